"""The block form at the most reactions that its shared memory has held from the start: 227 KB less the solver's vectors."""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu


def _most_reactions(nc, bt):
    """(17 bt + 3 nc + nr + bt / 32 + 5) doubles, 2 bt + bt / 32 + 1 ints, 64 + 16 bytes, in 227 KB."""
    return (227 * 1024 - 80 - 4 * (2 * bt + bt // 32 + 1)) // 8 - (17 * bt + 3 * nc + bt // 32 + 5)


def _mechanism(nc, nr):
    """nr reactions: those of a synthetic mechanism, over and over."""
    from laminarsmoke_b200.mech import blob, chemkin, synthetic
    s = synthetic.generate(nc, 6 * nc, 7)
    lines = s.kinetics.split("\n")
    first, end = lines.index("REACTIONS") + 1, len(lines) - 1 - lines[::-1].index("END")
    reactions, now = [], []
    for line in lines[first:end]:   # a reaction and its auxiliary lines
        if "=" in line and now:
            reactions.append(now)
            now = []
        now.append(line)
    reactions.append(now)
    body = [line for j in range(nr) for line in reactions[j % len(reactions)]]
    m = chemkin.compile_mechanism("\n".join(lines[:first] + body + lines[end:]), s.thermo)
    assert int(m.arrays["dims"][1]) == nr
    return blob.pack(m.arrays, m.species), m.species, m.arrays


@pytest.mark.parametrize("nc,bt", [(60, 128), (200, 256), (500, 512)])
def test_block_most_reactions(cuda, nc, bt):
    import torch
    from laminarsmoke_b200 import lsg
    from oracle.oracle import OracleMechanism
    data, species, A = _mechanism(nc, _most_reactions(nc, bt))
    Y, T = cells.synthetic_mixing(species, A["mw"], 3, seed=9, t_range=(800.0, 2400.0))
    m = lsg.Mechanism(data)
    y = np.ascontiguousarray(np.concatenate([Y, T[:, None]], axis=1).T)
    yd = torch.tensor(y, device=cuda)
    dy = torch.zeros_like(yd)
    ctx = lsg.ReactionStep(m, tmin_chem=3000.0)
    ctx.rhs_device(yd, dy)
    Yd, Td = torch.tensor(np.ascontiguousarray(2.0 * Y.T), device=cuda), torch.tensor(T, device=cuda)
    ctx.step_device(Yd, Td, 1e-9)   # below tmin_chem: renormalised
    torch.cuda.synchronize()
    ctx.check()
    np.testing.assert_allclose(Yd.cpu().numpy(), Y.T, rtol=1e-14)
    om = OracleMechanism(data)
    for k in range(3):   # as for the mechanism's own reactions; every reaction comes up to 86 times
        ref, _ = om.rhs(y[:, k])
        np.testing.assert_allclose(dy.cpu().numpy()[:, k], ref, rtol=1e-9, atol=1e-12 * np.abs(ref).max())
