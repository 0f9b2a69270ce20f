"""The batched form's two kernels on the same cells: the resident kernel (cells in shared memory from start to finish)
and the round scheme (RHS / solver kernels over a list of live cells) must give the same bits, because which of the two
integrates a cell depends on the size of its batch.  Calls that ask for the analytic Jacobian run the rounds, and at
constant volume, or with extended PLOG or fall-off reactions, these keep the forward differences: the same method."""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu

N = 700


def _mechanism(name):
    from laminarsmoke_b200 import mech
    from laminarsmoke_b200.mech import blob, chemkin, synthetic
    if name in ("xplog", "xfo"):
        from tests.test_gpu_extended import _mechanism as extended
        data, m = extended(name)
        return data, m.species, m.arrays
    if name == "syn28":
        s = synthetic.generate(28, 360, 7, physical=True)
        m = chemkin.compile_mechanism(s.kinetics, s.thermo)
        return blob.pack(m.arrays, m.species), m.species, m.arrays
    data, species = mech.load(name)
    return data, species, blob.unpack(data)[0]


def _states(name, species, A, n):
    if name.startswith("h2co"):
        Y, T = cells.h2co_mixing(species[:14], A["mw"][:14], n, seed=41)
        k = len(species) - 14
        if k:
            Y = np.concatenate([0.9 * Y, np.full((n, k), 0.1 / k)], axis=1)
    else:
        Y, T = cells.synthetic_mixing(species, A["mw"], n, 41, (900.0, 2200.0))
    T[::9] = 250.0             # skipped below tmin_chem
    T[4::50] = 7000.0          # above y_max_T: status -9
    Y[3::11, 0] = -1e-9        # clipped
    Y[5::13] *= 1.7            # renormalised
    return np.ascontiguousarray(Y.T), T


def _step(data, A, Y, T, dt, volume, precision, jacobian, **kw):
    """Every output of the step as bytes' worth of numpy arrays, and the kernel kinds that ran."""
    import torch
    from laminarsmoke_b200 import lsg
    n = T.size
    ctx = lsg.ReactionStep(lsg.Mechanism(data), tile=lsg.LSG_TILE_LANE, precision=precision, jacobian=jacobian,
                           tmin_chem=300.0, kernel_timing=1, **kw)
    dev = lambda x: torch.tensor(x, device="cuda")
    Yd, Td, dtd = dev(Y), dev(T), dev(dt)
    Q = torch.zeros(n, dtype=torch.float64, device="cuda")
    st = torch.zeros(n, dtype=torch.int32, device="cuda")
    ns = torch.zeros(n, dtype=torch.int32, device="cuda")
    cnt = torch.zeros((n, lsg.NCOUNTERS), dtype=torch.int64, device="cuda")
    out = dict(Q=Q, status=st, nsteps=ns, counters=cnt)
    if volume:
        rho = 101325.0 / (8314.4621 * T * (np.abs(Y) / A["mw"][:, None]).sum(0))
        ctx.step_cv_device(Yd, Td, dev(rho), dtd, **out)
    else:
        ctx.step_device(Yd, Td, dtd, **out)
    torch.cuda.synchronize()
    ctx.check()
    kinds = {k for k, (_, launches) in ctx.kernel_times().items() if launches}
    return dict(Y=Yd.cpu().numpy(), T=Td.cpu().numpy(), **{k: v.cpu().numpy() for k, v in out.items()}), kinds


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k].view(np.int64 if a[k].itemsize == 8 else np.int32),
                                      b[k].view(np.int64 if b[k].itemsize == 8 else np.int32), err_msg=k)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("name,volume", [("h2co", True), ("h2co+2", True), ("ch4", True), ("xplog", False), ("xfo", False),
                                         ("xfo", True)])
def test_resident_and_rounds_give_the_same_bits(cuda, name, volume, precision):
    data, species, A = _mechanism(name)
    Y, T = _states(name, species, A, N)
    dt = (1e-8 if name.startswith("x") else 1e-6) * 10.0 ** np.random.default_rng(4).uniform(-1.0, 0.0, N)
    for kw in (dict(), dict(max_steps=7)):   # to the end, and stopped on the way
        r, ran_r = _step(data, A, Y, T, dt, volume, precision, 0, **kw)
        s, ran_s = _step(data, A, Y, T, dt, volume, precision, 1, **kw)
        assert ran_r == {"group"} and "advance" in ran_s and "group" not in ran_s
        assert len(np.unique(r["status"])) >= 3
        _same(r, s)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_batch_size_does_not_show(cuda, precision):
    """28 species, 360 reactions at constant pressure: few cells fit a block, so that a small batch runs the resident
    kernel and a large one the rounds."""
    data, species, A = _mechanism("syn28")
    n = 148 * 32 * 12
    Y, T = _states("syn28", species, A, n)
    dt = np.full(n, 1e-9)
    whole, ran = _step(data, A, Y, T, dt, False, precision, 0)
    assert "advance" in ran and "group" not in ran
    part, ran = _step(data, A, np.ascontiguousarray(Y[:, :N]), T[:N], dt[:N], False, precision, 0)
    assert ran == {"group"}
    _same({k: np.ascontiguousarray(v[:N] if k == "counters" else v[..., :N]) for k, v in whole.items()}, part)


@pytest.mark.parametrize("name,precision,line", [("ch4", 1, 10 * 64), ("ch4", 0, 10 * 64), ("h2co+2", 1, 16 * 128),
                                                 ("h2co+2", 0, 16 * 48), ("h2co", 1, 28 * 128), ("h2co", 0, 28 * 48),
                                                 ("h2co+17", 1, 7 * 32)])
def test_large_calls_run_the_faster_kernel(cuda, name, precision, line):
    """The resident kernel up to `line` cells an SM (the cells that fit a block, so many times over), the rounds above; the
    cells are below tmin_chem, so that only the choice is run."""
    import torch
    data, species, A = _mechanism(name)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [sms * line, sms * line + 1]
    Y = np.full((len(species), sizes[-1]), 1.0)
    out = []
    for n, resident in zip(sizes, (True, False)):
        o, ran = _step(data, A, np.ascontiguousarray(Y[:, :n]), np.full(n, 290.0), np.full(n, 1e-6), False, precision, 0)
        assert (ran == {"group"}) == resident and ("init" in ran) != resident
        out.append(o)
    np.testing.assert_array_equal(out[0]["Y"], np.full((len(species), sizes[0]), 1.0 / len(species)))
    _same({k: np.ascontiguousarray(v[:sizes[0]] if k == "counters" else v[..., :sizes[0]]) for k, v in out[1].items()},
          out[0])


def test_call_too_large_for_the_rounds(cuda, h2co):
    """25 million cells: the rounds' records would take some 200 GB, so the resident kernel, which needs none, runs."""
    import torch
    from laminarsmoke_b200 import lsg
    n = 25000000
    ctx = lsg.ReactionStep(lsg.Mechanism(h2co[0]), tile=lsg.LSG_TILE_LANE, precision=1, tmin_chem=300.0)
    Y = torch.full((14, n), 2.0, dtype=torch.float64, device=cuda)
    T = torch.full((n,), 290.0, dtype=torch.float64, device=cuda)
    ctx.step_device(Y, T, 1e-6)
    torch.cuda.synchronize()
    ctx.check()
    assert bool((Y == 1.0 / 14.0).all())
