"""The warp form (one warp a cell, all FP64): batches around the cells of a grid, mechanisms with and without room for
their tables in shared memory, reactions in and outside the packed form -- against the oracle, and bit for bit
independent of the batch a cell is in."""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu


def _mechanism(name):
    from laminarsmoke_b200 import mech
    from laminarsmoke_b200.mech import blob, chemkin, synthetic
    if name == "syn28":   # 28 species, 360 reactions: too large to be staged beside four warps
        s = synthetic.generate(28, 360, 7, physical=True)
        m = chemkin.compile_mechanism(s.kinetics, s.thermo)
        data, species = blob.pack(m.arrays, m.species), m.species
    else:
        data, species = mech.load(name)
    return data, blob.unpack(data)[0], species


def _states(A, species, name, n):
    if name.startswith("h2co"):
        Y, T = cells.h2co_mixing(species[:14], A["mw"][:14], n, seed=31)
        k = len(species) - 14
        if k:
            Y = np.concatenate([0.9 * Y, np.full((n, k), 0.1 / k)], axis=1)
    else:
        Y, T = cells.synthetic_mixing(species, A["mw"], n, 31, (900.0, 2200.0))
    T[::7] = 250.0
    Y[3::11, 0] = -1e-9
    return np.ascontiguousarray(Y.T), T


@pytest.mark.parametrize("name,n,dt", [("h2co", 2401, 1e-6), ("h2co+1", 5, 1e-6), ("h2co+2", 5, 1e-6),
                                       ("h2co+17", 5, 1e-6), ("ch4", 300, 1e-7), ("syn28", 9, 1e-9)])
def test_warp_form(cuda, name, n, dt):
    from laminarsmoke_b200 import lsg
    from oracle.oracle import OracleMechanism
    data, A, species = _mechanism(name)
    Y, T = _states(A, species, name, n)
    kw = dict(rtol=1e-10, atol=1e-16, tmin_chem=300.0)
    ctx = lsg.ReactionStep(lsg.Mechanism(data), tile=lsg.LSG_TILE_WARP, **kw)

    def step(k):
        y, t = Y[:, :k].copy(), T[:k].copy()   # the step works in place
        Q, st, ns = ctx.step(y, t, dt)
        return y, t, Q, st, ns

    whole = step(n)
    for k in (1, 2, 149):
        if k < n:
            for a, b in zip(whole, step(k)):
                np.testing.assert_array_equal(a[..., :k], b)
    m = min(n, 160)
    Yo, To, _, sto, _ = OracleMechanism(data).reaction_step(np.ascontiguousarray(Y[:, :m].T), T[:m], dt, nthreads=8, **kw)
    np.testing.assert_array_equal(whole[3][:m], sto)
    assert np.abs(whole[1][:m] - To).max() <= 1e-6 * To.max()
    assert np.abs(whole[0][:, :m].T - Yo).max() <= 1e-9
