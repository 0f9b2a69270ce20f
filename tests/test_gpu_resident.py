"""The batched form's resident kernel (many cells of a block in shared memory): batch sizes around its tiles -- one
cell, one cell more and less than the cells a warp and a block hold, more cells than the grid holds at once -- against
the oracle, and bit for bit independent of the batch a cell is in."""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu

N = 148 * 28 + 5   # more than one block-full on every SM of a B200


def _states(name, n):
    from laminarsmoke_b200 import mech
    from laminarsmoke_b200.mech import blob
    data, species = mech.load(name)
    A, _ = blob.unpack(data)
    if name == "h2co":
        Y, T = cells.h2co_mixing(species, A["mw"], n, seed=23)
    else:
        Y, T = cells.synthetic_mixing(species, A["mw"], n, 23, (900.0, 2200.0))
    T[::7] = 250.0             # skipped below tmin_chem
    Y[3::11, 0] = -1e-9        # clipped
    Y[5::13] *= 1.7            # renormalised
    return data, A, np.ascontiguousarray(Y.T), T


def _step(ctx, A, Y, T, dt, reactor):
    Y, T = Y.copy(), T.copy()
    if reactor == "v":
        rho = 101325.0 / (8314.4621 * T * (np.abs(Y) / A["mw"][:, None]).sum(0))
        Q, st, ns = ctx.step_cv(Y, T, rho, dt)
    else:
        Q, st, ns = ctx.step(Y, T, dt)
    return Y, T, Q, st, ns


@pytest.mark.parametrize("name,reactor,precision", [("h2co", "p", 1), ("h2co", "v", 0), ("ch4", "p", 1), ("ch4", "v", 1)])
def test_resident_batch_sizes(cuda, name, reactor, precision):
    from laminarsmoke_b200 import lsg
    n = N if name == "h2co" else 148 * 10 + 3
    data, A, Y, T = _states(name, n)
    dt = 1e-6 * 10.0 ** np.random.default_rng(4).uniform(-1.0, 0.0, n)   # local time steps
    ctx = lsg.ReactionStep(lsg.Mechanism(data), tile=lsg.LSG_TILE_LANE, precision=precision, tmin_chem=300.0)
    whole = _step(ctx, A, Y, T, dt, reactor)
    assert set(np.unique(whole[3])) <= {0, 2}
    for k in (1, 2, 3, 27, 29, 148, 149, 297):
        part = _step(ctx, A, np.ascontiguousarray(Y[:, :k]), T[:k], dt[:k], reactor)
        for a, b in zip(whole, part):
            np.testing.assert_array_equal(a[..., :k], b)


@pytest.mark.parametrize("name", ["h2co", "ch4"])
def test_resident_against_oracle(cuda, name):
    from laminarsmoke_b200 import lsg
    from oracle.oracle import OracleMechanism
    data, A, Y, T = _states(name, 149)
    ctx = lsg.ReactionStep(lsg.Mechanism(data), tile=lsg.LSG_TILE_LANE, precision=1, tmin_chem=300.0,
                           rtol=1e-10, atol=1e-16)
    Yg, Tg, _, st, _ = _step(ctx, A, Y, T, 1e-6, "p")
    Yo, To, _, sto, _ = OracleMechanism(data).reaction_step(np.ascontiguousarray(Y.T), T, 1e-6, nthreads=8, rtol=1e-10,
                                                           atol=1e-16, tmin_chem=300.0)
    np.testing.assert_array_equal(st, sto)
    assert np.abs(Tg - To).max() <= 1e-6 * To.max()
    assert np.abs(Yg.T - Yo).max() <= 1e-9
