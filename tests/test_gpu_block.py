"""Block-per-cell step (mechanisms of 32 to 511 species) against the CPU oracle.

The H2/CO mechanism padded with chemically inert N2 copies keeps the real
chemistry's stiffness while the cell has 45, 165 or 315 ODE components, which
exercises the 128-, 256- and 512-thread blocks; the synthetic 120-species
mechanism is the large-mechanism configuration's chemistry.
"""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu

RTOL_T = 1e-6
ATOL_Y = 1e-9


def _padded_states(k, n, seed):
    from laminarsmoke_b200 import mech
    from laminarsmoke_b200.mech import blob
    data, species = mech.load(f"h2co+{k}")
    A, _ = blob.unpack(data)
    Y, T = cells.h2co_mixing(species[:14], A["mw"][:14], n, seed=seed)
    Y = np.concatenate([Y * 0.9, np.full((n, k), 0.1 / k)], axis=1)
    return data, Y, T


def _run(data, Y, T, dt, precision=0, **kw):
    import torch
    from laminarsmoke_b200 import lsg
    from oracle.oracle import OracleMechanism
    m = lsg.Mechanism(data)
    ctx = lsg.ReactionStep(m, precision=precision,
                           **{k: v for k, v in kw.items() if k in ("max_steps", "tmin_chem", "rtol", "atol")})
    n = Y.shape[0]
    Yd = torch.tensor(np.ascontiguousarray(Y.T), device="cuda")
    Td = torch.tensor(T, device="cuda")
    st = torch.zeros(n, dtype=torch.int32, device="cuda")
    ns = torch.zeros(n, dtype=torch.int32, device="cuda")
    Q = torch.zeros(n, dtype=torch.float64, device="cuda")
    ctx.step_device(Yd, Td, dt, Q=Q, status=st, nsteps=ns)
    torch.cuda.synchronize()
    ctx.check()
    kinds = ctx.kernel_times()
    Yo, To, Qo, sto, cnt = OracleMechanism(data).reaction_step(Y, T, dt, nthreads=8, **kw)
    return (Yd.cpu().numpy().T, Td.cpu().numpy(), Q.cpu().numpy(), st.cpu().numpy(), ns.cpu().numpy()), \
        (Yo, To, Qo, sto, cnt)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("k,ncells", [(30, 512), (150, 64), (300, 16)], ids=["n45", "n165", "n315"])
def test_block_padded_parity(cuda, k, ncells, precision):
    """FP64 block form, and the mixed-precision form: the tensor-core inverse of one 128-row tile (45
    components) or the in-place multi-tile inverse (165: two row tiles, 315: four), refined on the FP64
    residual."""
    data, Y, T = _padded_states(k, ncells, seed=11)
    (Yg, Tg, Qg, stg, nsg), (Yo, To, Qo, sto, cnt) = _run(data, Y, T, 1e-5, precision=precision)
    np.testing.assert_array_equal(stg, sto)
    rel_T = np.abs(Tg - To) / To
    abs_Y = np.abs(Yg - Yo).max(axis=1)
    same = nsg == cnt[:, 0]
    print(f"n={k + 15} precision={precision}: max rel T err {rel_T.max():.3e}, max abs Y err {abs_Y.max():.3e}, "
          f"cells within Y bound {np.mean(abs_Y <= ATOL_Y):.4f}, identical step counts {same.mean():.4f}")
    assert rel_T.max() <= RTOL_T
    # Rounding-level differences (tree-ordered sums over up to 315 components) send a few cells down a
    # different step sequence, which moves them by ~1e-8; the larger the system the more often.
    assert np.mean(abs_Y <= ATOL_Y) >= 0.9
    assert abs_Y.max() <= 1e-7
    np.testing.assert_allclose(Qg, Qo, rtol=1e-4, atol=1e-3 * np.abs(Qo).max())


def test_block_padded_tight(cuda):
    data, Y, T = _padded_states(30, 64, seed=12)
    (Yg, Tg, Qg, stg, nsg), (Yo, To, Qo, sto, cnt) = _run(data, Y, T, 1e-5, rtol=1e-10, atol=1e-16)
    assert np.abs(Tg - To).max() / To.min() <= RTOL_T
    assert np.abs(Yg - Yo).max() <= ATOL_Y


@pytest.mark.parametrize("k,ncells", [(18, 5), (21, 1), (22, 149), (49, 3), (82, 3), (105, 3), (113, 5), (114, 3)],
                         ids=["n33", "n36", "n37", "n64", "n97", "n120", "n128", "n129"])
def test_block_shared_factors_sizes(cuda, k, ncells):
    """FP64 factors in shared memory: component counts around the panels of eight columns, the substitution's four
    columns and the 32 rows of a lane group, the largest that it takes and the first that it does not."""
    data, Y, T = _padded_states(k, ncells, seed=13)
    (Yg, Tg, Qg, stg, nsg), (Yo, To, Qo, sto, cnt) = _run(data, Y, T, 1e-6, rtol=1e-10, atol=1e-16)
    np.testing.assert_array_equal(stg, sto)
    assert np.abs(Tg - To).max() / To.min() <= RTOL_T
    assert np.abs(Yg - Yo).max() <= ATOL_Y


@pytest.mark.parametrize("name", ["syn120", "syn500"])
def test_block_rhs_synthetic(cuda, name):
    """Thermo + rates of the 120- and 500-species synthetic mechanisms (800 / 3000
    reactions, third bodies, Troe fall-off) against the oracle's RHS."""
    import torch
    from laminarsmoke_b200 import lsg, mech
    from laminarsmoke_b200.mech import blob
    from oracle.oracle import OracleMechanism
    data, species = mech.load(name)
    A, _ = blob.unpack(data)
    Y, T = cells.synthetic_mixing(species, A["mw"], 48, seed=9, t_range=(800.0, 2400.0))
    y = np.ascontiguousarray(np.concatenate([Y, T[:, None]], axis=1).T)
    m = lsg.Mechanism(data)
    ctx = lsg.ReactionStep(m)
    yd = torch.tensor(y, device="cuda")
    dy = torch.zeros_like(yd)
    qr = torch.zeros(y.shape[1], dtype=torch.float64, device="cuda")
    ctx.rhs_device(yd, dy, qr=qr)
    torch.cuda.synchronize()
    ctx.check()
    dyg, qg = dy.cpu().numpy(), qr.cpu().numpy()
    om = OracleMechanism(data)
    for k in range(y.shape[1]):
        ref, qref = om.rhs(y[:, k])
        scale = np.abs(ref).max()
        np.testing.assert_allclose(dyg[:, k], ref, rtol=1e-9, atol=1e-12 * scale)
        assert abs(qg[k] - qref) <= 1e-9 * abs(qref) + 1e-6


def test_block_synthetic_120_step(cuda):
    """One step of the synthetic 120-species chemistry (T ~ U[800, 2400] K,
    dt = 5e-6 s) runs to valid statuses.  This chemistry is so stiff (time
    scales near 1e-13 s) that most cells end in Newton convergence failures in
    the oracle as well, after thousands of steps, so which cells fail depends on
    rounding: its parity is checked through the RHS above, the block step's
    through the padded H2/CO cases."""
    from laminarsmoke_b200 import mech
    from laminarsmoke_b200.mech import blob
    data, species = mech.load("syn120")
    A, _ = blob.unpack(data)
    Y, T = cells.synthetic_mixing(species, A["mw"], 24, seed=3, t_range=(800.0, 2400.0))
    (Yg, Tg, Qg, stg, nsg), _ = _run(data, Y, T, 5e-6)
    assert np.all(np.isin(stg, [2, -1, -2, -4, -5, -6]))
    assert np.all(np.isfinite(Yg)) and np.all(np.isfinite(Tg))
    np.testing.assert_allclose(Yg.sum(axis=1), 1.0, atol=1e-12)



@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_block_synthetic_120p_step(cuda, precision):
    """One step of the physically bounded 120-species / 800-reaction synthetic chemistry (barriers no lower
    than the endothermicity, rate constants at the collision limit; T ~ U[800, 2400] K, dt = 5e-6 s,
    thousands of BDF steps per cell) against the oracle.  At the default tolerances rounding-level
    differences move the step sequences of such long integrations apart by O(rtol); with rtol 1e-10 both
    integrations converge on the exact solution and are compared at the usual bounds."""
    from laminarsmoke_b200 import mech
    from laminarsmoke_b200.mech import blob
    data, species = mech.load("syn120p")
    A, _ = blob.unpack(data)
    Y, T = cells.synthetic_mixing(species, A["mw"], 32, seed=3, t_range=(800.0, 2400.0))
    for rtol, atol in ((1e-7, 1e-12), (1e-10, 1e-16)):
        (Yg, Tg, Qg, stg, nsg), (Yo, To, Qo, sto, cnt) = _run(data, Y, T, 5e-6, precision=precision, rtol=rtol,
                                                              atol=atol)
        rel_T = np.abs(Tg - To) / To
        abs_Y = np.abs(Yg - Yo).max(axis=1)
        print(f"syn120p precision={precision} rtol {rtol:g}: steps/cell {nsg.mean():.0f}, statuses equal {np.mean(stg == sto):.3f}, max rel T err {rel_T.max():.3e}, "
              f"max abs Y err {abs_Y.max():.3e}, cells within 1e-9 {np.mean(abs_Y <= ATOL_Y):.3f}, "
              f"steps {cnt[:, 0].mean():.0f}", flush=True)
    np.testing.assert_array_equal(stg, sto)
    assert np.all(stg == 2)
    assert rel_T.max() <= RTOL_T
    assert np.mean(abs_Y <= ATOL_Y) >= 0.9 and abs_Y.max() <= 1e-7
