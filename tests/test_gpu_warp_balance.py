"""The warp form's share of a mesh among the SMs: cells in the order of a mesh whose hot cells lie in a few columns."""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drg", [False, True], ids=["step", "drg"])
def test_hot_columns_take_no_longer_than_shuffled_cells(cuda, h2co, drg):
    """Lines of twice as many cells as there are SMs, ten hot columns: no more than half as long again as the same cells
    in random order (with the columns on ten SMs, several times as long), and the same result for every cell."""
    import torch
    from laminarsmoke_b200 import lsg
    data, species, A = h2co
    rows, line = 40, 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = rows * line
    Y, T = cells.h2co_mixing(species, A["mw"], n, seed=6, t_range=(1500.0, 2000.0))
    T[np.arange(n) % line >= 10] = 290.0   # below tmin_chem
    order = np.random.default_rng(2).permutation(n)
    ctx = lsg.ReactionStep(lsg.Mechanism(data), tile=lsg.LSG_TILE_WARP, tmin_chem=300.0)
    key = [species.index(s) for s in ("H2", "O2", "CO")]

    def run(pick):
        Y0 = torch.tensor(np.ascontiguousarray(Y[pick].T), device=cuda)
        T0 = torch.tensor(T[pick], device=cuda)
        best = None
        for _ in range(3):
            Yd, Td = Y0.clone(), T0.clone()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            if drg:
                ctx.step_drg_device(Yd, Td, 1e-5, key, min_T=300.0, first_cell_options_only=False)
            else:
                ctx.step_device(Yd, Td, 1e-5)
            b.record()
            torch.cuda.synchronize()
            ms = a.elapsed_time(b)
            best = ms if best is None else min(best, ms)
        ctx.check()
        return best, Yd.cpu().numpy(), Td.cpu().numpy()

    t_mesh, Ym, Tm = run(np.arange(n))
    t_mixed, Ys, Ts = run(order)
    print(f"mesh order {t_mesh:.1f} ms, shuffled {t_mixed:.1f} ms")
    np.testing.assert_array_equal(Ym[:, order], Ys)
    np.testing.assert_array_equal(Tm[order], Ts)
    assert t_mesh <= 1.5 * t_mixed
