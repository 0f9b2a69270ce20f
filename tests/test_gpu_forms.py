"""Which form runs a call: the resident kernel's tile on mechanisms of which no cell fits a block (under capture, with
the analytic Jacobian), and the autotuner's choice among the forms."""
import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rich():
    """15 species, 800 reactions: the rates of one evaluation alone exceed what the resident kernel has for them."""
    from laminarsmoke_b200.mech import blob, chemkin, synthetic
    s = synthetic.generate(15, 40, 7, physical=True)
    lines = s.kinetics.split("\n")
    first, end = lines.index("REACTIONS") + 1, len(lines) - 1 - lines[::-1].index("END")
    m = chemkin.compile_mechanism("\n".join(lines[:first] + 20 * lines[first:end] + lines[end:]), s.thermo)
    return blob.pack(m.arrays, m.species), m.species, m.arrays


def _fields(species, A, n):
    import torch
    Y, T = cells.synthetic_mixing(species, A["mw"], n, 17, (900.0, 2200.0))
    return torch.tensor(np.ascontiguousarray(Y.T), device="cuda"), torch.tensor(T, device="cuda")


def _step(ctx, Y, T, dt):
    import torch
    from laminarsmoke_b200 import lsg
    Yd, Td = Y.clone(), T.clone()
    cnt = torch.zeros((T.shape[0], lsg.NCOUNTERS), dtype=torch.int64, device="cuda")
    ctx.step_device(Yd, Td, dt, counters=cnt)
    torch.cuda.synchronize()
    ctx.check()
    return Yd.cpu().numpy(), Td.cpu().numpy(), cnt.cpu().numpy()


def test_group_tile_without_room_keeps_the_differences(cuda, rich):
    """LSG_TILE_GROUP takes forward differences whatever the Jacobian option says, in the rounds too."""
    from laminarsmoke_b200 import lsg
    data, species, A = rich
    Y, T = _fields(species, A, 150)
    out = [_step(lsg.ReactionStep(lsg.Mechanism(data), tile=tile, precision=lsg.LSG_PRECISION_MIXED, jacobian=j), Y, T, 1e-9)
           for tile, j in ((lsg.LSG_TILE_LANE, 0), (lsg.LSG_TILE_GROUP, 0), (lsg.LSG_TILE_GROUP, 1))]
    cnt = out[2][2]
    assert cnt[:, 2].min() > 0 and (cnt[:, 7] == 16 * cnt[:, 2]).all()   # 16 evaluations a Jacobian
    for o in out[1:]:
        for a, b in zip(out[0], o):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_group_tile_without_room_is_captured(cuda, rich, precision):
    """A captured call cannot wait for the host as the rounds do: it is the block form's step, bit for bit."""
    import torch
    from laminarsmoke_b200 import lsg
    data, species, A = rich
    Y, T = _fields(species, A, 150)
    m = lsg.Mechanism(data)
    Yr, Tr, _ = _step(lsg.ReactionStep(m, tile=lsg.LSG_TILE_BLOCK, precision=precision), Y, T, 1e-9)
    ctx = lsg.ReactionStep(m, tile=lsg.LSG_TILE_GROUP, precision=precision)
    _step(ctx, Y, T, 1e-9)   # a first call makes the buffers
    Yd, Td = Y.clone(), T.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.step_device(Yd, Td, 1e-9)
    for _ in range(2):
        Yd.copy_(Y)
        Td.copy_(T)
        graph.replay()
        torch.cuda.synchronize()
        ctx.check()
        np.testing.assert_array_equal(Td.cpu().numpy(), Tr)
        np.testing.assert_array_equal(Yd.cpu().numpy(), Yr)
    graph.reset()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_autotuner_skips_a_form_without_room(cuda, rich, precision):
    """Nothing but the rounds takes this mechanism below 32 species: the tuner says so and the step is theirs."""
    from laminarsmoke_b200 import lsg
    data, species, A = rich
    Y, T = _fields(species, A, 1100)
    m = lsg.Mechanism(data)
    ctx = lsg.ReactionStep(m, precision=precision, autotune=1)
    got = _step(ctx, Y, T, 1e-10)
    tile, width, rates = ctx.tuning()
    assert tile == lsg.LSG_TILE_LANE and {k for k, v in rates.items() if v > 0} == {"rounds16", "rounds32"}
    Yr, Tr, cnt = _step(lsg.ReactionStep(m, tile=lsg.LSG_TILE_LANE, precision=precision), Y, T, 1e-10)
    if width == 16:   # the lanes of a default call
        for a, b in zip(got, (Yr, Tr, cnt)):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_autotuner_honours_the_analytic_jacobian(cuda, h2co, precision):
    """A tuned context that asks for the analytic Jacobian integrates with it: one evaluation a Jacobian (its
    temperature column), whichever form would be the faster with differences."""
    from laminarsmoke_b200 import lsg
    data, species, A = h2co
    Y, T = cells.h2co_mixing(species, A["mw"], 2048, seed=8)
    import torch
    Y, T = torch.tensor(np.ascontiguousarray(Y.T), device=cuda), torch.tensor(T, device=cuda)
    ctx = lsg.ReactionStep(lsg.Mechanism(data), precision=precision, autotune=1, jacobian=lsg.LSG_JACOBIAN_ANALYTIC)
    cnt = _step(ctx, Y, T, 1e-5)[2]
    assert cnt[:, 2].sum() > 0 and (cnt[:, 7] == cnt[:, 2]).all()
    assert {k for k, v in ctx.tuning()[2].items() if v > 0} == {"rounds16", "rounds32"}


def test_autotuner_times_each_kernel_once(cuda, h2co):
    """Rounds and resident kernel are candidates of their own, and a tuned context's step sequences run one by one
    whichever of the two won, as LSG_TILE_LANE's do."""
    import torch
    from laminarsmoke_b200 import lsg
    data, species, A = h2co
    Y, T = cells.h2co_mixing(species, A["mw"], 1500, seed=8)
    Y, T = torch.tensor(np.ascontiguousarray(Y.T), device=cuda), torch.tensor(T, device=cuda)
    ctx = lsg.ReactionStep(lsg.Mechanism(data), precision=lsg.LSG_PRECISION_MIXED, autotune=1)
    got = _step(ctx, Y, T, 1e-5)
    tile, width, rates = ctx.tuning()
    assert {k for k, v in rates.items() if v > 0} == {"rounds16", "rounds32", "persistent", "group_4", "group_2"}
    assert ctx.launches() > 1000   # hundreds of rounds of four launches each, for two lane widths
    if width in (16, 4):
        want = _step(lsg.ReactionStep(lsg.Mechanism(data), precision=lsg.LSG_PRECISION_MIXED), Y, T, 1e-5)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
    Yd, Td = Y.clone(), T.clone()
    if tile in (lsg.LSG_TILE_LANE, lsg.LSG_TILE_GROUP):
        assert not ctx.step_sequence_graph(Yd, Td, 1e-5, 2)
    torch.cuda.synchronize()
    ctx.check()
