"""Two threads, a context and a stream each, whose calls launch the same kernel with different amounts of shared memory
at the same time: no call may fail because of the other's, and each gets its own answer."""
import threading

import numpy as np
import pytest

from laminarsmoke_b200 import cells

pytestmark = pytest.mark.gpu


def _states(name, species, A, n):
    if name.startswith("h2co"):
        Y, T = cells.h2co_mixing(species[:14], A["mw"][:14], n, seed=5)
        k = len(species) - 14
        if k:
            Y = np.concatenate([0.9 * Y, np.full((n, k), 0.1 / k)], axis=1)
        return Y, T
    return cells.synthetic_mixing(species, A["mw"], n, 5, (900.0, 2200.0))


def _worker(name, n, call, kw):
    """A function that makes `calls` calls in a row and returns the last one's outputs as numpy arrays."""
    import torch
    from laminarsmoke_b200 import lsg, mech
    from laminarsmoke_b200.mech import blob
    data, species = mech.load(name)
    Y, T = _states(name, species, blob.unpack(data)[0], n)
    # cells below tmin_chem are renormalised only, so that the calls are short and their launches close together
    ctx = lsg.ReactionStep(lsg.Mechanism(data), tmin_chem=5000.0, **kw)
    stream = torch.cuda.Stream()
    Y0, T0 = torch.tensor(np.ascontiguousarray(1.5 * Y.T), device="cuda"), torch.tensor(T, device="cuda")
    Yd = Y0.clone()
    torch.cuda.synchronize()

    def run(calls):
        with torch.cuda.stream(stream):
            Yd.copy_(Y0)
            for _ in range(calls):
                if call == "properties":
                    out = list(ctx.properties_device(Y0, T0).values())
                else:
                    ctx.step_device(Yd, T0, 1e-6)
                    out = [Yd]
        stream.synchronize()
        return [o.cpu().numpy() for o in out]
    return run


@pytest.mark.parametrize("call,kw,one,two", [
    ("step", dict(tile=1), ("h2co", 1), ("h2co", 3000)), ("step", dict(tile=2, precision=1), ("h2co", 1), ("h2co", 3000)),
    ("step", dict(), ("h2co+25", 3), ("h2co+90", 3)), ("properties", dict(), ("h2co", 500), ("ch4", 500))],
    ids=["warp", "resident", "block", "properties"])
def test_threads_with_different_sizes(cuda, call, kw, one, two):
    runs = [_worker(name, n, call, kw) for name, n in (one, two)]
    calls = 4000
    want = [r(calls) for r in runs]
    errors = []
    start = threading.Barrier(2)

    def loop(k):
        try:
            start.wait()
            for a, b in zip(runs[k](calls), want[k]):
                np.testing.assert_array_equal(a, b)
        except Exception as e:   # noqa: BLE001 (reported by the test's thread)
            errors.append(f"thread {k}: {e}")

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
