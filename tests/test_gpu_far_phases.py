"""The FP64 point form at phases of 2^32 to 1e13 and beyond, against the oracle
(GPU tests), and its time there.

Tolerance: as for the form's edges, (2e-15 + 3e-16 N) sum_j |z1_j + i z2_j|: the
phase has the oracle's bits at any size.  Time: phases of 1e9 to 1e13 take another
reduction to a turn and read their points again, some 60 integer instructions and a
few loads beside 110 to 190; a call of such phases is within 3 times one of small
phases (with CUDA's sincos() it was 8 to 9 times).
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


def _inputs(dim, n, p, extent, seed=0):
    rng = np.random.default_rng([dim, n, p, seed])
    return (rng.standard_normal((dim, n)), rng.standard_normal(n), rng.standard_normal(n),
            rng.uniform(-extent, extent, (dim, p)))


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("extent", [1e9, 5e9, 1e11, 2e12, 1e13, 1e15])
@pytest.mark.parametrize("p", [1, 700, 40_001])
def test_against_the_oracle(gsc, dim, extent, p):
    cov, z1, z2, pos = _inputs(dim, 75, p, extent)
    pos[:, ::7] *= 1e-9                      # small and large phases in one warp
    tol = (2e-15 + 3e-16 * 75) * np.sum(np.hypot(z1, z2))
    got = gsc.summate(cov, z1, z2, pos, form="plain")
    assert np.max(np.abs(got - oracle.summator(cov, z1, z2, pos, num_threads=NT))) <= tol
    if dim > 1:
        got = gsc.summate_incompr(cov, z1, z2, pos, form="plain")
        assert np.max(np.abs(got - oracle.summator_incompr(cov, z1, z2, pos, num_threads=NT))) <= tol


@pytest.mark.parametrize("extent", [1e9, 1e11])
def test_far_items_of_a_plan(gsc, extent):
    torch = pytest.importorskip("torch")
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    inputs = [_inputs(dim, 100, 5000, extent, seed=1) for dim in (1, 2, 3)]
    items = [{"cov": d(c), "z1": d(a), "z2": d(b), "pos": d(x),
              "out": torch.empty(5000, dtype=torch.float64, device="cuda")} for c, a, b, x in inputs]
    for r in (2, 4, 8):
        with gsc.Batch(items, form="plain", points_per_thread=r, tile_modes=8, units_per_block=4) as plan:
            plan.run()
            torch.cuda.synchronize()
        for (c, a, b, x), it in zip(inputs, items):
            tol = (2e-15 + 3e-16 * 100) * np.sum(np.hypot(a, b))
            ref = oracle.summator(c, a, b, x, num_threads=NT)
            assert np.max(np.abs(it["out"].cpu().numpy() - ref)) <= tol


@pytest.mark.parametrize("dim", [2, 3])
def test_time(gsc, dim):
    torch = pytest.importorskip("torch")
    out = torch.empty(100_000, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()

    def best(extent):
        args = [torch.from_numpy(a).cuda() for a in _inputs(dim, 500, 100_000, extent)]
        times = []
        for _ in range(15):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            gsc.summate_device(*args, out, stream=stream.cuda_stream)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    near, mid, far = best(100.0), best(1e10), best(1e12)
    print(f"dim {dim}: {near * 1e3:.0f}, {mid * 1e3:.0f}, {far * 1e3:.0f} us")
    assert mid <= 3.0 * near and far <= 3.0 * near
