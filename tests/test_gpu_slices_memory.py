"""The sliced FP64 grids' ways out when device memory is short, by allocations
that fail in a row (injected on the host): the digits of fewer rows at a time, no
splits of the modes, at last the FP64 MMA kernels alone (GPU tests).

Slabs of rows do not enter a value's sums: the same bits.  Without splits the
shared accumulator of levels 4 to 6 is truncated after other pairs of k-blocks:
the form's tolerance, as for the FP64 MMA: sum_j |z_j| |phase_j| 2^-51 for the
phases' rounding, N sum |z| 2^-53 of the oracle's and N max |z| 2^-50 of this form's
sums.  8192 modes are two segments, each split.
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


@pytest.mark.parametrize("shape,n,incompr", [((9, 130, 70), 200, False), ((1200, 40), 200, True), ((3, 90, 30), 8192, False)])
def test_every_step(gsc, shape, n, incompr):
    torch = pytest.importorskip("torch")
    from gstools_core import _native
    rng = np.random.default_rng([*shape, n])
    dim, points = len(shape), int(np.prod(shape))
    cov, z1, z2 = rng.normal(0.0, 0.4, (dim, n)), rng.standard_normal(n), rng.standard_normal(n)
    axes = tuple(rng.uniform(-20.0, 20.0) + rng.uniform(0.5, 1.5) * np.arange(s) for s in shape)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = (d(cov), d(z1), d(z2), tuple(d(a) for a in axes))
    call = gsc.summate_incompr_structured_device if incompr else gsc.summate_structured_device
    stream = torch.cuda.current_stream()

    def run(failures):
        out = torch.full((dim, points) if incompr else (points,), float("nan"), dtype=torch.float64, device="cuda")
        gsc.release_buffers()
        assert _native.lib.gsc_selftest_fail_allocs(0, failures) == 0
        try:
            call(*args, out, stream=stream.cuda_stream)
        finally:
            _native.lib.gsc_selftest_fail_allocs(0, 0)
        stream.synchronize()
        gsc.device_status()
        return out.cpu().numpy()

    want = run(0)
    flat = np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(dim, -1))
    ref = (oracle.summator_incompr if incompr else oracle.summator)(cov, z1, z2, flat, num_threads=NT)
    a = np.hypot(z1, z2)
    phase = np.abs(cov).T @ np.array([np.max(np.abs(x)) for x in axes])
    tol = np.sum(a * phase) * 2.0**-51 + n * np.sum(a) * 2.0**-53 + n * np.max(a) * 2.0**-50
    assert np.max(np.abs(want - ref)) <= tol
    # 10 (3) row tiles: slabs of 2 and 1 (0 is raised to 1), then no splits, then the FP64 MMA
    slabs = 2 if shape != (3, 90, 30) else 1
    for failures in range(1, slabs + 1):
        assert np.array_equal(run(failures), want), failures
    assert np.max(np.abs(run(slabs + 1) - ref)) <= tol
    mma = run(slabs + 2)
    assert not np.array_equal(mma, want)
    assert np.max(np.abs(mma - ref)) <= tol
    with pytest.raises(MemoryError, match="injected allocation failure"):
        run(slabs + 3)
    assert np.array_equal(run(0), want)
