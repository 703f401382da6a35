"""Device memory of the plain FP64 form's calls (GPU tests): the partial sums of
mode splits are bounded, and a call that does not get its workspace takes less
of it instead of failing.

Tolerance: as for the form's edges, (2e-15 + 3e-16 N) sum_j |z1_j + i z2_j|
(cosines to 9e-16 of a mode's amplitude, amplitudes to 2^-53 twice, and the
rounding of the oracle's running sum).
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


def _tolerance(z1, z2):
    return (2e-15 + 3e-16 * len(z1)) * np.sum(np.hypot(z1, z2))


def _device(torch, *arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


# fewer points than the GPU holds blocks for, so the modes are split.  Allocations
# that fail: the first (then without splits), or the first two (then also with the
# records of 65,536 modes at a time; 70,000 modes take two such builds)
@pytest.mark.parametrize("dim,incompr,n,p,failures", [
    (2, False, 700, 3001, 1), (3, True, 700, 3001, 1), (2, False, 70_000, 130, 2), (3, True, 70_000, 130, 2),
])
def test_less_workspace_when_memory_is_short(gsc, dim, incompr, n, p, failures):
    torch = pytest.importorskip("torch")
    from gstools_core import _native
    rng = np.random.default_rng(dim + n)
    cov, z1, z2 = rng.normal(0.0, 0.6, (dim, n)), rng.standard_normal(n), rng.standard_normal(n)
    pos = rng.uniform(-40.0, 40.0, (dim, p))
    args = _device(torch, cov, z1, z2, pos)
    out = torch.full((dim, p) if incompr else (p,), float("nan"), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()
    gsc.release_buffers()
    assert _native.lib.gsc_selftest_fail_allocs(0, failures) == 0
    try:
        (gsc.summate_incompr_device if incompr else gsc.summate_device)(*args, out, stream=stream.cuda_stream)
    finally:
        _native.lib.gsc_selftest_fail_allocs(0, 0)
    stream.synchronize()
    gsc.device_status()
    ref = (oracle.summator_incompr if incompr else oracle.summator)(cov, z1, z2, pos, num_threads=NT)
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= _tolerance(z1, z2)


def test_no_workspace_at_all_is_reported(gsc):
    """Every attempt fails: the error of the last, and the next call computes."""
    torch = pytest.importorskip("torch")
    from gstools_core import _native
    rng = np.random.default_rng(4)
    n, p = 500, 2000
    cov, z1, z2, pos = rng.normal(0.0, 0.6, (2, n)), rng.standard_normal(n), rng.standard_normal(n), rng.uniform(0, 9, (2, p))
    args = _device(torch, cov, z1, z2, pos)
    out = torch.empty(p, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()
    gsc.release_buffers()
    assert _native.lib.gsc_selftest_fail_allocs(0, 100) == 0
    try:
        with pytest.raises(MemoryError, match="injected allocation failure"):
            gsc.summate_device(*args, out, stream=stream.cuda_stream)
    finally:
        _native.lib.gsc_selftest_fail_allocs(0, 0)
    gsc.summate_device(*args, out, stream=stream.cuda_stream)
    stream.synchronize()
    ref = oracle.summator(cov, z1, z2, pos, num_threads=NT)
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= _tolerance(z1, z2)


def test_partial_sums_of_a_large_cloud_are_bounded(gsc):
    """28.8 million 3-D vectors x 4096 modes: the last wave of blocks would be
    fuller with four splits, whose partial sums are 2.8 GB.  A call keeps at most
    256 MB of them (a quarter more as allocated) and its mode records."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    n, p = 4096, 28_800_000
    cov, z1, z2 = rng.normal(0.0, 0.3, (3, n)), rng.standard_normal(n), rng.standard_normal(n)
    args = _device(torch, cov, z1, z2)
    pos = torch.rand((3, p), dtype=torch.float64, device="cuda") * 100.0
    out = torch.empty((3, p), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()
    gsc.summate_incompr_device(*args, pos[:, :1000].contiguous(), out[:, :1000].contiguous(), stream=stream.cuda_stream)
    stream.synchronize()
    gsc.release_buffers()
    before = torch.cuda.mem_get_info()[0]
    gsc.summate_incompr_device(*args, pos, out, stream=stream.cuda_stream)
    stream.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= 400 << 20
    at = torch.from_numpy(rng.integers(0, p, 50)).cuda()
    ref = oracle.summator_incompr(cov, z1, z2, np.ascontiguousarray(pos[:, at].cpu().numpy()), num_threads=NT)
    assert np.max(np.abs(out[:, at].cpu().numpy() - ref)) <= _tolerance(z1, z2)
