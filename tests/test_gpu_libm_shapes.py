"""Launch shapes of the sincos() form of the FP64 point kernels: one and four
points per thread, against the oracle, and the time of small calls (GPU tests).

Tolerance: phases and sums are those of the oracle but for CUDA's and glibc's
sincos (2 ulp) and the order of split sums: (4e-16 + 2^-53 (N + 64)) sum_j |z_j|
and the projector weights' |w_j| <= 1.
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n,p", [(1, 1), (64, 1), (33, 129), (1000, 700), (200, 100_001), (40, 160_000)])
def test_against_the_oracle(gsc, dim, n, p):
    rng = np.random.default_rng([dim, n, p])
    cov, z1, z2 = rng.normal(0.0, 0.6, (dim, n)), rng.standard_normal(n), rng.standard_normal(n)
    pos = rng.uniform(-40.0, 40.0, (dim, p))
    tol = (8e-16 + 2.0**-53 * (n + 64)) * np.sum(np.abs(z1) + np.abs(z2))
    got = gsc.summate(cov, z1, z2, pos, form="plain_libm")
    assert np.max(np.abs(got - oracle.summator(cov, z1, z2, pos, num_threads=NT))) <= tol
    if dim > 1:
        got = gsc.summate_incompr(cov, z1, z2, pos, form="plain_libm")
        assert np.max(np.abs(got - oracle.summator_incompr(cov, z1, z2, pos, num_threads=NT))) <= 2.0 * tol


def test_time_of_a_small_call(gsc):
    """One 3-D point x 64 modes: a thread's 32 modes in turn, as in the plain form, whose
    chain per mode is about a third as long.  (With four points per thread, three of
    them past the end, it took 8 times the plain form's call.)"""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(0)
    args = [torch.from_numpy(a).cuda() for a in
            (rng.normal(0.0, 0.6, (3, 64)), rng.standard_normal(64), rng.standard_normal(64), rng.uniform(0, 9, (3, 1)))]
    out = torch.empty(1, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()

    def best(form):
        times = []
        for _ in range(20):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(10):
                gsc.summate_device(*args, out, form=form, stream=stream.cuda_stream)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1) * 100.0)
        return min(times)

    plain, libm = best("plain"), best("plain_libm")
    print(f"plain {plain:.1f}, sincos() {libm:.1f} us")
    assert libm <= 4.0 * plain
