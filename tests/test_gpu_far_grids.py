"""FP64 grids whose phases reach 2^32 to 1e13: accuracy against the oracle, and
the time of the sliced form (GPU tests).

Tolerance: a phase is a sum of one rounded product per axis here and in the oracle,
in another order: sum_j |z_j| |phase_j| 2^-51, beside the rounding of the sums
(N sum |z| 2^-53 in the oracle, N max |z| 2^-50 here).
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


def _inputs(shape, n, origin):
    rng = np.random.default_rng([*shape, n])
    axes = tuple(origin + np.arange(s, dtype=np.float64) for s in shape)
    return rng.normal(0.0, 0.3, (len(shape), n)), rng.standard_normal(n), rng.standard_normal(n), axes


def _check(got, ref, cov, z1, z2, axes):
    a = np.hypot(z1, z2)
    phase = np.abs(cov).T @ np.array([np.max(np.abs(x)) for x in axes])
    tol = np.sum(a * phase) * 2.0**-51 + len(a) * np.sum(a) * 2.0**-53 + len(a) * np.max(a) * 2.0**-50
    assert np.max(np.abs(got - ref)) <= tol


@pytest.mark.parametrize("shape", [(45, 37), (3, 20, 33)])
@pytest.mark.parametrize("origin", [4e9, 1e11, 5e12])
@pytest.mark.parametrize("incompr", [False, True])
def test_against_the_oracle(gsc, shape, origin, incompr):
    cov, z1, z2, axes = _inputs(shape, 70, origin)
    flat = np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(len(shape), -1))
    call, want = ((gsc.summate_incompr_structured, oracle.summator_incompr) if incompr
                  else (gsc.summate_structured, oracle.summator))
    _check(call(cov, z1, z2, axes), want(cov, z1, z2, flat, num_threads=NT), cov, z1, z2, axes)


def test_one_far_mode_in_exact_arithmetic(gsc):
    """A single mode of short wave number and coordinates, whose products are exact:
    the cosine of a phase of 2^40 to FP64 accuracy."""
    k, x0 = 4194305.0, 262144.5                       # 23 and 20 bits
    axes = (x0 + np.arange(40.0), np.arange(30.0))
    flat = np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(2, -1))
    cov, z1, z2 = np.array([[k], [0.0]]), np.array([0.75]), np.array([-0.5])
    got = gsc.summate_structured(cov, z1, z2, axes)
    assert np.max(np.abs(got - oracle.summator(cov, z1, z2, flat))) <= 2e-15


@pytest.mark.parametrize("shape,incompr", [((1, 5000), True), ((300, 300), False)])
def test_time(gsc, shape, incompr):
    """Within half as long again as phases below 2^32 (the FP64 MMA takes 5 to 10 times that)."""
    torch = pytest.importorskip("torch")
    stream = torch.cuda.current_stream()
    points = int(np.prod(shape))
    out = torch.empty((len(shape), points) if incompr else points, dtype=torch.float64, device="cuda")
    call = gsc.summate_incompr_structured_device if incompr else gsc.summate_structured_device

    def best(origin):
        cov, z1, z2, axes = _inputs(shape, 400, origin)
        args = [torch.from_numpy(a).cuda() for a in (cov, z1, z2)]
        ax = tuple(torch.from_numpy(a).cuda() for a in axes)
        times = []
        for _ in range(20):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(5):
                call(*args, ax, out, stream=stream.cuda_stream)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1) * 200.0)
        return min(times)

    near, far = best(0.0), best(1e11)
    print(f"{shape}: {near:.0f}, {far:.0f} us")
    assert far <= 1.5 * near
