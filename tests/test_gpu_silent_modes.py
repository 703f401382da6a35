"""Modes of large weights that add nothing to the field, in the FP64 forms (GPU
tests): a wave vector along the first axis, whose projector weights are 0, and
the sine at k = 0.  The reference's sums leave them out exactly, so the forms'
fixed-point scales must not follow them.

Tolerance: the drop-in bar, 1e-12 of the field's RMS, with silent weights of 1e9
(the scale of such a weight would leave errors of 1e-8).
"""
import os

import numpy as np
import pytest

import oracle
from conftest import rel_err

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


def _modes(dim, n, incompr, seed=0):
    """Ordinary modes with two silent ones among the first 32 and one beyond."""
    rng = np.random.default_rng([dim, n, seed])
    cov, z1, z2 = rng.normal(0.0, 0.4, (dim, n)), rng.standard_normal(n), rng.standard_normal(n)
    for j, k0 in ((0, 0.5), (9, -0.25), (n - 1, 2.0)):
        cov[:, j] = 0.0
        z2[j] = 1e9
        if incompr:      # k0 is a power of two: 1 - k0 (k0 / k0^2) is 0 exactly
            cov[0, j], z1[j] = k0, -3e9
    return cov, z1, z2


def _mesh(axes):
    return np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(len(axes), -1))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [40, 4100])
@pytest.mark.parametrize("incompr", [False, True])
def test_points(gsc, dim, n, incompr):
    cov, z1, z2 = _modes(dim, n, incompr)
    pos = np.random.default_rng(1).uniform(-30.0, 30.0, (dim, 1500))
    call, want = ((gsc.summate_incompr, oracle.summator_incompr) if incompr else (gsc.summate, oracle.summator))
    assert rel_err(call(cov, z1, z2, pos, form="plain"), want(cov, z1, z2, pos, num_threads=NT)) <= 1e-12


@pytest.mark.parametrize("shape", [(40, 33), (3, 30, 25)])
@pytest.mark.parametrize("n", [40, 4100])
@pytest.mark.parametrize("incompr", [False, True])
def test_grids(gsc, shape, n, incompr):
    dim = len(shape)
    cov, z1, z2 = _modes(dim, n, incompr)
    axes = tuple(np.arange(s, dtype=np.float64) * 0.75 - 3.0 for s in shape)
    call, want = ((gsc.summate_incompr_structured, oracle.summator_incompr) if incompr
                  else (gsc.summate_structured, oracle.summator))
    assert rel_err(call(cov, z1, z2, axes), want(cov, z1, z2, _mesh(axes), num_threads=NT)) <= 1e-12


def test_weak_projector_weights(gsc):
    """Weights of 1e-6 to 1e-300 (k close to the first axis) of strong modes beside
    ordinary ones."""
    n = 64
    cov, z1, z2 = _modes(3, n, False, seed=1)
    z2[[0, 9, n - 1]] = 0.5
    cov[:, [0, 9, n - 1]] = 0.3
    for j, k1 in enumerate((1e-6, 1e-9, 1e-40, 1e-300)):
        cov[:, 10 + j] = (0.5, k1, 0.0)
        z1[10 + j] = 1e6
    axes = tuple(np.arange(s, dtype=np.float64) for s in (4, 20, 40))
    got = gsc.summate_incompr_structured(cov, z1, z2, axes, timing=True)
    assert "sep_f64_slices" in {k for k, _ in gsc.last_timings()}
    assert rel_err(got, oracle.summator_incompr(cov, z1, z2, _mesh(axes), num_threads=NT)) <= 1e-12


def test_fourier_and_batch(gsc):
    """The zero mode of the Fourier method, as points, as a grid and in a plan."""
    torch = pytest.importorskip("torch")
    cov, z1, z2 = _modes(2, 90, False, seed=2)
    sf = np.random.default_rng(3).uniform(0.1, 1.0, 90)
    pos = np.random.default_rng(4).uniform(-30.0, 30.0, (2, 2000))
    want = oracle.summator_fourier(sf, cov, z1, z2, pos, num_threads=NT)
    assert rel_err(gsc.summate_fourier(sf, cov, z1, z2, pos, form="plain"), want) <= 1e-12
    axes = tuple(np.arange(s, dtype=np.float64) for s in (50, 60))
    grid = oracle.summator_fourier(sf, cov, z1, z2, _mesh(axes), num_threads=NT)
    assert rel_err(gsc.summate_fourier_structured(sf, cov, z1, z2, axes), grid) <= 1e-12
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    item = {"cov": d(cov), "z1": d(sf * z1), "z2": d(sf * z2), "pos": d(pos),
            "out": torch.empty(2000, dtype=torch.float64, device="cuda")}
    with gsc.Batch([item], form="plain", points_per_thread=2, tile_modes=8, units_per_block=4) as plan:
        plan.run()
        torch.cuda.synchronize()
    assert rel_err(item["out"].cpu().numpy(), want) <= 1e-12
