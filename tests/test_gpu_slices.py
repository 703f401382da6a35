"""The FP64 structured form on the tensor cores (separable_slices.cu) at the
edges of its tiles, drains, segments and slabs, and on inputs that it leaves to
the FP64 MMA, against the oracle (GPU tests).

Tolerance.  The phases of the axes are rounded one by one, the oracle's in its
sum: 2^-51 |phase| of each mode's amplitude A at most.  F and G are held to
2^-54 of the largest amplitude and the products below 2^-70 of it dropped, with
the shared accumulator's truncation (64 products, 2^-24 of 2^-36 of it, per 32
modes): less than 2^-50 of the largest amplitude per mode.  The oracle's running
sum rounds by 2^-53 of its partial sum per mode.
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


def _inputs(seed, shape, n, k=0.4):
    rng = np.random.default_rng(seed)
    cov = rng.normal(0.0, k, (len(shape), n))
    axes = tuple(rng.uniform(-20.0, 20.0) + rng.uniform(0.5, 1.5) * np.arange(s) for s in shape)
    return cov, rng.standard_normal(n), rng.standard_normal(n), axes


def _points(axes, at=None):
    pos = np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(len(axes), -1))
    return pos if at is None else np.ascontiguousarray(pos[:, at])


def _tolerance(cov, z1, z2, axes):
    a = np.hypot(z1, z2)
    phase = np.abs(cov).T @ np.array([np.max(np.abs(x)) for x in axes])
    return np.sum(a * phase) * 2.0**-51 + len(a) * np.sum(a) * 2.0**-53 + len(a) * np.max(a) * 2.0**-50


def _check(gsc, cov, z1, z2, axes, incompr=False, at=None):
    call, want = ((gsc.summate_incompr_structured, oracle.summator_incompr) if incompr
                  else (gsc.summate_structured, oracle.summator))
    got = call(cov, z1, z2, axes, form="sep_f64")
    with np.errstate(all="ignore"):
        ref = want(cov, z1, z2, _points(axes, at), num_threads=NT)
    if at is not None:
        got = got[..., at]
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    fine = np.isfinite(ref)
    if fine.any():
        assert np.max(np.abs(got[fine] - ref[fine])) <= _tolerance(cov, z1, z2, axes)


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 300])
@pytest.mark.parametrize("columns", [2, 31, 33, 48, 79, 81, 97, 161])
def test_tiles(gsc, rows, columns):
    _check(gsc, *_inputs(rows * 1000 + columns, (rows, columns), 40))


@pytest.mark.parametrize("shape,incompr", [((5, 51, 37), False), ((3, 44, 33), True), ((130, 50), True),
                                            ((300, 2, 3), False), ((2, 3, 100), True)])
def test_slices_and_components(gsc, shape, incompr):
    _check(gsc, *_inputs(sum(shape), shape, 70), incompr=incompr)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 48, 65, 191, 193, 1025, 2049, 4096, 4097, 9000])
def test_drains_and_segments(gsc, n):
    _check(gsc, *_inputs(n, (20, 30), n))


def test_whole_k_range_in_one_part(gsc):
    """Enough tiles that no tile is split: every drain period runs out several times."""
    cov, z1, z2, axes = _inputs(3, (40, 512, 64), 700)
    at = np.random.default_rng(4).integers(0, 40 * 512 * 64, 4000)
    _check(gsc, cov, z1, z2, axes, at=at)


def test_coherent_modes(gsc):
    """All modes in phase with equal weights: every digit product of a k-block
    has one sign, the case the drain periods are made for."""
    n = 3000
    cov = np.tile(np.array([[0.3], [0.0]]), (1, n))
    axes = (np.arange(0.0, 8.0), np.arange(0.0, 40.0))
    for z in (1.0, 1.0 / 3.0, 0.998046875):
        _check(gsc, cov, np.full(n, z), np.zeros(n), axes)
        _check(gsc, cov, np.full(n, z), np.full(n, -z), axes)


def test_several_slabs(gsc):
    """More rows than one slab of F digits holds."""
    cov, z1, z2, axes = _inputs(5, (700, 256, 32), 256)
    at = np.random.default_rng(6).integers(0, 700 * 256 * 32, 20000)
    at[:3] = (0, 700 * 256 * 32 - 1, 131072)
    _check(gsc, cov, z1, z2, axes, at=at)


def test_amplitudes_of_many_scales(gsc):
    cov, z1, z2, axes = _inputs(7, (30, 40), 120)
    scale = 10.0 ** np.linspace(-40, 3, 120)
    _check(gsc, cov, z1 * scale, z2 * scale, axes)
    _check(gsc, cov, z1 * scale, z2 * scale, axes, incompr=True)
    _check(gsc, cov, np.zeros(120), np.zeros(120), axes)
    _check(gsc, cov, z1 * 1e-280, z2 * 1e-280, axes)       # past the sliced form's exponents
    _check(gsc, cov, z1 * 1e290, z2 * 1e290, axes)


@pytest.mark.parametrize("shape", [(30, 40), (5, 20, 40)])
@pytest.mark.parametrize("what", ["axis nan", "axis inf", "z nan", "k nan", "far"])
def test_left_to_the_fp64_mma(gsc, shape, what):
    cov, z1, z2, axes = _inputs(8, shape, 60)
    axes = [a.copy() for a in axes]
    if what.startswith("axis"):
        axes[0][2] = {"nan": np.nan, "inf": np.inf}[what.split()[1]]
    elif what == "z nan":
        z1[30] = np.nan
    elif what == "k nan":
        cov[1, 30] = np.nan
    else:
        cov[0, 30] = 3e9
    if what != "far":
        got = gsc.summate_structured(cov, z1, z2, tuple(axes), form="sep_f64")
        ref = oracle.summator(cov, z1, z2, _points(axes), num_threads=NT)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        fine = np.isfinite(ref)
        if fine.any():
            keep = [a[np.isfinite(a)] for a in axes]
            assert np.max(np.abs(got[fine] - ref[fine])) <= _tolerance(cov, z1, z2, keep)
    else:
        _check(gsc, cov, z1, z2, tuple(axes))


def test_device_call_and_replay(gsc):
    torch = pytest.importorskip("torch")
    cov, z1, z2, axes = _inputs(9, (17, 60, 50), 300)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = (d(cov), d(z1), d(z2), tuple(d(a) for a in axes))
    out = torch.full((17 * 60 * 50,), float("nan"), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()
    first = None
    for _ in range(3):
        gsc.summate_structured_device(*args, out, stream=stream.cuda_stream)
        stream.synchronize()
        got = out.cpu().numpy()
        first = got if first is None else first
        assert np.array_equal(first, got)
        out.fill_(float("nan"))
    gsc.device_status()
    ref = oracle.summator(cov, z1, z2, _points(axes), num_threads=NT)
    assert np.max(np.abs(first - ref)) <= _tolerance(cov, z1, z2, axes)


def test_smaller_slabs_when_memory_is_short(gsc):
    """A call whose digits do not fit (the first allocation fails, injected on
    the host) makes those of fewer rows at a time: the same bits."""
    torch = pytest.importorskip("torch")
    from gstools_core import _native
    cov, z1, z2, axes = _inputs(10, (9, 130, 70), 200)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    args = (d(cov), d(z1), d(z2), tuple(d(a) for a in axes))
    outs = [torch.full((9 * 130 * 70,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    stream = torch.cuda.current_stream()
    gsc.release_buffers()
    assert _native.lib.gsc_selftest_fail_alloc(0) == 0
    try:
        gsc.summate_structured_device(*args, outs[0], stream=stream.cuda_stream)
    finally:
        _native.lib.gsc_selftest_fail_alloc(-1)
    stream.synchronize()
    gsc.release_buffers()
    gsc.summate_structured_device(*args, outs[1], stream=stream.cuda_stream)
    stream.synchronize()
    gsc.device_status()
    a, b = (o.cpu().numpy() for o in outs)
    assert np.array_equal(a, b)
    ref = oracle.summator(cov, z1, z2, _points(axes), num_threads=NT)
    assert np.max(np.abs(a - ref)) <= _tolerance(cov, z1, z2, axes)
