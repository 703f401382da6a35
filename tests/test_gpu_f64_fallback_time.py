"""The FP64 MMA kernels, run for what the sliced form leaves to them and for
flagged x5 calls: how their tiles share the SMs (GPU tests).

A tile of 64 x 64 outputs takes an SM's FP64 pipe for a time t that depends on the
modes alone.  Tiles up to the number of SMs (152) take t together (1.3 t allows for
their tables), more of them what the busiest SM takes when each block gets the next
tile once it is free: 2 t for 160 tiles (1.3 times that), 7 t for 1000.  Blocks
placed several to an SM, or fixed shares of the tiles, exceed these: 3.6 t for 8
tiles, 3.7 t for 160, 7.3 t for 1000.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _time(torch, gsc, shape, n, incompr, tolerance=None, nan=False, origin=0.0):
    """Microseconds of a device call, the least of ten, on inputs that end on the FP64 MMA kernels."""
    rng = np.random.default_rng([*shape, n])
    cov, z1, z2 = rng.normal(0.0, 0.05, (len(shape), n)), np.ones(n), np.zeros(n)
    if nan:
        z2[0] = np.nan
    axes = tuple(torch.arange(s, dtype=torch.float64, device="cuda") - s // 2 + origin for s in shape)
    args = [torch.from_numpy(a).cuda() for a in (cov, z1, z2)]
    points = int(np.prod(shape))
    out = torch.empty((len(shape), points) if incompr else points, dtype=torch.float64, device="cuda")
    call = gsc.summate_incompr_structured_device if incompr else gsc.summate_structured_device
    stream = torch.cuda.current_stream()
    times = []
    for _ in range(10):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        call(*args, axes, out, tolerance=tolerance, stream=stream.cuda_stream)
        e1.record()
        e1.synchronize()
        times.append(e0.elapsed_time(e1) * 1e3)
    return min(times)


def test_few_tiles_of_phases_past_1e13(gsc):
    torch = pytest.importorskip("torch")
    one, eight = (_time(torch, gsc, (b, 8, 8), 200, False, origin=1e15) for b in (1, 8))
    print(f"{one:.0f} {eight:.0f} us")
    assert eight <= 1.3 * one


def test_more_tiles_than_sms(gsc):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    one = _time(torch, gsc, (1, 8, 8), 1000, False, nan=True)
    many = _time(torch, gsc, (100, 100, 100), 1000, True, nan=True)          # 100 x 2 x 5 tiles
    print(f"{one:.0f} {many:.0f} us")
    assert many <= -(-1000 // sms) * one


def test_flagged_x5_calls(gsc):
    """Coherent weights through the origin: the x5 form leaves the call to the FP64 MMA."""
    torch = pytest.importorskip("torch")
    few = _time(torch, gsc, (12, 40, 64), 2000, False, tolerance=1e-6)      # 12 tiles
    more = _time(torch, gsc, (40, 80, 100), 2000, False, tolerance=1e-6)    # 160
    print(f"{few:.0f} {more:.0f} us")
    assert more <= 1.3 * 2 * few
