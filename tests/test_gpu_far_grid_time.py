"""FP64 grids whose phases are all past the sliced form's range (2^32): what its
attempt adds to the FP64 MMA kernels that take the call (GPU test).

Both calls end on the same kernels, whose time depends on the sizes alone; the one
with a NaN weight leaves the sliced form before its tables.  10 % for the tables'
larger phases (a store by every warp to one word made it 20 %).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5000, 1), (300, 300)])
def test_far_phases_against_a_nan_weight(gsc, shape):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(0)
    points = int(np.prod(shape))
    out = torch.empty(points, dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()

    def best(origin, nan):
        cov, z1, z2 = rng.normal(0.0, 0.2, (2, 200)), rng.standard_normal(200), rng.standard_normal(200)
        if nan:
            z1[0] = np.nan
        args = [torch.from_numpy(a).cuda() for a in (cov, z1, z2)]
        axes = tuple(origin + torch.arange(s, dtype=torch.float64, device="cuda") for s in shape)
        times = []
        for _ in range(20):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            gsc.summate_structured_device(*args, axes, out, stream=stream.cuda_stream)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1) * 1e3)
        return min(times)

    nan, far = best(0.0, True), best(3e10, False)
    print(f"{shape}: {nan:.0f}, {far:.0f} us")
    assert far <= 1.1 * nan
