"""Split tiles of the x5 form whose parts stay within the exact range of the
leading sum while their total does not: sep_x5_join_kernel finds that, with
other blocks of the launch still at work, and the call is recomputed (GPU tests).

Modes of weight z1 = 1, z2 = 0 add in phase at the origin.  W = 2, and the
leading grid is 2^4 x 2^11 for a scalar and 2^5 x 2^11 for a vector field (a chunk
of 16 or 8 k-blocks of 16 modes may move a sum by 2^23 at most), so each mode
counts 2^14 or 2^15 there.  1024 (512) modes reach the limit of 2^24 and keep the
x5 result; twice as many reach 2^25 in four parts of 2^23 each.
"""
import os

import numpy as np
import pytest

import oracle
from conftest import rel_err

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


# one tile; 16 of them (so that blocks before and after the origin's tile run
# beside it); several components
@pytest.mark.parametrize("shape,incompr,n", [
    ((4, 16, 64), False, 512), ((4, 16, 64), False, 1024), ((4, 16, 64), False, 2048), ((30, 16, 900), False, 2048),
    ((4, 16, 64), True, 512), ((4, 16, 64), True, 1024),
])
def test_parts_within_the_bound(gsc, shape, incompr, n):
    torch = pytest.importorskip("torch")
    from gstools_core import _native
    past = n > (512 if incompr else 1024)
    bar = 1e-12 if past else 1e-6
    rng = np.random.default_rng(sum(shape))
    cov = rng.normal(0.0, 0.05, (3, n))
    if incompr:
        cov[0] = 0.0                      # the projector leaves component 0 whole
    z1, z2 = np.ones(n), np.zeros(n)
    axes = tuple(np.arange(s, dtype=np.float64) - s // 2 for s in shape)
    flat = np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(3, -1))
    name = "summate_incompr_structured" if incompr else "summate_structured"
    ref = (oracle.summator_incompr if incompr else oracle.summator)(cov, z1, z2, flat, num_threads=NT)
    host = getattr(gsc, name)
    for _ in range(3):
        assert rel_err(host(cov, z1, z2, axes, tolerance=1e-6), ref) <= bar
        if past:
            with pytest.raises(_native.GscError, match="leading sum"):
                host(cov, z1, z2, axes, form="sep_f16x5")
        else:
            assert rel_err(host(cov, z1, z2, axes, form="sep_f16x5"), ref) <= bar
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    out = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    args = (d(cov), d(z1), d(z2), tuple(d(a) for a in axes), out)
    for _ in range(3):
        getattr(gsc, name + "_device")(*args, tolerance=1e-6, stream=st)
        torch.cuda.synchronize()
        assert rel_err(out.cpu().numpy(), ref) <= bar
    gsc.device_status()                   # nothing left behind
    # an ordinary field afterwards
    w1, w2 = rng.standard_normal(n), rng.standard_normal(n)
    want = (oracle.summator_incompr if incompr else oracle.summator)(cov, w1, w2, flat, num_threads=NT)
    assert rel_err(host(cov, w1, w2, axes, tolerance=1e-6), want) <= 1e-6
