"""Tiles of the x5 form that are split over the modes (sep_x5_join_kernel): two,
three and four parts, ragged rows and columns, components that meet inside a
block of columns, against the oracle (GPU tests).

Tolerance: the form's bar, 1e-6 of the field's RMS, on max |err| against the
larger of that RMS and sqrt(sum(z1^2 + z2^2) / 2), as for every tile edge.
"""
import os

import numpy as np
import pytest

import oracle
from conftest import rms

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


# 16 modes per k-block, at least 8 k-blocks per part: 256 modes make 2 parts, 384
# three, 512 and more four (parts of unequal length at 530)
@pytest.mark.parametrize("n", [256, 384, 512, 530])
@pytest.mark.parametrize("shape,incompr", [
    ((1, 40), False), ((129, 33), False), ((127, 193), False), ((130, 257), False),
    ((3, 50, 31), False), ((2, 65, 64), False), ((2, 70, 65), True), ((150, 97), True), ((5, 26, 64), True),
])
def test_split_tiles(gsc, shape, incompr, n):
    rng = np.random.default_rng(sum(shape) + n)
    dim = len(shape)
    cov = rng.normal(0.0, 0.3, (dim, n))
    z1, z2 = rng.standard_normal(n), rng.standard_normal(n)
    axes = tuple(rng.uniform(-5.0, 5.0) + np.arange(s, dtype=np.float64) for s in shape)
    pos = np.ascontiguousarray(np.array(np.meshgrid(*axes, indexing="ij")).reshape(dim, -1))
    if incompr:
        ref = oracle.summator_incompr(cov, z1, z2, pos, num_threads=NT)
        out = gsc.summate_incompr_structured(cov, z1, z2, axes, form="sep_f16x5")
    else:
        ref = oracle.summator(cov, z1, z2, pos, num_threads=NT)
        out = gsc.summate_structured(cov, z1, z2, axes, form="sep_f16x5")
    scale = max(rms(ref), np.sqrt(np.sum(z1 ** 2 + z2 ** 2) / 2.0))
    assert np.max(np.abs(out - ref)) <= 1e-6 * scale
