"""The integer path of the FP64 kernels at the edges of its groups and ranges,
against the oracle (GPU tests).

Tolerance: the phases have the oracle's bits, so what remains is the cosine
(9e-16 of a mode's amplitude at most), the modes' amplitudes and projector
weights as integers (2^-53 of the largest of a group, twice) and the rounding
of the oracle's own running sum (2^-53 of the partial sum per mode):
(2e-15 + 3e-16 N) sum_j |z1_j + i z2_j|.
"""
import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 1


def _inputs(seed, dim, n, p, k=0.6, span=40.0):
    rng = np.random.default_rng(seed)
    return (rng.normal(0.0, k, (dim, n)), rng.standard_normal(n), rng.standard_normal(n),
            rng.uniform(-span, span, (dim, p)))


def _check(gsc, cov, z1, z2, pos):
    with np.errstate(all="ignore"):
        tol = (2e-15 + 3e-16 * len(z1)) * np.sum(np.hypot(z1, z2)) + 1e-300
        fields = [(gsc.summate, oracle.summator)]
        if cov.shape[0] > 1:
            fields.append((gsc.summate_incompr, oracle.summator_incompr))
        for call, want in fields:
            got, ref = call(cov, z1, z2, pos, form="plain"), want(cov, z1, z2, pos, num_threads=NT)
            np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
            fine = np.isfinite(ref)
            if fine.any():
                assert np.max(np.abs(got[fine] - ref[fine])) <= tol


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("p", [1, 127, 129, 1025, 30011])
def test_group_and_block_edges(gsc, dim, n, p):
    _check(gsc, *_inputs(dim * 1000 + n + p, dim, n, p))


@pytest.mark.parametrize("dim", [2, 3])
def test_amplitudes_of_many_scales(gsc, dim):
    """Amplitudes from 1e-290 to 1e280 inside one group, whole groups of tiny
    ones, zeros, and the axis directions where an angle's tangent is 0 or infinite."""
    cov, z1, z2, pos = _inputs(7, dim, 160, 900)
    z1[:32] *= 1e-290
    z2[:32] *= 1e-290
    z1[32:64] = 0.0
    z2[32:64] = 0.0
    z1[64:96:3] = 0.0
    z2[65:96:3] = 0.0
    z1[65], z1[68] = -1.5, -2.5
    _check(gsc, cov, z1, z2, pos)
    z1[96:128] *= 10.0 ** np.linspace(-30, 0, 32)
    _check(gsc, cov, z1, z2, pos)
    z1[100] = 1e280
    _check(gsc, cov, z1, z2, pos)
    z1[100], z2[101] = 1e305, -1e305      # past the integer scale: the exact path
    _check(gsc, cov, z1, z2, pos)


@pytest.mark.parametrize("dim", [1, 2, 3])
def test_phase_range(gsc, dim):
    """Zero and tiny phases, and phases either side of 2^32 rad."""
    cov, z1, z2, pos = _inputs(8, dim, 70, 1500, span=100.0)
    pos[:, :40] = 0.0
    pos[0, 40:60] = -0.0
    pos[:, 60:90] *= 1e-12
    pos[:, 90:110] = 5e-324
    cov[:, 3] = 0.0
    cov[0, 3] = 1e-14
    cov[:, 20:24] *= 1e7
    cov[:, 40] = 4.2e9 / (100.0 * dim)
    cov[:, 41] = 4.4e9 / (100.0 * dim)
    cov[:, 42] = 1e12
    cov[:, 60:66] *= 1e-9
    if dim > 1:
        cov[1, 50] = 0.0
    _check(gsc, cov, z1, z2, pos)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("what", ["pos nan", "pos inf", "k nan", "k inf", "z nan", "z inf"])
def test_not_finite(gsc, dim, what):
    cov, z1, z2, pos = _inputs(9, dim, 40, 700)
    where, value = what.split()
    value = {"nan": np.nan, "inf": np.inf}[value]
    if where == "pos":
        pos[dim - 1, 333] = value
    elif where == "k":
        cov[0, 35] = value
    else:
        z2[17] = value
    _check(gsc, cov, z1, z2, pos)
