"""The calls that users of this package make, as timed cases.

The package sums random Fourier modes at points (the randomization method) or
on structured grids, as a scalar, an incompressible vector or a Fourier-method
field.  Callers leave the default tolerance (1e-12 of the field's RMS, FP64)
or ask for 1e-6; hold their arrays on the GPU, or pass numpy arrays to the
drop-in calls; and sum one field at a time or a whole ensemble.  The sizes
are those of the benchmark's workloads (or fractions of them), of GSTools'
usual calls (1000 modes, meshes of a hundred points a side) and odd ones.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gstools-core_gb300"))
import gstools_core as gsc  # noqa: E402


def listed():
    return [
        # a conditioned field's value at its observation points: a call that is all latency
        _points("observations_2d", 2, 1000, 1000, length=10.0, extent=100.0),
        # what a script with default settings does: a 100 x 100 mesh, 1000 modes, numpy arrays in and out
        _mesh("drop_in_mesh_2d", 100, 100, 0, 1000, length=10.0, where="host"),
        # field values on the nodes of an unstructured 2-D mesh (the benchmark's first workload)
        _points("points_2d", 2, 100_000, 1000, length=10.0, extent=100.0),
        # the same where single-precision accuracy is enough
        _points("points_2d_1e6", 2, 100_000, 1000, length=10.0, extent=100.0, tolerance=1e-6),
        # a 3-D unstructured mesh with a rough (heavy-tailed) covariance, odd sizes
        _points("points_3d", 3, 250_007, 1999, spectrum="exponential", length=5.0, extent=1000.0),
        # the benchmark's large unstructured cloud, an eighth of its points
        _points("points_3d_1e6", 3, 2_097_152, 4096, spectrum="exponential", length=5.0, extent=1000.0, tolerance=1e-6),
        # velocities for particle tracking: an incompressible field at scattered points, numpy arrays
        _points("velocity_points_3d", 3, 60_000, 1500, field="incompr", length=8.0, extent=200.0, where="host"),
        # a 3-D geostatistical block model at the default tolerance, ragged sides
        _mesh("grid_3d", 160, 150, 130, 1000, length=12.0),
        # the benchmark's largest grid at single-precision accuracy
        _mesh("grid_3d_1e6", 256, 256, 256, 2000, spectrum="exponential", length=20.0, tolerance=1e-6),
        # a flow field on a grid for a transport solver (the benchmark's vector workload)
        _mesh("velocity_grid_3d_1e6", 192, 192, 192, 2048, field="incompr", length=8.0, tolerance=1e-6),
        # the Fourier method on a periodic 2-D grid
        _mesh("fourier_grid_2d", 512, 384, 0, 1024, field="fourier", length=30.0),
        # a Monte-Carlo ensemble planned once and replayed (the benchmark's ensemble, fewer and smaller items)
        _ensemble("ensemble_1e6", 48, 100_000, 4096, tolerance=1e-6),
    ]


def _points(name, dim, points, modes, *, field="scalar", spectrum="gaussian", length=10.0, extent=100.0,
            tolerance=0.0, where="gpu"):
    return {"name": name, "what": "points", "dim": dim, "points": points, "modes": modes, "field": field,
            "spectrum": spectrum, "length": length, "extent": extent, "tolerance": tolerance, "where": where}


def _mesh(name, n0, n1, n2, modes, *, field="scalar", spectrum="gaussian", length=10.0, spacing=1.0,
          tolerance=0.0, where="gpu"):
    return {"name": name, "what": "mesh", "n0": n0, "n1": n1, "n2": n2, "modes": modes, "field": field,
            "spectrum": spectrum, "length": length, "spacing": spacing, "tolerance": tolerance, "where": where}


def _ensemble(name, items, most_points, most_modes, *, tolerance=0.0):
    return {"name": name, "what": "ensemble", "items": items, "most_points": most_points,
            "most_modes": most_modes, "tolerance": tolerance}


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["points", "points", "mesh", "mesh", "ensemble"])
    tolerance = rng.choice([0.0, 1e-6])
    where = rng.choice(["gpu", "gpu", "host"])
    spectrum = rng.choice(["gaussian", "exponential"])
    field = rng.choice(["scalar", "scalar", "incompr", "fourier"])
    dim = rng.choice([2, 3])
    length = round(rng.uniform(2.0, 50.0), 3)
    if what == "ensemble":
        c = _ensemble("", rng.randint(8, 48), size(2000, 100_000), size(256, 4096), tolerance=tolerance)
        if tolerance == 0.0:     # the FP64 sums cost more: a third of the listed ensemble's work at most
            c["items"], c["most_points"] = min(c["items"], 24), min(c["most_points"], 40_000)
    elif what == "points":
        modes = size(64, 4096)
        most = 8.5e9 if tolerance else 4.9e8
        points = size(1000, min(2_000_000.0, most / modes / (2.0 if field == "incompr" else 1.0)))
        c = _points("", dim, points, modes, field=field, spectrum=spectrum, length=length,
                    extent=round(rng.uniform(50.0, 1000.0), 2), tolerance=tolerance, where=where)
    else:
        modes = size(64, 2048)
        most = 1.6e7 if tolerance else 3.1e6
        if field == "incompr":
            most /= 3.0
        side = (most ** 0.5 if dim == 2 else most ** (1.0 / 3.0))
        n = [size(20, min(side, 1200.0)) for _ in range(dim)]
        c = _mesh("", n[0], n[1], n[2] if dim == 3 else 0, modes, field=field, spectrum=spectrum, length=length,
                  spacing=rng.choice([0.5, 1.0, 1.25]), tolerance=tolerance, where=where)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _shape(case):
    return [case["n0"], case["n1"]] + ([case["n2"]] if case["n2"] else [])


def _modes(rng, dim, n, spectrum, length):
    """Wave vectors of a Gaussian (normal) or exponential (Student-t, one degree of freedom) covariance."""
    if spectrum == "gaussian":
        cov = rng.standard_normal((dim, n)) * (math.sqrt(2.0) / length)
    else:
        cov = rng.standard_normal((dim, n)) / np.abs(rng.standard_normal(n)) / length
    return cov, rng.standard_normal(n), rng.standard_normal(n)


def _fourier_modes(rng, dim, n, length, extent):
    """The n modes of the equidistant Fourier grid of a periodic box nearest zero (extent a side), a Gaussian
    covariance's spectrum factor on them, and their coefficients."""
    half = int(math.ceil(n ** (1.0 / dim))) // 2 + 1
    m = np.stack(np.meshgrid(*[np.arange(-half, half + 1)] * dim, indexing="ij")).reshape(dim, -1)
    m = m[:, np.argsort((m * m).sum(0), kind="stable")[:n]]
    k = m * (2.0 * math.pi / extent)
    k2 = (k * k).sum(0)
    density = (length / (2.0 * math.sqrt(math.pi))) ** dim * np.exp(-k2 * length * length / 4.0)
    factor = np.sqrt(2.0 * density * (2.0 * math.pi / extent) ** dim)
    n = k.shape[1]
    return factor, np.ascontiguousarray(k), rng.standard_normal(n), rng.standard_normal(n)


def _inputs(case, seed):
    """(spectrum factor or None, modes, z1, z2, positions or axes) as numpy arrays."""
    rng = np.random.default_rng([seed, 1711])
    if case["what"] == "points":
        dim, extent = case["dim"], case["extent"]
        where = rng.uniform(0.0, extent, (dim, case["points"]))
    else:
        shape = _shape(case)
        dim, extent = len(shape), case["spacing"] * max(shape)
        origin = np.round(rng.uniform(-10.0, 10.0, dim), 1)
        where = [origin[d] + case["spacing"] * np.arange(n, dtype=np.float64) for d, n in enumerate(shape)]
    if case["field"] == "fourier":
        factor, cov, z1, z2 = _fourier_modes(rng, dim, case["modes"], case["length"], extent)
    else:
        factor = None
        cov, z1, z2 = _modes(rng, dim, case["modes"], case["spectrum"], case["length"])
    return factor, cov, z1, z2, where


def _ensemble_sizes(case):
    """(dim, points, modes) of each realization: half 2-D, half 3-D, sizes log-uniform."""
    rng = np.random.default_rng([case["items"], case["most_points"], case["most_modes"]])
    fewest = min(256, case["most_modes"] // 2)
    sizes = []
    for i in range(case["items"]):
        points = math.exp(rng.uniform(math.log(1000.0), math.log(case["most_points"])))
        modes = math.exp(rng.uniform(math.log(fewest), math.log(case["most_modes"])))
        sizes.append((2 + (i % 2), int(round(points)), int(round(modes))))
    return sizes


def _ensemble_inputs(case, seed):
    """(modes, z1, z2, positions) of each realization; Gaussian and exponential spectra alternate in pairs."""
    rng = np.random.default_rng([seed, 1712])
    items = []
    for i, (dim, points, modes) in enumerate(_ensemble_sizes(case)):
        cov, z1, z2 = _modes(rng, dim, modes, "gaussian" if (i // 2) % 2 == 0 else "exponential", rng.uniform(2.0, 50.0))
        items.append((cov, z1, z2, rng.uniform(0.0, 500.0, (dim, points))))
    return items


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    tolerance = case["tolerance"] or None
    if case["what"] == "ensemble":
        items = []
        for cov, z1, z2, pos in _ensemble_inputs(case, seed):
            items.append({"cov": _gpu(cov), "z1": _gpu(z1), "z2": _gpu(z2), "pos": _gpu(pos),
                          "out": torch.empty(pos.shape[1], dtype=torch.float64, device="cuda")})
        return {"case": case, "items": items, "plan": gsc.Batch(items, tolerance=tolerance)}
    factor, cov, z1, z2, where = _inputs(case, seed)
    mesh = case["what"] == "mesh"
    field = case["field"]
    if case["where"] == "host":
        # the drop-in callers hold numpy arrays; a structured mesh comes expanded, as GSTools passes it
        if mesh:
            where = np.ascontiguousarray(np.array(np.meshgrid(*where, indexing="ij")).reshape(len(where), -1))
        call = {"scalar": gsc.summate, "incompr": gsc.summate_incompr, "fourier": gsc.summate_fourier}[field]
        lead = [] if factor is None else [factor]
        return {"case": case, "call": call, "args": (*lead, cov, z1, z2, where), "keys": {"tolerance": tolerance}}
    if mesh:
        points = math.prod(len(a) for a in where)
        where = tuple(_gpu(a) for a in where)
        call = {"scalar": gsc.summate_structured_device, "incompr": gsc.summate_incompr_structured_device,
                "fourier": gsc.summate_fourier_structured_device}[field]
    else:
        points = where.shape[1]
        where = _gpu(where)
        call = {"scalar": gsc.summate_device, "incompr": gsc.summate_incompr_device,
                "fourier": gsc.summate_fourier_device}[field]
    out = torch.empty((cov.shape[0], points) if field == "incompr" else (points,), dtype=torch.float64, device="cuda")
    lead = [] if factor is None else [_gpu(factor)]
    return {"case": case, "call": call, "args": (*lead, _gpu(cov), _gpu(z1), _gpu(z2), where, out),
            "keys": {"tolerance": tolerance, "stream": torch.cuda.current_stream().cuda_stream}}


def run(state):
    if "plan" in state:
        state["plan"].run_graph(torch.cuda.current_stream().cuda_stream)
        return [item["out"] for item in state["items"]]
    return state["call"](*state["args"], **state["keys"])


# ---------------------------------------------------------------------------
# work and 64-bit results
# ---------------------------------------------------------------------------
def _sum_work(dim, points, modes, outputs, extra_inputs=0):
    """Phase (2 dim - 1), sine and cosine (counted as one operation each), their weighted sum (4), and a
    multiply-add per output component of a vector field."""
    flops = points * modes * (2 * dim + 5 + (2 * outputs if outputs > 1 else 0))
    return {"bytes": 8 * (modes * (dim + 2) + extra_inputs + points * (dim + outputs)), "flops": flops}


def work(case):
    if case["what"] == "ensemble":
        total = {"bytes": 0, "flops": 0}
        for dim, points, modes in _ensemble_sizes(case):
            for k, v in _sum_work(dim, points, modes, 1).items():
                total[k] += v
        return total
    if case["what"] == "points":
        outputs = case["dim"] if case["field"] == "incompr" else 1
        return _sum_work(case["dim"], case["points"], case["modes"], outputs,
                         case["modes"] if case["field"] == "fourier" else 0)
    # a grid's exponentials factor by axis: one real multiply-add per output value and real part of a mode
    shape = _shape(case)
    points, dim = math.prod(shape), len(shape)
    outputs = dim if case["field"] == "incompr" else 1
    inputs = case["modes"] * (dim + 2 + (case["field"] == "fourier")) + sum(shape)
    if case["where"] == "host":
        inputs += points * dim          # the expanded mesh
    return {"bytes": 8 * (inputs + points * outputs), "flops": 4 * points * case["modes"] * outputs}


def _projector(cov):
    """e_1 - k k_1 / |k|^2 of each mode."""
    k2 = cov[0] / (cov * cov).sum(0)
    p = -cov * k2
    p[0] += 1.0
    return p


def _exact_points(cov, z1, z2, pos, incompr):
    cov, z1, z2, pos = (_gpu(a) for a in (cov, z1, z2, pos))
    dim, points = pos.shape
    if incompr:
        p = _projector(cov)
        c, s = (p * z1).T.contiguous(), (p * z2).T.contiguous()
    else:
        c, s = z1[:, None], z2[:, None]
    out = torch.empty((c.shape[1], points), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // max(1, cov.shape[1]))
    for a in range(0, points, step):
        x = pos[:, a:a + step]
        phase = x[0][:, None] * cov[0]
        for d in range(1, dim):
            phase = phase + x[d][:, None] * cov[d]
        out[:, a:a + step] = (torch.cos(phase) @ c + torch.sin(phase) @ s).T
    return out if incompr else out[0]


def _exact_mesh(cov, z1, z2, axes, incompr):
    cov, z1, z2 = _gpu(cov), _gpu(z1), _gpu(z2)
    axes = [_gpu(a) for a in axes]
    if len(axes) == 2:
        axes = [None] + axes
    first = cov.shape[0] - 2                         # the dimension of the rows' axis
    one, two = cov[first][:, None] * axes[1], cov[first + 1][:, None] * axes[2]
    row = torch.complex(torch.cos(one), torch.sin(one))
    column = torch.complex(torch.cos(two), torch.sin(two))
    weights = _projector(cov) if incompr else torch.ones_like(cov[:1])
    z = torch.complex(z1, -z2)
    right = [torch.cat([w[:, None] * column.real, -w[:, None] * column.imag]) for w in weights]
    slices = []
    for i in range(1 if axes[0] is None else axes[0].numel()):
        s = z
        if axes[0] is not None:
            phase = cov[0] * axes[0][i]
            s = z * torch.complex(torch.cos(phase), torch.sin(phase))
        f = row * s[:, None]
        left = torch.cat([f.real, f.imag]).T
        slices.append(torch.stack([left @ g for g in right]))
    out = torch.stack(slices, dim=1).reshape(len(right), -1)
    return out if incompr else out[0]


def exact(case, seed):
    if case["what"] == "ensemble":
        return [_exact_points(*item, False) for item in _ensemble_inputs(case, seed)]
    factor, cov, z1, z2, where = _inputs(case, seed)
    if factor is not None:
        z1, z2 = factor * z1, factor * z2
    incompr = case["field"] == "incompr"
    return (_exact_points if case["what"] == "points" else _exact_mesh)(cov, z1, z2, where, incompr)
