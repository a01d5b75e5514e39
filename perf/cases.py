"""Performance cases: one pass each through the public Python entry points.

The library takes and returns host arrays, so every pass is the whole call:
planning, copies, kernels and results.  Sizes, variograms and search radii are
those of hpgl_b200/workloads.py, of the benchmarks beside it and of the
reference's published setup (166 x 141 x 225 cells, radii 20, 12 neighbours).
"""

import math
import os
import tempfile

import numpy as np

from hpgl_b200 import cvariogram, serve, workloads
from hpgl_b200.geo_bsd import cdf, geo, sgs, sis

UNDEFINED = -99.0
# extent, as a multiple of the range, where the covariance falls to 1 %
EXTENT = {0: 1.0, 1: 1.54, 2: 1.24}


def _krige(name, kind, shape, informed, cov, ranges, radii, nmax, angle=0.0, nugget=0.0, categories=0,
           precision="fp64"):
    c = {"op": "krige", "kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2], "informed": informed,
         "cov": cov, "rx": float(ranges[0]), "ry": float(ranges[1]), "rz": float(ranges[2]), "sx": radii[0],
         "sy": radii[1], "sz": radii[2], "nmax": nmax, "angle": float(angle), "nugget": float(nugget),
         "categories": categories, "precision": precision}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one point's kriging weights: an interactive or scripted query, all latency
        {"name": "weights_24", "op": "weights", "n": 24, "cov": 1},
        # a small model, the size of a first trial of a variogram
        _krige("ok_50x50x20", "ok", (50, 50, 20), 0.02, 0, (10, 10, 5), (20, 20, 10), 12),
        # the default arithmetic on a field-scale cube
        _krige("sk_256x256x64_fp64", "sk", (256, 256, 64), 0.01, 1, (40, 20, 8), (80, 40, 16), 32, 30, 0.05),
        # the same job with the mixed-precision option
        _krige("sk_256x256x64_mixed", "sk", (256, 256, 64), 0.01, 1, (40, 20, 8), (80, 40, 16), 32, 30, 0.05,
               precision="mixed"),
        # the setup of the reference's published timings: dense data, few neighbours, odd sizes
        _krige("ok_166x141x225", "ok", (166, 141, 225), 0.2, 1, (10, 10, 10), (20, 20, 20), 12),
        # facies probabilities, four categories
        _krige("ik_200x200x100", "ik", (200, 200, 100), 0.015, 0, (25, 25, 6), (25, 25, 6), 24, categories=4),
        # clustered data, a smooth model, the largest neighbourhoods
        _krige("lvm_512x512x32", "lvm", (512, 512, 32), 0.005, 2, (30, 30, 4), (40, 40, 5), 64, nugget=0.01),
        # a sparse property with a dense secondary one, odd sizes
        _krige("cok1_161x119x47", "cok1", (161, 119, 47), 0.02, 0, (14, 14, 5), (14, 14, 5), 24),
        # the reference's large simulation test
        {"name": "sgs_166x141x225", "op": "simulate", "kind": "sgs", "nx": 166, "ny": 141, "nz": 225,
         "informed": 0.01, "range": 10.0, "radius": 20, "nmax": 12, "categories": 0},
        # a property file written and read back
        {"name": "inc_166x141x57", "op": "inc", "nx": 166, "ny": 141, "nz": 57, "informed": 0.8},
        # the experimental variogram of a whole cube
        {"name": "variogram_166x141x225", "op": "variogram", "nx": 166, "ny": 141, "nz": 225, "informed": 0.1,
         "lags": 20, "azimuth": 30.0},
        # a batch of unlike jobs handed to the server at once
        {"name": "serve_12_jobs", "op": "serve", "jobs": 12, "stream": 11, "cells": 600000},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _shape(rng, cells):
    a = [rng.uniform(2.5, 5.0), rng.uniform(2.5, 5.0), rng.uniform(0.8, 1.5)]
    s = (cells / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
    return [max(8, int(v * s)) for v in a]


def draw(rng):
    op = rng.choice(["krige"] * 8 + ["simulate"] * 2 + ["weights", "inc", "variogram", "serve"])
    if op == "weights":
        return {"op": op, "n": rng.randint(1, 64), "cov": rng.randint(0, 2)}
    if op == "inc":
        nx, ny, nz = _shape(rng, _log(rng, 5e4, 2e6))
        return {"op": op, "nx": nx, "ny": ny, "nz": nz, "informed": rng.uniform(0.1, 1.0)}
    if op == "variogram":
        nx, ny, nz = _shape(rng, _log(rng, 1e5, 4e6))
        return {"op": op, "nx": nx, "ny": ny, "nz": nz, "informed": rng.uniform(0.02, 0.15),
                "lags": rng.randint(6, 20), "azimuth": rng.uniform(0.0, 90.0)}
    if op == "serve":
        return {"op": op, "jobs": rng.randint(4, 12), "stream": rng.randint(100, 10000), "cells": rng.randint(100000, 600000)}
    if op == "simulate":
        nx, ny, nz = _shape(rng, _log(rng, 5e4, 2e6))
        kind = rng.choice(["sgs", "sis"])
        return {"op": op, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "informed": rng.uniform(0.005, 0.03),
                "range": rng.uniform(6.0, 12.0), "radius": rng.randint(8, 20), "nmax": rng.randint(8, 32),
                "categories": rng.randint(2, 4) if kind == "sis" else 0}
    kind = rng.choice(["ok", "ok", "sk", "sk", "lvm", "ik", "median", "cok1", "cok2"])
    nmax = rng.randint(8, 64)
    cells = _log(rng, 3e4, 4.2e6 if nmax <= 32 else 2e6)
    cov = rng.randint(0, 2)
    ranges = [rng.uniform(5, 30), rng.uniform(5, 30), rng.uniform(3, 8)]
    radii = [int(math.ceil(EXTENT[cov] * r)) for r in ranges]
    precision = rng.choice(["fp64", "mixed"]) if kind in ("ok", "sk", "lvm") else "fp64"
    return _krige(None, kind, _shape(rng, cells), _log(rng, 0.005, 0.2), cov, ranges, radii, nmax,
                  rng.choice([0.0, rng.uniform(0, 90)]), rng.uniform(0, 0.1),
                  rng.randint(3, 5) if kind == "ik" else 2 if kind == "median" else 0, precision)


# ---- inputs -------------------------------------------------------------------

def _waves(rng, cells, shape, count=6):
    """A smooth field at `cells`: waves of a few periods over the grid."""
    x, y, z = cells % shape[0], cells // shape[0] % shape[1], cells // (shape[0] * shape[1])
    out = np.zeros(len(cells))
    for _ in range(count):
        k = rng.uniform(0.5, 4.0, 3) * 2 * math.pi / np.array(shape)
        out += np.sin(k[0] * x + k[1] * y + k[2] * z + rng.uniform(0, 2 * math.pi))
    return out / math.sqrt(count / 2.0)


def _cells(rng, size, share):
    return np.flatnonzero(rng.random(size, dtype=np.float32) < share)


def _blob_cells(rng, shape, count):
    """About `count` cells in clusters of sigma 3 cells, as wells and pads cluster data."""
    centres = np.stack([rng.uniform(0, n, max(4, count // 200)) for n in shape], axis=1)
    p = np.floor(centres[rng.integers(0, len(centres), 2 * count)] + rng.normal(0, 3.0, (2 * count, 3))).astype(np.int64)
    p = p[np.all((p >= 0) & (p < np.array(shape)), axis=1)]
    idx = np.unique(p[:, 0] + shape[0] * (p[:, 1] + shape[1] * p[:, 2]))
    return np.sort(rng.permutation(idx)[:count])


def _prop(values, mask, shape):
    f = lambda a: np.reshape(a, shape, order="F")
    return geo.ContProperty(f(values), f(mask))


def _cont(rng, cells, shape, level=0.0):
    size = int(np.prod(shape))
    values = np.full(size, UNDEFINED, dtype=np.float32)
    mask = np.zeros(size, dtype=np.uint8)
    values[cells] = level + _waves(rng, cells, shape) + rng.normal(0, 0.3, len(cells))
    mask[cells] = 1
    return values, mask


def _codes(rng, cells, shape, categories):
    size = int(np.prod(shape))
    codes = np.zeros(size, dtype=np.uint8)
    mask = np.zeros(size, dtype=np.uint8)
    v = _waves(rng, cells, shape) + rng.normal(0, 0.3, len(cells))
    codes[cells] = np.searchsorted(np.quantile(v, np.arange(1, categories) / categories), v)
    mask[cells] = 1
    return codes, mask


def _mean_cube(rng, shape):
    mean = np.zeros(shape, dtype=np.float32, order="F")
    axes = [np.arange(n, dtype=np.float32) for n in shape]
    for _ in range(3):
        k = rng.uniform(0.2, 2.0, 3) * 2 * math.pi / np.array(shape)
        a, b, c = [np.sin(k[i] * axes[i] + rng.uniform(0, 6.28)).astype(np.float32) for i in range(3)]
        mean += a[:, None, None] * b[None, :, None] * c[None, None, :] * np.float32(0.3)
    return mean


class _Server:
    """A server that closes with the program that keeps it."""

    def __init__(self):
        self.server = serve.Server(hbm_budget_bytes=40 << 30, max_inflight=8)

    def __del__(self):
        if hasattr(self, "server"):
            self.server.close()


def _krige_inputs(case, rng):
    shape = (case["nx"], case["ny"], case["nz"])
    size = int(np.prod(shape))
    kind = case["kind"]
    s = {"radii": (case["sx"], case["sy"], case["sz"])}
    if kind == "lvm":
        cells = _blob_cells(rng, shape, max(1, int(size * case["informed"])))
        s["mean"] = _mean_cube(rng, shape)
        values, mask = _cont(rng, cells, shape)
        values[cells] = s["mean"].reshape(-1, order="F")[cells] + rng.normal(0, 0.3, len(cells))
    else:
        cells = _cells(rng, size, case["informed"])
        if case["categories"]:
            s["prop"] = geo.IndProperty(*[np.reshape(a, shape, order="F") for a in _codes(rng, cells, shape, case["categories"])],
                                        case["categories"])
            return s
        values, mask = _cont(rng, cells, shape, 2.0 if kind.startswith("cok") else 0.0)
    s["prop"] = _prop(values, mask, shape)
    if kind.startswith("cok"):
        every = np.arange(size)
        sec = (5.0 + 0.5 * _waves(rng, every, shape, 2) + rng.normal(0, 0.3, size)).astype(np.float32)
        smask = (rng.random(size) < 0.9).astype(np.uint8)
        s["secondary"] = _prop(np.where(smask > 0, sec, np.float32(UNDEFINED)), smask, shape)
        s["m1"], s["m2"] = float(values[cells].mean()), float(sec[smask > 0].mean())
        s["var2"] = float(sec[smask > 0].var())
    return s


def _serve_jobs(case, seed):
    """The jobs' grids, variograms and searches come from the stream, their data from the seed."""
    plan, rng = np.random.default_rng(case["stream"]), np.random.default_rng(seed)
    jobs = []
    for i in range(case["jobs"]):
        job = workloads.serve_job(plan, i, max_cells=case["cells"])
        n = len(job["mask"])
        cells = _cells(rng, n, float(job["mask"].mean()))
        job["mask"] = np.zeros(n, dtype=np.uint8)
        job["mask"][cells] = 1
        if job["kind"] == "ik":
            job["codes"] = np.zeros(n, dtype=np.uint8)
            job["codes"][cells] = rng.integers(0, 4, len(cells))
        else:
            job["values"] = np.full(n, UNDEFINED, dtype=np.float32)
            job["values"][cells] = rng.standard_normal(len(cells))
        jobs.append(job)
    return jobs


def _points(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    return rng.uniform(0, 50, 3).astype(np.float32), [rng.uniform(0, 50, n).astype(np.float32) for _ in range(3)]


def _inc_property(case, seed):
    rng = np.random.default_rng(seed)
    size = case["nx"] * case["ny"] * case["nz"]
    mask = (rng.random(size) < case["informed"]).astype(np.uint8)
    values = (1000.0 * rng.standard_normal(size) * 10.0 ** rng.integers(-3, 3, size)).astype(np.float32)
    return np.where(mask > 0, values, np.float32(UNDEFINED)), mask


def _variogram_property(case, seed):
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    x = np.arange(shape[0], dtype=np.float32)[:, None, None]
    v = np.asfortranarray(rng.standard_normal(shape, dtype=np.float32) + np.float32(0.02) * x)
    return v, np.asfortranarray((rng.random(shape, dtype=np.float32) < case["informed"]).astype(np.uint8))


def prepare(case, seed):
    op = case["op"]
    rng = np.random.default_rng(seed)
    s = {"op": op, "case": case}
    if op == "weights":
        s["centre"], s["points"] = _points(case, seed)
        return s
    if op == "serve":
        s["server"], s["jobs"] = _Server(), _serve_jobs(case, seed)
        return s
    shape = (case["nx"], case["ny"], case["nz"])
    s["shape"] = shape
    if op == "inc":
        s["prop"] = _prop(*_inc_property(case, seed), shape)
        s["folder"] = tempfile.TemporaryDirectory()
        return s
    if op == "variogram":
        s["data"] = _variogram_property(case, seed)
        ell = cvariogram.Ellipsoid(40.0, 4.0, 2.0, case["azimuth"], 0.0, 0.0)
        s["template"] = cvariogram.VariogramSearchTemplate(2.0, 2.0, 0.8, case["lags"], 0.0, ell)
        return s
    s["grid"] = geo.SugarboxGrid(*shape)
    if op == "simulate":
        cells = _cells(rng, int(np.prod(shape)), case["informed"])
        s["seed"] = int(rng.integers(1, 1 << 24))
        r = case["range"]
        if case["kind"] == "sgs":
            s["prop"] = _prop(*_cont(rng, cells, shape), shape)
            s["cdf"] = cdf.calc_cdf(s["prop"])
            s["cov"] = geo.CovarianceModel(type=1, ranges=(r, r, r), sill=0.4)
        else:
            k = case["categories"]
            s["prop"] = geo.IndProperty(*[np.reshape(a, shape, order="F") for a in _codes(rng, cells, shape, k)], k)
            s["data"] = [{"cov_model": geo.CovarianceModel(type=1, ranges=(r, r, r), sill=0.2),
                          "radiuses": (case["radius"],) * 3, "max_neighbours": case["nmax"]} for _ in range(k)]
            s["marginals"] = [1.0 / k] * k
        return s
    s.update(_krige_inputs(case, rng))
    sill = 0.25 if case["categories"] else 1.0
    s["cov"] = geo.CovarianceModel(type=case["cov"], ranges=(case["rx"], case["ry"], case["rz"]),
                                   angles=(case["angle"], 0.0, 0.0), sill=sill, nugget=case["nugget"] * sill)
    return s


# ---- one pass -----------------------------------------------------------------

def _run_krige(s):
    case = s["case"]
    kind, precision = case["kind"], case["precision"]
    a = (s["radii"], case["nmax"], s["cov"])
    if kind == "ok":
        return geo.ordinary_kriging(s["prop"], s["grid"], *a, precision=precision)
    if kind == "sk":
        return geo.simple_kriging(s["prop"], s["grid"], *a, mean=0.0, precision=precision)
    if kind == "lvm":
        return geo.lvm_kriging(s["prop"], s["grid"], s["mean"], *a, precision=precision)
    if kind == "cok1":
        return geo.simple_cokriging_markI(s["prop"], s["grid"], s["secondary"], s["m1"], s["m2"], s["var2"], 0.7, *a)
    if kind == "cok2":
        sec = geo.CovarianceModel(type=1, ranges=(20.0, 20.0, 6.0), sill=1.0, nugget=0.05)
        return geo.simple_cokriging_markII(s["grid"], {"data": s["prop"], "mean": s["m1"], "cov_model": s["cov"]},
                                           {"data": s["secondary"], "mean": s["m2"], "cov_model": sec}, 0.7,
                                           s["radii"], case["nmax"])
    if kind == "median":
        return geo.median_ik(s["prop"], s["grid"], (0.5, 0.5), *a, precision=precision)
    k = case["categories"]
    data = [{"cov_model": s["cov"], "radiuses": s["radii"], "max_neighbours": case["nmax"]} for _ in range(k)]
    return geo.indicator_kriging(s["prop"], s["grid"], data, [1.0 / k] * k, precision=precision)


def run(s):
    case, op = s["case"], s["op"]
    if op == "weights":
        return geo.simple_kriging_weights(s["centre"], *s["points"], ranges=(20.0, 15.0, 10.0), cov_type=case["cov"],
                                          nugget=0.05, angles=(30.0, 0.0, 0.0))
    if op == "serve":
        server = s["server"].server
        tickets = [server.submit(job, precision="fp64") for job in s["jobs"]]
        results = [server.result(t) for t in tickets]
        return [(r["out"], r["out_mask"]) for r in results]
    if op == "inc":
        path = os.path.join(s["folder"].name, "property.inc")
        geo.write_property(s["prop"], path, "PROPERTY", UNDEFINED)
        out = geo.load_cont_property(path, UNDEFINED, s["shape"])
    elif op == "variogram":
        return cvariogram.CalcVariograms(s["template"], s["data"])[1]
    elif op == "simulate" and case["kind"] == "sgs":
        out = sgs.sgs_simulation(s["prop"], s["grid"], s["cdf"], (case["radius"],) * 3, case["nmax"], s["cov"], s["seed"])
    elif op == "simulate":
        out = sis.sis_simulation(s["prop"], s["grid"], s["data"], s["seed"], s["marginals"])
    else:
        out = _run_krige(s)
    return out.data, out.mask


# ---- the work of a pass -------------------------------------------------------

def _system(n, ordinary=False):
    """A symmetric system of n neighbours: its covariances at 20 operations
    each, the factorisation and the triangular solves."""
    r = 2 if ordinary else 1
    return 2.0 / 3.0 * n ** 3 + 2.0 * r * n * n + 4.0 * n + 20.0 * (n * (n + 1) / 2.0 + n)


def work(case):
    op = case["op"]
    if op == "weights":
        return {"bytes": 16.0 * case["n"] + 12, "flops": _system(case["n"])}
    if op == "serve":
        plan, b, f = np.random.default_rng(case["stream"]), 0.0, 0.0
        for i in range(case["jobs"]):
            job = workloads.serve_job(plan, i, max_cells=case["cells"])
            n = len(job["mask"])
            f += n * _system(job["params"][0]["max_neighbours"], job["kind"] == "ok")
            b += n * (4.0 if job["kind"] == "ik" else 10.0)
        return {"bytes": b, "flops": f}
    n = float(case["nx"] * case["ny"] * case["nz"])
    if op == "inc":
        return {"bytes": n * (2 * 13.5 + 10.0), "flops": 0.0}
    if op == "variogram":
        area = math.pi * 4.0 * 2.0 * 2.0 * case["lags"]  # offsets in the tunnel, about
        return {"bytes": 5.0 * n, "flops": 4.0 * area * n * case["informed"] ** 2}
    if op == "simulate":
        k = 1 if case["categories"] <= 2 else case["categories"]
        b = 4.0 if case["categories"] else 10.0
        return {"bytes": b * n, "flops": k * n * (1.0 - case["informed"]) * _system(case["nmax"])}
    kind = case["kind"]
    systems = n if kind in ("ik", "median") else n * (1.0 - case["informed"])
    b = 4.0 if kind in ("ik", "median") else 15.0 if kind.startswith("cok") else 14.0 if kind == "lvm" else 10.0
    return {"bytes": b * n, "flops": systems * _system(case["nmax"] + kind.startswith("cok"), kind == "ok")}


# ---- the same results in 64 bits ----------------------------------------------

def _transform(ranges, angle):
    a = angle * math.pi / 180
    rz = np.array([[math.cos(a), math.sin(a), 0], [-math.sin(a), math.cos(a), 0], [0, 0, 1]])
    return np.diag([1.0, ranges[0] / ranges[1], ranges[0] / ranges[2]]) @ rz


def _covariance(cov, r, sill, nugget, h):
    if cov == 0:
        c = np.where(h > r, 0.0, 1 - 1.5 * h / r + 0.5 * (h / r) ** 3)
    else:
        c = np.exp(-3.0 * h / r) if cov == 1 else np.exp(-3.0 * (h / r) ** 2)
    return (sill - nugget) * np.where(h < 0.0001, 1.0, c)


def _exact_weights(case, seed):
    centre, points = _points(case, seed)
    p, c = np.stack(points, axis=1).astype(np.float64), centre.astype(np.float64)
    t = _transform((20.0, 15.0, 10.0), 30.0)
    h = lambda d: np.sqrt(((d @ t.T) ** 2).sum(-1))
    a = _covariance(case["cov"], 20.0, 1.0, 0.05, h(p[:, None] - p[None]))
    return np.linalg.solve(a, _covariance(case["cov"], 20.0, 1.0, 0.05, h(p - c)))


def _exact_variogram(case, seed):
    v, m = _variogram_property(case, seed)
    shape = v.shape
    a = case["azimuth"] * (3.14159265358 / 180.0)
    d1, d2 = (math.cos(a), math.sin(a)), (-math.sin(a), math.cos(a))
    reach = 2.0 * case["lags"]
    corners = [(i * reach * d1[0] + j * 4.0 * d2[0], i * reach * d1[1] + j * 4.0 * d2[1]) for i in (0, 1) for j in (-1, 1)]
    lo = [int(min(c[k] for c in corners)) for k in (0, 1)] + [-2]
    hi = [int(math.floor(max(c[k] for c in corners))) for k in (0, 1)] + [2]
    flat, inside = v.reshape(-1, order="F").astype(np.float64), m.reshape(-1, order="F")
    cells = np.flatnonzero(inside)
    x, y, z = cells % shape[0], cells // shape[0] % shape[1], cells // (shape[0] * shape[1])
    here = flat[cells]
    total, count = np.zeros(case["lags"]), np.zeros(case["lags"])
    for i in range(lo[0], hi[0] + 1):
        for j in range(lo[1], hi[1] + 1):
            for k in range(lo[2], hi[2] + 1):
                s1, s2 = i * d1[0] + j * d1[1], i * d2[0] + j * d2[1]
                side = math.sqrt((s2 / 4.0) ** 2 + (k / 2.0) ** 2)
                if not (side <= 1.0 and 0.8 * side <= s1):
                    continue
                dist = math.sqrt(i * i + j * j + k * k)
                lags = [l for l in range(math.ceil((dist - 1.0) / 2.0), math.floor((dist + 1.0) / 2.0) + 1)
                        if 0 <= l < case["lags"]]
                if not lags:
                    continue
                ok = (x + i >= 0) & (x + i < shape[0]) & (y + j >= 0) & (y + j < shape[1]) & (z + k >= 0) & (z + k < shape[2])
                to = cells[ok] + (i + shape[0] * (j + shape[1] * k))
                both = inside[to] > 0
                d = here[ok][both] - flat[to[both]]
                for l in lags:
                    total[l] += np.dot(d, d)
                    count[l] += len(d)
    return total / count / 2.0


def _sorted_offsets(keys):
    """Places of `keys` after std::sort by descending key: an introspective
    quicksort down to 16 elements, then an insertion sort.  Which of several
    equal offsets comes first decides which neighbours a node gets."""
    a = [(-k, i) for i, k in enumerate(keys)]
    less = lambda p, q: p[0] < q[0]
    todo = [(0, len(a))]
    while todo:
        lo, hi = todo.pop()
        while hi - lo > 16:
            mid, x, z = lo + (hi - lo) // 2, lo + 1, hi - 1
            if less(a[x], a[mid]):
                m = mid if less(a[mid], a[z]) else z if less(a[x], a[z]) else x
            else:
                m = x if less(a[x], a[z]) else z if less(a[mid], a[z]) else mid
            a[lo], a[m] = a[m], a[lo]
            p, i, j = a[lo], lo + 1, hi
            while True:
                while less(a[i], p):
                    i += 1
                j -= 1
                while less(p, a[j]):
                    j -= 1
                if not i < j:
                    break
                a[i], a[j] = a[j], a[i]
                i += 1
            todo.append((i, hi))
            hi = i
    for i in range(1, len(a)):
        v, j = a[i], i
        while j > 0 and less(v, a[j - 1]):
            a[j] = a[j - 1]
            j -= 1
        a[j] = v
    return [i for _, i in a]


def _exact_ok(case, seed):
    shape = (case["nx"], case["ny"], case["nz"])
    radii = (case["sx"], case["sy"], case["sz"])
    ranges = (case["rx"], case["ry"], case["rz"])
    t = np.diag([1.0, ranges[0] / ranges[1], ranges[0] / ranges[2]])
    value = lambda v: _covariance(0, ranges[0], 1.0, case["nugget"], np.sqrt(((np.asarray(v, dtype=np.float64) @ t) ** 2).sum(-1)))
    x, y, z = [np.arange(-r, r + 1) for r in radii]
    box = np.stack([g.reshape(-1) for g in np.meshgrid(z, y, x, indexing="ij")][::-1], axis=1)
    key = value(box)
    box, key = box[key > key.max() / 100], key[key > key.max() / 100]
    offsets = -box[_sorted_offsets(key)]
    prop = _krige_inputs(case, np.random.default_rng(seed))["prop"]
    mask, values = prop.mask.astype(bool), prop.data.astype(np.float64)
    pad = np.zeros([n + 2 * r for n, r in zip(shape, radii)], dtype=bool)
    inner = tuple(slice(r, r + n) for n, r in zip(shape, radii))
    pad[inner] = mask
    nodes = np.argwhere(~mask)
    count = np.zeros(len(nodes), dtype=np.int64)
    found = np.zeros((len(nodes), case["nmax"]), dtype=np.int64)
    live = np.arange(len(nodes))
    for k, o in enumerate(offsets):
        p = nodes[live] + o + np.array(radii)
        hit = live[pad[p[:, 0], p[:, 1], p[:, 2]]]
        found[hit, count[hit]] = k
        count[hit] += 1
        live = live[count[live] < case["nmax"]]
    out = values.copy()
    for n in range(1, case["nmax"] + 1):
        at = np.flatnonzero(count == n)
        if not len(at):
            continue
        o = offsets[found[at, :n]]
        a = np.ones((len(at), n + 1, n + 1))
        a[:, n, n] = 0.0
        a[:, :n, :n] = value(o[:, :, None] - o[:, None])
        b = np.ones((len(at), n + 1, 1))
        b[:, :n, 0] = value(o)
        w = np.linalg.solve(a, b)[:, :n, 0]
        cell = nodes[at][:, None] + o
        out[tuple(nodes[at].T)] = (w * values[cell[..., 0], cell[..., 1], cell[..., 2]]).sum(1)
    return out


def exact(case, seed):
    op = case["op"]
    if op == "weights":
        return _exact_weights(case, seed)
    if op == "inc":
        values, mask = _inc_property(case, seed)
        shape = (case["nx"], case["ny"], case["nz"])
        return np.reshape(np.array([float("%E" % v) for v in values]), shape, order="F"), None
    if op == "variogram":
        return _exact_variogram(case, seed)
    # kriging where the search and the systems are small enough for numpy: an
    # unrotated spherical model, data dense enough that the search walks its
    # template everywhere
    if op == "krige" and case["kind"] == "ok" and case["cov"] == 0 and case["angle"] == 0.0 and case["nmax"] <= 16 and \
            case["nx"] * case["ny"] * case["nz"] <= 60000 and case["informed"] >= 0.02 and \
            case["sx"] >= 2 * case["rx"] and case["sy"] >= 2 * case["ry"] and case["sz"] >= 2 * case["rz"]:
        return _exact_ok(case, seed), None
    return None
