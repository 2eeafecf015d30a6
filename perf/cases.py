"""The framework's measured cases: whole-grid kriging and simulation calls, as a
program makes them, from a few wells on a small grid to 16.8 M cells.

A case names a path ("kind"), how the call is made ("api"), the grid, the
conditioning points, the covariance model, the neighbour limit and the
precision. "host" cases call ``geo_bsd`` on numpy arrays, the way HPGL's Python
users do; "device" cases call the C ABI's ``_ex`` entry points on CUDA tensors,
the way a program that keeps its grids on the GPU does. Sizes and models are
those of ``geo_bsd.workloads``, of the test suite, or odd sizes between them.

Kinds: ok / sk (ordinary / simple kriging), lvm (locally varying mean), ik
(indicator kriging, one model per category), mik (median IK, two categories),
cok (collocated cokriging, Markov model I), sgs / sis (sequential Gaussian /
indicator simulation), loo (leave-one-out cross-validation with gradients).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpgl-reborn_b200"))
import geo_bsd  # noqa: E402
from geo_bsd import hpgl_wrap as W  # noqa: E402
from geo_bsd.loo import LooGeometry, loo_cv_mse  # noqa: E402

UNDEFINED = -99.0
COVS = {"spherical": 0, "exponential": 1, "gaussian": 2}
MARGINALS = (0.40, 0.25, 0.15, 0.12, 0.08)


def _case(name, kind, api, dims, points, cov, ranges, azimuth, nugget, k, precision="fp64", layout="uniform",
          variance=False):
    c = dict(name=name, kind=kind, api=api, nx=dims[0], ny=dims[1], nz=dims[2], points=points, cov=cov,
             range_x=ranges[0], range_y=ranges[1], range_z=ranges[2], azimuth=azimuth, nugget=nugget, k=k,
             precision=precision, layout=layout, variance=variance)
    if name is None:
        del c["name"]
    return c


def listed():
    return [
        # The smallest call: a handful of wells on a coarse grid, through the
        # Python API; host tables, launches and synchronisations are all of it.
        _case("few_wells", "ok", "host", (24, 20, 6), 30, "spherical", (10, 10, 5), 0.0, 0.1, 32, variance=True),
        # A sector model with a drift: every neighbourhood below the limit.
        _case("lvm_sparse", "lvm", "device", (97, 61, 43), 350, "exponential", (14, 11, 6), 20.0, 0.05, 32,
              variance=True),
        # Fitting a variogram by cross-validation: one loss with its gradients.
        _case("loo_gradient", "loo", "device", (200, 200, 50), 4000, "gaussian", (18, 18, 6), 30.0, 0.05, 24),
        # A half-million-cell grid with short neighbourhoods.
        _case("ok_small", "ok", "device", (100, 100, 50), 2000, "spherical", (10, 10, 5), 0.0, 0.1, 12,
              variance=True),
        # An odd-sized grid from and to pageable numpy arrays, automatic mean.
        _case("sk_api", "sk", "host", (151, 133, 57), 13700, "exponential", (17, 13, 6), 45.0, 0.05, 21),
        # The 8.4 M cell grid in double precision, with its kriging variance,
        _case("ok_grid", "ok", "device", (256, 256, 128), 83886, "exponential", (30, 15, 6), 30.0, 0.05, 32,
              variance=True),
        # and with the FP32-refined option.
        _case("ok_grid_refined", "ok", "device", (256, 256, 128), 83886, "exponential", (30, 15, 6), 30.0, 0.05, 32,
              precision="fp32_refined"),
        # Wells in clusters, long neighbourhoods, badly conditioned systems: the largest call.
        _case("ok_clustered", "ok", "device", (512, 512, 64), 33554, "gaussian", (40, 40, 8), 0.0, 1e-3, 64,
              layout="clustered"),
        # Facies probabilities: five categories, each with its own model.
        _case("ik_facies", "ik", "device", (200, 200, 100), 60000, "spherical", (18, 18, 6), 0.0, 0.1, 24),
        # A secondary attribute on half of the cells.
        _case("cokriging", "cok", "device", (160, 144, 80), 18432, "exponential", (30, 15, 6), 30.0, 0.05, 32),
        # One realisation of a continuous property,
        _case("sgs", "sgs", "device", (256, 256, 128), 83886, "exponential", (30, 15, 6), 30.0, 0.05, 32),
        # and one of a facies model.
        _case("sis", "sis", "device", (200, 200, 100), 60000, "spherical", (18, 18, 6), 0.0, 0.1, 24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges: grids of 2 k to 16 M cells with odd
    axes among them, 4 to 64 neighbours, any model, density and rotation."""
    kind = rng.choice(["ok", "ok", "ok", "sk", "sk", "lvm", "ik", "mik", "cok", "sgs", "sis", "loo"])
    if kind == "loo":
        dims = tuple(_log_int(rng, lo, hi) for lo, hi in ((60, 256), (60, 256), (20, 64)))
        return _case(None, "loo", "device", dims, _log_int(rng, 300, 8000), rng.choice(sorted(COVS)),
                     (rng.randint(8, 30), rng.randint(8, 30), rng.randint(3, 8)), rng.choice([0.0, 30.0, 110.0]), 0.05,
                     rng.randint(6, 32))
    ranges = (rng.randint(8, 32), rng.randint(8, 24), rng.randint(3, 8))
    k = _log_int(rng, 4, {"ok": 64, "sk": 64}.get(kind, 32))
    systems = len(MARGINALS) if kind in ("ik", "sis") else 1
    most = min({"sgs": 9.9e6, "sis": 9.9e6}.get(kind, 16e6), 9e11 / (systems * _flops(k, 2)))
    cells = math.exp(rng.uniform(math.log(2000.0), math.log(most)))
    flat = rng.uniform(0.15, 0.6)  # the grid's height against its width
    wide = (cells / flat) ** (1.0 / 3.0)
    skew = rng.uniform(0.8, 1.25)
    dims = (max(8, int(wide * skew)), max(8, int(wide / skew)), max(4, int(wide * flat)))
    n = dims[0] * dims[1] * dims[2]
    cov = rng.choice(sorted(COVS))
    nugget = rng.choice([0.05, 0.1, 0.2]) if cov == "gaussian" else rng.choice([0.0, 0.05, 0.1])
    points = max(4, int(n * math.exp(rng.uniform(math.log(0.003), math.log(0.02)))))
    api = rng.choice(["device", "host"]) if kind in ("ok", "sk") and n < 3e6 else "device"
    precision = rng.choice(["fp64", "fp64", "fp32_refined"]) if kind in ("ok", "sk", "lvm", "ik", "mik") else "fp64"
    variance = kind in ("ok", "sk", "lvm") and precision == "fp64" and rng.random() < 0.5
    return _case(None, kind, api, dims, points, cov, ranges, rng.choice([0.0, 0.0, 30.0, 75.0]), nugget, k, precision,
                 variance=variance)


# ------------------------------------------------------------------- inputs
def _dims(c):
    return c["nx"], c["ny"], c["nz"]


def _cells(c):
    return c["nx"] * c["ny"] * c["nz"]


def _ranges(c):
    return float(c["range_x"]), float(c["range_y"]), float(c["range_z"])


def _field(dims, ranges, gen):
    """A unit-variance Gaussian field (white noise under an anisotropic Gaussian
    kernel), flat with x fastest, on the GPU."""
    nx, ny, nz = dims
    f = torch.fft.rfftn(torch.randn((nz, ny, nx), generator=gen, device="cuda"))
    for axis, (n, a) in enumerate(zip((nz, ny, nx), reversed(ranges))):
        s = max(a / math.sqrt(12.0), 1e-6)
        w = (torch.fft.rfftfreq if axis == 2 else torch.fft.fftfreq)(n, device="cuda") * (2 * math.pi * s)
        shape = [1, 1, 1]
        shape[axis] = -1
        f = f * torch.exp(-0.5 * w * w).reshape(shape)
    f = torch.fft.irfftn(f, s=(nz, ny, nx)).reshape(-1)
    return (f - f.mean()) / f.std()


def _nodes(c, rng):
    """The conditioning cells: anywhere, or within 50 Gaussian clusters."""
    nx, ny, nz = _dims(c)
    if c["layout"] == "uniform":
        return np.sort(rng.choice(_cells(c), c["points"], replace=False))
    centres = np.stack([rng.uniform(0, d, 50) for d in _dims(c)], axis=1)
    p = np.rint(centres[rng.integers(0, 50, 4 * c["points"])] + rng.normal(0.0, 8.0, (4 * c["points"], 3)))
    p = p[((p >= 0) & (p < (nx, ny, nz))).all(axis=1)].astype(np.int64)
    node = p[:, 0] + nx * p[:, 1] + nx * ny * p[:, 2]
    _, first = np.unique(node, return_index=True)
    return np.sort(node[np.sort(first)[:c["points"]]])


def _inputs(c, seed):
    """The case's data, on the GPU, from the seed alone."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(int(seed))
    n = _cells(c)
    node = torch.from_numpy(_nodes(c, rng)).cuda()
    m = int(node.numel())
    mask = torch.zeros(n, dtype=torch.uint8, device="cuda")
    mask[node] = 1
    d = {"mask": mask, "node": node}
    kind = c["kind"]
    if kind in ("ik", "sis", "mik"):
        cuts = MARGINALS if kind != "mik" else (0.55, 0.45)
        field = _field(_dims(c), _ranges(c), gen)
        at = torch.sort(field[::max(1, n // 1000000)]).values
        at = at[[min(len(at) - 1, int(q * len(at))) for q in np.cumsum(cuts)[:-1]]]
        cats = torch.bucketize(field, at, right=True).to(torch.uint8)
        d["data"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        d["data"][node] = cats[node]
        return d
    if kind == "loo":
        d["values"] = _field(_dims(c), _ranges(c), gen)[node].double()
        return d
    data = torch.full((n,), UNDEFINED, device="cuda")
    z = torch.randn(m, generator=gen, device="cuda")
    data[node] = torch.exp(0.5 * z) if kind in ("ok", "sk") else z
    d["data"] = data
    if kind == "lvm":
        x, y = torch.arange(c["nx"], device="cuda"), torch.arange(c["ny"], device="cuda")
        a, b, e = rng.uniform(-0.02, 0.02, 3)
        mean = 0.3 + a * x[None, None, :] + b * y[None, :, None] + e * torch.arange(c["nz"], device="cuda")[:, None, None]
        wave = torch.sin(2 * math.pi * x / c["nx"])[None, None, :] * torch.cos(2 * math.pi * y / c["ny"])[None, :, None]
        d["mean"] = (mean + 0.4 * wave).float().reshape(-1).contiguous()
        d["data"][node] += d["mean"][node]
    if kind == "cok":
        have = torch.rand(n, generator=gen, device="cuda") < 0.5
        second = torch.randn(n, generator=gen, device="cuda")
        second[node] += 0.6 * data[node]
        d["second"] = torch.where(have, second, torch.full_like(second, UNDEFINED))
        d["second_mask"] = have.to(torch.uint8)
    return d


def _model(c):
    return dict(covariance_type=COVS[c["cov"]], ranges=_ranges(c), angles=(float(c["azimuth"]), 0.0, 0.0), sill=1.0,
                nugget=float(c["nugget"]))


def _search(c):
    return dict(radiuses=(c["range_x"], c["range_y"], c["range_z"]), max_neighbours=c["k"])


def _category_params(c):
    """One model per category, around the case's ranges."""
    out = (W._HPGL_IK_PARAMS * len(MARGINALS))()
    for i, p in enumerate(MARGINALS):
        f = 2.0 / 3.0 + i / 6.0
        r = [max(2, int(round(v * f))) for v in _ranges(c)]
        out[i] = W._HPGL_IK_PARAMS(covariance_type=COVS[c["cov"]], ranges=tuple(float(v) for v in r),
                                   angles=(float(c["azimuth"]), 0.0, 0.0), sill=1.0,
                                   nugget=c["nugget"] * (0.5 + 0.25 * i), radiuses=tuple(r), max_neighbours=c["k"],
                                   marginal_prob=p)
    return out


def _loo_matrix(c):
    """The anisotropy transform over ranges[0] for a rotation about z."""
    a = math.radians(c["azimuth"])
    rot = torch.tensor([[math.cos(a), math.sin(a), 0.0], [-math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]],
                       dtype=torch.float64, device="cuda")
    return torch.diag(1.0 / torch.tensor(_ranges(c), dtype=torch.float64, device="cuda")) @ rot


def _xyz(c, node):
    nx, ny = c["nx"], c["ny"]
    return torch.stack([node % nx, (node // nx) % ny, node // (nx * ny)], dim=1)


def _loo_neighbours(c, node):
    """The k nearest other points within the range, by the model's distance."""
    u = _xyz(c, node).double() @ _loo_matrix(c).T
    idx = []
    for part in torch.split(torch.arange(len(u), device="cuda"), 1024):
        h2 = (u[part][:, None, :] - u[None, :, :]).square().sum(-1)
        h2[torch.arange(len(part), device="cuda"), part] = math.inf
        h2 = torch.where(h2 < 1.0, h2, math.inf)
        val, at = torch.sort(h2, dim=1, stable=True)
        idx.append(torch.where(val[:, :c["k"]].isfinite(), at[:, :c["k"]], -1))
    idx = torch.cat(idx).int()
    return idx.contiguous(), (idx >= 0).sum(1).int()


def prepare(case, seed):
    c = case
    d = _inputs(c, seed)
    n = _cells(c)
    kind = c["kind"]
    s = {"case": c, "in": d, "dims": (C.c_int * 3)(*_dims(c))}
    if kind == "loo":
        nb, cnt = _loo_neighbours(c, d["node"])
        m = len(d["node"])
        s["geom"] = LooGeometry(pts_xyz=_xyz(c, d["node"]).int().contiguous(), values=d["values"],
                                targets=torch.arange(m, dtype=torch.int32, device="cuda"), nb_idx=nb, nb_cnt=cnt,
                                k=c["k"], cov_type=COVS[c["cov"]], nodes=d["node"].cpu().numpy())
        return s
    if c["api"] == "host":
        shape = _dims(c)
        s["prop"] = geo_bsd.ContProperty(d["data"].cpu().numpy().reshape(shape, order="F"),
                                         d["mask"].cpu().numpy().reshape(shape, order="F"))
        s["grid"] = geo_bsd.SugarboxGrid(*shape)
        mod = _model(c)
        s["model"] = geo_bsd.CovarianceModel(mod["covariance_type"], mod["ranges"], mod["angles"], 1.0, mod["nugget"])
        s["in"] = None
        return s
    opt = W._HPGL_B200_OPTIONS()
    opt.precision = W.FP32_REFINED if c["precision"] == "fp32_refined" else W.FP64_PLAIN
    opt.flags = W.FLAG_DEVICE_POINTERS
    s["opt"] = opt
    s["stream"] = torch.cuda.Stream()
    opt.stream = s["stream"].cuda_stream
    category = kind in ("ik", "mik", "sis")
    out = {"data": torch.empty(n, dtype=torch.uint8 if category else torch.float32, device="cuda"),
           "mask": torch.empty(n, dtype=torch.uint8, device="cuda")}
    if not category and kind != "sgs":  # the output starts as a clone of the input
        out["data"].copy_(d["data"])
        out["mask"].copy_(d["mask"])
    if kind in ("ok", "sk", "lvm", "cok", "sgs"):
        out["status"] = torch.empty(n, dtype=torch.int8, device="cuda")
        opt.status = out["status"].data_ptr()
    if c["variance"]:
        out["variance"] = torch.empty(n, dtype=torch.float64, device="cuda")
        opt.variance = out["variance"].data_ptr()
    if kind == "ik":
        out["probs"] = torch.empty(n * len(MARGINALS), device="cuda")
        opt.ik_probs = out["probs"].data_ptr()
    s["out"] = out
    if kind in ("ok", "sk"):
        s["par"] = W._HPGL_SK_PARAMS(automatic_mean=1, mean=0.0, **_model(c), **_search(c))
    elif kind == "lvm":
        s["par"] = W._HPGL_OK_PARAMS(**_model(c), **_search(c))
    elif kind == "mik":
        s["par"] = W._HPGL_MEDIAN_IK_PARAMS(marginal_probs=(0.55, 0.45), **_model(c), **_search(c))
    elif kind == "cok":
        s["par"] = W._HPGL_COK_M1_PARAMS(primary_mean=0.0, secondary_mean=0.0, secondary_variance=1.0,
                                         correlation_coef=0.6, **_model(c), **_search(c))
    elif kind == "sgs":
        s["par"] = W._HPGL_SGS_PARAMS(kriging_kind=1, seed=42, min_neighbours=0, **_model(c), **_search(c))
    else:
        s["par"] = _category_params(c)
    return s


# --------------------------------------------------------------------- pass
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "loo":
        return _run_loo(s)
    if c["api"] == "host":
        radiuses = (c["range_x"], c["range_y"], c["range_z"])
        call = geo_bsd.ordinary_kriging if kind == "ok" else geo_bsd.simple_kriging
        r = call(s["prop"], s["grid"], radiuses, c["k"], s["model"], precision=c["precision"],
                 return_variance=c["variance"])
        prop, var = r if c["variance"] else (r, None)
        out = {"data": prop.data, "mask": prop.mask}
        if var is not None:
            out["variance"] = var
        return out
    lib, d, o = W._hpgl_so, s["in"], s["out"]
    dims, opt, par = s["dims"], C.byref(s["opt"]), s["par"]
    if kind in ("sgs", "sis"):  # in place, on a copy of the conditioning data
        with torch.cuda.stream(s["stream"]):
            o["data"].copy_(d["data"])
            o["mask"].copy_(d["mask"])
        if kind == "sgs":
            rc = lib.hpgl_b200_sgs_ex(dims, o["data"].data_ptr(), o["mask"].data_ptr(), None, None, None,
                                      C.byref(par), opt)
        else:
            rc = lib.hpgl_b200_sis_ex(dims, o["data"].data_ptr(), o["mask"].data_ptr(), None, par, len(MARGINALS),
                                      None, 42, 0, opt)
        W.check(rc, kind)
        return o
    data, mask, out, out_mask = d["data"].data_ptr(), d["mask"].data_ptr(), o["data"].data_ptr(), o["mask"].data_ptr()
    if kind in ("ok", "sk"):
        rc = lib.hpgl_b200_cont_kriging_ex(0 if kind == "ok" else 1, dims, data, mask, C.byref(par), out, out_mask, opt)
    elif kind == "lvm":
        rc = lib.hpgl_b200_lvm_kriging_ex(dims, data, mask, d["mean"].data_ptr(), C.byref(par), out, out_mask, opt)
    elif kind == "ik":
        rc = lib.hpgl_b200_indicator_kriging_ex(dims, data, mask, par, len(MARGINALS), out, out_mask, opt)
    elif kind == "mik":
        rc = lib.hpgl_b200_median_ik_ex(dims, data, mask, C.byref(par), out, out_mask, opt)
    else:
        rc = lib.hpgl_b200_cokriging_ex(1, dims, data, mask, d["second"].data_ptr(), d["second_mask"].data_ptr(),
                                        C.byref(par), None, out, out_mask, opt)
    W.check(rc, kind)
    return o


def _loo_parameters(c):
    return [torch.tensor(v, dtype=torch.float64, requires_grad=True)
            for v in (_ranges(c), (float(c["azimuth"]), 0.0, 0.0), 1.0, float(c["nugget"]))]


def _run_loo(s):
    par = _loo_parameters(s["case"])
    values = s["geom"].values.detach().requires_grad_(True)
    loss = loo_cv_mse(s["geom"], *par, values)
    loss.backward()
    return {"loss": loss.detach(), "ranges": par[0].grad, "angles": par[1].grad, "sill": par[2].grad,
            "nugget": par[3].grad, "values": values.grad}


# --------------------------------------------------------------------- work
def _flops(n, rhs):
    """Assembly, factorisation and solves of one system of n neighbours."""
    return n ** 3 / 3 + n * n / 2 + 2 * rhs * n * n + 30 * (n * (n + 1) / 2 + n) + 2 * rhs * n


def work(case):
    c = case
    n, m, kind = _cells(c), c["points"], c["kind"]
    inside = 4.0 / 3.0 * math.pi * c["range_x"] * c["range_y"] * c["range_z"] * m / n
    k = min(float(c["k"]), max(1.0, inside))
    if kind == "loo":
        return {"bytes": m * (12 + 8 + 4 * k + 4 + 4 + 8), "flops": 4 * m * _flops(k, 3)}
    systems = {"ik": len(MARGINALS), "sis": len(MARGINALS)}.get(kind, 1)
    rhs = 2 if kind in ("ok", "cok") else 1
    per_cell = {"ik": 2 + 2 + 4 * len(MARGINALS), "mik": 4, "sis": 4, "lvm": 15, "cok": 16, "sgs": 11}.get(kind, 11)
    if c["api"] == "host":
        per_cell = 10
    per_cell += 8 if c["variance"] else 0
    return {"bytes": float(n * per_cell), "flops": float((n - m) * systems * _flops(k, rhs))}


# -------------------------------------------------------------------- exact
def _cov(c, d):
    """The model's covariance of displacements d [..., 3] in 64 bits."""
    r0 = c["range_x"]
    h = r0 * (d.double() @ _loo_matrix(c).T).square().sum(-1).sqrt()
    part = 1.0 - c["nugget"]
    if c["cov"] == "gaussian":
        v = part * torch.exp(-3 * (h / r0) ** 2)
    elif c["cov"] == "exponential":
        v = part * torch.exp(-3 * h / r0)
    else:
        v = torch.where(h > r0, 0.0, part * (1 - 1.5 * h / r0 + 0.5 * (h / r0) ** 3))
    return torch.where(h < 1e-4, 1.0, v)


def _exact_grid(c, seed):
    """OK / SK / LVM where every neighbourhood holds all of the points in reach
    (box and covariance above a hundredth of the sill); with more of them than
    the limit, equal covariances leave the choice to the search's order, and
    there is no one value."""
    d = _inputs(c, seed)
    node, mask, n = d["node"], d["mask"], _cells(c)
    p = _xyz(c, node)
    z = d["data"][node].double()
    rad = torch.tensor((c["range_x"], c["range_y"], c["range_z"]), device="cuda")
    simple = c["kind"] != "ok"
    if not simple and (c["cov"] != "spherical" or c["azimuth"]):
        return None  # points beyond the box may belong to an ordinary neighbourhood
    mean = torch.zeros(n, dtype=torch.float64, device="cuda")
    if c["kind"] == "lvm":
        mean = d["mean"].double()
        z = (d["data"][node] - d["mean"][node]).double()
    elif simple:
        mean += z.mean()
        z = (d["data"][node] - z.mean().float()).double()
    est, var = d["data"].double(), torch.zeros(n, dtype=torch.float64, device="cuda")
    status = torch.full((n,), -1, dtype=torch.int8, device="cuda")
    for cell in torch.split(torch.nonzero(mask == 0).reshape(-1), 20000):
        x = _xyz(c, cell)
        off = p[None, :, :] - x[:, None, :]
        b = _cov(c, off)
        near = (off.abs() <= rad).all(-1) & (b > 0.01)
        cnt = near.sum(1)
        if int(cnt.max()) > c["k"]:
            return None
        k = max(1, int(cnt.max()))
        at = torch.sort(near.byte(), dim=1, descending=True, stable=True).indices[:, :k]
        live = torch.arange(k, device="cuda")[None, :] < cnt[:, None]
        q = p[at]
        dq = q[:, :, None, :] - q[:, None, :, :]
        A = _cov(c, dq)
        if simple:
            A = A * (dq.abs() <= rad).all(-1)
        A = A * (live[:, :, None] & live[:, None, :]) + torch.diag_embed((~live).double())
        rhs = torch.stack([torch.gather(b, 1, at) * live, live.double(), z[at] * live], dim=2)
        y = torch.linalg.solve_triangular(torch.linalg.cholesky(A), rhs, upper=False)
        G = y.transpose(1, 2) @ y
        if simple:
            e, v = mean[cell] + G[:, 0, 2], 1.0 - G[:, 0, 0]
        else:
            mu = (G[:, 0, 1] - 1.0) / G[:, 1, 1]
            e, v = G[:, 0, 2] - mu * G[:, 1, 2], 1.0 - G[:, 0, 0] + mu * G[:, 0, 1] - mu
        none = cnt == 0
        est[cell] = torch.where(none, mean[cell] if simple else torch.full_like(e, UNDEFINED), e)
        var[cell] = torch.where(none, -1.0, v.clamp(min=0.0))
        status[cell] = none.to(torch.int8)
    out = {"data": est, "mask": None}
    if c["api"] == "host":
        shape = (c["nz"], c["ny"], c["nx"])
        out = {"data": est.reshape(shape).permute(2, 1, 0).contiguous(), "mask": None}
        if c["variance"]:
            out["variance"] = var.reshape(shape).permute(2, 1, 0).contiguous()
        return out
    out["status"] = status
    if c["variance"]:
        out["variance"] = var
    return out


def _exact_loo(c, seed):
    d = _inputs(c, seed)
    nb, cnt = _loo_neighbours(c, d["node"])
    ranges, angles, sill, nugget = (t.detach().cuda().requires_grad_(True) for t in _loo_parameters(c))
    z = d["values"].clone().requires_grad_(True)
    a = angles * (math.pi / 180.0)
    cs, sn = torch.cos(a), torch.sin(a)
    one, zero = torch.ones_like(cs[0]), torch.zeros_like(cs[0])
    rz = torch.stack([cs[0], sn[0], zero, -sn[0], cs[0], zero, zero, zero, one]).reshape(3, 3)
    ry = torch.stack([cs[1], zero, -sn[1], zero, one, zero, sn[1], zero, cs[1]]).reshape(3, 3)
    rx = torch.stack([one, zero, zero, zero, cs[2], sn[2], zero, -sn[2], cs[2]]).reshape(3, 3)
    M = torch.diag(1.0 / ranges) @ (rx @ ry @ rz)

    def cov(disp):
        u2 = (disp.double() @ M.T).square().sum(-1)
        same = (disp == 0).all(-1)
        u = torch.where(same, 1.0, u2).sqrt()
        part = sill - nugget
        if c["cov"] == "gaussian":
            v = part * torch.exp(-3 * u * u)
        elif c["cov"] == "exponential":
            v = part * torch.exp(-3 * u)
        else:
            v = torch.where(u > 1, torch.zeros_like(u), part * (1 - 1.5 * u + 0.5 * u ** 3))
        return torch.where(same, sill, v)

    p = _xyz(c, d["node"])
    live = torch.arange(c["k"], device="cuda")[None, :] < cnt[:, None]
    at = nb.long().clamp(min=0)
    q = p[at]
    A = cov(q[:, :, None, :] - q[:, None, :, :]) * (live[:, :, None] & live[:, None, :])
    A = A + torch.diag_embed((~live).double())
    rhs = torch.stack([cov(q - p[:, None, :]) * live, live.double(), z[at] * live], dim=2)
    y = torch.linalg.solve_triangular(torch.linalg.cholesky(A), rhs, upper=False)
    G = y.transpose(1, 2) @ y
    ok = cnt > 0
    s11 = torch.where(ok, G[:, 1, 1], 1.0)
    zhat = G[:, 0, 2] - (G[:, 0, 1] - 1.0) / s11 * G[:, 1, 2]
    err = torch.where(ok, zhat - z, 0.0)
    loss = (err * err).sum() / ok.sum().clamp(min=1)
    loss.backward()
    return {"loss": loss.detach(), "ranges": ranges.grad, "angles": angles.grad, "sill": sill.grad,
            "nugget": nugget.grad, "values": z.grad}


def exact(case, seed):
    if case["kind"] == "loo":
        return _exact_loo(case, seed)
    if case["kind"] in ("ok", "sk", "lvm") and _cells(case) * case["points"] < 1e9:
        return _exact_grid(case, seed)
    return None
