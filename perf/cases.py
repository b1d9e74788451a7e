"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain values.  `listed()` names twelve of them, `draw()`
gives further ones of the same ranges, `prepare()` makes the inputs a program
holds before the call (on the GPU, from a seed), `run()` is one pass through
the framework's public entry points, `work()` what the pass cannot do without,
and `exact()` the same results in 64 bits from plain torch and numpy.

Kinds of case:

* ``etkf``         one global ETKF cycle on a 2-D grid: H(X), then the analysis
* ``letkf_grid``   one LETKF cycle on a 2-D grid, batched or in the reference's
                   sequential grid-point order, reference semantics
* ``letkf_latlon`` one FP64 LETKF cycle on a lat-lon grid with levels
                   (Hunt transform, Gaspari-Cohn localisation)
* ``letkf_f32``    the same cycle in mixed precision on members kept in FP32
* ``batch``        many uneven global ETKF cases as one replayed CUDA graph
* ``enkf``         the stochastic EnKF with perturbed observations
* ``surrogate``    loss and gradients of the learned column operator
* ``text``         state written as text and read back, observation file read

Every cycle starts from the background the program keeps, so a pass can be
repeated and gives the same analysis.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from metada_gb300 import _lib
from metada_gb300 import kernels as K
from metada_gb300.algorithms import ETKF, LETKF, Ensemble, LatLonGeometry, ObsOperator, Observation, SimpleGeometry
from metada_gb300.synthetic import grf_fields_gpu

DEV = "cuda:0"
F64 = torch.float64
EARTH_KM = 6371.0


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # The reference tutorial's grid: the smallest cycle, where latency counts.
        {"name": "etkf_tutorial", "kind": "etkf", "nx": 36, "ny": 18, "k": 9, "p": 28, "semantics": "reference",
         "rho": 1.0},
        # The plain global analysis: 64 x 64 cells, 32 members, 1024 obs, FP64, reference semantics.
        {"name": "etkf_grid64", "kind": "etkf", "nx": 64, "ny": 64, "k": 32, "p": 1024, "semantics": "reference",
         "rho": 1.05},
        # A global analysis at the upper end of the uneven batch's sizes, symmetric square root, FP64.
        {"name": "etkf_hunt_200k", "kind": "etkf", "nx": 500, "ny": 400, "k": 64, "p": 20000, "semantics": "hunt",
         "rho": 1.05},
        # Local analyses of a 2-D grid with the default options (FP64, reference semantics, all points at once).
        {"name": "letkf_grid", "kind": "letkf_grid", "nx": 144, "ny": 72, "k": 32, "p": 2592, "radius": 6.0,
         "order": "batched", "rho": 1.05},
        # The tutorial's LETKF in the reference's own in-place order.
        {"name": "letkf_sequential", "kind": "letkf_grid", "nx": 36, "ny": 18, "k": 9, "p": 28, "radius": 10.0,
         "order": "sequential", "rho": 1.1},
        # The lat-lon configuration in FP64, the grid and the radius coarser by six (the same local obs counts).
        {"name": "letkf_latlon_fp64", "kind": "letkf_latlon", "nlon": 60, "nlat": 30, "nlev": 10, "nvar": 4, "k": 64,
         "p": 13890, "radius_km": 3000.0, "vradius": 2.0, "rho": 1.05},
        # The headline lat-lon configuration at full size, members kept in FP32.
        {"name": "letkf_latlon_f32", "kind": "letkf_f32", "nlon": 360, "nlat": 180, "nlev": 10, "nvar": 4, "k": 64,
         "p": 500000, "radius_km": 500.0, "vradius": 2.0, "rho": 1.05, "rtps": False, "clustered": 0.0,
         "patch_km": 0.0},
        # The high-resolution configuration (80 members, clustered obs, RTPS) on a grid coarser by four.
        {"name": "letkf_highres_f32", "kind": "letkf_f32", "nlon": 360, "nlat": 180, "nlev": 30, "nvar": 4, "k": 80,
         "p": 312500, "radius_km": 1200.0, "vradius": 2.0, "rho": 0.9, "rtps": True, "clustered": 0.6,
         "patch_km": 3200.0},
        # The uneven batch: independent global analyses in one graph, mixed precision.
        {"name": "uneven_batch", "kind": "batch", "ncases": 128, "n_max": 200000, "p_max": 50000, "fp64": False},
        # The EnKF on the lat-lon state, default precision.
        {"name": "enkf_latlon", "kind": "enkf", "n": 2592000, "k": 64, "p": 500000, "fp64": True},
        # One training batch of the learned column operator, forward and backward.
        {"name": "surrogate_train", "kind": "surrogate", "batch": 4096},
        # A state file written and read back, and an observation file read.
        {"name": "text_files", "kind": "text", "nx": 720, "ny": 360, "lines": 50000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["etkf", "etkf", "letkf_grid", "letkf_grid", "letkf_latlon", "letkf_f32", "letkf_f32", "batch",
                       "enkf", "surrogate", "text"])
    if kind == "etkf":
        nx = _log(rng, 20, 500)
        ny = max(15, int(nx * rng.uniform(0.4, 0.9)))
        k = rng.choice([9, 20, 32, 48, 64, 100, _log(rng, 8, 100)])
        return {"kind": kind, "nx": nx, "ny": ny, "k": k, "p": _log(rng, 25, min(20000, nx * ny // 2)),
                "semantics": rng.choice(["reference", "hunt"]), "rho": rng.choice([1.0, 1.05, 1.1])}
    if kind == "letkf_grid":
        order = rng.choice(["batched", "batched", "sequential"])
        nx = _log(rng, 20, 40) if order == "sequential" else _log(rng, 30, 160)
        ny = max(12, nx // 2 + rng.randint(-3, 3))
        k = rng.choice([9, 12, 20]) if order == "sequential" else rng.choice([9, 20, 32, 48, _log(rng, 8, 64)])
        return {"kind": kind, "nx": nx, "ny": ny, "k": k, "p": max(20, int(nx * ny * rng.uniform(0.04, 0.25))),
                "radius": rng.choice([3.0, 4.5, 6.0]), "order": order, "rho": rng.choice([1.0, 1.05, 1.1])}
    if kind == "letkf_latlon":
        nlon = 2 * _log(rng, 12, 30)
        nlat = nlon // 2 + rng.randint(-1, 1)
        return {"kind": kind, "nlon": nlon, "nlat": nlat, "nlev": rng.randint(3, 10), "nvar": rng.randint(1, 4),
                "k": rng.choice([20, 32, 40, 48, 64, rng.randint(10, 64)]),
                "p": int(nlon * nlat * rng.uniform(2.0, 7.7)), "radius_km": 360.0 / nlon * 500.0,
                "vradius": rng.choice([1.5, 2.0]), "rho": rng.choice([1.0, 1.05])}
    if kind == "letkf_f32":
        nlon = _log(rng, 60, 300)
        nlat = nlon // 2 + rng.randint(-3, 3)
        rtps = rng.random() < 0.5
        return {"kind": kind, "nlon": nlon, "nlat": nlat, "nlev": rng.randint(3, 20), "nvar": rng.randint(1, 5),
                "k": rng.choice([32, 40, 64, 80, 96, rng.randint(20, 96)]),
                "p": int(nlon * nlat * rng.uniform(2.0, 7.7)), "radius_km": 360.0 / nlon * rng.uniform(350.0, 500.0),
                "vradius": rng.choice([1.5, 2.0]), "rho": 0.9 if rtps else 1.05, "rtps": rtps,
                "clustered": 0.6 if rtps else 0.0, "patch_km": 360.0 / nlon * 3200.0}
    if kind == "batch":
        return {"kind": kind, "ncases": _log(rng, 8, 128), "n_max": _log(rng, 20000, 200000),
                "p_max": _log(rng, 5000, 50000), "fp64": rng.random() < 0.3}
    if kind == "enkf":
        return {"kind": kind, "n": _log(rng, 10000, 2500000), "k": rng.choice([20, 32, 48, 64, rng.randint(10, 64)]),
                "p": _log(rng, 500, 400000), "fp64": rng.random() < 0.7}
    if kind == "surrogate":
        return {"kind": kind, "batch": _log(rng, 256, 4096)}
    return {"kind": kind, "nx": _log(rng, 36, 720), "ny": _log(rng, 18, 360), "lines": _log(rng, 100, 50000)}


# ---------------------------------------------------------------- prepare ----
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _f32(x):
    """A config number as the framework reads it."""
    return float(np.float32(x))


def _grid_inputs(c, seed):
    """Truth and members (truth plus independent draws) of a smooth field, point obs at distinct cells."""
    g, r = _gen(seed), np.random.default_rng(seed)
    nx, ny, k, p = c["nx"], c["ny"], c["k"], c["p"]
    f = grf_fields_gpu(k + 1, ny, nx, 8.0 if min(nx, ny) >= 48 else 4.0, g, DEV).double().reshape(k + 1, nx * ny)
    X0 = (f[0][None] + f[1:]).contiguous()
    cells = r.choice(nx * ny, size=p, replace=False)
    xy = np.stack([cells % nx, cells // nx], axis=1).astype(np.int32)
    yo = f[0].cpu().numpy()[cells] + 0.5 * r.standard_normal(p)
    return X0, xy, yo


def _latlon_members(c, g, dtype):
    k, nv, nl, nlat, nlon = c["k"], c["nvar"], c["nlev"], c["nlat"], c["nlon"]
    s = math.sqrt(1.0 - 0.49)
    X = torch.empty((k, nv * nl * nlat * nlon), dtype=dtype, device=DEV)
    truth = None
    for i in range(-1, k):
        f = grf_fields_gpu(nv * nl, nlat, nlon, max(2.0, nlon / 45.0), g, DEV).view(nv, nl, nlat, nlon)
        for l in range(1, nl):
            f[:, l] = 0.7 * f[:, l - 1] + s * f[:, l]
        if truth is None:
            truth = f.reshape(-1).double()
        else:
            X[i] = truth + f.reshape(-1).to(dtype)
    return truth, X


def _latlon_obs(c, r):
    """Obs uniform on the sphere, a share of them in Gaussian patches, at continuous levels."""
    p = c["p"]
    lat = np.rad2deg(np.arcsin(r.uniform(-1.0, 1.0, p)))
    lon = r.uniform(0.0, 360.0, p)
    nc = int(round(c.get("clustered", 0.0) * p))
    if nc:
        cla, clo = np.rad2deg(np.arcsin(r.uniform(-0.9, 0.9, 20))), r.uniform(0.0, 360.0, 20)
        w = r.integers(0, 20, nc)
        sd = np.rad2deg(c["patch_km"] / EARTH_KM)
        lat[:nc] = np.clip(cla[w] + sd * r.standard_normal(nc), -89.9, 89.9)
        lon[:nc] = np.mod(clo[w] + sd * r.standard_normal(nc) / np.cos(np.deg2rad(cla[w])), 360.0)
    return lat, lon, r.uniform(0.0, max(c["nlev"] - 1.0, 0.0), p), r.integers(0, c["nvar"], p).astype(np.int32)


def _h_latlon(X, c, lat, lon, lev, var):
    """Bilinear / linear interpolation of members X (k x n) in 64 bits, p x k; plain torch."""
    nlon, nlat, nlev = c["nlon"], c["nlat"], c["nlev"]
    T = lambda a: torch.as_tensor(a, device=DEV).double()  # noqa: E731
    gx = T(lon) / (360.0 / nlon) - 0.5
    fx = gx - gx.floor()
    i0 = gx.floor().long() % nlon
    i1 = (i0 + 1) % nlon
    gy = ((T(lat) + 90.0) / (180.0 / nlat) - 0.5).clamp(0.0, nlat - 1.0)
    j0 = gy.floor().long().clamp(max=nlat - 2)
    fy = gy - j0
    gz = T(lev).clamp(0.0, nlev - 1.0)
    l0 = gz.floor().long().clamp(max=max(nlev - 2, 0))
    fz = gz - l0
    l1 = (l0 + 1).clamp(max=nlev - 1)
    vb = torch.as_tensor(var, device=DEV).long() * nlev
    out = torch.empty((lat.shape[0], X.shape[0]), dtype=F64, device=DEV)
    at = lambda x, l, j, i: x[((vb + l) * nlat + j) * nlon + i].double()  # noqa: E731
    for m in range(X.shape[0]):
        x = X[m]
        lo, hi = ((at(x, l, j0, i0) * (1 - fx) + at(x, l, j0, i1) * fx) * (1 - fy)
                  + (at(x, l, j0 + 1, i0) * (1 - fx) + at(x, l, j0 + 1, i1) * fx) * fy for l in (l0, l1))
        out[:, m] = lo * (1 - fz) + hi * fz
    return out


def _latlon_inputs(c, seed, dtype):
    g, r = _gen(seed), np.random.default_rng(seed)
    truth, X0 = _latlon_members(c, g, dtype)
    obs = _latlon_obs(c, r)
    yo = _h_latlon(truth[None], c, *obs)[:, 0].cpu().numpy() + r.standard_normal(c["p"])
    return X0, obs, yo


def _batch_inputs(c, seed):
    """Sizes log-uniform, members in FP32-representable values, obs at state nodes."""
    g, r = _gen(seed), np.random.default_rng(1000 + c["ncases"])  # sizes belong to the case, values to the seed
    shapes = [(_log_np(r, 1000, c["n_max"]), int(r.choice([20, 32, 48, 64, 100])), _log_np(r, 100, c["p_max"]))
              for _ in range(c["ncases"])]
    flat = torch.empty(sum(n * k for n, k, _ in shapes), dtype=F64, device=DEV)
    out, at = [], 0
    for n, k, p in shapes:
        truth = torch.randn(n, generator=g, device=DEV)
        X = flat[at: at + n * k].view(k, n)
        X.copy_(truth[None] + torch.randn((k, n), generator=g, device=DEV))
        node = torch.randint(0, n, (p,), generator=g, device=DEV)
        out.append({"at": at, "n": n, "k": k, "node": node,
                    "yo": truth[node].double() + torch.randn(p, generator=g, device=DEV, dtype=F64)})
        at += n * k
    return flat, out


def _log_np(r, lo, hi):
    return int(np.exp(r.uniform(np.log(lo), np.log(hi))))


def _enkf_inputs(c, seed):
    g = _gen(seed)
    n, k, p = c["n"], c["k"], c["p"]
    truth = torch.randn(n, generator=g, device=DEV, dtype=F64)
    X0 = torch.randn((k, n), generator=g, device=DEV, dtype=F64) + truth[None]
    node = torch.randint(0, n, (p,), generator=g, device=DEV)
    yo = truth[node] + 0.5 * torch.randn(p, generator=g, device=DEV, dtype=F64)
    eps = 0.5 * torch.randn((p, k), generator=g, device=DEV, dtype=F64)
    return X0, X0[:, node].T.contiguous(), yo, torch.full((p,), 0.25, dtype=F64, device=DEV), eps


def _mlp_inputs(c, seed):
    """Columns in the operator's ranges and their 16 channels; fan-in uniform weights."""
    g, r = _gen(seed), np.random.default_rng(seed)
    B, nl = c["batch"], 30
    T = 200.0 + 110.0 * torch.rand((B, nl), generator=g, device=DEV)
    q = torch.exp(math.log(1e-6) + math.log(2e4) * torch.rand((B, nl), generator=g, device=DEV))
    w = torch.rand((16, nl), generator=g, device=DEV) / nl
    tau = torch.exp(math.log(100.0) * torch.rand(16, generator=g, device=DEV))
    P = []
    for fo, fi in ((256, 64), (256, 256), (16, 256)):
        P += [r.uniform(-1.0, 1.0, fo * fi) / math.sqrt(fi), 0.1 * r.standard_normal(fo)]
    return T, q, w, tau, torch.tensor(np.concatenate(P), dtype=torch.float32, device=DEV)


def _obs_text(c, seed):
    r = np.random.default_rng(seed)
    m = c["lines"]
    z, y, x = r.integers(1, 40, m), r.integers(0, c["ny"], m), r.integers(0, c["nx"], m)
    v = r.standard_normal((m, 4)) * [0.3, 50.0, 30.0, 2.0]
    lines = ["-" * 80, "Time Z   Y   X   ZNU      XLONG_U    XLAT_U     Simple", "-" * 80]
    lines += ["0 %4d %4d %4d %8.4f %10.4f %10.4f %10.4f" % t
              for t in zip(z.tolist(), y.tolist(), x.tolist(), *v.T.tolist())]
    return ("\n".join(lines) + "\n").encode(), np.stack([x, y, z], axis=1), v


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("etkf", "letkf_grid"):
        X0, xy, yo = _grid_inputs(c, seed)
        cfg = {"inflation": c["rho"], "precision": "fp64"}
        if kind == "etkf":
            cfg["semantics"] = c["semantics"]
        else:
            cfg |= {"semantics": "reference", "order": c["order"], "localization_radius": c["radius"]}
        return {"kind": kind, "X0": X0, "geometry": SimpleGeometry(c["nx"], c["ny"]),
                "obs": Observation(yo, 0.5, grid_xy=xy), "op": ObsOperator(), "config": cfg}
    if kind == "letkf_latlon":
        X0, (lat, lon, lev, var), yo = _latlon_inputs(c, seed, F64)
        return {"kind": kind, "X0": X0, "geometry": LatLonGeometry(c["nlon"], c["nlat"], c["nlev"], c["nvar"]),
                "obs": Observation(yo, 1.0, lat=lat, lon=lon, lev=lev, var=var), "op": ObsOperator(),
                "config": {"inflation": c["rho"], "precision": "fp64", "semantics": "hunt",
                           "localization_radius": c["radius_km"], "vertical_radius": c["vradius"]}}
    if kind == "letkf_f32":
        X0, obs, yo = _latlon_inputs(c, seed, torch.float32)
        la, lo = LatLonGeometry(c["nlon"], c["nlat"], c["nlev"], c["nvar"]).columns()
        plane = c["nlat"] * c["nlon"]
        lat, lon, lev, var = (torch.from_numpy(a).to(DEV) for a in obs)
        return {"kind": kind, "case": dict(c), "X0": X0, "X": torch.empty_like(X0), "lat": lat, "lon": lon,
                "lev": lev, "var": var, "yo": torch.from_numpy(yo).to(DEV),
                "rvar": torch.ones(c["p"], dtype=F64, device=DEV), "col_lat": torch.from_numpy(la).to(DEV),
                "col_lon": torch.from_numpy(lo).to(DEV), "col_base": torch.arange(plane, device=DEV)}
    if kind == "batch":
        flat0, cases = _batch_inputs(c, seed)
        flat = torch.empty_like(flat0)
        plan = K.EtkfBatch([{"X": flat[d["at"]: d["at"] + d["n"] * d["k"]].view(d["k"], d["n"]), "yo": d["yo"],
                             "rvar": torch.ones_like(d["yo"]), "obs_node": d["node"], "rho": 1.05} for d in cases],
                           flags=0, precision=_lib.MG_PREC_FP64 if c["fp64"] else _lib.MG_PREC_MIXED)
        return {"kind": kind, "flat0": flat0, "flat": flat, "plan": plan}
    if kind == "enkf":
        X0, HX, yo, rvar, eps = _enkf_inputs(c, seed)
        return {"kind": kind, "X0": X0, "X": torch.empty_like(X0), "HX": HX, "yo": yo, "rvar": rvar, "eps": eps,
                "precision": _lib.MG_PREC_FP64 if c["fp64"] else _lib.MG_PREC_MIXED}
    if kind == "surrogate":
        T, q, w, tau, P = _mlp_inputs(c, seed)
        mlp = K.MLP(64, 256, 16)
        Y = K.column_op(T, q, w, tau)
        mlp.set_params(P, Y.mean(0), Y.std(0))
        return {"kind": kind, "mlp": mlp, "X": K.column_features(T, q, 64), "Y": Y}
    state = 280.0 + 15.0 * torch.randn(c["nx"] * c["ny"], generator=_gen(seed), device=DEV, dtype=F64)
    return {"kind": kind, "state": state, "nx": c["nx"], "ny": c["ny"], "text": _obs_text(c, seed)[0]}


# -------------------------------------------------------------------- run ----
def run(state):
    s, kind = state, state["kind"]
    if kind in ("etkf", "letkf_grid", "letkf_latlon"):
        ens = Ensemble(s["X0"].clone(), s["geometry"])
        alg = (ETKF if kind == "etkf" else LETKF)(ens, s["obs"], s["op"], s["config"])
        alg.Analyse()
        return {"members": ens.X, "mean": ens.mean_tensor()}
    if kind == "letkf_f32":
        c, X = s["case"], s["X"]
        X.copy_(s["X0"])
        HX = K.hx_latlon(X, c["nlon"], c["nlat"], c["nlev"], s["lat"], s["lon"], s["lev"], s["var"])
        off, idx, dist = K.select_geo(s["col_lat"], s["col_lon"], s["lat"], s["lon"], c["radius_km"])
        plane = c["nlat"] * c["nlon"]
        K.letkf_batched(X, col_base=s["col_base"], nlev=c["nlev"], n_var=c["nvar"], lev_stride=plane,
                        var_stride=c["nlev"] * plane, HX=HX, yo=s["yo"], rvar=s["rvar"], loc_off=off, loc_idx=idx,
                        loc_dist=dist, obs_lev=s["lev"], hsupport=c["radius_km"], vsupport=c["vradius"],
                        rho=c["rho"], flags=_lib.MG_RTPS if c["rtps"] else 0, precision=_lib.MG_PREC_MIXED,
                        want_mean=False)
        return {"members": X}
    if kind == "batch":
        s["flat"].copy_(s["flat0"])
        s["plan"].run(graph=True)
        s["plan"].finish()
        return {"members": s["flat"]}
    if kind == "enkf":
        s["X"].copy_(s["X0"])
        mean, diag = K.enkf(s["X"], s["HX"], s["yo"], s["rvar"], s["eps"], 1.05, precision=s["precision"])
        return {"members": s["X"], "mean": mean, "diag": diag}
    if kind == "surrogate":
        grad, loss = s["mlp"].gradients(s["X"], s["Y"])
        return {"grad": grad, "loss": torch.tensor(loss)}
    text = K.format_state(s["state"], s["nx"], s["ny"])
    values = K.parse_values(text)
    xyz, vals = K.parse_grid_obs(s["text"])
    return {"text": np.frombuffer(text, dtype=np.uint8), "values": values, "xyz": xyz, "vals": vals}


# ------------------------------------------------------------------- work ----
def _local_obs(c):
    """Expected local obs of one analysis."""
    if c["kind"] == "letkf_grid":
        return c["p"] / (c["nx"] * c["ny"]) * math.pi * c["radius"] ** 2
    cap = 0.5 * (1.0 - math.cos(c["radius_km"] / EARTH_KM))
    return c["p"] * cap * min(1.0, 2.0 * c["vradius"] / max(c["nlev"] - 1, 1))


def work(case):
    """Bytes: members and obs read once, analysis written once.  Operations: the products of the method (symmetric
    ones halved), 3 k^3 for a factorisation and inverse, 9 k^3 for a symmetric square root."""
    c, kind = case, case["kind"]
    if kind == "surrogate":
        B, np_ = c["batch"], 64 * 256 + 256 * 256 + 256 * 16
        return {"bytes": 4 * B * 80 + 8 * np_, "flops": 6 * B * np_ - 2 * B * 64 * 256}
    if kind == "text":
        n, m = c["nx"] * c["ny"], c["lines"]
        return {"bytes": n * (8 + 13 + 13 + 8) + m * (62 + 44), "flops": 0}
    if kind == "batch":
        r = np.random.default_rng(1000 + c["ncases"])
        b = f = 0
        for _ in range(c["ncases"]):
            n, k, p = _log_np(r, 1000, c["n_max"]), int(r.choice([20, 32, 48, 64, 100])), _log_np(r, 100, c["p_max"])
            b += 16 * n * k + 24 * p
            f += 2 * n * k * k + p * k * k + 9 * k ** 3
        return {"bytes": b, "flops": f}
    k, p = c["k"], c["p"]
    if kind == "enkf":
        return {"bytes": 16 * c["n"] * k + 16 * p * k + 16 * p + 8 * c["n"],
                "flops": 2 * c["n"] * k * k + 3 * p * k * k + 3 * k ** 3}
    if kind == "etkf":
        n = c["nx"] * c["ny"]
        return {"bytes": 16 * n * k + 8 * n + 24 * p,
                "flops": 2 * n * k * k + p * k * k + (3 if c["semantics"] == "reference" else 9) * k ** 3}
    if kind == "letkf_grid":
        n = c["nx"] * c["ny"]
        return {"bytes": 16 * n * k + 8 * n + 24 * p, "flops": n * (_local_obs(c) * k * k + 3 * k ** 3 + 2 * k * k)}
    pts = c["nlon"] * c["nlat"] * c["nlev"]
    size = 4 if kind == "letkf_f32" else 8
    return {"bytes": 2 * size * pts * c["nvar"] * k + 44 * p,
            "flops": pts * (_local_obs(c) * k * k + 9 * k ** 3 + 2 * c["nvar"] * k * k)}


# ------------------------------------------------------------------ exact ----
def _transform(A, b, k, scale, chol):
    """wa = scale A^-1 b and W = sqrt((k-1) scale) A^-1/2 (symmetric), or sqrt((k-1) scale) chol_L(A^-1)."""
    if chol:
        Pa = scale * torch.linalg.inv(A)
        return (Pa @ b[..., None])[..., 0], math.sqrt(k - 1) * torch.linalg.cholesky(0.5 * (Pa + Pa.mT))
    lam, V = torch.linalg.eigh(A)
    wa = (V @ ((V.mT @ b[..., None]) * (scale / lam)[..., None]))[..., 0]
    return wa, math.sqrt((k - 1) * scale) * (V * lam.rsqrt()[..., None, :]) @ V.mT


def _h_grid(X, c, xy):
    """IDW4 of the reference at integer cells: the cell itself by 1e12 against its neighbours by 1 and 1/sqrt(2)."""
    nx, ny = c["nx"], c["ny"]
    xy = torch.as_tensor(xy, device=DEV).long()
    i0, j0 = xy[:, 0], xy[:, 1]
    num = den = 0.0
    for dj in (0, 1):
        for di in (0, 1):
            i, j = (i0 + di).clamp(max=nx - 1), (j0 + dj).clamp(max=ny - 1)
            d = torch.sqrt(((i - i0) ** 2 + (j - j0) ** 2).double())
            w = torch.where(d == 0, torch.full_like(d, 1e12), 1.0 / d)
            num, den = num + w[:, None] * X[:, j * nx + i].T, den + w[:, None]
    return num / den


def _global(X, HX, yo, rinv, rho, compat):
    k = X.shape[0]
    ym = HX.mean(1, keepdim=True)
    Y, d = HX - ym, yo - ym[:, 0]
    A = Y.T @ (rinv[:, None] * Y) + (k - 1) / (1.0 if compat else rho) * torch.eye(k, dtype=F64, device=DEV)
    wa, W = _transform(A, Y.T @ (rinv * d), k, 1.0, compat)
    xm = X.mean(0)
    return xm[None] + (rho if compat else 1.0) * (wa[:, None] + W).T @ (X - xm[None]), xm


def _gc(z):
    z = z.abs()
    near = (((-0.25 * z + 0.5) * z + 0.625) * z - 5.0 / 3.0) * z * z + 1.0
    far = ((((z / 12.0 - 0.5) * z + 0.625) * z + 5.0 / 3.0) * z - 5.0) * z + 4.0 - 2.0 / (3.0 * z.clamp(min=1e-30))
    return torch.where(z <= 1.0, near, torch.where(z < 2.0, far, torch.zeros_like(z))).clamp(min=0.0)


def _exact_sequential(X, c, xy, yo):
    X, k, nx, ny = X.cpu().numpy().copy(), c["k"], c["nx"], c["ny"]
    rho, rad = _f32(c["rho"]), _f32(c["radius"])
    i0, j0 = xy[:, 0].astype(np.int64), xy[:, 1].astype(np.int64)
    nb, wt = [], []
    for dj in (0, 1):
        for di in (0, 1):
            i, j = np.minimum(i0 + di, nx - 1), np.minimum(j0 + dj, ny - 1)
            d = np.sqrt((i - i0) ** 2.0 + (j - j0) ** 2.0)
            nb.append(j * nx + i)
            wt.append(np.where(d == 0, 1e12, 1.0 / np.where(d == 0, 1.0, d)))
    nb, wt = np.array(nb), np.array(wt)
    for g in range(nx * ny):
        loc = np.nonzero(np.sqrt((g % nx - xy[:, 0]) ** 2.0 + (g // nx - xy[:, 1]) ** 2.0) <= rad)[0]
        x = X[:, g].copy()
        xm = x.mean()
        if not len(loc):
            X[:, g] = xm + (x - xm) * math.sqrt(rho)
            continue
        H = (X[:, nb[:, loc]] * wt[:, loc]).sum(1) / wt[:, loc].sum(0)
        Y = (H - H.mean(0)).T
        Pa = rho * np.linalg.inv((k - 1) * np.eye(k) + Y.T @ Y)
        wa = Pa @ (Y.T @ (yo[loc] - H.mean(0)))
        W = math.sqrt(k - 1) * np.linalg.cholesky(0.5 * (Pa + Pa.T))
        X[:, g] = xm + (x - xm) * wa + (x - xm) * W.sum(1)
    return X, X.mean(0)


def _exact_grid_batched(X, c, xy, yo):
    k, rho = c["k"], _f32(c["rho"])
    HX = _h_grid(X, c, xy)
    ym = HX.mean(1, keepdim=True)
    Y, d = HX - ym, torch.as_tensor(yo, device=DEV) - ym[:, 0]
    Z = (Y[:, :, None] * Y[:, None, :]).reshape(len(yo), k * k)
    P = torch.as_tensor(xy, device=DEV).double()
    g = torch.arange(X.shape[1], device=DEV)
    pts = torch.stack([g % c["nx"], g // c["nx"]], 1).double()
    out, xm, eye = torch.empty_like(X), X.mean(0), torch.eye(k, dtype=F64, device=DEV)
    for a in range(0, X.shape[1], 4096):
        q = pts[a: a + 4096]
        m = (((q[:, None] - P[None]) ** 2).sum(2).sqrt() <= _f32(c["radius"])).double()
        wa, W = _transform((m @ Z).view(-1, k, k) + (k - 1) * eye, m @ (Y * d[:, None]), k, rho, True)
        xp = (X[:, a: a + 4096] - xm[None, a: a + 4096]).T
        xa = xp * (wa + W.sum(2))
        xa = torch.where(m.sum(1, keepdim=True) > 0, xa, math.sqrt(rho) * xp)
        out[:, a: a + 4096] = xm[None, a: a + 4096] + xa.T
    return out, out.mean(0)


def _exact_latlon(X, c, obs, yo, rho, rtps):
    """Dense weights of every point against every obs, in chunks of columns."""
    k, nl, nv, plane = c["k"], c["nlev"], c["nvar"], c["nlon"] * c["nlat"]
    lat, lon, lev, var = obs
    HX = _h_latlon(X, c, lat, lon, lev, var)
    ym = HX.mean(1, keepdim=True)
    Y, d = HX - ym, torch.as_tensor(yo, device=DEV) - ym[:, 0]
    iu = torch.triu_indices(k, k, device=DEV)
    Z = Y[:, iu[0]] * Y[:, iu[1]]
    Yd = Y * d[:, None]
    T = lambda a: torch.deg2rad(torch.as_tensor(a, device=DEV).double())  # noqa: E731
    cla = T(-90.0 + (np.arange(c["nlat"]) + 0.5) * 180.0 / c["nlat"]).repeat_interleave(c["nlon"])
    clo = T((np.arange(c["nlon"]) + 0.5) * 360.0 / c["nlon"]).repeat(c["nlat"])
    la, lo = T(lat), T(lon)
    out = torch.empty((k, nv, nl, plane), dtype=F64, device=DEV)
    Xv = X.view(k, nv, nl, plane)
    eye = torch.eye(k, dtype=F64, device=DEV)
    diag = (k - 1) / (1.0 if rtps else rho)
    for l in range(nl):
        sel = slice(None)
        wv = 1.0
        if nl > 1:
            dl = (torch.as_tensor(lev, device=DEV) - l).abs()
            sel = torch.nonzero(dl <= c["vradius"])[:, 0]
            wv = _gc(dl[sel] / (0.5 * c["vradius"]))
        for a in range(0, plane, 2048):
            s = slice(a, min(a + 2048, plane))
            h = torch.sin(0.5 * (la[None, sel] - cla[s, None])) ** 2 + (
                torch.cos(cla[s, None]) * torch.cos(la[None, sel]) * torch.sin(0.5 * (lo[None, sel] - clo[s, None])) ** 2)
            km = 2.0 * EARTH_KM * torch.asin(h.clamp(max=1.0).sqrt())
            w = _gc(km / (0.5 * c["radius_km"])) * wv
            G = torch.empty((w.shape[0], k, k), dtype=F64, device=DEV)
            t = w @ Z[sel]
            G[:, iu[0], iu[1]] = t
            G[:, iu[1], iu[0]] = t
            wa, W = _transform(G + diag * eye, w @ Yd[sel], k, 1.0, False)
            none = (w.sum(1) == 0)[:, None, None]
            x = Xv[:, :, l, s].double()
            xm = x.mean(0)
            xp = (x - xm[None]).permute(2, 1, 0)  # points, variables, members
            xa = torch.where(none, xp * (1.0 if rtps else math.sqrt(rho)), xp @ W)
            inc = torch.where(none, torch.zeros_like(xa[..., :1]), xp @ wa[..., None])
            if rtps:
                sb, sa = xp.pow(2).sum(2, keepdim=True).sqrt(), xa.pow(2).sum(2, keepdim=True).sqrt()
                xa = torch.where(none, xa, xa * (1.0 + rho * (sb - sa) / sa))
            out[:, :, l, s] = (xm.T[..., None] + inc + xa).permute(2, 1, 0)
    out = out.view(k, -1)
    return out, out.mean(0)


def _exact_mlp(c, seed):
    """Weights rounded to BF16 as the network keeps them, everything else in 64 bits."""
    T, q, w, tau, P = _mlp_inputs(c, seed)
    X = torch.cat([(T - 255.0) / 30.0, 100.0 * q, torch.zeros((T.shape[0], 4), device=DEV)], 1).double()
    cq = q.double().cumsum(1)
    Y = ((w.double()[None] * torch.exp(-tau.double()[None, :, None] * cq[:, None])) * (T.double() ** 4 / 1e8)[:, None]).sum(2)
    Y = Y.float()
    t = ((Y - Y.mean(0)) / Y.std(0)).double()
    at, W = 0, []
    for fo, fi in ((256, 64), (256, 256), (16, 256)):
        W.append(P[at: at + fo * fi].bfloat16().double().view(fo, fi).requires_grad_())
        W.append(P[at + fo * fi: at + fo * fi + fo].double().requires_grad_())
        at += fo * fi + fo
    h = torch.nn.functional.silu(X @ W[0].T + W[1])
    h = torch.nn.functional.silu(h @ W[2].T + W[3])
    loss = ((h @ W[4].T + W[5] - t) ** 2).mean()
    loss.backward()
    return {"grad": torch.cat([x.grad.reshape(-1) for x in W]), "loss": loss.detach()}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "surrogate":
        return _exact_mlp(c, seed)
    if kind == "text":
        xyz, v = _obs_text(c, seed)[1:]
        state = 280.0 + 15.0 * torch.randn(c["nx"] * c["ny"], generator=_gen(seed), device=DEV, dtype=F64)
        back = np.array([float("%12.6f" % x) for x in state.tolist()])
        vals = np.array([[float("%.4f" % x) for x in row] for row in v.tolist()])
        return {"text": None, "values": back, "xyz": None, "vals": vals}
    if kind == "batch":
        flat, cases = _batch_inputs(c, seed)
        for d in cases:
            X = flat[d["at"]: d["at"] + d["n"] * d["k"]].view(d["k"], d["n"])
            X.copy_(_global(X, X[:, d["node"]].T, d["yo"], torch.ones_like(d["yo"]), 1.05, False)[0])
        return {"members": flat}
    if kind == "enkf":
        X, HX, yo, rvar, eps = _enkf_inputs(c, seed)
        k = c["k"]
        ym = HX.mean(1, keepdim=True)
        Y, d = HX - ym, yo - ym[:, 0]
        A = Y.T @ (Y / rvar[:, None]) + (k - 1) * torch.eye(k, dtype=F64, device=DEV)
        T = torch.linalg.solve(A, Y.T @ ((d[:, None] + eps - Y) / rvar[:, None]))
        xm = X.mean(0)
        Xp = math.sqrt(1.05) * (X - xm[None])
        Xa = xm[None] + Xp + T.T @ Xp
        am = Xa.mean(0)
        return {"members": Xa, "mean": am,
                "diag": {"innovation_norm": d.norm(), "background_spread": Xp.pow(2).mean().sqrt(),
                         "analysis_spread": (Xa - am[None]).pow(2).mean().sqrt()}}
    if kind in ("etkf", "letkf_grid"):
        X, xy, yo = _grid_inputs(c, seed)
        if kind == "etkf":
            Xa, m = _global(X, _h_grid(X, c, xy), torch.as_tensor(yo, device=DEV),
                            torch.full((len(yo),), 4.0, dtype=F64, device=DEV), _f32(c["rho"]),
                            c["semantics"] == "reference")
        else:
            Xa, m = (_exact_sequential if c["order"] == "sequential" else _exact_grid_batched)(X, c, xy, yo)
        return {"members": Xa, "mean": m}
    # Dense weights: points x obs in the vertical window x k^2 / 2 products, and an eigen-solve a point.
    pts = c["nlon"] * c["nlat"] * c["nlev"]
    window = min(1.0, 2.0 * c["vradius"] / max(c["nlev"] - 1, 1))
    if pts * (c["p"] * window * c["k"] ** 2 / 2 + 60.0 * c["k"] ** 3) > 2.5e12:
        return None
    X, obs, yo = _latlon_inputs(c, seed, torch.float32 if kind == "letkf_f32" else F64)
    rho = c["rho"] if kind == "letkf_f32" else _f32(c["rho"])
    Xa, m = _exact_latlon(X, c, obs, yo, rho, c.get("rtps", False))
    return {"members": Xa} if kind == "letkf_f32" else {"members": Xa, "mean": m}
