"""The work a user of the gridder has it do, as cases that can be timed.

Every case goes through the public Python entry points (the ctypes binding of
the C ABI): gridding and degridding of device tensors, a plan over a batch of
jobs, a request server, and the drop-in gridGPU on host arrays.  Inputs are
seeded synthetic observations with the shapes of the benchmark's workloads;
coordinates are float-representable, the convention of every caller here.

``exact`` evaluates the same sums in 64 bits with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "ska-gpu-grid_gb300"))
import gpugrid as gg  # noqa: E402
import synth  # noqa: E402

G = 8  # oversampling of every workload
DEV = "cuda"


def grid_case(name, pattern, n, vis, support, **more):
    c = {"name": name, "do": "grid", "pattern": pattern, "n": n, "vis": vis, "support": support,
         "pols": 1, "planes": 0, "gauss": False, "f64": False, "uv64": False,
         "mode": "auto", "compensated": True}
    c.update(more)
    return c


def listed():
    return [
        # the smallest request of the served mix: one short observation on a
        # 256^2 grid, where launches and latency are all there is
        grid_case("grid_small", "tracks", 256, 10_000, 8),
        # one ordinary facet of an odd size with FP64 coordinates, support 16
        grid_case("grid_ragged", "tracks", 777, 100_003, 16, uv64=True),
        # a full 64-antenna observation on 4096^2, support 8 (2016 baselines
        # x 2080 samples): the single-job FP32 workload
        grid_case("grid_tracks", "tracks", 4096, 2016 * 2080, 8),
        # w-projection of four polarisations: complex tables, one of 32
        # w-planes per visibility
        grid_case("grid_wproj", "tracks", 2048, 1 << 19, 16, pols=4, planes=32),
        # precision form: 8192^2, uniform disk with outliers, support 32, the
        # Gaussian evaluated on the device
        grid_case("grid_disk", "disk", 8192, 1 << 24, 32, gauss=True, uv64=True),
        # FP64 values and grid, as the reference's <double2, double2>
        grid_case("grid_f64", "uniform", 1024, 1 << 18, 16, f64=True, uv64=True),
        # the gather method asked for by name, on visibilities kept in order
        # of 32-cell uv tiles
        grid_case("gather_tracks", "tracks", 4096, 1 << 20, 8, mode="gather", presorted=True),
        # the default options (scatter, plain FP32 sums)
        grid_case("scatter_default", "tracks", 2048, 1 << 20, 8, mode="scatter",
                  compensated=False),
        # prediction: the visibilities of a full observation from a 4096^2 grid
        {"name": "degrid_tracks", "do": "degrid", "pattern": "tracks", "n": 4096,
         "vis": 2016 * 2080, "support": 8, "pols": 1, "gauss": False, "uv64": False,
         "compensated": True},
        # 256 jobs of mixed grid sides, supports and lengths in one plan
        {"name": "plan_batch", "do": "plan", "jobs": 256, "spec": 5},
        # the same mix as requests to the server, waited for one by one
        {"name": "serve_requests", "do": "serve", "jobs": 128, "spec": 7},
        # the drop-in call on host arrays, all FP64
        {"name": "host_dropin", "do": "host", "pattern": "uniform", "n": 1024, "vis": 1 << 18,
         "support": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["grid", "grid", "grid", "wproj", "disk", "f64", "gather", "scatter",
                       "degrid", "degrid", "plan", "serve", "host"])
    if kind in ("plan", "serve"):
        return {"do": kind, "jobs": _log(rng, 8, 160), "spec": rng.randrange(1 << 20)}
    support = rng.choice([8, 8, 16])
    pattern = rng.choice(["tracks", "tracks", "disk"])
    n = _log(rng, 200, 4096)
    uv64 = rng.random() < 0.3
    if kind == "host":
        return {"do": "host", "pattern": "uniform", "n": _log(rng, 128, 1024),
                "vis": _log(rng, 10_000, 1 << 18), "support": support}
    if kind == "degrid":
        return {"do": "degrid", "pattern": pattern, "n": n, "vis": _log(rng, 10_000, 1 << 21),
                "support": support, "pols": rng.choice([1, 1, 2]), "gauss": rng.random() < 0.2,
                "uv64": uv64, "compensated": rng.random() < 0.7}
    if kind == "grid":
        c = grid_case("", pattern, n, _log(rng, 10_000, 4_000_000), support, uv64=uv64,
                      pols=rng.choice([1, 1, 1, 2]), compensated=rng.random() < 0.8)
    elif kind == "wproj":
        c = grid_case("", pattern, n, _log(rng, 10_000, 1 << 19), support, uv64=uv64,
                      pols=rng.choice([1, 2, 4]), planes=_log(rng, 2, 64))
    elif kind == "disk":
        c = grid_case("", "disk", _log(rng, 512, 8192), _log(rng, 50_000, 1 << 23),
                      rng.choice([16, 32]), gauss=True, uv64=uv64,
                      compensated=rng.random() < 0.7)
    elif kind == "f64":
        c = grid_case("", rng.choice(["tracks", "uniform"]), _log(rng, 200, 2048),
                      _log(rng, 10_000, 1 << 18), support, f64=True, uv64=True)
    elif kind == "gather":
        c = grid_case("", pattern, n, _log(rng, 10_000, 1 << 20), support, uv64=uv64,
                      mode="gather", presorted=rng.random() < 0.5)
    else:
        c = grid_case("", pattern, n, _log(rng, 10_000, 1 << 20), support, uv64=uv64,
                      mode="scatter", compensated=rng.random() < 0.3)
    del c["name"]
    return c


# ---- inputs ---------------------------------------------------------------------

def _coords(c, seed):
    """(vis, 2) float-representable coordinates, float64, on the device"""
    n, vis = c["n"], c["vis"]
    if c["pattern"] == "tracks":
        return synth.job_tracks(n, vis, seed, device=DEV)[0]
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = torch.rand(vis, 2, generator=g, device=DEV, dtype=torch.float64)
    if c["pattern"] == "disk":
        rad, th = 0.45 * n * torch.sqrt(r[:, 0]), 2 * math.pi * r[:, 1]
        uv = n / 2 + torch.stack([rad * torch.cos(th), rad * torch.sin(th)], dim=1)
    else:
        uv = c["support"] + (n - 2 * c["support"]) * r
    return uv.float().double().contiguous()


def _values(c, seed, dtype):
    g = torch.Generator(device=DEV).manual_seed(seed + (1 << 32))
    v = torch.randn(c["vis"], c.get("pols", 1), 2, generator=g, device=DEV, dtype=dtype)
    if c["pattern"] == "disk":  # 1 % outliers
        hot = torch.rand(c["vis"], generator=g, device=DEV) < 0.01
        v[hot] *= 1e3
    return torch.view_as_complex(v)


def _table(support, dtype=torch.complex64):
    t = synth.gcf_table(synth.gaussian_gcf_1d(support))
    return torch.from_numpy(t).to(DEV, dtype).reshape(-1)


def _w_tables(support, planes):
    """planes x [G*G][S][S]: the Gaussian times the phase screen of a w-plane"""
    a = np.arange(support) - support // 2 + 1
    x = a[None, :] - np.arange(G)[:, None] / G                      # [sub][tap]
    r2 = x[None, :, None, :] ** 2 + x[:, None, :, None] ** 2        # [sy, sx, b, a]
    g = synth.gcf_table(synth.gaussian_gcf_1d(support)).reshape(r2.shape)
    w = np.arange(planes) / planes
    t = g[None] * np.exp(1j * math.pi * (4.0 / support) * w[:, None, None, None, None] * r2[None])
    return torch.from_numpy(t).to(DEV, torch.complex64).reshape(-1)


def _plane_index(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + (1 << 33))
    # consecutive samples of a track stay in one w-plane for a while
    runs = -(-c["vis"] // 64)
    w = torch.randint(c["planes"], (runs,), generator=g, device=DEV, dtype=torch.int32)
    return w.repeat_interleave(64)[: c["vis"]].contiguous()


def _specs(c):
    return synth.request_specs(c["jobs"], seed=c["spec"])


def _batch_inputs(c, seed):
    """[(n, S, uv float32, vals)] and where each job's grid lies in one buffer"""
    s = _specs(c)
    jobs, starts, at = [], [], 0
    for k in range(c["jobs"]):
        n, sup, vis = int(s["side"][k]), int(s["S"][k]), int(s["nvis"][k])
        uv, vals = synth.job_tracks(n, vis, seed * 100_003 + k, device=DEV)
        jobs.append((n, sup, uv.float(), vals))
        starts.append(at)
        at += n * n
    return jobs, starts, at


def _options(c):
    return gg.Options(mode=gg.MODES[c.get("mode", "auto")],
                      accum=gg.ACC_COMPENSATED if c["compensated"] else gg.ACC_PLAIN,
                      gcf_kind=gg.GCF_GAUSSIAN if c["gauss"] else gg.GCF_TABLE,
                      layout=gg.LAYOUT_INTERLEAVED, polarizations=c["pols"])


def _one(c, seed):
    """coordinates, values, tables (None: Gaussian) and plane index of a case"""
    f64 = c.get("f64", False)
    uv = _coords(c, seed)
    vals = _values(c, seed, torch.float64 if f64 else torch.float32)
    index = None
    if c.get("presorted"):
        key = (uv[:, 1] // 32).long() * (c["n"] // 32 + 1) + (uv[:, 0] // 32).long()
        order = torch.argsort(key, stable=True)
        uv, vals = uv[order].contiguous(), vals[order].contiguous()
    if c["gauss"]:
        tab = None
    elif c.get("planes", 0):
        tab, index = _w_tables(c["support"], c["planes"]), _plane_index(c, seed)
    else:
        tab = _table(c["support"], torch.complex128 if f64 else torch.complex64)
    return uv, vals, tab, index


def prepare(case, seed):
    c = case
    if c["do"] == "host":
        uv = _coords(c, seed).cpu().numpy()
        return {"do": "host", "n": c["n"], "support": c["support"], "vis": c["vis"],
                "uv": np.ascontiguousarray(uv).view(np.complex128).reshape(-1),
                "vals": _values(c, seed, torch.float64).cpu().numpy().reshape(-1),
                "gcf": synth.gcf_table(synth.gaussian_gcf_1d(c["support"])).reshape(-1),
                "out": np.zeros(gg.padded_size(c["n"], c["support"]), np.complex128)}
    if c["do"] in ("plan", "serve"):
        jobs, starts, cells = _batch_inputs(c, seed)
        out = torch.zeros(cells, dtype=torch.complex64, device=DEV)
        opts = gg.Options(mode=gg.MODE_AUTO, accum=gg.ACC_COMPENSATED,
                          layout=gg.LAYOUT_INTERLEAVED)
        state = {"do": c["do"], "out": out, "inputs": jobs}
        if c["do"] == "plan":
            tabs = {s: _table(s) for s in (8, 16)}
            ctx = gg.Context()
            todo = [gg.Context.make_job(out[a:a + n * n], uv, vals, tabs[sup], n, sup)
                    for (n, sup, uv, vals), a in zip(jobs, starts)]
            torch.cuda.synchronize()
            state.update(tables=tabs, context=ctx, plan=gg.Plan(ctx, opts, todo))
            return state
        srv = gg.Server(streams=3, max_batch_jobs=512, options=opts)
        ids = {s: srv.add_gcf(synth.gcf_table(synth.gaussian_gcf_1d(s)).astype(np.complex64))
               for s in (8, 16)}
        flags = gg.REQ_INPUTS_ON_DEVICE | gg.REQ_OUT_ON_DEVICE
        state["server"] = srv
        state["requests"] = [
            gg.Server.request(uv.data_ptr(), vals.data_ptr(), out[a:a + n * n].data_ptr(),
                              uv.shape[0], n, sup, ids[sup], flags=flags, uv_type=gg.C64)
            for (n, sup, uv, vals), a in zip(jobs, starts)]
        torch.cuda.synchronize()
        return state
    uv, vals, tab, index = _one(c, seed)
    if not c["uv64"]:
        uv = uv.float()
    state = {"do": c["do"], "context": gg.Context(), "options": _options(c), "uv": uv,
             "vals": vals, "table": tab, "index": index, "n": c["n"], "support": c["support"]}
    if c["do"] == "degrid":
        g = torch.Generator(device=DEV).manual_seed(seed + (1 << 34))
        state["grid"] = torch.view_as_complex(torch.randn(
            c["pols"], c["n"], c["n"], 2, generator=g, device=DEV))
        return state
    out = torch.zeros(c["pols"], c["n"], c["n"], device=DEV,
                      dtype=torch.complex128 if c["f64"] else torch.complex64)
    state["out"] = out
    state["job"] = gg.Context.make_job(out, uv, vals, tab, c["n"], c["support"], npts=c["vis"],
                                       gcf_index=index, n_gcf=max(1, c["planes"]))
    return state


def run(state):
    do = state["do"]
    if do == "grid":
        state["context"].grid_job(state["options"], state["job"])
        return state["out"]
    if do == "degrid":
        state["context"].degrid(state["options"], state["grid"], state["uv"], state["vals"],
                                state["table"], state["n"], state["support"])
        return state["vals"]
    if do == "plan":
        state["plan"].launch()
        return state["out"]
    if do == "serve":
        srv = state["server"]
        for t in [srv.submit(r) for r in state["requests"]]:
            srv.wait(t, timeout=60.0)
            srv.release(t)
        return state["out"]
    gg.gridGPU(state["out"], state["uv"], state["vals"], state["vis"], state["n"], state["gcf"],
               state["support"])
    return state["out"]


# ---- what a pass cannot do without -------------------------------------------------

def work(case):
    c = case
    if c["do"] in ("plan", "serve"):
        s = _specs(c)
        vis = s["nvis"].astype(np.float64)
        return {"bytes": float(16 * vis.sum() + 8 * (s["side"].astype(np.float64) ** 2).sum()),
                "flops": float(4 * (vis * s["S"].astype(np.float64) ** 2).sum())}
    vis, pols, s2 = c["vis"], c.get("pols", 1), c["support"] ** 2
    f64 = c["do"] == "host" or c.get("f64", False)
    cplx = 16 if f64 else 8
    uvb = 16 if c["do"] == "host" or c["uv64"] else 8
    planes = c.get("planes", 0)
    table = 0 if c.get("gauss") else max(1, planes) * G * G * s2 * cplx
    b = vis * (uvb + pols * cplx + (4 if planes else 0)) + table
    if c["do"] == "host":
        b += gg.padded_size(c["n"], c["support"]) * cplx
    else:
        b += pols * c["n"] ** 2 * cplx
    # a tap: complex times complex for the w-planes, complex times real for a
    # table or Gaussian without imaginary part, and the addition
    return {"bytes": float(b), "flops": float(vis * pols * s2 * (8 if planes else 4))}


# ---- the same in 64 bits ------------------------------------------------------------

def _steps(uv, n, s):
    """main cell's first tap and sub-kernel row of each coordinate"""
    fl = torch.floor(uv)
    sub = torch.floor(G * (uv - fl)).long()
    return fl.long() - s // 2 + 1, sub


def _taps(c, uv, tab, index):
    """grid cells (n*n: off the grid) and factors, (vis, S, S) each"""
    n, s = c["n"], c["support"]
    first, sub = _steps(uv, n, s)
    k = torch.arange(s, device=DEV)
    x, y = first[:, 0, None] + k, first[:, 1, None] + k
    okx, oky = (x >= 0) & (x < n), (y >= 0) & (y < n)
    cell = torch.where(okx[:, None, :] & oky[:, :, None], y[:, :, None] * n + x[:, None, :], n * n)
    if tab is None:
        d = (k - s // 2 + 1)[None, None, :] - sub[:, :, None].double() / G
        g = torch.exp(-d * d / (2.0 * (s / 4.0) ** 2))
        return cell, g[:, 1, :, None] * g[:, 0, None, :]
    row = sub[:, 1] * G + sub[:, 0]
    if index is not None:
        row = row + index.long() * (G * G)
    return cell, tab.reshape(-1, s, s)[row]


def _exact_grid(c, uv, vals, tab, index):
    n, s, pols = c["n"], c["support"], vals.shape[1]
    re = torch.zeros(pols, n * n + 1, dtype=torch.float64, device=DEV)
    im = torch.zeros_like(re)
    vals = vals.to(torch.complex128)
    if tab is not None:
        tab = tab.to(torch.complex128)
        if not bool((tab.imag != 0).any()):
            tab = tab.real.contiguous()
    step = max(1, (1 << 25) // (s * s))
    for a in range(0, uv.shape[0], step):
        cell, g = _taps(c, uv[a:a + step], tab, None if index is None else index[a:a + step])
        cell = cell.reshape(-1)
        for p in range(pols):
            v = vals[a:a + step, p, None, None]
            if g.is_complex():
                t = (v * g).reshape(-1)
                tr, ti = t.real.contiguous(), t.imag.contiguous()
            else:
                tr, ti = (v.real * g).reshape(-1), (v.imag * g).reshape(-1)
            re[p].index_add_(0, cell, tr)
            im[p].index_add_(0, cell, ti)
    return torch.complex(re[:, :-1], im[:, :-1])


def exact(case, seed):
    c = case
    if c["do"] in ("plan", "serve"):
        jobs, _, _ = _batch_inputs(c, seed)
        tabs = {s: _table(s) for s in (8, 16)}
        return torch.cat([_exact_grid({"n": n, "support": sup}, uv.double(), vals[:, None],
                                      tabs[sup], None).reshape(-1) for n, sup, uv, vals in jobs])
    if c["do"] == "host":
        n, s = c["n"], c["support"]
        tab = torch.from_numpy(synth.gcf_table(synth.gaussian_gcf_1d(s))).to(DEV).reshape(-1)
        g = _exact_grid(c, _coords(c, seed), _values(c, seed, torch.float64), tab, None)
        out = np.zeros(gg.padded_size(n, s), np.complex128)
        head = gg.grid_head(n, s)
        out[head:head + n * n] = g.reshape(-1).cpu().numpy()
        return out
    uv, vals, tab, index = _one(c, seed)
    n = c["n"]
    if c["do"] == "grid":
        return _exact_grid(c, uv, vals, tab, index).reshape(c["pols"], n, n)
    g = torch.Generator(device=DEV).manual_seed(seed + (1 << 34))
    grid = torch.view_as_complex(torch.randn(c["pols"], n, n, 2, generator=g, device=DEV))
    flat = torch.zeros(c["pols"], n * n + 1, dtype=torch.complex128, device=DEV)
    flat[:, :-1] = grid.reshape(c["pols"], -1)
    tab = None if tab is None else tab.to(torch.complex128)
    out = torch.empty(c["vis"], c["pols"], dtype=torch.complex128, device=DEV)
    step = max(1, (1 << 24) // (c["support"] ** 2))
    for a in range(0, c["vis"], step):
        cell, w = _taps(c, uv[a:a + step], tab, None)
        for p in range(c["pols"]):
            out[a:a + step, p] = (flat[p][cell] * w.conj()).sum((1, 2))
    return out
