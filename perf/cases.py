"""The work that users of the GPP / FF library have it do, as measurable cases.

A case is a dict of plain values: the entry point ("kind"), the shape, the
precision and the options.  The kinds:

  gpp    Context.gpp        the GPP sum (also its half sum, "half")
  real   Context.gpp_real   the real-valued GPP sum
  ff     Context.ff         the full-frequency kernels, with the band x G x G' schDt contraction
  serve  Server             a burst of uneven GPP requests over resident epsilon / wtilde

Inputs have the shapes and value distributions of the package's own synthetic
inputs (fortkernels_gb300.inputs), drawn on the GPU from the seed.  "where" says
where the caller's arrays live: "device" (the large arrays and the outputs are
GPU tensors, the calls only enqueue) or "host" (numpy arrays in and out).
"""
import math

import numpy as np
import torch

import __graft_entry__

fk = __graft_entry__.load_package()

TO1, LIMITTWO, LIMITONE = 1e-6, 0.25, 1.0 / (1e-6 * 4.0)


def _gpp(name, nb, nv, nc, ng, precision, where="device", dist="uniform", achstemp=False, half=False):
    return {"name": name, "kind": "gpp", "nb": nb, "nv": nv, "nc": nc, "ng": ng, "precision": precision,
            "where": where, "dist": dist, "achstemp": achstemp, "half": half}


def _real(name, nb, nv, nc, ng, precision, dist="branch"):
    return {"name": name, "kind": "real", "nb": nb, "nv": nv, "nc": nc, "ng": ng, "precision": precision,
            "where": "device", "dist": dist}


def _ff(name, nb, nv, nc, ng, nf, ne, precision, where="device", schdt=True):
    return {"name": name, "kind": "ff", "nb": nb, "nv": nv, "nc": nc, "ng": ng, "nf": nf, "ne": ne,
            "precision": precision, "where": where, "schdt": schdt}


def listed():
    return [
        # the smallest call: a drop-in user's first try, numpy arrays and the default precision; ragged sizes,
        # every branch of the solver
        _gpp("gpp_fp64_host_64x777x7", 64, 2, 777, 7, "fp64", where="host", dist="branch"),
        # a small ragged mixed call with the static remainder, as one of many in a self-energy loop
        _gpp("gpp_mixed_130x4099x70", 130, 2, 4099, 70, "mixed", dist="branch", achstemp=True),
        # the mini-app at full size, the benchmark's default, in both precisions
        _gpp("gpp_mixed_512x32768x20", 512, 2, 32768, 20, "mixed"),
        _gpp("gpp_fp64_512x32768x20", 512, 2, 32768, 20, "fp64"),
        # the reference's canonical command line `gppKer 512 2 32768 20` (ngpown = 32768 / 20)
        _gpp("gpp_mixed_512x32768x1638", 512, 2, 32768, 1638, "mixed"),
        # the sequential driver's half sum (gppsum = 1)
        _gpp("gpp_half_mixed_512x32768x20", 512, 2, 32768, 20, "mixed", dist="branch", half=True),
        # the real-valued driver
        _real("real_mixed_512x32768x20", 512, 2, 32768, 20, "mixed"),
        # a small full-frequency call at the default precision, ragged sizes
        _ff("ff_fp64_40x640x48x6", 40, 2, 640, 48, 6, 5, "fp64"),
        # the full-frequency contraction of the benchmark, in both precisions
        _ff("ff_mixed_512x4096x512x15", 512, 2, 4096, 512, 15, 10, "mixed"),
        _ff("ff_fp64_512x4096x512x15", 512, 2, 4096, 512, 15, 10, "fp64"),
        # the large full-frequency contraction: 17 GB for each of the two epsilon arrays
        _ff("ff_mixed_2048x8192x4096x32", 2048, 2, 8192, 4096, 32, 10, "mixed"),
        # a burst of uneven requests through the request server
        {"name": "serve_32_requests", "kind": "serve", "requests": 32, "nc_lo": 2048, "nc_hi": 32768, "levels": 4,
         "nv": 2, "plan": 7},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.choice(["gpp", "gpp", "gpp", "half", "real", "ff", "ff", "serve"])
        precision = rng.choice(["fp64", "mixed"])
        if kind == "serve":
            lo = _log_int(rng, 1000, 4096)
            return {"kind": "serve", "requests": rng.randint(8, 32), "nc_lo": lo, "nc_hi": _log_int(rng, lo, 32768),
                    "levels": rng.randint(2, 6), "nv": rng.randint(0, 4), "plan": rng.randint(0, 1 << 20)}
        nb, nv = _log_int(rng, 16, 1024), rng.choice([0, 1, 2, 2, 2, 4, 5])
        where = "host" if rng.random() < 0.15 else "device"
        dist = rng.choice(["uniform", "branch"])
        if kind == "ff":
            nc, ng = _log_int(rng, 300, 9000), _log_int(rng, 16, 1024)
            nf, ne = _log_int(rng, 4, 40), _log_int(rng, 3, 40)
            case = _ff("", nb, nv, nc, min(ng, nc), nf, ne, precision, where, rng.random() < 0.8)
        else:
            nc, ng = _log_int(rng, 300, 32768), _log_int(rng, 4, 1638)
            if kind == "real":
                case = _real("", nb, nv, nc, min(ng, nc), precision, dist)
            else:
                case = _gpp("", nb, nv, nc, min(ng, nc), precision, where, "branch" if kind == "half" else dist,
                            achstemp=kind == "gpp" and rng.random() < 0.2, half=kind == "half")
        del case["name"]
        w = work(case)
        if w["flops"] <= (6.5e11 if precision == "mixed" else 1.2e11) and (where == "device" or w["bytes"] < 4e8):
            return case


# ------------------------------------------------------------------ work

def _planes(c):
    """(R planes, A planes) an FF call reads: every R plane with the schDt contraction; the correction term's
    brackets of band energies U[-1, 1] against frequencies on [0, 2] (wx = 0.5 - e in [-0.5, 1.5])."""
    a = min(c["nf"], int(math.ceil(0.75 * (c["nf"] - 1))) + 1)
    return (c["nf"] if c["schdt"] else a), a


def work(c):
    if c["kind"] == "serve":
        flops = byts = 0
        for nb, nc, ng in _stream(c):
            flops += 8 * nb * 3 * ng * nc
            byts += 16 * (nb * nc + nb * ng + 2 * ng * nc + nb)
        return {"bytes": byts, "flops": flops}
    nb, nc, ng = c["nb"], c["nc"], c["ng"]
    if c["kind"] == "ff":
        r, a = _planes(c)
        rows = (2.0 / 15.0) * nb  # bands that read one plane of the correction term
        return {"bytes": 16 * (nb * nc + nb * ng + (r + a) * ng * nc + (nb * c["nf"] if c["schdt"] else 0)),
                "flops": 8 * nc * ng * (nb * r + rows * a) + 20 * nb * c["nf"] * c["ne"]}
    if c["kind"] == "real":
        return {"bytes": 8 * (nb * nc + nb * ng + 2 * ng * nc + nb), "flops": 2 * nb * 3 * ng * nc + 30 * 3 * ng * nc}
    if c["half"]:  # ig < igp over evenly spread columns, each term with its conjugate pair
        return {"bytes": 16 * (2 * nb * nc + 2 * ng * nc + nb), "flops": 8 * nb * 3 * ng * nc + 60 * 3 * ng * nc}
    return {"bytes": 16 * (nb * nc + nb * ng + 2 * ng * nc + nb),
            "flops": 8 * nb * (4 if c["achstemp"] else 3) * ng * nc + 60 * 3 * ng * nc}


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(gen, shape, lo, hi):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64).mul_(hi - lo).add_(lo)


def _cu(gen, shape):
    x = torch.rand(tuple(shape) + (2,), generator=gen, device="cuda", dtype=torch.float64)
    return torch.view_as_complex(x.sub_(0.5))


def _wtilde(gen, shape, dist, wx):
    """wtilde of the package's synthetic GPP inputs: re U[0.5, 2], im U[-0.05, 0.05], or ("branch") drawn around
    each frequency so that every branch of the solver is taken."""
    far = torch.complex(_rand(gen, shape, 0.5, 2.0), _rand(gen, shape, -0.05, 0.05))
    if dist == "uniform":
        return far
    centre = torch.tensor(wx, device="cuda", dtype=torch.float64)[
        torch.randint(0, 3, shape, generator=gen, device="cuda")]
    kind = torch.randint(0, 4, shape, generator=gen, device="cuda")
    mag = torch.where(kind == 0, _rand(gen, shape, 0.3, 0.7), 10.0 ** _rand(gen, shape, -5.0, -2.0))
    ang = _rand(gen, shape, 0.0, 2 * math.pi)
    near = torch.complex(centre + mag * torch.cos(ang), mag * torch.sin(ang))
    size = 10.0 ** _rand(gen, shape, -4.0, -1.0)
    zero = torch.complex(size * torch.cos(ang), size * torch.sin(ang))
    return torch.where(kind == 2, far, torch.where(kind == 3, zero, near))


def _inputs(c, seed):
    """The arrays of a gpp / real / ff case: the large ones on the GPU, the small ones numpy."""
    gen, rng = _gen(seed), np.random.default_rng(int(seed))
    nb, nv, nc, ng = c["nb"], c["nv"], c["nc"], c["ng"]
    p = {"number_bands": nb, "nvband": min(nv, nb), "ncouls": nc, "ngpown": ng,
         "vcoul": rng.uniform(0.1, 1.0, nc), "indinv": np.arange(nc, dtype=np.int32),
         "aqsmtemp": _cu(gen, (nb, nc)), "aqsntemp": _cu(gen, (nb, nc))}
    if c["kind"] == "ff":
        nf = c["nf"]
        grid = np.linspace(0.0, 2.0, nf)
        pref = np.append(np.diff(grid), grid[-1] - grid[-2]) / 3.14
        pref[0] *= 0.5
        pref[-1] *= 0.5
        p.update(nFreq=nf, nfreqeval=c["ne"], ekq=rng.uniform(-1.0, 1.0, nb), dFreqGrid=grid,
                 dFreqBrd=np.full(nf, 0.5 + 0.1j), pref=pref, pref_zb=0.5 / 3.14, freqevalmin=0.0, freqevalstep=0.5,
                 occ=1.0, inv_igp_index=np.arange(ng, dtype=np.int32))
        diag = torch.arange(ng, device="cuda")
        for key in ("I_epsR_array", "I_epsA_array"):
            p[key] = _cu(gen, (nf, ng, nc))
            p[key][:, diag, diag] += 1.0
    else:
        wx = [9.0, 10.0, 11.0]
        p["inv_igp_index"] = (np.arange(ng, dtype=np.int64) * nc // ng).astype(np.int32)
        p["wx_array"] = np.array(wx)
        p["I_eps_array"] = _cu(gen, (ng, nc))
        p["wtilde_array"] = _wtilde(gen, (ng, nc), c["dist"], wx)
        if c["kind"] == "real":
            for k in ("aqsmtemp", "aqsntemp", "I_eps_array", "wtilde_array"):
                p[k] = p[k].real.contiguous()
    return p


def _stream(c):
    """(number_bands, ncouls, ngpown) of each request of a served burst."""
    rng = np.random.default_rng(c["plan"])
    levels = np.unique(np.geomspace(c["nc_lo"], c["nc_hi"], c["levels"]).round().astype(int))
    return [(int(rng.choice([128, 256, 512, 1024])), int(nc), max(1, int(nc) // 64))
            for nc in rng.choice(levels, c["requests"])]


def _serve_inputs(c, seed):
    """Per ncouls of the stream: one pool of wavefunction rows and one epsilon / wtilde, which its requests share."""
    gen, rng = _gen(seed), np.random.default_rng(int(seed))
    pools = {}
    for nc in sorted({nc for _, nc, _ in _stream(c)}):
        ng = max(1, nc // 64)
        rows = max(nb for nb, n, _ in _stream(c) if n == nc)
        pools[nc] = {"aqsmtemp": _cu(gen, (rows, nc)), "aqsntemp": _cu(gen, (rows, nc)),
                     "I_eps_array": _cu(gen, (ng, nc)), "wtilde_array": _wtilde(gen, (ng, nc), "uniform", None),
                     "vcoul": torch.from_numpy(rng.uniform(0.1, 1.0, nc)).cuda(),
                     "inv_igp_index": torch.from_numpy((np.arange(ng) * nc // ng).astype(np.int32)).cuda(),
                     "indinv": torch.arange(nc, dtype=torch.int32, device="cuda"),
                     "wx_array": torch.tensor([9.0, 10.0, 11.0], dtype=torch.float64, device="cuda")}
    return pools


# ------------------------------------------------------------ prepare, run

_kept = {}  # the program's handle: one Context, kept while it works on one problem


def _context(c):
    key = repr(sorted((k, v) for k, v in c.items() if k != "name"))
    if _kept.get("key") != key:
        _kept.clear()
        _kept.update(key=key, ctx=fk.Context(0))
    return _kept["ctx"]


def prepare(case, seed):
    c = case
    if c["kind"] == "serve":
        pools = _serve_inputs(c, seed)
        stream = _stream(c)
        srv = fk.Server(0, hbm_bytes=16 << 30, max_active=16)
        torch.cuda.synchronize()
        for nc, q in pools.items():
            srv.resident_put(2 * nc, q["I_eps_array"])
            srv.resident_put(2 * nc + 1, q["wtilde_array"])
        out = {"achtemp": np.zeros((len(stream), 3), np.complex128),
               "asxtemp": np.zeros((len(stream), 3), np.complex128),
               "acht_n1_loc": np.zeros(sum(nb for nb, _, _ in stream), np.complex128)}
        reqs, at = [], 0
        for i, (nb, nc, ng) in enumerate(stream):
            p = {k: v for k, v in pools[nc].items() if k not in ("I_eps_array", "wtilde_array")}
            p.update(number_bands=nb, nvband=c["nv"], ncouls=nc, ngpown=ng)
            reqs.append((p, nc, {"achtemp": out["achtemp"][i], "asxtemp": out["asxtemp"][i],
                                 "acht_n1_loc": out["acht_n1_loc"][at:at + nb]}))
            at += nb
        return {"kind": "serve", "srv": srv, "reqs": reqs, "out": out}
    p = _inputs(c, seed)
    state = {"kind": c["kind"], "ctx": _context(c), "p": p, "precision": c["precision"], "flags": 0, "out": None}
    if c["kind"] == "ff":
        state["flags"] = fk.FK_FF_SPLIT_ACHD | (fk.FK_FF_SCHDT_GEMM if c["schdt"] else 0)
        shapes = {k: (c["ne"],) for k in ("asxDtemp", "achDtemp", "achDtemp_cor", "ach2Dtemp")}
        shapes.update(achsDtemp=(1,), schDt_matrix=(c["nb"], c["nf"]))
    else:
        shapes = {"achtemp": (3,), "asxtemp": (3,), "acht_n1_loc": (c["nb"],)}
        if c["kind"] == "gpp":
            state["flags"] = (fk.FK_GPP_HALF_SUM if c["half"] else 0) | (fk.FK_GPP_ACHSTEMP if c["achstemp"] else 0)
            shapes["achstemp"] = (1,) if c["achstemp"] else None
    if c["where"] == "host":
        for k, v in p.items():
            if isinstance(v, torch.Tensor):
                p[k] = v.cpu().numpy()
    else:
        if c["kind"] != "ff":  # the FF planner reads its small arrays on the host
            for k, v in p.items():
                if isinstance(v, np.ndarray):
                    p[k] = torch.from_numpy(v).cuda()
        dtype = torch.float64 if c["kind"] == "real" else torch.complex128
        state["out"] = {k: None if s is None else torch.zeros(s, dtype=dtype, device="cuda") for k, s in shapes.items()}
        torch.cuda.synchronize()  # the library works on its own stream
    return state


def run(state):
    if state["kind"] == "serve":
        srv = state["srv"]
        tickets = [srv.submit(p, eps_key=2 * nc, wtilde_key=2 * nc + 1, out=out) for p, nc, out in state["reqs"]]
        for t in tickets:
            srv.wait(t)
        return state["out"]
    call = {"gpp": state["ctx"].gpp, "real": state["ctx"].gpp_real, "ff": state["ctx"].ff}[state["kind"]]
    out = call(state["p"], state["precision"], state["flags"], out=state["out"])
    return {k: v for k, v in out.items() if v is not None}


# ------------------------------------------------------------------ exact

def _columns(p):
    """igp of each column and its vcoul, on the GPU (every index of these inputs maps inside [0, ncouls))."""
    dev = lambda a: a.cuda() if isinstance(a, torch.Tensor) else torch.from_numpy(np.asarray(a)).cuda()  # noqa: E731
    igp = dev(p["indinv"]).long()[dev(p["inv_igp_index"]).long()]
    return igp, dev(p["vcoul"])[igp]


def _exact_gpp(p, achstemp=False):
    nb, nv, nc, ng = p["number_bands"], p["nvband"], p["ncouls"], p["ngpown"]
    aqsn, aqsm = p["aqsntemp"][:nb], p["aqsmtemp"][:nb]
    igp, vc = _columns(p)
    wx = [float(x) for x in p["wx_array"]]
    ach, asx = torch.zeros(3, nb, dtype=torch.complex128, device="cuda"), torch.zeros(3, dtype=torch.complex128, device="cuda")
    stat = torch.zeros(1, dtype=torch.complex128, device="cuda")
    step = max(1, int(2e7) // nc)
    for h in range(0, ng, step):
        wt, eps = p["wtilde_array"][h:h + step], p["I_eps_array"][h:h + step]
        w = torch.conj(aqsm[:, igp[h:h + step]]) * vc[h:h + step]
        wt2 = wt * wt
        for iw in range(3):
            wd = wx[iw] - wt
            wdr = wd.real ** 2 + wd.imag ** 2
            delw = wt * torch.conj(wd) / wdr
            dr = delw.real ** 2 + delw.imag ** 2
            on = (wdr > LIMITTWO) & (dr < LIMITONE)
            zero = torch.zeros_like(eps)
            ach[iw] += 0.5 * (w * (aqsn @ torch.where(on, delw * eps, zero).T)).sum(1)
            if nv:
                om = wt2 * eps
                ssx = torch.where(on, om / wx[iw] ** 2,
                                  torch.where(dr > TO1, -om / (4.0 * wt2 * (delw + 0.5)) * delw, zero))
                asx[iw] += (w[:nv] * (aqsn[:nv] @ ssx.T)).sum()
        if achstemp:
            stat -= 0.5 * (w * (aqsn @ eps.T)).sum()
    out = {"achtemp": ach.sum(1), "asxtemp": asx, "acht_n1_loc": ach[2].clone()}
    if achstemp:
        out["achstemp"] = stat
    return out


def _exact_half(p):
    nb, nv, nc, ng = p["number_bands"], p["nvband"], p["ncouls"], p["ngpown"]
    aqsn, aqsm = p["aqsntemp"], p["aqsmtemp"]
    igp, vc = _columns(p)
    wx = [float(x) for x in p["wx_array"]]
    ig = torch.arange(nc, device="cuda")[None, :]
    ach, asx = torch.zeros(3, nb, dtype=torch.complex128, device="cuda"), torch.zeros(3, dtype=torch.complex128, device="cuda")
    step = max(1, int(2e7) // nc)
    for h in range(0, ng, step):
        g = igp[h:h + step]
        wt, eps = p["wtilde_array"][h:h + step], p["I_eps_array"][h:h + step]
        cm, v = torch.conj(aqsm[:, g]), vc[h:h + step]
        member = (ig < g[:, None] - 1) & (ig % 512 != 511)
        om = wt * wt * eps
        small = (om.abs() < TO1) & (ig < g[:, None])
        brk = torch.where(small.any(1), small.to(torch.int32).argmax(1), torch.full_like(g, nc))
        flag = ig < torch.minimum(g, brk)[:, None]
        zero = torch.zeros_like(eps)
        for iw in range(3):
            wd = wx[iw] - wt
            wdr = wd.real ** 2 + wd.imag ** 2
            delw = wt / wd
            on = (wdr < LIMITTWO) | (delw.real ** 2 + delw.imag ** 2 > LIMITONE)
            sch = torch.where(on, delw * eps, zero)
            d = torch.where(member, sch, zero)
            diag = torch.where((g > 0) & (g % 512 == 0), sch[torch.arange(len(g), device="cuda"), g], zero[:, 0])
            s = cm * (aqsn @ d.T) + torch.conj(cm * (aqsm @ d.T)) + cm * aqsn[:, g] * diag
            ach[iw, nv:] += 0.5 * (s * v)[nv:].sum(1)
            if nv:
                dl = wd * (0.5 / wt)
                off = (wdr < 0.25) | (dl.real ** 2 + dl.imag ** 2 < TO1)
                fsch = torch.where(off, zero, wt * eps / wd)
                fssx = torch.where(off, torch.where(wt.abs() > TO1, -om / (4.0 * wt * wt * (1.0 + dl)), zero),
                                   om / (wx[iw] ** 2 - wt * wt))
                keep2 = flag & (ig != g[:, None] - 1)
                for x, acc in ((fsch, 0), (fssx, 1)):
                    t = cm[:nv] * (aqsn[:nv] @ torch.where(flag, x, zero).T) \
                        + torch.conj(cm[:nv] * (aqsm[:nv] @ torch.where(keep2, x, zero).T))
                    if acc == 0:
                        ach[iw, :nv] += 0.5 * (t * v).sum(1)
                    else:
                        asx[iw] += (t * v).sum()
    return {"achtemp": ach.sum(1), "asxtemp": asx, "acht_n1_loc": ach[2].clone()}


def _exact_real(p):
    nb, nv, nc, ng = p["number_bands"], p["nvband"], p["ncouls"], p["ngpown"]
    aqsn, aqsm = p["aqsntemp"], p["aqsmtemp"]
    igp, vc = _columns(p)
    wx = [float(x) for x in p["wx_array"]]
    ach, asx = torch.zeros(3, nb, dtype=torch.float64, device="cuda"), torch.zeros(3, dtype=torch.float64, device="cuda")
    step = max(1, int(2e7) // nc)
    for h in range(0, ng, step):
        wt, eps = p["wtilde_array"][h:h + step], p["I_eps_array"][h:h + step]
        rows = wt.shape[0]
        w = aqsm[:, igp[h:h + step]] * vc[h:h + step]
        d, on = [], []
        for iw in range(3):
            wd = wx[iw] - wt
            delw = wt / wd
            d.append(delw * eps)
            on.append((wd * wd > LIMITTWO) & (delw * delw < LIMITONE))
            if nv:
                zero = torch.zeros_like(eps)
                sch = torch.where(on[iw], d[iw], zero)
                w2 = wt * wt
                ssx = torch.where(on[iw], w2 * eps / wx[iw] ** 2,
                                  torch.where(delw * delw > TO1, -w2 * eps / (4.0 * w2 * (delw + 0.5)) * delw, zero))
                ach[iw, :nv] += 0.5 * (w[:nv] * (aqsn[:nv] @ sch.T)).sum(1)
                asx[iw] += (w[:nv] * (aqsn[:nv] @ ssx.T)).sum()
        # the driver's 512-wide blocks: a masked term re-adds the value left at its block offset
        e = torch.zeros(3, rows, nc, dtype=torch.float64, device="cuda")
        val = torch.zeros(rows, 512, dtype=torch.float64, device="cuda")
        src = torch.zeros(rows, 512, dtype=torch.long, device="cuda")
        for b in range(0, nc, 512):
            n = min(512, nc - b)
            at = torch.arange(b, b + n, device="cuda").expand(rows, n)
            for iw in range(3):
                m = on[iw][:, b:b + n]
                val[:, :n] = torch.where(m, d[iw][:, b:b + n], val[:, :n])
                src[:, :n] = torch.where(m, at, src[:, :n])
                e[iw].scatter_add_(1, src[:, :n], val[:, :n])
        for iw in range(3):
            ach[iw, nv:] += 0.5 * (w[nv:] * (aqsn[nv:] @ e[iw].T)).sum(1)
    return {"achtemp": ach.sum(1), "asxtemp": asx, "acht_n1_loc": ach[2].clone()}


def _bracket(x, grid, none):
    """The last interval of the grid that x lies strictly inside; `none` (no interval, or the reference's
    default) maps to the last one."""
    inside = [k for k in range(len(grid) - 1) if grid[k] < x < grid[k + 1]]
    k = inside[-1] if inside else none
    return len(grid) - 2 if k == none else k


def _exact_ff(p, schdt):
    nb, nv, nf, ne = p["number_bands"], p["nvband"], p["nFreq"], p["nfreqeval"]
    aqsn, aqsm = p["aqsntemp"], p["aqsmtemp"]
    igp, vc = _columns(p)
    w = torch.conj(aqsm[:, igp])
    zeros = lambda *s: torch.zeros(s, dtype=torch.complex128, device="cuda")  # noqa: E731
    rw, rs, aw = zeros(nb, nf), zeros(nb, nf), zeros(nb, nf)
    for f in range(nf):
        t = w * (aqsn @ p["I_epsR_array"][f].T)
        rw[:, f], rs[:, f] = (t * vc).sum(1), t.sum(1)
        aw[:, f] = (w * (aqsn @ p["I_epsA_array"][f].T) * vc).sum(1)
    if not schdt:
        rs.zero_()
    rwh, awh, sch = rw.cpu().numpy(), aw.cpu().numpy(), rs.cpu().numpy()
    grid, ekq, brd = p["dFreqGrid"], p["ekq"], p["dFreqBrd"]
    asx = cor = 0j
    for n in range(nb):
        x = p["freqevalmin"] - ekq[n] + p["freqevalstep"]
        if n < nv:
            k = _bracket(abs(x), grid, 0)
            d = grid[k + 1] - grid[k]
            asx += p["occ"] * ((grid[k + 1] - abs(x)) / d * rwh[n, k] + (abs(x) - grid[k]) / d * rwh[n, k + 1])
        if (x > 0) == (n < nv):
            continue
        if x > 0:
            inside = [k for k in range(nf - 1) if grid[k] < x < grid[k + 1]]
            k, s = (inside[-1] if inside else 0), -0.5
        else:
            x, s = -x, -0.5
            k = _bracket(x, grid, 0)
        d = grid[k + 1] - grid[k]
        cor += s * ((grid[k + 1] - x) / d * (rwh[n, k] - awh[n, k])
                    + (x - grid[k]) / d * (rwh[n, k + 1] - awh[n, k + 1]))
    wxe = p["freqevalmin"] - ekq[None, :] + (np.arange(ne)[:, None] - 1) * p["freqevalstep"]
    achd = np.zeros(ne, np.complex128)
    for f in range(nf):
        achd -= ((1j * p["pref"][f] * sch[:, f])[None, :] / (wxe - (grid[f] - brd[f].real) + 1j * brd[f].imag)).sum(1)
    # the last (band, frequency) term of the zero-broadening sum, with the reference's integer freqeval arguments
    ew = int(p["freqevalmin"]) - ekq[-1] + (np.arange(ne) - 1.0) * int(p["freqevalstep"])
    fact = -np.log(np.clip((ew - grid[-1]) / (ew - grid[-2]), 1e-4, 1e4))
    a2 = -nb * 1j * p["pref_zb"] * 0.5 * (sch[-1, -1] + sch[-1, -2]) * fact
    return {"achsDtemp": np.array([-0.5 * rwh[:, 1].sum()]), "asxDtemp": np.full(ne, asx), "achDtemp": achd,
            "achDtemp_cor": np.full(ne, cor), "ach2Dtemp": a2, "schDt_matrix": sch}


def exact(case, seed):
    c = case
    if work(c)["flops"] > 4e12:
        return None
    if c["kind"] == "serve":
        pools, got = _serve_inputs(c, seed), []
        for nb, nc, ng in _stream(c):
            got.append(_exact_gpp(dict(pools[nc], number_bands=nb, nvband=c["nv"], ncouls=nc, ngpown=ng)))
        return {"achtemp": torch.stack([g["achtemp"] for g in got]), "asxtemp": torch.stack([g["asxtemp"] for g in got]),
                "acht_n1_loc": torch.cat([g["acht_n1_loc"] for g in got])}
    p = _inputs(c, seed)
    if c["kind"] == "ff":
        return _exact_ff(p, c["schdt"])
    if c["kind"] == "real":
        return _exact_real(p)
    out = _exact_half(p) if c["half"] else _exact_gpp(p, c["achstemp"])
    if c["where"] == "host" and not c["achstemp"]:  # the library's own output dict has the static remainder too, as 0
        out["achstemp"] = np.zeros(1, np.complex128)
    return out
