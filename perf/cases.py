"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values; `kind` names the entry point:

  dposv       CHAMELEON_dposv on LAPACK-layout device arrays (any leading dimension), default tile size
  dposv_tile  CHAMELEON_dposv_Tile on descriptors over the caller's arrays
  dpotrf_tile CHAMELEON_dpotrf_Tile on a tile-major descriptor, filled and read by Lap2Desc / Desc2Lap
  dpotrs      CHAMELEON_dpotrs_Tile with a factor kept from an earlier call
  mixed       CHAMELEON_B200_dposv_mixed_Tile on tile-major descriptors (low-precision factor, FP64 refinement)
  dsposv_host CHAMELEON_dsposv on pinned host arrays
  batch       CHAM_B200_dposv_batch / sposv_batch, systems of uneven orders
  inverse     CHAMELEON_dpotri / dtrtri on device arrays
  tile_step   one step of a task runtime on the tile kernels: CUDA_dpotrf, 2 x CUDA_dtrsm, 2 x CUDA_dsyrk, CUDA_dgemm
  serve       a wave of requests of mixed orders through the serving loop

Matrices have the values of CHAMELEON_dplgsy (entries uniform in [-0.5, 0.5], N added to the diagonal) and right-hand
sides those of CHAMELEON_dplrnt.  Column-major arrays are torch tensors of shape (columns, leading dimension).
"""
import ctypes
import math

import torch

import chameleon_b200 as cb

UPLO = {"lower": cb.ChamLower, "upper": cb.ChamUpper}
SERVE_BUDGET = 8e9   # device bytes of one server: several run side by side


def listed():
    return [
        # the smallest calls: one small system per call, where latency counts
        {"name": "dposv_203", "kind": "dposv", "n": 203, "nrhs": 3, "uplo": "upper", "pad": 5},
        # the plain FP64 configuration that the reference runs on CPUs
        {"name": "dposv_tile_2048", "kind": "dposv_tile", "n": 2048, "nb": 320, "nrhs": 1, "uplo": "lower"},
        # an ordinary solve of an odd order, odd leading dimension, LAPACK layout
        {"name": "dposv_5003", "kind": "dposv", "n": 5003, "nrhs": 17, "uplo": "upper", "pad": 4},
        # factorization alone, in the reference's own tile layout
        {"name": "dpotrf_tile_8192", "kind": "dpotrf_tile", "n": 8192, "nb": 512, "uplo": "lower"},
        # new right-hand sides for a factor at hand
        {"name": "dpotrs_8192", "kind": "dpotrs", "n": 8192, "nb": 512, "nrhs": 64, "uplo": "lower"},
        # the benchmark's headline solve, the largest
        {"name": "mixed_32768", "kind": "mixed", "n": 32768, "nb": 512, "nrhs": 64, "uplo": "lower", "prec": 2},
        # a mixed solve end to end from host memory, odd order
        {"name": "dsposv_host_6007", "kind": "dsposv_host", "n": 6007, "nrhs": 9, "uplo": "upper"},
        # the benchmark's uneven batch
        {"name": "batch_f64_8192", "kind": "batch", "count": 8192, "nmin": 16, "nmax": 512, "rmax": 8, "uplo": "lower",
         "fp32": False, "sizes": 2024},
        # a smaller FP32 batch
        {"name": "batch_f32_1500", "kind": "batch", "count": 1500, "nmin": 16, "nmax": 300, "rmax": 8, "uplo": "upper",
         "fp32": True, "sizes": 7},
        # the inverse of an SPD matrix from its factor
        {"name": "dpotri_2500", "kind": "inverse", "op": "potri", "n": 2500, "uplo": "lower"},
        # the tile kernels as a task runtime calls them
        {"name": "tile_step_512", "kind": "tile_step", "nb": 512},
        # the serving stream: a wave of requests, orders log-uniform, host inputs
        {"name": "serve_48", "kind": "serve", "count": 48, "nmin": 64, "nmax": 4096, "rmax": 32, "sizes": 77},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["dposv", "dposv", "dposv_tile", "dpotrf_tile", "dpotrs", "mixed", "mixed", "dsposv_host", "batch",
                       "batch", "inverse", "tile_step", "serve"])
    uplo = rng.choice(["lower", "upper"])
    nb = rng.choice([128, 200, 256, 320, 384, 512])
    if kind == "dposv":
        return {"kind": kind, "n": _log(rng, 16, 8000), "nrhs": _log(rng, 1, 64), "uplo": uplo, "pad": rng.randint(0, 9)}
    if kind == "dposv_tile":
        return {"kind": kind, "n": _log(rng, 200, 8192), "nb": nb, "nrhs": _log(rng, 1, 64), "uplo": uplo}
    if kind == "dpotrf_tile":
        return {"kind": kind, "n": _log(rng, 400, 10000), "nb": nb, "uplo": uplo}
    if kind == "dpotrs":
        return {"kind": kind, "n": _log(rng, 400, 10000), "nb": nb, "nrhs": _log(rng, 1, 128), "uplo": uplo}
    if kind == "mixed":
        return {"kind": kind, "n": _log(rng, 1000, 20000), "nb": rng.choice([256, 320, 384, 512, 512]),
                "nrhs": _log(rng, 1, 64), "uplo": uplo, "prec": rng.choice([2, 2, 2, 1])}
    if kind == "dsposv_host":
        return {"kind": kind, "n": _log(rng, 400, 8192), "nrhs": _log(rng, 1, 64), "uplo": uplo}
    if kind == "batch":
        nmax = _log(rng, 48, 512)
        return {"kind": kind, "count": _log(rng, 100, 8192), "nmin": rng.randint(1, 16), "nmax": nmax,
                "rmax": _log(rng, 1, 32), "uplo": uplo, "fp32": rng.random() < 0.4, "sizes": rng.randint(1, 1 << 20)}
    if kind == "inverse":
        return {"kind": kind, "op": rng.choice(["potri", "potri", "trtri"]), "n": _log(rng, 60, 4000), "uplo": uplo}
    if kind == "tile_step":
        return {"kind": kind, "nb": _log(rng, 48, 1024)}
    return {"kind": kind, "count": rng.randint(12, 64), "nmin": 64, "nmax": _log(rng, 600, 4096), "rmax": 32,
            "sizes": rng.randint(1, 1 << 20)}


# --- inputs -----------------------------------------------------------------------------------------------------------
def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _spd(n, ld, g):
    """A column-major n x n matrix (n, ld) whose either triangle is that of an SPD matrix."""
    a = torch.rand((n, ld), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    a[:, :n].diagonal().add_(float(n))
    return a


def _tri(n, upper, g):
    """A triangular factor with the entries' sizes of a dplgsy matrix's (zero in the triangle that is not referenced)."""
    a = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5).mul_(1.0 / math.sqrt(n))
    a.diagonal().copy_(math.sqrt(n) + torch.rand(n, dtype=torch.float64, device="cuda", generator=g))
    return a.tril() if upper else a.triu()


def _rhs(nrhs, n, g, pad=0):
    b = torch.zeros((nrhs, n + pad), dtype=torch.float64, device="cuda")
    b[:, :n] = torch.rand((nrhs, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    return b


def _sizes(case):
    """Orders and right-hand-side counts of a batch or a wave: part of the case, not of the seed."""
    g = _gen(case["sizes"], "cpu")
    c, lo, hi = case["count"], case["nmin"], case["nmax"]
    if case["kind"] == "serve":
        u = torch.rand(c, dtype=torch.float64, generator=g)
        n = torch.exp(math.log(lo) + u * (math.log(hi + 1) - math.log(lo))).floor().clamp(lo, hi).to(torch.int64)
    else:
        n = torch.randint(min(lo, hi), hi + 1, (c,), generator=g)
    k = torch.randint(1, case["rmax"] + 1, (c,), generator=g)
    return n, k


def _offsets(v):
    o = torch.zeros_like(v)
    o[1:] = torch.cumsum(v, 0)[:-1]
    return o


def _batch_inputs(case, seed):
    n, k = _sizes(case)
    a_off, b_off = _offsets(n * n), _offsets(n * k)
    g = _gen(seed)
    dt = torch.float32 if case["fp32"] else torch.float64
    a = torch.rand(int((n * n).sum()), dtype=dt, device="cuda", generator=g).sub_(0.5)
    b = torch.rand(int((n * k).sum()), dtype=dt, device="cuda", generator=g).sub_(0.5)
    rep = torch.repeat_interleave
    pos = torch.arange(int(n.sum()), dtype=torch.int64) - rep(_offsets(n), n)
    idx = rep(a_off, n) + pos * (rep(n, n) + 1)
    a[idx.cuda()] += rep(n, n).to(dt).cuda()
    return n, k, a_off, b_off, a, b


def _ptr(t, off=0):
    return ctypes.c_void_p(t.data_ptr() + off)


def _must(rc):
    if rc != 0:
        raise RuntimeError("status %d" % rc)


# --- prepare ----------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    cb.init()
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_dposv(case, seed):
    g = _gen(seed)
    n, ld = case["n"], case["n"] + case["pad"]
    a0, b0 = _spd(n, ld, g), _rhs(case["nrhs"], n, g, case["pad"])
    return {"run": _run_dposv, "case": case, "a0": a0, "b0": b0, "a": a0.clone(), "b": b0.clone()}


def _run_dposv(s):
    c = s["case"]
    s["a"].copy_(s["a0"])
    s["b"].copy_(s["b0"])
    ld = c["n"] + c["pad"]
    _must(cb.dposv(UPLO[c["uplo"]], c["n"], c["nrhs"], s["a"], ld, s["b"], ld))
    return [s["a"], s["b"]]


def _prepare_dposv_tile(case, seed):
    s = _prepare_dposv(dict(case, pad=0), seed)
    s["run"] = _run_dposv_tile
    s["da"] = cb.Desc.create(case["n"], case["n"], case["nb"], mat=s["a"])
    s["db"] = cb.Desc.create(case["n"], case["nrhs"], case["nb"], mat=s["b"])
    return s


def _run_dposv_tile(s):
    s["a"].copy_(s["a0"])
    s["b"].copy_(s["b0"])
    _must(cb.dposv_Tile(UPLO[s["case"]["uplo"]], s["da"], s["db"]))
    return [s["a"], s["b"]]


def _prepare_dpotrf_tile(case, seed):
    n = case["n"]
    a0 = _spd(n, n, _gen(seed))
    return {"run": _run_dpotrf_tile, "case": case, "a0": a0, "a": a0.clone(), "da": cb.Desc.create(n, n, case["nb"])}


def _run_dpotrf_tile(s):
    u, n, L = UPLO[s["case"]["uplo"]], s["case"]["n"], cb.lib()
    _must(L.CHAMELEON_Lap2Desc(u, _ptr(s["a0"]), n, s["da"].ptr))
    _must(cb.dpotrf_Tile(u, s["da"]))
    _must(L.CHAMELEON_Desc2Lap(u, s["da"].ptr, _ptr(s["a"]), n))
    return [s["a"]]


def _prepare_dpotrs(case, seed):
    g = _gen(seed)
    n = case["n"]
    a, b0 = _tri(n, case["uplo"] == "upper", g), _rhs(case["nrhs"], n, g)
    b = b0.clone()
    return {"run": _run_dpotrs, "case": case, "a": a, "b0": b0, "b": b, "da": cb.Desc.create(n, n, case["nb"], mat=a),
            "db": cb.Desc.create(n, case["nrhs"], case["nb"], mat=b)}


def _run_dpotrs(s):
    s["b"].copy_(s["b0"])
    _must(cb.dpotrs_Tile(UPLO[s["case"]["uplo"]], s["da"], s["db"]))
    return [s["b"]]


def _prepare_mixed(case, seed):
    g = _gen(seed)
    n, k, nb, L = case["n"], case["nrhs"], case["nb"], cb.lib()
    a, b = _spd(n, n, g), _rhs(k, n, g)
    s = {"run": _run_mixed, "case": case, "da": cb.Desc.create(n, n, nb), "db": cb.Desc.create(n, k, nb),
         "dx": cb.Desc.create(n, k, nb), "x": torch.zeros_like(b)}
    _must(L.CHAMELEON_Lap2Desc(cb.ChamUpperLower, _ptr(a), n, s["da"].ptr))
    _must(L.CHAMELEON_Lap2Desc(cb.ChamUpperLower, _ptr(b), n, s["db"].ptr))
    return s


def _run_mixed(s):
    c = s["case"]
    rc, info = cb.dposv_mixed_Tile(UPLO[c["uplo"]], c["prec"], s["da"], s["db"], s["dx"])
    _must(rc)
    _must(cb.lib().CHAMELEON_Desc2Lap(cb.ChamUpperLower, s["dx"].ptr, _ptr(s["x"]), c["n"]))
    return [s["x"]]


def _prepare_dsposv_host(case, seed):
    g = _gen(seed)
    n, k = case["n"], case["nrhs"]
    host = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (_spd(n, n, g), _rhs(k, n, g))]
    return {"run": _run_dsposv_host, "case": case, "a": host[0], "b": host[1],
            "x": torch.zeros((k, n), dtype=torch.float64, pin_memory=True)}


def _run_dsposv_host(s):
    c = s["case"]
    rc, it = cb.dsposv(UPLO[c["uplo"]], c["n"], c["nrhs"], s["a"], c["n"], s["b"], c["n"], s["x"], c["n"])
    _must(rc)
    return [s["x"]]


def _prepare_batch(case, seed):
    n, k, a_off, b_off, a0, b0 = _batch_inputs(case, seed)
    return {"run": _run_batch, "case": case, "a0": a0, "b0": b0, "a": a0.clone(), "b": b0.clone(),
            "n": n.to(torch.int32).cuda(), "k": k.to(torch.int32).cuda(), "ao": a_off.cuda(), "bo": b_off.cuda(),
            "info": torch.zeros(case["count"], dtype=torch.int32, device="cuda")}


def _run_batch(s):
    c, L = s["case"], cb.lib()
    s["a"].copy_(s["a0"])
    s["b"].copy_(s["b0"])
    f = L.CHAM_B200_sposv_batch if c["fp32"] else L.CHAM_B200_dposv_batch
    _must(f(UPLO[c["uplo"]], c["count"], _ptr(s["n"]), _ptr(s["k"]), _ptr(s["a"]), _ptr(s["ao"]), _ptr(s["b"]),
            _ptr(s["bo"]), _ptr(s["info"]), None))
    return [s["a"], s["b"], s["info"]]


def _prepare_inverse(case, seed):
    a0 = _tri(case["n"], case["uplo"] == "upper", _gen(seed))
    return {"run": _run_inverse, "case": case, "a0": a0, "a": a0.clone()}


def _run_inverse(s):
    c = s["case"]
    s["a"].copy_(s["a0"])
    if c["op"] == "potri":
        _must(cb.dpotri(UPLO[c["uplo"]], c["n"], s["a"], c["n"]))
    else:
        _must(cb.dtrtri(UPLO[c["uplo"]], cb.ChamNonUnit, c["n"], s["a"], c["n"]))
    return [s["a"]]


def _tile_inputs(case, seed):
    """Column 0 of a lower tile matrix (diagonal tile, two panel tiles) and the tiles that its step updates."""
    nb, g = case["nb"], _gen(seed)
    tiles = [_spd(nb, nb, g)] + [_rhs(nb, nb, g) for _ in range(2)]
    return tiles + [_spd(nb, nb, g), _rhs(nb, nb, g), _spd(nb, nb, g)]   # (1,1), (2,1), (2,2)


class _Handle:
    def __init__(self):
        self.h = ctypes.c_void_p()
        _must(cb.lib().CHAM_B200_Handle_Create(ctypes.byref(self.h), None))

    def __del__(self):
        try:
            cb.lib().CHAM_B200_Handle_Destroy(self.h)
        except Exception:
            pass


def _prepare_tile_step(case, seed):
    t0 = torch.stack(_tile_inputs(case, seed))
    return {"run": _run_tile_step, "case": case, "t0": t0, "t": t0.clone(), "h": _Handle(),
            "info": torch.zeros(1, dtype=torch.int32, device="cuda"), "one": ctypes.c_double(1.0),
            "neg": ctypes.c_double(-1.0)}


def _run_tile_step(s):
    nb, L, h, t = s["case"]["nb"], cb.lib(), s["h"].h, s["t"]
    t.copy_(s["t0"])
    p = [_ptr(t, 8 * nb * nb * i) for i in range(6)]
    one, neg = ctypes.byref(s["one"]), ctypes.byref(s["neg"])
    _must(L.CUDA_dpotrf(cb.ChamLower, nb, p[0], nb, None, 0, _ptr(s["info"]), h))
    for i in (1, 2):
        _must(L.CUDA_dtrsm(cb.ChamRight, cb.ChamLower, cb.ChamTrans, cb.ChamNonUnit, nb, nb, one, p[0], nb, p[i], nb, h))
    _must(L.CUDA_dsyrk(cb.ChamLower, cb.ChamNoTrans, nb, nb, neg, p[1], nb, one, p[3], nb, h))
    _must(L.CUDA_dgemm(cb.ChamNoTrans, cb.ChamTrans, nb, nb, nb, neg, p[2], nb, p[1], nb, one, p[4], nb, h))
    _must(L.CUDA_dsyrk(cb.ChamLower, cb.ChamNoTrans, nb, nb, neg, p[2], nb, one, p[5], nb, h))
    return [*t, s["info"]]


class _Server(cb.Server):
    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def _serve_inputs(case, seed):
    """One matrix whose leading blocks are the requests' matrices, and the right-hand sides."""
    g = _gen(seed)
    return _spd(case["nmax"], case["nmax"], g), _rhs(case["rmax"], case["nmax"], g)


def _prepare_serve(case, seed):
    a, b = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in _serve_inputs(case, seed)]
    n, k = _sizes(case)
    off = _offsets(n * k)
    x = torch.zeros(int((n * k).sum()), dtype=torch.float64, pin_memory=True)
    xs = [x[int(o):int(o) + int(m * r)].view(int(r), int(m)) for o, m, r in zip(off, n, k)]
    return {"run": _run_serve, "case": case, "a": a, "b": b, "x": x, "xs": xs, "nk": list(zip(n.tolist(), k.tolist())),
            "server": _Server(slots=4, hbm_budget_bytes=SERVE_BUDGET)}


def _run_serve(s):
    sv, ld = s["server"], s["case"]["nmax"]
    reqs = [sv.submit(s["a"], s["b"], x, N=n, nrhs=k, lda=ld, ldb=ld, ldx=n) for (n, k), x in zip(s["nk"], s["xs"])]
    sv.drain()
    for r in reqs:
        _must(r.status)
    return [s["x"]]


# --- work, tolerance, exact -------------------------------------------------------------------------------------------
def work(case):
    kind, n, k = case["kind"], case.get("n", 0), case.get("nrhs", 0)
    tri = n * (n + 1) // 2
    if kind in ("dposv", "dposv_tile"):
        return {"bytes": 8 * (2 * tri + 2 * n * k), "flops": n ** 3 / 3 + 2 * n * n * k}
    if kind == "dpotrf_tile":
        return {"bytes": 8 * 2 * tri, "flops": n ** 3 / 3}
    if kind == "dpotrs":
        return {"bytes": 8 * (tri + 2 * n * k), "flops": 2 * n * n * k}
    if kind in ("mixed", "dsposv_host"):
        return {"bytes": 8 * (tri + 2 * n * k), "flops": n ** 3 / 3 + 2 * n * n * k}
    if kind == "inverse":
        return {"bytes": 8 * 2 * tri, "flops": (2 if case["op"] == "potri" else 1) * n ** 3 / 3}
    if kind == "tile_step":
        nb = case["nb"]
        return {"bytes": 8 * (2 * 6 - 3) * nb * nb, "flops": (1 / 3 + 2 + 4) * nb ** 3}
    ns, ks = (v.double() for v in _sizes(case))
    flops = float((ns ** 3 / 3 + 2 * ns * ns * ks).sum())
    if kind == "batch":
        return {"bytes": (4 if case["fp32"] else 8) * float((ns * (ns + 1) + 2 * ns * ks).sum()), "flops": flops}
    return {"bytes": 8 * float((ns * (ns + 1) / 2 + 2 * ns * ks).sum()), "flops": flops}


def tolerance(case):
    # about four times the error against 64 bits that the path shows
    if case.get("fp32"):
        return {"rel": 2e-5}    # FP32 storage and sums, products of split 16-bit parts: 5e-6
    if case["kind"] in ("mixed", "dsposv_host", "serve"):
        return {"rel": 5e-14}   # refinement may stop at |r| <= eps sqrt(n) |A| |x|: up to 4e-14 at n = 32768
    return {"rel": 5e-15}       # FP64 sums: 1e-16 to 8e-16


def _factor(a, upper):
    """The Cholesky factor of the referenced triangle, as a (lower) matrix of torch's own layout."""
    s = a.tril() + a.tril(-1).T if upper else a.triu() + a.triu(1).T
    return torch.linalg.cholesky(s)


def _with_triangle(a, f, upper):
    """`a` with the referenced triangle of the column-major array replaced by the factor f (lower)."""
    return a.triu(1) + f if upper else a.tril(-1) + f.T


def _batched_exact(case, seed):
    n, k, a_off, b_off, a, b = _batch_inputs(case, seed)
    upper, dt = case["uplo"] == "upper", torch.float64
    a, b = a.to(dt), b.to(dt)
    order = torch.argsort(n).tolist()
    for at in range(0, len(order), 128):   # similar orders together, padded with the identity
        ids = order[at:at + 128]
        m, r = int(n[ids].max()), int(k[ids].max())
        s = torch.eye(m, dtype=dt, device="cuda").repeat(len(ids), 1, 1)
        y = torch.zeros((len(ids), m, r), dtype=dt, device="cuda")
        for q, i in enumerate(ids):
            ni, ki, ao, bo = int(n[i]), int(k[i]), int(a_off[i]), int(b_off[i])
            t = a[ao:ao + ni * ni].view(ni, ni)
            s[q, :ni, :ni] = t.tril() + t.tril(-1).T if upper else t.triu() + t.triu(1).T
            y[q, :ni, :ki] = b[bo:bo + ni * ki].view(ki, ni).T
        f = torch.linalg.cholesky(s)
        x = torch.cholesky_solve(y, f)
        for q, i in enumerate(ids):
            ni, ki, ao, bo = int(n[i]), int(k[i]), int(a_off[i]), int(b_off[i])
            t = a[ao:ao + ni * ni].view(ni, ni)
            t.copy_(_with_triangle(t, f[q, :ni, :ni], upper))
            b[bo:bo + ni * ki].view(ki, ni).copy_(x[q, :ni, :ki].T)
    return [a, b, None]


def exact(case, seed):
    kind, g, upper = case["kind"], _gen(seed), case.get("uplo") == "upper"
    if kind in ("dposv", "dposv_tile", "mixed", "dsposv_host"):
        n, ld = case["n"], case["n"] + case.get("pad", 0)
        a, b = _spd(n, ld, g), _rhs(case["nrhs"], n, g, ld - n)
        f = _factor(a[:, :n], upper)
        b[:, :n] = torch.cholesky_solve(b[:, :n].T, f).T
        if kind in ("mixed", "dsposv_host"):
            return [b]
        a[:, :n] = _with_triangle(a[:, :n], f, upper)
        return [a, b]
    if kind == "dpotrf_tile":
        a = _spd(case["n"], case["n"], g)
        return [_with_triangle(a, _factor(a, upper), upper)]
    if kind == "dpotrs":
        a, b = _tri(case["n"], upper, g), _rhs(case["nrhs"], case["n"], g)
        return [torch.cholesky_solve(b.T, a.tril() if upper else a.triu().T).T.contiguous()]
    if kind == "batch":
        return _batched_exact(case, seed)
    if kind == "inverse":
        n = case["n"]
        a = _tri(n, upper, g)
        eye = torch.eye(n, dtype=torch.float64, device="cuda")
        low = a.tril() if upper else a.triu().T   # the factor: L, or the transpose of U
        x = torch.linalg.solve_triangular(low, eye, upper=False)
        if case["op"] == "potri":
            x = x.T @ x
        return [_with_triangle(a, x.tril(), upper)]
    if kind == "tile_step":
        t = torch.stack(_tile_inputs(case, seed))
        f = _factor(t[0], False)
        t[0] = _with_triangle(t[0], f, False)
        for i in (1, 2):   # X L^T = P: tensors hold the transposes
            t[i] = torch.linalg.solve_triangular(f, t[i], upper=False)
        p, q = t[1].T, t[2].T
        for i, d in ((3, p @ p.T), (5, q @ q.T)):
            t[i] -= d.T.triu()
        t[4] -= (q @ p.T).T
        return [*t, None]
    a, b = _serve_inputs(case, seed)
    out = []
    for n, k in zip(*(v.tolist() for v in _sizes(case))):
        f = _factor(a[:n, :n], False)
        out.append(torch.cholesky_solve(b[:k, :n].T, f).T.reshape(-1))
    return [torch.cat(out)]
