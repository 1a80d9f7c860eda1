"""The work that users of the library have it do, as cases that can be timed and compared.

Nine families, one for each public path, over the sizes of the library's own configurations and tests:

* ``dropin``: one update through HCORE_dgemm on host arrays, as a task runtime calls it tile by tile;
* ``update``: a batch of low-rank updates in a plan (FP64, or FP32 end to end), its execute called directly
  or replayed from a CUDA graph;
* ``dense``: HCORE_dsyrk and HCORE_dgemmcd updates of dense tiles in a plan;
* ``apply``: HCORE_dgemmbdcd, a low-rank tile times a dense one into a dense one;
* ``factor``: HCORE_dpotrf of diagonal tiles and HCORE_dtrsm of the V factors below them;
* ``compress``: dense tiles to U, V factors and back (encode and decode);
* ``zgemm``: complex updates;
* ``panel``: one whole panel step of a TLR Cholesky in one call;
* ``predictor``: the rank predictor's forward pass and gradient.

The factors of a truncated update are determined only up to the sign of each column, and where two singular
values are close up to a rotation of their columns: any rounding decides.  What a user relies on is the tile
U V^T, so the passes that truncate end with the decompression that their program makes to read the tile
(HCORE_duncompress, as in the reference's own testing programs) and return whole dense tiles beside the ranks.
"""
import ctypes as C
import math

import numpy as np
import torch

import hcore_gb300 as hc

# HCORE_ / CBLAS constants
NO_TRANS, TRANS, LOWER, NON_UNIT, LEFT = 111, 112, 122, 131, 141
DEV = "cuda"


def listed():
    return [
        # the single-update configuration: nb 512, ranks 32, host arrays in and out
        {"name": "dropin_512", "kind": "dropin", "M": 512, "a": 32, "b": 32, "c": 32, "acc": 1e-8},
        # a short list of far-field updates of small tiles, executed directly: latency and launches
        {"name": "update_small", "kind": "update", "prec": "f64", "n": 16, "M": 250, "lo": 4, "hi": 12, "acc": 1e-8,
         "graph": False},
        # Schur updates with the ranks of a 2D covariance panel (a + c from 13 to 70), nb 1024, graph replay
        {"name": "update_panel_2d", "kind": "update", "prec": "f64", "n": 384, "M": 1024, "lo": 6, "hi": 34,
         "acc": 1e-8, "graph": True},
        # the large ranks of a 3D kernel: a + c beyond what one SM's shared memory holds
        {"name": "update_large_rank", "kind": "update", "prec": "f64", "n": 24, "M": 1000, "lo": 40, "hi": 110,
         "acc": 1e-7, "graph": False},
        # HCORE_sgemm end to end at a loose accuracy
        {"name": "update_f32", "kind": "update", "prec": "f32", "n": 256, "M": 512, "lo": 5, "hi": 24, "acc": 1e-4,
         "graph": True},
        # diagonal tiles updated by many low-rank tiles, and dense-C GEMM updates, nb 1024
        {"name": "dense_panel", "kind": "dense", "tiles": 32, "M": 1024, "updates": 24, "lo": 8, "hi": 32},
        # low-rank times dense into dense tiles of odd sizes
        {"name": "apply_odd", "kind": "apply", "tiles": 12, "M": 777, "N": 650, "K": 900, "rank": 40},
        # diagonal tiles factored and the V factors of their panels solved
        {"name": "factor_panel", "kind": "factor", "tiles": 8, "M": 1024, "factors": 12, "lo": 8, "hi": 32},
        # one small tile alone
        {"name": "factor_one", "kind": "factor", "tiles": 1, "M": 300, "factors": 3, "lo": 5, "hi": 16},
        # off-diagonal tiles compressed at 1e-8 relative and decompressed
        {"name": "compress_tiles", "kind": "compress", "tiles": 48, "M": 1024, "lo": 8, "hi": 40, "acc": 1e-8},
        # complex updates of the nb 512 shape
        {"name": "zgemm_batch", "kind": "zgemm", "n": 48, "M": 512, "lo": 16, "hi": 32, "acc": 1e-8},
        # POTRF, TRSM, SYRK and the recompressed updates of one panel in one call
        {"name": "panel_step", "kind": "panel", "nt": 16, "M": 512, "lo": 6, "hi": 24, "acc": 1e-8},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def ranks(lo, hi):
        x, y = sorted((logint(lo, hi), logint(lo, hi)))
        return {"lo": x, "hi": y}

    kind = rng.choice(["dropin", "update", "update", "dense", "apply", "factor", "compress", "zgemm", "panel",
                       "predictor"])
    if kind == "dropin":
        return {"kind": kind, "M": logint(128, 1024), "a": logint(4, 48), "b": logint(4, 48), "c": logint(4, 48),
                "acc": 1e-8}
    if kind == "update":
        if rng.random() < 0.25:
            return {"kind": kind, "prec": "f32", "n": logint(8, 256), "M": logint(256, 1024), **ranks(5, 24),
                    "acc": 1e-4, "graph": rng.random() < 0.5}
        if rng.random() < 0.25:
            return {"kind": kind, "prec": "f64", "n": logint(4, 24), "M": logint(512, 1100), **ranks(30, 110),
                    "acc": rng.choice([1e-6, 1e-7]), "graph": rng.random() < 0.5}
        return {"kind": kind, "prec": "f64", "n": logint(8, 384), "M": logint(200, 1024), **ranks(4, 34),
                "acc": rng.choice([1e-8, 1e-6]), "graph": rng.random() < 0.5}
    if kind == "dense":
        return {"kind": kind, "tiles": logint(2, 32), "M": logint(256, 1024), "updates": logint(1, 24), **ranks(4, 64)}
    if kind == "apply":
        return {"kind": kind, "tiles": logint(1, 16), "M": logint(200, 1024), "N": logint(100, 1024),
                "K": logint(200, 1024), "rank": logint(4, 100)}
    if kind == "factor":
        return {"kind": kind, "tiles": logint(1, 12), "M": logint(200, 1024), "factors": logint(1, 12), **ranks(4, 40)}
    if kind == "compress":
        return {"kind": kind, "tiles": logint(4, 48), "M": logint(256, 1024), **ranks(6, 40),
                "acc": rng.choice([1e-8, 1e-6])}
    if kind == "zgemm":
        return {"kind": kind, "n": logint(4, 48), "M": logint(128, 512), **ranks(6, 32), "acc": 1e-8}
    if kind == "panel":
        return {"kind": kind, "nt": logint(4, 20), "M": logint(256, 640), **ranks(5, 28), "acc": 1e-8}
    return {"kind": "predictor", "n": logint(200, 20000)}


# ---- inputs -------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _orth(g, n, M, r, dtype=torch.float64):
    """n matrices with r orthonormal columns of length M, as (n, r, M): column j of tile t is x[t, j].
    (Cholesky QR of Gaussian columns, twice.)"""
    x = torch.randn(n, r, M, generator=g, device=DEV, dtype=dtype)
    for _ in range(2):
        low = torch.linalg.cholesky(x @ x.mT)
        x = torch.linalg.solve_triangular(low, x, upper=False)
    return x


def _factors(g, ranks, M, rmax, decades=8.0, scale=None, dtype=torch.float64):
    """U and V (n, rmax, M) of tiles U V^T with Haar factors and singular values scale * 10^(-decades i / r),
    folded into V as HCORE's compression does; columns from a tile's own rank on are zero."""
    n = len(ranks)
    r = torch.tensor(ranks, device=DEV, dtype=torch.float64)[:, None]
    i = torch.arange(rmax, device=DEV, dtype=torch.float64)[None, :]
    sig = torch.where(i < r, 10.0 ** (-decades * i / r), torch.zeros((), device=DEV, dtype=torch.float64))
    if scale is not None:
        sig = sig * scale[:, None]
    u, v = _orth(g, n, M, rmax, torch.float64), _orth(g, n, M, rmax, torch.float64)
    if dtype.is_complex:
        ui, vi = _orth(g, n, M, rmax), _orth(g, n, M, rmax)
        u, v = torch.complex(u, ui) / math.sqrt(2.0), torch.complex(v, vi) / math.sqrt(2.0)
    u = u * (i < r)[:, :, None]
    v = v * sig[:, :, None]
    return u.to(dtype).contiguous(), v.to(dtype).contiguous()


def _ranks(seed, n, lo, hi):
    return [int(x) for x in np.random.default_rng(seed).integers(lo, hi + 1, n)]


def _scales(g, n):
    """tiles of a covariance matrix lose up to four decades with the distance of their clusters"""
    return 10.0 ** (-4.0 * torch.rand(n, generator=g, device=DEV, dtype=torch.float64))


def _spd(g, n, M):
    """dense diagonal covariance tiles exp(-|x - y|^2 / 0.01) + I of points in the unit square"""
    p = torch.rand(n, M, 2, generator=g, device=DEV, dtype=torch.float64)
    d2 = ((p[:, :, None, :] - p[:, None, :, :]) ** 2).sum(-1)
    return (torch.exp(-d2 / 0.01) + torch.eye(M, device=DEV, dtype=torch.float64)).contiguous()


def _update_inputs(case, seed):
    n, M, dtype = case["n"], case["M"], {"f64": torch.float64, "f32": torch.float32}[case.get("prec", "f64")]
    if case["kind"] == "zgemm":
        dtype = torch.complex128
    g = _gen(seed)
    ra, rb, rc = (_ranks([seed, q], n, case["lo"], case["hi"]) for q in (1, 2, 3))
    dec = 8.0 if dtype != torch.float32 else 5.0
    f = {}
    for name, r in (("A", ra), ("B", rb), ("C", rc)):
        f[name + "U"], f[name + "V"] = _factors(g, r, M, case["hi"], dec, _scales(g, n), dtype)
    return f, ra, rb, rc


def _uncompress_tasks(u, v, out):
    """HCORE_duncompress tasks of tiles (n, cols, M); the rank of each is filled in before a call"""
    n, cols, M = u.shape
    e = u.element_size()
    return [hc.DenseTask(kind=2, M=M, a=0, Au=u.data_ptr() + t * cols * M * e, lda=M,
                         Bv=v.data_ptr() + t * v.shape[1] * M * e, ldb=M, CD=out.data_ptr() + t * M * M * e, ldcd=M)
            for t in range(n)]


def _uncompress(tasks, ranks):
    for t, r in zip(tasks, ranks):
        t.a = int(r)
    hc.dense_batched(tasks, torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def work(case):
    return globals()["_work_" + case["kind"]](case)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


# ---- exact values -------------------------------------------------------------


def _truncated(left, right, acc, start=1, dtype=torch.float64):
    """The tile left @ right.T (M x k factors) truncated by the reference's rule: rank = first i >= start with
    sigma_i < acc.  Returns (rank, dense tile transposed, i.e. as a column-major buffer)."""
    qa, ra = torch.linalg.qr(left)
    qb, rb = torch.linalg.qr(right)
    u, s, vh = torch.linalg.svd((ra @ rb.mT).cpu())
    r = len(s)
    for i in range(start, len(s)):
        if float(s[i]) < acc:
            r = i
            break
    u = (u[:, :r] * s[:r]).to(left.device)
    return r, (qb @ vh[:r].mT.to(left.device)) @ (qa @ u).mT


def _exact_updates(f, ra, rb, rc, acc, alpha=-1.0, beta=1.0):
    ranks, tiles = [], []
    for t in range(len(ra)):
        w = torch.complex128 if f["AU"].dtype.is_complex else torch.float64
        au, av, bu, bv, cu, cv = (f[k][t].mT[:, :r[t]].to(w) for k, r in (
            ("AU", ra), ("AV", ra), ("BU", rb), ("BV", rb), ("CU", rc), ("CV", rc)))
        left = torch.cat([beta * cu, alpha * au], 1)
        right = torch.cat([cv, bu @ (av.mT @ bv).mT], 1)
        r, p = _truncated(left, right, acc)
        ranks.append(r)
        tiles.append(p)
    return np.array(ranks, dtype=np.int32), torch.stack(tiles)


# ---- dropin -------------------------------------------------------------------


def _dropin_inputs(case, seed):
    g = _gen(seed)
    f = {}
    for name, r in (("A", case["a"]), ("B", case["b"]), ("C", case["c"])):
        f[name + "U"], f[name + "V"] = _factors(g, [r], case["M"], r)
    return f


def _prepare_dropin(case, seed):
    f = {k: np.asfortranarray(v[0].cpu().numpy().T) for k, v in _dropin_inputs(case, seed).items()}
    return {"run": _run_dropin, "f": f, "case": case, "lib": hc.lib()}


def _run_dropin(s):
    c, f = s["case"], s["f"]
    M = c["M"]
    r, cu, cv, _ = hc.hcore_dgemm(M, -1.0, f["AU"], f["AV"], c["a"], f["BU"], f["BV"], c["b"], 1.0, f["CU"], f["CV"],
                                  c["c"], maxrk=c["a"] + c["c"], acc=c["acc"])
    tile = np.empty((M, M), order="F")
    rank = np.array([float(r)])
    dp = C.POINTER(C.c_double)
    p = lambda x: x.ctypes.data_as(dp)  # noqa: E731
    s["lib"].HCORE_duncompress(NO_TRANS, TRANS, M, M, 1.0, p(cu), p(rank), M, p(cv), p(rank), M, 0.0, p(tile), M)
    return {"rank": r, "tile": tile.T}


def _work_dropin(case):
    M, a, b, c = case["M"], case["a"], case["b"], case["c"]
    return {"bytes": 8.0 * M * (2 * (a + b + c) + M), "flops": _update_flops(M, a, b, c) + 2.0 * M * M * (a + c) / 2}


def _exact_dropin(case, seed):
    f = _dropin_inputs(case, seed)
    r, tiles = _exact_updates(f, [case["a"]], [case["b"]], [case["c"]], case["acc"])
    return {"rank": int(r[0]), "tile": tiles[0]}


# ---- update -------------------------------------------------------------------


def _update_flops(M, a, b, c):
    """two QRs of M x k, the SVD of their k x k core, the factor products and the rebuild of k/2 columns"""
    k = a + c
    return 4.0 * a * b * M + 4.0 * M * k * k + 22.0 * k ** 3 + 4.0 * M * k * k


def _prepare_update(case, seed):
    f, ra, rb, rc = _update_inputs(case, seed)
    n, M, dtype = case["n"], case["M"], f["AU"].dtype
    cap = 2 * case["hi"]
    cuo, cvo = (torch.zeros(n, cap, M, device=DEV, dtype=dtype) for _ in range(2))
    e = cuo.element_size()
    at = lambda x, t: x.data_ptr() + t * x.shape[1] * M * e  # noqa: E731
    tasks = [hc.LrTask(M=M, a=ra[t], b=rb[t], c=rc[t], rk=0, maxrk=cap, ld_newv=0, storage_maxrank=0, alpha=-1.0,
                       beta=1.0, acc=case["acc"], AU=at(f["AU"], t), AV=at(f["AV"], t), lda=M, BU=at(f["BU"], t),
                       BV=at(f["BV"], t), ldb=M, Bdense=None, CU=at(f["CU"], t), CV=at(f["CV"], t), ldc=M,
                       CUo=at(cuo, t), CVo=at(cvo, t), ldco=M) for t in range(n)]
    batch = hc.Batch(tasks, precision=hc.F64 if dtype == torch.float64 else hc.F32)
    s = {"run": _run_update, "f": f, "cuo": cuo, "cvo": cvo, "batch": batch, "graph": None}
    if dtype == torch.float64:
        s["tiles"] = torch.empty(n, M, M, device=DEV, dtype=dtype)
        s["tasks"] = _uncompress_tasks(cuo, cvo, s["tiles"])
    if case["graph"]:
        torch.cuda.synchronize()
        g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.stream(side):
            with torch.cuda.graph(g, stream=side):
                batch.execute(side.cuda_stream)
        torch.cuda.synchronize()
        s["graph"] = g
    return s


def _run_update(s):
    stream = torch.cuda.current_stream().cuda_stream
    if s["graph"] is not None:
        s["graph"].replay()
    else:
        s["batch"].execute(stream)
    ranks, status = s["batch"].results(stream)
    if "tiles" in s:
        _uncompress(s["tasks"], ranks)
        tiles = s["tiles"]
    else:  # FP32 tiles: the library decompresses FP64 only
        tiles = s["cvo"].mT @ s["cuo"]
    return {"ranks": ranks, "status": status, "tiles": tiles}


def _work_update(case):
    n, M, r = case["n"], case["M"], (case["lo"] + case["hi"]) / 2
    e = 8.0 if case["prec"] == "f64" else 4.0
    return {"bytes": n * e * M * (6 * r + M), "flops": n * (_update_flops(M, r, r, r) + 2.0 * M * M * r)}


def _exact_update(case, seed):
    k = 2 * case["hi"]
    if case["n"] * (case["M"] * k * k * 1e-9 + k ** 3 * 2e-9 + 4e-3) > 15:
        return None
    f, ra, rb, rc = _update_inputs(case, seed)
    ranks, tiles = _exact_updates(f, ra, rb, rc, case["acc"])
    return {"ranks": ranks, "status": np.zeros(case["n"], dtype=np.int32), "tiles": tiles}


# ---- dense --------------------------------------------------------------------


def _dense_inputs(case, seed):
    """every other tile takes dsyrk updates of its low-rank tiles, the others dgemmcd updates"""
    g = _gen(seed)
    n, M = case["updates"], case["M"]
    f = {}
    ra, rb = _ranks([seed, 1], n, case["lo"], case["hi"]), _ranks([seed, 2], n, case["lo"], case["hi"])
    f["AU"], f["AV"] = _factors(g, ra, M, case["hi"], 8.0, _scales(g, n))
    f["BU"], f["BV"] = _factors(g, rb, M, case["hi"], 8.0, _scales(g, n))
    return f, ra, rb, _spd(g, case["tiles"], M)


def _prepare_dense(case, seed):
    f, ra, rb, cd0 = _dense_inputs(case, seed)
    M, cd = case["M"], torch.empty_like(cd0)
    at = lambda x, t: x.data_ptr() + t * x.shape[1] * M * 8  # noqa: E731
    tasks = []
    for t in range(case["tiles"]):
        for u in range(case["updates"]):
            task = hc.DenseTask(kind=t % 2, M=M, a=ra[u], b=rb[u], alpha=-1.0, Au=at(f["AU"], u), Av=at(f["AV"], u),
                                lda=M, CD=at(cd, t), ldcd=M)
            if t % 2:
                task.Bu, task.Bv, task.ldb = at(f["BU"], u), at(f["BV"], u), M
            tasks.append(task)
    return {"run": _run_dense, "f": f, "cd0": cd0, "cd": cd, "plan": hc.DensePlan(tasks)}


def _run_dense(s):
    s["cd"].copy_(s["cd0"])
    s["plan"].execute(torch.cuda.current_stream().cuda_stream)
    return s["cd"]


def _work_dense(case):
    r, M, t, u = (case["lo"] + case["hi"]) / 2, case["M"], case["tiles"], case["updates"]
    return {"bytes": 8.0 * (4 * u * M * r + 2 * t * M * M), "flops": t * u * (1.5 * M * M * r + 4.0 * M * r * r)}


def _exact_dense(case, seed):
    f, ra, rb, cd = _dense_inputs(case, seed)
    syrk, gemm = torch.zeros_like(cd[0]), torch.zeros_like(cd[0])
    for u in range(case["updates"]):
        au, av, bu, bv = (f[k][u] for k in ("AU", "AV", "BU", "BV"))  # (r, M), column-major
        syrk += au.mT @ (av @ av.mT) @ au
        gemm += bu.mT @ (bv @ av.mT) @ au      # (Au (Av^T Bv) Bu^T)^T
    out = cd.clone()
    out[0::2] = torch.triu(out[0::2] - syrk)   # buffers are column-major: the lower triangle is kept
    out[1::2] -= gemm
    return out


# ---- apply --------------------------------------------------------------------


def _apply_inputs(case, seed):
    g, n, ld = _gen(seed), case["tiles"], max(case["M"], case["K"])
    au, av = _factors(g, [case["rank"]] * n, ld, case["rank"])
    bd = torch.randn(n, case["N"], case["K"], generator=g, device=DEV, dtype=torch.float64)
    cd = torch.randn(n, case["N"], case["M"], generator=g, device=DEV, dtype=torch.float64)
    return au, av, bd, cd


def _prepare_apply(case, seed):
    au, av, bd, cd0 = _apply_inputs(case, seed)
    M, N, K, r = case["M"], case["N"], case["K"], case["rank"]
    ld, cd = max(M, K), torch.empty_like(cd0)
    tasks = [hc.DenseTask(kind=3, M=M, N=N, kdim=K, a=r, alpha=-1.0, beta=1.0, Au=au.data_ptr() + t * r * ld * 8,
                          Av=av.data_ptr() + t * r * ld * 8, lda=ld, Bd=bd.data_ptr() + t * N * K * 8, ldb=K,
                          CD=cd.data_ptr() + t * N * M * 8, ldcd=M) for t in range(case["tiles"])]
    return {"run": _run_apply, "in": (au, av, bd), "cd0": cd0, "cd": cd, "tasks": tasks}


def _run_apply(s):
    s["cd"].copy_(s["cd0"])
    hc.dense_batched(s["tasks"], torch.cuda.current_stream().cuda_stream)
    return s["cd"]


def _work_apply(case):
    M, N, K, r, t = case["M"], case["N"], case["K"], case["rank"], case["tiles"]
    return {"bytes": 8.0 * t * (M * r + K * r + K * N + 2 * M * N), "flops": 2.0 * t * N * r * (K + M)}


def _exact_apply(case, seed):
    au, av, bd, cd = _apply_inputs(case, seed)
    return cd - (bd @ av[:, :, :case["K"]].mT) @ au[:, :, :case["M"]]


# ---- factor -------------------------------------------------------------------


def _factor_inputs(case, seed):
    g, n = _gen(seed), case["tiles"] * case["factors"]
    ranks = _ranks([seed, 1], n, case["lo"], case["hi"])
    _, v = _factors(g, ranks, case["M"], case["hi"], 8.0, _scales(g, n))
    return _spd(g, case["tiles"], case["M"]), v, ranks


def _prepare_factor(case, seed):
    d0, v0, ranks = _factor_inputs(case, seed)
    M, d, v = case["M"], torch.empty_like(d0), torch.empty_like(v0)
    at = lambda x, t: x.data_ptr() + t * x.shape[1] * M * 8  # noqa: E731
    potrf = [hc.PotrfTask(uplo=ord("L"), n=M, A=at(d, t), lda=M) for t in range(case["tiles"])]
    trsm = [hc.TrsmTask(side=LEFT, uplo=LOWER, trans=NO_TRANS, diag=NON_UNIT, M=M, N=r, alpha=1.0,
                        A=at(d, q // case["factors"]), lda=M, B=at(v, q), ldb=M) for q, r in enumerate(ranks)]
    return {"run": _run_factor, "d0": d0, "v0": v0, "d": d, "v": v, "potrf": potrf, "trsm": trsm}


def _run_factor(s):
    stream = torch.cuda.current_stream().cuda_stream
    s["d"].copy_(s["d0"])
    s["v"].copy_(s["v0"])
    info = hc.potrf_batched(s["potrf"], stream)
    hc.trsm_batched(s["trsm"], stream)
    return {"info": info, "tiles": s["d"], "factors": s["v"]}


def _work_factor(case):
    M, t = case["M"], case["tiles"]
    cols = case["factors"] * (case["lo"] + case["hi"]) / 2
    return {"bytes": 16.0 * t * (M * M + M * cols), "flops": t * (M ** 3 / 3.0 + 1.0 * M * M * cols)}


def _exact_factor(case, seed):
    d, v, _ = _factor_inputs(case, seed)
    low = torch.linalg.cholesky(d)
    tiles = torch.triu(low.mT) + torch.tril(d, -1)   # column-major buffers; the upper triangle is not touched
    per = v.view(case["tiles"], -1, case["M"])       # columns as rows
    return {"info": np.zeros(case["tiles"], dtype=np.int32), "tiles": tiles,
            "factors": torch.linalg.solve_triangular(low, per.mT, upper=False).mT.reshape(v.shape)}


# ---- compress -----------------------------------------------------------------


def _compress_inputs(case, seed):
    """tiles whose singular values fall geometrically to the rounding level, `rank` of them above acc"""
    g, n = _gen(seed), case["tiles"]
    ranks = _ranks([seed, 1], n, case["lo"], case["hi"])
    digits = -math.log10(case["acc"])
    # an odd count of columns: no singular value falls on the threshold itself
    count = lambda r: int(math.ceil(r * 16.0 / digits)) | 1  # noqa: E731
    u, v = _factors(g, [count(r) for r in ranks], case["M"], count(case["hi"]), 16.0, _scales(g, n))
    return u, v, (v.mT @ u).contiguous()             # column-major D = U V^T


def _prepare_compress(case, seed):
    _, _, d = _compress_inputs(case, seed)
    n, M, cap = case["tiles"], case["M"], 128
    u, v = (torch.zeros(n, cap, M, device=DEV, dtype=torch.float64) for _ in range(2))
    out = torch.empty_like(d)
    tasks = [hc.CompressTask(M=M, D=d.data_ptr() + t * M * M * 8, ldd=M, acc=case["acc"], relative=1, maxrank=cap,
                             U=u.data_ptr() + t * cap * M * 8, V=v.data_ptr() + t * cap * M * 8, ldo=M)
             for t in range(n)]
    return {"run": _run_compress, "d": d, "u": u, "v": v, "out": out, "tasks": tasks, "un": _uncompress_tasks(u, v, out)}


def _run_compress(s):
    ranks, status = hc.compress_batched(s["tasks"], torch.cuda.current_stream().cuda_stream)
    _uncompress(s["un"], ranks)
    return {"ranks": ranks, "status": status, "tiles": s["out"]}


def _work_compress(case):
    M, n, r = case["M"], case["tiles"], (case["lo"] + case["hi"]) / 2
    return {"bytes": 16.0 * n * M * M + 32.0 * n * M * r, "flops": n * (4.0 * M * M * r + 2.0 * M * M * r)}


def _exact_compress(case, seed):
    u, v, _ = _compress_inputs(case, seed)
    sig = torch.linalg.vector_norm(v, dim=2)
    keep = sig >= case["acc"] * sig.max(1, keepdim=True).values
    return {"ranks": keep.sum(1).to(torch.int32).cpu().numpy(), "status": np.zeros(case["tiles"], dtype=np.int32),
            "tiles": (v * keep[:, :, None]).mT @ u}


# ---- zgemm --------------------------------------------------------------------


def _prepare_zgemm(case, seed):
    f, ra, rb, rc = _update_inputs(case, seed)
    n, M, cap = case["n"], case["M"], 2 * case["hi"]
    z = lambda: torch.zeros(n, cap, M, device=DEV, dtype=torch.complex128)  # noqa: E731
    cu, cv = z(), z()
    at = lambda x, t: x.data_ptr() + t * x.shape[1] * M * 16  # noqa: E731
    tasks = [hc.ZlrTask(M=M, a=ra[t], b=rb[t], c=rc[t], rk=0, maxrk=cap, alpha=hc.DComplex(-1.0, 0.0),
                        beta=hc.DComplex(1.0, 0.0), acc=case["acc"], AU=at(f["AU"], t), AV=at(f["AV"], t), lda=M,
                        BU=at(f["BU"], t), BV=at(f["BV"], t), ldb=M, CU=at(cu, t), CV=at(cv, t), ldc=M)
             for t in range(n)]
    return {"run": _run_zgemm, "f": f, "cu": cu, "cv": cv, "tasks": tasks, "hi": case["hi"]}


def _run_zgemm(s):
    s["cu"][:, :s["hi"]].copy_(s["f"]["CU"])   # updated in place
    s["cv"][:, :s["hi"]].copy_(s["f"]["CV"])
    ranks, status = hc.zgemm_batched(s["tasks"], torch.cuda.current_stream().cuda_stream)
    r = int(ranks.max())
    keep = torch.arange(r, device=DEV)[None, :] < torch.from_numpy(ranks).to(DEV)[:, None]
    return {"ranks": ranks, "status": status, "tiles": (s["cv"][:, :r] * keep[:, :, None]).mT @ s["cu"][:, :r]}


def _work_zgemm(case):
    n, M, r = case["n"], case["M"], (case["lo"] + case["hi"]) / 2
    return {"bytes": n * 16.0 * M * (6 * r + M), "flops": 4.0 * n * (_update_flops(M, r, r, r) + 2.0 * M * M * r)}


def _exact_zgemm(case, seed):
    f, ra, rb, rc = _update_inputs(case, seed)
    ranks, tiles = _exact_updates(f, ra, rb, rc, case["acc"])
    return {"ranks": ranks, "status": np.zeros(case["n"], dtype=np.int32), "tiles": tiles}


# ---- panel --------------------------------------------------------------------


def _panel_inputs(case, seed):
    g, nt = _gen(seed), case["nt"]
    pairs = [(i, j) for j in range(nt) for i in range(j + 1, nt)]
    ranks = _ranks([seed, 1], len(pairs), case["lo"], case["hi"])
    cap = 2 * case["hi"]
    u, v = (torch.zeros(len(pairs), cap, case["M"], device=DEV, dtype=torch.float64) for _ in range(2))
    u[:, :case["hi"]], v[:, :case["hi"]] = _factors(g, ranks, case["M"], case["hi"], 8.0, _scales(g, len(pairs)))
    return pairs, ranks, u, v, _spd(g, nt, case["M"])


def _prepare_panel(case, seed):
    pairs, ranks, u0, v0, d0 = _panel_inputs(case, seed)
    nt, nb, cap = case["nt"], case["M"], u0.shape[1]
    u, v, d = (torch.empty_like(x) for x in (u0, v0, d0))
    rank0 = np.zeros(nt * nt, dtype=np.int32)
    dp, up, vp = (C.c_void_p * nt)(), (C.c_void_p * (nt * nt))(), (C.c_void_p * (nt * nt))()
    slot = []
    for t in range(nt):
        dp[t] = d.data_ptr() + t * nb * nb * 8
    for q, (i, j) in enumerate(pairs):
        slot.append(i + j * nt)
        up[slot[-1]] = u.data_ptr() + q * cap * nb * 8
        vp[slot[-1]] = v.data_ptr() + q * cap * nb * 8
        rank0[slot[-1]] = ranks[q]
    rank = rank0.copy()
    a = hc.TlrMatrix(nt=nt, nb=nb, D=C.addressof(dp), ldd=nb, U=C.addressof(up), V=C.addressof(vp),
                     rank=rank.ctypes.data, maxrank=cap)
    out = torch.empty(len(pairs), nb, nb, device=DEV, dtype=torch.float64)
    return {"run": _run_panel, "in": (u0, v0, d0), "buf": (u, v, d), "ptrs": (dp, up, vp), "rank0": rank0, "rank": rank,
            "slot": np.array(slot), "a": a, "cap": cap, "acc": case["acc"], "out": out,
            "un": _uncompress_tasks(u, v, out), "lib": hc.lib()}


def _run_panel(s):
    for x, y in zip(s["buf"], s["in"]):
        x.copy_(y)
    s["rank"][:] = s["rank0"]
    info, status = C.c_int(0), np.zeros_like(s["rank"])
    rc = s["lib"].hcore_gpu_tlr_panel_step(C.byref(s["a"]), 0, s["acc"], s["cap"], C.byref(info),
                                           status.ctypes.data_as(C.POINTER(C.c_int)),
                                           torch.cuda.current_stream().cuda_stream)
    ranks = s["rank"][s["slot"]]
    _uncompress(s["un"], ranks)
    return {"rc": rc, "info": info.value, "ranks": ranks, "status": status, "diagonal": s["buf"][2], "tiles": s["out"]}


def _work_panel(case):
    M, nt, r = case["M"], case["nt"], (case["lo"] + case["hi"]) / 2
    tiles, upd = nt * (nt - 1) / 2, (nt - 1) * (nt - 2) / 2
    return {"bytes": 8.0 * (2 * nt * M * M + tiles * (2 * M * r + M * M)),
            "flops": M ** 3 / 3.0 + (nt - 1) * (M * M * r + M * M * r) + upd * _update_flops(M, r, r, r) +
            tiles * 2.0 * M * M * r}


def _exact_panel(case, seed):
    pairs, ranks, u, v, d = _panel_inputs(case, seed)
    nt, M = case["nt"], case["M"]
    index = {p: q for q, p in enumerate(pairs)}
    low = torch.linalg.cholesky(d[0])
    diagonal = d.clone()
    diagonal[0] = torch.triu(low.mT) + torch.tril(d[0], -1)
    f = {(i, j): (u[q].mT[:, :ranks[q]], v[q].mT[:, :ranks[q]]) for (i, j), q in index.items()}
    for i in range(1, nt):
        f[i, 0] = (f[i, 0][0], torch.linalg.solve_triangular(low, f[i, 0][1], upper=False))
        ui, vi = f[i, 0]
        diagonal[i] = torch.triu(d[i] - ui @ (vi.mT @ vi) @ ui.mT)
    new, tiles = [], torch.empty(len(pairs), M, M, device=DEV, dtype=torch.float64)
    for q, (i, j) in enumerate(pairs):
        if j == 0:
            new.append(ranks[q])
            tiles[q] = f[i, 0][1] @ f[i, 0][0].mT
            continue
        (au, av), (bu, bv), (cu, cv) = f[i, 0], f[j, 0], f[i, j]
        r, tiles[q] = _truncated(torch.cat([cu, -au], 1), torch.cat([cv, bu @ (av.mT @ bv).mT], 1), case["acc"])
        new.append(r)
    return {"rc": 0, "info": 0, "ranks": np.array(new, dtype=np.int32), "status": np.zeros(nt * nt, dtype=np.int32),
            "diagonal": diagonal, "tiles": tiles}


# ---- predictor ----------------------------------------------------------------


def _predictor_inputs(case, seed):
    """features and log2(1 + rank) targets with the spread of a TLR panel's updates"""
    g, n = _gen(seed), case["n"]
    x = torch.randn(n, 6, generator=g, device=DEV, dtype=torch.float32)
    y = torch.log2(1.0 + 14.0 * torch.exp(0.5 * torch.randn(n, generator=g, device=DEV, dtype=torch.float32)))
    return x.contiguous(), y.contiguous()


def _prepare_predictor(case, seed):
    x, y = _predictor_inputs(case, seed)
    return {"run": _run_predictor, "x": x, "y": y, "net": hc.RankMLP(seed)}


def _run_predictor(s):
    stream = torch.cuda.current_stream().cuda_stream
    loss, grad = s["net"].gradient(s["x"], s["y"], stream)
    return {"loss": np.float32(loss), "gradient": grad, "ranks": s["net"].predict(s["x"], stream=stream)}


def _work_predictor(case):
    n, p = case["n"], hc.RankMLP.NPARAMS
    return {"bytes": 4.0 * (8 * n + 2 * p), "flops": 8.0 * n * p}


def _exact_predictor(case, seed):
    return None   # the network is defined with BF16 activations
