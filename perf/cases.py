"""Cases of the framework's performance measurement: FP64 products through the
public entry points, over the sizes, pair sets, error bounds and operand forms
that a program calls them with.

A case is a dict of plain values.  `kind` is the entry point:
  "device"   Handle.dgemm_device on device arrays (ozgb_dgemm_device),
  "ex"       Handle.dgemm_ex: op(A), op(B), alpha and beta (ozgb_dgemm_ex),
  "noalloc"  ozgb_dgemm_device_noalloc, the entry point without device allocation,
  "host"     Handle.setup + Handle.dgemm on plain numpy arrays (the drop-in call),
  "grouped"  Handle.dgemm_grouped, many independent products of any sizes.
The other fields are described at `listed`.

Inputs are (U - 0.5) exp(phi N), U uniform and N normal, the family of the test
suite and of bench.py, drawn on the device from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import ozaie_gb300 as oz
from ozaie_gb300 import Criterion, Mode, Profile

TAIL = 1e-4  # the elementwise criterion's tail, its default


def listed():
    return [
        # the smallest call a program makes, on device arrays: latency and launches
        case("tiny_fast", "device", 64, 64, 64),
        # odd sizes, no multiple of any tile, the accurate mode (full pair set)
        case("ragged_accurate", "device", 200, 136, 300, mode="accurate"),
        # the entry point for callers with a memory pool of their own, ragged
        case("noalloc_ragged", "noalloc", 777, 513, 640, slices=9),
        # the drop-in call on host arrays, a middle size of the reference's range
        case("host_512_accurate", "host", 512, 512, 512, mode="accurate"),
        # the drop-in call at the largest size of the reference's range
        case("host_2048_fast", "host", 2048, 2048, 2048),
        # an ordinary device product in the accurate mode
        case("square_1024_accurate", "device", 1024, 1024, 1024, mode="accurate"),
        # a BLAS-style update with transposes, padded leading dimensions and beta
        case("update_ragged", "ex", 1500, 777, 1333, transa=True, transb=True, alpha=-1.0, beta=1.0, pad=3),
        # the reference's own slice table and rounding (narrow slices)
        case("reference_profile_1024", "device", 1024, 1024, 1024, mode="accurate", profile="reference"),
        # the headline: slices chosen from the data for a normwise 1e-15
        case("adaptive_4096", "device", 4096, 4096, 4096, bound=1e-15),
        # the same knob held to the elementwise criterion, rectangular
        case("elementwise_3000", "device", 3000, 1000, 2000, bound=1e-13, criterion="elementwise"),
        # the batched workload: sizes log-uniform in [32, 2048], a bound on each
        case("grouped_512", "grouped", 32, 2048, 0, count=512, bound=1e-15),
        # a long inner dimension in the accurate mode
        case("long_k", "device", 4096, 4096, 32768, mode="accurate"),
    ]


def case(name, kind, M, N, K, mode="fast", profile="gb300", slices=0, bound=0.0, criterion="normwise", phi=1.0,
         transa=False, transb=False, alpha=1.0, beta=0.0, pad=0, count=0, graph=False):
    """M, N, K: the product's sizes; for "grouped" M and N are the smallest and
    the largest size of its `count` products.  mode: fast (triangular pair set) or
    accurate (full).  profile: the library's defaults or the reference's tables.
    slices: 0 for the profile's.  bound: requested relative error of the precision
    knob (0: none), under `criterion`.  phi: the spread of the inputs' exponents.
    pad: extra elements in each leading dimension.  graph: grouped calls replayed
    as CUDA graphs."""
    return {"name": name, "kind": kind, "M": M, "N": N, "K": K, "mode": mode, "profile": profile, "slices": slices,
            "bound": bound, "criterion": criterion, "phi": phi, "transa": transa, "transb": transb, "alpha": alpha,
            "beta": beta, "pad": pad, "count": count, "graph": graph}


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, odd ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["device", "device", "device", "device", "ex", "noalloc", "host", "grouped"])
    phi = rng.choice([0.5, 1.0, 2.0, 4.0])
    if kind == "grouped":
        lo = size(16, 128)
        c = case("", kind, lo, size(256, 2048), 0, count=size(8, 256), bound=rng.choice([0.0, 1e-8, 1e-11, 1e-15]), phi=phi,
                 graph=rng.random() < 0.3)
    elif kind == "noalloc":
        c = case("", kind, size(32, 1024), size(32, 1024), size(32, 1024), slices=rng.choice([3, 5, 7, 8, 9, 11]),
                 phi=phi)
    elif kind == "host":
        c = case("", kind, size(96, 2048), size(96, 2048), size(96, 2048), mode=rng.choice(["fast", "accurate"]),
                 phi=phi)
    elif kind == "ex":
        c = case("", kind, size(64, 3000), size(64, 3000), size(64, 3000), mode=rng.choice(["fast", "accurate"]),
                 phi=phi, transa=rng.random() < 0.5, transb=rng.random() < 0.5, alpha=rng.choice([-1.0, 1.0, 0.75]),
                 beta=rng.choice([0.0, 1.0]), pad=rng.choice([0, 1, 2, 8]))
    else:
        form = rng.choice(["fixed", "fixed", "reference", "normwise", "normwise", "elementwise"])
        if form == "reference":  # the sizes the reference takes
            c = case("", kind, size(128, 2048), size(128, 2048), size(128, 2048), profile="reference",
                     mode=rng.choice(["fast", "accurate"]), phi=phi)
        elif form == "fixed":
            c = case("", kind, size(48, 4096), size(48, 4096), size(48, 8192), mode=rng.choice(["fast", "accurate"]),
                     slices=rng.choice([0, 0, 4, 6, 9]), phi=phi)
        else:
            c = case("", kind, size(128, 4096), size(128, 4096), size(128, 8192), criterion=form,
                     bound=rng.choice([1e-8, 1e-11, 1e-13, 1e-15]), phi=phi)
    del c["name"]
    return c


def _draw_matrix(rows, cols, phi, gen, pad=0):
    """rows x cols values in a buffer with leading dimension cols + pad."""
    x = torch.empty((rows, cols + pad), dtype=torch.float64, device="cuda")
    x.normal_(0.0, phi, generator=gen).exp_()
    return x.mul_(torch.rand(x.shape, dtype=torch.float64, device="cuda", generator=gen).sub_(0.5))


def _sizes(c, seed):
    """The (M, N, K) of each product of a grouped case: every seed has the same
    sizes (the seed moves the values), log-uniform in [M, N]."""
    g = np.random.default_rng(7 + 1000 * c["count"])
    u = g.uniform(math.log(c["M"]), math.log(c["N"]), size=(c["count"], 3))
    return [tuple(int(v) for v in r) for r in np.rint(np.exp(u))]


def _inputs(c, seed):
    """Lists of the operands as stored, one entry per product; the outputs of a
    grouped case are views of one pool (also returned), 256-byte aligned."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    sizes = _sizes(c, seed) if c["kind"] == "grouped" else [(c["M"], c["N"], c["K"])]
    A, B, C, pool = [], [], [], None
    if c["kind"] == "grouped":
        at = np.cumsum([0] + [-(-M * N // 32) * 32 for M, N, _ in sizes])
        pool = torch.zeros(int(at[-1]), dtype=torch.float64, device="cuda")
        C = [pool[o:o + M * N].view(M, N) for o, (M, N, _) in zip(at, sizes)]
    for M, N, K in sizes:
        a, b = ((K, M) if c["transa"] else (M, K)), ((N, K) if c["transb"] else (K, N))
        A.append(_draw_matrix(a[0], a[1], c["phi"], gen, c["pad"]))
        B.append(_draw_matrix(b[0], b[1], c["phi"], gen, c["pad"]))
        if c["kind"] != "grouped":
            C.append(_draw_matrix(M, N, c["phi"], gen, c["pad"]) if c["beta"]
                     else torch.zeros((M, N + c["pad"]), dtype=torch.float64, device="cuda"))
    return sizes, A, B, C, pool


def _must(rc, h=None):
    if rc:
        raise RuntimeError("status %d: %s" % (rc, h.last_error() if h else ""))


def prepare(c, seed):
    sizes, A, B, C, pool = _inputs(c, seed)
    st = {"case": c, "A": A, "B": B, "C": C, "pool": pool, "stream": torch.cuda.current_stream().cuda_stream}
    if c["kind"] == "noalloc":
        st["lib"] = oz.load()
        return st
    h = oz.Handle()
    st["h"] = h
    if c["profile"] == "reference":
        h.set_profile(Profile.reference)
    if c["slices"]:
        h.set_slices(c["slices"])
    if c["bound"]:
        h.set_error_bound(c["bound"])
        h.set_error_criterion(Criterion[c["criterion"]], TAIL)
    if c["graph"]:
        h.set_graph(True)
    if c["kind"] == "grouped":
        st["probs"] = [{"M": M, "N": N, "K": K, "A": a.data_ptr(), "lda": K, "B": b.data_ptr(), "ldb": N,
                        "C": x.data_ptr(), "ldc": N, "error_bound": c["bound"]}
                       for (M, N, K), a, b, x in zip(sizes, A, B, C)]
    else:
        M, N, K = sizes[0]
        _must(h.setup(M, N, K, Mode[c["mode"]]), h)
    if c["kind"] == "host":
        st["A"], st["B"] = A[0].cpu().numpy(), B[0].cpu().numpy()
        st["C"] = np.empty((c["M"], c["N"]))
    return st


def run(st):
    c = st["case"]
    M, N, K, pad = c["M"], c["N"], c["K"], c["pad"]
    if c["kind"] == "host":
        _must(st["h"].dgemm(M, N, K, st["A"], st["B"], st["C"]), st["h"])
        return st["C"]
    if c["kind"] == "grouped":
        rc, _ = st["h"].dgemm_grouped(st["probs"], st["stream"])
        _must(rc, st["h"])
        return st["pool"]
    A, B, C = st["A"][0], st["B"][0], st["C"][0]
    if c["kind"] == "noalloc":
        _must(st["lib"].ozgb_dgemm_device_noalloc(M, N, K, ctypes.c_void_p(A.data_ptr()), K,
                                                  ctypes.c_void_p(B.data_ptr()), N, ctypes.c_void_p(C.data_ptr()), N,
                                                  c["slices"], ctypes.c_void_p(st["stream"])))
        return C
    if c["kind"] == "ex":
        # the update's C is kept by the program, which updates a copy of it
        X = C.clone() if c["beta"] else C
        _must(st["h"].dgemm_ex(c["transa"], c["transb"], M, N, K, c["alpha"], A.data_ptr(), A.shape[1], B.data_ptr(),
                               B.shape[1], c["beta"], X.data_ptr(), N + pad, st["stream"]), st["h"])
        return X
    _must(st["h"].dgemm_device(M, N, K, A.data_ptr(), K, B.data_ptr(), N, C.data_ptr(), N, st["stream"]), st["h"])
    return C


def exact(c, seed):
    sizes, A, B, C, pool = _inputs(c, seed)
    for (M, N, K), a, b, x in zip(sizes, A, B, C):
        a = a[:, :M].T if c["transa"] else a[:, :K]
        b = b[:, :K].T if c["transb"] else b[:, :N]
        x[:, :N] = c["alpha"] * (a @ b) + c["beta"] * x[:, :N]
    if c["kind"] == "grouped":
        return pool
    return C[0].cpu().numpy() if c["kind"] == "host" else C[0]


def _slice_pairs(c, K):
    """Slice-pair products of one element and K step: s(s + 1)/2 for the triangular
    set, s^2 for the full one.  With a bound, the fewest slices of 7 bits whose
    truncation alone meets it (the knob picks by the data, at least these)."""
    if c["bound"]:
        s = math.ceil(-math.log2(c["bound"]) / 7)
        return s * (s + 1) // 2
    if c["profile"] == "reference" and c["mode"] == "accurate":
        s = c["slices"] or 25
        return s * (s + 1) // 2
    s = c["slices"] or 8
    return s * s if c["mode"] == "accurate" else s * (s + 1) // 2


def work(c):
    sizes = _sizes(c, 0) if c["kind"] == "grouped" else [(c["M"], c["N"], c["K"])]
    nbytes = flops = 0
    for M, N, K in sizes:
        nbytes += 8 * (M * K + K * N + M * N * (2 if c["beta"] else 1))
        flops += 2 * M * N * K * _slice_pairs(c, K)
    return {"bytes": nbytes, "flops": flops}
