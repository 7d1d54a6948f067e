"""The calls this library is timed on: ε-self-joins through its public entry points.

A case is one call that a program makes: points, reference points and ε go in,
the pair list (or the CSR neighbour table) comes out.  The sizes, value
distributions and neighbour counts are those of the benchmark's workloads
(mistic/workloads.py) and of the tests, at full size, scaled down, or ragged:

  uniform   i.i.d. U[0,1)^d
  susy      heavy-tailed raw columns and nonlinear combinations of them,
            every column min-max scaled to [0,1]
  msd       correlated Gaussian with a decaying spectrum, standardised columns
  clusters  many Zipf-sized Gaussian clusters, L2-normalised rows
  mixture   1-50 anisotropic Gaussian clusters on a few dozen directions

Points are drawn on the GPU from the seed.  ε is calibrated on a sample of
them for a mean neighbour count and rounded to FP32, so that it does not
depend on the last bits of the calibration.

Pair lists are asked for sorted by (i, j), since their order is otherwise
that of the kernels' atomics.  All outputs are whole numbers (row ids and
offsets of the exact FP64 predicate), so there is no exact().
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "self-join-mistic_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mistic  # noqa: E402
from mistic import _lib as L  # noqa: E402


def listed():
    def case(name, gen, n, d, dtype, k, target, where, out, mode="auto"):
        return {"name": name, "gen": gen, "n": n, "d": d, "dtype": dtype, "k": k, "target": target,
                "where": where, "out": out, "mode": mode}
    return [
        # the smallest call anyone makes: a few thousand host rows in, pairs out
        # (the size of the library's own smoke run); latency and launches count
        case("first_call_4k", "uniform", 4_000, 18, "f64", 6, 32.0, "host", "pairs"),
        # a small planar point set with its neighbour table, ragged n
        case("planar_20k_table", "mixture", 20_011, 2, "f32", 2, 16.0, "host", "csr"),
        # the 100,000 x 18 uniform workload, rows already on the GPU
        case("uniform_100k", "uniform", 100_000, 18, "f64", 6, 32.0, "device", "pairs"),
        # the 5,000,000 x 18 workload, the largest ordinary low-dimensional set
        case("susy_5m", "susy", 5_000_000, 18, "f64", 6, 64.0, "device", "pairs"),
        # a ragged twentieth of it from a numpy array to a numpy array
        case("susy_250k_host", "susy", 250_007, 18, "f64", 6, 64.0, "host", "pairs"),
        # the 515,345 x 90 workload with its neighbour table
        case("msd_515k_table", "msd", 515_345, 90, "f64", 8, 16.0, "device", "csr"),
        # a fifth of the 5,000,000 x 384 workload: long FP32 rows, every pair a candidate
        case("clusters_1m_384", "clusters", 1_000_000, 384, "f32", 8, 16.0, "device", "pairs"),
        # a medium instance of the 2,000-instance batch on its own, d no multiple of anything
        case("mixture_200k_57", "mixture", 200_000, 57, "f32", 6, 16.0, "device", "csr"),
        # many points in the plane, odd n: the index and the CUDA-core filter carry it
        case("planar_2m", "mixture", 2_000_003, 2, "f32", 2, 16.0, "device", "pairs"),
        # uneven instances in one call: a share of the 2,000-instance batch
        {"name": "batch_48", "gen": "batch", "count": 48, "n_lo": 1_000, "n_hi": 200_000, "where": "device",
         "out": "pairs", "mode": "auto"},
        # the plain FP64 join, which a user takes as the yardstick
        case("fp64_30k", "uniform", 30_000, 18, "f64", 6, 32.0, "device", "pairs", mode="fp64"),
        # the entry point that allocates nothing
        {"name": "noalloc_30k", "gen": "mixture", "n": 30_000, "d": 32, "dtype": "f32", "k": 0, "target": 16.0,
         "where": "device", "out": "noalloc", "mode": "auto"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above."""
    fam = rng.choice(["uniform", "susy", "susy", "msd", "clusters", "mixture", "mixture", "batch", "fp64", "noalloc"])
    if fam == "batch":
        return {"gen": "batch", "count": rng.randint(4, 48), "n_lo": 1_000, "n_hi": _log_int(rng, 10_000, 200_000),
                "where": rng.choice(["host", "device"]), "out": "pairs", "mode": "auto"}
    c = {"gen": fam, "n": 0, "d": 0, "dtype": rng.choice(["f64", "f32"]), "k": 6,
         "target": rng.choice([4.0, 16.0, 64.0]), "where": rng.choice(["host", "device", "device"]),
         "out": rng.choice(["pairs", "pairs", "csr"]), "mode": "auto"}
    if fam == "uniform":
        c.update(n=_log_int(rng, 1_000, 200_000), d=rng.randint(6, 40))
    elif fam == "susy":
        c.update(n=_log_int(rng, 5_000, 4_000_000), d=18)
        if rng.random() < 0.2:
            c["mode"] = "fp32"
    elif fam == "msd":
        c.update(n=_log_int(rng, 5_000, 500_000), d=rng.randint(33, 126), k=8)
        if c["n"] < 100_000 and rng.random() < 0.2:
            c["mode"] = "tf32"
    elif fam == "clusters":
        c.update(n=_log_int(rng, 10_000, 900_000), d=rng.randint(127, 400), k=8)
    elif fam == "mixture":
        d = rng.choice([2, 3, 8, 18, 32, 57, 90])
        c.update(n=_log_int(rng, 1_000, 2_000_000 if d <= 3 else 300_000), d=d, k=min(6, d))
    elif fam == "fp64":
        c.update(gen=rng.choice(["uniform", "mixture"]), n=_log_int(rng, 1_000, 50_000), d=rng.randint(6, 40), mode="fp64")
    else:
        d = rng.randint(2, 64)
        c.update(gen="mixture", n=_log_int(rng, 1_000, 50_000), d=d, k=0, where="device", out="noalloc", target=16.0)
    return c


# ------------------------------------------------------------------ points


def _randn(shape, g):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)


def _uniform(n, d, g):
    return torch.rand((n, d), generator=g, device="cuda", dtype=torch.float64)


def _susy(n, d, g):
    raw_n = 8
    raw = torch.exp(0.8 * torch.randn((n, raw_n), generator=g, device="cuda", dtype=torch.float64))
    x = torch.empty((n, d), device="cuda", dtype=torch.float64)
    x[:, :raw_n] = raw
    spec = np.random.default_rng(1002)  # which columns combine is part of the workload, not of the seed
    for t in range(d - raw_n):
        a, b, c = (int(v) for v in spec.choice(raw_n, size=3, replace=False))
        if t % 3 == 0:
            v = raw[:, a] * raw[:, b]
        elif t % 3 == 1:
            v = raw[:, a] / (raw[:, b] + 0.5)
        else:
            v = torch.sqrt(raw[:, a] ** 2 + raw[:, b] ** 2 + raw[:, c] ** 2)
        x[:, raw_n + t] = v + 0.05 * torch.randn((n,), generator=g, device="cuda", dtype=torch.float64)
    lo, hi = x.min(dim=0).values, x.max(dim=0).values
    return (x - lo) / (hi - lo)


def _msd(n, d, g):
    q, _ = torch.linalg.qr(torch.randn((d, d), generator=g, device="cuda", dtype=torch.float64))
    scale = torch.arange(1, d + 1, device="cuda", dtype=torch.float64) ** -0.6
    x = (torch.randn((n, d), generator=g, device="cuda", dtype=torch.float64) * scale) @ q.T
    return (x - x.mean(dim=0)) / x.std(dim=0)


def _mix(n, d, n_clusters, rotations, rank, noise, eig_lo, weights, g):
    """Gaussian clusters of the given weights: eigenvalues log-uniform in
    [eig_lo, 1] on `rank` directions of one of `rotations` random rotations."""
    w = torch.as_tensor(weights, device="cuda", dtype=torch.float64)
    lab = torch.searchsorted(torch.cumsum(w / w.sum(), 0), torch.rand((n,), generator=g, device="cuda",
                                                                     dtype=torch.float64))
    lab = lab.clamp_(max=n_clusters - 1)
    centres = _randn((n_clusters, d), g) * 0.5
    u = torch.rand((n_clusters, rank), generator=g, device="cuda")
    sd = torch.exp(0.5 * math.log(eig_lo) * u)
    basis, _ = torch.linalg.qr(_randn((rotations, d, rank), g))
    x = torch.empty((n, d), device="cuda", dtype=torch.float32)
    for r in range(rotations):
        rows = torch.nonzero(lab % rotations == r).flatten()
        if rows.numel():
            z = _randn((rows.numel(), rank), g) * sd[lab[rows]]
            x[rows] = centres[lab[rows]] + z @ basis[r].T
    if noise > 0:
        x += noise * _randn((n, d), g)
    return x


def _clusters(n, d, g):
    zipf = 1.0 / np.arange(1, 1001, dtype=np.float64) ** 1.1
    x = _mix(n, d, 1000, 8, d, 0.0, 1e-3, zipf, g)
    x /= x.double().norm(dim=1, keepdim=True).float()
    return x


def _mixture(n, d, g):
    nc = 1 + (n + d) % 50  # of the case: the work does not change with the seed
    return _mix(n, d, nc, min(nc, 6), min(d, 32), 0.1, 1e-2, np.random.default_rng(n).random(nc) + 0.1, g)


def _points(gen, n, d, dtype, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    make = {"uniform": _uniform, "susy": _susy, "msd": _msd, "clusters": _clusters, "mixture": _mixture}[gen]
    x = make(n, d, g)
    return x.to(torch.float64 if dtype == "f64" else torch.float32).contiguous()


def _eps(x, target, seed):
    """ε for about `target` neighbours a point: the matching quantile of the
    squared distances within a sample of the rows."""
    n = x.shape[0]
    m = min(n, 8192 if n > 100_000 else 4096)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    idx = torch.randperm(n, generator=g, device="cuda")[:m] if n > m else torch.arange(n, device="cuda")
    s = x[idx].double()
    nrm = (s * s).sum(dim=1)
    d2 = nrm[:, None] + nrm[None, :] - 2.0 * (s @ s.T)
    d2.fill_diagonal_(math.inf)  # d2 holds every pair of the sample twice
    kth = max(2, min(int(round(target * m * (m - 1) / max(1, n - 1))), m * (m - 1)))
    v = float(torch.sort(d2.flatten()).values[kth - 1].clamp_min(0.0))
    return float(np.float32(math.sqrt(v)))


# ------------------------------------------------------------------ calls

_HANDLE = None


def _handle():
    """One library handle for the whole program, as a service keeps it."""
    global _HANDLE
    if _HANDLE is None:
        _HANDLE = mistic.Handle(0)
    return _HANDLE


class _Device:
    """A device array of the library's, for torch.as_tensor."""

    def __init__(self, ptr, count, typestr):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _array(ptr, count, typestr, where):
    """A library result of `count` numbers as a tensor (device) or numpy array (host), not copied."""
    ptr = ctypes.cast(ptr, ctypes.c_void_p).value
    if where == "device":
        return torch.as_tensor(_Device(ptr, count, typestr), device="cuda")
    size = int(typestr[2])
    return np.frombuffer((ctypes.c_char * (count * size)).from_address(ptr), dtype=typestr)


def _buffer(count, dtype, where):
    """The caller's own room for a result, -1 beyond its end."""
    if where == "device":
        return torch.full((count,), -1, dtype=getattr(torch, dtype), device="cuda")
    return np.full((count,), -1, dtype=dtype)


class _State:
    """What a program holds before the call: the inputs, ε, the options and its pair buffer."""


def prepare(case, seed):
    s = _State()
    s.case = case
    where, out = case["where"], case["out"]
    if case["gen"] == "batch":
        rng = np.random.default_rng(1000 * seed + 7)
        s.inst, s.keep, total = (L.Instance * case["count"])(), [], 0.0
        for i, (n, d, target) in enumerate(_batch_sizes(case)):
            x = _points("mixture", n, d, "f32", int(rng.integers(1 << 30)))
            p = s.inst[i]
            p.n, p.d, p.dtype, p.k, p.eps = n, d, L.F32, min(6, d), _eps(x, target, i)
            x = x if where == "device" else x.cpu().numpy()
            p.pts = _ptr(x)
            s.keep.append(x)
            total += n * target
        s.cap = int(1.5 * total) + 65_536
        s.opts = _handle().opts(mode=case["mode"], input_on_device=where == "device", pairs=where, sort_pairs=True)
        s.buf = _buffer(s.cap, "int64", where)
        return s
    x = _points(case["gen"], case["n"], case["d"], case["dtype"], seed)
    s.eps = _eps(x, case["target"], seed)
    s.x = x if where == "device" else x.cpu().numpy()
    # room for three times the neighbours expected
    edges = int(3.0 * case["target"] * case["n"]) + 131_072
    if out == "csr":
        s.cap, s.off, s.buf = edges, _buffer(case["n"] + 1, "int64", where), _buffer(edges, "int32", where)
        kw = {"csr": where}
    else:
        s.cap, s.buf = edges // 2, _buffer(edges // 2, "int64", where)
        kw = {"pairs": where, "sort_pairs": True}
        if where == "device":
            kw.update(pair_capacity=s.cap, pair_buffer=s.buf.data_ptr())
    s.opts = _handle().opts(mode=case["mode"], input_on_device=where == "device", **kw)
    return s


def _ptr(x):
    return x.data_ptr() if isinstance(x, torch.Tensor) else x.ctypes.data


def run(s):
    """One call; its pair count and the caller's buffers with the result in front."""
    c, h = s.case, _handle()
    where = c["where"]
    if c["gen"] == "batch":
        return _run_batch(s, h)
    dt = L.F64 if c["dtype"] == "f64" else L.F32
    if c["out"] == "noalloc":
        cnt = ctypes.c_uint64(0)
        st = h.lib.mistic_selfjoin_noalloc(s.x.data_ptr(), c["n"], c["d"], dt, s.eps, s.buf.data_ptr(), s.cap,
                                           ctypes.byref(cnt), None)
        if st != L.OK:
            raise mistic.MisticError(st, h.lib.mistic_strerror(st).decode())
        return cnt.value, torch.sort(s.buf).values  # this entry point has no order of its own
    r = h.selfjoin_raw(_ptr(s.x), c["n"], c["d"], dt, c["k"], s.eps, s.opts)
    if c["out"] == "csr":
        # the program's own copy of the table, then the library's goes back
        e = int(r.pairs_ordered_incl_self)
        s.off[:] = _array(r.csr_offsets, c["n"] + 1, "<i8", where)
        s.buf[:e] = _array(r.csr_nbrs, e, "<i4", where)
        _free(h, [r], where)
        return int(r.pairs_ij), s.off, s.buf
    if where == "host":
        if r.pairs_len:
            s.buf[:r.pairs_len] = _array(r.pairs, int(r.pairs_len), "<i8", where)
        _free(h, [r], where)
    return int(r.pairs_ij), s.buf


def _free(h, results, where):
    if where == "device":
        torch.cuda.current_stream().synchronize()  # the copies out of the results are done
    for r in results:
        h.lib.mistic_result_free(ctypes.byref(r))


def _run_batch(s, h):
    m, where = s.case["count"], s.case["where"]
    res = (L.Result * m)()
    st = h.lib.mistic_batch_selfjoin(h.h, s.inst, m, ctypes.byref(s.opts), res)
    if st != L.OK:
        raise mistic.MisticError(st, h.lib.mistic_last_error(h.h).decode())
    counts, at = [int(r.pairs_len) for r in res], 0
    for r, cnt in zip(res, counts):
        if cnt:
            s.buf[at:at + cnt] = _array(r.pairs, cnt, "<i8", where)
        at += cnt
    _free(h, res, where)
    return np.array(counts, dtype=np.int64), s.buf


def _batch_sizes(case):
    """(n, d, neighbours) of a batch's instances: the mix belongs to the case, the points to the seed."""
    rng = np.random.default_rng(7)
    for _ in range(case["count"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        yield n, int(rng.choice([2, 8, 18, 32, 57, 90])), float(rng.choice([4.0, 16.0, 64.0]))


# ------------------------------------------------------------------ work


def _work(n, d, esz, target, out, all_pairs):
    pairs = 0.5 * n * target
    outb = 8.0 * pairs if out != "csr" else 8.0 * (n + 1) + 4.0 * (2.0 * pairs + n)
    # distances: subtract, multiply, add for each of d coordinates, of every
    # pair where nothing prunes, of the result's own pairs where the index may
    evals = 0.5 * n * (n - 1) if all_pairs else pairs
    return {"bytes": float(n * d * esz + outb), "flops": float(3.0 * d * evals)}


def work(case):
    if case["gen"] == "batch":
        ws = [_work(n, d, 4, target, "pairs", False) for n, d, target in _batch_sizes(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    return _work(case["n"], case["d"], 8 if case["dtype"] == "f64" else 4, case["target"], case["out"],
                 case["out"] == "noalloc" or case["gen"] == "clusters")
