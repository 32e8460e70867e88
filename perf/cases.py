"""Performance cases of the one-sided Jacobi SVD library.

Each case is one piece of work that a program hands to the library through its
public entry points (jacobi-svd-cuda_b200/jsvd.py on libjsvd.so): the plain
drop-in, the QR-preconditioned and the blocked mixed-precision solvers on
device buffers, the mixed solver on host buffers, a packed batch of small
matrices, and the serving core.  Sizes are those of the library's workloads
(a 512 x 512 Gaussian matrix, a 4096 x 1024 matrix of condition 1e6, a batch
of matrices of 16..256 rows stored as FP32, a serving mix) and ragged or
generic ones around them.

The solvers return singular values unsorted and singular vectors with
arbitrary signs.  A program that wants the usual convention sorts them, and so
do the passes here: sigma in decreasing order, and, where a path is held to a
tolerance instead of to the bits, U and V in that order with the signs that
make the largest entry of every column of V positive.  The paths that
reproduce the reference's bytes (plain, batch) also return their outputs as
they come.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "jacobi-svd-cuda_b200"))

import jsvd  # noqa: E402


def listed():
    return [
        # the smallest call of a program that solves one little system at a
        # time, the reference's default epsilon: latency and launches
        {"name": "plain_64x48", "kind": "plain", "m": 64, "n": 48, "eps": 1e-9},
        # an odd, tall matrix through the drop-in
        {"name": "plain_1000x333", "kind": "plain", "m": 1000, "n": 333, "eps": 1e-9},
        # the square Gaussian workload, to full accuracy
        {"name": "plain_512x512", "kind": "plain", "m": 512, "n": 512, "eps": 1e-14},
        # the QR-preconditioned scalar sweep on a tall matrix
        {"name": "precond_2048x512", "kind": "precond", "m": 2048, "n": 512, "kappa": 1e6},
        # the blocked mixed-precision solver: a narrow matrix (no tensor-core
        # phase), a ragged one, the tall workload, a large one
        {"name": "mixed_600x200", "kind": "mixed", "m": 600, "n": 200, "kappa": 1e3},
        {"name": "mixed_1777x611", "kind": "mixed", "m": 1777, "n": 611, "kappa": 1e4},
        {"name": "mixed_4096x1024", "kind": "mixed", "m": 4096, "n": 1024, "kappa": 1e6},
        {"name": "mixed_8192x4096", "kind": "mixed", "m": 8192, "n": 4096, "kappa": 1e4},
        # the mixed solver called on host arrays: copies in and out included
        {"name": "host_mixed_2048x1024", "kind": "host", "m": 2048, "n": 1024, "kappa": 1e5},
        # the batch workload (16..256 rows, FP32 storage, sigma and V) and a
        # batch of small FP64 members with U as well
        {"name": "batch_f32_2000", "kind": "batch", "count": 2000, "m_lo": 16, "m_hi": 256, "f32": True, "u": False},
        {"name": "batch_f64_small_3000", "kind": "batch", "count": 3000, "m_lo": 16, "m_hi": 64, "f32": False,
         "u": True},
        # a burst of serving requests, small ones and large ones mixed
        {"name": "serve_burst_24", "kind": "serve", "count": 24, "m_lo": 32, "m_hi": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "precond", "mixed", "mixed", "mixed", "host", "batch", "batch", "serve"])
    if kind == "plain":
        m = _log_int(rng, 24, 1500)
        n = max(8, min(640, int(m * rng.uniform(0.2, 1.0))))
        return {"kind": kind, "m": m, "n": n, "eps": rng.choice([1e-9, 1e-12, 1e-14])}
    if kind in ("precond", "mixed", "host"):
        n = _log_int(rng, 70, {"precond": 768, "mixed": 2048, "host": 1100}[kind])
        m = min(8192, int(n * rng.uniform(1.0, 4.0)))
        return {"kind": kind, "m": m, "n": n, "kappa": float("%.3g" % 10.0 ** rng.uniform(1.0, 6.0))}
    if kind == "batch":
        hi = _log_int(rng, 40, 256)
        return {"kind": kind, "count": _log_int(rng, 150, 2000), "m_lo": rng.randint(8, hi // 2), "m_hi": hi,
                "f32": rng.random() < 0.6, "u": rng.random() < 0.4}
    return {"kind": kind, "count": rng.randint(6, 24), "m_lo": rng.randint(16, 64), "m_hi": _log_int(rng, 128, 1024)}


# ---- inputs ------------------------------------------------------------------


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _sigma(n, kappa, g, device):
    """n singular values from 1 down to 1/kappa, log-equidistant with a
    quarter of the spacing of jitter (so that neighbours stay apart)."""
    if n == 1:
        return torch.ones(1, dtype=torch.float64, device=device)
    step = math.log(kappa) / (n - 1)
    i = torch.arange(n, dtype=torch.float64, device=device)
    jitter = (torch.rand(n, generator=g, dtype=torch.float64, device=device) - 0.5) * 0.5
    jitter[0] = 0.0
    return torch.exp(-step * (i + jitter))


def _haar(m, n, g, device):
    q, r = torch.linalg.qr(torch.randn((m, n), generator=g, dtype=torch.float64, device=device))
    return q * torch.sign(torch.diagonal(r))


def _spectrum(m, n, kappa, seed):
    """A = U diag(sigma) V^T with Haar U and V; returns (A, U, sigma, V)."""
    dev = torch.device("cuda")
    g = _generator(seed, dev)
    s = _sigma(n, kappa, g, dev)
    u, v = _haar(m, n, g, dev), _haar(n, n, g, dev)
    return (u * s) @ v.T, u, s, v


def _plain_input(case, seed):
    dev = torch.device("cuda")
    return torch.randn((case["m"], case["n"]), generator=_generator(seed, dev), dtype=torch.float64, device=dev)


def _shapes(case, seed):
    """Shapes and condition numbers of the members of a batch or burst.  The
    shapes belong to the case, the values to the seed."""
    r = np.random.default_rng(case["count"] * 1000 + case["m_hi"])
    lo, hi = case["m_lo"], case["m_hi"]
    if case["kind"] == "serve":
        ms = np.floor(np.exp(r.uniform(math.log(lo), math.log(hi), size=case["count"]))).astype(int)
        ns = np.maximum(1, np.floor(ms * r.uniform(0.25, 1.0, size=case["count"]))).astype(int)
    else:
        ms = r.integers(lo, hi + 1, size=case["count"])
        ns = np.array([r.integers(min(8, m), m + 1) for m in ms])
    kappas = 10.0 ** np.random.default_rng(seed).uniform(1.0, 6.0, size=case["count"])
    return ms, ns, kappas


def _orthonormal_batch(ms, ns, rows, g, device):
    """Orthonormal factors (ms[i] x ns[i], zero-padded to rows x rows) of a
    batch of Gaussian matrices by three passes of CholeskyQR."""
    q = torch.randn((len(ms), rows, rows), generator=g, dtype=torch.float64, device=device)
    k = torch.arange(rows, device=device)
    live = k[None, :] < torch.as_tensor(ns, device=device)[:, None]
    q *= (k[None, :] < torch.as_tensor(ms, device=device)[:, None])[:, :, None]
    q *= live[:, None, :]
    pad = torch.diag_embed((~live).to(torch.float64))
    for p in range(3):
        gram = q.transpose(1, 2) @ q + pad
        if p == 0:
            gram += torch.diag_embed(1e-10 * torch.diagonal(gram, dim1=1, dim2=2))
        low = torch.linalg.cholesky(gram)
        q = torch.linalg.solve_triangular(low.transpose(1, 2), q, upper=True, left=False)
        q = q * live[:, None, :]
    return q


def _batch_matrices(case, seed):
    """The members as host arrays (FP32 or FP64), made in chunks on the GPU."""
    dev = torch.device("cuda")
    g = _generator(seed, dev)
    ms, ns, kappas = _shapes(case, seed)
    out = []
    for c0 in range(0, case["count"], 500):
        m, n, kap = ms[c0:c0 + 500], ns[c0:c0 + 500], kappas[c0:c0 + 500]
        rows = int(m.max())
        u = _orthonormal_batch(m, n, rows, g, dev)
        v = _orthonormal_batch(n, n, rows, g, dev)
        nt = torch.as_tensor(n, device=dev)[:, None].to(torch.float64)
        i = torch.arange(rows, dtype=torch.float64, device=dev)[None, :]
        jitter = (torch.rand((len(m), rows), generator=g, dtype=torch.float64, device=dev) - 0.5) * 0.5
        s = torch.exp(-torch.as_tensor(np.log(kap), device=dev)[:, None] / (nt - 1).clamp(min=1.0) * (i + jitter))
        a = ((u * s[:, None, :]) @ v.transpose(1, 2)).to(torch.float32 if case.get("f32") else torch.float64)
        a = a.cpu().numpy()
        out += [np.ascontiguousarray(a[j, :m[j], :n[j]]) for j in range(len(m))]
    return out


# ---- the usual order and signs -------------------------------------------------


def _ordered(u, s, v):
    """sigma decreasing, U and V in its order, the largest entry of every
    column of V positive."""
    s, order = torch.sort(s, descending=True)
    v = v.index_select(1, order)
    sign = torch.sign(torch.gather(v, 0, v.abs().argmax(dim=0, keepdim=True)))
    return {"u": u.index_select(1, order) * sign, "sigma": s, "v": v * sign}


def _ordered_host(u, s, v):
    order = np.argsort(-s, kind="stable")
    v = v[:, order]
    sign = np.sign(v[np.abs(v).argmax(axis=0), np.arange(v.shape[1])])
    out = {"sigma": s[order], "v": v * sign}
    if u is not None:
        out["u"] = u[:, order] * sign
    return out


# ---- the cases -----------------------------------------------------------------

_DEVICE_ENTRY = {"plain": jsvd.plain_svd_device, "precond": jsvd.precond_svd_device, "mixed": jsvd.mixed_svd_device}


_SERVER = []


def _server():
    """The process's serving core, started once as a serving program does."""
    if not _SERVER:
        _SERVER.append(jsvd.Server(jsvd.default_config(epsilon=1e-12), budget_bytes=4 << 30, large_path=2))
    return _SERVER[0]


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    if kind in _DEVICE_ENTRY:
        m, n = case["m"], case["n"]
        a = _plain_input(case, seed) if kind == "plain" else _spectrum(m, n, case["kappa"], seed)[0]
        return {"kind": kind, "a": a.contiguous(), "m": m, "n": n,
                "cfg": jsvd.default_config(epsilon=case.get("eps", 1e-14)),
                "u": torch.empty((m, n), dtype=torch.float64, device=dev),
                "s": torch.empty(n, dtype=torch.float64, device=dev),
                "v": torch.empty((n, n), dtype=torch.float64, device=dev)}
    if kind == "host":
        a = _spectrum(case["m"], case["n"], case["kappa"], seed)[0].cpu().numpy()
        return {"kind": kind, "a": a, "cfg": jsvd.default_config(epsilon=1e-14)}
    if kind == "batch":
        mats = _batch_matrices(case, seed)
        batch = jsvd.DeviceBatch(mats, dev, f32=case["f32"], want_u=case["u"], want_v=True)
        member = torch.from_numpy(np.repeat(np.arange(batch.count), batch.cols)).to(dev)
        return {"kind": kind, "batch": batch, "member": member, "cfg": jsvd.default_config(epsilon=1e-12)}
    mats = []
    ms, ns, kappas = _shapes(case, seed)
    for i in range(case["count"]):
        mats.append(_spectrum(int(ms[i]), int(ns[i]), kappas[i], seed * 1009 + i)[0].cpu().numpy())
    return {"kind": kind, "mats": mats, "server": _server()}


def run(state):
    kind = state["kind"]
    if kind in _DEVICE_ENTRY:
        sweeps = _DEVICE_ENTRY[kind](state["a"].data_ptr(), state["m"], state["n"], state["u"].data_ptr(),
                                     state["s"].data_ptr(), state["v"].data_ptr(), state["cfg"])
        if kind == "plain":  # the reference's bytes, and the spectrum in the usual order
            return {"u": state["u"], "sigma": state["s"], "v": state["v"], "sweeps": sweeps,
                    "spectrum": torch.sort(state["s"], descending=True)[0]}
        return _ordered(state["u"], state["s"], state["v"])
    if kind == "host":
        r = jsvd.svd(state["a"], "mixed", state["cfg"])
        return _ordered_host(r.u, r.sigma, r.v)
    if kind == "batch":
        b = state["batch"]
        b.solve(state["cfg"])
        # every member's singular values in decreasing order, member by member
        s, order = torch.sort(b.sigma, descending=True)
        spectrum = s[torch.sort(state["member"][order], stable=True)[1]]
        return {"sigma": b.sigma, "v": b.v, "u": b.u, "sweeps": b.sweeps, "spectrum": spectrum}
    server = state["server"]
    tickets = [server.submit(a) for a in state["mats"]]
    return [_ordered_host(None, s, v) for _, s, v, _, _ in (server.wait(t) for t in tickets)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "plain":
        s = torch.linalg.svdvals(_plain_input(case, seed).cpu())
        return {"u": None, "sigma": None, "v": None, "sweeps": None, "spectrum": s}
    if kind in ("precond", "mixed", "host"):
        # the factors that the input was made from
        _, u, s, v = _spectrum(case["m"], case["n"], case["kappa"], seed)
        return _ordered(u, s, v)
    if kind == "batch":
        mats = _batch_matrices(case, seed)
        s = np.concatenate([np.linalg.svd(a.astype(np.float64), compute_uv=False) for a in mats])
        return {"sigma": None, "v": None, "u": None, "sweeps": None, "spectrum": s}
    out = []
    ms, ns, kappas = _shapes(case, seed)
    for i in range(case["count"]):
        _, u, s, v = _spectrum(int(ms[i]), int(ns[i]), kappas[i], seed * 1009 + i)
        o = _ordered(u, s, v)
        out.append({"sigma": o["sigma"], "v": o["v"]})
    return out


def _svd_flops(m, n):
    """Golub-Van Loan's count for an SVD with m x n U, sigma and V by R-bidiagonalisation."""
    return 6.0 * m * n * n + 20.0 * n ** 3


def work(case):
    """The input read once, the outputs written once, and the operations of a
    direct (bidiagonalising) SVD of the same shape."""
    kind = case["kind"]
    if "m" in case:
        m, n = case["m"], case["n"]
        return {"bytes": 8.0 * (2 * m * n + n * n + n), "flops": _svd_flops(m, n)}
    ms, ns, _ = _shapes(case, 0)
    elem = 4.0 if case.get("f32") else 8.0
    total = {"bytes": 0.0, "flops": 0.0}
    for m, n in zip(ms.astype(float), ns.astype(float)):
        total["bytes"] += elem * m * n + 8.0 * (n + n * n) + (8.0 * m * n if case.get("u") else 0.0)
        total["flops"] += _svd_flops(m, n)
    return total
