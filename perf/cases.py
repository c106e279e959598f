"""The work a user of this library has it do, as cases that can be timed.

Every case is one pass through the public Python entry points, which hand device
(or page-locked host) pointers to the C-ABI. The matrices are of the two kinds
that the benchmark and the tests use: complex Gaussian entries, and
lowest-Landau-level (LLL) orbital matrices M_ik = z_i^k exp(-|z_i|^2/4) with
z ~ CN(0, n), which are ill-conditioned; the composite-fermion (CF) call builds
its matrices itself from one configuration and a batch of permutations.

The serving loop is not a case: its kernels stay resident for 0.2 s after the
last request, so a device-wide wait after a pass times that, not the request.
What it runs for a request is the batched mixed path at walker sizes, which the
smallest case stands for.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "lion-codes_gb300"))

import lufqhe  # noqa: E402

REF, FUSED, MIXED = lufqhe.MODE_PLAIN_FP64, lufqhe.MODE_PLAIN_FP64_FUSED, lufqhe.MODE_MIXED
PLAN_SIZES = (6, 8, 12, 16, 24, 32, 48)
# the CF columns' coefficients (k1, k2, r1, r2) and momenta (mu, nu)
CF_K, CF_MU, CF_NU = (1.0, 0.5, 0.5, 1.0), 0, 1


def listed():
    return [
        # one Monte Carlo walker's move: few matrices, latency and launches count
        {"name": "walker_lll16_k64", "kind": "batch", "ens": "lll", "n": 16, "pad": 0,
         "batch": 64, "mode": MIXED, "c64": False},
        # benchmark configuration 1: a small ensemble step
        {"name": "gauss8_4096", "kind": "batch", "ens": "gauss", "n": 8, "pad": 0,
         "batch": 4096, "mode": MIXED, "c64": False},
        # benchmark configuration 2: a full ensemble step, well-conditioned
        {"name": "gauss16_65536", "kind": "batch", "ens": "gauss", "n": 16, "pad": 0,
         "batch": 65536, "mode": MIXED, "c64": False},
        # benchmark configuration 3 (the default workload): the precision stress
        {"name": "lll24_32768", "kind": "batch", "ens": "lll", "n": 24, "pad": 0,
         "batch": 32768, "mode": MIXED, "c64": False},
        # the largest size of the FP32 path
        {"name": "lll32_8192", "kind": "batch", "ens": "lll", "n": 32, "pad": 0,
         "batch": 8192, "mode": MIXED, "c64": False},
        # an odd particle number and a ragged batch
        {"name": "lll19_20011", "kind": "batch", "ens": "lll", "n": 19, "pad": 0,
         "batch": 20011, "mode": MIXED, "c64": False},
        # the library's default mode: FP64 in the reference's arithmetic
        {"name": "plain_gauss16_65536", "kind": "batch", "ens": "gauss", "n": 16, "pad": 0,
         "batch": 65536, "mode": REF, "c64": False},
        # the largest size, FP64
        {"name": "fused_lll64_2048", "kind": "batch", "ens": "lll", "n": 64, "pad": 0,
         "batch": 2048, "mode": FUSED, "c64": False},
        # the reference-shaped call on its own complex64 buffers, with pair
        # products: as many matrices as the reference's fixture file holds,
        # copied into the call's buffer first as its Monte Carlo loop does
        {"name": "refcall16_1000", "kind": "refcall", "n": 16, "batch": 1000, "pair": True,
         "c64": True},
        # matrices and results in page-locked host memory, end to end
        {"name": "host_lll24_32768", "kind": "host", "ens": "lll", "n": 24, "batch": 32768,
         "mode": MIXED},
        # benchmark configuration 4 at a quarter of its count: a mixed-size
        # ensemble in one plan
        {"name": "plan_lll_49000", "kind": "plan", "total": 49000, "smallest": 6, "largest": 48,
         "mode": MIXED},
        # CF determinants of one configuration's permutations
        {"name": "cf11_131072", "kind": "cf", "n": 11, "np": 22, "batch": 131072, "mode": MIXED},
    ]


def _flops(n):
    """One n x n complex LUP: trailing complex MACs at 8 flops, multipliers at 6."""
    return 4.0 * (n - 1) * n * (2 * n - 1) / 3.0 + 3.0 * n * (n - 1)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any size, batch, kind, type and mode of the listed ranges."""
    budget = 7e8  # flops of one pass, below the largest listed cases'
    kind = rng.choice(("batch",) * 6 + ("refcall", "host", "plan", "cf"))
    mode = rng.choice((MIXED, MIXED, MIXED, REF, FUSED))
    if kind == "batch":
        n = _log_int(rng, 4, 64)
        ens = rng.choice(("gauss", "lll"))
        c64 = rng.random() < 0.2 and (ens == "gauss" or n <= 32)
        batch = _log_int(rng, 16, min(2 << 17, budget / _flops(n)))
        pad = rng.choice((0, 0, 1, (1 << (n - 1).bit_length()) - n))
        return {"kind": kind, "ens": ens, "n": n, "pad": pad, "batch": batch, "mode": mode,
                "c64": c64}
    if kind == "refcall":
        n = _log_int(rng, 4, 24)
        return {"kind": kind, "n": n, "batch": _log_int(rng, 64, 16384), "pair": rng.random() < 0.5,
                "c64": rng.random() < 0.7}
    if kind == "host":
        n = _log_int(rng, 6, 32)
        batch = _log_int(rng, 256, min(65536, budget / _flops(n)))
        return {"kind": kind, "ens": rng.choice(("gauss", "lll")), "n": n, "batch": batch,
                "mode": rng.choice((MIXED, MIXED, FUSED))}
    if kind == "plan":
        k = rng.randrange(len(PLAN_SIZES) - 2)
        return {"kind": kind, "total": _log_int(rng, 700, 40000), "smallest": PLAN_SIZES[k],
                "largest": PLAN_SIZES[rng.randrange(k + 2, len(PLAN_SIZES))], "mode": MIXED}
    n = 2 * rng.randrange(2, 16) + 1
    return {"kind": "cf", "n": n, "np": n + rng.randrange(0, 2 * n),
            "batch": _log_int(rng, 256, min(131072, 0.2 * budget / _flops(n))), "mode": mode}


def _plan_sizes(case):
    sizes = [n for n in PLAN_SIZES if case["smallest"] <= n <= case["largest"]]
    each, left = divmod(case["total"], len(sizes))
    return [(n, each + (i < left)) for i, n in enumerate(sizes)]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _gauss(batch, n, gen, sigma=1.0):
    x = torch.randn(batch, n, n, 2, dtype=torch.float64, device="cuda", generator=gen)
    return torch.view_as_complex(x * (sigma / math.sqrt(2.0)))


def _lll(batch, n, gen):
    z = torch.randn(batch, n, 2, dtype=torch.float64, device="cuda", generator=gen)
    z = torch.view_as_complex(z * math.sqrt(n / 2.0))
    A = torch.empty(batch, n, n, dtype=torch.complex128, device="cuda")
    row = torch.exp(-0.25 * (z.real ** 2 + z.imag ** 2)).to(torch.complex128)
    for k in range(n):
        A[:, :, k] = row
        row = row * z
    return A


def _dense(case, seed):
    """The batch's n x n matrices, complex128, on the GPU."""
    gen = _generator(seed)
    A = (_lll if case.get("ens") == "lll" else _gauss)(case["batch"], case["n"], gen)
    return A.to(torch.complex64) if case.get("c64") else A


def _cf_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, np_ = case["n"], case["np"]
    phi = rng.uniform(0.0, 2.0 * np.pi, np_)
    theta = rng.uniform(0.15, np.pi / 2 - 0.15, np_)
    perm = np.argsort(rng.random((case["batch"], np_)), axis=1)[:, :n].astype(np.int16) + 1
    return phi, theta, perm


def _empty_out(batch, device="cuda"):
    host = device == "cpu"
    return lufqhe.DetResult(*(torch.zeros(batch, dtype=d, device=device, pin_memory=host)
                              for d in (torch.float64, torch.float64, torch.int8, torch.int32)))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cf":
        phi, theta, perm = _cf_inputs(case, seed)
        return {"case": case, "cfg": lufqhe.CfConfig(phi, theta, *CF_K, CF_MU, CF_NU),
                "perm": torch.from_numpy(perm).cuda(), "out": _empty_out(case["batch"])}
    if kind == "plan":
        gen, groups, off = _generator(seed), [], 0
        for n, count in _plan_sizes(case):
            groups.append((_lll(count, n, gen), off))
            off += count
        out = _empty_out(off)
        return {"case": case, "out": out,
                "plan": lufqhe.Plan(groups, out, mode=case["mode"], autotune=False)}
    A = _dense(case, seed)
    if kind == "batch" and case["pad"]:
        n = case["n"]
        P = torch.zeros(case["batch"], n, n + case["pad"], dtype=A.dtype, device="cuda")
        P[:, :, :n] = A
        A = P
    if kind == "host":
        H = torch.empty(A.shape, dtype=A.dtype, pin_memory=True)
        H.copy_(A)
        return {"case": case, "A": H, "out": _empty_out(case["batch"], "cpu")}
    if kind == "refcall":
        return {"case": case, "A": A, "work": torch.empty_like(A)}
    return {"case": case, "A": A, "out": _empty_out(case["batch"])}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "refcall":
        state["work"].copy_(state["A"])
        lufqhe.lucoregpu_call(state["work"], pair_product=case["pair"])
        return state["work"]
    out = state["out"]
    if kind == "batch":
        lufqhe.batch_lup_det(state["A"], mode=case["mode"], out=out)
    elif kind == "host":
        lufqhe.batch_lup_det_host(state["A"], mode=case["mode"], out=out)
    elif kind == "plan":
        state["plan"].execute()
    else:
        lufqhe.cf_det(state["cfg"], state["perm"], case["n"], mode=case["mode"], out=out)
    return {"logabs": out.logabs, "phase": out.phase, "parity": out.parity, "status": out.status}


def work(case):
    kind, n = case["kind"], case.get("n")
    if kind == "plan":
        sizes = _plan_sizes(case)
        return {"bytes": sum(c * (16.0 * m * m + 21.0) for m, c in sizes),
                "flops": sum(c * _flops(m) for m, c in sizes)}
    batch = case["batch"]
    if kind == "cf":
        # permutation rows in; the orbital sums: about 40 flops per particle pair
        return {"bytes": batch * (2.0 * n + 21.0) + case["np"] * (n + 2) * 16.0,
                "flops": batch * (_flops(n) + 40.0 * n * (n - 1))}
    entry = 8.0 if case.get("c64") else 16.0
    if kind == "refcall":
        return {"bytes": batch * 2.0 * entry * n * n, "flops": batch * _flops(n)}
    return {"bytes": batch * (entry * n * n + 21.0), "flops": batch * _flops(n)}


def _slogdet(A):
    """log|det| and phase in 64 bits, after scaling columns and rows by powers of two."""
    logabs = np.zeros(A.shape[0])
    for axis in (1, 2):
        e = np.frexp(np.abs(A).max(axis=axis, keepdims=True))[1]
        A = A * np.ldexp(1.0, -e)
        logabs = logabs + math.log(2.0) * e.reshape(A.shape[0], -1).sum(axis=1)
    sign, la = np.linalg.slogdet(A)
    return logabs + la, np.angle(sign)


def _lup(A):
    """L\\U by columns in 64 bits, and the permutation's sign: implicit row
    scaling on |Re|, pivot on |Re| / scale, ties to the last row."""
    A = A.copy()
    batch, n = A.shape[0], A.shape[1]
    at = np.arange(batch)
    hold = np.abs(A.real).max(axis=2)
    sign = np.ones(batch)
    for j in range(n):
        q = np.abs(A[:, j:, j].real) / hold[:, j:]
        p = n - 1 - np.argmax(q[:, ::-1], axis=1)
        row = A[at, p].copy()
        A[at, p] = A[:, j]
        A[:, j] = row
        hold[at, p] = hold[:, j]
        sign = np.where(p == j, sign, -sign)
        A[:, j + 1:, j] /= A[:, j, j][:, None]
        A[:, j + 1:, j + 1:] -= A[:, j + 1:, j][:, :, None] * A[:, j, j + 1:][:, None, :]
    return A, sign


def _cf_matrices(case, seed):
    phi, theta, perm = _cf_inputs(case, seed)
    n, q1 = case["n"], (case["n"] - 3) // 2 + 1
    u = np.cos(theta) * np.exp(1j * phi)
    v = np.sin(theta) * np.exp(-1j * phi)
    tab = np.empty((case["np"], n), dtype=np.complex128)
    tab[:, q1] = (np.cos(theta) * np.sin(theta)) ** (q1 - 1)
    for j in range(1, q1 + 1):
        tab[:, q1 + j] = tab[:, q1 + j - 1] * (u / v)
        tab[:, q1 - j] = tab[:, q1 - j + 1] * (v / u)
    p = perm.astype(np.int64) - 1
    A = tab[p]
    up, vp = u[p], v[p]
    s1, s2 = np.zeros(p.shape, np.complex128), np.zeros(p.shape, np.complex128)
    k1, k2, r1, r2 = CF_K
    for s in range(n):
        a, c = up * vp[:, s:s + 1], up[:, s:s + 1] * vp
        d = a - c
        d[:, s] = 1.0
        t1, t2 = (k1 * a + k2 * c) / d, (r1 * a + r2 * c) / d
        t1[:, s] = t2[:, s] = 0.0
        s1 += t1
        s2 += t2
    A[:, :, n - 2] = tab[p, q1 + CF_MU] * s1
    A[:, :, n - 1] = tab[p, q1 + CF_NU] * s2
    return A


def exact(case, seed):
    kind = case["kind"]
    if kind == "refcall":
        A = _dense(case, seed).to(torch.complex128).cpu().numpy()
        F, sign = _lup(A)
        det = sign * np.prod(np.diagonal(F, axis1=1, axis2=2), axis=1)
        if case["pair"]:
            even = det.size // 2 * 2
            det[0:even:2] = det[0:even:2] * det[1:even:2]
        F[:, 0, 0] = det
        return F
    if kind == "plan":
        gen, parts = _generator(seed), []
        for n, count in _plan_sizes(case):
            parts.append(_slogdet(_lll(count, n, gen).cpu().numpy()))
        logabs, phase = (np.concatenate([p[i] for p in parts]) for i in (0, 1))
    elif kind == "cf":
        logabs, phase = _slogdet(_cf_matrices(case, seed))
    else:
        logabs, phase = _slogdet(_dense(case, seed).to(torch.complex128).cpu().numpy())
    return {"logabs": logabs, "phase": phase, "parity": None, "status": None}
