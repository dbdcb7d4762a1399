"""Performance cases of the solve phase: what a program that uses this package has it do.

A case is one call (or one short sequence of calls) through the public Python entry points on a
seeded workload of the package, timed on the GPU; see ``listed`` for what each stands for.
``prepare`` makes what such a program has in hand: the device setup of a matrix (uploaded once, kept
for every right-hand side of it) and inputs drawn from the seed.  ``run`` is one pass, ``exact`` the
same result in 64 bits from plain torch / numpy, ``work`` the bytes and operations of one pass that
no implementation can do without.
"""
from __future__ import annotations

import math
import os
import sys
from collections import OrderedDict
from concurrent.futures import ThreadPoolExecutor
from dataclasses import replace

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "algebraic-multilevel-preconditioner_b200"))

from s2l_b200 import capi, partition, sequence, setup_phase  # noqa: E402
from s2l_b200 import workloads as W  # noqa: E402

BASE = {"overlap": 1, "nev": 20, "one_level": "ras", "coarse": "deflated", "pou": "boolean", "imbalance": 0.0,
        "precision": "double", "approx": "none", "k": 1, "restart": 50}


def _case(name, entry, family, nx, nsub, **kw):
    return {"name": name, "entry": entry, "family": family, "nx": nx, "nsub": nsub, **BASE, **kw}


def listed():
    return [
        # the smallest call: one preconditioner apply on a small 2D problem (a caller's own Krylov
        # loop over the drop-in preconditioner); all latency and launches
        _case("apply_poisson2d_40", "apply", "poisson2d", 40, 4, coarse="additive"),
        # the reference's own CPU case: 2D Poisson 200^2, additive coarse term, LU, GMRES(30)
        _case("gmres_poisson2d_200", "gmres", "poisson2d", 200, 8, coarse="additive", restart=30),
        # BiCGStab with ASM and the multiplicity partition of unity on uneven parts of an odd grid
        _case("bicgstab_laplace3d_27", "bicgstab", "laplace3d", 27, 6, one_level="asm", coarse="additive",
              pou="multiplicity", imbalance=0.2),
        # an ordinary single solve: pressure Poisson of a bubbly flow, L L^T, deflated RAS
        _case("gmres_bubbles3d_48", "gmres", "bubbles3d", 48, 8),
        # a few right-hand sides at once (not a power of two) on an odd grid, overlap 2
        _case("block5_bubbles3d_37", "gmres_block", "bubbles3d", 37, 5, overlap=2, k=5),
        # nonsymmetric, FP32 LU factors under flexible FP64 GMRES(40)
        _case("gmres_convdiff3d_48_fp32", "gmres", "convdiff3d", 48, 12, nev=24, precision="single", restart=40),
        # the inexact local solver: one AMG V-cycle per subdomain
        _case("amg_bubbles3d_64", "gmres", "bubbles3d", 64, 16, approx="amg"),
        # one step of a time loop: refactorization for the next matrix, then its solve
        _case("refactor_bubbles3d_40", "refactor", "bubbles3d", 40, 8),
        # serving: requests on one matrix queued at once on the worker threads (host vectors)
        _case("serve8_bubbles3d_48_fp32", "serve", "bubbles3d", 48, 8, precision="single", k=8),
        # the benchmark's matrix (1.0M rows, 64 subdomains): the reference's configuration in FP64,
        # FP32 factors under flexible FP64 GMRES, and 16 right-hand sides at once
        _case("gmres_bubbles3d_100", "gmres", "bubbles3d", 100, 64),
        _case("gmres_bubbles3d_100_fp32", "gmres", "bubbles3d", 100, 64, precision="single"),
        _case("block16_bubbles3d_100_fp32", "gmres_block", "bubbles3d", 100, 64, precision="single", k=16),
    ]


def draw(rng):
    """One more case of the listed ranges: sizes log-uniform (odd ones among them), subdomains of
    about 1,500 to 16,000 rows in 3D and 400 to 6,000 in 2D, at most 32 of them."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["apply", "gmres", "gmres", "gmres_block", "bicgstab", "refactor", "serve"])
    family = rng.choice(["poisson2d", "laplace3d", "bubbles3d", "bubbles3d", "convdiff3d"])
    if entry in ("refactor", "serve"):
        family = "bubbles3d"
    if family == "poisson2d":
        nx = log_int(40, 260)
        rows = nx * nx
        nsub = max(2, min(32, int(rows / log_int(400, 6000))))
    else:
        nx = log_int(16, 40 if entry == "refactor" else 64)
        rows = nx ** 3
        nsub = max(2 if nx < 32 else 4, min(32, int(rows / log_int(1500, 16000))))
    kw = {"overlap": rng.choice([1, 1, 2]) if family == "bubbles3d" else 1, "coarse": rng.choice(["deflated", "additive"]),
          "imbalance": rng.choice([0.0, 0.0, 0.2]), "restart": rng.choice([30, 40, 50])}
    if entry in ("apply", "bicgstab") and rng.random() < 0.5:
        kw |= {"one_level": rng.choice(["ras", "asm"]), "pou": "multiplicity"}
    if entry == "gmres_block":
        kw["k"] = rng.randint(2, 16)
    if entry == "serve":
        kw["k"] = rng.randint(2, 12)
    if entry in ("gmres", "gmres_block", "serve") and rng.random() < 0.5:
        kw["precision"] = "single"
    if entry == "gmres" and family == "bubbles3d" and kw.get("precision") != "single" and rng.random() < 0.3:
        kw["approx"] = "amg"
    if entry == "refactor":
        kw |= {"coarse": "deflated", "overlap": 1}
    c = _case("drawn", entry, family, nx, nsub, **kw)
    del c["name"]
    return c


# ----------------------------------------------------------------------------- workloads and setups

def _workload(c) -> W.Workload:
    local = "cholesky" if c["family"] in ("bubbles3d", "laplace3d") else "lu"
    opts = setup_phase.SchwarzOptions(one_level=c["one_level"], coarse=c["coarse"], pou=c["pou"], overlap=c["overlap"],
                                      nev=c["nev"], local_factorization=local, local_approx=c["approx"])
    kind = "laplace2d" if c["family"] == "poisson2d" else c["family"]
    return W.Workload(c["family"], kind, c["nx"], c["nsub"], opts, restart=c["restart"],
                      nbubbles=200 if c["nx"] == 100 else max(4, c["nx"] ** 3 // 5000), imbalance=c["imbalance"])


def _flexible(c) -> bool:
    return c["precision"] == "single"


_HOST = {}            # the last host setup (its FP64 and FP32 device setups share it)
_KEPT = OrderedDict()  # device setups by case, the most recently used last
_KEPT_BYTES = 48e9
_CTX = None


def _host_setup(c):
    key = tuple(sorted((k, v) for k, v in c.items() if k not in ("name", "entry", "precision", "k", "restart")))
    if key not in _HOST:
        _HOST.clear()
        # threads, each with one BLAS thread: the factorizations release the interpreter's lock
        with ThreadPoolExecutor(os.cpu_count() or 1, initializer=setup_phase._one_thread_worker) as pool:
            _HOST[key] = W.build(_workload(c), use_cache=False, pool=pool)
    return _HOST[key]


def _context():
    global _CTX
    if _CTX is None:
        _CTX = capi.Context(0)
        _CTX.serve_start(4)
    return _CTX


def _device_setup(c):
    """The device setup of the case's matrix and the stream its calls run on, made once and kept
    (within _KEPT_BYTES of device memory), as a program keeps them for every solve of the matrix."""
    key = tuple(sorted((k, v) for k, v in c.items() if k != "name"))
    if key in _KEPT:
        _KEPT.move_to_end(key)
        return _KEPT[key]
    while _KEPT and sum(g.device_bytes() for g, _, _ in _KEPT.values()) > _KEPT_BYTES:
        _KEPT.popitem(last=False)[1][0].close()
    st = _host_setup(c)
    dev = setup_phase.with_factor_precision(st, "single") if c["precision"] == "single" else st
    g = capi.GpuSetup(_context(), dev, options={"refactor": 1} if c["entry"] == "refactor" else None)
    stream = torch.cuda.Stream()
    if c["entry"] != "serve":
        g.set_stream(stream.cuda_stream)
    light = None
    if c["entry"] == "refactor":  # what the next matrices of the sequence need of the setup
        light = replace(st, subdomains=[None] * st.nsub, E=np.zeros((0, 0)))
    _KEPT[key] = (g, stream, light)
    return _KEPT[key]


# ----------------------------------------------------------------------------- inputs

def _rows(c) -> int:
    return c["nx"] ** (2 if c["family"] == "poisson2d" else 3)


def _rhs(c, seed):
    """k right-hand sides U[-1, 1], the workloads' distribution."""
    gen = torch.Generator().manual_seed(int(seed))
    return 2.0 * torch.rand((c["k"], _rows(c)), generator=gen, dtype=torch.float64) - 1.0


def _moved(c, seed) -> W.Workload:
    """The matrix of the moving-bubble sequence at a time of the seed's."""
    t = 0.5 + 1.5 * float(torch.rand(1, generator=torch.Generator().manual_seed(int(seed) + 77)))
    return replace(_workload(c), time=t)


def prepare(case, seed):
    g, stream, light = _device_setup(case)
    s = {"case": case, "g": g, "stream": stream}
    b = _rhs(case, seed)
    if case["entry"] == "serve":
        s["b"] = [r.numpy() for r in b]
    else:
        s["b"] = (b[0] if case["entry"] != "gmres_block" else b).contiguous().cuda()
    if case["entry"] == "refactor":
        vals, _ = sequence.values_in_setup_order(W.make_problem(_moved(case, seed)).A, light)
        s["values"] = torch.from_numpy(np.ascontiguousarray(vals)).cuda()
    torch.cuda.synchronize()
    return s


def run(s):
    c, g, b = s["case"], s["g"], s["b"]
    kw = {"rtol": 1e-8}
    if c["entry"] != "bicgstab":
        kw |= {"restart": c["restart"], "flexible": _flexible(c), "strict": _flexible(c)}
    if c["entry"] == "serve":
        tickets = [g.submit(r, **kw) for r in b]
        out = []
        for t in tickets:
            x, _, status = t.wait()
            if status != capi.S2L_OK:
                raise RuntimeError(t.info()["error"])
            out.append(x)
            t.free()
        return out
    with torch.cuda.stream(s["stream"]):
        if c["entry"] == "apply":
            z = torch.empty_like(b)
            g.apply(b.data_ptr(), out=z.data_ptr())
            return z
        x = torch.zeros_like(b)
        if c["entry"] == "gmres_block":
            _, info = g.gmres_block((b.data_ptr(), c["k"]), device_out=x.data_ptr(), **kw)
            return {"x": x, "iterations": [r["iterations"] for r in info]}
        if c["entry"] == "refactor":
            g.refactor(s["values"].data_ptr())
        solve = g.bicgstab if c["entry"] == "bicgstab" else g.gmres
        _, info = solve(b.data_ptr(), device_out=x.data_ptr(), **kw)
        return {"x": x, "iterations": info["iterations"]}


# ----------------------------------------------------------------------------- work

ITERATIONS = {"poisson2d": 24, "laplace3d": 16, "bubbles3d": 14, "convdiff3d": 16}


def work(case):
    """Nominal: the iterations a family takes, per iteration one preconditioner apply (factor
    values once: one triangle where the factor is symmetric; coarse basis, E^-1), one product with A
    and one pass over the Krylov basis.  The fill of a factor is a fit to the workloads' own."""
    c = case
    n, nsub, two_d = _rows(c), c["nsub"], c["family"] == "poisson2d"
    nnz = (5 if two_d else 7) * n
    side = (n / nsub) ** (1 / 2 if two_d else 1 / 3) + 1.2 * c["overlap"]
    m = side ** (2 if two_d else 3)
    fill = m * (6.3 * math.log(m) if two_d else 0.48 * m ** (2 / 3))  # both triangles of one subdomain
    if c["family"] in ("bubbles3d", "laplace3d"):
        fill /= 2
    if c["approx"] == "amg":
        fill = 10.0 * m
    size = 4 if c["precision"] == "single" else 8
    n0 = nsub * c["nev"]
    k = c["k"]
    matrix = nnz * 12.0
    apply_bytes = nsub * fill * size + 8.0 * n * c["nev"] + 8.0 * n0 * n0 + (matrix if c["coarse"] == "deflated" else 0.0)
    apply_flops = 4.0 * nsub * fill + 4.0 * n * c["nev"] + 2.0 * n0 * n0
    if c["entry"] == "apply":
        return {"bytes": apply_bytes + 16.0 * n, "flops": apply_flops}
    its = ITERATIONS[c["family"]]
    basis = 8.0 * n * (its / 2 if c["entry"] != "bicgstab" else 6)
    step = apply_bytes + matrix + k * (basis + 32.0 * n)
    flops = k * (apply_flops + 2.0 * nnz + basis / 2)
    extra = 2 * nsub * fill * 8.0 if c["entry"] == "refactor" else 0.0
    return {"bytes": its * step + extra, "flops": its * flops}


# ----------------------------------------------------------------------------- 64-bit results

def _matrix(c, w):
    """The renumbered matrix of a workload (torch, CSR, on the GPU) and its symmetry."""
    prob = W.make_problem(w)
    _, n2o, _ = partition.renumber(W.make_partition(w, prob), c["nsub"])
    A = partition.permute(prob.A.tocsr(), n2o)
    t = torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)), torch.from_numpy(A.indices.astype(np.int64)),
                                torch.from_numpy(A.data.astype(np.float64)), size=A.shape).cuda()
    return t, torch.from_numpy(A.diagonal()).cuda(), prob.symmetric


def _solve(A, diag, symmetric, b):
    """A^-1 b in FP64 to a true residual of 1e-12: Jacobi CG, or Jacobi BiCGStab, restarted from
    its true residual."""
    x, bn = torch.zeros_like(b), float(b.norm())
    for _ in range(8):
        r = b - A @ x
        if float(r.norm()) <= 1e-12 * bn:
            return x
        stop = 0.3e-12 * bn
        if symmetric:
            z = r / diag
            p, rz = z.clone(), torch.dot(r, z)
            for it in range(6000):
                q = A @ p
                a = rz / torch.dot(p, q)
                x += a * p
                r -= a * q
                z = r / diag
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
                if it % 25 == 24 and float(r.norm()) <= stop:
                    break
        else:
            rh, rho, p, d = r.clone(), torch.dot(r, r), r.clone(), torch.zeros_like(x)
            for it in range(4000):
                y = p / diag
                v = A @ y
                a = rho / torch.dot(rh, v)
                s = r - a * v
                z = s / diag
                t = A @ z
                om = torch.dot(t, s) / torch.dot(t, t)
                d += a * y + om * z
                r = s - om * t
                rho, old = torch.dot(rh, r), rho
                p = r + (rho / old) * (a / om) * (p - om * v)
                if it % 25 == 24 and not float(r.norm()) > stop:
                    break
            if not bool(torch.isfinite(d).all()):
                return None
            x += d
    return x if float((b - A @ x).norm()) <= 1e-11 * bn else None


def _exact_apply(c, r):
    """Two-level Schwarz with dense local solves (small subdomains only)."""
    st = _host_setup(c)
    if max(s.n_local for s in st.subdomains) > 6000:
        return None
    r = r.numpy()
    z, x0, one = np.zeros(st.n), np.zeros(st.n), r
    if c["coarse"] != "none" and st.n0:
        Wc = np.zeros((st.n, st.n0)) if st.n * st.n0 < 3e8 else None
        if Wc is None:
            return None
        for i, s in enumerate(st.subdomains):
            Wc[s.l2g(), st.offsets[i]:st.offsets[i + 1]] = s.V
        x0 = Wc @ np.linalg.solve(Wc.T @ (st.A @ Wc), Wc.T @ r)
        if c["coarse"] == "deflated":
            one = r - st.A @ x0
    for s in st.subdomains:
        i = s.l2g()
        y = np.linalg.solve(s.Aii.toarray(), one[i])
        z[i] += y * (s.D if c["one_level"] == "ras" else 1.0)
    return torch.from_numpy(x0 + z)


def exact(case, seed):
    c, b = case, _rhs(case, seed)
    if c["entry"] == "apply":
        return _exact_apply(c, b[0])
    A, diag, symmetric = _matrix(c, _moved(c, seed) if c["entry"] == "refactor" else _workload(c))
    if c["entry"] == "refactor":  # the moved matrix in the order of the setup's own partition
        symmetric = True
    xs = [_solve(A, diag, symmetric, r.cuda()) for r in b]
    if c["entry"] == "serve":
        return xs
    if c["entry"] == "gmres_block":
        x = torch.stack(xs) if all(x is not None for x in xs) else None
        return {"x": x, "iterations": [None] * c["k"]}
    return {"x": xs[0], "iterations": None}
