"""The work that is timed: what a user of the reduced-order frequency sweep has it do, through
the Python front end (staccato_b200), over the range of sizes it is used with.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (inputs
on the GPU and one library handle a process), ``run`` is one pass, ``exact`` the same result in
64 bits by plain torch, ``work`` the bytes and operations the result cannot do without.

Refinement step counts and the error estimate of the mixed form (``steps``, ``berr``) describe the
route a system took and are not results; solutions, outputs, gradients and status words are.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from staccato_b200 import _capi, fe_tet10
from staccato_b200.adjoint import Param, backward
from staccato_b200.krylov import fom_sweep
from staccato_b200.project import DeviceCsr, orthonormalize, project, project_complex
from staccato_b200.rom import KrylovROMSubstructure
from staccato_b200.sweep import DeviceRom, solve_batched, sweep

C128, F64 = torch.complex128, torch.float64
TWO_PI = 2.0 * math.pi


def listed():
    return [
        # one design point of the smallest model: a few frequencies, where launches and latency count
        {"name": "point_r21", "kind": "sweep", "n": 21, "r": 1, "F": 8, "eta": 0.0, "damped": True, "near": False,
         "precision": "fp64", "f_lo": 20.0, "f_hi": 2000.0},
        # a small hysteretic model over one frequency band
        {"name": "plain_r64", "kind": "sweep", "n": 64, "r": 1, "F": 500, "eta": 0.02, "damped": False, "near": False,
         "precision": "fp64", "f_lo": 20.0, "f_hi": 2000.0},
        # the reference's middle order (odd) through its class: loads in, output DOFs out
        {"name": "back_transform_r189", "kind": "back_transform", "n": 189, "F": 1000, "n_in": 3, "loads": 2,
         "n_out": 12, "eta": 0.01, "damped": True},
        # many load cases close to resonance, Rayleigh and hysteretic damping
        {"name": "near_resonance_r256", "kind": "sweep", "n": 256, "r": 8, "F": 2048, "eta": 0.01, "damped": True,
         "near": True, "precision": "fp64", "f_lo": 10.0, "f_hi": 5000.0},
        # one call over an assembly's uneven models in the mixed precision, FP64 re-solve on
        {"name": "batch_mixed", "kind": "batch", "count": 16, "n_lo": 24, "n_hi": 512, "F_lo": 250, "F_hi": 1000,
         "eta": 0.02, "precision": "auto"},
        # the reference's largest order at a handful of frequencies
        {"name": "large_r2520", "kind": "sweep", "n": 2520, "r": 1, "F": 12, "eta": 0.02, "damped": False,
         "near": False, "precision": "fp64", "f_lo": 20.0, "f_hi": 2000.0},
        # one step of a gradient-based update: forward sweep with kept factors, adjoint backward
        {"name": "adjoint_r128", "kind": "adjoint", "n": 128, "r": 1, "F": 2000, "block": 8, "eta": 0.02},
        # projecting a solid model onto a real basis
        {"name": "project_tet10", "kind": "project", "nx": 10, "ny": 10, "nz": 40, "k": 96, "mats": 2},
        # projecting a damped model onto the complex Krylov basis
        {"name": "project_complex", "kind": "project_complex", "nx": 6, "ny": 6, "nz": 30, "k": 40, "mats": 3},
        # orthonormalising a basis
        {"name": "orthonormalize", "kind": "orthonormalize", "n": 107163, "k": 96},
        # full-order response of the solid model at one frequency, four load cases at once
        {"name": "fom_tet10", "kind": "fom", "nx": 10, "ny": 10, "nz": 40, "r": 4, "nf": 1},
        # interface Jacobians of a coupled assembly, one system a frequency
        {"name": "coupling_solves", "kind": "solve_batched", "count": 1000, "n": 24, "r": 1},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "back_transform", "batch", "large", "adjoint", "project",
                       "project_complex", "orthonormalize", "fom", "solve_batched"])
    if kind == "sweep":
        n, r = _logint(rng, 12, 600), rng.choice([1, 1, 2, 4, 5, 8])
        if n > 430:
            r = min(r, 4)
        F = max(4, min(_logint(rng, 8, 4000), int(2.0e11 / n ** 3)))
        return {"kind": "sweep", "n": n, "r": r, "F": F, "eta": rng.choice([0.0, 0.02]),
                "damped": rng.random() < 0.5, "near": n <= 300 and rng.random() < 0.3,
                "precision": rng.choice(["fp64", "fp64", "auto"]), "f_lo": 20.0, "f_hi": 2000.0}
    if kind == "back_transform":
        n = _logint(rng, 24, 400)
        return {"kind": kind, "n": n, "F": min(_logint(rng, 50, 3000), int(1.0e11 / n ** 3)), "n_in": rng.randint(1, 6),
                "loads": rng.randint(1, 4), "n_out": _logint(rng, 1, 200), "eta": rng.choice([0.0, 0.01]),
                "damped": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 16), "n_lo": 24, "n_hi": rng.randint(100, 512),
                "F_lo": rng.randint(50, 250), "F_hi": rng.randint(300, 1000), "eta": 0.02,
                "precision": rng.choice(["auto", "fp64"])}
    if kind == "large":
        n = _logint(rng, 700, 2520)
        return {"kind": "sweep", "n": n, "r": rng.choice([1, 2, 4]) if n < 2500 else 1, "F": rng.randint(2, 12), "eta": 0.02, "damped": rng.random() < 0.3,
                "near": False, "precision": "fp64", "f_lo": 20.0, "f_hi": 2000.0}
    if kind == "adjoint":
        block = rng.choice([4, 8])
        n = block * rng.randint(6, 24)
        return {"kind": kind, "n": n, "r": rng.choice([1, 1, 2, 3]), "F": _logint(rng, 100, 2000), "block": block,
                "eta": 0.02}
    if kind in ("project", "project_complex"):
        real = kind == "project"
        return {"kind": kind, "nx": rng.randint(3, 7), "ny": rng.randint(3, 7), "nz": rng.randint(8, 30),
                "k": rng.randint(8, 160) if real else rng.randint(6, 64), "mats": rng.randint(1, 3)}
    if kind == "orthonormalize":
        return {"kind": kind, "n": _logint(rng, 2000, 107163), "k": rng.randint(5, 130)}
    if kind == "fom":
        return {"kind": kind, "nx": rng.randint(2, 5), "ny": rng.randint(2, 5), "nz": rng.randint(8, 30),
                "r": rng.randint(1, 6), "nf": rng.randint(1, 3)}
    n = _logint(rng, 8, 200)
    return {"kind": "solve_batched", "count": _logint(rng, 20, 2000), "n": n, "r": rng.choice([1, 1, 2, 5])}


# ---------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _handle():
    """The program's library handle (legacy default stream, as torch's current one)."""
    return _capi.Handle(0)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, dtype=F64):
    return torch.randn(*shape, generator=g, dtype=dtype, device="cuda")


def _uniform(g, lo, hi, n):
    return lo + (hi - lo) * torch.rand(n, generator=g, dtype=F64, device="cuda")


def _modal_pair(g, n, f_lo, f_hi):
    """K = Q diag((2 pi f)^2) Q^T, f log-uniform in [f_lo, f_hi]; M = I + a little symmetric noise."""
    q, _ = torch.linalg.qr(_randn(g, n, n))
    lam = (TWO_PI * torch.exp(_uniform(g, math.log(f_lo), math.log(f_hi), n))) ** 2
    k = (q * lam[None, :]) @ q.T
    s = torch.triu(_randn(g, n, n))
    s = s + torch.triu(s, 1).T
    return q, lam, 0.5 * (k + k.T), torch.eye(n, dtype=F64, device="cuda") + (0.01 / math.sqrt(n)) * s


def _hyst(k, eta):
    return torch.complex(k, eta * k)


def _omega(g, F, f_lo, f_hi, k=None, m=None):
    if k is None:
        return TWO_PI * torch.linspace(max(1.0, f_lo / 20.0), f_hi, F, dtype=F64, device="cuda")
    # 60 % within 0.1 % of the generalised eigenfrequencies, the rest over the band
    li = torch.linalg.inv(torch.linalg.cholesky(m))
    fe = torch.sqrt(torch.clamp(torch.linalg.eigvalsh(li @ k @ li.T), min=0.0)) / TWO_PI
    near = torch.rand(F, generator=g, device="cuda") < 0.6
    pick = torch.randint(0, len(fe), (F,), generator=g, device="cuda")
    f = torch.where(near, fe[pick] * (1.0 + _uniform(g, -1e-3, 1e-3, F)), _uniform(g, f_lo, f_hi, F))
    return TWO_PI * f


def _cm(a):
    """Flat column-major copy of a matrix."""
    return a.t().contiguous().reshape(-1)


def _rom(g, n, r, F, eta, damped, near, f_lo, f_hi):
    _, _, k, m = _modal_pair(g, n, f_lo, f_hi)
    K, M = _hyst(k, eta), m.to(C128)
    D = (1e-5 * k + 2.0 * m).to(C128) if damped else None
    rhs = _randn(g, n, r, dtype=C128)
    return K, M, D, rhs, _omega(g, F, f_lo, f_hi, k if near else None, m)


def _device_rom(K, M, D, rhs, omega, eta=0.0, keep=False):
    rom = DeviceRom(n=K.shape[0], r=rhs.shape[1], F=len(omega), K=_cm(K), M=_cm(M), D=None if D is None else _cm(D),
                    rhs=_cm(rhs), omega=omega.contiguous(), eta=eta)
    rom.allocate_outputs("cuda", keep)
    return rom


def _batch_sizes(case, seed):
    rng = np.random.default_rng(case["count"] * 1000 + case["n_hi"])  # the assembly: the same for every seed
    ns = rng.integers(case["n_lo"], case["n_hi"] + 1, case["count"])
    Fs = rng.integers(case["F_lo"], case["F_hi"] + 1, case["count"])
    return [(int(n), int(r), int(F)) for n, r, F in zip(ns, rng.choice([1, 4], case["count"]), Fs)]


def _rom_inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "batch":
        return [_rom(g, n, r, F, case["eta"], False, False, 20.0, 2000.0) for n, r, F in _batch_sizes(case, seed)]
    return [_rom(g, case["n"], case["r"], case["F"], case["eta"], case["damped"], case["near"], case["f_lo"],
                 case["f_hi"])]


def _back_transform_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    _, _, k, m = _modal_pair(g, n, 20.0, 2000.0)
    D = (1e-5 * k + 2.0 * m).to(C128) if case["damped"] else None
    B, C = _randn(g, n, case["n_in"]).to(C128), _randn(g, case["n_out"], n).to(C128)
    load = _randn(g, case["n_in"], case["loads"]).to(C128)
    return _hyst(k, case["eta"]), m.to(C128), D, B, C, load, np.linspace(1.0, 2000.0, case["F"])


def _adjoint_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    q, lam, k, m = _modal_pair(g, n, 20.0, 2000.0)
    rhs, c = _randn(g, n, case["r"]).to(C128), _randn(g, n, dtype=C128)
    omega = TWO_PI * torch.linspace(1.0, 1500.0, case["F"], dtype=F64, device="cuda")
    return q, lam, k, m, rhs, c, omega


@functools.lru_cache(maxsize=8)
def _model(nx, ny, nz, free):
    """CSR pattern and values of the clamped block; free: the clamped DOFs taken out."""
    m = fe_tet10.clamped_block(nx, ny, nz)
    if not free:
        return m.indptr, m.indices, m.K, m.M
    keep = ~m.clamped
    new = np.cumsum(keep) - 1  # the clamped DOFs' rows and columns are empty
    indptr = np.concatenate([m.indptr[:-1][keep], m.indptr[-1:]])
    return indptr, new[m.indices].astype(np.int32), m.K, m.M


def _fe_inputs(case, seed, free=False):
    g = _gen(seed)
    indptr, indices, K, M = _model(case["nx"], case["ny"], case["nz"], free)
    csr = DeviceCsr.from_host(indptr, indices)
    # stiffness and density of this seed's material
    sk, sm = (1.0 + 0.2 * _uniform(g, -1.0, 1.0, 2)).tolist()
    Kd, Md = sk * torch.from_numpy(K).cuda(), sm * torch.from_numpy(M).cuda()
    return g, csr, [Kd, Md, 1e-5 * Kd + 2.0 * Md]


def _fom_freqs(case):
    return [300.0 + 600.0 * i / max(case["nf"] - 1, 1) for i in range(case["nf"])]


def _fom_inputs(case, seed):
    g, csr, vals = _fe_inputs(case, seed, free=True)
    loads = torch.zeros(case["r"], csr.n_rows, dtype=C128, device="cuda")
    dofs = torch.randperm(csr.n_rows, generator=g, device="cuda")[: case["r"]]
    loads[torch.arange(case["r"], device="cuda"), dofs] = 1e9
    return csr, [v.to(C128) for v in vals], loads


def _project_inputs(case, seed):
    g, csr, vals = _fe_inputs(case, seed)
    vals = vals[: case["mats"]]
    if case["kind"] == "project":
        return csr, vals, _randn(g, case["k"], csr.n_rows) / math.sqrt(csr.n_rows)
    return csr, [_hyst(v, 0.01) for v in vals], _randn(g, case["k"], csr.n_rows, dtype=C128) / math.sqrt(csr.n_rows)


def _ortho_inputs(case, seed):
    # Krylov-like columns: independent directions on a common part, of uneven size
    g = _gen(seed)
    V = _randn(g, case["k"], case["n"]) + 0.5 * _randn(g, 1, case["n"])
    return V * torch.exp(_uniform(g, -2.0, 2.0, case["k"]))[:, None]


def _solve_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    A = _randn(g, case["count"], n, n, dtype=C128) / math.sqrt(n) + 2.0 * torch.eye(n, dtype=C128, device="cuda")
    return A, _randn(g, case["count"], n, case["r"], dtype=C128)


PRECISION = {"fp64": _capi.SROM_FP64, "auto": _capi.SROM_MIXED_AUTO}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "handle": _handle()}
    if kind in ("sweep", "batch"):
        s["roms"] = [_device_rom(*rom) for rom in _rom_inputs(case, seed)]
        s["precision"] = PRECISION[case["precision"]]
        s["flags"] = 0 if case["precision"] == "fp64" else _capi.SROM_FLAG_FALLBACK_FP64
    elif kind == "back_transform":
        K, M, D, B, C, s["load"], s["freq"] = _back_transform_inputs(case, seed)
        s["sub"] = KrylovROMSubstructure(handle=s["handle"])
        s["sub"].set_reduced(K, M, D, B, C)
    elif kind == "adjoint":
        q, lam, k, m, rhs, s["c"], omega = _adjoint_inputs(case, seed)
        s["rom"] = _device_rom(k.to(C128), m.to(C128), None, rhs, omega, eta=case["eta"], keep=True)
        b = case["block"]
        s["params"] = [Param(U=_cm(q[:, j:j + b].to(C128)), s=lam[j:j + b].contiguous(), rank=b,
                             c0=complex(1.0, case["eta"])) for j in range(0, case["n"], b)]
        s["params"].append(Param(G=_cm(k.to(C128)), c0=1j))
    elif kind in ("project", "project_complex"):
        s["csr"], s["values"], s["V"] = _project_inputs(case, seed)
    elif kind == "orthonormalize":
        s["V"] = _ortho_inputs(case, seed)
    elif kind == "fom":
        s["csr"], s["values"], s["loads"] = _fom_inputs(case, seed)
        s["freq"] = _fom_freqs(case)
    else:
        s["A"], s["B"] = _solve_inputs(case, seed)
    return s


def run(s):
    kind, h = s["kind"], s["handle"]
    if kind in ("sweep", "batch"):
        sweep(h, s["roms"], precision=s["precision"], flags=s["flags"])
        return {"X": [r.X for r in s["roms"]], "info": [r.info for r in s["roms"]]}
    if kind == "back_transform":
        Y, info = s["sub"].back_transform_kmor(s["freq"], s["load"])
        return {"Y": Y, "info": info}
    if kind == "adjoint":
        rom = s["rom"]
        sweep(h, [rom], flags=_capi.SROM_FLAG_KEEP_FACTORS)
        X = rom.X.reshape(rom.F, rom.r, rom.n).transpose(1, 2)
        # J = sum |c^H x|^2: gbar = 2 c (c^H x)
        gbar = 2.0 * s["c"][None, :, None] * torch.einsum("i,fir->fr", s["c"].conj(), X)[:, None, :]
        grad, lam = backward(h, rom, gbar, s["params"], want_lambda=True)
        return {"X": X, "grad": grad, "lambda": lam}
    if kind == "project":
        return project(h, s["csr"], s["values"], s["V"])
    if kind == "project_complex":
        return project_complex(h, s["csr"], s["values"], s["V"])
    if kind == "orthonormalize":
        V = s["V"].clone()  # the program keeps the raw basis
        orthonormalize(h, V)
        return V
    if kind == "fom":
        K, M, D = s["values"]
        return fom_sweep(h, s["csr"], K, M, D, s["loads"], s["freq"])
    X, info = solve_batched(h, s["A"], s["B"])
    return {"X": X, "info": info}


# ---------------------------------------------------------------------------- 64-bit results
def _systems(K, M, D, omega, eta=0.0):
    """(chunk, A(w)) over the frequencies, a few GB of matrices at a time."""
    n = K.shape[0]
    step = max(1, int(1.0e9 / (16 * n * n)))
    for f in range(0, len(omega), step):
        w = omega[f:f + step, None, None]
        A = (1.0 + 1j * eta) * K - w * w * M
        yield slice(f, min(f + step, len(omega))), A if D is None else A + 1j * w * D


def _solutions(K, M, D, rhs, omega, eta=0.0):
    return torch.cat([torch.linalg.solve(A, rhs.expand(len(A), -1, -1)) for _, A in _systems(K, M, D, omega, eta)])


def _csr_mm(csr, vals, V):
    A = torch.sparse_csr_tensor(csr.rowptr, csr.colind.long(), vals, size=(csr.n_rows, csr.n_rows))
    return A @ V


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        X = [_solutions(*rom).transpose(1, 2).reshape(-1) for rom in _rom_inputs(case, seed)]
        return {"X": X, "info": [None] * len(X)}
    if kind == "back_transform":
        K, M, D, B, C, load, freq = _back_transform_inputs(case, seed)
        omega = TWO_PI * torch.from_numpy(freq).cuda()
        return {"Y": C @ _solutions(K, M, D, B @ load, omega), "info": None}
    if kind == "adjoint":
        q, lam, k, m, rhs, c, omega = _adjoint_inputs(case, seed)
        K, M, eta, b = k.to(C128), m.to(C128), case["eta"], case["block"]
        X = _solutions(K, M, None, rhs, omega, eta)
        gbar = 2.0 * c[None, :, None] * torch.einsum("i,fir->fr", c.conj(), X)[:, None, :]
        L = torch.cat([torch.linalg.solve(A.mH, gbar[f]) for f, A in _systems(K, M, None, omega, eta)])
        qc = q.to(C128)
        # -Re sum lambda^H dA x: one rank term a mode, then the loss factor
        modes = (1.0 + 1j * eta) * lam * torch.einsum("fjr,fjr->j", (qc.T @ L).conj(), qc.T @ X)
        last = 1j * torch.einsum("fir,fir->", L.conj(), K @ X)
        grad = -torch.cat([modes.real.reshape(-1, b).sum(1), last.real.reshape(1)])
        return {"X": X, "grad": grad, "lambda": L}
    if kind in ("project", "project_complex"):
        csr, vals, V = _project_inputs(case, seed)
        Vt = V.t().contiguous()
        return [V.conj() @ _csr_mm(csr, v, Vt) for v in vals]
    if kind == "orthonormalize":
        Q, R = torch.linalg.qr(_ortho_inputs(case, seed).t().contiguous())
        return (Q * torch.sign(torch.diagonal(R))[None, :]).t().contiguous()
    if kind == "fom":
        csr, (K, M, D), loads = _fom_inputs(case, seed)
        n = csr.n_rows
        if n > 16000:
            return None
        rows = torch.repeat_interleave(torch.arange(n, device="cuda"), csr.rowptr[1:] - csr.rowptr[:-1])
        out = []
        for f in _fom_freqs(case):
            w = TWO_PI * f
            A = torch.zeros(n, n, dtype=C128, device="cuda")
            A[rows, csr.colind.long()] = K - w * w * M + 1j * w * D
            out.append(torch.linalg.solve(A, loads.t()).t())
            del A
        return torch.stack(out)
    A, B = _solve_inputs(case, seed)
    return {"X": torch.linalg.solve(A, B), "info": None}


# ---------------------------------------------------------------------------- unavoidable work
def _sweep_work(n, r, F, mats):
    return {"bytes": 16.0 * (mats * n * n + n * r + F * n * r) + 8.0 * F,
            "flops": F * (8.0 / 3.0 * n ** 3 + 8.0 * n * n * r)}


def work(case):
    kind = case["kind"]
    if kind == "sweep":
        return _sweep_work(case["n"], case["r"], case["F"], 3 if case["damped"] else 2)
    if kind == "batch":
        parts = [_sweep_work(n, r, F, 2) for n, r, F in _batch_sizes(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "back_transform":
        n, F, q = case["n"], case["F"], case["loads"]
        w = _sweep_work(n, q, F, 3 if case["damped"] else 2)
        return {"bytes": 16.0 * (3 * n * n + n * case["n_in"] + case["n_out"] * n + F * case["n_out"] * q),
                "flops": w["flops"] + 8.0 * F * case["n_out"] * n * q}
    if kind == "adjoint":
        n, r, F = case["n"], case["r"], case["F"]
        w = _sweep_work(n, r, F, 2)
        # factors, solutions and adjoint solutions written once; two more triangles and the gradient terms
        return {"bytes": w["bytes"] + 16.0 * F * (n * n + n * r) + 16.0 * 2 * n * n,
                "flops": w["flops"] + F * r * (8.0 * n * n + 16.0 * n * n + 8.0 * n * n)}
    if kind in ("project", "project_complex"):
        indptr, _, _, _ = _model(case["nx"], case["ny"], case["nz"], False)
        n, nnz, k, q = len(indptr) - 1, float(indptr[-1]), case["k"], case["mats"]
        z, f = (8.0, 2.0) if kind == "project" else (16.0, 8.0)
        return {"bytes": z * nnz * q + 4.0 * nnz + 8.0 * n + z * n * k + z * k * k * q,
                "flops": f * q * (nnz * k + float(n) * k * k)}
    if kind == "orthonormalize":
        return {"bytes": 16.0 * case["n"] * case["k"], "flops": 2.0 * case["n"] * case["k"] ** 2}
    if kind == "fom":
        # elimination of a band of one cross-section of nodes (lower triangle) and the substitutions
        s = 3.0 * (2 * case["nx"] + 1) * (2 * case["ny"] + 1)
        n, bw = s * 2 * case["nz"], 2.0 * s
        return {"bytes": 16.0 * n * (bw + 2 * case["r"]) * case["nf"],
                "flops": case["nf"] * (4.0 * n * bw * bw + 16.0 * n * bw * case["r"])}
    n, r, F = case["n"], case["r"], case["count"]
    return {"bytes": 16.0 * F * (n * n + 2 * n * r), "flops": F * (8.0 / 3.0 * n ** 3 + 8.0 * n * n * r)}
