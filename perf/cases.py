"""Performance cases of the framework's public entry points.

``listed()`` names the workloads, ``draw(rng)`` gives others of the same
ranges, ``prepare`` makes what a program holds before the call (operators on
the device, sample vectors), ``run`` is one pass through the entry points, and
``exact`` restates it in plain torch FP64.  Geometry (lattices, neighbour
lists) depends on sizes only and is kept; every value depends on the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rsatb_b200 import lattice
from rsatb_b200.adjoint import KpmDosLoss
from rsatb_b200.calc import (Chebyshev, ISQRTMPreconditioner, KpmKernel, cg_solve,
                             evaluate_kpm_density, kpm_dos_moments)
from rsatb_b200.isqrt import inverse_sqrt_columns_batched
from rsatb_b200.transport import BASTIN, GREENWOOD, dc_spectrum_fftcheb
from rsatb_b200.vbcsr import BlockSpMat

DEV = "cuda"

# Energy windows (eV) that hold each model's spectrum for every seed.
WINDOW = {"graphene": (-8.9, 8.9), "tbg": (-11.0, 9.0), "silicon": (-21.5, 24.0),
          "diamond": (-9.2, 9.2)}


def listed():
    return [
        # One rescaled operator application on a small flake: the inner call
        # of a program's own propagation or Lanczos loop (latency).
        {"name": "apply_graphene_f64", "kind": "apply", "model": "graphene", "size": 60,
         "R": 8, "precision": "f64", "complex": True},
        # One S^-1/2 H S^-1/2 application on a mid-size LCAO crystal.
        {"name": "apply_diamond_f64", "kind": "apply", "model": "diamond", "size": 8, "R": 16,
         "precision": "f64", "complex": False},
        # Real-time propagation of a few wave packets over one time step.
        {"name": "propagate_graphene_f64", "kind": "propagate", "model": "graphene",
         "size": 200, "R": 4, "precision": "f64", "complex": True, "terms": 200},
        # Density of states of a pz flake: 7,200 orbitals, 8 random phases.
        {"name": "dos_graphene_f64", "kind": "dos", "model": "graphene", "size": 60, "R": 8,
         "precision": "f64", "complex": True, "moments": 512},
        # Density of states at a k-point: complex Hermitian sp3s* blocks.
        {"name": "dos_silicon_kpoint_f64", "kind": "dos", "model": "silicon_k", "size": 8,
         "R": 6, "precision": "f64", "complex": True, "moments": 400},
        # The mixed-precision DOS of a large non-orthogonal crystal (N = 262,144).
        {"name": "dos_diamond_f32", "kind": "dos", "model": "diamond", "size": 16, "R": 128,
         "precision": "f32", "complex": False, "moments": 256},
        # Kubo-Greenwood spectrum of twisted bilayer graphene, 47,632 atoms.
        {"name": "transport_tbg_f32", "kind": "transport", "model": "tbg", "size": 31,
         "tiles": 2, "R": 16, "precision": "f32", "moments": 2048, "bastin": False},
        # The same route in FP64 at a moment count that is no power of two.
        {"name": "transport_tbg_f64", "kind": "transport", "model": "tbg", "size": 15,
         "tiles": 2, "R": 5, "precision": "f64", "moments": 1000, "bastin": False},
        # Kubo-Bastin (all six tensor components) of a pz flake.
        {"name": "transport_bastin_f64", "kind": "transport", "model": "graphene", "size": 40,
         "tiles": 1, "R": 4, "precision": "f64", "moments": 512, "bastin": True},
        # Graph-local overlap factors: ragged batch of dense S^-1/2.
        {"name": "isqrt_batch", "kind": "isqrt", "problems": 1500, "n_min": 40, "n_max": 400},
        # One training step of a DOS loss over sp3s* block values.
        {"name": "adjoint_silicon_f64", "kind": "adjoint", "size": 8, "R": 32, "moments": 256},
        # S X = B for the exact Solve form: batched CG.
        {"name": "solve_diamond_f64", "kind": "solve", "size": 8, "R": 16, "precision": "f64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "propagate", "dos", "dos", "transport", "transport", "isqrt",
                       "adjoint", "solve"])
    precision = rng.choice(["f64", "f32"])
    if kind in ("apply", "propagate", "dos"):
        model = rng.choice(["graphene", "silicon_k", "diamond", "tbg"])
        c = {"kind": kind, "model": model, "R": _log(rng, 1, 64), "precision": precision,
             "complex": model in ("graphene", "silicon_k", "tbg")}
        if model == "graphene":
            c["size"] = _log(rng, 20, 250)
        elif model == "tbg":
            c["size"], c["tiles"] = rng.choice([5, 8, 11, 15]), rng.choice([1, 2])
        else:
            c["size"] = rng.randint(3, 10)
        if kind == "dos":
            c["moments"] = _log(rng, 50, 512)
        if kind == "propagate":
            c["terms"] = _log(rng, 20, 300)
        return c
    if kind == "transport":
        bastin = rng.random() < 0.3
        model = rng.choice(["graphene", "tbg", "tbg"])
        c = {"kind": kind, "model": model, "tiles": rng.choice([1, 2]), "R": _log(rng, 1, 16),
             "precision": precision, "bastin": bastin,
             "moments": rng.choice([256, 512, 1024, 2048]) if rng.random() < 0.6
             else _log(rng, 100, 1500)}
        c["size"] = rng.choice([5, 8, 11, 15]) if model == "tbg" else _log(rng, 10, 60)
        if model == "graphene":
            c["tiles"] = 1
        return c
    if kind == "isqrt":
        lo = _log(rng, 20, 200)
        return {"kind": kind, "problems": _log(rng, 30, 1200), "n_min": lo,
                "n_max": rng.randint(lo, 400)}
    if kind == "adjoint":
        return {"kind": kind, "size": rng.randint(2, 8), "R": _log(rng, 1, 32),
                "moments": _log(rng, 32, 256)}
    return {"kind": "solve", "size": rng.randint(3, 9), "R": _log(rng, 1, 64),
            "precision": precision}


# ------------------------------------------------------------------ geometry

@functools.lru_cache(maxsize=None)
def _geometry(model, size, tiles=1):
    """Pattern, mirror slots and the seed-independent block values."""
    if model == "graphene":
        H, pos, cell = lattice.graphene(size, size)
        disp = lattice.graphene_displacements(H, pos, cell)
        row_ptr, col_ind, b, base, dist2 = H.row_ptr, H.col_ind, 1, H.values, None
    elif model == "tbg":
        H, _, _, disp = lattice.twisted_bilayer_graphene(size, (tiles, tiles))
        row_ptr, col_ind, b, base, dist2 = H.row_ptr, H.col_ind, 1, H.values, None
    else:
        row_ptr, col_ind, dist2, _ = lattice.diamond_pattern(size, 8 if model == "silicon" else 11)
        disp, base, b = None, None, 5 if model == "silicon" else 8
    n = row_ptr.size - 1
    rows = np.repeat(np.arange(n, dtype=np.int64), np.diff(row_ptr))
    key = rows * n + col_ind
    mirror = np.searchsorted(key, col_ind.astype(np.int64) * n + rows)
    return {"row_ptr": row_ptr, "col_ind": col_ind, "b": b, "n": n, "rows": rows, "base": base,
            "dist2": dist2, "disp": disp, "mirror": torch.from_numpy(mirror)}


def _hermitian(geo, blocks, phase=None):
    """Blocks with V[j, i] = V[i, j]^H: the upper ones drawn, the lower mirrored."""
    rows = torch.from_numpy(geo["rows"]).to(DEV)
    cols = torch.from_numpy(geo["col_ind"]).to(DEV)
    mirror = geo["mirror"].to(DEV)
    if phase is not None:
        blocks = blocks * torch.polar(torch.ones_like(phase), phase)[:, None, None]
    flipped = blocks[mirror].transpose(1, 2)
    if blocks.is_complex():
        flipped = flipped.conj()
    out = torch.where((rows < cols)[:, None, None], blocks, flipped)
    return torch.where((rows == cols)[:, None, None], 0.5 * (blocks + flipped), out)


_SILICON = None


def _silicon_means():
    global _SILICON
    if _SILICON is None:
        _SILICON = (np.diag([-4.20, 1.715, 1.715, 1.715, 6.685]), np.array(
            [[-2.08, 1.43, 1.43, 1.43, 0.0], [-1.43, 0.43, 1.13, 1.13, -1.36],
             [-1.43, 1.13, 0.43, 1.13, -1.36], [-1.43, 1.13, 1.13, 0.43, -1.36],
             [0.0, 1.36, 1.36, 1.36, 0.0]]))
    return _SILICON


def _values(case, seed):
    """FP64 block values on the device: {"H": ..., "S": ..., "Z": ...}."""
    gen = torch.Generator(device=DEV).manual_seed(seed * 7919 + 17)
    model = case.get("model", "silicon" if case["kind"] == "adjoint" else "diamond")
    geo = _geometry("silicon" if model == "silicon_k" else model, case["size"],
                    case.get("tiles", 1))
    nnz, b = geo["col_ind"].size, geo["b"]
    f64 = {"device": DEV, "dtype": torch.float64}
    if model in ("graphene", "tbg"):
        # Hopping disorder of one per cent, symmetric.
        s = 1.0 + 0.01 * torch.rand(geo["n"], generator=gen, **f64)
        r = torch.from_numpy(geo["rows"]).to(DEV)
        c = torch.from_numpy(geo["col_ind"]).to(DEV).long()
        v = torch.from_numpy(geo["base"]).to(DEV) * (s[r] * s[c])[:, None, None]
        return geo, {"H": v}
    d2 = torch.from_numpy(geo["dist2"]).to(DEV)
    if model in ("silicon", "silicon_k"):
        on, nn = (torch.from_numpy(m).to(DEV) for m in _silicon_means())
        mean = torch.where((d2 == 0)[:, None, None], on,
                           torch.where((d2 == 3)[:, None, None], nn, 0.1 * nn))
        v = mean + 0.1 * torch.randn(nnz, b, b, generator=gen, **f64)
        ph = (2 * math.pi * torch.rand(nnz, generator=gen, **f64) if model == "silicon_k"
              else None)
        return geo, {"H": _hermitian(geo, v, ph)}
    r = d2.double().sqrt() * (3.567 / 4.0)
    H = torch.randn(nnz, b, b, generator=gen, **f64) * torch.exp(-r / 1.5)[:, None, None]
    S = 0.15 * torch.rand(nnz, b, b, generator=gen, **f64) * torch.exp(-r / 1.2)[:, None, None]
    S[d2 == 0] = torch.eye(b, **f64)
    S = _hermitian(geo, S)
    Z = -0.35 * S
    Z[d2 == 0] = torch.eye(b, **f64)
    return geo, {"H": _hermitian(geo, H), "S": S, "Z": Z}


def _matrix(geo, values, imaginary=False):
    return BlockSpMat(geo["row_ptr"], geo["col_ind"], values.cpu().numpy(), geo["b"],
                      imaginary=imaginary)


def _panel(n, R, cplx, precision, seed):
    """Sample vectors: random phases (complex) or signs (real), normalised."""
    gen = torch.Generator(device=DEV).manual_seed(seed * 104729 + 5)
    u = torch.rand(n, R, generator=gen, device=DEV, dtype=torch.float64)
    if cplx:
        x = torch.polar(torch.ones_like(u), 2 * math.pi * u)
        dt = torch.complex128 if precision == "f64" else torch.complex64
    else:
        x = torch.where(u < 0.5, -1.0, 1.0).double()
        dt = torch.float64 if precision == "f64" else torch.float32
    return (x / math.sqrt(n)).to(dt)


def _window(case):
    m = case.get("model", "silicon" if case["kind"] == "adjoint" else "diamond")
    return WINDOW["silicon" if m == "silicon_k" else m]


def _operator(case, geo, vals):
    pre = ISQRTMPreconditioner(_matrix(geo, vals["Z"])) if "Z" in vals else None
    c = Chebyshev(_matrix(geo, vals["H"]), *_window(case), preconditioner=pre)
    return c if case["precision"] == "f64" else c.astype("f32")


def _velocities(geo, vals):
    """Real parts W_a of V_a = i W_a: the bond moments at Gamma."""
    disp = torch.from_numpy(np.ascontiguousarray(geo["disp"])).to(DEV)
    return [vals["H"] * disp[:, a][:, None, None] for a in range(3)]


def _time_terms(n, t):
    """Chebyshev coefficients of a smooth propagator, n terms (t < n)."""
    k = 4 * n
    th = np.pi * (np.arange(k) + 0.5) / k
    f = np.exp(-1j * t * np.cos(th))
    c = 2.0 / k * (f[None, :] * np.cos(np.arange(n)[:, None] * th[None, :])).sum(1)
    c[0] *= 0.5
    return c


@functools.lru_cache(maxsize=None)
def _grid(nx=2000):
    return np.linspace(-0.995, 0.995, nx)


def _spd_batch(case, seed):
    """Ragged SPD batch A = Q diag(l) Q^T with condition numbers log-uniform in
    [1e2, 1e5]; returns sizes, offsets, A and the exact inverse square roots."""
    rng = np.random.default_rng(case["problems"])  # the sizes belong to the case
    n = np.sort(rng.integers(case["n_min"], case["n_max"] + 1, size=case["problems"]))
    rng = np.random.default_rng(seed)
    n = n.astype(np.int32)
    off = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)]).astype(np.int64)
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)
    A = torch.empty(int(off[-1]), dtype=torch.float64, device=DEV)
    parts = []
    for size in np.unique(n):
        idx = np.flatnonzero(n == size)
        m, c = int(size), idx.size
        G = torch.randn(c, m, m, dtype=torch.float64, device=DEV, generator=gen)
        for _ in range(3):  # Cholesky QR, repeated to orthogonality
            L = torch.linalg.cholesky_ex(G.transpose(1, 2) @ G)[0]
            G = torch.linalg.solve_triangular(L, G.transpose(1, 2), upper=False).transpose(1, 2)
        lk = torch.as_tensor(rng.uniform(np.log(1e2), np.log(1e5), size=c), device=DEV)[:, None]
        t = torch.linspace(0.0, 1.0, m, dtype=torch.float64, device=DEV)[None, :]
        lam = torch.exp(-lk + t * lk)
        M = (G * lam[:, None, :]) @ G.transpose(1, 2)
        A[off[idx[0]]:off[idx[-1] + 1]] = (0.5 * (M + M.transpose(1, 2))).reshape(-1)
        parts.append((G, lam))
    return n, off[:-1].copy(), A, parts


# ---------------------------------------------------------------- state, pass

def prepare(case, seed):
    kind = case["kind"]
    if kind == "isqrt":
        n, off, A, _ = _spd_batch(case, seed)
        return {"case": case, "n": n, "off": off, "A": A}
    geo, vals = _values(case, seed)
    st = {"case": case}
    N = geo["n"] * geo["b"]
    if kind == "adjoint":
        st["H"] = _matrix(geo, vals["H"])
        st["values"] = vals["H"].clone().requires_grad_(True)
        st["psi"] = _panel(N, case["R"], False, "f64", seed)
        st["x"] = _grid(400)
        st["target"] = 0.3 + 0.1 * np.cos(3 * st["x"] + seed)
        return st
    if kind == "solve":
        S = _matrix(geo, vals["S"])
        st["S"] = S if case["precision"] == "f64" else S.astype("f32")
        st["B"] = _panel(N, case["R"], False, case["precision"], seed)
        st["X"] = torch.empty_like(st["B"])
        return st
    st["op"] = _operator(case, geo, vals)
    cplx = case.get("complex", True)
    st["psi"] = _panel(N, case["R"], cplx, case["precision"], seed)
    if kind == "transport":
        V = [_matrix(geo, v, imaginary=True) for v in _velocities(geo, vals)]
        st["V"] = V if case["precision"] == "f64" else [v.astype("f32") for v in V]
    if kind in ("apply", "propagate"):
        st["out"] = torch.empty_like(st["psi"])
    if kind == "propagate":
        st["coeffs"] = _time_terms(case["terms"], 0.7 * case["terms"])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "apply":
        return st["op"].apply_op(st["psi"], st["out"])
    if kind == "propagate":
        return st["op"].propagate(st["psi"], st["out"], st["coeffs"])
    if kind == "dos":
        mu = kpm_dos_moments(st["op"], st["psi"], case["moments"])
        rho = evaluate_kpm_density(mu, _grid(), 1e-3, KpmKernel.Jackson)
        return {"mu": mu, "rho": rho}
    if kind == "transport":
        sigma, energy = dc_spectrum_fftcheb(
            st["op"], *st["V"], st["psi"], case["moments"],
            formulation=BASTIN if case["bastin"] else GREENWOOD)
        return {"sigma": sigma, "energy": energy}
    if kind == "isqrt":
        out, status, _ = inverse_sqrt_columns_batched(st["A"], st["n"], st["off"])
        return {"out": out, "status": status}
    if kind == "adjoint":
        st["values"].grad = None
        loss = KpmDosLoss.apply(st["values"], st["H"], st["psi"], *WINDOW["silicon"],
                                case["moments"], st["x"], st["target"])
        loss.backward()
        return {"loss": loss, "grad": st["values"].grad}
    st["X"].zero_()
    cg_solve(st["S"], st["B"], st["X"])
    return st["X"]


# ------------------------------------------------------------------- accounts

def work(case):
    kind = case["kind"]
    if kind == "isqrt":
        sizes = 0.5 * (case["n_min"] + case["n_max"])
        var = (case["n_max"] - case["n_min"]) ** 2 / 12.0
        n2, n3 = sizes ** 2 + var, sizes ** 3 + 3 * sizes * var
        # Eigenvalue-free count: ten Newton-Schulz steps of four products.
        return {"bytes": 16.0 * case["problems"] * n2, "flops": 80.0 * case["problems"] * n3}
    model = case.get("model", "silicon" if kind == "adjoint" else "diamond")
    geo = _geometry("silicon" if model == "silicon_k" else model, case["size"],
                    case.get("tiles", 1))
    nnz, b, N = geo["col_ind"].size, geo["b"], geo["n"] * geo["b"]
    s = 4 if case.get("precision") == "f32" else 8
    cm = model == "silicon_k"
    cv = case.get("complex", kind == "transport")
    mat = nnz * b * b * s * (2 if cm else 1) + 4 * (nnz + geo["n"])
    pan = N * case["R"] * s * (2 if cv else 1)
    fl = 2.0 * nnz * b * b * case["R"] * (4 if cm else 2 if cv else 1)
    forms = 3 if model == "diamond" and kind != "solve" else 1
    one = {"bytes": forms * mat + 2 * pan, "flops": forms * fl}
    if kind == "apply":
        return one
    if kind == "propagate":
        return {"bytes": forms * mat + case["terms"] * 3 * pan, "flops": case["terms"] * one["flops"]}
    if kind == "dos":
        k = (case["moments"] + 1) // 2
        return {"bytes": k * (forms * mat + 3 * pan), "flops": k * one["flops"]}
    if kind == "transport":
        # Per moment: one left step, three right ones, three currents, and the
        # two stores of three axes written and read.
        M = case["moments"]
        tf = 3 if case["bastin"] else 1
        fft = 6 * N * case["R"] * tf * 5.0 * 2 * M * math.log2(2 * M)
        return {"bytes": M * (4 * mat + 4 * 3 * pan + 2 * 6 * pan),
                "flops": M * 7 * fl + fft}
    if kind == "adjoint":
        M = case["moments"]
        return {"bytes": 4 * M * (mat + 3 * pan), "flops": 5 * M * fl}
    it = 20
    return {"bytes": it * (mat + 8 * pan), "flops": it * fl}


def tolerance(case):
    kind = case["kind"]
    f32 = case.get("precision") == "f32"
    if kind == "apply":
        return {"rel": 2e-6 if f32 else 4e-15}
    if kind == "propagate":  # rounding grows with the terms
        return {"rel": 8e-6 if f32 else 2e-14}
    if kind == "dos":
        return {"rel": 2e-6 if f32 else 2e-13}
    if kind == "transport":
        return {"rel": 8e-6 if f32 else 4e-13}
    if kind == "isqrt":  # split-TF32 phase, condition numbers to 1e5
        return {"rel": 1.5e-4}
    if kind == "adjoint":
        return {"rel": 1e-14}
    return {"rel": 2e-6 if f32 else 4e-8}  # solve: residual 1e-8


# ------------------------------------------------- FP64 restatement in torch

def _csr(geo, values):
    """The operator as a scalar FP64 (complex) sparse matrix."""
    b, n = geo["b"], geo["n"]
    r = torch.from_numpy(geo["rows"]).to(DEV)[:, None, None] * b
    c = torch.from_numpy(geo["col_ind"]).to(DEV).long()[:, None, None] * b
    k = torch.arange(b, device=DEV)
    idx = torch.stack([(r + k[None, :, None]).expand(-1, b, b).reshape(-1),
                       (c + k[None, None, :]).expand(-1, b, b).reshape(-1)])
    return torch.sparse_coo_tensor(idx, values.reshape(-1), (n * b, n * b)).coalesce().to_sparse_csr()


def _mm(A, X):
    if X.is_complex() and not A.is_complex():
        n, R = X.shape
        return torch.view_as_complex((A @ torch.view_as_real(X).reshape(n, 2 * R))
                                     .reshape(n, R, 2).contiguous())
    return A @ X


def _jackson(n):
    q = np.pi / (n + 1)
    i = np.arange(n)
    g = ((n + 1 - i) * np.cos(q * i) + np.sin(q * i) / np.tan(q)) / (n + 1)
    g[0] = 1.0
    return g


def exact(case, seed):
    kind = case["kind"]
    if kind == "isqrt":
        n, off, A, parts = _spd_batch(case, seed)
        out = [((G / lam.sqrt()[:, None, :]) @ G.transpose(1, 2)).reshape(-1) for G, lam in parts]
        return {"out": torch.cat(out), "status": np.zeros(n.size, np.int32)}
    geo, vals = _values(case, seed)
    prec = case.get("precision", "f64")
    up = (lambda v: v.float().double()) if prec == "f32" else (lambda v: v)
    H = _csr(geo, vals["H"] if vals["H"].is_complex() and prec == "f64" else
             vals["H"].to(torch.complex64).to(torch.complex128) if vals["H"].is_complex()
             else up(vals["H"]))
    N = geo["n"] * geo["b"]
    if kind == "solve":
        S = _csr(geo, up(vals["S"]))
        B = _panel(N, case["R"], False, prec, seed).double()
        X = torch.zeros_like(B)
        r = B.clone()
        p, rs = r.clone(), (r * r).sum(0)
        for _ in range(200):
            Sp = S @ p
            al = rs / (p * Sp).sum(0).clamp_min(1e-300)
            X += al * p
            r -= al * Sp
            new = (r * r).sum(0)
            if float(new.max()) < 1e-28:
                break
            p = r + new / rs.clamp_min(1e-300) * p
            rs = new
        return X
    emin, emax = _window(case)
    mid, hw = 0.5 * (emin + emax), 0.5 * (emax - emin)
    if "Z" in vals and kind != "adjoint":
        Z = _csr(geo, up(vals["Z"]))
        op = lambda X: (_mm(Z, _mm(H, _mm(Z, X))) - mid * X) / hw  # noqa: E731
    else:
        op = lambda X: (_mm(H, X) - mid * X) / hw  # noqa: E731
    cplx = case.get("complex", kind == "transport")
    psi = _panel(N, case["R"], cplx, prec, seed)
    psi = psi.to(torch.complex128) if cplx else psi.double()
    if kind == "apply":
        return op(psi)
    if kind == "propagate":
        c = _time_terms(case["terms"], 0.7 * case["terms"])
        if not cplx:
            c = c.real
        item = (lambda v: complex(v)) if cplx else (lambda v: float(v))
        t0, t1 = psi, op(psi)
        out = item(c[0]) * t0 + item(c[1]) * t1
        for k in range(2, case["terms"]):
            t0, t1 = t1, 2 * op(t1) - t0
            out += item(c[k]) * t1
        return out
    if kind == "dos":
        M = case["moments"]
        mu = _moments(op, psi, M)
        x = np.clip(_grid(), -1 + 1e-3, 1 - 1e-3)
        T = np.cos(np.arange(M)[None, :] * np.arccos(x)[:, None])
        w = _jackson(M) * mu.real * np.where(np.arange(M) == 0, 1.0, 2.0)
        return {"mu": mu, "rho": (T @ w) / (np.pi * np.sqrt(1 - x * x))}
    if kind == "transport":
        return _transport_exact(case, geo, vals, op, psi, mid, hw, up)
    return _adjoint_exact(case, seed, geo, op, psi, hw)


def _moments(op, psi, M):
    """Doubled recurrence: mu_2n = 2<t_n|t_n> - mu_0, mu_2n+1 = 2<t_n+1|t_n> - mu_1."""
    dot = lambda a, b: (a.conj() * b).sum() / psi.shape[1]  # noqa: E731
    mu = torch.zeros(M + 2, dtype=torch.complex128, device=DEV)
    t0, t1 = psi, op(psi)
    mu[0], mu[1] = dot(t0, t0), dot(t1, t0)
    n = 1
    while 2 * n < M:
        mu[2 * n] = 2 * dot(t1, t1) - mu[0]
        t0, t1 = t1, 2 * op(t1) - t0
        mu[2 * n + 1] = 2 * dot(t1, t0) - mu[1]
        n += 1
    return mu[:M].cpu().numpy()


def _transport_exact(case, geo, vals, op, psi, mid, hw, up):
    M, R, N = case["moments"], case["R"], psi.shape[0]
    V = [_csr(geo, up(v)) for v in _velocities(geo, vals)]
    cur = lambda a, X: (-1j / (2 * hw)) * _mm(V[a], X)  # noqa: E731
    g = torch.from_numpy(_jackson(M)).to(DEV)
    m = torch.arange(M, device=DEV, dtype=torch.float64)
    k = m + 0.5
    th = math.pi * m / (2 * M)
    half = torch.polar(torch.ones_like(th), th)
    eps, root = torch.cos(math.pi * k / M), torch.sin(math.pi * k / M)
    w3 = torch.where(m == 0, 1.0, 2.0) * g / math.pi
    pw = torch.where(m == 0, 1.0, 2.0) * g / math.pi * half

    def phi3(x):  # x_0 + 2 sum x_m cos(pi m (k + 1/2) / M)
        e = torch.fft.ifft(x * w3 * half, n=2 * M, dim=-1, norm="forward")
        return 0.5 * (e[..., :M] + torch.fft.ifft(x.conj() * w3 * half, n=2 * M, dim=-1,
                                                  norm="forward")[..., :M].conj())

    def phi(x, w):
        return torch.fft.ifft(x * w, n=2 * M, dim=-1, norm="forward")[..., :M]

    K = torch.zeros(M, 6, dtype=torch.complex128, device=DEV)
    comp = {(0, 0): 0, (0, 1): 1, (0, 2): 2, (1, 1): 3, (1, 2): 4, (2, 2): 5}
    rows = max(1, int(2e9 // (16 * 2 * M * 12)))
    group = max(1, int(4e10 // (16 * 6 * N * M)))  # samples held at once
    for s in range(0, R, group):
        l0 = psi[:, s:s + group].contiguous()
        w = l0.shape[1]
        left = torch.empty(3, N * w, M, dtype=torch.complex128, device=DEV)
        right = torch.empty_like(left)
        r0 = torch.cat([cur(a, l0) for a in range(3)], 1)
        l1, r1 = op(l0), op(r0)
        for n in range(M):
            for a in range(3):
                left[a, :, n] = cur(a, l0).reshape(-1)
                right[a, :, n] = r0[:, a * w:(a + 1) * w].reshape(-1)
            l0, l1 = l1, 2 * op(l1) - l0
            r0, r1 = r1, 2 * op(r1) - r0
        for q in range(0, N * w, rows):
            L, Rt = left[:, q:q + rows], right[:, q:q + rows]
            L3, R3 = phi3(L), phi3(Rt)
            if not case["bastin"]:
                for a in range(3):
                    K[:, comp[a, a]] += (L3[a].conj() * R3[a]).sum(0) / (1 - eps * eps).clamp_min(1e-14)
                continue
            L1, R1, L2, R2 = phi(L, pw), phi(Rt, pw), phi(L, pw * m), phi(Rt, pw * m)
            for (a, c), j in comp.items():
                t = L3[a].conj() * R1[c] + L1[a].conj() * R3[c]
                u = L2[a].conj() * R3[c] - L3[a].conj() * R2[c]
                K[:, j] += (eps * t + 1j * root * u).sum(0)
        del left, right
    K = (K / R).flip(0)
    e = eps.flip(0)
    if case["bastin"]:
        f = -K.imag
        trap = 0.5 * (f[1:] + f[:-1]) * (e[1:] - e[:-1])[:, None]
        sigma = torch.cat([torch.zeros(1, 6, dtype=torch.float64, device=DEV), trap.cumsum(0)])
    else:
        sigma = K.real
    return {"sigma": sigma, "energy": mid + hw * e}


def _adjoint_exact(case, seed, geo, op, psi, hw):
    M, R, b = case["moments"], case["R"], geo["b"]
    x = _grid(400)
    target = 0.3 + 0.1 * np.cos(3 * x + seed)
    n = np.arange(M)
    D = 2.0 * np.cos(n[None, :] * np.arccos(x)[:, None]) * (np.where(n == 0, 1.0, 2.0) * _jackson(M))
    D /= (np.pi * np.sqrt(1 - x * x))[:, None]
    t = [psi, op(psi)]
    for _ in range(2, M):
        t.append(2 * op(t[-1]) - t[-2])
    mu = torch.stack([(psi * v).sum() / R for v in t[:M]]).cpu().numpy()
    resid = D @ mu - target
    dmu = 2.0 * (resid @ D)
    lam2, lam1 = torch.zeros_like(psi), torch.zeros_like(psi)
    r = torch.from_numpy(geo["rows"]).to(DEV)
    c = torch.from_numpy(geo["col_ind"]).to(DEV).long()
    grad = torch.zeros(c.numel(), b, b, dtype=torch.float64, device=DEV)
    blocks = lambda v: v.reshape(-1, b, R)  # noqa: E731
    for k in range(M - 1, 0, -1):  # lambda_k, then lambda_k t_{k-1}^T
        lam = dmu[k] / R * psi + 2 * op(lam1) - lam2
        lam2, lam1 = lam1, lam
        grad += (1.0 if k == 1 else 2.0) * blocks(lam)[r] @ blocks(t[k - 1])[c].transpose(1, 2)
    return {"loss": torch.tensor(resid @ resid, dtype=torch.float64), "grad": grad / hw}
