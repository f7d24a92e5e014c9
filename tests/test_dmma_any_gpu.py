"""The any-shape FP64 tensor-core step (cheb_dmma_any.cuh), forced, at the edges
of its tiling: every block size it takes, widths around its column groups and
chunks, rows with no block and with more blocks than a load group, real,
complex and imaginary-unit values, FP64 and FP32 panels, against dense products;
and its fused column dots against the default kernels' moments."""
from __future__ import annotations

import numpy as np
import pytest

from _util import random_hermitian_bsr, rel_err

pytestmark = pytest.mark.gpu

KINDS = [("real", False, False, False), ("complex", True, False, True),
         ("imaginary", False, True, True), ("real_cplx_panel", False, False, True)]


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    torch.cuda.set_device(0)
    return torch


def _ragged(n, b, cm, seed):
    """Block rows of 0 to 11 blocks."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, 12, n)
    deg[:3] = 0, 1, 11
    ci = np.concatenate([np.sort(rng.permutation(n)[:d]) for d in deg]).astype(np.int32)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    v = rng.standard_normal((ci.size, b, b))
    if cm:
        v = v + 1j * rng.standard_normal(v.shape)
    A = np.zeros((n * b, n * b), dtype=v.dtype)
    for i in range(n):
        for k in range(rp[i], rp[i + 1]):
            A[i * b:(i + 1) * b, ci[k] * b:(ci[k] + 1) * b] = v[k]
    return rp, ci, v, A


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind", KINDS, ids=[k[0] for k in KINDS])
@pytest.mark.parametrize("b", [2, 3, 4, 5, 6, 7, 8])
def test_products_at_every_width(torch_cuda, monkeypatch, b, kind, precision):
    torch = torch_cuda
    from rsatb_b200.vbcsr import BlockSpMat
    _, cm, imag, cv = kind
    n = 23
    rp, ci, v, A = _ragged(n, b, cm, seed=b)
    M = BlockSpMat(rp, ci, v, b, n, imaginary=imag)
    if precision == "f32":
        M = M.astype("f32")
        A = A.astype(np.complex64 if cm else np.float32).astype(A.dtype)
    if imag:
        A = 1j * A
    dt = {("f64", True): torch.complex128, ("f64", False): torch.float64,
          ("f32", True): torch.complex64, ("f32", False): torch.float32}[(precision, cv)]
    monkeypatch.setenv("RSATB_STEP_KERNEL", "dmma_any")
    rng = np.random.default_rng(b)
    widths = [1, 2, 7, 8, 9, 16, 17, 24, 33, 48, 63, 64, 65, 127, 128]
    if not cv:
        widths += [129, 255, 256]
    for R in widths:
        X = rng.standard_normal((n * b, R))
        if cv:
            X = X + 1j * rng.standard_normal((n * b, R))
        Xd = torch.as_tensor(X).cuda().to(dt).contiguous()
        Yd = torch.full_like(Xd, float("nan"))
        M.mult_dense(Xd, Yd, alpha=0.5)
        want = 0.5 * (A @ Xd.cpu().numpy().astype(np.complex128 if cv else np.float64))
        # products and sums in FP64 whatever the panel, one rounding at the store
        tol = 1e-14 if precision == "f64" else 2e-7
        assert rel_err(Yd.cpu().numpy(), want) < tol, R
        assert np.all(Yd.cpu().numpy()[:b] == 0)  # the empty row


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("b,cm,R", [(5, True, 6), (5, False, 32), (5, False, 33), (8, False, 7),
                                    (8, False, 45), (3, False, 20), (4, True, 9), (8, True, 3),
                                    (2, False, 1)])
def test_dots_equal_the_register_kernel(torch_cuda, monkeypatch, b, cm, R, precision):
    """The doubled and the plain recurrence through both kernels."""
    torch = torch_cuda
    from rsatb_b200.calc import Chebyshev, kpm_dos_moments, kpm_dos_moments_plain
    from rsatb_b200.vbcsr import BlockSpMat
    n = 301
    A = random_hermitian_bsr(n, b, 4, seed=b + R, complex_values=cm, scale=0.3)
    M = BlockSpMat(A.row_ptr, A.col_ind, A.values, b, A.n_block_cols)
    M = M.astype("f32") if precision == "f32" else M
    bound = 1.5 * np.abs(A.to_dense()).sum(1).max()
    c = Chebyshev(M, -bound, bound)
    rng = np.random.default_rng(R)
    X = rng.choice([-1.0, 1.0], (n * b, R)) / np.sqrt(n * b)
    dt = {("f64", True): torch.complex128, ("f64", False): torch.float64,
          ("f32", True): torch.complex64, ("f32", False): torch.float32}[(precision, cm)]
    Xd = torch.as_tensor(X).cuda().to(dt).contiguous()
    got = {}
    for k in ("generic", "dmma_any"):
        monkeypatch.setenv("RSATB_STEP_KERNEL", k)
        got[k] = np.stack([kpm_dos_moments(c, Xd, 12), kpm_dos_moments_plain(c, Xd, 12)])
    tol = 1e-13 if precision == "f64" else 1e-5
    assert np.abs(got["generic"] - got["dmma_any"]).max() < tol * abs(got["generic"][0, 0])
