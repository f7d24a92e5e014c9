"""The arithmetic of the fused Greenwood row stage (fftcheb.cu, fused_transform)
replayed on the host for its four moment counts: the M-point input of the
DCT-III, the 16 x 16 x r plan with its exchange slots, the 4 x 4 16-point DFT with
its output order, the 2-, 4- and 8-point last pass, the factors formed from the
quarter table or read from the pass-B table, and the order of the outputs,
against the oracle's DCT-III (RowFFTWorkspace::dct_type3_batch,
rsatb/calc/fft.hpp:125-154).  The CUDA kernel itself is checked against the cuFFT
stage and the oracle, at every one of these counts, in test_transport_gpu.py."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

C8, S8, R2 = np.cos(np.pi / 8), np.sin(np.pi / 8), np.cos(np.pi / 4)
# v[j0 + 4 c] *= e^{2 pi i j0 c / 16} between the two radix-4 passes
INNER = {5: C8 + 1j * S8, 6: R2 + 1j * R2, 7: S8 + 1j * C8, 9: R2 + 1j * R2, 10: 1j,
         11: -R2 + 1j * R2, 13: S8 + 1j * C8, 14: -R2 + 1j * R2, 15: -C8 - 1j * S8}


def _energy(M, p):
    return np.where(p < (M + 1) // 2, 2 * p, 2 * (M - 1 - p) + 1)


def _dft4(a0, a1, a2, a3):
    s02, d02 = a0 + a2, a0 - a2
    s13, d13 = a1 + a3, 1j * (a1 - a3)
    return s02 + s13, d02 + d13, s02 - s13, d02 - d13


def _dft16(v):
    """dft16_inv on columns v[:, 0..15]; output k lands in column _at(k)."""
    v = v.copy()
    for j0 in range(4):
        v[:, j0], v[:, j0 + 4], v[:, j0 + 8], v[:, j0 + 12] = _dft4(
            v[:, j0], v[:, j0 + 4], v[:, j0 + 8], v[:, j0 + 12])
    for i, f in INNER.items():
        v[:, i] *= f
    for c in range(4):
        v[:, 4 * c], v[:, 4 * c + 1], v[:, 4 * c + 2], v[:, 4 * c + 3] = _dft4(
            v[:, 4 * c], v[:, 4 * c + 1], v[:, 4 * c + 2], v[:, 4 * c + 3])
    return v


def _at(k):
    return 4 * (k % 4) + k // 4


def _dft_r(u):
    """dft_r_inv: r = 1, 2, 4, 8 columns, natural order."""
    r = len(u)
    if r == 1:
        return u
    if r == 2:
        return [u[0] + u[1], u[0] - u[1]]
    if r == 4:
        return list(_dft4(*u))
    e, o = _dft4(u[0], u[2], u[4], u[6]), list(_dft4(u[1], u[3], u[5], u[7]))
    for k, f in ((1, R2 + 1j * R2), (2, 1j), (3, -R2 + 1j * R2)):
        o[k] = o[k] * f
    return [e[k] + o[k] for k in range(4)] + [e[k] - o[k] for k in range(4)]


def _twiddle(M, n):
    """twiddle: w^n from the quarter table w^j, j < M / 4."""
    q = np.exp(2j * np.pi * np.arange(M // 4) / M)
    return q[n % (M // 4)] * 1j ** ((n // (M // 4)) & 3)


def _pow16(b, b4):
    """Pow16: b^k, k = 0..15, as b4^(k // 4) b^(k % 4)."""
    lo = [np.ones_like(b), b, b * b]
    lo.append(lo[2] * b)
    hi = [np.ones_like(b), b4, b4 * b4]
    hi.append(hi[2] * b4)
    return np.stack([hi[k // 4] * lo[k % 4] for k in range(16)], axis=1)


def _write(size, slots, values):
    buf = np.full(size, np.nan, dtype=complex)
    flat = np.concatenate(slots)
    assert np.unique(flat).size == flat.size and 0 <= flat.min() and flat.max() < size
    for s, v in zip(slots, values):
        buf[s] = v
    return buf


@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_mpoint_plan_is_the_dct3(r):
    M, TPS = 256 * r, 16 * r
    size = 16 * 17 * r  # fused_xch
    rng = np.random.default_rng(r)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    w = rng.random(M)
    ph = w * np.exp(1j * np.pi * np.arange(M) / (2 * M))
    t = np.arange(TPS)
    # pass A
    n = t[:, None] + TPS * np.arange(16)[None, :]
    mirror = np.where(n > 0, M - n, 0)
    F = ph[n] * x[n] + np.where(n > 0, np.conj(ph[mirror]) * x[mirror], 0)
    v = _dft16(F)
    tw = _pow16(_twiddle(M, t), _twiddle(M, 4 * t))
    buf = _write(size, [k0 * 17 * r + t for k0 in range(16)],
                 [v[:, _at(k0)] * tw[:, k0] for k0 in range(16)])
    # pass B
    n0, k0 = t % r, t // r
    v = _dft16(np.stack([buf[k0 * 17 * r + n0 + r * n1] for n1 in range(16)], 1))
    e = np.arange(17 * r)
    wb = np.exp(2j * np.pi * (e // 17) * (e % 17) / (16 * r))  # the pass-B table
    buf = _write(size, [k1 * (16 * r + 1) + t for k1 in range(16)],
                 [v[:, _at(k1)] * (wb[n0 * 17 + k1] if r > 1 and k1 else 1) for k1 in range(16)])
    # pass C
    out = np.full(M, np.nan, dtype=complex)
    for j in range(16 // r):
        pi = t + TPS * j
        k1, k0 = pi & 15, pi >> 4
        u = _dft_r([buf[k1 * (16 * r + 1) + k0 * r + q] for q in range(r)])
        for q in range(r):
            out[k0 + 16 * k1 + 256 * q] = u[q]
    y = np.empty(M, dtype=complex)
    y[_energy(M, np.arange(M))] = out
    want = oracle.dct3((w * x)[None, :])[0]
    assert np.abs(y - want).max() <= 1e-12 * np.abs(want).max()


def test_dft16_output_order():
    rng = np.random.default_rng(3)
    z = rng.standard_normal((4, 16)) + 1j * rng.standard_normal((4, 16))
    d = _dft16(z)
    want = np.fft.ifft(z, axis=1) * 16
    assert np.allclose(np.stack([d[:, _at(k)] for k in range(16)], axis=1), want,
                       rtol=0, atol=1e-13)


@pytest.mark.parametrize("M", [1, 2, 3, 8, 17, 100])
def test_mpoint_input_is_the_dct3_at_any_length(M):
    """dct3_input_kernel's sequence and output order, odd lengths among them."""
    rng = np.random.default_rng(M)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    m = np.arange(M)
    z = np.where(m > 0, x[-m], 0)
    F = np.exp(1j * np.pi * m / (2 * M)) * (x - 1j * z)
    y = np.empty(M, dtype=complex)
    y[_energy(M, m)] = np.fft.ifft(F) * M
    assert np.abs(y - oracle.dct3(x)).max() <= 1e-12 * np.abs(y).max()
