"""The index arithmetic of the fused Greenwood row stage (fftcheb.cu,
fused_transform) replayed on the host for its four moment counts: the M-point
input of the DCT-III, the 16 x 16 x r plan with its exchange strides, and the
order of its outputs, against the oracle's DCT-III
(RowFFTWorkspace::dct_type3_batch, rsatb/calc/fft.hpp:125-154).  The CUDA kernel
itself is checked against the cuFFT stage and the oracle in
test_transport_gpu.py."""
from __future__ import annotations

import numpy as np
import pytest

import oracle


def _energy(M, p):
    return np.where(p < (M + 1) // 2, 2 * p, 2 * (M - 1 - p) + 1)


def _dft(v):
    n = v.shape[1]
    k = np.arange(n)
    return v @ np.exp(2j * np.pi * np.outer(k, k) / n)


@pytest.mark.parametrize("r", [1, 2, 4, 8])
def test_mpoint_plan_is_the_dct3(r):
    M, TPS = 256 * r, 16 * r
    rng = np.random.default_rng(r)
    x = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    ph = np.exp(1j * np.pi * np.arange(M) / (2 * M))
    w = np.exp(2j * np.pi / M)
    t = np.arange(TPS)
    # pass A
    n = t[:, None] + TPS * np.arange(16)[None, :]
    mirror = np.where(n > 0, M - n, 0)
    F = ph[n] * x[n] + np.where(n > 0, np.conj(ph[mirror]) * x[mirror], 0)
    v = _dft(F) * w ** (t[:, None] * np.arange(16)[None, :])
    buf = np.full(16 * 17 * r, np.nan, dtype=complex)
    for k0 in range(16):
        buf[k0 * 17 * r + t] = v[:, k0]
    # pass B
    n0, k0 = t % r, t // r
    v = np.stack([buf[k0 * 17 * r + n0 + r * n1] for n1 in range(16)], 1)
    v = _dft(v) * w ** (16 * n0[:, None] * np.arange(16)[None, :])
    buf[:] = np.nan
    for k1 in range(16):
        buf[k1 * (16 * r + 1) + t] = v[:, k1]
    # pass C
    out = np.full(M, np.nan, dtype=complex)
    for j in range(16 // r):
        pi = t + TPS * j
        k1, k0 = pi & 15, pi >> 4
        u = _dft(np.stack([buf[k1 * (16 * r + 1) + k0 * r + q] for q in range(r)], 1))
        for q in range(r):
            out[k0 + 16 * k1 + 256 * q] = u[:, q]
    y = np.empty(M, dtype=complex)
    y[_energy(M, np.arange(M))] = out
    assert np.abs(y - oracle.dct3(x)).max() <= 1e-12 * np.abs(y).max()


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
