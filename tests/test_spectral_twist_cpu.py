"""The z passes' twisted transform of length L >= nz (CPU, numpy).

* Modulo (z^L + i) the linear convolution of nz points wraps into the imaginary
  part, so the real part is the convolution itself, and the conjugate spectrum
  gives the correlation; the stencil folds as o >= 0 -> real part at o, o < 0 ->
  imaginary part at L + o.
* The 16 x N2 schedule with the twist split between constants of the 16-point
  stage and the twiddle exp(-2 pi i n2 (4 k1 + 1) / (4 L)) is that transform,
  and its inverse undoes it.
* The exchange holds every element once, in both layouts, and the accesses of 16
  lanes meant to be free of bank conflicts are.
"""
import numpy as np
import pytest

N2S = (3, 4, 5, 6, 8, 9, 10, 12, 15, 16, 18, 20, 24, 27, 32)


def _forward(x, n2s):
    L = 16 * n2s
    n1, n2 = np.arange(16)[:, None], np.arange(n2s)[None, :]
    v = x[n2s * n1 + n2] * np.exp(-2j * np.pi * n1 / 64)
    v = np.fft.fft(v, axis=0) * np.exp(-2j * np.pi * n2 * (4 * n1 + 1) / (4 * L))
    out = np.empty(L, complex)
    out[n1 + 16 * n2] = np.fft.fft(v, axis=1)
    return out


def _inverse(X, n2s):
    L = 16 * n2s
    n1, n2 = np.arange(16)[:, None], np.arange(n2s)[None, :]
    z = np.fft.ifft(X[n1 + 16 * n2], axis=1) * n2s * np.exp(2j * np.pi * n2 * (4 * n1 + 1) / (4 * L))
    y = np.fft.ifft(z, axis=0) * 16
    out = np.empty(L)
    out[n2s * n1 + n2] = (y * np.exp(2j * np.pi * n1 / 64)).real
    return out


@pytest.mark.parametrize("n2s", N2S)
def test_twisted_convolution(n2s):
    L = 16 * n2s
    rng = np.random.default_rng(n2s)
    for nz in (1, 7, L - 15, L - 1, L):
        T, S = rng.standard_normal(nz), rng.standard_normal(2 * nz - 1)      # S[o + nz - 1]
        x = np.zeros(L)
        x[:nz] = T
        fold = np.zeros(L, complex)
        o = np.arange(-(nz - 1), nz)
        np.add.at(fold, np.where(o < 0, L + o, o), np.where(o < 0, 1j, 1.0) * S)
        tq = np.exp(-2j * np.pi * np.arange(L) / (4 * L))
        Sh = np.fft.fft(fold * tq) / L
        F = _forward(x, n2s)
        assert np.abs(F - np.fft.fft(x * tq)).max() <= 1e-12 * max(1.0, np.abs(F).max())
        full = np.convolve(T, S)
        assert np.abs(_inverse(F * Sh, n2s)[:nz] - full[nz - 1:2 * nz - 1]).max() <= 1e-11 * np.abs(full).max()
        corr = np.convolve(T, S[::-1])
        assert np.abs(_inverse(F * Sh.conj(), n2s)[:nz] - corr[nz - 1:2 * nz - 1]).max() <= 1e-11 * np.abs(corr).max()


@pytest.mark.parametrize("plane", [False, True])
@pytest.mark.parametrize("n2s", N2S)
def test_exchange_layout(n2s, plane):
    pitch = 17 * n2s + (1 if plane and n2s % 2 == 0 else 0)
    slot = lambda r, c: c * pitch + r + r // 16  # noqa: E731
    r, c = np.meshgrid(np.arange(16 * n2s), np.arange(16))
    slots = slot(r, c).ravel()
    assert len(set(slots.tolist())) == slots.size and slots.max() < 16 * pitch
    lanes = np.arange(16)
    for n2 in range(n2s):
        if plane:       # 16 lanes across the lines
            assert len(set((slot(16 * n2 + 3, lanes) % 16).tolist())) == 16
        else:           # 16 lanes at consecutive k1
            assert len(set((slot(16 * n2 + lanes, 5) % 16).tolist())) == 16
    if n2s >= 16:       # 16 lanes at consecutive n2
        assert len(set((slot(16 * lanes + 3, 5) % 16).tolist())) == 16
