"""The z, y and x passes of the spectral cone stage and the transform that builds
S^ (spectral_z.cu, spectral_y.cu, spectral_x.cu), restated block by block and
thread by thread (CPU).

Threads of a block act stage by stage, numpy's DFT in the place of the short
ones.  Checked on the way: every exchange slot is written once per stage, lies
inside the block's shared memory and is written before it is read; global rows
are read inside their array and only where written (memory starts as NaN); rows
without TERMA are neither written nor read where the y pass goes by the flags;
rows asked for ahead lie inside the work arrays.  The five passes and the plane
layout together are the linear convolution, and its correlation with conj(S^).
"""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "conehead_gb300", "csrc")


def _src(name):
    return open(os.path.join(CSRC, name)).read()


N2S = [int(n) for n in re.findall(r"X\((\d+)\)", re.search(r"#define SPEC_N2\(X\)(.*)", _src("spectral_16n.cuh")).group(1))]
AHEAD = int(re.search(r"SPEC_AHEAD = (\d+)", _src("spectral_16n.cuh")).group(1))


def _threads(n2s):
    return max(16 * n2s, 256)


def _length(n):
    return next(16 * m for m in N2S if 16 * m >= n)


class Shared:
    """One block's exchange: `size` float2 slots."""

    def __init__(self, size):
        self.v = np.full(size, np.nan + 0j)

    def write(self, slots, values):
        flat = np.asarray(slots).ravel()
        assert flat.min() >= 0 and flat.max() < self.v.size and np.unique(flat).size == flat.size
        self.v[flat] = np.asarray(values).ravel()

    def read(self, slots):
        out = self.v[np.asarray(slots)]
        assert not np.isnan(out).any()
        return out


def _dft(v, axis, inv):
    return np.fft.ifft(v, axis=axis) * v.shape[axis] if inv else np.fft.fft(v, axis=axis)


def _twiddle(M, k):
    return np.exp(-2j * np.pi * np.asarray(k) / M)


# ------------------------------------------------------------------ z passes --
def _z_slot(n2s, plane):
    pitch = 17 * n2s + (1 if plane and n2s % 2 == 0 else 0)
    return (lambda r, c: c * pitch + r + (r >> 4)), 16 * pitch


def _z_forward(n2s, plane, nl, nz, T, flags, skip, A, lp):
    L = 16 * n2s
    slot, size = _z_slot(n2s, plane)
    t = np.arange(16 * n2s)
    n2, c = t % n2s, t // n2s
    tw = _twiddle(4 * L, (np.arange(L) % n2s) * (4 * (np.arange(L) // n2s) + 1))       # at m N2 + n2
    for l0 in range(0, nl, 16):
        live = np.array([l0 + i < nl and bool(flags[min(l0 + i, nl - 1)]) for i in range(16)])
        lines = min(16, nl - l0)
        if not live.any():
            if skip:
                continue
            if plane:                                      # 16-byte stores of two: past nl into the pitch
                assert l0 + 16 <= lp
                A[:, l0:l0 + 16] = 0
            else:
                A[l0:l0 + lines] = 0
            continue
        v = np.zeros((16, t.size), complex)
        for n1 in range(16):
            z = n2s * n1 + n2
            ok = live[c] & (z < nz)
            v[n1, ok] = T[l0 + c[ok], z[ok]]
        assert not np.isnan(v).any()
        v *= _twiddle(64, np.arange(16))[:, None]
        v = _dft(v, 0, False)
        sm = Shared(size)
        m = np.arange(16)[:, None]
        sm.write(slot(16 * n2[None] + m, c[None]), v * tw[m * n2s + n2[None]])
        u = np.arange(256)
        lo, hi = u & 15, u >> 4
        k1, cc = (hi, lo) if plane else (lo, hi)
        j = np.arange(n2s)[:, None]
        a = _dft(sm.read(slot(16 * j + k1[None], cc[None])), 0, False)
        ok = l0 + cc < nl
        for k2 in range(n2s):
            k = k1 + 16 * k2
            if plane:
                A[k[ok], l0 + cc[ok]] = a[k2, ok]
            else:
                A[l0 + cc[ok], k[ok]] = a[k2, ok]


def _z_inverse(n2s, plane, nl, nz, A, D):
    L = 16 * n2s
    slot, size = _z_slot(n2s, plane)
    u = np.arange(256)
    lo, hi = u & 15, u >> 4
    k1, cc = (hi, lo) if plane else (lo, hi)
    tw = _twiddle(4 * L, (np.arange(L) >> 4) * (4 * (np.arange(L) & 15) + 1)).conj()      # at 16 n2 + k1
    t = np.arange(16 * n2s)
    n2, c = t % n2s, t // n2s
    for l0 in range(0, nl, 16):
        ok = l0 + cc < nl
        a = np.zeros((n2s, 256), complex)
        for k2 in range(n2s):
            k = k1 + 16 * k2
            a[k2, ok] = A[k[ok], l0 + cc[ok]] if plane else A[l0 + cc[ok], k[ok]]
        assert not np.isnan(a).any()
        a = _dft(a, 0, True)
        j = np.arange(n2s)[:, None]
        sm = Shared(size)
        sm.write(slot(16 * j + k1[None], cc[None]), a * tw[16 * j + k1[None]])
        q = np.arange(16)[:, None]
        v = _dft(sm.read(slot(16 * n2[None] + q, c[None])), 0, True) * _twiddle(64, q).conj()
        for m in range(16):
            z = n2 + n2s * m
            w = (l0 + c < nl) & (z < nz)
            assert np.isnan(D[l0 + c[w], z[w]]).all()
            D[l0 + c[w], z[w]] = v[m, w].real


# -------------------------------------------------------------- y and x passes --
def _chain_slots(n2s):
    """Slots of the exchange of the y and x passes: row r at 16 r + line."""
    return lambda r, c: 16 * r + c


def _columns(n2s, rows, live):
    """Forward stages 1 and 2: rows(n) reads row n of the 16 lines; returns {(k1, c): a[k2]}."""
    slot = _chain_slots(n2s)
    t = np.arange(16 * n2s)
    c, h = t & 15, t >> 4
    v = np.zeros((16, t.size), complex)
    for n1 in range(8):
        n = n2s * n1 + h
        ok = live(n)
        v[n1, ok] = rows(n[ok], c[ok])
    assert not np.isnan(v).any()
    v = _dft(v, 0, False)
    m = np.arange(16)[:, None]
    sm = Shared(16 * n2s * 16)
    sm.write(slot(m * n2s + h[None], c[None]), v * _twiddle(16 * n2s, h[None] * m))
    u = np.arange(256)
    cc, k1 = u & 15, u >> 4
    j = np.arange(n2s)[:, None]
    return sm, _dft(sm.read(slot(k1[None] * n2s + j, cc[None])), 0, False), cc, k1


def _back(n2s, a, cc, k1, write):
    """Inverse stages A and B from a[k2] of threads (c, k1)."""
    slot = _chain_slots(n2s)
    j = np.arange(n2s)[:, None]
    sm = Shared(16 * n2s * 16)
    sm.write(slot(j * 16 + k1[None], cc[None]), _dft(a, 0, True) * _twiddle(16 * n2s, j * k1[None]).conj())
    t = np.arange(16 * n2s)
    c, h = t & 15, t >> 4
    q = np.arange(16)[:, None]
    v = _dft(sm.read(slot(h[None] * 16 + q, c[None])), 0, True)
    for m in range(8):
        write(h + n2s * m, c, v[m])


def _y_pass(n2s, inv, n0, ny, L, A, B, flags):
    """A [n0][ny][L], B [n0][M][L]; flags None: every row is read."""
    M, nkb = 16 * n2s, L // 16
    for blk in range(n0 * nkb):
        x, kz0 = blk // nkb, (blk % nkb) * 16
        nxt = blk + AHEAD
        if nxt < n0 * nkb:                                  # rows asked for, one per thread
            x2, row = nxt // nkb, np.arange(_threads(n2s))
            row = row[row < (M if inv else ny)]
            assert x2 < n0 and row.max() < (B if inv else A).shape[1] and (nxt % nkb) * 16 + 16 <= L
        if not inv:
            lines = None if flags is None else flags[x * ny:(x + 1) * ny]
            _, a, cc, k1 = _columns(n2s, lambda n, c: A[x, n, kz0 + c],
                                    lambda n: (n < ny) & (True if lines is None else lines[np.minimum(n, ny - 1)] != 0))
            for k2 in range(n2s):
                B[x, k1 + 16 * k2, kz0 + cc] = a[k2]
        else:
            u = np.arange(256)
            cc, k1 = u & 15, u >> 4
            a = np.stack([B[x, k1 + 16 * k2, kz0 + cc] for k2 in range(n2s)])
            assert not np.isnan(a).any()

            def write(y, c, v):
                ok = y < ny
                A[x, y[ok], kz0 + c[ok]] = v[ok]
            _back(n2s, a, cc, k1, write)


def _x_pass(n2s, nx, My, L, B, S, conj, beams=1):
    nkb = L // 16
    for blk in range(My * nkb):
        ky, kz0 = blk // nkb, (blk % nkb) * 16
        nxt = blk * beams + AHEAD
        if nxt < My * nkb * beams:
            blk2 = nxt // beams
            assert blk2 // nkb < My and (blk2 % nkb) * 16 + 16 <= L and 0 <= nxt - blk2 * beams < beams
        sm, a, cc, k1 = _columns(n2s, lambda n, c: B[n, ky, kz0 + c], lambda n: n < nx)
        for k2 in range(n2s):
            s = S[k1 + 16 * k2, ky, kz0 + cc]
            a[k2] *= s.conj() if conj else s

        def write(x, c, v):
            ok = x < nx
            B[x[ok], ky, kz0 + c[ok]] = v[ok]
        _back(n2s, a, cc, k1, write)


def _full(n2s, data, outer, cs, step, twist):
    """spec_full_kernel on the flat array `data`: `outer` the first elements of the blocks."""
    M = 16 * n2s
    along = step == 1
    sc, sn, sk = (17 * n2s, 17, 1) if along else (1, 16, 16 * n2s)
    t, u = np.arange(16 * n2s), np.arange(256)
    n2, c = (t % n2s, t // n2s) if along else (t >> 4, t & 15)
    k1, cc = (u & 15, u >> 4) if along else (u >> 4, u & 15)
    seen = np.zeros(data.size, int)
    for o in outer:
        i = n2s * np.arange(16)[:, None] + n2[None]
        v = data[o + c[None] * cs + i * step]
        if twist:
            v = v * _twiddle(4 * M, i)
        m = np.arange(16)[:, None]
        sm = Shared(16 * 17 * n2s)
        sm.write(m * sk + n2[None] * sn + c[None] * sc, _dft(v, 0, False) * _twiddle(M, n2[None] * m))
        j = np.arange(n2s)[:, None]
        a = _dft(sm.read(k1[None] * sk + j * sn + cc[None] * sc), 0, False)
        at = o + cc[None] * cs + (k1[None] + 16 * j) * step
        seen[at] += 1
        data[at] = a
    assert (seen == 1).all()


def _build(S, n, M):
    """S^ of the stencil S[o + n - 1], folded as spec_shat does, by three transforms in place."""
    F = np.zeros(M, complex)
    for iz in range(2 * n[2] - 1):
        oz = iz - (n[2] - 1)
        part = np.zeros(M[:2])
        ox, oy = np.arange(-(n[0] - 1), n[0]), np.arange(-(n[1] - 1), n[1])
        part[np.ix_(ox % M[0], oy % M[1])] = S[:, :, iz]
        F[:, :, oz if oz >= 0 else M[2] + oz] += part * (1 if oz >= 0 else 1j)
    flat = F.ravel()
    Mx, My, L = M
    nb = L // 16
    _full(L // 16, flat, [o * 16 * L for o in range(Mx * My // 16)], L, 1, True)
    _full(My // 16, flat, [(o // nb) * My * L + (o % nb) * 16 for o in range(Mx * nb)], 1, L, False)
    _full(Mx // 16, flat, [(o // nb) * L + (o % nb) * 16 for o in range(My * nb)], 1, My * L, False)
    return flat.reshape(M) / np.prod(M)


def _case(n, seed, part):
    rng = np.random.default_rng(seed)
    T = rng.standard_normal(n)
    flags = (rng.random(n[0] * n[1]) < part).astype(np.uint8)
    flags[: 5 * n[1]] = 0                                   # whole blocks without TERMA
    flags[-1] = 1
    T.reshape(-1, n[2])[flags == 0] = 0
    S = rng.standard_normal([2 * k - 1 for k in n])
    size = [4 * k for k in n]
    conv = np.fft.ifftn(np.fft.fftn(T, size, range(3)) * np.fft.fftn(S, size, range(3))).real
    corr = np.fft.ifftn(np.fft.fftn(T, size, range(3)) * np.fft.fftn(S[::-1, ::-1, ::-1], size, range(3))).real
    cut = tuple(slice(k - 1, 2 * k - 1) for k in n)
    zp = -(-n[2] // 4) * 4
    Tp = np.full((n[0] * n[1], zp), np.nan)                 # lines without TERMA and the pitch are never read
    Tp[flags != 0, :n[2]] = T.reshape(-1, n[2])[flags != 0]
    return Tp, flags, S, conv[cut], corr[cut]


@pytest.mark.parametrize("n,part,use_flags", [((9, 31, 41), 0.4, True), ((24, 20, 49), 0.7, True),
                                              ((25, 33, 70), 0.5, False), ((12, 40, 1), 0.6, True)])
def test_five_passes(n, part, use_flags):
    T, flags, S, conv, corr = _case(n, sum(n), part)
    M = (_length(2 * n[0] - 1), _length(2 * n[1] - 1), _length(n[2]))
    Sh = _build(S, n, M)
    nl = n[0] * n[1]
    if not use_flags:                                       # the cone operator: every line is read
        T[flags == 0, :n[2]] = 0
        flags = np.ones(nl, np.uint8)
    for conj, ref in ((False, conv), (True, corr)):
        A = np.full((nl, M[2]), np.nan + 0j)
        B = np.full((n[0], M[1], M[2]), np.nan + 0j)
        D = np.full((nl, n[2]), np.nan)
        _z_forward(M[2] // 16, False, nl, n[2], T, flags, True, A, 0)
        A3 = A.reshape(n[0], n[1], M[2])
        _y_pass(M[1] // 16, False, n[0], n[1], M[2], A3, B, flags if use_flags else None)
        _x_pass(M[0] // 16, n[0], M[1], M[2], B, Sh, conj)
        _y_pass(M[1] // 16, True, n[0], n[1], M[2], A3, B, None)
        _z_inverse(M[2] // 16, False, nl, n[2], A, D)
        assert np.abs(D.reshape(n) - ref).max() <= 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("n2s", N2S)
@pytest.mark.parametrize("plane", [False, True])
def test_z_passes(n2s, plane):
    """Each z length, both layouts, ragged line counts: forward is the twisted DFT, inverse undoes it."""
    L = 16 * n2s
    for nl, nz in ((35, L - 3), (16, L), (50, L // 2 + 1)):
        rng = np.random.default_rng(nl)
        flags = np.ones(nl, np.uint8)
        flags[16:32] = 0
        flags[3] = 0
        T = np.full((nl, -(-nz // 4) * 4), np.nan)
        T[flags != 0, :nz] = rng.standard_normal((int((flags != 0).sum()), nz))
        lp = -(-nl // 32) * 32
        A = np.full((L, lp) if plane else (nl, L), np.nan + 0j)
        D = np.full((nl, nz), np.nan)
        _z_forward(n2s, plane, nl, nz, T, flags, False, A, lp)
        x = np.zeros((nl, L))
        x[flags != 0, :nz] = T[flags != 0, :nz]
        ref = np.fft.fft(x * _twiddle(4 * L, np.arange(L)), axis=1)
        got = A[:, :nl].T if plane else A
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
        _z_inverse(n2s, plane, nl, nz, A, D)
        assert np.abs(D / L - x[:, :nz]).max() <= 1e-12 * np.abs(x).max()


@pytest.mark.parametrize("n2s", N2S)
def test_y_and_x_passes(n2s):
    """Each period: the y pair of passes and the x pass with a unit spectrum give M times their input."""
    M, L = 16 * n2s, 48
    rng = np.random.default_rng(n2s)
    for ny in (M // 2, M // 2 - 7, 1):
        flags = (rng.random(2 * ny) < 0.7).astype(np.uint8)
        x = rng.standard_normal((2, ny, L)) + 1j * rng.standard_normal((2, ny, L))
        A = np.where(flags.reshape(2, ny, 1) != 0, x, np.nan)
        x = np.where(flags.reshape(2, ny, 1) != 0, x, 0)
        B = np.full((2, M, L), np.nan + 0j)
        _y_pass(n2s, False, 2, ny, L, A, B, flags)
        pad = np.concatenate([x, np.zeros((2, M - ny, L))], axis=1)
        assert np.abs(B - np.fft.fft(pad, axis=1)).max() <= 1e-11 * max(1.0, np.abs(B).max())
        _y_pass(n2s, True, 2, ny, L, A, B, None)
        assert np.abs(A / M - x).max() <= 1e-12 * max(1.0, np.abs(x).max())
        C = np.full((ny, 2, L), np.nan + 0j)
        C[:] = x.transpose(1, 0, 2)
        _x_pass(n2s, ny, 2, L, C, np.ones((M, 2, L)), False, beams=3)
        assert np.abs(C / M - x.transpose(1, 0, 2)).max() <= 1e-12 * max(1.0, np.abs(x).max())


@pytest.mark.parametrize("n2s", N2S)
def test_full_lines(n2s):
    """The transform of full lines, along and across the contiguous axis, in place."""
    M = 16 * n2s
    rng = np.random.default_rng(n2s)
    x = rng.standard_normal((32, M)) + 1j * rng.standard_normal((32, M))
    d = x.ravel().copy()
    _full(n2s, d, [0, 16 * M], M, 1, True)
    ref = np.fft.fft(x * _twiddle(4 * M, np.arange(M)), axis=1)
    assert np.abs(d.reshape(x.shape) - ref).max() <= 1e-11 * np.abs(ref).max()
    y = rng.standard_normal((M, 32)) + 1j * rng.standard_normal((M, 32))
    d = y.ravel().copy()
    _full(n2s, d, [0, 16], 1, 32, False)
    ref = np.fft.fft(y, axis=0)
    assert np.abs(d.reshape(y.shape) - ref).max() <= 1e-11 * np.abs(ref).max()
