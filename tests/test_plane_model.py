"""numpy model of the plane kernel's index arithmetic (plane.cuh) against the direct spectral D
apply (CPU): the same buffers, places and exchanges, every access checked against its buffer, for
each grid size and both line paddings. Work items of a phase are independent of each other, so
the model takes a phase's stages over whole index ranges at once."""
import numpy as np
import pytest

SIZES = [*range(16, 129, 8), 144, 160]


def geometry(n, single):
    r2 = 4 if n <= 56 else (8 if n < 144 else 16)
    if not single:
        return n // r2, r2, n + n // r2
    return n // r2, r2, n + (4 if r2 == 4 else (8 if r2 == 8 and n % 16 == 0 else 0))


def wn(k, n):
    k = np.asarray(k)
    return np.where(k < n // 2, k, np.where(k == n // 2, 0, k - n))


def dft(v, s):  # along axis 0, unnormalised
    r = v.shape[0]
    m = np.exp(s * 2j * np.pi * np.outer(np.arange(r), np.arange(r)) / r)
    return np.tensordot(m, v, 1)


class Plane:
    """One x plane in the kernel's shared buffer."""

    def __init__(self, n, single):
        self.n, self.single = n, single
        self.r1, self.r2, self.ps2 = geometry(n, single)
        self.nq, self.nh = n // 2, n // 2 + 1
        self.buf = np.full(self.nq * self.ps2, np.nan, complex)
        self.tw = np.exp(2j * np.pi * np.arange(n) / n)

    def slot(self, k):
        return k if self.single else k + k // self.r2

    def row(self, r, c):
        second = self.slot(np.where(c == 0, self.nq, self.n - c))
        a = (r >> 1) * self.ps2 + np.where(r & 1, second, self.slot(c))
        assert np.all((a >= 0) & (a < self.buf.size))
        return a

    def inverse_y(self, G, j):
        n, r1, r2 = self.n, self.r1, self.r2
        c = np.arange(self.nq)
        for b in range(r2):
            ky = r2 * np.arange(r1) + b
            u = G[ky][:, c].copy()
            u[:, 0] = u[:, 0] + 1j * G[ky, self.nq]
            if j == 1:
                u = 1j * wn(ky, n)[:, None] * u
            u = dft(u, +1)
            for k1 in range(r1):
                self.buf[self.row(k1 * r2 + b, c)] = u[k1] * self.tw[b * k1]
        for k1 in range(r1):
            at = [self.row(k1 * r2 + b, c) for b in range(r2)]
            v = dft(np.array([self.buf[a] for a in at]), +1)
            for i in range(r2 // 2):
                a, h = v[2 * i], v[2 * i + 1]
                if j == 2:
                    a, h = 1j * c * a, 1j * c * h
                z0, z1 = a + 1j * h, np.conj(a) + 1j * np.conj(h)
                z0[0], z1[0] = a[0].real + 1j * h[0].real, a[0].imag + 1j * h[0].imag
                self.buf[at[2 * i]], self.buf[at[2 * i + 1]] = z0, z1

    def lines(self, real_op, forward=True, backward=True):
        n, r1, r2, nq = self.n, self.r1, self.r2, self.nq
        t = np.arange(r2)
        for pr in range(nq):
            E = self.buf[pr * self.ps2: pr * self.ps2 + self.ps2]
            p0 = 2 * pr
            y0 = p0 // r2 + r1 * (p0 % r2)
            y1 = y0 + r1
            assert y1 < n
            rows = np.arange(r1)[:, None]
            home = self.slot(r2 * rows + t)
            ex = rows * r2 + (t[None, :] ^ (rows & (r2 - 1))) if self.single else home
            assert home.max() < self.ps2 and ex.max() < self.ps2
            m = np.arange(r1)[:, None] + r1 * t[None, :]  # [k1][k2]
            if backward:
                u = dft(E[home], +1) * self.tw[np.arange(r1)[:, None] * t]
                E[ex] = u
                z = dft(E[ex].T.copy(), +1).T  # [k1][k2]
            else:
                z = None
            z = real_op(y0, y1, m, z)
            if forward:
                v = dft(z.T.copy(), -1).T * np.conj(self.tw[np.arange(r1)[:, None] * t])
                E[ex] = v
                E[home] = dft(E[ex], -1)

    def forward_y(self, j):
        n, r1, r2, nq = self.n, self.r1, self.r2, self.nq
        c = np.arange(nq)
        M = np.full((n, self.nh), np.nan, complex)
        zcol = np.empty(n, complex)
        for k1 in range(r1):
            at = [self.row(k1 * r2 + b, c) for b in range(r2)]
            v = []
            for i in range(r2 // 2):
                z, zq = self.buf[at[2 * i]], self.buf[at[2 * i + 1]]
                a, h = (z + np.conj(zq)) / 2, (z - np.conj(zq)) / 2j
                a[0], h[0] = z[0].real + 1j * zq[0].real, z[0].imag + 1j * zq[0].imag
                if j == 2:
                    a, h = 1j * c * a, 1j * c * h
                v += [a, h]
            v = dft(np.array(v), -1)
            for b in range(r2):
                self.buf[at[b]] = v[b] * np.conj(self.tw[k1 * b])
        for b in range(r2):
            u = dft(np.array([self.buf[self.row(k1 * r2 + b, c)] for k1 in range(r1)]), -1)
            for a in range(r1):
                ky = b + r2 * a
                zcol[ky] = u[a][0]
                M[ky, 1:nq] = u[a][1:] * (1j * wn(ky, n) if j == 1 else 1)
        ky = np.arange(n)
        z, zm = zcol, zcol[(n - ky) % n]
        w = 1j * wn(ky, n) if j == 1 else 1
        M[:, 0], M[:, nq] = w * (z + np.conj(zm)) / 2, w * (z - np.conj(zm)) / 2j
        return M


def columns_forward(M, n, r1, r2):
    """x transform of (x, ky, kz): R1-point DFTs over x = R2 a + b, result [k1][k2]."""
    tw = np.exp(-2j * np.pi * np.arange(n) / n)
    buf = np.empty((n,) + M.shape[1:], complex)
    for b in range(r2):
        u = dft(M[r2 * np.arange(r1) + b], -1)
        for k1 in range(r1):
            buf[k1 * r2 + b] = u[k1] * tw[b * k1]
    return np.array([dft(buf[k1 * r2: k1 * r2 + r2], -1) for k1 in range(r1)])


def columns_inverse(d, n, r1, r2):
    tw = np.exp(2j * np.pi * np.arange(n) / n)
    buf = np.empty((n,) + d.shape[2:], complex)
    for k1 in range(r1):
        v = dft(d[k1], +1)
        for b in range(r2):
            buf[k1 * r2 + b] = v[b] * tw[b * k1]
    out = np.empty_like(buf)
    for b in range(r2):
        u = dft(buf[[k1 * r2 + b for k1 in range(r1)]], +1)
        for a in range(r1):
            out[b + r2 * a] = u[a]
    return out


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("n", SIZES)
def test_phases_give_the_direct_d_apply(n, single):
    rng = np.random.default_rng(n)
    x_planes = rng.choice(n, 3, replace=False)
    r1, r2, _ = geometry(n, single)
    # a band-limited field whose x transform is cheap: few x modes on every (y, z)
    c = rng.standard_normal((n, n, n)) if n <= 32 else np.zeros((n, n, n))
    if n > 32:
        x = np.arange(n)[:, None, None]
        for mode in (0, 1, 5, n // 2):
            c += np.cos(2 * np.pi * mode * x / n + mode) * rng.standard_normal((1, n, n))
    k = 1 + rng.random((n, n, n))
    w = wn(np.arange(n), n)
    spec = np.fft.rfftn(c)
    d = spec.reshape((n, n, n // 2 + 1))
    kx = np.arange(r1)[:, None] + r1 * np.arange(r2)[None, :]
    G0 = columns_inverse(d[kx] / n ** 3, n, r1, r2)
    Gx = columns_inverse(1j * w[kx][..., None, None] * d[kx] / n ** 3, n, r1, r2)
    grads = [np.fft.irfftn(1j * ww * spec, s=c.shape, axes=(0, 1, 2)) for ww in
             (w[:, None, None], w[None, :, None], w[: n // 2 + 1][None, None, :])]
    for x in x_planes:
        for j in range(3):
            p = Plane(n, single)
            p.inverse_y(Gx[x] if j == 0 else G0[x], j)
            seen = np.full((n, n), np.nan)

            def op(y0, y1, m, z):
                seen[y0, m], seen[y1, m] = z.real, z.imag
                return z.real * k[x, y0, m] + 1j * z.imag * k[x, y1, m]

            p.lines(op)
            scale = np.abs(grads[j][x]).max()
            assert np.abs(seen - grads[j][x]).max() <= 1e-11 * scale
            M = p.forward_y(j)
            want = np.fft.fft(np.fft.rfft(k[x] * grads[j][x], axis=1), axis=0)
            if j == 1:
                want = 1j * w[:, None] * want
            if j == 2:
                want = 1j * w[: n // 2 + 1][None, :] * want
            assert np.abs(M - want).max() <= 1e-11 * np.abs(want).max()


@pytest.mark.parametrize("n", SIZES)
def test_transform_of_a_real_field_and_back(n):
    rng = np.random.default_rng(n)
    r1, r2, _ = geometry(n, True)
    f = rng.standard_normal((n, n))
    p = Plane(n, True)
    p.lines(lambda y0, y1, m, z: f[y0, m] + 1j * f[y1, m], backward=False)
    M = p.forward_y(0)
    want = np.fft.fft(np.fft.rfft(f, axis=1), axis=0)
    assert np.abs(M - want).max() <= 1e-11 * np.abs(want).max()
    out = np.empty((n, n))
    p = Plane(n, True)
    p.inverse_y(want / n ** 2, 0)

    def store(y0, y1, m, z):
        out[y0, m], out[y1, m] = z.real, z.imag

    p.lines(store, forward=False)
    assert np.abs(out - f).max() <= 1e-11 * np.abs(f).max()
    col = rng.standard_normal((n, 4)) + 1j * rng.standard_normal((n, 4))
    kx = np.arange(r1)[:, None] + r1 * np.arange(r2)[None, :]
    d = columns_forward(col, n, r1, r2)
    assert np.abs(d - np.fft.fft(col, axis=0)[kx]).max() <= 1e-10 * n
    assert np.abs(columns_inverse(d, n, r1, r2) / n - col).max() <= 1e-11 * n
