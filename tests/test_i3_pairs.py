"""The I3 sums by pairs of opposite shifts: the terms m and M - 1 - m of an
angle of FourierI3 (upstream src/quadrature.c:395-466) have the shifts a and
-a, one psi2 table and equal weights, and both follow from the chains of one
of them (I3Units in csrc/qb_kernels.cuh).

On the CPU the identity is checked in FP64 against the term-by-term sums, for
states of every kind (complex noise has Nyquist and anti-Hermitian content)
and for the packed real form.  On the GPU Cc and Cd are checked against the
oracle, which sums term by term: even and odd numbers of radial nodes (an odd
one leaves a node alone), one cell and several, all grid sizes.  The bounds are
the repository's: 1e-12 (relative L1) in FP64, 1e-5 (relative L2) in FP32.
"""
import numpy as np
import pytest

import orc
import qbgpu
from conftest import rel_l1

L, R = 6.0, 3.75
ETA = np.array([1.0, -1.0, -1.0, -1.0])


class Grid:
    def __init__(self, N, th):
        self.N = N
        self.kn = np.fft.fftfreq(N, 1.0 / N)
        self.idx = np.array([k if k < N // 2 else k + N for k in range(N)])
        kp = np.fft.fftfreq(2 * N, 0.5 / N)
        x = np.pi * R / L * (-kp[:, None] * np.sin(th) + kp[None, :] * np.cos(th))
        self.psi2 = np.sinc(x / np.pi)
        self.c, self.s = np.cos(th), np.sin(th)

    def shift(self, rho):
        return np.exp(1j * rho * np.pi / L * (self.kn[:, None] * self.c + self.kn[None, :] * self.s))

    def spec(self, f):
        out = np.zeros(f.shape[:-2] + (2 * self.N, 2 * self.N), complex)
        out[..., self.idx[:, None], self.idx[None, :]] = f
        return np.fft.fft2(out)

    def extract(self, Z):
        return np.fft.ifft2(Z)[..., self.idx[:, None], self.idx[None, :]]

    def chain(self, x):
        return np.fft.fft2(self.psi2 * np.fft.ifft2(x))


def states(N, n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "noise":                          # complex noise: Nyquist and anti-Hermitian content
        return 0.2 * (rng.normal(size=(n, 4, N, N)) + 1j * rng.normal(size=(n, 4, N, N))) / N
    Wv = qbgpu.gaussian_mixture_state(N, L, seed=seed, ncells=n)
    if kind == "kinks":                          # real velocity-space states with Nyquist content
        Wv = Wv * (1 + 0.1 * rng.normal(size=Wv.shape))
    return np.stack([orc.to_fourier(w) for w in Wv])


@pytest.mark.parametrize("N", [6, 8, 12])
@pytest.mark.parametrize("th", [0.0, 0.7, np.pi / 2])
@pytest.mark.parametrize("kind", ["noise", "kinks"])
def test_pair_identity(N, th, kind):
    g = Grid(N, th)
    W = states(N, 1, kind, 3)[0]
    Wh = g.spec(W)
    psi = g.shift(0.37 * R)
    P = g.spec(psi * W)
    T = np.stack([[g.chain(Wh[i] * P[j]) for j in range(4)] for i in range(4)])
    Y = np.einsum("j,jab,ijab->iab", ETA, Wh, T)
    Z = psi.conj() * g.extract(Y)
    Pm = g.spec(psi.conj() * W)
    direct = np.stack([g.extract(sum(ETA[i] * Pm[i] * g.chain(Wh[i] * Pm[j]) for i in range(4))) for j in range(4)])
    assert rel_l1(Z, direct) < 1e-12


@pytest.mark.parametrize("N", [6, 8, 12])
def test_packed_sums_separate(N):
    """A = Z_0 + i Z_1 on the frequencies -N/2 .. N/2 gives both parts where W
    has no Nyquist content"""
    g = Grid(N, 0.7)
    W = states(N, 1, "kinks", 5)[0]
    W[:, N // 2, :] = 0
    W[:, :, N // 2] = 0
    Wh = g.spec(W)
    assert np.abs(Wh.imag).max() < 1e-12 * np.abs(Wh).max()
    psi = g.shift(-0.6 * R)
    P = g.spec(psi * W)
    Y = np.stack([sum(ETA[j] * Wh[j] * g.chain(Wh[i] * P[j]) for j in range(4)) for i in range(4)])
    V = np.fft.ifft2(Y[0].real + 1j * Y[1].real)
    H = N // 2
    f = np.arange(-H, H + 1)
    ps = np.exp(1j * -0.6 * R * np.pi / L * (f[:, None] * g.c + f[None, :] * g.s))
    A = ps.conj() * V[f[:, None], f[None, :]]
    Am = A[::-1, ::-1].conj()
    z0, z1 = 0.5 * (A + Am), -0.5j * (A - Am)
    order = g.kn.astype(int) + H
    ref = psi.conj() * g.extract(Y)
    assert rel_l1(z0[np.ix_(order, order)], ref[0]) < 1e-12
    assert rel_l1(z1[np.ix_(order, order)], ref[1]) < 1e-12


def gpu_operators(N, J, M, W, precision):
    torch = pytest.importorskip("torch")
    q, ws = qbgpu.Quad(N, J, M, L, R), qbgpu.Workspace(N, precision=precision)
    cc, cd = qbgpu.collision_operators(ws, q, torch.from_numpy(W).cuda())
    return cc.cpu().numpy(), cd.cpu().numpy(), ws.i3_forms()


CASES = [(8, 4, 2, 1), (8, 4, 3, 5), (16, 4, 3, 2), (16, 8, 6, 1), (24, 4, 3, 2), (32, 4, 2, 1), (32, 4, 3, 3), (32, 4, 7, 1), (48, 4, 2, 1),
         (64, 4, 2, 2), (64, 4, 3, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("N,J,M,cells", CASES)
@pytest.mark.parametrize("kind", ["noise", "smooth"])
def test_pairs_against_oracle_fp64(N, J, M, cells, kind):
    W = states(N, cells, kind, 11)
    o = orc.Oracle(N, J, M, L, R)
    cc, cd, _ = gpu_operators(N, J, M, W, 64)
    for i in range(cells):
        assert rel_l1(cc[i], o.cc(W[i])) < 1e-12
        assert rel_l1(cd[i], o.cd(W[i])) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("N,J,M,cells", CASES)
def test_pairs_against_oracle_fp32(N, J, M, cells):
    # one cell of complex noise (complex form), the others smooth (real form where it has one)
    W = np.concatenate([states(N, 1, "noise", 12), states(N, cells, "smooth", 13)])
    o = orc.Oracle(N, J, M, L, R)
    cc, cd, _ = gpu_operators(N, J, M, W, 32)
    for i in range(cells + 1):
        assert np.linalg.norm(cc[i] - o.cc(W[i])) <= 1e-5 * np.linalg.norm(o.cc(W[i]))
        assert np.linalg.norm(cd[i] - o.cd(W[i])) <= 1e-5 * np.linalg.norm(o.cd(W[i]))
