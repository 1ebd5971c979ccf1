"""The workloads by which this framework's speed is judged: whole calls of its
public entry points over the range of sizes, precisions and boundary
conditions that its users run.

A case is a dict of plain values.  `kind` names the entry point:
  strang     one Strang step of N-grid cells on the device (qbgpu.inhom_step)
  maxwell    the same with Maxwell walls (qbgpu.inhom_step_maxwell)
  upstream   one InhomStepPeriodic call of the upstream C API on host buffers
  operators  Cc[W] and Cd[W] of a few cells (qbgpu.collision_operators)
  batch      one RK4 step of homogeneous instances of several grid sizes
             (qbgpu.homogeneous_batch)
  fno        loss and gradient of one surrogate training batch (FNO.gradients)
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inhom-quantum-boltzmann-fourier-c_b200")


def _qb():
    if "qbgpu" not in sys.modules:
        spec = importlib.util.spec_from_file_location("qbgpu", os.path.join(_PKG, "qbgpu.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules["qbgpu"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["qbgpu"]


# ---------------------------------------------------------------------------
# cases

def _step(kind, N, J, M, cells, prec=64, bc="periodic", field=False, xcells=0, name=None):
    c = {"kind": kind, "N": N, "J": J, "M": M, "cells": cells, "prec": prec, "bc": bc, "field": field, "xcells": xcells or cells}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the headline workload: 64 x-cells, the metric's grid and quadrature
        _step("strang", 32, 16, 16, 64, name="strang_n32_f64_64"),
        # the same grid in the FP32 form, a finer x line (64 of 256 x-cells)
        _step("strang", 32, 16, 16, 64, prec=32, xcells=256, name="strang_n32_f32_64"),
        # the large velocity grid and quadrature: FP64 (the largest case) and FP32, cells of a 1024-cell line
        _step("strang", 64, 32, 32, 16, xcells=1024, name="strang_n64_f64_16"),
        _step("strang", 64, 32, 32, 32, prec=32, xcells=1024, name="strang_n64_f32_32"),
        # the shipped drivers' run: 10 x-cells, J = M = 32, host buffers through the upstream C API
        _step("upstream", 32, 32, 32, 10, name="upstream_n32_host_10"),
        # a coarse grid with fixed ends and a magnetic field, an odd number of radial nodes and of cells
        _step("strang", 16, 12, 9, 33, bc="dirichlet", field=True, name="dirichlet_n16_f64_33"),
        # the smallest run, where launches and latency count
        _step("strang", 8, 4, 4, 3, name="strang_n8_f64_3"),
        # a short line between Maxwell walls at a reduced quadrature
        _step("maxwell", 32, 8, 6, 7, field=True, name="maxwell_n32_f64_7"),
        # the operator itself on one cell: parallelism only from the quadrature
        _step("operators", 32, 16, 16, 1, name="operators_n32_1"),
        # a radix-3 grid size in the FP32 form
        _step("strang", 48, 16, 16, 12, prec=32, xcells=1024, name="strang_n48_f32_12"),
        # independent homogeneous instances of mixed sizes, the largest grid among them
        {"kind": "batch", "sizes": "16,16,24,32,32,32,48,48,64,64,96,128", "J": 16, "M": 16, "prec": 64, "name": "batch_mixed_f64_12"},
        # one training batch of the surrogate network: forward and backward
        {"kind": "fno", "N": 32, "width": 32, "modes": 12, "layers": 4, "batch": 64, "name": "fno_gradients_n32_64"},
    ]


def _cost(c):
    """relative cost of a step or operator case: cells x terms x FFT work"""
    P = 2 * c["N"]
    return c["cells"] * c["J"] * c["M"] * P * P * math.log2(P)


_COST_MAX = 16 * 32 * 32 * 128 * 128 * math.log2(128)        # strang_n64_f64_16


def draw(rng):
    kind = rng.choice(["strang"] * 8 + ["maxwell", "upstream", "operators", "operators", "batch", "fno"])
    if kind == "batch":
        sizes = [rng.choice([16, 16, 24, 32, 32, 48, 64, 96]) for _ in range(rng.randint(3, 12))]
        return {"kind": "batch", "sizes": ",".join(str(n) for n in sizes), "J": rng.choice([8, 12, 16]), "M": rng.randint(6, 16), "prec": 64}
    if kind == "fno":
        return {"kind": "fno", "N": rng.choice([16, 24, 32]), "width": rng.choice([16, 24, 32]), "modes": rng.randint(4, 8),
                "layers": rng.randint(2, 4), "batch": round(math.exp(rng.uniform(math.log(8), math.log(128))))}
    if kind == "upstream":
        N = 32
    else:
        N = rng.choice([8, 16, 24, 32, 32, 32, 48, 64, 64])
    while True:
        J = rng.choice([4, 8, 12, 16, 16, 32])
        M = rng.choice([J, J, rng.randint(4, 24)])
        lo, hi = (1, 8) if kind == "operators" else (3, 96)
        cells = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
        prec = 64 if kind in ("operators", "upstream") else rng.choice([64, 64, 32])
        bc = rng.choice(["periodic", "periodic", "dirichlet"]) if kind == "strang" else "periodic"
        c = _step(kind, N, J, M, cells, prec, bc, rng.random() < 0.3, 1024 if prec == 32 else cells)
        if _cost(c) <= 0.5 * _COST_MAX:
            return c


# ---------------------------------------------------------------------------
# inputs

def _box(c):
    return (12.0, 7.5) if c["kind"] == "upstream" else (6.0, 3.75)        # the drivers' box; the metric's box


def _step_inputs(c, seed):
    """state (numpy, (cells, 4, N, N)), h, dt, magnetic field"""
    L, _ = _box(c)
    W = _qb().gaussian_mixture_state(c["N"], L, seed=seed + 1, ncells=c["cells"])
    h = 1.0 / c["xcells"]
    rng = np.random.default_rng(seed)
    B = rng.normal(size=(c["cells"], 3)) if c["field"] else np.zeros((c["cells"], 3))
    return W, h, 0.4 * h / L, B


def _walls(c, seed):
    L, _ = _box(c)
    return tuple(_qb().gaussian_mixture_state(c["N"], L, seed=seed + 1 + k)[0] for k in (1000, 2000))


def _hom_states(c, seed):
    return [_qb().gaussian_mixture_state(int(n), 6.0, seed=seed + 10 * i + 1)[0] for i, n in enumerate(c["sizes"].split(","))]


def _hom_fourier(W):
    """Fourier representation of one cell (numpy (4, N, N) -> complex (4, N, N))"""
    return np.fft.fft2(W) / (W.shape[-1] ** 2)


def _fno_inputs(c, seed):
    """states, targets, flat weights, input scales and output scales"""
    qb = _qb()
    X = qb.mixture_cells(c["N"], 6.0, c["batch"], 7 * seed + 1)
    Y = 0.5 * (X.mean(axis=0, keepdims=True) - X)
    w, m, nl = c["width"], c["modes"], c["layers"]
    K = (2 * m - 1) * m
    rng = np.random.default_rng(seed)
    parts = [rng.normal(size=w * 14) / math.sqrt(14), np.zeros(w)]
    for _ in range(nl):
        parts += [rng.normal(size=2 * w * w * K) / w, rng.normal(size=w * w) / math.sqrt(w), np.zeros(w)]
    parts += [rng.normal(size=4 * w) / math.sqrt(w), np.zeros(4)]
    theta = np.concatenate(parts).astype(np.float32)
    f = qb._features_np(X)
    in_scale = 1.0 / np.sqrt(np.mean(f * f, axis=(0, 2)))
    out_scale = np.sqrt(np.mean(Y.reshape(Y.shape[0], 4, -1) ** 2, axis=(0, 2)))
    return X, Y, theta, in_scale, out_scale


class _Host:
    """the upstream C API's handles of a driver: quadrature structs and step scratch"""

    def __init__(self, c, L, R):
        self.u = _qb().Upstream()
        self.quads = [self.u.fourier(1, c["J"], L, R), self.u.fourier(2, c["J"], L, R), self.u.fourier(3, c["J"], L, R, c["M"]),
                      self.u.fourier(4, c["J"], L, R)]
        self.interm = self.u.inhom_interm(c["cells"], L)

    def __del__(self):
        import ctypes
        self.u.L.InhomStepInterm_Delete(ctypes.byref(self.interm))
        for k, q in zip((1, 2, 3, 4), self.quads):
            self.u.quad_delete(k, q)


def prepare(case, seed):
    qb, c = _qb(), case
    s = {"case": c}
    if c["kind"] == "batch":
        s["states"] = [torch.from_numpy(_hom_fourier(W)).cuda() for W in _hom_states(c, seed)]
        return s
    if c["kind"] == "fno":
        X, Y, theta, in_scale, out_scale = _fno_inputs(c, seed)
        net = qb.FNO(c["N"], c["width"], c["modes"], c["layers"])
        net.set_params(theta)
        net.set_input_scale(in_scale)
        net.set_scale(out_scale)
        s.update(net=net, X=torch.from_numpy(X).cuda(), Y=torch.from_numpy(Y).cuda())
        return s
    L, R = _box(c)
    W, h, dt, B = _step_inputs(c, seed)
    s.update(h=h, dt=dt)
    if c["kind"] == "upstream":
        s["host"] = _Host(c, L, R)
        s.update(W=W, B=B, out=np.zeros_like(W))
        return s
    s["q"] = qb.Quad(c["N"], c["J"], c["M"], L, R)
    s["ws"] = qb.Workspace(c["N"], precision=c["prec"])
    s["W"] = torch.from_numpy(W).cuda()
    if c["kind"] == "operators":
        s["W"] = qb.to_fourier(s["W"])
        return s
    s["B"] = torch.from_numpy(B).cuda()
    s["out"] = torch.empty_like(s["W"])
    if c["kind"] == "maxwell":
        s["walls"] = [torch.from_numpy(x).cuda() for x in _walls(c, seed)]
    return s


_LAMBDA = 0.4        # accommodation coefficient of the Maxwell walls


def run(state):
    qb, s = _qb(), state
    kind = s["case"]["kind"]
    if kind == "strang":
        return qb.inhom_step(s["ws"], s["q"], s["W"], s["h"], s["dt"], s["B"], bc=s["case"]["bc"], out=s["out"])
    if kind == "maxwell":
        return qb.inhom_step_maxwell(s["ws"], s["q"], s["W"], s["h"], s["dt"], _LAMBDA, s["walls"][0], s["walls"][1], s["B"], out=s["out"])
    if kind == "operators":
        return qb.collision_operators(s["ws"], s["q"], s["W"])
    if kind == "upstream":
        h = s["host"]
        return h.u.inhom_step(s["W"], h.quads, s["h"], s["dt"], s["B"], L=12.0, interm=h.interm, out=s["out"])
    if kind == "batch":
        c = s["case"]
        return qb.homogeneous_batch(s["states"], 0.01, 1, rk4=True, J=c["J"], M=c["M"], L=6.0, R=3.75, precision=c["prec"])
    loss, grad = s["net"].gradients(s["X"], s["Y"])
    return {"loss": loss, "grad": grad}


# ---------------------------------------------------------------------------
# work

def _eval_flops(N, J, M):
    """flops of one collision evaluation: transforms of 2N x 2N grids at
    5 n log2 n (a padded input or an extracted output costs 3/4).  I3 by pairs
    of opposite shifts +-a: 16 chains of two transforms serve both nodes
    (f(v) g(v + a) is g(v) f(v - a) shifted), 4 spectra and 4 extracted sums a
    pair; I1 (J angles, 3 components), I4 (4 components): padded transform,
    product, transform; I2: two padded transforms; the outer transforms."""
    P2 = 4.0 * N * N
    F = 5.0 * P2 * math.log2(P2)
    i3 = (J * M / 2) * ((32 + 6) * F + 16 * (6 + 2 + 16) * P2)
    i14 = 7 * J * (1.75 * F + 10 * P2)
    i2 = 4 * J * (1.5 * F + 8 * P2)
    return i3 + i14 + i2 + 15 * F


def work(case):
    c = case
    if c["kind"] == "fno":
        N2, w, m, nl, b = c["N"] ** 2, c["width"], c["modes"], c["layers"], c["batch"]
        K = (2 * m - 1) * m
        fwd = 2.0 * N2 * 14 * w + nl * (2.0 * N2 * w * w + 8.0 * K * w * w + 4.0 * c["N"] * m * (c["N"] + 2 * (2 * m - 1)) * w * 2) + 8.0 * N2 * w
        params = w * 15 + nl * (2 * w * w * K + w * w + w) + 4 * w + 4
        return {"bytes": b * 4 * N2 * 16.0 + 8.0 * params, "flops": 3 * b * fwd}
    if c["kind"] == "batch":
        sizes = [int(n) for n in c["sizes"].split(",")]
        return {"bytes": sum(2 * 64.0 * n * n for n in sizes), "flops": sum(4 * _eval_flops(n, c["J"], c["M"]) for n in sizes)}
    cell = 4 * c["N"] ** 2
    if c["kind"] == "operators":
        return {"bytes": 3 * 16.0 * cell * c["cells"], "flops": c["cells"] * _eval_flops(c["N"], c["J"], c["M"])}
    ncol = c["cells"] - 2 if c["bc"] == "dirichlet" else c["cells"]
    return {"bytes": 2 * 8.0 * cell * c["cells"], "flops": 2 * ncol * _eval_flops(c["N"], c["J"], c["M"])}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits

def _sinc(x):
    return torch.where(x.abs() < 1e-8, torch.ones_like(x), torch.sin(x) / torch.where(x.abs() < 1e-8, torch.ones_like(x), x))


def _sin_sinc(x):
    return torch.where(x.abs() < 1e-8, x, torch.sin(x) ** 2 / torch.where(x.abs() < 1e-8, torch.ones_like(x), x))


class _Exact:
    """the collision operator by its defining sums (upstream src/collision.c, src/integrals.c, src/quadrature.c)"""

    def __init__(self, N, J, M, L, R):
        self.N, self.J, self.M, self.L, self.R = N, J, M, L, R
        dev = "cuda"
        kn = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device=dev)
        kp = torch.fft.fftfreq(2 * N, 0.5 / N, dtype=torch.float64, device=dev)
        self.kn = (kn[:, None], kn[None, :])
        self.kp = (kp[:, None], kp[None, :])
        self.idx = torch.tensor([k if k < N // 2 else k + N for k in range(N)], device=dev)
        self.rho, self.w = np.polynomial.legendre.leggauss(M)

    def along(self, k, th):
        return k[0] * math.cos(th) + k[1] * math.sin(th)

    def pad(self, f):
        N = self.N
        out = torch.zeros(f.shape[:-2] + (2 * N, 2 * N), dtype=torch.complex128, device=f.device)
        out[..., self.idx[:, None], self.idx[None, :]] = f.to(torch.complex128)
        return out

    def spec(self, f):
        return torch.fft.fft2(self.pad(f))

    def extract(self, Z):
        """Extract of the (normalised) inverse transform"""
        return torch.fft.ifft2(Z)[..., self.idx[:, None], self.idx[None, :]]

    def operators(self, W):
        """Cc, Cd of Fourier states W (n, 4, N, N)"""
        N, J, M, L, R = self.N, self.J, self.M, self.L, self.R
        P2 = 4.0 * N * N
        n = W.shape[0]
        Wh = self.spec(W)
        one = torch.zeros_like(W[:, 0])
        one[:, 0, 0] = 1.0
        oneh = self.spec(one)
        dth = math.pi / J
        S = [torch.zeros_like(Wh) for _ in range(2)]
        psi1 = [R * _sin_sinc(R * math.pi / (2 * L) * self.along(self.kp, i * dth)) for i in range(J)]
        Fcc, F4 = 2 * oneh - 4 * Wh[:, 0], 2 * Wh[:, 0] - oneh
        Q = torch.zeros_like(Wh[:, 0])
        eta = [1.0, -1.0, -1.0, -1.0]
        for j in range(J):
            th = j * dth
            p2 = R * _sin_sinc(R * math.pi / (2 * L) * self.along(self.kn, th + 0.5 * dth))
            phi = sum(-(2 * math.pi / J) ** 2 / math.cos(i * dth - th - 0.5 * dth) * psi1[i] for i in range(J))
            S[0] += phi * torch.fft.ifft2(Fcc[:, None] * self.spec(p2 * W))
            p1 = 2 * R * _sinc(R * math.pi / L * self.along(self.kp, th))
            p2 = 2 * R * math.pi / J * _sinc(R * math.pi / L * self.along(self.kn, th + math.pi / 2))
            S[1] += p1 * torch.fft.ifft2(F4[:, None] * self.spec(p2 * W))
            a = self.spec(2 * R * _sinc(R * math.pi / L * self.along(self.kn, th)) * W)
            b = self.spec(p2 * W)
            for i in range(4):
                Q += 2 * eta[i] * a[:, i] * b[:, i]
        X = torch.zeros_like(Wh)
        for j in range(J):
            th = j * dth
            sinc = _sinc(R * math.pi / L * self.along(self.kp, th + math.pi / 2))
            for m in range(M):
                Pt = self.spec(torch.exp(1j * (R * self.rho[m] * math.pi / L) * self.along(self.kn, th)) * W)
                f2 = 2 * R * (R * self.w[m]) * math.pi / J
                for i in range(4):
                    X += (eta[i] * f2) * Pt[:, i:i + 1] * torch.fft.fft2(sinc * torch.fft.ifft2(Wh[:, i:i + 1] * Pt))
        FS, F4s = torch.fft.fft2(S[0]), torch.fft.fft2(S[1])
        Cc, Cd = torch.zeros_like(W), torch.zeros_like(W)
        for j in range(1, 4):
            g, k = j % 3 + 1, (j + 1) % 3 + 1
            Cc[:, j] = self.extract(Wh[:, k] * FS[:, g] - Wh[:, g] * FS[:, k])
        for j in range(4):
            Z = (oneh if j == 0 else 0) * Q / 1.0 - Wh[:, j] * Q - 2 * eta[j] * X[:, j] + 2 * eta[j] * Wh[:, 0] * F4s[:, j] + 2 * Wh[:, j] * F4s[:, 0]
            if j == 0:
                Z = Z - 2 * sum(Wh[:, k] * F4s[:, k] for k in range(4))
            Cd[:, j] = self.extract(Z)
        return Cc, Cd

    def rhs(self, W, B):
        Cc, Cd = self.operators(W)
        C = Cc + Cd
        b = B.to(torch.complex128)[:, :, None, None]
        C[:, 1:] += 2 * torch.linalg.cross(b.expand(-1, -1, self.N, self.N), W[:, 1:], dim=1)
        return C

    def collide(self, V, dt, B):
        """velocity-space cells through one midpoint collision step"""
        N = self.N
        W = torch.fft.fft2(V) / (N * N)
        k = torch.arange(N, device=V.device)
        conj = W[..., (-k[:, None]) % N, (-k[None, :]) % N].conj()
        W = torch.where((k <= N // 2)[None, :], W, conj)
        mid = W + 0.5 * dt * self.rhs(W, B)
        W = W + dt * self.rhs(mid, B)
        return torch.fft.ifft2(W).real * (N * N)

    def cells(self, V, dt, B, per):
        return torch.cat([self.collide(V[i:i + per], dt, B[i:i + per]) for i in range(0, V.shape[0], per)])


def _minmod(a, b):
    one = torch.ones_like(a)
    return 0.5 * (torch.copysign(one, a) + torch.copysign(one, b)) * torch.minimum(a.abs(), b.abs())


def _limiter(V, A, h, dt):
    """minmod update of the interior of lines V (axis 0) with two ghost cells at each end"""
    al = V[1:] - V[:-1]
    hb = _minmod(al[1:], al[:-1])
    nu = dt * A / h
    d = torch.copysign(torch.ones_like(nu), nu) - nu
    S, Sa = 0.5 * A * d, 0.5 * A.abs() * d
    u, up, um = V[2:-2], V[3:-1], V[1:-3]
    h0, hp, hm = hb[1:-1], hb[2:], hb[:-2]
    return u + dt / (2 * h) * (-A * (up - um) + A.abs() * (up - 2 * u + um) - S * (hp - hm) + Sa * (hp - 2 * h0 + hm))


def _transport(W, A, h, dt, bc):
    if bc == "periodic":
        n = W.shape[0]
        i = torch.arange(-2, n + 2, device=W.device) % n
        return _limiter(W[i], A, h, dt)
    n = W.shape[0]
    al = torch.cat([W[1:] - W[:-1], torch.zeros_like(W[:1])])
    hb = torch.zeros_like(W)
    hb[1:n - 1] = _minmod(al[1:n - 1], al[:n - 2])
    nu = dt * A / h
    S = 0.5 * A * (torch.copysign(torch.ones_like(nu), nu) - nu)
    Sa = S * torch.copysign(torch.ones_like(A), A)
    sc = dt / (2 * h)
    out = W.clone()
    u, up, um, h0, hp, hm = W[1:-1], W[2:], W[:-2], hb[1:-1], hb[2:], hb[:-2]
    out[1:-1] = u + sc * (-A * (up - um) + A.abs() * (up - 2 * u + um) - S * (hp - hm) + Sa * (hp - 2 * h0 + hm))
    last = W[-1] + 2 * sc * (-A * (W[-1] - W[-2]) - S * (hb[-1] - hb[-2]))
    first = W[0] + 2 * sc * (-A * (W[1] - W[0]) - S * (hb[1] - hb[0]))
    out[-1] = torch.where(A >= 0, last, W[-1])
    out[0] = torch.where(A >= 0, W[0], first)
    return out


def _vx(N, L):
    return torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device="cuda") * (2 * L / N)


def _exact_step(c, W, h, dt, B, L, R, ex):
    A = _vx(c["N"], L)[:, None].expand(c["N"], c["N"])
    per = max(1, (1 << 26) // (16 * 16 * c["N"] * c["N"]))
    V = _transport(W, A, h, 0.5 * dt, c["bc"])
    if c["bc"] == "dirichlet":
        V[1:-1] = ex.cells(V[1:-1], dt, B[1:-1], per)
    else:
        V = ex.cells(V, dt, B, per)
    return _transport(V, A, h, 0.5 * dt, c["bc"])


def _exact_maxwell(c, W, h, dt, B, walls, L, ex):
    """Maxwell walls (upstream src/simulation.c:837-1165, src/finite_volume.c:186-323): per component the rows
    v_x = dv .. L, -L .. -dv (the row of -L serves both), diffuse and specular re-emission at both ends"""
    N = c["N"]
    half = N // 2
    rows = torch.tensor([r + 1 if r < half else r for r in range(N)], device="cuda")
    A = torch.tensor([(r + 1 if r < half else r - N) * (2 * L / N) for r in range(N)], dtype=torch.float64, device="cuda")[:, None].expand(N, N)
    right = lambda U: (A[:half] * U[:half]).sum()                       # noqa: E731
    left = lambda U: (A[half:].abs() * U[half:]).sum()                  # noqa: E731
    WL, WR = walls[0][:, rows], walls[1][:, rows]
    WL, WR = WL / right(WL[0]), WR / left(WR[0])

    def half_step(V):
        U = V[:, :, rows]
        fL, fR = left(U[0, 0]), right(U[-1, 0])
        mirror = U.flip(2, 3)
        a, b = U[0].clone(), U[-1].clone()
        a[:, :half] = (1 - _LAMBDA) * mirror[0][:, :half] + _LAMBDA * fL * WL[:, :half]
        b[:, half:] = (1 - _LAMBDA) * mirror[-1][:, half:] + _LAMBDA * fR * WR[:, half:]
        U = _limiter(torch.cat([a[None], a[None], U, b[None], b[None]]), A, h, 0.5 * dt)
        out = V.clone()
        out[:, :, 1:half] = U[:, :, :half - 1]
        out[:, :, half:] = U[:, :, half:]
        return out

    return half_step(ex.cells(half_step(W), dt, B, W.shape[0]))


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        out = []
        for W in _hom_states(c, seed):
            N = W.shape[-1]
            ex = _Exact(N, c["J"], c["M"], 6.0, 3.75)
            Z = torch.zeros((1, 3), dtype=torch.float64, device="cuda")
            Wf = torch.from_numpy(_hom_fourier(W)).cuda()[None]
            dt = 0.01
            k1 = ex.rhs(Wf, Z)
            k2 = ex.rhs(Wf + 0.5 * dt * k1, Z)
            k3 = ex.rhs(Wf + 0.5 * dt * k2, Z)
            k4 = ex.rhs(Wf + dt * k3, Z)
            out.append((Wf + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4))[0])
        return out
    if c["kind"] == "fno":
        return _exact_fno(c, seed)
    L, R = _box(c)
    W, h, dt, B = _step_inputs(c, seed)
    W, B = torch.from_numpy(W).cuda(), torch.from_numpy(B).cuda()
    ex = _Exact(c["N"], c["J"], c["M"], L, R)
    if c["kind"] == "operators":
        N = c["N"]
        Wf = torch.fft.fft2(W) / (N * N)
        k = torch.arange(N, device="cuda")
        Wf = torch.where((k <= N // 2)[None, :], Wf, Wf[..., (-k[:, None]) % N, (-k[None, :]) % N].conj())
        return ex.operators(Wf)
    if c["kind"] == "maxwell":
        return _exact_maxwell(c, W, h, dt, B, [torch.from_numpy(x).cuda() for x in _walls(c, seed)], L, ex)
    return _exact_step(c, W, h, dt, B, L, R, ex)


def _exact_fno(c, seed):
    X, Y, theta, in_scale, out_scale = _fno_inputs(c, seed)
    N, w, m, nl = c["N"], c["width"], c["modes"], c["layers"]
    K, P = (2 * m - 1) * m, c["N"] ** 2
    t = torch.from_numpy(theta).cuda().double().requires_grad_(True)
    o = [0]

    def take(*shape):
        k = int(np.prod(shape))
        o[0] += k
        return t[o[0] - k:o[0]].reshape(shape)

    f = torch.from_numpy(_qb_features(X) * in_scale[None, :, None]).cuda()
    p = torch.arange(N, dtype=torch.float64, device="cuda")
    kx = torch.arange(-(m - 1), m, dtype=torch.float64, device="cuda").repeat_interleave(m)
    ky = torch.arange(m, dtype=torch.float64, device="cuda").repeat(2 * m - 1)
    th = 2 * math.pi / N * (kx[:, None, None] * p[None, :, None] + ky[:, None, None] * p[None, None, :])
    E = torch.exp(-1j * th.reshape(K, P))
    h = torch.einsum("oi,bip->bop", take(w, 14), f) + take(w)[None, :, None]
    for k in range(nl):
        R = torch.complex(take(w, w, K), take(w, w, K))
        H = torch.einsum("bip,kp->bik", h.to(torch.complex128), E)
        O = torch.einsum("iok,bik->bok", R, H)
        u = torch.einsum("bok,kp->bop", O, E.conj()).real / P + torch.einsum("oi,bip->bop", take(w, w), h) + take(w)[None, :, None]
        h = torch.nn.functional.gelu(u) if k < nl - 1 else u
    y = torch.einsum("oi,bip->bop", take(4, w), h) + take(4)[None, :, None]
    target = torch.from_numpy(Y.reshape(Y.shape[0], 4, P) / out_scale[None, :, None]).cuda()
    loss = torch.mean((y - target) ** 2)
    loss.backward()
    return {"loss": float(loss.detach()), "grad": t.grad}


def _qb_features(W):
    W = W.reshape(W.shape[0], 4, -1)
    return np.stack([W[:, k] for k in range(4)] + [W[:, i] * W[:, j] for i in range(4) for j in range(i, 4)], axis=1)
