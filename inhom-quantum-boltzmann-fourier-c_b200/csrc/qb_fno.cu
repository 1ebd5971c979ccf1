// qb_fno.cu — a Fourier-neural-operator surrogate of the collision operator
// C[W] = Cc + Cd on one velocity-space cell, with hand-written forward,
// backward and Adam kernels (FP32 arithmetic, FP64 inputs and outputs; on
// request the pointwise maps and the truncated DFTs run on the tensor cores
// with BF16 operands and FP32 accumulation).
//
// Model (per cell; fields on the N x N velocity grid, point p = (l, k_v)):
//   x        = the 4 Pauli components and their 10 pairwise products (the
//              operator is cubic in W), each times a fixed input scale
//   h0       = A x + a                                  lift 14 -> w channels
//   layer l: H_i(k) = sum_p h_i(p) e^{-i theta(k,p)}     truncated DFT, modes
//            O_o(k) = sum_i R_l[i,o,k] H_i(k)            kx in [-m+1, m-1], ky in [0, m)
//            s_o(p) = Re sum_k O_o(k) e^{+i theta(k,p)} / N^2
//            u      = s + W_l h + b_l,  h' = gelu(u) (last layer: h' = u)
//   y        = Q h + q,  C~ = y * out_scale (per Pauli component)
// with theta(k, p) = 2 pi (kx l + ky k_v) / N.  The truncated transforms are
// separable matrix products (N x m then (2m-1) x N twiddle sums per field):
// only m of N frequencies per direction are kept, so this costs less than a
// full FFT and its adjoint is the same pair of sums.  Gradients use the
// complex convention dL/dRe + i dL/dIm: for O = R H, dR = dO conj(H) and
// dH = dO conj(R); for H = DFT(h) of a real field, dh = Re IDFT(dH) (no
// 1/N^2).  Every reduction (loss, weight gradients) is a fixed-order tree or
// a per-chunk partial sum reduced in order: results are deterministic.
#include "qb_engine.h"
#include "qb_kernels.cuh"
#include "qb_umma.cuh"

#include <cuda_bf16.h>

extern "C" {
#include "qbgpu.h"
}

#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

namespace {

constexpr int kFnoMaxWidth = 64;
constexpr int kFnoIn = 14;                   // input features: w_c (4) and w_i w_j, i <= j (10)

struct InScale { double s[kFnoIn]; };

struct Offsets {
	long A, a, Q, q;
	std::vector<long> Rr, Ri, W, b;
	long total;
};

Offsets offsets(int w, int K, int L) {
	Offsets o;
	long p = 0;
	o.A = p; p += (long)w * kFnoIn;
	o.a = p; p += w;
	for (int l = 0; l < L; l++) {
		o.Rr.push_back(p); p += (long)w * w * K;
		o.Ri.push_back(p); p += (long)w * w * K;
		o.W.push_back(p); p += (long)w * w;
		o.b.push_back(p); p += w;
	}
	o.Q = p; p += 4L * w;
	o.q = p; p += 4;
	o.total = p;
	return o;
}

__device__ __forceinline__ float gelu_f(float u) { return 0.5f * u * (1.0f + erff(u * 0.70710678118654752f)); }
__device__ __forceinline__ float dgelu_f(float u) {
	return 0.5f * (1.0f + erff(u * 0.70710678118654752f)) + u * expf(-0.5f * u * u) * 0.39894228040143268f;
}

// input features x[b][f][p] (FP32) of the FP64 state: f < 4: w_f; then the
// products w_i w_j (i <= j) in the order (0,0), (0,1), ..., (3,3); feature f
// is multiplied by sc.s[f]
__global__ void k_fno_in(int B, int P, const double *__restrict__ W, InScale sc, float *__restrict__ x) {
	const long n = (long)B * P;
	for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
		const long b = t / P, p = t % P;
		double w[4];
		for (int c = 0; c < 4; c++) w[c] = W[(b * 4 + c) * P + p];
		float *o = x + b * kFnoIn * P + p;
		int f = 0;
		for (int c = 0; c < 4; c++, f++) o[(long)f * P] = (float)(sc.s[f] * w[c]);
		for (int i = 0; i < 4; i++)
			for (int j = i; j < 4; j++, f++) o[(long)f * P] = (float)(sc.s[f] * w[i] * w[j]);
	}
}

// out[b][o][p] = sum_i M[o][i] in[b][i][p] + bias[o] (+ add[b][o][p]); act: store
// gelu in hout and u in uout.  trans: M^T (the backward of a pointwise map, M[i][o]).
// A thread keeps the CI (>= cin) inputs of a point in registers and takes every
// gridDim.y-th block of four outputs, the matrix rows as broadcast float4 reads.
// Bound by latency and L2: 64 cells, 32 x 32 channels at N = 32: 27 -> 18 us (the
// inputs were in local memory, their count known at run time only).
template <int CI>
__global__ void __launch_bounds__(256) k_fno_pointwise(int B, int P, int cin, int cout, int trans, const float *__restrict__ in,
                                                       const float *__restrict__ M, const float *__restrict__ bias,
                                                       const float *__restrict__ add, float *__restrict__ uout, float *__restrict__ hout, int act) {
	__shared__ __align__(16) float Ms[kFnoMaxWidth][CI];
	__shared__ float bs[kFnoMaxWidth];
	for (int i = threadIdx.x; i < cout * CI; i += blockDim.x) {
		const int o = i / CI, c = i % CI;
		Ms[o][c] = c < cin ? (trans ? M[c * cout + o] : M[o * cin + c]) : 0.0f;
	}
	for (int i = threadIdx.x; i < cout; i += blockDim.x) bs[i] = bias ? bias[i] : 0.0f;
	__syncthreads();
	const long n = (long)B * P;
	for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
		const long b = t / P, p = t % P;
		const float *x = in + b * cin * P + p;
		float v[CI];
#pragma unroll
		for (int i = 0; i < CI; i++) v[i] = i < cin ? x[(long)i * P] : 0.0f;
		for (int o0 = 4 * blockIdx.y; o0 < cout; o0 += 4 * gridDim.y) {
			const int no = min(4, cout - o0);
			float s[4];
#pragma unroll
			for (int q = 0; q < 4; q++) {
				if (q >= no) continue;
				s[q] = bs[o0 + q];
				if (add) s[q] += add[(b * cout + o0 + q) * P + p];
			}
#pragma unroll
			for (int q = 0; q < 4; q++) {
				if (q >= no) continue;
				const float4 *m = reinterpret_cast<const float4 *>(Ms[o0 + q]);
				float r = 0.0f;
#pragma unroll
				for (int i = 0; i < CI / 4; i++) {
					const float4 w = m[i];
					r = fmaf(w.x, v[4 * i], r);
					r = fmaf(w.y, v[4 * i + 1], r);
					r = fmaf(w.z, v[4 * i + 2], r);
					r = fmaf(w.w, v[4 * i + 3], r);
				}
				const float u = s[q] + r;
				const long oi = (b * cout + o0 + q) * P + p;
				if (uout) uout[oi] = u;
				hout[oi] = act ? gelu_f(u) : u;
			}
		}
	}
}

// the twiddle of the truncated transforms: tw[j] = e^{2 pi i j / N}, j < N, built once per network
// truncated forward DFT of every (b, c) field: H[b][c][k] = scale * sum_p f(p) e^{-i theta(k,p)}.
// Rows: a thread has one l and every (blockDim / N)-th ky, with the twiddle
// index advanced instead of reduced; columns: a thread gives kx and -kx from the same
// four sums.  64 cells x 32 channels at N = 32, 12 modes: 59 -> 16 us.
__global__ void __launch_bounds__(256) k_fno_dft(int N, int m, const float *__restrict__ f, const float2 *__restrict__ twg, float2 *__restrict__ H,
                                                 float scale) {
	extern __shared__ float sm[];
	const int P = N * N, K = (2 * m - 1) * m, pitch = N + 1;
	float2 *T = reinterpret_cast<float2 *>(sm);      // N x m
	float2 *tw = T + N * m;                          // N
	float *fs = reinterpret_cast<float *>(tw + N);   // N x (N + 1)
	const long bc = blockIdx.x;
	for (int i = threadIdx.x; i < P; i += blockDim.x) fs[(i / N) * pitch + i % N] = f[bc * P + i];
	for (int j = threadIdx.x; j < N; j += blockDim.x) tw[j] = twg[j];
	__syncthreads();
	const int ng = blockDim.x / N;                   // N <= 64
	if ((int)threadIdx.x < ng * N) {
		const int l = threadIdx.x % N;
		const float *row = fs + l * pitch;
		for (int ky = threadIdx.x / N; ky < m; ky += 2 * ng) {
			const int k2 = min(ky + ng, m - 1);
			float re = 0.0f, im = 0.0f, re2 = 0.0f, im2 = 0.0f;
			int j = 0, j2 = 0;
#pragma unroll 8
			for (int kv = 0; kv < N; kv++) {
				const float2 w = tw[j], w2 = tw[j2];
				const float v = row[kv];
				re = fmaf(v, w.x, re);
				im = fmaf(v, -w.y, im);
				re2 = fmaf(v, w2.x, re2);
				im2 = fmaf(v, -w2.y, im2);
				j += ky;
				if (j >= N) j -= N;
				j2 += k2;
				if (j2 >= N) j2 -= N;
			}
			T[l * m + ky] = make_float2(re, im);
			if (ky + ng < m) T[l * m + k2] = make_float2(re2, im2);
		}
	}
	__syncthreads();
	for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
		const int kx = t / m, ky = t % m;
		float ac = 0.0f, as = 0.0f, bcs = 0.0f, bs = 0.0f;
		int j = 0;
#pragma unroll 8
		for (int l = 0; l < N; l++) {
			const float2 w = tw[j], a = T[l * m + ky];
			ac = fmaf(a.x, w.x, ac);
			as = fmaf(a.x, w.y, as);
			bcs = fmaf(a.y, w.x, bcs);
			bs = fmaf(a.y, w.y, bs);
			j += kx;
			if (j >= N) j -= N;
		}
		float2 *h = H + bc * K;
		h[(m - 1 + kx) * m + ky] = make_float2(scale * (ac + bs), scale * (bcs - as));
		if (kx > 0) h[(m - 1 - kx) * m + ky] = make_float2(scale * (ac - bs), scale * (bcs + as));
	}
}

// truncated inverse: out[b][c][p] (=, or +=) scale * Re sum_k O[b][c][k] e^{+i theta(k,p)}, times
// dgelu(u[b][c][p]) when u is given (the step to the layer below in the backward
// pass).  The frequencies kx and -kx are summed as O(kx) +- O(-kx); a thread of the
// second stage has one kv and every (blockDim / N)-th row.  60 -> 24 us (as k_fno_dft).
__global__ void __launch_bounds__(256) k_fno_idft(int N, int m, const float2 *__restrict__ O, const float2 *__restrict__ twg, float *__restrict__ out,
                                                  float scale, int accumulate, const float *__restrict__ u) {
	extern __shared__ float sm[];
	const int P = N * N, K = (2 * m - 1) * m;
	float2 *S = reinterpret_cast<float2 *>(sm);      // m x m: O(kx) + O(-kx) (kx = 0: O(0))
	float2 *D = S + m * m;                           // m x m: O(kx) - O(-kx)
	float2 *U = D + m * m;                           // N x m
	float2 *tw = U + N * m;                          // N
	const long bc = blockIdx.x;
	for (int t = threadIdx.x; t < m * m; t += blockDim.x) {
		const int kx = t / m, ky = t % m;
		const float2 a = O[bc * K + (m - 1 + kx) * m + ky], b = O[bc * K + (m - 1 - kx) * m + ky];
		S[t] = kx == 0 ? a : make_float2(a.x + b.x, a.y + b.y);
		D[t] = make_float2(a.x - b.x, a.y - b.y);
	}
	for (int j = threadIdx.x; j < N; j += blockDim.x) tw[j] = twg[j];
	__syncthreads();
	for (int t = threadIdx.x; t < N * m; t += blockDim.x) {
		const int l = t / m, ky = t % m;
		float re = S[ky].x, im = S[ky].y;
		int j = l;
#pragma unroll 4
		for (int kx = 1; kx < m; kx++) {
			const float2 w = tw[j], a = S[kx * m + ky], b = D[kx * m + ky];
			re = fmaf(a.x, w.x, fmaf(-b.y, w.y, re));
			im = fmaf(a.y, w.x, fmaf(b.x, w.y, im));
			j += l;
			if (j >= N) j -= N;
		}
		U[t] = make_float2(re, im);
	}
	__syncthreads();
	const int ng = blockDim.x / N;
	if ((int)threadIdx.x >= ng * N) return;
	const int kv = threadIdx.x % N;
	for (int l0 = threadIdx.x / N; l0 < N; l0 += 4 * ng) {
		float s[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
		int j = 0;
#pragma unroll 4
		for (int ky = 0; ky < m; ky++) {
			const float2 w = tw[j];
#pragma unroll
			for (int q = 0; q < 4; q++) {
				const int l = min(l0 + q * ng, N - 1);
				const float2 a = U[l * m + ky];
				s[q] = fmaf(a.x, w.x, fmaf(-a.y, w.y, s[q]));
			}
			j += kv;
			if (j >= N) j -= N;
		}
#pragma unroll
		for (int q = 0; q < 4; q++) {
			const int l = l0 + q * ng;
			if (l >= N) continue;
			const long i = bc * P + l * N + kv;
			float v = scale * s[q];
			if (accumulate) v += out[i];
			if (u) v *= dgelu_f(u[i]);
			out[i] = v;
		}
	}
}

// mode mixing: fwd (conj = 0): out[b][o][k] = sum_i R[i][o][k] in[b][i][k]
//              bwd (conj = 1): out[b][i][k] = sum_o conj(R[i][o][k]) in[b][o][k]
// A thread has one k, four output channels and four cells, so the weights and
// the inputs are each read a quarter as often (from L2): 64 cells, 32 channels, 276
// modes: 38 -> 17 us.
__global__ void __launch_bounds__(128) k_fno_mix(int B, int w, int K, const float2 *__restrict__ in, const float *__restrict__ Rr,
                                                 const float *__restrict__ Ri, float2 *__restrict__ out, int conj) {
	const int nc = (w + 3) / 4, nb = (B + 3) / 4;
	const long n = (long)K * nc * nb;
	for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
		const int k = (int)(t % K), c0 = 4 * (int)(t / K % nc), b0 = 4 * (int)(t / ((long)K * nc));
		float re[4][4], im[4][4];
#pragma unroll
		for (int c = 0; c < 4; c++)
#pragma unroll
			for (int b = 0; b < 4; b++) re[c][b] = im[c][b] = 0.0f;
#pragma unroll 4
		for (int j = 0; j < w; j++) {
			float rr[4], ri[4];
			float2 v[4];
#pragma unroll
			for (int c = 0; c < 4; c++) {
				const int cc = min(c0 + c, w - 1);
				const long i = conj ? ((long)cc * w + j) * K + k : ((long)j * w + cc) * K + k;
				rr[c] = Rr[i];
				ri[c] = conj ? -Ri[i] : Ri[i];
			}
#pragma unroll
			for (int b = 0; b < 4; b++) v[b] = in[((long)min(b0 + b, B - 1) * w + j) * K + k];
#pragma unroll
			for (int c = 0; c < 4; c++)
#pragma unroll
				for (int b = 0; b < 4; b++) {
					re[c][b] = fmaf(rr[c], v[b].x, fmaf(-ri[c], v[b].y, re[c][b]));
					im[c][b] = fmaf(rr[c], v[b].y, fmaf(ri[c], v[b].x, im[c][b]));
				}
		}
#pragma unroll
		for (int c = 0; c < 4; c++)
#pragma unroll
			for (int b = 0; b < 4; b++)
				if (c0 + c < w && b0 + b < B) out[((long)(b0 + b) * w + c0 + c) * K + k] = make_float2(re[c][b], im[c][b]);
	}
}

// weight gradient of the mode mixing: dR[i][o][k] = sum_b GO[b][o][k] conj(H[b][i][k]).
// A block has 32 modes and one 4 x 4 block of (i, o); its four warps take a quarter
// of the cells each and add up in that order.  58 -> 28 us (as k_fno_mix)
__global__ void __launch_bounds__(128) k_fno_rgrad(int B, int w, int K, const float2 *__restrict__ GO, const float2 *__restrict__ H,
                                                   float *__restrict__ gRr, float *__restrict__ gRi) {
	__shared__ float2 sh[3][16][32];
	const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5, nt = (w + 3) / 4;
	const int k = blockIdx.x * 32 + lane, kk = min(k, K - 1), i0 = 4 * (blockIdx.y / nt), o0 = 4 * (blockIdx.y % nt);
	float2 acc[4][4];
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int o = 0; o < 4; o++) acc[i][o] = make_float2(0.0f, 0.0f);
	const int b0 = (int)((long)seg * B / 4), b1 = (int)((long)(seg + 1) * B / 4);
#pragma unroll 4
	for (int b = b0; b < b1; b++) {
		float2 g[4], h[4];
#pragma unroll
		for (int o = 0; o < 4; o++) g[o] = GO[((long)b * w + min(o0 + o, w - 1)) * K + kk];
#pragma unroll
		for (int i = 0; i < 4; i++) h[i] = H[((long)b * w + min(i0 + i, w - 1)) * K + kk];
#pragma unroll
		for (int i = 0; i < 4; i++)
#pragma unroll
			for (int o = 0; o < 4; o++) {
				acc[i][o].x = fmaf(g[o].x, h[i].x, fmaf(g[o].y, h[i].y, acc[i][o].x));
				acc[i][o].y = fmaf(g[o].y, h[i].x, fmaf(-g[o].x, h[i].y, acc[i][o].y));
			}
	}
	if (seg > 0) {
#pragma unroll
		for (int i = 0; i < 4; i++)
#pragma unroll
			for (int o = 0; o < 4; o++) sh[seg - 1][4 * i + o][lane] = acc[i][o];
	}
	__syncthreads();
	if (seg > 0 || k >= K) return;
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int o = 0; o < 4; o++) {
			if (i0 + i >= w || o0 + o >= w) continue;
			float2 v = acc[i][o];
#pragma unroll
			for (int q = 0; q < 3; q++) { v.x += sh[q][4 * i + o][lane].x; v.y += sh[q][4 * i + o][lane].y; }
			const long q = ((long)(i0 + i) * w + o0 + o) * K + k;
			gRr[q] = v.x;
			gRi[q] = v.y;
		}
}

// partial[chunk][cx][cy + 1] = sum over the chunk's (b, p) of X[b][a][p] * Y[b][c][p], and
// of X alone at c = cy.  Chunks of kChunk points, staged 64 at a time; a thread of
// the 16 x 16 block has the outputs (ty + 16 i, tx + 16 j).  Fixed order.  32 x 32 channels,
// 65 536 points: 44 us in two launches (the second for the sums of X) -> 26 us.
constexpr int kChunk = 128;
__global__ void __launch_bounds__(256) k_fno_outer(int B, int P, int cx, int cy, const float *__restrict__ X, const float *__restrict__ Y,
                                                   float *__restrict__ partial) {
	constexpr int T = 64, PT = T + 4;                    // points a stage, pitch (rows of 17 x 16 bytes)
	__shared__ __align__(16) float xs[kFnoMaxWidth][PT];
	__shared__ __align__(16) float ys[kFnoMaxWidth + 1][PT];
	const long n = (long)B * P;
	const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, ncy = cy + 1;
	float acc[4][5];
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int j = 0; j < 5; j++) acc[i][j] = 0.0f;
	if (threadIdx.x < T) ys[cy][threadIdx.x] = 1.0f;
	for (int s = 0; s < kChunk; s += T) {
		// four consecutive points are in one cell (P is a multiple of 4)
		const int q4 = 4 * (threadIdx.x & 15);
		const long t = (long)blockIdx.x * kChunk + s + q4;
		const bool ok = t < n;
		const long b = ok ? t / P : 0, p = ok ? t % P : 0;
		float4 v[8];
#pragma unroll
		for (int e = 0; e < 8; e++) {
			const int c = (threadIdx.x >> 4) + 16 * (e & 3), cn = e < 4 ? cx : cy;
			v[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			if (ok && c < cn) v[e] = *reinterpret_cast<const float4 *>((e < 4 ? X : Y) + (b * cn + c) * P + p);
		}
		__syncthreads();
#pragma unroll
		for (int e = 0; e < 8; e++) {
			const int c = (threadIdx.x >> 4) + 16 * (e & 3);
			if (c < (e < 4 ? cx : cy)) *reinterpret_cast<float4 *>(e < 4 ? &xs[c][q4] : &ys[c][q4]) = v[e];
		}
		__syncthreads();
#pragma unroll 2
		for (int q = 0; q < T; q += 4) {
			float4 x[4], y[5];
#pragma unroll
			for (int i = 0; i < 4; i++)
				if (16 * i < cx) x[i] = *reinterpret_cast<const float4 *>(&xs[min(ty + 16 * i, cx - 1)][q]);
#pragma unroll
			for (int j = 0; j < 5; j++)
				if (16 * j < ncy) y[j] = *reinterpret_cast<const float4 *>(&ys[min(tx + 16 * j, cy)][q]);
#pragma unroll
			for (int i = 0; i < 4; i++)
#pragma unroll
				for (int j = 0; j < 5; j++)
					if (16 * i < cx && 16 * j < ncy)
						acc[i][j] = fmaf(x[i].w, y[j].w, fmaf(x[i].z, y[j].z, fmaf(x[i].y, y[j].y, fmaf(x[i].x, y[j].x, acc[i][j]))));
		}
	}
	float *o = partial + (long)blockIdx.x * cx * ncy;
#pragma unroll
	for (int i = 0; i < 4; i++)
#pragma unroll
		for (int j = 0; j < 5; j++)
			if (ty + 16 * i < cx && tx + 16 * j < ncy) o[(ty + 16 * i) * ncy + tx + 16 * j] = acc[i][j];
}

// dM[a][c] = sum over the chunks of partial[.][a][c], db[a] = of partial[.][a][cy], in a
// fixed order: eight segments of chunks for 32 outputs a block, then the segments.
// One thread an output, 1024 chunks: 36 us; 512 chunks in segments: 9 us
__global__ void __launch_bounds__(256) k_fno_reduce(int nchunk, int cx, int cy, const float *__restrict__ partial, float *__restrict__ dM,
                                                    float *__restrict__ db) {
	__shared__ float sh[8][33];
	const int count = cx * (cy + 1), lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
	const int j = blockIdx.x * 32 + lane;
	const int c0 = (int)((long)seg * nchunk / 8), c1 = (int)((long)(seg + 1) * nchunk / 8);
	float s = 0.0f;
	if (j < count) {
#pragma unroll 8
		for (int c = c0; c < c1; c++) s += partial[(long)c * count + j];
	}
	sh[seg][lane] = s;
	__syncthreads();
	if (seg == 0 && j < count) {
		for (int q = 1; q < 8; q++) s += sh[q][lane];
		const int a = j / (cy + 1), c = j % (cy + 1);
		if (c < cy) dM[a * cy + c] = s;
		else db[a] = s;
	}
}

// dy = 2 (y - t / scale) / n, partial[block] = sum of squares (fixed tree)
__global__ void k_fno_loss(int B, int P, const float *__restrict__ y, const double *__restrict__ target, double s0, double s1, double s2,
                           double s3, float *__restrict__ dy, double *__restrict__ partial) {
	__shared__ double sh[256];
	const long n = (long)B * 4 * P;
	const double inv_n = 1.0 / (double)n;
	const double sc[4] = { s0, s1, s2, s3 };
	double acc = 0.0;
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
		const int c = (int)((i / P) % 4);
		const double d = (double)y[i] - target[i] / sc[c];
		acc += d * d;
		dy[i] = (float)(2.0 * d * inv_n);
	}
	sh[threadIdx.x] = acc;
	__syncthreads();
	for (int s = 128; s > 0; s >>= 1) {
		if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
		__syncthreads();
	}
	if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void k_fno_gelu_bwd(long n, const float *__restrict__ u, float *__restrict__ d) {
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) d[i] *= dgelu_f(u[i]);
}

__global__ void k_fno_out(long n, int P, const float *__restrict__ y, double s0, double s1, double s2, double s3, double *__restrict__ C) {
	const double sc[4] = { s0, s1, s2, s3 };
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
		C[i] = (double)y[i] * sc[(i / P) % 4];
}

__global__ void k_fno_adam(long n, float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v, float lr,
                           float b1, float b2, float eps, float c1, float c2) {
	for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
		const float gi = g[i];
		const float mi = b1 * m[i] + (1.0f - b1) * gi;
		const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
		m[i] = mi;
		v[i] = vi;
		w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	}
}

// ---------------------------------------------------------------------------
// The pointwise channel maps on the tensor cores (BF16 operands, FP32
// accumulation): for the points of a tile of 128 (rows of the flattened
// (b, p) index) D[row][n] = sum_k X[row][k] Wt[n][k] with one tcgen05.mma
// of M = 128, N = npad, K = 16 per step.
//   trans = 0 (forward map): X = in[b][k][p] (k < kin = cin), Wt[n][k] = M[n cin + k],
//            out = D + bias (+ add); act: uout = u, hout = gelu(u), else hout = u;
//   trans = 1 (its transpose, backward): X = in[b][k][p] (k < kin = cout),
//            Wt[n][k] = M[k cin + n] (n < nout = cin), hout = D.
// A (128 x 64 BF16) and B (npad x 64 BF16) are K-major with the 128-byte
// swizzle; D is 64 FP32 columns of tensor memory, row r in lane r, read back
// by the thread of that row.  Persistent CTAs of 128 threads stride over the
// tiles.  The MMA completion wait is bounded; a wait that runs out sets the
// error word and leaves the outputs of that tile undefined.
namespace fnomma {
constexpr int kThreads = 128, kRows = 128, kMaxK = 64, kCols = 64;
constexpr uint32_t oA = 0, oB = kRows * 128, kUsed = oB + kMaxK * 128;
// dynamic shared memory: the operands, 1024-byte alignment slack, and enough
// more that at most 7 CTAs share an SM (7 x 64 tensor-memory columns <= 512)
constexpr uint32_t kSmem = 33 * 1024;
static_assert(kUsed + 1024 <= kSmem, "operand tiles fit");
constexpr unsigned kPolls = 1u << 24;
}  // namespace fnomma

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
	__nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
	return *reinterpret_cast<uint32_t *>(&v);
}

__global__ void __launch_bounds__(fnomma::kThreads) k_fno_pointwise_mma(int B, int P, int cin, int cout, int trans,
                                                                         const float *__restrict__ in, const float *__restrict__ M,
                                                                         const float *__restrict__ bias, const float *__restrict__ add,
                                                                         float *__restrict__ uout, float *__restrict__ hout, int act,
                                                                         int *err) {
	using namespace fnomma;
	using namespace qb;
	extern __shared__ unsigned char smem_raw[];
	unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
	__shared__ uint64_t mbar;
	__shared__ uint32_t tslot;
	__shared__ int abort_flag;
	const int tid = threadIdx.x, warp = tid >> 5;
	const int kin = trans ? cout : cin, nout = trans ? cin : cout;
	const int kpad = (kin + 15) & ~15, npad = (nout + 15) & ~15;
	// B: the weights as Wt[n][k], BF16, zero beyond (nout, kin)
	for (int i = tid; i < kMaxK * (kMaxK / 2); i += kThreads) {
		const int n = i / (kMaxK / 2), k = 2 * (i % (kMaxK / 2));
		float w0 = 0.0f, w1 = 0.0f;
		if (n < nout) {
			if (k < kin) w0 = trans ? M[k * cin + n] : M[n * cin + k];
			if (k + 1 < kin) w1 = trans ? M[(k + 1) * cin + n] : M[n * cin + k + 1];
		}
		*reinterpret_cast<uint32_t *>(base + oB + umma::kmajor_off16(n, k)) = pack_bf16x2(w0, w1);
	}
	if (tid == 0) {
		umma::mbar_init(&mbar, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		abort_flag = 0;
	}
	if (warp == 0) tmem_alloc(&tslot, kCols);
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const uint32_t tmem = tslot;
	const uint32_t trow = tmem + ((uint32_t)(32 * warp) << 16);      // this warp's 32 lanes
	uint32_t idesc = 0;
	switch (npad) {
	case 16: idesc = umma::idesc_bf16<128, 16>(); break;
	case 32: idesc = umma::idesc_bf16<128, 32>(); break;
	case 48: idesc = umma::idesc_bf16<128, 48>(); break;
	default: idesc = umma::idesc_bf16<128, 64>(); break;
	}
	const long rows = (long)B * P, ntiles = (rows + kRows - 1) / kRows;
	unsigned phase = 0;
	for (long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
		const long row = tile * kRows + tid;
		const bool live = row < rows;
		const long b = live ? row / P : 0, p = live ? row % P : 0;
		// A: this thread's row (its point), BF16, zero beyond kin
		const float *x = in + b * (long)kin * P + p;
#pragma unroll 4
		for (int k = 0; k < kMaxK; k += 2) {
			const float x0 = (live && k < kin) ? x[(long)k * P] : 0.0f;
			const float x1 = (live && k + 1 < kin) ? x[(long)(k + 1) * P] : 0.0f;
			*reinterpret_cast<uint32_t *>(base + oA + umma::kmajor_off16(tid, k)) = pack_bf16x2(x0, x1);
		}
		umma::fence_async_smem();
		tmem_fence_before();
		__syncthreads();
		tmem_fence_after();
		if (tid == 0) {
			const uint32_t a0 = umma::smem_u32(base + oA), b0 = umma::smem_u32(base + oB);
			for (int k = 0; k < kpad; k += 16)
				umma::mma_f16(tmem, umma::desc_sw128(a0 + 2 * k, 16, 1024), umma::desc_sw128(b0 + 2 * k, 16, 1024), idesc, k > 0 ? 1u : 0u);
			umma::commit(&mbar);
		}
		if (!abort_flag && !umma::mbar_wait(&mbar, phase, kPolls)) {
			abort_flag = 1;
			if (err) atomicExch(err, 1);
		}
		phase ^= 1u;
		tmem_fence_after();
		// epilogue: this thread's row of D, 16 columns at a time
		for (int n0 = 0; n0 < npad; n0 += 16) {
			float d[16];
			umma::tmem_ld16(trow + (uint32_t)n0, d);
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
			if (!live) continue;
#pragma unroll
			for (int j = 0; j < 16; j++) {
				const int n = n0 + j;
				if (n >= nout) break;
				const long oi = (b * nout + n) * (long)P + p;
				float v = d[j];
				if (!trans) {
					if (bias) v += bias[n];
					if (add) v += add[oi];
					if (uout) uout[oi] = v;
					hout[oi] = act ? gelu_f(v) : v;
				} else {
					hout[oi] = v;
				}
			}
		}
		tmem_fence_before();
		__syncthreads();                      // D read and A free before the next tile's MMA
		tmem_fence_after();
	}
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (warp == 0) tmem_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------------------
// A grouped row GEMM on the tensor cores (BF16 operands, FP32 accumulation)
// for the separable truncated DFTs: for each of the
// bm.groups() groups and 128-row tiles of its bm.rows() rows,
// D[row][n] = sum_k A[row][k] Bg[n][k], k < K <= 128, n < Nn <= 128, with A
// read through the loader ld(g, row, k), Bg through bm(g, n, k) (rebuilt when a
// CTA moves to another group), and every row of D handed whole to the
// epilogue ep(g, row, d).  Operands K-major with the 128-byte swizzle in two
// 64-element atoms; D in 128 tensor-memory columns.  Persistent CTAs of 128
// threads; the MMA completion wait is bounded (a wait that runs out sets the
// error word).
namespace fnotc {
constexpr int kThreads = 128, kRows = 128, kMaxK = 128, kMaxN = 128, kCols = 128;
constexpr uint32_t oA = 0, oB = kRows * kMaxK * 2, kUsed = oB + kMaxN * kMaxK * 2;
// operands, alignment slack, and enough more that at most 3 CTAs share an SM (3 x 128 columns <= 512)
constexpr uint32_t kSmem = 72 * 1024;
static_assert(kUsed + 1024 <= kSmem, "operand tiles fit");
constexpr unsigned kPolls = 1u << 24;
__host__ __device__ constexpr uint32_t off(int R, int r, int k) {
	return (uint32_t)((k >> 6) * R * 128) + qb::umma::kmajor_off16(r, k & 63);
}
}  // namespace fnotc

template <class Ld, class Ep, class Bb>
__global__ void __launch_bounds__(fnotc::kThreads) k_fno_tc(const Ld ld, const Ep ep, const Bb bm, int K, int Nn, int *err) {
	using namespace fnotc;
	using namespace qb;
	extern __shared__ unsigned char smem_raw[];
	unsigned char *base = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
	__shared__ uint64_t mbar;
	__shared__ uint32_t tslot;
	__shared__ int abort_flag;
	const int tid = threadIdx.x, warp = tid >> 5;
	const int kpad = (K + 15) & ~15, npad = (Nn + 15) & ~15;
	if (tid == 0) {
		umma::mbar_init(&mbar, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		abort_flag = 0;
	}
	if (warp == 0) tmem_alloc(&tslot, kCols);
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const uint32_t tmem = tslot;
	const uint32_t trow = tmem + ((uint32_t)(32 * warp) << 16);
	const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(npad >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
	const long rows = bm.rows(), tpg = (rows + kRows - 1) / kRows, ntiles = tpg * bm.groups();
	unsigned phase = 0;
	int cur_g = -1;
	for (long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
		const int g = (int)(tile / tpg);
		const long row = (tile % tpg) * kRows + tid;
		const bool live = row < rows;
		if (g != cur_g) {                     // this group's B (the previous MMA has completed)
			for (int i = tid; i < npad * (kpad / 2); i += kThreads) {
				const int n = i / (kpad / 2), k = 2 * (i % (kpad / 2));
				const float b0 = (n < Nn && k < K) ? bm(g, n, k) : 0.0f;
				const float b1 = (n < Nn && k + 1 < K) ? bm(g, n, k + 1) : 0.0f;
				*reinterpret_cast<uint32_t *>(base + oB + off(npad, n, k)) = pack_bf16x2(b0, b1);
			}
			cur_g = g;
		}
		for (int k = 0; k < kpad; k += 2) {
			const float x0 = (live && k < K) ? ld(g, row, k) : 0.0f;
			const float x1 = (live && k + 1 < K) ? ld(g, row, k + 1) : 0.0f;
			*reinterpret_cast<uint32_t *>(base + oA + off(kRows, tid, k)) = pack_bf16x2(x0, x1);
		}
		umma::fence_async_smem();
		tmem_fence_before();
		__syncthreads();
		tmem_fence_after();
		if (tid == 0) {
			const uint32_t a0 = umma::smem_u32(base + oA), b0 = umma::smem_u32(base + oB);
			for (int k = 0; k < kpad; k += 16) {
				const uint32_t ao = (uint32_t)((k >> 6) * kRows * 128 + (k & 63) * 2);
				const uint32_t bo = (uint32_t)((k >> 6) * npad * 128 + (k & 63) * 2);
				umma::mma_f16(tmem, umma::desc_sw128(a0 + ao, 16, 1024), umma::desc_sw128(b0 + bo, 16, 1024), idesc, k > 0 ? 1u : 0u);
			}
			umma::commit(&mbar);
		}
		if (!abort_flag && !umma::mbar_wait(&mbar, phase, kPolls)) {
			abort_flag = 1;
			if (err) atomicExch(err, 1);
		}
		phase ^= 1u;
		tmem_fence_after();
		float d[kMaxN];
#pragma unroll
		for (int c = 0; c < kMaxN / 16; c++) {
			if (16 * c < npad) {
				float v[16];
				umma::tmem_ld16(trow + (uint32_t)(16 * c), v);
				asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
				for (int j = 0; j < 16; j++) d[16 * c + j] = v[j];
			}
		}
		if (live) ep(g, row, d);
		tmem_fence_before();
		__syncthreads();
		tmem_fence_after();
	}
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (warp == 0) tmem_dealloc(tmem, kCols);
}

// the truncated DFT of a field f (N x N real) to H (K complex, kx in [-m+1, m-1],
// ky in [0, m)) as two row GEMMs:
//   1. along kv: T[fld][ky][l] = sum_kv f[fld][l][kv] e^{-2 pi i ky kv / N}   (rows (fld, l), K = N, Nn = 2m)
//   2. along l:  H[fld][kx][ky] = scale sum_l T[fld][ky][l] e^{-2 pi i kx l / N} (rows (fld, ky), K = 2N, Nn = 2(2m-1))
// and its inverse out[fld][l][kv] (=, +=) scale Re sum_k O[fld][k] e^{+i theta}:
//   A. along kx: U[fld][l][ky] = sum_kx O[fld][kx][ky] e^{+2 pi i kx l / N}      (rows (fld, ky), K = 2(2m-1), Nn = 2N)
//   B. along ky: out = scale Re sum_ky U[fld][l][ky] e^{+2 pi i ky kv / N}        (rows (fld, l), K = 2m, Nn = N)
// one fixed FP32 [Nn][K] matrix in global memory (the twiddles) for `nrows` rows
struct BMat {
	const float *Bm; int K; long nrows;
	__device__ long rows() const { return nrows; }
	__device__ int groups() const { return 1; }
	__device__ float operator()(int, int n, int k) const { return Bm[(long)n * K + k]; }
};
struct LdDft1 { const float *f; int N; __device__ float operator()(int, long row, int k) const { return f[row * N + k]; } };
struct EpDft1 {
	float *T; int N, m;
	__device__ void operator()(int, long row, const float (&d)[fnotc::kMaxN]) const {
		const long fld = row / N;
		const int l = (int)(row % N);
		for (int ky = 0; ky < m; ky++) {
			float *t = T + (fld * m + ky) * 2L * N;
			t[l] = d[ky];
			t[N + l] = d[m + ky];
		}
	}
};
struct LdDft2 { const float *T; int N; __device__ float operator()(int, long row, int k) const { return T[row * 2L * N + k]; } };
struct EpDft2 {
	float2 *H; int m; float scale;
	__device__ void operator()(int, long row, const float (&d)[fnotc::kMaxN]) const {
		const int K = (2 * m - 1) * m, nk = 2 * m - 1;
		const long fld = row / m;
		const int ky = (int)(row % m);
		for (int kxi = 0; kxi < nk; kxi++) H[fld * K + kxi * m + ky] = make_float2(scale * d[kxi], scale * d[nk + kxi]);
	}
};
struct LdIdftA {
	const float2 *O; int m;
	__device__ float operator()(int, long row, int k) const {
		const int K = (2 * m - 1) * m, nk = 2 * m - 1;
		const long fld = row / m;
		const int ky = (int)(row % m);
		const float2 o = O[fld * K + (k % nk) * m + ky];
		return k < nk ? o.x : o.y;
	}
};
struct EpIdftA {
	float *U; int N, m;
	__device__ void operator()(int, long row, const float (&d)[fnotc::kMaxN]) const {
		const long fld = row / m;
		const int ky = (int)(row % m);
		for (int l = 0; l < N; l++) {
			float *u = U + (fld * N + l) * 2L * m;
			u[ky] = d[l];
			u[m + ky] = d[N + l];
		}
	}
};
struct LdIdftB { const float *U; int m; __device__ float operator()(int, long row, int k) const { return U[row * 2L * m + k]; } };
struct EpIdftB {
	float *out; int N; float scale; int accumulate;
	__device__ void operator()(int, long row, const float (&d)[fnotc::kMaxN]) const {
		float *o = out + row * N;           // row = fld N + l: out[fld][l][kv]
		for (int kv = 0; kv < N; kv++) o[kv] = accumulate ? o[kv] + scale * d[kv] : scale * d[kv];
	}
};

unsigned grid_for(long n) { return (unsigned)std::max<long>(1, std::min<long>((n + 255) / 256, 148L * 32)); }

}  // namespace

// the tensor-memory kernel of this file, for the engine's co-residency check
std::vector<qb::TmemKernel> qb::fno_tmem_kernels() {
	return { { (const void *)k_fno_pointwise_mma, fnomma::kSmem, fnomma::kThreads, fnomma::kCols, "k_fno_pointwise_mma" },
	         { (const void *)k_fno_tc<LdDft1, EpDft1, BMat>, fnotc::kSmem, fnotc::kThreads, fnotc::kCols, "k_fno_tc<dft 1>" },
	         { (const void *)k_fno_tc<LdDft2, EpDft2, BMat>, fnotc::kSmem, fnotc::kThreads, fnotc::kCols, "k_fno_tc<dft 2>" },
	         { (const void *)k_fno_tc<LdIdftA, EpIdftA, BMat>, fnotc::kSmem, fnotc::kThreads, fnotc::kCols, "k_fno_tc<idft A>" },
	         { (const void *)k_fno_tc<LdIdftB, EpIdftB, BMat>, fnotc::kSmem, fnotc::kThreads, fnotc::kCols, "k_fno_tc<idft B>" } };
}

namespace {

// every launch is counted (and timed while profiling is on) under its kernel's name
template <class... P, class... A>
void launch(const char *name, void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
	qb::ProfScope ps(name, s);
	k<<<grid, block, smem, s>>>(args...);
	QB_CUDA(cudaGetLastError());
}

}  // namespace

struct qb_fno {
	int N = 0, w = 0, m = 0, L = 0, K = 0, P = 0;
	Offsets off;
	double scale[4] = { 1, 1, 1, 1 };
	InScale inscale = { { 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1 } };
	long adam_t = 0;
	qb::DevBuf params, grads, am, av;
	int cap = 0;                                  // batch the activation buffers hold
	qb::DevBuf x, y, dy, dh, tmp, lossp, partial;
	std::vector<qb::DevBuf> h, u, H;             // h[0..L], u[0..L-1], H[0..L-1]
	qb::DevBuf GO, GH;
	int use_tc = 0;                               // pointwise maps and truncated DFTs on the tensor cores (BF16, FP32 accumulation)
	qb::DevBuf kerr;                              // error word of the bounded MMA waits
	qb::DevBuf twn;                               // the N-th roots of unity of the FP32 transforms
	qb::DevBuf twm, tscr, uscr;                   // tensor-core DFTs: the 4 twiddle matrices, stage scratch
	const float *Bm1 = nullptr, *Bm2 = nullptr, *BmA = nullptr, *BmB = nullptr;

	// the twiddle matrices of the two-stage DFT and inverse (FP32 [Nn][K], from FP64)
	void build_twiddles(cudaStream_t s) {
		if (twm.p != nullptr) return;
		const int nk = 2 * m - 1;
		const long n1 = 2L * m * N, n2 = 2L * nk * 2 * N, nA = 2L * N * 2 * nk, nB = (long)N * 2 * m;
		std::vector<float> h(n1 + n2 + nA + nB);
		auto c = [&](long a) { return (float)std::cos(2.0 * M_PI * (double)a / N); };
		auto sn = [&](long a) { return (float)std::sin(2.0 * M_PI * (double)a / N); };
		float *b1 = h.data(), *b2 = b1 + n1, *bA = b2 + n2, *bB = bA + nA;
		for (int n = 0; n < m; n++)
			for (int kv = 0; kv < N; kv++) { b1[n * N + kv] = c((long)n * kv); b1[(m + n) * N + kv] = -sn((long)n * kv); }
		for (int kxi = 0; kxi < nk; kxi++) {
			const int kx = kxi - (m - 1);
			for (int l = 0; l < N; l++) {
				const long a = (long)kx * l;
				b2[kxi * 2L * N + l] = c(a);         b2[kxi * 2L * N + N + l] = sn(a);
				b2[(nk + kxi) * 2L * N + l] = -sn(a); b2[(nk + kxi) * 2L * N + N + l] = c(a);
				bA[l * 2L * nk + kxi] = c(a);        bA[l * 2L * nk + nk + kxi] = -sn(a);
				bA[(N + l) * 2L * nk + kxi] = sn(a); bA[(N + l) * 2L * nk + nk + kxi] = c(a);
			}
		}
		for (int kv = 0; kv < N; kv++)
			for (int ky = 0; ky < m; ky++) { bB[kv * 2L * m + ky] = c((long)ky * kv); bB[kv * 2L * m + m + ky] = -sn((long)ky * kv); }
		twm.ensure(sizeof(float) * h.size());
		QB_CUDA(cudaMemcpyAsync(twm.p, h.data(), sizeof(float) * h.size(), cudaMemcpyHostToDevice, s));
		QB_CUDA(cudaStreamSynchronize(s));
		Bm1 = twm.as<float>(); Bm2 = Bm1 + n1; BmA = Bm2 + n2; BmB = BmA + nA;
	}

	template <class Ld, class Ep, class Bb> void row_gemm(const char *name, const Ld &ld, const Ep &ep, const Bb &bm, long tiles, int K, int Nn,
	                                                      cudaStream_t s) {
		static int attr_done[64] = {};
		int dev = 0;
		QB_CUDA(cudaGetDevice(&dev));
		if (!attr_done[dev & 63]) {
			qb::ensure_tmem_coresidency();
			QB_CUDA(cudaFuncSetAttribute(k_fno_tc<Ld, Ep, Bb>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fnotc::kSmem));
			attr_done[dev & 63] = 1;
		}
		const unsigned grid = (unsigned)std::max<long>(1, std::min<long>(tiles, 148L * 3));
		launch(name, k_fno_tc<Ld, Ep, Bb>, grid, fnotc::kThreads, (size_t)fnotc::kSmem, s, ld, ep, bm, K, Nn, kerr.as<int>());
	}

	// H[fld] = scale DFT(f[fld]) for the B w fields
	void dft(int B, const float *f, float2 *Hout, float scale, cudaStream_t s) {
		if (!use_tc) {
			launch("fno_dft", k_fno_dft, (unsigned)(B * w), 256, dft_smem(), s, N, m, f, twn.as<float2>(), Hout, scale);
			return;
		}
		ensure_err(s);
		build_twiddles(s);
		const long nf = (long)B * w;
		row_gemm("fno_dft_tc", LdDft1{ f, N }, EpDft1{ tscr.as<float>(), N, m }, BMat{ Bm1, N, nf * N }, (nf * N + 127) / 128, N, 2 * m, s);
		row_gemm("fno_dft_tc", LdDft2{ tscr.as<float>(), N }, EpDft2{ Hout, m, scale }, BMat{ Bm2, 2 * N, nf * m }, (nf * m + 127) / 128,
		         2 * N, 2 * (2 * m - 1), s);
	}
	// out[fld] (=, +=) scale Re IDFT(O[fld]), then times dgelu(u) when u is given
	void idft(int B, const float2 *O, float *out, float scale, int accumulate, const float *u, cudaStream_t s) {
		if (!use_tc) {
			launch("fno_idft", k_fno_idft, (unsigned)(B * w), 256, idft_smem(), s, N, m, O, twn.as<float2>(), out, scale, accumulate, u);
			return;
		}
		ensure_err(s);
		build_twiddles(s);
		const long nf = (long)B * w;
		row_gemm("fno_idft_tc", LdIdftA{ O, m }, EpIdftA{ uscr.as<float>(), N, m }, BMat{ BmA, 2 * (2 * m - 1), nf * m }, (nf * m + 127) / 128,
		         2 * (2 * m - 1), 2 * N, s);
		row_gemm("fno_idft_tc", LdIdftB{ uscr.as<float>(), m }, EpIdftB{ out, N, scale, accumulate }, BMat{ BmB, 2 * m, nf * N },
		         (nf * N + 127) / 128, 2 * m, N, s);
		const long nw = (long)B * w * P;
		if (u != nullptr) launch("fno_gelu_bwd", k_fno_gelu_bwd, grid_for(nw), 256, 0, s, nw, u, out);
	}
	// mode mixing: out[b][c][k] = sum over the other channel of R (or conj R, backward) times in;
	// FP32 in both modes (on the tensor cores, with a mode's matrix built for
	// each 128 cells, 117 us against 48 for 256 cells, 706 against 318 for 2048)
	void mix(int B, const float2 *in, const float *Rr, const float *Ri, float2 *out, int conj, cudaStream_t s) {
		launch("fno_mix", k_fno_mix, grid_for(2L * K * ((w + 3) / 4) * ((B + 3) / 4)), 128, 0, s, B, w, K, in, Rr, Ri, out, conj);
	}
	void ensure_err(cudaStream_t s) {
		if (kerr.p == nullptr) {
			kerr.ensure(sizeof(int));
			QB_CUDA(cudaMemsetAsync(kerr.p, 0, sizeof(int), s));
		}
	}

	float *P_(long o) { return params.as<float>() + o; }

	// out = M in + bias (+ add), gelu when act (uout keeps the pre-activation)
	void pointwise(int B, int cin, int cout, const float *in, const float *M, const float *bias, const float *add, float *uout,
	               float *hout, int act, cudaStream_t s) {
		if (use_tc) pointwise_mma(B, cin, cout, 0, in, M, bias, add, uout, hout, act, s);
		else pointwise_f32(B, cin, cout, 0, in, M, bias, add, uout, hout, act, s);
	}
	// grid: a thread a point; two (four) blocks share the outputs of a point while the
	// points alone do not fill the GPU twice
	void pointwise_f32(int B, int cin, int cout, int trans, const float *in, const float *M, const float *bias, const float *add, float *uout,
	                   float *hout, int act, cudaStream_t s) {
		auto go = [&](auto kern) {
			const unsigned gx = grid_for((long)B * P);
			const dim3 g(gx, gx < 1200 ? std::max(1, std::min(4, cout / 4)) : 1);
			qb::ProfScope ps("fno_pointwise", s);
			kern<<<g, 256, 0, s>>>(B, P, cin, cout, trans, in, M, bias, add, uout, hout, act);
			QB_CUDA(cudaGetLastError());
		};
		if (cin <= 4) go(k_fno_pointwise<4>);
		else if (cin <= 16) go(k_fno_pointwise<16>);
		else if (cin <= 32) go(k_fno_pointwise<32>);
		else go(k_fno_pointwise<64>);
	}
	// out = M^T in (the backward of a pointwise map)
	void pointwise_t(int B, int cin, int cout, const float *in, const float *M, float *out, cudaStream_t s) {
		if (use_tc) pointwise_mma(B, cin, cout, 1, in, M, nullptr, nullptr, nullptr, out, 0, s);
		else pointwise_f32(B, cout, cin, 1, in, M, nullptr, nullptr, nullptr, out, 0, s);
	}
	void pointwise_mma(int B, int cin, int cout, int trans, const float *in, const float *M, const float *bias, const float *add,
	                   float *uout, float *hout, int act, cudaStream_t s) {
		static int attr_done[64] = {};
		int dev = 0;
		QB_CUDA(cudaGetDevice(&dev));
		if (!attr_done[dev & 63]) {
			qb::ensure_tmem_coresidency();
			QB_CUDA(cudaFuncSetAttribute(k_fno_pointwise_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fnomma::kSmem));
			attr_done[dev & 63] = 1;
		}
		ensure_err(s);
		const long tiles = ((long)B * P + fnomma::kRows - 1) / fnomma::kRows;
		const unsigned grid = (unsigned)std::max<long>(1, std::min<long>(tiles, 148L * 7));
		launch("fno_pointwise_mma", k_fno_pointwise_mma, grid, fnomma::kThreads, (size_t)fnomma::kSmem, s, B, P, cin, cout, trans, in, M,
		       bias, add, uout, hout, act, kerr.as<int>());
	}
	float *G_(long o) { return grads.as<float>() + o; }

	void reserve(int B) {
		if (B <= cap) return;
		const long f = (long)B * w * P;
		x.ensure(sizeof(float) * B * (long)kFnoIn * P);
		y.ensure(sizeof(float) * B * 4L * P);
		dy.ensure(sizeof(float) * B * 4L * P);
		dh.ensure(sizeof(float) * f);
		tmp.ensure(sizeof(float) * f);
		h.resize(L + 1);
		u.resize(L);
		H.resize(L);
		for (int l = 0; l <= L; l++) h[l].ensure(sizeof(float) * f);
		for (int l = 0; l < L; l++) { u[l].ensure(sizeof(float) * f); H[l].ensure(sizeof(float2) * (long)B * w * K); }
		GO.ensure(sizeof(float2) * (long)B * w * K);
		GH.ensure(sizeof(float2) * (long)B * w * K);
		tscr.ensure(sizeof(float) * (long)B * w * m * 2 * N);
		uscr.ensure(sizeof(float) * (long)B * w * N * 2 * m);
		const long nchunk = ((long)B * P + kChunk - 1) / kChunk;
		partial.ensure(sizeof(float) * nchunk * kFnoMaxWidth * (kFnoMaxWidth + 1));
		lossp.ensure(sizeof(double) * 4096);
		cap = B;
	}

	size_t dft_smem() const { return sizeof(float) * (long)N * (N + 1) + sizeof(float2) * ((long)N * m + N); }
	size_t idft_smem() const { return sizeof(float2) * (2L * m * m + (long)N * m + N); }

	void forward(int B, const double *W, cudaStream_t s) {
		reserve(B);
		launch("fno_in", k_fno_in, grid_for((long)B * P), 256, 0, s, B, P, W, inscale, x.as<float>());
		pointwise(B, kFnoIn, w, x.as<float>(), P_(off.A), P_(off.a), nullptr, nullptr, h[0].as<float>(), 0, s);
		for (int l = 0; l < L; l++) {
			dft(B, h[l].as<float>(), H[l].as<float2>(), 1.0f, s);
			mix(B, H[l].as<float2>(), P_(off.Rr[l]), P_(off.Ri[l]), GO.as<float2>(), 0, s);
			idft(B, GO.as<float2>(), tmp.as<float>(), 1.0f / (float)P, 0, nullptr, s);
			pointwise(B, w, w, h[l].as<float>(), P_(off.W[l]), P_(off.b[l]), tmp.as<float>(), u[l].as<float>(), h[l + 1].as<float>(),
			          l < L - 1 ? 1 : 0, s);
		}
		pointwise(B, w, 4, h[L].as<float>(), P_(off.Q), P_(off.q), nullptr, nullptr, y.as<float>(), 0, s);
		QB_CUDA(cudaGetLastError());
	}

	// gradient of the pointwise map `out = M in + bias`: dM = sum dout in^T, dbias = sum dout
	void pw_grads(int B, int cin, int cout, const float *in, const float *dout, long offM, long offb, cudaStream_t s) {
		const long n = (long)B * P;
		const int nchunk = (int)((n + kChunk - 1) / kChunk);
		launch("fno_outer", k_fno_outer, nchunk, 256, 0, s, B, P, cout, cin, dout, in, partial.as<float>());
		launch("fno_reduce", k_fno_reduce, (cout * (cin + 1) + 31) / 32, 256, 0, s, nchunk, cout, cin, partial.as<float>(), G_(offM), G_(offb));
	}

	double loss_backward(int B, const double *target, cudaStream_t s) {
		const long n4 = (long)B * 4 * P;
		const int lb = 512;
		launch("fno_loss", k_fno_loss, lb, 256, 0, s, B, P, y.as<float>(), target, scale[0], scale[1], scale[2], scale[3], dy.as<float>(), lossp.as<double>());
		// projection
		pw_grads(B, w, 4, h[L].as<float>(), dy.as<float>(), off.Q, off.q, s);
		pointwise_t(B, w, 4, dy.as<float>(), P_(off.Q), dh.as<float>(), s);
		for (int l = L - 1; l >= 0; l--) {
			// dh holds du of layer l (the layers below the last have had their dgelu factor)
			pw_grads(B, w, w, h[l].as<float>(), dh.as<float>(), off.W[l], off.b[l], s);
			dft(B, dh.as<float>(), GO.as<float2>(), 1.0f / (float)P, s);
			{
				const unsigned nt = (unsigned)((w + 3) / 4);
				qb::ProfScope ps("fno_rgrad", s);
				k_fno_rgrad<<<dim3((unsigned)((K + 31) / 32), nt * nt), 128, 0, s>>>(B, w, K, GO.as<float2>(), H[l].as<float2>(), G_(off.Rr[l]), G_(off.Ri[l]));
				QB_CUDA(cudaGetLastError());
			}
			mix(B, GO.as<float2>(), P_(off.Rr[l]), P_(off.Ri[l]), GH.as<float2>(), 1, s);
			pointwise_t(B, w, w, dh.as<float>(), P_(off.W[l]), tmp.as<float>(), s);
			idft(B, GH.as<float2>(), tmp.as<float>(), 1.0f, 1, l > 0 ? u[l - 1].as<float>() : nullptr, s);
			std::swap(dh, tmp);
		}
		// lift
		pw_grads(B, kFnoIn, w, x.as<float>(), dh.as<float>(), off.A, off.a, s);
		QB_CUDA(cudaGetLastError());
		std::vector<double> lp(lb);
		QB_CUDA(cudaMemcpyAsync(lp.data(), lossp.p, sizeof(double) * lb, cudaMemcpyDeviceToHost, s));
		QB_CUDA(cudaStreamSynchronize(s));
		double l2 = 0;
		for (double v : lp) l2 += v;
		return l2 / (double)n4;
	}
};

namespace {
// splitmix64 normal variates for the initial weights
struct Rng {
	unsigned long long s;
	unsigned long long next() {
		unsigned long long z = (s += 0x9E3779B97F4A7C15ULL);
		z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
		z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
		return z ^ (z >> 31);
	}
	double uniform() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
	double normal() { return std::sqrt(-2.0 * std::log(uniform())) * std::cos(6.283185307179586 * uniform()); }
};

template <class F> int fno_guard(F &&f) {
	try {
		f();
		return 0;
	} catch (const std::exception &) {
		return -1;
	}
}
}  // namespace

extern "C" {

qb_fno *qb_fno_create(int N, int width, int modes, int layers, unsigned long long seed) {
	qb_fno *net = nullptr;
	fno_guard([&] {
		if (N < 4 || N > 64 || (N & 1)) QB_FAIL("qb_fno_create: N must be even, 4..64");
		if (width < 1 || width > kFnoMaxWidth) QB_FAIL("qb_fno_create: width must be 1..64");
		if (modes < 1 || 2 * modes - 1 > N) QB_FAIL("qb_fno_create: need 1 <= modes and 2 modes - 1 <= N");
		if (layers < 1 || layers > 16) QB_FAIL("qb_fno_create: layers must be 1..16");
		auto n = std::make_unique<qb_fno>();
		n->N = N; n->w = width; n->m = modes; n->L = layers; n->K = (2 * modes - 1) * modes; n->P = N * N;
		n->off = offsets(width, n->K, layers);
		const long np = n->off.total;
		std::vector<float> p(np, 0.0f);
		Rng r{ seed };
		auto fill = [&](long o, long cnt, double sd) { for (long i = 0; i < cnt; i++) p[o + i] = (float)(sd * r.normal()); };
		fill(n->off.A, (long)kFnoIn * width, std::sqrt(1.0 / kFnoIn));
		for (int l = 0; l < layers; l++) {
			fill(n->off.Rr[l], (long)width * width * n->K, 1.0 / width);
			fill(n->off.Ri[l], (long)width * width * n->K, 1.0 / width);
			fill(n->off.W[l], (long)width * width, std::sqrt(1.0 / width));
		}
		fill(n->off.Q, 4L * width, std::sqrt(1.0 / width));
		n->params.ensure(sizeof(float) * np);
		n->grads.ensure(sizeof(float) * np);
		n->am.ensure(sizeof(float) * np);
		n->av.ensure(sizeof(float) * np);
		QB_CUDA(cudaMemcpy(n->params.p, p.data(), sizeof(float) * np, cudaMemcpyHostToDevice));
		QB_CUDA(cudaMemset(n->am.p, 0, sizeof(float) * np));
		QB_CUDA(cudaMemset(n->av.p, 0, sizeof(float) * np));
		QB_CUDA(cudaMemset(n->grads.p, 0, sizeof(float) * np));
		std::vector<float2> tw(N);
		for (int j = 0; j < N; j++) tw[j] = make_float2((float)std::cos(2.0 * M_PI * j / N), (float)std::sin(2.0 * M_PI * j / N));
		n->twn.ensure(sizeof(float2) * N);
		QB_CUDA(cudaMemcpy(n->twn.p, tw.data(), sizeof(float2) * N, cudaMemcpyHostToDevice));
		net = n.release();
	});
	return net;
}

void qb_fno_free(qb_fno *net) { delete net; }

long qb_fno_num_params(const qb_fno *net) { return net ? net->off.total : -1; }

int qb_fno_grid_size(const qb_fno *net) { return net ? net->N : -1; }

int qb_fno_get_params(const qb_fno *net, float *host) {
	return fno_guard([&] {
		if (net == nullptr || host == nullptr) QB_FAIL("qb_fno_get_params: null network or buffer");
		QB_CUDA(cudaMemcpy(host, net->params.p, sizeof(float) * net->off.total, cudaMemcpyDeviceToHost));
	});
}

int qb_fno_set_params(qb_fno *net, const float *host) {
	return fno_guard([&] {
		if (net == nullptr || host == nullptr) QB_FAIL("qb_fno_set_params: null network or buffer");
		QB_CUDA(cudaMemcpy(net->params.p, host, sizeof(float) * net->off.total, cudaMemcpyHostToDevice));
	});
}

int qb_fno_set_scale(qb_fno *net, const double *scale) {
	return fno_guard([&] {
		if (net == nullptr || scale == nullptr) QB_FAIL("qb_fno_set_scale: null network or scales");
		for (int c = 0; c < 4; c++) {
			if (!(scale[c] > 0)) QB_FAIL("qb_fno_set_scale: scales must be positive");
			net->scale[c] = scale[c];
		}
	});
}

int qb_fno_set_input_scale(qb_fno *net, const double *scale) {
	return fno_guard([&] {
		if (net == nullptr || scale == nullptr) QB_FAIL("qb_fno_set_input_scale: null network or scales");
		for (int f = 0; f < kFnoIn; f++) {
			if (!(scale[f] > 0)) QB_FAIL("qb_fno_set_input_scale: scales must be positive");
			net->inscale.s[f] = scale[f];
		}
	});
}

int qb_fno_set_tensor_cores(qb_fno *net, int on) {
	return fno_guard([&] {
		if (net == nullptr) QB_FAIL("qb_fno_set_tensor_cores: null network");
		net->use_tc = on ? 1 : 0;
	});
}

int qb_fno_device_errors(const qb_fno *net) {
	int h = 0;
	if (net == nullptr || net->kerr.p == nullptr) return 0;
	if (cudaMemcpy(&h, net->kerr.p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
	return h;
}

int qb_fno_forward(qb_fno *net, int batch, const double *W, double *C, void *stream) {
	return fno_guard([&] {
		if (batch <= 0) return;
		if (net == nullptr || W == nullptr || C == nullptr) QB_FAIL("qb_fno_forward: null network or state");
		cudaStream_t s = (cudaStream_t)stream;
		net->forward(batch, W, s);
		const long n4 = (long)batch * 4 * net->P;
		launch("fno_out", k_fno_out, grid_for(n4), 256, 0, s, n4, net->P, net->y.as<float>(), net->scale[0], net->scale[1], net->scale[2], net->scale[3], C);
		QB_CUDA(cudaGetLastError());
	});
}

int qb_fno_gradients(qb_fno *net, int batch, const double *W, const double *target, float *grad_host, double *loss, void *stream) {
	return fno_guard([&] {
		if (batch <= 0) QB_FAIL("qb_fno_gradients: empty batch");
		if (net == nullptr || W == nullptr || target == nullptr) QB_FAIL("qb_fno_gradients: null network, state or target");
		cudaStream_t s = (cudaStream_t)stream;
		net->forward(batch, W, s);
		const double l = net->loss_backward(batch, target, s);
		if (loss) *loss = l;
		if (grad_host) {
			QB_CUDA(cudaMemcpyAsync(grad_host, net->grads.p, sizeof(float) * net->off.total, cudaMemcpyDeviceToHost, s));
			QB_CUDA(cudaStreamSynchronize(s));
		}
	});
}

int qb_fno_train_step(qb_fno *net, int batch, const double *W, const double *target, float lr, double *loss, void *stream) {
	return fno_guard([&] {
		if (batch <= 0) QB_FAIL("qb_fno_train_step: empty batch");
		if (net == nullptr || W == nullptr || target == nullptr) QB_FAIL("qb_fno_train_step: null network, state or target");
		cudaStream_t s = (cudaStream_t)stream;
		net->forward(batch, W, s);
		const double l = net->loss_backward(batch, target, s);
		if (loss) *loss = l;
		net->adam_t++;
		const float b1 = 0.9f, b2 = 0.999f;
		const float c1 = 1.0f - std::pow(b1, (float)net->adam_t), c2 = 1.0f - std::pow(b2, (float)net->adam_t);
		launch("fno_adam", k_fno_adam, grid_for(net->off.total), 256, 0, s, net->off.total, net->params.as<float>(), net->grads.as<float>(), net->am.as<float>(),
		                                                    net->av.as<float>(), lr, b1, b2, 1e-8f, c1, c2);
		QB_CUDA(cudaGetLastError());
	});
}

}  // extern "C"
