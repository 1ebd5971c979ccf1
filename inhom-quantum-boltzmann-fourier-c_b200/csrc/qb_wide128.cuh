// qb_wide128.cuh — the real form of the FP32 I3 sums at N = 64 with 32 values a
// thread.
//
// 512 threads hold a 128 x 128 complex FP32 grid, 32 values a thread, and transform
// it in three register stages with two exchanges through shared memory (128 = 32 4
// in both dimensions; the stages, the swizzle and the in-place exchanges are those
// of qb_wide64.cuh with 16 replaced by 32):
//   A  thread (l, tau), values k = tau + 4 r:             DFT32 over r -> q
//   B  item (q, lam), values (l = lam + 32 s, tau):       x w128^(tau q), DFT4 over tau
//      -> p and over s -> u, x w128^(lam u); two items a thread
//   C  thread (q + 32 p, u), values lam:                  DFT32 over lam -> v
// gives b(u + 4 v, q + 32 p).  With 8 values a thread (qb_full128.cuh) a transform
// takes three exchanges and two lane-pair shuffles.
#pragma once
#include "qb_full128.cuh"
#include "qb_wide64.cuh"

namespace qb {

// cos of 2 pi m / 32, folded to constants
__host__ __device__ constexpr double cos32(int m) {
	constexpr double q[9] = { 1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708, 0.70710678118654752440,
		                      0.55557023301960222474, 0.38268343236508977173, 0.19509032201612826785, 0.0 };
	m &= 31;
	return m <= 8 ? q[m] : m <= 16 ? -q[16 - m] : m <= 24 ? -q[m - 16] : q[32 - m];
}
// 32-point DFT in registers: natural order in, frequency f in x[pos32(f)]
__host__ __device__ constexpr int pos32(int f) { return (f & 3) * 8 + (f >> 2); }
template <int DIR> __device__ __forceinline__ void dft32(float2 (&x)[32]) {
#pragma unroll
	for (int n = 0; n < 8; n++) {
		dft4<DIR>(x[n], x[n + 8], x[n + 16], x[n + 24]);
#pragma unroll
		for (int k = 1; k < 4; k++) {                    // partial frequency k of residue n, times w32^(n k)
			if (n == 0) continue;
			float2 w;
			w.x = (float)cos32(n * k);
			w.y = (float)(DIR < 0 ? -cos32(n * k + 24) : cos32(n * k + 24));
			x[n + 8 * k] = cmul(x[n + 8 * k], w);
		}
	}
#pragma unroll
	for (int k = 0; k < 4; k++) {                        // frequency k + 4 m in x[8 k + m]
		float2 v[8];
#pragma unroll
		for (int n = 0; n < 8; n++) v[n] = x[8 * k + n];
		dft8<DIR>(v);
#pragma unroll
		for (int m = 0; m < 8; m++) x[8 * k + m] = v[m];
	}
}

struct Wide128 {
	static constexpr int P = 128, PP = P * P, NT = 512;
	float2 *U;
	const float2 *tw;                        // w128^e, e < 128, forward sign
	int t;
	__device__ __forceinline__ static int sw(int row) { return ((row & 3) << 2) | ((row >> 2) & 3); }
	__device__ __forceinline__ int row_a() const { return t >> 2; }
	__device__ __forceinline__ int col_a() const { return t & 3; }
	__device__ __forceinline__ int col_c() const { const int c = t & 127; return (c >> 2) + 32 * (c & 3); }
	__device__ __forceinline__ int row_c() const { return t >> 7; }
	template <class F> __device__ __forceinline__ void slots_a(const F &f) const {
		const int l = t >> 2, s = sw(l), b = l * P;
#pragma unroll
		for (int q = 0; q < 32; q++) f(q, U[b + (((t & 3) + 4 * (q & 3)) ^ s) + 16 * (q >> 2)]);
	}
	template <class F> __device__ __forceinline__ void slots_c(const F &f) const {
		const int c = t & 127, b = (t >> 7) * 32 * P;
#pragma unroll
		for (int m = 0; m < 32; m++) f(m, U[b + m * P + (c ^ sw(m))]);
	}
	template <int DIR> __device__ __forceinline__ void stage_b() const {
#pragma unroll
		for (int it = 0; it < 2; it++) {
			const int item = t + it * NT, q = item >> 5, lam = item & 31, s = sw(lam), b = lam * P + 16 * (q >> 2), h = 4 * (q & 3);
			float2 y[4][4], wq[3], wl[3];
#pragma unroll
			for (int c = 0; c < 4; c++)
#pragma unroll
				for (int r = 0; r < 4; r++) y[r][c] = U[b + ((c + h) ^ s) + 32 * P * r];
#pragma unroll
			for (int m = 0; m < 3; m++) {
				wq[m] = tw[(m + 1) * q];
				wl[m] = tw[(m + 1) * lam];
				if (DIR > 0) { wq[m].y = -wq[m].y; wl[m].y = -wl[m].y; }
			}
			const float2 (&w0)[3] = DIR > 0 ? wq : wl, (&w1)[3] = DIR > 0 ? wl : wq;
#pragma unroll
			for (int i = 0; i < 4; i++)
#pragma unroll
				for (int m = 1; m < 4; m++) {
					if (DIR > 0) y[i][m] = cmul(y[i][m], w0[m - 1]);
					else y[m][i] = cmul(y[m][i], w0[m - 1]);
				}
#pragma unroll
			for (int r = 0; r < 4; r++) dft4<DIR>(y[r][0], y[r][1], y[r][2], y[r][3]);
#pragma unroll
			for (int c = 0; c < 4; c++) dft4<DIR>(y[0][c], y[1][c], y[2][c], y[3][c]);
#pragma unroll
			for (int i = 0; i < 4; i++)
#pragma unroll
				for (int m = 1; m < 4; m++) {
					if (DIR > 0) y[m][i] = cmul(y[m][i], w1[m - 1]);
					else y[i][m] = cmul(y[i][m], w1[m - 1]);
				}
#pragma unroll
			for (int c = 0; c < 4; c++)
#pragma unroll
				for (int r = 0; r < 4; r++) U[b + ((c + h) ^ s) + 32 * P * r] = y[r][c];
		}
	}
};

// real grids in the vector order of A (value r = 4 h + e of thread t at 2048 h + 4 t +
// e): the real parts of the B-layout spectra
__global__ void __launch_bounds__(256) k_w128_real(const float2 *__restrict__ w, float *__restrict__ o) {
	const long g = (long)blockIdx.y * Wide128::PP;
	const int i = blockIdx.x * 256 + threadIdx.x, t = (i >> 2) & 511, r = 4 * (i >> 11) + (i & 3);
	o[g + i] = w[g + F128::brow(t >> 2) + (t & 3) + 4 * r].x;
}
// the transposed psi2 tables ([k][l]) in the vector order of C (value v of thread t)
__global__ void __launch_bounds__(256) k_psi128_real(const float *__restrict__ p, float *__restrict__ o) {
	const long g = (long)blockIdx.y * Wide128::PP;
	const int i = blockIdx.x * 256 + threadIdx.x, t = (i >> 2) & 511, v = 4 * (i >> 11) + (i & 3), c = t & 127;
	o[g + i] = p[g + ((c >> 2) + 32 * (c & 3)) * 128 + (t >> 7) + 4 * v];
}

// Real form of the I3 sums at N = 64 (the identity and what is dropped: see
// qb_full128.cuh): 2-CTA clusters, CTA r for components 2r, 2r + 1.  Per unit one
// transform of psi1 . (W_2r + i W_2r+1) gives P_2r and P_2r+1 (to L2, vector order of
// A); after a cluster barrier, for c = 0, 1 and both outputs j one packed chain of
// P_j . (W^_2c + i W^_2c+1), X_j in tensor memory, and for the other term of a pair
// Y_2c + i Y_2c+1 = sum_j eta_j W^_j . T (the first j waits in tensor memory), transformed
// into A_c = Z_2c + i Z_2c+1 on the frequencies -N/2 .. N/2 (zscr) and separated at the
// end.  WhR: real parts of W^ in vector order; psi2: in that of C; pscr: [cluster][8][PP]
// reals, the first four used; out: [slot][4][PP] B layout, zout: [slot][rank][4][N*N].
// Strang step of 32 cells, J = M = 32: 50.8 -> 40.5 ms against 8 values a thread
// (k_i3 kernels 43 -> 33 ms; shared-memory pipe 48%, issue 35%: latency of its L2 operands).
__global__ void __launch_bounds__(512, 1) k_i3_wide128r(const I3ParamsT<float2> p, const float *__restrict__ WhR, const float *__restrict__ psi2, float *pscr,
                                                        const int *kind) {
	using C = float2;
	using TM = F128TmemR;
	constexpr int N = 64, NN = N * N, P = 128, PP = P * P, H = N / 2, ZA = (N + 1) * (N + 1);
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned tmem_slot;
	C *U = reinterpret_cast<C *>(smem_raw), *tw = U + PP;
	cg::cluster_group cl = cg::this_cluster();
	const int rank = (int)cl.block_rank();
	const long cid = blockIdx.x / 2;
	const int chunk = (int)(cid % p.nchunk);
	const long cell = cid / p.nchunk;
	if (kind[cell] != 0) return;                             // both CTAs of the cluster leave before any barrier
	const int t = threadIdx.x, warp = t >> 5;
	if (warp == 0) tmem_alloc(&tmem_slot, TM::NCOLS);
	init_twiddles<128>(tw);
	const long slot = cell * p.nchunk + chunk;
	double2 *za = p.zscr + (slot * 2 + rank) * 2 * (long)ZA;
	for (int i = t; i < 2 * ZA; i += 512) za[i] = czero();
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const unsigned tbase = tmem_slot;
	{
		const float z[8] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
#pragma unroll 1
		for (int q = 0; q < 2; q++)
#pragma unroll 1
			for (int h = 0; h < 4; h++) tmem_st8r(TM::addr(tbase, q, h), z);
	}
	tmem_wait_st();
	const Wide128 F{ U, tw, t };
	const int kc = F.col_c(), ks = kc < H ? kc : (kc >= P - H ? kc - N : -1), zk = kc <= H ? kc : kc - P;
	float *Pall = pscr + cid * 8 * PP + 4 * t;
	const float *Wc = WhR + cell * 4 * PP + 4 * t;
	const double2 *sa = p.src + cell * p.src_cell + (long)p.src_comp[2 * rank] * NN + F.row_c() * N + ks;
	const double2 *sb = p.src + cell * p.src_cell + (long)p.src_comp[2 * rank + 1] * NN + F.row_c() * N + ks;
	auto ld4 = [](const float *a, int h) { return *reinterpret_cast<const float4 *>(a + 2048 * h); };
	auto ld4g = [](const float *a, int h) { return __ldcg(reinterpret_cast<const float4 *>(a + 2048 * h)); };
	const int u0 = (int)((long)chunk * p.nterms / p.nchunk), u1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
#pragma unroll 1
	for (int un = u0; un < u1; un++) {
		const int term = p.un.term(un);
		const bool pr = p.un.pair(un);
		const C *psi1 = p.psi1 + (long)term * NN;
		C x[32];
		// P_2rank + i P_2rank+1 = FFT2(Pad(psi1 . (W_2rank + i W_2rank+1)))
#pragma unroll
		for (int v = 0; v < 32; v++) x[v] = czero<C>();
		if (ks >= 0) {
#pragma unroll
			for (int v = 0; v < 16; v++) {                   // rows u + 4 v: v < 8 and v >= 24
				const int o = 4 * v * N;
				const double2 a = sa[o], b = sb[o];
				x[v < 8 ? v : v + 16] = cmul(psi1[F.row_c() * N + ks + o], mk<C>(a.x - b.y, a.y + b.x));
			}
		}
		dft32<-1>(x);
		F.slots_c([&](int m, C &v) { v = x[pos32(m)]; });
		__syncthreads();
		F.stage_b<-1>();
		__syncthreads();
		F.slots_a([&](int q, const C &v) { x[q] = v; });
		dft32<-1>(x);
		{
			float *Pa = Pall + 2 * rank * PP;
#pragma unroll
			for (int h = 0; h < 8; h++) {
				const C a = x[pos32(4 * h)], b = x[pos32(4 * h + 1)], c = x[pos32(4 * h + 2)], d = x[pos32(4 * h + 3)];
				__stcg(reinterpret_cast<float4 *>(Pa + 2048 * h), make_float4(a.x, b.x, c.x, d.x));
				__stcg(reinterpret_cast<float4 *>(Pa + PP + 2048 * h), make_float4(a.y, b.y, c.y, d.y));
			}
		}
		cl.sync();                                           // both CTAs' spectra are in L2
		const float *ps = psi2 + (long)p.psi2_idx[term] * PP + 4 * t;
		const float sc = (float)p.psi2_scale[term];
#pragma unroll 1
		for (int c = 0; c < 2; c++) {
			const float *W0 = Wc + 2 * c * PP, *P0 = Pall + 2 * c * PP;
			const float c0 = c == 0 ? sc : -sc;              // eta_2c; eta_2c+1 = -1
#pragma unroll 1
			for (int q = 0; q < 2; q++) {
				const int j = 2 * rank + q;
				const float *Pj = Pall + j * PP, *Wj = Wc + j * PP;
				const float cj = j == 0 ? sc : -sc;          // eta_j
#pragma unroll
				for (int h = 0; h < 8; h++) {
					const float4 a = ld4(W0, h), b = ld4(W0 + PP, h), f = ld4g(Pj, h);
					x[4 * h] = mk<C>(f.x * a.x, f.x * b.x);
					x[4 * h + 1] = mk<C>(f.y * a.y, f.y * b.y);
					x[4 * h + 2] = mk<C>(f.z * a.z, f.z * b.z);
					x[4 * h + 3] = mk<C>(f.w * a.w, f.w * b.w);
				}
				dft32<+1>(x);
				F.slots_a([&](int m, C &v) { v = x[pos32(m)]; });
				__syncthreads();
				F.stage_b<+1>();
				__syncthreads();
				F.slots_c([&](int m, const C &v) { x[m] = v; });
				dft32<+1>(x);
				{
					C y[32];
#pragma unroll
					for (int h = 0; h < 8; h++) {
						const float4 f = ld4(ps, h);
						y[4 * h] = cscale(x[pos32(4 * h)], f.x);
						y[4 * h + 1] = cscale(x[pos32(4 * h + 1)], f.y);
						y[4 * h + 2] = cscale(x[pos32(4 * h + 2)], f.z);
						y[4 * h + 3] = cscale(x[pos32(4 * h + 3)], f.w);
					}
#pragma unroll
					for (int v = 0; v < 32; v++) x[v] = y[v];
				}
				dft32<-1>(x);
				F.slots_c([&](int m, C &v) { v = x[pos32(m)]; });
				__syncthreads();
				F.stage_b<-1>();
				__syncthreads();
				F.slots_a([&](int m, const C &v) { x[m] = v; });
				dft32<-1>(x);
				// the real part is T of i = 2c, the imaginary part of 2c + 1
#pragma unroll
				for (int h = 0; h < 4; h++) {
					float a[8];
					tmem_ld8r(TM::addr(tbase, q, h), a);
					const float4 f0 = ld4g(P0, 2 * h), f1 = ld4g(P0, 2 * h + 1), g0 = ld4g(P0 + PP, 2 * h), g1 = ld4g(P0 + PP, 2 * h + 1);
					const float f[8] = { f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w }, g[8] = { g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w };
					tmem_wait_ld();
#pragma unroll
					for (int e = 0; e < 8; e++) {
						const C v = x[pos32(8 * h + e)];
						a[e] += c0 * (f[e] * v.x) - sc * (g[e] * v.y);
					}
					tmem_st8r(TM::addr(tbase, q, h), a);
				}
				if (pr) {
#pragma unroll
					for (int h = 0; h < 4; h++) {
						const float4 f0 = ld4(Wj, 2 * h), f1 = ld4(Wj, 2 * h + 1);
						const float f[8] = { f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w };
						C y[8];
#pragma unroll
						for (int e = 0; e < 8; e++) y[e] = cscale(x[pos32(8 * h + e)], cj * f[e]);
						if (q == 0) {
							tmem_st8(TM::yaddr(tbase, h), y);
						} else {
							C a[8];
							tmem_ld8(TM::yaddr(tbase, h), a);
							tmem_wait_ld();
#pragma unroll
							for (int e = 0; e < 8; e++) x[pos32(8 * h + e)] = cadd(a[e], y[e]);
						}
					}
				}
				tmem_wait_st();
			}
			if (!pr) continue;
			// A_c += conj(psi1) . IFFT2(Y_2c + i Y_2c+1)
			{
				C y[32];
#pragma unroll
				for (int r = 0; r < 32; r++) y[r] = x[pos32(r)];
#pragma unroll
				for (int r = 0; r < 32; r++) x[r] = y[r];
			}
			dft32<+1>(x);
			F.slots_a([&](int m, C &v) { v = x[pos32(m)]; });
			__syncthreads();
			F.stage_b<+1>();
			__syncthreads();
			F.slots_c([&](int m, const C &v) { x[m] = v; });
			__syncthreads();                                 // the next chain writes rows
			if (kc <= H || kc >= P - H) {
				dft32<+1>(x);
				double2 *A = za + c * ZA + zk + H;
#pragma unroll
				for (int v = 0; v < 32; v++) {
					if (v > 8 && v < 24) continue;               // rows 36 .. 95
					const int l = F.row_c() + 4 * v, zl = v < 9 ? l : l - P;
					if (zl > H || (zl == H && zk == -H) || (zl == -H && zk == H)) continue;
					// psi1 is tabulated on -N/2 .. N/2 - 1; at the upper end it is conj psi1(-k)
					const bool up = zl == H || zk == H;
					const int a = up ? -zl : zl, b = up ? -zk : zk;
					C w = psi1[(a < 0 ? a + N : a) * N + (b < 0 ? b + N : b)];
					if (!up) w.y = -w.y;
					zadd_mem(A + (zl + H) * (N + 1), w, x[pos32(v)]);
				}
			}
		}
		cl.sync();                                           // the partner is done with this unit's spectra
	}
	// A(k) = Z_2c(k) + i Z_2c+1(k) with both parts the transforms of real grids
	{
		double2 *zo = p.zout + (slot * 2 + rank) * 4 * (long)NN;
		for (int i = t; i < 2 * NN; i += 512) {
			const int c = i / NN, n = i % NN;
			int l = n / N, k = n % N;
			l = l < H ? l : l - N;
			k = k < H ? k : k - N;
			const double2 u = __ldcg(za + c * ZA + (l + H) * (N + 1) + k + H), v = __ldcg(za + c * ZA + (H - l) * (N + 1) + H - k);
			zo[(long)(2 * c) * NN + n] = make_double2(0.5 * (u.x + v.x), 0.5 * (u.y - v.y));
			zo[(long)(2 * c + 1) * NN + n] = make_double2(0.5 * (u.y + v.y), -0.5 * (u.x - v.x));
		}
	}
#pragma unroll 1
	for (int q = 0; q < 2; q++) {
		C *o = p.out + (slot * 4 + 2 * rank + q) * (long)PP + F128::brow(F.row_a()) + F.col_a();
#pragma unroll 1
		for (int h = 0; h < 4; h++) {
			float a[8];
			tmem_ld8r(TM::addr(tbase, q, h), a);
			tmem_wait_ld();
#pragma unroll
			for (int e = 0; e < 8; e++) o[4 * (8 * h + e)] = mk<C>(a[e], 0.0);
		}
	}
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (warp == 0) tmem_dealloc(tbase, TM::NCOLS);
}
constexpr size_t kWide128Smem = sizeof(float2) * (Wide128::PP + 128);

}  // namespace qb
