// qb_terms64.cuh — the I1, I2 and I4 term sums at N = 32 with 16 values a thread.
//
// One CTA of 256 threads per (cell, task, chunk) on the transforms of qb_wide64.cuh:
// two exchanges through shared memory a 2-D transform where the general kernels
// (k_i1_terms, k_i2_terms: 8 values a thread) take three and a change of order between
// the directions. FP64: two CTAs on an SM, whose accumulators and second operand (F,
// or the first transform of a product) are in tensor memory, since they and the
// transform do not fit 128 registers; FP32: three CTAs, accumulators in registers.
// Measured (Strang step, 64 cells, J = M = 16, the sums alone): I1 and I4 in FP64 1009 ->
// 666 us, I2 357 -> 280 us; I1 and I4 in FP32 734 -> 418 us. Both are bound by the
// shared-memory pipe and the latency of its barriers. I2 in FP32 stays with k_i2_terms.
#pragma once
#include "qb_wide64.cuh"

namespace qb {

template <class C> struct Terms64 {
	static constexpr bool WIDE = sizeof(C) == 16;
	static constexpr int P = 64, PP = P * P, N = 32, NN = N * N, NT = 256, CTAS = WIDE ? 2 : 3;
	static constexpr unsigned H = 4 * sizeof(C);             // columns of 16 values
	static constexpr unsigned COLS = (WIDE ? 4 : 2) * H;     // 256 or 64
	static constexpr size_t SMEM = sizeof(C) * (PP + 64);
	__device__ __forceinline__ static unsigned f(unsigned base) {        // the second operand
		const unsigned w = threadIdx.x >> 5;
		return base + ((32u * (w & 3u)) << 16) + (w >> 2) * (COLS / 2);
	}
	// 16 accumulators, visited four at a time by fn(index, value)
	struct Acc {
		unsigned ta;
		C r[WIDE ? 1 : 16];
		__device__ __forceinline__ void zero() {
			if constexpr (WIDE) {
				const C z[4] = { czero<C>(), czero<C>(), czero<C>(), czero<C>() };
#pragma unroll
				for (int h = 0; h < 4; h++) tmem_st4(ta + H / 4 * h, z);
				tmem_wait_st();
			} else {
#pragma unroll
				for (int e = 0; e < 16; e++) r[e] = czero<C>();
			}
		}
		template <class Fn> __device__ __forceinline__ void visit(int h, const Fn &fn) {
			if constexpr (WIDE) {
				C a[4];
				tmem_ld4(ta + H / 4 * h, a);
				tmem_wait_ld();
#pragma unroll
				for (int e = 0; e < 4; e++) fn(4 * h + e, a[e]);
				tmem_st4(ta + H / 4 * h, a);
			} else {
#pragma unroll
				for (int e = 0; e < 4; e++) fn(4 * h + e, r[4 * h + e]);
			}
		}
	};
	// this thread's values of Pad(psi . g) in the order of C
	template <class R> __device__ __forceinline__ static void load_pad(C (&x)[16], int ks, const R *psi, const double2 *g) {
#pragma unroll
		for (int v = 0; v < 16; v++) x[v] = czero<C>();
		if (ks >= 0) {
#pragma unroll
			for (int v = 0; v < 8; v++) {                    // rows u + 4 v: v < 4 and v >= 12
				const double2 w = g[4 * v * N];
				x[v < 4 ? v : v + 8] = cscale(mk<C>(w.x, w.y), psi[4 * v * N]);
			}
		}
	}
};

// the sums of k_i1_terms at P = 64
template <class C>
__global__ void __launch_bounds__(Terms64<C>::NT, Terms64<C>::CTAS) k_i1_terms64(const I1ParamsT<C> p) {
	using T = Terms64<C>;
	using R = typename CT<C>::R;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned tmem_slot;
	C *U = reinterpret_cast<C *>(smem_raw), *tw = U + T::PP;
	const int t = threadIdx.x;
	const int chunk = blockIdx.x % p.nchunk, task = (blockIdx.x / p.nchunk) % p.ntask;
	const long cell = blockIdx.x / (p.nchunk * p.ntask);
	if (t < 32) tmem_alloc(&tmem_slot, T::COLS);
	init_twiddles<64>(tw);
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const Wide64<C> F{ U, tw, t, 1 };
	const unsigned tf = T::f(tmem_slot);
	typename T::Acc acc{ tf + T::H, {} };
	acc.zero();
	{
		const C *w = p.What + cell * p.w_cell + (long)p.f_comp * T::PP + F.row_a() * T::P + F.col_a();
		const R fa = (R)p.fa, fb = (R)p.fb;
#pragma unroll
		for (int h = 0; h < 4; h++) {
			C f[4];
#pragma unroll
			for (int e = 0; e < 4; e++) {
				const C v = w[4 * (4 * h + e)];
				f[e].x = fa * v.x + fb;
				f[e].y = fa * v.y;
			}
			tmem_st4(tf + T::H / 4 * h, f);
		}
		tmem_wait_st();
	}
	const int kc = F.col_c(), ks = kc < T::N / 2 ? kc : (kc >= 3 * T::N / 2 ? kc - T::N : -1), oz = F.row_c() * T::N + ks;
	const double2 *g = p.g + cell * p.g_cell + (long)p.g_comp[task] * T::NN + oz;
	const int o = F.row_c() * T::P + kc;                     // element of C (+ 4 P v)
	const int t0 = (int)((long)chunk * p.nterms / p.nchunk), t1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
#pragma unroll 1
	for (int m = t0; m < t1; m++) {
		C x[16];
		T::load_pad(x, ks, p.psi2 + (long)m * T::NN + oz, g);
		F.forward(x);
		{
			C y[16];
#pragma unroll
			for (int h = 0; h < 4; h++) {
				C f[4];
				tmem_ld4(tf + T::H / 4 * h, f);
				tmem_wait_ld();
#pragma unroll
				for (int e = 0; e < 4; e++) y[4 * h + e] = cmul(f[e], x[pos16(4 * h + e)]);
			}
#pragma unroll
			for (int r = 0; r < 16; r++) x[r] = y[r];
		}
		F.inverse(x);
		const R *phi = p.phi + (long)m * T::PP + o;
#pragma unroll
		for (int h = 0; h < 4; h++)
			acc.visit(h, [&](int v, C &a) {
				const R f = phi[4 * T::P * v];
				a.x += f * x[pos16(v)].x;
				a.y += f * x[pos16(v)].y;
			});
		tmem_wait_st();
	}
	C *out = p.out + ((cell * p.ntask + task) * p.nchunk + chunk) * (long)T::PP + o;
#pragma unroll
	for (int h = 0; h < 4; h++) acc.visit(h, [&](int v, C &a) { out[4 * T::P * v] = a; });
	tmem_wait_st();
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (t < 32) tmem_dealloc(tmem_slot, T::COLS);
}

// the sums of k_i2_terms at P = 64 in FP64
__global__ void __launch_bounds__(Terms64<double2>::NT, Terms64<double2>::CTAS) k_i2_terms64(const I2ParamsT<double2> p) {
	using C = double2;
	using T = Terms64<C>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned tmem_slot;
	C *U = reinterpret_cast<C *>(smem_raw), *tw = U + T::PP;
	const int t = threadIdx.x;
	const int chunk = blockIdx.x % p.nchunk, task = (blockIdx.x / p.nchunk) % p.ntask;
	const long cell = blockIdx.x / (p.nchunk * p.ntask);
	if (t < 32) tmem_alloc(&tmem_slot, T::COLS);
	init_twiddles<64>(tw);
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const Wide64<C> F{ U, tw, t, 1 };
	const unsigned tf = T::f(tmem_slot);
	typename T::Acc acc{ tf + T::H, {} };
	acc.zero();
	const int kc = F.col_c(), ks = kc < T::N / 2 ? kc : (kc >= 3 * T::N / 2 ? kc - T::N : -1), oz = F.row_c() * T::N + ks;
	const double2 *f = p.src + cell * p.cell_stride + (long)p.f_comp[task] * T::NN + oz;
	const double2 *g = p.src + cell * p.cell_stride + (long)p.g_comp[task] * T::NN + oz;
	const int t0 = (int)((long)chunk * p.nterms / p.nchunk), t1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
#pragma unroll 1
	for (int m = t0; m < t1; m++) {
		C x[16];
		T::load_pad(x, ks, p.psi1 + (long)m * T::NN + oz, f);
		F.sync();                                            // the last transform's rows are read
		F.forward(x);
#pragma unroll
		for (int h = 0; h < 4; h++) {
			C a[4];
#pragma unroll
			for (int e = 0; e < 4; e++) a[e] = x[pos16(4 * h + e)];
			tmem_st4(tf + T::H / 4 * h, a);
		}
		tmem_wait_st();
		T::load_pad(x, ks, p.psi2 + (long)m * T::NN + oz, g);
		F.sync();
		F.forward(x);
#pragma unroll
		for (int h = 0; h < 4; h++) {
			C y[4];
			tmem_ld4(tf + T::H / 4 * h, y);
			tmem_wait_ld();
			acc.visit(h, [&](int r, C &a) { a = cfma(y[r & 3], x[pos16(r)], a); });
		}
		tmem_wait_st();
	}
	C *out = p.out + ((cell * p.ntask + task) * p.nchunk + chunk) * (long)T::PP + F.row_a() * T::P + F.col_a();
#pragma unroll
	for (int h = 0; h < 4; h++) acc.visit(h, [&](int r, C &a) { out[4 * r] = a; });
	tmem_wait_st();
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (t < 32) tmem_dealloc(tmem_slot, T::COLS);
}

}  // namespace qb
