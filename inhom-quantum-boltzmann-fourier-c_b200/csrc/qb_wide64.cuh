// qb_wide64.cuh — 64 x 64 transforms with 16 values a thread, and the I3 sums
// at N = 32 built on them.
//
// A group of 256 threads holds a 64 x 64 complex grid, 16 values a thread, and
// transforms it in three register stages with two exchanges through shared
// memory instead of the four stages and three exchanges of 8 values a thread.
// Inverse transform of a(l, k):
//   A  thread (l, tau), values k = tau + 4 r:             DFT16 over r -> q
//   B  thread (q, lam), values (l = lam + 16 s, tau):     x w64^(tau q), DFT4 over
//      tau -> p and over s -> u, x w64^(lam u)
//   C  thread (q + 16 p, u), values lam:                  DFT16 over lam -> v
// gives b(u + 4 v, q + 16 p); the forward transform is the mirror image (C, B,
// A with the same twiddles) and returns to the positions of A.  Every stage
// writes its results to the slots it read, so an exchange costs one barrier of
// the group, and a transform that starts at the positions where the last one
// ended needs none before it.
//
// Shared grid: slot(row, col) = 64 row + (col ^ sw(row)).  Eight lanes of 16-byte
// values (16 of 8 bytes) share a pass over the banks: of A two (four) rows x
// four consecutive columns, of B eight (16) consecutive rows, of C eight (16)
// consecutive columns.  With sw = bits (0, 2, 1) of the row (bits (1, 0, 3, 2) in
// FP32) each is free of bank conflicts without padding.
#pragma once
#include "qb_kernels.cuh"

namespace qb {

// 16-point DFT in registers: natural order in, frequency f in x[pos16(f)]
__host__ __device__ constexpr int pos16(int f) { return (f & 3) * 4 + (f >> 2); }
template <int DIR, class C> __device__ __forceinline__ void dft16(C (&x)[16]) {
	using R = typename CT<C>::R;
	constexpr double a = 0.92387953251128675613, b = 0.38268343236508977173;
#pragma unroll
	for (int n = 0; n < 4; n++) dft4<DIR>(x[n], x[n + 4], x[n + 8], x[n + 12]);
	// x[n + 4 k] holds partial frequency k of residue n: times w16^(n k)
	C w1, w3;
	w1.x = (R)a; w1.y = (R)(DIR < 0 ? -b : b);
	w3.x = (R)b; w3.y = (R)(DIR < 0 ? -a : a);
	x[5] = cmul(x[5], w1);
	x[6] = mul_w8<DIR>(x[6]);
	x[7] = cmul(x[7], w3);
	x[9] = mul_w8<DIR>(x[9]);
	x[10] = mul_i<DIR>(x[10]);
	x[11] = mul_w8_3<DIR>(x[11]);
	x[13] = cmul(x[13], w3);
	x[14] = mul_w8_3<DIR>(x[14]);
	C w9; w9.x = -w1.x; w9.y = -w1.y;                        // w16^9 = -w16
	x[15] = cmul(x[15], w9);
#pragma unroll
	for (int k = 0; k < 4; k++) dft4<DIR>(x[4 * k], x[4 * k + 1], x[4 * k + 2], x[4 * k + 3]);
	// frequency k + 4 m is in x[4 k + m]
}

template <class C> struct Wide64 {
	static constexpr int GT = 256;           // threads of a group
	C *U;                                    // the group's grid
	const C *tw;                             // w64^e, e < 64, forward sign
	int t, bar;                              // thread of the group, its named barrier
	static constexpr int HB = sizeof(C) == 16 ? 1 : 2, HM = (1 << HB) - 1;      // bits of q in the swizzled part of a column
	__device__ __forceinline__ static int sw(int row) { return ((row & HM) << 2) | ((row >> HB) & 3); }
	__device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(GT) : "memory"); }
	// A: this thread's row and first column
	__device__ __forceinline__ int row_a() const { return t >> 2; }
	__device__ __forceinline__ int col_a() const { return t & 3; }
	// C: this thread's column as a frequency / grid index and its first row (rows u + 4 v)
	__device__ __forceinline__ int col_c() const { const int c = t & 63; return (c >> 2) + 16 * (c & 3); }
	__device__ __forceinline__ int row_c() const { return t >> 6; }

	// slots of A: index q (columns tau + 4 q)
	template <class F> __device__ __forceinline__ void slots_a(const F &f) const {
		const int l = t >> 2, s = sw(l), b = l * 64;
#pragma unroll
		for (int q = 0; q < 16; q++) f(q, U[b + (((t & 3) + 4 * (q & HM)) ^ s) + (4 << HB) * (q >> HB)]);
	}
	// slots of B: index (s or u, tau or p)
	template <class F> __device__ __forceinline__ void slots_b(const F &f) const {
		const int q = t >> 4, lam = t & 15, s = sw(lam), b = lam * 64 + (4 << HB) * (q >> HB), h = 4 * (q & HM);
#pragma unroll
		for (int c = 0; c < 4; c++) {
			const int a = b + ((c + h) ^ s);
#pragma unroll
			for (int r = 0; r < 4; r++) f(r, c, U[a + 16 * 64 * r]);
		}
	}
	// slots of C: index lam
	template <class F> __device__ __forceinline__ void slots_c(const F &f) const {
		const int c = t & 63, b = (t >> 6) * 16 * 64;
#pragma unroll
		for (int m = 0; m < 16; m++) f(m, U[b + m * 64 + (c ^ sw(m))]);
	}
	// B of both directions: times w64^(c q) (inverse) or w64^(r lam) (forward), DFT4s, times the other
	template <int DIR> __device__ __forceinline__ void stage_b() const {
		const int q = t >> 4, lam = t & 15;
		C y[4][4];
		slots_b([&](int r, int c, const C &v) { y[r][c] = v; });
		C wq[3], wl[3];
#pragma unroll
		for (int m = 0; m < 3; m++) {
			wq[m] = tw[(m + 1) * q];
			wl[m] = tw[(m + 1) * lam];
			if (DIR > 0) { wq[m].y = -wq[m].y; wl[m].y = -wl[m].y; }
		}
		if (DIR > 0) {
#pragma unroll
			for (int r = 0; r < 4; r++)
#pragma unroll
				for (int c = 1; c < 4; c++) y[r][c] = cmul(y[r][c], wq[c - 1]);
		} else {
#pragma unroll
			for (int r = 1; r < 4; r++)
#pragma unroll
				for (int c = 0; c < 4; c++) y[r][c] = cmul(y[r][c], wl[r - 1]);
		}
#pragma unroll
		for (int r = 0; r < 4; r++) dft4<DIR>(y[r][0], y[r][1], y[r][2], y[r][3]);
#pragma unroll
		for (int c = 0; c < 4; c++) dft4<DIR>(y[0][c], y[1][c], y[2][c], y[3][c]);
		if (DIR > 0) {
#pragma unroll
			for (int r = 1; r < 4; r++)
#pragma unroll
				for (int c = 0; c < 4; c++) y[r][c] = cmul(y[r][c], wl[r - 1]);
		} else {
#pragma unroll
			for (int r = 0; r < 4; r++)
#pragma unroll
				for (int c = 1; c < 4; c++) y[r][c] = cmul(y[r][c], wq[c - 1]);
		}
		slots_b([&](int r, int c, C &v) { v = y[r][c]; });
	}
	// x[r] = a(row_a, col_a + 4 r) -> x[pos16(v)] = b(row_c + 4 v, col_c)
	__device__ __forceinline__ void inverse(C (&x)[16]) const {
		dft16<+1>(x);
		slots_a([&](int q, C &v) { v = x[pos16(q)]; });
		sync();
		stage_b<+1>();
		sync();
		slots_c([&](int m, const C &v) { x[m] = v; });
		dft16<+1>(x);
	}
	// x[v] = b(row_c + 4 v, col_c) -> x[pos16(r)] = a(row_a, col_a + 4 r)
	__device__ __forceinline__ void forward(C (&x)[16]) const {
		dft16<-1>(x);
		slots_c([&](int m, C &v) { v = x[pos16(m)]; });
		sync();
		stage_b<-1>();
		sync();
		slots_a([&](int q, const C &v) { x[q] = v; });
		dft16<-1>(x);
	}
};

// tensor memory of a thread of k_i3w: 16 accumulators of W words, then 16 values
// of P_j; four warps share a lane quarter.  W = 4 (FP64), 2 (FP32), 1 (FP32, real)
template <int W> struct WideTmem {
	static constexpr unsigned COLS = 128 * W, H = 16 * W;
	__device__ __forceinline__ static unsigned x(unsigned base) {
		const unsigned w = threadIdx.x >> 5;
		return base + ((32u * (w & 3u)) << 16) + (w >> 2) * 2u * H;
	}
	__device__ __forceinline__ static unsigned p(unsigned base) { return x(base) + H; }
};
// four FP32 complex values, or four reals
__device__ __forceinline__ void tmem_ld4(unsigned taddr, float2 (&v)[4]) {
	unsigned r[8];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
#pragma unroll
	for (int e = 0; e < 4; e++) { v[e].x = __uint_as_float(r[2 * e]); v[e].y = __uint_as_float(r[2 * e + 1]); }
}
__device__ __forceinline__ void tmem_st4(unsigned taddr, const float2 (&v)[4]) {
	unsigned r[8];
#pragma unroll
	for (int e = 0; e < 4; e++) { r[2 * e] = __float_as_uint(v[e].x); r[2 * e + 1] = __float_as_uint(v[e].y); }
	asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
	             :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
template <class C> constexpr size_t i3w_smem() {
	// two grids, the Y values in transit, psi2 (16 reals a thread of a group), the twiddles
	return sizeof(C) * (3 * 4096 + 64) + sizeof(typename CT<C>::R) * 4096;
}

// K4w: the I3 sums of the collision operator at N = 32 on a cluster of 2 CTAs
// of two groups, group g of CTA r for component j = 2 r + g.  Per unit
// (I3Units) a group writes P_j to the cluster's scratch in L2 and keeps it in
// tensor memory; after a cluster barrier it runs the chains of i = 0..3:
//   X_j += eta_i P_i . T_ij  (tensor memory),  y = eta_j W^_j . T_ij.
// Y_i of the CTA's two components goes to group i % 2 (through shared memory)
// which adds conj(psi1) . Extract(IFFT2(Y_i)) to the CTA's partial of Z_i.  The
// groups meet at that hand-over and at the cluster barrier only.  Ghat (W^) and
// pscr are in thread order (value r of thread t of A at 256 r + t): a warp's
// load is four full lines, where the natural order gives eight half lines and
// twice the cycles of the shared-memory and L1 pipe, which bounds this kernel.
// Measured (64 cells, J = M = 16, FP64): the Strang step 17.7 ms with 8
// values a thread (FP64 pipe 42%, shared-memory pipe 72%), 16.2 ms with 16
// values in the natural order, 15.5 ms in thread order.
// out: [slot][4][PP], zout: [slot][rank][4][N*N], slots of the term ranges (or
// (cell, chunk)); pscr: [cluster][2][4][PP] (two units in turn: one cluster
// barrier a unit).
// kind: null (every cell) or the per-cell form of k_nyquist_kind; this kernel
// then takes the cells of kind 1 (the real form k_i3wr takes kind 0).
template <class C>
__global__ void __launch_bounds__(512, Occ<C>::CTAS) k_i3w(const I3ParamsT<C> p, C *pscr, const int *kind) {
	using R = typename CT<C>::R;
	using TM = WideTmem<sizeof(C) / 4>;
	constexpr int N = 32, NN = N * N, P = 64, PP = P * P, GT = 256, H4 = TM::H / 4;
	if (kind != nullptr && kind[blockIdx.x / 2 / p.nchunk] != 1) return;     // both CTAs of the cluster leave before any barrier
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned tmem_slot;
	C *grids = reinterpret_cast<C *>(smem_raw), *Yb = grids + 2 * PP, *tw = Yb + PP;
	R *psi = reinterpret_cast<R *>(tw + 64);
	cg::cluster_group cl = cg::this_cluster();
	const int rank = (int)cl.block_rank();
	const int cid = (int)(blockIdx.x / 2);
	const int g = threadIdx.x / GT, t = threadIdx.x % GT, warp = threadIdx.x >> 5;
	if (warp == 0) tmem_alloc(&tmem_slot, TM::COLS);
	init_twiddles<64>(tw);
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const unsigned tx = TM::x(tmem_slot), tp = TM::p(tmem_slot);
	const Wide64<C> F{ grids + g * PP, tw, t, g + 1 };
	const int j = 2 * rank + g;
	const R etaj = (R)(j == 0 ? 1.0 : -1.0);
	const int oa = F.row_a() * P + F.col_a();                // element of A (+ 4 r)
	const int kc = F.col_c(), ks = kc < N / 2 ? kc : (kc >= 3 * N / 2 ? kc - N : -1);
	const int oz = F.row_c() * N + ks;                       // N-grid element of C: rows u + 4 v (v < 4), u + 4 v - 32 (v >= 12)
	C *Pall = pscr + (long)cid * 8 * PP + t;
	Yb += t;
	int psi_idx = -1, par = 0;
	long u, u1;
	if (p.rg.nslots > 0) {
		u = p.rg.start(cid);
		u1 = p.rg.start(cid + 1);
	} else {
		const int chunk = (int)(cid % p.nchunk);
		const long cell = cid / p.nchunk;
		u = cell * p.nterms + (long)chunk * p.nterms / p.nchunk;
		u1 = cell * p.nterms + (long)(chunk + 1) * p.nterms / p.nchunk;
	}
	// one segment per cell of the range (the (cell, chunk) grid has one)
#pragma unroll 1
	while (u < u1) {
		const long cell = u / p.nterms;
		const int t0 = (int)(u % p.nterms);
		const int t1 = (int)min((long)p.nterms, t0 + (u1 - u));
		u += t1 - t0;
		const long slot = p.rg.nslots > 0 ? (long)cid * p.rg.maxc + (cell - p.rg.first_cell(cid))
		                                  : cell * p.nchunk + (int)(cid % p.nchunk);
		const C *Wc = p.Ghat + cell * p.g_cell + t;
		const double2 *src = p.src + cell * p.src_cell + (long)p.src_comp[j] * NN + oz;
		double2 *Zo = p.zout + (slot * 2 + rank) * 4 * (long)NN + oz;
		{
			const C z[4] = { czero<C>(), czero<C>(), czero<C>(), czero<C>() };
#pragma unroll
			for (int h = 0; h < 4; h++) tmem_st4(tx + H4 * h, z);
			tmem_wait_st();
			if (ks >= 0) {
#pragma unroll 1
				for (int i = g; i < 4; i += 2)
#pragma unroll
					for (int v = 0; v < 8; v++) Zo[i * NN + 4 * v * N] = czero();
			}
		}
#pragma unroll 1
		for (int un = t0; un < t1; un++) {
			const int term = p.un.term(un);
			const bool pr = p.un.pair(un);
			const C *psi1 = p.psi1 + (long)term * NN + oz;
			C *Pu = Pall + par * 4 * PP;
			par ^= 1;
			C x[16];
			F.sync();                                        // the last chain's rows are read
			// P_j = FFT2(Pad(psi1 . W_j))
#pragma unroll
			for (int v = 0; v < 16; v++) x[v] = czero<C>();
			if (ks >= 0) {
#pragma unroll
				for (int v = 0; v < 8; v++) {
					const double2 w = src[4 * v * N];
					x[v < 4 ? v : v + 8] = cmul(psi1[4 * v * N], mk<C>(w.x, w.y));
				}
			}
			F.forward(x);
#pragma unroll
			for (int h = 0; h < 4; h++) {
				C a[4];
#pragma unroll
				for (int r = 0; r < 4; r++) {
					a[r] = x[pos16(4 * h + r)];
					__stcg(Pu + j * PP + GT * (4 * h + r), a[r]);
				}
				tmem_st4(tp + H4 * h, a);
			}
			tmem_wait_st();
			cl.sync();                                       // the unit's P grids are in L2
			if (p.psi2_idx[term] != psi_idx) {               // a new angle: its psi2 in the order of C
				psi_idx = p.psi2_idx[term];
				const R *s = p.psi2T + (long)psi_idx * PP + kc * P + F.row_c();
#pragma unroll
				for (int v = 0; v < 8; v++) psi[(8 * g + v) * GT + t] = s[4 * (8 * g + v)];
				__syncthreads();
			}
			const R sc = (R)p.psi2_scale[term];
#pragma unroll 1
			for (int i = 0; i < 4; i++) {
				const C *Wi = Wc + i * PP;
#pragma unroll
				for (int r = 0; r < 16; r++) x[r] = Wi[GT * r];
#pragma unroll
				for (int h = 0; h < 4; h++) {
					C a[4];
					tmem_ld4(tp + H4 * h, a);
					tmem_wait_ld();
#pragma unroll
					for (int r = 0; r < 4; r++) x[4 * h + r] = cmul(x[4 * h + r], a[r]);
				}
				F.inverse(x);
				{
					C y[16];
#pragma unroll
					for (int v = 0; v < 16; v++) y[v] = cscale(x[pos16(v)], psi[v * GT + t]);
#pragma unroll
					for (int v = 0; v < 16; v++) x[v] = y[v];
				}
				F.forward(x);
				// X_j += eta_i P_i . T_ij (psi2's scale applied here)
				const C *Pi = Pu + i * PP;
				const R ci = i == 0 ? sc : -sc;
#pragma unroll
				for (int h = 0; h < 4; h++) {
					C a[4], w[4];
#pragma unroll
					for (int r = 0; r < 4; r++) w[r] = __ldcg(Pi + GT * (4 * h + r));
					tmem_ld4(tx + H4 * h, a);
					tmem_wait_ld();
#pragma unroll
					for (int r = 0; r < 4; r++) {
						const C v = cmul(w[r], x[pos16(4 * h + r)]);
						a[r].x += ci * v.x;
						a[r].y += ci * v.y;
					}
					tmem_st4(tx + H4 * h, a);
				}
				if (pr) {
					// y = eta_j W^_j . T_ij; the group of i % 2 takes the sum of both
					const C *Wj = Wc + j * PP;
					const R cj = etaj * sc;
					const int hand = 3 + (i & 1);
#pragma unroll
					for (int r = 0; r < 16; r++) x[pos16(r)] = cscale(cmul(Wj[GT * r], x[pos16(r)]), cj);
					if ((i & 1) != g) {
#pragma unroll
						for (int r = 0; r < 16; r++) Yb[r * GT] = x[pos16(r)];
						asm volatile("bar.arrive %0, 512;" ::"r"(hand) : "memory");
					} else {
						asm volatile("bar.sync %0, 512;" ::"r"(hand) : "memory");
						C y[16];
#pragma unroll
						for (int r = 0; r < 16; r++) y[r] = cadd(Yb[r * GT], x[pos16(r)]);
						F.inverse(y);
						F.sync();                                // the next chain writes rows
						if (ks >= 0) {
							double2 *z = Zo + i * NN;
#pragma unroll
							for (int v = 0; v < 8; v++) {
								C w = psi1[4 * v * N];
								w.y = -w.y;
								zadd_mem(z + 4 * v * N, w, y[pos16(v < 4 ? v : v + 8)]);
							}
						}
					}
				}
				tmem_wait_st();
			}
		}
		C *o = p.out + (slot * 4 + j) * (long)PP + oa;
#pragma unroll
		for (int h = 0; h < 4; h++) {
			C a[4];
			tmem_ld4(tx + H4 * h, a);
			tmem_wait_ld();
#pragma unroll
			for (int r = 0; r < 4; r++) o[4 * (4 * h + r)] = a[r];
		}
	}
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (warp == 0) tmem_dealloc(tmem_slot, TM::COLS);
}

// ---------------------------------------------------------------------------
// k_i3w in real arithmetic (FP32 form, cells without Nyquist content): W^ and P
// are real and a chain maps real grids to real grids (qb_full128.cuh), so the
// chains of i = 2c and 2c + 1 share one complex transform of P_j . (W^_2c + i
// W^_2c+1), X_j (real) takes eta_2c P_2c . Re + eta_2c+1 P_2c+1 . Im, and Y_2c +
// i Y_2c+1 is packed the same way: two chains a unit and group.  A_c = Z_2c + i
// Z_2c+1 is summed on the frequencies -N/2 .. N/2 of both dimensions (the
// partner of -N/2 separates the two) in zscr and separated at the end.  WhR: the
// real parts of W^ in thread order; pscr: [cluster][4][4][PP]
// reals, the first half used.
__global__ void __launch_bounds__(512, 2) k_i3wr(const I3ParamsT<float2> p, const float *__restrict__ WhR, float *pscr, const int *kind) {
	using C = float2;
	using TM = WideTmem<1>;
	constexpr int N = 32, NN = N * N, P = 64, PP = P * P, GT = 256, H = N / 2, ZA = (N + 1) * (N + 1);
	const int cid = (int)(blockIdx.x / 2), chunk = cid % p.nchunk;
	const long cell = cid / p.nchunk;
	if (kind[cell] != 0) return;                             // both CTAs of the cluster leave before any barrier
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned tmem_slot;
	C *grids = reinterpret_cast<C *>(smem_raw), *Yb = grids + 2 * PP, *tw = Yb + PP;
	float *psi = reinterpret_cast<float *>(tw + 64);
	cg::cluster_group cl = cg::this_cluster();
	const int rank = (int)cl.block_rank();
	const int g = threadIdx.x / GT, t = threadIdx.x % GT, warp = threadIdx.x >> 5;
	if (warp == 0) tmem_alloc(&tmem_slot, TM::COLS);
	init_twiddles<64>(tw);
	const long slot = cell * p.nchunk + chunk;
	double2 *za = p.zscr + (slot * 2 + rank) * 2 * (long)ZA;
	for (int i = threadIdx.x; i < 2 * ZA; i += 512) za[i] = czero();
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const unsigned tx = TM::x(tmem_slot), tp = TM::p(tmem_slot);
	const Wide64<C> F{ grids + g * PP, tw, t, g + 1 };
	const int j = 2 * rank + g;
	const float etaj = j == 0 ? 1.f : -1.f;
	const int oa = F.row_a() * P + F.col_a();
	const int kc = F.col_c(), ks = kc < N / 2 ? kc : (kc >= 3 * N / 2 ? kc - N : -1);
	const int zk = kc <= H ? kc : kc - P;                    // this thread's column of C as a frequency
	const int oz = F.row_c() * N + ks;
	float *Pall = pscr + (long)cid * 16 * PP + t;          // where the complex form has this cluster's grids
	Yb += t;
	const double2 *src = p.src + cell * p.src_cell + (long)p.src_comp[j] * NN + oz;
	const float *Wc = WhR + cell * 4 * PP + t;
	{
		const float z[8] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
		tmem_st8r(tx, z);
		tmem_st8r(tx + 8, z);
		tmem_wait_st();
	}
	const int u0 = (int)((long)chunk * p.nterms / p.nchunk), u1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
	int psi_idx = -1, par = 0;
#pragma unroll 1
	for (int un = u0; un < u1; un++) {
		const int term = p.un.term(un);
		const bool pr = p.un.pair(un);
		float *Pu = Pall + par * 4 * PP;
		par ^= 1;
		C x[16];
		F.sync();                                            // the last chain's rows are read
		{
			// P_j = FFT2(Pad(psi1 . W_j)), real
			const C *psi1 = p.psi1 + (long)term * NN + oz;
#pragma unroll
			for (int v = 0; v < 16; v++) x[v] = czero<C>();
			if (ks >= 0) {
#pragma unroll
				for (int v = 0; v < 8; v++) {
					const double2 w = src[4 * v * N];
					x[v < 4 ? v : v + 8] = cmul(psi1[4 * v * N], mk<C>(w.x, w.y));
				}
			}
		}
		F.forward(x);
#pragma unroll
		for (int h = 0; h < 2; h++) {
			float a[8];
#pragma unroll
			for (int r = 0; r < 8; r++) {
				a[r] = x[pos16(8 * h + r)].x;
				__stcg(Pu + j * PP + GT * (8 * h + r), a[r]);
			}
			tmem_st8r(tp + 8 * h, a);
		}
		tmem_wait_st();
		cl.sync();                                           // the unit's P grids are in L2
		if (p.psi2_idx[term] != psi_idx) {                   // a new angle: its psi2 in the order of C
			psi_idx = p.psi2_idx[term];
			const float *s = p.psi2T + (long)psi_idx * PP + kc * P + F.row_c();
#pragma unroll
			for (int v = 0; v < 8; v++) psi[(8 * g + v) * GT + t] = s[4 * (8 * g + v)];
			__syncthreads();
		}
		const float sc = (float)p.psi2_scale[term];
#pragma unroll 1
		for (int c = 0; c < 2; c++) {
			const float *W0 = Wc + 2 * c * PP;
#pragma unroll
			for (int h = 0; h < 2; h++) {
				float a[8];
				tmem_ld8r(tp + 8 * h, a);
#pragma unroll
				for (int r = 0; r < 8; r++) x[8 * h + r] = mk<C>(W0[GT * (8 * h + r)], W0[PP + GT * (8 * h + r)]);
				tmem_wait_ld();
#pragma unroll
				for (int r = 0; r < 8; r++) x[8 * h + r] = cscale(x[8 * h + r], a[r]);
			}
			F.inverse(x);
			{
				C y[16];
#pragma unroll
				for (int v = 0; v < 16; v++) y[v] = cscale(x[pos16(v)], psi[v * GT + t]);
#pragma unroll
				for (int v = 0; v < 16; v++) x[v] = y[v];
			}
			F.forward(x);
			const float *P0 = Pu + 2 * c * PP;
			const float c0 = c == 0 ? sc : -sc;                  // eta_2c; eta_2c+1 = -1
#pragma unroll
			for (int h = 0; h < 2; h++) {
				float a[8];
				tmem_ld8r(tx + 8 * h, a);
				tmem_wait_ld();
#pragma unroll
				for (int r = 0; r < 8; r++) {
					const C v = x[pos16(8 * h + r)];
					a[r] += c0 * (__ldcg(P0 + GT * (8 * h + r)) * v.x) - sc * (__ldcg(P0 + PP + GT * (8 * h + r)) * v.y);
				}
				tmem_st8r(tx + 8 * h, a);
			}
			if (pr) {
				const float *Wj = Wc + j * PP;
				const float cj = etaj * sc;
				const int hand = 3 + c;
#pragma unroll
				for (int r = 0; r < 16; r++) x[pos16(r)] = cscale(x[pos16(r)], cj * Wj[GT * r]);
				if (c != g) {
#pragma unroll
					for (int r = 0; r < 16; r++) Yb[r * GT] = x[pos16(r)];
					asm volatile("bar.arrive %0, 512;" ::"r"(hand) : "memory");
				} else {
					asm volatile("bar.sync %0, 512;" ::"r"(hand) : "memory");
					C y[16];
#pragma unroll
					for (int r = 0; r < 16; r++) y[r] = cadd(Yb[r * GT], x[pos16(r)]);
					F.inverse(y);
					F.sync();                                // the next chain writes rows
					if (kc <= H || kc >= P - H) {
						const C *ps = p.psi1 + (long)term * NN;
#pragma unroll
						for (int v = 0; v < 16; v++) {
							if (v > 4 && v < 12) continue;       // rows 20 .. 47
							const int l = F.row_c() + 4 * v, zl = v < 5 ? l : l - P;
							if (zl > H || (zl == H && zk == -H) || (zl == -H && zk == H)) continue;
							// psi1 is tabulated on -N/2 .. N/2 - 1; at the upper end it is conj psi1(-k)
							const bool up = zl == H || zk == H;
							const int a = up ? -zl : zl, b = up ? -zk : zk;
							C w = ps[(a < 0 ? a + N : a) * N + (b < 0 ? b + N : b)];
							if (!up) w.y = -w.y;
							zadd_mem(za + c * ZA + (zl + H) * (N + 1) + zk + H, w, y[pos16(v)]);
						}
					}
				}
			}
			tmem_wait_st();
		}
	}
	__syncthreads();                                         // za is complete
	{
		double2 *zo = p.zout + (slot * 2 + rank) * 4 * (long)NN;
		for (int i = threadIdx.x; i < 2 * NN; i += 512) {
			const int c = i / NN, n = i % NN;
			int l = n / N, k = n % N;
			l = l < H ? l : l - N;
			k = k < H ? k : k - N;
			const double2 a = __ldcg(za + c * ZA + (l + H) * (N + 1) + k + H), b = __ldcg(za + c * ZA + (H - l) * (N + 1) + H - k);
			zo[(long)(2 * c) * NN + n] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
			zo[(long)(2 * c + 1) * NN + n] = make_double2(0.5 * (a.y + b.y), -0.5 * (a.x - b.x));
		}
	}
	C *o = p.out + (slot * 4 + j) * (long)PP + oa;
#pragma unroll
	for (int h = 0; h < 2; h++) {
		float a[8];
		tmem_ld8r(tx + 8 * h, a);
		tmem_wait_ld();
#pragma unroll
		for (int r = 0; r < 8; r++) o[4 * (8 * h + r)] = mk<C>(a[r], 0.0);
	}
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (warp == 0) tmem_dealloc(tmem_slot, TM::COLS);
}

}  // namespace qb
