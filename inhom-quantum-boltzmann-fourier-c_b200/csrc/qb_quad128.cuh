// qb_quad128.cuh — the I3 sums at N = 64 in FP64: a padded 128 x 128 grid as
// four 64 x 64 grids, one component's chains in one CTA.
//
// A padded FP64 grid (256 KB) does not fit a CTA's shared memory, but the
// four grids of its even / odd rows and columns do, one after the other.  With
// l = 2 m + pl, k = 2 n + pk and s = 2 pl + pk the inverse transform is
//   b(r + 64 sl, c + 64 sk) = sum_s (-1)^(sl pl + sk pk) w^(r pl + c pk) E_s(r, c),
//   E_s = IFFT64x64 of a(2 m + pl, 2 n + pk),  w = exp(2 pi i / 128),
// and the forward transform its mirror image: a chain FFT2(psi2 . IFFT2(a)) is
// four 64 x 64 inverse transforms, one pointwise 4 x 4 step at (r, c) (the
// butterflies, psi2 at its four points, the butterflies back) and four 64 x 64
// forward transforms.  Every thread owns the same eight (r, c) in all of them,
// so the E_s of a thread wait in places only it reads: two in shared memory,
// one in tensor memory, one in registers.  The 64 x 64 transforms hold 8
// values a thread, in one grid of pitch 65.
//
// Padding needs no transform of zeros: of the four points (r + 64 sl, c + 64
// sk) exactly one is outside the zero band, that of N-grid index (r, c), with
// sl = (r >= 32), sk = (c >= 32); so is Extract.
//
// Grids in global memory are in quad order, [s][64 m + n] (four contiguous
// 64 x 64 grids).
#pragma once
#include "qb_split128.cuh"

namespace qb {

struct Quad128 {
	using G = Geo<64, double2>;
	static constexpr int NT = 512, Q = 64 * 64;
	static constexpr long PP = 4L * Q;
	// the work grid, two waiting grids (8 values a thread), w^e for e < 128
	static constexpr size_t SMEM = sizeof(double2) * (G::GRID + 2 * 8 * NT + 128);
	static constexpr int TCOLS = 512;
	// tensor memory of a thread: X of s = 0, 1, 2 (32 words each), then one waiting grid
	__device__ __forceinline__ static unsigned taddr(unsigned base, int s) {
		const unsigned w = threadIdx.x >> 5;
		return base + ((32u * (w & 3u)) << 16) + (w >> 2) * 128u + 32u * (unsigned)s;
	}
};

// B-layout grids -> quad order
__global__ void __launch_bounds__(256) k_b_to_quad(const double2 *__restrict__ in, double2 *__restrict__ out) {
	const long g = (long)blockIdx.y * Quad128::PP;
	const int i = blockIdx.x * 256 + threadIdx.x;
	out[g + quad_from_b(i >> 13, (i >> 7) & 63, i & 127)] = in[g + i];
}

// 64-point transform of 8 values (fft1d) with the lane's twiddles w1 = w64^tau
// and w2 = w1^2 in registers (the powers by three levels of products); PRE: a
// CTA barrier before the line is used as scratch
template <int DIR, class Acc>
__device__ __forceinline__ void fft64_q(double2 (&x)[8], int tau, const Acc &sc, double2 w1, double2 w2, bool pre) {
	dft8<DIR>(x);
	if (DIR > 0) { w1.y = -w1.y; w2.y = -w2.y; }
	const double2 w3 = cmul(w1, w2), w4 = cmul(w2, w2);
	x[1] = cmul(x[1], w1);
	x[2] = cmul(x[2], w2);
	x[3] = cmul(x[3], w3);
	x[4] = cmul(x[4], w4);
	x[5] = cmul(x[5], cmul(w4, w1));
	x[6] = cmul(x[6], cmul(w4, w2));
	x[7] = cmul(x[7], cmul(w4, w3));
	if (pre) __syncthreads();
	fft1d_tail<64, DIR>(x, tau, sc);
}

// K4 (quad): the I3 sums of the collision operator on clusters of 4 CTAs, CTA j
// for component j.  Per unit (I3Units) CTA j writes P_j to the cluster's
// scratch (L2); after a cluster barrier the CTAs run the 16 chains in four
// rounds, CTA j that of i = (j + round) % 4:
//   X_j += eta_i P_i . T_ij   (tensor memory, s = 3 in the partial sum in L2)
//   Y_i += eta_j W^_j . T_ij  (cluster scratch in L2; one CTA a round and i)
// and after the last round CTA j transforms Y_j.  WhQ: W^ in quad order; pscr,
// yscr: [cluster][4][PP]; out: [slot][4][PP] quad order, zout: [slot][4][N*N],
// slots of the term ranges.
// Bound by the shared-memory pipe (28.8k of its cycles a chain for the
// transforms, 14k for the operands from L2) and the FP64 pipe (30k) together;
// the scratch of 33 clusters (P, Y and X: 75 MB) stays in L2.  Before, a grid
// was split over a CTA pair that exchanged 128 KB a chain and CTA, and every
// term ran its own chains: Strang step of 16 cells, J = M = 32: 218 -> 112 ms.
__global__ void __launch_bounds__(Quad128::NT, 1) k_i3_quad(const I3ParamsT<double2> p, const double2 *__restrict__ WhQ, double2 *pscr, double2 *yscr) {
	using F = Quad128;
	using G = F::G;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	__shared__ unsigned tmem_slot;
	double2 *Ug = reinterpret_cast<double2 *>(smem_raw), *st0 = Ug + G::GRID, *st1 = st0 + 8 * F::NT, *tw = st1 + 8 * F::NT;
	cg::cluster_group cl = cg::this_cluster();
	const int j = (int)cl.block_rank();
	const int cid = (int)(blockIdx.x / 4);
	const int tid = threadIdx.x, warp = tid >> 5, line = tid >> 3, tau = tid & 7;
	if (warp == 0) tmem_alloc(&tmem_slot, F::TCOLS);
	init_twiddles<128>(tw);
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	const unsigned tbase = tmem_slot;
	const double2 w1 = tw[2 * tau], w2 = tw[4 * tau];        // w64^tau, w64^(2 tau), forward sign
	double2 *Pall = pscr + (long)cid * 4 * F::PP, *Yall = yscr + (long)cid * 4 * F::PP;
	const int row = line * 64 + tau;                         // element of this thread in a row pass (+ 8 r)
	const double etaj = j == 0 ? 1.0 : -1.0;
	st0 += tid;
	st1 += tid;
	long u = p.rg.start(cid);
	const long u1 = p.rg.start(cid + 1);
#pragma unroll 1
	while (u < u1) {                                         // one segment per cell of the range
		const long cell = u / p.nterms;
		const int t0 = (int)(u % p.nterms);
		const int t1 = (int)min((long)p.nterms, t0 + (u1 - u));
		u += t1 - t0;
		const long slot = (long)cid * p.rg.maxc + (cell - p.rg.first_cell(cid));
		double2 *Xo = p.out + (slot * 4 + j) * F::PP + row;
		double2 *Zo = p.zout + (slot * 4 + j) * (long)F::Q + tau * 64 + line;        // rows tau + 8 e
#pragma unroll 1
		for (int s = 0; s < 3; s++)
#pragma unroll
			for (int e = 0; e < 8; e++) tmem_st(F::taddr(tbase, s) + 4 * e, czero());
		tmem_wait_st();
#pragma unroll
		for (int e = 0; e < 8; e++) {
			Xo[3 * F::Q + 8 * e] = czero();
			Zo[8 * e * 64] = czero();
		}
		const double2 *src = p.src + cell * p.src_cell + (long)p.src_comp[j] * F::Q + tau * 64 + line;
		const double2 *Wc = WhQ + cell * 4 * F::PP + row;
#pragma unroll 1
		for (int un = t0; un < t1; un++) {
			const int t = p.un.term(un);
			const bool pr = p.un.pair(un);
			const double2 *psi1 = p.psi1 + (long)t * F::Q + tau * 64 + line;
			// P_j: the four grids of FFT2(Pad(psi1 . W_j)), columns then rows
#pragma unroll 1
			for (int s = 0; s < 4; s++) {
				double2 x[8];
#pragma unroll
				for (int r = 0; r < 8; r++) {
					const int l = tau + 8 * r;
					double2 v = cmul(psi1[8 * r * 64], src[8 * r * 64]);
					if (s != 0) {
						v = cmul(v, tw[(s & 2 ? l : 0) + (s & 1 ? line : 0)]);
						if (((s & 2) && l >= 32) != ((s & 1) && line >= 32)) { v.x = -v.x; v.y = -v.y; }
					}
					x[r] = v;
				}
				fft64_q<-1>(x, tau, G::col(Ug, line), w1, w2, true);
#pragma unroll
				for (int e = 0; e < 8; e++) Ug[G::at(tau + 8 * e, line)] = x[e];
				__syncthreads();
#pragma unroll
				for (int r = 0; r < 8; r++) x[r] = Ug[G::at(line, tau + 8 * r)];
				fft64_q<-1>(x, tau, G::row(Ug, line), w1, w2, false);
				double2 *o = Pall + j * F::PP + s * F::Q + row;
#pragma unroll
				for (int e = 0; e < 8; e++) __stcg(o + 8 * e, x[e]);
			}
			cl.sync();                                       // the cluster's P grids are in L2
			const double *psi2 = p.psi2T + (long)p.psi2_idx[t] * F::PP + line * 128 + tau;
			const double sc = p.psi2_scale[t];
#pragma unroll 1
			for (int c = 0; c < 4; c++) {
				const int i = (j + c) & 3;
				double2 x[8];
				// inverse transforms of the four grids of W^_i . P_j
#pragma unroll 1
				for (int s = 0; s < 4; s++) {
					const double2 *g = Wc + i * F::PP + s * F::Q, *pj = Pall + j * F::PP + s * F::Q + row;
#pragma unroll
					for (int r = 0; r < 8; r++) x[r] = cmul(g[8 * r], __ldcg(pj + 8 * r));
					fft64_q<+1>(x, tau, G::row(Ug, line), w1, w2, s > 0);
#pragma unroll
					for (int e = 0; e < 8; e++) Ug[G::at(line, tau + 8 * e)] = x[e];
					__syncthreads();
#pragma unroll
					for (int r = 0; r < 8; r++) x[r] = Ug[G::at(tau + 8 * r, line)];
					fft64_q<+1>(x, tau, G::col(Ug, line), w1, w2, false);
					if (s < 2) {
						double2 *st = s == 0 ? st0 : st1;
#pragma unroll
						for (int e = 0; e < 8; e++) st[e * F::NT] = x[e];
					} else if (s == 2) {
						tmem_st8(F::taddr(tbase, 3), x);
						tmem_wait_st();
					}
				}
				// the pointwise step at (tau + 8 e, line)
				const double2 kc = tw[line];
#pragma unroll
				for (int e = 0; e < 8; e++) {
					const double2 kl = tw[tau + 8 * e];
					double2 e10;
					tmem_ld(F::taddr(tbase, 3) + 4 * e, e10);
					const double2 e00 = st0[e * F::NT], e01 = cmul(conj_c(kc), st1[e * F::NT]);
					const double f00 = sc * psi2[8 * e], f10 = sc * psi2[8 * e + 64];
					const double f01 = sc * psi2[8 * e + 64 * 128], f11 = sc * psi2[8 * e + 64 * 128 + 64];
					tmem_wait_ld();
					e10 = cmul(conj_c(kl), e10);
					const double2 e11 = cmul(conj_c(kl), cmul(conj_c(kc), x[e]));
					const double2 a0 = cadd(e00, e01), a1 = csub(e00, e01), b0 = cadd(e10, e11), b1 = csub(e10, e11);
					const double2 c00 = cscale(cadd(a0, b0), f00), c10 = cscale(csub(a0, b0), f10);
					const double2 c01 = cscale(cadd(a1, b1), f01), c11 = cscale(csub(a1, b1), f11);
					const double2 p0 = cadd(c00, c10), p1 = cadd(c01, c11), m0 = csub(c00, c10), m1 = csub(c01, c11);
					st0[e * F::NT] = cadd(p0, p1);
					st1[e * F::NT] = cmul(kc, csub(p0, p1));
					tmem_st(F::taddr(tbase, 3) + 4 * e, cmul(kl, cadd(m0, m1)));
					x[e] = cmul(kl, cmul(kc, csub(m0, m1)));
				}
				tmem_wait_st();
				// forward transforms, in the order s = 3 (in registers), 0, 1, 2
#pragma unroll 1
				for (int v = 0; v < 4; v++) {
					const int s = (v + 3) & 3;
					if (v == 1 || v == 2) {
						const double2 *st = v == 1 ? st0 : st1;
#pragma unroll
						for (int e = 0; e < 8; e++) x[e] = st[e * F::NT];
					} else if (v == 3) {
						tmem_ld8(F::taddr(tbase, 3), x);
						tmem_wait_ld();
					}
					fft64_q<-1>(x, tau, G::col(Ug, line), w1, w2, v > 0);
#pragma unroll
					for (int e = 0; e < 8; e++) Ug[G::at(tau + 8 * e, line)] = x[e];
					__syncthreads();
#pragma unroll
					for (int r = 0; r < 8; r++) x[r] = Ug[G::at(line, tau + 8 * r)];
					fft64_q<-1>(x, tau, G::row(Ug, line), w1, w2, false);
					// X_j += eta_i P_i . T_ij, four values at a time
					const double2 *pi = Pall + i * F::PP + s * F::Q + row;
					const double coef = i == 0 ? 1.0 : -1.0;
#pragma unroll
					for (int h = 0; h < 2; h++) {
						double2 a[4], w[4];
#pragma unroll
						for (int e = 0; e < 4; e++) w[e] = __ldcg(pi + 8 * (4 * h + e));
						if (s < 3) {
							tmem_ld4(F::taddr(tbase, s) + 16 * h, a);
							tmem_wait_ld();
						} else {
#pragma unroll
							for (int e = 0; e < 4; e++) a[e] = Xo[3 * F::Q + 8 * (4 * h + e)];
						}
#pragma unroll
						for (int e = 0; e < 4; e++) {
							const double2 y = cmul(w[e], x[4 * h + e]);
							a[e].x += coef * y.x;
							a[e].y += coef * y.y;
						}
						if (s < 3) tmem_st4(F::taddr(tbase, s) + 16 * h, a);
						else {
#pragma unroll
							for (int e = 0; e < 4; e++) Xo[3 * F::Q + 8 * (4 * h + e)] = a[e];
						}
					}
					// Y_i += eta_j W^_j . T_ij
					if (pr) {
						const double2 *wj = Wc + j * F::PP + s * F::Q;
						double2 *y = Yall + i * F::PP + s * F::Q + row;
						double2 a[8];
						if (c > 0) {
#pragma unroll
							for (int e = 0; e < 8; e++) a[e] = __ldcg(y + 8 * e);
						}
#pragma unroll
						for (int e = 0; e < 8; e++) {
							double2 b = cscale(cmul(wj[8 * e], x[e]), etaj);
							if (c > 0) b = cadd(a[e], b);
							__stcg(y + 8 * e, b);
						}
					}
					tmem_wait_st();
				}
				if (pr || c == 3) cl.sync();                 // one CTA a round adds to Y_i; the P grids are read
			}
			if (!pr) continue;
			// Z_j += conj(psi1) . Extract(IFFT2(Y_j))
#pragma unroll 1
			for (int s = 0; s < 4; s++) {
				const double2 *y = Yall + j * F::PP + s * F::Q + row;
				double2 x[8];
#pragma unroll
				for (int r = 0; r < 8; r++) x[r] = __ldcg(y + 8 * r);
				fft64_q<+1>(x, tau, G::row(Ug, line), w1, w2, s > 0);
#pragma unroll
				for (int e = 0; e < 8; e++) Ug[G::at(line, tau + 8 * e)] = x[e];
				__syncthreads();
#pragma unroll
				for (int r = 0; r < 8; r++) x[r] = Ug[G::at(tau + 8 * r, line)];
				fft64_q<+1>(x, tau, G::col(Ug, line), w1, w2, false);
				if (s == 0) {
#pragma unroll
					for (int e = 0; e < 8; e++) st0[e * F::NT] = x[e];
					continue;
				}
#pragma unroll
				for (int e = 0; e < 8; e++) {
					const int l = tau + 8 * e;
					double2 v = cmul(conj_c(tw[(s & 2 ? l : 0) + (s & 1 ? line : 0)]), x[e]);
					if (((s & 2) && e >= 4) != ((s & 1) && line >= 32)) { v.x = -v.x; v.y = -v.y; }
					v = cadd(st0[e * F::NT], v);
					if (s < 3) st0[e * F::NT] = v;
					else Zo[8 * e * 64] = cfma(conj_c(psi1[8 * e * 64]), v, Zo[8 * e * 64]);
				}
			}
		}
#pragma unroll 1
		for (int s = 0; s < 3; s++) {
			double2 a[8];
			tmem_ld8(F::taddr(tbase, s), a);
			tmem_wait_ld();
#pragma unroll
			for (int e = 0; e < 8; e++) Xo[s * F::Q + 8 * e] = a[e];
		}
	}
	tmem_fence_before();
	__syncthreads();
	tmem_fence_after();
	if (warp == 0) tmem_dealloc(tbase, F::TCOLS);
}

}  // namespace qb
