// qb_grid16.cuh — the I3 sums at N = 24 and 48 with a whole padded P x P grid, P = 16
// R (R = 3, 6), in one CTA.
//
// A 2-D transform is three register stages with two exchanges through the
// shared grid, as in qb_wide64.cuh with 4 replaced by R:
//   A  item (l, tau), values k = tau + R r:               DFT16 over r -> q
//   B  item (q, lam), values (l = lam + 16 s, tau):       x w_P^(tau q), DFT_R over tau
//      -> p and over s -> u, x w_P^(lam u)
//   C  item (q + 16 p, u), values lam:                    DFT16 over lam -> v
// gives b(u + R v, q + 16 p); the forward transform is the mirror image.  A and C
// have P R items of 16 values, B 256 items of R^2.  Every stage works item by
// item and writes the slots it read, so a thread never holds more than one
// item, whatever the number of items a thread.
#pragma once
#include <type_traits>
#include "qb_kernels.cuh"
#include "qb_radix.cuh"

namespace qb {

template <int R_, class C> struct Grid16 {
	static constexpr int R = R_, P = 16 * R, N = P / 2, PP = P * P, ITEMS = P * R;
	// threads: two items each of A and C at R = 6, one at R = 3 (whole warps)
	static constexpr int NT = R == 6 ? 288 : 160, IT = (ITEMS + NT - 1) / NT;
	// row pitch: 16 lanes of 8 bytes (8 of 16) of A are rows of R consecutive values, of
	// B 16 (8) rows; odd, and close to R modulo 16 (8)
	static constexpr int LDP = P + (R == 3 ? 3 : sizeof(C) == 8 ? 3 : 5);
	static constexpr int GRID = P * LDP;
	C *U;
	const C *tw;                             // w_P^e, e < P, forward sign

	__device__ __forceinline__ static int col_of(int c) { return c / R + 16 * (c % R); }      // grid column of column slot c of C
	// item of A: element (row, tau + R r) in x[r]
	template <class F> __device__ __forceinline__ void slots_a(int item, const F &f) const {
		C *u = U + (item / R) * LDP + item % R;
#pragma unroll
		for (int q = 0; q < 16; q++) f(q, u[R * q]);
	}
	// item of C: row slot u = item / P, column slot c = item % P
	template <class F> __device__ __forceinline__ void slots_c(int item, const F &f) const {
		C *u = U + (item / P) * 16 * LDP + item % P;
#pragma unroll
		for (int m = 0; m < 16; m++) f(m, u[m * LDP]);
	}
	template <int DIR> __device__ __forceinline__ void stage_b() const {
		for (int item = threadIdx.x; item < 256; item += NT) {
			const int q = item >> 4, lam = item & 15;
			C *u = U + lam * LDP + R * q;
			C y[R][R];                       // [s or u][tau or p]
#pragma unroll
			for (int r = 0; r < R; r++)
#pragma unroll
				for (int c = 0; c < R; c++) {
					C v = u[r * 16 * LDP + c];
					if (DIR > 0 ? c > 0 : r > 0) {
						C w = DIR > 0 ? tw[c * q] : tw[r * lam];
						if (DIR > 0) w.y = -w.y;
						v = cmul(v, w);
					}
					y[r][c] = v;
				}
#pragma unroll
			for (int r = 0; r < R; r++) dft_r<R, DIR>(y[r]);
#pragma unroll
			for (int c = 0; c < R; c++) {
				C v[R];
#pragma unroll
				for (int r = 0; r < R; r++) v[r] = y[r][c];
				dft_r<R, DIR>(v);
				const int fc = freq_of<R>(c);
#pragma unroll
				for (int r = 0; r < R; r++) {
					const int fr = freq_of<R>(r);
					if (DIR > 0 ? fr > 0 : fc > 0) {
						C w = DIR > 0 ? tw[fr * lam] : tw[fc * q];
						if (DIR > 0) w.y = -w.y;
						v[r] = cmul(v[r], w);
					}
					u[fr * 16 * LDP + fc] = v[r];
				}
			}
		}
	}
};

// k_i3g: clusters of 4 CTAs, CTA j for component j; RF: the real form (FP32), as in
// k_i3wr (qb_wide64.cuh): chains of i = 2c, 2c + 1 packed, real P, W^ and X_j.  Per unit CTA j
// writes P_j to the cluster's scratch in L2; after a cluster barrier it runs its
// chains (4, or 2 packed): X_j += eta_i P_i . T_ij, and for the other term of a pair
// y = eta_j W^_j . T_ij is transformed at once, item by item into the same grid,
// and conj(psi1) . Extract of it added to the CTA's own partial of Z_i (the sum
// over j is left to the assembly: half a chain more a chain, but no exchange
// between the CTAs).  W^, P, psi2 and X are in item order (value r of item i at
// ITEMS r + i).  Clusters take the (cell, chunk) pieces of the form `form` in turn.
// Bound by the latency of its operands from L2 at two CTAs of 9 warps an SM (P =
// 96, complex: shared-memory pipe 56%, issue 32%); against the three passes over
// global memory, see AnyRhs::fused_i3.
template <class C> struct I3GridP {
	using Rl = typename CT<C>::R;
	int ncells, nchunk, nunits, form;        // form 1: complex, 0: real
	I3Units un;
	const int *kind;                         // null: every cell complex
	const double2 *src;                      // N x N states [cell][4]
	const C *WI;                             // W^ in item order [cell][4]
	const Rl *WR;                            // its real parts (RF)
	const C *psi1;
	const Rl *psi2;                          // [angle] in the item order of C
	const double *scale;
	C *pscr;                                 // [cluster][2][4][PP]
	C *xscr;                                 // [cluster][4][PP], X of the forms that keep it in L2
	C *X;                                    // [cell][4][nchunk][PP] natural
	double2 *Z;                                  // [cell][4][4 nchunk][(N + 1)^2]
};
template <int R, class C, bool RF> struct I3Grid {
	static constexpr bool XS = R == 3 || RF; // X in shared memory
	using Xt = typename std::conditional<RF, float, C>::type;
	static constexpr size_t SMEM = sizeof(C) * (Grid16<R, C>::GRID + Grid16<R, C>::P) + (XS ? sizeof(Xt) * Grid16<R, C>::PP : 0);
	static constexpr int CTAS = R == 6 ? (sizeof(C) == 8 ? 2 : 1) : (sizeof(C) == 8 ? 3 : 2);
};
template <int R, class C, bool RF>
__global__ void __launch_bounds__((Grid16<R, C>::NT), (I3Grid<R, C, RF>::CTAS)) k_i3g(const I3GridP<C> p) {
	using F = Grid16<R, C>;
	using Rl = typename CT<C>::R;
	using Pt = typename std::conditional<RF, float, C>::type;       // P, W^ and X
	constexpr int P = F::P, N = F::N, NN = N * N, PP = F::PP, ITEMS = F::ITEMS, H = N / 2, ZS = N + 1, ZA = ZS * ZS;
	constexpr int NC = RF ? 2 : 4;
	constexpr bool XS = I3Grid<R, C, RF>::XS;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *U = reinterpret_cast<C *>(smem_raw), *tw = U + F::GRID;
	cg::cluster_group cl = cg::this_cluster();
	const int j = (int)cl.block_rank(), cid = (int)(blockIdx.x / 4), ncl = (int)(gridDim.x / 4);
	Pt *X = XS ? reinterpret_cast<Pt *>(tw + P) : reinterpret_cast<Pt *>(p.xscr + ((long)cid * 4 + j) * PP);
	init_twiddles<P>(tw);
	const F G{ U, tw };
	Pt *Pall = reinterpret_cast<Pt *>(p.pscr + (long)cid * 8 * PP);
	const Rl etaj = (Rl)(j == 0 ? 1.0 : -1.0);
	int par = 0;
#pragma unroll 1
	for (long piece = cid; piece < (long)p.ncells * p.nchunk; piece += ncl) {
		const long cell = piece / p.nchunk;
		const int chunk = (int)(piece % p.nchunk);
		if (p.kind != nullptr && p.kind[cell] != p.form) continue;
		const double2 *src = p.src + (cell * 4 + j) * NN;
		const Pt *Wc = RF ? reinterpret_cast<const Pt *>(p.WR) + cell * 4 * PP : reinterpret_cast<const Pt *>(p.WI) + cell * 4 * PP;
		const long nzp = 4L * p.nchunk;
		double2 *Zc = p.Z + (cell * 4 * nzp + chunk * 4 + j) * ZA;         // grid i at i nzp ZA
		for (int i = threadIdx.x; i < PP; i += F::NT) X[i] = Pt{};
		for (int i = threadIdx.x; i < NC * ZA; i += F::NT) Zc[(i / ZA) * nzp * ZA + i % ZA] = czero();
		const int u0 = (int)((long)chunk * p.nunits / p.nchunk), u1 = (int)((long)(chunk + 1) * p.nunits / p.nchunk);
		__syncthreads();
#pragma unroll 1
		for (int un = u0; un < u1; un++) {
			const int term = p.un.term(un);
			const bool pr = p.un.pair(un);
			const C *psi1 = p.psi1 + (long)term * NN;
			const Rl *psi2 = p.psi2 + (long)(term / p.un.M) * PP;
			const Rl sc = (Rl)p.scale[term];
			Pt *Pu = Pall + par * 4 * PP;
			par ^= 1;
			C x[16];
			// P_j = FFT2(Pad(psi1 . W_j))
#pragma unroll 1
			for (int item = threadIdx.x; item < ITEMS; item += F::NT) {
				const int u = item / P, k = F::col_of(item % P), ks = k < H ? k : (k >= P - H ? k - N : -1);
#pragma unroll
				for (int v = 0; v < 16; v++) {
					const int l = u + R * v, ls = l < H ? l : (l >= P - H ? l - N : -1);
					x[v] = czero<C>();
					if (ls >= 0 && ks >= 0) {
						const double2 w = src[ls * N + ks];
						x[v] = cmul(psi1[ls * N + ks], mk<C>(w.x, w.y));
					}
				}
				dft_r<16, -1>(x);
				G.slots_c(item, [&](int m, C &v) { v = x[(m & 3) * 4 + (m >> 2)]; });
			}
			__syncthreads();
			G.template stage_b<-1>();
			__syncthreads();
#pragma unroll 1
			for (int item = threadIdx.x; item < ITEMS; item += F::NT) {
				G.slots_a(item, [&](int q, const C &v) { x[q] = v; });
				dft_r<16, -1>(x);
#pragma unroll
				for (int r = 0; r < 16; r++) {
					const C v = x[(r & 3) * 4 + (r >> 2)];
					if constexpr (RF) __stcg(Pu + j * PP + ITEMS * r + item, v.x);
					else __stcg(Pu + j * PP + ITEMS * r + item, v);
				}
			}
			cl.sync();                                       // the unit's P grids are in L2
#pragma unroll 1
			for (int c = 0; c < NC; c++) {
				// inverse transform of W^_c . P_j (RF: (W^_2c + i W^_2c+1) . P_j)
#pragma unroll 1
				for (int item = threadIdx.x; item < ITEMS; item += F::NT) {
					const Pt *pj = Pu + j * PP + item, *w = Wc + (RF ? 2 * c : c) * PP + item;
#pragma unroll
					for (int r = 0; r < 16; r++) {
						if constexpr (RF) x[r] = cscale(mk<C>(w[ITEMS * r], w[PP + ITEMS * r]), __ldcg(pj + ITEMS * r));
						else x[r] = cmul(w[ITEMS * r], __ldcg(pj + ITEMS * r));
					}
					dft_r<16, +1>(x);
					G.slots_a(item, [&](int q, C &v) { v = x[(q & 3) * 4 + (q >> 2)]; });
				}
				__syncthreads();
				G.template stage_b<+1>();
				__syncthreads();
				// inverse, times psi2, forward: columns slots in place
#pragma unroll 1
				for (int item = threadIdx.x; item < ITEMS; item += F::NT) {
					Rl f[16];
#pragma unroll
					for (int v = 0; v < 16; v++) f[v] = psi2[ITEMS * v + item];
					G.slots_c(item, [&](int m, const C &v) { x[m] = v; });
					dft_r<16, +1>(x);
					C y[16];
#pragma unroll
					for (int v = 0; v < 16; v++) y[v] = cscale(x[(v & 3) * 4 + (v >> 2)], f[v]);
					dft_r<16, -1>(y);
					G.slots_c(item, [&](int m, C &v) { v = y[(m & 3) * 4 + (m >> 2)]; });
				}
				__syncthreads();
				G.template stage_b<-1>();
				__syncthreads();
				// T_cj: X_j, and the first stage of IFFT2(eta_j W^_j . T)
#pragma unroll 1
				for (int item = threadIdx.x; item < ITEMS; item += F::NT) {
					const Pt *pi = Pu + (RF ? 2 * c : c) * PP + item, *wj = Wc + j * PP + item;
					Pt *xo = X + item;
					G.slots_a(item, [&](int q, const C &v) { x[q] = v; });
					dft_r<16, -1>(x);
#pragma unroll
					for (int r = 0; r < 16; r++) {
						const C v = x[(r & 3) * 4 + (r >> 2)];
						if constexpr (RF) {
							const float c0 = c == 0 ? sc : -sc;          // eta_2c; eta_2c+1 = -1
							xo[ITEMS * r] += c0 * (__ldcg(pi + ITEMS * r) * v.x) - sc * (__ldcg(pi + PP + ITEMS * r) * v.y);
						} else {
							const Rl ci = c == 0 ? sc : -sc;
							const C a = cmul(__ldcg(pi + ITEMS * r), v);
							C o = xo[ITEMS * r];
							o.x += ci * a.x;
							o.y += ci * a.y;
							xo[ITEMS * r] = o;
						}
					}
					if (pr) {
						C y[16];
						const Rl cj = etaj * sc;
#pragma unroll
						for (int r = 0; r < 16; r++) {
							const C v = x[(r & 3) * 4 + (r >> 2)];
							if constexpr (RF) y[r] = cscale(v, cj * wj[ITEMS * r]);
							else y[r] = cscale(cmul(wj[ITEMS * r], v), cj);
						}
						dft_r<16, +1>(y);
						G.slots_a(item, [&](int q, C &v) { v = y[(q & 3) * 4 + (q >> 2)]; });
					}
				}
				if (!pr) continue;                               // the next chain writes the items just read
				__syncthreads();
				G.template stage_b<+1>();
				__syncthreads();
				double2 *Zi = Zc + c * nzp * ZA;
#pragma unroll 1
				for (int item = threadIdx.x; item < ITEMS; item += F::NT) {
					const int u = item / P, k = F::col_of(item % P), zk = k <= H ? k : k - P;
					if (zk < -H || (!RF && zk == H)) continue;
					G.slots_c(item, [&](int m, const C &v) { x[m] = v; });
					dft_r<16, +1>(x);
#pragma unroll
					for (int v = 0; v < 16; v++) {
						const int l = u + R * v, zl = l <= H ? l : l - P;
						if (zl < -H || (!RF && zl == H) || (zl == H && zk == -H) || (zl == -H && zk == H)) continue;
						// psi1 is tabulated on -N/2 .. N/2 - 1; at the upper end it is conj psi1(-k)
						const bool up = zl == H || zk == H;
						const int a = up ? -zl : zl, b = up ? -zk : zk;
						C w = psi1[(a < 0 ? a + N : a) * N + (b < 0 ? b + N : b)];
						if (!up) w.y = -w.y;
						zadd_mem(Zi + (zl + H) * ZS + zk + H, w, x[(v & 3) * 4 + (v >> 2)]);
					}
				}
				__syncthreads();                                 // the next chain writes rows
			}
			__syncthreads();                                     // the next unit's P_j writes columns
		}
		C *o = p.X + ((cell * 4 + j) * p.nchunk + chunk) * PP;
		for (int i = threadIdx.x; i < PP; i += F::NT) {
			// natural element i: item (l, tau), value r with k = tau + R r
			const int l = i / P, k = i % P;
			const Pt v = X[ITEMS * (k / R) + l * R + k % R];
			if constexpr (RF) o[i] = mk<C>(v, 0.0);
			else o[i] = v;
		}
		__syncthreads();                                         // X is read
	}
	cl.sync();
}

// W^ (natural order, ngrids grids) in item order, and its real parts (wr null: none)
template <int R, class C> __global__ void __launch_bounds__(256) k_to_items(const C *__restrict__ w, C *__restrict__ wi, float *__restrict__ wr) {
	using F = Grid16<R, C>;
	const long g = (long)blockIdx.y * F::PP;
	const int i = blockIdx.x * 256 + threadIdx.x;               // value r of item: ITEMS r + item
	if (i >= F::PP) return;
	const int item = i % F::ITEMS, r = i / F::ITEMS;
	const C v = w[g + (item / R) * F::P + item % R + R * r];
	wi[g + i] = v;
	if (wr != nullptr) wr[g + i] = (float)v.x;
}
// the transposed psi2 tables ([k][l]) in the item order of C
template <int R, class C> __global__ void __launch_bounds__(256) k_psi2_items(const typename CT<C>::R *__restrict__ t, typename CT<C>::R *__restrict__ o) {
	using F = Grid16<R, C>;
	const long g = (long)blockIdx.y * F::PP;
	const int i = blockIdx.x * 256 + threadIdx.x;
	if (i >= F::PP) return;
	const int item = i % F::ITEMS, v = i / F::ITEMS;
	o[g + i] = t[g + F::col_of(item % F::P) * F::P + item / F::P + R * v];
}

}  // namespace qb
