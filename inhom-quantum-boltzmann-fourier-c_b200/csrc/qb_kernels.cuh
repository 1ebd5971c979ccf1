// qb_kernels.cuh — collision kernels for sm_100a, generic over the working
// complex type C (double2: the plain FP64 path; float2: the FP32 precision
// form); the Wigner state itself is always FP64.
//
// Notation: N = velocity grid size, P = 2N padded size, all Fourier-space
// grids complex, element (l, k) at index k + n*l.  A P x P grid in shared
// memory is addressed through Geo::at(row, column): row pitch P + 1 for FP64
// (row passes, column passes and the in-line exchanges free of bank
// conflicts), a wider pitch and, at P = 64, an XOR column swizzle for FP32.
// A CTA has P*T threads (T = P/8 lanes per line,
// one line = one row or one column): thread tid works on line tid / T as
// lane tau = tid % T.
//
// The collision right-hand side is evaluated in factored form (upstream
// loops: src/integrals.c:90-379, src/collision.c:74-254):
//   x^ = FFT2(Pad(x)) for the four Pauli components (k_pad_fft)
//   I1/I4-type sums  S = sum_t phi_t . IFFT2(F . FFT2(Pad(psi2_t . g)))  (k_i1_terms)
//   I2-type sums     Q = sum_t FFT2(Pad(psi1_t f)) . FFT2(Pad(psi2_t g))  (k_i2_terms)
//   I3-type sums     X_r = sum_t sum_i coef_i P_{t,a_i} . FFT2(psi2_t . IFFT2(G_i . P_{t,r}))
//                    with P_{t,c} = FFT2(Pad(psi1_t . W_c))               (k_i3q here, k_i3w in
//                    qb_wide64.cuh and others at larger N; k_i3 for the single integrals)
//   then outer FFT/IFFT, Extract and the Pauli combination (k_fft_full, k_assemble).
// Moving the sums over quadrature terms inside the outer transforms is exact
// in real arithmetic; results agree with the upstream loop order to rounding.
#pragma once
#include <type_traits>
#include <cooperative_groups.h>
#include "qb_fft.cuh"

namespace qb {

namespace cg = cooperative_groups;

template <int P, class C = double2> struct Geo {
	static constexpr int N = P / 2;
	static constexpr int T = Len<P>::T;
	// row pitch: P + 1 makes every 16-byte (FP64) access pattern of the row,
	// column and exchange passes conflict-free; with 8-byte (FP32) values a
	// half-warp spans two lines, and the pads below halve the excess wavefronts
	// of P + 1 (bank model of all the patterns, 1.5x of ideal instead of 2x)
	static constexpr int LDP = sizeof(C) == 16 ? P + 1 : (P == 64 ? P + 8 : (P == 32 ? P + 4 : P + 2));
	// FP32 at P = 64: pitch P + 8 with the column index XOR-ed by 2 ((row >> 1) & 3)
	// makes every pattern conflict-free (a half-warp's two lines land on
	// opposite halves of the banks, and the swizzle spreads a column's rows)
	static constexpr bool SWZ = sizeof(C) == 8 && P == 64;
	__device__ __forceinline__ static int swz(int r) { return SWZ ? 2 * ((r >> 1) & 3) : 0; }
	// slot of element (row r, column c) of a grid in shared memory
	__device__ __forceinline__ static int at(int r, int c) { return r * LDP + (c ^ swz(r)); }
	// scratch accessors of a row / a column for the transforms
	struct RowA { C *p; int m; __device__ __forceinline__ C &operator()(int pos) const { return p[pos ^ m]; } };
	struct ColA { C *S; int c; __device__ __forceinline__ C &operator()(int pos) const { return S[at(pos, c)]; } };
	__device__ __forceinline__ static RowA row(C *S, int r) { return RowA{ S + r * LDP, swz(r) }; }
	__device__ __forceinline__ static ColA col(C *S, int c) { return ColA{ S, c }; }
	static constexpr int NT = P * T;            // threads per CTA
	static constexpr int GRID = P * LDP;        // smem slots of one padded grid
	// padded index -> index in the N grid, or -1 inside the zero band
	__device__ __forceinline__ static int src(int p) { return p < N / 2 ? p : (p >= 3 * N / 2 ? p - N : -1); }
	// N-grid index -> padded index (GridZeroPad, upstream src/grid.c:171-188)
	__device__ __forceinline__ static int pad(int k) { return k < N / 2 ? k : k + N; }
};

// resident CTAs per SM the term kernels are compiled for: the FP64 kernels
// need ~128 registers a thread (one 512-thread CTA per SM at P = 64); the
// FP32 ones fit two CTAs
template <class C> struct Occ { static constexpr int CTAS = 1; };
template <> struct Occ<float2> { static constexpr int CTAS = 2; };

// ---------------------------------------------------------------------------
// multipliers applied to the FP64 N-grid state before zero padding; the
// product is formed in the working precision C
template <class C> struct MulNone {
	__device__ __forceinline__ C operator()(int, double2 v) const { return mk<C>(v.x, v.y); }
};
template <class C> struct MulReal {           // psi (real N x N) .* v   (MultiplyPointwiseRC)
	const typename CT<C>::R *psi;
	__device__ __forceinline__ C operator()(int idx, double2 v) const { return cscale(mk<C>(v.x, v.y), psi[idx]); }
};
template <class C> struct MulCplx {           // psi (complex N x N) .* v   (MultiplyPointwiseCC)
	const C *psi;
	__device__ __forceinline__ C operator()(int idx, double2 v) const { return cmul(psi[idx], mk<C>(v.x, v.y)); }
};

// lane's 8 inputs of padded row `prow` of Pad(mul . src)
template <int P, class C, class Mul>
__device__ __forceinline__ void load_pad_row(C (&x)[8], int prow, int tau, const double2 *__restrict__ src, const Mul &mul) {
	using G = Geo<P, C>;
	const int l = G::src(prow);
#pragma unroll
	for (int r = 0; r < 8; r++) {
		const int k = G::src(tau + G::T * r);
		x[r] = (l >= 0 && k >= 0) ? mul(k + G::N * l, src[k + G::N * l]) : czero<C>();
	}
}

// FFT2 (direction DIR) of Pad(mul . src) into the smem grid S (in place, two passes)
template <int P, int DIR, class C, class Mul>
__device__ __forceinline__ void fft2_pad(C *S, const C *tw, const double2 *__restrict__ src, const Mul &mul) {
	using G = Geo<P, C>;
	const int line = threadIdx.x / G::T, tau = threadIdx.x % G::T;
	C x[8];
	load_pad_row<P>(x, line, tau, src, mul);
	fft1d_acc<P, DIR>(x, tau, G::row(S, line), tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[G::at(line, Len<P>::out_pos(tau, e))] = x[e];
	__syncthreads();
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = S[G::at(tau + G::T * r, line)];
	fft1d_acc<P, DIR>(x, tau, G::col(S, line), tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[G::at(Len<P>::out_pos(tau, e), line)] = x[e];
	__syncthreads();
}

// FFT2 of a full grid already in smem S (natural layout), in place
template <int P, int DIR, class C>
__device__ __forceinline__ void fft2_smem(C *S, const C *tw) {
	using G = Geo<P, C>;
	const int line = threadIdx.x / G::T, tau = threadIdx.x % G::T;
	C x[8];
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = S[G::at(line, tau + G::T * r)];
	fft1d_acc<P, DIR>(x, tau, G::row(S, line), tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[G::at(line, Len<P>::out_pos(tau, e))] = x[e];
	__syncthreads();
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = S[G::at(tau + G::T * r, line)];
	fft1d_acc<P, DIR>(x, tau, G::col(S, line), tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[G::at(Len<P>::out_pos(tau, e), line)] = x[e];
	__syncthreads();
}

// copy smem grid (pitch LDP) to a dense global P x P grid, coalesced
template <int P, class C>
__device__ __forceinline__ void smem_to_global(C *__restrict__ out, const C *S) {
	using G = Geo<P, C>;
	for (int i = threadIdx.x; i < P * P; i += G::NT) out[i] = S[G::at(i / P, i % P)];
}

// ---------------------------------------------------------------------------
// K1: padded forward spectra  out[b] = FFT2(Pad(src[b]))   (one CTA per grid);
// out2 (may be null, P = 64): the same in the thread order of k_i3w; outr (may be
// null): its real parts in that order
template <int P, class C>
__global__ void __launch_bounds__(Geo<P>::NT) k_pad_fft(const double2 *__restrict__ src, C *__restrict__ out, C *__restrict__ out2, float *__restrict__ outr) {
	using G = Geo<P, C>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *S = reinterpret_cast<C *>(smem_raw), *tw = S + G::GRID;
	init_twiddles<P>(tw);
	__syncthreads();
	const long b = blockIdx.x;
	fft2_pad<P, -1>(S, tw, src + b * G::N * G::N, MulNone<C>{});
	smem_to_global<P>(out + b * P * P, S);
	if (P == 64 && out2 != nullptr)
		for (int i = threadIdx.x; i < P * P; i += G::NT) {
			const C v = S[G::at((i & 255) >> 2, (i & 3) + 4 * (i >> 8))];
			out2[b * P * P + i] = v;
			if (outr != nullptr) outr[b * P * P + i] = (float)v.x;
		}
}

// ---------------------------------------------------------------------------
// K2: I1/I4-type term sums
//   S[cell][task][chunk] = sum_{t in chunk} phi_t . IFFT2(F . FFT2(Pad(psi2_t . g)))
//   g = gsrc[cell][g_comp[task]],  F = fa * What[cell][f_comp] + fb
template <class C> struct I1ParamsT {
	using R = typename CT<C>::R;
	int ntask, nchunk, nterms;
	const double2 *g; long g_cell;          // N x N grids (FP64 state)
	int g_comp[4];
	const C *What; long w_cell;             // P x P grids
	int f_comp; double fa, fb;
	const R *psi2;                          // nterms x N x N
	const R *phi;                           // nterms x P x P
	C *out;                                 // [cell][task][chunk][P*P]
};
using I1Params = I1ParamsT<double2>;

template <int P, class C>
__global__ void __launch_bounds__(Geo<P>::NT) k_i1_terms(const I1ParamsT<C> p) {
	using G = Geo<P, C>;
	using Lp = Len<P>;
	using R = typename CT<C>::R;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *S = reinterpret_cast<C *>(smem_raw), *F = S + G::GRID, *tw = S + 2 * G::GRID;
	const int chunk = blockIdx.x % p.nchunk;
	const int task = (blockIdx.x / p.nchunk) % p.ntask;
	const long cell = blockIdx.x / (p.nchunk * p.ntask);
	init_twiddles<P>(tw);
	const C *W = p.What + cell * p.w_cell + (long)p.f_comp * P * P;
	const R fa = (R)p.fa, fb = (R)p.fb;
	for (int i = threadIdx.x; i < P * P; i += G::NT) {
		const C w = W[i];
		C f; f.x = fa * w.x + fb; f.y = fa * w.y;
		F[G::at(i / P, i % P)] = f;
	}
	__syncthreads();
	const double2 *g = p.g + cell * p.g_cell + (long)p.g_comp[task] * G::N * G::N;
	const int t0 = (int)((long)chunk * p.nterms / p.nchunk), t1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
	const int line = threadIdx.x / G::T, tau = threadIdx.x % G::T;
	C acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = czero<C>();
	for (int t = t0; t < t1; t++) {
		C x[8];
		// rows: FFT of Pad(psi2_t . g)
		load_pad_row<P>(x, line, tau, g, MulReal<C>{p.psi2 + (long)t * G::N * G::N});
		fft1d_acc<P, -1>(x, tau, G::row(S, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) S[G::at(line, Lp::out_pos(tau, e))] = x[e];
		__syncthreads();
		// columns: FFT, multiply by F (convolution with f), inverse FFT
#pragma unroll
		for (int r = 0; r < 8; r++) x[r] = S[G::at(tau + G::T * r, line)];
		fft1d_acc<P, -1>(x, tau, G::col(S, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) x[e] = cmul(F[G::at(Lp::out_pos(tau, e), line)], x[e]);
		out_to_in_acc<P>(x, tau, G::col(S, line));
		fft1d_acc<P, +1>(x, tau, G::col(S, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) S[G::at(Lp::out_pos(tau, e), line)] = x[e];
		__syncthreads();
		// rows: inverse FFT, multiply by phi_t, accumulate
#pragma unroll
		for (int r = 0; r < 8; r++) x[r] = S[G::at(line, tau + G::T * r)];
		fft1d_acc<P, +1>(x, tau, G::row(S, line), tw);
		const R *phi = p.phi + (long)t * P * P + line * P;
#pragma unroll
		for (int e = 0; e < 8; e++) {
			const R f = phi[Lp::out_pos(tau, e)];
			acc[e].x += f * x[e].x;
			acc[e].y += f * x[e].y;
		}
		// no barrier: the next term's first pass writes only this group's row
	}
	C *o = p.out + ((cell * p.ntask + task) * p.nchunk + chunk) * (long)P * P + line * P;
#pragma unroll
	for (int e = 0; e < 8; e++) o[Lp::out_pos(tau, e)] = acc[e];
}

// ---------------------------------------------------------------------------
// K3: I2-type term sums
//   Q[cell][task][chunk] = sum_t FFT2(Pad(psi1_t . f)) . FFT2(Pad(psi2_t . g))
template <class C> struct I2ParamsT {
	using R = typename CT<C>::R;
	int ntask, nchunk, nterms;
	const double2 *src; long cell_stride;   // N x N grids (FP64 state)
	int f_comp[4], g_comp[4];
	const R *psi1, *psi2;                   // nterms x N x N each
	C *out;                                 // [cell][task][chunk][P*P]
};
using I2Params = I2ParamsT<double2>;

template <int P, class C>
__global__ void __launch_bounds__(Geo<P>::NT) k_i2_terms(const I2ParamsT<C> p) {
	using G = Geo<P, C>;
	using Lp = Len<P>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *A = reinterpret_cast<C *>(smem_raw), *B = A + G::GRID, *tw = A + 2 * G::GRID;
	const int chunk = blockIdx.x % p.nchunk;
	const int task = (blockIdx.x / p.nchunk) % p.ntask;
	const long cell = blockIdx.x / (p.nchunk * p.ntask);
	init_twiddles<P>(tw);
	__syncthreads();
	const double2 *f = p.src + cell * p.cell_stride + (long)p.f_comp[task] * G::N * G::N;
	const double2 *g = p.src + cell * p.cell_stride + (long)p.g_comp[task] * G::N * G::N;
	const int t0 = (int)((long)chunk * p.nterms / p.nchunk), t1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
	const int line = threadIdx.x / G::T, tau = threadIdx.x % G::T;
	C acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = czero<C>();
	for (int t = t0; t < t1; t++) {
		fft2_pad<P, -1>(A, tw, f, MulReal<C>{p.psi1 + (long)t * G::N * G::N});
		C x[8];
		load_pad_row<P>(x, line, tau, g, MulReal<C>{p.psi2 + (long)t * G::N * G::N});
		fft1d_acc<P, -1>(x, tau, G::row(B, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) B[G::at(line, Lp::out_pos(tau, e))] = x[e];
		__syncthreads();
#pragma unroll
		for (int r = 0; r < 8; r++) x[r] = B[G::at(tau + G::T * r, line)];
		fft1d_acc<P, -1>(x, tau, G::col(B, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) acc[e] = cfma(A[G::at(Lp::out_pos(tau, e), line)], x[e], acc[e]);
		__syncthreads();
	}
	// column-mapped accumulator -> smem -> coalesced store
#pragma unroll
	for (int e = 0; e < 8; e++) A[G::at(Lp::out_pos(tau, e), line)] = acc[e];
	__syncthreads();
	smem_to_global<P>(p.out + ((cell * p.ntask + task) * p.nchunk + chunk) * (long)P * P, A);
}

// ---------------------------------------------------------------------------
// K4: I3-type sums on a cluster of CS CTAs (one per source component), for the
// single integrals.
// CTA r of the cluster for (cell, chunk) computes P_r = FFT2(Pad(psi1_t . src_r))
// into its shared memory; the other CTAs read it through distributed shared
// memory.  For each of its combos (a, g, coef) it accumulates
//   X_r += coef * P_a . FFT2(psi2_t . IFFT2(G_g . P_r)).
// Contiguous ranges of the flattened (cell, term) work of the I3 sums, one per
// cluster: cluster k takes u in [start(k), start(k + 1)) of total = ncells x
// nterms, u = cell x nterms + term, and writes one partial per cell it
// touches to slot k x maxc + (cell - first_cell(k)).  Cell c's partials are
// those of clusters cluster_of(c nterms) .. cluster_of((c + 1) nterms - 1),
// summed in that order.  nslots = 0: the (cell, chunk) grid instead.
struct TermRanges {
	int nslots = 0, nterms = 0, maxc = 0;
	long total = 0;
	__host__ __device__ long start(int k) const { return (long)k * total / nslots; }
	__host__ __device__ int cluster_of(long u) const { return (int)(((u + 1) * nslots - 1) / total); }
	__host__ __device__ long first_cell(int k) const { return start(k) / nterms; }
};

// Units of the I3 sums.  The radial nodes of FourierI3 are Gauss-Legendre on
// [-R, R], so terms m and M - 1 - m of an angle have opposite shifts (psi1' =
// conj psi1) and equal weights (and one psi2 table), and both follow from the
// same chains T_ij = FFT2(psi2 . IFFT2(W^_i . P_j)):
//   X_j  += sum_i eta_i P_i . T_ij                       (the shift a)
//   Y_i   = sum_j eta_j W^_j . T_ij,
//   Z_i  += conj(psi1) . Extract(IFFT2(Y_i))             (the shift -a)
// because W_i(v) W_j(v - a) is W_i(v + a) W_j(v) shifted by a and psi2 commutes
// with shifts.  No product of N-grids reaches the aliases of the extracted
// points on the 2N grid, so the two forms agree for every W to rounding.  A
// pair takes 16 chains of two transforms instead of 32 and one transform a
// component more.  M = 0: the terms carry no such structure (caller-built
// tables) and every unit is one term; the middle node of an odd M is alone.
struct I3Units {
	int M = 0;
	__host__ __device__ int per_angle() const { return (M + 1) / 2; }
	__host__ __device__ int count(int nterms) const { return M > 0 ? nterms / M * per_angle() : nterms; }
	__device__ __forceinline__ int term(int u) const { return M > 0 ? u / per_angle() * M + u % per_angle() : u; }
	__device__ __forceinline__ bool pair(int u) const { return M > 0 && 2 * (u % per_angle()) != M - 1; }
};

// z += w y, the sums Z of both precisions: in FP64. Z is summed after the inverse
// transform, so the rounding of an FP32 sum of many units would spread over the
// whole velocity grid, where the energy weighs it with v^2; that of X stays where X
// is. With Z and the last transforms (k_assemble) in FP64, N = 32, J = M = 16, FP32:
// the energy production of Cd deviates by 2.6e-6 of the sum of |Cd| (rms of
// 48 cells) instead of 6.3e-6, and 1000 Strang steps (mean of 8 states) by 0.9e-6 from
// FP64 instead of 2.7e-6; term by term it was 2.7e-6 and 1.5e-6
template <class C> __device__ __forceinline__ void zadd(double2 &z, C w, C y) {
	z = cfma(widen(w), widen(y), z);
}
// the same in memory that this thread alone adds to (one order of the sums); in FP32
// without waiting for the old value: Strang step, 32 cells at N = 64, 41.9 -> 40.0 ms,
// 12 cells at N = 48, 8.1 -> 7.5 ms
__device__ __forceinline__ void zadd_mem(double2 *z, double2 w, double2 y) { *z = cfma(w, y, *z); }
__device__ __forceinline__ void zadd_mem(double2 *z, float2 w, float2 y) {
	const double2 v = cmul(widen(w), widen(y));
	atomicAdd(&z->x, v.x);
	atomicAdd(&z->y, v.y);
}

template <class C> struct I3ParamsT {
	using R = typename CT<C>::R;
	int nchunk, nterms;                                   // nterms: terms, or units of `un` in the kernels that pair them
	I3Units un;
	double2 *zout;                                        // Z_i partials, layout given at each kernel (pairing kernels)
	double2 *zscr;                                        // real forms: packed Z sums of the running cluster
	TermRanges rg;                                        // nslots > 0: one term range per cluster
	const double2 *src; long src_cell; int src_comp[4];   // N x N grids (FP64 state)
	const C *Ghat; long g_cell;                           // P x P grids, G_g at Ghat + cell*g_cell + g*P*P
	int ncombo[4]; int ca[4][4], cgi[4][4]; double ccoef[4][4];
	const C *psi1;                                        // nterms x N x N (complex)
	const R *psi2T;                                       // transposed P x P tables
	const int *psi2_idx; const double *psi2_scale;        // per term
	C *out;                                               // [cell][chunk][CS][P*P]
	int *err;                                             // error word of bounded waits (may be null)
};
using I3Params = I3ParamsT<double2>;

template <int P, int CS, class C>
__global__ void __launch_bounds__(Geo<P>::NT, Occ<C>::CTAS) k_i3(const I3ParamsT<C> p) {
	using G = Geo<P, C>;
	using Lp = Len<P>;
	using R = typename CT<C>::R;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *Pr = reinterpret_cast<C *>(smem_raw), *Ug = Pr + G::GRID, *tw = Pr + 2 * G::GRID;
	cg::cluster_group cluster = cg::this_cluster();
	const int rank = (int)cluster.block_rank();
	const long cid = blockIdx.x / CS;
	const int chunk = (int)(cid % p.nchunk);
	const long cell = cid / p.nchunk;
	init_twiddles<P>(tw);
	__syncthreads();
	const double2 *src = p.src + cell * p.src_cell + (long)p.src_comp[rank] * G::N * G::N;
	const int t0 = (int)((long)chunk * p.nterms / p.nchunk), t1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
	const int line = threadIdx.x / G::T, tau = threadIdx.x % G::T;
	C acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = czero<C>();
	const int nc = p.ncombo[rank];
	for (int t = t0; t < t1; t++) {
		fft2_pad<P, -1>(Pr, tw, src, MulCplx<C>{p.psi1 + (long)t * G::N * G::N});
		cluster.sync();
		const R *psi2 = p.psi2T + (long)p.psi2_idx[t] * P * P;
		const R sc = (R)p.psi2_scale[t];
		for (int c = 0; c < nc; c++) {
			const C *Gg = p.Ghat + cell * p.g_cell + (long)p.cgi[rank][c] * P * P;
			C x[8];
			// rows: IFFT of G_g . P_r
#pragma unroll
			for (int r = 0; r < 8; r++) {
				const int k = tau + G::T * r;
				x[r] = cmul(Gg[line * P + k], Pr[G::at(line, k)]);
			}
			fft1d_acc<P, +1>(x, tau, G::row(Ug, line), tw);
#pragma unroll
			for (int e = 0; e < 8; e++) Ug[G::at(line, Lp::out_pos(tau, e))] = x[e];
			__syncthreads();
			// columns: IFFT, multiply by psi2_t, FFT
#pragma unroll
			for (int r = 0; r < 8; r++) x[r] = Ug[G::at(tau + G::T * r, line)];
			fft1d_acc<P, +1>(x, tau, G::col(Ug, line), tw);
#pragma unroll
			for (int e = 0; e < 8; e++) {
				const R f = sc * psi2[line * P + Lp::out_pos(tau, e)];
				x[e].x *= f;
				x[e].y *= f;
			}
			out_to_in_acc<P>(x, tau, G::col(Ug, line));
			fft1d_acc<P, -1>(x, tau, G::col(Ug, line), tw);
#pragma unroll
			for (int e = 0; e < 8; e++) Ug[G::at(Lp::out_pos(tau, e), line)] = x[e];
			__syncthreads();
			// rows: FFT, multiply by P_a (remote), accumulate
#pragma unroll
			for (int r = 0; r < 8; r++) x[r] = Ug[G::at(line, tau + G::T * r)];
			fft1d_acc<P, -1>(x, tau, G::row(Ug, line), tw);
			const C *Pa = cluster.map_shared_rank(Pr, p.ca[rank][c]);
			const R coef = (R)p.ccoef[rank][c];
#pragma unroll
			for (int e = 0; e < 8; e++) {
				const C v = cmul(Pa[G::at(line, Lp::out_pos(tau, e))], x[e]);
				acc[e].x += coef * v.x;
				acc[e].y += coef * v.y;
			}
			__syncthreads();
		}
		cluster.sync();
	}
	C *o = p.out + ((cell * p.nchunk + chunk) * CS + rank) * (long)P * P + line * P;
#pragma unroll
	for (int e = 0; e < 8; e++) o[Lp::out_pos(tau, e)] = acc[e];
}

// ---------------------------------------------------------------------------
// K4q: the I3 sums of the collision operator at P = 16 and 32, all four
// components of a (cell, chunk) in one CTA of four groups of P T threads, group
// j for component j.  Per unit group j forms P_j, then the groups run the 16
// chains in four rounds, group j the chain of i = (j + round) % 4:
//   X_j += eta_i P_i . T_ij  (registers),  Y_i += eta_j W^_j . T_ij  (shared memory)
// In a round every i belongs to one group, so the Y sums need one CTA barrier
// a round and no atomics; after the last round group j transforms its own Y_j
// (see I3Units).  The P grids, work grids and Y sums of the four components
// (12 grids: 203 KB in FP64 at P = 32) replace the distributed shared memory
// of 4-CTA clusters, of which 33 fit the GPU (132 of 148 SMs), and a group's
// barriers hold back its own warps only.  Out as k_i3 with CS = 4; zout:
// [slot][4][N*N].
// Bound by latency at 16 warps an SM: Strang step of 33 cells at N = 16,
// J = 12, M = 9, FP64: 2.74 -> 1.70 ms (4-CTA clusters, term by term, before).
template <int P, class C> struct I3q {
	using G = Geo<P, C>;
	static constexpr int NT = 4 * G::NT;
	static constexpr size_t SMEM = sizeof(C) * (8 * (size_t)G::GRID + 4 * (size_t)P * P + P);
	static constexpr int CTAS = P == 16 ? 4 : (sizeof(C) == 8 ? 2 : 1);    // resident an SM, by registers and shared memory
};
template <int NT> __device__ __forceinline__ void group_sync(int g) {
	if constexpr (NT == 32) __syncwarp();
	else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(NT) : "memory");
}
template <int P, class C>
__global__ void __launch_bounds__(I3q<P, C>::NT, I3q<P, C>::CTAS) k_i3q(const I3ParamsT<C> p) {
	using G = Geo<P, C>;
	using Lp = Len<P>;
	using R = typename CT<C>::R;
	constexpr int GT = G::NT, N = G::N, NN = N * N;
	static_assert(P == 16 || P == 32, "P = 64 and up have kernels of their own");
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *Pg = reinterpret_cast<C *>(smem_raw), *Ug = Pg + 4 * G::GRID, *Yg = Ug + 4 * G::GRID, *tw = Yg + 4 * P * P;
	const int j = threadIdx.x / GT, tid = threadIdx.x % GT;
	const int line = tid / G::T, tau = tid % G::T;
	const int chunk = (int)(blockIdx.x % p.nchunk);
	const long cell = blockIdx.x / p.nchunk;
	init_twiddles<P>(tw);
	__syncthreads();
	C *Pj = Pg + j * G::GRID, *U = Ug + j * G::GRID;
	const double2 *src = p.src + cell * p.src_cell + (long)p.src_comp[j] * NN;
	const C *What = p.Ghat + cell * p.g_cell;
	const int u0 = (int)((long)chunk * p.nterms / p.nchunk), u1 = (int)((long)(chunk + 1) * p.nterms / p.nchunk);
	const R etaj = (R)(j == 0 ? 1.0 : -1.0);
	const int zk = G::src(line);                             // the extracted column of this thread, or -1
	C acc[8];
	double2 z[4];                                            // the thread's four extracted rows of column zk
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = czero<C>();
#pragma unroll
	for (int m = 0; m < 4; m++) z[m] = czero();
	// value index of the thread's m-th extracted row: T = 4: e = 0, 4 (rows below
	// P / 4), 3, 7 (from 3P / 4 on); T = 2: e = 2 m + tau
	auto zrow = [&](int m) { return G::src(Lp::out_pos(tau, P == 32 ? (m & 1) * 4 + (m >> 1) * 3 : 2 * m + tau)); };
	for (int u = u0; u < u1; u++) {
		const int t = p.un.term(u);
		const bool pr = p.un.pair(u);
		const C *psi1 = p.psi1 + (long)t * NN;
		C x[8];
		load_pad_row<P>(x, line, tau, src, MulCplx<C>{psi1});
		fft1d_acc<P, -1>(x, tau, G::row(Pj, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) Pj[G::at(line, Lp::out_pos(tau, e))] = x[e];
		group_sync<GT>(j);
#pragma unroll
		for (int r = 0; r < 8; r++) x[r] = Pj[G::at(tau + G::T * r, line)];
		fft1d_acc<P, -1>(x, tau, G::col(Pj, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) Pj[G::at(Lp::out_pos(tau, e), line)] = x[e];
		__syncthreads();
		const R *psi2 = p.psi2T + (long)p.psi2_idx[t] * P * P + line * P;
		const R sc = (R)p.psi2_scale[t];
#pragma unroll 1
		for (int c = 0; c < 4; c++) {
			const int i = (j + c) & 3;
			const C *Gg = What + i * P * P + line * P;
			// rows: IFFT of W^_i . P_j
#pragma unroll
			for (int r = 0; r < 8; r++) {
				const int k = tau + G::T * r;
				x[r] = cmul(Gg[k], Pj[G::at(line, k)]);
			}
			fft1d_acc<P, +1>(x, tau, G::row(U, line), tw);
#pragma unroll
			for (int e = 0; e < 8; e++) U[G::at(line, Lp::out_pos(tau, e))] = x[e];
			group_sync<GT>(j);
			// columns: IFFT, multiply by psi2_t, FFT
#pragma unroll
			for (int r = 0; r < 8; r++) x[r] = U[G::at(tau + G::T * r, line)];
			fft1d_acc<P, +1>(x, tau, G::col(U, line), tw);
#pragma unroll
			for (int e = 0; e < 8; e++) {
				const R f = sc * psi2[Lp::out_pos(tau, e)];
				x[e].x *= f;
				x[e].y *= f;
			}
			out_to_in_acc<P>(x, tau, G::col(U, line));
			fft1d_acc<P, -1>(x, tau, G::col(U, line), tw);
#pragma unroll
			for (int e = 0; e < 8; e++) U[G::at(Lp::out_pos(tau, e), line)] = x[e];
			group_sync<GT>(j);
			// rows: FFT, X_j += eta_i P_i . T_ij
#pragma unroll
			for (int r = 0; r < 8; r++) x[r] = U[G::at(line, tau + G::T * r)];
			fft1d_acc<P, -1>(x, tau, G::row(U, line), tw);
			const C *Pi = Pg + i * G::GRID;
			const R coef = (R)(i == 0 ? 1.0 : -1.0);
#pragma unroll
			for (int e = 0; e < 8; e++) {
				const C v = cmul(Pi[G::at(line, Lp::out_pos(tau, e))], x[e]);
				acc[e].x += coef * v.x;
				acc[e].y += coef * v.y;
			}
			if (pr) {
				// Y_i in the order of the threads (every group maps a thread to the same points)
				C *Y = Yg + i * P * P + tid;
				const C *Wj = What + j * P * P + line * P;
#pragma unroll
				for (int e = 0; e < 8; e++) {
					const C y = cscale(cmul(Wj[Lp::out_pos(tau, e)], x[e]), etaj);
					Y[e * GT] = c == 0 ? y : cadd(Y[e * GT], y);
				}
				__syncthreads();
			}
		}
		if (!pr) {
			__syncthreads();                                 // the P grids are read
			continue;
		}
		// Z_j += conj(psi1) . Extract(IFFT2(Y_j))
#pragma unroll
		for (int e = 0; e < 8; e++) x[e] = Yg[j * P * P + tid + e * GT];
		out_to_in_acc<P>(x, tau, G::row(U, line));
		fft1d_acc<P, +1>(x, tau, G::row(U, line), tw);
#pragma unroll
		for (int e = 0; e < 8; e++) U[G::at(line, Lp::out_pos(tau, e))] = x[e];
		group_sync<GT>(j);
		if (P == 16 || zk >= 0) {                            // P = 32: whole warps (lines 0 .. 7, 24 .. 31)
#pragma unroll
			for (int r = 0; r < 8; r++) x[r] = U[G::at(tau + G::T * r, line)];
			fft1d_acc<P, +1>(x, tau, G::col(U, line), tw);
			if (zk >= 0) {
#pragma unroll
				for (int m = 0; m < 4; m++) {
					C w = psi1[zrow(m) * N + zk];
					w.y = -w.y;
					C v;
					if constexpr (P == 32) v = x[(m & 1) * 4 + (m >> 1) * 3];
					else v = tau ? x[2 * m + 1] : x[2 * m];
					zadd(z[m], w, v);
				}
			}
		}
		group_sync<GT>(j);                                   // the next unit's chains reuse U
	}
	const long slot = cell * p.nchunk + chunk;
	C *o = p.out + (slot * 4 + j) * (long)P * P + line * P;
#pragma unroll
	for (int e = 0; e < 8; e++) o[Lp::out_pos(tau, e)] = acc[e];
	if (zk >= 0) {
		double2 *zo = p.zout + (slot * 4 + j) * (long)NN + zk;
#pragma unroll
		for (int m = 0; m < 4; m++) zo[zrow(m) * N] = z[m];
	}
}

// ---------------------------------------------------------------------------
// Tensor memory (TMEM) as accumulator storage.  A CTA allocates `ncols`
// columns of its SM's 128-lane TMEM; warp w reaches lanes 32 (w % 4) ..
// 32 (w % 4) + 31 (thread = lane), and the four warps that share a lane
// quarter split the columns (slot w / 4).  Loads and stores are warp-wide
// (tcgen05.ld / st .32x32b) and asynchronous until tcgen05.wait.
__device__ __forceinline__ void tmem_alloc(unsigned *slot_smem, unsigned ncols) {
	const unsigned a = (unsigned)__cvta_generic_to_shared(slot_smem);
	asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(ncols) : "memory");
	asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols) {
	asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// one complex value per thread at column `taddr` (+ 4 columns FP64, 2 FP32)
__device__ __forceinline__ void tmem_ld(unsigned taddr, double2 &v) {
	unsigned a, b, c, d;
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(taddr) : "memory");
	v.x = __hiloint2double((int)b, (int)a);
	v.y = __hiloint2double((int)d, (int)c);
}
__device__ __forceinline__ void tmem_st(unsigned taddr, double2 v) {
	const unsigned a = (unsigned)__double2loint(v.x), b = (unsigned)__double2hiint(v.x);
	const unsigned c = (unsigned)__double2loint(v.y), d = (unsigned)__double2hiint(v.y);
	asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_st(unsigned taddr, float2 v) {
	asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)) : "memory");
}

// eight consecutive complex values (32 columns FP64, 16 FP32) of this
// thread's lane in one warp-wide load or store
__device__ __forceinline__ void tmem_ld8(unsigned taddr, double2 (&v)[8]) {
	unsigned r[32];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
	             : "r"(taddr) : "memory");
#pragma unroll
	for (int e = 0; e < 8; e++) {
		v[e].x = __hiloint2double((int)r[4 * e + 1], (int)r[4 * e]);
		v[e].y = __hiloint2double((int)r[4 * e + 3], (int)r[4 * e + 2]);
	}
}
__device__ __forceinline__ void tmem_st8(unsigned taddr, const double2 (&v)[8]) {
	unsigned r[32];
#pragma unroll
	for (int e = 0; e < 8; e++) {
		r[4 * e] = (unsigned)__double2loint(v[e].x); r[4 * e + 1] = (unsigned)__double2hiint(v[e].x);
		r[4 * e + 2] = (unsigned)__double2loint(v[e].y); r[4 * e + 3] = (unsigned)__double2hiint(v[e].y);
	}
	asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
	             :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_ld8(unsigned taddr, float2 (&v)[8]) {
	unsigned r[16];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
	             : "r"(taddr) : "memory");
#pragma unroll
	for (int e = 0; e < 8; e++) { v[e].x = __uint_as_float(r[2 * e]); v[e].y = __uint_as_float(r[2 * e + 1]); }
}
__device__ __forceinline__ void tmem_st8(unsigned taddr, const float2 (&v)[8]) {
	unsigned r[16];
#pragma unroll
	for (int e = 0; e < 8; e++) { r[2 * e] = __float_as_uint(v[e].x); r[2 * e + 1] = __float_as_uint(v[e].y); }
	asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
	             :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// four consecutive FP64 complex values (16 columns) in one load or store
__device__ __forceinline__ void tmem_ld4(unsigned taddr, double2 (&v)[4]) {
	unsigned r[16];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
	             : "r"(taddr) : "memory");
#pragma unroll
	for (int e = 0; e < 4; e++) {
		v[e].x = __hiloint2double((int)r[4 * e + 1], (int)r[4 * e]);
		v[e].y = __hiloint2double((int)r[4 * e + 3], (int)r[4 * e + 2]);
	}
}
__device__ __forceinline__ void tmem_st4(unsigned taddr, const double2 (&v)[4]) {
	unsigned r[16];
#pragma unroll
	for (int e = 0; e < 4; e++) {
		r[4 * e] = (unsigned)__double2loint(v[e].x); r[4 * e + 1] = (unsigned)__double2hiint(v[e].x);
		r[4 * e + 2] = (unsigned)__double2loint(v[e].y); r[4 * e + 3] = (unsigned)__double2hiint(v[e].y);
	}
	asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
	             :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// eight FP32 reals (8 columns) in one load or store
__device__ __forceinline__ void tmem_ld8r(unsigned taddr, float (&v)[8]) {
	unsigned r[8];
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
	             : "r"(taddr) : "memory");
#pragma unroll
	for (int e = 0; e < 8; e++) v[e] = __uint_as_float(r[e]);
}
__device__ __forceinline__ void tmem_st8r(unsigned taddr, const float (&v)[8]) {
	unsigned r[8];
#pragma unroll
	for (int e = 0; e < 8; e++) r[e] = __float_as_uint(v[e]);
	asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
	             :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// ---------------------------------------------------------------------------
// K5: out[b] = FFT2(sum_{k<nparts} in[b*grid_stride + k*part_stride]) (full grids)
template <class C> struct FullParamsT {
	const C *in; long grid_stride, part_stride; int nparts;
	C *out;   // [b][P*P]
};
using FullParams = FullParamsT<double2>;

template <int P, class C>
__global__ void __launch_bounds__(Geo<P>::NT) k_fft_full(const FullParamsT<C> p) {
	using G = Geo<P, C>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	C *S = reinterpret_cast<C *>(smem_raw), *tw = S + G::GRID;
	init_twiddles<P>(tw);
	const long b = blockIdx.x;
	const C *in = p.in + b * p.grid_stride;
	{
		// all of the thread's elements of one partial are loaded together: the sums
		// wait for nparts memory latencies instead of nparts times the elements (one
		// cell at N = 32, 16 partials: 23 -> 10 us)
		C s[8];
#pragma unroll
		for (int e = 0; e < 8; e++) s[e] = in[threadIdx.x + e * G::NT];
#pragma unroll 2
		for (int k = 1; k < p.nparts; k++) {
			const C *ik = in + k * p.part_stride + threadIdx.x;
#pragma unroll
			for (int e = 0; e < 8; e++) s[e] = cadd(s[e], ik[e * G::NT]);
		}
#pragma unroll
		for (int e = 0; e < 8; e++) {
			const int i = threadIdx.x + e * G::NT;
			S[G::at(i / P, i % P)] = s[e];
		}
	}
	__syncthreads();
	fft2_smem<P, -1>(S, tw);
	smem_to_global<P>(p.out + b * (long)P * P, S);
}

// ---------------------------------------------------------------------------
// Sums of the I3 partials of each cell, in slot order: in[slot][len] (slots of
// a cell as in the assembly) -> out[cell][len].  The assembly has four CTAs a
// cell; with one cell and 74 partials it spent most of its time on them (N =
// 32: 390 us, 20 us behind this kernel), which spreads them over the GPU.
template <class C> struct SumSlotsT {
	const C *in; C *out; int len, nx;       // nx: slots a cell when rg.nslots = 0
	int per;                                // partials a slot (in[slot][per][len])
	TermRanges rg;
};
template <class C>
__global__ void __launch_bounds__(256) k_sum_slots(const SumSlotsT<C> p) {
	const int i = blockIdx.x * 256 + threadIdx.x;
	const long cell = blockIdx.y;
	if (i >= p.len) return;
	C s = czero<C>();
	long first = cell * p.nx, step = 1;
	int n = p.nx;
	if (p.rg.nslots > 0) {
		// after the first slot of a cell the others are the first of their cluster
		const TermRanges &g = p.rg;
		const int k0 = g.cluster_of(cell * (long)g.nterms);
		n = g.cluster_of((cell + 1) * (long)g.nterms - 1) - k0 + 1;
		const C *a = p.in + ((long)k0 * g.maxc + (cell - g.first_cell(k0))) * p.per * p.len + i;
		for (int r = 0; r < p.per; r++) s = cadd(s, a[(long)r * p.len]);
		first = (long)(k0 + 1) * g.maxc;
		step = g.maxc;
		n--;
	}
	const C *a = p.in + first * p.per * p.len + i;
	step *= (long)p.per * p.len;
	if (p.per == 1) {
#pragma unroll 8
		for (int k = 0; k < n; k++) s = cadd(s, a[k * step]);
	} else {
#pragma unroll 8
		for (int m = 0; m < 2 * n; m++) s = cadd(s, a[(m >> 1) * step + (long)(m & 1) * p.len]);   // per = 2
	}
	p.out[cell * p.len + i] = s;
}

// ---------------------------------------------------------------------------
// K6: assembly of Cc and Cd for one (cell, component j):
//   Zcc_j = Wh_h . FS_g - Wh_g . FS_h          ((g,h) = (2,3),(3,1),(1,2); upstream collision.c:232-253)
//   Zcd_j = s2 (-Wh_j + d_j0) . Q - eta2_j s1 X_j
//         + s1 (eta2_j Wh_0 . FS4_j + 2 Wh_j . FS4_0) - d_j0 2 s1 sum_c Wh_c . FS4_c   (collision.c:95-167)
//   Cc_j = s1 Extract(IFFT2(Zcc_j)), Cd_j = Extract(IFFT2(Zcd_j)) - eta2_j s1 Z_j
// (Z_j: the already extracted sums of I3Units)
// The inputs are in the working precision C; the sums and the inverse transforms
// are in FP64 in both (Asm): rounding after them spreads over the whole velocity grid
// (see zadd), before them it stays where W is.  mode 0 writes Cc and Cd; mode 1 writes
// base + dtc (Cc + Cd + CB) in FP64 with the magnetic rotation CB of `wcur`
// (upstream simulation.c:75-135).
template <class C> struct AsmParamsT {
	const C *What;                    // [cell][4][P*P]
	const C *FS;                      // [cell][3][P*P]  FFT2 of the Cc sums S_1..S_3, or null
	const C *FS4;                     // [cell][4][P*P]  FFT2 of the I4 sums, or null
	const C *Qp; int nq;              // [cell][4][nq][P*P] I2 partials, or null
	const C *Xp; int nx;              // [cell][nx][4][P*P] I3 partials, or null
	TermRanges xrg;                   // xrg.nslots > 0: Xp holds [slot][4][P*P] partials of term ranges
	bool xquad;                       // P = 128: Xp in quad order (Quad128) instead of the B layout
	const double2 *Zp; int nz;        // extracted I3 sums of the opposite shifts, [slot of Xp][nz][4][N*N], or null
	double s1, s2;
	int mode;
	double2 *out_cc, *out_cd;         // mode 0: [cell][4][N*N] (either may be null)
	const double2 *base, *wcur;       // mode 1: [cell][4][N*N]; base may be null (= 0)
	const double *B; double dtc;      // B: [cell][3], or null (no magnetic field)
	double2 *out;                     // mode 1
};
using AsmParams = AsmParamsT<double2>;

// the sum of the Z partials of a cell at point q, in slot order
template <class C>
__device__ __forceinline__ double2 zsum(const AsmParamsT<C> &p, long cell, int j, int NN, int q) {
	double2 z = czero();
	auto add = [&](long slot) {
		for (int r = 0; r < p.nz; r++) {
			z = cadd(z, p.Zp[((slot * p.nz + r) * 4 + j) * NN + q]);
		}
	};
	if (p.xrg.nslots > 0) {
		const TermRanges &g = p.xrg;
		const int k0 = g.cluster_of(cell * (long)g.nterms), k1 = g.cluster_of((cell + 1) * (long)g.nterms - 1);
		for (int k = k0; k <= k1; k++) add((long)k * g.maxc + (cell - g.first_cell(k)));
	} else {
		for (int k = 0; k < p.nx; k++) add(cell * p.nx + k);
	}
	return z;
}

// the assembly's type: FP64, but FP32 in the FP32 form at N = 8, where a step of
// launches costs 13 us more in FP64 (11 cells, J = M = 4: 153 against 133 us a
// midpoint step) and the FP32 form was never further from FP64 than term by term
template <int P, class C> struct Asm { using A = typename std::conditional<P == 16, C, double2>::type; };

template <int P, class C>
__global__ void __launch_bounds__(Geo<P>::NT) k_assemble(const AsmParamsT<C> p) {
	using A = typename Asm<P, C>::A;
	using G = Geo<P, A>;
	using R = typename CT<A>::R;
	constexpr int N = G::N, NN = N * N, PP = P * P;
	constexpr int PER = (NN + G::NT - 1) / G::NT;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	A *S = reinterpret_cast<A *>(smem_raw), *tw = S + G::GRID;
	const int j = blockIdx.x & 3;
	const long cell = blockIdx.x >> 2;
	init_twiddles<P>(tw);
	const R eta2[4] = { 2, -2, -2, -2 }, s1 = (R)p.s1, s2 = (R)p.s2;
	auto in = [](C v) { return mk<A>(v.x, v.y); };
	const C *Wh = p.What + cell * 4 * PP;
	double2 cc[PER], cd[PER];
#pragma unroll
	for (int u = 0; u < PER; u++) { cc[u] = czero(); cd[u] = czero(); }

	// --- Cc ---
	if (p.FS != nullptr && j > 0) {
		const int gi = (j % 3) + 1, hi = ((j + 1) % 3) + 1;    // j=1:(2,3) j=2:(3,1) j=3:(1,2)
		const C *FS = p.FS + cell * 3 * PP;
		for (int i = threadIdx.x; i < PP; i += G::NT) {
			S[G::at(i / P, i % P)] = csub(cmul(in(Wh[hi * PP + i]), in(FS[(gi - 1) * PP + i])),
			                              cmul(in(Wh[gi * PP + i]), in(FS[(hi - 1) * PP + i])));
		}
		__syncthreads();
		fft2_smem<P, +1>(S, tw);
#pragma unroll
		for (int u = 0; u < PER; u++) {
			const int q = threadIdx.x + u * G::NT;
			if (q < NN) {
				cc[u] = cscale(widen(S[G::at(G::pad(q / N), G::pad(q % N))]), p.s1);
			}
		}
		__syncthreads();
	}
	// --- Cd ---
	if (p.FS4 != nullptr || p.Qp != nullptr || p.Xp != nullptr) {
		// the partial sums of all the thread's elements together (as in k_fft_full)
		A zs[8];
#pragma unroll
		for (int e = 0; e < 8; e++) zs[e] = czero<A>();
		if (p.Qp != nullptr) {
#pragma unroll 1
			for (int ii = 0; ii < 4; ii++) {
				const C *Q = p.Qp + ((cell * 4 + ii) * p.nq) * (long)PP + threadIdx.x;
				A s[8];
#pragma unroll
				for (int e = 0; e < 8; e++) s[e] = czero<A>();
#pragma unroll 1
				for (int k = 0; k < p.nq; k++)
#pragma unroll
					for (int e = 0; e < 8; e++) s[e] = cadd(s[e], in(Q[(long)k * PP + e * G::NT]));
#pragma unroll
				for (int e = 0; e < 8; e++) { zs[e].x += eta2[ii] * s[e].x; zs[e].y += eta2[ii] * s[e].y; }
			}
#pragma unroll
			for (int e = 0; e < 8; e++) {
				A h = in(Wh[j * PP + threadIdx.x + e * G::NT]);
				h.x = -h.x; h.y = -h.y;
				if (j == 0) h.x += (R)1.0;
				const A v = cmul(h, zs[e]);
				zs[e].x = s2 * v.x;
				zs[e].y = s2 * v.y;
			}
		}
		if (p.Xp != nullptr) {
			A s[8];
#pragma unroll
			for (int e = 0; e < 8; e++) s[e] = czero<A>();
			auto add = [&](long slot) {
				const C *X = p.Xp + (slot * 4 + j) * (long)PP + threadIdx.x;
#pragma unroll
				for (int e = 0; e < 8; e++) s[e] = cadd(s[e], in(X[e * G::NT]));
			};
			if (p.xrg.nslots > 0) {
				const TermRanges &g = p.xrg;
				const int k0 = g.cluster_of(cell * (long)g.nterms), k1 = g.cluster_of((cell + 1) * (long)g.nterms - 1);
#pragma unroll 1
				for (int k = k0; k <= k1; k++) add((long)k * g.maxc + (cell - g.first_cell(k)));
			} else {
#pragma unroll 1
				for (int k = 0; k < p.nx; k++) add(cell * p.nx + k);
			}
#pragma unroll
			for (int e = 0; e < 8; e++) { zs[e].x -= eta2[j] * s1 * s[e].x; zs[e].y -= eta2[j] * s1 * s[e].y; }
		}
#pragma unroll
		for (int e = 0; e < 8; e++) {
			const int i = threadIdx.x + e * G::NT;
			A z = zs[e];
			if (p.FS4 != nullptr) {
				const C *F4 = p.FS4 + cell * 4 * PP;
				A v = cadd(cscale(cmul(in(Wh[i]), in(F4[j * PP + i])), eta2[j]), cscale(cmul(in(Wh[j * PP + i]), in(F4[i])), (R)2.0));
				if (j == 0) {
					A s = czero<A>();
					for (int c = 0; c < 4; c++) s = cadd(s, cmul(in(Wh[c * PP + i]), in(F4[c * PP + i])));
					v = csub(v, cscale(s, (R)2.0));
				}
				z.x += s1 * v.x; z.y += s1 * v.y;
			}
			S[G::at(i / P, i % P)] = z;
		}
		__syncthreads();
		fft2_smem<P, +1>(S, tw);
#pragma unroll
		for (int u = 0; u < PER; u++) {
			const int q = threadIdx.x + u * G::NT;
			if (q < NN) {
				cd[u] = widen(S[G::at(G::pad(q / N), G::pad(q % N))]);
				if (p.Zp != nullptr) {
					const double2 z = zsum(p, cell, j, NN, q);
					const double f = (j == 0 ? 2.0 : -2.0) * p.s1;
					cd[u].x -= f * z.x;
					cd[u].y -= f * z.y;
				}
			}
		}
	}
	// --- outputs (FP64) ---
#pragma unroll
	for (int u = 0; u < PER; u++) {
		const int q = threadIdx.x + u * G::NT;
		if (q >= NN) continue;
		const long o = (cell * 4 + j) * NN + q;
		if (p.mode == 0) {
			if (p.out_cc) p.out_cc[o] = cc[u];
			if (p.out_cd) p.out_cd[o] = cd[u];
		} else {
			const double2 *w = p.wcur + cell * 4 * NN + q;
			double2 cb = czero();          // -i [B, W] = 2 (B x w) . sigma
			if (p.B != nullptr) {        // null B: no magnetic field
				const double *B = p.B + cell * 3;
				if (j == 1) cb = make_double2(2 * (B[1] * w[3 * NN].x - B[2] * w[2 * NN].x), 2 * (B[1] * w[3 * NN].y - B[2] * w[2 * NN].y));
				if (j == 2) cb = make_double2(2 * (B[2] * w[1 * NN].x - B[0] * w[3 * NN].x), 2 * (B[2] * w[1 * NN].y - B[0] * w[3 * NN].y));
				if (j == 3) cb = make_double2(2 * (B[0] * w[2 * NN].x - B[1] * w[1 * NN].x), 2 * (B[0] * w[2 * NN].y - B[1] * w[1 * NN].y));
			}
			const double2 b = p.base ? p.base[o] : czero();      // null base: the right-hand side itself
			p.out[o] = make_double2(b.x + p.dtc * ((cc[u].x + cd[u].x) + cb.x), b.y + p.dtc * ((cc[u].y + cd[u].y) + cb.y));
		}
	}
}

// ---------------------------------------------------------------------------
// K7: velocity space -> Fourier space, one CTA per real N x N component:
//   FFT2 / N^2 with the Hermitian completion of upstream simulation.c:224-261
template <int N>
__global__ void __launch_bounds__(Len<N>::T * N) k_to_fourier(const double *__restrict__ Wv, double2 *__restrict__ Wf) {
	constexpr int T = Len<N>::T, LD = N + 1;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double2 *S = reinterpret_cast<double2 *>(smem_raw), *tw = S + N * LD;
	init_twiddles<N>(tw);
	__syncthreads();
	const long b = blockIdx.x;
	const double *in = Wv + b * N * N;
	const int line = threadIdx.x / T, tau = threadIdx.x % T;
	double2 x[8];
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = make_double2(in[line * N + tau + T * r], 0.0);
	fft1d<N, -1>(x, tau, S + line * LD, 1, tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[line * LD + Len<N>::out_pos(tau, e)] = x[e];
	__syncthreads();
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = S[(tau + T * r) * LD + line];
	fft1d<N, -1>(x, tau, S + line, LD, tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[Len<N>::out_pos(tau, e) * LD + line] = x[e];
	__syncthreads();
	const double scale = 1.0 / (N * N);
	double2 *out = Wf + b * N * N;
	for (int i = threadIdx.x; i < N * N; i += T * N) {
		const int l = i / N, k = i % N;
		if (k <= N / 2) {
			const double2 v = S[l * LD + k];
			out[i] = make_double2(v.x * scale, v.y * scale);
		} else {
			const int lc = (N - l) % N, kc = N - k;
			const double2 v = S[lc * LD + kc];
			out[i] = make_double2(v.x * scale, -(v.y * scale));
		}
	}
}

// K8: Fourier space -> velocity space: backward FFT2, real part (simulation.c:270-283)
template <int N>
__global__ void __launch_bounds__(Len<N>::T * N) k_from_fourier(const double2 *__restrict__ Wf, double *__restrict__ Wv) {
	constexpr int T = Len<N>::T, LD = N + 1;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double2 *S = reinterpret_cast<double2 *>(smem_raw), *tw = S + N * LD;
	init_twiddles<N>(tw);
	__syncthreads();
	const long b = blockIdx.x;
	const double2 *in = Wf + b * N * N;
	const int line = threadIdx.x / T, tau = threadIdx.x % T;
	double2 x[8];
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = in[line * N + tau + T * r];
	fft1d<N, +1>(x, tau, S + line * LD, 1, tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[line * LD + Len<N>::out_pos(tau, e)] = x[e];
	__syncthreads();
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = S[(tau + T * r) * LD + line];
	fft1d<N, +1>(x, tau, S + line, LD, tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[Len<N>::out_pos(tau, e) * LD + line] = x[e];
	__syncthreads();
	double *out = Wv + b * N * N;
	for (int i = threadIdx.x; i < N * N; i += T * N) out[i] = S[(i / N) * LD + (i % N)].x;
}

// K9: generic 2-D transform of n0 x n1 = L x L complex grids (FFTW-API plans).
// mode 0: c2c (in complex), mode 1: r2c (in real, out n0 x (L/2+1))
template <int L, int DIR>
__global__ void __launch_bounds__(Len<L>::T * L) k_fft2_generic(const void *__restrict__ in, double2 *__restrict__ out, int r2c) {
	constexpr int T = Len<L>::T, LD = L + 1;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	double2 *S = reinterpret_cast<double2 *>(smem_raw), *tw = S + L * LD;
	init_twiddles<L>(tw);
	__syncthreads();
	const int line = threadIdx.x / T, tau = threadIdx.x % T;
	double2 x[8];
#pragma unroll
	for (int r = 0; r < 8; r++) {
		const int i = line * L + tau + T * r;
		x[r] = r2c ? make_double2(((const double *)in)[i], 0.0) : ((const double2 *)in)[i];
	}
	fft1d<L, DIR>(x, tau, S + line * LD, 1, tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[line * LD + Len<L>::out_pos(tau, e)] = x[e];
	__syncthreads();
#pragma unroll
	for (int r = 0; r < 8; r++) x[r] = S[(tau + T * r) * LD + line];
	fft1d<L, DIR>(x, tau, S + line, LD, tw);
#pragma unroll
	for (int e = 0; e < 8; e++) S[Len<L>::out_pos(tau, e) * LD + line] = x[e];
	__syncthreads();
	if (r2c) {
		constexpr int H = L / 2 + 1;
		for (int i = threadIdx.x; i < L * H; i += T * L) out[i] = S[(i / H) * LD + (i % H)];
	} else {
		for (int i = threadIdx.x; i < L * L; i += T * L) out[i] = S[(i / L) * LD + (i % L)];
	}
}

}  // namespace qb
