// qb_radix.cuh — register DFTs of 2, 3, 4, 6, 8, 12 and 16 points (sm_100a),
// generic over the complex type: the stages of the any-N engine.
#pragma once
#include "qb_fft.cuh"

namespace qb {

template <int DIR, class C> __device__ __forceinline__ void dft3(C &x0, C &x1, C &x2) {
	using R = typename CT<C>::R;
	const C t1 = cadd(x1, x2);
	const C m = csub(x0, cscale(t1, (R)0.5));
	const C d = mul_i<DIR>(cscale(csub(x1, x2), (R)0.86602540378443864676));   // sin(2 pi / 3)
	x0 = cadd(x0, t1);
	x1 = cadd(m, d);
	x2 = csub(m, d);
}

// cos and sin of 2 pi m / R for R = 6, 12, 16 (the twiddles of the composite
// register DFTs; folded to constants when m is known at compile time)
__host__ __device__ constexpr double cos_r(int R, int m) {
	constexpr double h = 0.5, c3 = 0.86602540378443864676, c8 = 0.70710678118654752440;
	constexpr double a = 0.92387953251128675613, b = 0.38268343236508977173;
	if (R == 16) {
		const double t[16] = { 1, a, c8, b, 0, -b, -c8, -a, -1, -a, -c8, -b, 0, b, c8, a };
		return t[m];
	}
	if (R == 12) {
		const double t[12] = { 1, c3, h, 0, -h, -c3, -1, -c3, -h, 0, h, c3 };
		return t[m];
	}
	const double t[6] = { 1, h, -h, -1, -h, h };
	return t[m];
}
__host__ __device__ constexpr double sin_r(int R, int m) {
	if (R == 6) {
		constexpr double c3 = 0.86602540378443864676;
		const double t[6] = { 0, c3, c3, 0, -c3, -c3 };
		return t[m];
	}
	return cos_r(R, (m + 3 * R / 4) % R);     // sin x = cos(x - pi/2); R = 12, 16 are multiples of 4
}

template <int R1, int R2, int DIR, class C> __device__ __forceinline__ void dft_ct(C (&x)[R1 * R2]);

template <int RAD, int DIR, class C> __device__ __forceinline__ void dft_r(C (&v)[RAD]) {
	if constexpr (RAD == 16) dft_ct<4, 4, DIR>(v);
	else if constexpr (RAD == 12) dft_ct<4, 3, DIR>(v);
	else if constexpr (RAD == 8) dft8<DIR>(v);
	else if constexpr (RAD == 6) dft_ct<2, 3, DIR>(v);
	else if constexpr (RAD == 4) dft4<DIR>(v[0], v[1], v[2], v[3]);
	else if constexpr (RAD == 3) dft3<DIR>(v[0], v[1], v[2]);
	else dft2(v[0], v[1]);
}

// an R1 R2-point DFT in registers, in place: R2 DFTs of R1 points (stride
// R2), twiddles w_R^(n2 k1), R1 DFTs of R2 points.  Input in natural order;
// output frequency k1 + R1 k2 lands in slot k1 R2 + k2 (freq_of gives the
// frequency of a slot), so no second array of R values is live
template <int R1, int R2, int DIR, class C> __device__ __forceinline__ void dft_ct(C (&x)[R1 * R2]) {
	using R = typename CT<C>::R;
	constexpr int RR = R1 * R2;
#pragma unroll
	for (int n2 = 0; n2 < R2; n2++) {
		C v[R1];
#pragma unroll
		for (int n1 = 0; n1 < R1; n1++) v[n1] = x[n2 + R2 * n1];
		dft_r<R1, DIR>(v);
#pragma unroll
		for (int k1 = 0; k1 < R1; k1++) {
			const int m = (n2 * k1) % RR;
			if (m == 0) {
				x[n2 + R2 * k1] = v[k1];
			} else {
				C w;
				w.x = (R)cos_r(RR, m);
				w.y = (R)(DIR < 0 ? -sin_r(RR, m) : sin_r(RR, m));
				x[n2 + R2 * k1] = cmul(v[k1], w);
			}
		}
	}
#pragma unroll
	for (int k1 = 0; k1 < R1; k1++) {
		C v[R2];
#pragma unroll
		for (int n2 = 0; n2 < R2; n2++) v[n2] = x[k1 * R2 + n2];
		dft_r<R2, DIR>(v);
#pragma unroll
		for (int k2 = 0; k2 < R2; k2++) x[k1 * R2 + k2] = v[k2];
	}
}

// frequency held in slot s after dft_r<RAD> (the composite radices leave
// their output permuted; 2, 3, 4, 8 and the sub-DFTs are in natural order)
template <int RAD> __host__ __device__ constexpr int freq_of(int s) {
	if (RAD == 16) return s / 4 + 4 * (s % 4);
	if (RAD == 12) return s / 3 + 4 * (s % 3);
	if (RAD == 6) return s / 3 + 2 * (s % 3);
	return s;
}

}  // namespace qb
