// qb_radix.cuh — register DFTs of 2, 3, 4, 6, 8, 12 and 16 points (sm_100a),
// generic over the complex type: the stages of the any-N engine.
#pragma once
#include "qb_fft.cuh"

namespace qb {

// The FP32 transforms multiply by their constants without the mean error of a
// rounded constant. A rounded c = sqrt(1/2) or sqrt(3/4) scales everything it
// touches by 1 + (float)c / c, and the gains of a few transforms in a row do not cancel
// between the gain and the loss sums of the operator: with rounded constants they
// made up most of its production of mass (1.6e-7 of the gain sums at P = 96, with these
// 2.6e-8; the pairs (cos, sin) rounded to modulus 1, root16 and unit_root, are part of it).
__host__ __device__ constexpr float const_lo(double c) { return (float)(c - (double)(float)c); }
__device__ __forceinline__ double2 mul_const(double2 a, double c) { return cscale(a, c); }
__device__ __forceinline__ float2 mul_const(float2 a, double c) {
	return make_float2(fmaf(a.x, const_lo(c), a.x * (float)c), fmaf(a.y, const_lo(c), a.y * (float)c));
}

template <int DIR, class C> __device__ __forceinline__ void dft3(C &x0, C &x1, C &x2) {
	using R = typename CT<C>::R;
	const C t1 = cadd(x1, x2);
	const C m = csub(x0, cscale(t1, (R)0.5));
	const C d = mul_i<DIR>(mul_const(csub(x1, x2), 0.86602540378443864676));   // sin(2 pi / 3)
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

// v w_R^m, w_R = exp(DIR 2 pi i / R), m known at compile time
template <int RR, int DIR> __device__ __forceinline__ double2 mul_root(double2 v, int m) {
	return cmul(v, make_double2(cos_r(RR, m), DIR < 0 ? -sin_r(RR, m) : sin_r(RR, m)));
}
// cos(pi / 8) and sin(pi / 8) as the neighbouring FP32 values with |w|^2 - 1 nearest 0
__host__ __device__ constexpr float root16(double c) {
	const double m = c < 0 ? -c : c;
	const float r = m > 0.9 && m < 0.93 ? 0x1.d906bcp-1f : m > 0.38 && m < 0.39 ? 0x1.87de2ep-2f : (float)m;
	return c < 0 ? -r : r;
}
template <int RR, int DIR> __device__ __forceinline__ float2 mul_root(float2 v, int m) {
	if (4 * m == RR) return mul_i<DIR>(v);
	if (8 * m == RR || 8 * m == 3 * RR) {            // (+-1 + DIR i) sqrt(1/2)
		const float s = 8 * m == RR ? 1.0f : -1.0f;
		return mul_const(DIR < 0 ? make_float2(s * v.x + v.y, s * v.y - v.x) : make_float2(s * v.x - v.y, s * v.y + v.x), 0.70710678118654752440);
	}
	const double c = cos_r(RR, m), i = DIR < 0 ? -sin_r(RR, m) : sin_r(RR, m);
	if (RR == 16) return cmul(v, make_float2(root16(c), root16(i)));
	float2 z = cmul(v, make_float2((float)c, (float)i));
	z.x = fmaf(v.x, const_lo(c), fmaf(-v.y, const_lo(i), z.x));
	z.y = fmaf(v.x, const_lo(i), fmaf(v.y, const_lo(c), z.y));
	return z;
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
			x[n2 + R2 * k1] = m == 0 ? v[k1] : mul_root<RR, DIR>(v[k1], m);
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
