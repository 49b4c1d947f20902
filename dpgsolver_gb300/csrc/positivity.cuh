// Pieces of the positivity limiter shared by its own kernels (positivity.cu) and the fused stage kernel of the
// tensor-product meshes (kernels_tp_stage.cu).
#pragma once

#include <cmath>

#include "dpg_gpu_internal.cuh"

namespace dpg {
namespace pos {

// FP32 value of a double by integer operations only, truncating the mantissa (relative error < 2^-23): a conversion
// instruction would run on GB300's FP64 pipe, which bounds the screen's throughput otherwise.  Magnitudes below
// 2^-126 become 0 (absolute error far below EPS_PHYS), above the FP32 range, infinities and NaN become infinity (the
// screen then flags the volume).
__device__ __forceinline__ float trunc_to_float(double x)
{
	const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
	const int t = (int)(hi & 0x7fffffffu) - ((1023 - 127) << 20);   // exponent rebiased, mantissa's top 20 bits
	unsigned bits = __funnelshift_l(lo, (unsigned)t, 3);            // (t << 3) | (lo >> 29)
	bits = t < (1 << 20) ? 0u : t >= (255 << 20) ? 0x7f800000u : bits;
	return __uint_as_float(bits | (hi & 0x80000000u));
}

// convert_variables 'c' -> 'p' / 'p' -> 'c' of one coefficient (the reference's operation order)
template <int D>
__device__ void cons_to_prim(double* w)
{
	const double rho_inv = 1.0 / w[0];
	double rho2V2 = 0.0;
#pragma unroll
	for (int a = 0; a < D; ++a) {
		rho2V2 += w[1 + a] * w[1 + a];
		w[1 + a] = w[1 + a] * rho_inv;
	}
	w[D + 1] = 0.4 * (w[D + 1] - 0.5 * rho2V2 * rho_inv);
}
template <int D>
__device__ void prim_to_cons(double* w)
{
	double V2 = 0.0;
#pragma unroll
	for (int a = 0; a < D; ++a) {
		V2 += w[1 + a] * w[1 + a];
		w[1 + a] = w[0] * w[1 + a];
	}
	w[D + 1] = w[D + 1] / 0.4 + 0.5 * w[0] * V2;
}

// the reference's average_T / minimum_T over n coefficients (sequential sum)
__device__ inline double avg_seq(const double* x, int n)
{
	double s = 0.0;
#pragma unroll 1
	for (int i = 0; i < n; ++i) s += x[i];
	return s / (double)n;
}
__device__ inline double min_seq(const double* x, int n)
{
	double m = 1.7976931348623157e308;
#pragma unroll 1
	for (int i = 0; i < n; ++i)
		if (x[i] < m) m = x[i];
	return m;
}

// The serial part of enforce_positivity_highorder on one volume's primitive Bezier coefficients w [NV][NS]; false
// where an average is below EPS_PHYS (the reference stops there).
template <int D, int NS>
__device__ bool limit_volume(double* w)
{
	constexpr int NV = D + 2;
#pragma unroll 1
	for (int vr = 0; vr < NV; vr += NV - 1) {
		const double avg = avg_seq(w + vr * NS, NS);
		if (!(avg >= DPG_EPS_PHYS)) return false;
		const double mn = min_seq(w + vr * NS, NS);
		if (mn < DPG_EPS_PHYS) {
			const double p_ho = fmax(0.0, fmin(1.0, (avg - DPG_EPS_PHYS) / (avg - mn)));
#pragma unroll 1
			for (int v = 0; v < NV; ++v) {
				double* x = w + v * NS;
				double a = avg_seq(x, NS);
				if ((v == 0 || v == NV - 1) && a < DPG_EPS_PHYS) a = DPG_EPS_PHYS;
#pragma unroll 1
				for (int i = 0; i < NS; ++i) x[i] = p_ho * x[i] + (1 - p_ho) * a;
			}
		}
	}
	return true;
}

// 1D operators of the limiter as kernel parameters (read from the constant bank at compile-time indices)
struct PosOps {
	float ai32[25];    // bez1_inv in FP32 (the screen)
	float rs;          // bound of bez1_inv's absolute row sums (the screen's error bound)
	double a64[25];    // bez1: Bezier -> solution coefficients
	double ai64[25];   // bez1_inv: solution -> Bezier coefficients
};

// one 1D operator on n1 values (row-major A, output i = sum_k A[i][k] x[k])
template <int N1, typename T, typename A>
__device__ __forceinline__ void apply1(const A& a, const T (&x)[N1], T (&y)[N1])
{
#pragma unroll
	for (int i = 0; i < N1; ++i) {
		T acc = 0;
#pragma unroll
		for (int k = 0; k < N1; ++k) acc += (T)a[i * N1 + k] * x[k];
		y[i] = acc;
	}
}

// Host: the operators of a context with n1 points per direction.
template <int N1>
inline PosOps pos_ops(const dpg_gpu_ctx* c)
{
	PosOps ops{};
	for (int i = 0; i < N1 * N1; ++i) {
		ops.ai32[i] = (float)c->bez1_host[i + 25];
		ops.a64[i] = c->bez1_host[i];
		ops.ai64[i] = c->bez1_host[i + 25];
	}
	double rs = 0.0;
	for (int i = 0; i < N1; ++i) {
		double r = 0.0;
		for (int k = 0; k < N1; ++k) r += std::fabs(c->bez1_host[25 + i * N1 + k]);
		rs = r > rs ? r : rs;
	}
	ops.rs = (float)(rs * (1.0 + 1e-6));
	return ops;
}

} // namespace pos
} // namespace dpg
