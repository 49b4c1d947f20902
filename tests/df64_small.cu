// GPU check of the double-float square root and reciprocal square root (df64.cuh) on small operands: magnitudes from the
// smallest FP32 subnormal to 2^-90, the smallest normal number and its neighbours, and zero; and of the reciprocal where
// the operand or the result is a subnormal number.  Built and run by
// tests/test_gpu_split_rest.py; prints one line per check and exits 1 if any bound is missed.
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <vector>

#include "df64.cuh"

using dpg::df::df64;

__global__ void k_rcp(int n, const float2* x, float2* r)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const df64 y = dpg::df::rcp(dpg::df::from2(x[i]));
	r[i] = make_float2(y.hi, y.lo);
}

__global__ void k_roots(int n, const float2* x, double* s, float2* r)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const df64 a = dpg::df::from2(x[i]);
	s[i] = dpg::df::to_double(dpg::df::sqrt(a));
	const df64 y = dpg::df::rsqrt(a);
	r[i] = make_float2(y.hi, y.lo);
}

int main()
{
	std::vector<float2> x;
	uint64_t s = 99;
	auto u = [&] { s = s * 6364136223846793005ull + 1442695040888963407ull; return (double)(s >> 11) * (1.0 / 9007199254740992.0); };
	for (int e = -149; e <= -90; ++e)
		for (int k = 0; k < 64; ++k) x.push_back(dpg::df::split_double(std::ldexp(1.0 + (k ? u() : 0.0), e)));
	for (double v : {std::ldexp(1.0, -126), std::ldexp(1.0, -126) - std::ldexp(1.0, -149), std::ldexp(1.0, -126) + std::ldexp(1.0, -149)})
		x.push_back(dpg::df::split_double(v));
	const int n = (int)x.size();
	x.push_back(make_float2(0.f, 0.f));
	float2 *dx, *dr;
	double* ds;
	cudaMalloc(&dx, sizeof(float2) * (n + 1)); cudaMalloc(&dr, sizeof(float2) * (n + 1)); cudaMalloc(&ds, sizeof(double) * (n + 1));
	cudaMemcpy(dx, x.data(), sizeof(float2) * (n + 1), cudaMemcpyHostToDevice);
	k_roots<<<(n + 128) / 128, 128>>>(n + 1, dx, ds, dr);
	std::vector<double> rs(n + 1);
	std::vector<float2> rr(n + 1);
	const cudaError_t e = cudaDeviceSynchronize();
	cudaMemcpy(rs.data(), ds, sizeof(double) * (n + 1), cudaMemcpyDeviceToHost);
	cudaMemcpy(rr.data(), dr, sizeof(float2) * (n + 1), cudaMemcpyDeviceToHost);
	if (e != cudaSuccess) { std::printf("cuda error %s\n", cudaGetErrorString(e)); return 1; }
	double e_s = 0.0, e_r = 0.0;
	for (int i = 0; i < n; ++i) {
		const double a = (double)x[i].x + (double)x[i].y, q = std::sqrt(a);   // exact sum
		const double ds_ = std::fabs(rs[i] / q - 1.0), dr_ = std::fabs(((double)rr[i].x + (double)rr[i].y) * q - 1.0);
		e_s = ds_ <= e_s ? e_s : ds_;   // keeps a NaN
		e_r = dr_ <= e_r ? e_r : dr_;
	}
	// reciprocals: 1 / y for y in [2^-127, 2^-126), and for y in [2^126, 2^128), where 1 / y has 21 bits or more
	std::vector<float2> y;
	for (int ex : {-127, 126, 127})
		for (int k = 0; k < 512; ++k) y.push_back(dpg::df::split_double(std::ldexp(1.0 + 0.999 * u(), ex)));
	const int m = (int)y.size();
	cudaMemcpy(dx, y.data(), sizeof(float2) * m, cudaMemcpyHostToDevice);
	k_rcp<<<(m + 127) / 128, 128>>>(m, dx, dr);
	const cudaError_t e2 = cudaDeviceSynchronize();
	cudaMemcpy(rr.data(), dr, sizeof(float2) * m, cudaMemcpyDeviceToHost);
	if (e2 != cudaSuccess) { std::printf("cuda error %s\n", cudaGetErrorString(e2)); return 1; }
	double e_c[2] = {0.0, 0.0};
	for (int i = 0; i < m; ++i) {
		const double d = std::fabs(((double)rr[i].x + (double)rr[i].y) * ((double)y[i].x + (double)y[i].y) - 1.0);
		double& w = e_c[i >= 512];
		w = d <= w ? w : d;
	}
	int bad = 0;
	auto report = [&](const char* name, double err, double bound) {
		std::printf("check %-28s max_err %.3e bound %.1e %s\n", name, err, bound, err <= bound ? "ok" : "FAIL");
		bad += !(err <= bound);
	};
	report("sqrt (relative)", e_s, std::ldexp(1.0, -44));
	report("rsqrt (relative)", e_r, std::ldexp(1.0, -44));
	report("rcp of a subnormal (relative)", e_c[0], std::ldexp(1.0, -44));
	report("rcp to a subnormal (relative)", e_c[1], std::ldexp(1.0, -20));   // 2 units of 2^-149 in 2^-128
	report("sqrt(0)", std::fabs(rs[n]), 0.0);
	std::printf("%s\n", bad ? "FAILED" : "all checks passed");
	return bad ? 1 : 0;
}
