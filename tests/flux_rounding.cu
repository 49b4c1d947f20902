// Rounding of the numerical fluxes on the GPU: the forms that the large meshes take (numflux_.._rs, flux.cuh) against the plain
// ones, both measured against extended precision on the host (long double: 64 or 113 bits), rms per component over random
// states by regime.  Built and run by tests/test_gpu_flux_rounding.py; prints one line per check and exits 1 if an _rs form's
// rms error is larger than 1.15 times the plain form's (the sampling error of an rms over these states is 0.5 %).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "flux.cuh"

namespace {

typedef long double real;

struct Rng {   // 64-bit LCG (Knuth's MMIX constants), top 53 bits as a uniform double in [0, 1)
	uint64_t s;
	double in(double a, double b)
	{
		s = s * 6364136223846793005ull + 1442695040888963407ull;
		return a + (b - a) * ((double)(s >> 11) * (1.0 / 9007199254740992.0));
	}
};

template <int D>
void exact_flux(bool roe, const double* wl, const double* wr, const double* nd, real* F)
{
	const real G = DPG_GAMMA_D, GM = DPG_GM1_D;
	real WL[5], WR[5], n[3], uL[3], uR[3], V2L = 0, V2R = 0, VnL = 0, VnR = 0, fL[5], fR[5];
	for (int k = 0; k < D + 2; ++k) { WL[k] = wl[k]; WR[k] = wr[k]; }
	for (int a = 0; a < D; ++a) {
		n[a] = nd[a];
		uL[a] = WL[1 + a] / WL[0]; uR[a] = WR[1 + a] / WR[0];
		V2L += uL[a] * uL[a]; V2R += uR[a] * uR[a];
		VnL += n[a] * uL[a];  VnR += n[a] * uR[a];
	}
	const real pL = GM * (WL[D + 1] - 0.5L * WL[0] * V2L), pR = GM * (WR[D + 1] - 0.5L * WR[0] * V2R);
	fL[0] = WL[0] * VnL; fR[0] = WR[0] * VnR;
	for (int a = 0; a < D; ++a) { fL[1 + a] = WL[1 + a] * VnL + n[a] * pL; fR[1 + a] = WR[1 + a] * VnR + n[a] * pR; }
	fL[D + 1] = (WL[D + 1] + pL) * VnL; fR[D + 1] = (WR[D + 1] + pR) * VnR;
	if (!roe) {
		const real a = std::sqrt(V2L) + std::sqrt(G * pL / WL[0]), b = std::sqrt(V2R) + std::sqrt(G * pR / WR[0]), m = a > b ? a : b;
		for (int k = 0; k < D + 2; ++k) F[k] = 0.5L * (fL[k] + fR[k] + m * (WL[k] - WR[k]));
		return;
	}
	const real r = std::sqrt(WR[0] / WL[0]), rho = r * WL[0];
	real u[3], Vn = 0, V2 = 0;
	for (int a = 0; a < D; ++a) { u[a] = (r * uR[a] + uL[a]) / (r + 1); Vn += n[a] * u[a]; V2 += u[a] * u[a]; }
	const real HL = (WL[D + 1] + pL) / WL[0], HR = (WR[D + 1] + pR) / WR[0], H = (r * HR + HL) / (r + 1);
	const real c2 = GM * (H - 0.5L * V2), c = std::sqrt(c2);
	const real l1 = std::fmin(std::fabs(VnL - c), std::fabs(Vn - c)), l5 = std::fmax(std::fabs(VnR + c), std::fabs(Vn + c)), l2 = std::fabs(Vn);
	const real dp = pR - pL, dVn = VnR - VnL, lc1 = 0.5L * (l5 + l1) - l2, lc2 = 0.5L * (l5 - l1);
	const real d1 = lc1 * dp / c2 + lc2 * rho * dVn / c, d2 = lc1 * rho * dVn + lc2 * dp / c;
	F[0] = 0.5L * (fL[0] + fR[0] - l2 * (WR[0] - WL[0]) - d1);
	for (int a = 0; a < D; ++a) F[1 + a] = 0.5L * (fL[1 + a] + fR[1 + a] - l2 * (WR[1 + a] - WL[1 + a]) - d1 * u[a] - d2 * n[a]);
	F[D + 1] = 0.5L * (fL[D + 1] + fR[D + 1] - l2 * (WR[D + 1] - WL[D + 1]) - d1 * H - d2 * Vn);
}

template <int D>
__global__ void k_flux(int n, bool roe, bool rs, const double* L, const double* R, const double* N, double* F)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	constexpr int V = D + 2;
	double wl[V], wr[V], nn[D], f[V];
	for (int v = 0; v < V; ++v) { wl[v] = L[V * i + v]; wr[v] = R[V * i + v]; }
	for (int a = 0; a < D; ++a) nn[a] = N[D * i + a];
	if (roe && rs) dpg::numflux_roe_pike_rs<D>(wl, wr, nn, 0.5, f);
	else if (roe) dpg::numflux_roe_pike<D>(wl, wr, nn, f);
	else if (rs) dpg::numflux_lax_friedrichs_rs<D>(wl, wr, nn, 0.5, f);
	else dpg::numflux_lax_friedrichs<D>(wl, wr, nn, f);
	for (int v = 0; v < V; ++v) F[V * i + v] = f[v];
}

// speed and relative jump across the face: smooth flows, slow ones, uniform ones, supersonic ones, strong jumps
const struct { const char* name; double vel, jump; } kRegimes[] = {
	{"smooth", 0.6, 1e-3}, {"slow", 1e-3, 1e-5}, {"uniform", 0.6, 0.0}, {"uniform, slow", 1e-6, 0.0}, {"supersonic", 4.0, 1e-3}, {"jumps", 0.6, 0.5}};

template <int D>
int checks(bool roe)
{
	constexpr int V = D + 2, n = 1 << 15;
	double *dL, *dR, *dN, *dF;
	cudaMalloc(&dL, sizeof(double) * V * n); cudaMalloc(&dR, sizeof(double) * V * n);
	cudaMalloc(&dN, sizeof(double) * D * n); cudaMalloc(&dF, sizeof(double) * V * n);
	int bad = 0;
	for (const auto& g : kRegimes) {
		Rng r{77};
		std::vector<double> L(V * n), R(V * n), N(D * n), F(V * n);
		std::vector<real> E(V * n);
		for (int i = 0; i < n; ++i) {
			auto put = [&](double* w, double rho, const double* u, double p) {
				double V2 = 0.0;
				w[0] = rho;
				for (int a = 0; a < D; ++a) { w[1 + a] = rho * u[a]; V2 += u[a] * u[a]; }
				w[D + 1] = p / 0.4 + 0.5 * rho * V2;
			};
			const double rho = r.in(0.7, 1.4), p = r.in(0.7, 1.4);
			double u[3], s = 0.0;
			for (int a = 0; a < D; ++a) u[a] = r.in(-g.vel, g.vel);
			put(&L[V * i], rho, u, p);
			if (g.jump == 0.0) {
				for (int v = 0; v < V; ++v) R[V * i + v] = L[V * i + v];
			} else {
				for (int a = 0; a < D; ++a) u[a] += g.vel * g.jump * r.in(-1.0, 1.0);
				put(&R[V * i], rho * (1.0 + g.jump * r.in(-1.0, 1.0)), u, p * (1.0 + g.jump * r.in(-1.0, 1.0)));
			}
			for (int a = 0; a < D; ++a) { N[D * i + a] = r.in(-1.0, 1.0); s += N[D * i + a] * N[D * i + a]; }
			for (int a = 0; a < D; ++a) N[D * i + a] /= std::sqrt(s);
			exact_flux<D>(roe, &L[V * i], &R[V * i], &N[D * i], &E[V * i]);
		}
		cudaMemcpy(dL, L.data(), sizeof(double) * V * n, cudaMemcpyHostToDevice);
		cudaMemcpy(dR, R.data(), sizeof(double) * V * n, cudaMemcpyHostToDevice);
		cudaMemcpy(dN, N.data(), sizeof(double) * D * n, cudaMemcpyHostToDevice);
		double rms[2][3] = {};
		for (int rs = 0; rs < 2; ++rs) {
			k_flux<D><<<n / 128, 128>>>(n, roe, rs != 0, dL, dR, dN, dF);
			if (cudaMemcpy(F.data(), dF, sizeof(double) * V * n, cudaMemcpyDeviceToHost) != cudaSuccess) { std::printf("cuda error\n"); return 1; }
			for (int i = 0; i < V * n; ++i) {
				const int v = i % V;
				const double e = (double)((real)F[i] - E[i]) * 9007199254740992.0;
				rms[rs][v == 0 ? 0 : v <= D ? 1 : 2] += e * e / n / (v == 0 || v > D ? 1 : D);
			}
		}
		const char* what[3] = {"mass", "momentum", "energy"};
		for (int k = 0; k < 3; ++k) {
			const double a = std::sqrt(rms[0][k]), b = std::sqrt(rms[1][k]);
			const bool ok = b <= 1.15 * a;
			std::printf("check %s %dD %-14s %-8s rms / 2^-53: plain %.3g rs %.3g %s\n", roe ? "Roe-Pike" : "Lax-Friedrichs", D, g.name, what[k], a, b, ok ? "ok" : "FAIL");
			bad += !ok;
		}
	}
	cudaFree(dL); cudaFree(dR); cudaFree(dN); cudaFree(dF);
	return bad;
}

} // namespace

int main()
{
	const int bad = checks<3>(true) + checks<3>(false) + checks<2>(true) + checks<2>(false);
	std::printf("%s\n", bad ? "FAILED" : "all checks passed");
	return bad ? 1 : 0;
}
