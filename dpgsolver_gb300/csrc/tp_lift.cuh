// Last kernel of the tensor-product residual: face fluxes, mass matrix, back to the solution nodes, SSP-RK3 stage.
#pragma once

#include "tp_ops.cuh"

namespace dpg {
namespace tp {

template <int D, int NV, int N1>
inline size_t smem_lift(int E)
{
	const size_t N = ipow(N1, D), NF = ipow(N1, D - 1);
	return sizeof(Ops<N1>) + sizeof(double) * E * NV * (2 * N + 2 * D * NF) + 8;
}

// r (in: the weak divergence of this thread's node, collocated) += the lifted face fluxes, times 1 / detJ, at the solution
// nodes.  b0, b1: [E][NV][N]; sF: [E][2 D][NV][NF].
// OWN: the face fluxes are formed here from the traces, the same value on both sides, instead of read from nnf.
template <int D, int NV, int N1, bool OWN>
__device__ __forceinline__ void lift_body(const Ops<N1>* so, double* b0, double* b1, double* sF, int e0, int ne,
                                          const TpGeo& g, const double* nnf, const TpFaces& fa, double ji, double (&r)[NV])
{
	constexpr int N = ipow(N1, D), NF = ipow(N1, D - 1);
	const int e = threadIdx.x / N, i = threadIdx.x - e * N;
	const bool live = e < ne;
	// face fluxes in the element's node order, + outward
	for (int o = threadIdx.x; o < ne * 2 * D * NF; o += blockDim.x) {
		const int ee = o / (2 * D * NF), k = o - ee * 2 * D * NF, lf = k / NF, q = k - lf * NF;
		const int vf = g.vol_face[(size_t)(e0 + ee) * 2 * D + lf];
		const int f = vf >> 1, side = vf & 1;
		const int qs = side ? g.nc_inv[(size_t)f * NF + q] : q;
		const long long flip = side ? 0ll : (long long)0x8000000000000000ull;   // - outward flux of this element
		double y[NV];
		if constexpr (OWN) {
			const size_t t = (size_t)f * NF + qs;
			const int qr = side ? q : fa.nc[t];
			double WL[NV], WR[NV], n[D];
#pragma unroll
			for (int w = 0; w < NV; ++w) {
				WL[w] = fa.trace[((size_t)2 * f * NV + w) * NF + qs];
				WR[w] = fa.trace[((size_t)(2 * f + 1) * NV + w) * NF + qr];
			}
#pragma unroll
			for (int x = 0; x < D; ++x) n[x] = fa.nrm[t * D + x];
			if constexpr (NV == D + 2) {
				if (fa.num_flux == DPG_NUM_FLUX_ROE_PIKE) numflux_roe_pike_rs<D>(WL, WR, n, 0.5 * fa.jf[t], y);
				else                                      numflux_lax_friedrichs_rs<D>(WL, WR, n, 0.5 * fa.jf[t], y);
			} else {
				y[0] = numflux_upwind<D>(fa.b, WL[0], WR[0], n) * fa.jf[t];
			}
		} else {
#pragma unroll
			for (int w = 0; w < NV; ++w) y[w] = nnf[((size_t)f * NV + w) * NF + qs];
		}
#pragma unroll
		for (int w = 0; w < NV; ++w)
			sF[((size_t)(ee * 2 * D + lf) * NV + w) * NF + q] = __longlong_as_double(__double_as_longlong(y[w]) ^ flip);
	}
	__syncthreads();
	if (live) {
		auto face = [&](auto tag) {
			constexpr int A = decltype(tag)::value;
			const int ia = node_along<A, N1>(i), q = face_node<A, N1>(i);
			const double wm = so->wm[ia], wp = so->wp[ia];
			const double* F = sF + (size_t)(e * 2 * D + 2 * A) * NV * NF + q;
#pragma unroll
			for (int w = 0; w < NV; ++w) r[w] = fma(wp, F[(NV + w) * NF], fma(wm, F[w * NF], r[w]));
		};
		face(std::integral_constant<int, 0>{});
		face(std::integral_constant<int, 1>{});
		if constexpr (D == 3) face(std::integral_constant<int, 2>{});
#pragma unroll
		for (int w = 0; w < NV; ++w) b0[(e * NV + w) * N + i] = r[w] * ji;
	}
	__syncthreads();
	// back to the solution nodes: B^-1 in each direction
	auto pass = [&](auto tag, const double* src, double* dst) {
		constexpr int A = decltype(tag)::value;
		if (live) {
			const double* row = so->Bi + node_along<A, N1>(i) * N1;
			const int base = pencil_base<A, N1>(i);
			double op[N1];
#pragma unroll
			for (int j = 0; j < N1; ++j) op[j] = row[j];
#pragma unroll
			for (int w = 0; w < NV; ++w) {
				r[w] = pencil_dot<A, N1>(op, src + (e * NV + w) * N, base);
				if (A < D - 1) dst[(e * NV + w) * N + i] = r[w];
			}
		}
		if (A < D - 1) __syncthreads();
	};
	pass(std::integral_constant<int, 0>{}, b0, b1);
	pass(std::integral_constant<int, 1>{}, b1, b0);
	if constexpr (D == 3) pass(std::integral_constant<int, 2>{}, b0, b1);
}

// The stage's new value of one coefficient.
__device__ __forceinline__ double stage_value(int stage, double u0, double up, double r, double dt)
{
	if (stage == 0) return u0 + dt * r;
	if (stage == 1) return (1.0 / 4.0) * (3.0 * up + u0 + dt * r);
	return (1.0 / 3.0) * (up + 2.0 * u0 + 2.0 * dt * r);
}

} // namespace tp
} // namespace dpg
