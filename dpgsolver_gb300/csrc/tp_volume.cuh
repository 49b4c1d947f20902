// First kernel of the tensor-product residual (kernels_tp.cu, kernels_tp_general.cu): one thread per (element, node).
#pragma once

#include "tp_ops.cuh"

namespace dpg {
namespace tp {

// Shared memory (doubles): the operators, then two buffers of E NW N values and D - 1 of E NV N (the fluxes of direction
// 0 reuse the buffer the last B pass read from).
template <int D, int NV, int N1, bool TAN>
inline size_t smem_volume(int E)
{
	const size_t N = ipow(N1, D), NW = TAN ? 2 * NV : NV;
	return sizeof(Ops<N1>) + sizeof(double) * E * N * (2 * NW + (D - 1) * NV);
}

// kPeriodic: every face has two elements.  kWalls: the boundary states of boundary faces go to their side-1 trace slots.
// kViscous: kWalls, and the collocated values (G, G_t) instead of the weak divergence, which needs the gradients.
enum { kPeriodic = 0, kWalls = 1, kViscous = 2 };

// What follows the state in b0 (all threads synchronised): values at the Gauss points, traces, (boundary states,) and the weak
// divergence or the collocated values.  Each buffer is read by the traces between the barriers of the passes that write and
// overwrite it.
template <int D, int NV, int N1, bool TAN, int KIND>
__device__ __forceinline__ void volume_body(const Ops<N1>* so, double* b0, double* b1, double* fl, int e0, int ne, int E, bool first,
                                            const TpGeo& g, const TpBc& B, double* __restrict__ trace,
                                            double* __restrict__ trace_t, double* __restrict__ G, double* __restrict__ G_t,
                                            double bx, double by, double bz)
{
	constexpr int N = ipow(N1, D), NF = ipow(N1, D - 1), NW = TAN ? 2 * NV : NV;
	const int e = threadIdx.x / N, i = threadIdx.x - e * N;
	const bool live = e < ne;
	double m[D][D];   // of this node's element (affine) or node
	if (KIND != kViscous && live) {
#pragma unroll
		for (int x = 0; x < D; ++x)
#pragma unroll
			for (int r = 0; r < D; ++r)
				m[x][r] = g.affine ? g.met[(size_t)(e0 + e) * D * D + x + D * r]
				                   : g.met[((size_t)(e0 + e) * D * D + x + D * r) * N + i];
	}
	// values at the Gauss points: pass 0 b0 -> b1, pass 1 b1 -> b0, (pass 2 b0 -> b1)
	double s[NW];
	auto pass = [&](auto tag, const double* src, double* dst) {
		constexpr int A = decltype(tag)::value;
		if (live) {
			const double* row = so->B + node_along<A, N1>(i) * N1;
			const int base = pencil_base<A, N1>(i);
			double op[N1];
#pragma unroll
			for (int j = 0; j < N1; ++j) op[j] = row[j];
#pragma unroll
			for (int w = 0; w < NW; ++w) {
				s[w] = pencil_dot<A, N1>(op, src + (e * NW + w) * N, base);
				dst[(e * NW + w) * N + i] = s[w];
			}
		}
		__syncthreads();
	};
	// traces of the two local faces of direction a, in the element's own node order; value(element, side, face node, variable)
	auto traces = [&](int a, auto value) {
		for (int o = threadIdx.x; o < ne * 2 * NF; o += blockDim.x) {
			const int ee = o / (2 * NF), r = o - ee * 2 * NF, side = r / NF, q = r - side * NF;
			const size_t vf = (size_t)g.vol_face[(size_t)(e0 + ee) * 2 * D + 2 * a + side];
			double tr[NW];
#pragma unroll
			for (int w = 0; w < NW; ++w) {
				tr[w] = value(ee, side, q, w);
				if (w >= NV || !TAN || first) (w < NV ? trace : trace_t)[(vf * NV + (w < NV ? w : w - NV)) * NF + q] = tr[w];
			}
			if constexpr (KIND != kPeriodic) {
				const size_t f = vf >> 1;
				const int code = B.bc ? B.bc[f] : 0;
				if (code) {   // the only side of a boundary face: its nodes are in this order
					double n[D], x[3] = {0.0, 0.0, 0.0};
#pragma unroll
					for (int k = 0; k < D; ++k) { n[k] = B.nrm[(f * NF + q) * D + k]; x[k] = B.xyz[(f * NF + q) * D + k]; }
					using T = typename std::conditional<TAN, dual, double>::type;
					T sl[NV], sb[NV];
#pragma unroll
					for (int w = 0; w < NV; ++w) {
						if constexpr (TAN) sl[w] = dual(tr[w], tr[NV + w]);
						else sl[w] = tr[w];
					}
					if constexpr (NV == D + 2) boundary_state<D>(code, sl, n, x, B.bp, sb);
					else sb[0] = sl[0];
#pragma unroll
					for (int w = 0; w < NV; ++w) {
						const size_t k = ((vf + 1) * NV + w) * NF + q;
						if constexpr (TAN) { if (first) trace[k] = sb[w].v; trace_t[k] = sb[w].d; }
						else trace[k] = sb[w];
					}
				}
			}
		}
	};
	// The traces come straight from the solution nodes, whose first and last of a direction lie on the faces: only the tangential
	// directions are interpolated, N1 or no multiply-adds per face node, variable and step (2D: N1 for direction 0, none for
	// direction 1; 3D: 2 N1, N1, none).  Extrapolated from the Gauss points they would carry the rounding of three passes
	// with sums of up to 2.1 in magnitude: rms error of the residual of a vortex against extended precision, this way /
	// extrapolated / dense, HEX p = 1 1.16e-14 / 1.37e-14 / 1.40e-14, p = 2 1.20e-14 / 2.02e-14 / 1.70e-14, p = 3 2.67e-14 / 3.15e-14 / 5.17e-14, QUAD p = 1
	// 9.35e-14 / 9.73e-14 / 9.45e-14, jittered p = 3 3.12e-13 / 3.17e-13 / 3.36e-13.  Viscous face gradients amplify a jump's error by
	// ~4 p^2 / h: extrapolated, the energy residual at the 64x128 annulus' steady state stays at 2e-10 (this way and dense: below
	// 1e-10).
	auto along = [&](const double* u, int S, int q) {   // sum_j B[q][j] u[j S]
		double y = so->B[q * N1] * u[0];
#pragma unroll
		for (int j = 1; j < N1; ++j) y = fma(so->B[q * N1 + j], u[j * S], y);
		return y;
	};
	if constexpr (D == 2) {
		traces(0, [&](int ee, int side, int q, int w) { return along(b0 + (ee * NW + w) * N + side * (N1 - 1), N1, q); });
	} else {   // direction 0: along direction 1 first, into the space of the fluxes, [element][side][variable][k][q]
		for (int o = threadIdx.x; o < ne * 2 * NF; o += blockDim.x) {
			const int ee = o / (2 * NF), r = o - ee * 2 * NF, side = r / NF, kq = r - side * NF, k = kq / N1, q = kq - k * N1;
#pragma unroll
			for (int w = 0; w < NW; ++w)
				fl[((ee * 2 + side) * NW + w) * NF + kq] = along(b0 + (ee * NW + w) * N + side * (N1 - 1) + N1 * N1 * k, N1, q);
		}
	}
	pass(std::integral_constant<int, 0>{}, b0, b1);
	if constexpr (D == 2) {
		traces(1, [&](int ee, int side, int q, int w) { return b1[(ee * NW + w) * N + q + N1 * side * (N1 - 1)]; });
	} else {
		traces(0, [&](int ee, int side, int q, int w) {
			const int qb = q / N1;
			return along(fl + ((ee * 2 + side) * NW + w) * NF + q - qb * N1, N1, qb);
		});
		traces(1, [&](int ee, int side, int q, int w) {
			const int qb = q / N1;
			return along(b1 + (ee * NW + w) * N + q - qb * N1 + N1 * side * (N1 - 1), N1 * N1, qb);
		});
	}
	pass(std::integral_constant<int, 1>{}, b1, b0);
	if constexpr (D == 3) {
		traces(2, [&](int ee, int side, int q, int w) { return b0[(ee * NW + w) * N + q + N1 * N1 * side * (N1 - 1)]; });
		pass(std::integral_constant<int, 2>{}, b0, b1);
	}
	double* f0 = D == 3 ? b0 : b1;           // free: the fluxes of direction 0
	if (KIND == kViscous && live) {
#pragma unroll
		for (int w = 0; w < NW; ++w)
			if (w >= NV || !TAN || first) (w < NV ? G : G_t)[((size_t)(e0 + e) * NV + (w < NV ? w : w - NV)) * N + i] = s[w];
	}
	// reference fluxes of this node (TAN: their tangents)
	if (KIND != kViscous && live) {
		const double b[3] = {bx, by, bz};
		auto met = [&](int x, int r) { return m[x][r]; };
		auto put = [&](int r, int w, double y) { (r == 0 ? f0 : fl + (size_t)(r - 1) * E * NV * N)[(e * NV + w) * N + i] = y; };
		if constexpr (TAN) {
			dual sd[NV];
#pragma unroll
			for (int w = 0; w < NV; ++w) sd[w] = dual(s[w], s[NV + w]);
			ref_flux<D, NV>(sd, met, b, [&](int r, const dual (&fr)[NV]) {
#pragma unroll
				for (int w = 0; w < NV; ++w) put(r, w, fr[w].d);
			});
		} else {
			ref_flux<D, NV>(s, met, b, [&](int r, const double (&fr)[NV]) {
#pragma unroll
				for (int w = 0; w < NV; ++w) put(r, w, fr[w]);
			});
		}
	}
	if constexpr (KIND == kViscous) return;
	__syncthreads();
	// weak divergence
	if (live) {
		double acc[NV];
		auto add = [&](auto tag, const double* src) {
			constexpr int A = decltype(tag)::value;
			const double* row = so->Dw + node_along<A, N1>(i) * N1;
			const int base = pencil_base<A, N1>(i);
			double op[N1];
#pragma unroll
			for (int j = 0; j < N1; ++j) op[j] = row[j];
#pragma unroll
			for (int w = 0; w < NV; ++w) {
				const double* x = src + (e * NV + w) * N + base;
#pragma unroll
				for (int j = 0; j < N1; ++j)
					acc[w] = (A == 0 && j == 0) ? op[0] * x[0] : fma(op[j], x[j * ipow(N1, A)], acc[w]);
			}
		};
		add(std::integral_constant<int, 0>{}, f0);
		add(std::integral_constant<int, 1>{}, fl);
		if constexpr (D == 3) add(std::integral_constant<int, 2>{}, fl + (size_t)E * NV * N);
#pragma unroll
		for (int w = 0; w < NV; ++w) G[((size_t)(e0 + e) * NV + w) * N + i] = acc[w];
	}
}

template <int D, int NV, int N1, bool TAN, int KIND>
__global__ void __launch_bounds__(256) k_tp_volume(const double* u, const double* v, TpGeo g, TpBc B,
                                                   const __grid_constant__ Ops<N1> ops, double* __restrict__ trace,
                                                   double* __restrict__ trace_t, double* __restrict__ G,
                                                   double* __restrict__ G_t, int E, double bx, double by, double bz, TanStride ts)
{
	constexpr int N = ipow(N1, D), NW = TAN ? 2 * NV : NV;
	extern __shared__ double sm[];
	Ops<N1>* so = reinterpret_cast<Ops<N1>*>(sm);
	double* b0 = sm + sizeof(Ops<N1>) / sizeof(double);
	double* b1 = b0 + (size_t)E * NW * N;
	double* fl = b1 + (size_t)E * NW * N;   // [D - 1][E][NV][N]
	const int e0 = blockIdx.x * E, ne = min(E, g.n_vol - e0);
	const bool first = blockIdx.y == 0;   // TAN: the direction that writes the values all directions share
	if constexpr (TAN) {
		v += blockIdx.y * ts.dof;
		trace_t += blockIdx.y * ts.tr;
		(KIND == kViscous ? G_t : G) += blockIdx.y * ts.dof;
	}
	load_ops(so, ops);
	grid_wait();
	const size_t g0 = (size_t)e0 * NV * N;
	for (int k = threadIdx.x; k < ne * NV * N; k += blockDim.x) {
		if constexpr (TAN) {
			const int ee = k / (NV * N), r = k - ee * NV * N;
			b0[ee * NW * N + r] = u[g0 + k];
			b0[ee * NW * N + NV * N + r] = v[g0 + k];
		} else {
			b0[k] = u[g0 + k];
		}
	}
	__syncthreads();
	volume_body<D, NV, N1, TAN, KIND>(so, b0, b1, fl, e0, ne, E, first, g, B, trace, trace_t, G, G_t, bx, by, bz);
}

} // namespace tp
} // namespace dpg
