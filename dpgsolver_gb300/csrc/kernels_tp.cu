// FP64 form of the residual on tensor-product meshes of one order (QUAD, HEX, p = 1..4, periodic): the operators are
// applied one direction at a time in the collocated Gauss basis (tp_ops.cuh).
//
//   k_tp_volume : sol_coef -> values at the Gauss points (B passes) -> face traces of every local face, reference volume
//                 flux and its weak derivative (Dw passes), kept in the collocated basis
//   k_face      : numerical flux per face node (kernels_fp64.cu)
//   k_tp_lift   : + the face fluxes over the weights, / detJ, B^-1 passes -> rhs, ||rhs||_inf and the SSP-RK3 stage
//
// The FP64 pipe bounds all three (1.6-1.7 lanes per clock and SM on this GPU, 0.53 T operations/s), so the count of FP64
// instructions decides: HEX p = 3 Euler needs 210 per node in k_tp_volume and 110 in k_tp_lift where the dense
// operators need 28,672 / 64 x 5 = 2,240.  One thread per (element, node): the operands come from shared memory,
// whose traffic hides behind the FP64 issue rate.  A block holds as many elements as fill 256 threads, fewer on
// small meshes so that every SM has work.  32x32x8 HEX p = 3 Euler: k_tp_volume 183 us, k_tp_lift 100 us (the FP64
// pipe's measured rate) for 967 + 3,694 us of the dense kernels; the whole residual 0.39 against 4.78 ms.
//
// The linearisation (k_tp_volume with TAN, k_face_tan, k_tp_lift) carries (value, tangent) through the same passes.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "dpg_gpu_internal.cuh"
#include "dpg_host.h"
#include "tp_lift.cuh"
#include "tp_volume.cuh"

namespace dpg {

using namespace tp;

// stage < 0: residual only.  stage 0..2: SSP-RK3 stage update of sol (solp holds the step's initial state).  max_slot may
// be null (the linearisation).
template <int D, int NV, int N1, bool OWN>
__global__ void __launch_bounds__(256) k_tp_lift(const double* G, const double* nnf, TpGeo g, TpFaces fa,
                                                 const __grid_constant__ Ops<N1> ops, double* sol,
                                                 double* solp, double* __restrict__ rhs,
                                                 const double* __restrict__ dt_ptr, unsigned long long* max_slot, int stage,
                                                 int write_rhs, int E, TanStride ts)
{
	constexpr int N = ipow(N1, D), NF = ipow(N1, D - 1);
	extern __shared__ double sm[];
	Ops<N1>* so = reinterpret_cast<Ops<N1>*>(sm);
	double* b0 = sm + sizeof(Ops<N1>) / sizeof(double);
	double* b1 = b0 + (size_t)E * NV * N;
	double* sF = b1 + (size_t)E * NV * N;   // [E][2 D][NV][NF] face fluxes in the element's node order, + outward
	unsigned long long* s_max = reinterpret_cast<unsigned long long*>(sF + (size_t)E * NV * 2 * D * NF);
	G += blockIdx.y * ts.dof;
	nnf += blockIdx.y * ts.nf;
	rhs += blockIdx.y * ts.dof;
	const int e0 = blockIdx.x * E, ne = min(E, g.n_vol - e0);
	const int e = threadIdx.x / N, i = threadIdx.x - e * N;
	const bool live = e < ne;
	load_ops(so, ops);
	grid_wait();
	const size_t gi0 = (size_t)e0 * NV * N;
	const size_t gi = gi0 + (size_t)e * NV * N + i;
	double r[NV], u0[NV], up[NV], ji = 0.0;
	if (live) {   // every global operand of the node issued before the first barrier
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			r[w] = G[gi + w * N];
			u0[w] = stage >= 0 ? sol[gi + w * N] : 0.0;
			up[w] = stage >= 1 ? solp[gi + w * N] : 0.0;
		}
		ji = g.affine ? g.jinv[e0 + e] : g.jinv[(size_t)(e0 + e) * N + i];
	}
	lift_body<D, NV, N1, OWN>(so, b0, b1, sF, e0, ne, g, nnf, fa, ji, r);
	unsigned long long lmax = 0;
	if (live) {
		const double dt = (stage >= 0 ? *dt_ptr : 0.0);
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			const size_t k = gi + w * N;
			const unsigned long long ab = abs_bits_of(r[w]);
			lmax = ab > lmax ? ab : lmax;
			if (write_rhs) rhs[k] = r[w];
			if (stage == 0) solp[k] = u0[w];
			if (stage >= 0) sol[k] = stage_value(stage, u0[w], up[w], r[w], dt);
		}
	}
	if (max_slot) block_max_to(lmax, s_max, max_slot);
}

// ------------------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------------------
static bool near(double a, double b, double scale) { return std::fabs(a - b) <= 1e-11 * scale; }

// The 1D operators of order n1 - 1, and whether the element's dense operators are their products.
static bool build_ops(TpState* st, const dpg_element_ops& o)
{
	const int n1 = o.p + 1, d = o.d;
	double gll[16], wgll[16], gl[16], w[16], val[16], der[16];
	dpg_nodes_gll(n1, gll, wgll);
	dpg_nodes_gl(n1, gl, w);
	for (int q = 0; q < n1; ++q) {
		dpg_lagrange_1d(n1, gll, gl[q], val, der);
		for (int i = 0; i < n1; ++i) st->B[q * n1 + i] = val[i];
		dpg_lagrange_1d(n1, gl, gll[q], val, der);   // the inverse map: the collocated basis at the solution nodes
		for (int i = 0; i < n1; ++i) st->Bi[q * n1 + i] = val[i];
		dpg_lagrange_1d(n1, gl, gl[q], val, der);
		for (int i = 0; i < n1; ++i) { st->Dw[i * n1 + q] = w[q] / w[i] * der[i]; st->Ds[q * n1 + i] = der[i]; }
	}
	dpg_lagrange_1d(n1, gl, -1.0, st->lm, der);
	dpg_lagrange_1d(n1, gl, 1.0, st->lp, der);
	for (int i = 0; i < n1; ++i) { st->wm[i] = st->lm[i] / w[i]; st->wp[i] = st->lp[i] / w[i]; }
	// the dense operators entry by entry against products of n1 x n1 factors: interpolation, weak derivative, inverse mass
	// matrix, face traces and lifts
	const int n_s = o.n_s, n_c = o.n_c, n_fc = o.n_fc;
	double D1[25], M1[25], e1[2][5];   // l_s'(Gauss point), 1D inverse mass matrix, solution basis at -1 / +1
	for (int i = 0; i < n1; ++i)
		for (int j = 0; j < n1; ++j) {
			double t = 0.0, m = 0.0;
			for (int k = 0; k < n1; ++k) {
				t += st->Ds[i * n1 + k] * st->B[k * n1 + j];
				m += st->Bi[i * n1 + k] * st->Bi[j * n1 + k] / w[k];
			}
			D1[i * n1 + j] = t;
			M1[i * n1 + j] = m;
		}
	for (int s = 0; s < n1; ++s) {
		e1[0][s] = e1[1][s] = 0.0;
		for (int j = 0; j < n1; ++j) { e1[0][s] += st->lm[j] * st->B[j * n1 + s]; e1[1][s] += st->lp[j] * st->B[j * n1 + s]; }
	}
	std::vector<int> dig((size_t)n_s * 3);   // position along each direction of node k (solution and Gauss nodes alike)
	for (int k = 0; k < n_s; ++k)
		for (int a = 0, t = k; a < 3; ++a, t /= n1) dig[3 * k + a] = t % n1;
	for (int c = 0; c < n_c; ++c)
		for (int s = 0; s < n_s; ++s) {
			const int *ci = &dig[3 * c], *si = &dig[3 * s];
			double f[3], g[3], b = 1.0, wc = 1.0, m = 1.0;
			for (int a = 0; a < d; ++a) {
				f[a] = st->B[ci[a] * n1 + si[a]];
				g[a] = D1[ci[a] * n1 + si[a]];
				b *= f[a];
				wc *= w[ci[a]];
				m *= M1[ci[a] * n1 + si[a]];
			}
			if (!near(o.cv0_vs_vc[(size_t)c * n_s + s], b, 1.0) || !near(o.m_inv_ref[(size_t)c * n_s + s], m, 1e3)) return false;
			for (int r = 0; r < d; ++r) {
				double t = wc;
				for (int a = 0; a < d; ++a) t *= a == r ? g[a] : f[a];
				if (!near(o.tw1_vt_vc[((size_t)r * n_s + s) * n_c + c], t, 10.0)) return false;
			}
		}
	for (int lf = 0; lf < 2 * d; ++lf)
		for (int q = 0; q < n_fc; ++q) {
			int k[3] = {0, 0, 0}, t = q;
			double wf = 1.0;
			for (int a = 0; a < d; ++a)
				if (a != (lf >> 1)) { k[a] = t % n1; t /= n1; wf *= w[k[a]]; }
			for (int s = 0; s < n_s; ++s) {
				double y = e1[lf & 1][dig[3 * s + (lf >> 1)]];
				for (int a = 0; a < d; ++a)
					if (a != (lf >> 1)) y *= st->B[k[a] * n1 + dig[3 * s + a]];
				if (!near(o.cv0_vs_fc[((size_t)lf * n_fc + q) * n_s + s], y, 1.0) ||
				    !near(o.tw0_vt_fc[((size_t)lf * n_s + s) * n_fc + q], y * wf, 1.0))
					return false;
			}
		}
	return true;
}

void tp_free(dpg_gpu_ctx* c)
{
	TpState* st = (TpState*)c->tp;
	if (!st) return;
	for (void* p : st->allocs) cudaFree(p);
	delete st;
	c->tp = nullptr;
}

// Elements per block, at most 256 threads: the fewest warps on the fullest SM (a warp's FP64 instruction holds its SM's
// pipe for ~20 cycles however many of its lanes are in use), the larger block of equal ones.
static int block_elems(int n_vol, int N, int n_sm)
{
	int best = 1;
	int64_t cost = INT64_MAX;
	for (int E = 1; E <= most_elems(N); ++E) {
		const int64_t blocks = (n_vol + E - 1) / E, c = (blocks + n_sm - 1) / n_sm * ((E * N + 31) / 32);
		if (c <= cost) { cost = c; best = E; }
	}
	return best;
}

// Shared-memory opt-in at the largest block: one limit for every context of the process.
template <int D, int NV, int N1>
static int configure()
{
	constexpr int E = most_elems(ipow(N1, D));
	if (cudaFuncSetAttribute(k_tp_volume<D, NV, N1, false, kPeriodic>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_volume<D, NV, N1, false>(E)) ||
	    cudaFuncSetAttribute(k_tp_volume<D, NV, N1, true, kPeriodic>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_volume<D, NV, N1, true>(E)) ||
	    cudaFuncSetAttribute(k_tp_lift<D, NV, N1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_lift<D, NV, N1>(E)) ||
	    cudaFuncSetAttribute(k_tp_lift<D, NV, N1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_lift<D, NV, N1>(E)))
		return DPG_ERR_CUDA;
	return DPG_OK;
}

template <int D, int NV, int N1>
static int launch_volume(dpg_gpu_ctx* c, const double* u, const double* v, const TanWork* w)
{
	const TpState* st = (const TpState*)c->tp;
	constexpr int N = ipow(N1, D);
	const TpGeo geo = geo_of(c);
	const int E = st->E, grid = (geo.n_vol + E - 1) / E, threads = (E * N + 31) / 32 * 32;
	const Ops<N1> ops = ops_of<N1>(st);
	if (v)
		launch_chained(k_tp_volume<D, NV, N1, true, kPeriodic>, dim3(grid, w->nb), threads, smem_volume<D, NV, N1, true>(E), c->stream, u, v, geo, TpBc{}, ops, c->trace, w->trace_t, w->G, nullptr, E, c->b_adv[0], c->b_adv[1], c->b_adv[2], tan_stride(c));
	else
		launch_chained(k_tp_volume<D, NV, N1, false, kPeriodic>, grid, threads, smem_volume<D, NV, N1, false>(E), c->stream, u, nullptr, geo, TpBc{}, ops, c->trace, nullptr, st->G, nullptr, E, c->b_adv[0], c->b_adv[1], c->b_adv[2], TanStride{});
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

template <int D, int NV, int N1>
static int launch_lift(dpg_gpu_ctx* c, const double* G, const double* nnf, double* rhs, unsigned long long* max_slot, int stage,
                       bool write_rhs, int nb)
{
	const TpState* st = (const TpState*)c->tp;
	constexpr int N = ipow(N1, D);
	const TpGeo geo = geo_of(c);
	const bool own = st->own && nnf == c->nnf;
	const int E = st->E, grid = (geo.n_vol + E - 1) / E, threads = own ? own_threads<D, N1>(E) : (E * N + 31) / 32 * 32;
	launch_chained(own ? k_tp_lift<D, NV, N1, true> : k_tp_lift<D, NV, N1, false>, dim3(grid, nb), threads, smem_lift<D, NV, N1>(E), c->stream, G, nnf, geo, faces_of(c, c->trace), ops_of<N1>(st), c->sol, c->solp, rhs, c->ddt, max_slot, stage, write_rhs ? 1 : 0, E, tan_stride(c));
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

static int configure_any(dpg_gpu_ctx* c) { DPG_TP_DISPATCH(configure); }

int tp_volume(dpg_gpu_ctx* c) { DPG_TP_DISPATCH(launch_volume, c, c->sol, nullptr, nullptr); }
int tp_volume_tan(dpg_gpu_ctx* c, const double* u, const double* v, const TanWork& w)
{
	DPG_TP_DISPATCH(launch_volume, c, u, v, &w);
}
int tp_lift(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot)
{
	DPG_TP_DISPATCH(launch_lift, c, ((const TpState*)c->tp)->G, c->nnf, c->rhs, max_slot, stage, write_rhs, 1);
}
int tp_lift_tan(dpg_gpu_ctx* c, const TanWork& w, double* out)
{
	DPG_TP_DISPATCH(launch_lift, c, w.G, w.nnf_t, out, nullptr, -1, true, w.nb);
}
bool tp_own_faces(const dpg_gpu_ctx* c) { return ((const TpState*)c->tp)->own; }
bool tp_viscous(const dpg_gpu_ctx* c) { return ((const TpState*)c->tp)->viscous != 0; }

// Set-up.  Leaves c->tp null (the dense kernels of kernels_fp64.cu run) where the element is not one of the orders above
// or its operators are not the products of the 1D ones.
int tp_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim, bool general)
{
	const dpg_element_ops& o = sim->ops[0];
	if ((o.e_type != DPG_QUAD && o.e_type != DPG_HEX) || o.p < 1 || o.p + 1 > kN1Max) return DPG_OK;
	const int N = ipow(o.p + 1, o.d);
	if (o.n_s != N || o.n_c != N || o.n_fc != ipow(o.p + 1, o.d - 1) || o.n_fl != 2 * o.d) return DPG_OK;
	// Periodic meshes of fewer nodes keep the dense kernels for their summation order, not for speed: a Newton solve there runs
	// until its systems are near-singular and its residual is rounding, and ends elsewhere when a sum is
	// reordered (8x8 QUAD p = 2, uniform stream: by 6e-5 of the state).  The line lies above the small Newton problems of
	// the tests and the benchmark (900 nodes at most), whose results are kept.  us per step, 1D operators / dense (both with their own face fluxes): QUAD p = 1, 64 nodes 38.9 / 45.1, 900: 41.0 /
	// 45.1, 1,024: 41.2 / 46.0; QUAD p = 2, 576: 45.1 / 51.2, 1,296: 47.7 / 52; QUAD p = 4, 900: 53.4 / 67.6; HEX p = 1, 1,000: 55.3 / 59.0;
	// HEX p = 2, 729: 164 / 201; HEX p = 3, 768: 256 / 508.  One residual is equal on both sides up to p = 3 (37 to 47 us).
	constexpr int64_t kMinNodes = 1024;
	if (!general && (int64_t)sim->n_vol * N < kMinNodes) return DPG_OK;
	TpState* st = new TpState();
	st->n1 = o.p + 1;
	if (!build_ops(st, o)) { delete st; return DPG_OK; }
	c->tp = st;
	auto alloc = [&](double** p, size_t n) {
		void* q = nullptr;
		if (cudaMalloc(&q, n * sizeof(double)) != cudaSuccess) return (int)DPG_ERR_CUDA;
		st->allocs.push_back(q);
		*p = (double*)q;
		return (int)DPG_OK;
	};
	int rc;
	if ((rc = alloc(&st->G, (size_t)c->n_dof))) return rc;
	if (!c->g.affine) {
		std::vector<double> ji((size_t)sim->n_vol * N);
		for (int v = 0; v < sim->n_vol; ++v)
			for (int k = 0; k < N; ++k) ji[(size_t)v * N + k] = 1.0 / sim->jacobian_det_vc[sim->vol_geo_off[v] + k];
		if ((rc = alloc(&st->jn, ji.size()))) return rc;
		if (cudaMemcpy(st->jn, ji.data(), sizeof(double) * ji.size(), cudaMemcpyHostToDevice) != cudaSuccess) return DPG_ERR_CUDA;
	}
	st->E = block_elems(sim->n_vol, N, c->n_sm);
	// Below this many face nodes the lift and stage kernels form their elements' face fluxes (each flux twice, one launch less);
	// the FP64 pipe has the time.  us per step (with the limiter), so / with k_face: QUAD p = 1, 4,096 face nodes:
	// 41.3 / 47.6, 16,384: 55.5 / 50.1; QUAD p = 2, 1,536: 47.7 / 51.6, 15,000: 59.8 / 59.5; QUAD p = 3, 8,192: 51.5 / 53.8,
	// 20,000: 84.6 / 80.4; HEX p = 1, 6,144: 53.5 / 64.4, 12,000: 61.8 / 65.7, 32,928: 98.5 / 80.3; HEX p = 2, 13,824: 74.1 / 71.8;
	// HEX p = 3, 10,368: 76.0 / 76.1.  One residual gains 3 to 7 us of 31 to 36.
	const int64_t face_nodes = sim->face_geo_off[sim->n_face];
	if (!general && face_nodes <= kOwnFaceNodes) {
		if ((rc = alloc(&st->trace2, (size_t)2 * c->n_var * face_nodes))) return rc;
		st->own = true;
	}
	const int rc2 = configure_any(c);
	return rc2 ? rc2 : tp_configure_stage(c);
}

} // namespace dpg
