// One SSP-RK3 stage of a tensor-product mesh in one kernel: the lift with the stage update (tp_lift.cuh), the positivity limiter
// on the new state (the algorithm of positivity.cu), and the next stage's values at the Gauss points, traces and weak
// divergence (tp_volume.cuh).  All three work on the block's own elements, so the state stays in shared memory and a stage
// is two launches (this and the numerical fluxes) instead of four.
// Small meshes are bound by the launch chain and by each kernel's own latency (~5 us a kernel on 16x16 QUAD p = 2), large
// ones by the FP64 pipe, where the fusion saves the state's round trips through memory and the FP32 limiter hides.
#include "positivity.cuh"
#include "tp_lift.cuh"
#include "tp_volume.cuh"

namespace dpg {

using namespace tp;
using namespace pos;

// enforce_positivity_highorder on the block's elements: b0 [E][NV][NS] the state (also in global memory at sol), b1 of the
// same size as work space, flag [E].  All threads call; the pencil of thread t < E P is t % P of element t / P.
template <int D, int N1>
__device__ __forceinline__ void limit_block(const PosOps& ops, float amp, double* b0, double* b1, int* flag, int E, int ne,
                                            double* sol, int* __restrict__ err)
{
	constexpr int NS = ipow(N1, D), NV = D + 2, P = NS / N1;
	const int tid = threadIdx.x, el = tid / P, q = tid - el * P;
	const bool act = el < E, live = el < ne;
	float2* sbc = reinterpret_cast<float2*>(b1);
	if (tid < E) flag[tid] = 0;
	// the FP32 screen of k_positivity: coefficients and the bound of their error, direction by direction
	float b[NV][N1], c[NV][N1];
	auto pass = [&](const float (&x)[N1], float mx, int v) {
#pragma unroll
		for (int i = 0; i < N1; ++i) {
			float yb = 0.f;
#pragma unroll
			for (int k = 0; k < N1; ++k) yb += ops.ai32[i * N1 + k] * x[k];
			b[v][i] = yb;
			c[v][i] = ops.rs * mx;
		}
	};
	if (act) {
#pragma unroll
		for (int v = 0; v < NV; ++v) {
			float x[N1];
			float mx = 0.f;
#pragma unroll
			for (int k = 0; k < N1; ++k) {
				x[k] = trunc_to_float(live ? b0[(el * NV + v) * NS + q * N1 + k] : 1.0);
				mx = k == 0 ? fabsf(x[0]) : fmaxf(mx, fabsf(x[k]));
			}
			pass(x, mx, v);
		}
	}
#pragma unroll
	for (int dir = 1; dir < D; ++dir) {
		const int sp = dir == 1 ? 1 : N1, st = dir == 1 ? N1 : N1 * N1;
		if (act) {
#pragma unroll
			for (int v = 0; v < NV; ++v)
#pragma unroll
				for (int k = 0; k < N1; ++k)
					sbc[(el * NV + v) * NS + q % sp + sp * (k + N1 * (q / sp))] = make_float2(b[v][k], c[v][k]);
		}
		__syncthreads();
		if (act) {
#pragma unroll
			for (int v = 0; v < NV; ++v) {
				float x[N1];
				float mx = 0.f;
#pragma unroll
				for (int k = 0; k < N1; ++k) {
					const float2 t = sbc[(el * NV + v) * NS + q % st + st * (k + N1 * (q / st))];
					x[k] = t.x;
					mx = k == 0 ? t.y : fmaxf(mx, t.y);
				}
				pass(x, mx, v);
			}
		}
	}
	bool bad = false;
	if (live) {
#pragma unroll
		for (int i = 0; i < N1; ++i) {
			const float rho_lo = b[0][i] - amp * c[0][i];
			float m2 = 0.f;
#pragma unroll
			for (int a = 0; a < D; ++a) {
				const float m = fabsf(b[1 + a][i]) + amp * c[1 + a][i];
				m2 += m * m;
			}
			const float eE = amp * c[NV - 1][i];
			const float q2 = 0.5f * m2 / rho_lo, E_lo = b[NV - 1][i] - eE;
			const float p_lo = 0.4f * (E_lo - q2) - 9.5367431640625e-07f * (fabsf(b[NV - 1][i]) + eE + q2);
			bad |= !(rho_lo > 2.0f * (float)DPG_EPS_PHYS) || !(p_lo > 2.0f * (float)DPG_EPS_PHYS);
		}
		if (bad) flag[el] = 1;
	}
	if (!__syncthreads_or(bad)) return;
	// the reference's algorithm in FP64 for the flagged elements
	const int n_buf = E * NV * NS;
	for (int k = tid; k < n_buf; k += blockDim.x) b1[k] = k < ne * NV * NS ? b0[k] : 1.0;
	__syncthreads();
	auto pencils = [&](bool inv) {   // one direction after the other, in place
#pragma unroll
		for (int dir = 0; dir < D; ++dir) {
			const int st = dir == 0 ? 1 : dir == 1 ? N1 : N1 * N1;
			if (act) {
#pragma unroll
				for (int v = 0; v < NV; ++v) {
					double* p = b1 + (el * NV + v) * NS + q % st + st * N1 * (q / st);
					double x[N1], y[N1];
#pragma unroll
					for (int k = 0; k < N1; ++k) x[k] = p[st * k];
					if (inv) apply1<N1>(ops.ai64, x, y);
					else apply1<N1>(ops.a64, x, y);
#pragma unroll
					for (int k = 0; k < N1; ++k) p[st * k] = y[k];
				}
			}
			__syncthreads();
		}
	};
	auto convert = [&](bool to_prim) {
		for (int k = tid; k < E * NS; k += blockDim.x) {
			const int l = k / NS, node = k - l * NS;
			if (!flag[l]) continue;
			double w[NV];
#pragma unroll
			for (int v = 0; v < NV; ++v) w[v] = b1[(l * NV + v) * NS + node];
			if (to_prim) cons_to_prim<D>(w);
			else prim_to_cons<D>(w);
#pragma unroll
			for (int v = 0; v < NV; ++v) b1[(l * NV + v) * NS + node] = w[v];
		}
		__syncthreads();
	};
	pencils(true);
	convert(true);
	if (q == 0 && live && flag[el]) {
		if (!limit_volume<D, NS>(b1 + el * NV * NS)) {
			atomicOr(err, 1);   // average density or pressure below EPS_PHYS: the volume is left unchanged
			flag[el] = 0;
		}
	}
	__syncthreads();
	convert(false);
	pencils(false);
	for (int k = tid; k < n_buf; k += blockDim.x)
		if (flag[k / (NV * NS)]) { b0[k] = b1[k]; sol[k] = b1[k]; }
	__syncthreads();
}

template <int D, int NV, int N1>
static size_t smem_stage(int E)
{
	const size_t N = ipow(N1, D), NF = ipow(N1, D - 1);
	const size_t work = 2 * D * NF > (D - 1) * N ? 2 * D * NF : (D - 1) * N;   // face fluxes, then volume fluxes
	return sizeof(Ops<N1>) + sizeof(double) * E * NV * (2 * N + work) + 8 + sizeof(int) * E;
}

template <int D, int NV, int N1, int KIND, bool OWN>
__global__ void __launch_bounds__(256) k_tp_stage(double* G, const double* nnf, TpGeo g, TpFaces fa, TpBc B,
                                                  const __grid_constant__ Ops<N1> ops, const __grid_constant__ PosOps pops,
                                                  float amp, int* __restrict__ pos_err, double* sol,
                                                  double* solp, const double* __restrict__ dt_ptr,
                                                  unsigned long long* max_slot, int stage, int limit, int next,
                                                  double* __restrict__ trace, double* Gn, int E, double bx, double by, double bz)
{
	constexpr int N = ipow(N1, D), NF = ipow(N1, D - 1);
	constexpr int work = 2 * D * NF > (D - 1) * N ? 2 * D * NF : (D - 1) * N;
	extern __shared__ double sm[];
	Ops<N1>* so = reinterpret_cast<Ops<N1>*>(sm);
	double* b0 = sm + sizeof(Ops<N1>) / sizeof(double);
	double* b1 = b0 + (size_t)E * NV * N;
	double* sW = b1 + (size_t)E * NV * N;
	unsigned long long* s_max = reinterpret_cast<unsigned long long*>(sW + (size_t)E * NV * work);
	int* flag = reinterpret_cast<int*>(s_max + 1);
	const int e0 = blockIdx.x * E, ne = min(E, g.n_vol - e0);
	const int e = threadIdx.x / N, i = threadIdx.x - e * N;
	const bool live = e < ne;
	load_ops(so, ops);
	grid_wait();
	const size_t gi0 = (size_t)e0 * NV * N, gi = gi0 + (size_t)e * NV * N + i;
	double r[NV], u0[NV], up[NV], ji = 0.0;
	if (live) {
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			r[w] = G[gi + w * N];
			u0[w] = sol[gi + w * N];
			up[w] = stage >= 1 ? solp[gi + w * N] : 0.0;
		}
		ji = g.affine ? g.jinv[e0 + e] : g.jinv[(size_t)(e0 + e) * N + i];
	}
	lift_body<D, NV, N1, OWN>(so, b0, b1, sW, e0, ne, g, nnf, fa, ji, r);
	unsigned long long lmax = 0;
	__syncthreads();   // the last pass has read its buffer
	if (live) {
		const double dt = *dt_ptr;
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			const unsigned long long ab = abs_bits_of(r[w]);
			lmax = ab > lmax ? ab : lmax;
			const double un = stage_value(stage, u0[w], up[w], r[w], dt);
			if (stage == 0) solp[gi + w * N] = u0[w];
			sol[gi + w * N] = un;
			b0[(e * NV + w) * N + i] = un;
		}
	}
	block_max_to(lmax, s_max, max_slot);   // its barriers also publish b0
	if constexpr (NV == D + 2) {
		if (limit) limit_block<D, N1>(pops, amp, b0, b1, flag, E, ne, sol + gi0, pos_err);
	}
	if (!next) return;
	volume_body<D, NV, N1, false, KIND>(so, b0, b1, sW, e0, ne, E, true, g, B, trace, nullptr, KIND == kViscous ? Gn : G, nullptr,
	                                    bx, by, bz);
}

template <int D, int NV, int N1>
static int configure_stage(dpg_gpu_ctx* c)
{
	constexpr int E = most_elems(ipow(N1, D));
	constexpr cudaFuncAttribute A = cudaFuncAttributeMaxDynamicSharedMemorySize;
	const int sm = (int)smem_stage<D, NV, N1>(E);
	if (cudaFuncSetAttribute(k_tp_stage<D, NV, N1, kPeriodic, false>, A, sm) || cudaFuncSetAttribute(k_tp_stage<D, NV, N1, kPeriodic, true>, A, sm) ||
	    cudaFuncSetAttribute(k_tp_stage<D, NV, N1, kWalls, false>, A, sm))
		return DPG_ERR_CUDA;
	if constexpr (NV == D + 2)
		if (cudaFuncSetAttribute(k_tp_stage<D, NV, N1, kViscous, false>, A, sm)) return DPG_ERR_CUDA;
	return DPG_OK;
}

template <int D, int NV, int N1>
static int launch_stage(dpg_gpu_ctx* c, int stage, unsigned long long* max_slot, int next)
{
	const TpState* st = (const TpState*)c->tp;
	constexpr int N = ipow(N1, D);
	const TpGeo geo = geo_of(c);
	const TpBc B{st->bc, st->xyz, c->fc.nrm, st->bp};
	const int E = st->E, grid = (geo.n_vol + E - 1) / E, threads = st->own ? own_threads<D, N1>(E) : (E * N + 31) / 32 * 32;
	// own face fluxes: the neighbours still read this stage's traces, so the next stage's go to the other array
	double* const from = st->own && stage == 1 ? st->trace2 : c->trace;
	double* const to = st->own && stage == 0 ? st->trace2 : c->trace;
	const size_t sm = smem_stage<D, NV, N1>(E);
	const Ops<N1> ops = ops_of<N1>(st);
	const int limit = NV == D + 2 && c->positivity;
	const PosOps pops = limit ? pos_ops<N1>(c) : PosOps{};
	auto go = [&](auto kernel) {
		return launch_chained(kernel, grid, threads, sm, c->stream, st->G, c->nnf, geo, faces_of(c, from), B, ops, pops, c->pos_amp,
		                      c->pos_err, c->sol, c->solp, c->ddt, max_slot, stage, limit, next, to, st->Uc, E, c->b_adv[0], c->b_adv[1],
		                      c->b_adv[2]);
	};
	cudaError_t e;
	if constexpr (NV == D + 2) {
		e = st->viscous ? go(k_tp_stage<D, NV, N1, kViscous, false>)
		    : c->walls_or_visc ? go(k_tp_stage<D, NV, N1, kWalls, false>)
		    : st->own ? go(k_tp_stage<D, NV, N1, kPeriodic, true>) : go(k_tp_stage<D, NV, N1, kPeriodic, false>);
	} else {
		e = c->walls_or_visc ? go(k_tp_stage<D, NV, N1, kWalls, false>)
		    : st->own ? go(k_tp_stage<D, NV, N1, kPeriodic, true>) : go(k_tp_stage<D, NV, N1, kPeriodic, false>);
	}
	return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

int tp_configure_stage(dpg_gpu_ctx* c) { DPG_TP_DISPATCH(configure_stage, c); }
static int stage_any(dpg_gpu_ctx* c, int stage, unsigned long long* max_slot, int next)
{
	DPG_TP_DISPATCH(launch_stage, c, stage, max_slot, next);
}

// One SSP-RK3 step of c->sol, norms of the three residuals in max_slots[0..2].
int tp_step(dpg_gpu_ctx* c, unsigned long long* max_slots)
{
	int rc = c->walls_or_visc ? tp_general_front(c) : tp_volume(c);
	for (int stage = 0; stage < 3 && !rc; ++stage) {
		if ((rc = c->walls_or_visc ? tp_general_fluxes(c) : launch_face(c))) break;
		rc = stage_any(c, stage, max_slots + stage, stage < 2);
	}
	return rc;
}

} // namespace dpg
