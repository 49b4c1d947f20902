// Mixed orders (hp meshes) in the FP64 form of the DG residual: volumes grouped by order, each launch covering every
// group.
//
//   k_hp_trace  : per volume, the trace of every local face at the cubature of the face's order p_f (the larger
//                 order of its two volumes, compute_face_reference_order, face_solver.c:123-132), through the
//                 volume basis' operator cv0_vs_fc[p_f][p] (get_operator__cv0_vs_fc_T, compute_face_rlhs_T.c:67-80).
//   k_hp_face   : (Euler) per face node, the numerical flux with the left normal, scaled by jacobian_det_fc.
//   k_hp_volume : per volume, volume flux, the face fluxes of its local faces in local-face order (right sides
//                 reordered and negated; advection computes them here from the traces: an upwind flux costs less than a
//                 launch), one lift contraction over [tw1 | -tw0[p_f(0)] | -tw0[p_f(1)] | ...] (m_inv_ref folded in for
//                 affine groups), the mass-matrix inverse, ||rhs||_inf and the SSP-RK3 stage.
//   k_hp_advect : advection on affine elements, also of one order (TRI, TET): the same in one launch per stage.  Metrics and
//                 velocity are constant, so the volume part is sum_r a_r [lift_r Cv] u, d n_s^2 multiply-adds instead
//                 of (d + 1) n_s n_c; after the stage it writes the traces of the new state for the next one
//                 (two trace arrays in turn).
// A block processes E_b volumes of one group; the grid is the concatenation of the groups' blocks.  The per-face arrays
// (traces, fluxes, normals, node correspondence) are packed by face at the face-node offsets of the host data
// model (face_geo_off).
//
// Bound: the chain of a block on small meshes (~50 dependent FP64 multiply-adds behind its loads), the FP64 pipe on large ones
// (34,992 TETs p = 3: 79 % of its 0.53 T multiply-adds per second).  So a local face's order, side and offset come from
// one 16-byte entry per volume and local face in group order (they were five loads, one after the other); the operators are
// stored K-major, a warp reading consecutive entries, and staged in shared memory where they are small; a thread
// carries all variables of its node; blocks have one coefficient per thread at most (a block of 16 TETs of order 4 held
// its SM for 160 us, 3 of them spread over the chip) and the highest order comes first.
//   advection, us per SSP-RK3 step, before / now (before: dense k_trace, k_face, k_volume or this file's):
//     TRI 1..4 (mixed),  8,192: 105 / 58     TET 1..4 (mixed), 34,992: 2,288 / 918
//     TRI 1,   8,192: 39 / 27                TRI 4, 288: 46 / 24, 8,192: 103 / 80, 32,768: 308 / 263
//     TET 2,  34,992: 322 / 281              TET 3, 3,072: 165 / 93, 34,992: 906 / 783      TET 4, 3,072: 683 / 193
//   Euler (mixed), us per step: TRI 1..3, 1,152 volumes: 91 / 88; QUAD 1..4, 64: 337 / 131, 10,000: 792 / 514; HEX 1..3, 64:
//   1,659 / 449, 1,728: 2,998 / 1,012
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "dpg_gpu_internal.cuh"
#include "flux.cuh"

namespace dpg {

constexpr int kHpMaxGroups = DPG_P_MAX;
constexpr int kHpThreads = 128;
constexpr size_t kHpStageBytes = 16 * 1024;   // operators of a group up to this size are staged in shared memory

struct HpGroup {
	int p, n_vol, n_s, n_c, E_b, blk0;     // blk0: first block of the group in every launch
	int affine;                            // every volume affine: the lift carries m_inv_ref, scale by 1 / detJ
	int n_stage;                           // doubles of `ops` staged in shared memory by k_hp_volume (0: too many)
	int n_tr0, n_tr;                       // the trace operators' part of ops: first entry, entries
	const int* vols;                       // [n_vol] volume indices
	const int64_t* dof;                    // [n_vol] first coefficient
	const int4* side;                      // [n_vol][n_fl]: first K of the face in the lift; p_f | side << 8 | n_fc << 16; offset (lo, hi)
	const double* ops;                     // all K-major: Cv [n_s][n_c], lift, volume part [d n_c][n_s] (folded: their products
	                                       // [d][n_s][n_s]) | oL[p_f]: lift, face part [n_fl n_fc][n_s], negated .. |
	                                       // oT[p_f]: traces [n_s][n_fl n_fc] ..
	int oL[DPG_P_MAX + 1], oT[DPG_P_MAX + 1];
	const double* minv;                    // non-affine groups: [n_vol][n_s x n_s] in group order
	const double* met;                     // affine: [n_vol][d d]; else [n_vol][d d][n_c], group order
	const double* jinv;                    // affine: [n_vol]
};

struct HpDev {
	int n_groups, n_fl, n_blocks, nfc_max;
	int n_fc[DPG_P_MAX + 1];               // face cubature nodes by order
	HpGroup grp[kHpMaxGroups];
	const int64_t* dof_off;                // [n_vol + 1]
	const int* vol_face;                   // [n_vol][n_fl]: (face << 1) | side
	const int* face_p;                     // [n_face]
	const int64_t* fnode_off;              // [n_face + 1]
	const int* node_face;                  // [n_fnode]
	const int* nc;                         // [n_fnode] right node of each left node
	const int* nc_inv;                     // [n_fnode]
	const double* nrm;                     // [n_fnode][d]
	const double* jf;                      // [n_fnode]
	int64_t n_fnode;
};

struct HpState {
	HpDev dev{};
	std::vector<void*> allocs;
	double* trace[2] = {};                 // [2 n_var n_fnode]; the second: advection, in turn with the first
	double* nnf = nullptr;                 // [n_var n_fnode] (Euler)
	size_t smem_trace = 0, smem_volume = 0;
	int blocks = 0;
	bool folded = false;                   // k_hp_advect in the place of k_hp_volume
	bool own = false;                      // Euler, small meshes: k_hp_volume forms its elements' face fluxes
};

__device__ __forceinline__ int hp_group_of(const HpDev& h, int blk)
{
	int g = 0;
	while (g + 1 < h.n_groups && h.grp[g + 1].blk0 <= blk) ++g;
	return g;
}

__device__ __forceinline__ void hp_atomic_max_abs(unsigned long long* slot, double v)
{
	atomicMax(slot, (unsigned long long)__double_as_longlong(fabs(v)));
}

__device__ __forceinline__ int64_t side_offset(const int4& t) { return (int64_t)((unsigned long long)(unsigned)t.z | (unsigned long long)(unsigned)t.w << 32); }

// Traces of the block's ne volumes from their coefficients sU [ne][NV][n_s]; ops: the group's trace operators.
template <int NV>
__device__ __forceinline__ void hp_traces(const double* sU, const int4* sSide, const HpGroup& G, const double* ops, int n_fl, int nfm,
                                          int ne, double* __restrict__ trace)
{
	const int n_s = G.n_s, per_e = n_fl * nfm;
	for (int o = threadIdx.x; o < ne * per_e; o += blockDim.x) {
		const int e = o / per_e, r = o - e * per_e, lf = r / nfm, q = r - lf * nfm;
		const int4 t = sSide[e * n_fl + lf];
		const int pf = t.y & 255, side = (t.y >> 8) & 1, n_fc = t.y >> 16;
		if (q >= n_fc) continue;
		const double* op = ops + (G.oT[pf] - G.n_tr0) + lf * n_fc + q;
		const double* u = sU + e * NV * n_s;
		double acc[NV];
#pragma unroll
		for (int v = 0; v < NV; ++v) acc[v] = 0.0;
#pragma unroll 4
		for (int s = 0; s < n_s; ++s) {
			const double a = op[s * n_fl * n_fc];
#pragma unroll
			for (int v = 0; v < NV; ++v) acc[v] = fma(a, u[v * n_s + s], acc[v]);
		}
		double* y = trace + 2 * NV * side_offset(t) + (size_t)(side * NV) * n_fc + q;
#pragma unroll
		for (int v = 0; v < NV; ++v) y[(size_t)v * n_fc] = acc[v];
	}
}

template <int NV>
__global__ void __launch_bounds__(kHpThreads) k_hp_trace(const double* sol, const __grid_constant__ HpDev h, double* __restrict__ trace)
{
	extern __shared__ __align__(16) double sm[];
	const HpGroup& G = h.grp[hp_group_of(h, blockIdx.x)];
	const int n_s = G.n_s, n_fl = h.n_fl;
	const int e0 = (blockIdx.x - G.blk0) * G.E_b;
	const int ne = min(G.E_b, G.n_vol - e0);
	int4* sSide = reinterpret_cast<int4*>(sm);                    // [E_b][n_fl]
	double* sU = sm + 2 * G.E_b * n_fl;                           // [E_b][NV][n_s]
	double* sT = sU + G.E_b * NV * n_s;
	for (int i = threadIdx.x; i < ne * n_fl; i += blockDim.x) sSide[i] = G.side[(size_t)e0 * n_fl + i];
	if (G.n_stage)
		for (int i = threadIdx.x; i < G.n_tr; i += blockDim.x) sT[i] = G.ops[G.n_tr0 + i];
	grid_wait();
	for (int i = threadIdx.x; i < ne * NV * n_s; i += blockDim.x) {
		const int e = i / (NV * n_s), r = i - e * NV * n_s;
		sU[i] = sol[G.dof[e0 + e] + r];
	}
	__syncthreads();
	hp_traces<NV>(sU, sSide, G, G.n_stage ? sT : G.ops + G.n_tr0, n_fl, h.nfc_max, ne, trace);
}

// The numerical flux of a face node times its face Jacobian.
template <int D, int NV>
__device__ __forceinline__ void hp_numflux(const double* WL, const double* WR, const double* n, double j, int num_flux, const double* b, double* nf)
{
	if constexpr (NV == 1) {
		nf[0] = numflux_upwind<D>(b, WL[0], WR[0], n) * j;
	} else {
		if (num_flux == DPG_NUM_FLUX_ROE_PIKE) numflux_roe_pike_rs<D>(WL, WR, n, 0.5 * j, nf);
		else                                   numflux_lax_friedrichs_rs<D>(WL, WR, n, 0.5 * j, nf);
	}
}

template <int D, int NV>
__global__ void __launch_bounds__(128) k_hp_face(const double* trace, const __grid_constant__ HpDev h, double* __restrict__ nnf,
                                                 int num_flux)
{
	grid_wait();
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= h.n_fnode) return;
	const int f = h.node_face[t];
	const int64_t off = h.fnode_off[f];
	const int n_fc = (int)(h.fnode_off[f + 1] - off), q = (int)(t - off);
	const int qr = h.nc[t];
	double WL[NV], WR[NV], n[D], nf[NV];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		WL[v] = trace[2 * NV * off + (size_t)v * n_fc + q];
		WR[v] = trace[2 * NV * off + (size_t)(NV + v) * n_fc + qr];
	}
#pragma unroll
	for (int a = 0; a < D; ++a) n[a] = h.nrm[t * D + a];
	hp_numflux<D, NV>(WL, WR, n, h.jf[t], num_flux, nullptr, nf);
#pragma unroll
	for (int v = 0; v < NV; ++v) nnf[NV * off + (size_t)v * n_fc + q] = nf[v];
}

// stage < 0: residual only.  stage 0..2: SSP-RK3 stage update (solp holds the step's initial state).  flux: face fluxes
// or, OWN, traces: the block forms its elements' face fluxes itself.
template <int D, int NV, bool OWN>
__global__ void __launch_bounds__(kHpThreads) k_hp_volume(double* sol, double* solp, double* __restrict__ rhs, const double* flux,
                                                   const __grid_constant__ HpDev h, const double* __restrict__ dt_ptr,
                                                   unsigned long long* max_slot, int stage, int write_rhs, int num_flux,
                                                   double bx, double by, double bz)
{
	extern __shared__ __align__(16) double sm[];
	const HpGroup& G = h.grp[hp_group_of(h, blockIdx.x)];
	const int n_s = G.n_s, n_c = G.n_c, n_fl = h.n_fl, nfm = h.nfc_max, E_b = G.E_b;
	const int Kx = (D * n_c + n_fl * nfm) | 1;
	const int e0 = (blockIdx.x - G.blk0) * E_b;
	const int ne = min(E_b, G.n_vol - e0);
	const double b[3] = {bx, by, bz};
	int4* sSide = reinterpret_cast<int4*>(sm);          // [E_b][n_fl]
	double* sU = sm + 2 * E_b * n_fl;                   // [E_b][NV][n_s]
	double* sX = sU + (size_t)E_b * NV * n_s;           // [E_b][NV][Kx]
	double* sO = sX + (size_t)E_b * NV * Kx;            // staged operators
	for (int i = threadIdx.x; i < ne * n_fl; i += blockDim.x) sSide[i] = G.side[(size_t)e0 * n_fl + i];
	for (int i = threadIdx.x; i < G.n_stage; i += blockDim.x) sO[i] = G.ops[i];
	const double* ops = G.n_stage ? sO : G.ops;
	grid_wait();
	for (int i = threadIdx.x; i < ne * NV * n_s; i += blockDim.x) {
		const int e = i / (NV * n_s), r = i - e * NV * n_s;
		sU[i] = sol[G.dof[e0 + e] + r];
	}
	__syncthreads();
	// 1. fluxes of the local faces, in the volume's own node order (negated on right sides), packed after the volume part
	for (int o = threadIdx.x; o < ne * n_fl * nfm; o += blockDim.x) {
		const int e = o / (n_fl * nfm), r = o - e * n_fl * nfm;
		const int lf = r / nfm, q = r - lf * nfm;
		const int4 t = sSide[e * n_fl + lf];
		const int side = (t.y >> 8) & 1, n_fc = t.y >> 16;
		if (q >= n_fc) continue;
		const int64_t off = side_offset(t);
		const double sgn = side ? -1.0 : 1.0;
		double* x = sX + (size_t)e * NV * Kx + t.x + q;
		if constexpr (OWN) {
			const int other = side ? h.nc_inv[off + q] : h.nc[off + q], ql = side ? other : q, qr = side ? q : other;
			double WL[NV], WR[NV], n[D], nf[NV];
#pragma unroll
			for (int v = 0; v < NV; ++v) {
				WL[v] = flux[2 * NV * off + (size_t)v * n_fc + ql];
				WR[v] = flux[2 * NV * off + (size_t)(NV + v) * n_fc + qr];
			}
#pragma unroll
			for (int a = 0; a < D; ++a) n[a] = h.nrm[(off + ql) * D + a];
			hp_numflux<D, NV>(WL, WR, n, h.jf[off + ql], num_flux, b, nf);
#pragma unroll
			for (int v = 0; v < NV; ++v) x[(size_t)v * Kx] = sgn * nf[v];
		} else {
			const int qs = side ? h.nc_inv[off + q] : q;
#pragma unroll
			for (int v = 0; v < NV; ++v) x[(size_t)v * Kx] = sgn * flux[NV * off + (size_t)v * n_fc + qs];
		}
	}
	// 2. per volume node: s = cv0_vs_vc sol_coef, the physical flux and the reference flux fr[eq][r] = sum_x m_{x r} f[x][eq]
	for (int o = threadIdx.x; o < ne * n_c; o += blockDim.x) {
		const int e = o / n_c, c = o - e * n_c;
		const size_t ve = (size_t)(e0 + e);
		double m[D][D], s[NV];
#pragma unroll
		for (int x = 0; x < D; ++x)
#pragma unroll
			for (int r = 0; r < D; ++r)
				m[x][r] = G.affine ? G.met[ve * D * D + x + D * r] : G.met[(ve * D * D + x + D * r) * n_c + c];
#pragma unroll
		for (int v = 0; v < NV; ++v) s[v] = 0.0;
		const double* u = sU + (size_t)e * NV * n_s;
#pragma unroll 4
		for (int k = 0; k < n_s; ++k) {
			const double a = ops[k * n_c + c];
#pragma unroll
			for (int v = 0; v < NV; ++v) s[v] = fma(a, u[v * n_s + k], s[v]);
		}
		double* x0 = sX + (size_t)e * NV * Kx + c;
		if constexpr (NV == D + 2) {
			double f[D][D + 2];
			flux_euler<D>(s, f);
#pragma unroll
			for (int eq = 0; eq < NV; ++eq)
#pragma unroll
				for (int r = 0; r < D; ++r) {
					double acc = 0.0;
#pragma unroll
					for (int x = 0; x < D; ++x) acc += m[x][r] * f[x][eq];
					x0[(size_t)eq * Kx + r * n_c] = acc;
				}
		} else {
#pragma unroll
			for (int r = 0; r < D; ++r) {
				double acc = 0.0;
#pragma unroll
				for (int x = 0; x < D; ++x) acc += m[x][r] * (b[x] * s[0]);
				x0[r * n_c] = acc;
			}
		}
	}
	__syncthreads();
	// 3. lift: R_i = sum_k Lv[k][i] X[k] + sum_lf sum_q Lf[p_f(lf)][lf n_fc + q][i] X[k0(lf) + q], one accumulator per variable;
	// 4. mass-matrix inverse, RK stage, norm
	const double dt = (stage >= 0 ? *dt_ptr : 0.0);
	double lmax = 0.0;
	auto finish = [&](int e, int v, int i, double r) {
		lmax = fmax(lmax, fabs(r));
		if (isnan(r)) lmax = r;
		const size_t gi = (size_t)G.dof[e0 + e] + (size_t)v * n_s + i;
		const double s0 = sU[((size_t)e * NV + v) * n_s + i];
		if (write_rhs) rhs[gi] = r;
		if (stage < 0) return;
		double un;
		if (stage == 0) { solp[gi] = s0; un = s0 + dt * r; }
		else if (stage == 1) un = (1.0 / 4.0) * (3.0 * solp[gi] + s0 + dt * r);
		else un = (1.0 / 3.0) * (solp[gi] + 2.0 * s0 + 2.0 * dt * r);
		sol[gi] = un;
	};
	auto lift = [&](int e, int i, double (&acc)[NV]) {
		const double* x = sX + (size_t)e * NV * Kx;
#pragma unroll
		for (int v = 0; v < NV; ++v) acc[v] = 0.0;
		auto part = [&](const double* l, const double* xp, int n) {
#pragma unroll 4
			for (int k = 0; k < n; ++k) {
				const double a = l[k * n_s];
#pragma unroll
				for (int v = 0; v < NV; ++v) acc[v] = fma(a, xp[(size_t)v * Kx + k], acc[v]);
			}
		};
		part(ops + n_s * n_c + i, x, D * n_c);
		for (int lf = 0; lf < n_fl; ++lf) {
			const int4 t = sSide[e * n_fl + lf];
			const int n_fc = t.y >> 16;
			part(ops + G.oL[t.y & 255] + (size_t)lf * n_fc * n_s + i, x + t.x, n_fc);
		}
	};
	if (G.affine) {
		for (int o = threadIdx.x; o < ne * n_s; o += blockDim.x) {
			const int e = o / n_s, i = o - e * n_s;
			const double ji = G.jinv[e0 + e];
			double acc[NV];
			lift(e, i, acc);
#pragma unroll
			for (int v = 0; v < NV; ++v) finish(e, v, i, acc[v] * ji);
		}
	} else {
		double* sR = sO + G.n_stage;   // [E_b][NV][n_s]
		for (int o = threadIdx.x; o < ne * n_s; o += blockDim.x) {
			const int e = o / n_s, i = o - e * n_s;
			double acc[NV];
			lift(e, i, acc);
#pragma unroll
			for (int v = 0; v < NV; ++v) sR[((size_t)e * NV + v) * n_s + i] = acc[v];
		}
		__syncthreads();
		for (int o = threadIdx.x; o < ne * NV * n_s; o += blockDim.x) {
			const int ev = o / n_s, i = o - ev * n_s, e = ev / NV;
			const double* mi = G.minv + (size_t)(e0 + e) * n_s * n_s + (size_t)i * n_s;
			double acc = 0.0;
			for (int j = 0; j < n_s; ++j) acc = fma(mi[j], sR[(size_t)ev * n_s + j], acc);
			finish(e, ev - e * NV, i, acc);
		}
	}
	for (int off = 16; off > 0; off >>= 1) {
		const double other = __shfl_xor_sync(0xffffffffu, lmax, off);
		lmax = (isnan(other) || other > lmax) ? other : lmax;
	}
	if ((threadIdx.x & 31) == 0) hp_atomic_max_abs(max_slot, lmax);
}

// Advection on affine elements: the volume part folded, a thread per coefficient (E_b n_s <= kHpThreads), the traces of the
// new state for the next stage at the end.  Everything that no kernel writes is loaded before the wait.
template <int D>
__global__ void __launch_bounds__(kHpThreads) k_hp_advect(double* sol, double* solp, double* __restrict__ rhs, const double* trace,
                                                          const __grid_constant__ HpDev h, const double* __restrict__ dt_ptr,
                                                          unsigned long long* max_slot, int stage, int write_rhs,
                                                          double* __restrict__ next, double bx, double by, double bz)
{
	extern __shared__ __align__(16) double sm[];
	const HpGroup& G = h.grp[hp_group_of(h, blockIdx.x)];
	const int n_s = G.n_s, n_fl = h.n_fl, nfm = h.nfc_max, E_b = G.E_b, Kx = (n_fl * nfm) | 1;
	const int e0 = (blockIdx.x - G.blk0) * E_b;
	const int ne = min(E_b, G.n_vol - e0), tid = threadIdx.x;
	const double b[3] = {bx, by, bz};
	int4* sSide = reinterpret_cast<int4*>(sm);          // [E_b][n_fl]
	double* sU = sm + 2 * E_b * n_fl;                   // [E_b][n_s]
	double* sV = sU + E_b * n_s;                        // [E_b][n_s] the new state
	double* sX = sV + E_b * n_s;                        // [E_b][Kx]
	double* sO = sX + E_b * Kx;                         // staged operators
	for (int i = tid; i < ne * n_fl; i += kHpThreads) sSide[i] = G.side[(size_t)e0 * n_fl + i];
	for (int i = tid; i < G.n_stage; i += kHpThreads) sO[i] = G.ops[i];
	const double* ops = G.n_stage ? sO : G.ops;
	const bool live = tid < ne * n_s;
	const int e = live ? tid / n_s : 0, i = tid - e * n_s;
	const int64_t gi = G.dof[e0 + e] + i;
	const double ji = G.jinv[e0 + e];
	double a[D];
#pragma unroll
	for (int r = 0; r < D; ++r) {
		a[r] = 0.0;
#pragma unroll
		for (int c = 0; c < D; ++c) a[r] += G.met[(size_t)(e0 + e) * D * D + c + D * r] * b[c];
	}
	__syncthreads();
	// fluxes of the local faces, in the volume's own node order, negated on right sides
	const int n_item = ne * n_fl * nfm;
	struct Node { int64_t l, r; int dst; double n[D], j; };
	auto node = [&](int o) {
		Node t;
		const int el = o / (n_fl * nfm), rem = o - el * n_fl * nfm, lf = rem / nfm, q = rem - lf * nfm;
		const int4 sd = sSide[el * n_fl + lf];
		const int side = (sd.y >> 8) & 1, n_fc = sd.y >> 16;
		t.dst = -1;
		if (q >= n_fc) return t;
		const int64_t off = side_offset(sd);
		const int other = side ? h.nc_inv[off + q] : h.nc[off + q], ql = side ? other : q;
		t.l = 2 * off + ql;
		t.r = 2 * off + n_fc + (side ? q : other);
		t.dst = el * Kx + sd.x + q;
#pragma unroll
		for (int c = 0; c < D; ++c) t.n[c] = h.nrm[(off + ql) * D + c];
		t.j = side ? -h.jf[off + ql] : h.jf[off + ql];
		return t;
	};
	Node t;
	t.dst = -1;
	if (tid < n_item) t = node(tid);
	grid_wait();
	const double u0 = live ? sol[gi] : 0.0, up = live && stage >= 1 ? solp[gi] : 0.0, dt = stage >= 0 ? *dt_ptr : 0.0;
	for (int o = tid; o < n_item; o += kHpThreads) {
		if (o != tid) t = node(o);
		if (t.dst >= 0) sX[t.dst] = numflux_upwind<D>(b, trace[t.l], trace[t.r], t.n) * t.j;
	}
	if (live) sU[tid] = u0;
	__syncthreads();
	double lmax = 0.0;
	if (live) {
		// sum_r (sum_x m_{x r} b_x) [lift_r Cv] u, then the faces
		double y[D], acc = 0.0;
#pragma unroll
		for (int r = 0; r < D; ++r) y[r] = 0.0;
		const double *u = sU + e * n_s, *l = ops + i;
#pragma unroll 4
		for (int k = 0; k < n_s; ++k)
#pragma unroll
			for (int r = 0; r < D; ++r) y[r] = fma(l[(r * n_s + k) * n_s], u[k], y[r]);
		for (int lf = 0; lf < n_fl; ++lf) {
			const int4 sd = sSide[e * n_fl + lf];
			const int n_fc = sd.y >> 16;
			const double *lp = ops + G.oL[sd.y & 255] + lf * n_fc * n_s + i, *x = sX + e * Kx + sd.x;
#pragma unroll 4
			for (int q = 0; q < n_fc; ++q) acc = fma(lp[q * n_s], x[q], acc);
		}
#pragma unroll
		for (int r = 0; r < D; ++r) acc = fma(a[r], y[r], acc);
		const double r = acc * ji;
		lmax = isnan(r) ? r : fabs(r);
		if (write_rhs) rhs[gi] = r;
		if (stage >= 0) {
			double un;
			if (stage == 0) { solp[gi] = u0; un = u0 + dt * r; }
			else if (stage == 1) un = (1.0 / 4.0) * (3.0 * up + u0 + dt * r);
			else un = (1.0 / 3.0) * (up + 2.0 * u0 + 2.0 * dt * r);
			sol[gi] = un;
			sV[tid] = un;
		}
	}
	for (int off = 16; off > 0; off >>= 1) {
		const double other = __shfl_xor_sync(0xffffffffu, lmax, off);
		lmax = (isnan(other) || other > lmax) ? other : lmax;
	}
	if ((tid & 31) == 0) hp_atomic_max_abs(max_slot, lmax);
	if (next) {
		__syncthreads();
		hp_traces<1>(sV, sSide, G, ops + G.n_tr0, n_fl, nfm, ne, next);
	}
}

// ------------------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------------------
template <typename T>
static int hp_upload(HpState* s, T** dst, const T* src, size_t n)
{
	void* p = nullptr;
	if (cudaMalloc(&p, (n ? n : 1) * sizeof(T)) != cudaSuccess) return DPG_ERR_CUDA;
	s->allocs.push_back(p);
	if (n && src && cudaMemcpy(p, src, n * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) return DPG_ERR_CUDA;
	*dst = (T*)p;
	return DPG_OK;
}

static HpState* hp_state(const dpg_gpu_ctx* c) { return (HpState*)(c->hp ? c->hp : c->adv); }

void hp_free(dpg_gpu_ctx* c)
{
	for (void** slot : {&c->hp, &c->adv}) {
		HpState* s = (HpState*)*slot;
		if (!s) continue;
		for (void* p : s->allocs) cudaFree(p);
		delete s;
		*slot = nullptr;
	}
}

template <int D, int NV>
static int hp_set_smem(const HpState* s)
{
	if (s->smem_trace > kSmemOptIn || s->smem_volume > kSmemOptIn) return DPG_ERR_CUDA;
	return allow_smem((const void*)k_hp_trace<NV>) && allow_smem((const void*)k_hp_volume<D, NV, false>) &&
	       allow_smem((const void*)k_hp_volume<D, NV, true>) && allow_smem((const void*)k_hp_advect<D>) ? DPG_OK : DPG_ERR_CUDA;
}

// share: null with mixed orders (c->hp); else the device tables of a context of one order that takes hp_step and
// hp_residual for its FP64 residuals (c->adv: advection, affine, periodic).
int hp_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim, const OzTables* share)
{
	const int d = sim->d, NV = sim->n_var, n_vol = sim->n_vol, n_face = sim->n_face;
	const int n_fl = sim->ops[0].n_fl;
	if (sim->n_ops > kHpMaxGroups || (!sim->face_p && !share)) return DPG_ERR_UNSUPPORTED;
	if (share && sim->ops[0].n_s > kHpThreads) return DPG_OK;
	HpState* s = new HpState();
	(share ? c->adv : c->hp) = s;
	HpDev& h = s->dev;
	h.n_fl = n_fl;
	for (int k = 0; k < sim->n_ops; ++k) h.n_fc[sim->ops[k].p] = sim->ops[k].n_fc;
	h.nfc_max = 0;
	for (int k = 0; k < sim->n_ops; ++k) h.nfc_max = std::max(h.nfc_max, sim->ops[k].n_fc);
	int rc;
	// groups: the volumes of each order present, in volume order
	std::vector<std::vector<int>> members(sim->n_ops);
	for (int v = 0; v < n_vol; ++v) members[sim->vol_ops[v]].push_back(v);
	bool folded = NV == 1;   // advection, every element affine: k_hp_advect
	for (int v = 0; v < n_vol; ++v) folded = folded && sim->vol_affine[v];
	for (int k = 0; k < sim->n_ops; ++k) folded = folded && sim->ops[k].n_s <= kHpThreads;
	s->folded = folded;
	size_t smem_t = 0, smem_v = 0;
	int blocks = 0;
	for (int k = sim->n_ops - 1; k >= 0; --k) {   // the highest order (the longest blocks) first
		if (members[k].empty()) continue;
		const dpg_element_ops& o = sim->ops[k];
		HpGroup& G = h.grp[h.n_groups++];
		G = HpGroup{};
		const int kv = folded ? 0 : d * o.n_c;   // first K of the face part in the lift
		G.p = o.p; G.n_vol = (int)members[k].size(); G.n_s = o.n_s; G.n_c = o.n_c;
		G.affine = 1;
		for (int v : members[k]) G.affine &= sim->vol_affine[v];
		std::vector<int64_t> dof;
		std::vector<int4> side;
		for (int v : members[k]) {
			dof.push_back(sim->vol_dof_off[v]);
			int k0 = kv;
			for (int lf = 0; lf < n_fl; ++lf) {
				const int f = sim->vol_face[v * DPG_NFL_MAX + lf], pf = dpg_face_order(sim, f), n_fc = h.n_fc[pf];
				const int64_t off = sim->face_geo_off[f];
				side.push_back(int4{k0, pf | sim->vol_face_side[v * DPG_NFL_MAX + lf] << 8 | n_fc << 16, (int)(uint32_t)off, (int)(uint32_t)(off >> 32)});
				k0 += n_fc;
			}
		}
		if (!share && (rc = hp_upload(s, (int**)&G.vols, members[k].data(), members[k].size()))) return rc;
		if ((rc = hp_upload(s, (int64_t**)&G.dof, dof.data(), dof.size()))) return rc;
		if ((rc = hp_upload(s, (int4**)&G.side, side.data(), side.size()))) return rc;
		// operators, K-major; lift [tw1 | -tw0[p_f]], times m_inv_ref for an affine group (the sums of the single-group
		// lift operator)
		std::vector<double> ops;
		auto push_lift = [&](int K, auto entry) {   // entry(i, k)
			for (int kk = 0; kk < K; ++kk)
				for (int i = 0; i < o.n_s; ++i) {
					double acc = 0.0;
					if (G.affine)
						for (int j = 0; j < o.n_s; ++j) acc += o.m_inv_ref[(size_t)i * o.n_s + j] * entry(j, kk);
					else
						acc = entry(i, kk);
					ops.push_back(acc);
				}
		};
		auto tw1 = [&](int i, int kk) { return o.tw1_vt_vc[((size_t)(kk / o.n_c) * o.n_s + i) * o.n_c + kk % o.n_c]; };
		if (folded)   // d n_s^2 multiply-adds instead of (d + 1) n_s n_c, n_c >= n_s
			push_lift(d * o.n_s, [&](int i, int kk) {
				double acc = 0.0;
				for (int cc = 0; cc < o.n_c; ++cc) acc += tw1(i, kk / o.n_s * o.n_c + cc) * o.cv0_vs_vc[(size_t)cc * o.n_s + kk % o.n_s];
				return acc;
			});
		else {
			for (int j = 0; j < o.n_s; ++j)
				for (int cc = 0; cc < o.n_c; ++cc) ops.push_back(o.cv0_vs_vc[(size_t)cc * o.n_s + j]);
			push_lift(d * o.n_c, tw1);
		}
		for (int pf = o.p; pf <= DPG_P_MAX; ++pf) {
			const double* tw = dpg_face_tw0(&o, pf);
			if (!dpg_face_cv0(&o, pf) || !tw) continue;
			const int n_fc = h.n_fc[pf];
			G.oL[pf] = (int)ops.size();
			push_lift(n_fl * n_fc, [&](int i, int kk) { return -tw[((size_t)(kk / n_fc) * o.n_s + i) * n_fc + kk % n_fc]; });
		}
		G.n_tr0 = (int)ops.size();
		for (int pf = o.p; pf <= DPG_P_MAX; ++pf) {
			const double* cf = dpg_face_cv0(&o, pf);
			if (!cf || !dpg_face_tw0(&o, pf)) continue;
			G.oT[pf] = (int)ops.size();
			for (int j = 0; j < o.n_s; ++j)
				for (int q = 0; q < n_fl * h.n_fc[pf]; ++q) ops.push_back(cf[(size_t)q * o.n_s + j]);
		}
		G.n_tr = (int)ops.size() - G.n_tr0;
		G.n_stage = ops.size() * sizeof(double) <= kHpStageBytes ? (int)ops.size() : 0;
		if ((rc = hp_upload(s, (double**)&G.ops, ops.data(), ops.size()))) return rc;
		const size_t per_v = sizeof(double) * (2 * n_fl + NV * (o.n_s + ((kv + n_fl * h.nfc_max) | 1) + (folded || !G.affine ? o.n_s : 0)));
		const size_t per_t = sizeof(double) * (2 * n_fl + NV * o.n_s);
		G.E_b = std::max(1, std::min({16, kHpThreads / o.n_s, (int)((96 * 1024) / per_v)}));
		// small meshes leave every SM a block (us per Euler step, 288 TRI 1..3: 109 -> 80; k_hp_advect has less work than
		// staging per volume: 288 TRI 4 23 -> 31)
		if (!folded) G.E_b = std::min(G.E_b, (n_vol + c->n_sm - 1) / c->n_sm);
		smem_t = std::max(smem_t, G.E_b * per_t + (G.n_stage ? G.n_tr : 0) * sizeof(double));
		smem_v = std::max(smem_v, G.E_b * per_v + G.n_stage * sizeof(double));
		G.blk0 = blocks;
		blocks += (G.n_vol + G.E_b - 1) / G.E_b;
		if (share) {
			G.met = share->met[k]; G.jinv = share->jinv[k];
			continue;
		}
		// geometry in group order
		std::vector<double> met, jinv, minv;
		for (int v : members[k]) {
			const double* m = &sim->metrics_vc[(size_t)sim->vol_geo_off[v] * d * d];
			if (G.affine) {
				for (int kk = 0; kk < d * d; ++kk) met.push_back(m[(size_t)o.n_c * kk]);
				jinv.push_back(1.0 / sim->jacobian_det_vc[sim->vol_geo_off[v]]);
			} else {
				met.insert(met.end(), m, m + (size_t)o.n_c * d * d);
				if (sim->vol_minv_off[v + 1] > sim->vol_minv_off[v]) {
					minv.insert(minv.end(), &sim->m_inv[sim->vol_minv_off[v]], &sim->m_inv[sim->vol_minv_off[v]] + (size_t)o.n_s * o.n_s);
				} else {
					const double jd = sim->jacobian_det_vc[sim->vol_geo_off[v]];
					for (int kk = 0; kk < o.n_s * o.n_s; ++kk) minv.push_back(o.m_inv_ref[kk] / jd);
				}
			}
		}
		if ((rc = hp_upload(s, (double**)&G.met, met.data(), met.size()))) return rc;
		if (G.affine) { if ((rc = hp_upload(s, (double**)&G.jinv, jinv.data(), jinv.size()))) return rc; }
		else if ((rc = hp_upload(s, (double**)&G.minv, minv.data(), minv.size()))) return rc;
	}
	h.n_blocks = blocks;
	s->blocks = blocks;
	s->smem_trace = smem_t;
	s->smem_volume = smem_v;
	const int64_t n_fnode = h.n_fnode = sim->face_geo_off[n_face];
	if (share) {
		h.nc = share->nc; h.nc_inv = share->nc_inv; h.nrm = share->nrm; h.jf = share->jf;
	} else {
		// volumes and faces
		std::vector<int> vf((size_t)n_vol * n_fl);
		for (int v = 0; v < n_vol; ++v)
			for (int lf = 0; lf < n_fl; ++lf)
				vf[(size_t)v * n_fl + lf] = (sim->vol_face[v * DPG_NFL_MAX + lf] << 1) | sim->vol_face_side[v * DPG_NFL_MAX + lf];
		std::vector<int> node_face((size_t)n_fnode), ncinv((size_t)n_fnode);
		for (int f = 0; f < n_face; ++f) {
			const int64_t off = sim->face_geo_off[f];
			for (int q = 0; q < sim->face_nfc[f]; ++q) {
				node_face[off + q] = f;
				ncinv[off + sim->nc_fc[off + q]] = q;
			}
		}
		if ((rc = hp_upload(s, (int64_t**)&h.dof_off, sim->vol_dof_off, (size_t)n_vol + 1))) return rc;
		if ((rc = hp_upload(s, (int**)&h.vol_face, vf.data(), vf.size()))) return rc;
		if ((rc = hp_upload(s, (int**)&h.face_p, sim->face_p, (size_t)n_face))) return rc;
		if ((rc = hp_upload(s, (int64_t**)&h.fnode_off, sim->face_geo_off, (size_t)n_face + 1))) return rc;
		if ((rc = hp_upload(s, (int**)&h.node_face, node_face.data(), node_face.size()))) return rc;
		if ((rc = hp_upload(s, (int**)&h.nc, sim->nc_fc, (size_t)n_fnode))) return rc;
		if ((rc = hp_upload(s, (int**)&h.nc_inv, ncinv.data(), ncinv.size()))) return rc;
		if ((rc = hp_upload(s, (double**)&h.nrm, sim->normals_fc, (size_t)n_fnode * d))) return rc;
		if ((rc = hp_upload(s, (double**)&h.jf, sim->jacobian_det_fc, (size_t)n_fnode))) return rc;
	}
	for (int k = 0; k < (folded ? 2 : 1); ++k)
		if ((rc = hp_upload(s, &s->trace[k], (const double*)nullptr, (size_t)2 * NV * n_fnode))) return rc;
	s->own = NV > 1 && n_fnode <= kOwnFaceNodes;
	if (NV > 1 && !s->own && (rc = hp_upload(s, &s->nnf, (const double*)nullptr, (size_t)NV * n_fnode))) return rc;
	if (d == 2 && NV == 1) return hp_set_smem<2, 1>(s);
	if (d == 3 && NV == 1) return hp_set_smem<3, 1>(s);
	if (d == 2 && NV == 4) return hp_set_smem<2, 4>(s);
	if (d == 3 && NV == 5) return hp_set_smem<3, 5>(s);
	return DPG_ERR_UNSUPPORTED;
}

OzTables hp_tables(const dpg_gpu_ctx* c, const struct dpg_sim* sim)
{
	const HpState* s = (const HpState*)c->hp;
	const HpDev& h = s->dev;
	OzTables t;
	t.n_groups = h.n_groups;
	for (int i = 0; i < h.n_groups; ++i)
		for (int k = 0; k < sim->n_ops; ++k)
			if (sim->ops[k].p == h.grp[i].p) { t.vols[k] = h.grp[i].vols; t.met[k] = h.grp[i].met; t.jinv[k] = h.grp[i].jinv; }
	t.dof_off = h.dof_off; t.vol_face = h.vol_face; t.face_p = h.face_p; t.fnode_off = h.fnode_off; t.node_face = h.node_face;
	t.nc = h.nc; t.nrm = h.nrm; t.jf = h.jf;
	return t;
}

// which: 0 traces, 1 face fluxes (Euler), 2 volumes; from, next: see hp_step.
template <int D, int NV>
static int hp_launch(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot, int from, bool next)
{
	HpState* s = hp_state(c);
	const HpDev& h = s->dev;
	if (which == 0) {
		launch_chained(k_hp_trace<NV>, s->blocks, kHpThreads, s->smem_trace, c->stream, c->sol, h, s->trace[0]);
	} else if (which == 1) {
		if constexpr (NV > 1) {
			const int64_t n = h.n_fnode;
			const int ft = spread_threads(n, c->n_sm);
			if (s->own) return DPG_OK;
			launch_chained(k_hp_face<D, NV>, (unsigned)((n + ft - 1) / ft), ft, 0, c->stream, s->trace[0], h, s->nnf, c->num_flux);
		}
	} else if (NV == 1 && s->folded) {
		launch_chained(k_hp_advect<D>, s->blocks, kHpThreads, s->smem_volume, c->stream, c->sol, c->solp, c->rhs, s->trace[from], h,
		               c->ddt, max_slot, stage, write_rhs ? 1 : 0, next ? s->trace[1 - from] : nullptr, c->b_adv[0], c->b_adv[1],
		               c->b_adv[2]);
	} else {
		const bool own = NV == 1 || s->own;
		launch_chained(own ? k_hp_volume<D, NV, true> : k_hp_volume<D, NV, false>, s->blocks, kHpThreads, s->smem_volume, c->stream,
		               c->sol, c->solp, c->rhs, own ? s->trace[0] : s->nnf, h, c->ddt, max_slot, stage, write_rhs ? 1 : 0, c->num_flux,
		               c->b_adv[0], c->b_adv[1], c->b_adv[2]);
	}
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

static int hp_launch_any(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot, int from, bool next)
{
	if (c->d == 2 && c->n_var == 1) return hp_launch<2, 1>(c, which, stage, write_rhs, max_slot, from, next);
	if (c->d == 3 && c->n_var == 1) return hp_launch<3, 1>(c, which, stage, write_rhs, max_slot, from, next);
	if (c->d == 2 && c->n_var == 4) return hp_launch<2, 4>(c, which, stage, write_rhs, max_slot, from, next);
	if (c->d == 3 && c->n_var == 5) return hp_launch<3, 5>(c, which, stage, write_rhs, max_slot, from, next);
	return DPG_ERR_UNSUPPORTED;
}

int hp_launch_part(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot)
{
	return hp_launch_any(c, which, stage, write_rhs, max_slot, 0, false);
}

int hp_residual(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot)
{
	int rc;
	if ((rc = hp_launch_part(c, 0, stage, write_rhs, max_slot))) return rc;
	if ((rc = hp_launch_part(c, 1, stage, write_rhs, max_slot))) return rc;
	return hp_launch_part(c, 2, stage, write_rhs, max_slot);
}

// Kernels of one residual.
int hp_launches(const dpg_gpu_ctx* c) { return c->n_var == 1 || hp_state(c)->own ? 2 : 3; }

// Whether hp_step may take the place of three stages.
bool hp_steps(const dpg_gpu_ctx* c) { return c->prec_mode == DPG_PREC_FP64 && hp_state(c) && hp_state(c)->folded; }

// One SSP-RK3 step, norms of the three residuals in max_slots[0..2]: the traces once, then a launch per stage.
int hp_step(dpg_gpu_ctx* c, unsigned long long* max_slots)
{
	int rc = hp_launch_any(c, 0, 0, false, max_slots, 0, false);
	for (int stage = 0; stage < 3 && !rc; ++stage) rc = hp_launch_any(c, 2, stage, false, max_slots + stage, stage & 1, stage < 2);
	return rc;
}

} // namespace dpg
