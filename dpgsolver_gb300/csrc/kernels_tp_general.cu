// Boundary faces and the BR2 Navier-Stokes terms on tensor-product meshes (QUAD, HEX, p = 1..4, straight or curved), FP64,
// in the collocated Gauss basis (tp_ops.cuh):
//
//   k_tp_volume (kWalls / kViscous) : values at the Gauss points, face traces (constructor_s_fc_interp_T,
//                 boundary_T.c:134-145), boundary states into the side-1 slots of boundary faces
//                 (constructor_Boundary_Value_fcl, face_solver_T.c:92-115; formulas in flux.cuh)
//   k_tp_grad   : BR2.  Volume gradient g_x = 1/detJ sum_r m_xr Ds_r u (constructor_grad_xyz_p: m_inv tw0_vt_vc (detJ
//                 d/dx) u); the faces' liftings m_inv tw0_vt_fc (J_f n_x (s_num - s)), s_num = (s_l + s_r) / 2
//                 (compute_grad_coef_faces, dg/compute_grad_coef_dg_T.c:214-285), one factor l(+-1) / (w detJ) per node;
//                 per local face node the normal second-order flux of this side at the partially corrected gradient
//                 g + 1.01 NFMAX the face's own lifting (constructor_partial_grad_fc_interp,
//                 compute_face_rlhs_dg_T.c:245-296), whose trace is the factor c_q = sum_j l_j^2 / (w_j detJ_j); a
//                 boundary face has the interior gradient on both sides (constructor_Boundary_Value_T_grad_from_internal);
//                 the volume flux at the fully corrected gradient and its weak divergence
//   k_tp_face_br2 : inviscid numerical flux + the mean of the two sides' normal second-order fluxes
//                 (numerical_flux_central_T.c:75-100), the energy component zero on adiabatic no-slip walls
//                 (set_provided_Numerical_Flux_members), times jacobian_det_fc
//   k_tp_lift   : kernels_tp.cu
//
// Four launches per Navier-Stokes residual, three for Euler with walls.  Every sum is formed by one thread in a fixed
// order.  Bound: the FP64 pipe (about 320 instructions per node in k_tp_grad, which runs at its rate).  64x128 annulus, QUAD
// p = 3, one residual: k_tp_volume 22, k_tp_grad 86, k_tp_face_br2 21, k_tp_lift 18 us, 146 us in all; the dense form with
// stored gradients (two passes of element mass-matrix inverses per face, six launches) took 957 us.
// T = double: the residual; T = dual: its tangent (fvn, the face fluxes and G then hold tangents only).
#include <vector>

#include "tp_volume.cuh"

namespace dpg {

using namespace tp;

template <class T> struct Ld;
template <> struct Ld<double> {
	static constexpr bool tan = false;
	__device__ __forceinline__ static double at(const double* a, const double*, size_t k) { return a[k]; }
	__device__ __forceinline__ static double out(double x) { return x; }
};
template <> struct Ld<dual> {
	static constexpr bool tan = true;
	__device__ __forceinline__ static dual at(const double* a, const double* t, size_t k) { return dual(a[k], t[k]); }
	__device__ __forceinline__ static double out(dual x) { return x.d; }
};

struct TpVisc {
	double mu, kappa, scale;
	const int* bc;        // [n_face] or null
	const int* nc;        // [n_face][n_fc]
	const double* nrm;    // [n_face][n_fc][d]
	const double* jf;     // [n_face][n_fc]
};

template <class T, int D, int NV, int N1>
static size_t smem_grad(int E)
{
	const size_t N = ipow(N1, D), NF = ipow(N1, D - 1);
	return sizeof(Ops<N1>) + sizeof(T) * E * ((1 + D) * NV * N + 2 * D * NV * NF) + sizeof(double) * E * (2 * D * NF * D + N);
}

template <class T, int D, int NV, int N1>
__global__ void __launch_bounds__(256) k_tp_grad(const double* Uc, const double* Uc_t,
                                                 const double* trace, const double* trace_t, TpGeo g,
                                                 TpVisc V, const __grid_constant__ Ops<N1> ops, double* __restrict__ fvn,
                                                 double* __restrict__ G, int E, TanStride ts)
{
	constexpr int N = ipow(N1, D), NF = ipow(N1, D - 1);
	extern __shared__ double sm[];
	Ops<N1>* so = reinterpret_cast<Ops<N1>*>(sm);
	T* sU = reinterpret_cast<T*>(sm + sizeof(Ops<N1>) / sizeof(double));   // [E][NV][N]
	T* sG = sU + (size_t)E * NV * N;               // [D][E][NV][N] gradients of the volume part, then reference fluxes
	T* sJ = sG + (size_t)E * D * NV * N;           // [E][2 D][NV][NF] J_f (u_num - u)
	double* sN = reinterpret_cast<double*>(sJ + (size_t)E * 2 * D * NV * NF);   // [E][2 D][D][NF] normals
	double* sD = sN + (size_t)E * 2 * D * D * NF;  // [E][N] 1 / detJ
	if constexpr (Ld<T>::tan) {
		Uc_t += blockIdx.y * ts.dof;
		trace_t += blockIdx.y * ts.tr;
		fvn += blockIdx.y * ts.tr;
		G += blockIdx.y * ts.dof;
	}
	const int e0 = blockIdx.x * E, ne = min(E, g.n_vol - e0);
	const int e = threadIdx.x / N, i = threadIdx.x - e * N;
	const bool live = e < ne;
	load_ops(so, ops);
	grid_wait();
	for (int k = threadIdx.x; k < ne * NV * N; k += blockDim.x) sU[k] = Ld<T>::at(Uc, Uc_t, (size_t)e0 * NV * N + k);
	double m[D][D], ji = 0.0;
	if (live) {
		ji = g.affine ? g.jinv[e0 + e] : g.jinv[(size_t)(e0 + e) * N + i];
		sD[e * N + i] = ji;
#pragma unroll
		for (int x = 0; x < D; ++x)
#pragma unroll
			for (int r = 0; r < D; ++r)
				m[x][r] = g.affine ? g.met[(size_t)(e0 + e) * D * D + x + D * r]
				                   : g.met[((size_t)(e0 + e) * D * D + x + D * r) * N + i];
	}
	// jumps to the central trace at the faces, in the element's own node order; with the normal of side 0 both sides have
	// the same product n (u_num - u)
	for (int o = threadIdx.x; o < ne * 2 * D * NF; o += blockDim.x) {
		const int ee = o / (2 * D * NF), k = o - ee * 2 * D * NF, lf = k / NF, q = k - lf * NF;
		const int vf = g.vol_face[(size_t)(e0 + ee) * 2 * D + lf];
		const size_t f = (size_t)(vf >> 1);
		const int side = vf & 1, ql = side ? g.nc_inv[f * NF + q] : q, qr = side ? q : V.nc[f * NF + q];
		const double jh = 0.5 * V.jf[f * NF + ql];
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			const T sl = Ld<T>::at(trace, trace_t, (2 * f * NV + w) * NF + ql);
			const T sr = Ld<T>::at(trace, trace_t, ((2 * f + 1) * NV + w) * NF + qr);
			sJ[((size_t)(ee * 2 * D + lf) * NV + w) * NF + q] = jh * (sr - sl);
		}
#pragma unroll
		for (int x = 0; x < D; ++x) sN[((size_t)(ee * 2 * D + lf) * D + x) * NF + q] = V.nrm[(f * NF + ql) * D + x];
	}
	__syncthreads();
	// volume gradient at this node
	T gx[D][NV];
	if (live) {
		double jm[D][D];
#pragma unroll
		for (int x = 0; x < D; ++x)
#pragma unroll
			for (int r = 0; r < D; ++r) jm[x][r] = ji * m[x][r];
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			T dr[D];
			auto along = [&](auto tag) {
				constexpr int A = decltype(tag)::value;
				const double* row = so->Ds + node_along<A, N1>(i) * N1;
				dr[A] = pencil_dot<A, N1>(row, sU + (e * NV + w) * N, pencil_base<A, N1>(i));
			};
			along(std::integral_constant<int, 0>{});
			along(std::integral_constant<int, 1>{});
			if constexpr (D == 3) along(std::integral_constant<int, 2>{});
#pragma unroll
			for (int x = 0; x < D; ++x) {
				T acc = jm[x][0] * dr[0];
#pragma unroll
				for (int r = 1; r < D; ++r) acc += jm[x][r] * dr[r];
				gx[x][w] = acc;
				sG[((size_t)(x * E + e) * NV + w) * N + i] = gx[x][w];
			}
		}
	}
	__syncthreads();
	// per local face node: the partially corrected gradient and this side's normal second-order flux
	for (int o = threadIdx.x; o < ne * 2 * D * NF; o += blockDim.x) {
		const int ee = o / (2 * D * NF), k = o - ee * 2 * D * NF, lf = k / NF, q = k - lf * NF, a = lf >> 1;
		const int vf = g.vol_face[(size_t)(e0 + ee) * 2 * D + lf];
		const double* l = (lf & 1) ? so->lp : so->lm;
		const double* lw = (lf & 1) ? so->lwp : so->lwm;
		const int S = stride_of<N1>(a), base = face_base<N1>(a, q);
		double cq = 0.0, n[D];
#pragma unroll
		for (int j = 0; j < N1; ++j) cq = fma(lw[j], sD[ee * N + base + j * S], cq);
		cq *= V.scale;
#pragma unroll
		for (int x = 0; x < D; ++x) n[x] = sN[((size_t)(ee * 2 * D + lf) * D + x) * NF + q];
		T gq[D][NV], W[NV];
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			const T J = cq * sJ[((size_t)(ee * 2 * D + lf) * NV + w) * NF + q];
#pragma unroll
			for (int x = 0; x < D; ++x) {
				const T* y = sG + ((size_t)(x * E + ee) * NV + w) * N + base;
				T acc = l[0] * y[0];
#pragma unroll
				for (int j = 1; j < N1; ++j) acc += l[j] * y[j * S];
				gq[x][w] = acc + n[x] * J;
			}
			W[w] = Ld<T>::at(trace, trace_t, ((size_t)vf * NV + w) * NF + q);
		}
		auto emit = [&](int slot) {
			T F[NV];
			flux_viscous_normal<D>(V.mu, V.kappa, W, gq, n, F);
#pragma unroll
			for (int w = 0; w < NV; ++w) fvn[((size_t)slot * NV + w) * NF + q] = Ld<T>::out(F[w]);
		};
		emit(vf);
		if (V.bc && V.bc[vf >> 1]) {   // boundary face: the boundary state with the interior gradient
#pragma unroll
			for (int w = 0; w < NV; ++w) W[w] = Ld<T>::at(trace, trace_t, ((size_t)(vf + 1) * NV + w) * NF + q);
			emit(vf + 1);
		}
	}
	// fully corrected gradient, volume flux
	T fr[D][NV];
	if (live) {
		auto lift = [&](auto tag) {
			constexpr int A = decltype(tag)::value;
			const int ia = node_along<A, N1>(i), q = face_node<A, N1>(i);
#pragma unroll
			for (int sd = 0; sd < 2; ++sd) {
				const int lf = 2 * A + sd;
				const double c = ji * (sd ? so->wp[ia] : so->wm[ia]);
				double cn[D];
#pragma unroll
				for (int x = 0; x < D; ++x) cn[x] = c * sN[((size_t)(e * 2 * D + lf) * D + x) * NF + q];
#pragma unroll
				for (int w = 0; w < NV; ++w) {
					const T J = sJ[((size_t)(e * 2 * D + lf) * NV + w) * NF + q];
#pragma unroll
					for (int x = 0; x < D; ++x) gx[x][w] += cn[x] * J;
				}
			}
		};
		lift(std::integral_constant<int, 0>{});
		lift(std::integral_constant<int, 1>{});
		if constexpr (D == 3) lift(std::integral_constant<int, 2>{});
		T s[NV], F[D][NV];
#pragma unroll
		for (int w = 0; w < NV; ++w) s[w] = sU[(e * NV + w) * N + i];
		flux_viscous<D>(V.mu, V.kappa, s, gx, F);
		auto met = [&](int x, int r) { return m[x][r]; };
		ref_flux<D, NV>(s, met, (const double*)nullptr, [&](int r, const T (&f)[NV]) {
#pragma unroll
			for (int w = 0; w < NV; ++w) {
				T acc = f[w];
				if (w > 0) {
#pragma unroll
					for (int x = 0; x < D; ++x) acc += m[x][r] * F[x][w];
				}
				fr[r][w] = acc;
			}
		});
	}
	__syncthreads();   // every face has read the gradients
	if (live) {
#pragma unroll
		for (int r = 0; r < D; ++r)
#pragma unroll
			for (int w = 0; w < NV; ++w) sG[((size_t)(r * E + e) * NV + w) * N + i] = fr[r][w];
	}
	__syncthreads();
	if (live) {
#pragma unroll
		for (int w = 0; w < NV; ++w) {
			double acc = 0.0;
			auto add = [&](auto tag) {
				constexpr int A = decltype(tag)::value;
				const double* row = so->Dw + node_along<A, N1>(i) * N1;
				const T* x = sG + ((size_t)(A * E + e) * NV + w) * N + pencil_base<A, N1>(i);
#pragma unroll
				for (int j = 0; j < N1; ++j) acc = fma(row[j], Ld<T>::out(x[j * ipow(N1, A)]), acc);
			};
			add(std::integral_constant<int, 0>{});
			add(std::integral_constant<int, 1>{});
			if constexpr (D == 3) add(std::integral_constant<int, 2>{});
			G[((size_t)(e0 + e) * NV + w) * N + i] = acc;
		}
	}
}

template <class T, int D, int NV>
__global__ void __launch_bounds__(128) k_tp_face_br2(const double* trace, const double* trace_t,
                                                     const double* fvn, TpVisc V, int n_face, int n_fc,
                                                     int num_flux, double* __restrict__ nnf, TanStride ts)
{
	if constexpr (Ld<T>::tan) {
		trace_t += blockIdx.y * ts.tr;
		fvn += blockIdx.y * ts.tr;
		nnf += blockIdx.y * ts.nf;
	}
	grid_wait();
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= n_face * n_fc) return;
	const int f = t / n_fc, q = t - f * n_fc, qr = V.nc[t];
	const size_t iL = (size_t)(2 * f) * NV * n_fc + q, iR = (size_t)(2 * f + 1) * NV * n_fc + qr;
	T WL[NV], WR[NV], nf[NV];
	double n[D];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		WL[v] = Ld<T>::at(trace, trace_t, iL + (size_t)v * n_fc);
		WR[v] = Ld<T>::at(trace, trace_t, iR + (size_t)v * n_fc);
	}
#pragma unroll
	for (int a = 0; a < D; ++a) n[a] = V.nrm[(size_t)t * D + a];
	const double h = 0.5 * V.jf[t];
	if (num_flux == DPG_NUM_FLUX_ROE_PIKE) numflux_roe_pike_rs<D>(WL, WR, n, h, nf);
	else                                   numflux_lax_friedrichs_rs<D>(WL, WR, n, h, nf);
	const bool adiabatic = V.bc && V.bc[f] == DPG_BC_NOSLIP_ADIABATIC;
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		double y = Ld<T>::out(nf[v]) + h * (fvn[iL + (size_t)v * n_fc] + fvn[iR + (size_t)v * n_fc]);
		if (v == D + 1 && adiabatic) y = 0.0;   // prescribed: no energy flux through the wall
		nnf[((size_t)f * NV + v) * n_fc + q] = y;
	}
}

// ------------------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------------------
template <int D, int NV, int N1>
static int configure_general(dpg_gpu_ctx* c)
{
	constexpr int E = most_elems(ipow(N1, D));
	constexpr cudaFuncAttribute A = cudaFuncAttributeMaxDynamicSharedMemorySize;
	const int sv = (int)smem_volume<D, NV, N1, false>(E), st = (int)smem_volume<D, NV, N1, true>(E);
	if (cudaFuncSetAttribute(k_tp_volume<D, NV, N1, false, kWalls>, A, sv) || cudaFuncSetAttribute(k_tp_volume<D, NV, N1, true, kWalls>, A, st))
		return DPG_ERR_CUDA;
	if constexpr (NV == D + 2) {
		if (cudaFuncSetAttribute(k_tp_volume<D, NV, N1, false, kViscous>, A, sv) ||
		    cudaFuncSetAttribute(k_tp_volume<D, NV, N1, true, kViscous>, A, st) ||
		    cudaFuncSetAttribute(k_tp_grad<double, D, NV, N1>, A, (int)smem_grad<double, D, NV, N1>(E)) ||
		    cudaFuncSetAttribute(k_tp_grad<dual, D, NV, N1>, A, (int)smem_grad<dual, D, NV, N1>(E)))
			return DPG_ERR_CUDA;
	}
	return DPG_OK;
}

// What comes before the lift, of the state u (w null) or its tangents along v[nb][n_dof]: the traces and boundary states with
// the weak divergence or the collocated values (kFront), then (the gradients and) the face fluxes (kFluxes).
enum { kFront = 1, kFluxes = 2 };

template <int D, int NV, int N1>
static int before_lift(dpg_gpu_ctx* c, const double* u, const double* v, const TanWork* w, int parts)
{
	const TpState* st = (const TpState*)c->tp;
	constexpr int N = ipow(N1, D);
	const TpGeo geo = geo_of(c);
	const int E = st->E, n_blk = (geo.n_vol + E - 1) / E, threads = (E * N + 31) / 32 * 32;
	const dim3 grid(n_blk, w ? w->nb : 1);
	const Ops<N1> ops = ops_of<N1>(st);
	const TanStride ts = tan_stride(c);
	if (parts & kFront) {
		const TpBc B{st->bc, st->xyz, c->fc.nrm, st->bp};
		auto go = [&](auto kernel, size_t smem, double* G, double* G_t) {
			launch_chained(kernel, grid, threads, smem, c->stream, u, v, geo, B, ops, c->trace, w ? w->trace_t : nullptr, G, G_t, E,
			               c->b_adv[0], c->b_adv[1], c->b_adv[2], ts);
		};
		const size_t sm_v = smem_volume<D, NV, N1, false>(E), sm_t = smem_volume<D, NV, N1, true>(E);
		if constexpr (NV == D + 2) {
			if (st->viscous && w) go(k_tp_volume<D, NV, N1, true, kViscous>, sm_t, st->Uc, w->Uc_t);
			else if (st->viscous) go(k_tp_volume<D, NV, N1, false, kViscous>, sm_v, st->Uc, nullptr);
		}
		if (!st->viscous && w) go(k_tp_volume<D, NV, N1, true, kWalls>, sm_t, w->G, nullptr);
		else if (!st->viscous) go(k_tp_volume<D, NV, N1, false, kWalls>, sm_v, st->G, nullptr);
	}
	if (cudaGetLastError() != cudaSuccess) return DPG_ERR_CUDA;
	if (!(parts & kFluxes)) return DPG_OK;
	if (!st->viscous) return w ? launch_face_tan(c, *w) : launch_face(c);
	if constexpr (NV == D + 2) {
		const TpVisc V{st->mu, st->kappa, st->scale, st->bc, c->fc.nc, c->fc.nrm, c->fc.jf};
		const int64_t nq = (int64_t)c->fc.n_face * c->fc.n_fc;
		const int ft = spread_threads(nq * (w ? w->nb : 1), c->n_sm), n_fb = (int)((nq + ft - 1) / ft);
		if (w) {
			launch_chained(k_tp_grad<dual, D, NV, N1>, grid, threads, smem_grad<dual, D, NV, N1>(E), c->stream, st->Uc, w->Uc_t,
			               c->trace, w->trace_t, geo, V, ops, w->fvn, w->G, E, ts);
			launch_chained(k_tp_face_br2<dual, D, NV>, dim3(n_fb, w->nb), ft, 0, c->stream, c->trace, w->trace_t, w->fvn, V,
			               c->fc.n_face, c->fc.n_fc, c->num_flux, w->nnf_t, ts);
		} else {
			launch_chained(k_tp_grad<double, D, NV, N1>, grid, threads, smem_grad<double, D, NV, N1>(E), c->stream, st->Uc, nullptr,
			               c->trace, nullptr, geo, V, ops, st->fvn, st->G, E, ts);
			launch_chained(k_tp_face_br2<double, D, NV>, n_fb, ft, 0, c->stream, c->trace, nullptr, st->fvn, V, c->fc.n_face,
			               c->fc.n_fc, c->num_flux, c->nnf, ts);
		}
		return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
	}
	return DPG_ERR_UNSUPPORTED;
}

static int before_lift_any(dpg_gpu_ctx* c, const double* u, const double* v, const TanWork* w, int parts)
{
	DPG_TP_DISPATCH(before_lift, c, u, v, w, parts);
}
static int configure_general_any(dpg_gpu_ctx* c) { DPG_TP_DISPATCH(configure_general, c); }

int tp_general_front(dpg_gpu_ctx* c) { return before_lift_any(c, c->sol, nullptr, nullptr, kFront); }
int tp_general_fluxes(dpg_gpu_ctx* c) { return before_lift_any(c, c->sol, nullptr, nullptr, kFluxes); }

int tp_general_residual(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot)
{
	const int rc = before_lift_any(c, c->sol, nullptr, nullptr, kFront | kFluxes);
	return rc ? rc : tp_lift(c, stage, write_rhs, max_slot);
}

int tp_general_jvp(dpg_gpu_ctx* c, const double* u, const double* v, double* out, const TanWork& w)
{
	const int rc = before_lift_any(c, u, v, &w, kFront | kFluxes);
	return rc ? rc : tp_lift_tan(c, w, out);
}

int tp_general_launches(dpg_gpu_ctx* c) { return 3 + (((const TpState*)c->tp)->viscous ? 1 : 0); }

// Boundary conditions and viscous terms of a tensor-product context (after tp_prepare).
int tp_general_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim)
{
	TpState* st = (TpState*)c->tp;
	const int d = sim->d, n_face = sim->n_face, n_fc = sim->ops[0].n_fc;
	auto put = [&](void** dst, const void* src, size_t bytes) {
		void* p = nullptr;
		if (cudaMalloc(&p, bytes ? bytes : 8) != cudaSuccess) return (int)DPG_ERR_CUDA;
		st->allocs.push_back(p);
		*dst = p;
		return src && cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess ? (int)DPG_ERR_CUDA : (int)DPG_OK;
	};
	int rc;
	std::vector<int> bc(n_face, 0);
	bool any = false;
	for (int f = 0; f < n_face; ++f)
		if (sim->face_vol[2 * f + 1] < 0) { bc[f] = sim->face_bc[f]; any = true; }
	if (any) {
		std::vector<double> xyz((size_t)n_face * n_fc * d);
		for (int f = 0; f < n_face; ++f)
			for (int q = 0; q < n_fc; ++q)
				for (int a = 0; a < d; ++a)
					xyz[((size_t)f * n_fc + q) * d + a] = sim->xyz_fc[(size_t)sim->face_geo_off[f] * d + q + (size_t)n_fc * a];
		if ((rc = put((void**)&st->bc, bc.data(), sizeof(int) * bc.size()))) return rc;
		if ((rc = put((void**)&st->xyz, xyz.data(), sizeof(double) * xyz.size()))) return rc;
	}
	st->bp.omega = sim->bc_omega; st->bp.rho_b = sim->bc_rho; st->bp.E_b = sim->bc_E;
	for (int k = 0; k < 5; ++k) st->bp.ext[k] = sim->bc_state[k];
	if (sim->pde_index == DPG_PDE_NAVIER_STOKES) {
		if (c->n_var != d + 2) return DPG_ERR_UNSUPPORTED;
		st->viscous = 1;
		st->mu = sim->mu;
		st->kappa = DPG_GAMMA_D * sim->mu / sim->Pr;
		st->scale = 1.01 * 2 * d;
		if ((rc = put((void**)&st->Uc, nullptr, sizeof(double) * c->n_dof))) return rc;
		if ((rc = put((void**)&st->fvn, nullptr, sizeof(double) * (size_t)n_face * 2 * c->n_var * n_fc))) return rc;
	}
	return configure_general_any(c);
}

} // namespace dpg
