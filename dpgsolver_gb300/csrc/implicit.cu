// Implicit path: matrix-free Newton-GMRES with pseudo-transient continuation, on the GPU.
//
// Follows solve_implicit / implicit_step (solve_implicit.c:95-110, 232-256): at each Newton step the system
//     (I / dtau - dF/du) du = F(u),      F(u) = m_inv * rhs(u)  (the residual of dpg_gpu_compute_rhs)
// is solved and u += du, until ||F||_inf < tol (the reference's exit rule max_rhs < exit_tol_i).  The reference
// assembles the full Jacobian into a PETSc matrix and adds -M/dt on the diagonal (compute_CFL_ramping,
// dg/solve_dg.c:223-248); here the same system, left-scaled by m_inv, is solved matrix-free:
//   - Jacobian-vector products are finite differences of the residual kernels (the same kernels as the explicit
//     path, in the context's precision mode);
//   - GMRES(m) with right preconditioning and classical Gram-Schmidt with one re-orthogonalisation; the Krylov
//     residual decides convergence;
//   - preconditioners: none, block-Jacobi (the element-diagonal blocks of I/dtau - dF/du assembled by
//     finite-difference probing over an element colouring in which no two face neighbours share a colour, then
//     factorised by a batched LU with partial pivoting), the learned block inverse (mlp.cu), or block ILU(0) in
//     its diagonal form (below: the diagonal and face-neighbour blocks, probed over a distance-2 colouring, with
//     level-scheduled factorisation and triangular solves) -- the GPU counterpart of the reference's default
//     PETSc method, GMRES(60) + ILU(1) with rtol 1e-4 (external/petsc/options_files/petsc_options_gmres_default.txt);
//   - dtau follows switched evolution relaxation: dtau_k = dtau_0 * ||F_0|| / ||F_k||.
// All vectors stay on the device; reductions are two-pass and deterministic.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "dpg_gpu_internal.cuh"

namespace dpg {

// ------------------------------------------------------------------------------------------------------------
// vector kernels
// ------------------------------------------------------------------------------------------------------------
constexpr int kRedBlocks = 304;   // 2 x 152 SMs
constexpr int kRedThreads = 256;

__global__ void k_axpby(int64_t n, double a, const double* __restrict__ x, double b, double* __restrict__ y)
{
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
		y[i] = a * x[i] + b * y[i];
}

__global__ void k_lincomb3(int64_t n, double a, const double* __restrict__ x, double b, const double* __restrict__ y,
                           double* __restrict__ z)
{
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
		z[i] = a * x[i] + b * y[i];
}

constexpr int kDotChunk = 8;   // vectors per block of a multi-vector dot product
// Sums over the lanes of eight values; lane l returns the value 4 (l >> 4) + 2 ((l >> 3) & 1) + ((l >> 2) & 1).  9 FP64
// additions instead of 40; each value's tree is the one of eight separate butterflies.
__device__ __forceinline__ double warp_sum8(const double (&v)[8], int lane)
{
	double a[4], b[2];
	const bool h = lane & 16, q = lane & 8, e = lane & 4;
#pragma unroll
	for (int k = 0; k < 4; ++k) a[k] = (h ? v[k + 4] : v[k]) + __shfl_xor_sync(0xffffffffu, h ? v[k] : v[k + 4], 16);
#pragma unroll
	for (int k = 0; k < 2; ++k) b[k] = (q ? a[k + 2] : a[k]) + __shfl_xor_sync(0xffffffffu, q ? a[k] : a[k + 2], 8);
	double s = (e ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, e ? b[0] : b[1], 4);
	s += __shfl_xor_sync(0xffffffffu, s, 2);
	s += __shfl_xor_sync(0xffffffffu, s, 1);
	return s;
}

// partial[k * gridDim.x + block] = this block's part of V_k . w, eight vectors k per block (blockIdx.y).  With jz: w =
// shift z - jz first (the product with the pseudo-transient matrix), written by the blocks of the first eight vectors.
__global__ void __launch_bounds__(kRedThreads) k_multidot_partial(int64_t n, int nv, const double* __restrict__ V, int64_t ld,
                                                                  double* w, double* __restrict__ partial, int nb = 1,
                                                                  const double* __restrict__ shift = nullptr,
                                                                  const double* __restrict__ z = nullptr,
                                                                  const double* __restrict__ jz = nullptr)
{
	__shared__ double red[kRedThreads / 32][kDotChunk];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k0 = blockIdx.y * kDotChunk;
	double acc[kDotChunk];
#pragma unroll
	for (int k = 0; k < kDotChunk; ++k) acc[k] = 0.0;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		double wi;
		if (jz) {
			wi = shift[i / nb] * z[i] - jz[i];
			if (blockIdx.y == 0) w[i] = wi;
		} else {
			wi = w[i];
		}
#pragma unroll
		for (int k = 0; k < kDotChunk; ++k)
			if (k0 + k < nv) acc[k] += V[(k0 + k) * ld + i] * wi;
	}
	const double v = warp_sum8(acc, lane);
	if ((lane & 3) == 0) red[warp][4 * (lane >> 4) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1)] = v;
	__syncthreads();
	if (threadIdx.x < kDotChunk && k0 + (int)threadIdx.x < nv) {
		double s = 0.0;
		for (int wv = 0; wv < kRedThreads / 32; ++wv) s += red[wv][threadIdx.x];
		partial[(int64_t)(k0 + threadIdx.x) * gridDim.x + blockIdx.x] = s;
	}
}

// Orthogonalisation of small systems (at most 32 blocks of one element per thread): each block sums the partial dot
// products itself, so a Gram-Schmidt pass is two launches instead of three and the norm comes with the second pass
// (10 -> 5 small launches per Krylov iteration; their chain, not their work, bounds such a system).  The sums are those of
// k_reduce_partials: lane p holds block p's part.
//   h_k = sum of the parts of V_k . w;  w -= sum_k V_k h_k;  norm_partial (may be null): this block's part of w . w
constexpr int kSmallBlocks = 32;
__global__ void __launch_bounds__(kRedThreads) k_gs_pass(int64_t n, int nv, const double* __restrict__ V, int64_t ld,
                                                         const double* __restrict__ partial, double* __restrict__ h,
                                                         double* __restrict__ w, double* __restrict__ norm_partial)
{
	extern __shared__ double sh[];   // [nv] h
	__shared__ double red[kRedThreads / 32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, np = gridDim.x;
	for (int k0 = 8 * warp; k0 < nv; k0 += 8 * (kRedThreads / 32)) {
		double p[8];
#pragma unroll
		for (int k = 0; k < 8; ++k) p[k] = (lane < np && k0 + k < nv) ? partial[(int64_t)(k0 + k) * np + lane] : 0.0;
		const double s = warp_sum8(p, lane);
		const int k = k0 + 4 * (lane >> 4) + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1);
		if ((lane & 3) == 0 && k < nv) {
			sh[k] = s;
			if (blockIdx.x == 0) h[k] = s;
		}
	}
	__syncthreads();
	const int64_t i = blockIdx.x * (int64_t)kRedThreads + threadIdx.x;
	double wi = 0.0;
	if (i < n) {
		double s = 0.0;
#pragma unroll 8
		for (int k = 0; k < nv; ++k) s += V[k * ld + i] * sh[k];
		wi = w[i] - s;
		w[i] = wi;
	}
	if (!norm_partial) return;
	double v = wi * wi;
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	if (lane == 0) red[warp] = v;
	__syncthreads();
	if (threadIdx.x == 0) {
		double s = 0.0;
		for (int wv = 0; wv < kRedThreads / 32; ++wv) s += red[wv];
		norm_partial[blockIdx.x] = s;
	}
}

// h[i] += h2[i] (the two passes), h[j + 1] = ||w|| from its blocks' parts, w /= ||w|| when positive
__global__ void __launch_bounds__(kRedThreads) k_gs_finish(int64_t n, int j, const double* __restrict__ norm_partial,
                                                           double* __restrict__ h, const double* __restrict__ h2,
                                                           double* __restrict__ w)
{
	const int lane = threadIdx.x & 31;
	double v = lane < (int)gridDim.x ? norm_partial[lane] : 0.0;
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	const double norm = sqrt(fmax(v, 0.0));
	if (blockIdx.x == 0) {
		for (int i = threadIdx.x; i <= j; i += blockDim.x) h[i] += h2[i];
		if (threadIdx.x == 0) h[j + 1] = norm;
	}
	const int64_t i = blockIdx.x * (int64_t)kRedThreads + threadIdx.x;
	if (i < n && norm > 0.0) w[i] *= 1.0 / norm;
}

__global__ void k_reduce_partials(int nv, int nparts, const double* __restrict__ partial, double* __restrict__ out)
{
	const int k = blockIdx.x;
	if (k >= nv) return;
	__shared__ double red[32];
	double s = 0.0;
	for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += partial[(int64_t)k * nparts + i];
	for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.0;
		for (int i = 0; i < (int)(blockDim.x / 32); ++i) t += red[i];
		out[k] = t;
	}
}

// w -= sum_k V_k h_k   (h on the device)
__global__ void k_sub_combination(int64_t n, int nv, const double* __restrict__ V, int64_t ld,
                                  const double* __restrict__ h, double* __restrict__ w)
{
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		double s = 0.0;
		for (int k = 0; k < nv; ++k) s += V[k * ld + i] * h[k];
		w[i] -= s;
	}
}

// Arnoldi column j on the device: h[i] += h2[i] (the two Gram-Schmidt passes) and h[j+1] = ||w|| from h2[j+1] = w.w
__global__ void k_column_finish(int j, double* __restrict__ h, const double* __restrict__ h2)
{
	for (int i = threadIdx.x; i <= j; i += blockDim.x) h[i] += h2[i];
	if (threadIdx.x == 0) h[j + 1] = sqrt(fmax(h2[j + 1], 0.0));
}

// w /= *s when *s > 0 (the norm stays on the device)
__global__ void k_scale_inv(int64_t n, double* __restrict__ w, const double* __restrict__ s)
{
	const double v = *s;
	if (!(v > 0.0)) return;
	const double inv = 1.0 / v;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) w[i] *= inv;
}

// x += sum_k Z_k y_k
__global__ void k_add_combination(int64_t n, int nv, const double* __restrict__ Z, int64_t ld,
                                  const double* __restrict__ y, double* __restrict__ x)
{
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		double s = 0.0;
		for (int k = 0; k < nv; ++k) s += Z[k * ld + i] * y[k];
		x[i] += s;
	}
}

__global__ void k_absmax_partial(int64_t n, const double* __restrict__ x, double* __restrict__ partial)
{
	__shared__ double red[32];
	double m = 0.0;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const double v = fabs(x[i]);
		m = (v > m || isnan(v)) ? v : m;
	}
	for (int o = 16; o > 0; o >>= 1) {
		const double v = __shfl_xor_sync(0xffffffffu, m, o);
		m = (v > m || isnan(v)) ? v : m;
	}
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.0;
		for (int i = 0; i < (int)(blockDim.x / 32); ++i) t = (red[i] > t || isnan(red[i])) ? red[i] : t;
		partial[blockIdx.x] = t;
	}
}

// ------------------------------------------------------------------------------------------------------------
// block-Jacobi: probing, LU, solve
// ------------------------------------------------------------------------------------------------------------
// u_dst = u_src with eps added to local dof j of every element of colour `col`
__global__ void k_perturb(int n_vol, int nb, const double* __restrict__ u_src, double* __restrict__ u_dst,
                          const int* __restrict__ colour, int col, int j, double eps)
{
	const int64_t n = (int64_t)n_vol * nb;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const int e = (int)(i / nb), k = (int)(i - (int64_t)e * nb);
		u_dst[i] = u_src[i] + ((k == j && colour[e] == col) ? eps : 0.0);
	}
}

// B_e[k][j] = shift_e * delta_kj - (F1_e[k] - F0_e[k]) / eps for the elements of colour `col` (shift_e = 1/dtau_e)
__global__ void k_extract_column(int n_vol, int nb, const double* __restrict__ F1, const double* __restrict__ F0,
                                 const int* __restrict__ colour, int col, int j, double inv_eps,
                                 const double* __restrict__ shift, double* __restrict__ blocks)
{
	const int64_t n = (int64_t)n_vol * nb;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const int e = (int)(i / nb), k = (int)(i - (int64_t)e * nb);
		if (colour[e] != col) continue;
		blocks[((int64_t)e * nb + k) * nb + j] = (k == j ? shift[e] : 0.0) - (F1[i] - F0[i]) * inv_eps;
	}
}

// Probe directions p0 .. p0 + gridDim.y - 1 of the tangent probing, V[b][n]: probe p = colour * nb + j is e_j on every
// element of the colour.
__global__ void k_probe_directions(int n_vol, int nb, const int* __restrict__ colour, int p0, double* __restrict__ V)
{
	const int64_t n = (int64_t)n_vol * nb;
	const int col = (p0 + (int)blockIdx.y) / nb, j = (p0 + (int)blockIdx.y) % nb;
	double* dst = V + blockIdx.y * n;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const int e = (int)(i / nb), k = (int)(i - (int64_t)e * nb);
		dst[i] = (k == j && colour[e] == col) ? 1.0 : 0.0;
	}
}

// The block columns of those probes from their products JV[b][n] (nbr null: diagonal blocks only)
__global__ void k_extract_probes(int n_vol, int nb, int n_fl, const double* __restrict__ JV, const int* __restrict__ colour,
                                 const int* __restrict__ nbr, int p0, const double* __restrict__ shift,
                                 double* __restrict__ diag, double* __restrict__ offd)
{
	const int64_t n = (int64_t)n_vol * nb;
	const int col = (p0 + (int)blockIdx.y) / nb, j = (p0 + (int)blockIdx.y) % nb;
	const double* src = JV + blockIdx.y * n;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const int e = (int)(i / nb), k = (int)(i - (int64_t)e * nb);
		if (colour[e] == col) {
			diag[((int64_t)e * nb + k) * nb + j] = (k == j ? shift[e] : 0.0) - src[i];
			continue;
		}
		if (!nbr) continue;
		for (int s = 0; s < n_fl; ++s) {
			const int o = nbr[e * n_fl + s];
			if (o >= 0 && colour[o] == col) offd[(((int64_t)e * n_fl + s) * nb + k) * nb + j] = -src[i];
		}
	}
}

// every element's 1/dtau_e: one value for all
__global__ void k_fill(int n, double v, double* __restrict__ out)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = v;
}

// 1/dtau_e of the reference's CFL ramping (compute_dt_cfl_constrained, dg/solve_dg.c:284-318): one warp per
// element; lambda_e = the largest |V| + c over the element's Bezier coefficients ccSB0 u read as conservative
// states (compute_max_wavespeed), |b| for advection; dtau_e = cfl min(h_e / lambda_e, h_e^2 / mu).
__global__ void k_pseudo_dt(int n_vol, int n_s, int nv, const double* __restrict__ u, const double* __restrict__ bez,
                            const double* __restrict__ h, double adv_speed, double mu, double cfl,
                            double* __restrict__ inv_dtau)
{
	const int e = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
	if (e >= n_vol) return;
	const int d = nv - 2;
	double lam = (nv == 1) ? adv_speed : 0.0;
	if (nv > 1)
		for (int i = lane; i < n_s; i += 32) {
			double b[5] = {0, 0, 0, 0, 0};
			for (int var = 0; var < nv; ++var) {
				double acc = 0.0;
				for (int j = 0; j < n_s; ++j) acc += bez[(int64_t)i * n_s + j] * u[(int64_t)e * n_s * nv + j + (int64_t)n_s * var];
				b[var] = acc;
			}
			if (!(b[0] > 0.0)) continue;
			double V2 = 0.0;
			for (int a = 0; a < d; ++a) V2 += (b[1 + a] / b[0]) * (b[1 + a] / b[0]);
			const double p = 0.4 * (b[d + 1] - 0.5 * b[0] * V2);
			lam = fmax(lam, sqrt(V2) + sqrt(fmax(1.4 * p / b[0], 0.0)));
		}
	for (int o = 16; o > 0; o >>= 1) lam = fmax(lam, __shfl_xor_sync(0xffffffffu, lam, o));
	if (lane == 0) {
		const double he = h[e];
		double dt = (lam > 0.0) ? he / lam : 1e300;
		if (mu > 0.0) dt = fmin(dt, he * he / mu);
		inv_dtau[e] = 1.0 / (cfl * dt);
	}
}

// out = shift_e z - J z  (J z given), per element shift_e = 1/dtau_e
__global__ void k_shift_minus(int64_t n, int nb, const double* __restrict__ shift, const double* __restrict__ z,
                              const double* __restrict__ jz, double* __restrict__ out)
{
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
		out[i] = shift[i / nb] * z[i] - jz[i];
}

// out = shift_e z - (F1 - F0) / eps
__global__ void k_shift_minus_fd(int64_t n, int nb, const double* __restrict__ shift, const double* __restrict__ z,
                                 const double* __restrict__ F1, const double* __restrict__ F0, double inv_eps,
                                 double* __restrict__ out)
{
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
		out[i] = shift[i / nb] * z[i] - (F1[i] - F0[i]) * inv_eps;
}

// partial[block] = sum over its elements of max_k sum_j |B_e[k][j] - shift_e delta_kj| (the inf-norm of -dF/du_ee)
__global__ void k_block_norm_partial(int n_vol, int nb, const double* __restrict__ blocks,
                                     const double* __restrict__ shift, double* __restrict__ partial)
{
	__shared__ double red[32];
	double acc = 0.0;
	for (int e = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); e < n_vol; e += gridDim.x * (blockDim.x / 32)) {
		double mx = 0.0;
		for (int k = threadIdx.x & 31; k < nb; k += 32) {
			double sr = 0.0;
			for (int j = 0; j < nb; ++j) sr += fabs(blocks[((int64_t)e * nb + k) * nb + j] - (k == j ? shift[e] : 0.0));
			mx = fmax(mx, sr);
		}
		for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
		acc += ((threadIdx.x & 31) == 0) ? mx : 0.0;
	}
	for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.0;
		for (int i = 0; i < (int)(blockDim.x / 32); ++i) t += red[i];
		partial[blockIdx.x] = t;
	}
}

// In-place LU with partial pivoting of one nb x nb block per thread block (nb <= 128), row-major.
__global__ void k_lu_batched(int nb, double* __restrict__ blocks, int* __restrict__ piv, int* __restrict__ info)
{
	extern __shared__ double a[];
	__shared__ int s_p;
	__shared__ double s_pivval;
	const int e = blockIdx.x;
	double* g = blocks + (int64_t)e * nb * nb;
	for (int i = threadIdx.x; i < nb * nb; i += blockDim.x) a[i] = g[i];
	__syncthreads();
	for (int k = 0; k < nb; ++k) {
		if (threadIdx.x == 0) {
			int p = k;
			double best = fabs(a[k * nb + k]);
			for (int i = k + 1; i < nb; ++i)
				if (fabs(a[i * nb + k]) > best) { best = fabs(a[i * nb + k]); p = i; }
			s_p = p;
			s_pivval = best;
			piv[(int64_t)e * nb + k] = p;
			if (best == 0.0) atomicExch(info, e + 1);
		}
		__syncthreads();
		const int p = s_p;
		if (p != k)
			for (int j = threadIdx.x; j < nb; j += blockDim.x) {
				const double t = a[k * nb + j]; a[k * nb + j] = a[p * nb + j]; a[p * nb + j] = t;
			}
		__syncthreads();
		if (s_pivval != 0.0) {
			const double inv = 1.0 / a[k * nb + k];
			for (int i = k + 1 + threadIdx.x; i < nb; i += blockDim.x) a[i * nb + k] *= inv;
			__syncthreads();
			const int rem = nb - k - 1;
			for (int t = threadIdx.x; t < rem * rem; t += blockDim.x) {
				const int i = k + 1 + t / rem, j = k + 1 + t % rem;
				a[i * nb + j] -= a[i * nb + k] * a[k * nb + j];
			}
		}
		__syncthreads();
	}
	for (int i = threadIdx.x; i < nb * nb; i += blockDim.x) g[i] = a[i];
}

// z_e = (LU_e)^-1 r_e, one warp per element
__global__ void k_lu_solve(int n_vol, int nb, const double* __restrict__ lu, const int* __restrict__ piv,
                           const double* __restrict__ r, double* __restrict__ z)
{
	const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (warp >= n_vol) return;
	extern __shared__ double sh[];
	double* x = sh + (threadIdx.x >> 5) * nb;
	const double* a = lu + (int64_t)warp * nb * nb;
	for (int i = lane; i < nb; i += 32) x[i] = r[(int64_t)warp * nb + i];
	__syncwarp();
	if (lane == 0)
		for (int k = 0; k < nb; ++k) {
			const int p = piv[(int64_t)warp * nb + k];
			if (p != k) { const double t = x[k]; x[k] = x[p]; x[p] = t; }
		}
	__syncwarp();
	for (int i = 0; i < nb; ++i) {          // L y = P r (unit diagonal)
		double s = 0.0;
		for (int j = lane; j < i; j += 32) s += a[i * nb + j] * x[j];
		for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		if (lane == 0) x[i] -= s;
		__syncwarp();
	}
	for (int i = nb - 1; i >= 0; --i) {     // U z = y
		double s = 0.0;
		for (int j = i + 1 + lane; j < nb; j += 32) s += a[i * nb + j] * x[j];
		for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		if (lane == 0) x[i] = (x[i] - s) / a[i * nb + i];
		__syncwarp();
	}
	for (int i = lane; i < nb; i += 32) z[(int64_t)warp * nb + i] = x[i];
}

// z_e = P_e r_e / (shift_e + rho) with a dense per-element matrix (learned inverse), one warp per element
__global__ void k_block_apply(int n_vol, int nb, const float* __restrict__ P, const double* __restrict__ r,
                              double* __restrict__ z, const double* __restrict__ shift, double rho)
{
	const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
	if (warp >= n_vol) return;
	const float* a = P + (int64_t)warp * nb * nb;
	const double* x = r + (int64_t)warp * nb;
	const double scale = 1.0 / (shift[warp] + rho);
	for (int i = lane; i < nb; i += 32) {
		double s = 0.0;
		for (int j = 0; j < nb; ++j) s += (double)a[i * nb + j] * x[j];
		z[(int64_t)warp * nb + i] = scale * s;
	}
}

// ------------------------------------------------------------------------------------------------------------
// block ILU(0), diagonal form:  M = (D + L) D^-1 (D + U)
//   L, U the strictly lower / upper face-neighbour blocks of A = I/dtau - dF/du in the chosen element order (rank),
//   D_i = A_ii - sum_{k lower neighbour of i} A_ik D_k^-1 A_ki, so that M and A have the same diagonal and
//   neighbour blocks; on meshes whose face graph has no triangles (every mesh of this path except periodic
//   directions three elements wide) this is block ILU(0).  D_i^-1 is kept explicitly (Gauss-Jordan with partial
//   pivoting); each element's blocks of one level are independent, so the factorisation and both triangular
//   solves run level by level, one thread block per element.
// ------------------------------------------------------------------------------------------------------------
// the blocks of column j of every element of distance-2 colour `col`: the diagonal block of those elements and
// the neighbour block A_ik (k of colour col) of every other element i (at most one such k per i)
__global__ void k_extract_ilu(int n_vol, int nb, int n_fl, const double* __restrict__ F1, const double* __restrict__ F0,
                              const int* __restrict__ colour, const int* __restrict__ nbr, int col, int j,
                              double inv_eps, const double* __restrict__ shift, double* __restrict__ diag,
                              double* __restrict__ offd)
{
	const int64_t n = (int64_t)n_vol * nb;
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
		const int e = (int)(i / nb), k = (int)(i - (int64_t)e * nb);
		const double dF = (F1[i] - F0[i]) * inv_eps;
		if (colour[e] == col) {
			diag[((int64_t)e * nb + k) * nb + j] = (k == j ? shift[e] : 0.0) - dF;
			continue;
		}
		for (int s = 0; s < n_fl; ++s) {
			const int o = nbr[e * n_fl + s];
			if (o >= 0 && colour[o] == col) offd[(((int64_t)e * n_fl + s) * nb + k) * nb + j] = -dF;
		}
	}
}

// Per element of the level lists, what its row of the factorisation and of the sweeps touches: {element, number of lower
// neighbours, number of upper ones, then (slot, neighbour) of the lower and of the upper ones in slot order}.
constexpr int kIluDesc = 16;   // 3 + 2 * 6 local faces

// D_i = A_ii - sum_{k lower} A_ik D_k^-1 A_ki, kIluSlab columns per block (gridDim.y of them): the columns are independent,
// and one SM's FP64 pipe would take 14 us for each of a 36 x 36 element's four products (8x8 QUAD p = 2, one level:
// factor 204 us with a block per element, 40 us for update and inverse here).  diag holds A_ii on entry (elements of
// earlier levels already hold D_k^-1).
constexpr int kIluSlab = 4;
__global__ void __launch_bounds__(256) k_ilu_update_level(const int* __restrict__ desc, int nb, int n_fl,
                                                          const int* __restrict__ nbr, double* __restrict__ diag,
                                                          const double* __restrict__ offd)
{
	extern __shared__ double sh[];
	double* M = sh;                       // D_k^-1, then A_ik
	double* B = M + nb * nb;              // [nb][kIluSlab] A_ki
	double* T = B + nb * kIluSlab;        // [nb][kIluSlab] D_k^-1 A_ki
	double* D = T + nb * kIluSlab;        // [nb][kIluSlab]
	const int* d = desc + (size_t)blockIdx.x * kIluDesc;
	const int i = d[0], n_low = d[1];
	if (n_low == 0) return;
	const int c0 = blockIdx.y * kIluSlab, nc = min(kIluSlab, nb - c0);
	double* Di = diag + (int64_t)i * nb * nb;
	for (int t = threadIdx.x; t < nb * kIluSlab; t += blockDim.x) {
		const int r = t / kIluSlab, c = t - r * kIluSlab;
		D[t] = c < nc ? Di[r * nb + c0 + c] : 0.0;
	}
	for (int q = 0; q < n_low; ++q) {
		const int s = d[3 + 2 * q], k = d[4 + 2 * q];
		int sk = -1;
		for (int t = 0; t < n_fl; ++t)
			if (nbr[k * n_fl + t] == i) { sk = t; break; }
		if (sk < 0) continue;
		const double* Dk = diag + (int64_t)k * nb * nb;                           // D_k^-1
		const double* Aki = offd + ((int64_t)k * n_fl + sk) * nb * nb;
		const double* Aik = offd + ((int64_t)i * n_fl + s) * nb * nb;
		for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) M[t] = Dk[t];
		for (int t = threadIdx.x; t < nb * kIluSlab; t += blockDim.x) {
			const int r = t / kIluSlab, c = t - r * kIluSlab;
			B[t] = c < nc ? Aki[r * nb + c0 + c] : 0.0;
		}
		__syncthreads();
		for (int t = threadIdx.x; t < nb * kIluSlab; t += blockDim.x) {             // T = D_k^-1 A_ki
			const int r = t / kIluSlab, c = t - r * kIluSlab;
			double acc = 0.0;
			for (int p = 0; p < nb; ++p) acc += M[r * nb + p] * B[p * kIluSlab + c];
			T[t] = acc;
		}
		__syncthreads();
		for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) M[t] = Aik[t];
		__syncthreads();
		for (int t = threadIdx.x; t < nb * kIluSlab; t += blockDim.x) {             // D -= A_ik T
			const int r = t / kIluSlab, c = t - r * kIluSlab;
			double acc = 0.0;
			for (int p = 0; p < nb; ++p) acc += M[r * nb + p] * T[p * kIluSlab + c];
			D[t] -= acc;
		}
		__syncthreads();
	}
	for (int t = threadIdx.x; t < nb * kIluSlab; t += blockDim.x) {
		const int r = t / kIluSlab, c = t - r * kIluSlab;
		if (c < nc) Di[r * nb + c0 + c] = D[t];
	}
}

// D_i^-1 of the elements of one level, one block each, in shared memory (Gauss-Jordan with partial pivoting; the row
// exchanges are undone as column exchanges at the end).  Two barriers per pivot: every warp finds the pivot by itself
// and the exchanged row goes through buffers, since the chain of pivots, not the FP64 work, bounds it.
__global__ void __launch_bounds__(1024) k_ilu_invert_level(const int* __restrict__ desc, int nb, double* __restrict__ diag,
                                                           int* __restrict__ info)
{
	extern __shared__ double a[];         // [nb][nb]
	double* row = a + nb * nb;            // the pivot row over the pivot
	double* old = row + nb;               // the row that the pivot row changes places with
	double* col = old + nb;               // the factors of the rows after the exchange
	int* perm = (int*)(col + nb);
	const int i0 = desc[(size_t)blockIdx.x * kIluDesc];
	double* Di = diag + (int64_t)i0 * nb * nb;
	const int lane = threadIdx.x & 31;
	for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) a[t] = Di[t];
	__syncthreads();
	for (int k = 0; k < nb; ++k) {
		// largest |a_ik|, i >= k (lowest i of equal ones): magnitudes compared as integers, NaN never chosen
		long long best = -1;
		int p = k;
		for (int i = k + lane; i < nb; i += 32) {
			const long long v = __double_as_longlong(a[i * nb + k]) & 0x7FFFFFFFFFFFFFFFll;
			if (v <= 0x7FF0000000000000ll && v > best) { best = v; p = i; }
		}
		for (int o = 16; o > 0; o >>= 1) {
			const long long bv = __shfl_xor_sync(0xffffffffu, best, o);
			const int bp = __shfl_xor_sync(0xffffffffu, p, o);
			if (bv > best || (bv == best && bp < p)) { best = bv; p = bp; }
		}
		if (best <= 0) {   // the same in every warp: the block leaves together
			if (threadIdx.x == 0) atomicExch(info, i0 + 1);
			return;
		}
		for (int c = threadIdx.x; c < nb; c += blockDim.x) {
			const double inv = 1.0 / a[p * nb + k];
			row[c] = c == k ? inv : a[p * nb + c] * inv;
			old[c] = a[k * nb + c];
			col[c] = a[(c == p ? k : c) * nb + k];
			if (c == k) perm[k] = p;
		}
		__syncthreads();
		for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) {
			const int i = t / nb, c = t - i * nb;
			double v;
			if (i == k) v = row[c];
			else if (c == k) v = -col[i] * row[k];
			else {
				v = i == p ? old[c] : a[t];
				v -= col[i] * row[c];
			}
			a[t] = v;
		}
		__syncthreads();
	}
	for (int k = nb - 1; k >= 0; --k) {
		const int p = perm[k];
		if (p != k)
			for (int i = threadIdx.x; i < nb; i += blockDim.x) {
				const double t = a[i * nb + k]; a[i * nb + k] = a[i * nb + p]; a[i * nb + p] = t;
			}
		__syncthreads();
	}
	for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) Di[t] = a[t];
}

// One level of either triangular sweep, one thread block per element, four rows per warp (lane l the columns l, l + 32,
// ...).
//   FWD: x_i = D_i^-1 (b_i - sum_{k lower} A_ik x_k)    (b = r, x = w)
//   BWD: x_i = b_i - D_i^-1 sum_{j upper} A_ij x_j      (b = w, x = z)
// The levels are a chain of dependent launches, each with few elements, so its latency counts: the next level's
// blocks start early (programmatic dependent launch) and fetch their descriptor and matrices, which no level writes,
// before they wait for this one; the lane sums of a warp's four rows are folded together (6 FP64 additions instead of
// 20: the FP64 pipe takes ~20 cycles of the SM for each warp instruction).  A row's sum keeps one order: neighbours, then
// columns, then lanes l + (l ^ 16), ^ 8, ..  8x8 QUAD p = 2 (36 x 36 blocks): 25 us per level with one row after
// the other and a plain launch; 64x128 annulus QUAD p = 3 (64 x 64 blocks): 17 us.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Sums over the lanes of four rows' values; lane l returns the row 2 (l >> 4) + ((l >> 3) & 1).
__device__ __forceinline__ double warp_sum4(const double (&v)[4], int lane)
{
	const bool h = lane & 16, q = lane & 8;
	const double a = (h ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
	const double b = (h ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h ? v[1] : v[3], 16);
	double s = (q ? b : a) + __shfl_xor_sync(0xffffffffu, q ? a : b, 8);
	for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
	return s;
}

template <int CC, bool FWD>
__global__ void __launch_bounds__(CC <= 2 ? 512 : 896) k_ilu_sweep_level(const int* __restrict__ desc, int nb, int n_fl,
                                                                         const double* __restrict__ dinv,
                                                                         const double* __restrict__ offd, const double* b, double* x)
{
	constexpr int PRE = CC <= 2 ? 2 : 0;   // neighbour blocks fetched before the wait (register budget)
	__shared__ double y[128];
	grid_dependency_launch();
	int d[kIluDesc];
#pragma unroll
	for (int k = 0; k < kIluDesc / 4; ++k) {
		const int4 t = reinterpret_cast<const int4*>(desc + (size_t)blockIdx.x * kIluDesc)[k];
		d[4 * k] = t.x; d[4 * k + 1] = t.y; d[4 * k + 2] = t.z; d[4 * k + 3] = t.w;
	}
	const int i = d[0], n_low = d[1], n_use = FWD ? n_low : d[2];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	auto entry = [&](int q, int w) {   // (slot, neighbour) q of this sweep's list
		int v = 0;
#pragma unroll
		for (int k = 0; k < 6; ++k) v = (k == (FWD ? q : n_low + q)) ? d[3 + 2 * k + w] : v;
		return v;
	};
	auto fetch = [&](const double* M, double (&m)[4][CC]) {
#pragma unroll
		for (int t = 0; t < 4; ++t)
#pragma unroll
			for (int j = 0; j < CC; ++j) {
				const int row = 4 * warp + t, c = lane + 32 * j;
				m[t][j] = (row < nb && c < nb) ? M[(int64_t)row * nb + c] : 0.0;
			}
	};
	double dm[4][CC], am[PRE > 0 ? PRE : 1][4][CC];
	fetch(dinv + (int64_t)i * nb * nb, dm);
#pragma unroll
	for (int q = 0; q < PRE; ++q)
		if (q < n_use) fetch(offd + ((int64_t)i * n_fl + entry(q, 0)) * nb * nb, am[q]);
	grid_dependency_wait();
	const int row = 4 * warp + 2 * (lane >> 4) + ((lane >> 3) & 1);   // the row whose sum this lane gets
	const bool owner = (lane & 7) == 0 && row < nb;
	const double bv = owner ? __ldcg(b + (int64_t)i * nb + row) : 0.0;
	double acc[4] = {0.0, 0.0, 0.0, 0.0};
	auto times = [&](const double (&m)[4][CC], const double (&v)[CC]) {
#pragma unroll
		for (int j = 0; j < CC; ++j)
			if (lane + 32 * j < nb) {
#pragma unroll
				for (int t = 0; t < 4; ++t) acc[t] += m[t][j] * v[j];
			}
	};
	for (int q = 0; q < n_use; ++q) {
		double v[CC];
#pragma unroll
		for (int j = 0; j < CC; ++j) v[j] = lane + 32 * j < nb ? __ldcg(x + (int64_t)entry(q, 1) * nb + lane + 32 * j) : 0.0;
		if constexpr (PRE > 0) {
			if (q == 0) { times(am[0], v); continue; }
			if (q == 1) { times(am[1], v); continue; }
		}
		double m[4][CC];
		fetch(offd + ((int64_t)i * n_fl + entry(q, 0)) * nb * nb, m);
		times(m, v);
	}
	const double s = warp_sum4(acc, lane);
	if (owner) y[row] = FWD ? bv - s : s;
	__syncthreads();
#pragma unroll
	for (int t = 0; t < 4; ++t) acc[t] = 0.0;
	double yv[CC];
#pragma unroll
	for (int j = 0; j < CC; ++j) yv[j] = lane + 32 * j < nb ? y[lane + 32 * j] : 0.0;
	times(dm, yv);
	const double z = warp_sum4(acc, lane);
	if (owner) x[(int64_t)i * nb + row] = FWD ? z : bv - z;
}

// ------------------------------------------------------------------------------------------------------------
// host orchestration
// ------------------------------------------------------------------------------------------------------------
struct Implicit {
	int nb = 0, m = 0, n_colours = 0;
	int64_t n = 0;
	double *u = nullptr, *F0 = nullptr, *F1 = nullptr, *up = nullptr, *du = nullptr, *w = nullptr;
	double *V = nullptr, *Z = nullptr, *h = nullptr, *h2 = nullptr, *partial = nullptr;
	double* hcol_host = nullptr;  // pinned [m + 2]: the Arnoldi column, one copy per iteration
	double *blocks = nullptr;
	int *piv = nullptr, *colour = nullptr, *info = nullptr;
	float* P = nullptr;           // learned inverses [n_vol][nb][nb] (owned by the MLP state)
	double* forcing = nullptr;    // subtracted from F (nullptr: none)
	double rho = 0.0;             // mean inf-norm of the element blocks of dF/du (last assembly)
	double* forcing_buf = nullptr;
	TanWork probe;                // tangent probing: work space of a batch of directions,
	double *pV = nullptr, *pJV = nullptr;   // [probe.nb][n] the directions and their products
	double* inv_dtau = nullptr;   // [n_vol] 1/dtau_e of the current Newton step
	bool blocks_valid = false;
	bool u_traced = false;        // c->trace holds the traces of u (within one Krylov solve)
	bool tangent = true;          // Jacobian products by the analytic linearisation (false: finite differences)
	// block ILU (built on first use)
	int ilu_order = -1;           // element order of the levels: DPG_ILU_ORDER_* (-1: not built)
	int ilu_parts = 0;            // subdomains of the factorisation (contiguous ranges of the element order)
	int n_colours2 = 0;           // distance-2 colouring: no two elements within two face steps share a colour
	int* colour2 = nullptr;       // [n_vol]
	int* nbr = nullptr;           // [n_vol][n_fl] distinct face neighbours (-1: none)
	int* desc = nullptr;          // [n_vol][kIluDesc] rows of the elements grouped by level
	std::vector<int> level_ptr;   // [n_levels + 1]
	double* offd = nullptr;       // [n_vol][n_fl][nb][nb] A_{i, nbr[i][s]}
	double* wbuf = nullptr;       // [n] forward-sweep result
	double* ilu_in = nullptr;     // [n] right-hand side of the sweeps' graph
	double* ilu_out = nullptr;    // [n] result of the sweeps' graph
	cudaGraphExec_t ilu_graph = nullptr;   // forward and backward sweeps over all levels (one launch)
	bool ilu_valid = false;
};

static int grid_for(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 4 * 152 * 8); }

static Implicit* implicit_state(dpg_gpu_ctx* c, int m)
{
	Implicit* im = (Implicit*)c->implicit;
	if (im && im->m >= m) return im;
	if (im) implicit_free(c);
	im = new Implicit();
	im->nb = c->g.n_s * c->n_var;
	im->m = m;
	im->n = c->n_dof;
	const int64_t n = im->n;
	bool ok = true;
	auto al = [&](void** p, size_t bytes) { if (cudaMalloc(p, bytes ? bytes : 1) != cudaSuccess) ok = false; };
	al((void**)&im->u, n * 8); al((void**)&im->F0, n * 8); al((void**)&im->F1, n * 8); al((void**)&im->up, n * 8);
	al((void**)&im->du, n * 8); al((void**)&im->w, n * 8);
	al((void**)&im->V, (size_t)(m + 1) * n * 8); al((void**)&im->Z, (size_t)m * n * 8);
	al((void**)&im->h, (size_t)(m + 2) * 8); al((void**)&im->h2, (size_t)(m + 2) * 8);
	al((void**)&im->partial, (size_t)(m + 2) * kRedBlocks * 8);
	if (cudaMallocHost((void**)&im->hcol_host, (size_t)(m + 2) * 8) != cudaSuccess) ok = false;
	al((void**)&im->blocks, (size_t)c->g.n_vol * im->nb * im->nb * 8);
	al((void**)&im->piv, (size_t)c->g.n_vol * im->nb * 4); al((void**)&im->info, 4);
	al((void**)&im->colour, (size_t)c->g.n_vol * 4);
	al((void**)&im->inv_dtau, (size_t)c->g.n_vol * 8);
	c->implicit = im;
	if (!ok) { implicit_free(c); return nullptr; }
	// greedy element colouring: face neighbours get different colours
	std::vector<int> vf((size_t)c->g.n_vol * c->g.n_fl), col(c->g.n_vol, -1);
	cudaMemcpy(vf.data(), c->g.vol_face, vf.size() * 4, cudaMemcpyDeviceToHost);
	std::vector<std::vector<int>> face_vols(c->fc.n_face);
	for (int e = 0; e < c->g.n_vol; ++e)
		for (int lf = 0; lf < c->g.n_fl; ++lf) face_vols[vf[(size_t)e * c->g.n_fl + lf] >> 1].push_back(e);
	int nc = 0;
	for (int e = 0; e < c->g.n_vol; ++e) {
		std::vector<char> used(64, 0);
		for (int lf = 0; lf < c->g.n_fl; ++lf)
			for (int o : face_vols[vf[(size_t)e * c->g.n_fl + lf] >> 1])
				if (o != e && col[o] >= 0 && col[o] < 64) used[col[o]] = 1;
		int k = 0;
		while (used[k]) ++k;
		col[e] = k;
		nc = std::max(nc, k + 1);
	}
	im->n_colours = nc;
	cudaMemcpy(im->colour, col.data(), col.size() * 4, cudaMemcpyHostToDevice);
	return im;
}

void implicit_free(dpg_gpu_ctx* c)
{
	Implicit* im = (Implicit*)c->implicit;
	if (!im) return;
	void* ptrs[] = {im->u, im->F0, im->F1, im->up, im->du, im->w, im->V, im->Z, im->h, im->h2, im->partial,
	                im->blocks, im->piv, im->info, im->colour, im->forcing_buf, im->pV, im->pJV, im->colour2, im->nbr,
	                im->desc, im->offd, im->wbuf, im->inv_dtau, im->ilu_in, im->ilu_out};
	if (im->ilu_graph) cudaGraphExecDestroy(im->ilu_graph);
	for (void* p : ptrs) if (p) cudaFree(p);
	free_tangent_work(&im->probe);
	if (im->hcol_host) cudaFreeHost(im->hcol_host);
	delete im;
	c->implicit = nullptr;
}

// F = m_inv * rhs(u) (- forcing) through the residual kernels of the context's precision mode.
static int residual(dpg_gpu_ctx* c, const double* u, double* F)
{
	double* sol0 = c->sol;
	double* rhs0 = c->rhs;
	c->sol = const_cast<double*>(u);
	c->rhs = F;
	int rc = enqueue_residual_raw(c, c->dmax + kMaxStages);
	c->sol = sol0;
	c->rhs = rhs0;
	Implicit* im = (Implicit*)c->implicit;
	if (!rc && im && im->forcing)
		k_axpby<<<grid_for(im->n), 256, 0, c->stream>>>(im->n, -1.0, im->forcing, 1.0, F);
	return rc;
}

// blocks of a reduction over n values: those past the last value would only add zeros
static int red_blocks(int64_t n) { return (int)std::min<int64_t>(kRedBlocks, (n + kRedThreads - 1) / kRedThreads); }

static int absmax(dpg_gpu_ctx* c, Implicit* im, const double* x, double* out)
{
	k_absmax_partial<<<kRedBlocks, kRedThreads, 0, c->stream>>>(im->n, x, im->partial);
	k_absmax_partial<<<1, kRedThreads, 0, c->stream>>>(kRedBlocks, im->partial, im->h);
	if (cudaMemcpyAsync(out, im->h, 8, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	if (cudaStreamSynchronize(c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	return std::isfinite(*out) ? DPG_OK : DPG_ERR_NONFINITE;
}

// h[0..nv) = V[0..nv)^T w   (device result in im->h, copied to host_h)
static int multidot(dpg_gpu_ctx* c, Implicit* im, int nv, const double* V, const double* w, double* host_h)
{
	const int blocks = red_blocks(im->n);
	k_multidot_partial<<<dim3(blocks, (nv + kDotChunk - 1) / kDotChunk), kRedThreads, 0, c->stream>>>(
	    im->n, nv, V, im->n, const_cast<double*>(w), im->partial);
	k_reduce_partials<<<nv, 256, 0, c->stream>>>(nv, blocks, im->partial, im->h);
	if (cudaMemcpyAsync(host_h, im->h, 8 * nv, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	if (cudaStreamSynchronize(c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	return DPG_OK;
}

// Block columns by tangent probing: the directions of all (colour, column) pairs are independent, so they go through the
// linearisation's launches in batches (an 8x8 QUAD p = 2 mesh has 396 probes of ~60 us each one after another, bound by
// the launch chain on 4 blocks; all of them at once take ~1 ms).  nbr null: diagonal blocks only.
constexpr size_t kProbeBytes = (size_t)512 << 20;   // work space of a batch, kept with the implicit state; less where it does not fit

static int probe_blocks(dpg_gpu_ctx* c, Implicit* im, const int* colour, int n_colours, const int* nbr, double* diag, double* offd)
{
	const int nb = im->nb, n_vol = c->g.n_vol, n_probes = n_colours * nb;
	int rc;
	if (!im->probe.nb) {
		const size_t per = tangent_bytes(c) + 2 * sizeof(double) * im->n;
		const int most = (int)std::max<size_t>(1, std::min<size_t>(kProbeBytes / per, (size_t)n_probes));
		alloc_tangent_work(c, most, &im->probe, {{&im->pV, (size_t)im->n}, {&im->pJV, (size_t)im->n}});
	}
	// no room for one direction more: one after another through the buffers of the Krylov products
	const TanWork all = im->probe.nb ? im->probe : c->tan;
	double *V = im->probe.nb ? im->pV : im->up, *JV = im->probe.nb ? im->pJV : im->F1;
	for (int p0 = 0; p0 < n_probes; p0 += all.nb) {
		TanWork w = all;
		w.nb = std::min(all.nb, n_probes - p0);
		const dim3 grid((unsigned)std::min<int64_t>((im->n + 255) / 256, 1216), w.nb);
		k_probe_directions<<<grid, 256, 0, c->stream>>>(n_vol, nb, colour, p0, V);
		if ((rc = jvp_fp64(c, im->u, V, JV, w))) return rc;
		k_extract_probes<<<grid, 256, 0, c->stream>>>(n_vol, nb, c->g.n_fl, JV, colour, nbr, p0, im->inv_dtau, diag, offd);
	}
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

static int assemble_block_jacobi(dpg_gpu_ctx* c, Implicit* im, const double* F0)
{
	const int nb = im->nb, n_vol = c->g.n_vol;
	const double eps = 1e-7;
	int rc;
	// block column j of every element of one colour at once (no two face neighbours share a colour): the tangent
	// along e_j on those elements (exact), or a forward difference of the residual
	if (im->tangent && (rc = probe_blocks(c, im, im->colour, im->n_colours, nullptr, im->blocks, nullptr))) return rc;
	for (int col = 0; col < im->n_colours && !im->tangent; ++col)
		for (int j = 0; j < nb; ++j) {
			k_perturb<<<grid_for(im->n), 256, 0, c->stream>>>(n_vol, nb, im->u, im->up, im->colour, col, j, eps);
			if ((rc = residual(c, im->up, im->F1))) return rc;
			k_extract_column<<<grid_for(im->n), 256, 0, c->stream>>>(n_vol, nb, im->F1, F0, im->colour, col, j,
			                                                          1.0 / eps, im->inv_dtau, im->blocks);
		}
	{
		k_block_norm_partial<<<kRedBlocks, kRedThreads, 0, c->stream>>>(n_vol, nb, im->blocks, im->inv_dtau, im->partial);
		std::vector<double> parts(kRedBlocks);
		if (cudaMemcpyAsync(parts.data(), im->partial, 8 * kRedBlocks, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess)
			return DPG_ERR_CUDA;
		if (cudaStreamSynchronize(c->stream) != cudaSuccess) return DPG_ERR_CUDA;
		double t = 0.0;
		for (double v : parts) t += v;
		im->rho = t / n_vol;
	}
	if (cudaMemsetAsync(im->info, 0, 4, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	const size_t smem = (size_t)nb * nb * 8;
	if (smem > 48 * 1024 && cudaFuncSetAttribute(k_lu_batched, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem))
		return DPG_ERR_CUDA;
	k_lu_batched<<<n_vol, 256, smem, c->stream>>>(nb, im->blocks, im->piv, im->info);
	int info = 0;
	cudaMemcpyAsync(&info, im->info, 4, cudaMemcpyDeviceToHost, c->stream);
	if (cudaStreamSynchronize(c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	im->blocks_valid = (info == 0);
	return info == 0 ? DPG_OK : DPG_ERR_NONFINITE;
}

// ---- block ILU: structure (once per element order), assembly and factorisation (every Newton step), solve ----
constexpr int kIluMaxNb = 112;   // a block of 4 rows per warp, 28 warps

static size_t ilu_update_smem(int nb) { return ((size_t)nb * nb + 3 * (size_t)nb * kIluSlab) * 8; }
static size_t ilu_invert_smem(int nb) { return ((size_t)nb * nb + 3 * (size_t)nb) * 8 + (size_t)nb * 4; }

template <int CC, bool FWD>
static void launch_sweep_level(dpg_gpu_ctx* c, Implicit* im, int l, bool first, const double* b, double* x)
{
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3(im->level_ptr[l + 1] - im->level_ptr[l]);
	cfg.blockDim = dim3(32 * ((im->nb + 3) / 4));
	cfg.stream = c->stream;
	cudaLaunchAttribute at{};
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = &at;
	cfg.numAttrs = first ? 0 : 1;   // the first level waits for what wrote its right-hand side
	cudaLaunchKernelEx(&cfg, k_ilu_sweep_level<CC, FWD>, (const int*)(im->desc + (size_t)im->level_ptr[l] * kIluDesc), im->nb,
	                   c->g.n_fl, (const double*)im->blocks, (const double*)im->offd, b, x);
}

template <int CC>
static void enqueue_sweeps_of(dpg_gpu_ctx* c, Implicit* im, const double* r, double* z)
{
	const int n_levels = (int)im->level_ptr.size() - 1;
	bool first = true;
	for (int l = 0; l < n_levels; ++l) {
		if (im->level_ptr[l + 1] <= im->level_ptr[l]) continue;
		launch_sweep_level<CC, true>(c, im, l, first, r, im->wbuf);
		first = false;
	}
	for (int l = n_levels - 1; l >= 0; --l)
		if (im->level_ptr[l + 1] > im->level_ptr[l]) launch_sweep_level<CC, false>(c, im, l, false, im->wbuf, z);
}

static void enqueue_block_ilu_sweeps(dpg_gpu_ctx* c, Implicit* im, const double* r, double* z)
{
	switch ((im->nb + 31) / 32) {   // columns per lane (nb <= kIluMaxNb)
	case 1: return enqueue_sweeps_of<1>(c, im, r, z);
	case 2: return enqueue_sweeps_of<2>(c, im, r, z);
	case 3: return enqueue_sweeps_of<3>(c, im, r, z);
	default: return enqueue_sweeps_of<4>(c, im, r, z);
	}
}

static int ilu_build(dpg_gpu_ctx* c, Implicit* im, int order, int parts)
{
	if (parts < 1) parts = 1;
	if (im->ilu_order == order && im->ilu_parts == parts) return DPG_OK;
	const int n_vol = c->g.n_vol, n_fl = c->g.n_fl, nb = im->nb;
	if (nb > kIluMaxNb) return DPG_ERR_UNSUPPORTED;
	std::vector<int> vf((size_t)n_vol * n_fl);
	if (cudaMemcpy(vf.data(), c->g.vol_face, vf.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return DPG_ERR_CUDA;
	std::vector<std::vector<int>> face_vols(c->fc.n_face);
	for (int e = 0; e < n_vol; ++e)
		for (int lf = 0; lf < n_fl; ++lf) face_vols[vf[(size_t)e * n_fl + lf] >> 1].push_back(e);
	// distinct face neighbours (a periodic direction one or two elements wide repeats a neighbour, or the element)
	std::vector<int> nbr((size_t)n_vol * n_fl, -1);
	for (int e = 0; e < n_vol; ++e) {
		int cnt = 0;
		for (int lf = 0; lf < n_fl; ++lf)
			for (int o : face_vols[vf[(size_t)e * n_fl + lf] >> 1]) {
				if (o == e) continue;
				bool seen = false;
				for (int q = 0; q < cnt; ++q) seen |= (nbr[(size_t)e * n_fl + q] == o);
				if (!seen) nbr[(size_t)e * n_fl + cnt++] = o;
			}
	}
	// distance-2 colouring (greedy, volume order)
	std::vector<int> col2(n_vol, -1);
	int nc2 = 0;
	for (int e = 0; e < n_vol; ++e) {
		std::vector<char> used(256, 0);
		for (int a = 0; a < n_fl; ++a) {
			const int o = nbr[(size_t)e * n_fl + a];
			if (o < 0) continue;
			if (col2[o] >= 0) used[col2[o]] = 1;
			for (int b = 0; b < n_fl; ++b) {
				const int q = nbr[(size_t)o * n_fl + b];
				if (q >= 0 && q != e && col2[q] >= 0) used[col2[q]] = 1;
			}
		}
		int k = 0;
		while (k < 255 && used[k]) ++k;
		col2[e] = k;
		nc2 = std::max(nc2, k + 1);
	}
	// element order and levels: an element's level is one more than the highest level of its lower neighbours
	std::vector<int> col1(n_vol);
	if (cudaMemcpy(col1.data(), im->colour, (size_t)n_vol * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return DPG_ERR_CUDA;
	std::vector<int64_t> key(n_vol);
	for (int e = 0; e < n_vol; ++e) key[e] = (order == DPG_ILU_ORDER_COLOUR ? (int64_t)col1[e] * n_vol : 0) + e;
	std::vector<int> by_rank(n_vol), rank(n_vol), level(n_vol, 0);
	for (int e = 0; e < n_vol; ++e) by_rank[e] = e;
	std::sort(by_rank.begin(), by_rank.end(), [&](int a, int b) { return key[a] < key[b]; });
	for (int r = 0; r < n_vol; ++r) rank[by_rank[r]] = r;
	// subdomains: `parts` contiguous ranges of the element order, factorised independently (the couplings between
	// them are left out of L and U, as in a block-Jacobi method with ILU(0) inside each block); the probing colouring
	// above keeps every neighbour, so a left-out coupling cannot alias a kept one
	if (parts > 1)
		for (int e = 0; e < n_vol; ++e)
			for (int a = 0; a < n_fl; ++a) {
				int& o = nbr[(size_t)e * n_fl + a];
				if (o >= 0 && (int64_t)rank[o] * parts / n_vol != (int64_t)rank[e] * parts / n_vol) o = -1;
			}
	int n_levels = 0;
	for (int r = 0; r < n_vol; ++r) {
		const int e = by_rank[r];
		int lv = 0;
		for (int a = 0; a < n_fl; ++a) {
			const int o = nbr[(size_t)e * n_fl + a];
			if (o >= 0 && rank[o] < r) lv = std::max(lv, level[o] + 1);
		}
		level[e] = lv;
		n_levels = std::max(n_levels, lv + 1);
	}
	im->level_ptr.assign(n_levels + 1, 0);
	for (int e = 0; e < n_vol; ++e) ++im->level_ptr[level[e] + 1];
	for (int l = 0; l < n_levels; ++l) im->level_ptr[l + 1] += im->level_ptr[l];
	std::vector<int> elems(n_vol), fill(im->level_ptr.begin(), im->level_ptr.end() - 1);
	for (int r = 0; r < n_vol; ++r) { const int e = by_rank[r]; elems[fill[level[e]]++] = e; }
	std::vector<int> desc((size_t)n_vol * kIluDesc, 0);
	for (int t = 0; t < n_vol; ++t) {
		int* d = &desc[(size_t)t * kIluDesc];
		const int e = elems[t];
		d[0] = e;
		for (int up = 0; up < 2; ++up)
			for (int a = 0; a < n_fl; ++a) {
				const int o = nbr[(size_t)e * n_fl + a];
				if (o < 0 || (rank[o] > rank[e]) != (up == 1)) continue;
				const int q = d[1] + d[2];
				d[3 + 2 * q] = a;
				d[4 + 2 * q] = o;
				++d[1 + up];
			}
	}
	bool ok = true;
	auto al = [&](void** p, size_t bytes) { if (!*p && cudaMalloc(p, bytes ? bytes : 1) != cudaSuccess) ok = false; };
	al((void**)&im->colour2, (size_t)n_vol * 4); al((void**)&im->nbr, (size_t)n_vol * n_fl * 4);
	al((void**)&im->desc, (size_t)n_vol * kIluDesc * 4);
	al((void**)&im->offd, (size_t)n_vol * n_fl * nb * nb * 8); al((void**)&im->wbuf, (size_t)im->n * 8);
	al((void**)&im->ilu_in, (size_t)im->n * 8); al((void**)&im->ilu_out, (size_t)im->n * 8);
	if (!ok) return DPG_ERR_CUDA;
	if (cudaMemcpy(im->colour2, col2.data(), (size_t)n_vol * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
	    cudaMemcpy(im->nbr, nbr.data(), nbr.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
	    cudaMemcpy(im->desc, desc.data(), desc.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
	    cudaMemset(im->offd, 0, (size_t)n_vol * n_fl * nb * nb * 8) != cudaSuccess)
		return DPG_ERR_CUDA;
	if (cudaFuncSetAttribute(k_ilu_update_level, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ilu_update_smem(kIluMaxNb)) ||
	    cudaFuncSetAttribute(k_ilu_invert_level, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ilu_invert_smem(kIluMaxNb)))
		return DPG_ERR_CUDA;
	im->n_colours2 = nc2;
	// the sweeps of one application as a graph: 2 launches per level, replayed with the right-hand side copied into
	// ilu_in and the result taken from ilu_out (the operands' addresses stay fixed from here on)
	if (im->ilu_graph) { cudaGraphExecDestroy(im->ilu_graph); im->ilu_graph = nullptr; }
	{
		cudaGraph_t graph = nullptr;
		if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return DPG_ERR_CUDA;
		enqueue_block_ilu_sweeps(c, im, im->ilu_in, im->ilu_out);
		cudaError_t e = cudaStreamEndCapture(c->stream, &graph);
		if (e != cudaSuccess) return DPG_ERR_CUDA;
		e = cudaGraphInstantiate(&im->ilu_graph, graph, 0);
		cudaGraphDestroy(graph);
		if (e != cudaSuccess) { im->ilu_graph = nullptr; return DPG_ERR_CUDA; }
	}
	im->ilu_order = order;
	im->ilu_parts = parts;
	return DPG_OK;
}

static int assemble_block_ilu(dpg_gpu_ctx* c, Implicit* im, const double* F0)
{
	const int nb = im->nb, n_vol = c->g.n_vol, n_fl = c->g.n_fl;
	const double eps = 1e-7;
	int rc;
	im->ilu_valid = false;
	if (im->tangent && (rc = probe_blocks(c, im, im->colour2, im->n_colours2, im->nbr, im->blocks, im->offd))) return rc;
	for (int col = 0; col < im->n_colours2 && !im->tangent; ++col)
		for (int j = 0; j < nb; ++j) {
			k_perturb<<<grid_for(im->n), 256, 0, c->stream>>>(n_vol, nb, im->u, im->up, im->colour2, col, j, eps);
			if ((rc = residual(c, im->up, im->F1))) return rc;
			k_extract_ilu<<<grid_for(im->n), 256, 0, c->stream>>>(n_vol, nb, n_fl, im->F1, F0, im->colour2,
			                                                       im->nbr, col, j, 1.0 / eps, im->inv_dtau,
			                                                       im->blocks, im->offd);
		}
	if (cudaMemsetAsync(im->info, 0, 4, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	const int n_levels = (int)im->level_ptr.size() - 1, n_slab = (nb + kIluSlab - 1) / kIluSlab;
	const int threads = std::min(1024, std::max(128, (nb * nb / 4 + 31) / 32 * 32));
	for (int l = 0; l < n_levels; ++l) {
		const int cnt = im->level_ptr[l + 1] - im->level_ptr[l];
		const int* desc = im->desc + (size_t)im->level_ptr[l] * kIluDesc;
		if (cnt <= 0) continue;
		if (l > 0) k_ilu_update_level<<<dim3(cnt, n_slab), 256, ilu_update_smem(nb), c->stream>>>(desc, nb, n_fl, im->nbr, im->blocks, im->offd);
		k_ilu_invert_level<<<cnt, threads, ilu_invert_smem(nb), c->stream>>>(desc, nb, im->blocks, im->info);
	}
	int info = 0;
	if (cudaMemcpyAsync(&info, im->info, 4, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	if (cudaStreamSynchronize(c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	im->ilu_valid = (info == 0);
	return info == 0 ? DPG_OK : DPG_ERR_NONFINITE;
}

static int apply_block_ilu(dpg_gpu_ctx* c, Implicit* im, const double* r, double* z)
{
	if (cudaMemcpyAsync(im->ilu_in, r, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	if (cudaGraphLaunch(im->ilu_graph, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	if (cudaMemcpyAsync(z, im->ilu_out, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	return DPG_OK;
}

static int apply_precond(dpg_gpu_ctx* c, Implicit* im, int precond, const double* r, double* z)
{
	const int nb = im->nb, n_vol = c->g.n_vol;
	const int wpb = 8;
	if (precond == DPG_PRECOND_BLOCK_JACOBI) {
		k_lu_solve<<<(n_vol + wpb - 1) / wpb, 32 * wpb, (size_t)wpb * nb * 8, c->stream>>>(n_vol, nb, im->blocks, im->piv, r, z);
	} else if (precond == DPG_PRECOND_BLOCK_ILU) {
		const int rc = apply_block_ilu(c, im, r, z);
		if (rc) return rc;
	} else if (precond == DPG_PRECOND_MLP) {
		k_block_apply<<<(n_vol + wpb - 1) / wpb, 32 * wpb, 0, c->stream>>>(n_vol, nb, im->P, r, z, im->inv_dtau,
		                                                                   mlp_rho(c));
	} else {
		if (cudaMemcpyAsync(z, r, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	}
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

// F1 = dF/du z by the tangent; the first product of a Krylov solve also leaves the state's own traces in c->trace, which
// the next ones read
static int apply_J(dpg_gpu_ctx* c, Implicit* im, const double* z)
{
	TanWork w = c->tan;
	w.u_traced = im->u_traced;
	const int rc = jvp_fp64(c, im->u, z, im->F1, w);
	im->u_traced = true;
	return rc;
}

// A z = z / dtau_e - dF/du z: the analytic tangent, or (F(u + eps z) - F(u)) / eps
static int apply_A(dpg_gpu_ctx* c, Implicit* im, const double* z, double* out, double u_norm, double z_norm)
{
	if (im->tangent) {
		const int rc = apply_J(c, im, z);
		if (rc) return rc;
		k_shift_minus<<<grid_for(im->n), 256, 0, c->stream>>>(im->n, im->nb, im->inv_dtau, z, im->F1, out);
		return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
	}
	const double eps = std::sqrt(2.2e-16) * (1.0 + u_norm) / std::max(z_norm, 1e-300);
	k_lincomb3<<<grid_for(im->n), 256, 0, c->stream>>>(im->n, 1.0, im->u, eps, z, im->up);
	int rc = residual(c, im->up, im->F1);
	if (rc) return rc;
	k_shift_minus_fd<<<grid_for(im->n), 256, 0, c->stream>>>(im->n, im->nb, im->inv_dtau, z, im->F1, im->F0, 1.0 / eps,
	                                                          out);
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

static double host_norm2(dpg_gpu_ctx* c, Implicit* im, const double* x, int* rc)
{
	double h;
	*rc = multidot(c, im, 1, x, x, &h);
	return std::sqrt(std::max(h, 0.0));
}

// GMRES(m), right preconditioned, for A du = F0; returns iterations; du in im->du.
static int gmres(dpg_gpu_ctx* c, Implicit* im, int precond, double rtol, int max_it, double u_norm,
                 int* iters, double* rel_res)
{
	const int m = im->m;
	const int64_t n = im->n;
	int rc;
	im->u_traced = false;
	if (cudaMemsetAsync(im->du, 0, n * 8, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	const double bnorm = host_norm2(c, im, im->F0, &rc);
	if (rc) return rc;
	*iters = 0;
	*rel_res = 0.0;
	if (bnorm == 0.0) return DPG_OK;
	double rnorm = bnorm;
	// r = b - A du (du = 0 on the first cycle)
	if (cudaMemcpyAsync(im->V, im->F0, n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	std::vector<double> H((size_t)(m + 1) * m), cs(m), sn(m), g(m + 1), hcol(m + 1);
	while (*iters < max_it) {
		k_axpby<<<grid_for(n), 256, 0, c->stream>>>(n, 1.0 / rnorm, im->V, 0.0, im->V);
		std::fill(g.begin(), g.end(), 0.0);
		g[0] = rnorm;
		int j = 0;
		for (; j < m && *iters < max_it; ++j) {
			double* vj = im->V + (int64_t)j * n;
			double* zj = im->Z + (int64_t)j * n;
			if ((rc = apply_precond(c, im, precond, vj, zj))) return rc;
			double znorm = 0.0;   // only the finite-difference product needs it (its step size)
			if (!im->tangent) {
				znorm = host_norm2(c, im, zj, &rc);
				if (rc) return rc;
			}
			double* w = im->V + (int64_t)(j + 1) * n;
			// the product and classical Gram-Schmidt, twice, and the norm -- all on the device; one copy of the column per
			// iteration
			const int blocks = red_blocks(n);
			const dim3 dots(blocks, (j + kDotChunk) / kDotChunk);
			if (blocks <= kSmallBlocks) {
				if (im->tangent) {
					if ((rc = apply_J(c, im, zj))) return rc;
					k_multidot_partial<<<dots, kRedThreads, 0, c->stream>>>(n, j + 1, im->V, n, w, im->partial, im->nb, im->inv_dtau,
					                                                        zj, im->F1);
				} else {
					if ((rc = apply_A(c, im, zj, w, u_norm, znorm))) return rc;
					k_multidot_partial<<<dots, kRedThreads, 0, c->stream>>>(n, j + 1, im->V, n, w, im->partial);
				}
				double* norm_partial = im->partial + (size_t)(m + 1) * kRedBlocks;
				const size_t sm_h = (size_t)(j + 1) * 8;
				k_gs_pass<<<blocks, kRedThreads, sm_h, c->stream>>>(n, j + 1, im->V, n, im->partial, im->h, w, nullptr);
				k_multidot_partial<<<dots, kRedThreads, 0, c->stream>>>(n, j + 1, im->V, n, w, im->partial);
				k_gs_pass<<<blocks, kRedThreads, sm_h, c->stream>>>(n, j + 1, im->V, n, im->partial, im->h2, w, norm_partial);
				k_gs_finish<<<blocks, kRedThreads, 0, c->stream>>>(n, j, norm_partial, im->h, im->h2, w);
			} else {
				if ((rc = apply_A(c, im, zj, w, u_norm, znorm))) return rc;
				k_multidot_partial<<<dots, kRedThreads, 0, c->stream>>>(n, j + 1, im->V, n, w, im->partial);
				k_reduce_partials<<<j + 1, 256, 0, c->stream>>>(j + 1, blocks, im->partial, im->h);
				k_sub_combination<<<grid_for(n), 256, 0, c->stream>>>(n, j + 1, im->V, n, im->h, w);
				k_multidot_partial<<<dots, kRedThreads, 0, c->stream>>>(n, j + 1, im->V, n, w, im->partial);
				k_reduce_partials<<<j + 1, 256, 0, c->stream>>>(j + 1, blocks, im->partial, im->h2);
				k_sub_combination<<<grid_for(n), 256, 0, c->stream>>>(n, j + 1, im->V, n, im->h2, w);
				k_multidot_partial<<<blocks, kRedThreads, 0, c->stream>>>(n, 1, w, n, w, im->partial);
				k_reduce_partials<<<1, 256, 0, c->stream>>>(1, blocks, im->partial, im->h2 + j + 1);
				k_column_finish<<<1, 256, 0, c->stream>>>(j, im->h, im->h2);
				k_scale_inv<<<grid_for(n), 256, 0, c->stream>>>(n, w, im->h + j + 1);
			}
			if (cudaMemcpyAsync(im->hcol_host, im->h, 8 * (j + 2), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
			    cudaStreamSynchronize(c->stream) != cudaSuccess)
				return DPG_ERR_CUDA;
			for (int i = 0; i <= j + 1; ++i) hcol[i] = im->hcol_host[i];
			const double hn = hcol[j + 1];
			if (!std::isfinite(hn)) return DPG_ERR_NONFINITE;
			// Givens rotations
			for (int i = 0; i < j; ++i) {
				const double t = cs[i] * hcol[i] + sn[i] * hcol[i + 1];
				hcol[i + 1] = -sn[i] * hcol[i] + cs[i] * hcol[i + 1];
				hcol[i] = t;
			}
			const double den = std::hypot(hcol[j], hcol[j + 1]);
			cs[j] = den > 0 ? hcol[j] / den : 1.0;
			sn[j] = den > 0 ? hcol[j + 1] / den : 0.0;
			hcol[j] = den;
			hcol[j + 1] = 0.0;
			g[j + 1] = -sn[j] * g[j];
			g[j] = cs[j] * g[j];
			for (int i = 0; i <= j; ++i) H[(size_t)i * m + j] = hcol[i];
			++*iters;
			if (std::fabs(g[j + 1]) <= rtol * bnorm || hn == 0.0) { ++j; break; }
		}
		// y = H^-1 g (upper triangular j x j), du += Z y
		std::vector<double> y(j);
		for (int i = j - 1; i >= 0; --i) {
			double s = g[i];
			for (int k = i + 1; k < j; ++k) s -= H[(size_t)i * m + k] * y[k];
			y[i] = s / H[(size_t)i * m + i];
		}
		cudaMemcpyAsync(im->h, y.data(), 8 * j, cudaMemcpyHostToDevice, c->stream);
		k_add_combination<<<grid_for(n), 256, 0, c->stream>>>(n, j, im->Z, n, im->h, im->du);
		rnorm = std::fabs(g[j]);
		*rel_res = rnorm / bnorm;
		if (rnorm <= rtol * bnorm) break;
		// restart: r = b - A du
		const double dun = host_norm2(c, im, im->du, &rc);
		if (rc) return rc;
		if ((rc = apply_A(c, im, im->du, im->w, u_norm, dun))) return rc;
		k_lincomb3<<<grid_for(n), 256, 0, c->stream>>>(n, 1.0, im->F0, -1.0, im->w, im->V);
		rnorm = host_norm2(c, im, im->V, &rc);
		if (rc) return rc;
		*rel_res = rnorm / bnorm;
		if (rnorm <= rtol * bnorm) break;
	}
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

int implicit_solve(dpg_gpu_ctx* c, const dpg_newton_params* prm, dpg_newton_stats* st)
{
	const int m = std::max(2, std::min(prm->gmres_restart, 512));
	int rc;
	Implicit* im = implicit_state(c, m);
	if (!im) return DPG_ERR_CUDA;
	if (prm->precond == DPG_PRECOND_MLP && !c->mlp) return DPG_ERR_INVALID;
	if (prm->jacobian != DPG_JACOBIAN_TANGENT && prm->jacobian != DPG_JACOBIAN_FD) return DPG_ERR_INVALID;
	if (prm->precond < DPG_PRECOND_NONE || prm->precond > DPG_PRECOND_BLOCK_ILU) return DPG_ERR_INVALID;
	if (!(prm->cfl_initial >= 0.0)) return DPG_ERR_INVALID;
	if (prm->cfl_initial > 0.0 && c->n_var > 1 && !c->bez_full) return DPG_ERR_UNSUPPORTED;
	if (c->pos_dense) return DPG_ERR_UNSUPPORTED;   // the relaxed update of the Newton step: tensor-product volumes
	if (prm->precond == DPG_PRECOND_BLOCK_ILU) {
		if (prm->ilu_order != DPG_ILU_ORDER_VOLUME && prm->ilu_order != DPG_ILU_ORDER_COLOUR) return DPG_ERR_INVALID;
		if (prm->ilu_parts < 0) return DPG_ERR_INVALID;
		if ((rc = ilu_build(c, im, prm->ilu_order, prm->ilu_parts))) return rc;
	}
	im->tangent = prm->jacobian == DPG_JACOBIAN_TANGENT;
	if (im->tangent && ensure_tangent_buffers(c)) return DPG_ERR_CUDA;
	memset(st, 0, sizeof *st);
	const auto t0 = std::chrono::steady_clock::now();
	im->forcing = nullptr;
	if (prm->forcing) {
		if (!im->forcing_buf && cudaMalloc(&im->forcing_buf, im->n * 8) != cudaSuccess) return DPG_ERR_CUDA;
		if (cudaMemcpy(im->forcing_buf, prm->forcing, im->n * 8, cudaMemcpyHostToDevice) != cudaSuccess) return DPG_ERR_CUDA;
		im->forcing = im->forcing_buf;
	}
	if (cudaMemcpyAsync(im->u, c->sol, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	double fmax0 = 0.0;
	if ((rc = residual(c, im->u, im->F0))) return rc;
	if ((rc = absmax(c, im, im->F0, &fmax0))) return rc;
	double fmax = fmax0;
	st->residual_initial = fmax0;
	int k = 0;
	for (; k < prm->max_newton && fmax > prm->tol; ++k) {
		const double dtau = std::min(prm->dtau0 * fmax0 / fmax, prm->dtau_max);
		const double cfl = prm->cfl_initial * std::max(1.0, fmax0 / fmax);
		if (prm->cfl_initial > 0.0)
			k_pseudo_dt<<<(c->g.n_vol + 7) / 8, 256, 0, c->stream>>>(c->g.n_vol, c->g.n_s, c->n_var, im->u, c->bez_full,
			                                                         c->h_min, c->adv_speed, c->visc_mu, cfl,
			                                                         im->inv_dtau);
		else
			k_fill<<<grid_for(c->g.n_vol), 256, 0, c->stream>>>(c->g.n_vol, 1.0 / dtau, im->inv_dtau);
		const double u_norm = host_norm2(c, im, im->u, &rc);
		if (rc) return rc;
		int pc = prm->precond;
		if (pc == DPG_PRECOND_BLOCK_JACOBI) {
			const auto ta = std::chrono::steady_clock::now();
			if ((rc = assemble_block_jacobi(c, im, im->F0))) return rc;
			st->assembly_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - ta).count();
			if (prm->collect_blocks && c->mlp) mlp_collect(c, im->u, im->blocks, im->piv, im->inv_dtau, im->rho);
		} else if (pc == DPG_PRECOND_MLP) {
			if ((rc = mlp_predict(c, im->u, im->inv_dtau, &im->P))) return rc;
		} else if (pc == DPG_PRECOND_BLOCK_ILU) {
			const auto ta = std::chrono::steady_clock::now();
			if ((rc = assemble_block_ilu(c, im, im->F0))) return rc;
			st->assembly_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - ta).count();
		}
		int its = 0;
		double rel = 0.0;
		if ((rc = gmres(c, im, pc, prm->gmres_rtol, prm->max_gmres, u_norm, &its, &rel))) return rc;
		st->gmres_iterations += its;
		if (pc == DPG_PRECOND_MLP && rel > 10.0 * prm->gmres_rtol) {
			// the learned inverse did not give a converged Krylov solve: redo the step with exact block-Jacobi
			const auto ta = std::chrono::steady_clock::now();
			if ((rc = assemble_block_jacobi(c, im, im->F0))) return rc;
			st->assembly_seconds += std::chrono::duration<double>(std::chrono::steady_clock::now() - ta).count();
			if ((rc = gmres(c, im, DPG_PRECOND_BLOCK_JACOBI, prm->gmres_rtol, prm->max_gmres, u_norm, &its, &rel)))
				return rc;
			st->gmres_iterations += its;
			++st->fallback_steps;
		}
		// u += du ; F0 = F(u).  With positivity (Euler) the update is under-relaxed per volume and limited as in the
		// reference (update_coef_s_v, solve_implicit.c:724-731, 821-873).  A step that produces a non-finite residual
		// or breaks positivity beyond repair (where the reference stops) is undone and the pseudo time step of the next
		// attempt is reduced (fmax0 scaled so that dtau halves).
		if (cudaMemcpyAsync(im->up, im->u, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess)
			return DPG_ERR_CUDA;
		if (c->positivity) {
			if ((rc = launch_relaxed_update(c, im->u, im->du))) return rc;
			if ((rc = launch_positivity(c, im->u))) return rc;
		} else {
			k_axpby<<<grid_for(im->n), 256, 0, c->stream>>>(im->n, 1.0, im->du, 1.0, im->u);
		}
		const int pos_bad = positivity_error(c);
		if (pos_bad < 0) return DPG_ERR_CUDA;
		double fnew = 0.0;
		rc = pos_bad ? DPG_ERR_NONFINITE : residual(c, im->u, im->F0);
		if (rc == DPG_OK) rc = absmax(c, im, im->F0, &fnew);
		if (rc == DPG_ERR_NONFINITE) {
			if (cudaMemcpyAsync(im->u, im->up, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess)
				return DPG_ERR_CUDA;
			if ((rc = residual(c, im->u, im->F0))) return rc;
			if ((rc = absmax(c, im, im->F0, &fnew))) return rc;
			fmax0 *= 0.5;
			++st->rejected_steps;
			if (prm->verbose) printf("newton %2d  rejected (non-finite state), dtau halved\n", k);
		} else if (rc) {
			return rc;
		}
		fmax = fnew;
		if (prm->verbose)
			printf("newton %2d  %s %.3e  gmres %3d (rel %.2e)  ||F||_inf %.3e\n", k,
			       prm->cfl_initial > 0.0 ? "cfl" : "dtau", prm->cfl_initial > 0.0 ? cfl : dtau, its, rel, fmax);
	}
	st->newton_iterations = k;
	st->residual_final = fmax;
	if (cudaMemcpyAsync(c->sol, im->u, im->n * 8, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	if (cudaStreamSynchronize(c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	st->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
	return fmax <= prm->tol ? DPG_OK : DPG_ERR_NOT_CONVERGED;
}

} // namespace dpg
