// One-dimensional operators of the tensor-product elements (QUAD, HEX) and the device passes that apply them one
// direction at a time.
//
// The solution nodes are Gauss-Lobatto points, the cubature nodes of volumes and faces Gauss points, n1 = p + 1 of
// both per direction.  Every dense operator of the residual is a Kronecker product of 1D factors, and the
// mass matrix with that cubature is diagonal in the Lagrange basis of the Gauss points (the collocated basis):
//     cv0_vs_vc           = B (x) B (x) B                     B[q][i]  GLL Lagrange polynomial i at Gauss point q
//     cv0_vs_fc           = l(+-1)^T in the face's direction of the collocated values
//     m_inv tw1_vt_vc[r]  = B^-1 (x) .. diag(1 / detJ) Dw_r    Dw[i][j] = w_j / w_i l_i'(x_j)
//     m_inv tw0_vt_fc     = B^-1 (x) .. diag(1 / detJ) l_i(+-1) / w_i
// (for a non-affine element too: 1 / detJ is then one number per Gauss point).  An n1^d x n1^d product becomes d
// passes of n1 terms, a face lift one term per node.
#pragma once

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "dpg_gpu_internal.cuh"
#include "flux.cuh"

namespace dpg {
namespace tp {

constexpr int kN1Max = 5;   // orders 1..4

// Kernel parameter (constant bank), copied to shared memory by each block.
template <int N1>
struct Ops {
	double B[N1 * N1];     // [q][i]  GLL -> Gauss values
	double Bi[N1 * N1];    // [i][q]  its inverse
	double Dw[N1 * N1];    // [i][j]  weak derivative over the weights
	double Ds[N1 * N1];    // [i][j]  l_j'(x_i)
	double lm[N1], lp[N1]; // collocated basis at -1 and +1
	double wm[N1], wp[N1]; // the same over the weights
	double lwm[N1], lwp[N1]; // lm wm, lp wp
};

// Host state of a tensor-product context (dpg_gpu_ctx::tp).
struct TpState {
	int n1 = 0, E = 1;          // order + 1, elements per block
	bool own = false;           // small meshes: k_tp_lift and k_tp_stage form their elements' face fluxes
	double* trace2 = nullptr;   // own: the traces of every other stage
	double* G = nullptr;        // [n_vol][n_var][n1^d] weak divergence in the collocated basis
	double* jn = nullptr;       // non-affine: [n_vol][n1^d] 1 / detJ at the Gauss points
	double B[25], Bi[25], Dw[25], Ds[25], lm[5], lp[5], wm[5], wp[5];
	// boundary faces and viscous terms (kernels_tp_general.cu)
	int viscous = 0;
	double mu = 0.0, kappa = 0.0, scale = 0.0;   // viscosity, gamma mu / Pr, BR2 penalty 1.01 NFMAX
	BcParams bp{};
	const int* bc = nullptr;    // [n_face] 0 or the boundary code; null without boundary faces
	const double* xyz = nullptr;// [n_face][n_fc][d]
	double* Uc = nullptr;       // viscous: [n_dof] collocated values
	double* fvn = nullptr;      // viscous: [n_face][2][n_var][n_fc] normal second-order flux of each side
	std::vector<void*> allocs;
};

struct TpGeo {
	int n_vol, affine;
	const double* met;          // affine: [n_vol][d d]; else [n_vol][d d][n1^d]
	const double* jinv;         // affine: [n_vol]; else [n_vol][n1^d]
	const int* vol_face;        // [n_vol][2 d]  (face << 1) | side
	const int* nc_inv;          // [n_face][n_fc]
};

// What a kernel needs to form the numerical fluxes of its elements' faces by itself.
struct TpFaces {
	const double* trace;        // [n_face][2][n_var][n_fc]
	const int* nc;              // [n_face][n_fc]
	const double* nrm;          // [n_face][n_fc][d]
	const double* jf;           // [n_face][n_fc]
	int num_flux;
	double b[3];
};

// What boundary faces add: their codes and the positions and normals of the face nodes.
struct TpBc {
	const int* bc;
	const double* xyz;
	const double* nrm;
	BcParams bp;
};

template <int N1>
inline Ops<N1> ops_of(const TpState* st)
{
	Ops<N1> o;
	for (int k = 0; k < N1 * N1; ++k) { o.B[k] = st->B[k]; o.Bi[k] = st->Bi[k]; o.Dw[k] = st->Dw[k]; o.Ds[k] = st->Ds[k]; }
	for (int k = 0; k < N1; ++k) {
		o.lm[k] = st->lm[k]; o.lp[k] = st->lp[k]; o.wm[k] = st->wm[k]; o.wp[k] = st->wp[k];
		o.lwm[k] = st->lm[k] * st->wm[k]; o.lwp[k] = st->lp[k] * st->wp[k];
	}
	return o;
}

inline TpGeo geo_of(const dpg_gpu_ctx* c)
{
	const TpState* st = (const TpState*)c->tp;
	const GroupDev& g = c->g;
	return TpGeo{g.n_vol, g.affine, g.met, g.affine ? g.jinv : st->jn, g.vol_face, g.nc_inv};
}

inline TpFaces faces_of(const dpg_gpu_ctx* c, const double* trace)
{
	return {trace, c->fc.nc, c->fc.nrm, c->fc.jf, c->num_flux, {c->b_adv[0], c->b_adv[1], c->b_adv[2]}};
}
constexpr int most_elems(int N) { return 256 / N; }   // elements per block: at most 256 threads of one node each

// A launch of a kernel of <D, NV, N1> by the context's sizes.
#define DPG_TP_N1(F, D, NV, ...)                        \
	switch (((const TpState*)c->tp)->n1) {              \
	case 2: return F<D, NV, 2>(__VA_ARGS__);            \
	case 3: return F<D, NV, 3>(__VA_ARGS__);            \
	case 4: return F<D, NV, 4>(__VA_ARGS__);            \
	case 5: return F<D, NV, 5>(__VA_ARGS__);            \
	default: return DPG_ERR_UNSUPPORTED;                \
	}
#define DPG_TP_DISPATCH(F, ...)                                             \
	do {                                                                    \
		if (c->d == 2 && c->n_var == 4) { DPG_TP_N1(F, 2, 4, __VA_ARGS__) } \
		if (c->d == 3 && c->n_var == 5) { DPG_TP_N1(F, 3, 5, __VA_ARGS__) } \
		if (c->d == 2 && c->n_var == 1) { DPG_TP_N1(F, 2, 1, __VA_ARGS__) } \
		if (c->d == 3 && c->n_var == 1) { DPG_TP_N1(F, 3, 1, __VA_ARGS__) } \
		return DPG_ERR_UNSUPPORTED;                                         \
	} while (0)

template <int N1>
__device__ __forceinline__ void load_ops(Ops<N1>* s, const Ops<N1>& p)
{
	constexpr int n = (int)(sizeof(Ops<N1>) / sizeof(double));
	const double* src = reinterpret_cast<const double*>(&p);
	for (int k = threadIdx.x; k < n; k += blockDim.x) reinterpret_cast<double*>(s)[k] = src[k];
}

__host__ __device__ constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }

// Node i's value of one direction's pass over an array of n1^d nodes: sum_j op[i_a][j] x[.. j ..].
template <int A, int N1, class T>
__device__ __forceinline__ T pencil_dot(const double* row, const T* x, int base)
{
	constexpr int S = ipow(N1, A);
	T acc = row[0] * x[base];
#pragma unroll
	for (int j = 1; j < N1; ++j) acc += row[j] * x[base + j * S];
	return acc;
}
// A thread per face node too, as far as a block goes.
template <int D, int N1>
inline int own_threads(int E)
{
	const int n = ipow(N1, D), nf = 2 * D * ipow(N1, D - 1);
	return std::min(256, (E * (n > nf ? n : nf) + 31) / 32 * 32);
}

// Position of node i along direction A, and the first node of its pencil.
template <int A, int N1>
__device__ __forceinline__ int node_along(int i) { return (i / ipow(N1, A)) % N1; }
template <int A, int N1>
__device__ __forceinline__ int pencil_base(int i) { return i - node_along<A, N1>(i) * ipow(N1, A); }

// Face node q of direction a: the first node of its pencil; node i's face node.
template <int N1>
__device__ __forceinline__ int face_base(int a, int q)
{
	const int S = a == 0 ? 1 : (a == 1 ? N1 : N1 * N1);
	return (q % S) + (q / S) * (S * N1);
}
template <int A, int N1>
__device__ __forceinline__ int face_node(int i)
{
	constexpr int S = ipow(N1, A);
	return (i % S) + (i / (S * N1)) * S;
}

template <int N1>
__device__ __forceinline__ constexpr int stride_of(int a) { return a == 0 ? 1 : (a == 1 ? N1 : N1 * N1); }

// Reference volume flux of one node, handed to emit(r, fr_r) direction by direction: fr_r[eq] = sum_x m_xr f[x][eq]
// in contravariant form (the velocity along r once per direction instead of d products per equation).
template <int D, int NV, class T, class Met, class Emit>
__device__ __forceinline__ void ref_flux(const T* s, const Met& met, const double* b, Emit&& emit)
{
	if constexpr (NV == D + 2) {
		const T rho_inv = 1.0 / s[0], E = s[D + 1];
		T q = 0.0;   // (rho V)^2
#pragma unroll
		for (int a = 0; a < D; ++a) q += s[1 + a] * s[1 + a];
		const T p = DPG_GM1_D * (E - 0.5 * (q * rho_inv)), Ep = E + p;
#pragma unroll
		for (int r = 0; r < D; ++r) {
			double m[D];
#pragma unroll
			for (int x = 0; x < D; ++x) m[x] = met(x, r);
			T f0 = m[0] * s[1];
#pragma unroll
			for (int x = 1; x < D; ++x) f0 += m[x] * s[1 + x];
			const T W = f0 * rho_inv;
			T fr[NV];
			fr[0] = f0;
#pragma unroll
			for (int a = 0; a < D; ++a) fr[1 + a] = s[1 + a] * W + m[a] * p;
			fr[D + 1] = Ep * W;
			emit(r, fr);
		}
	} else {
#pragma unroll
		for (int r = 0; r < D; ++r) {
			T fr[NV];
			double mb = 0.0;
#pragma unroll
			for (int x = 0; x < D; ++x) mb += met(x, r) * b[x];
			fr[0] = mb * s[0];
			emit(r, fr);
		}
	}
}

__device__ __forceinline__ unsigned long long abs_bits_of(double v)
{
	return (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
}

// max |v| of the block (IEEE bits: NaN orders above +inf) into *slot; every thread calls.
__device__ __forceinline__ void block_max_to(unsigned long long m, unsigned long long* s_max, unsigned long long* slot)
{
	if (threadIdx.x == 0) *s_max = 0ull;
	__syncthreads();
	for (int o = 16; o > 0; o >>= 1) {
		const unsigned long long t = __shfl_xor_sync(0xffffffffu, m, o);
		m = t > m ? t : m;
	}
	if ((threadIdx.x & 31) == 0) atomicMax(s_max, m);
	__syncthreads();
	if (threadIdx.x == 0) atomicMax(slot, *s_max);
}

} // namespace tp
} // namespace dpg
