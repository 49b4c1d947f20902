// Device context and kernel launch declarations shared by the CUDA translation units.
#pragma once

#include <vector>
#include <cstdint>
#include <cuda_runtime.h>

#include "batch_alloc.h"
#include "dpg_gb300.h"
#include "dpg_simulation.h"

namespace dpg {

constexpr int kMaxStages = 3;

// Per-group device tables (one group = one (element type, order); the structured meshes of this path have one).
struct GroupDev {
	int n_vol, n_s, n_c, n_fl, n_fc, K;    // K = d*n_c + n_fl*n_fc (lift contraction length)
	const double* Cv;      // [n_c  x n_s]        cv0_vs_vc
	const double* Cf;      // [n_fl*n_fc x n_s]   cv0_vs_fc stacked over local faces
	const double* L;       // [n_s  x K]          [tw1_vt_vc[0..d) | -tw0_vt_fc[0..n_fl)], pre-multiplied by
	                       //                     m_inv_ref when every volume is affine
	const double* met;     // affine: [n_vol][d*d] (m_ij at i + d*j); else [n_vol][d*d][n_c]
	const double* jinv;    // [n_vol] 1/detJ (affine)
	const double* minv;    // [n_vol][n_s*n_s] (non-affine) or nullptr
	const int* vol_face;   // [n_vol][n_fl]  (face << 1) | side
	const int* nc_inv;     // [n_face][n_fc] inverse of nc_fc
	int affine;
};

struct FaceDev {
	int n_face, n_fc;
	const double* nrm;     // [n_face][n_fc][d]
	const double* jf;      // [n_face][n_fc]
	const int* nc;         // [n_face][n_fc]
};

// Work space of the linearisation for nb directions at once (their arrays one after another).
struct TanWork {
	int nb = 0;
	double* trace_t = nullptr;  // [nb][n_face][2][n_var][n_fc] tangents of the traces
	double* nnf_t = nullptr;    // [nb][n_face][n_var][n_fc]    tangents of the face fluxes
	double* G = nullptr;        // tensor-product meshes: [nb][n_dof] weak divergence
	double* Uc_t = nullptr;     // viscous: [nb][n_dof] collocated tangents
	double* fvn = nullptr;      // viscous: [nb][n_face][2][n_var][n_fc]
	bool u_traced = false;      // dense kernels: the traces of u are in place (ctx.trace)
};

// Strides between the directions of a launch (blockIdx.y): state-sized arrays, traces, face fluxes.
struct TanStride {
	size_t dof = 0, tr = 0, nf = 0;
};

} // namespace dpg

struct dpg_gpu_ctx {
	int dev = 0;
	cudaStream_t stream = nullptr;
	int d = 0, n_var = 0, n_eq = 0, pde = 0, num_flux = 0;
	int e_type = 0;             // element type of the (single) group (DPG_QUAD, DPG_HEX, DPG_TRI)
	double b_adv[3] = {0, 0, 0};
	int64_t n_dof = 0;

	dpg::GroupDev g{};
	dpg::FaceDev fc{};

	// state
	double* sol = nullptr;
	double* solp = nullptr;
	double* rhs = nullptr;
	double* trace = nullptr;    // [n_face][2][n_var][n_fc], each side in its own node order
	double* nnf = nullptr;      // [n_face][n_eq][n_fc], left node order, scaled by jacobian_det_fc
	unsigned long long* dmax = nullptr;   // [kMaxStages+1] max |rhs| bit patterns
	double* ddt = nullptr;      // device copy of dt (graph parameter)

	// owned device allocations (freed at destroy)
	void* allocs[32] = {};
	int n_allocs = 0;

	// precision
	int prec_mode = DPG_PREC_FP64;
	int n_slices = 0;
	void* split = nullptr;      // split-precision state (split_ops.cu)

	// CUDA graph of one SSP-RK3 step
	cudaGraphExec_t step_graph = nullptr;
	int step_graph_mode = -1;

	int n_sm = 1;
	int vol_block_elems = 1;
	int trace_block_elems = 1;
	int tan_block_elems = 1;     // elements per block of the linearisation's volume kernel
	dpg::TanWork tan;            // one direction (allocated on the first Jacobian-vector product)

	// positivity of density and pressure (Euler): limiter after every RK stage and Newton update (positivity.cu)
	int positivity = 0;          // on by default for Euler, as the reference's test_case_requires_positivity
	int pos_n1 = 0;              // solution points per direction
	double* bez1 = nullptr;      // [n1 x n1] Bernstein polynomials at the GLL nodes (Bezier -> solution coefficients)
	double* bez1_inv = nullptr;  // [n1 x n1] its inverse
	int pos_dense = 0;           // simplices, mixed orders: dense Bezier operators (no 1D factors)
	// the dense limiter per order group: its volumes (null: all, one order), operators (dense_limiter_tables), screen bound
	struct PosGroup { int n_vol, ns; const int* vols; const float* screen; const double *sbT, *bsT; float amp; };
	PosGroup pos_grp[DPG_P_MAX] = {};
	int n_pos_grp = 0;
	const int64_t* pos_dof_off = nullptr;   // [n_vol + 1], or null (one order)
	// local pseudo time steps of the implicit solve (the reference's CFL ramping)
	double* h_min = nullptr;     // [n_vol] shortest edge of each volume (chord between its end vertices)
	double* bez_full = nullptr;  // [n_s x n_s] solution -> Bezier coefficients (ccSB0_vs_vs), Euler-like PDEs
	double visc_mu = 0.0;        // constant viscosity (Navier-Stokes), 0 without second-order terms
	double adv_speed = 0.0;      // |b_adv| (advection)
	double bez1_host[50] = {};   // host copies: bez1 at [0, n1^2), bez1_inv at [25, 25 + n1^2) (kernel parameters)
	float pos_amp = 0.f;         // FP32 screen: bound of the coefficient error per unit of |A^-1| |u|
	int* pos_err = nullptr;      // bit 0: an average density / pressure below EPS_PHYS; bit 1: relaxation underflow
	double* jv_buf = nullptr;    // [2][n_dof] direction and product of dpg_gpu_jacobian_apply
	double* du_buf = nullptr;    // [n_dof] device copy of a host Newton update (dpg_gpu_positivity_update)

	void* tp = nullptr;         // QUAD / HEX of one order: 1D operators of the FP64 form (kernels_tp.cu)
	int walls_or_visc = 0;      // boundary faces or viscous terms: FP64 only, kernels_tp_general.cu (advection above p = 4:
	                            // the dense kernels, boundary traces copied)
	const int* bface = nullptr; // [n_bface] the boundary faces of that case
	int n_bface = 0;
	void* oz = nullptr;         // simplices: FP64 dense products on the tensor cores (kernels_oz.cu)
	void* hp = nullptr;         // mixed orders: volumes grouped by order (kernels_hp.cu)
	void* adv = nullptr;        // one order, simplices, advection: the same for the FP64 residual
	void* implicit = nullptr;   // Newton-GMRES work space (implicit.cu)
	void* mlp = nullptr;        // learned preconditioner (mlp.cu)
};

namespace dpg {
// The kernels of a residual are a chain, each a few us long on small meshes: the next kernel's launch is processed while the
// previous one runs (programmatic dependent launch), and its blocks wait for that kernel's end and memory before they
// touch anything a kernel writes.  In every kernel launched by launch_chained each thread that reads or writes what another
// kernel writes calls grid_wait before it does, and every block has such threads (in ks_* and k_oz_* the compute warps; the
// loading and issuing warps touch operators and shared memory only).  So a kernel that has ended means that all before it have.
// Inputs that another kernel writes are not `__restrict__`: such loads count as invariant (or as untouched by the wait),
// may be moved above it and go through the read-only path.  Blocks of small grids (at most half of the 152 SMs: two grids
// fit side by side) let the next kernel's blocks start at once (16x16 QUAD p = 2, 36 stages: 870 us with plain launches,
// 834 without this, 788 with it); for larger grids the early blocks pack onto the first free SMs and share their FP64
// pipes (61x47 QUAD p = 3: 473 us without, 553 with it).
__device__ __forceinline__ void grid_wait()
{
	if (gridDim.x * gridDim.y <= 76) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Threads per block (32, 64 or 128) of a kernel of n independent threads that the FP64 pipe bounds: the fewest warps on the
// fullest SM, since a warp's FP64 instruction holds its SM's pipe for ~20 cycles whoever else is idle.
inline int spread_threads(int64_t n, int n_sm)
{
	int best = 128;
	int64_t cost = INT64_MAX;
	for (int t = 128; t >= 32; t /= 2) {
		const int64_t blocks = (n + t - 1) / t, c = (blocks + n_sm - 1) / n_sm * (t / 32);
		if (c < cost) { cost = c; best = t; }
	}
	return best;
}

template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args)
{
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = stream;
	cudaLaunchAttribute at{};
	at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at.val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = &at;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Shared-memory opt-in of a kernel without static shared memory: the device's largest block, for every context of the process.
// The attribute belongs to the function: a limit of this context's size would refuse the launches of an earlier one with larger
// blocks.
constexpr int kSmemOptIn = 227 * 1024;
inline bool allow_smem(const void* kernel)
{
	return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemOptIn) == cudaSuccess;
}

// Up to this many face nodes of a mesh its volume or lift kernels form their elements' face fluxes themselves.
constexpr int64_t kOwnFaceNodes = 10000;

int launch_trace (dpg_gpu_ctx* c);
int launch_face  (dpg_gpu_ctx* c);
int launch_face_tan(dpg_gpu_ctx* c, const TanWork& w);   // tangents of the face fluxes
TanStride tan_stride(const dpg_gpu_ctx* c);
int launch_volume(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot);
// J v = d(m_inv rhs)/du . v at u (FP64 formulas, forward-mode tangents) for w.nb directions v[nb][n_dof] -> out[nb][n_dof]
// in one set of launches.
int jvp_fp64(dpg_gpu_ctx* c, const double* u, const double* v, double* out, const TanWork& w);
int ensure_tangent_buffers(dpg_gpu_ctx* c);             // c->tan
size_t tangent_bytes(const dpg_gpu_ctx* c);             // of a TanWork, per direction
// w for the largest batch up to `most` directions that fits (w->nb), with more buffers of the same batch: all or none
int alloc_tangent_work(dpg_gpu_ctx* c, int most, TanWork* w, std::initializer_list<DirBuffer> more = {});
void free_tangent_work(TanWork* w);

// tensor-product elements (kernels_tp.cu): traces and weak divergence, then lift, stage and norm; the tangents of the
// linearisation.  tp_prepare leaves c->tp null where the dense kernels run.
int  tp_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim, bool general);
int  tp_volume(dpg_gpu_ctx* c);
int  tp_lift(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot);
int  tp_volume_tan(dpg_gpu_ctx* c, const double* u, const double* v, const TanWork& w);
int  tp_lift_tan(dpg_gpu_ctx* c, const TanWork& w, double* out);
bool dense_own_faces(const dpg_gpu_ctx* c);  // no k_face: the dense volume kernel forms its elements' face fluxes
bool tp_own_faces(const dpg_gpu_ctx* c);     // the same: the lift and stage kernels form their elements' face fluxes
bool tp_viscous(const dpg_gpu_ctx* c);
void tp_free(dpg_gpu_ctx* c);
int  tp_general_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim);   // boundary faces, BR2 (after tp_prepare)
int  tp_general_residual(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot);
int  tp_general_jvp(dpg_gpu_ctx* c, const double* u, const double* v, double* out, const TanWork& w);
int  tp_general_launches(dpg_gpu_ctx* c);
int  tp_general_front(dpg_gpu_ctx* c);     // its first kernel, and those up to the face fluxes (the fused stages of tp_step)
int  tp_general_fluxes(dpg_gpu_ctx* c);
int  tp_configure_stage(dpg_gpu_ctx* c);
int  tp_step(dpg_gpu_ctx* c, unsigned long long* max_slots);   // one SSP-RK3 step with the limiter (kernels_tp_stage.cu)

// mixed orders (kernels_hp.cu): FP64 residual over volume groups of each order; which = 0 traces, 1 face fluxes,
// 2 volume terms (with the RK stage)
int  hp_residual(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot);
int  hp_launches(const dpg_gpu_ctx* c);
bool hp_steps(const dpg_gpu_ctx* c);                            // advection on affine elements:
int  hp_step(dpg_gpu_ctx* c, unsigned long long* max_slots);   // one SSP-RK3 step
int  hp_launch_part(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot);
void hp_free(dpg_gpu_ctx* c);

// simplices of enough work: FP64 residual with sliced operator products on the tensor cores (kernels_oz.cu); which as above
struct OzTables {                       // device tables of the context, by order (index into dpg_sim.ops)
	int n_groups = 0;                   // mixed orders: > 0
	const int* vols[DPG_P_MAX] = {};
	const double* met[DPG_P_MAX] = {};
	const double* jinv[DPG_P_MAX] = {};
	const int64_t* dof_off = nullptr;
	const int* vol_face = nullptr;
	const int* face_p = nullptr;
	const int64_t* fnode_off = nullptr;
	const int* node_face = nullptr;
	const int *nc = nullptr, *nc_inv = nullptr;
	const double* nrm = nullptr;
	const double* jf = nullptr;
};
int  hp_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim, const OzTables* share);
OzTables hp_tables(const dpg_gpu_ctx* c, const struct dpg_sim* sim);
int  oz_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim, const OzTables& tab);
int  oz_ready(dpg_gpu_ctx* c);
int  oz_residual(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot);
int  oz_launch_part(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot);
int  oz_error(dpg_gpu_ctx* c);
void oz_free(dpg_gpu_ctx* c);

// split-precision path (split_ops.cu)
int  split_prepare(dpg_gpu_ctx* c);
void split_free(dpg_gpu_ctx* c);
int  split_launch_trace (dpg_gpu_ctx* c);   // interpolation kernel (traces + volume fluxes)
int  split_launch_face  (dpg_gpu_ctx* c);
int  split_launch_volume(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot);
int  split_error(dpg_gpu_ctx* c);   // non-zero when a bounded device wait gave up
using TileConfig = dpg_tile_config;
int  split_get_tiles(dpg_gpu_ctx* c, TileConfig* t);
int  split_set_tiles(dpg_gpu_ctx* c, const TileConfig& t);   // validated; the caller drops the captured step graph
// elements per block of the wave rule: the fewest whole waves of blocks over n_sm SMs (plus extra_waves), elements
// spread evenly, at most 128 / NV data rows
int  wave_rule_eb(int n_vol, int NV, int n_sm, int extra_waves);
void invalidate_step_graph(dpg_gpu_ctx* c);

// residual of the context's precision mode from c->sol into c->rhs (no synchronisation)
int  enqueue_residual_raw(dpg_gpu_ctx* c, unsigned long long* max_slot);

// positivity (positivity.cu): the limiter on a state (no-op when c->positivity is 0) and the Newton update
// u += relax du with the per-volume under-relaxation (positivity on only); errors in c->pos_err
void dense_limiter_tables(const dpg_element_ops& o, std::vector<float>& screen, std::vector<double>& sbT, std::vector<double>& bsT);
int  launch_positivity(dpg_gpu_ctx* c, double* sol);
int  launch_relaxed_update(dpg_gpu_ctx* c, double* u, const double* du);
int  positivity_error(dpg_gpu_ctx* c);   // reads and clears c->pos_err
int  launch_axpy(dpg_gpu_ctx* c, int64_t n, double a, const double* x, double* y);   // y += a x

// implicit path (implicit.cu) and learned preconditioner (mlp.cu)
int  implicit_solve(dpg_gpu_ctx* c, const dpg_newton_params* prm, dpg_newton_stats* st);
void implicit_free(dpg_gpu_ctx* c);
int  mlp_collect(dpg_gpu_ctx* c, const double* u, const double* lu, const int* piv, const double* shift, double rho);
double mlp_rho(dpg_gpu_ctx* c);
int  mlp_predict(dpg_gpu_ctx* c, const double* u, const double* shift, float** P);
void mlp_free(dpg_gpu_ctx* c);
} // namespace dpg
