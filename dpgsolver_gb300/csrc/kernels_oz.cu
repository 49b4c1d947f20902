// FP64 residual of simplex meshes (TRI, TET; one order or an order per element; affine, periodic) with the dense operator
// products on the tcgen05 tensor cores.
//
// Simplex operators have no 1D factors, and the FP64 pipe of this GPU does 0.53 T multiply-adds per second: a TET of order
// 4 needs 110,000 of them per residual (Euler), 93 % in dense products.  Here every product runs as the sliced (Ozaki)
// scheme: operator rows and data columns are scaled by powers of two, cut into S = 8 signed 8-bit digits (62 bits of
// each operand's largest value) held as BF16, and the digit products of level a + b < 8 are accumulated in FP32,
// each level in an accumulator of its own (8 x 64 TMEM columns).  The level sums are joined in 64-bit integers and rounded
// to FP64 once, so an output is a correctly rounded sum up to the digits cut off, 2^-61 K of the largest products.
// An accumulator is exact while its integer sum is below 2^24 (random digits: an rms of 0.02 times that or less).  In the worst
// case, data digits at their extremes in line with the operator's own, levels 0 to 4 stay below it for every element (0.79
// times 2^24 at most), and all levels for every element but the TET of order 4 (K = 439), whose levels 5, 6 and 7 can
// reach 1.01, 1.23 and 1.45 times: an addition above 2^24 rounds by two units, 2^-51 of the largest product or less.
// Residuals against binary128 (TRI, TET, orders 2..4 and mixed; smooth and noisy states): 0.3 to 0.8 of the dense FP64
// kernels' largest error, 0.25 to 0.6 of their mean.  Fluxes, mass matrix scaling, RK stages and norms are FP64
// instructions.  A row with a value that is not finite gives NaN in all its outputs.
//
//   k_oz_interp : rows (element, variable) of the state -> values at the volume cubature nodes and face traces (a local
//                 face's operators for every order its face may have; the one it has is written)
//   k_oz_flux   : numerical flux per face node and reference volume flux per cubature node, into the rows of the lift's
//                 data (the right side of a face negated, in its own node order)
//   k_oz_lift   : data rows -> rhs (operators [tw1 | -tw0[p_f]] times m_inv), 1 / detJ, norm, SSP-RK3 stage
//
// A block holds 128 data rows (the MMA's M): 25 TETs or 32 TRIs of Euler.  24,576 TETs of orders 1..4: 739 us per residual
// (interpolation 239, fluxes 232, lift 268), dense kernels 2,116.  The fluxes are bound by the FP64 pipe (~210 slots per
// node: Roe-Pike and the volume flux); the other two by the chain digits -> MMAs -> accumulators of the one block that
// an SM holds (512 TMEM columns, 193 KB of shared memory): the products are 36 digit pairs per K of 32 columns.
// Moving a chunk's loads to whole sectors of 8 rows (lane = row, 32-byte part) and one barrier arrival per warp instead
// of per thread took the residual from 795 to 779 us.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "split_kernels.cuh"
#include "tp_ops.cuh"

namespace dpg {
namespace oz {

using namespace split;

constexpr int S = 8;
constexpr int kN = 64;                      // output columns of a tile: 8 accumulators of 64 TMEM columns
constexpr int kPart = kRows * 32 * 2;       // one digit part of a 32-wide K chunk of the data
constexpr int kDigSlot = S * kPart;         // 64 KB
constexpr int kOpSlot = S * kN * 32 * 2;    // 32 KB
constexpr int kOffOp = 2 * kDigSlot, kOffTab = kOffOp + 2 * kOpSlot;
constexpr int kMaxFl = 4;                   // local faces of a simplex
constexpr int kSmem = kOffTab + kRows * 4 + kRows * kMaxFl * 12 + 128;
constexpr int kMaxGroups = 4;

struct Group {
	int n_vol, n_s, n_c, blk0, KS, NT, KL, NL, ldx, n_col;
	int64_t node0;              // first of the group's volume nodes in k_oz_flux
	size_t svc0, xl0;           // offsets of the group's rows
	const int* vols;            // volume of each element of the group, or null (all, in order)
	const double* met;          // [n_vol][d d]
	const double* jinv;         // [n_vol]
	const uint8_t* tI;          // [NT][KS][S] operator tiles of kN rows
	const uint8_t* tL;          // [KL][S] tiles of NL rows
	const int *eI, *eL;         // scale exponents of the operator rows
	const int* col;             // [NT kN] output column: cubature node, or 1 << 16 | lf << 12 | p_f << 8 | face node; -1
};

struct Dev {
	int n_groups, n_blocks, n_fl, p_min;
	int64_t n_fnode, n_vnode;
	int n_fc[8];                // face nodes by order
	Group g[kMaxGroups];
	const int64_t* dof_off;     // [n_vol + 1], or null (n_s n_var per volume)
	const int* vol_face;        // [n_vol][n_fl]
	const int* face_p;          // [n_face], or null (one order)
	const int64_t* fnode_off;   // [n_face + 1], or null (n_fc[p_min] per face)
	const int* node_face;       // [n_fnode], or null
	const int* nc;
	const double* nrm;
	const double* jf;
	const int64_t* face_xl;     // [n_face][2] where a side's fluxes go in xl (variable 0, node 0)
	const int* face_ld;         // [n_face][2] row length there
};

__device__ __forceinline__ int group_of(const Dev& d, int blk)
{
	int k = 0;
	while (k + 1 < d.n_groups && d.g[k + 1].blk0 <= blk) ++k;
	return k;
}

// Scale exponent F of a data row from its exponent bound (|x| < 2^e): |x| 2^-F < 1/4.
__device__ __forceinline__ int row_scale(int e) { return col_exp_of(e, S) + 1; }
constexpr int kNonFinite = 1025;            // exp_bound of an infinity or NaN

// MMA stream of one K chunk: slices a of the operator times parts b < S - a of the data into accumulator a + b.
template <int a>
__device__ __forceinline__ void chunk_slices(uint32_t tmem, uint64_t xd, uint64_t od, uint32_t slice_step, uint32_t idesc, bool first)
{
	if constexpr (a < S) {
#pragma unroll
		for (int ks = 0; ks < 2; ++ks)
#pragma unroll
			for (int b = 0; b < S - a; ++b)
				tc::mma_bf16_elect(tmem + (uint32_t)((a + b) * kN), xd + (uint64_t)(b * (kPart >> 4) + 16 * ks),
				                   od + (uint64_t)(a * slice_step + 16 * ks), idesc, (first && ks == 0 && a == 0) ? 0u : 1u);
		chunk_slices<a + 1>(tmem, xd, od, slice_step, idesc, first);
	}
}

// Digits of 8 values of data row m, K columns kk0.. of a chunk.
__device__ __forceinline__ void write_digits(uint8_t* chunk, int m, int kk0, const double (&x)[8], int F)
{
	uint32_t lo[8], hi[8], lead[8];
#pragma unroll
	for (int j = 0; j < 8; ++j) {
		const long long mm = biased_mantissa<S>(x[j], 8 * S - F);
		lo[j] = (uint32_t)mm;
		hi[j] = (uint32_t)((unsigned long long)mm >> 32);
		lead[j] = (uint32_t)((int)(mm >> (8 * (S - 1))) + 128);
	}
	store_slices<S, 0>(chunk + tc::kmajor_offset(m, kk0, 32, 2), kPart, lo, hi, lead);
}

// The double nearest (hi 2^32 + lo) 2^e, |hi|, |lo| < 2^50, with integer instructions only: a conversion, an addition and a
// scaling on the FP64 pipe would cost ~80 cycles of the SM per warp and output.  The 82-bit sum is cut to its top 63 bits
// (at most 0.5 ulp + 2^-10).
__device__ __forceinline__ double joined(long long hi, long long lo, int e)
{
	long long A = hi + (lo >> 32);
	uint32_t B = (uint32_t)lo;
	const bool neg = A < 0;
	if (neg) { A = ~A + (B == 0); B = 0u - B; }
	const int sh = min(__clzll(A) - 1, 32);   // A's leading zeros but the sign's, at most the 32 bits of B
	const unsigned long long X = ((unsigned long long)A << sh) | ((unsigned long long)B >> (32 - sh));
	const int lz = __clzll((long long)X);
	const unsigned long long R = ((X << (lz - 1)) + 0x200) >> 10;     // 53 bits, or 2^53 (X < 2^63: lz >= 1)
	const int be = 63 - lz + (32 - sh) + e + 1023;        // biased exponent of the leading bit
	unsigned long long bits = ((unsigned long long)(be - 1) << 52) + R;
	if (be < 1 || be > 2046) bits = be < 1 ? 0ull : 0x7FF0000000000000ull;
	bits = X == 0 ? 0ull : bits;
	return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

// Columns c0 .. c0 + 7 of this thread's accumulator row as doubles, times 2^(e[c0 + j] + F - 16).  All lanes call.
__device__ __forceinline__ void combine8(uint32_t trow, int c0, const int* __restrict__ e, int F, double (&out)[8])
{
	float acc[S][8];
	__syncwarp();
#pragma unroll
	for (int L = 0; L < S; ++L) tc::tmem_ld8(trow + (uint32_t)(L * kN + c0), acc[L]);
	tc::tmem_ld_wait();
#pragma unroll
	for (int j = 0; j < 8; ++j) {
		long long hi = 0, lo = 0;   // units 2^-24 and 2^-56
#pragma unroll
		for (int L = 0; L < 4; ++L) {
			hi += (long long)__float2int_rn(acc[L][j] * __int_as_float((127 + 8 * L) << 23)) << (24 - 8 * L);
			lo += (long long)__float2int_rn(acc[L + 4][j] * __int_as_float((127 + 8 * (L + 4)) << 23)) << (24 - 8 * L);
		}
		out[j] = joined(hi, lo, e[c0 + j] + F - 72);
	}
}

// One arrival per warp, after the writes (and their fences) of all its lanes.
__device__ __forceinline__ void warp_arrive(uint64_t* bar)
{
	__syncwarp();
	if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

struct Bars {
	uint64_t full[2], freed[2], ready[2], done, acc_free;
	uint32_t tmem;
};

__device__ __forceinline__ uint32_t block_setup(Bars* B, int warp)
{
	if (warp == 0) { tc::tmem_alloc(&B->tmem, 512u); tc::tmem_relinquish(); }
	if (threadIdx.x == 0) {
		for (int i = 0; i < 2; ++i) {
			tc::mbar_init(&B->full[i], 1);
			tc::mbar_init(&B->freed[i], 1);
			tc::mbar_init(&B->ready[i], kComputeWarps);
		}
		tc::mbar_init(&B->done, 1);
		tc::mbar_init(&B->acc_free, kComputeWarps);
		tc::fence_mbar_init();
	}
	tc::fence_before_sync();
	__syncthreads();
	tc::fence_after_sync();
	return B->tmem;
}

__device__ __forceinline__ void block_end(uint32_t tmem, int warp)
{
	tc::fence_before_sync();
	__syncthreads();
	if (warp == 0) tc::tmem_dealloc(tmem, 512u);
}

template <int NV>
__global__ void __launch_bounds__(kBlockThreads, 1) k_oz_interp(const double* sol, const __grid_constant__ Dev d,
                                                                double* __restrict__ svc, double* __restrict__ trace, int* err)
{
	extern __shared__ __align__(1024) uint8_t sm[];
	const Group& g = d.g[group_of(d, blockIdx.x)];
	constexpr int EB = kRows / NV;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int e0 = (blockIdx.x - g.blk0) * EB, ne = min(EB, g.n_vol - e0), rows = ne * NV;
	int* colF = (int*)(sm + kOffTab);
	int64_t* fbase = (int64_t*)(colF + kRows);             // [EB][n_fl] trace offset of the face side
	int* fp = (int*)(fbase + kRows * kMaxFl);              // [EB][n_fl] order of the face
	__shared__ Bars B;
	if (tid < kRows) colF[tid] = -4000;
	const uint32_t tmem = block_setup(&B, warp);
	const int KS = g.KS, NT = g.NT, T = NT * KS;
	if (warp == kLoadWarp) {
		for (int t = 0; t < T; ++t) {
			const int s = t & 1;
			if (t >= 2 && !tc::mbar_wait(&B.freed[s], (uint32_t)((t / 2 - 1) & 1))) { fail(err, 1); break; }
			load_stage(sm + kOffOp + s * kOpSlot, g.tI + (size_t)t * kOpSlot, kOpSlot, &B.full[s]);
		}
	} else if (warp == kIssueWarp) {
		const uint32_t idesc = tc::make_idesc(kRows, kN, 1);
#pragma unroll 1
		for (int t = 0; t < T; ++t) {
			const int nt = t / KS, c = t - nt * KS, s = t & 1;
			if (nt == 0 && !tc::mbar_wait(&B.ready[c], 0)) fail(err, 6);
			if (nt > 0 && c == 0 && !tc::mbar_wait(&B.acc_free, (uint32_t)((nt - 1) & 1))) fail(err, 7);
			if (!tc::mbar_wait(&B.full[s], (uint32_t)((t / 2) & 1))) fail(err, 3);
			tc::fence_after_sync();
			chunk_slices<0>(tmem, tc::make_sdesc(tc::smem_u32(sm + c * kDigSlot), 128, 512),
			                tc::make_sdesc(tc::smem_u32(sm + kOffOp + s * kOpSlot), 128, 512), (kN * 64) >> 4, idesc, c == 0);
			tc::mma_commit_elect(&B.freed[s]);
			if (c == KS - 1) tc::mma_commit_elect(&B.done);
			__syncwarp();
		}
	} else {
		const int n_s = g.n_s, m_r = 8 * warp + (lane & 7), kg = lane >> 3;   // whole lines of 8 rows per load of a warp
		for (int k = tid; k < ne * d.n_fl; k += kCompute) {
			const int el = k / d.n_fl, lf = k - el * d.n_fl, v = g.vols ? g.vols[e0 + el] : e0 + el;
			const int vf = d.vol_face[(size_t)v * d.n_fl + lf], f = vf >> 1;
			const int pf = d.face_p ? d.face_p[f] : d.p_min;
			const int64_t off = d.fnode_off ? d.fnode_off[f] : (int64_t)f * d.n_fc[pf];
			fbase[k] = 2 * NV * off + (int64_t)(vf & 1) * NV * d.n_fc[pf];
			fp[k] = pf;
		}
		grid_wait();
		double x[2][8];
		{
			const int el = m_r / NV, var = m_r - el * NV, v = m_r < rows ? (g.vols ? g.vols[e0 + el] : e0 + el) : 0;
			const double* src = sol + (d.dof_off ? d.dof_off[v] : (int64_t)v * NV * n_s) + var * n_s;
			int e = -4000;
#pragma unroll
			for (int c = 0; c < 2; ++c)
#pragma unroll
				for (int j = 0; j < 8; ++j) {
					const int k = 32 * c + 8 * kg + j;
					x[c][j] = (m_r < rows && k < n_s) ? src[k] : 0.0;
					e = max(e, exp_bound(x[c][j]));
				}
			if (e > -4000) atomicMax(&colF[m_r], e);
		}
		compute_sync();
		{
			const int F = row_scale(colF[m_r]);
#pragma unroll 1
			for (int c = 0; c < KS; ++c) {
				double y[8];
#pragma unroll
				for (int j = 0; j < 8; ++j) y[j] = c == 0 ? x[0][j] : x[1][j];
				write_digits(sm + c * kDigSlot, m_r, 8 * kg, y, F);
				tc::fence_async_smem();
				warp_arrive(&B.ready[c]);
			}
		}
		const int m = 32 * (warp & 3) + lane, el = m / NV, var = m - el * NV;
		const bool live = m < rows, bad = colF[m] >= kNonFinite;
		const int F = row_scale(colF[m]);
		const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
		double* srow = svc + g.svc0 + ((size_t)e0 * NV + m) * g.n_c;
#pragma unroll 1
		for (int nt = 0; nt < NT; ++nt) {
			if (!tc::mbar_wait(&B.done, (uint32_t)(nt & 1))) fail(err, 5);
			tc::fence_after_sync();
#pragma unroll 1
			for (int c8 = warp >> 2; c8 < kN / 8; c8 += kColStride) {
				if (nt * kN + 8 * c8 >= g.n_col) break;   // padding columns
				double v[8];
				combine8(trow, 8 * c8, g.eI + nt * kN, F, v);
				if (!live) continue;
#pragma unroll
				for (int j = 0; j < 8; ++j) {
					const int code = g.col[nt * kN + 8 * c8 + j];
					if (code < 0) continue;
					const double y = bad ? __longlong_as_double(0x7FF8000000000000ll) : v[j];
					if (code < (1 << 16)) { srow[code] = y; continue; }
					const int lf = (code >> 12) & 15, pf = (code >> 8) & 15, q = code & 255;
					if (fp[el * d.n_fl + lf] == pf) trace[fbase[el * d.n_fl + lf] + (int64_t)var * d.n_fc[pf] + q] = y;
				}
			}
			tc::fence_before_sync();
			warp_arrive(&B.acc_free);
		}
	}
	block_end(tmem, warp);
}

// Face nodes first, then the volume nodes of the groups.
template <int D, int NV>
__global__ void __launch_bounds__(128) k_oz_flux(const double* trace, const double* svc,
                                                 const __grid_constant__ Dev d, double* __restrict__ xl, int num_flux)
{
	static_assert(NV == D + 2, "Euler");
	grid_wait();
	const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t < d.n_fnode) {
		const int f = d.node_face ? d.node_face[t] : (int)(t / d.n_fc[d.p_min]);
		const int64_t off = d.fnode_off ? d.fnode_off[f] : (int64_t)f * d.n_fc[d.p_min];
		const int n_fc = d.fnode_off ? (int)(d.fnode_off[f + 1] - off) : d.n_fc[d.p_min];
		const int q = (int)(t - off), qr = d.nc[t];
		double WL[NV], WR[NV], n[D], nf[NV];
#pragma unroll
		for (int v = 0; v < NV; ++v) {
			WL[v] = trace[2 * NV * off + (int64_t)v * n_fc + q];
			WR[v] = trace[2 * NV * off + (int64_t)(NV + v) * n_fc + qr];
		}
#pragma unroll
		for (int a = 0; a < D; ++a) n[a] = d.nrm[t * D + a];
		const double h = 0.5 * d.jf[t];
		if (num_flux == DPG_NUM_FLUX_ROE_PIKE) numflux_roe_pike_rs<D>(WL, WR, n, h, nf);
		else                                   numflux_lax_friedrichs_rs<D>(WL, WR, n, h, nf);
		double* xL = xl + d.face_xl[2 * f] + q;
		double* xR = xl + d.face_xl[2 * f + 1] + qr;
		const int lL = d.face_ld[2 * f], lR = d.face_ld[2 * f + 1];
#pragma unroll
		for (int v = 0; v < NV; ++v) {
			const double y = nf[v];
			xL[(size_t)v * lL] = y;
			xR[(size_t)v * lR] = __longlong_as_double(__double_as_longlong(y) ^ (long long)0x8000000000000000ull);
		}
		return;
	}
	const int64_t tv = t - d.n_fnode;
	if (tv >= d.n_vnode) return;
	int k = 0;
	while (k + 1 < d.n_groups && d.g[k + 1].node0 <= tv) ++k;
	const Group& g = d.g[k];
	const int64_t r = tv - g.node0;
	const int e = (int)(r / g.n_c), c = (int)(r - (int64_t)e * g.n_c);
	double s[NV];
#pragma unroll
	for (int v = 0; v < NV; ++v) s[v] = svc[g.svc0 + ((size_t)e * NV + v) * g.n_c + c];
	double* x = xl + g.xl0 + (size_t)e * NV * g.ldx + c;
	const double* m = g.met + (size_t)e * D * D;
	tp::ref_flux<D, NV>(s, [&](int a, int dir) { return m[a + D * dir]; }, nullptr, [&](int dir, const double (&fr)[NV]) {
#pragma unroll
		for (int v = 0; v < NV; ++v) x[(size_t)v * g.ldx + dir * g.n_c] = fr[v];
	});
}

template <int NV>
__global__ void __launch_bounds__(kBlockThreads, 1) k_oz_lift(const double* xl, const __grid_constant__ Dev d,
                                                              double* sol, double* solp,
                                                              double* __restrict__ rhs, const double* __restrict__ dt_ptr,
                                                              unsigned long long* max_slot, int stage, int write_rhs, int* err)
{
	extern __shared__ __align__(1024) uint8_t sm[];
	const Group& g = d.g[group_of(d, blockIdx.x)];
	constexpr int EB = kRows / NV;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int e0 = (blockIdx.x - g.blk0) * EB, ne = min(EB, g.n_vol - e0), rows = ne * NV;
	int* colF = (int*)(sm + kOffTab);
	__shared__ Bars B;
	if (tid < kRows) colF[tid] = -4000;
	const uint32_t tmem = block_setup(&B, warp);
	const int KL = g.KL;
	const uint32_t op_bytes = (uint32_t)(S * g.NL * 64);
	if (warp == kLoadWarp) {
		for (int c = 0; c < KL; ++c) {
			const int s = c & 1;
			if (c >= 2 && !tc::mbar_wait(&B.freed[s], (uint32_t)((c / 2 - 1) & 1))) { fail(err, 1); break; }
			load_stage(sm + kOffOp + s * kOpSlot, g.tL + (size_t)c * op_bytes, op_bytes, &B.full[s]);
		}
	} else if (warp == kIssueWarp) {
		const uint32_t idesc = tc::make_idesc(kRows, g.NL, 1);
#pragma unroll 1
		for (int c = 0; c < KL; ++c) {
			const int s = c & 1;
			if (!tc::mbar_wait(&B.full[s], (uint32_t)((c / 2) & 1))) fail(err, 3);
			if (!tc::mbar_wait(&B.ready[s], (uint32_t)((c / 2) & 1))) fail(err, 6);
			tc::fence_after_sync();
			chunk_slices<0>(tmem, tc::make_sdesc(tc::smem_u32(sm + s * kDigSlot), 128, 512),
			                tc::make_sdesc(tc::smem_u32(sm + kOffOp + s * kOpSlot), 128, 512), (uint32_t)(g.NL * 64) >> 4, idesc, c == 0);
			tc::mma_commit_elect(&B.freed[s]);
			__syncwarp();
		}
		tc::mma_commit_elect(&B.done);
		__syncwarp();
	} else {
		const int m_r = 8 * warp + (lane & 7), kg = lane >> 3;
		const double* xrow = xl + g.xl0 + ((size_t)e0 * NV + m_r) * g.ldx + 8 * kg;
		grid_wait();
		auto load = [&](int c, double (&x)[8]) {
			if (m_r < rows) {
				load_sector(xrow + 32 * c, x);
				load_sector(xrow + 32 * c + 4, x + 4);
			} else {
#pragma unroll
				for (int j = 0; j < 8; ++j) x[j] = 0.0;
			}
		};
		// the rows' scales first, a warp per row with whole lines per load; the digits below read the data again, from L2
		{
			const double* base = xl + g.xl0 + (size_t)e0 * NV * g.ldx;
			for (int r0 = warp; r0 < rows; r0 += 2 * kComputeWarps) {
				int e[2] = {-4000, -4000};
#pragma unroll 4
				for (int k = 2 * lane; k < g.ldx; k += 64) {
#pragma unroll
					for (int h = 0; h < 2; ++h) {
						const int r = r0 + h * kComputeWarps;
						const double2 t = r < rows ? *(const double2*)(base + (size_t)r * g.ldx + k) : make_double2(0.0, 0.0);
						e[h] = max(e[h], max(exp_bound(t.x), exp_bound(t.y)));
					}
				}
#pragma unroll
				for (int h = 0; h < 2; ++h) {
					const int mx = __reduce_max_sync(0xffffffffu, e[h]);
					if (lane == 0 && r0 + h * kComputeWarps < rows) colF[r0 + h * kComputeWarps] = mx;
				}
			}
		}
		compute_sync();
		{
			const int F = row_scale(colF[m_r]);
			auto digits = [&](int c, const double (&x)[8]) {
				const int s = c & 1;
				if (c >= 2 && !tc::mbar_wait(&B.freed[s], (uint32_t)((c / 2 - 1) & 1))) fail(err, 2);
				write_digits(sm + s * kDigSlot, m_r, 8 * kg, x, F);
				tc::fence_async_smem();
				warp_arrive(&B.ready[s]);
			};
			// three register sets in rotation: each load has two chunks of digit work to land in
			double x0[8], x1[8], x2[8];
			load(0, x0);
			if (KL > 1) load(1, x1);
			if (KL > 2) load(2, x2);
#pragma unroll 1
			for (int c = 0; c < KL; c += 3) {
				digits(c, x0);
				if (c + 3 < KL) load(c + 3, x0);
				if (c + 1 < KL) {
					digits(c + 1, x1);
					if (c + 4 < KL) load(c + 4, x1);
				}
				if (c + 2 < KL) {
					digits(c + 2, x2);
					if (c + 5 < KL) load(c + 5, x2);
				}
			}
		}
		const int m = 32 * (warp & 3) + lane, el = m / NV, var = m - el * NV, n_s = g.n_s;
		const bool live = m < rows, bad = colF[m] >= kNonFinite;
		const int F = row_scale(colF[m]);
		const uint32_t trow = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
		const int v = live ? (g.vols ? g.vols[e0 + el] : e0 + el) : 0;
		const size_t base = (size_t)(d.dof_off ? d.dof_off[v] : (int64_t)v * NV * n_s) + (size_t)var * n_s;
		const double ji = live ? g.jinv[e0 + el] : 0.0, dt = stage >= 0 ? *dt_ptr : 0.0;
		double u0[8], u1[8];
		auto state = [&](int c8) {
#pragma unroll
			for (int j = 0; j < 8; ++j) {
				const bool in = live && 8 * c8 + j < n_s;
				u0[j] = in && stage >= 0 ? sol[base + 8 * c8 + j] : 0.0;
				u1[j] = in && stage >= 1 ? solp[base + 8 * c8 + j] : 0.0;
			}
		};
		if ((warp >> 2) < g.NL / 8) state(warp >> 2);
		if (!tc::mbar_wait(&B.done, 0)) fail(err, 4);
		tc::fence_after_sync();
		unsigned long long lmax = 0;
#pragma unroll 1
		for (int c8 = warp >> 2; c8 < g.NL / 8; c8 += kColStride) {
			double r8[8];
			combine8(trow, 8 * c8, g.eL, F, r8);
#pragma unroll
			for (int j = 0; j < 8; ++j) {
				const int i = 8 * c8 + j;
				if (!live || i >= n_s) continue;
				const double r = bad ? __longlong_as_double(0x7FF8000000000000ll) : r8[j] * ji;
				const unsigned long long ab = tp::abs_bits_of(r);
				lmax = ab > lmax ? ab : lmax;
				const size_t k = base + i;
				if (write_rhs) rhs[k] = r;
				if (stage == 0) { solp[k] = u0[j]; sol[k] = u0[j] + dt * r; }
				else if (stage == 1) sol[k] = (1.0 / 4.0) * (3.0 * u1[j] + u0[j] + dt * r);
				else if (stage == 2) sol[k] = (1.0 / 3.0) * (u1[j] + 2.0 * u0[j] + 2.0 * dt * r);
			}
			if (c8 + kColStride < g.NL / 8) state(c8 + kColStride);
		}
		for (int o = 16; o > 0; o >>= 1) {
			const unsigned long long t = __shfl_xor_sync(0xffffffffu, lmax, o);
			lmax = t > lmax ? t : lmax;
		}
		if (lane == 0) atomicMax(max_slot, lmax);
	}
	block_end(tmem, warp);
}

// ------------------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------------------
struct State {
	Dev dev{};
	size_t n_svc = 0, n_xl = 0, n_trace = 0;
	double *svc = nullptr, *xl = nullptr, *trace = nullptr;   // allocated by oz_ready
	int* err = nullptr;
	std::vector<void*> allocs;
};

static int up(State* st, const void** dst, const void* src, size_t bytes)
{
	void* p = nullptr;
	if (cudaMalloc(&p, bytes ? bytes : 8) != cudaSuccess) return DPG_ERR_CUDA;
	st->allocs.push_back(p);
	*dst = p;
	return bytes && cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess ? DPG_ERR_CUDA : DPG_OK;
}

// Digit tiles [n tile][chunk][slice] of n_rows operator rows (row(i)[k], k < K) in tiles of N rows, and the row scales.
template <class Row>
static void slice_operator(int n_rows, int K, int N, int n_tiles, int n_chunks, Row row, std::vector<uint8_t>& tiles, std::vector<int>& ex)
{
	const size_t tb = (size_t)N * 64;
	tiles.assign(tb * S * n_tiles * n_chunks, 0);
	ex.assign((size_t)n_tiles * N, 0);
	for (int i = 0; i < n_rows; ++i) {
		double mx = 0.0;
		for (int k = 0; k < K; ++k) mx = std::max(mx, std::fabs(row(i, k)));
		int E = 0;
		if (mx > 0.0) { std::frexp(mx, &E); E += 2; }   // |a| 2^-E < 1/4
		ex[i] = E;
		const int nt = i / N, r = i - nt * N;
		for (int k = 0; k < K; ++k) {
			const double a = row(i, k);
			if (a == 0.0) continue;
			const long long m = std::llrint(std::ldexp(a, 8 * S - E)) + digit_bias<S>();
			const uint32_t o = tc::kmajor_offset(r, k % 32, 32, 2);
			for (int s = 0; s < S; ++s) {
				const int dgt = s == 0 ? (int)(m >> (8 * (S - 1))) : (int)((m >> (8 * (S - 1 - s))) & 255) - 128;
				const float f = (float)std::ldexp((double)dgt, -8 * s);
				uint32_t u;
				memcpy(&u, &f, 4);
				const uint16_t b = (uint16_t)(u >> 16);   // 8 significant bits: exact
				memcpy(&tiles[(((size_t)nt * n_chunks + k / 32) * S + s) * tb + o], &b, 2);
			}
		}
	}
}

} // namespace oz

using namespace oz;

void oz_free(dpg_gpu_ctx* c)
{
	State* st = (State*)c->oz;
	if (!st) return;
	for (void* p : st->allocs) cudaFree(p);
	delete st;
	c->oz = nullptr;
}

// Whether this path is the faster one.  A block's latency (operator tiles, digits, one accumulator set) is 15..60 us per
// kernel whatever the mesh; the dense kernels' time is their FP64 multiply-adds, 0.45 T per second on a full chip, and a
// chain per block that is two to three times as long where orders are mixed.  Measured, us per residual, this path /
// the dense kernels, by volumes:
//   multiply-adds per volume   small              medium               large
//   TET 1,   800               1,296:  42 / 31    6,000:  73 / 50     24,576: 201 / 135
//   TRI 3, 2,400               1,152:  48 / 35    8,192:  89 / 89     32,768: 296 / 264
//   TRI 4, 4,680               1,152:  49 / 38    8,192:  90 / 131    32,768: 296 / 407
//   TET 2, 5,200               1,296:  56 / 46    6,000: 113 / 131    24,576: 370 / 426
//   TET 3, 19,000                384:  66 / 54    1,296:  73 / 94     24,576: 556 / 1263
//   TET 4, 110,000                48: 122 / 68    1,296: 145 / 420     6,000: 361 / 1335
//   TRI 1..3 (mixed)              72:  46 / 44    1,152:  46 / 47      8,192:  80 / 72
//   TRI 1..4 (mixed)              72:  48 / 66    8,192:  90 / 125    32,768: 276 / 290
//   TET 1..2 (mixed)              48:  54 / 66      384:  54 / 68      3,072:  66 / 97
//   TET 1..4 (mixed)              48: 125 / 194   3,072: 155 / 360    24,576: 779 / 2116
// So: 4,500 multiply-adds or more per volume of the highest order, and with one order 2e7 in all.
static bool worth_it(const struct dpg_sim* sim)
{
	double total = 0.0, most = 0.0;
	for (int v = 0; v < sim->n_vol; ++v) {
		const dpg_element_ops& o = sim->ops[sim->vol_ops[v]];
		const double w = (double)sim->n_var * (o.n_c * o.n_s + o.n_s * (sim->d * o.n_c + 2 * o.n_fl * o.n_fc));
		total += w;
		most = std::max(most, w);
	}
	return most >= 4500.0 && (total >= 2e7 || sim->n_ops > 1);
}

// Set-up; leaves c->oz null where the dense FP64 kernels run.  groups: the device tables of a mixed-order context (volume
// lists, metrics), or null with one order.
int oz_prepare(dpg_gpu_ctx* c, const struct dpg_sim* sim, const OzTables& tab)
{
	const int d = sim->d, NV = sim->n_var, n_face = sim->n_face, n_vol = sim->n_vol;
	const int e_type = sim->ops[0].e_type, n_fl = sim->ops[0].n_fl;
	if ((e_type != DPG_TRI && e_type != DPG_TET) || NV != d + 2 || sim->n_ops > kMaxGroups) return DPG_OK;
	if (!worth_it(sim)) return DPG_OK;
	for (int f = 0; f < n_face; ++f)
		if (sim->face_vol[2 * f + 1] < 0) return DPG_OK;
	for (int v = 0; v < n_vol; ++v)
		if (!sim->vol_affine[v]) return DPG_OK;
	int p_max = 0;
	for (int k = 0; k < sim->n_ops; ++k) {
		if (sim->ops[k].n_s > 64 || sim->ops[k].p > 7 || sim->ops[k].n_fc > 255) return DPG_OK;
		p_max = std::max(p_max, sim->ops[k].p);
	}
	State* st = new State();
	c->oz = st;
	Dev& D = st->dev;
	D.n_fl = n_fl;
	D.p_min = sim->ops[0].p;
	for (int k = 0; k < sim->n_ops; ++k) D.n_fc[sim->ops[k].p] = sim->ops[k].n_fc;
	std::vector<std::vector<int>> members(sim->n_ops);
	for (int v = 0; v < n_vol; ++v) members[sim->vol_ops[v]].push_back(v);
	std::vector<int> slot(n_vol), grp(n_vol), kf((size_t)kMaxGroups * 8, 0);   // kf: first K of a face order in a group's rows
	int rc, blocks = 0;
	const int EB = kRows / NV;
	std::vector<uint8_t> tiles;
	std::vector<int> ex;
	for (int k = sim->n_ops - 1; k >= 0; --k) {   // the highest order (the longest blocks) first
		if (members[k].empty()) continue;
		const dpg_element_ops& o = sim->ops[k];
		const int gi = D.n_groups++;
		Group& g = D.g[gi];
		g.n_vol = (int)members[k].size(); g.n_s = o.n_s; g.n_c = o.n_c;
		g.blk0 = blocks;
		blocks += (g.n_vol + EB - 1) / EB;
		for (int i = 0; i < g.n_vol; ++i) { slot[members[k][i]] = i; grp[members[k][i]] = gi; }
		g.vols = tab.n_groups ? tab.vols[k] : nullptr;
		g.met = tab.met[k];
		g.jinv = tab.jinv[k];
		g.node0 = D.n_vnode;
		D.n_vnode += (int64_t)g.n_vol * g.n_c;
		g.svc0 = st->n_svc;
		st->n_svc += (size_t)g.n_vol * NV * g.n_c;
		// interpolation: volume nodes, then the face nodes of every face order
		std::vector<const double*> rows;
		std::vector<int> col;
		for (int cc = 0; cc < o.n_c; ++cc) { rows.push_back(&o.cv0_vs_vc[(size_t)cc * o.n_s]); col.push_back(cc); }
		int K = d * o.n_c;
		struct Part { int pf, n_fc, k0; const double* tw; };
		std::vector<Part> parts;
		for (int pf = o.p; pf <= p_max; ++pf) {
			const double *cf = dpg_face_cv0(&o, pf), *tw = dpg_face_tw0(&o, pf);
			if (!cf || !tw) continue;
			const int n_fc = D.n_fc[pf];
			for (int lf = 0; lf < n_fl; ++lf)
				for (int q = 0; q < n_fc; ++q) {
					rows.push_back(&cf[((size_t)lf * n_fc + q) * o.n_s]);
					col.push_back(1 << 16 | lf << 12 | pf << 8 | q);
				}
			kf[gi * 8 + pf] = K;
			parts.push_back({pf, n_fc, K, tw});
			K += n_fl * n_fc;
		}
		g.KS = (o.n_s + 31) / 32;
		g.n_col = (int)rows.size();
		g.NT = ((int)rows.size() + kN - 1) / kN;
		col.resize((size_t)g.NT * kN, -1);
		slice_operator((int)rows.size(), o.n_s, kN, g.NT, g.KS, [&](int i, int kk) { return rows[i][kk]; }, tiles, ex);
		if ((rc = up(st, (const void**)&g.tI, tiles.data(), tiles.size()))) return rc;
		if ((rc = up(st, (const void**)&g.eI, ex.data(), sizeof(int) * ex.size()))) return rc;
		if ((rc = up(st, (const void**)&g.col, col.data(), sizeof(int) * col.size()))) return rc;
		// lift: m_inv_ref [tw1 | -tw0[p_f] ..]
		g.KL = (K + 31) / 32;
		g.ldx = 32 * g.KL;
		g.NL = (o.n_s + 15) / 16 * 16;
		g.xl0 = st->n_xl;
		st->n_xl += (size_t)g.n_vol * NV * g.ldx;
		std::vector<double> L((size_t)o.n_s * K), Lm((size_t)o.n_s * K);
		for (int i = 0; i < o.n_s; ++i) {
			for (int r = 0; r < d; ++r)
				for (int cc = 0; cc < o.n_c; ++cc) L[(size_t)i * K + r * o.n_c + cc] = o.tw1_vt_vc[((size_t)r * o.n_s + i) * o.n_c + cc];
			for (const Part& pt : parts)
				for (int lf = 0; lf < n_fl; ++lf)
					for (int q = 0; q < pt.n_fc; ++q)
						L[(size_t)i * K + pt.k0 + lf * pt.n_fc + q] = -pt.tw[((size_t)lf * o.n_s + i) * pt.n_fc + q];
		}
		for (int i = 0; i < o.n_s; ++i)
			for (int j = 0; j < o.n_s; ++j) {
				const double m = o.m_inv_ref[(size_t)i * o.n_s + j];
				for (int kk = 0; kk < K; ++kk) Lm[(size_t)i * K + kk] += m * L[(size_t)j * K + kk];
			}
		slice_operator(o.n_s, K, g.NL, 1, g.KL, [&](int i, int kk) { return Lm[(size_t)i * K + kk]; }, tiles, ex);
		if ((rc = up(st, (const void**)&g.tL, tiles.data(), tiles.size()))) return rc;
		if ((rc = up(st, (const void**)&g.eL, ex.data(), sizeof(int) * ex.size()))) return rc;
	}
	D.n_blocks = blocks;
	D.n_fnode = sim->face_geo_off[n_face];
	D.dof_off = tab.dof_off; D.vol_face = tab.vol_face; D.face_p = tab.face_p; D.fnode_off = tab.fnode_off;
	D.node_face = tab.node_face; D.nc = tab.nc; D.nrm = tab.nrm; D.jf = tab.jf;
	std::vector<int64_t> fx((size_t)2 * n_face);
	std::vector<int> fl((size_t)2 * n_face);
	for (int f = 0; f < n_face; ++f) {
		const int pf = dpg_face_order(sim, f);
		for (int s = 0; s < 2; ++s) {
			const int v = sim->face_vol[2 * f + s], lf = sim->face_lf[2 * f + s];
			const Group& g = D.g[grp[v]];
			fx[2 * f + s] = (int64_t)g.xl0 + (int64_t)slot[v] * NV * g.ldx + kf[grp[v] * 8 + pf] + (int64_t)lf * D.n_fc[pf];
			fl[2 * f + s] = g.ldx;
		}
	}
	if ((rc = up(st, (const void**)&D.face_xl, fx.data(), sizeof(int64_t) * fx.size()))) return rc;
	if ((rc = up(st, (const void**)&D.face_ld, fl.data(), sizeof(int) * fl.size()))) return rc;
	const int zero = 0;
	if ((rc = up(st, (const void**)&st->err, &zero, sizeof zero))) return rc;
	st->n_trace = (size_t)2 * NV * D.n_fnode;
	const void* fns[4] = {(const void*)k_oz_interp<4>, (const void*)k_oz_lift<4>, (const void*)k_oz_interp<5>, (const void*)k_oz_lift<5>};
	for (const void* f : fns)
		if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)) return DPG_ERR_CUDA;
	return DPG_OK;
}

// The work arrays, on the first FP64 residual (a context that runs in split precision does without them); before any capture.
int oz_ready(dpg_gpu_ctx* c)
{
	State* st = (State*)c->oz;
	if (!st || st->xl) return DPG_OK;
	double* xl = nullptr;
	auto get = [](void** p, size_t bytes) { return cudaMalloc(p, bytes) == cudaSuccess; };
	if (!alloc_directions(1, {{&st->svc, st->n_svc}, {&st->trace, st->n_trace}, {&xl, st->n_xl}}, {}, get, [](void* p) { cudaFree(p); })) {
		cudaGetLastError();   // answered by the caller: the dense kernels take over
		return DPG_ERR_CUDA;
	}
	for (double* p : {st->svc, st->trace, xl}) st->allocs.push_back(p);
	// the K slots of other face orders and the padding stay zero
	if (cudaMemsetAsync(xl, 0, st->n_xl * sizeof(double), c->stream) != cudaSuccess) return DPG_ERR_CUDA;
	st->xl = xl;
	return DPG_OK;
}

template <int D, int NV>
static int launch_part(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot)
{
	State* st = (State*)c->oz;
	const Dev& d = st->dev;
	if (which == 0) {
		launch_chained(k_oz_interp<NV>, d.n_blocks, kBlockThreads, kSmem, c->stream, c->sol, d, st->svc, st->trace, st->err);
	} else if (which == 1) {
		const int64_t n = d.n_fnode + d.n_vnode;
		launch_chained(k_oz_flux<D, NV>, (unsigned)((n + 127) / 128), 128, 0, c->stream, st->trace, st->svc, d, st->xl, c->num_flux);
	} else {
		launch_chained(k_oz_lift<NV>, d.n_blocks, kBlockThreads, kSmem, c->stream, st->xl, d, c->sol, c->solp, c->rhs, c->ddt, max_slot,
		               stage, write_rhs ? 1 : 0, st->err);
	}
	return cudaGetLastError() == cudaSuccess ? DPG_OK : DPG_ERR_CUDA;
}

int oz_launch_part(dpg_gpu_ctx* c, int which, int stage, bool write_rhs, unsigned long long* max_slot)
{
	const int rc = oz_ready(c);
	if (rc) return rc;
	return c->d == 2 ? launch_part<2, 4>(c, which, stage, write_rhs, max_slot) : launch_part<3, 5>(c, which, stage, write_rhs, max_slot);
}

int oz_residual(dpg_gpu_ctx* c, int stage, bool write_rhs, unsigned long long* max_slot)
{
	int rc;
	for (int k = 0; k < 3; ++k)
		if ((rc = oz_launch_part(c, k, stage, write_rhs, max_slot))) return rc;
	return DPG_OK;
}

// non-zero when a bounded wait gave up
int oz_error(dpg_gpu_ctx* c)
{
	int e = 0;
	cudaMemcpyAsync(&e, ((State*)c->oz)->err, sizeof e, cudaMemcpyDeviceToHost, c->stream);
	cudaStreamSynchronize(c->stream);
	return e;
}

} // namespace dpg
