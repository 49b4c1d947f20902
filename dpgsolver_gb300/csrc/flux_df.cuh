// Fluxes of the split path in double-float arithmetic (df64.cuh): the numerical fluxes Roe-Pike, Lax-Friedrichs and
// upwind, and the reference-space volume flux.  Same formulas and operation order as the FP64 versions (flux.cuh and
// the FP64 form's volume kernel), evaluated on the FP32 pipe.  Sums use the one-TwoSum addition: its error is
// ~2^-47 of the larger operand, the forward-error behaviour of FP64 arithmetic at 48 bits (a difference of nearly
// equal operands is as accurate as the operands are); the results agree with FP64 to ~1e-14 of the flux scale.
#pragma once

#include "df64.cuh"

namespace dpg {
namespace df {

// gamma - 1 and gamma as double-floats (0.4 and 1.4 are not FP32 numbers)
__device__ __forceinline__ df64 gm1() { return df64{0.4f, (float)(0.4 - (double)0.4f)}; }
__device__ __forceinline__ df64 gam() { return df64{1.4f, (float)(1.4 - (double)1.4f)}; }

__device__ __forceinline__ df64 min_abs(df64 a, df64 b) { return abs_less(a, b) ? absd(a) : absd(b); }
__device__ __forceinline__ df64 max_abs(df64 a, df64 b) { return abs_less(b, a) ? absd(a) : absd(b); }

// (gamma - 1) (E - rho V.V / 2) of a state with velocity u.
template <int D>
__device__ __forceinline__ df64 pressure(const df64* W, const df64* u)
{
	return mul(gm1(), (Sum(W[D + 1]) -= prod(scale(W[0], 0.5f), dot<D>(u, u))).value());
}

// Roe-Pike flux (the formula of flux.cuh numflux_roe_pike, with the entropy fix of min/max_abs_real).
template <int D>
__device__ __forceinline__ void numflux_roe_pike(const df64* WL, const df64* WR, const df64* n, df64* nF)
{
	df64 uL[D], uR[D];
	const df64 rhoL = WL[0], rhoR = WR[0], EL = WL[D + 1], ER = WR[D + 1];
	const df64 rhoL_inv = rcp(rhoL), rhoR_inv = rcp(rhoR);
#pragma unroll
	for (int a = 0; a < D; ++a) { uL[a] = mul(WL[1 + a], rhoL_inv); uR[a] = mul(WR[1 + a], rhoR_inv); }
	const df64 VnL = dot<D>(n, uL), VnR = dot<D>(n, uR);
	const df64 pL = pressure<D>(WL, uL), EpL = add_s(EL, pL);
	const df64 pR = pressure<D>(WR, uR), EpR = add_s(ER, pR);
	const df64 r = sqrt(mul(rhoR, rhoL_inv)), rP1_inv = rcp(add_s(r, mk(1.f))), rho = mul(r, rhoL);
	auto roe = [&](df64 xL, df64 xR) { return mul((Sum(prod(r, xR)) += xL).value(), rP1_inv); };
	df64 u[D];
#pragma unroll
	for (int a = 0; a < D; ++a) u[a] = roe(uL[a], uR[a]);
	const df64 Vn = dot<D>(n, u), V2 = dot<D>(u, u), H = roe(mul(EpL, rhoL_inv), mul(EpR, rhoR_inv));
	const df64 c2 = mul(gm1(), sub_s(H, scale(V2, 0.5f))), c_inv = rsqrt(c2), c = mul(c2, c_inv);
	const df64 l1 = min_abs(sub_s(VnL, c), sub_s(Vn, c)), l5 = max_abs(add_s(VnR, c), add_s(Vn, c)), l234 = absd(Vn);
	const df64 drho = sub_s(rhoR, rhoL), dE = sub_s(ER, EL), dp = sub_s(pR, pL), dVn = sub_s(VnR, VnL);
	const df64 lc1 = sub_s(scale(add_s(l5, l1), 0.5f), l234), lc2 = scale(sub_s(l5, l1), 0.5f);
	const df64 dpc = mul(dp, c_inv), rdv = mul(rho, dVn);
	const df64 disInter1 = mul((Sum(prod(lc1, dpc)) += prod(lc2, rdv)).value(), c_inv);
	const df64 disInter2 = (Sum(prod(lc1, rdv)) += prod(lc2, dpc)).value();
	const df64 rhoVnL = mul(rhoL, VnL), rhoVnR = mul(rhoR, VnR), np = ((Sum(pL) += pR) -= disInter2).value();
	Sum f0(rhoVnL);
	f0 += rhoVnR; f0 -= prod(l234, drho); f0 -= disInter1;
	nF[0] = scale(f0.value(), 0.5f);
#pragma unroll
	for (int a = 0; a < D; ++a) {
		Sum f(prod(rhoVnL, uL[a]));
		f += prod(rhoVnR, uR[a]); f += prod(n[a], np);
		f -= prod(l234, sub_s(WR[1 + a], WL[1 + a])); f -= prod(disInter1, u[a]);
		nF[1 + a] = scale(f.value(), 0.5f);
	}
	Sum fE(prod(VnL, EpL));
	fE += prod(VnR, EpR); fE -= prod(l234, dE); fE -= prod(disInter1, H); fE -= prod(disInter2, Vn);
	nF[D + 1] = scale(fE.value(), 0.5f);
}

// Lax-Friedrichs flux (the formula of flux.cuh numflux_lax_friedrichs, the normal flux through V . n).
template <int D>
__device__ __forceinline__ void numflux_lax_friedrichs(const df64* WL, const df64* WR, const df64* n, df64* nF)
{
	df64 uL[D], uR[D];
	const df64 iL = rcp(WL[0]), iR = rcp(WR[0]);
#pragma unroll
	for (int a = 0; a < D; ++a) { uL[a] = mul(WL[1 + a], iL); uR[a] = mul(WR[1 + a], iR); }
	const df64 VnL = dot<D>(n, uL), VnR = dot<D>(n, uR), pL = pressure<D>(WL, uL), pR = pressure<D>(WR, uR);
	const df64 maxlL = add_s(sqrt(dot<D>(uL, uL)), sqrt(mul(mul(gam(), pL), iL)));
	const df64 maxlR = add_s(sqrt(dot<D>(uR, uR)), sqrt(mul(mul(gam(), pR), iR)));
	const df64 maxV = abs_less(maxlR, maxlL) ? maxlL : maxlR, pLR = add_s(pL, pR);
	auto flux = [&](df64 xL, df64 xR, df64 dW, df64 ny) {   // xL VnL + xR VnR + maxV dW + ny pLR
		Sum f(prod(xL, VnL));
		f += prod(xR, VnR); f += prod(maxV, dW); f += prod(ny, pLR);
		return scale(f.value(), 0.5f);
	};
	nF[0] = scale(((Sum(prod(WL[0], VnL)) += prod(WR[0], VnR)) += prod(maxV, sub_s(WL[0], WR[0]))).value(), 0.5f);
#pragma unroll
	for (int a = 0; a < D; ++a) nF[1 + a] = flux(WL[1 + a], WR[1 + a], sub_s(WL[1 + a], WR[1 + a]), n[a]);
	nF[D + 1] = scale(((Sum(prod(add_s(WL[D + 1], pL), VnL)) += prod(add_s(WR[D + 1], pR), VnR)) +=
	                   prod(maxV, sub_s(WL[D + 1], WR[D + 1]))).value(), 0.5f);
}

// Upwind flux of linear advection (the formula of flux.cuh numflux_upwind).
template <int D>
__device__ __forceinline__ df64 numflux_upwind(const df64* b, df64 wl, df64 wr, const df64* n)
{
	df64 bn = mk(0.f);
#pragma unroll
	for (int a = 0; a < D; ++a) bn = add_s(bn, mul(b[a], n[a]));
	const bool left = bn.hi > 2.220446049250313e-16f || (bn.hi == 2.220446049250313e-16f && bn.lo > 0.f);
	return mul(bn, left ? wl : wr);
}

// Reference-space volume flux fr[r][eq] = sum_x m[x][r] f[x][eq] (m_xr = detJ dr/dx, the cofactor metrics) of one
// node, handed to emit(r, fr_r) one reference direction at a time: the per-node quantities (1/rho, velocity,
// pressure) are formed once and the direction loop stays rolled (one copy of its code; the metric column m[.][r] is
// read by mcol(x, r)).  Euler: the contraction is taken through W_r = sum_x m[x][r] u_x.  Sums use the sloppy
// addition: each flux is accurate to ~2^-46 of its largest term, below the resolution of the row-scaled digits it
// feeds.
template <int D, int NV, class MCol, class Emit>
__device__ __forceinline__ void ref_flux_rows(const df64* s, const MCol& mcol, const df64* b, Emit&& emit)
{
	if constexpr (NV == D + 2) {
		const df64 rho_inv = rcp(s[0]), E = s[D + 1];
		df64 u[D];
#pragma unroll
		for (int a = 0; a < D; ++a) u[a] = mul(s[1 + a], rho_inv);
		const df64 p = pressure<D>(s, u), Ep = add_s(E, p);
#pragma unroll 1
		for (int r = 0; r < D; ++r) {
			df64 m[D];
#pragma unroll
			for (int x = 0; x < D; ++x) m[x] = mcol(x, r);
			const df64 W = dot<D>(m, u);
			df64 fr[NV];
			fr[0] = dot<D>(m, s + 1);
#pragma unroll
			for (int a = 0; a < D; ++a) fr[1 + a] = (Sum(prod(s[1 + a], W)) += prod(m[a], p)).value();
			fr[D + 1] = mul(Ep, W);
			emit(r, fr);
		}
	} else {
#pragma unroll 1
		for (int r = 0; r < D; ++r) {
			df64 fr[NV];
			fr[0] = mul(mcol(0, r), mul(b[0], s[0]));
#pragma unroll
			for (int x = 1; x < D; ++x) fr[0] = add_s(fr[0], mul(mcol(x, r), mul(b[x], s[0])));
			emit(r, fr);
		}
	}
}

} // namespace df
} // namespace dpg
