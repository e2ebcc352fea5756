// FP32 iterations in difference form (defect correction) for the FP64
// finishing phase of batched first-order AUSM solves.
//
// The FP32 variant's residual stops dropping near 5 orders: each face flux
// F(q) is O(1) and carries FP32 rounding of that size, and a converged cell's
// residual is the near-cancelling sum of such fluxes.  Here the state is split
// into a base state q_b, fixed between rebases and held in FP64, and an FP32
// difference d = q - q_b.  The residual is
//
//     R(q) = R64(q_b) + [R(q_b + d) - R(q_b)],
//
// where R64(q_b) is evaluated once per rebase in FP64 (k_base_residual) and the
// bracket is evaluated per stage in FP32 by algebra in which every term carries
// a factor of the difference (ausm_delta_face): (a+da)(b+db) - ab = da(b+db) +
// a db, sqrt(x+dx) - sqrt(x) = dx / (sqrt(x+dx) + sqrt(x)), and so on.  The
// rounding of the bracket is then FP32 rounding of the *change* of each face
// flux since the base, not of the flux itself, so the residual keeps falling
// below the FP32 floor; rebasing every few dozen iterations keeps the
// differences, and hence their rounding, small against the residual.
//
// The reference's AUSM (AusmScheme.cpp:12-243, 716-871) has branches: the
// Mach and pressure splits at |M| = 1 and the |M| <= 0.25 fix of the
// dissipation.  All are continuous functions of M, so a difference across a
// branch point is summed piece by piece through the branch point
// (piecewise_delta), each piece again a small difference.
//
// Conserved differences dW = W - W_b are carried in FP32 across iterations (the
// base W_b is FP64, in the engine's W0 array); primitives follow from them in
// difference form too.  Boundary ghost states are evaluated in FP64 from the
// cell's full FP64 state (base + difference) with the FP64 face normals, the
// same arithmetic that gives the ghost's base state, so their difference is
// exact to FP32 rounding of the difference.
//
// The discrete equations are the reference's; the converged state is the
// FP64 path's converged state to the accuracy of the FP64 base residual.  The
// iterates are not bit-identical to the reference's.
#include "launch_common.cuh"

namespace e3d {
namespace {

// ------------------------------------------------------------ face flux in difference form

// One cell's state as base primitives + differences, with the quantities of
// the AUSM flux that do not depend on the face: enthalpy, speed of sound and
// rho c as base value + difference (the normal Mach number is formed per face).
// Kept per cell as two 32-byte records, one sector and one load each: the base
// half changes only when the base does, the difference half is written with the
// differences.  Formed at every face instead, a cell's half-dozen divisions and
// square roots were done five times and its states gathered in four pieces.
// B200, 280k cells, 100 iterations: 17.4 ms with the states, 15.3 with the
// records and neighbours from the mate slots; what bounds it now is the 256
// bytes of neighbours' records a cell takes from L2 each stage (rolled loops and
// 5 to 8 resident blocks all stay within 15.3-16.0 ms).
struct alignas(32) DBase {
	float u, v, w, p, H, ic, F1, r;  // ic = 1/c, F1 = rho c
};
struct alignas(32) DDiff {
	float du, dv, dw, dp, dH, dc, ic1, dF1;  // dc = c' - c, ic1 = 1/c'
};
struct DCell {
	DBase b;
	DDiff d;
};

__device__ __forceinline__ void load_record(const float* __restrict__ a, int c, float o[8]) {
	asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
	             : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
	             : "l"(a + 8 * (size_t)c)
	             : "memory");
}
__device__ __forceinline__ void store_record(float* a, int c, const float o[8]) {
	asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a + 8 * (size_t)c), "f"(o[0]),
	             "f"(o[1]), "f"(o[2]), "f"(o[3]), "f"(o[4]), "f"(o[5]), "f"(o[6]), "f"(o[7])
	             : "memory");
}
__device__ __forceinline__ DCell load_cell(const float* __restrict__ base, const float* __restrict__ diff, int c) {
	float x[8], y[8];
	load_record(base, c, x);
	load_record(diff, c, y);
	return DCell{{x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]}, {y[0], y[1], y[2], y[3], y[4], y[5], y[6], y[7]}};
}

__device__ __forceinline__ DBase base_record(const Q5<float>& b, float g, float gr) {
	DBase s;
	const float qq = b.u * b.u + b.v * b.v + b.w * b.w;
	const float pr = b.p * (1.f / b.r);
	const float x = g * pr;
	s.u = b.u;
	s.v = b.v;
	s.w = b.w;
	s.p = b.p;
	s.r = b.r;
	s.H = 0.5f * qq + gr * pr;
	s.ic = rsqrtf(x);  // 1/c, and c = x/c: one reciprocal square root for both
	s.F1 = b.r * (x * s.ic);
	return s;
}
__device__ __forceinline__ DDiff diff_record(const DBase& b, const Q5<float>& d, float g, float gr) {
	DDiff s;
	s.du = d.u;
	s.dv = d.v;
	s.dw = d.w;
	s.dp = d.p;
	const float dqq = d.u * (2.f * b.u + d.u) + d.v * (2.f * b.v + d.v) + d.w * (2.f * b.w + d.w);
	const float pr = b.p * (1.f / b.r);
	const float dpr = (d.p - pr * d.r) / (b.r + d.r);  // p'/r' - p/r
	s.dH = 0.5f * dqq + gr * dpr;
	const float x = g * pr, x1 = g * (pr + dpr);
	s.ic1 = rsqrtf(x1);
	const float c = x * b.ic, c1 = x1 * s.ic1;
	s.dc = g * dpr / (c + c1);
	s.dF1 = d.r * c1 + b.r * s.dc;
	return s;
}
__device__ __forceinline__ void store_diff(float* a, int c, const DDiff& s) {
	const float o[8] = {s.du, s.dv, s.dw, s.dp, s.dH, s.dc, s.ic1, s.dF1};
	store_record(a, c, o);
}

// normal Mach number of a cell at a face: M = V/c and M' - M = (dV - M dc)/c'
__device__ __forceinline__ void dmach(const DCell& s, float nx, float ny, float nz, float& M, float& dM) {
	const float V = s.b.u * nx + s.b.v * ny + s.b.w * nz;
	const float dV = s.d.du * nx + s.d.dv * ny + s.d.dw * nz;
	M = V * s.b.ic;
	dM = (dV - M * s.d.dc) * s.d.ic1;
}

// F = (rho c, rho u c, rho v c, rho w c, rho H c) of one side and its difference
__device__ __forceinline__ void side_flux(const DCell& s, float F[5], float dF[5]) {
	const DBase& b = s.b;
	const DDiff& d = s.d;
	F[0] = b.F1;
	dF[0] = d.dF1;
	F[1] = b.F1 * b.u;
	dF[1] = d.dF1 * (b.u + d.du) + b.F1 * d.du;
	F[2] = b.F1 * b.v;
	dF[2] = d.dF1 * (b.v + d.dv) + b.F1 * d.dv;
	F[3] = b.F1 * b.w;
	dF[3] = d.dF1 * (b.w + d.dw) + b.F1 * d.dw;
	F[4] = b.F1 * b.H;
	dF[4] = d.dF1 * (b.H + d.dH) + b.F1 * d.dH;
}

// f(x + d) - f(x) for a continuous function of three pieces split at lo < hi;
// i0, i1 are the pieces of x and x + d (by the reference's branch tests) and
// piece(i, x0, e) = f_i(x0 + e) - f_i(x0) on piece i.  Across branch points
// the difference is summed through them, so every term stays a difference.
template <class P>
__device__ __forceinline__ float piecewise_delta(float x, float d, float lo, float hi, int i0, int i1, P piece) {
	if (i0 == i1) return piece(i0, x, d);
	float acc = 0.f, x0 = x, rest = d;
	if (i1 > i0) {
		for (int i = i0; i < i1; i++) {
			const float bp = i == 0 ? lo : hi;
			const float e = bp - x0;
			acc += piece(i, x0, e);
			rest -= e;
			x0 = bp;
		}
	} else {
		for (int i = i0; i > i1; i--) {
			const float bp = i == 2 ? hi : lo;
			const float e = bp - x0;
			acc += piece(i, x0, e);
			rest -= e;
			x0 = bp;
		}
	}
	return acc + piece(i1, x0, rest);
}

// branch of the Mach / pressure splits (AusmScheme.cpp:777-833): M <= -1, -1 < M < 1, M >= 1
__device__ __forceinline__ int split_piece(float M) { return M <= -1.f ? 0 : (M < 1.f ? 1 : 2); }
// branch of the dissipation's |M| with the |M| <= 0.25 fix (AusmScheme.cpp:201-209)
__device__ __forceinline__ int fix_piece(float M) { return M < -0.25f ? 0 : (M <= 0.25f ? 1 : 2); }

// Difference of the AUSM convective (fc) and dissipative (fd, when DISS) face
// fluxes between the states (bL+dL, bR+dR) and (bL, bR).
template <bool DISS>
__device__ __forceinline__ void ausm_delta_face(const DCell& L, const DCell& R, float nx, float ny, float nz, float nn,
                                                float fc[5], float fd[5]) {
	float LM, LdM, RM, RdM;
	dmach(L, nx, ny, nz, LM, LdM);
	dmach(R, nx, ny, nz, RM, RdM);
	// plus splits of the left state
	const int iL0 = split_piece(LM), iL1 = split_piece(LM + LdM);
	const float MLp = iL0 == 0 ? 0.f : (iL0 == 1 ? 0.25f * (LM + 1.f) * (LM + 1.f) : LM);
	const float PLp = iL0 == 0 ? 0.f : (iL0 == 1 ? 0.25f * (LM + 1.f) * (LM + 1.f) * (2.f - LM) : 1.f);
	const float dMLp = piecewise_delta(LM, LdM, -1.f, 1.f, iL0, iL1, [](int i, float x, float e) {
		return i == 0 ? 0.f : (i == 1 ? 0.25f * e * (2.f * (x + 1.f) + e) : e);
	});
	const float dPLp = piecewise_delta(LM, LdM, -1.f, 1.f, iL0, iL1, [](int i, float x, float e) {
		return i == 1 ? 0.25f * e * (3.f - 3.f * x * x - 3.f * x * e - e * e) : 0.f;
	});
	// minus splits of the right state
	const int iR0 = split_piece(RM), iR1 = split_piece(RM + RdM);
	const float MRm = iR0 == 0 ? RM : (iR0 == 1 ? -0.25f * (RM - 1.f) * (RM - 1.f) : 0.f);
	const float PRm = iR0 == 0 ? 1.f : (iR0 == 1 ? 0.25f * (1.f - RM) * (1.f - RM) * (2.f + RM) : 0.f);
	const float dMRm = piecewise_delta(RM, RdM, -1.f, 1.f, iR0, iR1, [](int i, float x, float e) {
		return i == 0 ? e : (i == 1 ? -0.25f * e * (2.f * (x - 1.f) + e) : 0.f);
	});
	const float dPRm = piecewise_delta(RM, RdM, -1.f, 1.f, iR0, iR1, [](int i, float x, float e) {
		return i == 1 ? 0.25f * e * (-3.f + 3.f * x * x + 3.f * x * e + e * e) : 0.f;
	});
	const float M = MLp + MRm, dM = dMLp + dMRm;
	const float dpLp = L.d.dp * (PLp + dPLp) + L.b.p * dPLp;  // (p P)' - p P
	const float dpRm = R.d.dp * (PRm + dPRm) + R.b.p * dPRm;
	float FL[5], dFL[5], FR[5], dFR[5];
	side_flux(L, FL, dFL);
	side_flux(R, FR, dFR);
	const float h = 0.5f * nn;
#pragma unroll
	for (int k = 0; k < 5; k++) {
		const float S = FL[k] + FR[k], dS = dFL[k] + dFR[k];
		fc[k] = h * (dM * (S + dS) + M * dS);  // 0.5 M (FL+FR) |S|
	}
	const float dps = (dpLp + dpRm) * nn;
	fc[1] += nx * dps;
	fc[2] += ny * dps;
	fc[3] += nz * dps;
	if (DISS) {
		const int j0 = fix_piece(M), j1 = fix_piece(M + dM);
		const float aM = j0 == 0 ? -M : (j0 == 1 ? (M * M + 0.0625f) * 2.f : M);
		const float daM = piecewise_delta(M, dM, -0.25f, 0.25f, j0, j1, [](int i, float x, float e) {
			return i == 0 ? -e : (i == 1 ? 2.f * e * (2.f * x + e) : e);
		});
#pragma unroll
		for (int k = 0; k < 5; k++) {
			const float D = FR[k] - FL[k], dD = dFR[k] - dFL[k];
			fd[k] = h * (daM * (D + dD) + aM * dD);  // 0.5 |M| (FR-FL) |S|
		}
	}
}

// Primitive differences from conserved differences dw = W - W_b, with b the
// base primitives of W_b: u = m/rho, p = (gamma-1)(rhoE - rho q^2/2).
__device__ __forceinline__ Q5<float> prim_delta(const DBase& b, const float dw[5], float gm1) {
	Q5<float> d;
	const float r1 = b.r + dw[0];
	d.r = dw[0];
	d.u = (dw[1] - b.u * dw[0]) / r1;
	d.v = (dw[2] - b.v * dw[0]) / r1;
	d.w = (dw[3] - b.w * dw[0]) / r1;
	const float u1 = b.u + d.u, v1 = b.v + d.v, w1 = b.w + d.w;
	const float dqq = d.u * (b.u + u1) + d.v * (b.v + v1) + d.w * (b.w + w1);
	d.p = gm1 * (dw[4] - 0.5f * (dw[0] * (u1 * u1 + v1 * v1 + w1 * w1) + b.r * dqq));
	return d;
}

__device__ __forceinline__ Q5<double> freestream64(const FusedView<float>& v, const Physics& ph, int gi) {
	const double* f = v.case_free ? v.case_free + 5 * v.gcase[gi] : ph.free;
	return Q5<double>{f[0], f[1], f[2], f[3], f[4]};
}

// ------------------------------------------------------------ stage kernels (tiles of real cells)

// one RK stage: flux differences, residual, conserved-difference update,
// primitive differences and the boundary ghosts' differences; the first stage
// forms the local time step from the full state as well
#ifndef E3D_DELTA_MIN_BLOCKS
#define E3D_DELTA_MIN_BLOCKS 6
#endif
template <int MODE>
__global__ void __launch_bounds__(128, E3D_DELTA_MIN_BLOCKS) k_delta_flux_tiles(FusedView<float> v, Physics ph, float alpha, float beta,
                                                             int last, const int4* __restrict__ work) {
	const int4 t = work[blockIdx.x];
	const int c = t.x + threadIdx.x;
	if (c >= t.y) return;
	constexpr bool DISS = MODE != STAGE_NODISS, FIRST = MODE == STAGE_FIRST;
	const float g = float(ph.gamma), gr = float(ph.gr), gm1 = float(ph.gm1);
	const int NR = v.NR;
	const float keep = 1.f - beta;
	float ac[5], ad[5];
#pragma unroll
	for (int q = 0; q < 5; q++) {
		ac[q] = 0.f;
		ad[q] = (!DISS || keep != 0.f) ? v.Rd[q * (size_t)NR + c] : 0.f;
		if (DISS) ad[q] *= keep;
	}
	const DCell own = load_cell(v.rec_base, v.rec_in, c);
	Q5<float> q{0.f, 0.f, 0.f, 0.f, 0.f};
	float cc = 0.f, srad = 0.f;
	if (FIRST) {
		q = Q5<float>{own.b.r + v.dW[c], own.b.u + own.d.du, own.b.v + own.d.dv, own.b.w + own.d.dw, own.b.p + own.d.dp};
		cc = sqrtf(g * q.p / q.r);
	}
	const float4* geo = reinterpret_cast<const float4*>(v.sgeo) + 4 * (size_t)c;
	unsigned ghosts = 0;  // slots with a ghost neighbour
#pragma unroll
	for (int k = 0; k < 4; k++) {
		const int mt = v.slot_mate[4 * (size_t)c + k];
		const bool left = mt >= 0;
		const int m = left ? mt : ~mt, nb = m < 4 * NR ? m >> 2 : m - 3 * NR;
		if (nb >= NR) ghosts |= 1u << k;
		const DCell nbr = load_cell(v.rec_base, v.rec_in, nb);
		const float4 n = geo[k];
		if (FIRST) srad += (fabsf(q.u * n.x + q.v * n.y + q.w * n.z) + cc) * n.w;
		float fc[5], fd[5];
		// one call with the sides selected by value: a branch on the orientation
		// would run the face arithmetic twice in warps whose cells differ
		ausm_delta_face<DISS>(left ? own : nbr, left ? nbr : own, n.x, n.y, n.z, n.w, fc, fd);
#pragma unroll
		for (int q = 0; q < 5; q++) {
			ac[q] += left ? fc[q] : -fc[q];
			if (DISS) ad[q] += (left ? fd[q] : -fd[q]) * beta;
		}
	}
	const float V = v.vol[c];
	float dt;
	if (FIRST) {
		dt = float(ph.cfl) * V / srad;
		v.dt[c] = dt;
	} else {
		dt = v.dt[c];
	}
	const float coef = alpha * dt / V;
	float dw[5];
#pragma unroll
	for (int q = 0; q < 5; q++) {
		const float rc = v.Rb[q * NR + c] + ac[q];  // R64(q_b) - D64(q_b) + change of the convective sum
		dw[q] = v.dW[q * NR + c] - coef * (rc - ad[q]);
		if (last) v.Rc[q * NR + c] = rc;  // Rc - Rd is the full residual (norms)
		if (DISS) v.Rd[q * NR + c] = ad[q];
		if (last) v.dW[q * NR + c] = dw[q];  // next iteration's W0 - W_b
	}
	const Q5<float> dq = prim_delta(own.b, dw, gm1);
	store_diff(v.rec_out, c, diff_record(own.b, dq, g, gr));
	if (last) st5(v.Pout, v.NA, c, dq);  // wall pressures read it once an iteration
	// boundary ghosts in FP64: full state of the cell, FP64 face normal
	while (ghosts) {
		const int k = __ffs(ghosts) - 1;
		ghosts &= ghosts - 1;
		const int mt = v.slot_mate[4 * (size_t)c + k], nb = (mt >= 0 ? mt : ~mt) - 3 * NR;
		const int gi = nb - NR;
		const int kind = v.gkind[gi];
		if (kind == GK_NONE) continue;
		const Q5<double> b64 = ld5(v.Pb64, v.NA, c);
		const Q5<double> q64{b64.r + (double)dq.r, b64.u + (double)dq.u, b64.v + (double)dq.v, b64.w + (double)dq.w,
		                     b64.p + (double)dq.p};
		const int f = v.slot_face[4 * c + k];
		const double* n = v.nhat64 + 3 * (size_t)f;
		const Q5<double> g64 = ghost_state<double>(kind, q64, freestream64(v, ph, gi), n[0], n[1], n[2], ph.gamma);
		const Q5<double> gb = ld5(v.Pb64, v.NA, nb);
		const Q5<float> dg{(float)(g64.r - gb.r), (float)(g64.u - gb.u), (float)(g64.v - gb.v), (float)(g64.w - gb.w),
		                   (float)(g64.p - gb.p)};
		float b8[8];
		load_record(v.rec_base, nb, b8);
		const DBase bg{b8[0], b8[1], b8[2], b8[3], b8[4], b8[5], b8[6], b8[7]};
		store_diff(v.rec_out, nb, diff_record(bg, dg, g, gr));
		if (last) st5(v.Pout, v.NA, nb, dg);
	}
}

// ------------------------------------------------------------ rebase

__device__ __forceinline__ void zero_cell(float* d0, float* d1, int NA, int c) {
	const Q5<float> z{0.f, 0.f, 0.f, 0.f, 0.f};
	st5(d0, NA, c, z);
	st5(d1, NA, c, z);
}

// real cells: W_b += dW, base primitives from W_b (FP64 and FP32 copies), differences cleared
__global__ void k_rebase_cells(int NR, int NA, double* __restrict__ Wb, float* __restrict__ dW, double gm1,
                               double* __restrict__ Pb64, float* __restrict__ Pb32, float* d0, float* d1) {
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= NR) return;
	double w[5];
	for (int q = 0; q < 5; q++) {
		w[q] = Wb[(size_t)q * NR + c] + (double)dW[(size_t)q * NR + c];
		Wb[(size_t)q * NR + c] = w[q];
		dW[(size_t)q * NR + c] = 0.f;
	}
	Q5<double> p;
	p.r = w[0];
	p.u = w[1] / w[0];
	p.v = w[2] / w[0];
	p.w = w[3] / w[0];
	p.p = gm1 * (w[4] - 0.5 * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) / w[0]);
	st5(Pb64, NA, c, p);
	st5(Pb32, NA, c, Q5<float>{(float)p.r, (float)p.u, (float)p.v, (float)p.w, (float)p.p});
	zero_cell(d0, d1, NA, c);
}

// boundary ghosts: base state from the owner cell's base state (FP64 normals)
__global__ void k_rebase_ghosts(FusedView<float> v, Physics ph, double* __restrict__ Pb64, float* __restrict__ Pb32,
                                float* d0, float* d1) {
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= v.NR) return;
	for (int k = 0; k < 4; k++) {
		const int g = v.slot_nbr[4 * c + k];
		if (g < v.NR) continue;
		const int kind = v.gkind[g - v.NR];
		if (kind == GK_NONE) continue;
		const int f = v.slot_face[4 * c + k];
		const double* n = v.nhat64 + 3 * (size_t)f;
		const Q5<double> q =
		    ghost_state<double>(kind, ld5(Pb64, v.NA, c), freestream64(v, ph, g - v.NR), n[0], n[1], n[2], ph.gamma);
		st5(Pb64, v.NA, g, q);
		st5(Pb32, v.NA, g, Q5<float>{(float)q.r, (float)q.u, (float)q.v, (float)q.w, (float)q.p});
		zero_cell(d0, d1, v.NA, g);
	}
}

// connexion ghosts: copies of their origin cells
__global__ void k_rebase_halo(int n, const int* __restrict__ dst, const int* __restrict__ src, int NA,
                              double* __restrict__ Pb64, float* __restrict__ Pb32, float* d0, float* d1) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= n) return;
	const Q5<double> q = ld5(Pb64, NA, src[t]);
	st5(Pb64, NA, dst[t], q);
	st5(Pb32, NA, dst[t], Q5<float>{(float)q.r, (float)q.u, (float)q.v, (float)q.w, (float)q.p});
	zero_cell(d0, d1, NA, dst[t]);
}

// every cell's records for the new base: differences zero
__global__ void k_rebase_records(int NA, const float* __restrict__ Pb32, float g, float gr, float* __restrict__ base,
                                 float* __restrict__ d0, float* __restrict__ d1) {
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= NA) return;
	const DBase b = base_record(ld5(Pb32, NA, c), g, gr);
	const float o[8] = {b.u, b.v, b.w, b.p, b.H, b.ic, b.F1, b.r};
	store_record(base, c, o);
	const DDiff d = diff_record(b, Q5<float>{0.f, 0.f, 0.f, 0.f, 0.f}, g, gr);
	store_diff(d0, c, d);
	store_diff(d1, c, d);
}

// base residual in FP64: Rb = sum(+-Fc) - sum(+-Fd) of the base state (first-order AUSM,
// FP64 face normals and areas); the carried dissipation difference restarts at zero
__global__ void __launch_bounds__(128) k_base_residual(FusedView<float> v, Physics ph, const double* __restrict__ area64,
                                                       float* __restrict__ Rb, float* __restrict__ Rd) {
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= v.NR) return;
	double ac[5] = {0., 0., 0., 0., 0.}, ad[5] = {0., 0., 0., 0., 0.};
	const Q5<double> qc = ld5(v.Pb64, v.NA, c);
	for (int k = 0; k < 4; k++) {
		const int s = 4 * c + k;
		const bool left = v.slot_mate[s] >= 0;
		const Q5<double> qn = ld5(v.Pb64, v.NA, v.slot_nbr[s]);
		const int f = v.slot_face[s];
		const double* n = v.nhat64 + 3 * (size_t)f;
		const Q5<double>& L = left ? qc : qn;
		const Q5<double>& R = left ? qn : qc;
		double fc[5], fd[5];
		flux_ausm_conv<double>(L, R, n[0], n[1], n[2], area64[f], ph.gamma, ph.gr, fc);
		flux_ausm_diss<double>(L, R, n[0], n[1], n[2], area64[f], ph.gamma, ph.gr, fd);
		for (int q = 0; q < 5; q++) {
			ac[q] += left ? fc[q] : -fc[q];
			ad[q] += left ? fd[q] : -fd[q];
		}
	}
	for (int q = 0; q < 5; q++) {
		Rb[(size_t)q * v.NR + c] = (float)(ac[q] - ad[q]);
		Rd[(size_t)q * v.NR + c] = 0.f;
	}
}

inline int grid_of(long long n, int tpb) { return (int)((n + tpb - 1) / tpb); }

}  // namespace

namespace delta {

cudaError_t launch_iterations(const FusedView<float>& v0, const FusedView<float>& v1, const Physics& ph,
                              const PersistArgs& a, const ReduceArgs& r, cudaStream_t st) {
	if (a.n_work <= 0) return cudaSuccess;
	int parity = a.start_parity;
	for (int it = 0; it < a.iters; it++) {
		for (int s = 0; s < a.stages; s++) {
			const FusedView<float>& v = parity ? v1 : v0;
			const float al = float(a.alpha[s]), be = float(a.beta[s]);
			const int last = s == a.stages - 1;
			const auto kernel = s == 0               ? k_delta_flux_tiles<STAGE_FIRST>
			                    : a.beta[s] != 0.0 ? k_delta_flux_tiles<STAGE_DISS>
			                                       : k_delta_flux_tiles<STAGE_NODISS>;
			kernel<<<a.n_work, 128, 0, st>>>(v, ph, al, be, last, a.work);
			parity ^= 1;
		}
		end_iteration<float>(parity ? v1 : v0, r, it, a.iters, st);
	}
	return cudaGetLastError();
}

void launch_rebase(const FusedView<float>& v, const Physics& ph, double* Wb, const double* area64, int n_halo,
                   const int* halo_dst, const int* halo_src, float* d0, float* d1, cudaStream_t st) {
	double* Pb64 = const_cast<double*>(v.Pb64);
	float* Pb32 = const_cast<float*>(v.Pb);
	if (v.NR > 0) {
		k_rebase_cells<<<grid_of(v.NR, 256), 256, 0, st>>>(v.NR, v.NA, Wb, v.dW, ph.gm1, Pb64, Pb32, d0, d1);
		k_rebase_ghosts<<<grid_of(v.NR, 256), 256, 0, st>>>(v, ph, Pb64, Pb32, d0, d1);
	}
	if (n_halo > 0) k_rebase_halo<<<grid_of(n_halo, 256), 256, 0, st>>>(n_halo, halo_dst, halo_src, v.NA, Pb64, Pb32, d0, d1);
	if (v.NA > 0)
		k_rebase_records<<<grid_of(v.NA, 256), 256, 0, st>>>(v.NA, Pb32, float(ph.gamma), float(ph.gr),
		                                                     const_cast<float*>(v.rec_base), const_cast<float*>(v.rec_in),
		                                                     v.rec_out);
	if (v.NR > 0) k_base_residual<<<grid_of(v.NR, 128), 128, 0, st>>>(v, ph, area64, v.Rb, v.Rd);
}

}  // namespace delta
}  // namespace e3d
