// Kernels of the residual/update path.
//
// Granular kernels (FP64) mirror one reference strategy method each and keep
// the reference's array meanings, so the drop-in adapters can call them one by
// one.  Fused kernels (templated on T) do the same arithmetic per RK stage in
// two passes: k_recon (gradient + limiter + MUSCL face states, ghost cells
// included) and k_flux_update (both fluxes, residual gather, conservative
// update, boundary conditions).  Every per-cell sum runs over the cell's slots
// in ascending face id, the reference's accumulation order, and no kernel uses
// atomics: each cell (or ghost) is written by exactly one thread.
#pragma once
#include <cooperative_groups.h>

#include "physics.cuh"
#include "views.hpp"

namespace e3d {
// Internal linkage: k64.cu and k32.cu each compile their own copy.
namespace {

// Five-variable arrays use a packed layout: [n] vectors of (rho, u, v, w)
// followed by [n] p.  A gather of one cell's state touches two memory sectors
// (one 16/32-byte vector + one scalar) instead of five.
template <class T>
struct Vec4;
template <>
struct Vec4<float> {
	using type = float4;
};
template <>
struct Vec4<double> {
	using type = double4;
};

// Four values as one memory instruction.  A double4 in C++ is two 16-byte
// accesses; sm_100 has 32-byte ones, half the instructions and L1 tag look-ups
// of every gathered FP64 state.  B200, 663k tets FP64: flux pass without
// dissipation 88 -> 74 us, with 121 -> 117, first reconstruction 154 -> 145;
// strategy-level central flux on 41k cells 14.4 -> 12.4.
__device__ __forceinline__ float4 ldv4(const float* __restrict__ p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ double4 ldv4(const double* __restrict__ p) {
	double4 a;
	asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(a.z), "=d"(a.w) : "l"(p) : "memory");
	return a;
}
__device__ __forceinline__ void stv4(float* p, const float4& a) { *reinterpret_cast<float4*>(p) = a; }
__device__ __forceinline__ void stv4(double* p, const double4& a) {
	asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a.x), "d"(a.y), "d"(a.z), "d"(a.w) : "memory");
}

template <class T>
__device__ __forceinline__ Q5<T> ld5(const T* __restrict__ P, int n, int c) {
	const typename Vec4<T>::type a = ldv4(P + 4 * (size_t)c);
	Q5<T> q;
	q.r = a.x;
	q.u = a.y;
	q.v = a.z;
	q.w = a.w;
	q.p = P[4 * (size_t)n + c];
	return q;
}
template <class T>
__device__ __forceinline__ void st5(T* __restrict__ P, int n, int c, const Q5<T>& q) {
	typename Vec4<T>::type a;
	a.x = q.r;
	a.y = q.u;
	a.z = q.v;
	a.w = q.w;
	stv4(P + 4 * (size_t)c, a);
	P[4 * (size_t)n + c] = q.p;
}
template <class T>
__device__ __forceinline__ T& qv(Q5<T>& q, int v) { return (&q.r)[v]; }
template <class T>
__device__ __forceinline__ T qv(const Q5<T>& q, int v) { return (&q.r)[v]; }

// Launched with programmatic serialization (launch_next): the next kernel's blocks
// may take their places while this one's last blocks run, and every kernel waits
// here for all memory of the one before it.  Only data that no kernel of an
// iteration writes (topology, geometry) may be read before the wait, and only
// pointers to such data may be `const __restrict__` parameters of the kernel: the
// qualifiers promise constant data from the kernel's first instruction on, and allow
// loads past the coherent path, while here the kernel before may still be writing.
__device__ __forceinline__ void start_after_previous() {
	cudaTriggerProgrammaticLaunchCompletion();
	cudaGridDependencySynchronize();
}

// Thread index -> cell of a per-block range: real cells [r0, r1) then ghost
// cells [NR+g0, NR+g1).
__device__ __forceinline__ int range_cell(int t, int r0, int r1, int NR, int g0, int g1) {
	const int nr = r1 - r0;
	if (t < nr) return r0 + t;
	t -= nr;
	if (t < g1 - g0) return NR + g0 + t;
	return -1;
}

// ===================================================================== granular
// Solver::saveW0 (Solver/src/Solver.cpp:161-210).
__global__ void k_save_w0(GeoView g, StateView s, Physics ph, int r0, int r1) {
	start_after_previous();
	const int c = r0 + blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= r1) return;
	const Q5<double> q = ld5(s.prim, g.NA, c);
	const int n = g.NR;
	s.w0[c] = q.r;
	s.w0[n + c] = q.r * q.u;
	s.w0[2 * n + c] = q.r * q.v;
	s.w0[3 * n + c] = q.r * q.w;
	s.w0[4 * n + c] = 0.5 * q.r * (q.u * q.u + q.v * q.v + q.w * q.w) + 1. / (ph.gamma - 1.0) * q.p;
}

// Timestep::computeSpectralRadius (Solver/src/Timestep.cpp:26-121): the cell's
// own state on every face.
__global__ void k_spectral_radius(GeoView g, StateView s, Physics ph, int r0, int r1) {
	start_after_previous();
	const int c = r0 + blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= r1) return;
	const Q5<double> q = ld5(s.prim, g.NA, c);
	const double cc = sqrt(ph.gamma * q.p / q.r);
	double sr = 0.0;
	for (int k = g.slot_ptr[c]; k < g.slot_ptr[c + 1]; k++) {
		const int f = g.slot_face[k];
		const double nx = g.nhat[3 * f], ny = g.nhat[3 * f + 1], nz = g.nhat[3 * f + 2], ds = g.area[f];
		sr += (fabs((q.u) * nx + (q.v) * ny + (q.w) * nz) + (cc)) * ds;
	}
	s.srad[c] = sr;
}

// Timestep::computeTimestep (Timestep.cpp:123-148).
__global__ void k_timestep(GeoView g, StateView s, Physics ph, int r0, int r1) {
	start_after_previous();
	const int c = r0 + blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= r1) return;
	s.dt[c] = ph.cfl * g.vol[c] / s.srad[c];
}

// Gradients are stored cell-major, GRAD_LD values a cell (variable-major, 3 each),
// limiters packed like the primitives: a face's two sides are two runs of 160
// bytes instead of 40 separate rows.  These kernels run on one block of a mesh at
// a time and are bound by latency, so each takes several lanes per cell: one per
// variable (gradients, limiters), one per slot (fluxes).  Every sum keeps the
// reference's order.  B200, back to back on 41k cells, one thread per cell / this
// form: Venkatakrishnan 14.4 / 10.3, central flux 14.4 / 12.4, Roe dissipation 18.5 /
// 16.5 us; on 25k cells Barth-Jespersen 16.9 / 8.2, smoothing 21 / 9 us.

// Writes variable v's gradient of the ghosts owned by real cell c: reflected for ghosts of the
// first n_real_boundaries markers, zero for the others (GreenGauss.cpp:68-81,
// 175-232; LeastSquares.cpp:62-75, 127-184).
__device__ __forceinline__ void write_ghost_grads(const GeoView& g, const StateView& s, int c, int v, const double gr[3]) {
	for (int k = g.slot_ptr[c]; k < g.slot_ptr[c + 1]; k++) {
		const int nb = g.slot_nbr[k];
		if (nb < g.NR) continue;
		const double* n = g.sgeo + 4 * (size_t)k;
		double go[3] = {0.0, 0.0, 0.0};
		if (g.grefl[nb - g.NR]) reflect_grad(gr, n[0], n[1], n[2], go);
		for (int d = 0; d < 3; d++) s.grad[GRAD_LD * (size_t)nb + 3 * v + d] = go[d];
	}
}

__device__ __forceinline__ double ld5q(const double* __restrict__ P, int n, int c, int q) {
	return q < 4 ? P[4 * (size_t)c + q] : P[4 * (size_t)n + c];
}

// GreenGauss::computeGradients (Solver/src/GreenGauss.cpp:86-166) and
// LeastSquares::computeGradients (Solver/src/LeastSquares.cpp:80-119), five lanes per cell.
template <int GRAD>
__global__ void k_grad(GeoView g, StateView s, int r0, int r1) {
	start_after_previous();
	const int t = blockIdx.x * blockDim.x + threadIdx.x, c = r0 + t / 5, v = t % 5;
	if (c >= r1) return;
	double gr[3] = {0.0, 0.0, 0.0};
	const double q0 = ld5q(s.prim, g.NA, c, v);
	const int k1 = g.slot_ptr[c + 1];
	for (int k = g.slot_ptr[c]; k < k1; k++) {
		const double qn = ld5q(s.prim, g.NA, g.slot_nbr[k], v);
		if (GRAD == GRAD_GREEN_GAUSS) {
			const int f = g.slot_face[k];
			// 0.5*(q_L+q_R)*(+-S): addition commutes, so owner/neighbour order is exact
			const double a = 0.5 * (q0 + qn);
			const bool left = g.slot_mate[k] >= 0;
			for (int d = 0; d < 3; d++) {
				const double n = g.S[3 * (size_t)f + d];
				gr[d] += a * (left ? n : -n);
			}
		} else {
			const double dq = qn - q0;
			for (int d = 0; d < 3; d++) gr[d] += g.lsw[3 * (size_t)k + d] * dq;
		}
	}
	if (GRAD == GRAD_GREEN_GAUSS) {
		const double V = g.vol[c];
		for (int d = 0; d < 3; d++) gr[d] /= V;
	}
	for (int d = 0; d < 3; d++) s.grad[GRAD_LD * (size_t)c + 3 * v + d] = gr[d];
	write_ghost_grads(g, s, c, v, gr);
}

// BarthJespersen::computeLimiters / Venkatakrishnan::computeLimiters
// (Solver/src/BarthJespersen.cpp:88-331, Venkatakrishnan.cpp:87-324), all cells, five lanes per cell.
template <int LIM>
__global__ void k_limiter(GeoView g, StateView s, Physics ph, int r0, int r1, int g0, int g1) {
	start_after_previous();
	const int t = blockIdx.x * blockDim.x + threadIdx.x, v = t % 5;
	const int c = range_cell(t / 5, r0, r1, g.NR, g0, g1);
	if (c < 0) return;
	const double q0 = ld5q(s.prim, g.NA, c, v);
	double mx = q0, mn = q0;
	const int k0 = g.slot_ptr[c], k1 = g.slot_ptr[c + 1];
	for (int k = k0; k < k1; k++) {
		const double qn = ld5q(s.prim, g.NA, g.slot_nbr[k], v);
		if (qn > mx) mx = qn;
		if (qn < mn) mn = qn;
	}
	const double dmax = mx - q0, dmin = mn - q0;
	const double eps2 = ph.k3 * g.vol[c];
	const double* gr = s.grad + GRAD_LD * (size_t)c + 3 * v;
	const double gx = gr[0], gy = gr[1], gz = gr[2];
	CellLimiter<double, LIM> lim;
	for (int k = k0; k < k1; k++) {
		const double* r = g.srv + 3 * (size_t)k;
		double d2 = 0.0;
		d2 += gx * r[0];
		d2 += gy * r[1];
		d2 += gz * r[2];
		lim.face(d2, dmax, dmin, ph.omega, eps2);
	}
	s.lim[v < 4 ? 4 * (size_t)c + v : 4 * (size_t)g.NA + c] = lim.value(dmax, dmin);
}

// State of cell c at a face it sees at r, from its gradient and limiter.
__device__ __forceinline__ Q5<double> face_state(const GeoView& g, const StateView& s, int c, const double* __restrict__ r) {
	Q5<double> q = ld5(s.prim, g.NA, c);
	const Q5<double> phi = ld5(s.lim, g.NA, c);
	double gr[GRAD_LD];
#pragma unroll
	for (int i = 0; i < GRAD_LD / 4; i++) {
		const double4 x = ldv4(s.grad + GRAD_LD * (size_t)c + 4 * i);
		gr[4 * i] = x.x;
		gr[4 * i + 1] = x.y;
		gr[4 * i + 2] = x.z;
		gr[4 * i + 3] = x.w;
	}
	const double rx = r[0], ry = r[1], rz = r[2];
#pragma unroll
	for (int v = 0; v < 5; v++) qv(q, v) = recon(qv(q, v), qv(phi, v), gr[3 * v], gr[3 * v + 1], gr[3 * v + 2], rx, ry, rz);
	return q;
}

// Fluxes gathered per cell, one lane per slot, LPC lanes per cell (4: tetrahedra,
// 8: up to 6 slots); lane k then adds up variable k over the slots in order.
// Convective (DISS = false): FluxScheme::computeFluxConv / AusmScheme::computeFluxConv
// (FluxScheme.cpp:83-207, AusmScheme.cpp:716-871).  Dissipative:
// RoeScheme::computeFluxDiss / AusmScheme::computeFluxDiss (RoeScheme.cpp:87-291,
// AusmScheme.cpp:84-243), Rd <- (1-beta) Rd + beta * D.
template <int SCHEME, bool DISS, int LPC>
__global__ void __launch_bounds__(128, 6) k_flux(GeoView g, StateView s, Physics ph, double beta, int r0, int r1) {
	start_after_previous();
	__shared__ double sm[4][5][33];
	const int lane = threadIdx.x & 31, k = lane & (LPC - 1), first = lane - k;
	const int c = r0 + (blockIdx.x * 128 + threadIdx.x) / LPC;
	int s0 = 4 * c, n = 4;
	if (LPC != 4) {
		s0 = c < r1 ? g.slot_ptr[c] : 0;
		n = c < r1 ? g.slot_ptr[c + 1] - s0 : 0;
	}
	double (*x)[33] = sm[threadIdx.x >> 5];
	if (c < r1 && k < n) {
		const int sl = s0 + k, mt = g.slot_mate[sl];
		const bool left = mt >= 0;
		const Q5<double> qo = face_state(g, s, c, g.srv + 3 * (size_t)sl);
		const Q5<double> qn = face_state(g, s, g.slot_nbr[sl], g.srv + 3 * (size_t)(left ? mt : ~mt));
		Q5<double> L, R;
		for (int v = 0; v < 5; v++) {
			qv(L, v) = left ? qv(qo, v) : qv(qn, v);
			qv(R, v) = left ? qv(qn, v) : qv(qo, v);
		}
		const double4 geo = ldv4(g.sgeo + 4 * (size_t)sl);
		const double nx = geo.x, ny = geo.y, nz = geo.z, nn = geo.w;
		double fl[5];
		if (DISS) {
			if (SCHEME == FLUX_ROE) flux_roe_diss(L, R, nx, ny, nz, nn, ph.gr, ph.gm1, fl);
			else flux_ausm_diss(L, R, nx, ny, nz, nn, ph.gamma, ph.gr, fl);
			for (int v = 0; v < 5; v++) fl[v] *= beta;
		} else {
			if (SCHEME == FLUX_ROE) flux_central(L, R, nx, ny, nz, nn, ph.gr, fl);
			else flux_ausm_conv(L, R, nx, ny, nz, nn, ph.gamma, ph.gr, fl);
		}
#pragma unroll
		for (int v = 0; v < 5; v++) x[v][lane] = left ? fl[v] : -fl[v];
	}
	__syncwarp();
	if (c >= r1) return;
	double* out = DISS ? s.rd : s.rc;
	for (int v = k; v < 5; v += LPC) {
		double acc = DISS ? out[v * (size_t)g.NR + c] * (1.0 - beta) : 0.0;
		for (int i = 0; i < n; i++) acc += x[v][first + i];
		out[v * (size_t)g.NR + c] = acc;
	}
}

// Conservative update and primitive recovery, W0 - alpha*dt/V*(Rc-Rd)
// (Updater::updateInternalBlock, Solver/src/Updater.cpp:31-76).
template <class T>
__device__ __forceinline__ Q5<T> conservative_update(const double w0[5], T coef, const T rc[5], const T rd[5], T gm1,
                                                     double wn[5]) {
	for (int v = 0; v < 5; v++) wn[v] = w0[v] - (double)(coef) * (double)(rc[v] - rd[v]);
	Q5<T> q;
#ifdef E3D_SHARED_SIDES
	if constexpr (sizeof(T) == 8) {  // contracted FP64 batch kernels: one reciprocal of rho
		const double ir = 1.0 / wn[0];
		q.r = wn[0];
		q.u = wn[1] * ir;
		q.v = wn[2] * ir;
		q.w = wn[3] * ir;
		q.p = gm1 * (wn[4] - 0.5 * (wn[1] * wn[1] + wn[2] * wn[2] + wn[3] * wn[3]) * ir);
		return q;
	}
#endif
	q.r = (T)wn[0];
	q.u = (T)(wn[1] / wn[0]);
	q.v = (T)(wn[2] / wn[0]);
	q.w = (T)(wn[3] / wn[0]);
	q.p = (T)((double)gm1 * (wn[4] - 0.5 * (wn[1] * wn[1] + wn[2] * wn[2] + wn[3] * wn[3]) / wn[0]));
	return q;
}

__global__ void k_update(GeoView g, StateView s, Physics ph, double alpha, int r0, int r1) {
	start_after_previous();
	const int c = r0 + blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= r1) return;
	const int n = g.NR;
	double w0[5], rc[5], rd[5], wn[5];
	for (int v = 0; v < 5; v++) {
		w0[v] = s.w0[v * n + c];
		rc[v] = s.rc[v * n + c];
		rd[v] = s.rd[v * n + c];
	}
	const double coef = alpha * s.dt[c] / g.vol[c];
	const Q5<double> q = conservative_update<double>(w0, coef, rc, rd, ph.gamma - 1.0, wn);
	st5(s.prim, g.NA, c, q);
}

// Ghost states of the first n_real_boundaries markers (Updater::updateBoundary,
// Updater.cpp:84-87, and the *CellIds::updateBoundary implementations).
template <class T>
__device__ __forceinline__ Q5<T> ghost_state(int kind, const Q5<T>& qi, const Q5<T>& fr, T nx, T ny, T nz, T gamma) {
	if (kind == GK_FARFIELD) return bc_farfield(qi, fr, nx, ny, nz, gamma);
	return bc_slip(qi, nx, ny, nz);
}

__global__ void k_bc(GeoView g, StateView s, Physics ph, int g0, int g1) {
	start_after_previous();
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= g1 - g0) return;
	const int gi = g0 + t, c = g.NR + gi;
	const int kind = g.gkind[gi];
	if (kind == GK_NONE) return;
	const int k = g.slot_ptr[c];
	const int f = g.slot_face[k], in = g.slot_nbr[k];
	Q5<double> fr;
	fr.r = ph.free[0];
	fr.u = ph.free[1];
	fr.v = ph.free[2];
	fr.w = ph.free[3];
	fr.p = ph.free[4];
	const Q5<double> q = ghost_state(kind, ld5(s.prim, g.NA, in), fr, g.nhat[3 * f], g.nhat[3 * f + 1],
	                                 g.nhat[3 * f + 2], ph.gamma);
	st5(s.prim, g.NA, c, q);
}

// Inter-block halo: connexion ghost primitives <- origin cell primitives, once
// per outer iteration (BlockCommunicator::updateBoundaries, serial path
// MPI/src/BlockCommunicator.cpp:212-268; the other 35 copied values are
// rewritten before any read).  Writes every buffer in `bufs`.
// CentralIrsSmoother::smoothResidual (Solver/src/CentralIrsSmoother.cpp:12-166):
// one Jacobi step of central implicit residual smoothing, eps = 0.8, applied to
// the convective and the dissipative residuals of the real cells.  Pass 1: the
// start value J1 = R / (1 + eps N) (N = the cell's face count) of all ten arrays.
// The reference fills J1 of the dissipative v-momentum from the w-momentum and
// never fills J1 of the dissipative w-momentum (:90); these two follow the
// formula of the other eight here.
constexpr double IRS_EPS = 0.8;
// One thread per (cell, array): blockIdx.y = 0..4 convective, 5..9 dissipative.
__global__ void k_irs_start(GeoView g, StateView s, double* __restrict__ j1, int r0, int r1) {
	start_after_previous();
	const int c = r0 + blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
	if (c >= r1) return;
	const int na = g.slot_ptr[c + 1] - g.slot_ptr[c];
	const double* r = q < 5 ? s.rc + q * (size_t)g.NR : s.rd + (q - 5) * (size_t)g.NR;
	j1[q * (size_t)g.NR + c] = (r[c] + 0.) / (1. + IRS_EPS * na);
}

// Pass 2: R = (R + eps * sum of J1 over the real neighbours in slot order) / (1 + eps N),
// in place (each thread reads only its own R and the neighbours' J1).
__global__ void k_irs_smooth(GeoView g, StateView s, const double* j1, int r0, int r1) {
	start_after_previous();
	const int c = r0 + blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
	if (c >= r1) return;
	const int k0 = g.slot_ptr[c], k1 = g.slot_ptr[c + 1];
	const double* j = j1 + q * (size_t)g.NR;
	double sum = 0.;
	for (int k = k0; k < k1; k++) {
		const int nb = g.slot_nbr[k];
		if (nb < g.NR) sum += j[nb];
	}
	double& r = q < 5 ? s.rc[q * (size_t)g.NR + c] : s.rd[(q - 5) * (size_t)g.NR + c];
	r = (r + IRS_EPS * sum) / (1. + IRS_EPS * (k1 - k0));
}

template <class T>
__global__ void k_halo(int n, const int* __restrict__ dst, const int* __restrict__ src, int NA, T* b0, T* b1) {
	start_after_previous();
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= n) return;
	const int d = dst[t], o = src[t];
	const Q5<T> q = ld5(b0, NA, o);
	st5(b0, NA, d, q);
	if (b1) st5(b1, NA, d, q);
}

// The halo of a block-sharded case, split at the transport: pack gathers the
// primitives of the origin cells another process needs into an entry-major
// buffer (buf[5*i + q], q = rho u v w p), unpack writes received entries into
// the connexion ghosts of both state buffers, as k_halo does for local ones.
template <class T>
__global__ void k_halo_pack(int n, const int* __restrict__ src, int NA, const T* __restrict__ P,
                            T* __restrict__ buf) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= n) return;
	const Q5<T> q = ld5(P, NA, src[t]);
	T* o = buf + 5 * (size_t)t;
	o[0] = q.r;
	o[1] = q.u;
	o[2] = q.v;
	o[3] = q.w;
	o[4] = q.p;
}

template <class T>
__global__ void k_halo_unpack(int n, const int* __restrict__ dst, int NA, const T* __restrict__ buf, T* b0, T* b1) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= n) return;
	const T* i = buf + 5 * (size_t)t;
	const Q5<T> q{i[0], i[1], i[2], i[3], i[4]};
	st5(b0, NA, dst[t], q);
	if (b1) st5(b1, NA, dst[t], q);
}

// ===================================================================== fused
// Slot data of one real cell.  NSL = 4 is the all-tetrahedron fast path:
// slots of cell c are 4c..4c+3, so per-slot arrays load as vectors.  NSL = 0
// reads the slot range from slot_ptr (any cell type).
template <class T, int NSL>
struct SlotRange {
	int s0, n;
	__device__ __forceinline__ SlotRange(const FusedView<T>& v, int c) {
		if (NSL == 4) {
			s0 = 4 * c;
			n = 4;
		} else {
			s0 = v.slot_ptr[c];
			n = v.slot_ptr[c + 1] - s0;
		}
	}
};
constexpr int MAXSL = 6;  // hexahedra

// A tetrahedron's four slots from s0 on: 3 consecutive values each (r-vectors, LS
// weights, signed area vectors), and one integer each
template <class T>
__device__ __forceinline__ void load3(const T* __restrict__ a, int s0, T o[4][3]) {
	T f[12];
	if constexpr (sizeof(T) == 4) {
		const float4* p = reinterpret_cast<const float4*>(a + 3 * (size_t)s0);
		const float4 x = __ldg(p), y = __ldg(p + 1), z = __ldg(p + 2);
		const float g[12] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
#pragma unroll
		for (int i = 0; i < 12; i++) f[i] = g[i];
	} else {
		const double2* p = reinterpret_cast<const double2*>(a + 3 * (size_t)s0);
#pragma unroll
		for (int i = 0; i < 6; i++) {
			const double2 t = __ldg(p + i);
			f[2 * i] = t.x;
			f[2 * i + 1] = t.y;
		}
	}
#pragma unroll
	for (int k = 0; k < 4; k++)
		for (int d = 0; d < 3; d++) o[k][d] = f[3 * k + d];
}
__device__ __forceinline__ void load_int(const int* __restrict__ a, int s0, int o[4]) {
	const int4 x = __ldg(reinterpret_cast<const int4*>(a + s0));
	o[0] = x.x;
	o[1] = x.y;
	o[2] = x.z;
	o[3] = x.w;
}

#define E3D_SLOTS(k, r) for (int k = 0; k < (NSL == 4 ? 4 : MAXSL); k++) if (NSL == 4 || k < r.n)

// First-order AUSM with each cell's side quantities formed once (built only
// where E3D_SHARED_SIDES is defined: the FP64 batch kernels with contraction,
// which are not held to the reference's operation order).  The reference forms
// a side's p/rho, speed of sound, enthalpy and c-scaled flux vector again in
// every face flux, convective and dissipative alike (AusmScheme.cpp:716-871,
// 102-243); a cell's own side is the same at all its faces, so here it is
// formed once per cell and the neighbour's once per face, the normal Mach
// number is V times 1/c, and c and 1/c come from one reciprocal square root.
// Same formulas otherwise, including the branch tests.
template <class T>
struct AusmSide {
	T u, v, w, p, ic;  // velocity, pressure, 1/c
	T F[5];            // rho c (1, u, v, w, H)
};
template <class T>
__device__ __forceinline__ AusmSide<T> ausm_side(const Q5<T>& q, T g, T gr) {
	AusmSide<T> s;
	const T pr = q.p / q.r;
	const T x = g * pr;
	s.ic = rsqrt(x);  // 1/c, and c = x/c: one reciprocal square root for both
	const T c = x * s.ic;
	const T H = T(0.5) * (q.u * q.u + q.v * q.v + q.w * q.w) + gr * pr;
	s.u = q.u;
	s.v = q.v;
	s.w = q.w;
	s.p = q.p;
	s.F[0] = q.r * c;
	s.F[1] = s.F[0] * q.u;
	s.F[2] = s.F[0] * q.v;
	s.F[3] = s.F[0] * q.w;
	s.F[4] = s.F[0] * H;
	return s;
}
template <class T, bool DISS>
__device__ __forceinline__ void ausm_face_sides(const AusmSide<T>& L, const AusmSide<T>& R, T nx, T ny, T nz, T nn,
                                                T fc[5], T fd[5]) {
	const T ML = (L.u * nx + L.v * ny + L.w * nz) * L.ic;
	const T MR = (R.u * nx + R.v * ny + R.w * nz) * R.ic;
	T pLp, MLp, pRm, MRm;
	if (ML <= T(-1.0)) {
		pLp = T(0);
		MLp = T(0);
	} else if (ML < T(1.0)) {
		MLp = T(0.25) * (ML + T(1.0)) * (ML + T(1.0));
		pLp = L.p * MLp * (T(2.0) - ML);
	} else {
		MLp = ML;
		pLp = L.p;
	}
	if (MR <= T(-1.0)) {
		pRm = R.p;
		MRm = MR;
	} else if (MR < T(1.0)) {
		MRm = T(-0.25) * (MR - T(1.0)) * (MR - T(1.0));
		pRm = -R.p * MRm * (T(2.0) + MR);
	} else {
		pRm = T(0);
		MRm = T(0);
	}
	const T M = MLp + MRm;
	const T hM = T(0.5) * M * nn, ps = (pLp + pRm) * nn;
	for (int k = 0; k < 5; k++) fc[k] = hM * (L.F[k] + R.F[k]);
	fc[1] += nx * ps;
	fc[2] += ny * ps;
	fc[3] += nz * ps;
	if (DISS) {
		const T delta = T(0.25);
		T Mf = M;
		if (!(tabs(Mf) > delta)) Mf = (Mf * Mf + delta * delta) / (T(2.0) * delta);
		const T ha = T(0.5) * tabs(Mf) * nn;
		for (int k = 0; k < 5; k++) fd[k] = ha * (R.F[k] - L.F[k]);
	}
}

// Pass 1 of a stage, one thread per real tetrahedron: gradient, limiter and MUSCL
// face states of the cell and of its ghost cells.
template <class T, int GRAD, int LIM>
__device__ __forceinline__ void recon_cell(const FusedView<T>& v, const Physics& ph, int c) {
	const int s0 = 4 * c;
	const Q5<T> q0 = ld5(v.Pin, v.NA, c);
	int nb[4];
	load_int(v.slot_nbr, s0, nb);
	T w[4][3];
	if (GRAD == GRAD_GREEN_GAUSS) load3(v.sS, s0, w);
	else load3(v.lsw, s0, w);
	T gr[5][3];
	for (int q = 0; q < 5; q++) gr[q][0] = gr[q][1] = gr[q][2] = T(0.0);
	Q5<T> mx = q0, mn = q0;
#pragma unroll
	for (int k = 0; k < 4; k++) {
		const Q5<T> qn = ld5(v.Pin, v.NA, nb[k]);
		for (int q = 0; q < 5; q++) {
			if (GRAD == GRAD_GREEN_GAUSS) {
				// 0.5*(q_L+q_R)*(+-S): addition commutes, so owner/neighbour order is exact
				const T a = T(0.5) * (qv(q0, q) + qv(qn, q));
				gr[q][0] += a * w[k][0];
				gr[q][1] += a * w[k][1];
				gr[q][2] += a * w[k][2];
			} else {
				const T dq = qv(qn, q) - qv(q0, q);
				gr[q][0] += w[k][0] * dq;
				gr[q][1] += w[k][1] * dq;
				gr[q][2] += w[k][2] * dq;
			}
			if (qv(qn, q) > qv(mx, q)) qv(mx, q) = qv(qn, q);
			if (qv(qn, q) < qv(mn, q)) qv(mn, q) = qv(qn, q);
		}
	}
	const T V = v.vol[c];
	if (GRAD == GRAD_GREEN_GAUSS)
		for (int d = 0; d < 3; d++)
			for (int q = 0; q < 5; q++) gr[q][d] /= V;
	T rv[4][3];
	load3(v.srv, s0, rv);
	const T eps2 = T(ph.k3) * V;
	if constexpr (sizeof(T) == 4) {
		// FP32: the face value q + phi (g.r) reuses the limiter's d2 = g.r
		Q5<T> fs[4];
		for (int q = 0; q < 5; q++) {
			const T dmax = qv(mx, q) - qv(q0, q), dmin = qv(mn, q) - qv(q0, q);
			T d2[4];
			CellLimiter<T, LIM> lim;
#pragma unroll
			for (int k = 0; k < 4; k++) {
				d2[k] = gr[q][0] * rv[k][0];
				d2[k] += gr[q][1] * rv[k][1];
				d2[k] += gr[q][2] * rv[k][2];
				lim.face(d2[k], dmax, dmin, T(ph.omega), eps2);
			}
			const T phi = lim.value(dmax, dmin);
#pragma unroll
			for (int k = 0; k < 4; k++) qv(fs[k], q) = qv(q0, q) + phi * d2[k];
		}
#pragma unroll
		for (int k = 0; k < 4; k++) st5(v.FS, v.NS, s0 + k, fs[k]);
	} else {
		// FP64: the reference's accumulation order
		T phi[5];
		for (int q = 0; q < 5; q++) {
			const T dmax = qv(mx, q) - qv(q0, q), dmin = qv(mn, q) - qv(q0, q);
			CellLimiter<T, LIM> lim;
#pragma unroll
			for (int k = 0; k < 4; k++) {
				T d2 = T(0.0);
				d2 += gr[q][0] * rv[k][0];
				d2 += gr[q][1] * rv[k][1];
				d2 += gr[q][2] * rv[k][2];
				lim.face(d2, dmax, dmin, T(ph.omega), eps2);
			}
			phi[q] = lim.value(dmax, dmin);
		}
#pragma unroll
		for (int k = 0; k < 4; k++) {
			Q5<T> fs;
			for (int q = 0; q < 5; q++)
				qv(fs, q) = recon(qv(q0, q), phi[q], gr[q][0], gr[q][1], gr[q][2], rv[k][0], rv[k][1], rv[k][2]);
			st5(v.FS, v.NS, s0 + k, fs);
		}
	}
	// ghost cells of this cell's boundary faces: gradient (reflected or zero),
	// limiter (the ghost's only neighbour is c) and face state.  The slot neighbours
	// are read again (a cache hit) rather than held through the pass, which takes
	// the FP32 pass from 32-68 bytes of spills to none.
	load_int(v.slot_nbr, s0, nb);
#pragma unroll
	for (int k = 0; k < 4; k++) {
		if (nb[k] >= v.NR) {
			const int g = nb[k];
			int ms = v.slot_mate[s0 + k];
			ms = ms >= 0 ? ms : ~ms;
			const Q5<T> qg = ld5(v.Pin, v.NA, g);
			const T nx = v.sgeo[4 * (size_t)(s0 + k)], ny = v.sgeo[4 * (size_t)(s0 + k) + 1],
			        nz = v.sgeo[4 * (size_t)(s0 + k) + 2];
			const T g0 = v.srv[3 * (size_t)ms], g1 = v.srv[3 * (size_t)ms + 1], g2 = v.srv[3 * (size_t)ms + 2];
			const bool refl = v.grefl[g - v.NR] != 0;
			const T eps2g = T(ph.k3) * v.vol[g];
			Q5<T> fs;
			for (int q = 0; q < 5; q++) {
				T gg[3] = {T(0.0), T(0.0), T(0.0)};
				if (refl) reflect_grad(gr[q], nx, ny, nz, gg);
				T gmx = qv(qg, q), gmn = qv(qg, q);
				if (qv(q0, q) > gmx) gmx = qv(q0, q);
				if (qv(q0, q) < gmn) gmn = qv(q0, q);
				T d2 = T(0.0);
				d2 += gg[0] * g0;
				d2 += gg[1] * g1;
				d2 += gg[2] * g2;
				const T dmx = gmx - qv(qg, q), dmn = gmn - qv(qg, q);
				const T lf = (LIM == LIM_BARTH_JESPERSEN) ? limiter_bj_face(d2, dmx, dmn, T(ph.omega))
				                                          : limiter_venkat_face(d2, dmx, dmn, eps2g);
				T pg = T(INFINITY);
				if (lf < pg) pg = lf;
				qv(fs, q) = recon(qv(qg, q), pg, gg[0], gg[1], gg[2], g0, g1, g2);
			}
			st5(v.FS, v.NS, ms, fs);
		}
	}
}

// resident blocks per SM the FP32 reconstruction pass is compiled for (64 registers)
#ifndef E3D_RECON_MIN_BLOCKS
#define E3D_RECON_MIN_BLOCKS 8
#endif
template <int GRAD, int LIM>
__global__ void __launch_bounds__(128, E3D_RECON_MIN_BLOCKS) k_recon(FusedView<float> v, Physics ph) {
	start_after_previous();
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c < v.NR) recon_cell<float, GRAD, LIM>(v, ph, c);
}

// Reconstruction with one lane per (cell, variable): FP64, and both precisions on
// cells other than tetrahedra.  Gradient, limiter and face states of one variable
// depend on that variable alone, so five lanes per cell run the same per-variable
// arithmetic as recon_cell, in the same order (FP64: bit for bit), with a fifth of
// its gradient/limiter state and the slot weights read per slot: 48 registers
// instead of 128, 40 resident warps per SM instead of 16 (663k tets FP64: 118 us
// at 6 blocks of 64 registers, 115 at 8).  A block covers RV_CELLS cells (5 *
// RV_CELLS threads, cell-major: the four lanes of a cell's (rho, u, v, w) read and
// write one 32-byte vector together).  Measured on B200 (3.07M tets, FP64 second
// order): 2.61 TB/s against 2.44 for the one-thread-per-cell pass.  With slot
// counts known only at run time, one thread per cell kept its slot arrays in local
// memory: 65k hexahedra FP64 40 us a launch, 23 here (7 resident blocks; 25 at 8).
constexpr int RV_CELLS = 32;

template <class T>
__device__ __forceinline__ T ldq(const T* __restrict__ P, int n, int c, int q) {
	return q < 4 ? P[4 * (size_t)c + q] : P[4 * (size_t)n + c];
}
template <class T>
__device__ __forceinline__ void stq(T* __restrict__ P, int n, int c, int q, T x) {
	if (q < 4) P[4 * (size_t)c + q] = x;
	else P[4 * (size_t)n + c] = x;
}

template <class T, int GRAD, int LIM, int NSL>
__global__ void __launch_bounds__(5 * RV_CELLS, NSL == 4 ? 8 : 7) k_recon_var(FusedView<T> v, Physics ph) {
	const int c = blockIdx.x * RV_CELLS + threadIdx.x / 5, q = threadIdx.x % 5;
	if (c >= v.NR) return start_after_previous();
	const SlotRange<T, NSL> sr(v, c);
	int nb[MAXSL];
	if (NSL == 4) {
		load_int(v.slot_nbr, sr.s0, nb);
	} else {
#pragma unroll
		E3D_SLOTS(k, sr) nb[k] = __ldg(v.slot_nbr + sr.s0 + k);
	}
	const T V = v.vol[c];
	start_after_previous();
	const T q0 = ldq(v.Pin, v.NA, c, q);
	T gr[3] = {T(0.0), T(0.0), T(0.0)};
	T mx = q0, mn = q0;
	{
		const T* __restrict__ wa = (GRAD == GRAD_GREEN_GAUSS ? v.sS : v.lsw) + 3 * (size_t)sr.s0;
#pragma unroll
		E3D_SLOTS(k, sr) {
			const T w[3] = {__ldg(wa + 3 * k), __ldg(wa + 3 * k + 1), __ldg(wa + 3 * k + 2)};
			const T qn = ldq(v.Pin, v.NA, nb[k], q);
			if (GRAD == GRAD_GREEN_GAUSS) {
				const T a = T(0.5) * (q0 + qn);
				gr[0] += a * w[0];
				gr[1] += a * w[1];
				gr[2] += a * w[2];
			} else {
				const T dq = qn - q0;
				gr[0] += w[0] * dq;
				gr[1] += w[1] * dq;
				gr[2] += w[2] * dq;
			}
			if (qn > mx) mx = qn;
			if (qn < mn) mn = qn;
		}
	}
	if (GRAD == GRAD_GREEN_GAUSS)
		for (int d = 0; d < 3; d++) gr[d] /= V;
	const T* __restrict__ ra = v.srv + 3 * (size_t)sr.s0;
	const T eps2 = T(ph.k3) * V;
	const T dmax = mx - q0, dmin = mn - q0;
	CellLimiter<T, LIM> lim;
#pragma unroll
	E3D_SLOTS(k, sr) {
		T d2 = T(0.0);
		d2 += gr[0] * __ldg(ra + 3 * k);
		d2 += gr[1] * __ldg(ra + 3 * k + 1);
		d2 += gr[2] * __ldg(ra + 3 * k + 2);
		lim.face(d2, dmax, dmin, T(ph.omega), eps2);
	}
	const T phi = lim.value(dmax, dmin);
#pragma unroll
	E3D_SLOTS(k, sr)
	stq(v.FS, v.NS, sr.s0 + k, q,
	    recon(q0, phi, gr[0], gr[1], gr[2], __ldg(ra + 3 * k), __ldg(ra + 3 * k + 1), __ldg(ra + 3 * k + 2)));
	// ghost cells of this cell's boundary faces (recon_cell's tail, one variable)
#pragma unroll
	E3D_SLOTS(k, sr) {
		if (nb[k] < v.NR) continue;
		const int g = nb[k];
		int ms = v.slot_mate[sr.s0 + k];
		ms = ms >= 0 ? ms : ~ms;
		const T qg = ldq(v.Pin, v.NA, g, q);
		const T* n = v.sgeo + 4 * (size_t)(sr.s0 + k);
		const T g0 = v.srv[3 * (size_t)ms], g1 = v.srv[3 * (size_t)ms + 1], g2 = v.srv[3 * (size_t)ms + 2];
		T gg[3] = {T(0.0), T(0.0), T(0.0)};
		if (v.grefl[g - v.NR] != 0) reflect_grad(gr, n[0], n[1], n[2], gg);
		T gmx = qg, gmn = qg;
		if (q0 > gmx) gmx = q0;
		if (q0 < gmn) gmn = q0;
		T d2 = T(0.0);
		d2 += gg[0] * g0;
		d2 += gg[1] * g1;
		d2 += gg[2] * g2;
		const T dmx = gmx - qg, dmn = gmn - qg;
		const T lf = (LIM == LIM_BARTH_JESPERSEN) ? limiter_bj_face(d2, dmx, dmn, T(ph.omega))
		                                          : limiter_venkat_face(d2, dmx, dmn, T(ph.k3) * v.vol[g]);
		T pg = T(INFINITY);
		if (lf < pg) pg = lf;
		stq(v.FS, v.NS, ms, q, recon(qg, pg, gg[0], gg[1], gg[2], g0, g1, g2));
	}
}

// Pass 2 of a stage, one thread per real cell: convective and dissipative
// fluxes of each face (computed identically from both sides), residual gather,
// conservative update into Pout and the ghost states of the cell's boundary
// faces.  ORDER1 reads cell states directly (first order).  LAST stores the
// final conservative state as the next W0 when carry_w0 is set.
//
// DISS = false is used for stages with beta = 0: the reference still evaluates
// the dissipative flux (its guard is always true) but Rd*(1-0) + sum(D*0) equals
// Rd for finite fluxes, so the flux and the Rd store are skipped.  Rc is stored
// only at the last stage, the one the norms (and callers) read.
//
// One face at a time (FP64: the slot loop stays rolled).  Holding all four
// slots' mates, normals and neighbours live took the FP64 Roe pass to 128
// registers and 23 % resident warps, with instruction-cache misses from four
// copies of the flux; one copy needs 96.  Neighbours of a tetrahedron follow
// from the mate slot (real slot 4c+k, ghost g's only slot 4 NR + g), so
// slot_nbr is not read, and beta = 1 drops Rd unread (a value that is not finite
// included: 0 * NaN does not reach the new Rd).  B200, us a launch with / without
// dissipation: 663k tets FP64 Roe 136 / 100 -> 121 / 88, and 152 / 102 -> 126 / 74
// with the 32-byte accesses (second pair on another box); 3.07M FP32 Roe 184 / 147 ->
// 175 / 144 (FP32 keeps the loop unrolled: 178 / 156 rolled).
// FIRST (the first stage): W0 (unless carried) and the local time step
// (Timestep.cpp:26-148) are formed here from the state the stage starts from,
// with the normals the fluxes read anyway, instead of in a pass of their own or
// in the first reconstruction (663k tets FP64 second order, us an iteration:
// first reconstruction 145 -> 115, this pass 117 -> 129; 3.07M FP32 185 -> 160 and
// 180 -> 192).
enum StageMode : int { STAGE_NODISS, STAGE_DISS, STAGE_FIRST };
template <class T>
__device__ __forceinline__ T conserved(const Q5<T>& q, int k, double gamma) {
	if (k == 4) return T(0.5) * q.r * (q.u * q.u + q.v * q.v + q.w * q.w) + T(1.) / (T(gamma) - T(1.0)) * q.p;
	return k == 0 ? q.r : k == 1 ? q.r * q.u : k == 2 ? q.r * q.v : q.r * q.w;
}
template <class T, int SCHEME, bool ORDER1, int NSL, int MODE>
__device__ __forceinline__ void flux_update_cell(const FusedView<T>& v, const Physics& ph, T alpha, T beta, int last,
                                                 int carry_w0, int c) {
	constexpr int UNROLL = NSL == 4 && sizeof(T) == 4 ? 4 : 1;
	constexpr bool DISS = MODE != STAGE_NODISS, FIRST = MODE == STAGE_FIRST;
	const int NR = v.NR;
	const SlotRange<T, NSL> sr(v, c);
	const T g = T(ph.gamma), gr = T(ph.gr), gm1 = T(ph.gm1);
	const T keep = T(1.0) - beta;
	T ac[5], ad[5];
	for (int q = 0; q < 5; q++) {
		ac[q] = T(0.0);
		ad[q] = (!DISS || keep != T(0.0)) ? v.Rd[q * (size_t)NR + c] : T(0.0);
		if (DISS) ad[q] *= keep;
	}
	Q5<T> qc;
	if (ORDER1 || FIRST) qc = ld5(v.Pin, v.NA, c);
	const T cc = FIRST ? tsqrt(g * qc.p / qc.r) : T(0.0);
	T srad = T(0.0);
#ifdef E3D_SHARED_SIDES
	constexpr bool shared_sides = ORDER1 && SCHEME == FLUX_AUSM;
	AusmSide<T> own;
	if constexpr (shared_sides) own = ausm_side(qc, g, gr);
#endif
	unsigned ghosts = 0;  // slots with a ghost neighbour
#pragma unroll UNROLL
	for (int k = 0; k < (NSL == 4 ? 4 : sr.n); k++) {
		const int s = sr.s0 + k;
		const int mt = v.slot_mate[s];
		const bool left = mt >= 0;
		const int m = left ? mt : ~mt;
		const int nb = NSL == 4 ? (m < 4 * NR ? m >> 2 : m - 3 * NR) : v.slot_nbr[s];
		if (nb >= NR) ghosts |= 1u << k;
		Q5<T> qo, qn;
		if (ORDER1) {
			qo = qc;
			qn = ld5(v.Pin, v.NA, nb);
		} else {
			qo = ld5(v.FS, v.NS, s);
			qn = ld5(v.FS, v.NS, m);
		}
		const typename Vec4<T>::type geo = ldv4(v.sgeo + 4 * (size_t)s);
		if (FIRST) srad += (tabs((qc.u) * geo.x + (qc.v) * geo.y + (qc.w) * geo.z) + (cc)) * geo.w;
		Q5<T> L, R;
		for (int q = 0; q < 5; q++) {
			qv(L, q) = left ? qv(qo, q) : qv(qn, q);
			qv(R, q) = left ? qv(qn, q) : qv(qo, q);
		}
		T fc[5], fd[5];
#ifdef E3D_SHARED_SIDES
		if constexpr (shared_sides) {
			const AusmSide<T> nbr = ausm_side(qn, g, gr);
			// sides selected by value: a branch on the orientation would run the
			// face arithmetic twice in warps whose cells differ
			ausm_face_sides<T, DISS>(left ? own : nbr, left ? nbr : own, geo.x, geo.y, geo.z, geo.w, fc, fd);
		} else
#endif
		if (SCHEME == FLUX_ROE) {
			flux_central(L, R, geo.x, geo.y, geo.z, geo.w, gr, fc);
			if (DISS) flux_roe_diss(L, R, geo.x, geo.y, geo.z, geo.w, gr, gm1, fd);
		} else {
			flux_ausm_conv(L, R, geo.x, geo.y, geo.z, geo.w, g, gr, fc);
			if (DISS) flux_ausm_diss(L, R, geo.x, geo.y, geo.z, geo.w, g, gr, fd);
		}
		for (int q = 0; q < 5; q++) {
			ac[q] += left ? fc[q] : -fc[q];
			if (DISS) ad[q] += (left ? fd[q] : -fd[q]) * beta;
		}
	}
	double w0[5], wn[5];
	for (int q = 0; q < 5; q++) {
		if (last) v.Rc[q * (size_t)NR + c] = ac[q];
		if (DISS) v.Rd[q * (size_t)NR + c] = ad[q];
		if (FIRST && !carry_w0) {
			w0[q] = (double)conserved(qc, q, ph.gamma);
			v.W0[q * (size_t)NR + c] = w0[q];
		} else {
			w0[q] = v.W0[q * (size_t)NR + c];
		}
	}
	const T V = v.vol[c];
	T dt;
	if (FIRST) {
		dt = T(ph.cfl) * V / srad;
		v.dt[c] = dt;
	} else {
		dt = v.dt[c];
	}
	const T coef = alpha * dt / V;
	const Q5<T> qnew = conservative_update<T>(w0, coef, ac, ad, gm1, wn);
	st5(v.Pout, v.NA, c, qnew);
	if (last && carry_w0)
		for (int q = 0; q < 5; q++) v.W0[q * (size_t)NR + c] = wn[q];
	while (ghosts) {
		const int s = sr.s0 + __ffs(ghosts) - 1;
		ghosts &= ghosts - 1;
		int nb;
		if (NSL == 4) {
			const int mt = v.slot_mate[s];
			nb = (mt >= 0 ? mt : ~mt) - 3 * NR;
		} else {
			nb = v.slot_nbr[s];
		}
		const int kind = v.gkind[nb - NR];
		if (kind == GK_NONE) continue;
		// freestream of the ghost's case (batched cases differ in Mach and alpha)
		const double* f = v.case_free ? v.case_free + 5 * v.gcase[nb - NR] : ph.free;
		const Q5<T> fr{T(f[0]), T(f[1]), T(f[2]), T(f[3]), T(f[4])};
		const T* n = v.sgeo + 4 * (size_t)s;
		st5(v.Pout, v.NA, nb, ghost_state(kind, qnew, fr, n[0], n[1], n[2], g));
	}
}

// resident blocks per SM the FP64 flux pass is compiled for (5: 96 registers;
// 663k tets, Roe: 126 us at 5, 131 at 6, 136 at 7)
#ifndef E3D_FLUX64_MIN_BLOCKS
#define E3D_FLUX64_MIN_BLOCKS 5
#endif
template <class T, int SCHEME, bool ORDER1, int NSL, int MODE>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : E3D_FLUX64_MIN_BLOCKS) k_flux_update(FusedView<T> v, Physics ph, T alpha, T beta, int last, int carry_w0) {
	start_after_previous();
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c < v.NR) flux_update_cell<T, SCHEME, ORDER1, NSL, MODE>(v, ph, alpha, beta, last, carry_w0, c);
}

// FP64 pass 2 with one lane per slot, LPC lanes per cell (4: tetrahedra; 8: up to
// 6 slots).  flux_update_cell runs a cell's face fluxes one after the other in
// one thread, a dependent chain of ~2,000 FP64 operations (Roe): on a small mesh
// a launch is that latency (3k cells: 19 us, here 11).  Here each lane
// forms one face's flux, then the cell's lanes exchange them through shared
// memory and lane k adds up variable k over the slots in ascending face id
// (the reference's order, so FP64 results are the same bits) and updates it;
// lane 0 has the energy too.
template <int SCHEME, bool ORDER1, int LPC, int MODE>
__device__ __forceinline__ void flux_update_slots(const FusedView<double>& v, const Physics& ph, double alpha, double beta, int last,
                                                  int carry_w0, int c, bool in_range, double (*sm)[33]) {
	constexpr unsigned FULL = 0xffffffffu;
	constexpr bool DISS = MODE != STAGE_NODISS, FIRST = MODE == STAGE_FIRST;
	const int lane = threadIdx.x & 31, k = lane & (LPC - 1), first = lane - k;
	const int NR = v.NR;
	const double g = ph.gamma, gr = ph.gr, gm1 = ph.gm1;
	int s0 = LPC * c, n = LPC;
	if (LPC != 4) {
		s0 = v.slot_ptr[c];
		n = v.slot_ptr[c + 1] - s0;
	}
	const bool on = in_range && k < n;
	const int s = s0 + (k < n ? k : 0);
	const int mt = v.slot_mate[s];
	const bool left = mt >= 0;
	const int m = left ? mt : ~mt;
	const int nb = LPC == 4 ? (m < 4 * NR ? m >> 2 : m - 3 * NR) : v.slot_nbr[s];
	const double4 geo = ldv4(v.sgeo + 4 * (size_t)s);
	const double vol = v.vol[c];
	start_after_previous();
	const Q5<double> qo = ORDER1 ? ld5(v.Pin, v.NA, c) : ld5(v.FS, v.NS, s);
	const Q5<double> qn = ORDER1 ? ld5(v.Pin, v.NA, nb) : ld5(v.FS, v.NS, m);
	// this lane's share of the cell: variable k, and variable 4 on lane 0
	const int qk = k < 4 ? k : 0;
	const double keep = 1.0 - beta;
	double rd = 0.0, rd4 = 0.0;
	if (!DISS || keep != 0.0) {  // beta = 1 (the first stage) drops the old value
		rd = v.Rd[(size_t)qk * NR + c];
		if (k == 0) rd4 = v.Rd[4 * (size_t)NR + c];
	}
	Q5<double> qc;
	if (FIRST) qc = ORDER1 ? qo : ld5(v.Pin, v.NA, c);
	double w0, w04 = 0.0;
	if (FIRST && !carry_w0) {
		w0 = conserved(qc, qk, ph.gamma);
		w04 = conserved(qc, 4, ph.gamma);
		if (in_range && k < 4) v.W0[(size_t)k * NR + c] = w0;
		if (in_range && k == 0) v.W0[4 * (size_t)NR + c] = w04;
	} else {
		w0 = v.W0[(size_t)qk * NR + c];
		if (k == 0) w04 = v.W0[4 * (size_t)NR + c];
	}
	double dt;
	if (FIRST) {  // ahead of the fluxes, whose arithmetic covers its divisions
		sm[10][lane] = (fabs((qc.u) * geo.x + (qc.v) * geo.y + (qc.w) * geo.z) + (sqrt(g * qc.p / qc.r))) * geo.w;
		__syncwarp();
		double srad = 0.0;
#pragma unroll
		for (int i = 0; i < (LPC == 4 ? 4 : MAXSL); i++) {
			if (LPC != 4 && i >= n) break;
			srad += sm[10][first + i];
		}
		dt = ph.cfl * vol / srad;
		if (in_range && k == 0) v.dt[c] = dt;
	} else {
		dt = v.dt[c];
	}
	const double coef = alpha * dt / vol;
	{
		Q5<double> L, R;
		for (int q = 0; q < 5; q++) {
			qv(L, q) = left ? qv(qo, q) : qv(qn, q);
			qv(R, q) = left ? qv(qn, q) : qv(qo, q);
		}
		double fc[5], fd[5];
		if (SCHEME == FLUX_ROE) {
			flux_central(L, R, geo.x, geo.y, geo.z, geo.w, gr, fc);
			if (DISS) flux_roe_diss(L, R, geo.x, geo.y, geo.z, geo.w, gr, gm1, fd);
		} else {
			flux_ausm_conv(L, R, geo.x, geo.y, geo.z, geo.w, g, gr, fc);
			if (DISS) flux_ausm_diss(L, R, geo.x, geo.y, geo.z, geo.w, g, gr, fd);
		}
#pragma unroll
		for (int q = 0; q < 5; q++) {
			sm[q][lane] = left ? fc[q] : -fc[q];
			if (DISS) sm[5 + q][lane] = left ? fd[q] : -fd[q];
		}
	}
	__syncwarp();
	double ac = 0.0, ad = DISS ? rd * keep : rd, ac4 = 0.0, ad4 = DISS ? rd4 * keep : rd4;
#pragma unroll
	for (int i = 0; i < (LPC == 4 ? 4 : MAXSL); i++) {
		if (LPC != 4 && i >= n) break;
		ac += sm[qk][first + i];
		if (DISS) ad += sm[5 + qk][first + i] * beta;
		if (k == 0) {
			ac4 += sm[4][first + i];
			if (DISS) ad4 += sm[9][first + i] * beta;
		}
	}
	const double wn = w0 - coef * (ac - ad);
	const double wn4 = w04 - coef * (ac4 - ad4);
	const double r = __shfl_sync(FULL, wn, first);
	const double mx = __shfl_sync(FULL, wn, first + 1), my = __shfl_sync(FULL, wn, first + 2),
	             mz = __shfl_sync(FULL, wn, first + 3);
	// one division per lane: the velocity component, on lane 0 the kinetic energy
	const double x = (k == 0 ? 0.5 * (mx * mx + my * my + mz * mz) : wn) / r;
	const double qnew = k == 0 ? r : x;
	const double pnew = (gm1 * (wn4 - x));
	if (in_range && k < 4) {
		if (last) v.Rc[(size_t)k * NR + c] = ac;
		if (DISS) v.Rd[(size_t)k * NR + c] = ad;
		v.Pout[4 * (size_t)c + k] = qnew;
		if (last && carry_w0) v.W0[(size_t)k * NR + c] = wn;
		if (k == 0) {
			if (last) v.Rc[4 * (size_t)NR + c] = ac4;
			if (DISS) v.Rd[4 * (size_t)NR + c] = ad4;
			v.Pout[4 * (size_t)v.NA + c] = pnew;
			if (last && carry_w0) v.W0[4 * (size_t)NR + c] = wn4;
		}
	}
	// boundary conditions of the cell's ghost cells
	const bool ghost = on && nb >= NR;
	if (__any_sync(FULL, ghost)) {
		Q5<double> q;
		q.r = __shfl_sync(FULL, qnew, first);
		q.u = __shfl_sync(FULL, qnew, first + 1);
		q.v = __shfl_sync(FULL, qnew, first + 2);
		q.w = __shfl_sync(FULL, qnew, first + 3);
		q.p = __shfl_sync(FULL, pnew, first);
		const int kind = ghost ? v.gkind[nb - NR] : (int)GK_NONE;
		if (kind != GK_NONE) {
			// freestream of the ghost's case (batched cases differ in Mach and alpha)
			const double* f = v.case_free ? v.case_free + 5 * v.gcase[nb - NR] : ph.free;
			const Q5<double> fr{f[0], f[1], f[2], f[3], f[4]};
			st5(v.Pout, v.NA, nb, ghost_state(kind, q, fr, geo.x, geo.y, geo.z, g));
		}
	}
}

template <int SCHEME, bool ORDER1, int LPC, int MODE>
__global__ void __launch_bounds__(128, 4)
    k_flux_slots(FusedView<double> v, Physics ph, double alpha, double beta, int last, int carry_w0) {
	__shared__ double sm[4][MODE == STAGE_FIRST ? 11 : MODE == STAGE_DISS ? 10 : 5][33];
	const int c = (blockIdx.x * 128 + threadIdx.x) / LPC;
	const bool in_range = c < v.NR;
	if (!__any_sync(0xffffffffu, in_range)) start_after_previous();
	else
		flux_update_slots<SCHEME, ORDER1, LPC, MODE>(v, ph, alpha, beta, last, carry_w0, in_range ? c : v.NR - 1,
		                                                in_range, sm[threadIdx.x >> 5]);
}

// ===================================================================== reductions
// End of an outer iteration: residual norms (Convergence::calculate*Rms,
// PostProcessing/src/Convergence.cpp:27-143), wall forces
// (AerodynamicParameters::computeAerodynamic, AerodynamicParameters.cpp:189-232)
// and the inter-block halo.  k_tail does every parallel part in one launch
// (chunk sums of (Rc-Rd)^2, per-face force terms, halo copies) and writes the
// sums' inputs to slot *pend of a small ring; k_tail_sums then adds up all
// pending iterations at once, one thread block per (iteration, mesh block).
// The force sums keep the reference's wall-face order, a serial chain of FP64
// adds (2.7k faces: 71 us per iteration as a kernel of its own); with up to
// 32 iterations pending (tail_slots) the chains run side by side, and their time is
// paid once per call instead of once per iteration.  B200, tail and sums of one
// iteration back to back, as six kernels / these two: 1.3k cells 23.5 / 13.3 us, 48k
// 47 / 19, 304k (2,738 wall faces) 85 / 30; the sums, most of it, are now shared by
// the iterations of the ring.

// Sum of n values in ascending order by one warp (every lane returns it): the
// next 128 are in flight while 128 are added from shared memory.
__device__ __forceinline__ double warp_ordered_sum(const double* __restrict__ x, int n, double* buf) {
	const int lane = threadIdx.x & 31;
	double nx[4], acc = 0.;
#pragma unroll
	for (int j = 0; j < 4; j++) nx[j] = 32 * j + lane < n ? x[32 * j + lane] : 0.;
	for (int base = 0; base < n; base += 128) {
		__syncwarp();
#pragma unroll
		for (int j = 0; j < 4; j++) buf[32 * j + lane] = nx[j];
		__syncwarp();
		const int m = min(128, n - base);
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const int i = base + 128 + 32 * j + lane;
			nx[j] = i < n ? x[i] : 0.;
		}
		if (m == 128) {
			const double2* b2 = reinterpret_cast<const double2*>(buf);
#pragma unroll 16
			for (int i = 0; i < 64; i++) {
				const double2 t = b2[i];
				acc += t.x;
				acc += t.y;
			}
		} else {
			for (int i = 0; i < m; i++) acc += buf[i];
		}
	}
	return acc;
}

// Force terms of one wall face: fy, fx, cmx, cmy, cmz.
__device__ __forceinline__ void wall_face_terms(double p0, double p1, double denom, const double* __restrict__ S,
                                                const double* __restrict__ fc, double out[5]) {
	const double pbc = 0.5 * (p0 + p1);
	const double cp = (pbc - 1.) / denom;
	const double fx = cp * S[0], fy = cp * S[1], fz = cp * S[2];
	const double x = fc[0], y = fc[1], z = fc[2];
	out[0] = fy;
	out[1] = fx;
	out[2] = y * fz - z * fy;
	out[3] = z * fx - x * fz;
	out[4] = x * fy - y * fx;
}

// grid = one block per norm chunk (at most TAIL_CHUNK cells of one mesh block),
// then wall faces, then halo entries, TAIL_TPB of each per block.  The chunks are
// listed: a grid of the largest mesh block's chunks for each of them launches
// mostly empty blocks, and keeps partials for them (B200, one 384k-cell mesh beside
// 250 of 750 cells, 100 first-order iterations of the batch: FP32 35.8 ms so, 16.4
// listed; FP64 61.8 and 42.6).  The last block to finish moves *pend on, after every
// block has read it.
template <class T>
__global__ void __launch_bounds__(TAIL_TPB) k_tail(ReduceArgs a, const T* Rc, const T* Rd, T* P, T* P2) {
	const int t = threadIdx.x, n_norm = a.n_chunks, n_wb = (a.n_wall + TAIL_TPB - 1) / TAIL_TPB;
	int w = blockIdx.x;
	const int4 ch = w < n_norm ? a.chunk[w] : make_int4(0, 0, 0, 0);
	start_after_previous();
	const int slot = *a.pend;
	if (w < n_norm) {
		const bool frozen = a.block_work && a.block_work[ch.z] == a.block_work[ch.z + 1];
		const int beg = ch.x, end = frozen ? beg : ch.y;
		double acc[5] = {0., 0., 0., 0., 0.};
#pragma unroll
		for (int j = 0; j < TAIL_CHUNK / TAIL_TPB; j++) {
			const int c = beg + j * TAIL_TPB + t;
			if (c < end)
#pragma unroll
				for (int q = 0; q < 5; q++) {
					const double r = (double)Rc[q * (size_t)a.NR + c] - (double)Rd[q * (size_t)a.NR + c];
					acc[q] += r * r;
				}
		}
		__shared__ double sm[5][TAIL_TPB / 32];
#pragma unroll
		for (int q = 0; q < 5; q++) {
			for (int h = 16; h > 0; h >>= 1) acc[q] += __shfl_down_sync(0xffffffffu, acc[q], h);
			if ((t & 31) == 0) sm[q][t >> 5] = acc[q];
		}
		__syncthreads();
		if (t < 5) {
			double s = 0.;
			for (int i = 0; i < TAIL_TPB / 32; i++) s += sm[t][i];
			a.partial[((size_t)slot * 5 + t) * n_norm + w] = s;
		}
	} else if ((w -= n_norm) < n_wb) {
		const int i = w * TAIL_TPB + t;
		if (i < a.n_wall) {
			const int f = a.wall_face[i];
			const size_t i0 = 4 * (size_t)a.NA + a.face_lr[2 * f], i1 = 4 * (size_t)a.NA + a.face_lr[2 * f + 1];
			double p0 = (double)P[i0], p1 = (double)P[i1], o[5];
			if (a.Pb64) {
				p0 += a.Pb64[i0];
				p1 += a.Pb64[i1];
			}
			wall_face_terms(p0, p1, a.wall_denom ? a.wall_denom[i] : a.denom, a.S + 3 * (size_t)f, a.fc + 3 * (size_t)f, o);
#pragma unroll
			for (int q = 0; q < 5; q++) a.wall_terms[((size_t)slot * 5 + q) * a.n_wall + i] = o[q];
		}
	} else {
		const int i = (w - n_wb) * TAIL_TPB + t;
		if (i < a.n_halo) {
			const int d = a.halo_dst[i];
			const Q5<T> q = ld5(P, a.NA, a.halo_src[i]);
			st5(P, a.NA, d, q);
			st5(P2, a.NA, d, q);
			if (a.rec) {
				const float4* r = reinterpret_cast<const float4*>(a.rec + 8 * (size_t)a.halo_src[i]);
				const float4 x = r[0], y = r[1];
				for (float* o : {a.rec, a.rec2}) {
					reinterpret_cast<float4*>(o + 8 * (size_t)d)[0] = x;
					reinterpret_cast<float4*>(o + 8 * (size_t)d)[1] = y;
				}
			}
		}
	}
	__syncthreads();
	if (t == 0) {
		__threadfence();
		if (atomicAdd(a.ticket, 1u) == gridDim.x - 1) {
			*a.ticket = 0u;
			*a.pend = slot + 1;
		}
	}
}

// hist[(*d_iter + i)*stride + b*10 + ...] for the pending iterations i (grid.y)
// of block b (grid.x), warp q summing component q: norm chunks by a fixed tree,
// wall faces in order.  Sets *bad when a norm is not finite (NaN propagates
// silently in the reference).  The last block clears *pend and, with `advance`,
// moves *d_iter on.
__global__ void __launch_bounds__(160) k_tail_sums(ReduceArgs a, int advance) {
	start_after_previous();
	__shared__ __align__(16) double buf[5][128];
	const int q = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x, i = blockIdx.y;
	const int base = *a.d_iter;
	const double* part = a.partial + ((size_t)i * 5 + q) * a.n_chunks + a.chunk_off[b];
	const int nc = a.chunk_off[b + 1] - a.chunk_off[b];
	double s = 0.;
	for (int k = lane; k < nc; k += 32) s += part[k];
	for (int h = 16; h > 0; h >>= 1) s += __shfl_down_sync(0xffffffffu, s, h);
	const int beg = a.wall_off[b], end = a.wall_off[b + 1];
	const double f = warp_ordered_sum(a.wall_terms + ((size_t)i * 5 + q) * a.n_wall + beg, end - beg, buf[q]);
	if (lane == 0) {
		double* out = a.hist + (size_t)(base + i) * a.stride + b * 10;
		out[q] = s;
		out[5 + q] = f;
		if (!isfinite(s)) *a.d_bad = 1;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		if (atomicAdd(a.ticket, 1u) == gridDim.x * gridDim.y - 1) {
			*a.ticket = 0u;
			*a.pend = 0;
			if (advance) *a.d_iter = base + gridDim.y;
		}
	}
}

// ===================================================================== batches
// Phases of one outer iteration over a work list (tiles of real cells of the
// active cases), shared by the persistent kernel and the tiled per-pass
// kernels.  TPB threads cooperate on one tile.

// Sum of (Rc-Rd)^2 over the cells of tile w, fixed tree order (red: [5][TPB]).
template <class T, int TPB>
__device__ __forceinline__ void tile_norms(const FusedView<T>& vf, const PersistArgs& a, int w, double (*red)[TPB]) {
	const int4 t = a.work[w];
	double acc[5] = {0., 0., 0., 0., 0.};
	for (int c = t.x + threadIdx.x; c < t.y; c += TPB)
		for (int q = 0; q < 5; q++) {
			const double r = (double)vf.Rc[q * vf.NR + c] - (double)vf.Rd[q * vf.NR + c];
			acc[q] += r * r;
		}
	for (int q = 0; q < 5; q++) red[q][threadIdx.x] = acc[q];
	__syncthreads();
	for (int h = TPB / 2; h > 0; h >>= 1) {
		if (threadIdx.x < h)
			for (int q = 0; q < 5; q++) red[q][threadIdx.x] += red[q][threadIdx.x + h];
		__syncthreads();
	}
	if (threadIdx.x < 5) a.wpart[(size_t)w * 5 + threadIdx.x] = red[threadIdx.x][0];
	__syncthreads();
}

// Force terms of wall faces i0, i0+stride, ... (frozen cases included: cheap, ignored by the host).
template <class T>
__device__ __forceinline__ void wall_terms_range(const FusedView<T>& vf, const PersistArgs& a, int i0, int stride) {
	for (int i = i0; i < a.n_wall; i += stride) {
		const int f = a.wall_face[i];
		const T* p = vf.Pin + 4 * (size_t)vf.NA;
		double o[5];
		wall_face_terms((double)p[a.face_lr[2 * f]], (double)p[a.face_lr[2 * f + 1]],
		                a.wall_denom ? a.wall_denom[i] : a.denom, a.S + 3 * (size_t)f, a.fc + 3 * (size_t)f, o);
		for (int q = 0; q < 5; q++) a.wall_terms[q * (size_t)a.n_wall + i] = o[q];
	}
}

// Inter-block halo copies i0, i0+stride, ... into both primitive buffers.
template <class T>
__device__ __forceinline__ void halo_range(const FusedView<T>& vf, const PersistArgs& a, int i0, int stride) {
	for (int i = i0; i < a.n_halo; i += stride) {
		const Q5<T> q = ld5(vf.Pin, vf.NA, a.halo_src[i]);
		st5(const_cast<T*>(vf.Pin), vf.NA, a.halo_dst[i], q);
		st5(vf.Pout, vf.NA, a.halo_dst[i], q);
	}
}

// Per-block sums of block b into history slot `slot`: tiles in a fixed tree
// order, wall faces sequentially in the reference's order.
template <int TPB>
__device__ __forceinline__ void block_sums(const PersistArgs& a, int b, int slot, double (*red)[TPB], double (*wbuf)[128]) {
	const int w0 = a.block_work[b], w1 = a.block_work[b + 1], warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	double acc[5] = {0., 0., 0., 0., 0.};
	for (int w = w0 + threadIdx.x; w < w1; w += TPB)
		for (int q = 0; q < 5; q++) acc[q] += a.wpart[(size_t)w * 5 + q];
	for (int q = 0; q < 5; q++) red[q][threadIdx.x] = acc[q];
	__syncthreads();
	for (int h = TPB / 2; h > 0; h >>= 1) {
		if (threadIdx.x < h)
			for (int q = 0; q < 5; q++) red[q][threadIdx.x] += red[q][threadIdx.x + h];
		__syncthreads();
	}
	double* out = a.hist + (size_t)slot * a.stride + b * 10;
	if (threadIdx.x < 5) {
		out[threadIdx.x] = red[threadIdx.x][0];
		if (!isfinite(red[threadIdx.x][0]) && w1 > w0) *a.d_bad = 1;
	}
	const int beg = a.wall_off[b], end = a.wall_off[b + 1];
	for (int q = warp; q < 5; q += TPB / 32) {
		const double f = warp_ordered_sum(a.wall_terms + q * (size_t)a.n_wall + beg, end - beg, wbuf[warp]);
		if (lane == 0) out[5 + q] = f;
	}
	__syncthreads();
}

// Persistent form: one cooperative launch runs `iters` outer iterations;
// phases are separated by grid-wide barriers.  Tiles of converged cases are
// absent from the work list.
template <class T, int GRAD, int LIM, int SCHEME, bool ORDER2, int TPB>
__global__ void __launch_bounds__(TPB, 512 / TPB) k_persistent(FusedView<T> v0, FusedView<T> v1, Physics ph,
                                                               PersistArgs a) {
	namespace cg = cooperative_groups;
	cg::grid_group grid = cg::this_grid();
	__shared__ double red[5][TPB];
	__shared__ __align__(16) double wbuf[TPB / 32][128];
	const int base = *a.d_iter;
	int parity = a.start_parity;  // which primitive buffer holds the current state
	for (int it = 0; it < a.iters; it++) {
		for (int s = 0; s < a.stages; s++) {
			const FusedView<T>& v = parity ? v1 : v0;
			if (ORDER2) {
				for (int w = blockIdx.x; w < a.n_work; w += gridDim.x) {
					const int4 t = a.work[w];
					for (int c = t.x + threadIdx.x; c < t.y; c += TPB) recon_cell<T, GRAD, LIM>(v, ph, c);
				}
				grid.sync();
			}
			const T al = T(a.alpha[s]), be = T(a.beta[s]);
			const int last = s == a.stages - 1;
			for (int w = blockIdx.x; w < a.n_work; w += gridDim.x) {
				const int4 t = a.work[w];
				for (int c = t.x + threadIdx.x; c < t.y; c += TPB) {
					if (s == 0) flux_update_cell<T, SCHEME, !ORDER2, 4, STAGE_FIRST>(v, ph, al, be, last, a.carry, c);
					else if (a.beta[s] != 0.0) flux_update_cell<T, SCHEME, !ORDER2, 4, STAGE_DISS>(v, ph, al, be, last, a.carry, c);
					else flux_update_cell<T, SCHEME, !ORDER2, 4, STAGE_NODISS>(v, ph, al, be, last, a.carry, c);
				}
			}
			grid.sync();
			parity ^= 1;
		}
		const FusedView<T>& vf = parity ? v1 : v0;  // Pin of the next stage = current state
		for (int w = blockIdx.x; w < a.n_work; w += gridDim.x) tile_norms<T, TPB>(vf, a, w, red);
		wall_terms_range(vf, a, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
		halo_range(vf, a, blockIdx.x * TPB + threadIdx.x, gridDim.x * TPB);
		grid.sync();
		const int slot = min(base + it, a.hist_capacity - 1);
		for (int b = blockIdx.x; b < a.nblocks; b += gridDim.x) block_sums<TPB>(a, b, slot, red, wbuf);
		grid.sync();
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) *a.d_iter = base + a.iters;
}

// Tiled per-pass form: the same phases as separate launches over the work
// list (one block of 128 threads per tile of at most 128 cells), captured in a
// CUDA graph by the host.  Each pass keeps only its own registers and shared
// memory, so more warps stay resident than in the persistent kernel.
template <class T, int GRAD, int LIM>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 4) k_recon_tiles(FusedView<T> v, Physics ph,
                                                                             const int4* __restrict__ work) {
	start_after_previous();
	const int4 t = work[blockIdx.x];
	const int c = t.x + threadIdx.x;
	if (c < t.y) recon_cell<T, GRAD, LIM>(v, ph, c);
}

template <class T, int SCHEME, bool ORDER1, int MODE>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 8 : 4) k_flux_update_tiles(FusedView<T> v, Physics ph, T alpha,
                                                                                   T beta, int last, int carry_w0,
                                                                                   const int4* __restrict__ work) {
	start_after_previous();
	const int4 t = work[blockIdx.x];
	const int c = t.x + threadIdx.x;
	if (c < t.y) flux_update_cell<T, SCHEME, ORDER1, 4, MODE>(v, ph, alpha, beta, last, carry_w0, c);
}

}  // namespace
}  // namespace e3d
