// Launcher templates shared by k64.cu and k32.cu (each instantiates its T).
#pragma once
#include "kernels.cuh"
#include "launch.hpp"

namespace e3d {

template <class T>
void launch_halo(int n, const int* dst, const int* src, int NA, T* b0, T* b1, cudaStream_t st) {
	if (n > 0) launch_next(k_halo<T>, (n + 127) / 128, 128, 0, st, n, dst, src, NA, b0, b1);
}

template <class T>
void launch_halo_pack(int n, const int* src, int NA, const T* P, T* buf, cudaStream_t st) {
	if (n > 0) k_halo_pack<T><<<(n + 127) / 128, 128, 0, st>>>(n, src, NA, P, buf);
}

template <class T>
void launch_halo_unpack(int n, const int* dst, int NA, const T* buf, T* b0, T* b1, cudaStream_t st) {
	if (n > 0) k_halo_unpack<T><<<(n + 127) / 128, 128, 0, st>>>(n, dst, NA, buf, b0, b1);
}

template <class T>
void launch_tail(const ReduceArgs& a, const T* Rc, const T* Rd, T* P, T* P2, cudaStream_t st) {
	const auto blocks = [](int n) { return (n + TAIL_TPB - 1) / TAIL_TPB; };
	const int grid = a.n_chunks + blocks(a.n_wall) + blocks(a.n_halo);
	launch_next(k_tail<T>, grid, TAIL_TPB, 0, st, a, Rc, Rd, P, P2);
}

// Which pass reconstructs: see k_recon_var.
template <class T, int GRAD, int LIM>
void recon_pass(const FusedView<T>& v, const Physics& ph, cudaStream_t st) {
	const int grid = (v.NR + 127) / 128, gv = (v.NR + RV_CELLS - 1) / RV_CELLS;
	if (!v.tet4) launch_next(k_recon_var<T, GRAD, LIM, 0>, gv, 5 * RV_CELLS, 0, st, v, ph);
	else if constexpr (sizeof(T) == 8) launch_next(k_recon_var<T, GRAD, LIM, 4>, gv, 5 * RV_CELLS, 0, st, v, ph);
	else launch_next(k_recon<GRAD, LIM>, grid, 128, 0, st, v, ph);
}

template <class T>
void launch_recon(const FusedView<T>& v, const Physics& ph, int grad, int lim, cudaStream_t st) {
	if (v.NR <= 0) return;
	if (grad == GRAD_LEAST_SQUARES) {
		if (lim == LIM_VENKATAKRISHNAN) recon_pass<T, GRAD_LEAST_SQUARES, LIM_VENKATAKRISHNAN>(v, ph, st);
		else recon_pass<T, GRAD_LEAST_SQUARES, LIM_BARTH_JESPERSEN>(v, ph, st);
	} else {
		if (lim == LIM_VENKATAKRISHNAN) recon_pass<T, GRAD_GREEN_GAUSS, LIM_VENKATAKRISHNAN>(v, ph, st);
		else recon_pass<T, GRAD_GREEN_GAUSS, LIM_BARTH_JESPERSEN>(v, ph, st);
	}
}

// Largest mesh whose FP64 flux pass runs one lane per slot.  Below it a launch is
// latency: four times the threads, each with a quarter of the chain.  Above it the
// exchange through shared memory (and, on hexahedra, two idle lanes of eight) costs
// more than it hides.  B200, us a launch with dissipation, per cell / per slot.
// Tetrahedra: Roe 25k 22 / 15, 132k 40 / 34, 216k 54 / 52 (second order 57 / 58; without
// dissipation 25 / 30), 384k 81 / 92; AUSM 25k 16.5 / 12.7, 83k 19.9 / 20.5, 132k 25 / 27.
// Hexahedra: Roe 20k 26 / 19, 64k 32 / 36; AUSM 20k 20.5 / 16.2, 64k 23 / 29.
// FP32 gains little (3k 10 / 8, 48k 10.5 / 10.6) and keeps one form, so that the
// batch kernels and this path round alike.
constexpr int slot_pass_cells(int scheme, bool tet) {
	return scheme == FLUX_ROE ? (tet ? 180000 : 40000) : (tet ? 60000 : 30000);
}

template <class T>
void launch_flux_update(const FusedView<T>& v, const Physics& ph, int scheme, bool order1, bool first, double alpha,
                        double beta, int last, int carry, cudaStream_t st) {
	if (v.NR <= 0) return;
	const int grid = (v.NR + 127) / 128, g4 = (v.NR + 31) / 32, g8 = (v.NR + 15) / 16;
	const bool slots = sizeof(T) == 8 && v.NR <= slot_pass_cells(scheme, v.tet4);
	const T a = T(alpha), b = T(beta);
#define E3D_FLUX_D(S, O, D)                                                                                \
	do {                                                                                                   \
		if constexpr (sizeof(T) == 8)                                                                      \
			if (slots) {                                                                                   \
				if (v.tet4) launch_next(k_flux_slots<S, O, 4, D>, g4, 128, 0, st, v, ph, a, b, last, carry);        \
				else launch_next(k_flux_slots<S, O, 8, D>, g8, 128, 0, st, v, ph, a, b, last, carry);               \
				break;                                                                                     \
			}                                                                                              \
		if (v.tet4) launch_next(k_flux_update<T, S, O, 4, D>, grid, 128, 0, st, v, ph, a, b, last, carry);          \
		else launch_next(k_flux_update<T, S, O, 0, D>, grid, 128, 0, st, v, ph, a, b, last, carry);                 \
	} while (0)
#define E3D_FLUX(S, O)                                                                                     \
	do {                                                                                                   \
		if (first) E3D_FLUX_D(S, O, STAGE_FIRST);                                                          \
		else if (beta != 0.0) E3D_FLUX_D(S, O, STAGE_DISS);                                                \
		else E3D_FLUX_D(S, O, STAGE_NODISS);                                                               \
	} while (0)
	if (scheme == FLUX_AUSM) {
		if (order1) E3D_FLUX(FLUX_AUSM, true);
		else E3D_FLUX(FLUX_AUSM, false);
	} else {
		if (order1) E3D_FLUX(FLUX_ROE, true);
		else E3D_FLUX(FLUX_ROE, false);
	}
#undef E3D_FLUX
#undef E3D_FLUX_D
}

}  // namespace e3d
