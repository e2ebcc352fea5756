// Batch launchers (persistent cooperative kernel and tiled per-pass form).
// Included by k32.cu and k64.cu with E3D_BATCH_NS = batch, and by k64f.cu
// with E3D_BATCH_NS = batch_fast: the same kernels compiled with FMA
// contraction for the FP64 finishing phase of batched solves.
#pragma once
#include "kernels.cuh"
#include "launch.hpp"

#ifndef E3D_BATCH_NS
#define E3D_BATCH_NS batch
#endif

namespace e3d {
namespace E3D_BATCH_NS {

// ---- persistent batch kernel (cooperative launch)
constexpr int PERSIST_TPB = 128;

template <class T, int GRAD, int LIM, int SCHEME, bool ORDER2>
void* persistent_fn() {
	return reinterpret_cast<void*>(&k_persistent<T, GRAD, LIM, SCHEME, ORDER2, PERSIST_TPB>);
}

template <class T>
void* persistent_select(int grad, int lim, int scheme, bool order2) {
#define E3D_P(G, L, S)                                                                      \
	if (grad == G && lim == L && scheme == S)                                               \
		return order2 ? persistent_fn<T, G, L, S, true>() : persistent_fn<T, G, L, S, false>();
	E3D_P(GRAD_GREEN_GAUSS, LIM_BARTH_JESPERSEN, FLUX_ROE)
	E3D_P(GRAD_GREEN_GAUSS, LIM_BARTH_JESPERSEN, FLUX_AUSM)
	E3D_P(GRAD_GREEN_GAUSS, LIM_VENKATAKRISHNAN, FLUX_ROE)
	E3D_P(GRAD_GREEN_GAUSS, LIM_VENKATAKRISHNAN, FLUX_AUSM)
	E3D_P(GRAD_LEAST_SQUARES, LIM_BARTH_JESPERSEN, FLUX_ROE)
	E3D_P(GRAD_LEAST_SQUARES, LIM_BARTH_JESPERSEN, FLUX_AUSM)
	E3D_P(GRAD_LEAST_SQUARES, LIM_VENKATAKRISHNAN, FLUX_ROE)
	E3D_P(GRAD_LEAST_SQUARES, LIM_VENKATAKRISHNAN, FLUX_AUSM)
#undef E3D_P
	return nullptr;
}

template <class T>
int persistent_blocks_per_sm(int grad, int lim, int scheme, bool order2) {
	int n = 0;
	void* fn = persistent_select<T>(grad, lim, scheme, order2);
	if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, PERSIST_TPB, 0) != cudaSuccess) return 0;
	return n;
}

template <class T>
cudaError_t launch_persistent(const FusedView<T>& v0, const FusedView<T>& v1, const Physics& ph, const PersistArgs& a,
                              int grad, int lim, int scheme, bool order2, int grid, cudaStream_t st) {
	void* fn = persistent_select<T>(grad, lim, scheme, order2);
	if (!fn) return cudaErrorInvalidValue;
	FusedView<T> x0 = v0, x1 = v1;
	Physics p = ph;
	PersistArgs q = a;
	void* args[] = {&x0, &x1, &p, &q};
	return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(PERSIST_TPB), args, 0, st);
}

// ---- tiled per-pass batch iterations (enqueued on `st`, captured by the caller)
template <class T, int GRAD, int LIM>
void recon_tiles(const FusedView<T>& v, const Physics& ph, int n_work, const int4* work, cudaStream_t st) {
	launch_next(k_recon_tiles<T, GRAD, LIM>, n_work, 128, 0, st, v, ph, work);
}

template <class T, int SCHEME, bool ORDER1>
void flux_tiles(const FusedView<T>& v, const Physics& ph, bool first, bool diss, T al, T be, int last, int carry,
                int n_work, const int4* work, cudaStream_t st) {
	const auto kernel = first  ? k_flux_update_tiles<T, SCHEME, ORDER1, STAGE_FIRST>
	                    : diss ? k_flux_update_tiles<T, SCHEME, ORDER1, STAGE_DISS>
	                           : k_flux_update_tiles<T, SCHEME, ORDER1, STAGE_NODISS>;
	launch_next(kernel, n_work, 128, 0, st, v, ph, al, be, last, carry, work);
}

template <class T>
cudaError_t launch_tiled_iterations(const FusedView<T>& v0, const FusedView<T>& v1, const Physics& ph,
                                    const PersistArgs& a, const ReduceArgs& r, int grad, int lim, int scheme, bool order2,
                                    cudaStream_t st) {
	if (a.n_work <= 0) return cudaSuccess;
	int parity = a.start_parity;
	for (int it = 0; it < a.iters; it++) {
		for (int s = 0; s < a.stages; s++) {
			const FusedView<T>& v = parity ? v1 : v0;
			if (order2) {
				if (grad == GRAD_LEAST_SQUARES) {
					if (lim == LIM_VENKATAKRISHNAN)
						recon_tiles<T, GRAD_LEAST_SQUARES, LIM_VENKATAKRISHNAN>(v, ph, a.n_work, a.work, st);
					else
						recon_tiles<T, GRAD_LEAST_SQUARES, LIM_BARTH_JESPERSEN>(v, ph, a.n_work, a.work, st);
				} else {
					if (lim == LIM_VENKATAKRISHNAN)
						recon_tiles<T, GRAD_GREEN_GAUSS, LIM_VENKATAKRISHNAN>(v, ph, a.n_work, a.work, st);
					else
						recon_tiles<T, GRAD_GREEN_GAUSS, LIM_BARTH_JESPERSEN>(v, ph, a.n_work, a.work, st);
				}
			}
			const T al = T(a.alpha[s]), be = T(a.beta[s]);
			const int last = s == a.stages - 1;
			const bool diss = a.beta[s] != 0.0;
			const auto flux = scheme == FLUX_AUSM ? (order2 ? flux_tiles<T, FLUX_AUSM, false> : flux_tiles<T, FLUX_AUSM, true>)
			                                      : (order2 ? flux_tiles<T, FLUX_ROE, false> : flux_tiles<T, FLUX_ROE, true>);
			flux(v, ph, s == 0, diss, al, be, last, a.carry, a.n_work, a.work, st);
			parity ^= 1;
		}
		end_iteration<T>(parity ? v1 : v0, r, it, a.iters, st);
	}
	return cudaGetLastError();
}

}  // namespace E3D_BATCH_NS
}  // namespace e3d
