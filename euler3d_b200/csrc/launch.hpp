// Host-callable kernel launchers.  k64.cu (built with -fmad=false, so double
// arithmetic keeps the reference's rounding) defines the FP64 granular kernels
// and the double instantiations; k32.cu defines the float instantiations.
#pragma once
#include <cuda_runtime.h>

#include "views.hpp"

namespace e3d {

// Launches a kernel that starts with start_after_previous(): its blocks are
// scheduled while the previous kernel on the stream drains, which hides the
// launch, the ramp-up and the loads before the wait.  Captured launches become
// programmatic graph edges.  B200, a pass with / without: 20 iterations of 1.3k
// cells FP64 749 / 829 us, 50 of 48k 3337 / 3505, strategy calls on 82k 1336 / 1580;
// no difference from 300k cells.  The difference form's stages are launched without
// (15.6 / 15.3 ms for 100 iterations).
template <class... P, class... A>
void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
	cudaLaunchAttribute attr{};
	attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr.val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cfg.attrs = &attr;
	cfg.numAttrs = 1;
	cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// ---- granular FP64 drop-in kernels (one per reference strategy method) ----
void launch_save_w0(const GeoView&, const StateView&, const Physics&, int r0, int r1, cudaStream_t);
void launch_spectral_radius(const GeoView&, const StateView&, const Physics&, int r0, int r1, cudaStream_t);
void launch_timestep(const GeoView&, const StateView&, const Physics&, int r0, int r1, cudaStream_t);
void launch_gradients(const GeoView&, const StateView&, int kind, int r0, int r1, cudaStream_t);
void launch_limiters(const GeoView&, const StateView&, const Physics&, int kind, int r0, int r1, int g0, int g1,
                     cudaStream_t);
void launch_flux_conv(const GeoView&, const StateView&, const Physics&, int scheme, int r0, int r1, cudaStream_t);
void launch_flux_diss(const GeoView&, const StateView&, const Physics&, int scheme, double beta, int r0, int r1,
                      cudaStream_t);
void launch_update(const GeoView&, const StateView&, const Physics&, double alpha, int r0, int r1, cudaStream_t);
void launch_bc(const GeoView&, const StateView&, const Physics&, int g0, int g1, cudaStream_t);
// central implicit residual smoothing of Rc and Rd (j1: 10 x NR FP64 scratch)
void launch_smooth(const GeoView&, const StateView&, double* j1, int r0, int r1, cudaStream_t);

// ---- shared by both paths, per precision ----
template <class T>
void launch_halo(int n, const int* dst, const int* src, int NA, T* b0, T* b1, cudaStream_t);
// halo entries of a block-sharded case: gather into / scatter from an
// entry-major buffer of 5 values per entry (k_halo_pack, k_halo_unpack)
template <class T>
void launch_halo_pack(int n, const int* src, int NA, const T* P, T* buf, cudaStream_t);
template <class T>
void launch_halo_unpack(int n, const int* dst, int NA, const T* buf, T* b0, T* b1, cudaStream_t);

// end of an iteration (k_tail), then the sums of the iterations in its ring (k_tail_sums);
// P: current primitives, P2: the other buffer (halo ghosts are written to both)
template <class T>
void launch_tail(const ReduceArgs&, const T* Rc, const T* Rd, T* P, T* P2, cudaStream_t);
// n: pending iterations; advance: move *d_iter on by n
void launch_tail_sums(const ReduceArgs&, int n, bool advance, cudaStream_t);

// tail of iteration `it` of `iters` of a batch launch (current state in v.Pin), with the sums once the ring is full
template <class T>
void end_iteration(const FusedView<T>& v, const ReduceArgs& r, int it, int iters, cudaStream_t st) {
	ReduceArgs a = r;
	a.rec = const_cast<float*>(v.rec_in);
	a.rec2 = v.rec_out;
	launch_tail<T>(a, v.Rc, v.Rd, const_cast<T*>(v.Pin), v.Pout, st);
	const int in_ring = it % r.slots + 1;
	if (in_ring == r.slots || it == iters - 1) launch_tail_sums(r, in_ring, true, st);
}

// ---- fused stage kernels ----
template <class T>
void launch_recon(const FusedView<T>&, const Physics&, int grad, int lim, cudaStream_t);

// batch launchers: threads per block; per namespace: resident blocks per SM of
// the persistent kernel, its cooperative launch, and the tiled per-pass form.
// `batch` is built with the working precision's flags (FP64: no contraction,
// the same arithmetic as the single-case path); `batch_fast` holds FP64
// kernels built with FMA contraction (k64f.cu).
constexpr int kPersistThreads = 128;
namespace batch {
template <class T>
int persistent_blocks_per_sm(int grad, int lim, int scheme, bool order2);
template <class T>
cudaError_t launch_persistent(const FusedView<T>& v0, const FusedView<T>& v1, const Physics& ph, const PersistArgs& a,
                              int grad, int lim, int scheme, bool order2, int grid, cudaStream_t st);
// the same iterations as separate per-pass launches over the work list
template <class T>
cudaError_t launch_tiled_iterations(const FusedView<T>& v0, const FusedView<T>& v1, const Physics& ph,
                                    const PersistArgs& a, const ReduceArgs& r, int grad, int lim, int scheme, bool order2,
                                    cudaStream_t st);
}  // namespace batch
namespace batch_fast {
template <class T>
int persistent_blocks_per_sm(int grad, int lim, int scheme, bool order2);
template <class T>
cudaError_t launch_persistent(const FusedView<T>& v0, const FusedView<T>& v1, const Physics& ph, const PersistArgs& a,
                              int grad, int lim, int scheme, bool order2, int grid, cudaStream_t st);
// the same iterations as separate per-pass launches over the work list
template <class T>
cudaError_t launch_tiled_iterations(const FusedView<T>& v0, const FusedView<T>& v1, const Physics& ph,
                                    const PersistArgs& a, const ReduceArgs& r, int grad, int lim, int scheme, bool order2,
                                    cudaStream_t st);
}  // namespace batch_fast

// FP32 iterations in difference form (delta.cu): first-order AUSM, all-tetrahedron
// meshes, tiled per-pass form.  v0/v1 carry the base and difference arrays.
namespace delta {
cudaError_t launch_iterations(const FusedView<float>& v0, const FusedView<float>& v1, const Physics& ph,
                              const PersistArgs& a, const ReduceArgs& r, cudaStream_t st);
// new base state from W_b + dW (Wb: the FP64 base conserved state, updated in
// place), base ghosts, base residual in FP64; differences d0, d1 cleared
void launch_rebase(const FusedView<float>& v, const Physics& ph, double* Wb, const double* area64, int n_halo,
                   const int* halo_dst, const int* halo_src, float* d0, float* d1, cudaStream_t st);
}  // namespace delta

template <class T>
void launch_flux_update(const FusedView<T>&, const Physics&, int scheme, bool order1, bool first, double alpha,
                        double beta, int last, int carry, cudaStream_t);

}  // namespace e3d
