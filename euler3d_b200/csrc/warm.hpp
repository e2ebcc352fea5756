// Device helpers around the solver state that are not part of the residual
// path: per-cell features for the warm-start surrogate, writing a predicted
// conservative state into the solver, and widening an FP32 solver to FP64.
#pragma once
#include <cuda_runtime.h>

namespace e3d {

// Per-slot geometry of the fused path from the FP64 per-face arrays: unit
// normal and area (face orientation), area vector signed outward for the
// slot's owner, and the owner's r-vector.  sS may be null.
template <class T>
void launch_slot_geometry(int NS, const int* slot_face, const int* slot_mate, const double* S, const double* nhat,
                          const double* area, const double* rl, const double* rr, T* sgeo, T* sS, T* srv,
                          cudaStream_t st);
// n values in the working precision
template <class T>
void launch_convert(size_t n, const double* x, T* y, cudaStream_t st);

// FP64 copy of an FP32 packed primitive state, into both ping-pong buffers
// (only P0 when P1 is null).
// With W (the carried FP64 conservative state, [5][NR]) the real cells are
// recomputed from it exactly; ghost cells are widened from P32.
void launch_widen_state(int NA, int NR, const float* P32, const double* W, double gm1, double* P0, double* P1,
                        cudaStream_t st);

// Wall faces in clusters of at most WALL_CLUSTER consecutive ones of one case
// (cluster k: wall faces [first[k], first[k+1])): their centres and boxes.
constexpr int WALL_CLUSTER = 64;
void launch_wall_clusters(int n, const int* first, const int* wall_face, const double* fc, float4* centre, float4* box,
                          cudaStream_t st);

// Raw surrogate inputs of real cells [c0, c0 + n), [n][8] floats:
// x, y, z (centroid), distance to the nearest wall-face centre of the cell's
// case (clusters [case_cluster[cs], case_cluster[cs+1])), Mach, alpha
// (degrees), 0, 0.  Cells of a case without wall faces get distance 1.
void launch_cell_features(int c0, int n, int nb, const int* roff, const int* block_case, const float* centroid,
                          const int* case_cluster, const int* first, const float4* centre, const float4* box,
                          const float* case_mach_aoa, float* out, cudaStream_t st);

// Writes a conservative state (rho, rho u, rho v, rho w, rho E), [n][ld]
// floats, into real cells [c0, c0 + n): primitives of both ping-pong buffers (T) and,
// when W is non-null, the carried FP64 state.  A cell whose prediction is not
// physical (non-finite, rho or p below 1e-3 of freestream) keeps the
// freestream state of its case.  Returns nothing; the count of such cells is
// added to *n_fallback (device int).
template <class T>
void launch_apply_conservative(int c0, int n, int NR, int NA, int nb, const int* roff, const int* block_case,
                               const float* Wpred, int ld, const double* case_free, double gamma, T* P0, T* P1,
                               double* W, int* n_fallback, cudaStream_t st);

// Conservative state of every real cell from the packed primitives, [NR][8]
// floats (5 used).
template <class T>
void launch_prims_to_conservative(int NR, int NA, const T* P, double gamma, float* out, cudaStream_t st);

// One block's state array in file order and double precision: values
// [at, at + m) of [rows][n] into out.  Packed: five-variable arrays over all cells
// (ld = NA); rows: [row][real cell] (ld = NR); grad: [cell][GRAD_LD] as
// [var][cell][dim].  Real cell i of the block is device cell r0 + pos[i], ghost
// nr + j is g0 + j.
enum StateLayout : int { STATE_PACKED, STATE_ROWS, STATE_GRAD };
template <class T>
void launch_state_out(StateLayout layout, const T* dev, int ld, int n, int r0, int nr, int g0, const int* pos, size_t at,
                      size_t m, double* out, cudaStream_t st);

}  // namespace e3d
