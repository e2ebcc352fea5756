// Device-array views shared by the host engine and the kernel translation units.
//
// Cell numbering on the device: all real cells of all blocks first (block after
// block, each in its file order), then all ghost cells (block after block, in
// marker order).  Faces are numbered block after block in the reference's
// creation order.  A "slot" is one (cell, face) incidence; a cell's slots are
// contiguous and follow ascending face id, which is the reference's summation
// order for every per-cell accumulation.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace e3d {

enum GradKind : int { GRAD_GREEN_GAUSS = 0, GRAD_LEAST_SQUARES = 1 };
enum LimKind : int { LIM_BARTH_JESPERSEN = 0, LIM_VENKATAKRISHNAN = 1 };
enum FluxKind : int { FLUX_ROE = 0, FLUX_AUSM = 1 };
enum GhostKind : int { GK_NONE = 0, GK_WALL = 1, GK_FARFIELD = 2, GK_SYMMETRY = 3 };

struct Physics {
	double gamma, gm1, gr;  // gamma, gamma-1, gamma/(gamma-1)
	double cfl;
	double omega, k3;       // BJ shift, Venkatakrishnan K^3
	double free[5];         // freestream rho, u, v, w, p
};

// Mesh topology and FP64 geometry (granular drop-in kernels).
struct GeoView {
	int NR, NG, NA, NF, NS;
	int tet4;              // 1 when every real cell has exactly 4 slots
	const int* slot_ptr;   // NA+1
	const int* slot_face;  // NS
	const int* slot_nbr;   // NS
	const int* slot_mate;  // NS as in FusedView
	const double* sgeo;    // 4*NS n, |S| of the slot's face (face orientation)
	const double* srv;     // 3*NS r-vector of the slot's owner
	const double* S;       // 3*NF area vector, left -> right
	const double* nhat;    // 3*NF S/|S| as the reference normalises it
	const double* area;    // NF
	const double* vol;     // NA
	const double* lsw;     // 3*NS (real-cell slots)
	const signed char* gkind;  // NG boundary-condition kind of each ghost
	const signed char* grefl;  // NG 1: gradient reflected, 0: gradient zero
};

constexpr int GRAD_LD = 16;  // stored gradient values per cell: [var][dim], 15 used

// FP64 state arrays in the reference's meaning (drop-in path).
struct StateView {
	double* prim;  // 5*NA packed: [cell] x (rho,u,v,w), then [cell] p
	double* rc;    // 5*NR
	double* rd;    // 5*NR
	double* w0;    // 5*NR
	double* grad;  // 16*NA [cell][var][dim], padded
	double* lim;   // 5*NA packed like prim
	double* dt;    // NR
	double* srad;  // NR
};

// Fused-path view in working precision T.
template <class T>
struct FusedView {
	int NR, NG, NA, NS;
	int tet4;               // 1 when every real cell has exactly 4 slots (slot = 4c+k)
	const int* slot_ptr;    // NA+1
	const int* slot_nbr;    // NS
	const int* slot_mate;   // NS  >=0: owner is the face's left cell, mate slot index; <0: ~mate, owner is right
	const T* sgeo;          // 4*NS  nx, ny, nz, |S| of the face (face orientation)
	const T* sS;            // 3*NS  area vector signed outward for the owner (Green-Gauss)
	const T* srv;           // 3*NS  r-vector of the owner at the face
	const T* lsw;           // 3*NS  least-squares weights (real slots)
	const T* vol;           // NA
	const signed char* gkind;
	const signed char* grefl;
	const T* Pin;           // 5*NA
	T* Pout;                // 5*NA
	T* FS;                  // 5*NS reconstructed face states [var][slot]
	T* Rc;                  // 5*NR
	T* Rd;                  // 5*NR
	double* W0;             // 5*NR
	T* dt;                  // NR
	const double* case_free;  // 5 per case, or null: every ghost uses Physics::free
	const int* gcase;         // NG case index of each ghost (with case_free)
	// difference form (delta.cu; null otherwise): Pin/Pout hold differences from
	// the base primitives Pb (FP32 copy of Pb64), dW the carried conserved
	// differences from the FP64 base W_b, Rb the FP64-evaluated base residual
	const float* Pb;          // 5*NA
	const double* Pb64;       // 5*NA
	const float* rec_base;    // 8*NA per-cell flux quantities of the base state
	const float* rec_in;      // 8*NA and their differences, of Pin
	float* rec_out;           // 8*NA of Pout
	float* dW;                // 5*NR
	float* Rb;                // 5*NR
	const int* slot_face;     // NS  (FP64 face normals of boundary slots)
	const double* nhat64;     // 3*NF
};

// End of an iteration (k_tail, k_tail_sums): norm chunks, wall terms and halo
// of one iteration into ring slot *pend, then the per-block sums of all pending
// iterations into hist[(*d_iter + i)*stride + b*10 + (0..4 norms, 5..9 forces)].
constexpr int TAIL_TPB = 256;     // threads per block of k_tail
constexpr int TAIL_CHUNK = 1024;  // cells per norm chunk: 48 blocks at 48k cells, 3,000 at 3.07M
constexpr int TAIL_SLOTS = 32;    // iterations the ring holds at most
// Iterations the ring of a solver holds.  One iteration's slot is 40 bytes a norm chunk
// and wall face; 64 meshes with 230k wall faces would keep 0.3 GB in 32 of them.  The
// ring stays within 8 bytes a cell or 16 MB, whichever is more: fewer iterations'
// chains then run side by side, but so many faces come in many blocks, whose chains do
// too (B200, 100 iterations of 64 meshes with 578 wall faces each, 10 slots / 32: FP32
// 45.8 / 45.8 ms, FP64 120.2 / 119.8; 1,339 / 1,373 MB).
inline int tail_slots(size_t n_chunks, size_t n_wall, size_t n_cells, size_t hist_capacity) {
	const size_t slot = 5 * sizeof(double) * (n_chunks + n_wall), room = n_cells > (2u << 20) ? 8 * n_cells : 16u << 20;
	size_t n = slot ? room / slot : TAIL_SLOTS;
	n = n < hist_capacity ? n : hist_capacity;
	return n < 1 ? 1 : n < TAIL_SLOTS ? (int)n : TAIL_SLOTS;
}
struct ReduceArgs {
	int NR, NA, nblocks;
	int n_chunks;          // norm chunks of all blocks, one block after the other
	const int4* chunk;     // first cell, end, block
	const int* chunk_off;  // nblocks+1 chunk offsets
	int slots;             // iterations the ring holds
	double* partial;       // slots*5*n_chunks
	const int* wall_off;   // nblocks+1
	const int* wall_face;
	int n_wall;
	double* wall_terms;    // slots*5*n_wall
	const int* face_lr;
	const double* S;
	const double* fc;
	double denom;          // 0.5*gamma*M*M*cmac
	const double* wall_denom;  // per wall face (cases of a batch differ in Mach), or null
	int n_halo;
	const int* halo_dst;
	const int* halo_src;
	double* hist;
	int stride;
	int* d_iter;
	int* d_bad;
	int* pend;             // iterations in the ring
	unsigned* ticket;      // blocks of the running launch that are done
	const int* block_work; // batches: nblocks+1 work-item offsets, a block without items is frozen; else null
	const double* Pb64;    // difference form: FP64 base primitives (wall pressures are base + difference), else null
	float *rec, *rec2;     // difference form: 8 values a cell of either buffer, copied with the halo; else null
};

// One launch of the persistent batch kernel: several outer iterations over the
// work list (tiles of real cells of the active cases).
struct PersistArgs {
	int n_work;            // work items (tiles)
	const int4* work;      // x: first cell, y: end cell, z: block, w: unused
	const int* block_work; // nblocks+1: work items of block b are [block_work[b], block_work[b+1])
	int nblocks;
	int stages;
	double alpha[5], beta[5];
	int carry;
	int iters;             // outer iterations in this launch
	int start_parity;      // 0: state in P0 (view v0 reads it), 1: state in P1
	// reductions
	double* wpart;         // n_work*5 per-tile sums of (Rc-Rd)^2
	const int* wall_off;
	const int* wall_face;
	int n_wall;
	double* wall_terms;
	const double* wall_denom;
	double denom;
	const int* face_lr;
	const double* S;
	const double* fc;
	double* hist;          // [iteration][block][10]
	int stride;
	int* d_iter;           // iteration counter (advanced by `iters` at the end)
	int hist_capacity;
	int* d_bad;
	// halo
	int n_halo;
	const int* halo_dst;
	const int* halo_src;
};

}  // namespace e3d
