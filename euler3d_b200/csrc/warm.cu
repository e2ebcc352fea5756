// Surrogate inputs, warm-start state writes and FP32 -> FP64 widening.
#include <cmath>

#include "views.hpp"
#include "warm.hpp"

namespace e3d {
namespace {

constexpr int TPB = 256;
inline int grid_for(long long n) { return (int)((n + TPB - 1) / TPB); }

__device__ __forceinline__ int block_of(const int* __restrict__ roff, int nb, int c) {
	int lo = 0, hi = nb;  // roff[lo] <= c < roff[hi]
	while (hi - lo > 1) {
		const int mid = (lo + hi) >> 1;
		if (roff[mid] <= c) lo = mid;
		else hi = mid;
	}
	return lo;
}

template <class T>
__global__ void k_slot_geometry(int NS, const int* __restrict__ slot_face, const int* __restrict__ slot_mate,
                                const double* __restrict__ S, const double* __restrict__ nhat,
                                const double* __restrict__ area, const double* __restrict__ rl,
                                const double* __restrict__ rr, T* __restrict__ sgeo, T* __restrict__ sS,
                                T* __restrict__ srv) {
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= NS) return;
	const int F = slot_face[k];
	const bool left = slot_mate[k] >= 0;
	for (int d = 0; d < 3; d++) {
		sgeo[4 * (size_t)k + d] = (T)nhat[3 * (size_t)F + d];
		if (sS) sS[3 * (size_t)k + d] = (T)(left ? S[3 * (size_t)F + d] : -S[3 * (size_t)F + d]);
		srv[3 * (size_t)k + d] = (T)(left ? rl[3 * (size_t)F + d] : rr[3 * (size_t)F + d]);
	}
	sgeo[4 * (size_t)k + 3] = (T)area[F];
}

__global__ void k_widen_state(int NA, int NR, const float* __restrict__ P32, const double* __restrict__ W, double gm1,
                              double* __restrict__ P0, double* __restrict__ P1) {
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= NA) return;
	double q[5];
	if (W && c < NR) {
		const double r = W[c];
		q[0] = r;
		q[1] = W[(size_t)NR + c] / r;
		q[2] = W[2 * (size_t)NR + c] / r;
		q[3] = W[3 * (size_t)NR + c] / r;
		q[4] = gm1 * (W[4 * (size_t)NR + c] - 0.5 * r * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]));
	} else {
		for (int v = 0; v < 4; v++) q[v] = (double)P32[4 * (size_t)c + v];
		q[4] = (double)P32[4 * (size_t)NA + c];
	}
	for (int v = 0; v < 4; v++) P0[4 * (size_t)c + v] = q[v];
	P0[4 * (size_t)NA + c] = q[4];
	if (P1) {
		for (int v = 0; v < 4; v++) P1[4 * (size_t)c + v] = q[v];
		P1[4 * (size_t)NA + c] = q[4];
	}
}

template <class T>
__global__ void k_convert(size_t n, const double* __restrict__ x, T* __restrict__ y) {
	const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (i < n) y[i] = (T)x[i];
}

template <class T>
__global__ void k_state_out(StateLayout layout, const T* __restrict__ dev, int ld, int n, int r0, int nr, int g0,
                            const int* __restrict__ pos, size_t at, size_t m, double* __restrict__ out) {
	const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (t >= m) return;
	size_t j = at + t;
	int d = 0;
	if (layout == STATE_GRAD) {  // [var][cell][dim]
		d = (int)(j % 3);
		j /= 3;
	}
	const int q = (int)(j / n), i = (int)(j % n);
	const int c = i < nr ? r0 + pos[i] : g0 + (i - nr);
	size_t src;
	if (layout == STATE_GRAD) src = GRAD_LD * (size_t)c + 3 * q + d;
	else if (layout == STATE_ROWS) src = q * (size_t)ld + c;
	else src = q < 4 ? 4 * (size_t)c + q : 4 * (size_t)ld + c;
	out[t] = (double)dev[src];
}

// Wall-face centres in FP32 and the box of each cluster of consecutive ones
// (cluster k: faces [first[k], first[k+1])); one block of WALL_CLUSTER threads per cluster.
__global__ void __launch_bounds__(WALL_CLUSTER) k_wall_clusters(const int* __restrict__ first,
                                                                const int* __restrict__ wall_face,
                                                                const double* __restrict__ fc, float4* __restrict__ centre,
                                                                float4* __restrict__ box) {
	const int b = first[blockIdx.x], e = first[blockIdx.x + 1], i = min(b + (int)threadIdx.x, e - 1);
	const int f = wall_face[i];
	float3 lo = make_float3((float)fc[3 * (size_t)f], (float)fc[3 * (size_t)f + 1], (float)fc[3 * (size_t)f + 2]), hi = lo;
	centre[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
	__shared__ float3 slo[WALL_CLUSTER / 32], shi[WALL_CLUSTER / 32];
	for (int h = 16; h > 0; h >>= 1) {
		lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, h));
		lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, h));
		lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, h));
		hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, h));
		hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, h));
		hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, h));
	}
	if ((threadIdx.x & 31) == 0) {
		slo[threadIdx.x >> 5] = lo;
		shi[threadIdx.x >> 5] = hi;
	}
	__syncthreads();
	if (threadIdx.x != 0) return;
	for (int w = 1; w < WALL_CLUSTER / 32; w++) {
		lo = make_float3(fminf(lo.x, slo[w].x), fminf(lo.y, slo[w].y), fminf(lo.z, slo[w].z));
		hi = make_float3(fmaxf(hi.x, shi[w].x), fmaxf(hi.y, shi[w].y), fmaxf(hi.z, shi[w].z));
	}
	box[2 * blockIdx.x] = make_float4(lo.x, lo.y, lo.z, 0.f);
	box[2 * blockIdx.x + 1] = make_float4(hi.x, hi.y, hi.z, 0.f);
}

__device__ __forceinline__ float wall_distance2(float x, float y, float z, const float4 w) {
	const float dx = x - w.x, dy = y - w.y, dz = z - w.z;
	return dx * dx + dy * dy + dz * dz;
}

// Features of real cells [c0, c0 + n).  The nearest wall face of every cell over
// all faces is cells x faces work with three FP64 conversions a pair (384k cells x
// 3,200 faces: 1,795 us).  A warp's 32 consecutive cells lie close together, so
// it takes the wall cluster nearest to their box first and then only those whose
// box comes within the largest distance found (the whole warm start of that mesh,
// network and buffers included, went from 4.8 to 1.1 ms).  The distances are the
// same FP32 expressions, and a box's is rounded the same way from components no
// larger than the face's, so the minimum is unchanged.
__global__ void __launch_bounds__(TPB) k_cell_features(int c0, int n, int nb, const int* __restrict__ roff,
                                                       const int* __restrict__ block_case, const float* __restrict__ cen,
                                                       const int* __restrict__ case_cluster,
                                                       const int* __restrict__ first, const float4* __restrict__ centre,
                                                       const float4* __restrict__ box, const float* __restrict__ case_ma,
                                                       float* __restrict__ out) {
	constexpr unsigned FULL = 0xffffffffu;
	const int t = blockIdx.x * TPB + threadIdx.x, lane = threadIdx.x & 31;
	if (t - lane >= n) return;
	const int c = c0 + min(t, n - 1);
	const int cs = block_case[block_of(roff, nb, c)];
	const float x = cen[3 * (size_t)c], y = cen[3 * (size_t)c + 1], z = cen[3 * (size_t)c + 2];
	float d2 = 3.4e38f;
	const int k0 = case_cluster[cs], k1 = case_cluster[cs + 1];
	const auto cluster = [&](int k) {
		const int e = first[k + 1];
#pragma unroll 8
		for (int i = first[k]; i < e; i++) d2 = fminf(d2, wall_distance2(x, y, z, __ldg(centre + i)));
	};
	if (__all_sync(FULL, cs == __shfl_sync(FULL, cs, 0))) {
		float3 lo = make_float3(x, y, z), hi = lo;
		for (int h = 16; h > 0; h >>= 1) {
			lo.x = fminf(lo.x, __shfl_xor_sync(FULL, lo.x, h));
			lo.y = fminf(lo.y, __shfl_xor_sync(FULL, lo.y, h));
			lo.z = fminf(lo.z, __shfl_xor_sync(FULL, lo.z, h));
			hi.x = fmaxf(hi.x, __shfl_xor_sync(FULL, hi.x, h));
			hi.y = fmaxf(hi.y, __shfl_xor_sync(FULL, hi.y, h));
			hi.z = fmaxf(hi.z, __shfl_xor_sync(FULL, hi.z, h));
		}
		const auto box_distance2 = [&](int k) {
			const float4 a = __ldg(box + 2 * k), b = __ldg(box + 2 * k + 1);
			const float dx = fmaxf(fmaxf(a.x - hi.x, lo.x - b.x), 0.f), dy = fmaxf(fmaxf(a.y - hi.y, lo.y - b.y), 0.f),
			            dz = fmaxf(fmaxf(a.z - hi.z, lo.z - b.z), 0.f);
			return dx * dx + dy * dy + dz * dz;
		};
		float best = 3.4e38f;
		int kb = k0;
		for (int k = k0 + lane; k < k1; k += 32) {
			const float d = box_distance2(k);
			if (d < best) {
				best = d;
				kb = k;
			}
		}
		for (int h = 16; h > 0; h >>= 1) {
			const float ob = __shfl_xor_sync(FULL, best, h);
			const int ok = __shfl_xor_sync(FULL, kb, h);
			if (ob < best || (ob == best && ok < kb)) {
				best = ob;
				kb = ok;
			}
		}
		if (k1 > k0) cluster(kb);
		for (int base = k0; base < k1; base += 32) {
			float far = d2;
			for (int h = 16; h > 0; h >>= 1) far = fmaxf(far, __shfl_xor_sync(FULL, far, h));
			const int k = base + lane;
			// the margin covers a differently contracted sum of squares
			unsigned todo = __ballot_sync(FULL, k < k1 && k != kb && box_distance2(min(k, k1 - 1)) * 0.99999f <= far);
			while (todo) {
				cluster(base + __ffs(todo) - 1);
				todo &= todo - 1;
			}
		}
	} else {
		for (int k = k0; k < k1; k++) cluster(k);
	}
	if (t >= n) return;
	float4* o = reinterpret_cast<float4*>(out + 8 * (size_t)t);
	o[0] = make_float4(x, y, z, k1 > k0 ? sqrtf(d2) : 1.f);
	o[1] = make_float4(case_ma[2 * cs], case_ma[2 * cs + 1], 0.f, 0.f);
}

template <class T>
__global__ void k_apply_conservative(int c0, int n, int NR, int NA, int nb, const int* __restrict__ roff,
                                     const int* __restrict__ block_case, const float* __restrict__ Wp, int ld,
                                     const double* __restrict__ case_free, double gamma, T* __restrict__ P0,
                                     T* __restrict__ P1, double* __restrict__ W, int* __restrict__ n_fallback) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x, c = c0 + t;
	if (t >= n) return;
	const int cs = block_case[block_of(roff, nb, c)];
	const double* f = case_free + 5 * (size_t)cs;
	const double gm1 = gamma - 1.0;
	double w[5];
	for (int v = 0; v < 5; v++) w[v] = (double)Wp[(size_t)ld * t + v];
	double q[5];
	q[0] = w[0];
	q[1] = w[1] / w[0];
	q[2] = w[2] / w[0];
	q[3] = w[3] / w[0];
	q[4] = gm1 * (w[4] - 0.5 * w[0] * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]));
	bool ok = true;
	for (int v = 0; v < 5; v++) ok = ok && isfinite(q[v]);
	ok = ok && q[0] > 1e-3 * f[0] && q[4] > 1e-3 * f[4];
	if (!ok) {
		for (int v = 0; v < 5; v++) q[v] = f[v];
		w[0] = f[0];
		w[1] = f[0] * f[1];
		w[2] = f[0] * f[2];
		w[3] = f[0] * f[3];
		w[4] = 0.5 * f[0] * (f[1] * f[1] + f[2] * f[2] + f[3] * f[3]) + 1. / gm1 * f[4];
		atomicAdd(n_fallback, 1);
	}
	for (int v = 0; v < 4; v++) {
		P0[4 * (size_t)c + v] = (T)q[v];
		P1[4 * (size_t)c + v] = (T)q[v];
	}
	P0[4 * (size_t)NA + c] = (T)q[4];
	P1[4 * (size_t)NA + c] = (T)q[4];
	if (W)
		for (int v = 0; v < 5; v++) W[(size_t)v * NR + c] = w[v];
}

template <class T>
__global__ void k_prims_to_conservative(int NR, int NA, const T* __restrict__ P, double gamma, float* __restrict__ out) {
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= NR) return;
	const double r = (double)P[4 * (size_t)c], u = (double)P[4 * (size_t)c + 1], v = (double)P[4 * (size_t)c + 2],
	             w = (double)P[4 * (size_t)c + 3], p = (double)P[4 * (size_t)NA + c];
	float* o = out + 8 * (size_t)c;
	o[0] = (float)r;
	o[1] = (float)(r * u);
	o[2] = (float)(r * v);
	o[3] = (float)(r * w);
	o[4] = (float)(0.5 * r * (u * u + v * v + w * w) + p / (gamma - 1.0));
	o[5] = o[6] = o[7] = 0.f;
}

}  // namespace

template <class T>
void launch_prims_to_conservative(int NR, int NA, const T* P, double gamma, float* out, cudaStream_t st) {
	if (NR > 0) k_prims_to_conservative<T><<<grid_for(NR), TPB, 0, st>>>(NR, NA, P, gamma, out);
}
template void launch_prims_to_conservative<float>(int, int, const float*, double, float*, cudaStream_t);
template void launch_prims_to_conservative<double>(int, int, const double*, double, float*, cudaStream_t);

template <class T>
void launch_slot_geometry(int NS, const int* slot_face, const int* slot_mate, const double* S, const double* nhat,
                          const double* area, const double* rl, const double* rr, T* sgeo, T* sS, T* srv,
                          cudaStream_t st) {
	if (NS > 0)
		k_slot_geometry<T><<<grid_for(NS), TPB, 0, st>>>(NS, slot_face, slot_mate, S, nhat, area, rl, rr, sgeo, sS, srv);
}
template void launch_slot_geometry<float>(int, const int*, const int*, const double*, const double*, const double*,
                                          const double*, const double*, float*, float*, float*, cudaStream_t);
template void launch_slot_geometry<double>(int, const int*, const int*, const double*, const double*, const double*,
                                           const double*, const double*, double*, double*, double*, cudaStream_t);

template <class T>
void launch_convert(size_t n, const double* x, T* y, cudaStream_t st) {
	if (n > 0) k_convert<T><<<grid_for((long long)n), TPB, 0, st>>>(n, x, y);
}
template void launch_convert<float>(size_t, const double*, float*, cudaStream_t);
template void launch_convert<double>(size_t, const double*, double*, cudaStream_t);

void launch_widen_state(int NA, int NR, const float* P32, const double* W, double gm1, double* P0, double* P1,
                        cudaStream_t st) {
	if (NA > 0) k_widen_state<<<grid_for(NA), TPB, 0, st>>>(NA, NR, P32, W, gm1, P0, P1);
}

template <class T>
void launch_state_out(StateLayout layout, const T* dev, int ld, int n, int r0, int nr, int g0, const int* pos, size_t at,
                      size_t m, double* out, cudaStream_t st) {
	if (m > 0) k_state_out<T><<<grid_for((long long)m), TPB, 0, st>>>(layout, dev, ld, n, r0, nr, g0, pos, at, m, out);
}
template void launch_state_out<float>(StateLayout, const float*, int, int, int, int, int, const int*, size_t, size_t,
                                      double*, cudaStream_t);
template void launch_state_out<double>(StateLayout, const double*, int, int, int, int, int, const int*, size_t, size_t,
                                       double*, cudaStream_t);

void launch_wall_clusters(int n, const int* first, const int* wall_face, const double* fc, float4* centre, float4* box,
                          cudaStream_t st) {
	if (n > 0) k_wall_clusters<<<n, WALL_CLUSTER, 0, st>>>(first, wall_face, fc, centre, box);
}

void launch_cell_features(int c0, int n, int nb, const int* roff, const int* block_case, const float* centroid,
                          const int* case_cluster, const int* first, const float4* centre, const float4* box,
                          const float* case_mach_aoa, float* out, cudaStream_t st) {
	if (n > 0)
		k_cell_features<<<grid_for(n), TPB, 0, st>>>(c0, n, nb, roff, block_case, centroid, case_cluster, first, centre,
		                                             box, case_mach_aoa, out);
}

template <class T>
void launch_apply_conservative(int c0, int n, int NR, int NA, int nb, const int* roff, const int* block_case,
                               const float* Wpred, int ld, const double* case_free, double gamma, T* P0, T* P1,
                               double* W, int* n_fallback, cudaStream_t st) {
	if (n > 0)
		k_apply_conservative<T><<<grid_for(n), TPB, 0, st>>>(c0, n, NR, NA, nb, roff, block_case, Wpred, ld, case_free,
		                                                     gamma, P0, P1, W, n_fallback);
}

template void launch_apply_conservative<float>(int, int, int, int, int, const int*, const int*, const float*, int,
                                               const double*, double, float*, float*, double*, int*, cudaStream_t);
template void launch_apply_conservative<double>(int, int, int, int, int, const int*, const int*, const float*, int,
                                                const double*, double, double*, double*, double*, int*, cudaStream_t);

}  // namespace e3d
