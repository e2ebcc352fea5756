// Warm-start surrogate: training and inference kernels (see surrogate.hpp).
//
// A training step is three launches.  k_mlp takes tiles of 64 rows through the
// whole network and back: the weights stay in shared memory, the activations
// of a tile never leave the SM between layers, GELU'(z) stays in registers from
// the forward to the backward pass (one erf for both), and only the BF16
// activations and gradients that the weight gradients need are written out.
// k_wgrad forms dW = g^T a over slices of rows, k_update adds up the partials in
// a fixed order and applies Adam.  Inference is k_mlp's forward half alone.
// All GEMMs are mma.sync m16n8k16 with BF16 operands and FP32 accumulators, k
// ascending.  Per row the step is 0.2 MFLOP of GEMM but 384 erf and 384 exp, so
// the CUDA cores, not the tensor cores, bound it.  No floating-point atomics
// anywhere: every sum is a fixed-order loop or tree, so a training run is
// reproducible bit for bit.
// B200: a 16,384-row step took 334 us as 25 launches with every activation in
// global memory; 65 us in this form.  A 384k-row forward pass: 940 us in 5
// launches; 335 us in one.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>

#include "surrogate.hpp"
#include "warm.hpp"

namespace e3d {
namespace {

using S = SurrogateShape;
constexpr int H = S::H;

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ uint16_t f2bf(float x) {
	const __nv_bfloat16 b = __float2bfloat16_rn(x);
	return *reinterpret_cast<const uint16_t*>(&b);
}
__device__ __forceinline__ float bf2f(uint16_t u) { return __uint_as_float(((uint32_t)u) << 16); }

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x) {
	// splitmix64 finaliser
	x += 0x9E3779B97F4A7C15ull;
	x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
	x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
	return x ^ (x >> 31);
}

// freestream conservative state of (Mach, alpha in degrees), the reference's
// nondimensionalisation (rho = 1, p = 1, |u| = M sqrt(gamma))
__device__ __forceinline__ void wfree(float mach, float aoa_deg, float gamma, float w[5]) {
	const float a = aoa_deg * 0.017453292519943295f;
	const float q = mach * sqrtf(gamma);
	const float u = q * cosf(a), v = q * sinf(a);
	w[0] = 1.f;
	w[1] = u;
	w[2] = v;
	w[3] = 0.f;
	w[4] = 0.5f * (u * u + v * v) + 1.f / (gamma - 1.f);
}

// ------------------------------------------------------------------ tensor-core fragments
__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
	asm volatile(
	    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
	    "{%0,%1,%2,%3};\n"
	    : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
	    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool TRANS>
__device__ __forceinline__ void ldsm4(uint32_t r[4], const uint16_t* p) {
	const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
	if (TRANS)
		asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
		             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
		             : "r"(a));
	else
		asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
		             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
		             : "r"(a));
}

constexpr int TR = 64;         // rows of a tile
constexpr int MLP_TPB = 512;   // 16 warps: 4 (16 rows) x 4 (32 columns) of a 64 x 128 layer
constexpr int LDH = H + 8;     // shared rows of 128 BF16 values, padded: 8 rows of a matrix hit 32 banks
constexpr int LDX = S::IN + 8;
// per-block sums of the output layer and the biases: W4, b4, b3, b2, b1
constexpr int PA_B4 = S::OUT * H, PA_B3 = PA_B4 + S::OUT, PA_B2 = PA_B3 + H, PA_B1 = PA_B2 + H, PA_N = PA_B1 + H;

struct MlpShared {
	uint16_t w1[H][LDX], w2[H][LDH], w3[H][LDH];
	uint16_t x[TR][LDX], a1[TR][LDH], a2[TR][LDH], a3[TR][LDH], g2[TR][LDH];
	float w4[H][12];  // W4 transposed: the 5 outputs' weights of one input, padded against bank conflicts
	float b1[H], b2[H], b3[H], b4[S::OUT], norm[S::N_NORM];
	float t[TR][S::OUT], d4[TR][S::OUT];  // targets (inference: freestream state), dL/dy
	float red[PA_N];
	float loss[MLP_TPB / 32];
};

// One warp's 16 x 32 part of (64 x K) * (K x 128); B row-major [n][k] or, BT, [k][n].
template <int K, int LDA, int LDB, bool BT>
__device__ __forceinline__ void warp_gemm(float acc[4][4], const uint16_t (*A)[LDA], const uint16_t (*B)[LDB], int m0,
                                          int n0) {
	const int lane = threadIdx.x & 31, r = lane & 7, id = lane >> 3;
#pragma unroll
	for (int j = 0; j < 4; j++)
#pragma unroll
		for (int i = 0; i < 4; i++) acc[j][i] = 0.f;
#pragma unroll
	for (int k0 = 0; k0 < K; k0 += 16) {
		uint32_t a[4], b[2][4];
		ldsm4<false>(a, &A[m0 + r + (id & 1) * 8][k0 + (id >> 1) * 8]);
#pragma unroll
		for (int h = 0; h < 2; h++)
			if (BT) ldsm4<true>(b[h], &B[k0 + r + (id & 1) * 8][n0 + 16 * h + (id >> 1) * 8]);
			else ldsm4<false>(b[h], &B[n0 + 16 * h + r + (id >> 1) * 8][k0 + (id & 1) * 8]);
#pragma unroll
		for (int j = 0; j < 4; j++) mma_bf16(acc[j], a, b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
	}
}
__device__ __forceinline__ uint32_t pack2(float a, float b) { return (uint32_t)f2bf(a) | ((uint32_t)f2bf(b) << 16); }

// z = acc + bias, h = GELU(z) to shared memory; gd = GELU'(z) kept by the thread
template <bool TRAIN>
__device__ __forceinline__ void gelu_layer(const float acc[4][4], const float* bias, uint16_t (*out)[LDH], float gd[4][4],
                                           int m0, int n0) {
	const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
	for (int j = 0; j < 4; j++) {
		const int n = n0 + 8 * j + 2 * t;
		float h[4];
#pragma unroll
		for (int i = 0; i < 4; i++) {
			const float z = acc[j][i] + bias[n + (i & 1)];
			const float e = 1.f + erff(z * 0.70710678118654752f);
			h[i] = 0.5f * z * e;
			if (TRAIN) gd[j][i] = 0.5f * e + z * 0.39894228040143268f * expf(-0.5f * z * z);
		}
		*reinterpret_cast<uint32_t*>(&out[m0 + g][n]) = pack2(h[0], h[1]);
		*reinterpret_cast<uint32_t*>(&out[m0 + g + 8][n]) = pack2(h[2], h[3]);
	}
}
__device__ __forceinline__ void store_grad(const float acc[4][4], const float gd[4][4], uint16_t (*out)[LDH], int m0, int n0) {
	const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
	for (int j = 0; j < 4; j++) {
		const int n = n0 + 8 * j + 2 * t;
		*reinterpret_cast<uint32_t*>(&out[m0 + g][n]) = pack2(acc[j][0] * gd[j][0], acc[j][1] * gd[j][1]);
		*reinterpret_cast<uint32_t*>(&out[m0 + g + 8][n]) = pack2(acc[j][2] * gd[j][2], acc[j][3] * gd[j][3]);
	}
}
// a tile's first `rows` rows of 128 values to global memory
__device__ __forceinline__ void copy_rows(const uint16_t (*src)[LDH], uint16_t* __restrict__ dst, int rows) {
	for (int i = threadIdx.x; i < TR * (H / 8); i += MLP_TPB) {
		const int r = i / (H / 8), c = i % (H / 8);
		if (r < rows) reinterpret_cast<uint4*>(dst)[(size_t)r * (H / 8) + c] = *reinterpret_cast<const uint4*>(&src[r][8 * c]);
	}
}
// 5 values of a 16-byte-aligned row
__device__ __forceinline__ void load5(const float* p, float o[S::N_OUT]) {
	const float4 v = *reinterpret_cast<const float4*>(p);
	o[0] = v.x;
	o[1] = v.y;
	o[2] = v.z;
	o[3] = v.w;
	o[4] = p[4];
}
__device__ __forceinline__ float colsum16(const uint16_t (*g)[LDH], int r0, int j) {
	float s = 0.f;
#pragma unroll
	for (int r = 0; r < 16; r++) s += bf2f(g[r0 + r][j]);
	return s;
}

struct MlpArgs {
	int n;                // rows
	const float* feat;    // [.][8] raw features
	const float* state;   // [.][8] conservative states (training)
	long long n_store;    // > 0: row i is a hashed draw from n_store samples; 0: row i
	uint64_t seed;
	long long step;
	const float* norm;
	float gamma;
	const float* master;  // FP32 parameters (biases)
	const uint16_t* wb;   // BF16 weights
	uint16_t *x, *a1, *a2, *g1, *g2, *g3;  // training: operands of the weight gradients
	float* part;          // training: [block][PA_N]
	float* lossp;         // training: [block] squared-error sums
	float* out;           // inference: [n][8] conservative states
};

// The network forward, and with TRAIN back to the first layer, over tiles of TR
// rows.  One block per SM (163 KB of shared memory), weights loaded once.
template <bool TRAIN>
__global__ void __launch_bounds__(MLP_TPB, 1) k_mlp(MlpArgs p) {
	extern __shared__ __align__(16) unsigned char dyn[];
	MlpShared& s = *reinterpret_cast<MlpShared*>(dyn);
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * 32;
	for (int i = t; i < H * S::IN / 8; i += MLP_TPB)
		*reinterpret_cast<uint4*>(&s.w1[i / 2][8 * (i % 2)]) = reinterpret_cast<const uint4*>(p.wb + S::OFF_W1)[i];
	for (int i = t; i < H * H / 8; i += MLP_TPB) {
		*reinterpret_cast<uint4*>(&s.w2[i / 16][8 * (i % 16)]) = reinterpret_cast<const uint4*>(p.wb + S::OFF_W2)[i];
		*reinterpret_cast<uint4*>(&s.w3[i / 16][8 * (i % 16)]) = reinterpret_cast<const uint4*>(p.wb + S::OFF_W3)[i];
	}
	for (int i = t; i < S::N_OUT * H; i += MLP_TPB) s.w4[i % H][i / H] = bf2f(p.wb[S::OFF_W4 + i]);
	if (t < H) {
		s.b1[t] = p.master[S::OFF_B1 + t];
		s.b2[t] = p.master[S::OFF_B2 + t];
		s.b3[t] = p.master[S::OFF_B3 + t];
	}
	if (t < S::OUT) s.b4[t] = p.master[S::OFF_B4 + t];
	if (t < S::N_NORM) s.norm[t] = p.norm[t];
	__syncthreads();
	const int row8 = t >> 3, j8 = t & 7;          // 8 lanes per row: inputs, outputs
	const int col = t & (H - 1), r16 = (t >> 7) * 16;  // 16 rows of one column: sums over rows
	float se = 0.f, w4sum[S::N_OUT] = {0.f, 0.f, 0.f, 0.f, 0.f}, b4sum = 0.f, b3sum = 0.f, b2sum = 0.f, b1sum = 0.f;
	const int n_tiles = (p.n + TR - 1) / TR;
	for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
		const int i0 = tile * TR, rows = min(TR, p.n - i0);
		const bool valid = row8 < rows;
		{  // standardised features, scaled targets
			const long long i = i0 + (valid ? row8 : 0);
			long long src = i;
			if (p.n_store > 0)
				src = (long long)(mix64(p.seed ^ mix64((uint64_t)p.step * 0x100000001B3ull + (uint64_t)i)) %
				                  (uint64_t)p.n_store);
			const float f = p.feat[(size_t)src * 8 + j8];
			const uint16_t xv = valid && j8 < S::N_IN ? f2bf((f - s.norm[j8]) / s.norm[8 + j8]) : (uint16_t)0;
			s.x[row8][j8] = xv;
			s.x[row8][8 + j8] = 0;
			const float mach = __shfl_sync(0xffffffffu, f, (lane & 24) + 4), aoa = __shfl_sync(0xffffffffu, f, (lane & 24) + 5);
			float wf[5];
			wfree(mach, aoa, p.gamma, wf);
			const float w = j8 == 0 ? wf[0] : j8 == 1 ? wf[1] : j8 == 2 ? wf[2] : j8 == 3 ? wf[3] : wf[4];
			if (TRAIN) {
				if (valid) {
					p.x[(size_t)i * S::IN + j8] = xv;
					p.x[(size_t)i * S::IN + 8 + j8] = 0;
				}
				s.t[row8][j8] = j8 < S::N_OUT ? (p.state[(size_t)src * 8 + j8] - w) / s.norm[16 + j8] : 0.f;
			} else {
				s.t[row8][j8] = w;
			}
		}
		__syncthreads();
		float acc[4][4], gd1[4][4], gd2[4][4], gd3[4][4];
		warp_gemm<S::IN, LDX, LDX, false>(acc, s.x, s.w1, m0, n0);
		gelu_layer<TRAIN>(acc, s.b1, s.a1, gd1, m0, n0);
		__syncthreads();
		warp_gemm<H, LDH, LDH, false>(acc, s.a1, s.w2, m0, n0);
		gelu_layer<TRAIN>(acc, s.b2, s.a2, gd2, m0, n0);
		__syncthreads();
		warp_gemm<H, LDH, LDH, false>(acc, s.a2, s.w3, m0, n0);
		gelu_layer<TRAIN>(acc, s.b3, s.a3, gd3, m0, n0);
		__syncthreads();
		{  // output layer: each of a row's 8 lanes takes 16 of the 128 inputs
			float y[S::N_OUT] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
			for (int k = 0; k < 16; k += 2) {
				const int j = 16 * j8 + ((k + 2 * j8) & 15);  // staggered: the lanes' reads spread over the banks
				const uint32_t v = *reinterpret_cast<const uint32_t*>(&s.a3[row8][j]);
				const float x0 = bf2f((uint16_t)(v & 0xFFFFu)), x1 = bf2f((uint16_t)(v >> 16));
				float wa[S::N_OUT], wc[S::N_OUT];
				load5(s.w4[j], wa);
				load5(s.w4[j + 1], wc);
#pragma unroll
				for (int q = 0; q < S::N_OUT; q++) y[q] += wa[q] * x0 + wc[q] * x1;
			}
#pragma unroll
			for (int q = 0; q < S::N_OUT; q++)
				for (int h = 4; h > 0; h >>= 1) y[q] += __shfl_xor_sync(0xffffffffu, y[q], h);
			const float yq = (j8 == 0 ? y[0] : j8 == 1 ? y[1] : j8 == 2 ? y[2] : j8 == 3 ? y[3] : y[4]) + s.b4[j8];
			if (TRAIN) {
				const float e = valid && j8 < S::N_OUT ? yq - s.t[row8][j8] : 0.f;
				s.d4[row8][j8] = 2.f * e / (float)(p.n * S::N_OUT);
				se += e * e;
			} else if (valid) {
				p.out[(size_t)(i0 + row8) * 8 + j8] = j8 < S::N_OUT ? s.t[row8][j8] + s.norm[16 + j8] * yq : 0.f;
			}
		}
		if (!TRAIN) continue;  // the next tile's first write to a3 is behind three barriers
		__syncthreads();
#pragma unroll
		for (int r = 0; r < 16; r++) {
			const float a = bf2f(s.a3[r16 + r][col]);
			float d[S::N_OUT];
			load5(s.d4[r16 + r], d);
#pragma unroll
			for (int q = 0; q < S::N_OUT; q++) w4sum[q] += d[q] * a;
			if (col < S::OUT) b4sum += s.d4[r16 + r][col];
		}
		{  // g3 = GELU'(z3) * (d4 W4)
			const int g = lane >> 2, c2 = 2 * (lane & 3);
			float da[S::N_OUT], db[S::N_OUT];
			load5(s.d4[m0 + g], da);
			load5(s.d4[m0 + g + 8], db);
#pragma unroll
			for (int j = 0; j < 4; j++)
#pragma unroll
				for (int i = 0; i < 2; i++) {
					float w[S::N_OUT], u = 0.f, v = 0.f;
					load5(s.w4[n0 + 8 * j + c2 + i], w);
#pragma unroll
					for (int q = 0; q < S::N_OUT; q++) {
						u += da[q] * w[q];
						v += db[q] * w[q];
					}
					acc[j][i] = u;
					acc[j][2 + i] = v;
				}
		}
		__syncthreads();
		store_grad(acc, gd3, s.a3, m0, n0);  // a3 is read no more: it holds g3 from here
		__syncthreads();
		copy_rows(s.a3, p.g3 + (size_t)i0 * H, rows);
		b3sum += colsum16(s.a3, r16, col);
		warp_gemm<H, LDH, LDH, true>(acc, s.a3, s.w3, m0, n0);
		store_grad(acc, gd2, s.g2, m0, n0);
		__syncthreads();
		copy_rows(s.g2, p.g2 + (size_t)i0 * H, rows);
		b2sum += colsum16(s.g2, r16, col);
		warp_gemm<H, LDH, LDH, true>(acc, s.g2, s.w2, m0, n0);
		store_grad(acc, gd1, s.a3, m0, n0);  // g1
		__syncthreads();
		copy_rows(s.a3, p.g1 + (size_t)i0 * H, rows);
		copy_rows(s.a1, p.a1 + (size_t)i0 * H, rows);
		copy_rows(s.a2, p.a2 + (size_t)i0 * H, rows);
		b1sum += colsum16(s.a3, r16, col);
	}
	if constexpr (TRAIN) {
		// the four row groups' sums in order, then the block's squared error
		for (int grp = 0; grp < 4; grp++) {
			__syncthreads();
			if ((t >> 7) == grp) {
				const bool z = grp == 0;
#pragma unroll
				for (int q = 0; q < S::OUT; q++) {
					float& r = s.red[q * H + col];
					const float v = q < S::N_OUT ? w4sum[q < S::N_OUT ? q : 0] : 0.f;
					r = z ? v : r + v;
				}
				if (col < S::OUT) s.red[PA_B4 + col] = z ? b4sum : s.red[PA_B4 + col] + b4sum;
				s.red[PA_B3 + col] = z ? b3sum : s.red[PA_B3 + col] + b3sum;
				s.red[PA_B2 + col] = z ? b2sum : s.red[PA_B2 + col] + b2sum;
				s.red[PA_B1 + col] = z ? b1sum : s.red[PA_B1 + col] + b1sum;
			}
		}
		for (int h = 16; h > 0; h >>= 1) se += __shfl_down_sync(0xffffffffu, se, h);
		if (lane == 0) s.loss[warp] = se;
		__syncthreads();
		for (int i = t; i < PA_N; i += MLP_TPB) p.part[(size_t)blockIdx.x * PA_N + i] = s.red[i];
		if (t == 0) {
			float l = 0.f;
			for (int w = 0; w < MLP_TPB / 32; w++) l += s.loss[w];
			p.lossp[blockIdx.x] = l;
		}
	}
}

// Weight gradients dW[o][i] = sum_rows g[row][o] a[row][i] of one slice of rows
// (blockIdx.x) of layer 3, 2 or 1 (blockIdx.y), tiles of 64 rows in two buffers:
// the next one loads while this one is multiplied.  part: [slice][2 H H + H IN].
constexpr int WG_TPB = 256;
constexpr int WG_N = 2 * H * H + H * S::IN;
struct WgShared {
	uint16_t g[2][TR][LDH], a[2][TR][LDH];
};
__device__ __forceinline__ void cp16(void* dst, const void* src, bool on) {
	const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
	const int n = on ? 16 : 0;
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n));
}
// rows [r0, r0 + TR) of a [.][COLS] matrix, rows at or past `end` as zeros
template <int COLS>
__device__ __forceinline__ void load_tile(uint16_t (*dst)[LDH], const uint16_t* __restrict__ src, int r0, int end) {
	for (int i = threadIdx.x; i < TR * (COLS / 8); i += WG_TPB) {
		const int r = i / (COLS / 8), c = i % (COLS / 8);
		const bool on = r0 + r < end;
		cp16(&dst[r][8 * c], src + (size_t)(on ? r0 + r : 0) * COLS + 8 * c, on);
	}
}

template <int IN>  // columns of a: 128, or 16 for the first layer
__device__ __forceinline__ void wgrad_slice(WgShared& s, const uint16_t* __restrict__ g, const uint16_t* __restrict__ a,
                                            int r0, int r1, float* __restrict__ out) {
	// 8 warps: 2 (64 outputs) x 4 (32 inputs); 8 (16 outputs) x 1 (16 inputs)
	constexpr int MT = IN == H ? 4 : 1, NT = IN == H ? 4 : 2;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane & 7, id = lane >> 3;
	const int m0 = IN == H ? (warp & 1) * 64 : warp * 16, n0 = IN == H ? (warp >> 1) * 32 : 0;
	float acc[MT][NT][4];
#pragma unroll
	for (int i = 0; i < MT; i++)
#pragma unroll
		for (int j = 0; j < NT; j++)
#pragma unroll
			for (int k = 0; k < 4; k++) acc[i][j][k] = 0.f;
	load_tile<H>(s.g[0], g, r0, r1);
	load_tile<IN>(s.a[0], a, r0, r1);
	asm volatile("cp.async.commit_group;\n");
	int buf = 0;
	for (int b = r0; b < r1; b += TR, buf ^= 1) {
		if (b + TR < r1) {
			load_tile<H>(s.g[buf ^ 1], g, b + TR, r1);
			load_tile<IN>(s.a[buf ^ 1], a, b + TR, r1);
		}
		asm volatile("cp.async.commit_group;\n");
		asm volatile("cp.async.wait_group 1;\n");
		__syncthreads();
#pragma unroll
		for (int k0 = 0; k0 < TR; k0 += 16) {
			uint32_t fa[MT][4], fb[NT / 2][4];
#pragma unroll
			for (int i = 0; i < MT; i++)
				ldsm4<true>(fa[i], &s.g[buf][k0 + r + (id >> 1) * 8][m0 + 16 * i + (id & 1) * 8]);
#pragma unroll
			for (int j = 0; j < NT / 2; j++)
				ldsm4<true>(fb[j], &s.a[buf][k0 + r + (id & 1) * 8][n0 + 16 * j + (id >> 1) * 8]);
#pragma unroll
			for (int i = 0; i < MT; i++)
#pragma unroll
				for (int j = 0; j < NT; j++) mma_bf16(acc[i][j], fa[i], fb[j >> 1][2 * (j & 1)], fb[j >> 1][2 * (j & 1) + 1]);
		}
		__syncthreads();
	}
	const int gg = lane >> 2, t2 = 2 * (lane & 3);
#pragma unroll
	for (int i = 0; i < MT; i++)
#pragma unroll
		for (int j = 0; j < NT; j++) {
			const int o = m0 + 16 * i + gg, n = n0 + 8 * j + t2;
			*reinterpret_cast<float2*>(&out[(size_t)o * IN + n]) = make_float2(acc[i][j][0], acc[i][j][1]);
			*reinterpret_cast<float2*>(&out[(size_t)(o + 8) * IN + n]) = make_float2(acc[i][j][2], acc[i][j][3]);
		}
}

__global__ void __launch_bounds__(WG_TPB) k_wgrad(MlpArgs p, int rows, float* __restrict__ part) {
	extern __shared__ __align__(16) unsigned char dyn[];
	WgShared& s = *reinterpret_cast<WgShared*>(dyn);
	const int r0 = blockIdx.x * rows, r1 = min(p.n, r0 + rows);
	float* out = part + (size_t)blockIdx.x * WG_N;
	if (blockIdx.y == 0) wgrad_slice<H>(s, p.g3, p.a2, r0, r1, out);
	else if (blockIdx.y == 1) wgrad_slice<H>(s, p.g2, p.a1, r0, r1, out + H * H);
	else wgrad_slice<S::IN>(s, p.g1, p.x, r0, r1, out + 2 * H * H);
}

struct AdamArgs {
	float *w, *m, *v;
	uint16_t* wb;
	float lr, b1, b2, eps, c1, c2;
};
// Gradient of parameter i: its partials in four interleaved runs, each in block or
// slice order, then the runs' sums in order; Adam with UPDATE.  A thread per run:
// one thread per parameter, 64 dependent adds over loads 145 KB apart, took 17 us.
// The last block adds up the loss.
constexpr int UP_RUNS = 4, UP_PARAMS = 256 / UP_RUNS;
template <bool UPDATE>
__global__ void __launch_bounds__(256) k_update(int blocks_a, const float* __restrict__ pa, int slices,
                                                const float* __restrict__ pw, float* __restrict__ grad, AdamArgs a,
                                                const float* __restrict__ lossp, int n, double* __restrict__ loss) {
	if (blockIdx.x == gridDim.x - 1) {
		if (threadIdx.x == 0) {
			double l = 0.0;
#pragma unroll 8
			for (int i = 0; i < blocks_a; i++) l += (double)lossp[i];
			*loss = l / ((double)n * S::N_OUT);
		}
		return;
	}
	const int lp = threadIdx.x % UP_PARAMS, run = threadIdx.x / UP_PARAMS;
	const int i = min(blockIdx.x * UP_PARAMS + lp, S::N_PARAM - 1);
	const float* src;
	int count, stride;
	const auto from_slices = [&](int off) {
		src = pw + off;
		count = slices;
		stride = WG_N;
	};
	const auto from_blocks = [&](int off) {
		src = pa + off;
		count = blocks_a;
		stride = PA_N;
	};
	if (i < S::OFF_B1) from_slices(2 * H * H + i);
	else if (i < S::OFF_W2) from_blocks(PA_B1 + i - S::OFF_B1);
	else if (i < S::OFF_B2) from_slices(H * H + i - S::OFF_W2);
	else if (i < S::OFF_W3) from_blocks(PA_B2 + i - S::OFF_B2);
	else if (i < S::OFF_B3) from_slices(i - S::OFF_W3);
	else if (i < S::OFF_W4) from_blocks(PA_B3 + i - S::OFF_B3);
	else from_blocks(i - S::OFF_W4);  // W4, b4
	float g = 0.f;
#pragma unroll 8
	for (int k = run; k < count; k += UP_RUNS) g += src[(size_t)k * stride];
	__shared__ float sums[UP_RUNS][UP_PARAMS];
	sums[run][lp] = g;
	__syncthreads();
	if (run != 0 || blockIdx.x * UP_PARAMS + lp >= S::N_PARAM) return;
	for (int r = 1; r < UP_RUNS; r++) g += sums[r][lp];
	if (!UPDATE) {
		grad[i] = g;
		return;
	}
	const float mi = a.b1 * a.m[i] + (1.f - a.b1) * g;
	const float vi = a.b2 * a.v[i] + (1.f - a.b2) * g * g;
	a.m[i] = mi;
	a.v[i] = vi;
	const float wi = a.w[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
	a.w[i] = wi;
	a.wb[i] = f2bf(wi);
}

__global__ void k_to_bf16(int n, const float* __restrict__ w, uint16_t* __restrict__ wb) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) wb[i] = f2bf(w[i]);
}

// feature statistics: per-block sums of x and x^2 (double) over STAT_ROWS rows,
// 16 threads a row group (0..5 features, 8..12 target deviations), fixed order
constexpr int STAT_ROWS = 2048;
__global__ void __launch_bounds__(256) k_feat_stats(long long n, const float* __restrict__ feat,
                                                    const float* __restrict__ state, float gamma,
                                                    double* __restrict__ part) {
	const int j = threadIdx.x & 15, grp = threadIdx.x >> 4;
	const long long r0 = (long long)blockIdx.x * STAT_ROWS, r1 = min(n, r0 + STAT_ROWS);
	double s = 0.0, s2 = 0.0;
	for (long long b = r0 + grp; b < r1; b += 16) {
		double x = 0.0;
		if (j < 8) {
			if (j < S::N_IN) x = (double)feat[b * 8 + j];
		} else if (j - 8 < S::N_OUT) {
			float wf[5];
			wfree(feat[b * 8 + 4], feat[b * 8 + 5], gamma, wf);
			const int q = j - 8;
			x = (double)state[b * 8 + q] - (double)(q == 0 ? wf[0] : q == 1 ? wf[1] : q == 2 ? wf[2] : q == 3 ? wf[3] : wf[4]);
		}
		s += x;
		s2 += x * x;
	}
	__shared__ double red[16][32];
	red[grp][j] = s;
	red[grp][16 + j] = s2;
	__syncthreads();
	if (threadIdx.x < 32) {
		double v = 0.0;
		for (int k = 0; k < 16; k++) v += red[k][threadIdx.x];
		part[(size_t)blockIdx.x * 32 + threadIdx.x] = v;
	}
}

inline void ok(cudaError_t e, const char* what) {
	if (e != cudaSuccess) throw Error(E3D_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
inline int blocks(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// ------------------------------------------------------------------ Surrogate
Surrogate::Surrogate(int device, uint64_t seed, double gamma) : device_(device), gamma_(gamma), seed_(seed) {
	if (device_ >= 0) ok(cudaSetDevice(device_), "cudaSetDevice");
	ok(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking), "cudaStreamCreate");
	ok(cudaEventCreateWithFlags(&params_ready_, cudaEventDisableTiming), "event");
	int dev = 0;
	ok(cudaGetDevice(&dev), "cudaGetDevice");
	ok(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev), "SM count");
	const auto smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
	ok(cudaFuncSetAttribute(k_mlp<true>, smem, (int)sizeof(MlpShared)), "shared memory");
	ok(cudaFuncSetAttribute(k_mlp<false>, smem, (int)sizeof(MlpShared)), "shared memory");
	ok(cudaFuncSetAttribute(k_wgrad, smem, (int)sizeof(WgShared)), "shared memory");
	// Kaiming-uniform initialisation from a seeded generator (host), padding entries zero
	std::vector<float> w(S::N_PARAM, 0.f);
	std::mt19937_64 rng(seed);
	auto fill = [&](int off, int rows, int cols, int used_rows, int used_cols) {
		const float bound = std::sqrt(6.f / (float)used_cols);
		std::uniform_real_distribution<float> u(-bound, bound);
		for (int r = 0; r < rows; r++)
			for (int c = 0; c < cols; c++) w[off + r * cols + c] = (r < used_rows && c < used_cols) ? u(rng) : 0.f;
	};
	fill(S::OFF_W1, H, S::IN, H, S::N_IN);
	fill(S::OFF_W2, H, H, H, H);
	fill(S::OFF_W3, H, H, H, H);
	fill(S::OFF_W4, S::OUT, H, S::N_OUT, H);
	for (int i = 0; i < S::OUT * H; i++) w[S::OFF_W4 + i] *= 0.1f;  // small initial output: start near freestream
	master_.upload(w);
	std::vector<float> z(S::N_PARAM, 0.f);
	m1_.upload(z);
	m2_.upload(z);
	grad_.upload(z);
	wb_.alloc(S::N_PARAM);
	norm_h_.assign(S::N_NORM, 0.f);
	for (int j = 0; j < 8; j++) norm_h_[8 + j] = 1.f;
	for (int q = 0; q < 8; q++) norm_h_[16 + q] = 1.f;
	norm_.upload(norm_h_);
	loss_d_.alloc(1);
	upload_params();
}

Surrogate::~Surrogate() {
	if (params_ready_) cudaEventDestroy(params_ready_);
	if (st_) cudaStreamDestroy(st_);
}

void Surrogate::upload_params() {
	k_to_bf16<<<blocks(S::N_PARAM, 256), 256, 0, st_>>>(S::N_PARAM, master_.p, wb_.p);
	ok(cudaGetLastError(), "to_bf16");
}

void Surrogate::add_samples_device(const float* feat, const float* state, long long n, cudaStream_t producer) {
	if (n <= 0) return;
	if (producer) ok(cudaStreamSynchronize(producer), "sync");
	if (n_samples_ + n > cap_samples_) {
		const long long cap = std::max(n_samples_ + n, cap_samples_ * 3 / 2 + 1024);
		DevBuf<float> f2, s2;
		f2.alloc((size_t)cap * 8);
		s2.alloc((size_t)cap * 8);
		if (n_samples_) {
			ok(cudaMemcpyAsync(f2.p, feat_.p, (size_t)n_samples_ * 8 * sizeof(float), cudaMemcpyDeviceToDevice, st_),
			   "grow");
			ok(cudaMemcpyAsync(s2.p, state_.p, (size_t)n_samples_ * 8 * sizeof(float), cudaMemcpyDeviceToDevice, st_),
			   "grow");
		}
		ok(cudaStreamSynchronize(st_), "sync");
		std::swap(feat_.p, f2.p);
		std::swap(feat_.n, f2.n);
		std::swap(state_.p, s2.p);
		std::swap(state_.n, s2.n);
		cap_samples_ = cap;
	}
	ok(cudaMemcpyAsync(feat_.p + (size_t)n_samples_ * 8, feat, (size_t)n * 8 * sizeof(float), cudaMemcpyDeviceToDevice,
	                   st_),
	   "samples");
	ok(cudaMemcpyAsync(state_.p + (size_t)n_samples_ * 8, state, (size_t)n * 8 * sizeof(float),
	                   cudaMemcpyDeviceToDevice, st_),
	   "samples");
	ok(cudaStreamSynchronize(st_), "sync");
	n_samples_ += n;
}

void Surrogate::add_samples_host(const float* feat6, const float* state5, long long n) {
	if (n <= 0) return;
	std::vector<float> f((size_t)n * 8, 0.f), s((size_t)n * 8, 0.f);
	for (long long i = 0; i < n; i++) {
		for (int j = 0; j < 6; j++) f[i * 8 + j] = feat6[i * 6 + j];
		for (int q = 0; q < 5; q++) s[i * 8 + q] = state5[i * 5 + q];
	}
	DevBuf<float> fd, sd;
	fd.upload(f);
	sd.upload(s);
	add_samples_device(fd.p, sd.p, n, nullptr);
}

void Surrogate::add_solution(Engine& e) {
	const int nr = e.n_real_total();
	DevBuf<float> f, s;
	f.alloc((size_t)nr * 8);
	s.alloc((size_t)nr * 8);
	e.cell_features(f.p);
	e.conservative_rows(s.p);
	add_samples_device(f.p, s.p, nr, e.stream());
}

void Surrogate::clear_samples() {
	n_samples_ = 0;
	normalised_ = false;
}

void Surrogate::fit_normalisation() {
	if (n_samples_ < 2) throw Error(E3D_ERR_STATE, "surrogate: no training samples");
	const int nb = (int)((n_samples_ + STAT_ROWS - 1) / STAT_ROWS);
	DevBuf<double> part;
	part.alloc((size_t)nb * 32);
	k_feat_stats<<<nb, 256, 0, st_>>>(n_samples_, feat_.p, state_.p, (float)gamma_, part.p);
	ok(cudaGetLastError(), "feat_stats");
	std::vector<double> h((size_t)nb * 32);
	ok(cudaMemcpyAsync(h.data(), part.p, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st_), "stats");
	ok(cudaStreamSynchronize(st_), "sync");
	double s[16] = {0}, s2[16] = {0};
	for (int b = 0; b < nb; b++)
		for (int j = 0; j < 16; j++) {
			s[j] += h[(size_t)b * 32 + j];
			s2[j] += h[(size_t)b * 32 + 16 + j];
		}
	const double n = (double)n_samples_;
	for (int j = 0; j < 8; j++) {
		const double mu = s[j] / n, var = std::max(0.0, s2[j] / n - mu * mu);
		norm_h_[j] = (float)mu;
		norm_h_[8 + j] = (float)std::max(std::sqrt(var), 1e-6);
		const double t2 = s2[8 + j] / n;  // target scale: RMS deviation from freestream
		norm_h_[16 + j] = (float)std::max(std::sqrt(t2), 1e-6);
	}
	norm_.upload(norm_h_);
	normalised_ = true;
}

void Surrogate::ensure_work(int n) {
	x_.reserve((size_t)n * S::IN);
	for (auto* b : {&a1_, &a2_, &g1_, &g2_, &g3_}) b->reserve((size_t)n * H);
	lossp_.reserve((size_t)sms_);
	part_.reserve((size_t)sms_ * PA_N);
	wpart_.reserve((size_t)kSlices * WG_N);
}

// Loss and gradient partials of n rows (part_, wpart_, lossp_); `grad`: gradient
// into grad_ and the loss into *loss, else one Adam step as well.
void Surrogate::step_rows(int n, const float* feat, const float* state, long long n_store, const AdamStep* adam,
                          double* loss) {
	MlpArgs p{};
	p.n = n;
	p.feat = feat;
	p.state = state;
	p.n_store = n_store;
	p.seed = seed_;
	p.step = step_;
	p.norm = norm_.p;
	p.gamma = (float)gamma_;
	p.master = master_.p;
	p.wb = wb_.p;
	p.x = x_.p;
	p.a1 = a1_.p;
	p.a2 = a2_.p;
	p.g1 = g1_.p;
	p.g2 = g2_.p;
	p.g3 = g3_.p;
	p.part = part_.p;
	p.lossp = lossp_.p;
	const int grid = std::min(sms_, blocks(n, TR));
	k_mlp<true><<<grid, MLP_TPB, sizeof(MlpShared), st_>>>(p);
	// slices of whole tiles, at most kSlices of them
	const int rows = blocks(blocks(n, TR), kSlices) * TR, slices = blocks(n, rows);
	k_wgrad<<<dim3(slices, 3), WG_TPB, sizeof(WgShared), st_>>>(p, rows, wpart_.p);
	AdamArgs a{};
	if (adam)
		a = AdamArgs{master_.p, m1_.p, m2_.p, wb_.p, adam->lr, adam->b1, adam->b2, adam->eps, adam->c1, adam->c2};
	const int ug = blocks(S::N_PARAM, UP_PARAMS) + 1;
	if (adam) k_update<true><<<ug, 256, 0, st_>>>(grid, part_.p, slices, wpart_.p, grad_.p, a, lossp_.p, n, loss);
	else k_update<false><<<ug, 256, 0, st_>>>(grid, part_.p, slices, wpart_.p, grad_.p, a, lossp_.p, n, loss);
	ok(cudaGetLastError(), "training step");
}

double Surrogate::train(int steps, int batch, double lr, std::vector<float>* loss_per_step) {
	if (steps <= 0) return 0.0;
	if (batch < 64 || batch > (1 << 20)) throw Error(E3D_ERR_ARG, "surrogate: batch must be in [64, 2^20]");
	if (n_samples_ < 2) throw Error(E3D_ERR_STATE, "surrogate: no training samples");
	if (!normalised_) fit_normalisation();
	ensure_work(batch);
	hist_.reserve((size_t)steps);
	AdamStep ad{0.f, 0.9f, 0.999f, 1e-8f, 1.f, 1.f};
	for (int s = 0; s < steps; s++) {
		// cosine decay to 5% of lr over this call
		const double frac = steps > 1 ? (double)s / (steps - 1) : 1.0;
		ad.lr = (float)(lr * (0.05 + 0.95 * 0.5 * (1.0 + std::cos(3.14159265358979 * frac))));
		ad.c1 = 1.f - std::pow(ad.b1, (float)(step_ + 1));
		ad.c2 = 1.f - std::pow(ad.b2, (float)(step_ + 1));
		step_rows(batch, feat_.p, state_.p, n_samples_, &ad, hist_.p + s);
		step_++;
	}
	ok(cudaGetLastError(), "train");
	std::vector<double> h(steps);
	ok(cudaMemcpyAsync(h.data(), hist_.p, steps * sizeof(double), cudaMemcpyDeviceToHost, st_), "loss history");
	ok(cudaStreamSynchronize(st_), "sync");
	if (loss_per_step) loss_per_step->assign(h.begin(), h.end());
	const int k = std::min(steps, 50);
	double m = 0.0;
	for (int i = steps - k; i < steps; i++) m += h[i];
	return m / k;
}

double Surrogate::gradient(const float* feat6, const float* state5, int n, std::vector<float>& grad) {
	if (n < 1 || n > (1 << 20)) throw Error(E3D_ERR_ARG, "surrogate: sample count out of range");
	std::vector<float> f((size_t)n * 8, 0.f), s((size_t)n * 8, 0.f);
	for (int i = 0; i < n; i++) {
		for (int j = 0; j < 6; j++) f[(size_t)i * 8 + j] = feat6[(size_t)i * 6 + j];
		for (int q = 0; q < 5; q++) s[(size_t)i * 8 + q] = state5[(size_t)i * 5 + q];
	}
	DevBuf<float> fd, sd;
	fd.upload(f);
	sd.upload(s);
	ensure_work(n);
	step_rows(n, fd.p, sd.p, 0, nullptr, loss_d_.p);
	double loss = 0.0;
	ok(cudaMemcpyAsync(&loss, loss_d_.p, sizeof(double), cudaMemcpyDeviceToHost, st_), "loss");
	grad.resize(S::N_PARAM);
	ok(cudaMemcpyAsync(grad.data(), grad_.p, S::N_PARAM * sizeof(float), cudaMemcpyDeviceToHost, st_), "grad");
	ok(cudaStreamSynchronize(st_), "sync");
	return loss;
}

// Rows queued on `st`, behind the parameters' last update.
void Surrogate::predict_device(const float* feat, long long n, float* state, cudaStream_t st) {
	if (st != st_) {
		ok(cudaEventRecord(params_ready_, st_), "event");
		ok(cudaStreamWaitEvent(st, params_ready_, 0), "event");
	}
	const long long chunk = 1 << 30;  // rows of a launch fit an int
	for (long long b0 = 0; b0 < n; b0 += chunk) {
		MlpArgs p{};
		p.n = (int)std::min<long long>(chunk, n - b0);
		p.feat = feat + b0 * 8;
		p.norm = norm_.p;
		p.gamma = (float)gamma_;
		p.master = master_.p;
		p.wb = wb_.p;
		p.out = state + b0 * 8;
		k_mlp<false><<<std::min(sms_, blocks(p.n, TR)), MLP_TPB, sizeof(MlpShared), st>>>(p);
	}
	ok(cudaGetLastError(), "predict");
}

void Surrogate::predict_host(const float* feat6, long long n, float* state5) {
	if (n <= 0) return;
	std::vector<float> f((size_t)n * 8, 0.f);
	for (long long i = 0; i < n; i++)
		for (int j = 0; j < 6; j++) f[i * 8 + j] = feat6[i * 6 + j];
	DevBuf<float> fd, sd;
	fd.upload(f);
	sd.alloc((size_t)n * 8);
	predict_device(fd.p, n, sd.p, st_);
	std::vector<float> s((size_t)n * 8);
	ok(cudaMemcpyAsync(s.data(), sd.p, s.size() * sizeof(float), cudaMemcpyDeviceToHost, st_), "predict");
	ok(cudaStreamSynchronize(st_), "sync");
	for (long long i = 0; i < n; i++)
		for (int q = 0; q < 5; q++) state5[i * 5 + q] = s[i * 8 + q];
}

// Features, network and state write of kWarmRows cells at a time, on the engine's
// stream: the two buffers stay (64 MB at most) instead of 64 bytes a cell
// allocated and freed on every call.
int Surrogate::warm_start(Engine& e) {
	const int nr = (int)e.n_real_total(), m = std::min(nr, kWarmRows);
	warm_f_.reserve((size_t)m * 8);
	warm_w_.reserve((size_t)m * 8);
	e.clear_fallbacks();
	for (int c0 = 0; c0 < nr; c0 += m) {
		const int n = std::min(m, nr - c0);
		e.cell_features(warm_f_.p, c0, n);
		predict_device(warm_f_.p, n, warm_w_.p, e.stream());
		e.apply_conservative(warm_w_.p, 8, c0, n);
	}
	return e.fallbacks();
}

void Surrogate::get_params(float* out) const {
	ok(cudaMemcpy(out, master_.p, S::N_PARAM * sizeof(float), cudaMemcpyDeviceToHost), "params");
}
void Surrogate::set_params(const float* in) {
	ok(cudaMemcpyAsync(master_.p, in, S::N_PARAM * sizeof(float), cudaMemcpyHostToDevice, st_), "params");
	upload_params();
	ok(cudaStreamSynchronize(st_), "sync");
}
void Surrogate::get_normalisation(float* out) const { std::memcpy(out, norm_h_.data(), S::N_NORM * sizeof(float)); }
void Surrogate::set_normalisation(const float* in) {
	norm_h_.assign(in, in + S::N_NORM);
	norm_.upload(norm_h_);
	normalised_ = true;
}

}  // namespace e3d
