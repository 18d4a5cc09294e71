// mlp.cu -- the gain network of the learned form and its training.
//
// Network: 65 -> 256 -> 256 -> 64, GELU (erf form) after the two hidden
// layers, sigmoid on the output.  Weights and activations are BF16 with FP32
// accumulation on the tensor cores (mma.sync m16n8k16); FP32 master weights,
// biases, pre-activations, gradients and AdamW moments.
//
// Layouts (all row-major):
//   public parameter blob (host, float): W1[65][256] b1[256] W2[256][256]
//     b2[256] W3[256][64] b3[64]  -- W[in][out]
//   device master (float): the same with W1 padded to [80][256] (rows 65..79
//     stay zero: their inputs are zero, so their gradients are zero)
//   device working copy (bf16): the matrices in the order of the MMA's B
//     fragments, 16 bytes a lane (frag_at)
//   features: bf16 [rows][80] (65 used), gains: float [rows][64]
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bm4dof.h"
#include "internal.hpp"

namespace bm4dof {

namespace {

using bf16 = __nv_bfloat16;

constexpr int kIn = 65, kInP = 80, kHid = 256, kOut = 64;

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
	asm volatile(
	    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
	    "{%0,%1,%2,%3};\n"
	    : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float gelu(float x)
{
	return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
}

__device__ __forceinline__ float gelu_grad(float x)
{
	// d/dx x*Phi(x) = Phi(x) + x*phi(x)
	const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
	const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
	return cdf + x * pdf;
}

__device__ __forceinline__ void ldmatrix(uint32_t (&r)[4], const bf16 *p)
{
	const uint32_t s = (uint32_t)__cvta_generic_to_shared(p);
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
	             : "r"(s)
	             : "memory");
}

// float features [n][65] -> bf16 [n][80] (zero padded)
__global__ void pack_features_kernel(const float *__restrict__ f, long long n, bf16 *__restrict__ X)
{
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n * kInP;
	     i += (long long)gridDim.x * blockDim.x) {
		const long long r = i / kInP;
		const int c = (int)(i % kInP);
		X[i] = __float2bfloat16_rn(c < kIn ? f[r * kIn + c] : 0.f);
	}
}

// ---------------------------------------------------------------------------
// Weights as B operands of mma.m16n8k16, in fragment order: for a tile of 8
// outputs and a pair of k-steps, lane (g = lane / 4, t = lane % 4) holds
// k = 2t, 2t+1, 2t+8, 2t+9 of output g of both steps in 16 bytes.
// ---------------------------------------------------------------------------
constexpr int kInF = 96;                 // inputs padded to whole pairs of k-steps
constexpr int kFragF1 = 0, kFragF2 = kFragF1 + kInF * kHid, kFragF3 = kFragF2 + kHid * kHid,
              kFragB3 = kFragF3 + kHid * kOut, kFragB2 = kFragB3 + kOut * kHid, kFragSize = kFragB2 + kHid * kHid;
static_assert(kFragB3 == kMlpWtSize, "the forward operands");

// Place of B(k, n) in a fragment-ordered operand of K rows.
__host__ __device__ __forceinline__ int frag_at(int k, int n, int K)
{
	const int pair = k >> 5, ks = k >> 4 & 1, kk = k & 15;
	const int t = (kk & 7) >> 1, half = kk >> 3, lane = (n & 7) * 4 + t;
	return (((n >> 3) * (K >> 5) + pair) * 32 + lane) * 8 + ks * 4 + half * 2 + (kk & 1);
}

// acc[mi][j] = A (MI x 16 rows, K columns, shared, pitch ldA, 16-byte rows) . B tiles tile0 + j
template <int K, int MI, int NT>
__device__ __forceinline__ void rows_mma(const bf16 *A, int ldA, const bf16 *__restrict__ B, int tile0,
                                         float (&acc)[MI][NT][4])
{
	const int lane = threadIdx.x & 31;
	const bf16 *ap = A + ((lane & 7) + (lane & 8)) * ldA + (lane >> 4) * 8;
#pragma unroll
	for (int mi = 0; mi < MI; mi++)
#pragma unroll
		for (int j = 0; j < NT; j++) acc[mi][j][0] = acc[mi][j][1] = acc[mi][j][2] = acc[mi][j][3] = 0.f;
#pragma unroll 4
	for (int p = 0; p < K / 32; p++) {
		uint4 b[NT];
#pragma unroll
		for (int j = 0; j < NT; j++)
			b[j] = __ldg(reinterpret_cast<const uint4 *>(B) + ((size_t)(tile0 + j) * (K / 32) + p) * 32 + lane);
#pragma unroll
		for (int ks = 0; ks < 2; ks++)
#pragma unroll
			for (int mi = 0; mi < MI; mi++) {
				uint32_t a[4];
				ldmatrix(a, ap + mi * 16 * ldA + p * 32 + ks * 16);
#pragma unroll
				for (int j = 0; j < NT; j++) mma_bf16(acc[mi][j], a, ks ? b[j].z : b[j].x, ks ? b[j].w : b[j].y);
			}
	}
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b)
{
	__nv_bfloat162 v = __floats2bfloat162_rn(a, b);
	return *reinterpret_cast<uint32_t *>(&v);
}

// Forward pass over n feature rows, 64 rows a CTA.  A warp takes 32 (the last
// layer: 8) columns of all 64 rows, so that a fragment of the weights, 16 bytes
// a lane out of L2, serves eight products; the activations come from shared
// memory by ldmatrix.
//
// What bounds it: the tensor cores' rate through mma.sync and erff.  1.36 million
// rows: 5.1 -> 1.45 ms (16 rows a warp, two 4-byte loads of weights a product
// before).
constexpr int kFwdRows = 64, kFwdThreads = 256;

__global__ void __launch_bounds__(kFwdThreads, 2)
mlp_forward_kernel(const bf16 *__restrict__ X, long long n, MlpWeights w, float *__restrict__ out)
{
	constexpr int P = kHid + 8;          // row pitch without bank conflicts
	extern __shared__ __align__(16) unsigned char msm[];
	bf16 *A = reinterpret_cast<bf16 *>(msm), *B = A + kFwdRows * P;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
	auto hidden = [&](float (&p)[4][4][4], const float *bias, bf16 *to) {
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const int c = warp * 32 + j * 8 + 2 * t;
			const float b0 = __ldg(bias + c), b1 = __ldg(bias + c + 1);
#pragma unroll
			for (int mi = 0; mi < 4; mi++)
#pragma unroll
				for (int h = 0; h < 2; h++)
					*reinterpret_cast<uint32_t *>(to + (mi * 16 + g + 8 * h) * P + c) =
					    pack_bf16(gelu(p[mi][j][2 * h] + b0), gelu(p[mi][j][2 * h + 1] + b1));
		}
	};
	for (long long r0 = (long long)blockIdx.x * kFwdRows; r0 < n; r0 += (long long)gridDim.x * kFwdRows) {
		// 64 rows of 96 bf16 (80 in memory, then zeros) in 16-byte pieces
		for (int i = tid; i < kFwdRows * (kInF / 8); i += kFwdThreads) {
			const int r = i / (kInF / 8), c8 = i % (kInF / 8);
			uint4 v = make_uint4(0, 0, 0, 0);
			if (r0 + r < n && c8 < kInP / 8) v = __ldg(reinterpret_cast<const uint4 *>(X + (r0 + r) * kInP) + c8);
			*reinterpret_cast<uint4 *>(B + r * P + c8 * 8) = v;
		}
		__syncthreads();
		float p[4][4][4];
		rows_mma<kInF, 4, 4>(B, P, w.frag + kFragF1, warp * 4, p);
		hidden(p, w.b1, A);
		__syncthreads();
		rows_mma<kHid, 4, 4>(A, P, w.frag + kFragF2, warp * 4, p);
		hidden(p, w.b2, B);
		__syncthreads();
		float o[4][1][4];
		rows_mma<kHid, 4, 1>(B, P, w.frag + kFragF3, warp, o);
		const int c = warp * 8 + 2 * t;
		const float b0 = __ldg(w.b3 + c), b1 = __ldg(w.b3 + c + 1);
#pragma unroll
		for (int mi = 0; mi < 4; mi++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const long long row = r0 + mi * 16 + g + 8 * h;
				if (row < n)
					*reinterpret_cast<float2 *>(out + row * kOut + c) =
					    make_float2(1.f / (1.f + expf(-(o[mi][0][2 * h] + b0))), 1.f / (1.f + expf(-(o[mi][0][2 * h + 1] + b1))));
			}
		__syncthreads();
	}
}

constexpr size_t kForwardSmem = sizeof(bf16) * 2 * kFwdRows * (kHid + 8);

// ---------------------------------------------------------------------------
// Training.  One step is three launches:
//   train_rows_kernel   forward and backward of 32 rows per CTA, all layers; the
//                       pre-activations stay in registers (a warp's columns are
//                       the same in the forward and the backward pass of a
//                       layer); leaves the BF16 activations and gradients of
//                       every layer, and per-CTA sums for the biases and the loss
//   weight_grad_kernel  the three products activations^T . gradients, 64 x 64
//                       tiles, the rows split over CTAs
//   update_kernel       the splits summed in a fixed order (no atomics: a step is
//                       reproducible), AdamW, and the weights' BF16 copies
// Separate kernels per layer with 16 CTAs walking all 8192 rows took 5.6 ms for
// a step of 8192 rows; these take 32 + 12 + 10 us.  What bounds them: the latency
// of one wave of CTAs (4.8 GFLOP are 3 us of the tensor cores' time), the
// weights' trip through L2 to every CTA, and erff.
//
// ---------------------------------------------------------------------------
constexpr int kTrainRows = 32, kTrainThreads = 512;   // rows and threads per CTA of train_rows_kernel
constexpr int kGradTile = 64, kMaxSplits = 16, kSplitRows = 512;
constexpr int kBiases = kHid + kHid + kOut;

// Sum of a column's values over the lanes that hold its rows (g = 0 .. 7).
__device__ __forceinline__ float column_sum(float v)
{
	v += __shfl_xor_sync(0xffffffffu, v, 4);
	v += __shfl_xor_sync(0xffffffffu, v, 8);
	v += __shfl_xor_sync(0xffffffffu, v, 16);
	return v;
}

struct TrainRows {
	const float *feat, *target;
	long long n;
	const bf16 *frag;
	const float *master;
	bf16 *X, *H1, *H2, *D1, *D2, *D3;   // [rows][96], [rows][256] x 2, then the gradients
	float *bias_part, *loss_part;       // [CTAs][kBiases], [CTAs]
};

__global__ void __launch_bounds__(kTrainThreads, 2)
train_rows_kernel(TrainRows a)
{
	constexpr int XP = kInF + 8, HP = kHid + 8, OP = kOut + 8;   // pitches without bank conflicts
	__shared__ __align__(16) bf16 Xs[kTrainRows * XP], Hs[kTrainRows * HP], Gs[kTrainRows * HP], Ds[kTrainRows * OP];
	__shared__ float s_loss[kTrainThreads / 32], s_db3[2][kOut];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
	const long long r0 = (long long)blockIdx.x * kTrainRows;
	for (int i = tid; i < kTrainRows * kInF; i += kTrainThreads) {
		const int r = i / kInF, c = i % kInF;
		const bf16 v = __float2bfloat16_rn(c < kIn && r0 + r < a.n ? a.feat[(r0 + r) * kIn + c] : 0.f);
		Xs[r * XP + c] = v;
		a.X[(r0 + r) * kInF + c] = v;
	}
	__syncthreads();
	const int c0 = warp * 16;            // this warp's columns of the hidden layers
	float p1[2][2][4], p2[2][2][4];
	// hidden layer: pre-activations to p, activations to shared memory and H
	auto hidden = [&](float (&p)[2][2][4], const float *bias, bf16 *out, bf16 *H) {
#pragma unroll
		for (int j = 0; j < 2; j++) {
			const int c = c0 + j * 8 + 2 * t;
			const float b0 = __ldg(bias + c), b1 = __ldg(bias + c + 1);
#pragma unroll
			for (int mi = 0; mi < 2; mi++)
#pragma unroll
				for (int h = 0; h < 2; h++) {
					const int r = mi * 16 + g + 8 * h;
					p[mi][j][2 * h] += b0;
					p[mi][j][2 * h + 1] += b1;
					const uint32_t v = pack_bf16(gelu(p[mi][j][2 * h]), gelu(p[mi][j][2 * h + 1]));
					*reinterpret_cast<uint32_t *>(out + r * HP + c) = v;
					*reinterpret_cast<uint32_t *>(H + (r0 + r) * kHid + c) = v;
				}
		}
	};
	rows_mma<kInF, 2, 2>(Xs, XP, a.frag + kFragF1, warp * 2, p1);
	hidden(p1, a.master + kMlpOffB1, Hs, a.H1);
	__syncthreads();
	rows_mma<kHid, 2, 2>(Hs, HP, a.frag + kFragF2, warp * 2, p2);
	hidden(p2, a.master + kMlpOffB2, Gs, a.H2);
	__syncthreads();
	float *bias_part = a.bias_part + (size_t)blockIdx.x * kBiases;
	{
		// output layer: sigmoid, squared error, its gradient; a warp takes 8 columns
		// of 16 rows
		const int m0 = (warp >> 3) * 16;
		float o[1][1][4];
		rows_mma<kHid, 1, 1>(Gs + m0 * HP, HP, a.frag + kFragF3, warp & 7, o);
		const int c = (warp & 7) * 8 + 2 * t;
		const float b0 = __ldg(a.master + kMlpOffB3 + c), b1 = __ldg(a.master + kMlpOffB3 + c + 1);
		const float scale = 2.f / (float)(a.n * kOut);
		float loss = 0.f, s0 = 0.f, s1 = 0.f;
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int r = m0 + g + 8 * h;
			float d[2] = {0.f, 0.f};
			if (r0 + r < a.n) {
				const float *tg = a.target + (r0 + r) * kOut + c;
#pragma unroll
				for (int q = 0; q < 2; q++) {
					const float y = 1.f / (1.f + expf(-(o[0][0][2 * h + q] + (q ? b1 : b0))));
					const float e = y - tg[q];
					loss += e * e;
					d[q] = scale * e * y * (1.f - y);
				}
			}
			s0 += d[0];
			s1 += d[1];
			const uint32_t v = pack_bf16(d[0], d[1]);
			*reinterpret_cast<uint32_t *>(Ds + r * OP + c) = v;
			*reinterpret_cast<uint32_t *>(a.D3 + (r0 + r) * kOut + c) = v;
		}
		s0 = column_sum(s0);
		s1 = column_sum(s1);
		if (g == 0) { s_db3[warp >> 3][c] = s0; s_db3[warp >> 3][c + 1] = s1; }
#pragma unroll
		for (int s = 16; s > 0; s >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, s);
		if (lane == 0) s_loss[warp] = loss;
	}
	__syncthreads();
	if (tid < kOut) bias_part[2 * kHid + tid] = s_db3[0][tid] + s_db3[1][tid];
	if (tid == 0) {
		float l = 0.f;
		for (int i = 0; i < kTrainThreads / 32; i++) l += s_loss[i];
		a.loss_part[blockIdx.x] = l;
	}
	// gradient of a hidden layer: d = (dH) GELU'(p), to shared memory (when another
	// layer follows) and D, its column sums to the bias
	auto back = [&](const float (&dh)[2][2][4], const float (&p)[2][2][4], bf16 *out, bf16 *D, float *db) {
#pragma unroll
		for (int j = 0; j < 2; j++) {
			const int c = c0 + j * 8 + 2 * t;
			float s0 = 0.f, s1 = 0.f;
#pragma unroll
			for (int mi = 0; mi < 2; mi++)
#pragma unroll
				for (int h = 0; h < 2; h++) {
					const int r = mi * 16 + g + 8 * h;
					const float d0 = dh[mi][j][2 * h] * gelu_grad(p[mi][j][2 * h]);
					const float d1 = dh[mi][j][2 * h + 1] * gelu_grad(p[mi][j][2 * h + 1]);
					s0 += d0;
					s1 += d1;
					const uint32_t v = pack_bf16(d0, d1);
					if (out) *reinterpret_cast<uint32_t *>(out + r * HP + c) = v;
					*reinterpret_cast<uint32_t *>(D + (r0 + r) * kHid + c) = v;
				}
			s0 = column_sum(s0);
			s1 = column_sum(s1);
			if (g == 0) { db[c] = s0; db[c + 1] = s1; }
		}
	};
	float dh[2][2][4];
	rows_mma<kOut, 2, 2>(Ds, OP, a.frag + kFragB3, warp * 2, dh);
	back(dh, p2, Hs, a.D2, bias_part + kHid);     // Hs is free: layer 2 has read it
	__syncthreads();
	rows_mma<kHid, 2, 2>(Hs, HP, a.frag + kFragB2, warp * 2, dh);
	back(dh, p1, nullptr, a.D1, bias_part);
}

__device__ __forceinline__ void ldmatrix_t(uint32_t (&r)[4], const bf16 *p)
{
	const uint32_t s = (uint32_t)__cvta_generic_to_shared(p);
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
	             : "r"(s)
	             : "memory");
}

// part[split][offset ..] = A^T . B over the split's rows, one 64 x 64 tile per CTA:
// layer 2 (16 tiles), layer 3 (4), layer 1 (8, its last rows cut off at 80).
__global__ void __launch_bounds__(128)
weight_grad_kernel(const bf16 *__restrict__ X, const bf16 *__restrict__ H1, const bf16 *__restrict__ H2,
                   const bf16 *__restrict__ D1, const bf16 *__restrict__ D2, const bf16 *__restrict__ D3, int rows,
                   int split_rows, float *__restrict__ part)
{
	constexpr int KB = 32, SP = kGradTile + 8;
	__shared__ __align__(16) bf16 As[2][KB * SP], Bs[2][KB * SP];
	const int tile = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
	const bf16 *A, *B;
	int lda, ldb, m0, n0, M, N, off;
	if (tile < 16) { A = H1; B = D2; lda = ldb = kHid; m0 = tile / 4 * 64; n0 = tile % 4 * 64; M = N = kHid; off = kMlpOffW2; }
	else if (tile < 20) { A = H2; B = D3; lda = kHid; ldb = kOut; m0 = (tile - 16) * 64; n0 = 0; M = kHid; N = kOut; off = kMlpOffW3; }
	else { A = X; B = D1; lda = kInF; ldb = kHid; m0 = (tile - 20) / 4 * 64; n0 = (tile - 20) % 4 * 64; M = kInP; N = kHid; off = kMlpOffW1; }
	const int k0 = blockIdx.y * split_rows, k1 = min(rows, k0 + split_rows);
	// a 32 x 64 block of an operand: 256 pieces of 16 bytes, two per thread; columns
	// past the operand's width (layer 1's second tile) stay zero
	auto load = [&](bf16 *s, const bf16 *p, int ld, int c0, int r0) {
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int i = tid + h * 128, r = i >> 3, c = (i & 7) * 8;
			const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s + r * SP + c);
			const bool in = c0 + c < ld;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(p + (size_t)(r0 + r) * ld + (in ? c0 + c : 0)),
			             "r"(in ? 16 : 0));
		}
	};
	float acc[8][4];
#pragma unroll
	for (int j = 0; j < 8; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
	int buf = 0;
	if (k0 < k1) {
		load(As[0], A, lda, m0, k0);
		load(Bs[0], B, ldb, n0, k0);
	}
	asm volatile("cp.async.commit_group;\n");
	for (int k = k0; k < k1; k += KB, buf ^= 1) {
		if (k + KB < k1) {
			load(As[buf ^ 1], A, lda, m0, k + KB);
			load(Bs[buf ^ 1], B, ldb, n0, k + KB);
		}
		asm volatile("cp.async.commit_group;\n");
		asm volatile("cp.async.wait_group 1;\n");
		__syncthreads();
		// rows are the summed index: both operands come out of shared memory
		// transposed
#pragma unroll
		for (int ks = 0; ks < KB; ks += 16) {
			uint32_t af[4];
			// 8 x 8 blocks (k, m): (0, 0), (0, 8), (8, 0), (8, 8)
			ldmatrix_t(af, As[buf] + (ks + (lane >> 4) * 8 + (lane & 7)) * SP + warp * 16 + (lane >> 3 & 1) * 8);
#pragma unroll
			for (int j = 0; j < 8; j += 2) {
				uint32_t bq[4];
				// blocks (k, n): (0, 0), (8, 0), (0, 8), (8, 8)
				ldmatrix_t(bq, Bs[buf] + (ks + (lane >> 3 & 1) * 8 + (lane & 7)) * SP + j * 8 + (lane >> 4) * 8);
				mma_bf16(acc[j], af, bq[0], bq[1]);
				mma_bf16(acc[j + 1], af, bq[2], bq[3]);
			}
		}
		__syncthreads();
	}
	float *out = part + (size_t)blockIdx.y * kMlpMasterSize + off;
#pragma unroll
	for (int j = 0; j < 8; j++)
#pragma unroll
		for (int h = 0; h < 2; h++) {
			const int m = m0 + warp * 16 + g + 8 * h, c = n0 + j * 8 + 2 * t;
			if (m < M && c < N)
				*reinterpret_cast<float2 *>(out + (size_t)m * N + c) = make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
		}
}

// The weight's BF16 copies: in the forward pass' operand and, for training, in the
// backward one's.
__device__ __forceinline__ void store_weight(int i, float v, bf16 *frag, bool train)
{
	const bf16 b = __float2bfloat16_rn(v);
	if (i < kMlpOffB1) {
		frag[kFragF1 + frag_at(i / kHid, i % kHid, kInF)] = b;
	} else if (i >= kMlpOffW2 && i < kMlpOffB2) {
		const int j = i - kMlpOffW2, k = j / kHid, o = j % kHid;
		frag[kFragF2 + frag_at(k, o, kHid)] = b;
		if (train) frag[kFragB2 + frag_at(o, k, kHid)] = b;
	} else if (i >= kMlpOffW3 && i < kMlpOffB3) {
		const int j = i - kMlpOffW3, k = j / kOut, o = j % kOut;
		frag[kFragF3 + frag_at(k, o, kHid)] = b;
		if (train) frag[kFragB3 + frag_at(o, k, kOut)] = b;
	}
}

// (the inputs past the master's 80 are cleared by the caller)
__global__ void pack_weights_kernel(const float *__restrict__ m, bf16 *__restrict__ frag, int train)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpMasterSize; i += gridDim.x * blockDim.x)
		store_weight(i, m[i], frag, train != 0);
}

__device__ __forceinline__ bool is_bias(int i)
{
	return (i >= kMlpOffB1 && i < kMlpOffW2) || (i >= kMlpOffB2 && i < kMlpOffW3) || i >= kMlpOffB3;
}

struct Update {
	const float *part, *bias_part, *loss_part;
	int splits, ctas;
	float *grad, *loss;                  // grad: written when step is 0
	int step;
	float *p, *m, *v;
	float lr, b1, b2, eps, wd, c1, c2;
	bf16 *frag;
};

// Sums of the splits (weights: a thread each; biases and the loss: a warp each),
// then AdamW; weight decay on the matrices, not the biases.
__global__ void __launch_bounds__(256)
update_kernel(Update u)
{
	auto apply = [&](int i, float g) {
		if (!u.step) {
			u.grad[i] = g;
			return;
		}
		const float mi = u.b1 * u.m[i] + (1.f - u.b1) * g;
		const float vi = u.b2 * u.v[i] + (1.f - u.b2) * g * g;
		u.m[i] = mi;
		u.v[i] = vi;
		float q = u.p[i];
		const bool bias = is_bias(i);
		if (!bias) q -= u.lr * u.wd * q;
		q -= u.lr * (mi / u.c1) / (sqrtf(vi / u.c2) + u.eps);
		u.p[i] = q;
		if (!bias) store_weight(i, q, u.frag, true);
	};
	const int nthreads = gridDim.x * blockDim.x, id = blockIdx.x * blockDim.x + threadIdx.x;
	for (int i = id; i < kMlpMasterSize; i += nthreads) {
		if (is_bias(i)) continue;
		float g = 0.f;
#pragma unroll 4
		for (int s = 0; s < u.splits; s++) g += u.part[(size_t)s * kMlpMasterSize + i];
		apply(i, g);
	}
	const int lane = threadIdx.x & 31;
	for (int b = id >> 5; b <= kBiases; b += nthreads >> 5) {
		double s = 0.0;
		for (int c = lane; c < u.ctas; c += 32) s += b < kBiases ? u.bias_part[(size_t)c * kBiases + b] : u.loss_part[c];
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		if (lane != 0) continue;
		if (b == kBiases) *u.loss = (float)s;
		else apply(b < kHid ? kMlpOffB1 + b : b < 2 * kHid ? kMlpOffB2 + b - kHid : kMlpOffB3 + b - 2 * kHid, (float)s);
	}
}

int blocks_for(long long n, int threads, int cap = 4096)
{
	long long b = (n + threads - 1) / threads;
	return (int)std::max<long long>(1, std::min<long long>(b, cap));
}

}  // namespace

cudaError_t launch_mlp_forward(const uint16_t *X, long long n, const MlpWeights &w, float *out, int nsm,
                               cudaStream_t st)
{
	if (n <= 0) return cudaSuccess;
	cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                                     (int)kForwardSmem);
	if (e != cudaSuccess) return e;
	const long long need = (n + kFwdRows - 1) / kFwdRows;
	const int nb = (int)std::min<long long>(need, (long long)nsm * 2);
	mlp_forward_kernel<<<nb, kFwdThreads, kForwardSmem, st>>>(reinterpret_cast<const bf16 *>(X), n, w, out);
	return cudaGetLastError();
}

cudaError_t launch_pack_weights(const float *master, uint16_t *wt, cudaStream_t st)
{
	cudaError_t e = cudaMemsetAsync(wt, 0, sizeof(bf16) * kFragF2, st);
	if (e != cudaSuccess) return e;
	pack_weights_kernel<<<256, 256, 0, st>>>(master, reinterpret_cast<bf16 *>(wt), 0);
	return cudaGetLastError();
}

MlpWeights mlp_weights(const uint16_t *wt, const float *master)
{
	MlpWeights w;
	w.frag = reinterpret_cast<const bf16 *>(wt);
	w.b1 = master + kMlpOffB1;
	w.b2 = master + kMlpOffB2;
	w.b3 = master + kMlpOffB3;
	return w;
}

void mlp_public_to_master(const float *pub, float *master)
{
	std::memset(master, 0, sizeof(float) * kMlpMasterSize);
	for (int k = 0; k < kIn; k++)
		for (int o = 0; o < kHid; o++) master[kMlpOffW1 + k * kHid + o] = pub[k * kHid + o];
	std::memcpy(master + kMlpOffB1, pub + kIn * kHid, sizeof(float) * (kMlpMasterSize - kMlpOffB1));
}

void mlp_master_to_public(const float *master, float *pub)
{
	for (int k = 0; k < kIn; k++)
		for (int o = 0; o < kHid; o++) pub[k * kHid + o] = master[kMlpOffW1 + k * kHid + o];
	std::memcpy(pub + kIn * kHid, master + kMlpOffB1, sizeof(float) * (kMlpMasterSize - kMlpOffB1));
}

}  // namespace bm4dof

using namespace bm4dof;

// ---------------------------------------------------------------------------
// trainer

struct bm4dof_trainer {
	int device = 0, nsm = 0;
	unsigned batch = 0;
	long long step = 0;
	cudaStream_t st = nullptr;
	float *master = nullptr, *grad = nullptr, *m1 = nullptr, *m2 = nullptr;
	bf16 *frag = nullptr;        // the weights in fragment order
	// activations and gradients of one batch (rows padded to whole CTAs)
	bf16 *X = nullptr, *H1 = nullptr, *H2 = nullptr, *D1 = nullptr, *D2 = nullptr, *D3 = nullptr;
	float *part = nullptr, *bias_part = nullptr, *loss_part = nullptr, *loss = nullptr;
};

namespace {

#define TCK(expr)                                                                            \
	do {                                                                                     \
		cudaError_t e_ = (expr);                                                             \
		if (e_ != cudaSuccess) {                                                             \
			set_error(std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " #expr);  \
			return e_ == cudaErrorMemoryAllocation ? BM4DOF_ERR_NO_MEMORY : BM4DOF_ERR_CUDA; \
		}                                                                                    \
	} while (0)

void free_trainer(bm4dof_trainer *t)
{
	void *ps[] = {t->master, t->grad, t->m1, t->m2, t->frag, t->X, t->H1, t->H2, t->D1, t->D2, t->D3,
	              t->part, t->bias_part, t->loss_part, t->loss};
	for (void *p : ps)
		if (p) cudaFree(p);
	if (t->st) cudaStreamDestroy(t->st);
	delete t;
}

// forward + backward of n rows (n <= batch), then the gradients into t->grad
// (u.step 0) or an AdamW step; the loss into t->loss
bm4dof_status train_batch(bm4dof_trainer *t, const float *feat, const float *target, long long n, Update u)
{
	cudaStream_t st = t->st;
	const int ctas = (int)((n + kTrainRows - 1) / kTrainRows), rows = ctas * kTrainRows;
	TrainRows a;
	a.feat = feat;
	a.target = target;
	a.n = n;
	a.frag = t->frag;
	a.master = t->master;
	a.X = t->X;
	a.H1 = t->H1;
	a.H2 = t->H2;
	a.D1 = t->D1;
	a.D2 = t->D2;
	a.D3 = t->D3;
	a.bias_part = t->bias_part;
	a.loss_part = t->loss_part;
	train_rows_kernel<<<ctas, kTrainThreads, 0, st>>>(a);
	// rows split into pieces of at least kSplitRows, whole 32-row blocks each
	const int want = std::max(1, std::min(kMaxSplits, (rows + kSplitRows - 1) / kSplitRows));
	const int split_rows = ((rows + want - 1) / want + 31) / 32 * 32, splits = (rows + split_rows - 1) / split_rows;
	weight_grad_kernel<<<dim3(28, splits), 128, 0, st>>>(t->X, t->H1, t->H2, t->D1, t->D2, t->D3, rows, split_rows, t->part);
	u.part = t->part;
	u.bias_part = t->bias_part;
	u.loss_part = t->loss_part;
	u.splits = splits;
	u.ctas = ctas;
	u.grad = t->grad;
	u.loss = t->loss;
	u.p = t->master;
	u.m = t->m1;
	u.v = t->m2;
	u.frag = t->frag;
	update_kernel<<<blocks_for(kMlpMasterSize, 256), 256, 0, st>>>(u);
	TCK(cudaGetLastError());
	return BM4DOF_OK;
}

cudaError_t pack_trainer(bm4dof_trainer *t)
{
	pack_weights_kernel<<<256, 256, 0, t->st>>>(t->master, t->frag, 1);
	return cudaGetLastError();
}

bool trainer_ok(bm4dof_trainer *t, const void *feat, const void *target, unsigned n)
{
	if (!t || !feat || !target || n == 0 || n > t->batch) {
		set_error("bm4dof_trainer: bad argument (null pointer or n outside [1, batch])");
		return false;
	}
	return true;
}

}  // namespace

extern "C" {

bm4dof_status bm4dof_trainer_create(bm4dof_trainer **out, int device, unsigned batch, unsigned seed)
{
	clear_error();
	if (!out || batch == 0) { set_error("bm4dof_trainer_create: bad argument"); return BM4DOF_ERR_ARGUMENT; }
	*out = nullptr;
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
		cudaGetLastError();
		set_error("bm4dof_trainer_create: no CUDA device");
		return BM4DOF_ERR_NO_DEVICE;
	}
	if (device < 0 || device >= ndev) { set_error("bm4dof_trainer_create: bad device"); return BM4DOF_ERR_ARGUMENT; }
	TCK(cudaSetDevice(device));
	bm4dof_trainer *t = new bm4dof_trainer();
	t->device = device;
	t->batch = batch;
	cudaDeviceGetAttribute(&t->nsm, cudaDevAttrMultiProcessorCount, device);
	const size_t ctas = ((size_t)batch + kTrainRows - 1) / kTrainRows, B = ctas * kTrainRows;
	bool ok = cudaStreamCreateWithFlags(&t->st, cudaStreamNonBlocking) == cudaSuccess &&
	          cudaMalloc(&t->master, sizeof(float) * kMlpMasterSize) == cudaSuccess &&
	          cudaMalloc(&t->grad, sizeof(float) * kMlpMasterSize) == cudaSuccess &&
	          cudaMalloc(&t->m1, sizeof(float) * kMlpMasterSize) == cudaSuccess &&
	          cudaMalloc(&t->m2, sizeof(float) * kMlpMasterSize) == cudaSuccess &&
	          cudaMalloc(&t->frag, sizeof(bf16) * kFragSize) == cudaSuccess &&
	          cudaMalloc(&t->X, sizeof(bf16) * B * kInF) == cudaSuccess &&
	          cudaMalloc(&t->H1, sizeof(bf16) * B * kHid) == cudaSuccess &&
	          cudaMalloc(&t->H2, sizeof(bf16) * B * kHid) == cudaSuccess &&
	          cudaMalloc(&t->D1, sizeof(bf16) * B * kHid) == cudaSuccess &&
	          cudaMalloc(&t->D2, sizeof(bf16) * B * kHid) == cudaSuccess &&
	          cudaMalloc(&t->D3, sizeof(bf16) * B * kOut) == cudaSuccess &&
	          cudaMalloc(&t->part, sizeof(float) * kMaxSplits * kMlpMasterSize) == cudaSuccess &&
	          cudaMalloc(&t->bias_part, sizeof(float) * ctas * kBiases) == cudaSuccess &&
	          cudaMalloc(&t->loss_part, sizeof(float) * ctas) == cudaSuccess &&
	          cudaMalloc(&t->loss, sizeof(float)) == cudaSuccess;
	if (!ok) {
		cudaGetLastError();
		free_trainer(t);
		set_error("bm4dof_trainer_create: device allocation failed");
		return BM4DOF_ERR_NO_MEMORY;
	}
	// He-style uniform initialisation from a fixed LCG (host), zero biases
	std::vector<float> pub(kMlpPublicSize, 0.f);
	uint64_t s = 0x9E3779B97F4A7C15ull ^ seed;
	auto uni = [&s]() {
		s = s * 6364136223846793005ull + 1442695040888963407ull;
		return (float)((s >> 40) * (1.0 / 16777216.0)) * 2.f - 1.f;
	};
	const int fan[3] = {kIn, kHid, kHid}, outs[3] = {kHid, kHid, kOut};
	size_t o = 0;
	for (int l = 0; l < 3; l++) {
		const float a = std::sqrt(3.f / (float)fan[l]);
		for (int i = 0; i < fan[l] * outs[l]; i++) pub[o + i] = a * uni();
		o += (size_t)fan[l] * outs[l] + outs[l];
	}
	std::vector<float> master(kMlpMasterSize);
	mlp_public_to_master(pub.data(), master.data());
	TCK(cudaMemcpyAsync(t->master, master.data(), sizeof(float) * kMlpMasterSize, cudaMemcpyHostToDevice, t->st));
	TCK(cudaMemsetAsync(t->m1, 0, sizeof(float) * kMlpMasterSize, t->st));
	TCK(cudaMemsetAsync(t->m2, 0, sizeof(float) * kMlpMasterSize, t->st));
	TCK(cudaMemsetAsync(t->grad, 0, sizeof(float) * kMlpMasterSize, t->st));
	TCK(cudaMemsetAsync(t->frag, 0, sizeof(bf16) * kFragSize, t->st));   // inputs 80..95 stay zero
	TCK(pack_trainer(t));
	TCK(cudaStreamSynchronize(t->st));
	*out = t;
	return BM4DOF_OK;
}

bm4dof_status bm4dof_trainer_get_stream(bm4dof_trainer *t, void **stream)
{
	clear_error();
	if (!t || !stream) { set_error("bm4dof_trainer_get_stream: null argument"); return BM4DOF_ERR_ARGUMENT; }
	*stream = static_cast<void *>(t->st);
	return BM4DOF_OK;
}

void bm4dof_trainer_destroy(bm4dof_trainer *t)
{
	if (!t) return;
	cudaSetDevice(t->device);
	cudaStreamSynchronize(t->st);
	free_trainer(t);
}

bm4dof_status bm4dof_trainer_params(bm4dof_trainer *t, float *params, size_t n, int set)
{
	clear_error();
	if (!t || !params || n != (size_t)kMlpPublicSize) {
		set_error("bm4dof_trainer_params: bad argument (the blob holds " + std::to_string(kMlpPublicSize) + " floats)");
		return BM4DOF_ERR_ARGUMENT;
	}
	TCK(cudaSetDevice(t->device));
	std::vector<float> master(kMlpMasterSize);
	if (set) {
		mlp_public_to_master(params, master.data());
		TCK(cudaMemcpyAsync(t->master, master.data(), sizeof(float) * kMlpMasterSize, cudaMemcpyHostToDevice, t->st));
		TCK(pack_trainer(t));
		TCK(cudaStreamSynchronize(t->st));
	} else {
		TCK(cudaMemcpyAsync(master.data(), t->master, sizeof(float) * kMlpMasterSize, cudaMemcpyDeviceToHost, t->st));
		TCK(cudaStreamSynchronize(t->st));
		mlp_master_to_public(master.data(), params);
	}
	return BM4DOF_OK;
}

bm4dof_status bm4dof_trainer_state(bm4dof_trainer *t, float *moment1, float *moment2, size_t n,
                                   unsigned long long *steps, int set)
{
	clear_error();
	if (!t || !moment1 || !moment2 || !steps || n != (size_t)kMlpPublicSize) {
		set_error("bm4dof_trainer_state: bad argument (each moment holds " + std::to_string(kMlpPublicSize) +
		          " floats)");
		return BM4DOF_ERR_ARGUMENT;
	}
	TCK(cudaSetDevice(t->device));
	std::vector<float> m1(kMlpMasterSize), m2(kMlpMasterSize);
	if (set) {
		// the padded inputs of W1 never receive a gradient: their moments stay 0
		mlp_public_to_master(moment1, m1.data());
		mlp_public_to_master(moment2, m2.data());
		TCK(cudaMemcpyAsync(t->m1, m1.data(), sizeof(float) * kMlpMasterSize, cudaMemcpyHostToDevice, t->st));
		TCK(cudaMemcpyAsync(t->m2, m2.data(), sizeof(float) * kMlpMasterSize, cudaMemcpyHostToDevice, t->st));
		TCK(cudaStreamSynchronize(t->st));
		t->step = (long long)*steps;
	} else {
		TCK(cudaMemcpyAsync(m1.data(), t->m1, sizeof(float) * kMlpMasterSize, cudaMemcpyDeviceToHost, t->st));
		TCK(cudaMemcpyAsync(m2.data(), t->m2, sizeof(float) * kMlpMasterSize, cudaMemcpyDeviceToHost, t->st));
		TCK(cudaStreamSynchronize(t->st));
		mlp_master_to_public(m1.data(), moment1);
		mlp_master_to_public(m2.data(), moment2);
		*steps = (unsigned long long)t->step;
	}
	return BM4DOF_OK;
}

bm4dof_status bm4dof_trainer_grad(bm4dof_trainer *t, const float *feat, const float *target, unsigned n,
                                  float *grads, float *loss)
{
	clear_error();
	if (!trainer_ok(t, feat, target, n)) return BM4DOF_ERR_ARGUMENT;
	TCK(cudaSetDevice(t->device));
	bm4dof_status s = train_batch(t, feat, target, n, Update{});
	if (s != BM4DOF_OK) return s;
	std::vector<float> g(kMlpMasterSize);
	float l = 0.f;
	TCK(cudaMemcpyAsync(g.data(), t->grad, sizeof(float) * kMlpMasterSize, cudaMemcpyDeviceToHost, t->st));
	TCK(cudaMemcpyAsync(&l, t->loss, sizeof(float), cudaMemcpyDeviceToHost, t->st));
	TCK(cudaStreamSynchronize(t->st));
	if (grads) mlp_master_to_public(g.data(), grads);
	if (loss) *loss = l / (float)((size_t)n * kOut);
	return BM4DOF_OK;
}

bm4dof_status bm4dof_trainer_step(bm4dof_trainer *t, const float *feat, const float *target, unsigned n,
                                  float lr, float weight_decay, float *loss)
{
	clear_error();
	if (!trainer_ok(t, feat, target, n)) return BM4DOF_ERR_ARGUMENT;
	TCK(cudaSetDevice(t->device));
	Update u{};
	u.step = 1;
	u.lr = lr;
	u.b1 = 0.9f;
	u.b2 = 0.999f;
	u.eps = 1e-8f;
	u.wd = weight_decay;
	u.c1 = 1.f - std::pow(u.b1, (float)(t->step + 1));
	u.c2 = 1.f - std::pow(u.b2, (float)(t->step + 1));
	bm4dof_status s = train_batch(t, feat, target, n, u);
	if (s != BM4DOF_OK) return s;
	t->step++;
	if (loss) {
		float l = 0.f;
		TCK(cudaMemcpyAsync(&l, t->loss, sizeof(float), cudaMemcpyDeviceToHost, t->st));
		TCK(cudaStreamSynchronize(t->st));
		*loss = l / (float)((size_t)n * kOut);
	}
	return BM4DOF_OK;
}

bm4dof_status bm4dof_trainer_predict(bm4dof_trainer *t, const float *feat, unsigned n, float *gains)
{
	clear_error();
	if (!t || !feat || !gains || n == 0 || n > t->batch) {
		set_error("bm4dof_trainer_predict: bad argument");
		return BM4DOF_ERR_ARGUMENT;
	}
	TCK(cudaSetDevice(t->device));
	pack_features_kernel<<<blocks_for((long long)n * kInP, 256), 256, 0, t->st>>>(feat, n, t->X);
	TCK(launch_mlp_forward(reinterpret_cast<const uint16_t *>(t->X), n, mlp_weights(reinterpret_cast<const uint16_t *>(t->frag), t->master), gains,
	                       t->nsm, t->st));
	TCK(cudaStreamSynchronize(t->st));
	return BM4DOF_OK;
}

}  // extern "C"
