// filter.cu -- collaborative filtering of each patch group, exact FP32.
//
// Restates VideoNLB::computeBayesEstimateStep1/2 and their _vbm3d bodies
// (src/core/nldct.cpp:1799-2006, 2015-2242) bit for bit:
//   * all-members-equal groups are left untouched and keep the previous
//     group's aggregation weights (1986-1999, 2222-2235) -- flagged here and
//     completed by fixup_equal_kernel;
//   * Z = G.B, the dense sPC x sPC patch transform, accumulated over the inner
//     index in increasing order with one rounded multiply and one rounded add
//     per term -- the order of the sequential sgemm the reference is built
//     with (productMatrix, src/core/matrix_funs.cpp:136-164);
//   * orthonormal Haar along the member axis (1846-1860), hard threshold at
//     (beta*sigma)^2 keeping coefficient (0,0) (1901-1908) or the empirical
//     Wiener gain against the basic estimate (2123-2135), inverse Haar, and
//     the inverse transform Z.Binv^T (1926-1931, 2155-2159);
//   * group weight 1/sigma^2/#kept in float (1935) or 1/sigma^2/sum(w^2) in
//     double (2167), the Wiener sum taken in the reference's order.
// The result is written as per-member estimates and weights; the gather forms
// the products (w*window[p])*g that the reference adds into its image
// (2296-2297, 2385-2386).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "common.cuh"

namespace bm4dof {

namespace {

constexpr int kFilterThreads = 256;

__device__ __forceinline__ int nsp_of(int np)
{
	// member stride of the shared-memory group tiles: a multiple of 4 (float4
	// access) plus 4, which spreads consecutive rows over distinct banks
	return ((np + 3) / 4) * 4 + 4;
}

template <int NS>
__device__ __forceinline__ void haar_forward(float (&z)[NS], float is2)
{
#pragma unroll
	for (int s = 2, h = 1; s <= NS; s *= 2, h *= 2)
#pragma unroll
		for (int n = 0; n < NS; n += s) {
			const float z0 = __fmul_rn(z[n], is2);
			const float z1 = __fmul_rn(z[n + h], is2);
			z[n] = __fadd_rn(z0, z1);
			z[n + h] = __fsub_rn(z0, z1);
		}
}

template <int NS>
__device__ __forceinline__ void haar_inverse(float (&z)[NS], float is2)
{
#pragma unroll
	for (int s = NS, h = NS / 2; s >= 2; s /= 2, h /= 2)
#pragma unroll
		for (int n = 0; n < NS; n += s) {
			const float z0 = __fmul_rn(z[n], is2);
			const float z1 = __fmul_rn(z[n + h], is2);
			z[n] = __fadd_rn(z0, z1);
			z[n + h] = __fsub_rn(z0, z1);
		}
}

// std::max(a, 0.f) as libstdc++ evaluates it ((a < 0) ? 0 : a, NaN kept)
__device__ __forceinline__ float max0(float a) { return a < 0.f ? 0.f : a; }

// Order-invariant shrinkage of one coefficient's Haar rows z, with y the basic
// estimate's (step 2) or z itself (step 1); returns its share of the group weight.
template <int NS, int STEP>
__device__ __forceinline__ float shrink_invariant(float (&z)[NS], const float (&y)[NS], float bs2, float sigma2, float bm2)
{
	float vi = 0.f;
#pragma unroll
	for (int n = 1; n < NS; n++) vi = __fadd_rn(vi, __fmul_rn(y[n], y[n]));
	vi = __fdiv_rn(vi, (float)(NS - 1));
	const float v0 = STEP == 1 ? max0(__fsub_rn(__fmul_rn(y[0], y[0]), sigma2)) : __fmul_rn(y[0], y[0]);
	const float w0 = __fdiv_rn(v0, __fadd_rn(v0, bm2));
	z[0] = __fmul_rn(z[0], w0);
	if (STEP == 1) vi = max0(__fsub_rn(vi, sigma2));
	const float wi = __fdiv_rn(vi, __fadd_rn(vi, bs2));
#pragma unroll
	for (int n = 1; n < NS; n++) z[n] = __fmul_rn(z[n], wi);
	return __fadd_rn(__fmul_rn(w0, w0), __fmul_rn(__fmul_rn((float)(NS - 1), wi), wi));
}

// One transform coefficient k of one channel: Haar over the NS members,
// shrinkage, inverse Haar.  Returns the number of kept coefficients (step 1).
// With order invariance (nldct.cpp:1865-1900, 2101-2122) one Wiener gain
// serves the mean row and one all other rows; the coefficient's share of the
// group weight, w0^2 + (NS-1) wi^2, goes to *contrib.
template <int NS, int STEP>
__device__ int shrink_column(float *zcol, const float *ycol, float *w2col, int k, float bs2,
                             float is2, bool oinv, float sigma2, float bm2, float *contrib)
{
	float z[NS];
#pragma unroll
	for (int n = 0; n < NS; n++) z[n] = zcol[n];
	haar_forward<NS>(z, is2);
	int kept = 0;
	if (oinv) {
		float y[NS];
#pragma unroll
		for (int n = 0; n < NS; n++) y[n] = STEP == 1 ? z[n] : ycol[n];
		if (STEP == 2) haar_forward<NS>(y, is2);
		*contrib = shrink_invariant<NS, STEP>(z, y, bs2, sigma2, bm2);
	} else if (STEP == 1) {
#pragma unroll
		for (int n = 0; n < NS; n++) {
			if (__fmul_rn(z[n], z[n]) > bs2 || (k == 0 && n == 0)) kept++;
			else z[n] = 0.f;
		}
	} else {
		float y[NS];
#pragma unroll
		for (int n = 0; n < NS; n++) y[n] = ycol[n];
		haar_forward<NS>(y, is2);
#pragma unroll
		for (int n = 0; n < NS; n++) {
			const float yy = __fmul_rn(y[n], y[n]);
			const float w = __fdiv_rn(yy, __fadd_rn(yy, bs2));
			z[n] = __fmul_rn(z[n], w);
			w2col[n] = __fmul_rn(w, w);
		}
	}
	haar_inverse<NS>(z, is2);
#pragma unroll
	for (int n = 0; n < NS; n++) zcol[n] = z[n];
	return kept;
}

template <int STEP>
__device__ int shrink_dispatch(int ns, float *zcol, const float *ycol, float *w2col, int k,
                               float bs2, float is2, bool oinv, float sigma2, float bm2, float *contrib)
{
#define SHRINK(N) shrink_column<N, STEP>(zcol, ycol, w2col, k, bs2, is2, oinv, sigma2, bm2, contrib)
	switch (ns) {
	case 1: return SHRINK(1);
	case 2: return SHRINK(2);
	case 4: return SHRINK(4);
	case 8: return SHRINK(8);
	case 16: return SHRINK(16);
	default: return SHRINK(32);
	}
#undef SHRINK
}

// out(n, q) = sum_r in(n, r) * M[r*spc + q], r increasing, for a block of 4
// members starting at n0.  in is a [r][nsp] tile, out a [q][nsp] tile.
__device__ __forceinline__ void product4(const float *in, const float *M, float *out, int spc,
                                         int nsp, int q, int n0)
{
	float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
	for (int r = 0; r < spc; r++) {
		const float4 g = *reinterpret_cast<const float4 *>(in + r * nsp + n0);
		const float b = M[r * spc + q];
		a0 = __fadd_rn(a0, __fmul_rn(g.x, b));
		a1 = __fadd_rn(a1, __fmul_rn(g.y, b));
		a2 = __fadd_rn(a2, __fmul_rn(g.z, b));
		a3 = __fadd_rn(a3, __fmul_rn(g.w, b));
	}
	*reinterpret_cast<float4 *>(out + q * nsp + n0) = make_float4(a0, a1, a2, a3);
}

// Any patch shape.
template <int STEP>
__global__ void __launch_bounds__(kFilterThreads, STEP == 2 ? 3 : 4)
filter_exact_kernel(Image noisy, Image basic, const Tile *__restrict__ tiles, int ntiles,
                    StepParams sp, const float *__restrict__ basis, const float *__restrict__ binv,
                    long long g_begin, long long g_end,
                    const uint8_t *__restrict__ nsimp, const uint32_t *__restrict__ idx,
                    const uint8_t *__restrict__ alive, float *__restrict__ vals,
                    float *__restrict__ wslot, float *__restrict__ wgroup, uint8_t *__restrict__ eq)
{
	extern __shared__ __align__(16) float sm[];
	const int px = sp.px, pt = sp.pt, C = sp.C;
	const int spc = px * px * pt, np = sp.np;
	const int nsp = nsp_of(np);
	const int tile_f = C * spc * nsp;          // floats of one group tile (all channels)
	const int bsz = ((spc * spc + 3) / 4) * 4; // basis sizes padded: the group tiles
	                                           // below must start on 16-byte boundaries
	float *Bt = sm;                            // Bt[p*spc + k] = basis[k*spc + p]
	float *Bi = Bt + bsz;                      // Bi[k*spc + p] = binv[k*spc + p]
	float *Gn = Bi + bsz;                      // noisy group   [c][p][n]
	float *Zn = Gn + tile_f;                   // its transform [c][k][n]
	float *Gb = Zn + tile_f;                   // basic group (step 2); later Wiener w^2
	float *Zb = Gb + tile_f;
	__shared__ int s_mx[kMaxNp], s_my[kMaxNp], s_mt[kMaxNp];
	__shared__ int s_kept, s_ns, s_tile, s_equal;
	__shared__ float s_w;

	const int tid = threadIdx.x;
	for (int i = tid; i < spc * spc; i += blockDim.x) {
		const int k = i / spc, p = i % spc;
		Bt[p * spc + k] = basis[i];
		Bi[i] = binv[i];
	}

	const float sigma2 = __fmul_rn(sp.sigma, sp.sigma);
	const float bsig = __fmul_rn(sp.beta, sp.sigma);
	const float bs2 = __fmul_rn(bsig, bsig);
	const float bmsig = __fmul_rn(sp.beta_mean, sp.sigma);
	const float bm2 = __fmul_rn(bmsig, bmsig);
	const bool oinv = sp.order_inv != 0;
	const float is2 = (float)(1.0 / sqrt(2.0));

	for (long long g = g_begin + blockIdx.x; g < g_end; g += gridDim.x) {
		__syncthreads();
		if (!alive[g]) continue;
		if (tid == 0) {
			const int ti = tile_of(tiles, ntiles, g);
			s_tile = ti;
			s_ns = nsimp[g];
			s_kept = 0;
			s_equal = 0;
		}
		__syncthreads();
		const int ns = s_ns;
		const Tile T = tiles[s_tile];
		if (tid < ns) {
			const uint32_t lin = idx[g * np + tid];
			const uint32_t whl = (uint32_t)T.w * T.h;
			s_mt[tid] = (int)(lin / whl);
			s_my[tid] = (int)((lin % whl) / T.w);
			s_mx[tid] = (int)(lin % T.w);
		}
		__syncthreads();

		// gather the group: member-fastest tiles G[c][p][n] (nldct.cpp:1334-1339)
		const int per = C * spc;
		for (int it = tid; it < ns * per; it += blockDim.x) {
			const int n = it / per, r = it % per;
			const int c = r / spc, p = r % spc;
			const int ht = p / (px * px), hy = (p / px) % px, hx = p % px;
			const size_t a = noisy.at(T.ox + s_mx[n] + hx, T.oy + s_my[n] + hy, s_mt[n] + ht, c);
			Gn[(c * spc + p) * nsp + n] = __ldg(noisy.p + a);
			if (STEP == 2) Gb[(c * spc + p) * nsp + n] = __ldg(basic.p + a);
		}
		__syncthreads();

		const long long slot0 = (g - g_begin) * np;   // slots are chunk-relative
		// all-equal test (nldct.cpp:1986-1999, 2222-2235)
		int differs = 0;
		if (ns > 1)
			for (int r = tid; r < per; r += blockDim.x) {
				const float *row = Gn + r * nsp;
				for (int n = 1; n < ns; n++) differs |= row[n] != row[0];
			}
		const int any = __syncthreads_or(differs);
		if (ns > 1 && !any) {
			// unweighted: the weights are set later (fixup_equal_kernel)
			for (int it = tid; it < ns * per; it += blockDim.x) {
				const int n = it / per, r = it % per;
				const int c = r / spc, p = r % spc;
				vals[((slot0 + n) * C + c) * spc + term_of(px, pt, p)] = Gn[r * nsp + n];
			}
			if (tid == 0) eq[g] = 1;
			continue;
		}

		// forward transform(s): Z(n,k) = sum_p G(n,p) B(p,k)
		const int nblk = (ns + 3) / 4;
		const int nprod = (STEP == 2 ? 2 : 1) * C * spc * nblk;
		for (int it = tid; it < nprod; it += blockDim.x) {
			int r = it;
			const int k = r % spc; r /= spc;
			const int nb = r % nblk; r /= nblk;
			const int c = r % C; r /= C;
			const float *in = (r == 0 ? Gn : Gb) + c * spc * nsp;
			float *out = (r == 0 ? Zn : Zb) + c * spc * nsp;
			product4(in, Bt, out, spc, nsp, k, nb * 4);
		}
		__syncthreads();

		// Haar, shrinkage, inverse Haar per (channel, coefficient)
		int kept = 0;
		for (int it = tid; it < C * spc; it += blockDim.x) {
			const int k = it % spc;
			kept += shrink_dispatch<STEP>(ns, Zn + it * nsp, Zb + it * nsp, Gb + it * ns, k, bs2, is2, oinv,
			                              sigma2, bm2, Gb + it);
		}
		if (STEP == 1 && kept) atomicAdd(&s_kept, kept);
		__syncthreads();

		// inverse transform Ghat(n,p) = sum_k Z(n,k) Binv[k*spc + p] into Gn,
		// while one lane forms the group weight
		if (tid < 32) {
			if (tid == 0) {
				if (oinv) {
					// float sum of the coefficients' shares in (c, k) order
					float v = 0.f;
					for (int i = 0; i < C * spc; i++) v = __fadd_rn(v, Gb[i]);
					s_w = STEP == 1 ? __fdiv_rn(__fdiv_rn(1.f, sigma2), v) : (float)(1.0 / (double)sigma2 / (double)v);
				} else if (STEP == 1) {
					s_w = __fdiv_rn(__fdiv_rn(1.f, sigma2), (float)s_kept);
				} else {
					float v = 0.f;   // sum of w^2 in the reference's (c, k, n) order
					for (int i = 0; i < C * spc * ns; i++) v = __fadd_rn(v, Gb[i]);
					s_w = (float)(1.0 / (double)sigma2 / (double)v);
				}
			}
		} else {
			const int ninv = C * spc * nblk;
			for (int it = tid - 32; it < ninv; it += blockDim.x - 32) {
				int r = it;
				const int p = r % spc; r /= spc;
				const int nb = r % nblk; r /= nblk;
				const int c = r;
				product4(Zn + c * spc * nsp, Bi, Gn + c * spc * nsp, spc, nsp, p, nb * 4);
			}
		}
		__syncthreads();

		// the estimates; the gather forms (w * window[p]) * ghat (nldct.cpp:2296-2297, 2385-2386)
		const float w = s_w;
		for (int it = tid; it < ns * per; it += blockDim.x) {
			const int n = it / per, r = it % per;
			const int c = r / spc, p = r % spc;
			vals[((slot0 + n) * C + c) * spc + term_of(px, pt, p)] = Gn[r * nsp + n];
		}
		if (tid < ns) wslot[slot0 + tid] = w;
		if (tid == 0) { wgroup[g] = w; eq[g] = 0; }
	}
}

// ---------------------------------------------------------------------------
// The same filter by warps, for the patch shapes of the benchmark and default
// parameters (4x4x4, 8x8, 7x7): a lane is one member of one group, 32 / L groups
// of up to L members to a warp, no barriers.
//
//   * A lane forms all SPC transform coefficients of its member, one register
//     each: out[q] = sum_r in[r] M[r][q], r increasing, every product and sum
//     rounded by itself -- the generic kernel's results, bit for bit.
//   * The members' pixels are staged, then transposed, through one (step 2: two)
//     shared tiles per warp [element][lane]; Haar transform, shrinkage and its
//     inverse take a coefficient's members as one row of the tile.
//   * 4x4x4 DCT (DCT4): the products.  A basis value is (ax ay) at with |a| one of
//     three numbers (h, A, B), so the 64 products of one pixel have 27 magnitudes
//     and the 64 of one coefficient at most 8.  Products are formed once per
//     magnitude and frame (36 per pixel, 9 per coefficient on average, signs of
//     the frame factor included) and added or subtracted: the same rounded
//     terms, since rounding is symmetric.  173 instead of 256 operations for a
//     pixel's part of a forward and an inverse transform.
//   * Other shapes: the basis in shared memory, four values per load for the
//     whole warp, products in pairs (f32x2), sums one at a time.
//
// What bounds it: the FP32 pipe and issue slots (4x4x4, step 2: pipe busy 62 %,
// issue 69 % of the cycles; the products are 80 % of the instructions).  Filter
// time, per-group CTAs or four groups per CTA -> this kernel (ms, both steps):
// 1920x1080x24 308 -> 174, 640x360x3x14 90.5 -> 27.8, 767x511 colour image with
// defaults 19.8 -> 8.0, 853x481x16 with defaults 10.9 -> 3.8.  On the way: the
// basis multiplied out densely 242 on 1920x1080x24 with a frame's code unrolled,
// 185 with a row's, 174 with the weight's chain of sums beside the inverse
// transform.
// ---------------------------------------------------------------------------
constexpr int kFwWarps = 4, kTileP = 36;   // row pitch: rows 8 apart share no bank in 16-byte accesses

// (x0 * y0, x1 * y1), each rounded as __fmul_rn (mul.rn.f32x2)
__device__ __forceinline__ void mul2(float x0, float x1, float y0, float y1, float &p0, float &p1)
{
	unsigned long long x, y, z;
	asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(x0), "f"(x1));
	asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(y0), "f"(y1));
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(z) : "l"(x), "l"(y));
	asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(z));
}

// 4-point DCT: a[k][n] = sign(k, n) * magnitude(k, n); magnitudes by class: 0 = h
// (k even), 1 = A, 2 = B (k odd: A where n and k are both outer or both inner).
__host__ __device__ constexpr bool dct4_neg(int k, int n)
{
	return k == 1 ? n >= 2 : k == 2 ? (n == 1 || n == 2) : k == 3 ? (n & 1) != 0 : false;
}
__host__ __device__ constexpr int dct4_class(int k, int n)
{
	return (k & 1) == 0 ? 0 : ((k == 1) == (n == 0 || n == 3) ? 1 : 2);
}

// f(0), f(1), .. with the index as a compile-time constant (arrays indexed by it
// stay in registers)
template <class F, int... I>
__device__ __forceinline__ void static_for_(F f, std::integer_sequence<int, I...>) { (f(std::integral_constant<int, I>{}), ...); }
template <int N, class F>
__device__ __forceinline__ void static_for(F f) { static_for_(f, std::make_integer_sequence<int, N>{}); }

// The DCT's tables in shared memory, read by whole warps: the loops below take a
// row (four pixels or coefficients) per pass, so that their code (300
// instructions) stays in the instruction cache; unrolled over a frame it did
// not, and a third of the issue slots went to fetching it.
struct Dct4Tables {
	// forward, by whether the pixel's frame and row are inner: (mag x) (mag y) (mag t)
	// for the classes of x (by magnitude), ky and kt
	float fwd[4][28];
	// inverse, by the classes of kt and ky: magnitudes x, then outer/inner rows and frames
	float inv[9][12];
	// sign(k_t, n_t) sign(k_y, n_y): by pixel frame and row for every kt, ky, and by
	// kt and ky for every pixel frame and row
	float fwd_sign[16][16], inv_sign[16][16];

	__device__ void fill(const float *mag, int tid, int nthreads)
	{
		auto m = [&](int c) { return c == 0 ? mag[0] : c == 1 ? mag[1] : mag[2]; };
		for (int i = tid; i < 4 * 27; i += nthreads) {
			const int v = i / 27, x = i / 9 % 3, y = i / 3 % 3, t = i % 3;
			// class 0 is k = 0 and 2, class 1 is k = 1, class 2 is k = 3
			const int cy = dct4_class(y == 0 ? 0 : 2 * y - 1, v & 1), ct = dct4_class(t == 0 ? 0 : 2 * t - 1, v >> 1);
			fwd[v][i % 27] = __fmul_rn(__fmul_rn(m(x), m(cy)), m(ct));
		}
		for (int i = tid; i < 9 * 12; i += nthreads) {
			const int v = i / 12, x = i / 4 % 3, y = i / 2 % 2, t = i % 2;
			const int ky = v % 3 == 0 ? 0 : 2 * (v % 3) - 1, kt = v / 3 == 0 ? 0 : 2 * (v / 3) - 1;
			inv[v][i % 12] = __fmul_rn(__fmul_rn(m(x), m(dct4_class(ky, y))), m(dct4_class(kt, t)));
		}
		for (int i = tid; i < 256; i += nthreads) {
			const int a = i >> 6, b = i >> 4 & 3, c = i >> 2 & 3, d = i & 3;
			fwd_sign[i >> 4][i & 15] = dct4_neg(c, a) != dct4_neg(d, b) ? -1.f : 1.f;
			inv_sign[i >> 4][i & 15] = dct4_neg(a, c) != dct4_neg(b, d) ? -1.f : 1.f;
		}
	}
};

template <int N>
__device__ __forceinline__ void load_table(const float *t, float (&v)[N])
{
#pragma unroll
	for (int i = 0; i < N; i += 4) {
		const float4 q = *reinterpret_cast<const float4 *>(t + i);
		v[i] = q.x;
		v[i + 1] = q.y;
		v[i + 2] = q.z;
		v[i + 3] = q.w;
	}
}

// a + p * s for s = 1 or -1: the product is exact, so this is the rounded sum or
// difference that a separate add gives
__device__ __forceinline__ float add_signed(float a, float p, float s, bool neg) { return __fmaf_rn(neg ? -p : p, s, a); }

// out[(kt, ky, kx)] = sum over the pixels (nt, ny, nx) of col[.. * kTileP] * basis
__device__ __forceinline__ void dct4_forward(const float *col, const Dct4Tables &tab, float (&out)[64])
{
#pragma unroll
	for (int k = 0; k < 64; k++) out[k] = 0.f;
#pragma unroll 1
	for (int it = 0; it < 16; it++) {
		const int nt = it >> 2, ny = it & 3;
		float m[28], sg[16];
		load_table(tab.fwd[(nt == 1 || nt == 2 ? 2 : 0) + (ny == 1 || ny == 2 ? 1 : 0)], m);
		load_table(tab.fwd_sign[it], sg);
		static_for<4>([&](auto nx) {
			const float g = col[(it * 4 + nx) * kTileP];
			static_for<3>([&](auto cx) {
				constexpr int ix = dct4_class(cx == 0 ? 0 : 2 * cx - 1, nx);
				float p[9];
#pragma unroll
				for (int q = 0; q < 8; q += 2) mul2(g, g, m[ix * 9 + q], m[ix * 9 + q + 1], p[q], p[q + 1]);
				p[8] = __fmul_rn(g, m[ix * 9 + 8]);
				static_for<64>([&](auto k) {
					constexpr int kt = k / 16, ky = k / 4 % 4, kx = k % 4;
					constexpr int cy = ky % 2 ? (ky + 1) / 2 : 0, ct = kt % 2 ? (kt + 1) / 2 : 0;
					if constexpr ((kx % 2 ? (kx + 1) / 2 : 0) == cx)
						out[k] = add_signed(out[k], p[cy * 3 + ct], sg[kt * 4 + ky], dct4_neg(kx, nx));
				});
			});
		});
	}
}

// out[(nt, ny, nx)] = sum over the coefficients (kt, ky, kx) of col[..] * basis;
// also(r) is called with each coefficient in turn
template <class F>
__device__ __forceinline__ void dct4_inverse(const float *col, const Dct4Tables &tab, float (&out)[64], F also)
{
#pragma unroll
	for (int k = 0; k < 64; k++) out[k] = 0.f;
#pragma unroll 1
	for (int it = 0; it < 16; it++) {
		const int kt = it >> 2, ky = it & 3;
		float m[12], sg[16];
		load_table(tab.inv[(kt & 1 ? (kt + 1) / 2 : 0) * 3 + (ky & 1 ? (ky + 1) / 2 : 0)], m);
		load_table(tab.inv_sign[it], sg);
		static_for<4>([&](auto kx) {
			const float z = col[(it * 4 + kx) * kTileP];
			also(it * 4 + kx);
			// outer (nx = 0, 3) and inner columns; even kx have one magnitude
			static_for<2>([&](auto xi) {
				if constexpr (kx % 2 == 1 || xi == 0) {
					constexpr int ix = dct4_class(kx, xi);
					float p[4];   // outer/inner rows, outer/inner frames
					mul2(z, z, m[ix * 4], m[ix * 4 + 1], p[0], p[1]);
					mul2(z, z, m[ix * 4 + 2], m[ix * 4 + 3], p[2], p[3]);
					static_for<64>([&](auto n) {
						constexpr int nt = n / 16, ny = n / 4 % 4, nx = n % 4;
						constexpr bool inx = kx % 2 == 0 || ((nx == 1 || nx == 2) == (xi == 1));
						constexpr int q = (ny == 1 || ny == 2 ? 2 : 0) + (nt == 1 || nt == 2 ? 1 : 0);
						if constexpr (inx) out[n] = add_signed(out[n], p[q], sg[nt * 4 + ny], dct4_neg(kx, nx));
					});
				}
			});
		});
	}
}

// out[q] = sum_r col[r * kTileP] * M[r][q], any basis; M rows of SP floats; also(r)
// is called with each r in turn
template <int SPC, int SP, class F>
__device__ __forceinline__ void dense_product(const float *col, const float *M, float (&out)[64], F also)
{
#pragma unroll
	for (int q = 0; q < 64; q++) out[q] = 0.f;
#pragma unroll 1
	for (int r = 0; r < SPC; r++) {
		const float g = col[r * kTileP];
		const float *m = M + r * SP;
		also(r);
#pragma unroll
		for (int q = 0; q < SP; q += 4) {
			const float4 b = *reinterpret_cast<const float4 *>(m + q);
			float p[4];
			mul2(g, g, b.x, b.y, p[0], p[1]);
			mul2(g, g, b.z, b.w, p[2], p[3]);
#pragma unroll
			for (int i = 0; i < 4; i++)
				if (q + i < SPC) out[q + i] = __fadd_rn(out[q + i], p[i]);
		}
	}
}

// A row of members: 16-byte accesses where there are four of them
template <int NS>
__device__ __forceinline__ void load_row(const float *row, float (&z)[NS])
{
	if constexpr (NS >= 4) {
#pragma unroll
		for (int n = 0; n < NS; n += 4) {
			const float4 v = *reinterpret_cast<const float4 *>(row + n);
			z[n] = v.x;
			z[n + 1] = v.y;
			z[n + 2] = v.z;
			z[n + 3] = v.w;
		}
	} else {
#pragma unroll
		for (int n = 0; n < NS; n++) z[n] = row[n];
	}
}

template <int NS>
__device__ __forceinline__ void store_row(float *row, const float (&z)[NS])
{
	if constexpr (NS >= 4) {
#pragma unroll
		for (int n = 0; n < NS; n += 4)
			*reinterpret_cast<float4 *>(row + n) = make_float4(z[n], z[n + 1], z[n + 2], z[n + 3]);
	} else {
#pragma unroll
		for (int n = 0; n < NS; n++) row[n] = z[n];
	}
}

// The coefficients k0, k0 + step, .. of one group: Haar over the members,
// shrinkage, inverse Haar; step 2 leaves w^2 in the basic estimate's rows.
template <int NS, int STEP, int SPC>
__device__ int shrink_rows(float *zt, float *yt, float *ct, int k0, int step, float bs2, float is2, bool oinv, float sigma2,
                           float bm2)
{
	int kept = 0;
#pragma unroll 1
	for (int k = k0; k < SPC; k += step) {
		float *zr = zt + k * kTileP, *yr = yt + k * kTileP;
		float z[NS], y[NS];
		load_row<NS>(zr, z);
		haar_forward<NS>(z, is2);
		if (STEP == 2) {
			load_row<NS>(yr, y);
			haar_forward<NS>(y, is2);
		}
		if (oinv) {
			if (STEP == 1) {
#pragma unroll
				for (int n = 0; n < NS; n++) y[n] = z[n];
			}
			ct[k * kTileP] = shrink_invariant<NS, STEP>(z, y, bs2, sigma2, bm2);
		} else if (STEP == 1) {
#pragma unroll
			for (int n = 0; n < NS; n++) {
				if (__fmul_rn(z[n], z[n]) > bs2 || (k == 0 && n == 0)) kept++;
				else z[n] = 0.f;
			}
		} else {
#pragma unroll
			for (int n = 0; n < NS; n++) {
				const float yy = __fmul_rn(y[n], y[n]);
				const float w = __fdiv_rn(yy, __fadd_rn(yy, bs2));
				z[n] = __fmul_rn(z[n], w);
				y[n] = __fmul_rn(w, w);
			}
			store_row<NS>(yr, y);
		}
		haar_inverse<NS>(z, is2);
		store_row<NS>(zr, z);
	}
	return kept;
}

template <int STEP, int PX, int PT, int L, bool DCT4>
__global__ void __launch_bounds__(32 * kFwWarps, DCT4 ? 3 : 2)
filter_warp_kernel(Image noisy, Image basic, const Tile *__restrict__ tiles, int ntiles, StepParams sp,
                   const float *__restrict__ basis, const float *__restrict__ binv, long long g_begin, long long g_end,
                   int run, const uint8_t *__restrict__ nsimp, const uint32_t *__restrict__ idx,
                   const uint8_t *__restrict__ alive, float *__restrict__ vals, float *__restrict__ wslot,
                   float *__restrict__ wgroup, uint8_t *__restrict__ eq)
{
	constexpr int SPC = PX * PX * PT, SP = (SPC + 3) / 4 * 4, NG = 32 / L, kTile = SPC * kTileP;
	constexpr int RW = PX <= 4 ? 4 : 8, RM = 32 / RW;   // lanes per row of pixels, members staged at once
	extern __shared__ __align__(16) float sm[];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int gi = lane / L, n = lane % L;              // this lane's group and member
	float *Bt = sm;                                     // Bt[p][k] = basis[k][p]   (not DCT4)
	float *Bi = Bt + (DCT4 ? 0 : SPC * SP);             // Bi[k][p] = binv[k][p]
	float *T1 = Bi + (DCT4 ? 0 : SPC * SP) + warp * STEP * kTile, *T2 = STEP == 2 ? T1 + kTile : T1;
	float *ct = T1 + 32 + gi;                           // weight shares (order invariance): the rows' padding
	__shared__ __align__(16) typename std::conditional<DCT4, Dct4Tables, int>::type tab;
	if constexpr (DCT4) {
		tab.fill(sp.dct4, threadIdx.x, blockDim.x);
		__syncthreads();
	} else {
		for (int i = threadIdx.x; i < SPC * SP; i += blockDim.x) {
			const int r = i / SP, q = i % SP;
			Bt[i] = q < SPC ? basis[q * SPC + r] : 0.f;
			Bi[i] = q < SPC ? binv[r * SPC + q] : 0.f;
		}
		__syncthreads();
	}
	const int C = sp.C, np = sp.np;
	const float sigma2 = __fmul_rn(sp.sigma, sp.sigma);
	const float bsig = __fmul_rn(sp.beta, sp.sigma);
	const float bs2 = __fmul_rn(bsig, bsig);
	const float bmsig = __fmul_rn(sp.beta_mean, sp.sigma);
	const float bm2 = __fmul_rn(bmsig, bmsig);
	const bool oinv = sp.order_inv != 0;
	const float is2 = (float)(1.0 / sqrt(2.0));
	const unsigned mygroup = (L == 32 ? 0xffffffffu : (1u << L) - 1u) << (gi * L);

	// runs of consecutive groups; the warp takes NG processed ones at a time
	for (long long r0 = g_begin + ((long long)blockIdx.x * kFwWarps + warp) * run; r0 < g_end;
	     r0 += (long long)gridDim.x * kFwWarps * run) {
		unsigned todo = __ballot_sync(0xffffffffu, lane < run && r0 + lane < g_end && alive[r0 + lane]);
		while (todo) {
			// group gi is the gi-th of the next set bits
			unsigned bits = todo;
			for (int i = 0; i < gi; i++) bits &= bits - 1;
			bool on = bits != 0u;
			const long long g = r0 + (on ? __ffs(bits) - 1 : __ffs(todo) - 1);
#pragma unroll
			for (int i = 0; i < NG; i++) todo &= todo - 1;
			const int ns = nsimp[g];
			const Tile T = tiles[tile_of(tiles, ntiles, g)];
			const long long slot0 = (g - g_begin) * np;
			size_t base;       // the member's first pixel in its video
			{
				const uint32_t lin = idx[g * np + (n < ns ? n : 0)], whl = (uint32_t)T.w * T.h;
				base = noisy.at(T.ox + (int)(lin % T.w), T.oy + (int)((lin % whl) / T.w), (int)(lin / whl), 0);
			}
			// all-equal test (nldct.cpp:1986-1999, 2222-2235): decided by the first
			// element as a rule
			{
				const float v = __ldg(noisy.p + base);
				// (shuffles and ballots outside the conditions: every lane takes part)
				const float v0 = __shfl_sync(0xffffffffu, v, gi * L);
				bool differs = n < ns && v != v0;
				unsigned any = __ballot_sync(0xffffffffu, differs) & mygroup;
				bool maybe = on && ns > 1 && any == 0u;
				if (__any_sync(0xffffffffu, maybe)) {
					for (int i = 0; i < C * SPC; i++) {
						const int c = i / SPC, p = i % SPC;
						const size_t at = noisy.at(p % PX, p / PX % PX, p / (PX * PX), c);
						const float u = __ldg(noisy.p + base + at);
						const float u0 = __shfl_sync(0xffffffffu, u, gi * L);
						differs |= n < ns && u != u0;
					}
					any = __ballot_sync(0xffffffffu, differs) & mygroup;
					maybe = maybe && any == 0u;
					if (maybe) {
						// left as it is; its weights are set later (fixup_equal_kernel)
						for (int i = 0; i < C * SPC && n < ns; i++) {
							const int c = i / SPC, p = i % SPC;
							vals[((slot0 + n) * C + c) * SPC + term_of(PX, PT, p)] =
							    __ldg(noisy.p + base + noisy.at(p % PX, p / PX % PX, p / (PX * PX), c));
						}
						if (n == 0) eq[g] = 1;
						on = false;
					}
					if (!__any_sync(0xffffffffu, on)) continue;
				}
			}
			const bool full = __all_sync(0xffffffffu, ns == L) && !oinv;
			int kept = 0;
			float wsum = 0.f;
			for (int c = 0; c < C; c++) {
				__syncwarp();
				// stage the members' pixels, RM members' rows at a time
#pragma unroll
				for (int m0 = 0; m0 < 32; m0 += RM) {
					const int m = m0 + lane / RW, hx = lane % RW;
					const size_t mb = __shfl_sync(0xffffffffu, (unsigned long long)base, m) + (size_t)c * noisy.plane() + hx;
					if (hx < PX) {
						float v[PX * PT];
#pragma unroll
						for (int r = 0; r < PX * PT; r++)
							v[r] = __ldg(noisy.p + mb + (size_t)(r / PX) * noisy.plane() * C + (size_t)(r % PX) * noisy.P);
#pragma unroll
						for (int r = 0; r < PX * PT; r++) T1[(r * PX + hx) * kTileP + m] = v[r];
						if (STEP == 2) {
#pragma unroll
							for (int r = 0; r < PX * PT; r++)
								v[r] = __ldg(basic.p + mb + (size_t)(r / PX) * noisy.plane() * C + (size_t)(r % PX) * noisy.P);
#pragma unroll
							for (int r = 0; r < PX * PT; r++) T2[(r * PX + hx) * kTileP + m] = v[r];
						}
					}
				}
				__syncwarp();
				float o[64];
#pragma unroll 1
				for (int b = 0; b < STEP; b++) {
					float *col = (b ? T2 : T1) + lane;
					if constexpr (DCT4) dct4_forward(col, tab, o);
					else dense_product<SPC, SP>(col, Bt, o, [](int) {});
#pragma unroll
					for (int k = 0; k < SPC; k++) col[k * kTileP] = o[k];
				}
				__syncwarp();
				{
					float *zt = T1 + gi * L, *yt = T2 + gi * L;
#define ROWS(N) kept += shrink_rows<N, STEP, SPC>(zt, yt, ct, n, L, bs2, is2, oinv, sigma2, bm2)
					switch (ns) {
					case 1: ROWS(1); break;
					case 2: ROWS(2); break;
					case 4: ROWS(4); break;
					case 8: ROWS(8); break;
					case 16: if constexpr (L >= 16) ROWS(16); break;
					default: if constexpr (L >= 32) ROWS(32); break;
					}
#undef ROWS
				}
				__syncwarp();
				if (oinv) {
					// float sum of the coefficients' shares in (c, k) order
					for (int k = 0; k < SPC; k++) wsum = __fadd_rn(wsum, ct[k * kTileP]);
				} else if (STEP == 2 && !full) {
					// sum of w^2 in the reference's (c, k, n) order
					const float *yt = T2 + gi * L;
					for (int k = 0; k < SPC; k++)
						for (int i = 0; i < ns; i++) wsum = __fadd_rn(wsum, yt[k * kTileP + i]);
				}
				__syncwarp();
				const auto inverse = [&](auto also) {
					if constexpr (DCT4) dct4_inverse(T1 + lane, tab, o, also);
					else dense_product<SPC, SP>(T1 + lane, Bi, o, also);
				};
				if (STEP == 2 && full) {
					// the same sum for whole groups, beside the inverse transform: a chain
					// of SPC * L dependent adds that would stall the warp by itself
					inverse([&](int k) {
						const float *row = T2 + gi * L + k * kTileP;
#pragma unroll
						for (int i = 0; i < L; i += 4) {
							const float4 q = *reinterpret_cast<const float4 *>(row + i);
							wsum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(wsum, q.x), q.y), q.z), q.w);
						}
					});
				} else {
					inverse([](int) {});
				}
				if (on && n < ns) {
					float *to = vals + ((slot0 + n) * C + c) * SPC;
					if constexpr (SPC % 8 == 0) {
#pragma unroll
						for (int p = 0; p < SPC; p += 8) {
							// element order of term_of: for 4x4 patches columns of rows
							float e[8];
#pragma unroll
							for (int i = 0; i < 8; i++) {
								const int q = p + i;
								e[i] = o[PX == 4 ? (q & ~15) | (q & 3) << 2 | (q >> 2 & 3) : q];
							}
							asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to + p), "f"(e[0]),
							             "f"(e[1]), "f"(e[2]), "f"(e[3]), "f"(e[4]), "f"(e[5]), "f"(e[6]), "f"(e[7])
							             : "memory");
						}
					} else {
#pragma unroll
						for (int p = 0; p < SPC; p++) to[p] = o[p];
					}
				}
			}
			// the group's weight
#pragma unroll
			for (int s = L / 2; s > 0; s >>= 1) kept += __shfl_xor_sync(0xffffffffu, kept, s);
			float w;
			if (STEP == 1) w = __fdiv_rn(__fdiv_rn(1.f, sigma2), oinv ? wsum : (float)kept);
			else w = (float)(1.0 / (double)sigma2 / (double)wsum);
			if (on && n < ns) wslot[slot0 + n] = w;
			if (on && n == 0) { wgroup[g] = w; eq[g] = 0; }
		}
	}
}
// Groups whose members are all equal keep the aggregation weights left by the
// previous processed groups of their tile (the reference's aggreWeights vector
// is not rewritten, nldct.cpp:1998, 2234): member n takes the weight of the
// latest earlier group with more than n members, or 1 if there is none
// (its initial value, nldct.cpp:754, 824).
__global__ void fixup_equal_kernel(const Tile *__restrict__ tiles, int ntiles, StepParams sp,
                                   long long g_begin, long long g_end,
                                   const uint8_t *__restrict__ nsimp, const uint8_t *__restrict__ alive,
                                   const uint8_t *__restrict__ eq, const float *__restrict__ wgroup,
                                   float *__restrict__ wslot)
{
	for (long long g = g_begin + blockIdx.x * (long long)blockDim.x + threadIdx.x; g < g_end;
	     g += (long long)gridDim.x * blockDim.x) {
		if (!alive[g] || !eq[g]) continue;
		const Tile T = tiles[tile_of(tiles, ntiles, g)];
		const int ns = nsimp[g];
		const long long slot0 = (g - g_begin) * sp.np;
		// the group for member n + 1 is the one for member n or lies before it: one walk
		// back serves them all (flat 854x480x8: 1580 -> 107 ms of filter, 39 -> 2.7 s on
		// a flat 1280x720x16, where the walk goes back to the first group)
		long long q = g;
		int members = 0;     // of group q
		float w = 1.f;
		for (int n = 0; n < ns; n++) {
			while (members <= n && q > T.g0) {
				q--;
				if (alive[q] && !eq[q] && nsimp[q] > n) {
					members = nsimp[q];
					w = wgroup[q];
				}
			}
			wslot[slot0 + n] = members > n ? w : 1.f;
		}
	}
}

}  // namespace

size_t filter_smem_bytes(const StepParams &sp)
{
	const int nsp = ((sp.np + 3) / 4) * 4 + 4;
	const size_t tile_f = (size_t)sp.C * sp.spc * nsp;
	const size_t bsz = ((size_t)sp.spc * sp.spc + 3) / 4 * 4;
	return sizeof(float) * (2 * bsz + 4 * tile_f);
}

namespace {

struct FilterArgs {
	const Image &noisy, &basic;
	const Tile *tiles;
	int ntiles;
	const StepParams &sp;
	const float *basis, *binv;
	long long g_begin, g_end;
	const uint8_t *nsimp;
	const uint32_t *idx;
	const uint8_t *alive;
	float *vals, *wslot, *wgroup;
	uint8_t *eq;
	int nsm;
	cudaStream_t st;
};

template <int STEP>
cudaError_t launch_exact(const FilterArgs &a)
{
	auto kern = filter_exact_kernel<STEP>;
	const size_t smem = filter_smem_bytes(a.sp);
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e != cudaSuccess) return e;
	const int blocks = (int)std::min<long long>(a.g_end - a.g_begin, (long long)a.nsm * 8);
	kern<<<blocks, kFilterThreads, smem, a.st>>>(a.noisy, a.basic, a.tiles, a.ntiles, a.sp, a.basis, a.binv, a.g_begin,
	                                            a.g_end, a.nsimp, a.idx, a.alive, a.vals, a.wslot, a.wgroup, a.eq);
	return cudaGetLastError();
}

template <int STEP, int PX, int PT, int L, bool DCT4>
cudaError_t launch_warp_t(const FilterArgs &a)
{
	auto kern = filter_warp_kernel<STEP, PX, PT, L, DCT4>;
	constexpr int SPC = PX * PX * PT, SP = (SPC + 3) / 4 * 4, NG = 32 / L;
	const size_t smem = sizeof(float) * ((DCT4 ? 0 : 2 * SPC * SP) + kFwWarps * STEP * SPC * kTileP);
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e != cudaSuccess) return e;
	int per_sm = 0;
	e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kFwWarps, smem);
	if (e != cudaSuccess) return e;
	// runs of up to 32 groups per warp (the processed ones are packed), shorter
	// where that would leave warps idle
	const long long n = a.g_end - a.g_begin, warps = (long long)a.nsm * std::max(per_sm, 1) * kFwWarps;
	const int run = (int)std::min<long long>(32, (n + warps * NG - 1) / (warps * NG) * NG);
	const long long need = (n + (long long)run * kFwWarps - 1) / ((long long)run * kFwWarps);
	const int blocks = (int)std::min<long long>(need, (long long)a.nsm * std::max(per_sm, 1));
	kern<<<blocks, 32 * kFwWarps, smem, a.st>>>(a.noisy, a.basic, a.tiles, a.ntiles, a.sp, a.basis, a.binv, a.g_begin,
	                                           a.g_end, run, a.nsimp, a.idx, a.alive, a.vals, a.wslot, a.wgroup, a.eq);
	return cudaGetLastError();
}

// L lanes per group: the largest power of two up to nSimilarPatches (a group
// never has more members), at least 8.
template <int PX, int PT, bool DCT4>
cudaError_t launch_warp(const FilterArgs &a)
{
	const int np = a.sp.np;
	if (a.sp.step1)
		return np >= 32 ? launch_warp_t<1, PX, PT, 32, DCT4>(a)
		                : np >= 16 ? launch_warp_t<1, PX, PT, 16, DCT4>(a) : launch_warp_t<1, PX, PT, 8, DCT4>(a);
	return np >= 32 ? launch_warp_t<2, PX, PT, 32, DCT4>(a)
	                : np >= 16 ? launch_warp_t<2, PX, PT, 16, DCT4>(a) : launch_warp_t<2, PX, PT, 8, DCT4>(a);
}

}  // namespace

cudaError_t launch_filter(const Image &noisy, const Image &basic, const Tile *tiles, int ntiles,
                          const StepParams &sp, const float *basis, const float *binv,
                          long long g_begin, long long g_end,
                          const uint8_t *nsimp, const uint32_t *idx, const uint8_t *alive,
                          float *vals, float *wslot, float *wgroup, uint8_t *eq, int nsm,
                          cudaStream_t st)
{
	if (g_end <= g_begin) return cudaSuccess;
	const FilterArgs a = {noisy, basic, tiles, ntiles, sp,    basis,  binv, g_begin, g_end,
	                      nsimp, idx,   alive, vals,   wslot, wgroup, eq,   nsm,     st};
	cudaError_t e;
	if (sp.px == 4 && sp.pt == 4 && sp.dct4[0] > 0.f) e = launch_warp<4, 4, true>(a);
	else if (sp.px == 8 && sp.pt == 1) e = launch_warp<8, 1, false>(a);
	else if (sp.px == 7 && sp.pt == 1) e = launch_warp<7, 1, false>(a);
	else e = sp.step1 ? launch_exact<1>(a) : launch_exact<2>(a);
	if (e != cudaSuccess) return e;
	const long long n = g_end - g_begin;
	const int fb = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
	fixup_equal_kernel<<<fb, 256, 0, st>>>(tiles, ntiles, sp, g_begin, g_end, nsimp, alive, eq, wgroup, wslot);
	return cudaGetLastError();
}

}  // namespace bm4dof
