// tvl1.cu -- TV-L1 optical flow (Zach, Pock and Bischof's dual method) on the
// GPU, batched over frame pairs.  It produces the flows the denoiser takes as
// input, the step the reference runs before its path (lib/tvl1flow, driven by
// scripts/tvl1flow-seq.sh).
//
// Restates, with the same float/double arithmetic (except |grad u| of the dual
// update, taken in float instead of the reference's double hypot):
//   tvl1flow_lib.c   image_normalization (299-336), Dual_TVL1_optic_flow
//                    (93-263), Dual_TVL1_optic_flow_multiscale (344-474);
//   mask.c           divergence (40-88), forward_gradient (96-139),
//                    centered_gradient (147-203), gaussian (211-333, the
//                    reflecting boundary);
//   zoom.c           zoom_size (24-35), zoom_out (42-77), zoom_in (84-112);
//   bicubic_interpolation.c  bicubic_interpolation_at (141-232, Neumann
//                    boundary, including its use of sx for the row above),
//                    bicubic_interpolation_warp (239-262);
//   main.c           the number of scales (147-153).
//
// Layout: every array is [pair][y][x] at its pyramid level.  Each frame pair
// is one unit of the batch; all pairs of a video go in one call, and a pair and
// the same pair backwards share the normalised images, their smoothing and
// their pyramids.
//
// FP64 runs at 1/64 of the FP32 rate here, so the reference's double sums
// (Gaussian, bicubic cells, normalisation) are formed in pairs of floats with
// an error bound; where the bound leaves the rounding to float open (about one
// value in 2^10 to 2^16) the value is formed again in double.  The results are
// those of the double code bit for bit.
//
// The fixed-point iterations of one level run in one cooperative launch with
// the state of each tile in shared memory and registers (level_kernel); a level
// whose pairs do not fit on the chip runs from L2 (iterate_kernel).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "divide.hpp"
#include "internal.hpp"

namespace cg = cooperative_groups;

namespace bm4dof {

namespace {

constexpr int kMaxIterations = 300;         // tvl1flow_lib.c:23
constexpr double kPresmoothSigma = 0.8;     // tvl1flow_lib.c:24
constexpr float kGradIsZero = 1e-10f;       // tvl1flow_lib.c:25
constexpr float kZoomSigmaZero = 0.6f;      // zoom.c:16
constexpr int kGaussWindow = 5;             // mask.c:23
constexpr int kMaxGauss = 64;               // taps passed with the launch

// ---- pairs of floats (Knuth's and Dekker's exact sum and product) ----------------
struct Pair { float h, l; };

__device__ __forceinline__ Pair two_sum(float a, float b)
{
	const float s = a + b, t = s - a;
	return {s, (a - (s - t)) + (b - t)};
}

__device__ __forceinline__ Pair two_prod(float a, float b)
{
	const float p = a * b;
	return {p, __fmaf_rn(a, b, -p)};
}

// acc + p (a pair), the low parts summed in float
__device__ __forceinline__ void add_pair(Pair &acc, Pair p)
{
	const Pair s = two_sum(acc.h, p.h);
	acc.h = s.h;
	acc.l += s.l + p.l;
}

// acc.h + acc.l rounded to float when every number within e of it rounds alike
// (also false for NaN)
__device__ __forceinline__ bool rounds(Pair acc, float e, float &r)
{
	r = acc.h + (acc.l + e);
	return r == acc.h + (acc.l - e);
}

// ---- bicubic interpolation (bicubic_interpolation.c) ---------------------------
__device__ __forceinline__ int neumann(int x, int n, bool &out)
{
	if (x < 0) { out = true; return 0; }
	if (x >= n) { out = true; return n - 1; }
	return x;
}

__device__ __forceinline__ double cubic_cell(const double v[4], double x)
{
	return v[1] + 0.5 * x * (v[2] - v[0] + x * (2.0 * v[0] - 5.0 * v[1] + 4.0 * v[2] - v[3] +
	                                            x * (3.0 * (v[1] - v[2]) + v[3] - v[0])));
}

struct Cell {
	int xs[4], ys[4];
	float x, y;     // position within the cell
	bool out;
};

__device__ __forceinline__ Cell cell_of(float uu, float vv, int nx, int ny)
{
	Cell c;
	const int sx = uu < 0 ? -1 : 1;
	const int sy = vv < 0 ? -1 : 1;
	c.out = false;
	c.xs[1] = neumann((int)uu, nx, c.out);
	c.ys[1] = neumann((int)vv, ny, c.out);
	c.xs[0] = neumann((int)uu - sx, nx, c.out);
	c.ys[0] = neumann((int)vv - sx, ny, c.out);   // sx, as the reference has it
	c.xs[2] = neumann((int)uu + sx, nx, c.out);
	c.ys[2] = neumann((int)vv + sy, ny, c.out);
	c.xs[3] = neumann((int)uu + 2 * sx, nx, c.out);
	c.ys[3] = neumann((int)vv + 2 * sy, ny, c.out);
	c.x = uu - c.xs[1];
	c.y = vv - c.ys[1];
	return c;
}

__device__ __noinline__ float bicubic_double(const float *in, const Cell &c, int nx)
{
	double v[4];
	for (int a = 0; a < 4; a++) {
		double col[4];
		for (int b = 0; b < 4; b++) col[b] = (double)in[c.xs[a] + nx * c.ys[b]];
		v[a] = cubic_cell(col, (double)c.y);
	}
	return (float)cubic_cell(v, (double)c.x);
}

// The four weights of cubic_cell at x in [0, 1], each to 2^-45:
//   -x/2 + x^2 - x^3/2,  1 - 5x^2/2 + 3x^3/2,  x/2 + 2x^2 - 3x^3/2,  (x^3 - x^2)/2
__device__ __forceinline__ void cubic_weights(float x, Pair w[4])
{
	const Pair x2 = two_prod(x, x);
	Pair x3 = two_prod(x2.h, x);
	x3.l = __fmaf_rn(x2.l, x, x3.l);
	Pair a = two_prod(2.5f, x2.h), b = two_prod(1.5f, x3.h);
	a.l = __fmaf_rn(2.5f, x2.l, a.l);
	b.l = __fmaf_rn(1.5f, x3.l, b.l);
	w[0] = x2;
	add_pair(w[0], {-0.5f * x, 0.f});
	add_pair(w[0], {-0.5f * x3.h, -0.5f * x3.l});
	w[1] = {1.f, 0.f};
	add_pair(w[1], {-a.h, -a.l});
	add_pair(w[1], b);
	w[2] = {2.f * x2.h, 2.f * x2.l};
	add_pair(w[2], {0.5f * x, 0.f});
	add_pair(w[2], {-b.h, -b.l});
	w[3] = {0.5f * x3.h, 0.5f * x3.l};
	add_pair(w[3], {-0.5f * x2.h, -0.5f * x2.l});
#pragma unroll
	for (int k = 0; k < 4; k++) {
		const float h = w[k].h + w[k].l;
		w[k].l -= h - w[k].h;
		w[k].h = h;
	}
}

// The bicubic value in pairs of floats.  With M the largest of the 16 pixels
// and both weight sums at most 1.25, the weights' errors give 2^-41.7 M and the
// rounded low parts of the two levels of sums 2 x 2^-42.5 M, together less than
// 2^-40 M.  The products' low parts are exact for M from 1e-20 to 1e30.
// About 240 FP32 operations a value, and 70 for each axis' weights, in place of
// 65 of the FP64 pipe and 16 conversions on it: the zoom of 18 flows from
// 320x180 to 640x360 took 1677 us in double and takes 153 us.
__device__ __forceinline__ float bicubic_value(const float *in, const Cell &c, const Pair wx[4], const Pair wy[4],
                                               bool fast, int nx)
{
	if (fast) {
		Pair acc = {0.f, 0.f};
		float M = 0.f;
#pragma unroll
		for (int b = 0; b < 4; b++) {
			const float *row = in + nx * c.ys[b];
			Pair s = {0.f, 0.f};
#pragma unroll
			for (int a = 0; a < 4; a++) {
				const float v = row[c.xs[a]];
				M = fmaxf(M, fabsf(v));
				Pair p = two_prod(wx[a].h, v);
				p.l = __fmaf_rn(wx[a].l, v, p.l);
				if (a == 0) s = p;
				else add_pair(s, p);
			}
			Pair p = two_prod(wy[b].h, s.h);
			p.l = __fmaf_rn(wy[b].l, s.h, __fmaf_rn(wy[b].h, s.l, p.l));
			add_pair(acc, p);
		}
		float r;
		if (M <= 1e30f && (M >= 1e-20f || M == 0.f)) {
			if (rounds(acc, 0x1p-40f * M, r)) return r;
			// Halfway positions give halves of a unit often (a zoom by 2: one value
			// in 32).  Their weights are sixteenths, and with all pixels within 2^8
			// of each other every low part is a multiple of 2^-8 units of the
			// smallest below 2^21 of them: pairs and doubles are both exact.
			if (2.f * c.x == floorf(2.f * c.x) && 2.f * c.y == floorf(2.f * c.y)) {
				float mn = M;
#pragma unroll
				for (int k = 0; k < 16; k++) {
					const float v = fabsf(in[c.xs[k % 4] + nx * c.ys[k / 4]]);
					if (v != 0.f) mn = fminf(mn, v);
				}
				if (mn * 256.f >= M) return acc.h + acc.l;
			}
		}
	}
	return bicubic_double(in, c, nx);
}

__device__ __forceinline__ bool in_cell(const Cell &c) { return c.x >= 0.f && c.x <= 1.f && c.y >= 0.f && c.y <= 1.f; }

// the three warped values of one pixel, 0 outside the image
__device__ __noinline__ float3 warp_at(const float *I1, const float *I1x, const float *I1y, float uu, float vv, int nx,
                                       int ny)
{
	const Cell c = cell_of(uu, vv, nx, ny);
	if (c.out) return make_float3(0.f, 0.f, 0.f);
	Pair wx[4], wy[4];
	cubic_weights(c.x, wx);
	cubic_weights(c.y, wy);
	const bool fast = in_cell(c);
	float3 r;
	r.x = bicubic_value(I1, c, wx, wy, fast, nx);
	r.y = bicubic_value(I1x, c, wx, wy, fast, nx);
	r.z = bicubic_value(I1y, c, wx, wy, fast, nx);
	return r;
}

// ---- per-pixel stencils of mask.c ------------------------------------------------
__device__ __forceinline__ float divergence_at(const float *v1, const float *v2, int i, int j, int nx, int ny)
{
	const int p = i * nx + j;
	const bool top = i == 0, bot = i == ny - 1, lef = j == 0, rig = j == nx - 1;
	if (!top && !bot && !lef && !rig) return (v1[p] - v1[p - 1]) + (v2[p] - v2[p - nx]);
	if (top && lef) return v1[0] + v2[0];
	if (top && rig) return -v1[nx - 2] + v2[nx - 1];
	if (bot && lef) return v1[p] - v2[p - nx];
	if (bot && rig) return -v1[p - 1] - v2[p - nx];
	if (top) return v1[j] - v1[j - 1] + v2[j];
	if (bot) return v1[p] - v1[p - 1] - v2[p - nx];
	if (lef) return v1[p] + v2[p] - v2[p - nx];
	return -v1[p - 1] + v2[p] - v2[p - nx];   // right column
}

__device__ __forceinline__ void forward_gradient_at(const float *f, int i, int j, int nx, int ny, float &fx,
                                                    float &fy)
{
	const int p = i * nx + j;
	fx = j < nx - 1 ? f[p + 1] - f[p] : 0.f;
	fy = i < ny - 1 ? f[p + nx] - f[p] : 0.f;
}

// ---- kernels ---------------------------------------------------------------------
// the smallest and largest value of every image, by parts: part[image][gridDim.x][2]
__global__ void __launch_bounds__(256) minmax_kernel(const float *__restrict__ I0, const float *__restrict__ I1,
                                                     int n, int size, float *__restrict__ part)
{
	const int img = blockIdx.y;
	const float *a = (img < n ? I0 + (size_t)img * size : I1 + (size_t)(img - n) * size);
	__shared__ float s[2][8];
	float mn = a[0], mx = a[0];
	for (long long i = blockIdx.x * 256 + threadIdx.x; i < size; i += 256 * gridDim.x) {
		mn = fminf(mn, a[i]);
		mx = fmaxf(mx, a[i]);
	}
	for (int d = 16; d; d >>= 1) {
		mn = fminf(mn, __shfl_xor_sync(~0u, mn, d));
		mx = fmaxf(mx, __shfl_xor_sync(~0u, mx, d));
	}
	if (threadIdx.x % 32 == 0) {
		s[0][threadIdx.x / 32] = mn;
		s[1][threadIdx.x / 32] = mx;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int k = 1; k < 8; k++) {
			mn = fminf(mn, s[0][k]);
			mx = fmaxf(mx, s[1][k]);
		}
		part[((size_t)img * gridDim.x + blockIdx.x) * 2] = mn;
		part[((size_t)img * gridDim.x + blockIdx.x) * 2 + 1] = mx;
	}
}

// 255 (I - min) / (max - min) of both images of every pair, min and max over
// both; O holds the n first images and then the n second ones.
// The reference divides 255 d, exact in double, by den in double and rounds to
// float.  The pair p is that product; the quotient's correction c comes from a
// remainder good to 2^-24 of one and a half units of q, so q + c is good to
// 2^-43 q.
__global__ void __launch_bounds__(256) normalize_kernel(const float *__restrict__ I0, const float *__restrict__ I1,
                                                        int n, int size, const float *__restrict__ part, int parts,
                                                        float *__restrict__ O)
{
	const int img = blockIdx.y, pair = img < n ? img : img - n;
	const float *a = (img < n ? I0 : I1) + (size_t)pair * size;
	const float *p0 = part + (size_t)pair * parts * 2, *p1 = part + (size_t)(n + pair) * parts * 2;
	float mn0 = p0[0], mx0 = p0[1], mn1 = p1[0], mx1 = p1[1];
	for (int k = 1; k < parts; k++) {
		mn0 = fminf(mn0, p0[2 * k]);
		mx0 = fmaxf(mx0, p0[2 * k + 1]);
		mn1 = fminf(mn1, p1[2 * k]);
		mx1 = fmaxf(mx1, p1[2 * k + 1]);
	}
	const float mx = mx0 > mx1 ? mx0 : mx1;
	const float mn = mn0 < mn1 ? mn0 : mn1;
	const float den = mx - mn;
	float *o = O + (size_t)img * size;
	const bool scaled = den > 0x1p-30f && den < 0x1p60f;
	const float y = scaled ? __frcp_rn(den) : 0.f;
	for (long long i = blockIdx.x * 256 + threadIdx.x; i < size; i += 256 * gridDim.x) {
		const float v = a[i];
		if (!(den > 0)) {
			o[i] = v;
			continue;
		}
		const float d = v - mn;
		const Pair p = two_prod(255.f, d);
		const float q = p.h * y;
		const float c = (__fmaf_rn(-den, q, p.h) + p.l) * y;
		float r;
		if (!(scaled && (q > 0x1p-60f || d == 0.f) && rounds({q, c}, 0x1p-43f * q, r)))
			r = (float)(255.0 * (double)d / (double)den);
		o[i] = r;
	}
}

struct Gauss {
	double d[kMaxGauss];
	float h[kMaxGauss], l[kMaxGauss];   // d as a pair of floats
	float e;                            // error bound of the pairs' sum, over the largest pixel
	int taps;
};

// one pass of the separable Gaussian with the reflecting boundary of mask.c
// (rows: step 1 along x; columns: along y).  The sum of the pairs: every low
// part is below (taps + 2) 2^-24 M and is rounded twice a tap.  18 images of
// 640x360, 11 taps: 42 us a pass (109 us for as many in double).
template <int ALONG_Y>
__global__ void __launch_bounds__(256) gauss_pass_kernel(const float *__restrict__ in, float *__restrict__ out, int nx,
                                                         int ny, __grid_constant__ const Gauss g)
{
	const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
	if (x >= nx || y >= ny) return;
	const size_t base = (size_t)blockIdx.z * nx * ny;
	const int n = ALONG_Y ? ny : nx, pos = ALONG_Y ? y : x, step = ALONG_Y ? nx : 1;
	const float *line = in + base + (ALONG_Y ? x : y * nx);
	auto at = [&](int m) {
		if (m < 0) m = -m;
		else if (m >= n) m = n - (m - n) - 1;
		return line[m * step];
	};
	const float v = at(pos);
	float M = fabsf(v);
	Pair acc = two_prod(g.h[0], v);
	acc.l = __fmaf_rn(g.l[0], v, acc.l);
	for (int j = 1; j < g.taps; j++) {
		const float a = at(pos - j), b = at(pos + j);
		M = fmaxf(M, fmaxf(fabsf(a), fabsf(b)));
		const Pair s = two_sum(a, b);
		Pair p = two_prod(g.h[j], s.h);
		p.l = __fmaf_rn(g.l[j], s.h, __fmaf_rn(g.h[j], s.l, p.l));
		add_pair(acc, p);
	}
	float r;
	if (!(rounds(acc, g.e * M, r) && M <= 1e30f && (M >= 1e-20f || M == 0.f))) {
		double sum = g.d[0] * (double)v;
		for (int j = 1; j < g.taps; j++) sum += g.d[j] * ((double)at(pos - j) + (double)at(pos + j));
		r = (float)sum;
	}
	out[base + (size_t)y * nx + x] = r;
}

// zoom_out's resampling (after the smoothing) and zoom_in, with an optional
// scale of the values (the flow's 1/zfactor), of two planes at once: plane z
// of in0 and of in1
__global__ void __launch_bounds__(256) resample_kernel(const float *__restrict__ in0, const float *__restrict__ in1,
                                                       int nx, int ny, float *__restrict__ out0,
                                                       float *__restrict__ out1, int nxx, int nyy, float fx, float fy,
                                                       float scale, int use_scale)
{
	const int j1 = blockIdx.x * 32 + threadIdx.x, i1 = blockIdx.y * 8 + threadIdx.y;
	if (j1 >= nxx || i1 >= nyy) return;
	const Cell c = cell_of((float)j1 / fx, (float)i1 / fy, nx, ny);
	Pair wx[4], wy[4];
	cubic_weights(c.x, wx);
	cubic_weights(c.y, wy);
	const bool fast = in_cell(c);
	const size_t src = (size_t)blockIdx.z * nx * ny, dst = (size_t)blockIdx.z * nxx * nyy + (size_t)i1 * nxx + j1;
	float a = bicubic_value(in0 + src, c, wx, wy, fast, nx);
	float b = bicubic_value(in1 + src, c, wx, wy, fast, nx);
	if (use_scale) {
		a *= scale;
		b *= scale;
	}
	out0[dst] = a;
	out1[dst] = b;
}

__global__ void __launch_bounds__(256) centered_gradient_kernel(const float *__restrict__ in, float *__restrict__ dx,
                                                                float *__restrict__ dy, int nx, int ny)
{
	const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 8 + threadIdx.y;
	if (j >= nx || i >= ny) return;
	const size_t base = (size_t)blockIdx.z * nx * ny;
	const float *f = in + base;
	const int k = i * nx + j;
	const int l = j > 0 ? k - 1 : k, r = j < nx - 1 ? k + 1 : k;
	const int u = i > 0 ? k - nx : k, d = i < ny - 1 ? k + nx : k;
	dx[base + k] = 0.5f * (f[r] - f[l]);
	dy[base + k] = 0.5f * (f[d] - f[u]);
}

// The images of a level.  Pair k < m takes first[k] to second[k]; pair m + k,
// where there is one, is pair k backwards.  The gradients are those of second,
// and where pairs go backwards too, those of first before them.
struct LevelImages {
	const float *first, *second, *gx, *gy;
	int m, mirrored, nx, ny;
	__device__ const float *i0(int pair) const { return at(pair < m ? first : second, pair); }
	__device__ const float *i1(int pair) const { return at(pair < m ? second : first, pair); }
	__device__ size_t grad(int pair) const
	{
		return (size_t)(!mirrored ? pair : pair < m ? m + pair : pair - m) * nx * ny;
	}
	__device__ const float *at(const float *p, int pair) const
	{
		return p + (size_t)(pair < m ? pair : pair - m) * nx * ny;
	}
};

// The fixed-point update of u at one pixel (tvl1flow_lib.c:176-218): v1, v2
// before the divergence is added.
__device__ __forceinline__ void threshold(float wx, float wy, float g, float rho, float l_t, float &d1, float &d2)
{
	if (rho < -l_t * g) {
		d1 = l_t * wx;
		d2 = l_t * wy;
	} else if (rho > l_t * g) {
		d1 = -l_t * wx;
		d2 = -l_t * wy;
	} else if (g < kGradIsZero) {
		d1 = d2 = 0.f;
	} else {
		const float fi = -rho / g;
		d1 = fi * wx;
		d2 = fi * wy;
	}
}

// ---- one level with its state on the chip ------------------------------------------
struct LevelArgs {
	LevelImages im;
	float *u1, *u2;          // [pair][y][x]
	float *ring;             // [2][4][pair][y][x], tile borders only: p11, p12, p21, p22
	float *partial;          // [2][gridDim.x]
	unsigned *arrived;       // [pair], zero at the launch
	int *error;
	size_t plane;            // floats of one of the eight planes of ring
	int pair0, tw, th, ntx, tiles, warps;
	float tau, lambda, theta, eps2;
};

constexpr int kTileW = 32, kPitch = kTileW + 2;
constexpr int kMaxPolls = 1 << 22;   // a barrier's limit, about 2 s

constexpr size_t level_smem(int ppt) { return sizeof(float) * 6 * kPitch * (8 * ppt + 2); }

__device__ __forceinline__ unsigned load_acquire(const unsigned *p)
{
	unsigned v;
	asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}

// All warping steps of one level for gridDim.x / tiles pairs, a block a tile of
// up to 32 x 8 PPT pixels (tvl1flow_lib.c:123-246).
//
// What bounds it: the iterations, each a few hundred thousand pixels of about
// 150 instructions between two exchanges with the neighbours.  Run from L2 the
// state is 96 bytes a pixel and iteration and three grid barriers; here u and p
// stay in shared memory, the constants of the warping step in registers, and an
// iteration has one barrier among the blocks of the pair.  A block updates u
// also on the column right of its tile and the row below it (from the same
// numbers as their owner), so that only the border of p is exchanged, in two
// buffers by turns: a block that writes one has passed the barrier after which
// all have read it.  A pair that has converged leaves the others running.
// 18 pairs of 320x180, five warping steps: 5325 us (2235 iterating, 3090
// warping) from L2, 1600 us here, with 52 % of the issue slots; at 160x90 and
// below (2140 us before, 870 us now) the barriers' and exchanges' latency.
//
// The sums are formed per thread, warp, block and then over the pair's tiles in
// one order, the same in every block, so all decide alike.
template <int PPT>
__global__ void __launch_bounds__(256, 4) level_kernel(__grid_constant__ const LevelArgs a)
{
	extern __shared__ float sm[];
	__shared__ float s_red[8], s_err;
	__shared__ int s_fail;
	constexpr int kSize = kPitch * (8 * PPT + 2);
	float *const U1 = sm, *const U2 = sm + kSize, *const P11 = sm + 2 * kSize, *const P12 = sm + 3 * kSize,
	      *const P21 = sm + 4 * kSize, *const P22 = sm + 5 * kSize;
	const int nx = a.im.nx, ny = a.im.ny, size = nx * ny;
	const int pair = a.pair0 + blockIdx.x / a.tiles, tile = blockIdx.x % a.tiles;
	const int x0 = tile % a.ntx * a.tw, y0 = tile / a.ntx * a.th;
	const int W = min(a.tw, nx - x0), H = min(a.th, ny - y0);
	const int t = threadIdx.x, lane = t % 32, warp = t / 32;
	const bool right = x0 + W < nx, below = y0 + H < ny;
	const bool col_on = lane < W;
	const bool edge = x0 + lane == 0 || x0 + lane == nx - 1;
	const int o = (warp + 1) * kPitch + lane + 1;   // pixel k of a thread: row warp + 8 k
	// the pixel of the ring that this thread also updates
	const int rr = t < 64 ? t : H, rc = t < 64 ? W : t - 64;
	const bool ring_on = t < 64 ? right && t < H : below && t - 64 < W;
	const bool ring_edge = x0 + rc == 0 || x0 + rc == nx - 1;
	const int ro = (rr + 1) * kPitch + rc + 1;
	const size_t base = (size_t)pair * size;
	const float *I0 = a.im.i0(pair), *I1 = a.im.i1(pair);
	const float *I1x = a.im.gx + a.im.grad(pair), *I1y = a.im.gy + a.im.grad(pair);
	float *const u1 = a.u1 + base, *const u2 = a.u2 + base;
	const int g0 = (y0 + warp) * nx + x0 + lane, gr = (y0 + rr) * nx + x0 + rc;

	for (int i = t; i < 6 * kSize; i += 256) sm[i] = 0.f;
	if (t == 0) s_fail = 0;
	__syncthreads();
	if (col_on)
		for (int k = 0; k < PPT; k++)
			if (warp + 8 * k < H) {
				U1[o + 8 * k * kPitch] = u1[g0 + 8 * k * nx];
				U2[o + 8 * k * kPitch] = u2[g0 + 8 * k * nx];
			}
	if (ring_on) {
		U1[ro] = u1[gr];
		U2[ro] = u2[gr];
	}
	const float l_t = a.lambda * a.theta, taut = a.tau / a.theta;
	unsigned it = 0;
	for (int wp = 0; wp < a.warps; wp++) {
		// the warped image and gradient at this step's flow, and the constant part of rho
		float cx[PPT + 1], cy[PPT + 1], cr[PPT + 1];
#pragma unroll
		for (int k = 0; k <= PPT; k++) {
			const bool on = k == PPT ? ring_on : col_on && warp + 8 * k < H;
			const int so = k == PPT ? ro : o + 8 * k * kPitch;
			cx[k] = cy[k] = cr[k] = 0.f;
			if (on) {
				const float v1 = U1[so], v2 = U2[so];
				const int j = x0 + (k == PPT ? rc : lane), i = y0 + (k == PPT ? rr : warp + 8 * k);
				const float3 w = warp_at(I1, I1x, I1y, (float)j + v1, (float)i + v2, nx, ny);
				cx[k] = w.y;
				cy[k] = w.z;
				cr[k] = w.x - w.y * v1 - w.z * v2 - I0[i * nx + j];
			}
		}
		for (int n = 0; n < kMaxIterations; n++, it++) {
			// u, at the tile and its ring
			float err = 0.f;
#pragma unroll
			for (int k = 0; k <= PPT; k++) {
				const bool on = k == PPT ? ring_on : col_on && warp + 8 * k < H;
				const int so = k == PPT ? ro : o + 8 * k * kPitch;
				const bool side = k == PPT ? ring_edge : edge;
				if (on) {
					const float wx = cx[k], wy = cy[k], g = wx * wx + wy * wy;
					const float u1k = U1[so], u2k = U2[so];
					float d1, d2;
					threshold(wx, wy, g, cr[k] + (wx * u1k + wy * u2k), l_t, d1, d2);
					// p is 0 outside the image, p11 and p21 in its last column and p12
					// and p22 in its last row; the order of the sum is the reference's
					const float h1 = P11[so] - P11[so - 1], h2 = P21[so] - P21[so - 1];
					const float a1 = P12[so], b1 = P12[so - kPitch], a2 = P22[so], b2 = P22[so - kPitch];
					const float dp1 = side ? h1 + a1 - b1 : h1 + (a1 - b1);
					const float dp2 = side ? h2 + a2 - b2 : h2 + (a2 - b2);
					const float n1 = (u1k + d1) + a.theta * dp1, n2 = (u2k + d2) + a.theta * dp2;
					U1[so] = n1;
					U2[so] = n2;
					if (k < PPT) err += (n1 - u1k) * (n1 - u1k) + (n2 - u2k) * (n2 - u2k);
				}
			}
			for (int d = 16; d; d >>= 1) err += __shfl_xor_sync(~0u, err, d);
			if (lane == 0) s_red[warp] = err;
			__syncthreads();
			// p, and the tile's border of it to the neighbours
			float *const out = a.ring + (size_t)(it & 1) * 4 * a.plane + base;
#pragma unroll 2
			for (int k = 0; k < PPT; k++) {
				const int r = warp + 8 * k, so = o + 8 * k * kPitch;
				if (!(col_on && r < H)) continue;
				const bool last_x = x0 + lane == nx - 1, last_y = y0 + r == ny - 1;
				const float u1k = U1[so], u2k = U2[so];
				const float u1x = last_x ? 0.f : U1[so + 1] - u1k, u1y = last_y ? 0.f : U1[so + kPitch] - u1k;
				const float u2x = last_x ? 0.f : U2[so + 1] - u2k, u2y = last_y ? 0.f : U2[so + kPitch] - u2k;
				// |grad u| in float (the reference's double hypot rounded to
				// float agrees to the last bit or one unit), and 1.0 + x rounded
				// once to float, as the reference's double sum of two floats is
				const float ng1 = 1.f + taut * sqrtf(u1x * u1x + u1y * u1y);
				const float ng2 = 1.f + taut * sqrtf(u2x * u2x + u2y * u2y);
				const float y1 = __frcp_rn(ng1), y2 = __frcp_rn(ng2);
				const float q11 = divide_by(P11[so] + taut * u1x, ng1, y1);
				const float q12 = divide_by(P12[so] + taut * u1y, ng1, y1);
				const float q21 = divide_by(P21[so] + taut * u2x, ng2, y2);
				const float q22 = divide_by(P22[so] + taut * u2y, ng2, y2);
				P11[so] = q11;
				P12[so] = q12;
				P21[so] = q21;
				P22[so] = q22;
				if (lane == 0 || lane == W - 1 || r == 0 || r == H - 1) {
					float *const q = out + g0 + 8 * k * nx;
					__stcg(q, q11);
					__stcg(q + a.plane, q12);
					__stcg(q + 2 * a.plane, q21);
					__stcg(q + 3 * a.plane, q22);
				}
			}
			__syncthreads();
			float *const part = a.partial + (size_t)(it & 1) * gridDim.x;
			if (t == 0) {
				float e = 0.f;
				for (int k = 0; k < 8; k++) e += s_red[k];
				__stcg(part + blockIdx.x, e);
				__threadfence();
				atomicAdd(a.arrived + pair, 1u);
				const unsigned target = (it + 1) * (unsigned)a.tiles;
				int polls = 0;
				while ((int)(load_acquire(a.arrived + pair) - target) < 0)
					if (++polls == kMaxPolls) {
						s_fail = 1;
						atomicExch(a.error, 1);
						break;
					}
			}
			__syncthreads();
			if (s_fail) return;
			// the neighbours' borders, and the pair's mean squared update
			if (warp == 7) {
				float e = 0.f;
				const float *const mine = part + blockIdx.x - tile;
				for (int k = lane; k < a.tiles; k += 32) e += __ldcg(mine + k);
				for (int d = 16; d; d >>= 1) e += __shfl_xor_sync(~0u, e, d);
				if (lane == 0) s_err = e / (float)size;
			} else if (t < 96) {
				if (ring_on) {   // all four on the right column and the row below
					const float *const q = out + gr;
					P11[ro] = __ldcg(q);
					P12[ro] = __ldcg(q + a.plane);
					P21[ro] = __ldcg(q + 2 * a.plane);
					P22[ro] = __ldcg(q + 3 * a.plane);
				}
			} else if (t < 161) {   // the column to the left, and below it where the tile has a row there
				const int r = t - 96;
				if (x0 > 0 && r < H + (below ? 1 : 0)) {
					const float *const q = out + (y0 + r) * nx + x0 - 1;
					P11[(r + 1) * kPitch] = __ldcg(q);
					P21[(r + 1) * kPitch] = __ldcg(q + 2 * a.plane);
				}
			} else if (t >= 161 && t < 194) {   // the row above, and its corner on the right
				const int c = t - 161;
				if (y0 > 0 && c < W + (right ? 1 : 0)) {
					const float *const q = out + (y0 - 1) * nx + x0 + c;
					P12[c + 1] = __ldcg(q + a.plane);
					P22[c + 1] = __ldcg(q + 3 * a.plane);
				}
			}
			__syncthreads();
			if (!(s_err > a.eps2)) {
				it++;
				break;
			}
		}
	}
	if (col_on)
		for (int k = 0; k < PPT; k++)
			if (warp + 8 * k < H) {
				u1[g0 + 8 * k * nx] = U1[o + 8 * k * kPitch];
				u2[g0 + 8 * k * nx] = U2[o + 8 * k * kPitch];
			}
}

// ---- one warping step from L2, for a level that does not fit on the chip -----------
// the three warps of a warping step and the constant parts of rho
__global__ void __launch_bounds__(256) warp_kernel(LevelImages im, const float *__restrict__ u1,
                                                   const float *__restrict__ u2, float *__restrict__ I1wx,
                                                   float *__restrict__ I1wy, float *__restrict__ grad,
                                                   float *__restrict__ rho_c)
{
	const int j = blockIdx.x * 32 + threadIdx.x, i = blockIdx.y * 8 + threadIdx.y, pair = blockIdx.z;
	if (j >= im.nx || i >= im.ny) return;
	const int p = i * im.nx + j;
	const size_t q = (size_t)pair * im.nx * im.ny + p, g = im.grad(pair);
	const float3 w = warp_at(im.i1(pair), im.gx + g, im.gy + g, (float)j + u1[q], (float)i + u2[q], im.nx, im.ny);
	I1wx[q] = w.y;
	I1wy[q] = w.z;
	grad[q] = w.y * w.y + w.z * w.z;
	rho_c[q] = w.x - w.y * u1[q] - w.z * u2[q] - im.i0(pair)[p];
}

struct IterArgs {
	const float *I1wx, *I1wy, *grad, *rho_c;
	float *u1, *u2, *p11, *p12, *p21, *p22;
	float *partial;          // [2][npairs][bpp]
	int *active;             // [npairs]
	int *iters;              // [npairs]
	int nx, ny, npairs, bpp;
	float tau, lambda, theta, eps2;
};

// The fixed-point iterations of one warping step for every pair
// (tvl1flow_lib.c:163-246).  Block b serves pair b / bpp.
__global__ void __launch_bounds__(256) iterate_kernel(IterArgs a)
{
	cg::grid_group grid = cg::this_grid();
	__shared__ float red[256];
	__shared__ int s_any;
	const int pair = blockIdx.x / a.bpp, sub = blockIdx.x % a.bpp;
	const int size = a.nx * a.ny;
	const long long base = (long long)pair * size;
	const float l_t = a.lambda * a.theta;
	const float taut = a.tau / a.theta;
	for (int n = 0; n < kMaxIterations; n++) {
		const bool act = a.active[pair] != 0;
		float err = 0.f;
		if (act) {
			// thresholding, divergence of p, update of u (in place: only the
			// pixel's own u is read)
			for (int p = sub * blockDim.x + threadIdx.x; p < size; p += a.bpp * blockDim.x) {
				const long long q = base + p;
				const int i = p / a.nx, j = p % a.nx;
				const float wx = a.I1wx[q], wy = a.I1wy[q], g = a.grad[q];
				const float u1k = a.u1[q], u2k = a.u2[q];
				const float rho = a.rho_c[q] + (wx * u1k + wy * u2k);
				float d1, d2;
				threshold(wx, wy, g, rho, l_t, d1, d2);
				const float v1 = u1k + d1, v2 = u2k + d2;
				const float dp1 = divergence_at(a.p11 + base, a.p12 + base, i, j, a.nx, a.ny);
				const float dp2 = divergence_at(a.p21 + base, a.p22 + base, i, j, a.nx, a.ny);
				const float n1 = v1 + a.theta * dp1, n2 = v2 + a.theta * dp2;
				a.u1[q] = n1;
				a.u2[q] = n2;
				err += (n1 - u1k) * (n1 - u1k) + (n2 - u2k) * (n2 - u2k);
			}
		}
		red[threadIdx.x] = err;
		__syncthreads();
		for (int h = blockDim.x / 2; h > 0; h >>= 1) {
			if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
			__syncthreads();
		}
		float *part = a.partial + (size_t)(n & 1) * a.npairs * a.bpp;
		if (threadIdx.x == 0) part[pair * a.bpp + sub] = red[0];
		grid.sync();
		if (act) {
			// gradient of u, update of the dual variable p
			for (int p = sub * blockDim.x + threadIdx.x; p < size; p += a.bpp * blockDim.x) {
				const long long q = base + p;
				const int i = p / a.nx, j = p % a.nx;
				float u1x, u1y, u2x, u2y;
				forward_gradient_at(a.u1 + base, i, j, a.nx, a.ny, u1x, u1y);
				forward_gradient_at(a.u2 + base, i, j, a.nx, a.ny, u2x, u2y);
				// |grad u| in float (the reference's double hypot rounded to
				// float agrees to the last bit or one unit; FP64 is slow here),
				// and 1.0 + x rounded once to float, as the reference's
				// double sum of two floats is
				const float g1 = sqrtf(u1x * u1x + u1y * u1y);
				const float g2 = sqrtf(u2x * u2x + u2y * u2y);
				const float ng1 = 1.f + taut * g1;
				const float ng2 = 1.f + taut * g2;
				a.p11[q] = (a.p11[q] + taut * u1x) / ng1;
				a.p12[q] = (a.p12[q] + taut * u1y) / ng1;
				a.p21[q] = (a.p21[q] + taut * u2x) / ng2;
				a.p22[q] = (a.p22[q] + taut * u2y) / ng2;
			}
		}
		// every block decides the same way for every pair
		if (threadIdx.x == 0) s_any = 0;
		__syncthreads();
		for (int k = threadIdx.x; k < a.npairs; k += blockDim.x) {
			if (!a.active[k]) continue;
			float e = 0.f;
			for (int b = 0; b < a.bpp; b++) e += part[k * a.bpp + b];
			e /= (float)size;
			if (e > a.eps2 && n + 1 < kMaxIterations) atomicOr(&s_any, 1);
		}
		__syncthreads();
		const int any = s_any;
		grid.sync();   // everyone has read this iteration's active flags
		if (blockIdx.x == 0)
			for (int k = threadIdx.x; k < a.npairs; k += blockDim.x) {
				if (!a.active[k]) continue;
				float e = 0.f;
				for (int b = 0; b < a.bpp; b++) e += part[k * a.bpp + b];
				e /= (float)size;
				a.iters[k] = n + 1;
				if (!(e > a.eps2 && n + 1 < kMaxIterations)) a.active[k] = 0;
			}
		grid.sync();
		if (!any) break;
	}
}

__global__ void set_int_kernel(int *p, int n, int v)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// Gaussian taps of mask.c:211-237, computed on the host in double
int gauss_taps(double sigma, std::vector<double> &B)
{
	const double den = 2 * sigma * sigma;
	const int size = (int)(kGaussWindow * sigma) + 1;
	B.assign(size, 0.0);
	for (int i = 0; i < size; i++) B[i] = 1 / (sigma * sqrt(2.0 * 3.1415926)) * exp(-i * i / den);
	double norm = 0;
	for (int i = 0; i < size; i++) norm += B[i];
	norm *= 2;
	norm -= B[0];
	for (int i = 0; i < size; i++) B[i] /= norm;
	return size;
}

dim3 grid_of(int nx, int ny, int n) { return dim3((nx + 31) / 32, (ny + 7) / 8, n); }

// n images of nx x ny: in (kept) -> tmp -> out
cudaError_t gaussian(const float *in, float *tmp, float *out, int nx, int ny, int n, double sigma, cudaStream_t st)
{
	std::vector<double> B;
	const int taps = gauss_taps(sigma, B);
	if (taps > kMaxGauss || taps > nx || taps > ny) return cudaErrorInvalidValue;   // "sigma too large"
	Gauss g = {};
	g.taps = taps;
	for (int j = 0; j < taps; j++) {
		g.d[j] = B[j];
		g.h[j] = (float)B[j];
		g.l[j] = (float)(B[j] - (double)g.h[j]);
	}
	g.e = (float)(3.0 * taps * (taps + 4) * 0x1p-48);
	gauss_pass_kernel<0><<<grid_of(nx, ny, n), dim3(32, 8), 0, st>>>(in, tmp, nx, ny, g);
	gauss_pass_kernel<1><<<grid_of(nx, ny, n), dim3(32, 8), 0, st>>>(tmp, out, nx, ny, g);
	return cudaGetLastError();
}

// Tiles of 32 x 8 PPT pixels: the smallest that lets all pairs run at once (more
// blocks share the work of a small level), else the largest, whose launch takes
// as many pairs as fit; 0 pairs when not even one does.
struct LevelPlan {
	const void *kernel;
	size_t smem;
	int ntx, tiles, tw, th, pairs;
};

cudaError_t plan_level(int nx, int ny, int npairs, int nsm, LevelPlan &pl)
{
	const void *const kernels[4] = {(const void *)level_kernel<1>, (const void *)level_kernel<2>,
	                                (const void *)level_kernel<4>, (const void *)level_kernel<8>};
	for (int k = 0; k < 4; k++) {
		const int th = 8 << k;
		pl.kernel = kernels[k];
		pl.smem = level_smem(1 << k);
		cudaError_t e = cudaFuncSetAttribute(pl.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem);
		int per_sm = 0;
		if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pl.kernel, 256, pl.smem);
		if (e != cudaSuccess) return e;
		pl.ntx = (nx + kTileW - 1) / kTileW;
		const int nty = (ny + th - 1) / th;
		pl.tw = (nx + pl.ntx - 1) / pl.ntx;
		pl.th = (ny + nty - 1) / nty;
		const long long tiles = (long long)pl.ntx * nty;
		pl.pairs = (int)std::min<long long>(npairs, (long long)per_sm * nsm / tiles);
		pl.tiles = (int)tiles;
		if (pl.pairs == npairs) break;
	}
	if (nx < 3 || ny < 3) pl.pairs = 0;   // the divergence of a line of one or two pixels has its own form
	return cudaSuccess;
}

}  // namespace

int tvl1_scales(int nx, int ny, int nscales, float zfactor)
{
	// main.c:147-153: the smallest level is about 16 pixels across
	const float N = (float)(1 + log(hypot(nx, ny) / 16.0) / log(1 / zfactor));
	if (N < nscales) nscales = (int)N;
	return nscales;
}

// The flow of npairs frame pairs (I0[k] -> I1[k], each nx x ny, device
// memory) into u (x displacement) and v (y displacement), [pair][y][x].
// mirrored: I0 and I1 hold npairs / 2 images, and the second half of the pairs
// is the first one backwards (I1[k] -> I0[k]).
// ws: device workspace of tvl1_workspace_floats(...) floats; iws: 2 npairs + 2
// ints, the last one set where a barrier ran into its limit.
size_t tvl1_workspace_floats(int nx, int ny, int npairs, int nscales, float zfactor)
{
	size_t total = 0;
	int w = nx, h = ny;
	for (int s = 0; s < nscales; s++) {
		total += (size_t)4 * w * h * npairs;   // I0, I1, u1, u2 of the level
		const int nw = (int)((float)w * zfactor + 0.5f), nh = (int)((float)h * zfactor + 0.5f);
		w = nw;
		h = nh;
	}
	total += (size_t)13 * nx * ny * npairs;    // per-level work arrays, sized for level 0
	total += (size_t)2 * npairs * 1024 + 8192; // partial sums
	return total;
}

cudaError_t tvl1_flow(const float *I0, const float *I1, int nx, int ny, int npairs, bool mirrored,
                      const Tvl1Params &pr, float *u, float *v, float *ws, int *iws, int nsm, cudaStream_t st,
                      std::string &why)
{
	const int nscales = pr.nscales;
	const int fscale = std::min(pr.fscale, nscales);
	const int m = mirrored ? npairs / 2 : npairs;   // images on each side
	if (2 * (long long)m > 65535) { why = "too many frame pairs for one cooperative launch"; return cudaErrorInvalidValue; }
	std::vector<int> NX(nscales), NY(nscales);
	std::vector<float *> img(nscales), lu(nscales), lv(nscales);   // img: the m first images, the m second ones
	NX[0] = nx;
	NY[0] = ny;
	for (int s = 1; s < nscales; s++) {   // zoom_size (zoom.c:24-35)
		NX[s] = (int)((float)NX[s - 1] * pr.zfactor + 0.5f);
		NY[s] = (int)((float)NY[s - 1] * pr.zfactor + 0.5f);
	}
	float *w = ws;
	for (int s = 0; s < nscales; s++) {
		const size_t n = (size_t)NX[s] * NY[s] * npairs;
		img[s] = w; w += 2 * n;
		lu[s] = s == 0 ? u : w; w += n;
		lv[s] = s == 0 ? v : w; w += n;
	}
	const size_t n0 = (size_t)nx * ny * npairs;
	float *I1x = w, *I1y = w + n0, *ring = w + 2 * n0, *I1wx = ring, *I1wy = w + 3 * n0, *grad = w + 4 * n0,
	      *rho_c = w + 5 * n0, *p11 = w + 6 * n0, *p12 = w + 7 * n0, *p21 = w + 8 * n0, *p22 = w + 9 * n0,
	      *tmp = w, *tmp2 = w + 2 * n0;   // 2 n0 each, before the gradients are needed
	float *partial = w + 13 * n0;
	int *active = iws, *iters = iws + npairs, *error = iws + 2 * npairs;
	cudaMemsetAsync(error, 0, sizeof(int), st);

	// normalisation and pre-smoothing (tvl1flow_lib.c:385-390)
	const int size = nx * ny;
	const int parts = std::max(1, std::min(32, size / 4096));
	minmax_kernel<<<dim3(parts, 2 * m), 256, 0, st>>>(I0, I1, m, size, partial);
	normalize_kernel<<<dim3(std::max(1, std::min(64, size / 1024)), 2 * m), 256, 0, st>>>(I0, I1, m, size, partial,
	                                                                                     parts, tmp2);
	cudaError_t e = gaussian(tmp2, tmp, img[0], nx, ny, 2 * m, kPresmoothSigma, st);
	if (e != cudaSuccess) { why = "image too small for the Gaussian pre-smoothing"; return e; }
	// pyramid (zoom_out, zoom.c:42-77)
	const float zsig = (float)(kZoomSigmaZero * sqrt(1.0 / (pr.zfactor * pr.zfactor) - 1.0));
	for (int s = 1; s < nscales; s++) {
		e = gaussian(img[s - 1], tmp, tmp2, NX[s - 1], NY[s - 1], 2 * m, (double)zsig, st);
		if (e != cudaSuccess) { why = "pyramid level too small for the Gaussian"; return e; }
		const size_t half = (size_t)m * NX[s - 1] * NY[s - 1];
		resample_kernel<<<grid_of(NX[s], NY[s], m), dim3(32, 8), 0, st>>>(
		    tmp2, tmp2 + half, NX[s - 1], NY[s - 1], img[s], img[s] + (size_t)m * NX[s] * NY[s], NX[s], NY[s],
		    pr.zfactor, pr.zfactor, 1.f, 0);
	}
	const size_t nc = (size_t)NX[nscales - 1] * NY[nscales - 1] * npairs;
	cudaMemsetAsync(lu[nscales - 1], 0, sizeof(float) * nc, st);
	cudaMemsetAsync(lv[nscales - 1], 0, sizeof(float) * nc, st);

	int per_sm = 0;
	e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, iterate_kernel, 256, 0);
	if (e != cudaSuccess) return e;
	const int maxb = std::max(1, per_sm) * nsm;
	if (npairs > maxb) { why = "too many frame pairs for one cooperative launch"; return cudaErrorInvalidValue; }
	const float scale = (float)1.0 / pr.zfactor;
	for (int s = nscales - 1; s >= 0; s--) {
		const int sx = NX[s], sy = NY[s];
		if (s >= fscale) {
			const size_t n = (size_t)sx * sy;
			LevelImages im;
			im.first = img[s];
			im.second = img[s] + m * n;
			im.gx = I1x;
			im.gy = I1y;
			im.m = m;
			im.mirrored = mirrored;
			im.nx = sx;
			im.ny = sy;
			centered_gradient_kernel<<<grid_of(sx, sy, mirrored ? 2 * m : m), dim3(32, 8), 0, st>>>(
			    mirrored ? im.first : im.second, I1x, I1y, sx, sy);
			LevelPlan pl;
			e = plan_level(sx, sy, npairs, nsm, pl);
			if (e != cudaSuccess) return e;
			if (pl.pairs > 0) {
				LevelArgs a;
				a.im = im;
				a.u1 = lu[s];
				a.u2 = lv[s];
				a.ring = ring;
				a.plane = n * npairs;
				a.partial = partial;
				a.arrived = (unsigned *)active;
				a.error = error;
				a.tw = pl.tw;
				a.th = pl.th;
				a.ntx = pl.ntx;
				a.tiles = pl.tiles;
				a.warps = pr.warps;
				a.tau = pr.tau;
				a.lambda = pr.lambda;
				a.theta = pr.theta;
				a.eps2 = pr.epsilon * pr.epsilon;
				cudaMemsetAsync(active, 0, sizeof(int) * npairs, st);
				for (a.pair0 = 0; a.pair0 < npairs; a.pair0 += pl.pairs) {
					void *args[] = {&a};
					e = cudaLaunchCooperativeKernel(pl.kernel, dim3(std::min(pl.pairs, npairs - a.pair0) * pl.tiles),
					                                dim3(256), args, pl.smem, st);
					if (e != cudaSuccess) { why = "cooperative launch failed"; return e; }
				}
			} else {
				cudaMemsetAsync(p11, 0, sizeof(float) * 4 * n0, st);   // p11, p12, p21, p22 (contiguous)
				const int bpp = std::max(1, std::min(maxb / npairs, (int)((n + 255) / 256)));
				for (int wp = 0; wp < pr.warps; wp++) {
					warp_kernel<<<grid_of(sx, sy, npairs), dim3(32, 8), 0, st>>>(im, lu[s], lv[s], I1wx, I1wy, grad, rho_c);
					set_int_kernel<<<(npairs + 255) / 256, 256, 0, st>>>(active, npairs, 1);
					IterArgs a;
					a.I1wx = I1wx;
					a.I1wy = I1wy;
					a.grad = grad;
					a.rho_c = rho_c;
					a.u1 = lu[s];
					a.u2 = lv[s];
					a.p11 = p11;
					a.p12 = p12;
					a.p21 = p21;
					a.p22 = p22;
					a.partial = partial;
					a.active = active;
					a.iters = iters;
					a.nx = sx;
					a.ny = sy;
					a.npairs = npairs;
					a.bpp = bpp;
					a.tau = pr.tau;
					a.lambda = pr.lambda;
					a.theta = pr.theta;
					a.eps2 = pr.epsilon * pr.epsilon;
					void *args[] = {&a};
					e = cudaLaunchCooperativeKernel((const void *)iterate_kernel, dim3(npairs * bpp), dim3(256), args, 0, st);
					if (e != cudaSuccess) { why = "cooperative launch failed"; return e; }
				}
			}
		}
		// zoom the flow to the next finer level and scale it (tvl1flow_lib.c:429-459);
		// levels below fscale only pass it up
		if (s == 0) break;
		const float fx = (float)NX[s - 1] / sx, fy = (float)NY[s - 1] / sy;
		resample_kernel<<<grid_of(NX[s - 1], NY[s - 1], npairs), dim3(32, 8), 0, st>>>(
		    lu[s], lv[s], sx, sy, lu[s - 1], lv[s - 1], NX[s - 1], NY[s - 1], fx, fy, scale, 1);
	}
	return cudaGetLastError();
}

}  // namespace bm4dof
