// search_block.cu -- the exact patch search for blocks of 2 x 2 neighbouring
// reference patches, one warp per block.
//
// Same neighbour lists as search.cu's kernel, which computes every group by
// itself in the reference's summation order.  Here:
//
//   * Shared differences.  Neighbouring reference patches lie S < P pixels
//     apart (P the patch width, S the grid step) and overlap.  For one
//     displacement, the squared differences of the (P + S) x (P + S) pixels of
//     the four patches are summed in 3 x 3 cells (columns and rows [0, S),
//     [S, P), [P, P + S)); each patch's distance is the sum of its four cells.
//     4x4 patches of step 2 (S = 2): 36 differences per frame for four
//     distances instead of 64.
//   * One multiply-add per difference (fma.rn), packed in pairs (f32x2), where
//     the reference's order needs a product and a sum.  The distances so formed
//     are not the reference's last bits, but within eps of them.
//   * Streaming selection.  Every lane keeps the minima of its distances; the
//     K-th smallest of the warp's 64 minima per patch bounds the K-th smallest
//     distance from above, and only candidates within that bound (widened by
//     eps) are listed, about 70 of 3969.
//   * Certified order.  Two listed distances further apart than their error
//     bounds compare as the reference's do.  Where the K nearest are all that
//     far apart from their neighbours in rank, the list is the reference's.
//     Otherwise the listed candidates' distances are formed again in the
//     reference's order; what is still equal then (std::partial_sort's heap
//     decides) is left to search.cu's kernel, as are groups whose list
//     overflows and sources with values that are not finite.
//   * Blocks that do not pay.  The four windows of a block follow their own
//     flows; where those differ the block covers the windows' union, which may
//     cost more than the four windows one by one (Cost).  And in a block of
//     one value every group finds itself and its neighbours at distance 0, a tie.
//     Such blocks are left to search.cu's kernel before they are computed: flat
//     854x480x8, 4x4x4, both steps, 40.1 ms with them computed, 31.8 without.
//
// What bounds it: issue slots and L1.  Per displacement of a block (four
// distances) of 4x4x4 patches with S = 2 a warp issues 168 packed or scalar FP32
// instructions (288 lane operations, where four separate patches take 768), 41
// loads and about 170 others (addresses, cells, minima, listing); on
// 480x272x12 the FP32 pipe is busy 48 % of the cycles, the L1 data path 60 %,
// the issue slots 53 %.  168 registers (12 warps per SM) hold a frame of the
// reference block (36 values) and the 63 sums of 7 displacements; 5
// displacements at 128 registers load more per distance (67 against 60.5 ms on
// 854x480x20), scalar FP32 instructions issue more (77 ms), the reference block
// in shared memory instead of registers 64 ms.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "internal.hpp"
#include "search_common.cuh"

namespace bm4dof {

namespace {

constexpr int kWarps = 4;              // blocks in flight per CTA
constexpr int kRows = 7;               // displacements per lane along y
constexpr int kMaxRounds = 256;        // rounds of 32 columns of displacements per block

typedef float2 f32x2;

__device__ __forceinline__ f32x2 pack2(float a, float b) { return make_float2(a, b); }

__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b)
{
	a = v.x; b = v.y;
}

// (the reference patches are kept negated)
__device__ __forceinline__ f32x2 sub2(f32x2 neg_ref, f32x2 v) { return __fadd2_rn(neg_ref, v); }

__device__ __forceinline__ f32x2 sqacc2(f32x2 d, f32x2 acc)
{
	return __ffma2_rn(d, d, acc);
}

// One frame of the temporal range: the displacements (of the block's first
// patch) that any of its patches searches, and each patch's own window in it.
struct BlockFrame {
	int qt, dx0, dy0, uw;              // frame, first displacement, displacements per row
	int ibase;                         // first item (one column of up to kRows displacements)
	float inv_uw;
	unsigned win[4];                   // per patch: first column, columns, first row, rows (bytes)
};

template <int P, int S>
struct Shape {
	static constexpr int W = P + S;                     // pixels of the block along an axis
	static constexpr int NB = P - S;                    // width of the shared middle
	static constexpr int kPitch = (2 * S + NB + 3) / 4 * 4;   // floats of one reference row: S pairs, the middle
	static constexpr bool kRefRegs = W * W <= 49;       // a frame of the reference block fits registers
};

template <int P, int S, int PT>
struct WarpShared {
	// listed candidates per patch: image patches have few candidates but keep up
	// to 32 of them, from windows where many are alike
	static constexpr int kListCap = PT == 1 ? 384 : 256;
	BlockFrame fr[kMaxFrames];
	uint2 list[4][kListCap];           // approximate distance, item << 3 | row
	float near_d[64];                  // one patch's nearest candidates: distance,
	unsigned near_c[64];               // item << 3 | row
};

// The terms j and j + 1 of the middle's row, onto its sum.
template <int NB>
__device__ __forceinline__ void add_mid(int j, const float (&r)[NB > 0 ? NB : 1], const float (&v)[NB > 0 ? NB : 1],
                                        float &acc)
{
	if (j + 1 < NB) {
		float d0, d1;
		unpack2(sub2(pack2(r[j], r[j + 1]), pack2(v[j], v[j + 1])), d0, d1);
		acc = __fmaf_rn(d1, d1, __fmaf_rn(d0, d0, acc));
	} else if (j < NB) {
		const float d = __fadd_rn(r[j], v[j]);
		acc = __fmaf_rn(d, d, acc);
	}
}

// Cells of kRows vertically adjacent displacements.  col: the candidate
// block's first pixel of the first displacement.
template <int P, int S, int PT>
__device__ __forceinline__ void block_cells(const float *col, size_t rpitch, size_t cpitch, size_t tpitch, int chn,
                                            const float *ref_s, f32x2 (&ac)[kRows][3], float (&mid)[kRows][3])
{
	using Sh = Shape<P, S>;
	constexpr int W = Sh::W, NB = Sh::NB, PI = Sh::kPitch;
#pragma unroll
	for (int r = 0; r < kRows; r++)
#pragma unroll
		for (int k = 0; k < 3; k++) {
			ac[r][k] = make_float2(0.f, 0.f);
			mid[r][k] = 0.f;
		}
	for (int c = 0; c < chn; c++)
#pragma unroll 1
		for (int ht = 0; ht < PT; ht++) {
			const float *rs = ref_s + (c * PT + ht) * W * PI;
			f32x2 rac[Sh::kRefRegs ? W : 1][S];
			float rmid[Sh::kRefRegs ? W : 1][NB > 0 ? NB : 1];
			if constexpr (Sh::kRefRegs) {
#pragma unroll
				for (int y = 0; y < W; y++) {
#pragma unroll
					for (int i = 0; i < S; i++) rac[y][i] = *reinterpret_cast<const f32x2 *>(rs + y * PI + 2 * i);
#pragma unroll
					for (int j = 0; j < NB; j++) rmid[y][j] = rs[y * PI + 2 * S + j];
				}
			}
			const float *row = col + ht * tpitch + c * cpitch;
#pragma unroll
			for (int yy = 0; yy < kRows + W - 1; yy++) {
				f32x2 vac[S];
				float vm[NB > 0 ? NB : 1];
#pragma unroll
				for (int i = 0; i < S; i++) vac[i] = pack2(__ldg(row + i), __ldg(row + P + i));
#pragma unroll
				for (int j = 0; j < NB; j++) vm[j] = __ldg(row + S + j);
				row += rpitch;
				if constexpr (Sh::kRefRegs) {
					// term by term over all displacements: consecutive instructions are
					// independent of one another
#pragma unroll
					for (int i = 0; i < S; i++)
#pragma unroll
						for (int r = 0; r < kRows; r++) {
							const int hy = yy - r;
							if (hy < 0 || hy >= W) continue;
							const int seg = hy < S ? 0 : (hy < P ? 1 : 2);
							ac[r][seg] = sqacc2(sub2(rac[hy][i], vac[i]), ac[r][seg]);
						}
#pragma unroll
					for (int j = 0; j < NB; j += 2)
#pragma unroll
						for (int r = 0; r < kRows; r++) {
							const int hy = yy - r;
							if (hy < 0 || hy >= W) continue;
							const int seg = hy < S ? 0 : (hy < P ? 1 : 2);
							add_mid<NB>(j, rmid[hy], vm, mid[r][seg]);
						}
				} else {
#pragma unroll
					for (int r = 0; r < kRows; r++) {
						const int hy = yy - r;
						if (hy < 0 || hy >= W) continue;
						const int seg = hy < S ? 0 : (hy < P ? 1 : 2);
						// (a vector read of the reference row, the same for all lanes)
						float q[PI];
#pragma unroll
						for (int i = 0; i < PI; i += 4) {
							const float4 v4 = *reinterpret_cast<const float4 *>(rs + hy * PI + i);
							q[i] = v4.x;
							q[i + 1] = v4.y;
							q[i + 2] = v4.z;
							q[i + 3] = v4.w;
						}
						float qm[NB > 0 ? NB : 1];
#pragma unroll
						for (int j = 0; j < NB; j++) qm[j] = q[2 * S + j];
#pragma unroll
						for (int i = 0; i < S; i++)
							ac[r][seg] = sqacc2(sub2(pack2(q[2 * i], q[2 * i + 1]), vac[i]), ac[r][seg]);
#pragma unroll
						for (int j = 0; j < NB; j += 2) add_mid<NB>(j, qm, vm, mid[r][seg]);
					}
				}
			}
		}
}

struct BlockArgs {
	const Tile *tiles;
	int ntiles;
	const int *grid;
	const uint32_t *traj;
	int nfm;
	long long nblocks;
	const unsigned *bad_source;
	uint8_t *nsimp;
	uint32_t *idx;
	uint32_t *glist;                   // groups left to the per-group kernel (or none: nsimp stays as it is)
	unsigned *gcount;
	float eps;                         // relative error bound between two sums of one distance
};

// What a frame's share of a block costs here more than its four patches' candidates
// cost in search.cu's kernel; a block whose frames cost more than kSpare together is
// cheaper there.  In 1/1024 nanoseconds of the whole GPU and per channel, fitted to
// both kernels' times (854x480x8, windows of 9, 21 and 39; 8x8 and 7x7 also 7x7
// windows): a block takes 13 ns and, for every 32 columns of displacements, 0.025
// (4x4x4) or 0.036 a pixel of the block; a group 10 (4x4x4) or 50 and 0.011 a
// candidate.  4x4x4, step 2, 21x21 windows over 5 frames: 49 against 137 ns, so the
// columns may rise from 315 to 1090.  Without the rule flows with a noise of 8 / 20
// pixels took 21.9 / 52.2 ms (480x272x10, both steps) where the per-group kernel
// takes 15.0 / 16.0.
template <int P, int S, int PT>
struct Cost {
	static constexpr int kColumn = (int)((P == 4 ? 0.025f : 0.036f) * PT * (P + S) * (P + S) * 32.f + 0.5f);
	static constexpr int kCandidate = 11;
	static constexpr int kSpare = (P == 4 ? 4 * 10 - 13 : 4 * 50 - 13) * 1024;
};

constexpr float kTiny = 1e-35f;        // below this the products may underflow
constexpr float kMaxFinite = 3.0e38f;

// The largest approximate distance that a candidate no further away than one
// at approximate distance v can have.
__device__ __forceinline__ float widen(float v, float eps) { return fminf(v + (2.f * eps * v + kTiny), kMaxFinite); }

// Upper bounds of the K-th smallest of the warp's 64 values per patch (a, b per
// lane; distances as their bits, which order alike), at most hi; hi where fewer
// than K are below it.  The bound descends in halving steps from 2^bits (2^23 is
// a factor of two) to 2^17 (1.6 %); the four patches' steps are independent.
__device__ __forceinline__ void kth_bounds(const unsigned (&a)[4], const unsigned (&b)[4], const int (&K)[4],
                                           unsigned (&hi)[4], int bits)
{
#pragma unroll
	for (int k = 0; k < 4; k++) {
		// the largest finite value bounds the K-th, if K of them are finite
		const unsigned fa = a[k] < 0x7f800000u ? a[k] : 0u, fb = b[k] < 0x7f800000u ? b[k] : 0u;
		const unsigned top = __reduce_max_sync(0xffffffffu, max(fa, fb));
		const int c = __popc(__ballot_sync(0xffffffffu, a[k] < 0x7f800000u)) +
		              __popc(__ballot_sync(0xffffffffu, b[k] < 0x7f800000u));
		if (c >= K[k]) hi[k] = min(hi[k], top);
	}
#pragma unroll 1
	for (int s = bits; s >= 17; s--) {
#pragma unroll
		for (int k = 0; k < 4; k++) {
			const unsigned m = max(hi[k], 1u << s) - (1u << s);
			const int c = __popc(__ballot_sync(0xffffffffu, a[k] <= m)) + __popc(__ballot_sync(0xffffffffu, b[k] <= m));
			hi[k] = c >= K[k] ? m : hi[k];
		}
	}
}

template <int P, int S, int PT, int MINB>
__global__ void __launch_bounds__(32 * kWarps, MINB)
search_block_kernel(Image src, StepParams sp, BlockArgs a)
{
	using Sh = Shape<P, S>;
	using WS = WarpShared<P, S, PT>;
	constexpr int W = Sh::W, PI = Sh::kPitch, kListCap = WS::kListCap;
	extern __shared__ __align__(16) unsigned char smem[];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int chn = sp.chn_search;
	const size_t per_warp = sizeof(WS) + sizeof(float) * chn * PT * W * PI;
	WS &ws = *reinterpret_cast<WS *>(smem + warp * per_warp);
	float *ref_s = reinterpret_cast<float *>(smem + warp * per_warp + sizeof(WS));
	if (*a.bad_source) return;
	const unsigned lt = (1u << lane) - 1u;
	const int hw = (sp.wx - 1) / 2;
	const float eps = a.eps;

	for (long long blk = (long long)blockIdx.x * kWarps + warp; blk < a.nblocks; blk += (long long)gridDim.x * kWarps) {
		__syncwarp();
		// ---- the block: up to four reference patches, S apart -----------------
		int ti = 0;
		while (ti + 1 < a.ntiles && a.tiles[ti + 1].blk0 <= blk) ti++;
		const Tile T = a.tiles[ti];
		const unsigned lb = (unsigned)(blk - T.blk0);
		const int bi = (int)(lb % (unsigned)T.bkx), bj = (int)(lb / (unsigned)T.bkx % (unsigned)T.bky),
		          bf = (int)(lb / ((unsigned)T.bkx * T.bky));
		// columns: a regular pair, or one left-over column with a missing left one
		const bool px2 = bi < T.prx, py2 = bj < T.pry;
		const int xi = px2 ? 2 * bi : T.prx + bi, yi = py2 ? 2 * bj : T.pry + bj;
		const int X0 = a.grid[T.gx + xi] - (px2 ? 0 : S), Y0 = a.grid[T.gy + yi] - (py2 ? 0 : S);
		const int t = a.grid[T.gf + bf];
		const unsigned have = (px2 ? 3u : 2u) & 3u;           // bit kx: that column of patches exists
		const unsigned havey = (py2 ? 3u : 2u) & 3u;
		auto exists = [&](int k) { return ((have >> (k & 1)) & (havey >> (k >> 1)) & 1u) != 0u; };
		auto group = [&](int k) -> long long {
			const int gx = px2 ? xi + (k & 1) : xi, gy = py2 ? yi + (k >> 1) : yi;
			return T.g0 + ((long long)bf * T.ny + gy) * T.nx + gx;
		};
		int t0, t1;
		temporal_range(sp, t, t0, t1);
		const int nwt = t1 - t0 + 1;
		const unsigned wh = (unsigned)T.w * T.h;

		// ---- frames: windows of the patches and their union --------------------
		int items = 0;
		int cand[4] = {0, 0, 0, 0};
		bool wide = false;
		BlockFrame f;
		if (lane < nwt) {
			int lox[4], loy[4], nx[4], ny[4];
			int ux0 = 0x7fffffff, uy0 = 0x7fffffff, ux1 = -0x7fffffff, uy1 = -0x7fffffff;
#pragma unroll
			for (int k = 0; k < 4; k++) {
				lox[k] = loy[k] = nx[k] = ny[k] = 0;
				if (!exists(k)) continue;
				const uint32_t c = a.traj[group(k) * a.nfm + lane];
				const int cx = (int)(c & 0xffffu), cy = (int)(c >> 16);
				const int shx = min(0, cx - hw) + max(0, cx + hw - T.w + P);
				const int shy = min(0, cy - hw) + max(0, cy + hw - T.h + P);
				const int rx0 = max(0, cx - hw - shx), ry0 = max(0, cy - hw - shy);
				nx[k] = max(0, min(T.w - P, cx + hw - shx) - rx0 + 1);
				ny[k] = max(0, min(T.h - P, cy + hw - shy) - ry0 + 1);
				cand[k] = nx[k] * ny[k];
				// as displacements of the block's first patch position
				lox[k] = rx0 - (X0 + (k & 1) * S);
				loy[k] = ry0 - (Y0 + (k >> 1) * S);
				if (cand[k]) {
					ux0 = min(ux0, lox[k]);
					uy0 = min(uy0, loy[k]);
					ux1 = max(ux1, lox[k] + nx[k]);
					uy1 = max(uy1, loy[k] + ny[k]);
				}
			}
			const int uw = max(0, ux1 - ux0), uh = max(0, uy1 - uy0);
			wide = uw > 255 || uh > 255;
			items = uw * ((uh + kRows - 1) / kRows);
			f.qt = visit_frame(lane, t, t1);
			f.dx0 = ux0;
			f.dy0 = uy0;
			f.uw = uw;
			f.inv_uw = 1.f / (float)max(uw, 1);
#pragma unroll
			for (int k = 0; k < 4; k++)
				f.win[k] = cand[k] ? (unsigned)(lox[k] - ux0) | (unsigned)nx[k] << 8 | (unsigned)(loy[k] - uy0) << 16 |
				                         (unsigned)ny[k] << 24
				                   : 0u;
		}
		int ii = items;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const int u = __shfl_up_sync(0xffffffffu, ii, o);
			if (lane >= o) ii += u;
		}
		if (lane < nwt) {
			f.ibase = ii - items;
			ws.fr[lane] = f;
		}
		const int nitems = __shfl_sync(0xffffffffu, ii, 31);
		int K[4];
#pragma unroll
		for (int k = 0; k < 4; k++) K[k] = min(sp.np, __reduce_add_sync(0xffffffffu, cand[k]));
		// (in one condition with the next: another exit here costs the main loop registers)
		using Co = Cost<P, S, PT>;
		const int four = (cand[0] + cand[1] + cand[2] + cand[3]) << ((px2 ? 0 : 1) + (py2 ? 0 : 1));
		wide |= __reduce_add_sync(0xffffffffu, items * Co::kColumn - four * Co::kCandidate) * chn > Co::kSpare;
		// ---- reference pixels: per row S pairs (left, right), then the middle --
		// (not unrolled: 54.5 -> 53.9 ms on 854x480x20, both steps)
		bool flat = true;
#pragma unroll 1
		for (int i = lane; i < chn * PT * W * W; i += 32) {
			const int x = i % W, y = i / W % W, ht = i / (W * W) % PT, c = i / (W * W * PT);
			const float *first = src.p + src.at(T.ox, T.oy, t, c) + (long long)Y0 * src.P + X0;
			const float v = first[ht * src.plane() * src.C + (long long)y * src.P + x];
			flat &= v == *first;
			const int at = x < S ? 2 * x : (x < P ? 2 * S + x - S : 2 * (x - P) + 1);
			ref_s[((c * PT + ht) * W + y) * PI + at] = -v;
		}
		wide |= __all_sync(0xffffffffu, flat);
		if (__any_sync(0xffffffffu, wide) || nitems > 32 * kMaxRounds) {
			// windows far apart (a motion boundary, a rough flow), or a flat block
			if (a.glist && lane < 4 && exists(lane)) a.glist[atomicAdd(a.gcount, 1u)] = (uint32_t)group(lane);
			continue;
		}
		__syncwarp();

		// ---- distances and candidate lists --------------------------------------
		unsigned ma[4], mb[4], thr[4];
		int cnt[4];                        // listed candidates
		float tapp[4];                     // candidates up to this are listed
#pragma unroll
		for (int k = 0; k < 4; k++) {
			ma[k] = mb[k] = thr[k] = 0x7f800000u;
			cnt[k] = 0;
			tapp[k] = kMaxFinite;
		}
		int fi = 0;
		int round = 0;
#pragma unroll 1
		for (int base = 0; base < nitems; base += 32, round++) {
			const int it = min(base + lane, nitems - 1);
			while (fi + 1 < nwt && ws.fr[fi + 1].ibase <= it) fi++;
			const BlockFrame &fr = ws.fr[fi];
			const int rel = it - fr.ibase;
			const int strip = (int)(((float)rel + 0.5f) * fr.inv_uw), dx = rel - strip * fr.uw;
			const int dy = strip * kRows;
			const float *col = src.p + src.at(T.ox, T.oy, fr.qt, 0) + (long long)(Y0 + fr.dy0 + dy) * src.P + X0 + fr.dx0 + dx;
			f32x2 ac[kRows][3];
			float mid[kRows][3];
			block_cells<P, S, PT>(col, src.P, src.plane(), src.plane() * src.C, chn, ref_s, ac, mid);
			// the four patches' distances from the nine cells
			float d[4][kRows];
#pragma unroll
			for (int r = 0; r < kRows; r++) {
				float lo[3], hi[3];
#pragma unroll
				for (int s = 0; s < 3; s++) {
					float x0, x1;
					unpack2(ac[r][s], x0, x1);
					lo[s] = x0 + mid[r][s];
					hi[s] = mid[r][s] + x1;
				}
				d[0][r] = lo[0] + lo[1];
				d[1][r] = hi[0] + hi[1];
				d[2][r] = lo[1] + lo[2];
				d[3][r] = hi[1] + hi[2];
			}
			// candidates outside a patch's own window (and of lanes past the end) drop
			// out; rare: all four windows are mostly the same
			unsigned rows[4];                  // bit r: inside
			bool all_in = true;
#pragma unroll
			for (int k = 0; k < 4; k++) {
				const unsigned w = fr.win[k];
				const bool inx = base + lane < nitems && (unsigned)dx - (w & 255u) < (w >> 8 & 255u);
				const int first = max((int)(w >> 16 & 255u) - dy, 0), last = min((int)(w >> 16 & 255u) + (int)(w >> 24) - dy, kRows);
				rows[k] = inx && first < last ? (1u << last) - (1u << first) : 0u;
				all_in &= rows[k] == (1u << kRows) - 1u;
			}
			if (!__all_sync(0xffffffffu, all_in)) {
#pragma unroll 1
				for (int once = 0; once < 1; once++)   // (a loop: as selects they would cost every round)
#pragma unroll
					for (int k = 0; k < 4; k++)
#pragma unroll
						for (int r = 0; r < kRows; r++)
							if (!(rows[k] >> r & 1u)) d[k][r] = __int_as_float(0x7f800000);
			}
			float least[4];
#pragma unroll
			for (int k = 0; k < 4; k++) {
				const float m0 = fminf(fminf(d[k][0], d[k][1]), fminf(d[k][2], d[k][3]));
				const float m1 = fminf(fminf(d[k][4], d[k][5]), d[k][6]);
				ma[k] = min(ma[k], __float_as_uint(m0));
				mb[k] = min(mb[k], __float_as_uint(m1));
				least[k] = fminf(m0, m1);
			}
			if (round < 4 || round % 6 == 5 || base + 32 >= nitems) {
				kth_bounds(ma, mb, K, thr, round == 0 ? 28 : 23);
#pragma unroll
				for (int k = 0; k < 4; k++) tapp[k] = widen(__uint_as_float(thr[k]), eps);
			}
#pragma unroll
			for (int k = 0; k < 4; k++) {
				if (!__any_sync(0xffffffffu, least[k] <= tapp[k])) continue;
				int n = cnt[k];
#pragma unroll
				for (int r = 0; r < kRows; r++) {
					const bool hit = d[k][r] <= tapp[k];
					const unsigned m = __ballot_sync(0xffffffffu, hit);
					if (!m) continue;
					const int at = n + __popc(m & lt);
					if (hit && at < kListCap)
						ws.list[k][at] = make_uint2(__float_as_uint(d[k][r]), (unsigned)it << 3 | (unsigned)r);
					n += __popc(m);
				}
				if (n > kListCap) n = 0x10000;     // entries were lost: the group is left over
				else if (n > kListCap / 2) {
					// drop what the bound has fallen below
					__syncwarp();
					int left = 0;
					for (int e = 0; e < n; e += 32) {
						const uint2 q = e + lane < n ? ws.list[k][e + lane] : make_uint2(0x7f800000u, 0u);
						const bool keep = __uint_as_float(q.x) <= tapp[k];
						const unsigned m = __ballot_sync(0xffffffffu, keep);
						if (keep) ws.list[k][left + __popc(m & lt)] = q;
						left += __popc(m);
						__syncwarp();
					}
					n = left;
				}
				cnt[k] = n;
			}
		}
		__syncwarp();

		// ---- the K nearest of every patch ----------------------------------------
#pragma unroll 1
		for (int k = 0; k < 4; k++) {
			if (!exists(k)) continue;
			const long long g = group(k);
			const int Kk = k == 0 ? K[0] : k == 1 ? K[1] : k == 2 ? K[2] : K[3];
			const unsigned th = k == 0 ? thr[0] : k == 1 ? thr[1] : k == 2 ? thr[2] : thr[3];
			const int nc = k == 0 ? cnt[0] : k == 1 ? cnt[1] : k == 2 ? cnt[2] : cnt[3];
			bool ok = nc <= kListCap;
			float lim = widen(__uint_as_float(th), eps);
			int n = 0;
			if (ok) {
				// a tighter bound from the list where more than 64 are left
				for (int e = 0; e < nc; e += 32)
					n += __popc(__ballot_sync(0xffffffffu, e + lane < nc && __uint_as_float(ws.list[k][min(e + lane, kListCap - 1)].x) <= lim));
				if (n > 64) {
					unsigned lo = 0u, hi = th;
#pragma unroll 1
					for (int it = 0; it < 24 && n > 64; it++) {
						const unsigned m = lo + ((hi - lo) >> 1);
						int below = 0;
						for (int e = 0; e < nc; e += 32)
							below += __popc(__ballot_sync(0xffffffffu, e + lane < nc && ws.list[k][min(e + lane, kListCap - 1)].x <= m));
						if (below >= Kk) { hi = m; n = below; } else lo = m;
					}
					lim = widen(__uint_as_float(hi), eps);
				}
				// the candidates within it, side by side
				n = 0;
				for (int e = 0; e < nc; e += 32) {
					const uint2 q = e + lane < nc ? ws.list[k][e + lane] : make_uint2(0x7f800000u, 0u);
					const bool keep = __uint_as_float(q.x) <= lim;
					const unsigned m = __ballot_sync(0xffffffffu, keep);
					const int at = n + __popc(m & lt);
					if (keep && at < 64) {
						ws.near_d[at] = __uint_as_float(q.x);
						ws.near_c[at] = q.y;
					}
					n += __popc(m);
				}
				__syncwarp();
				ok = n >= Kk && n <= 64;
			}
			float dv[2] = {0.f, 0.f};
			int px_[2] = {0, 0}, py_[2] = {0, 0}, pt_[2] = {0, 0};   // position in the tile, frame
			int rank[2] = {64, 64};
			if (ok) {
				const int halves = n > 32 ? 2 : 1;
#pragma unroll
				for (int h = 0; h < 2; h++)
					if (lane + 32 * h < n) {
						dv[h] = ws.near_d[lane + 32 * h];
						const unsigned q = ws.near_c[lane + 32 * h];
						const int item = (int)(q >> 3), row = (int)(q & 7u);
						int fi2 = 0;
						while (fi2 + 1 < nwt && ws.fr[fi2 + 1].ibase <= item) fi2++;
						const BlockFrame &fr = ws.fr[fi2];
						const int rel = item - fr.ibase, strip = (int)(((float)rel + 0.5f) * fr.inv_uw);
						px_[h] = X0 + (k & 1) * S + fr.dx0 + rel - strip * fr.uw;
						py_[h] = Y0 + (k >> 1) * S + fr.dy0 + strip * kRows + row;
						pt_[h] = fr.qt;
					}
				// pass 0: the approximate distances, each from its neighbours in rank by
				// more than their errors; pass 1: formed again in the reference's order
				for (int pass = 0; pass < 2; pass++) {
					rank[0] = rank[1] = 0;
					for (int j = 0; j < n; j++) {
						const float o = ws.near_d[j];
						rank[0] += o < dv[0] || (o == dv[0] && j < lane) ? 1 : 0;
						if (halves == 2) rank[1] += o < dv[1] || (o == dv[1] && j < lane + 32) ? 1 : 0;
					}
					if (lane >= n) rank[0] = 64;
					if (lane + 32 >= n) rank[1] = 64;
					__syncwarp();
					if (rank[0] < 64) ws.near_d[rank[0]] = dv[0];   // in order now
					if (rank[1] < 64) ws.near_d[rank[1]] = dv[1];
					__syncwarp();
					bool doubt = false;
#pragma unroll
					for (int h = 0; h < 2; h++)
						if (rank[h] < Kk) {
							const float e2 = pass ? 0.f : 2.f * eps, tiny = pass ? 0.f : kTiny;
							const float nextd = rank[h] + 1 < n ? ws.near_d[rank[h] + 1] : __int_as_float(0x7f800000);
							doubt |= nextd - dv[h] <= __fmaf_rn(e2, nextd, tiny) && rank[h] + 1 < n;
							// tau rule: the distances at ranks 1, 2, 4, .. are compared with tau2
							doubt |= !pass && (rank[h] & (rank[h] - 1)) == 0 &&
							         fabsf(dv[h] - sp.tau2) <= __fmaf_rn(e2, sp.tau2, tiny);
						}
					ok = !__any_sync(0xffffffffu, doubt);
					if (ok || pass) break;
					const float *rp = src.p + src.at(T.ox, T.oy, t, 0) + (long long)(Y0 + (k >> 1) * S) * src.P + X0 + (k & 1) * S;
#pragma unroll
					for (int h = 0; h < 2; h++)
						if (lane + 32 * h < n) {
							const float *qp = src.p + src.at(T.ox + px_[h], T.oy + py_[h], pt_[h], 0);
							float s = 0.f;
							for (int c = 0; c < chn; c++)
								for (int ht = 0; ht < PT; ht++)
									for (int hy = 0; hy < P; hy++)
										for (int hx = 0; hx < P; hx++) {
											const size_t o = (size_t)ht * src.plane() * src.C + c * src.plane() + (size_t)hy * src.P + hx;
											const float df = __fsub_rn(rp[o], qp[o]);
											s = __fadd_rn(s, __fmul_rn(df, df));
										}
							dv[h] = s;
						}
					__syncwarp();
#pragma unroll
					for (int h = 0; h < 2; h++)
						if (lane + 32 * h < n) ws.near_d[lane + 32 * h] = dv[h];
					__syncwarp();
				}
			}
			if (!ok) {
				if (a.glist && lane == 0) a.glist[atomicAdd(a.gcount, 1u)] = (uint32_t)g;
				__syncwarp();
				continue;
			}
			// tau rule (nldct.cpp:1284-1289): n doubles while the next distance is below tau2
			unsigned below = 0u;   // bit b: the distance at rank 2^b is below tau2
#pragma unroll
			for (int h = 0; h < 2; h++)
				if (rank[h] < Kk && rank[h] > 0 && (rank[h] & (rank[h] - 1)) == 0 && dv[h] < sp.tau2)
					below |= 1u << (31 - __clz(rank[h]));
			below = __reduce_or_sync(0xffffffffu, below);
			int ns = 1;
			while (2 * ns <= Kk && (below >> (31 - __clz(ns)) & 1u)) ns *= 2;
			if (lane == 0) a.nsimp[g] = (uint8_t)ns;
#pragma unroll
			for (int h = 0; h < 2; h++)
				if (rank[h] < ns) a.idx[g * sp.np + rank[h]] = (uint32_t)pt_[h] * wh + (uint32_t)py_[h] * T.w + px_[h];
			__syncwarp();
		}
	}
}

// Values whose squared differences could overflow, and NaN: the block search
// relies on finite sums, so such a source is left to the per-group kernel.
__global__ void check_source_kernel(Image src, int chn, unsigned *__restrict__ bad)
{
	const size_t rows = (size_t)src.H * chn * src.F;
	bool b = false;
	for (size_t r = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); r < rows;
	     r += (size_t)gridDim.x * (blockDim.x >> 5)) {
		const size_t y = r % src.H, c = r / src.H % chn, t = r / ((size_t)src.H * chn);
		const float *row = src.p + src.at(0, (int)y, (int)t, (int)c);
		for (int x = threadIdx.x & 31; x < src.W; x += 32) b |= !(fabsf(row[x]) <= 1e17f);
	}
	if (__any_sync(0xffffffffu, b) && (threadIdx.x & 31) == 0) *bad = 1u;
}

template <int P, int S, int PT, int MINB>
cudaError_t launch_block(const Image &src, const StepParams &sp, const BlockArgs &a, int nsm, cudaStream_t st)
{
	auto kern = search_block_kernel<P, S, PT, MINB>;
	const size_t per_warp = sizeof(WarpShared<P, S, PT>) +
	                        sizeof(float) * sp.chn_search * PT * Shape<P, S>::W * Shape<P, S>::kPitch;
	const size_t smem = per_warp * kWarps;
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e != cudaSuccess) return e;
	int per_sm = 0;
	e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kWarps, smem);
	if (e != cudaSuccess) return e;
	const long long need = (a.nblocks + kWarps - 1) / kWarps;
	const long long blocks = std::min<long long>(need, (long long)nsm * std::max(per_sm, 1));
	kern<<<(int)blocks, 32 * kWarps, smem, st>>>(src, sp, a);
	return cudaGetLastError();
}

}  // namespace

// The patch shapes and grid steps of the benchmark and default parameters; other
// shapes, and tiles too small to give a single column or row a left neighbour,
// keep the per-group kernel.  Per-group kernel -> blocks (ms, both steps):
// 854x480x20 4x4x4 112.6 -> 57.6; 640x360x3x14 4x4x4 88.0 -> 42; 256x256 8x8
// 1.62 -> 0.19; 767x511 colour image, defaults (39x39 windows) 41.8 -> 2.3;
// 853x481x16 defaults (8x8 and 7x7, 7x7 windows) 29.9 -> 4.9.
bool block_search_supported(const StepParams &sp, const Plan &pl)
{
	if (!pl.blocks_ok || sp.np <= 1 || sp.search_strip == 7 || sp.search_ctas == 4) return false;
	const int p = sp.px, s = pl.step, t = sp.pt;
	return (p == 4 && t == 4 && (s == 2 || s == 3)) || (p == 8 && t == 1 && (s == 3 || s == 4 || s == 6)) ||
	       (p == 7 && t == 1 && (s == 3 || s == 4));
}

// Pixels a block of patches reaches past its tile: S on either side, and the
// unused rows of the last column of displacements.
size_t block_search_guard(int pitch) { return (size_t)16 * pitch + 64; }

cudaError_t launch_search_block(const Image &src, const Tile *tiles, int ntiles, const int *grid, const uint32_t *traj,
                                const StepParams &sp, int step, long long nblocks, uint8_t *nsimp, uint32_t *idx,
                                uint32_t *glist, unsigned *gcount, unsigned *bad_source, int nsm, cudaStream_t st)
{
	const long long rows = (long long)src.H * sp.chn_search * src.F;
	check_source_kernel<<<(int)std::min<long long>((rows + 7) / 8, 8ll * nsm), 256, 0, st>>>(src, sp.chn_search, bad_source);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess || nblocks <= 0) return e;
	BlockArgs a;
	a.tiles = tiles;
	a.ntiles = ntiles;
	a.grid = grid;
	a.traj = traj;
	a.nfm = search_frames_max(sp);
	a.nblocks = nblocks;
	a.bad_source = bad_source;
	a.nsimp = nsimp;
	a.idx = idx;
	a.glist = glist;
	a.gcount = gcount;
	// a distance of m terms, all positive, relative to their exact sum: the
	// reference's sequential sum is within (m + 1) u (u = 2^-24), the cells'
	// within (0.57 m + 4) u (the largest cell holds 36 of 64 terms); 2.5 (m + 8) u
	// covers both with room to spare
	a.eps = 2.5f * (float)(sp.spc * sp.chn_search + 8) * 5.9604645e-8f;
	const int p = sp.px;
	if (p == 4) return step == 2 ? launch_block<4, 2, 4, 3>(src, sp, a, nsm, st) : launch_block<4, 3, 4, 3>(src, sp, a, nsm, st);
	if (p == 7) return step == 3 ? launch_block<7, 3, 1, 3>(src, sp, a, nsm, st) : launch_block<7, 4, 1, 3>(src, sp, a, nsm, st);
	if (step == 3) return launch_block<8, 3, 1, 3>(src, sp, a, nsm, st);
	if (step == 4) return launch_block<8, 4, 1, 3>(src, sp, a, nsm, st);
	return launch_block<8, 6, 1, 3>(src, sp, a, nsm, st);
}

}  // namespace bm4dof
