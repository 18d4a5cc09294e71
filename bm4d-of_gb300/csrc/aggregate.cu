// aggregate.cu -- deterministic aggregation, reference-grid bookkeeping,
// normalisation, tile rebuild and colour transforms.
//
// The reference adds every group's estimates into a per-tile image and weight
// image one group after another (computeAggregationStep1/2,
// src/core/nldct.cpp:2259-2425), so each pixel's float sum follows the
// processing order (group, then member).  Here the same sums are formed as a
// gather with no float atomics: every member patch ("slot") is listed under
// the blocks of pixels it touches, each block's slots are ordered by slot
// number (= processing order), and the block's pixels add the terms of the
// slots that cover them in that order.  The result is bit-identical to the
// sequential scatter.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "internal.hpp"

namespace bm4dof {

namespace {


__device__ __forceinline__ void group_position(const Tile &T, const int *grid, long long g,
                                               int &x, int &y, int &t)
{
	const long long local = g - T.g0;
	x = grid[T.gx + (int)(local % T.nx)];
	y = grid[T.gy + (int)((local / T.nx) % T.ny)];
	t = grid[T.gf + (int)(local / ((long long)T.nx * T.ny))];
}

// ---------------------------------------------------------------------------
// mask(index[0]) = false (nldct.cpp:2325-2329, 2418-2422).  A group whose best
// match is not itself may switch off a later reference position; those rare
// cases become edges killer -> victim.  The index carries the channel stride
// (t*w*h*C + y*w + x) while the mask has one channel, so for C > 1 the cleared
// position is another frame of the mask; indices past the mask are ignored
// (the reference writes out of bounds there).
// ---------------------------------------------------------------------------
__global__ void kill_edges_kernel(const Tile *__restrict__ tiles, int ntiles,
                                  const int *__restrict__ grid, const int *__restrict__ inv,
                                  StepParams sp, long long G, const uint32_t *__restrict__ idx,
                                  unsigned long long *__restrict__ edges, unsigned *__restrict__ nedges,
                                  unsigned cap)
{
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < G;
	     g += (long long)gridDim.x * blockDim.x) {
		const Tile T = tiles[tile_of(tiles, ntiles, g)];
		int x, y, t;
		group_position(T, grid, g, x, y, t);
		const unsigned long long wh = (unsigned long long)T.w * T.h;
		const uint32_t lin = idx[g * sp.np];
		const unsigned long long mt = lin / wh, rem = lin % wh;
		// the reference's index value, interpreted as a one-channel mask index
		const unsigned long long m = mt * wh * sp.C + rem;
		const unsigned long long own = ((unsigned long long)t * T.h + y) * T.w + x;
		if (m >= wh * sp.F || m <= own) continue;
		const int tt = (int)(m / wh), ty = (int)((m % wh) / T.w), tx = (int)(m % T.w);
		const int xi = inv[T.gx + T.nx + tx];
		const int yi = inv[T.gy + T.ny + ty];
		const int fi = inv[T.gf + T.nf + tt];
		if (xi < 0 || yi < 0 || fi < 0) continue;
		const long long victim = T.g0 + ((long long)fi * T.ny + yi) * T.nx + xi;
		const unsigned e = atomicAdd(nedges, 1u);
		if (e < cap) edges[e] = ((unsigned long long)g << 32) | (unsigned long long)victim;
	}
}

// The switch-offs as a fixed point on the device: a victim is dead when a
// live killer points at it; repeat until nothing changes (at most n + 1
// rounds: every round that changes something settles at least one more
// group).  One CTA, so that the rounds need only CTA barriers.
__global__ void __launch_bounds__(1024)
kill_fixpoint_kernel(const unsigned long long *__restrict__ edges, const unsigned *__restrict__ nedges,
                     unsigned cap, uint8_t *__restrict__ alive, uint8_t *__restrict__ killed)
{
	__shared__ int changed;
	const unsigned n = min(*nedges, cap);
	for (unsigned round = 0; round <= n; round++) {
		for (unsigned e = threadIdx.x; e < n; e += blockDim.x) killed[edges[e] & 0xffffffffull] = 0;
		if (threadIdx.x == 0) changed = 0;
		__syncthreads();
		for (unsigned e = threadIdx.x; e < n; e += blockDim.x) {
			const unsigned long long v = edges[e];
			if (alive[v >> 32]) killed[v & 0xffffffffull] = 1;
		}
		__syncthreads();
		for (unsigned e = threadIdx.x; e < n; e += blockDim.x) {
			const long long w = (long long)(edges[e] & 0xffffffffull);
			const uint8_t a = killed[w] ? 0 : 1;
			if (alive[w] != a) {
				alive[w] = a;
				changed = 1;
			}
		}
		__syncthreads();
		if (!changed) break;
		__syncthreads();
	}
}

// Paste trick (doPasteBoost, nldct.cpp:2302-2322 and 2395-2415): a
// processed group switches off every member's position and its four
// neighbours outside the border band of 2*sPx (linear offsets -w, +w, -1, +1,
// so a band wider than the tile crosses rows; unsigned comparisons as the
// reference's).  Only reference positions are ever read from the mask, so a
// switch-off is an edge from a group to a later group of its tile, and a
// group is processed exactly when none of its killers is:
//     alive(g) = no alive k < g with an edge k -> g,
// the reference's sequential order restated as a recursion with one solution.
// It is evaluated by frontier rounds: a group is settled dead as soon as one
// killer is alive, alive once all its killers are dead (a count of pending
// killers per group); each settled group is pushed once and, when popped,
// settles or counts down its victims.  The first rounds run over the whole
// GPU, the tail in one CTA; every round count is fixed on the host side, so
// the sequence is stream ordered and graph capturable.
constexpr unsigned kUndecided = 0u, kAlive = 1u, kDead = 2u;

template <class Fn>
__device__ __forceinline__ void paste_victims(const Tile &T, const int *__restrict__ grid, const StepParams &sp,
                                              long long g, const uint8_t *__restrict__ nsimp,
                                              const uint32_t *__restrict__ idx, Fn fn)
{
	const unsigned w = (unsigned)T.w, h = (unsigned)T.h, band = 2u * (unsigned)sp.px, F = (unsigned)sp.F;
	const int ns = nsimp[g];
	for (int m = 0; m < ns; m++) {
		// member position as the one-channel mask index (t*h + y)*w + x
		const unsigned ind1 = idx[g * sp.np + m];
		const unsigned mx = ind1 % w, my = (ind1 / w) % h, mt = ind1 / (w * h);
#pragma unroll
		for (int q = 0; q < 5; q++) {
			unsigned vx = mx, vy = my, vt = mt;
			if (q == 1) { if (!(my > band)) continue; vy = my - 1; }
			if (q == 2) {
				if (!(my < h - band)) continue;
				if (++vy == h) { vy = 0; vt++; }
			}
			if (q == 3) { if (!(mx > band)) continue; vx = mx - 1; }
			if (q == 4) {
				if (!(mx < w - band)) continue;
				if (++vx == w) { vx = 0; if (++vy == h) { vy = 0; vt++; } }
			}
			if (vt >= F) continue;                          // past the mask
			const int xi = grid[T.gx + T.nx + vx], yi = grid[T.gy + T.ny + vy], fi = grid[T.gf + T.nf + vt];
			if (xi < 0 || yi < 0 || fi < 0) continue;       // not a reference position
			const long long v = T.g0 + ((long long)fi * T.ny + yi) * T.nx + xi;
			if (v > g) fn(v);                               // earlier groups are settled already
		}
	}
}

__global__ void paste_count_kernel(const Tile *__restrict__ tiles, int ntiles, const int *__restrict__ grid,
                                   StepParams sp, long long G, const uint8_t *__restrict__ nsimp,
                                   const uint32_t *__restrict__ idx, unsigned *__restrict__ pending)
{
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < G;
	     g += (long long)gridDim.x * blockDim.x) {
		const Tile T = tiles[tile_of(tiles, ntiles, g)];
		paste_victims(T, grid, sp, g, nsimp, idx, [&](long long v) { atomicAdd(&pending[v], 1u); });
	}
}

__global__ void paste_init_kernel(long long G, const unsigned *__restrict__ pending, unsigned *__restrict__ state,
                                  uint32_t *__restrict__ queue, unsigned *__restrict__ count)
{
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < G;
	     g += (long long)gridDim.x * blockDim.x) {
		const bool free_ = pending[g] == 0u;
		state[g] = free_ ? kAlive : kUndecided;
		if (free_) queue[atomicAdd(count, 1u)] = (uint32_t)g;
	}
}

// Pops group g: an alive group settles its undecided victims dead, a dead
// one counts them down (the last killer to die settles a victim alive).
__device__ __forceinline__ void paste_settle(const Tile *__restrict__ tiles, int ntiles,
                                             const int *__restrict__ grid, const StepParams &sp, long long g,
                                             const uint8_t *__restrict__ nsimp, const uint32_t *__restrict__ idx,
                                             unsigned *state, unsigned *pending, uint32_t *qout, unsigned *nout)
{
	const Tile T = tiles[tile_of(tiles, ntiles, g)];
	const unsigned sg = state[g];
	paste_victims(T, grid, sp, g, nsimp, idx, [&](long long v) {
		if (sg == kAlive) {
			if (atomicCAS(&state[v], kUndecided, kDead) == kUndecided) qout[atomicAdd(nout, 1u)] = (uint32_t)v;
		} else if (atomicSub(&pending[v], 1u) == 1u) {
			if (atomicCAS(&state[v], kUndecided, kAlive) == kUndecided) qout[atomicAdd(nout, 1u)] = (uint32_t)v;
		}
	});
}

__global__ void paste_round_kernel(const Tile *__restrict__ tiles, int ntiles, const int *__restrict__ grid,
                                   StepParams sp, const uint8_t *__restrict__ nsimp,
                                   const uint32_t *__restrict__ idx, unsigned *state, unsigned *pending,
                                   const uint32_t *__restrict__ qin, const unsigned *__restrict__ nin,
                                   uint32_t *__restrict__ qout, unsigned *nout)
{
	const unsigned n = *nin;
	for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		paste_settle(tiles, ntiles, grid, sp, qin[i], nsimp, idx, state, pending, qout, nout);
}

// The remaining rounds in one CTA (small frontiers), until the frontier is
// empty: every group is pushed at most once, so at most G + 1 rounds.
__global__ void __launch_bounds__(1024)
paste_finish_kernel(const Tile *__restrict__ tiles, int ntiles, const int *__restrict__ grid, StepParams sp,
                    long long G, const uint8_t *__restrict__ nsimp, const uint32_t *__restrict__ idx,
                    unsigned *state, unsigned *pending, uint32_t *q0, uint32_t *q1, unsigned *n_in,
                    unsigned *n_pair)
{
	uint32_t *qin = q0, *qout = q1;
	unsigned *nin = n_in;
	for (long long r = 0; r <= G; r++) {
		unsigned *nout = n_pair + (r & 1);
		if (threadIdx.x == 0) *nout = 0u;
		__syncthreads();
		const unsigned n = *(volatile unsigned *)nin;
		if (n == 0u) break;
		for (unsigned i = threadIdx.x; i < n; i += blockDim.x)
			paste_settle(tiles, ntiles, grid, sp, qin[i], nsimp, idx, state, pending, qout, nout);
		__syncthreads();
		uint32_t *t = qin;
		qin = qout;
		qout = t;
		nin = nout;
	}
}

__global__ void paste_alive_kernel(long long G, const unsigned *__restrict__ state, uint8_t *__restrict__ alive)
{
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < G;
	     g += (long long)gridDim.x * blockDim.x)
		alive[g] = state[g] == kAlive ? 1 : 0;
}

__global__ void count_alive_kernel(const Tile *__restrict__ tiles, int ntiles, long long G,
                                   const uint8_t *__restrict__ alive, unsigned *__restrict__ counts)
{
	// per-thread counts of the current tile, then one atomic per group of
	// lanes holding the same tile (one counter per tile: plain per-group
	// atomics serialise on it)
	int ct = -1;
	unsigned cnt = 0;
	for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < G;
	     g += (long long)gridDim.x * blockDim.x) {
		if (!alive[g]) continue;
		const int t = tile_of(tiles, ntiles, g);
		if (t != ct) {
			if (cnt) atomicAdd(&counts[ct], cnt);
			ct = t;
			cnt = 0;
		}
		cnt++;
	}
	const unsigned same = __match_any_sync(0xffffffffu, ct);
	const unsigned total = __reduce_add_sync(same, cnt);
	if (ct >= 0 && total && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&counts[ct], total);
}

// places held before they are looked up and added: 512 / 1024 / 2048 took 130 /
// 116 / 144 ms on 1920x1080x24 (barriers against resident CTAs)
constexpr int kGatherThreads = 128, kEntCap = 1024;

// ---------------------------------------------------------------------------
// bins: 16 x 16 pixels x BT frames of one tile (BT = 1 for one-frame patches,
// else 4).  Every member patch ("slot") is listed in each bin it touches; a
// CTA then adds one bin's slots to its pixels in slot order.
//
// The lists are small (about 2.5 entries of 4 bytes per 4x4x4 member, 2.1 per
// 8x8 one) and their order does not matter: the gather orders a bin's slots
// by a bitmap over the groups around it.  Aggregation with k-way merges of
// per-pixel lists (and a weight beside every estimate) -> with bins:
// 256x256 image, 8x8 patches 6.4 -> 0.37 ms; 767x511 colour image, defaults
// 30.1 -> 2.1 ms; 853x481x16, defaults 35.4 -> 1.9 ms; 1920x1080x24, 4x4x4
// patches 144 -> 114 ms.  Those merges kept 64 list heads in local memory for
// 8x8 patches; here a slot is listed once per bin, and its terms are half the
// bytes.
// ---------------------------------------------------------------------------
struct BinRange {
	int x0, x1, y0, y1, t0, t1;   // first and last bin along each axis
};

__device__ __forceinline__ BinRange bins_of(const Tile &T, const StepParams &sp, uint32_t lin)
{
	const uint32_t wh = (uint32_t)T.w * T.h;
	const int t = (int)(lin / wh), r = (int)(lin % wh), y = r / T.w, x = r % T.w;
	const int bt = bin_frames(sp.px, sp.pt);
	BinRange b;
	b.x0 = x / kBinX;
	b.x1 = (x + sp.px - 1) / kBinX;
	b.y0 = y / kBinY;
	b.y1 = (y + sp.px - 1) / kBinY;
	b.t0 = t / bt;
	b.t1 = (t + sp.pt - 1) / bt;
	return b;
}

// FILL = false: entries per bin; FILL = true: the entries, at the cursors.
//
// Neighbouring groups touch the same few bins, so plain atomics on the bins'
// counters serialise (10 G entries/s on 4x4x4 patches).  A CTA therefore takes
// kListSlots consecutive slots, counts their entries per bin in a small hash
// table in shared memory, and takes each bin's share with one atomic.  An entry
// that finds no place in the table (members spread over more bins than it
// holds) goes to the global counter by itself.
constexpr int kListThreads = 256, kListSlots = 1024, kListTable = 1024, kListProbes = 16;

template <bool FILL>
__global__ void __launch_bounds__(kListThreads)
bin_list_kernel(const Tile *__restrict__ tiles, int ntiles, StepParams sp, long long ga, long long gb,
                const uint8_t *__restrict__ nsimp, const uint32_t *__restrict__ idx,
                const uint8_t *__restrict__ alive, unsigned *__restrict__ cnt, unsigned *__restrict__ list)
{
	__shared__ unsigned s_key[kListTable], s_cnt[kListTable];   // s_cnt: entries, then the next list place
	const unsigned np = sp.np;
	const long long nslots = (gb - ga) * (long long)np;
	for (long long s0 = (long long)blockIdx.x * kListSlots; s0 < nslots; s0 += (long long)gridDim.x * kListSlots) {
		for (int i = threadIdx.x; i < kListTable; i += kListThreads) {
			s_key[i] = 0xffffffffu;
			s_cnt[i] = 0u;
		}
		__syncthreads();
		for (int pass = 0; pass < (FILL ? 2 : 1); pass++) {
			for (int k = threadIdx.x; k < kListSlots && s0 + k < nslots; k += kListThreads) {
				const unsigned slot = (unsigned)(s0 + k);   // chunk-relative
				const long long g = ga + slot / np;
				const int n = (int)(slot % np);
				if (!alive[g] || n >= nsimp[g]) continue;
				const Tile T = tiles[tile_of(tiles, ntiles, g)];
				const BinRange b = bins_of(T, sp, idx[g * np + n]);
				for (int t = b.t0; t <= b.t1; t++)
					for (int y = b.y0; y <= b.y1; y++)
						for (int x = b.x0; x <= b.x1; x++) {
							const unsigned bin = (unsigned)(T.bin0 + ((long long)t * T.nby + y) * T.nbx + x);
							unsigned h = bin * 2654435761u >> 22;   // kListTable = 1024 places
							int tries = 0;
							for (; tries < kListProbes; tries++, h = (h + 1) & (kListTable - 1)) {
								const unsigned key = pass ? s_key[h] : atomicCAS(&s_key[h], 0xffffffffu, bin);
								if (key == bin || (!pass && key == 0xffffffffu)) break;
							}
							if (tries < kListProbes) {
								const unsigned at = atomicAdd(&s_cnt[h], 1u);
								if (FILL && pass) list[at] = slot;
							} else if (FILL == (pass != 0)) {
								const unsigned at = atomicAdd(&cnt[bin], 1u);
								if (FILL) list[at] = slot;
							}
						}
			}
			__syncthreads();
			if (pass == 0)
				for (int i = threadIdx.x; i < kListTable; i += kListThreads)
					if (s_cnt[i]) s_cnt[i] = atomicAdd(&cnt[s_key[i]], s_cnt[i]);
			__syncthreads();
		}
	}
}

// List space of every bin that has entries (in any order of the bins), the
// fill cursors, and the non-empty bins.  heads: [0] list space taken, [1]
// non-empty bins, [2] the gather's next bin.
__global__ void bin_alloc_kernel(unsigned nbins, const unsigned *__restrict__ cnt, unsigned *__restrict__ cursor,
                                 unsigned *__restrict__ bins, unsigned *__restrict__ heads)
{
	const unsigned lane = threadIdx.x & 31u;
	for (unsigned b0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; b0 < nbins; b0 += gridDim.x * blockDim.x) {
		const unsigned b = b0 + lane;
		const unsigned c = b < nbins ? cnt[b] : 0u;
		unsigned s = c;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const unsigned u = __shfl_up_sync(0xffffffffu, s, o);
			if (lane >= (unsigned)o) s += u;
		}
		const unsigned full = __ballot_sync(0xffffffffu, c != 0u);
		if (full == 0u) continue;
		unsigned base = 0, at = 0;
		if (lane == 31) {
			base = atomicAdd(&heads[0], s);
			at = atomicAdd(&heads[1], (unsigned)__popc(full));
		}
		base = __shfl_sync(0xffffffffu, base, 31);
		at = __shfl_sync(0xffffffffu, at, 31);
		if (c) {
			cursor[b] = base + s - c;
			bins[at + __popc(full & ((1u << lane) - 1u))] = b;
		}
	}
}

// Adds a column of PX terms w * v to the rows R .. R + PX - 1 of a lane's 8 sums.  The
// markers keep the compiler from merging the cases of R into one that indexes
// the sums dynamically, which would put them in local memory.
template <int R, int PX, int CC>
__device__ __forceinline__ void add_rows(float (&a)[8][CC], float (&wa)[8], const float (&v)[CC][PX], float w)
{
	asm volatile("" ::"n"(R));
#pragma unroll
	for (int h = 0; h < PX; h++)
		if (R + h >= 0 && R + h < 8) {
#pragma unroll
			for (int c = 0; c < CC; c++) a[(R + h) & 7][c] = __fadd_rn(a[(R + h) & 7][c], __fmul_rn(w, v[c][h]));
			wa[(R + h) & 7] = __fadd_rn(wa[(R + h) & 7], w);
		}
	asm volatile("" ::"n"(R + 16));
}

__device__ __forceinline__ void load_column(const float *p, float (&v)[4])
{
	const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
	v[0] = q.x;
	v[1] = q.y;
	v[2] = q.z;
	v[3] = q.w;
}

__device__ __forceinline__ void load_column(const float *p, float (&v)[2])
{
	const float2 q = __ldg(reinterpret_cast<const float2 *>(p));
	v[0] = q.x;
	v[1] = q.y;
}

// Ordered gather of one bin per CTA at a time.
//
// Order: the slots of a bin come from groups of a small box of the reference
// grid (about 25 x 25 x 15 groups for 4x4x4 patches), and a slot's place in
// the box -- (frame, row, column, member), row by row -- rises with its
// number.  So the CTA marks its slots in a bitmap over the box and reads the
// marks back in order.  A box larger than the bitmap is taken in several
// passes, each starting at the first mark not yet taken, so any spread of the
// members is served.
//
// Sums: each of the four warps owns 8 x 8 pixels x BT frames, with their sums
// in registers, and adds a slot's terms to the pixels the slot covers, slots in
// order: the order of the reference's scatter loop for every pixel.  Only the
// terms a lane needs are loaded, each once; U slots' loads are in flight before
// the first is added.  4x4 patches and 2x2 ones of several frames: a lane owns one column of 8
// pixels of one of four frames; the patch's terms of that column and frame are one 16- or
// 8-byte load (term_of orders them so), and the rows they fall on are the same
// for the whole warp.  Other patches: a lane owns pixels (x, y) and (x, y + 4); by
// that mapping 2x2x4 patches took 11.3 ms (240x180x8), by columns 6.3.
template <int PX, int BT, int CC, int U>
__global__ void __launch_bounds__(kGatherThreads)
bin_gather_kernel(const Tile *__restrict__ tiles, int ntiles, StepParams sp, long long ga,
                  const uint32_t *__restrict__ idx, const float *__restrict__ vals, const float *__restrict__ wslot,
                  const float *__restrict__ win, const unsigned *__restrict__ cnt,
                  const unsigned *__restrict__ cursor, const unsigned *__restrict__ bins, unsigned *__restrict__ heads,
                  const unsigned *__restrict__ list, float *__restrict__ acc, float *__restrict__ wacc)
{
	constexpr int kBitWords = BT == 1 ? 512 : 2048;
	constexpr bool kColumn = PX == 4 || PX == 2;
	static_assert(!kColumn || BT == 4, "a lane's frame is one of four");
	__shared__ unsigned s_bits[kBitWords];
	__shared__ uint4 s_ent[kEntCap];         // slot, place relative to the bin, weight
	__shared__ float s_win[64];
	__shared__ unsigned s_warp[2][kGatherThreads / 32];
	__shared__ int s_box[6];
	__shared__ unsigned s_bin;
	__shared__ unsigned long long s_next;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int px = PX ? PX : sp.px, pt = sp.pt, np = sp.np, spc = px * px * pt;
	const unsigned nfull = heads[1];
	for (int i = tid; i < px * px; i += kGatherThreads) s_win[i] = win[i];
	for (;;) {
		__syncthreads();
		if (tid == 0) s_bin = atomicAdd(&heads[2], 1u);
		if (tid < 6) s_box[tid] = (tid & 1) ? -1 : 0x7fffffff;
		__syncthreads();
		if (s_bin >= nfull) break;
		const unsigned bin = bins[s_bin];
		int ti = 0;
		while (ti + 1 < ntiles && tiles[ti + 1].bin0 <= (long long)bin) ti++;
		const Tile T = tiles[ti];
		const int lb = (int)((long long)bin - T.bin0);
		const int X0 = lb % T.nbx * kBinX, Y0 = lb / T.nbx % T.nby * kBinY, F0 = lb / (T.nbx * T.nby) * BT;
		const unsigned n = cnt[bin];
		const unsigned *lst = list + (cursor[bin] - n);   // the cursor stands past the last entry
		const unsigned l0 = (unsigned)(ga - T.g0);        // of the tile's first group in the chunk (may wrap)
		const unsigned wh = (unsigned)T.w * T.h;
		const unsigned nx = T.nx, ny = T.ny;

		// the box of groups
		{
			int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
			for (unsigned i = tid; i < n; i += kGatherThreads) {
				const unsigned l = l0 + lst[i] / np, r = l / nx;
				const int v[3] = {(int)(l % nx), (int)(r % ny), (int)(r / ny)};
#pragma unroll
				for (int k = 0; k < 3; k++) { lo[k] = min(lo[k], v[k]); hi[k] = max(hi[k], v[k]); }
			}
#pragma unroll
			for (int k = 0; k < 3; k++) {
				lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
				hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
				if (lane == 0) { atomicMin(&s_box[2 * k], lo[k]); atomicMax(&s_box[2 * k + 1], hi[k]); }
			}
		}
		__syncthreads();
		const int gx0 = s_box[0], gy0 = s_box[2], gt0 = s_box[4];
		const unsigned bnx = (unsigned)(s_box[1] - gx0 + 1), bny = (unsigned)(s_box[3] - gy0 + 1);
		const unsigned long long volume = (unsigned long long)(s_box[5] - gt0 + 1) * bny * bnx * np;
		auto place = [&](unsigned slot) -> unsigned long long {
			const unsigned q = slot / np, l = l0 + q, r = l / nx;
			const unsigned x = l % nx - gx0, y = r % ny - gy0, t = r / ny - gt0;
			return ((unsigned long long)(t * bny + y) * bnx + x) * np + (slot - q * np);
		};

		// this warp's pixels; sum s of a lane is pixel (x, ly(s)) of frame lf(s)
		const int qx = X0 + (warp & 1) * 8, qy = Y0 + (warp >> 1) * 8;
		const int x = qx + (lane & 7), y = qy + (lane >> 3);
		constexpr int NS = kColumn ? 8 : 2 * BT;
		auto ly = [&](int s) { return kColumn ? qy + s : y + 4 * (s & 1); };
		auto lf = [&](int s) { return kColumn ? F0 + (lane >> 3) : F0 + (s >> 1); };
		float a[NS][CC], wa[NS];
#pragma unroll
		for (int s = 0; s < NS; s++) {
			const bool in = x < T.w && ly(s) < T.h && lf(s) < sp.F;
			const size_t at = (size_t)ly(s) * T.w + x;
#pragma unroll
			for (int c = 0; c < CC; c++) a[s][c] = in ? acc[T.pix0 * CC + ((size_t)lf(s) * CC + c) * wh + at] : 0.f;
			wa[s] = in ? wacc[T.pix0 + (size_t)lf(s) * wh + at] : 0.f;
		}

		unsigned long long p0 = 0;
		for (;;) {
			// marks of the slots at places [p0, p0 + bits)
			for (int i = tid; i < kBitWords; i += kGatherThreads) s_bits[i] = 0u;
			if (tid == 0) s_next = ~0ull;
			__syncthreads();
			unsigned long long nxt = ~0ull;
			for (unsigned i = tid; i < n; i += kGatherThreads) {
				const unsigned long long p = place(lst[i]);
				if (p < p0) continue;
				if (p - p0 < (unsigned long long)kBitWords * 32u) atomicOr(&s_bits[(unsigned)(p - p0) >> 5], 1u << ((unsigned)(p - p0) & 31u));
				else nxt = p < nxt ? p : nxt;
			}
			if (nxt != ~0ull) atomicMin(&s_next, nxt);
			__syncthreads();
			const unsigned q0 = (unsigned)(p0 / np), m0 = (unsigned)(p0 - (unsigned long long)q0 * np);
			const int words = (int)min((unsigned long long)kBitWords, (volume - p0 + 31) / 32);
			// the marks in order, one word per thread and round; the places found
			// gather in s_ent until it is full (or the words run out)
			unsigned have = 0;
			for (int w0 = 0, odd = 0;; w0 += kGatherThreads, odd ^= 1) {
				const bool last = w0 >= words;
				unsigned bits = last ? 0u : s_bits[w0 + tid], rank = 0, total = 0;
				if (!last) {
					const unsigned c = __popc(bits);
					unsigned s = c;
#pragma unroll
					for (int o = 1; o < 32; o <<= 1) {
						const unsigned u = __shfl_up_sync(0xffffffffu, s, o);
						if (lane >= o) s += u;
					}
					if (lane == 31) s_warp[odd][warp] = s;
					__syncthreads();
					rank = s - c;
#pragma unroll
					for (int k = 0; k < kGatherThreads / 32; k++) {
						if (k < warp) rank += s_warp[odd][k];
						total += s_warp[odd][k];
					}
				}
				unsigned done = 0;
				while (done < total || (last && have)) {
					const unsigned room = (unsigned)kEntCap - have;
					while (bits && rank - done < room) {
						const int b = __ffs(bits) - 1;
						bits &= bits - 1;
						s_ent[have + rank - done].x = (unsigned)((w0 + tid) * 32 + b);
						rank++;
					}
					const unsigned put = min(room, total - done);
					have += put;
					done += put;
					if (have < (unsigned)kEntCap && !last) continue;
					const int ne = (int)have;
					have = 0;
					__syncthreads();
					for (int e = tid; e < ne; e += kGatherThreads) {
						const unsigned p = m0 + s_ent[e].x, qq = p / np, m = p - qq * np, q = q0 + qq;
						const unsigned gx = q % bnx + gx0, r = q / bnx, gy = r % bny + gy0, gt = r / bny + gt0;
						const unsigned slot = ((gt * ny + gy) * nx + gx - l0) * np + m;
						const unsigned lin = __ldg(idx + (size_t)ga * np + slot);
						const int ot = (int)(lin / wh), rr = (int)(lin % wh), oy = rr / T.w, ox = rr % T.w;
						s_ent[e] = make_uint4(slot, (unsigned)(ox - X0 + 8) | (unsigned)(oy - Y0 + 8) << 8 |
						                                (unsigned)(ot - F0 + 16) << 16,
						                      __float_as_uint(__ldg(wslot + slot)), 0u);
					}
					__syncthreads();
					for (int e = 0; e < ne; e += 32) {
						bool hit = false;
						if (e + lane < ne) {
							const unsigned pos = s_ent[e + lane].y;
							const int rx = (int)(pos & 255u) - 8 + X0 - qx, ry = (int)(pos >> 8 & 255u) - 8 + Y0 - qy;
							hit = rx < 8 && rx + px > 0 && ry < 8 && ry + px > 0;
						}
						unsigned m = __ballot_sync(0xffffffffu, hit);
						if constexpr (kColumn) {
							while (m) {
								float v[U][CC][PX ? PX : 1];
								float wt[U];
								int row[U];
								bool ok[U];
#pragma unroll
								for (int u = 0; u < U; u++) {
									row[u] = -PX;
									ok[u] = false;
									if (!m) continue;
									const uint4 q = s_ent[e + __ffs(m) - 1];
									m &= m - 1;
									const unsigned dx = (unsigned)(x - X0 + 8) - (q.y & 255u);
									const unsigned dt = (unsigned)((lane >> 3) + 16) - (q.y >> 16);
									row[u] = (int)(q.y >> 8 & 255u) - 8 + Y0 - qy;
									ok[u] = dx < (unsigned)PX && dt < (unsigned)pt;
									wt[u] = __uint_as_float(q.z);   // no window for these patches
									const float *col = vals + (size_t)q.x * (spc * CC) + (dt * PX + dx) * PX;
#pragma unroll
									for (int c = 0; c < CC; c++)
										if (ok[u]) load_column(col + c * spc, v[u][c]);
								}
#pragma unroll
								for (int u = 0; u < U; u++)
									if (ok[u]) {
										switch (row[u]) {   // the same for the whole warp
										case -3: add_rows<-3, PX>(a, wa, v[u], wt[u]); break;
										case -2: add_rows<-2, PX>(a, wa, v[u], wt[u]); break;
										case -1: add_rows<-1, PX>(a, wa, v[u], wt[u]); break;
										case 0: add_rows<0, PX>(a, wa, v[u], wt[u]); break;
										case 1: add_rows<1, PX>(a, wa, v[u], wt[u]); break;
										case 2: add_rows<2, PX>(a, wa, v[u], wt[u]); break;
										case 3: add_rows<3, PX>(a, wa, v[u], wt[u]); break;
										case 4: add_rows<4, PX>(a, wa, v[u], wt[u]); break;
										case 5: add_rows<5, PX>(a, wa, v[u], wt[u]); break;
										case 6: add_rows<6, PX>(a, wa, v[u], wt[u]); break;
										case 7: add_rows<7, PX>(a, wa, v[u], wt[u]); break;
										}
									}
							}
						} else {
							while (m) {
								float v[U][NS][CC], wt[U][2];
								unsigned fm[U];
								bool ok[U][2];
#pragma unroll
								for (int u = 0; u < U; u++) {
									fm[u] = 0u;
									ok[u][0] = ok[u][1] = false;
									if (!m) continue;
									const uint4 q = s_ent[e + __ffs(m) - 1];
									m &= m - 1;
									const int dx = x - X0 + 8 - (int)(q.y & 255u), dy = y - Y0 + 8 - (int)(q.y >> 8 & 255u);
									const int rt = (int)(q.y >> 16) - 16;
									const bool okx = (unsigned)dx < (unsigned)px;
									ok[u][0] = okx && (unsigned)dy < (unsigned)px;
									ok[u][1] = okx && (unsigned)(dy + 4) < (unsigned)px;
									const float *row = vals + (size_t)q.x * (spc * CC);
#pragma unroll
									for (int h = 0; h < 2; h++) {
										const int d = (dy + 4 * h) * px + dx;
										// as the reference forms it
										wt[u][h] = ok[u][h] ? __fmul_rn(__uint_as_float(q.z), s_win[d]) : 0.f;
#pragma unroll
										for (int f = 0; f < BT; f++) {
											const int dt = f - rt;
											if ((unsigned)dt >= (unsigned)pt) continue;
											fm[u] |= 1u << f;
#pragma unroll
											for (int c = 0; c < CC; c++)
												if (ok[u][h]) v[u][2 * f + h][c] = __ldg(row + (c * spc + dt * px * px + d));
										}
									}
								}
#pragma unroll
								for (int u = 0; u < U; u++)
#pragma unroll
									for (int s = 0; s < NS; s++)
										if ((fm[u] >> (s >> 1) & 1u) && ok[u][s & 1]) {
#pragma unroll
											for (int c = 0; c < CC; c++) a[s][c] = __fadd_rn(a[s][c], __fmul_rn(wt[u][s & 1], v[u][s][c]));
											wa[s] = __fadd_rn(wa[s], wt[u][s & 1]);
										}
							}
						}
					}
					__syncthreads();
				}
				if (last) break;
			}
			p0 = s_next;
			__syncthreads();
			if (p0 == ~0ull) break;
		}
#pragma unroll
		for (int s = 0; s < NS; s++) {
			if (!(x < T.w && ly(s) < T.h && lf(s) < sp.F)) continue;
			const size_t at = (size_t)ly(s) * T.w + x;
#pragma unroll
			for (int c = 0; c < CC; c++) acc[T.pix0 * CC + ((size_t)lf(s) * CC + c) * wh + at] = a[s][c];
			wacc[T.pix0 + (size_t)lf(s) * wh + at] = wa[s];
		}
	}
}

template <int PX, int BT, int CC, int U>
cudaError_t gather_t(const BinArgs &a, const Tile *tiles, int ntiles, const StepParams &sp, long long ga,
                     const uint32_t *idx, const float *vals, const float *wslot, const float *win, float *acc,
                     float *wacc, int nsm, cudaStream_t st)
{
	auto kern = bin_gather_kernel<PX, BT, CC, U>;
	int per_sm = 0;
	cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kGatherThreads, 0);
	if (e != cudaSuccess) return e;
	const long long blocks = std::min<long long>((long long)nsm * std::max(per_sm, 1), a.nbins);
	kern<<<(int)blocks, kGatherThreads, 0, st>>>(tiles, ntiles, sp, ga, idx, vals, wslot, win, a.cnt, a.cursor, a.bins,
	                                            a.heads, a.list, acc, wacc);
	return cudaGetLastError();
}

// Slots whose loads are in flight: 4x4 patches take one 16-byte load per
// channel (2 / 4 slots: 117 / 114 ms of aggregation on 1920x1080x24, 16.2 /
// 14.7 ms on 640x360x3x14; 8 by gather_depth 2), the others one or two 4-byte
// loads per frame and channel.
template <int CC, class... Args>
cudaError_t gather_c(const StepParams &sp, Args... args)
{
	if (sp.px == 4) return sp.gather_depth == 2 && CC == 1 ? gather_t<4, 4, CC, CC == 1 ? 8 : 4>(args...) : gather_t<4, 4, CC, 4>(args...);
	if (sp.px == 2 && sp.pt != 1) return gather_t<2, 4, CC, 4>(args...);
	if (sp.pt != 1) return gather_t<0, 4, CC, 1>(args...);
	if (sp.px == 7) return gather_t<7, 1, CC, CC == 1 ? 4 : 2>(args...);
	if (sp.px == 8) return gather_t<8, 1, CC, CC == 1 ? 4 : 2>(args...);
	return gather_t<0, 1, CC, 2>(args...);
}

// ---------------------------------------------------------------------------
// colour transforms (src/utils/lib_videot.hpp:727-838), same float expressions
// ---------------------------------------------------------------------------
__device__ __forceinline__ void yuv_forward(float *v, int C)
{
	if (C == 3) {
		const float a = __fdiv_rn(1.f, sqrtf(3.f));
		const float b = __fdiv_rn(1.f, sqrtf(2.f));
		const float c = __fmul_rn(__fmul_rn(2.f, a), sqrtf(2.f));
		const float r = v[0], g = v[1], bl = v[2];
		v[0] = __fmul_rn(a, __fadd_rn(__fadd_rn(r, g), bl));
		v[1] = __fmul_rn(b, __fsub_rn(r, bl));
		v[2] = __fmul_rn(c, __fadd_rn(__fsub_rn(__fmul_rn(0.25f, r), __fmul_rn(0.5f, g)), __fmul_rn(0.25f, bl)));
	} else if (C == 4) {
		const float a = 0.5f;
		const float b = __fdiv_rn(1.f, sqrtf(2.f));
		const float Gr = v[0], R = v[1], B = v[2], Gb = v[3];
		v[0] = __fmul_rn(a, __fadd_rn(__fadd_rn(__fadd_rn(Gr, R), B), Gb));
		v[1] = __fmul_rn(b, __fsub_rn(R, B));
		v[2] = __fmul_rn(a, __fsub_rn(__fadd_rn(__fadd_rn(-Gr, R), B), Gb));
		v[3] = __fmul_rn(b, __fadd_rn(-Gr, Gb));
	}
}

__device__ __forceinline__ void yuv_inverse(float *v, int C)
{
	if (C == 3) {
		const float a = __fdiv_rn(1.f, sqrtf(3.f));
		const float b = __fdiv_rn(1.f, sqrtf(2.f));
		const float c = __fdiv_rn(a, b);
		const float ch = __fmul_rn(c, 0.5f);
		const float y = v[0], u = v[1], w = v[2];
		v[0] = __fadd_rn(__fadd_rn(__fmul_rn(a, y), __fmul_rn(b, u)), __fmul_rn(ch, w));
		v[1] = __fsub_rn(__fmul_rn(a, y), __fmul_rn(c, w));
		v[2] = __fadd_rn(__fsub_rn(__fmul_rn(a, y), __fmul_rn(b, u)), __fmul_rn(ch, w));
	} else if (C == 4) {
		const float a = 0.5f;
		const float b = __fdiv_rn(1.f, sqrtf(2.f));
		const float Gr = v[0], R = v[1], B = v[2], Gb = v[3];
		v[0] = __fsub_rn(__fsub_rn(__fmul_rn(a, Gr), __fmul_rn(a, B)), __fmul_rn(b, Gb));
		v[1] = __fadd_rn(__fadd_rn(__fmul_rn(a, Gr), __fmul_rn(b, R)), __fmul_rn(a, B));
		v[2] = __fadd_rn(__fsub_rn(__fmul_rn(a, Gr), __fmul_rn(b, R)), __fmul_rn(a, B));
		v[3] = __fadd_rn(__fsub_rn(__fmul_rn(a, Gr), __fmul_rn(a, B)), __fmul_rn(b, Gb));
	}
}

__global__ void color_kernel(Image in, Image out, int forward)
{
	const long long n = (long long)in.W * in.H * in.F;
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
	     i += (long long)gridDim.x * blockDim.x) {
		const int x = (int)(i % in.W), y = (int)((i / in.W) % in.H), t = (int)(i / ((long long)in.W * in.H));
		float v[4];
		for (int c = 0; c < in.C; c++) v[c] = in.p[in.at(x, y, t, c)];
		if (forward) yuv_forward(v, in.C); else yuv_inverse(v, in.C);
		for (int c = 0; c < in.C; c++) out.p[out.at(x, y, t, c)] = v[c];
	}
}

// computeWeightedAggregation (nldct.cpp:2436-2448) on every tile, then the
// inner-region rebuild of subBuildTight (lib_videot.hpp:1101-1163) and the
// inverse colour transform: one thread per output pixel.
__global__ void finalize_kernel(const Tile *__restrict__ tiles, int nW, int wTmp, int hTmp, StepParams sp,
                                Image noisy, const float *__restrict__ acc, const float *__restrict__ wacc,
                                Image out, int inverse_color)
{
	const long long n = (long long)out.W * out.H * out.F;
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
	     i += (long long)gridDim.x * blockDim.x) {
		const int X = (int)(i % out.W), Y = (int)((i / out.W) % out.H);
		const int t = (int)(i / ((long long)out.W * out.H));
		const Tile T = tiles[(Y / hTmp) * nW + X / wTmp];
		const int x = X - T.ox, y = Y - T.oy;
		const size_t pix = ((size_t)t * T.h + y) * T.w + x;
		const float wt = wacc[T.pix0 + pix];
		float v[4];
		for (int c = 0; c < sp.C; c++) {
			const float a = acc[T.pix0 * sp.C + (((size_t)t * sp.C + c) * T.h + y) * T.w + x];
			v[c] = wt > 0.f ? __fdiv_rn(a, wt) : __fdiv_rn(a, noisy.p[noisy.at(X, Y, t, c)]);
		}
		if (inverse_color) yuv_inverse(v, sp.C);
		for (int c = 0; c < sp.C; c++) out.p[out.at(X, Y, t, c)] = v[c];
	}
}

inline int grid_for(long long n, int threads, int cap = 65535)
{
	long long b = (n + threads - 1) / threads;
	if (b < 1) b = 1;
	return (int)(b < cap ? b : cap);
}

}  // namespace

cudaError_t launch_kill_edges(const Tile *tiles, int ntiles, const int *grid, const int *inv,
                              const StepParams &sp, long long G, const uint32_t *idx,
                              unsigned long long *edges, unsigned *nedges, unsigned cap, cudaStream_t st)
{
	kill_edges_kernel<<<grid_for(G, 256, 8192), 256, 0, st>>>(tiles, ntiles, grid, inv, sp, G, idx, edges, nedges, cap);
	return cudaGetLastError();
}

cudaError_t launch_kill_fixpoint(const unsigned long long *edges, const unsigned *nedges, unsigned cap,
                                 uint8_t *alive, uint8_t *killed, cudaStream_t st)
{
	kill_fixpoint_kernel<<<1, 1024, 0, st>>>(edges, nedges, cap, alive, killed);
	return cudaGetLastError();
}

cudaError_t launch_paste_resolve(const Tile *tiles, int ntiles, const int *grid, const StepParams &sp, long long G,
                                 const uint8_t *nsimp, const uint32_t *idx, PasteScratch w, uint8_t *alive, int nsm,
                                 cudaStream_t st)
{
	if (G <= 0) return cudaSuccess;
	cudaError_t e = cudaMemsetAsync(w.pending, 0, sizeof(unsigned) * (size_t)G, st);
	if (e == cudaSuccess) e = cudaMemsetAsync(w.counts, 0, sizeof(unsigned) * (kPasteRounds + 3), st);
	if (e != cudaSuccess) return e;
	const int b = grid_for(G, 256, 8 * nsm);
	paste_count_kernel<<<b, 256, 0, st>>>(tiles, ntiles, grid, sp, G, nsimp, idx, w.pending);
	paste_init_kernel<<<b, 256, 0, st>>>(G, w.pending, w.state, w.q0, w.counts);
	// the wide rounds: round r reads counts[r] and queue r & 1
	for (int r = 0; r < kPasteRounds; r++)
		paste_round_kernel<<<b, 256, 0, st>>>(tiles, ntiles, grid, sp, nsimp, idx, w.state, w.pending,
		                                      (r & 1) ? w.q1 : w.q0, w.counts + r, (r & 1) ? w.q0 : w.q1,
		                                      w.counts + r + 1);
	const bool odd = (kPasteRounds & 1) != 0;
	paste_finish_kernel<<<1, 1024, 0, st>>>(tiles, ntiles, grid, sp, G, nsimp, idx, w.state, w.pending,
	                                        odd ? w.q1 : w.q0, odd ? w.q0 : w.q1, w.counts + kPasteRounds,
	                                        w.counts + kPasteRounds + 1);
	paste_alive_kernel<<<b, 256, 0, st>>>(G, w.state, alive);
	return cudaGetLastError();
}

cudaError_t launch_count_alive(const Tile *tiles, int ntiles, long long G, const uint8_t *alive,
                               unsigned *counts, cudaStream_t st)
{
	count_alive_kernel<<<grid_for(G, 256, 8192), 256, 0, st>>>(tiles, ntiles, G, alive, counts);
	return cudaGetLastError();
}

int bin_entries_per_member(const StepParams &sp)
{
	const int bt = bin_frames(sp.px, sp.pt), s = sp.px > 1 ? 2 : 1;
	return s * s * ((sp.pt + bt - 2) / bt + 1);
}

cudaError_t launch_aggregate(const BinArgs &a, const Tile *tiles, int ntiles, const StepParams &sp, long long ga,
                             long long gb, const uint8_t *nsimp, const uint32_t *idx, const uint8_t *alive,
                             const float *vals, const float *wslot, const float *win, float *acc, float *wacc, int nsm,
                             unsigned *launches, cudaStream_t st)
{
	if (gb <= ga || a.nbins == 0) return cudaSuccess;
	*launches += 4;
	cudaError_t e = cudaMemsetAsync(a.heads, 0, sizeof(unsigned) * (kBinHeads + (size_t)a.nbins), st);   // heads, cnt
	if (e != cudaSuccess) return e;
	const int lb = grid_for((gb - ga) * sp.np, kListSlots, 16384);
	bin_list_kernel<false><<<lb, kListThreads, 0, st>>>(tiles, ntiles, sp, ga, gb, nsimp, idx, alive, a.cnt, nullptr);
	bin_alloc_kernel<<<grid_for(a.nbins, 256, 4096), 256, 0, st>>>(a.nbins, a.cnt, a.cursor, a.bins, a.heads);
	bin_list_kernel<true><<<lb, kListThreads, 0, st>>>(tiles, ntiles, sp, ga, gb, nsimp, idx, alive, a.cursor, a.list);
	e = cudaGetLastError();
	if (e != cudaSuccess) return e;
	if (sp.C == 1) return gather_c<1>(sp, a, tiles, ntiles, sp, ga, idx, vals, wslot, win, acc, wacc, nsm, st);
	if (sp.C == 3) return gather_c<3>(sp, a, tiles, ntiles, sp, ga, idx, vals, wslot, win, acc, wacc, nsm, st);
	return gather_c<4>(sp, a, tiles, ntiles, sp, ga, idx, vals, wslot, win, acc, wacc, nsm, st);
}

cudaError_t launch_color(const Image &in, const Image &out, int forward, cudaStream_t st)
{
	color_kernel<<<grid_for((long long)in.W * in.H * in.F, 256, 16384), 256, 0, st>>>(in, out, forward);
	return cudaGetLastError();
}

cudaError_t launch_finalize(const Tile *tiles, int nW, int wTmp, int hTmp, const StepParams &sp,
                            const Image &noisy, const float *acc, const float *wacc, const Image &out,
                            int inverse_color, cudaStream_t st)
{
	finalize_kernel<<<grid_for((long long)out.W * out.H * out.F, 256, 16384), 256, 0, st>>>(
		tiles, nW, wTmp, hTmp, sp, noisy, acc, wacc, out, inverse_color);
	return cudaGetLastError();
}

}  // namespace bm4dof
