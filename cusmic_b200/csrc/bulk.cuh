// Dense detection pass: one streaming kernel for every frame of a batch,
// whatever its width, alignment or noise model.
//
// What the pass needs from every pixel is only whether its sig_raw =
// lap / (2 noise) can exceed min(cr_threshold, neighbor_threshold); the exact
// value matters for the ~1% of pixels where it can.  So the work is split:
//
//  * block floors (once per call): a lower bound of the noise over every
//    32 x 32 block, turned into a threshold T = 2 min(cr, nb) (1 - 1e-12) x
//    floor.  With an error map floor_kernel takes min(max(error, 0)) over the
//    block (NaN counts as 0), once for each distinct map.  With the noise
//    model (src/filters.cuh:107-123) it stores a lower bound of the block's
//    clean values as an ordered key (from the row minima prepare_kernel keeps
//    of the non-hole pixels; the hole fill lowers it with the values it
//    writes) and the block's largest gain and smallest read noise when they
//    are maps.  Between passes
//    only replacement changes clean,
//    and replace_kernel lowers the key of the block it writes into, so the key
//    stays a lower bound of the block's values.  Every 5 x 5 median window of
//    a block lies in the block's 3 x 3 neighbourhood of blocks (border-mapped
//    positions included; wrap adds the blocks at the opposite edges, constant
//    adds zero), so the smallest key there bounds every window's median from
//    below, and the model evaluated at it with the block's gain and read noise
//    bounds the noise from below: the model is non-decreasing in the median
//    and in the read noise and non-increasing in the gain;
//  * sig_bulk_kernel (the full first pass): the Laplacian of every pixel against T of
//    its block.  Every pixel whose sig_raw exceeds min(cr, nb) passes (the
//    product is rounded by at most 2^-53 relative, the margin is 1e-12 and
//    the upper bound of the Laplacian used here is never below the
//    reference's value).  Passing pixels are written with that bound to a
//    per-warp region of the `pre` list (no atomics);
//  * classify_kernel: sig_raw of each listed pixel, lap / (2 noise), with the
//    exact noise (error map, or the noise model from the pixel's own 5 x 5
//    median); above cr_threshold -> high candidate list, else above
//    neighbor_threshold -> low list (src/filters.cuh:125-135), and the same
//    classes into the HIGH / LOW planes that late passes update.  The
//    candidate kernels recompute every value they threshold exactly.
//
// sig_bulk_kernel is warp-specialised.  A producer warp copies clean row
// segments (BK_COLS columns plus halo columns) into a ring of BK_SLOTS rows in
// shared memory: one `cp.async.bulk` for the 16-byte aligned body of a row
// and up to four single elements with 8-byte `cp.async` (an unaligned first
// or last element, the border columns -1 and w), so rows of any width and
// alignment stream the same way.  A row whose aligned body starts on an odd
// cell is stored one cell to the right (its shift).  Each ring row has a
// "full" mbarrier (the body's transaction bytes plus the producer's cp.async
// arrive) and an "empty" mbarrier on which each of the four consumer warps
// arrives when it is done with the row.  The producer computes the copies of
// an item's rows once per item (they differ by row offsets only), so its
// per-row work is a wait on the row's empty barrier and the issue.  (The S1, S2 and
// CAND planes were zeroed by the call's first launch.)  A block takes items
// of BK_COLS x BK_ROWS pixels from a ticket counter (items of frames that
// stopped are skipped there) and the ring runs straight through from one item
// into the next.
//
// The Laplacian (src/filters.cuh:86-105): each consumer thread evaluates four
// consecutive columns x .. x + 3 (lane ct of the four warps: x = x0 + 4 ct)
// and keeps the quarter values of the rows above and at the current row, and
// the current row's left and right neighbours, in registers.  Differences the reference computes twice
// are computed once: down(y) = q(y) - q(y+1) and up(y+1) = q(y+1) - q(y) are
// exact negatives of each other in round-to-nearest, and so are right(x) and
// left(x+1); negation changes at most the sign of a zero difference.
// positive(v) is replaced by an upper bound: v with its high word cleared when
// the sign bit is set (0 or a subnormal instead of the reference's 0 for a
// negative v).  Floating-point addition is monotone, so the sum is never below
// the reference's Laplacian for finite inputs; where a term is NaN the
// reference's sig_raw is NaN and its pixel is never a candidate, and a value
// here only lists a pixel that the candidate kernel drops.
//
// Non-finite input pixels (holes, sig = 0 in the reference) are not tested
// here; the candidate kernel drops candidates that are holes.
//
// Borders (Laplacian border mode: nearest for mirror and reflect): rows
// outside the frame are copied from their border-mapped row, or from a zero
// row in constant mode; columns -1 and w are copied from their border-mapped
// columns (zeros in constant mode), so the evaluation has no border cases.
//
// Every wait is bounded (about one second of SM clock).  A wait that runs out
// sets Control::fault (pass_control then stops every active frame
// and marks it faulted; the host reports CUSMIC_CUDA_ERROR) and the ring's
// abort word, which ends the block's other waits early; before the block
// exits, its producer waits (again bounded) for the copies it still has in
// flight into shared memory.
#pragma once
#include "detect.cuh"

namespace cb {

constexpr int BK_CWARPS = 4;                     // consumer warps
constexpr int BK_THREADS = 32 * (BK_CWARPS + 1); // plus one producer warp
constexpr int BK_HALF = 64 * BK_CWARPS;          // columns of one pair set (256)
constexpr int BK_COLS = 2 * BK_HALF;             // columns per item (512)
constexpr int BK_ROWS = 32;                      // most rows per item
constexpr int BK_SLOTS = 8;                      // ring rows (power of two)
constexpr int BK_CELLS = BK_COLS + 4;            // cells of a row: columns x0 - 2 .. x0 + BK_COLS + 1
constexpr int BK_STRIDE = BK_CELLS + 2;          // ring row length: room for a shift of one cell
constexpr int BK_BLOCKS_PER_SM = 6;
constexpr int BK_REGION = 4 * 32 * BK_ROWS;      // pre-list entries one consumer warp can write per item
constexpr int FLOOR_BLOCK = 32;                  // noise-floor granularity (square)
constexpr long long BK_WAIT_CYCLES = 1LL << 31;
static_assert((BK_SLOTS & (BK_SLOTS - 1)) == 0, "ring depth must be a power of two");
static_assert(BK_ROWS == FLOOR_BLOCK, "an item spans one row of floor blocks");
static_assert(BK_HALF % FLOOR_BLOCK == 0, "pair sets start on a floor block");
static_assert((BK_STRIDE * 8) % 16 == 0, "ring rows must stay 16-byte aligned");

struct __align__(128) BulkRing {
	double c[BK_SLOTS][BK_STRIDE]; // clean; column x0 - 2 + c at cell c + shift
	int2 meta[BK_SLOTS];           // first ring row of an item: {item index, y1}; index < 0: end
	int shift[BK_SLOTS];           // 0 or 1
	unsigned long long full[BK_SLOTS], empty[BK_SLOTS];
	unsigned long long poison; // never completes (injected failures only)
	int abort;
};

// A pixel that passed the floor test, with its Laplacian bound.
struct PreCand {
	unsigned pixel, frame;
	double lap;
};

// One 32 x 32 block whose floor floor_kernel computes: kind 0 = an error map
// (frames that share a map share its thresholds), 1 = a noise-model frame.
struct FloorJob {
	int frame, x0, y0, kind;
	long long out; // index into the threshold array
};

// Zeros for constant-mode rows and columns outside the frame.
__device__ __align__(16) double bulk_zero_row[BK_CELLS];

__device__ __forceinline__ unsigned smem_u32(const void *p)
{
	return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long *b, unsigned bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(b)),
		"r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *b)
{
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(b)) : "memory");
}

// As mbar_arrive, by the lanes with `mine` set, without a branch.
__device__ __forceinline__ void mbar_arrive_if(unsigned long long *b, bool mine)
{
	asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %1, 0;\n"
		     " @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}\n" ::"r"(smem_u32(b)), "r"((int)mine)
		: "memory");
}

// Arrive on b once every cp.async this thread issued so far has landed.
__device__ __forceinline__ void mbar_arrive_cp_async(unsigned long long *b)
{
	asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(b)) : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned long long *b, unsigned parity)
{
	unsigned done;
	asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
		     " selp.u32 %0, 1, 0, p;\n}\n"
		: "=r"(done)
		: "r"(smem_u32(b)), "r"(parity)
		: "memory");
	return done != 0;
}

// Wait until the phase of parity `parity` of barrier b has completed; false
// after about `limit` SM cycles, or as soon as the block aborted.
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity, const int *abort,
	long long limit = BK_WAIT_CYCLES)
{
	if (mbar_test(b, parity))
		return true;
	const long long t0 = clock64();
	for (unsigned i = 1;; ++i) {
		if (mbar_test(b, parity))
			return true;
		if ((i & 15) == 0 && (*(const volatile int *)abort || clock64() - t0 > limit))
			return false;
	}
}

// mbar_wait for a whole warp (every lane calls it and gets the same answer): one
// vote when the phase has completed already, no divergent branch.
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long *b, unsigned parity, const int *abort)
{
	if (__all_sync(0xffffffffu, mbar_test(b, parity)))
		return true;
	const long long t0 = clock64();
	for (unsigned i = 1;; ++i) {
		if (__all_sync(0xffffffffu, mbar_test(b, parity)))
			return true;
		if ((i & 15) == 0 && __any_sync(0xffffffffu, *(const volatile int *)abort ||
			clock64() - t0 > BK_WAIT_CYCLES))
			return false;
	}
}

// An injected failure (Control::poison_wait): a wait, bounded by `limit`
// cycles, on barrier b, which was initialised for one arrival that never
// comes.  It runs out and returns false, like a wait whose copies never land.
__device__ __forceinline__ bool poisoned_wait(unsigned long long *b, const int *abort, long long limit)
{
	return mbar_wait(b, 0, abort, limit);
}

// Global -> shared bulk copy completing on barrier bar (16-byte aligned
// addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes,
	unsigned long long *bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
		::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
		: "memory");
}

// The copies of ring row r of an item starting at column x0 of a w x h frame
// whose clean buffer starts `mis` elements past a 16-byte boundary (0 or 1).
// Cells are relative to the row's shift.
struct BulkRow {
	int shift;         // 0 or 1
	long long src;     // body: element offset into clean (-1: the zero row)
	int cell, n;       // body: destination cell and element count (even, maybe 0)
	// Single-element copies: an unaligned first element (head), an odd last
	// element (tail), columns -1 (left) and w (right).  Source: element
	// offset into clean, -1 for a zero, NO_COPY when there is none.
	long long hsrc, tsrc, lsrc, rsrc;
	int hcell, tcell, lcell, rcell;
	unsigned bytes; // transaction bytes of the body
};
constexpr long long NO_COPY = -2;

CB_HD BulkRow bulk_row(int w, int h, int lm, int mis, int x0, int r)
{
	BulkRow b;
	b.hsrc = b.tsrc = b.lsrc = b.rsrc = NO_COPY;
	b.hcell = b.tcell = b.lcell = b.rcell = 0;
	const int my = border_index(r, h, lm);
	if (my < 0) { // constant mode, row outside the frame
		b.shift = 0;
		b.src = -1;
		b.cell = 0;
		b.n = BK_CELLS;
		b.bytes = 8u * BK_CELLS;
		return b;
	}
	const long long ro = (long long)my * w;
	const int a = x0 - 2 < 0 ? 0 : x0 - 2;
	const int e = x0 + BK_COLS + 2 < w ? x0 + BK_COLS + 2 : w;
	const int head = (int)((mis + ro + a) & 1); // element a is 8 bytes off a 16-byte boundary
	const int a1 = a + head;
	b.shift = a1 & 1; // cell of a1 (x0 is even) made even
	const int len = e - a1 > 0 ? e - a1 : 0;
	b.src = ro + a1;
	b.cell = a1 - x0 + 2 + b.shift;
	b.n = len & ~1;
	b.bytes = 8u * (unsigned)b.n;
	if (head) {
		b.hsrc = ro + a;
		b.hcell = a - x0 + 2 + b.shift;
	}
	if (len & 1) {
		b.tsrc = ro + e - 1;
		b.tcell = e - 1 - x0 + 2 + b.shift;
	}
	if (x0 == 0) { // column -1
		const int mx = border_index(-1, w, lm);
		b.lsrc = mx < 0 ? -1 : ro + mx;
		b.lcell = 1 + b.shift;
	}
	if (w <= x0 + BK_COLS) { // column w
		const int mx = border_index(w, w, lm);
		b.rsrc = mx < 0 ? -1 : ro + mx;
		b.rcell = w - x0 + 2 + b.shift;
	}
	return b;
}

// Floors of 32 x 32 blocks (see the head of this file): of each distinct
// error map (one lane per column, all 32 rows in flight), and of each
// noise-model frame (from prepare_kernel's row minima, one lane per row).
// One warp per block.
//
// Noise-model blocks of frames without gain or read-noise maps are left to
// model_floor_kernel.
__device__ __forceinline__ bool thread_floor_job(const FloorJob &jb, const FrameDesc &fd)
{
	return jb.kind && !fd.gain_map && !fd.rn_map;
}

__device__ __forceinline__ void floor_jobs(const FrameDesc *__restrict__ frames,
	const FloorJob *__restrict__ jobs, int njobs, const DetectParams &prm, BlockFloor *floors)
{
	const int lane = threadIdx.x & 31;
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	const double tmin2 = fmin(prm.thi2, prm.tlo2);
	for (int j = gw; j < njobs; j += nw) {
		const FloorJob jb = jobs[j];
		const FrameDesc &fd = frames[jb.frame];
		if (thread_floor_job(jb, fd))
			continue; // warp-uniform
		const int w = fd.w, x = jb.x0 + lane;
		const int n = (jb.y0 + FLOOR_BLOCK < fd.h ? jb.y0 + FLOOR_BLOCK : fd.h) - jb.y0;
		if (jb.kind) { // noise model: ordered keys of clean, -gain, read noise
			const long long at = (long long)jb.y0 * w + x;
			unsigned long long key = ~0ull, gkey = ~0ull, rkey = ~0ull;
			// Clean: the smallest of the block rows' high words (prepare_kernel;
			// lane = row), as a key with its low word cleared: no larger than
			// the smallest key of the block's non-hole values.
			{
				const uint32_t m = lane < n ? plane_ptr(fd, P_ROWMIN)[(long long)(jb.y0 + lane) * fd.words +
					jb.x0 / 32] : 0xffffffffu;
				const uint32_t hi = __reduce_min_sync(0xffffffffu, m);
				if (hi != 0xffffffffu)
					key = (unsigned long long)hi << 32;
			}
			if (x < w && (fd.gain_map || fd.rn_map))
				for (int k = 0; k < n; ++k) {
					if (fd.gain_map)
						gkey = min(gkey, order_key(-fd.gain_map[at + (long long)k * w]));
					if (fd.rn_map)
						rkey = min(rkey, order_key(fd.rn_map[at + (long long)k * w]));
				}
#pragma unroll
			for (int o = 16; o; o >>= 1) {
				key = min(key, __shfl_xor_sync(0xffffffffu, key, o));
				gkey = min(gkey, __shfl_xor_sync(0xffffffffu, gkey, o));
				rkey = min(rkey, __shfl_xor_sync(0xffffffffu, rkey, o));
			}
			if (lane == 0)
				floors[jb.out] = BlockFloor{0.0, key, gkey, rkey};
			continue;
		}
		const double *col = fd.error + (long long)jb.y0 * w + x;
		double v[FLOOR_BLOCK];
#pragma unroll
		for (int k = 0; k < FLOOR_BLOCK; ++k)
			v[k] = x < w && k < n ? col[(long long)k * w] : INFINITY;
		double m = INFINITY;
#pragma unroll
		for (int k = 0; k < FLOOR_BLOCK; ++k)
			m = dmin(m, v[k] > 0 ? v[k] : 0.0);
#pragma unroll
		for (int o = 16; o; o >>= 1)
			m = dmin(m, __shfl_xor_sync(0xffffffffu, m, o));
		const double T = tmin2 * m;
		if (lane == 0)
			floors[jb.out].thr = T >= 0 ? T : 0.0; // NaN lists everything
	}
}

__global__ void __launch_bounds__(256)
floor_kernel(const FrameDesc *__restrict__ frames, const FloorJob *__restrict__ jobs, int njobs,
	DetectParams prm, BlockFloor *floors)
{
	floor_jobs(frames, jobs, njobs, prm, floors);
}

// Floors of the noise-model blocks of frames without gain or read-noise maps,
// one thread per block: the smallest of the block rows' high words
// (prepare_kernel's row minima) as a key with its low word cleared.
__global__ void __launch_bounds__(256)
model_floor_kernel(const FrameDesc *__restrict__ frames, const FloorJob *__restrict__ jobs, int njobs,
	BlockFloor *floors)
{
	for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < njobs; j += gridDim.x * blockDim.x) {
		const FloorJob jb = jobs[j];
		const FrameDesc &fd = frames[jb.frame];
		if (!thread_floor_job(jb, fd))
			continue;
		const int n = min(FLOOR_BLOCK, fd.h - jb.y0);
		const uint32_t *m = plane_ptr(fd, P_ROWMIN) + (long long)jb.y0 * fd.words + jb.x0 / 32;
		uint32_t v[FLOOR_BLOCK], hi = 0xffffffffu;
#pragma unroll
		for (int k = 0; k < FLOOR_BLOCK; ++k) // every load in flight at once
			v[k] = k < n ? m[(long long)k * fd.words] : 0xffffffffu;
#pragma unroll
		for (int k = 0; k < FLOOR_BLOCK; ++k)
			hi = min(hi, v[k]);
		floors[jb.out] = BlockFloor{0.0, hi != 0xffffffffu ? (unsigned long long)hi << 32 : ~0ull,
			~0ull, ~0ull};
	}
}

__device__ __forceinline__ int nbr_block(int b, int n, int i, bool wrap)
{
	// i = 0..2: b - 1 .. b + 1; i = 3..6 (wrap mode near an edge only): the two
	// blocks at each edge.  -1: none.
	if (i < 3)
		return b - 1 + i >= 0 && b - 1 + i < n ? b - 1 + i : -1;
	if (!wrap || (b > 1 && b < n - 2))
		return -1;
	const int v = i == 3 ? 0 : i == 4 ? 1 : i == 5 ? n - 2 : n - 1;
	return v >= 0 && v < n ? v : -1;
}

__device__ __forceinline__ double model_threshold(const FrameDesc &fd, int bx, int by, int mode,
	double tmin2)
{
	const BlockFloor *bf = fd.floors;
	const int w = fd.w, h = fd.h;
	const int bw = (w + FLOOR_BLOCK - 1) / FLOOR_BLOCK, bh = (h + FLOOR_BLOCK - 1) / FLOOR_BLOCK;
	const bool wrap = mode == WRAP;
	unsigned long long key = ~0ull;
	for (int i = 0; i < 7; ++i) {
		const int yy = nbr_block(by, bh, i, wrap);
		if (yy < 0)
			continue;
		for (int j = 0; j < 7; ++j) {
			const int xx = nbr_block(bx, bw, j, wrap);
			if (xx >= 0)
				key = min(key, bf[yy * bw + xx].key);
		}
	}
	// In constant mode a window reaching past the frame holds zeros.
	if (mode == CONSTANT && (bx == 0 || by == 0 || (bx + 1) * FLOOR_BLOCK + 2 > w ||
		(by + 1) * FLOOR_BLOCK + 2 > h))
		key = min(key, order_key(0.0));
	double m = order_value(key);
	m = m < SIGNAL_FLOOR ? SIGNAL_FLOOR : m;
	const BlockFloor &own = bf[by * bw + bx];
	const double g = fd.gain_map ? -order_value(own.gkey) : fd.gain;
	const double rn = fd.rn_map ? order_value(own.rkey) : fd.rn;
	return tmin2 * (sqrt(rn * rn + g * m) / g);
}

static_assert(FLOOR_BLOCK == 32, "a bit word of a row lies in one floor block");

// model_threshold of block (bx, by) of a noise-model frame; outside wrap mode
// only the 3 x 3 neighbouring blocks count, read directly (sig_bulk_kernel of 64
// noise-model frames of 256 to 4096 pixels a side: 386 us with model_threshold's
// loops over a wrapped range, 370 us).
__device__ __forceinline__ double block_threshold(const FrameDesc &fd, int bx, int by, int mode,
	double tmin2)
{
	if (mode == WRAP)
		return model_threshold(fd, bx, by, mode, tmin2);
	const BlockFloor *bf = fd.floors;
	const int bw = (fd.w + FLOOR_BLOCK - 1) / FLOOR_BLOCK, bh = (fd.h + FLOOR_BLOCK - 1) / FLOOR_BLOCK;
	unsigned long long key = ~0ull;
#pragma unroll
	for (int i = -1; i <= 1; ++i)
#pragma unroll
		for (int j = -1; j <= 1; ++j) {
			const int yy = by + i, xx = bx + j;
			if (yy >= 0 && yy < bh && xx >= 0 && xx < bw)
				key = min(key, bf[yy * bw + xx].key);
		}
	if (mode == CONSTANT && (bx == 0 || by == 0 || (bx + 1) * FLOOR_BLOCK + 2 > fd.w ||
		(by + 1) * FLOOR_BLOCK + 2 > fd.h))
		key = min(key, order_key(0.0));
	double m = order_value(key);
	m = m < SIGNAL_FLOOR ? SIGNAL_FLOOR : m;
	const BlockFloor &own = bf[by * bw + bx];
	const double g = fd.gain_map ? -order_value(own.gkey) : fd.gain;
	const double rn = fd.rn_map ? order_value(own.rkey) : fd.rn;
	return tmin2 * (sqrt(rn * rn + g * m) / g);
}

// Upper bound of positive(v): v when its sign bit is clear; otherwise the
// high word cleared (0 or a subnormal).
__device__ __forceinline__ double pos_ub(double v)
{
	const int hi = __double2hiint(v);
	return __hiloint2double(hi & ~(hi >> 31), __double2loint(v));
}

__device__ __forceinline__ unsigned hi_word(double v)
{
	return (unsigned)__double2hiint(v);
}

// The copies of an in-frame row `by` elements (a whole number of row pairs)
// away from the row b describes: only the element offsets into clean change
// (-1, a zero, stays).
__device__ __forceinline__ BulkRow shift_row(BulkRow b, long long by)
{
	b.src += by;
	if (b.hsrc >= 0)
		b.hsrc += by;
	if (b.tsrc >= 0)
		b.tsrc += by;
	if (b.lsrc >= 0)
		b.lsrc += by;
	if (b.rsrc >= 0)
		b.rsrc += by;
	return b;
}

// Issue the copies of one ring row (one lane: the bulk copy completes on
// the row's full barrier by its transaction bytes, the single-element copies
// by the thread's cp.async arrival).
__device__ __forceinline__ void bulk_issue(BulkRing &R, int slot, const BulkRow &b, const double *clean)
{
	double *row = R.c[slot];
	R.shift[slot] = b.shift;
	mbar_expect_tx(&R.full[slot], b.bytes);
	if (b.n)
		bulk_copy(row + b.cell, b.src < 0 ? bulk_zero_row : clean + b.src, 8u * b.n, &R.full[slot]);
	if (b.hsrc != NO_COPY)
		cp_async8(row + b.hcell, clean + b.hsrc);
	if (b.tsrc != NO_COPY)
		cp_async8(row + b.tcell, clean + b.tsrc);
	if (b.lsrc != NO_COPY)
		cp_async8(row + b.lcell, b.lsrc < 0 ? bulk_zero_row : clean + b.lsrc);
	if (b.rsrc != NO_COPY)
		cp_async8(row + b.rcell, b.rsrc < 0 ? bulk_zero_row : clean + b.rsrc);
	mbar_arrive_cp_async(&R.full[slot]);
}

// Rows the producer warp issues at a time, one per lane.  A row's copies take a
// lane a chain of instructions, which the consumers' share of the issue slots
// stretches: one row at a time, sig_bulk_kernel took 354 us on 64 ragged frames of
// 256 to 4096 pixels a side and 47 on 256 of 40 to 200, with four 331 and 38
// (two: 341 and 39; eight leave too few slots for the next group, 358 and 38, and
// prep_detect_kernel 300 us for 268).  A lane's slot held the row BK_SLOTS
// back, which an earlier group issued.
constexpr int BK_ISSUE = 4;
static_assert(BK_ISSUE <= BK_SLOTS && BK_ISSUE <= 32, "a lane per row, rows of earlier groups ahead");

// Take the next items' indices from ctl->ticket (whole warp).
__device__ __forceinline__ int next_ticket(Control *ctl)
{
	int t = 0;
	if ((threadIdx.x & 31) == 0)
		t = atomicAdd(&ctl->ticket, 1);
	return __shfl_sync(0xffffffffu, t, 0);
}

// End of the items: an end marker in ring row g (whole warp).
__device__ __forceinline__ bool bulk_end(BulkRing &R, int &g)
{
	const int slot = g & (BK_SLOTS - 1);
	if (g >= BK_SLOTS && !mbar_wait_warp(&R.empty[slot], ((g / BK_SLOTS) - 1) & 1, &R.abort))
		return false;
	if ((threadIdx.x & 31) == 0) {
		R.meta[slot] = make_int2(-1, 0);
		mbar_arrive(&R.full[slot]);
		mbar_arrive(&R.full[slot]);
	}
	++g;
	return true;
}

// The producer warp's rows of one item: rows y0 - 1 .. y1 from ring row g on,
// issue(lane's slot, lane's row, its copies) once the slot is free.  The copies
// of an item's in-frame rows differ only by their row offsets, in two classes
// by row parity (the 16-byte phase of a row start alternates when w is odd),
// so they are computed once per item (kept in `base`, shared memory); rows
// outside the frame (border-mapped or zero) are computed on their own.
template <class Issue>
__device__ __forceinline__ bool bulk_rows(BulkRing &R, int &g, BulkRow (&base)[2], int t, int w, int h, int lm,
	int mis, int x0, int y0, int y1, Issue issue)
{
	const int lane = threadIdx.x & 31;
	const int ra = y0 - 1 < 0 ? 0 : y0 - 1; // first in-frame row of the item
	if (lane < 2)
		base[lane] = bulk_row(w, h, lm, mis, x0, lane && ra + 1 < h ? ra + 1 : ra);
	__syncwarp();
	for (int r0 = y0 - 1; r0 <= y1; r0 += BK_ISSUE) {
		const int r = r0 + lane, d = r - ra;
		const bool mine = lane < BK_ISSUE && r <= y1;
		const int q = g + lane, slot = q & (BK_SLOTS - 1);
		BulkRow b;
		bool ok = true;
		if (mine) {
			b = r < 0 || r >= h ? bulk_row(w, h, lm, mis, x0, r)
				: shift_row(base[d & 1], (long long)(d & ~1) * w);
			ok = q < BK_SLOTS || mbar_wait(&R.empty[slot], ((q / BK_SLOTS) - 1) & 1, &R.abort);
		}
		if (!__all_sync(0xffffffffu, ok))
			return false;
		if (mine) {
			if (r == y0 - 1)
				R.meta[slot] = make_int2(t, y1);
			issue(slot, r, b);
		}
		g += min(BK_ISSUE, y1 - r0 + 1);
	}
	__syncwarp(); // before the next item's base
	return true;
}

// Producer of sig_bulk_kernel (the whole producer warp); g counts the ring rows
// issued.  Returns false after a fault.
__device__ __forceinline__ bool bulk_producer(BulkRing &R, const FrameDesc *__restrict__ frames,
	const FrameState *__restrict__ state, const int4 *__restrict__ items, int nitems, int lm,
	Control *ctl, int &g, BulkRow (&base)[2])
{
	int next = next_ticket(ctl);
	for (;;) {
		// Next active item.
		int t = -1;
		while (next < nitems) {
			const int cand = next;
			next = next_ticket(ctl);
			const int4 it = items[cand];
			if (!state[it.x].active)
				continue;
			if ((uintptr_t)frames[it.x].clean & 7) // the host rejects such buffers
				return false;
			t = cand;
			break;
		}
		if (t < 0)
			return bulk_end(R, g);
		const int4 it = items[t]; // items never cross a 32-row floor block
		const FrameDesc &fd = frames[it.x];
		const double *clean = fd.clean;
		const int mis = (int)(((uintptr_t)clean >> 3) & 1);
		if (!bulk_rows(R, g, base, t, fd.w, fd.h, lm, mis, it.y, it.z, it.w,
			[&](int slot, int, const BulkRow &b) { bulk_issue(R, slot, b, clean); }))
			return false;
	}
}

// Columns x - 1 .. x + 4 of a ring row (x = the lane's first column, at cell
// c + shift; c even, so every 16-byte load is aligned).
__device__ __forceinline__ void load_six(const double *row, int c, int shift, double (&v)[6])
{
	if (shift == 0) {
		const double2 a = *reinterpret_cast<const double2 *>(row + c);
		const double2 b = *reinterpret_cast<const double2 *>(row + c + 2);
		v[0] = row[c - 1];
		v[1] = a.x;
		v[2] = a.y;
		v[3] = b.x;
		v[4] = b.y;
		v[5] = row[c + 4];
	} else {
		const double2 a = *reinterpret_cast<const double2 *>(row + c);
		const double2 b = *reinterpret_cast<const double2 *>(row + c + 2);
		const double2 d = *reinterpret_cast<const double2 *>(row + c + 4);
		v[0] = a.x;
		v[1] = a.y;
		v[2] = b.x;
		v[3] = b.y;
		v[4] = d.x;
		v[5] = d.y;
	}
}

// A consumer warp's part of an item whose columns in the frame (w wide) end
// before the warp's: it frees the ring rows [g, g + n) as they arrive.  (Working
// through its masked lanes cost sig_bulk_kernel 52 us instead of 47 on 256 frames
// of 40 to 200 pixels a side and 372 instead of 354 on 64 of 256 to 4096, whose
// last columns leave warps without work.)
__device__ __forceinline__ bool bulk_pass_by(BulkRing &R, int g, int n)
{
	for (int i = g; i < g + n; ++i) {
		const int slot = i & (BK_SLOTS - 1);
		if (!mbar_wait_warp(&R.full[slot], (i / BK_SLOTS) & 1, &R.abort))
			return false;
		if ((threadIdx.x & 31) == 0)
			mbar_arrive(&R.empty[slot]);
	}
	return true;
}

// Consumer warps of sig_bulk_kernel: lane ct of the four warps evaluates
// columns x0 + 4 ct .. x0 + 4 ct + 3.  Returns false after a fault.
__device__ __forceinline__ bool bulk_consumer(BulkRing &R, const FrameDesc *__restrict__ frames,
	const int4 *__restrict__ items, const DetectParams &prm, PreCand *pre, int *pre_counts)
{
	const double tmin2 = fmin(prm.thi2, prm.tlo2);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int ct = warp * 32 + lane; // 0 .. 127
	const int c0 = 2 + 4 * ct;       // cell of the lane's first column (before the row's shift)
	const unsigned below = (1u << lane) - 1u;
	int g = 0;
	bool ok = true;
	for (;;) {
		ok = mbar_wait_warp(&R.full[g & (BK_SLOTS - 1)], (g / BK_SLOTS) & 1, &R.abort);
		if (!ok)
			break;
		const int2 meta = R.meta[g & (BK_SLOTS - 1)];
		if (meta.x < 0)
			break;
		const int t = meta.x, y1 = meta.y;
		const int4 it = items[t];
		const int f = it.x, x0 = it.y, y0 = it.z;
		const FrameDesc &fd = frames[f];
		const int w = fd.w, x = x0 + 4 * ct;
		if (x0 + 128 * warp >= w) { // none of the warp's columns
			ok = bulk_pass_by(R, g, y1 - y0 + 2);
			if (!ok)
				break;
			if (lane == 0)
				pre_counts[t * BK_CWARPS + warp] = 0;
			g += y1 - y0 + 2;
			continue;
		}
		// High word of the block threshold per column (all ones: not a pixel).
		unsigned thr[4];
		{
			unsigned tv = 0xffffffffu;
			if (x < w) {
				const int bx = x / FLOOR_BLOCK, by = y0 / FLOOR_BLOCK;
				const double T = fd.error ? fd.floors[by * ((w + FLOOR_BLOCK - 1) / FLOOR_BLOCK) + bx].thr
					: block_threshold(fd, bx, by, prm.mode, tmin2);
				tv = hi_word(T >= 0 ? T : 0.0); // NaN lists everything
			}
#pragma unroll
			for (int i = 0; i < 4; ++i)
				thr[i] = x + i < w ? tv : 0xffffffffu;
		}
		ok = mbar_wait_warp(&R.full[(g + 1) & (BK_SLOTS - 1)], ((g + 1) / BK_SLOTS) & 1, &R.abort);
		if (!ok)
			break;
		// Row y0 - 1 (values) and row y0 (values and neighbours), as quarters.
		double q[4], up[4], ql, qr;
		{
			double u[6], c[6];
			load_six(R.c[g & (BK_SLOTS - 1)], c0, R.shift[g & (BK_SLOTS - 1)], u);
			load_six(R.c[(g + 1) & (BK_SLOTS - 1)], c0, R.shift[(g + 1) & (BK_SLOTS - 1)], c);
			ql = c[0] * 0.25;
			qr = c[5] * 0.25;
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				q[i] = c[i + 1] * 0.25;
				up[i] = q[i] - u[i + 1] * 0.25;
			}
		}
		__syncwarp();
		if (lane == 0) { // both rows are in registers now
			mbar_arrive(&R.empty[g & (BK_SLOTS - 1)]);
			mbar_arrive(&R.empty[(g + 1) & (BK_SLOTS - 1)]);
		}
		PreCand *region = pre + ((long long)t * BK_CWARPS + warp) * BK_REGION;
		int cnt = 0;
#pragma unroll 2
		for (int y = y0; y < y1; ++y) {
			const int gd = g + 2 + (y - y0); // ring row of y + 1
			const int sd = gd & (BK_SLOTS - 1);
			ok = mbar_wait_warp(&R.full[sd], (gd / BK_SLOTS) & 1, &R.abort);
			if (!ok)
				break;
			double n[6];
			load_six(R.c[sd], c0, R.shift[sd], n);
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&R.empty[sd]); // row y + 1 is in registers
			// Horizontal differences: left(x+i) = h[i], right(x+i) = -h[i+1].
			double h[5];
			h[0] = q[0] - ql;
#pragma unroll
			for (int i = 0; i < 3; ++i)
				h[i + 1] = q[i] - q[i + 1];
			h[4] = q[3] - qr;
			const long long pix0 = (long long)y * w + x;
			// The four columns' Laplacians first (independent chains), then
			// the list appends.
			double lap[4];
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				const double qd = n[i + 1] * 0.25;
				const double d = q[i] - qd;
				const double lft = i == 0 ? h[0] : -h[i], rgt = i == 3 ? h[4] : h[i + 1];
				lap[i] = (pos_ub(up[i] + lft) + pos_ub(up[i] + rgt)) +
					(pos_ub(d + lft) + pos_ub(d + rgt));
				up[i] = -d;
				q[i] = qd;
			}
			ql = n[0] * 0.25;
			qr = n[5] * 0.25;
			bool pass[4];
#pragma unroll
			for (int i = 0; i < 4; ++i)
				pass[i] = hi_word(lap[i]) >= thr[i];
			if (__any_sync(0xffffffffu, pass[0] | pass[1] | pass[2] | pass[3])) {
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					const unsigned bal = __ballot_sync(0xffffffffu, pass[i]);
					if (pass[i])
						region[cnt + __popc(bal & below)] =
							PreCand{(unsigned)(pix0 + i), (unsigned)f, lap[i]};
					cnt += __popc(bal);
				}
			}
		}
		if (!ok)
			break;
		if (lane == 0)
			pre_counts[t * BK_CWARPS + warp] = cnt;
		g += y1 - y0 + 2;
	}
	return ok;
}

__global__ void __launch_bounds__(BK_THREADS, BK_BLOCKS_PER_SM)
sig_bulk_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const int4 *__restrict__ items, int nitems, DetectParams prm, Control *ctl, PreCand *pre,
	int *pre_counts)
{
	__shared__ BulkRing R;
	__shared__ BulkRow base[2]; // the producer's row copies of the current item
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (tid == 0) {
		for (int i = 0; i < BK_SLOTS; ++i) {
			mbar_init(&R.full[i], 2); // the producer's transaction bytes and cp.async arrive
			mbar_init(&R.empty[i], BK_CWARPS);
		}
		mbar_init(&R.poison, 1);
		R.abort = 0;
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
	}
	__syncthreads();
	// An injected failure of either step (prepare or detection; prepare_kernel
	// has no wait of its own).
	const long long poison = ctl->poison_wait[0] > ctl->poison_wait[1] ? ctl->poison_wait[0]
		: ctl->poison_wait[1];
	bool ok;
	int issued = 0; // ring rows issued (producer warp)
	if (warp == BK_CWARPS)
		ok = bulk_producer(R, frames, state, items, nitems, lap_mode(prm.mode), ctl, issued, base);
	else if (warp == 0 && blockIdx.x == 0 && poison > 0)
		ok = __all_sync(0xffffffffu, poisoned_wait(&R.poison, &R.abort, poison));
	else
		ok = bulk_consumer(R, frames, items, prm, pre, pre_counts);
	if (!ok && lane == 0) {
		R.abort = 1;
		atomicOr(&ctl->fault, FAULT_COPY);
	}
	__syncthreads();
	// After a fault: wait (bounded) for the copies still in flight into this
	// block's shared memory (on the normal path the consumers waited for every
	// issued row).
	if (warp == BK_CWARPS && lane == 0 && R.abort)
		for (int q = issued - BK_SLOTS < 0 ? 0 : issued - BK_SLOTS; q < issued; ++q) {
			const long long t0 = clock64();
			while (!mbar_test(&R.full[q & (BK_SLOTS - 1)], (q / BK_SLOTS) & 1) &&
				clock64() - t0 < BK_WAIT_CYCLES) {
			}
		}
}

// Entries a warp of classify_kernel stages per list before it appends them.
constexpr int CL_CAP = 128;

struct ClassifyStage {
	uint2 buf[8][2][CL_CAP]; // per warp: high, low
	int n[8][2];             // left at the end
	unsigned long long at[2];
};

// sig_raw of the listed pixels, lap / (2 noise) (src/filters.cuh:125-135),
// with the error map or the exact noise model at the pixel: a warp per item,
// whose four regions it reads as one list, a lane per entry, the next 32
// entries loading meanwhile.  The high list grows from the front of the
// candidate buffer, the low list from its back; a NaN goes to the high list
// (the candidate kernel decides).  Error-map entries listed with a bound of
// +inf get their exact Laplacian first.  A warp appends 128 entries at a time,
// the block's warps together what is left.  (A warp per region, with 20 of 32
// lanes busy and two block barriers for each eight regions, took 66 us on 16
// frames of 2048 x 2048.)  MODEL: the batch has noise-model frames.
template <bool MODEL>
__global__ void __launch_bounds__(256, MODEL ? 3 : 6)
classify_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const int4 *__restrict__ items, int nitems, const PreCand *__restrict__ pre,
	const int *__restrict__ pre_counts, DetectParams prm, Control *ctl, uint2 *cands)
{
	static_assert(BK_CWARPS == 4, "an item's counts are one int4");
	__shared__ ClassifyStage S;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	// After a bounded wait of the dense kernel ran out, the counts of the
	// items it left are stale: list nothing (the loop control then stops
	// every frame and the call reports the fault).
	if (*(const volatile int *)&ctl->fault)
		return;
	const unsigned long long cap = ctl->cand_cap;
	const unsigned below = (1u << lane) - 1u;
	int nst[2] = {0, 0};
	auto put = [&](int li, bool take, uint2 e) { // called by the whole warp
		const unsigned b = __ballot_sync(0xffffffffu, take);
		const int k = __popc(b);
		if (nst[li] + k > CL_CAP) {
			__syncwarp();
			unsigned long long at = 0;
			if (lane == 0)
				at = atomicAdd(li ? &ctl->pass[0].n_low : &ctl->pass[0].n_cand, (unsigned long long)nst[li]);
			at = __shfl_sync(0xffffffffu, at, 0);
			for (int i = lane; i < nst[li]; i += 32)
				cands[li ? cap - 1 - (at + i) : at + i] = S.buf[warp][li][i];
			nst[li] = 0;
			__syncwarp();
		}
		if (take)
			S.buf[warp][li][nst[li] + __popc(b & below)] = e;
		nst[li] += k;
	};
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	for (int i = gw; i < nitems; i += nw) {
		const int f = items[i].x;
		if (!state[f].active)
			continue; // warp-uniform
		const FrameDesc &fd = frames[f];
		const int4 c = reinterpret_cast<const int4 *>(pre_counts)[i];
		const int c1 = c.x + c.y, c2 = c1 + c.z, n = c2 + c.w;
		const PreCand *e = pre + (long long)i * BK_CWARPS * BK_REGION;
		auto entry = [&](int j) { // of the item's four regions as one list
			const int part = (j >= c.x) + (j >= c1) + (j >= c2);
			const int start = part == 0 ? 0 : part == 1 ? c.x : part == 2 ? c1 : c2;
			return j < n ? e[(long long)part * BK_REGION + j - start] : PreCand{0u, 0u, 0.0};
		};
		PreCand next = entry(lane);
		for (int k0 = 0; k0 < n; k0 += 32) {
			const PreCand pc = next;
			if (k0 + 32 < n)
				next = entry(k0 + 32 + lane);
			int cls = 0;
			if (k0 + lane < n) {
				const unsigned pix = pc.pixel, px = pix % (unsigned)fd.w, py = pix / (unsigned)fd.w;
				double lap = pc.lap, nz;
				if (!MODEL || fd.error) {
					nz = fd.error[pix];
					// A bound of +inf marks a pixel whose Laplacian reads a hole
					// (prep_detect_kernel) or overflowed: the exact Laplacian of
					// the filled working pixels.
					if (lap == INFINITY)
						lap = lap_at(fd, (int)px, (int)py, lap_mode(prm.mode));
				} else if (px >= 2 && py >= 2 && (int)px + 2 < fd.w && (int)py + 2 < fd.h) {
					double win[25];
					const double *src = fd.clean + pix - 2 * (long long)fd.w - 2;
#pragma unroll
					for (int a = 0; a < 5; ++a)
#pragma unroll
						for (int b = 0; b < 5; ++b)
							win[a * 5 + b] = src[(long long)a * fd.w + b];
					nz = noise_from_median(fd, pix, median_network(win));
				} else {
					nz = noise_model_at(fd, (int)px, (int)py, prm.mode);
				}
				const double v = lap / (2 * nz);
				cls = v > prm.cr || v != v ? 1 : v > prm.nb ? 2 : 0;
				if (cls) // the class planes that late passes keep up to date
					atomicOr(plane_ptr(fd, cls == 1 ? P_HIGH : P_LOW) + (long long)py * fd.words + (px >> 5),
						1u << (px & 31));
			}
			put(0, cls == 1, make_uint2((unsigned)f, pc.pixel));
			put(1, cls == 2, make_uint2((unsigned)f, pc.pixel));
		}
	}
	if (lane < 2)
		S.n[warp][lane] = lane ? nst[1] : nst[0];
	__syncthreads();
	if (threadIdx.x < 2) {
		int sum = 0;
		for (int v = 0; v < 8; ++v)
			sum += S.n[v][threadIdx.x];
		S.at[threadIdx.x] = sum ? atomicAdd(threadIdx.x ? &ctl->pass[0].n_low : &ctl->pass[0].n_cand,
			(unsigned long long)sum) : 0ull;
	}
	__syncthreads();
#pragma unroll
	for (int li = 0; li < 2; ++li) {
		unsigned long long at = S.at[li];
		for (int v = 0; v < warp; ++v)
			at += S.n[v][li];
		for (int i = lane; i < nst[li]; i += 32)
			cands[li ? cap - 1 - (at + i) : at + i] = S.buf[warp][li][i];
	}
}

} // namespace cb
