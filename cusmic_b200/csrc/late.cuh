// Late detection passes (every pass after the first), all of them in one launch
// whose blocks meet at barriers.
//
// A pass of the reference (src/cleaner.cuh:102-142) recomputes the whole
// detection chain on the current clean pixels, and between two passes only
// the pixels that the replacement wrote change.  Every quantity of the chain
// at a pixel p reads clean pixels within a fixed Chebyshev distance of p,
// measured in the frame (mirror, reflect and nearest map a window position
// onto an in-frame pixel no farther from p; constant reads a zero) or on the
// torus (wrap):
//
//   sig_raw = lap / (2 noise)       distance 2 (lap 1, noise-model median 2)
//   sig = sig_raw - med5(sig_raw)   distance 4
//   fine = med3 -> med7             distance 4
//   S1, S2, CAND                    distance 4
//   grown pixel (two dilations)     distance 6 (S2, S1 and CAND within 2)
//
// So with D the targets whose value the last replacement changed (the chg
// list that replace_targets writes), pass k + 1 differs from pass k only near
// D.  A late pass keeps the bit planes of the previous one and works on lists
// that start from D, in stages separated by barriers:
//
//  1. Half a warp per pixel of D (a lane per row of its 13 x 13
//     neighbourhood): the pixels within 2 are listed for re-evaluation (once
//     each, claimed in the EVAL plane); the HIGH pixels within 4 go to the high
//     list and the LOW pixels within 6 to the low list (once each, claimed in
//     the LISTED plane, by their old classes).
//  2. A thread per re-evaluated pixel: its exact sig_raw, hence its class
//     (sig_raw > cr_threshold or NaN: HIGH, else > neighbor_threshold: LOW;
//     classify_kernel's first-pass classes are supersets, from the Laplacian
//     upper bound).  A pixel that enters a class joins that list (its old class
//     listed it in stage 1 already if it keeps it); one that leaves HIGH loses
//     its S1 and CAND bits (sig <= sig_raw <= cr_threshold), one that leaves
//     both classes its S2 bit.
//  3. The high list's pixels that are HIGH now: significance and seed test, as
//     in a full pass but setting or clearing each bit.
//  4. The low list and the growth (low_list, growth_rows).
//  5. The replacement of the targets whose window holds a new pixel, and the
//     loop control.
//
// What stays exact: S1 and CAND everywhere, S2 of every HIGH pixel and of
// every LOW pixel with a CAND pixel within 2 (the only S2 bits growth reads): a
// LOW pixel whose CAND neighbourhood changed is within 6 of D.  Outside HIGH
// sig <= cr_threshold, and a pixel outside both classes has sig <=
// neighbor_threshold, so its bits are zero.
//
// Why one launch and lists: after the first pass little changes (16 frames of
// 2048 x 2048: 64,998 targets in the first pass, then 799, 688 and 290 changed
// pixels), so the passes are chains of latencies.  As eight launches each,
// scanning row marks and bit planes, in a graph's while node, passes 2 to 4
// took 0.30 ms of that batch's 1.04 ms, and a call without a graph issued 24
// launches for them whatever was left to do.
#pragma once

#include "bulk.cuh"
#include "common.cuh"
#include "detect.cuh"
#include "kernels.cuh"

namespace cb {

// One block of 24 warps per SM: the fewest arrivals at a grid barrier, with 80
// registers a thread.  (The candidate evaluation and the replacement want more: 124
// bytes of spill stores and 224 of loads a thread; with 32 warps of 64 registers 192
// and 364.)  Whole calls with 1024, 768, 640 and 512 threads, in us: 256 cutouts of 40
// to 200 pixels a side 316, 305, 296, 297; one 2048 x 2048 frame 377, 370, 363, 365;
// five of 1018 x 1001 550, 540, 537, 535; 64 ragged frames of 256 to 4096 pixels a side
// 2710, 2713, 2723, 2763; a 2048 x 2048 frame at thresholds of 1 and 0.5 3013, 3197, not
// timed, 3819.
constexpr int LATE_THREADS = 768;
constexpr int LATE_WARPS = LATE_THREADS / 32;

__device__ __forceinline__ int wrap_index(int i, int n)
{
	i %= n;
	return i < 0 ? i + n : i;
}

// The bound of a grid barrier's wait, in SM cycles (about 17 s), and the arrivals
// it waits for beyond the grid's (an injected failure: one that never comes).
// Every block of the team is running, so a block waits only while others work,
// and the bound cuts off no stage that ends: the longest single item is a
// replacement whose nearest donor is thousands of pixels away (1000 pixels: 7 ms).
struct BarrierWait {
	long long limit;
	unsigned missing;
};
constexpr long long BARRIER_CYCLES = 1LL << 35;

// The late launch's team: the blocks that have started when it is closed.  A block
// joins with its number (the order of the starts) and takes the first stage's share
// of that number among gridDim.x; the first barrier closes the team once the whole
// grid has started, or JOIN_CYCLES (about 17 us) after the first block got there, and
// the team's blocks do the missing shares.  So only running blocks meet at the
// barriers, and the launch needs no more SMs than are free: beside another stream's
// kernel that stays, or on a context with part of the SMs, a cooperative launch
// (whose blocks all have to fit at once) waits or is refused.  A block that comes
// too late leaves at once.  (Closing the team before the first stage cost every call
// the 2 us between the first block's start and the last one's.)
constexpr long long JOIN_CYCLES = 1 << 15;
constexpr unsigned TEAM_CLOSED = 1u << 31; // in Control::arrived

// False: too late.
__device__ __forceinline__ bool join_team(Control *ctl, Team &team)
{
	if (threadIdx.x == 0)
		team = Team{atomicAdd(&ctl->arrived, 1u), 0u};
	__syncthreads();
	return !(team.block & TEAM_CLOSED);
}

// Barrier of the team: the k-th call returns once every block has arrived k times,
// with their earlier writes visible (B.calls starts zero); the first one sets the
// team's size.  A wait that runs out faults every frame and returns false, and so do
// the barrier's other blocks that see the fault (the last one to arrive, whose own
// wait is over at once, among them) and every later barrier.
struct BarrierState {
	unsigned calls;
	int open;
};

__device__ __forceinline__ bool grid_barrier(Control *ctl, BarrierState &B, FrameState *state, int nf,
	const BarrierWait &bw, Team &team)
{
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		atomicAdd(&ctl->barrier, 1u);
		const unsigned call = ++B.calls;
		unsigned n = team.blocks;
		const long long t0 = clock64();
		bool ok;
		for (;;) {
			unsigned fault, count, here, size; // one round trip
			asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];\n"
				: "=r"(fault), "=r"(count), "=r"(here), "=r"(size)
				: "l"(__cvta_generic_to_global(&ctl->fault))
				: "memory");
			const long long waited = clock64() - t0;
			if (!n)
				n = here & TEAM_CLOSED ? size : here == gridDim.x ? here : 0u;
			if (!n && team.block == 0 && waited > JOIN_CYCLES) {
				n = atomicOr(&ctl->arrived, TEAM_CLOSED);
				*(volatile unsigned *)&ctl->team = n;
			}
			ok = fault == 0;
			if (!ok || (n && (int)(count - call * n - bw.missing) >= 0))
				break;
			if (waited > bw.limit) {
				ok = false;
				break;
			}
		}
		team.blocks = n;
		if (!ok) {
			atomicOr(&ctl->fault, FAULT_BARRIER);
			for (int f = 0; f < nf; ++f)
				state[f].fault = FAULT_BARRIER;
		}
		__threadfence();
		B.open = ok;
	}
	__syncthreads();
	return B.open != 0;
}

// A block's entries for the three lists of stage 1: their numbers, then their
// first slots.
struct ListSlots {
	int n[3];
	unsigned long long at[3];
};

// Stage 1 (called by every thread of the grid, in blocks of WARPS warps).  A
// block's warps reserve their list slots together, one atomic per list: an
// atomic per warp and list on the same three counters (0.8 ns each, one after
// another) held this stage for 82 us on 64,998 changed targets.
template <int WARPS>
__device__ __forceinline__ void late_neighbours(const FrameDesc *__restrict__ frames, const uint2 *targets,
	const unsigned *chg, PassLists &L, int mode, uint2 *cands, uint2 *low, uint2 *eval, ListSlots &R, Team team)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const long long n = (long long)L.n_chg;
	const bool wrap = mode == WRAP;
	const int dy = (lane & 15) - 6, ay = dy < 0 ? -dy : dy;
	// Entries per block and sweep: fewer for a short list, which spreads it.
	const long long share = (n + team.blocks - 1) / team.blocks;
	const int chunk = share < 2 * WARPS ? (int)share : 2 * WARPS;
	for (long long base = (long long)team.block * chunk; base < n; base += (long long)team.blocks * chunk) {
		const int own_entry = 2 * warp + (lane >> 4);
		const long long i = base + own_entry;
		bool valid = own_entry < chunk && i < n && dy <= 6;
		uint2 t = make_uint2(0u, 0u);
		int x = 0, yy = 0, w = 1, words = 1;
		uint32_t *high = nullptr, *lowp = nullptr, *ep = nullptr, *lp = nullptr;
		bool torus = false; // the row's window crosses the frame's edge on the torus
		if (valid) {
			t = targets[chg[i]];
			const FrameDesc &fd = frames[t.x];
			w = fd.w;
			words = fd.words;
			x = (int)(t.y % (unsigned)w);
			yy = (int)(t.y / (unsigned)w) + dy;
			if (wrap)
				yy = wrap_index(yy, fd.h);
			valid = yy >= 0 && yy < fd.h;
			torus = wrap && (x < 6 || x + 6 >= w);
			const long long row = (long long)(valid ? yy : 0) * words;
			high = plane_ptr(fd, P_HIGH) + row;
			lowp = plane_ptr(fd, P_LOW) + row;
			ep = plane_ptr(fd, P_EVAL) + row;
			lp = plane_ptr(fd, P_LISTED) + row;
		}
		// Pieces of the lane's row: its window [x - 6, x + 6] at once (at most
		// two words), or on the torus across an edge column by column.
		const int pieces = wrap ? (__syncthreads_or(valid && torus) ? 13 : 1) : 1;
		for (int p = 0; p < pieces; ++p) { // block-uniform
			unsigned long long m2 = 0, m4 = 0, m6 = 0; // bits from column 32 k
			int k = 0;
			if (valid && torus) {
				const int dx = p - 6, ax = dx < 0 ? -dx : dx, c = wrap_index(x + dx, w);
				k = c >> 5;
				m6 = 1ull << (c & 31);
				m4 = ax <= 4 && ay <= 4 ? m6 : 0ull;
				m2 = ax <= 2 && ay <= 2 ? m6 : 0ull;
			} else if (valid && p == 0) {
				auto span = [&](int r) { // columns x - r .. x + r in the frame
					const int a = max(x - r, 0), b = min(x + r, w - 1);
					return ((1ull << (b - a + 1)) - 1ull) << (a - 32 * k);
				};
				k = max(x - 6, 0) >> 5;
				m6 = span(6);
				m4 = ay <= 4 ? span(4) : 0ull;
				m2 = ay <= 2 ? span(2) : 0ull;
			}
			unsigned long long ne = 0, nh = 0, nl = 0;
			if (m6) {
				const bool two = (m6 >> 32) != 0;
				const unsigned long long H = high[k] | (unsigned long long)(two ? high[k + 1] : 0u) << 32;
				const unsigned long long W = lowp[k] | (unsigned long long)(two ? lowp[k + 1] : 0u) << 32;
				const unsigned long long want = (H & m4) | (W & ~H & m6);
				auto claim = [&](uint32_t *word, uint32_t bits) { return bits ? atomicOr(word, bits) : 0u; };
				const uint32_t e0 = claim(ep + k, (uint32_t)m2), e1 = claim(ep + k + 1, (uint32_t)(m2 >> 32));
				const uint32_t l0 = claim(lp + k, (uint32_t)want), l1 = claim(lp + k + 1, (uint32_t)(want >> 32));
				ne = m2 & ~(e0 | (unsigned long long)e1 << 32);
				const unsigned long long got = want & ~(l0 | (unsigned long long)l1 << 32);
				nh = got & H;
				nl = got & ~H;
			}
			// Positions in the three lists: counts (at most 13 per lane) side
			// by side in one scan of the warp, then the block's.
			int sum = __popcll(ne) | __popcll(nh) << 10 | __popcll(nl) << 20;
			const int own = sum;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const int v = __shfl_up_sync(0xffffffffu, sum, o);
				if (lane >= o)
					sum += v;
			}
			const int total = __shfl_sync(0xffffffffu, sum, 31);
			if (threadIdx.x < 3)
				R.n[threadIdx.x] = 0;
			__syncthreads();
			int mine = 0; // lanes 0..2: the warp's first entry of the list in the block's
			if (lane < 3 && total)
				mine = atomicAdd(&R.n[lane], (total >> (10 * lane)) & 1023);
			__syncthreads();
			if (threadIdx.x < 3) {
				const int c = R.n[threadIdx.x];
				unsigned long long *counter = threadIdx.x == 0 ? &L.n_eval : threadIdx.x == 1 ? &L.n_cand : &L.n_low;
				R.at[threadIdx.x] = c ? atomicAdd(counter, (unsigned long long)c) : 0ull;
			}
			__syncthreads();
			const unsigned pix = (unsigned)((long long)yy * w + 32 * k);
			auto put = [&](uint2 *list, int which, unsigned long long bits) {
				unsigned long long slot = R.at[which] + __shfl_sync(0xffffffffu, mine, which) +
					(((sum - own) >> (10 * which)) & 1023);
				for (; bits; bits &= bits - 1)
					list[slot++] = make_uint2(t.x, pix + __ffsll((long long)bits) - 1);
			};
			put(eval, 0, ne);
			put(cands, 1, nh);
			put(low, 2, nl);
		}
	}
}

// Stage 1 when much of the frames changed: a warp per row of 32 words, which takes
// all of CRMASK in place of D.  (Every changed pixel is in the mask, and what is
// evaluated again for the others comes out as it was.)  No claims: each pixel is
// listed by its own word.  Claims of 13 rows for each of a million changed targets
// took a 2048 x 2048 frame 1.2 ms, more than the pass's evaluations; the rows'
// words take 30 us whatever changed, and then four million pixels are classified.
// Hence the rule: when the changed targets are over a 64th of the pixels and a
// quarter of the mask.
__device__ __forceinline__ bool late_by_rows(const Control *ctl, const PassLists &L, const RowItems &rows)
{
	const unsigned long long n = L.n_chg;
	return 64 * n > rows.px && 4 * n > ctl->n_targets;
}

// Columns 32 k - 6 .. 32 k + 37 of row y of a plane (bit 0: the first); zero
// outside the frame, or on the torus what the column or row there maps to.
__device__ __forceinline__ unsigned long long window6(const uint32_t *plane, int w, int h, int words, int y,
	int k, bool torus)
{
	if (torus)
		y = wrap_index(y, h);
	if (y < 0 || y >= h)
		return 0ull;
	const uint32_t *row = plane + (long long)y * words;
	const unsigned long long l = k > 0 ? row[k - 1] >> 26 : 0u, c = row[k], r = k + 1 < words ? row[k + 1] & 63u : 0u;
	unsigned long long m = l | c << 6 | r << 38;
	if (torus && (k == 0 || 32 * k + 37 >= w))
		for (int j = 0; j < 44; ++j) {
			const int x = 32 * k - 6 + j;
			if (x < 0 || x >= w) {
				const int t = wrap_index(x, w);
				m |= (unsigned long long)((row[t >> 5] >> (t & 31)) & 1u) << j;
			}
		}
	return m;
}

__device__ __forceinline__ void late_rows(const FrameDesc *__restrict__ frames, const FrameState *state,
	const RowItems &rows, PassLists &L, int mode, uint2 *cands, uint2 *low, uint2 *eval, Team team)
{
	const int lane = threadIdx.x & 31;
	const int gw = (team.block * blockDim.x + threadIdx.x) >> 5, nw = (team.blocks * blockDim.x) >> 5;
	auto wide2 = [](unsigned long long m) { return m | m << 1 | m >> 1 | m << 2 | m >> 2; };
	for (int i = gw; i < rows.n; i += nw) {
		const int2 item = rows.rows[i];
		if (!state[item.x].active)
			continue; // warp-uniform
		const FrameDesc &fd = frames[item.x];
		const int w = fd.w, words = fd.words, y = item.y;
		for (int k0 = 0; k0 < words; k0 += 32) {
			const int k = k0 + lane;
			uint32_t ne = 0, nh = 0, nl = 0;
			if (k < words) {
				unsigned long long m2 = 0, m4 = 0, m6 = 0;
#pragma unroll 1
				for (int dy = -6; dy <= 6; ++dy) {
					const unsigned long long m = window6(plane_ptr(fd, P_CRMASK), w, fd.h, words, y + dy, k,
						mode == WRAP);
					m6 |= m;
					m4 |= dy >= -4 && dy <= 4 ? m : 0ull;
					m2 |= dy >= -2 && dy <= 2 ? m : 0ull;
				}
				const uint32_t clip = w - 32 * k >= 32 ? 0xffffffffu : (1u << (w - 32 * k)) - 1u;
				const long long o = (long long)y * words + k;
				const uint32_t H = plane_ptr(fd, P_HIGH)[o], W = plane_ptr(fd, P_LOW)[o];
				ne = (uint32_t)(wide2(m2) >> 6) & clip;
				nh = (uint32_t)(wide2(wide2(m4)) >> 6) & H;
				nl = (uint32_t)(wide2(wide2(wide2(m6))) >> 6) & W & ~H;
			}
			const unsigned pix = (unsigned)((long long)y * w + 32 * k);
			auto put = [&](uint2 *list, unsigned long long *count, uint32_t bits) {
				if (!__any_sync(0xffffffffu, bits != 0))
					return;
				unsigned long long slot = warp_append(count, __popc(bits));
				for (; bits; bits &= bits - 1)
					list[slot++] = make_uint2((unsigned)item.x, pix + __ffs((int)bits) - 1);
			};
			put(eval, &L.n_eval, ne);
			put(cands, &L.n_cand, nh);
			put(low, &L.n_low, nl);
		}
	}
}

// The class of lane's re-evaluated pixel t (0: none, 1: HIGH, 2: LOW) into the
// planes and lists; called by the whole warp, `have`: the lane has one.  GATED:
// the S1, S2 and CAND words are read where a bit can be set and has to go (they
// are set in the classes only), which saves loads but adds a round trip.
template <bool GATED>
__device__ __forceinline__ void late_class(const FrameDesc *__restrict__ frames, uint2 t, int cls, bool have,
	PassLists &L, uint2 *cands, uint2 *low)
{
	const int lane = threadIdx.x & 31;
	bool to_high = false, to_low = false;
	if (have) {
		const FrameDesc &fd = frames[t.x];
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		const long long o = (long long)y * fd.words + (x >> 5);
		const uint32_t bit = 1u << (x & 31);
		uint32_t *H = plane_ptr(fd, P_HIGH) + o, *W = plane_ptr(fd, P_LOW) + o;
		uint32_t *s1 = plane_ptr(fd, P_S1) + o, *s2 = plane_ptr(fd, P_S2) + o, *cd = plane_ptr(fd, P_CAND) + o;
		const bool oh = (*H & bit) != 0, ol = (*W & bit) != 0; // only this thread writes the pixel's bits
		const bool out_high = !GATED || (oh && cls != 1), out = !GATED || ((oh || ol) && cls == 0);
		const bool o1 = out_high && (*s1 & bit), oc = out_high && (*cd & bit), o2 = out && (*s2 & bit);
		to_high = cls == 1 && !oh;
		to_low = cls == 2 && !ol;
		if (to_high)
			atomicOr(H, bit);
		if (oh && cls != 1)
			atomicAnd(H, ~bit);
		if (to_low)
			atomicOr(W, bit);
		if (ol && cls != 2)
			atomicAnd(W, ~bit);
		if (o1 && cls != 1)
			atomicAnd(s1, ~bit);
		if (oc && cls != 1)
			atomicAnd(cd, ~bit);
		if (o2 && cls == 0)
			atomicAnd(s2, ~bit);
		plane_ptr(fd, P_EVAL)[o] = 0u; // every claim of the plane ends in this stage
	}
	const unsigned bh = __ballot_sync(0xffffffffu, to_high), bl = __ballot_sync(0xffffffffu, to_low);
	if (!(bh | bl))
		return;
	unsigned long long at = 0;
	if (lane == 0 && bh)
		at = atomicAdd(&L.n_cand, (unsigned long long)__popc(bh));
	if (lane == 1 && bl)
		at = atomicAdd(&L.n_low, (unsigned long long)__popc(bl));
	const unsigned long long ah = __shfl_sync(0xffffffffu, at, 0), al = __shfl_sync(0xffffffffu, at, 1);
	const unsigned below = (1u << lane) - 1u;
	if (to_high)
		cands[ah + __popc(bh & below)] = t;
	if (to_low)
		low[al + __popc(bl & below)] = t;
}

__device__ __forceinline__ int class_of(double v, const DetectParams &prm)
{
	return v > prm.cr || v != v ? 1 : v > prm.nb ? 2 : 0;
}

// Stage 2 (called by every warp of the grid).  On noise-model frames a pixel
// whose Laplacian is at most its floor block's bound cannot pass either
// threshold; the others wait in the warp's queue Q (64 entries) for the
// median of their window.  Short lists (LATE_SHORT) do both at once, a warp per
// median.  Long ones take two launches, since a thread per median takes 25
// values in registers: LATE_TESTS at full occupancy, which marks the entries it
// settles, then LATE_MEDIANS, 32 of the others at a time (in one launch with
// the medians' registers they took 190 us on 64 ragged noise-model frames of 256
// to 4096 pixels a side, as two 103 and 37).
//
// A long list finds the block thresholds written since the last replacement
// (late_neighbours_kernel).
enum LatePart { LATE_SHORT, LATE_TESTS, LATE_MEDIANS };
constexpr unsigned EVAL_DONE = 0xffffffffu; // the frame of an entry that is settled

template <LatePart PART, bool MODEL = true>
__device__ __forceinline__ void late_classes(const FrameDesc *__restrict__ frames, uint2 *eval,
	const DetectParams &prm, PassLists &L, uint2 *cands, uint2 *low, uint2 *Q, Team team)
{
	const int lane = threadIdx.x & 31;
	const long long gw = (team.block * (long long)blockDim.x + threadIdx.x) >> 5;
	const long long nw = ((long long)team.blocks * blockDim.x) >> 5;
	const long long n = (long long)L.n_eval;
	const int mode = prm.mode, lm = lap_mode(mode);
	const double tmin2 = fmin(prm.thi2, prm.tlo2);
	int nq = 0; // queued (warp-uniform)
	auto drain = [&](int count) { // the first `count` <= 32 queued pixels
		__syncwarp();
		uint2 t = make_uint2(0u, 0u);
		int cls = 0;
		if (PART == LATE_SHORT) {
			t = Q[lane < count ? lane : 0];
			for (int q = 0; q < count; ++q) {
				const uint2 u = Q[q];
				const FrameDesc &fd = frames[u.x];
				const int w = fd.w, x = (int)(u.y % (unsigned)w), y = (int)(u.y / (unsigned)w);
				double c = INFINITY;
				if (lane < 25) {
					const int cx = x + lane % 5 - 2, cy = y + lane / 5 - 2;
					c = cx >= 0 && cy >= 0 && cx < w && cy < fd.h ? fd.clean[(long long)cy * w + cx]
						: clean_at(fd, cx, cy, mode);
				}
				const double lap = lap_at(fd, x, y, lm); // every lane: one round trip with the window
				const double m = __shfl_sync(0xffffffffu, warp_sort32(c), 12);
				const int k = class_of(lap / (2 * noise_from_median(fd, u.y, m)), prm);
				if (lane == q)
					cls = k;
			}
		} else if (lane < count) {
			t = Q[lane];
			const FrameDesc &fd = frames[t.x];
			const int w = fd.w, x = (int)(t.y % (unsigned)w), y = (int)(t.y / (unsigned)w);
			double nz, lap;
			if (x >= 2 && y >= 2 && x + 2 < w && y + 2 < fd.h) {
				double v[25];
				const double *src = fd.clean + t.y - 2 * (long long)w - 2;
#pragma unroll
				for (int a = 0; a < 5; ++a)
#pragma unroll
					for (int b = 0; b < 5; ++b)
						v[a * 5 + b] = src[(long long)a * w + b];
				lap = lap_formula(v[12], v[7], v[17], v[11], v[13]);
				nz = noise_from_median(fd, t.y, median_network(v));
			} else {
				nz = noise_model_at(fd, x, y, mode);
				lap = lap_at(fd, x, y, lm);
			}
			cls = class_of(lap / (2 * nz), prm);
		}
		__syncwarp();
		if (lane + 32 < nq)
			Q[lane] = Q[lane + 32];
		nq -= count;
		__syncwarp();
		late_class<PART != LATE_SHORT>(frames, t, cls, lane < count, L, cands, low);
	};
	// Long lists go to the warps in runs of 32, whose loads share lines; short
	// ones are dealt one by one, so that few medians wait behind each other.
	const long long first = PART == LATE_SHORT ? gw : gw * 32, step = PART == LATE_SHORT ? nw : 1;
	for (long long base = first; base < n; base += nw * 32) {
		const long long e = base + lane * step;
		uint2 t = make_uint2(0u, 0u);
		int cls = 0;
		bool have = e < n, wait = false;
		if (have)
			t = eval[e];
		if (PART == LATE_MEDIANS) {
			wait = have && t.x != EVAL_DONE;
		} else if (have) {
			const FrameDesc &fd = frames[t.x];
			const int w = fd.w, x = (int)(t.y % (unsigned)w), y = (int)(t.y / (unsigned)w);
			double lap;
			if (x >= 1 && y >= 1 && x + 1 < w && y + 1 < fd.h) {
				const double *c = fd.clean + t.y;
				lap = lap_formula(c[0], c[-w], c[w], c[-1], c[1]);
			} else {
				lap = lap_at(fd, x, y, lm);
			}
			if (!MODEL || fd.error) {
				cls = class_of(lap / (2 * fd.error[t.y]), prm);
			} else {
				const double T = PART == LATE_SHORT ? block_threshold(fd, x >> 5, y >> 5, mode, tmin2)
					: fd.floors[(y >> 5) * ((w + 31) >> 5) + (x >> 5)].thr;
				wait = !(T >= 0 && lap <= T);
			}
		}
		if (PART != LATE_MEDIANS)
			late_class<PART != LATE_SHORT>(frames, t, cls, have && !wait, L, cands, low);
		if (PART == LATE_TESTS) {
			if (MODEL && have && !wait)
				eval[e].x = EVAL_DONE;
			continue;
		}
		const unsigned b = __ballot_sync(0xffffffffu, wait);
		if (b) {
			if (wait)
				Q[nq + __popc(b & ((1u << lane) - 1u))] = t;
			nq += __popc(b);
			if (nq >= 32)
				drain(32);
		}
	}
	if (nq)
		drain(nq);
}

// The entries of a list (count() many, which thread 0 asks) by blocks: a thread per
// entry tests it (keep), then the block's warps take the survivors (work, by the
// whole warp) from a queue in shared memory.  A block's share shrinks with the list,
// so that a short one spreads over the team.  The entries of a short list are dealt
// to the blocks one by one, so neighbouring entries, whose survivors come in
// clusters, go to different blocks; those of a long one in runs of 32, whose tests'
// loads share lines.  aside: other work of every warp, done before the first
// sweep's barrier, beside other warps' tests.  many: called by the whole block with
// the survivors of chunk k queued; it may take some.
//
// What is the same for the whole block stays in shared memory: the work holds
// every register of a thread (80 at this block size), and what lives across it
// spills.
struct LateQueue {
	uint16_t e[LATE_THREADS];
	int n;
	int chunk, run; // run: entries dealt at a time, as a power of two
	Team team;
	unsigned end; // (no list has 2^32 entries: a pixel takes more than 50 bytes of lists)

	// Entry of slot j of the block's k-th chunk.
	__device__ __forceinline__ unsigned entry(unsigned k, unsigned j) const
	{
		const unsigned i = k * chunk + j;
		return ((team.block + team.blocks * (i >> run)) << run) + (i & ((1u << run) - 1u));
	}
};

template <class Count, class Keep, class Many, class Work, class Aside>
__device__ __forceinline__ void block_sweep(Count count, LateQueue &Q, Team team, Keep keep, Many many, Work work,
	Aside aside)
{
	const int warp = threadIdx.x >> 5;
	if (threadIdx.x == 0) { // (a barrier of the team lies between two sweeps)
		const long long n = count(), share = (n + team.blocks - 1) / team.blocks;
		Q.chunk = share < LATE_THREADS ? (int)share : LATE_THREADS;
		Q.run = share < LATE_THREADS ? 0 : 5;
		Q.team = team;
		Q.end = (unsigned)n;
	}
	for (int k = 0;; ++k) { // block-uniform
		if (threadIdx.x == 0)
			Q.n = 0;
		__syncthreads();
		if (k == 0)
			aside();
		if ((int)threadIdx.x < Q.chunk) {
			const unsigned e = Q.entry(k, threadIdx.x);
			if (e < Q.end && keep(e))
				Q.e[atomicAdd(&Q.n, 1)] = (uint16_t)threadIdx.x;
		}
		__syncthreads();
		many(k);
		for (int q = warp; q < Q.n; q += LATE_WARPS)
			work(Q.entry(k, Q.e[q]));
		__syncthreads();
		if (!Q.chunk || Q.entry(k + 1, 0) >= Q.end)
			return;
	}
}

// Stage 3: the listed pixels that are HIGH (and no hole) now, a warp each.
template <class Count>
__device__ __forceinline__ void late_candidates(const FrameDesc *__restrict__ frames, const uint2 *cands,
	const DetectParams &prm, Count count, LateQueue &Q, Team team, double *P, double *S, double (*T)[63])
{
	const int lane = threadIdx.x & 31;
	block_sweep(count, Q, team, [&](unsigned e) {
		const uint2 t = cands[e];
		const FrameDesc &fd = frames[t.x];
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		return test_bit(plane_ptr(fd, P_HIGH), fd.words, x, y) &
			!test_bit(plane_ptr(fd, P_HOLE), fd.words, x, y);
	}, [](int) {}, [&](unsigned e) {
		const uint2 t = cands[e];
		const FrameDesc &fd = frames[t.x];
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		const bool excl = test_bit(plane_ptr(fd, P_EXCL), fd.words, x, y);
		const Sig g = candidate_sig<false, PATH_ANY>(fd, x, y, P, S, prm, false);
		if (g.s1 && !excl) // warp-uniform
			seed_eval(fd, x, y, g.lo, g.hi, g.noise, prm, P, T, false, true, [&] { return exact_sig(g); });
		else if (lane == 0)
			write_bit(plane_ptr(fd, P_CAND) + (long long)y * fd.words + (x >> 5), 1u << (x & 31), false);
	}, [] {});
}

// Stage 4, the high list's part: eight lanes grow around each listed pixel.
// The entries are dealt to the blocks in fours, and within a block to its last
// warps first (its first ones have the low list's entries).
__device__ __forceinline__ void late_grow(const FrameDesc *__restrict__ frames, FrameState *state,
	const uint2 *cands, const PassLists &L, Control *ctl, int par, uint2 *targets, Team team)
{
	const long long n = (long long)L.n_cand;
	const int back = LATE_WARPS - 1 - (threadIdx.x >> 5), lane = threadIdx.x & 31;
	for (long long base = 4 * ((long long)back * team.blocks + team.block); base < n;
	     base += 4ll * LATE_WARPS * team.blocks) { // warp-uniform
		const long long e = base + (lane >> 3);
		const uint2 t = e < n ? cands[e] : make_uint2(0u, 0u);
		const FrameDesc &fd = frames[t.x];
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		if (e < n && (lane & 7) == 0)
			plane_ptr(fd, P_LISTED)[(long long)y * fd.words + (x >> 5)] = 0u;
		grow_group(fd, (int)t.x, x, y, e < n, GROW_LATE, true, state, ctl, par, targets);
	}
}

// Stage 4: the growth, and the low list's pixels near a CAND pixel, a warp each.
__device__ __forceinline__ void late_low(const FrameDesc *__restrict__ frames, FrameState *state,
	const uint2 *cands, const uint2 *low, const DetectParams &prm, const PassLists &L, Control *ctl, int par,
	uint2 *targets, const RowItems &rows, LateQueue &Q, Team team, double *P, double *S)
{
	block_sweep([&] { return (long long)L.n_low; }, Q, team, [&](unsigned e) {
		const uint2 t = low[e];
		const FrameDesc &fd = frames[t.x];
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		plane_ptr(fd, P_LISTED)[(long long)y * fd.words + (x >> 5)] = 0u;
		return low_near(fd, x, y);
	}, [](int) {}, [&](unsigned e) {
		low_eval<PATH_ANY>(frames, state, low[e], prm, ctl, par, targets, P, S, false);
	}, [&] {
		if (grows_by_rows(L.n_cand, rows))
			grow_rows(frames, state, rows, true, ctl, par, targets, team);
		else
			late_grow(frames, state, cands, L, ctl, par, targets, team);
	});
}

// Stage 5: the replacement, by warps (few targets are left to do).  A target
// whose last replacement used a window of radius r <= KEEP_RADIUS_MAX without
// a pixel of FRESH (what this pass's growth flagged) keeps its value: donors
// are never added (the mask only grows) and keep their values, so the smaller
// windows still hold none, the same window holds the same donors, and the same
// median would come out.  A new target is itself a FRESH pixel.
//
// A block with LATE_BY_THREADS or more of a chunk's targets left (LATE_THREADS at
// most) gives them a thread each first, as replace_targets does (the 25 values spill,
// and are still faster than a warp per target).
constexpr int LATE_BY_THREADS = 256;

// (Called by the whole block; a function of its own, so that its registers are not
// the kernel's.)
__device__ __noinline__ void late_replace_threads(const FrameDesc *__restrict__ frames, const uint2 *targets,
	uint8_t *radius, unsigned *chg, unsigned long long *n_chg, LateQueue &Q, int k)
{
	const int n = Q.n, lane = threadIdx.x & 31;
	int left = -1; // the thread's slot, if it is left to the warps
	unsigned e = 0;
	bool changed = false;
	if ((int)threadIdx.x < n) {
		const int slot = Q.e[threadIdx.x];
		e = Q.entry(k, slot);
		const uint2 t = targets[e];
		const FrameDesc &fd = frames[t.x];
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		double v;
		if (first_window_value(fd, x, y, v)) {
			double &dst = fd.clean[t.y];
			changed = __double_as_longlong(dst) != __double_as_longlong(v);
			dst = v;
			radius[e] = 2;
			if (!fd.error) // keep the block's floor a lower bound of its clean values
				atomicMin(&fd.floors[(y >> 5) * ((fd.w + 31) >> 5) + (x >> 5)].key, order_key(v));
		} else {
			left = slot;
		}
	}
	const unsigned b = __ballot_sync(0xffffffffu, changed);
	unsigned long long at = 0;
	if (lane == 0 && b)
		at = atomicAdd(n_chg, (unsigned long long)__popc(b));
	at = __shfl_sync(0xffffffffu, at, 0);
	if (changed)
		chg[at + __popc(b & ((1u << lane) - 1u))] = e;
	__syncthreads();
	if (threadIdx.x == 0)
		Q.n = 0;
	__syncthreads();
	if (left >= 0)
		Q.e[atomicAdd(&Q.n, 1)] = (uint16_t)left;
	__syncthreads();
}

__device__ __forceinline__ void late_replace(const FrameDesc *__restrict__ frames, const FrameState *state,
	int par, const uint2 *targets, const Control *ctl, uint8_t *radius, unsigned *chg, unsigned long long *n_chg,
	LateQueue &Q, Team team)
{
	const unsigned fresh0 = (unsigned)ctl->fresh0;
	block_sweep([&] { return (long long)ctl->n_targets; }, Q, team, [&](unsigned e) {
		const uint2 t = targets[e];
		const int r = radius[e]; // (a new target's is not set yet)
		if (!replaces(state[t.x], par))
			return false;
		if (e >= fresh0 || r > KEEP_RADIUS_MAX)
			return true;
		const FrameDesc &fd = frames[t.x];
		return fresh_in_window(fd, (int)(t.y % (unsigned)fd.w), (int)(t.y / (unsigned)fd.w), r);
	}, [&](int k) {
		if (Q.n >= LATE_BY_THREADS) // block-uniform
			late_replace_threads(frames, targets, radius, chg, n_chg, Q, k);
	}, [&](unsigned e) {
		const uint2 t = targets[e];
		const FrameDesc &fd = frames[t.x];
		bool changed = false;
		const int r = replace_one(fd, (int)(t.y % (unsigned)fd.w), (int)(t.y / (unsigned)fd.w), &changed);
		if ((threadIdx.x & 31) == 0) {
			radius[e] = (uint8_t)(r < 255 ? r : 255);
			if (changed)
				chg[atomicAdd(n_chg, 1ull)] = e;
		}
	}, [] {});
}

// Stages 1 and 2 of the first late pass, which starts from every target of the
// full pass: launches of their own, whose registers let 48 and more warps per
// SM hide the claims' and loads' latency.
constexpr int LN_THREADS = 512;

__global__ void __launch_bounds__(LN_THREADS, 3)
late_neighbours_kernel(const FrameDesc *__restrict__ frames, const FrameState *state, DetectParams prm,
	Control *ctl, uint2 *cands, uint2 *low, uint2 *eval, const uint2 *targets, const unsigned *chg,
	RowItems rows, const FloorJob *__restrict__ jobs, int njobs)
{
	__shared__ ListSlots slots;
	// The noise-model blocks' thresholds, for the long lists' LATE_TESTS (a
	// thread per block; the replacement lowered the floors).
	const double tmin2 = fmin(prm.thi2, prm.tlo2);
	for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < njobs; j += gridDim.x * blockDim.x) {
		const FloorJob jb = jobs[j];
		const FrameDesc &fd = frames[jb.frame];
		if (!fd.error)
			fd.floors[(jb.y0 >> 5) * ((fd.w + 31) >> 5) + (jb.x0 >> 5)].thr =
				block_threshold(fd, jb.x0 >> 5, jb.y0 >> 5, prm.mode, tmin2);
	}
	if (late_by_rows(ctl, ctl->pass[1], rows)) {
		late_rows(frames, state, rows, ctl->pass[1], prm.mode, cands, low, eval, whole_grid());
		return;
	}
	late_neighbours<LN_THREADS / 32>(frames, targets, chg, ctl->pass[1], prm.mode, cands, low, eval, slots,
		whole_grid());
}

// MODEL: the batch has noise-model frames (launch_late has the choice of parts).
template <LatePart PART, bool MODEL>
__global__ void __launch_bounds__(256, PART == LATE_MEDIANS ? 2 : 6)
late_classes_kernel(const FrameDesc *__restrict__ frames, DetectParams prm, Control *ctl, uint2 *cands,
	uint2 *low, uint2 *eval)
{
	constexpr bool QUEUED = PART != LATE_TESTS;
	__shared__ uint2 queue[QUEUED ? 8 : 1][64];
	late_classes<PART, MODEL>(frames, eval, prm, ctl->pass[1], cands, low, queue[QUEUED ? threadIdx.x >> 5 : 0],
		whole_grid());
}

struct LateShared {
	double patches[LATE_WARPS][81];
	double scratch[LATE_WARPS][CS_RUNS]; // sorted runs or triples of a warp's patch
	uint2 queue[LATE_WARPS][64];
	LateQueue Q;
	ListSlots slots;
};

// Passes 1 .. maxiter - 1 (the full pass is number 0; maxiter >= 2), the first of
// them from stage 3.  cands: the high list; low, eval: buffers of as many entries as the
// batch has pixels (the first pass's pre list, which is done with); chg: the
// changed targets' indices.
__global__ void __launch_bounds__(LATE_THREADS, 1)
late_passes_kernel(const FrameDesc *__restrict__ frames, FrameState *state, int nf, DetectParams prm,
	Control *ctl, int maxiter, uint2 *cands, uint2 *low, uint2 *eval, uint2 *targets, uint8_t *radius,
	unsigned *chg, RowItems rows, BarrierWait bw)
{
	extern __shared__ __align__(16) unsigned char late_smem[];
	LateShared &S = *reinterpret_cast<LateShared *>(late_smem);
	const int warp = threadIdx.x >> 5;
	__shared__ Team team;
	__shared__ struct {
		int any;
		unsigned long long n_chg;
		long long n_cand;
	} begin;
	if (threadIdx.x == 32) { // beside the join: these change only after the team's first barrier
		begin.any = *(volatile int *)&ctl->any[0];
		begin.n_chg = *(volatile unsigned long long *)&ctl->pass[1].n_chg;
		begin.n_cand = *(volatile long long *)&ctl->pass[1].n_cand;
	}
	__shared__ BarrierState barrier;
	if (threadIdx.x == 0)
		barrier.calls = 0;
	if (!join_team(ctl, team))
		return;
	const bool first = team.block == 0 && threadIdx.x == 0;
	double (*triples)[63] = reinterpret_cast<double (*)[63]>(&S.scratch[warp][0]);
	static_assert(3 * 63 <= CS_RUNS, "the triples fit the runs' scratch");
	// Whether the loop ends before the pass of parity par: every frame stopped after
	// the last pass, or its replacement changed no value, so that this pass would
	// repeat it and find nothing new.
	auto ends = [&](int any, unsigned long long n_chg, int par, unsigned blocks) {
		if (any && !n_chg)
			pass_control(state, nf, ctl, par, Team{team.block, blocks});
		return !any || !n_chg;
	};
	if (ends(begin.any, begin.n_chg, 1, gridDim.x))
		return; // (nobody closes the team)
	for (int it = 1;; ++it) {
		const int par = it & 1;
		PassLists &L = ctl->pass[par], &next = ctl->pass[par ^ 1];
		if (it > 1) {
			if (late_by_rows(ctl, L, rows))
				late_rows(frames, state, rows, L, prm.mode, cands, low, eval, team);
			else
				late_neighbours<LATE_WARPS>(frames, targets, chg, L, prm.mode, cands, low, eval, S.slots, team);
			// The last growth's FRESH bits: its replacement is done.
			for (long long i = (long long)ctl->fresh0 + team.block * (long long)blockDim.x + threadIdx.x;
			     i < (long long)ctl->n_targets; i += (long long)team.blocks * blockDim.x) {
				const uint2 t = targets[i];
				const FrameDesc &fd = frames[t.x];
				plane_ptr(fd, P_FRESH)[(long long)(t.y / (unsigned)fd.w) * fd.words +
					((t.y % (unsigned)fd.w) >> 5)] = 0u;
			}
			if (!grid_barrier(ctl, barrier, state, nf, bw, team))
				return;
			late_classes<LATE_SHORT>(frames, eval, prm, L, cands, low, S.queue[warp], team);
			if (!grid_barrier(ctl, barrier, state, nf, bw, team))
				return;
		}
		if (first) { // what the coming stages and the next pass append to
			ctl->fresh0 = ctl->n_targets;
			next = PassLists{};
			ctl->any[par] = 0;
		}
		// The block's share; in the first pass of the grid's shares, then of those
		// whose blocks did not come, a barrier after each round.
		do { // block-uniform
			const unsigned share = (it > 1 ? 0u : barrier.calls * team.blocks) + team.block;
			const unsigned shares = it > 1 ? team.blocks : gridDim.x;
			if (share < shares)
				late_candidates(frames, cands, prm, [&] { return it > 1 ? (long long)L.n_cand : begin.n_cand; },
					S.Q, Team{share, shares}, S.patches[warp], S.scratch[warp], triples);
			if (!grid_barrier(ctl, barrier, state, nf, bw, team))
				return;
		} while (it == 1 && barrier.calls * team.blocks < gridDim.x);
		late_low(frames, state, cands, low, prm, L, ctl, par, targets, rows, S.Q, team, S.patches[warp],
			S.scratch[warp]);
		if (!grid_barrier(ctl, barrier, state, nf, bw, team))
			return;
		pass_control(state, nf, ctl, par, team);
		late_replace(frames, state, par, targets, ctl, radius, chg, &next.n_chg, S.Q, team);
		if (it + 1 >= maxiter || !grid_barrier(ctl, barrier, state, nf, bw, team))
			return;
		const int any = *(volatile int *)&ctl->any[par];
		if (ends(any, *(volatile unsigned long long *)&next.n_chg, par ^ 1, team.blocks))
			return;
	}
}

} // namespace cb
