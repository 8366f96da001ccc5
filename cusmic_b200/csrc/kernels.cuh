// Per-pass kernels around the detection kernel: preparation, bit-packed growth
// and mask update, loop control, replacement, restoration.
//
// Row kernels give one warp a frame row at a time (a row-item list of
// {frame, y} covers ragged batches), so each warp instruction reads 32
// consecutive float64 pixels and the bit planes fall out of __ballot_sync.
#pragma once
#include "common.cuh"
#include "select.cuh"

namespace cb {

__device__ __forceinline__ int warp_sum_int(int v)
{
#pragma unroll
	for (int o = 16; o; o >>= 1)
		v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

__device__ __forceinline__ int warp_inclusive_count(int cnt)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		int v = __shfl_up_sync(0xffffffffu, cnt, o);
		if (lane >= o)
			cnt += v;
	}
	return cnt;
}

__device__ __forceinline__ int warp_exclusive_count(int cnt)
{
	return warp_inclusive_count(cnt) - cnt;
}

// Append `cnt` entries per lane to a global list; returns this lane's first slot.
__device__ __forceinline__ unsigned long long warp_append(unsigned long long *counter, int cnt)
{
	const int lane = threadIdx.x & 31;
	int incl = cnt;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		int v = __shfl_up_sync(0xffffffffu, incl, o);
		if (lane >= o)
			incl += v;
	}
	int total = __shfl_sync(0xffffffffu, incl, 31);
	unsigned long long base = 0;
	if (lane == 31 && total)
		base = atomicAdd(counter, (unsigned long long)total);
	base = __shfl_sync(0xffffffffu, base, 31);
	return base + (unsigned long long)(incl - cnt);
}

// Map validation of the host entry point on the device (reference
// src/api.cu:107-114 runs it on the host): sets `bit` in *flags if any of the
// n values is not finite, or (minimum 1) not positive, or (minimum 0)
// negative.
__global__ void __launch_bounds__(256)
validate_kernel(const double *__restrict__ v, long long n, int minimum, unsigned *flags, unsigned bit)
{
	bool bad = false;
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
	     i += (long long)gridDim.x * blockDim.x) {
		const double x = v[i];
		bad |= !isfinite(x) || (minimum == 1 && x <= 0) || (minimum == 0 && x < 0);
	}
	if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0)
		atomicOr(flags, bit);
}

// The same for the maps of a device call, in one launch that tells the two
// failures apart: of map i, bit 2 i of *flags is set by a value that is not
// finite, bit 2 i + 1 by one that is not positive (minimum 1) or negative
// (minimum 0).  Bound by reading each value once, two per load where the map is
// 16-byte aligned: 9 us for one 2048 x 2048 map, where the tensor library's
// checks (isfinite in four passes, a comparison and two reductions) took 60 us
// of device time in 11 launches.
struct MapChecks {
	struct {
		const double *v;
		long long n;
		int minimum;
	} map[4];
	int count;
};

__global__ void __launch_bounds__(256)
check_maps_kernel(MapChecks c, unsigned *flags)
{
	const long long stride = (long long)gridDim.x * blockDim.x;
	const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	unsigned bad = 0;
	for (int k = 0; k < c.count; ++k) {
		const double *v = c.map[k].v;
		const long long n = c.map[k].n;
		const int minimum = c.map[k].minimum;
		bool inf = false, low = false;
		auto test = [&](double x) {
			inf |= !isfinite(x);
			low |= minimum == 1 ? x <= 0 : minimum == 0 ? x < 0 : false;
		};
		const long long pairs = ((uintptr_t)v & 15u) == 0 ? n / 2 : 0;
		const double2 *v2 = reinterpret_cast<const double2 *>(v);
#pragma unroll 4
		for (long long i = first; i < pairs; i += stride) {
			const double2 x = v2[i];
			test(x.x);
			test(x.y);
		}
		for (long long i = 2 * pairs + first; i < n; i += stride)
			test(v[i]);
		bad |= (unsigned)inf << (2 * k) | (unsigned)low << (2 * k + 1);
	}
	bad = __reduce_or_sync(0xffffffffu, bad);
	if (bad && (threadIdx.x & 31) == 0)
		atomicOr(flags, bad);
}

// What a call's first launch zeroes: the n16 16-byte words of the bit planes
// that nothing writes before the first pass, and the output masks (of which
// finish_kernel sets the flagged pixels): `bytes` bytes, the frames' masks back
// to back, from the first descriptor's (a plan's buffers change, its launches
// do not).
struct ZeroRange {
	uint4 *planes;
	long long n16;
	const FrameDesc *frames;
	long long bytes;
};

// The masks of that: the aligned body by 16 bytes, the ends byte by byte.
__device__ __forceinline__ void zero_masks(const ZeroRange &z)
{
	if (!z.bytes)
		return;
	const long long stride = (long long)gridDim.x * blockDim.x;
	const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	uint8_t *mask = z.frames[0].mask_out;
	const long long head = min(z.bytes, (long long)(-(uintptr_t)mask & 15u));
	const long long body = (z.bytes - head) / 16, tail = z.bytes - head - 16 * body;
	uint4 *m16 = reinterpret_cast<uint4 *>(mask + head);
	for (long long j = first; j < body; j += stride)
		m16[j] = make_uint4(0u, 0u, 0u, 0u);
	if (first < head)
		mask[first] = 0;
	if (first < tail)
		mask[head + 16 * body + first] = 0;
}

// The same in a launch of its own, after prepare: for a batch whose output masks
// take an input mask's place.
__global__ void __launch_bounds__(256)
zero_masks_kernel(ZeroRange z)
{
	zero_masks(z);
}

// Per-frame state and loop control of a call, and the zeroing, with grid-stride
// loops of 16-byte stores.
__device__ __forceinline__ void init_state(FrameState *state, int nf, Control *ctl, int maxiter,
	unsigned long long cand_cap, long long poison_prepare, long long poison_detect, const ZeroRange &z)
{
	const long long stride = (long long)gridDim.x * blockDim.x;
	const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	for (long long j = first; j < z.n16; j += stride)
		z.planes[j] = make_uint4(0u, 0u, 0u, 0u);
	zero_masks(z);
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < nf) {
		FrameState s = {};
		s.active = maxiter > 0;
		state[i] = s;
	}
	if (i == 0) {
		Control c = {};
		c.cand_cap = cand_cap;
		c.poison_wait[0] = poison_prepare;
		c.poison_wait[1] = poison_detect;
		*ctl = c;
	}
}

__global__ void init_kernel(FrameState *state, int nf, Control *ctl, int maxiter,
	unsigned long long cand_cap, long long poison_prepare = 0, long long poison_detect = 0,
	ZeroRange zero = ZeroRange{})
{
	init_state(state, nf, ctl, maxiter, cand_cap, poison_prepare, poison_detect, zero);
}

// IEEE bits mapped to an unsigned total order (reference src/replace.cuh:37-48).
__device__ __forceinline__ unsigned long long order_key(double v)
{
	unsigned long long b = (unsigned long long)__double_as_longlong(v);
	return (b >> 63) ? ~b : b ^ (1ull << 63);
}

__device__ __forceinline__ double order_value(unsigned long long k)
{
	return __longlong_as_double((long long)((k >> 63) ? k ^ (1ull << 63) : ~k));
}

// Reference src/image.cuh:24-48: holes, exclusions, clean = data (+ bg), the
// static donor plane (the reference's is_donor with an empty mask) and the
// per-frame facts the initial fill needs (src/cleaner.cuh:78-100).  A warp
// loads several chunks of 32 pixels before using them, so enough bytes are in
// flight per SM to approach the HBM bandwidth (launch_prepare).

// Frame kinds of prepare_row: the input maps it reads and whether it writes
// noise-model row minima (PREP_ANY decides per row).
enum PrepKind { PREP_ANY, PREP_PLAIN, PREP_MASK, PREP_MAPS, PREP_MODEL, PREP_MODEL_MAPS };

CB_HD int prep_kind(const FrameDesc &fd)
{
	const bool mask = fd.mask, bgmap = fd.bg_map;
	if (fd.floors && !fd.error) // noise-model frame: row minima for the floors
		return mask || bgmap ? PREP_MODEL_MAPS : PREP_MODEL;
	return bgmap ? PREP_MAPS : mask ? PREP_MASK : PREP_PLAIN;
}


// One row of prepare_kernel for the frame kinds that occur: MASK = input
// mask, BGMAP = background map.  Descriptor fields are held in registers (the
// stores below go through pointers the compiler cannot prove distinct from
// them).
//
// W words of the row at once, the rest in groups of 4.  Memory bounds it (64
// ragged noise-model frames of 256 to 4096 pixels a side, 178 Mpix of 24 bytes:
// 858 us with 8 words in flight and a tail group of 8, 705 us).  On small frames
// it was bound by its last lines, where lane 0 tested each frame flag before
// setting it, three waits in a row behind the other rows' additions to the
// sector (256 frames of 40 to 200 pixels: 68 us, 17 without).
template <bool MASK, bool BGMAP, bool ROWMIN, int W, bool OUT>
__device__ __forceinline__ void prepare_row(const FrameDesc &fd, FrameState &st, int f, int y, Control *ctl,
	uint2 *holes)
{
	const int lane = threadIdx.x & 31;
	const int w = fd.w, words = fd.words;
	const long long rowpix = (long long)y * w, roww = (long long)y * words;
	const double *__restrict__ data = fd.data + rowpix;
	// MASK / BGMAP false: the frame has none; true: it may have one.
	const uint8_t *__restrict__ mask = MASK && fd.mask ? fd.mask + rowpix : nullptr;
	const double *__restrict__ bgmap = BGMAP && fd.bg_map ? fd.bg_map + rowpix : nullptr;
	double *__restrict__ clean = fd.clean + rowpix;
	// A separate output buffer (a frame with a background): its pixels now,
	// (x + bg) - bg as the reference's restore computes them, the input at a
	// hole; finish_kernel writes only the flagged ones.
	double *__restrict__ out = OUT && fd.out && fd.out != fd.clean ? fd.out + rowpix : nullptr;
	const double bgv = fd.bg;
	const bool has_bg = fd.has_bg;
	uint32_t *hole_plane = plane_ptr(fd, P_HOLE) + roww, *excl_plane = plane_ptr(fd, P_EXCL) + roww;
	uint32_t *donor_plane = plane_ptr(fd, P_DONOR) + roww;
	// Noise-model frames with floors: per bit word the smallest high word of
	// the ordered keys of the non-hole clean values (a lower bound for the
	// block floors, which the hole fill then lowers with the values it writes).
	uint32_t *rowmin = ROWMIN ? plane_ptr(fd, P_ROWMIN) + roww : nullptr;
	uint32_t any_hole = 0, any_allowed = 0; // of this lane's words
	int ndonor = 0;
	for (int seg = 0; seg < words; seg += 32) {
		uint32_t my_h = 0, my_e = 0, my_d = 0, my_m = 0xffffffffu;
		// Words k = seg + c and on, `count` of them; FULL: all inside the row.
		auto group = [&](int c, auto count, auto full) {
			constexpr int U = decltype(count)::value;
			constexpr bool FULL = decltype(full)::value;
			const int xl = 32 * (seg + c) + lane;
			double d[U], bg[U];
			bool m[U];
#pragma unroll
			for (int u = 0; u < U; ++u) {
				const int x = xl + 32 * u;
				d[u] = 0;
				bg[u] = bgv;
				m[u] = false;
				if (FULL || x < w) {
					d[u] = data[x];
					if (MASK && mask)
						m[u] = mask[x] != 0;
					if (BGMAP && bgmap)
						bg[u] = bgmap[x];
				}
			}
			// Without a mask most groups are all donors, which one ballot
			// shows: the value is finite only where the pixel is.
			if (FULL && !MASK) {
				bool good = true;
#pragma unroll
				for (int u = 0; u < U; ++u)
					good = good && isfinite(has_bg ? d[u] + 1 * bg[u] : d[u]);
				if (__all_sync(0xffffffffu, good)) {
#pragma unroll
					for (int u = 0; u < U; ++u) {
						const double v = has_bg ? d[u] + 1 * bg[u] : d[u];
						clean[xl + 32 * u] = v;
						if (OUT && out)
							out[xl + 32 * u] = v + -1 * bg[u];
						const uint32_t mw = ROWMIN
							? __reduce_min_sync(0xffffffffu, (uint32_t)(order_key(v) >> 32)) : 0u;
						if (lane == c + u) {
							my_d = 0xffffffffu;
							my_m = mw;
						}
					}
					return;
				}
			}
#pragma unroll
			for (int u = 0; u < U; ++u) {
				const int x = xl + 32 * u;
				const bool valid = FULL || x < w, hole = valid && !isfinite(d[u]);
				double v = hole ? 0 : d[u];
				if (has_bg)
					v += 1 * bg[u];
				if (valid) {
					clean[x] = v;
					if (OUT && out)
						out[x] = hole ? d[u] : v + -1 * bg[u];
				}
				const uint32_t hw = __ballot_sync(0xffffffffu, hole);
				const uint32_t ew = MASK ? __ballot_sync(0xffffffffu, valid && (hole || m[u])) : hw;
				const uint32_t dw = __ballot_sync(0xffffffffu, valid && !hole && !m[u] && isfinite(v));
				const uint32_t mw = ROWMIN ? __reduce_min_sync(0xffffffffu,
					valid && !hole ? (uint32_t)(order_key(v) >> 32) : 0xffffffffu) : 0u;
				if (lane == c + u) {
					my_h = hw;
					my_e = ew;
					my_d = dw;
					my_m = mw;
				}
			}
		};
		const int n = min(32, words - seg);
		int c = 0;
		for (; c + W <= n && 32 * (seg + c + W) <= w; c += W)
			group(c, std::integral_constant<int, W>{}, std::true_type{});
		for (; c < n; c += 4) {
			if (W > 4 && 32 * (seg + c + 4) <= w)
				group(c, std::integral_constant<int, 4>{}, std::true_type{});
			else
				group(c, std::integral_constant<int, 4>{}, std::false_type{});
		}
		const int k = seg + lane;
		if (k < words) {
			hole_plane[k] = my_h;
			excl_plane[k] = my_e;
			donor_plane[k] = my_d;
			if (ROWMIN)
				rowmin[k] = my_m;
			any_hole |= my_h;
			any_allowed |= ~my_e & (w - 32 * k >= 32 ? 0xffffffffu : (1u << (w - 32 * k)) - 1u);
			ndonor += __popc(my_d);
		}
		if (holes && __any_sync(0xffffffffu, my_h != 0)) { // list the segment's holes for the fill
			unsigned long long slot = warp_append(&ctl->n_holes, __popc(my_h));
			for (uint32_t b = my_h; b; b &= b - 1)
				holes[slot++] = make_uint2((unsigned)f, (unsigned)(rowpix + 32 * k + __ffs(b) - 1));
		}
	}
	any_hole = __ballot_sync(0xffffffffu, any_hole != 0);
	any_allowed = __ballot_sync(0xffffffffu, any_allowed != 0);
	ndonor = __reduce_add_sync(0xffffffffu, ndonor);
	if (lane == 0) {
		if (any_hole)
			atomicAdd(&st.holes, 1ull);
		if (ndonor)
			atomicAdd(&st.donors, (unsigned long long)ndonor);
		else if (any_allowed)
			atomicAdd(&st.allowed, 1ull);
	}
}

// One warp per row (grid-stride over the row list), in segments of 32 words
// (1024 pixels): lane j keeps the HOLE, EXCL and DONOR words of the
// segment's word j, so each plane gets one coalesced store per segment.  The
// other planes were zeroed before the kernel.  With `holes`, each segment's
// holes are appended to that list (count in ctl->n_holes) for the hole fill.
// KIND: the frame kind every row has (PREP_ANY: decided per row); W: the words
// of a row in flight; OUT: some frame of the batch has a separate output buffer;
// MINB: blocks per SM, which leaves the registers for W.
template <int KIND, int W, bool OUT, int MINB>
__global__ void __launch_bounds__(256, MINB)
prepare_kernel(const FrameDesc *__restrict__ frames, FrameState *state, const int2 *__restrict__ rows,
	int nrows, Control *ctl = nullptr, uint2 *holes = nullptr)
{
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	int2 next = gw < nrows ? rows[gw] : make_int2(0, 0);
	for (int r = gw; r < nrows; r += nw) {
		const int2 item = next;
		if (r + nw < nrows) // the next row's entry loads during this row
			next = rows[r + nw];
		const FrameDesc &fd = frames[item.x];
		FrameState &st = state[item.x];
		switch (KIND == PREP_ANY ? prep_kind(fd) : KIND) {
		case PREP_MODEL:
			prepare_row<false, false, true, W, OUT>(fd, st, item.x, item.y, ctl, holes);
			break;
		case PREP_MODEL_MAPS:
			prepare_row<true, true, true, W, OUT>(fd, st, item.x, item.y, ctl, holes);
			break;
		case PREP_MASK:
			prepare_row<true, false, false, W, OUT>(fd, st, item.x, item.y, ctl, holes);
			break;
		case PREP_PLAIN:
			prepare_row<false, false, false, W, OUT>(fd, st, item.x, item.y, ctl, holes);
			break;
		default:
			prepare_row<true, true, false, W, OUT>(fd, st, item.x, item.y, ctl, holes);
		}
	}
}

// Reference src/replace.cuh:50-56.
__device__ __forceinline__ double midpoint(double lo, double hi)
{
	if (fabs(lo) < 1 && fabs(hi) < 1)
		return (lo + hi) / 2;
	return lo / 2 + hi / 2;
}

// Ascending bitonic network over the 32 lanes with the reference's exchange
// (src/replace.cuh:68-83): strict < comparisons, so equal values (such as -0
// and +0) end in the same lanes as in the reference.
__device__ __forceinline__ double bitonic32(double v)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int span = 2; span <= 32; span *= 2) {
#pragma unroll
		for (int step = span / 2; step; step /= 2) {
			double peer = __shfl_xor_sync(0xffffffffu, v, step);
			bool lower = ((lane & span) == 0) == ((lane & step) == 0);
			v = lower ? (peer < v ? peer : v) : (v < peer ? peer : v);
		}
	}
	return v;
}

struct Window {
	int x0, x1, y0, y1;
};

__device__ __forceinline__ bool donor_at(const uint32_t *don, const uint32_t *crm, int words,
	int x, int y)
{
	long long o = (long long)y * words + (x >> 5);
	return ((don[o] & ~crm[o]) >> (x & 31)) & 1u;
}

// The cells at Chebyshev distance r (>= 1) of (x, y) inside a w x h frame, in
// row-major order: `top` cells of the row above the middle rows, `sides` (0 to 2)
// of each of the `mid` middle rows, then the row below.
struct Ring {
	int x0, y, r, top, mid, sides, n; // n: all cells, at most 2 (w + h)
	int left, right, ymid;            // columns of the sides, first middle row
};

CB_HD Ring ring_cells(int w, int h, int x, int y, int r)
{
	Ring q;
	const int x1 = x + r < w ? x + r : w - 1, y1 = y + r < h ? y + r : h - 1;
	q.x0 = x - r > 0 ? x - r : 0;
	q.y = y;
	q.r = r;
	q.top = y - r >= 0 ? x1 - q.x0 + 1 : 0;
	q.ymid = y - r >= 0 ? y - r + 1 : 0;
	q.mid = (y + r < h ? y1 - 1 : y1) - q.ymid + 1;
	q.sides = (x - r >= 0) + (x + r < w);
	q.left = x - r >= 0 ? x - r : x + r;
	q.right = x + r;
	q.n = q.top + q.mid * q.sides + (y + r < h ? x1 - q.x0 + 1 : 0);
	return q;
}

CB_HD void ring_cell(const Ring &q, int pos, int &cx, int &cy)
{
	if (pos < q.top) {
		cx = q.x0 + pos;
		cy = q.y - q.r;
		return;
	}
	pos -= q.top;
	if (pos < q.mid * q.sides) {
		const int row = q.sides == 2 ? pos >> 1 : pos;
		cx = q.sides == 2 && (pos & 1) ? q.right : q.left;
		cy = q.ymid + row;
		return;
	}
	cx = q.x0 + pos - q.mid * q.sides;
	cy = q.y + q.r;
}

// Distance from bit c (which may lie outside 0 .. 31) to the nearest set bit of
// the word b (not zero).
CB_HD int bit_distance(uint32_t b, int c)
{
	int best = 1 << 30;
	const uint32_t low = c < 0 ? 0u : c >= 31 ? b : b & ((2u << c) - 1u), high = c <= 0 ? b : c > 31 ? 0u : b >> c;
#if defined(__CUDA_ARCH__)
	if (low)
		best = c - (31 - __clz((int)low));
	if (high)
		best = min(best, __ffs((int)high) - 1 - (c < 0 ? c : 0));
#else
	if (low)
		best = c - (31 - __builtin_clz(low));
	if (high && __builtin_ctz(high) - (c < 0 ? c : 0) < best)
		best = __builtin_ctz(high) - (c < 0 ? c : 0);
#endif
	return best;
}

// Chebyshev distance from (x, y) to the frame's nearest donor (0: it has none),
// by the whole warp: the bit words of boxes of radius 16, 32, 64, ... until one
// holds a donor within its radius, (2 R + 1)^2 / 32 words for the last.  Bound by
// the warp's chain of loads.  Counting every window of a growing radius cell by
// cell reads 4/3 R^3 cells: the replacement of one target 100 pixels from its
// donors took 6.4 ms, 300 pixels 129 ms, 1000 pixels seconds; with the words and
// the rim alone (far_window_median) 0.27, 2.2 and 6.7 ms.
__device__ __noinline__ int nearest_donor(const FrameDesc &fd, const uint32_t *don, const uint32_t *crm,
	int x, int y)
{
	const int lane = threadIdx.x & 31, limit = max(fd.w, fd.h);
	for (int R = 16;; R *= 2) {
		const int ya = max(0, y - R), yb = min(fd.h - 1, y + R);
		const int k0 = max(0, x - R) >> 5, nk = (min(fd.w - 1, x + R) >> 5) - k0 + 1, n = (yb - ya + 1) * nk;
		unsigned best = 0xffffffffu;
#pragma unroll 4
		for (int i = lane; i < n; i += 32) {
			const int row = i / nk, k = k0 + i - row * nk;
			const long long o = (long long)(ya + row) * fd.words + k;
			const uint32_t b = don[o] & ~crm[o];
			if (b)
				best = min(best, (unsigned)max(abs(ya + row - y), bit_distance(b, x - 32 * k)));
		}
		best = __reduce_min_sync(0xffffffffu, best);
		if (best <= (unsigned)R)
			return (int)best;
		if (R >= limit)
			return 0;
	}
}

// The donor of rank `rank` in key order among a ring's cells: an MSB-first radix
// select over ordered 64-bit keys (same ranks as reference
// src/replace.cuh:85-109).
__device__ double ring_rank(const FrameDesc &fd, const uint32_t *don, const uint32_t *crm, const Ring &q,
	int rank)
{
	const int lane = threadIdx.x & 31;
	unsigned long long prefix = 0, used = 0;
	for (int bit = 63; bit >= 0; --bit) {
		const unsigned long long flag = 1ull << bit;
		int below = 0;
		for (int pos = lane; pos < q.n; pos += 32) {
			int x, y;
			ring_cell(q, pos, x, y);
			if (!donor_at(don, crm, fd.words, x, y))
				continue;
			const unsigned long long k = order_key(fd.clean[(long long)y * fd.w + x]);
			below += (k & used) == prefix && !(k & flag);
		}
		below = warp_sum_int(below);
		used |= flag;
		if (rank >= below) {
			prefix |= flag;
			rank -= below;
		}
	}
	return order_value(prefix);
}

// The warp's 32 S keys in ascending unsigned order, by a bitonic network:
// element i = 32 s + lane in slot s of the lane.
template <int S>
__device__ __forceinline__ void sort_keys(unsigned long long (&k)[S])
{
	const int lane = threadIdx.x & 31;
	// Ascending where bit `size` of i is clear.
#pragma unroll
	for (int size = 2; size <= 32 * S; size <<= 1) {
#pragma unroll
		for (int j = size >> 1; j > 0; j >>= 1) {
			if (j >= 32) { // partner in the same lane, slot s ^ (j / 32)
#pragma unroll
				for (int s = 0; s < S; ++s) {
					const int t = s ^ (j >> 5);
					if (t < s)
						continue;
					const bool asc = ((32 * s + lane) & size) == 0;
					const unsigned long long a = k[s], b = k[t];
					const bool swap = asc ? b < a : a < b;
					k[s] = swap ? b : a;
					k[t] = swap ? a : b;
				}
			} else { // partner lane ^ j, same slot
#pragma unroll
				for (int s = 0; s < S; ++s) {
					const unsigned long long p = __shfl_xor_sync(0xffffffffu, k[s], j);
					const bool keep_min = ((lane & j) == 0) == (((32 * s + lane) & size) == 0);
					k[s] = keep_min ? (p < k[s] ? p : k[s]) : (k[s] < p ? p : k[s]);
				}
			}
		}
	}
}

// The donors of up to 32 S cells (cell(pos, x, y) for pos < n) in key order, for
// the median: lane l holds the keys of cells l + 32 s (all ones for a non-donor or
// past the last cell, which sort last), a bitonic network sorts the warp's 32 S
// keys in unsigned order (the order ring_rank's radix select ranks by),
// and the keys of ranks (nd - 1) / 2 and nd / 2 come back as lo and hi.  About 20
// to 30 dependent exchange steps instead of a radix select's 64 warp reductions per
// rank, so a replacement whose window grew past 5 x 5 no longer holds its
// launch for tens of microseconds.
struct DonorMedian {
	double lo, hi; // the two central donors (unset without a donor)
	int nd, r;     // donors; radius of the window
};

template <int S, class Cell>
__device__ __forceinline__ DonorMedian sorted_median(const FrameDesc &fd, const uint32_t *don,
	const uint32_t *crm, int n, Cell cell)
{
	const int lane = threadIdx.x & 31;
	unsigned long long k[S];
	int nd = 0;
#pragma unroll
	for (int s = 0; s < S; ++s) {
		const int pos = lane + 32 * s;
		k[s] = ~0ull;
		if (pos < n) {
			int x, y;
			cell(pos, x, y);
			if (donor_at(don, crm, fd.words, x, y))
				k[s] = order_key(fd.clean[(long long)y * fd.w + x]);
		}
		nd += __popc(__ballot_sync(0xffffffffu, k[s] != ~0ull));
	}
	if (!nd)
		return DonorMedian{0, 0, 0, 0};
	sort_keys(k);
	const int rl = (nd - 1) / 2, rh = nd / 2;
	unsigned long long vl = 0, vh = 0;
#pragma unroll
	for (int s = 0; s < S; ++s) { // register slots chosen by unrolled tests, not indexed
		if (s == rl >> 5)
			vl = k[s];
		if (s == rh >> 5)
			vh = k[s];
	}
	return DonorMedian{order_value(__shfl_sync(0xffffffffu, vl, rl & 31)),
		order_value(__shfl_sync(0xffffffffu, vh, rh & 31)), nd, 0};
}

// A window of 33 .. 32 S cells (r is left zero).
template <int S>
__device__ __noinline__ DonorMedian sorted_window_median(const FrameDesc &fd, const uint32_t *don,
	const uint32_t *crm, Window win)
{
	const int ww = win.x1 - win.x0 + 1, area = ww * (win.y1 - win.y0 + 1);
	return sorted_median<S>(fd, don, crm, area, [&](int pos, int &x, int &y) {
		x = win.x0 + pos % ww;
		y = win.y0 + pos / ww;
	});
}

// The smallest window around (x, y) that holds a donor, for a pixel whose windows
// of up to 128 cells hold none (r = 0: the frame has no donor).  No smaller window
// holds a donor, so all of them lie on the window's rim: only its cells are read.
__device__ __noinline__ DonorMedian far_window_median(const FrameDesc &fd, const uint32_t *don,
	const uint32_t *crm, int x, int y)
{
	DonorMedian m{0, 0, 0, 0};
	const int r = nearest_donor(fd, don, crm, x, y);
	if (!r)
		return m;
	const Ring q = ring_cells(fd.w, fd.h, x, y, r);
	if (q.n <= 128) {
		m = sorted_median<4>(fd, don, crm, q.n, [&](int pos, int &cx, int &cy) { ring_cell(q, pos, cx, cy); });
	} else {
		int cnt = 0;
		for (int pos = threadIdx.x & 31; pos < q.n; pos += 32) {
			int cx, cy;
			ring_cell(q, pos, cx, cy);
			cnt += donor_at(don, crm, fd.words, cx, cy);
		}
		m.nd = warp_sum_int(cnt);
		m.lo = ring_rank(fd, don, crm, q, (m.nd - 1) / 2);
		m.hi = m.nd % 2 ? m.lo : ring_rank(fd, don, crm, q, m.nd / 2);
	}
	m.r = r;
	return m;
}

// Reference src/replace.cuh:111-153 for one pixel, by the whole warp: the
// median of the donors in the clipped (2r+1)^2 window, r = 2, 3, ... until a
// donor exists; lane 0 writes it.  Returns r (0: the frame has no donor).
__device__ __forceinline__ int replace_one(const FrameDesc &fd, int x, int y, bool *changed = nullptr)
{
	const int lane = threadIdx.x & 31;
	const int w = fd.w, h = fd.h, words = fd.words;
	const uint32_t *don = plane_ptr(fd, P_DONOR), *crm = plane_ptr(fd, P_CRMASK);
	const int limit = max(w, h);
	for (int r = 2; r <= limit; ++r) {
		Window win = {max(0, x - r), min(w - 1, x + r), max(0, y - r), min(h - 1, y + r)};
		const int ww = win.x1 - win.x0 + 1, area = ww * (win.y1 - win.y0 + 1);
		double lo, hi;
		int nd;
		if (area <= 32) {
			bool d = false;
			double v = INFINITY;
			if (lane < area) {
				// The value loads with the donor bits and is dropped for a
				// non-donor (whose pixel another warp may be writing).
				int cx = win.x0 + lane % ww, cy = win.y0 + lane / ww;
				const double c = fd.clean[(long long)cy * w + cx];
				d = donor_at(don, crm, words, cx, cy);
				if (d)
					v = c;
			}
			nd = __popc(__ballot_sync(0xffffffffu, d));
			if (!nd)
				continue;
			v = bitonic32(v);
			lo = __shfl_sync(0xffffffffu, v, (nd - 1) / 2);
			hi = __shfl_sync(0xffffffffu, v, nd / 2);
		} else if (area <= 64) {
			const DonorMedian m = sorted_window_median<2>(fd, don, crm, win);
			if (!m.nd)
				continue;
			nd = m.nd, lo = m.lo, hi = m.hi;
		} else if (area <= 128) {
			const DonorMedian m = sorted_window_median<4>(fd, don, crm, win);
			if (!m.nd)
				continue;
			nd = m.nd, lo = m.lo, hi = m.hi;
		} else {
			const DonorMedian m = far_window_median(fd, don, crm, x, y);
			if (!m.r)
				return 0;
			r = m.r, nd = m.nd, lo = m.lo, hi = m.hi;
		}
		if (lane == 0) {
			const double v = nd % 2 ? 0.0 + lo : midpoint(lo, hi);
			double &dst = fd.clean[(long long)y * w + x];
			if (changed)
				*changed = __double_as_longlong(dst) != __double_as_longlong(v);
			dst = v;
			// Keep the block's floor a lower bound of its clean values.
			if (fd.floors && !fd.error)
				atomicMin(&fd.floors[(y >> 5) * ((w + 31) >> 5) + (x >> 5)].key, order_key(v));
		}
		return r;
	}
	return 0;
}

// Largest window radius whose FRESH neighbourhood replace_kernel inspects.
constexpr int KEEP_RADIUS_MAX = 15;

// Any FRESH pixel in the (2r + 1)^2 window of (x, y) clipped to the frame
// (r <= KEEP_RADIUS_MAX: a window row spans at most two bit words).
__device__ __forceinline__ bool fresh_in_window(const FrameDesc &fd, int x, int y, int r)
{
	const uint32_t *fr = plane_ptr(fd, P_FRESH);
	const int x0 = max(0, x - r), x1 = min(fd.w - 1, x + r);
	const int k0 = x0 >> 5, k1 = x1 >> 5;
	const unsigned long long span = ((1ull << (x1 - x0 + 1)) - 1ull) << (x0 & 31);
	const int ya = max(0, y - r), yb = min(fd.h - 1, y + r);
	const uint32_t *c0 = fr + (long long)ya * fd.words + k0;
	const int dk = k1 - k0; // 0 or 1
	unsigned long long any = 0;
#pragma unroll 4
	for (int i = 0; i <= yb - ya; ++i) { // independent loads, no early exit
		const uint32_t *c = c0 + (long long)i * fd.words;
		any |= (c[0] | (unsigned long long)c[dk] << 32) & span;
	}
	return any != 0;
}

// Bits of columns x - 2 .. x + 2 of row y of a bit plane (bit i: column
// x - 2 + i; columns outside the frame read as zero: the words' padding bits
// are zero, and words before the row's first or after its last read as zero).
// The second word is read only where the five columns reach into it.
__device__ __forceinline__ uint32_t bits5(const uint32_t *plane, int words, int x, int y)
{
	const int a = x - 2, k = a >> 5, s = a & 31; // k >= -1
	const uint32_t *row = plane + (long long)y * words;
	const uint32_t lo = k >= 0 ? row[k] : 0u, hi = s > 27 && k + 1 < words ? row[k + 1] : 0u;
	return __funnelshift_r(lo, hi, s) & 0x1fu;
}

// replace_one's first window (radius 2, clipped to the frame: at most 25
// cells) evaluated by one thread: the donor bits of its five rows, the
// donors' values, a sorting network over the 25 cells (non-donors as +inf)
// and the same median (rank (nd - 1) / 2, or the midpoint of ranks
// (nd - 1) / 2 and nd / 2).  Equal nonzero donors are the same bits, and an
// odd count's 0.0 + lo drops a zero's sign, so any sort gives the bits of
// replace_one's exchange network except when an even count's two middle
// values are zeros and the window holds zeros of both signs.  Returns false
// for that window and for one without a donor: the caller's warp then runs
// replace_one (the exchange network, expanding windows).
__device__ __forceinline__ bool first_window_value(const FrameDesc &fd, int x, int y, double &out)
{
	const int w = fd.w, h = fd.h, words = fd.words;
	const uint32_t *don = plane_ptr(fd, P_DONOR), *crm = plane_ptr(fd, P_CRMASK);
	uint32_t rb[5];
	int nd = 0;
#pragma unroll
	for (int dy = 0; dy < 5; ++dy) {
		const int yy = y - 2 + dy;
		rb[dy] = yy >= 0 && yy < h ? bits5(don, words, x, yy) & ~bits5(crm, words, x, yy) : 0u;
		nd += __popc(rb[dy]);
	}
	if (nd == 0)
		return false;
	double v[25];
	bool pz = false, nz = false; // donors of +0 and of -0
#pragma unroll
	for (int c = 0; c < 25; ++c) {
		const int dy = c / 5, dx = c % 5;
		v[c] = INFINITY;
		if ((rb[dy] >> dx) & 1u) {
			v[c] = fd.clean[(long long)(y - 2 + dy) * w + (x - 2 + dx)];
			pz |= v[c] == 0 && !signbit(v[c]);
			nz |= v[c] == 0 && signbit(v[c]);
		}
	}
	sort_network(v);
	const int k1 = (nd - 1) / 2, k2 = nd / 2;
	double lo = 0, hi = 0;
#pragma unroll
	for (int c = 0; c < 25; ++c) {
		lo = c == k1 ? v[c] : lo;
		hi = c == k2 ? v[c] : hi;
	}
	if (!(nd % 2) && lo == 0 && hi == 0 && pz && nz)
		return false;
	out = nd % 2 ? 0.0 + lo : midpoint(lo, hi);
	return true;
}

// Items the thread path of a block leaves, replaced by all of its warps.
struct WindowQueue {
	long long e[256];
	int n;
};

// Whether the replacement after a pass of parity par runs for a frame: the
// pass flagged a pixel and a donor is left (reference src/cleaner.cuh:128-142).
__device__ __forceinline__ bool replaces(const FrameState &s, int par)
{
	return s.todo[par] && s.donors > s.masked;
}

// Per-frame loop control after a pass (reference src/cleaner.cuh:128-142,
// 175-181): a frame with new pixels but no donors fails, a frame without new
// pixels stops (its later passes would repeat this one), the others replace
// and continue.  Runs in the replacement's grid (a thread per frame): the
// replacement reads only todo[par] and the donor counts, which this leaves alone.
__device__ __forceinline__ void pass_control(FrameState *state, int nf, Control *ctl, int par, Team team)
{
	const int fault = *(volatile int *)&ctl->fault;
	for (int f = team.block * blockDim.x + threadIdx.x; f < nf; f += team.blocks * blockDim.x) {
		FrameState &s = state[f];
		s.todo[par ^ 1] = 0;
		if (!s.active)
			continue;
		++s.passes;
		bool on = false;
		if (fault) // this pass's detection is incomplete: stop, report
			s.fault = fault;
		else if (s.todo[par] && s.donors <= s.masked)
			s.error = 1;
		else
			on = s.todo[par] != 0;
		s.active = on;
		if (on)
			ctl->any[par] = 1;
	}
}

// Replacement after a pass of parity par (src/replace.cuh:111-153), for the
// frames whose pass flagged new pixels.  A thread per target evaluates its
// first window (first_window_value); the targets it leaves (windows inside a
// cluster of flagged pixels) are queued in shared memory and the block's warps
// replace them with replace_one, spread over all eight warps so that a cluster
// does not hold one warp for many targets.  Targets are in the mask, so never
// donors: no target reads another's value.
//
// With chg, the indices of the targets whose value changed (bit for bit) are
// appended there (count in n_chg): the next pass starts from those pixels.
__device__ __forceinline__ void replace_targets(const FrameDesc *__restrict__ frames,
	const FrameState *state, int par, const uint2 *list, long long n, uint8_t *radius, unsigned *chg,
	unsigned long long *n_chg, WindowQueue &Q)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
	const long long stride = (long long)gridDim.x * blockDim.x;
	__syncthreads();
	if (threadIdx.x == 0)
		Q.n = 0;
	__syncthreads();
	for (long long base = blockIdx.x * (long long)blockDim.x; base < n; base += stride) { // block-uniform
		const long long e = base + threadIdx.x;
		bool changed = false;
		if (e < n) {
			const uint2 t = list[e];
			if (replaces(state[t.x], par)) {
				const FrameDesc &fd = frames[t.x];
				const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
				double v;
				if (first_window_value(fd, x, y, v)) {
					double &dst = fd.clean[(long long)y * fd.w + x];
					changed = __double_as_longlong(dst) != __double_as_longlong(v);
					dst = v;
					if (radius)
						radius[e] = 2;
					// Keep the block's floor a lower bound of its clean values.
					if (fd.floors && !fd.error)
						atomicMin(&fd.floors[(y >> 5) * ((fd.w + 31) >> 5) + (x >> 5)].key, order_key(v));
				} else {
					Q.e[atomicAdd(&Q.n, 1)] = e;
				}
			}
		}
		if (chg) {
			const unsigned b = __ballot_sync(0xffffffffu, changed);
			unsigned long long at = 0;
			if (lane == 0 && b)
				at = atomicAdd(n_chg, (unsigned long long)__popc(b));
			at = __shfl_sync(0xffffffffu, at, 0);
			if (changed)
				chg[at + __popc(b & ((1u << lane) - 1u))] = (unsigned)e;
		}
		__syncthreads();
		const int nq = Q.n;
		for (int q = warp; q < nq; q += nwarps) {
			const long long eq = Q.e[q];
			const uint2 t = list[eq];
			const FrameDesc &fd = frames[t.x];
			bool ch = false;
			const int r = replace_one(fd, (int)(t.y % (unsigned)fd.w), (int)(t.y / (unsigned)fd.w), &ch);
			if (lane == 0) {
				if (radius)
					radius[eq] = (uint8_t)(r < 255 ? r : 255);
				if (chg && ch)
					chg[atomicAdd(n_chg, 1ull)] = (unsigned)eq;
			}
		}
		__syncthreads();
		if (threadIdx.x == 0)
			Q.n = 0;
		__syncthreads();
	}
}

// The replacement after a full pass of parity par (every target of the frames
// that flagged pixels), with the pass's loop control in the same grid.
// Without chg (no late passes follow) the next full pass's lists are reset.
__global__ void __launch_bounds__(256, 3)
replace_kernel(const FrameDesc *__restrict__ frames, FrameState *state, int nf, const uint2 *list,
	Control *ctl, int par, uint8_t *radius, unsigned *chg)
{
	__shared__ WindowQueue Q;
	pass_control(state, nf, ctl, par, whole_grid());
	if (!chg && blockIdx.x == 0 && threadIdx.x == 0) {
		ctl->pass[par ^ 1] = PassLists{};
		ctl->any[par ^ 1] = 0;
	}
	replace_targets(frames, state, par, list, (long long)ctl->n_targets, radius, chg,
		&ctl->pass[par ^ 1].n_chg, Q);
}

// Initial fill of non-finite pixels (src/cleaner.cuh:78-100) for frames with
// a finite donor, from the hole list prepare wrote (holes are never donors, so
// the order does not matter): a thread per hole (first_window_value), the
// block's warps for the holes it leaves (replace_kernel's queue).
__global__ void __launch_bounds__(256)
fill_list_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const uint2 *__restrict__ holes, const unsigned long long *count)
{
	__shared__ WindowQueue Q;
	const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
	const long long n = (long long)*count;
	const long long stride = (long long)gridDim.x * blockDim.x;
	if (threadIdx.x == 0)
		Q.n = 0;
	__syncthreads();
	for (long long base = blockIdx.x * (long long)blockDim.x; base < n; base += stride) { // block-uniform
		const long long e = base + threadIdx.x;
		if (e < n) {
			const uint2 t = holes[e];
			if (state[t.x].donors) {
				const FrameDesc &fd = frames[t.x];
				const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
				double r;
				if (first_window_value(fd, x, y, r)) {
					fd.clean[(long long)y * fd.w + x] = r;
					// Keep the block's floor a lower bound of its clean values.
					if (fd.floors && !fd.error)
						atomicMin(&fd.floors[(y >> 5) * ((fd.w + 31) >> 5) + (x >> 5)].key, order_key(r));
				} else {
					Q.e[atomicAdd(&Q.n, 1)] = e;
				}
			}
		}
		__syncthreads();
		const int nq = Q.n;
		for (int q = warp; q < nq; q += nwarps) {
			const uint2 t = holes[Q.e[q]];
			const FrameDesc &fd = frames[t.x];
			replace_one(fd, (int)(t.y % (unsigned)fd.w), (int)(t.y / (unsigned)fd.w));
		}
		__syncthreads();
		if (threadIdx.x == 0)
			Q.n = 0;
		__syncthreads();
	}
}

// The same fill without a hole list: one warp per row scans the row's HOLE
// words.
__global__ void __launch_bounds__(256)
fill_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const int2 *__restrict__ rows, int nrows)
{
	const int lane = threadIdx.x & 31;
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	for (int ri = gw; ri < nrows; ri += nw) {
		const int2 item = rows[ri];
		const FrameState &st = state[item.x];
		if (!st.holes || !st.donors)
			continue; // warp-uniform
		const FrameDesc &fd = frames[item.x];
		const uint32_t *hp = plane_ptr(fd, P_HOLE) + (long long)item.y * fd.words;
		for (int k0 = 0; k0 < fd.words; k0 += 32) {
			const uint32_t hw = k0 + lane < fd.words ? hp[k0 + lane] : 0u;
			for (unsigned m = __ballot_sync(0xffffffffu, hw != 0); m; m &= m - 1) {
				const int j = __ffs(m) - 1;
				for (uint32_t bits = __shfl_sync(0xffffffffu, hw, j); bits; bits &= bits - 1)
					replace_one(fd, 32 * (k0 + j) + __ffs(bits) - 1, item.y);
			}
		}
	}
}

// The end of a call (reference src/image.cuh:50-70).  prepare wrote every
// output pixel but the flagged ones, and the masks start zero, so what is left
// is sparse: the flagged pixels' mask bytes and, for a frame with a background
// (whose working pixels are a buffer of their own), their values, from the
// target list; and the non-finite inputs of the frames whose working pixels are
// the output, bit for bit, from the HOLE words (a warp per row).  Writing every
// mask byte from the CRMASK words took 24 us on 16 frames of 2048 x 2048 and
// 108 us on 64 ragged frames, whose rows are not aligned; zeroing the masks in
// the first launch and this take 6 + 14 and 31 + 26 us.
__global__ void __launch_bounds__(256)
finish_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const int2 *__restrict__ rows, int nrows, const uint2 *__restrict__ targets,
	const Control *__restrict__ ctl)
{
	const long long n = (long long)ctl->n_targets, stride = (long long)gridDim.x * blockDim.x;
	for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += stride) {
		const uint2 t = targets[e];
		const FrameDesc &fd = frames[t.x];
		fd.mask_out[t.y] = 1;
		if (fd.out != fd.clean)
			fd.out[t.y] = fd.clean[t.y] + -1 * (fd.bg_map ? fd.bg_map[t.y] : fd.bg);
	}
	const int lane = threadIdx.x & 31;
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	for (int r = gw; r < nrows; r += nw) {
		const int2 item = rows[r];
		const FrameDesc &fd = frames[item.x];
		if (!state[item.x].holes || fd.out != fd.clean)
			continue; // warp-uniform
		const uint32_t *hole = plane_ptr(fd, P_HOLE) + (long long)item.y * fd.words;
		const long long rowpix = (long long)item.y * fd.w;
		for (int k = lane; k < fd.words; k += 32)
			for (uint32_t hb = hole[k]; hb; hb &= hb - 1) {
				const long long i = rowpix + 32 * k + __ffs(hb) - 1;
				fd.clean[i] = fd.data[i];
			}
	}
}

// The same for a call without the zeroed masks and the separate output
// buffers (the allocation-free entry point): clean -= bg in place, non-finite
// inputs restored, every mask byte from the bit plane.
__global__ void __launch_bounds__(256)
restore_kernel(const FrameDesc *__restrict__ frames, const int2 *__restrict__ rows, int nrows)
{
	const int lane = threadIdx.x & 31;
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	for (int r = gw; r < nrows; r += nw) {
		const int2 item = rows[r];
		const FrameDesc &fd = frames[item.x];
		// Descriptor fields in registers (the stores below could alias it).
		const int w = fd.w, y = item.y, words = fd.words;
		const uint32_t *hole = plane_ptr(fd, P_HOLE) + (long long)y * words;
		const uint32_t *crm = plane_ptr(fd, P_CRMASK) + (long long)y * words;
		const long long rowpix = (long long)y * w;
		double *clean = fd.clean + rowpix;
		const double *data = fd.data + rowpix, *bgmap = fd.bg_map ? fd.bg_map + rowpix : nullptr;
		uint8_t *mask_out = fd.mask_out + rowpix;
		const double bgv = fd.bg;
		const bool has_bg = fd.has_bg;
		constexpr int ROW_UNROLL = 4; // words whose loads are issued before their use
		for (int xb = 0; xb < w; xb += 32 * ROW_UNROLL) {
			double v[ROW_UNROLL], bg[ROW_UNROLL];
			uint32_t hb[ROW_UNROLL], cb[ROW_UNROLL];
#pragma unroll
			for (int u = 0; u < ROW_UNROLL; ++u) {
				const int x = xb + 32 * u + lane;
				v[u] = 0;
				bg[u] = bgv;
				hb[u] = cb[u] = 0;
				if (x < w) {
					v[u] = clean[x];
					hb[u] = hole[x >> 5];
					cb[u] = crm[x >> 5];
					if (bgmap)
						bg[u] = bgmap[x];
				}
			}
#pragma unroll
			for (int u = 0; u < ROW_UNROLL; ++u) {
				const int x = xb + 32 * u + lane;
				if (x < w) {
					double o = v[u];
					if (has_bg)
						o += -1 * bg[u];
					if ((hb[u] >> (x & 31)) & 1u)
						o = data[x];
					clean[x] = o;
					mask_out[x] = (cb[u] >> (x & 31)) & 1u;
				}
			}
		}
	}
}

// maxiter == 0 (reference src/image.cuh:72-92): background round trip only.
__global__ void __launch_bounds__(256)
copy_kernel(const FrameDesc *__restrict__ frames, const int2 *__restrict__ rows, int nrows)
{
	const int lane = threadIdx.x & 31;
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	for (int r = gw; r < nrows; r += nw) {
		const int2 item = rows[r];
		const FrameDesc &fd = frames[item.x];
		const long long rowpix = (long long)item.y * fd.w;
		for (int x = lane; x < fd.w; x += 32) {
			const long long i = rowpix + x;
			const double d = fd.data[i];
			double v = isfinite(d) ? d : 0;
			if (fd.has_bg) {
				double bg = fd.bg_map ? fd.bg_map[i] : fd.bg;
				v += 1 * bg;
				v += -1 * bg;
			}
			fd.clean[i] = isfinite(d) ? v : d;
			fd.mask_out[i] = 0;
		}
	}
}

// Up to four copies of 8-byte words between any memory the device can
// address, page-locked host memory included (read or written over the bus by
// the kernel itself, so no copy engine is involved).
struct WordCopy {
	const unsigned long long *src;
	unsigned long long *dst;
	long long n8;
};

struct WordCopies {
	WordCopy part[6];
	int n;
};

__global__ void __launch_bounds__(256)
word_copy_kernel(WordCopies c)
{
	const long long stride = (long long)gridDim.x * blockDim.x;
	for (int k = 0; k < c.n; ++k)
		for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < c.part[k].n8; i += stride)
			c.part[k].dst[i] = c.part[k].src[i];
}

// The cleaned values of the listed targets (the cumulative mask as
// {frame, pixel}): vals[i] = clean of target i.  Without a background every
// other output pixel equals its input bit for bit, so these values and the
// list are all of a frame's result that differs from its input.
__global__ void __launch_bounds__(256)
gather_targets_kernel(const FrameDesc *__restrict__ frames, const uint2 *__restrict__ list,
	const unsigned long long *count, double *vals)
{
	const unsigned long long n = *count, stride = (unsigned long long)gridDim.x * blockDim.x;
	for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
	     i += stride) {
		const uint2 t = list[i];
		vals[i] = frames[t.x].clean[t.y];
	}
}

} // namespace cb
