// Shared definitions of the cusmic_b200 kernels: border mapping, frame
// descriptors, per-frame state, bit-plane layout and small device helpers.
//
// HBM layout of one call (all per frame, frames back to back):
//   clean      float64 [h][w]      working pixels; the caller's output buffer
//   bit planes uint32  [N_PLANES][frames][h][words], words = ceil(w / 32); bit b of
//              word (y, k) is pixel (y, 32 k + b); padding bits are zero
//   targets    uint2   {frame, pixel} list of replacement targets
#pragma once
#include <cstddef>
#include <cstdint>
#include <cmath>
#include <cuda_runtime.h>

#if defined(__CUDACC__)
#define CB_HD __host__ __device__ __forceinline__
#else
#define CB_HD inline
#endif

namespace cb {

using std::fabs;
using std::fmax;
using std::fmin;
using std::isfinite;
using std::isnan;
using std::sqrt;

enum Border { REFLECT = 0, CONSTANT = 1, NEAREST = 2, MIRROR = 3, WRAP = 4 };

// Bit planes of a frame.
enum Plane {
	P_HOLE,   // non-finite input pixel
	P_EXCL,   // excluded from seeds and donors: hole or masked
	P_DONOR,  // static donor: not excluded and finite after background
	P_CRMASK, // cumulative cosmic-ray mask
	P_HIGH,   // holds every pixel with sig_raw > cr_threshold (or NaN) on the
	          // current clean pixels (a superset after the first pass)
	P_LOW,    // with HIGH, holds every pixel with sig_raw > neighbor_threshold
	P_S1,     // significance > cr_threshold
	P_S2,     // significance > neighbor_threshold
	P_CAND,   // seed: S1, not excluded, contrast test passed
	P_FRESH,  // pixels that the last late pass added to the mask
	P_EVAL,   // late passes: pixels claimed for re-evaluation (zero between passes)
	P_LISTED, // late passes: pixels claimed for the work lists (zero between passes)
	P_ROWMIN, // noise-model frames: per row and bit word, the smallest high word of
	          // the ordered keys of its finite input pixels (all ones: none)
	N_PLANES
};

static_assert(P_S2 == P_S1 + 1 && P_CAND == P_S1 + 2,
	"S1, S2 and CAND are zeroed as one range (clear_detect_words)");

constexpr double FINE_FLOOR = 0.01;   // reference src/filters.cuh:21
constexpr double SIGNAL_FLOOR = 1e-5; // reference src/filters.cuh:22

// scipy.ndimage border conventions, reference src/filters.cuh:24-44: returns
// the in-range index a coordinate reads, or -1 for a constant (zero) pad.
CB_HD int border_index(int x, int n, int mode)
{
	if (x >= 0 && x < n)
		return x;
	if (mode == CONSTANT)
		return -1;
	if (mode == NEAREST)
		return x < 0 ? 0 : n - 1;
	if (n == 1)
		return 0;
	// One reflection or turn (the windows' offsets are a few pixels) without
	// the divisions of the general case.
	const int once = mode == REFLECT ? (x < 0 ? -x - 1 : 2 * n - 1 - x)
		: mode == MIRROR ? (x < 0 ? -x : 2 * (n - 1) - x) : (x < 0 ? x + n : x - n);
	if (once >= 0 && once < n)
		return once;
	int period = mode == REFLECT ? 2 * n : mode == MIRROR ? 2 * (n - 1) : n;
	x %= period;
	if (x < 0)
		x += period;
	if (mode == REFLECT && x >= n)
		return period - x - 1;
	if (mode == MIRROR && x >= n)
		return period - x;
	return x;
}

CB_HD int clampi(int x, int lo, int hi)
{
	return x < lo ? lo : x > hi ? hi : x;
}

// Noise floor of a 32 x 32 block of a frame (see bulk.cuh): the detection
// threshold of an error-map block, or for a noise-model block lower bounds
// kept as ordered keys (a smaller key is a smaller value): of its clean values
// (lowered by every replacement inside the block), of -gain and of the read
// noise over the block (gain and read-noise maps only).  All-ones keys: no
// value seen yet.
struct BlockFloor {
	double thr;
	unsigned long long key, gkey, rkey;
};

// One frame of a (possibly ragged) batch, as the kernels see it.
struct FrameDesc {
	const double *data, *error, *gain_map, *rn_map, *bg_map;
	const uint8_t *mask;
	double *clean;     // working pixels, restored in place into the output
	double *out;       // output pixels: clean itself (null means the same), or for a frame
	                   // with a background the caller's buffer while clean is a
	                   // workspace buffer: prepare then writes every output pixel
	                   // except the flagged ones, which restore writes
	uint8_t *mask_out; // uint8 output mask
	uint32_t *bits;    // N_PLANES planes of `plane` words
	BlockFloor *floors; // the frame's block floors, row-major by block (null: none)
	// Noise-model frames, first pass: sig_raw and the noise at every pixel
	// within two of a HIGH pixel (region_sig_kernel), which the high-list
	// candidates read instead of recomputing their windows (null: none).
	double *sig_raw, *noise;
	double gain, rn, bg;
	long long plane;   // words per plane of this frame = h * words
	long long pstride; // words from one plane to the next (planes of all frames of a
	                   // batch are interleaved plane by plane, so pstride >= plane)
	int w, h, words, has_bg;
};

// Device-side control state of a frame.  Passes are numbered from 0; what a
// pass appends or flags is kept by the pass's parity, so the next pass can
// start from it while its own is still empty.
struct FrameState {
	unsigned int active;  // the next detection pass runs for this frame
	unsigned int error;   // a target had no finite donor
	unsigned int passes;  // detection passes run
	unsigned int fault;   // a bounded wait inside a kernel ran out (the frame stopped): FaultBit
	unsigned int todo[2]; // by parity: the pass flagged a new pixel (set by many warps)
	unsigned int map_flags, pad; // frame 0: failed map checks of the call (check_maps_kernel)
	// Static donors, and those of them that are in the mask.
	unsigned long long donors, masked;
	// Nonzero if the frame has a hole; if it has an allowed pixel in a row
	// (or tile) without a donor.  Many warps set both, by additions whose
	// result nobody waits for: a test before the store waits behind the other
	// warps' additions to the sector, and plain stores to it are slower still
	// (prep_detect_kernel on one 2048 x 2048 frame: 52 us with tests, 95 with
	// stores alone, 32; on two of 8192 x 8192: 512, 755, 488).
	unsigned long long holes, allowed;
};

// Lengths of one pass's work lists.
struct PassLists {
	unsigned long long n_cand; // high list: pixels whose significance is evaluated
	unsigned long long n_low;  // low list: pixels whose sig_raw can only exceed neighbor
	unsigned long long n_eval; // late passes: pixels whose sig_raw is evaluated again
	unsigned long long n_chg;  // targets whose value the replacement before changed
};

// What ran out: a copy into the dense kernels' ring, or a grid barrier.
enum FaultBit { FAULT_COPY = 1, FAULT_BARRIER = 2 };

// Loop control shared by the per-pass kernels.
struct Control {
	unsigned long long n_targets; // length of the target list
	unsigned long long n_holes;   // length of the hole list prepare_kernel writes
	unsigned long long cand_cap;  // capacity of the candidate buffer (first pass: high from
	                              // the front, low from the back)
	PassLists pass[2];            // by parity
	unsigned long long n_region;  // first pass: pixels of the noise-model sig_raw map (listed)
	unsigned long long fresh0;    // late passes: targets listed before the last growth
	int any[2];                   // by parity: a frame goes on after the pass
	int ticket;                   // next item of the bulk detection kernel
	unsigned pad;
	// Read as one 16-byte word by grid_barrier:
	alignas(16) int fault;        // a bounded wait ran out (FaultBit)
	unsigned barrier;             // arrivals at the late passes' grid barriers
	unsigned arrived;             // blocks of the late passes that started (join_team)
	unsigned team;                // how many of them work, once that is closed
	// Injected failures (0: none): the bound, in SM cycles, of one extra wait
	// on a barrier that nothing completes, for prepare ([0]) and for the dense
	// detection ([1]); one warp of the dense detection's first block makes it.
	long long poison_wait[2];
};

static_assert(offsetof(Control, fault) % 16 == 0 && offsetof(Control, team) == offsetof(Control, fault) + 12,
	"grid_barrier reads the four as one word");

// The blocks that share a launch's work: this one's number and how many there are
// (all of the grid's, except in the late passes).
struct Team {
	unsigned block, blocks;
};

#ifdef __CUDACC__
__device__ __forceinline__ Team whole_grid()
{
	return Team{blockIdx.x, gridDim.x};
}
#endif

CB_HD uint32_t *plane_ptr(const FrameDesc &f, int p)
{
	return f.bits + (long long)p * f.pstride;
}

CB_HD bool test_bit(const uint32_t *plane, int words, int x, int y)
{
	return (plane[(long long)y * words + (x >> 5)] >> (x & 31)) & 1u;
}

#ifdef __CUDACC__
// Sets or clears bit `bit` of *word, for a caller that is the only writer of
// that bit (other bits of the word may change concurrently): an atomic only
// when the bit changes.  `fresh`: the plane was zeroed for this pass, so only
// a set needs an atomic and nothing is read.
__device__ __forceinline__ void write_bit(uint32_t *word, uint32_t bit, bool value, bool fresh = false)
{
	if (fresh) {
		if (value)
			atomicOr(word, bit);
		return;
	}
	const bool now = (*(volatile uint32_t *)word & bit) != 0;
	if (value && !now)
		atomicOr(word, bit);
	else if (!value && now)
		atomicAnd(word, ~bit);
}
#endif

} // namespace cb
