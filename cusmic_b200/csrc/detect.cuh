// Detection pass of one L.A.Cosmic iteration.
//
// Reference chain (src/cleaner.cuh:102-126): laplacian -> [median5 ->
// noise_model] -> snr -> median5 -> significance -> median3 -> median7 ->
// fine_structure -> detect, every stage a full-frame float64 pass with 25 to
// 49 gathers per pixel.  Two exact facts about that chain let this pass read
// each pixel once and evaluate medians only where a threshold can pass:
//
//  * the Laplacian is a sum of clipped terms, so lap >= 0 and sig_raw =
//    lap / (2 noise) >= 0; hence med5(sig_raw) >= 0 and sig = sig_raw -
//    med5(sig_raw) <= sig_raw.  A pixel whose sig_raw does not exceed
//    min(cr, neighbor) (both >= 0) can set neither `sig > cr` nor
//    `sig > neighbor`, so its 5 x 5 median is never needed (NaN compares
//    false either way);
//  * fine structure (med3 -> med7) is only read by detect behind
//    `sig > cr_threshold` on a non-excluded pixel (src/filters.cuh:164-175).
//
// So a pass has three steps:
//   A  dense: a division-free, median-free test that keeps a superset of the
//      pixels whose sig_raw exceeds min(cr, neighbor) in a candidate list.  The
//      kernels of bulk.cuh and prep_detect.cuh do that; those below
//      (sig_stream_kernel and sig_model_kernel, which also clear the S1/S2/CAND
//      words) serve the call without device allocation only: with an error map
//      each warp walks a strip of 32 columns down the frame with a rolling 3-row
//      register window, with the noise model a tile kernel bounds the noise from
//      below by the tile's minimum;
//   B  a candidate: exact sig_raw over the 5 x 5 window (with the exact noise model
//      where there is no error map), sig against both thresholds, the S1/S2 bits
//      and the candidate's seed slot;
//   C  a seed: the contrast test and the CAND bit, by counts over the 49 3 x 3
//      windows, or from their medians where those leave it open.
// Every value that feeds a threshold is computed in the reference's operation
// order (no FMA), so the bits equal the reference's.
//
// Borders: the chained filters read intermediates at border-mapped positions
// (med7 reads med3 at border_index(x), med5 reads sig_raw there).  B and C
// fold each window position with the median's border map before evaluating
// the intermediate, except that the medians of clean under mirror, reflect or
// wrap are taken directly on border-extended clean pixels: those border maps
// are invariant under a group of isometries that folds any coordinate onto
// its image, so both give the same multiset.  The Laplacian itself reads its
// neighbours with nearest semantics for mirror and reflect
// (src/filters.cuh:95-97).
#pragma once
#include "common.cuh"
#include "kernels.cuh"
#include "select.cuh"

namespace cb {

struct DetectParams {
	double contrast, cr, nb;
	double thi2;  // 2 cr (1 - 1e-12): division-free superset test for sig_raw > cr
	double tlo2;  // 2 nb (1 - 1e-12): the same for sig_raw > neighbor
	double rcontrast; // 1 / contrast
	int mode;
};

// Kernel A's two superset tests (see sig_stream_kernel): bit 0 = can exceed
// cr_threshold, bit 1 = can only exceed neighbor_threshold.
__device__ __forceinline__ uint32_t candidate_class(double lap, double nz, const DetectParams &p)
{
	if (lap > p.thi2 * nz)
		return 1u;
	return lap > p.tlo2 * nz ? 2u : 0u;
}

// Seed slot of candidate e (frame NO_SEED when the candidate is not a seed).
struct Seed {
	unsigned frame, pixel;
	double sig, noise;
};
constexpr unsigned NO_SEED = 0xffffffffu;

constexpr int STREAM_ROWS = 32; // rows per strip item of sig_stream_kernel
constexpr int MTILE = 32;       // square tile of sig_model_kernel
constexpr int MHALO = MTILE + 4;

__device__ __forceinline__ double positive(double v)
{
	return v < 0 ? 0 : v;
}

// Reference src/filters.cuh:98-104, same operation order.
__device__ __forceinline__ double lap_formula(double c0, double u0, double d0, double l0, double r0)
{
	double c = c0 / 4;
	double up = c - u0 / 4;
	double down = c - d0 / 4;
	double left = c - l0 / 4;
	double right = c - r0 / 4;
	return (positive(up + left) + positive(up + right)) + (positive(down + left) + positive(down + right));
}

__device__ __forceinline__ int lap_mode(int mode)
{
	return mode == MIRROR || mode == REFLECT ? NEAREST : mode;
}

// The same Laplacian from quarter values q = x / 4 (exact: a power-of-two
// scaling), so a streaming kernel can scale each pixel once.
__device__ __forceinline__ double lap_quarters(double qc, double qu, double qd, double ql, double qr)
{
	double up = qc - qu;
	double down = qc - qd;
	double left = qc - ql;
	double right = qc - qr;
	return (positive(up + left) + positive(up + right)) + (positive(down + left) + positive(down + right));
}

// clean at (x, y) under a border mode (0 outside for constant).
__device__ __forceinline__ double clean_at(const FrameDesc &fd, int x, int y, int mode)
{
	int mx = border_index(x, fd.w, mode), my = border_index(y, fd.h, mode);
	return mx < 0 || my < 0 ? 0.0 : fd.clean[(long long)my * fd.w + mx];
}

// The Laplacian at an in-frame pixel (reference src/filters.cuh:98-104).
__device__ __forceinline__ double lap_at(const FrameDesc &fd, int x, int y, int lm)
{
	return lap_formula(fd.clean[(long long)y * fd.w + x], clean_at(fd, x, y - 1, lm),
		clean_at(fd, x, y + 1, lm), clean_at(fd, x - 1, y, lm), clean_at(fd, x + 1, y, lm));
}

// Noise model at an in-frame pixel from its 5 x 5 median of clean
// (src/filters.cuh:107-123).
__device__ __forceinline__ double noise_from_median(const FrameDesc &fd, long long i, double m)
{
	double g = fd.gain_map ? fd.gain_map[i] : fd.gain;
	double rn = fd.rn_map ? fd.rn_map[i] : fd.rn;
	m = m < SIGNAL_FLOOR ? SIGNAL_FLOOR : m;
	return sqrt(rn * rn + g * m) / g;
}

__device__ __forceinline__ void clear_detect_words(const FrameDesc &fd, long long word, int lane)
{
	if (lane < 3)
		plane_ptr(fd, P_S1 + lane)[word] = 0u;
}

// Append the candidates of one strip item (lane = column, bit k of `rows` =
// row y0 + k) with a single atomic per item; the high list grows from the
// front of the buffer, the low list from its back.
__device__ __forceinline__ void stream_flush(int f, int w, int x, int y0, uint32_t hi, uint32_t lo,
	Control *ctl, int par, uint2 *cands)
{
	if (__any_sync(0xffffffffu, hi != 0)) {
		unsigned long long slot = warp_append(&ctl->pass[par].n_cand, __popc(hi));
		while (hi) {
			const int k = __ffs(hi) - 1;
			hi &= hi - 1;
			cands[slot++] = make_uint2((unsigned)f, (unsigned)((long long)(y0 + k) * w + x));
		}
	}
	if (__any_sync(0xffffffffu, lo != 0)) {
		unsigned long long slot = warp_append(&ctl->pass[par].n_low, __popc(lo));
		while (lo) {
			const int k = __ffs(lo) - 1;
			lo &= lo - 1;
			cands[ctl->cand_cap - 1 - slot++] =
				make_uint2((unsigned)f, (unsigned)((long long)(y0 + k) * w + x));
		}
	}
}

// A, error-map frames: one warp per item {frame, x0, y0}: 32 columns from x0,
// rows y0 .. y0 + STREAM_ROWS - 1.  Each warp streams its rows through a
// shared-memory ring filled with cp.async, SR_LEAD rows ahead of the row it
// evaluates, so many row loads are in flight per warp without holding
// registers.  A ring row holds the row's 32 columns plus one halo column on
// each side, each cell already border-mapped with the Laplacian's border mode
// (zero outside for constant), so the evaluation has no border cases.
//
// The kernel only has to find supersets of {sig_raw > cr} and {sig_raw >
// neighbor}: B evaluates sig_raw exactly for every candidate and drops the
// others.  So instead of dividing it tests lap > (2 t (1 - 1e-12)) noise: the
// product is rounded by at most 2^-53 relative and 2 t scales exactly, so
// every pixel with fl(lap / (2 noise)) > t passes (NaN, infinite or zero noise
// give the same outcome as the division, or a larger superset).
constexpr int SR_DEPTH = 8; // ring rows per warp (power of two)
constexpr int SR_LEAD = 5;  // rows issued ahead of the row being evaluated

struct StreamRing {
	double c[SR_DEPTH][34]; // clean, columns x0 - 1 .. x0 + 32
	double e[SR_DEPTH][32]; // error map, columns x0 .. x0 + 31
	uint32_t hole[SR_DEPTH];
};

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem)
{
	unsigned s = (unsigned)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
	unsigned s = (unsigned)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void cp_async_commit()
{
	asm volatile("cp.async.commit_group;\n" ::);
}

template <int N> __device__ __forceinline__ void cp_async_wait()
{
	asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Every lane issues its cells of ring row r (one commit group per row, empty
// past the last needed row so group counting stays uniform).
__device__ __forceinline__ void stream_issue(StreamRing &R, const FrameDesc &fd, int r, int r_end,
	int y0, int y1, int x0, int lane, int lm, int mx, int mx_halo, int xc)
{
	if (r <= r_end) {
		const int slot = r & (SR_DEPTH - 1);
		const int my = border_index(r, fd.h, lm);
		const double *row = fd.clean + (long long)(my < 0 ? 0 : my) * fd.w;
		if (my >= 0 && mx >= 0)
			cp_async8(&R.c[slot][1 + lane], row + mx);
		else
			R.c[slot][1 + lane] = 0.0;
		if (lane == 0 || lane == 31) {
			const int hi = lane == 0 ? 0 : 33;
			if (my >= 0 && mx_halo >= 0)
				cp_async8(&R.c[slot][hi], row + mx_halo);
			else
				R.c[slot][hi] = 0.0;
		}
		if (r >= y0 && r < y1) {
			cp_async8(&R.e[slot][lane], fd.error + (long long)r * fd.w + xc);
			if (lane == 0)
				cp_async4(&R.hole[slot], plane_ptr(fd, P_HOLE) + (long long)r * fd.words + (x0 >> 5));
		}
	}
	cp_async_commit();
}

__global__ void __launch_bounds__(256)
sig_stream_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const int4 *__restrict__ items, int nitems, DetectParams prm, Control *ctl, int par, uint2 *cands)
{
	__shared__ StreamRing rings[8];
	const int lane = threadIdx.x & 31;
	StreamRing &R = rings[threadIdx.x >> 5];
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	const int lm = lap_mode(prm.mode);
	for (int it = gw; it < nitems; it += nw) {
		const int4 item = items[it];
		if (!state[item.x].active)
			continue; // warp-uniform
		const FrameDesc &fd = frames[item.x];
		const int w = fd.w, h = fd.h, words = fd.words;
		const int x0 = item.y, y0 = item.z, y1 = min(y0 + STREAM_ROWS, h);
		const int x = x0 + lane, xc = min(x, w - 1);
		const bool valid = x < w;
		const int mx = border_index(x, w, lm);
		const int mx_halo = border_index(lane == 0 ? x0 - 1 : x0 + 32, w, lm);
		const int r_end = y1; // the row below the last output row
		for (int r = y0 - 1; r < y0 - 1 + SR_LEAD + 1; ++r)
			stream_issue(R, fd, r, r_end, y0, y1, x0, lane, lm, mx, mx_halo, xc);
		uint32_t hi = 0, lo = 0; // bit k: row y0 + k of this lane's column is a candidate
		double qu = 0, qc = 0;   // quarter values of the rows above and at y
		for (int y = y0; y < y1; ++y) {
			// Groups issued: rows y0 - 1 .. y + SR_LEAD - 1; row y + 1 is done
			// once at most SR_LEAD - 2 newer groups are pending.
			cp_async_wait<SR_LEAD - 2>();
			__syncwarp();
			const int s = y & (SR_DEPTH - 1), sd = (y + 1) & (SR_DEPTH - 1);
			if (y == y0) {
				qu = R.c[(y - 1) & (SR_DEPTH - 1)][1 + lane] * 0.25;
				qc = R.c[s][1 + lane] * 0.25;
			}
			const double qd = R.c[sd][1 + lane] * 0.25;
			const double lap = lap_quarters(qc, qu, qd, R.c[s][lane] * 0.25, R.c[s][lane + 2] * 0.25);
			const uint32_t cls = valid && !((R.hole[s] >> lane) & 1u)
				? candidate_class(lap, R.e[s][lane], prm) : 0u;
			hi |= (cls & 1u) << (y - y0);
			lo |= (cls >> 1) << (y - y0);
			qu = qc;
			qc = qd;
			clear_detect_words(fd, (long long)y * words + (x0 >> 5), lane);
			__syncwarp();
			stream_issue(R, fd, y + SR_LEAD, r_end, y0, y1, x0, lane, lm, mx, mx_halo, xc);
		}
		cp_async_wait<0>();
		__syncwarp();
		stream_flush(item.x, w, x, y0, hi, lo, ctl, par, cands);
	}
}

__device__ __forceinline__ void tile_flush(int f, int w, int x, int ybase, uint32_t hi, uint32_t lo,
	Control *ctl, int par, uint2 *cands)
{
	if (__any_sync(0xffffffffu, hi != 0)) {
		unsigned long long slot = warp_append(&ctl->pass[par].n_cand, __popc(hi));
		while (hi) {
			const int j = __ffs(hi) - 1;
			hi &= hi - 1;
			cands[slot++] = make_uint2((unsigned)f, (unsigned)((long long)(ybase + 8 * j) * w + x));
		}
	}
	if (__any_sync(0xffffffffu, lo != 0)) {
		unsigned long long slot = warp_append(&ctl->pass[par].n_low, __popc(lo));
		while (lo) {
			const int j = __ffs(lo) - 1;
			lo &= lo - 1;
			cands[ctl->cand_cap - 1 - slot++] =
				make_uint2((unsigned)f, (unsigned)((long long)(ybase + 8 * j) * w + x));
		}
	}
}

// A, noise-model frames: one block per MTILE x MTILE tile with its clean
// pixels (halo 2, border-extended) in shared memory.  The noise model is
// monotone non-decreasing in the 5 x 5 median in floating point (max, g * m,
// rn^2 + ., sqrt and / g are each monotone for g > 0), and the median of a
// window is at least the minimum m_lo of the tile and its halo, so
// noise(m_lo) <= noise(med5) and lap / (2 noise(m_lo)) >= sig_raw.  The tile
// therefore applies the superset tests of sig_stream_kernel with noise(m_lo)
// in place of the noise, without any median.  Scalar gain and read
// noise make noise(m_lo) one value per tile; maps evaluate it per pixel.
__global__ void __launch_bounds__(256)
sig_model_kernel(const FrameDesc *__restrict__ frames, const FrameState *__restrict__ state,
	const int4 *__restrict__ tiles, int ntiles, DetectParams prm, Control *ctl, int par, uint2 *cands)
{
	__shared__ double C[MHALO * MHALO];
	__shared__ double wmin[8];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int mode = prm.mode, lm = lap_mode(mode);
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const int4 tile = tiles[t];
		if (!state[tile.x].active)
			continue; // block-uniform
		const FrameDesc &fd = frames[tile.x];
		const int w = fd.w, h = fd.h, words = fd.words, x0 = tile.y, y0 = tile.z;
		double vmin = INFINITY;
		for (int k = tid; k < MHALO * MHALO; k += 256) {
			const double v = clean_at(fd, x0 - 2 + k % MHALO, y0 - 2 + k / MHALO, mode);
			C[k] = v;
			vmin = dmin(vmin, v);
		}
#pragma unroll
		for (int o = 16; o; o >>= 1)
			vmin = dmin(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
		if (lane == 0)
			wmin[warp] = vmin;
		__syncthreads();
		double m_lo = wmin[0];
#pragma unroll
		for (int i = 1; i < 8; ++i)
			m_lo = dmin(m_lo, wmin[i]);
		const bool scalar_noise = !fd.gain_map && !fd.rn_map;
		const double nz_tile = scalar_noise ? noise_from_median(fd, 0, m_lo) : 0.0;
		const uint32_t *holes = plane_ptr(fd, P_HOLE);
		uint32_t hi = 0, lo = 0; // bit j: row warp + 8 j of this lane's column
#pragma unroll 1
		for (int oy = warp; oy < MTILE; oy += 8) {
			const int x = x0 + lane, y = y0 + oy;
			if (y >= h)
				break; // warp-uniform
			uint32_t cls = 0;
			if (x < w) {
				const int cx = lane + 2, cy = oy + 2;
				double l, r, u, d;
				if (lm == WRAP || lm == CONSTANT) {
					l = C[cy * MHALO + cx - 1];
					r = C[cy * MHALO + cx + 1];
					u = C[(cy - 1) * MHALO + cx];
					d = C[(cy + 1) * MHALO + cx];
				} else {
					l = C[cy * MHALO + clampi(x - 1, 0, w - 1) - x0 + 2];
					r = C[cy * MHALO + clampi(x + 1, 0, w - 1) - x0 + 2];
					u = C[(clampi(y - 1, 0, h - 1) - y0 + 2) * MHALO + cx];
					d = C[(clampi(y + 1, 0, h - 1) - y0 + 2) * MHALO + cx];
				}
				const double lap = lap_formula(C[cy * MHALO + cx], u, d, l, r);
				const double nz = scalar_noise ? nz_tile
					: noise_from_median(fd, (long long)y * w + x, m_lo);
				const uint32_t hw = holes[(long long)y * words + (x0 >> 5)];
				cls = (hw >> lane) & 1u ? 0u : candidate_class(lap, nz, prm);
			}
			hi |= (cls & 1u) << (oy >> 3);
			lo |= (cls >> 1) << (oy >> 3);
			clear_detect_words(fd, (long long)y * words + (x0 >> 5), lane);
		}
		// Bits j of this lane are rows y0 + warp + 8 j: append as rows of a
		// strip starting at y0 + warp with stride 8.
		tile_flush(tile.x, w, x0 + lane, y0 + warp, hi, lo, ctl, par, cands);
		__syncthreads();
	}
}

// Noise model at an in-frame pixel (exact: its own 5 x 5 median of clean
// under the border mode).
__device__ __noinline__ double noise_model_at(const FrameDesc &fd, int x, int y, int mode)
{
	int mx[5], my[5];
#pragma unroll
	for (int i = 0; i < 5; ++i) {
		mx[i] = border_index(x + i - 2, fd.w, mode);
		my[i] = border_index(y + i - 2, fd.h, mode);
	}
	double v[25];
#pragma unroll
	for (int c = 0; c < 25; ++c) {
		const int cx = mx[c % 5], cy = my[c / 5];
		v[c] = (cx | cy) < 0 ? 0.0 : fd.clean[(long long)cy * fd.w + cx];
	}
	return noise_from_median(fd, (long long)y * fd.w + x, median_network(v));
}

// Ascending bitonic network over the 32 lanes (compare-exchange form).
__device__ __forceinline__ double warp_sort32(double v)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int span = 2; span <= 32; span *= 2) {
#pragma unroll
		for (int step = span / 2; step; step /= 2) {
			const double peer = __shfl_xor_sync(0xffffffffu, v, step);
			const bool lower = ((lane & span) == 0) == ((lane & step) == 0);
			// The lower lane keeps the smaller value, the upper the larger;
			// on equal values either choice is the same value.
			v = (peer < v) == lower ? peer : v;
		}
	}
	return v;
}

// B: one warp per candidate.  Lane l < 25 evaluates sig_raw at window cell l
// (row-major, folded by the median's border map; zero outside for constant),
// a 32-lane bitonic network (+inf padding) gives the 5 x 5 median, and
// sig = sig_raw(center) - median decides the S1/S2 bits and the seed list.  A
// window holding a NaN takes the reference's exact rule in lane 0.
//
// LOW: the low list (sig_raw can exceed only neighbor_threshold), run after
// the seed kernel.  Only the S2 bit can be set there, and S2 is read only by
// the second growth step, i.e. within distance 2 of a CAND pixel; candidates
// with no CAND bit in their clipped 5 x 5 neighbourhood are skipped.
//
// A candidate whose patch serves (patch_serves: every one under mirror, reflect
// and wrap, else those at least 4 pixels from every edge) stages the 9 x 9 patch
// of border-extended clean pixels around it in the warp's shared memory and
// takes, on noise-model frames, its 25 noise windows from it, and away from the
// edges its Laplacians; the others read border-mapped values from global
// memory.  The patch stays for a seed test of the same pixel.  (With every
// candidate near an edge on the border-mapped path, 25 gathered medians per
// lane, the late passes of 256 cutouts took 163 us, 130 with the patch.)
// Which frames a kernel variant serves: any (decided per frame), error-map
// frames only, or noise-model frames only (a variant compiles one path and
// needs fewer registers).
enum FramePath { PATH_ANY = 0, PATH_ERROR = 1, PATH_MODEL = 2 };

template <int PATH>
__device__ __forceinline__ bool has_error_map(const FrameDesc &fd)
{
	return PATH == PATH_ERROR ? true : PATH == PATH_MODEL ? false : fd.error != nullptr;
}

template <int PATH>
__device__ __forceinline__ bool serves(const FrameDesc &fd)
{
	return PATH == PATH_ANY || (fd.error != nullptr) == (PATH == PATH_ERROR);
}

// Scratch doubles per warp that candidate_sig needs: the sorted vertical runs
// of the 9 x 9 patch on noise-model frames (CS_RUNS), else only the 25 window
// values of the NaN rule.
constexpr int CS_RUNS = 225;

// The 25 noise medians of a staged candidate (src/filters.cuh:46-70, the
// median<5> that noise_model reads), lane l < 25 returning the median of the
// 5 x 5 block of the 9 x 9 patch P at rows l / 5 .. + 4, columns l % 5 .. + 4
// (the window of window cell l).  Clean pixels are never NaN, so the middle
// order statistic is the reference's value (its sign of a zero aside, which
// max(m, 1e-5) removes).
//
// The 25 blocks share their columns: the 45 vertical runs of five (9 columns
// x 5 row offsets) are sorted once per warp into S (S[(r * 5 + i) * 9 + c] =
// i-th smallest of rows r .. r + 4 of column c).  A block of five sorted
// columns whose rows are then sorted is sorted both ways, and its median is the
// median of the 13 cells (i, j) with (i + 1)(j + 1) <= 13 and
// (5 - i)(5 - j) <= 13: every other cell has at least 13 cells known to be no
// larger (or no smaller) than it, six on each side.  So a lane sorts only the
// rank rows of its five columns and takes a median of 13.
__device__ __forceinline__ double patch_window_median(const double *P, double *S)
{
	const int lane = threadIdx.x & 31;
	for (int k = lane; k < 45; k += 32) {
		const int r = k / 9, c = k % 9;
		const double *p = P + r * 9 + c;
		double a = p[0], b = p[9], d = p[18], e = p[27], f = p[36];
		sort5(a, b, d, e, f);
		double *s = S + r * 45 + c;
		s[0] = a;
		s[9] = b;
		s[18] = d;
		s[27] = e;
		s[36] = f;
	}
	__syncwarp();
	double med = 0;
	if (lane < 25) {
		const double *R = S + (lane / 5) * 45 + lane % 5; // rank row i at R + 9 i, columns 0..4
		double band[13];
		int nb = 0;
#pragma unroll
		for (int i = 0; i < 5; ++i) {
			double a = R[9 * i], b = R[9 * i + 1], c = R[9 * i + 2], d = R[9 * i + 3], e = R[9 * i + 4];
			sort5(a, b, c, d, e);
			const double row[5] = {a, b, c, d, e};
#pragma unroll
			for (int j = 0; j < 5; ++j)
				if ((i + 1) * (j + 1) <= 13 && (5 - i) * (5 - j) <= 13)
					band[nb++] = row[j];
		}
		med = median_network(band);
	}
	__syncwarp();
	return med;
}

// What a warp finds out about a candidate's significance sig = center - med5:
// the threshold tests, bounds of sig (equal when it was computed), and what
// exact_sig needs to compute it.
struct Sig {
	bool s1, s2;      // sig > cr, sig > neighbor
	double lo, hi;    // lo <= sig <= hi
	double noise;     // at the pixel
	double center, v; // sig_raw at the pixel; the lane's window value (lanes < 25)
};

// The exact significance (called by the whole warp).
__device__ __forceinline__ double exact_sig(const Sig &g)
{
	if (g.lo == g.hi)
		return g.lo;
	const double v = (threadIdx.x & 31) < 25 ? g.v : INFINITY;
	return g.center - __shfl_sync(0xffffffffu, warp_sort32(v), 12);
}

__device__ __forceinline__ bool interior4(const FrameDesc &fd, int x, int y)
{
	return x >= 4 && y >= 4 && x + 4 < fd.w && y + 4 < fd.h;
}

// Whether the 9 x 9 patch around (x, y), border-extended, holds the windows of
// the pixel's medians: away from the edges, and under mirror, reflect and wrap
// everywhere.  Those border maps are invariant under a group of isometries
// that folds any coordinate onto its image, so the median at a folded position
// and the one at the position itself on the extended pixels have the same
// multiset.  (nearest and constant fold medians, not pixels.)
__device__ __forceinline__ bool patch_serves(const FrameDesc &fd, int x, int y, int mode)
{
	return interior4(fd, x, y) || (mode != NEAREST && mode != CONSTANT);
}

// That patch, three rows of a column per lane (lane 9 g + c < 27: rows 3 g ..
// 3 g + 2 of column c).
__device__ __forceinline__ void load_patch(const FrameDesc &fd, int x, int y, int mode, double (&p)[3])
{
	const int lane = threadIdx.x & 31;
	p[0] = p[1] = p[2] = 0;
	if (lane < 27) {
		int cx = x - 4 + lane % 9, cy[3];
#pragma unroll
		for (int i = 0; i < 3; ++i)
			cy[i] = y - 4 + 3 * (lane / 9) + i;
		if (!interior4(fd, x, y)) { // warp-uniform
			cx = border_index(cx, fd.w, mode);
#pragma unroll
			for (int i = 0; i < 3; ++i)
				cy[i] = border_index(cy[i], fd.h, mode);
		}
#pragma unroll
		for (int i = 0; i < 3; ++i)
			p[i] = fd.clean[(long long)cy[i] * fd.w + cx];
	}
}

__device__ __forceinline__ void store_patch(double *P, const double (&p)[3])
{
	const int lane = threadIdx.x & 31;
	__syncwarp(); // earlier reads of P
	if (lane < 27) {
		double *q = P + 27 * (lane / 9) + lane % 9;
		q[0] = p[0];
		q[9] = p[1];
		q[18] = p[2];
	}
	__syncwarp();
}

// S: the warp's scratch of at least CS_RUNS doubles on noise-model frames
// (25 otherwise).
//
// No sort: fl(center - v) falls as v grows, so sig > t, the test at the
// window's rank 12 value, holds exactly when it holds at 13 or more of the 25
// values (a ballot per threshold).  The window median lies between 0 (sig_raw
// is never negative for positive noise) and SIG_MED_HI when 13 values do,
// which bounds sig for the contrast test; only a seed that these bounds leave
// undecided has its window sorted (exact_sig).
constexpr double SIG_MED_HI = 1.5;

template <bool LOW, int PATH = PATH_ANY>
__device__ __forceinline__ Sig candidate_sig(const FrameDesc &fd, int x, int y, double *P, double *S,
	const DetectParams &prm, bool fresh, bool skip = false)
{
	const int lane = threadIdx.x & 31;
	const int w = fd.w, h = fd.h, mode = prm.mode, lm = lap_mode(mode);
	const bool err = has_error_map<PATH>(fd);
	const bool inside = interior4(fd, x, y), staged = patch_serves(fd, x, y, mode); // warp-uniform
	Sig g;
	double v = INFINITY, nz = 0;
	// The lane's window cell, folded into the frame (negative: a zero).
	int mx = x + lane % 5 - 2, my = y + lane / 5 - 2;
	if (!inside) {
		mx = border_index(mx, w, mode);
		my = border_index(my, h, mode);
	}
	const bool cell = lane < 25, real = cell && (mx | my) >= 0;
	const long long at = (long long)my * w + mx;
	if (staged) {
		double p[3];
		load_patch(fd, x, y, mode, p);
		if (cell && err) // loads with the patch
			nz = fd.error[at];
		store_patch(P, p);
		if (!err) { // warp-uniform
			const double m = patch_window_median(P, S);
			if (cell)
				nz = noise_from_median(fd, at, m);
		}
	} else if (real) {
		nz = err ? fd.error[at] : noise_model_at(fd, mx, my, mode);
	}
	if (cell) {
		double lap = 0;
		if (inside) {
			const double *q = P + (lane / 5 + 2) * 9 + lane % 5 + 2; // the window cell
			lap = lap_formula(q[0], q[-9], q[9], q[-1], q[1]);
		} else if (real) {
			lap = lap_at(fd, mx, my, lm);
		}
		v = real ? lap / (2 * nz) : 0.0;
	}
	const double center = __shfl_sync(0xffffffffu, v, 12);
	g.center = center;
	g.v = v;
	g.noise = __shfl_sync(0xffffffffu, nz, 12);
	if (__any_sync(0xffffffffu, cell && !(v >= 0))) { // a NaN, or a negative noise
		double med;
		if (__any_sync(0xffffffffu, isnan(v))) {
			// The reference's NaN rule on the 25 values, in the warp's scratch
			// (a register array indexed at run time would live in local memory).
			__syncwarp();
			if (cell)
				S[lane] = v;
			__syncwarp();
			med = lane == 0 ? window_median_exact(S, 25) : 0.0;
			med = __shfl_sync(0xffffffffu, med, 0);
			__syncwarp();
		} else {
			med = __shfl_sync(0xffffffffu, warp_sort32(v), 12);
		}
		g.lo = g.hi = center - med;
		g.s1 = g.lo > prm.cr;
		g.s2 = g.lo > prm.nb;
	} else {
		const double d = center - v;
		g.s2 = __popc(__ballot_sync(0xffffffffu, cell && d > prm.nb)) >= 13;
		if (!LOW) {
			g.s1 = __popc(__ballot_sync(0xffffffffu, cell && d > prm.cr)) >= 13;
			g.hi = center;
			g.lo = g.s1 ? prm.cr : -INFINITY; // (read for S1 pixels)
			if (__popc(__ballot_sync(0xffffffffu, cell && v <= SIG_MED_HI)) >= 13)
				g.lo = fmax(g.lo, center - SIG_MED_HI);
		}
	}
	if (lane == 0 && !skip) {
		// Set or clear: a late pass keeps the bits of the previous pass and
		// re-evaluates some pixels.
		const long long word = (long long)y * fd.words + (x >> 5);
		const uint32_t bit = 1u << (x & 31);
		write_bit(plane_ptr(fd, P_S2) + word, bit, g.s2, fresh);
		if (!LOW)
			write_bit(plane_ptr(fd, P_S1) + word, bit, g.s1, fresh);
	}
	return g;
}

// candidate_sig plus the seed slot of candidate e (list-based kernels).  A
// hole (src/filters.cuh:137-146: sig = 0) gets no bit and no seed; its flag
// is loaded before the evaluation and only read after it.
template <int PATH = PATH_ANY>
__device__ __forceinline__ void candidate_eval(const FrameDesc &fd, uint2 t, long long e, int x, int y,
	double *P, double *S, const DetectParams &prm, Seed *seeds, bool fresh, bool hole = false)
{
	const long long word = (long long)y * fd.words + (x >> 5);
	const uint32_t bit = 1u << (x & 31);
	const uint32_t excl = plane_ptr(fd, P_EXCL)[word];
	const Sig g = candidate_sig<false, PATH>(fd, x, y, P, S, prm, fresh, hole);
	const bool seed = !hole && g.s1 && !(excl & bit); // warp-uniform
	const double sig = seed ? exact_sig(g) : 0.0;
	if ((threadIdx.x & 31) == 0) {
		seeds[e] = seed ? Seed{t.x, t.y, sig, g.noise} : Seed{NO_SEED, 0, 0.0, 0.0};
		if (!seed) // the seed kernel decides the CAND bit of a seed
			write_bit(plane_ptr(fd, P_CAND) + word, bit, false, fresh);
	}
}

// The first pass's evaluation of a noise-model candidate by one thread: its 25
// window values from the sig_raw map (region_sig_kernel), their median by a
// sorting network (NaN-free windows: any network gives the median's value, a
// zero's sign aside, which no threshold sees), the S1 / S2 bits and the seed
// slot, as candidate_eval.  A window cell past an edge reads its border-mapped
// pixel (zero in constant mode), which mirror, reflect and nearest keep within
// two pixels of the candidate, so the map holds it; wrap maps it to the far
// side of the frame.  (A warp evaluating each edge candidate on its own, 25
// border-mapped noise medians per lane, held the launch for 121 us on a
// 1531 x 1023 frame with maps, 154 us on five of 1018 x 1001 and 122 us on 256
// cutouts of 40 to 200 pixels; those calls went from 853 to 770, 1193 to 1058
// and 736 to 593 us.)  Returns false for a candidate within two pixels of an
// edge under wrap and for a window holding a NaN: the warp evaluates those.
__device__ __forceinline__ bool map_candidate(const FrameDesc &fd, uint2 t, long long e, int x, int y,
	const DetectParams &prm, Seed *seeds)
{
	const int w = fd.w, h = fd.h;
	const bool inside = x >= 2 && y >= 2 && x + 2 < w && y + 2 < h;
	if (!inside && prm.mode == WRAP)
		return false;
	int mx[5], my[5];
#pragma unroll
	for (int i = 0; i < 5; ++i) {
		mx[i] = x + i - 2;
		my[i] = y + i - 2;
		if (!inside) {
			mx[i] = border_index(mx[i], w, prm.mode);
			my[i] = border_index(my[i], h, prm.mode);
		}
	}
	double v[25];
	bool nan = false;
#pragma unroll
	for (int c = 0; c < 25; ++c) {
		const int cx = mx[c % 5], cy = my[c / 5];
		v[c] = (cx | cy) < 0 ? 0.0 : fd.sig_raw[(long long)cy * w + cx];
		nan |= isnan(v[c]);
	}
	if (nan)
		return false;
	const long long word = (long long)y * fd.words + (x >> 5);
	const uint32_t bit = 1u << (x & 31);
	const bool hole = (plane_ptr(fd, P_HOLE)[word] & bit) != 0;
	const uint32_t excl = plane_ptr(fd, P_EXCL)[word];
	const double nz = fd.noise[(long long)y * w + x];
	const double center = v[12];
	const double sig = center - median_network(v);
	if (!hole) { // a hole's significance is zero: no bit (the planes start zeroed)
		write_bit(plane_ptr(fd, P_S2) + word, bit, sig > prm.nb, true);
		write_bit(plane_ptr(fd, P_S1) + word, bit, sig > prm.cr, true);
	}
	const bool seed = !hole && sig > prm.cr && !(excl & bit);
	seeds[e] = seed ? Seed{t.x, t.y, sig, nz} : Seed{NO_SEED, 0, 0.0, 0.0};
	return true;
}

// B, high list: one warp per candidate.  Holes have sig = 0
// (src/filters.cuh:137-146): no bit, no seed; the dense kernel does not test
// the hole plane itself.
// PATH: the frames this launch serves (FramePath); the other launch of a
// mixed batch takes the rest of the list.
template <int PATH>
__global__ void __launch_bounds__(256, 4)
candidate_high_kernel(const FrameDesc *__restrict__ frames, const uint2 *__restrict__ cands,
	DetectParams prm, Control *ctl, int par, Seed *seeds)
{
	__shared__ double patches[8][81];
	__shared__ double scratch[8][CS_RUNS];
	double *P = patches[threadIdx.x >> 5], *S = scratch[threadIdx.x >> 5];
	const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	const long long n = (long long)ctl->pass[par].n_cand;
	uint2 next = gw < n ? cands[gw] : make_uint2(0u, 0u);
	for (long long e = gw; e < n; e += nw) {
		const uint2 t = next;
		if (e + nw < n) // the next entry loads during this evaluation
			next = cands[e + nw];
		const FrameDesc &fd = frames[t.x];
		if (!serves<PATH>(fd))
			continue; // warp-uniform
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		const bool hole = test_bit(plane_ptr(fd, P_HOLE), fd.words, x, y);
		candidate_eval<PATH>(fd, t, e, x, y, P, S, prm, seeds, true, hole);
	}
}

// B, high list, first pass on noise-model frames: a thread per candidate
// whose window the sig_raw map holds (map_candidate); the warp evaluates the
// others (wrap's frame edges, windows with a NaN) one after another with
// candidate_eval.  Its own launch bounds: the thread path holds 25 window
// values, the warp path (candidate_high_kernel) runs at four blocks per SM.
__global__ void __launch_bounds__(256, 2)
candidate_map_kernel(const FrameDesc *__restrict__ frames, const uint2 *__restrict__ cands,
	DetectParams prm, Control *ctl, Seed *seeds)
{
	constexpr int PATH = PATH_MODEL;
	__shared__ double patches[8][81];
	__shared__ double scratch[8][CS_RUNS];
	double *P = patches[threadIdx.x >> 5], *S = scratch[threadIdx.x >> 5];
	const long long n = (long long)ctl->pass[0].n_cand;
	const int lane = threadIdx.x & 31;
	const long long stride = (long long)gridDim.x * blockDim.x;
	for (long long base = blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31); base < n;
	     base += stride) { // warp-uniform
		const long long e = base + lane;
		uint2 t = make_uint2(0u, 0u);
		bool defer = false;
		if (e < n) {
			t = cands[e];
			const FrameDesc &fd = frames[t.x];
			if (serves<PATH>(fd)) {
				const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
				defer = !(fd.sig_raw && map_candidate(fd, t, e, x, y, prm, seeds));
			}
		}
		for (unsigned m = __ballot_sync(0xffffffffu, defer); m; m &= m - 1) {
			const int j = __ffs(m) - 1;
			const uint2 tj = make_uint2(__shfl_sync(0xffffffffu, t.x, j),
				__shfl_sync(0xffffffffu, t.y, j));
			const FrameDesc &fd = frames[tj.x];
			const int x = (int)(tj.y % (unsigned)fd.w), y = (int)(tj.y / (unsigned)fd.w);
			const bool hole = test_bit(plane_ptr(fd, P_HOLE), fd.words, x, y);
			candidate_eval<PATH>(fd, tj, base + j, x, y, P, S, prm, seeds, true, hole);
		}
	}
}

// Growth (reference src/filters.cuh:177-193 twice, src/cleaner.cuh:123-125):
// grown = dilate3x3(dilate3x3(CAND) & S1) & S2, clipped to the frame; fresh =
// grown & ~CRMASK joins the mask and the target list (src/cleaner.cuh:22-37).
//
// It is driven by the work lists, because what can grow lies within two pixels of one: 58,520 of 67 million pixels are CAND on
// 16 frames of 2048 x 2048.  (The row sweeps over the bit planes that this
// replaced took 126 us in the four passes of those frames, bound by their
// chains of dependent word loads, most of which found nothing.)
//
// first: the pass's planes were zeroed, so everything that grows grows from a
// CAND pixel's own 5 x 5 neighbourhood.  Otherwise pixels may also grow
// because an S1 or S2 bit near an old CAND pixel was set; every bit set in the
// pass belongs to a listed pixel, and the S1 cells within one pixel of it that
// touch a CAND pixel dilate into its 5 x 5 neighbourhood.  There a
// LOW pixel's S2 bit may date from an earlier pass (it is evaluated again, on
// its own, wherever its CAND neighbourhood changed), so only HIGH pixels count.

// Eight lanes work on a listed pixel (x, y), lane r < 5 of them on row
// y - 2 + r: the S1 cells within one pixel of (x, y) that touch a CAND pixel,
// dilated, with S2 set (late passes: and HIGH) and not in the mask yet, join
// the mask and the target list.  A lane loads its row's words together, and
// the rows meet by shuffles: a few hundred instructions in all, where a thread
// per pixel unrolls over a thousand, whose fetching took most of the time of
// a late pass's growth (11 us for 34 pixels).
enum GrowKind {
	GROW_FIRST, // the full pass: any S2 pixel
	GROW_LATE,  // HIGH pixels only, and the new pixels' FRESH bits
	GROW_SELF   // only (x, y) itself, whose S2 bit was just found set
};

// Called by the whole warp (on: the lane's group has a pixel; fd, x, y, f are
// its group's).  track: set FRESH bits.
__device__ __forceinline__ void grow_group(const FrameDesc &fd, int f, int x, int y, bool on, GrowKind kind,
	bool track, FrameState *state, Control *ctl, int par, uint2 *targets)
{
	const int lane = threadIdx.x & 31, r = lane & 7, yy = y - 2 + r;
	const int words = fd.words, w = fd.w, k = (x - 2) >> 5, s = (x - 2) & 31; // k >= -1
	const bool in = on && r < 5 && yy >= 0 && yy < fd.h;
	uint32_t c = 0, s1 = 0, s2 = 0, old = 0, donor = 0;
	if (in) {
		c = bits5(plane_ptr(fd, P_CAND), words, x, yy);
		s1 = bits5(plane_ptr(fd, P_S1), words, x, yy);
		s2 = kind == GROW_SELF ? (r == 2 ? 4u : 0u) : bits5(plane_ptr(fd, P_S2), words, x, yy);
		if (kind == GROW_LATE)
			s2 &= bits5(plane_ptr(fd, P_HIGH), words, x, yy);
		old = bits5(plane_ptr(fd, P_CRMASK), words, x, yy);
		donor = bits5(plane_ptr(fd, P_DONOR), words, x, yy);
	}
	uint32_t v = c | __shfl_up_sync(0xffffffffu, c, 1, 8) | __shfl_down_sync(0xffffffffu, c, 1, 8);
	v = r >= 1 && r <= 3 ? (v | (v << 1) | (v >> 1)) & s1 & 0xeu : 0u; // columns x - 1 .. x + 1
	const uint32_t d = (v | (v << 1) | (v >> 1)) & 0x1fu;
	uint32_t g = d | __shfl_up_sync(0xffffffffu, d, 1, 8) | __shfl_down_sync(0xffffffffu, d, 1, 8);
	g &= s2 & ~old;
	if (!__any_sync(0xffffffffu, g != 0))
		return;
	uint32_t now = 0;
	if (g) { // (columns left of the frame have no S2 bits)
		uint32_t *crm = plane_ptr(fd, P_CRMASK) + (long long)yy * words + k;
		const unsigned long long wide = (unsigned long long)g << s;
		const uint32_t lo = (uint32_t)wide, hi = (uint32_t)(wide >> 32);
		const uint32_t o0 = lo ? atomicOr(crm, lo) : 0u, o1 = hi ? atomicOr(crm + 1, hi) : 0u;
		now = g & ~(uint32_t)((o0 | (unsigned long long)o1 << 32) >> s);
		if (track && now) {
			uint32_t *fr = plane_ptr(fd, P_FRESH) + (long long)yy * words + k;
			const unsigned long long n = (unsigned long long)now << s;
			if ((uint32_t)n)
				atomicOr(fr, (uint32_t)n);
			if (n >> 32)
				atomicOr(fr + 1, (uint32_t)(n >> 32));
		}
	}
	// The new pixels into the target list, and their frames' state: once for
	// the warp when its groups share a frame.
	const unsigned some = __ballot_sync(0xffffffffu, now != 0);
	if (!some)
		return;
	unsigned long long slot = warp_append(&ctl->n_targets, __popc(now));
	const int lost = __popc(now & donor);
	const int lead = __ffs(some) - 1, f0 = __shfl_sync(0xffffffffu, f, lead);
	const bool same = __all_sync(0xffffffffu, !now || f == f0);
	const int sum = (int)__reduce_add_sync(0xffffffffu, (unsigned)lost);
	if (now && (!same || lane == lead)) {
		const int gone = same ? sum : lost;
		atomicOr(&state[f].todo[par], 1u);
		if (gone)
			atomicAdd(&state[f].masked, (unsigned long long)gone);
	}
	const unsigned base = (unsigned)((long long)yy * w + x - 2);
	for (; now; now &= now - 1)
		targets[slot++] = make_uint2((unsigned)f, base + __ffs(now) - 1);
}

// The same for every pixel of the frames, a warp per row of 32 words: two dilations
// on bit words, for a pass whose high list holds over a 16th of the pixels (eight
// lanes for each of 0.9 million listed pixels of a 2048 x 2048 frame took about 250 us,
// the rows 20; at a 64th the two are even).
// late: HIGH pixels only, the new pixels' FRESH bits, and the high list's LISTED bits
// cleared.  A function of its own: its registers are not its callers'.
// (The rows come with the batch's pixels: a load of those would delay the rule.)
struct RowItems {
	const int2 *rows;
	int n;
	unsigned long long px;
};

__device__ __forceinline__ bool grows_by_rows(unsigned long long n_cand, const RowItems &rows)
{
	return 16 * n_cand > rows.px;
}

// Columns 32 k - 2 .. 32 k + 33 of row y of a plane (bit 0: the first), zero outside.
__device__ __forceinline__ unsigned long long window2(const uint32_t *plane, int words, int h, int y, int k)
{
	if (y < 0 || y >= h)
		return 0ull;
	const uint32_t *row = plane + (long long)y * words;
	const unsigned long long l = k > 0 ? row[k - 1] >> 30 : 0u, r = k + 1 < words ? row[k + 1] & 3u : 0u;
	return l | (unsigned long long)row[k] << 2 | r << 34;
}

__device__ __noinline__ void grow_rows(const FrameDesc *__restrict__ frames, FrameState *state,
	const RowItems &rows, bool late, Control *ctl, int par, uint2 *targets, Team team)
{
	const int lane = threadIdx.x & 31;
	const int gw = (team.block * blockDim.x + threadIdx.x) >> 5, nw = (team.blocks * blockDim.x) >> 5;
	for (int i = gw; i < rows.n; i += nw) {
		const int2 item = rows.rows[i];
		const int f = item.x, y = item.y;
		if (!state[f].active)
			continue; // warp-uniform
		const FrameDesc &fd = frames[f];
		const int words = fd.words, h = fd.h;
		for (int k0 = 0; k0 < words; k0 += 32) {
			const int k = k0 + lane;
			const long long o = (long long)y * words + k;
			uint32_t now = 0;
			int lost = 0;
			if (k < words) {
				if (late)
					plane_ptr(fd, P_LISTED)[o] = 0u;
				unsigned long long c[5], v = 0; // CAND; S1 cells that touch one
#pragma unroll
				for (int r = 0; r < 5; ++r)
					c[r] = window2(plane_ptr(fd, P_CAND), words, h, y - 2 + r, k);
#pragma unroll
				for (int r = 0; r < 3; ++r) {
					const unsigned long long m = c[r] | c[r + 1] | c[r + 2];
					if (m)
						v |= (m | m << 1 | m >> 1) & window2(plane_ptr(fd, P_S1), words, h, y - 1 + r, k);
				}
				uint32_t g = (uint32_t)((v | v << 1 | v >> 1) >> 2);
				if (g) {
					g &= plane_ptr(fd, P_S2)[o];
					if (late)
						g &= plane_ptr(fd, P_HIGH)[o];
				}
				if (g) // (low pixels join the mask beside this)
					now = g & ~atomicOr(plane_ptr(fd, P_CRMASK) + o, g);
				if (now) {
					lost = __popc(now & plane_ptr(fd, P_DONOR)[o]);
					if (late)
						atomicOr(plane_ptr(fd, P_FRESH) + o, now);
				}
			}
			if (!__any_sync(0xffffffffu, now != 0))
				continue;
			unsigned long long slot = warp_append(&ctl->n_targets, __popc(now));
			lost = __reduce_add_sync(0xffffffffu, lost);
			if (lane == 0) {
				atomicOr(&state[f].todo[par], 1u);
				if (lost)
					atomicAdd(&state[f].masked, (unsigned long long)lost);
			}
			const unsigned pix = (unsigned)((long long)y * fd.w + 32 * k);
			for (; now; now &= now - 1)
				targets[slot++] = make_uint2((unsigned)f, pix + __ffs((int)now) - 1);
		}
	}
}

// Any CAND pixel within two pixels of (x, y) (S2 is read only by the second
// growth step, within that distance of a CAND pixel), and no hole there.
__device__ __forceinline__ bool low_near(const FrameDesc &fd, int x, int y)
{
	const uint32_t *cand = plane_ptr(fd, P_CAND);
	const bool hole = test_bit(plane_ptr(fd, P_HOLE), fd.words, x, y);
	uint32_t any = 0;
#pragma unroll
	for (int d = -2; d <= 2; ++d)
		any |= y + d >= 0 && y + d < fd.h ? bits5(cand, fd.words, x, y + d) : 0u;
	return any && !hole;
}

// The warp's evaluation of a low-list pixel near a CAND pixel: its S2 bit,
// which, when set, may grow the pixel itself.
template <int PATH>
__device__ __forceinline__ void low_eval(const FrameDesc *__restrict__ frames, FrameState *state, uint2 t,
	const DetectParams &prm, Control *ctl, int par, uint2 *targets, double *P, double *S, bool fresh)
{
	const FrameDesc &fd = frames[t.x];
	const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
	const Sig g = candidate_sig<true, PATH>(fd, x, y, P, S, prm, fresh);
	if (g.s2) // warp-uniform
		grow_group(fd, (int)t.x, x, y, (threadIdx.x & 31) < 8, GROW_SELF, !fresh, state, ctl, par, targets);
}

// Low list and growth of a full pass (run after the seeds): a lane per low
// entry tests its neighbourhood, the warp evaluates the survivors one after
// another.  `grow`: this launch grows the high list (a mixed batch launches
// the low list once per kind of frame, and grows once).
template <int PATH>
__global__ void __launch_bounds__(256, PATH == PATH_ERROR ? 4 : 3)
low_grow_kernel(const FrameDesc *__restrict__ frames, FrameState *state, const uint2 *__restrict__ cands,
	DetectParams prm, Control *ctl, int par, uint2 *targets, int grow, RowItems rows)
{
	__shared__ double patches[8][81];
	__shared__ double scratch[8][PATH == PATH_ERROR ? 25 : CS_RUNS];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const long long stride = (long long)gridDim.x * blockDim.x;
	long long nc = grow ? (long long)ctl->pass[par].n_cand : 0;
	const long long nl = (long long)ctl->pass[par].n_low;
	if (grows_by_rows((unsigned long long)nc, rows)) {
		grow_rows(frames, state, rows, false, ctl, par, targets, whole_grid());
		nc = 0;
	}
	const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5, nw = stride >> 5;
	// Entries per warp and sweep: 32 for a long list, fewer for a short one,
	// whose survivors then land on different warps.  (Dealing the entries to the
	// warps one by one spreads them better, but no two lanes' loads share a line
	// then: 60 instead of 48 us on 16 frames of 2048 x 2048.)
	auto chunk_of = [&](long long n) { return n >= nw * 32 ? 32 : n > nw ? (int)((n + nw - 1) / nw) : 1; };
	const int cc = chunk_of(nc), cl = chunk_of(nl);
	for (long long base = gw * cc; base < nc; base += nw * cc) { // warp-uniform
		const long long e = base + lane;
		uint2 t = make_uint2(0u, 0u);
		bool cand = false;
		if (lane < cc && e < nc) {
			t = cands[e];
			const FrameDesc &fd = frames[t.x];
			cand = test_bit(plane_ptr(fd, P_CAND), fd.words, (int)(t.y % (unsigned)fd.w),
				(int)(t.y / (unsigned)fd.w));
		}
		for (unsigned m = __ballot_sync(0xffffffffu, cand); m;) { // four CAND pixels at a time
			int j = -1;
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				if (q == lane >> 3)
					j = __ffs(m) - 1;
				m &= m - 1;
			}
			const unsigned f = __shfl_sync(0xffffffffu, t.x, j & 31), pix = __shfl_sync(0xffffffffu, t.y, j & 31);
			const FrameDesc &fd = frames[f];
			grow_group(fd, (int)f, (int)(pix % (unsigned)fd.w), (int)(pix / (unsigned)fd.w), j >= 0, GROW_FIRST,
				false, state, ctl, par, targets);
		}
	}
	const unsigned long long cap = ctl->cand_cap;
	for (long long base = gw * cl; base < nl; base += nw * cl) { // warp-uniform
		const long long e = base + lane;
		uint2 t = make_uint2(0, 0);
		bool near = false;
		if (lane < cl && e < nl) {
			t = cands[cap - 1 - e];
			const FrameDesc &fd = frames[t.x];
			near = serves<PATH>(fd) && low_near(fd, (int)(t.y % (unsigned)fd.w), (int)(t.y / (unsigned)fd.w));
		}
		for (unsigned m = __ballot_sync(0xffffffffu, near); m; m &= m - 1) {
			const int j = __ffs(m) - 1;
			const uint2 tj = make_uint2(__shfl_sync(0xffffffffu, t.x, j), __shfl_sync(0xffffffffu, t.y, j));
			low_eval<PATH>(frames, state, tj, prm, ctl, par, targets, patches[warp], scratch[warp], true);
		}
	}
}

// Element RANK < 32 of the 64 values held as (a, b) = slots (lane, 32 + lane)
// of a warp, by an ascending bitonic network: a sorts ascending and b
// descending, the half-cleaner keeps the 32 smallest in a, and only a is
// merged further.  NaN-free inputs; on equal values either choice of a
// compare-exchange is the same value.
template <int RANK>
__device__ __forceinline__ double warp_rank64(double a, double b)
{
	static_assert(RANK >= 0 && RANK < 32, "the lower half holds the rank");
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
		for (int j = k >> 1; j > 0; j >>= 1) {
			const double pa = __shfl_xor_sync(0xffffffffu, a, j);
			const double pb = __shfl_xor_sync(0xffffffffu, b, j);
			const bool mina = ((lane & j) == 0) == ((lane & k) == 0);
			const bool minb = ((lane & j) == 0) == (((lane + 32) & k) == 0);
			a = (pa < a) == mina ? pa : a;
			b = (pb < b) == minb ? pb : b;
		}
	}
	a = dmin(a, b);
#pragma unroll
	for (int j = 16; j > 0; j >>= 1) {
		const double pa = __shfl_xor_sync(0xffffffffu, a, j);
		a = (pa < a) == ((lane & j) == 0) ? pa : a;
	}
	return __shfl_sync(0xffffffffu, a, RANK);
}

// How many of the 49 3 x 3 windows of a 9 x 9 patch hold five or more pixels
// above t_hi, and how many hold five or more below t_lo (called by the whole
// warp, the patch as load_patch distributes it).  The patch becomes 81 bits
// per threshold by ballots; lane 8 k + j (j < 7) sums the three columns, then
// the three rows, of the seven windows starting in row j, bit-sliced.
struct WindowCounts {
	int above, below;
};

__device__ __forceinline__ WindowCounts count_windows(const double (&p)[3], double t_hi, double t_lo)
{
	const int lane = threadIdx.x & 31, j = lane & 7;
	uint32_t rows[3];
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		const uint32_t up = __ballot_sync(0xffffffffu, lane < 27 && p[k] > t_hi);
		const uint32_t dn = __ballot_sync(0xffffffffu, lane < 27 && p[k] < t_lo);
		// The one of rows j .. j + 2 that is k modulo 3.
		rows[k] = (lane < 8 ? up : dn) >> (9 * ((j + 2 - k) / 3));
	}
	uint32_t one[3], two[3]; // a row's sums of three columns: ones and twos
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		const uint32_t a = rows[k], b = a >> 1, c = a >> 2;
		one[k] = a ^ b ^ c;
		two[k] = (a & b) | (c & (a ^ b));
	}
	const uint32_t z = one[0] ^ one[1] ^ one[2];
	const uint32_t carry = (one[0] & one[1]) | (one[2] & (one[0] ^ one[1]));
	const uint32_t x1 = two[0] ^ two[1], c1 = two[0] & two[1], x2 = two[2] ^ carry, c2 = two[2] & carry;
	const uint32_t odd = x1 ^ x2, c3 = x1 & x2;
	// z + 2 (odd + 2 (c1 + c2 + c3)) >= 5
	const uint32_t five = ((c1 & c2) | ((c1 | c2 | c3) & (odd | z))) & 0x7fu;
	const int n = j < 7 && lane < 16 ? __popc(five) : 0;
	const unsigned sum = __reduce_add_sync(0xffffffffu, (unsigned)(lane < 8 ? n : n << 8));
	return WindowCounts{(int)(sum & 0xffu), (int)(sum >> 8)};
}

// The warp's fine-structure test of a seed at (x, y) (src/filters.cuh:148-175):
// fine = max((med3 - med7) / noise, 0.01) with med7 the median of the 49 3 x 3
// medians around it, and CAND = sig / fine > contrast.
//
// A seed whose patch serves (patch_serves) is decided without any 3 x 3 median
// but its own: the test holds at med7 exactly when it holds with 25 or more of
// the 49 medians in med7's place (it can only turn true as that value grows),
// a median m satisfies it when med3 - m < sig noise / contrast (and sig / 0.01
// > contrast), and m > t exactly when five or more of its nine pixels are.  So
// the seed is CAND when 25 windows hold five pixels above t_hi = med3 - sig_lo
// noise / contrast, and not when 25 hold five below t_lo, the same with sig_hi,
// both with a margin of 1e-12 for the roundings (of two products here, of a
// difference and two divisions in the test).  sig need not be exact for that:
// sig_lo and sig_hi bound it.  What these counts leave open, values outside
// the range where the margin covers the roundings, and the other seeds take
// the medians and the exact sig (from exact(), called by the whole warp).
//
// (Sorting the 25 window values, 63 column triples and 49 medians across the
// warp took about 950 warp instructions per candidate and seed on error maps.
// The candidates and seeds of 16 frames of 2048 x 2048 took 168 us with it and
// 95 with the counts, 379 and 213 us where the error map underestimates the
// noise of most frames; the noise-model seeds of 64 ragged frames 476 and
// 251 us.)
template <class Exact>
__device__ __forceinline__ void seed_eval(const FrameDesc &fd, int x, int y, double sig_lo, double sig_hi,
	double noise, const DetectParams &prm, double *P, double (*T)[63], bool fresh, bool staged,
	Exact exact)
{
	const int lane = threadIdx.x & 31;
	const int w = fd.w, h = fd.h, mode = prm.mode;
	const bool patch = patch_serves(fd, x, y, mode); // warp-uniform
	int verdict = -1; // undecided
	if (patch) {
		double p[3];
		if (staged) { // the candidate evaluation left this patch in P
			const double *q = P + (lane < 27 ? 27 * (lane / 9) + lane % 9 : 0);
			p[0] = q[0];
			p[1] = q[9];
			p[2] = q[18];
		} else {
			load_patch(fd, x, y, mode, p);
			store_patch(P, p);
		}
		const double k = prm.contrast, floor_k = k * FINE_FLOOR;
		const bool sane = noise > 1e-100 && noise < 1e100 && sig_hi < 1e100 && k > 1e-100 && k < 1e100;
		if (sane && sig_hi < floor_k * (1 - 1e-12)) {
			verdict = 0;
		} else if (sane && sig_lo > floor_k * (1 + 1e-12)) {
			// The seed's own 3 x 3 median: the value of rank 4, by counting.
			const double own = lane < 9 ? P[30 + 9 * (lane / 3) + lane % 3] : 0.0;
			int rank = 0;
#pragma unroll
			for (int i = 0; i < 9; ++i) {
				const double o = P[30 + 9 * (i / 3) + i % 3];
				rank += i < lane ? o <= own : o < own;
			}
			const unsigned at = __ballot_sync(0xffffffffu, lane < 9 && rank == 4);
			const double med3 = __shfl_sync(0xffffffffu, own, __ffs(at) - 1);
			const double ql = sig_lo * noise * prm.rcontrast, qh = sig_hi * noise * prm.rcontrast;
			const double t_hi = (med3 - ql * (1 - 1e-12)) + 1e-15 * (fabs(med3) + ql);
			const double t_lo = (med3 - qh * (1 + 1e-12)) - 1e-15 * (fabs(med3) + qh);
			const WindowCounts n = count_windows(p, t_hi, t_lo);
			verdict = n.above >= 25 ? 1 : n.below >= 25 ? 0 : -1;
		}
	}
	bool cand = verdict > 0;
	if (verdict < 0) { // warp-uniform
		const double sig = exact();
		double m3[2] = {INFINITY, INFINITY};
		if (patch) {
			__syncwarp();
			for (int k = lane; k < 63; k += 32) {
				double a = P[k], b = P[k + 9], c = P[k + 18];
				cas(a, b);
				cas(b, c);
				cas(a, b);
				T[0][k] = a;
				T[1][k] = b;
				T[2][k] = c;
			}
			__syncwarp();
#pragma unroll
			for (int s = 0; s < 2; ++s) {
				const int j = lane + 32 * s;
				if (j < 49) {
					const int k = (j / 7) * 9 + j % 7; // window rows j/7 .. +2, columns j%7 .. +2
					const double *lo = &T[0][k], *mid = &T[1][k], *hi = &T[2][k];
					m3[s] = med3(dmax(dmax(lo[0], lo[1]), lo[2]), med3(mid[0], mid[1], mid[2]),
						dmin(dmin(hi[0], hi[1]), hi[2]));
				}
			}
		} else {
#pragma unroll
			for (int s = 0; s < 2; ++s) {
				const int j = lane + 32 * s;
				if (j < 49) {
					int qx = x + j % 7 - 3, qy = y + j / 7 - 3;
					double m = 0;
					if (!(mode == CONSTANT && (qx < 0 || qx >= w || qy < 0 || qy >= h))) {
						qx = clampi(qx, 0, w - 1); // nearest folds the medians
						qy = clampi(qy, 0, h - 1);
						int mx[3], my[3];
#pragma unroll
						for (int i = 0; i < 3; ++i) {
							mx[i] = border_index(qx + i - 1, w, mode);
							my[i] = border_index(qy + i - 1, h, mode);
						}
						double v[9];
#pragma unroll
						for (int c = 0; c < 9; ++c)
							v[c] = (mx[c % 3] | my[c / 3]) < 0 ? 0.0
								: fd.clean[(long long)my[c / 3] * w + mx[c % 3]];
						m = median9(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8]);
					}
					m3[s] = m;
				}
			}
		}
		const double med3c = __shfl_sync(0xffffffffu, m3[0], 24);
		const double med7 = warp_rank64<24>(m3[0], m3[1]);
		double fine = (med3c - med7) / noise;
		fine = fine < FINE_FLOOR ? FINE_FLOOR : fine;
		cand = sig / fine > prm.contrast;
	}
	if (lane == 0)
		write_bit(plane_ptr(fd, P_CAND) + (long long)y * fd.words + (x >> 5), 1u << (x & 31), cand,
			fresh);
}

// C (list-based): one warp per seed slot.
__global__ void __launch_bounds__(256)
seed_kernel(const FrameDesc *__restrict__ frames, const Seed *__restrict__ seeds, DetectParams prm,
	const Control *ctl, int par)
{
	__shared__ double patches[8][81];
	__shared__ double triples[8][3][63];
	const int warp = threadIdx.x >> 5;
	const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	const long long n = (long long)ctl->pass[par].n_cand;
	Seed next = gw < n ? seeds[gw] : Seed{NO_SEED, 0, 0.0, 0.0};
	for (long long e = gw; e < n; e += nw) {
		const Seed sd = next;
		if (e + nw < n) // the next slot loads during this evaluation
			next = seeds[e + nw];
		if (sd.frame == NO_SEED)
			continue; // warp-uniform
		const FrameDesc &fd = frames[sd.frame];
		seed_eval(fd, (int)(sd.pixel % (unsigned)fd.w), (int)(sd.pixel / (unsigned)fd.w), sd.sig, sd.sig,
			sd.noise, prm, patches[warp], triples[warp], true, false, [&] { return sd.sig; });
	}
}

// B and C fused, high list: one warp per candidate, and a candidate that is
// a seed gets its fine-structure test from the same warp at once (it needs
// only its own sig and noise and the clean pixels within 4), so no seed list
// is walked.  Error-map frames only: noise-model candidates run
// candidate_map_kernel.  With `seeds` (a batch that also runs seed_kernel) each
// served entry's slot is marked empty.
__global__ void __launch_bounds__(256, 4)
candidate_seed_kernel(const FrameDesc *__restrict__ frames, const uint2 *__restrict__ cands,
	DetectParams prm, Control *ctl, Seed *seeds)
{
	// The scratch of candidate_sig holds just the 25 values of the NaN rule, and
	// the triples of the seed test serve as it.
	constexpr int PATH = PATH_ERROR;
	__shared__ double patches[8][81];
	__shared__ double triples[8][3][63];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	double *P = patches[warp];
	const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	const long long n = (long long)ctl->pass[0].n_cand;
	uint2 next = gw < n ? cands[gw] : make_uint2(0u, 0u);
	for (long long e = gw; e < n; e += nw) {
		const uint2 t = next;
		if (e + nw < n) // the next entry loads during this evaluation
			next = cands[e + nw];
		const FrameDesc &fd = frames[t.x];
		if (!serves<PATH>(fd))
			continue; // warp-uniform
		const int x = (int)(t.y % (unsigned)fd.w), y = (int)(t.y / (unsigned)fd.w);
		const long long word = (long long)y * fd.words + (x >> 5);
		const uint32_t bit = 1u << (x & 31);
		const bool hole = (plane_ptr(fd, P_HOLE)[word] & bit) != 0;
		const uint32_t excl = plane_ptr(fd, P_EXCL)[word];
		if (seeds && lane == 0)
			seeds[e] = Seed{NO_SEED, 0, 0.0, 0.0};
		const Sig g = candidate_sig<false, PATH>(fd, x, y, P, &triples[warp][0][0], prm, true, hole);
		if (!hole && g.s1 && !(excl & bit)) // warp-uniform
			seed_eval(fd, x, y, g.lo, g.hi, g.noise, prm, P, triples[warp], true, true,
				[&] { return exact_sig(g); });
	}
}

} // namespace cb
