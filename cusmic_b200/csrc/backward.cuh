// Adjoint of the cleaned pixels with the detection mask frozen.
//
// With the final mask fixed, the forward is piecewise linear in (data, bg):
//   unflagged finite pixel p: out_p = (x_p + bg_p) - bg_p     -> d/dx_p = 1
//   non-finite pixel p:       out_p = x_p (returned as is)     -> identity
//   flagged pixel p:          out_p = sel(x_d + bg_d) - bg_p, where sel is the
//     replacement median over the final donors: one donor d (odd count) or
//     the two central donors with weight 1/2 each (even count).
// So dL/dx_d += w_d g_p, dL/dbg_d += w_d g_p and dL/dbg_p -= g_p.  The donor
// selected at a rank is recomputed (not stored): donors are ordered by their
// IEEE total-order key, ties by lowest linear index.
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace cb {

// Words of 32 pixels whose loads a warp of bwd_dense_kernel issues before their
// use (memory bounds it; three frames of 777 x 900 with a background map: 24 us
// one word at a time, 13.5 with 4, 11 with 8, as with 16; eight of 1024 x 1024: 29
// and 26).
constexpr int BWD_WORDS = 8;

// Pass-through part: grad_data = g off the mask, 0 on it; with background
// maps, grad_bg = -g on the mask and 0 elsewhere.
__global__ void __launch_bounds__(256)
bwd_dense_kernel(const FrameDesc *__restrict__ frames, const int2 *__restrict__ rows, int nrows,
	const double *__restrict__ g, double *__restrict__ gx, double *__restrict__ gbg_map,
	const long long *__restrict__ offsets)
{
	const int lane = threadIdx.x & 31;
	const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
	for (int r = gw; r < nrows; r += nw) {
		const int2 item = rows[r];
		const FrameDesc &fd = frames[item.x];
		const uint32_t *crm = plane_ptr(fd, P_CRMASK) + (long long)item.y * fd.words;
		const long long base = offsets[item.x] + (long long)item.y * fd.w;
		const int w = fd.w;
		for (int xb = 0; xb < w; xb += 32 * BWD_WORDS) {
			double gi[BWD_WORDS];
			uint32_t cw[BWD_WORDS];
#pragma unroll
			for (int u = 0; u < BWD_WORDS; ++u) {
				const int x = xb + 32 * u + lane;
				if (x < w) {
					gi[u] = g[base + x];
					cw[u] = crm[x >> 5];
				}
			}
#pragma unroll
			for (int u = 0; u < BWD_WORDS; ++u) {
				const int x = xb + 32 * u + lane;
				if (x < w) {
					const bool flagged = (cw[u] >> lane) & 1u;
					gx[base + x] = flagged ? 0.0 : gi[u];
					if (gbg_map)
						gbg_map[base + x] = flagged ? -gi[u] : 0.0;
				}
			}
		}
	}
}

// data + bg of an in-frame pixel: the value the forward's replacement compared
// (donors are finite inputs).
__device__ __forceinline__ double donor_value(const FrameDesc &fd, long long i)
{
	double c = fd.data[i];
	if (fd.has_bg)
		c += 1 * (fd.bg_map ? fd.bg_map[i] : fd.bg);
	return c;
}

// Linear index of the donor at `rank` in (key, linear index) order, for a
// window of at most 32 cells held one per lane (key = ~0 for non-donors).
__device__ __forceinline__ int donor_at_rank32(unsigned long long key, int idx, int rank)
{
	const int lane = threadIdx.x & 31;
	unsigned long long v = key;
#pragma unroll
	for (int span = 2; span <= 32; span *= 2) {
#pragma unroll
		for (int step = span / 2; step; step /= 2) {
			unsigned long long peer = __shfl_xor_sync(0xffffffffu, v, step);
			bool lower = ((lane & span) == 0) == ((lane & step) == 0);
			v = lower ? (peer < v ? peer : v) : (v < peer ? peer : v);
		}
	}
	const unsigned long long k = __shfl_sync(0xffffffffu, v, rank);
	const int less = __popc(__ballot_sync(0xffffffffu, key < k));
	unsigned same = __ballot_sync(0xffffffffu, key == k);
	for (int t = rank - less; t > 0; --t)
		same &= same - 1;
	return __shfl_sync(0xffffffffu, idx, __ffs(same) - 1);
}

// Both central donors of up to 32 S cells in row-major order (cell(pos, x, y) for
// pos < n): lane l holds the keys of cells l + 32 s, the warp sorts a copy, and a
// rank's donor is the (rank - less)-th one with the sorted key, in cell (= linear
// index) order.  Returns the number of donors (0: d_lo and d_hi unset).
//
// (A radix select reads the window 64 times, bit by bit, for each rank: a
// few clusters of flagged pixels held the launch for 49 us on eight frames of
// 1024 x 1024, 18 with the sort.)
template <int S, class Cell>
__device__ __forceinline__ int sorted_donors(const FrameDesc &fd, const uint32_t *don, const uint32_t *crm,
	int n, Cell cell, long long &d_lo, long long &d_hi)
{
	const int lane = threadIdx.x & 31;
	unsigned long long own[S], k[S];
	int nd = 0;
#pragma unroll
	for (int s = 0; s < S; ++s) {
		const int pos = lane + 32 * s;
		own[s] = ~0ull;
		if (pos < n) {
			int x, y;
			cell(pos, x, y);
			if (donor_at(don, crm, fd.words, x, y))
				own[s] = order_key(donor_value(fd, (long long)y * fd.w + x));
		}
		k[s] = own[s];
		nd += __popc(__ballot_sync(0xffffffffu, own[s] != ~0ull));
	}
	if (!nd)
		return 0;
	sort_keys(k);
	auto donor = [&](int rank) {
		unsigned long long v = 0;
#pragma unroll
		for (int s = 0; s < S; ++s)
			if (s == rank >> 5)
				v = k[s];
		v = __shfl_sync(0xffffffffu, v, rank & 31);
		int skip = rank;
#pragma unroll
		for (int s = 0; s < S; ++s)
			skip -= __popc(__ballot_sync(0xffffffffu, own[s] < v));
		int pos = -1; // warp-uniform
#pragma unroll
		for (int s = 0; s < S; ++s) {
			unsigned m = __ballot_sync(0xffffffffu, own[s] == v);
			const int c = __popc(m);
			if (pos < 0 && skip < c) {
				for (; skip > 0; --skip)
					m &= m - 1;
				pos = 32 * s + __ffs(m) - 1;
			} else if (pos < 0) {
				skip -= c;
			}
		}
		int x, y;
		cell(pos, x, y);
		return (long long)y * fd.w + x;
	};
	d_lo = donor((nd - 1) / 2);
	d_hi = nd % 2 ? d_lo : donor(nd / 2);
	return nd;
}

// A window of 33 .. 32 S cells.
template <int S>
__device__ __noinline__ int sorted_window_donors(const FrameDesc &fd, const uint32_t *don,
	const uint32_t *crm, Window win, long long &d_lo, long long &d_hi)
{
	const int ww = win.x1 - win.x0 + 1, area = ww * (win.y1 - win.y0 + 1);
	return sorted_donors<S>(fd, don, crm, area, [&](int pos, int &x, int &y) {
		x = win.x0 + pos % ww;
		y = win.y0 + pos / ww;
	}, d_lo, d_hi);
}

// Linear index of the donor at `rank` in (key, linear index) order among a
// ring's cells: radix select of the key, then the (rank - less)-th donor with
// that key in row-major (= linear index) order.
__device__ long long ring_donor(const FrameDesc &fd, const uint32_t *don, const uint32_t *crm,
	const Ring &q, int rank)
{
	const int lane = threadIdx.x & 31;
	unsigned long long prefix = 0, used = 0;
	int r = rank;
	for (int bit = 63; bit >= 0; --bit) {
		const unsigned long long flag = 1ull << bit;
		int below = 0;
		for (int pos = lane; pos < q.n; pos += 32) {
			int x, y;
			ring_cell(q, pos, x, y);
			if (!donor_at(don, crm, fd.words, x, y))
				continue;
			unsigned long long k = order_key(donor_value(fd, (long long)y * fd.w + x));
			below += (k & used) == prefix && !(k & flag);
		}
		below = warp_sum_int(below);
		used |= flag;
		if (r >= below) {
			prefix |= flag;
			r -= below;
		}
	}
	// r is now the number of equal keys to skip in row-major order.
	for (int pos0 = 0; pos0 < q.n; pos0 += 32) {
		const int pos = pos0 + lane;
		bool match = false;
		int x = 0, y = 0;
		if (pos < q.n) {
			ring_cell(q, pos, x, y);
			match = donor_at(don, crm, fd.words, x, y) &&
				order_key(donor_value(fd, (long long)y * fd.w + x)) == prefix;
		}
		unsigned m = __ballot_sync(0xffffffffu, match);
		int c = __popc(m);
		if (r < c) {
			for (int t = r; t > 0; --t)
				m &= m - 1;
			int src = __ffs(m) - 1;
			int sx = __shfl_sync(0xffffffffu, x, src), sy = __shfl_sync(0xffffffffu, y, src);
			return (long long)sy * fd.w + sx;
		}
		r -= c;
	}
	return -1; // unreachable when rank < donor count
}

// far_window_median's two central donors, as linear indices.
__device__ __noinline__ int far_window_donors(const FrameDesc &fd, const uint32_t *don, const uint32_t *crm,
	int x, int y, int &nd, long long &d_lo, long long &d_hi)
{
	const int r = nearest_donor(fd, don, crm, x, y);
	if (!r)
		return 0;
	const Ring q = ring_cells(fd.w, fd.h, x, y, r);
	if (q.n <= 128) {
		nd = sorted_donors<4>(fd, don, crm, q.n, [&](int pos, int &cx, int &cy) { ring_cell(q, pos, cx, cy); },
			d_lo, d_hi);
		return r;
	}
	int cnt = 0;
	for (int pos = threadIdx.x & 31; pos < q.n; pos += 32) {
		int cx, cy;
		ring_cell(q, pos, cx, cy);
		cnt += donor_at(don, crm, fd.words, cx, cy);
	}
	nd = warp_sum_int(cnt);
	d_lo = ring_donor(fd, don, crm, q, (nd - 1) / 2);
	d_hi = nd % 2 ? d_lo : ring_donor(fd, don, crm, q, nd / 2);
	return r;
}

// One warp per flagged pixel: recompute its final replacement window and
// donors, scatter w * g to the selected donor(s).
__global__ void __launch_bounds__(256)
bwd_scatter_kernel(const FrameDesc *__restrict__ frames, const uint2 *__restrict__ list,
	const unsigned long long *count, const long long *__restrict__ offsets,
	const double *__restrict__ g, double *gx, double *gbg_map, double *gbg_scalar)
{
	const int lane = threadIdx.x & 31;
	const long long gw = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
	const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
	const long long n = (long long)*count;
	for (long long e = gw; e < n; e += nw) {
		const uint2 t = list[e];
		const FrameDesc &fd = frames[t.x];
		const int w = fd.w, h = fd.h;
		const int x = (int)(t.y % (unsigned)w), y = (int)(t.y / (unsigned)w);
		const uint32_t *don = plane_ptr(fd, P_DONOR), *crm = plane_ptr(fd, P_CRMASK);
		const long long off = offsets[t.x];
		const double gp = g[off + t.y];
		const int limit = max(w, h);
		for (int r = 2; r <= limit; ++r) {
			Window win = {max(0, x - r), min(w - 1, x + r), max(0, y - r), min(h - 1, y + r)};
			const int ww = win.x1 - win.x0 + 1, area = ww * (win.y1 - win.y0 + 1);
			long long d_lo, d_hi;
			int nd;
			if (area <= 32) {
				unsigned long long key = ~0ull;
				int idx = 0;
				bool d = false;
				if (lane < area) {
					int cx = win.x0 + lane % ww, cy = win.y0 + lane / ww;
					d = donor_at(don, crm, fd.words, cx, cy);
					idx = cy * w + cx;
					if (d)
						key = order_key(donor_value(fd, idx));
				}
				nd = __popc(__ballot_sync(0xffffffffu, d));
				if (!nd)
					continue;
				d_lo = donor_at_rank32(key, idx, (nd - 1) / 2);
				d_hi = nd % 2 ? d_lo : donor_at_rank32(key, idx, nd / 2);
			} else if (area <= 128) {
				nd = area <= 64 ? sorted_window_donors<2>(fd, don, crm, win, d_lo, d_hi)
					: sorted_window_donors<4>(fd, don, crm, win, d_lo, d_hi);
				if (!nd)
					continue;
			} else if (!far_window_donors(fd, don, crm, x, y, nd, d_lo, d_hi)) {
				break;
			}
			if (lane == 0) {
				// Odd count: the middle donor, weight 1.  Even: the two central
				// donors, weight 1/2 each (midpoint either form).
				const double wl = nd % 2 ? gp : gp / 2, wh = nd % 2 ? 0.0 : gp / 2;
				atomicAdd(&gx[off + d_lo], wl);
				if (!(nd % 2))
					atomicAdd(&gx[off + d_hi], wh);
				if (gbg_map) {
					atomicAdd(&gbg_map[off + d_lo], wl);
					if (!(nd % 2))
						atomicAdd(&gbg_map[off + d_hi], wh);
				}
				if (gbg_scalar && fd.has_bg)
					atomicAdd(&gbg_scalar[t.x], (wl + wh) - gp);
			}
			break;
		}
	}
}

} // namespace cb
