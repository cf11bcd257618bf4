// Device pieces of the pairlist walk shared by the plain and the batched
// builds: the reference's exact pair test, the walk of a run of rows, and the
// join of a slice's far entries.
#pragma once

#include "mb2_internal.cuh"

namespace mb2 {

// ExclusionView::row_contains / same_body (src/Interactions/DeviceExclusions.h:22-75):
// b is excluded from the row [row_b, row_e) of the CSR or shares its rigid body.
__device__ __forceinline__ bool is_excluded(const Exclusions& ex, int b, int row_b, int row_e,
											int body) {
	if (body >= 0 && ex.rigid_body_id[b] == body) return true;
	for (int e = row_b; e < row_e; ++e)
		if (ex.neighbors[e] == b) return true;
	return false;
}

// Exact reference test: wrap_diff(pj - pi).length2() <= rc2, same rounding.
__device__ __forceinline__ bool exact_hit(const Box& box, const float4& pi, const float4& pj,
										  float rc2) {
	const float3 d = wrap_diff(box, __fsub_rn(pj.x, pi.x), __fsub_rn(pj.y, pi.y),
							   __fsub_rn(pj.z, pi.z));
	return len2(d.x, d.y, d.z) <= rc2;
}

// Most rows a warp walks, and the shared memory it does so in.
constexpr uint32_t kWalkRows = 8;
struct WalkShared {
	float4 rows[kWalkRows];                // position, original index in .w
	int4 excl[kWalkRows];                  // exclusion row [x, y), rigid body z
	unsigned long long base[kWalkRows];    // index of the row's entry 0 in the list
	float4 cand[64];                       // candidates that passed the run's test, index in .w
};

// One cell grid's arrays and the list being written.
struct WalkArrays {
	const float4* sorted_pos;
	const uint32_t* s2o;
	const uint32_t* begin;  // this grid's cells
	const uint32_t* end;
	const StencilEntry* stencil;
	int ns;
	uint32_t* nbr;
	uint32_t cap;
	int hshift;
	uint32_t* row_len;
	uint32_t* row_back;
};

// nearest image of x (a multiple of l away): x - l rint(x / l), one rounding;
// inv = 0 (an open axis) leaves x.
__device__ __forceinline__ float nearest(float x, float l, float inv, float* k) {
	constexpr float kRound = 12582912.0f;  // 1.5 * 2^23: adding it rounds to nearest
	*k = __fsub_rn(__fmaf_rn(x, inv, kRound), kRound);
	return __fmaf_rn(*k, -l, x);
}

// The rows [rb, re) of one cell c (at most kWalkRows), walked by one warp.
//
// The lanes take the cell's pruned stencil 32 cells at a time (cells whose
// Morton code precedes c hold only earlier particles and are skipped), lay
// their candidate ranges end to end (a warp scan of the lengths) and load 32
// candidates a round, each lane finding its candidate's cell by a binary
// search over the running totals held one per lane and read with shuffles. A
// candidate is moved into the image nearest the rows' coordinate box once for
// all rows, dropped when its distance from that box is beyond the radius, and
// otherwise queued in shared memory; each time the queue holds 32, one per
// lane, they are tested against every row. So the cost of finding, loading
// and moving a candidate is shared by the run's rows, the test that is left is
// three differences and a sum of squares, and all lanes hold a candidate.
//
// A cheap distance decides all but candidates within rounding of the radius
// (fast_lo < d^2 <= fast_hi), which take the reference's exact test behind a
// warp vote, so the pair set is the reference's bit for bit. Where the image
// nearest the box need not be the one nearest each row (a box edge below twice
// the radius and the run's extent), each row takes its own; particles far
// outside the box (exact_all) take the exact test throughout.
//
// A row's hits are appended with two ballots: near entries (within split2)
// from the front of its slots, far ones from the back, or (near_last) the other
// way round; join_back_slice then moves the back part behind the front part. Entries past cap are only counted
// (the host then grows the list and walks again). Returns the rows' total and
// longest lengths in *total and *longest (the same in every lane).
template <bool kExcl>
__device__ __forceinline__ void walk_run(const WalkArrays& w, const WalkGrid& wg, const Box& box,
										 const Exclusions& ex, WalkShared& sh, uint32_t rb,
										 uint32_t re, uint32_t c, bool exact_all,
										 uint32_t* total_out, uint32_t* longest_out) {
	const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
	const int nr = static_cast<int>(re - rb);
	const int cells = 1 << wg.m;
	const float len[3] = {box.size[0], box.size[1], box.size[2]};
	const float inv[3] = {box.periodic[0] ? box.inv[0] : 0.0f, box.periodic[1] ? box.inv[1] : 0.0f,
						  box.periodic[2] ? box.inv[2] : 0.0f};
	// The rows and their coordinate box.
	const uint32_t mine = rb + min(lane & (kWalkRows - 1u), static_cast<uint32_t>(nr - 1));
	const float4 q = w.sorted_pos[mine];
	const int own = static_cast<int>(w.s2o[mine]);
	float mid[3] = {q.x, q.y, q.z}, half[3] = {q.x, q.y, q.z};
#pragma unroll
	for (int a = 0; a < 3; ++a) {
		float lo = mid[a], hi = mid[a];
#pragma unroll
		for (uint32_t o = kWalkRows / 2; o > 0; o >>= 1) {
			lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
			hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
		}
		mid[a] = 0.5f * (lo + hi);
		half[a] = 0.5f * (hi - lo) + wg.eps[a];
	}
	if (lane < static_cast<uint32_t>(nr)) {
		sh.rows[lane] = make_float4(q.x, q.y, q.z, __int_as_float(own));
		if (kExcl) {
			int4 e = make_int4(0, 0, -1, 0);
			if (ex.offsets && static_cast<uint32_t>(own) < ex.num_particles) {
				e.x = ex.offsets[own];
				e.y = ex.offsets[own + 1];
			}
			if (ex.rigid_body_id) e.z = ex.rigid_body_id[own];
			sh.excl[lane] = e;
		}
		const uint32_t h = 1u << w.hshift;
		sh.base[lane] = (static_cast<unsigned long long>(mine >> w.hshift) * w.cap << w.hshift) +
						(mine & (h - 1u));
	}
	__syncwarp();
	const float gate = wg.fast_hi * 1.00001f, rc = sqrtf(gate);
	bool per_row = false;
#pragma unroll
	for (int a = 0; a < 3; ++a)
		per_row = per_row || (box.periodic[a] && len[a] <= 2.0f * (rc + half[a] + wg.eps[a]));
	uint32_t row_len = 0, row_back = 0;  // of row `lane`
	uint32_t queued = 0;
	const bool split = wg.split2 < INFINITY;

	auto test = [&](uint32_t m) {
		const bool there = lane < m;
		const float4 p = sh.cand[lane];
		const uint32_t j = __float_as_uint(p.w);
		const int bj = there ? static_cast<int>(w.s2o[j]) : 0;
		for (int r = 0; r < nr; ++r) {
			const float4 row = sh.rows[r];
			float dx = p.x - row.x, dy = p.y - row.y, dz = p.z - row.z;
			if (per_row) {
				float k;
				dx = nearest(dx, len[0], inv[0], &k);
				dy = nearest(dy, len[1], inv[1], &k);
				dz = nearest(dz, len[2], inv[2], &k);
			}
			const float d2 = dx * dx + dy * dy + dz * dz;
			const bool later = there && j > rb + static_cast<uint32_t>(r);
			bool hit = later && d2 < wg.fast_lo && !exact_all;
			const bool band = later && !hit && (d2 <= wg.fast_hi || exact_all);
			if (__any_sync(0xFFFFFFFFu, band)) {
				if (band) hit = exact_hit(box, w.sorted_pos[rb + r], w.sorted_pos[j], wg.rc2);
			}
			if (kExcl && hit) {
				const int4 e = sh.excl[r];
				hit = !is_excluded(ex, bj, e.x, e.y, e.z);
			}
			const bool front = !split || (d2 <= wg.split2) != (wg.near_last != 0);
			const uint32_t nm = __ballot_sync(0xFFFFFFFFu, hit && front);
			const uint32_t fm = __ballot_sync(0xFFFFFFFFu, hit && !front);
			if ((nm | fm) == 0u) continue;
			const uint32_t all = __shfl_sync(0xFFFFFFFFu, row_len, r);
			const uint32_t back = __shfl_sync(0xFFFFFFFFu, row_back, r);
			if (hit) {
				const uint32_t place = all + static_cast<uint32_t>(__popc((nm | fm) & lt));
				const uint32_t slot =
					front ? all - back + static_cast<uint32_t>(__popc(nm & lt))
						  : w.cap - 1u - (back + static_cast<uint32_t>(__popc(fm & lt)));
				const uint32_t flip = bj < __float_as_int(row.w) ? kOrientBit : 0u;
				if (place < w.cap)
					w.nbr[sh.base[r] + (static_cast<unsigned long long>(slot) << w.hshift)] = j | flip;
			}
			if (static_cast<int>(lane) == r) {
				row_len += static_cast<uint32_t>(__popc(nm | fm));
				row_back += static_cast<uint32_t>(__popc(fm));
			}
		}
	};

	const uint32_t lvl = (1u << (3 * wg.m)) - 1u;
	const uint32_t mx = 0x24924924u & lvl, my = 0x12492492u & lvl, mz = 0x09249249u & lvl;
	// A neighbour's cell code is the home code plus the stencil entry's
	// interleaved offset on each axis, carried through the other axes' bits
	// (set to one) and masked: modulo 2^m per axis, so open axes also check
	// the plain coordinate range.
	const uint32_t cxo = c | ~mx, cyo = c | ~my, czo = c | ~mz;
	const int cx = static_cast<int>(compact_by3(c >> 2)), cy = static_cast<int>(compact_by3(c >> 1)),
			  cz = static_cast<int>(compact_by3(c));
	for (int k0 = 0; k0 < w.ns; k0 += 32) {
		uint32_t jb = 0, je = 0;
		const int k = k0 + static_cast<int>(lane);
		if (k < w.ns) {
			const StencilEntry se = w.stencil[k];
			bool in = true;
			if (!box.periodic[0]) in = in && static_cast<unsigned>(cx + se.dx) < static_cast<unsigned>(cells);
			if (!box.periodic[1]) in = in && static_cast<unsigned>(cy + se.dy) < static_cast<unsigned>(cells);
			if (!box.periodic[2]) in = in && static_cast<unsigned>(cz + se.dz) < static_cast<unsigned>(cells);
			if (in) {
				const uint32_t d = static_cast<uint32_t>(se.pad);
				const uint32_t nc = ((cxo + (d & mx)) & mx) | ((cyo + (d & my)) & my) |
									((czo + (d & mz)) & mz);
				if (nc >= c) {  // earlier cells hold only earlier particles
					const uint32_t b = w.begin[nc];
					jb = b > rb + 1u ? b : rb + 1u;
					je = w.end[nc];
				}
			}
		}
		// An empty cell (begin = end = 0) or one that ends at the rows has jb >= je.
		const uint32_t cnt = je > jb ? je - jb : 0u;
		uint32_t incl = cnt;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
			if (static_cast<int>(lane) >= o) incl += v;
		}
		const uint32_t stream = __shfl_sync(0xFFFFFFFFu, incl, 31);
		const uint32_t off = jb - (incl - cnt);  // candidate t of this cell is off + t
		for (uint32_t t0 = 0; t0 < stream; t0 += 32u) {
			const uint32_t t = t0 + lane;
			int owner = 0;  // first lane whose running total exceeds t
#pragma unroll
			for (int step = 16; step > 0; step >>= 1) {
				const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, owner + step - 1);
				if (v <= t) owner += step;
			}
			const uint32_t j = __shfl_sync(0xFFFFFFFFu, off, owner & 31) + t;
			bool pass = false;
			float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
			if (t < stream) {
				p = w.sorted_pos[j];
				float k0f, k1f, k2f;
				const float dx = nearest(p.x - mid[0], len[0], inv[0], &k0f);
				const float dy = nearest(p.y - mid[1], len[1], inv[1], &k1f);
				const float dz = nearest(p.z - mid[2], len[2], inv[2], &k2f);
				const float gx = fmaxf(0.0f, fabsf(dx) - half[0]);
				const float gy = fmaxf(0.0f, fabsf(dy) - half[1]);
				const float gz = fmaxf(0.0f, fabsf(dz) - half[2]);
				pass = exact_all || gx * gx + gy * gy + gz * gz <= gate;
				p.x = __fmaf_rn(k0f, -len[0], p.x);
				p.y = __fmaf_rn(k1f, -len[1], p.y);
				p.z = __fmaf_rn(k2f, -len[2], p.z);
				p.w = __uint_as_float(j);
			}
			const uint32_t pm = __ballot_sync(0xFFFFFFFFu, pass);
			if (pass) sh.cand[queued + static_cast<uint32_t>(__popc(pm & lt))] = p;
			queued += static_cast<uint32_t>(__popc(pm));
			__syncwarp();
			if (queued >= 32u) {
				test(32u);
				queued -= 32u;
				const float4 rest = sh.cand[32u + lane];
				__syncwarp();
				sh.cand[lane] = rest;
				__syncwarp();
			}
		}
	}
	if (queued) test(queued);
	__syncwarp();
	if (lane < static_cast<uint32_t>(nr)) {
		w.row_len[rb + lane] = row_len;
		w.row_back[rb + lane] = row_back;
	}
	*total_out = __reduce_add_sync(0xFFFFFFFFu, row_len);
	*longest_out = __reduce_max_sync(0xFFFFFFFFu, row_len);
}

// Moves the back entries of a slice's rows (stored backwards from the end of
// each row's cap slots) to follow the front ones, so that a row is one
// contiguous run, each part in candidate order but the back one reversed. One
// warp per slice of H rows; len, back: of row (lane mod H). Lane l copies
// entries l / H, l / H + 32 / H, ... of that row, so each load and store
// instruction touches neighbouring words. Destinations precede sources (front +
// back <= cap) and every batch is loaded before it is stored, so the in-place
// copy is safe.
__device__ __forceinline__ void join_back_slice(uint32_t* __restrict__ nbr, uint32_t len,
												uint32_t back, uint32_t slice, uint32_t cap,
												int hshift) {
	const uint32_t lane = threadIdx.x & 31u;
	const uint32_t h = 1u << hshift;
	const uint32_t r = lane & (h - 1u), kk = lane >> hshift, step = 32u >> hshift;
	const uint32_t front = len - back;
	uint32_t most = back;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xFFFFFFFFu, most, o));
	uint32_t* base = nbr + static_cast<size_t>(slice) * cap * h + r;
	for (uint32_t k0 = 0; k0 < most; k0 += step) {
		const uint32_t k = k0 + kk;
		uint32_t v = 0u;
		if (k < back) v = base[static_cast<size_t>(cap - back + k) * h];
		__syncwarp();
		if (k < back) base[static_cast<size_t>(front + k) * h] = v;
		__syncwarp();
	}
}

}  // namespace mb2
