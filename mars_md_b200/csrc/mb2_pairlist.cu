// Pairlist build over Morton-sorted particles.
//
// Replaces BuildCellRangesKernel / BuildCellNeighborsKernel /
// ZOrderCellNeighborKernel (src/PatchOperation/PairListKernels/ZOrderNeighbor.h)
// and the grow-and-retry loop of ZOrderPairlist::find_neighbors_zorder
// (src/PatchOperation/PairListKernels/ZOrderPairlist.cpp:208-366).
//
// The pair SET is the reference's: for sorted i < sorted j, keep (i, j) when
// wrap_diff(pos_j - pos_i).length2() <= rc^2 (float, exactly as the reference
// rounds it) and the pair is not excluded. Only the search differs.
//
// Search. Cells are the top 3m bits of the 30-bit Morton key; a cell's
// particles are a contiguous run of the sorted array. The stencil is every
// cell whose box-to-box distance from the home cell can be within rc (a
// pruned sphere, not the reference's (2r+1)^3 cube), at the cell level chosen
// per run to minimise the walk's cost (choose_cell_grid). A warp owns up to 8
// consecutive sorted particles (walk_rows) and walks them in runs of one cell: its
// lanes find and load 32 candidates of the cell's stencil at a time, drop those
// too far from the run's coordinate box, and test the rest, one a lane, against
// every row of the run (walk_run). The test is a cheap minimum-image distance; only
// candidates inside a rounding band around rc (sized from the float ulp of the
// box) take the exact reference computation.
//
// Storage. A half list in sliced ELL form: rows of H consecutive particles
// form a slice; entry k of row i sits at ((i / H) * cap + k) * H + i % H, so
// that G = 32 / H lanes per row reading k..k+G-1 of H rows touch one 128-byte
// line. row_len[i] holds the row's length. Bit 31 of an entry records the
// reference's pair orientation: set when the original index of j is smaller
// than that of i (the reference computes that pair as j -> i).
#include "mb2_internal.cuh"
#include "mb2_walk.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>

namespace mb2 {

namespace {

double ulp_of(double x) {
	x = std::fabs(x);
	if (x < 1e-30) return 1e-45;
	return std::ldexp(1.0, static_cast<int>(std::floor(std::log2(x))) - 23);
}

}  // namespace

CellGrid choose_cell_grid(const float* extent, const int* periodic, float rc_list, size_t n,
						  double rows, int m_lo, int m_hi) {
	CellGrid best;
	double best_cost = -1.0;
	const double rc = static_cast<double>(rc_list);
	for (int m = m_lo; m <= m_hi; ++m) {
		const int cells = 1 << m;
		const double num_cells = std::ldexp(1.0, 3 * m);
		if (m > m_lo && num_cells > 2.0 * static_cast<double>(n)) break;
		std::vector<int> off[3];
		std::vector<double> gap[3];
		double wmin[3] = {0, 0, 0};
		for (int a = 0; a < 3; ++a) {
			if (m == 0) {
				off[a] = {0};
				gap[a] = {0.0};
				wmin[a] = extent[a];
				continue;
			}
			// Real-space cell widths: cell c spans Morton coordinates
			// [c 2^k, (c+1) 2^k) of the 0..1023 scale over the domain, so it is
			// extent * 2^k / 1023 wide, except the last, extent * (2^k - 1) / 1023.
			const int k = 10 - m;
			wmin[a] = static_cast<double>(extent[a]) * (std::ldexp(1.0, k) - 1.0) / 1023.0 *
					  (1.0 - 1e-6);
			const int r = static_cast<int>(std::floor(rc / wmin[a])) + 1;
			if (periodic[a] && 2 * r + 1 >= cells) {
				for (int d = 0; d < cells; ++d) {
					off[a].push_back(d);
					gap[a].push_back(0.0);
				}
			} else {
				for (int d = -r; d <= r; ++d) {
					off[a].push_back(d);
					gap[a].push_back(std::max(0, std::abs(d) - 1) * wmin[a]);
				}
			}
		}
		std::vector<StencilEntry> st;
		const double lim = rc * rc * (1.0 + 1e-4) + 1e-6;
		for (size_t x = 0; x < off[0].size(); ++x)
			for (size_t y = 0; y < off[1].size(); ++y)
				for (size_t z = 0; z < off[2].size(); ++z) {
					const double g2 =
						gap[0][x] * gap[0][x] + gap[1][y] * gap[1][y] + gap[2][z] * gap[2][z];
					if (g2 <= lim) {
						// pad: the offsets modulo 2^m interleaved into Morton bit
						// positions (x at 3k + 2, y at 3k + 1, z at 3k).
						const auto wrap = [cells](int v) {
							return static_cast<uint32_t>(((v % cells) + cells) % cells);
						};
						const uint32_t d = (split_by3(wrap(off[0][x])) << 2) |
										   (split_by3(wrap(off[1][y])) << 1) |
										   split_by3(wrap(off[2][z]));
						st.push_back(StencilEntry{off[0][x], off[1][y], off[2][z],
												  static_cast<int>(d)});
					}
				}
		const double per_cell = static_cast<double>(n) / num_cells;
		// What the walk spends on a row: finding the stencil's cells (some 3 warp
		// instructions each) and loading and placing their candidates (2.4 each, of
		// the half that follow the rows), shared by the rows of a run; a run is
		// what a warp's rows have in one cell. (The tests against the rows
		// themselves hardly depend on the level.) Against counting cells and
		// candidates alone: 131,071 beads 411 -> 333 us.
		const double run = std::max(1.0, rows / (1.0 + (rows - 1.0) / std::max(per_cell, 1e-6)));
		const double cost = static_cast<double>(st.size()) * (3.0 + 1.2 * per_cell) / run;
		if (best_cost < 0.0 || cost < best_cost) {
			best_cost = cost;
			best.m = m;
			best.shift = 3 * (10 - m);
			best.num_stencil = static_cast<int>(st.size());
			best.stencil = st;
		}
	}
	return best;
}

void fast_test_band(const Box& box, float rc_list, float* fast_lo, float* fast_hi) {
	// Each minimum-image component differs from the reference's wrap_diff by at
	// most a few ulp of the largest coordinate magnitude; bound |d^2 - d_ref^2|.
	double mag = 0.0;
	for (int a = 0; a < 3; ++a)
		mag = std::max({mag, std::fabs(static_cast<double>(box.origin[a])),
						std::fabs(static_cast<double>(box.origin[a]) + box.size[a]),
						static_cast<double>(box.size[a])});
	const double rc = rc_list;
	const double per_axis = 4.0 * ulp_of(2.0 * mag);
	const double delta = 2.0 * rc * 3.0 * per_axis * 2.0 + rc * rc * 1e-6;
	*fast_lo = static_cast<float>(rc * rc - delta);
	*fast_hi = static_cast<float>(rc * rc + delta);
}

namespace {

__global__ void __launch_bounds__(256) cell_ranges_kernel(const uint32_t* __restrict__ keys,
														  uint32_t n, int shift,
														  uint32_t* __restrict__ begin,
														  uint32_t* __restrict__ end) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint32_t c = keys[i] >> shift;
	if (i == 0 || (keys[i - 1] >> shift) != c) begin[c] = i;
	if (i + 1 == n || (keys[i + 1] >> shift) != c) end[c] = i + 1;
}

// The walk: each warp owns rows_per_warp consecutive sorted particles and walks
// them in runs of one cell (walk_run). Bound by issuing the tests. Against one
// warp a particle, which found, loaded and exactly tested every candidate anew
// for each row: 131,071 beads 564 -> 347 us, 512 systems of 500 to 20,000 beads
// 1.31 -> 0.76 ms; about even up to 20,000 particles, where a warp has one or two
// rows. Against one lane a particle, which ran the appends of 32 rows one
// candidate at a time: 300,007 beads, 20 steps with a rebuild, 5.36 -> 4.92 ms.
// Statistics are added once per block.
template <bool kExcl>
__global__ void __launch_bounds__(256) build_walk_kernel(
	const uint32_t* __restrict__ keys, WalkArrays w, WalkGrid wg, uint32_t n, Box box,
	Exclusions ex, uint32_t rows_per_warp, const unsigned long long* __restrict__ outside,
	unsigned long long* __restrict__ stats) {
	__shared__ WalkShared shared[8];
	__shared__ uint32_t part[2][8];
	const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
	const uint32_t i0 = (blockIdx.x * 8u + warp) * rows_per_warp;
	uint32_t total = 0, longest = 0;
	if (i0 < n) {
		const uint32_t rows = min(rows_per_warp, n - i0);
		const bool exact_all = *outside != 0ull;
		const uint32_t cell = keys[i0 + min(lane, rows - 1u)] >> wg.shift;
		for (uint32_t r = 0; r < rows;) {
			const uint32_t c = __shfl_sync(0xFFFFFFFFu, cell, r);
			const uint32_t same = __ballot_sync(0xFFFFFFFFu, cell == c && lane >= r && lane < rows);
			const uint32_t run = static_cast<uint32_t>(__popc(same));
			uint32_t t, l;
			walk_run<kExcl>(w, wg, box, ex, shared[warp], i0 + r, i0 + r + run, c, exact_all, &t, &l);
			total += t;
			longest = max(longest, l);
			r += run;
			__syncwarp();
		}
	}
	if (lane == 0) {
		part[0][warp] = total;
		part[1][warp] = longest;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		unsigned long long sum = 0, most = 0;
		for (int k = 0; k < 8; ++k) {
			sum += part[0][k];
			most = max(most, static_cast<unsigned long long>(part[1][k]));
		}
		if (sum) {
			atomicAdd(stats, sum);
			atomicMax(stats + 1, most);
		}
	}
}

__global__ void __launch_bounds__(256) export_kernel(const uint32_t* __restrict__ nbr,
													 const uint32_t* __restrict__ row_len,
													 const uint32_t* __restrict__ row_off,
													 const uint32_t* __restrict__ s2o, uint32_t n,
													 uint32_t cap, int hshift,
													 int2* __restrict__ out) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const int a = static_cast<int>(s2o[i]);
	const int h = 1 << hshift;
	const uint32_t* base = nbr + (static_cast<size_t>(i >> hshift) * cap << hshift) + (i & (h - 1));
	const uint32_t len = row_len[i], off = row_off[i];
	for (uint32_t k = 0; k < len; ++k) {
		const int b = static_cast<int>(s2o[base[static_cast<size_t>(k) * h] & ~kOrientBit]);
		out[off + k] = make_int2(a < b ? a : b, a < b ? b : a);
	}
}

// After a storing walk: each slice's far entries joined to its near ones.
__global__ void __launch_bounds__(256) join_back_kernel(uint32_t* __restrict__ nbr,
													   const uint32_t* __restrict__ row_len,
													   const uint32_t* __restrict__ row_back,
													   uint32_t n, uint32_t cap, int hshift) {
	const uint32_t slice = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
	const uint32_t slices = (n + (1u << hshift) - 1u) >> hshift;
	if (slice >= slices) return;  // whole warp
	const uint32_t i = (slice << hshift) + (threadIdx.x & ((1u << hshift) - 1u));
	join_back_slice(nbr, i < n ? row_len[i] : 0u, i < n ? row_back[i] : 0u, slice, cap, hshift);
}

__global__ void __launch_bounds__(256) displacement_kernel(const float4* __restrict__ cur,
														   const float4* __restrict__ prev,
														   uint32_t n, float3 len,
														   unsigned int* __restrict__ out) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	// The word so far, read before the loads so its latency overlaps theirs:
	// a warp whose maximum is not above it has nothing to raise.
	const unsigned int seen = (threadIdx.x & 31) == 0 ? *reinterpret_cast<volatile unsigned int*>(out) : 0u;
	float d2 = 0.0f;
	if (i < n) {
		const float4 c = cur[i], p = prev[i];
		const float dx = min_image(__fsub_rn(c.x, p.x), len.x);
		const float dy = min_image(__fsub_rn(c.y, p.y), len.y);
		const float dz = min_image(__fsub_rn(c.z, p.z), len.z);
		d2 = len2(dx, dy, dz);
		if (isnan(d2)) d2 = 0.0f;  // a NaN coordinate does not trip the skin check
	}
	// Non-negative floats order like their bit patterns.
	const unsigned int bits = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(d2));
	if ((threadIdx.x & 31) == 0 && bits > seen) atomicMax(out, bits);
}

__global__ void __launch_bounds__(256) pack_kernel(const float4* pos, const int* type_ids,
												   const uint32_t* s2o, uint32_t n,
												   float4* sorted_pos, unsigned long long* odd,
												   float3 far_lo, float3 far_hi, float4* clear_a,
												   float4* clear_b, DisplacementTrack track) {
	chain_begin();
	chain_wait();
	const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
	// The tracked word so far, read before the loads (see displacement_kernel).
	const unsigned int seen = track.d2max && (threadIdx.x & 31) == 0
								  ? *reinterpret_cast<volatile unsigned int*>(track.d2max)
								  : 0u;
	float d2 = 0.0f;
	if (s < n) {
		const uint32_t o = s2o[s];
		float4 p = pos[o];
		const int type = type_ids ? type_ids[o] : 0;
		float4 ref = p;
		if (track.ref_sorted) ref = track.ref_sorted[s];
		// Accumulators of the step that follows, cleared here instead of by
		// separate memsets (one launch less each on short steps).
		if (clear_a) clear_a[s] = make_float4(0.f, 0.f, 0.f, 0.f);
		if (clear_b) clear_b[s] = make_float4(0.f, 0.f, 0.f, 0.f);
		if (odd) {
			if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) atomicAdd(odd, 1ull);
			if (p.x < far_lo.x || p.x > far_hi.x || p.y < far_lo.y || p.y > far_hi.y ||
				p.z < far_lo.z || p.z > far_hi.z)
				odd[1] = 1ull;
		}
		if (track.d2max) d2 = tracked_d2(track, p, ref);
		p.w = __int_as_float(type);
		sorted_pos[s] = p;
	}
	if (track.d2max) {
		raise_track(track, d2, seen, 0xFFFFFFFFu);
	}
}

}  // namespace

void cell_ranges(const uint32_t* keys, uint32_t n, int shift, uint32_t* begin, uint32_t* end,
				 size_t num_cells, cudaStream_t st) {
	MB2_CUDA(cudaMemsetAsync(begin, 0, num_cells * sizeof(uint32_t), st));
	MB2_CUDA(cudaMemsetAsync(end, 0, num_cells * sizeof(uint32_t), st));
	if (n == 0) return;
	MB2_LAUNCH cell_ranges_kernel<<<(n + 255) / 256, 256, 0, st>>>(keys, n, shift, begin, end);
}

void build_walk(const float4* sorted_pos, const uint32_t* keys, const uint32_t* s2o,
				const uint32_t* begin, const uint32_t* end, const StencilEntry* stencil,
				int num_stencil, const WalkGrid& wg, uint32_t n, const Box& box,
				const Exclusions& ex, uint32_t* nbr, uint32_t cap, int hshift, uint32_t* row_len,
				uint32_t* row_back, const unsigned long long* outside, unsigned long long* stats,
				cudaStream_t st) {
	MB2_CUDA(cudaMemsetAsync(stats, 0, 2 * sizeof(unsigned long long), st));
	if (n == 0) return;
	const bool excl = ex.offsets != nullptr || ex.rigid_body_id != nullptr;
	const WalkArrays w{sorted_pos, s2o, begin,  end,    stencil, num_stencil,
					   nbr,        cap, hshift, row_len, row_back};
	const uint32_t rows = walk_rows(n);
	auto kern = excl ? build_walk_kernel<true> : build_walk_kernel<false>;
	MB2_LAUNCH kern<<<(n + 8 * rows - 1) / (8 * rows), 256, 0, st>>>(keys, w, wg, n, box, ex, rows,
																	 outside, stats);
}

void join_back(uint32_t* nbr, const uint32_t* row_len, const uint32_t* row_back, uint32_t n,
			  uint32_t cap, int hshift, cudaStream_t st) {
	if (n == 0) return;
	const uint32_t slices = (n + (1u << hshift) - 1u) >> hshift;
	const uint32_t blocks = (slices + 7u) / 8u;  // 8 warps (slices) per block
	MB2_LAUNCH join_back_kernel<<<blocks, 256, 0, st>>>(nbr, row_len, row_back, n, cap, hshift);
}

void export_pairs(const uint32_t* nbr, const uint32_t* row_len, const uint32_t* row_off,
				  const uint32_t* s2o, uint32_t n, uint32_t cap, int hshift, int2* out,
				  cudaStream_t st) {
	if (n == 0) return;
	MB2_LAUNCH export_kernel<<<(n + 255) / 256, 256, 0, st>>>(nbr, row_len, row_off, s2o, n, cap,
															  hshift, out);
}

void max_displacement_sq(const float4* cur, const float4* prev, uint32_t n, const Box& box,
						 unsigned int* out_bits, cudaStream_t st) {
	MB2_CUDA(cudaMemsetAsync(out_bits, 0, sizeof(unsigned int), st));
	if (n == 0) return;
	const float3 len = make_float3(box.periodic[0] ? box.size[0] : 0.0f,
								   box.periodic[1] ? box.size[1] : 0.0f,
								   box.periodic[2] ? box.size[2] : 0.0f);
	MB2_LAUNCH displacement_kernel<<<(n + 255) / 256, 256, 0, st>>>(cur, prev, n, len, out_bits);
}

DisplacementTrack displacement_track(const Box& box, const float4* ref_sorted,
									 unsigned int* d2max) {
	DisplacementTrack t;
	t.ref_sorted = ref_sorted;
	t.d2max = d2max;
	for (int a = 0; a < 3; ++a) {
		t.len[a] = box.periodic[a] ? box.size[a] : 0.0f;
		t.lo[a] = box.origin[a] - kTrackBand;
		t.hi[a] = box.origin[a] + box.size[a] + kTrackBand;
	}
	return t;
}

void pack_sorted_positions(const float4* pos, const int* type_ids, const uint32_t* s2o,
						   uint32_t n, float4* sorted_pos, cudaStream_t st,
						   unsigned long long* odd, const Box* box, float4* clear_a,
						   float4* clear_b, const DisplacementTrack& track) {
	if (n == 0) return;
	float lo[3] = {-INFINITY, -INFINITY, -INFINITY}, hi[3] = {INFINITY, INFINITY, INFINITY};
	for (int a = 0; odd && a < 3; ++a) {
		if (!box->periodic[a]) continue;
		lo[a] = box->origin[a] - 0.5f * box->size[a];
		hi[a] = box->origin[a] + 1.5f * box->size[a];
	}
	launch_chained(pack_kernel, (n + 255) / 256, 256, 0, st, pos, type_ids, s2o, n, sorted_pos,
				   odd, make_float3(lo[0], lo[1], lo[2]), make_float3(hi[0], hi[1], hi[2]), clear_a,
				   clear_b, track);
}

}  // namespace mb2
