// Z-order (Morton) sort: encode, stable LSD radix sort of (key, index),
// inverse map and gather of sorted positions.
//
// Replaces MortonEncodeKernel / InverseIndexKernel / ReorderDataKernel
// (src/PatchOperation/ZOrderKernels/ZOrderKernels.h:27-83) and the CUB call in
// device_radix_sort_pairs_cub (src/PatchOperation/ZOrderKernels/CUDASort.cu:13-98).
//
// Radix sort layout: four passes of 8 bits, one launch each. All four digit
// histograms come from one read of the keys up front; in a pass each CTA takes
// a tile of consecutive elements (by ticket, so that every earlier tile is
// running or done), ranks it stably (warps in order, a warp's rounds in order,
// lanes in order by __match_any_sync), publishes its digit counts, and adds up
// the counts of the tiles before it, whatever they have published: their own
// counts, or all counts up to theirs ("decoupled look-back", D. Merrill and M.
// Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016).
// Stable per pass, so four passes equal a stable sort on the 32-bit key,
// which is the CUB SortPairs contract the reference relies on. Against a
// histogram, three scan and a scatter launch a pass (each element read twice
// and twenty launches in all), 16,384 to 131,072 elements took 62 us of device
// time and 1,000,003 106 us; now 52 us with its launches at 131,072, 99 us at 1,000,003.
#include <algorithm>
#include <utility>

#include "mb2_internal.cuh"

namespace mb2 {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Elements per thread of a tile: small tiles spread a small array over more
// SMs, large ones shorten the look-back and its publications.
constexpr int kSmallItems = 4;
constexpr int kLargeItems = 16;
constexpr uint32_t kSmallTileMaxN = 1u << 18;

// Look-back word: a tag in the top four bits (2 pass + 1: the tile's own
// count, 2 pass + 2: the count of all tiles up to and including it; anything
// less is an earlier pass's or the zero of the start: nothing yet), the count
// below. So one array, cleared once, serves the four passes.
constexpr int kTagShift = 60;
constexpr unsigned long long kCount = (1ull << kTagShift) - 1ull;

__global__ void __launch_bounds__(256) morton_encode_kernel(const float4* __restrict__ pos,
															uint32_t n, float3 lo, float3 range,
															uint32_t* __restrict__ keys,
															uint32_t* __restrict__ idx) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const float4 p = pos[i];
	const uint32_t x = morton_coord(p.x, lo.x, range.x);
	const uint32_t y = morton_coord(p.y, lo.y, range.y);
	const uint32_t z = morton_coord(p.z, lo.z, range.z);
	keys[i] = split_by3(z) | (split_by3(y) << 1) | (split_by3(x) << 2);
	idx[i] = i;
}

// The digit counts of all four passes, added into hist[4][256].
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const uint32_t* __restrict__ keys,
																  uint32_t n,
																  uint32_t* __restrict__ hist) {
	__shared__ uint32_t counts[4][256];
	for (int p = 0; p < 4; ++p) counts[p][threadIdx.x] = 0;
	__syncthreads();
	for (uint32_t i = blockIdx.x * kSortThreads + threadIdx.x; i < n; i += gridDim.x * kSortThreads) {
		const uint32_t k = keys[i];
#pragma unroll
		for (int p = 0; p < 4; ++p) atomicAdd(&counts[p][(k >> (8 * p)) & 255u], 1u);
	}
	__syncthreads();
	for (int p = 0; p < 4; ++p) {
		const uint32_t c = counts[p][threadIdx.x];
		if (c) atomicAdd(&hist[p * 256 + threadIdx.x], c);
	}
}

// One pass: tile -> its place in the output. hist: this pass's 256 digit
// counts; status[tile][256]: look-back words; ticket: zero at the start. The
// tickets promise that every earlier tile publishes its counts; should they not
// come within max_polls all the same (0: not waited for at all), the tile counts
// the keys before it itself, which takes no other tile: the wait is bounded and
// the result is the sort either way. place_of (the last pass of a sort whose
// values are 0 .. n - 1): place_of[value] = output slot, the inverse of the
// permutation.
template <int kItems>
__global__ void __launch_bounds__(kSortThreads) radix_pass_kernel(
	const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t n,
	int pass, const uint32_t* __restrict__ hist, unsigned long long* status, uint32_t* ticket,
	uint32_t max_polls, uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
	uint32_t* __restrict__ place_of) {
	__shared__ uint32_t warp_count[kSortWarps][256];
	__shared__ uint32_t warp_tot[2][kSortWarps];
	__shared__ uint32_t tile_sh;
	__shared__ uint32_t to_global[256];  // output slot of digit d less its slot in the tile
	__shared__ uint32_t sorted_key[kSortThreads * kItems], sorted_val[kSortThreads * kItems];
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d = threadIdx.x;
	const int shift = 8 * pass;
	const unsigned long long own = 2ull * pass + 1ull, all = own + 1ull;
	if (threadIdx.x == 0) tile_sh = atomicAdd(ticket, 1u);
	for (int w = 0; w < kSortWarps; ++w) warp_count[w][d] = 0;
	__syncthreads();
	const uint32_t tile = tile_sh;
	const uint32_t base = (tile * kSortThreads + warp * 32) * kItems + lane;
	uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
	for (int k = 0; k < kItems; ++k) {
		const uint32_t i = base + k * 32;
		key[k] = i < n ? keys_in[i] : 0xFFFFFFFFu;
		val[k] = i < n ? vals_in[i] : 0u;
	}
	// Rank within the warp's part of the tile. Elements past the end hold the
	// largest key and follow every other, so they move nobody.
#pragma unroll
	for (int k = 0; k < kItems; ++k) {
		const uint32_t digit = (key[k] >> shift) & 255u;
		const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
		const uint32_t before = __popc(peers & ((1u << lane) - 1u));
		const uint32_t c = warp_count[warp][digit];
		__syncwarp();
		if (before == 0) warp_count[warp][digit] = c + __popc(peers);
		__syncwarp();
		rank[k] = c + before;
	}
	__syncthreads();
	// Thread d: the tile's count of digit d, and each warp's place in it.
	uint32_t count = 0;
#pragma unroll
	for (int w = 0; w < kSortWarps; ++w) {
		const uint32_t c = warp_count[w][d];
		warp_count[w][d] = count;
		count += c;
	}
	volatile unsigned long long* row = status + static_cast<size_t>(tile) * 256u + d;
	*row = ((tile == 0 ? all : own) << kTagShift) | count;
	// First output slot of digit d, and its first slot in the tile: exclusive
	// scans of the global and of the tile's counts.
	const uint32_t h = hist[d];
	uint32_t incl = h, tincl = count;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
		const uint32_t tv = __shfl_up_sync(0xFFFFFFFFu, tincl, o);
		if (lane >= o) {
			incl += v;
			tincl += tv;
		}
	}
	if (lane == 31) {
		warp_tot[0][warp] = incl;
		warp_tot[1][warp] = tincl;
	}
	__syncthreads();
	uint32_t first = incl - h, tfirst = tincl - count;
	for (int w = 0; w < warp; ++w) {
		first += warp_tot[0][w];
		tfirst += warp_tot[1][w];
	}
	// The tile in order in shared memory, while the look-back's words arrive.
#pragma unroll
	for (int w = 0; w < kSortWarps; ++w) warp_count[w][d] += tfirst;
	__syncthreads();
#pragma unroll
	for (int k = 0; k < kItems; ++k) {
		const uint32_t slot = warp_count[warp][(key[k] >> shift) & 255u] + rank[k];
		sorted_key[slot] = key[k];
		sorted_val[slot] = val[k];
	}
	// Counts of the tiles before this one, eight words in flight at a time.
	unsigned long long prefix = 0;
	bool alone = false;  // not told within max_polls
	if (tile > 0) {
		constexpr int kBatch = 8;
		int64_t t = static_cast<int64_t>(tile) - 1;
		uint32_t polls = 0;
		bool done = false;
		alone = max_polls == 0u;
		while (!done && !alone) {
			unsigned long long v[kBatch];
#pragma unroll
			for (int q = 0; q < kBatch; ++q)
				v[q] = t - q >= 0 ? *static_cast<volatile unsigned long long*>(
										status + static_cast<size_t>(t - q) * 256u + d)
								  : 0ull;
			int used = 0;
#pragma unroll
			for (int q = 0; q < kBatch; ++q) {
				if (!done && used == q && (v[q] >> kTagShift) >= own) {
					prefix += v[q] & kCount;
					done = (v[q] >> kTagShift) == all;
					used = q + 1;
				}
			}
			t -= used;
			if (!done && used == 0 && ++polls >= max_polls) alone = true;
		}
		if (!alone) *row = (all << kTagShift) | (prefix + count);
	}
	to_global[d] = first + static_cast<uint32_t>(prefix) - tfirst;
	const uint32_t start = tile * (kSortThreads * kItems);
	if (__syncthreads_or(alone)) {
		warp_count[0][d] = 0u;
		__syncthreads();
		for (uint32_t i = threadIdx.x; i < start; i += kSortThreads)
			atomicAdd(&warp_count[0][(keys_in[i] >> shift) & 255u], 1u);
		__syncthreads();
		prefix = warp_count[0][d];
		*row = (all << kTagShift) | (prefix + count);
		to_global[d] = first + static_cast<uint32_t>(prefix) - tfirst;
		__syncthreads();
	}
	// Written in tile order, so that a digit's elements are neighbouring stores.
	const uint32_t here = min(static_cast<uint32_t>(kSortThreads * kItems), n - start);
#pragma unroll
	for (int k = 0; k < kItems; ++k) {
		const uint32_t slot = k * kSortThreads + threadIdx.x;
		if (slot < here) {
			const uint32_t out_key = sorted_key[slot];
			const uint32_t dst = to_global[(out_key >> shift) & 255u] + slot;
			const uint32_t out_val = sorted_val[slot];
			keys_out[dst] = out_key;
			vals_out[dst] = out_val;
			if (place_of) place_of[out_val] = dst;
		}
	}
}

// out[s] = in[s2o[s]] for 4- or 16-byte elements (DeviceParticle::permute).
template <typename T>
__global__ void __launch_bounds__(256) permute_kernel(const T* __restrict__ in,
													  const uint32_t* __restrict__ s2o, uint32_t n,
													  T* __restrict__ out) {
	const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
	if (s < n) out[s] = in[s2o[s]];
}

// RemapIndicesKernel (ZOrderKernels.h:87-101): in-range indices go through inv.
__global__ void __launch_bounds__(256) remap_kernel(int* __restrict__ idx, size_t count,
													const uint32_t* __restrict__ inv, uint32_t n) {
	const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
	if (i >= count) return;
	const int v = idx[i];
	if (v >= 0 && static_cast<uint32_t>(v) < n) idx[i] = static_cast<int>(inv[v]);
}

}  // namespace

namespace {

// Up to this many pairs the sort counts, for every element, the elements that
// precede it: n^2 comparisons spread over the whole GPU (64 M of them at 8,192
// pairs) in one launch, where the passes above would be six launches of a few
// CTAs. With the copy back 13.3 us at 1,000 pairs, 19.5 at 4,096 and 33.8 at
// 8,192, where the passes take 33.8 (35 at 16,384): above it the squares win.
constexpr uint32_t kRankSortMax = 8192;

// Stable rank of 32 elements a CTA, lane = element; each of the CTA's warps
// compares them with an eighth of the keys, which all lanes read together
// (four keys a shared-memory load, broadcast). Bound by issuing the
// comparisons: 8.9 us at 4,096 pairs.
__global__ void __launch_bounds__(256) rank_sort_kernel(const uint32_t* __restrict__ keys,
														const uint32_t* __restrict__ vals,
														uint32_t n, uint32_t* __restrict__ keys_out,
														uint32_t* __restrict__ vals_out) {
	extern __shared__ uint4 keys4[];
	__shared__ uint32_t part[8][32];
	uint32_t* sk = reinterpret_cast<uint32_t*>(keys4);
	const uint32_t quads = (n + 3u) / 4u;
	for (uint32_t i = threadIdx.x; i < quads * 4u; i += blockDim.x) sk[i] = i < n ? keys[i] : 0xFFFFFFFFu;
	__syncthreads();
	const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
	const uint32_t first = blockIdx.x * 32u, i = first + lane;
	const uint32_t key = i < n ? sk[i] : 0u;
	// Keys before the CTA's elements precede on a tie, keys after them do not;
	// among the 32 themselves the position decides.
	const uint32_t q0 = first / 4u, q1 = min(q0 + 8u, quads);
	uint32_t rank = 0;
	for (uint32_t q = warp; q < q0; q += 8u) {
		const uint4 k = keys4[q];
		rank += (k.x <= key) + (k.y <= key) + (k.z <= key) + (k.w <= key);
	}
	for (uint32_t q = q1 + warp; q < quads; q += 8u) {
		const uint4 k = keys4[q];
		rank += (k.x < key) + (k.y < key) + (k.z < key) + (k.w < key);
	}
	for (uint32_t q = q0 + warp; q < q1; q += 8u)
		for (uint32_t c = 4u * q; c < 4u * q + 4u; ++c)
			if (c < n) rank += sk[c] < key || (sk[c] == key && c < i);
	part[warp][lane] = rank;
	__syncthreads();
	if (warp == 0 && i < n) {
#pragma unroll
		for (int w = 1; w < 8; ++w) rank += part[w][lane];
		keys_out[rank] = key;
		vals_out[rank] = vals[i];
	}
}

// The sorted pairs back into the caller's arrays.
__global__ void __launch_bounds__(256) copy_pairs_kernel(const uint32_t* __restrict__ keys_in,
														 const uint32_t* __restrict__ vals_in,
														 uint32_t n, uint32_t* __restrict__ keys,
														 uint32_t* __restrict__ vals,
														 uint32_t* __restrict__ place_of) {
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint32_t v = vals_in[i];
	keys[i] = keys_in[i];
	vals[i] = v;
	if (place_of) place_of[v] = i;
}

uint32_t sort_tiles(uint32_t n) {
	const uint32_t tile = kSortThreads * (n <= kSmallTileMaxN ? kSmallItems : kLargeItems);
	return (n + tile - 1) / tile;
}

// Words before the look-back rows: the four histograms, a ticket for each
// pass.
constexpr size_t kSortHeadWords = 4 * 256 + 8;

}  // namespace

size_t sort_work_words(uint32_t n) {
	if (n <= kRankSortMax) return 0;
	return kSortHeadWords + static_cast<size_t>(sort_tiles(n)) * 256u * 2u;
}

void radix_sort_pairs_into(uint32_t* keys, uint32_t* vals, uint32_t n, uint32_t* keys_alt,
						   uint32_t* vals_alt, uint32_t* work, cudaStream_t st, uint32_t* place_of,
						   uint32_t max_polls) {
	if (n == 0) return;
	if (n == 1) {
		if (place_of) MB2_CUDA(cudaMemsetAsync(place_of, 0, sizeof(uint32_t), st));
		return;
	}
	if (n <= kRankSortMax) {
		const size_t smem = static_cast<size_t>((n + 3u) / 4u) * sizeof(uint4);
		MB2_LAUNCH rank_sort_kernel<<<(n + 31) / 32, 256, smem, st>>>(keys, vals, n, keys_alt,
																	  vals_alt);
		MB2_LAUNCH copy_pairs_kernel<<<(n + 255) / 256, 256, 0, st>>>(keys_alt, vals_alt, n, keys,
																	  vals, place_of);
		return;
	}
	const uint32_t tiles = sort_tiles(n);
	uint32_t* tickets = work + 4 * 256;
	unsigned long long* status = reinterpret_cast<unsigned long long*>(work + kSortHeadWords);
	MB2_CUDA(cudaMemsetAsync(work, 0, sort_work_words(n) * sizeof(uint32_t), st));
	MB2_LAUNCH radix_hist_kernel<<<std::min(tiles, 592u), kSortThreads, 0, st>>>(keys, n, work);
	uint32_t *ks = keys, *vs = vals, *kd = keys_alt, *vd = vals_alt;
	auto pass_kernel = n <= kSmallTileMaxN ? radix_pass_kernel<kSmallItems>
										   : radix_pass_kernel<kLargeItems>;
	for (int pass = 0; pass < 4; ++pass) {
		MB2_LAUNCH pass_kernel<<<tiles, kSortThreads, 0, st>>>(
			ks, vs, n, pass, work + 256 * pass, status, tickets + pass, max_polls, kd, vd,
			pass == 3 ? place_of : nullptr);
		std::swap(ks, kd);
		std::swap(vs, vd);
	}
	// Four passes: the sorted data is back in the caller's buffers.
}

void radix_sort_pairs(Scratch& s, uint32_t* keys, uint32_t* vals, uint32_t n, cudaStream_t st,
					  uint32_t* place_of, uint32_t max_polls) {
	if (n == 0) return;
	s.ensure_sort(n, sort_work_words(n));
	radix_sort_pairs_into(keys, vals, n, s.keys_alt.ptr, s.vals_alt.ptr, s.work.ptr, st, place_of,
						  max_polls);
}

void morton_encode(const float4* pos, uint32_t n, const float* bmin, const float* bmax,
				   uint32_t* keys, uint32_t* idx, cudaStream_t st) {
	float3 lo = make_float3(bmin[0], bmin[1], bmin[2]);
	// range = fmaxf(box_max - box_min, 1e-6f), per axis, in float (MortonCode.h:97-109)
	float3 range = make_float3(fmaxf(bmax[0] - bmin[0], 1e-6f), fmaxf(bmax[1] - bmin[1], 1e-6f),
							   fmaxf(bmax[2] - bmin[2], 1e-6f));
	if (n == 0) return;
	MB2_LAUNCH morton_encode_kernel<<<(n + 255) / 256, 256, 0, st>>>(pos, n, lo, range, keys, idx);
}

void permute_gather(const void* in, const uint32_t* s2o, uint32_t n, int elem_bytes, void* out,
					cudaStream_t st) {
	if (n == 0) return;
	if (elem_bytes == 16)
		MB2_LAUNCH permute_kernel<float4><<<(n + 255) / 256, 256, 0, st>>>(
			static_cast<const float4*>(in), s2o, n, static_cast<float4*>(out));
	else
		MB2_LAUNCH permute_kernel<uint32_t><<<(n + 255) / 256, 256, 0, st>>>(
			static_cast<const uint32_t*>(in), s2o, n, static_cast<uint32_t*>(out));
}

void remap_indices(int* idx, size_t count, const uint32_t* inv, uint32_t n, cudaStream_t st) {
	if (count == 0) return;
	MB2_LAUNCH remap_kernel<<<static_cast<unsigned>((count + 255) / 256), 256, 0, st>>>(idx, count,
																						inv, n);
}

}  // namespace mb2
