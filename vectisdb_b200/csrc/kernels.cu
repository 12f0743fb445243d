// kernels.cu -- precompiled device primitives (see kernels.hpp).
#include "kernels.hpp"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <type_traits>

#include <utility>

#include "device_lib.cuh"

namespace vgpu {
namespace kern {

using namespace vgpu_dev;

namespace {

constexpr int kScanBlock = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanBlock * kScanItems;

unsigned GridFor(uint64_t n, int block) {
	uint64_t g = (n + block - 1) / block;
	if (g == 0) {
		g = 1;
	}
	const uint64_t cap = static_cast<uint64_t>(Runtime::Get().props().sm_count) * 32;
	return static_cast<unsigned>(g < cap ? g : cap);
}

template <typename T> __device__ __forceinline__ T BlockScanExclusive(T v, T *scratch /*33*/, T *total) {
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5;
	const int nwarps = blockDim.x >> 5;
	T x = v;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		T y = __shfl_up_sync(0xffffffffu, x, o);
		if (lane >= o) x += y;
	}
	if (lane == 31) scratch[warp] = x;
	__syncthreads();
	if (warp == 0) {
		T w = (lane < nwarps) ? scratch[lane] : T(0);
		T s = w;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			T y = __shfl_up_sync(0xffffffffu, s, o);
			if (lane >= o) s += y;
		}
		if (lane < nwarps) scratch[lane] = s - w;
		if (lane == 31) scratch[32] = s;
	}
	__syncthreads();
	T r = scratch[warp] + x - v;
	*total = scratch[32];
	__syncthreads();
	return r;
}

template <typename T> __global__ void __launch_bounds__(kScanBlock) ScanTileSums(const T *in, uint64_t n, T *sums) {
	__shared__ T scratch[33];
	const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile + static_cast<uint64_t>(threadIdx.x) * kScanItems;
	T local = 0;
#pragma unroll
	for (int i = 0; i < kScanItems; i++) {
		if (base + i < n) local += in[base + i];
	}
	T total;
	BlockScanExclusive<T>(local, scratch, &total);
	if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Single CTA: exclusive scan of the tile sums in place, grand total to *total.
template <typename T> __global__ void __launch_bounds__(1024) ScanSums(T *sums, uint64_t count, T *total) {
	__shared__ T scratch[33];
	T carry = 0;
	for (uint64_t c0 = 0; c0 < count; c0 += blockDim.x) {
		const uint64_t i = c0 + threadIdx.x;
		T v = i < count ? sums[i] : T(0);
		T chunk_total;
		T ex = BlockScanExclusive<T>(v, scratch, &chunk_total);
		if (i < count) sums[i] = carry + ex;
		carry += chunk_total;
	}
	if (threadIdx.x == 0 && total) *total = carry;
}

template <typename T>
__global__ void __launch_bounds__(kScanBlock) ScanApply(const T *in, T *out, uint64_t n, const T *sums) {
	__shared__ T scratch[33];
	const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kScanTile + static_cast<uint64_t>(threadIdx.x) * kScanItems;
	T vals[kScanItems];
	T local = 0;
#pragma unroll
	for (int i = 0; i < kScanItems; i++) {
		vals[i] = base + i < n ? in[base + i] : T(0);
		local += vals[i];
	}
	T total;
	T run = BlockScanExclusive<T>(local, scratch, &total) + sums[blockIdx.x];
#pragma unroll
	for (int i = 0; i < kScanItems; i++) {
		if (base + i < n) out[base + i] = run;
		run += vals[i];
	}
}

// Values one CTA scans in one launch (16 per thread): the tile counts of a materialization of up to
// 2^24 rows. The three-launch form costs more in launches than in work at these sizes.
constexpr int kSmallScanItems = 16;
constexpr uint64_t kSmallScanMax = 1024 * kSmallScanItems;

// Single CTA, in place allowed: each thread loads a run of up to 16 consecutive values at once (all
// loads issued before any is used), the block scans the run sums, then each thread writes its run's
// exclusive prefixes from registers (every read precedes the block scan's barrier, every write follows).
template <typename T> __global__ void __launch_bounds__(1024) ScanSmall(const T *in, T *out, uint64_t n, T *total) {
	__shared__ T scratch[33];
	const uint64_t per = (n + blockDim.x - 1) / blockDim.x;
	const uint64_t b = static_cast<uint64_t>(threadIdx.x) * per;
	T vals[kSmallScanItems];
	T local = 0;
#pragma unroll
	for (int k = 0; k < kSmallScanItems; k++) {
		const uint64_t i = b + k;
		vals[k] = (static_cast<uint64_t>(k) < per && i < n) ? in[i] : T(0);
		local += vals[k];
	}
	T all;
	T run = BlockScanExclusive<T>(local, scratch, &all);
#pragma unroll
	for (int k = 0; k < kSmallScanItems; k++) {
		const uint64_t i = b + k;
		if (static_cast<uint64_t>(k) < per && i < n) {
			out[i] = run;
			run += vals[k];
		}
	}
	if (threadIdx.x == 0 && total) *total = all;
}

template <typename T> void ExclusiveScan(const T *in, T *out, uint64_t n, T *total, Arena &arena) {
	cudaStream_t s = arena.stream();
	if (n <= kSmallScanMax) {
		LaunchScope scope("scan_small", s, 2 * n * sizeof(T), n);
		ScanSmall<T><<<1, 1024, 0, s>>>(in, out, n, total);
		VGPU_CUDA(cudaGetLastError());
		return;
	}
	const uint64_t tiles = n == 0 ? 1 : (n + kScanTile - 1) / kScanTile;
	T *sums = arena.AllocT<T>(tiles);
	{
		LaunchScope scope("scan_tiles", s, n * sizeof(T), n);
		ScanTileSums<T><<<static_cast<unsigned>(tiles), kScanBlock, 0, s>>>(in, n, sums);
	}
	{
		LaunchScope scope("scan_sums", s, tiles * sizeof(T), tiles);
		ScanSums<T><<<1, 1024, 0, s>>>(sums, tiles, total);
	}
	if (n > 0) {
		LaunchScope scope("scan_apply", s, 2 * n * sizeof(T), n);
		ScanApply<T><<<static_cast<unsigned>(tiles), kScanBlock, 0, s>>>(in, out, n, sums);
	}
	VGPU_CUDA(cudaGetLastError());
}

__global__ void UnpackValidityKernel(const uint8_t *bitmap, uint8_t *bytes, uint64_t n) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		bytes[i] = (bitmap[i >> 3] >> (i & 7)) & 1u;
	}
}

__global__ void PackValidityKernel(const uint8_t *bytes, uint8_t *bitmap, uint64_t n) {
	const uint64_t nbytes = (n + 7) / 8;
	for (uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b < nbytes; b += (uint64_t)gridDim.x * blockDim.x) {
		uint8_t v = 0;
		for (int k = 0; k < 8; k++) {
			uint64_t i = b * 8 + k;
			if (i < n && bytes[i]) v |= static_cast<uint8_t>(1u << k);
		}
		bitmap[b] = v;
	}
}

template <typename T> __global__ void GatherKernel(const T *src, const uint32_t *idx, uint64_t n, T *dst) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		dst[i] = src[idx[i]];
	}
}

struct CopyArgs {
	BufferCopy c[kMaxCopies];
};

// blockIdx.y picks the buffer. Bound by the bytes; one launch, since a few kilobytes are copied as often as not.
__global__ void __launch_bounds__(256) CopyBuffersKernel(CopyArgs a) {
	const BufferCopy &c = a.c[blockIdx.y];
	const uint64_t vecs = (c.bytes + 15) / 16, stride = (uint64_t)gridDim.x * blockDim.x;
	const uint4 *src = static_cast<const uint4 *>(c.src);
	uint4 *dst = static_cast<uint4 *>(c.dst);
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < vecs; i += stride) dst[i] = src[i];
}

// Key bits zero-extended to 64 bits, minus `bias`.
template <typename T> __global__ void WidenKernel(const T *src, uint64_t n, uint64_t bias, uint64_t *dst) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		dst[i] = static_cast<uint64_t>(src[i]) - bias;
	}
}

// ---- value ranges of columns ------------------------------------------------------------------------
//
// One launch for up to kMaxBoundsColumns columns (blockIdx.y picks the column), bound by reading them
// once: 16-byte loads, four in flight per thread, one atomic pair per CTA (a pair per warp serializes on
// the two words once thousands of warps reach them: a 10M-row INT32 key column 28 -> 19 us; 2^24 INT64
// keys and their INT32 values 0.095 ms in two kernels, one of them writing the keys widened, -> 0.046 ms,
// 4.4 TB/s). Values travel as an order-preserving
// unsigned image (signed values with the sign bit flipped); the minimum is kept as the maximum of the
// complemented image, so one zero fill is the identity of both.

//
// With `ranks`, also an estimate of each column's distinct values (HyperLogLog: of the hashes that share their
// low 8 bits, the most leading zeros in the rest) over one value in 1024, as a cheap hash picks them: a
// multiplication per value, and the rest for one warp step in thirty (8M INT64 values 0.028 -> 0.029 ms; every value
// taken, or one in eight, which is nearly every step of a warp: 0.041 ms).
constexpr int kDistinctShift = 10;

struct BoundsArgs {
	BoundsColumn c[kMaxBoundsColumns];
	unsigned long long *out;
	unsigned int *ranks;  // kDistinctRanks per column, or null
	unsigned long long *pairs;  // two words per column, or null
};

// Out of line: few values come here, and the kernel's eight unrolled readers stay small.
__device__ __noinline__ void NoteValue(u64 v, uint32_t *ranks) {
	const u64 h = mix64(v);
	const uint32_t rank = static_cast<uint32_t>(__clzll(static_cast<long long>(h | (kDistinctRanks - 1)))) + 1u;
	uint32_t *r = ranks + (h & (kDistinctRanks - 1));
	if (*reinterpret_cast<volatile uint32_t *>(r) < rank) atomicMax(r, rank);
}

template <typename T, bool kBool, bool kPairs>
__device__ __forceinline__ void RangeOf(const T *p, uint64_t n, T &mn, T &mx, uint32_t *ranks, uint2 &seen) {
	auto take = [&](T v) {
		if constexpr (kBool) v = v != 0 ? 1 : 0;
		mn = v < mn ? v : mn;
		mx = v > mx ? v : mx;
		if constexpr (sizeof(T) >= 4 && !kPairs) {
			u32 w = static_cast<u32>(v);
			if constexpr (sizeof(T) == 8) w ^= static_cast<u32>(static_cast<u64>(v) >> 32);
			if (w * 0x9e3779b1u < (1u << (32 - kDistinctShift)) && ranks) NoteValue(static_cast<u64>(v), ranks);
		}
	};
	constexpr uint64_t kPer = 16 / sizeof(T);
	const uint64_t skew = reinterpret_cast<uintptr_t>(p) & 15u;
	uint64_t head = skew ? (16 - skew) / sizeof(T) : 0;  // values before the first 16-byte boundary
	if (head > n) head = n;
	const uint64_t vecs = (n - head) / kPer;
	const uint64_t tail = head + vecs * kPer;
	const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
	if (tid < head) take(p[tid]);
	if (tid < n - tail) take(p[tail + tid]);  // both ends are shorter than a warp
	const uint4 *v = reinterpret_cast<const uint4 *>(p + head);
	auto take4 = [&](const uint4 &q) {
		T x[kPer];
		memcpy(x, &q, 16);
#pragma unroll
		for (uint64_t j = 0; j < kPer; j++) take(x[j]);
	};
	uint64_t i = tid;
	for (; i + 3 * stride < vecs; i += 4 * stride) {
		const uint4 a = v[i], b = v[i + stride], c = v[i + 2 * stride], d = v[i + 3 * stride];
		take4(a);
		take4(b);
		take4(c);
		take4(d);
		if constexpr (kPairs) {
			T x[kPer], y[kPer], z[kPer], w[kPer];
			memcpy(x, &a, 16);
			memcpy(y, &b, 16);
			memcpy(z, &c, 16);
			memcpy(w, &d, 16);
#pragma unroll
			for (uint64_t j = 0; j < kPer; j++) seen.x += (x[j] == y[j] ? 1u : 0u) + (z[j] == w[j] ? 1u : 0u);
			seen.y += 2 * kPer;
		}
	}
	for (; i < vecs; i += stride) take4(v[i]);
}

template <typename T, bool kPairs, bool kBool = false>
__device__ __forceinline__ void RangeImage(const void *p, uint64_t n, unsigned long long &lo, unsigned long long &hi,
                                           uint32_t *ranks, uint2 &seen) {
	T mn = std::numeric_limits<T>::max(), mx = std::numeric_limits<T>::lowest();
	RangeOf<T, kBool, kPairs>(static_cast<const T *>(p), n, mn, mx, ranks, seen);
	constexpr unsigned long long kFlip = std::is_signed<T>::value ? 1ull << 63 : 0ull;
	const bool any = mn <= mx;  // a thread without values leaves the identity
	lo = any ? static_cast<unsigned long long>(mn) ^ kFlip : ~0ull;
	hi = any ? static_cast<unsigned long long>(mx) ^ kFlip : 0ull;
}

constexpr int kBoundsBlock = 256;

template <bool kPairs> __global__ void __launch_bounds__(kBoundsBlock) ColumnBoundsKernel(BoundsArgs a) {
	const BoundsColumn &c = a.c[blockIdx.y];
	unsigned long long lo = ~0ull, hi = 0ull;
	__shared__ uint32_t shared_ranks[kDistinctRanks];
	static_assert(kDistinctRanks == kBoundsBlock, "one rank per thread");
	shared_ranks[threadIdx.x] = 0;
	uint32_t *ranks = a.ranks ? shared_ranks : nullptr;
	uint2 seen = make_uint2(0, 0);  // equal pairs, pairs
	__syncthreads();
	switch (c.kind) {
	case BoundsKind::U8: RangeImage<uint8_t, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::U16: RangeImage<uint16_t, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::U32: RangeImage<uint32_t, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::U64: RangeImage<unsigned long long, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::I16: RangeImage<int16_t, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::I32: RangeImage<int32_t, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::I64: RangeImage<long long, kPairs>(c.data, c.rows, lo, hi, ranks, seen); break;
	case BoundsKind::BOOL: RangeImage<uint8_t, kPairs, true>(c.data, c.rows, lo, hi, ranks, seen); break;
	}
	__shared__ unsigned long long slo[kBoundsBlock / 32], shi[kBoundsBlock / 32];
	for (int o = 16; o > 0; o >>= 1) {
		const unsigned long long x = __shfl_xor_sync(0xffffffffu, lo, o), y = __shfl_xor_sync(0xffffffffu, hi, o);
		lo = x < lo ? x : lo;
		hi = y > hi ? y : hi;
	}
	__shared__ uint2 sseen[kBoundsBlock / 32];
	if constexpr (kPairs) {
		seen.x = __reduce_add_sync(0xffffffffu, seen.x);
		seen.y = __reduce_add_sync(0xffffffffu, seen.y);
	}
	if ((threadIdx.x & 31) == 0) {
		slo[threadIdx.x >> 5] = lo;
		shi[threadIdx.x >> 5] = hi;
		sseen[threadIdx.x >> 5] = seen;
	}
	__syncthreads();
	if (kPairs && threadIdx.x == 32) {
		unsigned long long equal = 0, all = 0;
		for (int w = 0; w < kBoundsBlock / 32; w++) {
			equal += sseen[w].x;
			all += sseen[w].y;
		}
		if (equal) atomicAdd(a.pairs + 2 * blockIdx.y, equal);
		if (all) atomicAdd(a.pairs + 2 * blockIdx.y + 1, all);
	}
	if (threadIdx.x == 0) {
		for (int w = 1; w < kBoundsBlock / 32; w++) {
			lo = slo[w] < lo ? slo[w] : lo;
			hi = shi[w] > hi ? shi[w] : hi;
		}
		atomicMax(a.out + 2 * blockIdx.y, ~lo);
		atomicMax(a.out + 2 * blockIdx.y + 1, hi);
	}
	if (!kPairs && a.ranks) {  // (the values were all taken before the barrier above)
		// few CTAs raise a rank the others have raised before: looked at first (a thousand CTAs' atomics on the
		// same eight lines took 20 us)
		unsigned int *to = a.ranks + blockIdx.y * kDistinctRanks + threadIdx.x;
		const uint32_t r = shared_ranks[threadIdx.x];
		if (r != 0 && r > __ldcg(to)) atomicMax(to, r);
	}
}

__global__ void IotaKernel(uint32_t *out, uint64_t n) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		out[i] = static_cast<uint32_t>(i);
	}
}

// ---- LSD radix sort: 8-bit digits, stable warp-ordered local ranking ----------------------------

constexpr int kSortBlock = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortBlock * kSortItems;
constexpr int kSortWarps = kSortBlock / 32;

__device__ __forceinline__ uint32_t LaneMaskLt() {
	uint32_t m;
	asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
	return m;
}

__global__ void __launch_bounds__(kSortBlock) RadixHistKernel(const uint64_t *keys, uint64_t n, int shift,
                                                              uint32_t *hist, uint32_t ntiles) {
	__shared__ uint32_t counts[256];
	for (int i = threadIdx.x; i < 256; i += kSortBlock) counts[i] = 0;
	__syncthreads();
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const uint64_t base = static_cast<uint64_t>(blockIdx.x) * kSortTile + static_cast<uint64_t>(warp) * 32 * kSortItems;
#pragma unroll 4
	for (int k = 0; k < kSortItems; k++) {
		const uint64_t idx = base + static_cast<uint64_t>(k) * 32 + lane;
		const bool valid = idx < n;
		const uint32_t active = __ballot_sync(0xffffffffu, valid);
		if (valid) {
			const uint32_t d = static_cast<uint32_t>(keys[idx] >> shift) & 255u;
			const uint32_t peers = __match_any_sync(active, d);
			if ((peers & LaneMaskLt()) == 0) atomicAdd(&counts[d], static_cast<uint32_t>(__popc(peers)));
		}
	}
	__syncthreads();
	for (int d = threadIdx.x; d < 256; d += kSortBlock) hist[static_cast<uint64_t>(d) * ntiles + blockIdx.x] = counts[d];
}

// Scatter of one pass: the tile's keys are ranked stably (warp-ordered: a warp's items in order, warps
// in order), placed in shared memory in digit order, then written out by consecutive threads to
// consecutive positions of each digit's run, so the global stores are coalesced runs instead of one
// scattered store per key.
__global__ void __launch_bounds__(kSortBlock) RadixScatterKernel(const uint64_t *kin, const uint32_t *vin,
                                                                 uint64_t *kout, uint32_t *vout, uint64_t n, int shift,
                                                                 const uint32_t *offsets, uint32_t ntiles) {
	__shared__ uint32_t wcount[kSortWarps][256];
	__shared__ uint32_t tile_start[256];  // first local position of each digit in the tile
	__shared__ uint32_t global_start[256];
	__shared__ uint64_t skeys[kSortTile];  // the tile in digit order: keys, then (reused) values
	__shared__ uint8_t sdig[kSortTile];
	for (int i = threadIdx.x; i < kSortWarps * 256; i += kSortBlock) (&wcount[0][0])[i] = 0;
	__syncthreads();
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const uint64_t tile0 = static_cast<uint64_t>(blockIdx.x) * kSortTile;
	const uint64_t base = tile0 + static_cast<uint64_t>(warp) * 32 * kSortItems;
	uint64_t keys[kSortItems];
	uint32_t vals[kSortItems];
	uint32_t rank[kSortItems];
#pragma unroll
	for (int k = 0; k < kSortItems; k++) {
		const uint64_t idx = base + static_cast<uint64_t>(k) * 32 + lane;
		const bool valid = idx < n;
		keys[k] = valid ? kin[idx] : 0ull;
		vals[k] = !valid ? 0u : vin ? vin[idx] : static_cast<uint32_t>(idx);
	}
#pragma unroll
	for (int k = 0; k < kSortItems; k++) {
		const uint64_t idx = base + static_cast<uint64_t>(k) * 32 + lane;
		const bool valid = idx < n;
		const uint32_t active = __ballot_sync(0xffffffffu, valid);
		uint32_t peers = 0, d = 0;
		if (valid) {
			d = static_cast<uint32_t>(keys[k] >> shift) & 255u;
			peers = __match_any_sync(active, d);
			rank[k] = wcount[warp][d] + static_cast<uint32_t>(__popc(peers & LaneMaskLt()));
		}
		__syncwarp();
		if (valid && (peers & LaneMaskLt()) == 0) wcount[warp][d] += static_cast<uint32_t>(__popc(peers));
		__syncwarp();
	}
	__syncthreads();
	if (threadIdx.x < 256) {  // per digit: warps' starts within the digit, the digit's count in the tile
		uint32_t run = 0;
		for (int w = 0; w < kSortWarps; w++) {
			const uint32_t c = wcount[w][threadIdx.x];
			wcount[w][threadIdx.x] = run;
			run += c;
		}
		tile_start[threadIdx.x] = run;  // the count, turned into a start below
		global_start[threadIdx.x] = offsets[static_cast<uint64_t>(threadIdx.x) * ntiles + blockIdx.x];
	}
	__syncthreads();
	if (threadIdx.x < 32) {  // exclusive scan of the 256 digit counts by one warp (8 per lane)
		uint32_t c[8], sum = 0;
#pragma unroll
		for (int j = 0; j < 8; j++) {
			c[j] = tile_start[threadIdx.x * 8 + j];
			sum += c[j];
		}
		uint32_t incl = sum;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
			if (lane >= o) incl += y;
		}
		uint32_t run = incl - sum;
#pragma unroll
		for (int j = 0; j < 8; j++) {
			tile_start[threadIdx.x * 8 + j] = run;
			run += c[j];
		}
	}
	__syncthreads();
	uint32_t lpos[kSortItems];
#pragma unroll
	for (int k = 0; k < kSortItems; k++) {
		const uint64_t idx = base + static_cast<uint64_t>(k) * 32 + lane;
		if (idx < n) {
			const uint32_t d = static_cast<uint32_t>(keys[k] >> shift) & 255u;
			lpos[k] = tile_start[d] + wcount[warp][d] + rank[k];
			skeys[lpos[k]] = keys[k];
			sdig[lpos[k]] = static_cast<uint8_t>(d);
		}
	}
	__syncthreads();
	const uint32_t valid_rows = static_cast<uint32_t>(n - tile0 < kSortTile ? n - tile0 : kSortTile);
	for (uint32_t i = threadIdx.x; i < valid_rows; i += kSortBlock) {
		const uint32_t d = sdig[i];
		kout[global_start[d] + (i - tile_start[d])] = skeys[i];
	}
	__syncthreads();
	uint32_t *svals = reinterpret_cast<uint32_t *>(skeys);
#pragma unroll
	for (int k = 0; k < kSortItems; k++) {
		const uint64_t idx = base + static_cast<uint64_t>(k) * 32 + lane;
		if (idx < n) svals[lpos[k]] = vals[k];
	}
	__syncthreads();
	for (uint32_t i = threadIdx.x; i < valid_rows; i += kSortBlock) {
		const uint32_t d = sdig[i];
		vout[global_start[d] + (i - tile_start[d])] = svals[i];
	}
}

// ---- join -----------------------------------------------------------------------------------------

// Load-balanced expansion of the match pairs (a merge path over the left rows' output offsets): each
// CTA owns a fixed tile of output positions, finds once which left rows those positions span, stages
// those rows' offsets in shared memory (when they fit) and every thread places its outputs by a search
// there; writes are coalesced across the tile. Left rows with no match share an offset with the next
// row, so "last row whose offset <= o" skips them.
constexpr int kExpandBlock = 256;
constexpr int kExpandItems = 8;
constexpr int kExpandTile = kExpandBlock * kExpandItems;
constexpr int kExpandWindow = 4096;

__device__ __forceinline__ uint64_t LastAtMost(const uint64_t *offsets, uint64_t a, uint64_t b, uint64_t o) {
	// offsets[a] <= o; returns the last index in [a, b) with offsets[index] <= o
	uint64_t lo = a + 1, hi = b;
	while (lo < hi) {
		const uint64_t mid = (lo + hi) >> 1;
		if (offsets[mid] <= o) lo = mid + 1;
		else hi = mid;
	}
	return lo - 1;
}

__global__ void __launch_bounds__(kExpandBlock) JoinExpandKernel(const uint64_t *offsets, const uint64_t *lower,
                                                                 uint64_t n_left, const uint32_t *sorted_perm,
                                                                 uint64_t total, uint32_t *out_left, uint32_t *out_right) {
	__shared__ uint64_t s_off[kExpandWindow];
	__shared__ uint64_t s_first, s_end;
	for (uint64_t tile = blockIdx.x; tile * kExpandTile < total; tile += gridDim.x) {
		const uint64_t o_begin = tile * kExpandTile;
		const uint64_t o_last = o_begin + kExpandTile < total ? o_begin + kExpandTile - 1 : total - 1;
		if (threadIdx.x == 0) {
			const uint64_t first = LastAtMost(offsets, 0, n_left, o_begin);
			s_first = first;
			s_end = LastAtMost(offsets, first, n_left, o_last) + 1;
		}
		__syncthreads();
		const uint64_t first = s_first, end = s_end, window = end - first;
		const bool staged = window <= kExpandWindow;
		if (staged) {
			for (uint64_t r = threadIdx.x; r < window; r += kExpandBlock) s_off[r] = offsets[first + r];
		}
		__syncthreads();
		for (int t = 0; t < kExpandItems; ++t) {
			const uint64_t o = o_begin + static_cast<uint64_t>(t) * kExpandBlock + threadIdx.x;
			if (o > o_last) break;
			uint64_t i;
			if (staged) {
				uint32_t lo = 1, hi = static_cast<uint32_t>(window);
				while (lo < hi) {
					const uint32_t mid = (lo + hi) >> 1;
					if (s_off[mid] <= o) lo = mid + 1;
					else hi = mid;
				}
				i = first + lo - 1;
			} else {
				i = LastAtMost(offsets, first, end, o);
			}
			const uint64_t j = o - (staged ? s_off[i - first] : offsets[i]);
			out_left[o] = static_cast<uint32_t>(i);
			out_right[o] = sorted_perm[lower[i] + j];
		}
		__syncthreads();
	}
}

// ---- materializing join over short runs ---------------------------------------------------------------
//
// The right rows of each key, contiguous and in row order, then two passes over the left rows: one counts the
// matches of each tile (the starts of the tiles in the same launch, see tile_scanner), one writes every output
// column of the tile's matches, consecutive threads writing consecutive output rows. No pair of row numbers,
// no per-row offset and no sorted key is written: 4M left rows against 1M right ones with 7.3M matches, three
// columns out, 0.574 ms of kernels by sorting, offsets, expansion and a gather per column, 0.221 ms here (the emit pass, bound
// by random reads of 8-byte right values, 0.113 ms; 0.088 with the values in run order, see the caller).

// info of the kernels below: [0] runs listed for the last of them, [1] the longest run, [2] the cursor of the runs'
// places; zero at the first launch. A run past kJoinRunLimit makes the result useless: from then on they return.
// (Read through L1: a load of that one word past it from every warp took as long as the rest of such a pass.)
__device__ __forceinline__ bool JoinRunTooLong(const uint32_t *info) { return __ldg(info + 1) > kJoinRunLimit; }

// Dense keys: an entry per key value, x = end of its run in `rows`, y = its length. Adds to one entry queue at its
// address (0.7 ns each: a key in every second of 4M rows held this kernel for 1.4 ms), so a warp with equal
// neighbours adds each of its keys once and looks at the counts it meets: the pass ends soon after one is too long.
template <typename K>
__global__ void JoinEntryCountKernel(const K *keys, uint64_t n, uint64_t bias, uint2 *entries, uint32_t *info) {
	const uint32_t lane = threadIdx.x & 31;
	for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
		// (this launch writes the word: past L1, once for the CTA)
		if (__syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile uint32_t *>(info + 1) > kJoinRunLimit)) return;
		const uint64_t i = base + threadIdx.x;
		const uint64_t k = static_cast<uint64_t>(keys[i < n ? i : n - 1]) - bias;
		const uint64_t next = __shfl_down_sync(0xffffffffu, k, 1);
		const uint32_t live = __ballot_sync(0xffffffffu, i < n);
		if (__any_sync(0xffffffffu, lane < 31 && i + 1 < n && next == k)) {
			const uint32_t peers = __match_any_sync(0xffffffffu, k) & live;
			if (i < n && static_cast<uint32_t>(__ffs(peers) - 1) == lane) {
				const uint32_t count = atomicAdd(&entries[k].y, __popc(peers)) + __popc(peers);
				if (count > kJoinRunLimit) atomicMax(info + 1, count);
			}
		} else if (i < n) {
			atomicAdd(&entries[k].y, 1u);
		}
	}
}

// Runs laid out tile by tile in whatever order the tiles arrive (a run's place does not matter); entry x becomes
// its start.
__global__ void __launch_bounds__(256) JoinEntryPlaceKernel(uint2 *entries, uint64_t count, uint32_t *info) {
	__shared__ uint32_t scratch[33], base;
	const bool stop = threadIdx.x == 0 && *reinterpret_cast<volatile uint32_t *>(info + 1) > kJoinRunLimit;  // (written here)
	if (__syncthreads_or(stop)) return;
	uint32_t longest = 0;
	for (uint64_t first = blockIdx.x * 1024ull; first < count; first += gridDim.x * 1024ull) {
		const uint64_t i = first + threadIdx.x * 4ull;
		uint32_t c[4], sum = 0;
#pragma unroll
		for (int j = 0; j < 4; j++) {
			c[j] = i + j < count ? entries[i + j].y : 0u;
			sum += c[j];
			longest = max(longest, c[j]);
		}
		uint32_t total;
		uint32_t at = BlockScanExclusive<uint32_t>(sum, scratch, &total);
		if (threadIdx.x == 0) base = total ? atomicAdd(info + 2, total) : 0u;
		__syncthreads();
		at += base;
#pragma unroll
		for (int j = 0; j < 4; j++) {
			if (i + j < count) entries[i + j].x = at;
			at += c[j];
		}
		__syncthreads();
	}
	__shared__ uint32_t most;
	if (threadIdx.x == 0) most = 0;
	__syncthreads();
	longest = __reduce_max_sync(0xffffffffu, longest);
	if ((threadIdx.x & 31) == 0) atomicMax(&most, longest);
	__syncthreads();
	if (threadIdx.x == 0 && most > *reinterpret_cast<volatile uint32_t *>(info + 1)) atomicMax(info + 1, most);
}

// Each right row's number into its key's run, in any order; entry x moves to the run's end.
template <typename K>
__global__ void JoinEntryFillKernel(const K *keys, uint64_t n, uint64_t bias, uint2 *entries, uint32_t *rows,
                                    const uint32_t *info) {
	if (JoinRunTooLong(info)) return;
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		rows[atomicAdd(&entries[static_cast<uint64_t>(keys[i]) - bias].x, 1u)] = static_cast<uint32_t>(i);
	}
}

// Row order within the runs. A thread sorts a run of up to 16 rows in registers and local memory; longer ones
// go to a list for the kernel after.
constexpr uint32_t kRunShort = 16, kRunWarp = 256;

__global__ void JoinEntrySortKernel(const uint2 *entries, uint64_t count, uint32_t *rows, uint32_t *list, uint32_t *info) {
	if (JoinRunTooLong(info)) return;
	const uint32_t lane = threadIdx.x & 31;
	for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); w < count; w += (uint64_t)gridDim.x * blockDim.x) {
		const uint64_t k = w + lane;
		const uint2 e = k < count ? entries[k] : make_uint2(0, 0);
		const uint32_t listed = __ballot_sync(0xffffffffu, e.y > kRunShort);
		if (listed) {
			uint32_t at = 0;
			if (lane == 0) at = atomicAdd(info, __popc(listed));
			at = __shfl_sync(0xffffffffu, at, 0);
			if (e.y > kRunShort) list[at + __popc(listed & ((1u << lane) - 1))] = static_cast<uint32_t>(k);
		}
		if (e.y < 2) continue;
		uint32_t *r = rows + (e.x - e.y);
		if (e.y == 2) {
			const uint32_t a = r[0], b = r[1];
			if (a > b) {
				r[0] = b;
				r[1] = a;
			}
		} else if (e.y <= kRunShort) {
			uint32_t v[kRunShort];
			for (uint32_t i = 0; i < e.y; i++) {
				const uint32_t x = r[i];
				uint32_t j = i;
				for (; j > 0 && v[j - 1] > x; j--) v[j] = v[j - 1];
				v[j] = x;
			}
			for (uint32_t i = 0; i < e.y; i++) r[i] = v[i];
		}
	}
}

// Listed runs. Up to 256 rows a warp ranks them: a row's place is the number of smaller ones (row numbers differ),
// counted while the others pass by. Longer ones a CTA sorts in shared memory by a bitonic network over the next power
// of two.
__global__ void __launch_bounds__(256) JoinEntrySortLongKernel(const uint2 *entries, uint32_t *rows, const uint32_t *list,
                                                              const uint32_t *info) {
	__shared__ uint32_t v[kJoinRunLimit];
	if (__syncthreads_or(JoinRunTooLong(info))) return;
	const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
	for (uint32_t item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < info[0]; item += warps) {
		const uint2 e = entries[list[item]];
		if (e.y > kRunWarp) continue;
		uint32_t *r = rows + (e.x - e.y);
		if (e.y <= 32) {
			const uint32_t own = lane < e.y ? r[lane] : 0xffffffffu;
			uint32_t rank = 0;
#pragma unroll
			for (int l = 0; l < 32; l++) rank += __shfl_sync(0xffffffffu, own, l) < own ? 1u : 0u;
			if (lane < e.y) r[rank] = own;
			continue;
		}
		constexpr int kEach = kRunWarp / 32;
		uint32_t own[kEach], rank[kEach];
#pragma unroll
		for (int j = 0; j < kEach; j++) {
			own[j] = j * 32 + lane < e.y ? r[j * 32 + lane] : 0xffffffffu;
			rank[j] = 0;
		}
#pragma unroll
		for (int s = 0; s < kEach; s++) {
			if (s * 32 >= e.y) break;
			for (int l = 0; l < 32; l++) {  // (rows past the run's end are above every row)
				const uint32_t other = __shfl_sync(0xffffffffu, own[s], l);
#pragma unroll
				for (int j = 0; j < kEach; j++) rank[j] += other < own[j] ? 1u : 0u;
			}
		}
		__syncwarp();
#pragma unroll
		for (int j = 0; j < kEach; j++) {
			if (j * 32 + lane < e.y) r[rank[j]] = own[j];
		}
	}
	for (uint32_t item = blockIdx.x; item < info[0]; item += gridDim.x) {
		const uint2 e = entries[list[item]];
		if (e.y <= kRunWarp) continue;
		uint32_t *r = rows + (e.x - e.y);
		const uint32_t size = 1u << (32 - __clz(e.y - 1));
		for (uint32_t i = threadIdx.x; i < size; i += blockDim.x) v[i] = i < e.y ? r[i] : 0xffffffffu;
		__syncthreads();
		for (uint32_t k = 2; k <= size; k <<= 1) {
			for (uint32_t j = k >> 1; j > 0; j >>= 1) {
				for (uint32_t i = threadIdx.x; i < size; i += blockDim.x) {
					const uint32_t o = i ^ j;
					if (o > i) {
						const uint32_t a = v[i], b = v[o];
						if ((a > b) == ((i & k) == 0)) {
							v[i] = b;
							v[o] = a;
						}
					}
				}
				__syncthreads();
			}
		}
		for (uint32_t i = threadIdx.x; i < e.y; i += blockDim.x) r[i] = v[i];
		__syncthreads();
	}
}

// A left key's run: its first place in the right rows' order, and its length.
__device__ __forceinline__ uint2 JoinRunOf(const JoinRunsView &v, uint64_t key) {
	const uint64_t k = key - v.bias;  // below the bias wraps past every bucket: no match
	if (v.entries) {
		if (k >= v.nb) return make_uint2(0, 0);
		const uint2 e = reinterpret_cast<const uint2 *>(v.entries)[k];
		return make_uint2(e.x - e.y, e.y);
	}
	u32 count = 0;
	const long long at = vgpu_join_run(k, reinterpret_cast<const u64 *>(v.sorted), v.dir, v.nb, v.shift, &count);
	return make_uint2(at < 0 ? 0u : static_cast<uint32_t>(at), count);
}

constexpr int kJoinBlock = 256, kJoinItems = 4, kJoinTile = kJoinBlock * kJoinItems;

// Tile starts of the matches: chain (zero at launch) = total (u64, the top bit set when a wait ran out), ticket and
// longest tile (u32 each), tile counts (u32, an even number of them), tile starts + 1 (u64). A tile of more
// than 2^31 matches counts as failed too: the caller takes the other way.
template <typename K>
__global__ void __launch_bounds__(kJoinBlock) JoinMatchCountKernel(const K *keys, uint64_t n, JoinRunsView view, uint64_t ntiles,
                                                              uint64_t *chain, uint64_t wait_ns) {
	__shared__ uint32_t scratch[33], bound, next;
	__shared__ unsigned long long wide;
	uint32_t *words = reinterpret_cast<uint32_t *>(chain + 1);
	u32 *counts = reinterpret_cast<u32 *>(chain + 2);
	u64 *starts = reinterpret_cast<u64 *>(chain + 2 + (ntiles + 1) / 2);
	if (view.info && *(view.info + 1) > kJoinRunLimit) return;  // (written by earlier launches)
	if (threadIdx.x == 0) next = atomicAdd(words, 1u);
	__syncthreads();
	const uint32_t ticket = next;
	__syncthreads();  // read by every thread: the following ticket comes in the same word
	if (ticket == 0) {
		const u64 t = tile_scanner(counts, starts, ntiles, scratch, &bound, wait_ns);
		if (threadIdx.x == 0) tiles_total(reinterpret_cast<u64 *>(chain), t);
		return;
	}
	uint32_t longest = 0;
	for (uint64_t tile = ticket - 1ull; tile < ntiles;) {
		const uint64_t row0 = tile * kJoinTile + threadIdx.x * static_cast<uint64_t>(kJoinItems);
		K k[kJoinItems];
#pragma unroll
		for (int i = 0; i < kJoinItems; i++) k[i] = row0 + i < n ? keys[row0 + i] : K(0);
		uint64_t sum = 0;
#pragma unroll
		for (int i = 0; i < kJoinItems; i++) sum += row0 + i < n ? JoinRunOf(view, static_cast<uint64_t>(k[i])).y : 0u;
		if (threadIdx.x == 0) {
			wide = 0;
			next = atomicAdd(words, 1u);
		}
		__syncthreads();
		for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
		if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&wide, static_cast<unsigned long long>(sum));
		__syncthreads();
		const uint64_t total = wide, after = next - 1ull;
		if (threadIdx.x == 0) {
			if (total >> 31) atomicOr(reinterpret_cast<unsigned long long *>(chain), 1ull << 62);
			st_relaxed(counts + tile, static_cast<u32>(total >> 31 ? 0 : total) + 1u);
			longest = max(longest, static_cast<uint32_t>(total >> 31 ? 0x7fffffffull : total));
		}
		__syncthreads();
		tile = after;
	}
	if (threadIdx.x == 0 && longest) atomicMax(words + 1, longest);
}

template <typename T> __device__ __forceinline__ void JoinCopy(const JoinOut &c, uint64_t from, uint64_t to) {
	static_cast<T *>(c.dst)[to] = static_cast<const T *>(c.src)[from];
}

template <typename K>
__global__ void __launch_bounds__(kJoinBlock) JoinEmitKernel(const K *keys, uint64_t n, JoinRunsView view, uint64_t ntiles,
                                                            const uint64_t *starts, const uint32_t *rows, JoinOuts outs,
                                                            uint32_t parts) {
	__shared__ uint32_t scratch[33], offset[kJoinTile], first[kJoinTile];
	for (uint64_t item = blockIdx.x; item < ntiles * parts; item += gridDim.x) {
		const uint64_t tile = item / parts;
		const uint32_t part = static_cast<uint32_t>(item % parts);
		const uint64_t row0 = tile * kJoinTile + threadIdx.x * static_cast<uint64_t>(kJoinItems);
		K k[kJoinItems];
#pragma unroll
		for (int i = 0; i < kJoinItems; i++) k[i] = row0 + i < n ? keys[row0 + i] : K(0);
		uint2 run[kJoinItems];
		uint32_t sum = 0;
#pragma unroll
		for (int i = 0; i < kJoinItems; i++) {
			run[i] = row0 + i < n ? JoinRunOf(view, static_cast<uint64_t>(k[i])) : make_uint2(0, 0);
			sum += run[i].y;
		}
		uint32_t total;
		uint32_t at = BlockScanExclusive<uint32_t>(sum, scratch, &total);
#pragma unroll
		for (int i = 0; i < kJoinItems; i++) {
			offset[threadIdx.x * kJoinItems + i] = at;
			first[threadIdx.x * kJoinItems + i] = run[i].x;
			at += run[i].y;
		}
		__syncthreads();
		const uint64_t base = starts[tile] - 1;
		for (uint32_t o = part * kJoinBlock + threadIdx.x; o < total; o += kJoinBlock * parts) {
			uint32_t r = 0;  // the last row whose matches start at or before o (rows without any share their start)
#pragma unroll
			for (uint32_t step = kJoinTile / 2; step > 0; step >>= 1) r += offset[r + step] <= o ? step : 0u;
			const uint64_t left = tile * kJoinTile + r, place = first[r] + (o - offset[r]);
			const uint64_t right = rows ? rows[place] : place;
			for (int c = 0; c < outs.n; c++) {
				const JoinOut &col = outs.c[c];
				const uint64_t from = col.right ? right : left, to = base + o;
				switch (col.width) {
				case 1: JoinCopy<uint8_t>(col, from, to); break;
				case 2: JoinCopy<uint16_t>(col, from, to); break;
				case 4: JoinCopy<uint32_t>(col, from, to); break;
				case 8: JoinCopy<uint64_t>(col, from, to); break;
				default: JoinCopy<uint4>(col, from, to); break;
				}
			}
		}
		__syncthreads();
	}
}

// Each left key's run: its first place in the right rows' order, and its length.
template <typename K>
__global__ void JoinRunKernel(const K *keys, uint64_t n, JoinRunsView view, uint64_t *lower, uint64_t *count) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		const uint2 run = JoinRunOf(view, static_cast<uint64_t>(keys[i]));
		lower[i] = run.x;
		count[i] = run.y;
	}
}

// Radix directory over a sorted key array (see vgpu_join_find): position i writes the entries of the
// buckets that start at i, so every one of the nb + 1 entries is written exactly once.
__global__ void JoinDirectoryKernel(const uint64_t *sorted, uint64_t n, uint32_t shift, uint64_t nb, uint32_t *dir) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= n; i += (uint64_t)gridDim.x * blockDim.x) {
		const uint64_t lo = i == 0 ? 0 : (sorted[i - 1] >> shift) + 1;
		const uint64_t hi = i == n ? nb : (sorted[i] >> shift);
		for (uint64_t b = lo; b <= hi && b <= nb; ++b) dir[b] = static_cast<uint32_t>(i);
	}
}

// Dense key tables (see JoinDenseFill): plain stores, then a count of the entries that were written. Keys
// are distinct exactly when that count equals the row count, so nothing has to be claimed by
// compare-and-swap: 2^24 keys into a 32 MB table of 2-byte entries took 0.40 ms with 16-bit swaps; the
// fill, the stores (bound by one L2 sector write per key) and the count together take 0.16 ms.
template <typename K, typename V, typename E>
__global__ void JoinFillKernel(const K *keys, const V *values, uint64_t n, uint64_t bias, uint64_t base, E *table) {
	const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
	uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	for (; i + 3 * stride < n; i += 4 * stride) {
		K k[4];
		V v[4];
#pragma unroll
		for (int j = 0; j < 4; j++) {
			k[j] = keys[i + j * stride];
			v[j] = values[i + j * stride];
		}
#pragma unroll
		for (int j = 0; j < 4; j++) table[static_cast<uint64_t>(k[j]) - bias] = static_cast<E>(static_cast<uint64_t>(v[j]) + base);
	}
	for (; i < n; i += stride) table[static_cast<uint64_t>(keys[i]) - bias] = static_cast<E>(static_cast<uint64_t>(values[i]) + base);
}

template <typename K> __global__ void JoinFillRowsKernel(const K *keys, uint64_t n, uint64_t bias, uint32_t *table) {
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		table[static_cast<uint64_t>(keys[i]) - bias] = static_cast<uint32_t>(i + 1);
	}
}

// Entries that differ from the empty marker (zero, or all ones).
template <typename E> __global__ void __launch_bounds__(256) JoinCountKernel(const E *table, uint64_t entries, E empty,
                                                                            uint32_t *occupied) {
	constexpr uint64_t kPer = 16 / sizeof(E);
	const uint64_t vecs = entries / kPer, stride = (uint64_t)gridDim.x * blockDim.x;
	const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
	uint32_t c = 0;
	const uint4 *v = reinterpret_cast<const uint4 *>(table);
	for (uint64_t i = tid; i < vecs; i += stride) {
		const uint4 q = v[i];
		E x[kPer];
		memcpy(x, &q, 16);
#pragma unroll
		for (uint64_t j = 0; j < kPer; j++) c += x[j] != empty ? 1u : 0u;
	}
	if (tid < entries - vecs * kPer) c += table[vecs * kPer + tid] != empty ? 1u : 0u;
	c = __reduce_add_sync(0xffffffffu, c);
	__shared__ uint32_t warps[8];
	if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = c;
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int w = 1; w < 8; w++) c += warps[w];
		if (c) atomicAdd(occupied, c);
	}
}

__global__ void CountAdjacentEqualKernel(const uint64_t *sorted, uint64_t n, uint32_t *out) {
	uint32_t local = 0;
	for (uint64_t i = 1 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		local += sorted[i] == sorted[i - 1] ? 1u : 0u;
	}
	if (local) atomicAdd(out, local);
}

// Longest run of equal keys in a sorted array: every run start finds its end by a galloping then a
// binary search, and the lengths meet in one atomic maximum.
__global__ void MaxRunLengthKernel(const uint64_t *sorted, uint64_t n, uint32_t *out) {
	uint32_t local = 0;
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		const uint64_t k = sorted[i];
		if (i > 0 && sorted[i - 1] == k) continue;
		// gallop: `good` holds k, `bad` is the first probe past the run (or n)
		uint64_t good = i, step = 1, bad = n;
		while (good + step < n) {
			if (sorted[good + step] != k) {
				bad = good + step;
				break;
			}
			good += step;
			step <<= 1;
		}
		// the run ends in (good, bad]: binary search for the first position without k
		uint64_t a = good + 1, b = bad;
		while (a < b) {
			const uint64_t mid = (a + b) >> 1;
			if (sorted[mid] == k) a = mid + 1;
			else b = mid;
		}
		const uint64_t len = a - i;
		local = max(local, len > 0xffffffffull ? 0xffffffffu : static_cast<uint32_t>(len));
	}
	if (local) atomicMax(out, local);
}

// Work list of a partitioned aggregation pass. Item = (partition, first row, end row, split index or
// ~0). Partitions above `split_rows` rows become ceil(size / split_rows) chunks sharing one split
// index; everything is ordered longest first by size class (chunks of split partitions, then
// partitions by descending floor(log2(size))), so the longest items start first and the persistent
// CTAs finish together. Empty partitions produce no item. One CTA.
constexpr int kPlanBlock = 1024;

__global__ void __launch_bounds__(kPlanBlock) PlanWorkKernel(const uint32_t *offsets, uint64_t stride, uint32_t P,
                                                             const uint32_t *total_rows, uint32_t min_split,
                                                             uint32_t ctas, uint4 *items, uint32_t *counts,
                                                             uint32_t *split_info, uint32_t max_split) {
	__shared__ uint32_t cls_count[34];
	__shared__ uint32_t cls_cursor[34];
	__shared__ uint32_t n_split;
	__shared__ uint32_t split_rows;
	if (threadIdx.x < 34) cls_count[threadIdx.x] = 0;
	if (threadIdx.x == 0) {
		n_split = 0;
		// chunks small enough that every CTA gets several items on average
		const uint32_t total = *total_rows;
		// rounded up, so fewer than 4 * ctas partitions exceed it: the caller sizes the split tables from
		// that bound without reading the plan back
		const uint64_t quarter = 4ull * (ctas ? ctas : 1);
		const uint32_t even = static_cast<uint32_t>((total + quarter - 1) / quarter);
		split_rows = even > min_split ? even : min_split;
	}
	__syncthreads();
	const uint32_t total = *total_rows;
	const uint32_t S = split_rows;
	for (uint32_t p = threadIdx.x; p < P; p += blockDim.x) {
		const uint32_t r0 = offsets[static_cast<uint64_t>(p) * stride];
		const uint32_t r1 = p + 1 < P ? offsets[static_cast<uint64_t>(p + 1) * stride] : total;
		const uint32_t size = r1 - r0;
		if (size == 0) continue;
		const bool split = size > S;
		const uint32_t nch = split ? (size + S - 1) / S : 1u;
		const int cls = split ? 33 : 31 - __clz(size);
		atomicAdd(&cls_count[cls], nch);
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		uint32_t run = 0;
		for (int c = 33; c >= 0; --c) {
			cls_cursor[c] = run;
			run += cls_count[c];
		}
		counts[0] = run;
	}
	__syncthreads();
	for (uint32_t p = threadIdx.x; p < P; p += blockDim.x) {
		const uint32_t r0 = offsets[static_cast<uint64_t>(p) * stride];
		const uint32_t r1 = p + 1 < P ? offsets[static_cast<uint64_t>(p + 1) * stride] : total;
		const uint32_t size = r1 - r0;
		if (size == 0) continue;
		const bool split = size > S;
		const uint32_t nch = split ? (size + S - 1) / S : 1u;
		const int cls = split ? 33 : 31 - __clz(size);
		const uint32_t pos = atomicAdd(&cls_cursor[cls], nch);
		uint32_t sidx = ~0u;
		if (split) {
			sidx = atomicAdd(&n_split, 1u);
			if (sidx < max_split) {
				split_info[2 * sidx] = nch;
				split_info[2 * sidx + 1] = 0;
			}
		}
		for (uint32_t c = 0; c < nch; ++c) {
			const uint32_t a = r0 + c * S;
			const uint32_t b = (c + 1 == nch) ? r1 : a + S;
			items[pos + c] = make_uint4(p, a, b, sidx);
		}
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		counts[1] = n_split;
		counts[3] = *total_rows;  // read back with the split count: the partitioned row count
	}
}

} // namespace

void JoinDirectory(const uint64_t *sorted, uint64_t n, uint32_t shift, uint64_t nb, uint32_t *dir, cudaStream_t stream) {
	LaunchScope scope("join_directory", stream, n * 8 + (nb + 1) * 4, n);
	JoinDirectoryKernel<<<GridFor(n + 1, 256), 256, 0, stream>>>(sorted, n, shift, nb, dir);
	VGPU_CUDA(cudaGetLastError());
}

namespace {

// f(typed key pointer) for a key column of `width` bytes, read as unsigned.
template <typename F> void WithKeys(const void *keys, size_t width, F &&f) {
	switch (width) {
	case 1: return f(static_cast<const uint8_t *>(keys));
	case 2: return f(static_cast<const uint16_t *>(keys));
	case 4: return f(static_cast<const uint32_t *>(keys));
	case 8: return f(static_cast<const uint64_t *>(keys));
	default: Fail(VGPU_ERR_INTERNAL, "join keys: width must be 1, 2, 4 or 8 bytes");
	}
}

template <typename F> void WithValues(const void *values, size_t width, F &&f) {
	switch (width) {
	case 1: return f(static_cast<const uint8_t *>(values));
	case 2: return f(static_cast<const uint16_t *>(values));
	case 4: return f(static_cast<const uint32_t *>(values));
	default: Fail(VGPU_ERR_INTERNAL, "join table: value width must be 1, 2 or 4 bytes");
	}
}

template <typename E> void LaunchCount(const E *table, uint64_t entries, E empty, uint32_t *occupied, cudaStream_t stream) {
	const unsigned grid = std::min<unsigned>(GridFor(entries * sizeof(E) / 16 + 1, 256), Runtime::Get().props().sm_count * 8);
	JoinCountKernel<E><<<grid, 256, 0, stream>>>(table, entries, empty, occupied);
}

} // namespace

void JoinDenseFill(const void *keys, size_t kwidth, const void *values, size_t vwidth, uint64_t n, uint64_t bias,
                   uint64_t range, uint32_t vmin, void *table, size_t width, uint32_t *occupied, cudaStream_t stream) {
	LaunchScope scope("join_dense_table", stream, n * (kwidth + vwidth) + (range + 1) * width, n);
	// 8-byte entries and row numbers mark an empty key with 0, narrower values with all ones
	const bool ones = values != nullptr && width != 8;
	VGPU_CUDA(cudaMemsetAsync(table, ones ? 0xff : 0, (range + 1) * width, stream));
	VGPU_CUDA(cudaMemsetAsync(occupied, 0, 4, stream));
	const unsigned grid = GridFor((n + 3) / 4, 256);
	WithKeys(keys, kwidth, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		if (!values) {
			JoinFillRowsKernel<K><<<GridFor(n, 256), 256, 0, stream>>>(k, n, bias, static_cast<uint32_t *>(table));
			return;
		}
		WithValues(values, vwidth, [&](auto *v) {
			using V = std::remove_const_t<std::remove_pointer_t<decltype(v)>>;
			const uint64_t base = width == 8 ? 1ull << 32 : 0ull - vmin;
			switch (width) {
			case 1: JoinFillKernel<K, V, uint8_t><<<grid, 256, 0, stream>>>(k, v, n, bias, base, static_cast<uint8_t *>(table)); break;
			case 2: JoinFillKernel<K, V, uint16_t><<<grid, 256, 0, stream>>>(k, v, n, bias, base, static_cast<uint16_t *>(table)); break;
			case 4: JoinFillKernel<K, V, uint32_t><<<grid, 256, 0, stream>>>(k, v, n, bias, base, static_cast<uint32_t *>(table)); break;
			case 8: JoinFillKernel<K, V, uint64_t><<<grid, 256, 0, stream>>>(k, v, n, bias, base, static_cast<uint64_t *>(table)); break;
			default: Fail(VGPU_ERR_INTERNAL, "join table: entry width must be 1, 2, 4 or 8 bytes");
			}
		});
	});
	VGPU_CUDA(cudaGetLastError());
	switch (width) {
	case 1: LaunchCount<uint8_t>(static_cast<uint8_t *>(table), range + 1, 0xffu, occupied, stream); break;
	case 2: LaunchCount<uint16_t>(static_cast<uint16_t *>(table), range + 1, 0xffffu, occupied, stream); break;
	case 4: LaunchCount<uint32_t>(static_cast<uint32_t *>(table), range + 1, ones ? 0xffffffffu : 0u, occupied, stream); break;
	default: LaunchCount<uint64_t>(static_cast<uint64_t *>(table), range + 1, 0ull, occupied, stream); break;
	}
	VGPU_CUDA(cudaGetLastError());
}

void ColumnBounds(const BoundsColumn *cols, int n, uint64_t *out, cudaStream_t stream, bool distinct, uint64_t *pairs) {
	if (n <= 0) return;
	if (pairs && distinct) Fail(VGPU_ERR_INTERNAL, "column bounds: distinct counts or pairs, not both");
	if (pairs) VGPU_CUDA(cudaMemsetAsync(pairs, 0, static_cast<size_t>(n) * 16, stream));
	VGPU_CUDA(cudaMemsetAsync(out, 0, BoundsWords(n, distinct) * 8, stream));
	unsigned int *ranks = distinct ? reinterpret_cast<unsigned int *>(out + 2 * n) : nullptr;
	for (int first = 0; first < n; first += kMaxBoundsColumns) {
		BoundsArgs a;
		const int count = std::min(n - first, kMaxBoundsColumns);
		uint64_t bytes = 0, rows = 0, widest = 0;
		for (int j = 0; j < count; j++) {
			a.c[j] = cols[first + j];
			const uint64_t b = a.c[j].rows * BoundsWidth(a.c[j].kind);
			bytes += b;
			rows += a.c[j].rows;
			widest = std::max(widest, b);
		}
		if (widest == 0) continue;
		a.out = reinterpret_cast<unsigned long long *>(out + 2 * first);
		a.ranks = ranks ? ranks + static_cast<size_t>(first) * kDistinctRanks : nullptr;
		a.pairs = pairs ? reinterpret_cast<unsigned long long *>(pairs + 2 * first) : nullptr;
		LaunchScope scope("column_bounds", stream, bytes, rows);
		// four 16-byte loads per thread, at most eight CTAs per SM over all columns
		const uint64_t cap = std::max<uint64_t>(1, static_cast<uint64_t>(Runtime::Get().props().sm_count) * 8 / count);
		const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(cap, (widest + kBoundsBlock * 64 - 1) / (kBoundsBlock * 64)));
		const dim3 ctas(grid, static_cast<unsigned>(count));
		if (pairs) ColumnBoundsKernel<true><<<ctas, kBoundsBlock, 0, stream>>>(a);
		else ColumnBoundsKernel<false><<<ctas, kBoundsBlock, 0, stream>>>(a);
		VGPU_CUDA(cudaGetLastError());
	}
}

uint64_t DistinctEstimate(const uint64_t *words, int n, int column, BoundsKind kind) {
	if (BoundsWidth(kind) < 4) return 0;
	const uint32_t *ranks = reinterpret_cast<const uint32_t *>(words + 2 * n) + static_cast<size_t>(column) * kDistinctRanks;
	double sum = 0;
	int empty = 0;
	for (int i = 0; i < kDistinctRanks; i++) {
		sum += std::ldexp(1.0, -static_cast<int>(ranks[i]));
		empty += ranks[i] == 0;
	}
	const double m = kDistinctRanks, raw = 0.7213 / (1 + 1.079 / m) * m * m / sum;
	const double picked = raw <= 2.5 * m && empty ? m * std::log(m / empty) : raw;
	return static_cast<uint64_t>(picked * (1 << kDistinctShift)) + 1;
}

BoundsKind SignedBoundsKind(ValueType t) {
	switch (t) {
	case ValueType::INT16: return BoundsKind::I16;
	case ValueType::INT32:
	case ValueType::DICTIONARY_STRING: return BoundsKind::I32;
	case ValueType::INT64: return BoundsKind::I64;
	case ValueType::BOOLEAN: return BoundsKind::BOOL;
	default: Fail(VGPU_ERR_INTERNAL, "min/max statistics need an integer column");
	}
}

// Multi-match inline table: entry[k] = the key's match count in the low `cbits` bits, then one
// `vbits`-bit slot per match holding value bits - vmin (the matches of a key in no particular order).
// A match reserves its slot by adding 1 to the count and then ORs its value into that slot; a key
// with more than rmax matches (rmax < 2^cbits, so the count never wraps before it is seen) counts in
// *overflow and the table is not valid.
template <typename K, typename T, typename E>
__global__ void JoinDenseMultiKernel(const K *keys, const T *values, uint64_t n, uint64_t bias, uint32_t vmin,
                                     uint32_t vbits, uint32_t cbits, uint32_t rmax, E *table, uint32_t *overflow) {
	const E cmask = (E(1) << cbits) - 1;
	uint32_t local = 0;
	for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
		E *slot = table + (static_cast<uint64_t>(keys[i]) - bias);
		const E old = atomicAdd(slot, E(1));
		const uint32_t j = static_cast<uint32_t>(old & cmask);
		if (j >= rmax) {
			local++;
			continue;
		}
		const E v = static_cast<E>(static_cast<uint32_t>(values[i]) - vmin);
		atomicOr(slot, v << (cbits + j * vbits));
	}
	if (local) atomicAdd(overflow, local);
}

void JoinDenseMulti(const void *keys, size_t kwidth, const void *values, size_t vwidth, uint64_t n, uint64_t bias,
                    uint64_t range, uint32_t vmin, uint32_t vbits, uint32_t cbits, uint32_t rmax, void *table, bool wide,
                    uint32_t *overflow, cudaStream_t stream) {
	const size_t ew = wide ? 8 : 4;
	if (cbits < 1 || cbits > 3 || rmax >= (1u << cbits) || cbits + rmax * vbits > ew * 8) {
		Fail(VGPU_ERR_INTERNAL, "multi-match join table: slots do not fit the entry");
	}
	LaunchScope scope("join_dense_multi", stream, n * (kwidth + vwidth) + (range + 1) * ew, n);
	VGPU_CUDA(cudaMemsetAsync(table, 0, (range + 1) * ew, stream));
	VGPU_CUDA(cudaMemsetAsync(overflow, 0, 4, stream));
	const unsigned grid = GridFor(n, 256);
	WithKeys(keys, kwidth, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		WithValues(values, vwidth, [&](auto *v) {
			using V = std::remove_const_t<std::remove_pointer_t<decltype(v)>>;
			if (wide) {
				JoinDenseMultiKernel<K, V, unsigned long long><<<grid, 256, 0, stream>>>(
				    k, v, n, bias, vmin, vbits, cbits, rmax, static_cast<unsigned long long *>(table), overflow);
			} else {
				JoinDenseMultiKernel<K, V, unsigned int><<<grid, 256, 0, stream>>>(
				    k, v, n, bias, vmin, vbits, cbits, rmax, static_cast<unsigned int *>(table), overflow);
			}
		});
	});
	VGPU_CUDA(cudaGetLastError());
}

void CountAdjacentEqual(const uint64_t *sorted, uint64_t n, uint32_t *out, cudaStream_t stream) {
	VGPU_CUDA(cudaMemsetAsync(out, 0, 4, stream));
	if (n < 2) return;
	LaunchScope scope("count_adjacent_equal", stream, n * 8, n);
	CountAdjacentEqualKernel<<<GridFor(n, 256), 256, 0, stream>>>(sorted, n, out);
	VGPU_CUDA(cudaGetLastError());
}

void MaxRunLength(const uint64_t *sorted, uint64_t n, uint32_t *out, cudaStream_t stream) {
	VGPU_CUDA(cudaMemsetAsync(out, 0, 4, stream));
	if (n == 0) return;
	LaunchScope scope("max_run_length", stream, n * 8, n);
	MaxRunLengthKernel<<<GridFor(n, 256), 256, 0, stream>>>(sorted, n, out);
	VGPU_CUDA(cudaGetLastError());
}

uint64_t PlanWorkCapacity(uint32_t P, uint64_t rows, uint32_t min_split) {
	return static_cast<uint64_t>(P) + rows / (min_split ? min_split : 1) + 1;
}

namespace {
constexpr int kHeavyBlock = 1024;
constexpr uint32_t kHeavyBins = 1024;  // counts at or above the last bin share it
static_assert(kHeavyBins == kHeavyBlock, "a thread per bin");

__device__ uint64_t HeavyBlockSum(uint64_t v, uint64_t *scratch) {
	for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
	if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
	__syncthreads();
	uint64_t total = 0;
	for (uint32_t w = 0; w < blockDim.x / 32; ++w) total += scratch[w];
	__syncthreads();
	return total;
}

// The sample's counts: a histogram, their sum, and a list of the keys seen min_count times or more, so that the
// one CTA that selects walks those alone (a thread per slot; walking the whole table four times from one CTA took
// 82 us, the two kernels together take 21).
__global__ void __launch_bounds__(kHeavyBlock) HeavyCountKernel(const uint64_t *keys, const uint32_t *counts,
                                                                uint32_t min_count, HeavyScratch *g, uint2 *list) {
	__shared__ uint32_t hist[kHeavyBins], warp_base[kHeavyBlock / 32], base;
	__shared__ uint64_t scratch[32];
	const uint32_t s = blockIdx.x * kHeavyBlock + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	hist[threadIdx.x] = 0;
	const uint64_t key = keys[s];
	const uint32_t c = key == ~0ull ? 0u : counts[s];
	const uint32_t chosen = __ballot_sync(0xffffffffu, c >= min_count);
	if (lane == 0) warp_base[warp] = __popc(chosen);
	__syncthreads();
	// most sampled keys share a few small counts: lanes of one bin add once
	const uint32_t bin = c < kHeavyBins ? c : kHeavyBins - 1;
	const uint32_t peers = __match_any_sync(0xffffffffu, bin);
	if (bin && static_cast<uint32_t>(__ffs(peers) - 1) == lane) atomicAdd(&hist[bin], __popc(peers));
	if (threadIdx.x == 0) {
		uint32_t total = 0;
		for (uint32_t w = 0; w < kHeavyBlock / 32; ++w) {
			const uint32_t n = warp_base[w];
			warp_base[w] = total;
			total += n;
		}
		base = total ? atomicAdd(&g->listed, total) : 0;
	}
	const uint64_t sampled = HeavyBlockSum(c, scratch);
	if (threadIdx.x == 0 && sampled) atomicAdd(reinterpret_cast<unsigned long long *>(&g->sampled), sampled);
	if (c >= min_count) {  // mixed keys of the direct-partitioned group-by: below 2^31
		list[base + warp_base[warp] + __popc(chosen & ((1u << lane) - 1))] = make_uint2(static_cast<uint32_t>(key), c);
	}
	if (hist[threadIdx.x]) atomicAdd(&g->hist[threadIdx.x], hist[threadIdx.x]);
}

__global__ void __launch_bounds__(kHeavyBlock) HeavySelectKernel(const HeavyScratch *g, uint2 *list, uint32_t *hmap,
                                                                 uint32_t dbits, uint32_t *hkeys, uint32_t K,
                                                                 uint32_t min_count, bool require_cover,
                                                                 uint32_t *n_heavy) {
	__shared__ uint64_t scratch[32];
	__shared__ uint32_t above[kHeavyBlock / 32];
	__shared__ uint32_t n_keys;
	const uint32_t dmask = (1u << dbits) - 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	constexpr uint32_t kWon = 0x80000000u;
	if (threadIdx.x == 0) n_keys = 0;
	// the smallest threshold from min_count up whose keys fit in K: keys with counts in this thread's bin or above
	uint32_t keys_at = g->hist[threadIdx.x];
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t o = __shfl_down_sync(0xffffffffu, keys_at, d);
		if (lane + d < 32) keys_at += o;
	}
	if (lane == 0) above[warp] = keys_at;
	__syncthreads();
	for (uint32_t w = warp + 1; w < kHeavyBlock / 32; ++w) keys_at += above[w];
	const uint32_t t = min(min_count, kHeavyBins) + __syncthreads_count(threadIdx.x >= min_count && keys_at > K);
	const uint32_t listed = g->listed;
	// claim each candidate's partition; the winner marks its entry
	for (uint32_t i = threadIdx.x; i < listed; i += kHeavyBlock) {
		const uint2 e = list[i];
		if (e.y < t) continue;
		if (atomicCAS(&hmap[e.x >> dbits], ~0u, 0xfffe0000u | (e.x & dmask)) == ~0u) list[i].y = e.y | kWon;
	}
	__syncthreads();
	uint64_t covered = 0;
	for (uint32_t i = threadIdx.x; i < listed; i += kHeavyBlock) {
		const uint2 e = list[i];
		if (!(e.y & kWon)) continue;
		const uint32_t idx = atomicAdd(&n_keys, 1u);
		if (idx < K) {
			hmap[e.x >> dbits] = (idx << 16) | (e.x & dmask);
			hkeys[idx] = e.x;
			covered += e.y & ~kWon;
		} else {
			hmap[e.x >> dbits] = ~0u;
			list[i].y = e.y & ~kWon;
		}
	}
	covered = HeavyBlockSum(covered, scratch);
	const bool drop = require_cover && covered * 10 < g->sampled;
	if (drop) {
		for (uint32_t i = threadIdx.x; i < listed; i += kHeavyBlock) {
			const uint2 e = list[i];
			if (e.y & kWon) hmap[e.x >> dbits] = ~0u;
		}
	}
	if (threadIdx.x == 0) *n_heavy = drop ? 0u : (n_keys < K ? n_keys : K);
}
} // namespace

void HeavySelect(const uint64_t *sample_keys, const uint32_t *sample_counts, uint32_t SC, HeavyScratch *scratch,
                 uint64_t *list, uint32_t *hmap, uint32_t dbits, uint32_t *heavy_keys, uint32_t K, uint32_t min_count,
                 bool require_cover, uint32_t *n_heavy, cudaStream_t stream) {
	if (SC % kHeavyBlock != 0) {
		Fail(VGPU_ERR_INTERNAL, "heavy_select: sample table size must be a multiple of 1024");
	}
	if (min_count < 1) min_count = 1;
	uint2 *entries = reinterpret_cast<uint2 *>(list);
	{
		LaunchScope scope("heavy_count", stream, static_cast<uint64_t>(SC) * 12, SC);
		HeavyCountKernel<<<SC / kHeavyBlock, kHeavyBlock, 0, stream>>>(sample_keys, sample_counts, min_count, scratch,
		                                                               entries);
		VGPU_CUDA(cudaGetLastError());
	}
	LaunchScope scope("heavy_select", stream, 0, 0);
	HeavySelectKernel<<<1, kHeavyBlock, 0, stream>>>(scratch, entries, hmap, dbits, heavy_keys, K, min_count, require_cover,
	                                                 n_heavy);
	VGPU_CUDA(cudaGetLastError());
}

void PlanWork(const uint32_t *offsets, uint64_t stride, uint32_t P, const uint32_t *total_rows, uint32_t min_split,
              uint32_t ctas, void *items, uint32_t *counts, uint32_t *split_info, uint32_t max_split,
              cudaStream_t stream) {
	LaunchScope scope("plan_work", stream, static_cast<uint64_t>(P) * 8, P);
	PlanWorkKernel<<<1, kPlanBlock, 0, stream>>>(offsets, stride, P, total_rows, min_split, ctas,
	                                             static_cast<uint4 *>(items), counts, split_info, max_split);
	VGPU_CUDA(cudaGetLastError());
}

void ExclusiveScanU32(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *total, Arena &arena) {
	ExclusiveScan<uint32_t>(in, out, n, total, arena);
}

void ExclusiveScanU64(const uint64_t *in, uint64_t *out, uint64_t n, uint64_t *total, Arena &arena) {
	ExclusiveScan<uint64_t>(in, out, n, total, arena);
}

void UnpackValidity(const uint8_t *bitmap, uint8_t *bytes, uint64_t n, cudaStream_t stream) {
	if (n == 0) return;
	LaunchScope scope("unpack_validity", stream, n / 8 + n, n);
	UnpackValidityKernel<<<GridFor(n, 256), 256, 0, stream>>>(bitmap, bytes, n);
	VGPU_CUDA(cudaGetLastError());
}

void PackValidity(const uint8_t *bytes, uint8_t *bitmap, uint64_t n, cudaStream_t stream) {
	if (n == 0) return;
	LaunchScope scope("pack_validity", stream, n + n / 8, n);
	PackValidityKernel<<<GridFor((n + 7) / 8, 256), 256, 0, stream>>>(bytes, bitmap, n);
	VGPU_CUDA(cudaGetLastError());
}

void Gather(const void *src, size_t width, const uint32_t *idx, uint64_t n, void *dst, cudaStream_t stream) {
	if (n == 0) return;
	LaunchScope scope("gather", stream, n * (width * 2 + 4), n);
	const unsigned grid = GridFor(n, 256);
	switch (width) {
	case 1:
		GatherKernel<uint8_t><<<grid, 256, 0, stream>>>(static_cast<const uint8_t *>(src), idx, n, static_cast<uint8_t *>(dst));
		break;
	case 2:
		GatherKernel<uint16_t><<<grid, 256, 0, stream>>>(static_cast<const uint16_t *>(src), idx, n, static_cast<uint16_t *>(dst));
		break;
	case 4:
		GatherKernel<uint32_t><<<grid, 256, 0, stream>>>(static_cast<const uint32_t *>(src), idx, n, static_cast<uint32_t *>(dst));
		break;
	case 8:
		GatherKernel<uint64_t><<<grid, 256, 0, stream>>>(static_cast<const uint64_t *>(src), idx, n, static_cast<uint64_t *>(dst));
		break;
	case 16:
		GatherKernel<uint4><<<grid, 256, 0, stream>>>(static_cast<const uint4 *>(src), idx, n, static_cast<uint4 *>(dst));
		break;
	default:
		Fail(VGPU_ERR_INTERNAL, "gather: unsupported width");
	}
	VGPU_CUDA(cudaGetLastError());
}

void CopyBuffers(const BufferCopy *copies, int n, cudaStream_t stream) {
	for (int first = 0; first < n; first += kMaxCopies) {
		CopyArgs a;
		const int count = std::min(n - first, kMaxCopies);
		uint64_t most = 0, bytes = 0;
		for (int j = 0; j < count; j++) {
			a.c[j] = copies[first + j];
			most = std::max(most, a.c[j].bytes);
			bytes += a.c[j].bytes;
		}
		if (most == 0) continue;
		LaunchScope scope("copy_buffers", stream, 2 * bytes, 0);
		const uint64_t cap = std::max<uint64_t>(1, static_cast<uint64_t>(Runtime::Get().props().sm_count) * 8 / count);
		const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(cap, (most + 4095) / 4096));
		CopyBuffersKernel<<<dim3(grid, static_cast<unsigned>(count)), 256, 0, stream>>>(a);
		VGPU_CUDA(cudaGetLastError());
	}
}

void WidenKeys(const void *src, size_t width, uint64_t n, uint64_t bias, uint64_t *dst, cudaStream_t stream) {
	if (n == 0) return;
	LaunchScope scope("widen_keys", stream, n * (width + 8), n);
	WithKeys(src, width, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		WidenKernel<K><<<GridFor(n, 256), 256, 0, stream>>>(k, n, bias, dst);
	});
	VGPU_CUDA(cudaGetLastError());
}

void Iota(uint32_t *out, uint64_t n, cudaStream_t stream) {
	if (n == 0) return;
	LaunchScope scope("iota", stream, n * 4, n);
	IotaKernel<<<GridFor(n, 256), 256, 0, stream>>>(out, n);
	VGPU_CUDA(cudaGetLastError());
}

void RadixSortPairs(uint64_t *keys, uint32_t *values, uint64_t *keys_alt, uint32_t *values_alt, uint64_t n, int bits,
                    Arena &arena) {
	cudaStream_t s = arena.stream();
	if (n <= 1 || bits <= 0) {
		Iota(values, n, s);
		return;
	}
	const uint64_t ntiles64 = (n + kSortTile - 1) / kSortTile;
	if (ntiles64 > 0xffffffffull) Fail(VGPU_ERR_UNSUPPORTED, "radix sort: too many rows");
	const uint32_t ntiles = static_cast<uint32_t>(ntiles64);
	uint32_t *hist = arena.AllocT<uint32_t>(static_cast<size_t>(ntiles) * 256);
	uint32_t *total = arena.AllocT<uint32_t>(1);
	uint64_t *kin = keys, *kout = keys_alt;
	const uint32_t *vin = nullptr;  // the first pass takes each key's position
	uint32_t *vout = values_alt, *vspare = values;
	const int passes = (bits + 7) / 8;
	for (int p = 0; p < passes; p++) {
		const int shift = 8 * p;
		{
			LaunchScope scope("radix_hist", s, n * 8, n);
			RadixHistKernel<<<ntiles, kSortBlock, 0, s>>>(kin, n, shift, hist, ntiles);
		}
		ExclusiveScanU32(hist, hist, static_cast<uint64_t>(ntiles) * 256, total, arena);
		{
			LaunchScope scope("radix_scatter", s, n * 24, n);
			RadixScatterKernel<<<ntiles, kSortBlock, 0, s>>>(kin, vin, kout, vout, n, shift, hist, ntiles);
		}
		VGPU_CUDA(cudaGetLastError());
		std::swap(kin, kout);
		vin = vout;
		std::swap(vout, vspare);
	}
	if (kin != keys) {
		VGPU_CUDA(cudaMemcpyAsync(keys, kin, n * 8, cudaMemcpyDeviceToDevice, s));
		VGPU_CUDA(cudaMemcpyAsync(values, vin, n * 4, cudaMemcpyDeviceToDevice, s));
	}
}

void JoinExpand(const uint64_t *offsets, const uint64_t *lower, uint64_t n_left, const uint32_t *sorted_perm,
                uint64_t total, uint32_t *out_left, uint32_t *out_right, cudaStream_t stream) {
	if (total == 0) return;
	LaunchScope scope("join_expand", stream, total * 8, total);
	const uint64_t tiles = (total + kExpandTile - 1) / kExpandTile;
	const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(tiles, 148ull * 8));
	JoinExpandKernel<<<grid, kExpandBlock, 0, stream>>>(offsets, lower, n_left, sorted_perm, total, out_left, out_right);
	VGPU_CUDA(cudaGetLastError());
}

void JoinRuns(const void *keys, size_t kwidth, uint64_t n, const JoinRunsView &view, uint64_t *lower, uint64_t *count,
              cudaStream_t stream) {
	if (n == 0) return;
	LaunchScope scope("join_runs", stream, n * (kwidth + 16), n);
	WithKeys(keys, kwidth, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		JoinRunKernel<K><<<GridFor(n, 256), 256, 0, stream>>>(k, n, view, lower, count);
	});
	VGPU_CUDA(cudaGetLastError());
}

void JoinDenseRuns(const void *keys, size_t kwidth, uint64_t n, uint64_t bias, uint64_t range, uint64_t *entries,
                   uint32_t *rows, uint32_t *list, uint32_t *info, cudaStream_t stream) {
	LaunchScope scope("join_runs_dense", stream, n * (2 * kwidth + 4) + (range + 1) * 8, n);
	auto *e = reinterpret_cast<uint2 *>(entries);
	VGPU_CUDA(cudaMemsetAsync(entries, 0, (range + 1) * 8, stream));
	VGPU_CUDA(cudaMemsetAsync(info, 0, 12, stream));
	WithKeys(keys, kwidth, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		JoinEntryCountKernel<K><<<GridFor(n, 256), 256, 0, stream>>>(k, n, bias, e, info);
		JoinEntryPlaceKernel<<<GridFor((range + 1024) / 4, 256), 256, 0, stream>>>(e, range + 1, info);
		JoinEntryFillKernel<K><<<GridFor(n, 256), 256, 0, stream>>>(k, n, bias, e, rows, info);
	});
	JoinEntrySortKernel<<<GridFor(range + 1, 256), 256, 0, stream>>>(e, range + 1, rows, list, info);
	JoinEntrySortLongKernel<<<Runtime::Get().props().sm_count * 2, 256, 0, stream>>>(e, rows, list, info);
	VGPU_CUDA(cudaGetLastError());
}

uint64_t WaitLimitNs() {
	const char *env = std::getenv("VGPU_WAIT_LIMIT_NS");
	return env ? std::min<uint64_t>(std::strtoull(env, nullptr, 10), 10000000000ull) : 2000000000ull;
}

uint64_t JoinChainWords(uint64_t n_left) {
	const uint64_t tiles = (n_left + kJoinTile - 1) / kJoinTile;
	return 2 + (tiles + 1) / 2 + tiles;
}

void JoinCountMatches(const void *keys, size_t kwidth, uint64_t n, const JoinRunsView &view, uint64_t *chain,
                      cudaStream_t stream) {
	LaunchScope scope("join_count", stream, n * kwidth, n);
	const uint64_t tiles = (n + kJoinTile - 1) / kJoinTile;
	VGPU_CUDA(cudaMemsetAsync(chain, 0, JoinChainWords(n) * 8, stream));
	const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(tiles + 1, static_cast<uint64_t>(Runtime::Get().props().sm_count) * 8));
	WithKeys(keys, kwidth, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		JoinMatchCountKernel<K><<<grid, kJoinBlock, 0, stream>>>(k, n, view, tiles, chain, WaitLimitNs());
	});
	VGPU_CUDA(cudaGetLastError());
}

void JoinEmit(const void *keys, size_t kwidth, uint64_t n, const JoinRunsView &view, const uint64_t *chain,
              const uint32_t *rows, const JoinOuts &outs, uint64_t total, uint32_t longest, cudaStream_t stream) {
	// CTAs that share a tile's matches (and each find all of its runs): a few left rows with many matches each are
	// otherwise left to as few CTAs (15600 left rows with 64 each: 0.28 -> 0.03 ms)
	const uint32_t parts = std::max<uint32_t>(1, longest / 4096);
	uint64_t row_bytes = 0;
	for (int c = 0; c < outs.n; c++) row_bytes += outs.c[c].width;
	LaunchScope scope("join_emit", stream, n * kwidth + 2 * total * row_bytes, total);
	const uint64_t tiles = (n + kJoinTile - 1) / kJoinTile;
	const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(tiles * parts, static_cast<uint64_t>(Runtime::Get().props().sm_count) * 8));
	WithKeys(keys, kwidth, [&](auto *k) {
		using K = std::remove_const_t<std::remove_pointer_t<decltype(k)>>;
		JoinEmitKernel<K><<<grid, kJoinBlock, 0, stream>>>(k, n, view, tiles, chain + 2 + (tiles + 1) / 2, rows, outs, parts);
	});
	VGPU_CUDA(cudaGetLastError());
}

// ---- running total (the stream pipeline's RUNNING_SUM window primitive) ----------------------------
//
// Three passes over tiles of 4096 values (1024 threads x 4 consecutive values): each tile's total; one
// block turning the totals into per-tile starting values that continue from the carried state; each
// tile's inclusive scan from its starting value. Integer values are summed as unsigned words of at
// least their width (wrap-around, truncated on store), floats in their own type.

namespace {

constexpr int kSumThreads = 1024;
constexpr int kSumItems = 4;
constexpr uint64_t kSumTile = uint64_t(kSumThreads) * kSumItems;

template <class T, class A> __device__ __forceinline__ A SumLoad(const T *p) {
	if constexpr (sizeof(T) == 2) {
		return static_cast<A>(static_cast<uint16_t>(*p));
	} else if constexpr (std::is_integral<T>::value) {
		return static_cast<A>(*p);
	} else {
		return *p;
	}
}

template <class T, class A> __device__ __forceinline__ void SumStore(T *p, A v) {
	*p = static_cast<T>(v);
}

// Block-wide scan of one value per thread (1024 threads): inclusive and exclusive prefixes and the
// block total, all in the same addition order.
template <class A> __device__ void SumBlockScan(A x, A *warp_sums, A &incl, A &excl, A &total) {
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5;
	for (int d = 1; d < 32; d <<= 1) {
		const A y = __shfl_up_sync(0xffffffffu, x, d);
		if (lane >= d) x = static_cast<A>(x + y);
	}
	A prev = __shfl_up_sync(0xffffffffu, x, 1);
	if (lane == 31) warp_sums[warp] = x;
	__syncthreads();
	if (warp == 0) {
		A w = warp_sums[lane];
		for (int d = 1; d < 32; d <<= 1) {
			const A y = __shfl_up_sync(0xffffffffu, w, d);
			if (lane >= d) w = static_cast<A>(w + y);
		}
		warp_sums[lane] = w;
	}
	__syncthreads();
	if (warp == 0) {
		incl = x;
		excl = lane == 0 ? A(0) : prev;
	} else {
		const A before = warp_sums[warp - 1];
		incl = static_cast<A>(before + x);
		excl = lane == 0 ? before : static_cast<A>(before + prev);
	}
	total = warp_sums[31];
	__syncthreads();  // warp_sums is rewritten by the next call
}

template <class T, class A>
__global__ void __launch_bounds__(kSumThreads) SumTileTotalsKernel(const T *data, uint64_t rows, A *totals) {
	__shared__ A warp_sums[32];
	const uint64_t base = blockIdx.x * kSumTile + uint64_t(threadIdx.x) * kSumItems;
	A s = A(0);
	for (int j = 0; j < kSumItems; j++) {
		if (base + j < rows) s = static_cast<A>(s + SumLoad<T, A>(data + base + j));
	}
	A incl, excl, total;
	SumBlockScan(s, warp_sums, incl, excl, total);
	if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

// One block: totals[i] becomes the value before tile i (the carried state plus the tiles before it).
template <class T, class A>
__global__ void __launch_bounds__(kSumThreads) SumTileStartsKernel(A *totals, uint64_t tiles, const T *state) {
	__shared__ A warp_sums[32];
	A carry = SumLoad<T, A>(state);
	for (uint64_t c = 0; c < tiles; c += kSumThreads) {
		const uint64_t i = c + threadIdx.x;
		const A x = i < tiles ? totals[i] : A(0);
		A incl, excl, chunk;
		SumBlockScan(x, warp_sums, incl, excl, chunk);
		if (i < tiles) totals[i] = static_cast<A>(carry + excl);
		carry = static_cast<A>(carry + chunk);
	}
}

template <class T, class A>
__global__ void __launch_bounds__(kSumThreads) SumTileScanKernel(T *data, uint64_t rows, const A *starts, T *state) {
	__shared__ A warp_sums[32];
	const uint64_t base = blockIdx.x * kSumTile + uint64_t(threadIdx.x) * kSumItems;
	A v[kSumItems];
	A s = A(0);
	for (int j = 0; j < kSumItems; j++) {
		v[j] = base + j < rows ? SumLoad<T, A>(data + base + j) : A(0);
		s = static_cast<A>(s + v[j]);
	}
	A incl, excl, total;
	SumBlockScan(s, warp_sums, incl, excl, total);
	A run = static_cast<A>(starts[blockIdx.x] + excl);
	for (int j = 0; j < kSumItems; j++) {
		run = static_cast<A>(run + v[j]);
		if (base + j < rows) {
			SumStore<T, A>(data + base + j, run);
			if (base + j == rows - 1) SumStore<T, A>(state, run);
		}
	}
}

template <class T, class A> void RunningSumTyped(void *data, uint64_t rows, void *state, void *scratch, cudaStream_t stream) {
	const uint64_t tiles = (rows + kSumTile - 1) / kSumTile;
	T *d = static_cast<T *>(data);
	T *st = static_cast<T *>(state);
	A *sums = static_cast<A *>(scratch);
	SumTileTotalsKernel<T, A><<<static_cast<unsigned>(tiles), kSumThreads, 0, stream>>>(d, rows, sums);
	SumTileStartsKernel<T, A><<<1, kSumThreads, 0, stream>>>(sums, tiles, st);
	SumTileScanKernel<T, A><<<static_cast<unsigned>(tiles), kSumThreads, 0, stream>>>(d, rows, sums, st);
	VGPU_CUDA(cudaGetLastError());
}

} // namespace

size_t RunningSumScratchBytes(uint64_t rows) {
	return static_cast<size_t>((rows + kSumTile - 1) / kSumTile) * sizeof(uint64_t) + 16;
}

void RunningSum(void *data, ValueType t, uint64_t rows, void *state, void *scratch, cudaStream_t stream) {
	if (rows == 0) return;
	if (rows >= (1ull << 32)) Fail(VGPU_ERR_INVALID_ARGUMENT, "running sum: at most 2^32 - 1 rows per call");
	LaunchScope scope("vgpu_running_sum", stream, 2 * rows * TypeSize(t) + rows * TypeSize(t), rows);
	switch (t) {
	case ValueType::INT16:
		RunningSumTyped<int16_t, uint32_t>(data, rows, state, scratch, stream);
		break;
	case ValueType::INT32:
		RunningSumTyped<int32_t, uint32_t>(data, rows, state, scratch, stream);
		break;
	case ValueType::INT64:
		RunningSumTyped<int64_t, uint64_t>(data, rows, state, scratch, stream);
		break;
	case ValueType::FLOAT32:
		RunningSumTyped<float, float>(data, rows, state, scratch, stream);
		break;
	case ValueType::FLOAT64:
		RunningSumTyped<double, double>(data, rows, state, scratch, stream);
		break;
	default:
		Fail(VGPU_ERR_UNSUPPORTED, std::string("running sum: unsupported type ") + TypeName(t));
	}
}

} // namespace kern
} // namespace vgpu
