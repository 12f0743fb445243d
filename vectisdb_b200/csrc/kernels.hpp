// kernels.hpp -- precompiled (nvcc, sm_100a) device primitives used by the executor. Every entry
// point launches on the given stream, takes temporaries from the given arena and never synchronizes.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#include "runtime.hpp"

namespace vgpu {
namespace kern {

//! out[i] = sum(in[0..i)), *total = sum(in) (device scalar). In-place (out == in) is allowed.
void ExclusiveScanU32(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *total, Arena &arena);
void ExclusiveScanU64(const uint64_t *in, uint64_t *out, uint64_t n, uint64_t *total, Arena &arena);

//! Running total in place: data[i] = *state + data[0] + ... + data[i] for `rows` values of type `t`
//! (INT16/INT32/INT64 wrapping in their width, FLOAT32/FLOAT64 in their own precision), then
//! *state = data[rows - 1] (device scalar of type `t`), so consecutive calls continue one total.
//! `scratch` holds RunningSumScratchBytes(rows) bytes. Three launches, no host synchronization.
size_t RunningSumScratchBytes(uint64_t rows);
void RunningSum(void *data, ValueType t, uint64_t rows, void *state, void *scratch, cudaStream_t stream);

//! Arrow LSB-first bitmap <-> one byte per row.
void UnpackValidity(const uint8_t *bitmap, uint8_t *bytes, uint64_t n, cudaStream_t stream);
void PackValidity(const uint8_t *bytes, uint8_t *bitmap, uint64_t n, cudaStream_t stream);

//! dst[o] = src[idx[o]] for `width`-byte values (1, 2, 4, 8 or 16).
void Gather(const void *src, size_t width, const uint32_t *idx, uint64_t n, void *dst, cudaStream_t stream);

//! Several buffers copied in one launch per kMaxCopies of them: sources and destinations 16-byte aligned, with room up
//! to the next multiple of 16 bytes.
constexpr int kMaxCopies = 24;
struct BufferCopy {
	const void *src;
	void *dst;
	uint64_t bytes;
};
void CopyBuffers(const BufferCopy *copies, int n, cudaStream_t stream);

//! Raw key bits zero-extended to 64 bits (the reference's WidenKeyKernel semantics,
//! cuda_engine/src/operators/gpu_groupby.cu:76-94), minus `bias`.
void WidenKeys(const void *src, size_t width, uint64_t n, uint64_t bias, uint64_t *dst, cudaStream_t stream);

//! How a column's values are read for ColumnBounds (BOOL: one byte, zero or not).
enum class BoundsKind : int { U8, U16, U32, U64, I16, I32, I64, BOOL };
constexpr int kMaxBoundsColumns = 8;
struct BoundsColumn {
	const void *data;
	uint64_t rows;
	BoundsKind kind;
};
inline size_t BoundsWidth(BoundsKind k) {
	return k == BoundsKind::U8 || k == BoundsKind::BOOL ? 1 : k == BoundsKind::U16 || k == BoundsKind::I16 ? 2
	       : k == BoundsKind::U32 || k == BoundsKind::I32 ? 4 : 8;
}
//! The unsigned kind of a `width`-byte column's raw bits, zero-extended.
inline BoundsKind RawBoundsKind(size_t width) {
	return width == 1 ? BoundsKind::U8 : width == 2 ? BoundsKind::U16 : width == 4 ? BoundsKind::U32 : BoundsKind::U64;
}
//! The kind of an integer, boolean or dictionary column's values.
BoundsKind SignedBoundsKind(ValueType t);
//! Smallest and largest value of each of `n` columns, one launch per kMaxBoundsColumns of them: two words
//! per column in `out` (device, 2n words), read back with BoundsLow / BoundsHigh. A column without rows
//! gives the largest value of its 64-bit kind as the smallest and the other way round.
//! With `distinct`, kDistinctRanks 32-bit ranks per column follow in `out` (BoundsWords in all), from which
//! DistinctEstimate (on the words read back) gives about how many distinct values a 4- or 8-byte column has
//! (within some 7%; 0 for narrower ones).
//! With `pairs` (2n words) instead, also how many pairs of values far apart it looked at, [2c + 1], and how many of those were
//! equal, [2c]: their share is the chance that two rows have the same value.
void ColumnBounds(const BoundsColumn *cols, int n, uint64_t *out, cudaStream_t stream, bool distinct = false,
                  uint64_t *pairs = nullptr);
constexpr int kDistinctRanks = 256;
inline size_t BoundsWords(int n, bool distinct) {
	return static_cast<size_t>(n) * (2 + (distinct ? kDistinctRanks / 2 : 0));
}
uint64_t DistinctEstimate(const uint64_t *words, int n, int column, BoundsKind kind);
inline bool BoundsSigned(BoundsKind k) {
	return k == BoundsKind::I16 || k == BoundsKind::I32 || k == BoundsKind::I64;
}
//! The column's bounds as the 64-bit pattern of its value (two's complement for the signed kinds).
inline uint64_t BoundsLow(const uint64_t *words, BoundsKind k) {
	return ~words[0] ^ (BoundsSigned(k) ? 1ull << 63 : 0ull);
}
inline uint64_t BoundsHigh(const uint64_t *words, BoundsKind k) {
	return words[1] ^ (BoundsSigned(k) ? 1ull << 63 : 0ull);
}

//! Stable LSD radix sort of keys over their low `bits` bits (8-bit digits), `values` becoming the sorted
//! keys' positions in the input. Results end in (keys, values); (keys_alt, values_alt) are the ping-pong buffers.
void RadixSortPairs(uint64_t *keys, uint32_t *values, uint64_t *keys_alt, uint32_t *values_alt, uint64_t n, int bits,
                    Arena &arena);

void Iota(uint32_t *out, uint64_t n, cudaStream_t stream);

//! Left row i owns outputs [offsets[i], offsets[i + 1]) (offsets ascending, offsets[0] = 0): output o
//! becomes (i, sorted_perm[lower[i] + o - offsets[i]]). Load-balanced: fixed tiles of outputs per CTA,
//! the left rows a tile spans staged in shared memory.
void JoinExpand(const uint64_t *offsets, const uint64_t *lower, uint64_t n_left, const uint32_t *sorted_perm,
                uint64_t total, uint32_t *out_left, uint32_t *out_right, cudaStream_t stream);

//! Where a left key's right rows are: dense keys by an entry per key value (JoinDenseRuns), else a sorted key
//! array with its radix directory (`entries` null).
struct JoinRunsView {
	const uint64_t *entries = nullptr;
	const uint64_t *sorted = nullptr;
	const uint32_t *dir = nullptr;
	uint64_t nb = 0;  // entries, or directory buckets
	uint64_t bias = 0;
	uint32_t shift = 0;
	const uint32_t *info = nullptr;  // of JoinDenseRuns, with entries: the count does nothing when a run is too long
};
//! For each left row (raw keys): the first place of its run in the right rows' order, and the run's length.
void JoinRuns(const void *keys, size_t kwidth, uint64_t n, const JoinRunsView &view, uint64_t *lower, uint64_t *count,
              cudaStream_t stream);
//! Longest run JoinDenseRuns puts in row order.
constexpr uint32_t kJoinRunLimit = 4096;
//! The rows of each key value contiguous in `rows` [n], in row order, and an entry per value of the range (range
//! + 1 words of `entries`), without sorting the keys. `list` [n / 17 + 1] and `info` [3] are scratch; info[1]
//! becomes the longest run's length, or one past kJoinRunLimit as soon as a run is: the rest is then left out, and the
//! caller sorts instead.
void JoinDenseRuns(const void *keys, size_t kwidth, uint64_t n, uint64_t bias, uint64_t range, uint64_t *entries,
                   uint32_t *rows, uint32_t *list, uint32_t *info, cudaStream_t stream);
//! Longest wait in ns of a kernel for tiles counted in the same launch (VGPU_WAIT_LIMIT_NS, for testing: up to 10 s;
//! with 0 every wait that is not over at its first look runs out).
uint64_t WaitLimitNs();
//! Matches of the left rows (raw keys): chain [JoinChainWords] = the total (bits 62 and 63 set when a tile has 2^31
//! or a wait ran out), [1] >> 32 = the most matches of one tile of left rows, then the tiles' starts for JoinEmit.
uint64_t JoinChainWords(uint64_t n_left);
void JoinCountMatches(const void *keys, size_t kwidth, uint64_t n, const JoinRunsView &view, uint64_t *chain,
                      cudaStream_t stream);
struct JoinOut {
	const void *src;
	void *dst;
	int width;   // 1, 2, 4, 8 or 16
	bool right;  // a column of the right side
};
constexpr int kMaxJoinOuts = 16;
struct JoinOuts {
	JoinOut c[kMaxJoinOuts];
	int n = 0;
};
//! Every output column of the matches, left rows in order and each one's matches in the order of `rows`; without
//! `rows` the right columns are in that order themselves. `longest`: the most matches of one tile.
void JoinEmit(const void *keys, size_t kwidth, uint64_t n, const JoinRunsView &view, const uint64_t *chain,
              const uint32_t *rows, const JoinOuts &outs, uint64_t total, uint32_t longest, cudaStream_t stream);

//! Radix directory of a sorted (biased) key array: dir[b] = first position whose key >> shift >= b,
//! for b in [0, nb]; dir needs nb + 1 entries and nb must exceed every key >> shift.
void JoinDirectory(const uint64_t *sorted, uint64_t n, uint32_t shift, uint64_t nb, uint32_t *dir, cudaStream_t stream);
//! Dense join table over the raw keys (`kwidth` bytes, zero-extended) minus `bias` (their minimum), all <=
//! `range`: range + 1 entries of `width` bytes, built without sorting. Without values (width 4): row index
//! + 1 of the key's row, 0 = no key. With a 1-, 2- or 4-byte value column: width 8 holds (1 << 32 | value
//! bits), 0 = no key; width 1, 2 or 4 holds value bits - vmin, all ones = no key (every value's offset must
//! stay below that marker). *occupied = entries written: below n when a key repeats, and the table is then
//! not a valid lookup.
void JoinDenseFill(const void *keys, size_t kwidth, const void *values, size_t vwidth, uint64_t n, uint64_t bias,
                   uint64_t range, uint32_t vmin, void *table, size_t width, uint32_t *occupied, cudaStream_t stream);
//! Dense multi-match table over the same keys, built without sorting, for a join that contributes
//! one right column of at most 4 bytes: entry[k] (4 bytes, or 8 when `wide`) holds k's match count in its
//! low `cbits` bits (1..3) and one `vbits`-bit slot per match above them, each the value bits - vmin. A key
//! with more than `rmax` matches (rmax < 2^cbits, cbits + rmax * vbits within the entry) counts in
//! *overflow, and the table is then not valid.
void JoinDenseMulti(const void *keys, size_t kwidth, const void *values, size_t vwidth, uint64_t n, uint64_t bias,
                    uint64_t range, uint32_t vmin, uint32_t vbits, uint32_t cbits, uint32_t rmax, void *table, bool wide,
                    uint32_t *overflow, cudaStream_t stream);
//! *out = number of positions i > 0 with sorted[i] == sorted[i - 1].
void CountAdjacentEqual(const uint64_t *sorted, uint64_t n, uint32_t *out, cudaStream_t stream);
//! *out = the length of the longest run of equal keys in `sorted` (saturating at 2^32 - 1).
void MaxRunLength(const uint64_t *sorted, uint64_t n, uint32_t *out, cudaStream_t stream);

//! Counts of a sample by how often its keys were seen; zeroed by the caller of HeavySelect.
struct HeavyScratch {
	uint32_t hist[1024];
	uint64_t sampled;
	uint32_t listed, pad;
};
//! Work list of a partitioned aggregation pass over `P` partitions whose row ranges start at
//! offsets[p * stride] (the last ends at *total_rows): 16-byte items (partition, first row, end row,
//! split index or ~0u), longest first, into `items` (capacity PlanWorkCapacity). Partitions larger
//! than max(min_split, ceil(total / (4 * ctas))) rows are split into chunks (so at most 4 * ctas and
//! at most total / min_split partitions are split); chunks of one partition share a
//! split index s with split_info[2s] = chunk count and split_info[2s+1] = 0 (a completion counter).
//! counts[0] = items, counts[1] = split partitions (split_info is written for the first max_split),
//! counts[3] = *total_rows.
//! Heavy keys of a direct-partitioned group-by from a sample: sample_keys/sample_counts ([SC], key ~0
//! = empty) hold the sampled rows' mixed keys and counts. Keys seen at least
//! t times, t >= min_count the smallest threshold that selects at most K keys, claim their
//! partition (key >> dbits; the first claim wins, one heavy key per partition): hmap[p] = (index << 16)
//! | (key & (2^dbits - 1)), heavy_keys[index] = key, *n_heavy = keys selected. hmap must hold ~0 on
//! entry. With require_cover, a selection covering under a tenth of the sampled rows is dropped. `list`:
//! scratch for SC entries.
void HeavySelect(const uint64_t *sample_keys, const uint32_t *sample_counts, uint32_t SC, HeavyScratch *scratch,
                 uint64_t *list, uint32_t *hmap, uint32_t dbits, uint32_t *heavy_keys, uint32_t K, uint32_t min_count,
                 bool require_cover, uint32_t *n_heavy, cudaStream_t stream);
uint64_t PlanWorkCapacity(uint32_t P, uint64_t rows, uint32_t min_split);
void PlanWork(const uint32_t *offsets, uint64_t stride, uint32_t P, const uint32_t *total_rows, uint32_t min_split,
              uint32_t ctas, void *items, uint32_t *counts, uint32_t *split_info, uint32_t max_split,
              cudaStream_t stream);

} // namespace kern
} // namespace vgpu
