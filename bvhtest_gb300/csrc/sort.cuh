// Internal interface of the onesweep radix sort (sort.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace bvhgb {
// Sets the kernels' shared-memory attributes; call once before any stream capture.
int sort_prepare();
// Scratch bytes for sorting n pairs on key bits [beginBit, endBit).
size_t sort_temp_bytes(uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit);
// Device word that the look-back sets to a non-zero error bit if a bounded wait gives up.
uint32_t *sort_error_word(void *temp, uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit);
// Stable ascending sort; temp must hold sort_temp_bytes(...) bytes. tileKeys = keys per CTA of the
// onesweep passes (2048, 4096 or 8192; the result does not depend on it); 0 takes the process-wide
// setting (bvhgb_sort_set_default_tile), which leaves the choice to the number of pairs unless it was changed.
constexpr uint32_t kSortTileDefault = 8192;  // the batched pipeline's, and the choice for the largest sorts
bool sort_tile_valid(uint32_t tileKeys);
// Polls of an unpublished predecessor before a look-back gives up (0xFFFFFFFF: the default).
int sort_set_spin_limit(uint32_t limit, uint32_t *previous);
// The lowest bit of a Morton cell: 2^32 cells for up to 8M triangles, 2^40 for more (the densest cells of the
// benchmark scenes then hold a few dozen; 33.5M triangles in 64 clusters put over 256 into some of 2^32).
__host__ __device__ constexpr uint32_t morton_cell_bit(uint32_t n) { return n <= (1u << 23) ? 31u : 23u; }
// A hashed table that the kernel making the keys counts every cell_sample(n)-th one's cell in. The sort raises
// *heavy where a count is heavy_cell(n) or more (groups of about 320, 448 and 640 keys). Null and 0: none.
__host__ __device__ constexpr uint32_t cell_sample(uint32_t n) { return n <= (1u << 20) ? 16u : n <= (1u << 23) ? 32u : 64u; }
__host__ __device__ constexpr uint32_t heavy_cell(uint32_t n) { return n <= (1u << 20) ? 20u : n <= (1u << 23) ? 14u : 10u; }
struct MortonCells {
  const uint32_t *count = nullptr;
  uint32_t words = 0;
  uint32_t *heavy = nullptr;
};
// The stable ascending sort of n 63-bit Morton keys; temp as for sort_pairs on bits [0, 63). *gate
// and *cells.heavy (device) are 0 after; where they are not before, the full sort makes the order. *route
// receives how it was made: 0 by the upper bits and their groups, 1 by the full sort after a long group, 2 by the full
// sort at once, for a full cell (not written up to 4,096 pairs).
int sort_morton(void *temp, const uint64_t *keysIn, uint64_t *keysOut, const uint32_t *valsIn, uint32_t *valsOut,
                uint32_t n, uint32_t *gate, uint32_t *route, const MortonCells &cells, cudaStream_t s);
// The sort's alternate buffers, (keyBytes + 4) * n bytes of the temp space that hold nothing between sorts.
void *sort_alternate(void *temp, uint32_t n, uint32_t keyBytes, uint32_t beginBit, uint32_t endBit);
int sort_pairs(void *temp, const void *keysIn, void *keysOut, const uint32_t *valsIn, uint32_t *valsOut, uint32_t n,
               uint32_t keyBytes, uint32_t beginBit, uint32_t endBit, cudaStream_t s, uint32_t tileKeys = 0);
// The values of the first k pairs of a stable ascending sort of (keys, vals), 32-bit keys, in that
// order, into valsOut[0, k) (k <= n), without sorting all n pairs; temp must hold
// select_temp_bytes(n, k) bytes.
size_t select_temp_bytes(uint32_t n, uint32_t k);
int select_smallest(void *temp, const uint32_t *keys, const uint32_t *vals, uint32_t n, uint32_t k, uint32_t *valsOut,
                    cudaStream_t s, uint32_t tileKeys = 0);

// The same for many segments of one key array at once: segment g keeps its keep[g] smallest keys (ties
// in index order), in index order, as (g << 32 | key, index within the segment) from place outOff[g] on.
// A stable sort of the kept pairs is then every segment's prefix of its own stable sort. Segments
// without a row keep all their keys. All arrays are on the device.
constexpr uint32_t kSegTile = 8192, kSegThreads = 512, kSegBins = 2048;
struct SegTile {
  uint32_t seg, start, len, local;  // keys [start, start + len); 'local' is the first one's index in its segment
};
struct SegSelect {
  uint32_t segs, tiles, rows;  // rows: segments that select
  const SegTile *tile;         // in order, tileOff[g] .. tileOff[g + 1] - 1 for segment g
  const uint32_t *tileOff, *row, *rowSeg, *keep, *outOff;  // row[g] or kNone; rowSeg[row] = g
  uint2 *state;                // per row: digits of the threshold found so far, keys below them
  uint2 *count;                // per tile: keys below and at the threshold
};
// hist: rows x kSegBins counts of the keys' upper 11 bits (cleared on return).
int select_segments(const SegSelect &q, const uint32_t *keys, uint32_t *hist, uint64_t *outKeys, uint32_t *outVals,
                    cudaStream_t s);
#ifdef __CUDACC__
// Adds one key per lane (bin 0xFFFFFFFF: none) to a block's counts; lanes with the same bin add together.
__device__ __forceinline__ void count_bin(uint32_t *bins, uint32_t bin) {
  const uint32_t peers = __match_any_sync(0xFFFFFFFFu, bin);
  if (bin != 0xFFFFFFFFu && (peers & ((1u << (threadIdx.x & 31u)) - 1u)) == 0u) atomicAdd(&bins[bin], (uint32_t)__popc(peers));
}
#endif
}  // namespace bvhgb
