// Resident-order sorts: a stable LSD radix sort of (key, value) pairs with
// 8-bit digits (uploads and the P2P mode's per-step sort), and the leaf
// counting sort that refreshes the order of resident bodies.
//
// The radix sort orders bodies by (scene, Morton leaf key) so each leaf's bodies are
// contiguous: leaf membership and occupancy then come from runs of equal
// keys, and the deposit is a segmented reduction over those runs.  The sort
// is stable, so the resident order is a deterministic function of the input.
//
// One launch per 8-bit pass (k_sort_pass).  The digit totals of every pass
// come with the keys (k_keys counts them), so a tile only needs the counts of
// the tiles before it: tiles are numbered by a ticket, publish their digit
// counts and look back over their predecessors' (Merrill & Garland,
// "Single-pass parallel prefix scan with decoupled look-back", 2016).  Ranks
// inside a tile come from eight ballots per key and per-warp digit counters
// (a match over 32 distinct digits takes about 230 cycles, the ballots about
// 40), and a tile is put in digit order in shared memory before it is
// written, so the stores run along digit runs.  What bounds a pass: memory
// at millions of keys, latency (ticket, loads, ranks, look-back) below.
// With histogram, scan and scatter launches per pass and separate fills of the
// tree buffers before -> now, upload with sort and deposit, us: 4,096 bodies
// 91 -> 18, 65,536 99 -> 25, 250,000 107 -> 43, 1,048,576 147 -> 104,
// 5,242,880 539 -> 432; with the caller's buffer read in place and what else
// k_gather says, 18, 22, 37, 78 and 306.
#include <cuda_runtime.h>

#include "rfmm_device.cuh"
#include "rfmm_kernels.h"

namespace rfmm {

constexpr uint32_t kSortThreads = 256u;
constexpr uint32_t kSortWarps = kSortThreads / 32u;

// Keys per thread of a tile: many small tiles while they fit the GPU twice
// over (latency), large ones beyond (fewer look-backs, longer digit runs;
// 8 / 12 / 16 keys at 5,242,880 bodies: 479 / 453 / 438 us per upload).
constexpr uint32_t kSortItemsSmall = 4u, kSortItemsLarge = 16u;
constexpr uint32_t kSortSmallTiles = 304u;  // 2 per SM
static uint32_t sort_tiles(uint32_t n) {
  const uint32_t small = (n + kSortThreads * kSortItemsSmall - 1u) / (kSortThreads * kSortItemsSmall);
  if (small <= kSortSmallTiles) return small;
  return (n + kSortThreads * kSortItemsLarge - 1u) / (kSortThreads * kSortItemsLarge);
}
size_t sort_status_words(uint32_t capacity) {
  const uint32_t t = sort_tiles(capacity);
  return 256u * (size_t)(t < kSortSmallTiles ? kSortSmallTiles : t);  // smaller sorts may use more tiles
}

// Block-wide exclusive scan of one value per thread (256 threads).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *warp_sums) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (uint32_t off = 1u; off < 32u; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31u) warp_sums[warp] = x;
  __syncthreads();
  uint32_t before = 0u;
#pragma unroll
  for (uint32_t w = 0; w < kSortWarps; w++)
    if (w < warp) before += warp_sums[w];
  __syncthreads();
  return before + x - v;
}

// A tile's published count of one digit: bits 0-31 the count, 32-33 what it
// is, 34-63 the pass it belongs to (SortState::epoch, so words left by earlier
// passes read as absent).
constexpr uint32_t kSortOwn = 1u;   // the tile's own count
constexpr uint32_t kSortUpTo = 2u;  // the count of every tile up to this one
// Top bit of a count up to a tile: that tile, or one before it, gave up
// waiting.  (Counts stay below 2^31.  As a fourth kind of word, told apart in
// the look-back's loop, it took 0.5 us a pass at 65,536 keys.)
constexpr uint32_t kSortFailed = 0x80000000u;
constexpr uint32_t kSortPolls = 1u << 22;  // polls of a tile's wait for its predecessors, a few seconds
__device__ __forceinline__ unsigned long long sort_word(uint32_t epoch, uint32_t kind, uint32_t count) {
  return ((unsigned long long)((epoch << 2) | kind) << 32) | count;
}

template <uint32_t kItems>
__global__ void __launch_bounds__(kSortThreads) k_sort_pass(
    const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in,
    const uint32_t *__restrict__ tile_map, uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out,
    uint32_t n, uint32_t shift, uint32_t *__restrict__ totals, unsigned long long *__restrict__ status,
    SortState *__restrict__ state, Counters *__restrict__ ctr, uint32_t max_polls) {
  constexpr uint32_t kTileKeys = kSortThreads * kItems, kAll = 0xFFFFFFFFu;
  __shared__ uint32_t s_key[kTileKeys], s_val[kTileKeys];
  __shared__ uint32_t s_cnt[kSortWarps][256];  // per warp: digit counts, then first rank in the tile
  __shared__ uint32_t s_out[256];              // per digit: output index minus index in the tile
  __shared__ uint32_t s_sums[kSortWarps];
  __shared__ uint32_t s_tile, s_epoch, s_stop;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
#pragma unroll
  for (uint32_t w = 0; w < kSortWarps; w++) s_cnt[w][tid] = 0u;
  grid_dependency_wait();  // keys and totals, or the previous pass, are complete
  if (tid == 0u) {
    s_tile = atomicAdd(&state->ticket, 1u);
    s_epoch = *reinterpret_cast<volatile uint32_t *>(&state->epoch);
    s_stop = 0u;
  }
  const uint32_t total = totals[tid];
  __syncthreads();
  const uint32_t tile = s_tile, epoch = s_epoch;
  const uint32_t base = tile * kTileKeys + warp * 32u * kItems + lane;

  // Warp w holds the tile's keys [32 kItems w, 32 kItems (w + 1)), 32 at a
  // time: first the lanes with the same digit (independent ballots), then the
  // ranks, one 32-key row after the other through the warp's counters.
  uint32_t key[kItems], rank[kItems];
#pragma unroll
  for (uint32_t i = 0; i < kItems; i++) key[i] = base + 32u * i < n ? keys_in[base + 32u * i] : 0u;
#pragma unroll
  for (uint32_t i = 0; i < kItems; i++) {
    uint32_t peers = __ballot_sync(kAll, base + 32u * i < n);
#pragma unroll
    for (uint32_t b = 0; b < 8u; b++) {
      const bool bit = (key[i] >> (shift + b)) & 1u;
      const uint32_t ones = __ballot_sync(kAll, bit);
      peers &= bit ? ones : ~ones;
    }
    rank[i] = peers;
  }
#pragma unroll
  for (uint32_t i = 0; i < kItems; i++) {
    const uint32_t peers = rank[i], below = __popc(peers & ((1u << lane) - 1u));
    const bool valid = base + 32u * i < n;
    uint32_t *c = &s_cnt[warp][(key[i] >> shift) & 255u];
    const uint32_t before = *c;
    __syncwarp();
    if (valid && below == 0u) *c = before + __popc(peers);
    __syncwarp();
    rank[i] = before + below;
  }
  __syncthreads();

  // Values, needed after the look-back (first pass: a key's value is its slot).
  uint32_t val[kItems];
#pragma unroll
  for (uint32_t i = 0; i < kItems; i++) {
    const uint32_t at = base + 32u * i;
    if (vals_in != nullptr) {
      val[i] = at < n ? vals_in[at] : 0u;
    } else {
      val[i] = tile_map != nullptr && at < n ? tile_map[at / kTile] * kTile + at % kTile : at;
    }
  }

  // Thread t: digit t.  Counts per warp become first ranks inside the tile.
  uint32_t count = 0u;
  {
    uint32_t c[kSortWarps];
#pragma unroll
    for (uint32_t w = 0; w < kSortWarps; w++) {
      c[w] = s_cnt[w][tid];
      count += c[w];
    }
    volatile unsigned long long *mine = status + (size_t)tile * 256u + tid;
    *mine = sort_word(epoch, tile == 0u ? kSortUpTo : kSortOwn, count);
    const uint32_t first = block_exclusive_scan(count, s_sums);
    uint32_t run = first;
#pragma unroll
    for (uint32_t w = 0; w < kSortWarps; w++) {
      s_cnt[w][tid] = run;
      run += c[w];
    }
    const uint32_t digit0 = block_exclusive_scan(total, s_sums);
    // Look back until a tile that knows its whole prefix.  Tickets number
    // tiles in the order their CTAs began, so every predecessor is running;
    // the wait is bounded all the same, and a tile that gives up, or finds that
    // one before it did, publishes that with its count and writes nothing.
    uint32_t before = 0u;
    if (tile != 0u) {
      // Four predecessors per round trip, nearest first (1 / 4 / 8 / 16 at
      // 1,048,576 bodies: 109 / 104 / 105 / 116 us per upload).
      constexpr uint32_t kBack = 4u;
      uint32_t back = tile;  // tiles [back, tile) are counted in `before`
      bool open = true;
      for (uint32_t polls = 0u; open;) {
        unsigned long long w[kBack];
#pragma unroll
        for (uint32_t j = 0; j < kBack; j++)
          w[j] = back > j ? *reinterpret_cast<volatile unsigned long long *>(status + (size_t)(back - 1u - j) * 256u + tid)
                          : 0ull;
        uint32_t used = 0u;
#pragma unroll
        for (uint32_t j = 0; j < kBack; j++) {
          const uint32_t tag = (uint32_t)(w[j] >> 32);
          if (open && used == j && (tag >> 2) == (epoch & 0x3FFFFFFFu) && (tag & 3u) != 0u) {
            before += (uint32_t)w[j];
            used = j + 1u;
            open = (tag & 3u) != kSortUpTo;
          }
        }
        back -= used;
        if (open && used == 0u && ++polls == max_polls) {
          if (atomicCAS(&ctr->error, 0u, (uint32_t)kDevErrSortTimeout) == 0u) ctr->error_info = tile;
          before |= kSortFailed;
          break;
        }
      }
      if (before >= kSortFailed) s_stop = 1u;
      *mine = sort_word(epoch, kSortUpTo, before + count);
    }
    s_out[tid] = digit0 + before - first;
  }
  __syncthreads();

  // Digit order in shared memory, then out along the digit runs.
#pragma unroll
  for (uint32_t i = 0; i < kItems; i++) {
    const uint32_t from = base + 32u * i;
    if (from < n) {
      const uint32_t at = s_cnt[warp][(key[i] >> shift) & 255u] + rank[i];
      s_key[at] = key[i];
      s_val[at] = val[i];
    }
  }
  __syncthreads();
  if (s_stop == 0u) {
    const uint32_t here = min(kTileKeys, n - tile * kTileKeys);
#pragma unroll
    for (uint32_t i = 0; i < kItems; i++) {
      const uint32_t at = i * kSortThreads + tid;
      if (at < here) {
        const uint32_t k = s_key[at], out = s_out[(k >> shift) & 255u] + at;
        if (out < n) {  // defensive: offsets from the counts stay below n
          keys_out[out] = k;
          vals_out[out] = s_val[at];
        }
      }
    }
  }
  // The last CTA leaves the state ready for the next pass: this pass's
  // totals cleared, a new epoch, tickets from zero.
  if (tid == 0u) s_tile = atomicAdd(&state->done, 1u);
  __syncthreads();
  if (s_tile == gridDim.x - 1u) {
    totals[tid] = 0u;
    if (tid == 0u) {
      state->ticket = 0u;
      state->done = 0u;
      state->epoch = epoch + 1u;
    }
  }
}

// Keys keys[0] (and their digit totals, s.totals) are in place; the values
// start as the keys' slots (tile_map: as in launch_keys).
int radix_sort(const LaunchCtx &L, SortScratch &s, uint32_t n, uint32_t bits, const uint32_t *tile_map) {
  const uint32_t ntiles = sort_tiles(n);
  const auto pass = ntiles * kSortThreads * kSortItemsSmall >= n ? k_sort_pass<kSortItemsSmall>
                                                                 : k_sort_pass<kSortItemsLarge>;
  int cur = 0;
  for (uint32_t shift = 0; shift < bits; shift += 8u) {
    launch_step_kernel(L, pass, dim3(ntiles), dim3(kSortThreads), 0, (const uint32_t *)s.keys[cur],
                       (const uint32_t *)(shift == 0u ? nullptr : s.vals[cur]), tile_map, s.keys[cur ^ 1],
                       s.vals[cur ^ 1], n, shift, s.totals + 256u * (shift / 8u), s.status, s.state, L.ctr, kSortPolls);
    cur ^= 1;
  }
  return cur;
}

void launch_sort_wait_check(cudaStream_t stream, uint32_t polls, SortWaitCheck *check) {
  static_assert(SortWaitCheck::kTileKeys == kSortThreads * kSortItemsSmall, "small tiles");
  k_sort_pass<kSortItemsSmall><<<1, kSortThreads, 0, stream>>>(
      check->keys, nullptr, nullptr, check->out_keys, check->out_vals, 3u * SortWaitCheck::kTileKeys, 0u,
      check->totals, check->status, &check->state, &check->ctr, polls);
}

// What the two launches of the check must leave: tiles 1 and 2 marked failed
// for every digit, the output as it was, and the state ready for a next pass.
bool sort_wait_check_failed_closed(const SortWaitCheck &h, uint32_t poison) {
  for (uint32_t i = 0; i < 3u * SortWaitCheck::kTileKeys; i++)
    if (h.out_keys[i] != poison || h.out_vals[i] != poison) return false;
  for (uint32_t i = 256u; i < 3u * 256u; i++)
    if ((uint32_t)(h.status[i] >> 32) != ((SortWaitCheck::kEpoch << 2) | kSortUpTo) ||
        (uint32_t)h.status[i] < kSortFailed)
      return false;
  return h.state.ticket == 0u && h.state.done == 0u && h.state.epoch == SortWaitCheck::kEpoch + 1u;
}

// ------------------------------------------------ leaf counting-sort resort
//
// The periodic refresh of the resident leaf order.  The leaf counts of the
// current positions are already known (integrate deposited them into the next
// step's moments), so bodies are bucketed by leaf with one exclusive scan of
// the counts in Morton order of the leaves and one scatter:
//   k_leaf_block_sums  per 4096-leaf block of a scene, the sum of its counts
//   k_leaf_block_scan  per scene, exclusive scan of its block sums (+ body_off)
//   k_leaf_offsets     per block, exclusive scan of its counts -> first slot of
//                      every leaf (starts, at the scene's cell offset)
//   k_leaf_scatter     every body takes the next slot of its leaf (one atomic
//                      per leaf run of a warp) and moves there with its id
// Bodies of one leaf land in an arbitrary order, which no result depends on:
// each body's update reads only its own state and the tree, and the moment
// sums are exact integers.

namespace {

constexpr uint32_t kLeafBlock = 4096u;
constexpr uint32_t kLeafThreads = 1024u;

__device__ __forceinline__ uint32_t compact3(uint32_t v) {  // inverse of a 3-D bit spread
  v &= 0x09249249u;
  v = (v | (v >> 2)) & 0x030C30C3u;
  v = (v | (v >> 4)) & 0x0300F00Fu;
  v = (v | (v >> 8)) & 0x030000FFu;
  v = (v | (v >> 16)) & 0x000003FFu;
  return v;
}

__device__ __forceinline__ uint32_t spread3s(uint32_t v) {
  v &= 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// Count of the leaf with Morton index m (x in bit 0) of scene S.
__device__ __forceinline__ uint32_t leaf_count(const SceneDesc &S, const uint4 *mom, uint32_t m) {
  const uint32_t D = S.depth;
  const uint32_t x = compact3(m), y = compact3(m >> 1), z = compact3(m >> 2);
  return mom[S.cell_off + level_offset_d(D) + (x | (y << D) | (z << (2u * D)))].x;
}

// Sum over the 1024-thread block (every thread gets the total).
__device__ __forceinline__ uint32_t block_sum_1024(uint32_t v, uint32_t *warp_buf) {
  for (uint32_t off = 16u; off > 0u; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
  __syncthreads();
  if ((threadIdx.x & 31u) == 0u) warp_buf[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = warp_buf[threadIdx.x & 31u];
  for (uint32_t off = 16u; off > 0u; off >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, off);
  return t;
}

}  // namespace

// The leaf-sort kernels walk scene rows: row y is scene y, or, with an
// active-scene list (serving slots), rows y, y + gridDim, ... take the listed
// scenes in turn.
__device__ __forceinline__ uint32_t scene_rows(const uint32_t *scene_list, const Counters *ctr,
                                               uint32_t scenes) {
  return scene_list != nullptr ? min(ctr->scenes_active, scenes) : scenes;
}

__global__ void __launch_bounds__(kLeafThreads) k_leaf_block_sums(const SceneDesc *__restrict__ scenes,
                                                                  uint32_t nscenes,
                                                                  const uint32_t *__restrict__ scene_list,
                                                                  const Counters *__restrict__ ctr,
                                                                  const uint4 *__restrict__ mom,
                                                                  uint32_t *__restrict__ block_sums,
                                                                  uint32_t max_blocks,
                                                                  unsigned long long *__restrict__ stamp) {
  __shared__ uint32_t warp_buf[32];
  grid_dependency_wait();  // the deposit of the current positions is complete
  stamp_begin(stamp);      // first of the resort's four kernels
  const uint32_t rows = scene_rows(scene_list, ctr, nscenes);
  for (uint32_t y = blockIdx.y; y < rows; y += gridDim.y) {
    const uint32_t sc = scene_list != nullptr ? scene_list[y] : y;
    const SceneDesc &S = scenes[sc];
    const uint32_t leaves = 1u << (3u * S.depth);
    const uint32_t base = blockIdx.x * kLeafBlock;
    if (S.n == 0u || base >= leaves) continue;  // block-uniform
    uint32_t v = 0u;
    for (uint32_t k = 0; k < kLeafBlock / kLeafThreads; k++) {
      const uint32_t m = base + k * kLeafThreads + threadIdx.x;
      if (m < leaves) v += leaf_count(S, mom, m);
    }
    v = block_sum_1024(v, warp_buf);
    if (threadIdx.x == 0) block_sums[sc * max_blocks + blockIdx.x] = v;
  }
}

// One warp per scene: exclusive scan of the scene's block sums (at most 64
// blocks: depth <= 6), offset by the scene's first slot.
__global__ void __launch_bounds__(32) k_leaf_block_scan(const SceneDesc *__restrict__ scenes,
                                                        uint32_t nscenes,
                                                        const uint32_t *__restrict__ scene_list,
                                                        const Counters *__restrict__ ctr,
                                                        uint32_t *__restrict__ block_sums,
                                                        uint32_t max_blocks) {
  grid_dependency_wait();
  const uint32_t rows = scene_rows(scene_list, ctr, nscenes);
  for (uint32_t y = blockIdx.x; y < rows; y += gridDim.x) {
    const uint32_t sc = scene_list != nullptr ? scene_list[y] : y;
    const SceneDesc &S = scenes[sc];
    if (S.n == 0u) continue;
    const uint32_t lane = threadIdx.x;
    const uint32_t nb = ((1u << (3u * S.depth)) + kLeafBlock - 1u) / kLeafBlock;
    uint32_t *row = block_sums + sc * max_blocks;
    // Lane l holds blocks 2l and 2l + 1.
    const uint32_t a = 2u * lane < nb ? row[2u * lane] : 0u;
    const uint32_t b = 2u * lane + 1u < nb ? row[2u * lane + 1u] : 0u;
    uint32_t x = a + b;
    for (uint32_t off = 1u; off < 32u; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, off);
      if (lane >= off) x += t;
    }
    const uint32_t before = S.body_off + x - (a + b);
    if (2u * lane < nb) row[2u * lane] = before;
    if (2u * lane + 1u < nb) row[2u * lane + 1u] = before + a;
  }
}

__global__ void __launch_bounds__(kLeafThreads) k_leaf_offsets(const SceneDesc *__restrict__ scenes,
                                                               uint32_t nscenes,
                                                               const uint32_t *__restrict__ scene_list,
                                                               const Counters *__restrict__ ctr,
                                                               const uint4 *__restrict__ mom,
                                                               const uint32_t *__restrict__ block_offs,
                                                               uint32_t max_blocks,
                                                               uint32_t *__restrict__ starts) {
  __shared__ uint32_t warp_sums[32];
  grid_dependency_wait();
  const uint32_t rows = scene_rows(scene_list, ctr, nscenes);
  for (uint32_t y = blockIdx.y; y < rows; y += gridDim.y) {
    const uint32_t sc = scene_list != nullptr ? scene_list[y] : y;
    const SceneDesc &S = scenes[sc];
    const uint32_t leaves = 1u << (3u * S.depth);
    const uint32_t base = blockIdx.x * kLeafBlock;
    if (S.n == 0u || base >= leaves) continue;  // block-uniform
    // Thread t owns leaves base + 4t .. 4t+3 (a contiguous run of the Morton order).
    constexpr uint32_t kPer = kLeafBlock / kLeafThreads;
    uint32_t c[kPer], total = 0u;
    for (uint32_t k = 0; k < kPer; k++) {
      const uint32_t m = base + threadIdx.x * kPer + k;
      c[k] = m < leaves ? leaf_count(S, mom, m) : 0u;
      total += c[k];
    }
    // Exclusive scan of the thread totals across the block.
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = total;
    for (uint32_t off = 1u; off < 32u; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, x, off);
      if (lane >= off) x += t;
    }
    if (lane == 31u) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t v = warp_sums[lane];
      for (uint32_t off = 1u; off < 32u; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, off);
        if (lane >= off) v += t;
      }
      warp_sums[lane] = v;
    }
    __syncthreads();
    uint32_t run = block_offs[sc * max_blocks + blockIdx.x] + (warp ? warp_sums[warp - 1] : 0u) + x - total;
    for (uint32_t k = 0; k < kPer; k++) {
      const uint32_t m = base + threadIdx.x * kPer + k;
      if (m < leaves) starts[S.cell_off + m] = run;
      run += c[k];
    }
    __syncthreads();  // warp_sums is rewritten by the next row
  }
}

// Each CTA moves the bodies of one tile at a time (every tile once, or the
// active tiles of a tile list in turn).  Slots are reserved in two levels so
// a dense leaf (tens of thousands of bodies) sees one global atomic per CTA:
// runs of neighbouring lanes in one leaf reserve their offsets in a
// shared-memory table of the CTA's leaves, then one thread per leaf reserves
// the CTA's whole block of that leaf from `starts`.  (One global atomic per
// run instead: uniform 1,048,576 bodies 19 us per re-sort, but Plummer 152,
// queued on the core leaves.  Two or four tiles per CTA: Plummer 23.2 and
// 24.5, clusters 5,242,880 81 and 92.)  With the re-sort's launches chained,
// a list of the table's used slots instead of scans over it, and lane runs
// instead of a match, before -> now, us: Plummer 1,048,576 32.5 -> 23.2,
// clusters 5,242,880 105 -> 80, 256 scenes 392 -> 318, uniform 65,536 14 -> 10.
constexpr uint32_t kScatterSlots = 2u * kTile;  // > bodies per CTA, so probing always ends

template <bool kList>
__global__ void __launch_bounds__(256) k_leaf_scatter(const SceneDesc *__restrict__ scenes,
                                                      const uint32_t *__restrict__ tile_scene,
                                                      const uint32_t *__restrict__ tile_list,
                                                      const Counters *__restrict__ ctr,
                                                      const float4 *__restrict__ part_in,
                                                      const uint32_t *__restrict__ ids_in,
                                                      float4 *__restrict__ part_out,
                                                      uint32_t *__restrict__ ids_out,
                                                      uint32_t *__restrict__ starts, uint32_t tiles,
                                                      unsigned long long *__restrict__ stamp) {
  constexpr uint32_t kAll = 0xFFFFFFFFu, kNone = 0xFFFFFFFFu;
  __shared__ uint32_t hkey[kScatterSlots], hcnt[kScatterSlots];
  __shared__ uint16_t used[kTile];  // table slots in use
  __shared__ uint32_t nused;
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t i = threadIdx.x; i < kScatterSlots; i += blockDim.x) {
    hkey[i] = kNone;
    hcnt[i] = 0u;
  }
  if (threadIdx.x == 0u) nused = 0u;
  grid_dependency_wait();  // the leaves' first slots are known
  const uint32_t ntiles = kList ? min(ctr->tiles_active, tiles) : tiles;
  // Without a list the grid has one tile per CTA: the loop runs once.
  for (uint32_t i = blockIdx.x; i < ntiles; i += kList ? gridDim.x : ntiles) {
    const uint32_t tile = kList ? tile_list[i] : i;
    const SceneDesc &S = scenes[tile_scene[tile]];
    const uint32_t slot = tile * kTile + threadIdx.x;
    float4 p0, p1;
    uint32_t key = kNone, id = 0u;
    if (slot - S.body_off < S.n) {
      load_body(part_in, slot, p0, p1);
      id = ids_in[slot];
      uint32_t cx, cy, cz;
      cells_of_position(p0.x, p0.y, p0.z, S.depth, cx, cy, cz);
      key = S.cell_off + (spread3s(cx) | (spread3s(cy) << 1) | (spread3s(cz) << 2));
    }
    __syncthreads();  // the table is clear
    const uint32_t prev = __shfl_up_sync(kAll, key, 1);
    const uint32_t heads = __ballot_sync(kAll, lane == 0u || key != prev);
    const uint32_t head = 31u - (uint32_t)__clz((int)(heads & (kAll >> (31u - lane))));  // of this lane's run
    uint32_t h = 0u, base = 0u;
    if (key != kNone && lane == head) {
      const uint32_t after = lane == 31u ? 0u : heads & (kAll << (lane + 1u));
      h = (key * 2654435761u) >> 23;  // 9-bit multiplicative hash
      for (uint32_t probe = 0; probe < kScatterSlots; probe++) {
        const uint32_t was = atomicCAS(&hkey[h], kNone, key);
        if (was == kNone) used[atomicAdd(&nused, 1u)] = (uint16_t)h;
        if (was == kNone || was == key) break;
        h = (h + 1u) & (kScatterSlots - 1u);
      }
      base = atomicAdd(&hcnt[h], (after != 0u ? (uint32_t)__ffs((int)after) - 1u : 32u) - lane);
    }
    h = __shfl_sync(kAll, h, head);
    const uint32_t off = __shfl_sync(kAll, base, head) + (lane - head);
    __syncthreads();
    // One global reservation per (CTA, leaf); hcnt becomes the CTA's first slot.
    const uint32_t leaves = nused;
    if (threadIdx.x < leaves) {
      const uint32_t u = used[threadIdx.x];
      hcnt[u] = atomicAdd(&starts[hkey[u]], hcnt[u]);
    }
    __syncthreads();
    if (key != kNone) {
      const uint32_t dst = hcnt[h] + off;
      if (dst < tiles * kTile) {  // defensive: counts and positions always agree
        store_body(part_out, dst, p0, p1);
        ids_out[dst] = id;
      }
    }
    if (kList) {  // the table is cleared for the next tile
      __syncthreads();
      if (threadIdx.x < leaves) {
        const uint32_t u = used[threadIdx.x];
        hkey[u] = kNone;
        hcnt[u] = 0u;
      }
      if (threadIdx.x == 0u) nused = 0u;
    }
  }
  stamp_end(stamp);  // last of the resort's four kernels
}

uint32_t leaf_sort_blocks(uint32_t max_depth) {
  return ((1u << (3u * max_depth)) + kLeafBlock - 1u) / kLeafBlock;
}

void leaf_counting_sort(const LaunchCtx &L, uint32_t scenes, uint32_t max_depth, const uint4 *counts,
                        uint32_t *block_scratch, uint32_t *starts, const float4 *part_in,
                        const uint32_t *ids_in, float4 *part_out, uint32_t *ids_out,
                        uint32_t tiles) {
  const uint32_t nb = leaf_sort_blocks(max_depth);
  // With lists (serving slots), a few rows of CTAs walk the active scenes and
  // a persistent grid the active tiles.
  const uint32_t rows = L.scene_list != nullptr ? (scenes < 32u ? scenes : 32u) : scenes;
  launch_step_kernel(L, k_leaf_block_sums, dim3(nb, rows), dim3(kLeafThreads), 0, L.scenes, scenes, L.scene_list,
                     (const Counters *)L.ctr, counts, block_scratch, nb, stamp_rec(L, 4u));
  launch_step_kernel(L, k_leaf_block_scan, dim3(rows), dim3(32), 0, L.scenes, scenes, L.scene_list,
                     (const Counters *)L.ctr, block_scratch, nb);
  launch_step_kernel(L, k_leaf_offsets, dim3(nb, rows), dim3(kLeafThreads), 0, L.scenes, scenes, L.scene_list,
                     (const Counters *)L.ctr, counts, (const uint32_t *)block_scratch, nb, starts);
  const uint32_t wave = 8u * L.sms;
  launch_step_kernel(L, L.tile_list != nullptr ? k_leaf_scatter<true> : k_leaf_scatter<false>,
                     dim3(L.tile_list != nullptr && tiles > wave ? wave : tiles), dim3(256), 0, L.scenes, L.tile_scene,
                     L.tile_list, (const Counters *)L.ctr, part_in, ids_in, part_out, ids_out, starts, tiles,
                     stamp_rec(L, 4u));
}

}  // namespace rfmm
