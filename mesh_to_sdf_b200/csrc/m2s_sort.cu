// Stable LSD radix sort of (u32 key, u32 value) pairs on the device: the LBVH
// build, Morton-ordered query batches, the mesh check and the viewer's cell
// order.
//
// One kernel counts the digits of every pass in a single read of the keys, and
// each 8-bit pass is then one kernel that reads its pairs once and writes them
// once.  A tile learns where its digits go from the tiles before it: it
// publishes its digit counts, then adds up the counts (or, where a tile has
// them already, the running totals) of the tiles before it, newest first.
// Tiles take their numbers from a counter as their blocks start, so the tiles
// a block waits for have started before it.  A wait is bounded all the same:
// past its limit the thread counts its digit in the tiles before it from the
// keys themselves (a pass never overwrites its input), slower but the same sum.
// (The look-back is Merrill and Garland's, "Single-pass Parallel Prefix Scan with
// Decoupled Look-back", 2016; one kernel a digit with it is Adinets and Merrill's
// "Onesweep", 2022.)
//
// Bound: HBM, 16 bytes a pair and pass (8 read, 8 written).  Before, each pass
// read the keys again for per-tile counts, scanned 256 counts a tile in three
// launches and ranked a tile in eight steps of three block barriers: 16.7M
// pairs 176 us a pass in the scatter alone, 20 launches a sort; now 132 us a
// pass (2.0 TB/s: 2,048 tiles, two an SM at a time, are seven waves of about
// 19 us, a tile's chain of loads, ranks and totals) and 5 launches: the sort
// 1.08 -> 0.57 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>

#include "m2s_internal.cuh"

namespace m2s {
namespace {

constexpr int kThreads = 256;  // one per digit value
constexpr int kWarps = kThreads / 32;
constexpr int kDigits = 256;
constexpr int kMaxPasses = 4;

__device__ __forceinline__ uint32_t total_order_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7FFFFFFFu) : ~key);
}

// What a pass reads: pairs, or the floats whose indices are to be ordered by
// f32::total_cmp (the first pass of the cell order: no pairs written for it).
struct PairSource {
  const uint32_t *keys, *vals;
  __device__ uint32_t key(uint64_t i) const { return keys[i]; }
  __device__ uint32_t val(uint64_t i) const { return vals[i]; }
};
struct FloatSource {
  const float* d;
  __device__ uint32_t key(uint64_t i) const { return total_order_key(d[i]); }
  __device__ uint32_t val(uint64_t i) const { return (uint32_t)i; }
};

// Zeroed before a sort.
struct __align__(16) SortState {
  uint32_t hist[kMaxPasses][kDigits];  // digit counts, then each digit's first place
  uint32_t tiles[kMaxPasses];          // next tile number of a pass
  uint32_t done;                       // blocks that have counted
  uint32_t lo_inv, hi;                 // extremes of the floats: ~(least key), greatest key
};

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += warp_sums[w];
  __syncthreads();
  return before + x - v;
}

// Digit counts of every pass; the block that finishes last turns them into
// each digit's first place.  MINMAX (floats): also the extremes of the values
// that are no NaN, out[0] and out[1], starting from f32::MAX and -f32::MAX.
template <class Source, int PASSES, bool MINMAX>
__global__ void __launch_bounds__(kThreads) k_sort_count(Source src, uint64_t n, SortState* st, float* out) {
  __shared__ uint32_t h[PASSES][kDigits];
  __shared__ uint32_t warp_sums[kWarps];
  __shared__ bool last;
  for (int p = 0; p < PASSES; ++p) h[p][threadIdx.x] = 0;
  __syncthreads();
  uint32_t lo_inv = 0, hi = 0;
  const uint64_t stride = (uint64_t)gridDim.x * kThreads;
  constexpr int kUnroll = 4;
  for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += kUnroll * stride) {
    uint32_t key[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) key[u] = i + u * stride < n ? src.key(i + u * stride) : 0u;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      if (i + u * stride >= n) continue;
#pragma unroll
      for (int p = 0; p < PASSES; ++p) atomicAdd(&h[p][(key[u] >> (8 * p)) & 0xFFu], 1u);
      if (MINMAX && !isnan(key_float(key[u]))) {
        lo_inv = max(lo_inv, ~key[u]);
        hi = max(hi, key[u]);
      }
    }
  }
  if (MINMAX) {
    lo_inv = __reduce_max_sync(0xFFFFFFFFu, lo_inv);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if ((threadIdx.x & 31) == 0) {
      if (lo_inv) atomicMax(&st->lo_inv, lo_inv);
      if (hi) atomicMax(&st->hi, hi);
    }
  }
  __syncthreads();
  for (int p = 0; p < PASSES; ++p) {
    const uint32_t c = h[p][threadIdx.x];
    if (c) atomicAdd(&st->hist[p][threadIdx.x], c);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int p = 0; p < PASSES; ++p) {
    const uint32_t c = __ldcg(&st->hist[p][threadIdx.x]);
    st->hist[p][threadIdx.x] = block_exclusive_scan(c, warp_sums);
  }
  if (MINMAX && threadIdx.x == 0) {
    const uint32_t l = __ldcg(&st->lo_inv), g = __ldcg(&st->hi);
    const bool any = l != 0u || g != 0u;  // no key is both 0 and 0xFFFFFFFF
    out[0] = key_float(any ? min(~l, total_order_key(FLT_MAX)) : 0xFFFFFFFFu);
    out[1] = key_float(any ? max(g, total_order_key(-FLT_MAX)) : 0u);
  }
}

// A tile's word for one digit: its count (kCount) or the count up to and with
// it (kTotal) in the low bits; 0 until it is published.  Words carry all that
// is exchanged, so they need no ordering.  32 bits hold counts below 2^30.
template <class Word>
struct TileWord {
  static constexpr int kBits = sizeof(Word) * 8 - 2;
  static constexpr Word kCount = (Word)1 << kBits, kTotal = (Word)2 << kBits, kValue = kCount - 1;
};
__device__ __forceinline__ uint32_t ld_word(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
constexpr uint32_t kPolls = 1u << 16;  // in vain, at most (some 50 ms; a tile takes microseconds)
constexpr uint32_t kAhead = 8;

// The lanes of the warp whose d (9 bits) is this lane's, by a ballot per bit
// (16.7M pairs 0.57 ms against 0.67 with __match_any_sync).
__device__ __forceinline__ uint32_t same_digit(uint32_t d) {
  uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const bool set = (d >> b) & 1u;
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, set);
    peers &= set ? m : ~m;
  }
  return peers;
}

// One pass.  A warp ranks its ITEMS * 32 neighbouring pairs 32 at a time (the
// lanes of one digit find each other by ballots, the digit's count so
// far in the warp's own table), so ranking takes no block barrier and keeps
// the input order; the tile is then ordered in shared memory and written out
// digit run by digit run.
template <int THREADS, int ITEMS, class Source, class Word, bool KEYS_OUT>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_sort_pass(Source src, uint32_t* __restrict__ kout,
                                                                       uint32_t* __restrict__ vout, uint64_t n,
                                                                       int shift, const uint32_t* __restrict__ first,
                                                                       Word* words, uint32_t* next_tile,
                                                                       uint32_t max_polls) {
  using W = TileWord<Word>;
  constexpr int kTile = THREADS * ITEMS, kTileWarps = THREADS / 32;
  extern __shared__ uint32_t s_mem[];
  uint32_t* s_key = s_mem;  // kTile keys, kTile values, then per warp:
  uint32_t* s_val = s_mem + kTile;
  uint32_t(*count)[kDigits] = reinterpret_cast<uint32_t(*)[kDigits]>(s_mem + 2 * kTile);  // digit counts, then places
  __shared__ uint32_t dest[kDigits];  // a digit's first place in the output less that in the tile
  __shared__ uint32_t warp_sums[kWarps], s_tile;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = atomicAdd(next_tile, 1u);
  for (uint32_t i = threadIdx.x; i < kTileWarps * kDigits; i += THREADS) (&count[0][0])[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = (uint64_t)tile * kTile;
  const uint32_t tile_n = (uint32_t)min((uint64_t)kTile, n - base);
  uint32_t key[ITEMS], rank[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t t = warp * (ITEMS * 32) + i * 32 + lane;
    key[i] = t < tile_n ? src.key(base + t) : 0u;
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t t = warp * (ITEMS * 32) + i * 32 + lane;
    const uint32_t d = t < tile_n ? (key[i] >> shift) & 0xFFu : 0x100u;
    const uint32_t peers = same_digit(d);
    const uint32_t before = peers & ((1u << lane) - 1u);
    uint32_t c = 0;
    if (before == 0u && d < 0x100u) {  // the first lane of its digit
      c = count[warp][d];
      count[warp][d] = c + __popc(peers);
    }
    rank[i] = __shfl_sync(0xFFFFFFFFu, c, __ffs(peers) - 1) + __popc(before);
    __syncwarp();
  }
  __syncthreads();
  // From here thread d < 256 has digit d: its count in the tile, its place there.
  const uint32_t d = threadIdx.x;
  const bool has = THREADS == kDigits || d < kDigits;
  uint32_t total = 0;
  Word* row = words + (uint64_t)tile * kDigits + d;
  if (has) {
    for (int w = 0; w < kTileWarps; ++w) total += count[w][d];
    st_word(row, (tile == 0 ? W::kTotal : W::kCount) | (Word)total);
  }
  uint32_t x = total;
  if (warp < kWarps) {
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
      if ((int)lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
  }
  __syncthreads();
  uint32_t in_tile = x - total;
  if (has) {
    for (uint32_t w = 0; w < warp; ++w) in_tile += warp_sums[w];
    uint32_t at = in_tile;
    for (int w = 0; w < kTileWarps; ++w) {
      const uint32_t c = count[w][d];
      count[w][d] = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t t = warp * (ITEMS * 32) + i * 32 + lane;
    if (t < tile_n) {
      const uint32_t pos = count[warp][(key[i] >> shift) & 0xFFu] + rank[i];
      s_key[pos] = key[i];
      s_val[pos] = src.val(base + t);
    }
  }
  if (has) {
    // The digit's count in the tiles before this one, kAhead of them at a time:
    // the tiles of a wave publish their counts together and then look back over
    // each other, so one at a time each would wait through hundreds of loads.
    uint64_t before = 0;
    uint32_t polls = 0;
    for (uint32_t j = tile; j > 0;) {
      if (polls == max_polls) {  // gave up: count tiles 0 .. j - 1
        const uint64_t end = (uint64_t)j * kTile;
        for (uint64_t i = 0; i < end; ++i) before += ((src.key(i) >> shift) & 0xFFu) == d ? 1u : 0u;
        break;
      }
      Word w[kAhead];
#pragma unroll
      for (uint32_t a = 0; a < kAhead; ++a)
        w[a] = a < j ? ld_word(words + (uint64_t)(j - 1u - a) * kDigits + d) : (Word)0;
      bool found = false;
      uint32_t taken = 0;
#pragma unroll
      for (uint32_t a = 0; a < kAhead; ++a) {
        if (found || taken != a || w[a] == 0) continue;  // after a total, or after one not yet there
        before += w[a] & W::kValue;
        found = (w[a] & W::kTotal) != 0;
        ++taken;
      }
      if (found) break;
      j -= taken;
      if (taken == 0) ++polls;
    }
    if (tile != 0) st_word(row, W::kTotal | (Word)(before + total));
    dest[d] = first[d] + (uint32_t)before - in_tile;
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < tile_n; t += THREADS) {
    const uint32_t k = s_key[t];
    const uint32_t to = dest[(k >> shift) & 0xFFu] + t;
    if (KEYS_OUT) kout[to] = k;
    vout[to] = s_val[t];
  }
}

// Tiles: 8,192 pairs once there are 2^20 pairs, 2,048 below, so that a sort
// fills the GPU (512 x 16 / 1,024 x 16 / 256 x 16 threads x pairs: 16.7M pairs
// 0.57 / 0.62 / 0.58 ms, 4M 0.18 / 0.20 / 0.22; 256 x 8 / 256 x 4 / 512 x 4: 1M
// 0.104 / 0.127 / 0.102 ms, 82,000 0.05 all).
constexpr int kLargeThreads = 512, kLargeItems = 16, kSmallThreads = 256, kSmallItems = 8;
constexpr uint64_t kLargeMin = 1ull << 20;
struct SortPlan {
  DevBuf<uint8_t> space;
  SortState* st = nullptr;
  uint8_t* words = nullptr;
  uint64_t tiles = 0;
  bool big = false;   // counts that need 64-bit words
  bool wide = false;  // large tiles
  uint32_t max_polls = kPolls;
  int init(uint64_t n, int passes, cudaStream_t s) {
    big = big || n >= (1ull << 30);
    wide = n >= kLargeMin;
    const uint64_t tile = (big || wide) ? kLargeThreads * kLargeItems : kSmallThreads * kSmallItems;
    tiles = (n + tile - 1) / tile;
    const uint64_t word_bytes = (uint64_t)passes * tiles * kDigits * (big ? 8 : 4);
    int r = space.alloc(sizeof(SortState) + word_bytes, s);
    if (r) return r;
    st = reinterpret_cast<SortState*>(space.p);
    words = space.p + sizeof(SortState);
    M2S_CUDA(cudaMemsetAsync(space.p, 0, sizeof(SortState) + word_bytes, s));
    return M2S_OK;
  }
  template <int THREADS, int ITEMS, class Source, class Word, bool KEYS_OUT>
  int launch(Source src, uint32_t* kout, uint32_t* vout, uint64_t n, int p, cudaStream_t s) {
    auto* kern = k_sort_pass<THREADS, ITEMS, Source, Word, KEYS_OUT>;
    constexpr int smem = (2 * THREADS * ITEMS + THREADS / 32 * kDigits) * 4;
    if (smem > 48 * 1024 - 2048) M2S_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kern<<<(unsigned)tiles, THREADS, smem, s>>>(src, kout, vout, n, 8 * p, st->hist[p],
                                                reinterpret_cast<Word*>(words) + (uint64_t)p * tiles * kDigits,
                                                &st->tiles[p], max_polls);
    M2S_CUDA(cudaGetLastError());
    return M2S_OK;
  }
  template <class Source, bool KEYS_OUT>
  int pass(Source src, uint32_t* kout, uint32_t* vout, uint64_t n, int p, cudaStream_t s) {
    if (big) return launch<kLargeThreads, kLargeItems, Source, unsigned long long, KEYS_OUT>(src, kout, vout, n, p, s);
    if (wide) return launch<kLargeThreads, kLargeItems, Source, uint32_t, KEYS_OUT>(src, kout, vout, n, p, s);
    return launch<kSmallThreads, kSmallItems, Source, uint32_t, KEYS_OUT>(src, kout, vout, n, p, s);
  }
};

unsigned count_blocks(uint64_t n) {
  return (unsigned)std::min<uint64_t>((n + 4 * kThreads - 1) / (4 * kThreads), 148ull * 8ull);
}

}  // namespace

namespace {
int sort_pairs(SortPlan& plan, uint32_t* keys, uint32_t* vals, uint64_t n, int key_bits, cudaStream_t s,
               bool keep_keys) {
  if (n <= 1) return M2S_OK;
  if (key_bits <= 0 || key_bits > 32 || n > 0xFFFFFFFFull) return M2S_ERR_INVALID_ARGUMENT;
  const int passes = (key_bits + 7) / 8;
  DevBuf<uint32_t> k2, v2;
  int r;
  if ((r = plan.init(n, passes, s)) || (r = k2.alloc(n, s)) || (r = v2.alloc(n, s))) return r;
  const PairSource in{keys, vals};
  const unsigned cb = count_blocks(n);
  switch (passes) {
    case 1: k_sort_count<PairSource, 1, false><<<cb, kThreads, 0, s>>>(in, n, plan.st, nullptr); break;
    case 2: k_sort_count<PairSource, 2, false><<<cb, kThreads, 0, s>>>(in, n, plan.st, nullptr); break;
    case 3: k_sort_count<PairSource, 3, false><<<cb, kThreads, 0, s>>>(in, n, plan.st, nullptr); break;
    default: k_sort_count<PairSource, 4, false><<<cb, kThreads, 0, s>>>(in, n, plan.st, nullptr);
  }
  M2S_CUDA(cudaGetLastError());
  uint32_t *ka = keys, *va = vals, *kb = k2.p, *vb = v2.p;
  for (int p = 0; p < passes; ++p) {
    const PairSource src{ka, va};
    if (p + 1 < passes || keep_keys) r = plan.pass<PairSource, true>(src, kb, vb, n, p, s);
    else r = plan.pass<PairSource, false>(src, kb, vb, n, p, s);
    if (r) return r;
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (ka != keys) {
    if (keep_keys) M2S_CUDA(cudaMemcpyAsync(keys, ka, n * 4, cudaMemcpyDeviceToDevice, s));
    M2S_CUDA(cudaMemcpyAsync(vals, va, n * 4, cudaMemcpyDeviceToDevice, s));
  }
  return M2S_OK;
}

}  // namespace

int radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint64_t n, int key_bits, cudaStream_t s, bool keep_keys) {
  SortPlan plan;
  return sort_pairs(plan, keys, vals, n, key_bits, s, keep_keys);
}

int radix_sort_pairs_with(uint32_t* keys, uint32_t* vals, uint64_t n, int key_bits, uint32_t max_polls, bool big,
                          cudaStream_t s) {
  SortPlan plan;
  plan.max_polls = max_polls;
  plan.big = big;
  return sort_pairs(plan, keys, vals, n, key_bits, s, true);
}

int sort_floats(const float* d, uint64_t n, uint32_t* order, float* minmax, cudaStream_t s) {
  if (n == 0) return M2S_OK;
  if (n > 0xFFFFFFFFull) return M2S_ERR_INVALID_ARGUMENT;
  SortPlan plan;
  DevBuf<uint32_t> k1, k2, v2;
  int r;
  if ((r = plan.init(n, 4, s)) || (r = k1.alloc(n, s)) || (r = k2.alloc(n, s)) || (r = v2.alloc(n, s))) return r;
  const FloatSource in{d};
  const unsigned cb = count_blocks(n);
  if (minmax) k_sort_count<FloatSource, 4, true><<<cb, kThreads, 0, s>>>(in, n, plan.st, minmax);
  else k_sort_count<FloatSource, 4, false><<<cb, kThreads, 0, s>>>(in, n, plan.st, nullptr);
  M2S_CUDA(cudaGetLastError());
  if ((r = plan.pass<FloatSource, true>(in, k2.p, v2.p, n, 0, s))) return r;
  if ((r = plan.pass<PairSource, true>(PairSource{k2.p, v2.p}, k1.p, order, n, 1, s))) return r;
  if ((r = plan.pass<PairSource, true>(PairSource{k1.p, order}, k2.p, v2.p, n, 2, s))) return r;
  return plan.pass<PairSource, false>(PairSource{k2.p, v2.p}, nullptr, order, n, 3, s);
}

}  // namespace m2s
