// Stable LSD radix sort of (uint32 key, uint32 value) pairs, and the Morton
// codes the photon-beam pipeline sorts.
//
// Reference design: PPB_RadixSort_LocalSort.comp (block-local 4-bit sort by
// four 1-bit split passes with a Blelloch scan + 16-bin histogram),
// PPB_RadixSort_PrefixSum.comp and PPB_RadixSort_GlobalSort.comp (scan of
// the histograms, scatter), driven from RenderTechniquePPB.cpp:465-491; keys
// from expandBits/getMortonCode (PPB_PT.comp:317-333).
//
// GB300 design: the same stable order (a stable LSD sort's result does not
// depend on its digit width) from 8-bit digits, so 32-bit keys take 4
// passes instead of the reference's 8.  Up to 8,192 pairs are sorted by one
// CTA in one launch.  Beyond that one histogram kernel computes the digit
// counts of every pass at once; each digit pass is then ONE kernel over
// tiles of 4,096 to 8,192 keys: stable in-tile ranking from eight warp
// ballots of the digit bits, a decoupled look-back across tiles (one thread
// a digit; tile ids taken in launch order from an atomic counter, so every
// tile waits only on tiles already running), shared-memory staging and a
// coalesced scatter.  Each pass reads and writes every pair once (16 B/key
// per pass).  Spins are bounded: a wait that runs out sets the context's
// error word instead of hanging.
#include "vcr_internal.h"
#include "sort.cuh"

namespace vcr {

constexpr uint32_t kFlagA = 1u << 30;                 // tile aggregate published
constexpr uint32_t kFlagP = 2u << 30;                 // inclusive prefix published
constexpr uint32_t kCountMask = (1u << 30) - 1u;

struct SortScratch {
  uint32_t* hist;     // [4][256] digit counts per pass
  uint32_t* tiles;    // [4] tile counters
  uint32_t* desc;     // [4][ntiles][256] look-back words
  uint32_t* keys_tmp; // n
  uint32_t* vals_tmp; // n
};

static SortScratch carve(void* base, uint32_t n) {
  uint32_t* p = reinterpret_cast<uint32_t*>(base);
  SortScratch s;
  s.hist = p;
  s.tiles = p + kSortMaxPasses * kSortRadix;
  s.desc = p + kSortMaxPasses * kSortRadix + kSortMaxPasses;
  uint8_t* b = reinterpret_cast<uint8_t*>(base) + sort_round256(sort_scratch_header_bytes(n));
  s.keys_tmp = reinterpret_cast<uint32_t*>(b);
  s.vals_tmp = reinterpret_cast<uint32_t*>(b + sort_round256((size_t)n * 4));
  return s;
}

// Mask of pass p's digit: 8 bits, or the bits left below end_bit in the
// last pass (so bits at or above end_bit never decide the order).
__host__ __device__ __forceinline__ uint32_t digit_mask(uint32_t begin_bit, uint32_t end_bit, uint32_t p) {
  const uint32_t w = end_bit - (begin_bit + kSortDigitBits * p);
  return w >= kSortDigitBits ? (uint32_t)kSortRadix - 1u : (1u << w) - 1u;
}

// Digit counts of all passes in one read of the keys.  A CTA's counters are
// one word a digit value and lane, lane l's on bank l, so a warp's 32 atomic
// adds never meet on a bank, whatever the keys are (in one array of 256
// counters three to four of 32 random digits share a bank, and equal keys
// one word): 128 KB for the four passes, one CTA of 1,024 threads an SM.
// 2^26 random keys: 59 us = 4.5 TB/s (235 us with one array).
constexpr int kHistThreads = 1024;
constexpr int kHistItems = 16;                               // keys a thread reads at once
constexpr uint32_t kHistKeys = kHistThreads * kHistItems;    // keys of a chunk
constexpr uint32_t kHistPass = kSortRadix * 32;              // counters of a pass

__global__ void __launch_bounds__(kHistThreads) sort_hist_kernel(const uint32_t* __restrict__ keys, uint32_t n,
                                                                 uint32_t begin_bit, uint32_t end_bit, uint32_t passes,
                                                                 uint32_t* __restrict__ hist) {
  extern __shared__ __align__(16) uint32_t s_dyn[];
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t i = threadIdx.x; i < passes * kHistPass; i += kHistThreads) s_dyn[i] = 0u;
  __syncthreads();
  uint32_t* mine = s_dyn + lane;
  const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0u;  // a chunk is a multiple of 16 bytes
  const auto count = [&](uint32_t key) {
#pragma unroll
    for (uint32_t p = 0; p < (uint32_t)kSortMaxPasses; ++p)
      if (p < passes) {
        const uint32_t d = (key >> (begin_bit + kSortDigitBits * p)) & digit_mask(begin_bit, end_bit, p);
        atomicAdd(mine + p * kHistPass + d * 32u, 1u);
      }
  };
  for (uint64_t c = blockIdx.x; c * kHistKeys < n; c += gridDim.x) {
    const uint32_t base = (uint32_t)(c * kHistKeys);
    if (vec && n - base >= kHistKeys) {  // 16 bytes a load; which lane counts a key does not matter
      const uint4* v = reinterpret_cast<const uint4*>(keys + base) + threadIdx.x;
      uint4 q[kHistItems / 4];
#pragma unroll
      for (int j = 0; j < kHistItems / 4; ++j) q[j] = __ldg(v + kHistThreads * j);
#pragma unroll
      for (int j = 0; j < kHistItems / 4; ++j) {
        count(q[j].x);
        count(q[j].y);
        count(q[j].z);
        count(q[j].w);
      }
    } else {
      for (uint32_t i = base + threadIdx.x; i < n && i - base < kHistKeys; i += kHistThreads) count(__ldg(keys + i));
    }
  }
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < passes * kSortRadix; r += kHistThreads) {  // a digit value's 32 counters
    uint32_t sum = 0;
#pragma unroll 8
    for (uint32_t i = 0; i < 32u; ++i) sum += s_dyn[r * 32u + ((lane + i) & 31u)];
    if (sum) atomicAdd(hist + r, sum);
  }
}

// The lanes of a warp that hold the same digit as this one (of those with
// ok), from eight ballots of the digit's bits.
template <bool kFull>
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool ok) {
  uint32_t peers = kFull ? 0xffffffffu : __ballot_sync(0xffffffffu, ok);
#pragma unroll
  for (int i = 0; i < kSortDigitBits; ++i) {
    const bool bit = (d >> i) & 1u;
    const uint32_t b = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? b : ~b;
  }
  return peers;
}

// Stable ranks of a warp's keys among its keys with the same digit: item j
// of lane l is the warp's key 32 j + l, the first `count` are keys.  The
// lowest lane of each group of equal digits advances the warp's running
// count in wc[256] (zero on entry, the warp's digit counts afterwards).
// Four items' ballots are taken before their counts, which follow one
// another, so the ballots of one item overlap the counting of the others.
// (Ranks are below 2^16: two a register.)
template <int kItems, bool kFull>
__device__ __forceinline__ void warp_rank(const uint32_t (&key)[kItems], uint32_t (&rank)[(kItems + 1) / 2], uint32_t count,
                                          uint32_t shift, uint32_t dmask, uint32_t* wc) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  constexpr int kGroup = kItems < 4 ? kItems : 4;
#pragma unroll
  for (int g = 0; g < kItems; g += kGroup) {
    uint32_t peers[kGroup];
#pragma unroll
    for (int j = 0; j < kGroup; ++j)
      peers[j] = digit_peers<kFull>((key[g + j] >> shift) & dmask, kFull || 32u * (g + j) + lane < count);
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      const uint32_t d = (key[g + j] >> shift) & dmask;
      const bool ok = kFull || 32u * (g + j) + lane < count;
      const uint32_t leader = ok ? __ffs(peers[j]) - 1u : lane;
      uint32_t base = 0;
      if (ok && lane == leader) {
        base = wc[d];
        wc[d] = base + __popc(peers[j]);
      }
      base = __shfl_sync(0xffffffffu, base, leader);
      const uint32_t r = base + __popc(peers[j] & lt);
      if ((g + j) & 1) rank[(g + j) / 2] |= r << 16;
      else rank[(g + j) / 2] = r;
      __syncwarp();
    }
  }
}

// Exclusive scans of two values a thread over the first 256 threads of a CTA
// (all threads call it); `sums` holds 16 words of shared memory.
__device__ __forceinline__ uint2 scan256(uint32_t x, uint32_t y, uint32_t* sums) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t ix = x, iy = y;
  if (warp < 8u) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t vx = __shfl_up_sync(0xffffffffu, ix, o), vy = __shfl_up_sync(0xffffffffu, iy, o);
      if (lane >= (uint32_t)o) {
        ix += vx;
        iy += vy;
      }
    }
    if (lane == 31u) {
      sums[warp] = ix;
      sums[8 + warp] = iy;
    }
  }
  __syncthreads();
  uint2 r = make_uint2(ix - x, iy - y);
#pragma unroll
  for (uint32_t w = 0; w < 7u; ++w)
    if (w < warp && warp < 8u) {
      r.x += sums[w];
      r.y += sums[8 + w];
    }
  return r;
}

// A load that stays where it is written: moved up before the ranking, as the
// compiler likes to, the values' registers push others to the stack.
__device__ __forceinline__ uint32_t load_here(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// One digit pass over tiles of kT x kI keys (tile ids in launch order from an
// atomic counter).  Warp w ranks the tile's keys [32 kI w, 32 kI (w + 1));
// then one thread a digit: the exclusive prefix over the warps, the tile's
// digit starts and the digit's global base (block scans of the tile's and
// the whole sort's counts) and the decoupled look-back, kAhead predecessors
// a poll.  A tile publishes its counts, makes its first poll and puts its
// keys and values in digit order in shared memory before it waits for the
// answer.
//
// 2^26 pairs: 443 us a pass = 2.4 TB/s (552 us with 4,096-key tiles of 256
// threads, values and look-back after one another).  Bound by the shared
// memory pipe (half of its wavefronts: three to four of 32 random digits
// share a bank in each of the counting, staging and base reads) and the
// ballots' issue (42 %); leaving the look-back out gave 15 %, storing in
// input order instead of scattered nothing.
//
// kFull: every key of the tile exists.
template <int kT, int kI, int kAhead, bool kFull>
__device__ __forceinline__ void sort_tile(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                          uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n,
                                          uint32_t shift, uint32_t dmask, uint32_t pass, const SortScratch& sc,
                                          uint32_t spin_limit, int* __restrict__ err, uint32_t tile, uint32_t* s_dyn,
                                          uint32_t* s_off, uint32_t* s_sums) {
  constexpr uint32_t kTile = kT * kI, kWarps = kT / 32;
  uint32_t* s_keys = s_dyn;                // [kTile] the tile's keys in digit order
  uint32_t* s_vals = s_keys + kTile;       // [kTile] their values
  uint32_t* s_wcnt = s_vals + kTile;       // [kWarps][256]

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t tile0 = tile * kTile;
  const uint32_t count = min(kTile, n - tile0);
  const uint32_t first = warp * (32 * kI);  // the warp's first key of the tile
  const uint32_t mine = count > first ? min(count - first, 32u * kI) : 0u;
  uint32_t key[kI], rank[(kI + 1) / 2];
  const uint32_t* kp = kin + tile0 + first + lane;
#pragma unroll
  for (int j = 0; j < kI; ++j) key[j] = (kFull || 32u * j + lane < mine) ? kp[32 * j] : 0u;
  uint32_t val[kI];
  uint32_t* wc = s_wcnt + warp * kSortRadix;
  warp_rank<kI, kFull>(key, rank, mine, shift, dmask, wc);
#pragma unroll
  for (int j = 0; j < kI; ++j) {
    const uint32_t local = first + 32u * j + lane;
    val[j] = tile0 + local;
    if (vin && (kFull || 32u * j + lane < mine)) val[j] = load_here(vin + tile0 + local);
  }
  __syncthreads();
  const uint32_t d = threadIdx.x;  // one thread a digit
  const bool digit = d < (uint32_t)kSortRadix;
  uint32_t total = 0;
  volatile uint32_t* desc = sc.desc + (size_t)pass * ((size_t)gridDim.x * kSortRadix);
  uint32_t ahead[kAhead];  // the words of tiles t, t - 1, ...
  int t = (int)tile - 1;
  const auto look = [&]() {
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      ahead[i] = t - i >= 0 ? desc[(size_t)(t - i) * kSortRadix + d] : kFlagP + 0u;
  };
  if (digit) {
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) {
      const uint32_t c = s_wcnt[w * kSortRadix + d];
      s_wcnt[w * kSortRadix + d] = total;  // exclusive prefix over warps
      total += c;
    }
    desc[(size_t)tile * kSortRadix + d] = (tile == 0 ? kFlagP : kFlagA) | total;
  }
  const uint2 starts = scan256(digit ? total : 0u, digit ? sc.hist[pass * kSortRadix + d] : 0u, s_sums);
  if (digit) {
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) s_wcnt[w * kSortRadix + d] += starts.x;
    look();  // under way while the tile is put in order
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kI; ++j)
    if (kFull || 32u * j + lane < mine) {
      const uint32_t pos = wc[(key[j] >> shift) & dmask] + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
      s_keys[pos] = key[j];
      s_vals[pos] = val[j];
    }
  if (digit) {
    uint32_t excl = 0, spins = 0;
    bool found = t < 0;
    while (!found) {
      int used = 0;
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const uint32_t flag = ahead[i] & ~kCountMask;
        if (flag == 0u) break;
        excl += ahead[i] & kCountMask;
        ++used;
        if (flag == kFlagP) {
          found = true;
          break;
        }
      }
      if (found) break;
      t -= used;
      if (used < kAhead && ++spins > spin_limit) {
        atomicExch(err, 2);  // look-back wait ran out
        break;
      }
      look();
    }
    if (tile != 0) desc[(size_t)tile * kSortRadix + d] = kFlagP | (excl + total);
    s_off[d] = starts.y + excl - starts.x;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kI; ++j) {
    const uint32_t i = j * kT + threadIdx.x;
    if (kFull || i < count) {
      const uint32_t k = s_keys[i], o = s_off[(k >> shift) & dmask] + i;
      if (o < n) {  // always true unless a look-back wait ran out (error word set)
        kout[o] = k;
        vout[o] = s_vals[i];
      }
    }
  }
}

constexpr int kSortThreads = 512;
constexpr int kSortAhead = 4;

template <int kI>
__global__ void __launch_bounds__(kSortThreads, 2) sort_pass_kernel(const uint32_t* __restrict__ kin,
                                                             const uint32_t* __restrict__ vin,
                                                             uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                             uint32_t n, uint32_t shift, uint32_t dmask, uint32_t pass,
                                                             SortScratch sc, uint32_t spin_limit,
                                                             int* __restrict__ err) {
  constexpr int kT = kSortThreads;
  static_assert(kT >= kSortRadix, "one thread a digit in the tile-level steps");
  extern __shared__ __align__(16) uint32_t s_dyn[];
  __shared__ uint32_t s_tile, s_off[kSortRadix], s_sums[16];
  if (threadIdx.x == 0) s_tile = atomicAdd(sc.tiles + pass, 1u);
  uint32_t* s_wcnt = s_dyn + 2 * kT * kI;
  for (uint32_t i = threadIdx.x; i < kT / 32u * kSortRadix; i += kT) s_wcnt[i] = 0u;
  __syncthreads();
  const uint32_t tile = s_tile;
  if (n - tile * (uint32_t)(kT * kI) >= (uint32_t)(kT * kI))
    sort_tile<kT, kI, kSortAhead, true>(kin, vin, kout, vout, n, shift, dmask, pass, sc, spin_limit, err, tile, s_dyn,
                                    s_off, s_sums);
  else
    sort_tile<kT, kI, kSortAhead, false>(kin, vin, kout, vout, n, shift, dmask, pass, sc, spin_limit, err, tile, s_dyn,
                                     s_off, s_sums);
}

template <int kI>
static cudaError_t sort_pass(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, uint32_t n,
                             uint32_t shift, uint32_t dmask, uint32_t pass, const SortScratch& sc, uint32_t spins,
                             int* d_err, cudaStream_t st) {
  constexpr int kT = kSortThreads;
  constexpr size_t smem = (size_t)(2 * kT * kI + kT / 32 * kSortRadix) * sizeof(uint32_t);
  const auto kern = sort_pass_kernel<kI>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<(n + kT * kI - 1) / (kT * kI), kT, smem, st>>>(kin, vin, kout, vout, n, shift, dmask, pass, sc, spins, d_err);
  return cudaGetLastError();
}

// A sort of few keys in one launch of one CTA: keys and values stay in shared
// memory over all digit passes (seven launches, most of them one small tile,
// otherwise).  3,001 pairs: 53 -> 16.5 us a call, 8,192: 59 -> 31 us.
constexpr int kSmallThreads = 1024;
constexpr int kSmallItems = 8;
constexpr uint32_t kSmallKeys = kSmallThreads * kSmallItems;

template <int kI>
__global__ void __launch_bounds__(kSmallThreads) sort_small_kernel(const uint32_t* kin, const uint32_t* vin,
                                                                   uint32_t* kout, uint32_t* vout, uint32_t n,
                                                                   uint32_t begin_bit, uint32_t end_bit) {
  constexpr uint32_t kWarps = kSmallThreads / 32;
  extern __shared__ __align__(16) uint32_t s_dyn[];
  uint32_t* s_keys = s_dyn;
  uint32_t* s_vals = s_keys + kSmallThreads * kI;
  uint32_t* s_wcnt = s_vals + kSmallThreads * kI;  // [kWarps][256]
  __shared__ uint32_t s_start[kSortRadix], s_part[4][kSortRadix], s_sums[16];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t first = warp * (32 * kI), mine = n > first ? min(n - first, 32u * kI) : 0u;
  uint32_t key[kI], val[kI], rank[(kI + 1) / 2];
#pragma unroll
  for (int j = 0; j < kI; ++j) {
    const uint32_t i = first + 32u * j + lane;
    key[j] = i < n ? kin[i] : 0u;
    val[j] = !vin ? i : i < n ? vin[i] : 0u;
  }
  const uint32_t passes = (end_bit - begin_bit + kSortDigitBits - 1) / kSortDigitBits;
  uint32_t* wc = s_wcnt + warp * kSortRadix;
  for (uint32_t p = 0; p < passes; ++p) {
    const uint32_t shift = begin_bit + kSortDigitBits * p, dmask = digit_mask(begin_bit, end_bit, p);
    for (uint32_t i = lane; i < (uint32_t)kSortRadix; i += 32u) wc[i] = 0u;
    __syncwarp();
    warp_rank<kI, false>(key, rank, mine, shift, dmask, wc);
    __syncthreads();
    // four threads a digit: the exclusive prefix over their quarter of the warps
    const uint32_t d = threadIdx.x & (kSortRadix - 1u), quarter = threadIdx.x / kSortRadix;
    uint32_t total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps / 4; ++w) {
      uint32_t* c = s_wcnt + (quarter * (kWarps / 4) + w) * kSortRadix + d;
      const uint32_t x = *c;
      *c = total;
      total += x;
    }
    s_part[quarter][d] = total;
    __syncthreads();
    uint32_t all = 0;
    if (threadIdx.x < (uint32_t)kSortRadix)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t x = s_part[q][d];
        s_part[q][d] = all;
        all += x;
      }
    const uint32_t start = scan256(all, 0u, s_sums).x;
    if (threadIdx.x < (uint32_t)kSortRadix) s_start[d] = start;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kI; ++j)
      if (32u * j + lane < mine) {
        const uint32_t e = (key[j] >> shift) & dmask;
        const uint32_t pos = s_start[e] + s_part[warp / (kWarps / 4)][e] + wc[e] + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
        s_keys[pos] = key[j];
        s_vals[pos] = val[j];
      }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kI; ++j) {
      const uint32_t i = first + 32u * j + lane;
      if (i < n) {
        key[j] = s_keys[i];
        val[j] = s_vals[i];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kI; ++j) {
    const uint32_t i = first + 32u * j + lane;
    if (i < n) {
      kout[i] = key[j];
      vout[i] = val[j];
    }
  }
}

template <int kI>
static cudaError_t sort_small(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, uint32_t n,
                              uint32_t begin_bit, uint32_t end_bit, cudaStream_t st) {
  constexpr size_t smem = (size_t)(2 * kSmallThreads * kI + kSmallThreads / 32 * kSortRadix) * sizeof(uint32_t);
  const auto kern = sort_small_kernel<kI>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<1, kSmallThreads, smem, st>>>(kin, vin, kout, vout, n, begin_bit, end_bit);
  return cudaGetLastError();
}

// Runs the passes for bits [begin_bit, end_bit) in 8-bit digits (the last
// digit narrower when the range is not a multiple of 8 bits).  The pass
// chain ping-pongs between `out` and the scratch copy so the last pass
// lands in `out`; in-place calls (in == out) with an odd pass count start
// from a copy.
cudaError_t sort_pairs_enqueue(int sm_count, int* d_err, void* scratch, const uint32_t* kin, const uint32_t* vin,
                               uint32_t* kout, uint32_t* vout, uint32_t n, uint32_t begin_bit, uint32_t end_bit,
                               cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (n <= kSmallKeys) {
    if (n <= 1u * kSmallThreads) return sort_small<1>(kin, vin, kout, vout, n, begin_bit, end_bit, st);
    if (n <= 2u * kSmallThreads) return sort_small<2>(kin, vin, kout, vout, n, begin_bit, end_bit, st);
    if (n <= 4u * kSmallThreads) return sort_small<4>(kin, vin, kout, vout, n, begin_bit, end_bit, st);
    return sort_small<kSmallItems>(kin, vin, kout, vout, n, begin_bit, end_bit, st);
  }
  uint32_t passes = (end_bit - begin_bit + kSortDigitBits - 1) / kSortDigitBits;
  const uint32_t spins = wait_limits().sort_lookback;
  SortScratch sc = carve(scratch, n);
  const uint32_t sms = (uint32_t)std::max(sm_count, 1);
  // Keys a thread: the larger the tile, the fewer look-backs; the smaller,
  // the sooner all SMs have two.  Whole sorts of 30- and 32-bit keys at 8 /
  // 12 / 16 a thread: 100,000 pairs 47 / 57 / 60 us, 1 M 75 / 76 / 75, 3.2 M
  // 147 / 142 / 152, 10.3 M 377 / 352 / 339, 2^26 2.19 / 1.96 / 1.83 ms.
  const uint32_t items = n <= (1u << 20) ? 8u : n <= (1u << 23) ? 12u : 16u;
  const uint32_t ntiles = (n + kSortThreads * items - 1u) / (kSortThreads * items);
  cudaError_t e = cudaMemsetAsync(
      scratch, 0, ((size_t)kSortMaxPasses * (kSortRadix + 1) + (size_t)passes * ntiles * kSortRadix) * 4, st);
  if (e != cudaSuccess) return e;
  const uint32_t hist_smem = passes * kHistPass * (uint32_t)sizeof(uint32_t);
  if ((e = cudaFuncSetAttribute(sort_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSortMaxPasses * kHistPass * sizeof(uint32_t))) != cudaSuccess)
    return e;
  const uint32_t chunks = (n + kHistKeys - 1u) / kHistKeys;
  sort_hist_kernel<<<std::min(chunks, sms), kHistThreads, hist_smem, st>>>(kin, n, begin_bit, end_bit, passes, sc.hist);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const uint32_t* ck = kin;
  const uint32_t* cv = vin;
  // Destinations alternate; the first one is `out` when that makes the last
  // pass land in `out` (odd count) unless the input aliases `out`, in which
  // case the chain starts in scratch and ends with one copy.
  bool alias = (kin == kout) || (vin && vin == vout);
  bool first_to_out = (passes % 2u == 1u) && !alias;
  for (uint32_t p = 0; p < passes; ++p) {
    bool to_out = ((p % 2u) == 0u) == first_to_out;
    uint32_t* nk = to_out ? kout : sc.keys_tmp;
    uint32_t* nv = to_out ? vout : sc.vals_tmp;
    const uint32_t shift = begin_bit + kSortDigitBits * p, dmask = digit_mask(begin_bit, end_bit, p);
    if (items == 8) e = sort_pass<8>(ck, cv, nk, nv, n, shift, dmask, p, sc, spins, d_err, st);
    else if (items == 12) e = sort_pass<12>(ck, cv, nk, nv, n, shift, dmask, p, sc, spins, d_err, st);
    else e = sort_pass<16>(ck, cv, nk, nv, n, shift, dmask, p, sc, spins, d_err, st);
    if (e != cudaSuccess) return e;
    ck = nk;
    cv = nv;
  }
  if (ck != kout) {
    if ((e = cudaMemcpyAsync(kout, ck, (size_t)n * 4, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(vout, cv, (size_t)n * 4, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Morton codes
// ---------------------------------------------------------------------------
// Spread the low 10 bits of v so two zeros separate each (Karras 2012; the
// reference's 8-bit expandBits is PPB_PT.comp:319-325).
__device__ __forceinline__ uint32_t expand10(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

__device__ __forceinline__ uint32_t quant(float p, float b0, float ext, float cells) {
  float q = ((p - b0) / ext) * cells;
  q = fminf(fmaxf(q, 0.0f), cells - 1.0f);
  return (uint32_t)q;
}

// bits == 30: 10 bits per axis over the box [b0, b1] (x << 2 | y << 1 | z);
// bits == 24: the reference's getMortonCode (PPB_PT.comp:327-333), relative
// position / 256 clamped to [0, 255] per axis.
__global__ void morton_kernel(const float* __restrict__ pts, uint32_t n, f3 b0, f3 b1, int bits,
                              uint32_t* __restrict__ codes) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  f3 p = mk(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
  if (bits == 24) {
    f3 r = p - b0;
    uint32_t x = (uint32_t)fminf(fmaxf(r.x / 256.0f, 0.0f), 255.0f);
    uint32_t y = (uint32_t)fminf(fmaxf(r.y / 256.0f, 0.0f), 255.0f);
    uint32_t z = (uint32_t)fminf(fmaxf(r.z / 256.0f, 0.0f), 255.0f);
    codes[i] = (expand10(x) << 2) + (expand10(y) << 1) + expand10(z);
    return;
  }
  f3 e = b1 - b0;
  uint32_t x = quant(p.x, b0.x, e.x, 1024.0f), y = quant(p.y, b0.y, e.y, 1024.0f), z = quant(p.z, b0.z, e.z, 1024.0f);
  codes[i] = (expand10(x) << 2) | (expand10(y) << 1) | expand10(z);
}

vcr_status morton_launch(vcr_ctx* ctx, const float* d_pts, uint32_t n, const float b0[3], const float b1[3],
                         int bits, uint32_t* d_codes, cudaStream_t st) {
  if (n == 0) return VCR_OK;
  morton_kernel<<<(n + 255) / 256, 256, 0, st>>>(d_pts, n, mk(b0[0], b0[1], b0[2]), mk(b1[0], b1[1], b1[2]), bits,
                                                 d_codes);
  VCR_CUDA(ctx, cudaGetLastError());
  return VCR_OK;
}

}  // namespace vcr

using namespace vcr;

extern "C" VCR_API vcr_status vcr_radix_sort_pairs(vcr_ctx* ctx, const uint32_t* d_keys_in, const uint32_t* d_vals_in,
                                                   uint32_t* d_keys_out, uint32_t* d_vals_out, uint32_t n,
                                                   uint32_t begin_bit, uint32_t end_bit, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  if (n && (!d_keys_in || !d_keys_out || !d_vals_out)) return fail(ctx, VCR_ERR_INVALID, "null sort buffer");
  if (begin_bit >= end_bit || end_bit > 32) return fail(ctx, VCR_ERR_INVALID, "bit range [%u, %u)", begin_bit, end_bit);
  if (n > (1u << 30) - 1u) return fail(ctx, VCR_ERR_UNSUPPORTED, "sort of %u keys (max 2^30 - 1)", n);
  if (d_vals_in == d_vals_out && d_keys_in != d_keys_out)
    return fail(ctx, VCR_ERR_INVALID, "values may alias only together with keys");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  vcr_status st = ensure_scratch(ctx, sort_scratch_bytes(n));
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  VCR_CUDA(ctx, sort_pairs_enqueue(ctx->sm_count, ctx->d_error, ctx->d_scratch, d_keys_in, d_vals_in, d_keys_out,
                                   d_vals_out, n, begin_bit, end_bit, s));
  VCR_CUDA(ctx, cudaEventRecord(ctx->work_done, s));
  return VCR_OK;
}

extern "C" VCR_API vcr_status vcr_morton_codes(vcr_ctx* ctx, const float* d_points, uint32_t n,
                                               const float bounds_min[3], const float bounds_max[3],
                                               uint32_t bits, uint32_t* d_codes, void* stream) {
  if (!ctx) return fail(nullptr, VCR_ERR_INVALID, "null context");
  VCR_CUDA(ctx, cudaSetDevice(ctx->device));
  if (n && (!d_points || !d_codes || !bounds_min || !bounds_max)) return fail(ctx, VCR_ERR_INVALID, "null argument");
  if (bits != 30 && bits != 24) return fail(ctx, VCR_ERR_INVALID, "Morton bits must be 30 or 24");
  return morton_launch(ctx, d_points, n, bounds_min, bounds_max, (int)bits, d_codes, (cudaStream_t)stream);
}
