// Kernel-map generation: for every query row and kernel offset, probe the
// coordinate table; results land in an offset-major neighbour table
// nbr[K][n_query] (what the convolution kernels consume) and, on request, in
// CSR-over-offsets pair lists (the reference's per-offset in/out vectors,
// engine/grid/maps.hpp:19-79).
//
// Pass 1 (k_kmap_probe): one thread per query row keeps the row in registers
// (one vectorised 16-byte load for W = 4), loops over the K offsets held in
// shared memory, probes, writes nbr[k][q] (coalesced: consecutive lanes are
// consecutive rows) and counts hits per offset with warp ballots.
// On small maps the offsets are split over gridDim.y, so that more blocks share the chain of probes.
// Pass 2 (k_kmap_scan): exclusive scan of the per-(offset, block) hit counts; the last block turns
// the per-offset totals into offset_ptr[K+1].
// Pass 3 (k_kmap_pairs, optional): ballot compaction of nbr into (a, q) pair
// lists at deterministic positions (pairs of one offset sorted by query row),
// with no sort and no atomics. The reference instead sorts all triplets by
// offset (engine/grid/lattice_gpu.cuh:440-488).
#include "rmn_common.cuh"

#include <string.h>

#include <mutex>

namespace rmn {

constexpr int kKmapBlock = 256;

// The scan of pass 2 by the last block of the probing kernel, on maps of up to kTailCounts counts: a launch of its own takes
// longer there (900 rows x 27 offsets: 6.4 us of a pass of 53). Warp w takes the counted offsets w, w + 8, ...
constexpr uint32_t kTailCounts = 4096;
struct TailScan {
  uint32_t* ticket;  // NULL: k_kmap_scan does it
  uint32_t* totals;
  int64_t* offset_ptr;
  volatile int64_t* host_ptr;
};
__device__ __forceinline__ void scan_counts_in_last_block(const TailScan& tail, uint32_t* block_counts, uint32_t n_blocks, int K,
                                                          int mirror_half) {
  __shared__ uint32_t s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(tail.ticket, 1u) == gridDim.x * gridDim.y - 1 ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto scan = [&](auto v) {  // inclusive, over the warp
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const auto t = __shfl_up_sync(0xFFFFFFFFu, v, d);
      if (lane >= d) v += t;
    }
    return v;
  };
  for (int k = warp; k < K - mirror_half; k += kKmapBlock / 32) {
    uint32_t* counts = block_counts + (size_t)k * n_blocks;
    uint32_t carry = 0;
    for (uint32_t base = 0; base < n_blocks; base += 128) {
      uint32_t v[4], sum = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t i = base + lane * 4 + j;
        v[j] = i < n_blocks ? __ldcg(counts + i) : 0u;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t x = v[j];
        v[j] = sum;
        sum += x;
      }
      const uint32_t incl = scan(sum), before = carry + incl - sum;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t i = base + lane * 4 + j;
        if (i < n_blocks) counts[i] = before + v[j];
      }
      carry += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    if (lane == 0) {
      tail.totals[k] = carry;
      if (k < mirror_half) tail.totals[K - 1 - k] = carry;
    }
  }
  __syncthreads();
  uint32_t* flags = tail.totals + K;  // [0] "pair lists did not fit", [1] half
  if (threadIdx.x == 0) {
    flags[0] = 0;
    flags[1] = (uint32_t)mirror_half;
  }
  if (warp) return;
  int64_t carry = 0;
  for (int base = 0; base < K; base += 32) {
    const int k = base + lane;
    const int64_t t = k < K ? (int64_t)__ldcg(tail.totals + k) : 0, incl = scan(t);
    if (k < K) {
      tail.offset_ptr[k] = carry + incl - t;
      if (tail.host_ptr) tail.host_ptr[k] = carry + incl - t;
    }
    carry += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  if (lane == 0) {
    tail.offset_ptr[K] = carry;
    if (tail.host_ptr) tail.host_ptr[K] = carry;
  }
}

// The packed key is linear in the coordinates: key(c + off) = key(c) + sum_i (off_i << shift_i)
// in 64-bit modular arithmetic, so each probe costs one 64-bit add on top of the range test
// (a neighbour outside the table's bounding box is a miss without touching memory).
template <int W>
__global__ void __launch_bounds__(kKmapBlock) k_kmap_probe(
    const TableHeader* __restrict__ h, const Slot* __restrict__ slots,
    const int32_t* __restrict__ query, uint32_t n_query, const int32_t* __restrict__ offsets,
    int K, int32_t* __restrict__ nbr, uint32_t* __restrict__ block_counts, uint32_t n_blocks,
    uint32_t* __restrict__ scan_ticket, TailScan tail) {
  after_previous_kernel();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int D = W - 1;
  const int k_begin = (int)((uint32_t)K * blockIdx.y / gridDim.y), k_end = (int)((uint32_t)K * (blockIdx.y + 1) / gridDim.y);
  if (!tail.ticket && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *scan_ticket = 0;
  long long* s_delta = reinterpret_cast<long long*>(smem_raw);           // [K]
  int32_t* s_off = reinterpret_cast<int32_t*>(s_delta + K);              // [K][D]
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(s_off + K * D);          // [K]
  for (int i = k_begin * D + threadIdx.x; i < k_end * D; i += kKmapBlock) s_off[i] = offsets[i];
  for (int k = k_begin + threadIdx.x; k < k_end; k += kKmapBlock) {
    long long d = 0;
#pragma unroll
    for (int a = 0; a < D; ++a) d += (long long)offsets[k * D + a] << h->shift[a + 1];
    s_delta[k] = d;
    s_cnt[k] = 0;
  }
  __syncthreads();

  const uint32_t capacity = h->capacity, pos_shift = h->pos_shift;
  const uint32_t q = blockIdx.x * kKmapBlock + threadIdx.x;
  const bool active = q < n_query;
  int32_t c[W];
  if (active) {
    load_row<W>(query, q, c);
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) c[i] = 0;
  }
  // distance from the box minimum per column, the packed centre key, and the box spans
  uint32_t dist[W], span[W];
  long long ckey = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const int32_t mn = h->mn[i];
    dist[i] = (uint32_t)c[i] - (uint32_t)mn;
    span[i] = (uint32_t)(h->mx[i] - mn);
    ckey += (long long)((long long)c[i] - (long long)mn) << h->shift[i];
  }
  const bool batch_ok = active && dist[0] <= span[0];
  const int lane = threadIdx.x & 31;
  // Offsets are handled kUnroll at a time: the first-probe loads of a batch are issued before any
  // is examined, so a thread keeps several table reads in flight. With the region's first axis
  // varying fastest, a batch of three is the x-1 / x / x+1 triple that shares one table line.
  // Only the HOME slot is read here. One lookup in eight has to walk on (a foreign key with the
  // passed-over bit), but in almost every warp some lane does, so walking inside this loop made
  // every warp pay a second and third dependent table read per offset; those lookups are noted in
  // a bit mask instead (64 offsets per chunk) and finished, thread by thread, after the chunk.
  constexpr int kUnroll = 3;
  for (int chunk0 = k_begin; chunk0 < k_end; chunk0 += 64) {
    const int chunk_end = min(k_end, chunk0 + 64);
    unsigned long long pending = 0ull;
    for (int k0 = chunk0; k0 < chunk_end; k0 += kUnroll) {
      unsigned long long key[kUnroll];
      ulonglong2 first[kUnroll];
      bool valid[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = min(k0 + u, chunk_end - 1);
        bool in_box = batch_ok && (k0 + u < chunk_end);
#pragma unroll
        for (int a = 0; a < D; ++a) in_box = in_box && (dist[a + 1] + (uint32_t)s_off[k * D + a] <= span[a + 1]);
        valid[u] = in_box;
        key[u] = (unsigned long long)(ckey + s_delta[k]);
        first[u] = make_ulonglong2(kEmptyKey, 0ull);
        if (in_box) first[u] = load_slot(slots + hash_key(key[u], capacity, pos_shift));
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int k = k0 + u;
        if (k < chunk_end) {  // uniform across the block
          const uint32_t found = (uint32_t)(first[u].y >> 32);
          uint32_t uid = 0xFFFFFFFFu;
          if (valid[u]) {
            if (first[u].x == key[u]) uid = found & ~kPassedBit;
            else if (first[u].x != kEmptyKey && (found & kPassedBit)) pending |= 1ull << (k - chunk0);
          }
          if (active) __stcs(nbr + (size_t)k * n_query + q, (int32_t)uid);
          const uint32_t hits = __ballot_sync(0xFFFFFFFFu, uid != 0xFFFFFFFFu);
          if (lane == 0) atomicAdd(&s_cnt[k], (uint32_t)__popc(hits));
        }
      }
    }
    while (pending) {  // the lookups that walk on: from the slot behind the home slot
      const int k = chunk0 + __ffsll((long long)pending) - 1;
      pending &= pending - 1ull;
      const unsigned long long key = (unsigned long long)(ckey + s_delta[k]);
      uint32_t s = next_slot(hash_key(key, capacity, pos_shift), capacity);
      for (uint32_t probe = 1; probe < (capacity >> 3); ++probe) {
        const ulonglong2 v = load_slot(slots + s);
        const uint32_t found = (uint32_t)(v.y >> 32);
        if (v.x == key) {
          __stcs(nbr + (size_t)k * n_query + q, (int32_t)(found & ~kPassedBit));
          atomicAdd(&s_cnt[k], 1u);
          break;
        }
        if (v.x == kEmptyKey || !(found & kPassedBit)) break;
        s = next_slot(s, capacity);
      }
    }
  }
  __syncthreads();
  for (int k = k_begin + threadIdx.x; k < k_end; k += kKmapBlock)
    block_counts[(size_t)k * n_blocks + blockIdx.x] = s_cnt[k];
  if (tail.ticket) scan_counts_in_last_block(tail, block_counts, n_blocks, K, 0);
}

// Self map with a point-symmetric region (stride-1 convolution: the query rows ARE the table's
// rows, offsets[K-1-k] == -offsets[k], offsets[K/2] == 0). A pair (q -> a) at offset k implies
// (a -> q) at offset K-1-k, so only the first K/2 offsets are probed; every hit also fills its
// mirror entry (one scattered 4-byte store instead of a second probe) and the centre offset is
// the identity. The mirrored half of nbr must hold -1 before the launch.
template <int W>
__global__ void __launch_bounds__(kKmapBlock) k_kmap_probe_self(
    const TableHeader* __restrict__ h, const Slot* __restrict__ slots,
    const int32_t* __restrict__ coords, uint32_t n, const int32_t* __restrict__ offsets, int K,
    int32_t* __restrict__ nbr, uint32_t* __restrict__ block_counts, uint32_t n_blocks,
    uint32_t* __restrict__ scan_ticket, const uint32_t* __restrict__ index_state, TailScan tail) {
  after_previous_kernel();
  if (index_state && *index_state == ~0u) return;  // kIndexInUse: k_kmap_blocks_self has written the map
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int D = W - 1;
  const int half = K / 2;
  const int k_begin = (int)((uint32_t)half * blockIdx.y / gridDim.y);
  const int k_end = (int)((uint32_t)half * (blockIdx.y + 1) / gridDim.y);
  if (!tail.ticket && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *scan_ticket = 0;
  long long* s_delta = reinterpret_cast<long long*>(smem_raw);   // [half]
  int32_t* s_off = reinterpret_cast<int32_t*>(s_delta + (half > 0 ? half : 1));  // [half][D]
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(s_off + (half > 0 ? half : 1) * D);  // [half]
  for (int i = k_begin * D + threadIdx.x; i < k_end * D; i += kKmapBlock) s_off[i] = offsets[i];
  for (int k = k_begin + threadIdx.x; k < k_end; k += kKmapBlock) {
    long long d = 0;
#pragma unroll
    for (int a = 0; a < D; ++a) d += (long long)offsets[k * D + a] << h->shift[a + 1];
    s_delta[k] = d;
    s_cnt[k] = 0;
  }
  __syncthreads();

  const uint32_t capacity = h->capacity, pos_shift = h->pos_shift;
  const uint32_t q = blockIdx.x * kKmapBlock + threadIdx.x;
  const bool active = q < n;
  int32_t c[W];
  if (active) {
    load_row<W>(coords, q, c);
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) c[i] = 0;
  }
  uint32_t dist[W], span[W];
  long long ckey = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const int32_t mn = h->mn[i];
    dist[i] = (uint32_t)c[i] - (uint32_t)mn;
    span[i] = (uint32_t)(h->mx[i] - mn);
    ckey += (long long)((long long)c[i] - (long long)mn) << h->shift[i];
  }
  const int lane = threadIdx.x & 31;
  if (active && blockIdx.y == 0) __stcs(nbr + (size_t)half * n + q, (int32_t)q);  // centre offset: identity
  // (Deferring the few lookups that walk past their home slot to a second loop, as the general builder does,
  // made this kernel slower: 0.153 against 0.144 ms.)
  for (int k = k_begin; k < k_end; ++k) {
    bool in_box = active;
#pragma unroll
    for (int a = 0; a < D; ++a) in_box = in_box && (dist[a + 1] + (uint32_t)s_off[k * D + a] <= span[a + 1]);
    uint32_t uid = 0xFFFFFFFFu;
    if (in_box) uid = table_find(slots, capacity, pos_shift, (unsigned long long)(ckey + s_delta[k]));
    if (active) {
      __stcs(nbr + (size_t)k * n + q, (int32_t)uid);
      if (uid != 0xFFFFFFFFu) nbr[(size_t)(K - 1 - k) * n + uid] = (int32_t)q;  // mirror entry
    }
    const uint32_t hits = __ballot_sync(0xFFFFFFFFu, uid != 0xFFFFFFFFu);
    if (lane == 0) atomicAdd(&s_cnt[k], (uint32_t)__popc(hits));
  }
  __syncthreads();
  for (int k = k_begin + threadIdx.x; k < k_end; k += kKmapBlock)
    block_counts[(size_t)k * n_blocks + blockIdx.x] = s_cnt[k];
  if (threadIdx.x == 0 && blockIdx.y == 0) {
    const uint32_t row0 = blockIdx.x * kKmapBlock;
    block_counts[(size_t)half * n_blocks + blockIdx.x] = row0 < n ? min((uint32_t)kKmapBlock, n - row0) : 0u;
  }
  if (tail.ticket) scan_counts_in_last_block(tail, block_counts, n_blocks, K, half);
}

// One block of 1024 threads per counted offset: exclusive scan of block_counts[k][0..n_blocks) in place, totals[k] = number
// of pairs of offset k. The last block to finish writes offset_ptr[0..K] = exclusive scan of the totals, to host_ptr too
// (mapped page-locked memory) where a host wants them.
// mirror_half > 0 (self map): offsets K-1-k and k hold the same number of pairs, so only the first mirror_half + 1 offsets
// have counts and blocks; the flag word records the half: the pair lists of the mirrored offsets are then the exchanged
// lists of their mirror offsets (written by k_kmap_pairs together with the originals).
__global__ void __launch_bounds__(1024) k_kmap_scan(uint32_t* __restrict__ block_counts, uint32_t n_blocks, int K,
                                                    int mirror_half, uint32_t* __restrict__ totals,
                                                    int64_t* __restrict__ offset_ptr, volatile int64_t* host_ptr) {
  after_previous_kernel();
  __shared__ uint32_t warp_sums[32];
  __shared__ int64_t warp_sums64[32];
  __shared__ uint32_t s_last;
  uint32_t* flags = totals + K;  // [0] "pair lists did not fit" (see rmn_kmap_pairs_status), [1] half, [2] ticket
  uint32_t* counts = block_counts + (size_t)blockIdx.x * n_blocks;
  const uint32_t per = (n_blocks + 1023u) / 1024u;
  const uint32_t begin = min(n_blocks, threadIdx.x * per), end = min(n_blocks, begin + per);
  uint32_t sum = 0;
  for (uint32_t i = begin; i < end; ++i) sum += counts[i];
  uint32_t incl = sum;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warp_sums[lane], wi = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t t = __shfl_up_sync(0xFFFFFFFFu, wi, d);
      if (lane >= d) wi += t;
    }
    warp_sums[lane] = wi - w;
    if (lane == 31) {
      totals[blockIdx.x] = wi;
      __threadfence();
      s_last = atomicAdd(flags + 2, 1u) == gridDim.x - 1 ? 1u : 0u;
    }
  }
  __syncthreads();
  uint32_t run = warp_sums[warp] + incl - sum;
  for (uint32_t i = begin; i < end; ++i) {
    uint32_t v = counts[i];
    counts[i] = run;
    run += v;
  }
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    flags[0] = 0;
    flags[1] = (uint32_t)mirror_half;
  }
  const int per_k = (K + 1023) / 1024, k0 = min(K, (int)threadIdx.x * per_k), k1 = min(K, k0 + per_k);
  auto total = [&](int k) { return __ldcg(totals + (k >= K - mirror_half ? K - 1 - k : k)); };
  int64_t sum64 = 0;
  for (int k = k0; k < k1; ++k) sum64 += total(k);
  int64_t incl64 = sum64;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int64_t t = __shfl_up_sync(0xFFFFFFFFu, incl64, d);
    if (lane >= d) incl64 += t;
  }
  if (lane == 31) warp_sums64[warp] = incl64;
  __syncthreads();
  int64_t pos = incl64 - sum64;
  for (int w = 0; w < warp; ++w) pos += warp_sums64[w];
  for (int k = k0; k < k1; ++k) {
    const uint32_t t = total(k);
    offset_ptr[k] = pos;
    if (host_ptr) host_ptr[k] = pos;
    if (k >= K - mirror_half) totals[k] = t;
    pos += t;
    if (k == K - 1) {
      offset_ptr[K] = pos;
      if (host_ptr) host_ptr[K] = pos;
    }
  }
}

// Block b covers query rows [b*256, b*256+256). Warp w handles offsets
// k = w, w+8, ...; for each it walks the 8 row groups of the block keeping a
// running prefix, so no block-level synchronisation is needed.
__device__ __forceinline__ void kmap_pairs_body(
    const int32_t* __restrict__ nbr, uint32_t n_query, int K,
    const int64_t* __restrict__ offset_ptr, const uint32_t* __restrict__ block_prefix,
    uint32_t n_blocks, int32_t* __restrict__ a_idx, int32_t* __restrict__ q_idx,
    unsigned long long capacity, uint32_t* __restrict__ overflow) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t row0 = blockIdx.x * kKmapBlock;
  // Self map (flag word after the overflow word = K / 2): only the offsets up to the centre are walked;
  // a pair (a, q) of offset k < K / 2 is also stored, exchanged, at the same rank of offset K-1-k, whose
  // list therefore comes out sorted by table row.
  const int mirror_half = (int)overflow[1];
  const int K_full = K;
  K -= mirror_half;
  for (int k = warp; k < K; k += (int)(blockDim.x >> 5)) {
    const unsigned long long base = (unsigned long long)offset_ptr[k];
    unsigned long long pos = base + block_prefix[(size_t)k * n_blocks + blockIdx.x];
    const bool mirror = k < mirror_half;
    const unsigned long long mbase = mirror ? (unsigned long long)offset_ptr[K_full - 1 - k] : 0ull;
    // all eight row groups are loaded before the first ballot (eight independent 128-byte reads in flight)
    int32_t av[kKmapBlock / 32];
#pragma unroll
    for (int g = 0; g < kKmapBlock / 32; ++g) {
      const uint32_t q = row0 + g * 32 + lane;
      av[g] = q < n_query ? __ldcs(nbr + (size_t)k * n_query + q) : -1;
    }
#pragma unroll
    for (int g = 0; g < kKmapBlock / 32; ++g) {
      const uint32_t q = row0 + g * 32 + lane;
      const int32_t a = av[g];
      const uint32_t hits = __ballot_sync(0xFFFFFFFFu, a >= 0);
      if (a >= 0) {
        const unsigned long long p = pos + __popc(hits & ((1u << lane) - 1u));
        if (p < capacity) {
          __stcs(a_idx + p, a);
          __stcs(q_idx + p, (int32_t)q);
        } else {
          *overflow = 1;
        }
        if (mirror) {
          const unsigned long long d = mbase + (p - base);
          if (d < capacity) {
            __stcs(a_idx + d, (int32_t)q);
            __stcs(q_idx + d, a);
          } else {
            *overflow = 1;
          }
        }
      }
      pos += __popc(hits);
    }
  }
}

__global__ void __launch_bounds__(kKmapBlock) k_kmap_pairs(
    const int32_t* __restrict__ nbr, uint32_t n_query, int K, const int64_t* __restrict__ offset_ptr,
    const uint32_t* __restrict__ block_prefix, uint32_t n_blocks, int32_t* __restrict__ a_idx,
    int32_t* __restrict__ q_idx, unsigned long long capacity, uint32_t* __restrict__ overflow) {
  kmap_pairs_body(nbr, n_query, K, offset_ptr, block_prefix, n_blocks, a_idx, q_idx, capacity, overflow);
}

// The same compaction built to become resident BESIDE a convolution CTA: 128 threads of at most 32 registers. A convolution
// CTA (768 threads x 80 registers) leaves 4096 registers of an SM free, and one shared-memory / L1 split serves all CTAs of
// an SM, so this kernel asks for the largest one. It runs at a fraction of the stand-alone speed (4 KB of loads in flight per
// SM); a pass with 14.8 M pairs takes 40 us longer with the lists than without.
__global__ void __maxnreg__(32) k_kmap_pairs_background(
    const int32_t* __restrict__ nbr, uint32_t n_query, int K, const int64_t* __restrict__ offset_ptr,
    const uint32_t* __restrict__ block_prefix, uint32_t n_blocks, int32_t* __restrict__ a_idx,
    int32_t* __restrict__ q_idx, unsigned long long capacity, uint32_t* __restrict__ overflow) {
  kmap_pairs_body(nbr, n_query, K, offset_ptr, block_prefix, n_blocks, a_idx, q_idx, capacity, overflow);
}

// n entries "no neighbour" (a launch that overlaps its neighbours, where a memset would not)
__global__ void __launch_bounds__(256) k_kmap_clear(int32_t* __restrict__ nbr, size_t n, uint32_t* __restrict__ ticket) {
  after_previous_kernel();
  if (ticket && blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
  // single words up to the first 16-byte boundary and behind the last one
  const size_t head = min(n, (size_t)(((16 - ((uintptr_t)nbr & 15)) & 15) / 4)), vecs = (n - head) / 4, tail = head + 4 * vecs;
  const size_t first = (size_t)blockIdx.x * 256 + threadIdx.x, step = (size_t)gridDim.x * 256;
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (size_t i = first; i < vecs; i += step) reinterpret_cast<uint4*>(nbr + head)[i] = ones;
  if (first < head) nbr[first] = -1;
  if (tail + first < n) nbr[tail + first] = -1;
}
inline cudaError_t clear_entries(int32_t* nbr, size_t n, uint32_t* ticket, cudaStream_t stream) {
  const size_t blocks = (n / 4 + 255) / 256 + 1;
  count_launch();
  return launch_overlapped(k_kmap_clear, dim3((uint32_t)(blocks < 148 * 8 ? blocks : 148 * 8)), dim3(256), 0, stream, nbr, n, ticket);
}

// The public map from an ordered one. k_kmap_positions: the position of every row, and which of its entries exist, a bit each, in
// the row's words of `masks` [words][n]. k_kmap_unorder, offset by offset: entries of neighbouring rows lie anywhere in the 4 n bytes
// of that offset, of which what is read again is in the L2 (19 MB for 4.8 M rows), whose 32-byte pieces bound it; so only the
// entries that exist are read. The masks lie in the last offsets' places in the public table, which a launch without them fills
// at the end. Counts are those of k_kmap_probe_self. us, before the masks
// and with them: 4.8 M shuffled clip rows x 81 offsets at 32 % 1750 and 1363, 2.1 M voxels of rooms x 27 at 46 % 271 and 214, 2.2 M
// of lidar sweeps x 27 in their own order 117 and 153.
__global__ void __launch_bounds__(256) k_kmap_positions(const int32_t* __restrict__ order, const int32_t* __restrict__ ordered,
                                                        uint32_t n, int K, int32_t* __restrict__ position,
                                                        uint32_t* __restrict__ masks, uint32_t* __restrict__ scan_ticket) {
  after_previous_kernel();
  const uint32_t p = blockIdx.x * 256 + threadIdx.x;
  if (p == 0) *scan_ticket = 0;
  if (p >= n) return;
  const uint32_t row = (uint32_t)__ldg(order + p);
  position[row] = (int32_t)p;
  for (int k0 = 0; k0 < K; k0 += 32, masks += n) {
    uint32_t mask = 0;
#pragma unroll 8
    for (int k = k0; k < min(k0 + 32, K); ++k) mask |= (__ldcs(ordered + (size_t)k * n + p) >= 0 ? 1u : 0u) << (k - k0);
    masks[row] = mask;
  }
}
constexpr int kUnorderBlocks = 4;  // blocks of kKmapBlock rows that a CUDA block takes
__global__ void __launch_bounds__(kKmapBlock) k_kmap_unorder(const int32_t* __restrict__ ordered, const int32_t* __restrict__ position,
                                                             const uint32_t* masks, uint32_t n, int k0, int half, int32_t* nbr,
                                                             uint32_t* __restrict__ block_counts, uint32_t n_blocks) {
  after_previous_kernel();
  const int k = k0 + (int)blockIdx.y;
  const size_t first = (size_t)k * n;
  const uint32_t block0 = blockIdx.x * kUnorderBlocks;
  uint32_t exists[kUnorderBlocks];
  int32_t v[kUnorderBlocks];
#pragma unroll
  for (int j = 0; j < kUnorderBlocks; ++j) {
    const uint32_t row = (block0 + j) * kKmapBlock + threadIdx.x;
    exists[j] = row >= n ? 0u : masks ? (masks[(size_t)(k / 32) * n + row] >> (k & 31)) & 1u : 1u;
  }
#pragma unroll
  for (int j = 0; j < kUnorderBlocks; ++j) {
    const uint32_t row = (block0 + j) * kKmapBlock + threadIdx.x;
    v[j] = exists[j] ? __ldg(ordered + first + (uint32_t)__ldg(position + row)) : -1;
  }
#pragma unroll
  for (int j = 0; j < kUnorderBlocks; ++j) {
    const uint32_t row = (block0 + j) * kKmapBlock + threadIdx.x;
    if (row < n) __stcs(nbr + first + row, v[j]);
    if (k > half) continue;
    const int count = __syncthreads_count(v[j] >= 0);
    if (threadIdx.x == 0 && block0 + j < n_blocks) block_counts[(size_t)k * n_blocks + block0 + j] = (uint32_t)count;
  }
}

__global__ void __launch_bounds__(256) k_kmap_transpose(const int32_t* __restrict__ nbr,
                                                        uint32_t n_query, int K, uint32_t n_a,
                                                        int32_t* __restrict__ nbr_t) {
  after_previous_kernel();
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (uint64_t)K * n_query) return;
  const int32_t a = __ldg(nbr + i);
  if (a < 0 || (uint32_t)a >= n_a) return;
  const uint64_t k = i / n_query;
  const uint32_t q = (uint32_t)(i - k * n_query);
  nbr_t[k * n_a + (uint32_t)a] = (int32_t)q;
}

inline uint32_t kmap_blocks(uint32_t n_query) { return (n_query + kKmapBlock - 1) / kKmapBlock; }

// Self maps of three and more dimensions whose hash table takes most of the 126 MB L2 (94 MB from 1.97 M rows on, see
// table_capacity) may go over the occupancy index, see k_block_choose; below that a probe of the table is an L2 hit in any order
// of the rows (1.2 M shuffled rows x 27 offsets: 137 us by probing, 240 us with the index).
inline bool may_use_block_index(uint32_t n, int W, int K) {
  return W >= 4 && (size_t)n * 64 > ((size_t)120 << 20) && (K & 1) && K >= 9 && K <= 2048;
}

// counts per (offset, 256 query rows), totals, flags
inline size_t kmap_counts_bytes(uint32_t n_query, int K) {
  return (((size_t)K * kmap_blocks(n_query) + (size_t)K + 64) * sizeof(uint32_t) + 255) & ~(size_t)255;
}

}  // namespace rmn

#include "rmn_kmap_blocks.cuh"

using namespace rmn;

extern "C" int rmn_region_volume(int region_type, int D, const int32_t* kernel_size, int n_custom) {
  if (D < 1 || D >= RMN_MAX_W) return -RMN_ERR_BAD_ARG;
  if (region_type == RMN_CUSTOM) return n_custom;
  if (!kernel_size) return -RMN_ERR_BAD_ARG;
  long long v = 1;
  if (region_type == RMN_HYPER_CUBE) {
    for (int a = 0; a < D; ++a) v *= kernel_size[a];
  } else if (region_type == RMN_HYPER_CROSS) {
    for (int a = 0; a < D; ++a) v += kernel_size[a] - 1;
  } else {
    return -RMN_ERR_BAD_ARG;
  }
  return v > 0 && v < (1 << 20) ? (int)v : -RMN_ERR_BAD_ARG;
}

extern "C" int rmn_region_offsets(int region_type, int D, const int32_t* kernel_size,
                                  const int32_t* dilation, const int32_t* tensor_stride,
                                  const int32_t* custom_offsets, int n_custom, int32_t* offsets) {
  const int K = rmn_region_volume(region_type, D, kernel_size, n_custom);
  if (K < 0) return K;
  if (!dilation || !tensor_stride || !offsets) return -RMN_ERR_BAD_ARG;
  if (region_type == RMN_CUSTOM && n_custom > 0 && !custom_offsets) return -RMN_ERR_BAD_ARG;
  for (int k = 0; k < K; ++k) {
    int32_t* o = offsets + (size_t)k * D;
    for (int a = 0; a < D; ++a) o[a] = 0;
    if (region_type == RMN_HYPER_CUBE) {
      int idx = k;
      for (int a = 0; a < D; ++a) {
        const int ks = kernel_size[a];
        const int cur = idx % ks;
        const int step = dilation[a] * tensor_stride[a];
        o[a] = (ks % 2 == 0) ? cur * step : (cur - ks / 2) * step;
        idx /= ks;
      }
    } else if (region_type == RMN_HYPER_CROSS) {
      if (k == 0) continue;
      int ind = k - 1, axis = 0;
      while (axis < D && ind >= kernel_size[axis] - 1) {
        ind -= kernel_size[axis] - 1;
        ++axis;
      }
      const int r = (kernel_size[axis] - 1) / 2;
      const int co = ind < r ? ind + 1 : ind - 2 * r;
      o[axis] = co * dilation[axis] * tensor_stride[axis];
    } else {
      for (int a = 0; a < D; ++a)
        o[a] = (int32_t)((long long)custom_offsets[(size_t)k * D + a] * tensor_stride[a] *
                         dilation[a]);
    }
  }
  return K;
}

extern "C" size_t rmn_kmap_workspace_bytes(uint32_t n_query, int K) {
  if (K < 1) K = 1;
  return kmap_counts_bytes(n_query, K) + (may_use_block_index(n_query, RMN_MAX_W, K) ? block_index_bytes(n_query) : 0);
}

// Blocks that share the offsets of a row block (gridDim.y): about four blocks per SM in all, three offsets each at least.
static unsigned offset_split(uint32_t n_blocks, int K) {
  const uint32_t want = 148u * 4u / n_blocks, most = ((uint32_t)K + 2u) / 3u;
  const uint32_t split = want < most ? want : most;
  return split > 1 ? split : 1u;
}

static int kmap_build(const void* d_table, const int32_t* d_query, uint32_t n_query, int W, const int32_t* d_offsets, int K,
                      bool self, int32_t* d_nbr, int64_t* d_offset_ptr, void* d_workspace, size_t workspace_bytes,
                      int64_t* host_ptr, cudaStream_t stream) {
  if (!d_table || W < 2 || W > RMN_MAX_W || K < 1 || K > 4096 || (self && (K & 1) == 0) || !d_offsets || !d_offset_ptr ||
      !d_workspace)
    return RMN_ERR_BAD_ARG;
  if (workspace_bytes < rmn_kmap_workspace_bytes(n_query, K)) return RMN_ERR_ALLOC;
  if (n_query == 0) {
    RMN_CUDA_TRY(cudaMemsetAsync(d_offset_ptr, 0, sizeof(int64_t) * (K + 1), stream));
    if (host_ptr) memset(host_ptr, 0, sizeof(int64_t) * (K + 1));
    return RMN_OK;
  }
  if (!d_query || !d_nbr || !coords_aligned(d_query, W)) return RMN_ERR_BAD_ARG;
  int64_t* host_alias = nullptr;
  if (host_ptr) {
    void* p = nullptr;
    RMN_CUDA_TRY(cudaHostGetDevicePointer(&p, host_ptr, 0));
    host_alias = static_cast<int64_t*>(p);
  }
  const uint32_t nb = kmap_blocks(n_query);
  uint32_t* block_counts = reinterpret_cast<uint32_t*>(d_workspace);
  uint32_t* totals = block_counts + (size_t)K * nb;
  uint32_t* ticket = totals + K + 2;
  auto* h = reinterpret_cast<const TableHeader*>(d_table);
  auto* slots =
      reinterpret_cast<const Slot*>(reinterpret_cast<const char*>(d_table) + sizeof(TableHeader));
  const int half = self ? K / 2 : 0;
  const int hs = half > 0 ? half : 1;
  const TailScan tail{(uint64_t)(K - half) * nb <= kTailCounts ? ticket : nullptr, totals, d_offset_ptr, host_alias};
  const size_t self_smem = (size_t)hs * 8 + (size_t)hs * (W - 1) * 4 + (size_t)hs * 4;
  if (self && may_use_block_index(n_query, W, K) && ((uintptr_t)d_workspace & 15) == 0) {
    const BlockIndex ix = block_index(static_cast<char*>(d_workspace) + kmap_counts_bytes(n_query, K), n_query);
    const dim3 grid(148 * 8), block(256);
    const size_t smem = (size_t)8 * kKmapBlock * 12 + (size_t)K * 4 + (size_t)half * 4;
    RMN_DISPATCH_W(W, if constexpr (kW >= 4) {
      BlockSample* sample = reinterpret_cast<BlockSample*>(ix.perm);
      RMN_CUDA_TRY(launch_overlapped(k_block_sample<kW>, dim3(kChooseRows / 256), block, 0, stream, h, slots, d_query, n_query,
                                     sample));
      RMN_LAUNCH_CHECK();
      RMN_CUDA_TRY(launch_overlapped(k_block_choose, dim3(148 * 2), dim3(1024), 0, stream, h, n_query, sample, ix,
                                     d_nbr + (size_t)(half + 1) * n_query, (size_t)half * n_query));
      RMN_LAUNCH_CHECK();
      RMN_CUDA_TRY(launch_overlapped(k_block_insert<kW>, grid, block, 0, stream, h, d_query, n_query, ix));
      RMN_LAUNCH_CHECK();
      RMN_CUDA_TRY(launch_overlapped(k_block_bases, dim3((ix.capacity + 255) / 256), block, 0, stream, ix));
      RMN_LAUNCH_CHECK();
      RMN_CUDA_TRY(launch_overlapped(k_block_scatter<kW>, grid, block, 0, stream, h, d_query, n_query, ix));
      RMN_LAUNCH_CHECK();
      RMN_CUDA_TRY(launch_overlapped(k_kmap_blocks_self<kW>, dim3(148 * 6), dim3(kKmapBlock), smem, stream, h, slots, d_query,
                                     n_query, d_offsets, K, d_nbr, block_counts, nb, ticket, ix));
      RMN_LAUNCH_CHECK();
      RMN_CUDA_TRY(launch_overlapped(k_kmap_probe_self<kW>, dim3(nb, offset_split(nb, half)), dim3(kKmapBlock), self_smem,
                                     stream, h, slots, d_query, n_query, d_offsets, K, d_nbr, block_counts, nb, ticket,
                                     ix.state, TailScan{}));
    });
  } else if (self) {
    if (half > 0 || tail.ticket)  // the mirrored half starts as "no neighbour"
      RMN_CUDA_TRY(clear_entries(d_nbr + (size_t)(half + 1) * n_query, (size_t)half * n_query, tail.ticket, stream));
    RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_kmap_probe_self<kW>, dim3(nb, offset_split(nb, half)), dim3(kKmapBlock),
                                                     self_smem, stream, h, slots, d_query, n_query, d_offsets, K, d_nbr,
                                                     block_counts, nb, ticket, nullptr, tail)));
  } else {
    if (tail.ticket) RMN_CUDA_TRY(clear_entries(d_nbr, 0, tail.ticket, stream));
    const size_t smem = (size_t)K * 8 + (size_t)K * (W - 1) * 4 + (size_t)K * 4;
    RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(
                        k_kmap_probe<kW>, dim3(nb, offset_split(nb, K)), dim3(kKmapBlock), smem, stream, h, slots, d_query, n_query, d_offsets, K, d_nbr, block_counts, nb, ticket, tail)));
  }
  RMN_LAUNCH_CHECK();
  if (tail.ticket) return RMN_OK;
  RMN_CUDA_TRY(launch_overlapped(k_kmap_scan, dim3(self ? half + 1 : K), dim3(1024), 0, stream,
                        block_counts, nb, K, half, totals, d_offset_ptr, host_alias));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" size_t rmn_kmap_ordered_workspace_bytes(uint32_t n_rows, int W, int K) {
  if (W > RMN_MAX_W || !may_use_block_index(n_rows, W, K)) return 0;
  return kmap_counts_bytes(n_rows, K) + block_index_bytes(n_rows, true) + kBlockBuckets * sizeof(uint32_t) + 32;
}

extern "C" int rmn_kmap_build_ordered(const void* d_table, const int32_t* d_coords, uint32_t n_rows, int W,
                                      const int32_t* d_offsets, int K, int32_t* d_order, int32_t* d_nbr, void* d_workspace,
                                      size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  const size_t need = rmn_kmap_ordered_workspace_bytes(n_rows, W, K);
  if (need == 0) return RMN_ERR_UNSUPPORTED;
  if (!d_table || !d_coords || !d_offsets || !d_order || !d_nbr || !d_workspace || !coords_aligned(d_coords, W) ||
      ((uintptr_t)d_workspace & 15))
    return RMN_ERR_BAD_ARG;
  if (workspace_bytes < need) return RMN_ERR_ALLOC;
  auto* h = reinterpret_cast<const TableHeader*>(d_table);
  auto* slots = reinterpret_cast<const Slot*>(reinterpret_cast<const char*>(d_table) + sizeof(TableHeader));
  // counts of the probing kernel (not needed, but it keeps them), the index, the buckets
  uint32_t* counts = static_cast<uint32_t*>(d_workspace);
  const uint32_t nb = kmap_blocks(n_rows);
  char* index = static_cast<char*>(d_workspace) + kmap_counts_bytes(n_rows, K);
  BlockIndex ix = block_index(index, n_rows, true);
  BlockSample* sample = reinterpret_cast<BlockSample*>(ix.perm);
  ix.perm = d_order;
  ix.buckets = reinterpret_cast<uint32_t*>(index + ((block_index_bytes(n_rows, true) + 15) & ~(size_t)15));
  const int half = K / 2;
  const dim3 grid(148 * 8), block(256), slot_grid((ix.capacity + 255) / 256);
  const size_t self_smem = (size_t)half * 8 + (size_t)half * (W - 1) * 4 + (size_t)half * 4;
  RMN_DISPATCH_W(W, if constexpr (kW >= 4) {
    RMN_CUDA_TRY(launch_overlapped(k_block_sample<kW>, dim3(kChooseRows / 256), block, 0, stream, h, slots, d_coords, n_rows,
                                   sample));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_block_choose, dim3(148 * 2), dim3(1024), 0, stream, h, n_rows, sample, ix,
                                   d_nbr + (size_t)(half + 1) * n_rows, (size_t)half * n_rows));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_block_insert<kW>, grid, block, 0, stream, h, d_coords, n_rows, ix));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_block_assign<false>, slot_grid, block, 0, stream, h, ix));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_block_bucket_sums, dim3(1), dim3(1024), 0, stream, ix));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_block_assign<true>, slot_grid, block, 0, stream, h, ix));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_block_scatter<kW>, grid, block, 0, stream, h, d_coords, n_rows, ix));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_kmap_ordered<kW>, dim3(148 * 4), dim3(kKmapBlock), ordered_smem(K), stream, h, slots,
                                   d_coords, n_rows, d_offsets, K, d_nbr, ix));
    RMN_LAUNCH_CHECK();
    RMN_CUDA_TRY(launch_overlapped(k_kmap_probe_self<kW>, dim3(nb, offset_split(nb, half)), dim3(kKmapBlock), self_smem, stream,
                                   h, slots, d_coords, n_rows, d_offsets, K, d_nbr, counts, nb,
                                   counts + (size_t)K * nb + K + 2, ix.state, TailScan{}));
    RMN_LAUNCH_CHECK();
  });
  return RMN_OK;
}

extern "C" int rmn_kmap_build_from_ordered(const int32_t* d_order, const int32_t* d_ordered_nbr, uint32_t n_rows, int K,
                                           int32_t* d_nbr, int64_t* d_offset_ptr, int64_t* host_ptr, void* d_workspace,
                                           size_t workspace_bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (rmn_kmap_ordered_workspace_bytes(n_rows, RMN_MAX_W, K) == 0) return RMN_ERR_UNSUPPORTED;
  if (!d_order || !d_ordered_nbr || !d_nbr || !d_offset_ptr || !d_workspace || ((uintptr_t)d_workspace & 15)) return RMN_ERR_BAD_ARG;
  if (workspace_bytes < rmn_kmap_workspace_bytes(n_rows, K)) return RMN_ERR_ALLOC;
  int64_t* host_alias = nullptr;
  if (host_ptr) RMN_CUDA_TRY(cudaHostGetDevicePointer(reinterpret_cast<void**>(&host_alias), host_ptr, 0));
  const uint32_t nb = kmap_blocks(n_rows);
  const int half = K / 2;
  uint32_t* block_counts = static_cast<uint32_t*>(d_workspace);
  uint32_t* totals = block_counts + (size_t)K * nb;
  // (where a build has its index)
  int32_t* position = reinterpret_cast<int32_t*>(static_cast<char*>(d_workspace) + kmap_counts_bytes(n_rows, K));
  const int words = (K + 31) / 32, masked = K - words;
  uint32_t* masks = reinterpret_cast<uint32_t*>(d_nbr + (size_t)masked * n_rows);
  RMN_CUDA_TRY(launch_overlapped(k_kmap_positions, dim3((n_rows + 255) / 256), dim3(256), 0, stream, d_order, d_ordered_nbr, n_rows, K,
                                 position, masks, totals + K + 2));
  RMN_LAUNCH_CHECK();
  const uint32_t row_blocks = (nb + kUnorderBlocks - 1) / kUnorderBlocks;
  for (const uint32_t* m = masks;; m = nullptr) {
    RMN_CUDA_TRY(launch_overlapped(k_kmap_unorder, dim3(row_blocks, m ? masked : words), dim3(kKmapBlock), 0, stream, d_ordered_nbr,
                                   (const int32_t*)position, m, n_rows, m ? 0 : masked, half, d_nbr, block_counts, nb));
    RMN_LAUNCH_CHECK();
    if (!m) break;
  }
  RMN_CUDA_TRY(launch_overlapped(k_kmap_scan, dim3(half + 1), dim3(1024), 0, stream, block_counts, nb, K, half, totals, d_offset_ptr,
                                 host_alias));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_kmap_build(const void* d_table, const int32_t* d_query, uint32_t n_query, int W,
                              const int32_t* d_offsets, int K, int32_t* d_nbr,
                              int64_t* d_offset_ptr, void* d_workspace, size_t workspace_bytes,
                              void* stream_) {
  return kmap_build(d_table, d_query, n_query, W, d_offsets, K, false, d_nbr, d_offset_ptr, d_workspace, workspace_bytes,
                    nullptr, (cudaStream_t)stream_);
}

extern "C" int rmn_kmap_build_self(const void* d_table, const int32_t* d_coords, uint32_t n_rows, int W,
                                   const int32_t* d_offsets, int K, int32_t* d_nbr, int64_t* d_offset_ptr,
                                   void* d_workspace, size_t workspace_bytes, void* stream_) {
  return kmap_build(d_table, d_coords, n_rows, W, d_offsets, K, true, d_nbr, d_offset_ptr, d_workspace, workspace_bytes,
                    nullptr, (cudaStream_t)stream_);
}

extern "C" int rmn_kmap_build_host(const void* d_table, const int32_t* d_query, uint32_t n_query, int W,
                                   const int32_t* d_offsets, int K, int self, int32_t* d_nbr, int64_t* d_offset_ptr,
                                   int64_t* h_offset_ptr_pinned, void* d_workspace, size_t workspace_bytes, void* stream_) {
  if (!h_offset_ptr_pinned) return RMN_ERR_BAD_ARG;
  return kmap_build(d_table, d_query, n_query, W, d_offsets, K, self != 0, d_nbr, d_offset_ptr, d_workspace,
                    workspace_bytes, h_offset_ptr_pinned, (cudaStream_t)stream_);
}

static int kmap_pairs_launch(const int32_t* d_nbr, uint32_t n_query, int K, const int64_t* d_offset_ptr,
                             const void* d_workspace, int32_t* d_a_idx, int32_t* d_q_idx, uint64_t capacity,
                             cudaStream_t stream, bool background) {
  if (K < 1 || !d_offset_ptr || !d_workspace) return RMN_ERR_BAD_ARG;
  if (n_query == 0 || capacity == 0) return RMN_OK;
  if (!d_nbr || !d_a_idx || !d_q_idx) return RMN_ERR_BAD_ARG;
  const uint32_t nb = kmap_blocks(n_query);
  const uint32_t* block_prefix = reinterpret_cast<const uint32_t*>(d_workspace);
  // the word after the totals flags a capacity overflow (zeroed by the build, read by rmn_kmap_pairs_status)
  uint32_t* overflow = const_cast<uint32_t*>(block_prefix) + (size_t)K * nb + K;
  if (!background) {
    k_kmap_pairs<<<nb, kKmapBlock, 0, stream>>>(d_nbr, n_query, K, d_offset_ptr, block_prefix, nb, d_a_idx,
                                                d_q_idx, capacity, overflow);
  } else {
    static std::once_flag once[64];
    int dev = 0;
    RMN_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64)
      std::call_once(once[dev], [] {
        cudaFuncSetAttribute(k_kmap_pairs_background, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
      });
    k_kmap_pairs_background<<<nb, 128, 0, stream>>>(d_nbr, n_query, K, d_offset_ptr, block_prefix, nb, d_a_idx,
                                                    d_q_idx, capacity, overflow);
  }
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_kmap_pairs_status(const void* d_workspace, uint32_t n_query, int K, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (K < 1 || !d_workspace) return RMN_ERR_BAD_ARG;
  if (n_query == 0) return RMN_OK;
  const uint32_t* flag = reinterpret_cast<const uint32_t*>(d_workspace) + (size_t)K * kmap_blocks(n_query) + K;
  uint32_t v = 0;
  RMN_CUDA_TRY(cudaMemcpyAsync(&v, flag, sizeof(v), cudaMemcpyDeviceToHost, stream));
  RMN_CUDA_TRY(cudaStreamSynchronize(stream));
  return v ? RMN_ERR_ALLOC : RMN_OK;
}

extern "C" int rmn_kmap_pairs(const int32_t* d_nbr, uint32_t n_query, int K,
                              const int64_t* d_offset_ptr, const void* d_workspace,
                              int32_t* d_a_idx, int32_t* d_q_idx, uint64_t capacity,
                              void* stream_) {
  return kmap_pairs_launch(d_nbr, n_query, K, d_offset_ptr, d_workspace, d_a_idx, d_q_idx, capacity,
                           (cudaStream_t)stream_, false);
}

extern "C" int rmn_kmap_pairs_background(const int32_t* d_nbr, uint32_t n_query, int K,
                                         const int64_t* d_offset_ptr, const void* d_workspace,
                                         int32_t* d_a_idx, int32_t* d_q_idx, uint64_t capacity,
                                         void* stream_) {
  return kmap_pairs_launch(d_nbr, n_query, K, d_offset_ptr, d_workspace, d_a_idx, d_q_idx, capacity,
                           (cudaStream_t)stream_, true);
}

extern "C" int rmn_kmap_transpose(const int32_t* d_nbr, uint32_t n_query, int K, uint32_t n_a,
                                  int32_t* d_nbr_t, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (K < 1) return RMN_ERR_BAD_ARG;
  if (n_a == 0) return RMN_OK;
  if (!d_nbr_t) return RMN_ERR_BAD_ARG;
  RMN_CUDA_TRY(clear_entries(d_nbr_t, (size_t)K * n_a, nullptr, stream));
  if (n_query == 0) return RMN_OK;
  if (!d_nbr) return RMN_ERR_BAD_ARG;
  const uint64_t total = (uint64_t)K * n_query;
  RMN_CUDA_TRY(launch_overlapped(k_kmap_transpose, dim3((uint32_t)((total + 255) / 256)), dim3(256), 0, stream, d_nbr, n_query, K,
                                 n_a, d_nbr_t));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}
