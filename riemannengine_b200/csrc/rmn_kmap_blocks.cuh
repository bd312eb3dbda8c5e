// Self map over an occupancy index: the rows of a map grouped into 4 x 4 x 4 blocks of voxels, one 64-bit mask per block.
//
// What bounds k_kmap_probe_self on a large map whose rows come in no spatial order is random access: a hash-table line per
// (row, x-triple of offsets), and for every hit a scattered 4-byte store of the mirror entry into a table that no cache holds;
// once the table lines that the rows of a stretch touch exceed the L2 the probes go to DRAM as well. Here a row looks up the
// blocks that its neighbourhood can touch (at most 8 per position on the axes behind the third; the slots of all blocks stay
// in L2), and every offset is a bit test; a hit ranks its bit in the mask and reads the row number from `perm`, where the rows
// of a block lie next to one another. All K offsets are computed, nothing is mirrored, and the table is written once,
// coalesced. 4.8 M rows of four shuffled clips x 81 offsets: 3650 us by probing, 2324 with the index, still bound by the row
// numbers' random reads (26 per row; more registers or wider shared entries leave less L1 and are slower: 2030 and 2350 us
// against 1980 us for the kernel alone). Rows that do come in spatial order are probed in 1480 us and take 2240 with the index,
// and thin clouds 290 and 1080: k_block_choose decides on the device, and where the index does not serve, its kernels end at
// once and k_kmap_probe_self runs behind them (25 - 30 us later than it would by itself).
//
// Included by rmn_kmap.cu.
#pragma once

namespace rmn {

struct __align__(32) BlockSlot {  // one 32-byte sector: a lookup is one access
  unsigned long long key;   // packed block coordinates, kEmptyKey when free
  unsigned long long free;  // bit per voxel of the block: 0 where a row exists (so that a fill with ones is "empty")
  uint32_t base;            // position in perm of the first row of the block
  uint32_t pad[3];
};

// Index in a workspace of block_index_bytes(n). One slot per eight rows, so that the slots fit the L2 where the hash table
// does not: a surface fills a block with about twenty rows. Rows that lie too thinly for that (a lidar sweep) do not fit.
struct BlockIndex {
  BlockSlot* slots;
  uint32_t* counter;      // rows numbered so far, minus one
  uint32_t* state;        // one of the three below
  int32_t* perm;          // row numbers, block by block
  uint32_t* slot_of_row;  // build scratch
  uint32_t* buckets;      // of an ordered map (k_block_assign), NULL otherwise
  uint32_t capacity;
};
constexpr uint32_t kBlockBucketBits = 13, kBlockBuckets = 1u << kBlockBucketBits;
constexpr uint32_t kIndexInUse = ~0u, kIndexNotChosen = 0u, kIndexFull = 1u;  // full: the blocks did not fit
// (a surface loads two slots in five: runs of 32 taken slots occur, runs of 128 do not; 4.8 M clip rows overflowed at 32 in
// some scenes, and took 3.0 ms by the hash table)
constexpr uint32_t kBlockMaxProbes = 128;
// (For an ordered map, whose lookups wait for the longest of 27, it is one per four: 1141 -> 1004 us.)
inline uint32_t block_index_capacity(uint32_t n, bool ordered = false) { return n / (ordered ? 4 : 8) + 64; }
inline size_t block_index_bytes(uint32_t n, bool ordered = false) {
  return (size_t)block_index_capacity(n, ordered) * sizeof(BlockSlot) + 32 + (size_t)n * 8;
}
inline BlockIndex block_index(void* workspace, uint32_t n, bool ordered = false) {
  BlockIndex b;
  b.capacity = block_index_capacity(n, ordered);
  b.slots = static_cast<BlockSlot*>(workspace);
  b.counter = reinterpret_cast<uint32_t*>(b.slots + b.capacity);
  b.state = b.counter + 1;
  b.perm = reinterpret_cast<int32_t*>(b.counter + 8);
  b.slot_of_row = reinterpret_cast<uint32_t*>(b.perm + n);
  b.buckets = nullptr;
  return b;
}

__device__ __forceinline__ uint32_t block_hash(unsigned long long key, uint32_t capacity) {
  uint32_t h = (uint32_t)key ^ ((uint32_t)(key >> 32) * 0x9E3779B1u);
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return __umulhi(h, capacity);
}

// Coordinates of a row relative to the box, split into block and position. The first three spatial columns are the block's
// axes (in fewer dimensions a block has too few rows for the index); the low bits that all rows share (tensor stride) are left
// out of them.
template <int W>
struct BlockCoords {
  static_assert(W >= 4, "three spatial columns");
  static constexpr int NA = 3;
  uint32_t local;           // 2 bits per block axis, in nibbles
  uint32_t block[NA];       // block coordinate per block axis
  unsigned long long key;   // packed block coordinates with the remaining columns
  uint32_t dist[W];         // distance from the box minimum per column

  __device__ __forceinline__ void load(const TableHeader* h, const int32_t (&c)[W]) {
    local = 0;
    key = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      dist[i] = (uint32_t)c[i] - (uint32_t)h->mn[i];
      unsigned long long field = dist[i];
      if (i >= 1 && i <= NA) {
        const uint32_t s = h->low_shift(i - 1);
        local |= ((dist[i] >> s) & 3u) << (4 * (i - 1));
        block[i - 1] = (dist[i] >> s) >> 2;
        field = block[i - 1];
      }
      key |= field << h->shift[i];
    }
  }
  static __device__ __forceinline__ uint32_t bit(uint32_t nibbles) {  // position of a voxel in its block's mask
    return (nibbles & 3u) | ((nibbles >> 2) & 0xCu) | ((nibbles >> 4) & 0x30u);
  }
};

// Whether the index serves this map, by two samples of its rows.
// Working set: the part of the hash table that the rows of a stretch touch goes with the part of the map's space which the
// stretch covers. Of 8192 rows in sequence every other one marks its coarse cell (eight per block axis, four on the other
// axes); the part of 8192 rows spread over the map that lie in marked cells, by the same part of the stretch's other rows (the
// marks do not reach every cell), is the part covered. Measured, by (part x table): 27 offsets, 41 MiB 650 us probed and 801
// with the index, 48 MiB 413 and 501, 55 MiB 1064 and 1037, 61 MiB 606 and 621, 82 MiB 902 and 803, 219 MiB 1601 and 1058;
// 81 offsets, 14 MiB 1394 and 1822, 55 MiB 2585 and 1832.
// Density: 64 rows count the rows of their blocks in the hash table; the mean of 1 / count is blocks per row. With more than
// 0.6 of the slots taken, the runs of taken slots grow towards kBlockMaxProbes.
// k_block_sample reads the rows (a single SM would wait 50 us for these random reads); in k_block_choose every block counts and
// decides, then all clear the slots or, where k_kmap_probe_self will run, fill the mirrored half of the table with "no
// neighbour" - work that hides the launches of the kernels behind it.
constexpr uint32_t kChooseRows = 8192, kChooseCells = 47 * 1024, kChooseBlocks = 64;
constexpr float kChooseBytes = 51.f * (1 << 20), kChooseLoad = 0.6f;

struct BlockSample {                            // lies in perm, which is not needed before the choice
  uint16_t sequence[kChooseRows];               // coarse cells of rows in sequence
  uint16_t spread[kChooseRows];                 // and of rows spread over the map
  uint32_t rows[kChooseBlocks * 64 / 32];       // rows found by every 32 lookups of voxels, 64 per sampled block
};

template <int W>
__global__ void __launch_bounds__(256) k_block_sample(const TableHeader* __restrict__ h, const Slot* __restrict__ slots,
                                                      const int32_t* __restrict__ coords, uint32_t n,
                                                      BlockSample* __restrict__ sample) {
  after_previous_kernel();
  const uint32_t t = blockIdx.x * 256 + threadIdx.x;  // kChooseRows in all
  auto cell = [&](uint32_t row) {
    int32_t c[W];
    load_row<W>(coords, row, c);
    unsigned long long key = (uint32_t)c[0] - (uint32_t)h->mn[0];
#pragma unroll
    for (int a = 1; a < W; ++a) {
      const int width = 32 - __clz((int)((uint32_t)h->mx[a] - (uint32_t)h->mn[a])), bits = a <= 3 ? 3 : 2;
      key = key * 8 + (((uint32_t)c[a] - (uint32_t)h->mn[a]) >> (width > bits ? width - bits : 0));
    }
    return (uint16_t)block_hash(key, kChooseCells);
  };
  sample->sequence[t] = cell(n / 8 * 3 + t);
  sample->spread[t] = cell((uint32_t)((uint64_t)t * n / kChooseRows));
  if (t >= kChooseBlocks * 64) return;
  int32_t c[W];
  load_row<W>(coords, (uint32_t)((uint64_t)(t / 64) * n / kChooseBlocks), c);
  unsigned long long key = 0;
  bool in_box = true;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    uint32_t d = (uint32_t)c[i] - (uint32_t)h->mn[i];
    if (i >= 1 && i <= 3) {
      const uint32_t s = h->low_shift(i - 1);
      d = (((d >> s) & ~3u) | ((t >> (2 * (i - 1))) & 3u)) << s;
      in_box = in_box && d <= (uint32_t)h->mx[i] - (uint32_t)h->mn[i];
    }
    key |= (unsigned long long)d << h->shift[i];
  }
  const bool found = in_box && table_find(slots, h->capacity, h->pos_shift, key) != 0xFFFFFFFFu;
  const uint32_t votes = __ballot_sync(0xFFFFFFFFu, found);
  if ((t & 31) == 0) sample->rows[t / 32] = (uint32_t)__popc(votes);
}

__global__ void __launch_bounds__(1024) k_block_choose(const TableHeader* __restrict__ h, uint32_t n,
                                                       const BlockSample* __restrict__ sample, BlockIndex ix,
                                                       int32_t* __restrict__ mirrored, size_t n_mirrored) {
  after_previous_kernel();
  __shared__ __align__(16) uint8_t s_marked[kChooseCells];
  __shared__ uint32_t s_inside[2], s_serves;
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < kChooseCells / 16; i += 1024) reinterpret_cast<uint4*>(s_marked)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid < 2) s_inside[tid] = 0u;
  static_assert(kChooseRows == 8 * 1024, "rows of a thread");
  __align__(16) uint16_t sequence[8], spread[8];
  *reinterpret_cast<uint4*>(sequence) = reinterpret_cast<const uint4*>(sample->sequence)[tid];
  *reinterpret_cast<uint4*>(spread) = reinterpret_cast<const uint4*>(sample->spread)[tid];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; i += 2) s_marked[sequence[i]] = 1;
  __syncthreads();
  uint32_t near = 0, far = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i & 1) near += s_marked[sequence[i]];
    far += s_marked[spread[i]];
  }
  near = __reduce_add_sync(0xFFFFFFFFu, near);
  far = __reduce_add_sync(0xFFFFFFFFu, far);
  if ((tid & 31) == 0) {
    atomicAdd(&s_inside[0], near);
    atomicAdd(&s_inside[1], far);
  }
  __syncthreads();
  if (tid < 32) {
    float blocks = 0.f;
#pragma unroll
    for (uint32_t j = tid; j < kChooseBlocks; j += 32) blocks += 1.f / (float)(sample->rows[2 * j] + sample->rows[2 * j + 1]);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) blocks += __shfl_xor_sync(0xFFFFFFFFu, blocks, d);
    const float part = fminf(1.f, 0.5f * (float)s_inside[1] / (float)s_inside[0]);
    const float set = part * ((float)h->capacity * sizeof(Slot));
    if (tid == 0)
      s_serves = (ix.buckets || set > kChooseBytes) && blocks / kChooseBlocks * (float)n <= kChooseLoad * (float)(n / 8) ? 1u : 0u;
  }
  __syncthreads();
  const bool serves = s_serves != 0u;
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
  const size_t first = blockIdx.x * 1024 + tid, step = gridDim.x * 1024;
  if (first == 0) {
    *ix.state = serves ? kIndexInUse : kIndexNotChosen;
    *ix.counter = ~0u;
  }
  if (serves) {
    for (size_t i = first; i < 2 * (size_t)ix.capacity; i += step) reinterpret_cast<uint4*>(ix.slots)[i] = ones;
    if (ix.buckets)
      for (size_t i = first; i < kBlockBuckets; i += step) ix.buckets[i] = 0u;
  } else {  // single words up to the first 16-byte boundary and behind the last one
    const size_t head = ((16 - ((uintptr_t)mirrored & 15)) & 15) / 4, vecs = (n_mirrored - head) / 4;
    const size_t tail = head + 4 * vecs;
    for (size_t i = first; i < vecs; i += step) __stcs(reinterpret_cast<uint4*>(mirrored + head) + i, ones);
    if (first < head) mirrored[first] = -1;
    if (tail + first < n_mirrored) mirrored[tail + first] = -1;
  }
}

template <int W>
__global__ void __launch_bounds__(256) k_block_insert(const TableHeader* __restrict__ h, const int32_t* __restrict__ coords,
                                                      uint32_t n, BlockIndex ix) {
  after_previous_kernel();
  for (uint32_t row = blockIdx.x * 256 + threadIdx.x; row < n; row += gridDim.x * 256) {
    if (*(volatile uint32_t*)ix.state != kIndexInUse) return;
    int32_t c[W];
    load_row<W>(coords, row, c);
    BlockCoords<W> b;
    b.load(h, c);
    uint32_t s = block_hash(b.key, ix.capacity);
    bool placed = false;
    for (uint32_t probe = 0; probe < kBlockMaxProbes; ++probe) {
      unsigned long long cur = *(volatile unsigned long long*)&ix.slots[s].key;
      if (cur == kEmptyKey) cur = atomicCAS(&ix.slots[s].key, kEmptyKey, b.key);
      if (cur == kEmptyKey || cur == b.key) {
        placed = true;
        break;
      }
      if (++s == ix.capacity) s = 0;
    }
    if (!placed) {
      *(volatile uint32_t*)ix.state = kIndexFull;
      return;
    }
    atomicAnd(&ix.slots[s].free, ~(1ull << b.bit(b.local)));
    ix.slot_of_row[row] = s;
  }
}

// The ranges of perm in an ordered map: blocks that share the highest bits of their key - batch, further axes, layers of blocks along
// the third axis - lie together, so that the rows which a stretch of the convolution gathers stay in the L2. (Rows of blocks
// along the second axis, too: 1004 -> 992 us, and more to add up.) Rows per bucket, their exclusive sums (one block), and a
// range for every block.
__device__ __forceinline__ uint32_t block_bucket(const TableHeader* h, unsigned long long key) {
  return (uint32_t)(key >> (h->total_bits > kBlockBucketBits ? h->total_bits - kBlockBucketBits : 0u));
}
template <bool kAssign>
__global__ void __launch_bounds__(256) k_block_assign(const TableHeader* __restrict__ h, BlockIndex ix) {
  after_previous_kernel();
  if (*ix.state != kIndexInUse) return;
  const uint32_t s = blockIdx.x * 256 + threadIdx.x;
  if (s >= ix.capacity || ix.slots[s].key == kEmptyKey) return;
  const uint32_t first = atomicAdd(ix.buckets + block_bucket(h, ix.slots[s].key), (uint32_t)__popcll(~ix.slots[s].free));
  if constexpr (kAssign) ix.slots[s].base = first;
}
__global__ void __launch_bounds__(1024) k_block_bucket_sums(BlockIndex ix) {
  after_previous_kernel();
  if (*ix.state != kIndexInUse) return;
  __shared__ uint32_t s_warp[32];
  constexpr uint32_t PER = kBlockBuckets / 1024;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* mine = reinterpret_cast<uint4*>(ix.buckets + threadIdx.x * PER);
  uint32_t sum = 0;
  for (uint32_t i = 0; i < PER / 4; ++i) {
    const uint4 v = mine[i];
    sum += v.x + v.y + v.z + v.w;
  }
  uint32_t incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= (uint32_t)d) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t run = incl - sum;
  for (uint32_t w = 0; w < warp; ++w) run += s_warp[w];
  for (uint32_t i = 0; i < PER / 4; ++i) {
    const uint4 v = mine[i];
    mine[i] = make_uint4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
    run += v.x + v.y + v.z + v.w;
  }
}

// Gives every block its range of perm. Which range a block gets depends on the order of the atomics; what the index
// returns does not.
__global__ void __launch_bounds__(256) k_block_bases(BlockIndex ix) {
  after_previous_kernel();
  __shared__ uint32_t s_warp[8], s_base;
  if (*ix.state != kIndexInUse) return;
  const uint32_t s = blockIdx.x * 256 + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t count = s < ix.capacity ? (uint32_t)__popcll(~__ldg(&ix.slots[s].free)) : 0u;
  uint32_t incl = count;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const uint32_t v = s_warp[w];
      s_warp[w] = run;
      run += v;
    }
    s_base = run ? atomicAdd(ix.counter, run) + 1u : 0u;  // (the counter starts at all ones)
  }
  __syncthreads();
  if (count) ix.slots[s].base = s_base + s_warp[warp] + incl - count;
}

template <int W>
__global__ void __launch_bounds__(256) k_block_scatter(const TableHeader* __restrict__ h, const int32_t* __restrict__ coords,
                                                       uint32_t n, BlockIndex ix) {
  after_previous_kernel();
  if (*ix.state != kIndexInUse) return;
  for (uint32_t row = blockIdx.x * 256 + threadIdx.x; row < n; row += gridDim.x * 256) {
    const uint32_t s = ix.slot_of_row[row];
    int32_t c[W];
    load_row<W>(coords, row, c);
    BlockCoords<W> b;
    b.load(h, c);
    const unsigned long long below = (1ull << b.bit(b.local)) - 1ull;
    ix.perm[__ldg(&ix.slots[s].base) + (uint32_t)__popcll(~__ldg(&ix.slots[s].free) & below)] = (int32_t)row;
  }
}

// One thread per row, as in k_kmap_probe, in blocks that stay (one setup each, and few to launch where the index is not in
// use: 2450 -> 2324 us for the four clips). Offsets that reach further than two voxels (in units of the map's grid) along a
// block axis look their row up in the hash table instead. Where the blocks did not fit, the mirrored half of the table is
// filled with "no neighbour" for k_kmap_probe_self, which follows.
template <int W>
__global__ void __launch_bounds__(kKmapBlock, 6) k_kmap_blocks_self(
    const TableHeader* __restrict__ h, const Slot* __restrict__ slots, const int32_t* __restrict__ coords, uint32_t n,
    const int32_t* __restrict__ offsets, int K, int32_t* __restrict__ nbr, uint32_t* __restrict__ block_counts,
    uint32_t n_blocks, uint32_t* __restrict__ scan_ticket, BlockIndex ix) {
  after_previous_kernel();
  if (*ix.state != kIndexInUse) {
    if (*ix.state == kIndexFull)
      for (uint32_t row = blockIdx.x * kKmapBlock + threadIdx.x; row < n; row += gridDim.x * kKmapBlock)
        for (int k = K / 2 + 1; k < K; ++k) __stcs(nbr + (size_t)k * n + row, -1);
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *scan_ticket = 0;
  using B = BlockCoords<W>;
  constexpr int D = W - 1, NA = B::NA, CELLS = 1 << NA;
  constexpr uint32_t kNever = 1u << 28, kFar = 1u << 29, kNewOuter = 1u << 30;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* s_occ = reinterpret_cast<unsigned long long*>(smem_raw);  // [CELLS][256] masks around every row
  uint32_t* s_base = reinterpret_cast<uint32_t*>(s_occ + CELLS * kKmapBlock);   // [CELLS][256]
  uint32_t* s_off = s_base + CELLS * kKmapBlock;                                // [K] offset in nibbles modulo 8, flags
  uint32_t* s_cnt = s_off + K;                                                  // [half]
  __shared__ uint32_t s_reach[2 * NA];  // largest step down / up per block axis
  const int half = K / 2;
  if (threadIdx.x < 2 * NA) s_reach[threadIdx.x] = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += kKmapBlock) {
    uint32_t e = 0;
    int32_t step[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int32_t o = __ldg(offsets + k * D + a);
      const uint32_t s = h->low_shift(a);
      if (o & ((1 << s) - 1)) e |= kNever;  // off the map's grid
      step[a] = o >> s;
      if (step[a] < -2 || step[a] > 2) e |= kFar;
      e |= ((uint32_t)step[a] & 7u) << (4 * a);
    }
    bool new_outer = k == 0;
#pragma unroll
    for (int a = NA; a < D; ++a) new_outer |= k > 0 && __ldg(offsets + k * D + a) != __ldg(offsets + (k - 1) * D + a);
    if (new_outer) e |= kNewOuter;
    if (!(e & (kNever | kFar))) {
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        if (step[a] < 0) atomicMax(&s_reach[2 * a], (uint32_t)-step[a]);
        if (step[a] > 0) atomicMax(&s_reach[2 * a + 1], (uint32_t)step[a]);
      }
    }
    s_off[k] = e;
  }

  for (uint32_t row_block = blockIdx.x; row_block < n_blocks; row_block += gridDim.x) {
    __syncthreads();  // (the offsets are there, the counts of the block before are written)
    for (int k = threadIdx.x; k < half; k += kKmapBlock) s_cnt[k] = 0;
    __syncthreads();
    const uint32_t q = row_block * kKmapBlock + threadIdx.x;
    const bool active = q < n;
    const int lane = threadIdx.x & 31;
    int32_t c[W];
#pragma unroll
    for (int i = 0; i < W; ++i) c[i] = h->mn[i];
    if (active) load_row<W>(coords, q, c);
    B b;
    b.load(h, c);
    // per block axis: the neighbouring block on the side of the row's half of its block, if any offset reaches it
    long long side[NA];
    uint32_t reach = 0;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const uint32_t l = (b.local >> (4 * a)) & 3u;
      const uint32_t last = (((uint32_t)(h->mx[a + 1] - h->mn[a + 1])) >> h->low_shift(a)) >> 2;
      const bool up = l >= 2;
      if (up ? (l + s_reach[2 * a + 1] > 3 && b.block[a] < last) : (s_reach[2 * a] > l && b.block[a] > 0)) reach |= 1u << a;
      side[a] = (up ? 1ll : -1ll) * (1ll << h->shift[a + 1]);
    }
    unsigned long long* occ = s_occ + threadIdx.x;
    uint32_t* base = s_base + threadIdx.x;
    int32_t* dst = nbr + q;
    for (int k = 0; k < K; ++k, dst += n) {
      const uint32_t e = s_off[k];
      if (e & kNewOuter) {  // (same for the whole block) look up the blocks around the row
        unsigned long long key0 = b.key;
        bool in_box = active;
#pragma unroll
        for (int a = NA; a < D; ++a) {
          const int32_t o = __ldg(offsets + k * D + a);
          in_box = in_box && b.dist[a + 1] + (uint32_t)o <= (uint32_t)(h->mx[a + 1] - h->mn[a + 1]);
          key0 += (unsigned long long)((long long)o << h->shift[a + 1]);
        }
        constexpr int BATCH = CELLS < 4 ? CELLS : 4;  // independent lookups in flight
#pragma unroll
        for (int i0 = 0; i0 < CELLS; i0 += BATCH) {
          ulonglong2 v[BATCH];
          uint32_t at[BATCH];
#pragma unroll
          for (int j = 0; j < BATCH; ++j) {
            const int i = i0 + j;
            v[j] = make_ulonglong2(kEmptyKey, ~0ull);
            at[j] = 0;
            if (in_box && (i & ~reach) == 0) {
              unsigned long long key = key0;
#pragma unroll
              for (int a = 0; a < NA; ++a)
                if ((i >> a) & 1) key += (unsigned long long)side[a];
              at[j] = block_hash(key, ix.capacity);
              v[j] = __ldg(reinterpret_cast<const ulonglong2*>(ix.slots + at[j]));
            }
          }
#pragma unroll
          for (int j = 0; j < BATCH; ++j) {
            const int i = i0 + j;
            unsigned long long key = key0;
#pragma unroll
            for (int a = 0; a < NA; ++a)
              if ((i >> a) & 1) key += (unsigned long long)side[a];
            for (uint32_t probe = 1; v[j].x != key && v[j].x != kEmptyKey && probe < kBlockMaxProbes; ++probe) {
              if (++at[j] == ix.capacity) at[j] = 0;
              v[j] = __ldg(reinterpret_cast<const ulonglong2*>(ix.slots + at[j]));
            }
            const bool found = v[j].x == key;
            occ[i * kKmapBlock] = found ? ~v[j].y : 0ull;
            if (found) base[i * kKmapBlock] = __ldg(&ix.slots[at[j]].base);
          }
        }
      }
      uint32_t uid = 0xFFFFFFFFu;
      bool hit = false;
      if (!(e & (kNever | kFar))) {
        const uint32_t p = b.local + (e & 0xFFFu), bit = B::bit(p);
        // bits 2, 6 and 10: is the voxel in the row's own block or in the next one along the axis
        const uint32_t cell = ((((p & 0x444u) * 0x124u) >> 10) & 7u) * kKmapBlock;
        const unsigned long long m = occ[cell];
        hit = (m >> bit) & 1ull;
        if (hit) uid = (uint32_t)__ldg(ix.perm + base[cell] + __popcll(m & ((1ull << bit) - 1ull)));
      } else if (e & kFar && !(e & kNever)) {
        bool in_box = active;
        unsigned long long key = 0;
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const uint32_t d = b.dist[i] + (i > 0 ? (uint32_t)__ldg(offsets + k * D + i - 1) : 0u);
          in_box = in_box && d <= (uint32_t)(h->mx[i] - h->mn[i]);
          key |= (unsigned long long)d << h->shift[i];
        }
        if (in_box) uid = table_find(slots, h->capacity, h->pos_shift, key);
        hit = uid != 0xFFFFFFFFu;
      }
      if (active) __stcs(dst, (int32_t)uid);
      if (k < half) {  // (the other half has the same counts, see k_kmap_scan)
        const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
        if (lane == 0) atomicAdd(&s_cnt[k], (uint32_t)__popc(hits));
      }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < half; k += kKmapBlock) block_counts[(size_t)k * n_blocks + row_block] = s_cnt[k];
    if (threadIdx.x == 0)
      block_counts[(size_t)half * n_blocks + row_block] = min((uint32_t)kKmapBlock, n - row_block * kKmapBlock);
  }
}

// The map in the order of perm, block by block (rmn_kmap_build_ordered): position p is row perm[p], entries are row numbers,
// nothing is counted. The positions of a CUDA block lie in a dozen or two blocks of the index, so these are looked up with the
// 26 around them once for all their rows, a warp per block and a lane per cell; rows test bits in shared memory, and the row
// numbers that they read lie next to one another. What
// bounds it is issued instructions (55 % of the slots, 58 % of the load/store pipe) and the latency that four blocks an SM do not
// cover: 4.8 M clip rows x 81 offsets with the index 2250 us by k_kmap_blocks_self, 1700 by the same
// kernel walking perm, 1200 here (270 the index, 260 looking blocks up, 550 the rows, of them 160 the stores).
// Where the index is not in use perm becomes the identity, and k_kmap_probe_self follows.
constexpr int kOrderedCells = 27, kOrderedChunk = 32;  // blocks in shared memory at a time
struct OrderedHalf {  // half of a block's mask (32 voxels) and the position in perm of its first row
  uint32_t mask, base;
};
inline size_t ordered_smem(int K) { return (size_t)kOrderedChunk * kOrderedCells * 2 * sizeof(OrderedHalf) + (size_t)K * 4; }

template <int W>
__global__ void __launch_bounds__(kKmapBlock, 4) k_kmap_ordered(
    const TableHeader* __restrict__ h, const Slot* __restrict__ slots, const int32_t* __restrict__ coords, uint32_t n,
    const int32_t* __restrict__ offsets, int K, int32_t* __restrict__ nbr, BlockIndex ix) {
  after_previous_kernel();
  if (*ix.state != kIndexInUse) {
    for (uint32_t row = blockIdx.x * kKmapBlock + threadIdx.x; row < n; row += gridDim.x * kKmapBlock) {
      ix.perm[row] = (int32_t)row;
      if (*ix.state == kIndexFull)
        for (int k = K / 2 + 1; k < K; ++k) __stcs(nbr + (size_t)k * n + row, -1);
    }
    return;
  }
  using B = BlockCoords<W>;
  constexpr int D = W - 1, NA = B::NA;
  constexpr uint32_t kCube = 1u << 27, kNever = 1u << 28, kFar = 1u << 29, kNewOuter = 1u << 30;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  OrderedHalf* s_half = reinterpret_cast<OrderedHalf*>(smem_raw);                               // [chunk][cell][half]
  uint32_t* s_off = reinterpret_cast<uint32_t*>(s_half + kOrderedChunk * kOrderedCells * 2);  // [K] nibbles modulo 8, flags
  __shared__ unsigned long long s_key[kKmapBlock];  // of the blocks of this CUDA block, moved along the outer axes
  __shared__ uint8_t s_sides[kKmapBlock];           // bit 2 a (+ 1): the box goes on below (above) the block along axis a
  __shared__ uint32_t s_slot[kKmapBlock], s_heads[kKmapBlock / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int k = tid; k < K; k += kKmapBlock) {
    uint32_t e = 0;
    int32_t step[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int32_t o = __ldg(offsets + k * D + a);
      const uint32_t s = h->low_shift(a);
      if (o & ((1 << s) - 1)) e |= kNever;  // off the map's grid
      step[a] = o >> s;
      if (step[a] < -2 || step[a] > 2) e |= kFar;
      e |= ((uint32_t)step[a] & 7u) << (4 * a);
    }
    bool new_outer = k == 0;
#pragma unroll
    for (int a = NA; a < D; ++a) new_outer |= k > 0 && __ldg(offsets + k * D + a) != __ldg(offsets + (k - 1) * D + a);
    if (new_outer) e |= kNewOuter;
    bool cube = new_outer && k + kOrderedCells <= K;  // the 27 steps of -1, 0, 1, the first axis fastest
    for (int j = 0; cube && j < kOrderedCells; ++j)
      for (int a = 0, c = j; a < D; ++a, c /= 3)
        cube = cube && __ldg(offsets + (k + j) * D + a) == (a < NA ? (c % 3 - 1) * (1 << h->low_shift(a)) : __ldg(offsets + k * D + a));
    if (cube) e |= kCube;
    s_off[k] = e;
  }
  // this lane's cell: its distance in keys, and the sides of a block on which the box has to go on
  unsigned long long cell_step = 0;
  uint32_t cell_sides = 0;
#pragma unroll
  for (int a = 0, c = (int)lane; a < NA; ++a, c /= 3) {
    const int d = c % 3 - 1;
    cell_step += (unsigned long long)((long long)d * (1ll << h->shift[a + 1]));
    if (d) cell_sides |= 1u << (2 * a + (d > 0 ? 1 : 0));
  }
  const uint32_t n_blocks = (n + kKmapBlock - 1) / kKmapBlock;
  for (uint32_t row_block = blockIdx.x; row_block < n_blocks; row_block += gridDim.x) {
    const uint32_t q = row_block * kKmapBlock + tid;
    const bool active = q < n;
    const uint32_t row = active ? (uint32_t)__ldg(ix.perm + q) : 0u;
    int32_t c[W];
#pragma unroll
    for (int i = 0; i < W; ++i) c[i] = h->mn[i];
    if (active) load_row<W>(coords, row, c);
    B b;
    b.load(h, c);
    // number the blocks of these positions
    __syncthreads();  // (the lists of the positions before have been read)
    s_slot[tid] = active ? __ldg(ix.slot_of_row + row) : ~0u;
    __syncthreads();
    const bool head = active && (tid == 0 || s_slot[tid] != s_slot[tid - 1]);
    const uint32_t heads = __ballot_sync(0xFFFFFFFFu, head);
    if (lane == 0) s_heads[warp] = __popc(heads);
    __syncthreads();
    uint32_t mine = __popc(heads & ((2u << lane) - 1u)) - 1u, n_own = 0;
#pragma unroll
    for (uint32_t w = 0; w < kKmapBlock / 32; ++w) {
      if (w < warp) mine += s_heads[w];
      n_own += s_heads[w];
    }
    if (head) {
      uint32_t sides = 0;
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const uint32_t last = (((uint32_t)(h->mx[a + 1] - h->mn[a + 1])) >> h->low_shift(a)) >> 2;
        sides |= (b.block[a] > 0 ? 1u : 0u) << (2 * a) | (b.block[a] < last ? 2u : 0u) << (2 * a);
      }
      s_sides[mine] = (uint8_t)sides;
    }
    int32_t* dst = nbr + q;
    for (int k0 = 0, k1; k0 < K; k0 = k1) {  // the offsets that share their steps along the outer axes
      for (k1 = k0 + 1; k1 < K && !(s_off[k1] & kNewOuter);) ++k1;
      if (head) {
        unsigned long long key = b.key;
        bool in_box = true;
#pragma unroll
        for (int a = NA; a < D; ++a) {
          const int32_t o = __ldg(offsets + k0 * D + a);
          in_box = in_box && b.dist[a + 1] + (uint32_t)o <= (uint32_t)(h->mx[a + 1] - h->mn[a + 1]);
          key += (unsigned long long)((long long)o << h->shift[a + 1]);
        }
        s_key[mine] = in_box ? key : kEmptyKey;
      }
      for (uint32_t chunk = 0; chunk < n_own; chunk += kOrderedChunk) {
        __syncthreads();  // (the keys are there, the cells before have been read)
        constexpr uint32_t WARPS = kKmapBlock / 32;
        for (uint32_t j = warp; j < kOrderedChunk && chunk + j < n_own; j += 2 * WARPS) {  // two lookups in flight
          unsigned long long key[2];
          uint32_t at[2];
          ulonglong2 v[2];
#pragma unroll
          for (uint32_t i = 0; i < 2; ++i) {
            const uint32_t own = j + i * WARPS;
            const unsigned long long origin = own < kOrderedChunk && chunk + own < n_own ? s_key[chunk + own] : kEmptyKey;
            key[i] = origin + cell_step;
            at[i] = block_hash(key[i], ix.capacity);
            v[i] = make_ulonglong2(kEmptyKey, ~0ull);
            if (lane < kOrderedCells && origin != kEmptyKey && !(cell_sides & ~s_sides[chunk + own]))
              v[i] = __ldg(reinterpret_cast<const ulonglong2*>(ix.slots + at[i]));
          }
#pragma unroll
          for (uint32_t i = 0; i < 2; ++i) {
            const uint32_t own = j + i * WARPS;
            for (uint32_t probe = 1; v[i].x != key[i] && v[i].x != kEmptyKey && probe < kBlockMaxProbes; ++probe) {
              if (++at[i] == ix.capacity) at[i] = 0;
              v[i] = __ldg(reinterpret_cast<const ulonglong2*>(ix.slots + at[i]));
            }
            const bool found = v[i].x == key[i];
            const uint32_t lo = found ? (uint32_t)~v[i].y : 0u, hi = found ? (uint32_t)(~v[i].y >> 32) : 0u;
            const uint32_t base = found ? __ldg(&ix.slots[at[i]].base) : 0u;
            if (lane < kOrderedCells && own < kOrderedChunk)
              *reinterpret_cast<uint4*>(s_half + (own * kOrderedCells + lane) * 2) = make_uint4(lo, base, hi, base + __popc(lo));
          }
        }
        __syncthreads();
        if (!active || mine - chunk >= (uint32_t)kOrderedChunk) continue;
        const OrderedHalf* half_of = s_half + (mine - chunk) * kOrderedCells * 2;
        // cell beside the block along an axis, from the nibble of a position: 0..3 the block itself, 4, 5 above, 6, 7 below
        auto beside = [](uint32_t nibble) { return nibble & 4u ? (nibble & 2u ? 0u : 2u) : 1u; };
        int32_t* out = dst + (size_t)k0 * n;
        int k = k0;
        if (s_off[k0] & kCube) {
          // Steps -1, 0, 1 along the first axis are neighbouring bits of a row of four, whose ranks differ by the bits between
          // them, and at the block's edge one bit of the block beside it.
          const uint32_t x = b.local & 3u, edge_x = x ? 0u : 3u;
          const int edge_cell = x < 2u ? -2 : 2;
          uint32_t cell_y[3], shift_y[3];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const uint32_t y = (((b.local >> 4) & 3u) + (uint32_t)i - 1u) & 7u;
            cell_y[i] = beside(y) * 6u;
            shift_y[i] = 4u * (y & 3u);
          }
#pragma unroll
          for (int iz = 0; iz < 3; ++iz) {
            const uint32_t z = (((b.local >> 8) & 3u) + (uint32_t)iz - 1u) & 7u;
            const OrderedHalf* plane = half_of + beside(z) * 18u + 2u + ((z >> 1) & 1u);
            const uint32_t shift_z = 16u * (z & 1u);
#pragma unroll
            for (int iy = 0; iy < 3; ++iy) {
              const OrderedHalf* cell = plane + cell_y[iy];
              const uint2 own = *reinterpret_cast<const uint2*>(cell), edge = *reinterpret_cast<const uint2*>(cell + edge_cell);
              const uint32_t shift = shift_y[iy] + shift_z, at = shift + x, edge_at = shift + edge_x;
              const uint32_t edge_bit = (edge.x >> edge_at) & 1u;
              const uint32_t window = ((own.x >> shift) & 15u) << 1 | (x == 0u ? edge_bit : 0u) | (x == 3u ? edge_bit << 5 : 0u);
              const uint32_t hits = window >> x;
              const uint32_t centre = own.y + __popc(own.x & ((1u << at) - 1u));
              const uint32_t other = edge.y + __popc(edge.x & ((1u << edge_at) - 1u));
              int32_t v[3] = {-1, -1, -1};
              if (hits & 1u) v[0] = __ldg(ix.perm + (x ? centre - 1u : other));
              if (hits & 2u) v[1] = __ldg(ix.perm + centre);
              if (hits & 4u) v[2] = __ldg(ix.perm + (x < 3u ? centre + ((hits >> 1) & 1u) : other));
#pragma unroll
              for (int i = 0; i < 3; ++i, out += n) __stcs(out, v[i]);
            }
          }
          k += kOrderedCells;
        }
        for (; k < k1; ++k, out += n) {
          const uint32_t e = s_off[k];
          uint32_t uid = 0xFFFFFFFFu;
          if (!(e & (kNever | kFar))) {
            const uint32_t p = b.local + (e & 0xFFFu), bit = B::bit(p);
            const uint32_t cell = 9 * beside((p >> 8) & 7u) + 3 * beside((p >> 4) & 7u) + beside(p & 7u);
            const OrderedHalf m = half_of[cell * 2 + (bit >> 5)];
            if ((m.mask >> (bit & 31u)) & 1u) uid = (uint32_t)__ldg(ix.perm + m.base + __popc(m.mask & ((1u << (bit & 31u)) - 1u)));
          } else if (!(e & kNever)) {
            bool in_box = true;
            unsigned long long key = 0;
#pragma unroll
            for (int i = 0; i < W; ++i) {
              const uint32_t d = b.dist[i] + (i > 0 ? (uint32_t)__ldg(offsets + k * D + i - 1) : 0u);
              in_box = in_box && d <= (uint32_t)(h->mx[i] - h->mn[i]);
              key |= (unsigned long long)d << h->shift[i];
            }
            if (in_box) uid = table_find(slots, h->capacity, h->pos_shift, key);
          }
          __stcs(out, (int32_t)uid);
        }
      }
    }
  }
}

}  // namespace rmn
