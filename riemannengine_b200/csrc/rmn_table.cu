// Coordinate hash table: dedup insert with first-occurrence numbering, lookup,
// stride alignment. Integer work bound by HBM/L2 bandwidth.
//
// Build pipeline (all on the caller's stream, no host synchronisation):
//   header cleared
//   -> fill + range (slots to the empty pattern, column min/max; the last block plans the bit packing)
//   -> insert (one 16-byte CAS on the packed key, atomicMin on the first row; marks and counts the repeated rows)
//   -> finalize (number of unique rows, stored into the host's memory first where the caller waits for it; unique ids, mapping,
//      unique coordinates; identity inverse when nothing was a duplicate)
//   -> inverse (only does work when there were duplicates)
// Up to kSmallRows rows one block does all of it in one launch.
// Numbering unique rows by first occurrence reproduces the reference CPU map
// (engine/grid/lattice_cpu.hpp:419-444) deterministically; the reference GPU
// map lets a CAS race pick the surviving duplicate
// (engine/grid/lattice_gpu.cu:30-51).
#include "rmn_common.cuh"

#include <cuda_bf16.h>

#include <limits.h>
#include <string.h>
#include <stddef.h>

#include <atomic>
#include <mutex>

namespace rmn {

int tc_copy_status_async(uint32_t* host_dst, cudaStream_t stream);  // rmn_conv_tc.cu
int tc_clear_status();
const uint32_t* tc_status_device_address();

constexpr int kRowsPerBlock = 256;
constexpr uint32_t kGrid = 148 * 8;  // blocks of the passes that may have nothing to do

// Scratch of a build of n rows: slot of every row, one bit per row that is not the first of its key, and how many of these
// every kSuperBlocks blocks of 256 rows hold (with them and the bits of its own super-block a block of k_finalize numbers its
// rows without a scan: 5 to 8 us less than a pass that counts and scans)
struct Scratch {
  uint32_t* slot_of_row;
  uint32_t* super_repeats;
  uint32_t* repeat_bits;
};
constexpr uint32_t kSuperBlocks = 64, kSuperRows = kSuperBlocks * kRowsPerBlock;
// Counted by k_insert, or where many duplicates are expected by k_super_repeats from the bits: there the atomics would serialise
// (1.2 M rows on 0.27 M strided cells: insert 33 us without them, 60 with sixteen counters per super-block, 80 with one).
constexpr size_t super_words(size_t n) { return ((n + kSuperRows - 1) / kSuperRows + 3) / 4 * 4; }
constexpr size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }
constexpr size_t scratch_bytes(size_t n) {
  const size_t nb = (n + kRowsPerBlock - 1) / kRowsPerBlock;
  return align16(n * 4) + super_words(n) * 4 + nb * (kRowsPerBlock / 8) + 256;
}
inline Scratch scratch(void* workspace, uint32_t n) {
  char* p = reinterpret_cast<char*>(((uintptr_t)workspace + 15) & ~(uintptr_t)15);
  Scratch s;
  s.slot_of_row = reinterpret_cast<uint32_t*>(p);
  s.super_repeats = reinterpret_cast<uint32_t*>(p + align16((size_t)n * 4));
  s.repeat_bits = s.super_repeats + super_words(n);
  return s;
}

// Words that a build stores into page-locked host memory for a host that polls: rmn_table_info's four, the convolution
// kernels' status word and, last, the number of this build.
struct HostPost {
  volatile uint32_t* words;  // NULL: nobody waits
  const uint32_t* conv_status;
  uint32_t sequence;

  __device__ void store(const TableHeader* h, uint32_t n_unique) const {
    if (!words) return;
    words[0] = n_unique;
    words[1] = *(const volatile uint32_t*)&h->status;
    words[2] = h->capacity;
    words[3] = h->n_rows;
    words[4] = conv_status ? *conv_status : 0u;
    __threadfence_system();
    words[5] = sequence;
  }
};

__device__ void plan_packing(TableHeader* h);

// One thread: the header's constants, the decoded column bounds and the key packing.
__device__ void write_header(TableHeader* h, uint32_t W, uint32_t n, uint32_t capacity) {
  h->magic = kTableMagic;
  h->W = W;
  h->n_rows = n;
  h->capacity = capacity;
  for (uint32_t c = 0; c < RMN_MAX_W; ++c) {
    const uint32_t en = *(volatile uint32_t*)&h->mn_enc[c], ex = *(volatile uint32_t*)&h->mx_enc[c];
    h->mn[c] = (c < W && n > 0) ? (int32_t)(~en ^ 0x80000000u) : 0;
    h->mx[c] = (c < W && n > 0) ? (int32_t)(ex ^ 0x80000000u) : 0;
    h->bits[c] = 0;
    h->shift[c] = 0;
  }
  const uint32_t o = *(volatile uint32_t*)&h->x_or;
  h->pos_shift = o ? (uint32_t)(__ffs((int)o) - 1) : 0u;
  plan_packing(h);
}

// (a launch that overlaps its neighbours, where a memset would not)
__global__ void __launch_bounds__(64) k_clear_header(uint32_t* __restrict__ words) {
  after_previous_kernel();
  words[threadIdx.x] = 0u;
}

// First pass of a build, on a cleared header: fills the slots with the empty
// pattern (all ones) and reduces the column bounds of the rows in the same pass (the fill writes, the
// reduction reads: one launch moves both at HBM speed). The last block to finish writes the header's
// constants, decodes the bounds and plans the key packing.
template <int W>
__global__ void __launch_bounds__(256) k_fill_range(const int32_t* __restrict__ coords, uint32_t n,
                                                    TableHeader* h, uint4* __restrict__ slots, uint32_t capacity, Scratch sc) {
  after_previous_kernel();
  __shared__ int32_t s_mn[8][W], s_mx[8][W];
  constexpr int NA = W - 1 < 3 ? W - 1 : 3;
  __shared__ uint32_t s_or[8][NA];
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < capacity; i += gridDim.x * blockDim.x)
    slots[i] = ones;
  const uint32_t bit_words = (n + kRowsPerBlock - 1) / kRowsPerBlock * (kRowsPerBlock / 32);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < bit_words; i += gridDim.x * blockDim.x) sc.repeat_bits[i] = 0u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < super_words(n); i += gridDim.x * blockDim.x) sc.super_repeats[i] = 0u;
  int32_t mn[W], mx[W];
#pragma unroll
  for (int c = 0; c < W; ++c) { mn[c] = INT_MAX; mx[c] = INT_MIN; }
  // OR of (x - x of row 0) over the rows: its trailing zeros are the bits of a spatial column that all rows share
  uint32_t first[NA], col_or[NA];
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    first[a] = n > 0 ? (uint32_t)__ldg(coords + 1 + a) : 0u;
    col_or[a] = 0;
  }
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    int32_t v[W];
    load_row<W>(coords, r, v);
#pragma unroll
    for (int c = 0; c < W; ++c) { mn[c] = min(mn[c], v[c]); mx[c] = max(mx[c], v[c]); }
#pragma unroll
    for (int a = 0; a < NA; ++a) col_or[a] |= (uint32_t)v[1 + a] - first[a];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < W; ++c) {
    const int32_t a = __reduce_min_sync(0xFFFFFFFFu, mn[c]);
    const int32_t b = __reduce_max_sync(0xFFFFFFFFu, mx[c]);
    if (lane == 0) { s_mn[warp][c] = a; s_mx[warp][c] = b; }
  }
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const uint32_t o = __reduce_or_sync(0xFFFFFFFFu, col_or[a]);
    if (lane == 0) s_or[warp][a] = o;
  }
  __syncthreads();
  // one atomic per block and column (per-warp atomics on eight addresses serialise badly); blocks that
  // saw no row leave the zero ("no row yet") in place
  if (threadIdx.x < W && blockIdx.x * blockDim.x < n) {
    int32_t a = s_mn[0][threadIdx.x], b = s_mx[0][threadIdx.x];
#pragma unroll
    for (int w2 = 1; w2 < 8; ++w2) { a = min(a, s_mn[w2][threadIdx.x]); b = max(b, s_mx[w2][threadIdx.x]); }
    atomicMax(&h->mn_enc[threadIdx.x], ~((uint32_t)a ^ 0x80000000u));
    atomicMax(&h->mx_enc[threadIdx.x], (uint32_t)b ^ 0x80000000u);
  }
  if (threadIdx.x >= 32 && threadIdx.x < 32 + NA && blockIdx.x * blockDim.x < n) {
    const int a = (int)threadIdx.x - 32;
    uint32_t o = 0;
#pragma unroll
    for (int w2 = 0; w2 < 8; ++w2) o |= s_or[w2][a];
    if (o) atomicOr(a == 0 ? &h->x_or : &h->yz_or[a - 1], o);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&h->range_blocks_done, 1u) == gridDim.x - 1) {
    __threadfence();
    write_header(h, W, n, capacity);
  }
}

// One thread: bit widths and shifts of the packed key from the bounding box in the header.
__device__ void plan_packing(TableHeader* h) {
  uint32_t total = 0;
  // packing order: spatial columns first (column 1 in the lowest bits: its low three bits pick
  // the position inside a bucket), the batch column last
  for (uint32_t i = 0; i < h->W; ++i) {
    const uint32_t c = i + 1 < h->W ? i + 1 : 0;
    uint32_t b = 0;
    if (h->n_rows > 0) {
      const uint32_t span = (uint32_t)h->mx[c] - (uint32_t)h->mn[c];
      b = span == 0 ? 0 : 32 - __clz(span);
    }  // empty table: bounds are zero and every probe ends on a free slot
    h->bits[c] = b;
    h->shift[c] = total > 63 ? 63 : total;
    total += b;
  }
  h->total_bits = total;
  if (total > 63) h->status = RMN_ERR_RANGE;
}

// 16-byte atomic compare-and-swap of a whole slot against the empty pattern (all ones); returns
// the slot's previous content.
__device__ __forceinline__ void cas_slot(Slot* slot, unsigned long long key, unsigned long long rows,
                                         unsigned long long& old_key, unsigned long long& old_rows) {
  asm volatile(
      "{\n\t.reg .b128 c, d, o;\n\t"
      "mov.b128 c, {%2, %2};\n\t"
      "mov.b128 d, {%3, %4};\n\t"
      "atom.relaxed.gpu.global.cas.b128 o, [%5], c, d;\n\t"
      "mov.b128 {%0, %1}, o;\n\t}"
      : "=l"(old_key), "=l"(old_rows)
      : "l"(~0ull), "l"(key), "l"(rows), "l"(slot)
      : "memory");
}

constexpr uint32_t kNoRow = 0xFFFFFFFFu;

// Claims the slot of a row's key: {key, first_row = row, uid = row}. Without duplicates the unique numbering is the row
// numbering and the slot is final after this single 16-byte compare-and-swap. A row that finds its key taken lowers
// first_row; the larger of the two rows is not the first of its key and goes to *repeat (every row but the smallest loses
// once; kNoRow: none did). look_first: read a slot before the compare-and-swap and spare it, and
// the atomic minimum, where the key is there already with a smaller row - the usual case among many duplicates (1.2 M rows
// on 0.27 M strided cells: 60 -> 25 us), a second round trip to the slot without them.
__device__ __forceinline__ bool insert_row(Slot* slots, uint32_t capacity, uint32_t pos_shift, unsigned long long key,
                                           uint32_t row, bool look_first, uint32_t* slot_of_row, uint32_t* repeat) {
  uint32_t s = hash_key(key, capacity, pos_shift);
  const unsigned long long mine = (unsigned long long)row | ((unsigned long long)row << 32);
  for (uint32_t probe = 0; probe < (capacity >> 3); ++probe) {
    unsigned long long cur_key = kEmptyKey, cur_rows = ~0ull;
    if (look_first) {
      const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(slots + s));
      cur_key = v.x;
      cur_rows = v.y;
    }
    if (cur_key == kEmptyKey) {
      cas_slot(&slots[s], key, mine, cur_key, cur_rows);
    }
    if (cur_key == kEmptyKey || cur_key == key) {
      if (cur_key == key) {
        uint32_t other = (uint32_t)cur_rows;
        if (other > row) other = atomicMin(&slots[s].first_row, row);
        *repeat = other > row ? other : row;
      }
      slot_of_row[row] = s;
      return true;
    }
    // another key lives here and this one walks on: leave word for the lookups (kPassedBit)
    // (all ones: the key has been seen before its rows)
    if (cur_rows == ~0ull || !((uint32_t)(cur_rows >> 32) & kPassedBit)) atomicOr(&slots[s].uid, kPassedBit);
    s = next_slot(s, capacity);
  }
  return false;
}

template <int W>
__global__ void __launch_bounds__(256) k_insert(const int32_t* __restrict__ coords, uint32_t n,
                                                TableHeader* h, Slot* slots,
                                                Scratch sc, int look_first) {
  after_previous_kernel();
  if (h->status != RMN_OK) return;
  const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t repeat = kNoRow;
  if (row < n) {
    Packer<W> pk;
    pk.load(h);
    int32_t c[W];
    load_row<W>(coords, row, c);
    unsigned long long key;
    pk.pack(c, key);
    if (!insert_row(slots, h->capacity, h->pos_shift, key, row, look_first != 0, sc.slot_of_row, &repeat))
      atomicExch(&h->status, (uint32_t)RMN_ERR_PROBE_LIMIT);
  }
  const uint32_t own = __ballot_sync(0xFFFFFFFFu, repeat == row);  // (rows of a warp share a word)
  if ((threadIdx.x & 31) == 0 && own) atomicOr(sc.repeat_bits + (row >> 5), own);
  if (repeat != kNoRow && repeat != row) {
    atomicOr(sc.repeat_bits + (repeat >> 5), 1u << (repeat & 31));
    if (!look_first) atomicAdd(sc.super_repeats + repeat / kSuperRows, 1u);
  }
  // one atomic per block: the rows' own would serialise on the words
  const int dups = __syncthreads_count(repeat != kNoRow);
  const int dups_here = dups && !look_first ? __syncthreads_count(repeat == row) : 0;
  if (threadIdx.x == 0) {
    if (dups_here) atomicAdd(sc.super_repeats + blockIdx.x / kSuperBlocks, (uint32_t)dups_here);
    if (dups) atomicAdd(&h->n_dups, (uint32_t)dups);
  }
}

__global__ void __launch_bounds__(256) k_super_repeats(uint32_t n, const TableHeader* __restrict__ h, Scratch sc) {
  after_previous_kernel();
  if (h->status != RMN_OK || h->n_dups == 0) return;
  const uint32_t words = (n + kRowsPerBlock - 1) / kRowsPerBlock * (kRowsPerBlock / 32);
  const uint32_t super = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  uint32_t count = 0;
#pragma unroll
  for (uint32_t i = 0; i < kSuperRows / 32; i += 32) {
    const uint32_t at = super * (kSuperRows / 32) + i + lane;
    if (at < words) count += __popc(__ldg(sc.repeat_bits + at));
  }
  count = __reduce_add_sync(0xFFFFFFFFu, count);
  if (lane == 0 && super * (kSuperRows / 32) < words) sc.super_repeats[super] = count;
}

// (one thread, behind k_insert) the number of unique rows: every row but the first of its key has lost once
__device__ __forceinline__ void publish_unique(TableHeader* h, uint32_t n, const HostPost& post) {
  const bool ok = h->status == RMN_OK;
  const uint32_t n_unique = ok ? n - h->n_dups : 0u;
  if (ok) h->n_unique = n_unique;
  post.store(h, n_unique);
}
__global__ void k_publish_unique(uint32_t n, TableHeader* h) {
  after_previous_kernel();
  publish_unique(h, n, HostPost{});
}

template <int W>
__global__ void __launch_bounds__(kRowsPerBlock) k_finalize(
    const int32_t* __restrict__ coords, uint32_t n, TableHeader* h, Slot* slots,
    Scratch sc, int64_t* __restrict__ mapping, int32_t* __restrict__ unique_coords, int64_t* __restrict__ inverse,
    HostPost post) {
  after_previous_kernel();
  if (blockIdx.x == 0 && threadIdx.x == 0) publish_unique(h, n, post);
  if (h->status != RMN_OK) return;
  const uint32_t row = blockIdx.x * kRowsPerBlock + threadIdx.x;
  if (h->n_dups == 0) {
    // Fast path (all rows distinct): unique row == input row, already stored in the slots by
    // k_insert; only the identity mapping and the coordinate copy remain (both streaming).
    if (row < n) {
      if (mapping) mapping[row] = (int64_t)row;
      if (inverse) inverse[row] = (int64_t)row;
      if (unique_coords) {
        int32_t c[W];
        load_row<W>(coords, row, c);
#pragma unroll
        for (int i = 0; i < W; ++i) unique_coords[(size_t)row * W + i] = c[i];
      }
    }
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // repeated rows before this block
  __shared__ uint32_t s_before[kRowsPerBlock / 32];
  uint32_t before = 0;
  const uint32_t super = blockIdx.x / kSuperBlocks;
  for (uint32_t i = threadIdx.x; i < super; i += kRowsPerBlock) before += __ldg(sc.super_repeats + i);
  for (uint32_t i = super * (kSuperRows / 32) + threadIdx.x; i < blockIdx.x * (kRowsPerBlock / 32); i += kRowsPerBlock)
    before += __popc(__ldg(sc.repeat_bits + i));
  before = __reduce_add_sync(0xFFFFFFFFu, before);
  if (lane == 0) s_before[warp] = before;
  __syncthreads();
  if (row >= n) return;
  before = 0;
#pragma unroll
  for (int w = 0; w < kRowsPerBlock / 32; ++w) before += s_before[w];
  const uint32_t* bits = sc.repeat_bits + blockIdx.x * (kRowsPerBlock / 32);
  if ((__ldg(bits + warp) >> lane) & 1u) return;
  uint32_t uid = blockIdx.x * kRowsPerBlock - before + __popc(~__ldg(bits + warp) & ((1u << lane) - 1u));
  for (int w = 0; w < warp; ++w) uid += __popc(~__ldg(bits + w));
  const uint32_t s = sc.slot_of_row[row];
  slots[s].uid = uid | (slots[s].uid & kPassedBit);
  if (mapping) mapping[uid] = (int64_t)row;
  if (unique_coords) {
    int32_t c[W];
    load_row<W>(coords, row, c);
#pragma unroll
    for (int i = 0; i < W; ++i) unique_coords[(size_t)uid * W + i] = c[i];
  }
}

__global__ void __launch_bounds__(256) k_inverse(const Slot* __restrict__ slots,
                                                 const uint32_t* __restrict__ slot_of_row,
                                                 uint32_t n, const TableHeader* h,
                                                 int64_t* __restrict__ inverse) {
  after_previous_kernel();
  // without duplicates k_finalize has already written the identity
  if (h->n_dups == 0 || h->status != RMN_OK) return;
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < n; row += gridDim.x * blockDim.x)
    inverse[row] = (int64_t)(slots[slot_of_row[row]].uid & ~kPassedBit);
}

// The whole build of a small table by one block: what a chain of six launches costs there is the launches (900 rows:
// 20 us with their gaps).
constexpr uint32_t kSmallRows = 2048;
template <int W>
__global__ void __launch_bounds__(1024) k_build_small(const int32_t* __restrict__ coords, uint32_t n, TableHeader* h,
                                                      Slot* slots, uint32_t capacity, Scratch sc,
                                                      int64_t* __restrict__ mapping, int32_t* __restrict__ unique_coords,
                                                      int64_t* __restrict__ inverse, int look_first, HostPost post) {
  after_previous_kernel();
  constexpr int NA = W - 1 < 3 ? W - 1 : 3;
  __shared__ TableHeader s_h;
  __shared__ uint32_t s_ok;
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (tid < sizeof(TableHeader) / 4) reinterpret_cast<uint32_t*>(&s_h)[tid] = 0u;
  if (tid == 0) s_ok = 1u;
  const uint4 ones = make_uint4(~0u, ~0u, ~0u, ~0u);
  for (uint32_t i = tid; i < capacity; i += 1024) reinterpret_cast<uint4*>(slots)[i] = ones;
  int32_t row_c[2][W];
  int32_t mn[W], mx[W];
  uint32_t first[NA], col_or[NA];
#pragma unroll
  for (int c = 0; c < W; ++c) { mn[c] = INT_MAX; mx[c] = INT_MIN; }
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    first[a] = (uint32_t)__ldg(coords + 1 + a);
    col_or[a] = 0;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t row = tid + i * 1024;
    if (row >= n) continue;
    load_row<W>(coords, row, row_c[i]);
#pragma unroll
    for (int c = 0; c < W; ++c) { mn[c] = min(mn[c], row_c[i][c]); mx[c] = max(mx[c], row_c[i][c]); }
#pragma unroll
    for (int a = 0; a < NA; ++a) col_or[a] |= (uint32_t)row_c[i][1 + a] - first[a];
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < W; ++c) {
    const int32_t a = __reduce_min_sync(0xFFFFFFFFu, mn[c]), b = __reduce_max_sync(0xFFFFFFFFu, mx[c]);
    if (lane == 0 && a <= b) {
      atomicMax(&s_h.mn_enc[c], ~((uint32_t)a ^ 0x80000000u));
      atomicMax(&s_h.mx_enc[c], (uint32_t)b ^ 0x80000000u);
    }
  }
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const uint32_t o = __reduce_or_sync(0xFFFFFFFFu, col_or[a]);
    if (lane == 0 && o) atomicOr(a == 0 ? &s_h.x_or : &s_h.yz_or[a - 1], o);
  }
  __syncthreads();
  if (tid == 0) write_header(&s_h, W, n, capacity);
  __syncthreads();
  const bool range_ok = s_h.status == RMN_OK;
  uint32_t dups = 0;
  if (range_ok) {
    Packer<W> pk;
    pk.load(&s_h);
    uint32_t repeat[2] = {kNoRow, kNoRow};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t row = tid + i * 1024;
      if (row >= n) continue;
      unsigned long long key;
      pk.pack(row_c[i], key);
      if (!insert_row(slots, capacity, s_h.pos_shift, key, row, look_first != 0, sc.slot_of_row, &repeat[i])) s_ok = 0u;
    }
    dups = (uint32_t)(__syncthreads_count(repeat[0] != kNoRow) + __syncthreads_count(repeat[1] != kNoRow));
    if (tid == 0) {
      s_h.n_dups = dups;
      if (!s_ok) s_h.status = RMN_ERR_PROBE_LIMIT;
    }
    __syncthreads();
  }
  const bool ok = range_ok && s_h.status == RMN_OK;
  if (ok && dups == 0) {
    if (tid == 0) s_h.n_unique = n;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t row = tid + i * 1024;
      if (row >= n) continue;
      if (mapping) mapping[row] = (int64_t)row;
      if (inverse) inverse[row] = (int64_t)row;
      if (unique_coords) {
#pragma unroll
        for (int c = 0; c < W; ++c) unique_coords[(size_t)row * W + c] = row_c[i][c];
      }
    }
  } else if (ok) {
    __shared__ uint32_t s_warp[33];
    uint32_t carry = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t row = tid + i * 1024;
      const uint32_t s = row < n ? sc.slot_of_row[row] : 0u;
      const bool is_first = row < n && __ldcg(&slots[s].first_row) == row;
      const uint32_t bits = __ballot_sync(0xFFFFFFFFu, is_first);
      if (lane == 0) s_warp[tid >> 5] = (uint32_t)__popc(bits);
      __syncthreads();
      uint32_t before = carry, total = 0;
      for (uint32_t w = 0; w < 32; ++w) {
        if (w < (tid >> 5)) before += s_warp[w];
        total += s_warp[w];
      }
      carry += total;
      if (is_first) {
        const uint32_t uid = before + __popc(bits & ((1u << lane) - 1u));
        slots[s].uid = uid | (__ldcg(&slots[s].uid) & kPassedBit);
        if (mapping) mapping[uid] = (int64_t)row;
        if (unique_coords) {
#pragma unroll
          for (int c = 0; c < W; ++c) unique_coords[(size_t)uid * W + c] = row_c[i][c];
        }
      }
      __syncthreads();
    }
    if (tid == 0) s_h.n_unique = carry;
    if (inverse)
      for (uint32_t row = tid; row < n; row += 1024)
        inverse[row] = (int64_t)(__ldcg(&slots[sc.slot_of_row[row]].uid) & ~kPassedBit);
  }
  __syncthreads();
  if (tid < sizeof(TableHeader) / 4) reinterpret_cast<uint32_t*>(h)[tid] = reinterpret_cast<const uint32_t*>(&s_h)[tid];
  if (tid == 0) post.store(&s_h, s_h.n_unique);
}

template <int W>
__global__ void __launch_bounds__(256) k_find(const TableHeader* __restrict__ h,
                                              const Slot* __restrict__ slots,
                                              const int32_t* __restrict__ query, uint32_t n,
                                              int32_t* __restrict__ rows) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  Packer<W> pk;
  pk.load(h);
  const uint32_t capacity = h->capacity;
  int32_t c[W];
  load_row<W>(query, q, c);
  unsigned long long key;
  uint32_t uid = 0xFFFFFFFFu;
  if (pk.pack(c, key)) uid = table_find(slots, capacity, h->pos_shift, key);
  rows[q] = (int32_t)uid;
}

struct StrideArg {
  int32_t s[RMN_MAX_W];
};

// floor(c / s) * s; s == 1 and powers of two without a division
__device__ __forceinline__ int32_t floor_to(int32_t c, int32_t s) {
  if ((s & (s - 1)) == 0) return c & -s;
  int32_t q = c / s;
  if (c < 0 && q * s != c) --q;  // floor for negative coordinates
  return q * s;
}

// One thread per row (1.2 M rows of four columns: 24 -> 8 us against one thread per element with a 64-bit remainder).
// kVec: rows of four columns as one 16-byte access (aligned pointers).
template <int W, bool kVec>
__global__ void __launch_bounds__(256) k_stride(const int32_t* __restrict__ coords, uint32_t n, StrideArg st,
                                                int32_t* __restrict__ out) {
  after_previous_kernel();
  const uint32_t row = blockIdx.x * 256 + threadIdx.x;
  if (row >= n) return;
  int32_t c[W];
  if constexpr (kVec) {
    load_row<W>(coords, row, c);
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) c[i] = __ldg(coords + (size_t)row * W + i);
  }
#pragma unroll
  for (int i = 1; i < W; ++i) c[i] = floor_to(c[i], st.s[i - 1]);
  store_row<W, kVec>(out, row, c);
}

// Sum or mean of the rows of every voxel: the first row of a voxel is copied, the others - few, in a lidar sweep - are
// added to it (atomics), and only voxels of several rows are divided. (960 K points, 4 channels: 57 us by zero fills, two
// index_add, a ones tensor, a clamp and a division.)
__global__ void __launch_bounds__(256) k_segment_first(const float* __restrict__ feats, const int64_t* __restrict__ mapping,
                                                       uint32_t m, int C, float* __restrict__ out, uint32_t* __restrict__ count) {
  after_previous_kernel();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (size_t)m * C) return;
  const size_t u = i / C, c = i - u * C;
  out[i] = __ldg(feats + (size_t)__ldg(mapping + u) * C + c);
  if (c == 0) count[u] = 1u;
}
__global__ void __launch_bounds__(256) k_segment_first4(const float4* __restrict__ feats, const int64_t* __restrict__ mapping,
                                                        uint32_t m, float4* __restrict__ out, uint32_t* __restrict__ count) {
  after_previous_kernel();
  const uint32_t u = blockIdx.x * 256 + threadIdx.x;
  if (u >= m) return;
  out[u] = __ldg(feats + __ldg(mapping + u));
  count[u] = 1u;
}
__global__ void __launch_bounds__(256) k_segment_add(const float* __restrict__ feats, const int64_t* __restrict__ inverse,
                                                     const int64_t* __restrict__ mapping, uint32_t n, int C,
                                                     float* __restrict__ out, uint32_t* __restrict__ count) {
  after_previous_kernel();
  const uint32_t row = blockIdx.x * 256 + threadIdx.x;
  if (row >= n) return;
  const size_t u = (size_t)__ldg(inverse + row);
  if ((uint32_t)__ldg(mapping + u) == row) return;
  for (int c = 0; c < C; ++c) atomicAdd(out + u * C + c, __ldg(feats + (size_t)row * C + c));
  atomicAdd(count + u, 1u);
}
__global__ void __launch_bounds__(256) k_segment_divide(uint32_t m, int C, const uint32_t* __restrict__ count,
                                                        float* __restrict__ out) {
  after_previous_kernel();
  const uint32_t u = blockIdx.x * 256 + threadIdx.x;
  if (u >= m) return;
  const uint32_t k = __ldg(count + u);
  if (k > 1u)
    for (int c = 0; c < C; ++c) out[(size_t)u * C + c] = __fdiv_rn(out[(size_t)u * C + c], (float)k);
}

// Continuous (field) coordinates -> integer voxel coordinates, the reference's rule in float32:
// batch column lroundf(v), spatial column j: stride_j * (int)floor(v / stride_j)
// (engine/grid/lattice_cpu.hpp:944-984, engine/grid/lattice_gpu.cu:78-151). One thread per row, streaming.
template <int W, bool kVec>
__global__ void __launch_bounds__(256) k_field_quantize(const float* __restrict__ field, uint32_t n, StrideArg st,
                                                        int32_t* __restrict__ out) {
  after_previous_kernel();
  const uint32_t row = blockIdx.x * 256 + threadIdx.x;
  if (row >= n) return;
  float v[W];
  if constexpr (kVec) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(field) + row);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) v[i] = __ldg(field + (size_t)row * W + i);
  }
  int32_t c[W];
  c[0] = (int32_t)lroundf(v[0]);
#pragma unroll
  for (int i = 1; i < W; ++i) {
    const int32_t s = st.s[i - 1];
    c[i] = s == 1 ? (int32_t)floorf(v[i]) : s * (int32_t)floorf(__fdiv_rn(v[i], (float)s));
  }
  store_row<W, kVec>(out, row, c);
}

// out = (int32)floor((double)v / q) on EVERY column (q <= 0: floor only): the discretisation step of
// sparse_quantize (engine/helpers/discretization.cpp:97-102), computed in float64 as there.
template <typename T>
__global__ void __launch_bounds__(256) k_discretize(const T* __restrict__ in, uint64_t total, double q,
                                                    int32_t* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  double v = (double)in[i];
  if (q > 0.0) v = __ddiv_rn(v, q);
  out[i] = (int32_t)floor(v);
}

// Multilinear splat of a field onto the 2^D lattice corners around every point
// (engine/tensor/field.cpp:61-94): corner-major rows (row = corner * n + point), coordinates
// floor(v) + corner bit per spatial axis (batch column floor(v)), features scaled by
// prod_axis (bit ? frac : 1 - frac). One thread per (output row, 4-channel group).
template <typename T>
__global__ void __launch_bounds__(256) k_field_splat(const float* __restrict__ field, const T* __restrict__ feats,
                                                     uint32_t n, int W, int C, int32_t* __restrict__ out_coords,
                                                     T* __restrict__ out_feats) {
  const int groups = (C + 3) / 4;
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t rows = (uint64_t)n << (W - 1);
  if (t >= rows * groups) return;
  const uint64_t row = t / groups;
  const int g = (int)(t % groups);
  const uint32_t corner = (uint32_t)(row / n), point = (uint32_t)(row % n);
  float w = 1.0f;
  for (int a = 0; a < W; ++a) {
    const float v = field[(size_t)point * W + a];
    const float fl = floorf(v);
    int32_t c = (int32_t)fl;
    if (a > 0) {
      const float frac = v - fl;
      const bool upper = (corner >> (a - 1)) & 1u;
      w *= upper ? frac : 1.0f - frac;
      c += upper ? 1 : 0;
    }
    if (g == 0) out_coords[row * W + a] = c;
  }
  for (int ch = g * 4; ch < min(C, g * 4 + 4); ++ch)
    out_feats[row * C + ch] = (T)((float)feats[(size_t)point * C + ch] * w);
}

// out[(row * K + k)] = coords[row] + offsets[k] on the spatial columns (batch column copied)
__global__ void __launch_bounds__(256) k_expand(const int32_t* __restrict__ coords, uint64_t total, int W, int K,
                                                const int32_t* __restrict__ offsets, int32_t* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int col = (int)(i % (uint64_t)W);
  const uint64_t rk = i / (uint64_t)W;
  const int k = (int)(rk % (uint64_t)K);
  const uint64_t row = rk / (uint64_t)K;
  int32_t c = __ldg(coords + row * W + col);
  if (col > 0) c += __ldg(offsets + (size_t)k * (W - 1) + (col - 1));
  out[i] = c;
}

}  // namespace rmn

using namespace rmn;

extern "C" int rmn_coords_expand(const int32_t* d_coords, uint32_t n_rows, int W, const int32_t* d_offsets, int K,
                                 int32_t* d_out, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (W < 2 || W > RMN_MAX_W || K < 1) return RMN_ERR_BAD_ARG;
  if (n_rows == 0) return RMN_OK;
  if (!d_coords || !d_offsets || !d_out) return RMN_ERR_BAD_ARG;
  const uint64_t total = (uint64_t)n_rows * (uint64_t)K * (uint64_t)W;
  if ((uint64_t)n_rows * (uint64_t)K >= 0x7FFFFFFFull) return RMN_ERR_TOO_LARGE;
  k_expand<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(d_coords, total, W, K, d_offsets, d_out);
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_field_quantize(const float* d_field, uint32_t n_rows, int W, const int32_t* tensor_stride,
                                  int32_t* d_out, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (W < 2 || W > RMN_MAX_W || !tensor_stride) return RMN_ERR_BAD_ARG;
  if (n_rows == 0) return RMN_OK;
  if (!d_field || !d_out) return RMN_ERR_BAD_ARG;
  StrideArg st;
  for (int a = 0; a < RMN_MAX_W; ++a) st.s[a] = 1;
  for (int a = 0; a < W - 1; ++a) {
    if (tensor_stride[a] <= 0) return RMN_ERR_BAD_ARG;
    st.s[a] = tensor_stride[a];
  }
  const uint32_t nb = (n_rows + 255) / 256;
  if (W == 4 && !((uintptr_t)d_field & 15) && !((uintptr_t)d_out & 15))
    RMN_CUDA_TRY(launch_overlapped(k_field_quantize<4, true>, dim3(nb), dim3(256), 0, stream, d_field, n_rows, st, d_out));
  else
    RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_field_quantize<kW, false>, dim3(nb), dim3(256), 0, stream, d_field, n_rows,
                                                     st, d_out)));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_segment_reduce(const float* d_feats, uint32_t n_rows, int channels, const int64_t* d_inverse,
                                  const int64_t* d_mapping, uint32_t n_unique, int mean, float* d_out, uint32_t* d_counts,
                                  void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (channels < 1 || n_unique > n_rows) return RMN_ERR_BAD_ARG;
  if (n_unique == 0) return RMN_OK;
  if (!d_feats || !d_inverse || !d_mapping || !d_out || !d_counts) return RMN_ERR_BAD_ARG;
  if (channels == 4 && !((uintptr_t)d_feats & 15) && !((uintptr_t)d_out & 15)) {
    RMN_CUDA_TRY(launch_overlapped(k_segment_first4, dim3((n_unique + 255) / 256), dim3(256), 0, stream,
                        (const float4*)d_feats, d_mapping, n_unique, (float4*)d_out, d_counts));
  } else {
    const size_t total = (size_t)n_unique * channels;
    if (total >= ((size_t)1 << 39)) return RMN_ERR_TOO_LARGE;
    RMN_CUDA_TRY(launch_overlapped(k_segment_first, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream,
                        d_feats, d_mapping, n_unique, channels, d_out, d_counts));
  }
  RMN_LAUNCH_CHECK();
  if (n_unique == n_rows) return RMN_OK;
  RMN_CUDA_TRY(launch_overlapped(k_segment_add, dim3((n_rows + 255) / 256), dim3(256), 0, stream,
                        d_feats, d_inverse, d_mapping, n_rows, channels, d_out, d_counts));
  RMN_LAUNCH_CHECK();
  if (!mean) return RMN_OK;
  RMN_CUDA_TRY(launch_overlapped(k_segment_divide, dim3((n_unique + 255) / 256), dim3(256), 0, stream,
                        n_unique, channels, d_counts, d_out));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_coords_discretize(const void* d_in, int in_type, uint64_t n_elems, double quantization_size,
                                     int32_t* d_out, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (n_elems == 0) return RMN_OK;
  if (!d_in || !d_out || n_elems >= ((uint64_t)1 << 39)) return RMN_ERR_BAD_ARG;
  if (quantization_size != quantization_size) return RMN_ERR_BAD_ARG;  // NaN
  const uint32_t nb = (uint32_t)((n_elems + 255) / 256);
  switch (in_type) {
    case 0: k_discretize<float><<<nb, 256, 0, stream>>>((const float*)d_in, n_elems, quantization_size, d_out); break;
    case 1: k_discretize<double><<<nb, 256, 0, stream>>>((const double*)d_in, n_elems, quantization_size, d_out); break;
    case 2: k_discretize<int32_t><<<nb, 256, 0, stream>>>((const int32_t*)d_in, n_elems, quantization_size, d_out); break;
    default: return RMN_ERR_UNSUPPORTED;
  }
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_field_splat(const float* d_field, const void* d_feats, int dtype, uint32_t n_rows, int W, int C,
                               int32_t* d_out_coords, void* d_out_feats, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (W < 2 || W > RMN_MAX_W || C < 1) return RMN_ERR_BAD_ARG;
  if (n_rows == 0) return RMN_OK;
  if (!d_field || !d_feats || !d_out_coords || !d_out_feats) return RMN_ERR_BAD_ARG;
  const uint64_t rows = (uint64_t)n_rows << (W - 1);
  if (rows >= 0x7FFFFFFFull) return RMN_ERR_TOO_LARGE;
  const uint64_t threads = rows * (uint64_t)((C + 3) / 4);
  const uint32_t nb = (uint32_t)((threads + 255) / 256);
  if (dtype == RMN_F32)
    k_field_splat<float><<<nb, 256, 0, stream>>>(d_field, (const float*)d_feats, n_rows, W, C, d_out_coords,
                                                 (float*)d_out_feats);
  else if (dtype == RMN_BF16)
    k_field_splat<__nv_bfloat16><<<nb, 256, 0, stream>>>(d_field, (const __nv_bfloat16*)d_feats, n_rows, W, C,
                                                         d_out_coords, (__nv_bfloat16*)d_out_feats);
  else
    return RMN_ERR_UNSUPPORTED;
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" size_t rmn_table_bytes(uint32_t n_rows) {
  return sizeof(TableHeader) + sizeof(Slot) * (size_t)table_capacity(n_rows);
}

extern "C" size_t rmn_table_build_workspace_bytes(uint32_t n_rows) {
  return scratch_bytes(n_rows);
}

static int table_build_args(const int32_t* d_coords, uint32_t n_rows, int W, const void* d_table, size_t table_bytes,
                            const void* d_workspace, size_t workspace_bytes) {
  if (!d_table || W < 2 || W > RMN_MAX_W || n_rows >= 0x7FFFFFFFu) return RMN_ERR_BAD_ARG;
  if (n_rows > 0 && (!d_coords || !d_workspace)) return RMN_ERR_BAD_ARG;
  if (((uintptr_t)d_table & 15) || !coords_aligned(d_coords, W)) return RMN_ERR_BAD_ARG;
  if (table_bytes < rmn_table_bytes(n_rows) ||
      (n_rows > 0 && workspace_bytes < rmn_table_build_workspace_bytes(n_rows)))
    return RMN_ERR_ALLOC;
  return RMN_OK;
}

static int table_build_begin(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table, void* d_workspace,
                             int look_first, cudaStream_t stream) {
  auto* h = reinterpret_cast<TableHeader*>(d_table);
  auto* slots = reinterpret_cast<Slot*>(reinterpret_cast<char*>(d_table) + sizeof(TableHeader));
  const uint32_t capacity = table_capacity(n_rows);
  const Scratch sc = scratch(d_workspace, n_rows);
  static_assert(sizeof(TableHeader) == 64 * 4, "a thread per word");
  RMN_CUDA_TRY(launch_overlapped(k_clear_header, dim3(1), dim3(64), 0, stream, reinterpret_cast<uint32_t*>(h)));
  RMN_LAUNCH_CHECK();
  {
    const uint32_t fill_blocks = (capacity + 255u) / 256u;
    const uint32_t blocks = fill_blocks < kGrid ? fill_blocks : kGrid;
    RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_fill_range<kW>, dim3(blocks), dim3(256), 0, stream,
                        d_coords, n_rows, h, reinterpret_cast<uint4*>(slots), capacity, sc)));
    RMN_LAUNCH_CHECK();
  }
  if (n_rows == 0) return RMN_OK;
  const uint32_t nb = (n_rows + kRowsPerBlock - 1) / kRowsPerBlock;
  RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_insert<kW>, dim3(nb), dim3(256), 0, stream,
                        d_coords, n_rows, h, slots, sc, look_first)));
  RMN_LAUNCH_CHECK();
  if (look_first) {
    const uint32_t supers = (n_rows + kSuperRows - 1) / kSuperRows;
    RMN_CUDA_TRY(launch_overlapped(k_super_repeats, dim3((supers + 7) / 8), dim3(256), 0, stream, n_rows, h, sc));
    RMN_LAUNCH_CHECK();
  }
  return RMN_OK;
}

static int table_build_finish(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table, int64_t* d_mapping,
                              int64_t* d_inverse, int32_t* d_unique_coords, void* d_workspace, const HostPost& post,
                              cudaStream_t stream) {
  auto* h = reinterpret_cast<TableHeader*>(d_table);
  auto* slots = reinterpret_cast<Slot*>(reinterpret_cast<char*>(d_table) + sizeof(TableHeader));
  const Scratch sc = scratch(d_workspace, n_rows);
  const uint32_t nb = (n_rows + kRowsPerBlock - 1) / kRowsPerBlock;
  RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_finalize<kW>, dim3(nb), dim3(kRowsPerBlock), 0, stream,
                        d_coords, n_rows, h, slots, sc, d_mapping, d_unique_coords, d_inverse, post)));
  RMN_LAUNCH_CHECK();
  if (d_inverse) {  // optional: only the quantisation modes that average or sample features read it
    RMN_CUDA_TRY(launch_overlapped(k_inverse, dim3(nb < kGrid ? nb : kGrid), dim3(256), 0, stream,
                        slots, sc.slot_of_row, n_rows, h, d_inverse));
    RMN_LAUNCH_CHECK();
  }
  return RMN_OK;
}

static int table_build(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table, int64_t* d_mapping,
                       int64_t* d_inverse, int32_t* d_unique_coords, void* d_workspace, int look_first,
                       const HostPost& post, cudaStream_t stream) {
  if (n_rows > 0 && n_rows <= kSmallRows) {
    auto* h = reinterpret_cast<TableHeader*>(d_table);
    auto* slots = reinterpret_cast<Slot*>(reinterpret_cast<char*>(d_table) + sizeof(TableHeader));
    RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_build_small<kW>, dim3(1), dim3(1024), 0, stream,
                        d_coords, n_rows, h, slots, table_capacity(n_rows), scratch(d_workspace, n_rows), d_mapping,
                        d_unique_coords, d_inverse, look_first, post)));
    RMN_LAUNCH_CHECK();
    return RMN_OK;
  }
  const int rc = table_build_begin(d_coords, n_rows, W, d_table, d_workspace, look_first, stream);
  if (rc != RMN_OK || n_rows == 0) return rc;
  return table_build_finish(d_coords, n_rows, W, d_table, d_mapping, d_inverse, d_unique_coords, d_workspace, post, stream);
}

// First half of a build: header, slot fill + bounding box, insert, number of unique rows. When it has
// run, the header is final (number of unique rows, status): a caller may read it back while the second
// half is still running.
extern "C" int rmn_table_build_begin(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table,
                                     size_t table_bytes, void* d_workspace, size_t workspace_bytes,
                                     void* stream_) {
  const int rc = table_build_args(d_coords, n_rows, W, d_table, table_bytes, d_workspace, workspace_bytes);
  if (rc != RMN_OK) return rc;
  const int st = table_build_begin(d_coords, n_rows, W, d_table, d_workspace, 0, (cudaStream_t)stream_);
  if (st != RMN_OK || n_rows == 0) return st;
  RMN_CUDA_TRY(launch_overlapped(k_publish_unique, dim3(1), dim3(1), 0, (cudaStream_t)stream_, n_rows,
                                 reinterpret_cast<TableHeader*>(d_table)));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

// Second half: unique ids, mapping, unique coordinates, inverse. Same table, coordinates and workspace as
// the first half, on the same stream.
extern "C" int rmn_table_build_finish(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table,
                                      int64_t* d_mapping, int64_t* d_inverse, int32_t* d_unique_coords,
                                      void* d_workspace, void* stream_) {
  if (!d_table || W < 2 || W > RMN_MAX_W || n_rows >= 0x7FFFFFFFu) return RMN_ERR_BAD_ARG;
  if (n_rows == 0) return RMN_OK;
  if (!d_coords || !d_mapping || !d_workspace) return RMN_ERR_BAD_ARG;
  return table_build_finish(d_coords, n_rows, W, d_table, d_mapping, d_inverse, d_unique_coords, d_workspace,
                            HostPost{}, (cudaStream_t)stream_);
}

extern "C" int rmn_table_build(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table,
                               size_t table_bytes, int64_t* d_mapping, int64_t* d_inverse,
                               int32_t* d_unique_coords, void* d_workspace,
                               size_t workspace_bytes, void* stream_) {
  if (n_rows > 0 && n_rows < 0x7FFFFFFFu && !d_mapping) return RMN_ERR_BAD_ARG;
  const int rc = table_build_args(d_coords, n_rows, W, d_table, table_bytes, d_workspace, workspace_bytes);
  if (rc != RMN_OK) return rc;
  return table_build(d_coords, n_rows, W, d_table, d_mapping, d_inverse, d_unique_coords, d_workspace, 0, HostPost{},
                     (cudaStream_t)stream_);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of rmn_table_build.
//
// Some hosts may not allocate device memory once they are running: a perception
// loop with a fixed memory plan treats cudaMalloc as forbidden because it
// synchronises the whole device and can fail from fragmentation in the middle
// of a drive, and a plug-in loaded into somebody else's process may be handed
// input and output buffers but no allocator to ask for scratch. Such callers
// own the table, mapping and inverse buffers (they are outputs) yet have
// nowhere to put the build's scratch (slot-of-row array + block counters).
// Here that scratch lives in a file-scope device array of fixed size, so the
// call needs nothing beyond its inputs and outputs. The price is a hard row
// limit and 4.2 MiB of device memory held by every GPU that loads the library.
//
// The host symbol below is only a handle: kernels must be given the device
// address obtained with cudaGetSymbolAddress, which is looked up once per
// device (with that device current) on the first call made on it.
// ---------------------------------------------------------------------------
constexpr uint32_t kStaticMaxRows = 1u << 20;
constexpr size_t kStaticScratchBytes = rmn::scratch_bytes(kStaticMaxRows);
static __device__ __align__(256) unsigned char g_table_static_scratch[kStaticScratchBytes];

static int static_scratch_address(void** out) {
  constexpr int kMaxDevices = 64;
  static void* address[kMaxDevices] = {};
  static std::mutex lock;
  int dev = 0;
  RMN_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return RMN_ERR_BAD_ARG;
  std::lock_guard<std::mutex> guard(lock);
  if (!address[dev]) {
    void* p = nullptr;
    // the current device is `dev`: the address returned belongs to this device's copy of the array
    RMN_CUDA_TRY(cudaGetSymbolAddress(&p, g_table_static_scratch));
    if (!p) return RMN_ERR_CUDA;
    address[dev] = p;
  }
  *out = address[dev];
  return RMN_OK;
}

extern "C" uint32_t rmn_table_build_static_max_rows(void) { return kStaticMaxRows; }

extern "C" int rmn_table_build_static(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table,
                                      size_t table_bytes, int64_t* d_mapping, int64_t* d_inverse,
                                      int32_t* d_unique_coords, void* stream_) {
  if (n_rows > kStaticMaxRows) return RMN_ERR_TOO_LARGE;
  void* scratch = nullptr;
  const int rc = static_scratch_address(&scratch);
  if (rc != RMN_OK) return rc;
  // Nothing in the scratch has to start at zero: the build's first pass clears the bits and counts of
  // repeated rows and the insert pass writes the slot of every row before anything reads them, so
  // whatever an earlier call left behind is overwritten.
  return rmn_table_build(d_coords, n_rows, W, d_table, table_bytes, d_mapping, d_inverse,
                         d_unique_coords, scratch, kStaticScratchBytes, stream_);
}

// Small read-backs go through a kernel that stores into page-locked host memory, not through a copy
// engine: a device-to-host cudaMemcpyAsync waits its turn behind every copy already queued on that
// engine, on whatever stream, so the 256-byte header of a table build would sit behind the previous
// step's 150 MB result on its way to the host (measured: 6 ms behind two such copies, 14 us on an idle
// link) and the step behind it. Stores from an SM share the link but not the queue.
__global__ void k_words_to_host(const uint32_t* __restrict__ src, uint32_t n_words, const uint32_t* __restrict__ extra,
                                volatile uint32_t* __restrict__ dst) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_words; i += gridDim.x * blockDim.x) dst[i] = src[i];
  if (extra && blockIdx.x == 0 && threadIdx.x == 0) dst[n_words] = *extra;
  __threadfence_system();
}

// device-side alias of a page-locked host block, or NULL when the block is not mapped into the device
static void* device_alias(void* host_block) {
  void* d = nullptr;
  if (cudaHostGetDevicePointer(&d, host_block, 0) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return d;
}

extern "C" int rmn_readback_small(const void* d_src, void* h_dst_pinned, size_t bytes, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (bytes == 0) return RMN_OK;
  if (!d_src || !h_dst_pinned || (bytes & 3) || ((uintptr_t)d_src & 3) || ((uintptr_t)h_dst_pinned & 3) ||
      bytes > (1u << 20))
    return RMN_ERR_BAD_ARG;
  void* alias = device_alias(h_dst_pinned);
  if (!alias) {  // not page-locked / not mapped: the copy engine it is
    RMN_CUDA_TRY(cudaMemcpyAsync(h_dst_pinned, d_src, bytes, cudaMemcpyDeviceToHost, stream));
    return RMN_OK;
  }
  const uint32_t n_words = (uint32_t)(bytes / 4);
  k_words_to_host<<<(n_words + 255) / 256 < 64 ? (n_words + 255) / 256 : 64, 256, 0, stream>>>(
      static_cast<const uint32_t*>(d_src), n_words, nullptr, static_cast<volatile uint32_t*>(alias));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_table_info(const void* d_table, uint32_t info[4], void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!d_table || !info) return RMN_ERR_BAD_ARG;
  // The header is read back through a page-locked staging block owned by the calling thread: a copy into
  // pageable memory is staged by the driver and costs several microseconds more, and this read-back is the
  // one host synchronisation of a table build.
  // The same wait also brings back the status word of the convolution kernels (a bounded wait that ran out
  // in a kernel queued before this read-back on a stream this one is ordered after): every table build
  // of a host thus checks the convolutions that went before it without a synchronisation of its own.
  struct Staging {
    TableHeader header;
    uint32_t conv_status;  // directly behind the header: k_words_to_host stores it as word n_words
  };
  static_assert(sizeof(TableHeader) % 4 == 0 && offsetof(Staging, conv_status) == sizeof(TableHeader), "layout");
  thread_local Staging* staging = nullptr;
  if (!staging) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(Staging), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    staging = static_cast<Staging*>(p);
  }
  TableHeader pageable;
  TableHeader* dst = staging ? &staging->header : &pageable;
  void* alias = staging ? device_alias(staging) : nullptr;
  const uint32_t* d_conv_status = alias ? tc_status_device_address() : nullptr;
  if (alias && d_conv_status) {
    // header and status word in one launch, stored by the SM (see k_words_to_host)
    staging->header.magic = 0;
    staging->conv_status = 0;
    k_words_to_host<<<1, 64, 0, stream>>>(static_cast<const uint32_t*>(d_table), (uint32_t)(sizeof(TableHeader) / 4),
                                          d_conv_status, reinterpret_cast<volatile uint32_t*>(alias));
    RMN_LAUNCH_CHECK();
  } else {
    RMN_CUDA_TRY(cudaMemcpyAsync(dst, d_table, sizeof(TableHeader), cudaMemcpyDeviceToHost, stream));
    if (staging) {
      staging->conv_status = 0;
      RMN_CUDA_TRY(tc_copy_status_async(&staging->conv_status, stream) == RMN_OK ? cudaSuccess : cudaErrorUnknown);
    }
  }
  RMN_CUDA_TRY(cudaStreamSynchronize(stream));
  const TableHeader h = *dst;
  if (h.magic != kTableMagic) return RMN_ERR_BAD_ARG;
  info[0] = h.n_unique;
  info[1] = h.status;
  info[2] = h.capacity;
  info[3] = h.n_rows;
  if (h.status == RMN_OK && staging && staging->conv_status != 0) {
    const int st = (int)staging->conv_status;
    tc_clear_status();
    return st;
  }
  return (int)h.status;
}

// What a waiting host polls: page-locked words of the calling thread, never freed (a build may still store into them).
struct HostWords {
  uint32_t* host = nullptr;
  uint32_t* device = nullptr;
  uint32_t sequence = 0;
};
static HostWords& host_words() {
  thread_local HostWords w;
  if (!w.host) {
    void* p = nullptr;
    if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
    } else if (void* alias = device_alias(p)) {
      memset(p, 0, 64);
      w.host = static_cast<uint32_t*>(p);
      w.device = static_cast<uint32_t*>(alias);
    }
  }
  return w;
}

// The host waits by polling a word that the build stores, not for the stream: no read-back kernel, no event, no second
// stream, and the host goes on while the second half of the build runs.
extern "C" int rmn_table_build_counted(const int32_t* d_coords, uint32_t n_rows, int W, void* d_table, size_t table_bytes,
                                       int64_t* d_mapping, int64_t* d_inverse, int32_t* d_unique_coords, void* d_workspace,
                                       size_t workspace_bytes, int expect_duplicates, uint32_t info[4], void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!info) return RMN_ERR_BAD_ARG;
  int rc = table_build_args(d_coords, n_rows, W, d_table, table_bytes, d_workspace, workspace_bytes);
  if (rc != RMN_OK) return rc;
  HostWords& hw = host_words();
  HostPost post{};
  if (hw.host && n_rows > 0) {
    post.words = hw.device;
    post.conv_status = tc_status_device_address();
    post.sequence = ++hw.sequence ? hw.sequence : ++hw.sequence;
  }
  rc = table_build(d_coords, n_rows, W, d_table, d_mapping, d_inverse, d_unique_coords, d_workspace, expect_duplicates, post,
                   stream);
  if (rc != RMN_OK) return rc;
  if (!post.words) return rmn_table_info(d_table, info, stream_);
  const volatile uint32_t* words = hw.host;
  for (uint32_t spin = 1; words[5] != post.sequence; ++spin) {
    if (spin % 4096 != 0) {
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
      continue;
    }
    const cudaError_t e = cudaStreamQuery(stream);
    if (e == cudaErrorNotReady) {
      cudaGetLastError();
      continue;
    }
    if (e != cudaSuccess) return RMN_ERR_CUDA;
    if (words[5] == post.sequence) break;
    return rmn_table_info(d_table, info, stream_);  // the build has ended without storing
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  for (int i = 0; i < 4; ++i) info[i] = words[i];
  if (info[1] == RMN_OK && words[4] != 0) {
    const int st = (int)words[4];
    tc_clear_status();
    return st;
  }
  return (int)info[1];
}

extern "C" int rmn_table_find(const void* d_table, const int32_t* d_query, uint32_t n_query, int W,
                              int32_t* d_rows, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!d_table || W < 2 || W > RMN_MAX_W) return RMN_ERR_BAD_ARG;
  if (n_query == 0) return RMN_OK;
  if (!d_query || !d_rows || !coords_aligned(d_query, W)) return RMN_ERR_BAD_ARG;
  auto* h = reinterpret_cast<const TableHeader*>(d_table);
  auto* slots =
      reinterpret_cast<const Slot*>(reinterpret_cast<const char*>(d_table) + sizeof(TableHeader));
  const uint32_t nb = (n_query + 255) / 256;
  RMN_DISPATCH_W(W, k_find<kW><<<nb, 256, 0, stream>>>(h, slots, d_query, n_query, d_rows));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

extern "C" int rmn_coords_stride(const int32_t* d_coords, uint32_t n_rows, int W,
                                 const int32_t* out_tensor_stride, int32_t* d_out, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (W < 2 || W > RMN_MAX_W || !out_tensor_stride) return RMN_ERR_BAD_ARG;
  if (n_rows == 0) return RMN_OK;
  if (!d_coords || !d_out) return RMN_ERR_BAD_ARG;
  StrideArg st;
  for (int a = 0; a < RMN_MAX_W; ++a) st.s[a] = 1;
  for (int a = 0; a < W - 1; ++a) {
    if (out_tensor_stride[a] <= 0) return RMN_ERR_BAD_ARG;
    st.s[a] = out_tensor_stride[a];
  }
  const uint32_t nb = (n_rows + 255) / 256;
  if (W == 4 && !((uintptr_t)d_coords & 15) && !((uintptr_t)d_out & 15))
    RMN_CUDA_TRY(launch_overlapped(k_stride<4, true>, dim3(nb), dim3(256), 0, stream, d_coords, n_rows, st, d_out));
  else
    RMN_DISPATCH_W(W, RMN_CUDA_TRY(launch_overlapped(k_stride<kW, false>, dim3(nb), dim3(256), 0, stream, d_coords, n_rows, st,
                                                     d_out)));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}
