// fp32 convolution on the tensor cores (sm_100a): the forward pass, and the input gradient on transposed weights.
//   out[j] = sum_k F[nbr[k][j]] . W[k]
//
// An fp32 number is the sum of three bf16 numbers x0 + x1 + x2 of eight significant bits each, every one the nearest to what the
// ones before it leave. Of the nine products of the parts of two numbers the six with i + j <= 2 are multiplied, the smallest
// first; the others lie below 2^-24 of the product. Tensor memory adds with truncation, so no sum stays there for long: after
// every stage (32 channels of an offset) it is read back and added, rounded to nearest, to sums in registers. These are added up in
// groups of stages, whose sums lie in shared memory, so that no long chain rounds at the size of the result: what the addition of a
// group leaves out begins the next group's sum (sum_and_rest), and two of the additions are rounded so that they take out the bias of
// the truncation (sum_outward). Error against 64 bits (2-norm) here / by k_conv_f32, whose sums of an offset are chains of
// multiply-adds: 30 000 random rows at 66 %, 32 -> 32, numbers of either sign 0.71e-7 / 1.22e-7, positive ones 0.41e-7 / 0.54e-7,
// 64 -> 64 0.86e-7 / 1.59e-7 and 0.46e-7 / 0.58e-7 (without groups 1.26e-7 and 1.06e-7, and some 4 % faster);
// 343 offsets, 32 -> 32 1.13e-7 / 1.54e-7 and 0.48e-7 / 0.58e-7, 64 -> 64 1.16e-7 / 1.84e-7 and 0.46e-7 / 0.58e-7 (without what is
// left out 1.55e-7 and 0.69e-7 there).
// (Read back every other stage, it is 2.7e-7.)
//
// Sums that are not finite are computed again with fp32 multiply-adds: infinities and NaN do not survive the split (inf - inf),
// nor do numbers that round to infinity in bf16. Numbers below 2^-102 lose their last parts, which fall below the normal numbers of
// bf16, up to 2^-126 of them in all; products below 2^-102 lose parts in the sums. So the kernel that prepares the weights also
// finds the largest and the smallest magnitude of the weights and of the features (one pass over these, 13 MB of 102 K rows, which
// the gathers then find in the L2), and if there is such a number or product, sums below 2^-90 times the largest operand (or 1) are
// computed again, too, zeros among them: what a sum of up to 2^11 such terms can have lost lies below 2^-25 of any other. The
// drain only marks their rows, and when the pipeline has ended sixteen of the CTA's warps take the marked ones (exact_rows):
// nothing in the pipeline waits for them, however many they are. 40 003 rows of infinities, 64 -> 64: 0.88 ms, 5.2 ms
// where the drain computed each row itself.
//
// The kernel is built like k_conv_ta (rmn_conv_ta.cuh): gather warps fetch rows into registers, split them there and store the
// parts into tensor memory as the A operand; W[k] comes as a prepared image by bulk copies. 20 warps: 8 gather (two groups of
// four), 2 MMA, 1 weights, 1 idle, 8 drain. Group g, issuer g and accumulators g make up stream g: one of the two row tiles of a
// super-tile (T = 2), or every other stage of a single one (T = 1). Waits are bounded, results bit-reproducible.
//
// What bounds it is the gather warps' chain of fetching, splitting (eleven instructions per two numbers) and storing a stage,
// some 600 cycles, against 12 MMAs of 16 to 32 cycles: 56 % of the issue slots and 22 % of the tensor pipe are busy at 32 -> 32, 61
// and 46 % at 64 -> 64. us with the weight image, back to back / k_conv_f32: 101 930 rows at 66 %, 32 -> 32 64 / 166, 64 -> 64
// 133 / 523; 48 503 rows at 45 %, 32 -> 64 44 / 116, 64 -> 32 62 / 141; 119 755 lidar voxels at 4 %, 32 -> 32 57 / 52, 64 -> 64
// 127 / 112 (k_conv_f32 goes with the rows that exist: see f3_asks_for_thin_tables. Blocks of 32 rows none of which exists are not
// split here, which took 13 and 22 us off).
#include "rmn_common.cuh"
#include "rmn_tc.cuh"

#include <cuda_bf16.h>

#include <cmath>

namespace rmn {

const uint32_t* tc_status_device_address();  // rmn_conv_tc.cu
void count_tc_launch();
int f32_conv_if(const float* src, const float* w, const int32_t* nbr, uint32_t n_dst, int K, int c_red, int c_col, float* out,
                const float* ep_scale, const float* ep_shift, int ep_relu, const uint32_t* only_if, cudaStream_t stream);

namespace tc {

template <int CC, int T_>
struct F3Cfg {
  static constexpr int T = T_, STREAMS = 2, PARTS = 3;
  static constexpr int KB = 32;                         // reduction channels of a stage
  static constexpr int A_COLS = PARTS * KB / 2;         // tensor-memory columns of one A slot
  static constexpr int ACC_BUFS = 2, ACC_COLS = STREAMS * ACC_BUFS * CC;
  static constexpr int FIT = (512 - ACC_COLS) / (STREAMS * A_COLS);
  static constexpr int SLOTS = FIT >= 4 ? 4 : 2;        // A slots per stream
  static constexpr uint32_t PART_BYTES = KB * CC * 2, B_BYTES = PARTS * PART_BYTES;
  static constexpr int B_STAGES = 8;
  static constexpr int BARRIERS = 2 * B_STAGES + 2 * STREAMS * SLOTS + 2 * STREAMS * ACC_BUFS;
  static constexpr uint32_t EP_OFFSET = 1024;  // behind the barriers: 2 * CC floats of epilogue scale / shift
  static constexpr uint32_t RING_OFFSET = 2048;  // W[k]
  static constexpr uint32_t TOTAL_OFFSET = RING_OFFSET + B_STAGES * B_BYTES;  // sums of the stages before the present group
  static constexpr int TOTAL_VECS = (T > 1 ? 2 : 1) * CC / 8;                 // float4 of each drain thread
  static constexpr uint32_t SMEM = TOTAL_OFFSET + TOTAL_VECS * 256 * 16;
  static_assert(FIT >= 2 && BARRIERS * 8 + 4 <= 1024 && (CC == 32 || CC == 64), "tensor / shared memory");
};
// Marks of a CTA's rows that are computed again, one bit each; rows beyond this many share them.
constexpr uint32_t kF3Marks = 8192;

constexpr int kF3MmaWarp = 8, kF3WeightWarp = 10, kF3DrainWarp0 = 12, kF3Warps = 20, kF3Threads = kF3Warps * 32;
// Registers: 640 threads x 96 at launch = 256 x 112 (gather) + 128 x 48 (MMA, weights) + 256 x 104 (drain)
constexpr int kF3GatherRegs = 112, kF3IssueRegs = 48, kF3DrainRegs = 104, kF3ExactRegs = 96;

struct F3Args {
  const float* src;      // [*, c_red]
  const uint8_t* image;  // k_f3_image of w
  const float* w;        // [K][c_red][c_col]
  const int32_t* nbr;
  float* out;            // [n_dst, c_col]
  const float* ep_scale;
  const float* ep_shift;
  const uint4* ranges;  // k_f3_image's
  uint32_t* thin;       // k_f3_image's, or NULL: 1 where k_conv_f32 does this pass
  uint32_t* status;
  uint32_t n_dst, n_super, n_ranges;
  int K, c_red, c_col, n_kb, relu, group;
};

// Largest magnitude and smallest but zero of some numbers, as bits without the sign, shifted up by one: .x and .z are the largest
// (weights, features), .y and .w the smallest minus one, where zero wraps around to the largest integer.
__device__ __forceinline__ void take_range(float v, uint32_t& most, uint32_t& least) {
  const uint32_t u = __float_as_uint(v) << 1;
  most = max(most, u);
  least = min(least, u - 1u);
}
constexpr uint4 kNoRange{0u, ~0u, 0u, ~0u};
__device__ __forceinline__ void merge_ranges(uint4 r, uint4* shared) {  // by a whole warp
  r.x = __reduce_max_sync(0xFFFFFFFFu, r.x);
  r.y = __reduce_min_sync(0xFFFFFFFFu, r.y);
  r.z = __reduce_max_sync(0xFFFFFFFFu, r.z);
  r.w = __reduce_min_sync(0xFFFFFFFFu, r.w);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&shared->x, r.x);
    atomicMin(&shared->y, r.y);
    atomicMax(&shared->z, r.z);
    atomicMin(&shared->w, r.w);
  }
}
// Magnitude (bits, shifted up by one) below which a sum is computed again
__device__ __forceinline__ uint32_t least_sum(uint4 r) {
  constexpr uint32_t kTiny = 25u << 24;  // 2^-102
  const bool lossy = r.y < kTiny || r.w < kTiny || (r.y >> 24) + (r.w >> 24) < 2 * 127 - 102;
  return lossy ? min(max(max(r.x, r.z), 127u << 24), (255u << 24) - 1u) - (90u << 24) : 0u;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t p;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo));
  return p;
}
// bf16 pair nearest to (lo, hi), which keep what is left
__device__ __forceinline__ uint32_t take_part(float& lo, float& hi) {
  const uint32_t p = pack_bf16(lo, hi);
  asm("{\n\t.reg .b64 v, q;\n\t"
      "mov.b64 v, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\t"
      "sub.rn.f32x2 v, v, q;\n\tmov.b64 {%0, %1}, v;\n\t}"
      : "+f"(lo), "+f"(hi)
      : "f"(__uint_as_float(p << 16)), "f"(__uint_as_float(p & 0xFFFF0000u)));
  return p;
}

// Order of the 32 channels of a stage along K (what the gather's loads and stores make of them), and of the CC columns of an
// image (for the drain's loads, see n_channel in rmn_conv_ta.cuh).
__device__ __forceinline__ constexpr uint32_t f3_k_channel(uint32_t p) {
  return 16 * (p >> 4) + 8 * ((p >> 1) & 1u) + 2 * ((p >> 2) & 3u) + (p & 1u);
}
template <int CC>
__device__ __forceinline__ constexpr uint32_t f3_n_channel(uint32_t p) {
  return (CC / 4) * ((p >> 1) & 3u) + 2 * (p >> 3) + (p & 1u);
}

// Image of the weights: per stage (offset, 32-channel block) and block of CC columns the three parts, each the MN-major swizzled
// operand of 32 lines. One thread per line and eight columns. reverse: offset k of the image is W[K - 1 - k]. plain (or NULL): the
// weights as [K][c_red][c_col] in the image's order of offsets. The blocks from image_blocks on read the n_x numbers of x. ranges:
// what each block has read. thin (or NULL): a last block looks at kF3Samples of the n_entries entries of the table, spread evenly,
// and says whether fewer than one in sixteen is a neighbour.
constexpr uint32_t kF3Samples = 4096;
template <int CC>
__global__ void __launch_bounds__(256) k_f3_image(const float* __restrict__ w, int K, int c_red, int c_col, int n_kb, int blocks,
                                                  int transpose, int reverse, uint4* __restrict__ image,
                                                  float* __restrict__ plain, uint32_t image_blocks, const float4* __restrict__ x,
                                                  size_t n_x, uint4* __restrict__ ranges, const int32_t* __restrict__ nbr,
                                                  uint64_t n_entries, uint32_t* __restrict__ thin) {
  after_previous_kernel();
  if (thin && blockIdx.x == gridDim.x - 1) {
    uint32_t found = 0;
#pragma unroll 16
    for (uint32_t i = threadIdx.x; i < kF3Samples; i += 256)  // (multiples of the golden ratio)
      found += __ldg(nbr + __umul64hi(i * 0x9E3779B97F4A7C15ull, n_entries)) >= 0 ? 1u : 0u;
    __shared__ uint32_t s_found;
    if (threadIdx.x == 0) s_found = 0u;
    __syncthreads();
    found = __reduce_add_sync(0xFFFFFFFFu, found);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_found, found);
    __syncthreads();
    if (threadIdx.x == 0) *thin = s_found < kF3Samples / 16 ? 1u : 0u;
    return;
  }
  const uint32_t range_blocks = gridDim.x - image_blocks - (thin ? 1u : 0u);
  __shared__ uint4 s_range;
  if (threadIdx.x == 0) s_range = kNoRange;
  __syncthreads();
  uint4 range = kNoRange;
  if (blockIdx.x >= image_blocks) {
    const size_t step = (size_t)range_blocks * 256;
#pragma unroll 4
    for (size_t i = (size_t)(blockIdx.x - image_blocks) * 256 + threadIdx.x; i < n_x / 4; i += step) {
      const float4 v = __ldg(x + i);
      take_range(v.x, range.z, range.w);
      take_range(v.y, range.z, range.w);
      take_range(v.z, range.z, range.w);
      take_range(v.w, range.z, range.w);
    }
  }
  constexpr uint32_t CPL = CC / 8, CHUNKS = 32 * CPL;
  const uint32_t lines = (uint32_t)(K * n_kb * blocks) * CHUNKS;
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; blockIdx.x < image_blocks && i < lines; i += image_blocks * 256) {
    const uint32_t block = i / CHUNKS, p = i % CHUNKS / CPL, c = i % CPL;
    const int stage = (int)block / blocks, k = stage / n_kb, col0 = ((int)block % blocks) * CC;
    const int ci = stage % n_kb * 32 + (int)f3_k_channel(p);
    const float* wk = w + (size_t)(reverse ? K - 1 - k : k) * c_red * c_col;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int co = col0 + (int)f3_n_channel<CC>(c * 8 + q);
      const bool in = ci < c_red && co < c_col;
      v[q] = in ? __ldg(wk + (transpose ? (size_t)co * c_red + ci : (size_t)ci * c_col + co)) : 0.f;
      if (plain && in) plain[((size_t)k * c_red + ci) * c_col + co] = v[q];
      take_range(v[q], range.x, range.y);
    }
    uint4* dst = image + (size_t)block * 3 * CHUNKS + p * CPL + swz<CC * 2>(p, c);
#pragma unroll
    for (int part = 0; part < 3; ++part)
      dst[part * CHUNKS] = make_uint4(take_part(v[0], v[1]), take_part(v[2], v[3]), take_part(v[4], v[5]), take_part(v[6], v[7]));
  }
  merge_ranges(range, &s_range);
  __syncthreads();
  if (threadIdx.x == 0) ranges[blockIdx.x] = s_range;
}

// 32 channels of a gather warp's 32 rows: lane t holds channels 8 c .. 8 c + 7 and 16 + 8 c .. 16 + 8 c + 7 (c = t / 2 & 1) of row
// t / 4 + 8 (t & 1) of each half of 16, see RowBlock in rmn_conv_ta.cuh. The registers keep their place until they are split.
struct F3Rows {
  uint32_t v[2][16];
  bool any;  // (the same in all lanes) one of the rows exists
  __device__ __forceinline__ void load(const float* __restrict__ src_lane, int c_red, int32_t idx, int kb, int lane) {
    const int mine = (lane >> 2) + 8 * (lane & 1), ch = kb * 32 + 8 * ((lane >> 1) & 1);
    any = __any_sync(0xFFFFFFFFu, idx >= 0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int32_t row = __shfl_sync(0xFFFFFFFFu, idx, h * 16 + mine);
      const float* p = src_lane + (size_t)(uint32_t)row * (uint32_t)c_red + kb * 32;
      ldg32_or_zero<0>(p, row >= 0 && ch < c_red, v[h]);
      ldg32_or_zero<8>(p + 16, row >= 0 && ch + 16 < c_red, v[h]);
    }
  }
  __device__ __forceinline__ void store_zeros(uint32_t taddr) const {  // (of rows none of which exists: v is zero)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      {
        tc_st16x64b(taddr + ((uint32_t)(h * 16) << 16), v[h]);  // 32 columns, and the 16 behind them
        uint32_t p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = v[h][i];
        tc_st16x64b(taddr + ((uint32_t)(h * 16) << 16) + 32, p);
      }
  }
  __device__ __forceinline__ void split_store(uint32_t taddr) const {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(v[h][i]);
#pragma unroll
      for (int part = 0; part < 3; ++part) {
        uint32_t p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = take_part(x[2 * i], x[2 * i + 1]);
        tc_st16x64b(taddr + ((uint32_t)(h * 16) << 16) + part * 16, p);
      }
    }
  }
};

__device__ __forceinline__ float f3_finish(float v, float scale, float shift, int relu) {
  v = fmaf(v, scale, shift);
  return relu ? relu_f32(v) : v;
}

// a + b, rounded away from zero. Truncation costs a stage some 6e-8 of its sum on average, so the whole sum as much; two of the sums
// of groups, at about half of the whole and at its end, rounded like this give most of it back (a later one than at half gave back up
// to 4e-8 too much). Sums that are exact stay so.
__device__ __forceinline__ float sum_outward(float a, float b) {
  const float up = __fadd_ru(a, b), down = __fadd_rd(a, b);
  return up >= 0.f ? up : down;
}

// a becomes a + b, and b what its rounding has left out (Knuth's TwoSum), with which the next group begins
__device__ __forceinline__ void sum_and_rest(float& a, float& b) {
  const float s = __fadd_rn(a, b), part = __fsub_rn(s, a);
  b = __fadd_rn(__fsub_rn(a, __fsub_rn(s, part)), __fsub_rn(b, part));
  a = s;
}

// Rows row0 .. row0 + 3 (columns col0 .. col0 + CC - 1) by fp32 multiply-adds, by a whole warp: a lane per column of every 32
template <int CC>
__device__ __forceinline__ void exact_rows(const F3Args& a, uint32_t row0, int col0, const float* s_ep, int lane) {
  constexpr int NC = CC / 32;
  if (row0 >= a.n_dst) return;
  float sum[4][NC];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < NC; ++c) sum[r][c] = 0.f;
  auto entry = [&](int k, int r) { return k < a.K && row0 + r < a.n_dst ? __ldg(a.nbr + (size_t)k * a.n_dst + row0 + r) : -1; };
  int32_t next[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) next[r] = entry(0, r);
#pragma unroll 1
  for (int k = 0; k < a.K; ++k) {
    int32_t idx[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      idx[r] = next[r];
      next[r] = entry(k + 1, r);
    }
    if ((idx[0] & idx[1] & idx[2] & idx[3]) < 0) continue;  // none exists
    float part[4][NC];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < NC; ++c) part[r][c] = 0.f;
    const float* w = a.w + (size_t)k * a.c_red * a.c_col;
#pragma unroll 1
    for (int c0 = 0; c0 < a.c_red; c0 += 32) {
      float x[4];  // a channel per lane
#pragma unroll
      for (int r = 0; r < 4; ++r)
        x[r] = idx[r] >= 0 && c0 + lane < a.c_red ? __ldg(a.src + (size_t)idx[r] * a.c_red + c0 + lane) : 0.f;
#pragma unroll 1
      for (int ci = 0; ci < 32 && c0 + ci < a.c_red; ci += 4) {
        float v[4][NC];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int col = col0 + 32 * c + lane;
            v[e][c] = __ldg(w + (size_t)(c0 + ci + e) * a.c_col + (col < a.c_col ? col : 0));  // (columns past the last are dropped)
          }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float xe = __shfl_sync(0xFFFFFFFFu, x[r], ci + e);
#pragma unroll
            for (int c = 0; c < NC; ++c) part[r][c] = fmaf(xe, v[e][c], part[r][c]);
          }
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (idx[r] >= 0) sum[r][c] += part[r][c];
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int at = 32 * c + lane;
      if (row0 + r < a.n_dst && col0 + at < a.c_col)
        a.out[(size_t)(row0 + r) * a.c_col + col0 + at] = f3_finish(sum[r][c], s_ep[at], s_ep[CC + at], a.relu);
    }
}

// blockIdx.y: block of CC columns
template <int CC, int T_>
__global__ void __launch_bounds__(kF3Threads, 1) k_conv_f3(const __grid_constant__ F3Args a) {
  using C = F3Cfg<CC, T_>;
  constexpr int T = T_, SLOTS = C::SLOTS, BST = C::B_STAGES, SWB = CC * 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint32_t s_marks[kF3Marks / 32], s_marked;
  __shared__ uint4 s_range;
  uint64_t* b_full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* b_empty = b_full + BST;
  uint64_t* a_full = b_empty + BST;              // [stream][slot]
  uint64_t* a_empty = a_full + 2 * SLOTS;        // [stream][slot]
  uint64_t* acc_full = a_empty + 2 * SLOTS;      // [stream][buffer]
  uint64_t* acc_empty = acc_full + 4;            // [stream][buffer]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 4);
  float* s_ep = reinterpret_cast<float*>(smem + C::EP_OFFSET);  // scale | shift

  // (uniform for the compiler, see k_conv_ta)
  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  if (tid < kF3Marks / 32) s_marks[tid] = 0u;
  if (tid == 0) {
    s_marked = 0u;
    s_range = kNoRange;
    for (int s = 0; s < BST; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], T > 1 ? 2 : 1);
    }
    for (int s = 0; s < 2 * SLOTS; ++s) {
      mbar_init(&a_full[s], 4);
      mbar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < 4; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], T > 1 ? 4 : 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  // (tensor memory is taken behind the kernels before this one and ahead of the next: see release_next_kernel)
  wait_previous_kernels();
  if (a.thin && __ldg(a.thin)) return;
  if (warp == kF3MmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const int col0 = (int)blockIdx.y * CC;
  if (tid < CC) {
    const bool in = col0 + tid < a.c_col;
    s_ep[tid] = a.ep_scale && in ? __ldg(a.ep_scale + col0 + tid) : 1.f;
    s_ep[CC + tid] = a.ep_shift && in ? __ldg(a.ep_shift + col0 + tid) : 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  release_next_kernel();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t smem_base = smem_u32(smem) + C::RING_OFFSET;
  const int n_stages = a.K * a.n_kb;
  // stages of a stream per super-tile
  auto stages_of = [&](int stream) { return T > 1 ? n_stages : (n_stages + 1 - stream) / 2; };
  bool timed_out = false;

  if (warp < kF3MmaWarp) {
    // ------------------------------ gather ---------------------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kF3GatherRegs));
    constexpr int STEP = T > 1 ? 1 : 2;
    const int g = warp >> 2, t = T > 1 ? g : 0;
    const float* src_lane = a.src + 8 * ((lane >> 1) & 1);
    const uint32_t a_base = tmem_base + C::ACC_COLS + g * SLOTS * C::A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t bars = smem_u32(a_full + g * SLOTS);  // full barriers; the empty ones lie 2 * SLOTS further

    // Cursor over the table entries of this lane's rows and the channel blocks that go with them; kEnd behind the last one
    constexpr int32_t kEnd = INT32_MIN;
    uint32_t st = blockIdx.x;
    int k = a.K, kb = 0, kb_next = 0;
    const int32_t* entry = a.nbr;
    bool row_ok = false, fresh = true;
    auto next = [&]() -> int32_t {
      for (;;) {
        if (k < a.K) {
          const int32_t v = row_ok ? __ldg(entry) : -1;
          kb = kb_next;
          kb_next += STEP;
          while (kb_next >= a.n_kb) {
            kb_next -= a.n_kb;
            ++k;
            entry += a.n_dst;
          }
          return v;
        }
        if (!fresh) st += gridDim.x;
        fresh = false;
        if (st >= a.n_super) {
          fresh = true;  // stay here
          return kEnd;
        }
        const uint32_t row = st * (kTileM * T) + t * kTileM + (warp & 3) * 32 + lane;
        row_ok = row < a.n_dst;
        entry = a.nbr + row;
        k = 0;
        kb_next = T > 1 ? 0 : g;
        while (kb_next >= a.n_kb) {
          kb_next -= a.n_kb;
          ++k;
          entry += a.n_dst;
        }
      }
    };
    // (entries are fetched four stages ahead, rows two, in windows unrolled by hand: see k_conv_ta)
    uint32_t cnt = 0, zero = 0;  // zero: slots whose rows of this warp are zeros already
    F3Rows b0, b1;
    auto load = [&](F3Rows& b, int32_t idx, int block) { b.load(src_lane, a.c_red, idx, block, lane); };
    auto arrive = [&]() {  // the block stored last has reached tensor memory
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + ((cnt - 1u) % SLOTS) * 8);
    };
    auto put = [&](const F3Rows& b) {
      if (cnt) arrive();
      const uint32_t s = cnt % SLOTS, ph = (cnt / SLOTS) & 1u;
      ++cnt;
      if (!mbar_wait(bars + (2 * SLOTS + s) * 8, ph ^ 1u)) timed_out = true;
      tc_fence_after();
      __syncwarp();
      if (b.any) {
        b.split_store(a_base + s * C::A_COLS);
        zero &= ~(1u << s);
      } else if (!((zero >> s) & 1u)) {
        b.store_zeros(a_base + s * C::A_COLS);
        zero |= 1u << s;
      }
    };
    int32_t w0, w1, w2, w3;
    int x0, x1, x2, x3;
    w0 = next(), x0 = kb;
    w1 = next(), x1 = kb;
    load(b0, w0, x0);
    load(b1, w1, x1);
    bool live0 = w0 != kEnd, live1 = w1 != kEnd;
    w2 = next(), x2 = kb;
    w3 = next(), x3 = kb;
    w0 = next(), x0 = kb;
    w1 = next(), x1 = kb;
    while (live0) {
      put(b0);
      load(b0, w2, x2);
      live0 = w2 != kEnd;
      w2 = next(), x2 = kb;
      if (!live1) break;
      put(b1);
      load(b1, w3, x3);
      live1 = w3 != kEnd;
      w3 = next(), x3 = kb;
      if (!live0) break;
      put(b0);
      load(b0, w0, x0);
      live0 = w0 != kEnd;
      w0 = next(), x0 = kb;
      if (!live1) break;
      put(b1);
      load(b1, w1, x1);
      live1 = w1 != kEnd;
      w1 = next(), x1 = kb;
      if (__any_sync(0xFFFFFFFFu, timed_out)) break;
    }
    if (cnt) arrive();
  } else if (warp < kF3DrainWarp0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kF3IssueRegs));
    if (warp < kF3MmaWarp + 2) {
      // ------------------------------ MMA issuers ----------------------------------------
      constexpr uint32_t IDESC = instr_desc(kTileM, CC, true);
      constexpr uint64_t B_DESC0 = smem_desc_sw_const(C::PART_BYTES, 8 * SWB, SWB == 128 ? 2u : 4u);
      constexpr uint32_t B_DESC_HI = (uint32_t)(B_DESC0 >> 32);
      const int stream = warp - kF3MmaWarp, mine = stages_of(stream);
      uint32_t cnt = 0, b_base = 0;
      for (uint32_t st = blockIdx.x; st < a.n_super && !timed_out; st += gridDim.x, b_base += (uint32_t)n_stages) {
        for (int i = 0; i < mine; ++i, ++cnt) {
          const uint32_t b_it = b_base + (T > 1 ? i : 2 * i + stream), bs = b_it % BST, s = cnt % SLOTS;
          const uint32_t buf = cnt & 1u;
          if (!mbar_wait(&b_full[bs], (b_it / BST) & 1u)) { timed_out = true; goto mma_done; }
          if (!mbar_wait(&a_full[stream * SLOTS + s], (cnt / SLOTS) & 1u)) { timed_out = true; goto mma_done; }
          if (!mbar_wait(&acc_empty[stream * 2 + buf], ((cnt >> 1) & 1u) ^ 1u)) {
            timed_out = true;
            goto mma_done;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (stream * 2 + buf) * CC;
          const uint32_t a_tmem = tmem_base + C::ACC_COLS + (stream * SLOTS + s) * C::A_COLS;
          const uint32_t b_lo = ((smem_base + bs * C::B_BYTES) >> 4) + (uint32_t)(B_DESC0 & 0xFFFFFFFFu);
          static_for<12>([&](auto xc) {
            constexpr int x = decltype(xc)::value, j = x & 1;
            constexpr int pa[6] = {2, 1, 0, 1, 0, 0}, pb[6] = {0, 1, 2, 0, 1, 0};
            const uint64_t b_desc = ((uint64_t)B_DESC_HI << 32) | (b_lo + ((pb[x / 2] * C::PART_BYTES + j * 16 * SWB) >> 4));
            tc_mma_bf16_ta_elect(d_tmem, a_tmem + pa[x / 2] * 16 + j * 8, b_desc, IDESC, x > 0 ? 1u : 0u);
          });
          tc_commit_elect(&a_empty[stream * SLOTS + s]);
          tc_commit_elect(&b_empty[bs]);
          tc_commit_elect(&acc_full[stream * 2 + buf]);
        }
      }
    mma_done:;
    } else if (warp == kF3WeightWarp && lane == 0) {
      // ------------------------------ weights --------------------------------------------
      const uint8_t* image = a.image + (size_t)blockIdx.y * C::B_BYTES;
      uint32_t b_it = 0;
      for (uint32_t st = blockIdx.x; st < a.n_super && !timed_out; st += gridDim.x) {
        for (int i = 0; i < n_stages; ++i, ++b_it) {
          const uint32_t s = b_it % BST;
          if (!mbar_wait(&b_empty[s], ((b_it / BST) & 1u) ^ 1u)) { timed_out = true; break; }
          bulk_load(smem_base + s * C::B_BYTES, image + (size_t)i * gridDim.y * C::B_BYTES, C::B_BYTES, smem_u32(&b_full[s]));
        }
      }
      // no copy may be in flight when the CTA exits: wait for the last round of the ring
      for (uint32_t i = b_it > BST ? b_it - BST : 0; i < b_it; ++i)
        if (!mbar_wait(&b_full[i % BST], (i / BST) & 1u)) timed_out = true;
    }
  } else if (warp < kF3Warps) {
    // ------------------------------ drain ----------------------------------------------
    // Four warps per set, one per 32 rows. T = 2: set d adds up stream d; T = 1: set d half d of the rows, of both streams.
    // Lane t holds, of rows t / 4 and t / 4 + 8 of a half, CC / 4 channels from (t % 4) * CC / 4 on.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kF3DrainRegs));
    constexpr int HALVES = T > 1 ? 2 : 1;
    const int set = (warp - kF3DrainWarp0) >> 2, u = lane & 3;
    const uint32_t quad = warp & 3;
    const int longest = stages_of(0);
    {
      uint4 range = kNoRange;
      for (uint32_t i = tid - kF3DrainWarp0 * 32; i < a.n_ranges; i += 256) {
        const uint4 r = __ldg(a.ranges + i);
        range = make_uint4(max(range.x, r.x), min(range.y, r.y), max(range.z, r.z), min(range.w, r.w));
      }
      merge_ranges(range, &s_range);
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    float4* total = reinterpret_cast<float4*>(smem + C::TOTAL_OFFSET) + tid - kF3DrainWarp0 * 32;  // vector q: total[256 q]
    uint32_t cnt[2] = {0, 0}, mark = (T > 1 ? set * 4 : 0) + quad;  // of this warp's block of 32 rows
    for (uint32_t st = blockIdx.x; st < a.n_super && !timed_out; st += gridDim.x, mark += 4 * T) {
      float sum[HALVES][CC / 8][4];
#pragma unroll
      for (int h = 0; h < HALVES; ++h)
#pragma unroll
        for (int v = 0; v < CC / 8; ++v)
#pragma unroll
          for (int e = 0; e < 4; ++e) sum[h][v][e] = 0.f;
      int d = 0;
      for (bool grouped = false;; grouped = true) {
        const int end = min(longest, d + a.group);
#pragma unroll 1
        for (; d < end && !timed_out; ++d) {
#pragma unroll
          for (int x = 0; x < (T > 1 ? 1 : 2); ++x) {
            const int stream = T > 1 ? set : x;
            if (d >= stages_of(stream)) continue;
            const uint32_t acc = stream * 2 + (cnt[x] & 1u), ph = (cnt[x] >> 1) & 1u;
            ++cnt[x];
            if (!mbar_wait(&acc_full[acc], ph)) timed_out = true;
            timed_out = __any_sync(0xFFFFFFFFu, timed_out);
            if (timed_out) break;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {
              const uint32_t taddr = tmem_base + ((quad * 32u + (T > 1 ? h : set) * 16u) << 16) + acc * CC;
              uint32_t r[CC / 32][16];
#pragma unroll
              for (int q = 0; q < CC / 32; ++q) tc_ld16x256b(taddr + q * 32, r[q]);
              tc_wait_ld();
#pragma unroll
              for (int v = 0; v < CC / 2; ++v) sum[h][v / 4][v % 4] += __uint_as_float(r[v / 16][v % 16]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
          }
        }
        // Outward: the last two sums of two or three groups; of more, the first that holds half of the stages and the last.
        const bool outward = d == longest || (2 * d >= longest && 2 * (d - a.group) < longest);
        if (grouped && outward) {
#pragma unroll
          for (int q = 0; q < C::TOTAL_VECS; ++q) {
            float(&f)[4] = sum[q / (CC / 8)][q % (CC / 8)];
            const float4 before = total[256 * q];
            f[0] = sum_outward(before.x, f[0]);
            f[1] = sum_outward(before.y, f[1]);
            f[2] = sum_outward(before.z, f[2]);
            f[3] = sum_outward(before.w, f[3]);
          }
        }
        if (timed_out || d == longest) break;
        if (grouped && !outward) {
#pragma unroll
          for (int q = 0; q < C::TOTAL_VECS; ++q) {
            float(&f)[4] = sum[q / (CC / 8)][q % (CC / 8)];
            float4 all = total[256 * q];
            sum_and_rest(all.x, f[0]);
            sum_and_rest(all.y, f[1]);
            sum_and_rest(all.z, f[2]);
            sum_and_rest(all.w, f[3]);
            total[256 * q] = all;
          }
        } else {
#pragma unroll
          for (int q = 0; q < C::TOTAL_VECS; ++q) {
            float(&f)[4] = sum[q / (CC / 8)][q % (CC / 8)];
            total[256 * q] = make_float4(f[0], f[1], f[2], f[3]);
            f[0] = f[1] = f[2] = f[3] = 0.f;
          }
        }
      }
      if (timed_out) break;
      const uint32_t least = least_sum(s_range);
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t row = st * (kTileM * T) + (T > 1 ? set : 0) * kTileM + quad * 32 + (T > 1 ? h : set) * 16 + i * 8 + (lane >> 2);
          bool bad = false;
#pragma unroll
          for (int v = 0; v < CC / 8; ++v)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              bad = bad || (__float_as_uint(sum[h][v][2 * i + e]) << 1) - least >= (255u << 24) - least;  // small, or not finite
            }
          if (bad && row < a.n_dst) {  // (rare)
            atomicOr(&s_marks[mark % (kF3Marks / 32)], 1u << ((T > 1 ? h : set) * 16 + i * 8 + (lane >> 2)));
            s_marked = 1u;
          }
          if (row < a.n_dst) {
            float* dst = a.out + (size_t)row * a.c_col;
#pragma unroll
            for (int v = 0; v < CC / 8; v += 2) {
              const int c = u * (CC / 4) + v * 2;
              if (col0 + c < a.c_col) {
                float4 f;
                f.x = f3_finish(sum[h][v][2 * i], s_ep[c], s_ep[CC + c], a.relu);
                f.y = f3_finish(sum[h][v][2 * i + 1], s_ep[c + 1], s_ep[CC + c + 1], a.relu);
                f.z = f3_finish(sum[h][v + 1][2 * i], s_ep[c + 2], s_ep[CC + c + 2], a.relu);
                f.w = f3_finish(sum[h][v + 1][2 * i + 1], s_ep[c + 3], s_ep[CC + c + 3], a.relu);
                *reinterpret_cast<float4*>(dst + col0 + c) = f;
              }
            }
          }
        }
      }
    }
  }

  if (timed_out) atomicExch(a.status, (uint32_t)RMN_ERR_TIMEOUT);
  tc_fence_before();
  const bool failed = __syncthreads_or(timed_out);
  if (warp == kF3MmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
  // ------------------------------ marked rows ------------------------------------------
  if (failed || !s_marked || (warp >= kF3MmaWarp && warp < kF3DrainWarp0)) return;
  __builtin_assume(warp < kF3Warps);
  if (warp < kF3Warps) {  // (all that are left: whole warpgroups)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kF3ExactRegs));
  }
  const uint32_t worker = warp < kF3MmaWarp ? warp : warp - (kF3DrainWarp0 - kF3MmaWarp);
  const uint32_t mine = (a.n_super - blockIdx.x + gridDim.x - 1) / gridDim.x * (32 * T);  // groups of four rows
  for (uint32_t i = worker; i < mine; i += 16) {
    if (!((s_marks[i / 8 % (kF3Marks / 32)] >> (i % 8 * 4)) & 15u)) continue;
    exact_rows<CC>(a, (blockIdx.x + i / (32 * T) * gridDim.x) * (kTileM * T) + i % (32 * T) * 4, col0, s_ep, lane);
  }
}

template <int CC, int T>
int launch_f3(F3Args a, uint32_t blocks, uint32_t fit, cudaStream_t stream) {
  using C = F3Cfg<CC, T>;
  static SmemOptIn opt_in;
  RMN_CUDA_TRY(opt_in.apply(reinterpret_cast<const void*>(&k_conv_f3<CC, T>), C::SMEM));
  a.n_super = (a.n_dst + kTileM * T - 1) / (kTileM * T);
  // Stages of a group: n stages in g groups leave a rounding error within them that goes with sqrt(n) / g, and some of the last sum.
  // Adding up a group costs the drain what a stage or two do, so few of them where they are short; but two from four stages on, for
  // the rounding that takes out the bias (7 offsets, 32 -> 64, positive numbers 0.66e-7 with one, 0.48e-7 with two, 0.57e-7
  // by multiply-adds).
  const int stages = a.K * a.n_kb, steps = T > 1 ? stages : (stages + 1) / 2;
  int groups = (int)(std::cbrt((double)stages) + 1e-6);
  if (groups < 2 && stages >= 4) groups = 2;
  if (groups < (stages + 47) / 48) groups = (stages + 47) / 48;
  a.group = (steps + groups - 1) / groups;
  RMN_CUDA_TRY(launch_overlapped(k_conv_f3<CC, T>, dim3(fit < a.n_super ? fit : a.n_super, blocks), dim3(kF3Threads), C::SMEM,
                                 stream, a));
  RMN_LAUNCH_CHECK();
  count_tc_launch();
  return RMN_OK;
}

constexpr uint32_t kF3ImageBlocks = 148 * 2, kF3RangeBlocks = 148 * 4;

template <int CC>
int run_f3(F3Args a, uint32_t n_src, int transpose, int reverse, uint8_t* image, float* plain, uint4* ranges, cudaStream_t stream) {
  int dev = 0, sms = 148;
  RMN_CUDA_TRY(cudaGetDevice(&dev));
  RMN_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t blocks = (uint32_t)(a.c_col + CC - 1) / CC, fit = (uint32_t)sms > blocks ? (uint32_t)sms / blocks : 1u;
  const uint32_t lines = (uint32_t)(a.K * a.n_kb) * blocks * 32 * (CC / 8);
  const size_t n_x = (size_t)n_src * a.c_red;
  const uint32_t image_blocks = (lines + 255) / 256 < kF3ImageBlocks ? (lines + 255) / 256 : kF3ImageBlocks;
  const uint32_t range_blocks = n_x / 8192 < kF3RangeBlocks ? (uint32_t)(n_x / 8192) + 1 : kF3RangeBlocks;
  RMN_CUDA_TRY(launch_overlapped(k_f3_image<CC>, dim3(image_blocks + range_blocks + (a.thin ? 1u : 0u)), dim3(256), 0, stream, a.w,
                                 a.K, a.c_red, a.c_col, a.n_kb, (int)blocks, transpose, reverse, reinterpret_cast<uint4*>(image),
                                 plain, image_blocks, reinterpret_cast<const float4*>(a.src), n_x, ranges, a.nbr,
                                 (uint64_t)a.K * a.n_dst, a.thin));
  RMN_LAUNCH_CHECK();
  a.ranges = ranges;
  a.n_ranges = image_blocks + range_blocks;
  a.image = image;
  if (plain) a.w = plain;
  // row tiles of the busiest SM: pairs of them share their weights, single ones leave fewer SMs idle at the end
  const uint32_t tiles = (a.n_dst + kTileM - 1) / kTileM, pairs = (tiles + 1) / 2;
  const uint32_t rounds2 = (pairs + fit - 1) / fit * 2, rounds1 = (tiles + fit - 1) / fit;
  const int st = rounds2 <= rounds1 ? launch_f3<CC, 2>(a, blocks, fit, stream) : launch_f3<CC, 1>(a, blocks, fit, stream);
  if (st != RMN_OK || !a.thin) return st;
  return f32_conv_if(a.src, a.w, a.nbr, a.n_dst, a.K, a.c_red, a.c_col, a.out, a.ep_scale, a.ep_shift, a.relu, a.thin, stream);
}

}  // namespace tc
}  // namespace rmn

using namespace rmn;

// The image of the weights, behind it the weights themselves in its order, then the ranges of k_f3_image's blocks
static size_t f3_image_bytes(int K, int c_in, int c_out) {
  const size_t cc = c_out <= 32 ? 32 : 64, columns = (c_out + cc - 1) / cc * cc;
  return (size_t)K * ((c_in + 31) / 32) * 32 * columns * 3 * 2;
}
static size_t f3_plain_bytes(int K, int c_in, int c_out) { return (size_t)K * c_in * c_out * sizeof(float); }  // (a multiple of 128)
extern "C" size_t rmn_conv_f32_scratch_bytes(uint32_t n_dst, int K, int c_in, int c_out) {
  if (n_dst == 0 || K < 1 || K > 4096 || c_in < 16 || c_in > 1024 || c_in % 8 || c_out < 4 || c_out > 1024 || c_out % 4) return 0;
  return f3_image_bytes(K, c_in, c_out) + f3_plain_bytes(K, c_in, c_out) +
         (tc::kF3ImageBlocks + tc::kF3RangeBlocks + 1) * sizeof(uint4);  // (and k_f3_image's word on the table)
}

// Little work is the multiply-add kernel's: these kernels need the weights prepared by a launch of their own, which a host that
// waits for nothing else pays for, and few rows leave most SMs idle while every row tile walks all offsets in turn. Passes of
// one layer, us there / here, forward alone and with its gradients, by the rows x offsets x channels in x out of the layer, in
// millions: 221 (8000 rows 32 -> 32) 69 / 66 and 168 / 173; 442 (32 -> 64) 75 / 67 and 168 / 172; 553 (20 000 rows 32 -> 32)
// 91 / 72 and 175 / 172; 663 (8000 rows 64 -> 48) 94 / 75 and 181 / 169; 90 (strided, 11 000 rows, 8 offsets) 94 / 99. (Device
// time alone, back to back: 221 16.1 / 15.7, 442 23 / 18, 553 39 / 25, 664 41 / 28.)
extern "C" int rmn_conv_f32_pays(uint32_t n_dst, int K, int c_in, int c_out) {
  return rmn_conv_f32_scratch_bytes(n_dst, K, c_in, c_out) > 0 && (double)n_dst * K * c_in * c_out >= 500e6;
}

// Thin tables are the multiply-add kernel's, which goes with the entries that are neighbours. Whether a table is thin is known on
// the device alone; both kernels are launched then, and one does nothing, for 5 us. So it is asked where that is little: us of
// the two kernels here / there, lidar sweeps of 119 755 voxels, 64 -> 64, 27 offsets (4 % neighbours) 139 / 121, 125 offsets (1.2 %)
// 548 / 270, 343 offsets (0.6 %) 1426 / 578, 32 -> 32 69 / 64, 231 / 172, 611 / 419; a shell at 66 % 142 / 531 and 73 / 176. The
// lines between lie at 5.0 % (32 -> 64) to 6.6 % (32 -> 32). A self map of 27 offsets has 3.7 % at least.
// Asked, the passes over 125 and 343 offsets take 183 and 436 (32 -> 32), 280 and 595 (64 -> 64); a shell's over 125 258 -> 263 and
// 519 -> 527.
static bool f3_asks_for_thin_tables(uint32_t n_dst, int K, int c_in, int c_out) {
  return (double)n_dst * K * c_in * c_out >= (K > 27 ? 8e9 : 40e9);
}

extern "C" int rmn_conv_forward_f32(const float* d_feats, uint32_t n_src, int c_in, const float* d_weights, int K, int c_out,
                                    int transpose, int reverse, const int32_t* d_nbr, uint32_t n_dst, float* d_out,
                                    const float* d_scale, const float* d_shift, int relu, void* d_scratch, size_t scratch_bytes,
                                    void* stream_) {
  if (n_dst == 0) return RMN_OK;
  const size_t need = rmn_conv_f32_scratch_bytes(n_dst, K, c_in, c_out);
  if (need == 0) return RMN_ERR_UNSUPPORTED;
  // (with no source rows every table entry is -1 and nothing is read through d_feats)
  if (!d_weights || !d_nbr || !d_out || !d_scratch || (n_src > 0 && !d_feats)) return RMN_ERR_BAD_ARG;
  // (weights are read by single elements: a view into a larger buffer of parameters need not be aligned)
  if (((uintptr_t)d_feats & 31) || ((uintptr_t)d_out & 15) || ((uintptr_t)d_scratch & 15))
    return RMN_ERR_UNSUPPORTED;
  if (scratch_bytes < need) return RMN_ERR_ALLOC;
  tc::F3Args a = {};
  a.src = d_feats;
  a.w = d_weights;
  a.nbr = d_nbr;
  a.out = d_out;
  a.ep_scale = d_scale;
  a.ep_shift = d_shift;
  a.status = const_cast<uint32_t*>(tc_status_device_address());
  a.n_dst = n_dst;
  a.K = K;
  a.c_red = c_in;
  a.c_col = c_out;
  a.n_kb = (c_in + 31) / 32;
  a.relu = relu;
  if (!a.status) return RMN_ERR_CUDA;
  uint8_t* image = static_cast<uint8_t*>(d_scratch);
  const bool ask = f3_asks_for_thin_tables(n_dst, K, c_in, c_out);
  // (for exact_rows, whose lanes read neighbouring columns, and k_conv_f32, which reads four elements at a time)
  uint8_t* behind = image + f3_image_bytes(K, c_in, c_out);
  float* plain = transpose || reverse || (ask && ((uintptr_t)d_weights & 15)) ? reinterpret_cast<float*>(behind) : nullptr;
  uint4* ranges = reinterpret_cast<uint4*>(behind + f3_plain_bytes(K, c_in, c_out));
  if (ask) a.thin = reinterpret_cast<uint32_t*>(ranges + tc::kF3ImageBlocks + tc::kF3RangeBlocks);
  return c_out <= 32 ? tc::run_f3<32>(a, n_src, transpose, reverse, image, plain, ranges, (cudaStream_t)stream_)
                     : tc::run_f3<64>(a, n_src, transpose, reverse, image, plain, ranges, (cudaStream_t)stream_);
}
