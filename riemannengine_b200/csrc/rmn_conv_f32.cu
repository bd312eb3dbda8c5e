// fp32 convolution passes for channel counts that are multiples of four: exact fp32 products and
// accumulation on the CUDA cores, work only for the neighbours that exist.
//
//   forward         out[j]  = sum_k F[nbr[k][j]]   . W[k]
//   backward input  dF[i]   = sum_k dY[nbr_t[k][i]] . W[k]^T   (the forward pass on transposed weights)
//   backward weight dW[k]   = sum_j F[nbr[k][j]]^T . dY[j]
//
// Half or more of a table's entries are empty (35 % of a shell's, 54 % of a room's, 95 % of a lidar sweep's), and a
// row-stationary register tile multiplies them as zeros. Both kernels compact the rows that have a neighbour at
// an offset first and multiply only those. All sums run in a fixed order: no atomics, bit-reproducible.
// The hosts run the forward pass and the input gradient here where little is to be done or the channel counts do not suit the
// tensor cores (rmn_conv_f32_pays), elsewhere by rmn_conv_f32_tc.cu.
#include "rmn_common.cuh"
#include "rmn_tc.cuh"

namespace rmn {

namespace {
__device__ __forceinline__ void ffma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float v) {
  unsigned long long p;
  asm("mov.b64 %0, {%1, %1};" : "=l"(p) : "f"(v));
  return p;
}
}  // namespace

// ------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------
// Every warp works on its own: it owns 32 output rows x 32 * NV columns, whose sums it keeps in shared memory, and
// walks over its offsets without a CTA barrier. Per offset it compacts the rows that have a neighbour (ballot) and takes
// them in batches of up to 8 * RGS lines: gather into the warp's ring (cp.async, one batch ahead), then RGS row groups
// (line l belongs to group l mod RGS) times 8 * NV column groups of four columns in registers, W[k] read through L1
// (the warps of an SM use the same few slices at a time), and the result added to the sums of its rows. The tile's
// height follows the number of lines: the kernel is bound by issued instructions.
// Where the rows alone would not fill the GPU, the offsets are dealt to `splits` warps per 32 rows, whose sums are
// added in split order.
// Measured on 101 930 rows, 65 % of the 27 entries present, 32 -> 32: 0.477 ms as a row-stationary 64 x 64 tile,
// 0.171 ms like this. Packed FFMA2 gains nothing: it runs at half the rate of FFMA (66 against 70 TFLOP/s measured)
// and its operands need MOVs; W[k] shared through shared memory (a barrier per offset) is no faster at 32 columns and
// 1.15 times slower at 64.
constexpr int kFwRows = 32, kFwLists = 4, kFwStages = 2;
constexpr int kFwLine = 36;  // 32 floats and four of padding: the row groups' reads do not conflict

template <int NV>
struct F32FwCfg {
  static constexpr int C = 32 * NV, CGS = 8 * NV, RGS = 32 / CGS;  // column and row groups of a warp
  static constexpr int BATCH = 8 * RGS;                            // lines of a full batch
  static constexpr int STAGE_WORDS = BATCH * kFwLine;
  static constexpr int WARP_WORDS = kFwRows * C + kFwStages * STAGE_WORDS + kFwLists * kFwRows + kFwLists * kFwRows / 4;
};

// acc[i][n] (+)= T lines of A x four columns of W, over cn chunks of four channels
// a: the lane's first line, `step` floats from its next one; wp: row ci of W, the lane's columns
template <int T>
__device__ __forceinline__ void f32_tile(float (&acc)[8][4], const float* a, int step, const float* wp, int c_col, int cn) {
#pragma unroll 2
  for (int c = 0; c < cn; ++c) {
    float4 b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      b[e] = __ldg(reinterpret_cast<const float4*>(wp));
      wp += c_col;
    }
#pragma unroll
    for (int i = 0; i < T; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(a + i * step + c * 4);
      const float av[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[i][0] = fmaf(av[e], b[e].x, acc[i][0]);
        acc[i][1] = fmaf(av[e], b[e].y, acc[i][1]);
        acc[i][2] = fmaf(av[e], b[e].z, acc[i][2]);
        acc[i][3] = fmaf(av[e], b[e].w, acc[i][3]);
      }
    }
  }
}

// sums of the rows += acc; acc = 0. dst: the rows of the row group's lines (eight bytes), live: how many of them count
template <int T>
__device__ __forceinline__ void f32_add_rows(float (&acc)[8][4], float* s_acc, int stride, const uint8_t* dst, int live) {
  const uint2 rows = *reinterpret_cast<const uint2*>(dst);
#pragma unroll
  for (int i = 0; i < T; ++i) {
    if (i < live) {
      float4* p = reinterpret_cast<float4*>(s_acc + (int)(((i < 4 ? rows.x : rows.y) >> (8 * (i % 4))) & 0xFFu) * stride);
      float4 v = *p;
      v.x += acc[i][0];
      v.y += acc[i][1];
      v.z += acc[i][2];
      v.w += acc[i][3];
      *p = v;
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) acc[i][n] = 0.f;
  }
}

template <int NV>
__global__ void __launch_bounds__(256)
    k_conv_f32(const float* __restrict__ src, const float* __restrict__ w, const int32_t* __restrict__ nbr, uint32_t n_dst,
               int K, int c_red, int c_col, int splits, float* __restrict__ out, const float* __restrict__ ep_scale,
               const float* __restrict__ ep_shift, int ep_relu, const uint32_t* __restrict__ only_if) {
  after_previous_kernel();
  if (only_if && !__ldg(only_if)) return;
  using Cfg = F32FwCfg<NV>;
  constexpr int C = Cfg::C, BATCH = Cfg::BATCH, RGS = Cfg::RGS;
  extern __shared__ __align__(16) float smem_f[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int groups = (int)(blockDim.x >> 5) / splits, split = warp % splits, group = warp / splits;
  float* s_acc = smem_f + warp * Cfg::WARP_WORDS;                                      // [32][C]
  float* s_ring = s_acc + kFwRows * C;                                                 // [stages][BATCH][kFwLine]
  int32_t* s_src = reinterpret_cast<int32_t*>(s_ring + kFwStages * Cfg::STAGE_WORDS);  // [lists][32] source rows
  uint8_t* s_dst = reinterpret_cast<uint8_t*>(s_src + kFwLists * kFwRows);             // [lists][batch][group][8] rows
  const uint32_t row0 = (blockIdx.x * groups + group) * kFwRows;
  const int n0 = blockIdx.y * C;
  const int n_chunks = (c_red + 31) / 32;
  const int rg = lane / Cfg::CGS, cg = lane % Cfg::CGS;

  for (int i = lane; i < kFwRows * C / 4; i += 32) reinterpret_cast<float4*>(s_acc)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  // (columns past the last are computed from column 0 and dropped)
  const int col = n0 + cg * 4 < c_col ? n0 + cg * 4 : 0;

  // An item is a batch (lines start .. start + count of the list in `slot`) and a 32-channel chunk j of offset k.
  struct Item {
    int k, j, slot, start, count;
  };
  int32_t idx = -1;
  auto load_idx = [&](int k) { idx = (k < K && row0 + lane < n_dst) ? __ldg(nbr + (size_t)k * n_dst + row0 + lane) : -1; };
  int pk = split - splits, pm = 0, pb = 0, pj = 0, lists = -1;
  load_idx(split);
  auto fetch = [&](int stage) -> Item {  // starts the gather of the next item
    while (pb >= pm && pk < K) {         // the current list is used up: the next offset that has a row
      pk += splits;
      if (pk >= K) break;
      const uint32_t have = __ballot_sync(0xFFFFFFFFu, idx >= 0);
      pm = __popc(have);
      pb = pj = 0;
      if (pm) {
        ++lists;
        const int base = (lists % kFwLists) * kFwRows, p = __popc(have & ((1u << lane) - 1u));
        if (idx >= 0) {
          s_src[base + p] = idx;
          s_dst[base + p / BATCH * BATCH + (p % RGS) * 8 + p % BATCH / RGS] = (uint8_t)lane;
        }
        __syncwarp();
      }
      load_idx(pk + splits);
    }
    Item it{K, 0, 0, 0, 0};
    if (pk < K) {
      it = Item{pk, pj, (lists % kFwLists) * kFwRows, pb, min(BATCH, pm - pb)};
      const int ch = lane & 7, cn = min(8, (c_red - pj * 32) >> 2);
      if (ch < cn) {  // eight lanes copy 32 floats of a row
        const float* s = src + pj * 32 + ch * 4;
        const uint32_t d = tc::smem_u32(s_ring + stage * Cfg::STAGE_WORDS + ch * 4);
        const int32_t* rows = s_src + it.slot + pb;
#pragma unroll
        for (int q = 0; q < BATCH / 4; ++q) {
          const int r = q * 4 + (lane >> 3);
          if (r < it.count) tc::cp_async16(d + r * (kFwLine * 4), s + (size_t)rows[r] * c_red, 16u);
        }
      }
      if (++pj == n_chunks) {
        pj = 0;
        pb += BATCH;
      }
    }
    tc::cp_async_commit();
    return it;
  };

  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int n = 0; n < 4; ++n) acc[i][n] = 0.f;

  Item it = fetch(0);
  for (int stage = 0; it.k < K; stage ^= 1) {
    const Item next = fetch(stage ^ 1);
    tc::cp_async_wait<1>();
    __syncwarp();
    const float* a = s_ring + stage * Cfg::STAGE_WORDS + rg * kFwLine;
    const float* wp = w + ((size_t)it.k * c_red + it.j * 32) * c_col + col;
    const uint8_t* dst = s_dst + it.slot + it.start + rg * 8;
    const int cn = min(8, (c_red - it.j * 32) >> 2), live = (it.count - rg + RGS - 1) / RGS;
    const bool last = it.j + 1 == n_chunks;
#define RMN_F32_TILE(T_)                                                            \
  {                                                                                 \
    f32_tile<T_>(acc, a, RGS * kFwLine, wp, c_col, cn);                             \
    if (last) f32_add_rows<T_>(acc, s_acc + cg * 4, C, dst, live);                  \
  }
    if (it.count > 6 * RGS) RMN_F32_TILE(8)
    else if (it.count > 4 * RGS) RMN_F32_TILE(6)
    else if (it.count > 2 * RGS) RMN_F32_TILE(4)
    else RMN_F32_TILE(2)
#undef RMN_F32_TILE
    __syncwarp();  // the stage and the list may be written again
    it = next;
  }
  tc::cp_async_wait<0>();
  if (splits > 1) __syncthreads();
  else __syncwarp();

  // the split's share of the rows: add the splits' sums in order, apply act(sum * scale + shift), store
  const float* base = smem_f + group * splits * Cfg::WARP_WORDS;
  for (int e = split * 32 + lane; e < kFwRows * C / 4; e += splits * 32) {
    const uint32_t row = row0 + e / (C / 4);
    const int n = n0 + (e % (C / 4)) * 4;
    if (row >= n_dst || n >= c_col) continue;
    float4 v = reinterpret_cast<const float4*>(base)[e];
    for (int s2 = 1; s2 < splits; ++s2) {
      const float4 t = reinterpret_cast<const float4*>(base + s2 * Cfg::WARP_WORDS)[e];
      v.x += t.x;
      v.y += t.y;
      v.z += t.z;
      v.w += t.w;
    }
    float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (ep_scale) f[q] *= __ldg(ep_scale + n + q);
      if (ep_shift) f[q] += __ldg(ep_shift + n + q);
      if (ep_relu) f[q] = relu_f32(f[q]);
    }
    *reinterpret_cast<float4*>(out + (size_t)row * c_col + n) = make_float4(f[0], f[1], f[2], f[3]);
  }
}

template <int NV>
static int launch_conv_f32(const float* src, const float* w, const int32_t* nbr, uint32_t n_dst, int K, int c_red, int c_col,
                           float* out, const float* ep_scale, const float* ep_shift, int ep_relu, const uint32_t* only_if,
                           cudaStream_t stream) {
  using Cfg = F32FwCfg<NV>;
  static SmemOptIn opt_in;
  RMN_CUDA_TRY(opt_in.apply(reinterpret_cast<const void*>(&k_conv_f32<NV>), 8 * Cfg::WARP_WORDS * 4));
  const uint32_t tiles_n = (uint32_t)(c_col + Cfg::C - 1) / Cfg::C;
  // Offsets are split while fewer than four rounds of warps (16 fit on an SM) would exist, so that the last round costs
  // little (101 930 rows: 0.186 ms with one round, 0.171 with four). A CTA is four warps, or the eight that share the
  // rows of a small problem.
  const uint32_t row_groups = (n_dst + kFwRows - 1) / kFwRows;
  int splits = 1;
  while (splits < 8 && splits * 2 <= K && row_groups * tiles_n * splits < 148u * 16u * 4u) splits *= 2;
  const int warps = splits == 8 ? 8 : 4;
  const uint32_t groups = warps / splits;
  dim3 grid((row_groups + groups - 1) / groups, tiles_n);
  RMN_CUDA_TRY(launch_overlapped(k_conv_f32<NV>, dim3(grid), dim3(warps * 32), (size_t)warps * Cfg::WARP_WORDS * 4, stream,
                                 src, w, nbr, n_dst, K, c_red, c_col, splits, out, ep_scale, ep_shift, ep_relu, only_if));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

// ------------------------------------------------------------------------------------------
// backward weight
// ------------------------------------------------------------------------------------------
// Grid (row chunks, offsets, 32 x COT channel tiles). A CTA walks its chunk in passes of kWgPass rows: the rows that
// have a neighbour at the offset are compacted into a pair list in shared memory, then each of the eight warps takes
// every eighth batch of kWgBatch pairs (two batches in flight, cp.async into the warp's own ring: no CTA barrier) and
// adds their outer products to its 32 x COT tile, 8 x (COT / 8) sums per lane (packed FFMA2 here: the plain form needs
// more registers than two CTAs per SM leave, 93 against 82 us). The warps' tiles are added in warp order at the end;
// k_reduce_f32 adds the chunks' partials in chunk order. 48 503 rows, 46 % present, 32 -> 64: 0.387 ms as a
// row-stationary 64 x 64 tile, 0.082 ms like this.
constexpr int kWgPass = 1024, kWgBatch = 16, kWgWarps = 8;

template <int COT>
struct F32WgCfg {
  static constexpr int RING = 2 * kWgBatch * (32 + COT);  // floats per warp
  static constexpr size_t SMEM = (size_t)kWgWarps * RING * 4 + kWgPass * 8;
  static_assert(kWgWarps * RING >= 32 * COT, "the final reduction reuses the rings");
};

template <int COT>
__global__ void __launch_bounds__(kWgWarps * 32, 2)
    k_wgrad_f32(const float* __restrict__ feats, const float* __restrict__ grad_out, const int32_t* __restrict__ nbr,
                uint32_t n_dst, int K, int c_in, int c_out, uint32_t chunk_rows, int tiles_co, float* __restrict__ partial) {
  after_previous_kernel();
  using Cfg = F32WgCfg<COT>;
  constexpr int NV = COT / 32;  // 4-column groups per lane, 32 columns apart
  extern __shared__ __align__(16) float smem_f[];
  __shared__ int s_warp_cnt[kWgWarps];
  int32_t* s_in = reinterpret_cast<int32_t*>(smem_f + kWgWarps * Cfg::RING);  // [kWgPass]
  int32_t* s_out = s_in + kWgPass;                                             // [kWgPass]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int k = blockIdx.y, ci0 = (blockIdx.z / tiles_co) * 32, co0 = (blockIdx.z % tiles_co) * COT;
  const uint32_t j_begin = blockIdx.x * chunk_rows, j_end = min(n_dst, j_begin + chunk_rows);
  const int32_t* table = nbr + (size_t)k * n_dst;
  float* ring = smem_f + warp * Cfg::RING;
  const int cig = lane >> 3, cog = lane & 7;

  unsigned long long acc[8][2 * NV];  // pairs of columns
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int n = 0; n < 2 * NV; ++n) acc[i][n] = 0ull;

  for (uint32_t j0 = j_begin; j0 < j_end; j0 += kWgPass) {
    // compaction: warp v owns rows [128 v, 128 v + 128) of the pass, so the list keeps the row order
    int32_t idx[4];
    uint32_t have[4];
    int mine = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint32_t j = j0 + warp * 128 + g * 32 + lane;
      idx[g] = j < j_end ? __ldg(table + j) : -1;
      have[g] = __ballot_sync(0xFFFFFFFFu, idx[g] >= 0);
      mine += __popc(have[g]);
    }
    __syncthreads();  // the previous pass no longer reads the list or the counts
    if (lane == 0) s_warp_cnt[warp] = mine;
    __syncthreads();
    int base = 0, total = 0;
#pragma unroll
    for (int v = 0; v < kWgWarps; ++v) {
      if (v < warp) base += s_warp_cnt[v];
      total += s_warp_cnt[v];
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      if (idx[g] >= 0) {
        const int p = base + __popc(have[g] & ((1u << lane) - 1u));
        s_in[p] = idx[g];
        s_out[p] = (int32_t)(j0 + warp * 128 + g * 32 + lane);
      }
      base += __popc(have[g]);
    }
    __syncthreads();

    const int n_batches = (total + kWgBatch - 1) / kWgBatch;
    auto fetch = [&](int b, int stage) {
      if (b < n_batches) {
        float* f = ring + stage * kWgBatch * (32 + COT);
        float* g = f + kWgBatch * 32;
        // eight lanes copy 32 floats of a row; pairs past the end and channels past the last are zero-filled
#pragma unroll
        for (int q = 0; q < kWgBatch / 4; ++q) {
          const int p = q * 4 + (lane >> 3), e = b * kWgBatch + p, ci = ci0 + (lane & 7) * 4;
          const bool ok = e < total && ci < c_in;
          tc::cp_async16(tc::smem_u32(f + p * 32 + (lane & 7) * 4), ok ? feats + (size_t)s_in[e] * c_in + ci : feats,
                         ok ? 16u : 0u);
#pragma unroll
          for (int h = 0; h < NV; ++h) {
            const int co = co0 + h * 32 + (lane & 7) * 4;
            const bool okg = e < total && co < c_out;
            tc::cp_async16(tc::smem_u32(g + p * COT + h * 32 + (lane & 7) * 4),
                           okg ? grad_out + (size_t)s_out[e] * c_out + co : grad_out, okg ? 16u : 0u);
          }
        }
      }
      tc::cp_async_commit();
    };
    fetch(warp, 0);
    int stage = 0;
    for (int b = warp; b < n_batches; b += kWgWarps, stage ^= 1) {
      fetch(b + kWgWarps, stage ^ 1);
      tc::cp_async_wait<1>();
      __syncwarp();
      const float* f = ring + stage * kWgBatch * (32 + COT) + cig * 8;
      const float* g = ring + stage * kWgBatch * (32 + COT) + kWgBatch * 32 + cog * 4;
#pragma unroll 4
      for (int p = 0; p < kWgBatch; ++p) {
        const float4 f0 = *reinterpret_cast<const float4*>(f + p * 32), f1 = *reinterpret_cast<const float4*>(f + p * 32 + 4);
        ulonglong2 gv[NV];
#pragma unroll
        for (int h = 0; h < NV; ++h) gv[h] = *reinterpret_cast<const ulonglong2*>(g + p * COT + h * 32);
        const float fv[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const unsigned long long ff = twice(fv[i]);
#pragma unroll
          for (int h = 0; h < NV; ++h) {
            ffma2(acc[i][2 * h], ff, gv[h].x);
            ffma2(acc[i][2 * h + 1], ff, gv[h].y);
          }
        }
      }
      __syncwarp();  // every lane is done with this half of the ring before it is filled again
    }
    tc::cp_async_wait<0>();
  }
  // tiles of the warps, added in warp order
  __syncthreads();
  for (int v = 0; v < kWgWarps; ++v) {
    if (warp == v) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int h = 0; h < NV; ++h) {
          float4* p = reinterpret_cast<float4*>(smem_f + (cig * 8 + i) * COT + h * 32 + cog * 4);
          const float4 t = v == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *p;
          const float2 a = *reinterpret_cast<float2*>(&acc[i][2 * h]), b = *reinterpret_cast<float2*>(&acc[i][2 * h + 1]);
          *p = make_float4(t.x + a.x, t.y + a.y, t.z + b.x, t.w + b.y);
        }
    }
    __syncthreads();
  }
  float* dst = partial + ((size_t)blockIdx.x * K + k) * c_in * c_out;
  for (int e = tid; e < 32 * COT / 4; e += kWgWarps * 32) {
    const int ci = ci0 + e / (COT / 4), co = co0 + (e % (COT / 4)) * 4;
    if (ci < c_in && co < c_out)
      *reinterpret_cast<float4*>(dst + (size_t)ci * c_out + co) = reinterpret_cast<const float4*>(smem_f)[e];
  }
}

// out[reverse ? K - 1 - k : k][co][ci] = w[k][ci][co]: 32 x 32 tiles through shared memory
template <typename T>
__global__ void __launch_bounds__(256) k_transpose_weights(const T* __restrict__ w, int K, int c_in, int c_out, int reverse,
                                                           T* __restrict__ out) {
  after_previous_kernel();
  __shared__ T tile[32][33];
  const int k = blockIdx.z, x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int ci0 = blockIdx.y * 32, co0 = blockIdx.x * 32;
  for (int r = y; r < 32; r += 8)
    if (ci0 + r < c_in && co0 + x < c_out) tile[r][x] = w[((size_t)k * c_in + ci0 + r) * c_out + co0 + x];
  __syncthreads();
  T* dst = out + (size_t)(reverse ? K - 1 - k : k) * c_in * c_out;
  for (int r = y; r < 32; r += 8)
    if (co0 + r < c_out && ci0 + x < c_in) dst[(size_t)(co0 + r) * c_in + ci0 + x] = tile[x][r];
}

// out[e] = sum over the chunks of partial[chunk][e], in chunk order; four elements per thread
__global__ void __launch_bounds__(128) k_reduce_f32(const float4* __restrict__ partial, uint32_t n_chunks, size_t vecs,
                                                    float4* __restrict__ out) {
  after_previous_kernel();
  const size_t e = (size_t)blockIdx.x * 128 + threadIdx.x;
  if (e >= vecs) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (uint32_t c = 0; c < n_chunks; ++c) {
    const float4 v = __ldcs(partial + (size_t)c * vecs + e);
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  out[e] = s;
}

// Row chunks of the weight gradient: enough CTAs for about four waves of two per SM (chunks of at least one pass),
// but no more partials than that needs.
static uint32_t f32_wgrad_chunk_rows(uint32_t n_dst, int K, int c_in, int c_out) {
  const uint32_t tiles = (uint32_t)((c_in + 31) / 32) * (uint32_t)(c_out <= 32 ? 1 : (c_out + 63) / 64);
  uint32_t chunks = (148u * 2u * 4u + (uint32_t)K * tiles - 1) / ((uint32_t)K * tiles);
  uint32_t rows = (n_dst + chunks - 1) / chunks;
  return (rows < (uint32_t)kWgPass ? (uint32_t)kWgPass : (rows + kWgPass - 1) / kWgPass * kWgPass);
}

bool f32_fast_shape(int c_in, int c_out) { return c_in % 4 == 0 && c_out % 4 == 0; }

static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// RMN_ERR_UNSUPPORTED where the shape or an alignment is not covered (the generic kernels take it then). only_if (or NULL): on the
// device, nothing is done where it holds 0.
int f32_conv_if(const float* src, const float* w, const int32_t* nbr, uint32_t n_dst, int K, int c_red, int c_col, float* out,
                const float* ep_scale, const float* ep_shift, int ep_relu, const uint32_t* only_if, cudaStream_t stream) {
  if (!f32_fast_shape(c_red, c_col) || !aligned16(src) || !aligned16(w) || !aligned16(out)) return RMN_ERR_UNSUPPORTED;
  return c_col <= 32
             ? launch_conv_f32<1>(src, w, nbr, n_dst, K, c_red, c_col, out, ep_scale, ep_shift, ep_relu, only_if, stream)
             : launch_conv_f32<2>(src, w, nbr, n_dst, K, c_red, c_col, out, ep_scale, ep_shift, ep_relu, only_if, stream);
}
int f32_conv(const float* src, const float* w, const int32_t* nbr, uint32_t n_dst, int K, int c_red, int c_col,
             float* out, const float* ep_scale, const float* ep_shift, int ep_relu, cudaStream_t stream) {
  return f32_conv_if(src, w, nbr, n_dst, K, c_red, c_col, out, ep_scale, ep_shift, ep_relu, nullptr, stream);
}

size_t f32_wgrad_workspace_bytes(uint32_t n_dst, int K, int c_in, int c_out) {
  const uint32_t rows = f32_wgrad_chunk_rows(n_dst, K, c_in, c_out);
  return (size_t)((n_dst + rows - 1) / rows) * K * c_in * c_out * sizeof(float);
}

int f32_conv_backward_weight(const float* feats, const float* grad_out, uint32_t n_dst, const int32_t* nbr, int K, int c_in,
                             int c_out, float* dw, float* workspace, cudaStream_t stream) {
  if (!f32_fast_shape(c_in, c_out) || !aligned16(feats) || !aligned16(grad_out) || !aligned16(dw) || !aligned16(workspace))
    return RMN_ERR_UNSUPPORTED;
  const uint32_t rows = f32_wgrad_chunk_rows(n_dst, K, c_in, c_out), chunks = (n_dst + rows - 1) / rows;
  const int cot = c_out <= 32 ? 32 : 64, tiles_co = (c_out + cot - 1) / cot;
  dim3 grid(chunks, K, (c_in + 31) / 32 * tiles_co);
  if (grid.z > 65535u) return RMN_ERR_UNSUPPORTED;  // (a launch takes no more)
  if (cot == 32) {
    static SmemOptIn opt_in;
    RMN_CUDA_TRY(opt_in.apply(reinterpret_cast<const void*>(&k_wgrad_f32<32>), F32WgCfg<32>::SMEM));
    RMN_CUDA_TRY(launch_overlapped(k_wgrad_f32<32>, dim3(grid), dim3(kWgWarps * 32), F32WgCfg<32>::SMEM, stream,
                                   feats, grad_out, nbr, n_dst, K, c_in, c_out, rows, tiles_co, workspace));
  } else {
    static SmemOptIn opt_in;
    RMN_CUDA_TRY(opt_in.apply(reinterpret_cast<const void*>(&k_wgrad_f32<64>), F32WgCfg<64>::SMEM));
    RMN_CUDA_TRY(launch_overlapped(k_wgrad_f32<64>, dim3(grid), dim3(kWgWarps * 32), F32WgCfg<64>::SMEM, stream,
                                   feats, grad_out, nbr, n_dst, K, c_in, c_out, rows, tiles_co, workspace));
  }
  RMN_LAUNCH_CHECK();
  const size_t vecs = (size_t)K * c_in * c_out / 4;
  RMN_CUDA_TRY(launch_overlapped(k_reduce_f32, dim3((uint32_t)((vecs + 127) / 128)), dim3(128), 0, stream,
                                 reinterpret_cast<const float4*>(workspace), chunks, vecs,
                                 reinterpret_cast<float4*>(dw)));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

}  // namespace rmn

using namespace rmn;

extern "C" int rmn_conv_transpose_weights(const void* d_weights, int K, int c_in, int c_out, int dtype, int reverse,
                                          void* d_out, void* stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!d_weights || !d_out || K < 1 || K > 65535 || c_in < 1 || c_out < 1 || c_in > 65536 || c_out > 65536 ||
      (dtype != RMN_F32 && dtype != RMN_BF16))
    return RMN_ERR_BAD_ARG;
  const dim3 grid((c_out + 31) / 32, (c_in + 31) / 32, K);
  if (dtype == RMN_F32)
    RMN_CUDA_TRY(launch_overlapped(k_transpose_weights<uint32_t>, dim3(grid), dim3(256), 0, stream,
                                   (const uint32_t*)d_weights, K, c_in, c_out, reverse, (uint32_t*)d_out));
  else
    RMN_CUDA_TRY(launch_overlapped(k_transpose_weights<uint16_t>, dim3(grid), dim3(256), 0, stream,
                                   (const uint16_t*)d_weights, K, c_in, c_out, reverse, (uint16_t*)d_out));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}
