// Tensor-core convolution with the gathered operand in tensor memory (sm_100a, bf16 x bf16 -> fp32):
//   out[j] = sum_k F[nbr[k][j]] . W[k]
// the forward pass, and the input gradient on transposed weights. The weights come as an image prepared by
// k_weight_image (rmn_conv_weight_image): the entry points that bring no scratch for it run k_conv_tc instead.
//
// What bounds k_conv_tc is the load/store data pipe: a gathered 128-byte row is two wavefronts into shared memory, a
// zero row of a missing neighbour (54 % of a room's table) one, and the MMAs read every row back through the same pipe.
// Here a row goes from global memory to registers (two wavefronts: two lanes fetch 64 bytes at a time with 32-byte
// loads) and from there to tensor memory (tcgen05.st), where tcgen05.mma takes its A operand: a missing row is read from
// nowhere. It is not free: its stage is stored and multiplied all the same. 1.2 M x 27 entries, 64 -> 64: 215 us with no entry
// present, 270 at 46 %, 371 with all; the load/store pipe is 79 % busy at 46 %, half of it with the rows that exist, the tensor
// pipe 48 %. The order in which the registers of a row reach tensor memory is a permutation
// of its channels, which the weight image repeats along K; its columns are permuted so that the epilogue's
// tcgen05.ld gives every lane 32 contiguous bytes of an output row; and W[k] arrives by one bulk copy per stage.
//
// Persistent CTAs, one per SM, over super-tiles of T x 128 output rows. 24 warps: 16 gather (four groups of four: group g
// serves tile g % T), 2 MMA, 1 weights, 1 idle, 4 epilogue. A (tile, offset) stage costs the warp that issues its MMAs some 150
// cycles of barrier, fence and commit latency beside 128 of math at 64 columns, and one such warp is what bound tables of few
// entries. So two issue, each for half of the tiles; where a super-tile is a single tile of up to 64 columns, one takes its even
// stages and one its odd ones, into accumulators of their own that the epilogue adds (SPLIT; sums half as
// long, truncated half as often: of 230 400 results at 900 rows 256 -> 256 222 are not the bf16 number nearest to the 64-bit sum,
// with one accumulator 404; of 576 000 at 9000 rows 64 -> 64 168 and 261). Rows are fetched past the L1: a
// hit there passes the load/store pipe in twice the wavefronts of a miss. us before and after both: 1.2 M rows of rooms 64 -> 64
// 281 and 271, sorted by blocks 300 and 274, 32 -> 32 154 and 149; 240 000 lidar voxels 64 -> 64 57 and 51; 850 rows 256 -> 256
// 21.5 and 19.6. Waits are bounded (g_tc_status), results are bit-reproducible: every accumulator adds its offsets in ascending
// order, planned or not.
//
// Included by rmn_conv_tc.cu.
#pragma once

namespace rmn {
namespace tc {

// CC: columns of a CTA (of the whole product, or one of its 64-column blocks), T: row tiles that share one stage of W[k]
template <int CR, int CC, int T_>
struct TaCfg {
  static constexpr int KB = 64;                 // reduction channels per stage ...
  static constexpr int OPS = CR < KB ? 2 : 1;   // ... those of two offsets where a row has only 32 ...
  static constexpr int NKB = CR < KB ? 1 : CR / KB;  // ... or one of the NKB blocks of an offset
  static constexpr int T = T_;
  static constexpr int GROUPS = 4, PHASES = GROUPS / T;         // the PHASES groups of a tile take its stages in turn
  static constexpr int A_COLS = KB / 2;                         // tensor-memory columns of one A slot
  static constexpr int SPLIT = T == 1 && CC <= 64 ? 2 : 1;      // sums of a tile: even and odd stages apart, see the issuers
  static constexpr int ISSUERS = T > 1 ? 2 : SPLIT;
  static constexpr int SUM_COLS = T * SPLIT * CC;
  static constexpr int ACC_BUFS = SUM_COLS * 2 + GROUPS * 2 * A_COLS <= 512 ? 2 : 1;
  static constexpr int ACC_COLS = SUM_COLS * ACC_BUFS;
  static constexpr int FIT = (512 - ACC_COLS) / (GROUPS * A_COLS);
  static constexpr int SLOTS = FIT >= 4 ? 4 : 2;                // A slots per group
  static constexpr uint32_t B_BYTES = KB * CC * 2;
  static constexpr int B_STAGES = B_BYTES * 8 <= 64 * 1024 ? 8 : 4;
  static constexpr uint32_t BAR_OFFSET = B_STAGES * B_BYTES;
  static constexpr int BARRIERS = 2 * B_STAGES + 2 * GROUPS * SLOTS + 2 * ACC_BUFS * T;
  static constexpr uint32_t EP_OFFSET = BAR_OFFSET + 1024;                // 2 * CC floats of epilogue scale / shift
  static constexpr uint32_t STATS_OFFSET = EP_OFFSET + 2 * CC * 4;        // per-warp channel statistics, 4 * 2 * CC floats
  static constexpr uint32_t SMEM = STATS_OFFSET + 4 * 2 * CC * 4;
  static_assert(CR * OPS == KB * NKB && (OPS == 1 || CC <= 64), "stages");
  static_assert(FIT >= 2 && BARRIERS * 8 + 4 <= 1024, "tensor / shared memory");
};

// Registers: 768 threads x 80 at launch = 512 x 88 (gather) + 128 x 48 (MMA, weights) + 128 x 80 (epilogue)
constexpr int kTaGatherWarps = 16, kTaMmaWarp = 16, kTaWeightWarp = 18, kTaEpWarp0 = 20;  // MMA: 16 and 17
constexpr int kTaThreads = (kTaEpWarp0 + 4) * 32;
constexpr int kTaGatherRegs = 88, kTaIssueRegs = 48;

// Channel order of the operands (see RowBlock and the epilogue): of every 32 reduction channels, position 4 w + 2 c + e
// holds channel 16 c + 2 w + e (c < 2); within a block of N output channels, position 8 g + 2 u + e holds channel
// N / 4 * u + 2 g + e (u < 4).
__device__ __forceinline__ constexpr uint32_t k_channel(uint32_t p) {
  return (p & ~31u) + 16 * ((p >> 1) & 1u) + 2 * ((p & 31u) >> 2) + (p & 1u);
}
template <int N>
__device__ __forceinline__ constexpr uint32_t n_channel(uint32_t p) {
  return (N / 4) * ((p >> 1) & 3u) + 2 * (p >> 3) + (p & 1u);
}

// The weight image: per offset and KB-channel block, the MN-major swizzled operand image of the stage (one line of 128 or
// 64 bytes per reduction position and 64-column atom, 16-byte chunk c of line p at swz(p, c)). Where a stage has two
// offsets their lines follow one another; the second half of an odd last stage is zero. One thread per chunk.
// w has w_red <= CR and w_col <= CC channels, the rest is zero. transpose: w is [K][w_col][w_red] (input gradient);
// reverse: offset k of the image is W[K - 1 - k]. One more block turns the batch norm of `fold` into epilogue scale and shift.
template <int CC>
constexpr int ta_tiles() { return CC <= 64 ? 4 : (CC <= 128 ? 2 : 1); }

__device__ __forceinline__ void fold_batch_norm(const rmn_bn_fold& fold, uint32_t w_col, uint32_t c_col) {
  for (uint32_t c = threadIdx.x; c < c_col; c += 256) {
    auto param = [&](const void* p, float absent) {
      if (!p || c >= w_col) return absent;
      return fold.param_dtype == RMN_F32 ? static_cast<const float*>(p)[c]
                                         : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[c]);
    };
    const float s = param(fold.gamma, 1.f) / sqrtf(param(fold.var, 1.f) + fold.eps);
    fold.scale[c] = s;
    fold.shift[c] = param(fold.beta, 0.f) + (param(fold.conv_bias, 0.f) - param(fold.mean, 0.f)) * s;
  }
}
template <int CR, int CC>
__device__ __forceinline__ void image_chunk(const __nv_bfloat16* __restrict__ w, int K, uint32_t w_red, uint32_t w_col,
                                            int transpose, int reverse, uint4* __restrict__ image, uint32_t i) {
  using C = TaCfg<CR, CC, ta_tiles<CC>()>;
  constexpr int KB = C::KB, NBLK = CC < 64 ? CC : 64, CPL = NBLK / 8, CHUNKS = KB * CC / 8;
  if (i >= (uint32_t)((K + C::OPS - 1) / C::OPS) * C::NKB * CHUNKS) return;
  const uint32_t stage = i / CHUNKS, r = i % CHUNKS;
  const uint32_t atom = r / (KB * CPL), p = (r / CPL) % KB, c = r % CPL;
  const uint32_t ci = k_channel(C::OPS > 1 ? p % CR : stage % C::NKB * KB + p);
  const int k = (int)(C::OPS > 1 ? stage * C::OPS + p / CR : stage / C::NKB);
  const __nv_bfloat16* wk = w + (size_t)(reverse ? K - 1 - k : k) * w_red * w_col;
  uint32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint16_t e[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t co = atom * NBLK + n_channel<NBLK>(c * 8 + q * 2 + h);
      e[h] = k >= K || ci >= w_red || co >= w_col
                 ? (uint16_t)0
                 : *reinterpret_cast<const uint16_t*>(wk + (transpose ? (size_t)co * w_red + ci : (size_t)ci * w_col + co));
    }
    v[q] = e[0] | ((uint32_t)e[1] << 16);
  }
  image[stage * CHUNKS + atom * (KB * CPL) + p * CPL + swz<NBLK * 2>(p, c)] = make_uint4(v[0], v[1], v[2], v[3]);
}

template <int CR, int CC>
__global__ void __launch_bounds__(256) k_weight_image(const __nv_bfloat16* __restrict__ w, int K, uint32_t w_red,
                                                      uint32_t w_col, int transpose, int reverse, rmn_bn_fold fold,
                                                      uint4* __restrict__ image) {
  after_previous_kernel();
  if (fold.scale && blockIdx.x == gridDim.x - 1) return fold_batch_norm(fold, w_col, CC);
  image_chunk<CR, CC>(w, K, w_red, w_col, transpose, reverse, image, blockIdx.x * 256 + threadIdx.x);
}

// The 32 rows of a gather warp on their way from global to tensor memory: 64 channels of one row each, or the 32 channels
// of two (OPS = 2, idx2: the rows of the second offset). Two lanes share a row of each half of 16 (lane t: row
// t / 4 + 8 (t & 1), 32-byte piece t / 2 & 1 of every 64 bytes). The registers are loaded in the order tcgen05.st.16x64b
// takes them in, so nothing is moved in between: a move, like a spill, of a register whose load is in flight waits for
// the load (four lanes per row and 16x256b stores would halve the pieces per row, but need the moves and three times the
// registers).
struct RowBlock {
  uint32_t v[2][16];
  template <int CR, int OPS>
  __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ src_lane, int32_t idx, int32_t idx2, int lane) {
    const int mine = (lane >> 2) + 8 * (lane & 1);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int32_t row = __shfl_sync(0xFFFFFFFFu, idx, h * 16 + mine);
      const __nv_bfloat16* p = src_lane + (size_t)(uint32_t)row * CR;
      ldg32_or_zero<0>(p, row >= 0, v[h]);
      if constexpr (OPS == 1) {
        ldg32_or_zero<8>(p + 32, row >= 0, v[h]);
      } else {
        const int32_t row2 = __shfl_sync(0xFFFFFFFFu, idx2, h * 16 + mine);
        ldg32_or_zero<8>(src_lane + (size_t)(uint32_t)row2 * CR, row2 >= 0, v[h]);
      }
    }
  }
  __device__ __forceinline__ void store(uint32_t taddr) const {
    tc_st16x64b(taddr, v[0]);
    tc_st16x64b(taddr + (16u << 16), v[1]);
  }
};

// kPlan: the rows are processed in the internal order of a convolution plan (rmn_plan.cu): `nbr` is the plan's permuted
// table [K][n_dst] (n_dst = the padded position count), `perm` maps a position to the output row it is stored to (-1:
// padding) and `tile_mask` holds, per 128-row tile, the offsets at which any row of the tile has a neighbour: other
// (tile, offset) pairs take no gather, no slot and no MMA, offsets that no tile of the super-tile has no copy of W[k].
// Without a plan `perm` may be the order of an ordered map (rmn_kmap_build_ordered), or NULL.
// kStats: the epilogue also accumulates, per output channel, the sum and the sum of squares of the values it stores
// and writes them to stats_partial[blockIdx.x][2][CC].
// The columns [CC * blockIdx.y, CC * (blockIdx.y + 1)) of n_cols are computed.
template <int CR, int CC, int T_, bool kStats, bool kPlan>
__global__ void __launch_bounds__(kTaThreads, 1)
    k_conv_ta(const __nv_bfloat16* __restrict__ src, const uint8_t* __restrict__ image, const int32_t* __restrict__ nbr,
              uint32_t n_dst, int K, __nv_bfloat16* __restrict__ out, uint32_t n_super, const float* __restrict__ ep_scale,
              const float* __restrict__ ep_shift, const __nv_bfloat16* __restrict__ ep_add, int ep_relu, uint32_t n_cols, float* __restrict__ stats_partial,
              const int32_t* __restrict__ perm, const uint32_t* __restrict__ tile_mask) {
  using C = TaCfg<CR, CC, T_>;
  constexpr int KB = C::KB, NKB = C::NKB, OPS = C::OPS, T = C::T, G = C::GROUPS, PH = C::PHASES, SLOTS = C::SLOTS, BST = C::B_STAGES;
  constexpr int NI = C::ISSUERS, SPLIT = C::SPLIT, NT = T > 1 ? T / NI : 1;  // NT: tiles of an issuer
  constexpr int KSTEP = PH > NKB ? PH / NKB : 1;  // every KSTEP-th offset belongs to one group of a tile ...
  constexpr int NB = NKB > PH ? NKB / PH : 1;     // ... with NB of its channel blocks, PH apart
  constexpr int NBLK = CC < 64 ? CC : 64;         // columns of one atom
  constexpr int SWB = NBLK * 2;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* b_full = reinterpret_cast<uint64_t*>(smem + C::BAR_OFFSET);
  uint64_t* b_empty = b_full + BST;
  uint64_t* a_full = b_empty + BST;                  // [group][slot]
  uint64_t* a_empty = a_full + G * SLOTS;            // [group][slot]
  uint64_t* acc_full = a_empty + G * SLOTS;          // [buffer][tile]
  uint64_t* acc_empty = acc_full + C::ACC_BUFS * T;  // [buffer][tile]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + C::ACC_BUFS * T);
  float* s_ep = reinterpret_cast<float*>(smem + C::EP_OFFSET);  // per-channel scale | shift
  static_assert(KSTEP <= 2 || !kPlan, "planned tiles count their offsets modulo 2");
  const uint32_t col0 = blockIdx.y * CC;
  const int n_off = (K + OPS - 1) / OPS;  // offsets, or pairs of them
  const bool has_ep = ep_scale != nullptr || ep_shift != nullptr || ep_add != nullptr || ep_relu != 0;

  // (the shuffle makes the warp number uniform for the compiler, too: with tid >> 5 the MMA warp's loop leaves the uniform
  // datapath, 919 -> 1005 us in a pass of thirty small layers)
  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < BST; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], NI / SPLIT);
    }
    for (int s = 0; s < G * SLOTS; ++s) {
      mbar_init(&a_full[s], 4);
      mbar_init(&a_empty[s], 1);
    }
    for (int a = 0; a < C::ACC_BUFS * T; ++a) {
      mbar_init(&acc_full[a], SPLIT);
      mbar_init(&acc_empty[a], 128);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  // (tensor memory is taken behind the kernels before this one and ahead of the next: see release_next_kernel)
  wait_previous_kernels();
  if (warp == kTaMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (has_ep && tid < CC) {
    s_ep[tid] = ep_scale ? __ldg(ep_scale + col0 + tid) : 1.f;
    s_ep[CC + tid] = ep_shift ? __ldg(ep_shift + col0 + tid) : 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  release_next_kernel();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const uint32_t smem_base = smem_u32(smem);
  bool timed_out = false;

  if (warp < kTaGatherWarps) {
    // ------------------------------ gather ---------------------------------------------
    // Stages of a tile are its (offset, channel block) pairs in order; group g takes every PH-th one from g / T on. A warp
    // fills the 32 lanes of tensor memory it may access with its 32 rows of the tile.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTaGatherRegs));
    const int g = warp >> 2, t = g % T, k_first = (g / T) / NKB * OPS;
    const __nv_bfloat16* src_lane = src + ((g / T) % NKB) * KB + ((lane >> 1) & 1) * 16;
    const uint32_t a_base = tmem_base + C::ACC_COLS + g * SLOTS * C::A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t bars = smem_u32(a_full + g * SLOTS);  // full barriers; the empty ones lie G * SLOTS further

    // Cursor over the table entries of this lane's rows (OPS = 2: `second` goes with the entry returned); kEnd behind the
    // last one
    constexpr int32_t kEnd = INT32_MIN;
    uint32_t st = blockIdx.x, todo = 0;
    int k = K, kb = NB - 1;
    const int32_t* entry = nbr;
    bool row_ok = false, fresh = true;
    int32_t last = -1, second = -1;
    auto next = [&]() -> int32_t {
      if constexpr (NB > 1) {
        if (++kb < NB) return last;
        kb = 0;
      }
      for (;;) {
        if constexpr (kPlan) {
          if (todo) {
            const int kk = __ffs(todo) - 1;
#pragma unroll
            for (int i = 0; i < KSTEP; ++i) todo &= todo - 1u;
            last = row_ok ? __ldg(entry + (size_t)kk * n_dst) : -1;
            return last;
          }
        } else {
          if (k < K) {
            last = row_ok ? __ldg(entry) : -1;
            if constexpr (OPS == 2) second = row_ok && k + 1 < K ? __ldg(entry + n_dst) : -1;
            entry += (size_t)(KSTEP * OPS) * n_dst;
            k += KSTEP * OPS;
            return last;
          }
        }
        if (!fresh) st += gridDim.x;
        fresh = false;
        if (st >= n_super) {
          last = kEnd;
          fresh = true;  // stay here
          return kEnd;
        }
        const uint32_t row = st * (kTileM * T) + t * kTileM + (warp & 3) * 32 + lane;
        row_ok = row < n_dst;
        if constexpr (kPlan) {
          entry = nbr + row;
          todo = __ldg(tile_mask + (size_t)st * T + t);
#pragma unroll
          for (int i = 0; i < KSTEP - 1; ++i)
            if (i < k_first) todo &= todo - 1u;
        } else {
          k = k_first;
          entry = nbr + (size_t)k_first * n_dst + row;
        }
      }
    };
    // Table entries are fetched four stages ahead of their use, rows two: two row blocks live in registers, each loaded
    // again as soon as it has been stored. (The windows are unrolled by hand: a rotating window would copy registers
    // whose loads are in flight, and a copy waits for its source. A spilled register of a block does the same: 80
    // registers were 3 times slower.)
    uint32_t cnt = 0;
    RowBlock b0, b1;
    auto load = [&](RowBlock& b, int32_t idx, int32_t idx2, int block) {
      b.template load<CR, OPS>(src_lane + (NB > 1 ? block * PH * KB : 0), idx, idx2, lane);
    };
    auto arrive = [&]() {  // the block stored last has reached tensor memory
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + ((cnt - 1u) % SLOTS) * 8);
    };
    auto put = [&](const RowBlock& b) {
      if (cnt) arrive();
      const uint32_t s = cnt % SLOTS, ph = (cnt / SLOTS) & 1u;
      ++cnt;
      if (!mbar_wait(bars + (G * SLOTS + s) * 8, ph ^ 1u)) timed_out = true;
      tc_fence_after();
      __syncwarp();
      b.store(a_base + s * C::A_COLS);
    };
    constexpr int ODD = NB > 1 ? 1 : 0;
    static_assert(NB <= 2, "the blocks of an offset alternate");
    int32_t w0, w1, w2, w3, x0 = -1, x1 = -1, x2 = -1, x3 = -1;
    w0 = next(), x0 = second;
    w1 = next(), x1 = second;
    load(b0, w0, x0, 0);
    load(b1, w1, x1, ODD);
    bool live0 = w0 != kEnd, live1 = w1 != kEnd;
    w2 = next(), x2 = second;
    w3 = next(), x3 = second;
    w0 = next(), x0 = second;
    w1 = next(), x1 = second;
    while (live0) {
      put(b0);
      load(b0, w2, x2, 0);
      live0 = w2 != kEnd;
      w2 = next(), x2 = second;
      if (!live1) break;
      put(b1);
      load(b1, w3, x3, ODD);
      live1 = w3 != kEnd;
      w3 = next(), x3 = second;
      if (!live0) break;
      put(b0);
      load(b0, w0, x0, 0);
      live0 = w0 != kEnd;
      w0 = next(), x0 = second;
      if (!live1) break;
      put(b1);
      load(b1, w1, x1, ODD);
      live1 = w1 != kEnd;
      w1 = next(), x1 = second;
      if (__any_sync(0xFFFFFFFFu, timed_out)) break;
    }
    if (cnt) arrive();
  } else if (warp < kTaEpWarp0) {
    // (one instruction for the whole warpgroup, ahead of its roles)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTaIssueRegs));
    if (warp < kTaMmaWarp + NI) {
      // ------------------------------ MMA issuer -----------------------------------------
      // The warp's tiles are t0 .. t0 + T / NI - 1. Warp-uniform code, one elected lane issues. B descriptors differ only in the
      // start address field. Masks of a plan come through a warp vote (the ballot of "bit `lane` of the mask" is the mask
      // itself), whose result is warp-uniform by construction, so that branches on it keep the loop on the uniform datapath.
      const int issuer = warp - kTaMmaWarp, t0 = SPLIT > 1 ? 0 : issuer * NT;
      constexpr uint32_t IDESC = instr_desc(kTileM, CC, true);
      constexpr uint64_t B_DESC0 = smem_desc_sw_const(KB * SWB, 8 * SWB, SWB == 128 ? 2u : 4u);
      constexpr uint32_t B_DESC_HI = (uint32_t)(B_DESC0 >> 32);
      uint32_t cnts = 0;  // stages taken from each group so far, modulo 8 (one byte per group)
      uint32_t b_it = 0, tile_iter = 0;
      for (uint32_t st = blockIdx.x; st < n_super && !timed_out; st += gridDim.x, ++tile_iter) {
        const uint32_t buf = tile_iter % C::ACC_BUFS, acc_ph = (tile_iter / C::ACC_BUFS) & 1u;
        uint32_t m[NT] = {}, todo = 0;
        if constexpr (kPlan) {
  #pragma unroll
          for (int t = 0; t < T; ++t) {
            const uint32_t v = __ballot_sync(0xFFFFFFFFu, (__ldg(tile_mask + (size_t)st * T + t) >> lane) & 1u);
            todo |= v;
  #pragma unroll
            for (int i = 0; i < NT; ++i)
              if (t == t0 + i) m[i] = v;
          }
        }
        uint32_t started = 0, odd = 0;  // per tile: an MMA has been issued; parity of its offset count
        for (int k = 0; kPlan ? todo != 0 : k < n_off; ++k) {
          if constexpr (kPlan) {
            k = __ffs(todo) - 1;
            todo &= todo - 1u;
          }
  #pragma unroll
          for (int kb = 0; kb < NKB; ++kb, ++b_it) {
            if (SPLIT > 1 && ((k * NKB + kb) & 1) != issuer) continue;
            const uint32_t bs = b_it % BST;
            if (!mbar_wait(&b_full[bs], (b_it / BST) & 1u)) { timed_out = true; goto mma_done; }
            const uint32_t b_lo = ((smem_base + bs * C::B_BYTES) >> 4) + (uint32_t)(B_DESC0 & 0xFFFFFFFFu);
  #pragma unroll
            for (int i = 0; i < NT; ++i) {
              const int t = t0 + i;
              if constexpr (kPlan) {
                if (!((m[i] >> k) & 1u)) continue;
              }
              const uint32_t g = t + T * (KSTEP > 1 ? (kPlan ? (odd >> t) & 1u : (uint32_t)k % KSTEP) * NKB + kb : kb % PH);
              const uint32_t c = (cnts >> (8 * g)) & 7u, s = c % SLOTS;
              const uint32_t begun = (started >> t) & 1u;
              if (!mbar_wait(&a_full[g * SLOTS + s], (c / SLOTS) & 1u)) { timed_out = true; goto mma_done; }
              if (!begun && !mbar_wait(&acc_empty[buf * T + t], acc_ph ^ 1u)) { timed_out = true; goto mma_done; }
              tc_fence_after();
              const uint32_t d_tmem = tmem_base + (SPLIT > 1 ? buf * 2 + issuer : buf * T + t) * CC;
              const uint32_t a_tmem = tmem_base + C::ACC_COLS + (g * SLOTS + s) * C::A_COLS;
  #pragma unroll
              for (int j = 0; j < KB / 16; ++j) {
                // MN-major B: 8-row K groups 8 * SWB apart (SBO), 64-column atoms KB * SWB apart (LBO), a K step is 16 lines
                const uint64_t b_desc = ((uint64_t)B_DESC_HI << 32) | (b_lo + (uint32_t)((j * 16 * SWB) >> 4));
                tc_mma_bf16_ta_elect(d_tmem, a_tmem + j * 8, b_desc, IDESC, j > 0 ? 1u : begun);
              }
              tc_commit_elect(&a_empty[g * SLOTS + s]);
              cnts = (cnts + (1u << (8 * g))) & 0x07070707u;
              started |= 1u << t;
              if (kPlan && KSTEP > 1 && kb == NKB - 1) odd ^= 1u << t;
            }
            tc_commit_elect(&b_empty[bs]);
          }
        }
  #pragma unroll
        for (int i = 0; i < NT; ++i) {
          const int t = t0 + i;
          if (!((started >> t) & 1u) && !mbar_wait(&acc_empty[buf * T + t], acc_ph ^ 1u)) { timed_out = true; goto mma_done; }
          tc_commit_elect(&acc_full[buf * T + t]);
        }
      }
    mma_done:;
    } else {
      // ------------------------------ weights --------------------------------------------
      if (warp == kTaWeightWarp && lane == 0) {
        uint32_t b_it = 0;
        for (uint32_t st = blockIdx.x; st < n_super && !timed_out; st += gridDim.x) {
          uint32_t todo = 0;
          if constexpr (kPlan) {
  #pragma unroll
            for (int t = 0; t < T; ++t) todo |= __ldg(tile_mask + (size_t)st * T + t);
          }
          for (int k = 0; (kPlan ? todo != 0 : k < n_off) && !timed_out; ++k) {
            if constexpr (kPlan) {
              k = __ffs(todo) - 1;
              todo &= todo - 1u;
            }
            for (int kb = 0; kb < NKB; ++kb, ++b_it) {
              const uint32_t s = b_it % BST;
              if (!mbar_wait(&b_empty[s], ((b_it / BST) & 1u) ^ 1u)) { timed_out = true; break; }
              bulk_load(smem_base + s * C::B_BYTES, image + ((size_t)(k * NKB + kb) * n_cols + col0) * (KB * 2), C::B_BYTES,
                        smem_u32(&b_full[s]));
            }
          }
        }
        // no copy may be in flight when the CTA exits: wait for the last round of the ring
        for (uint32_t i = b_it > BST ? b_it - BST : 0; i < b_it; ++i)
          if (!mbar_wait(&b_full[i % BST], (i / BST) & 1u)) timed_out = true;
      }
    }
  } else {
    // ------------------------------ epilogue -------------------------------------------
    // tcgen05.ld.16x256b and the column order of the weight image give lane t CC / 4 contiguous channels (of every
    // 64-column block) of the rows t / 4 and t / 4 + 8: four lanes store a whole 128-byte line.
    const uint32_t quad = warp & 3, u = lane & 3;
    constexpr int NW = NBLK / 8;  // words a lane stores per row and block
    float* s_st = reinterpret_cast<float*>(smem + C::STATS_OFFSET) + quad * 2 * CC;
    if constexpr (kStats) {
      for (int c = lane; c < 2 * CC; c += 32) s_st[c] = 0.f;
      __syncwarp();
    }
    uint32_t tile_iter = 0;
    for (uint32_t st = blockIdx.x; st < n_super && !timed_out; st += gridDim.x, ++tile_iter) {
      const uint32_t buf = tile_iter % C::ACC_BUFS, acc_ph = (tile_iter / C::ACC_BUFS) & 1u;
#pragma unroll 1
      for (int t = 0; t < T; ++t) {
        if (!mbar_wait(&acc_full[buf * T + t], acc_ph)) timed_out = true;
        timed_out = __any_sync(0xFFFFFFFFu, timed_out);
        if (timed_out) break;
        tc_fence_after();
        bool tile_any = true;  // false: no MMA wrote this tile's accumulator (no neighbour at any offset)
        if constexpr (kPlan) tile_any = __any_sync(0xFFFFFFFFu, __ldg(tile_mask + (size_t)st * T + t) != 0);
        uint32_t rows[4];  // output rows t / 4 + 8 i of this warp's 32
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t pos = st * (kTileM * T) + t * kTileM + quad * 32 + i * 8 + (lane >> 2);
          rows[i] = pos < n_dst ? pos : 0xFFFFFFFFu;
          if (kPlan || (perm && pos < n_dst)) rows[i] = (uint32_t)__ldg(perm + pos);  // (-1: padding of a plan)
        }
#pragma unroll 1
        for (int nb = 0; nb < CC / NBLK; ++nb) {
          const int ch = nb * NBLK + u * (NBLK / 4);  // this lane's first channel
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t taddr = tmem_base + ((quad * 32u + h * 16u) << 16) + (buf * T + t) * SPLIT * CC + nb * NBLK;
            uint32_t w0[NW], w1[NW];  // rows 2 h and 2 h + 1: first what is added to them, then the result
            if (ep_add) {
              auto fetch = [&](uint32_t row, uint32_t (&w)[NW]) {
                const uint4* a = reinterpret_cast<const uint4*>(ep_add + (size_t)row * n_cols + col0 + ch);
#pragma unroll
                for (int v = 0; v < NW / 4; ++v) {
                  const uint4 x = row != 0xFFFFFFFFu ? __ldg(a + v) : make_uint4(0u, 0u, 0u, 0u);
                  w[4 * v] = x.x, w[4 * v + 1] = x.y, w[4 * v + 2] = x.z, w[4 * v + 3] = x.w;
                }
              };
              fetch(rows[2 * h], w0);
              fetch(rows[2 * h + 1], w1);
            }
#pragma unroll
            for (int q = 0; q < NBLK / 32; ++q) {
              uint32_t r[16];
              if (tile_any) {
                tc_ld16x256b(taddr + q * 32, r);
                if (SPLIT > 1 && n_off * NKB > 1) {  // the odd stages' sum
                  uint32_t odd[16];
                  tc_ld16x256b(taddr + CC + q * 32, odd);
                  tc_wait_ld();
#pragma unroll
                  for (int v = 0; v < 16; ++v) r[v] = __float_as_uint(__uint_as_float(r[v]) + __uint_as_float(odd[v]));
                } else {
                  tc_wait_ld();
                }
              } else {
#pragma unroll
                for (int v = 0; v < 16; ++v) r[v] = 0u;
              }
#pragma unroll
              for (int gg = 0; gg < 4; ++gg) {
                float f[4] = {__uint_as_float(r[4 * gg]), __uint_as_float(r[4 * gg + 1]), __uint_as_float(r[4 * gg + 2]),
                              __uint_as_float(r[4 * gg + 3])};
                if (has_ep) {
                  const int c = ch + 2 * (q * 4 + gg);
                  const float2 sc = *reinterpret_cast<const float2*>(s_ep + c);
                  const float2 sh = *reinterpret_cast<const float2*>(s_ep + CC + c);
                  f[0] = fmaf(f[0], sc.x, sh.x);
                  f[1] = fmaf(f[1], sc.y, sh.y);
                  f[2] = fmaf(f[2], sc.x, sh.x);
                  f[3] = fmaf(f[3], sc.y, sh.y);
                  if (ep_add) {
                    const float2 a0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w0[q * 4 + gg]));
                    const float2 a1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w1[q * 4 + gg]));
                    f[0] += a0.x, f[1] += a0.y, f[2] += a1.x, f[3] += a1.y;
                  }
                  if (ep_relu) {
#pragma unroll
                    for (int v = 0; v < 4; ++v) f[v] = relu_f32(f[v]);
                  }
                }
                const __nv_bfloat162 p0 = __floats2bfloat162_rn(f[0], f[1]), p1 = __floats2bfloat162_rn(f[2], f[3]);
                w0[q * 4 + gg] = *reinterpret_cast<const uint32_t*>(&p0);
                w1[q * 4 + gg] = *reinterpret_cast<const uint32_t*>(&p1);
              }
            }
            if (rows[2 * h] != 0xFFFFFFFFu) {
              uint4* d = reinterpret_cast<uint4*>(out + (size_t)rows[2 * h] * n_cols + col0 + ch);
#pragma unroll
              for (int v = 0; v < NW / 4; ++v) d[v] = make_uint4(w0[4 * v], w0[4 * v + 1], w0[4 * v + 2], w0[4 * v + 3]);
            }
            if (rows[2 * h + 1] != 0xFFFFFFFFu) {
              uint4* d = reinterpret_cast<uint4*>(out + (size_t)rows[2 * h + 1] * n_cols + col0 + ch);
#pragma unroll
              for (int v = 0; v < NW / 4; ++v) d[v] = make_uint4(w1[4 * v], w1[4 * v + 1], w1[4 * v + 2], w1[4 * v + 3]);
            }
            if constexpr (kStats) {
              // statistics of the values as stored (rounded to bf16), over the eight lanes that hold the same channels
              const float l0 = rows[2 * h] != 0xFFFFFFFFu ? 1.f : 0.f, l1 = rows[2 * h + 1] != 0xFFFFFFFFu ? 1.f : 0.f;
#pragma unroll
              for (int v = 0; v < NW; ++v) {
                const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w0[v]));
                const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w1[v]));
                float sum[4] = {l0 * a.x + l1 * b.x, l0 * a.y + l1 * b.y, l0 * a.x * a.x + l1 * b.x * b.x,
                                l0 * a.y * a.y + l1 * b.y * b.y};
#pragma unroll
                for (int d = 4; d < 32; d <<= 1)
#pragma unroll
                  for (int x = 0; x < 4; ++x) sum[x] += __shfl_xor_sync(0xFFFFFFFFu, sum[x], d);
                if (lane < 4) {
                  s_st[ch + 2 * v] += sum[0];
                  s_st[ch + 2 * v + 1] += sum[1];
                  s_st[CC + ch + 2 * v] += sum[2];
                  s_st[CC + ch + 2 * v + 1] += sum[3];
                }
              }
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&acc_empty[buf * T + t]);
      }
    }
    if constexpr (kStats) {
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the four epilogue warps, added in warp order
      const float* all = reinterpret_cast<const float*>(smem + C::STATS_OFFSET);
      for (int c = (int)(quad * 32) + lane; c < 2 * CC; c += 128)
        stats_partial[((size_t)blockIdx.x * 2 + c / CC) * n_cols + col0 + c % CC] = all[c] + all[2 * CC + c] + all[4 * CC + c] + all[6 * CC + c];
    }
  }

  if (timed_out) atomicExch(&g_tc_status, (uint32_t)RMN_ERR_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  if (warp == kTaMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

// grid_out receives the number of CTAs, i.e. of [2][CC] partials written to stats_partial.
template <int CR, int CC, int T, bool kStats, bool kPlan>
int launch_ta(const void* src, const void* image, const int32_t* nbr, uint32_t n_dst, int K, void* out, const float* ep_scale,
              const float* ep_shift, const void* ep_add, int ep_relu, uint32_t n_cols, int sms, cudaStream_t stream, float* stats_partial,
              uint32_t* grid_out, const void* plan, const int32_t* order) {
  using C = TaCfg<CR, CC, T>;
  auto kern = k_conv_ta<CR, CC, T, kStats, kPlan>;
  const int32_t* perm = order;
  const uint32_t* tile_mask = nullptr;
  if constexpr (kPlan) {
    const PlanLayout L = plan_layout(n_dst, K);
    const char* base = static_cast<const char*>(plan);
    perm = reinterpret_cast<const int32_t*>(base + L.perm);
    tile_mask = reinterpret_cast<const uint32_t*>(base + L.tile_mask);
    nbr = reinterpret_cast<const int32_t*>(base + L.nbr_p);
    n_dst = L.n_pos;  // positions, a multiple of every super-tile size
  }
  static SmemOptIn opt_in;
  RMN_CUDA_TRY(opt_in.apply(reinterpret_cast<const void*>(kern), C::SMEM));
  const uint32_t n_super = (n_dst + kTileM * C::T - 1) / (kTileM * C::T);
  const uint32_t n_blocks = n_cols / CC, fit = (uint32_t)sms > n_blocks ? (uint32_t)sms / n_blocks : 1u;
  const uint32_t grid = fit < n_super ? fit : n_super;  // one CTA per SM owns its tensor memory
  RMN_CUDA_TRY(launch_overlapped(kern, dim3(grid, n_blocks), dim3(kTaThreads), C::SMEM, stream, (const __nv_bfloat16*)src,
                                 (const uint8_t*)image, nbr, n_dst, K, (__nv_bfloat16*)out, n_super, ep_scale, ep_shift,
                                 (const __nv_bfloat16*)ep_add, ep_relu, n_cols, stats_partial, perm, tile_mask));
  RMN_LAUNCH_CHECK();
  count_tc_launch();
  if (grid_out) *grid_out = grid;
  return RMN_OK;
}

// K rounded up to whole stages, times the bytes of one offset's weights
template <int CR, int CC>
size_t image_bytes(int K) {
  using C = TaCfg<CR, CC, ta_tiles<CC>()>;
  return (size_t)((K + C::OPS - 1) / C::OPS) * C::NKB * C::B_BYTES;
}

template <int CR, int CC>
int launch_image(const void* w, int K, int w_red, int w_col, int transpose, int reverse, const rmn_bn_fold& fold, void* image,
                 cudaStream_t stream) {
  const uint32_t chunks = (uint32_t)(image_bytes<CR, CC>(K) / 16);
  RMN_CUDA_TRY(launch_overlapped(k_weight_image<CR, CC>, dim3((chunks + 255) / 256 + (fold.scale ? 1 : 0)), dim3(256), 0,
                                 stream, (const __nv_bfloat16*)w, K, (uint32_t)w_red, (uint32_t)w_col, transpose, reverse, fold,
                                 (uint4*)image));
  RMN_LAUNCH_CHECK();
  return RMN_OK;
}

}  // namespace tc

#define RMN_TA_SHAPES(CASE) \
  CASE(32, 32) CASE(32, 64) CASE(64, 32) CASE(64, 64) CASE(64, 128) CASE(128, 64) CASE(128, 128) CASE(128, 256) CASE(256, 128) CASE(256, 256)

size_t ta_image_bytes(int K, int c_red, int c_col);

// The images of up to kImageJobs layers in one launch: what one of them costs a network of small layers is the launch between two
// convolutions (3 to 4 us each: 113 us of a network of thirty layers, 24 like this; the pass, which the host bounds, 877 to 866).
constexpr int kImageJobs = 24;
struct ImageJobs {
  int n;
  uint32_t first[kImageJobs + 1];  // block range of every job; its last block folds the batch norm, if there is one
  rmn_weight_job job[kImageJobs];
};
__global__ void __launch_bounds__(256) k_weight_images(const __grid_constant__ ImageJobs jobs) {
  after_previous_kernel();
  int j = 0;
  while (blockIdx.x >= jobs.first[j + 1]) ++j;
  const rmn_weight_job& job = jobs.job[j];
  if (job.fold.scale && blockIdx.x + 1 == jobs.first[j + 1]) return tc::fold_batch_norm(job.fold, (uint32_t)job.w_out, (uint32_t)job.c_out);
  const uint32_t i = (blockIdx.x - jobs.first[j]) * 256 + threadIdx.x;
#define RMN_TA_CASE(R, Cc)                                                                                             \
  if (job.c_in == R && job.c_out == Cc)                                                                                \
    return tc::image_chunk<R, Cc>(static_cast<const __nv_bfloat16*>(job.weights), job.K, (uint32_t)job.w_in,           \
                                  (uint32_t)job.w_out, 0, 0, static_cast<uint4*>(job.image), i);
  RMN_TA_SHAPES(RMN_TA_CASE)
#undef RMN_TA_CASE
}

int ta_weight_images(const rmn_weight_job* jobs, int n_jobs, cudaStream_t stream) {
  for (int done = 0; done < n_jobs; done += kImageJobs) {
    ImageJobs a = {};
    a.n = n_jobs - done < kImageJobs ? n_jobs - done : kImageJobs;
    for (int j = 0; j < a.n; ++j) {
      a.job[j] = jobs[done + j];
      const size_t chunks = ta_image_bytes(a.job[j].K, a.job[j].c_in, a.job[j].c_out) / 16;
      a.first[j + 1] = a.first[j] + (uint32_t)((chunks + 255) / 256) + (a.job[j].fold.scale ? 1u : 0u);
    }
    RMN_CUDA_TRY(launch_overlapped(k_weight_images, dim3(a.first[a.n]), dim3(256), 0, stream, a));
    RMN_LAUNCH_CHECK();
  }
  return RMN_OK;
}

constexpr int kPlanMinWeight = 128 * 128;

// 0: no kernel for these channel counts
size_t ta_image_bytes(int K, int c_red, int c_col) {
#define RMN_TA_CASE(R, Cc) if (c_red == R && c_col == Cc) return tc::image_bytes<R, Cc>(K);
  RMN_TA_SHAPES(RMN_TA_CASE)
#undef RMN_TA_CASE
  return 0;
}

// image of c_red x c_col products of [K][w_red][w_col] weights (transpose: given as [K][w_col][w_red])
int ta_weight_image(const void* w, int K, int w_red, int w_col, int c_red, int c_col, int transpose, int reverse,
                    const rmn_bn_fold& fold, void* image, cudaStream_t stream) {
#define RMN_TA_CASE(R, Cc) \
  if (c_red == R && c_col == Cc) return tc::launch_image<R, Cc>(w, K, w_red, w_col, transpose, reverse, fold, image, stream);
  RMN_TA_SHAPES(RMN_TA_CASE)
#undef RMN_TA_CASE
  return RMN_ERR_UNSUPPORTED;
}

// Whether to run single row tiles and 64-column blocks, not super-tiles of all columns. Super-tiles share a copy of W[k] and
// a gathered row among all columns, but few of them leave SMs idle: the time goes with the tiles of the busiest SM, a
// tile on its own costing about 30 % more, and one of more than 128 columns 60 % more than one of 64.
bool ta_small(uint32_t n_dst, int c_col, int sms) {
  const uint32_t tiles = (n_dst + tc::kTileM - 1) / tc::kTileM, t = c_col <= 64 ? 4u : c_col <= 128 ? 2u : 1u;
  const uint32_t blocks = c_col <= 64 ? 1u : (uint32_t)c_col / 64, fit = (uint32_t)sms > blocks ? (uint32_t)sms / blocks : 1u;
  const uint32_t supers = (tiles + t - 1) / t;
  const uint32_t whole = (supers + sms - 1) / sms * t * (c_col > 128 ? 16u : 10u), single = (tiles + fit - 1) / fit * 13u;
  return single < whole;
}

// stats_partial != nullptr: also leave per-CTA channel statistics ([*n_partials][2][c_col] floats)
int ta_conv(const void* src, const void* image, const int32_t* nbr, uint32_t n_dst, int K, int c_red, int c_col, void* out,
            const float* ep_scale, const float* ep_shift, const void* ep_add, int ep_relu, float* stats_partial, uint32_t* n_partials,
            cudaStream_t stream, const void* plan, const int32_t* order) {
  if (ta_image_bytes(K, c_red, c_col) == 0) return RMN_ERR_UNSUPPORTED;  // (the cases below match blocks of columns)
  int dev = 0, sms = 148;
  RMN_CUDA_TRY(cudaGetDevice(&dev));
  RMN_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
#define RMN_TA_ARGS \
  src, image, nbr, n_dst, K, out, ep_scale, ep_shift, ep_add, ep_relu, (uint32_t)c_col, sms, stream, stats_partial, n_partials, plan, order
  if (ta_small(n_dst, c_col, sms)) {
    plan = nullptr;
#define RMN_TA_CASE(R, Cc)                                                                   \
  if (c_red == R && (Cc == 32 ? c_col == 32 : c_col != 32))                                  \
    return stats_partial ? tc::launch_ta<R, Cc, 1, true, false>(RMN_TA_ARGS)                 \
                         : tc::launch_ta<R, Cc, 1, false, false>(RMN_TA_ARGS);
    RMN_TA_CASE(32, 32) RMN_TA_CASE(32, 64) RMN_TA_CASE(64, 32) RMN_TA_CASE(64, 64) RMN_TA_CASE(128, 64) RMN_TA_CASE(256, 64)
#undef RMN_TA_CASE
  }
  // A plan pays where a skipped tile saves more MMA time than the gather of its rows takes anyway: from 128 x 128 channels
  // on (1.2 M rows: 128->128 716 -> 645 us, but 64->64 281 -> 288, 32->64 221 -> 249). The rows come out the same.
#define RMN_TA_CASE(R, Cc)                                                                       \
  if (c_red == R && c_col == Cc) {                                                               \
    constexpr int T = tc::ta_tiles<Cc>();                                                        \
    if constexpr (R * Cc >= kPlanMinWeight) {                                                    \
      if (plan && K <= kPlanMaxK)                                                                \
        return stats_partial ? tc::launch_ta<R, Cc, T, true, true>(RMN_TA_ARGS)                  \
                             : tc::launch_ta<R, Cc, T, false, true>(RMN_TA_ARGS);                \
    }                                                                                            \
    return stats_partial ? tc::launch_ta<R, Cc, T, true, false>(RMN_TA_ARGS)                     \
                         : tc::launch_ta<R, Cc, T, false, false>(RMN_TA_ARGS);                   \
  }
  RMN_TA_SHAPES(RMN_TA_CASE)
#undef RMN_TA_CASE
#undef RMN_TA_ARGS
  return RMN_ERR_UNSUPPORTED;
}

}  // namespace rmn
