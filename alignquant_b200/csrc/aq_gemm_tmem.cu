// Mixed W4/W8 x A8 GEMM for large row counts on the Blackwell tensor cores (sm_100a).
//
// A streaming pass (expand_kernel) widens the weights to int8 in the workspace, in the operand
// layout of the MMA; then one persistent CTA per SM computes 128-row x (64 TN)-column output tiles
// and walks K in stages of two 64-wide steps through a shared-memory ring.  Every 64 x 64 weight tile
// has its own scale, so no integer sum may span two K64 tiles (alignquant/kernels/cuda/linear.cu:951-963):
// every int32 result leaves tensor memory, is converted and added to an FP32 register with one fused
// multiply-add.  That drain, not the tensor pipe, bounds the kernel.
//
// What a drain costs (measured with resident operands, cycles per SM for the 128 x 256 results of
// one K64 step, from event times at a nominal 1.92 GHz: good to some per cent): the arithmetic alone 375 (one I2F
// and half a packed FMA per result, i.e. 1.5 issue slots, or 384 cycles), with its tensor-memory loads 590 (a load
// occupies the register file's write port as arithmetic does), with barriers and MMAs 680-750, the tensor pipe
// 248.  This kernel: 850 (16384 x 19456 x 2560 with quantizer and expansion 1.15 POPS; the version before it, which
// widened W4 tiles inside the GEMM and drained with eight warps, 0.67).  What brought it there:
//   * sixteen drain warps, four per scheduler, each owning 32 rows x 16 TN columns: a warp that
//     waits for a barrier or a tensor-memory load leaves its scheduler to three others (eight
//     warps with twice the columns: 1040-1090 cycles per step);
//   * a hand-over covers 192 or 256 accumulator columns: one K step of a wide tile or two of a
//     128-column one; every hand-over costs each warp some forty instructions;
//   * barriers are polled by whole warps and arrived on by one predicated lane.  Polling with one
//     lane and a shuffle costs 2.5 times as much (436 against 178 cycles per step for the bare
//     hand-over), a branch around the arrival 80 cycles per step;
//   * the loop's registers: sums, loaded columns and little else (scales come from a ring in shared
//     memory).  The 128- and 192-column kernels spill nothing, the 256-column one some 90 bytes; an instantiation of it
//     without the output transform spills 68 and is slower (16384 x 19456 x 2560 1381 -> 1446 us);
//   * no work for single warps: next to sixteen busy warps an ordinary instruction of a single warp
//     takes 5 to 10 cycles, so a warp that issues copies or widens tiles step by step falls behind
//     the drain.  Hence two copies per stage and the expansion in a pass of its own.
//
// Roles of the 20 warps:
//   * warps 0-15 drain (tensor-memory lane quarter = warp % 4, column group = warp / 4) and store
//     finished tiles through tensor-map copies;
//   * warp 16 issues tcgen05.mma kind::i8 (M=128, N=64 TN, K=32, twice per step) into one of two
//     256-column accumulators and commits to mbarriers (stage free, accumulator full);
//   * warp 17 streams the operands -- activations with a tensor-map copy (64-byte swizzle, rows past
//     M read as zero), expanded weights with one bulk copy per stage -- and lays down the scales;
//   * warps 18-19 only make up the warpgroup whose registers the drain takes.
// The roles meet only in mbarriers, so copies and MMAs of the next output tile run while the
// finished one is stored.
//
// Few output tiles leave SMs idle; their K range is then split over a thread-block cluster (one
// output tile per cluster, at most eight CTAs) and the FP32 partial tiles meet in distributed
// shared memory, added in split order.
//
// Every mbarrier wait is bounded; on a time-out the CTA raises a device status word
// (read by aq_device_status), stops issuing, gives copies in flight time to land,
// frees its tensor memory and returns.
#include <cooperative_groups.h>
#include <cuda.h>

#include <mutex>

#include "aq_common.cuh"
#include "aq_ptx.cuh"
#include "aq_tile_math.cuh"
#include "aq_tcgen05.cuh"

namespace cg = cooperative_groups;

namespace aq {

__device__ int g_gemm_status = 0;

namespace {

constexpr int kBM = 128;
constexpr int kABytes = kBM * kTile;  // 8192
constexpr int kMaxNk = 512;
constexpr int kDrainWarps = 16;
constexpr int kMmaWarp = 16;
constexpr int kCopyWarp = 17;
constexpr int kThreads = 20 * 32;
constexpr int kAccs = 2;
constexpr int kAccColumns = 256;
constexpr int kTmemColumns = kAccs * kAccColumns;
constexpr int kScaleSlots = 16;     // K steps whose scales are kept: more than the copies can be ahead of the drain
constexpr int kScaleRow = 12;       // floats per step: TN <= 4 weight scales, then eight activation scales (tile mode)
constexpr int kTurnRows = 15;       // rows a drain warp turns through shared memory at a time (output transform)
constexpr int kTurnFloats = 65;     // floats per turned row
constexpr int kTurnBytes = 4096;    // shared memory in which a drain warp turns its results

// TN = weight tile rows (64 columns each) of the CTA tile.  A stage of the ring holds two K steps:
// the activation blocks of both, then the weight tiles of both.
template <int TN>
struct Layout {
  static constexpr int kCols = TN * kTile;
  static constexpr int kBBytes = TN * kW8TileBytes;      // weight operand of a K step
  static constexpr int kStageBytes = 2 * (kABytes + kBBytes);  // a multiple of the 1024-byte operand alignment
  static constexpr int kStages = TN == 4 ? 3 : 4;        // 144, 160 or 128 KiB
  static constexpr int kSub = TN == 2 ? 2 : 1;           // K steps per hand-over of an accumulator
  static constexpr int kWarpCols = kCols / 4;            // columns of a drain warp
  // Registers: the block is launched with 96 per thread; the 64 sums and 32 loaded columns of a
  // TN = 4 drain thread take what the other four warps can spare.
  static constexpr int kDrainRegs = TN == 4 ? 112 : 104;
  static constexpr int kOtherRegs = TN == 4 ? 32 : 64;
  static_assert(kDrainWarps * 32 * kDrainRegs + (kThreads - kDrainWarps * 32) * kOtherRegs <= kThreads * 96,
                "setmaxnreg would wait for registers that the block does not have");
  // ready[S], empty[S], acc_full[kAccs], acc_empty[kAccs], final
  static constexpr int kNumBars = 2 * kStages + 2 * kAccs + 1;
  static constexpr int kScaleBytes = kScaleSlots * kScaleRow * 4;
  static constexpr int kSmemBytes = kStages * kStageBytes + kDrainWarps * kTurnBytes + kScaleBytes + kNumBars * 8 + 16;
  // a stage is refilled once its MMAs are done, and at most 2 kSub steps wait for the drain behind it
  static_assert(2 * kStages + 2 * kSub <= kScaleSlots, "a scale must outlive its step");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of a CTA");
  static_assert(kBM * (kCols + 1) * 4 <= kStages * kStageBytes, "the split-K exchange tile must fit into the ring");
};

struct GemmParams {
  const float* act_scales;
  const TileRecord* records;
  const uint8_t* operand;  // expanded weights of tile rows j_base ..
  const int32_t* u_metadata;
  void* out;
  int32_t* acc_dump;
  int64_t m;
  int n_j;
  int n_k;
  int j_base;  // first tile row of this launch
  int scale_mode;
  int out_dtype;
  int m_blocks;
  int n_blocks;
  int n_j_total;       // tile rows of the layer (n_j: end of this launch's range)
  int64_t row_stride;  // output values per row
  uint32_t band_magic;  // 2^32 / (16 n_blocks), rounded down
};

// Output tile `t` -> (row block, column block).  Tiles are numbered through bands of 16 row
// blocks, column blocks slowest: CTAs that run at the same time share a few weight strips and a
// few activation blocks, which is what the L2 has to deliver.
__device__ __forceinline__ void tile_position(const GemmParams& p, int t, int& mb, int& nb) {
  const uint32_t band_tiles = static_cast<uint32_t>(p.n_blocks) * 16u;
  uint32_t band = __umulhi(static_cast<uint32_t>(t), p.band_magic);  // t / band_tiles or one less
  uint32_t in_band = static_cast<uint32_t>(t) - band * band_tiles;
  if (in_band >= band_tiles) {
    in_band -= band_tiles;
    ++band;
  }
  const uint32_t rows = static_cast<uint32_t>(p.m_blocks) - band * 16u;
  if (rows >= 16u) {
    nb = static_cast<int>(in_band >> 4);
    mb = static_cast<int>(band * 16u + (in_band & 15u));
  } else {
    nb = static_cast<int>(in_band / rows);
    mb = static_cast<int>(band * 16u + in_band % rows);
  }
}

// A position in a ring of barriers: slot and the parity of its current phase.
template <int kSlots>
struct RingPosition {
  int slot = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ void advance() {
    if (++slot == kSlots) {
      slot = 0;
      parity ^= 1u;
    }
  }
};

// kCount results: acc pairs += float(v) * scale, multiply and add rounded separately (operation
// order of linear.cu:958-962); the two sums of a pair are added with one packed instruction.  kFused:
// acc = fma(float(v), scale, acc), one rounding per tile, two sums per instruction.
template <bool kFused, int kCount>
__device__ __forceinline__ void drain(uint64_t* acc, const int* v, float scale) {
  const uint64_t scale2 = pack2(__float_as_uint(scale), __float_as_uint(scale));
#pragma unroll
  for (int i = 0; i < kCount / 2; ++i) {
    if (kFused) {
      const uint64_t f = pack2(__float_as_uint(__int2float_rn(v[2 * i])), __float_as_uint(__int2float_rn(v[2 * i + 1])));
      acc[i] = fma2(f, scale2, acc[i]);
    } else {
      const float p0 = __fmul_rn(__int2float_rn(v[2 * i]), scale);
      const float p1 = __fmul_rn(__int2float_rn(v[2 * i + 1]), scale);
      acc[i] = add2(acc[i], pack2(__float_as_uint(p0), __float_as_uint(p1)));
    }
  }
}

// kCount consecutive FP32 sums (packed pairs) of one row per lane -> 32 rows of the result from row0
// on, through the warp's turning buffer and tensor-map stores: lanes lay their rows down in the
// map's swizzle and one lane hands the block over, so that neither rows past M nor the stores
// themselves hold the warp up.  (Storing from registers, 16 bytes per lane, touches 32 lines per
// instruction: 4 us per 256-column output tile; whole line segments through shared memory: 1.7 us.)
template <int kCount>
__device__ __forceinline__ void store_rows(const CUtensorMap* map, int dtype, uint8_t* region, int row0, int col0, int cols, int lane,
                                           const uint64_t* acc) {
  const uint32_t dst = smem_u32(region);
  auto room = [&]() {  // the buffer's previous block has left it
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
  };
  auto hand_over = [&](int col, uint32_t from) {
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) tensor_store_2d(map, col, row0, from);
  };
  if constexpr (kCount == 48) {  // three blocks of 16 columns without a swizzle
    const bool f32 = dtype == AQ_F32, bf16 = dtype == AQ_BF16;
    if (!f32) room();
#pragma unroll
    for (int h = 0; h < 3; ++h) {
      if (f32) room();  // a block of floats is 2 KiB
      const int block = f32 ? 0 : h * 1024;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint64_t x = acc[h * 8 + 2 * i], y = acc[h * 8 + 2 * i + 1];
        if (f32) {
          reinterpret_cast<uint4*>(region + lane * 64)[i] = make_uint4(static_cast<uint32_t>(x), static_cast<uint32_t>(x >> 32),
                                                                       static_cast<uint32_t>(y), static_cast<uint32_t>(y >> 32));
        } else {
          float a, b, c, d;
          unpack2(x, a, b);
          unpack2(y, c, d);
          const __nv_bfloat162 b0 = __floats2bfloat162_rn(a, b), b1 = __floats2bfloat162_rn(c, d);
          const __half2 h0 = __floats2half2_rn(a, b), h1 = __floats2half2_rn(c, d);
          reinterpret_cast<uint2*>(region + block + lane * 32)[i] =
              make_uint2(bf16 ? *reinterpret_cast<const uint32_t*>(&b0) : *reinterpret_cast<const uint32_t*>(&h0),
                         bf16 ? *reinterpret_cast<const uint32_t*>(&b1) : *reinterpret_cast<const uint32_t*>(&h1));
        }
      }
      if (f32) {
        if (col0 + h * 16 < cols) hand_over(col0 + h * 16, dst);
      } else if (h == 2) {
        hand_over(col0, dst);
        if (lane == 0) {
          if (col0 + 16 < cols) tensor_store_2d(map, col0 + 16, row0, dst + 1024);
          if (col0 + 32 < cols) tensor_store_2d(map, col0 + 32, row0, dst + 2048);
        }
      }
    }
  } else if (dtype == AQ_F32) {  // 32 columns = 128 bytes at a time, 128-byte swizzle
#pragma unroll
    for (int h = 0; h < kCount / 32; ++h) {
      room();
      uint4* row = reinterpret_cast<uint4*>(region + lane * 128);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t a = acc[h * 16 + 2 * i], b = acc[h * 16 + 2 * i + 1];
        row[i ^ (lane & 7)] = make_uint4(static_cast<uint32_t>(a), static_cast<uint32_t>(a >> 32), static_cast<uint32_t>(b),
                                         static_cast<uint32_t>(b >> 32));
      }
      hand_over(col0 + h * 32, dst);
    }
  } else {  // 64 columns with the 128-byte swizzle or 32 with the 64-byte swizzle
    room();
    uint4* row = reinterpret_cast<uint4*>(region + lane * (kCount * 2));
    const int swz = kCount == 64 ? lane & 7 : (lane >> 1) & 3;
    const bool bf16 = dtype == AQ_BF16;
#pragma unroll
    for (int i = 0; i < kCount / 8; ++i) {
      uint32_t w[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float a, b;
        unpack2(acc[4 * i + h], a, b);
        const __nv_bfloat162 vb = __floats2bfloat162_rn(a, b);
        const __half2 vh = __floats2half2_rn(a, b);
        w[h] = bf16 ? *reinterpret_cast<const uint32_t*>(&vb) : *reinterpret_cast<const uint32_t*>(&vh);
      }
      row[i ^ swz] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    hand_over(col0, dst);
  }
}

// Debug aid: the exact integer tile sums (W4 tiles were fed 16*w to the MMA).
__device__ __forceinline__ void dump16(const GemmParams& p, int64_t row, int j, int k, int column, const int* v) {
  if (row >= p.m || j >= p.n_j) return;
  const int shift = (p.records[static_cast<int64_t>(j) * p.n_k + k].offset_flag & kW4Flag) ? 4 : 0;
  int4* o = reinterpret_cast<int4*>(p.acc_dump + ((row * p.n_j_total + j) * p.n_k + k) * kTile + column);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[i] = make_int4(v[4 * i] >> shift, v[4 * i + 1] >> shift, v[4 * i + 2] >> shift, v[4 * i + 3] >> shift);
  }
}

// Output transforms of a finished 128-column tile whose FP32 sums lie in shared memory (rows of `stride` floats), where a
// CTA has one output tile only and so the stage ring to put them in.  A warp takes 16 rows of one tile row; a pair
// of lanes owns a row (lane 2 r + h its elements 32 h .. 32 h + 31), so that five of the six butterfly stages stay in
// registers, in the order of inverse_u_row and with its roundings.  (inverse_u_row has two elements per lane and some
// twenty dependent shuffles a row, 20 us for the 32 rows of a drain warp: 128 x 1024 x 1024 29.9 us, now 13.)
__device__ __forceinline__ void turn_rows(float* sums, int stride, const int32_t* meta, int lane) {
  const int half = lane & 1;
  float* own = sums + (lane >> 1) * stride;
  if (meta == nullptr || meta[0] == 0) return;
  double e[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) e[i] = static_cast<double>(own[32 * half + i]) * static_cast<double>(meta[3 * kTile + 32 * half + i]);
#pragma unroll
  for (int stride_of = 1; stride_of < 32; stride_of <<= 1) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if ((i & stride_of) == 0) {
        const double a = e[i], b = e[i + stride_of];
        e[i] = a + b;
        e[i + stride_of] = a - b;
      }
    }
  }
  __syncwarp();
  // lane h ends up with elements 16 h + i and 32 + 16 h + i, i < 16; an eighth of them, which is exact, and the sign
  // that follows commute with the rounding to FP32
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const double sent = half ? e[i] : e[16 + i];
    const double kept = half ? e[16 + i] : e[i];
    const double got = __shfl_xor_sync(0xffffffffu, sent, 1);
    const double a = half ? got : kept, b = half ? kept : got;
    own[16 * half + i] = static_cast<float>((a + b) * 0.125);
    own[32 + 16 * half + i] = static_cast<float>((a - b) * 0.125);
  }
}

// kTurn: one output tile per CTA, with output transforms (TN = 2).
template <int TN, bool kDump, bool kFused, bool kTurn>
__global__ void __launch_bounds__(kThreads, 1)
tmem_gemm_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap out_map, const GemmParams p) {
  using S = Layout<TN>;
  constexpr int kStages = S::kStages;
  constexpr int kStageBytes = S::kStageBytes;
  constexpr int kSub = S::kSub;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* stages = smem;
  uint8_t* turn = smem + kStages * kStageBytes;
  float* scale_ring = reinterpret_cast<float*>(turn + kDrainWarps * kTurnBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes + kDrainWarps * kTurnBytes + S::kScaleBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + S::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_k = p.n_k;
  const int tiles = p.m_blocks * p.n_blocks;
  // split-K over a thread-block cluster along z: this CTA walks K steps [k_begin, k_begin + steps)
  cg::cluster_group cluster = cg::this_cluster();
  const int split_k = static_cast<int>(cluster.num_blocks());
  const int split = static_cast<int>(cluster.block_rank());
  const int k_begin = static_cast<int>(static_cast<int64_t>(n_k) * split / split_k);
  const int steps = static_cast<int>(static_cast<int64_t>(n_k) * (split + 1) / split_k) - k_begin;

  const uint32_t bar0 = smem_u32(bars);
  auto ready = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (2 * kStages + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (2 * kStages + kAccs + b); };
  const uint32_t final_bar = bar0 + 8u * (2 * kStages + 2 * kAccs);

  // one thread per barrier: the initialisations would otherwise run one after the other
  if (threadIdx.x < S::kNumBars) {
    const int i = threadIdx.x;
    // acc_empty: one arrival per drain warp; all others: one (a commit or the copies' expect_tx)
    const uint32_t count = (i >= 2 * kStages + kAccs && i < 2 * kStages + 2 * kAccs) ? kDrainWarps : 1;
    mbar_init(bar0 + 8u * i, count);
    if (i == 0) *abort_flag = 0;
    mbar_init_fence();
    fence_proxy_async();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(kTmemColumns))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Not before the allocation: a dependent kernel that shares the SM and takes tensor memory itself would get it first
  // and keep it while it waits for this grid.
  grid_launch_dependents();
  bool ok = true;

  if (warp >= kDrainWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::kOtherRegs));
    RingPosition<kStages> at;
    if (warp == kMmaWarp) {
      // ---------------- MMA issuer ---------------------------------------------------------
      // The whole warp walks the loop so that addresses and descriptors stay warp-uniform
      // values (the MMA takes them from uniform registers); one elected lane issues.
      constexpr uint32_t idesc_columns = S::kCols;
      const uint32_t idesc = instr_desc_i8(idesc_columns);
      // the low word of a descriptor carries the address in 16-byte units, the rest is constant
      const uint64_t a_desc0 = smem_desc_sw64(smem_u32(stages));
      const uint64_t b_desc0 = smem_desc_sw64(smem_u32(stages) + 2 * kABytes);
      uint32_t unit = 0;  // hand-overs so far
      for (int tile_index = blockIdx.x; tile_index < tiles && ok; tile_index += gridDim.x) {
        for (int kt = 0; kt < steps && ok; kt += 2) {
          ok = mbar_wait(ready(at.slot), at.parity, abort_flag, &g_gemm_status, 2);
          const uint32_t stage = static_cast<uint32_t>(at.slot) * (kStageBytes / 16);
          const bool pair = kt + 1 < steps;
#pragma unroll
          for (int unit_of_stage = 0; unit_of_stage < 2 / kSub; ++unit_of_stage) {
            if (!ok || (unit_of_stage == 1 && !pair)) break;
            const uint32_t b = unit & 1u;
            // a fresh barrier counts as past the phase of parity 1: both accumulators start out free
            ok = mbar_wait(acc_empty(b), ((unit >> 1) & 1u) ^ 1u, abort_flag, &g_gemm_status, 5);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
              // Both operands: rows of 64 bytes, the second K32 half of a row starts 32 bytes in.
              // Every K step starts a fresh integer sum: the first MMA overwrites the accumulator.
#pragma unroll
              for (int sub = 0; sub < kSub; ++sub) {
                const int half = unit_of_stage + sub;
                const uint64_t a_desc = a_desc0 + (stage + half * (kABytes / 16));
                const uint64_t b_desc = b_desc0 + (stage + half * (S::kBBytes / 16));
                const uint32_t d = tmem_base + b * kAccColumns + static_cast<uint32_t>(sub * S::kCols);
                if (sub == 0 || pair) {
                  tc_mma_i8(d, a_desc, b_desc, idesc, 0u);
                  tc_mma_i8(d, a_desc + 2, b_desc + 2, idesc, 1u);
                }
              }
              tc_commit(acc_full(b));
              if (kSub == 2 || unit_of_stage == 1 || !pair) tc_commit(empty(at.slot));
            }
            __syncwarp();
            ++unit;
          }
          at.advance();
        }
      }
      if (!ok) {
        // make sure nothing issued is still running before tensor memory is freed
        if (elect_one()) tc_commit(final_bar);
        __syncwarp();
        for (uint32_t i = 0; i < (1u << 20) && !mbar_try_wait(final_bar, 0); ++i) {
        }
      }
    } else if (warp == kCopyWarp) {
      // ---------------- operand copies and scales --------------------------------------------
      // Two copies per stage.  Lanes 0-7 fetch the weight scales of its two steps (lane = 4 step +
      // tile row), lanes 8-23 under tile scales those of the activations (eight 16-row groups per
      // step), a stage ahead.
      grid_dependency_wait();  // activations and expanded weights come from preceding kernels
      const bool of_weights = lane < 8;
      const int scale_step = of_weights ? lane >> 2 : (lane - 8) >> 3;
      const int scale_index = of_weights ? lane & 3 : (lane - 8) & 7;
      const bool fetches = of_weights ? scale_index < TN : (lane < 24 && p.scale_mode == AQ_SCALE_TILE);
      const int scale_stride = of_weights ? 2 : 1;  // floats from one K step to the next
      float* const scale_dst = scale_ring + (of_weights ? 0 : 4) + scale_index;
      int step = scale_step;  // over all output tiles
      for (int tile_index = blockIdx.x; tile_index < tiles && ok; tile_index += gridDim.x) {
        int mb, nb;
        tile_position(p, tile_index, mb, nb);
        const int j = p.j_base + nb * TN + scale_index;
        int left = steps - scale_step;  // this lane's scales of the tile that are still to be fetched, two steps apart
        if (!(fetches && (of_weights ? j < p.n_j : static_cast<int64_t>(mb) * kBM + 16 * scale_index < p.m))) left = 0;
        const float* scale_src = of_weights ? &p.records[static_cast<int64_t>(j) * n_k + k_begin + scale_step].scale
                                            : p.act_scales + (static_cast<int64_t>(mb) * 8 + scale_index) * n_k + k_begin + scale_step;
        float next_scale = left > 0 ? *scale_src : 0.0f;
        const uint8_t* b_src = p.operand + (static_cast<int64_t>(nb) * n_k + k_begin) * S::kBBytes;
        for (int kt = 0; kt < steps; kt += 2, at.advance()) {
          const float scale = next_scale;
          scale_src += 2 * scale_stride;
          left -= 2;
          next_scale = left > 0 ? *scale_src : 0.0f;
          const bool pair = kt + 1 < steps;
          ok = mbar_wait(empty(at.slot), at.parity ^ 1u, abort_flag, &g_gemm_status, 1);
          if (!ok) break;
          if (lane < 24) scale_dst[(step % kScaleSlots) * kScaleRow] = scale;
          __syncwarp();
          if (elect_one()) {
            const uint32_t dst = smem_u32(stages + at.slot * kStageBytes);
            const uint32_t bar = ready(at.slot);
            mbar_expect_tx(bar, 2 * kABytes + (pair ? 2 : 1) * S::kBBytes);
            tensor_copy_3d(dst, &x_map, 0, mb * kBM, k_begin + kt, bar);
            bulk_copy(dst + 2 * kABytes, b_src, (pair ? 2 : 1) * S::kBBytes, bar);
          }
          __syncwarp();
          b_src += 2 * S::kBBytes;
          step += pair ? 2 : 1;
        }
      }
    }
    if (*abort_flag != 0) {
      // bulk copies may still be in flight: give them a bounded time to land before the CTA
      // and its shared memory go away
      for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::kDrainRegs));
    // ---------------- drain: int32 accumulator -> scaled FP32 registers -------------
    grid_dependency_wait();  // the activation scales come from the preceding kernel, and it may read what is stored here
    constexpr int kWarpCols = S::kWarpCols;
    const int quarter = warp & 3;                  // tensor-memory lane quarter this warp may read
    const int group = warp >> 2;                   // column group
    const int tl = group * kWarpCols / kTile;      // (first) weight tile row of the warp's columns
    const int tile_col = group * kWarpCols % kTile;
    // TN = 3: 48 columns; those of the second and third group begin in one tile row and end in the next
    const int tl_last = (group * kWarpCols + kWarpCols - 1) / kTile;
    const bool middle_in_last = tile_col == 48;
    const int row = quarter * 32 + lane;
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(group * kWarpCols);
    const float* row_scale_ring = scale_ring + 4 + (row >> 4);
    const float* col_scale_ring = scale_ring + tl;
    const int to_last = tl_last - tl;
    const bool tile_mode = p.scale_mode == AQ_SCALE_TILE;
    uint32_t unit = 0;  // hand-overs so far: accumulator unit % 2, phase (unit / 2) % 2
    uint32_t step = 0;  // K steps so far
    uint64_t acc[kWarpCols / 2];  // FP32 sums as packed pairs
    int mb, nb;
    auto token_scale = [&]() {  // of this lane's row in output tile (mb, nb), fetched while the tile before is stored
      const int64_t r = static_cast<int64_t>(mb) * kBM + row;
      return !tile_mode && r < p.m ? p.act_scales[r] : 0.0f;
    };
    tile_position(p, blockIdx.x, mb, nb);
    float a_scale = token_scale();
    for (int tile_index = blockIdx.x; tile_index < tiles && ok; tile_index += gridDim.x) {
      const int64_t row0 = static_cast<int64_t>(mb) * kBM + quarter * 32;
      const int64_t grow = row0 + lane;
      const int j = p.j_base + nb * TN + tl;
#pragma unroll
      for (int i = 0; i < kWarpCols / 2; ++i) acc[i] = 0ull;
      // Rows past M and columns past N take part like all others (zeros and stale columns) and
      // are not stored.  The loop holds 16 TN sums, 32 loaded columns and little else: what does not
      // fit the warp's registers is spilled inside of it (a version that kept pointers and the next
      // scales in registers ran at 1950 instead of 870 cycles per 256-column step).
      const uint32_t end = step + steps;
#pragma unroll 1
      while (step != end) {
        const uint32_t b = unit & 1u;
        ok = mbar_wait(acc_full(b), (unit >> 1) & 1u, abort_flag, &g_gemm_status, 7);
        if (!ok) break;
        tc_fence_after();
        const uint32_t slot = (step % kScaleSlots) * kScaleRow;
        if (tile_mode) a_scale = row_scale_ring[slot];
        float scale0 = __fmul_rn(a_scale, col_scale_ring[slot]);
        float scale1 = 0.0f;
        if (kSub == 2 && step + 1 != end) {  // with an odd number of steps the last stale columns add nothing
          const uint32_t slot1 = ((step + 1) % kScaleSlots) * kScaleRow;
          if (tile_mode) a_scale = row_scale_ring[slot1];
          scale1 = __fmul_rn(a_scale, col_scale_ring[slot1]);
        }
        if (TN == 3) scale1 = __fmul_rn(a_scale, col_scale_ring[slot + to_last]);
        auto hand_back = [&]() {
          tc_fence_before();
          __syncwarp();
          mbar_arrive_lane0(acc_empty(b), lane);
        };
        const uint32_t col = taddr + b * kAccColumns;
        const int k = k_begin + static_cast<int>(step + steps - end);
        int v0[32];
        tc_ld32(col, v0);
        if constexpr (TN == 2) {
          // the warp's 32 columns of both K steps: everything is loaded and handed back before the arithmetic
          int v1[32];
          tc_ld32(col + S::kCols, v1);
          tc_wait_ld32(v0);
          tc_wait_ld32(v1);
          hand_back();
          drain<kFused, 32>(acc, v0, scale0);
          drain<kFused, 32>(acc, v1, scale1);
          if (kDump) {
            for (int c = 0; c < 2; ++c) dump16(p, grow, j, k, tile_col + 16 * c, v0 + 16 * c);
            if (step + 1 != end) {
              for (int c = 0; c < 2; ++c) dump16(p, grow, j, k + 1, tile_col + 16 * c, v1 + 16 * c);
            }
          }
        } else if constexpr (TN == 3) {
          int v1[16];
          tc_ld16(col + 32, v1);
          tc_wait_ld32(v0);
          tc_wait_ld(v1);
          hand_back();
          const float scale_middle = middle_in_last ? scale1 : scale0;
          drain<kFused, 16>(acc, v0, scale0);
          drain<kFused, 16>(acc + 8, v0 + 16, scale_middle);
          drain<kFused, 16>(acc + 16, v1, scale1);
          if (kDump) {
            dump16(p, grow, j, k, tile_col, v0);
            dump16(p, grow, j + (tile_col + 16) / kTile, k, (tile_col + 16) % kTile, v0 + 16);
            dump16(p, grow, j + (tile_col + 32) / kTile, k, (tile_col + 32) % kTile, v1);
          }
        } else {
          // 64 columns: there are registers for half of them at a time
          tc_wait_ld32(v0);
          drain<kFused, 32>(acc, v0, scale0);
          if (kDump) {
            for (int c = 0; c < 2; ++c) dump16(p, grow, j, k, 16 * c, v0 + 16 * c);
          }
          tc_ld32(col + 32, v0);
          tc_wait_ld32(v0);
          hand_back();
          drain<kFused, 32>(acc + 16, v0, scale0);
          if (kDump) {
            for (int c = 0; c < 2; ++c) dump16(p, grow, j, k, 32 + 16 * c, v0 + 16 * c);
          }
        }
        ++unit;
        step = (kSub == 2 && step + 1 == end) ? end : step + kSub;
      }

      if (tile_index + static_cast<int>(gridDim.x) < tiles) {
        tile_position(p, tile_index + gridDim.x, mb, nb);
        a_scale = token_scale();
      }
      // ---------------- epilogue -------------------------------------------------------
      if constexpr (kTurn) {
        // The sums go to shared memory over the stage ring, whose last operands have been consumed.
        constexpr int kRow = S::kCols + 1;
        float* sums = reinterpret_cast<float*>(stages);
#pragma unroll
        for (int c = 0; c < kWarpCols / 2; ++c) unpack2(acc[c], sums[row * kRow + group * kWarpCols + 2 * c], sums[row * kRow + group * kWarpCols + 2 * c + 1]);
        asm volatile("bar.sync 1, %0;" ::"n"(kDrainWarps * 32) : "memory");
        const int turned = p.j_base + nb * TN + (warp & 1);  // tile row of this warp, of rows 16 (warp / 2) ..
        const int64_t first = static_cast<int64_t>(mb) * kBM + (warp >> 1) * 16;
        if (turned < p.n_j && first < p.m) {
          float* region = sums + (warp >> 1) * 16 * kRow + (warp & 1) * kTile;
          const int32_t* meta = p.u_metadata + static_cast<int64_t>(turned) * 4 * kTile;
          turn_rows(region, kRow, meta, lane);
          __syncwarp();
          const bool identity = meta[0] == 0;
          const int t_lo = identity ? lane : meta[kTile + lane], t_hi = identity ? lane + 32 : meta[kTile + lane + 32];
          const int from_lo = (t_lo & 31) + (t_lo < 32 ? 0 : 32), from_hi = (t_hi & 31) + (t_hi < 32 ? 0 : 32);
          const float left_lo = identity ? 1.0f : static_cast<float>(meta[2 * kTile + lane]);
          const float left_hi = identity ? 1.0f : static_cast<float>(meta[2 * kTile + lane + 32]);
          const int rows_here = p.m - first < 16 ? static_cast<int>(p.m - first) : 16;
          for (int r = 0; r < rows_here; ++r) {
            const int64_t o = (first + r) * p.row_stride + static_cast<int64_t>(turned) * kTile + lane;
            store_any(p.out, p.out_dtype, o, region[r * kRow + from_lo] * left_lo);
            store_any(p.out, p.out_dtype, o + 32, region[r * kRow + from_hi] * left_hi);
          }
        }
      } else if (split_k > 1) {
        // split-K: the CTA's FP32 tile goes to shared memory (over the stage ring, whose last
        // operands have been consumed; rows padded by one float so that a warp writing one row
        // per lane hits 32 banks) for the exchange below
        float* dst = reinterpret_cast<float*>(stages) + row * (S::kCols + 1) + group * kWarpCols;
#pragma unroll
        for (int c = 0; c < kWarpCols / 2; ++c) unpack2(acc[c], dst[2 * c], dst[2 * c + 1]);
      } else if (ok && j < p.n_j) {
        const int64_t n_cols = p.row_stride;
        const int32_t* meta = p.u_metadata ? p.u_metadata + static_cast<int64_t>(j) * 4 * kTile : nullptr;
        if (TN != 4 || meta == nullptr || meta[0] == 0) {
          if (row0 < p.m) store_rows<kWarpCols>(&out_map, p.out_dtype, turn + warp * kTurnBytes, static_cast<int>(row0), j * kTile + tile_col,
                                                static_cast<int>(p.row_stride), lane, acc);
        } else if constexpr (TN == 4) {
          // Output transform: a few rows at a time change from one lane per row to two columns
          // per lane (the stage ring already belongs to the next output tile).
          float* region = reinterpret_cast<float*>(turn + warp * kTurnBytes);
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          for (int r0 = 0; r0 < 32; r0 += kTurnRows) {
            __syncwarp();
            if (lane >= r0 && lane < r0 + kTurnRows) {
              float* dst = region + (lane - r0) * kTurnFloats;
#pragma unroll
              for (int c = 0; c < kWarpCols / 2; ++c) unpack2(acc[c], dst[2 * c], dst[2 * c + 1]);
            }
            __syncwarp();
#pragma unroll 1
            for (int r = 0; r < kTurnRows && r0 + r < 32; ++r) {
              const int64_t gr = row0 + r0 + r;
              if (gr >= p.m) break;
              float lo = region[r * kTurnFloats + lane];
              float hi = region[r * kTurnFloats + lane + 32];
              inverse_u_row(lo, hi, meta, lane);
              const int64_t o = gr * n_cols + static_cast<int64_t>(j) * kTile + lane;
              store_any(p.out, p.out_dtype, o, lo);
              store_any(p.out, p.out_dtype, o + 32, hi);
            }
          }
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  if (split_k > 1) {
    // ---------------- split-K exchange through cluster shared memory ------------------------
    // CTA r of the cluster finishes rows r, r + split_k, ...: it adds the split sums in split
    // order (the reference reducer's order, linear.cu:1339-1343), applies the inverse output
    // transform and stores.  The second barrier keeps every CTA's tile alive until read.
    cluster.sync();
    if (warp < kDrainWarps) {
      int mb, nb;
      tile_position(p, blockIdx.x, mb, nb);
      const int64_t m0 = static_cast<int64_t>(mb) * kBM;
      const int tiles_here = min(TN, p.n_j - p.j_base - nb * TN);
      const float* xchg = reinterpret_cast<const float*>(stages);
      const int64_t n_cols = p.row_stride;
      const float* remote[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) remote[s] = cluster.map_shared_rank(xchg, s < split_k ? s : 0);
      const int64_t rows_left = p.m - m0 - split;  // owned rows: split, split + split_k, ... below p.m
      const int owned = rows_left <= 0 ? 0
                        : static_cast<int>(((rows_left < kBM - split ? rows_left : kBM - split) + split_k - 1) / split_k);
      const int pairs = owned * tiles_here;  // (row, weight tile row) pairs, dealt to the drain warps
      for (int q = warp; q < pairs; q += kDrainWarps) {
        const int row = split + split_k * (q / tiles_here);
        const int tl = q % tiles_here;
        const int offset = row * (S::kCols + 1) + tl * kTile + lane;
        // all remote loads of the pair are issued before the first add
        float a[8], b[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          a[s] = 0.0f;
          b[s] = 0.0f;
          if (s < split_k) {
            a[s] = remote[s][offset];
            b[s] = remote[s][offset + 32];
          }
        }
        float lo = a[0], hi = b[0];
#pragma unroll
        for (int s = 1; s < 8; ++s) {
          if (s < split_k) {
            lo = __fadd_rn(lo, a[s]);
            hi = __fadd_rn(hi, b[s]);
          }
        }
        const int j = p.j_base + nb * TN + tl;
        const int32_t* meta = p.u_metadata ? p.u_metadata + static_cast<int64_t>(j) * 4 * kTile : nullptr;
        if (meta != nullptr && meta[0] != 0) inverse_u_row(lo, hi, meta, lane);
        const int64_t o = (m0 + row) * n_cols + static_cast<int64_t>(j) * kTile + lane;
        store_any(p.out, p.out_dtype, o, lo);
        store_any(p.out, p.out_dtype, o + 32, hi);
      }
    }
    cluster.sync();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(kTmemColumns))
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Weight tiles -> the GEMM's operand: every tile as 64 rows of 64 bytes in the 64-byte-swizzle
// layout (a W4 tile widened to 16*w), the TN tile rows of a CTA tile side by side:
// [tile row / TN][k][tile row % TN][4096 bytes], so that the operand of a stage is one copy.
//
// Widening inside the GEMM costs every 128-row block of the activations again, and what it costs
// there is not bandwidth but instructions of single warps next to sixteen draining ones: 1900
// cycles per K step instead of 750 for the bare drain.  Here it is a streaming pass over the weights.
// A CTA takes eight consecutive tiles of a tile row; all their loads are in flight together.
// ---------------------------------------------------------------------------------------------
constexpr int kExpandTiles = 8;

__global__ void __launch_bounds__(256) expand_kernel(const TileRecord* __restrict__ records, const uint8_t* __restrict__ payload,
                                                     int n_k, int j_base, int tn, uint8_t* __restrict__ operand) {
  const int k0 = blockIdx.x * kExpandTiles;
  const int row = blockIdx.y;
  const TileRecord* recs = records + static_cast<int64_t>(j_base + row) * n_k;
  const int n = threadIdx.x >> 2;                      // row of the tile
  const int k16 = (threadIdx.x & 3) ^ ((n >> 1) & 3);  // 16-byte chunk of that row that this thread's slot holds
  uint32_t of[kExpandTiles];
#pragma unroll
  for (int i = 0; i < kExpandTiles; ++i) of[i] = k0 + i < n_k ? __ldg(&recs[k0 + i].offset_flag) : 0u;
  uint4 v[kExpandTiles];
#pragma unroll
  for (int i = 0; i < kExpandTiles; ++i) {
    const uint8_t* tile = payload + static_cast<int64_t>(of[i] & ~kW4Flag) * kW4TileBytes;
    const int at = (of[i] & kW4Flag) ? n * 32 + (k16 >> 1) * 16 : static_cast<int>(threadIdx.x) * 16;
    if (k0 + i < n_k) v[i] = __ldg(reinterpret_cast<const uint4*>(tile + at));
  }
  grid_launch_dependents();
  grid_dependency_wait();  // the GEMM before may still read the operand of its own weights
  uint8_t* dst = operand + ((static_cast<int64_t>(row / tn) * n_k + k0) * tn + row % tn) * kW8TileBytes + threadIdx.x * 16;
#pragma unroll
  for (int i = 0; i < kExpandTiles; ++i) {
    if (k0 + i >= n_k) break;
    if (of[i] & kW4Flag) {
      const int shift = (k16 & 1) ? 0 : 4;
      v[i].x = (v[i].x << shift) & 0xf0f0f0f0u;
      v[i].y = (v[i].y << shift) & 0xf0f0f0f0u;
      v[i].z = (v[i].z << shift) & 0xf0f0f0f0u;
      v[i].w = (v[i].w << shift) & 0xf0f0f0f0u;
    }
    *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(i) * tn * kW8TileBytes) = v[i];
  }
}

// The workspace starts with the arrival counters of the stream-K kernel, which have to stay zero.
constexpr int64_t kScratchOffset = 64 * 1024;
// Expanded weights at a time: a layer above this is run in several passes over its columns.  Not so few that a pass
// leaves SMs idle: with 64 MiB, which the L2 would keep, 129 x 34816 x 5120 ran three passes of 96 output tiles, 157
// us against 127 in one, and 129 x 65536 x 2048 131 against 104.
constexpr int64_t kScratchBytes = 256LL << 20;

// Tile rows per pass, the passes of about one size: the tile width and the K ranges are chosen for a pass.
int rows_per_pass(int n_j, int n_k) {
  if (n_k > kMaxNk) return n_j;  // refused at the launch; a scratch of this size holds at least 24 tile rows up to there
  int64_t most = kScratchBytes / (static_cast<int64_t>(n_k) * kW8TileBytes);
  if (most >= n_j) return n_j;
  most = most / 12 * 12;  // whole CTA tiles of every width
  const int64_t passes = (n_j + most - 1) / most;
  return static_cast<int>(((n_j + passes - 1) / passes + 11) / 12 * 12);
}

int launch_expand(const TileRecord* records, const uint8_t* payload, int n_k, int j_base, int rows, int tn, uint8_t* operand,
                  cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>((n_k + kExpandTiles - 1) / kExpandTiles), static_cast<unsigned>(rows), 1);
  config.blockDim = dim3(256, 1, 1);
  config.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = use_dependent_launch() ? 1 : 0;
  return check_cuda(cudaLaunchKernelEx(&config, expand_kernel, records, payload, n_k, j_base, tn, operand), "weight expansion launch");
}

template <int TN>
int set_shared_memory(int device) {
  static std::once_flag once[64];
  cudaError_t attr_status = cudaSuccess;
  std::call_once(once[device & 63], [&] {
    const void* kernels[8] = {
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, false, false, false>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, false, true, false>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, true, false, false>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, true, true, false>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, false, false, TN == 2>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, false, true, TN == 2>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, true, false, TN == 2>),
        reinterpret_cast<const void*>(tmem_gemm_kernel<TN, true, true, TN == 2>)};
    for (const void* kernel : kernels) {
      if (attr_status == cudaSuccess) {
        attr_status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<TN>::kSmemBytes);
      }
    }
  });
  return check_cuda(attr_status, "cudaFuncSetAttribute(tmem_gemm_kernel)");
}

// Clusters of `split` CTAs that can be resident at once (SMs of different GPU processing clusters do
// not form one: 48 clusters of three need more than 144 SMs); cached per device.
template <int TN>
int resident_clusters(int split, int device) {
  static std::mutex mutex;
  static int cache[64][9];  // 0: not asked yet, -1: failed
  std::lock_guard<std::mutex> lock(mutex);
  int& slot = cache[device & 63][split];
  if (slot == 0) {
    int clusters = 0;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(1, 1, static_cast<unsigned>(split));
    config.blockDim = dim3(kThreads, 1, 1);
    config.dynamicSmemBytes = static_cast<size_t>(Layout<TN>::kSmemBytes);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = static_cast<unsigned>(split);
    config.attrs = attr;
    config.numAttrs = 1;
    if (set_shared_memory<TN>(device) != AQ_OK ||
        cudaOccupancyMaxActiveClusters(&clusters, reinterpret_cast<const void*>(tmem_gemm_kernel<TN, false, true, false>), &config) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    slot = clusters > 0 ? clusters : -1;
  }
  return slot > 0 ? slot : 0;
}

template <int TN>
int launch_shape(const CUtensorMap& x_map, const CUtensorMap& out_map, const GemmParams& p, bool dump, bool fused, int split, int sm_count,
                 int device, cudaStream_t stream) {
  using S = Layout<TN>;
  int rc = set_shared_memory<TN>(device);
  if (rc != AQ_OK) return rc;
  const int tiles = p.m_blocks * p.n_blocks;
  cudaLaunchConfig_t config = {};
  // a persistent CTA per SM; with K ranges one cluster per output tile
  config.gridDim = dim3(static_cast<unsigned>(split > 1 || tiles < sm_count ? tiles : sm_count), 1, static_cast<unsigned>(split));
  config.blockDim = dim3(kThreads, 1, 1);
  config.dynamicSmemBytes = static_cast<size_t>(S::kSmemBytes);
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(split);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attr;
  config.numAttrs = use_dependent_launch() ? 2 : 1;
  const bool turn = TN == 2 && split == 1 && p.u_metadata != nullptr;
  const auto kernel = turn ? (dump ? (fused ? tmem_gemm_kernel<TN, true, true, TN == 2> : tmem_gemm_kernel<TN, true, false, TN == 2>)
                                   : (fused ? tmem_gemm_kernel<TN, false, true, TN == 2> : tmem_gemm_kernel<TN, false, false, TN == 2>))
                           : (dump ? (fused ? tmem_gemm_kernel<TN, true, true, false> : tmem_gemm_kernel<TN, true, false, false>)
                                   : (fused ? tmem_gemm_kernel<TN, false, true, false> : tmem_gemm_kernel<TN, false, false, false>));
  const cudaError_t status = cudaLaunchKernelEx(&config, kernel, x_map, out_map, p);
  return check_cuda(status, "tensor-memory GEMM launch");
}

int device_sm_count(int* count) {
  int device = 0;
  int rc = check_cuda(cudaGetDevice(&device), "cudaGetDevice");
  if (rc != AQ_OK) return rc;
  static int sm_counts[64] = {0};
  if (sm_counts[device & 63] == 0) {
    int value = 0;
    rc = check_cuda(cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    if (rc != AQ_OK) return rc;
    sm_counts[device & 63] = value;
  }
  *count = sm_counts[device & 63];
  return AQ_OK;
}

// Tile width and number of K ranges of a problem.
struct Choice {
  int tn;
  int split;
  double cost;  // modelled SM cycles of a pass
};

// The cheapest of the three tile widths and up to eight K ranges by a model in SM cycles: a CTA's K
// steps, its hand-over from one output tile to the next, and the exchange of a split.  Measured on
// B200 (cycles): a K step 850 / 730 / 527 for TN = 4 / 3 / 2, a hand-over 1800 / 3000 / 1400, an exchange
// 4000 per tile row.  The wide tile wins where there are many output tiles (16384 x 19456 x 2560: 1287 us
// against 1537 and 1575); the others where it would leave most of a last wave idle (2048 x 5120 x 3072:
// 69 us against 77); K ranges only pay for a few row blocks (128 x 5120 x 3072: 16 us against 21).
// `n_j`: tile rows of a pass (with the whole layer's, 34816 x 5120 at 48 rows ran three passes of 48 CTAs).
// AQ_OPT_GEMM_TILE and AQ_OPT_GEMM_SPLIT force a choice.
Choice choose(int64_t m, int n_j, int n_k, int forced_tile, int forced_split, int sm_count, int device) {
  const int64_t m_blocks = (m + kBM - 1) / kBM;
  static const double kStep[5] = {0, 0, 527, 730, 850};
  static const double kHandOver[5] = {0, 0, 1400, 3000, 1800};
  Choice best = {4, 1, 0.0};
  double best_cost = 0.0;
  for (int tn = 4; tn >= 2; --tn) {
    if (forced_tile == AQ_GEMM_TILE_WIDE && tn != 4) continue;
    if (forced_tile == AQ_GEMM_TILE_NARROW && tn != 3) continue;
    if (forced_tile == AQ_GEMM_TILE_PAIRED && tn != 2) continue;
    const int64_t tiles = m_blocks * ((n_j + tn - 1) / tn);
    for (int split = 1; split <= 8; ++split) {
      int64_t at_once = sm_count;
      if (forced_split >= 1 && forced_split <= 8) {
        if (split != forced_split) continue;
      } else if (split > 1) {
        if (n_k / split < 4 || tiles * split > sm_count) break;
        at_once = tn == 4 ? resident_clusters<4>(split, device) : tn == 3 ? resident_clusters<3>(split, device) : resident_clusters<2>(split, device);
        if (tiles > at_once) continue;
      }
      const int64_t waves = (tiles + at_once - 1) / at_once;
      const double cost = static_cast<double>(waves) * ((n_k + split - 1) / split * kStep[tn] + kHandOver[tn]) + (split > 1 ? 4000.0 * tn : 0.0);
      if (best_cost == 0.0 || cost < best_cost) {
        best_cost = cost;
        best = {tn, split, cost};
      }
    }
  }
  while (best.split > 1 && n_k / best.split < 4) --best.split;
  return best;
}

}  // namespace

// Up to 128 rows the kernel that reads the packed weights once, where that pass costs less than their expansion and
// the GEMM for many rows, both by their models (expansion: 2.1 cycles per tile, measured: 14 us for 12288 tiles, but not
// less than 4000, and a launch).  Measured (us, gemm_rows_kernel / the other): 64 rows 34816 x 5120 57 / 91, 1024 x 1024
// 6.1 / 9.4, 3072 x 3072 9.5 / 13; 128 rows 34816 x 5120 65 / 91, 16384 x 3072 21.5 / 28.4, 1024 x 1024 8.4 / 9.5,
// 19456 x 64 8.9 / 7.2, 19456 x 2560 (152 CTAs: a second wave of four) 36 / 33.
GemmPlan plan_gemm(int64_t m, int n_j, int n_k) {
  const int forced_tile = gemm_tile_option();
  const int forced_split = gemm_split_option();
  int sm_count = 148;
  if (device_sm_count(&sm_count) != AQ_OK) sm_count = 148;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) device = 0;
  GemmPlan plan = {};
  plan.fused = !gemm_separate_rounding();
  plan.rows_per_pass = rows_per_pass(n_j, n_k);
  const Choice choice = choose(m, plan.rows_per_pass, n_k, forced_tile, forced_split, sm_count, device);
  plan.tn = choice.tn;
  plan.split = choice.split;
  if (n_k > kMaxNk) return plan;  // the launch says why
  if (m <= kBM && plan.fused && forced_tile == AQ_GEMM_TILE_AUTO) {
    const int passes = (n_j + plan.rows_per_pass - 1) / plan.rows_per_pass;
    const double tiles = static_cast<double>(n_j) * n_k;
    // Above what the L2 keeps the expanded weights come from HBM again: 14000 cycles more, whatever the size.
    const double again = static_cast<double>(plan.rows_per_pass) * n_k * kW8TileBytes > 64e6 ? 14000.0 : 0.0;
    const double cost = passes * (choice.cost + again + 4500.0) + (2.1 * tiles > 4000.0 ? 2.1 * tiles : 4000.0);
    double rows_cost = 0.0;
    const int rows_split = gemm_rows_split(m, n_j, n_k, forced_split, &rows_cost);
    if (forced_split >= 1 || rows_cost < cost) {
      plan.few_rows = true;
      plan.split = rows_split;
      return plan;
    }
  }
  // Up to three tile rows fill up the last CTA tile.  A layer that is cut into passes asks for the whole scratch, not
  // for its longest pass, so that what suffices for a layer suffices for every smaller one.
  const int64_t tile_row = static_cast<int64_t>(n_k) * kW8TileBytes;
  plan.workspace_bytes = kScratchOffset + (plan.rows_per_pass == n_j ? n_j * tile_row : kScratchBytes) + 3 * tile_row;
  return plan;
}

int launch_tmem_gemm(const LinearArgs& a, const GemmPlan& plan, cudaStream_t stream) {
  if (a.n_k > kMaxNk) {
    return fail(AQ_ERR_INVALID, "the GEMM kernel supports K up to %d, got %d", kMaxNk * kTile,
                a.n_k * kTile);
  }
  if (plan.few_rows) return launch_gemm_rows(a, plan.split, stream);
  int device = 0;
  int rc = check_cuda(cudaGetDevice(&device), "cudaGetDevice");
  if (rc != AQ_OK) return rc;
  int sm_count = 0;
  rc = device_sm_count(&sm_count);
  if (rc != AQ_OK) return rc;
  if (a.m >= (1LL << 31)) return fail(AQ_ERR_INVALID, "the GEMM kernel supports fewer than 2^31 rows");
  alignas(64) CUtensorMap x_map;
  rc = encode_activation_map(&x_map, a.xq, a.m, a.n_k, kBM, 2);
  if (rc != AQ_OK) return rc;
  const int rows_at_once = plan.rows_per_pass;
  // With transforms and one K range a row's 64 columns have to meet in one warp: in the stage ring where every CTA has
  // only one 128-column tile, else (the ring belongs to the next tile) in the drain warps of a 256-column one.
  int tn = plan.tn;
  if (a.u_metadata != nullptr && plan.split == 1) tn = (a.m + kBM - 1) / kBM * ((plan.rows_per_pass + 1) / 2) <= sm_count ? 2 : 4;
  alignas(64) CUtensorMap out_map;
  rc = encode_result_map(&out_map, a.out, a.out_dtype, a.m, static_cast<int64_t>(a.n_j) * kTile, tn == 4 ? 64 : tn == 3 ? 16 : 32, 32);
  if (rc != AQ_OK) return rc;
  const bool dump = a.acc_dump != nullptr;
  uint8_t* operand = static_cast<uint8_t*>(a.workspace) + kScratchOffset;
  for (int j_base = 0; j_base < a.n_j; j_base += rows_at_once) {
    const int rows = a.n_j - j_base < rows_at_once ? a.n_j - j_base : rows_at_once;
    rc = launch_expand(a.records, a.payload, a.n_k, j_base, rows, tn, operand, stream);
    if (rc != AQ_OK) return rc;
    GemmParams p;
    p.act_scales = a.act_scales;
    p.records = a.records;
    p.operand = operand;
    p.u_metadata = a.u_metadata;
    p.out = a.out;
    p.acc_dump = a.acc_dump;
    p.m = a.m;
    p.n_j = j_base + rows;
    p.n_k = a.n_k;
    p.j_base = j_base;
    p.row_stride = static_cast<int64_t>(a.n_j) * kTile;
    p.n_j_total = a.n_j;
    p.scale_mode = a.scale_mode;
    p.out_dtype = a.out_dtype;
    p.m_blocks = static_cast<int>((a.m + kBM - 1) / kBM);
    p.n_blocks = (rows + tn - 1) / tn;
    p.band_magic = static_cast<uint32_t>((1ULL << 32) / (static_cast<uint64_t>(p.n_blocks) * 16));
    if (static_cast<int64_t>(p.m_blocks) * p.n_blocks >= (1LL << 31) / 16) return fail(AQ_ERR_INVALID, "the GEMM kernel supports fewer output tiles");
    rc = tn == 4   ? launch_shape<4>(x_map, out_map, p, dump, plan.fused, plan.split, sm_count, device, stream)
         : tn == 3 ? launch_shape<3>(x_map, out_map, p, dump, plan.fused, plan.split, sm_count, device, stream)
                          : launch_shape<2>(x_map, out_map, p, dump, plan.fused, plan.split, sm_count, device, stream);
    if (rc != AQ_OK) return rc;
  }
  return AQ_OK;
}

int take_gemm_status() {
  int status = 0;
  if (cudaMemcpyFromSymbol(&status, g_gemm_status, sizeof(int)) != cudaSuccess) return -1;
  if (status != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int));
  }
  return status;
}

}  // namespace aq
