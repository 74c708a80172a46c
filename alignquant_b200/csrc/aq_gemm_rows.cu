// Mixed W4/W8 x A8 GEMM for up to 128 rows on the Blackwell tensor cores (sm_100a).
//
// With few rows the weights are the large operand: they are read once, straight from the prepared
// image, and they are the M side of the MMA.  A CTA takes two tile rows (128 output columns) and a
// range of K; D is 128 columns x NT activation rows (NT = 32, 64 or 128), so nothing is spent on
// padding the rows to 128.  Above 64 rows there is no padding to save and the sides change: with the rows on the M side
// a drain lane has one row and one tile row, so that one scale serves all of its results of a step (with the
// weights there, a multiplication and a shared-memory read for every pair of results: 1060 cycles a step, now 660).  What
// bounds it is the weight stream; the GEMM of aq_gemm_tmem.cu expands the
// weights into a workspace first (2.4 times the bytes written and read again) and drains 128 x 256 results
// per step whatever the rows: 34816 x 5120 at 48 rows took 167 us there.
//
//   * a stage of the ring holds SUB K steps (four, two for NT = 128).  The packed tiles of a tile row's
//     steps are contiguous, so a stage is two bulk copies and one tensor-map copy of the activations;
//   * eight warps widen a stage in place: every warp reads its tile (half a tile for NT = 128) into registers,
//     the eight meet at a barrier, then each lays its tile down in its operand slot (64-byte swizzle, W4 as 16*w);
//   * one warp issues tcgen05.mma kind::i8 (M = 128, N = NT, K = 32) into one of two accumulators of
//     SUB x NT columns: a hand-over covers a whole stage;
//   * eight warps drain: 32 columns x NT / 2 rows each (NT = 128: 32 rows x 64 columns), one packed multiply
//     (activation scale x weight scale; NT = 128: one per step) and one packed fused multiply-add per two results,
//     tiles in increasing k: the roundings of aq_gemm_tmem.cu, bit for bit;
//   * K ranges of a thread-block cluster meet in distributed shared memory, added in split order.
//
// Every wait is bounded, as in aq_gemm_tmem.cu.
#include <cooperative_groups.h>
#include <cuda.h>

#include <mutex>

#include "aq_common.cuh"
#include "aq_ptx.cuh"
#include "aq_tile_math.cuh"
#include "aq_tcgen05.cuh"

namespace cg = cooperative_groups;

namespace aq {

__device__ int g_gemm_rows_status = 0;

namespace {

constexpr int kDrainWarps = 8;
constexpr int kWidenWarps = 8;
constexpr int kMmaWarp = kDrainWarps + kWidenWarps;
constexpr int kCopyWarp = kMmaWarp + 1;
constexpr int kWarps = 20;  // whole warpgroups, for the registers: two warps have no role
constexpr int kThreads = kWarps * 32;
// Registers: the block is launched with 96 per thread; a drain thread of 128 rows holds 64 sums, 32
// loaded values and their scales.
constexpr int kDrainRegs = 144;
constexpr int kOtherRegs = 64;
static_assert(kDrainWarps * 32 * kDrainRegs + (kThreads - kDrainWarps * 32) * kOtherRegs <= kThreads * 96,
              "setmaxnreg would wait for registers that the block does not have");
constexpr int kMmaRows = 2 * kTile;  // output columns of a CTA: the M side of the MMA

template <int NT>
struct RowsLayout {
  static constexpr int kSub = NT == 128 ? 2 : 4;             // K steps per stage
  static constexpr int kStages = NT == 128 ? 6 : 4;
  static constexpr int kABytes = kSub * 2 * kW8TileBytes;    // weight operand, and the packed tiles before they are widened
  static constexpr int kBBytes = kSub * NT * kTile;          // activations
  static constexpr int kStageBytes = kABytes + kBBytes;      // 40, 48 or 32 KiB
  static constexpr int kAccColumns = kSub * NT;              // at most 256
  static constexpr int kTmemColumns = 2 * kAccColumns;
  static constexpr int kWarpsPerTile = kWidenWarps / (2 * kSub);
  static constexpr bool kRowsOnM = NT == 128;                // lanes of an accumulator: activation rows, else output columns
  static constexpr int kCols = NT / 2;                       // accumulator columns of a drain warp (activation rows; kRowsOnM: output columns)
  static constexpr int kXchgRow = kMmaRows + (kRowsOnM ? 1 : 4);  // floats per activation row of the exchange tile
  // landed[S], ready[S], empty[S], acc_full[2], acc_empty[2], final
  static constexpr int kNumBars = 3 * kStages + 5;
  static constexpr int kSmemBytes = kStages * kStageBytes + NT * 4 + kNumBars * 8 + 16;
  static_assert(NT * kXchgRow * 4 <= kStages * kStageBytes, "the exchange tile must fit into the ring");
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of a CTA");
};

struct RowsParams {
  const float* act_scales;
  const TileRecord* records;
  const uint8_t* payload;
  const int32_t* u_metadata;
  void* out;
  int32_t* acc_dump;
  int m;
  int n_j;
  int n_k;
  int out_dtype;
};

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t both(float v) { return pack2(__float_as_uint(v), __float_as_uint(v)); }

template <int NT, bool kToken, bool kDump>
__global__ void __launch_bounds__(kThreads, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap x_map, const RowsParams p) {
  using S = RowsLayout<NT>;
  constexpr int kSub = S::kSub;
  constexpr int kStages = S::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* stages = smem;
  float* row_scales = reinterpret_cast<float*>(smem + kStages * S::kStageBytes);  // [NT], per-token mode
  uint64_t* bars = reinterpret_cast<uint64_t*>(row_scales + NT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + S::kNumBars);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_k = p.n_k;
  cg::cluster_group cluster = cg::this_cluster();
  const int split_k = static_cast<int>(cluster.num_blocks());
  const int split = static_cast<int>(cluster.block_rank());
  const int k_begin = static_cast<int>(static_cast<int64_t>(n_k) * split / split_k);
  const int steps = static_cast<int>(static_cast<int64_t>(n_k) * (split + 1) / split_k) - k_begin;
  const int n_stages = (steps + kSub - 1) / kSub;
  const int j0 = blockIdx.x * 2;

  const uint32_t bar0 = smem_u32(bars);
  auto landed = [&](int s) { return bar0 + 8u * s; };
  auto ready = [&](int s) { return bar0 + 8u * (kStages + s); };
  auto empty = [&](int s) { return bar0 + 8u * (2 * kStages + s); };
  auto acc_full = [&](int b) { return bar0 + 8u * (3 * kStages + b); };
  auto acc_empty = [&](int b) { return bar0 + 8u * (3 * kStages + 2 + b); };
  const uint32_t final_bar = bar0 + 8u * (3 * kStages + 4);

  if (threadIdx.x < S::kNumBars) {
    const int i = threadIdx.x;
    const bool of_widen = i >= kStages && i < 2 * kStages;
    const bool of_drain = i >= 3 * kStages + 2 && i < 3 * kStages + 4;
    mbar_init(bar0 + 8u * i, of_widen ? kWidenWarps : of_drain ? kDrainWarps : 1);
    if (i == 0) *abort_flag = 0;
    mbar_init_fence();
    fence_proxy_async();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(static_cast<uint32_t>(S::kTmemColumns))
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
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
  if (warp == kCopyWarp) {
    // ---------------- copies ----------------------------------------------------------------------
    // Lane l keeps place and size of stage l's packed tiles (of stage 32 b + l in the b-th block of 32), so that no
    // stage waits for a record.
    uint32_t first0 = 0, bytes0 = 0, first1 = 0, bytes1 = 0;
    auto load_places = [&](int st0) {
      const int first = (st0 + lane) * kSub;
      if (first >= steps) return;
      const int last = min(first + kSub, steps) - 1;
      const TileRecord* recs = p.records + static_cast<int64_t>(j0) * n_k + k_begin;
      const TileRecord rf = recs[first];
      first0 = rf.offset_flag & ~kW4Flag;
      bytes0 = span_bytes(rf, recs[last]);
      if (j0 + 1 < p.n_j) {
        const TileRecord rg = recs[n_k + first];
        first1 = rg.offset_flag & ~kW4Flag;
        bytes1 = span_bytes(rg, recs[n_k + last]);
      }
    };
    auto weights = [&](int st, int slot) {
      if ((st & 31) == 0) load_places(st);
      const uint32_t place = __shfl_sync(0xffffffffu, first0, st & 31), size = __shfl_sync(0xffffffffu, bytes0, st & 31);
      const uint32_t place1 = __shfl_sync(0xffffffffu, first1, st & 31), size1 = __shfl_sync(0xffffffffu, bytes1, st & 31);
      if (lane == 0) {
        const uint32_t dst = smem_u32(stages + slot * S::kStageBytes);
        mbar_expect_tx(landed(slot), size + size1 + S::kBBytes);
        bulk_copy(dst, p.payload + static_cast<int64_t>(place) * kW4TileBytes, size, landed(slot));
        if (size1 != 0) bulk_copy(dst + S::kABytes / 2, p.payload + static_cast<int64_t>(place1) * kW4TileBytes, size1, landed(slot));
      }
      __syncwarp();
    };
    auto activations = [&](int st, int slot) {
      if (lane == 0) {
        tensor_copy_3d(smem_u32(stages + slot * S::kStageBytes) + S::kABytes, &x_map, 0, 0, k_begin + st * kSub, landed(slot));
      }
      __syncwarp();
    };
    // the weights do not depend on the preceding kernel: the ring is filled with them before it ends
    const int ahead = min(kStages, n_stages);
    for (int st = 0; st < ahead; ++st) weights(st, st);
    grid_dependency_wait();
    for (int st = 0; st < ahead; ++st) activations(st, st);
    int slot = 0;
    uint32_t parity = 0;
    for (int st = ahead; st < n_stages; ++st) {
      ok = mbar_wait(empty(slot), parity, abort_flag, &g_gemm_rows_status, 81);
      if (!ok) break;
      weights(st, slot);
      activations(st, slot);
      if (++slot == kStages) {
        slot = 0;
        parity ^= 1u;
      }
    }
  } else if (warp == kMmaWarp) {
    const uint32_t idesc = instr_desc_i8(NT);
    const uint64_t a_desc0 = smem_desc_sw64(smem_u32(stages));
    const uint64_t b_desc0 = smem_desc_sw64(smem_u32(stages) + S::kABytes);
    int slot = 0;
    uint32_t parity = 0;
    for (int st = 0; st < n_stages; ++st) {
      const uint32_t b = st & 1;
      ok = mbar_wait(ready(slot), parity, abort_flag, &g_gemm_rows_status, 82);
      // a fresh barrier counts as past the phase of parity 1: both accumulators start out free
      ok = ok && mbar_wait(acc_empty(b), ((st >> 1) & 1u) ^ 1u, abort_flag, &g_gemm_rows_status, 85);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t stage = static_cast<uint32_t>(slot) * (S::kStageBytes / 16);
        const int here = min(kSub, steps - st * kSub);
#pragma unroll
        for (int s = 0; s < kSub; ++s) {
          if (s < here) {
            const uint64_t a_desc = a_desc0 + (stage + s * (2 * kW8TileBytes / 16));
            const uint64_t b_desc = b_desc0 + (stage + s * (NT * kTile / 16));
            const uint32_t d = tmem_base + b * S::kAccColumns + static_cast<uint32_t>(s * NT);
            tc_mma_i8(d, S::kRowsOnM ? b_desc : a_desc, S::kRowsOnM ? a_desc : b_desc, idesc, 0u);
            tc_mma_i8(d, (S::kRowsOnM ? b_desc : a_desc) + 2, (S::kRowsOnM ? a_desc : b_desc) + 2, idesc, 1u);
          }
        }
        tc_commit(acc_full(b));
        tc_commit(empty(slot));
      }
      __syncwarp();
      if (++slot == kStages) {
        slot = 0;
        parity ^= 1u;
      }
    }
    if (!ok) {
      // make sure nothing issued is still running before tensor memory is freed
      if (elect_one()) tc_commit(final_bar);
      __syncwarp();
      for (uint32_t i = 0; i < (1u << 20) && !mbar_try_wait(final_bar, 0); ++i) {
      }
    }
  } else if (warp < kMmaWarp) {
    // ---------------- widening ------------------------------------------------------------------
    const int w = warp - kDrainWarps;
    const int tile = w / S::kWarpsPerTile;  // step of the stage, tile row
    const int s = tile >> 1, r = tile & 1;
    constexpr int kVecs = 8 / S::kWarpsPerTile;  // 16-byte vectors of a lane
    const int t0 = (w % S::kWarpsPerTile) * (256 / S::kWarpsPerTile) + lane;  // slot t: row t / 4, chunk t % 4 of the tile
    const bool row_exists = j0 + r < p.n_j;
    const TileRecord* recs = p.records + static_cast<int64_t>(row_exists ? j0 + r : j0) * n_k + k_begin;
    // Lane l keeps the place of the warp's tile among the packed tiles of stage l, and its W4 flag.
    uint32_t lane_of = 0;
    auto load_places = [&](int st0) {
      const int at = (st0 + lane) * kSub;
      if (at + s >= steps) return;
      const uint32_t of = recs[at + s].offset_flag, first = recs[at].offset_flag;
      lane_of = (((of & ~kW4Flag) - (first & ~kW4Flag)) * kW4TileBytes) | (of & kW4Flag);
    };
    int slot = 0;
    uint32_t parity = 0;
    for (int st = 0; st < n_stages; ++st) {
      if ((st & 31) == 0) load_places(st);
      const uint32_t of = __shfl_sync(0xffffffffu, lane_of, st & 31);
      // the eight warps meet at a barrier in every stage: after a time-out they still walk all stages
      ok = ok && mbar_wait(landed(slot), parity, abort_flag, &g_gemm_rows_status, 83);
      const bool works = ok && row_exists && st * kSub + s < steps;
      const uint8_t* packed = stages + slot * S::kStageBytes + r * (S::kABytes / 2) + (of & ~kW4Flag);
      const bool w4 = (of & kW4Flag) != 0;
      uint4 v[kVecs];
      if (works) {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) {
          const int t = t0 + 32 * i;
          const int n = t >> 2, k16 = (t & 3) ^ ((n >> 1) & 3);
          v[i] = *reinterpret_cast<const uint4*>(packed + (w4 ? n * 32 + (k16 >> 1) * 16 : t * 16));
          if (w4) {
            const int shift = (k16 & 1) ? 0 : 4;
            v[i].x = (v[i].x << shift) & 0xf0f0f0f0u;
            v[i].y = (v[i].y << shift) & 0xf0f0f0f0u;
            v[i].z = (v[i].z << shift) & 0xf0f0f0f0u;
            v[i].w = (v[i].w << shift) & 0xf0f0f0f0u;
          }
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kWidenWarps * 32) : "memory");  // every packed tile has been read
      if (works) {
        uint8_t* operand = stages + slot * S::kStageBytes + (s * 2 + r) * kW8TileBytes;
#pragma unroll
        for (int i = 0; i < kVecs; ++i) *reinterpret_cast<uint4*>(operand + (t0 + 32 * i) * 16) = v[i];
      }
      fence_proxy_async();
      __syncwarp();
      mbar_arrive_lane0(ready(slot), lane);
      if (++slot == kStages) {
        slot = 0;
        parity ^= 1u;
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDrainRegs));
    // ---------------- drain: lane = output column, registers = activation rows; kRowsOnM: the other way round ----------
    constexpr int kCols = S::kCols;
    constexpr bool kRowsOnM = S::kRowsOnM;
    constexpr int kXchgRow = S::kXchgRow;
    const int quarter = warp & 3;  // tensor-memory lane quarter this warp may read
    const int group = warp >> 2;   // accumulator columns group * kCols ..
    const int j = j0 + (kRowsOnM ? group : quarter >> 1);
    const TileRecord* recs = p.records + static_cast<int64_t>(j < p.n_j ? j : j0) * n_k + k_begin;
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(group * kCols);
    float w_next[kSub];
#pragma unroll
    for (int s = 0; s < kSub; ++s) w_next[s] = s < steps ? __ldg(&recs[s].scale) : 0.0f;
    grid_dependency_wait();  // the activation scales come from the preceding kernel, and it may read what is stored here
    // 16-row groups of the warp (kRowsOnM: of the lane), one scale each per step under tile scales
    constexpr int kRowGroups = kRowsOnM ? 1 : kCols / 16;
    const int m_row = quarter * 32 + lane;  // kRowsOnM: this lane's activation row
    float g_next[kToken ? 1 : kSub][kRowGroups];
    // Ordinary loads, as for all that the preceding kernel writes: it may still be writing while this one is resident,
    // and the read-only path does not see that (stale scales at 128 x 3072 x 3072).
    auto group_scales = [&](int at) {
      if constexpr (!kToken) {
#pragma unroll
        for (int s = 0; s < kSub; ++s) {
#pragma unroll
          for (int g = 0; g < kRowGroups; ++g) {
            const int row_group = kRowsOnM ? m_row >> 4 : group * kRowGroups + g;
            g_next[s][g] = at + s < steps && row_group * 16 < p.m
                               ? p.act_scales[static_cast<int64_t>(row_group) * n_k + k_begin + at + s]
                               : 0.0f;
          }
        }
      }
    };
    group_scales(0);
    float token_scale = 0.0f;
    if constexpr (kToken && kRowsOnM) {
      if (m_row < p.m) token_scale = p.act_scales[m_row];
    } else if (kToken) {
      if (threadIdx.x < NT) row_scales[threadIdx.x] = static_cast<int>(threadIdx.x) < p.m ? p.act_scales[threadIdx.x] : 0.0f;
      asm volatile("bar.sync 2, %0;" ::"n"(kDrainWarps * 32) : "memory");
    }
    const ulonglong2* my_scales = reinterpret_cast<const ulonglong2*>(row_scales + group * kCols);
    uint64_t acc[kCols / 2];
#pragma unroll
    for (int i = 0; i < kCols / 2; ++i) acc[i] = 0ull;
#pragma unroll 1
    for (int st = 0; st < n_stages; ++st) {
      const uint32_t b = st & 1;
      float w_s[kSub];
      float g_s[kToken ? 1 : kSub][kRowGroups];
#pragma unroll
      for (int s = 0; s < kSub; ++s) {
        w_s[s] = w_next[s];
        if constexpr (!kToken) {
#pragma unroll
          for (int g = 0; g < kRowGroups; ++g) g_s[s][g] = g_next[s][g];
        }
      }
      const int at = st * kSub;
#pragma unroll
      for (int s = 0; s < kSub; ++s) w_next[s] = at + kSub + s < steps ? __ldg(&recs[at + kSub + s].scale) : 0.0f;
      group_scales(at + kSub);
      ok = mbar_wait(acc_full(b), (st >> 1) & 1u, abort_flag, &g_gemm_rows_status, 87);
      if (!ok) break;
      tc_fence_after();
      // Columns at a time, and steps (NT = 32: four, NT = 64: two) whose loads are on their way together: eight warps
      // do not hide the latency of one load after the other.  Steps past the range load stale columns.
      constexpr int kPart = kCols < 32 ? kCols : 32;
      constexpr int kSteps = kCols <= 32 ? 64 / kPart : 1;
#pragma unroll
      for (int s0 = 0; s0 < kSub; s0 += kSteps) {
#pragma unroll
        for (int c0 = 0; c0 < kCols; c0 += kPart) {
          int v[kSteps][kPart];
#pragma unroll
          for (int h = 0; h < kSteps; ++h) {
            const uint32_t col = taddr + b * S::kAccColumns + static_cast<uint32_t>((s0 + h) * NT + c0);
            if constexpr (kPart == 16) tc_ld16(col, v[h]);
            else tc_ld32(col, v[h]);
          }
#pragma unroll
          for (int h = 0; h < kSteps; ++h) {
            if constexpr (kPart == 16) tc_wait_ld(v[h]);
            else tc_wait_ld32(v[h]);
          }
#pragma unroll
          for (int h = 0; h < kSteps; ++h) {
            const int s = s0 + h;
            if (at + s >= steps) break;
            const uint64_t w2 = kRowsOnM ? both(__fmul_rn(kToken ? token_scale : g_s[kToken ? 0 : s][0], w_s[s])) : both(w_s[s]);
#pragma unroll
            for (int i = 0; i < kPart; i += 4) {
              uint64_t scale_a, scale_b;
              if constexpr (kRowsOnM) {
                scale_a = scale_b = w2;
              } else if constexpr (kToken) {
                const ulonglong2 a = my_scales[(c0 + i) / 4];
                scale_a = mul2(a.x, w2);
                scale_b = mul2(a.y, w2);
              } else {
                scale_a = scale_b = both(__fmul_rn(g_s[s][(c0 + i) / 16], w_s[s]));
              }
              const int* e = v[h] + i;
              const uint64_t f0 = pack2(__float_as_uint(__int2float_rn(e[0])), __float_as_uint(__int2float_rn(e[1])));
              const uint64_t f1 = pack2(__float_as_uint(__int2float_rn(e[2])), __float_as_uint(__int2float_rn(e[3])));
              acc[(c0 + i) / 2] = fma2(f0, scale_a, acc[(c0 + i) / 2]);
              acc[(c0 + i) / 2 + 1] = fma2(f1, scale_b, acc[(c0 + i) / 2 + 1]);
            }
            if (kDump && j < p.n_j) {
              const int k = k_begin + at + s;
              const int shift = (recs[at + s].offset_flag & kW4Flag) ? 4 : 0;
#pragma unroll
              for (int i = 0; i < kPart; ++i) {
                const int row = kRowsOnM ? m_row : group * kCols + c0 + i;
                const int column = kRowsOnM ? c0 + i : (quarter & 1) * 32 + lane;
                if (row < p.m) p.acc_dump[((static_cast<int64_t>(row) * p.n_j + j) * n_k + k) * kTile + column] = v[h][i] >> shift;
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      mbar_arrive_lane0(acc_empty(b), lane);
    }
    // The sums go to shared memory over the ring: the last accumulator is only full once every operand
    // has been consumed.  (After a time-out the results are void and copies may land among them.)
    float* xchg = reinterpret_cast<float*>(stages);
#pragma unroll
    for (int i = 0; i < kCols / 2; ++i) {
      float lo, hi;
      unpack2(acc[i], lo, hi);
      const int column = group * kCols + 2 * i;  // of the accumulator
      xchg[kRowsOnM ? m_row * kXchgRow + column : column * kXchgRow + quarter * 32 + lane] = lo;
      xchg[kRowsOnM ? m_row * kXchgRow + column + 1 : (column + 1) * kXchgRow + quarter * 32 + lane] = hi;
    }
  }
  if (*abort_flag != 0) {
    // bulk copies may still be in flight: give them a bounded time to land before the CTA
    // and its shared memory go away
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }

  // ---------------- rows split, split + split_k, ... of the CTA's columns -------------------------
  // The K ranges' sums are added in split order (linear.cu:1339-1343), transformed back and stored, a
  // (row, tile row) pair per warp.  The second barrier keeps every CTA's sums alive until read.
  if (split_k > 1) {
    cluster.sync();
  } else {
    __syncthreads();
  }
  if (warp < kDrainWarps) {
    const int tiles_here = min(2, p.n_j - j0);
    const int owned = p.m > split ? (p.m - split + split_k - 1) / split_k : 0;
    const float* xchg = reinterpret_cast<const float*>(stages);
    const float* remote[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) remote[s] = split_k > 1 ? cluster.map_shared_rank(xchg, s < split_k ? s : 0) : xchg;
    const int64_t n_cols = static_cast<int64_t>(p.n_j) * kTile;
    if (split_k == 1 && p.u_metadata == nullptr) {
      // Eight warps do not hide chains of integer arithmetic: with the row, the tile row and the address worked out for
      // every pair, as below, a pair takes 280 cycles, 9000 for a CTA of 128 rows (128 x 18944 x 1024 17.6 us, now 12.1).
      constexpr int kTogether = 4;  // rows whose loads do not wait for the stores of the row before
      const int tl = tiles_here == 2 ? warp & 1 : 0;
      const int first = tiles_here == 2 ? warp >> 1 : warp, every = kDrainWarps / tiles_here;
      const float* from = xchg + first * S::kXchgRow + tl * kTile + lane;
      const int from_step = every * S::kXchgRow;
      const int64_t to_step = every * n_cols;
      auto store = [&](auto* out) {
        int64_t to = first * n_cols + static_cast<int64_t>(j0 + tl) * kTile + lane;
        int row = first;
        for (; row + (kTogether - 1) * every < p.m; row += kTogether * every) {
          float lo[kTogether], hi[kTogether];
#pragma unroll
          for (int h = 0; h < kTogether; ++h, from += from_step) {
            lo[h] = from[0];
            hi[h] = from[32];
          }
#pragma unroll
          for (int h = 0; h < kTogether; ++h, to += to_step) {
            store_out(out, to, lo[h]);
            store_out(out, to + 32, hi[h]);
          }
        }
        for (; row < p.m; row += every, from += from_step, to += to_step) {
          store_out(out, to, from[0]);
          store_out(out, to + 32, from[32]);
        }
      };
      if (p.out_dtype == AQ_F32) store(static_cast<float*>(p.out));
      else if (p.out_dtype == AQ_BF16) store(static_cast<__nv_bfloat16*>(p.out));
      else store(static_cast<__half*>(p.out));
    } else {
      for (int q = warp; q < owned * tiles_here; q += kDrainWarps) {
        const int row = split + split_k * (q / tiles_here);
        const int tl = q % tiles_here;
        const int offset = row * S::kXchgRow + tl * kTile + lane;
        float a[8], b[8];
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          a[s] = b[s] = 0.0f;
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
        const int j = j0 + tl;
        const int32_t* meta = p.u_metadata ? p.u_metadata + static_cast<int64_t>(j) * 4 * kTile : nullptr;
        if (meta != nullptr && meta[0] != 0) inverse_u_row(lo, hi, meta, lane);
        const int64_t o = static_cast<int64_t>(row) * n_cols + static_cast<int64_t>(j) * kTile + lane;
        store_any(p.out, p.out_dtype, o, lo);
        store_any(p.out, p.out_dtype, o + 32, hi);
      }
    }
  }
  if (split_k > 1) cluster.sync();

  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(S::kTmemColumns))
                 : "memory");
  }
}

template <int NT>
const void* kernel_of(bool token, bool dump) {
  return token ? (dump ? reinterpret_cast<const void*>(gemm_rows_kernel<NT, true, true>) : reinterpret_cast<const void*>(gemm_rows_kernel<NT, true, false>))
               : (dump ? reinterpret_cast<const void*>(gemm_rows_kernel<NT, false, true>) : reinterpret_cast<const void*>(gemm_rows_kernel<NT, false, false>));
}

struct Shape {
  int nt;
  int index;  // 0, 1, 2
  int smem;
  const void* kernels[4];  // [token][dump]
};

const Shape& shape_for(int64_t m) {
  static const Shape shapes[3] = {
      {32, 0, RowsLayout<32>::kSmemBytes, {kernel_of<32>(false, false), kernel_of<32>(false, true), kernel_of<32>(true, false), kernel_of<32>(true, true)}},
      {64, 1, RowsLayout<64>::kSmemBytes, {kernel_of<64>(false, false), kernel_of<64>(false, true), kernel_of<64>(true, false), kernel_of<64>(true, true)}},
      {128, 2, RowsLayout<128>::kSmemBytes, {kernel_of<128>(false, false), kernel_of<128>(false, true), kernel_of<128>(true, false), kernel_of<128>(true, true)}}};
  return shapes[m <= 32 ? 0 : m <= 64 ? 1 : 2];
}

int set_shared_memory(const Shape& shape, int device) {
  static std::once_flag once[64][3];
  cudaError_t status = cudaSuccess;
  std::call_once(once[device & 63][shape.index], [&] {
    for (const void* kernel : shape.kernels) {
      if (status == cudaSuccess) status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, shape.smem);
    }
  });
  return check_cuda(status, "cudaFuncSetAttribute(gemm_rows_kernel)");
}

void fill_config(cudaLaunchConfig_t* config, cudaLaunchAttribute* attr, const Shape& shape, int pairs, int split) {
  config->gridDim = dim3(static_cast<unsigned>(pairs), 1, static_cast<unsigned>(split));
  config->blockDim = dim3(kThreads, 1, 1);
  config->dynamicSmemBytes = static_cast<size_t>(shape.smem);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = static_cast<unsigned>(split);
  config->attrs = attr;
  config->numAttrs = 1;
}

// Clusters of `split` CTAs that can be resident at once; cached per device.
int resident_clusters(const Shape& shape, int split, int device) {
  static std::mutex mutex;
  static int cache[64][3][9];  // 0: not asked yet, -1: failed
  std::lock_guard<std::mutex> lock(mutex);
  int& slot = cache[device & 63][shape.index][split];
  if (slot == 0) {
    int clusters = 0;
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attr[1];
    fill_config(&config, attr, shape, 1, split);
    if (set_shared_memory(shape, device) != AQ_OK || cudaOccupancyMaxActiveClusters(&clusters, shape.kernels[2], &config) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    slot = clusters > 0 ? clusters : -1;
  }
  return slot > 0 ? slot : 0;
}

}  // namespace

// K ranges and their cost by a model in SM cycles: a K step of two tiles (measured 490, 560 and 660 for 32, 64
// and 128 rows), what a CTA costs beside its steps, the exchange (more with every row that changes hands: 128 x 4736 x 5120
// gains 9 us from a second range, which its steps alone would put at 14); clusters in waves.
// `forced` (AQ_OPT_GEMM_SPLIT) >= 1: that number.
int gemm_rows_split(int64_t m, int n_j, int n_k, int forced, double* cost) {
  const int pairs = (n_j + 1) / 2;
  const double step = m <= 32 ? 490.0 : m <= 64 ? 560.0 : 660.0;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) device = 0;
  const Shape& shape = shape_for(m);
  int best = 1;
  double best_cost = 0.0;
  for (int split = 1; split <= 8; ++split) {
    if (forced >= 1 ? split != forced : split > 1 && n_k / split < 4) continue;
    const int at_once = split == 1 ? num_sms() : resident_clusters(shape, split, device);
    if (at_once <= 0 && forced < 1) continue;
    const int waves = at_once > 0 ? (pairs + at_once - 1) / at_once : pairs;
    const double this_cost = static_cast<double>(waves) * ((n_k + split - 1) / split * step + 8000.0) + (split > 1 ? 1500.0 + 40.0 * static_cast<double>(m) : 0.0);
    if (best_cost == 0.0 || this_cost < best_cost) {
      best_cost = this_cost;
      best = split;
    }
  }
  while (best > 1 && n_k / best < 4) --best;
  if (cost != nullptr) *cost = best_cost;
  return best;
}

int launch_gemm_rows(const LinearArgs& a, int split, cudaStream_t stream) {
  int device = 0;
  int rc = check_cuda(cudaGetDevice(&device), "cudaGetDevice");
  if (rc != AQ_OK) return rc;
  const Shape& shape = shape_for(a.m);
  rc = set_shared_memory(shape, device);
  if (rc != AQ_OK) return rc;
  alignas(64) CUtensorMap x_map;
  rc = encode_activation_map(&x_map, a.xq, a.m, a.n_k, shape.nt, shape.nt == 128 ? RowsLayout<128>::kSub : RowsLayout<32>::kSub);
  if (rc != AQ_OK) return rc;
  RowsParams p;
  p.act_scales = a.act_scales;
  p.records = a.records;
  p.payload = a.payload;
  p.u_metadata = a.u_metadata;
  p.out = a.out;
  p.acc_dump = a.acc_dump;
  p.m = static_cast<int>(a.m);
  p.n_j = a.n_j;
  p.n_k = a.n_k;
  p.out_dtype = a.out_dtype;
  cudaLaunchConfig_t config = {};
  cudaLaunchAttribute attr[2];
  fill_config(&config, attr, shape, (a.n_j + 1) / 2, split);
  config.stream = stream;
  if (use_dependent_launch()) {
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    config.numAttrs = 2;
  }
  void* args[] = {&x_map, &p};
  return check_cuda(cudaLaunchKernelExC(&config, shape.kernels[(a.scale_mode == AQ_SCALE_TOKEN ? 2 : 0) + (a.acc_dump != nullptr ? 1 : 0)], args),
                    "row GEMM launch");
}

int take_gemm_rows_status() {
  int status = 0;
  if (cudaMemcpyFromSymbol(&status, g_gemm_rows_status, sizeof(int)) != cudaSuccess) return -1;
  if (status != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_gemm_rows_status, &zero, sizeof(int));
  }
  return status;
}

}  // namespace aq
