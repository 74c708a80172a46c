// One-time re-layout of a layer's artifact tensors into the prepared image.
//
// Source (alignquant/quantization/artifact.py:62-73, 131-199): per-precision arenas
// of 64x64 tiles in "Layout-B" physical order.  Element (k, n) of a tile is byte
//     256*(n/4) + 16*v + k%16,  v = 8*(k/32) + 4*(t/4) + ((t%4) ^ ((n/4)%4)),
//     t = (k/16)%2 + 2*(n%4),
// i.e. every aligned 16-byte vector holds 16 consecutive k of one output column.
// W4 tiles store the same order two values per byte, low nibble first.
//
// Destination (include/alignquant_b200.h): tiles in (j, k) order behind an array of
// 8-byte records.  A W8 tile is 64 rows (output columns n) of 64 bytes (k), the
// 16-byte chunk c = k/16 of row n stored at slot c ^ ((n/2) % 4): the K-major
// 64-byte-swizzle operand layout of tcgen05.mma, which also makes the small-M
// kernels' 16-byte shared-memory reads conflict free.  A W4 tile is 64 rows of 32
// bytes: chunk h = k/32 holds k%32 < 16 in the low nibbles and k%32 >= 16 in the high
// nibbles of the same bytes, so one shift-and-mask widens a word.
#include "aq_common.cuh"

namespace aq {
namespace {

__device__ __forceinline__ int layout_b_vector(int n, int k16) {
  const int vs = n >> 2;
  const int t = (k16 & 1) + 2 * (n & 3);
  const int v = 8 * (k16 >> 1) + 4 * (t >> 2) + ((t & 3) ^ (vs & 3));
  return vs * 16 + v;  // index of the 16-element vector inside the tile
}

// A CTA takes eight consecutive tiles of a tile row: their place follows from one count of the W4 tiles
// before them, and the loads of all eight are in flight together.  With a tile per CTA the kernel was a
// chain of four dependent loads per 2 or 4 KiB (16384 x 3072: 28 us; now the call's 19 us are Python's).
constexpr int kRepackTiles = 8;

__global__ void __launch_bounds__(256) repack_kernel(
    const uint8_t* __restrict__ state_bits, const uint8_t* __restrict__ w4_payload,
    const float* __restrict__ w4_scales, const int8_t* __restrict__ w8_payload,
    const float* __restrict__ w8_scales, const int32_t* __restrict__ w4_row_offsets,
    const int32_t* __restrict__ w8_row_offsets, int n_k, int groups, TileRecord* __restrict__ records,
    uint8_t* __restrict__ payload) {
  __shared__ int warp_count[8];
  const int j = static_cast<int>(blockIdx.x / groups);
  const int k0 = static_cast<int>(blockIdx.x % groups) * kRepackTiles;
  const int64_t row_base = static_cast<int64_t>(j) * n_k;
  const int32_t first4 = __ldg(&w4_row_offsets[j]), first8 = __ldg(&w8_row_offsets[j]);
  auto is_w4_tile = [&](int k) {
    const int64_t bit = row_base + k;
    return (__ldg(&state_bits[bit >> 3]) >> (bit & 7)) & 1;
  };
  uint32_t w4_mask = 0;  // bit i: tile k0 + i is W4
#pragma unroll
  for (int i = 0; i < kRepackTiles; ++i) {
    if (k0 + i < n_k) w4_mask |= static_cast<uint32_t>(is_w4_tile(k0 + i)) << i;
  }

  // W4 tiles of row j that precede k0
  int count = 0;
  for (int i = threadIdx.x; i < k0; i += 256) count += is_w4_tile(i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
  if ((threadIdx.x & 31) == 0) warp_count[threadIdx.x >> 5] = count;
  __syncthreads();
  int before4 = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) before4 += warp_count[w];
  const int64_t group4 = static_cast<int64_t>(first4) + before4;
  const int64_t group8 = static_cast<int64_t>(first8) + (k0 - before4);
  const int64_t group_units = group4 + 2 * group8;  // 2048-byte units

  if (threadIdx.x < kRepackTiles && k0 + static_cast<int>(threadIdx.x) < n_k) {
    const int i = threadIdx.x;
    const int w4_before = __popc(w4_mask & ((1u << i) - 1u));
    const bool is_w4 = (w4_mask >> i) & 1u;
    TileRecord rec;
    rec.offset_flag = static_cast<uint32_t>(group_units + 2 * i - w4_before) | (is_w4 ? kW4Flag : 0u);
    rec.scale = is_w4 ? w4_scales[group4 + w4_before] * 0.0625f : w8_scales[group8 + i - w4_before];
    records[row_base + k0 + i] = rec;
  }

  // W8 tile: destination chunk r = 4*n + slot  <-  Layout-B vector of (n, k16 = slot ^ ((n/2)%4)).
  // W4 tile: destination chunk u = 2*n + h; a source vector of 16 int4 is 8 bytes, those of
  // k%32 in [0,16) (nibble i = k offset i) and k%32 in [16,32) make a chunk.
  const int r8 = threadIdx.x;
  const int from8 = layout_b_vector(r8 >> 2, (r8 & 3) ^ ((r8 >> 3) & 3));
  const int n4 = (threadIdx.x & 127) >> 1, h4 = threadIdx.x & 1;
  const int from4a = layout_b_vector(n4, 2 * h4), from4b = layout_b_vector(n4, 2 * h4 + 1);
  uint4 v[kRepackTiles];
#pragma unroll
  for (int i = 0; i < kRepackTiles; ++i) {
    if (k0 + i >= n_k) break;
    const int w4_before = __popc(w4_mask & ((1u << i) - 1u));
    if (!((w4_mask >> i) & 1u)) {
      v[i] = __ldg(reinterpret_cast<const uint4*>(w8_payload + (group8 + i - w4_before) * kW8TileBytes) + from8);
    } else if (threadIdx.x < 128) {
      const uint2* src = reinterpret_cast<const uint2*>(w4_payload + (group4 + w4_before) * kW4TileBytes);
      const uint2 a = __ldg(src + from4a), b = __ldg(src + from4b);
      v[i] = make_uint4(a.x, a.y, b.x, b.y);
    }
  }
#pragma unroll
  for (int i = 0; i < kRepackTiles; ++i) {
    if (k0 + i >= n_k) break;
    const int w4_before = __popc(w4_mask & ((1u << i) - 1u));
    uint4* dst = reinterpret_cast<uint4*>(payload + (group_units + 2 * i - w4_before) * kW4TileBytes);
    if (!((w4_mask >> i) & 1u)) {
      dst[r8] = v[i];
    } else if (threadIdx.x < 128) {
      const uint64_t av = (static_cast<uint64_t>(v[i].y) << 32) | v[i].x;
      const uint64_t bv = (static_cast<uint64_t>(v[i].w) << 32) | v[i].z;
      uint32_t out[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        uint32_t word = 0;
#pragma unroll
        for (int byte = 0; byte < 4; ++byte) {
          const int e = 4 * w + byte;
          const uint32_t low = static_cast<uint32_t>(av >> (4 * e)) & 0xfu;
          const uint32_t high = static_cast<uint32_t>(bv >> (4 * e)) & 0xfu;
          word |= (low | (high << 4)) << (8 * byte);
        }
        out[w] = word;
      }
      dst[threadIdx.x] = make_uint4(out[0], out[1], out[2], out[3]);
    }
  }
  // The projections fetch the image before their grid_dependency_wait, so the wait is not what makes it visible to
  // them: it has to have reached device scope when the last CTA ends, which is when a dependent kernel may begin.
  __threadfence();
}

}  // namespace

int launch_repack(const uint8_t* state_bits, const uint8_t* w4_payload, const float* w4_scales,
                  const int8_t* w8_payload, const float* w8_scales, const int32_t* w4_row_offsets,
                  const int32_t* w8_row_offsets, int n_j, int n_k, void* prepared,
                  cudaStream_t stream) {
  const int64_t tiles = static_cast<int64_t>(n_j) * n_k;
  TileRecord* records = static_cast<TileRecord*>(prepared);
  uint8_t* payload = static_cast<uint8_t*>(prepared) + records_bytes(tiles);
  const int groups = (n_k + kRepackTiles - 1) / kRepackTiles;
  repack_kernel<<<static_cast<unsigned>(static_cast<int64_t>(n_j) * groups), 256, 0, stream>>>(
      state_bits, w4_payload, w4_scales, w8_payload, w8_scales, w4_row_offsets, w8_row_offsets,
      n_k, groups, records, payload);
  return check_cuda(cudaGetLastError(), "repack launch");
}

}  // namespace aq
