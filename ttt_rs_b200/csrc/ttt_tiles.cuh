// Shared-memory tile formats per element type, and the per-thread "slab" (register tile) helpers.
//
// bf16 I/O: a tile is one swizzled bf16 plane written directly by TMA; tensor-core operands are read from it
// with ldmatrix and element-wise code reads the same bytes.
// f32 I/O: TMA lands the raw float tile (two swizzled 128-byte-row halves); all threads then split it into
// three bf16 planes (see Pk<3>) that ldmatrix reads, while element-wise code reads the raw floats.
#pragma once

#include <type_traits>

#include "ttt_common.cuh"

namespace ttt {

template <typename T>
struct TileFmt;

template <>
struct TileFmt<__nv_bfloat16> {
  static constexpr int NP = 1;
  static constexpr uint32_t RAW_BYTES = TILE_BF16_BYTES;
  static constexpr uint32_t PLANE_OFF = 0;              // plane 0 is the raw tile
  static constexpr uint32_t BYTES = TILE_BF16_BYTES;    // per tile, multiple of 1024
  static constexpr uint32_t ELT = 2;
  static constexpr int TMA_BOXES = 1;                   // one [16 x 64] box
  static constexpr int TMA_BOX_COLS = 64;
};
template <>
struct TileFmt<float> {
  static constexpr int NP = 3;
  static constexpr uint32_t RAW_BYTES = TILE_F32_BYTES;
  static constexpr uint32_t PLANE_OFF = TILE_F32_BYTES;
  static constexpr uint32_t BYTES = TILE_F32_BYTES + 3 * TILE_BF16_BYTES;  // 10240
  static constexpr uint32_t ELT = 4;
  static constexpr int TMA_BOXES = 2;                   // two [16 x 32] boxes
  static constexpr int TMA_BOX_COLS = 32;
};

// element pair (row, col..col+1), col even, from the raw tile
template <typename T>
__device__ __forceinline__ float2 ld_pair(uint32_t tile, int row, int col);
template <>
__device__ __forceinline__ float2 ld_pair<__nv_bfloat16>(uint32_t tile, int row, int col) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(tile + off_bf16(row, col)));
  return make_float2(bf16_lo(v), bf16_hi(v));
}
template <>
__device__ __forceinline__ float2 ld_pair<float>(uint32_t tile, int row, int col) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(tile + off_f32(row, col)));
  return v;
}
template <typename T>
__device__ __forceinline__ void st_pair(uint32_t tile, int row, int col, float x, float y);
template <>
__device__ __forceinline__ void st_pair<__nv_bfloat16>(uint32_t tile, int row, int col, float x, float y) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile + off_bf16(row, col)), "r"(pack_bf16(x, y)) : "memory");
}
template <>
__device__ __forceinline__ void st_pair<float>(uint32_t tile, int row, int col, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(tile + off_f32(row, col)), "f"(x), "f"(y) : "memory");
}

// f32 only: split a raw float tile into its three bf16 operand planes. All 128 threads take part.
__device__ __forceinline__ void split_tile_f32(uint32_t tile, int tid) {
  const int row = tid >> 3, c0 = (tid & 7) << 3;
  float v[8];
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(tile + off_f32(row, c0)));
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(tile + off_f32(row, c0 + 4)));
  uint32_t pl[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const Pk<3> s = split_pack<3>(v[2 * i], v[2 * i + 1]);
    pl[0][i] = s.p[0];
    pl[1][i] = s.p[1];
    pl[2][i] = s.p[2];
  }
  const uint32_t dst = tile + TileFmt<float>::PLANE_OFF + off_bf16(row, c0);
#pragma unroll
  for (int p = 0; p < 3; ++p)
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + p * TILE_BF16_BYTES), "r"(pl[p][0]),
                 "r"(pl[p][1]), "r"(pl[p][2]), "r"(pl[p][3])
                 : "memory");
}

// Issue the TMA load(s) of one [16 x 64] tile whose first row is `row0` of the 2-D view [rows, 64].
template <typename T>
__device__ __forceinline__ void tma_load_tile(uint32_t tile, const CUtensorMap* tm, int row0, uint32_t bar) {
  if constexpr (TileFmt<T>::TMA_BOXES == 1) {
    tma_load_2d(tile, tm, 0, row0, bar);
  } else {
    tma_load_2d(tile, tm, 0, row0, bar);
    tma_load_2d(tile + 2048, tm, 32, row0, bar);
  }
}
template <typename T>
__device__ __forceinline__ void tma_store_tile(const CUtensorMap* tm, int row0, uint32_t tile) {
  if constexpr (TileFmt<T>::TMA_BOXES == 1) {
    tma_store_2d(tm, 0, row0, tile);
  } else {
    tma_store_2d(tm, 0, row0, tile);
    tma_store_2d(tm, 32, row0, tile + 2048);
  }
}

// One of the caller's tiles, as the TTT-Linear kernels hold it.  SEG = 64: the tile above.  SEG = 32: the tiles of a PAIR of
// 32-wide heads side by side, so that the 64-wide kernels serve two such streams at once: two boxes of 16 rows x 32 columns
// of the 2-D view [B*H*seq, 32], one per head, the second behind the first.  In float32 a box row is 128 bytes and the pair
// has the layout of the 64-wide tile (two 128-byte-swizzled halves); in bf16 it is 64 bytes, swizzled over 64 bytes.
template <typename T, int SEG>
__device__ __forceinline__ uint32_t off_io(int row, int col) {
  if constexpr (sizeof(T) == 4) return off_f32(row, col);
  else if constexpr (SEG == 64) return off_bf16(row, col);
  else return static_cast<uint32_t>(((col >> 5) << 10) + row * 64 + (((((col & 31) >> 3) ^ (row >> 1)) & 3) << 4) + ((col & 7) << 1));
}
template <typename T, int SEG>
__device__ __forceinline__ float2 ld_io(uint32_t tile, int row, int col) {
  const uint32_t a = tile + off_io<T, SEG>(row, col);
  if constexpr (sizeof(T) == 4) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
  } else {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
    return make_float2(bf16_lo(v), bf16_hi(v));
  }
}
template <typename T, int SEG>
__device__ __forceinline__ void st_io(uint32_t tile, int row, int col, float x, float y) {
  const uint32_t a = tile + off_io<T, SEG>(row, col);
  if constexpr (sizeof(T) == 4) asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(a), "f"(x), "f"(y) : "memory");
  else asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(pack_bf16(x, y)) : "memory");
}
// ldmatrix.x4 lane offset into the tile's operand planes, columns kc..kc+15 (lane_off_A, which is also lane_off_B_kn)
template <typename T, int SEG>
__device__ __forceinline__ uint32_t lane_off_io(int lane, int kc) {
  if constexpr (sizeof(T) == 2 && SEG == 32) return off_io<T, SEG>((lane & 7) + (((lane >> 3) & 1) << 3), kc + ((lane >> 4) << 3));
  else return lane_off_A(lane, kc);
}
// A warp's 16 x 16 slab of a tile, columns nb..nb+15, as column pairs x[nt][r]: in bf16 the four pairs of a thread are the four
// 8 x 8 blocks of one ldmatrix / stmatrix, in place of an access each with an address of its own.
template <typename T, int SEG>
__device__ __forceinline__ void ld_slab(uint32_t tile, int lane, int nb, float2 (&x)[2][2]) {
  if constexpr (sizeof(T) == 2) {
    uint32_t v[4];
    ldsm_x4(v, tile + lane_off_io<T, SEG>(lane, nb));
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i >> 1][i & 1] = make_float2(bf16_lo(v[i]), bf16_hi(v[i]));
  } else {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int r = 0; r < 2; ++r) x[nt][r] = ld_io<T, SEG>(tile, (lane >> 2) + 8 * r, nb + 8 * nt + 2 * (lane & 3));
  }
}
template <typename T, int SEG>
__device__ __forceinline__ void st_slab(uint32_t tile, int lane, int nb, const float2 (&x)[2][2]) {
  if constexpr (sizeof(T) == 2) {
    stsm_x4(tile + lane_off_io<T, SEG>(lane, nb), pack_bf16(x[0][0].x, x[0][0].y), pack_bf16(x[0][1].x, x[0][1].y),
            pack_bf16(x[1][0].x, x[1][0].y), pack_bf16(x[1][1].x, x[1][1].y));
  } else {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int r = 0; r < 2; ++r) st_io<T, SEG>(tile, (lane >> 2) + 8 * r, nb + 8 * nt + 2 * (lane & 3), x[nt][r].x, x[nt][r].y);
  }
}
// Operand planes of a 16 x 16 block whose fragments are b[nt][r] (rows 8r.., columns 8nt.. of it): `at` is the address of
// the planes plus lane_off_A of the block's first column.
template <int NP>
__device__ __forceinline__ void stsm_np(uint32_t at, const Pk<NP>& b00, const Pk<NP>& b01, const Pk<NP>& b10, const Pk<NP>& b11) {
#pragma unroll
  for (int p = 0; p < NP; ++p) stsm_x4(at + p * TILE_BF16_BYTES, b00.p[p], b01.p[p], b10.p[p], b11.p[p]);
}
// `stream` (SEG = 32: pair) and first token of the tile; `seq` tokens per stream
template <typename T, int SEG>
__device__ __forceinline__ void tma_load_io(uint32_t tile, const CUtensorMap* tm, int stream, int t0, int seq, uint32_t bar) {
  if constexpr (SEG == 64) {
    tma_load_tile<T>(tile, tm, stream * seq + t0, bar);
  } else {
    tma_load_2d(tile, tm, 0, (2 * stream) * seq + t0, bar);
    tma_load_2d(tile + TileFmt<T>::RAW_BYTES / 2, tm, 0, (2 * stream + 1) * seq + t0, bar);
  }
}
template <typename T, int SEG>
__device__ __forceinline__ void tma_store_io(const CUtensorMap* tm, int stream, int t0, int seq, uint32_t tile) {
  if constexpr (SEG == 64) {
    tma_store_tile<T>(tm, stream * seq + t0, tile);
  } else {
    tma_store_2d(tm, 0, (2 * stream) * seq + t0, tile);
    tma_store_2d(tm, 0, (2 * stream + 1) * seq + t0, tile + TileFmt<T>::RAW_BYTES / 2);
  }
}
// Byte `o` of such a tile (operand planes included) belongs to a row that a mini-batch of MB tokens does not fill.
template <typename T, int SEG, int MB>
__device__ __forceinline__ bool io_pad(uint32_t o) {
  constexpr uint32_t BOX = (SEG == 32) ? TileFmt<T>::RAW_BYTES / 2 : 2048, ROW = BOX / CS;
  return o >= TileFmt<T>::RAW_BYTES || (o % BOX) >= MB * ROW;
}

}  // namespace ttt
