// Device-side building blocks shared by the fused TTT inner-loop kernels (sm_100a).
//
// Role: what the reference's tile library provides to its fused kernels (shared-memory tiles with an XOR
// swizzle, per-thread register tiles, cooperative loads/stores, "mma", row/column reductions:
// rust/thundercube/src/tiles/st.rs:9-47, tiles/mma.rs:71-187, cube/reduce.rs:131-259) is provided here by
//   * TMA tile loads/stores (cp.async.bulk.tensor, 128-byte swizzle) completed on mbarriers,
//   * ldmatrix / movmatrix fragment moves,
//   * warp-level tensor-core products mma.sync.m16n8k16 (bf16 operands, f32 accumulate),
//   * warp-shuffle row reductions plus a tiny shared-memory exchange across the four warps of a CTA.
//
// Data layout convention used by every kernel: a "tile" is 16 tokens (rows) x 64 features (columns).
// Warp w of the CTA owns columns [16w, 16w+16).  Inside a warp, lane = 4*g + t holds, of its 16x16 slab,
// rows {g, g+8} and columns {8*nt + 2t, 8*nt + 2t + 1 : nt = 0,1}: this is the accumulator layout of
// mma.m16n8k16, so products chain without moving data.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ttt {

constexpr int CS = 16;        // mini-batch length (tokens per stage)
constexpr int HD = 64;        // head dim
constexpr int NTHREADS = 128; // 4 warps per (batch, head) stream
constexpr uint32_t TILE_BF16_BYTES = CS * HD * 2;  // 2048
constexpr uint32_t TILE_F32_BYTES = CS * HD * 4;   // 4096
constexpr uint32_t SPIN_LIMIT = 1u << 22;          // bounded mbarrier wait (iterations of try_wait)

// status words written by kernels: [0] error code, [1] where, [2] block, [3] stage
enum : uint32_t { KST_OK = 0, KST_TIMEOUT = 6 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ----------------------------------------------------------------------------------------------------
// mbarrier + TMA
// ----------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One lane of a converged warp, the same every time.  Unlike a comparison of the lane number it leaves the addresses of
// what follows in the uniform registers that the bulk-copy instructions want.
__device__ __forceinline__ bool elect_one() {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(v));
  return v != 0;
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// Returns false if the phase did not complete within SPIN_LIMIT polls (caller reports and leaves).
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
  }
  return false;
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// 2-D tiled TMA load into this CTA's shared memory, completion counted in bytes on `bar`.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tm, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tm), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// 2-D tiled TMA store from shared memory (bulk async-group completion).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, int x, int y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(tm), "r"(x),
               "r"(y), "r"(src)
               : "memory");
}
// Untiled bulk copy global -> shared (both 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bulk_store_1d(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* tm) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tm) : "memory");
}

// ----------------------------------------------------------------------------------------------------
// Swizzled tile addressing (matches CU_TENSOR_MAP_SWIZZLE_128B; tile bases are 1024-byte aligned)
// ----------------------------------------------------------------------------------------------------
// bf16 tile [16][64]: 128 bytes per row.
__device__ __forceinline__ uint32_t off_bf16(int row, int col) {
  return static_cast<uint32_t>(row * 128 + ((((col >> 3) ^ row) & 7) << 4) + ((col & 7) << 1));
}
// f32 tile [16][64] stored as two half tiles [16][32] of 128-byte rows (2048 bytes each).
__device__ __forceinline__ uint32_t off_f32(int row, int col) {
  return static_cast<uint32_t>(((col >> 5) << 11) + row * 128 + (((((col & 31) >> 2) ^ row) & 7) << 4) +
                               ((col & 3) << 2));
}

// ----------------------------------------------------------------------------------------------------
// Fragment moves
// ----------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// the counterpart of ldsm_x4: the same lanes' addresses, the same fragments
__device__ __forceinline__ void stsm_x4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Transpose an 8x8 matrix of 16-bit values held one register per lane across the warp.
__device__ __forceinline__ uint32_t movm_t(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t a0, const uint32_t a1, const uint32_t a2,
                                         const uint32_t a3, const uint32_t b0, const uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// pack two floats into bf16x2 (lo = first element)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// ----------------------------------------------------------------------------------------------------
// Operand planes.  NP = 1: operands are bf16.  NP = 3: a float is carried as three bf16 planes
// (x = p0 + p1 + p2, 24 mantissa bits) and a product uses the six plane pairs whose weight is >= 2^-16,
// which reproduces float32 operand precision on the bf16 tensor-core path.
// ----------------------------------------------------------------------------------------------------
template <int NP>
struct Pk {  // one 32-bit fragment register position (a pair of elements), NP planes
  uint32_t p[NP];
};

template <int NP>
__device__ __forceinline__ Pk<NP> split_pack(float x, float y);
template <>
__device__ __forceinline__ Pk<1> split_pack<1>(float x, float y) {
  Pk<1> r;
  r.p[0] = pack_bf16(x, y);
  return r;
}
template <>
__device__ __forceinline__ Pk<3> split_pack<3>(float x, float y) {
  Pk<3> r;
  float2 v = make_float2(x, y);
  const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    r.p[i] = pack_bf16(v.x, v.y);
    if (i < 2) v = __ffma2_rn(make_float2(bf16_lo(r.p[i]), bf16_hi(r.p[i])), minus, v);  // the remainder, exact
  }
  return r;
}

// One k-step of N independent products C_n += A_n . B_n.
//
// float32 (three planes): the tensor core adds products to its accumulator with truncation, which biases long chained sums,
// so each k-step is summed from zero (the five cross terms and the leading term apart) and joined to the running float32
// accumulator with ordinary round-to-nearest adds, packed in pairs.  The tiles of a call take turns, so that two chains of
// dependent products are in flight; 96 streams of 64 stages: forward 207 -> 205 us, backward 502 -> 453 us.
template <int NP, int N>
__device__ __forceinline__ void mma_np_n(float (*const (&c)[N])[4], const Pk<NP> (*const (&a)[N])[4],
                                         const Pk<NP> (*const (&b)[N])[2]) {
  auto mma1 = [&](float (&d)[4], int n, int pa, int pb) {
    mma_bf16(d, (*a[n])[0].p[pa], (*a[n])[1].p[pa], (*a[n])[2].p[pa], (*a[n])[3].p[pa], (*b[n])[0].p[pb], (*b[n])[1].p[pb]);
  };
  if constexpr (NP == 1) {
#pragma unroll
    for (int n = 0; n < N; ++n) mma1(*c[n], n, 0, 0);
  } else {
    float x[N][4] = {}, h[N][4] = {};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int n = 0; n < N; ++n) {
        constexpr int PA[6] = {1, 2, 0, 0, 1, 0}, PB[6] = {1, 0, 2, 0, 0, 1};
        if (i == 3) mma1(h[n], n, 0, 0);
        else mma1(x[n], n, PA[i], PB[i]);
      }
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const float2 lo = make_float2(x[n][i], x[n][i + 1]);
        const float2 v = __fadd2_rn(make_float2((*c[n])[i], (*c[n])[i + 1]),
                                    __fadd2_rn(make_float2(h[n][i], h[n][i + 1]), lo));
        (*c[n])[i] = v.x;
        (*c[n])[i + 1] = v.y;
      }
  }
}
template <int NP>
__device__ __forceinline__ void mma_np(float (&c)[4], const Pk<NP> (&a)[4], const Pk<NP> (&b)[2]) {
  mma_np_n<NP, 1>({&c}, {&a}, {&b});
}
template <int NP>
__device__ __forceinline__ void mma_np2(float (&c0)[4], const Pk<NP> (&a0)[4], const Pk<NP> (&b0)[2], float (&c1)[4],
                                        const Pk<NP> (&a1)[4], const Pk<NP> (&b1)[2]) {
  mma_np_n<NP, 2>({&c0, &c1}, {&a0, &a1}, {&b0, &b1});
}

// two k-steps of two products (the joins of one accumulator follow one another, so the sums are those of two calls of mma_np2):
// a product of the float32 planes waits for the one before it, and a lone warp on its scheduler has only its own others to
// fill that
template <int NP>
__device__ __forceinline__ void mma_np2x2(float (&c0)[4], float (&c1)[4], const Pk<NP> (&a0)[4], const Pk<NP> (&b00)[2],
                                          const Pk<NP> (&b01)[2], const Pk<NP> (&a1)[4], const Pk<NP> (&b10)[2],
                                          const Pk<NP> (&b11)[2]) {
  mma_np_n<NP, 4>({&c0, &c1, &c0, &c1}, {&a0, &a0, &a1, &a1}, {&b00, &b01, &b10, &b11});
}

template <int NP>
__device__ __forceinline__ Pk<NP> movm_t_np(const Pk<NP>& a) {
  Pk<NP> r;
#pragma unroll
  for (int i = 0; i < NP; ++i) r.p[i] = movm_t(a.p[i]);
  return r;
}

// ldmatrix x4 over NP planes (plane stride in bytes)
template <int NP>
__device__ __forceinline__ void ldsm_np(Pk<NP> (&r)[4], uint32_t addr, uint32_t plane_stride, bool trans) {
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    uint32_t v[4];
    if (trans)
      ldsm_x4_t(v, addr + p * plane_stride);
    else
      ldsm_x4(v, addr + p * plane_stride);
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i].p[p] = v[i];
  }
}

// Lane address helpers for ldmatrix.x4 on a swizzled bf16 tile [16][64].
//  A operand (16 rows x 16 k-columns starting at kc): regs = {rows0-7/k-lo, rows8-15/k-lo, rows0-7/k-hi, rows8-15/k-hi}
__device__ __forceinline__ uint32_t lane_off_A(int lane, int kc) {
  const int m = lane >> 3, r = lane & 7;
  return off_bf16(r + ((m & 1) << 3), kc + ((m >> 1) << 3));
}
//  B operand read from a tile stored [n][k] (rows index the product's N, columns its K), both 8-row n-tiles,
//  16 k-columns starting at kc: regs = {n0-7/k-lo, n0-7/k-hi, n8-15/k-lo, n8-15/k-hi}
__device__ __forceinline__ uint32_t lane_off_B_nk(int lane, int kc) {
  const int m = lane >> 3, r = lane & 7;
  return off_bf16(r + ((m >> 1) << 3), kc + ((m & 1) << 3));
}
//  B operand read (with .trans) from a tile stored [k][n] (rows index the product's K = 16 tokens, columns
//  its N): two adjacent 8-column n-tiles starting at nc: regs = {k0-7/n-tile0, k8-15/n-tile0, k0-7/n-tile1, k8-15/n-tile1}
__device__ __forceinline__ uint32_t lane_off_B_kn(int lane, int nc) {
  const int m = lane >> 3, r = lane & 7;
  return off_bf16(r + ((m & 1) << 3), nc + ((m >> 1) << 3));
}

// ----------------------------------------------------------------------------------------------------
// Packed float32x2 arithmetic (one instruction per column pair on sm_100).
// ----------------------------------------------------------------------------------------------------
typedef float2 F2;
__device__ __forceinline__ F2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ F2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ F2 f2fma(F2 a, F2 b, F2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ F2 f2mul(F2 a, F2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ F2 f2add(F2 a, F2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ F2 f2sub(F2 a, F2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ F2 f2neg(F2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float f2hsum(F2 a) { return a.x + a.y; }
// accumulator quad {r0e0, r0e1, r1e0, r1e1} viewed as the column pair of row r
__device__ __forceinline__ F2 pr(const float (&c)[4], int r) { return make_float2(c[2 * r], c[2 * r + 1]); }

// ----------------------------------------------------------------------------------------------------
// Reductions
// ----------------------------------------------------------------------------------------------------
// sum over the 4 lanes that share a row (lane bits 0,1)
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}
// sum over the 8 lanes that share a column pair (lane bits 2,3,4)
__device__ __forceinline__ float col_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  return v;
}

template <typename T>
__device__ __forceinline__ float ld_as_float(const void* base, size_t idx);
template <>
__device__ __forceinline__ float ld_as_float<float>(const void* base, size_t idx) {
  return static_cast<const float*>(base)[idx];
}
template <>
__device__ __forceinline__ float ld_as_float<__nv_bfloat16>(const void* base, size_t idx) {
  return __bfloat162float(static_cast<const __nv_bfloat16*>(base)[idx]);
}
template <typename T>
__device__ __forceinline__ void st_from_float(void* base, size_t idx, float v);
template <>
__device__ __forceinline__ void st_from_float<float>(void* base, size_t idx, float v) {
  static_cast<float*>(base)[idx] = v;
}
template <>
__device__ __forceinline__ void st_from_float<__nv_bfloat16>(void* base, size_t idx, float v) {
  static_cast<__nv_bfloat16*>(base)[idx] = __float2bfloat16_rn(v);
}


// ---- tensor memory as a per-thread scratchpad (no tensor-core instruction touches it) ---------------------------
// A warp can address the 32 tensor-memory lanes of its quarter (warp index % 4) only, and with the 32x32b shape lane l
// of the warp gets lane 32 (warp % 4) + l: N consecutive columns of that lane are N private 32-bit words of the
// thread.  A kernel whose per-thread float32 state crowds its registers keeps it there between the places that use
// it: a load + store round trip of 32 columns costs about 100 cycles (measured by probe_chain_latency.cu).
// taddr = allocation base + (first lane of the quarter << 16) + column.
__device__ __forceinline__ void tmem_alloc(uint32_t smem_slot, int columns) {  // one whole warp; a power of 2 >= 32
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, int columns) {  // the warp that allocated
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}
__device__ __forceinline__ void tmem_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 32 columns <-> an [8][4] register array (the accumulator fragments of eight 16 x 8 tiles).  The load waits for its
// data; the store does not wait: tmem_wait_st() before the next load of the same columns.
__device__ __forceinline__ void tmem_ld_8x4(uint32_t taddr, float (&r)[8][4]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=f"(r[0][0]), "=f"(r[0][1]), "=f"(r[0][2]), "=f"(r[0][3]), "=f"(r[1][0]), "=f"(r[1][1]), "=f"(r[1][2]), "=f"(r[1][3]), "=f"(r[2][0]), "=f"(r[2][1]), "=f"(r[2][2]), "=f"(r[2][3]), "=f"(r[3][0]), "=f"(r[3][1]), "=f"(r[3][2]), "=f"(r[3][3]), "=f"(r[4][0]), "=f"(r[4][1]), "=f"(r[4][2]), "=f"(r[4][3]), "=f"(r[5][0]), "=f"(r[5][1]), "=f"(r[5][2]), "=f"(r[5][3]), "=f"(r[6][0]), "=f"(r[6][1]), "=f"(r[6][2]), "=f"(r[6][3]), "=f"(r[7][0]), "=f"(r[7][1]), "=f"(r[7][2]), "=f"(r[7][3])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_8x4(uint32_t taddr, const float (&r)[8][4]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
      ::"f"(r[0][0]), "f"(r[0][1]), "f"(r[0][2]), "f"(r[0][3]), "f"(r[1][0]), "f"(r[1][1]), "f"(r[1][2]), "f"(r[1][3]), "f"(r[2][0]), "f"(r[2][1]), "f"(r[2][2]), "f"(r[2][3]), "f"(r[3][0]), "f"(r[3][1]), "f"(r[3][2]), "f"(r[3][3]), "f"(r[4][0]), "f"(r[4][1]), "f"(r[4][2]), "f"(r[4][3]), "f"(r[5][0]), "f"(r[5][1]), "f"(r[5][2]), "f"(r[5][3]), "f"(r[6][0]), "f"(r[6][1]), "f"(r[6][2]), "f"(r[6][3]), "f"(r[7][0]), "f"(r[7][1]), "f"(r[7][2]), "f"(r[7][3]), "r"(taddr)
      : "memory");
}

// ---- tcgen05.mma --------------------------------------------------------------------------------------------------
// shared-memory matrix descriptor for a K-major bf16 tile of 128-byte rows with 128-byte swizzle: start address >> 4,
// stride between 8-row groups = 1024 bytes, descriptor version 1 (sm_100), layout type 2 (SWIZZLE_128B)
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}
// instruction descriptor, kind::f16: D float32 (bit 4), A and B bf16 (bits 7, 10), both K-major, N >> 3 at bit 17,
// M >> 4 at bit 24
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {  // N: a multiple of 16, 16..256, at M = 128
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ---- programmatic dependent launch ------------------------------------------------------------------------------
// One element of TokenEtaParams, in two halves with the kernel's own work between them (the loads are on their way during it)
struct TokenEtaElement {
  __nv_bfloat16 a, b;
  template <class P>
  __device__ __forceinline__ void load(const P& p, int i) {
    if (i < p.n) {
      a = static_cast<const __nv_bfloat16*>(p.idx)[i];
      b = static_cast<const __nv_bfloat16*>(p.learnable)[i];
    }
  }
  template <class P>
  __device__ __forceinline__ void store(const P& p, int i) const {
    if (i < p.n) {  // the sum rounded as an addition of its own would leave it; a NaN stays one
      const float s = __bfloat162float(__float2bfloat16_rn(__bfloat162float(a) + __bfloat162float(b)));
      static_cast<__nv_bfloat16*>(p.out)[i] = __float2bfloat16_rn(s < 0.f ? 0.f : s);
    }
  }
};

// A kernel launched with launch_dependent may begin while the kernel before it on the stream drains: its launch and
// prologue (and loads of data that neither the kernel before nor an unfinished one writes) are off the chain.
// pdl_wait: everything before on the stream is complete and visible.  pdl_go: the next kernel may begin; called after
// pdl_wait, or by a kernel that is only ever launched behind everything before it (the scans of the backwards), so that at most
// one kernel is unfinished when a later one starts.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Both, for a kernel that reads nothing before: only its launch and what it sets up for itself overlap the kernel before it.  (The
// products, the prologue, the epilogue and the three-group scan of a layer: 1 x 1001 tokens x 768 107 -> 97 us, 4 x 43 tokens x 1024
// 57 -> 47, a token of 51 sequences as graphs replay it 35.8 -> 27.0.)  Only where it does not matter which SMs the kernel before
// leaves first: blocks that several to an SM are to be spread evenly fill those (ttt_linear_fwd.cu).
__device__ __forceinline__ void pdl_join() {
  pdl_wait();
  pdl_go();
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace ttt
