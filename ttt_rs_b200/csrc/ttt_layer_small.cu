// The outer layer's steps either side of the inner loop for few tokens (decode steps, short prompts), bf16: the projections
// with everything the prologue does, and the post norm (+ gate) with the output projection, one launch each.
//
// What bounds them: at 8 rows the weights (a few MB, resident in L2 from one step to the next) have to reach the SMs once;
// on 128 x 256 tensor-core tiles that is ten CTAs' work and a chain of loads, 7.4 us per product.  Here a CTA owns 16 (or 8)
// output features and its eight warps split the contraction, so 145 CTAs (2304 + 12 features) pull the weights at once with
// all loads of a warp in flight, and the products (mma.sync, 16-row tiles) are an afterthought.  Semantics as in
// ttt_layer.cu (rust/layer/src/ttt.rs:152-299).
//
// Operand order: the contraction index may be permuted at will as long as both operands agree, so a thread takes eight
// consecutive elements of its row (one 16-byte load) and feeds them to two k-steps: elements 0..3 are its share of the
// first, 4..7 of the second.
#include "ttt_kernels.h"
#include "ttt_common.cuh"

namespace ttt {

constexpr int SM_THREADS = 256, SM_WARPS = 8;

// These kernels begin while the kernel before them runs (launch_dependent).  What that one may be writing -- activations,
// for the first of them weights too -- is read by ordinary loads behind pdl_wait: the non-coherent path promises data that
// nobody writes while the kernel runs, and such a load may be moved above the wait.  It is left to the output kernel's
// weights: its predecessor, the inner step, writes none, and everything before that has finished when it starts.
__device__ __forceinline__ uint4 ld4(const void* p) { return *static_cast<const uint4*>(p); }
__device__ __forceinline__ uint4 ldg4(const void* p) { return __ldg(static_cast<const uint4*>(p)); }

// acc[mt][nt] += A . B^T over one 32-wide slice: a[mt][half] rows 16 mt + g + 8 half, b[nt] rows 8 nt + g
template <int MT, int NT>
__device__ __forceinline__ void slice_mma(float (&acc)[MT][NT][4], const uint4 (&a)[MT][2], const uint4 (&b)[NT]) {
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      mma_bf16(acc[mt][nt], a[mt][0].x, a[mt][1].x, a[mt][0].y, a[mt][1].y, b[nt].x, b[nt].y);
      mma_bf16(acc[mt][nt], a[mt][0].z, a[mt][1].z, a[mt][0].w, a[mt][1].w, b[nt].z, b[nt].w);
    }
}
// the warps' partial tiles summed in warp order; thread e of the block gets the pair e of tile mt: row e / (4 NT), columns
// 2 (e % (4 NT)), + 1 (threads beyond 64 NT get nothing)
template <int MT, int NT>
__device__ __forceinline__ float2 tile_sum(float* red, const float (&acc)[MT][NT][4], int mt) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  constexpr int LD = 8 * NT + 2;  // floats per row of a partial tile (even: pairs stay aligned)
  __syncthreads();                // the previous tile has been read
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      *reinterpret_cast<float2*>(&red[(warp * 16 + g + 8 * r) * LD + 8 * nt + 2 * t]) =
          make_float2(acc[mt][nt][2 * r], acc[mt][nt][2 * r + 1]);
  __syncthreads();
  float2 s = make_float2(0.f, 0.f);
  if (tid < 64 * NT) {
    const int row = tid / (4 * NT), c = 2 * (tid % (4 * NT));
#pragma unroll
    for (int w = 0; w < SM_WARPS; ++w) {
      const float2 v = *reinterpret_cast<const float2*>(&red[(w * 16 + row) * LD + c]);
      s.x += v.x;
      s.y += v.y;
    }
  }
  return s;
}

// Projections: x [M, K] . w[N, K]^T with the head split, the rotary rotation and the learning-rate gate on the way out;
// token_eta by the first block.
template <int MT>
__global__ void __launch_bounds__(SM_THREADS) ttt_layer_small_proj_kernel(const SmallProjParams p) {
  constexpr int NT = 2;
  __shared__ float red[SM_WARPS * 16 * (8 * NT + 2)];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16;
  const __nv_bfloat16* const x = static_cast<const __nv_bfloat16*>(p.x);
  const __nv_bfloat16* const w = static_cast<const __nv_bfloat16*>(p.w);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float acc[MT][NT][4] = {};
  pdl_wait();
  pdl_go();
  TokenEtaElement te;
  if (blockIdx.x == 0) te.load(p.te, tid);
#pragma unroll 4
  for (int k = warp * 32 + 8 * t; k < p.K; k += SM_WARPS * 32) {
    uint4 a[MT][2], b[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const int n = n0 + 8 * nt + g;
      b[nt] = n < p.N ? ld4(w + (size_t)n * p.ldw + k) : zero;
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int m = 16 * mt + g + 8 * r;
        a[mt][r] = m < p.M ? ld4(x + (size_t)m * p.ldx + k) : zero;
      }
    slice_mma(acc, a, b);
  }
  if (blockIdx.x == 0) te.store(p.te, tid);
  const int C = p.H * p.F;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    float2 v = tile_sum<MT, NT>(red, acc, mt);
    const int m = 16 * mt + tid / (4 * NT), n = n0 + 2 * (tid % (4 * NT));
    if (tid >= 64 * NT || m >= p.M || n >= p.N) continue;
    if (n >= p.lr_col) {  // learning-rate logits (then padding rows)
      const int h0 = n - p.lr_col, b = m / p.T, tok = m % p.T;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int h = h0 + e;
        if (h >= p.H) continue;
        float z = e ? v.y : v.x;
        if (p.lr_bias != nullptr) z += ld_as_float<__nv_bfloat16>(p.lr_bias, (size_t)h);
        st_from_float<__nv_bfloat16>(p.lr_out, ((size_t)b * p.H + h) * p.lr_ld + tok, p.base_lr / p.F / (1.f + expf(-z)));
      }
      continue;
    }
    const int blk = n / C, c = n - blk * C;  // 0 q, 1 k, 2 v, 3 gate
    if (blk == 3) {
      *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.gate) + (size_t)m * C + c) = pack_bf16(v.x, v.y);
      continue;
    }
    const int h = c / p.F, f = c - h * p.F, b = m / p.T, tok = m % p.T;
    if (blk < 2 && p.rope_mode != 0) {
      const int pos = p.rope_mode == 1 ? (p.start_idx + tok) % p.pos_mod : p.start_idx + tok;
      float sn, cs;
      sincosf(pos * exp2f(-((float)f / p.F) * log2f(p.rope_theta)), &sn, &cs);
      v = make_float2(v.x * cs - v.y * sn, v.y * cs + v.x * sn);
    }
    void* const dst = blk == 0 ? p.xq : blk == 1 ? p.xk : p.xv;
    *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(dst) + (((size_t)b * p.H + h) * p.T + tok) * p.F + f) =
        pack_bf16(v.x, v.y);
  }
}

// Output side: y = (LN(inner_out) [* gelu(gate)]) . w[C, C]^T.  Every CTA normalises the rows for itself (they are few).
template <int MT>
__global__ void __launch_bounds__(SM_THREADS) ttt_layer_small_out_kernel(const SmallOutParams p) {
  constexpr int NT = 1;
  extern __shared__ __align__(16) uint8_t so_smem[];
  __shared__ float red[SM_WARPS * 16 * (8 * NT + 2)];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 8, C = p.H * p.F;
  const int ld = C + 32;  // bf16 elements per row of the operand tile: 64 bytes of padding
  __nv_bfloat16* const rows = reinterpret_cast<__nv_bfloat16*>(so_smem);
  const __nv_bfloat16* const w = static_cast<const __nv_bfloat16*>(p.w);
  // the first weight slices are on their way while the kernel before this one (the inner loop's step, which writes no
  // weights) finishes and the rows are normalised
  constexpr int PRE = 3;
  uint4 pre[PRE];
#pragma unroll
  for (int i = 0; i < PRE; ++i) {
    const int k = (i * SM_WARPS + warp) * 32 + 8 * t;
    pre[i] = k < C ? ldg4(w + (size_t)(n0 + g) * p.ldw + k) : make_uint4(0u, 0u, 0u, 0u);
  }
  pdl_wait();
  pdl_go();
  for (int m = warp; m < 16 * MT; m += SM_WARPS) {
    if (m >= p.M) {  // padding rows of the last tile
      for (int c = 8 * lane; c < C; c += 256) *reinterpret_cast<uint4*>(rows + m * ld + c) = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const int b = m / p.T, tok = m % p.T;
    float v[8][8];  // up to 2048 features
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = 8 * lane + 256 * i;
      if (c < C) {
        const int h = c / p.F, f = c - h * p.F;
        const uint4 q = ld4(static_cast<const __nv_bfloat16*>(p.inner_out) + (((size_t)b * p.H + h) * p.T + tok) * p.F + f);
        const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[i][2 * j] = bf16_lo(u[j]);
          v[i][2 * j + 1] = bf16_hi(u[j]);
          s += v[i][2 * j] + v[i][2 * j + 1];
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = s / C;
    float q2 = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (8 * lane + 256 * i < C)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[i][j] -= mean;
          q2 = fmaf(v[i][j], v[i][j], q2);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    const float rstd = 1.f / sqrtf(q2 / C + p.eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = 8 * lane + 256 * i;
      if (c < C) {
        const uint4 gq = ldg4(static_cast<const __nv_bfloat16*>(p.ln_w) + c), bq = ldg4(static_cast<const __nv_bfloat16*>(p.ln_b) + c);
        const uint32_t gu[4] = {gq.x, gq.y, gq.z, gq.w}, bu[4] = {bq.x, bq.y, bq.z, bq.w};
        float y[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          y[2 * j] = fmaf(v[i][2 * j] * rstd, bf16_lo(gu[j]), bf16_lo(bu[j]));
          y[2 * j + 1] = fmaf(v[i][2 * j + 1] * rstd, bf16_hi(gu[j]), bf16_hi(bu[j]));
        }
        if (p.gate != nullptr) {
          const uint4 tq = ld4(static_cast<const __nv_bfloat16*>(p.gate) + (size_t)m * p.ld_gate + c);
          const uint32_t tu[4] = {tq.x, tq.y, tq.z, tq.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float a = (j & 1) ? bf16_hi(tu[j >> 1]) : bf16_lo(tu[j >> 1]);
            y[j] *= 0.5f * a * (1.f + tanhf(0.7978845608028654f * (a + 0.044715f * a * a * a)));
          }
        }
        *reinterpret_cast<uint4*>(rows + m * ld + c) =
            make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
      }
    }
  }
  __syncthreads();
  float acc[MT][NT][4] = {};
  int i = 0;
#pragma unroll 4
  for (int k = warp * 32 + 8 * t; k < C; k += SM_WARPS * 32, ++i) {
    uint4 a[MT][2], b[NT];
    b[0] = i == 0 ? pre[0] : i == 1 ? pre[1] : i == 2 ? pre[2] : ldg4(w + (size_t)(n0 + g) * p.ldw + k);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int r = 0; r < 2; ++r) a[mt][r] = *reinterpret_cast<const uint4*>(rows + (16 * mt + g + 8 * r) * ld + k);
    slice_mma(acc, a, b);
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    const float2 v = tile_sum<MT, NT>(red, acc, mt);
    const int m = 16 * mt + tid / (4 * NT), n = n0 + 2 * (tid % (4 * NT));
    if (tid < 64 * NT && m < p.M)
      *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(p.y) + (size_t)m * C + n) = pack_bf16(v.x, v.y);
  }
}

cudaError_t launch_layer_small_proj(const SmallProjParams& p, cudaStream_t st) {
  const int grid = (p.N + 15) / 16;
  return launch_dependent(p.M <= 16 ? ttt_layer_small_proj_kernel<1> : ttt_layer_small_proj_kernel<2>, grid, SM_THREADS, 0, st, p);
}

template <int MT>
static cudaError_t launch_out_t(const SmallOutParams& p, cudaStream_t st) {
  const int C = p.H * p.F, smem = 16 * MT * (C + 32) * 2;
  static DeviceValue ready;
  int most = 0;
  const cudaError_t e = ready.get(0, &most, [](int* n) {
    *n = 16 * MT * (2048 + 32) * 2;
    return cudaFuncSetAttribute(ttt_layer_small_out_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, *n);
  });
  if (e != cudaSuccess) return e;
  return launch_dependent(ttt_layer_small_out_kernel<MT>, C / 8, SM_THREADS, smem, st, p);
}
cudaError_t launch_layer_small_out(const SmallOutParams& p, cudaStream_t st) {
  return p.M <= 16 ? launch_out_t<1>(p, st) : launch_out_t<2>(p, st);
}

}  // namespace ttt
