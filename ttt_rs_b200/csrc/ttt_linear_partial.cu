// One mini-batch of fewer than (or exactly) 16 tokens of the TTT-Linear inner model: the decode step (1 token) and
// the tail of a sequence whose length is not a multiple of the mini-batch.
//
// Reference semantics: `TTTInnerModel::forward` runs whole mini-batches and then calls `forward_mini_batch` once on
// the remainder, i.e. the remainder is ONE mini-batch of its own length r with eta[i][j] = token_eta[i] * lr[j]
// (rust/core/src/inner.rs:25-50, rust/core/src/linear.rs:91-149); token by token generation therefore runs with
// r = 1 (rust/layer/src/ttt.rs:253-256).  The reference's fused kernels refuse these shapes
// (rust/fused/src/linear_fused_tile/wrapper.rs:152-172); only its unfused tensor-op path covers them.
//
// Work per stream is tiny (r <= 16 rows against an F x F state, F = 64 or 32): CUDA cores, and the time is the chain of
// dependent steps -- load the state, z = x W + b, LayerNorm statistics, gradient, second LayerNorm, update.  So:
//   * one 4-warp CTA per stream; warp w holds rows [w F/4, (w + 1) F/4) of W (lane: F/32 adjacent columns, coalesced 64- or
//     128-byte rows), so z is a partial sum per warp, met in shared memory: one barrier;
//   * from there on a row belongs to one warp (row i to warp i % 4): every row sum is a warp shuffle, no barrier; the
//     gradients of all rows meet in shared memory once more for the output and the update.
// The state is read and written exactly once, three barriers in all.  (One thread per column with the row sums crossing
// warps ten times: 22 us for 9 rows of 12 streams, 4.1 us for one row of 96.)
#include "ttt_kernels.h"
#include "ttt_common.cuh"

namespace ttt {

constexpr int PT_WARPS = 4;

// N adjacent columns; VEC: as one access (the pointers are aligned to it), else element by element
template <typename T, bool VEC, int N>
__device__ __forceinline__ void ld_cols(const void* base, size_t idx, float (&v)[N]) {
  if constexpr (N == 1 || !VEC) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = ld_as_float<T>(base, idx + i);
  } else if constexpr (sizeof(T) == 2) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(static_cast<const T*>(base) + idx);
    v[0] = bf16_lo(u);
    v[1] = bf16_hi(u);
  } else {
    const float2 u = *reinterpret_cast<const float2*>(static_cast<const T*>(base) + idx);
    v[0] = u.x;
    v[1] = u.y;
  }
}
template <typename T, bool VEC, int N>
__device__ __forceinline__ void st_cols(void* base, size_t idx, const float (&v)[N]) {
  if constexpr (N == 1 || !VEC) {
#pragma unroll
    for (int i = 0; i < N; ++i) st_from_float<T>(base, idx + i, v[i]);
  } else if constexpr (sizeof(T) == 2) *reinterpret_cast<uint32_t*>(static_cast<T*>(base) + idx) = pack_bf16(v[0], v[1]);
  else *reinterpret_cast<float2*>(static_cast<T*>(base) + idx) = make_float2(v[0], v[1]);
}
// sums of N values over the warp, all of them in every lane
template <int N>
__device__ __forceinline__ void warp_sums(float (&v)[N]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
}

template <int RM, int FD>
struct PartialSmem {
  float q[RM][FD], k[RM][FD], g[RM][FD];  // g: the rows' gradients
  float z[PT_WARPS][2][RM][FD];           // the warps' partial K W and Q W
  float attn[RM][RM];
  float lr[RM], te[RM];
};

// RM: compile-time bound on the number of rows (1 for the decode step, 4, or 16).
template <typename T, int RM, int FD, bool VEC>
__global__ void __launch_bounds__(32 * PT_WARPS) ttt_linear_partial_kernel(const LinPartialParams p) {
  constexpr int NC = FD / 32, KR = FD / PT_WARPS;            // columns per lane, rows of W per warp
  constexpr int RW = (RM + PT_WARPS - 1) / PT_WARPS;         // rows of the mini-batch per warp
  constexpr int NT = 32 * PT_WARPS;
  constexpr float INV_F = 1.f / FD;
  __shared__ __align__(16) PartialSmem<RM, FD> sm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int stream = blockIdx.x, head = stream % p.H, r = p.R;
  const size_t row0 = (size_t)stream * p.row_ld + p.row_off;
  const int c0 = NC * lane, k0 = KR * warp;

  float w[KR][NC];
  if (!p.state_settled) pdl_wait();
#pragma unroll
  for (int k = 0; k < KR; ++k) ld_cols<T, VEC>(p.w0, (size_t)stream * FD * FD + (size_t)(k0 + k) * FD + c0, w[k]);
  if (p.state_settled) pdl_wait();
  pdl_go();
  for (int e = tid; e < r * FD; e += NT) {
    sm.q[0][e] = ld_as_float<T>(p.xq, row0 * FD + e);
    sm.k[0][e] = ld_as_float<T>(p.xk, row0 * FD + e);
  }
  if (tid < r) {
    sm.lr[tid] = ld_as_float<T>(p.lr, (size_t)stream * p.lr_ld + p.row_off + tid);
    sm.te[tid] = ld_as_float<T>(p.token_eta, (size_t)tid);
  }
  float bias[NC], gam[NC], bet[NC], v[RW][NC];
  ld_cols<T, VEC>(p.b0, (size_t)stream * FD + c0, bias);
  ld_cols<T, VEC>(p.ln_g, (size_t)head * FD + c0, gam);
  ld_cols<T, VEC>(p.ln_b, (size_t)head * FD + c0, bet);
#pragma unroll
  for (int j = 0; j < RW; ++j)
    if (warp + PT_WARPS * j < r) ld_cols<T, VEC>(p.xv, (row0 + warp + PT_WARPS * j) * FD + c0, v[j]);
  __syncthreads();

  // ---- this warp's share of Z1 = K W and Zq = Q W; Attn[i][j] = Q[i] . K[j] for j <= i
#pragma unroll
  for (int i = 0; i < RM; ++i)
    if (i < r) {
      float a[NC] = {}, b[NC] = {};
#pragma unroll
      for (int k = 0; k < KR; k += 4) {
        const float4 kk = *reinterpret_cast<const float4*>(&sm.k[i][k0 + k]), qq = *reinterpret_cast<const float4*>(&sm.q[i][k0 + k]);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          a[c] = fmaf(kk.w, w[k + 3][c], fmaf(kk.z, w[k + 2][c], fmaf(kk.y, w[k + 1][c], fmaf(kk.x, w[k][c], a[c]))));
          b[c] = fmaf(qq.w, w[k + 3][c], fmaf(qq.z, w[k + 2][c], fmaf(qq.y, w[k + 1][c], fmaf(qq.x, w[k][c], b[c]))));
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        sm.z[warp][0][i][c0 + c] = a[c];
        sm.z[warp][1][i][c0 + c] = b[c];
      }
    }
  for (int e = tid; e < r * r; e += NT) {
    const int i = e / r, j = e - i * r;
    if (j > i) continue;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int k = 0; k < FD; k += 8) {
      const float4 qa = *reinterpret_cast<const float4*>(&sm.q[i][k]), ka = *reinterpret_cast<const float4*>(&sm.k[j][k]);
      const float4 qb = *reinterpret_cast<const float4*>(&sm.q[i][k + 4]), kb = *reinterpret_cast<const float4*>(&sm.k[j][k + 4]);
      s0 = fmaf(qa.w, ka.w, fmaf(qa.z, ka.z, fmaf(qa.y, ka.y, fmaf(qa.x, ka.x, s0))));
      s1 = fmaf(qb.w, kb.w, fmaf(qb.z, kb.z, fmaf(qb.y, kb.y, fmaf(qb.x, kb.x, s1))));
    }
    sm.attn[i][j] = s0 + s1;
  }
  __syncthreads();

  // ---- per row (i = warp + 4 j): LayerNorm statistics of Z1 (two-pass variance), G = dL/dZ1
  float z[RW][NC], st[RW], mean[RW];
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    const int i = min(warp + PT_WARPS * j, r - 1);  // (rows beyond the last: computed on the last one's values, not kept)
    st[j] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      z[j][c] = bias[c] + ((sm.z[0][0][i][c0 + c] + sm.z[1][0][i][c0 + c]) + (sm.z[2][0][i][c0 + c] + sm.z[3][0][i][c0 + c]));
      st[j] += z[j][c];
    }
  }
  warp_sums(st);
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    mean[j] = st[j] * INV_F;
    st[j] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      z[j][c] -= mean[j];
      st[j] = fmaf(z[j][c], z[j][c], st[j]);
    }
  }
  warp_sums(st);
  float gx[RW][NC], sums[2 * RW], rstd[RW];
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    rstd[j] = 1.f / sqrtf(st[j] * INV_F + p.eps);
    sums[2 * j] = sums[2 * j + 1] = 0.f;
    const int i = min(warp + PT_WARPS * j, r - 1);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      z[j][c] *= rstd[j];  // x_hat
      const float tgt = (warp + PT_WARPS * j < r) ? v[j][c] - sm.k[i][c0 + c] : 0.f;
      gx[j][c] = (gam[c] * z[j][c] + bet[c] - tgt) * gam[c];
      sums[2 * j] += gx[j][c];
      sums[2 * j + 1] = fmaf(gx[j][c], z[j][c], sums[2 * j + 1]);
    }
  }
  warp_sums(sums);
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    const int i = warp + PT_WARPS * j;
    if (i < r) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        sm.g[i][c0 + c] = (gx[j][c] - sums[2 * j] * INV_F - z[j][c] * sums[2 * j + 1] * INV_F) * rstd[j];
    }
  }
  __syncthreads();

  // ---- state update with the last row of eta: W -= (te[r-1] lr o K)^T G, b -= sum_j te[r-1] lr[j] G[j]
  const float te_last = sm.te[r - 1];
  float b_in[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) b_in[c] = bias[c];
  for (int j = 0; j < r; ++j) {
    const float e = te_last * sm.lr[j];
    float gl[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      gl[c] = e * sm.g[j][c0 + c];
      bias[c] -= gl[c];
    }
#pragma unroll
    for (int k = 0; k < KR; k += 4) {
      const float4 kk = *reinterpret_cast<const float4*>(&sm.k[j][k0 + k]);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        w[k][c] = fmaf(-kk.x, gl[c], w[k][c]);
        w[k + 1][c] = fmaf(-kk.y, gl[c], w[k + 1][c]);
        w[k + 2][c] = fmaf(-kk.z, gl[c], w[k + 2][c]);
        w[k + 3][c] = fmaf(-kk.w, gl[c], w[k + 3][c]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < KR; ++k) st_cols<T, VEC>(p.w_out, (size_t)stream * FD * FD + (size_t)(k0 + k) * FD + c0, w[k]);

  // ---- Zbar = Zq - sum_{j<=i} te[i] lr[j] (1 + Attn[i][j]) G[j];  out = Q + LN(Zbar)
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    const int i = min(warp + PT_WARPS * j, r - 1);
    float s[NC] = {};
    for (int l = 0; l <= i; ++l) {
      const float m = sm.lr[l] * (1.f + sm.attn[i][l]);
#pragma unroll
      for (int c = 0; c < NC; ++c) s[c] = fmaf(m, sm.g[l][c0 + c], s[c]);
    }
    st[j] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float zq = b_in[c] + ((sm.z[0][1][i][c0 + c] + sm.z[1][1][i][c0 + c]) + (sm.z[2][1][i][c0 + c] + sm.z[3][1][i][c0 + c]));
      z[j][c] = zq - sm.te[i] * s[c];
      st[j] += z[j][c];
    }
  }
  warp_sums(st);
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    mean[j] = st[j] * INV_F;
    st[j] = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      z[j][c] -= mean[j];
      st[j] = fmaf(z[j][c], z[j][c], st[j]);
    }
  }
  warp_sums(st);
#pragma unroll
  for (int j = 0; j < RW; ++j) {
    const int i = warp + PT_WARPS * j;
    if (i < r) {
      const float rs = 1.f / sqrtf(st[j] * INV_F + p.eps);
      float o[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) o[c] = sm.q[i][c0 + c] + gam[c] * z[j][c] * rs + bet[c];
      st_cols<T, VEC>(p.out, (row0 + i) * FD + c0, o);
    }
  }
  // (in place or not: every warp read the old state before the first barrier)
  if (warp == 0) st_cols<T, VEC>(p.b_out, (size_t)stream * FD + c0, bias);
}

template <typename T, int FD, bool VEC>
static cudaError_t launch_partial_t(const LinPartialParams& p, int nstreams, cudaStream_t st) {
  auto kfn = p.R == 1   ? ttt_linear_partial_kernel<T, 1, FD, VEC>
             : p.R <= 4 ? ttt_linear_partial_kernel<T, 4, FD, VEC>
                        : ttt_linear_partial_kernel<T, 16, FD, VEC>;
  return launch_dependent(kfn, nstreams, 32 * PT_WARPS, 0, st, p);
}
template <typename T>
static cudaError_t launch_partial_d(int head_dim, const LinPartialParams& p, int nstreams, cudaStream_t st) {
  if (head_dim == 32) return launch_partial_t<T, 32, false>(p, nstreams, st);
  // column pairs as one access where every tensor starts on one (any tensor of its own does; a view may not)
  uintptr_t all = 0;
  for (const void* q : {p.w0, p.b0, p.ln_g, p.ln_b, p.xv, (const void*)p.out, (const void*)p.w_out, (const void*)p.b_out})
    all |= reinterpret_cast<uintptr_t>(q);
  return all % (2 * sizeof(T)) == 0 ? launch_partial_t<T, 64, true>(p, nstreams, st)
                                    : launch_partial_t<T, 64, false>(p, nstreams, st);
}

cudaError_t launch_linear_partial(int dtype, int head_dim, const LinPartialParams& p, int nstreams, cudaStream_t st) {
  return dtype == 1 ? launch_partial_d<__nv_bfloat16>(head_dim, p, nstreams, st)
                    : launch_partial_d<float>(head_dim, p, nstreams, st);
}

}  // namespace ttt
