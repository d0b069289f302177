// The steps of the outer TTT layer on either side of the inner loop, as two bandwidth-bound kernels (sm_100a).
//
// Reference semantics: rust/layer/src/ttt.rs:152-299 (`get_qkv`, `get_lr`, `conv_qk`, `forward`), rotary embedding
// rust/core/src/util.rs:284-392 (PyTorch twin reference/ttt.py:215-270,701-915).  There the projections' outputs
// are reshaped and permuted to [B,H,T,F] (one materialised copy per tensor), rotated by separate element-wise
// kernels, the learning-rate gate is a chain of small tensor ops, and after the inner loop the result is permuted
// back and normalised by further kernels.  Here:
//   * ttt_layer_prologue_kernel reads the projection output once in its native [B*T, columns] layout and writes
//     XQ, XK, XV in the inner loop's [B,H,T,F] layout with the shared-QK causal convolutions and the rotary
//     rotation applied on the way, plus ttt_lr_eta = base_lr * sigmoid(logit + bias) / F in [B,H,T];
//   * ttt_layer_epilogue_kernel reads the inner loop's [B,H,T,F] output once and writes [B,T,H*F] with the post
//     LayerNorm and the optional gelu(tanh) gate applied.
// Every global access is a full 128-byte (bf16) or 256-byte (f32) row segment per 8 / 32 lanes; no shared-memory
// staging is needed because a (token, head) row of F = 64 or 32 features is contiguous in both layouts.
#include "ttt_kernels.h"
#include "ttt_common.cuh"

namespace ttt {

template <typename T>
struct Vec8;  // eight consecutive elements
template <>
struct Vec8<__nv_bfloat16> {
  uint4 raw;
  __device__ __forceinline__ void load(const void* p) { raw = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void store(void* p) const { *reinterpret_cast<uint4*>(p) = raw; }
  __device__ __forceinline__ void load_once(const void* p) { raw = __ldcs(reinterpret_cast<const uint4*>(p)); }
  __device__ __forceinline__ void store_once(void* p) const { __stcs(reinterpret_cast<uint4*>(p), raw); }
  __device__ __forceinline__ void unpack(float (&f)[8]) const {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = bf16_lo(w[i]);
      f[2 * i + 1] = bf16_hi(w[i]);
    }
  }
  __device__ __forceinline__ void pack(const float (&f)[8]) {
    raw.x = pack_bf16(f[0], f[1]);
    raw.y = pack_bf16(f[2], f[3]);
    raw.z = pack_bf16(f[4], f[5]);
    raw.w = pack_bf16(f[6], f[7]);
  }
};
template <>
struct Vec8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const void* p) {
    a = reinterpret_cast<const float4*>(p)[0];
    b = reinterpret_cast<const float4*>(p)[1];
  }
  __device__ __forceinline__ void store(void* p) const {
    reinterpret_cast<float4*>(p)[0] = a;
    reinterpret_cast<float4*>(p)[1] = b;
  }
  __device__ __forceinline__ void load_once(const void* p) {
    a = __ldcs(reinterpret_cast<const float4*>(p));
    b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
  }
  __device__ __forceinline__ void store_once(void* p) const {
    __stcs(reinterpret_cast<float4*>(p), a);
    __stcs(reinterpret_cast<float4*>(p) + 1, b);
  }
  __device__ __forceinline__ void unpack(float (&f)[8]) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  __device__ __forceinline__ void pack(const float (&f)[8]) {
    a = make_float4(f[0], f[1], f[2], f[3]);
    b = make_float4(f[4], f[5], f[6], f[7]);
  }
};

constexpr int PRO_THREADS = 256;
constexpr int PRO_TCHUNK = 32;   // tokens per warp task, at most
constexpr int PRO_MAXK = 4;      // causal convolution taps supported
constexpr int PRO_MAXPOS = 64;   // rotary table rows (positions modulo the mini-batch length)

// One warp task = (batch b, group of HPW heads, chunk of PRO_TCHUNK tokens), HPW = 4 heads of 64 features or 8 heads of
// 32.  Lane = SUBS*hq + sub (SUBS = F/8) handles head HPW*hgroup + hq, features [8*sub, 8*sub+8) = rotary pairs
// 4*sub .. 4*sub+3, and walks the chunk's tokens in groups of PRO_TG whose loads are all issued before any of them is
// used (memory-level parallelism).
constexpr int PRO_TG = 4;

template <typename T, bool CONV, int FD>
__global__ void __launch_bounds__(PRO_THREADS, (CONV || sizeof(T) == 4) ? 1 : 3) ttt_layer_prologue_kernel(const LayerProParams p) {
  __shared__ float2 rope_tab[PRO_MAXPOS][32];  // (cos, sin) per position and pair (the first FD/2 pairs are used)
  constexpr int F = FD, SUBS = FD / 8, HPW = 32 / SUBS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int H = p.H, NT = p.T;
  const bool rope = p.rope_mode != 0;
  const bool rope_wrap = p.rope_mode == 1;
  const float log2_theta = log2f(p.rope_theta);
  if (rope && rope_wrap) {
    for (int e = tid; e < p.pos_mod * 32; e += PRO_THREADS) {
      const int pos = e >> 5, i = e & 31;
      const float inv_freq = exp2f(-(2.f * i / F) * log2_theta);
      float s, c;
      sincosf(pos * inv_freq, &s, &c);
      rope_tab[pos][i] = make_float2(c, s);
    }
  }
  pdl_join();
  if (sizeof(T) == 2 && blockIdx.x == 0) {
    TokenEtaElement te;
    te.load(p.te, tid);
    te.store(p.te, tid);
  }
  __syncthreads();

  const int hq = lane / SUBS, sub = lane % SUBS;
  const int hgroups = (H + HPW - 1) / HPW, tchunks = (NT + p.tchunk - 1) / p.tchunk;
  const long ntasks = (long)p.B * hgroups * tchunks;
  const int KC = p.conv_k;

  for (long task = (long)blockIdx.x * (PRO_THREADS / 32) + warp; task < ntasks; task += (long)gridDim.x * (PRO_THREADS / 32)) {
    const int tc = (int)(task % tchunks);
    const int hg = (int)((task / tchunks) % hgroups);
    const int b = (int)(task / ((long)tchunks * hgroups));
    const int h = HPW * hg + hq;
    if (h >= H) continue;
    const int col = h * F + 8 * sub;  // first of this lane's 8 columns inside a projection block
    const int t0 = tc * p.tchunk, t1 = min(NT, t0 + p.tchunk);

    // convolution taps and biases of this lane's 8 channels (loop-invariant); window slot j holds token
    // t-(PRO_MAXK-1)+j and taps are right-aligned (the last tap multiplies token t), so slots older than the kernel
    // length get zero weights
    float wq[CONV ? PRO_MAXK : 1][8], wk[CONV ? PRO_MAXK : 1][8], bq[8], bk[8];
    float hist[CONV ? PRO_MAXK - 1 : 1][8];  // the previous PRO_MAXK-1 rows of the shared projection (oldest first)
    if constexpr (CONV) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        bq[c] = ld_as_float<T>(p.conv_q_b, (size_t)(col + c));
        bk[c] = ld_as_float<T>(p.conv_k_b, (size_t)(col + c));
#pragma unroll
        for (int j = 0; j < PRO_MAXK; ++j) {
          const int wj = j - (PRO_MAXK - KC);
          wq[j][c] = (wj >= 0) ? ld_as_float<T>(p.conv_q_w, (size_t)(col + c) * KC + wj) : 0.f;
          wk[j][c] = (wj >= 0) ? ld_as_float<T>(p.conv_k_w, (size_t)(col + c) * KC + wj) : 0.f;
        }
      }
#pragma unroll
      for (int j = 0; j < PRO_MAXK - 1; ++j) {
        const int tt = t0 - (PRO_MAXK - 1) + j;
        if (tt >= 0) {
          Vec8<T> v;
          v.load(static_cast<const T*>(p.q_src) + ((size_t)b * NT + tt) * p.ld_src + col);
          v.unpack(hist[j]);
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) hist[j][c] = 0.f;
        }
      }
    }

    for (int tb = t0; tb < t1; tb += PRO_TG) {
      Vec8<T> vq[PRO_TG], vk[PRO_TG], vv[PRO_TG];
#pragma unroll
      for (int u = 0; u < PRO_TG; ++u) {
        if (tb + u < t1) {
          const size_t srow = ((size_t)b * NT + tb + u) * p.ld_src + col;
          vq[u].load(static_cast<const T*>(p.q_src) + srow);
          if constexpr (!CONV) vk[u].load(static_cast<const T*>(p.k_src) + srow);
          vv[u].load(static_cast<const T*>(p.v_src) + srow);
        }
      }
#pragma unroll
      for (int u = 0; u < PRO_TG; ++u) {
        const int t = tb + u;
        if (t < t1) {
          float fq[8], fk[8];
          if constexpr (CONV) {
            float cur[8];
            vq[u].unpack(cur);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              float aq = bq[c], ak = bk[c];
#pragma unroll
              for (int j = 0; j < PRO_MAXK - 1; ++j) {
                aq = fmaf(wq[j][c], hist[j][c], aq);
                ak = fmaf(wk[j][c], hist[j][c], ak);
              }
              fq[c] = fmaf(wq[PRO_MAXK - 1][c], cur[c], aq);
              fk[c] = fmaf(wk[PRO_MAXK - 1][c], cur[c], ak);
            }
#pragma unroll
            for (int j = 0; j < PRO_MAXK - 2; ++j)
#pragma unroll
              for (int c = 0; c < 8; ++c) hist[j][c] = hist[j + 1][c];
#pragma unroll
            for (int c = 0; c < 8; ++c) hist[PRO_MAXK - 2][c] = cur[c];
          } else {
            vq[u].unpack(fq);
            vk[u].unpack(fk);
          }
          if (rope) {
            const int pos = p.start_idx + t;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float2 cs;
              if (rope_wrap) {
                cs = rope_tab[pos % p.pos_mod][4 * sub + j];
              } else {
                const float inv_freq = exp2f(-(2.f * (4 * sub + j) / F) * log2_theta);
                sincosf(pos * inv_freq, &cs.y, &cs.x);
              }
              const float q0 = fq[2 * j], q1 = fq[2 * j + 1], k0 = fk[2 * j], k1 = fk[2 * j + 1];
              fq[2 * j] = q0 * cs.x - q1 * cs.y;
              fq[2 * j + 1] = q1 * cs.x + q0 * cs.y;
              fk[2 * j] = k0 * cs.x - k1 * cs.y;
              fk[2 * j + 1] = k1 * cs.x + k0 * cs.y;
            }
          }
          if (CONV || rope) {
            vq[u].pack(fq);
            vk[u].pack(fk);
          }
          const size_t drow = (((size_t)b * H + h) * NT + t) * F + 8 * sub;
          vq[u].store(static_cast<T*>(p.xq) + drow);
          vk[u].store(static_cast<T*>(p.xk) + drow);
          vv[u].store(static_cast<T*>(p.xv) + drow);
        }
      }
    }
  }

  // ttt_lr_eta[b,h,t] = base_lr / F * sigmoid(logit[b*T+t][h] + bias[h])
  const long nlr = (long)p.B * H * NT;
  for (long e = (long)blockIdx.x * PRO_THREADS + tid; e < nlr; e += (long)gridDim.x * PRO_THREADS) {
    const int t = (int)(e % NT);
    const int h = (int)((e / NT) % H);
    const int b = (int)(e / ((long)NT * H));
    float z = ld_as_float<T>(p.lr_logits, ((size_t)b * NT + t) * p.ld_lr + h);
    if (p.lr_bias != nullptr) z += ld_as_float<T>(p.lr_bias, (size_t)h);
    st_from_float<T>(p.lr_out, ((size_t)b * H + h) * p.lr_ld_out + t, p.base_lr / F / (1.f + expf(-z)));
  }
}

// One CTA per tile of TT consecutive tokens of one batch element, persistent, tiles double-buffered.  Load: for every head the
// tile's TT rows of F features are one contiguous segment of the [B,H,T,F] tensor; a thread copies its 16-byte column chunk of
// its rows asynchronously to a [TT][H*F] tile in shared memory.  Row phase: a warp per row takes mean and variance (two
// sweeps over registers).  Column phase: a thread per 16-byte chunk of columns and row group, its weights and biases in
// registers, applies the norm and the optional gate and stores to [B,T,H*F].  Bound by shared-memory and issue slots before
// memory: 65536 tokens, bf16: 55.6 -> 49.3 -> 45 us at 768 features (the last with tiles of a row per warp), 118 -> 93 us at
// 2048; gated 289 -> 233 us, float32 gated 678 -> 327 us at 2048 (a warp that also wrote its row read 4 to 16 KB of weights and
// biases for it from shared memory).
// CTAs per SM: one fewer for float32 without a gate, which is at 0.9 of the memory rate with two (67 against 76 us at 768).
// MAXCH: 16-byte chunks of one row per lane (rows of up to 32 * MAXCH chunks = 512 * MAXCH bytes).
constexpr int EPI_THREADS = 384;
// A CTA's tiles: tile `first + i * stride` of a batch of sequences cut into `per_b` tiles each, as (sequence, tile in it); stepped
// without dividing (two 64-bit divisions per tile were a third of the instructions)
struct TileWalk {
  int b, t, per_b, step_b, step_t;
  long left;  // tiles from this one to the last
  __device__ __forceinline__ TileWalk(long first, long stride, long ntiles, int per_b_) : per_b(per_b_) {
    b = (int)(first / per_b);
    t = (int)(first - (long)b * per_b);
    step_b = (int)(stride / per_b);
    step_t = (int)(stride - (long)step_b * per_b);
    left = ntiles - first;
  }
  __device__ __forceinline__ bool valid() const { return left > 0; }
  __device__ __forceinline__ void step(long stride) {
    left -= stride;
    b += step_b;
    t += step_t;
    if (t >= per_b) {
      t -= per_b;
      ++b;
    }
  }
};
template <typename T, int MAXCH, int FD, bool GATE>
__global__ void __launch_bounds__(MAXCH == 16 ? 512 : EPI_THREADS, (MAXCH == 16 ? 2 : 3) - (sizeof(T) == 4 && !GATE ? 1 : 0))
    ttt_layer_epilogue_kernel(const LayerEpiParams p) {
  constexpr int HD = FD;  // features per head in this instantiation
  const int TT = p.tile_rows;
  constexpr int EPC = 16 / sizeof(T);  // elements per 16-byte chunk
  constexpr int NPAIR = EPC / 2;
  extern __shared__ __align__(16) uint8_t epi_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int H = p.H, NT = p.T, C = H * HD;
  const int nch = C / EPC, ngroups = p.row_groups;
  const size_t tile_bytes = (size_t)TT * C * sizeof(T);
  float2* stat = reinterpret_cast<float2*>(epi_smem + 2 * tile_bytes);  // per row: mean, rstd
  const int tiles_per_b = (NT + TT - 1) / TT;
  const long ntiles = (long)p.B * tiles_per_b;
  const int my_ch = tid % nch, my_grp = tid / nch, c_own = my_ch * EPC;
  const int h_own = c_own / HD, f_own = c_own - h_own * HD;
  auto unpack = [](const uint4 raw, F2 (&v)[NPAIR]) {
    if constexpr (sizeof(T) == 2) {
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = f2(bf16_lo(w[k]), bf16_hi(w[k]));
    } else {
      v[0] = f2(__uint_as_float(raw.x), __uint_as_float(raw.y));
      v[1] = f2(__uint_as_float(raw.z), __uint_as_float(raw.w));
    }
  };
  pdl_join();
  TileWalk ahead(blockIdx.x, gridDim.x, ntiles, tiles_per_b), cur = ahead;
  auto fetch = [&](int buf) {  // the next tile that is not on its way yet
    if (ahead.valid() && my_grp < ngroups) {
      const int b = ahead.b, t0 = ahead.t * TT;
      const int rows = min(TT, NT - t0);
      const uint32_t dst = smem_u32(epi_smem + buf * tile_bytes) + (uint32_t)(c_own * sizeof(T));
      const T* z = static_cast<const T*>(p.inner_out) + (((size_t)b * H + h_own) * NT + t0) * HD + f_own;
      for (int r = my_grp; r < rows; r += ngroups)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(r * C * sizeof(T))),
                     "l"(z + (size_t)r * HD)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ahead.step(gridDim.x);
  };
  F2 gam[NPAIR], bet[NPAIR];
#pragma unroll
  for (int k = 0; k < NPAIR; ++k) {
    gam[k] = f2(ld_as_float<T>(p.ln_w, (size_t)c_own + 2 * k), ld_as_float<T>(p.ln_w, (size_t)c_own + 2 * k + 1));
    bet[k] = f2(ld_as_float<T>(p.ln_b, (size_t)c_own + 2 * k), ld_as_float<T>(p.ln_b, (size_t)c_own + 2 * k + 1));
  }
  int buf = 0;
  fetch(0);
  for (; cur.valid(); cur.step(gridDim.x), buf ^= 1) {
    const int b = cur.b, t0 = cur.t * TT;
    const int rows = min(TT, NT - t0);
    fetch(buf ^ 1);  // that buffer was released by the barrier that ended the last tile
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // this tile has landed for every thread
    const uint8_t* tile = epi_smem + buf * tile_bytes;
    for (int r = warp; r < rows; r += nwarps) {
      const uint4* row = reinterpret_cast<const uint4*>(tile + (size_t)r * C * sizeof(T));
      F2 acc = f2(0.f);
#pragma unroll
      for (int j = 0; j < MAXCH; ++j)
        if (j * 32 + lane < nch) {
          F2 v[NPAIR];
          unpack(row[j * 32 + lane], v);
#pragma unroll
          for (int k = 0; k < NPAIR; ++k) acc = f2add(acc, v[k]);
        }
      float s = f2hsum(acc);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const float mean = s / C;
      acc = f2(0.f);
      asm volatile("" ::: "memory");  // (read again rather than kept: the registers are better spent on warps)
#pragma unroll
      for (int j = 0; j < MAXCH; ++j)
        if (j * 32 + lane < nch) {
          F2 v[NPAIR];
          unpack(row[j * 32 + lane], v);
#pragma unroll
          for (int k = 0; k < NPAIR; ++k) {
            const F2 d = f2sub(v[k], f2(mean));
            acc = f2fma(d, d, acc);
          }
        }
      float q = f2hsum(acc);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (lane == 0) stat[r] = make_float2(mean, 1.f / sqrtf(q / C + p.eps));
    }
    __syncthreads();
    if (my_grp < ngroups) {
      for (int r = my_grp; r < rows; r += ngroups) {
        const size_t tok = (size_t)b * NT + t0 + r;
        const float2 st = stat[r];
        F2 y[NPAIR];
        unpack(*reinterpret_cast<const uint4*>(tile + ((size_t)r * C + c_own) * sizeof(T)), y);
#pragma unroll
        for (int k = 0; k < NPAIR; ++k) y[k] = f2fma(f2sub(y[k], f2(st.x)), f2mul(gam[k], f2(st.y)), bet[k]);
        if constexpr (GATE) {
          // (gate rows are only 8-byte aligned: two 8-byte loads)
          const uint2* gp = reinterpret_cast<const uint2*>(static_cast<const T*>(p.gate) + tok * p.ld_gate + c_own);
          const uint2 g0 = gp[0], g1 = gp[1];
          F2 g[NPAIR];
          unpack(make_uint4(g0.x, g0.y, g1.x, g1.y), g);
          // gelu, tanh form (rust/layer/src/ttt.rs:290-293; constants thundercube/src/unary_ops.rs:136-137)
          auto gelu = [](float x) { return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x))); };
#pragma unroll
          for (int k = 0; k < NPAIR; ++k) y[k] = f2mul(y[k], f2(gelu(g[k].x), gelu(g[k].y)));
        }
        T* dst = static_cast<T*>(p.y) + tok * C + c_own;
        if constexpr (sizeof(T) == 2)
          *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(y[0].x, y[0].y), pack_bf16(y[1].x, y[1].y),
                                                      pack_bf16(y[2].x, y[2].y), pack_bf16(y[3].x, y[3].y));
        else
          *reinterpret_cast<float4*>(dst) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
      }
    }
    __syncthreads();  // done with this buffer before the next iteration refills it
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

static int sm_count() {
  int n = 148;
  return device_sms(&n) == cudaSuccess ? n : 148;
}

// Grid of the two prologue kernels: one warp per (batch, group of 256 / head_dim heads, token chunk), capped.  The chunk
// is halved down to one group of PRO_TG tokens while the tasks leave schedulers without a second warp: a chunk is a chain
// of loads and stores, and a short prompt's time is that chain (1 x 1001 tokens, 12 heads: 20.4 us with chunks of 32).
static int prologue_grid(int B, int H, int T, int head_dim, int first_chunk, int per_sm, int* tchunk) {
  const int hpw = 256 / head_dim;
  const long cap = (long)sm_count() * per_sm;
  int ch = first_chunk;
  auto tasks = [&](int c) { return (long)B * ((H + hpw - 1) / hpw) * ((T + c - 1) / c); };
  while (ch > PRO_TG && tasks(ch) < (long)sm_count() * 8) ch /= 2;
  *tchunk = ch;
  const long want = (tasks(ch) + PRO_THREADS / 32 - 1) / (PRO_THREADS / 32);
  return (int)(want < 1 ? 1 : (want > cap ? cap : want));
}

template <typename T, int FD>
static cudaError_t launch_pro_t(const LayerProParams& p, int grid, cudaStream_t st) {
  if (p.conv_q_w != nullptr)
    return launch_dependent(ttt_layer_prologue_kernel<T, true, FD>, grid, PRO_THREADS, 0, st, p);
  return launch_dependent(ttt_layer_prologue_kernel<T, false, FD>, grid, PRO_THREADS, 0, st, p);
}

cudaError_t launch_layer_prologue(int dtype, int head_dim, const LayerProParams& p0, cudaStream_t st) {
  LayerProParams p = p0;
  const int grid = prologue_grid(p.B, p.H, p.T, head_dim, PRO_TCHUNK, 8, &p.tchunk);
  if (head_dim == 32) return dtype == 1 ? launch_pro_t<__nv_bfloat16, 32>(p, grid, st) : launch_pro_t<float, 32>(p, grid, st);
  return dtype == 1 ? launch_pro_t<__nv_bfloat16, 64>(p, grid, st) : launch_pro_t<float, 64>(p, grid, st);
}

template <typename T, int MAXCH, int FD, bool GATE>
static cudaError_t launch_epi_g(LayerEpiParams p, cudaStream_t st) {
  const int C = p.H * FD, nch = C / (16 / (int)sizeof(T));
  constexpr int TT = 64 / MAXCH, MAXT = MAXCH == 16 ? 512 : EPI_THREADS;
  auto kfn = ttt_layer_epilogue_kernel<T, MAXCH, FD, GATE>;
  // Row groups g, rows of a tile, threads.  128 MB of input, bf16 / bf16 gated, us (g, rows, threads):
  //   up to 72 chunks (four groups use the threads that a row per warp wants): 448 features (4, 16, 224) 72 / 140, (1, 11, 64)
  //     78 / 166, (6, 12, 384) 78 / 154; 64 features (4, 16, 32) 227 / 302, (4, 4, 32) 246 / 320, (16, 16, 128) 244 / 319
  //   up to 95: two groups, 640 features (2, 12, 160) 64 / 132, (4, 16, 320) 69 / 141; 704 (2, 12, 192) 62 / 138, (1, 11, 96) 65 / 153
  //   more: whole blocks of a warp per row, 768 features (4, 12, 384) 59 / 124, (4, 16, 384) 63 / 125; float32, 448 features
  //     (3, 12, 384) 48 / 91, (1, 11, 128) 54 / 114
  // Rows of more than 512 bytes x 4 (TT < 16): as many groups as fit, a row per warp.
  p.row_groups = MAXT / nch < TT ? MAXT / nch : TT;
  int threads = (p.row_groups * nch + 31) & ~31;
  p.tile_rows = threads / 32 < TT ? threads / 32 : TT;
  if (TT == 16) {
    p.row_groups = nch <= 72 ? 4 : nch < 96 ? 2 : MAXT / nch;
    p.tile_rows = nch <= 72 ? 16 : 12;
    threads = nch < 96 ? (p.row_groups * nch + 31) & ~31 : MAXT;
  }
  const size_t smem = 2 * (size_t)p.tile_rows * C * sizeof(T) + p.tile_rows * sizeof(float2);
  static DeviceValue resident;
  int per_sm = 1;
  cudaError_t e = resident.get((uint32_t)C, &per_sm, [&](int* n) {
    constexpr int CMAX = 512 * MAXCH / (int)sizeof(T);  // the widest row of this instantiation
    const cudaError_t a = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               2 * TT * CMAX * (int)sizeof(T) + TT * (int)sizeof(float2));
    return a != cudaSuccess ? a : cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kfn, threads, smem);
  });
  if (e != cudaSuccess) return e;
  const long ntiles = (long)p.B * ((p.T + p.tile_rows - 1) / p.tile_rows);
  const long cap = (long)sm_count() * (per_sm < 1 ? 1 : per_sm);
  const int grid = (int)(ntiles < cap ? ntiles : cap);
  return launch_dependent(kfn, grid < 1 ? 1 : grid, threads, smem, st, p);
}
template <typename T, int MAXCH, int FD>
static cudaError_t launch_epi_t(const LayerEpiParams& p, cudaStream_t st) {
  return p.gate != nullptr ? launch_epi_g<T, MAXCH, FD, true>(p, st) : launch_epi_g<T, MAXCH, FD, false>(p, st);
}

template <int FD>
static cudaError_t launch_epi_f(int dtype, const LayerEpiParams& p, cudaStream_t st) {
  // chunks of one row per lane: H*F elements / (elements per 16 bytes) / 32 lanes
  const int C = p.H * FD;
  if (dtype == 1) return C <= 1024 ? launch_epi_t<__nv_bfloat16, 4, FD>(p, st) : launch_epi_t<__nv_bfloat16, 8, FD>(p, st);
  if (C <= 512) return launch_epi_t<float, 4, FD>(p, st);
  return C <= 1024 ? launch_epi_t<float, 8, FD>(p, st) : launch_epi_t<float, 16, FD>(p, st);
}

cudaError_t launch_layer_epilogue(int dtype, int head_dim, const LayerEpiParams& p, cudaStream_t st) {
  return head_dim == 32 ? launch_epi_f<32>(dtype, p, st) : launch_epi_f<64>(dtype, p, st);
}

}  // namespace ttt

// =====================================================================================================
// Backward of the two layer steps (training).  Reference: Burn autodiff over the tensor ops of
// rust/layer/src/ttt.rs:152-299; here each step's gradient is one more bandwidth-bound pass.
// =====================================================================================================
namespace ttt {

// Prologue backward (configuration without the shared-QK convolutions): gradients of XQ, XK, XV [B,H,T,F] go back
// to the projection layout [B*T, ld] with the inverse rotation applied to q and k; the gradient of ttt_lr_eta goes
// back through the sigmoid to the logits' columns (lr = c sigma(z), c = base_lr / F  =>  dz = dlr * lr * (1 - lr/c));
// padding columns after the H logit columns are zeroed.
template <typename T, int FD>
__global__ void __launch_bounds__(PRO_THREADS, sizeof(T) == 2 ? 3 : 1) ttt_layer_prologue_bwd_kernel(const LayerProBwdParams p) {
  __shared__ float2 rope_tab[PRO_MAXPOS][32];
  constexpr int F = FD, SUBS = FD / 8, HPW = 32 / SUBS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int H = p.H, NT = p.T;
  const bool rope = p.rope_mode != 0, rope_wrap = p.rope_mode == 1;
  const float log2_theta = log2f(p.rope_theta);
  if (rope && rope_wrap) {
    for (int e = tid; e < p.pos_mod * 32; e += PRO_THREADS) {
      const int pos = e >> 5, i = e & 31;
      float s, c;
      sincosf(pos * exp2f(-(2.f * i / F) * log2_theta), &s, &c);
      rope_tab[pos][i] = make_float2(c, s);
    }
  }
  __syncthreads();
  const int hq = lane / SUBS, sub = lane % SUBS;
  const int hgroups = (H + HPW - 1) / HPW, tchunks = (NT + p.tchunk - 1) / p.tchunk;
  const long ntasks = (long)p.B * hgroups * tchunks;
  for (long task = (long)blockIdx.x * (PRO_THREADS / 32) + warp; task < ntasks; task += (long)gridDim.x * (PRO_THREADS / 32)) {
    const int hg = (int)(task % hgroups);
    const int tc = (int)((task / hgroups) % tchunks);
    const int b = (int)(task / ((long)tchunks * hgroups));
    const int h = HPW * hg + hq;
    if (h >= H) continue;
    const int col = h * F + 8 * sub;
    const int t0 = tc * p.tchunk, t1 = min(NT, t0 + p.tchunk);
    for (int tb = t0; tb < t1; tb += PRO_TG) {
      Vec8<T> vq[PRO_TG], vk[PRO_TG], vv[PRO_TG];
#pragma unroll
      for (int u = 0; u < PRO_TG; ++u) {
        if (tb + u < t1) {
          const size_t srow = (((size_t)b * H + h) * NT + tb + u) * F + 8 * sub;
          vq[u].load(static_cast<const T*>(p.dxq) + srow);
          vk[u].load(static_cast<const T*>(p.dxk) + srow);
          vv[u].load(static_cast<const T*>(p.dxv) + srow);
        }
      }
#pragma unroll
      for (int u = 0; u < PRO_TG; ++u) {
        const int t = tb + u;
        if (t < t1) {
          if (rope) {
            float fq[8], fk[8];
            vq[u].unpack(fq);
            vk[u].unpack(fk);
            const int pos = p.start_idx + t;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float2 cs;
              if (rope_wrap) {
                cs = rope_tab[pos % p.pos_mod][4 * sub + j];
              } else {
                sincosf(pos * exp2f(-(2.f * (4 * sub + j) / F) * log2_theta), &cs.y, &cs.x);
              }
              // transpose of the forward rotation
              const float q0 = fq[2 * j], q1 = fq[2 * j + 1], k0 = fk[2 * j], k1 = fk[2 * j + 1];
              fq[2 * j] = q0 * cs.x + q1 * cs.y;
              fq[2 * j + 1] = q1 * cs.x - q0 * cs.y;
              fk[2 * j] = k0 * cs.x + k1 * cs.y;
              fk[2 * j + 1] = k1 * cs.x - k0 * cs.y;
            }
            vq[u].pack(fq);
            vk[u].pack(fk);
          }
          const size_t drow = ((size_t)b * NT + t) * p.ld_dst + col;
          vq[u].store_once(static_cast<T*>(p.dq_dst) + drow);
          vk[u].store_once(static_cast<T*>(p.dk_dst) + drow);
          vv[u].store_once(static_cast<T*>(p.dv_dst) + drow);
        }
      }
    }
  }
  // logits' columns, four elements of a thread at a time (their loads in flight together)
  const float inv_c = (float)F / p.base_lr;
  const long nlr = (long)p.B * NT * p.lr_cols, step = (long)gridDim.x * PRO_THREADS;
  for (long e0 = (long)blockIdx.x * PRO_THREADS + tid; e0 < nlr; e0 += 4 * step) {
    float lr[4], dl[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long e = e0 + u * step, row = e / p.lr_cols;  // b * T + t
      const int h = (int)(e % p.lr_cols);
      lr[u] = dl[u] = 0.f;
      if (e < nlr && h < H) {
        const int t = (int)(row % NT), b = (int)(row / NT);
        const size_t i = ((size_t)b * H + h) * NT + t;
        lr[u] = ld_as_float<T>(p.lr, i);
        dl[u] = ld_as_float<T>(p.dlr, i);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long e = e0 + u * step;
      if (e < nlr) st_from_float<T>(p.dlogits_dst, (size_t)(e / p.lr_cols) * p.ld_dlr + (int)(e % p.lr_cols), dl[u] * lr[u] * (1.f - lr[u] * inv_c));
    }
  }
}

// Epilogue backward, one pass over the token tiles: with dn = dy * gelu(g) and n = gamma x_hat + beta (without a gate dn = dy)
//   dg = dy * n * gelu'(g),  dz = rstd * (dx - mean(dx) - x_hat * mean(dx * x_hat)),  dx = dn * gamma,
//   d weight[c] = sum over tokens of dn * x_hat,  d bias[c] = sum of dn.
// Bound by memory (dy and the inner output read once, dz written once), so everything happens while a tile of TT tokens is
// in shared memory, both operands double-buffered with asynchronous copies.  Row phase: a warp per row, two rounds of
// shuffles (the mean; then the variance and both sums of dx together).  Column phase: a thread per 16-byte chunk of columns
// and row group, which writes dz straight to [B,H,T,F] and keeps its columns' parameter sums in registers over all of the
// CTA's tiles; the row groups meet in shared memory at the end and leave one [2][C] row of `partials` per CTA.
// 65536 tokens x 768, bf16: 187 -> 86 -> 72 us without a gate (the last step: packed arithmetic, tiles of a row per warp, no
// divisions), 359 -> 208 us with one; float32 409 -> 104 us (the parameter sums were a kernel of their own that read both
// operands again).  TT: with a gate (whose row phase is bound by tanh) half, so
// that the tanh values that the column phase uses again fit beside two CTAs' tiles.
constexpr int EPI_BWD_THREADS = 384;
template <typename T, int MAXCH, int FD, bool GATE>
__global__ void __launch_bounds__(MAXCH == 16 ? 512 : EPI_BWD_THREADS, (sizeof(T) == 2 || MAXCH == 16) ? 2 : 3)
    ttt_layer_epilogue_bwd_kernel(const LayerEpiBwdParams p) {
  constexpr int HD = FD;  // features per head in this instantiation
  const int TT = p.tile_rows;
  constexpr int EPC = 16 / sizeof(T);
  extern __shared__ __align__(16) uint8_t epi_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int H = p.H, NT = p.T, C = H * HD;
  const int nch = C / EPC, ngroups = p.row_groups;
  const size_t tile_bytes = (size_t)TT * C * sizeof(T);
  float4* stat = reinterpret_cast<float4*>(epi_smem + 4 * tile_bytes);  // per row: mean, rstd, mean(dx), mean(dx x_hat)
  float* gam = reinterpret_cast<float*>(stat + TT);
  float* th_tile = gam + C;  // with a gate: the row phase's tanh values [TT][C], for the column phase
  for (int c = tid; c < C; c += blockDim.x) gam[c] = ld_as_float<T>(p.ln_w, (size_t)c);
  const int tiles_per_b = (NT + TT - 1) / TT;
  const long ntiles = (long)p.B * tiles_per_b;
  const int my_ch = tid % nch, my_grp = tid / nch, c_own = my_ch * EPC;
  const int h_own = c_own / HD, f_own = c_own - h_own * HD;

  // the next tile that is not on its way yet: the inner output to buffer `buf`, dy to buffer 2 + buf (both [TT][C])
  TileWalk ahead(blockIdx.x, gridDim.x, ntiles, tiles_per_b), cur = ahead;
  auto fetch = [&](int buf) {
    if (ahead.valid()) {
      const int b = ahead.b, t0 = ahead.t * TT;
      const int rows = min(TT, NT - t0);
      if (my_grp < ngroups) {
        const uint32_t dst = smem_u32(epi_smem + buf * tile_bytes) + (uint32_t)(c_own * sizeof(T));
        const T* z = static_cast<const T*>(p.inner_out) + (((size_t)b * H + h_own) * NT + t0) * HD + f_own;
        const T* y = static_cast<const T*>(p.dy) + ((size_t)b * NT + t0) * C + c_own;
        for (int r = my_grp; r < rows; r += ngroups) {
          const uint32_t d = dst + (uint32_t)(r * C * sizeof(T));
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(z + (size_t)r * HD) : "memory");
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 2 * (uint32_t)tile_bytes), "l"(y + (size_t)r * C)
                       : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ahead.step(gridDim.x);
  };
  constexpr int NPAIR = EPC / 2;
  auto chunk = [](const void* src, F2 (&f)[NPAIR]) {
    const uint4 v = *reinterpret_cast<const uint4*>(src);
    if constexpr (sizeof(T) == 2) {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) f[k] = f2(bf16_lo(w[k]), bf16_hi(w[k]));
    } else {
      f[0] = f2(__uint_as_float(v.x), __uint_as_float(v.y));
      f[1] = f2(__uint_as_float(v.z), __uint_as_float(v.w));
    }
  };
  auto gate_chunk = [&](size_t tok, int c0, F2 (&g)[NPAIR]) {  // (rows of the gate buffer are aligned to 8 bytes only)
    const uint2* src = reinterpret_cast<const uint2*>(static_cast<const T*>(p.gate) + tok * p.ld_gate + c0);
    const uint2 a = src[0], b = src[1];
    if constexpr (sizeof(T) == 2) {
      const uint32_t w[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
      for (int k = 0; k < 4; ++k) g[k] = f2(bf16_lo(w[k]), bf16_hi(w[k]));
    } else {
      g[0] = f2(__uint_as_float(a.x), __uint_as_float(a.y));
      g[1] = f2(__uint_as_float(b.x), __uint_as_float(b.y));
    }
  };
  auto gelu_tanh = [](float g) { return tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g)); };

  F2 ag[NPAIR], ab[NPAIR], gam_own[NPAIR], bet_own[NPAIR];
#pragma unroll
  for (int k = 0; k < NPAIR; ++k) {
    const size_t c = (size_t)(c_own + 2 * k);
    ag[k] = ab[k] = f2(0.f);
    gam_own[k] = f2(ld_as_float<T>(p.ln_w, c), ld_as_float<T>(p.ln_w, c + 1));
    bet_own[k] = GATE ? f2(ld_as_float<T>(p.ln_b, c), ld_as_float<T>(p.ln_b, c + 1)) : f2(0.f);
  }
  int buf = 0;
  fetch(0);
  for (; cur.valid(); cur.step(gridDim.x), buf ^= 1) {
    const int b = cur.b, t0 = cur.t * TT;
    const int rows = min(TT, NT - t0);
    fetch(buf ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const uint8_t* zt = epi_smem + buf * tile_bytes;
    const uint8_t* yt = zt + 2 * tile_bytes;
    for (int r = warp; r < rows; r += nwarps) {
      const T* zr = reinterpret_cast<const T*>(zt) + (size_t)r * C;
      const T* yr = reinterpret_cast<const T*>(yt) + (size_t)r * C;
      // (row sums in the order of the columns: a learning-rate position's gradient is a difference of large sums and shows their last
      // bits)
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < MAXCH; ++j)
        if (j * 32 + lane < nch) {
          F2 v[NPAIR];
          chunk(zr + (j * 32 + lane) * EPC, v);
#pragma unroll
          for (int k = 0; k < NPAIR; ++k) s = s + v[k].x + v[k].y;
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const float mean = s / C;
      float q = 0.f, m1 = 0.f, m2 = 0.f;
#pragma unroll
      for (int j = 0; j < MAXCH; ++j)
        if (j * 32 + lane < nch) {
          const int c0 = (j * 32 + lane) * EPC;
          F2 v[NPAIR], dn[NPAIR];
          chunk(zr + c0, v);
          chunk(yr + c0, dn);
          if constexpr (GATE) {
            F2 g[NPAIR], th[NPAIR];
            gate_chunk((size_t)b * NT + t0 + r, c0, g);
#pragma unroll
            for (int k = 0; k < NPAIR; ++k) {
              th[k] = f2(gelu_tanh(g[k].x), gelu_tanh(g[k].y));
              dn[k] = f2mul(dn[k], f2mul(f2mul(g[k], f2(0.5f)), f2add(th[k], f2(1.f))));
            }
#pragma unroll
            for (int k = 0; k < NPAIR; k += 2)
              *reinterpret_cast<float4*>(&th_tile[(size_t)r * C + c0 + 2 * k]) = make_float4(th[k].x, th[k].y, th[k + 1].x, th[k + 1].y);
          }
#pragma unroll
          for (int k = 0; k < NPAIR; ++k) {
            const F2 x = f2sub(v[k], f2(mean)), dx = f2mul(dn[k], *reinterpret_cast<const F2*>(&gam[c0 + 2 * k]));
            q = fmaf(x.y, x.y, fmaf(x.x, x.x, q));
            m1 = m1 + dx.x + dx.y;
            m2 = fmaf(dx.y, x.y, fmaf(dx.x, x.x, m2));
          }
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        q += __shfl_xor_sync(0xffffffffu, q, o);
        m1 += __shfl_xor_sync(0xffffffffu, m1, o);
        m2 += __shfl_xor_sync(0xffffffffu, m2, o);
      }
      const float rstd = 1.f / sqrtf(q / C + p.eps);
      if (lane == 0) stat[r] = make_float4(mean, rstd, m1 / C, m2 * rstd / C);
    }
    __syncthreads();
    if (my_grp < ngroups) {
      T* out = static_cast<T*>(p.d_inner) + (((size_t)b * H + h_own) * NT + t0) * HD + f_own;
      for (int r = my_grp; r < rows; r += ngroups) {
        const float4 st = stat[r];
        const size_t tok = (size_t)b * NT + t0 + r;
        F2 z[NPAIR], dn[NPAIR];
        chunk(reinterpret_cast<const T*>(zt) + (size_t)r * C + c_own, z);
        chunk(reinterpret_cast<const T*>(yt) + (size_t)r * C + c_own, dn);
        if constexpr (GATE) {
          F2 g[NPAIR], dg[NPAIR];
          gate_chunk(tok, c_own, g);
#pragma unroll
          for (int k = 0; k < NPAIR; ++k) {
            const F2 th = *reinterpret_cast<const F2*>(&th_tile[(size_t)r * C + c_own + 2 * k]);
            const F2 half = f2fma(th, f2(0.5f), f2(0.5f)), g2 = f2mul(g[k], g[k]);  // 0.5 (1 + tanh)
            const F2 slope = f2fma(g2, f2(3.f * 0.044715f * 0.7978845608028654f), f2(0.7978845608028654f));
            const F2 dgelu = f2fma(f2mul(f2mul(g[k], f2(0.5f)), f2fma(f2neg(th), th, f2(1.f))), slope, half);
            const F2 n = f2fma(gam_own[k], f2mul(f2sub(z[k], f2(st.x)), f2(st.y)), bet_own[k]);
            dg[k] = f2mul(f2mul(dn[k], n), dgelu);
            dn[k] = f2mul(dn[k], f2mul(g[k], half));
          }
          uint2* dst = reinterpret_cast<uint2*>(static_cast<T*>(p.dgate) + tok * p.ld_dgate + c_own);
          if constexpr (sizeof(T) == 2) {
            dst[0] = make_uint2(pack_bf16(dg[0].x, dg[0].y), pack_bf16(dg[1].x, dg[1].y));
            dst[1] = make_uint2(pack_bf16(dg[2].x, dg[2].y), pack_bf16(dg[3].x, dg[3].y));
          } else {
            dst[0] = make_uint2(__float_as_uint(dg[0].x), __float_as_uint(dg[0].y));
            dst[1] = make_uint2(__float_as_uint(dg[1].x), __float_as_uint(dg[1].y));
          }
        }
#pragma unroll
        for (int k = 0; k < NPAIR; ++k) {
          const F2 xh = f2mul(f2sub(z[k], f2(st.x)), f2(st.y));
          ag[k] = f2fma(dn[k], xh, ag[k]);
          ab[k] = f2add(ab[k], dn[k]);
          z[k] = f2mul(f2fma(xh, f2(-st.w), f2fma(dn[k], gam_own[k], f2(-st.z))), f2(st.y));
        }
        uint4 o;
        if constexpr (sizeof(T) == 2)
          o = make_uint4(pack_bf16(z[0].x, z[0].y), pack_bf16(z[1].x, z[1].y), pack_bf16(z[2].x, z[2].y), pack_bf16(z[3].x, z[3].y));
        else
          o = make_uint4(__float_as_uint(z[0].x), __float_as_uint(z[0].y), __float_as_uint(z[1].x), __float_as_uint(z[1].y));
        *reinterpret_cast<uint4*>(out + (size_t)r * HD) = o;
      }
    }
    __syncthreads();  // done with this buffer before the next iteration refills it
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // row groups to shared memory ([group][2][C] float32, over the tile buffers), summed in group order
  float* red = reinterpret_cast<float*>(epi_smem);
  if (my_grp < ngroups) {
#pragma unroll
    for (int k = 0; k < NPAIR; ++k) {
      *reinterpret_cast<F2*>(&red[(size_t)my_grp * 2 * C + c_own + 2 * k]) = ag[k];
      *reinterpret_cast<F2*>(&red[(size_t)my_grp * 2 * C + C + c_own + 2 * k]) = ab[k];
    }
  }
  __syncthreads();
  for (int c = tid; c < 2 * C; c += blockDim.x) {
    float sum = red[c];
    for (int g = 1; g < ngroups; ++g) sum += red[(size_t)g * 2 * C + c];
    p.partials[(size_t)blockIdx.x * 2 * C + c] = sum;
  }
}

// d post_norm_weight / d post_norm_bias: the CTAs' partial rows added in a fixed order.  A CTA owns 32 columns;
// its 8 warps each add an interleaved eighth of the parts (lanes = columns, so every load is one coalesced 128-byte
// row segment), and the eight sums are combined in warp order through shared memory.
__global__ void __launch_bounds__(256) ttt_layer_epilogue_bwd_reduce_kernel(const float* partials, int nparts, int C,
                                                                            float* dw, float* db) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;  // column of the [2][C] row
  float s = 0.f;
  if (c < 2 * C)
    for (int i = warp; i < nparts; i += 8) s += partials[(size_t)i * 2 * C + c];
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < 2 * C) {
    float tot = red[0][lane];
#pragma unroll
    for (int w = 1; w < 8; ++w) tot += red[w][lane];
    if (c < C)
      dw[c] = tot;
    else
      db[c - C] = tot;
  }
}

cudaError_t launch_layer_prologue_bwd(int dtype, int head_dim, const LayerProBwdParams& p0, cudaStream_t st) {
  LayerProBwdParams p = p0;
  // as many blocks as are resident, each warp several short tasks: a task per warp was 1.7 rounds of them at 65536 tokens x 768
  // (130 us; 107 with two blocks of eight warps per SM, head groups of the same tokens side by side and streaming stores)
  const int grid = prologue_grid(p.B, p.H, p.T, head_dim, PRO_TG, 2, &p.tchunk);
  if (head_dim == 32) {
    if (dtype == 1) ttt_layer_prologue_bwd_kernel<__nv_bfloat16, 32><<<grid, PRO_THREADS, 0, st>>>(p);
    else ttt_layer_prologue_bwd_kernel<float, 32><<<grid, PRO_THREADS, 0, st>>>(p);
  } else {
    if (dtype == 1) ttt_layer_prologue_bwd_kernel<__nv_bfloat16, 64><<<grid, PRO_THREADS, 0, st>>>(p);
    else ttt_layer_prologue_bwd_kernel<float, 64><<<grid, PRO_THREADS, 0, st>>>(p);
  }
  return cudaGetLastError();
}

// CTAs of the epilogue backward, at most: each leaves one row of partial sums
constexpr int EPI_BWD_MAX_CTAS = 148 * 4;
size_t layer_epilogue_bwd_workspace_bytes(int B, int H, int T, int head_dim) {
  const size_t ntok = (size_t)B * T;  // (a tile holds at least one token)
  return (ntok < EPI_BWD_MAX_CTAS ? ntok : EPI_BWD_MAX_CTAS) * 2 * (size_t)H * head_dim * sizeof(float);
}

template <typename T, int MAXCH, int FD, bool GATE>
static cudaError_t launch_epi_bwd_g(LayerEpiBwdParams p, cudaStream_t st) {
  const int C = p.H * FD, nch = C / (16 / (int)sizeof(T));
  constexpr int TT = (GATE ? 32 : 64) / MAXCH, MAXT = MAXCH == 16 ? 512 : EPI_BWD_THREADS;
  auto kfn = ttt_layer_epilogue_bwd_kernel<T, MAXCH, FD, GATE>;
  // as many row groups as fit a CTA, but no more than a tile has rows, and with a gate a warp for each of them (the row phase is
  // bound by tanh; 128 MB of bf16 input: 64 features 1397 us with 64 threads for 8 rows, 872 with 256)
  p.row_groups = MAXT / nch < TT ? MAXT / nch : TT;
  int threads = (p.row_groups * nch + 31) & ~31;
  if (GATE && threads < 32 * TT) threads = 32 * TT;
  // a row of the tile per warp where the tile is not smaller than that (twelve warps of sixteen rows took two turns), unless a
  // row has so few chunks that the column phase would run on a part of the block (64 features: 552 us with 4 rows, 445 with 16)
  p.tile_rows = threads / 32 < TT && nch > 16 ? threads / 32 : TT;
  if (p.row_groups > p.tile_rows) p.row_groups = p.tile_rows;
  const size_t smem = 4 * (size_t)p.tile_rows * C * sizeof(T) + p.tile_rows * sizeof(float4) +
                      (size_t)(GATE ? p.tile_rows + 1 : 1) * C * sizeof(float);
  static DeviceValue resident;
  int per_sm = 1;
  cudaError_t e = resident.get((uint32_t)C, &per_sm, [&](int* n) {
    constexpr int CMAX = 512 * MAXCH / (int)sizeof(T);  // the widest row of this instantiation
    const cudaError_t a = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               4 * TT * CMAX * (int)sizeof(T) + TT * 16 + (GATE ? TT + 1 : 1) * CMAX * 4);
    return a != cudaSuccess ? a : cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kfn, threads, smem);
  });
  if (e != cudaSuccess) return e;
  const long ntiles = (long)p.B * ((p.T + p.tile_rows - 1) / p.tile_rows);
  long grid = (long)sm_count() * (per_sm < 1 ? 1 : per_sm);
  if (grid > EPI_BWD_MAX_CTAS) grid = EPI_BWD_MAX_CTAS;
  if (grid > ntiles) grid = ntiles;
  kfn<<<(int)grid, threads, smem, st>>>(p);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  ttt_layer_epilogue_bwd_reduce_kernel<<<(2 * C + 31) / 32, 256, 0, st>>>(p.partials, (int)grid, C, p.d_ln_w, p.d_ln_b);
  return cudaGetLastError();
}

template <typename T, int MAXCH, int FD>
static cudaError_t launch_epi_bwd_t(const LayerEpiBwdParams& p, cudaStream_t st) {
  return p.gate != nullptr ? launch_epi_bwd_g<T, MAXCH, FD, true>(p, st) : launch_epi_bwd_g<T, MAXCH, FD, false>(p, st);
}
template <int FD>
static cudaError_t launch_epi_bwd_f(int dtype, const LayerEpiBwdParams& p, cudaStream_t st) {
  const int C = p.H * FD;
  if (dtype == 1) return C <= 1024 ? launch_epi_bwd_t<__nv_bfloat16, 4, FD>(p, st) : launch_epi_bwd_t<__nv_bfloat16, 8, FD>(p, st);
  if (C <= 512) return launch_epi_bwd_t<float, 4, FD>(p, st);
  return C <= 1024 ? launch_epi_bwd_t<float, 8, FD>(p, st) : launch_epi_bwd_t<float, 16, FD>(p, st);
}

cudaError_t launch_layer_epilogue_bwd(int dtype, int head_dim, const LayerEpiBwdParams& p, cudaStream_t st) {
  return head_dim == 32 ? launch_epi_bwd_f<32>(dtype, p, st) : launch_epi_bwd_f<64>(dtype, p, st);
}

// ----------------------------------------------------------------------------------------------------
// Shared-QK convolutions as a differentiable step (training path of the shared-QK layout; inference applies them
// inside the prologue kernel).  A thread owns four adjacent channels and walks LAYER_CONV_CHUNK tokens of one batch
// row with a rolling window, so every global access of a warp is one contiguous row piece.
// ----------------------------------------------------------------------------------------------------
template <typename T>
struct Vec4;
template <>
struct Vec4<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const void* p, float (&f)[4]) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    f[0] = bf16_lo(r.x); f[1] = bf16_hi(r.x); f[2] = bf16_lo(r.y); f[3] = bf16_hi(r.y);
  }
  static __device__ __forceinline__ void store(void* p, const float (&f)[4]) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
  }
};
template <>
struct Vec4<float> {
  static __device__ __forceinline__ void load(const void* p, float (&f)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    f[0] = r.x; f[1] = r.y; f[2] = r.z; f[3] = r.w;
  }
  static __device__ __forceinline__ void store(void* p, const float (&f)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  }
};

template <typename T>
__global__ void __launch_bounds__(256) ttt_layer_conv_kernel(const LayerConvParams p) {
  const int ncg = p.C / 4, nch = (p.T + LAYER_CONV_CHUNK - 1) / LAYER_CONV_CHUNK;
  const long total = (long)p.B * nch * ncg;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    const int cg = (int)(idx % ncg);
    const long rest = idx / ncg;
    const int ch = (int)(rest % nch), b = (int)(rest / nch);
    const int c0 = 4 * cg, t0 = ch * LAYER_CONV_CHUNK, t1 = min(t0 + LAYER_CONV_CHUNK, p.T);
    float wq[4][4], wk[4][4], bq[4], bk[4];  // [channel][tap]
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      Vec4<T>::load(static_cast<const T*>(p.wq) + (size_t)(c0 + c) * 4, wq[c]);
      Vec4<T>::load(static_cast<const T*>(p.wk) + (size_t)(c0 + c) * 4, wk[c]);
    }
    Vec4<T>::load(static_cast<const T*>(p.bq) + c0, bq);
    Vec4<T>::load(static_cast<const T*>(p.bk) + c0, bk);
    const T* xb = static_cast<const T*>(p.x) + (size_t)b * p.T * p.ld_x + c0;
    float win[3][4];  // x at t-3, t-2, t-1
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int t = t0 - 3 + d;
      if (t >= 0) {
        Vec4<T>::load(xb + (size_t)t * p.ld_x, win[d]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) win[d][c] = 0.f;
      }
    }
    for (int t = t0; t < t1; ++t) {
      float xv[4], q[4], k[4];
      Vec4<T>::load(xb + (size_t)t * p.ld_x, xv);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        q[c] = bq[c] + wq[c][0] * win[0][c] + wq[c][1] * win[1][c] + wq[c][2] * win[2][c] + wq[c][3] * xv[c];
        k[c] = bk[c] + wk[c][0] * win[0][c] + wk[c][1] * win[1][c] + wk[c][2] * win[2][c] + wk[c][3] * xv[c];
        win[0][c] = win[1][c];
        win[1][c] = win[2][c];
        win[2][c] = xv[c];
      }
      const size_t o = ((size_t)b * p.T + t) * p.C + c0;
      Vec4<T>::store(static_cast<T*>(p.q) + o, q);
      Vec4<T>::store(static_cast<T*>(p.k) + o, k);
    }
  }
}

// dx[t] = sum_j wq[j] dq[t + 3 - j] + wk[j] dk[t + 3 - j] (terms beyond the sequence end dropped); parameter
// gradients d w[j] = sum_t d out[t] x[t - 3 + j], d b = sum_t d out[t], as per-chunk partials (summed afterwards in a
// fixed order).  The chunk is walked from its last token to its first.
template <typename T>
__global__ void __launch_bounds__(256) ttt_layer_conv_bwd_kernel(const LayerConvBwdParams p) {
  const int ncg = p.C / 4, nch = (p.T + LAYER_CONV_CHUNK - 1) / LAYER_CONV_CHUNK;
  const long total = (long)p.B * nch * ncg;
  for (long idx = (long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    const int cg = (int)(idx % ncg);
    const long rest = idx / ncg;
    const int ch = (int)(rest % nch), b = (int)(rest / nch);
    const int c0 = 4 * cg, t0 = ch * LAYER_CONV_CHUNK, t1 = min(t0 + LAYER_CONV_CHUNK, p.T);
    float wq[4][4], wk[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      Vec4<T>::load(static_cast<const T*>(p.wq) + (size_t)(c0 + c) * 4, wq[c]);
      Vec4<T>::load(static_cast<const T*>(p.wk) + (size_t)(c0 + c) * 4, wk[c]);
    }
    const T* xb = static_cast<const T*>(p.x) + (size_t)b * p.T * p.ld_x + c0;
    const T* dqb = static_cast<const T*>(p.dq) + (size_t)b * p.T * p.C + c0;
    const T* dkb = static_cast<const T*>(p.dk) + (size_t)b * p.T * p.C + c0;
    float gq[3][4], gk[3][4];  // d out at t+1, t+2, t+3
    float xw[4][4];            // x at t, t-1, t-2, t-3
    float aq[5][4], ak[5][4];  // accumulators: taps 0..3, bias
#pragma unroll
    for (int j = 0; j < 5; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) aq[j][c] = ak[j][c] = 0.f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int t = t1 + d;
      if (t < p.T) {
        Vec4<T>::load(dqb + (size_t)t * p.C, gq[d]);
        Vec4<T>::load(dkb + (size_t)t * p.C, gk[d]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) gq[d][c] = gk[d][c] = 0.f;
      }
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const int t = t1 - 1 - d;
      if (t >= 0) {
        Vec4<T>::load(xb + (size_t)t * p.ld_x, xw[d]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) xw[d][c] = 0.f;
      }
    }
    for (int t = t1 - 1; t >= t0; --t) {
      float dqv[4], dkv[4], dx[4];
      Vec4<T>::load(dqb + (size_t)t * p.C, dqv);
      Vec4<T>::load(dkb + (size_t)t * p.C, dkv);
      float xn[4];  // x at t-4, for the next step
      if (t - 4 >= 0) {
        Vec4<T>::load(xb + (size_t)(t - 4) * p.ld_x, xn);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) xn[c] = 0.f;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // tap j multiplies x[t - 3 + j]: its transpose sends d out[t + 3 - j] to x[t]
        dx[c] = wq[c][3] * dqv[c] + wq[c][2] * gq[0][c] + wq[c][1] * gq[1][c] + wq[c][0] * gq[2][c] +
                wk[c][3] * dkv[c] + wk[c][2] * gk[0][c] + wk[c][1] * gk[1][c] + wk[c][0] * gk[2][c];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          aq[j][c] += dqv[c] * xw[3 - j][c];
          ak[j][c] += dkv[c] * xw[3 - j][c];
        }
        aq[4][c] += dqv[c];
        ak[4][c] += dkv[c];
        gq[2][c] = gq[1][c]; gq[1][c] = gq[0][c]; gq[0][c] = dqv[c];
        gk[2][c] = gk[1][c]; gk[1][c] = gk[0][c]; gk[0][c] = dkv[c];
        xw[0][c] = xw[1][c]; xw[1][c] = xw[2][c]; xw[2][c] = xw[3][c]; xw[3][c] = xn[c];
      }
      Vec4<T>::store(static_cast<T*>(p.dx) + ((size_t)b * p.T + t) * p.C + c0, dx);
    }
    float* row = p.partials + ((size_t)b * nch + ch) * 10 * p.C;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      *reinterpret_cast<float4*>(row + (size_t)j * p.C + c0) = make_float4(aq[j][0], aq[j][1], aq[j][2], aq[j][3]);
      *reinterpret_cast<float4*>(row + (size_t)(5 + j) * p.C + c0) = make_float4(ak[j][0], ak[j][1], ak[j][2], ak[j][3]);
    }
  }
}

static int conv_grid(const long total) {
  const long want = (total + 255) / 256, cap = (long)sm_count() * 8;
  return (int)(want < 1 ? 1 : (want > cap ? cap : want));
}

cudaError_t launch_layer_conv(int dtype, const LayerConvParams& p, cudaStream_t st) {
  const long total = (long)p.B * ((p.T + LAYER_CONV_CHUNK - 1) / LAYER_CONV_CHUNK) * (p.C / 4);
  if (dtype == 1)
    ttt_layer_conv_kernel<__nv_bfloat16><<<conv_grid(total), 256, 0, st>>>(p);
  else
    ttt_layer_conv_kernel<float><<<conv_grid(total), 256, 0, st>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_layer_conv_bwd(int dtype, const LayerConvBwdParams& p, cudaStream_t st) {
  const int nch = (p.T + LAYER_CONV_CHUNK - 1) / LAYER_CONV_CHUNK;
  const long total = (long)p.B * nch * (p.C / 4);
  if (dtype == 1)
    ttt_layer_conv_bwd_kernel<__nv_bfloat16><<<conv_grid(total), 256, 0, st>>>(p);
  else
    ttt_layer_conv_bwd_kernel<float><<<conv_grid(total), 256, 0, st>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // sum the chunks' partial rows [10 C] in a fixed order: first 5 C -> the q parameters, last 5 C -> the k parameters
  ttt_layer_epilogue_bwd_reduce_kernel<<<(10 * p.C + 31) / 32, 256, 0, st>>>(p.partials, p.B * nch, 5 * p.C,
                                                                            p.dparams_q, p.dparams_k);
  return cudaGetLastError();
}

}  // namespace ttt
