// The parameter generation in front of the scan (models/dest_module.py:541-559), one read of the distance features:
//   dt[b, l, h, k] = softplus(dist[b, l, k, :] . Wdt[h, :] + tok[b, l, h]) * mask[b, l, k]
//   B [b, l, g, k] = dist[b, l, k, :] . Wb[g, :] + tok[b, l, H + g]          (C, and the second direction's B / C with
//                                                                             their own token terms, alike)
// where the reference runs dt_proj / bc_proj as two Linear layers over dist, transposes both results to the
// (b, l, h, k) layout the scan wants, adds the per-token terms, applies softplus and multiplies by the mask in
// separate elementwise passes.  Here a thread owns one state k of one point: it holds the M distance features in
// registers, forms every output row, and stores each row coalesced over k in the scan's layout.
// Backward: g = d(out) / d(pre) per output row; ddist = sum_r g[r] W[r, :]; the weight gradient sum_k g[r, k] dist[k, j]
// is formed per point from shared-memory tiles and accumulated per block; the token terms are g summed over k in a
// fixed order.
#include "issm_common.cuh"

#include <type_traits>

namespace issm {

constexpr int GLUE_MAX_ROWS = 16;
constexpr int GLUE_FWD_BLOCKS = 148 * 16;

struct GlueArgs {
  int L, K, H, G, back, RW, RO;                            // RW = H + 2G weight rows; RO = H + 2G (+ 2G) output rows
  const void* dist; int64_t d_sb, d_sl, d_sk;
  const float* w; const float* wbc;                        // dt rows (H, M); B / C rows (2G, M)
  const float* tok;                                        // (b, L, RO)
  const float* mask;                                       // (b, L, K) or null
  void* dt; void* bc;                                      // (b, L, H, K), (b, L, RO - H, K)
  const void* ddt;                                         // (b, L, H, K) or null
  const void* gb[4]; int64_t gb_rs;                        // gradients of B, C (, second B, second C): rows of G x K, gb_rs elements per point; null: zero
  void* ddist;                                             // (b, L, K, M)
  float* dwpart;                                           // (blocks, GLUE_MAX_ROWS * M) partial weight gradients
  float* dtok;                                             // (b, L, RO)
};

template <typename T, int M>
__device__ __forceinline__ void load_feats(const T* p, float (&d)[M]) {
  if constexpr (sizeof(T) == 2 && M % 8 == 0) {
#pragma unroll
    for (int c = 0; c < M / 8; ++c) {
      const uint4 u = ((const uint4*)p)[c];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        d[c * 8 + 2 * i] = __uint_as_float(w[i] << 16);
        d[c * 8 + 2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      }
    }
  } else if constexpr (sizeof(T) == 4 && M % 4 == 0) {
#pragma unroll
    for (int c = 0; c < M / 4; ++c) {
      const float4 u = ((const float4*)p)[c];
      d[c * 4] = u.x; d[c * 4 + 1] = u.y; d[c * 4 + 2] = u.z; d[c * 4 + 3] = u.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < M; ++j) d[j] = ldf(p + j);
  }
}

template <typename T, int M>
__device__ __forceinline__ void store_feats(T* p, const float (&d)[M]) {
  if constexpr (sizeof(T) == 2 && M % 8 == 0) {
#pragma unroll
    for (int c = 0; c < M / 8; ++c) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(d[c * 8 + 2 * i], d[c * 8 + 2 * i + 1]);
        w[i] = *(const uint32_t*)&h;
      }
      ((uint4*)p)[c] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  } else if constexpr (sizeof(T) == 4 && M % 4 == 0) {
#pragma unroll
    for (int c = 0; c < M / 4; ++c) ((float4*)p)[c] = make_float4(d[c * 4], d[c * 4 + 1], d[c * 4 + 2], d[c * 4 + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < M; ++j) stf(p + j, d[j]);
  }
}

__device__ __forceinline__ float glue_sigmoid(float v) { return __fdividef(1.f, 1.f + __expf(-v)); }

// softplus with threshold 20 in the log2 domain (hardware ex2 / lg2); below -4 the series of log1p in u = e^v, where
// lg2(1 + u) would lose the low bits of u
__device__ __forceinline__ float glue_softplus(float v) {
  float u, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(u) : "f"(v * 1.4426950408889634f));
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.f + u));
  const float series = u * fmaf(u, fmaf(u, 0.33333333f, -0.5f), 1.f);
  const float r = v < -4.f ? series : s * 0.6931471805599453f;
  return v <= 20.f ? r : v;
}

// one block per point (b, l); a thread owns two adjacent states and computes them with packed fp32 instructions,
// reading four weights per shared-memory access
// TD: element type of dist (and ddist), T: of dt / bc and their gradients (float dist with bfloat16 outputs is what
// autocast hands the block: the features stay float32, the activations are bfloat16)
// Weights wait in shared memory as pairs (w, w): a 128-bit access gives two packed operands, where the scalar form cost a move
// per multiply-add.  Blocks walk the points with a grid stride, so the weights are laid out once per block and not per point.
// 16 x 4096 points x 256 states x 16 features bf16: 312 us before.
// The dt rows are padded to a multiple of four (zero weights) and the B / C rows follow: rows are worked on four at a time, four
// independent chains of multiply-adds (one row at a time left the fp32 pipe waiting for its own results).
constexpr int GLUE_PAD_ROWS = 20;
__host__ __device__ __forceinline__ int glue_hp(int H) { return (H + 3) & ~3; }
template <int M>
__device__ __forceinline__ void weights_to_smem(const GlueArgs& a, float2* sw, int rows) {
  const int hp = glue_hp(a.H);
  for (int i = threadIdx.x; i < rows * M; i += blockDim.x) {
    const int r = i / M, j = i % M;
    const float w = r < hp ? (r < a.H ? a.w[r * M + j] : 0.f) : (r - hp < 2 * a.G ? a.wbc[(r - hp) * M + j] : 0.f);
    sw[i] = make_float2(w, w);
  }
}
// pre[q] += sum_j dp[j] w[q][j] for four consecutive rows
template <int M>
__device__ __forceinline__ void quad_dot(const float2* w, const float2 (&dp)[M], float2 (&pre)[4]) {
#pragma unroll
  for (int c = 0; c < M; c += 2)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 v = *(const float4*)(w + q * M + c);
      pre[q] = __ffma2_rn(dp[c], make_float2(v.x, v.y), pre[q]);
      pre[q] = __ffma2_rn(dp[c + 1], make_float2(v.z, v.w), pre[q]);
    }
}
template <typename TD, typename T, int M>
__global__ void __launch_bounds__(128) k_glue_fwd(GlueArgs a, int npoints) {
  __shared__ __align__(16) float2 sw[GLUE_PAD_ROWS * M];
  weights_to_smem<M>(a, sw, GLUE_PAD_ROWS);
  __syncthreads();
  const bool pair_store = !(a.K & 1);                      // rows of an even number of states keep pairs aligned
  auto put = [&](T* p, float2 v, bool two) {
    if (pair_store) {
      if constexpr (sizeof(T) == 2) *(__nv_bfloat162*)p = __float22bfloat162_rn(v);
      else *(float2*)p = v;
    } else {
      stf(p, v.x);
      if (two) stf(p + 1, v.y);
    }
  };
  const unsigned half = (a.K + 1) / 2, items = (unsigned)npoints * half;
  const int hp = glue_hp(a.H), nbc = 2 * a.G;
  // item = (point, pair of states); consecutive threads take consecutive pairs
  for (unsigned item = blockIdx.x * blockDim.x + threadIdx.x; item < items; item += gridDim.x * blockDim.x) {
    const unsigned row = item / half, b = row / a.L, l = row - b * a.L;
    const int k = 2 * (int)(item - row * half);
    const TD* drow = (const TD*)a.dist + b * a.d_sb + l * a.d_sl + (int64_t)k * a.d_sk;
    const float* tok = a.tok + (size_t)row * a.RO;
    const bool two = k + 1 < a.K;
    float d0[M], d1[M];
    load_feats<TD, M>(drow, d0);
    load_feats<TD, M>(drow + (two ? a.d_sk : 0), d1);
    float2 mk = make_float2(1.f, 1.f);
    if (a.mask) mk = make_float2(a.mask[(size_t)row * a.K + k], a.mask[(size_t)row * a.K + (two ? k + 1 : k)]);
    float2 dp[M];
#pragma unroll
    for (int j = 0; j < M; ++j) dp[j] = make_float2(d0[j], d1[j]);
    T* out = (T*)a.dt + (size_t)row * a.H * a.K + k;
#pragma unroll 1
    for (int r = 0; r < hp; r += 4) {
      float2 pre[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { const float t = r + q < a.H ? __ldg(tok + r + q) : 0.f; pre[q] = make_float2(t, t); }
      quad_dot<M>(sw + r * M, dp, pre);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (r + q < a.H) put(out, __fmul2_rn(make_float2(glue_softplus(pre[q].x), glue_softplus(pre[q].y)), mk), two);
        out += a.K;
      }
    }
    out = (T*)a.bc + (size_t)row * (a.RO - a.H) * a.K + k;
    const float* tk = tok + a.H;
#pragma unroll 1
    for (int r = 0; r < nbc; r += 4) {
      float2 pre[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) pre[q] = make_float2(0.f, 0.f);
      quad_dot<M>(sw + (hp + r) * M, dp, pre);              // rows past the last one have zero weights
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (r + q < nbc) {
          const float t = __ldg(tk + r + q);
          put(out + (r + q) * a.K, __fadd2_rn(pre[q], make_float2(t, t)), two);
          if (a.back) {
            const float u = __ldg(tk + nbc + r + q);
            put(out + (nbc + r + q) * a.K, __fadd2_rn(pre[q], make_float2(u, u)), two);
          }
        }
    }
  }
}

constexpr int GLUE_BWD_WARPS = 4;
constexpr int GLUE_BWD_BLOCKS = 148 * 3;                   // two (16 features) or three blocks of four warps per SM: registers

// Backward: a warp takes whole points and walks their states 64 at a time, two adjacent states per lane; it shares nothing with
// the other warps of the block but the weights, so there is no block barrier in the walk.  Per 64 states:
//  (1) g = d out / d pre per row and ddist = sum_r g[r] W[r, :] with packed pairs; the inputs of the next 64 states are loaded
//      (packed, in registers) before the current ones are worked on;
//  (2) g and the features go through the warp's part of shared memory for the weight gradient sum_k g[r, k] dist[k, j]: a lane
//      owns NR / 2 rows x M / 2 features of it and every eighth state - 48 multiply-adds for four shared-memory reads at
//      10 rows x 16 features - in registers over the whole walk.
// Bound: the fp32 pipe (450 multiply-adds per (point, state)); the block-wide version with staged inputs held 12 warps per SM
// that met at three barriers per point and used a fifth of the issue slots: 16 x 4096 x 256 x 16 bf16 1730 us.
// NR: weight rows padded to 12 or 20 (dt rows to a multiple of four, then the B / C rows).
template <typename TD, typename T, int M, int NR>
__global__ void __launch_bounds__(GLUE_BWD_WARPS * 32, M == 16 ? 2 : 3) k_glue_bwd(GlueArgs a, int npoints, int pairs_ok) {
  constexpr int RH = NR / 2, MH = M / 2, GS = NR, DS = M + 4;      // rows / features of a lane's tile; row strides in shared memory
  __shared__ __align__(16) float2 sw[NR * M];
  __shared__ __align__(16) float sg_all[GLUE_BWD_WARPS][64 * GS];
  __shared__ __align__(16) float sd_all[GLUE_BWD_WARPS][64 * DS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* sg = sg_all[warp];
  float* sd = sd_all[warp];
  weights_to_smem<M>(a, sw, NR);
  for (int i = lane; i < 64 * GS; i += 32) sg[i] = 0.f;
  __syncthreads();
  const int rh = lane & 1, jh = (lane >> 1) & 1, kq = lane >> 2;   // the lane's tile and its share of the states
  float2 acc[RH][MH / 2];
#pragma unroll
  for (int r = 0; r < RH; ++r)
#pragma unroll
    for (int j = 0; j < MH / 2; ++j) acc[r][j] = make_float2(0.f, 0.f);
  constexpr int FW = M * (int)sizeof(TD) / 8;              // 8-byte words of one state's features
  typedef typename std::conditional<sizeof(T) == 2, uint32_t, float2>::type GP;      // a pair of gradients as loaded
  auto up = [](GP v) {
    if constexpr (sizeof(T) == 2) return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    else return v;
  };
  const int per = gridDim.x * GLUE_BWD_WARPS, first = blockIdx.x * GLUE_BWD_WARPS + warp;
  const int nstep = (a.K + 63) / 64, nb = a.RO - a.H, hp = glue_hp(a.H);      // steps per point; B / C gradient rows; padded dt rows
  const bool has_bc = a.gb[0] || a.gb[1] || a.gb[2] || a.gb[3];
  uint2 fx[2][FW];
  GP gh[8];                                  // dt gradient rows, loaded eight at a time
  float2 mk;
  auto pair_at = [&](const T* p, bool in0, bool in1) {
    GP v;
    if constexpr (sizeof(T) == 2) {
      if (pairs_ok) v = in0 ? *(const uint32_t*)p : 0u;
      else v = (in0 ? (uint32_t)*(const uint16_t*)p : 0u) | (in1 ? (uint32_t)*((const uint16_t*)p + 1) << 16 : 0u);
    } else {
      if (pairs_ok) v = in0 ? *(const float2*)p : make_float2(0.f, 0.f);
      else v = make_float2(in0 ? p[0] : 0.f, in1 ? p[1] : 0.f);
    }
    return v;
  };
  auto load = [&](int pt, int step) {                      // features, mask and the first eight dt gradient rows of 64 states
    const int k = step * 64 + 2 * lane;
    const bool in0 = k < a.K, in1 = k + 1 < a.K;
    const int b = pt / a.L, l = pt - b * a.L;
    const TD* d = (const TD*)a.dist + b * a.d_sb + l * a.d_sl;
#pragma unroll
    for (int s2 = 0; s2 < 2; ++s2) {
      const bool in = s2 ? in1 : in0;
      const uint2* p = (const uint2*)(d + (int64_t)(k + s2) * a.d_sk);
      if constexpr (FW % 2 == 0) {
#pragma unroll
        for (int c = 0; c < FW / 2; ++c) {
          const uint4 v = in ? ((const uint4*)p)[c] : make_uint4(0, 0, 0, 0);
          fx[s2][2 * c] = make_uint2(v.x, v.y);
          fx[s2][2 * c + 1] = make_uint2(v.z, v.w);
        }
      } else {
#pragma unroll
        for (int c = 0; c < FW; ++c) fx[s2][c] = in ? p[c] : make_uint2(0, 0);
      }
    }
    mk = make_float2(in0 ? 1.f : 0.f, in1 ? 1.f : 0.f);
    if (a.mask) {
      if (in0) mk.x = a.mask[(int64_t)pt * a.K + k];
      if (in1) mk.y = a.mask[(int64_t)pt * a.K + k + 1];
    }
    if (a.ddt) {
      const T* g = (const T*)a.ddt + (int64_t)pt * a.H * a.K + k;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < a.H) gh[r] = pair_at(g + (int64_t)r * a.K, in0, in1);
    }
  };
  float tsum[NR + 8];
#pragma unroll
  for (int r = 0; r < NR + 8; ++r) tsum[r] = 0.f;
  if (first < npoints) load(first, 0);
  for (int pt = first; pt < npoints; pt += per) {
    const float* tok = a.tok + (int64_t)pt * a.RO;
    for (int step = 0; step < nstep; ++step) {
      const int k = step * 64 + 2 * lane;
      const bool in0 = k < a.K, in1 = k + 1 < a.K;
      float2 dp[M], dd[M], m2 = mk;
      GP g8[8];
#pragma unroll
      for (int s2 = 0; s2 < 2; ++s2) {                     // features: float pairs over the two states; rows of sd
        float f[M];
#pragma unroll
        for (int c = 0; c < FW; ++c) {
          if constexpr (sizeof(TD) == 2) {
            f[4 * c] = __uint_as_float(fx[s2][c].x << 16); f[4 * c + 1] = __uint_as_float(fx[s2][c].x & 0xffff0000u);
            f[4 * c + 2] = __uint_as_float(fx[s2][c].y << 16); f[4 * c + 3] = __uint_as_float(fx[s2][c].y & 0xffff0000u);
          } else {
            f[2 * c] = __uint_as_float(fx[s2][c].x); f[2 * c + 1] = __uint_as_float(fx[s2][c].y);
          }
        }
#pragma unroll
        for (int j = 0; j < M; ++j) { if (s2) dp[j].y = f[j]; else dp[j].x = f[j]; }
#pragma unroll
        for (int c = 0; c < M / 4; ++c) *(float4*)(sd + (2 * lane + s2) * DS + c * 4) = make_float4(f[c * 4], f[c * 4 + 1], f[c * 4 + 2], f[c * 4 + 3]);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) g8[r] = gh[r];
      // gradients of the B / C rows of this step and the inputs of the next one
      GP gb[8];
      auto row_grad = [&](int q) {                         // B / C gradient row q of this step
        const int which = q / a.G;
        const T* p = (const T*)a.gb[which];
        return p ? pair_at(p + (int64_t)pt * a.gb_rs + (int64_t)(q - which * a.G) * a.K + k, in0, in1) : GP{};
      };
      if (has_bc) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r < nb) gb[r] = row_grad(r);
      }
      if (step + 1 < nstep) load(pt, step + 1);
      else if (pt + per < npoints) load(pt + per, 0);
#pragma unroll
      for (int j = 0; j < M; ++j) dd[j] = make_float2(0.f, 0.f);
#pragma unroll
      for (int rq = 0; rq < NR; rq += 4) {
        float2 g[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) g[q] = make_float2(0.f, 0.f);
        if (rq < hp) {
          if (a.ddt) {
            float2 pre[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) { const float t = rq + q < a.H ? __ldg(tok + rq + q) : 0.f; pre[q] = make_float2(t, t); }
            quad_dot<M>(sw + rq * M, dp, pre);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int r = rq + q;
              const float2 s2 = make_float2(pre[q].x <= 20.f ? glue_sigmoid(pre[q].x) : 1.f, pre[q].y <= 20.f ? glue_sigmoid(pre[q].y) : 1.f);
              float2 go = make_float2(0.f, 0.f);
              if (r < a.H) go = r < 8 ? up(g8[r & 7]) : up(pair_at((const T*)a.ddt + ((int64_t)pt * a.H + r) * a.K + k, in0, in1));
              g[q] = __fmul2_rn(__fmul2_rn(go, m2), s2);
              tsum[r] += g[q].x + g[q].y;
            }
          }
        } else if (has_bc) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int c = rq - hp + q, c2 = c + 2 * a.G;   // both directions share the weight row
            if (c >= 2 * a.G) continue;
            g[q] = c == 0 ? up(gb[0]) : c == 1 ? up(gb[1]) : up(row_grad(c));
            if (a.back) g[q] = __fadd2_rn(g[q], c2 == 2 ? up(gb[2]) : c2 == 3 ? up(gb[3]) : up(row_grad(c2)));
          }
        }
#pragma unroll
        for (int c = 0; c < M; c += 2)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 v = *(const float4*)(sw + (rq + q) * M + c);
            dd[c] = __ffma2_rn(g[q], make_float2(v.x, v.y), dd[c]);
            dd[c + 1] = __ffma2_rn(g[q], make_float2(v.z, v.w), dd[c + 1]);
          }
        *(float4*)(sg + (2 * lane) * GS + rq) = make_float4(g[0].x, g[1].x, g[2].x, g[3].x);
        *(float4*)(sg + (2 * lane + 1) * GS + rq) = make_float4(g[0].y, g[1].y, g[2].y, g[3].y);
      }
      if (has_bc) {                                        // token terms of the B / C rows (each output row has its own)
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < nb) {
            const float2 v = q < 4 ? up(gb[q & 3]) : up(row_grad(q));
            tsum[NR + q] += v.x + v.y;
          }
        for (int q = 8; q < nb; ++q) {                     // more than two groups: straight to the token gradient
          const float2 v = up(row_grad(q));
          const float t = warp_sum(v.x + v.y);
          if (lane == 0) { float* o = a.dtok + (int64_t)pt * a.RO + a.H + q; *o = step ? *o + t : t; }
        }
      }
      TD* ddist = (TD*)a.ddist + ((int64_t)pt * a.K + k) * M;
      {
        float f[M];
#pragma unroll
        for (int j = 0; j < M; ++j) f[j] = dd[j].x;
        if (in0) store_feats<TD, M>(ddist, f);
#pragma unroll
        for (int j = 0; j < M; ++j) f[j] = dd[j].y;
        if (in1) store_feats<TD, M>(ddist + M, f);
      }
      __syncwarp();
#pragma unroll 2
      for (int i = 0; i < 8; ++i) {
        const float* gp = sg + (kq + 8 * i) * GS + rh * RH;
        const float* dq = sd + (kq + 8 * i) * DS + jh * MH;
        float gv[RH];
#pragma unroll
        for (int r = 0; r < RH; r += 2) { const float2 v = *(const float2*)(gp + r); gv[r] = v.x; gv[r + 1] = v.y; }
#pragma unroll
        for (int j = 0; j < MH / 2; ++j) {
          const float2 dv = *(const float2*)(dq + 2 * j);
#pragma unroll
          for (int r = 0; r < RH; ++r) acc[r][j] = __ffma2_rn(make_float2(gv[r], gv[r]), dv, acc[r][j]);
        }
      }
      __syncwarp();
    }
    // token gradients of the point: sums over its states
#pragma unroll
    for (int r = 0; r < NR + 8; ++r) {
      const bool head = r < NR;
      const int o = head ? r : a.H + r - NR;
      if (head ? r < a.H : r - NR < nb) {
        const float t = warp_sum(tsum[r]);
        if (lane == 0) a.dtok[(int64_t)pt * a.RO + o] = t;
      }
      tsum[r] = 0.f;
    }
  }
  // the eight shares of the states, then the four warps, in a fixed order
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RH; ++r)
#pragma unroll
    for (int j = 0; j < MH / 2; ++j) {
      float2 v = acc[r][j];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (kq == 0) *(float2*)(sg + (rh * RH + r) * M + jh * MH + 2 * j) = v;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < a.RW * M; i += blockDim.x) {
    const int r = i / M, at = (r < a.H ? r : hp + r - a.H) * M + i % M;
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < GLUE_BWD_WARPS; ++w) t += sg_all[w][at];
    a.dwpart[(size_t)blockIdx.x * GLUE_MAX_ROWS * M + i] = t;
  }
}

// dweight (RW, M) from the per-block partials: 32 outputs by 8 groups per block; a group sums its contiguous share of
// the partials, the groups are combined in a fixed order
__global__ void __launch_bounds__(256) k_glue_reduce(const float* __restrict__ part, int blocks, int stride, int n, float* __restrict__ dw) {
  __shared__ float red[8][32];
  const int o = blockIdx.x * 32 + threadIdx.x, grp = threadIdx.y;
  const int per = (blocks + 7) / 8;
  float acc = 0.f;
  if (o < n) {
    const int i1 = min(blocks, (grp + 1) * per);
#pragma unroll 4
    for (int i = grp * per; i < i1; ++i) acc += part[(size_t)i * stride + o];
  }
  red[grp][threadIdx.x] = acc;
  __syncthreads();
  if (grp == 0 && o < n) {
    float tot = 0.f;
#pragma unroll
    for (int g = 0; g < 8; ++g) tot += red[g][threadIdx.x];
    dw[o] = tot;
  }
}

static int glue_validate(const issm_glue_params* p, bool bwd) {
  if (!p) return ISSM_ERR_NULL;
  if (p->batch <= 0 || p->batch > 65535 || p->seqlen <= 0 || p->nstates <= 0 || p->nheads <= 0 || p->ngroups <= 0) return ISSM_ERR_SHAPE;
  if (p->nfeat != 4 && p->nfeat != 8 && p->nfeat != 16) return ISSM_ERR_SHAPE;
  if (p->nheads + 2 * p->ngroups > GLUE_MAX_ROWS || p->nheads + 4 * p->ngroups > GLUE_MAX_ROWS + 8) return ISSM_ERR_SHAPE;
  if (p->io_dtype != ISSM_F32 && p->io_dtype != ISSM_BF16) return ISSM_ERR_DTYPE;
  if (p->dist_dtype != p->io_dtype && !(p->dist_dtype == ISSM_F32 && p->io_dtype == ISSM_BF16)) return ISSM_ERR_DTYPE;
  if (!p->dist || !p->weight || !p->tok) return ISSM_ERR_NULL;
  if (!bwd && (!p->dt || !p->bc)) return ISSM_ERR_NULL;
  if (bwd && (!p->ddist || !p->dweight || !p->dtok)) return ISSM_ERR_NULL;
  const size_t es = p->dist_dtype == ISSM_F32 ? 4 : 2;
  if (((uintptr_t)p->dist % 16) || (p->dist_sb * es) % 16 || (p->dist_sl * es) % 16 || (p->dist_sk * es) % (p->nfeat * es >= 16 ? 16 : p->nfeat * es))
    return ISSM_ERR_ALIGN;
  return ISSM_OK;
}
static GlueArgs glue_args(const issm_glue_params& p) {
  GlueArgs a{};
  a.L = p.seqlen; a.K = p.nstates; a.H = p.nheads; a.G = p.ngroups; a.back = p.has_back;
  a.RW = p.nheads + 2 * p.ngroups; a.RO = a.RW + (p.has_back ? 2 * p.ngroups : 0);
  a.dist = p.dist; a.d_sb = p.dist_sb; a.d_sl = p.dist_sl; a.d_sk = p.dist_sk;
  a.w = p.weight; a.wbc = p.weight_bc ? p.weight_bc : p.weight + (size_t)p.nheads * p.nfeat; a.tok = p.tok; a.mask = p.mask; a.dt = p.dt; a.bc = p.bc;
  a.ddt = p.ddt; a.ddist = p.ddist; a.dwpart = (float*)p.workspace; a.dtok = p.dtok;
  const int64_t part = (int64_t)p.ngroups * p.nstates;
  a.gb_rs = p.dbc ? (a.RO - p.nheads) * (int64_t)p.nstates : part;
  for (int i = 0; i < (p.has_back ? 4 : 2); ++i)
    a.gb[i] = p.dbc ? (const void*)((const char*)p.dbc + i * part * (p.io_dtype == ISSM_F32 ? 4 : 2)) : p.dbc_part[i];
  return a;
}

// ---- token terms ---------------------------------------------------------------------------------------------------
// one thread per (point, output row): float copies of up to five narrow tensors into one array, and the way back
struct TokSrc { const void* src[5]; void* dst[5]; int64_t sb[5], sl[5]; int f32[5]; };
__global__ void k_glue_tok(TokSrc t, int L, int H, int G, int RO, unsigned n, const float* __restrict__ bias, float* __restrict__ tok,
                           const float* __restrict__ dtok) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned row = i / RO;
  int r = (int)(i - row * RO), s = 0, w = H;
  if (r >= H) { s = 1 + (r - H) / G; r = (r - H) % G; w = G; }
  if (tok) {
    const unsigned b = row / L, l = row - b * L;
    const int64_t at = b * t.sb[s] + l * t.sl[s] + r;
    float v = t.f32[s] ? ((const float*)t.src[s])[at] : ldf((const bf16*)t.src[s] + at);
    if (s == 0 && bias) v += bias[r];
    tok[i] = v;
  } else if (t.dst[s]) {
    const float v = dtok[i];
    if (t.f32[s]) ((float*)t.dst[s])[(size_t)row * w + r] = v;
    else stf((bf16*)t.dst[s] + (size_t)row * w + r, v);
  }
}
}  // namespace issm

using namespace issm;

extern "C" size_t issm_b200_sizeof_glue_tok(void) { return sizeof(issm_glue_tok); }
static int glue_tok_run(const issm_glue_tok* p, void* stream, bool pack) {
  if (!p) return ISSM_ERR_NULL;
  if (p->batch <= 0 || p->seqlen <= 0 || p->nheads <= 0 || p->ngroups <= 0 || (p->nsrc != 3 && p->nsrc != 5)) return ISSM_ERR_SHAPE;
  const int RO = p->nheads + (p->nsrc - 1) * p->ngroups;
  const int64_t n = (int64_t)p->batch * p->seqlen * RO;
  if (n > 0x7fffffff) return ISSM_ERR_SHAPE;
  if (pack ? !p->tok : !p->dtok) return ISSM_ERR_NULL;
  TokSrc t{};
  for (int i = 0; i < p->nsrc; ++i) {
    if (p->dtype[i] != ISSM_F32 && p->dtype[i] != ISSM_BF16) return ISSM_ERR_DTYPE;
    if (pack && !p->src[i]) return ISSM_ERR_NULL;
    t.src[i] = p->src[i]; t.dst[i] = p->dsrc[i]; t.sb[i] = p->sb[i]; t.sl[i] = p->sl[i]; t.f32[i] = p->dtype[i] == ISSM_F32;
  }
  ISSM_LAUNCH(k_glue_tok, (unsigned)cdiv64(n, 256), 256, 0, (cudaStream_t)stream, t, p->seqlen, p->nheads, p->ngroups, RO, (unsigned)n, p->dt_bias,
              pack ? p->tok : nullptr, p->dtok);
  return ISSM_OK;
}
extern "C" int issm_b200_glue_tok_pack(const issm_glue_tok* p, void* stream) { return glue_tok_run(p, stream, true); }
extern "C" int issm_b200_glue_tok_unpack(const issm_glue_tok* p, void* stream) { return glue_tok_run(p, stream, false); }

extern "C" size_t issm_b200_sizeof_glue_params(void) { return sizeof(issm_glue_params); }

extern "C" int issm_b200_glue_fwd(const issm_glue_params* p, void* stream) {
  int rc = glue_validate(p, false);
  if (rc) return rc;
  const GlueArgs a = glue_args(*p);
  if ((int64_t)p->batch * p->seqlen * ((p->nstates + 1) / 2) > 0x7fffffff - 148 * 16 * 128) return ISSM_ERR_SHAPE;
  const int npoints = p->batch * p->seqlen;
  const int64_t want = cdiv64((int64_t)npoints * ((p->nstates + 1) / 2), 128);
  const unsigned grid = (unsigned)(want < GLUE_FWD_BLOCKS ? want : GLUE_FWD_BLOCKS);
  cudaStream_t s = (cudaStream_t)stream;
#define GLUE_FWD_M(TD, T)                                                                             \
  do {                                                                                                \
    if (p->nfeat == 16) ISSM_LAUNCH((k_glue_fwd<TD, T, 16>), grid, 128, 0, s, a, npoints);            \
    else if (p->nfeat == 8) ISSM_LAUNCH((k_glue_fwd<TD, T, 8>), grid, 128, 0, s, a, npoints);         \
    else ISSM_LAUNCH((k_glue_fwd<TD, T, 4>), grid, 128, 0, s, a, npoints);                            \
  } while (0)
  if (p->io_dtype == ISSM_F32) GLUE_FWD_M(float, float);
  else if (p->dist_dtype == ISSM_F32) GLUE_FWD_M(float, bf16);
  else GLUE_FWD_M(bf16, bf16);
#undef GLUE_FWD_M
  return ISSM_OK;
}

static int glue_bwd_blocks(const issm_glue_params* p) {
  const int64_t need = cdiv64((int64_t)p->batch * p->seqlen, GLUE_BWD_WARPS);
  const int64_t most = p->nfeat == 16 ? 148 * 2 : GLUE_BWD_BLOCKS;
  return (int)(need < most ? need : most);
}

extern "C" size_t issm_b200_glue_workspace_bytes(const issm_glue_params* p) {
  if (!p || p->batch <= 0 || p->seqlen <= 0) return 0;
  return align_up((size_t)glue_bwd_blocks(p) * GLUE_MAX_ROWS * 16 * sizeof(float), 256);
}

extern "C" int issm_b200_glue_bwd(const issm_glue_params* p, void* stream) {
  int rc = glue_validate(p, true);
  if (rc) return rc;
  if (!p->workspace || p->workspace_bytes < issm_b200_glue_workspace_bytes(p)) return ISSM_ERR_WORKSPACE;
  if ((int64_t)p->batch * p->seqlen > 0x7fffffff) return ISSM_ERR_SHAPE;
  const GlueArgs a = glue_args(*p);
  const int blocks = glue_bwd_blocks(p), npoints = p->batch * p->seqlen;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t es = p->io_dtype == ISSM_F32 ? 4 : 2;
  // pairs of gradients are one access where every row of states starts on the pair's alignment
  const int pairs_ok = !(p->nstates & 1) && !((uintptr_t)p->ddt % (2 * es)) && !((uintptr_t)p->dbc % (2 * es)) &&
                       !(((uintptr_t)p->dbc_part[0] | (uintptr_t)p->dbc_part[1] | (uintptr_t)p->dbc_part[2] | (uintptr_t)p->dbc_part[3]) % (2 * es));
#define GLUE_BWD(TD, TT, MM)                                                                          \
  do {                                                                                                \
    if (glue_hp(a.H) + 2 * a.G <= 12) ISSM_LAUNCH((k_glue_bwd<TD, TT, MM, 12>), blocks, GLUE_BWD_WARPS * 32, 0, s, a, npoints, pairs_ok); \
    else ISSM_LAUNCH((k_glue_bwd<TD, TT, MM, 20>), blocks, GLUE_BWD_WARPS * 32, 0, s, a, npoints, pairs_ok);            \
  } while (0)
#define GLUE_BWD_M(TD, TT)                                                                            \
  do {                                                                                                \
    if (p->nfeat == 16) GLUE_BWD(TD, TT, 16); else if (p->nfeat == 8) GLUE_BWD(TD, TT, 8); else GLUE_BWD(TD, TT, 4); \
  } while (0)
  if (p->io_dtype == ISSM_F32) GLUE_BWD_M(float, float);
  else if (p->dist_dtype == ISSM_F32) GLUE_BWD_M(float, bf16);
  else GLUE_BWD_M(bf16, bf16);
#undef GLUE_BWD_M
#undef GLUE_BWD
  const int n = a.RW * p->nfeat;
  ISSM_LAUNCH(k_glue_reduce, (n + 31) / 32, dim3(32, 8), 0, s, a.dwpart, blocks, GLUE_MAX_ROWS * p->nfeat, n, p->dweight);
  return ISSM_OK;
}
