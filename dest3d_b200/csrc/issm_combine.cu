// out_i = (a_i + b_i) * scale_i for up to eight arrays in ONE launch: the sums that join the two scan directions
// (models/dest_module.py:574 and the gradients of what the directions share: dt, z, A, D, dt_bias, initial states).
// HBM-bound: 16-byte accesses, four in flight per thread; the sum is formed in float and rounded once.
#include "issm_common.cuh"

namespace issm {
namespace {
struct AddArgs { issm_add_item item[ISSM_ADD_MAX]; unsigned first_block[ISSM_ADD_MAX + 1]; int n; };
constexpr int kThreads = 256, kVec = 4;                   // 16 KB of each operand per block

__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b, float s) {
  const float lo = (__uint_as_float(a << 16) + __uint_as_float(b << 16)) * s;
  const float hi = (__uint_as_float(a & 0xffff0000u) + __uint_as_float(b & 0xffff0000u)) * s;
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__global__ void __launch_bounds__(kThreads) k_add_multi(const __grid_constant__ AddArgs p) {
  int k = 0;
  while (k + 1 < p.n && blockIdx.x >= p.first_block[k + 1]) ++k;
  const issm_add_item& it = p.item[k];
  const int64_t nv = it.n / (it.dtype == ISSM_BF16 ? 8 : 4);                  // whole 16-byte vectors
  const int64_t v0 = (int64_t)(blockIdx.x - p.first_block[k]) * (kThreads * kVec) + threadIdx.x;
  const uint4* a = (const uint4*)it.a;
  const uint4* b = (const uint4*)it.b;
  uint4 x[kVec], y[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int64_t v = v0 + i * kThreads;
    if (v < nv) { x[i] = a[v]; y[i] = b[v]; }
  }
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int64_t v = v0 + i * kThreads;
    if (v >= nv) continue;
    uint4 o;
    if (it.dtype == ISSM_BF16) {
      o = make_uint4(add2(x[i].x, y[i].x, it.scale), add2(x[i].y, y[i].y, it.scale), add2(x[i].z, y[i].z, it.scale), add2(x[i].w, y[i].w, it.scale));
    } else {
      auto f = [&](uint32_t u, uint32_t w) { return __float_as_uint((__uint_as_float(u) + __uint_as_float(w)) * it.scale); };
      o = make_uint4(f(x[i].x, y[i].x), f(x[i].y, y[i].y), f(x[i].z, y[i].z), f(x[i].w, y[i].w));
    }
    ((uint4*)it.out)[v] = o;
  }
  if (blockIdx.x == p.first_block[k]) {                   // the elements past the last whole vector
    const int64_t e = nv * (it.dtype == ISSM_BF16 ? 8 : 4) + threadIdx.x;
    if (e < it.n) {
      if (it.dtype == ISSM_BF16) ((bf16*)it.out)[e] = __float2bfloat16_rn((ldf((const bf16*)it.a + e) + ldf((const bf16*)it.b + e)) * it.scale);
      else ((float*)it.out)[e] = (((const float*)it.a)[e] + ((const float*)it.b)[e]) * it.scale;
    }
  }
}

// A projection's operands are 0.1 to 10 MB each at the detector's sizes, so a conversion is its launch: six of them in one.
struct CastArgs { issm_cast_item item[ISSM_ADD_MAX]; unsigned first_block[ISSM_ADD_MAX + 1]; int n; };
constexpr int kCast = kThreads * 2 * 8;                    // elements per block
__global__ void __launch_bounds__(kThreads) k_cast_multi(const __grid_constant__ CastArgs p) {
  int k = 0;
  while (k + 1 < p.n && blockIdx.x >= p.first_block[k + 1]) ++k;
  const issm_cast_item& it = p.item[k];
  const int64_t e0 = (int64_t)(blockIdx.x - p.first_block[k]) * kCast + threadIdx.x * 8;
  const float* sf = (const float*)it.src;
  const bf16* sh = (const bf16*)it.src;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int64_t e = e0 + i * (kThreads * 8);
    if (e + 8 <= it.n) {
      if (it.to_bf16) {
        const float4 u = *(const float4*)(sf + e), v = *(const float4*)(sf + e + 4);
        const __nv_bfloat162 o[4] = {__floats2bfloat162_rn(u.x, u.y), __floats2bfloat162_rn(u.z, u.w), __floats2bfloat162_rn(v.x, v.y),
                                     __floats2bfloat162_rn(v.z, v.w)};
        const uint32_t* w = (const uint32_t*)o;
        *(uint4*)((bf16*)it.dst + e) = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
        const uint4 w = *(const uint4*)(sh + e);
        auto lo = [](uint32_t x) { return __uint_as_float(x << 16); };
        auto hi = [](uint32_t x) { return __uint_as_float(x & 0xffff0000u); };
        *(float4*)((float*)it.dst + e) = make_float4(lo(w.x), hi(w.x), lo(w.y), hi(w.y));
        *(float4*)((float*)it.dst + e + 4) = make_float4(lo(w.z), hi(w.z), lo(w.w), hi(w.w));
      }
    } else {
      for (int64_t j = e; j < it.n && j < e + 8; ++j) {
        if (it.to_bf16) stf((bf16*)it.dst + j, sf[j]);
        else ((float*)it.dst)[j] = ldf(sh + j);
      }
    }
  }
}
}  // namespace
}  // namespace issm

using namespace issm;
extern "C" int issm_b200_add_multi(const issm_add_item* items, int32_t count, void* stream) {
  if (!items) return ISSM_ERR_NULL;
  if (count < 0 || count > ISSM_ADD_MAX) return ISSM_ERR_SHAPE;
  AddArgs p{};
  uint64_t blocks = 0;
  for (int i = 0; i < count; ++i) {
    const issm_add_item& it = items[i];
    if (it.n == 0) continue;
    if (it.n < 0) return ISSM_ERR_SHAPE;
    if (!it.a || !it.b || !it.out) return ISSM_ERR_NULL;
    if (it.dtype != ISSM_F32 && it.dtype != ISSM_BF16) return ISSM_ERR_DTYPE;
    if (((uintptr_t)it.a | (uintptr_t)it.b | (uintptr_t)it.out) & 15) return ISSM_ERR_ALIGN;
    p.item[p.n] = it;
    p.first_block[p.n] = (unsigned)blocks;
    ++p.n;
    const int64_t nv = it.n / (it.dtype == ISSM_BF16 ? 8 : 4);
    blocks += (uint64_t)(nv > 0 ? cdiv64(nv, kThreads * kVec) : 1);
  }
  if (!p.n) return ISSM_OK;
  if (blocks > 0x7fffffffull) return ISSM_ERR_SHAPE;
  p.first_block[p.n] = (unsigned)blocks;
  ISSM_LAUNCH(k_add_multi, (unsigned)blocks, kThreads, 0, (cudaStream_t)stream, p);
  return ISSM_OK;
}

extern "C" int issm_b200_cast_multi(const issm_cast_item* items, int32_t count, void* stream) {
  if (!items) return ISSM_ERR_NULL;
  if (count < 0 || count > ISSM_ADD_MAX) return ISSM_ERR_SHAPE;
  CastArgs p{};
  uint64_t blocks = 0;
  for (int i = 0; i < count; ++i) {
    const issm_cast_item& it = items[i];
    if (it.n == 0) continue;
    if (it.n < 0) return ISSM_ERR_SHAPE;
    if (!it.src || !it.dst) return ISSM_ERR_NULL;
    if (((uintptr_t)it.src | (uintptr_t)it.dst) & 15) return ISSM_ERR_ALIGN;
    p.item[p.n] = it;
    p.first_block[p.n++] = (unsigned)blocks;
    blocks += (uint64_t)cdiv64(it.n, kCast);
  }
  if (!p.n) return ISSM_OK;
  if (blocks > 0x7fffffffull) return ISSM_ERR_SHAPE;
  p.first_block[p.n] = (unsigned)blocks;
  ISSM_LAUNCH(k_cast_multi, (unsigned)blocks, kThreads, 0, (cudaStream_t)stream, p);
  return ISSM_OK;
}
