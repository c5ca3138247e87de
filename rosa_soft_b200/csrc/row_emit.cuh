// What a resolved row writes: the functors that the match kernels call once per (token, head) with
// the winning match length and route (0, 0: no match).
#pragma once

#include "chain_match.cuh"
#include "common.cuh"

namespace rosa {
namespace {

template <typename T>
__device__ __forceinline__ bool is_positive(T x) { return (float)x > 0.0f; }

// Routed value signs as T or as int8, the winner and optionally the routed token.
template <typename T, typename OutT>
struct SignEmit {
  const T* v;
  OutT* out;
  int32_t* route_token;
  unsigned long long* best;
  int Hv, group, Dv, vec;

  // a row that the chained matcher gave up (length -1) and nobody has resolved yet
  __device__ __forceinline__ bool pending(int64_t th) const { return best[th] == kChainGaveUp; }

  __device__ __forceinline__ void operator()(int64_t g, int h, int H, int start, int length,
                                             int route) const {
    const int64_t th = g * H + h;
    const int64_t src_token = route > 0 ? (int64_t)start + route : -1;
    best[th] = ((unsigned long long)(unsigned)length << 32) | (unsigned)route;
    if (route_token != nullptr) route_token[th] = (int32_t)src_token;
    const T* src = v + (src_token * Hv + (group == 1 ? h : h / group)) * Dv;
    OutT* o = out + th * Dv;
    if (vec) {
      // 16 bytes of output at a time from as many value components
      constexpr int kOutPer = 16 / (int)sizeof(OutT);
      constexpr int kInPer = 16 / (int)sizeof(T);
      for (int d0 = 0; d0 < Dv; d0 += kOutPer) {
        alignas(16) OutT vals[kOutPer];
#pragma unroll
        for (int x = 0; x < kOutPer; ++x) vals[x] = (OutT)0;
        if (route > 0) {
#pragma unroll
          for (int wd = 0; wd < kOutPer / kInPer; ++wd) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src + d0) + wd);
            const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int x = 0; x < kInPer; ++x)
              vals[wd * kInPer + x] = is_positive<T>(e[x]) ? (OutT)1.0f : (OutT)-1.0f;
          }
        }
        *reinterpret_cast<uint4*>(o + d0) = *reinterpret_cast<const uint4*>(vals);
      }
      return;
    }
    for (int d = 0; d < Dv; ++d)
      o[d] = route <= 0 ? (OutT)0 : is_positive<T>(src[d]) ? (OutT)1.0f : (OutT)-1.0f;
  }
};

// Payload row of the successor and the position of the match (-2: the row is pending).
struct PayloadEmit {
  const float* payload;
  float* out;
  int64_t* matched_end;
  int Hp, group, Dp, vec;

  __device__ __forceinline__ bool pending(int64_t th) const { return matched_end[th] == -2; }

  __device__ __forceinline__ void operator()(int64_t g, int h, int H, int start, int length,
                                             int route) const {
    const int64_t th = g * H + h;
    matched_end[th] = length < 0 ? -2 : (int64_t)route - 1;
    if (out == nullptr) return;
    float* o = out + th * Dp;
    const float* src = payload + (((int64_t)start + route) * Hp + (group == 1 ? h : h / group)) * Dp;
    if (vec) {
      for (int d = 0; d < Dp; d += 4)
        *reinterpret_cast<float4*>(o + d) = route > 0
            ? __ldg(reinterpret_cast<const float4*>(src + d)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      return;
    }
    for (int d = 0; d < Dp; ++d) o[d] = route > 0 ? src[d] : 0.0f;
  }
};

inline PayloadEmit make_payload_emit(const FwdArgs& a, const float* payload, float* out,
                                     int64_t* matched_end) {
  const auto aligned = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  return {payload, out, matched_end, a.Hv, a.H / a.Hv, a.Dv,
          a.Dv % 4 == 0 && aligned(payload) && aligned(out)};
}

// Calls f with the functor of the call's value type and output form.
template <typename T, typename OutT>
inline SignEmit<T, OutT> make_sign_emit(const FwdArgs& a, OutT* out) {
  constexpr int kOutPer = 16 / (int)sizeof(OutT);
  const auto aligned = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  return {(const T*)a.v, out, a.route_token, a.best, a.Hv, a.H / a.Hv, a.Dv,
          a.Dv % kOutPer == 0 && aligned(a.v) && aligned(out) && (a.Dv * (int)sizeof(T)) % 16 == 0 &&
              kOutPer >= 16 / (int)sizeof(T)};
}

template <typename F>
inline int with_sign_emit(const FwdArgs& a, F f) {
  if (a.out_i8 != nullptr) {
    if (a.dtype == ROSA_B200_F32) return f(make_sign_emit<float>(a, a.out_i8));
    if (a.dtype == ROSA_B200_F16) return f(make_sign_emit<__half>(a, a.out_i8));
    return f(make_sign_emit<__nv_bfloat16>(a, a.out_i8));
  }
  if (a.dtype == ROSA_B200_F32) return f(make_sign_emit<float>(a, (float*)a.out));
  if (a.dtype == ROSA_B200_F16) return f(make_sign_emit<__half>(a, (__half*)a.out));
  return f(make_sign_emit<__nv_bfloat16>(a, (__nv_bfloat16*)a.out));
}

}  // namespace
}  // namespace rosa
