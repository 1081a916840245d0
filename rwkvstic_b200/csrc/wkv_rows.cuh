// WKV-4 over rows laid out [stream][T][C] for the many-rows paths: max-trick state rows of stream s at
// aa / bb / pp + s * state_stride, advanced in place; y = gate * wkv goes over k (fp32) or, rounded to the
// matrices' 16-bit type, to out16.
//
// The recurrence is sequential in t, but it is a scan whose state composes: after n steps without input
// the state (aa, bb, pp) is (aa, bb, pp + n*w), and two states add after bringing them to a common
// exponent.  A CTA takes 32 channels of one stream (a lane per channel, so a row is one 128-byte line) and
// n <= 16 consecutive steps per warp: every warp runs its steps from the empty state, meets the other
// warps once in shared memory, adds up the states in front of it (one maximum, then independent
// exponentials), and runs its steps again (now from L2) with outputs.  States are added in groups of 16
// warps (the state in front of a group is the one in front of the previous group plus that group's 16),
// and n depends on T alone, so a stream's bits do not depend on how many warps a CTA has.  Longer
// sequences continue with the carried state.
// Kept as loops over four steps: with all steps of a warp unrolled and held in registers the kernel took
// 152 instead of 62 us (8 streams x 512 tokens, 2560 channels; 0.65 instructions issued per clock and
// scheduler, the rest waits for L2); requesting the next four steps ahead gained nothing, two at a time
// lost 30 %.  The two passes over 64-step chunks that this replaces took 85 us, and 48 instead of 10 us for
// one stream of 333 tokens at 4096 channels.
#pragma once

#include "common.cuh"
#include "dense_gemv.cuh"

namespace b200 {

constexpr int kWkvSteps = 16;      // steps per warp at most
constexpr int kWkvGroup = 16, kWkvWarpsMax = 2 * kWkvGroup;

__device__ __forceinline__ unsigned short to_bits16(float v, int is_bf16) {
  return is_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

struct WkvParams {
  const float *w, *u;               // [C] decay (negative), first
  float* k;                         // [streams][T][C]
  const float *v, *gate;
  float *aa, *bb, *pp;
  long long state_stride;
  unsigned short* out16;            // null: y over k
  int is_bf16;
  int T, C, steps;                  // steps per warp, 1..kWkvSteps
};

__global__ void __launch_bounds__(kWkvWarpsMax * 32, 1) wkv_span_kernel(const WkvParams P) {
  __shared__ float sa[kWkvWarpsMax][32], sb[kWkvWarpsMax][32], sp[kWkvWarpsMax][32];   // local state of every warp's steps
  __shared__ float ca[32], cb[32], cp[32];                                             // carried state
  griddep_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5, n = P.steps;
  const int c = blockIdx.x * 32 + lane, C = P.C, T = P.T;
  const size_t so = size_t(blockIdx.y) * P.state_stride + c;
  const float wv = __ldg(P.w + c), uv = __ldg(P.u + c);
  if (warp == 0) {     // touched a whole step ago: on their way from DRAM while the GEMM in front still runs
    asm volatile("prefetch.global.L2 [%0];" ::"l"(P.aa + so));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(P.bb + so));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(P.pp + so));
  }
  griddep_wait();
  if (warp == 0) { ca[lane] = P.aa[so]; cb[lane] = P.bb[so]; cp[lane] = P.pp[so]; }
  const size_t base = size_t(blockIdx.y) * T * C + c;
  const unsigned uC = unsigned(C);
  constexpr int U = 4;      // steps fetched at a time
  for (int t0 = 0; t0 < T; t0 += W * n) {
    const int first = t0 + warp * n, len = min(n, T - first);      // this warp's steps; len <= 0: none left
    const size_t row = base + size_t(first) * C;
    const float *kp = P.k + row, *vp = P.v + row, *gp = P.gate + row;
    if (first + n < T) {                                           // somebody follows: a full chunk
      float a = 0.f, b = 0.f, p = -1e30f;
      int t = 0;
      for (; t + U <= n; t += U) {
        float kk[U], vv[U];
#pragma unroll
        for (int i = 0; i < U; ++i) { kk[i] = __ldcg(kp + unsigned(t + i) * uC); vv[i] = __ldcg(vp + unsigned(t + i) * uC); }
#pragma unroll
        for (int i = 0; i < U; ++i) wkv_advance(kk[i], vv[i], wv, a, b, p);
      }
      for (; t < n; ++t) wkv_advance(__ldcg(kp + unsigned(t) * uC), __ldcg(vp + unsigned(t) * uC), wv, a, b, p);
      sa[warp][lane] = a; sb[warp][lane] = b; sp[warp][lane] = p;
    }
    __syncthreads();
    // (a, b, p) after the steps of warps j0 .. j0 + cnt - 1
    auto advance = [&](float& a, float& b, float& p, int j0, int cnt) {
      // finite for a decay of minus infinity (a channel that forgets at once): 0 steps of it are 0, not NaN
      const float wn = fmaxf(wv * float(n), -1e36f);
      float m = p + float(cnt) * wn;
      for (int j = 0; j < cnt; ++j) m = fmaxf(m, sp[j0 + j][lane] + float(cnt - 1 - j) * wn);
      const float e0 = expf(p + float(cnt) * wn - m);
      a *= e0; b *= e0;
#pragma unroll 4
      for (int j = 0; j < cnt; ++j) {
        const float e = expf(sp[j0 + j][lane] + float(cnt - 1 - j) * wn - m);
        a = fmaf(e, sa[j0 + j][lane], a); b = fmaf(e, sb[j0 + j][lane], b);
      }
      p = m;
    };
    float a = ca[lane], b = cb[lane], p = cp[lane];
    const bool more = t0 + W * n < T;
    float na = a, nb = b, np = p;                                  // warp 0: the state carried to the next turn
    if (more && warp == 0)
      for (int g = 0; g < W; g += kWkvGroup) advance(na, nb, np, g, kWkvGroup);
    if (len > 0) {
      const int g0 = warp & ~(kWkvGroup - 1);
      if (g0 > 0) advance(a, b, p, 0, kWkvGroup);
      if (warp > g0) advance(a, b, p, g0, warp - g0);
      auto put = [&](int t, float y) {
        if (P.out16) P.out16[row + unsigned(t) * uC] = to_bits16(y, P.is_bf16);
        else P.k[row + unsigned(t) * uC] = y;
      };
      int t = 0;
      for (; t + U <= len; t += U) {
        float kk[U], vv[U], gg[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const unsigned o = unsigned(t + i) * uC;
          kk[i] = __ldcg(kp + o); vv[i] = __ldcg(vp + o); gg[i] = __ldcg(gp + o);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) put(t + i, gg[i] * wkv_step(kk[i], vv[i], wv, uv, a, b, p));
      }
      for (; t < len; ++t) {
        const unsigned o = unsigned(t) * uC;
        const float k1 = __ldcg(kp + o), v1 = __ldcg(vp + o), g1 = __ldcg(gp + o);
        put(t, g1 * wkv_step(k1, v1, wv, uv, a, b, p));
      }
    }
    if (len > 0 && first + len == T) { P.aa[so] = a; P.bb[so] = b; P.pp[so] = p; }
    if (more) {
      __syncthreads();      // everyone has read the carried state and the local states
      if (warp == 0) { ca[lane] = na; cb[lane] = nb; cp[lane] = np; }
      // the next turn's barrier comes before anyone reads them
    }
  }
}

// One step per stream (T = 1): a thread per (stream, channel).
__global__ void __launch_bounds__(128) wkv_step_kernel(const WkvParams P, int n) {
  griddep_launch_dependents();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const int s = idx / P.C, c = idx - s * P.C;
  const float wv = __ldg(P.w + c), uv = __ldg(P.u + c);
  const size_t so = size_t(s) * P.state_stride + c;
  asm volatile("prefetch.global.L2 [%0];" ::"l"(P.aa + so));
  asm volatile("prefetch.global.L2 [%0];" ::"l"(P.bb + so));
  asm volatile("prefetch.global.L2 [%0];" ::"l"(P.pp + so));
  griddep_wait();
  float a = P.aa[so], b = P.bb[so], p = P.pp[so];
  const float k = __ldcg(P.k + idx), v = __ldcg(P.v + idx), g = __ldcg(P.gate + idx);
  const float y = g * wkv_step(k, v, wv, uv, a, b, p);
  if (P.out16) P.out16[idx] = to_bits16(y, P.is_bf16);
  else P.k[idx] = y;
  P.aa[so] = a; P.bb[so] = b; P.pp[so] = p;
}

// Steps per warp and warps per CTA: T spread over 32 warps; 32 warps in one CTA, or 16 (two CTAs per SM)
// where CTAs of 32 would be more than one per SM (2 streams x 2560 channels are 160 of them: bf16 prompt of
// 2 x 701 tokens 10730 -> 10542 us).
inline void wkv_span_shape(int streams, int T, int C, int sms, int* warps, int* steps) {
  const int n = (T + kWkvWarpsMax - 1) / kWkvWarpsMax;
  *steps = n < kWkvSteps ? n : kWkvSteps;
  const int W = (long long)streams * (C / 32) > sms ? kWkvGroup : kWkvWarpsMax, need = (T + *steps - 1) / *steps;
  *warps = need < W ? need : W;
}

}  // namespace b200
