// Typical sampling on the device: one cluster of CTAs per row of logits, no sort and no host round trip.
//
// What the reference's sampler computes on the host per token (samplers/typical.py:1-17):
//   p = softmax(logits); nl = -log p; ent = sum(nl * p) (NaN terms skipped); s = |nl - ent|;
//   sort by s, running sum of p in that order, cutoff = number of running sums < tau;
//   every p whose s is larger than the s at the cutoff position becomes 0; p <- p^(1/temp);
//   one draw from the resulting (unnormalised) distribution.
// The sort only serves to find one threshold: the smallest value t among the s_i for which the
// mass of {i : s_i <= t} reaches tau.  Here it is found in two steps.  A histogram of mass over 1024
// equal intervals of s gives the interval that holds t; the tokens of that interval (a few hundred
// of 50277) go to a list in shared memory, and a radix select over the bit patterns of their s (s >= 0,
// so float order is unsigned-integer order) gives t.  A row that puts more tokens into the interval
// than the list holds takes the radix select over the whole row.  Masses are fixed point (p * 2^31
// rounded to nearest, 32-bit shared-memory atomics, which are native; 64-bit totals): integer sums do
// not depend on arrival order, so every run sees the same totals, and the rounding (2.3e-10 per token)
// stays below what the reference's fp32 running sum resolves.  The draw is an inverse-CDF walk in
// index order with a uniform number the caller supplies, so a run is reproducible from its seed.
//
// What bounds it: instruction issue and the latency of dependent passes, not bytes.  The row is read
// from memory once, into the shared memory of its cluster (each CTA holds a slice), and the four passes
// over it (maximum, softmax sums, histogram, draw sums with the candidates set aside) run from there.
// Measured at n = 50277: 1 row 19 us, 74 rows 30, 148 rows 40, 256 rows 76 (two waves of clusters), against
// 62 us for 1 row and 111 for 256 with one CTA of 1024 threads per row and eight passes through L2.  ncu
// (256 rows): 0.57 instructions issued per clock and scheduler, the rest fixed latencies and barriers.
#pragma once

#include <cooperative_groups.h>

#include <utility>

#include "common.cuh"

namespace b200 {

constexpr int kSampleThreads = 512;
constexpr int kSampleWarps = kSampleThreads / 32;
constexpr int kSampleMaxCluster = 8;
constexpr int kSampleBins = 2 * kSampleThreads;    // intervals of s; the last one also takes everything beyond
constexpr float kSampleBinsPerUnit = 64.f;         // 1/64 nat each
constexpr int kSampleListCap = 1280;               // candidates the list holds
constexpr int kSampleHists = 8;                    // select over the whole row: lane l adds into histogram l % 8
constexpr int kSampleHistStride = 257;             // odd stride: equal bins of different histograms in different banks
constexpr float kMassScale = 2147483648.0f;        // 2^31
// Two CTAs share an SM (its 228 KB hold two slices of this many logits and the scratch), so that one
// computes while the other waits for loads or its cluster.  Shared memory beyond that is not used.
constexpr int kSampleMaxSlice = 25600;
static_assert(kSampleMaxSlice <= 63 * kSampleThreads, "a thread's tokens must fit its 64-bit candidate mask");

struct TypicalRow {
  float mx;       // largest logit
  float inv_z;    // 1 / sum exp(l - mx)
  float log_z;    // log of that sum
  float ent;      // entropy in nats
};

// The surprise -log p of a logit is log_z - (l - mx): one subtraction instead of a logarithm of an
// exponential (and exact where the reference's fp32 -log(softmax) carries the rounding of p).
__device__ __forceinline__ float typical_shift(float l, const TypicalRow& r) {
  return fabsf((r.log_z - (l - r.mx)) - r.ent);
}
__device__ __forceinline__ float typical_prob(float l, const TypicalRow& r) {
  return expf(l - r.mx) * r.inv_z;
}
__device__ __forceinline__ unsigned typical_mass(float p) { return p > 0.f ? __float2uint_rn(p * kMassScale) : 0u; }
// Interval of s: floor(s * 64), at most kSampleBins - 1 (also for NaN).  The sum with 2^23, rounded
// towards zero, holds the integer in its mantissa.
__device__ __forceinline__ int typical_bin(float s) {
  const float top = (float(kSampleBins) - 0.5f) / kSampleBinsPerUnit;
  return __float_as_int(__fmaf_rz(fminf(s, top), kSampleBinsPerUnit, 8388608.0f)) - 0x4B000000;
}

struct SampleShared {
  union {
    unsigned hist[2][kSampleBins];                           // mass per interval; lane parity picks the copy
    struct { uint2 cand[kSampleListCap]; unsigned bins[256]; } list;   // (bits of s, mass) of the candidates; rank 0's is used
    unsigned radix[kSampleHists][kSampleHistStride];
    double part[kSampleThreads];                             // draw mass per thread
  };
  double warp_z[kSampleWarps], warp_dz[kSampleWarps];
  unsigned long long warp_sum[kSampleWarps];
  float warp_mx[kSampleWarps];
  // one entry per CTA of the cluster, written by that CTA
  double z[kSampleMaxCluster], dz[kSampleMaxCluster], total[kSampleMaxCluster];
  float mx[kSampleMaxCluster];
  TypicalRow row;
  unsigned long long below;     // mass in front of the interval / of the prefix
  unsigned prefix;              // bits of the threshold found so far
  int bin;                      // interval of the threshold; kSampleBins: everything is kept
  int count;                    // candidates (rank 0's)
  unsigned thresh;              // bits of the threshold
};

// Sum of v over the threads before this one.
__device__ __forceinline__ unsigned long long sample_exclusive_scan(unsigned long long v, SampleShared& S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();              // warp_sum may still be read from an earlier call
  if (lane == 31) S.warp_sum[warp] = inc;
  __syncthreads();
  unsigned long long before = inc - v;
  for (int w = 0; w < warp; ++w) before += S.warp_sum[w];
  return before;
}

// logits [rows][ldx]; u: one uniform number in [0,1) per draw, read at u[row + rows * step] where
// step = *history_count when a history is kept and 0 otherwise; out[row] = sampled id;
// probs_out (nullable) [rows][n]: the masked, tempered, unnormalised probabilities the draw used.
// A cluster handles a row, each of its CTAs `slice` consecutive logits.  kInSmem: the slice is held in
// dynamic shared memory (4 * slice bytes); else (rows beyond 8 x kSampleMaxSlice logits) every pass
// reads it from memory.
template <bool kInSmem>
__global__ void __launch_bounds__(kSampleThreads, 2)
sample_typical_kernel(const float* __restrict__ x, int n, long long ldx, float temp, float tau,
                      const float* __restrict__ u, long long* __restrict__ out, float* __restrict__ probs_out,
                      long long* __restrict__ hist, int* __restrict__ hist_count, int hist_cap, int slice) {
  extern __shared__ float held[];
  __shared__ SampleShared S;
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  auto started = cluster.barrier_arrive();     // met before the first access to another CTA's memory
  const int rank = int(cluster.block_rank()), C = int(cluster.num_blocks());
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row_id = int(blockIdx.x) / C, rows = int(gridDim.x) / C;
  const long long first = (long long)rank * slice;
  const int lo = int(first < n ? first : n), len = int(first + slice < n ? first + slice : n) - lo;
  const float* row = x + size_t(row_id) * ldx + lo;
  auto logit = [&](int i) -> float { return kInSmem ? held[i] : __ldg(row + i); };

  // ---- the slice into shared memory, and the largest logit
  float mx = -INFINITY;
  for (int base = tid; base < len; base += 16 * kSampleThreads) {
    float l[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int i = base + j * kSampleThreads;
      l[j] = i < len ? __ldg(row + i) : -INFINITY;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int i = base + j * kSampleThreads;
      if (kInSmem && i < len) held[i] = l[j];
      mx = fmaxf(mx, l[j]);
    }
  }
  mx = warp_max(mx);
  if (lane == 0) S.warp_mx[warp] = mx;
  __syncthreads();
  cluster.barrier_wait(std::move(started));    // every CTA of the cluster runs, so its shared memory exists
  if (tid < C) {
    for (int w = 0; w < kSampleWarps; ++w) mx = fmaxf(mx, S.warp_mx[w]);
    *cluster.map_shared_rank(&S.mx[rank], tid) = mx;
  }
  for (int i = tid; i < 2 * kSampleBins; i += kSampleThreads) (&S.hist[0][0])[i] = 0u;
  cluster.sync();
  mx = S.mx[0];
  for (int c = 1; c < C; ++c) mx = fmaxf(mx, S.mx[c]);

  // ---- Z = sum e^d and sum d e^d (d = l - mx), every term in fp64; entropy = log Z - (sum d e^d) / Z
  double z = 0.0, dz = 0.0;
  auto add4 = [&](const float (&d)[4]) {
    float e[4], de[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      e[j] = expf(d[j]);
      de[j] = e[j] > 0.f ? d[j] * e[j] : 0.f;
    }
    z += (double(e[0]) + double(e[1])) + (double(e[2]) + double(e[3]));
    dz += (double(de[0]) + double(de[1])) + (double(de[2]) + double(de[3]));
  };
  int at = tid;
  for (; at + 3 * kSampleThreads < len; at += 4 * kSampleThreads) {
    float d[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) d[j] = logit(at + j * kSampleThreads) - mx;
    add4(d);
  }
  for (; at < len; at += kSampleThreads) {
    const float d = logit(at) - mx, e = expf(d);
    z += double(e);
    if (e > 0.f) dz += double(d * e);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    z += __shfl_xor_sync(0xffffffffu, z, o);
    dz += __shfl_xor_sync(0xffffffffu, dz, o);
  }
  if (lane == 0) { S.warp_z[warp] = z; S.warp_dz[warp] = dz; }
  __syncthreads();
  if (tid < C) {
    z = 0.0; dz = 0.0;
    for (int w = 0; w < kSampleWarps; ++w) { z += S.warp_z[w]; dz += S.warp_dz[w]; }
    *cluster.map_shared_rank(&S.z[rank], tid) = z;
    *cluster.map_shared_rank(&S.dz[rank], tid) = dz;
  }
  cluster.sync();
  if (tid == 0) {
    z = 0.0; dz = 0.0;
    for (int c = 0; c < C; ++c) { z += S.z[c]; dz += S.dz[c]; }     // the same order in every CTA
    const double lz = log(z);
    S.row.mx = mx;
    S.row.inv_z = float(1.0 / z);
    S.row.log_z = float(lz);
    S.row.ent = float(lz - dz / z);
    S.bin = kSampleBins;
    S.below = 0ull;
  }
  __syncthreads();
  const TypicalRow r = S.row;

  // ---- mass per interval of s, and the interval in which the running mass reaches tau
  const unsigned long long tau_fixed = __double2ull_ru(double(tau) * double(kMassScale));
  {
    unsigned* h = S.hist[tid & 1];
    int i = tid;
    for (; i + 3 * kSampleThreads < len; i += 4 * kSampleThreads) {
      unsigned m[4];
      int b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float l = logit(i + j * kSampleThreads);
        m[j] = typical_mass(typical_prob(l, r));
        b[j] = typical_bin(typical_shift(l, r));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (m[j]) atomicAdd(&h[b[j]], m[j]);
    }
    for (; i < len; i += kSampleThreads) {
      const float l = logit(i);
      const unsigned m = typical_mass(typical_prob(l, r));
      if (m) atomicAdd(&h[typical_bin(typical_shift(l, r))], m);
    }
  }
  cluster.sync();
  {
    // thread t owns intervals 2t and 2t + 1; every CTA adds up the whole cluster's histograms
    unsigned long long a0 = 0ull, a1 = 0ull;
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint2 v = *reinterpret_cast<const uint2*>(cluster.map_shared_rank(&S.hist[k][2 * tid], c));
        a0 += v.x; a1 += v.y;
      }
    const unsigned long long before = sample_exclusive_scan(a0 + a1, S);
    if (before + a0 + a1 >= tau_fixed && (tid == 0 || before < tau_fixed)) {    // true in one thread, or in none
      const bool low = before + a0 >= tau_fixed;
      S.bin = 2 * tid + (low ? 0 : 1);
      S.below = low ? before : before + a0;
    }
    if (tid == 0) S.count = 0;
  }
  cluster.sync();               // nobody reads a histogram any more: their memory becomes the list
  const int bin = S.bin;

  // ---- draw sums, q_i = keep_i ? p_i^(1/temp) : 0 in index order.  A thread owns `chunk` consecutive
  // tokens (odd: no bank conflicts).  Below the interval a token is kept; inside it is a candidate, noted
  // in the thread's mask and, with its mass, in rank 0's list.
  const float inv_temp = 1.0f / temp;
  const bool tempered = temp != 1.0f;
  auto temper = [&](float q) { return tempered && q > 0.f ? powf(q, inv_temp) : q; };
  const int chunk = ((slice + kSampleThreads - 1) / kSampleThreads) | 1;
  const int i0 = min((long long)tid * chunk, (long long)len), i1 = min((long long)i0 + chunk, (long long)len);
  double mine = 0.0;
  unsigned long long mask = 0ull;
  {
    uint2* cand0 = cluster.map_shared_rank(&S.list.cand[0], 0);
    int* count0 = cluster.map_shared_rank(&S.count, 0);
    auto candidate = [&](int i, float l, float s) {
      if (kInSmem) mask |= 1ull << (i - i0);
      const unsigned m = typical_mass(typical_prob(l, r));
      if (m) {
        const int slot = atomicAdd(count0, 1);
        if (slot < kSampleListCap) cand0[slot] = make_uint2(__float_as_uint(s), m);
      }
    };
    // four tokens at a time without branches but for the rare candidates: some lane keeps each of them
    for (int i = i0; i < i1; i += 4) {
      float l[4], s[4], q[4];
      int b[4];
      bool any = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        l[j] = i + j < i1 ? logit(i + j) : -INFINITY;
        s[j] = typical_shift(l[j], r);
        b[j] = i + j < i1 ? typical_bin(s[j]) : 2 * kSampleBins;
        q[j] = b[j] < bin ? typical_prob(l[j], r) : 0.f;
        any = any || b[j] == bin;
      }
      if (kInSmem) {
#pragma unroll
        for (int j = 0; j < 4; ++j) mine += double(temper(q[j]));
      }
      if (any) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (b[j] == bin) candidate(i + j, l[j], s[j]);
      }
    }
  }
  cluster.sync();

  // ---- the threshold: radix select, a byte of it per pass, over the list (rank 0 alone) or the row (all)
  const bool keep_all = bin == kSampleBins;
  if (!keep_all) {
    const int count = *cluster.map_shared_rank(&S.count, 0);
    const bool listed = count <= kSampleListCap;
    if (!listed || rank == 0) {
      unsigned known = 0u, prefix = 0u;
      unsigned long long below = listed ? S.below : 0ull;
      for (int shift = 24; shift >= 0; shift -= 8) {
        unsigned long long v = 0ull;
        if (listed) {
          if (tid < 256) S.list.bins[tid] = 0u;
          __syncthreads();
          for (int i = tid; i < count; i += kSampleThreads) {
            const uint2 e = S.list.cand[i];
            if ((e.x & known) == prefix) atomicAdd(&S.list.bins[(e.x >> shift) & 255u], e.y);
          }
          __syncthreads();
          if (tid < 256) v = S.list.bins[tid];
        } else {
          cluster.sync();       // the previous pass's totals have been read
          for (int i = tid; i < kSampleHists * kSampleHistStride; i += kSampleThreads) (&S.radix[0][0])[i] = 0u;
          __syncthreads();
          for (int i = tid; i < len; i += kSampleThreads) {
            const float l = logit(i);
            const unsigned key = __float_as_uint(typical_shift(l, r));
            if ((key & known) == prefix) {
              const unsigned m = typical_mass(typical_prob(l, r));
              if (m) atomicAdd(&S.radix[lane & (kSampleHists - 1)][(key >> shift) & 255u], m);
            }
          }
          cluster.sync();
          if (tid < 256)
            for (int c = 0; c < C; ++c)
              for (int k = 0; k < kSampleHists; ++k) v += *cluster.map_shared_rank(&S.radix[k][tid], c);
        }
        const unsigned long long before = below + sample_exclusive_scan(v, S);
        if (before + v >= tau_fixed && (tid == 0 || before < tau_fixed)) {
          S.prefix = prefix | unsigned(tid) << shift;
          S.below = before;
        }
        __syncthreads();
        prefix = S.prefix; below = S.below;
        known |= 255u << shift;
      }
      if (listed) {
        if (tid < C) *cluster.map_shared_rank(&S.thresh, tid) = prefix;
      } else if (tid == 0) {
        S.thresh = prefix;
      }
    }
  }
  cluster.sync();
  const float thresh = keep_all ? 0.f : __uint_as_float(S.thresh);
  auto weight = [&](float l) -> float {
    const float p = typical_prob(l, r);
    return temper((keep_all || typical_shift(l, r) <= thresh) ? p : 0.f);
  };
  if (kInSmem) {
    for (; mask; mask &= mask - 1) mine += double(weight(logit(i0 + __ffsll(mask) - 1)));
  } else {
    for (int i = i0; i < i1; ++i) mine += double(weight(logit(i)));
  }
  if (probs_out)
    for (int i = tid; i < len; i += kSampleThreads) probs_out[size_t(row_id) * n + lo + i] = weight(logit(i));

  // ---- the draw: inverse CDF over the CTAs of the cluster, the threads of one CTA, the tokens of one thread
  S.part[tid] = mine;
  __syncthreads();
  if (warp == 0) {
    // lane l owns the partial sums of threads [16 l, 16 l + 16)
    constexpr int kPer = kSampleThreads / 32;
    double loc = 0.0;
    for (int k = 0; k < kPer; ++k) loc += S.part[lane * kPer + k];
    double inc = loc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    const double cta_total = __shfl_sync(0xffffffffu, inc, 31);
    if (lane < C) *cluster.map_shared_rank(&S.total[rank], lane) = cta_total;
    // u holds rows * history_capacity numbers when a history is kept: replays beyond the capacity reuse the last one
    int step = (hist && hist_count) ? *hist_count : 0;
    const int seen = step;
    if (step >= hist_cap && hist_cap > 0) step = hist_cap - 1;
    const double uniform = double(u[row_id + size_t(rows) * step]);
    cluster.sync();             // the last access to another CTA's memory
    double total = 0.0, base = 0.0;
    for (int c = 0; c < C; ++c) { if (c == rank) base = total; total += S.total[c]; }
    const double target = uniform * total;
    int owner_cta = -1, last_cta = 0;
    double run = 0.0;
    for (int c = 0; c < C; ++c) {
      run += S.total[c];
      if (S.total[c] > 0.0) { last_cta = c; if (owner_cta < 0 && run >= target) owner_cta = c; }
    }
    if (owner_cta < 0) owner_cta = last_cta;   // rounding can leave the target past the end: the last that holds any mass
    if (rank != owner_cta) return;
    inc += base;
    const unsigned hit = __ballot_sync(0xffffffffu, loc > 0.0 && inc >= target);
    const unsigned nonzero = __ballot_sync(0xffffffffu, loc > 0.0);
    const int owner = hit ? __ffs(hit) - 1 : (nonzero ? 31 - __clz(nonzero) : 0);
    // the thread of that group whose tokens hold the target (the same search, in the owner's order)
    run = __shfl_sync(0xffffffffu, inc - loc, owner);
    int c = -1, last = owner * kPer;
    double run_last = run;
    for (int k = 0; k < kPer; ++k) {
      const double v = S.part[owner * kPer + k];
      if (v > 0.0) {
        last = owner * kPer + k; run_last = run;
        if (run + v >= target) { c = last; break; }
      }
      run += v;
    }
    if (c < 0) c = last;
    run = run_last;
    // its tokens, 32 at a time
    const int j0 = min((long long)c * chunk, (long long)len), j1 = min((long long)j0 + chunk, (long long)len);
    int pick = -1, kept = j0;
    for (int b = j0; b < j1 && pick < 0; b += 32) {
      const float q = b + lane < j1 ? weight(logit(b + lane)) : 0.f;
      double sum = double(q);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += t;
      }
      const unsigned at = __ballot_sync(0xffffffffu, q > 0.f && run + sum >= target);
      const unsigned any = __ballot_sync(0xffffffffu, q > 0.f);
      if (at) pick = b + __ffs(at) - 1;
      if (any) kept = b + 31 - __clz(any);
      run += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) {
      const long long id = (long long)lo + (pick < 0 ? kept : pick);
      out[row_id] = id;
      if (hist && hist_count && row_id == 0) {
        if (seen < hist_cap) hist[seen] = id;
        *hist_count = seen + 1;
      }
    }
  } else {
    cluster.sync();
  }
}

// CTAs per row: the fewest whose slices fit two to an SM, and more while the launch still leaves SMs
// without a CTA and a slice has four tokens or more per thread (50277 logits: 19 us for 1 row with 8 CTAs,
// 27 for 37 rows with 4, 30 for 74 rows with 2).
inline int sample_cluster(int rows, int n, int sms) {
  int c = 1;
  while (c < kSampleMaxCluster && (n + c - 1) / c > kSampleMaxSlice) c *= 2;
  while (c < kSampleMaxCluster && (long long)rows * 2 * c <= sms && n / (2 * c) >= 4 * kSampleThreads) c *= 2;
  return c;
}

}  // namespace b200
