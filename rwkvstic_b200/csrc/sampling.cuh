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
// Measured at n = 50277, logits from HBM: 1 row 27 us, 37 rows 38, 74 rows 44, 148 rows 57, 256 rows 102 (two
// waves of clusters), against 68, 72, 72, 74 and 138 with one CTA of 1024 threads per row and eight passes
// through L2.  Sums in fp64 per term and in fixed parts are 9 us of it at 256 rows and 1 at 1 row: parts added up
// in the order of whatever CTAs a row got would save 5 of the 9, but then the last bit of a row's sums would
// depend on the number of rows in the call; terms built from the bits of the fp32 number instead of converted
// cost 4 more.
#pragma once

#include <cooperative_groups.h>

#include <utility>

#include "common.cuh"

namespace b200 {

constexpr int kSampleThreads = 512;
constexpr int kSampleWarps = kSampleThreads / 32;
constexpr int kSampleMaxCluster = 8;
constexpr int kSampleParts = kSampleMaxCluster;    // a row is summed in this many parts, whatever its CTAs
constexpr int kSampleBins = 2 * kSampleThreads;    // intervals of s; the last one also takes everything beyond
constexpr float kSampleBinsPerUnit = 64.f;         // 1/64 nat each
constexpr int kSampleListCap = 1280;               // candidates the list holds
constexpr int kSampleHists = 8;                    // select over the whole row: lane l adds into histogram l % 8
constexpr int kSampleHistStride = 257;             // odd stride: equal bins of different histograms in different banks
constexpr float kMassScale = 2147483648.0f;        // 2^31
// Two CTAs share an SM (its 228 KB hold two slices of this many logits and the scratch), so that one
// computes while the other waits for loads or its cluster.  Shared memory beyond that is not used.
constexpr int kSampleMaxSlice = 25600;
// consecutive tokens per thread and part (odd: no bank conflicts)
__host__ __device__ constexpr int sample_chunk(int part) { return ((part + kSampleThreads - 1) / kSampleThreads) | 1; }
static_assert(sample_chunk(kSampleMaxSlice) <= 64 && 2 * sample_chunk(kSampleMaxSlice / 2) <= 64 && 4 * sample_chunk(kSampleMaxSlice / 4) <= 64 &&
                  8 * sample_chunk(kSampleMaxSlice / 8) <= 64, "a thread's tokens must fit its 64-bit candidate mask");

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
    struct { double a[kSampleParts * kSampleWarps], b[kSampleParts * kSampleWarps]; } sums;   // per part and warp
    double part[kSampleThreads];                             // draw mass per thread
  };
  unsigned long long warp_sum[kSampleWarps];
  float warp_mx[kSampleWarps];
  // one entry per part of the row, or CTA of the cluster, written by the CTA that has it
  double z[kSampleParts], dz[kSampleParts], total[kSampleParts];
  float mx[kSampleMaxCluster];
  TypicalRow row;
  unsigned long long below;     // mass in front of the interval / of the prefix
  unsigned prefix;              // bits of the threshold found so far
  int bin;                      // interval of the threshold; kSampleBins: everything is kept
  int count;                    // candidates (rank 0's)
  unsigned thresh;              // bits of the threshold
  double uniform;               // the number the draw is made with
  int seen;                     // draws in the history before this one
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

// Sums over a warp of N values per lane, each by the butterfly of distances 16, 8, 4, 2, 1, of which a lane follows one
// value only: lane l returns the total of value l / (32 / N).
template <int N>
__device__ __forceinline__ double sample_warp_totals(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int n = N;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n /= 2;
#pragma unroll
      for (int i = 0; i < N / 2; ++i)
        if (i < n) {
          const double keep = lane & o ? v[i + n] : v[i], give = lane & o ? v[i] : v[i + n];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

// logits [rows][ldx]; u: one uniform number in [0,1) per draw, read at u[row + rows * step] where
// step = *history_count when a history is kept and 0 otherwise; out[row] = sampled id;
// probs_out (nullable) [rows][n]: the masked, tempered, unnormalised probabilities the draw used.
// A cluster handles a row of kSampleParts parts of `part` consecutive logits (the last ones may be shorter or
// empty); each of its CTAs takes kParts consecutive ones, its slice.  Sums of fp64 terms are formed
// per part, by all threads of the CTA in the same order, and added in the order of the parts, so a row's
// probabilities and its draw do not depend on how many CTAs it got, and with that on the rows beside it.
// kInSmem: the slice is held in dynamic shared memory (4 bytes a logit); else (rows beyond 8 x
// kSampleMaxSlice logits) every pass reads it from memory.
template <bool kInSmem, int kParts>
__global__ void __launch_bounds__(kSampleThreads, 2)
sample_typical_kernel(const float* __restrict__ x, int n, long long ldx, float temp, float tau,
                      const float* __restrict__ u, long long* __restrict__ out, float* __restrict__ probs_out,
                      long long* __restrict__ hist, int* __restrict__ hist_count, int hist_cap, int part) {
  extern __shared__ float held[];
  __shared__ SampleShared S;
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  auto started = cluster.barrier_arrive();     // met before the first access to another CTA's memory
  const int rank = int(cluster.block_rank()), C = int(cluster.num_blocks());   // kSampleParts / kParts
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row_id = int(blockIdx.x) / C, rows = int(gridDim.x) / C;
  const long long slice = (long long)kParts * part, first = rank * slice;
  const int lo = int(first < n ? first : n), len = int(first + slice < n ? first + slice : n) - lo;
  const float* row = x + size_t(row_id) * ldx + lo;
  auto logit = [&](int i) -> float { return kInSmem ? held[i] : __ldg(row + i); };

  if (tid == 0) {
    // u holds rows * history_capacity numbers when a history is kept: replays beyond the capacity reuse the last one
    int step = (hist && hist_count) ? *hist_count : 0;
    S.seen = step;
    if (step >= hist_cap && hist_cap > 0) step = hist_cap - 1;
    S.uniform = double(u[row_id + size_t(rows) * step]);
  }

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
  cluster.sync();
  mx = S.mx[0];
  for (int c = 1; c < C; ++c) mx = fmaxf(mx, S.mx[c]);

  // ---- Z = sum e^d and sum d e^d (d = l - mx), every term in fp64; entropy = log Z - (sum d e^d) / Z
  // sums of the parts, over the warps in their order (part_total); the lanes that hold a part's sum of their warp write it
  constexpr int kPartLanes = 32 / kParts;
  const int lane_part = lane / kPartLanes;
  const bool lane_writes = lane % kPartLanes == 0;
  auto part_total = [&](const double* w, int p) {
    double t = 0.0;
    for (int i = 0; i < kSampleWarps; ++i) t += w[p * kSampleWarps + i];
    return t;
  };
  double zs[kParts], dzs[kParts];
#pragma unroll
  for (int p = 0; p < kParts; ++p) {
    const int end = min(len, (p + 1) * part);
    double z = 0.0, dz = 0.0;
    int at = p * part + tid;
    for (; at + 3 * kSampleThreads < end; at += 4 * kSampleThreads) {
      float e[4], de[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d = logit(at + j * kSampleThreads) - mx;
        e[j] = expf(d);
        de[j] = e[j] > 0.f ? d * e[j] : 0.f;
      }
      z += (double(e[0]) + double(e[1])) + (double(e[2]) + double(e[3]));
      dz += (double(de[0]) + double(de[1])) + (double(de[2]) + double(de[3]));
    }
    for (; at < end; at += kSampleThreads) {
      const float d = logit(at) - mx, e = expf(d);
      z += double(e);
      if (e > 0.f) dz += double(d * e);
    }
    zs[p] = z; dzs[p] = dz;
  }
  {
    const double z = sample_warp_totals(zs), dz = sample_warp_totals(dzs);
    if (lane_writes) { S.sums.a[lane_part * kSampleWarps + warp] = z; S.sums.b[lane_part * kSampleWarps + warp] = dz; }
  }
  __syncthreads();
  if (tid < kSampleParts) {                  // thread: a part of this CTA and a CTA to tell
    const int p = tid / C, to = tid - p * C;
    *cluster.map_shared_rank(&S.z[rank * kParts + p], to) = part_total(S.sums.a, p);
    *cluster.map_shared_rank(&S.dz[rank * kParts + p], to) = part_total(S.sums.b, p);
  }
  cluster.sync();
  for (int i = tid; i < 2 * kSampleBins; i += kSampleThreads) (&S.hist[0][0])[i] = 0u;
  if (tid == 0) {
    double z = 0.0, dz = 0.0;
    for (int p = 0; p < kSampleParts; ++p) { z += S.z[p]; dz += S.dz[p]; }
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
  // tokens of every part.  Below the interval a token is kept; inside it is a candidate, noted in the
  // thread's mask and, with its mass, in rank 0's list.
  const float inv_temp = 1.0f / temp;
  const bool tempered = temp != 1.0f;
  auto temper = [&](float q) { return tempered && q > 0.f ? powf(q, inv_temp) : q; };
  const int chunk = sample_chunk(part);
  auto part_begin = [&](int p) { return int(min((long long)p * part + (long long)tid * chunk, (long long)min(len, (p + 1) * part))); };
  auto part_end = [&](int p) { return int(min((long long)p * part + (long long)(tid + 1) * chunk, (long long)min(len, (p + 1) * part))); };
  double mine[kParts];                       // per part
  unsigned long long mask = 0ull;            // bit p * chunk + j: token j of the thread's in part p is a candidate
  {
    uint2* cand0 = cluster.map_shared_rank(&S.list.cand[0], 0);
    int* count0 = cluster.map_shared_rank(&S.count, 0);
    auto candidate = [&](int bit, float l, float s) {
      if (kInSmem) mask |= 1ull << bit;
      const unsigned m = typical_mass(typical_prob(l, r));
      if (m) {
        const int slot = atomicAdd(count0, 1);
        if (slot < kSampleListCap) cand0[slot] = make_uint2(__float_as_uint(s), m);
      }
    };
#pragma unroll 1
    for (int p = 0; p < kParts; ++p) {
      const int i0 = part_begin(p), i1 = part_end(p);
      double sum = 0.0;
      int i = i0;
      // four tokens at a time without branches but for the rare candidates: some lane keeps each of them
      for (; i + 3 < i1; i += 4) {
        float l[4], s[4], q[4];
        int b[4];
        bool any = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          l[j] = logit(i + j);
          s[j] = typical_shift(l[j], r);
          b[j] = typical_bin(s[j]);
          q[j] = b[j] < bin ? typical_prob(l[j], r) : 0.f;
          any = any || b[j] == bin;
        }
        if (kInSmem) {
#pragma unroll
          for (int j = 0; j < 4; ++j) sum += double(temper(q[j]));
        }
        if (any) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (b[j] == bin) candidate(p * chunk + i + j - i0, l[j], s[j]);
        }
      }
      for (; i < i1; ++i) {
        const float l = logit(i), s = typical_shift(l, r);
        const int b = typical_bin(s);
        if (kInSmem && b < bin) sum += double(temper(typical_prob(l, r)));
        if (b == bin) candidate(p * chunk + i - i0, l, s);
      }
      mine[p] = sum;
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
  if (probs_out)
    for (int i = tid; i < len; i += kSampleThreads) probs_out[size_t(row_id) * n + lo + i] = weight(logit(i));

  // ---- the draw: inverse CDF over the parts, the threads of one part, the tokens of one thread
#pragma unroll
  for (int p = 0; p < kParts; ++p) {
    double sum = mine[p];
    const int i0 = part_begin(p);
    if (kInSmem) {
      for (unsigned long long some = mask >> (p * chunk) & ((1ull << chunk) - 1); some; some &= some - 1)
        sum += double(weight(logit(i0 + __ffsll(some) - 1)));
    } else {
      const int i1 = part_end(p);
      for (int i = i0; i < i1; ++i) sum += double(weight(logit(i)));
    }
    mine[p] = sum;
  }
  {
    double v[kParts];
#pragma unroll
    for (int p = 0; p < kParts; ++p) v[p] = mine[p];
    const double sum = sample_warp_totals(v);
    if (lane_writes) S.sums.a[lane_part * kSampleWarps + warp] = sum;
  }
  __syncthreads();
  if (tid < kSampleParts) {
    const int p = tid / C, to = tid - p * C;
    *cluster.map_shared_rank(&S.total[rank * kParts + p], to) = part_total(S.sums.a, p);
  }
  cluster.sync();               // the last access to another CTA's memory
  double total = 0.0;
  for (int p = 0; p < kSampleParts; ++p) total += S.total[p];
  const double target = S.uniform * total;
  int owner_part = -1, last_part = 0;
  double base = 0.0, before = 0.0, last_before = 0.0;      // mass in front of the owner's part
  for (int p = 0; p < kSampleParts; ++p) {
    const double v = S.total[p];
    if (v > 0.0) {
      last_part = p; last_before = before;
      if (owner_part < 0 && before + v >= target) { owner_part = p; base = before; }
    }
    before += v;
  }
  // rounding can leave the target past the end: the last that holds any mass
  if (owner_part < 0) { owner_part = last_part; base = last_before; }
  if (owner_part / kParts != rank) return;
  const int mine_part = owner_part - rank * kParts;
  S.part[tid] = mine[mine_part];
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
    inc += base;
    const unsigned hit = __ballot_sync(0xffffffffu, loc > 0.0 && inc >= target);
    const unsigned nonzero = __ballot_sync(0xffffffffu, loc > 0.0);
    const int owner = hit ? __ffs(hit) - 1 : (nonzero ? 31 - __clz(nonzero) : 0);
    // the thread of that group whose tokens hold the target (the same search, in the owner's order)
    double run = __shfl_sync(0xffffffffu, inc - loc, owner);
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
    const int end = min(len, (mine_part + 1) * part);
    const int j0 = int(min((long long)mine_part * part + (long long)c * chunk, (long long)end)), j1 = min(j0 + chunk, end);
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
        if (S.seen < hist_cap) hist[S.seen] = id;
        *hist_count = S.seen + 1;      // every CTA has read it: it did before the first cluster barrier
      }
    }
  }
}

inline int sample_part(int n) { return n / kSampleParts + (n % kSampleParts != 0); }

// CTAs per row: the fewest whose slices fit two to an SM, and more while the launch still leaves SMs
// without a CTA and a slice has four tokens or more per thread (50277 logits: 27 us for 1 row with 8 CTAs,
// 38 for 37 rows with 4, 44 for 74 rows with 2).
inline int sample_cluster(int rows, int n, int sms) {
  int c = 1;
  while (c < kSampleMaxCluster && sample_part(n) > c * (kSampleMaxSlice / kSampleParts)) c *= 2;
  while (c < kSampleMaxCluster && (long long)rows * 2 * c <= sms && n / (2 * c) >= 4 * kSampleThreads) c *= 2;
  return c;
}

}  // namespace b200
