// Many activation rows through UNQUANTISED bf16 / fp16 matrices on the 5th-generation tensor cores:
// the reference's TORCH-mode matvec for T > 1 rows (agnostic/backends/torch.py:162-164,
// `x.to(W.dtype).matmul(W).to(x.dtype)`; AgnosticRWKV applies every matrix to all rows of a sequence
// at once, agnosticRwkv.py:123-169).
//
//   out[r][n] = epilogue( round_T( sum_k x_T[r][k] * W[n][k] ) )        fp32 accumulation
//
//   A = 128 weight rows    x 128 bytes of K (64 elements; a TMA box of W[N][K], 128-byte swizzle)
//   B = Rt activation rows x 128 bytes of K (a TMA box of the rows already rounded to T; Rt = 16..240)
//   D = 128 lanes x activation rows fp32 columns in tensor memory, two buffers (columns 0 and 256): the
//       epilogue of a tile runs under the MMAs of the next.
//
// Same skeleton and the same two forms as tile_gemm.cuh: a CTA on 128 weight rows x Rt activation rows, or
// a pair of CTAs (tcgen05.mma.cta_group::2) on 256 x 2*Rt, up to 256 x 256.  Persistent CTAs, an operand
// ring that runs on across tiles, warp 0 = TMA producer, warp 1 = MMA issuer (kind::f16), warps 4..19 =
// epilogue through tcgen05.ld; no digit planes, no per-row scalars.  With few rows and therefore few
// tiles K is cut into slices (work item = tile x slice): a slice parks its fp32 partial sums in a scratch
// buffer and draws a ticket; the CTA that draws a tile's last ticket adds the slices IN SLICE ORDER (so
// the result does not depend on which CTA finished when) and runs the epilogue.  Nobody waits for anybody.
// Every wait is bounded; on expiry the CTA sets a status bit, drains its copies and still frees its
// tensor memory.
#pragma once

#include "dense_step.cuh"
#include "tile_gemm.cuh"

namespace b200 {

constexpr int kDgRowsSingle = 240, kDgRowsPair = 128;            // activation rows a CTA holds of a tile, at most
constexpr int kDgRingBytes = 186 * 1024;
constexpr int kDgMaxStages = 8;                                  // barriers: full 0..7, empty 8..15
constexpr int kDgSmem = kGemmOffRing + kDgRingBytes;
constexpr int kDgSplitMaxItems = 640;                            // tiles x slices of a split launch (its tickets)
constexpr int kDgSplitMaxRows = 1024;                            // calls of up to this many rows may split K
constexpr long long kDgSplitMaxCells = 640ll * 64;               // tiles x slices x tile height that the scratch holds
constexpr size_t kDgSplitBytes = size_t(kDgSplitMaxCells) * 128 * 4;   // 21 MB of partial sums

struct DGemmSeg {
  CUtensorMap wmap;     // W as bytes [K*2/128][N][128 B], box [kc][128][128], 128-byte swizzle
  CUtensorMap xmap;     // rows as bytes [K*2/128][Rpad][128 B], box [kc][Rt][128], 128-byte swizzle
  void* out;            // [R][ldo] of float, or of T when out_t is set
  const float* res;     // [R][ldres] added last, or null
  const float* gate;    // [R][ldgate] multiplies the product first, or null
  long long ldo, ldres, ldgate;
  int N, act, out_t;
};

struct DGemmParams {
  DGemmSeg seg[kMaxSeg];
  int nseg, ksteps, R;  // ksteps = K * 2 / 128
  int pair;             // tiles of a CTA pair: 256 weight rows x 2*Rt activation rows; else 128 x Rt
  int Rt, row_tiles;
  int tiles_seg[kMaxSeg];
  int ntiles;
  int is_bf16;
  int kc;               // K steps of 128 bytes per stage, 1 or 2
  int stages;           // ring depth: as many stages of stage_bytes as fit the ring, at most 8
  int stage_bytes;      // kc * (128 + Rt) * 128, a multiple of 1024
  int ksplit;           // K slices per tile (1: none; > 1 only with single-CTA tiles; divides ksteps)
  float* sk_part;       // [ntiles][ksplit][Rt][128] partial sums of the slices
  unsigned* sk_count;   // [ntiles] tickets, zero between launches
  int* status;
};

// Instruction descriptor of kind::f16: D fp32, A and B of the same 16-bit type, both K-major, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int M, int N, int is_bf16) {
  return (1u << 4) | (uint32_t(is_bf16 ? 1 : 0) << 7) | (uint32_t(is_bf16 ? 1 : 0) << 10) | (uint32_t(N >> 3) << 17) |
         (uint32_t(M >> 4) << 24);
}

template <bool kPair>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (kPair)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ float round16(float v, int is_bf16) {
  return is_bf16 ? __bfloat162float(__float2bfloat16_rn(v)) : __half2float(__float2half_rn(v));
}
__device__ __forceinline__ unsigned short bits16(float v, int is_bf16) {
  return is_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}

struct DGemmTile { int seg, n0, row0; };
__device__ __forceinline__ DGemmTile dgemm_tile(const DGemmParams& P, int t) {
  int s = 0;
  while (s < P.nseg - 1 && t >= P.tiles_seg[s]) { t -= P.tiles_seg[s]; ++s; }
  const int wt = t / P.row_tiles;                       // tiles that share a weight tile are consecutive
  return {s, wt * (P.pair ? 256 : 128), (t - wt * P.row_tiles) * (P.pair ? 2 * P.Rt : P.Rt)};
}

// kPair: two CTAs of a cluster work on one tile with tcgen05.mma.cta_group::2 (see tile_gemm.cuh).
template <bool kPair>
__global__ void __launch_bounds__(kGemmThreads, 1) dense_tile_gemm_kernel(const __grid_constant__ DGemmParams P) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int Rt = P.Rt, S = P.ksplit;
  const int nk = P.ksteps / S;            // K steps of one work item
  const int nitems_all = P.ntiles * S;
  const int NS = P.stages, KC = P.kc;
  const int rank = kPair ? int(cluster_ctarank()) : 0;                    // which half of the tile this CTA holds
  const int first_item = kPair ? int(blockIdx.x >> 1) : int(blockIdx.x), item_stride = kPair ? int(gridDim.x >> 1) : int(gridDim.x);
  const uint32_t a_chunk = 128u * 128u, b_chunk = uint32_t(Rt) * 128u;
  const uint32_t a_bytes = uint32_t(KC) * a_chunk;      // a stage: KC weight chunks, then KC row chunks

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + 8);
  const uint32_t acc_full0 = smem_u32(bars + 16), acc_empty0 = smem_u32(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 256);
  volatile int* issued_ptr = reinterpret_cast<volatile int*>(smem + 260);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 264);
  unsigned char* ring = smem + kGemmOffRing;

  if (tid == 0) {
    for (int i = 0; i < kDgMaxStages; ++i) { mbar_init(full0 + 8 * i, 1); mbar_init(empty0 + 8 * i, 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(acc_full0 + 8 * i, 1); mbar_init(acc_empty0 + 8 * i, (kPair ? 2 : 1) * kGemmEpiWarps); }
    *abort_flag = 0;
    *issued_ptr = 0;
    fence_mbar_init();
  }
  if (warp == 2) tmem_alloc<kPair>(smem_u32(tmem_slot));
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_sync();             // the partner's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  griddep_launch_dependents();

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    const uint32_t ring0 = smem_u32(ring), stage_bytes = uint32_t(P.stage_bytes);
    const uint32_t full_at = kPair ? leader_addr(full0) : full0;
    const uint32_t tx_bytes = kPair ? 2u * stage_bytes : stage_bytes;
    struct Cursor { int it, k, left; DGemmTile T; };      // work item, K step of the copy, K steps left of the item
    auto start = [&](Cursor& c) {
      if (c.it < nitems_all) { c.T = dgemm_tile(P, c.it / S); c.k = S == 1 ? 0 : (c.it % S) * nk; c.left = nk; }
    };
    auto next = [&](Cursor& c) {
      c.k += KC;
      if ((c.left -= KC) <= 0) { c.it += item_stride; start(c); }
    };
    Cursor ld;
    ld.it = first_item;
    start(ld);
    // Weights are constants: the first ring of them is requested before the launch dependency resolves.
    int early = 0;
    for (; early < NS && ld.it < nitems_all; ++early, next(ld)) {
      if (elect_one()) {
        if (rank == 0) mbar_arrive_expect_tx(full0 + 8 * early, tx_bytes);
        tma_operand_3d<kPair>(ring0 + uint32_t(early) * stage_bytes, &P.seg[ld.T.seg].wmap, 0, ld.T.n0 + rank * 128, ld.k, full_at + 8 * early);
      }
    }
    *issued_ptr = early;
    griddep_wait();   // the activation rows come from the kernel in front of this launch
    int issued = 0, slot = 0;
    uint32_t phase = 0;
    ld.it = first_item;
    for (start(ld); ld.it < nitems_all; next(ld)) {
      const DGemmSeg& Sg = P.seg[ld.T.seg];
      const uint32_t bar = full_at + 8 * slot, dst = ring0 + uint32_t(slot) * stage_bytes;
      if (issued >= early) {
        if (!warp_wait(empty0 + 8 * slot, phase ^ 1u, abort_flag, P.status, B200RWKV_STATUS_WAIT_EMPTY)) break;
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(full0 + 8 * slot, tx_bytes);
          tma_operand_3d<kPair>(dst, &Sg.wmap, 0, ld.T.n0 + rank * 128, ld.k, bar);   // rows past N are zero-filled
        }
      }
      if (elect_one()) tma_operand_3d<kPair>(dst + a_bytes, &Sg.xmap, 0, ld.T.row0 + rank * Rt, ld.k, bar);   // rows past the buffer too
      ++issued;
      if (++slot == NS) { slot = 0; phase ^= 1u; }
    }
    *issued_ptr = issued;
    if (kPair && ld.it >= nitems_all) ring_drain(empty0, slot, phase, NS, abort_flag, P.status, B200RWKV_STATUS_WAIT_EMPTY);
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer (the even CTA's, for both)
    if (rank == 0) {
      const uint32_t idesc = umma_idesc_f16(kPair ? 256 : 128, kPair ? 2 * Rt : Rt, P.is_bf16);
      const uint32_t ring0 = smem_u32(ring), stage_bytes = uint32_t(P.stage_bytes);
      bool ok = true;
      int iter = 0, slot = 0;
      uint32_t phase = 0;
      for (int it = first_item; it < nitems_all && ok; it += item_stride, ++iter) {
        const int buf = iter & 1, use = iter >> 1;
        const uint32_t tacc = tmem + uint32_t(buf * kGemmAcc1Col);
        if (!warp_wait(acc_empty0 + 8 * buf, uint32_t(use & 1) ^ 1u, abort_flag, P.status, B200RWKV_STATUS_WAIT_EMPTY)) break;
        uint32_t acc = 0u;    // the first MMA of a tile overwrites the accumulator
        for (int k0 = 0; k0 < nk; k0 += KC) {
          if (!warp_wait(full0 + 8 * slot, phase, abort_flag, P.status, B200RWKV_STATUS_WAIT_FULL)) { ok = false; break; }
          if (elect_one()) {
            tc_fence_after();
            const uint32_t a = ring0 + uint32_t(slot) * stage_bytes;
            const uint64_t ad = umma_desc(a), bd = umma_desc(a + a_bytes);
            auto chunk = [&](uint64_t a64, uint64_t b64, uint32_t first) {    // straight-line issue, see tile_gemm.cuh
#pragma unroll
              for (int k = 0; k < 4; ++k)   // 16 elements = 32 bytes of K per instruction: +2 in the descriptors' 16-byte units
                umma_f16<kPair>(tacc, a64 + uint64_t(2 * k), b64 + uint64_t(2 * k), idesc, k == 0 ? first : 1u);
            };
            chunk(ad, bd, acc);
            if (KC > 1 && nk - k0 > 1) chunk(ad + uint64_t(a_chunk >> 4), bd + uint64_t(b_chunk >> 4), 1u);
            umma_commit<kPair>(empty0 + 8 * slot);
            if (k0 + KC >= nk) umma_commit<kPair>(acc_full0 + 8 * buf);
          }
          acc = 1u;
          if (++slot == NS) { slot = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------------- epilogue: four warps per TMEM lane quadrant
    const int q = warp & 3, eg = (warp - 4) >> 2;
    constexpr int EG = kGemmEpiWarps / 4, CH = kGemmChunk;
    const int et = tid - 128;
    const int rows_tile = kPair ? 2 * Rt : Rt, nchunks = rows_tile / CH;   // TMEM column = row of the tile
    volatile int* last_flag = reinterpret_cast<volatile int*>(smem + 272);   // K split: this CTA drew a tile's last ticket
    griddep_wait();
    bool ok = true;
    int iter = 0;
    for (int it = first_item; it < nitems_all && ok; it += item_stride, ++iter) {
      const int tile = it / S, slice = it - tile * S;
      const DGemmTile T = dgemm_tile(P, tile);
      const DGemmSeg& Sg = P.seg[T.seg];
      const int n0 = T.n0 + rank * 128, row0 = T.row0;
      const int buf = iter & 1, use = iter >> 1;
      const uint32_t acc_empty = acc_empty0 + 8 * buf;
      auto drained = [&]() {
        tc_fence_before();
        if (lane == 0) {
          if (kPair) mbar_arrive_leader(acc_empty); else mbar_arrive(acc_empty);
        }
      };
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(acc_full0 + 8 * buf, uint32_t(use & 1), abort_flag));
      if (!ok) {
        if (lane == 0 && P.status) atomicOr(P.status, B200RWKV_STATUS_WAIT_FULL);
        break;
      }
      tc_fence_after();
      int last_item = -1;     // this warp's last item that really reads TMEM
      for (int item = eg; item < nchunks; item += EG)
        if (row0 + item * CH < P.R) last_item = item;
      if (last_item < 0) drained();
      const int rlast = P.R - 1;
      // rounding to the matrices' type, activation, gate, residual and store for 8 rows of one output column
      auto finish = [&](const float (&acc)[CH], int j0) {
        const int n = n0 + q * 32 + lane;
        const bool nvalid = n < Sg.N;
        const int nc = nvalid ? n : Sg.N - 1;
        float yv[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) yv[j] = round16(acc[j], P.is_bf16);
        if (Sg.act == ACT_RELUSQ) {
#pragma unroll
          for (int j = 0; j < CH; ++j) { const float t = fmaxf(yv[j], 0.f); yv[j] = __fmul_rn(t, t); }
        } else if (Sg.act == ACT_SIGMOID) {
#pragma unroll
          for (int j = 0; j < CH; ++j) yv[j] = sigmoidf_(yv[j]);
        }
        if (Sg.gate) {
          float gv[CH];
#pragma unroll
          for (int j = 0; j < CH; ++j) { const int r = min(row0 + j0 + j, rlast); gv[j] = __ldcg(Sg.gate + size_t(r) * Sg.ldgate + nc); }
#pragma unroll
          for (int j = 0; j < CH; ++j) yv[j] = __fmul_rn(yv[j], gv[j]);
        }
        if (Sg.res) {
          float rv[CH];
#pragma unroll
          for (int j = 0; j < CH; ++j) { const int r = min(row0 + j0 + j, rlast); rv[j] = __ldcg(Sg.res + size_t(r) * Sg.ldres + nc); }
#pragma unroll
          for (int j = 0; j < CH; ++j) yv[j] = __fadd_rn(rv[j], yv[j]);
        }
#pragma unroll
        for (int j = 0; j < CH; ++j) {
          const int r = row0 + j0 + j;
          if (r <= rlast && nvalid) {
            if (Sg.out_t) static_cast<unsigned short*>(Sg.out)[size_t(r) * Sg.ldo + n] = bits16(yv[j], P.is_bf16);
            else static_cast<float*>(Sg.out)[size_t(r) * Sg.ldo + n] = yv[j];
          }
        }
      };
      // K split: this slice's partial sums go to [tile][slice][row][128 weight rows] (single-CTA tiles only)
      float* sk = S > 1 ? P.sk_part + (size_t(tile) * S + slice) * Rt * 128 + q * 32 + lane : nullptr;
#pragma unroll 1
      for (int item = eg; item < nchunks; item += EG) {
        const int j0 = item * CH;
        if (row0 + j0 >= P.R) continue;   // warp-uniform
        int d[CH];
        tmem_ld8(tmem + (uint32_t(q * 32) << 16) + uint32_t(buf * kGemmAcc1Col + j0), d);
        tmem_ld_wait();
        if (item == last_item) drained();
        float acc[CH];
#pragma unroll
        for (int j = 0; j < CH; ++j) acc[j] = __int_as_float(d[j]);
        if (S == 1) {
          finish(acc, j0);
        } else {
#pragma unroll
          for (int j = 0; j < CH; ++j) sk[size_t(j0 + j) * 128] = acc[j];   // 32 lanes = 128 consecutive bytes per store
        }
      }
      if (S > 1) {
        __threadfence();                                   // this thread's partial sums are visible before the ticket
        named_bar_sync(1, kGemmEpiWarps * 32);
        if (et == 0) {
          const unsigned ticket = atomicAdd(P.sk_count + tile, 1u);
          __threadfence();                                 // and the other slices' sums before the reads below
          *last_flag = ticket == unsigned(S - 1) ? 1 : 0;
        }
        named_bar_sync(1, kGemmEpiWarps * 32);
        if (*last_flag) {
          const float* all = P.sk_part + size_t(tile) * S * Rt * 128 + q * 32 + lane;
#pragma unroll 1
          for (int item = eg; item < nchunks; item += EG) {
            const int j0 = item * CH;
            if (row0 + j0 >= P.R) continue;
            float acc[CH];
#pragma unroll
            for (int j = 0; j < CH; ++j) acc[j] = 0.f;
            for (int sl = 0; sl < S; ++sl) {               // slice order: the sum does not depend on who came last
#pragma unroll
              for (int j = 0; j < CH; ++j) acc[j] += __ldcg(all + (size_t(sl) * Rt + j0 + j) * 128);
            }
            finish(acc, j0);
          }
          if (et == 0) P.sk_count[tile] = 0u;              // leave the tickets zero for the next launch
        }
        named_bar_sync(1, kGemmEpiWarps * 32);             // last_flag is rewritten by the next work item
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && rank == 0 && *abort_flag) {      // copies that may still be in flight into shared memory
    const int issued = *issued_ptr;
    const unsigned long long t0 = globaltimer_ns();
    for (int i = issued > NS ? issued - NS : 0; i < issued; ++i) {
      const uint32_t bar = full0 + 8 * (i % NS), parity = uint32_t(i / NS) & 1u;
      while (!mbar_try_wait(bar, parity) && globaltimer_ns() - t0 < kWaitLimitNs / 10) {
      }
    }
  }
  if (kPair) cluster_sync();             // nothing of the pair's work touches either CTA any more
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc<kPair>(tmem);
  }
}

// ---- rows in front of the GEMMs ---------------------------------------------------------------------
// A CTA takes rows_per_cta consecutive activation rows (row r: stream r / Tn, position r % Tn): layer
// norm of x[r]; the token-shift carry is the stream's state row for its first row and the layer norm of
// x[r - 1] otherwise (agnosticRwkv.py:125-127: roll + push); out[m][r] = T(lerp(carry, ln, mix[m])).
// Walking consecutive rows, the CTA already holds the layer norm of x[r - 1] from its previous turn and
// only rebuilds it for the first row it takes; a row's arithmetic is the same either way.  The layer norm
// of every stream's last row is the stream's next carry: with one row per stream the CTA that read the
// state row writes it back itself; with more rows it is parked in a scratch row (sibling CTAs still read
// the old one), and the next preparation launch commits it.
// With `last_only` the CTA of stream b normalises x[(b+1)*Tn - 1] and writes out[0][b] = T(ln): the
// rows the head is applied to (agnosticRwkv.py:184).
// The form is rows_stream_kernel's (tile_gemm.cuh): a thread owns the same 4*G inputs of every row, their
// parameters are fetched before the launch dependency resolves and held in the thread's own slots of shared
// memory, the row stays in registers and the next one is requested ahead.
// Against a CTA of 256 threads that re-read the parameters from L2 for every row and kept rows in shared
// memory, us per call: fp16 1.5B 48 streams 1763 -> 1608, bf16 3B 2 x 701 tokens 10896 -> 10730 (with the
// copies of the carries, two a block, that the commit replaces).
struct DRowsPrepParams {
  const float* x;            // [R][D]
  const float *ln_w, *ln_b;
  const float* carry;        // state row of stream 0; stream b at carry + b * carry_stride
  long long carry_stride;
  float* carry_out;          // stream b's new carry goes to carry_out + b * carry_out_stride
  long long carry_out_stride;
  const float* mix[3];
  unsigned short* out[3];    // T [Rpad][D]
  int nmix, D, Tn, last_only, is_bf16;
  int R, rows_per_cta;       // rows of the call (streams with last_only); consecutive rows per CTA
  int hold_ln;               // ln_w and ln_b fit shared memory beside the mix vectors
  // A carry that the previous preparation launch parked: stream b's D floats go from commit_src + b * D to
  // commit_dst + b * carry_stride, by the CTA of the stream's last row.  Null: none.
  const float* commit_src;
  float* commit_dst;
};

template <int G, int NT_MAX, int MIN_CTAS>
__global__ void __launch_bounds__(NT_MAX, MIN_CTAS)
dense_rows_prep_kernel(const __grid_constant__ DRowsPrepParams P) {
  extern __shared__ __align__(128) unsigned char rp_smem[];
  float* red = reinterpret_cast<float*>(rp_smem);
  const int tid = threadIdx.x, NT = blockDim.x, nwarps = NT >> 5, D = P.D, NG = P.D >> 2;
  float4* mix = reinterpret_cast<float4*>(rp_smem + kStreamRedBytes);       // [nmix][NG], then ln_w, ln_b
  float4* ln = mix + P.nmix * NG;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  griddep_launch_dependents();
#pragma unroll
  for (int i = 0; i < G; ++i) {
    const int g = tid + i * NT;
    if (g < NG) {
      if (P.hold_ln) {
        const float4 w = ld_param_v4(reinterpret_cast<const float4*>(P.ln_w) + g), b = ld_param_v4(reinterpret_cast<const float4*>(P.ln_b) + g);
        ln[g] = w; ln[NG + g] = b;
      }
#pragma unroll
      for (int m = 0; m < 3; ++m)
        if (m < P.nmix) mix[m * NG + g] = ld_param_v4(reinterpret_cast<const float4*>(P.mix[m]) + g);
    }
  }
  const float4* lnw = P.hold_ln ? ln : reinterpret_cast<const float4*>(P.ln_w);
  const float4* lnb = P.hold_ln ? ln + NG : reinterpret_cast<const float4*>(P.ln_b);
  griddep_wait();

  auto load = [&](const float* row, float4 (&v)[G]) {
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int g = tid + i * NT;
      v[i] = g < NG ? __ldcg(reinterpret_cast<const float4*>(row) + g) : zero4;
    }
  };
  int phase = 0;
  auto norm = [&](float4 (&a)[G]) {      // torch.py:102-110
    float s[1] = {0.f};
#pragma unroll
    for (int i = 0; i < G; ++i) s[0] += (a[i].x + a[i].y) + (a[i].z + a[i].w);      // groups past the end hold zeros
    stream_reduce<1, 0>(s, red, phase, nwarps);
    const float mean = s[0] / float(D);
    float q[1] = {0.f};
#pragma unroll
    for (int i = 0; i < G; ++i) {
      a[i].x -= mean; a[i].y -= mean; a[i].z -= mean; a[i].w -= mean;
      if (tid + i * NT < NG) {
        q[0] = fmaf(a[i].x, a[i].x, q[0]); q[0] = fmaf(a[i].y, a[i].y, q[0]);
        q[0] = fmaf(a[i].z, a[i].z, q[0]); q[0] = fmaf(a[i].w, a[i].w, q[0]);
      }
    }
    stream_reduce<1, 0>(q, red, phase, nwarps);
    const float sd = sqrtf(q[0] / float(D) + 1e-5f);
    // n / sd by the correctly rounded reciprocal and the exact remainder of the first quotient (Markstein,
    // 1990): the division's own result without its range checks (every mantissa of sd against 160 numerators on
    // a CPU: no difference; fp16 1.5B 48 streams 1613 us, 1648 with the division).  Below 2^-100 the remainder of n
    // loses bits and the quotient may be one off in its last place; a quotient by infinity stays 0.
    const float rcp = 1.0f / sd, neg = sd < INFINITY ? -sd : 0.f;
    auto quot = [&](float n) { const float q0 = n * rcp; return fmaf(fmaf(neg, q0, n), rcp, q0); };
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int g = tid + i * NT;
      if (g < NG) {
        const float4 w = lnw[g], b = lnb[g];
        a[i] = make_float4(w.x * quot(a[i].x) + b.x, w.y * quot(a[i].y) + b.y, w.z * quot(a[i].z) + b.z, w.w * quot(a[i].w) + b.w);
      }
    }
  };
  const bool shift = !P.last_only && P.nmix > 0;
  const int first = blockIdx.x * P.rows_per_cta, end = min(first + P.rows_per_cta, P.R);
  auto source = [&](int idx) { return P.x + (P.last_only ? size_t(idx + 1) * P.Tn - 1 : size_t(idx)) * D; };
  float4 x[G], nx[G], pv[G];
  load(source(first), x);
  int stream = P.last_only ? first : first / P.Tn, pos = P.last_only ? P.Tn - 1 : first - stream * P.Tn;
  if (shift && pos > 0) {                       // this CTA begins inside a stream
    load(source(first - 1), pv);
    norm(pv);
  }
  for (int idx = first; idx < end; ++idx) {
    if (idx + 1 < end) load(source(idx + 1), nx);
    const bool last = pos == P.Tn - 1;
    if (P.commit_src && last) {
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int g = tid + i * NT;
        if (g < NG)
          reinterpret_cast<float4*>(P.commit_dst + size_t(stream) * P.carry_stride)[g] = __ldcg(reinterpret_cast<const float4*>(P.commit_src + size_t(stream) * D) + g);
      }
    }
    if (shift && pos == 0) load(P.carry + size_t(stream) * P.carry_stride, pv);
    norm(x);
    if (shift && last && P.carry_out) {
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const int g = tid + i * NT;
        if (g < NG) reinterpret_cast<float4*>(P.carry_out + size_t(stream) * P.carry_out_stride)[g] = x[i];
      }
    }
    const size_t orow = size_t(idx) * D;
    auto store4 = [&](unsigned short* out, int g, float a, float b, float c, float d) {
      ushort4 o;
      o.x = bits16(a, P.is_bf16); o.y = bits16(b, P.is_bf16); o.z = bits16(c, P.is_bf16); o.w = bits16(d, P.is_bf16);
      reinterpret_cast<ushort4*>(out + orow)[g] = o;
    };
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int g = tid + i * NT;
      if (g < NG) {
        if (!shift) store4(P.out[0], g, x[i].x, x[i].y, x[i].z, x[i].w);
        else {
#pragma unroll
          for (int m = 0; m < 3; ++m)
            if (m < P.nmix) {
              const float4 w = mix[m * NG + g];
              store4(P.out[m], g, lerp_like_torch(pv[i].x, x[i].x, w.x), lerp_like_torch(pv[i].y, x[i].y, w.y),
                     lerp_like_torch(pv[i].z, x[i].z, w.z), lerp_like_torch(pv[i].w, x[i].w, w.w));
            }
        }
      }
      pv[i] = x[i];
      x[i] = nx[i];
    }
    if (P.last_only) ++stream;
    else if (++pos == P.Tn) { pos = 0; ++stream; }
  }
}

// Shape of a launch: the fewest groups per thread that 1024 threads allow; resident CTAs by registers (64 a
// thread, 40 with one group and at most 768 threads) and shared memory.
struct DRowsShape { int G, threads, slots_per_sm, hold_ln; size_t smem; };
inline DRowsShape dense_rows_prep_shape(int D, int nmix) {
  DRowsShape sh;
  const int NG = D / 4;
  sh.G = (NG + 1023) / 1024;
  sh.threads = ((NG + sh.G - 1) / sh.G + 31) / 32 * 32;
  const size_t limit = size_t(224) * 1024;
  sh.hold_ln = size_t(kStreamRedBytes) + size_t(nmix + 2) * D * 4 <= limit ? 1 : 0;
  sh.smem = size_t(kStreamRedBytes) + size_t(nmix + (sh.hold_ln ? 2 : 0)) * D * 4;
  const int by_regs = sh.G == 1 && sh.threads <= 768 ? 1536 / sh.threads : 1024 / sh.threads, by_smem = int(limit / (sh.smem + 1024));
  sh.slots_per_sm = by_regs < 1 || by_smem < 1 ? 1 : by_regs < by_smem ? by_regs : by_smem;
  return sh;
}

}  // namespace b200
