// Mixed-precision rotate + average, pipelined (4 pols, complex<float>): the hot kernel.
//
// Work comes from a table of items; an item is one resident integration and a
// contiguous range of directions (the single-integration call is one item; a
// batched call has one item per integration chunk).  An item is cut into units
// = (group of TPB 32-baseline tiles, group of (NC/TPB)*DPW directions,
// timestep slab); units of all items are numbered consecutively, so uneven
// chunks share one launch.  The host assigns units to the persistent blocks
// longest first, each to the least-loaded block, and passes the result as an
// order table (block b visits order[b], order[b + grid], ... up to a -1), so
// blocks finish together even when unit sizes differ by 100x.
//
// A unit is a sequence of chunks = (timestep, CH channels).  The visibility
// tensor of an item is viewed as a 2-D array [channel][row*8 floats]; a chunk
// is one TMA box of 256 floats (32 baselines x 4 pols x complex) by CH
// channels per tile, loaded with cp.async.bulk.tensor from the item's tensor
// map into a shared-memory stage, completing on the stage's "full" mbarrier.
// Boxes past the last row or channel are zero-filled by the TMA unit; rows of
// a partial tile that belong to the next timestep are loaded but not used.
// Every warp releases a stage through its "empty" mbarrier; lane 0 of warp 0
// then refills it with the chunk one ring length ahead.  (A separate producer
// warp would make 9 warps, 3 on one SM sub-partition, and cap registers at
// 168.)  All waits are bounded and report a device error instead of hanging.
//
// Per (row, direction) the phase turns(c) = A + c*B is formed once per
// timestep in double-float arithmetic (~1e-12 turns) as 32-bit fixed-point
// fractions of a turn: no FP64 instructions in this kernel (GB300 runs them
// at ~1/70 of the FP32 rate).  A block of 16 channels is a polynomial in the
// channel step's phasor w, evaluated by Horner's rule from its last channel:
//     sum_k V[c0 + k] z w^k = z (V[c0] + w (V[c0+1] + w (...))),
// so a channel costs one complex multiply-add per pol and no phasor recurrence
// of its own; z, table-accurate (twiddle_turns), enters once per block.  w has a
// relative error eta of ~1e-7, w^k one of k eta; z is taken at the block's middle
// channel and divided by w^8 as rounded, which leaves (k - 8) eta: half the drift
// of a recurrence from the block's start (~5e-7; it reaches the cal phases only
// through baselines that the reference-antenna pass does not cover, with weight
// ~1/S).  Sums: FP32 over 64 channels, folded into Kahan pairs.
//
// What bounds it: HBM and the issue of FFMA2, 8 per (row, channel, direction) at
// 2 to 2.6 issue slots each; a recurrence of the phasors took 4 scalar FMAs more.
// 32-chunk batched workload, 8 directions a chunk (52.3 GB): 9.6 ms, 5.4 TB/s, in
// a call of 10.97 -> 10.50 ms.
//
// Shared-memory reads: lane i reads its 32 bytes as two 16-byte halves; lanes
// with bit 2 set read the upper half first so that each quarter-warp covers
// all 32 banks (conflict-free).  Those lanes hold pols (2,3,0,1) in register
// slots (0,1,2,3) and swap back when writing out.
#pragma once

#include "leap_common.cuh"

namespace leapgb {

// One item of a pipelined launch (device memory; the tensor map needs 128-byte alignment).
struct alignas(128) PipeItem {
  CUtensorMap map;        // [channel][rows*8 floats], box 256 x CH
  const float* uvw_f;     // [rows][6] split UVWs
  double2* out;           // nslab == 1: avg + dir0*4*nbl; else this item's [nslab][ndir][4][nbl] partials
  int64_t rows;
  int32_t T, C, t_per_slab, nslab;
  int32_t tgroups, dgroups, dir0, ndir;
  int32_t unit_begin, pad_[3];
};

struct PipeParams {
  const PipeItem* items;
  const int32_t* order;    // [nslots]: block b visits units order[b], order[b + grid], ... until -1
  int32_t nslots;
  int32_t nitems, units;
  int32_t nbl;
  const float* dirk;       // [ndir_total][12]
  const float2* twiddle;   // [kTwiddleSize]
  int* err;
};

constexpr int kPipeMaxItems = 128;
// Channels summed in FP32 before a Kahan fold.  At 32 the fold was ~6% of the FMA-pipe work;
// FP32 partial sums over 64 channels (~2e-8 of the sum of |terms|) stay far below the phasor
// drift between reseeds (~1e-6).  Measured: 32-chunk batched workload 11.47 -> 11.10 ms per
// call (cal-phase difference from the FP64 form over 256 directions: median 1.1e-7 -> 1.2e-7
// rad, maximum 4.7e-6 -> 4.2e-6); 128-antenna 1-tile call 2.58 -> 2.49 ms.
constexpr int kPipeFold = 64;
constexpr int kPipeItemBytes = 32 * 4 * 8;  // one channel of one tile: 32 baselines x 4 pols x complex<float>

// Channels per chunk (one Horner block) and ring depth: 1 tile x 16 channels = 16 KB stages, 4 deep; 2 tiles =
// 32 KB, 4 deep; 4 tiles = 64 KB stages, 3 deep (192 KB of the 227 KB of shared memory).
template <int TPB> struct PipeShape;
template <> struct PipeShape<1> { static constexpr int CH = 16, STAGES = 4; };
template <> struct PipeShape<2> { static constexpr int CH = 16, STAGES = 4; };
template <> struct PipeShape<4> { static constexpr int CH = 16, STAGES = 3; };

template <int TPB>
__host__ __device__ constexpr int pipe_stage_bytes() { return TPB * PipeShape<TPB>::CH * kPipeItemBytes; }

template <int TPB>
__host__ __device__ constexpr int pipe_smem_bytes() {
  return PipeShape<TPB>::STAGES * (pipe_stage_bytes<TPB>() + 16) + kTwiddleSize * 8 + kPipeMaxItems * 4;
}

// Position in a block's chunk sequence: slot s of the order table, unit u = order[s].
struct ChunkCursor {
  int s, u, item, t, cb;
  int t_hi;
};

// Item holding unit u: the last item whose first unit is <= u (binary search; units of
// an item are consecutive and items are in unit order).
__device__ __forceinline__ int find_item(const int* unit_begin, int nitems, int u) {
  int lo = 0, hi = nitems - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (unit_begin[mid] <= u) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int slot_unit(const PipeParams& p, int s) { return s < p.nslots ? __ldg(p.order + s) : -1; }

__device__ __forceinline__ void cursor_unit(ChunkCursor& k, const PipeParams& p, const int* unit_begin) {
  k.item = find_item(unit_begin, p.nitems, k.u);
  const PipeItem& it = p.items[k.item];
  const int slab = (k.u - it.unit_begin) % it.nslab;
  k.t = slab * it.t_per_slab;
  k.t_hi = min(it.T, k.t + it.t_per_slab);
  k.cb = 0;
}

template <int TPB>
__device__ __forceinline__ void cursor_next(ChunkCursor& k, const PipeParams& p, const int* unit_begin) {
  k.cb += PipeShape<TPB>::CH;
  if (k.cb < p.items[k.item].C) return;
  k.cb = 0;
  if (++k.t < k.t_hi) return;
  k.s += gridDim.x;
  k.u = slot_unit(p, k.s);
  if (k.u >= 0) cursor_unit(k, p, unit_begin);
}

template <int TPB>
__device__ __forceinline__ void issue_chunk(const ChunkCursor& k, const PipeParams& p, unsigned char* stage_mem,
                                           uint64_t* full, int st) {
  constexpr int CH = PipeShape<TPB>::CH;
  const PipeItem& it = p.items[k.item];
  const int l = k.u - it.unit_begin;
  const int tg = l / (it.dgroups * it.nslab);
  mbar_arrive_expect_tx(&full[st], pipe_stage_bytes<TPB>());
  unsigned char* dst = stage_mem + st * pipe_stage_bytes<TPB>();
#pragma unroll
  for (int ts = 0; ts < TPB; ++ts)
    tma_load_2d(dst + ts * CH * kPipeItemBytes, &it.map, (k.t * p.nbl + (tg * TPB + ts) * 32) * 8, k.cb, &full[st]);
}

// Paired FP32 FMAs (FFMA2) run two directions in their halves: a direction pair's phasors and sums are natural
// register pairs, and a visibility component enters as the addend (v, v).  (With two pols in the halves the
// step's phasor has to be doubled instead, in moves of every direction: 13.2 against 10.5 ms for the 32-chunk
// batched workload; scalar FMAs: 12.5 ms.)
struct PipeStep {  // the phasor w = r + i of a direction pair, and -i
  float2 r, i, ni;
};

__device__ __forceinline__ PipeStep pipe_step(float2 r, float2 i) { return PipeStep{r, i, make_float2(-i.x, -i.y)}; }

// p = p * w + v for the 4 pols of one channel and the first N direction pairs: 16 paired FMAs each.  FIRST: p = v.
template <int N, bool FIRST, int DP>
__device__ __forceinline__ void pipe_horner(const unsigned char* src, int h, float2 (&pr)[DP][4], float2 (&pi)[DP][4],
                                            const PipeStep (&w)[DP]) {
  const float4 x0 = *reinterpret_cast<const float4*>(src + 16 * h);
  const float4 x1 = *reinterpret_cast<const float4*>(src + 16 * (1 - h));
  const float vr[4] = {x0.x, x0.z, x1.x, x1.z}, vi[4] = {x0.y, x0.w, x1.y, x1.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 a = make_float2(vr[q], vr[q]), b = make_float2(vi[q], vi[q]);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (FIRST) {
        pr[j][q] = a;
        pi[j][q] = b;
      } else {
        const float2 nr = __ffma2_rn(pi[j][q], w[j].ni, __ffma2_rn(pr[j][q], w[j].r, a));
        pi[j][q] = __ffma2_rn(pr[j][q], w[j].i, __ffma2_rn(pi[j][q], w[j].r, b));
        pr[j][q] = nr;
      }
    }
  }
}

// Kahan fold of x into (s, -c): both halves as the scalar sequence y = x - c, t = s + y, c = (t - s) - y, s = t
// (a - b as fma(b, -1, a), one rounding).
__device__ __forceinline__ void pipe_fold(float2& s, float2& nc, float2 x) {
  const float2 neg = make_float2(-1.f, -1.f);
  const float2 y = __fadd2_rn(x, nc);
  const float2 t = __fadd2_rn(s, y);
  nc = __fadd2_rn(y, __ffma2_rn(t, neg, s));
  s = t;
}

// acc += z sum_k V[k] w^k over the n channels of a chunk, for the first N direction pairs.  z: the phasor of the
// chunk's middle channel, at turns a + b (in 2^-32 of a turn) per direction; (ur, ui) = 1 / w^8.
template <int N, int CH, int DP>
__device__ __forceinline__ void pipe_chunk(const unsigned char* src, int h, int n, const PipeStep (&w)[DP],
                                           const float2 (&ur)[DP], const float2 (&ui)[DP], const uint32_t (&turns)[2 * DP],
                                           const float2* tab, float2 (&acc_r)[DP][4], float2 (&acc_i)[DP][4]) {
  float2 pr[DP][4], pi[DP][4];
  pipe_horner<N, true>(src + (n - 1) * kPipeItemBytes, h, pr, pi, w);
  if (n == CH) {
#pragma unroll
    for (int k = CH - 2; k >= 0; --k) pipe_horner<N, false>(src + k * kPipeItemBytes, h, pr, pi, w);
  } else {
    for (int k = n - 2; k >= 0; --k) pipe_horner<N, false>(src + k * kPipeItemBytes, h, pr, pi, w);
  }
#pragma unroll
  for (int j = 0; j < N; ++j) {
    float2 zr, zi;
    twiddle_turns(turns[2 * j], tab, zr.x, zi.x);
    twiddle_turns(turns[2 * j + 1], tab, zr.y, zi.y);
    const float2 nzi = make_float2(-zi.x, -zi.y);
    const PipeStep x = pipe_step(__ffma2_rn(nzi, ui[j], __fmul2_rn(zr, ur[j])), __ffma2_rn(zi, ur[j], __fmul2_rn(zr, ui[j])));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc_r[j][q] = __ffma2_rn(pi[j][q], x.ni, __ffma2_rn(pr[j][q], x.r, acc_r[j][q]));
      acc_i[j][q] = __ffma2_rn(pr[j][q], x.i, __ffma2_rn(pi[j][q], x.r, acc_i[j][q]));
    }
  }
}

// 1 / w^8 as rounded: conj(w^8) (2 - |w^8|^2), |w^8| = 1 to ~1e-6.
__device__ __forceinline__ void pipe_unturn8(float wr, float wi, float& ur, float& ui) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float r = fmaf(wr, wr, -wi * wi);
    wi = 2.f * wr * wi;
    wr = r;
  }
  const float f = 2.f - fmaf(wr, wr, wi * wi);
  ur = wr * f;
  ui = -wi * f;
}

template <int NC, int DPW, int TPB>
__global__ void __launch_bounds__(NC * 32, 1) rotate_average_mixed_pipe(const PipeParams p) {
  constexpr int CH = PipeShape<TPB>::CH;
  constexpr int NS = PipeShape<TPB>::STAGES;
  constexpr int WPT = NC / TPB;  // warps (direction groups of DPW) per tile
  constexpr int DP = DPW / 2;    // direction pairs per warp
  static_assert(NC % TPB == 0 && DPW % 4 == 0, "warps divide among tiles, directions into pairs and halves");
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* stage_mem = smem;
  float2* tab = reinterpret_cast<float2*>(smem + NS * pipe_stage_bytes<TPB>());
  uint64_t* full = reinterpret_cast<uint64_t*>(tab + kTwiddleSize);
  uint64_t* empty = full + NS;
  int* unit_begin = reinterpret_cast<int*>(empty + NS);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool producer = threadIdx.x == 0;
  for (int i = threadIdx.x; i < kTwiddleSize; i += blockDim.x) tab[i] = __ldg(p.twiddle + i);
  for (int i = threadIdx.x; i < p.nitems; i += blockDim.x) unit_begin[i] = p.items[i].unit_begin;
  __syncthreads();
  ChunkCursor pc{};  // producer cursor, NS chunks ahead of the consumers
  uint32_t issued = 0;
  if (producer) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], NC);
    }
    fence_mbar_init();
    pc.s = blockIdx.x;
    pc.u = slot_unit(p, pc.s);
    pc.item = 0;
    if (pc.u >= 0) cursor_unit(pc, p, unit_begin);
    for (; issued < NS && pc.u >= 0; ++issued) {
      issue_chunk<TPB>(pc, p, stage_mem, full, issued);
      cursor_next<TPB>(pc, p, unit_begin);
    }
  }
  __syncthreads();

  const int h = (lane >> 2) & 1;  // read order of the two 16-byte halves
  // The warps of a tile take its direction groups in an order that differs from tile to tile, so that the groups
  // past the last direction idle on different schedulers (a warp's scheduler is its number modulo 4).
  const int ts = warp / WPT;
  const int dsub = WPT >= 4 ? (warp + 2 * ts) % WPT : (warp + ts / 2) % WPT;
  uint32_t it = 0;
  bool ok = true;
  int item = 0;
  for (int sl = blockIdx.x; ok; sl += gridDim.x) {
    const int u = slot_unit(p, sl);
    if (u < 0) break;
    item = find_item(unit_begin, p.nitems, u);
    const PipeItem& I = p.items[item];
    const int l = u - I.unit_begin;
    const int tg = l / (I.dgroups * I.nslab);
    const int dg = (l / I.nslab) % I.dgroups;
    const int slab = l % I.nslab;
    const int t_lo = slab * I.t_per_slab, t_hi = min(I.T, t_lo + I.t_per_slab);
    const int C = I.C;
    const int b = (tg * TPB + ts) * 32 + lane;
    const bool valid = b < p.nbl;
    const int jd0 = (dg * WPT + dsub) * DPW;  // first direction of this warp within the item
    // A tile wholly past the last baseline (the last tile group when nbl is not a multiple
    // of 32 * TPB) only takes part in the stage hand-over.
    const bool active = jd0 < I.ndir && (tg * TPB + ts) * 32 < p.nbl;
    // The second half of the warp's directions is past the last one.  Not looked at with 4 tiles, whose items fill
    // their 8 directions as a rule: the second path costs the full one 1.5% there.
    const bool half = TPB < 4 && jd0 + DPW / 2 >= I.ndir;

    // Kahan pairs (sum, negated compensation) of direction pair j, pol slot q.
    float2 sr[DP][4], si[DP][4], cr[DP][4], ci[DP][4];
#pragma unroll
    for (int j = 0; j < DP; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) sr[j][q] = si[j][q] = cr[j][q] = ci[j][q] = make_float2(0.f, 0.f);

    // The row's split UVWs are loaded one timestep ahead, so that the set-up of a
    // timestep does not wait on a global load.
    float xn[6];
#pragma unroll
    for (int i = 0; i < 6; ++i)
      xn[i] = active ? __ldg(I.uvw_f + 6 * (static_cast<int64_t>(t_lo) * p.nbl + (valid ? b : 0)) + i) : 0.f;
    for (int t = t_lo; t < t_hi && ok; ++t) {
      uint32_t pa[DPW], pb[DPW];
      PipeStep w[DP];
      float2 ur[DP], ui[DP];  // 1 / w^8
      if (active) {
        // turns(c) = A + c*B, A = -(l*u + m*v + (n-1)*w)*f0/c, B likewise with df.
        float x[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) x[i] = xn[i];
        if (t + 1 < t_hi) {
          const int64_t rn = static_cast<int64_t>(t + 1) * p.nbl + (valid ? b : 0);
#pragma unroll
          for (int i = 0; i < 6; ++i) xn[i] = __ldg(I.uvw_f + 6 * rn + i);
        }
#pragma unroll
        for (int j = 0; j < DPW; ++j) {
          const int d = I.dir0 + min(jd0 + j, I.ndir - 1);
          float ka[6], kb[6];
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            ka[i] = __ldg(p.dirk + 12 * d + i);
            kb[i] = __ldg(p.dirk + 12 * d + 6 + i);
          }
          pa[j] = df_dot3_turns_u32(ka, x);
          pb[j] = df_dot3_turns_u32(kb, x);
        }
#pragma unroll
        for (int j = 0; j < DP; ++j) {
          float2 r, i;
          twiddle_turns(pb[2 * j], tab, r.x, i.x);
          twiddle_turns(pb[2 * j + 1], tab, r.y, i.y);
          w[j] = pipe_step(r, i);
          pipe_unturn8(r.x, i.x, ur[j].x, ui[j].x);
          pipe_unturn8(r.y, i.y, ur[j].y, ui[j].y);
        }
      }
      // FP32 partial sums of up to kPipeFold channels, then a Kahan fold.
      float2 acc_r[DP][4], acc_i[DP][4];
#pragma unroll
      for (int j = 0; j < DP; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc_r[j][q] = acc_i[j][q] = make_float2(0.f, 0.f);
      for (int cb = 0; cb < C; cb += CH, ++it) {
        const int n = min(CH, C - cb);
        const int st = it % NS;
        if (!mbar_wait_bounded(&full[st], (it / NS) & 1)) {
          atomicOr(p.err, kDevErrTimeout);
          ok = false;
          break;
        }
        if (active) {
          const unsigned char* src = stage_mem + st * pipe_stage_bytes<TPB>() + ts * CH * kPipeItemBytes + lane * 32;
          uint32_t turns[DPW];
#pragma unroll
          for (int j = 0; j < DPW; ++j) turns[j] = pa[j] + static_cast<uint32_t>(cb + 8) * pb[j];
          if (half)
            pipe_chunk<DP / 2, CH>(src, h, n, w, ur, ui, turns, tab, acc_r, acc_i);
          else
            pipe_chunk<DP, CH>(src, h, n, w, ur, ui, turns, tab, acc_r, acc_i);
          if ((cb + CH) % kPipeFold == 0 || cb + CH >= C) {
#pragma unroll
            for (int j = 0; j < DP; ++j)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                pipe_fold(sr[j][q], cr[j][q], acc_r[j][q]);
                pipe_fold(si[j][q], ci[j][q], acc_i[j][q]);
                acc_r[j][q] = acc_i[j][q] = make_float2(0.f, 0.f);
              }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[st]);
        if (producer && pc.u >= 0) {
          // Refill this stage with the chunk NS ahead once every warp released it.
          if (!mbar_wait_bounded(&empty[st], (it / NS) & 1)) {
            atomicOr(p.err, kDevErrTimeout);
            ok = false;
          } else {
            issue_chunk<TPB>(pc, p, stage_mem, full, st);
            cursor_next<TPB>(pc, p, unit_begin);
            ++issued;
          }
        }
        __syncwarp();
      }
    }
    if (ok && active && valid) {
      // nslab == 1: out points at avg[dir0]; else at this item's partials.
      double2* out = I.out + static_cast<int64_t>(I.nslab > 1 ? slab : 0) * I.ndir * 4 * p.nbl;
#pragma unroll
      for (int j = 0; j < DPW; ++j) {
        const int jd = jd0 + j;
        if (jd < I.ndir) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int pol = q ^ (2 * h), i = j >> 1;
            const bool odd = j & 1;
            out[(static_cast<int64_t>(jd) * 4 + pol) * p.nbl + b] =
                make_double2(static_cast<double>(odd ? sr[i][q].y : sr[i][q].x) + static_cast<double>(odd ? cr[i][q].y : cr[i][q].x),
                             static_cast<double>(odd ? si[i][q].y : si[i][q].x) + static_cast<double>(odd ? ci[i][q].y : ci[i][q].x));
          }
        }
      }
    }
  }
  if (producer) {
    // Do not leave while copies issued by this block may still land in shared memory.
    for (uint32_t j = (issued > NS ? issued - NS : 0); j < issued; ++j)
      if (!mbar_wait_bounded(&full[j % NS], (j / NS) & 1)) atomicOr(p.err, kDevErrTimeout);
  }
}

// Per-item slab reduction: out[begin + i] = sum over the item's slabs of partial[s][i],
// i < ndir * per_dir (per_dir = pols * nbl for avgData, nI1 for the reference rows).
struct ReduceItem {
  const double2* partial;  // [nslab][ndir][per_dir]
  int64_t begin;           // first flat output index of the item
  int32_t nslab, ndir;
};

static __global__ void reduce_item_slabs(const ReduceItem* __restrict__ items, int nitems, int per_dir,
                                         double2* __restrict__ avg) {
  const ReduceItem r = items[blockIdx.y];
  const int64_t n = static_cast<int64_t>(r.ndir) * per_dir;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    // Four partial sums (slabs s = j mod 4), added in a fixed order: four loads in flight.
    double re[4] = {0.0, 0.0, 0.0, 0.0}, im[4] = {0.0, 0.0, 0.0, 0.0};
    int s = 0;
    for (; s + 4 <= r.nslab; s += 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 v = r.partial[static_cast<int64_t>(s + j) * n + i];
        re[j] += v.x;
        im[j] += v.y;
      }
    }
    for (int j = 0; s < r.nslab; ++s, ++j) {
      const double2 v = r.partial[static_cast<int64_t>(s) * n + i];
      re[j] += v.x;
      im[j] += v.y;
    }
    avg[r.begin + i] = make_double2((re[0] + re[1]) + (re[2] + re[3]), (im[0] + im[1]) + (im[2] + im[3]));
  }
}

}  // namespace leapgb
