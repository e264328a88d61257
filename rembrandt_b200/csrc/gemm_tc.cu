// Persistent, warp-specialised tcgen05 GEMM / implicit-GEMM convolution for sm_100a.
//
//   warp 0      A producer: TMA loads (tiled, im2col, or whole image rows) of the A operand, one lane per box
//   warp 1      MMA issuer (one elected lane issues): tcgen05.mma, fp32 accumulators in TMEM; owns TMEM alloc/dealloc
//   warps 2..9  epilogue: tcgen05.ld -> bias / ReLU / mask -> swizzled smem -> TMA store (bf16), or fp32 TMA
//               store / reduce-add (split-K, gradient accumulation). Two warps share each TMEM lane quarter and
//               alternate column slabs: with one warp per scheduler the epilogue is bound by instruction latency.
//   warp 10     B producer: TMA loads of the B operand, one lane per box (or the resident panel, once)
//
// What was measured on this kernel and shaped it:
//   * one thread's TMA loads go one after the other while loads issued by different threads overlap, so the loads of a
//     stage are spread over two producer warps and over lanes;
//   * what a producer or the MMA issuer does per k-block in instructions counts as much as what it asks for: with the
//     coordinates divided out of the k-block's number, and the MMAs issued from a branch of one lane, each took ~1200
//     cycles per k-block whatever the size of its boxes; walking taps and pixels by additions and issuing from converged
//     code took 10-30 % off every layer (weight gradient of 128 -> 128 on 256 x 19 x 19: 51 -> 36 us);
//   * im2col-mode loads cost up to ~2.8 ns per pixel row per SM and tiled loads 1-1.7 ns per row, independent of the
//     row's bytes: rows are kept 128 bytes wide (64 channels) even when that means a half-empty, zero-filled chunk;
//   * the L2 delivers 10-12 TB/s into the shared memories, which is what binds layers of 64 and more channels; tiles are
//     as wide as the layer allows (N <= 256);
//   * a work item may cover two 128-row sub-tiles (mt = 2; up to four in flat mode) that share one B stage and use an
//     accumulator each; when
//     the whole B panel fits in shared memory and the CTA only ever needs that one panel, it is loaded once per CTA
//     and stays resident (b_resident); split-K (fp32 reduce-add epilogue) spreads long reductions over all SMs;
//   * which of these a forward / data-grad launch uses is decided by timing the candidates the first time a shape
//     is seen (the launches are idempotent), see `launch`.
//   * stride-1 convolutions can load whole input rows once for all filter taps (A_FLAT_K, the comment at flat_geom):
//     what binds the im2col form is that every tap brings the same pixels into shared memory again.
// With two accumulator sets in TMEM the epilogue of work item i overlaps the main loop of item i+1; a
// 256 x 256 item needs all 512 columns and runs without that overlap.
//
// Every mbarrier wait is bounded; on a timeout the CTA raises an abort flag, records
// RB_STATUS_MBAR_TIMEOUT in the status word, drains its outstanding TMA copies (bounded),
// frees TMEM and returns. No TMA load here uses cluster multicast.
#include "gemm_tc.cuh"
#include "ptx.cuh"
#include "common.cuh"
#include "launch.cuh"
#include <ctype.h>
#include <stdlib.h>
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

namespace rb {

constexpr int BM = 128;
constexpr int GEMM_THREADS = 352;   // A-producer warp, MMA warp, 8 epilogue warps, B-producer warp
// Register budget: 352 threads x 144 registers leave 14.8 K of the SM's 64 K registers free, which is what one
// 128-thread block of the exchange kernels (80 registers per thread, 10 K) needs to run beside a resident CTA of this
// kernel. Above 155 registers those blocks no longer fit and the gradient exchange stops overlapping the backward
// pass (measured: 2.29 instead of 1.98 ms per AlexNet step on 2 GPUs); tests/test_register_budget.py keeps watch.
// Registers are handed out to whole warps, four warps at a time: the CTA's 11 warps take 12 x 32 x 144 = 55296, and
// the 10240 left are exactly the four warps x 80 registers of an exchange block. Hence the hard cap.
constexpr int GEMM_MAX_REGS = 144;
constexpr int PRODUCER_B_WARP = 10;
constexpr int EPI_WARPS = 8;
constexpr int MAX_STAGES = 8;
constexpr int MAX_A_STAGES = 3;   // flat mode
constexpr int TILE_SMEM_BYTES = 192 * 1024;   // B panel (if resident) + stage ring
// The lean instantiation (weight-gradients that run beside other kernels of the step): what it leaves of an SM's shared memory
// holds a block of the normalisation kernels (17 KB), and its registers leave room for one (20 - 26 K of 34.8 K). With 96 KB
// a 256-column tile has two stages instead of three: Go network's step at 256 boards 1567 us, with 144 KB 1529, with all of
// the shared memory (nothing beside it) 1650.
constexpr int LEAN_TILE_BYTES = 144 * 1024;
constexpr int LEAN_MAX_REGS = 80;
constexpr int STAGING_BYTES = 32 * 1024;      // epilogue: 8 warps x one slab of 32 rows x 128 B
constexpr int GEMM_SMEM_BYTES = TILE_SMEM_BYTES + STAGING_BYTES + 1024 /*align*/ + 512 /*barriers*/;
constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;  // 2 s

struct SharedCtl {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t b_full;
  uint64_t a_full[MAX_A_STAGES];    // flat mode: the A ring has its own barriers
  uint64_t a_empty[MAX_A_STAGES];
  uint64_t mask_bar[EPI_WARPS];
  uint32_t tmem_base;
  volatile int abort_flag;
};

__device__ __forceinline__ bool ctl_wait(SharedCtl* ctl, uint64_t* bar, uint32_t parity, unsigned int* status) {
  if (mbar_try_wait(bar, parity)) return true;    // the common case costs one instruction, no read of the abort flag
  if (ctl->abort_flag) return false;
  if (mbar_wait_bounded(bar, parity, WAIT_LIMIT_NS)) return true;
  ctl->abort_flag = 1;
  if (status) atomicOr(status, RB_STATUS_MBAR_TIMEOUT);
  return false;
}

// The same for a whole converged warp: the result is the same in every lane. Where lane 0 alone has seen the phase, the
// barrier at the end orders the other lanes (one of which may be the elected one that issues) after what it acquired; the
// shuffle alone orders no memory.
__device__ __forceinline__ bool ctl_wait_warp(SharedCtl* ctl, uint64_t* bar, uint32_t parity, unsigned int* status) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  int ok = 0;
  if ((threadIdx.x & 31) == 0) ok = ctl_wait(ctl, bar, parity, status) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();
  return ok != 0;
}

// Role profile (built only with -DRB_GEMM_PROFILE, see `python -m rembrandt_b200._build --profile`): cycles that the
// roles of ONE CTA (block 3) spend waiting, summed over launches -- [0] A producer on a free stage, [1] B producer on
// a free stage, [2] MMA issuer on a filled stage, [3] MMA issuer on a drained accumulator, [4] the CTA's whole run,
// and for ONE epilogue warp (warp 2) in the bf16 epilogue: [5] waiting for a filled accumulator, [6] proxy fence +
// issue of the TMA store of a slab, [7] a slab's way from TMEM through registers into shared memory.
// A role that hardly waits is the one the others wait for. `rb_gemm_role_profile` reads and clears the counters.
#ifdef RB_GEMM_PROFILE
__device__ unsigned long long g_role_cycles[8];
__device__ __forceinline__ bool ctl_wait_role(SharedCtl* ctl, uint64_t* bar, uint32_t parity, unsigned int* status,
                                              int slot) {
  const long long t0 = clock64();
  const bool r = ctl_wait(ctl, bar, parity, status);
  if (blockIdx.x == 3) atomicAdd(&g_role_cycles[slot], (unsigned long long)(clock64() - t0));
  return r;
}
__device__ __forceinline__ bool ctl_wait_warp_role(SharedCtl* ctl, uint64_t* bar, uint32_t parity, unsigned int* status,
                                                   int slot) {
  const long long t0 = clock64();
  const bool r = ctl_wait_warp(ctl, bar, parity, status);
  if (blockIdx.x == 3 && (threadIdx.x & 31) == 0) atomicAdd(&g_role_cycles[slot], (unsigned long long)(clock64() - t0));
  return r;
}
#else
__device__ __forceinline__ bool ctl_wait_warp_role(SharedCtl* ctl, uint64_t* bar, uint32_t parity, unsigned int* status,
                                                   int) {
  return ctl_wait_warp(ctl, bar, parity, status);
}
__device__ __forceinline__ bool ctl_wait_role(SharedCtl* ctl, uint64_t* bar, uint32_t parity, unsigned int* status,
                                              int) {
  return ctl_wait(ctl, bar, parity, status);
}
#endif

#ifdef RB_GEMM_PROFILE
#define RB_PROF_T0(cond) const long long prof_t0_ = (cond) ? clock64() : 0
#define RB_PROF_ADD(cond, slot) \
  if ((cond) && blockIdx.x == 3 && (threadIdx.x & 31) == 0) \
    atomicAdd(&g_role_cycles[slot], (unsigned long long)(clock64() - prof_t0_))
#else
#define RB_PROF_T0(cond)
#define RB_PROF_ADD(cond, slot)
#endif

// base pixel (w, h, n) of output position `pix` of a P x Q grid for the im2col tensor maps
__device__ __forceinline__ void pixel_coords(int P, int Q, int stride, int lower_h, int lower_w, int pix, int& w, int& h, int& n) {
  const int pq = P * Q;
  n = pix / pq;
  const int r2 = pix - n * pq;
  const int pp = r2 / Q;
  const int qq = r2 - pp * Q;
  w = qq * stride + lower_w;
  h = pp * stride + lower_h;
}

// One unit of a CTA's work list: tile (tm, tn) over k-blocks [kb0, kb1). `tail` >= 0 marks a part of a cut item of
// the last wave (index among the cut items); its sums go to the fp32 workspace instead of D.
struct WorkItem {
  int tm, tn, kb0, kb1, tail, phase;
};
template <bool PHASES, class Params>
__device__ __forceinline__ WorkItem decode_work(const Params& p, int work, int m_items, int direct, int kb_per_split) {
  WorkItem w;
  int rem;
  w.phase = 0;
  if constexpr (PHASES) {
    for (int k = 1; k < p.phases; ++k) w.phase = work >= p.ph[k].work0 ? k : w.phase;
    const GemmPhase& ph = p.ph[w.phase];
    rem = work - ph.work0;
    m_items = ph.m_items;
    w.kb0 = 0;
    w.kb1 = ph.num_kb;
    w.tail = -1;
  } else if (p.tail_items > 0 && work >= direct) {
    const int w2 = work - direct;
    const int part = w2 / p.tail_items;
    w.tail = w2 - part * p.tail_items;
    rem = direct + w.tail;
    const int kbs = (p.num_kb + p.tail_split - 1) / p.tail_split;
    w.kb0 = part * kbs;
    w.kb1 = min(p.num_kb, w.kb0 + kbs);
  } else {
    const int per = m_items * p.n_tiles;
    const int z = work / per;
    rem = work - z * per;
    w.kb0 = z * kb_per_split;
    w.kb1 = min(p.num_kb, w.kb0 + kb_per_split);
    w.tail = -1;
  }
  w.tn = rem / m_items;
  w.tm = rem - w.tn * m_items;
  return w;
}

// Flat mode: row of D (and mask, addend) that position `f` belongs to, -1 for the zero columns and rows between images.
__device__ __forceinline__ long long flat_row(const GemmTcParams& p, int f) {
  const int g = f / p.fl_pitch, q = f - g * p.fl_pitch;
  const int n = g / p.fl_hp, i = g - n * p.fl_hp;
  if (q >= p.cv_Q || i >= p.cv_P || n * p.cv_P * p.cv_Q >= p.M) return -1;
  if (p.sc_stride)
    return ((long long)n * p.sc_H + i * p.sc_stride + p.sc_a) * p.sc_W + q * p.sc_stride + p.sc_b;
  return ((long long)n * p.cv_P + i) * p.cv_Q + q;
}

__device__ __forceinline__ int dgrad_tap(const GemmTcParams& p, int tap) {
  if (p.dg_dv == 0) return tap;
  const int u = tap / p.cv_S;
  return p.dg_base + u * p.dg_du + (tap - u * p.cv_S) * p.dg_dv;
}

// One k-block of a resident B panel (weights: never a weight-grad's operand), by one thread.
__device__ __forceinline__ void load_b(const GemmTcParams& p, uint8_t* sb, uint64_t* bar, int kb, int n0) {
  const int b_split = p.b_split > 0 ? p.b_split : 1;
  const int b_rows = p.bn_load / b_split;
  if (p.b_mode == B_TILED_K) {
    for (int q = 0; q < b_split; ++q)
      tma_load_2d(sb + q * b_rows * p.bk * 2, &p.tm_b, bar, kb * p.bk, n0 + q * b_rows);
  } else if (p.b_mode == B_TILED_K3) {
    const int tap = kb / p.cv_cchunks;
    const int cc = kb - tap * p.cv_cchunks;
    for (int q = 0; q < b_split; ++q)
      tma_load_3d(sb + q * b_rows * p.bk * 2, &p.tm_b, bar, cc * p.bk, dgrad_tap(p, tap), n0 + q * b_rows);
  } else if (p.b_mode == B_DGRAD_MN) {
    const int tap = kb / p.cv_cchunks;
    const int cc = kb - tap * p.cv_cchunks;
    for (int j = 0; j < p.bn_load / 64; ++j)
      tma_load_3d(sb + j * p.bk * 128, &p.tm_b, bar, n0 + 64 * j, dgrad_tap(p, tap), cc * p.bk);
  } else if (p.b_mode == B_TILED_MN) {
    for (int j = 0; j < p.bn_load / 64; ++j) tma_load_2d(sb + j * p.bk * 128, &p.tm_b, bar, n0 + 64 * j, kb * p.bk);
  }
}

// The MMAs of one k-block, fully unrolled: MT sub-tiles x KK 16-deep steps (x 2 for a tile wider than 256 columns).
// The issuing warp's instruction stream is what bounds the kernel when operands arrive in time (a single extra
// branch per MMA in this loop cost 44 % on a weight-grad launch), so nothing here is computed per MMA that can be
// computed per k-block, and only the first MMA into an accumulator carries a predicate.
// The steps of one accumulator share an election and take one addition per operand each, and whether the next stage has
// arrived is asked before the MMAs of this one are issued: a k-block cost the issuing warp ~100 cycles of waiting for its own
// barrier and ~35 per MMA beyond what the tensor core needs (with the coordinates worked out before the dependency wait, see
// `ahead_done`: 3 x 3, 64 -> 64 on 128 x 8 x 8: 8.8 -> 7.5 us; 128 -> 128 on 256 x 19 x 19, weight gradient: 33.6 -> 31.3).
template <int KK, int MT, bool WIDE, bool PAIR>
__device__ __forceinline__ void issue_kblock(uint32_t d_tmem, uint32_t acc_stride, uint32_t a_lo, uint32_t a_hi, uint32_t a_sub,
                                             uint32_t b_lo, uint32_t b_hi, uint32_t a_adv, uint32_t b_adv, uint32_t idesc,
                                             uint32_t idesc2, uint32_t b_wide_off, bool fresh) {
#pragma unroll
  for (int j = 0; j < MT; ++j) {
    tc_mma_steps<KK, PAIR>(d_tmem + (uint32_t)j * acc_stride, a_lo + (uint32_t)j * a_sub, a_hi, b_lo, b_hi, a_adv, b_adv, idesc,
                           fresh ? 0u : 1u);
    if (WIDE)
      tc_mma_steps<KK, false>(d_tmem + 256u, a_lo, a_hi, b_lo + b_wide_off, b_hi, a_adv, b_adv, idesc2, fresh ? 0u : 1u);
  }
}

// What the issuing warp needs for the k-blocks of one work item, fixed for the launch.
struct IssueCtx {
  uint32_t ring_u32, tiles_u32, stage_bytes, b_bytes, b_in_stage;   // b_in_stage: offset of B inside a stage
  uint32_t acc_stride, a_adv, b_adv, idesc, idesc2;
  uint32_t a_desc0_lo, b_desc0_lo, a_hi, b_hi, a_sub, b_wide_off;   // descriptors: the address in the lower word is filled in
  int stages, b_resident;
};

// k-blocks [kb0, kb1) of one work item; returns false after a wait that ran out.
template <int KK, int MT, bool WIDE, bool PAIR>
__device__ __forceinline__ bool issue_item(const IssueCtx& c, SharedCtl* ctl, unsigned int* status, uint32_t d_tmem,
                                           int kb0, int kb1, int& s, uint32_t& ph) {
  bool ready = mbar_test_wait(&ctl->full[s], ph);
  for (int kb = kb0; kb < kb1; ++kb) {
    if (!__all_sync(0xffffffffu, ready) && !ctl_wait_warp_role(ctl, &ctl->full[s], ph, status, 2)) return false;
    tc_fence_after();
    const uint32_t sa = c.ring_u32 + (uint32_t)s * c.stage_bytes;
    const uint32_t sb = c.b_resident ? c.tiles_u32 + (uint32_t)kb * c.b_bytes : sa + c.b_in_stage;
    uint64_t* const done = &ctl->empty[s];
    if (++s == c.stages) { s = 0; ph ^= 1u; }
    ready = mbar_test_wait(&ctl->full[s], ph);      // the answer is under way while these are issued
    // descriptors differ from the templates only in the 14-bit start address (no carry out of it: shared memory
    // ends below 256 KB)
    issue_kblock<KK, MT, WIDE, PAIR>(d_tmem, c.acc_stride, c.a_desc0_lo | (sa >> 4), c.a_hi, c.a_sub, c.b_desc0_lo | (sb >> 4),
                                     c.b_hi, c.a_adv, c.b_adv, c.idesc, c.idesc2, c.b_wide_off, kb == kb0);
    // stage is free once these MMAs have read it (in both CTAs of a pair)
    if (PAIR) tc_commit2_both(done);
    else tc_commit(done);
  }
  return true;
}

// Flat mode: the k-blocks of one work item, channel chunk by channel chunk. An A stage holds the chunk's input rows, so
// filter tap (r, s) of sub-tile j is a descriptor offset of r * pitch + s positions into it: the swizzle is a function of
// the address alone, so a tile may start at any of its rows.
struct FlatCtx {
  uint32_t a_ring_u32, b_ring_u32, a_stage_bytes, row_units;   // row_units: one position in 16-byte units
  uint32_t lead_units, pitch_units, b_tap_units;               // b_tap_units: from tap to tap of the resident panel
  int cchunks, R, S, a_stages, b_stages, b_resident;
};
template <int KK, int MT, bool PAIR>
__device__ __forceinline__ bool issue_flat_item(const IssueCtx& c, const FlatCtx& f, SharedCtl* ctl, unsigned int* status,
                                                uint32_t d_tmem, int& as, uint32_t& aph, int& bs, uint32_t& bph) {
  bool fresh = true;
  bool a_ready = mbar_test_wait(&ctl->a_full[as], aph);
  bool b_ready = !f.b_resident && mbar_test_wait(&ctl->full[bs], bph);
  for (int cc = 0; cc < f.cchunks; ++cc) {
    if (!__all_sync(0xffffffffu, a_ready) && !ctl_wait_warp_role(ctl, &ctl->a_full[as], aph, status, 2)) return false;
    uint32_t a_row = ((f.a_ring_u32 + (uint32_t)as * f.a_stage_bytes) >> 4) + f.lead_units;
    uint32_t b_tap = (f.b_ring_u32 + (uint32_t)cc * c.b_bytes) >> 4;
    uint64_t* const a_done = &ctl->a_empty[as];
    if (++as == f.a_stages) { as = 0; aph ^= 1u; }
    a_ready = mbar_test_wait(&ctl->a_full[as], aph);
    for (int r = 0; r < f.R; ++r, a_row += f.pitch_units) {
      uint32_t a_tap = a_row;
      for (int sx = 0; sx < f.S; ++sx, a_tap += f.row_units) {
        if (f.b_resident) {
          tc_fence_after();
          issue_kblock<KK, MT, false, PAIR>(d_tmem, c.acc_stride, c.a_desc0_lo | a_tap, c.a_hi, c.a_sub, c.b_desc0_lo | b_tap,
                                            c.b_hi, c.a_adv, c.b_adv, c.idesc, c.idesc2, 0u, fresh);
          b_tap += f.b_tap_units;
        } else {
          if (!__all_sync(0xffffffffu, b_ready) && !ctl_wait_warp_role(ctl, &ctl->full[bs], bph, status, 2)) return false;
          tc_fence_after();
          const uint32_t b_at = (f.b_ring_u32 + (uint32_t)bs * c.b_bytes) >> 4;
          uint64_t* const done = &ctl->empty[bs];
          if (++bs == f.b_stages) { bs = 0; bph ^= 1u; }
          b_ready = mbar_test_wait(&ctl->full[bs], bph);
          issue_kblock<KK, MT, false, PAIR>(d_tmem, c.acc_stride, c.a_desc0_lo | a_tap, c.a_hi, c.a_sub, c.b_desc0_lo | b_at,
                                            c.b_hi, c.a_adv, c.b_adv, c.idesc, c.idesc2, 0u, fresh);
          if (PAIR) tc_commit2_both(done);
          else tc_commit(done);
        }
        fresh = false;
      }
    }
    // every MMA that reads this A stage has been issued before this point
    if (PAIR) tc_commit2_both(a_done);
    else tc_commit(a_done);
  }
  return true;
}

// The bf16 epilogue of 32 columns of one row: packed fp32 adds for the bias, one conversion per pair,
// ReLU and the mask of the previous layer's ReLU on the packed bf16 pair (rounding is monotone, so clamping after it gives
// the same bits as clamping before), into 16-byte chunks of a 128-byte swizzled slab row (chunk index XOR row mod 8, the
// layout the store's tensor map expects).
// What a launch does not use is not there at all: two epilogue warps share a scheduler, and with the flags tested per
// element a 32 x 64 slab took 2300 cycles, most of them branches.
// PART: only the first `valid` of the 32 columns exist, the others are written as zeros (16 channels of 32: element by element
// this took ~4000 cycles per 32 x 32 group and kept the issuing warp waiting for accumulators: ResNet-20's step at 128 images,
// whose first stage has 16 channels: 1362 -> 1310 us).
template <bool BIAS, bool RELU, bool MASK, bool ADD, bool PART, bool SCALE = false>
__device__ __forceinline__ void epilogue_half(const uint32_t (&v)[32], uint8_t* row, int swz, int half, const float* bias,
                                              const uint4* mask, const uint4* add, int valid, const float* scale = nullptr) {
  const __nv_bfloat162 zero2 = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 o;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
    float4 bq[2];   // eight columns' worth at a time: all 32 would put the kernel over its register budget
    if (BIAS && !PART) {
      bq[0] = __ldg(reinterpret_cast<const float4*>(bias + q * 8));
      bq[1] = __ldg(reinterpret_cast<const float4*>(bias + q * 8 + 4));
    } else if (BIAS) {
      float* const b1 = reinterpret_cast<float*>(&bq[0]);
#pragma unroll
      for (int e = 0; e < 8; ++e) b1[e] = q * 8 + e < valid ? __ldg(bias + q * 8 + e) : 0.f;
    }
    const float* bb = reinterpret_cast<const float*>(&bq[0]);
    float sc[8];
    if (SCALE) {
#pragma unroll
      for (int e = 0; e < 8; ++e) sc[e] = !PART || q * 8 + e < valid ? __ldg(scale + q * 8 + e) : 0.f;
    }
    const uint4 av = ADD ? add[q] : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t* aw = reinterpret_cast<const uint32_t*>(&av);
    const __nv_bfloat162* m2 = reinterpret_cast<const __nv_bfloat162*>(&mask[q]);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float x0 = __uint_as_float(v[q * 8 + 2 * e]), x1 = __uint_as_float(v[q * 8 + 2 * e + 1]);
      if (SCALE) {
        x0 = fmaf(x0, sc[2 * e], bb[2 * e]);
        x1 = fmaf(x1, sc[2 * e + 1], bb[2 * e + 1]);
      } else if (BIAS) {
        add2_f32(v[q * 8 + 2 * e], v[q * 8 + 2 * e + 1], bb[2 * e], bb[2 * e + 1], x0, x1);
      }
      if (ADD) {
        x0 += __uint_as_float(aw[e] << 16);
        x1 += __uint_as_float(aw[e] & 0xFFFF0000u);
      }
      __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
      if (RELU) h = __hmax2(h, zero2);
      uint32_t w = *reinterpret_cast<uint32_t*>(&h);
      if (MASK) w &= __hgt2_mask(m2[e], zero2);
      if (PART) w = q * 8 + 2 * e + 1 < valid ? w : q * 8 + 2 * e < valid ? w & 0xFFFFu : 0u;
      ow[e] = w;
    }
    *reinterpret_cast<uint4*>(row + ((half * 4 + q) ^ swz) * 16) = o;
  }
}

template <bool EXT, bool PART>
__device__ __forceinline__ void epilogue_kinds(int kind, bool addend, const uint32_t (&v)[32], uint8_t* row, int swz, int half,
                                               const float* bias, const uint4* m, const uint4* av, int valid) {
  if (EXT && addend) {                  // data-gradients: no bias, no ReLU
    if (kind & 4) epilogue_half<false, false, true, EXT, PART>(v, row, swz, half, bias, m, av, valid);
    else epilogue_half<false, false, false, EXT, PART>(v, row, swz, half, bias, m, av, valid);
    return;
  }
  switch (kind) {   // 1: bias, 2: ReLU, 4: mask
    case 0: epilogue_half<false, false, false, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    case 1: epilogue_half<true, false, false, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    case 2: epilogue_half<false, true, false, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    case 3: epilogue_half<true, true, false, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    case 4: epilogue_half<false, false, true, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    case 5: epilogue_half<true, false, true, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    case 6: epilogue_half<false, true, true, false, PART>(v, row, swz, half, bias, m, av, valid); break;
    default: epilogue_half<true, true, true, false, PART>(v, row, swz, half, bias, m, av, valid); break;
  }
}

// The epilogue of a convolution whose normalisation is known beforehand (inference): scale, shift, residual and ReLU.
template <bool PART>
__device__ __forceinline__ void epilogue_norm(bool relu, bool addend, const uint32_t (&v)[32], uint8_t* row, int swz, int half,
                                              const float* bias, const float* scale, const uint4* m, const uint4* av,
                                              int valid) {
  if (addend) {
    if (relu) epilogue_half<true, true, false, true, PART, true>(v, row, swz, half, bias, m, av, valid, scale);
    else epilogue_half<true, false, false, true, PART, true>(v, row, swz, half, bias, m, av, valid, scale);
  } else {
    if (relu) epilogue_half<true, true, false, false, PART, true>(v, row, swz, half, bias, m, av, valid, scale);
    else epilogue_half<true, false, false, false, PART, true>(v, row, swz, half, bias, m, av, valid, scale);
  }
}

// PAIR: the instantiation that runs as clusters of two CTAs (p.pair != 0). It is a kernel of its own because a
// kernel that contains cta_group::2 instructions can only be launched with an even cluster size.
// EXT: the instantiation whose bf16 epilogue can scatter rows and take an addend. The tests for these cost the epilogue of
// every other launch what they do not use: 1 x 1 layers, which are bound by it, ran 8 % slower with them (NIN's training
// step at 64 images: 1255 instead of 1186 us).
// FLAT: the instantiation for A_FLAT_K, whose rows are always scattered (EXT).
// NORM: the instantiation for launches with a scale (EXT).
// PHASES: the instantiation for several output phases of a strided data-gradient (EXT).
// LEAN: the instantiation for fp32 output with fewer registers (74: the bf16 epilogues are what takes 138) and less shared
// memory, for launches beside which others are to run.
template <bool PAIR, bool EXT, bool FLAT, bool NORM, bool LEAN, bool PHASES = false>
__global__ void __maxnreg__(LEAN ? LEAN_MAX_REGS : GEMM_MAX_REGS) gemm_tc_kernel(
    const __grid_constant__ std::conditional_t<PHASES, GemmPhasesParams, GemmTcParams> p) {
#ifdef RB_GEMM_PROFILE
  const long long t_kernel0 = clock64();
#endif
  extern __shared__ uint8_t smem_raw[];
  // tiles start on a 1024-byte boundary (swizzle atoms); control block follows the tiles
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = tiles + (LEAN ? LEAN_TILE_BYTES : TILE_SMEM_BYTES);
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(staging + STAGING_BYTES);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);   // known to be the same in all lanes
  const int lane = threadIdx.x & 31;

  // CTA pairs: rank of this CTA in its pair, and the persistent loop runs over pairs
  constexpr bool pair = PAIR;
  const uint32_t cta_rank = pair ? cluster_ctarank() : 0u;
  const int cta_id = pair ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int cta_step = pair ? (int)(gridDim.x >> 1) : (int)gridDim.x;

  const int mt = p.mt;
  const int a_bytes = BM * p.bk * 2;            // one 128-row sub-tile
  const int b_bytes = p.bn_load * p.bk * 2;
  const int panel_bytes = p.b_resident ? p.num_kb * b_bytes : 0;
  const int stage_bytes = mt * a_bytes + (p.b_resident ? 0 : b_bytes);
  uint8_t* ring = tiles + panel_bytes;
  const int stages = p.stages;

  const bool box = !FLAT && p.a_mode == A_BOX_K;
  const int bx_groups = box ? (p.cv_P + mt * p.bx_rows - 1) / (mt * p.bx_rows) : 1;   // work items per image
  const int m_units = FLAT  ? (p.fl_units + mt - 1) / mt
                      : box ? (p.M / (p.cv_P * p.cv_Q)) * bx_groups
                            : (p.M + BM * mt - 1) / (BM * mt);
  const int m_items = pair ? (m_units + 1) >> 1 : m_units;   // a pair's item is two CTA-sized units
  const int n_tiles = p.n_tiles;
  // whole items first, then the parts of the cut items of the last wave (tail cut; never in flat mode)
  const int direct = m_items * n_tiles - p.tail_items;
  int num_work = p.tail_items > 0 ? direct + p.tail_items * p.tail_split : m_items * n_tiles * p.split_k;
  if constexpr (PHASES) num_work = p.ph[p.phases - 1].work0 + p.ph[p.phases - 1].m_items * n_tiles;
  // flat mode: [A ring: fl_a_stages x fl_a_bytes][B ring: stages x b_bytes, or the resident panel]
  uint8_t* const b_ring = FLAT ? tiles + p.fl_a_stages * p.fl_a_bytes : tiles;
  const int kb_per_split = (p.num_kb + p.split_k - 1) / p.split_k;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      // one arrival per producer warp that fills it (a pair: both CTAs' producers arrive on the leader's barrier)
      mbar_init(&ctl->full[s], FLAT ? (pair ? 2 : 1) : pair ? 4 : (p.b_resident ? 1 : 2));
      mbar_init(&ctl->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&ctl->acc_full[a], 1);
      mbar_init(&ctl->acc_empty[a], pair ? 2 * EPI_WARPS : EPI_WARPS);
    }
    mbar_init(&ctl->b_full, 1);
    for (int a = 0; FLAT && a < MAX_A_STAGES; ++a) {
      mbar_init(&ctl->a_full[a], pair ? 2 : 1);
      mbar_init(&ctl->a_empty[a], 1);
    }
    for (int w = 0; w < EPI_WARPS; ++w) mbar_init(&ctl->mask_bar[w], 1);
    ctl->abort_flag = 0;
    mbar_fence_init();
    if constexpr (PHASES)
      for (int k = 0; k < p.phases; ++k) tma_prefetch_desc(&p.ph[k].tm_a);
    else
      tma_prefetch_desc(&p.tm_a);
    tma_prefetch_desc(&p.tm_b);
    if (!PHASES) tma_prefetch_desc(&p.tm_d);
    if (!PHASES && p.epi == EPI_BF16 && p.mask_src) tma_prefetch_desc(&p.tm_mask);
    if (p.tail_items > 0) tma_prefetch_desc(&p.tm_ws);
  }
  if (warp == 1) {
    if (pair) {
      tmem_alloc2(&ctl->tmem_base, 512);   // both CTAs of the pair execute this; each gets the same address
      tmem_relinquish2();
    } else {
      tmem_alloc(&ctl->tmem_base, 512);
      tmem_relinquish();
    }
  }
  if (p.a_mode == A_BOX_MN && p.wb_rows * p.wb_w < p.bk) {
    // the k-block's rows that no box ever writes: zeros in every stage and both operands
    const int first = p.wb_rows * p.wb_w * 8, per_block = p.bk * 8;        // in 16-byte units per 64-column block
    const int blocks = stages * stage_bytes / (p.bk * 128);
    for (int i = threadIdx.x; i < blocks * per_block; i += GEMM_THREADS)
      if (i % per_block >= first) *reinterpret_cast<uint4*>(ring + (size_t)i * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  if (pair) cluster_sync_all();   // the peer's barriers are initialised before anything of ours signals them
  tc_fence_after();
  // Programmatic dependent launch (option `pdl`): what touches only this CTA's own shared memory, TMEM and the launch
  // parameters may run while the kernels before this one on the stream are still finishing. Every warp that touches anything
  // else (operands, bias, mask, output, workspace) calls `ahead_done` first, which returns when they have completed and
  // flushed: the producers right before their first load, when its coordinates have been worked out and its stage claimed
  // (1 - 2 us of integer divisions and first touches of code and parameters). Without the launch attribute the instructions
  // do nothing. The issuing warp does not call it: it waits for the first stage meanwhile, so the time that the kernels before
  // this one still take after its blocks are resident counts against its wait limit (WAIT_LIMIT_NS; those that release their
  // dependents early take a few milliseconds at most).
  bool ahead = true;
  auto ahead_done = [&ahead]() {
    if (!ahead) return;
    ahead = false;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  };
  const uint32_t tmem_base = ctl->tmem_base;

  if (warp == 0 || warp == PRODUCER_B_WARP) {
    // ------------------------------ producers ------------------------------
    // One thread gets its TMA instructions through one after the other; boxes issued by other threads overlap with them.
    // So the loads of a stage are spread: warp 0 issues the A loads (one lane per box, all lanes of a mode execute the same
    // instruction), warp PRODUCER_B_WARP the B loads, and both arrive on the stage's `full` barrier with the
    // bytes they bring.
    const bool is_a = warp == 0;
    int s = 0, issued = 0;
    uint32_t ph = 0;
    bool ok = true;
    if (FLAT && (is_a || !p.b_resident)) {
      // A: a stage is the fl_rows input rows of one channel chunk, one lane per row, every one fl_pitch positions of which
      // those outside the image arrive as zeros. B: one (tap, channel chunk) tile per stage, one lane per box.
      const int nst = is_a ? p.fl_a_stages : stages;
      uint64_t* const fullb = is_a ? ctl->a_full : ctl->full;
      uint64_t* const emptyb = is_a ? ctl->a_empty : ctl->empty;
      const uint32_t full0_leader = pair ? mapa_shared(smem_u32(fullb), 0u) : 0u;
      const int row_bytes = p.bk * 2;
      const uint32_t tx = is_a ? (uint32_t)(p.fl_rows * p.fl_pitch * row_bytes) : (uint32_t)b_bytes;
      const bool mn = p.b_mode == B_DGRAD_MN;
      const int b_split = p.b_split > 0 ? p.b_split : 1, b_rows = p.bn_load / b_split;
      const int nload = is_a ? p.fl_rows : (mn ? p.bn_load / 64 : b_split);
      auto claim = [&]() -> bool {   // wait for a free stage and announce its bytes
        int w_ok = 1;
        if (lane == 0) {
          w_ok = ctl_wait_role(ctl, &emptyb[s], ph ^ 1u, p.status, is_a ? 0 : 1) ? 1 : 0;
          if (w_ok) {
            if (pair) mbar_expect_tx_cluster(full0_leader + (uint32_t)s * 8u, tx);
            else mbar_expect_tx(&fullb[s], tx);
          }
        }
        return __shfl_sync(0xffffffffu, w_ok, 0) != 0;
      };
      for (int work = cta_id; work < num_work && ok; work += cta_step) {
        const int tn = work / m_items;
        const int tm = (work - tn * m_items) * (pair ? 2 : 1) + (int)cta_rank;
        const int n0 = tn * p.bn + (pair ? (int)cta_rank * p.bn_load : 0);
        const int f0 = tm * mt * p.fl_step;
        const int g0 = f0 / p.fl_pitch;
        // the item's first position always lies at fl_lead, whatever its column: both CTAs of a pair use one descriptor
        uint8_t* const row0 = tiles + (p.fl_lead - (f0 - g0 * p.fl_pitch)) * row_bytes;
        for (int cc = 0; cc < p.cv_cchunks && ok; ++cc) {
          if (is_a) {
            if (!claim()) { ok = false; break; }
            ahead_done();
            for (int i = lane; i < nload; i += 32) {
              const int g = g0 + i, n = g / p.fl_hp, h = g - n * p.fl_hp - p.fl_pad_h;
              uint8_t* to = row0 + s * p.fl_a_bytes + i * p.fl_pitch * row_bytes;
              if (pair) tma2_load_4d(to, &p.tm_a, full0_leader + (uint32_t)s * 8u, cc * p.bk, -p.fl_pad_w, h, n);
              else tma_load_4d(to, &p.tm_a, &fullb[s], cc * p.bk, -p.fl_pad_w, h, n);
            }
            __syncwarp();
            ++issued;
            if (++s == nst) { s = 0; ph ^= 1u; }
            continue;
          }
          for (int r = 0; r < p.fl_R && ok; ++r)
            for (int sx = 0; sx < p.cv_S; ++sx) {
              if (!claim()) { ok = false; break; }
              ahead_done();
              if (lane < nload) {
                const int wtap = p.dg_dv == 0 ? r * p.cv_S + sx : p.dg_base + r * p.dg_du + sx * p.dg_dv;
                const int c0 = mn ? n0 + 64 * lane : cc * p.bk, c2 = mn ? cc * p.bk : n0 + lane * b_rows;
                uint8_t* to = b_ring + s * b_bytes + lane * (mn ? p.bk * 128 : b_rows * row_bytes);
                if (pair) tma2_load_3d(to, &p.tm_b, full0_leader + (uint32_t)s * 8u, c0, wtap, c2);
                else tma_load_3d(to, &p.tm_b, &fullb[s], c0, wtap, c2);
              }
              __syncwarp();
              ++issued;
              if (++s == nst) { s = 0; ph ^= 1u; }
            }
        }
      }
      if (!ok && lane == 0 && pair && cta_rank != 0) {
        const uint64_t t0 = globaltimer_ns();   // as below
        while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      } else if (!ok && lane == 0) {
        // drain: wait (bounded) until the copies already issued have landed
        const int back = min(issued, nst);
        for (int i = 0; i < back; ++i) {
          if (s == 0) { s = nst; ph ^= 1u; }
          --s;
          mbar_wait_bounded(&fullb[s], ph, 100000000ull);
        }
      }
    } else if (!FLAT && (is_a || !p.b_resident)) {
      // Loads this warp issues per stage, one lane each. What a lane's load needs is worked out once per launch (where in a
      // stage it goes) or per work item (its pixel, tap or column), and carried from k-block to k-block by additions: with
      // the divisions by run-time values that the coordinates otherwise take, a k-block cost the warp ~1200 cycles.
      const int a_split = p.a_split > 0 ? p.a_split : 1, b_split = p.b_split > 0 ? p.b_split : 1;
      const bool a_mn_blocks = p.a_mode == A_TILED_MN || p.a_mode == A_BOX_MN;
      const int mode = is_a ? p.a_mode : 8 + p.b_mode;
      int nload;
      if (is_a) nload = box ? mt : (a_mn_blocks ? 2 : a_split) * mt;
      else if (p.b_mode == B_TILED_MN || p.b_mode == B_DGRAD_MN) nload = p.bn_load / 64;
      else if (p.b_mode == B_IM2COL_MN || p.b_mode == B_BOX_MN)
        nload = p.wg_taps > 1 ? p.wg_taps * (p.wg_cw / 64) : p.bn_load / 64;
      else nload = b_split;
      // a pair counts every load on the leader's `full` barriers
      const uint32_t full0_leader = pair ? mapa_shared(smem_u32(&ctl->full[0]), 0u) : 0u;
      const uint32_t my_tx = p.a_mode == A_BOX_MN ? (uint32_t)(nload * p.wb_rows * p.wb_w * 128)
                             : !is_a ? (uint32_t)b_bytes
                             : box ? (uint32_t)(mt * p.bx_rows * p.cv_Q * p.bk * 2)   // the boxes bring whole rows only
                                   : (uint32_t)(mt * a_bytes);
      // sub-tile of this lane's A load, and which of the sub-tile's boxes it is; where the load goes inside a stage
      const int aj = a_mn_blocks ? (lane >> 1) : lane / a_split;
      const int aq = a_mn_blocks ? (lane & 1) : lane - aj * a_split;
      const int a_rows = BM / a_split, b_rows = p.bn_load / b_split;
      int dst;
      if (box && is_a) dst = lane * a_bytes;
      else if (is_a) dst = aj * a_bytes + (a_mn_blocks ? aq * p.bk * 128 : aq * a_rows * p.bk * 2);
      else dst = mt * a_bytes + lane * (p.b_mode == B_TILED_K || p.b_mode == B_TILED_K3 ? b_rows * p.bk * 2 : p.bk * 128);
      // the taps of a convolution are walked in order; a weight-grad walks pixels, bk at a time
      const int cchunks = p.cv_cchunks > 0 ? p.cv_cchunks : 1;
      int taps_w = p.cv_S > 0 ? p.cv_S : 1, dg_base = p.dg_base;
      const CUtensorMap* map_a = &p.tm_a;
      int step_q = 0, step_p = 0, step_n = 0;
      if (mode == 8 + B_IM2COL_MN) {
        step_q = p.bk % p.cv_Q;
        step_p = (p.bk / p.cv_Q) % p.cv_P;
        step_n = p.bk / (p.cv_Q * p.cv_P);
      }
      const int wg_apt = p.wg_taps > 1 ? p.wg_cw / 64 : 32;     // 64-column blocks per tap of a tile (one tap: all of them)
      const int wg_t = lane / wg_apt, wg_c = 64 * (lane - wg_t * wg_apt);
      for (int work = cta_id; work < num_work && ok; work += cta_step) {
        const WorkItem it = decode_work<PHASES>(p, work, m_items, direct, kb_per_split);
        if constexpr (PHASES) {
          taps_w = p.ph[it.phase].S;
          dg_base = p.ph[it.phase].dg_base;
          map_a = &p.ph[it.phase].tm_a;
        }
        const int tn = it.tn, kb0 = it.kb0, kb1 = it.kb1;
        const int tm = pair ? it.tm * 2 + (int)cta_rank : it.tm;
        const int m0 = tm * BM * mt;
        int a_w = 0, a_h = 0, a_n = 0;   // first pixel of this lane's A load
        if (mode == A_IM2COL_K && lane < nload) {
          if constexpr (PHASES) {
            const GemmPhase& ph = p.ph[it.phase];
            pixel_coords(ph.P, ph.Q, 1, ph.lower_h, ph.lower_w, m0 + aj * BM + aq * a_rows, a_w, a_h, a_n);
          } else {
            pixel_coords(p.cv_P, p.cv_Q, p.cv_stride, p.cv_lower_h, p.cv_lower_w, m0 + aj * BM + aq * a_rows, a_w, a_h, a_n);
          }
        }
        if (mode == A_BOX_K) {   // lane j loads sub-tile j: image a_n, first output row a_h
          a_n = tm / bx_groups;
          a_h = ((tm - a_n * bx_groups) * mt + lane) * p.bx_rows;
        }
        const int n0 = tn * p.bn + (pair ? (int)cta_rank * p.bn_load : 0);   // a pair's CTA loads its half of the rows
        // filter tap (r, sx), its number, and channel chunk of k-block kb
        int tap = kb0 / cchunks;
        int cc = kb0 - tap * cchunks;
        int r = tap / taps_w;
        int sx = tap - r * taps_w;
        // weight-grad: this lane's tap and channel, and the k-block's first pixel (column, row, image) or box
        int wg_r = 0, wg_s = 0, wg_c0 = wg_c, px = 0, py = 0, pn = 0;
        if (p.wgrad) {
          int b_tap;
          if (p.wg_taps > 1) {
            b_tap = min(tn * p.wg_taps + wg_t, p.wg_ntaps - 1);   // slots past the last tap reload it; the epilogue skips them
          } else {
            b_tap = tn / p.wg_ctiles;
            wg_c0 = (tn - b_tap * p.wg_ctiles) * p.bn + 64 * lane;
          }
          wg_r = b_tap / taps_w;
          wg_s = b_tap - wg_r * taps_w;
          if (mode == 8 + B_IM2COL_MN) {
            const int pix = kb0 * p.bk, pq = p.cv_P * p.cv_Q;
            pn = pix / pq;
            py = (pix - pn * pq) / p.cv_Q;
            px = pix - pn * pq - py * p.cv_Q;
          } else if (p.a_mode == A_BOX_MN) {
            const int per = p.wb_groups * p.wb_pieces;
            pn = kb0 / per;
            py = (kb0 - pn * per) / p.wb_pieces;       // row group
            px = kb0 - pn * per - py * p.wb_pieces;    // piece of the row
          }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          int w_ok = 1;
          if (lane == 0) {
            w_ok = ctl_wait_role(ctl, &ctl->empty[s], ph ^ 1u, p.status, is_a ? 0 : 1) ? 1 : 0;
            if (w_ok) {
              if (pair) mbar_expect_tx_cluster(full0_leader + (uint32_t)s * 8u, my_tx);
              else mbar_expect_tx(&ctl->full[s], my_tx);
            }
          }
          w_ok = __shfl_sync(0xffffffffu, w_ok, 0);
          if (!w_ok) { ok = false; break; }
          uint8_t* to = ring + s * stage_bytes + dst;
          uint64_t* bar = &ctl->full[s];
          const uint32_t bar2 = full0_leader + (uint32_t)s * 8u;   // pairs: the leader's barrier of this stage
          ahead_done();
          if (lane < nload) {
            // pairs: K-major A; K-major B or filters as they lie
            switch (mode) {
              case A_TILED_K:
                if (pair) tma2_load_2d(to, &p.tm_a, bar2, kb * p.bk, m0 + aj * BM + aq * a_rows);
                else tma_load_2d(to, &p.tm_a, bar, kb * p.bk, m0 + aj * BM + aq * a_rows);
                break;
              case A_IM2COL_K:
                if (pair) tma2_load_im2col_4d(to, &p.tm_a, bar2, cc * p.bk, a_w, a_h, a_n, (uint16_t)sx, (uint16_t)r);
                else tma_load_im2col_4d(to, map_a, bar, cc * p.bk, a_w, a_h, a_n, (uint16_t)sx, (uint16_t)r);
                break;
              case A_TILED_MN:   // two boxes of 64 rows(M) x bk per sub-tile
                if (!pair) tma_load_2d(to, &p.tm_a, bar, m0 + aj * BM + 64 * aq, kb * p.bk);
                break;
              case A_BOX_K:
                if (!pair) tma_load_4d(to, &p.tm_a, bar, cc * p.bk, sx - p.bx_pad_w, a_h + r - p.bx_pad_h, a_n);
                break;
              case A_BOX_MN:
                if (!pair) tma_load_4d(to, &p.tm_a, bar, m0 + aj * BM + 64 * aq, px * p.wb_w, py * p.wb_rows, pn);
                break;
              case 8 + B_TILED_K:
                if (pair) tma2_load_2d(to, &p.tm_b, bar2, kb * p.bk, n0 + lane * b_rows);
                else tma_load_2d(to, &p.tm_b, bar, kb * p.bk, n0 + lane * b_rows);
                break;
              case 8 + B_TILED_MN:
                if (!pair) tma_load_2d(to, &p.tm_b, bar, n0 + 64 * lane, kb * p.bk);
                break;
              case 8 + B_IM2COL_MN:
                if (!pair)
                  tma_load_im2col_4d(to, &p.tm_b, bar, wg_c0, px * p.cv_stride + p.cv_lower_w,
                                     py * p.cv_stride + p.cv_lower_h, pn, (uint16_t)wg_s, (uint16_t)wg_r);
                break;
              case 8 + B_BOX_MN:
                if (!pair)
                  tma_load_4d(to, &p.tm_b, bar, wg_c0, px * p.wb_w + wg_s - p.wb_pad_w, py * p.wb_rows + wg_r - p.wb_pad_h,
                              pn);
                break;
              default: {   // B_TILED_K3, B_DGRAD_MN: tap of the filters in memory
                const int wtap = p.dg_dv == 0 ? tap : dg_base + r * p.dg_du + sx * p.dg_dv;
                const bool k3 = p.b_mode == B_TILED_K3;
                const int c0 = k3 ? cc * p.bk : n0 + 64 * lane, c2 = k3 ? n0 + lane * b_rows : cc * p.bk;
                if (pair) tma2_load_3d(to, &p.tm_b, bar2, c0, wtap, c2);
                else tma_load_3d(to, &p.tm_b, bar, c0, wtap, c2);
                break;
              }
            }
          }
          __syncwarp();
          if (++cc == cchunks) {
            cc = 0;
            ++tap;
            if (++sx == taps_w) { sx = 0; ++r; }
          }
          if (p.a_mode == A_BOX_MN) {
            if (++px == p.wb_pieces) {
              px = 0;
              if (++py == p.wb_groups) { py = 0; ++pn; }
            }
          } else if (mode == 8 + B_IM2COL_MN) {
            px += step_q;
            py += step_p;
            pn += step_n;
            if (px >= p.cv_Q) { px -= p.cv_Q; ++py; }
            if (py >= p.cv_P) { py -= p.cv_P; ++pn; }
          }
          ++issued;
          if (++s == stages) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok && lane == 0 && pair && cta_rank != 0) {
        // this CTA's copies complete on the leader's barriers, which cannot be waited on from here: give them time
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
      } else if (!ok && lane == 0) {
        // drain: wait (bounded) until the copies already issued have landed
        const int back = min(issued, stages);
        for (int i = 0; i < back; ++i) {
          if (s == 0) { s = stages; ph ^= 1u; }
          --s;
          mbar_wait_bounded(&ctl->full[s], ph, 100000000ull);
        }
      }
    } else {
      // resident B: this warp loads the one panel the CTA will ever need, k-blocks spread over its lanes
      if (blockIdx.x < num_work) {
        if (lane == 0) mbar_expect_tx(&ctl->b_full, (uint32_t)panel_bytes);
        __syncwarp();
        ahead_done();
        for (int kb = lane; kb < p.num_kb; kb += 32) load_b(p, b_ring + kb * b_bytes, &ctl->b_full, kb, 0);
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // the whole warp runs this, converged, and one elected thread issues (see tc_mma_f16)
    if (cta_rank == 0) {   // of a pair, only the leader issues
      const bool a_mn = p.a_mode == A_TILED_MN || p.a_mode == A_BOX_MN;
      const bool b_mn = p.b_mode != B_TILED_K && p.b_mode != B_TILED_K3;
      // a tile wider than 256 columns is two MMAs side by side (256 + the rest) that share the A descriptor
      const uint32_t idesc = make_idesc_bf16(pair ? 2 * BM : BM, (uint32_t)min(p.bn, 256), a_mn ? 1u : 0u, b_mn ? 1u : 0u);
      const uint32_t idesc2 = p.bn > 256 ? make_idesc_bf16(BM, (uint32_t)(p.bn - 256), a_mn ? 1u : 0u, b_mn ? 1u : 0u) : 0u;
      const uint32_t b_wide_off = (256u * (uint32_t)p.bk * 2u) >> 4;   // 256 rows (K-major) or 4 blocks on
      // K-major: rows of bk*2 bytes, 8-row atoms -> SBO = 8*bk*2; swizzle 128B (bk=64) or 64B (bk=32)
      // MN-major: 64-element (128 B) rows per k, atoms of 8 k -> SBO = 1024, LBO = bk*128 between 64-wide blocks
      const uint32_t k_layout = (p.bk == 64) ? 2u : 4u;
      const uint32_t a_lbo = a_mn ? (uint32_t)p.bk * 128u : 16u;
      const uint32_t a_sbo = a_mn ? 1024u : (uint32_t)p.bk * 16u;
      const uint32_t a_lay = a_mn ? 2u : k_layout;
      const uint32_t b_lbo = b_mn ? (uint32_t)p.bk * 128u : 16u;
      const uint32_t b_sbo = b_mn ? 1024u : (uint32_t)p.bk * 16u;
      const uint32_t b_lay = b_mn ? 2u : k_layout;
      const uint32_t a_adv = a_mn ? (2048u >> 4) : (32u >> 4);  // per 16-deep MMA, in 16-byte units
      const uint32_t b_adv = b_mn ? (2048u >> 4) : (32u >> 4);
      const int kk_steps = p.bk / 16;
      const uint32_t set_cols = (uint32_t)(mt * p.acc_stride);

      int s = 0;
      uint32_t ph = 0;
      int acc = 0;
      uint32_t acc_ph = 0;
      bool ok = true;
      if (p.b_resident && blockIdx.x < num_work) ok = ctl_wait_warp(ctl, &ctl->b_full, 0u, p.status);
      // what the unrolled issue code needs, fixed for the launch
      IssueCtx ic;
      ic.ring_u32 = smem_u32(ring);
      ic.tiles_u32 = smem_u32(tiles);
      ic.stage_bytes = (uint32_t)stage_bytes;
      ic.b_bytes = (uint32_t)b_bytes;
      ic.b_in_stage = (uint32_t)(mt * a_bytes);
      ic.acc_stride = (uint32_t)p.acc_stride;
      ic.a_adv = a_adv;
      ic.b_adv = b_adv;
      ic.idesc = idesc;
      ic.idesc2 = idesc2;
      const uint64_t a_desc0 = make_smem_desc(0u, a_lbo, a_sbo, a_lay), b_desc0 = make_smem_desc(0u, b_lbo, b_sbo, b_lay);
      ic.a_desc0_lo = (uint32_t)a_desc0;
      ic.a_hi = (uint32_t)(a_desc0 >> 32);
      ic.b_desc0_lo = (uint32_t)b_desc0;
      ic.b_hi = (uint32_t)(b_desc0 >> 32);
      ic.a_sub = (uint32_t)(FLAT ? p.fl_step * p.bk * 2 : a_bytes) >> 4;     // next sub-tile of the stage
      ic.b_wide_off = b_wide_off;
      ic.stages = stages;
      ic.b_resident = p.b_resident;
      if (FLAT) {
        FlatCtx fc;
        fc.a_ring_u32 = smem_u32(tiles);
        fc.b_ring_u32 = smem_u32(b_ring);
        fc.a_stage_bytes = (uint32_t)p.fl_a_bytes;
        fc.row_units = (uint32_t)(p.bk * 2) >> 4;
        fc.lead_units = (uint32_t)p.fl_lead * fc.row_units;
        fc.pitch_units = (uint32_t)p.fl_pitch * fc.row_units;
        fc.b_tap_units = (uint32_t)(p.cv_cchunks * b_bytes) >> 4;
        fc.cchunks = p.cv_cchunks;
        fc.R = p.fl_R;
        fc.S = p.cv_S;
        fc.a_stages = p.fl_a_stages;
        fc.b_stages = stages;
        fc.b_resident = p.b_resident;
        int as = 0;
        uint32_t aph = 0;
        const int kind = (kk_steps == 4 ? 0 : 4) + mt;
        for (int work = cta_id; work < num_work && ok; work += cta_step) {
          if (!ctl_wait_warp_role(ctl, &ctl->acc_empty[acc], acc_ph ^ 1u, p.status, 3)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)acc * set_cols;
          switch (kind) {
            case 1: ok = issue_flat_item<4, 1, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            case 2: ok = issue_flat_item<4, 2, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            case 3: ok = issue_flat_item<4, 3, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            case 4: ok = issue_flat_item<4, 4, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            case 5: ok = issue_flat_item<2, 1, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            case 6: ok = issue_flat_item<2, 2, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            case 7: ok = issue_flat_item<2, 3, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
            default: ok = issue_flat_item<2, 4, PAIR>(ic, fc, ctl, p.status, d_tmem, as, aph, s, ph); break;
          }
          if (!ok) break;
          if (pair) tc_commit2_both(&ctl->acc_full[acc]);
          else tc_commit(&ctl->acc_full[acc]);
          if (++acc == p.acc_bufs) { acc = 0; acc_ph ^= 1u; }
        }
      }
      const int issue_kind = (kk_steps == 4 ? 0 : 3) + (idesc2 ? 2 : (mt == 2 ? 1 : 0));
      for (int work = cta_id; work < num_work && ok && !FLAT; work += cta_step) {
        const WorkItem it = decode_work<PHASES>(p, work, m_items, direct, kb_per_split);
        if (!ctl_wait_warp_role(ctl, &ctl->acc_empty[acc], acc_ph ^ 1u, p.status, 3)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)acc * set_cols;
        switch (issue_kind) {
          case 0: ok = issue_item<4, 1, false, PAIR>(ic, ctl, p.status, d_tmem, it.kb0, it.kb1, s, ph); break;
          case 1: ok = issue_item<4, 2, false, PAIR>(ic, ctl, p.status, d_tmem, it.kb0, it.kb1, s, ph); break;
          case 3: ok = issue_item<2, 1, false, PAIR>(ic, ctl, p.status, d_tmem, it.kb0, it.kb1, s, ph); break;
          case 4: ok = issue_item<2, 2, false, PAIR>(ic, ctl, p.status, d_tmem, it.kb0, it.kb1, s, ph); break;
          default:   // one tile wider than 256 columns: never for pairs (refused on the host)
            if (PAIR) ok = false;
            else if (issue_kind == 2) ok = issue_item<4, 1, true, false>(ic, ctl, p.status, d_tmem, it.kb0, it.kb1, s, ph);
            else ok = issue_item<2, 1, true, false>(ic, ctl, p.status, d_tmem, it.kb0, it.kb1, s, ph);
            break;
        }
        if (!ok) break;
        if (pair) tc_commit2_both(&ctl->acc_full[acc]);
        else tc_commit(&ctl->acc_full[acc]);
        if (++acc == p.acc_bufs) { acc = 0; acc_ph ^= 1u; }
      }
    }
  } else if (warp < 2 + EPI_WARPS) {
    // ------------------------------ epilogue ------------------------------
    ahead_done();
    const int lane_base = (warp & 3) * 32;  // TMEM lanes this warp may read
    const uint32_t set_cols = (uint32_t)(mt * p.acc_stride);
    const int col_half = (warp - 2) >> 2;        // which of the two warps of this lane quarter
    uint8_t* stg = staging + (warp - 2) * 4096;  // one 32-row x 128-byte slab buffer per warp
    // a second one (bf16 epilogue, short main loops) lets a slab be worked on while the store of the one before it is
    // still reading shared memory, which takes as long as the slab itself while the output is on its way to memory
    const uint32_t flip_buf = p.epi_bufs == 2 ? (uint32_t)STAGING_BYTES : 0u;
    uint32_t buf_off = 0u;
    const bool has_bias = p.bias != nullptr;
    uint64_t* mbar_m = &ctl->mask_bar[warp - 2];
    uint32_t mask_ph = 0;
    const int epi_kind = (has_bias ? 1 : 0) | (p.relu ? 2 : 0) | (p.mask_src ? 4 : 0);
    int acc = 0;
    uint32_t acc_ph = 0;
    bool ok = true;
    for (int work = cta_id; work < num_work && ok; work += cta_step) {
      const WorkItem it = decode_work<PHASES>(p, work, m_items, direct, kb_per_split);
      const int tn = it.tn;
      const int tm = pair ? it.tm * 2 + (int)cta_rank : it.tm;
      const bool tail = it.tail >= 0;
      {
        RB_PROF_T0(warp == 2);
        if (!ctl_wait(ctl, &ctl->acc_full[acc], acc_ph, p.status)) { ok = false; break; }
        RB_PROF_ADD(warp == 2, 5);
      }
      tc_fence_after();
      int col0;        // first column of D this tile writes
      int col_limit;   // tile-local bound on stored columns
      if (p.wgrad && p.wg_taps > 1) {
        col0 = 0;            // columns are mapped per 32-column chunk below
        col_limit = p.bn;
      } else if (p.wgrad) {
        const int tap = tn / p.wg_ctiles;
        const int c0 = (tn - tap * p.wg_ctiles) * p.bn;
        col0 = tap * p.wg_cpad + c0;
        col_limit = min(p.bn, p.wg_cpad - c0);
      } else {
        col0 = tn * p.bn;
        col_limit = min(p.bn, p.n_store - col0);
      }
      for (int j = 0; j < mt; ++j) {
        int row0 = tm * BM * mt + j * BM + lane_base;   // first row of this warp's 32-row band
        int band_rows = 32;                             // rows of the band that belong to this tile
        if (box) {
          // the sub-tile is bx_rows whole output rows of one image: consecutive rows of D, fewer at the image's
          // lower edge; tile rows past them are computed from stale shared memory and dropped here
          const int b_n = tm / bx_groups;
          const int b_p = ((tm - b_n * bx_groups) * mt + j) * p.bx_rows;
          const int valid = max(0, min(p.bx_rows, p.cv_P - b_p)) * p.cv_Q;
          band_rows = max(0, min(32, valid - lane_base));
          row0 = (b_n * p.cv_P + b_p) * p.cv_Q + lane_base;
          if (band_rows == 0 && !tail) continue;
        }
        const uint32_t t_addr =
            tmem_base + (uint32_t)acc * set_cols + (uint32_t)(j * p.acc_stride) + ((uint32_t)lane_base << 16);
        if (!LEAN && p.epi == EPI_BF16 && !tail) {
          // row of D that this lane's row belongs to (-1: none); only scattered rows and an addend need it
          const bool scatter = FLAT || PHASES || (EXT && p.sc_stride != 0);
          const bool addend = EXT && p.add_src != nullptr;
          long long drow_of = -1;
          if (FLAT) drow_of = flat_row(p, (tm * mt + j) * p.fl_step + lane_base + lane);
          else if constexpr (PHASES) {
            const GemmPhase& ph = p.ph[it.phase];
            if (row0 + lane < ph.M)
              drow_of = scatter_row(row0 + lane, ph.P, ph.Q, p.sc_stride, ph.sc_a, ph.sc_b, p.sc_H, p.sc_W);
          } else if ((scatter || addend) && lane < band_rows && row0 + lane < p.M)
            drow_of = scatter ? scatter_row(row0 + lane, p.cv_P, p.cv_Q, p.sc_stride, p.sc_a, p.sc_b, p.sc_H, p.sc_W)
                              : (long long)(row0 + lane);
          // 64-column slabs: TMEM -> registers -> bias / ReLU / mask -> swizzled shared memory -> TMA store.
          // Each warp owns a 4 KB slab buffer and issues its own stores, so no cross-warp sync is needed.
          // the two warps of a lane quarter alternate slabs, starting with the other warp on the second sub-tile, so
          // that a tile with an odd number of slabs (96 columns = a full and a half slab) splits evenly between them
          for (int c = ((col_half + j) & 1) * 64; c < p.bn && col0 + c < p.n_store; c += 128) {
            uint8_t* buf = stg - buf_off;
            if (lane == 0) {   // the store that last used this buffer has read it
              if (flip_buf) tma_store_wait_read<1>();
              else tma_store_wait_read<0>();
            }
            buf_off ^= flip_buf;
            __syncwarp();
            const int gcol = col0 + c;
            uint4 mreg[8];
            if (p.mask_src && scatter) {
#pragma unroll
              for (int ch = 0; ch < 8; ++ch) {
                mreg[ch] = make_uint4(0u, 0u, 0u, 0u);
                if (drow_of >= 0 && gcol + ch * 8 < p.n_store)
                  mreg[ch] = *reinterpret_cast<const uint4*>(p.mask_src + drow_of * p.ldd + gcol + ch * 8);
              }
            } else if (p.mask_src) {
              // the mask slab arrives through TMA into the slab buffer (same box and swizzle as the output),
              // is copied to registers, and the buffer is then reused for the output
              if (lane == 0) {
                mbar_expect_tx(mbar_m, 4096u);
                tma_load_2d(buf, &p.tm_mask, mbar_m, gcol, row0);
              }
              if (!mbar_wait_bounded(mbar_m, mask_ph, WAIT_LIMIT_NS)) {
                ctl->abort_flag = 1;
                if (p.status) atomicOr(p.status, RB_STATUS_MBAR_TIMEOUT);
              }
              mask_ph ^= 1u;
#pragma unroll
              for (int ch = 0; ch < 8; ++ch)
                mreg[ch] = *reinterpret_cast<const uint4*>(buf + lane * 128 + ((ch ^ (lane & 7)) * 16));
              __syncwarp();
            }
            RB_PROF_T0(warp == 2);
            uint8_t* const slab_row = buf + lane * 128;
            const int swz = lane & 7;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              uint32_t v[32];
              const int nbase = gcol + half * 32;
              if (nbase >= p.n_store) continue;            // these columns do not exist in D: the store clips them
              tmem_ld_32x32(t_addr + (uint32_t)(c + half * 32), v);
              tmem_ld_wait();
              const float* bias = p.bias + nbase;
              const uint4* m = &mreg[half * 4];
              uint4 av[4];
              if (addend) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  av[q] = make_uint4(0u, 0u, 0u, 0u);
                  if (drow_of >= 0 && nbase + q * 8 < p.n_store)
                    av[q] = *reinterpret_cast<const uint4*>(p.add_src + drow_of * p.ldd + nbase + q * 8);
                }
              }
              const int valid = p.n_valid - nbase;
              if (NORM) {
                if (valid >= 32) epilogue_norm<false>(p.relu != 0, addend, v, slab_row, swz, half, bias, p.scale + nbase, m, av, valid);
                else epilogue_norm<true>(p.relu != 0, addend, v, slab_row, swz, half, bias, p.scale + nbase, m, av, valid);
              } else if (valid >= 32) epilogue_kinds<EXT, false>(epi_kind, addend, v, slab_row, swz, half, bias, m, av, valid);
              else epilogue_kinds<EXT, true>(epi_kind, addend, v, slab_row, swz, half, bias, m, av, valid);
            }
            RB_PROF_ADD(warp == 2, 7);
#ifdef RB_GEMM_PROFILE
            const long long prof_t1_ = clock64();
#endif
            if (scatter) {
              // eight lanes write the 128 bytes of a row, four rows at a time
              __syncwarp();
#pragma unroll
              for (int it = 0; it < 8; ++it) {
                const int rr = it * 4 + (lane >> 3), ch = lane & 7;
                const long long dr = __shfl_sync(0xffffffffu, drow_of, rr);
                if (dr >= 0 && gcol + ch * 8 < p.n_store)
                  *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.D) + dr * p.ldd + gcol + ch * 8) =
                      *reinterpret_cast<const uint4*>(buf + rr * 128 + ((ch ^ (rr & 7)) * 16));
              }
              __syncwarp();
              if (lane == 0) tma_store_commit();   // every slab is one group, also an empty one (see the wait above)
              continue;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (band_rows < 32) {
              // ragged band (box mode): the rows after the tile's last belong to other tiles, so the valid rows are
              // copied out by hand, 16 bytes at a time, instead of a 32-row TMA store
              if (lane < band_rows) {
                bf16* drow = reinterpret_cast<bf16*>(p.D) + (long long)(row0 + lane) * p.ldd + gcol;
#pragma unroll
                for (int ch = 0; ch < 8; ++ch)
                  if (gcol + ch * 8 < p.n_store)
                    *reinterpret_cast<uint4*>(drow + ch * 8) =
                        *reinterpret_cast<const uint4*>(buf + lane * 128 + ((ch ^ (lane & 7)) * 16));
              }
              __syncwarp();
              if (lane == 0) tma_store_commit();
            } else if (lane == 0) {
              if (row0 < p.M) tma_store_2d(&p.tm_d, buf, gcol, row0);
              tma_store_commit();
            }
#ifdef RB_GEMM_PROFILE
            if (warp == 2 && blockIdx.x == 3 && lane == 0)
              atomicAdd(&g_role_cycles[6], (unsigned long long)(clock64() - prof_t1_));
#endif
          }
          continue;
        }
        for (int c = ((col_half + j) & 1) * 32; c < p.bn; c += 64) {
          uint32_t v[32];
          tmem_ld_32x32(t_addr + (uint32_t)c, v);
          tmem_ld_wait();
          if (!tail && c >= col_limit) continue;
          int gcol = tail ? c : col0 + c;
          if (!tail && p.wgrad && p.wg_taps > 1) {
            const int t = c / p.wg_cw, cc = c - t * p.wg_cw;
            const int tap = tn * p.wg_taps + t;
            if (tap >= p.wg_ntaps || cc >= p.wg_cpad) continue;
            gcol = tap * p.wg_cpad + cc;
          }
          // fp32 output: 32-column chunk -> swizzled slab buffer -> one TMA store (overwrite) or TMA reduce-add
          // (accumulate / split-K) per warp, instead of eight 16-byte red instructions per thread
          if (lane == 0) tma_store_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 o = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((q ^ (lane & 7)) * 16)) = o;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && (tail || row0 < p.M)) {
            // a part of a cut item adds into its rows of the workspace; everything else goes to D
            if (tail) tma_reduce_add_2d(&p.tm_ws, stg, gcol, (it.tail * mt + j) * BM + lane_base);
            else if (p.epi == EPI_F32_STORE) tma_store_2d(&p.tm_d, stg, gcol, row0);
            else tma_reduce_add_2d(&p.tm_d, stg, gcol, row0);
            tma_store_commit();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        // the accumulators of both CTAs of a pair are refilled by the leader: it waits for both epilogues
        if (pair) mbar_arrive_cluster(mapa_shared(smem_u32(&ctl->acc_empty[acc]), 0u));
        else mbar_arrive(&ctl->acc_empty[acc]);
      }
      if (++acc == p.acc_bufs) { acc = 0; acc_ph ^= 1u; }
    }
    if (lane == 0) tma_store_wait_all<0>();   // every output store has completed before the CTA exits
  }

  tc_fence_before();
  __syncthreads();
#ifdef RB_GEMM_PROFILE
  if (blockIdx.x == 3 && threadIdx.x == 0) atomicAdd(&g_role_cycles[4], (unsigned long long)(clock64() - t_kernel0));
#endif
  // a pair frees its TMEM together, after both epilogues have read it and nothing signals a peer's barrier any more
  if (pair) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    if (pair) tmem_dealloc2(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

#include "wgrad_rows.cuh"

// =============================== host side ===============================

typedef void (*Kernel)(GemmTcParams);
static const Kernel KERNELS[] = {   // without and with CTA pairs
    gemm_tc_kernel<false, false, false, false, false>, gemm_tc_kernel<true, false, false, false, false>,
    gemm_tc_kernel<false, true, false, false, false>,  gemm_tc_kernel<true, true, false, false, false>,
    gemm_tc_kernel<false, true, true, false, false>,   gemm_tc_kernel<true, true, true, false, false>,
    gemm_tc_kernel<false, true, false, true, false>,   gemm_tc_kernel<true, true, false, true, false>,
    gemm_tc_kernel<false, true, true, true, false>,    gemm_tc_kernel<true, true, true, true, false>,
    gemm_tc_kernel<false, false, false, false, true>};
constexpr int LEAN_KERNEL = 10;
static void (*const PHASES_KERNEL)(GemmPhasesParams) = gemm_tc_kernel<false, true, false, false, false, true>;
static int tile_bytes(const GemmTcParams& p) { return p.lean ? LEAN_TILE_BYTES : TILE_SMEM_BYTES; }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const int*, const int*, cuuint32_t, cuuint32_t,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn g_encode_tiled = nullptr;
static EncodeIm2colFn g_encode_im2col = nullptr;
static int g_num_sms = 0;
static int g_driver_version = 0;
static int g_pair_clusters = 0;   // clusters of two CTAs of the kernel that the device runs at once (0 = none)

static void options_from_env();

static int ensure_driver_entry() {
  options_from_env();
  if (g_encode_tiled && g_encode_im2col) return 0;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || !fn)
    return -1;
  g_encode_tiled = reinterpret_cast<EncodeTiledFn>(fn);
  fn = nullptr;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &qres) != cudaSuccess || !fn)
    return -1;
  g_encode_im2col = reinterpret_cast<EncodeIm2colFn>(fn);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDriverGetVersion(&g_driver_version);
  for (auto kern : KERNELS)
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES) != cudaSuccess) return -2;
  if (cudaFuncSetAttribute(wgrad_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES) != cudaSuccess) return -2;
  if (cudaFuncSetAttribute(PHASES_KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES) != cudaSuccess) return -2;
  {   // how many CTA pairs fit at once: the persistent loop of pair mode runs exactly that many clusters
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(g_num_sms / 2 * 2));
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = GEMM_SMEM_BYTES;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, gemm_tc_kernel<true, true, true, false, false>, &cfg) != cudaSuccess) nc = 0;
    cudaGetLastError();   // a refused query must not be taken for a failed launch later
    g_pair_clusters = nc > g_num_sms / 2 ? g_num_sms / 2 : nc;
  }
  return 0;
}

// 2-D bf16 map: dims {inner, outer}, outer pitch in elements, box {bi, bo}.
static int make_map_2d(CUtensorMap* m, const void* ptr, uint64_t inner, uint64_t outer, uint64_t pitch_elems,
                       uint32_t bi, uint32_t bo, CUtensorMapSwizzle sw) {
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {pitch_elems * 2};
  cuuint32_t box[2] = {bi, bo};
  cuuint32_t es[2] = {1, 1};
  CUresult r = g_encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(100 + (int)r);
}
static int make_map_3d(CUtensorMap* m, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t pitch1,
                       uint64_t pitch2, uint32_t b0, uint32_t b1, uint32_t b2, CUtensorMapSwizzle sw) {
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {pitch1 * 2, pitch2 * 2};
  cuuint32_t box[3] = {b0, b1, b2};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = g_encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(100 + (int)r);
}
// NHWC bf16 im2col map. The base pixel ranges over [lower, dim + upper) per spatial axis;
// a load fetches `pixels` base pixels (w fastest, then h, then n) x `channels` channels.
static int make_map_im2col(CUtensorMap* m, const void* ptr, int N, int H, int W, int C, int lower_h, int lower_w,
                           int upper_h, int upper_w, int stride, uint32_t channels, uint32_t pixels,
                           CUtensorMapSwizzle sw) {
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
  cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)C * W * 2, (cuuint64_t)C * W * H * 2};
  int lower[2] = {lower_w, lower_h};
  int upper[2] = {upper_w, upper_h};
  cuuint32_t es[4] = {1, (cuuint32_t)stride, (cuuint32_t)stride, 1};
  CUresult r = g_encode_im2col(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, lower,
                               upper, channels, pixels, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return -(200 + (int)r);
  // Drivers up to 13.1 mis-handle im2col maps of tensors smaller than 128 KiB unless bit 21 of the
  // second descriptor word is cleared (same adjustment CUTLASS applies to its im2col descriptors).
  if (g_driver_version <= 13010 && (size_t)N * H * W * C * 2 < 131072) {
    reinterpret_cast<uint64_t*>(m)[1] &= ~(1ull << 21);
  }
  return 0;
}

// Output map of the bf16 epilogue: columns [0, n_store) x rows [0, M), 64 x 32 boxes, 128-byte swizzle.
static int make_map_out(CUtensorMap* m, void* D, int n_store, int M, long long ldd) {
  return make_map_2d(m, D, (uint64_t)n_store, (uint64_t)M, (uint64_t)ldd, 64, 32, CU_TENSOR_MAP_SWIZZLE_128B);
}

// fp32 output map: 32-column x 32-row boxes (128-byte rows), 128-byte swizzle; used by TMA store / reduce-add.
static int make_map_out_f32(CUtensorMap* m, void* D, long long n_cols, int M, long long ldd) {
  cuuint64_t dims[2] = {(cuuint64_t)n_cols, (cuuint64_t)M};
  cuuint64_t strides[1] = {(cuuint64_t)ldd * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t es[2] = {1, 1};
  CUresult r = g_encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, D, dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(300 + (int)r);
}

// 4-D bf16 tiled map over an NHWC tensor: dims {C, W, H, N}, pixel pitch `ld` elements, box {bc, bw, bh, 1}.
static int make_map_nhwc(CUtensorMap* m, const void* ptr, uint64_t C, uint64_t W, uint64_t H, uint64_t N, uint64_t ld,
                         uint32_t bc, uint32_t bw, uint32_t bh, CUtensorMapSwizzle sw) {
  cuuint64_t dims[4] = {C, W, H, N};
  cuuint64_t strides[3] = {ld * 2, ld * W * 2, ld * W * H * 2};
  cuuint32_t box[4] = {bc, bw, bh, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = g_encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(400 + (int)r);
}

// ---- options ----------------------------------------------------------------------------------------------------
// Switches of the planner. Their initial values come from the environment (RB_GEMM_*), read once when the library
// is first used; afterwards they change only through rb_gemm_set_option (tests, experiments).
struct GemmOptions {
  int force_mt = 0;          // RB_GEMM_FORCE_MT: 1 | 2, flat mode up to 4, sub-tiles per item (0 = planner's choice)
  int force_resident = -1;   // RB_GEMM_FORCE_RESIDENT: 0 | 1
  int force_halo = -1;       // RB_GEMM_FORCE_HALO: whole input rows for all taps (flat mode): 0 = never, 1 = whenever feasible
  int force_taps = 0;        // RB_GEMM_FORCE_TAPS: filter taps per weight-grad tile
  int force_tail = -1;       // RB_GEMM_FORCE_TAIL: 0 = never cut the last wave, 1 = whenever feasible
  int force_wide = -1;       // RB_GEMM_FORCE_WIDE: 0 = tiles of at most 256 columns, 1 = one wide tile when N <= 512
  int force_box = -1;        // RB_GEMM_FORCE_BOX: 0 = never load A as tap-shifted boxes, 1 = whenever feasible
  int force_pair = -1;       // RB_GEMM_FORCE_PAIR: 0 = never run as CTA pairs (cta_group::2), 1 = whenever feasible
  int pdl = 2;               // RB_GEMM_PDL: programmatic stream serialization (blocks become resident while the kernel
                             // before them finishes; see launch.cuh): 0 = off, 1 = this kernel only, 2 = every kernel
                             // of a step. Beside exchange kernels on other streams use at most 1: the waiting blocks
                             // of elementwise kernels fill the SMs' thread slots and the exchange kernels starve.
  int bk32 = 0;              // RB_GEMM_BK32: keep 32-channel chunks for channel counts such as 96
  int bn_cap = 256;          // RB_GEMM_BN_CAP: upper bound on the tile width chosen by the planner
  int a_split = 1;           // RB_GEMM_A_SPLIT / RB_GEMM_B_SPLIT: TMA boxes per K-major tile
  int b_split = 1;
  int force_rows = -1;       // RB_GEMM_FORCE_ROWS: weight-gradients from whole rows: 0 = never, n = the n-th plan wherever there is one
  int autotune = 1;          // RB_GEMM_AUTOTUNE: 0 = cost model only, even in tuning mode
  int deterministic = 0;     // RB_GEMM_DETERMINISTIC: 1 = no launch lets several CTAs add into the same output element
                             // (no reduction split, no tail cut), so results are bit-identical from run to run, and the
                             // order of additions does not depend on what is measured as the fastest (no flat mode)
};
static GemmOptions g_opt;
static std::once_flag g_opt_once;
static int g_tune_mode = 0;   // set by rb_gemm_tune_mode: launches of unseen shapes time their candidates

static int* option_slot(const char* name) {
  struct { const char* name; int* slot; } table[] = {
      {"force_mt", &g_opt.force_mt}, {"force_resident", &g_opt.force_resident}, {"force_halo", &g_opt.force_halo},
      {"force_taps", &g_opt.force_taps}, {"force_tail", &g_opt.force_tail}, {"force_wide", &g_opt.force_wide},
      {"force_box", &g_opt.force_box}, {"force_pair", &g_opt.force_pair}, {"force_rows", &g_opt.force_rows}, {"pdl", &g_opt.pdl},
      {"bk32", &g_opt.bk32}, {"bn_cap", &g_opt.bn_cap}, {"a_split", &g_opt.a_split}, {"b_split", &g_opt.b_split},
      {"autotune", &g_opt.autotune}, {"deterministic", &g_opt.deterministic}};
  for (auto& t : table)
    if (strcmp(t.name, name) == 0) return t.slot;
  return nullptr;
}
static void options_from_env() {
  std::call_once(g_opt_once, [] {
    const char* names[] = {"force_mt", "force_resident", "force_halo", "force_taps", "force_tail", "force_wide", "force_box",
                           "force_pair", "force_rows", "pdl", "bk32", "bn_cap", "a_split", "b_split", "autotune", "deterministic"};
    for (const char* n : names) {
      char env[64] = "RB_GEMM_";
      size_t k = strlen(env);
      for (const char* c = n; *c && k + 1 < sizeof(env); ++c) env[k++] = (char)toupper((unsigned char)*c);
      env[k] = 0;
      const char* e = getenv(env);
      if (e) *option_slot(n) = atoi(e);
    }
  });
}

int pdl_enabled() {
  options_from_env();
  return g_opt.pdl >= 2 ? 1 : 0;
}

// ---- tile-shape planning -----------------------------------------------------------------------------------
// Cost model in "rows": the kernel is bound by the 128-byte rows it fills into shared memory per k-block
// (see the header comment), so an item costs about k-blocks x (rows of A + rows of B) plus its epilogue, and a
// launch costs rounds x item (persistent CTAs, one per SM). The planner picks sub-tiles per item (mt),
// the reduction split, B residency and whether the last wave is cut along the reduction to minimise that.
struct Plan {
  int mt, split, resident, tail;   // tail: parts per cut item of the last wave (0 = no cut)
  double cost;
  int pair = 0;                    // run as CTA pairs (never with resident B or a tail cut)
};

// CTA pairs need K-major operands loaded by plain or im2col TMA, a tile of at most 256 columns whose halves are whole
// boxes of the B map (the map's box is bn / b_split rows, so b_split must be even), and more than one pair's rows.
static bool pair_ok(const GemmTcParams& p) {
  if (g_opt.force_pair == 0 || g_pair_clusters <= 0) return false;
  if (p.a_mode != A_TILED_K && p.a_mode != A_IM2COL_K && p.a_mode != A_FLAT_K) return false;
  if (p.b_mode == B_DGRAD_MN) {
    if (p.bn > 256 || p.bn % 128 != 0) return false;   // each CTA loads whole 64-column blocks
    return p.M > 2 * BM;
  }
  if (p.b_mode != B_TILED_K && p.b_mode != B_TILED_K3) return false;
  if (p.bn > 256 || p.bn % 16 != 0 || p.b_split < 2 || p.b_split % 2 != 0) return false;
  return p.M > 2 * BM;
}
// Boxes per tile for K-major operands (each box is issued by its own lane). A box must keep whole 8-row swizzle
// atoms, start on a 1024-byte boundary in shared memory and have at most 256 rows.
static int pick_box_split(int sp, int rows, int bk) {
  if (sp < 1) sp = 1;
  while (rows / sp > 256) sp <<= 1;
  while (sp > 1 && (rows % sp != 0 || (rows / sp) % 8 != 0 || ((rows / sp) * bk * 2) % 1024 != 0)) sp >>= 1;
  return sp < 1 ? 1 : sp;
}

// Boxes per B tile such that half a tile is a whole number of boxes whenever the shape allows pairs.
static int pairable_b_split(int bn, int bk) {
  int sp = pick_box_split(g_opt.b_split, bn, bk);
  if (g_opt.force_pair != 0 && sp % 2 != 0 && bn <= 256) {
    const int sp2 = pick_box_split(sp * 2, bn, bk);
    if (sp2 % 2 == 0) sp = sp2;
  }
  return sp;
}

static bool split_ok(int s, int num_kb) { return s == 1 || (s - 1) * ((num_kb + s - 1) / s) < num_kb; }

static int acc_stride_for(int bn) { return bn > 256 ? 512 : (bn > 128 ? 256 : 128); }

// Work items along M for `mt` sub-tiles per item (box mode: whole output rows per sub-tile, per image).
static int m_items_of(const GemmTcParams& p, int mt) {
  if (p.a_mode == A_BOX_K) {
    const int groups = (p.cv_P + mt * p.bx_rows - 1) / (mt * p.bx_rows);
    return (p.M / (p.cv_P * p.cv_Q)) * groups;
  }
  const int units = p.a_mode == A_FLAT_K ? (p.fl_units + mt - 1) / mt : (p.M + BM * mt - 1) / (BM * mt);
  return p.pair ? (units + 1) / 2 : units;
}

// Parts per cut item for `items` work items on `sms` SMs (0 = cutting does not pay or is not possible): the last
// wave must be at most half full, every SM gets at most one part, a part keeps at least four k-blocks. A launch with
// fewer items than half the SMs (small batches, 7 x 7 layers) is one such wave: all of its items are cut.
static int tail_parts(long long items, int sms, int num_kb) {
  const int rem = (int)(items % sms);
  if (rem == 0 || rem * 2 > sms) return 0;
  int s = sms / rem;
  if (s > num_kb / 4) s = num_kb / 4;
  if (s > 16) s = 16;
  while (s > 1 && !split_ok(s, num_kb)) --s;
  return s >= 2 ? s : 0;
}

// ---- flat mode -----------------------------------------------------------------------------------------------
// A stride-1 convolution over rows of positions: every image row is fl_pitch positions long (the output row plus the zero
// columns that the filter reaches, those at a row's end shared with the next row's beginning), every image fl_hp rows
// (likewise), and all of them lie one after the other. Output position f then reads positions f + r * pitch + s, for every
// filter tap (r, s) at the same distance, so one copy of the rows in shared memory serves all R * S taps of a channel chunk:
// a tap is an offset in the A descriptor. What lies on zero columns and rows is computed and not stored (19 x 19: 11 %,
// 13 x 13: 16 %, 32 x 32: 6 %, 56 x 56: 4 %).
// Why: loaded tap by tap, a 128-row tile takes R * S x 16 KB per chunk from the L2, which delivers ~41 bytes per cycle and
// SM: 128 -> 128 channels at two sub-tiles per item ask for 94, so the tensor pipe was 40 % busy; this asks for 25 to 41.
// 96 -> 256 on 128 x 27 x 27, 5 x 5: data-gradient 115 -> 89 us; 256 -> 384 on 128 x 13 x 13: 42 -> 35; 16 -> 16 on
// 128 x 32 x 32: 19.6 -> 16.2; 64 -> 128 on 64 x 128 x 128: data-gradient 205 -> 187.
// Counted on 32 images of the first of these: 604 -> 198 MB into shared memory, 62 -> 55 us.
// Sub-tiles start 128 positions apart, or, on rows of at least 128 positions with at most 128 outputs, one row apart.
// Rows of 113 to 127 positions are made 128 long for that: 3 x 3, 64 -> 64 / 128 / 256, 16 images of 112 x 112, as they are
// 44 / 58 / 107 us, 128 long 34 / 41 / 59 (tap by tap: 34 / 36 / 54); from 124 on they do not fit as they are. Shorter rows
// would gain too (111: 44 / 47 / 81 against 32 / 38 / 56; 99: 29 / 39 / 60 against 30 / 37 / 52), but there the tap-by-tap plans
// are as fast or faster (32 / 38 / 54; 29 / 32 / 48) and the measurement takes those.
static bool flat_geom(GemmTcParams& p, int N, int H, int W, int R, int S, int pad_h, int pad_w) {
  const int P = p.cv_P, Q = p.cv_Q;
  const int share_w = std::max(0, std::min({pad_w, S - 1, Q + S - 1 - pad_w - W}));
  const int share_h = std::max(0, std::min({pad_h, R - 1, P + R - 1 - pad_h - H}));
  p.fl_pitch = Q + S - 1 - share_w;
  if (p.bk == 32) p.fl_pitch = (p.fl_pitch + 1) / 2 * 2;   // rows of 64-byte positions have to start on 128 bytes
  if (p.fl_pitch > 112 && p.fl_pitch < BM) p.fl_pitch = BM;   // a sub-tile per row: whole-row items need no rows in between
  p.fl_hp = P + R - 1 - share_h;
  const bool by_rows = p.fl_pitch >= BM && Q <= BM;
  p.fl_step = by_rows ? p.fl_pitch : BM;
  const long long rows = (long long)N * p.fl_hp - (p.fl_hp - P);
  const long long positions = rows * p.fl_pitch;
  if (p.fl_pitch > 256 || pad_h < 0 || pad_w < 0 || positions > (1ll << 30)) return false;   // a box has at most 256 columns
  p.fl_units = (int)(by_rows ? rows : (positions + BM - 1) / BM);
  p.fl_R = R;
  p.fl_pad_h = pad_h;
  p.fl_pad_w = pad_w;
  return true;
}

static int gcd_of(int a, int b) { return b == 0 ? a : gcd_of(b, a % b); }

// Input rows and bytes of an A stage for `mt` sub-tiles per item.
static void flat_stage(GemmTcParams& p, int mt) {
  const int pitch = p.fl_pitch, row_bytes = p.bk * 2;
  const bool by_rows = p.fl_step != BM, shared = pitch < p.cv_Q + p.cv_S - 1;
  const int off_max = by_rows ? 0 : pitch - gcd_of(pitch, mt * p.fl_step);     // column of an item's first position
  const int last = off_max + (mt - 1) * p.fl_step + (by_rows ? p.cv_Q : BM) - 1 + (shared ? p.cv_S - 1 : 0);
  p.fl_rows = last / pitch + p.fl_R;
  p.fl_lead = off_max;
  const int loaded = p.fl_lead + p.fl_rows * pitch;
  const int read = p.fl_lead + (mt - 1) * p.fl_step + BM + (p.fl_R - 1) * pitch + p.cv_S - 1;
  p.fl_a_bytes = (std::max(loaded, read) * row_bytes + 1023) / 1024 * 1024;
}

// Fill in what follows from a plan; returns the grid size, or 0 when the plan does not fit.
static int apply_flat_plan(GemmTcParams& p, const Plan& pl) {
  if (pl.tail || pl.split != 1 || p.bn > 256 || pl.mt < 1 || pl.mt > 4) return 0;
  if (p.fl_units < pl.mt) return 0;
  p.mt = pl.mt;
  p.split_k = 1;
  p.b_resident = pl.resident;
  if (pl.pair) {
    if (!pair_ok(p) || pl.resident || p.fl_units <= pl.mt) return 0;
    p.pair = 1;
    p.bn_load = p.bn / 2;
    if (p.b_mode != B_DGRAD_MN) p.b_split = p.b_split / 2;
  }
  p.acc_stride = 32;
  while (p.acc_stride < p.bn) p.acc_stride *= 2;
  if (p.mt * p.acc_stride > 512) return 0;
  p.acc_bufs = 2 * p.mt * p.acc_stride <= 512 ? 2 : 1;
  flat_stage(p, p.mt);
  const int b_bytes = p.bn_load * p.bk * 2;
  p.fl_a_stages = 2;
  const int room = TILE_SMEM_BYTES - p.fl_a_stages * p.fl_a_bytes;
  if (p.b_resident) {
    if (p.n_tiles != 1 || room < p.num_kb * b_bytes) return 0;
    p.stages = 2;                       // unused
    if (room >= p.num_kb * b_bytes + p.fl_a_bytes) p.fl_a_stages = 3;
  } else {
    if (room < 2 * b_bytes) return 0;
    p.stages = std::min(room / b_bytes, MAX_STAGES);
  }
  p.epi_bufs = 1;
  p.tail_items = p.tail_split = 0;
  const long long work = (long long)m_items_of(p, p.mt) * p.n_tiles;
  if (p.pair) return 2 * (int)std::min<long long>(work, g_pair_clusters);
  return (int)std::min<long long>(work, g_num_sms);
}

// Cycles of a launch, to rank plans by: MMA time (a 128 x N x 16 step takes N / 2 cycles, or what its operands take at 128
// bytes per cycle from shared memory), L2 delivery (41 bytes per cycle and SM), ~150 cycles per k-block for the issuing warp,
// an epilogue of ~900 cycles per 32 x 64 slab and warp, overlapped when there are two accumulator sets.
static double flat_cost(const GemmTcParams& p, int grid) {
  const double steps = (double)p.num_kb * (p.bk / 16) * p.mt;
  const double step = std::max(p.bn / 2.0, 32.0 + (p.pair ? p.bn / 8.0 : p.bn / 4.0));
  const double bytes = (double)p.cv_cchunks * p.fl_rows * p.fl_pitch * p.bk * 2 +
                       (p.b_resident ? 0.0 : (double)p.num_kb * p.bn_load * p.bk * 2);
  const double loop = std::max(steps * step, bytes / 41.0) + p.num_kb * (p.b_resident ? 60.0 : 150.0);
  const double epi = p.mt * ((p.bn + 63) / 64) * 0.5 * 900.0;
  const double item = p.acc_bufs == 2 ? std::max(loop, epi) + 200.0 : loop + epi + 600.0;
  const long long work = (long long)m_items_of(p, p.mt) * p.n_tiles;
  const long long ctas = p.pair ? grid / 2 : grid;
  return (double)((work + ctas - 1) / ctas) * item + (p.acc_bufs == 2 ? epi : 0.0);
}

// The plans that fit, best first by flat_cost; returns how many.
static int flat_plans(const GemmTcParams& p, Plan* out, int max_plans) {
  int n = 0;
  for (int pass = 0; pass < 2 && n == 0; ++pass)   // the force options restrict the search (ignored when infeasible)
  for (int mt = 1; mt <= 4; ++mt) {
    if (pass == 0 && g_opt.force_mt && mt != g_opt.force_mt) continue;
    for (int kind = 0; kind < 3; ++kind) {
      Plan pl{mt, 1, kind == 1, 0, 0.0};
      pl.pair = kind == 2;
      if (pass == 0 && g_opt.force_resident >= 0 && pl.resident != g_opt.force_resident) continue;
      GemmTcParams q = p;
      const int grid = apply_flat_plan(q, pl);
      if (grid <= 0) continue;
      pl.cost = flat_cost(q, grid);
      int at = std::min(n, max_plans);
      while (at > 0 && out[at - 1].cost > pl.cost) --at;
      if (at == max_plans) continue;
      n = std::min(n + 1, max_plans);
      for (int i = n - 1; i > at; --i) out[i] = out[i - 1];
      out[at] = pl;
    }
  }
  return n;
}

static Plan plan_shape(const GemmTcParams& p, bool allow_split, int fixed_split, bool b_is_weights) {
  if (p.a_mode == A_FLAT_K) {
    Plan best{1, 1, 0, 0, 1e300};
    flat_plans(p, &best, 1);
    return best;
  }
  if (g_opt.deterministic) {   // one CTA per output tile, its k-blocks in order
    allow_split = false;
    fixed_split = 1;
  }
  const int a_bytes = BM * p.bk * 2, b_bytes = p.bn_load * p.bk * 2;
  const double epi_elem = (p.epi == EPI_BF16) ? 1.2 : 1.6;
  Plan best{1, 1, 0, 0, 1e300};
  // the force options restrict the search (ignored when infeasible)
  const int force_mt = g_opt.force_mt, force_res = g_opt.force_resident;
  for (int pass = 0; pass < 2 && best.cost >= 1e299; ++pass)
  for (int mt = 1; mt <= 2; ++mt) {
    if (pass == 0 && force_mt && mt != force_mt) continue;
    if (mt == 2 && (p.M <= BM || p.bn > 256)) continue;
    if (mt == 2 && p.a_mode == A_BOX_K && p.cv_P <= p.bx_rows) continue;
    const int acc_stride = acc_stride_for(p.bn);
    const int acc_bufs = (2 * mt * acc_stride <= 512) ? 2 : 1;
    const int m_items = m_items_of(p, mt);
    const long long tiles = (long long)m_items * p.n_tiles;
    // up to one part per SM (a layer with a single output tile, e.g. the weight-grad of a 1 x 1 convolution on 96
    // channels, would otherwise leave SMs idle), each part at least eight k-blocks long
    const int split_cap = g_num_sms > 0 ? g_num_sms : 148;
    const int max_split = allow_split ? (p.num_kb / 8 > split_cap ? split_cap : (p.num_kb / 8 < 1 ? 1 : p.num_kb / 8)) : 1;
    for (int s = (fixed_split > 0 ? fixed_split : 1); s <= (fixed_split > 0 ? fixed_split : max_split); ++s) {
      if (!split_ok(s, p.num_kb)) continue;
      for (int res = 0; res <= 1; ++res) {
        if (pass == 0 && force_res >= 0 && res != force_res) continue;
        const long long panel = (long long)p.num_kb * b_bytes;
        if (res) {
          if (!b_is_weights || p.n_tiles != 1 || s != 1 || panel > 112 * 1024) continue;
          if ((tile_bytes(p) - panel) / (mt * a_bytes) < 3) continue;
        } else if (tile_bytes(p) / (mt * a_bytes + b_bytes) < 2) {
          continue;
        }
        const int kbs = (p.num_kb + s - 1) / s;
        const double rows_kb = mt * BM + (res ? 0 : p.bn_load);
        const double mainloop = kbs * rows_kb * (p.bk / 64.0);
        const double epi = mt * p.bn * epi_elem;
        const double item = acc_bufs == 2 ? (mainloop > epi ? mainloop : epi) + 0.15 * epi : mainloop + epi;
        for (int tail = 0; tail <= 1; ++tail) {
          int parts = 0;
          if (tail) {
            if (p.epi != EPI_BF16 || s != 1 || !p.ws || g_opt.force_tail == 0 || g_opt.deterministic) continue;
            parts = tail_parts(tiles, g_num_sms, p.num_kb);
            if (parts == 0) continue;
            const long long need = (tiles % g_num_sms) * mt * BM * (long long)p.bn * 4;
            if (need > p.ws_bytes) continue;
          } else if (pass == 0 && g_opt.force_tail == 1 && p.epi == EPI_BF16 && s == 1 && p.ws &&
                     tail_parts(tiles, g_num_sms, p.num_kb) > 0) {
            continue;
          }
          double rounds = (double)((tiles * s + g_num_sms - 1) / g_num_sms);
          if (parts) rounds = (double)(tiles / g_num_sms) + 1.0 / parts + 0.1;   // + the fix-up pass
          const double cost = rounds * item + (res ? (double)p.num_kb * p.bn_load * (p.bk / 64.0) : 0.0);
          if (cost < best.cost * 0.97) best = Plan{mt, s, res, parts, cost};
        }
      }
    }
  }
  return best;
}

// Fill in what follows from a plan; returns the grid size, or 0 when the plan does not fit.
static int apply_plan(GemmTcParams& p, const Plan& pl) {
  if (p.a_mode == A_FLAT_K) return apply_flat_plan(p, pl);
  if (pl.mt < 1 || pl.mt > 2) return 0;   // what issue_item is built for
  p.mt = pl.mt;
  p.split_k = pl.split;
  p.b_resident = pl.resident;
  if (pl.pair) {
    if (!pair_ok(p) || pl.resident || pl.tail || p.M <= BM * pl.mt) return 0;
    p.pair = 1;
    p.bn_load = p.bn / 2;      // rows of B per CTA
    if (p.b_mode != B_DGRAD_MN) p.b_split = p.b_split / 2;
  }
  p.acc_stride = acc_stride_for(p.bn);
  p.acc_bufs = (2 * p.mt * p.acc_stride <= 512) ? 2 : 1;
  if (p.mt * p.acc_stride > 512) return 0;
  const int a_bytes = BM * p.bk * 2, b_bytes = p.bn_load * p.bk * 2;
  const int panel = p.b_resident ? p.num_kb * b_bytes : 0;
  const int stage = p.mt * a_bytes + (p.b_resident ? 0 : b_bytes);
  if (panel >= tile_bytes(p)) return 0;
  p.stages = (tile_bytes(p) - panel) / stage;
  // Two slab buffers per epilogue warp where the main loop is too short to hide the epilogue and the stages that are left
  // still cover a whole item or are four.
  p.epi_bufs = 1;
  if (p.epi == EPI_BF16 && p.num_kb <= 4 && TILE_SMEM_BYTES - STAGING_BYTES > panel) {
    const int left = (TILE_SMEM_BYTES - STAGING_BYTES - panel) / stage;
    if (left >= 4 || (left >= 2 && left >= p.num_kb)) {
      p.epi_bufs = 2;
      p.stages = left;
    }
  }
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  if (p.stages < 2) return 0;
  if (p.mt == 2 && p.M <= BM) return 0;
  if (p.mt == 2 && p.a_mode == A_BOX_K && p.cv_P <= p.bx_rows) return 0;
  const int m_items = m_items_of(p, p.mt);
  const long long items = (long long)m_items * p.n_tiles;
  p.tail_items = 0;
  p.tail_split = 0;
  long long work = items * p.split_k;
  if (pl.tail > 0) {
    if (p.epi != EPI_BF16 || p.split_k != 1 || !p.ws) return 0;
    p.tail_items = (int)(items % g_num_sms);
    p.tail_split = pl.tail;
    const long long rows = (long long)p.tail_items * p.mt * BM;
    if (p.tail_items == 0 || rows * p.bn * 4 > p.ws_bytes || !split_ok(pl.tail, p.num_kb)) return 0;
    cuuint64_t dims[2] = {(cuuint64_t)p.bn, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)p.bn * 4};
    cuuint32_t box[2] = {32, 32};
    cuuint32_t es[2] = {1, 1};
    if (g_encode_tiled(&p.tm_ws, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.ws, dims, strides, box, es,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return 0;
    work = items - p.tail_items + (long long)p.tail_items * p.tail_split;
  }
  if (p.pair) return 2 * (int)(work < g_pair_clusters ? work : g_pair_clusters);
  return work < g_num_sms ? (int)work : g_num_sms;
}

// Epilogue of the cut items: D = act(workspace + bias), masked, as bf16; the workspace rows are cleared again so
// that the next launch that uses the workspace finds zeros. One thread per 8 columns.
struct TailFixArgs {
  float* ws;
  __nv_bfloat16* D;
  const float* bias;
  const __nv_bfloat16* mask;
  long long ldd;
  const __nv_bfloat16* add;
  const float* scale;
  int M, bn, rows_per_item, m_items, direct, tail_items, n_valid, n_store, relu;
  int sc_stride, sc_a, sc_b, sc_H, sc_W;   // see GemmTcParams
  int box, P, Q, bx_rows, bx_groups, mt;   // box mode: rows of a sub-tile are whole output rows of one image
};
__global__ void tail_fix_kernel(const TailFixArgs a) {
  pdl_prolog();
  const int gpr = a.bn / 8;
  const long long groups = (long long)a.tail_items * a.rows_per_item * gpr;
  const float act_lo = a.relu ? 0.f : -INFINITY;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < groups;
       g += (long long)gridDim.x * blockDim.x) {
    const int c8 = (int)(g % gpr);
    const long long wr = g / gpr;                    // row of the workspace
    const int ti = (int)(wr / a.rows_per_item);
    const int r = (int)(wr - (long long)ti * a.rows_per_item);
    const int rem = a.direct + ti;
    const int tn = rem / a.m_items, tm = rem - tn * a.m_items;
    long long row = (long long)tm * a.rows_per_item + r;
    bool live = true;
    if (a.box) {
      const int j = r / BM, i = r - j * BM;
      const int n_img = tm / a.bx_groups;
      const int p_sub = ((tm - n_img * a.bx_groups) * a.mt + j) * a.bx_rows;
      live = i < max(0, min(a.bx_rows, a.P - p_sub)) * a.Q;
      row = ((long long)n_img * a.P + p_sub) * a.Q + i;
    }
    const int col = tn * a.bn + c8 * 8;
    float4* src = reinterpret_cast<float4*>(a.ws + wr * a.bn + c8 * 8);
    const float4 v0 = src[0], v1 = src[1];
    src[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    src[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!live || row >= a.M || col >= a.n_store) continue;
    if (a.sc_stride) row = scatter_row((int)row, a.P, a.Q, a.sc_stride, a.sc_a, a.sc_b, a.sc_H, a.sc_W);
    float extra[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (a.add) load8(a.add + row * a.ldd + col, extra);
    float f[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int n = col + e;
      if (a.scale && n < a.n_valid) f[e] *= __ldg(a.scale + n);
      f[e] = n < a.n_valid ? fmaxf(f[e] + (a.bias ? __ldg(a.bias + n) : 0.f) + extra[e], act_lo) : 0.f;
    }
    if (a.mask) {
      float m[8];
      load8(a.mask + row * a.ldd + col, m);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (!(m[e] > 0.f)) f[e] = 0.f;
    }
    store8(a.D + row * a.ldd + col, f);
  }
}

// One output phase that no filter tap reaches: mask(add) or zeros. One thread per 8 channels.
__global__ void fill_phase_kernel(const __nv_bfloat16* add, const __nv_bfloat16* __restrict__ mask, __nv_bfloat16* dx,
                                  long long groups, int P, int Q, int stride, int a, int b, int H, int W, int Cp) {
  pdl_prolog();
  const int cg = Cp / 8;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < groups; g += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(g / cg), c = (int)(g - (long long)m * cg) * 8;
    const long long o = scatter_row(m, P, Q, stride, a, b, H, W) * Cp + c;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (add) load8(add + o, f);
    if (mask) {
      float k[8];
      load8(mask + o, k);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (!(k[e] > 0.f)) f[e] = 0.f;
    }
    store8(dx + o, f);
  }
}
static int fill_phase(const __nv_bfloat16* add, const __nv_bfloat16* mask, __nv_bfloat16* dx, int N, int P, int Q, int stride,
                      int a, int b, int H, int W, int Cp, cudaStream_t stream) {
  const long long groups = (long long)N * P * Q * (Cp / 8);
  long long blocks = (groups + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  launch_pdl(fill_phase_kernel, (int)blocks, 256, 0, stream, add, mask, dx, groups, P, Q, stride, a, b, H, W, Cp);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// What the most recent launch of this process used (for benchmarks and tests; not synchronised between threads):
// {sub-tiles per item, reduction split, resident B, tail parts, CTA pairs, tile width, A load mode, stages, grid}.
static int g_last_launch[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
static int g_last_cuda_error = 0;   // what the runtime answered to the last launch that failed

static int run_plan(GemmTcParams p, const Plan& pl, cudaStream_t stream) {
  const int grid = apply_plan(p, pl);
  if (grid <= 0) return -3;
  const int last[9] = {p.mt, p.split_k, p.b_resident, pl.tail, p.pair, p.bn, p.a_mode, p.stages, grid};
  memcpy(g_last_launch, last, sizeof(last));
  {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = (size_t)(GEMM_SMEM_BYTES - TILE_SMEM_BYTES + tile_bytes(p));
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    int n_at = 0;
    if (p.pair) {
      at[n_at].id = cudaLaunchAttributeClusterDimension;
      at[n_at].val.clusterDim.x = 2;
      at[n_at].val.clusterDim.y = 1;
      at[n_at].val.clusterDim.z = 1;
      ++n_at;
    }
    if (g_opt.pdl >= 1) {   // the kernel's prologue may overlap the end of the work before it on the stream
      at[n_at].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[n_at].val.programmaticStreamSerializationAllowed = 1;
      ++n_at;
    }
    cfg.attrs = n_at ? at : nullptr;
    cfg.numAttrs = (unsigned)n_at;
    const int form = p.a_mode == A_FLAT_K ? 2 : p.scale || p.sc_stride != 0 || p.add_src != nullptr ? 1 : 0;
    const int which = p.lean ? LEAN_KERNEL : (p.scale ? 2 * (form + 2) : 2 * form) + (p.pair ? 1 : 0);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, KERNELS[which], p);
    if (e != cudaSuccess) {
      g_last_cuda_error = (int)e;
      cudaGetLastError();
      return -4;
    }
  }
  if (p.tail_items > 0) {
    TailFixArgs f;
    f.ws = p.ws;
    f.D = reinterpret_cast<__nv_bfloat16*>(p.D);
    f.bias = p.bias;
    f.mask = p.mask_src;
    f.add = p.add_src;
    f.scale = p.scale;
    f.sc_stride = p.sc_stride;
    f.sc_a = p.sc_a;
    f.sc_b = p.sc_b;
    f.sc_H = p.sc_H;
    f.sc_W = p.sc_W;
    f.ldd = p.ldd;
    f.M = p.M;
    f.bn = p.bn;
    f.rows_per_item = p.mt * BM;
    f.m_items = m_items_of(p, p.mt);
    f.box = p.a_mode == A_BOX_K ? 1 : 0;
    f.P = p.cv_P;
    f.Q = p.cv_Q;
    f.bx_rows = p.bx_rows;
    f.bx_groups = f.box ? (p.cv_P + p.mt * p.bx_rows - 1) / (p.mt * p.bx_rows) : 1;
    f.mt = p.mt;
    f.direct = f.m_items * p.n_tiles - p.tail_items;
    f.tail_items = p.tail_items;
    f.n_valid = p.n_valid;
    f.n_store = p.n_store;
    f.relu = p.relu;
    const long long groups = (long long)p.tail_items * f.rows_per_item * (p.bn / 8);
    long long blocks = (groups + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    launch_pdl(tail_fix_kernel, (int)blocks, 256, 0, stream, f);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) g_last_cuda_error = (int)e;
  return e == cudaSuccess ? 0 : -4;
}

// Shapes whose output is overwritten (bf16 epilogue: forward and data-grad passes) can be tuned by measurement:
// in tuning mode (rb_gemm_tune_mode(1), which a network switches on while it runs each of its convolution shapes
// once on scratch operands at build time) a launch of a shape that has no cached plan times every feasible
// (sub-tiles per item, resident B, tail cut) choice on the given stream and caches the fastest. The cost model
// alone mis-ranks them by up to 30 % (it knows rows filled, not how much of the epilogue is exposed). Outside
// tuning mode a launch never times anything: it takes the cached plan, or the cost model's.
// Box plans depend on the extents of the output rows, not on their product alone: at odd sizes two phases of a strided
// data-gradient have the same M, N and k-blocks with rows and columns exchanged.
// Flat plans depend on the pitch and the rows per image, which follow from paddings and input extents as well.
typedef std::tuple<int, int, int, int, int, int, int, int, int, int, int, int, int, int, int, int> PlanKey;
static std::map<PlanKey, Plan> g_plan_cache;
static std::mutex g_plan_mutex;

static PlanKey plan_key(const GemmTcParams& p) {
  return PlanKey(p.a_mode, p.b_mode, p.M, p.N, p.num_kb, p.bn, p.bk, p.n_tiles, p.cv_stride,
                 // (a forward pass with its normalisation takes the plan that was measured for the one without: it is not timed
                 // by itself)
                 (p.mask_src ? 1 : 0) | (p.add_src && !p.scale ? 2 : 0) | (p.sc_stride ? 4 : 0), p.cv_P, p.cv_Q, p.cv_S,
                 p.cv_cchunks, p.fl_pitch, p.fl_hp);
}

// CTA pairs must win by 3 %: measured alone they tie to within 2 % on the layers tried, and inside a training step (other
// kernels beside them) the plain plans did better.
constexpr float PAIR_MARGIN = 0.97f;

// Times a launch (the best of two after a first one); true, with its time in *best_ms, when it beats `margin` times *best_ms.
template <class Run>
static bool time_launches(cudaStream_t stream, Run run, float* best_ms, float margin = 1.0f) {
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float ms = 1e30f;
  bool ok = true;
  for (int rep = 0; rep < 3 && ok; ++rep) {
    cudaEventRecord(e0, stream);
    ok = run() == 0;
    cudaEventRecord(e1, stream);
    ok = ok && cudaEventSynchronize(e1) == cudaSuccess;
    float t = 0.f;
    if (ok) cudaEventElapsedTime(&t, e0, e1);
    if (ok && rep > 0 && t < ms) ms = t;   // the first run warms the caches
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!ok || ms >= *best_ms * margin) return false;
  *best_ms = ms;
  return true;
}

// Times the candidates of `p` (3 launches each, best of the last 2); returns the best time in ms, or a negative
// value when nothing could be run.
static float tune_plan(const GemmTcParams& p, bool b_is_weights, cudaStream_t stream, Plan* out,
                       const Plan* given = nullptr) {
  // the candidates: the one given, or plain plans first (sub-tiles x resident B x tail cut), then CTA pairs
  Plan cands[12];
  int n_cands = 0;
  if (given) cands[n_cands++] = *given;
  for (int pr = 0; pr <= (pair_ok(p) ? 1 : 0) && !given; ++pr) {
    for (int mt = 1; mt <= 2; ++mt) {
      for (int res = 0; res <= (pr ? 0 : 1); ++res) {
        if (res && (!b_is_weights || p.n_tiles != 1)) continue;
        for (int tail = 0; tail <= (pr ? 0 : 1); ++tail) {
          Plan cand{mt, 1, res, 0, 0.0};
          cand.pair = pr;
          if (tail) {
            if (!p.ws || g_opt.force_tail == 0 || g_opt.deterministic) continue;
            cand.tail = tail_parts((long long)m_items_of(p, mt) * p.n_tiles, g_num_sms, p.num_kb);
            if (cand.tail == 0) continue;
          }
          GemmTcParams q = p;
          if (apply_plan(q, cand) <= 0 || (res && q.stages < 3)) continue;
          cands[n_cands++] = cand;
        }
      }
    }
  }
  float best_ms = 1e30f;
  // pairs are timed after every plain plan and must win by PAIR_MARGIN (a plan that is given: the caller's business)
  for (int c = 0; c < n_cands; ++c)
    if (time_launches(stream, [&]() { return run_plan(p, cands[c], stream); }, &best_ms,
                      cands[c].pair && !given ? PAIR_MARGIN : 1.0f))
      *out = cands[c];
  return best_ms < 1e29f ? best_ms : -1.f;
}

static bool tunable(const GemmTcParams& p, cudaStream_t stream) {
  if (!g_tune_mode || !g_opt.autotune || p.epi != EPI_BF16) return false;
  if (g_opt.force_mt || g_opt.force_resident >= 0 || g_opt.force_pair == 1) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
}

static int launch(GemmTcParams& p, bool allow_split, int fixed_split, bool b_is_weights, cudaStream_t stream) {
  if (p.M <= 0 || p.n_tiles <= 0 || p.num_kb <= 0) return 0;
  Plan pl = plan_shape(p, allow_split, fixed_split, b_is_weights);
  if (pl.cost >= 1e299) return -3;
  bool forced = g_opt.force_mt || g_opt.force_resident >= 0 || g_opt.force_tail >= 0;
  if (g_opt.force_pair == 1 && pair_ok(p)) {   // pairs wherever they are feasible (tests, experiments)
    const int most = p.a_mode == A_FLAT_K ? 4 : 2;
    for (int mt = g_opt.force_mt ? std::min(g_opt.force_mt, most) : 2; mt >= 1; --mt) {
      Plan pp{mt, pl.split, 0, 0, 0.0};
      pp.pair = 1;
      GemmTcParams q = p;
      if (apply_plan(q, pp) > 0) {
        pl = pp;
        forced = true;
        break;
      }
      if (g_opt.force_mt) break;
    }
  }
  const Plan model = pl;
  if (p.epi == EPI_BF16 && !forced) {
    std::lock_guard<std::mutex> lock(g_plan_mutex);
    auto it = g_plan_cache.find(plan_key(p));
    if (it != g_plan_cache.end()) {
      Plan cached = it->second;
      if (cached.tail && (!p.ws || g_opt.deterministic)) cached.tail = 0;   // tuned with a workspace, launched without
      pl = cached;
    } else if (tunable(p, stream)) {
      Plan best = pl;
      if (tune_plan(p, b_is_weights, stream, &best) > 0.f) pl = best;
      g_plan_cache[plan_key(p)] = pl;
    }
  }
  const int rc = run_plan(p, pl, stream);
  // a plan from the cache that does not fit this launch (a smaller workspace, options changed since): the cost model's
  return rc == -3 ? run_plan(p, model, stream) : rc;
}

static int round_bn(int n, int cap) {
  int bn = ((n + 31) / 32) * 32;
  if (bn > cap) bn = cap;
  return bn;
}

// Tile width for `n` output columns: among 1..4 column tiles (width a multiple of `gran`, at most 256), the one
// whose plan is cheapest. `setup(p, bn)` must fill the fields that depend on the width.
template <class Setup>
static int pick_bn(GemmTcParams& p, int n, int gran, bool allow_split, int fixed_split, bool b_is_weights,
                   Setup setup) {
  int best_bn = 0;
  double best_cost = 1e300;
  const int cap = g_opt.bn_cap > 0 ? g_opt.bn_cap : 256;
  for (int nt = 1; nt <= 4; ++nt) {
    int bn = (n + nt - 1) / nt;
    const int g = (nt > 1 && gran < 64) ? 64 : gran;   // the bf16 epilogue stores 64-column slabs
    bn = (bn + g - 1) / g * g;
    if (bn > 256 || bn > cap || bn == best_bn) continue;
    setup(p, bn);
    const Plan pl = plan_shape(p, allow_split, fixed_split, b_is_weights);
    if (pl.cost < best_cost * 0.97) { best_cost = pl.cost; best_bn = bn; }
  }
  if (best_bn == 0) best_bn = 256;
  setup(p, best_bn);
  return best_bn;
}

// Tile width chosen by measurement for a convolution shape (key: the plan key with the width left out).
static std::map<PlanKey, int> g_bn_cache;

}  // namespace rb

using namespace rb;

extern "C" {

// Dense GEMM on bf16 operands:  D[M x N] = op(A) * op(B)^T-style contraction over K.
//   a_mn = 0: A is [M][K] (K contiguous, pitch lda)     a_mn = 1: A is [K][M] (M contiguous, pitch lda)
//   b_mn = 0: B is [N][K] (K contiguous, pitch ldb)     b_mn = 1: B is [K][N] (N contiguous, pitch ldb)
//   epi = 0: bf16 D (+bias, ReLU, mask);  epi = 1: fp32 D overwritten;  epi = 2: fp32 D accumulated (red.add)
// split_k <= 0 lets the library choose; epi 0/1 force split_k = 1.
int rb_gemm_tc(const void* A, int a_mn, long long lda, const void* B, int b_mn, long long ldb, int M, int N, int K,
               void* D, long long ldd, int epi, const float* bias, int relu, const void* mask_src, int n_valid,
               int n_store, int split_k, int bn_cap, float* ws, long long ws_bytes, unsigned int* status,
               cudaStream_t stream) {
  int rc = ensure_driver_entry();
  if (rc) return rc;
  if ((n_store > 0 ? n_store : N) % 32 != 0 || ldd % 8 != 0) return -11;  // epilogue writes 32-column chunks
  GemmTcParams p;
  memset(&p, 0, sizeof(p));
  p.ws = ws;
  p.ws_bytes = ws ? ws_bytes : 0;
  const bool any_mn = a_mn || b_mn;
  p.bk = (!any_mn && (K % 64 != 0) && (K % 32 == 0)) ? 32 : 64;
  if (bn_cap <= 0) bn_cap = 256;
  p.bn = round_bn(N, bn_cap);
  if (b_mn || (epi == EPI_BF16 && N > p.bn)) p.bn = ((p.bn + 63) / 64) * 64;
  p.bn_load = p.bn;
  p.M = M;
  p.N = N;
  p.num_kb = (K + p.bk - 1) / p.bk;
  p.n_tiles = (N + p.bn - 1) / p.bn;
  const CUtensorMapSwizzle ksw = p.bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  if (a_mn) {
    p.a_mode = A_TILED_MN;
    rc = make_map_2d(&p.tm_a, A, M, K, lda, 64, p.bk, CU_TENSOR_MAP_SWIZZLE_128B);
  } else {
    p.a_mode = A_TILED_K;
    p.a_split = pick_box_split(g_opt.a_split, BM, p.bk);
    rc = make_map_2d(&p.tm_a, A, K, M, lda, p.bk, BM / p.a_split, ksw);
  }
  if (rc) return rc;
  if (b_mn) {
    p.b_mode = B_TILED_MN;
    rc = make_map_2d(&p.tm_b, B, N, K, ldb, 64, p.bk, CU_TENSOR_MAP_SWIZZLE_128B);
  } else {
    p.b_mode = B_TILED_K;
    p.b_split = pairable_b_split(p.bn, p.bk);
    rc = make_map_2d(&p.tm_b, B, K, N, ldb, p.bk, p.bn / p.b_split, ksw);
  }
  if (rc) return rc;
  p.epi = epi;
  p.relu = relu;
  p.n_valid = n_valid > 0 ? n_valid : N;
  p.n_store = n_store > 0 ? n_store : N;
  p.ldd = ldd;
  p.D = D;
  p.bias = bias;
  p.mask_src = reinterpret_cast<const __nv_bfloat16*>(mask_src);
  p.status = status;
  if (epi == EPI_BF16) {
    rc = make_map_out(&p.tm_d, D, p.n_store, M, ldd);
    if (rc) return rc;
    if (mask_src) rc = make_map_out(&p.tm_mask, const_cast<void*>(mask_src), p.n_store, M, ldd);
    if (rc) return rc;
  } else {
    rc = make_map_out_f32(&p.tm_d, D, p.n_store, M, ldd);
    if (rc) return rc;
  }
  if (epi != EPI_F32_ATOMIC) split_k = 1;
  if (split_k > p.num_kb) split_k = p.num_kb;
  while (split_k > 1 && !split_ok(split_k, p.num_kb)) --split_k;
  return launch(p, epi == EPI_F32_ATOMIC && split_k <= 0, split_k > 0 ? split_k : 0, !b_mn, stream);
}

}  // extern "C"

namespace rb {

// What turns a forward convolution into (one output phase of) a data-gradient: filters read as they lie (B_DGRAD_MN),
// rows scattered, an addend.
struct DgradForm {
  int packed;                              // the filters are transposed and flipped: [n_store][taps][Cp], K-major
  int taps, base, du, dv;                  // filter taps of the layer, and which of them tap (u, v) is
  int sc_stride, sc_a, sc_b, sc_H, sc_W;
  const void* add;
};

// A normalisation in the epilogue of a forward pass, with an optional residual.
struct NormForm {
  const float* scale;
  const void* residual;
};

// x NHWC bf16 [N][H][W][Cp]; w bf16 [Kout][R*S][Cp], or with `dg` the filters [k_rows][taps][n_store] of the layer whose
// data-gradient this is (or their packed form); y bf16 [N*P*Q][ldy]. Base pixel range: lower = -pad, P / Q given by the
// caller.
static int conv_forward_form(const void* x, int N, int H, int W, int Cp, const void* w, int Kout, int R, int S, int stride,
                             int pad_h, int pad_w, int P, int Q, void* y, long long ldy, const float* bias, int relu,
                             const void* mask_src, int n_valid, int n_store, int k_rows, const DgradForm* dg, const NormForm* norm,
                             float* ws, long long ws_bytes, unsigned int* status, cudaStream_t stream) {
  int rc = ensure_driver_entry();
  if (rc) return rc;
  GemmTcParams p;
  memset(&p, 0, sizeof(p));
  p.ws = ws;
  p.ws_bytes = ws ? ws_bytes : 0;
  // The TMA unit is bound by rows (requests), not bytes: 64-channel (128-byte) rows halve the rows per MMA. A channel
  // count such as 96 therefore runs as two 64-channel chunks whose upper half lies outside the tensor and is
  // zero-filled by the TMA unit (both operands), rather than as three 32-channel chunks: a third more MMA work,
  // a third fewer loads, and the loads are what binds.
  p.bk = (Cp % 64 == 0 || (Cp > 64 && g_opt.bk32 != 1)) ? 64 : 32;   // option bk32: keep 32-channel chunks
  if (Cp % 32 != 0) return -10;
  if ((n_store > 0 ? n_store : Kout) % 32 != 0 || ldy % 8 != 0) return -11;
  const CUtensorMapSwizzle ksw = p.bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  const int n_cols = n_store > 0 ? n_store : Kout;
  p.M = N * P * Q;
  p.N = Kout;
  p.cv_cchunks = (Cp + p.bk - 1) / p.bk;
  p.num_kb = R * S * p.cv_cchunks;
  p.epi = EPI_BF16;
  p.a_mode = A_IM2COL_K;
  const bool mn = dg && !dg->packed;
  p.b_mode = mn ? B_DGRAD_MN : B_TILED_K3;
  pick_bn(p, n_cols, 32, false, 1, true, [n_cols, mn](GemmTcParams& q, int bn) {
    q.bn = bn;
    q.bn_load = mn ? (bn + 63) / 64 * 64 : bn;
    q.n_tiles = (n_cols + bn - 1) / bn;
  });
  if (dg) {
    p.dg_base = dg->base;
    p.dg_du = dg->du;
    p.dg_dv = dg->dv;
    p.sc_stride = dg->sc_stride;
    p.sc_a = dg->sc_a;
    p.sc_b = dg->sc_b;
    p.sc_H = dg->sc_H;
    p.sc_W = dg->sc_W;
    p.add_src = reinterpret_cast<const __nv_bfloat16*>(dg->add);
  }
  if (norm) {
    p.scale = norm->scale;
    p.add_src = reinterpret_cast<const __nv_bfloat16*>(norm->residual);
  }
  p.cv_P = P;
  p.cv_Q = Q;
  p.cv_stride = stride;
  p.cv_lower_h = -pad_h;
  p.cv_lower_w = -pad_w;
  p.cv_S = S;
  p.relu = relu;
  p.n_valid = n_valid > 0 ? n_valid : Kout;
  p.n_store = n_store > 0 ? n_store : Kout;
  p.ldd = ldy;
  p.D = y;
  p.bias = bias;
  p.mask_src = reinterpret_cast<const __nv_bfloat16*>(mask_src);
  p.status = status;
  // upper corner so that the base pixel takes exactly P x Q positions
  const int upper_h = (P - 1) * stride - pad_h - (H - 1);
  const int upper_w = (Q - 1) * stride - pad_w - (W - 1);
  p.a_split = pick_box_split(g_opt.a_split, BM, p.bk);
  const bool one_by_one = R == 1 && S == 1 && stride == 1 && pad_h == 0 && pad_w == 0 && P == H && Q == W;
  rc = make_map_out(&p.tm_d, y, p.n_store, p.M, ldy);
  if (rc) return rc;
  if (mask_src) rc = make_map_out(&p.tm_mask, const_cast<void*>(mask_src), p.n_store, p.M, ldy);
  if (rc) return rc;
  // How the A operand is loaded (`how`: LOAD_BOX = tap-shifted tiled boxes of whole output rows, LOAD_FLAT = whole input
  // rows once for all taps, else the im2col map, or plain tiled rows for a 1 x 1 convolution) and what depends on the tile
  // width: column tiling, the filter map's box.
  enum { LOAD_BOX = 1, LOAD_FLAT = 2 };
  auto configure = [&](GemmTcParams& q, int how, int bn) -> int {
    int e;
    if (how == LOAD_FLAT) {
      q.a_mode = A_FLAT_K;
      q.a_split = 1;
      if (!flat_geom(q, N, H, W, R, S, pad_h, pad_w)) return -3;
      e = make_map_nhwc(&q.tm_a, x, Cp, W, H, N, Cp, q.bk, q.fl_pitch, 1, ksw);
    } else if (how == LOAD_BOX) {
      q.a_mode = A_BOX_K;
      q.a_split = 1;
      q.bx_rows = BM / Q;
      q.bx_pad_h = pad_h;
      q.bx_pad_w = pad_w;
      e = make_map_nhwc(&q.tm_a, x, Cp, W, H, N, Cp, q.bk, Q, q.bx_rows, ksw);
    } else if (one_by_one) {
      // a 1 x 1 convolution is a plain GEMM over the pixel rows: tiled loads, which the TMA unit serves 2-3x
      // faster per row than im2col-mode loads
      q.a_mode = A_TILED_K;
      e = make_map_2d(&q.tm_a, x, Cp, (uint64_t)q.M, Cp, q.bk, BM / q.a_split, ksw);
    } else {
      q.a_mode = A_IM2COL_K;
      e = make_map_im2col(&q.tm_a, x, N, H, W, Cp, -pad_h, -pad_w, upper_h, upper_w, stride, q.bk, BM / q.a_split, ksw);
    }
    if (e) return e;
    q.bn = q.bn_load = bn;
    q.n_tiles = (n_cols + bn - 1) / bn;
    if (mn) {
      q.bn_load = (bn + 63) / 64 * 64;
      return make_map_3d(&q.tm_b, w, n_cols, dg->taps, k_rows, n_cols, (uint64_t)dg->taps * n_cols, 64, 1, q.bk,
                         CU_TENSOR_MAP_SWIZZLE_128B);
    }
    q.b_split = pairable_b_split(bn, q.bk);
    const uint64_t taps = dg ? dg->taps : R * S;
    return make_map_3d(&q.tm_b, w, Cp, taps, Kout, Cp, taps * Cp, q.bk, 1, bn / q.b_split, ksw);
  };
  // Candidates beside the default (im2col loads, tiles of at most 256 columns):
  //  * between 257 and 512 output columns, ONE tile as wide as the layer (two MMAs side by side, one accumulator
  //    set, no overlap of epilogue and main loop) instead of narrower tiles that each load the A operand again;
  //  * for stride-1 convolutions with more than one tap and output rows of at most 128 positions, box loads:
  //    cheaper per row for the TMA unit, at the price of tile rows that are computed and dropped when Q does not
  //    divide 128 (and when bx_rows does not divide P).
  //  * for stride-1 convolutions with more than one tap, flat mode: the first five plans by its cost model. On 76 layers and
  //    directions of this framework's networks these held the best plan that beat the other modes in all but one, which
  //    loses 3 %.
  // Which is fastest is decided by measurement in tuning mode and remembered per shape; without a measurement the
  // default is taken.
  const int bn_default = p.bn;
  const int bn_wide = (n_cols > 256 && n_cols <= 512 && g_opt.force_wide != 0 && g_opt.bn_cap >= 256) ? n_cols : 0;
  const bool box_ok = stride == 1 && R * S > 1 && Q <= BM && g_opt.force_box != 0;
  // flat mode: the widths of one to four equal column tiles of at most 256 columns, 0 for those that are not
  const int flat_cap = g_opt.bn_cap > 0 ? std::min(g_opt.bn_cap, 256) : 256;
  auto flat_bn = [n_cols, flat_cap](int nt) {
    const int per = (n_cols + nt - 1) / nt, bn = nt == 1 ? (per + 31) / 32 * 32 : (per + 63) / 64 * 64;
    return bn > flat_cap || bn * (nt - 1) >= n_cols ? 0 : bn;
  };
  GemmTcParams key_p = p;
  const bool flat_fits = stride == 1 && R * S > 1 && flat_geom(key_p, N, H, W, R, S, pad_h, pad_w);
  // (flat mode adds the channel chunks outside the taps, all others inside: with `deterministic` timing must not choose the order)
  const bool flat_ok = flat_fits && g_opt.force_halo != 0 && !g_opt.deterministic;
  auto flat_candidates = [&]() {      // (width, plan), best first
    std::vector<std::pair<int, Plan>> all;
    for (int nt = 1; nt <= 4 && flat_ok; ++nt) {
      GemmTcParams q = p;
      if (!flat_bn(nt) || configure(q, LOAD_FLAT, flat_bn(nt))) continue;
      Plan plans[12];
      const int n = flat_plans(q, plans, 12);
      for (int i = 0; i < n; ++i) all.push_back({flat_bn(nt), plans[i]});
    }
    std::stable_sort(all.begin(), all.end(), [](const std::pair<int, Plan>& a, const std::pair<int, Plan>& b) {
      return a.second.cost < b.second.cost;
    });
    return all;
  };
  int use = bn_default;   // low 16 bits: tile width; above: how A is loaded
  if (bn_wide || box_ok || flat_ok) {
    key_p.bn = key_p.n_tiles = 0;
    const PlanKey ckey = plan_key(key_p);
    std::lock_guard<std::mutex> lock(g_plan_mutex);   // released at the end of this block, before `launch` takes it
    auto it = g_bn_cache.find(ckey);
    const auto forced = g_opt.force_halo == 1 ? flat_candidates() : std::vector<std::pair<int, Plan>>();
    if (!forced.empty()) {
      use = forced[0].first | (LOAD_FLAT << 16);
    } else if (g_opt.force_wide == 1 || g_opt.force_box == 1) {
      use = ((bn_wide && g_opt.force_wide == 1) ? bn_wide : bn_default) |
            ((box_ok && g_opt.force_box == 1) ? LOAD_BOX << 16 : 0);
    } else if (it != g_bn_cache.end()) {
      use = it->second;   // as far as it still applies: the options may have changed since it was measured
      if ((use >> 16) == LOAD_FLAT && (!flat_ok || (use & 0xFFFF) > flat_cap)) use = bn_default;
      if ((use >> 16) == LOAD_BOX && !box_ok) use &= 0xFFFF;
      if ((use >> 16) != LOAD_FLAT && (use & 0xFFFF) != bn_default && (use & 0xFFFF) != bn_wide)
        use = bn_default | (use & ~0xFFFF);
    } else if (tunable(p, stream)) {
      float best_ms = 1e30f;
      auto measure = [&](int how, int bn, const Plan* given) {
        GemmTcParams q = p;
        if (configure(q, how, bn)) return;
        Plan pl{1, 1, 0, 0, 0.0};
        const float ms = tune_plan(q, true, stream, &pl, given);
        if (ms > 0.f && ms < best_ms * (given && given->pair ? PAIR_MARGIN : 1.0f)) {
          best_ms = ms;
          use = bn | (how << 16);
          g_plan_cache[plan_key(q)] = pl;
        }
      };
      for (int how = 0; how <= (box_ok ? LOAD_BOX : 0); ++how)
        for (int bn : {bn_default, bn_wide})
          if (bn) measure(how, bn, nullptr);
      const auto flat = flat_candidates();
      for (int pair = 0; pair <= 1; ++pair)
        for (size_t i = 0; i < flat.size() && i < 5; ++i)
          if (flat[i].second.pair == pair) measure(LOAD_FLAT, flat[i].first, &flat[i].second);
      g_bn_cache[ckey] = use;
    }
  }
  GemmTcParams q = p;
  rc = configure(q, use >> 16, use & 0xFFFF);
  if (rc == 0) rc = launch(q, false, 1, true, stream);
  if (rc != -3 || (use >> 16) != LOAD_FLAT) return rc;
  // nothing was launched: no flat plan fits this convolution, under these options, at the width that was measured
  rc = configure(p, 0, bn_default);
  return rc ? rc : launch(p, false, 1, true, stream);
}

// ---- weight-gradients from whole rows (wgrad_rows.cuh) ------------------------------------------------------------------
// The cheapest plan for each division of a shape into items (filter rows, channel blocks, how positions line up), cheapest first.
// Modelled in cycles: MMAs (a 128 x N x 16 step takes N / 2, at least 49), L2 delivery (41 bytes per cycle and SM), a fixed part
// per chunk, the additions into dw (19 bytes per cycle and SM).
static std::vector<WgradRowsParams> rows_plans(int N, int H, int W, int Cp, int Kout, int R, int S, int pad_h, int pad_w, int P,
                                               int Q, int tile) {
  std::vector<std::pair<double, WgradRowsParams>> all;
  if (S > 8 || R * S < 2 || pad_h < 0 || pad_w < 0 || Cp % 32 != 0) return {};
  const int sms = g_num_sms > 0 ? g_num_sms : 148;
  WgradRowsParams p;
  memset(&p, 0, sizeof(p));
  p.R = R;
  p.S = S;
  p.pad_h = pad_h;
  p.pad_w = pad_w;
  p.Cp = Cp;
  p.Kout = Kout;
  p.xw = Cp % 64 == 0 || Cp > 128 ? 64 : 32;      // 32 and 96 channels without empty halves
  p.dyw = Kout > 32 ? 64 : 32;
  p.cblocks = (Cp + p.xw - 1) / p.xw;
  p.dy_blocks = Kout > 64 ? 2 : 1;
  p.m_tiles = (Kout + BM - 1) / BM;
  p.tile_bytes = tile;
  const int most = 256 / p.xw, pieces = (S + most - 1) / most, xpos = p.xw * 2, dypos = p.dyw * 2;
  const int per_mma = p.per_mma = (S + pieces - 1) / pieces;
  const int share = std::max(0, std::min({pad_w, S - 1, Q + S - 1 - pad_w - W}));
  auto kb = [](long long bytes) { return (int)((bytes + 1023) / 1024 * 1024); };
  for (int nr : {1, R}) {
    for (int ncb = 1; ncb <= std::min(4, p.cblocks); ++ncb) {
      if (nr * ncb * S * p.xw > 512 || nr * ncb * pieces > 4 || (nr == R && R == 1)) continue;
      for (int run = 0; run <= 1; ++run) {
        const int wdy = run ? Q + S - 1 - share : (Q + 15) / 16 * 16, wx = run ? wdy : wdy + S - 1;
        if (wx > 256) continue;
        double best_cost = -1.0;
        WgradRowsParams best;
        for (int rows = 1; rows <= std::min(P, 256 - nr + 1); ++rows) {
          for (int images = 1; images <= (rows == P && nr == 1 ? std::min(N, 16) : 1); ++images) {
            WgradRowsParams q = p;
            q.nr = nr;
            q.ncb = ncb;
            q.rows = rows;
            q.images = images;
            const long long dy_pos = (long long)rows * images * wdy, x_pos = (long long)(rows + nr - 1) * images * wx;
            q.segs = run ? 1 : rows * images;
            q.steps = (int)(run ? (dy_pos + 15) / 16 : wdy / 16);
            q.dy_seg = wdy * dypos >> 4;
            q.x_seg = wx * xpos >> 4;
            q.x_row = wx * xpos >> 4;
            q.dy_bytes = (int)(dy_pos * dypos);
            q.x_bytes = (int)(x_pos * xpos);
            q.dy_block = kb((run ? q.steps * 16ll : dy_pos) * dypos);
            q.x_block = kb((run ? x_pos + 16 + S : x_pos) * xpos);
            q.clear = run;
            const long long stage = (long long)q.dy_blocks * q.dy_block + (long long)ncb * q.x_block;
            if (stage * 2 > tile) break;
            q.stages = (int)std::min<long long>(tile / stage, MAX_STAGES);
            q.row_groups = (P + rows - 1) / rows;
            q.chunks = (N + images - 1) / images * q.row_groups;
            q.groups_r = R / nr;
            q.groups_c = (p.cblocks + ncb - 1) / ncb;
            const int per = q.groups_r * q.groups_c * q.m_tiles;
            q.splits = std::max(1, std::min(q.chunks, sms / per));
            q.work = per * q.splits;
            double mma = 0.0;
            for (int s0 = 0; s0 < S; s0 += per_mma) mma += std::max(49.0, 0.5 * p.xw * std::min(per_mma, S - s0));
            mma *= (double)nr * ncb * q.segs * q.steps;
            // (a position of 64 bytes takes the TMA unit as long as one of 128: ~2.3 cycles)
            const double load = std::max(((double)q.dy_blocks * q.dy_bytes + (double)ncb * q.x_bytes) / 41.0,
                                         2.3 * ((double)q.dy_blocks * dy_pos + (double)ncb * x_pos));
            const double chunk = std::max(mma, load) + (q.stages == 2 ? 0.15 * load + 200.0 : 120.0);
            const double epilogue = (double)nr * ncb * S * p.xw * (std::min(Kout, BM) + 31) / 32 * 32 * 4 / 19.0 + 2500.0;
            const double cost = ((q.work + sms - 1) / sms) * ((double)((q.chunks + q.splits - 1) / q.splits) * chunk + epilogue);
            if (best_cost < 0.0 || cost < best_cost) {
              best_cost = cost;
              best = q;
            }
          }
        }
        if (best_cost >= 0.0) all.push_back({best_cost, best});
      }
    }
  }
  std::stable_sort(all.begin(), all.end(), [](const std::pair<double, WgradRowsParams>& a, const std::pair<double, WgradRowsParams>& b) {
    return a.first < b.first;
  });
  std::vector<WgradRowsParams> plans;
  for (const auto& a : all) plans.push_back(a.second);
  return plans;
}

// What was measured as the fastest for a weight-gradient: a plan, or none of them (`rows` = 0: gemm_tc_kernel).
typedef std::tuple<int, int, int, int, int, int, int, int, int, int, int, int> RowsKey;
static std::map<RowsKey, WgradRowsParams> g_rows_cache;
// With less work than this the general kernel adds up from 1 to 16 parts, row plans from 24 to 49, whose order is left open, and runs
// repeat less closely: LeNet's parameters after eight steps at 17 images, two captured runs, differ by 4e-4 of an update in the median
// with the general kernel and by 2.7e-2 with row plans (one value at a rounding edge falls either way). It is not the faster of the
// two everywhere below the line: a launch of row plans takes 0.3 to 2.5 us less of 6 to 8 (32 -> 32 channels on 8 x 32 x 32, 0.15
// GFLOP: 8.1 -> 5.6) or up to 2.5 more (256 -> 256 on 4 x 4 x 4: 4.3 -> 6.8).
constexpr double ROWS_MIN_FLOPS = 0.2e9;
// Row plans have to win by this much: two timings of one launch differ by up to 2 %, and between equals the general kernel adds up
// fewer parts. 512 -> 512 on 64 x 32 x 32: without the margin a row plan of 192.9 us was kept over 189.1; with it the general kernel
// in four tunings of four.
constexpr float ROWS_MARGIN = 0.97f;

static int run_rows(WgradRowsParams p, const void* x, int N, int H, int W, const void* dy, long long lddy, int P, int Q, float* dw,
                    unsigned int* status, cudaStream_t stream) {
  p.status = status;
  p.x = reinterpret_cast<const __nv_bfloat16*>(x);
  p.dy = reinterpret_cast<const __nv_bfloat16*>(dy);
  p.lddy = lddy;
  p.N = N;
  p.H = H;
  p.W = W;
  p.P = P;
  p.Q = Q;
  const int wdy = p.dy_seg * 16 / (p.dyw * 2), wx = p.x_seg * 16 / (p.xw * 2);
  cuuint64_t dims_dy[4] = {(cuuint64_t)p.Kout, (cuuint64_t)Q, (cuuint64_t)P, (cuuint64_t)N};
  cuuint64_t dims_x[4] = {(cuuint64_t)p.Cp, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
  cuuint64_t str_dy[3] = {(cuuint64_t)lddy * 2, (cuuint64_t)lddy * Q * 2, (cuuint64_t)lddy * Q * P * 2};
  cuuint64_t str_x[3] = {(cuuint64_t)p.Cp * 2, (cuuint64_t)p.Cp * W * 2, (cuuint64_t)p.Cp * W * H * 2};
  cuuint32_t box_dy[4] = {(cuuint32_t)p.dyw, (cuuint32_t)wdy, (cuuint32_t)p.rows, (cuuint32_t)p.images};
  cuuint32_t box_x[4] = {(cuuint32_t)p.xw, (cuuint32_t)wx, (cuuint32_t)(p.rows + p.nr - 1), (cuuint32_t)p.images};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = g_encode_tiled(&p.tm_dy, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(dy), dims_dy, str_dy, box_dy, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, p.dyw == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS)
    r = g_encode_tiled(&p.tm_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(x), dims_x, str_x, box_x, es,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, p.xw == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return -(400 + (int)r);
  const long long ldd = (long long)p.R * p.S * p.Cp;
  const int rc = make_map_out_f32(&p.tm_dw, dw, ldd, p.Kout, ldd);
  if (rc) return rc;
  const int grid = std::min(p.work, g_num_sms);
  const int last[9] = {p.nr, p.splits, p.ncb, p.rows, p.images, p.clear ? 0 : p.segs, A_ROWS, p.stages, grid};
  memcpy(g_last_launch, last, sizeof(last));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = (size_t)(GEMM_SMEM_BYTES - TILE_SMEM_BYTES + p.tile_bytes);
  cfg.stream = stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = g_opt.pdl >= 1 ? 1u : 0u;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, wgrad_rows_kernel, p);
  if (e == cudaSuccess) return 0;
  g_last_cuda_error = (int)e;
  cudaGetLastError();
  return -4;
}

// The output phases of a strided data-gradient (conv_dgrad below) that have filter taps.
struct DgradPhase {
  int a, b;                    // positions (s i + a, s j + b)
  int r0, c0, U, V, pt, pl;    // first tap, taps, padding of the stride-1 convolution that the phase is
  int Hp, Wp;                  // positions
};

// All of them in ONE launch (GemmPhasesParams). Launched one by one, a phase's work of a few us lies between the set-up and the
// drain of its own launch, and leaves SMs idle at its end. 3 x 3 / 2, us for four launches and for one, on a replayed graph:
// 64 <- 128 channels on 32 x 64 x 64: 41.8, 20.9; 256 <- 512 on 32 x 16 x 16: 52.6, 17.8; 32 <- 64 on 128 x 16 x 16: 24.3, 7.8;
// 32 <- 32 on 512 x 32 x 32: 68.6, 47.2. The filters are read in place or from their packed copy, the phases with more taps come
// first, and tile width and sub-tiles per item are common to all.
static int run_phases(GemmPhasesParams p, int bn, int mt, int n_cols, cudaStream_t stream) {
  p.bn = bn;
  p.bn_load = p.b_mode == B_DGRAD_MN ? (bn + 63) / 64 * 64 : bn;
  p.n_tiles = (n_cols + bn - 1) / bn;
  p.mt = mt;
  p.acc_stride = acc_stride_for(bn);
  p.acc_bufs = 2 * mt * p.acc_stride <= 512 ? 2 : 1;
  if (bn > 256 || mt * p.acc_stride > 512) return -3;
  p.stages = std::min(TILE_SMEM_BYTES / (mt * BM * p.bk * 2 + p.bn_load * p.bk * 2), MAX_STAGES);
  if (p.stages < 2) return -3;
  int work = 0;
  for (int k = 0; k < p.phases; ++k) {
    p.ph[k].work0 = work;
    p.ph[k].m_items = (p.ph[k].M + BM * mt - 1) / (BM * mt);
    work += p.ph[k].m_items * p.n_tiles;
  }
  const int grid = std::min(work, g_num_sms);
  const int last[9] = {mt, 1, 0, 0, 0, bn, p.a_mode, p.stages, grid};
  memcpy(g_last_launch, last, sizeof(last));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = GEMM_SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = g_opt.pdl >= 1 ? 1u : 0u;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, PHASES_KERNEL, p);
  if (e == cudaSuccess) return 0;
  g_last_cuda_error = (int)e;
  cudaGetLastError();
  return -4;
}

typedef std::tuple<int, int, int, int, int, int, int, int, int, int, int, int, int, int> PhasesKey;
static std::map<PhasesKey, std::pair<int, int>> g_phases_cache;      // tile width (0: one launch per phase) and sub-tiles

// `separate`: runs the phases one by one. Returns -3 when that is what is to be done and nothing has been launched.
template <class Separate>
static int dgrad_phases(const void* dy, int N, int P, int Q, int Kp, const void* w, bool packed, int Kout, int Cp, int c_valid,
                        int R, int S, int stride, int pad_h, int pad_w, int H, int W, void* dx, const void* add, const void* mask,
                        const DgradPhase* phases, int n_phases, unsigned int* status, cudaStream_t stream, Separate separate) {
  int rc = ensure_driver_entry();
  if (rc) return rc;
  GemmPhasesParams p;
  memset(&p, 0, sizeof(p));
  p.bk = (Kp % 64 == 0 || (Kp > 64 && g_opt.bk32 != 1)) ? 64 : 32;
  if (Kp % 32 != 0) return -10;
  const CUtensorMapSwizzle ksw = p.bk == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  p.N = Cp;
  p.a_mode = A_IM2COL_K;
  p.b_mode = packed ? B_TILED_K3 : B_DGRAD_MN;
  p.cv_cchunks = (Kp + p.bk - 1) / p.bk;
  p.cv_stride = 1;
  p.a_split = pick_box_split(g_opt.a_split, BM, p.bk);
  p.split_k = 1;
  p.epi = EPI_BF16;
  p.epi_bufs = 1;
  p.n_valid = c_valid;
  p.n_store = Cp;
  p.ldd = Cp;
  p.D = dx;
  p.add_src = reinterpret_cast<const __nv_bfloat16*>(add);
  p.mask_src = reinterpret_cast<const __nv_bfloat16*>(mask);
  p.status = status;
  p.sc_stride = stride;
  p.sc_H = H;
  p.sc_W = W;
  p.dg_du = packed ? stride * S : -stride * S;
  p.dg_dv = packed ? stride : -stride;
  p.phases = n_phases;
  int order[MAX_PHASES];
  for (int k = 0; k < n_phases; ++k) order[k] = k;
  std::stable_sort(order, order + n_phases, [&](int x, int y) { return phases[x].U * phases[x].V > phases[y].U * phases[y].V; });
  double rows_kb = 0.0;      // 128-row tiles x k-blocks of the launch
  for (int k = 0; k < n_phases; ++k) {
    const DgradPhase& f = phases[order[k]];
    GemmPhase& g = p.ph[k];
    g.M = N * f.Hp * f.Wp;
    g.num_kb = f.U * f.V * p.cv_cchunks;
    g.P = f.Hp;
    g.Q = f.Wp;
    g.lower_h = -f.pt;
    g.lower_w = -f.pl;
    g.S = f.V;
    g.dg_base = (f.r0 + stride * (f.U - 1)) * S + f.c0 + stride * (f.V - 1);
    if (packed) g.dg_base = R * S - 1 - g.dg_base;      // tap t lies at R * S - 1 - t
    g.sc_a = f.a;
    g.sc_b = f.b;
    p.M = std::max(p.M, g.M);
    p.num_kb = std::max(p.num_kb, g.num_kb);
    rows_kb += (double)((g.M + BM - 1) / BM) * g.num_kb;
    rc = make_map_im2col(&g.tm_a, dy, N, P, Q, Kp, -f.pt, -f.pl, f.Hp - f.pt - P, f.Wp - f.pl - Q, 1, p.bk, BM / p.a_split, ksw);
    if (rc) return rc;
  }
  auto with_b = [&](GemmPhasesParams& q, int bn) -> int {      // the filters' map, whose box depends on the tile width
    const uint64_t taps = (uint64_t)R * S;
    if (!packed)
      return make_map_3d(&q.tm_b, w, Cp, taps, Kout, Cp, taps * Cp, 64, 1, q.bk, CU_TENSOR_MAP_SWIZZLE_128B);
    q.b_split = pick_box_split(g_opt.b_split, bn, q.bk);
    return make_map_3d(&q.tm_b, w, Kp, taps, Cp, Kp, taps * Kp, q.bk, 1, bn / q.b_split, ksw);
  };
  // Candidates: one to four equal column tiles, one or two sub-tiles. The model ranks them by rows filled per SM (see Plan) plus
  // what is left when the longest item ends last.
  std::pair<int, int> cands[8], best(0, 0);
  int n_cands = 0;
  double best_cost = 1e300;
  const int cap = g_opt.bn_cap > 0 ? std::min(g_opt.bn_cap, 256) : 256;
  for (int nt = 1; nt <= 4; ++nt) {
    const int per = (Cp + nt - 1) / nt, bn = nt == 1 ? (per + 31) / 32 * 32 : (per + 63) / 64 * 64;
    if (bn > cap || bn * (nt - 1) >= Cp) continue;
    for (int mt = 1; mt <= 2; ++mt) {
      if (g_opt.force_mt && mt != std::min(g_opt.force_mt, 2)) continue;
      if (mt == 2 && p.M <= BM) continue;
      const double item = p.num_kb * (mt * BM + bn) * (p.bk / 64.0) + 0.3 * mt * bn;
      const double cost = rows_kb / mt * nt * (mt * BM + bn) * (p.bk / 64.0) / g_num_sms + 0.5 * item;
      cands[n_cands++] = {bn, mt};
      if (std::max(cost, item) < best_cost) {
        best_cost = std::max(cost, item);
        best = cands[n_cands - 1];
      }
    }
  }
  if (n_cands == 0) return -3;
  {
    const PhasesKey key(N, P, Q, Kp, Cp, H, W, R, S, stride, pad_h, pad_w, packed ? 1 : 0, (mask ? 1 : 0) | (add ? 2 : 0));
    std::unique_lock<std::mutex> lock(g_plan_mutex);
    auto it = g_phases_cache.find(key);
    if (it != g_phases_cache.end()) {
      if (!g_opt.force_mt && it->second.first <= cap) best = it->second;
    } else if (tunable(p, stream)) {
      float best_ms = 1e30f;
      for (int i = 0; i < n_cands; ++i) {
        GemmPhasesParams q = p;
        if (with_b(q, cands[i].first) == 0 &&
            time_launches(stream, [&]() { return run_phases(q, cands[i].first, cands[i].second, Cp, stream); }, &best_ms))
          best = cands[i];
      }
      lock.unlock();      // launches of their own, which look their plans up
      if (time_launches(stream, separate, &best_ms, 0.95f)) best = {0, 0};
      lock.lock();
      g_phases_cache[key] = best;
    }
  }
  if (best.first == 0) return -3;
  rc = with_b(p, best.first);
  return rc ? rc : run_phases(p, best.first, best.second, Cp, stream);
}

// See rb_conv_dgrad_tc; `add_masked`: add is zero already where the mask is.
static int conv_dgrad(const void* dy, int N, int P, int Q, int Kp, const void* w, const void* wt, int Kout, int Cp, int c_valid,
                      int R, int S, int stride, int pad_h, int pad_w, int H, int W, void* dx, const void* add,
                     const void* mask, int add_masked, float* ws, long long ws_bytes, unsigned int* status, cudaStream_t stream) {
  if (stride < 1 || Cp % 32 != 0 || ((uintptr_t)add & 15u)) return -10;
  std::vector<DgradPhase> all, with_taps;
  for (int a = 0; a < stride; ++a)
    for (int b = 0; b < stride; ++b) {
      DgradPhase f;
      f.a = a;
      f.b = b;
      f.r0 = (a + pad_h) % stride;
      f.c0 = (b + pad_w) % stride;
      f.U = f.r0 < R ? (R - f.r0 + stride - 1) / stride : 0;
      f.V = f.c0 < S ? (S - f.c0 + stride - 1) / stride : 0;
      f.pt = f.U - 1 - (a + pad_h - f.r0) / stride;
      f.pl = f.V - 1 - (b + pad_w - f.c0) / stride;
      f.Hp = a < H ? (H - a + stride - 1) / stride : 0;
      f.Wp = b < W ? (W - b + stride - 1) / stride : 0;
      if (f.Hp <= 0 || f.Wp <= 0) continue;
      const bool taps = f.U > 0 && f.V > 0;
      if (stride > 1 && taps && (f.pt < 0 || f.pl < 0)) return -20;
      all.push_back(f);
      if (taps) with_taps.push_back(f);
    }
  // The phases' epilogue and fill_phase_kernel read and write 16 bytes at a time, without a map whose making would say no.
  if (stride > 1 && (((uintptr_t)dx | (uintptr_t)mask) & 15u)) return -10;
  for (const DgradPhase& f : all) {
    if ((f.U > 0 && f.V > 0) || (add == dx && (!mask || add_masked))) continue;
    const int rc = fill_phase((const __nv_bfloat16*)add, (const __nv_bfloat16*)mask, (__nv_bfloat16*)dx, N, f.Hp, f.Wp, stride, f.a,
                              f.b, H, W, Cp, stream);
    if (rc) return rc;
  }
  auto separate = [&]() -> int {
    for (const DgradPhase& f : with_taps) {
      DgradForm dg;
      dg.packed = wt != nullptr;
      dg.taps = R * S;
      dg.base = (f.r0 + stride * (f.U - 1)) * S + f.c0 + stride * (f.V - 1);
      dg.du = -stride * S;
      dg.dv = -stride;
      if (wt) {   // tap t lies at R * S - 1 - t
        dg.base = R * S - 1 - dg.base;
        dg.du = -dg.du;
        dg.dv = -dg.dv;
      }
      dg.sc_stride = stride > 1 ? stride : 0;
      dg.sc_a = f.a;
      dg.sc_b = f.b;
      dg.sc_H = H;
      dg.sc_W = W;
      dg.add = add;
      const int rc = conv_forward_form(dy, N, P, Q, Kp, wt ? wt : w, Cp, f.U, f.V, 1, f.pt, f.pl, f.Hp, f.Wp, dx, Cp, nullptr, 0,
                                       mask, c_valid, Cp, Kout, &dg, nullptr, ws, ws_bytes, status, stream);
      if (rc) return rc;
    }
    return 0;
  };
  // an option that forces a form the one launch does not have is for the launches of the phases
  const bool forced = g_opt.force_halo == 1 || g_opt.force_box == 1 || g_opt.force_wide == 1 || g_opt.force_pair == 1 ||
                      g_opt.force_tail == 1 || g_opt.force_resident >= 0;
  if (with_taps.size() >= 2 && with_taps.size() <= MAX_PHASES && !forced) {
    const int rc = dgrad_phases(dy, N, P, Q, Kp, wt ? wt : w, wt != nullptr, Kout, Cp, c_valid, R, S, stride, pad_h, pad_w, H, W, dx,
                                add, mask, with_taps.data(), (int)with_taps.size(), status, stream, separate);
    if (rc != -3) return rc;
  }
  return separate();
}

// See rb_conv_wgrad_tc: by gemm_tc_kernel.
static int conv_wgrad(const void* x, int N, int H, int W, int Cp, const void* dy, long long lddy, int Kout, int R,
                      int S, int stride, int pad_h, int pad_w, int P, int Q, float* dw, int split_k, int beside,
                      unsigned int* status, cudaStream_t stream) {
  int rc = 0;
  GemmTcParams p;
  memset(&p, 0, sizeof(p));
  p.bk = 64;
  p.lean = beside ? 1 : 0;
  p.M = Kout;
  p.N = R * S * Cp;
  const long long pixels = (long long)N * P * Q;
  p.num_kb = (int)((pixels + p.bk - 1) / p.bk);
  p.wg_cpad = Cp;
  p.epi = EPI_F32_ATOMIC;
  if (split_k > p.num_kb) split_k = p.num_kb;
  while (split_k > 1 && !split_ok(split_k, p.num_kb)) --split_k;
  const int taps = R * S;
  p.wg_ntaps = taps;
  const bool auto_split = split_k <= 0;
  const int fixed = split_k > 0 ? split_k : 0;
  // candidates: (a) one tap per tile, 1..4 channel tiles; (b) several taps side by side when a tap is narrow
  double best_cost = 1e300;
  int best_bn = 0, best_taps = 1;
  auto setup = [Cp, taps](GemmTcParams& q, int bn, int T) {
    q.bn = q.bn_load = bn;
    q.wg_taps = T;
    if (T > 1) {
      q.wg_cw = bn / T;
      q.wg_ctiles = 1;
      q.n_tiles = (taps + T - 1) / T;
    } else {
      q.wg_cw = bn;
      q.wg_ctiles = (Cp + bn - 1) / bn;
      q.n_tiles = taps * q.wg_ctiles;
    }
  };
  for (int nt = 1; nt <= 4; ++nt) {
    int bn = (Cp + nt - 1) / nt;
    bn = (bn + 63) / 64 * 64;
    if (bn > 256) continue;
    setup(p, bn, 1);
    const Plan pl = plan_shape(p, auto_split, fixed, false);
    if (pl.cost < best_cost * 0.97) { best_cost = pl.cost; best_bn = bn; best_taps = 1; }
  }
  const int cw = (Cp + 63) / 64 * 64;
  for (int T = 2; T * cw <= 256 && T <= taps; ++T) {
    setup(p, T * cw, T);
    const Plan pl = plan_shape(p, auto_split, fixed, false);
    // a tile with idle tap slots still pays for them: scale by the slots actually computed
    const double waste = (double)(p.n_tiles * T) / taps;
    if (pl.cost * waste < best_cost * 0.97) { best_cost = pl.cost * waste; best_bn = T * cw; best_taps = T; }
  }
  {  // option force_taps = T takes the T-taps-per-tile candidate when it is feasible
    const int T = g_opt.force_taps;
    if (T == 1 && best_taps != 1) { best_taps = 1; best_bn = cw > 256 ? 256 : cw; }
    if (T > 1 && T * cw <= 256 && T <= taps) { best_taps = T; best_bn = T * cw; }
  }
  if (best_bn == 0) return -3;
  setup(p, best_bn, best_taps);
  p.wgrad = 1;
  p.cv_P = P;
  p.cv_Q = Q;
  p.cv_stride = stride;
  p.cv_lower_h = -pad_h;
  p.cv_lower_w = -pad_w;
  p.cv_S = S;
  // How the pixels of a k-block are loaded:
  //  * a 1 x 1 convolution at stride 1 reads plain rows of both tensors (96 -> 96 on 64 x 54 x 54: 14.0 -> 13.1 us);
  //  * at stride 1, boxes of whole output rows (or pieces of one) of one image where these fill the k-blocks to 95 %,
  //    that is rows of 8, 16, 32 or a multiple of 64: an im2col load takes up to twice as long per pixel row (64 -> 128
  //    on 64 x 128 x 128: 266 -> 218 us; 32 -> 32 on 128 x 32 x 32: 36 -> 31, 5 x 5 on 16 x 16: 29 -> 25);
  //  * else the im2col map: what a box leaves empty is MMA work for nothing (19 x 19 boards, 0.80 full: 46 us from im2col
  //    loads, 48 from boxes; 13 x 13, 0.66 full: 38 against 50).
  const bool plain = taps == 1 && stride == 1 && pad_h == 0 && pad_w == 0 && P == H && Q == W;
  int box_rows = 0, box_w = 0, box_pieces = 1, box_groups = 1;
  if (!plain && stride == 1 && g_opt.force_box != 0) {
    box_pieces = (Q + p.bk - 1) / p.bk;
    box_w = (Q + box_pieces - 1) / box_pieces;
    box_rows = box_pieces > 1 ? 1 : p.bk / Q;
    if (box_rows > P) box_rows = P;
    box_groups = (P + box_rows - 1) / box_rows;
    const double util = (double)P * Q / ((double)box_groups * box_pieces * p.bk);
    if (util < 0.95 && g_opt.force_box != 1) box_rows = 0;
  }
  if (plain) {
    p.a_mode = A_TILED_MN;
    p.b_mode = B_TILED_MN;
    p.wgrad = 0;
    rc = make_map_2d(&p.tm_a, dy, Kout, (uint64_t)pixels, lddy, 64, p.bk, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!rc) rc = make_map_2d(&p.tm_b, x, Cp, (uint64_t)pixels, Cp, 64, p.bk, CU_TENSOR_MAP_SWIZZLE_128B);
  } else if (box_rows > 0) {
    p.a_mode = A_BOX_MN;
    p.b_mode = B_BOX_MN;
    p.wb_rows = box_rows;
    p.wb_w = box_w;
    p.wb_pieces = box_pieces;
    p.wb_groups = box_groups;
    p.wb_pad_h = pad_h;
    p.wb_pad_w = pad_w;
    p.num_kb = N * box_groups * box_pieces;
    if (split_k > p.num_kb) split_k = p.num_kb;
    rc = make_map_nhwc(&p.tm_a, dy, Kout, Q, P, N, lddy, 64, box_w, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!rc) rc = make_map_nhwc(&p.tm_b, x, Cp, W, H, N, Cp, 64, box_w, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
  } else {
    p.a_mode = A_TILED_MN;
    p.b_mode = B_IM2COL_MN;
    const int upper_h = (P - 1) * stride - pad_h - (H - 1);
    const int upper_w = (Q - 1) * stride - pad_w - (W - 1);
    rc = make_map_2d(&p.tm_a, dy, Kout, (uint64_t)pixels, lddy, 64, p.bk, CU_TENSOR_MAP_SWIZZLE_128B);
    if (!rc)
      rc = make_map_im2col(&p.tm_b, x, N, H, W, Cp, -pad_h, -pad_w, upper_h, upper_w, stride, 64, p.bk,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  }
  if (rc) return rc;
  p.epi = EPI_F32_ATOMIC;
  p.n_valid = p.N;
  p.n_store = p.N;
  p.ldd = (long long)R * S * Cp;
  p.D = dw;
  rc = make_map_out_f32(&p.tm_d, dw, p.ldd, Kout, p.ldd);
  if (rc) return rc;
  p.status = status;
  if (split_k > p.num_kb) split_k = p.num_kb;
  while (split_k > 1 && !split_ok(split_k, p.num_kb)) --split_k;
  return launch(p, split_k <= 0, split_k > 0 ? split_k : 0, false, stream);
}

// See rb_conv_wgrad_tc and rb_conv_wgrad_tune.
static int wgrad_by_plan(const void* x, int N, int H, int W, int Cp, const void* dy, long long lddy, int Kout, int R, int S,
                         int stride, int pad_h, int pad_w, int P, int Q, float* dw, int split_k, int beside, bool measure,
                         unsigned int* status, cudaStream_t stream) {
  const int rc = ensure_driver_entry();
  if (rc) return rc;
  auto plain = [&]() {
    return conv_wgrad(x, N, H, W, Cp, dy, lddy, Kout, R, S, stride, pad_h, pad_w, P, Q, dw, split_k, beside, status, stream);
  };
  // options of the other kernel
  const bool forced = g_opt.force_mt || g_opt.force_taps || g_opt.force_box >= 0 || g_opt.force_resident >= 0 ||
                      (g_opt.bn_cap > 0 && g_opt.bn_cap < 256);
  if (stride != 1 || R * S < 2 || split_k > 0 || N < 1 || P < 1 || Q < 1) return measure ? 0 : plain();
  if (measure && (!g_opt.autotune || g_opt.deterministic || g_opt.force_rows >= 0 || forced)) return 1;
  if (g_opt.deterministic || g_opt.force_rows == 0 || forced) return plain();
  auto run = [&](const WgradRowsParams& p) { return run_rows(p, x, N, H, W, dy, lddy, P, Q, dw, status, stream); };
  auto plans = [&]() {
    return rows_plans(N, H, W, Cp, Kout, R, S, pad_h, pad_w, P, Q, beside ? LEAN_TILE_BYTES : TILE_SMEM_BYTES);
  };
  if (g_opt.force_rows > 0) {
    const auto all = plans();
    return all.empty() ? plain() : run(all[std::min<size_t>((size_t)g_opt.force_rows, all.size()) - 1]);
  }
  if (2.0 * N * P * Q * R * S * Cp * Kout < ROWS_MIN_FLOPS) return measure ? 0 : plain();
  const RowsKey key(N, H, W, Cp, Kout, R, S, pad_h, pad_w, P, Q, beside ? 1 : 0);
  std::unique_lock<std::mutex> lock(g_plan_mutex);
  const auto it = g_rows_cache.find(key);
  if (it != g_rows_cache.end()) {
    const WgradRowsParams p = it->second;
    lock.unlock();
    return measure ? 0 : p.rows ? run(p) : plain();
  }
  if (!measure) {
    lock.unlock();
    return plain();
  }
  WgradRowsParams best;
  memset(&best, 0, sizeof(best));
  float best_ms = 1e30f;
  lock.unlock();      // launches of their own, which look their plans up
  time_launches(stream, plain, &best_ms);
  best_ms *= ROWS_MARGIN;
  const auto all = plans();
  for (size_t i = 0; i < all.size() && i < 4; ++i)
    if (time_launches(stream, [&]() { return run(all[i]); }, &best_ms)) best = all[i];
  lock.lock();
  g_rows_cache[key] = best;
  return 0;
}

}  // namespace rb

extern "C" {

// Convolution forward (also a stride-1 data-grad on flipped and transposed filters).
//   x   NHWC bf16 [N][H][W][Cp]      w  bf16 [Kout][R*S][Cp]     y  bf16 [N*P*Q][ldy]
//   base pixel range: lower = -pad_lo, P/Q given by the caller.
int rb_conv_fprop_tc(const void* x, int N, int H, int W, int Cp, const void* w, int Kout, int R, int S, int stride,
                     int pad_h, int pad_w, int P, int Q, void* y, long long ldy, const float* bias, int relu,
                     const void* mask_src, int n_valid, int n_store, float* ws, long long ws_bytes,
                     unsigned int* status, cudaStream_t stream) {
  return conv_forward_form(x, N, H, W, Cp, w, Kout, R, S, stride, pad_h, pad_w, P, Q, y, ldy, bias, relu, mask_src, n_valid,
                           n_store, 0, nullptr, nullptr, ws, ws_bytes, status, stream);
}

// The same followed by a normalisation that is known beforehand, in the epilogue:
// y = act(scale * conv(x) + shift [+ residual]), scale and shift per output column, residual laid out like y; shift and residual
// on a 16-byte boundary.
int rb_conv_fprop_norm(const void* x, int N, int H, int W, int Cp, const void* w, int Kout, int R, int S, int stride,
                       int pad_h, int pad_w, int P, int Q, void* y, long long ldy, const float* scale, const float* shift,
                       const void* residual, int relu, int n_valid, int n_store, float* ws, long long ws_bytes,
                       unsigned int* status, cudaStream_t stream) {
  if (!scale || !shift || ((uintptr_t)shift & 15u) || ((uintptr_t)residual & 15u)) return -10;
  const NormForm form = {scale, residual};
  return conv_forward_form(x, N, H, W, Cp, w, Kout, R, S, stride, pad_h, pad_w, P, Q, y, ldy, shift, relu, nullptr, n_valid,
                           n_store, 0, nullptr, &form, ws, ws_bytes, status, stream);
}

// Convolution data-grad: dx[N][H][W][Cp] = mask(add + the gradient), from dy NHWC bf16 [N][P][Q][Kp] and the forward
// filters w bf16 [Kout][R*S][Cp]. Channels >= c_valid of dx are written as zeros.
//   stride 1: a forward convolution of dy, its filters read in place. stride s: s x s output phases; phase (a, b), the
//   positions (s i + a, s j + b), is a stride-1 convolution of dy with every s-th filter tap, whose rows the epilogue
//   scatters. A phase without taps gets mask(add), and nothing has to be done when add is dx itself and there is no mask.
//   wt: null, or the filters transposed and flipped (rb_pack_dgrad_filters): then these are read, as a K-major operand.
//   add, mask: optional, layout of dx; add may be dx. All three on a 16-byte boundary (else an error). Returns -20 for a strided geometry with a
//   phase of negative padding.
int rb_conv_dgrad_tc(const void* dy, int N, int P, int Q, int Kp, const void* w, const void* wt, int Kout, int Cp, int c_valid,
                     int R, int S, int stride, int pad_h, int pad_w, int H, int W, void* dx, const void* add,
                     const void* mask, float* ws, long long ws_bytes, unsigned int* status, cudaStream_t stream) {
  return conv_dgrad(dy, N, P, Q, Kp, w, wt, Kout, Cp, c_valid, R, S, stride, pad_h, pad_w, H, W, dx, add, mask, 0, ws, ws_bytes,
                    status, stream);
}

// dx += mask(the gradient) where dx is zero already at the places that the mask zeroes: positions that no filter tap reaches
// stay as they are, without a launch that would write them again.
int rb_conv_dgrad_onto_tc(const void* dy, int N, int P, int Q, int Kp, const void* w, const void* wt, int Kout, int Cp,
                          int c_valid, int R, int S, int stride, int pad_h, int pad_w, int H, int W, void* dx, const void* mask,
                          float* ws, long long ws_bytes, unsigned int* status, cudaStream_t stream) {
  return conv_dgrad(dy, N, P, Q, Kp, w, wt, Kout, Cp, c_valid, R, S, stride, pad_h, pad_w, H, W, dx, dx, mask, 1, ws, ws_bytes,
                    status, stream);
}

// Convolution weight-grad:  dw[Kout][R*S][Cp] (fp32) (+)= sum over pixels dy[pix][k] * x[pix shifted by tap][c].
//   The result is always accumulated into dw (red.add), so dw holds zeros or the running gradient on entry.
//   beside: the launch is to leave room on the SMs for kernels that run at the same time (the lean instantiation, or less
//   shared memory).
//   Which kernel runs is what rb_conv_wgrad_tune has measured for the shape; without a measurement, with an explicit split and
//   with `deterministic` (measurements must not choose the order of additions), gemm_tc_kernel.
int rb_conv_wgrad_tc(const void* x, int N, int H, int W, int Cp, const void* dy, long long lddy, int Kout, int R,
                     int S, int stride, int pad_h, int pad_w, int P, int Q, float* dw, int split_k, int beside,
                     unsigned int* status, cudaStream_t stream) {
  return wgrad_by_plan(x, N, H, W, Cp, dy, lddy, Kout, R, S, stride, pad_h, pad_w, P, Q, dw, split_k, beside, false, status, stream);
}

// Times gemm_tc_kernel and the first four plans of wgrad_rows_kernel by its model on these operands, which are scratch (dw is
// added into many times), and remembers which was the fastest. Synchronises the stream: never inside a capture. Does nothing for
// a shape that has been measured, or that has no such plans. Returns 1 where an option is in the way of measuring: to be asked
// again.
int rb_conv_wgrad_tune(const void* x, int N, int H, int W, int Cp, const void* dy, long long lddy, int Kout, int R, int S,
                       int pad_h, int pad_w, int P, int Q, float* dw, int beside, unsigned int* status, cudaStream_t stream) {
  return wgrad_by_plan(x, N, H, W, Cp, dy, lddy, Kout, R, S, 1, pad_h, pad_w, P, Q, dw, 0, beside, true, status, stream);
}

// Planner options by name (see GemmOptions); returns 0, or -1 for an unknown name.
int rb_gemm_set_option(const char* name, int value) {
  options_from_env();
  int* slot = option_slot(name);
  if (!slot) return -1;
  *slot = value;
  return 0;
}

int rb_gemm_get_option(const char* name, int* value) {
  options_from_env();
  int* slot = option_slot(name);
  if (!slot) return -1;
  *value = *slot;
  return 0;
}

// Tuning mode: while on, a bf16-epilogue launch of a shape without a cached plan times its candidates (it
// synchronises the stream, so it must not run inside a stream capture) and caches the winner.
int rb_gemm_tune_mode(int on) {
  g_tune_mode = on ? 1 : 0;
  return 0;
}

int rb_gemm_clear_plans() {
  std::lock_guard<std::mutex> lock(g_plan_mutex);
  g_plan_cache.clear();
  g_bn_cache.clear();
  g_phases_cache.clear();
  g_rows_cache.clear();
  return 0;
}

// out[0..7]: the role-profile counters (all zero in a build without -DRB_GEMM_PROFILE, returns 1 then); cleared on read.
int rb_gemm_role_profile(unsigned long long* out) {
  for (int i = 0; i < 8; ++i) out[i] = 0ull;
#ifdef RB_GEMM_PROFILE
  cudaDeviceSynchronize();
  if (cudaMemcpyFromSymbol(out, g_role_cycles, sizeof(unsigned long long) * 8) != cudaSuccess) return -1;
  const unsigned long long zeros[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (cudaMemcpyToSymbol(g_role_cycles, zeros, sizeof(zeros)) != cudaSuccess) return -1;
  return 0;
#else
  return 1;
#endif
}

// Runtime error code of the last launch that failed (a launcher's return value of -4), 0 if none did.
int rb_gemm_last_cuda_error() { return g_last_cuda_error; }

// out[0..8]: the tile plan of the most recent launch, see g_last_launch.
int rb_gemm_last_launch(int* out) {
  memcpy(out, g_last_launch, sizeof(g_last_launch));
  return 0;
}

int rb_num_sms() {
  ensure_driver_entry();
  return g_num_sms;
}

}  // extern "C"
