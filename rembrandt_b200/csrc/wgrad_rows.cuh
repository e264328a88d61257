// Weight-gradient of a stride-1 convolution from whole rows of positions (included by gemm_tc.cu).
//
//   dw[k][tap][c] += sum over positions f of dy[f][k] * x[f + offset of the tap][c]
//
// A stage in shared memory is a chunk of output rows: boxes of dy and of x with 64 or 32 channels per position, as TMA writes
// them, zeros outside the image. Both are MN-major operands (the reduction runs over positions), so filter tap s of a row is the
// same box of x one position further on: the operand descriptor starts there, and one MMA covers several taps side by side, its
// 64- or 32-column blocks one position apart. What is loaded per chunk serves S taps times one or more blocks of channels
// instead of one tap: tap by tap, 128 -> 128 channels ask for 94 bytes per cycle and SM from the L2, which delivers 41; this way
// for 41. Us a launch (back to back, inputs larger than the L2), tap by tap and from rows: 3 x 3, 128 -> 128 on 256 x 19 x 19:
// 30.4, 25.3; 64 -> 64 on 32 x 64 x 64: 24.1, 16.7; 128 -> 128 on 32 x 32 x 32: 16.1, 12.8; 256 -> 384 on 128 x 13 x 13: 42.7, 36.2;
// 64 -> 128 on 64 x 128 x 128: 152, 119; 32 -> 32 on 128 x 32 x 32: 24.1, 13.1; 5 x 5, 32 -> 32 on 128 x 16 x 16: 23.4, 10.0;
// 96 -> 256 on 128 x 27 x 27: 104, 88. Where tap by tap loads two sub-tiles per item (256 and more channels on both sides, rows that
// fill its k-blocks), it is as fast (3 x 3, 512 -> 512 on 64 x 32 x 32: 0.97 of the measured peak either way) and stays.
// A launch takes ~4 us to start and drain, and the additions into dw 2.5 us per 192 columns (all CTAs add 14 MB at 5.5 TB/s): with
// less than a few us of MMAs per CTA these are what bounds it.
//
// How positions line up in the two operands:
//   by rows   every output row is a reduction of its own, as many positions as the row has, rounded up to 16 (dy is zero there)
//   in a run  the rows of a chunk lie one after the other, the zero columns that the filter reaches included (those at a row's
//             end shared with the next row's beginning), and the whole chunk is one reduction: what bounds small images, whose
//             rows are no multiple of 16 (13 x 13: 192 positions for 169 outputs instead of 208). Positions behind the boxes are
//             zeros from the start of the kernel, in both operands.
// Either way zero columns of dy meet pixels at the border, which belong to no output of that tap. Finite ones add nothing; an
// infinity or a NaN would turn sums into NaN that it has no part in. So a slab with a sum that is not finite is not added but taken
// again, over the outputs alone (rows_again). For finite sums that costs the test: nothing to 0.5 us a launch (3 x 3, 32 -> 32 on
// 128 x 16 x 16: 7.3 -> 7.5 us; 64 -> 64 on 32 x 64 x 64: 17.4 -> 17.5; 128 -> 128 on 256 x 19 x 19: 26.1 -> 26.2).
//
// A work item is 128 output channels x (filter rows x blocks of channels) of at most 512 accumulator columns over a range of
// chunks; items that share a range run at the same time. The sums are added into dw by TMA.
// Warp 0 loads, warp 1 issues, warps 2 - 9 add up, as in gemm_tc_kernel.
#pragma once

struct alignas(64) WgradRowsParams {
  CUtensorMap tm_x, tm_dy, tm_dw;
  int work;                          // items
  int m_tiles, groups_r, groups_c;   // item = (range of chunks, block group, filter row group, 128 output channels)
  int splits, chunks;                // ranges, chunks in all
  int row_groups, rows, images;      // a chunk: `rows` output rows of `images` images; row groups per image
  int nr, ncb;                       // filter rows and channel blocks per item
  int xw, dyw;                       // channels per block of x and dy: 64 (128-byte positions) or 32
  int per_mma;                       // taps side by side in one MMA
  int R, S, cblocks, pad_h, pad_w, Cp, Kout;
  int segs, steps;                   // reductions per chunk, 16 positions at a time
  int dy_seg, x_seg;                 // 16-byte units from one to the next
  int x_row;                         // 16-byte units from filter row to filter row
  int dy_blocks;                     // blocks of dy per item
  int dy_block, x_block;             // bytes per block of a stage
  int dy_bytes, x_bytes;             // bytes that a box brings
  int stages, tile_bytes;
  int clear;                         // shared memory behind the boxes has to be zeros
  const __nv_bfloat16 *x, *dy;       // for sums that are taken again
  long long lddy;
  int N, H, W, P, Q;
  unsigned int* status;
};

// The MMAs of one 16-position step (or four) into NM accumulators.
template <int KK, int NM>
__device__ __forceinline__ void rows_steps(const uint32_t (&d)[NM], const uint32_t (&off)[NM], const uint32_t (&idesc)[NM],
                                           uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t a_step,
                                           uint32_t b_step, uint32_t accumulate) {
#pragma unroll
  for (int j = 0; j < NM; ++j)
    tc_mma_steps<KK, false>(d[j], a_lo, a_hi, b_lo + off[j], b_hi, a_step, b_step, idesc[j], accumulate);
}

template <int NM>
__device__ __forceinline__ bool rows_item(const WgradRowsParams& p, SharedCtl* ctl, uint32_t tiles_u32, uint32_t stage_bytes,
                                          uint32_t tmem, int ncb, int c0, int c1, int& s, uint32_t& ph) {
  uint32_t d[NM], off[NM], idesc[NM];
  const int per = p.per_mma, pieces = (p.S + per - 1) / per, pos = p.xw * 2;      // pos: bytes of a position of x
#pragma unroll
  for (int j = 0; j < NM; ++j) {
    const int unit = j / pieces, s0 = (j - unit * pieces) * per, taps = min(per, p.S - s0);
    const int ri = unit / ncb, cb = unit - ri * ncb;
    d[j] = tmem + (uint32_t)((unit * p.S + s0) * p.xw);
    off[j] = (uint32_t)((cb * p.x_block >> 4) + ri * p.x_row + s0 * (pos >> 4));
    idesc[j] = make_idesc_bf16(BM, (uint32_t)(p.xw * taps), 1u, 1u);
  }
  // blocks of A: dy blocks (one block: rows past the layer's channels are not stored); of B: one position apart
  const uint32_t dpos = (uint32_t)p.dyw * 2u;
  const uint64_t a_desc = make_smem_desc(0u, p.dy_blocks > 1 ? (uint32_t)p.dy_block : dpos, 8u * dpos, p.dyw == 64 ? 2u : 4u);
  const uint64_t b_desc = make_smem_desc(0u, (uint32_t)pos, 8u * (uint32_t)pos, p.xw == 64 ? 2u : 4u);
  const uint32_t a_step = dpos, b_step = (uint32_t)pos;      // 16 positions, in 16-byte units
  const uint32_t a_hi = (uint32_t)(a_desc >> 32), b_hi = (uint32_t)(b_desc >> 32);
  uint32_t accumulate = 0u;
  for (int c = c0; c < c1; ++c) {
    if (!ctl_wait_warp(ctl, &ctl->full[s], ph, p.status)) return false;
    tc_fence_after();
    uint32_t a = (uint32_t)a_desc | ((tiles_u32 + (uint32_t)s * stage_bytes) >> 4);
    uint32_t b = (uint32_t)b_desc | ((tiles_u32 + (uint32_t)s * stage_bytes + (uint32_t)(p.dy_blocks * p.dy_block)) >> 4);
    for (int seg = 0; seg < p.segs; ++seg, a += (uint32_t)p.dy_seg, b += (uint32_t)p.x_seg) {
      uint32_t a1 = a, b1 = b;
      int st = p.steps;
      for (; st >= 4; st -= 4, a1 += 4u * a_step, b1 += 4u * b_step) {
        rows_steps<4, NM>(d, off, idesc, a1, a_hi, b1, b_hi, a_step, b_step, accumulate);
        accumulate = 1u;
      }
      if (st >= 2) {
        rows_steps<2, NM>(d, off, idesc, a1, a_hi, b1, b_hi, a_step, b_step, accumulate);
        accumulate = 1u;
        a1 += 2u * a_step;
        b1 += 2u * b_step;
        st -= 2;
      }
      if (st) {
        rows_steps<1, NM>(d, off, idesc, a1, a_hi, b1, b_hi, a_step, b_step, accumulate);
        accumulate = 1u;
      }
    }
    tc_commit(&ctl->empty[s]);
    if (++s == p.stages) { s = 0; ph ^= 1u; }
  }
  return true;
}

// Item `work`: output channels, filter rows, channel blocks, chunks.
struct RowsItem {
  int m0, r0, cb0, ncb, c0, c1;
};
__device__ __forceinline__ RowsItem rows_item_of(const WgradRowsParams& p, int work) {
  RowsItem it;
  const int groups = p.groups_r * p.groups_c, t = work / p.m_tiles, sp = t / groups, g = t - sp * groups, gc = g / p.groups_r;
  it.m0 = (work - t * p.m_tiles) * BM;
  it.r0 = (g - gc * p.groups_r) * p.nr;
  it.cb0 = gc * p.ncb;
  it.ncb = min(p.ncb, p.cblocks - it.cb0);
  it.c0 = (int)((long long)sp * p.chunks / p.splits);
  it.c1 = (int)((long long)(sp + 1) * p.chunks / p.splits);
  return it;
}

// What accumulator column `c` of an item holds: channel `chan` of tap (row r, `tap`).
struct RowsColumn {
  int r, tap, chan;
};
__device__ __forceinline__ RowsColumn rows_column_of(const WgradRowsParams& p, const RowsItem& it, int c) {
  const int unit_cols = p.S * p.xw, unit = c / unit_cols, in_unit = c - unit * unit_cols, ri = unit / it.ncb;
  RowsColumn at;
  at.r = it.r0 + ri;
  at.tap = in_unit / p.xw;
  at.chan = (it.cb0 + unit - ri * it.ncb) * p.xw + in_unit - at.tap * p.xw;
  return at;
}

// A slab of 32 accumulator columns (c ...) of an item on its way to dw: TMEM -> registers -> the warp's staging buffer.
__device__ __forceinline__ void rows_load(uint32_t tmem, int c, uint32_t (&v)[32]) {
  tmem_ld_32x32(tmem + (uint32_t)c + ((threadIdx.x >> 5 & 3u) << 21), v);
  tmem_ld_wait();
}
__device__ __forceinline__ void rows_stage(uint8_t* staged, const uint32_t (&v)[32]) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) tma_store_wait_read<0>();
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 8; ++q)
    *reinterpret_cast<uint4*>(staged + lane * 128 + ((q ^ (lane & 7)) * 16)) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}
__device__ __forceinline__ bool rows_add(const WgradRowsParams& p, uint8_t* staged, const RowsItem& it, const RowsColumn& at, bool not_yet) {
  fence_proxy_async_smem();
  __syncwarp();
  if (__any_sync(0xffffffffu, not_yet)) return false;
  if ((threadIdx.x & 31) == 0) {
    tma_reduce_add_2d(&p.tm_dw, staged, (at.r * p.S + at.tap) * p.Cp + at.chan, it.m0 + (int)(threadIdx.x >> 5 & 3) * 32);
    tma_store_commit();
  }
  return true;
}

// A slab with sums that are not finite: these are taken again, over output positions, pixels outside the image as zeros. In
// doubles, so that the order does not matter; four columns at a time and one position after the other: slow, and only ever needed
// for infinities and NaN. A sum that has become NaN is done: a launch whose operands are all NaN takes 1 to 2 ms, one with a single
// infinite pixel 1 to 17, and where every sum is infinite and none NaN (512 -> 512 on 64 x 32 x 32, 22016 positions an item) 0.5 s,
// which is below the limit that waits have.
__device__ __forceinline__ void rows_again(const WgradRowsParams& p, uint8_t* staged, uint32_t tmem, int work, int c) {
  const RowsItem it = rows_item_of(p, work);
  const RowsColumn col = rows_column_of(p, it, c);
  const int lane = threadIdx.x & 31, m = it.m0 + (int)(threadIdx.x >> 5 & 3) * 32 + lane;
  {
    uint32_t v[32];
    rows_load(tmem, c, v);
    rows_stage(staged, v);
  }
#pragma unroll 1
  for (int j = 0; j < 32 && m < p.Kout; j += 4) {
    float* const at = reinterpret_cast<float*>(staged + lane * 128 + ((j / 4) ^ (lane & 7)) * 16);
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    uint32_t again = 0u;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if ((__float_as_uint(at[e]) & 0x7f800000u) == 0x7f800000u) again |= 1u << e;
    uint32_t open = again;      // those that are not NaN so far
    for (int k = it.c0; k < it.c1 && open; ++k) {
      const int grp = k / p.row_groups, h0 = (k - grp * p.row_groups) * p.rows;
      const int n1 = min(p.N, (grp + 1) * p.images), h1 = min(p.P, h0 + p.rows);
      for (int n = grp * p.images; n < n1; ++n)
        for (int h = h0; h < h1; ++h) {
          const int y = h + col.r - p.pad_h, w0 = p.pad_w - col.tap;
          const int w1 = y >= 0 && y < p.H ? p.W : 0;      // pixels of this row
          const __nv_bfloat16* dy = p.dy + ((long long)n * p.P + h) * p.Q * p.lddy + m;
          const __nv_bfloat16* x = p.x + (((long long)n * p.H + y) * p.W - w0) * p.Cp + col.chan + j;
#pragma unroll 1
          for (int q = 0; q < p.Q; ++q, dy += p.lddy, x += p.Cp) {
            const uint2 four = q >= w0 && q - w0 < w1 ? *reinterpret_cast<const uint2*>(x) : make_uint2(0u, 0u);
            const double d = (double)__bfloat162float(*dy);
            sum[0] += d * (double)__uint_as_float(four.x << 16);
            sum[1] += d * (double)__uint_as_float(four.x & 0xffff0000u);
            sum[2] += d * (double)__uint_as_float(four.y << 16);
            sum[3] += d * (double)__uint_as_float(four.y & 0xffff0000u);
          }
        }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (isnan(sum[e])) open &= ~(1u << e);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (again & (1u << e)) at[e] = (float)sum[e];
  }
  rows_add(p, staged, it, col, false);
}

__global__ void __maxnreg__(LEAN_MAX_REGS) wgrad_rows_kernel(const __grid_constant__ WgradRowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = tiles + p.tile_bytes;
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(staging + STAGING_BYTES);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t stage_bytes = (uint32_t)(p.dy_blocks * p.dy_block + p.ncb * p.x_block);
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->acc_full[0], 1);
    mbar_init(&ctl->acc_empty[0], EPI_WARPS);
    ctl->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&p.tm_x);
    tma_prefetch_desc(&p.tm_dy);
    tma_prefetch_desc(&p.tm_dw);
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
  }
  if (p.clear) {
    for (uint32_t i = threadIdx.x; i < (uint32_t)p.tile_bytes / 16; i += GEMM_THREADS)
      *reinterpret_cast<uint4*>(tiles + i * 16) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  if (warp == 0) {
    int s = 0, issued = 0;
    uint32_t ph = 0;
    bool ok = true;
    pdl_prolog();
    for (int work = blockIdx.x; work < p.work && ok; work += gridDim.x) {
      const RowsItem it = rows_item_of(p, work);
      const int boxes = p.dy_blocks + it.ncb;
      int grp = it.c0 / p.row_groups, rg = it.c0 - grp * p.row_groups;
      for (int c = it.c0; c < it.c1; ++c) {
        int w_ok = 1;
        if (lane == 0) {
          w_ok = ctl_wait(ctl, &ctl->empty[s], ph ^ 1u, p.status) ? 1 : 0;
          if (w_ok) mbar_expect_tx(&ctl->full[s], (uint32_t)(p.dy_blocks * p.dy_bytes + it.ncb * p.x_bytes));
        }
        if (!__shfl_sync(0xffffffffu, w_ok, 0)) { ok = false; break; }
        uint8_t* const stage = tiles + (uint32_t)s * stage_bytes;
        if (lane < p.dy_blocks)
          tma_load_4d(stage + lane * p.dy_block, &p.tm_dy, &ctl->full[s], it.m0 + p.dyw * lane, 0, rg * p.rows, grp * p.images);
        else if (lane < boxes)
          tma_load_4d(stage + p.dy_blocks * p.dy_block + (lane - p.dy_blocks) * p.x_block, &p.tm_x, &ctl->full[s],
                      (it.cb0 + lane - p.dy_blocks) * p.xw, -p.pad_w, rg * p.rows + it.r0 - p.pad_h, grp * p.images);
        __syncwarp();
        if (++rg == p.row_groups) { rg = 0; ++grp; }
        ++issued;
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
    }
    if (!ok && lane == 0) {
      // drain: wait (bounded) until the copies already issued have landed
      const int back = min(issued, p.stages);
      for (int i = 0; i < back; ++i) {
        if (s == 0) { s = p.stages; ph ^= 1u; }
        --s;
        mbar_wait_bounded(&ctl->full[s], ph, 100000000ull);
      }
    }
  } else if (warp == 1) {
    // (waits for the first stage, whose load waits for the kernels before this one)
    int s = 0;
    uint32_t ph = 0, acc_ph = 0;
    const int pieces = (p.S + p.per_mma - 1) / p.per_mma;
    const uint32_t tiles_u32 = smem_u32(tiles);
    for (int work = blockIdx.x; work < p.work; work += gridDim.x) {
      const RowsItem it = rows_item_of(p, work);
      if (!ctl_wait_warp(ctl, &ctl->acc_empty[0], acc_ph ^ 1u, p.status)) break;
      tc_fence_after();
      bool ok;
      switch (p.nr * it.ncb * pieces) {
        case 1: ok = rows_item<1>(p, ctl, tiles_u32, stage_bytes, tmem_base, it.ncb, it.c0, it.c1, s, ph); break;
        case 2: ok = rows_item<2>(p, ctl, tiles_u32, stage_bytes, tmem_base, it.ncb, it.c0, it.c1, s, ph); break;
        case 3: ok = rows_item<3>(p, ctl, tiles_u32, stage_bytes, tmem_base, it.ncb, it.c0, it.c1, s, ph); break;
        default: ok = rows_item<4>(p, ctl, tiles_u32, stage_bytes, tmem_base, it.ncb, it.c0, it.c1, s, ph); break;
      }
      if (!ok) break;
      tc_commit(&ctl->acc_full[0]);
      acc_ph ^= 1u;
    }
  } else if (warp < 2 + EPI_WARPS) {
    pdl_prolog();
    const int lane_base = (warp & 3) * 32, col_half = (warp - 2) >> 2;
    uint8_t* const stg = staging + (warp - 2) * 4096;
    uint32_t acc_ph = 0;
    for (int work = blockIdx.x; work < p.work; work += gridDim.x) {
      const RowsItem it = rows_item_of(p, work);
      if (!ctl_wait(ctl, &ctl->acc_full[0], acc_ph, p.status)) break;
      tc_fence_after();
      const int cols = p.nr * it.ncb * p.S * p.xw;
      uint32_t odd = 0u;      // slabs that rows_again takes
      for (int c = col_half * 32; c < cols; c += 64) {
        const RowsColumn at = rows_column_of(p, it, c);
        if (at.chan >= p.Cp || it.m0 + lane_base >= p.Kout) continue;
        uint32_t v[32];
        rows_load(tmem_base, c, v);
        rows_stage(stg, v);
        // One value that is not finite leaves the sum of all so (a sum that overflows is looked at for nothing). Worked out while
        // the stores are on their way, and asked in place of the warp's own barrier.
        float all[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 32; ++q) all[q & 3] += __uint_as_float(v[q]);
        float one = (all[0] + all[1]) + (all[2] + all[3]);
        asm volatile("" : "+f"(one));
        const bool bad = (__float_as_uint(one) & 0x7f800000u) == 0x7f800000u && it.m0 + lane_base + lane < p.Kout;
        if (!rows_add(p, stg, it, at, bad)) odd |= 1u << (c >> 5);
      }
      for (; odd; odd &= odd - 1) rows_again(p, stg, tmem_base, work, (__ffs(odd) - 1) * 32);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->acc_empty[0]);
      acc_ph ^= 1u;
    }
    if (lane == 0) tma_store_wait_all<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}
