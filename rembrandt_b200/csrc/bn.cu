// Spatial batch normalisation on NHWC bf16 tensors (rows = N*H*W, columns = channels):
//   forward (training): per-channel batch mean / inverse std, running-statistic update with a caller-given
//   factor, then y = act(gamma * xhat + beta [+ residual]);  inference uses the running statistics.
//   backward: dgamma = sum dy*xhat, dbeta = sum dy, dx = gamma*istd/M * (M*dy - dbeta - xhat*dgamma).
// Replaces cuDNN BatchNormalizationForwardTraining/Inference/Backward as used by the reference's
// BNormConv2d and residual operators, including its "add into a copy of x" residual trick
// (src/operator/conv.rs:494-535,595-608,1601-1644).
#include "launch.cuh"
#include "common.cuh"

namespace rb {

// How the kernels below cover a [rows][C] tensor: a thread owns one group of 8 channels (16 bytes) for its whole life
// and walks down the rows, so everything that belongs to a channel (shift, mean, scale, ...) is fetched once and kept
// in registers. A block holds `gpb` = min(C / 8, 256) neighbouring groups x 256 / gpb rows (rounded down: 96 channels
// use 252 of its 256 threads), blockIdx.y covers wider tensors slab by slab. Any multiple of 8 channels fits.
struct RowCover {
  int gpb, rl, g, rr, c0;
  bool live;
};
__device__ __forceinline__ RowCover row_cover(int C) {
  RowCover w;
  const int cg = C >> 3;
  w.gpb = cg < 256 ? cg : 256;
  w.rl = 256 / w.gpb;
  w.rr = threadIdx.x / w.gpb;
  w.g = threadIdx.x - w.rr * w.gpb;
  w.c0 = (blockIdx.y * w.gpb + w.g) * 8;
  w.live = w.rr < w.rl && w.c0 < C;
  return w;
}
static inline dim3 row_grid(long long rows, int C, int rows_per_thread, int max_blocks) {
  const int cg = C / 8, gpb = cg < 256 ? cg : 256, rl = 256 / gpb;
  const int slabs = (cg + gpb - 1) / gpb;
  long long b = (rows + (long long)rl * rows_per_thread - 1) / ((long long)rl * rows_per_thread);
  if (b > max_blocks / slabs) b = max_blocks / slabs;
  if (b < 1) b = 1;
  return dim3((unsigned)b, (unsigned)slabs);
}

// Scratch of the two-launch forms: two buffers of 2 * C sums and two words. A call adds into the buffer named by `next`;
// the kernel after the reduction reads the sums from the buffer the reduction noted in `used`, clears the other buffer,
// whose sums belong to the call before and have been read, and names it for the next call. Each word is written by one
// kernel and read by the other, so no block can see a change of its own launch, and calls that share a scratch only have
// to be ordered on one stream. What this saves over a kernel that finishes the sums is a launch between two dependent
// ones (2.5 us); letting the reduction's last block finish them instead costs 3.5 us (fence, counter, reload).
struct BnScratch {
  float* sums;            // null: `plain` holds the sums and is cleared by whoever finishes them
  unsigned int* next;
  unsigned int* used;
};
static inline BnScratch bn_scratch(float* ws, int C) {
  return BnScratch{ws, (unsigned int*)(ws + 4 * (long long)C), (unsigned int*)(ws + 4 * (long long)C) + 16};
}

// Where the batch statistics go and how the running ones follow them.
struct BnStats {
  float* mean;
  float* istd;
  float* run_mean;
  float* run_var;
  const unsigned int* step_ptr;
  float eps, factor;
  int avg_kind;
};

// mean/istd from the sums; running statistics: r = (1-f) r + f batch ; sums re-zeroed.
// With a step counter (`step_ptr`, the network's device-side count of training steps) the factor is derived on
// the device, so that a captured CUDA graph keeps averaging correctly: avg_kind 1 = cumulative 1 / (1 + t),
// avg_kind 2 = exponential `factor` with 1 at t = 0; avg_kind 0 (or no counter) uses `factor` as given.
// `inv_rows` = 1 / rows: every thread of the apply kernel does this for its eight channels, and two divisions per channel
// were half of its instructions (92416 x 128: 18 us, 2.4 instructions per cycle and SM).
__device__ __forceinline__ void bn_batch_stats(float s0, float s1, float shift, float inv_rows, float eps, float& mean,
                                               float& var, float& istd) {
  const float ms = s0 * inv_rows;             // mean of the shifted values
  var = fmaxf(s1 * inv_rows - ms * ms, 0.f);
  mean = shift + ms;
  istd = rsqrtf(var + eps);
}
__device__ __forceinline__ void bn_store_stats(const BnStats& f, int c, long long rows, float mean, float var,
                                               float istd) {
  float factor = f.factor;
  if (f.step_ptr && f.avg_kind) {
    const unsigned int t = *f.step_ptr;
    factor = f.avg_kind == 1 ? 1.f / (1.f + (float)t) : (t == 0u ? 1.f : factor);
  }
  f.mean[c] = mean;
  f.istd[c] = istd;
  if (f.run_mean) {
    const float unbiased = rows > 1 ? var * (float)rows / (float)(rows - 1) : var;
    f.run_mean[c] = (1.f - factor) * f.run_mean[c] + factor * mean;
    f.run_var[c] = (1.f - factor) * f.run_var[c] + factor * unbiased;
  }
}

// Forward: sums[c] += sum (x - k_c), sums[C+c] += sum (x - k_c)^2 with the shift k_c = x[0][c] (the channel's value in
// the first row). Shifted sums keep the variance E[(x-k)^2] - E[x-k]^2 free of the cancellation that plain
// E[x^2] - E[x]^2 suffers when a channel's mean is large against its spread (the shift lies inside the data's range,
// so both terms are of the order of the variance). Backward: sums of dy and dy * xhat.
// Bound by load latency at the sizes of a training step (2 - 24 MB, mostly in L2): eight 16-byte loads are in flight per
// thread (92416 x 128: forward 17 -> 10 us against one load at a time).
template <int BACKWARD, int MASK>
__global__ void __launch_bounds__(256) bn_reduce_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dy,
                                                        const bf16* __restrict__ y, const float* __restrict__ mean,
                                                        const float* __restrict__ istd, long long rows, int C,
                                                        float* __restrict__ plain, const BnScratch ws) {
  pdl_prolog();
  constexpr int U = BACKWARD ? 4 : 8;
  __shared__ float red0[2048];
  __shared__ float red1[2048];
  const RowCover w = row_cover(C);
  float* sums = plain;
  if (ws.sums) {
    const unsigned int b = *ws.next & 1u;
    sums = ws.sums + b * (2 * (long long)C);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *ws.used = b;
  }
  float a0[8], a1[8], mu[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { a0[j] = 0.f; a1[j] = 0.f; }
  if (w.live) {
    if (BACKWARD) {
#pragma unroll
      for (int j = 0; j < 8; ++j) mu[j] = mean[w.c0 + j];
    } else {
      load8(x + w.c0, mu);   // the shift: row 0 of these channels
    }
    const long long step = (long long)gridDim.x * w.rl;
    for (long long r = (long long)blockIdx.x * w.rl + w.rr; r < rows; r += step * U) {
      uint4 xv[U], gv[BACKWARD ? U : 1], yv[MASK ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long ru = r + step * u;
        if (ru < rows) {
          const long long o = ru * C + w.c0;
          xv[u] = *reinterpret_cast<const uint4*>(x + o);
          if (BACKWARD) gv[u] = *reinterpret_cast<const uint4*>(dy + o);
          if (MASK) yv[u] = *reinterpret_cast<const uint4*>(y + o);   // ReLU after the normalisation
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r + step * u >= rows) break;
        float v[8];
        unpack8(xv[u], v);
        if (!BACKWARD) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float d = v[j] - mu[j];
            a0[j] += d;
            a1[j] += d * d;
          }
        } else {
          float g[8];
          unpack8(gv[u], g);
          if (MASK) {
            float yy[8];
            unpack8(yv[u], yy);
#pragma unroll
            for (int j = 0; j < 8; ++j) if (!(yy[j] > 0.f)) g[j] = 0.f;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) { a0[j] += g[j]; a1[j] += g[j] * (v[j] - mu[j]); }
        }
      }
    }
    if (BACKWARD) {
#pragma unroll
      for (int j = 0; j < 8; ++j) a1[j] *= istd[w.c0 + j];
    }
  }
  // red[rr][channel of the block]: rl * gpb * 8 <= 2048 floats
  if (w.rr < w.rl) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      red0[(w.rr * w.gpb + w.g) * 8 + j] = a0[j];
      red1[(w.rr * w.gpb + w.g) * 8 + j] = a1[j];
    }
  }
  __syncthreads();
  const int width = w.gpb * 8, base = blockIdx.y * width;
  for (int c = threadIdx.x; c < width && base + c < C; c += 256) {
    float s0 = 0.f, s1 = 0.f;
    for (int k = 0; k < w.rl; ++k) { s0 += red0[k * width + c]; s1 += red1[k * width + c]; }
    atomicAdd(sums + base + c, s0);
    atomicAdd(sums + C + base + c, s1);
  }
}

static void launch_bn_reduce(const bf16* x, const bf16* dy, const bf16* y, const float* mean, const float* istd,
                             long long rows, int C, float* plain, int backward, const BnScratch& ws, cudaStream_t st) {
  // Two blocks per SM: every block adds 2 * C sums to the same addresses, and in the backward pass of a captured step the
  // weight-gradient beside it leaves room for one or two. Fastest or equal without a neighbour too, on the 14 sizes tried: forward
  // (us a layer with its application; 1, 2, 3, 4 blocks) 92416 x 128: 20.7, 18.9, 18.7, 20.9, 131072 x 64: 17.0, 15.2, 15.5, 16.6,
  // 8192 x 64: 6.0, 5.9, 6.0, 6.0; backward (2, 4) 92416 x 128: 24.1, 26.5, 2048 x 512: 9.0, 9.0. The Go network's step at 256
  // boards, weight-gradients beside and in line, with four 1421 and 1531 us, with two 1408 and 1521.
  const dim3 grid = row_grid(rows, C, 8, 148 * 2);
  auto go = [&](auto kern) { launch_pdl(kern, grid, dim3(256), 0, st, x, dy, y, mean, istd, rows, C, plain, ws); };
  if (!backward) go(bn_reduce_kernel<0, 0>);
  else if (y) go(bn_reduce_kernel<1, 1>);
  else go(bn_reduce_kernel<1, 0>);
}

// The sums of 8 channels, for the kernel after a reduction. Which of the scratch's two buffers holds them is only known
// after a load, so both are read at the same time.
__device__ __forceinline__ void bn_load_sums(const BnScratch& ws, const float* plain, int C, int c0, float (&s0)[8],
                                             float (&s1)[8]) {
  if (!ws.sums) {
#pragma unroll
    for (int j = 0; j < 8; ++j) { s0[j] = plain[c0 + j]; s1[j] = plain[C + c0 + j]; }
    return;
  }
  const float* p = ws.sums;
  auto get = [&](const float* q, float (&v)[8]) {
    const float4 lo = *reinterpret_cast<const float4*>(q), hi = *reinterpret_cast<const float4*>(q + 4);
    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
    v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
  };
  get(p + c0, s0);
  get(p + C + c0, s1);
  float t0[8], t1[8];
  get(p + 2 * (long long)C + c0, t0);
  get(p + 3 * (long long)C + c0, t1);
  const bool second = (*ws.used & 1u) != 0u;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s0[j] = second ? t0[j] : s0[j];
    s1[j] = second ? t1[j] : s1[j];
  }
}
// ... and the handing over of the other buffer to the next call (BnScratch). Loads of the buffer that is cleared here may
// still be under way in other blocks: bn_load_sums throws those away.
// This and what else is stored once per channel is done by blocks of their own, the last of each slab, one thread per
// channel: done by blocks that also have rows to do, its chains of loads and stores delay the end of the launch.
__device__ __forceinline__ bool bn_is_keeper(const BnScratch& ws) { return ws.sums && blockIdx.x == gridDim.x - 1; }
__device__ __forceinline__ long long bn_row_blocks(const BnScratch& ws) { return (long long)gridDim.x - (ws.sums ? 1 : 0); }
__device__ __forceinline__ void bn_hand_over(const BnScratch& ws, int C) {
  const unsigned int b = *ws.used & 1u;
  float* other = ws.sums + (b ^ 1u) * (2 * (long long)C);
  for (int c = blockIdx.y * 256 + threadIdx.x; c < 2 * C; c += 256 * gridDim.y) other[c] = 0.f;
  if (blockIdx.y == 0 && threadIdx.x == 0) *ws.next = b ^ 1u;
}

// Statistics from sums that the caller keeps (cleared here), for scratches of 2 * C floats.
__global__ void bn_finalize_kernel(float* __restrict__ sums, const bf16* __restrict__ x_row0, long long rows, int C,
                                   const BnStats st) {
  pdl_prolog();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float mean, var, istd;
  bn_batch_stats(sums[c], sums[C + c], bf2f(x_row0[c]), 1.f / (float)rows, st.eps, mean, var, istd);
  bn_store_stats(st, c, rows, mean, var, istd);
  sums[c] = 0.f;
  sums[C + c] = 0.f;
}

// y = act(gamma * (x - mean) * istd + beta [+ residual]), with mean and istd from st.mean / st.istd (BN_GIVEN), from the
// running statistics (BN_INFER) or from a reduction's sums (BN_SUMS: every block works them out for its own channels). Per row
// and thread: 16 bytes in (32 with a residual), 16 out, one subtract and one fused multiply-add per channel; four rows in
// flight. A thread used to fetch all five values of all its eight channels again for every row, and 64-bit divide to find
// them: 92416 x 128 took 22 us, now 11 with given statistics or running ones. From sums it takes 13 (cold caches; 18 with
// two divisions per channel and more blocks than fit at once).
enum { BN_GIVEN = 0, BN_INFER = 1, BN_SUMS = 2 };
template <int FROM, int RES>
__global__ void __launch_bounds__(256) bn_apply_kernel(const bf16* __restrict__ x, const BnStats st, const BnScratch ws,
                                                       const float* __restrict__ gamma, const float* __restrict__ beta,
                                                       const bf16* __restrict__ residual, bf16* __restrict__ y,
                                                       long long rows, int C, int c_valid, int relu) {
  pdl_prolog();
  constexpr int U = 4;
  const RowCover w = row_cover(C);
  if (FROM == BN_SUMS && bn_is_keeper(ws)) {
    const float* sums = ws.sums + (*ws.used & 1u) * (2 * (long long)C);
    const int width = w.gpb * 8, base = blockIdx.y * width;
    for (int c = base + threadIdx.x; c < base + width && c < C; c += 256) {
      float m, var, is;
      bn_batch_stats(sums[c], sums[C + c], bf2f(x[c]), 1.f / (float)rows, st.eps, m, var, is);
      bn_store_stats(st, c, rows, m, var, is);
    }
    bn_hand_over(ws, C);
    return;
  }
  if (!w.live) return;
  const long long step = bn_row_blocks(ws) * w.rl;
  long long r = (long long)blockIdx.x * w.rl + w.rr;
  uint4 xv[U], rv[RES ? U : 1];
  auto fetch = [&]() {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long ru = r + step * u;
      if (ru < rows) {
        xv[u] = *reinterpret_cast<const uint4*>(x + ru * C + w.c0);
        if (RES) rv[u] = *reinterpret_cast<const uint4*>(residual + ru * C + w.c0);
      }
    }
  };
  fetch();      // the first rows are under way while the statistics are worked out
  float mu[8], sc[8], be[8];
  if (FROM == BN_SUMS) {
    float shift[8], s0[8], s1[8];
    const float inv_rows = 1.f / (float)rows;
    load8(x + w.c0, shift);   // the shift of the sums: row 0
    bn_load_sums(ws, nullptr, C, w.c0, s0, s1);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float var;
      bn_batch_stats(s0[j], s1[j], shift[j], inv_rows, st.eps, mu[j], var, sc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = w.c0 + j;
    if (FROM == BN_INFER) {
      mu[j] = st.run_mean[c];
      sc[j] = rsqrtf(st.run_var[c] + st.eps);
    } else if (FROM == BN_GIVEN) {
      mu[j] = st.mean[c];
      sc[j] = st.istd[c];
    }
    sc[j] *= c < c_valid ? gamma[c] : 0.f;
    be[j] = c < c_valid ? beta[c] : 0.f;
  }
  const bool whole = w.c0 + 8 <= c_valid;
  for (; r < rows; r += step * U, fetch()) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long ru = r + step * u;
      if (ru >= rows) break;
      float v[8], q[8];
      unpack8(xv[u], v);
      if (RES) unpack8(rv[u], q);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float o = (v[j] - mu[j]) * sc[j] + be[j];
        if (RES) o += q[j];
        if (relu) o = fmaxf(o, 0.f);
        v[j] = (whole || w.c0 + j < c_valid) ? o : 0.f;
      }
      store8(y + ru * C + w.c0, v);
    }
  }
}

template <int FROM>
static void launch_bn_apply(const bf16* x, const BnStats& stats, const BnScratch& ws, const float* gamma, const float* beta,
                            const bf16* residual, bf16* y, long long rows, int C, int c_valid, int relu,
                            cudaStream_t st) {
  // with the statistics to work out a block costs ~500 instructions before its first row: no more blocks than fit at once
  dim3 grid = row_grid(rows, C, 4, 148 * (FROM == BN_SUMS ? 3 : 8));
  if (ws.sums) ++grid.x;   // the blocks that store what exists once per channel
  auto go = [&](auto kern) {
    launch_pdl(kern, grid, dim3(256), 0, st, x, stats, ws, gamma, beta, residual, y, rows, C, c_valid, relu);
  };
  if (residual) go(bn_apply_kernel<FROM, 1>);
  else go(bn_apply_kernel<FROM, 0>);
}

// Scale and shift of normalisations by running statistics, for the epilogues of the convolutions before them
// (rb_conv_fprop_norm): y = x * scale + shift. One block per layer; `units` holds per layer where gamma, beta, the running mean
// and the running variance lie in `params` and where the layer's scale and shift go in `out`, its channels, padded and not, and
// eps as a bit pattern.
__global__ void __launch_bounds__(256) bn_fold_kernel(const float* __restrict__ params, const long long* __restrict__ units,
                                                      float* __restrict__ out) {
  pdl_prolog();
  const long long* u = units + 8 * (long long)blockIdx.x;
  const int C = (int)u[5], c_valid = (int)u[6];
  const float eps = __int_as_float((int)u[7]);
  for (int c = threadIdx.x; c < C; c += 256) {
    float scale = 0.f, shift = 0.f;
    if (c < c_valid) {
      scale = params[u[0] + c] * rsqrtf(params[u[3] + c] + eps);
      shift = params[u[1] + c] - params[u[2] + c] * scale;
    }
    out[u[4] + c] = scale;
    out[u[4] + C + c] = shift;
  }
}

// dx = gamma * istd * (dy - (dbeta + xhat * dgamma) / rows), with [dbeta | dgamma] of this batch from `plain` or from a
// scratch; in the latter case they are also accumulated into the gradient buffers.
template <int MASK>
__global__ void __launch_bounds__(256) bn_bwd_apply_kernel(const bf16* __restrict__ x, const bf16* __restrict__ dy,
                                                           const bf16* __restrict__ y, const float* __restrict__ mean,
                                                           const float* __restrict__ istd,
                                                           const float* __restrict__ gamma, const float* plain,
                                                           const BnScratch ws, float* __restrict__ dgamma,
                                                           float* __restrict__ dbeta, bf16* __restrict__ dx,
                                                           long long rows, int C, int c_valid) {
  pdl_prolog();
  constexpr int U = MASK ? 2 : 3;
  const RowCover w = row_cover(C);
  if (bn_is_keeper(ws)) {
    const float* sums = ws.sums + (*ws.used & 1u) * (2 * (long long)C);
    const int width = w.gpb * 8, base = blockIdx.y * width;
    for (int c = base + threadIdx.x; c < base + width && c < c_valid; c += 256) {
      dbeta[c] += sums[c];
      dgamma[c] += sums[C + c];
    }
    bn_hand_over(ws, C);
    return;
  }
  if (!w.live) return;
  const long long step = bn_row_blocks(ws) * w.rl;
  long long r = (long long)blockIdx.x * w.rl + w.rr;
  uint4 xv[U], gv[U], yv[MASK ? U : 1];
  auto fetch = [&]() {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long ru = r + step * u;
      if (ru < rows) {
        const long long o = ru * C + w.c0;
        xv[u] = *reinterpret_cast<const uint4*>(x + o);
        gv[u] = *reinterpret_cast<const uint4*>(dy + o);
        if (MASK) yv[u] = *reinterpret_cast<const uint4*>(y + o);
      }
    }
  };
  fetch();      // the first rows are under way while the sums arrive
  float mu[8], sc[8], kb[8], kg[8];
  const float invm = 1.f / (float)rows;
  bn_load_sums(ws, plain, C, w.c0, kb, kg);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = w.c0 + j;
    mu[j] = sc[j] = 0.f;
    if (c < c_valid) {
      mu[j] = mean[c];
      sc[j] = gamma[c] * istd[c];
      kb[j] *= invm;
      kg[j] *= invm * istd[c];
    }
  }
  for (; r < rows; r += step * U, fetch()) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long ru = r + step * u;
      if (ru >= rows) break;
      float v[8], g[8];
      unpack8(xv[u], v);
      unpack8(gv[u], g);
      if (MASK) {
        float yy[8];
        unpack8(yv[u], yy);
#pragma unroll
        for (int j = 0; j < 8; ++j) if (!(yy[j] > 0.f)) g[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = w.c0 + j < c_valid ? sc[j] * (g[j] - (kb[j] + (v[j] - mu[j]) * kg[j])) : 0.f;
      store8(dx + ru * C + w.c0, v);
    }
  }
}

static void launch_bn_bwd_apply(const bf16* x, const bf16* dy, const bf16* y, const float* mean, const float* istd,
                                const float* gamma, const float* plain, const BnScratch& ws, float* dgamma,
                                float* dbeta, bf16* dx, long long rows, int C, int c_valid, cudaStream_t st) {
  // Two blocks per SM, which find room beside a weight-gradient and are the fastest alone: 92416 x 128, us a layer with its sums, by
  // 2, 4, 8 blocks: 24.1, 25.2, 28.3, 32768 x 128: 14.1, 15.8, 15.8. Steps with weight-gradients beside and in line, with eight and
  // with two: the Go network at 256 boards 1432 and 1569 us, 1408 and 1521; ResNet-18 at 32 images 1417 and 1595, 1406 and 1582.
  dim3 grid = row_grid(rows, C, 4, 148 * 2);
  if (ws.sums) ++grid.x;   // the blocks that store what exists once per channel
  auto go = [&](auto kern) {
    launch_pdl(kern, grid, dim3(256), 0, st, x, dy, y, mean, istd, gamma, plain, ws, dgamma, dbeta, dx, rows, C, c_valid);
  };
  if (y) go(bn_bwd_apply_kernel<1>);
  else go(bn_bwd_apply_kernel<0>);
}

// The gradients of a batch into the gradient buffers, for scratches of 2 * C floats.
__global__ void bn_grad_accum_kernel(float* __restrict__ sums, float* __restrict__ dgamma, float* __restrict__ dbeta,
                                     int C, int c_valid) {
  pdl_prolog();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  if (c < c_valid) {
    dbeta[c] += sums[c];
    dgamma[c] += sums[C + c];
  }
  sums[c] = 0.f;
  sums[C + c] = 0.f;
}

}  // namespace rb

using namespace rb;

extern "C" {

// sums: 2*C floats of scratch that must be zero on entry and is zero again on return.
int rb_bn_fwd_train(const void* x, long long rows, int C, int c_valid, float* sums, float eps, float factor,
                    float* mean, float* istd, float* run_mean, float* run_var, const float* gamma, const float* beta,
                    const void* residual, void* y, int relu, int avg_kind, const unsigned int* step_ptr,
                    cudaStream_t st) {
  if (C % 8) return -10;
  const BnStats stats = {mean, istd, run_mean, run_var, step_ptr, eps, factor, avg_kind};
  const BnScratch none = {};
  launch_bn_reduce((const bf16*)x, nullptr, nullptr, nullptr, nullptr, rows, C, sums, 0, none, st);
  launch_pdl(bn_finalize_kernel, dim3((C + 127) / 128), dim3(128), 0, st, sums, (const bf16*)x, rows, C, stats);
  launch_bn_apply<BN_GIVEN>((const bf16*)x, stats, none, gamma, beta, (const bf16*)residual, (bf16*)y, rows, C, c_valid,
                            relu, st);
  return RB_LAUNCH_OK();
}

// The same in two launches: `ws` is 4*C + 32 floats, on a 16-byte boundary, zero before their first use, and used for nothing
// but calls of the two-launch forms with the same C: one buffer of sums is left as it is (BnScratch).
int rb_bn_fwd_train_ws(const void* x, long long rows, int C, int c_valid, float* ws, float eps, float factor,
                       float* mean, float* istd, float* run_mean, float* run_var, const float* gamma,
                       const float* beta, const void* residual, void* y, int relu, int avg_kind,
                       const unsigned int* step_ptr, cudaStream_t st) {
  if (C % 8 || ((uintptr_t)ws & 15u)) return -10;
  const BnStats stats = {mean, istd, run_mean, run_var, step_ptr, eps, factor, avg_kind};
  const BnScratch scr = bn_scratch(ws, C);
  launch_bn_reduce((const bf16*)x, nullptr, nullptr, nullptr, nullptr, rows, C, nullptr, 0, scr, st);
  launch_bn_apply<BN_SUMS>((const bf16*)x, stats, scr, gamma, beta, (const bf16*)residual, (bf16*)y, rows, C, c_valid, relu,
                           st);
  return RB_LAUNCH_OK();
}

// One launch, which works out the inverse deviations itself: the argument that once was scratch for them is not looked at.
int rb_bn_fwd_infer(const void* x, long long rows, int C, int c_valid, float eps, const float* run_mean,
                    const float* run_var, float* /* scratch */, const float* gamma, const float* beta,
                    const void* residual, void* y, int relu, cudaStream_t st) {
  if (C % 8) return -10;
  const BnStats stats = {nullptr, nullptr, (float*)run_mean, (float*)run_var, nullptr, eps, 0.f, 0};
  launch_bn_apply<BN_INFER>((const bf16*)x, stats, BnScratch{}, gamma, beta, (const bf16*)residual, (bf16*)y, rows, C,
                            c_valid, relu, st);
  return RB_LAUNCH_OK();
}

int rb_bn_fold(const float* params, const long long* units, int n_units, float* out, cudaStream_t st) {
  if (n_units <= 0) return 0;
  launch_pdl(bn_fold_kernel, dim3(n_units), dim3(256), 0, st, params, units, out);
  return RB_LAUNCH_OK();
}

// y_relu: forward output when a ReLU followed the normalisation (masks dy), else null.
// dgamma/dbeta are accumulated (the optimizer zeroes them).
int rb_bn_bwd(const void* x, const void* dy, const void* y_relu, long long rows, int C, int c_valid, float* sums,
              const float* mean, const float* istd, const float* gamma, float* dgamma, float* dbeta, void* dx,
              cudaStream_t st) {
  if (C % 8) return -10;
  const BnScratch none = {};
  launch_bn_reduce((const bf16*)x, (const bf16*)dy, (const bf16*)y_relu, mean, istd, rows, C, sums, 1, none, st);
  launch_bn_bwd_apply((const bf16*)x, (const bf16*)dy, (const bf16*)y_relu, mean, istd, gamma, sums, none, dgamma, dbeta,
                      (bf16*)dx, rows, C, c_valid, st);
  launch_pdl(bn_grad_accum_kernel, dim3((C + 127) / 128), dim3(128), 0, st, sums, dgamma, dbeta, C, c_valid);
  return RB_LAUNCH_OK();
}

// The same in two launches, with the scratch of rb_bn_fwd_train_ws.
int rb_bn_bwd_ws(const void* x, const void* dy, const void* y_relu, long long rows, int C, int c_valid, float* ws,
                 const float* mean, const float* istd, const float* gamma, float* dgamma, float* dbeta, void* dx,
                 cudaStream_t st) {
  if (C % 8 || ((uintptr_t)ws & 15u)) return -10;
  const BnScratch scr = bn_scratch(ws, C);
  launch_bn_reduce((const bf16*)x, (const bf16*)dy, (const bf16*)y_relu, mean, istd, rows, C, nullptr, 1, scr, st);
  launch_bn_bwd_apply((const bf16*)x, (const bf16*)dy, (const bf16*)y_relu, mean, istd, gamma, nullptr, scr, dgamma, dbeta,
                      (bf16*)dx, rows, C, c_valid, st);
  return RB_LAUNCH_OK();
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------------
// Allocation-free variant (declared and documented in bn_noalloc.h).
#include "bn_noalloc.h"

namespace rb {
// Scratch for the per-channel sums: part of the library's device image, one copy per GPU.
static __device__ __align__(256) float g_bn_noalloc_scratch[2 * RB_BN_NOALLOC_MAX_CHANNELS];
constexpr int kMaxDevices = 64;
// Device address of the array above, per device. The array's name is only a host-side handle; kernels
// must be given the address that cudaGetSymbolAddress returns for the device they run on.
static float* g_bn_noalloc_ptr[kMaxDevices] = {nullptr};
}  // namespace rb

extern "C" {

int rb_bn_fwd_train_noalloc(const void* x, long long rows, int C, int c_valid, float eps, float factor, float* mean,
                            float* istd, float* run_mean, float* run_var, const float* gamma, const float* beta,
                            const void* residual, void* y, int relu, cudaStream_t stream) {
  if (C % 8) return RB_BN_NOALLOC_E_CHANNEL_ALIGN;
  if (C > RB_BN_NOALLOC_MAX_CHANNELS) return RB_BN_NOALLOC_E_TOO_MANY_CHANNELS;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return RB_BN_NOALLOC_E_DEVICE;
  if (g_bn_noalloc_ptr[dev] == nullptr) {
    // first call on this device: resolve the array's device address (the device is current here)
    float* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_bn_noalloc_scratch) != cudaSuccess || p == nullptr)
      return RB_BN_NOALLOC_E_SYMBOL;
    g_bn_noalloc_ptr[dev] = p;
  }
  float* sums = g_bn_noalloc_ptr[dev];
  // the array keeps whatever the previous call left: clear the part this call accumulates into
  if (cudaMemsetAsync(sums, 0, sizeof(float) * 2 * (size_t)C, stream) != cudaSuccess) return RB_BN_NOALLOC_E_LAUNCH;
  const BnStats stats = {mean, istd, run_mean, run_var, nullptr, eps, factor, 0};
  bn_reduce_kernel<0, 0><<<row_grid(rows, C, 8, 148 * 4), 256, 0, stream>>>((const bf16*)x, nullptr, nullptr, nullptr,
                                                                          nullptr, rows, C, sums, BnScratch{});
  bn_finalize_kernel<<<(C + 127) / 128, 128, 0, stream>>>(sums, (const bf16*)x, rows, C, stats);
  const dim3 grid = row_grid(rows, C, 4, 148 * 8);
  if (residual)
    bn_apply_kernel<BN_GIVEN, 1><<<grid, 256, 0, stream>>>((const bf16*)x, stats, BnScratch{}, gamma, beta,
                                                         (const bf16*)residual, (bf16*)y, rows, C, c_valid, relu);
  else
    bn_apply_kernel<BN_GIVEN, 0><<<grid, 256, 0, stream>>>((const bf16*)x, stats, BnScratch{}, gamma, beta, nullptr, (bf16*)y,
                                                         rows, C, c_valid, relu);
  return cudaGetLastError() == cudaSuccess ? RB_BN_NOALLOC_OK : RB_BN_NOALLOC_E_LAUNCH;
}

const char* rb_bn_noalloc_strerror(int code) {
  switch (code) {
    case RB_BN_NOALLOC_OK: return "ok";
    case RB_BN_NOALLOC_E_CHANNEL_ALIGN: return "channel count must be a multiple of 8";
    case RB_BN_NOALLOC_E_TOO_MANY_CHANNELS: return "channel count exceeds RB_BN_NOALLOC_MAX_CHANNELS (4096)";
    case RB_BN_NOALLOC_E_DEVICE: return "current CUDA device could not be determined or its index is >= 64";
    case RB_BN_NOALLOC_E_SYMBOL: return "cudaGetSymbolAddress failed for the built-in scratch array";
    case RB_BN_NOALLOC_E_LAUNCH: return "a kernel launch or the scratch-clearing memset failed";
    default: return "unknown code";
  }
}

}  // extern "C"
