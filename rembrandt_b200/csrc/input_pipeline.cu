// Input pipeline on the GPU: one pass from staged u8 images (planar, [N][C][H][W], the reference's
// "WHC bytes, first dimension fastest") to the bf16 NHWC tensor the first convolution reads:
//   u8 -> float (optionally /255) -> subtract element-wise mean -> random / centre crop (with zero
//   padding for negative offsets) -> horizontal flip -> PCA lighting noise -> optional space-to-depth.
// Covers the reference's cast_bytes[_normalized], cuDNN strided-transform crop, batch_blockmap256_flip,
// cuDNN add-tensor mean subtraction and batch_map_preproc_pca3_noise (src/operator/mod.rs:653-778,
// src/operator/input.rs:288-419) in a single kernel. Crop offsets and flip coins are per sample by
// default; `per_batch` reproduces the reference's one-draw-per-batch behaviour.
//
// An output pixel (Y,X) holds the f*f*C values of source pixels (Y*stride+dy, X*stride+dx), channel = (dy*f+dx)*C + c.
// With f == stride this is space-to-depth: an s-strided k x k convolution becomes a stride-1 ceil(k/f) x ceil(k/f)
// convolution on f*f*C channels. With f = k and the convolution's own stride each output pixel holds the whole
// receptive field of a first layer, which then is a plain matrix product.
#include "launch.cuh"
#include "common.cuh"

namespace rb {

struct InputArgs {
  const uint8_t* src;   // [N][C][H][W]
  const float* mean;    // optional [C][H][W]
  bf16* dst;            // [N][OH][OW][Cp]
  int N, C, H, W;
  int crop_h, crop_w;   // extent of the crop window
  int OH, OW, Cp, f;
  int stride;           // source pixels between neighbouring output pixels (f: space-to-depth)
  int border;           // this many rows / columns around the crop window are zeros, whatever the image holds there
  int ones;             // channel that holds 1 in every pixel (-1: none)
  int lo_y, hi_y, lo_x, hi_x;  // inclusive range of the window's top-left corner (may be negative)
  int random_crop, random_flip, per_batch;
  float scale;          // 1/255 when normalising, else 1
  float mean_scale;     // multiplies the mean before subtraction
  float pca_sigma;      // 0 disables
  float pca_vals[3];
  float pca_vecs[9];    // row c, column j
  uint64_t seed;
  uint32_t step;
  const uint32_t* step_ptr;  // optional device counter added to `step` (keeps captured graphs fresh)
};

__device__ __forceinline__ void sample_draw(const InputArgs& a, int n, int& oy, int& ox, int& flip, float (&shift)[3]) {
  uint32_t r[4] = {0u, 0u, 0u, 0u};
  const bool lighting = a.pca_sigma > 0.f && a.C == 3;
  uint32_t step = a.step;
  if (a.random_crop || a.random_flip || lighting) {      // (nothing to draw: inference, and networks without augmentation)
    if (a.step_ptr) step += *a.step_ptr;
    Philox::gen(a.seed, a.per_batch ? 0ull : (uint64_t)n, step, r);
  }
  if (a.random_crop) {
    oy = a.lo_y + (int)(r[0] % (uint32_t)(a.hi_y - a.lo_y + 1));
    ox = a.lo_x + (int)(r[1] % (uint32_t)(a.hi_x - a.lo_x + 1));
  } else {
    // rounded down: padding absorbed from the first layer lowers both ends and must not move the centre
    oy = (a.lo_y + a.hi_y) >> 1;
    ox = (a.lo_x + a.hi_x) >> 1;
  }
  flip = a.random_flip ? (int)(r[2] & 1u) : 0;
  shift[0] = shift[1] = shift[2] = 0.f;
  if (lighting) {
    uint32_t q[4];
    Philox::gen(a.seed ^ 0x5bd1e995ull, (uint64_t)n, step, q);
    // Box-Muller: three normals from four uniforms
    const float u0 = fmaxf(u32_to_unit(q[0]), 1e-7f), u1 = u32_to_unit(q[1]);
    const float u2 = fmaxf(u32_to_unit(q[2]), 1e-7f), u3 = u32_to_unit(q[3]);
    const float m0 = sqrtf(-2.f * __logf(u0)), m1 = sqrtf(-2.f * __logf(u2));
    const float al[3] = {a.pca_sigma * m0 * __cosf(6.2831853f * u1), a.pca_sigma * m0 * __sinf(6.2831853f * u1),
                         a.pca_sigma * m1 * __cosf(6.2831853f * u3)};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      shift[c] = al[0] * a.pca_vals[0] * a.pca_vecs[c * 3 + 0] + al[1] * a.pca_vals[1] * a.pca_vecs[c * 3 + 1] +
                 al[2] * a.pca_vals[2] * a.pca_vecs[c * 3 + 2];
  }
}

// Value of crop-window position (y, x) in channel c; zero outside the window, in its border and outside the image.
__device__ __forceinline__ bool input_source(const InputArgs& a, int y, int x, int oy, int ox, int flip, int& sy, int& sx) {
  const bool in = y >= a.border && y < a.crop_h - a.border && x >= a.border && x < a.crop_w - a.border;
  sy = oy + y;
  sx = ox + (flip ? a.crop_w - 1 - x : x);
  return in && sy >= 0 && sy < a.H && sx >= 0 && sx < a.W;
}

__global__ void input_kernel(InputArgs a) {
  pdl_prolog();
  const int groups = a.Cp / 8;
  const long long total = (long long)a.N * a.OH * a.OW * groups;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int gidx = (int)(i % groups);
    long long t = i / groups;
    const int X = (int)(t % a.OW); t /= a.OW;
    const int Y = (int)(t % a.OH);
    const int n = (int)(t / a.OH);
    int oy, ox, flip;
    float shift[3];
    sample_draw(a, n, oy, ox, flip, shift);
    float out[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int ch = gidx * 8 + j;
      float v = ch == a.ones ? 1.f : 0.f;
      const int blk = ch / a.C, c = ch - blk * a.C;
      if (blk < a.f * a.f) {
        const int dy = blk / a.f, dx = blk - dy * a.f;
        int sy, sx;
        if (input_source(a, Y * a.stride + dy, X * a.stride + dx, oy, ox, flip, sy, sx)) {
          const long long si = ((long long)c * a.H + sy) * a.W + sx;
          v = (float)a.src[(long long)n * a.C * a.H * a.W + si] * a.scale;
          if (a.mean) v -= a.mean_scale * a.mean[si];
          if (c < 3) v += shift[c];
        }
      }
      out[j] = v;
    }
    store8(a.dst + i * 8, out);
  }
}

// q = e / d by one multiply-high; exact for e * d < 2^32 (the host checks the largest e of a block).
struct Divider {
  uint32_t d, magic;
};
__device__ __forceinline__ uint32_t fast_div(uint32_t e, const Divider& v) { return v.d == 1u ? e : __umulhi(e, v.magic); }

// Staged variant: one block per (sample, `rows` output rows). The source rows that these need are read four pixels at a
// time (two aligned words, shifted), several loads in flight per thread, converted (scale, mean, lighting shift, crop /
// flip / zero padding) and kept in shared memory as bf16 planes [row][channel][pitch]; then every thread writes 16-byte
// channel groups. A thread keeps the same channel group throughout, so where its eight values lie relative to a pixel is
// worked out once, in registers. A block moves a few KB: latency and instruction count are what it costs, not bandwidth: which
// of four pixels exist is worked out for all four at once, pixels beyond an edge are loaded and dropped, and nothing is drawn where
// nothing is random. With the four tested one by one, and tiles small enough for eight blocks per SM (of which four fit), us for
// LeNet's input at 64 images, the CIFAR network's at 128, AlexNet's at 128, ResNet-18's at 32, VGG-A's at 64: 13.1, 22.8, 54.7, 52.1,
// 72.3; now 5.8, 10.6, 46.8, 40.7, 60.1.
__global__ void __launch_bounds__(256) input_tile_kernel(InputArgs a, int rows, int pitch, Divider by_q, Divider by_c,
                                                         Divider by_ow) {
  pdl_prolog();
  extern __shared__ __align__(16) uint8_t input_smem[];
  bf16* st = reinterpret_cast<bf16*>(input_smem);   // [0] = 0, [1] = 1, planes from [8]
  __shared__ int s_draw[3];
  __shared__ float s_shift[4];
  const int n = blockIdx.y, Y0 = blockIdx.x * rows;
  const int nrow = min(rows, a.OH - Y0);
  if (threadIdx.x == 0) {
    int oy, ox, flip;
    float shift[3];
    sample_draw(a, n, oy, ox, flip, shift);
    s_draw[0] = oy; s_draw[1] = ox; s_draw[2] = flip;
    s_shift[0] = shift[0]; s_shift[1] = shift[1]; s_shift[2] = shift[2]; s_shift[3] = 0.f;
    st[0] = f2bf(0.f);
    st[1] = f2bf(1.f);
  }
  __syncthreads();
  const int oy = s_draw[0], ox = s_draw[1], flip = s_draw[2];
  const uint8_t* img = a.src + (long long)n * a.C * a.H * a.W;
  const uint8_t* src_end = a.src + (long long)a.N * a.C * a.H * a.W;
  const int lines = ((nrow - 1) * a.stride + a.f) * a.C;
  const uint32_t quads = (uint32_t)lines * by_q.d;
  constexpr int U = 4;
  for (uint32_t e0 = threadIdx.x; e0 < quads; e0 += 256 * U) {
    uint32_t lo[U], hi[U];   // the two words of four neighbouring source pixels, or those pixels one by one in `lo`
    int sh[U], at[U], idx[U], ch[U];
    uint32_t ok[U];          // which of the four positions hold a source pixel
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t e = e0 + u * 256;
      at[u] = -1;
      ok[u] = 0u;
      lo[u] = hi[u] = 0u;
      sh[u] = 0;
      idx[u] = 0;
      ch[u] = 3;
      if (e >= quads) continue;
      const uint32_t line = fast_div(e, by_q);
      const int x0 = 4 * (int)(e - line * by_q.d);
      const int t = (int)fast_div(line, by_c);
      const int c = (int)line - t * (int)by_c.d;
      at[u] = 8 + (int)line * pitch + x0;
      ch[u] = min(c, 3);
      const int y = Y0 * a.stride + t, sy = oy + y;
      if (y < a.border || y >= a.crop_h - a.border || sy < 0 || sy >= a.H) continue;
      // source column of position x0 (not flipped) or x0 + 3 (flipped): the lowest of the four
      const int sx = ox + (flip ? a.crop_w - 4 - x0 : x0);
      // which of the four lie in the window and in the image: k0 .. k1 - 1
      const int k0 = max(max(a.border - x0, flip ? sx + 4 - a.W : -sx), 0);
      const int k1 = min(min(a.crop_w - a.border - x0, flip ? sx + 4 : a.W - sx), 4);
      if (k0 >= k1) continue;
      ok[u] = (1u << k1) - (1u << k0);
      idx[u] = (c * a.H + sy) * a.W + sx;
      const uint8_t* px = img + idx[u];
      const int off = (int)(reinterpret_cast<uintptr_t>(px) & 3u);
      const uint8_t* w = px - off;
      if (w >= a.src && w + 8 <= src_end) {      // (pixels of other rows may come along: they are dropped below)
        lo[u] = *reinterpret_cast<const uint32_t*>(w);
        hi[u] = *reinterpret_cast<const uint32_t*>(w + 4);
        sh[u] = off * 8;
      } else {   // the first or last of the batch
#pragma unroll 1
        for (int k = 0; k < 4; ++k)
          if (ok[u] & (1u << (flip ? 3 - k : k))) lo[u] |= (uint32_t)px[k] << (8 * k);
      }
    }
    float mu[U][4];
    if (a.mean) {
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          mu[u][k] = 0.f;
          if (ok[u] & (1u << k)) mu[u][k] = a.mean[idx[u] + (flip ? 3 - k : k)];
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (at[u] < 0) continue;
      uint32_t px = __funnelshift_r(lo[u], hi[u], sh[u]);
      if (flip) px = __byte_perm(px, 0u, 0x0123);
      const float shift = s_shift[ch[u]];
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k] = (float)((px >> (8 * k)) & 255u) * a.scale;
        if (a.mean) v[k] -= a.mean_scale * mu[u][k];
        v[k] += shift;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (!(ok[u] & (1u << k))) v[k] = 0.f;
      __nv_bfloat162 two[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
      *reinterpret_cast<uint2*>(st + at[u]) = *reinterpret_cast<uint2*>(two);
    }
  }
  const int groups = a.Cp / 8;
  const int per = 256 / groups;                       // pixels per pass of the block
  const int g = threadIdx.x % groups, first = threadIdx.x / groups;
  int off[8], sel[8];                                 // sel: all ones where the value moves with the pixel
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int ch = g * 8 + j;
    const int blk = ch / a.C, c = ch - blk * a.C;
    const int dy = blk / a.f, dx = blk - dy * a.f;
    sel[j] = blk < a.f * a.f ? -1 : 0;
    off[j] = sel[j] ? 8 + (dy * a.C + c) * pitch + dx : (ch == a.ones ? 1 : 0);
  }
  __syncthreads();
  if (first >= per) return;
  const int row_step = a.stride * a.C * pitch;
  bf16* drow = a.dst + (((long long)n * a.OH + Y0) * a.OW) * a.Cp + g * 8;
  const uint16_t* raw = reinterpret_cast<const uint16_t*>(st);
  for (int i = first; i < nrow * a.OW; i += per) {
    const int Y = (int)fast_div((uint32_t)i, by_ow), X = i - Y * a.OW;
    const int base = Y * row_step + X * a.stride;
    uint32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = raw[off[j] + (base & sel[j])];
    *reinterpret_cast<uint4*>(drow + (long long)i * a.Cp) =
        make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16), v[4] | (v[5] << 16), v[6] | (v[7] << 16));
  }
}

// Synthetic N(0,1) activations (bf16, padded channels zero) and uniform labels, generated on the device.
__global__ void synth_normal_kernel(bf16* __restrict__ dst, long long pixels, int C, int Cp, uint64_t seed,
                                    uint32_t step) {
  pdl_prolog();
  const long long total = pixels * Cp;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total / 4;
       i += (long long)gridDim.x * blockDim.x) {
    uint32_t r[4];
    Philox::gen(seed, (uint64_t)i, step, r);
    const float u0 = fmaxf(u32_to_unit(r[0]), 1e-7f), u1 = u32_to_unit(r[1]);
    const float u2 = fmaxf(u32_to_unit(r[2]), 1e-7f), u3 = u32_to_unit(r[3]);
    const float m0 = sqrtf(-2.f * __logf(u0)), m1 = sqrtf(-2.f * __logf(u2));
    float z[4] = {m0 * __cosf(6.2831853f * u1), m0 * __sinf(6.2831853f * u1), m1 * __cosf(6.2831853f * u3),
                  m1 * __sinf(6.2831853f * u3)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long e = i * 4 + j;
      const int c = (int)(e % Cp);
      dst[e] = f2bf(c < C ? z[j] : 0.f);
    }
  }
}

__global__ void synth_labels_kernel(int* __restrict__ labels, int n, int classes, uint64_t seed, uint32_t step) {
  pdl_prolog();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t r[4];
  Philox::gen(seed ^ 0x9e3779b97f4a7c15ull, (uint64_t)i, step, r);
  labels[i] = (int)(r[0] % (uint32_t)classes);
}

}  // namespace rb

using namespace rb;

extern "C" {

int rb_input_u8(const void* src, const float* mean, void* dst, int N, int C, int H, int W, int crop_h, int crop_w,
                int OH, int OW, int Cp, int f, int stride, int border, int ones, int lo_y, int hi_y, int lo_x, int hi_x, int random_crop,
                int random_flip, int per_batch, float scale, float mean_scale, float pca_sigma, const float* pca_vals,
                const float* pca_vecs, unsigned long long seed, unsigned int step, const unsigned int* step_ptr,
                cudaStream_t st) {
  if (Cp % 8) return -10;
  InputArgs a;
  a.src = (const uint8_t*)src; a.mean = mean; a.dst = (bf16*)dst;
  a.N = N; a.C = C; a.H = H; a.W = W; a.crop_h = crop_h; a.crop_w = crop_w;
  a.OH = OH; a.OW = OW; a.Cp = Cp; a.f = f; a.stride = stride; a.border = border; a.ones = ones;
  a.lo_y = lo_y; a.hi_y = hi_y; a.lo_x = lo_x; a.hi_x = hi_x;
  a.random_crop = random_crop; a.random_flip = random_flip; a.per_batch = per_batch;
  a.scale = scale; a.mean_scale = mean_scale; a.pca_sigma = pca_sigma;
  for (int i = 0; i < 3; ++i) a.pca_vals[i] = pca_vals ? pca_vals[i] : 0.f;
  for (int i = 0; i < 9; ++i) a.pca_vecs[i] = pca_vecs ? pca_vecs[i] : 0.f;
  a.seed = seed; a.step = step; a.step_ptr = step_ptr;
  // Output rows per block: as many as leave every SM two blocks and the planes in 32 KB (fewer rows are staged twice
  // when windows overlap, and a block's fixed cost, 3 - 4 us, is shared by more of them: with 4 blocks per SM 8.5 instead of 6.2 us
  // for LeNet's input, 14.4 instead of 11.3 for the CIFAR network's; the larger ones are as fast from 2 to 4).
  const int seg_w = (OW - 1) * stride + f;
  const int quads = (seg_w + 3) / 4;
  const int pitch = 4 * (quads | 1);
  int rows = 0;
  for (int r = 16; r >= 1; r >>= 1) {
    const long long lines = ((long long)(r - 1) * stride + f) * C;
    const long long smem = (8 + lines * pitch) * 2;
    if (smem > (r == 1 ? 40 * 1024 : 32 * 1024)) continue;
    if (lines * quads * quads >= 0xFFFFFFFFll || (long long)r * OW * OW >= 0xFFFFFFFFll) continue;   // see Divider
    rows = r;
    if ((long long)N * ((OH + r - 1) / r) >= 148 * 2) break;
  }
  if (rows > 0 && Cp <= 2048 && N <= 65535 && (long long)C * H * W < 0x7FFFFFFF) {
    const size_t smem = (8 + (size_t)((rows - 1) * stride + f) * C * pitch) * 2;
    auto divider = [](int d) { return Divider{(uint32_t)d, (uint32_t)((0x100000000ull + d - 1) / d)}; };
    launch_pdl(input_tile_kernel, dim3((unsigned)((OH + rows - 1) / rows), (unsigned)N), dim3(256), smem, st, a, rows,
               pitch, divider(quads), divider(C), divider(OW));
  } else {
    const long long total = (long long)N * OH * OW * (Cp / 8);
    long long blocks = (total + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    launch_pdl(input_kernel, (int)blocks, 256, 0, st, a);
  }
  return RB_LAUNCH_OK();
}

int rb_synth_normal(void* dst, long long pixels, int C, int Cp, unsigned long long seed, unsigned int step,
                    cudaStream_t st) {
  if ((pixels * Cp) % 4) return -10;
  long long blocks = (pixels * Cp / 4 + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  launch_pdl(synth_normal_kernel, (int)blocks, 256, 0, st, (bf16*)dst, pixels, C, Cp, seed, step);
  return RB_LAUNCH_OK();
}

int rb_synth_labels(int* labels, int n, int classes, unsigned long long seed, unsigned int step, cudaStream_t st) {
  launch_pdl(synth_labels_kernel, (n + 255) / 256, 256, 0, st, labels, n, classes, seed, step);
  return RB_LAUNCH_OK();
}

}  // extern "C"
