// The planner of the tensor-core convolutions without a GPU: csrc/gemm_tc.cu compiled with the CUDA calls of its host code
// replaced, so that a launch is only noted and a plan's time is what `fake_ms` says. Run with the name of a scenario
// (test_conv_plans.py); says what is wrong and returns 1.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

static int g_launches = 0;
static float fake_ms();
#define cudaLaunchKernelEx(...) (++g_launches, cudaSuccess)
#define cudaEventCreate(e) ((void)(e), cudaSuccess)
#define cudaEventDestroy(e) ((void)(e), cudaSuccess)
#define cudaEventRecord(e, s) ((void)(e), cudaSuccess)
#define cudaEventSynchronize(e) ((void)(e), cudaSuccess)
#define cudaEventElapsedTime(t, a, b) (*(t) = fake_ms(), cudaSuccess)
#define cudaStreamIsCapturing(s, c) ((void)(s), (void)(c), cudaSuccess)
#define cudaGetLastError() cudaSuccess
#include "gemm_tc.cu"

static CUresult no_tiled(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                         const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                         CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
static CUresult no_im2col(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const int*,
                          const int*, cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                          CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}

// {sub-tiles, split, resident, tail, pair, width, A load mode, ...} of the last launch
enum { MT = 0, PAIR = 4, WIDTH = 5, MODE = 6 };
static float (*g_time)(const int* launch) = nullptr;
static float fake_ms() { return g_time ? g_time(g_last_launch) : 1.f; }
static float flat_is_fastest(const int* l) { return l[MODE] == A_FLAT_K ? 1.f : 2.f; }
static float flat_of_256_is_fastest(const int* l) { return l[MODE] == A_FLAT_K && l[WIDTH] == 256 ? 1.f : 2.f; }

// A forward convolution, stride 1, on images of H x H.
static int conv(int N, int C, int Ko, int H, int R, int pad) {
  const int P = H + 2 * pad - R + 1;
  void* const at = (void*)0x1000;   // never read: nothing is launched
  return rb_conv_fprop_tc(at, N, H, H, C, at, Ko, R, R, 1, pad, pad, P, P, at, Ko, nullptr, 0, nullptr, Ko, Ko, nullptr, 0,
                          nullptr, 0);
}
static void measure(float (*time)(const int*), int N, int C, int Ko, int H, int R, int pad) {
  g_time = time;
  g_tune_mode = 1;
  conv(N, C, Ko, H, R, pad);
  g_tune_mode = 0;
}

static int g_wrong = 0;
static void expect(bool ok, const char* what) {
  if (ok) return;
  printf("wrong: %s (mode %d, width %d, sub-tiles %d, pair %d)\n", what, g_last_launch[MODE], g_last_launch[WIDTH],
         g_last_launch[MT], g_last_launch[PAIR]);
  g_wrong = 1;
}

// Flat mode is remembered, and no plan of it fits a later launch: other options, or other paddings of the same output
// (3 x 3, 256 columns, rows of 111: padding 0 fits at a row pitch of 128, padding 1 does not at 112).
static void remembered_flat_does_not_fit() {
  measure(flat_is_fastest, 4, 64, 128, 108, 3, 1);
  expect(conv(4, 64, 128, 108, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K, "measured as flat");
  g_opt.force_pair = 0;   // all plans of this one are CTA pairs
  expect(conv(4, 64, 128, 108, 3, 1) == 0, "flat with pairs switched off since");
  g_opt.force_pair = -1;
  measure(flat_of_256_is_fastest, 4, 64, 256, 113, 3, 0);
  expect(conv(4, 64, 256, 113, 3, 0) == 0 && g_last_launch[MODE] == A_FLAT_K, "measured as flat, padding 0");
  expect(conv(4, 64, 256, 111, 3, 1) == 0, "the same output at padding 1");
}

// What was measured for one row pitch says nothing about another: the same output at padding 1 (33) and 0 (34).
static void paddings_are_measured_apart() {
  measure(flat_is_fastest, 16, 64, 64, 32, 3, 1);
  expect(conv(16, 64, 64, 32, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K, "measured as flat");
  expect(conv(16, 64, 64, 34, 3, 0) == 0 && g_last_launch[MODE] != A_FLAT_K, "not measured at padding 0");
  measure(flat_is_fastest, 16, 64, 64, 34, 3, 0);
  expect(conv(16, 64, 64, 34, 3, 0) == 0 && g_last_launch[MODE] == A_FLAT_K, "measured as flat at padding 0");
}

// Three and four sub-tiles per item exist in flat mode only; a launch of another mode that is asked for them as CTA pairs must
// not have accumulators that nothing computes.
static void sub_tiles_of_other_modes() {
  g_opt.force_pair = 1;
  for (int mt = 1; mt <= 4; ++mt) {
    g_opt.force_mt = mt;
    expect(conv(16, 64, 64, 32, 3, 1) == 0 && g_last_launch[PAIR] == 1 && g_last_launch[MT] == (mt < 2 ? mt : 2), "im2col");
    void* const at = (void*)0x1000;
    expect(rb_gemm_tc(at, 0, 64, at, 0, 64, 4096, 64, 64, at, 64, 0, nullptr, 0, nullptr, 0, 0, 0, 0, nullptr, 0, nullptr, 0) == 0 &&
               g_last_launch[PAIR] == 1 && g_last_launch[MT] == (mt < 2 ? mt : 2),
           "matrix product");
    g_opt.force_halo = 1;
    expect(conv(16, 64, 64, 32, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K && g_last_launch[MT] == mt, "flat");
    g_opt.force_halo = -1;
  }
}

// `deterministic`: every plan that timing may choose from adds the products of an output in one order. Flat mode has another
// one (channel chunks outside, taps inside), so it is not among them, measured or forced.
static void deterministic_keeps_one_order() {
  measure(flat_is_fastest, 16, 128, 64, 32, 3, 1);
  expect(conv(16, 128, 64, 32, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K, "measured as flat");
  g_opt.deterministic = 1;
  expect(conv(16, 128, 64, 32, 3, 1) == 0 && g_last_launch[MODE] != A_FLAT_K, "measured before");
  g_opt.force_halo = 1;
  expect(conv(16, 128, 64, 32, 3, 1) == 0 && g_last_launch[MODE] != A_FLAT_K, "forced");
  g_opt.force_halo = -1;
  g_bn_cache.clear();
  g_plan_cache.clear();
  measure(flat_is_fastest, 16, 128, 64, 32, 3, 1);
  expect(conv(16, 128, 64, 32, 3, 1) == 0 && g_last_launch[MODE] != A_FLAT_K, "measured under the option");
}

// CTA pairs are taken where they win by 3 %, also in flat mode, whichever of the candidates is timed first.
static float flat_pairs_win(const int* l, float by) { return l[MODE] != A_FLAT_K ? 2.f : l[PAIR] ? 1.f / by : 1.f; }
static void pairs_win_by_a_margin() {
  const struct { float (*time)(const int*); int pair; const char* what; } tries[] = {
      {[](const int* l) { return flat_pairs_win(l, 1.02f); }, 0, "pairs 2 % faster"},
      {[](const int* l) { return flat_pairs_win(l, 1.05f); }, 1, "pairs 5 % faster"},
      {[](const int* l) { return flat_pairs_win(l, 0.99f); }, 0, "pairs slower"}};
  for (auto& t : tries)
    for (int Ko : {64, 128, 256, 384}) {
      g_bn_cache.clear();
      g_plan_cache.clear();
      measure(t.time, 16, 128, Ko, 32, 3, 1);
      expect(conv(16, 128, Ko, 32, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K && g_last_launch[PAIR] == t.pair, t.what);
    }
}

// `bn_cap` bounds the tile width of flat plans too, forced, measured, and measured before the option was set.
static void flat_tiles_within_the_cap() {
  g_opt.bn_cap = 128;
  g_opt.force_halo = 1;
  for (int Ko : {64, 128, 192, 256, 512}) expect(conv(16, 64, Ko, 32, 3, 1) == 0 && g_last_launch[WIDTH] <= 128, "forced");
  g_opt.force_halo = -1;
  measure(flat_is_fastest, 16, 64, 256, 32, 3, 1);
  expect(conv(16, 64, 256, 32, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K && g_last_launch[WIDTH] <= 128, "measured");
  g_opt.bn_cap = 256;
  g_bn_cache.clear();
  measure(flat_of_256_is_fastest, 16, 64, 256, 32, 3, 1);
  expect(conv(16, 64, 256, 32, 3, 1) == 0 && g_last_launch[MODE] == A_FLAT_K && g_last_launch[WIDTH] == 256, "measured at 256");
  g_opt.bn_cap = 128;
  expect(conv(16, 64, 256, 32, 3, 1) == 0 && g_last_launch[WIDTH] <= 128, "the cap came later");
}

// The epilogue reads a residual (inference) or an addend (data-gradients) in 16-byte pieces: another alignment is an error.
static void addends_are_aligned() {
  for (int off = 0; off < 32; off += 2) {
    const int want = off % 16 == 0 ? 0 : -10;
    void *const at = (void*)0x1000, *const add = (void*)(0x2000 + (size_t)off);
    for (int R : {1, 3}) {
      const int pad = R / 2, before = g_launches;
      expect(rb_conv_fprop_norm(at, 2, 8, 8, 32, at, 32, R, R, 1, pad, pad, 8, 8, at, 32, (const float*)at, (const float*)at, add,
                                1, 32, 32, nullptr, 0, nullptr, 0) == want, "residual");
      expect((g_launches != before) == (want == 0), "residual: launched");
      for (int stride : {1, 2})
        expect(rb_conv_dgrad_tc(at, 2, 8 / stride, 8 / stride, 32, at, nullptr, 32, 32, 32, R, R, stride, pad, pad, 8, 8, at, add,
                                nullptr, nullptr, 0, nullptr, 0) == want, "addend");
    }
  }
}

// The same for the output and the mask of a strided data-gradient, whose phases share one launch, have none (1 x 1) or are
// too many for one (stride 3): refused before anything is launched. A geometry that is not taken keeps its own answer.
static void strided_outputs_are_aligned() {
  const struct { int R, stride, pad, rc; } tries[] = {{1, 2, 0, 0}, {2, 2, 0, 0}, {3, 2, 1, 0}, {5, 2, 2, 0}, {1, 3, 0, 0},
                                                      {3, 3, 0, 0}, {5, 3, 2, 0}, {3, 2, 6, -20}, {2, 2, 1, -20}};
  for (auto& t : tries)
    for (int off = 0; off < 32; off += 2)
      for (int form = 0; form < 3; ++form) {
        const int P = (12 + 2 * t.pad - t.R) / t.stride + 1, before = g_launches;
        // (an addend, which the third form's output is, is looked at first)
        const int want = off % 16 != 0 && (form == 2 || !t.rc) ? -10 : t.rc;
        void *const at = (void*)0x1000, *const odd = (void*)(0x2000 + (size_t)off);
        void *const dx = form == 1 ? at : odd, *const mask = form == 0 ? nullptr : odd;
        const int rc = form == 2 ? rb_conv_dgrad_onto_tc(at, 2, P, P, 32, at, nullptr, 32, 32, 32, t.R, t.R, t.stride, t.pad, t.pad, 12,
                                                         12, dx, mask, nullptr, 0, nullptr, 0)
                                 : rb_conv_dgrad_tc(at, 2, P, P, 32, at, nullptr, 32, 32, 32, t.R, t.R, t.stride, t.pad, t.pad, 12, 12,
                                                    dx, nullptr, mask, nullptr, 0, nullptr, 0);
        expect(rc == want, form == 1 ? "mask" : "output");
        expect((g_launches != before) == (want == 0), "launched");
      }
}

// Weight-gradients: row plans are taken where the best of them wins by 3 %, whichever is timed first; the first of equal ones.
static float g_rows_ms[4];
static int g_rows_seen;
static float rows_take(const int* l) { return l[MODE] != A_ROWS ? 1.f : g_rows_ms[std::min(g_rows_seen++ / 3, 3)]; }
static int wgrad(int N, int C, int Ko, int H, int R, int pad, int beside, bool measure = false, long long lddy = 0) {
  void* const at = (void*)0x1000;
  const int P = H + 2 * pad - R + 1;
  if (measure) return rb_conv_wgrad_tune(at, N, H, H, C, at, Ko, Ko, R, R, pad, pad, P, P, (float*)at, beside, nullptr, 0);
  return rb_conv_wgrad_tc(at, N, H, H, C, at, lddy ? lddy : Ko, Ko, R, R, 1, pad, pad, P, P, (float*)at, 0, beside, nullptr, 0);
}
static void row_plans_win_by_a_margin() {
  g_time = rows_take;
  const struct { float ms[4]; bool rows; const char* what; } tries[] = {
      {{1.02f, 1.01f, 1.f, 1.f}, false, "slower"}, {{.98f, .99f, 1.f, 1.f}, false, "2 % faster"},
      {{.98f, .96f, 1.f, .99f}, true, "the second 4 % faster"}, {{.9f, .96f, .91f, .99f}, true, "the first 10 % faster"},
      {{.96f, .965f, .955f, .95f}, true, "all by little"}};
  for (auto& t : tries)
    for (int beside = 0; beside <= 1; ++beside) {
      rb_gemm_clear_plans();
      g_rows_seen = 0;
      memcpy(g_rows_ms, t.ms, sizeof(g_rows_ms));
      expect(wgrad(64, 32, 32, 32, 3, 1, beside, true) == 0, t.what);
      expect(g_rows_seen == 12, "four row plans timed three times");
      expect(wgrad(64, 32, 32, 32, 3, 1, beside) == 0 && (g_last_launch[MODE] == A_ROWS) == t.rows, t.what);
      int took[9];
      memcpy(took, g_last_launch, sizeof(took));
      g_opt.force_rows = 1 + (int)(std::min_element(t.ms, t.ms + 4) - t.ms);
      expect(wgrad(64, 32, 32, 32, 3, 1, beside) == 0 && (memcmp(took, g_last_launch, sizeof(took)) == 0) == t.rows, "the fastest");
      g_opt.force_rows = -1;
    }
}

// What stands in the way of measuring a weight-gradient is said, and nothing is remembered; what was measured is for that shape, those
// paddings and that form alone; shapes of little work and `deterministic` stay with the general kernel.
static float rows_are_fastest(const int* l) { return l[MODE] == A_ROWS ? 1.f : 2.f; }
static void row_plans_are_remembered() {
  g_time = rows_are_fastest;
  int* const in_the_way[] = {&g_opt.deterministic, &g_opt.force_mt, &g_opt.force_taps, &g_opt.force_box, &g_opt.force_resident,
                             &g_opt.force_rows, &g_opt.bn_cap, &g_opt.autotune};
  for (int* option : in_the_way) {
    const int was = *option;
    *option = option == &g_opt.bn_cap ? 128 : option == &g_opt.autotune ? 0 : 1;
    expect(wgrad(64, 32, 32, 32, 3, 1, 0, true) == 1 && g_rows_cache.empty(), "an option in the way");
    *option = was;
    expect(wgrad(64, 32, 32, 32, 3, 1, 0) == 0 && g_last_launch[MODE] != A_ROWS, "not measured");
  }
  for (int beside = 0; beside <= 1; ++beside) {
    expect(wgrad(64, 32, 32, 32, 3, 1, beside) == 0 && g_last_launch[MODE] != A_ROWS, "the other form was measured");
    expect(wgrad(64, 32, 32, 32, 3, 1, beside, true) == 0 && g_rows_cache.size() == 1u + beside, "measured");
    expect(wgrad(64, 32, 32, 32, 3, 1, beside) == 0 && g_last_launch[MODE] == A_ROWS, "measured");
    const WgradRowsParams& p = g_rows_cache.rbegin()->second;
    expect(p.stages * (p.dy_blocks * p.dy_block + p.ncb * p.x_block) <= (beside ? LEAN_TILE_BYTES : TILE_SMEM_BYTES), "fits");
    expect(wgrad(63, 32, 32, 32, 3, 1, beside) == 0 && g_last_launch[MODE] != A_ROWS, "another batch");
    expect(wgrad(64, 32, 32, 34, 3, 0, beside) == 0 && g_last_launch[MODE] != A_ROWS, "the same output at padding 0");
    expect(wgrad(64, 32, 32, 32, 3, 1, beside, false, 64) == 0 && g_last_launch[MODE] == A_ROWS, "longer rows of dy");
    g_opt.deterministic = 1;
    expect(wgrad(64, 32, 32, 32, 3, 1, beside) == 0 && g_last_launch[MODE] != A_ROWS, "deterministic");
    g_opt.deterministic = 0;
  }
  const size_t before = g_rows_cache.size();      // 0.199 GFLOP
  expect(wgrad(42, 32, 32, 16, 3, 1, 0, true) == 0 && g_rows_cache.size() == before, "little work");
  expect(wgrad(42, 32, 32, 16, 3, 1, 0) == 0 && g_last_launch[MODE] != A_ROWS, "little work");
  expect(wgrad(43, 32, 32, 16, 3, 1, 0, true) == 0 && g_rows_cache.size() == before + 1, "enough work");
  rb_gemm_clear_plans();
  expect(wgrad(64, 32, 32, 32, 3, 1, 0) == 0 && g_last_launch[MODE] != A_ROWS, "forgotten");
}

int main(int argc, char** argv) {
  const struct { const char* name; void (*run)(); } scenarios[] = {
      {"remembered_flat_does_not_fit", remembered_flat_does_not_fit},
      {"paddings_are_measured_apart", paddings_are_measured_apart},
      {"sub_tiles_of_other_modes", sub_tiles_of_other_modes},
      {"deterministic_keeps_one_order", deterministic_keeps_one_order},
      {"pairs_win_by_a_margin", pairs_win_by_a_margin},
      {"flat_tiles_within_the_cap", flat_tiles_within_the_cap},
      {"addends_are_aligned", addends_are_aligned},
      {"strided_outputs_are_aligned", strided_outputs_are_aligned},
      {"row_plans_win_by_a_margin", row_plans_win_by_a_margin},
      {"row_plans_are_remembered", row_plans_are_remembered}};
  g_encode_tiled = no_tiled;
  g_encode_im2col = no_im2col;
  g_num_sms = 148;
  g_pair_clusters = 74;
  for (auto& s : scenarios)
    if (argc > 1 && strcmp(argv[1], s.name) == 0) {
      s.run();
      return g_wrong;
    }
  printf("no such scenario\n");
  return 2;
}
