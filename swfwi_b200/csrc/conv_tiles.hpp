// Shapes of the row-tile convolution (k_conv3x3_tg in precond.cu) and the
// widths that it serves: plain functions, for the kernel, its launcher and
// host checks.
#pragma once
#include <cstddef>
#ifdef __CUDACC__
#define SWFWI_HD __host__ __device__
#else
#define SWFWI_HD
#endif

namespace swfwi {

constexpr int kMaxTmemCols = 256;   // tensor-memory columns that one CTA may take
// columns allocated for n: a power of two, at most kMaxTmemCols
SWFWI_HD constexpr int tmem_cols(int n) { return n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : kMaxTmemCols)); }

namespace tg {
constexpr int kGroupBytes = 160;                  // 10 pixels x 16 bytes
constexpr int kPlaneRow = 16 * kGroupBytes;       // one ky row of the 16 groups
constexpr int kCopyThreads = 320, kThreads = kCopyThreads + 32 + 128;
constexpr int kMaxStages = 6;
constexpr size_t kMaxSmem = 226 * 1024;
// output channels a CTA forms: all, or half where their weights would leave
// no room for two stages
SWFWI_HD constexpr int cols(int cin, int cout) {
  return cin / 16 * 9 * 32 * cout > 150 * 1024 - cin / 16 * 2 * kPlaneRow && cout % 32 == 0 ? cout / 2 : cout;
}
SWFWI_HD constexpr int weight_bytes(int cin, int cout) { return cin / 16 * 9 * 32 * cols(cin, cout); }
SWFWI_HD constexpr int stage_rows(int cin) { return cin <= 48 ? 3 : 1; }
SWFWI_HD constexpr int stage_bytes(int cin) { return cin / 16 * 2 * stage_rows(cin) * kPlaneRow; }
// stages: as many as leave room for a second CTA where weights and two
// stages are small, else for one
SWFWI_HD constexpr int stages(int cin, int cout) {
  const int w = weight_bytes(cin, cout), sb = stage_bytes(cin), half = 110 * 1024;
  const int n = w + 2 * sb <= half ? (half - w) / sb : ((int)kMaxSmem - 1024 - w) / sb;
  return n < kMaxStages ? n : kMaxStages;
}
SWFWI_HD constexpr size_t smem(int cin, int cout) {
  return (size_t)weight_bytes(cin, cout) + (size_t)stages(cin, cout) * stage_bytes(cin) + 256;
}
// Dynamic shared memory of a launch, raised where needed so that no more CTAs
// are resident on an SM than its tensor memory holds.
SWFWI_HD constexpr size_t launch_smem(int cin, int cout) {
  const int fit = 512 / tmem_cols(2 * cols(cin, cout));   // CTAs whose accumulators fit
  const size_t need = smem(cin, cout), cap = 228 * 1024 / (fit + 1) - 1024 + 16;
  return need > cap ? need : cap;
}
// The widths it takes: weights and two stages fit, and so do two accumulators
// in the tensor memory that a CTA allocates.
SWFWI_HD constexpr bool fits(int cin, int cout) {
  return stages(cin, cout) >= 2 && 2 * cols(cin, cout) <= kMaxTmemCols;
}
}  // namespace tg

}  // namespace swfwi
