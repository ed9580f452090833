// Launcher of the resident time loop (resident.cuh): how a batch is cut into
// launches, slabs and row chunks.
#include <algorithm>
#include "common.hpp"
#include "resident.hpp"
#include "resident.cuh"

namespace swfwi {

namespace {

constexpr size_t kMaxSmem = 227 * 1024;

int device_sms() {
  int dev = 0, n = 0;
  SWFWI_CUDA(cudaGetDevice(&dev));
  SWFWI_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
  return n;
}

int depth_groups(int nz) { return (nz - 6) / 4 + ((nz - 6) % 4 == 3 ? 1 : 0); }
int row_floats(int nz) { return 4 * depth_groups(nz) + 8; }

// most points of any `width` consecutive rows
int window_max(const std::vector<int> &hist, int width) {
  int sum = 0, most = 0;
  for (int x = 0; x < (int)hist.size(); x++) {
    sum += hist[x];
    if (x >= width) sum -= hist[x - width];
    most = std::max(most, sum);
  }
  return most;
}

// most strip cells in reach of any slab (backward)
int stage_cells(int nx, int nz, int bx0, int cps) {
  const int rows = nx - 12, nzs = std::max(nz - 6 - bx0, 0);
  int most = 0;
  auto overlap = [](int a0, int a1, int b0, int b1) { return std::max(std::min(a1, b1) - std::max(a0, b0), 0); };
  for (int c = 0; c < cps; c++) {
    const int ra = resident_detail::slab_first(rows, cps, c), rb = resident_detail::slab_first(rows, cps, c + 1) + 12;
    most = std::max(most, 6 * overlap(ra, rb, bx0 - 6, nx - bx0 + 6) +
                              nzs * (overlap(ra, rb, bx0 - 6, bx0) + overlap(ra, rb, nx - bx0, nx - bx0 + 6)));
  }
  return most;
}

// Row chunks of a slab of `rmax` rows: the count with the smallest estimate
// of a step's issue time.  A warp task costs about 10 instructions a row to
// fill the queue (12 rows), 62 for each u2 row (2 more than its outputs)
// and 58 for each output row (25 more where it also images); a round of
// `warps` tasks takes its tasks per scheduler times that, but no less than
// one task alone at about 2.5 cycles an instruction.
int row_chunks(bool back, int rmax, int ngroups, int warps) {
  double best = 1e30;
  int best_k = 1;
  for (int k = 1; k <= std::min(rmax, kResidentChunks); k++) {
    if ((long long)k * ngroups * ngroups >= (1 << 20)) break;
    const int L = (rmax + k - 1) / k;
    const int per_field = (k * ngroups + 29) / 30;
    const double cost = 120.0 + 62.0 * (L + 2) + (back ? 70.0 : 58.0) * L + 60.0;
    int left = per_field * (back ? 2 : 1);
    double t = 0;
    while (left > 0) {
      const int a = std::min(left, warps);
      t += cost * std::max(2.5, (double)((a + 3) / 4));
      left -= a;
    }
    if (t < best) {
      best = t;
      best_k = k;
    }
  }
  return best_k;
}

template <int ARITH, bool BACK, bool WIDE>
void launch_t(const ResidentArgs &a, size_t smem, cudaStream_t st) {
  allow_smem(fd_resident<ARITH, BACK, WIDE>, kMaxSmem);
  ResidentArgs b = a;
  void *args[] = {&b};
  SWFWI_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(fd_resident<ARITH, BACK, WIDE>),
                                         dim3(a.nslots * a.cps), dim3(kResidentThreads), args, smem, st));
}

}  // namespace

// thin: slabs may have fewer than 6 rows
static ResidentPlan plan_slabs(bool thin, int arith, bool back, int n, int nx, int nz, int bx0, bool strips,
                               const std::vector<int> &src_hist, const std::vector<int> &rec_hist) {
  ResidentPlan p;
  const int rows = nx - 12;
  if (n <= 0 || rows < 1 || nz < 16) return p;
  const int sms = device_sms(), zp = row_floats(nz);
  if (6LL * depth_groups(nz) * depth_groups(nz) >= (1 << 20)) return p;   // the index divisions by multiplication
  const int most = std::min(sms, thin ? rows : std::max(rows / 6, 1));   // a slab's halo: its neighbours' edge rows
  auto smem_of = [&](int cps, int &rmax, int &cs, int &cr, int &cg) {
    rmax = (rows + cps - 1) / cps;
    cs = window_max(src_hist, rmax + 12);
    cr = window_max(rec_hist, rmax + 12);
    cg = back && strips ? stage_cells(nx, nz, bx0, cps) : 0;
    return resident_smem(back, false, rmax, zp, cs, cr, cg);
  };
  // fewest slabs whose fields fit beside their lists, from the fewest whose
  // fields fit alone
  const int floats_row = (back ? 6 : 3) * zp, fixed = (back ? 48 : 24) * zp;
  const int rfit = ((int)(kMaxSmem / 4) - fixed) / floats_row;
  if (rfit < 1) return p;
  int cps = 0, rmax, cs, cr, cg;
  for (int c = (rows + rfit - 1) / rfit; c <= most && !cps; c++)
    if (smem_of(c, rmax, cs, cr, cg) <= kMaxSmem) cps = c;
  if (!cps) return p;
  const int slots_max = std::max(1, sms / cps);
  const int rounds = (n + slots_max - 1) / slots_max;
  p.slots = (n + rounds - 1) / rounds;
  p.rounds = rounds;
  p.cps = std::min(most, sms / p.slots);
  p.smem = smem_of(p.cps, p.rmax, p.cap_src, p.cap_rec, p.cap_stage);
  while (p.smem > kMaxSmem && p.cps > cps) p.smem = smem_of(--p.cps, p.rmax, p.cap_src, p.cap_rec, p.cap_stage);
  p.thin = rows / p.cps < 6;
  p.rows = rows;
  if (p.smem > kMaxSmem) return ResidentPlan();
  // The two-pass form: in REF arithmetic wherever it fits, in FAST up to two
  // rounds of u2 items.  Microseconds a forward step, two-pass / march: REF 1
  // shot of 533 x 193 2.7 / 4.8, 8 shots 6.0 / 8.3, 16 shots 10.0 / 11.8, 1
  // shot of 993 x 343 4.4 / 6.0; FAST 1 shot of 533 x 193 (282 items) 2.3 /
  // 2.9, 4 shots (799) 3.5 / 3.6, 8 shots (1457) 5.1 / 4.4, 1 shot of 993 x
  // 343 (756) 3.9 / 4.0, 2 shots (1344) 5.0 / 4.6.
  const long long u2_items = (back ? 2LL : 1LL) * (p.rmax + 2) * depth_groups(nz);
  const size_t two = resident_smem(back, true, p.rmax, zp, p.cap_src, p.cap_rec, p.cap_stage);
  p.wide = (arith == ARITH_REF || u2_items <= 800) && two <= kMaxSmem &&
           u2_items * depth_groups(nz) < (1 << 20);   // the index divisions by multiplication
  if (p.wide) p.smem = two;
  p.zp = zp;
  p.ngroups = depth_groups(nz);
  p.ogroups = (nz - 7) / 4;
  // helper warps: with one, strips and records hold up the exchange; more
  // than three take warps from the march (1 shot of 533 x 193, backward:
  // 10.6 / 6.2 / 5.5 / 5.5 us a step with 1 / 2 / 3 / 4)
  p.helpers = 3;
  p.chunks = row_chunks(back, p.rmax, p.ngroups, kResidentThreads / 32 - p.helpers);
  if (resident_halo(p.slots, p.cps, rows, p.thin, 2, p.ogroups) >= (1u << 31)) return ResidentPlan();
  p.halo = resident_halo(p.slots, p.cps, rows, p.thin, back ? 2 : 1, p.ogroups) + 1;   // and the launch's flag
  p.ok = true;
  return p;
}

// Slabs of fewer than 6 rows only in the two-pass form, which gains by them
// (533 x 193, 148 slabs against 86: 1 shot forward, REF, 2.5 / 3.2 us a step;
// an encoded epoch of 800 steps, FAST, 10.6 / 12.7 ms).
ResidentPlan plan_resident(int arith, bool back, int n, int nx, int nz, int bx0, bool strips,
                           const std::vector<int> &src_hist, const std::vector<int> &rec_hist) {
  const ResidentPlan p = plan_slabs(true, arith, back, n, nx, nz, bx0, strips, src_hist, rec_hist);
  return p.thin && !p.wide ? plan_slabs(false, arith, back, n, nx, nz, bx0, strips, src_hist, rec_hist) : p;
}

// Estimated microseconds a step (B200, fits to timed sweeps of 1..96 shots of
// 272 x 142, 533 x 193 and 993 x 343 padded points; within about 15 %).  A
// resident round costs its latency (points, exchange, barriers) plus its
// largest slab's march; a streamed step its launches plus its points.
// Measured forward / backward, FAST: 1 shot of 533 x 193 3.0 / 5.5 resident
// against 9.0 / 18.9 streamed; 20 shots 6.5 / 18.6 against 13.0 / 31.5; 96
// shots 28.8 / 114 against 36.1 / 108; 1 shot of 993 x 343 3.8 / 8.0 against
// 9.2 / 19.1; 10 shots 12.2 / 46 against 15.5 / 34; 96 shots 113 / 599
// against 87 / 227.
double resident_us(const ResidentPlan &p, int arith, bool back) {
  const double x = (double)p.rmax * p.ngroups;
  const bool ref = arith == ARITH_REF;
  double round;
  if (p.wide)
    round = back ? (ref ? 1.5 + 0.0066 * x : 1.7 + 0.0028 * x) + 0.045 * p.ogroups
                 : (ref ? 2.4 + 0.0028 * x : 2.1 + 0.0021 * x);
  else
    round = back ? (ref ? 3.5 + 0.0066 * x : 2.9 + 0.0028 * x) + 0.045 * p.ogroups
                 : (ref ? 3.9 + 0.0027 * x : 2.7 + 0.00113 * x);
  return p.rounds * round;
}
double streamed_us(int arith, bool back, double points, bool own_velocity) {
  const double m = points * 1e-6;
  if (arith == ARITH_REF) return back ? 30 + 10 * m : 14 + 3.9 * m;
  return back ? 17.5 + 6.6 * m : 8.3 + (own_velocity ? 4.9 : 2.4) * m;
}

void launch_resident(int arith, bool back, const ResidentPlan &p, ResidentArgs a, int nslots, cudaStream_t st) {
  a.nslots = nslots;
  a.cps = p.cps;
  a.rmax = p.rmax;
  a.zp = p.zp;
  a.ngroups = p.ngroups;
  a.ogroups = p.ogroups;
  a.gmagic = (1u << 20) / (unsigned)p.ngroups + 1;
  a.omagic = (1u << 20) / (unsigned)p.ogroups + 1;
  const int nzs = std::max(a.nz - 6 - a.bx0, 1);
  a.nzs_magic = (unsigned)((1ull << 32) / nzs + 1);
  a.chunks = p.chunks;
  a.thin = p.thin ? 1 : 0;
  a.helpers = p.helpers;
  a.cap_src = p.cap_src;
  a.cap_rec = p.cap_rec;
  a.cap_stage = p.cap_stage;
  const size_t halo = resident_halo(nslots, p.cps, p.rows, p.thin, back ? 2 : 1, p.ogroups);
  a.quit = reinterpret_cast<int *>(a.halo + halo);
  SWFWI_CUDA(cudaMemsetAsync(a.halo, 0, sizeof(uint4) * (halo + 1), st));
  auto go = [&](auto wide) {
    constexpr bool W = decltype(wide)::value;
    if (arith == ARITH_REF) {
      if (back) launch_t<ARITH_REF, true, W>(a, p.smem, st);
      else launch_t<ARITH_REF, false, W>(a, p.smem, st);
    } else {
      if (back) launch_t<ARITH_FAST, true, W>(a, p.smem, st);
      else launch_t<ARITH_FAST, false, W>(a, p.smem, st);
    }
  };
  if (p.wide) go(std::true_type());
  else go(std::false_type());
  note_launch();
}

}  // namespace swfwi
