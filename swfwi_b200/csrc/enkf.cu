// The ensemble Kalman analysis of swfwi's EnFWI (src/enfwi/enkfanalyze.cpp)
// on the GPU, in FP64.
//
// calGainMatrix (enkfanalyze.cpp:185-341) forms, over rows = nt*ng data
// samples and N members, HA' = HA - rowmean(HA), the perturbed data
// D = dobs + pert, gamma = pert - rowmean(pert), band = HA' + gamma, the SVD
// band = U S V', and the N x N gain t4 = HA'^T U SSqInv U^T (D - HA) with
// SSqInv = diag(1/s_i^2) for the first clipPosition(S) singular values.
// With U = band V S^-1 that is
//   t4 = X2 V diag(s_i^-4, i < clip) V^T X3,
//   X1 = band^T band,  X2 = HA'^T band,  X3 = band^T (D - HA),
// and s_i^2, V the eigenpairs of X1.  The three N x N cross products are
// the only work over the data (O(rows N^2)); one fused pass forms them row
// by row (row means, perturbation, band and residual never reach HBM), a
// fixed-order reduction sums the per-CTA partials, one CTA solves the N x N
// eigen problem (parallel-ordered two-sided Jacobi in FP64 shared memory),
// sorts it and applies clipPosition, and a few small kernels form V and t4,
// which stays in device memory for the member update.
//
// analyze (enkfanalyze.cpp:57-111) then moves each member by
// A' t4 (A' = members - their float mean), in physical velocity.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>
#include "common.hpp"
#include "kernels.cuh"

namespace swfwi {
namespace {

constexpr int kMaxMembers = 64;   // members per analysis (one 64 x 64 tile)
constexpr int kThreads = 256;

// ---- counter-based normal draws (Philox4x32-10 of Salmon et al. 2011,
// "Parallel random numbers: as easy as 1, 2, 3"; Box-Muller transform)
__device__ __forceinline__ void philox_round(uint32_t (&c)[4], const uint32_t (&k)[2]) {
  const uint32_t m0 = 0xD2511F53u, m1 = 0xCD9E8D57u;
  const uint32_t hi0 = __umulhi(m0, c[0]), lo0 = m0 * c[0];
  const uint32_t hi1 = __umulhi(m1, c[2]), lo1 = m1 * c[2];
  const uint32_t n0 = hi1 ^ c[1] ^ k[0], n1 = lo1, n2 = hi0 ^ c[3] ^ k[1], n3 = lo0;
  c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
}

__device__ __forceinline__ double normal_draw(unsigned long long seed, unsigned long long index) {
  uint32_t c[4] = {(uint32_t)index, (uint32_t)(index >> 32), 0u, 0u};
  uint32_t k[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
#pragma unroll
  for (int r = 0; r < 10; r++) {
    philox_round(c, k);
    k[0] += 0x9E3779B9u;
    k[1] += 0xBB67AE85u;
  }
  const double u1 = ((double)c[0] + 1.0) * 2.3283064365386963e-10;   // (0, 1]
  const double u2 = (double)c[1] * 2.3283064365386963e-10;           // [0, 1)
  return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

// ---- max |HA'| as initPerturbation picks it: the first element (member-
// major order) whose float |x| is largest.  key = float bits of |x| above
// the inverted element index, so the largest key is that element.
__global__ void k_maxkey(unsigned long long *best, const float *hona, long long rows, int n) {
  unsigned long long mine = 0;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < rows;
       r += (long long)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int i = 0; i < n; i++) s += (double)hona[i * rows + r];
    const double mean = s / n;
    for (int i = 0; i < n; i++) {
      const double x = (double)hona[i * rows + r] - mean;
      const uint32_t key = __float_as_uint(fabsf((float)x));
      const uint32_t inv = 0xFFFFFFFFu - (uint32_t)(i * rows + r);
      const unsigned long long v = ((unsigned long long)key << 32) | inv;
      mine = v > mine ? v : mine;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, o);
    mine = other > mine ? other : mine;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(best, mine);
}

// sigma = |HA'| of that element times the perturbation factor
// (initPerturbation, enkfanalyze.cpp:621-635)
__global__ void k_value_at(double *sigma, const unsigned long long *best, const float *hona, long long rows,
                           int n, float sigfac) {
  const uint32_t idx = 0xFFFFFFFFu - (uint32_t)(*best & 0xFFFFFFFFull);
  const long long r = idx % rows;
  const int i0 = (int)(idx / rows);
  double s = 0.0;
  for (int i = 0; i < n; i++) s += (double)hona[i * rows + r];
  *sigma = fabs((double)hona[i0 * rows + r] - s / n) * (double)sigfac;
}

// D += A B on the FP64 tensor cores: A 8 x 4 (lane: row lane / 4, column
// lane % 4), B 4 x 8 (row lane % 4, column lane / 4), D row lane / 4,
// columns 2 * (lane % 4) and the next.
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// ---- the three cross products, one pass over the rows, a CTA per SM and 32
// rows at a time.  A warp takes 8 rows x 16 members (a lane 4 members of a
// row): it reads HA, draws the perturbation, sums both by row, and once the
// four warps of a row have their sums writes HA', band and D - HA to shared
// memory, [member][row] with a stride that serves the products' fragments
// (an A and a B fragment of the same operand are the same 8 x 4 values)
// without bank conflicts.  The products run on the FP64 tensor cores, an
// 8 x 32 strip of X1, X2 and X3 a warp, while half of the warps draw the
// next rows.  Both use the FP64 pipe, which bounds it: 61 % busy, 44 with
// products and 17 with draws.  461000 rows of 64 members: 0.71 ms; 1.92 with
// 4 x 4 tiles of plain FP64 a thread, row sums by 16 threads of 256 and
// everything in turn.  partials[cta][3][64][64].
constexpr int kCrossThreads = 512;
constexpr int kRows = 32;         // rows of a chunk
constexpr int kLdr = kRows + 4;   // 4 mod 16: an 8 x 4 fragment covers the banks once

__host__ __device__ constexpr size_t cross_smem_bytes() {
  return sizeof(double) * (3 * kMaxMembers * kLdr + 2 * 4 * kRows);
}

template <bool DRAW>
__global__ void __launch_bounds__(kCrossThreads, 1)
k_cross(double *partials, const float *hona, const float *dobs, const double *z, long long rows, int n,
        const double *sigma_dev, unsigned long long seed) {
  extern __shared__ __align__(16) double cross_sm[];
  double *sh = cross_sm;                        // HA'   [64][kLdr]
  double *sp = sh + kMaxMembers * kLdr;         // band
  double *sr = sp + kMaxMembers * kLdr;         // D - HA
  double *sums = sr + kMaxMembers * kLdr;       // [2][member set][row]
  const double sigma = *sigma_dev;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // producer: row lrow of the chunk, members 16 * set + 4 * q + lane / 8
  const int set = warp >> 2, lrow = (warp & 3) * 8 + (lane & 7), m0 = 16 * set + (lane >> 3);
  // products: rows of tile ti, columns of tiles tj .. tj+3
  const int ti = warp >> 1, tj = (warp & 1) * 4, tiles = (n + 7) / 8;
  const int frag = (lane >> 2) * kLdr + (lane & 3);
  double a1[4][2] = {}, a2[4][2] = {}, a3[4][2] = {};
  double h[4], p[4], d = 0.0;

  auto draw = [&](long long r0) {
    const long long r = r0 + lrow;
    const bool rok = r < rows;
    double s = 0.0, u = 0.0;
    d = rok ? (double)dobs[r] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = m0 + 4 * q;
      h[q] = p[q] = 0.0;
      if (rok && i < n) {
        h[q] = (double)hona[i * rows + r];
        p[q] = sigma * (DRAW ? normal_draw(seed, (unsigned long long)(i * rows + r)) : z[i * rows + r]);
      }
      s += h[q];
      u += p[q];
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      u += __shfl_xor_sync(0xffffffffu, u, o);
    }
    if (lane < 8) {
      sums[set * kRows + lrow] = s;
      sums[(4 + set) * kRows + lrow] = u;
    }
  };
  auto finish = [&](long long r0) {
    const bool rok = r0 + lrow < rows;
    double s = 0.0, u = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      s += sums[k * kRows + lrow];
      u += sums[(4 + k) * kRows + lrow];
    }
    const double mh = s / n, mp = u / n;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int i = m0 + 4 * q;
      const bool ok = rok && i < n;
      const double hap = h[q] - mh;
      sh[i * kLdr + lrow] = ok ? hap : 0.0;
      sp[i * kLdr + lrow] = ok ? hap + (p[q] - mp) : 0.0;
      sr[i * kLdr + lrow] = ok ? (d + p[q]) - h[q] : 0.0;
    }
  };
  auto products = [&] {
    if (ti >= tiles || tj >= tiles) return;
#pragma unroll 2
    for (int k = 0; k < kRows; k += 4) {
      const double gb = sp[ti * 8 * kLdr + frag + k], gh = sh[ti * 8 * kLdr + frag + k];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int o = (tj + j) * 8 * kLdr + frag + k;   // members past n are zeros
        const double b = sp[o], r = sr[o];
        mma_f64(a1[j], gb, b);
        mma_f64(a2[j], gh, b);
        mma_f64(a3[j], gb, r);
      }
    }
  };

  const long long step = (long long)gridDim.x * kRows;
  long long r0 = (long long)blockIdx.x * kRows;
  draw(r0);
  __syncthreads();
  finish(r0);
  for (; r0 < rows; r0 += step) {
    __syncthreads();   // this chunk is in shared memory
    if (warp & 4) {
      products();
      draw(r0 + step);
    } else {
      draw(r0 + step);
      products();
    }
    __syncthreads();   // its products and the next one's sums are done
    finish(r0 + step);
  }
  double *out = partials + (long long)blockIdx.x * 3 * kMaxMembers * kMaxMembers;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int e = (ti * 8 + (lane >> 2)) * kMaxMembers + (tj + j) * 8 + 2 * (lane & 3);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      out[e + c] = a1[j][c];
      out[kMaxMembers * kMaxMembers + e + c] = a2[j][c];
      out[2 * kMaxMembers * kMaxMembers + e + c] = a3[j][c];
    }
  }
}

// Sum of the per-CTA partials in CTA order (deterministic).
__global__ void __launch_bounds__(64) k_sum_partials(double *x, const double *partials, int nparts) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = 3 * kMaxMembers * kMaxMembers;
  if (e >= m) return;
  double s = 0.0;
#pragma unroll 8
  for (int b = 0; b < nparts; b++) s += partials[(long long)b * m + e];
  x[e] = s;
}

// ---- analyze's update: the members' float mean (createAMean,
// enkfanalyze.cpp:568-580), A' in double, A' t4, and
// v <- velTrans(velRecover(v) + (A' t4)_i) (enkfanalyze.cpp:72-108).  A CTA
// takes 128 model points: their values of every member stay in shared memory
// (one read and one write of HBM), the mean is summed there in member order,
// and A' t4 runs on the FP64 tensor cores, 16 points x all members a warp.
// 64 members of 129519 points: 87 us; 318 with a thread per point, its 64
// sums of 64 terms re-read from L1 and spilled.
constexpr int kTile = 128;          // points of a CTA
constexpr int kLdp = kTile + 8;     // floats a member row: 8 mod 32
constexpr int kLdg = kMaxMembers + 4;   // doubles a column of t4: 4 mod 16

__host__ __device__ constexpr size_t update_smem_bytes() {
  return sizeof(double) * kMaxMembers * kLdg + sizeof(float) * (kMaxMembers * kLdp + kTile);
}

__device__ __forceinline__ void update_members(float *vels, long long model, int n, const double *t4, float dx,
                                               float dt) {
  extern __shared__ __align__(16) double update_sm[];
  double *g = update_sm;                                      // t4, column i at i * kLdg, zeros past n
  float *sv = reinterpret_cast<float *>(g + kMaxMembers * kLdg);   // [64][kLdp]
  float *mean = sv + kMaxMembers * kLdp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tiles = (n + 7) / 8;
  for (int e = tid; e < kMaxMembers * kMaxMembers; e += kThreads) {
    const int i = e / kMaxMembers, j = e - i * kMaxMembers;
    g[i * kLdg + j] = i < n && j < n ? t4[i * n + j] : 0.0;
  }
  const float dx2 = __fmul_rn(dx, dx), dt2 = __fmul_rn(dt, dt);
  for (long long p0 = (long long)blockIdx.x * kTile; p0 < model; p0 += (long long)gridDim.x * kTile) {
    __syncthreads();
    for (int e = tid; e < n * kTile; e += kThreads) {
      const int j = e / kTile, k = e - j * kTile;
      sv[j * kLdp + k] = p0 + k < model ? vels[j * model + p0 + k] : 1.0f;
    }
    __syncthreads();
    if (tid < kTile) {
      float s = 0.0f;
#pragma unroll 8
      for (int j = 0; j < n; j++) s = __fadd_rn(s, sv[j * kLdp + tid]);
      mean[tid] = __fdiv_rn(s, (float)n);
    }
    __syncthreads();
    // every member's A' t4 from the values before any of them is written:
    // a warp reads and writes its own points only
    const int pt = warp * 16 + (lane >> 2);
    const double mu[2] = {(double)mean[pt], (double)mean[pt + 8]};
    double acc[2][8][2] = {};
    for (int k = 0; k < n; k += 4) {
      const int j = k + (lane & 3);
      double a[2];
#pragma unroll
      for (int t = 0; t < 2; t++) a[t] = j < n ? (double)sv[j * kLdp + pt + 8 * t] - mu[t] : 0.0;
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (i < tiles) {
          const double b = g[(i * 8 + (lane >> 2)) * kLdg + j];
          mma_f64(acc[0][i], a[0], b);
          mma_f64(acc[1][i], a[1], b);
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const int m = i * 8 + 2 * (lane & 3) + c;
          if (m < n) {
            float *v = sv + m * kLdp + pt + 8 * t;
            const float phys = __fsqrt_rn(__fdiv_rn(dx2, __fmul_rn(dt2, *v)));
            const float upd = (float)((double)phys + acc[t][i][c]);
            *v = __fdiv_rn(dx2, __fmul_rn(__fmul_rn(dt2, upd), upd));
          }
        }
    __syncthreads();
    for (int e = tid; e < n * kTile; e += kThreads) {
      const int j = e / kTile, k = e - j * kTile;
      if (p0 + k < model) vels[j * model + p0 + k] = sv[j * kLdp + k];
    }
  }
}

__global__ void __launch_bounds__(kThreads)
k_update(float *vels, long long model, int n, const double *t4, float dx, float dt) {
  update_members(vels, model, n, t4, dx, dt);
}

// the same after a device-side gain: nothing moves if the gain was not finite
__global__ void __launch_bounds__(kThreads)
k_update_guarded(float *vels, long long model, int n, const double *t4, float dx, float dt, const int *status) {
  if (status[1]) return;
  update_members(vels, model, n, t4, dx, dt);
}

__global__ void k_mean(float *mean, const float *vels, long long model, int n) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < model;
       p += (long long)gridDim.x * blockDim.x) {
    float s = 0.0f;
    for (int j = 0; j < n; j++) s = __fadd_rn(s, vels[j * model + p]);
    mean[p] = __fdiv_rn(s, (float)n);
  }
}

unsigned grid_of(long long n, int per) {
  long long g = (n + per - 1) / per;
  return (unsigned)std::max(1LL, std::min(g, 4096LL));
}

// ---- the gain from the cross products.  x = [X1 | X2 | X3], each K x K
// row-major (K = kMaxMembers), first n x n used.
//
// Eigenvalues of the symmetric X1 by two-sided Jacobi in the round-robin
// (tournament) ordering, one CTA: each round rotates n/2 disjoint index
// pairs at once, A <- J^T A J with J the product of the round's plane
// rotations, n-1 rounds a sweep (n odd: one player idles, a zero row).
// Sweeps stop when the off-diagonal square sum is at most 1e-30 of the
// total (or after 100).  Eigenvalues sorted descending (ties by index),
// s_k = sqrt(max(lambda_k, 0)), c = clipPosition(s)
// (src/enfwi/Matrix.cpp:170-185).  The rotations go to `rot` and k_vectors
// applies them to the rows of V, which do not depend on each other; then
//   t4 = (X2 V_c diag(s^-4)) (V_c^T X3),  written column-major (the
// reference's Matrix): t4[j*n + i] = row i, column j.
// status[0] = c, status[1] = 1 if any cross product is not finite,
// status[2] = rounds.
//
// What bounds it is the chain of a round: a pair's angle (two reciprocal
// roots in FP64), then everybody's rotation.  So A has two copies, read and
// written in turn: while 496 threads rotate the 2 x 2 blocks of a round, one
// a thread and the upper triangle only, the warp of the angles forms the
// next round's off-diagonal elements itself from the same copy and goes on
// to their angles; a round has one barrier.  Rows and columns are kept by
// their place in the tournament (pair k's players at k and 32 + k), so that
// a round moves every element by the same permutation and a thread's
// addresses never change.  64 members: 0.39 ms, and 0.05 for V; 2.07 ms with
// columns, rows, angles and V in turn in one CTA, 0.54 with one barrier but
// player indices and the angle by square root and division.
constexpr int kPairs = kMaxMembers / 2;
constexpr int kBlocks = kPairs * (kPairs - 1) / 2;
constexpr int kAngleWarp = (kBlocks + 31) / 32;
constexpr int kGainThreads = (kAngleWarp + 1) * 32;
constexpr int kLd = kMaxMembers + 1;   // the two rows that share a row of the triangle's storage
constexpr int kTriangle = kMaxMembers * kLd / 2;
constexpr int kMaxSweeps = 100;
// rotations of at most kMaxSweeps, and the round formed ahead of the last
constexpr int kMaxRotations = (kMaxSweeps * (kMaxMembers - 1) + 1) * kPairs;

// The players of pair k in the first round of m - 1, and of every sweep:
// round r pairs (r + k, r - k) modulo m-1, pair 0 player m-1 with player r.
// From a round to the next the player at place k (k > 0) moves to k - 1,
// the one at 0 to 32 + 1, at 32 + k (k > 0) to 32 + k + 1, the last of
// these to the last place k; the one at 32 stays.
__device__ __forceinline__ int player_u(int k) { return k; }
__device__ __forceinline__ int player_w(int k, int m) { return m - 1 - k; }
__device__ __forceinline__ int place_next(int place, int half) {
  if (half == 1 || place == kPairs) return place;
  if (place < kPairs) return place == 0 ? kPairs + 1 : place - 1;
  return place == kPairs + half - 1 ? half - 1 : place + 1;
}
__device__ __forceinline__ int place_before(int place, int half) {
  if (half == 1 || place == kPairs) return place;
  if (place < kPairs) return place == half - 1 ? kPairs + half - 1 : place + 1;
  return place == kPairs + 1 ? 0 : place - 1;
}
// the same for the values of a pair's two players, one pair a lane
__device__ __forceinline__ void pass_on(double &u, double &w, int lane, int half) {
  const double up = __shfl_down_sync(0xffffffffu, u, 1);
  const double dn = __shfl_up_sync(0xffffffffu, lane == 0 ? u : w, 1);
  const double nu = half == 1 ? u : lane == half - 1 ? w : up;
  w = lane == 0 ? w : dn;
  u = nu;
}
// element (i, j) of the triangle, i != j: rows i and 63 - i share kLd doubles
__device__ __forceinline__ int at(int i, int j) {
  const int lo = min(i, j), hi = max(i, j);
  return lo < kPairs ? lo * kLd + hi : (kMaxMembers - 1 - lo) * kLd + kMaxMembers - hi - 1;
}

__global__ void __launch_bounds__(kGainThreads)
k_eigen(double2 *rot, double *sv_out, int *ord_out, int *status, const double *x, int n) {
  __shared__ double A[2][kTriangle];
  __shared__ double w[kMaxMembers], sv[kMaxMembers];
  __shared__ double2 cs[2][kPairs];
  __shared__ double red[2][kAngleWarp + 1];
  __shared__ int ord[kMaxMembers], flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = kMaxMembers, m = (n + 1) & ~1, half = m / 2;

  if (tid == 0) flag = 0;
  for (int e = tid; e < 2 * kTriangle; e += kGainThreads) (&A[0][0])[e] = 0.0;
  if (tid < K) w[tid] = 0.0;
  __syncthreads();
  for (int e = tid; e < n * n; e += kGainThreads) {
    const int i = e / n, j = e - i * n;
    const double a = x[i * K + j], b = x[K * K + i * K + j], c = x[2 * K * K + i * K + j];
    if (!isfinite(a) || !isfinite(b) || !isfinite(c)) flag = 1;
    // player p's place
    const int pi = i < half ? i : kPairs + m - 1 - i, pj = j < half ? j : kPairs + m - 1 - j;
    if (i < j) A[0][at(pi, pj)] = a;
    if (i == j) w[i] = a;
  }
  __syncthreads();
  if (flag) {
    if (tid == 0) {
      status[0] = 0;
      status[1] = 1;
      status[2] = 0;
    }
    return;
  }

  // this thread's elements, read at f and written, a round on, at g: the
  // block of pairs ba < bb; or (angles) the four that form the next
  // element of pair `lane`
  int ba = 0, bb = 0, f[4] = {}, g[4] = {}, own = 0;
  bool su = false, sw = false;   // angles: the next players are their pairs' second now
  const bool angles = warp == kAngleWarp && lane < half;
  if (tid < half * (half - 1) / 2) {
    int t = tid;
    while (t >= half - 1 - ba) t -= half - 1 - ba++;
    bb = ba + 1 + t;
  }
  const bool block = bb > 0;
  if (angles) {
    const int i = place_before(lane, half), j = place_before(kPairs + lane, half);
    ba = i % kPairs;
    bb = j % kPairs;
    su = i >= kPairs;
    sw = j >= kPairs;
    own = half == 1 ? at(0, kPairs) : at(place_next(lane, half), place_next(kPairs + lane, half));
  }
  if (block || (angles && ba != bb)) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int i = ba + (e & 2 ? kPairs : 0), j = bb + (e & 1 ? kPairs : 0);
      f[e] = at(i, j);
      g[e] = at(place_next(i, half), place_next(j, half));
    }
  }

  // the rotation of pair `lane` from its off-diagonal element o:
  // cos 2 theta = |d| / h, h = sqrt(d^2 + 4 o^2), and c, s of the half angle.
  // du, dw: the diagonal, which it moves
  double du = 0.0, dw = 0.0;
  auto angle = [&](double o, int buf, long long r) {
    double c = 1.0, s = 0.0;
    const double d = dw - du, o2 = 2.0 * o, h2 = fma(d, d, o2 * o2);
    if (o != 0.0 && h2 > 0.0 && h2 < 1e300) {
      const double rh = rsqrt(h2), y = 0.5 * rh, cc = fma(fabs(d), y, 0.5), rc = rsqrt(cc);
      c = cc * rc;
      s = (d >= 0.0 ? o2 : -o2) * y * rc;
      const double t = s * rc;
      du = fma(-t, o, du);
      dw = fma(t, o, dw);
    }
    cs[buf][lane] = make_double2(c, s);
    rot[r * kPairs + lane] = make_double2(c, s);
  };
  if (warp == kAngleWarp) {
    if (angles) {
      du = w[player_u(lane)];
      dw = w[player_w(lane, m)];
      angle(A[0][at(lane, kPairs + lane)], 0, 0);
    }
  }

  int cur = 0;          // the copy to read
  long long r = 0;      // rounds begun; angles are ready for this one
  for (int sweep = 0; sweep < kMaxSweeps; sweep++) {
    __syncthreads();
    double off = 0.0, tot = 0.0;
    for (int e = tid; e < kTriangle; e += kGainThreads) off += A[cur][e] * A[cur][e];
    // the diagonal is a round ahead (the angles formed last): tot exceeds
    // the total by no more than off
    if (angles) tot = du * du + dw * dw;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if (lane == 0) {
      red[0][warp] = off;
      red[1][warp] = tot;
    }
    __syncthreads();
    off = 0.0;
    for (int k = 0; k <= kAngleWarp; k++) off += red[0][k];
    off *= 2.0;
    tot = red[1][kAngleWarp] + off;
    if (off <= 1e-30 * tot || off == 0.0) break;
    for (int round = 0; round < m - 1; round++) {
      const double *B = A[cur];
      double *D = A[cur ^ 1];
      const double2 *rc = cs[r & 1];
      if (block) {
        const double xpp = B[f[0]], xpq = B[f[1]], xqp = B[f[2]], xqq = B[f[3]];
        const double2 ra = rc[ba], rb = rc[bb];
        const double ypp = rb.x * xpp - rb.y * xpq, ypq = rb.y * xpp + rb.x * xpq;
        const double yqp = rb.x * xqp - rb.y * xqq, yqq = rb.y * xqp + rb.x * xqq;
        D[g[0]] = ra.x * ypp - ra.y * yqp;
        D[g[2]] = ra.y * ypp + ra.x * yqp;
        D[g[1]] = ra.x * ypq - ra.y * yqq;
        D[g[3]] = ra.y * ypq + ra.x * yqq;
      } else if (warp == kAngleWarp) {
        double o = 0.0;
        if (angles && ba != bb) {
          const double2 ra = rc[ba], rb = rc[bb];
          const double cb = sw ? rb.y : rb.x, sb = sw ? rb.x : -rb.y;
          const double ca = su ? ra.y : ra.x, sa = su ? ra.x : -ra.y;
          o = ca * (cb * B[f[0]] + sb * B[f[1]]) + sa * (cb * B[f[2]] + sb * B[f[3]]);
        }
        pass_on(du, dw, lane, half);
        if (angles) {
          D[own] = 0.0;   // the pair's own element is rotated to zero
          angle(o, (r + 1) & 1, r + 1);
        }
      }
      __syncthreads();
      cur ^= 1;
      r++;
    }
  }
  // round r, formed ahead, is in the diagonal and goes into V; in A it would
  // move elements that are at rounding level.  Places are the first round's
  if (angles) {
    w[player_u(lane)] = du;
    w[player_w(lane, m)] = dw;
  }
  __syncthreads();
  // descending order of the eigenvalues, ties by index
  if (tid < n) {
    int rank = 0;
    const double wi = w[tid];
    for (int j = 0; j < n; j++) rank += (w[j] > wi || (w[j] == wi && j < tid)) ? 1 : 0;
    ord[rank] = tid;
  }
  __syncthreads();
  if (tid < n) {
    sv[tid] = sqrt(fmax(w[ord[tid]], 0.0));
    sv_out[tid] = sv[tid];
    ord_out[tid] = ord[tid];
  }
  __syncthreads();
  if (tid == 0) {
    // clipPosition (Matrix.cpp:170-185); relativeError is a float literal
    const double rel = (double)0.001f;
    double sum = 0.0;
    int pos;
    for (pos = 0; pos < n - 1; pos++) {
      sum += fabs(sv[pos]);
      if (rel / (1 - rel) * sum > (n - pos + 1) * sv[pos + 1]) break;
    }
    status[0] = pos + 1;
    status[1] = 0;
    status[2] = (int)r + 1;
  }
}

// Row blockIdx.x of V = the product of the rotations, one warp: lane k holds
// the row's entries of pair k's two players and passes them on.  A round is
// two dependent operations and a shuffle; its rotations are loaded 8 to 16
// rounds ahead.
__global__ void __launch_bounds__(32) k_vectors(double *v, const double2 *rot, const int *status, int n) {
  const int row = blockIdx.x, lane = threadIdx.x, m = (n + 1) & ~1, half = m / 2;
  const int rounds = status[2];
  if (status[1]) return;
  constexpr int kAhead = 8;
  double2 c[kAhead], next[kAhead];
  const double2 *from = rot + min(lane, half - 1);
  auto load = [&](double2 (&x)[kAhead], int r) {
#pragma unroll
    for (int e = 0; e < kAhead; e++) x[e] = from[(long long)min(r + e, rounds - 1) * kPairs];
  };
  double u = player_u(lane) == row ? 1.0 : 0.0, w = player_w(lane, m) == row ? 1.0 : 0.0;
  if (lane >= half) u = w = 0.0;
  load(c, 0);
  for (int r = 0; r < rounds; r += kAhead) {
    load(next, r + kAhead);
#pragma unroll
    for (int e = 0; e < kAhead; e++)
      if (r + e < rounds) {
        if (r + e > 0) pass_on(u, w, lane, half);
        const double nu = c[e].x * u - c[e].y * w;
        w = c[e].y * u + c[e].x * w;
        u = nu;
      }
#pragma unroll
    for (int e = 0; e < kAhead; e++) c[e] = next[e];
  }
  // the last rotation is the first of a sweep: places are the first round's
  if (lane < half) {
    v[row * kMaxMembers + player_u(lane)] = u;
    v[row * kMaxMembers + player_w(lane, m)] = w;
  }
}

// left[i][k] = (X2 V)[i][ord[k]] s_k^-4 (first 64 threads, i = blockIdx.x);
// right[k][i] = (V^T X3)[ord[k]][i] (the others, k = blockIdx.x)
__global__ void __launch_bounds__(2 * kMaxMembers)
k_sides(double *left, double *right, const double *x, const double *v, const double *sv, const int *ord,
        const int *status, int n) {
  const int K = kMaxMembers, c = status[0], b = blockIdx.x, t = threadIdx.x % kMaxMembers;
  if (status[1]) return;
  if (threadIdx.x < kMaxMembers) {
    if (t >= c) return;
    const int col = ord[t];
    double l = 0.0;
#pragma unroll 8
    for (int j = 0; j < n; j++) l += x[K * K + b * K + j] * v[j * K + col];
    const double s2 = sv[t] * sv[t];
    left[b * K + t] = l * (1.0 / (s2 * s2));
  } else {
    if (b >= c || t >= n) return;
    const int col = ord[b];
    double r = 0.0;
#pragma unroll 8
    for (int j = 0; j < n; j++) r += v[j * K + col] * x[2 * K * K + j * K + t];
    right[b * K + t] = r;
  }
}

// row i = threadIdx.x, column j = blockIdx.x of t4
__global__ void __launch_bounds__(kMaxMembers)
k_gain(double *t4, const double *left, const double *right, const int *status, int n) {
  const int K = kMaxMembers, i = threadIdx.x, j = blockIdx.x, c = status[0];
  if (status[1] || i >= n) return;
  double acc = 0.0;
#pragma unroll 8
  for (int k = 0; k < c; k++) acc += left[i * K + k] * right[k * K + j];
  t4[j * n + i] = acc;
}

// Device memory of one analysis, held by the caller until its results are
// back.  The results come first: sigma, status ([0] clip, [1] non-finite
// cross products, [2] rounds), t4.
struct GainScratch {
  static constexpr size_t kSquare = (size_t)kMaxMembers * kMaxMembers;
  static constexpr int kResults = 3;   // doubles before t4
  static constexpr size_t bytes(int nparts) {
    return sizeof(double) * (kResults + 1 + 7 * kSquare + 2 * kMaxMembers + 2 * (size_t)kMaxRotations +
                             nparts * 3 * kSquare);
  }
  Scratch mem;
  double *sigma, *t4, *x, *v, *left, *right, *sv, *partials;
  int *status, *ord;
  double2 *rot;
  unsigned long long *best;

  explicit GainScratch(int nparts) : mem(bytes(nparts)) {
    double *p = static_cast<double *>(mem.get());
    auto take = [&p](size_t doubles) {
      double *q = p;
      p += doubles;
      return q;
    };
    sigma = take(1);
    status = reinterpret_cast<int *>(take(2));
    t4 = take(kSquare);
    best = reinterpret_cast<unsigned long long *>(take(1));   // rot below: 16-byte aligned
    rot = reinterpret_cast<double2 *>(take(2 * (size_t)kMaxRotations));
    x = take(3 * kSquare);
    v = take(kSquare);
    left = take(kSquare);
    right = take(kSquare);
    sv = take(kMaxMembers);
    ord = reinterpret_cast<int *>(take(kMaxMembers));
    partials = take(nparts * 3 * kSquare);
  }
};

int cross_parts(long long rows) {
  int dev = 0, sms = 148;
  SWFWI_CUDA(cudaGetDevice(&dev));
  SWFWI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return (int)std::min<long long>((rows + kRows - 1) / kRows, sms);
}

// The analysis's device part: sigma (first call), cross products, gain into
// sc.t4 [n*n] (column-major), sc.status, sc.sigma.
void gain_on_device(const float *hona, const float *dobs, const double *z, long long rows, int n, float sigfac,
                    const double *sigma_in, unsigned long long seed, int nparts, GainScratch &sc, cudaStream_t st) {
  if (!(*sigma_in > 0.0)) {
    // initPerturbation's first call: sigma = max|HA'| * sigmaFactor
    SWFWI_CUDA(cudaMemsetAsync(sc.best, 0, sizeof(unsigned long long), st));
    k_maxkey<<<grid_of(rows, kThreads), kThreads, 0, st>>>(sc.best, hona, rows, n);
    note_launch();
    k_value_at<<<1, 1, 0, st>>>(sc.sigma, sc.best, hona, rows, n, sigfac);
    note_launch();
  } else {
    SWFWI_CUDA(cudaMemcpyAsync(sc.sigma, sigma_in, sizeof(double), cudaMemcpyHostToDevice, st));
  }
  allow_smem(z ? k_cross<false> : k_cross<true>, cross_smem_bytes());
  if (z)
    k_cross<false><<<nparts, kCrossThreads, cross_smem_bytes(), st>>>(sc.partials, hona, dobs, z, rows, n, sc.sigma,
                                                                      seed);
  else
    k_cross<true><<<nparts, kCrossThreads, cross_smem_bytes(), st>>>(sc.partials, hona, dobs, nullptr, rows, n,
                                                                     sc.sigma, seed);
  note_launch();
  k_sum_partials<<<3 * kMaxMembers * kMaxMembers / 64, 64, 0, st>>>(sc.x, sc.partials, nparts);
  note_launch();
  k_eigen<<<1, kGainThreads, 0, st>>>(sc.rot, sc.sv, sc.ord, sc.status, sc.x, n);
  note_launch();
  k_vectors<<<n, 32, 0, st>>>(sc.v, sc.rot, sc.status, n);
  note_launch();
  k_sides<<<n, 2 * kMaxMembers, 0, st>>>(sc.left, sc.right, sc.x, sc.v, sc.sv, sc.ord, sc.status, n);
  note_launch();
  k_gain<<<n, kMaxMembers, 0, st>>>(sc.t4, sc.left, sc.right, sc.status, n);
  note_launch();
  SWFWI_CUDA(cudaGetLastError());
}

// sigma, clip and (unless null) t4 to the host, in one copy
void fetch_gain(GainScratch &sc, int n, double *sigma, double *t4, int *clip, cudaStream_t st) {
  std::vector<double> h(GainScratch::kResults + (t4 ? (size_t)n * n : 0));
  SWFWI_CUDA(cudaMemcpyAsync(h.data(), sc.sigma, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, st));
  SWFWI_CUDA(cudaStreamSynchronize(st));
  sc.mem.idle();
  int hs[2];
  std::memcpy(hs, &h[1], sizeof(hs));
  *sigma = h[0];
  if (t4) std::memcpy(t4, &h[GainScratch::kResults], sizeof(double) * n * n);
  if (hs[1]) throw Error(SWFWI_ERR_NONFINITE, "non-finite data in the analysis");
  if (clip) *clip = hs[0];
}

template <typename F, typename... Args>
void launch_update(F kernel, long long model, cudaStream_t st, Args... args) {
  allow_smem(kernel, update_smem_bytes());
  kernel<<<(unsigned)std::min<long long>((model + kTile - 1) / kTile, 444), kThreads, update_smem_bytes(), st>>>(
      args...);
  note_launch();
  SWFWI_CUDA(cudaGetLastError());
}

}  // namespace
}  // namespace swfwi

using namespace swfwi;

extern "C" int swfwi_enkf_gain_matrix(const float *hona, const float *dobs, const double *z, long long rows,
                                      int n, float sigfac, double *sigma, unsigned long long seed,
                                      double *t4, int *clip, void *stream) {
  return guarded([&] {
    SWFWI_REQUIRE(hona && dobs && sigma && t4, "null pointer");
    SWFWI_REQUIRE(n >= 2 && n <= kMaxMembers, "members must be 2..64");
    SWFWI_REQUIRE(rows > 0 && rows * n < 0xFFFFFFFFLL, "rows x members must be below 2^32");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int nparts = cross_parts(rows);
    GainScratch sc(nparts);
    gain_on_device(hona, dobs, z, rows, n, sigfac, sigma, seed, nparts, sc, st);
    fetch_gain(sc, n, sigma, t4, clip, st);
  });
}

extern "C" int swfwi_enkf_analyze(const float *hona, const float *dobs, const double *z, long long rows, int n,
                                  float sigfac, double *sigma, unsigned long long seed, float *vels,
                                  long long model_size, float dx, float dt, double *t4_out, int *clip,
                                  void *stream) {
  return guarded([&] {
    SWFWI_REQUIRE(hona && dobs && sigma && vels && model_size > 0, "null pointer or empty model");
    SWFWI_REQUIRE(n >= 2 && n <= kMaxMembers, "members must be 2..64");
    SWFWI_REQUIRE(rows > 0 && rows * n < 0xFFFFFFFFLL, "rows x members must be below 2^32");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int nparts = cross_parts(rows);
    GainScratch sc(nparts);
    gain_on_device(hona, dobs, z, rows, n, sigfac, sigma, seed, nparts, sc, st);
    // a non-finite gain leaves the members unchanged: the update skips when
    // status[1] is set
    launch_update(k_update_guarded, model_size, st, vels, model_size, n, (const double *)sc.t4, dx, dt,
                  (const int *)sc.status);
    fetch_gain(sc, n, sigma, t4_out, clip, st);
  });
}

extern "C" int swfwi_enkf_update(float *vels, long long model_size, int n, const double *t4, float dx,
                                 float dt, void *stream) {
  return guarded([&] {
    SWFWI_REQUIRE(vels && t4 && model_size > 0, "bad update arguments");
    SWFWI_REQUIRE(n >= 2 && n <= kMaxMembers, "members must be 2..64");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    Scratch g(sizeof(double) * n * n);
    SWFWI_CUDA(cudaMemcpyAsync(g.get(), t4, sizeof(double) * n * n, cudaMemcpyHostToDevice, st));
    launch_update(k_update, model_size, st, vels, model_size, n, static_cast<const double *>(g.get()), dx, dt);
    SWFWI_CUDA(cudaStreamSynchronize(st));
    g.idle();
  });
}

extern "C" int swfwi_enkf_mean(float *mean, const float *vels, long long model_size, int n, void *stream) {
  return guarded([&] {
    SWFWI_REQUIRE(mean && vels && model_size > 0 && n >= 1, "bad mean arguments");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    k_mean<<<grid_of(model_size, kThreads), kThreads, 0, st>>>(mean, vels, model_size, n);
    note_launch();
    SWFWI_CUDA(cudaGetLastError());
  });
}
