// Resident time loop: a whole sweep of the 4th-order-time / 10th-order-space
// scheme in one launch, the wavefields held in shared memory.
//
// A streaming step (stream_rq.cuh, stream_rq2.cuh) is one launch a time step
// and another for the points around it; on grids of up to a few million
// points those launches, and the queue fill of short tasks, cost several
// times the arithmetic.  Here one cooperative launch runs every step.  Each
// slot (shot, supershot or ensemble member) is cut along x into `cps` slabs
// of whole columns, one CTA a slab, one CTA an SM.  A CTA keeps, for its R
// rows (x) and all depths, the two fields of a propagation with a 6-row halo
// on each side, 1/vt, and in the backward sweep the second propagation's
// fields and the image: HBM sees only the recorded samples, the boundary
// strips and the source values.
//
// A step: sources are added to the current fields (and their halo copies),
// one CTA barrier, then the compute warps march over the rows with the
// streaming kernels' register queue and arithmetic (the same operations in
// the same order: the same bits), writing the next field over the previous
// one in shared memory, while helper warps record receivers, save or
// prefetch strips and source values and collect the neighbours' edge rows;
// one CTA barrier ends the step.
//
// Lanes: an item is (row chunk, group of 4 depths); items are numbered chunk
// by chunk and a warp takes 30 of them plus one on each side, whose u2 the
// edge items need (z neighbours come by shuffle; an item at a chunk's first
// or last group needs no neighbour).  Partly filled depth slices, which cost
// the streaming kernels up to a quarter of their lanes, do not occur.
//
// Slabs of a few rows (one supershot over all SMs) leave that march a warp or
// two a scheduler and a chain of ten loads and L + 2 rows of u2 for L rows of
// output: 2450 (FAST) and 4500 (REF) cycles a step for a row a chunk.  The
// two-pass form (WIDE) has an item per u2 row and depth group, then, after a
// barrier of the compute warps, one per output row and group, u2 going
// through shared memory: no row is formed twice and nothing is serial, for 13
// loads a u2 item instead of 3 to 7.  (More warps than 16, or a barrier before
// the neighbours' rows are polled, made a step slower: 1 shot of 533 x 193
// REF 2.5 us with 512 threads, 3.1 with 768, 3.5 with 1024.)
//
// Edge rows travel through L2 as 8-byte {value, step tag} pairs, each one
// 64-bit access, written by the lanes that compute them and polled by the
// neighbour's helpers: no fence, no flag and no grid barrier.  Two buffers alternate: a CTA writes
// step n's rows only after it has received its neighbours' rows of step n-1,
// which they computed after receiving step n-2's.  Slabs of fewer than 6 rows
// (one shot of a small grid on all SMs) need rows of slabs further away: the
// buffer then has a place for every row, read by whoever is within 6 of it;
// who reads a CTA's rows is again who it reads.  Every CTA of the grid is
// resident (cooperative launch), every wait is bounded: on timeout the CTA
// raises the launch's flag, which the others' waits look at, and the
// caller's, which stays up until the host has seen it; it makes its results
// NaN, so that they cannot pass for a sweep's, and leaves.
#pragma once
#include <type_traits>
#include "kernels.cuh"
#include "stream.cuh"

namespace swfwi {

struct ResidentArgs {
  int nx, nz, pitch;         // padded grid, floats between global rows
  long long fstride;         // floats between slots' global fields
  int cps;                   // CTAs (slabs) per slot
  int nslots;                // grid = nslots * cps
  int nt;                    // time steps of the records (strides below)
  int steps;                 // steps to run
  int bx0, bsize;
  int chunks;                // row chunks a slab is split into
  int helpers;               // helper warps (the last ones of the CTA)
  int rmax;                  // rows of the largest slab
  int zp;                    // floats per shared row
  int ngroups, ogroups;      // depth groups per row: all, and those that hold outputs
  unsigned omagic;           // the same for ogroups and indices below 6 * ogroups
  unsigned gmagic;           // 2^20 / ngroups + 1: id / ngroups = id * gmagic >> 20 for id * ngroups < 2^20
  const float *rcp;          // 1/vt origin, pitched
  long long vel_stride;      // floats between slots' reciprocals (0: shared)
  const float2 *coef_x;
  const float *damp_x, *damp_z;
  int ramp;
  float *p0, *p1;            // global fields (origins): forward writes the final pair, backward reads it
  int store_state;           // forward: write the final pair
  PointSet src, rec;         // positions x*pitch + z
  const float *vals;         // source values: vals + it*it_stride + slot*slot_stride + i*i_stride
  long long it_stride, slot_stride;
  int i_stride;
  float *dcal;               // forward: records [slot][nt][ngrec] (null: none)
  const float *vsrc;         // backward: receiver sources, same layout
  int ngrec;
  float *strips;             // [slot][nt][bsize] (forward: written if not null; backward: read)
  float *image;              // backward: origin of the slots' images, updated in place
  float dt;
  int cap_src, cap_rec, cap_stage;   // list capacities (entries)
  unsigned nzs_magic;        // 2^32 / nzs + 1: u / nzs = high word of u * nzs_magic, nzs = depths of a side strip
  int thin;                  // slabs of fewer than 6 rows (two-pass form only): exchange buffer by row, not by slab
  uint4 *halo;               // zeroed before the launch
  int *quit;                 // this launch's flag: a wait gave up (zeroed before the launch)
  int *err;                  // the caller's
  long long patience;        // cycles a wait may take; 0: one unsuccessful poll
};

constexpr int kResidentThreads = 512;
constexpr int kResidentChunks = 64;   // most row chunks of a slab

// Shared memory of one CTA, in floats: the fields [2 * NF][rmax+12][zp] (S
// current/previous, then G), 1/vt [rmax][zp], the image [rmax][zp]
// (backward), the depths' sponge coefficients [2][zp], the point lists, the
// prefetched strips, the chunk starts and the slab's numbers.
struct ResidentSlab {
  int slot, R, xa;                          // own rows xa .. xa+R-1; shared row r is absolute row xa-6+r
  int nsrc, nrec;
  int nstrip, nbot, bot0, nlft, lft0, rgt0;   // strip cells in reach, see strip_cell
  int band;                                 // backward: a source in reach is a strip cell
  int give_up, drawn;                       // a wait gave up; receive batches drawn
};
struct ResidentLayout {
  int v, im, cf, src, rec, stage, cs, slab, args, u2, total;   // u2: the two-pass form's, [NF][rmax+2][zp]
  __host__ __device__ ResidentLayout(bool back, int rmax, int zp, int cap_src, int cap_rec, int cap_stage) {
    v = (back ? 4 : 2) * (rmax + 12) * zp;
    im = v + rmax * zp;
    cf = im + (back ? rmax * zp : 0);
    src = cf + 2 * zp;             // offset, index, value, image: cap_src each
    rec = src + 4 * cap_src;       // offset, index, value: cap_rec each
    stage = rec + 3 * cap_rec;
    cs = stage + cap_stage;
    slab = cs + kResidentChunks + 1;
    args = (slab + (int)(sizeof(ResidentSlab) / 4) + 3) / 4 * 4;   // a copy of the launch arguments
    u2 = (args + (int)((sizeof(ResidentArgs) + 3) / 4) + 3) / 4 * 4;
    total = u2;
  }
};
inline size_t resident_smem(bool backward, bool wide, int rmax, int zp, int cap_src, int cap_rec, int cap_stage) {
  return 4 * ((size_t)ResidentLayout(backward, rmax, zp, cap_src, cap_rec, cap_stage).total +
              (wide ? (backward ? 2 : 1) * (rmax + 2) * zp : 0));
}
// uint4 elements of the exchange buffer: [slot][slab][propagation][parity]
// [side][6][ogroups][2], or (thin) [slot][row][propagation][parity][ogroups][2]
inline size_t resident_halo(int nslots, int cps, int rows, bool thin, int nfields, int ogroups) {
  return (size_t)nslots * (thin ? rows : 12 * cps) * nfields * 2 * ogroups * 2;
}

namespace resident_detail {
using namespace stream_detail;

// Two pairs a 16-byte access.  Each pair is one 64-bit element of it: the
// memory model makes an element of a vector access one scalar access, so a
// value and its tag cannot be seen apart (as four 32-bit elements they could).
__device__ __forceinline__ unsigned long long pair_of(float v, uint32_t tag) {
  return (unsigned long long)tag << 32 | __float_as_uint(v);
}
__device__ __forceinline__ void put_pair2(uint4 *dst, float a, float b, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(dst), "l"(pair_of(a, tag)), "l"(pair_of(b, tag))
               : "memory");
}
__device__ __forceinline__ uint4 get_pair2(const uint4 *src) {
  unsigned long long a, b;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(src) : "memory");
  return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
}
__device__ __forceinline__ void cp4(uint32_t dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// rows of slab c of a slot: [first, first + n)
__host__ __device__ __forceinline__ int slab_first(int rows, int cps, int c) { return (int)((long long)rows * c / cps); }

// Imaging weight of step `it` (the reference's ramp, fwiframework.cpp:170).
__device__ __forceinline__ float image_scale(float dt, int it) {
  const float t = dt * (float)it;
  return (double)t > 0.4 ? 1.0f : (float)(((double)t - 0.3) / 0.1);
}

// Boundary strip cell e of a slab (its rows in reach): 6 below the
// model for the rows [bx0-6, nx-bx0+6), then the depths [6, nz-bx0) of the 6
// rows left and of the 6 rows right of the model.  g: its index in a step's
// strip, o: its shared offset.  Each of the three runs is contiguous in g.
__device__ __forceinline__ void strip_cell(const ResidentArgs &a, const ResidentSlab &b, int e, int &g, int &o) {
  const int w = 6, b0 = a.bx0, nzs = a.nz - 6 - b0;
  if (e < b.nbot * w) {
    const int k = e / w, iz = e - k * w, x = b.bot0 + k;
    g = (b.bot0 - (b0 - w)) * w + e;
    o = (x - (b.xa - 6)) * a.zp + a.nz - b0 + iz;
  } else {
    const int u = e - b.nbot * w, k = nzs > 1 ? (int)__umulhi((unsigned)u, a.nzs_magic) : u, iz = u - k * nzs;
    const bool left = k < b.nlft;
    const int x = left ? b.lft0 + k : b.rgt0 + k - b.nlft;
    const int col = left ? x - (b0 - w) : x - (a.nx - b0) + w;
    g = w * (a.nx - 2 * (b0 - w)) + col * nzs + iz;
    o = (x - (b.xa - 6)) * a.zp + 6 + iz;
  }
}

// The helper warps' part of a step besides the exchange: records and strips
// of the current field and the next step's source values (forward), the
// source values of this step and the strips and receiver sources of the
// next (backward).  Not inlined: the march needs the registers.
template <bool BACK>
__device__ __noinline__ void helper_step(const ResidentArgs &a, float *F, int cur, int n, int ht, int hn) {
  const ResidentLayout l(BACK, a.rmax, a.zp, a.cap_src, a.cap_rec, a.cap_stage);
  const ResidentSlab &b = *reinterpret_cast<const ResidentSlab *>(F + l.slab);
  const int it = BACK ? a.nt - 1 - n : n;
  const int *src_idx = reinterpret_cast<const int *>(F + l.src) + a.cap_src;
  float *src_val = F + l.src + 2 * a.cap_src;
  const int *rec_off = reinterpret_cast<const int *>(F + l.rec), *rec_idx = rec_off + a.cap_rec;
  const float *vals = a.vals + (long long)b.slot * a.slot_stride;
  const float *A = F + cur * (a.rmax + 12) * a.zp;
  if constexpr (!BACK) {
    if (a.dcal) {
      float *d = a.dcal + ((long long)b.slot * a.nt + it) * a.ngrec;
      for (int k = ht; k < b.nrec; k += hn) d[rec_idx[k]] = A[rec_off[k]];
    }
    if (it + 1 < a.nt)
      for (int k = ht; k < b.nsrc; k += hn)
        src_val[k] = vals[(long long)(it + 1) * a.it_stride + (long long)src_idx[k] * a.i_stride];
    if (b.nstrip) {
      float *d = a.strips + ((long long)b.slot * a.nt + it) * a.bsize;
      for (int e = ht; e < b.nstrip; e += hn) {
        int g, o;
        strip_cell(a, b, e, g, o);
        __stcs(d + g, A[o]);
      }
    }
  } else {
    for (int k = ht; k < b.nsrc; k += hn)
      cp4(smem_u32(src_val + k), vals + (long long)it * a.it_stride + (long long)src_idx[k] * a.i_stride);
    if (it > 0) {
      float *rec_val = F + l.rec + 2 * a.cap_rec;
      const float *v = a.vsrc + ((long long)b.slot * a.nt + it - 1) * a.ngrec;
      for (int k = ht; k < b.nrec; k += hn) cp4(smem_u32(rec_val + k), v + rec_idx[k]);
      const float *s = a.strips + ((long long)b.slot * a.nt + it - 1) * a.bsize;
      const uint32_t stage = smem_u32(F + l.stage);
      for (int e = ht; e < b.nstrip; e += hn) {
        int g, o;
        strip_cell(a, b, e, g, o);
        cp4(stage + 4 * e, s + g);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
}

// True where a strip has a cell: the 6 rows and depths around the model.
__device__ __forceinline__ bool in_strips(const ResidentArgs &a, int x, int z) {
  const int b0 = a.bx0;
  if (x < b0 - 6 || x >= a.nx - b0 + 6 || z < 6 || z >= a.nz - b0 + 6) return false;
  return z >= a.nz - b0 || x < b0 || x >= a.nx - b0;
}

// The points of the current fields before a step's march: sources in
// (forward); the last step's sources out of the rebuilt field, its image at
// them, the strips and the receiver sources in (backward).  A source that
// lies in the strips is imaged, then overwritten by them.
template <bool BACK>
__device__ __noinline__ void point_step(const ResidentArgs &a, float *F, int cur, int n) {
  const ResidentLayout l(BACK, a.rmax, a.zp, a.cap_src, a.cap_rec, a.cap_stage);
  const ResidentSlab &b = *reinterpret_cast<const ResidentSlab *>(F + l.slab);
  const int tid = threadIdx.x, nthreads = blockDim.x, field = (a.rmax + 12) * a.zp;
  const int *src_off = reinterpret_cast<const int *>(F + l.src);
  const float *src_val = F + l.src + 2 * a.cap_src;
  if constexpr (!BACK) {
    for (int k = tid; k < b.nsrc; k += nthreads) {
      float *s = F + cur * field + src_off[k];
      *s = __fadd_rn(*s, src_val[k]);
    }
  } else {
    if (n > 0) {
      const float scale = image_scale(a.dt, a.nt - n);   // of the step before
      float *src_img = F + l.src + 3 * a.cap_src;
      for (int k = tid; k < b.nsrc; k += nthreads) {
        float *s = F + cur * field + src_off[k];
        const float v = __fsub_rn(*s, src_val[k]);
        *s = v;
        src_img[k] = __fsub_rn(src_img[k], __fmul_rn(__fmul_rn(v, F[(2 + (cur ^ 1)) * field + src_off[k]]), scale));
      }
    }
    if (b.band) __syncthreads();
    for (int e = tid; e < b.nstrip; e += nthreads) {
      int g, o;
      strip_cell(a, b, e, g, o);
      F[cur * field + o] = F[l.stage + e];
    }
    const int *rec_off = reinterpret_cast<const int *>(F + l.rec);
    const float *rec_val = F + l.rec + 2 * a.cap_rec;
    for (int k = tid; k < b.nrec; k += nthreads) {
      float *g = F + (2 + cur) * field + rec_off[k];
      *g = __fadd_rn(*g, rec_val[k]);
    }
  }
}

// The neighbours' edge rows of the fields step n forms: batches of kRecv
// groups a lane, taken by whichever warp is free (the helpers at once, the
// compute warps as they finish).
constexpr int kRecv = 2;
template <bool BACK, bool WIDE>
__device__ __noinline__ void receive_step(const ResidentArgs &a, float *F, int cur, int n) {
  constexpr int NF = BACK ? 2 : 1;
  const ResidentLayout l(BACK, a.rmax, a.zp, a.cap_src, a.cap_rec, a.cap_stage);
  ResidentSlab &b = *reinterpret_cast<ResidentSlab *>(F + l.slab);
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, field = (a.rmax + 12) * a.zp;
  const bool has_l = b.xa > 6, has_r = b.xa + b.R < a.nx - 6;
  const int nper = 6 * a.ogroups, nside = (has_l ? 1 : 0) + (has_r ? 1 : 0);   // groups a side, sides
  const int ntotal = NF * nside * nper, nbatch = (ntotal + 32 * kRecv - 1) / (32 * kRecv);
  const size_t side = (size_t)nper * 2;
  const uint32_t tag = (uint32_t)(n + 1);
  for (;;) {
    int k = 0;
    if (lane == 0) k = atomicAdd(&b.drawn, 1);
    k = __shfl_sync(0xffffffffu, k, 0) - n * (nbatch + nwarps);   // every warp draws one past the end a step
    if (k >= nbatch) break;
    const uint4 *from[kRecv];
    float *to[kRecv];
    unsigned todo = 0;
#pragma unroll
    for (int e = 0; e < kRecv; e++) {
      const int u = (k * kRecv + e) * 32 + lane;
      from[e] = nullptr;
      to[e] = nullptr;
      if (u < ntotal) {
        const int f = BACK && u >= nper * nside ? 1 : 0, v = u - f * nper * nside;
        const int sd = v >= nper ? 1 : 0, gidx = v - sd * nper;
        const bool left = has_l && sd == 0;   // rows before the slab: the left neighbour's last rows
        const int rr = (int)(((unsigned)gidx * a.omagic) >> 20), grp = gidx - rr * a.ogroups;
        if (WIDE && a.thin) {
          const int row = (left ? b.xa - 12 : b.xa + b.R - 6) + rr;   // row 0: absolute row 6
          if (row < 0 || row >= a.nx - 12) continue;
          from[e] = a.halo + (((size_t)b.slot * (a.nx - 12) + row) * NF + f) * 4 * a.ogroups +
                    ((size_t)(n & 1) * a.ogroups + grp) * 2;
        } else {
          const int nb = left ? (int)blockIdx.x - 1 : (int)blockIdx.x + 1;
          from[e] = a.halo + ((size_t)nb * NF + f) * 4 * side + ((size_t)(n & 1) * 2 + (left ? 1 : 0)) * side +
                    (size_t)gidx * 2;
        }
        to[e] = F + (2 * f + (cur ^ 1)) * field + (left ? rr : b.R + 6 + rr) * a.zp + 4 + 4 * grp;
        todo |= 1u << e;
      }
    }
    long long t0 = 0;
    auto late = [&](int spin) {   // bounded: a.patience cycles, or until another CTA gave up
      if (a.patience > 0 && (spin & 255) != 255) return false;
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (now - t0 < a.patience && !*(volatile int *)a.quit) return false;
      *(volatile int *)a.quit = 1;
      *(volatile int *)a.err = 1;
      b.give_up = 1;
      return true;
    };
    for (int spin = 0; todo; spin++) {
      uint4 x[kRecv], y[kRecv];
#pragma unroll
      for (int e = 0; e < kRecv; e++)
        if (todo >> e & 1) {
          x[e] = get_pair2(from[e]);
          y[e] = get_pair2(from[e] + 1);
        }
#pragma unroll
      for (int e = 0; e < kRecv; e++)
        if ((todo >> e & 1) && x[e].y == tag && x[e].w == tag && y[e].y == tag && y[e].w == tag) {
          st4(to[e], make_float4(__uint_as_float(x[e].x), __uint_as_float(x[e].z), __uint_as_float(y[e].x),
                                 __uint_as_float(y[e].z)));
          todo &= ~(1u << e);
        }
      if (todo && late(spin)) break;
    }
    __syncwarp();
  }
}

// A wait gave up in step n: what the CTA would still have written is NaN, the
// records from the next step on and the final pair, or the image.
template <bool BACK>
__device__ __noinline__ void spoil_results(const ResidentArgs &a, float *F, int n) {
  const ResidentLayout l(BACK, a.rmax, a.zp, a.cap_src, a.cap_rec, a.cap_stage);
  const ResidentSlab &b = *reinterpret_cast<const ResidentSlab *>(F + l.slab);
  const int tid = threadIdx.x, nthreads = blockDim.x;
  const float nan = __int_as_float(0x7fffffff);
  if (!BACK && a.dcal) {
    const int *rec_idx = reinterpret_cast<const int *>(F + l.rec) + a.cap_rec;
    for (int it = n + 1; it < a.steps; it++)
      for (int k = tid; k < b.nrec; k += nthreads)
        a.dcal[((long long)b.slot * a.nt + it) * a.ngrec + rec_idx[k]] = nan;
  }
  if (BACK || a.store_state)
    for (int i = tid; i < b.R * a.zp; i += nthreads) {
      const int r = i / a.zp, z = i - r * a.zp;
      if (z < 6 || z >= a.nz - 6) continue;
      const long long p = (long long)b.slot * a.fstride + (long long)(b.xa + r) * a.pitch + z;
      if constexpr (BACK) a.image[p] = nan;
      else a.p0[p] = a.p1[p] = nan;
    }
}

// The compute warps' part of a step in two passes (ct of cn threads).
template <int ARITH, bool BACK>
__device__ __forceinline__ void march_wide(const ResidentArgs &a, const ResidentLayout &l, float *F, int slot, int xa,
                                           int R, int cur, int n, int ct, int cn) {
  constexpr int NF = BACK ? 2 : 1;
  const int ZP = a.zp, nz = a.nz, field = (a.rmax + 12) * ZP, G = a.ngroups, ufield = (a.rmax + 2) * ZP;
  float *U = F + l.u2;
  // u2 row ur (of propagation f) belongs to shared row ur + 5
  for (int id = ct; id < NF * (R + 2) * G; id += cn) {
    const int rr = (int)(((unsigned)id * a.gmagic) >> 20), grp = id - rr * G;
    const int f = BACK && rr >= R + 2 ? 1 : 0, ur = rr - f * (R + 2), zg = 4 + 4 * grp;
    const float *A = F + (2 * f + cur) * field + ur * ZP + zg;   // five rows before
    const float *C = A + 5 * ZP;
    float4 xm[6], xp[6];
#pragma unroll
    for (int k = 1; k <= 5; k++) {
      xm[k] = ld4(A + (5 - k) * ZP);
      xp[k] = ld4(A + (5 + k) * ZP);
    }
    const float4 v1 = ld4(C - 4), v2 = ld4(C), v3 = ld4(C + 4);
    float zn[20];
    zn[0] = zn[1] = zn[2] = zn[17] = zn[18] = zn[19] = 0.f;
    zn[3] = C[grp > 0 ? -5 : -4];   // the first depth of the first group is no output's neighbour
    zn[16] = C[8];
    zn[4] = v1.x; zn[5] = v1.y; zn[6] = v1.z; zn[7] = v1.w;
    zn[8] = v2.x; zn[9] = v2.y; zn[10] = v2.z; zn[11] = v2.w;
    zn[12] = v3.x; zn[13] = v3.y; zn[14] = v3.z; zn[15] = v3.w;
    float4 u;
    if constexpr (ARITH == ARITH_FAST) {
      const float2 lo = lap_pair_fast<0>(zn, xm, xp), hi = lap_pair_fast<1>(zn, xm, xp);
      u = make_float4(lo.x, lo.y, hi.x, hi.y);
    } else {
      float uu[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float m[6], q[6];
        m[0] = q[0] = 0.f;
#pragma unroll
        for (int k = 1; k <= 5; k++) {
          m[k] = get(xm[k], i);
          q[k] = get(xp[k], i);
        }
        uu[i] = lap_pt<ARITH>(zn, i, m, q);
      }
      u = make_float4(uu[0], uu[1], uu[2], uu[3]);
    }
    st4(U + f * ufield + ur * ZP + zg, u);
  }
  asm volatile("bar.sync 1, %0;" ::"r"(cn) : "memory");

  const bool has_l = xa > 6, has_r = xa + R < a.nx - 6;
  const float scale = BACK ? image_scale(a.dt, a.nt - 1 - n) : 0.0f;
  const uint32_t tag = (uint32_t)(n + 1);
  const unsigned span = (unsigned)max(a.nx - 2 * a.ramp, 0);
  const int O = a.ogroups;
  for (int id = ct; id < NF * R * O; id += cn) {
    const int rr = (int)(((unsigned)id * a.omagic) >> 20), grp = id - rr * O;
    const int f = BACK && rr >= R ? 1 : 0, j = rr - f * R, zg = 4 + 4 * grp;
    const bool damped = !BACK || f == 1;
    const int at = (j + 6) * ZP + zg;
    const float *u = U + f * ufield + (j + 1) * ZP + zg;
    const float4 um = ld4(u - ZP), uc = ld4(u), up = ld4(u + ZP);
    const float ucl = u[-1], ucr = u[4];
    float *B = F + (2 * f + (cur ^ 1)) * field + at;
    const float4 c4 = ld4(F + (2 * f + cur) * field + at), p4 = ld4(B), r4 = ld4(F + l.v + at - 6 * ZP);
    const bool ramp_row = damped && (unsigned)(j + xa - a.ramp) >= span;
    float4 o;
    if constexpr (ARITH == ARITH_FAST) {
      float2 cf0 = make_float2(2.f, 2.f), cf1 = cf0, pc0 = make_float2(-1.f, -1.f), pc1 = pc0;
      if (damped) {
        const float4 c = ld4(F + l.cf + zg), p = ld4(F + l.cf + ZP + zg);
        cf0 = lo2(c);
        cf1 = hi2(c);
        pc0 = lo2(p);
        pc1 = hi2(p);
      }
      if (ramp_row) {
        const float2 cx = a.coef_x[xa + j];
        if (pc0.x == -1.f) { cf0.x = cx.x; pc0.x = cx.y; }
        if (pc0.y == -1.f) { cf0.y = cx.x; pc0.y = cx.y; }
        if (pc1.x == -1.f) { cf1.x = cx.x; pc1.x = cx.y; }
        if (pc1.y == -1.f) { cf1.y = cx.x; pc1.y = cx.y; }
      }
      const float2 o0 = update_pair_coef(lo2(c4), lo2(p4), lo2(r4), lo2(uc),
                                         make_float2(__fadd_rn(ucl, uc.y), __fadd_rn(uc.x, uc.z)), lo2(um), lo2(up),
                                         cf0, pc0);
      const float2 o1 = update_pair_coef(hi2(c4), hi2(p4), hi2(r4), hi2(uc),
                                         make_float2(__fadd_rn(uc.y, uc.w), __fadd_rn(uc.z, ucr)), hi2(um), hi2(up),
                                         cf1, pc1);
      o = make_float4(o0.x, o0.y, o1.x, o1.y);
    } else {
      const float dxr = ramp_row ? a.damp_x[xa + j] : 0.f;
      float4 dz = make_float4(-1.f, -1.f, -1.f, -1.f);
      if (damped) dz = ld4(F + l.cf + zg);
      float oo[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float delta = 0.f;
        const float dist = get(dz, i) >= 0.f ? get(dz, i) : dxr;
        if (damped) delta = __fmul_rn(__fmul_rn(0.05f, dist), dist);
        oo[i] = update_pt<ARITH>(get(c4, i), get(p4, i), get(r4, i), get(uc, i), i == 0 ? ucl : get(uc, i - 1),
                                 i == 3 ? ucr : get(uc, i + 1), get(um, i), get(up, i), delta);
      }
      o = make_float4(oo[0], oo[1], oo[2], oo[3]);
    }
    // border depths stay zero
    o.x = zg >= 6 && zg < nz - 6 ? o.x : 0.f;
    o.y = zg + 1 >= 6 && zg + 1 < nz - 6 ? o.y : 0.f;
    o.z = zg + 2 < nz - 6 ? o.z : 0.f;
    o.w = zg + 3 < nz - 6 ? o.w : 0.f;
    st4(B, o);
    if constexpr (BACK) {
      if (f == 0) {
        const float4 g4 = ld4(F + (2 + cur) * field + at);
        float *im = F + l.im + at - 6 * ZP;
        float4 m = ld4(im);
        m.x = __fsub_rn(m.x, __fmul_rn(__fmul_rn(o.x, g4.x), scale));
        m.y = __fsub_rn(m.y, __fmul_rn(__fmul_rn(o.y, g4.y), scale));
        m.z = __fsub_rn(m.z, __fmul_rn(__fmul_rn(o.z, g4.z), scale));
        m.w = __fsub_rn(m.w, __fmul_rn(__fmul_rn(o.w, g4.w), scale));
        st4(im, m);
      }
    }
    if (a.thin) {
      uint4 *d = a.halo + ((((unsigned)(slot * (a.nx - 12) + xa - 6 + j) * NF + f) * 2 + (n & 1)) * O + grp) * 2;
      put_pair2(d, o.x, o.y, tag);
      put_pair2(d + 1, o.z, o.w, tag);
    } else {
      uint4 *h = a.halo + (((blockIdx.x * NF + f) * 4 + (n & 1) * 2) * (unsigned)(6 * O) + grp) * 2;
      if (j < 6 && has_l) {
        uint4 *d = h + (unsigned)(j * O * 2);
        put_pair2(d, o.x, o.y, tag);
        put_pair2(d + 1, o.z, o.w, tag);
      }
      if (j >= R - 6 && has_r) {
        uint4 *d = h + (unsigned)((j - R + 12) * O * 2);
        put_pair2(d, o.x, o.y, tag);
        put_pair2(d + 1, o.z, o.w, tag);
      }
    }
  }
}

}  // namespace resident_detail

template <int ARITH, bool BACK, bool WIDE>
__global__ void __launch_bounds__(kResidentThreads, 1) fd_resident(const __grid_constant__ ResidentArgs a) {
  using namespace resident_detail;
  constexpr int NF = BACK ? 2 : 1;   // propagations
  extern __shared__ __align__(16) float F[];
  const ResidentLayout l(BACK, a.rmax, a.zp, a.cap_src, a.cap_rec, a.cap_stage);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthreads = blockDim.x, cwarps = (nthreads >> 5) - a.helpers;
  const int ZP = a.zp, nz = a.nz, field = (a.rmax + 12) * ZP;
  ResidentSlab &sb = *reinterpret_cast<ResidentSlab *>(F + l.slab);
  // what the calls below read the arguments from
  ResidentArgs &sa = *reinterpret_cast<ResidentArgs *>(F + l.args);
  int *cs = reinterpret_cast<int *>(F + l.cs);

  // ---- set up
  {
    const int slot = blockIdx.x / a.cps, slab = blockIdx.x - slot * a.cps;
    const int s0 = slab_first(a.nx - 12, a.cps, slab), R = slab_first(a.nx - 12, a.cps, slab + 1) - s0, xa = 6 + s0;
    if (tid == 0) {
      sa = a;
      // strip rows in reach: going back the halo rows too, forward the own
      // rows and, of a sponge of fewer than 6 points, the rows outside the
      // computing zone (their cells stay zero)
      const int w = 6, b0 = a.bx0, ra = BACK || slab == 0 ? xa - 6 : xa,
                rb = BACK || slab == a.cps - 1 ? xa + R + 6 : xa + R;
      sb.slot = slot;
      sb.R = R;
      sb.xa = xa;
      sb.nsrc = sb.nrec = 0;
      sb.bot0 = max(ra, b0 - w);
      sb.nbot = max(min(rb, a.nx - b0 + w) - sb.bot0, 0);
      sb.lft0 = max(ra, b0 - w);
      sb.nlft = max(min(rb, b0) - sb.lft0, 0);
      sb.rgt0 = max(ra, a.nx - b0);
      const int nrgt = max(min(rb, a.nx - b0 + w) - sb.rgt0, 0);
      sb.nstrip = a.strips ? sb.nbot * w + (sb.nlft + nrgt) * max(nz - 6 - b0, 0) : 0;
      sb.band = 0;
      sb.give_up = 0;
      sb.drawn = 0;
    }
    for (int i = tid; i < NF * 2 * field; i += nthreads) F[i] = 0.0f;
    for (int i = tid; i <= a.chunks; i += nthreads) cs[i] = slab_first(R, a.chunks, i);
    for (int z = tid; z < ZP; z += nthreads) {
      const float d = z < nz ? a.damp_z[z] : -1.f;
      if constexpr (ARITH == ARITH_FAST) {
        const float2 c = fast_damp_coef(d >= 0.f ? d : 0.0f);
        F[l.cf + z] = c.x;
        F[l.cf + ZP + z] = c.y;
      } else {
        F[l.cf + z] = d;
      }
    }
    const float *rcp = a.rcp + (long long)slot * a.vel_stride;
    for (int i = tid; i < R * ZP; i += nthreads) {
      const int r = i / ZP, z = i - r * ZP;
      const bool in = z >= 6 && z < nz - 6;
      F[l.v + i] = in ? rcp[(long long)(xa + r) * a.pitch + z] : 1.0f;
      if constexpr (BACK)
        F[l.im + i] = in ? a.image[(long long)slot * a.fstride + (long long)(xa + r) * a.pitch + z] : 0.0f;
    }
    __syncthreads();
    if constexpr (BACK) {
      // current source field: p0 (the field the last step advanced from);
      // previous: p1 (the newest)
      const float *g0 = a.p0 + (long long)slot * a.fstride, *g1 = a.p1 + (long long)slot * a.fstride;
      for (int i = tid; i < (R + 12) * ZP; i += nthreads) {
        const int r = i / ZP, z = i - r * ZP;
        if (z < nz) {
          F[i] = g0[(long long)(xa - 6 + r) * a.pitch + z];
          F[field + i] = g1[(long long)(xa - 6 + r) * a.pitch + z];
        }
      }
    }
    // the points of the slab (receivers of the forward sweep: own rows; the
    // others also in the halo rows), in any order: positions are distinct
    int *src_off = reinterpret_cast<int *>(F + l.src), *src_idx = src_off + a.cap_src;
    int *rec_off = reinterpret_cast<int *>(F + l.rec), *rec_idx = rec_off + a.cap_rec;
    const int sshot = a.src.slot_shot ? a.src.slot_shot[slot] : slot;
    for (int i = tid; i < a.src.per_shot; i += nthreads) {
      const int p = a.src.pos[(long long)sshot * a.src.per_shot + i];
      if (p < 0) continue;
      const int x = p / a.pitch, z = p - x * a.pitch, r = x - (xa - 6);
      if (r < 0 || r >= R + 12) continue;
      if (BACK && in_strips(a, x, z)) sb.band = 1;
      const int k = atomicAdd(&sb.nsrc, 1);
      if (k < a.cap_src) {
        src_off[k] = r * ZP + z;
        src_idx[k] = i;
      }
    }
    if (BACK || a.dcal) {
      const int rshot = a.rec.slot_shot ? a.rec.slot_shot[slot] : slot;
      for (int i = tid; i < a.rec.per_shot; i += nthreads) {
        const int p = a.rec.pos[(long long)rshot * a.rec.per_shot + i];
        if (p < 0) continue;
        const int x = p / a.pitch, z = p - x * a.pitch, r = x - (xa - 6);
        if (BACK ? (r < 0 || r >= R + 12) : (r < 6 || r >= R + 6)) continue;
        const int k = atomicAdd(&sb.nrec, 1);
        if (k < a.cap_rec) {
          rec_off[k] = r * ZP + z;
          rec_idx[k] = i;
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      sb.nsrc = min(sb.nsrc, a.cap_src);
      sb.nrec = min(sb.nrec, a.cap_rec);
    }
    __syncthreads();
    const float *vals = a.vals + (long long)slot * a.slot_stride;
    const int it0 = BACK ? a.nt - 1 : 0;
    for (int k = tid; k < sb.nsrc; k += nthreads) {
      F[l.src + 2 * a.cap_src + k] =
          BACK ? 0.0f : vals[(long long)it0 * a.it_stride + (long long)src_idx[k] * a.i_stride];
      if constexpr (BACK) {
        const int r = src_off[k] / ZP;
        F[l.src + 3 * a.cap_src + k] = r >= 6 && r < R + 6 ? F[l.im + src_off[k] - 6 * ZP] : 0.0f;
      }
    }
    if constexpr (BACK) {
      const float *vsrc = a.vsrc + ((long long)slot * a.nt + it0) * a.ngrec;
      for (int k = tid; k < sb.nrec; k += nthreads) F[l.rec + 2 * a.cap_rec + k] = vsrc[rec_idx[k]];
      const float *strips = a.strips + ((long long)slot * a.nt + it0) * a.bsize;
      for (int e = tid; e < sb.nstrip; e += nthreads) {
        int g, o;
        strip_cell(sa, sb, e, g, o);
        F[l.stage + e] = strips[g];
      }
    }
    __syncthreads();
  }
  const int R = sb.R, xa = sb.xa;
  const bool points = BACK || sb.nsrc > 0;

  const bool has_l = xa > 6, has_r = xa + R < a.nx - 6;

  // ---- the compute warps' items
  const int K = a.chunks, G = a.ngroups, items = K * G;
  const int wtasks = (items + 29) / 30;
  const int L = (R + K - 1) / K;   // rows of the longest chunk

  int cur = 0;                     // which of a propagation's two buffers is current
  for (int n = 0; n < a.steps; n++) {
    if (points) {
      point_step<BACK>(sa, F, cur, n);
      __syncthreads();
    }

    if (WIDE && warp < cwarps) {
      march_wide<ARITH, BACK>(sa, l, F, sb.slot, xa, R, cur, n, tid, 32 * cwarps);
    } else if (!WIDE && warp < cwarps) {
      const float scale = BACK ? image_scale(a.dt, a.nt - 1 - n) : 0.0f;
      const uint32_t tag = (uint32_t)(n + 1);
      for (int task = warp; task < NF * wtasks; task += cwarps) {
        const int f = BACK ? (task >= wtasks ? 1 : 0) : 0;   // 0: source field, 1: receiver field
        const bool damped = !BACK || f == 1;
        const int id = (task - f * wtasks) * 30 + lane - 1;
        const int idc = min(max(id, 0), items - 1);
        const int chunk = (int)(((unsigned)idc * a.gmagic) >> 20), grp = idc - chunk * G;
        const int c0 = cs[chunk], c1 = cs[chunk + 1];
        const int zg = 4 + 4 * grp;
        const bool outlane = lane >= 1 && lane <= 30 && id < items && grp < a.ogroups;
        bool zok[4];
#pragma unroll
        for (int i = 0; i < 4; i++) zok[i] = zg + i >= 6 && zg + i < nz - 6;
        const float *A = F + (2 * f + cur) * field + c0 * ZP + zg;
        float *B = F + (2 * f + (cur ^ 1)) * field + (c0 + 6) * ZP + zg;
        const float *rv = F + l.v + c0 * ZP + zg;
        const float *gc = F + (2 + cur) * field + (c0 + 6) * ZP + zg;   // receiver field at the outputs (BACK)
        float *im = F + l.im + c0 * ZP + zg;
        // this step's place for the first edge row's group in the exchange buffer
        const unsigned hl = ((blockIdx.x * NF + f) * 4 + (n & 1) * 2) * (unsigned)(12 * a.ogroups) + 2 * grp;

        // sponge, as in the streaming kernels: the bottom ramp per depth,
        // the row's coefficients on left/right ramp rows
        float dz[4] = {-1.f, -1.f, -1.f, -1.f};
        float2 coefz[2] = {make_float2(2.f, 2.f), make_float2(2.f, 2.f)};
        float2 pcz[2] = {make_float2(-1.f, -1.f), make_float2(-1.f, -1.f)};
        if (damped) {
          const float4 c = ld4(F + l.cf + zg);
          if constexpr (ARITH == ARITH_FAST) {
            const float4 p = ld4(F + l.cf + ZP + zg);
            coefz[0] = lo2(c);
            coefz[1] = hi2(c);
            pcz[0] = lo2(p);
            pcz[1] = hi2(p);
          } else {
            dz[0] = c.x; dz[1] = c.y; dz[2] = c.z; dz[3] = c.w;
          }
        }
        const int j_lo = a.ramp - xa - c0;   // output rows j < j_lo or >= j_lo + span: ramp rows
        const unsigned span = (unsigned)max(a.nx - 2 * a.ramp, 0);

        float4 q[11];   // own values of 11 rows; at march step i slot i % 11 takes row c0 + i
#pragma unroll
        for (int i = 0; i < 10; i++) q[i] = ld4(A + i * ZP);
        const float *An = A + 10 * ZP;   // the row to load
        const float *Ac = A + 5 * ZP;    // the row whose u2 is formed
        float4 um = make_float4(0.f, 0.f, 0.f, 0.f), uc = um;

        // march step i = i0 + U: load row c0+i, u2 of row c0+i-5, output row j = i - 12
        auto step = [&](auto uu, int j) {
          constexpr int U = decltype(uu)::value;
          q[U] = ld4(An);
          An += ZP;
#define SWFWI_Q(k) q[(U + 1 + (k)) % 11]
          const float4 v1 = ld4(Ac - 4), v3 = ld4(Ac + 4), v2 = SWFWI_Q(5);
          Ac += ZP;
          float zn[20];
          zn[0] = zn[1] = zn[2] = zn[17] = zn[18] = zn[19] = 0.f;
          zn[3] = __shfl_up_sync(0xffffffffu, v1.w, 1);
          zn[16] = __shfl_down_sync(0xffffffffu, v3.x, 1);
          zn[4] = v1.x; zn[5] = v1.y; zn[6] = v1.z; zn[7] = v1.w;
          zn[8] = v2.x; zn[9] = v2.y; zn[10] = v2.z; zn[11] = v2.w;
          zn[12] = v3.x; zn[13] = v3.y; zn[14] = v3.z; zn[15] = v3.w;
          float4 up;
          if constexpr (ARITH == ARITH_FAST) {
            const float a5[6] = {-4.0f * SWFWI_A0, SWFWI_A1, SWFWI_A2, SWFWI_A3, SWFWI_A4, SWFWI_A5};
            float2 acc[2];
#pragma unroll
            for (int pr = 0; pr < 2; pr++) {
              const int i = 2 * pr;
              acc[pr] = __fmul2_rn(make_float2(a5[0], a5[0]), pr == 0 ? lo2(v2) : hi2(v2));
#pragma unroll
              for (int kk = 1; kk <= 5; kk++) {
                float2 zs;
                if (kk & 1)   // unaligned depth pairs: two scalar adds
                  zs = make_float2(__fadd_rn(zn[8 + i - kk], zn[8 + i + kk]), __fadd_rn(zn[9 + i - kk], zn[9 + i + kk]));
                else
                  zs = __fadd2_rn(make_float2(zn[8 + i - kk], zn[9 + i - kk]), make_float2(zn[8 + i + kk], zn[9 + i + kk]));
                const float2 xs = pr == 0 ? __fadd2_rn(lo2(SWFWI_Q(5 - kk)), lo2(SWFWI_Q(5 + kk)))
                                          : __fadd2_rn(hi2(SWFWI_Q(5 - kk)), hi2(SWFWI_Q(5 + kk)));
                acc[pr] = __ffma2_rn(make_float2(a5[kk], a5[kk]), __fadd2_rn(zs, xs), acc[pr]);
              }
            }
            up = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
          } else {
            float uu4[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
              float xm[6], xp[6];
              xm[0] = xp[0] = 0.f;
#pragma unroll
              for (int d = 1; d <= 5; d++) {
                xm[d] = get(SWFWI_Q(5 - d), i);
                xp[d] = get(SWFWI_Q(5 + d), i);
              }
              uu4[i] = lap_pt<ARITH>(zn, i, xm, xp);
            }
            up = make_float4(uu4[0], uu4[1], uu4[2], uu4[3]);
          }
          if (j >= 0) {
            const float ucl = __shfl_up_sync(0xffffffffu, uc.w, 1);
            const float ucr = __shfl_down_sync(0xffffffffu, uc.x, 1);
            const float4 c4 = SWFWI_Q(4);
            const float4 p4 = ld4(B), r4 = ld4(rv);
            const bool ramp_row = __builtin_expect(damped && (unsigned)(j - j_lo) >= span, 0);
            float4 o;
            if constexpr (ARITH == ARITH_FAST) {
              float2 cf0 = coefz[0], cf1 = coefz[1], pc0 = pcz[0], pc1 = pcz[1];
              if (ramp_row) {
                const float2 cx = a.coef_x[min(xa + c0 + j, a.nx - 1)];
                if (pc0.x == -1.f) { cf0.x = cx.x; pc0.x = cx.y; }
                if (pc0.y == -1.f) { cf0.y = cx.x; pc0.y = cx.y; }
                if (pc1.x == -1.f) { cf1.x = cx.x; pc1.x = cx.y; }
                if (pc1.y == -1.f) { cf1.y = cx.x; pc1.y = cx.y; }
              }
              const float2 o0 = update_pair_coef(lo2(c4), lo2(p4), lo2(r4), lo2(uc),
                                                 make_float2(__fadd_rn(ucl, uc.y), __fadd_rn(uc.x, uc.z)), lo2(um),
                                                 lo2(up), cf0, pc0);
              const float2 o1 = update_pair_coef(hi2(c4), hi2(p4), hi2(r4), hi2(uc),
                                                 make_float2(__fadd_rn(uc.y, uc.w), __fadd_rn(uc.z, ucr)), hi2(um),
                                                 hi2(up), cf1, pc1);
              o = make_float4(o0.x, o0.y, o1.x, o1.y);
            } else {
              const float dxr = ramp_row ? a.damp_x[min(xa + c0 + j, a.nx - 1)] : 0.f;
              float oo[4];
#pragma unroll
              for (int i = 0; i < 4; i++) {
                float delta = 0.f;
                const float dist = dz[i] >= 0.f ? dz[i] : dxr;
                if (damped) delta = __fmul_rn(__fmul_rn(0.05f, dist), dist);
                const float uzm = i == 0 ? ucl : get(uc, i - 1);
                const float uzp = i == 3 ? ucr : get(uc, i + 1);
                oo[i] = update_pt<ARITH>(get(c4, i), get(p4, i), get(r4, i), get(uc, i), uzm, uzp, get(um, i),
                                         get(up, i), delta);
              }
              o = make_float4(oo[0], oo[1], oo[2], oo[3]);
            }
            if (outlane && c0 + j < c1) {
              // border depths stay zero
              o.x = zok[0] ? o.x : 0.f;
              o.y = zok[1] ? o.y : 0.f;
              o.z = zok[2] ? o.z : 0.f;
              o.w = zok[3] ? o.w : 0.f;
              st4(B, o);
              if constexpr (BACK) {
                if (f == 0) {
                  const float4 g4 = ld4(gc);
                  float4 m = ld4(im);
                  m.x = __fsub_rn(m.x, __fmul_rn(__fmul_rn(o.x, g4.x), scale));
                  m.y = __fsub_rn(m.y, __fmul_rn(__fmul_rn(o.y, g4.y), scale));
                  m.z = __fsub_rn(m.z, __fmul_rn(__fmul_rn(o.z, g4.z), scale));
                  m.w = __fsub_rn(m.w, __fmul_rn(__fmul_rn(o.w, g4.w), scale));
                  st4(im, m);
                }
              }
              const int row = c0 + j;
              if (row < 6 && has_l) {
                uint4 *d = a.halo + (hl + (unsigned)(row * a.ogroups * 2));
                put_pair2(d, o.x, o.y, tag);
                put_pair2(d + 1, o.z, o.w, tag);
              }
              if (row >= R - 6 && has_r) {
                uint4 *d = a.halo + (hl + (unsigned)((row - R + 12) * a.ogroups * 2));
                put_pair2(d, o.x, o.y, tag);
                put_pair2(d + 1, o.z, o.w, tag);
              }
            }
            B += ZP;
            rv += ZP;
            if constexpr (BACK) {
              gc += ZP;
              im += ZP;
            }
          }
#undef SWFWI_Q
          um = uc;
          uc = up;
        };
#define SWFWI_STEP(U)                                   \
  step(std::integral_constant<int, (U)>{}, j);          \
  if (++j >= L) break;
        for (int j = -2;;) {
          SWFWI_STEP(10) SWFWI_STEP(0) SWFWI_STEP(1) SWFWI_STEP(2) SWFWI_STEP(3) SWFWI_STEP(4)
          SWFWI_STEP(5) SWFWI_STEP(6) SWFWI_STEP(7) SWFWI_STEP(8) SWFWI_STEP(9)
        }
#undef SWFWI_STEP
      }
    } else {
      const int hn = 32 * a.helpers;
      helper_step<BACK>(sa, F, cur, n, tid - (nthreads - hn), hn);
    }
    if (n + 1 < a.steps && (has_l || has_r)) receive_step<BACK, WIDE>(sa, F, cur, n);
    if constexpr (BACK) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    cur ^= 1;
    if (sb.give_up) {   // uniform: written before the barrier, never cleared
      spoil_results<BACK>(sa, F, n);
      return;
    }
  }

  // ---- results
  const long long out = (long long)sb.slot * a.fstride;
  if constexpr (BACK) {
    // the last step's source points
    const float scale = image_scale(a.dt, a.nt - a.steps);
    const int *src_off = reinterpret_cast<const int *>(F + l.src);
    for (int k = tid; k < sb.nsrc; k += nthreads) {
      const int o = src_off[k], r = o / ZP;
      if (r < 6 || r >= R + 6) continue;
      const float v = __fsub_rn(F[cur * field + o], F[l.src + 2 * a.cap_src + k]);
      F[l.im + o - 6 * ZP] = __fsub_rn(F[l.src + 3 * a.cap_src + k],
                                       __fmul_rn(__fmul_rn(v, F[(2 + (cur ^ 1)) * field + o]), scale));
    }
    __syncthreads();
    for (int i = tid; i < R * ZP; i += nthreads) {
      const int r = i / ZP, z = i - r * ZP;
      if (z >= 6 && z < nz - 6) a.image[out + (long long)(xa + r) * a.pitch + z] = F[l.im + i];
    }
  } else if (a.store_state) {
    // p0: the field the last step advanced from, p1: the newest
    for (int i = tid; i < R * ZP; i += nthreads) {
      const int r = i / ZP, z = i - r * ZP;
      if (z >= 6 && z < nz - 6) {
        const long long p = out + (long long)(xa + r) * a.pitch + z;
        a.p0[p] = F[(cur ^ 1) * field + i + 6 * ZP];
        a.p1[p] = F[cur * field + i + 6 * ZP];
      }
    }
  }
}

}  // namespace swfwi
