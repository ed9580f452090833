// The LSRTM operator's time loops with the fields in shared memory: a whole
// sweep of a batch of shots in one cooperative launch, as the resident time
// loop of the FWI propagator (resident.cuh) runs its sweeps.  Included by
// lsrtm.cu, whose kernels define the scheme and which decides between the two
// (Prtm::resident).  The arithmetic and its order are theirs, point by point
// and so bit by bit, but for one sum of FAST Born modelling: the launched
// kernel contracts vv a + vv b to an FMA with one product unrounded, while
// here each vv times the field is rounded once, as the row is loaded.  The
// two differ by 1 to 2e-6 relative L2, equally far from 64 bits (1.65e-5).
//
// A shot is cut along x into `cps` slabs, one CTA each, with 2 halo rows a
// side.  The stencils are latency- and launch-bound as separate launches
// (each step two or three launches over fields that sit in L2: 33 us a step
// of Born modelling for 20 shots of 521 x 211, against about 1 us of
// arithmetic); here a step is one pass over shared memory and two CTA
// barriers, with the edge rows exchanged as {value, step} pairs.
//
// What k_prtm_aux does between the stencil steps is folded into the pass:
//  * the sponge of the new field is applied as it is stored and that of the
//    previous field as it is read (both fields of a pair are tapered once a
//    step); the smaller weight multiplies first, which is the reference's
//    order (ib ascending, z before x) because the weights grow with ib;
//  * Born's injection adds S mod to the previous field as it is read;
//  * imaging adds to the slab's image in shared memory;
//  * ring, source and receiver cells are touched before the pass, in the
//    halo rows too.
// The exact transpose's field b is always -W a of the step before (plus the
// injected data), so it is formed from the previous a as it is read; the
// grid's outer two cells, which its stencil masks, never reach the image.
#pragma once
#include "resident.cuh"

namespace swfwi {
namespace {

enum PrtmSweep { PRTM_BORN = 0, PRTM_SOURCE = 1, PRTM_MIGRATE = 2, PRTM_TRANSPOSE = 3 };

constexpr int kPrtmThreads = 512;
constexpr int kPrtmChunks = 64;

struct PrtmResident {
  PrtmGeo g;
  PrtmCoef c;
  int nslots, cps, rmax, zp, ngroups, ogroups, chunks, helpers;
  unsigned gmagic, nz_magic;
  int cap_rec, cap_ring;
  const float *vv, *mod, *wl;
  float *s0, *s1, *g0, *g1;    // fields [slot][fsz]: state read (backward; REF Born's receiver pair) and written
  int keep_g;                  // REF: Born reads and writes the receiver pair, the migration writes it
  float *dat, *ring, *img;
  long long ring_stride, img_stride;
  uint4 *halo;                 // zeroed before the launch
  int *quit, *err;             // a wait gave up: the launch's flag (zeroed before it), the caller's
  long long patience;          // cycles a wait may take; 0: one unsuccessful poll
};

struct PrtmSlab {
  int slot, R, xa;             // own rows xa .. xa+R-1; shared row r is row xa-2+r
  int src_off;                 // shared offset of the source, -1: out of reach
  int nrec, nring, ntop, top0, nlft, lft0, rgt0;
  int give_up, drawn;
};

struct PrtmLayout {
  int v, x, wz, wx, rec, stage, cs, slab, args, total;
  __host__ __device__ PrtmLayout(int mode, int rmax, int zp, int cap_rec, int cap_ring) {
    const int field = (rmax + 4) * zp;
    v = (mode == PRTM_SOURCE ? 2 : 4) * field;
    x = v + field;                                      // model (Born) or image (backward) of the own rows
    wz = x + (mode == PRTM_SOURCE ? 0 : rmax * zp);
    wx = wz + zp;
    rec = wx + (rmax + 4);                              // offset, index, value: cap_rec each
    stage = rec + 3 * cap_rec;
    cs = stage + cap_ring;
    slab = cs + kPrtmChunks + 1;
    args = (slab + (int)(sizeof(PrtmSlab) / 4) + 3) / 4 * 4;
    total = args + (int)((sizeof(PrtmResident) + 3) / 4);
  }
};

// Sponge weights of a cell: smaller first.
__device__ __forceinline__ float prtm_taper(float v, float wz, float wx) {
  return __fmul_rn(__fmul_rn(v, fminf(wz, wx)), fmaxf(wz, wx));
}

// Ring cell e of a slab: 4 for each model row, then the model depths of the
// two rows on each side.  gi: its index in a step's ring, o: shared offset.
__device__ __forceinline__ void prtm_ring_cell(const PrtmResident &a, const PrtmSlab &b, int e, int &gi, int &o) {
  const PrtmGeo &g = a.g;
  if (e < 4 * b.ntop) {
    const int x = b.top0 + (e >> 2), k = e & 3;   // padded row
    gi = 4 * (x - g.nb) + k;
    o = (x - (b.xa - 2)) * a.zp + (k < 2 ? g.nb - 2 + k : g.nb + g.nz + k - 2);
  } else {
    const int u = e - 4 * b.ntop, k = g.nz > 1 ? (int)__umulhi((unsigned)u, a.nz_magic) : u, mz = u - k * g.nz;
    const bool left = k < b.nlft;
    const int x = left ? b.lft0 + k : b.rgt0 + k - b.nlft, mx = x - g.nb;
    gi = 4 * g.nx + mz + g.nz * (left ? mx + 2 : 2 + mx - g.nx);
    o = (x - (b.xa - 2)) * a.zp + g.nb + mz;
  }
}

template <int MODE>
__device__ __noinline__ void prtm_points(const PrtmResident &a, float *F, int cur, int n) {
  const PrtmLayout l(MODE, a.rmax, a.zp, a.cap_rec, a.cap_ring);
  const PrtmSlab &b = *reinterpret_cast<const PrtmSlab *>(F + l.slab);
  const int tid = threadIdx.x, nthreads = blockDim.x, field = (a.rmax + 4) * a.zp;
  if constexpr (MODE == PRTM_BORN || MODE == PRTM_SOURCE) {
    if (tid == 0 && b.src_off >= 0) {
      float *s = F + cur * field + b.src_off;
      *s = __fadd_rn(*s, a.wl[n]);
    }
  } else {
    const int it = a.g.nt - 1 - n;
    for (int e = tid; e < b.nring; e += nthreads) {
      int gi, o;
      prtm_ring_cell(a, b, e, gi, o);
      F[cur * field + o] = F[l.stage + e];
    }
    if (tid == nthreads - 1 && b.src_off >= 0 && it + 1 < a.g.nt) {
      float *s = F + (cur ^ 1) * field + b.src_off;
      *s = __fsub_rn(*s, a.wl[it + 1]);
    }
    const int *off = reinterpret_cast<const int *>(F + l.rec);
    const float *val = F + l.rec + 2 * a.cap_rec;
    for (int k = tid; k < b.nrec; k += nthreads) {
      if constexpr (MODE == PRTM_MIGRATE) {
        float *q = F + (2 + cur) * field + off[k];
        *q = __fadd_rn(*q, val[k]);
      } else {   // into b = -a of the step before (the model is off the sponge)
        float *q = F + (2 + (cur ^ 1)) * field + off[k];
        *q = __fsub_rn(*q, val[k]);
      }
    }
  }
}

template <int MODE>
__device__ __noinline__ void prtm_helper(const PrtmResident &a, float *F, int cur, int n, int ht, int hn) {
  using namespace resident_detail;
  const PrtmLayout l(MODE, a.rmax, a.zp, a.cap_rec, a.cap_ring);
  const PrtmSlab &b = *reinterpret_cast<const PrtmSlab *>(F + l.slab);
  const int field = (a.rmax + 4) * a.zp;
  const int *off = reinterpret_cast<const int *>(F + l.rec), *idx = off + a.cap_rec;
  if constexpr (MODE == PRTM_BORN) {
    float *d = a.dat + (long long)b.slot * a.g.nt * a.g.ng + n;
    const float *G = F + (2 + cur) * field;
    for (int k = ht; k < b.nrec; k += hn) {
      float *q = d + (long long)idx[k] * a.g.nt;
      *q = __fadd_rn(*q, G[off[k]]);
    }
  } else if constexpr (MODE == PRTM_SOURCE) {
    float *r = a.ring + (long long)b.slot * a.ring_stride + (long long)n * 4 * (a.g.nx + a.g.nz);
    for (int e = ht; e < b.nring; e += hn) {
      int gi, o;
      prtm_ring_cell(a, b, e, gi, o);
      const int row = o / a.zp, z = o - row * a.zp;
      r[gi] = prtm_taper(F[cur * field + o], F[l.wz + z], F[l.wx + row]);
    }
  } else {
    const int it = a.g.nt - 1 - n;
    if (it > 0) {
      const float *r = a.ring + (long long)b.slot * a.ring_stride + (long long)(it - 1) * 4 * (a.g.nx + a.g.nz);
      const uint32_t stage = smem_u32(F + l.stage);
      for (int e = ht; e < b.nring; e += hn) {
        int gi, o;
        prtm_ring_cell(a, b, e, gi, o);
        cp4(stage + 4 * e, r + gi);
      }
      const float *d = a.dat + (long long)b.slot * a.g.nt * a.g.ng + it - 1;
      const uint32_t val = smem_u32(F + l.rec + 2 * a.cap_rec);
      for (int k = ht; k < b.nrec; k += hn) cp4(val + 4 * k, d + (long long)idx[k] * a.g.nt);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
}

// The neighbours' edge rows of the fields step n forms (receive_step of
// resident.cuh, with 2 rows a side).
template <int MODE>
__device__ __noinline__ void prtm_receive(const PrtmResident &a, float *F, int cur, int n) {
  using namespace resident_detail;
  constexpr int NF = MODE == PRTM_SOURCE ? 1 : 2;
  const PrtmLayout l(MODE, a.rmax, a.zp, a.cap_rec, a.cap_ring);
  PrtmSlab &b = *reinterpret_cast<PrtmSlab *>(F + l.slab);
  const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5, field = (a.rmax + 4) * a.zp;
  const bool has_l = b.xa > 2, has_r = b.xa + b.R < a.g.nxpad - 2;
  const int nper = 2 * a.ogroups, nside = (has_l ? 1 : 0) + (has_r ? 1 : 0);
  const int ntotal = NF * nside * nper, nbatch = (ntotal + 31) / 32;
  const size_t side = (size_t)nper * 2;
  const uint32_t tag = (uint32_t)(n + 1);
  for (;;) {
    int k = 0;
    if (lane == 0) k = atomicAdd(&b.drawn, 1);
    k = __shfl_sync(0xffffffffu, k, 0) - n * (nbatch + nwarps);   // every warp draws one past the end a step
    if (k >= nbatch) break;
    const int u = k * 32 + lane;
    bool todo = u < ntotal;
    const int f = NF == 2 && u >= nper * nside ? 1 : 0, v = u - f * nper * nside;
    const int sd = v >= nper ? 1 : 0, gidx = v - sd * nper;
    const bool left = has_l && sd == 0;   // rows before the slab: the left neighbour's last rows
    const int rr = gidx >= a.ogroups ? 1 : 0, grp = gidx - rr * a.ogroups;
    const int nb = left ? (int)blockIdx.x - 1 : (int)blockIdx.x + 1;
    const uint4 *from = a.halo + ((size_t)nb * NF + f) * 4 * side + ((size_t)(n & 1) * 2 + (left ? 1 : 0)) * side +
                        (size_t)gidx * 2;
    float *to = F + (2 * f + (cur ^ 1)) * field + (left ? rr : b.R + 2 + rr) * a.zp + 4 * grp;
    long long t0 = 0;
    for (int spin = 0; todo; spin++) {
      const uint4 x = get_pair2(from), y = get_pair2(from + 1);
      if (x.y == tag && x.w == tag && y.y == tag && y.w == tag) {
        st4(to, make_float4(__uint_as_float(x.x), __uint_as_float(x.z), __uint_as_float(y.x), __uint_as_float(y.z)));
        todo = false;
      } else if (a.patience == 0 || (spin & 255) == 255) {
        // bounded: a.patience cycles, or until another CTA gave up
        const long long now = clock64();
        if (t0 == 0) t0 = now;
        if (now - t0 >= a.patience || *(volatile int *)a.quit) {
          *(volatile int *)a.quit = 1;
          *(volatile int *)a.err = 1;
          b.give_up = 1;
          break;
        }
      }
    }
    __syncwarp();
  }
}

// A wait gave up in step n: what the CTA would still have written is NaN, the
// data from the next step on, the source pair or the image.
template <int MODE>
__device__ __noinline__ void prtm_spoil(const PrtmResident &a, float *F, int n) {
  const PrtmLayout l(MODE, a.rmax, a.zp, a.cap_rec, a.cap_ring);
  const PrtmSlab &b = *reinterpret_cast<const PrtmSlab *>(F + l.slab);
  const int tid = threadIdx.x, nthreads = blockDim.x, nzp = a.g.nzpad, nb = a.g.nb;
  const float nan = __int_as_float(0x7fffffff);
  if constexpr (MODE == PRTM_BORN) {
    const int *idx = reinterpret_cast<const int *>(F + l.rec) + a.cap_rec;
    for (int k = 0; k < b.nrec; k++)
      for (int it = n + 1 + tid; it < a.g.nt; it += nthreads)
        a.dat[((long long)b.slot * a.g.ng + idx[k]) * a.g.nt + it] = nan;
  } else {
    for (int i = tid; i < b.R * nzp; i += nthreads) {
      const int r = i / nzp, z = i - r * nzp, mx = b.xa + r - nb, mz = z - nb;
      if constexpr (MODE == PRTM_SOURCE) {
        const long long p = (long long)b.slot * a.g.fsz + (long long)(b.xa + r) * nzp + z;
        if (z >= 2 && z < nzp - 2) a.s0[p] = a.s1[p] = nan;
      } else {
        if (mx >= 0 && mx < a.g.nx && mz >= 0 && mz < a.g.nz)
          a.img[(long long)b.slot * a.img_stride + (long long)mx * a.g.nz + mz] = nan;
      }
    }
  }
}

template <int ARITH, int MODE>
__global__ void __launch_bounds__(kPrtmThreads, 1) k_prtm_resident(const __grid_constant__ PrtmResident a) {
  using namespace resident_detail;
  constexpr int NF = MODE == PRTM_SOURCE ? 1 : 2;   // 0: source pair, 1: receiver pair
  constexpr bool BACKW = MODE == PRTM_MIGRATE || MODE == PRTM_TRANSPOSE;
  extern __shared__ __align__(16) float F[];
  const PrtmLayout l(MODE, a.rmax, a.zp, a.cap_rec, a.cap_ring);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthreads = blockDim.x;
  const int cwarps = (nthreads >> 5) - a.helpers;
  const int ZP = a.zp, nzp = a.g.nzpad, field = (a.rmax + 4) * ZP, nb = a.g.nb;
  PrtmSlab &sb = *reinterpret_cast<PrtmSlab *>(F + l.slab);
  PrtmResident &sa = *reinterpret_cast<PrtmResident *>(F + l.args);
  int *cs = reinterpret_cast<int *>(F + l.cs);

  // ---- set up
  {
    const int slot = blockIdx.x / a.cps, slab = blockIdx.x - slot * a.cps;
    const int s0 = slab_first(a.g.nxpad - 4, a.cps, slab), R = slab_first(a.g.nxpad - 4, a.cps, slab + 1) - s0;
    const int xa = 2 + s0;
    if (tid == 0) {
      sa = a;
      // ring rows in reach: going back the halo rows too, forward the own
      // rows and, of a sponge of fewer than 4 cells, the grid's outer rows
      // (their cells stay zero)
      const int ra = BACKW || slab == 0 ? xa - 2 : xa, rb = BACKW || slab == a.cps - 1 ? xa + R + 2 : xa + R;
      sb.slot = slot;
      sb.R = R;
      sb.xa = xa;
      const int sp = a.g.spos[slot], sx = sp / nzp, sz = sp - sx * nzp, sr = sx - (xa - 2);
      sb.src_off = sr >= 0 && sr < R + 4 ? sr * ZP + sz : -1;
      sb.nrec = 0;
      sb.top0 = max(ra, nb);
      sb.ntop = max(min(rb, nb + a.g.nx) - sb.top0, 0);
      sb.lft0 = max(ra, nb - 2);
      sb.nlft = max(min(rb, nb) - sb.lft0, 0);
      sb.rgt0 = max(ra, nb + a.g.nx);
      const int nrgt = max(min(rb, nb + a.g.nx + 2) - sb.rgt0, 0);
      sb.nring = MODE == PRTM_BORN ? 0 : 4 * sb.ntop + (sb.nlft + nrgt) * a.g.nz;
      sb.give_up = 0;
      sb.drawn = 0;
    }
    for (int i = tid; i < 2 * NF * field; i += nthreads) F[i] = 0.0f;
    for (int i = tid; i <= a.chunks; i += nthreads) cs[i] = slab_first(R, a.chunks, i);
    for (int z = tid; z < ZP; z += nthreads) {
      const int ib = min(z, nzp - 1 - z);
      F[l.wz + z] = ib >= 0 && ib < nb ? a.g.w[ib] : 1.0f;
    }
    for (int r = tid; r < R + 4; r += nthreads) {
      const int x = xa - 2 + r, ib = min(x, a.g.nxpad - 1 - x);
      F[l.wx + r] = ib < nb ? a.g.w[ib] : 1.0f;
    }
    for (int i = tid; i < (R + 4) * ZP; i += nthreads) {
      const int r = i / ZP, z = i - r * ZP;
      F[l.v + i] = z < nzp ? a.vv[(long long)(xa - 2 + r) * nzp + z] : 0.0f;
    }
    if constexpr (MODE != PRTM_SOURCE) {
      const float *x = MODE == PRTM_BORN ? a.mod : a.img + (long long)slot * a.img_stride;
      for (int i = tid; i < R * ZP; i += nthreads) {
        const int r = i / ZP, z = i - r * ZP, mx = xa + r - nb, mz = z - nb;
        F[l.x + i] = mx >= 0 && mx < a.g.nx && mz >= 0 && mz < a.g.nz ? x[(long long)mx * a.g.nz + mz] : 0.0f;
      }
    }
    __syncthreads();
    if constexpr (BACKW || MODE == PRTM_BORN) {
      // backward: the source pair (s0 the field the ring belongs to); Born
      // continuing from earlier fields: the receiver pair (g0 the newest)
      const long long off = (long long)slot * a.g.fsz;
      const float *q0 = MODE == PRTM_BORN ? a.g0 + off : a.s0 + off, *q1 = MODE == PRTM_BORN ? a.g1 + off : a.s1 + off;
      if (BACKW || a.keep_g) {
        float *d0 = F + (MODE == PRTM_BORN ? 2 * field : 0), *d1 = d0 + field;
        for (int i = tid; i < (R + 4) * ZP; i += nthreads) {
          const int r = i / ZP, z = i - r * ZP;
          if (z >= nzp) continue;
          const long long p = (long long)(xa - 2 + r) * nzp + z;
          d0[i] = MODE == PRTM_BORN ? prtm_taper(q0[p], F[l.wz + z], F[l.wx + r]) : q0[p];
          d1[i] = q1[p];
        }
      }
    }
    if constexpr (MODE != PRTM_SOURCE) {
      int *off = reinterpret_cast<int *>(F + l.rec), *idx = off + a.cap_rec;
      for (int i = tid; i < a.g.ng; i += nthreads) {
        const int p = a.g.rpos[(long long)slot * a.g.ng + i];
        const int x = p / nzp, z = p - x * nzp, r = x - (xa - 2);
        if (BACKW ? (r < 0 || r >= R + 4) : (r < 2 || r >= R + 2)) continue;
        const int k = atomicAdd(&sb.nrec, 1);
        if (k < a.cap_rec) {
          off[k] = r * ZP + z;
          idx[k] = i;
        }
      }
    }
    __syncthreads();
    if (tid == 0) sb.nrec = min(sb.nrec, a.cap_rec);
    __syncthreads();
    if constexpr (BACKW) {
      const int it = a.g.nt - 1;
      const int *idx = reinterpret_cast<const int *>(F + l.rec) + a.cap_rec;
      const float *d = a.dat + (long long)slot * a.g.nt * a.g.ng + it;
      for (int k = tid; k < sb.nrec; k += nthreads) F[l.rec + 2 * a.cap_rec + k] = d[(long long)idx[k] * a.g.nt];
      const float *r = a.ring + (long long)slot * a.ring_stride + (long long)it * 4 * (a.g.nx + a.g.nz);
      for (int e = tid; e < sb.nring; e += nthreads) {
        int gi, o;
        prtm_ring_cell(sa, sb, e, gi, o);
        F[l.stage + e] = r[gi];
      }
    }
    __syncthreads();
  }
  const int R = sb.R, xa = sb.xa;
  const bool points = BACKW || sb.src_off >= 0;
  const bool has_l = xa > 2, has_r = xa + R < a.g.nxpad - 2;
  const int K = a.chunks, G = a.ngroups, items = K * G, wtasks = (items + 29) / 30, L = (R + K - 1) / K;
  const float k0 = a.c.c0, k11 = a.c.c11, k12 = a.c.c12, k21 = a.c.c21, k22 = a.c.c22;
  int cur = 0;

  for (int n = 0; n < a.g.nt; n++) {
    if (points) {
      prtm_points<MODE>(sa, F, cur, n);
      __syncthreads();
    }
    if (warp < cwarps) {
      const uint32_t tag = (uint32_t)(n + 1);
      // the new field's sponge; REF Born leaves the last field as the
      // unfused loop does, to be tapered by the next call
      const bool taper_new = MODE == PRTM_SOURCE || MODE == PRTM_MIGRATE || (MODE == PRTM_BORN && n + 1 < a.g.nt);
      for (int task = warp; task < wtasks; task += cwarps) {
        const int id = task * 30 + lane - 1, idc = min(max(id, 0), items - 1);
        const int chunk = (int)(((unsigned)idc * a.gmagic) >> 20), grp = idc - chunk * G;
        const int c0 = cs[chunk], c1 = cs[chunk + 1], zg = 4 * grp;
        const bool outlane = lane >= 1 && lane <= 30 && id < items && grp < a.ogroups;
        bool zok[4];
#pragma unroll
        for (int i = 0; i < 4; i++) zok[i] = zg + i >= 2 && zg + i < nzp - 2;
        const float *S = F + cur * field + c0 * ZP + zg;             // row c0 + i of the march
        float *SP = F + (cur ^ 1) * field + (c0 + 2) * ZP + zg;      // output rows
        const float *Gc = S + 2 * field;
        float *GP = SP + 2 * field;
        const float *V = F + l.v + c0 * ZP + zg;
        float *X = F + l.x + c0 * ZP + zg;
        const float *wx = F + l.wx + c0 + 2;
        const float4 wz = ld4(F + l.wz + zg);
        const unsigned hp = (blockIdx.x * NF * 4 + (n & 1) * 2) * (unsigned)(4 * a.ogroups) + 2 * grp;

        float4 qs[5], qg[5];   // rows c0+i-4 .. c0+i: the source field; the receiver field (Born: times vv)
        auto load = [&](auto uu) {
          constexpr int U = decltype(uu)::value;
          qs[U] = ld4(S);
          S += ZP;
          if constexpr (NF == 2) {
            float4 v = ld4(Gc);
            if constexpr (MODE == PRTM_BORN) {
              const float4 w = ld4(V);
              v = make_float4(__fmul_rn(w.x, v.x), __fmul_rn(w.y, v.y), __fmul_rn(w.z, v.z), __fmul_rn(w.w, v.w));
            }
            qg[U] = v;
            Gc += ZP;
          }
          V += ZP;
        };
        // stencil sums of the queue's centre row (FAST: the FMA chain; REF:
        // left to right, the centre term given)
        auto sums = [&](const float4 (&q)[5], auto uu, const float (&first)[4], float (&s)[4]) {
          constexpr int U = decltype(uu)::value;
          const float4 m2 = q[(U + 1) % 5], m1 = q[(U + 2) % 5], c = q[(U + 3) % 5], p1 = q[(U + 4) % 5], p2 = q[U];
          const float zn[8] = {__shfl_up_sync(0xffffffffu, c.z, 1), __shfl_up_sync(0xffffffffu, c.w, 1), c.x, c.y, c.z,
                               c.w, __shfl_down_sync(0xffffffffu, c.x, 1), __shfl_down_sync(0xffffffffu, c.y, 1)};
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float z1 = __fadd_rn(zn[i + 1], zn[i + 3]), z2 = __fadd_rn(zn[i], zn[i + 4]);
            const float x1 = __fadd_rn(get(m1, i), get(p1, i)), x2 = __fadd_rn(get(m2, i), get(p2, i));
            float t = first[i];
            if constexpr (ARITH == ARITH_REF) {
              t = __fadd_rn(t, __fmul_rn(k11, z1));
              t = __fadd_rn(t, __fmul_rn(k12, z2));
              t = __fadd_rn(t, __fmul_rn(k21, x1));
              t = __fadd_rn(t, __fmul_rn(k22, x2));
            } else {
              t = fmaf(k11, z1, t);
              t = fmaf(k12, z2, t);
              t = fmaf(k21, x1, t);
              t = fmaf(k22, x2, t);
            }
            s[i] = t;
          }
        };
        // march step i: load row c0+i; output row j = i - 4
        auto step = [&](auto uu, int j) {
          constexpr int U = decltype(uu)::value;
          load(uu);
          const float4 vc4 = ld4(V - 3 * ZP);   // vv at the output row
          const float4 c4 = qs[(U + 3) % 5], p4 = ld4(SP);
          const float wr = wx[j];
          float so[4], go[4];
          {
            const float first[4] = {__fmul_rn(k0, c4.x), __fmul_rn(k0, c4.y), __fmul_rn(k0, c4.z), __fmul_rn(k0, c4.w)};
            float s[4];
            sums(qs, uu, first, s);
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const float p = BACKW ? get(p4, i) : prtm_taper(get(p4, i), get(wz, i), wr);
              if constexpr (ARITH == ARITH_REF)
                so[i] = __double2float_rn(__dadd_rn(__dsub_rn(__dmul_rn(2.0, (double)get(c4, i)), (double)p),
                                                    (double)__fmul_rn(get(vc4, i), s[i])));
              else
                so[i] = fmaf(s[i], get(vc4, i), fmaf(2.0f, get(c4, i), -p));
              if (MODE == PRTM_SOURCE || (MODE == PRTM_BORN && taper_new)) so[i] = prtm_taper(so[i], get(wz, i), wr);
            }
          }
          if constexpr (MODE == PRTM_BORN) {
            const float4 g4 = ld4(Gc - 3 * ZP), gp4 = ld4(GP), m4 = ld4(X), vu4 = qg[(U + 3) % 5];
            if constexpr (ARITH == ARITH_REF) {
              // every product's sum goes to double on its own
              const float4 m2 = qg[(U + 1) % 5], m1 = qg[(U + 2) % 5], p1 = qg[(U + 4) % 5], p2 = qg[U];
              const float zn[8] = {__shfl_up_sync(0xffffffffu, vu4.z, 1), __shfl_up_sync(0xffffffffu, vu4.w, 1),
                                   vu4.x, vu4.y, vu4.z, vu4.w, __shfl_down_sync(0xffffffffu, vu4.x, 1),
                                   __shfl_down_sync(0xffffffffu, vu4.y, 1)};
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const float p = prtm_taper(__fadd_rn(get(gp4, i), __fmul_rn(get(p4, i), get(m4, i))), get(wz, i), wr);
                double t = __dsub_rn(__dmul_rn(2.0, (double)get(g4, i)), (double)p);
                t = __dadd_rn(t, (double)__fmul_rn(__fmul_rn(k0, get(vc4, i)), get(g4, i)));
                t = __dadd_rn(t, (double)__fmul_rn(k11, __fadd_rn(zn[i + 1], zn[i + 3])));
                t = __dadd_rn(t, (double)__fmul_rn(k12, __fadd_rn(zn[i], zn[i + 4])));
                t = __dadd_rn(t, (double)__fmul_rn(k21, __fadd_rn(get(m1, i), get(p1, i))));
                t = __dadd_rn(t, (double)__fmul_rn(k22, __fadd_rn(get(m2, i), get(p2, i))));
                go[i] = __double2float_rn(t);
              }
            } else {
              const float first[4] = {k0 * vu4.x, k0 * vu4.y, k0 * vu4.z, k0 * vu4.w};
              float s[4];
              sums(qg, uu, first, s);
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const float p = prtm_taper(__fadd_rn(get(gp4, i), __fmul_rn(get(p4, i), get(m4, i))), get(wz, i), wr);
                go[i] = __fadd_rn(fmaf(2.0f, get(g4, i), -p), s[i]);
              }
            }
            if (taper_new) {
#pragma unroll
              for (int i = 0; i < 4; i++) go[i] = prtm_taper(go[i], get(wz, i), wr);
            }
          } else if constexpr (BACKW) {
            const float4 g4 = qg[(U + 3) % 5], gp4 = ld4(GP);
            const float first[4] = {__fmul_rn(k0, g4.x), __fmul_rn(k0, g4.y), __fmul_rn(k0, g4.z), __fmul_rn(k0, g4.w)};
            if constexpr (MODE == PRTM_MIGRATE) {
              float s[4];
              sums(qg, uu, first, s);
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const float p = prtm_taper(get(gp4, i), get(wz, i), wr);
                float t;
                if constexpr (ARITH == ARITH_REF)
                  t = __double2float_rn(__dadd_rn(__dsub_rn(__dmul_rn(2.0, (double)get(g4, i)), (double)p),
                                                  (double)__fmul_rn(get(vc4, i), s[i])));
                else
                  t = fmaf(s[i], get(vc4, i), fmaf(2.0f, get(g4, i), -p));
                go[i] = prtm_taper(t, get(wz, i), wr);
              }
            } else {
              // k_prtm_born_transpose's FMA chain in either arithmetic
              const float4 m2 = qg[(U + 1) % 5], m1 = qg[(U + 2) % 5], p1 = qg[(U + 4) % 5], p2 = qg[U];
              const float zn[8] = {__shfl_up_sync(0xffffffffu, g4.z, 1), __shfl_up_sync(0xffffffffu, g4.w, 1), g4.x,
                                   g4.y, g4.z, g4.w, __shfl_down_sync(0xffffffffu, g4.x, 1),
                                   __shfl_down_sync(0xffffffffu, g4.y, 1)};
#pragma unroll
              for (int i = 0; i < 4; i++) {
                float t = first[i];
                t = fmaf(k11, __fadd_rn(zn[i + 1], zn[i + 3]), t);
                t = fmaf(k12, __fadd_rn(zn[i], zn[i + 4]), t);
                t = fmaf(k21, __fadd_rn(get(m1, i), get(p1, i)), t);
                t = fmaf(k22, __fadd_rn(get(m2, i), get(p2, i)), t);
                const float wp = __fmul_rn(get(wz, i), wr);
                const float b = __fmul_rn(wp, -get(gp4, i));
                go[i] = __fmul_rn(wp, fmaf(get(vc4, i), t, fmaf(2.0f, get(g4, i), b)));
              }
            }
          }
          if (outlane && c0 + j < c1) {
#pragma unroll
            for (int i = 0; i < 4; i++) {   // border cells stay zero
              so[i] = zok[i] ? so[i] : 0.0f;
              if constexpr (NF == 2) go[i] = zok[i] ? go[i] : 0.0f;
            }
            st4(SP, make_float4(so[0], so[1], so[2], so[3]));
            if constexpr (NF == 2) st4(GP, make_float4(go[0], go[1], go[2], go[3]));
            if constexpr (BACKW) {
              const float4 g4 = qg[(U + 3) % 5];
              const float4 m = ld4(X);
              float o[4];
#pragma unroll
              for (int i = 0; i < 4; i++) {
                if constexpr (MODE == PRTM_MIGRATE) o[i] = __fadd_rn(get(m, i), __fmul_rn(so[i], go[i]));
                else o[i] = fmaf(so[i], -get(g4, i), get(m, i));
              }
              st4(X, make_float4(o[0], o[1], o[2], o[3]));
            }
            const int row = c0 + j;
            if (row < 2 && has_l) {
              uint4 *d = a.halo + (hp + (unsigned)(row * a.ogroups * 2));
              put_pair2(d, so[0], so[1], tag);
              put_pair2(d + 1, so[2], so[3], tag);
              if constexpr (NF == 2) {
                uint4 *e = d + 16 * a.ogroups;   // the receiver pair's block: 4 sides of 4 * ogroups
                put_pair2(e, go[0], go[1], tag);
                put_pair2(e + 1, go[2], go[3], tag);
              }
            }
            if (row >= R - 2 && has_r) {
              uint4 *d = a.halo + (hp + (unsigned)((row - R + 4) * a.ogroups * 2));
              put_pair2(d, so[0], so[1], tag);
              put_pair2(d + 1, so[2], so[3], tag);
              if constexpr (NF == 2) {
                uint4 *e = d + 16 * a.ogroups;
                put_pair2(e, go[0], go[1], tag);
                put_pair2(e + 1, go[2], go[3], tag);
              }
            }
          }
          SP += ZP;
          if constexpr (NF == 2) GP += ZP;
          X += ZP;
        };
        load(std::integral_constant<int, 0>{});
        load(std::integral_constant<int, 1>{});
        load(std::integral_constant<int, 2>{});
        load(std::integral_constant<int, 3>{});
#define SWFWI_PRTM_STEP(U)                       \
  step(std::integral_constant<int, (U)>{}, j);   \
  if (++j >= L) break;
        for (int j = 0;;) {
          SWFWI_PRTM_STEP(4) SWFWI_PRTM_STEP(0) SWFWI_PRTM_STEP(1) SWFWI_PRTM_STEP(2) SWFWI_PRTM_STEP(3)
        }
#undef SWFWI_PRTM_STEP
      }
    } else {
      const int hn = 32 * a.helpers;
      prtm_helper<MODE>(sa, F, cur, n, tid - (nthreads - hn), hn);
    }
    if (n + 1 < a.g.nt && (has_l || has_r)) prtm_receive<MODE>(sa, F, cur, n);
    if constexpr (BACKW) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    cur ^= 1;
    if (sb.give_up) {   // uniform: written before the barrier, never cleared
      prtm_spoil<MODE>(sa, F, n);
      return;
    }
  }

  // ---- results
  const long long off = (long long)sb.slot * a.g.fsz;
  if constexpr (MODE == PRTM_SOURCE || MODE == PRTM_BORN) {
    // source sweep: s0 = the field the last step advanced from, tapered, s1 =
    // the newest; Born: g0 = the newest, g1 = the one before
    if (MODE == PRTM_SOURCE || a.keep_g) {
      const float *older = F + (MODE == PRTM_BORN ? 2 * field : 0) + (cur ^ 1) * field;
      const float *newest = F + (MODE == PRTM_BORN ? 2 * field : 0) + cur * field;
      for (int i = tid; i < R * ZP; i += nthreads) {
        const int r = i / ZP, z = i - r * ZP, k = i + 2 * ZP;
        if (z < 2 || z >= nzp - 2) continue;
        const long long p = off + (long long)(xa + r) * nzp + z;
        if constexpr (MODE == PRTM_SOURCE) {
          a.s0[p] = prtm_taper(older[k], F[l.wz + z], F[l.wx + r + 2]);
          a.s1[p] = newest[k];
        } else {
          a.g0[p] = newest[k];
          a.g1[p] = older[k];
        }
      }
    }
  } else {
    if (MODE == PRTM_MIGRATE && a.keep_g) {
      // the receiver pair as the unfused loop leaves it: g0 the field the
      // last step advanced from, g1 the newest, both tapered
      const float *older = F + (2 + (cur ^ 1)) * field, *newest = F + (2 + cur) * field;
      for (int i = tid; i < R * ZP; i += nthreads) {
        const int r = i / ZP, z = i - r * ZP, k = i + 2 * ZP;
        if (z < 2 || z >= nzp - 2) continue;
        const long long p = off + (long long)(xa + r) * nzp + z;
        a.g0[p] = prtm_taper(older[k], F[l.wz + z], F[l.wx + r + 2]);
        a.g1[p] = newest[k];
      }
    }
    float *img = a.img + (long long)sb.slot * a.img_stride;
    for (int i = tid; i < R * ZP; i += nthreads) {
      const int r = i / ZP, z = i - r * ZP, mx = xa + r - nb, mz = z - nb;
      if (mx >= 0 && mx < a.g.nx && mz >= 0 && mz < a.g.nz) img[(long long)mx * a.g.nz + mz] = F[l.x + i];
    }
  }
}

}  // namespace
}  // namespace swfwi
