// Learned preconditioner: BF16 convolutions on the fifth-generation tensor
// cores (forward, data gradient and weight gradient: tcgen05.mma with FP32
// accumulators in tensor memory), the encoder-decoder around them, its
// training step and the features/scatter between the padded model grid and
// the network's image.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <random>
#include "conv_tiles.hpp"
#include "kernels.cuh"
#include "precond.hpp"
#include "stream.cuh"

namespace swfwi {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kEw = 256;   // threads of the elementwise kernels
constexpr int kDotThreads = 32;    // of the channel sums: kEw / C runs x C / 8 groups
constexpr int kRowThreads = 128;   // threads of those that take an image row a blockIdx.y

inline void noted() { g_kernel_launches.fetch_add(1, std::memory_order_relaxed); }
inline unsigned blocks_for(long long n, int threads = kEw) {
  long long b = (n + threads - 1) / threads;
  return (unsigned)std::max(1LL, std::min(b, 148LL * 64));
}

// The network's forward kernels are launched with programmatic stream
// serialisation: the next one's blocks are set up while this one ends, and
// touch memory only after entering, when all it wrote is visible.  A proposal
// is 30 launches of a few microseconds: 232 us for 480 x 160 without, 188 so.
__device__ __forceinline__ void let_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void enter() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
void launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  SWFWI_CUDA(cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...));
  noted();
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}

// ---------------------------------------------------------------- 3x3 conv, tcgen05
// Implicit GEMM on the fifth-generation tensor cores.  A CTA of 128 threads
// owns 128 consecutive pixels of the flattened (n, h, w) index (M = 128) and
// every output channel (N = cout, a multiple of 16 up to 256); K = 9 taps x
// cin, 16 channels per MMA.  The taps go in rounds of T (9, 3 or 1, the most
// whose tiles fit the shared-memory budget): per round the threads copy, for
// each of its taps, the 128 shifted pixel rows (zero-filled outside the
// image) and the tap's weights into shared memory with cp.async, as K-major
// core matrices without swizzle (8 rows x 16 bytes; the 8-row groups 256 B
// apart, the two 8-channel halves of a 16-channel chunk 128 B apart).  With
// more than one round, two stages: while the tensor cores run one round, the
// copies of the next land in the other stage.  One thread issues a round's
// T x cin/16 tcgen05.mma into the FP32 accumulator in tensor memory and
// commits them to the stage's mbarrier; a stage is refilled only after its
// barrier shows those MMAs done (bounded waits).  Narrow layers take all 9
// taps in one round: one copy, MMA and commit latency per CTA instead of 9.
// The epilogue reads the accumulator 16 columns at a time (warp w holds the
// tensor-memory lanes, i.e. pixels, 32w .. 32w+31) and writes BF16 with
// bias and ReLU, or FP32 (optionally added to the output).  A wait that
// gives up sets g_conv_timeout; the CTA still frees its tensor memory.
// (The row-tile kernel below replaces this one wherever its stages fit.)
__device__ int g_conv_timeout;

namespace tc {
__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// shared-memory matrix descriptor: start address, leading (K) byte offset
// 128, stride (8-row group) byte offset 256, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(256u >> 4) << 32) |
         (1ull << 46);
}
// 16 bytes global -> shared, zero-filled when !valid (src is then not read)
__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// bytes of one stage of T taps (A and B tiles)
__host__ __device__ inline int stage_bytes(int cin, int cout, int T) { return T * (cin / 16) * (4096 + 32 * cout); }
constexpr int kStageBudget = 96 * 1024;   // shared memory the stages may take
// taps per round: the most of 9, 3, 1 whose stages fit the budget
__host__ __device__ inline int taps_per_round(int cin, int cout) {
  if (stage_bytes(cin, cout, 9) <= kStageBudget) return 9;
  return 2 * stage_bytes(cin, cout, 3) <= kStageBudget ? 3 : 1;
}
}  // namespace tc

template <bool F32>
__global__ void __launch_bounds__(128) k_conv3x3_tc(const bf16 *__restrict__ in, int cin,
                                                    const bf16 *__restrict__ w, const float *__restrict__ bias,
                                                    void *out, int accum, int cout, int N, int H, int W) {
  using namespace stream_detail;
  extern __shared__ __align__(1024) unsigned char sm[];
  const int KC = cin / 16, T = tc::taps_per_round(cin, cout), R = 9 / T;
  const int SB = tc::stage_bytes(cin, cout, T), NS = R > 1 ? 2 : 1;
  // stage s at sm + s*SB: the round's A tiles (T x KC x 4 KB, tap-major),
  // then its B tiles (T x KC x cout x 32 B)
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + NS * SB);   // one per stage
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long HW = (long long)H * W, P = (long long)N * HW;
  const long long p0 = (long long)blockIdx.x * 128;
  const uint32_t ncols = (uint32_t)tmem_cols(cout);
  // thread tid copies A row tid (its pixel, decoded once; valid = inside the
  // batch) and the B rows co = tid, tid + 128, ... of every tap
  const long long pm = p0 + tid;
  const bool pin = pm < P;
  const int pn = pin ? (int)(pm / HW) : 0, pr = pin ? (int)(pm - (long long)pn * HW) : 0;
  const int ph = pr / W, pw = pr - ph * W;
  // the row's place in a 16-channel chunk's A tile (core matrix, row within it)
  const uint32_t arow = (uint32_t)((tid >> 3) * 256 + (tid & 7) * 16);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::saddr(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t taddr = *tslot;
  // kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B, both
  // K-major, N = cout, M = 128
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(cout >> 3) << 17) | ((128u >> 4) << 24);
  const uint32_t sbase = tc::saddr(sm);

  auto load_round = [&](int rd) {
    const uint32_t sa = sbase + (uint32_t)((rd % NS) * SB), sb = sa + (uint32_t)(T * KC * 4096);
    for (int t = 0; t < T; t++) {
      const int tap = rd * T + t, ky = tap / 3, kx = tap - 3 * ky;
      const uint32_t at = sa + (uint32_t)(t * KC * 4096) + arow, bt = sb + (uint32_t)(t * KC * cout * 32);
      const int hh = ph + ky - 1, xx = pw + kx - 1;
      const bool ok = pin && hh >= 0 && hh < H && xx >= 0 && xx < W;
      const bf16 *src = ok ? in + (((long long)pn * H + hh) * W + xx) * cin : in;
      // 16 bytes per step along the pixel's channels: chunk q >> 1, half q & 1
      for (int q = 0; q < 2 * KC; q++)
        tc::cp16(at + (uint32_t)((q >> 1) * 4096 + (q & 1) * 128), ok ? src + q * 8 : in, ok);
      for (int co = tid; co < cout; co += 128) {
        const bf16 *wr = w + ((long long)co * 9 + tap) * cin;
        const uint32_t brow = bt + (uint32_t)((co >> 3) * 256 + (co & 7) * 16);
        for (int q = 0; q < 2 * KC; q++)
          tc::cp16(brow + (uint32_t)((q >> 1) * cout * 32 + (q & 1) * 128), wr + q * 8, true);
      }
    }
    tc::cp_commit();
  };

  bool ok = true;
  load_round(0);
  for (int rd = 0; rd < R && ok; rd++) {
    if (rd + 1 < R) {
      // the next round's stage was read by the MMAs of round rd-1: wait for them
      if (rd >= 1 && !__syncthreads_and(mbar_wait(&bar[(rd + 1) & 1], (uint32_t)(((rd - 1) >> 1) & 1)))) {
        ok = false;
        break;
      }
      load_round(rd + 1);
      tc::cp_wait<1>();   // this round's copies are complete, the next round's may be in flight
    } else {
      tc::cp_wait<0>();
    }
    // the tiles were written through the generic proxy; the MMA reads them
    // through the async proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sa = sbase + (uint32_t)((rd % NS) * SB), sb = sa + (uint32_t)(T * KC * 4096);
      for (int kc = 0; kc < T * KC; kc++) {   // (tap within the round, 16-channel chunk)
        const uint64_t ad = tc::kmajor_desc(sa + kc * 4096);
        const uint64_t bd = tc::kmajor_desc(sb + kc * cout * 32);
        const uint32_t acc = (rd > 0 || kc > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(taddr),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       tc::saddr(&bar[rd & 1]))
                   : "memory");
    }
  }
  // the last commit (round R-1, its barrier's ((R-1)/2 + 1)-th phase) covers every MMA
  if (ok && !__syncthreads_and(mbar_wait(&bar[(R - 1) & 1], (uint32_t)(((R - 1) >> 1) & 1)))) ok = false;
  tc::cp_wait<0>();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    const long long p = p0 + warp * 32 + lane;
    for (int c0 = 0; c0 < cout; c0 += 16) {
      uint32_t r[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
            "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (p < P) {
        if constexpr (F32) {
          float4 *o = reinterpret_cast<float4 *>(reinterpret_cast<float *>(out) + p * cout + c0);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            float4 v = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                   __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
            if (accum) {
              const float4 q = o[i];
              v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
            }
            o[i] = v;
          }
        } else {
          uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<bf16 *>(out) + p * cout + c0);
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 8; i++)
            pk[i] = pack_bf16(fmaxf(__uint_as_float(r[2 * i]) + bias[c0 + 2 * i], 0.0f),
                              fmaxf(__uint_as_float(r[2 * i + 1]) + bias[c0 + 2 * i + 1], 0.0f));
          o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
      }
    }
  } else if (tid == 0) {
    atomicExch(&g_conv_timeout, 1);
    // bounded: whatever MMAs are still in flight, before their tensor memory goes
    mbar_wait(&bar[0], 0u);
    mbar_wait(&bar[1], 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------- 3x3 conv, tcgen05, row tiles
// The same implicit GEMM with row-aligned tiles in a persistent kernel.  A
// tile's 128 pixels are 16 groups of 8 consecutive pixels of one image row
// each.  For every group the three input rows it needs (h-1, h, h+1) are
// staged once, 10 pixels wide (the group and a one-pixel halo), as 16-byte
// rows per 8-channel half: A(tap ky, kx) is then the staged rows of ky seen
// from a start address shifted by kx rows, with the 8-row groups 160 B apart
// -- the three column taps share one copy, and the input is copied 30/8 times
// instead of 9.
// A CTA keeps the weights of its output channels in shared memory and walks
// over tiles: 320 threads copy (a thread one pixel and 8-channel half of every
// 16 channels, no divisions beyond its group's place once a tile) into a ring
// of stages, a stage being a tile's three rows or one of them (stage_rows), a
// warp issues the MMAs, and four warps drain one accumulator while the next is
// formed.  The copies bound it.  One tile a CTA with everything in turn took
// 114 us for 16 -> 16 channels on 1.2 million pixels.
// The MMAs of an output are those of that form in the same order (taps, then
// channels): the same bits.

// KC = cin / 16 is a template parameter: loops by constants.
template <bool F32, int KC>
__global__ void __launch_bounds__(tg::kThreads) k_conv3x3_tg(const bf16 *__restrict__ in, const bf16 *__restrict__ w,
                                                             const float *__restrict__ bias, void *out, int accum,
                                                             int cout, int N, int H, int W) {
  using namespace stream_detail;
  extern __shared__ __align__(1024) unsigned char sm[];
  constexpr int cin = 16 * KC, NKY = KC <= 3 ? 3 : 1, R = 3 / NKY;
  const int S = tg::stages(cin, cout), SB = tg::stage_bytes(cin), WB = tg::weight_bytes(cin, cout);
  const int NC = tg::cols(cin, cout), co0 = blockIdx.y * NC;   // this CTA's output channels
  uint64_t *full = reinterpret_cast<uint64_t *>(sm + WB + S * SB), *empty = full + tg::kMaxStages;
  uint64_t *ready = empty + tg::kMaxStages, *taken = ready + 2;   // an accumulator is formed, is read
  uint32_t *tslot = reinterpret_cast<uint32_t *>(taken + 2);
  volatile int *bad = reinterpret_cast<volatile int *>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned GW = (unsigned)(W + 7) / 8, groups = (unsigned)N * H * GW;
  const int tiles = (int)((groups + 15) / 16);
  const uint32_t ncols = (uint32_t)tmem_cols(2 * NC);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::saddr(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int k = 0; k < tg::kMaxStages; k++) {
      mbar_init(&full[k], tg::kCopyThreads);
      mbar_init(&empty[k], 1);
    }
    for (int k = 0; k < 2; k++) {
      mbar_init(&ready[k], 1);
      mbar_init(&taken[k], 128);
    }
    *bad = 0;
    fence_mbar_init();
  }
  const uint32_t sbase = tc::saddr(sm);
  enter();
  // weights: 9 taps x [kc] x NC rows in K-major core matrices
  for (int u = tid; u < 9 * NC * 2 * KC; u += tg::kThreads) {
    const int q = u % (2 * KC), v = u / (2 * KC), co = v % NC, tap = v / NC;
    tc::cp16(sbase + (uint32_t)((tap * KC + (q >> 1)) * NC * 32 + ((co >> 3) * 2 + (q & 1)) * 128 + (co & 7) * 16),
             w + ((long long)(co0 + co) * 9 + tap) * cin + q * 8, true);
  }
  tc::cp_commit();
  tc::cp_wait<0>();
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t taddr = *tslot;
  // not before this CTA holds its tensor memory: a block of the next kernel
  // that took it would wait for this one
  let_next();

  if (warp < tg::kCopyThreads / 32) {
    // ---- copies: pixel px of group g, channels 8 * half .. of every 16
    const int half = tid & 1, t = tid >> 1, g = t / 10, px = t - 10 * g;
    const uint32_t dst0 = sbase + (uint32_t)(WB + half * NKY * tg::kPlaneRow + g * tg::kGroupBytes + px * 16);
    auto landed = [&](int unit) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::saddr(&full[unit % S])) : "memory");
    };
    int unit = 0;
    bool stop = false;
    for (int tile = blockIdx.x; tile < tiles && !stop; tile += gridDim.x) {
      const unsigned gi = (unsigned)tile * 16 + g, row = gi / GW;
      const int n = (int)(row / (unsigned)H), h = (int)(row - (unsigned)n * H), x = (int)(gi - row * GW) * 8 + px - 1;
      const bool col = gi < groups && x >= 0 && x < W;
      const bf16 *src0 = in + (((long long)n * H + h - 1) * W + x) * cin + 8 * half;
      for (int rd = 0; rd < R; rd++, unit++) {
        const int st = unit % S;
        if (*bad || (unit >= S && !mbar_wait(&empty[st], (uint32_t)((unit / S - 1) & 1)))) {
          *bad = 1;
          stop = true;
          break;
        }
        const uint32_t dst = dst0 + (uint32_t)(st * SB);
#pragma unroll
        for (int k = 0; k < NKY; k++) {
          const int ky = rd * NKY + k, y = h + ky - 1;
          const bool ok = col && y >= 0 && y < H;
          const bf16 *src = src0 + (long long)ky * W * cin;
#pragma unroll
          for (int kc = 0; kc < KC; kc++)
            tc::cp16(dst + (uint32_t)((kc * 2 * NKY + k) * tg::kPlaneRow), ok ? src + 16 * kc : in, ok);
        }
        tc::cp_commit();
        if (unit > 0) {
          tc::cp_wait<1>();
          landed(unit - 1);
        }
      }
    }
    tc::cp_wait<0>();
    if (unit > 0) landed(unit - 1);
  } else if (warp == tg::kCopyThreads / 32) {
    // ---- MMAs
    if (lane == 0) {
      // kind::f16: FP32 accumulator, BF16 A and B, both K-major, N = NC, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NC >> 3) << 17) | ((128u >> 4) << 24);
      int unit = 0, k = 0;
      bool stop = false;
      for (int tile = blockIdx.x; tile < tiles && !stop; tile += gridDim.x, k++) {
        const int buf = k & 1;
        if (*bad || (k >= 2 && !mbar_wait(&taken[buf], (uint32_t)((k / 2 - 1) & 1)))) {
          *bad = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc0 = taddr + (uint32_t)(buf * NC);
        for (int rd = 0; rd < R; rd++, unit++) {
          const int st = unit % S;
          if (*bad || !mbar_wait(&full[st], (uint32_t)((unit / S) & 1))) {
            *bad = 1;
            stop = true;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = sbase + (uint32_t)(WB + st * SB);
          for (int t = 0; t < 3 * NKY; t++) {
            const int kyl = t / 3, kx = t - 3 * kyl;
            for (int kc = 0; kc < KC; kc++) {
              // A rows: group g at g*160, row i of the group at (i + kx)*16;
              // the channel halves NKY planes apart
              const uint32_t a_addr = sa + (uint32_t)((kc * 2 * NKY + kyl) * tg::kPlaneRow + kx * 16);
              const uint64_t ad = (uint64_t)((a_addr >> 4) & 0x3FFFu) |
                                  ((uint64_t)((uint32_t)(NKY * tg::kPlaneRow) >> 4) << 16) |
                                  ((uint64_t)((uint32_t)tg::kGroupBytes >> 4) << 32) | (1ull << 46);
              const uint64_t bd = tc::kmajor_desc(sbase + (uint32_t)(((rd * 3 * NKY + t) * KC + kc) * NC * 32));
              const uint32_t acc = (rd > 0 || t > 0 || kc > 0) ? 1u : 0u;
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(acc0),
                  "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                  : "memory");
            }
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           tc::saddr(&empty[st]))
                       : "memory");
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         tc::saddr(&ready[buf]))
                     : "memory");
      }
      // a wait gave up: bounded, the MMAs still in flight
      if (*bad && k > 0) mbar_wait(&ready[(k - 1) & 1], (uint32_t)(((k - 1) / 2) & 1));
    }
    __syncwarp();
  } else {
    // ---- epilogue: warp q holds the tensor-memory lanes 32 q .., q = warp % 4
    const int q = warp & 3, r = q * 32 + lane, g = r >> 3, i = r & 7;
    int k = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, k++) {
      const int buf = k & 1;
      const unsigned gi = (unsigned)tile * 16 + g, row = gi / GW;
      const int x = (int)(gi - row * GW) * 8 + i;
      const bool valid = gi < groups && x < W;
      const long long p = valid ? (long long)row * W + x : 0;
      const bool got = mbar_wait(&ready[buf], (uint32_t)((k / 2) & 1));
      if (!got) *bad = 1;
      // one decision a warp: the reads of tensor memory are whole warps'
      if (__any_sync(0xffffffffu, !got || *bad)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c0 = 0; c0 < NC; c0 += 16) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr + (uint32_t)(buf * NC) + ((uint32_t)(q * 32) << 16) + (uint32_t)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 16 >= NC) {   // the accumulator is read: the MMAs may have it back
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::saddr(&taken[buf])) : "memory");
        }
        if (valid) {
          if constexpr (F32) {
            float4 *o = reinterpret_cast<float4 *>(reinterpret_cast<float *>(out) + p * cout + co0 + c0);
#pragma unroll
            for (int e = 0; e < 4; e++) {
              float4 x4 = make_float4(__uint_as_float(v[4 * e]), __uint_as_float(v[4 * e + 1]),
                                      __uint_as_float(v[4 * e + 2]), __uint_as_float(v[4 * e + 3]));
              if (accum) {
                const float4 b = o[e];
                x4.x += b.x; x4.y += b.y; x4.z += b.z; x4.w += b.w;
              }
              o[e] = x4;
            }
          } else {
            uint4 *o = reinterpret_cast<uint4 *>(reinterpret_cast<bf16 *>(out) + p * cout + co0 + c0);
            const float *bs = bias + co0 + c0;
            uint32_t pk[8];
#pragma unroll
            for (int e = 0; e < 8; e++)
              pk[e] = pack_bf16(fmaxf(__uint_as_float(v[2 * e]) + bs[2 * e], 0.0f),
                                fmaxf(__uint_as_float(v[2 * e + 1]) + bs[2 * e + 1], 0.0f));
            o[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            o[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *bad) atomicExch(&g_conv_timeout, 1);
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------- weight gradient, tcgen05
// part[chunk][co][tap * cin + ci] = sum_{p in chunk} dz[p][co] x[p + tap][ci]
// as D (M x N) = A (M x K) B (K x N) on the fifth-generation tensor cores:
// M = output channels (padded to 128 with zero rows), N = a tile of the
// 9 * cin (tap, input channel) columns, K = the chunk's pixels, 16 per MMA.
// Both operands are MN-major (NHWC keeps a pixel's channels contiguous), as
// core matrices without swizzle: 8 pixels x 16 bytes (8 channels), the
// 8-channel groups 128 B apart, the two 8-pixel halves of a 16-pixel step
// all of a pixel's groups apart.  Rows of D past cout come from whatever lies
// behind A and are never read.
// Rounds of kWgRound steps go through a ring of stages: two groups of 128
// threads copy alternate rounds with cp.async (a thread one 8-channel half
// of every 16 of a pixel: the pixel's place in the image and its border tests
// once a round, no divisions) and arrive on the stage's `full` barrier when
// their copies have landed, a ninth warp issues the round's MMAs and commits
// them to its `empty` barrier; nothing else synchronises, and all waits are
// bounded.  The copies bound it: 1.2 million pixels take 113 us for 16 -> 16
// channels and 374 for 48 -> 16; 222 and 645 with one group, two stages, a
// CTA barrier a round and zeros copied into A's groups past cout.
// The chunks are summed afterwards in a fixed order (k_reduce_rows):
// training stays bit-reproducible.
constexpr int kWgRound = 4;   // 16-pixel steps per round (64 pixels)
constexpr int kWgThreads = 288;

__host__ __device__ inline int wg_tiles(int cin) { return (9 * cin + 255) / 256; }
__host__ __device__ inline int wg_cols(int cin) { return ((9 * cin + wg_tiles(cin) - 1) / wg_tiles(cin) + 15) / 16 * 16; }
__host__ __device__ inline int wg_stage_bytes(int cin, int cout) { return kWgRound * 32 * (cout + wg_cols(cin)); }
// stages: four if two CTAs then fit an SM (their accumulators take half of
// the tensor memory each), or three, or four for one CTA
__host__ __device__ inline int wg_stages(int cin, int cout) {
  const int sb = wg_stage_bytes(cin, cout), two = 112 * 1024;
  return 4 * sb <= two ? 4 : 3 * sb <= two ? 3 : 4;
}

// CIN is a template parameter: the copies' loops are by constants.
template <int CIN>
__global__ void __launch_bounds__(kWgThreads) k_wgrad_tc(const bf16 *__restrict__ dz, int cout,
                                                         const bf16 *__restrict__ x, float *__restrict__ part, int N,
                                                         int H, int W, int ppc) {
  using namespace stream_detail;
  extern __shared__ __align__(1024) unsigned char sm[];
  constexpr int cin = CIN;
  const int NT = 9 * cin, NNmax = wg_cols(cin);
  const int n0 = blockIdx.y * NNmax, NN = min(NNmax, NT - n0);   // this CTA's columns
  const int SB = wg_stage_bytes(cin, cout), S = wg_stages(cin, cout);
  uint64_t *full = reinterpret_cast<uint64_t *>(sm + S * SB), *empty = full + 4, *done = empty + 4;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  volatile int *bad = reinterpret_cast<volatile int *>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long HW = (long long)H * W, P = (long long)N * HW;
  const long long pb = (long long)blockIdx.x * ppc, pe = min(P, pb + ppc);
  const int R = (int)((pe - pb + 16 * kWgRound - 1) / (16 * kWgRound));   // rounds
  const uint32_t ncols = (uint32_t)tmem_cols(NN);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::saddr(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int k = 0; k < 4; k++) {
      mbar_init(&full[k], 128);
      mbar_init(&empty[k], 1);
    }
    mbar_init(done, 1);
    *bad = 0;
    fence_mbar_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t taddr = *tslot;
  const uint32_t sbase = tc::saddr(sm);

  if (warp < 8) {
    // ---- copies: pixel pi of the rounds rd = warp / 4, + 2, ..., channels
    // 8 * half .. of every 16
    const int half = tid & 1, pi = (tid >> 1) & 63, ks = pi >> 4, r = pi & 15;
    const uint32_t da = (uint32_t)(ks * 32 * cout + (r >> 3) * 16 * cout + half * 128 + (r & 7) * 16);
    const uint32_t db = (uint32_t)(kWgRound * 32 * cout + ks * 32 * NN + (r >> 3) * 16 * NN + half * 128 + (r & 7) * 16);
    int rd = warp >> 2;
    long long p = pb + (long long)rd * 64 + pi;
    int h = (int)((p % HW) / W), w = (int)(p % W);
    const int tap0 = n0 / cin, c0 = n0 - tap0 * cin + 8 * half;
    auto landed = [&](int round) {
      // written through the generic proxy, read by the MMAs through the async proxy
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::saddr(&full[round % S])) : "memory");
    };
    int last = -1;   // this group's round that has been copied but not announced
    for (; rd < R; rd += 2) {
      const int st = rd % S;
      if (*bad) break;
      if (rd >= S && !mbar_wait(&empty[st], (uint32_t)((rd / S - 1) & 1))) {
        *bad = 1;
        break;
      }
      const uint32_t stage = sbase + (uint32_t)(st * SB);
      const bool in = p < pe;
      const bf16 *za = in ? dz + p * cout + 8 * half : dz;
      for (int g = 0; g < cout; g += 16) tc::cp16(stage + da + (uint32_t)(g * 16), in ? za + g : dz, in);
      // bit 3 * ky + kx: the tap's pixel is inside the image
      unsigned rows = (h > 0 ? 1u : 0u) | 2u | (h + 1 < H ? 4u : 0u);
      const unsigned cols = (w > 0 ? 1u : 0u) | 2u | (w + 1 < W ? 4u : 0u);
      unsigned vm = ((rows & 1u) ? cols : 0u) | ((rows & 2u) ? cols << 3 : 0u) | ((rows & 4u) ? cols << 6 : 0u);
      if (!in) vm = 0u;
      const bf16 *xp = x + p * cin;
      if constexpr (9 * CIN <= 256) {
#pragma unroll
        for (int tap = 0; tap < 9; tap++) {
          const bool ok = vm >> tap & 1u;
          const bf16 *src = xp + ((tap / 3 - 1) * W + tap % 3 - 1) * cin + 8 * half;
#pragma unroll
          for (int c = 0; c < cin; c += 16)
            tc::cp16(stage + db + (uint32_t)((tap * cin + c) * 16), ok ? src + c : x, ok);
        }
      } else {
        int tap = tap0, c = c0, kx = tap0 % 3;
        const bf16 *src = xp + ((tap0 / 3 - 1) * W + kx - 1) * cin;
#pragma unroll 2
        for (int g = 0; g < NN; g += 16) {
          const bool ok = vm >> tap & 1u;
          tc::cp16(stage + db + (uint32_t)(g * 16), ok ? src + c : x, ok);
          c += 16;
          if (c >= cin) {
            c -= cin;
            tap++;
            kx++;
            src += cin;
            if (kx == 3) {
              kx = 0;
              src += (W - 3) * cin;
            }
          }
        }
      }
      tc::cp_commit();
      if (last >= 0) {
        tc::cp_wait<1>();
        landed(last);
      }
      last = rd;
      p += 128;
      w += 128;
      while (w >= W) {
        w -= W;
        if (++h == H) h = 0;
      }
    }
    tc::cp_wait<0>();
    if (last >= 0) landed(last);
  } else if (lane == 0) {
    // ---- MMAs.  kind::f16: FP32 accumulator, BF16 A and B, both MN-major, N = NN, M = 128
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                           ((uint32_t)(NN >> 3) << 17) | ((128u >> 4) << 24);
    for (int rd = 0; rd < R; rd++) {
      const int st = rd % S;
      if (*bad) break;
      if (!mbar_wait(&full[st], (uint32_t)((rd / S) & 1))) {
        *bad = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sa = sbase + (uint32_t)(st * SB), sb = sa + (uint32_t)(kWgRound * 32 * cout);
      for (int ks = 0; ks < kWgRound; ks++) {
        // MN-major descriptors: leading (K-half) offset, stride (8-channel group) offset 128
        const uint64_t ad = (uint64_t)(((sa + ks * 32 * cout) >> 4) & 0x3FFFu) | ((uint64_t)(uint32_t)cout << 16) |
                            ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
        const uint64_t bd = (uint64_t)(((sb + ks * NN * 32) >> 4) & 0x3FFFu) | ((uint64_t)(uint32_t)NN << 16) |
                            ((uint64_t)(128u >> 4) << 32) | (1ull << 46);
        const uint32_t acc = (rd > 0 || ks > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(taddr),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       tc::saddr(&empty[st]))
                   : "memory");
    }
    // whatever has been issued
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc::saddr(done))
                 : "memory");
  }
  __syncwarp();
  if (!mbar_wait(done, 0u)) *bad = 1;
  __syncthreads();
  const bool ok = *bad == 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok && warp < 4 && warp * 32 < cout) {   // lanes = output channels
    const int co = warp * 32 + lane;
    float *dst = part + ((long long)blockIdx.x * cout + co) * NT + n0;
    for (int c0 = 0; c0 < NN; c0 += 16) {
      uint32_t r[16];
      if (R > 0) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int i = 0; i < 16; i++) r[i] = 0u;   // an empty chunk contributes zeros
      }
      if (co < cout) {
        float4 *o = reinterpret_cast<float4 *>(dst + c0);
#pragma unroll
        for (int i = 0; i < 4; i++)
          o[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                             __uint_as_float(r[4 * i + 3]));
      }
    }
  } else if (!ok && tid == 0) {
    atomicExch(&g_conv_timeout, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Sums of partials, two sets a launch: out[i] = sum over r = 0..rows-1, in
// order, of part[r * len + i].  A block takes 32 columns: its warps fetch 128
// rows at a time into shared memory, one of them adds the rows.  (With a
// column a thread, 9 blocks of loads in turn, 437 rows of 2304 columns took
// 49 us and the 256 rows of a bias 23.)
struct RowSum {
  const float *part;
  int rows;
  long long len;
  float *out;
};
constexpr int kSumRows = 128;
__global__ void __launch_bounds__(kEw) k_reduce_rows(RowSum a, RowSum b, unsigned ablocks) {
  __shared__ float buf[2][kSumRows][32];
  const RowSum &x = blockIdx.x < ablocks ? a : b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long i = (long long)(blockIdx.x < ablocks ? blockIdx.x : blockIdx.x - ablocks) * 32 + lane;
  const bool in = i < x.len;
  auto fetch = [&](int r0, float (*to)[32]) {
#pragma unroll
    for (int k = 0; k < kSumRows / 8; k++) {
      const int r = r0 + warp + 8 * k;
      to[warp + 8 * k][lane] = in && r < x.rows ? x.part[(long long)r * x.len + i] : 0.0f;
    }
  };
  float s = 0.0f;
  fetch(0, buf[0]);
  for (int r0 = 0, k = 0; r0 < x.rows; r0 += kSumRows, k ^= 1) {
    __syncthreads();
    if (r0 + kSumRows < x.rows) fetch(r0 + kSumRows, buf[k ^ 1]);
    if (warp == 0) {
      const int m = min(kSumRows, x.rows - r0);
#pragma unroll 16
      for (int r = 0; r < m; r++) s += buf[k][r][lane];
    }
  }
  if (warp == 0 && in) x.out[i] = s;
}

// --------------------------------------------------------- elementwise parts
__global__ void k_pack3(const float *__restrict__ x3, bf16 *__restrict__ x16, long long P) {
  let_next();
  enter();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
       p += (long long)gridDim.x * blockDim.x) {
    uint4 lo, hi;
    lo.x = pack_bf16(x3[3 * p], x3[3 * p + 1]);
    lo.y = pack_bf16(x3[3 * p + 2], 0.0f);
    lo.z = lo.w = 0u;
    hi.x = hi.y = hi.z = hi.w = 0u;
    uint4 *o = reinterpret_cast<uint4 *>(x16 + p * 16);
    o[0] = lo;
    o[1] = hi;
  }
}

__global__ void k_pool(const bf16 *__restrict__ in, bf16 *__restrict__ out, int N, int H, int W,
                       int C) {
  let_next();
  enter();
  const int Ho = H / 2, Wo = W / 2, cp = C / 2;
  const long long total = (long long)N * Ho * Wo * cp;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int c = 2 * (int)(e % cp);
    long long q = e / cp;
    const int wo = (int)(q % Wo);
    q /= Wo;
    const int ho = (int)(q % Ho);
    const int n = (int)(q / Ho);
    const long long r0 = ((long long)(n * H + 2 * ho) * W + 2 * wo) * C + c;
    const long long r1 = r0 + (long long)W * C;
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(in + r0);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(in + r0 + C);
    const __nv_bfloat162 d = *reinterpret_cast<const __nv_bfloat162 *>(in + r1);
    const __nv_bfloat162 f = *reinterpret_cast<const __nv_bfloat162 *>(in + r1 + C);
    const float lo = (((__low2float(a) + __low2float(b)) + __low2float(d)) + __low2float(f)) * 0.25f;
    const float hi = (((__high2float(a) + __high2float(b)) + __high2float(d)) + __high2float(f)) * 0.25f;
    reinterpret_cast<uint32_t *>(out)[(((long long)(n * Ho + ho) * Wo + wo) * C + c) / 2] = pack_bf16(lo, hi);
  }
}

// 8 channels of a pixel: 16 bytes BF16, 32 bytes FP32
struct alignas(16) F8 {
  float4 a, b;
};
__device__ __forceinline__ F8 ld8(const float *p) {
  return {*reinterpret_cast<const float4 *>(p), *reinterpret_cast<const float4 *>(p + 4)};
}
__device__ __forceinline__ float lo_f(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi_f(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

// cat[n][h][w] = (low[n][h/2][w/2][0..C1), skip[n][h][w][0..C2)), 16 bytes a
// thread, an image row a blockIdx.y
__global__ void __launch_bounds__(kRowThreads)
k_upcat(const bf16 *__restrict__ low, int C1, const bf16 *__restrict__ skip, int C2, bf16 *__restrict__ cat, int H,
        int W) {
  let_next();
  enter();
  const int g1 = C1 / 8, g2 = C2 / 8, gt = g1 + g2;
  const int e = blockIdx.x * kRowThreads + threadIdx.x, row = blockIdx.y;
  if (e >= W * gt) return;
  const int w = e / gt, g = e - w * gt, n = row / H, h = row - n * H;
  const uint4 *src = g < g1 ? reinterpret_cast<const uint4 *>(low) +
                                  ((long long)(n * (H / 2) + h / 2) * (W / 2) + w / 2) * g1 + g
                            : reinterpret_cast<const uint4 *>(skip) + ((long long)row * W + w) * g2 + g - g1;
  reinterpret_cast<uint4 *>(cat)[(long long)row * W * gt + e] = *src;
}

// ReLU gradient of a layer, rounded to BF16 for the tensor-core products:
// dz = y > 0 ? dY : 0, 8 channels a thread, an image row a blockIdx.y.  Where
// dY is a plain function of other gradients it is formed here and never
// stored: kPlain: a is dY; kLow: the four fine gradients (a: dcat, of Ct
// channels) of an upsampled pixel; kSkip: the skip's share of a concatenation
// (channels C1.. of a) plus a quarter of the pooled gradient b; kOut: the
// output layer's, a[pixel] times b[channel].
enum { kPlain, kLow, kSkip, kOut };
template <int MODE>
__global__ void __launch_bounds__(kRowThreads)
k_relu_mask(const float *__restrict__ a, const float *__restrict__ b, int Ct, int C1, const bf16 *__restrict__ y,
            bf16 *__restrict__ dz, int H, int W, int C) {
  const int g8 = C / 8, e = blockIdx.x * kRowThreads + threadIdx.x, row = blockIdx.y;
  if (e >= W * g8) return;
  const int w = e / g8, c = (e - w * g8) * 8;
  const long long p = (long long)row * W + w;
  float v[8];
  auto put = [&](const F8 &x) {
    v[0] = x.a.x; v[1] = x.a.y; v[2] = x.a.z; v[3] = x.a.w;
    v[4] = x.b.x; v[5] = x.b.y; v[6] = x.b.z; v[7] = x.b.w;
  };
  auto add = [&](const F8 &x) {
    v[0] += x.a.x; v[1] += x.a.y; v[2] += x.a.z; v[3] += x.a.w;
    v[4] += x.b.x; v[5] += x.b.y; v[6] += x.b.z; v[7] += x.b.w;
  };
  if constexpr (MODE == kPlain) {
    put(ld8(a + p * C + c));
  } else if constexpr (MODE == kLow) {
    // pixel rows of the fine grid are 2 * row and the next: 2 n H + 2 h
    const float *r0 = a + (((long long)row * 2) * (2 * W) + 2 * w) * Ct + c, *r1 = r0 + (long long)2 * W * Ct;
    put(ld8(r0));
    add(ld8(r0 + Ct));
    add(ld8(r1));
    add(ld8(r1 + Ct));
  } else if constexpr (MODE == kSkip) {
    const int n = row / H, h = row - n * H;
    put(ld8(a + p * Ct + C1 + c));
    F8 q = ld8(b + ((long long)(n * (H / 2) + h / 2) * (W / 2) + w / 2) * C + c);
    q.a.x *= 0.25f; q.a.y *= 0.25f; q.a.z *= 0.25f; q.a.w *= 0.25f;
    q.b.x *= 0.25f; q.b.y *= 0.25f; q.b.z *= 0.25f; q.b.w *= 0.25f;
    add(q);
  } else {
    const float d = a[p];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = d * b[c + k];
  }
  const uint4 m = *reinterpret_cast<const uint4 *>(y + p * C + c);
  uint4 o;
  o.x = pack_bf16(lo_f(m.x) > 0.0f ? v[0] : 0.0f, hi_f(m.x) > 0.0f ? v[1] : 0.0f);
  o.y = pack_bf16(lo_f(m.y) > 0.0f ? v[2] : 0.0f, hi_f(m.y) > 0.0f ? v[3] : 0.0f);
  o.z = pack_bf16(lo_f(m.z) > 0.0f ? v[4] : 0.0f, hi_f(m.z) > 0.0f ? v[5] : 0.0f);
  o.w = pack_bf16(lo_f(m.w) > 0.0f ? v[6] : 0.0f, hi_f(m.w) > 0.0f ? v[7] : 0.0f);
  *reinterpret_cast<uint4 *>(dz + p * C + c) = o;
}

// y[p] = b + sum_c w[c] u[p][c]   (FP32)
__global__ void k_out_fwd(const bf16 *__restrict__ u, const float *__restrict__ w,
                          const float *__restrict__ b, float *__restrict__ y, long long P, int C) {
  let_next();
  enter();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
       p += (long long)gridDim.x * blockDim.x) {
    float s = 0.0f;
    for (int c = 0; c < C; c += 8) {
      const uint4 v = *reinterpret_cast<const uint4 *>(u + p * C + c);
      s = fmaf(w[c], lo_f(v.x), s);
      s = fmaf(w[c + 1], hi_f(v.x), s);
      s = fmaf(w[c + 2], lo_f(v.y), s);
      s = fmaf(w[c + 3], hi_f(v.y), s);
      s = fmaf(w[c + 4], lo_f(v.z), s);
      s = fmaf(w[c + 5], hi_f(v.z), s);
      s = fmaf(w[c + 6], lo_f(v.w), s);
      s = fmaf(w[c + 7], hi_f(v.w), s);
    }
    y[p] = s + b[0];
  }
}

// part[slot][c] = sum over the slot's pixels of a[p][c] * (WGT ? wgt[p] : 1):
// slot s of kRedBlocks has `runs` = kEw / C runs, run k the pixels
// s * runs + k, + kRedBlocks * runs, ..., added in order and then run by run.
// 8 channels a thread and 16 loads in flight; the slots are summed by
// k_reduce_rows.  39 MB (16 channels of 480 x 160 x 16 pixels) in 2-byte loads
// took 78 us.
template <bool WGT>
__global__ void __launch_bounds__(kDotThreads) k_chan_dot(const bf16 *__restrict__ a, const float *__restrict__ wgt,
                                                          long long P, int C, float *__restrict__ part) {
  __shared__ float red[kEw];   // [run][C]: C * runs <= kEw
  const int g8 = C / 8, runs = kEw / C, run = threadIdx.x / g8, c = (threadIdx.x - run * g8) * 8;
  if (run < runs) {
    float s[8] = {};
    const long long step = (long long)gridDim.x * runs;
    constexpr int kDeep = 16;
    for (long long p0 = (long long)blockIdx.x * runs + run; p0 < P; p0 += kDeep * step) {
      uint4 v[kDeep];
      float f[kDeep];
#pragma unroll
      for (int k = 0; k < kDeep; k++) {
        const long long p = p0 + k * step;
        v[k] = p < P ? *reinterpret_cast<const uint4 *>(a + p * C + c) : make_uint4(0u, 0u, 0u, 0u);
        f[k] = WGT && p < P ? wgt[p] : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < kDeep; k++) {
        if (p0 + k * step >= P) break;
        const uint32_t q[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
        for (int h = 0; h < 4; h++) {
          s[2 * h] = WGT ? fmaf(lo_f(q[h]), f[k], s[2 * h]) : s[2 * h] + lo_f(q[h]);
          s[2 * h + 1] = WGT ? fmaf(hi_f(q[h]), f[k], s[2 * h + 1]) : s[2 * h + 1] + hi_f(q[h]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 8; k++) red[run * C + c + k] = s[k];
  }
  __syncthreads();
  for (int k = threadIdx.x; k < C; k += kDotThreads) {
    float t = 0.0f;
    for (int r = 0; r < runs; r++) t += red[r * C + k];
    part[(long long)blockIdx.x * C + k] = t;
  }
}

// part[block] = the block's sum of a (fixed order)
__global__ void k_sum(const float *__restrict__ a, long long n, float *__restrict__ part) {
  __shared__ float red[kEw / 32];
  float s = 0.0f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    s += a[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < kEw / 32; w++) t += red[w];
    part[blockIdx.x] = t;
  }
}

// dy = scale (y - t); loss += (y - t)^2 (FP64)
__global__ void k_mse(const float *__restrict__ y, const float *__restrict__ t, float *__restrict__ dy,
                      long long P, float scale, double *__restrict__ loss) {
  double s = 0.0;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P;
       p += (long long)gridDim.x * blockDim.x) {
    const float r = y[p] - t[p];
    dy[p] = scale * r;
    s += (double)r * r;
  }
  // one addition to the loss a block
  __shared__ double red[kEw / 32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kEw / 32; w++) s += red[w];
    atomicAdd(loss, s);
  }
}

// wt[ci][tap][co] = w[co][8 - tap][ci]: the data gradient as a forward conv
__global__ void k_flip(const bf16 *__restrict__ w, bf16 *__restrict__ wt, int cout, int cin) {
  const long long total = (long long)cout * 9 * cin;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int co = (int)(e % cout);
    const long long q = e / cout;
    const int tap = (int)(q % 9);
    const int ci = (int)(q / 9);
    wt[e] = w[((long long)co * 9 + (8 - tap)) * cin + ci];
  }
}

__global__ void k_adam(float *__restrict__ p, float *__restrict__ m, float *__restrict__ v,
                       const float *__restrict__ g, long long n, float lr_t, float b1, float b2,
                       float eps) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr_t * mi / (sqrtf(vi) + eps);
  }
}

__global__ void k_to_bf16(const float *__restrict__ a, bf16 *__restrict__ b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    b[i] = __float2bfloat16_rn(a[i]);
}

// Interior statistics, per block: part[block][0..3] = sum a^2, sum b,
// sum b^2, max c (c >= 0); the block that ends last adds them in block order
// into s[0..3], one thread a sum (a launch of its own, one thread for all of
// them, took 41 us), and leaves `done` at zero.
__global__ void k_stats(const float *__restrict__ a, const float *__restrict__ b,
                        const float *__restrict__ c, int nzpad, int x0, int z0, int nx, int nz,
                        double *__restrict__ part, double *__restrict__ s, unsigned *__restrict__ done) {
  double sa = 0, sb = 0, sb2 = 0, mc = 0;
  const long long total = (long long)nx * nz;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(e / nz), iz = (int)(e - (long long)ix * nz);
    const long long q = (long long)(x0 + ix) * nzpad + z0 + iz;
    if (a) sa += (double)a[q] * a[q];
    if (b) { sb += b[q]; sb2 += (double)b[q] * b[q]; }
    if (c) mc = fmax(mc, (double)fmaxf(c[q], 0.0f));
  }
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_down_sync(0xffffffffu, sa, o);
    sb += __shfl_down_sync(0xffffffffu, sb, o);
    sb2 += __shfl_down_sync(0xffffffffu, sb2, o);
    mc = fmax(mc, __shfl_down_sync(0xffffffffu, mc, o));
  }
  __shared__ double red[kEw / 32][4];
  __shared__ bool last;
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = sa;
    red[threadIdx.x >> 5][1] = sb;
    red[threadIdx.x >> 5][2] = sb2;
    red[threadIdx.x >> 5][3] = mc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t0 = 0, t1 = 0, t2 = 0, t3 = 0;
    for (int w = 0; w < kEw / 32; w++) {
      t0 += red[w][0];
      t1 += red[w][1];
      t2 += red[w][2];
      t3 = fmax(t3, red[w][3]);
    }
    part[4 * blockIdx.x] = t0;
    part[4 * blockIdx.x + 1] = t1;
    part[4 * blockIdx.x + 2] = t2;
    part[4 * blockIdx.x + 3] = t3;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double all[4 * kEw];
  for (int i = threadIdx.x; i < 4 * kEw; i += kEw) all[i] = i < 4 * (int)gridDim.x ? __ldcg(part + i) : 0.0;
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0;
    for (int i = 0; i < (int)gridDim.x; i++) {
      const double v = all[4 * i + threadIdx.x];
      t = threadIdx.x == 3 ? fmax(t, v) : t + v;
    }
    s[threadIdx.x] = t;
  }
  if (threadIdx.x == 0) *done = 0;
}

__global__ void k_features(const float *__restrict__ gr, const float *__restrict__ vel,
                           const float *__restrict__ il, int nzpad, int x0, int z0, int nx, int nz,
                           int Hp, int Wp, const double *__restrict__ s, float *__restrict__ x3) {
  let_next();
  enter();
  const double cnt = (double)nx * nz;
  const double rms = sqrt(s[0] / cnt);
  const double mean = s[1] / cnt;
  const double var = fmax(s[2] / cnt - mean * mean, 0.0);
  const double sd = sqrt(var);
  const double imax = s[3];
  const long long total = (long long)Hp * Wp;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int h = (int)(e / Wp), w = (int)(e - (long long)h * Wp);
    float f0 = 0, f1 = 0, f2 = 0;
    if (h < nx && w < nz) {
      const long long q = (long long)(x0 + h) * nzpad + z0 + w;
      if (rms > 0) f0 = (float)(gr[q] / rms);
      if (sd > 0) f1 = (float)((vel[q] - mean) / sd);
      if (il && imax > 0) f2 = (log10f((float)(fmaxf(il[q], 0.0f) / imax) + 1e-6f) + 3.0f) / 3.0f;
    }
    x3[3 * e] = f0;
    x3[3 * e + 1] = f1;
    x3[3 * e + 2] = f2;
  }
}

__global__ void k_target(const float *__restrict__ dv, int nzpad, int x0, int z0, int nx, int nz,
                         int Hp, int Wp, const double *__restrict__ s, float *__restrict__ t) {
  const double rms = sqrt(s[0] / ((double)nx * nz));
  const long long total = (long long)Hp * Wp;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int h = (int)(e / Wp), w = (int)(e - (long long)h * Wp);
    float v = 0;
    if (h < nx && w < nz && rms > 0) v = (float)(dv[(long long)(x0 + h) * nzpad + z0 + w] / rms);
    t[e] = v;
  }
}

// the whole padded grid: y in the interior, zeros around it
__global__ void k_scatter(const float *__restrict__ y, int nxpad, int nzpad, int x0, int z0, int nx, int nz,
                          int Wp, float *__restrict__ dir) {
  let_next();
  enter();
  const long long total = (long long)nxpad * nzpad;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e / nzpad), ix = x - x0, iz = (int)(e - (long long)x * nzpad) - z0;
    dir[e] = ix >= 0 && ix < nx && iz >= 0 && iz < nz ? y[(long long)ix * Wp + iz] : 0.0f;
  }
}

__global__ void k_illum(float *__restrict__ illum, const float *__restrict__ p, long long fstride,
                        int n, int nxpad, int nzpad, int pitch) {
  const long long total = (long long)nxpad * nzpad;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(e / nzpad), z = (int)(e - (long long)x * nzpad);
    float s = 0.0f;
    for (int j = 0; j < n; j++) {
      const float v = p[j * fstride + (long long)x * pitch + z];
      s = fmaf(v, v, s);
    }
    illum[e] += s;
  }
}

// Dynamic shared memory of a launch: two stages, the barriers, the tensor
// memory address and the decoded pixels -- raised where needed so that no
// more CTAs are resident on an SM than its 512 tensor-memory columns hold
// (a CTA that cannot allocate would wait inside tcgen05.alloc).
size_t conv_tc_smem(int cin, int cout) {
  const int T = tc::taps_per_round(cin, cout);
  const size_t need = (T == 9 ? 1 : 2) * (size_t)tc::stage_bytes(cin, cout, T) + 32;
  const int fit = 512 / tmem_cols(cout);   // CTAs whose accumulators fit
  if (fit >= 16) return need;                 // 16 CTAs of 128 threads fill an SM
  const size_t sm_bytes = 228 * 1024, reserve = 1024;   // per SM, per CTA
  const size_t cap = sm_bytes / (fit + 1) - reserve + 16;   // fit + 1 CTAs no longer fit
  return std::max(need, cap);
}

template <bool F32>
void conv_tc_go(const bf16 *in, int cin, const bf16 *w, const float *bias, void *out, bool accum, int cout,
                int N, int H, int W, cudaStream_t st) {
  static const bool attr = [] {
    SWFWI_CUDA(cudaFuncSetAttribute(k_conv3x3_tc<F32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)conv_tc_smem(128, 256)));   // the largest accepted widths
    return true;
  }();
  (void)attr;
  const long long P = (long long)N * H * W;
  k_conv3x3_tc<F32><<<(unsigned)((P + 127) / 128), 128, conv_tc_smem(cin, cout), st>>>(
      in, cin, w, bias, out, accum ? 1 : 0, cout, N, H, W);
  noted();
}

constexpr int kRedBlocks = 256;           // blocks of the channel sums

void reduce_rows(const RowSum &a, const RowSum &b, cudaStream_t st) {
  const unsigned na = (unsigned)((a.len + 31) / 32), nb = b.rows ? (unsigned)((b.len + 31) / 32) : 0;
  k_reduce_rows<<<na + nb, kEw, 0, st>>>(a, b, na);
  noted();
}

// Pixels per chunk of a weight gradient: a multiple of one round (64), about
// 444 CTAs (3 per SM) over the column tiles.
long long wgrad_pix_per_chunk(long long P, int cin) {
  const long long chunks = std::max(1, 444 / wg_tiles(cin));
  return 64 * std::max(1LL, (P + 64 * chunks - 1) / (64 * chunks));
}

size_t wgrad_tc_smem(int cin, int cout) {
  const size_t need = (size_t)wg_stages(cin, cout) * wg_stage_bytes(cin, cout) + 9 * 8 + 8;
  const int fit = 512 / tmem_cols(wg_cols(cin));   // CTAs whose accumulators fit
  const size_t cap = 228 * 1024 / (fit + 1) - 1024 + 16;   // fit + 1 CTAs no longer fit
  return std::max(need, cap);
}

template <int CIN>
void wgrad_tc_cin(const bf16 *dz, int cout, const bf16 *x, float *part, int N, int H, int W, long long ppc,
                  unsigned chunks, cudaStream_t st) {
  static const bool attr = [] {
    SWFWI_CUDA(cudaFuncSetAttribute(k_wgrad_tc<CIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    227 * 1024));
    return true;
  }();
  (void)attr;
  dim3 grid(chunks, wg_tiles(CIN));
  k_wgrad_tc<CIN><<<grid, kWgThreads, wgrad_tc_smem(CIN, cout), st>>>(dz, cout, x, part, N, H, W, (int)ppc);
}

// bias: partials of the bias gradient to sum in the same launch (rows 0: none)
void wgrad_tc_go(const bf16 *dz, int cout, const bf16 *x, int cin, float *dw, float *part, const RowSum &bias, int N,
                 int H, int W, cudaStream_t st) {
  const long long P = (long long)N * H * W;
  const long long ppc = wgrad_pix_per_chunk(P, cin);
  const unsigned chunks = (unsigned)((P + ppc - 1) / ppc);
  switch (cin) {
    case 16: wgrad_tc_cin<16>(dz, cout, x, part, N, H, W, ppc, chunks, st); break;
    case 32: wgrad_tc_cin<32>(dz, cout, x, part, N, H, W, ppc, chunks, st); break;
    case 48: wgrad_tc_cin<48>(dz, cout, x, part, N, H, W, ppc, chunks, st); break;
    case 64: wgrad_tc_cin<64>(dz, cout, x, part, N, H, W, ppc, chunks, st); break;
    case 96: wgrad_tc_cin<96>(dz, cout, x, part, N, H, W, ppc, chunks, st); break;
    case 128: wgrad_tc_cin<128>(dz, cout, x, part, N, H, W, ppc, chunks, st); break;
    default: throw Error(SWFWI_ERR_BAD_ARG, "weight gradient: input width must be 16/32/48/64/96/128");
  }
  noted();
  reduce_rows({part, (int)chunks, (long long)cout * 9 * cin, dw}, bias, st);
}

// Partial channel sums of a (times wgt, if given) for out[C], in a fixed order.
RowSum chan_sum(const bf16 *a, const float *wgt, long long P, int C, float *out, float *part, cudaStream_t st) {
  if (wgt) k_chan_dot<true><<<kRedBlocks, kDotThreads, 0, st>>>(a, wgt, P, C, part);
  else k_chan_dot<false><<<kRedBlocks, kDotThreads, 0, st>>>(a, nullptr, P, C, part);
  noted();
  return {part, kRedBlocks, C, out};
}

int roundup8(int v) { return (v + 7) / 8 * 8; }

// grid of the kernels that take an image row a blockIdx.y, 8 of C channels a thread
dim3 row_grid(int C, int rows, int W) {
  return dim3((unsigned)((W * (C / 8) + kRowThreads - 1) / kRowThreads), (unsigned)rows);
}

}  // namespace

template <bool F32, int KC>
void conv_tg_kc(const bf16 *in, const bf16 *w, const float *bias, void *out, bool accum, int cout, int N, int H,
                int W, cudaStream_t st) {
  static const bool attr = [] {
    SWFWI_CUDA(cudaFuncSetAttribute(k_conv3x3_tg<F32, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    227 * 1024));
    return true;
  }();
  (void)attr;
  const long long tiles = ((long long)N * H * ((W + 7) / 8) + 15) / 16;
  const size_t smem = tg::launch_smem(16 * KC, cout);
  const int halves = cout / tg::cols(16 * KC, cout);
  const long long ctas = std::max(1LL, (smem <= 112 * 1024 ? 296LL : 148LL) / halves);   // one or two an SM
  // tiles evenly over the CTAs
  const long long per = (tiles + ctas - 1) / ctas;
  launch_after(k_conv3x3_tg<F32, KC>, dim3((unsigned)((tiles + per - 1) / per), (unsigned)halves), tg::kThreads, smem,
               st, in, w, bias, out, accum ? 1 : 0, cout, N, H, W);
}

// true when a row-tile kernel exists for cin
template <bool F32>
bool conv_tg_go(const bf16 *in, int cin, const bf16 *w, const float *bias, void *out, bool accum, int cout,
                int N, int H, int W, cudaStream_t st) {
  switch (cin / 16) {
    case 1: conv_tg_kc<F32, 1>(in, w, bias, out, accum, cout, N, H, W, st); return true;
    case 2: conv_tg_kc<F32, 2>(in, w, bias, out, accum, cout, N, H, W, st); return true;
    case 3: conv_tg_kc<F32, 3>(in, w, bias, out, accum, cout, N, H, W, st); return true;
    case 4: conv_tg_kc<F32, 4>(in, w, bias, out, accum, cout, N, H, W, st); return true;
    case 6: conv_tg_kc<F32, 6>(in, w, bias, out, accum, cout, N, H, W, st); return true;
    case 8: conv_tg_kc<F32, 8>(in, w, bias, out, accum, cout, N, H, W, st); return true;
    default: return false;
  }
}

void launch_conv3x3(const bf16 *in, int cin, const bf16 *w, const float *bias, void *out,
                    bool out_f32, bool accum, int cout, int N, int H, int W, cudaStream_t st) {
  SWFWI_REQUIRE(cin > 0 && cin % 16 == 0 && cin <= 128 && cout > 0 && cout % 16 == 0 && cout <= 256,
                "conv widths must be multiples of 16, at most 128 in and 256 out");
  SWFWI_REQUIRE(N > 0 && H > 0 && W > 0, "conv image size out of range");
  SWFWI_REQUIRE(out_f32 || bias, "BF16 conv output needs a bias");
  // row tiles (each input row staged once) where weights, two stages and two
  // accumulators fit, and their group index 32 bits; else the pixel-run tiles
  const bool rows = tg::fits(cin, cout) && (long long)N * H * ((W + 7) / 8) < (1LL << 31) - 32;
  if (out_f32) {
    if (!(rows && conv_tg_go<true>(in, cin, w, bias, out, accum, cout, N, H, W, st)))
      conv_tc_go<true>(in, cin, w, bias, out, accum, cout, N, H, W, st);
  } else {
    if (!(rows && conv_tg_go<false>(in, cin, w, bias, out, false, cout, N, H, W, st)))
      conv_tc_go<false>(in, cin, w, bias, out, false, cout, N, H, W, st);
  }
}

size_t conv3x3_wgrad_scratch(int cout, int cin, int N, int H, int W) {
  const long long P = (long long)N * H * W;
  const long long ppc = wgrad_pix_per_chunk(P, cin);
  return (size_t)((P + ppc - 1) / ppc) * cout * 9 * cin;
}

void launch_conv3x3_wgrad(const bf16 *dz, int cout, const bf16 *x, int cin, float *dw, float *scratch,
                          size_t scratch_floats, int N, int H, int W, cudaStream_t st) {
  SWFWI_REQUIRE(cout > 0 && cout % 16 == 0 && cout <= 128, "weight gradient: output width must be a multiple of 16, at most 128");
  SWFWI_REQUIRE(cin == 16 || cin == 32 || cin == 48 || cin == 64 || cin == 96 || cin == 128,
                "weight gradient: input width must be 16/32/48/64/96/128");
  SWFWI_REQUIRE(scratch && scratch_floats >= conv3x3_wgrad_scratch(cout, cin, N, H, W),
                "weight gradient scratch too small");
  wgrad_tc_go(dz, cout, x, cin, dw, scratch, RowSum{}, N, H, W, st);
}

void launch_illum_accum(float *illum, const float *p, long long fstride, int n, int nxpad, int nzpad,
                        int pitch, cudaStream_t st) {
  const long long total = (long long)nxpad * nzpad;
  k_illum<<<blocks_for(total), kEw, 0, st>>>(illum, p, fstride, n, nxpad, nzpad, pitch);
  noted();
}

// ------------------------------------------------------------------ network
Preconditioner::Preconditioner(const int widths[4]) {
  for (int i = 0; i < 4; i++) {
    SWFWI_REQUIRE(widths[i] > 0 && widths[i] % 16 == 0 && widths[i] <= 64,
                  "preconditioner widths must be multiples of 16 up to 64");
    w_[i] = widths[i];
  }
  const int c0 = w_[0], c1 = w_[1], c2 = w_[2], c3 = w_[3];
  const int io[kConvs][2] = {{kInCh, c0}, {c0, c0}, {c0, c1}, {c1, c1}, {c1, c2},
                             {c2, c2},    {c2, c3}, {c3, c3}, {c3 + c2, c2}, {c2, c2},
                             {c2 + c1, c1}, {c1, c1}, {c1 + c0, c0}, {c0, c0}};
  long long off = 0;
  size_t maxw = 0;
  for (int l = 0; l < kConvs; l++) {
    ConvSpec s{io[l][0], io[l][1], 0, 0};
    s.w_off = off;
    off += (long long)s.cout * 9 * s.cin;
    s.b_off = off;
    off += s.cout;
    maxw = std::max(maxw, (size_t)s.cout * 9 * s.cin);
    conv_.push_back(s);
  }
  out_w_ = off;
  off += c0;
  out_b_ = off;
  off += 1;
  nparam_ = off;
  params_.resize(nparam_);
  grads_.resize(nparam_);
  m_.resize(nparam_);
  v_.resize(nparam_);
  wbf_.resize(nparam_);
  wflip_.resize(maxw);
  red_.resize(8 + 4 * 256);   // loss, statistics and their per-block partials
  done_.resize(1);
  done_.zero(st_);
  // He-uniform conv weights, zero biases, small output layer (seeded)
  std::vector<float> h(nparam_, 0.0f);
  std::mt19937 gen(12345u);
  for (const ConvSpec &s : conv_) {
    const float lim = std::sqrt(6.0f / (9.0f * s.cin));
    std::uniform_real_distribution<float> U(-lim, lim);
    for (long long i = 0; i < (long long)s.cout * 9 * s.cin; i++) h[s.w_off + i] = U(gen);
  }
  {
    const float lim = 1.0f / std::sqrt((float)c0);
    std::uniform_real_distribution<float> U(-lim, lim);
    for (int i = 0; i < c0; i++) h[out_w_ + i] = U(gen);
  }
  set_params(h.data());
}

void Preconditioner::refresh_bf16() {
  k_to_bf16<<<blocks_for(nparam_), kEw, 0, st_>>>(params_.get(), wbf_.get(), nparam_);
  noted();
}

void Preconditioner::set_params(const float *host) {
  SWFWI_REQUIRE(host, "null parameters");
  params_.upload(host, nparam_, st_);
  refresh_bf16();
  reset_optimizer();
}

void Preconditioner::reset_optimizer() {
  m_.zero(st_);
  v_.zero(st_);
  grads_.zero(st_);
  step_ = 0;
  SWFWI_CUDA(cudaStreamSynchronize(st_));
}

void Preconditioner::get_params(float *host) {
  SWFWI_CUDA(cudaMemcpyAsync(host, params_.get(), sizeof(float) * nparam_, cudaMemcpyDeviceToHost, st_));
  SWFWI_CUDA(cudaStreamSynchronize(st_));
}

void Preconditioner::get_grads(float *host) {
  SWFWI_CUDA(cudaMemcpyAsync(host, grads_.get(), sizeof(float) * nparam_, cudaMemcpyDeviceToHost, st_));
  SWFWI_CUDA(cudaStreamSynchronize(st_));
}

void Preconditioner::conv_fwd(int l, const bf16 *in, bf16 *out, long long, int H, int W) {
  const ConvSpec &s = conv_[l];
  launch_conv3x3(in, s.cin, wbf_.get() + s.w_off, params_.get() + s.b_off, out, false, false, s.cout,
                 N_, H, W, st_);
}

void Preconditioner::forward(const float *x, float *y, int N, int H, int W) {
  SWFWI_REQUIRE(x && N > 0 && H > 0 && W > 0 && H % 8 == 0 && W % 8 == 0,
                "network input must be N x H x W with H and W multiples of 8");
  SWFWI_REQUIRE((long long)N * H <= 65535, "network batch too large");
  N_ = N;
  H_ = H;
  W_ = W;
  const int c0 = w_[0], c1 = w_[1], c2 = w_[2], c3 = w_[3];
  const long long P0 = (long long)N * H * W, P1 = P0 / 4, P2 = P0 / 16, P3 = P0 / 64;
  x16_.resize(P0 * kInCh);
  a0_.resize(P0 * c0); s0_.resize(P0 * c0); p0_.resize(P1 * c0);
  a1_.resize(P1 * c1); s1_.resize(P1 * c1); p1_.resize(P2 * c1);
  a2_.resize(P2 * c2); s2_.resize(P2 * c2); p2_.resize(P3 * c2);
  a3_.resize(P3 * c3); b3_.resize(P3 * c3);
  cat2_.resize(P2 * (c3 + c2)); a4_.resize(P2 * c2); u2_.resize(P2 * c2);
  cat1_.resize(P1 * (c2 + c1)); a5_.resize(P1 * c1); u1_.resize(P1 * c1);
  cat0_.resize(P0 * (c1 + c0)); a6_.resize(P0 * c0); u0_.resize(P0 * c0);
  y_.resize(P0);
  launch_after(k_pack3, blocks_for(P0), kEw, 0, st_, x, x16_.get(), P0);
  const int H1 = H / 2, W1 = W / 2, H2 = H / 4, W2 = W / 4, H3 = H / 8, W3 = W / 8;
  conv_fwd(0, x16_.get(), a0_.get(), P0, H, W);
  conv_fwd(1, a0_.get(), s0_.get(), P0, H, W);
  launch_after(k_pool, blocks_for(P1 * c0 / 2), kEw, 0, st_, s0_.get(), p0_.get(), N, H, W, c0);
  conv_fwd(2, p0_.get(), a1_.get(), P1, H1, W1);
  conv_fwd(3, a1_.get(), s1_.get(), P1, H1, W1);
  launch_after(k_pool, blocks_for(P2 * c1 / 2), kEw, 0, st_, s1_.get(), p1_.get(), N, H1, W1, c1);
  conv_fwd(4, p1_.get(), a2_.get(), P2, H2, W2);
  conv_fwd(5, a2_.get(), s2_.get(), P2, H2, W2);
  launch_after(k_pool, blocks_for(P3 * c2 / 2), kEw, 0, st_, s2_.get(), p2_.get(), N, H2, W2, c2);
  conv_fwd(6, p2_.get(), a3_.get(), P3, H3, W3);
  conv_fwd(7, a3_.get(), b3_.get(), P3, H3, W3);
  launch_after(k_upcat, row_grid(c3 + c2, N * H2, W2), kRowThreads, 0, st_,
               b3_.get(), c3, s2_.get(), c2, cat2_.get(), H2, W2);
  conv_fwd(8, cat2_.get(), a4_.get(), P2, H2, W2);
  conv_fwd(9, a4_.get(), u2_.get(), P2, H2, W2);
  launch_after(k_upcat, row_grid(c2 + c1, N * H1, W1), kRowThreads, 0, st_,
               u2_.get(), c2, s1_.get(), c1, cat1_.get(), H1, W1);
  conv_fwd(10, cat1_.get(), a5_.get(), P1, H1, W1);
  conv_fwd(11, a5_.get(), u1_.get(), P1, H1, W1);
  launch_after(k_upcat, row_grid(c1 + c0, N * H, W), kRowThreads, 0, st_,
               u1_.get(), c1, s0_.get(), c0, cat0_.get(), H, W);
  conv_fwd(12, cat0_.get(), a6_.get(), P0, H, W);
  conv_fwd(13, a6_.get(), u0_.get(), P0, H, W);
  launch_after(k_out_fwd, blocks_for(P0), kEw, 0, st_, u0_.get(), params_.get() + out_w_, params_.get() + out_b_,
                                              y_.get(), P0, c0);
  if (y) SWFWI_CUDA(cudaMemcpyAsync(y, y_.get(), sizeof(float) * P0, cudaMemcpyDeviceToDevice, st_));
}

template <int MODE>
void Preconditioner::conv_bwd(int l, const bf16 *in, const bf16 *out, const float *a, const float *b, int Ct, int C1,
                              float *dX, int H, int W) {
  const ConvSpec &s = conv_[l];
  const long long P = (long long)N_ * H * W;
  k_relu_mask<MODE><<<row_grid(s.cout, N_ * H, W), kRowThreads, 0, st_>>>(a, b, Ct, C1, out, dz_.get(), H, W, s.cout);
  noted();
  const RowSum bias = chan_sum(dz_.get(), nullptr, P, s.cout, grads_.get() + s.b_off, bpart_.get(), st_);
  wgrad_tc_go(dz_.get(), s.cout, in, s.cin, grads_.get() + s.w_off, part_.get(), bias, N_, H, W, st_);
  if (dX) {
    k_flip<<<blocks_for((long long)s.cout * 9 * s.cin), kEw, 0, st_>>>(wbf_.get() + s.w_off, wflip_.get(),
                                                                        s.cout, s.cin);
    noted();
    launch_conv3x3(dz_.get(), s.cout, wflip_.get(), nullptr, dX, true, false, s.cin, N_, H, W, st_);
  }
}

double Preconditioner::backward(const float *t) {
  SWFWI_REQUIRE(t && N_ > 0, "backward needs a forward and a target");
  const int N = N_, H = H_, W = W_;
  const int c0 = w_[0], c1 = w_[1], c2 = w_[2], c3 = w_[3];
  const long long P0 = (long long)N * H * W, P1 = P0 / 4, P2 = P0 / 16, P3 = P0 / 64;
  const int H1 = H / 2, W1 = W / 2, H2 = H / 4, W2 = W / 4, H3 = H / 8, W3 = W / 8;
  const long long big = std::max({P0 * c0, P1 * std::max(c0, c1), P2 * std::max(c1, c2), P3 * std::max(c2, c3)});
  dy_.resize(P0);
  dA_.resize(big);
  dCat0_.resize(P0 * (c1 + c0));
  dCat1_.resize(P1 * (c2 + c1));
  dCat2_.resize(P2 * (c3 + c2));
  dz_.resize(big);
  bpart_.resize((size_t)kRedBlocks * 64);
  size_t need = kRedBlocks;
  {
    const int hw[4][2] = {{H, W}, {H1, W1}, {H2, W2}, {H3, W3}};
    const int level[kConvs] = {0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0};
    for (int l = 0; l < kConvs; l++)
      need = std::max(need, conv3x3_wgrad_scratch(conv_[l].cout, conv_[l].cin, N, hw[level[l]][0],
                                                  hw[level[l]][1]));
  }
  part_.resize(need);
  grads_.zero(st_);
  red_.zero(st_);
  k_mse<<<(unsigned)std::min<long long>(blocks_for(P0), 592), kEw, 0, st_>>>(y_.get(), t, dy_.get(), P0,
                                                                             2.0f / (float)P0, red_.get());
  noted();
  // output layer
  k_sum<<<kRedBlocks, kEw, 0, st_>>>(dy_.get(), P0, part_.get());
  noted();
  reduce_rows({part_.get(), kRedBlocks, 1, grads_.get() + out_b_},
              chan_sum(u0_.get(), dy_.get(), P0, c0, grads_.get() + out_w_, bpart_.get(), st_), st_);
  // A layer's output gradient is formed where it is masked (k_relu_mask):
  // from the output layer, the four copies of an upsampled pixel, a skip's
  // two shares, or the convolution above.
  // decoder level 0
  conv_bwd<kOut>(13, a6_.get(), u0_.get(), dy_.get(), params_.get() + out_w_, 0, 0, dA_.get(), H, W);
  conv_bwd<kPlain>(12, cat0_.get(), a6_.get(), dA_.get(), nullptr, 0, 0, dCat0_.get(), H, W);
  // decoder level 1
  conv_bwd<kLow>(11, a5_.get(), u1_.get(), dCat0_.get(), nullptr, c1 + c0, 0, dA_.get(), H1, W1);
  conv_bwd<kPlain>(10, cat1_.get(), a5_.get(), dA_.get(), nullptr, 0, 0, dCat1_.get(), H1, W1);
  // decoder level 2
  conv_bwd<kLow>(9, a4_.get(), u2_.get(), dCat1_.get(), nullptr, c2 + c1, 0, dA_.get(), H2, W2);
  conv_bwd<kPlain>(8, cat2_.get(), a4_.get(), dA_.get(), nullptr, 0, 0, dCat2_.get(), H2, W2);
  // bottleneck
  conv_bwd<kLow>(7, a3_.get(), b3_.get(), dCat2_.get(), nullptr, c3 + c2, 0, dA_.get(), H3, W3);
  conv_bwd<kPlain>(6, p2_.get(), a3_.get(), dA_.get(), nullptr, 0, 0, dA_.get(), H3, W3);
  // encoder level 2
  conv_bwd<kSkip>(5, a2_.get(), s2_.get(), dCat2_.get(), dA_.get(), c3 + c2, c3, dA_.get(), H2, W2);
  conv_bwd<kPlain>(4, p1_.get(), a2_.get(), dA_.get(), nullptr, 0, 0, dA_.get(), H2, W2);
  // encoder level 1
  conv_bwd<kSkip>(3, a1_.get(), s1_.get(), dCat1_.get(), dA_.get(), c2 + c1, c2, dA_.get(), H1, W1);
  conv_bwd<kPlain>(2, p0_.get(), a1_.get(), dA_.get(), nullptr, 0, 0, dA_.get(), H1, W1);
  // encoder level 0
  conv_bwd<kSkip>(1, a0_.get(), s0_.get(), dCat0_.get(), dA_.get(), c1 + c0, c1, dA_.get(), H, W);
  conv_bwd<kPlain>(0, x16_.get(), a0_.get(), dA_.get(), nullptr, 0, 0, nullptr, H, W);
  double loss = 0;
  SWFWI_CUDA(cudaMemcpyAsync(&loss, red_.get(), sizeof(double), cudaMemcpyDeviceToHost, st_));
  SWFWI_CUDA(cudaStreamSynchronize(st_));
  int timeout = 0;
  SWFWI_CUDA(cudaMemcpyFromSymbol(&timeout, g_conv_timeout, sizeof(int)));
  if (timeout) {
    const int zero = 0;
    SWFWI_CUDA(cudaMemcpyToSymbol(g_conv_timeout, &zero, sizeof(int)));
    throw Error(SWFWI_ERR_TIMEOUT, "a convolution's bounded wait on its tensor-core MMAs gave up");
  }
  if (!std::isfinite(loss)) throw Error(SWFWI_ERR_NONFINITE, "preconditioner loss is not finite");
  return loss / (double)P0;
}

void Preconditioner::adam_step(float lr, float beta1, float beta2, float eps) {
  step_++;
  const double bc1 = 1.0 - std::pow((double)beta1, (double)step_);
  const double bc2 = 1.0 - std::pow((double)beta2, (double)step_);
  const float lr_t = (float)(lr * std::sqrt(bc2) / bc1);
  k_adam<<<blocks_for(nparam_), kEw, 0, st_>>>(params_.get(), m_.get(), v_.get(), grads_.get(), nparam_,
                                               lr_t, beta1, beta2, eps);
  noted();
  refresh_bf16();
}

double Preconditioner::train_step(const float *x, const float *t, int N, int H, int W, float lr) {
  forward(x, nullptr, N, H, W);
  const double loss = backward(t);
  adam_step(lr);
  return loss;
}

void Preconditioner::stats(const float *a, const float *b, const float *c, int nzpad, int x0, int z0, int nx,
                           int nz) {
  constexpr int blocks = 256;
  red_.resize(8 + 4 * blocks);
  static_assert(blocks <= kEw, "k_stats sums at most kEw blocks");
  k_stats<<<blocks, kEw, 0, st_>>>(a, b, c, nzpad, x0, z0, nx, nz, red_.get() + 8, red_.get(), done_.get());
  noted();
}

void Preconditioner::features(const float *grad, const float *vel, const float *illum, int nxpad,
                              int nzpad, int bx0, int bxn, int bz0, int bzn, float *x3) {
  SWFWI_REQUIRE(grad && vel && x3, "null field");
  const int nx = nxpad - bx0 - bxn, nz = nzpad - bz0 - bzn;
  SWFWI_REQUIRE(nx > 0 && nz > 0, "empty interior");
  const int Hp = roundup8(nx), Wp = roundup8(nz);
  stats(grad, vel, illum, nzpad, bx0, bz0, nx, nz);
  launch_after(k_features, blocks_for((long long)Hp * Wp), kEw, 0, st_, grad, vel, illum, nzpad, bx0, bz0, nx, nz, Hp,
                                                                Wp, red_.get(), x3);
}

void Preconditioner::target(const float *dv, int nxpad, int nzpad, int bx0, int bxn, int bz0, int bzn,
                            float *t) {
  SWFWI_REQUIRE(dv && t, "null field");
  const int nx = nxpad - bx0 - bxn, nz = nzpad - bz0 - bzn;
  SWFWI_REQUIRE(nx > 0 && nz > 0, "empty interior");
  const int Hp = roundup8(nx), Wp = roundup8(nz);
  stats(dv, nullptr, nullptr, nzpad, bx0, bz0, nx, nz);
  k_target<<<blocks_for((long long)Hp * Wp), kEw, 0, st_>>>(dv, nzpad, bx0, bz0, nx, nz, Hp, Wp, red_.get(), t);
  noted();
}

void Preconditioner::scatter(const float *y, int nxpad, int nzpad, int bx0, int bxn, int bz0, int bzn,
                             float *dir) {
  SWFWI_REQUIRE(y && dir, "null field");
  const int nx = nxpad - bx0 - bxn, nz = nzpad - bz0 - bzn;
  SWFWI_REQUIRE(nx > 0 && nz > 0, "empty interior");
  launch_after(k_scatter, blocks_for((long long)nxpad * nzpad), kEw, 0, st_, y, nxpad, nzpad, bx0, bz0, nx, nz,
               roundup8(nz), dir);
}

void Preconditioner::propose(const float *grad, const float *vel, const float *illum, int nxpad,
                             int nzpad, int bx0, int bxn, int bz0, int bzn, float *dir) {
  const int nx = nxpad - bx0 - bxn, nz = nzpad - bz0 - bzn;
  const int Hp = roundup8(nx), Wp = roundup8(nz);
  feat_.resize((size_t)Hp * Wp * 3);
  outimg_.resize((size_t)Hp * Wp);
  features(grad, vel, illum, nxpad, nzpad, bx0, bxn, bz0, bzn, feat_.get());
  forward(feat_.get(), outimg_.get(), 1, Hp, Wp);
  scatter(outimg_.get(), nxpad, nzpad, bx0, bxn, bz0, bzn, dir);
}

}  // namespace swfwi
