// The 3x3 convolution of the proposal network on the fifth-generation tensor
// cores: an implicit GEMM with M = 128 pixels (a patch 8 wide and 16 high of one
// image), N = 32, 64, 96 or 128 output channels and K = 9 taps x input channels,
// the accumulators in tensor memory (TMEM), operands in shared memory, fetched
// by the tensor memory accelerator (TMA).
//
// What bounded it was the traffic from L2 into shared memory (about 38 bytes per
// clock and SM): a tile fetched anew for each of the nine taps, with its weights,
// reached 30 % of the tensor peak on the widest layers and 15 % on the narrow ones.
// So a K step is one horizontal shift (dx) of KC = 64 or 32 input
// channels: one 4-D TMA box (KC channels, 8 columns, 18 rows, 1 image) from a
// row above the patch, in the 128- or 64-byte swizzled K-major layout. A row
// of eight pixels is one 8-row group of that layout, so the three vertical
// taps of the box are the same operand started one group (8 x 2 KC bytes, a
// whole swizzle period) further on. The pixels outside the image come back
// as zeros, which is the convolution's padding and lets patches overhang the
// image's edge. A block takes several patches at a time, which share the
// weights, and keeps all nine taps' weights in shared memory for its whole
// life where they fit, else streams three taps a step.
//
// With resident weights the patches also share boxes: `s` patches (2 or 4) take
// every s-th column of 8 s columns, so that patch c's shift dx is the box of the
// columns c + dx - 1, c + dx - 1 + s, ..., which patch c + 1 reads at shift
// dx - 1. s + 2 boxes of a step serve the 3 s shifts (a 5-D map splits the
// columns by their remainder): a layer of 32 channels over 81 images of 256^2
// took 335 us with a box per patch and shift, 222 so.
//
// Blocks are persistent, one per SM: warp 0 issues the TMA loads into a ring
// of stages, warp 1 issues tcgen05.mma (kind::f16, bf16 inputs, f32
// accumulation) and commits each stage back to the loader, and sixteen more
// read the accumulators out of TMEM (one pixel and 32 channels per thread at a
// time) and apply the epilogue of the mma.sync kernel (bias, accumulate, ReLU,
// mask, bf16) while the next patches are multiplied into the other half of
// TMEM. Four epilogue warps, one per scheduler, took longer over their chains
// of dependent instructions than the loads and MMAs of a narrow layer.
//
// No unit is full now: at batch 8 the tcgen05 pipe is active 54 % of the time on
// 256^2 x 32 -> 32 channels and 56 % on 64^2 x 384 -> 128, L2 into the SMs takes 7
// and 18 % of its rate. What is left is the latency of loads, MMAs and epilogue
// over the few groups of patches that a block has.
//
// The weight gradient (k_conv3_dw_tc, further down) is the same machinery with
// K = pixels and both operands read channel-contiguous (MN-major).
//
// Every wait on an mbarrier gives up after about two seconds of device time;
// the block then records the failure in a device flag
// (rang_b200_nn_device_status) and returns after its own copies have landed
// (again with a limit) and its TMEM is freed.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "nn_conv_tc.h"

namespace {

using bf16 = __nv_bfloat16;

constexpr int TC_TW = 8, TC_TH = 16, TC_M = TC_TW * TC_TH;  // pixels per patch
constexpr int TC_ROWS = TC_TH + 2;                          // with the rows above and below
constexpr int TC_MAX_STAGES = 6;
constexpr int TC_SMEM = 225 * 1024;  // of the 227 KB a block may use
constexpr unsigned long long WAIT_NS = 2000000000ull;  // a wait gives up after this long

__device__ int g_conv_tc_error = 0;

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(bar)), "r"(bytes) : "memory");
}
// True once the phase of this parity has completed; false after limit_ns.
__device__ __forceinline__ bool mbar_wait_for(uint64_t* bar, uint32_t parity, unsigned long long limit_ns) {
  const uint32_t a = saddr(bar);
  unsigned long long t0 = 0;
  for (uint32_t i = 0;; i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 255u) == 64u) {  // the global timer is slow: not on short waits
      const unsigned long long t = now_ns();
      if (i == 64u)
        t0 = t;
      else if (t - t0 > limit_ns)
        return false;
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) { return mbar_wait_for(bar, parity, WAIT_NS); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(saddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(saddr(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2,
                                            int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], "
      "[%2];" ::"r"(saddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(saddr(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          saddr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(saddr(bar)), "r"(c0), "r"(c1)
      : "memory");
}

// Shared-memory matrix descriptors, as the two words of the 64-bit value. Low
// word: the address and, for MN-major operands, the leading byte offset (1 for
// K-major, whose swizzled layouts do not use it), both in 16-byte units; moving
// an operand by d bytes adds d / 16 to it. High word: the stride byte offset
// (8-row groups are 8 x row_bytes apart), descriptor version 1, layout type 2
// (128-byte swizzle) or 4 (64-byte swizzle).
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lead_bytes = 16) {
  return ((addr >> 4) & 0x3FFFu) | (((lead_bytes >> 4) & 0x3FFFu) << 16);
}
__host__ __device__ constexpr uint32_t desc_hi(uint32_t row_bytes) {
  return (((8u * row_bytes) >> 4) & 0x3FFFu) | (1u << 14) | ((row_bytes == 128 ? 2u : 4u) << 29);
}
// Instruction descriptor: f32 accumulator, bf16 A and B, both K-major, M = 128, N.
__host__ __device__ constexpr uint32_t instr_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                     uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %2};\n\t"
      "mov.b64 b, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}\n" ::"r"(tmem_d),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc));
}
// One lane of a converged warp (the same one each time).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// The smallest power of two of TMEM columns (32 to 512) that holds n.
__host__ __device__ constexpr uint32_t tmem_columns(int n) {
  uint32_t c = 32;
  while (c < (uint32_t)n) c *= 2;
  return c;
}

// 32 bytes of global memory, 32-byte aligned: a whole sector per lane. Lanes
// hold pixels, 64 or more bytes apart, and 16-byte stores reached L2 as half
// sectors.
__device__ __forceinline__ void store32(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

template <int KC, int BN>
struct TcConv {
  static constexpr int ROW = 2 * KC;                      // bytes of a staged pixel
  static constexpr int A_PATCH = TC_ROWS * TC_TW * ROW;   // one dx box of one patch
  static constexpr int B_TAP = BN * ROW;                  // one tap's weights of KC channels
  static constexpr int MT = BN == 32 ? 4 : 2;             // patches at a time, at most
  static constexpr uint32_t COLUMNS = tmem_columns(2 * MT * BN);
};
// How one launch runs (conv3_run): patches at a time, ring stages, whether
// the weights stay in shared memory, patch groups, output-channel tiles.
struct TcConvRun {
  int mt, stages, resident, groups, nt, tiles_x, tiles_y;
  int wide;   // the output takes 32-byte stores
  int share;  // the patches share boxes (a group is mt patches of interleaved columns)
};
// Past the stages and the resident weights: full, empty, weights, accumulator
// full and empty, done, the TMEM address, the failure flag, the bias.
constexpr int TC_EPI_WARPS = 16, TC_THREADS = 64 + 32 * TC_EPI_WARPS;
constexpr int TC_CONTROL = (2 * TC_MAX_STAGES + 6) * 8 + 16 + 128 * 4;

// Patch q of the batch (patches past the last lie in an image past the last:
// their loads return zeros and nothing is stored).
struct PatchAt {
  int img, x0, y0;
};
__device__ __forceinline__ PatchAt patch_at(int q, int tiles_x, int tiles_y) {
  const int row = q / tiles_x, img = row / tiles_y;
  return PatchAt{img, (q - row * tiles_x) * TC_TW, (row - img * tiles_y) * TC_TH};
}

template <int KC, int BN>
__global__ void __launch_bounds__(TC_THREADS, 1)
    k_conv3_tc(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tw, const TcConvArgs a,
               const TcConvRun run) {
  using L = TcConv<KC, BN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int nc = a.Cin / KC;
  const int stage_bytes = (run.share ? run.mt + 2 : run.mt) * L::A_PATCH + (run.resident ? 0 : 3 * L::B_TAP);
  const int nj = run.share ? nc : 3 * nc;  // steps of a patch group
  unsigned char* weights = smem + run.stages * stage_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(weights + (run.resident ? 9 * nc * L::B_TAP : 0));
  uint64_t* empty = full + TC_MAX_STAGES;
  uint64_t* wfull = empty + TC_MAX_STAGES;
  uint64_t* tfull = wfull + 1;
  uint64_t* tempty = tfull + 2;
  uint64_t* done = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* bad = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* bias = reinterpret_cast<float*>(tmem_slot + 4);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (int)(blockIdx.x % (unsigned)run.nt) * BN;  // this block's output channels
  const int g0 = (int)(blockIdx.x / (unsigned)run.nt), gstep = (int)(gridDim.x / (unsigned)run.nt);

  if (threadIdx.x == 0) {
    for (int s = 0; s < run.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(wfull, 1);
    for (int i = 0; i < 2; i++) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], TC_EPI_WARPS);
    }
    mbar_init(done, 1);
    *bad = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < BN) bias[threadIdx.x] = a.bias ? a.bias[n0 + threadIdx.x] : 0.0f;
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                 "r"(L::COLUMNS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {  // loader
    if (run.resident) {
      mbar_expect_tx(wfull, (uint32_t)(9 * nc * L::B_TAP));
      for (int i = 0; i < 9 * nc; i++)
        tma_load_2d(weights + i * L::B_TAP, &tw, wfull, (i / nc) * a.Cin + (i % nc) * KC, n0);
    }
    int it = 0;
    for (int g = g0; g < run.groups && !*bad; g += gstep) {
      for (int j = 0; j < nj; j++, it++) {  // channel block cb, horizontal tap dx
        const int s = it % run.stages, cb = run.share ? j : j / 3, dx = run.share ? 0 : j - 3 * cb;
        if (it >= run.stages && !mbar_wait(&empty[s], ((it / run.stages) - 1) & 1)) {
          *bad = 1;
          break;
        }
        unsigned char* st = smem + s * stage_bytes;
        mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
        if (run.share) {  // box b: columns x0 + b - 1 and every mt-th after it
          const PatchAt q = patch_at(g, run.tiles_x, run.tiles_y);  // x0 in columns over mt
          for (int b = 0; b < run.mt + 2; b++) {
            const int i = b == 0 ? q.x0 - 1 : b <= run.mt ? q.x0 : q.x0 + 1, r = b == 0 ? run.mt - 1 : (b - 1) % run.mt;
            tma_load_5d(st + b * L::A_PATCH, &tin, &full[s], cb * KC, r, i, q.y0 - 1, q.img);
          }
        }
        for (int m = 0; m < run.mt && !run.share; m++) {
          const PatchAt q = patch_at(g * run.mt + m, run.tiles_x, run.tiles_y);
          tma_load_4d(st + m * L::A_PATCH, &tin, &full[s], cb * KC, q.x0 + dx - 1, q.y0 - 1, q.img);
        }
        if (!run.resident)
          for (int dy = 0; dy < 3; dy++)
            tma_load_2d(st + run.mt * L::A_PATCH + dy * L::B_TAP, &tw, &full[s], (3 * dy + dx) * a.Cin + cb * KC, n0);
      }
    }
    // every load has landed before the block can leave
    if (run.resident && !mbar_wait(wfull, 0)) *bad = 1;
    for (int i = it > run.stages ? it - run.stages : 0; i < it; i++)
      if (!mbar_wait(&full[i % run.stages], (i / run.stages) & 1)) *bad = 1;
  } else if (warp == 1) {  // MMA issuer: the warp waits, one lane issues
    // The issue loop is unrolled onto descriptor words that differ by constants:
    // with descriptors formed per MMA by one lane, an MMA took 125 clocks
    // whatever its N (64 clocks of tensor time at N = 128, 16 at 32).
    constexpr uint32_t idesc = instr_desc(BN), hi = desc_hi(L::ROW);
    const bool leader = elect_one();
    if (run.resident && !mbar_wait(wfull, 0)) *bad = 1;
    const uint32_t wlo = desc_lo(saddr(weights));
    int s = 0, item = 0;
    uint32_t phase = 0;  // of stage s
    for (int g = g0; g < run.groups && !*bad; g += gstep, item++) {
      const int ab = item & 1;
      if (item >= 2 && !mbar_wait(&tempty[ab], ((item >> 1) - 1) & 1)) {
        *bad = 1;
        break;
      }
      tc_fence_after();
      const uint32_t acc = tmem + (uint32_t)(ab * run.mt * BN);
      for (int j = 0; j < nj; j++) {
        const int cb = run.share ? j : j / 3, dx = run.share ? 0 : j - 3 * cb;
        if (!mbar_wait(&full[s], phase)) {
          *bad = 1;
          break;
        }
        tc_fence_after();
        const uint32_t alo = desc_lo(saddr(smem + s * stage_bytes));
        if (leader && run.share) {
#pragma unroll
          for (int m = 0; m < L::MT; m++)
            if (m < run.mt) {
#pragma unroll
              for (int i = 0; i < 9; i++) {  // dx, then dy: the order of the other form's sums
                const int dx3 = i / 3, dy = i % 3;
                const uint32_t blo = wlo + (uint32_t)((3 * dy + dx3) * nc + cb) * (L::B_TAP / 16);
#pragma unroll
                for (int k = 0; k < KC / 16; k++)
                  umma(acc + (uint32_t)(m * BN),
                       alo + (uint32_t)(((m + dx3) * L::A_PATCH + dy * TC_TW * L::ROW + 32 * k) / 16), hi,
                       blo + (uint32_t)(2 * k), hi, idesc, (j | i | k) != 0);
              }
            }
          umma_commit(&empty[s]);
        } else if (leader) {
#pragma unroll
          for (int dy = 0; dy < 3; dy++) {
            const uint32_t blo = run.resident ? wlo + (uint32_t)((3 * dy + dx) * nc + cb) * (L::B_TAP / 16)
                                              : alo + (uint32_t)(run.mt * (L::A_PATCH / 16) + dy * (L::B_TAP / 16));
#pragma unroll
            for (int m = 0; m < L::MT; m++)
              if (m < run.mt) {
#pragma unroll
                for (int k = 0; k < KC / 16; k++)
                  umma(acc + (uint32_t)(m * BN),
                       alo + (uint32_t)((m * L::A_PATCH + dy * TC_TW * L::ROW + 32 * k) / 16), hi,
                       blo + (uint32_t)(2 * k), hi, idesc, (j | dy | k) != 0);
              }
          }
          umma_commit(&empty[s]);
        }
        __syncwarp();
        if (++s == run.stages) {
          s = 0;
          phase ^= 1;
        }
      }
      if (leader) umma_commit(&tfull[ab]);
      __syncwarp();
    }
    if (leader) umma_commit(done);  // arrives once every MMA issued above has completed
  } else if (warp >= 2) {  // epilogue: warp w reads TMEM lanes 32 (w mod 4) ..
    // Sets of four warps take the patches' 32-channel chunks in turn.
    const int quad = warp & 3, r = quad * 32 + lane, set = (warp - 2) >> 2;
    int item = 0;
    for (int g = g0; g < run.groups; g += gstep, item++) {
      const int ab = item & 1;
      const bool ok = mbar_wait(&tfull[ab], (item >> 1) & 1);
      if (!ok) *bad = 1;
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      for (int i = set; i < run.mt * (BN / 32); i += TC_EPI_WARPS / 4) {
        const int m = i / (BN / 32), c = (i - m * (BN / 32)) * 32;
        const PatchAt q = patch_at(run.share ? g : g * run.mt + m, run.tiles_x, run.tiles_y);
        const int x = run.share ? (q.x0 + r % TC_TW) * run.mt + m : q.x0 + r % TC_TW, y = q.y0 + r / TC_TW;
        const bool in = q.img < a.batch && x < a.W && y < a.H;
        const int64_t p = in ? ((int64_t)q.img * a.H + y) * a.W + x : 0;
        float v[32];
        __syncwarp();  // lanes outside the image skip the stores below
        tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((ab * run.mt + m) * BN + c), v);
        if (!in) continue;
        uint4* o = reinterpret_cast<uint4*>(a.out + p * a.ld_out + n0 + c);
        const uint4* mask = a.mask ? reinterpret_cast<const uint4*>(a.mask + p * a.ld_mask + n0 + c) : nullptr;
#pragma unroll
        for (int h = 0; h < 2; h++) {  // sixteen channels
          float* u = v + 16 * h;
#pragma unroll
          for (int k = 0; k < 16; k++) u[k] += bias[c + 16 * h + k];
          if (a.accumulate) {
            const uint4 old[2] = {o[2 * h], o[2 * h + 1]};
            const bf16* ob = reinterpret_cast<const bf16*>(old);
#pragma unroll
            for (int k = 0; k < 16; k++) u[k] += __bfloat162float(ob[k]);
          }
          if (a.relu) {
#pragma unroll
            for (int k = 0; k < 16; k++) u[k] = fmaxf(u[k], 0.0f);
          }
          if (mask) {
            const uint4 mv[2] = {mask[2 * h], mask[2 * h + 1]};
            const bf16* mb = reinterpret_cast<const bf16*>(mv);
#pragma unroll
            for (int k = 0; k < 16; k++)
              if (!(__bfloat162float(mb[k]) > 0.0f)) u[k] = 0.0f;
          }
          uint32_t res[8];
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(u[2 * k], u[2 * k + 1]);
            res[k] = *reinterpret_cast<const uint32_t*>(&b2);
          }
          if (run.wide) {
            store32(o + 2 * h, res);
          } else {
            o[2 * h] = make_uint4(res[0], res[1], res[2], res[3]);
            o[2 * h + 1] = make_uint4(res[4], res[5], res[6], res[7]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[ab]);
    }
  }
  __syncwarp();
  const bool ok = mbar_wait(done, 0);
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::COLUMNS));
  }
  if (threadIdx.x == 0 && (*bad || !ok)) atomicExch(&g_conv_tc_error, 1);
}

// ------------------------------------------------------------------ weight gradient

// dw[co][tap][ci] += sum_q dz[q - off(tap)][co] in[q][ci] on the tcgen05 path:
// M = output channels (of several vertical taps), N = BN input channels, K =
// the pixels of a range of patches (one patch, 128 pixels, per K step). A
// block takes one horizontal tap: per patch the A operand is the dz box at
// that shift, 18 rows high, and the B operand the input's patch, so that the
// three vertical taps share one fetch of each. Both are channel-contiguous
// (MN-major): a box of C channels is its pixels (the K index) as rows of 2C
// bytes in the 2C-byte swizzle, 8-row groups (image rows of the patch) 16C
// bytes apart, channel groups one box apart. A vertical tap is the dz operand
// started one image row, 16C bytes, further on, so with 64 output channels the
// "channel groups" of M = 128 are two vertical taps, 16C bytes apart, and with
// 32 four of them: two and one accumulators instead of three, the last tap's
// share unused (with M padded by zeros instead, 32 output channels ran at 51
// TFLOP/s). The block's sums, accumulated in TMEM over its patches, are added
// to dw with vector atomics.
template <int CO, int CB, int BN>  // CO: 32, 64 or 128 output channels per block
struct TcDw {
  static constexpr int CA = CO < 64 ? CO : 64;                  // channels of a dz box
  static constexpr int A_BOX = TC_ROWS * TC_TW * CA * 2, B_BOX = TC_M * CB * 2;
  static constexpr int A_BYTES = (CO / CA) * A_BOX, B_BYTES = (BN / CB) * B_BOX;
  static constexpr int STAGE = A_BYTES + B_BYTES;
  static constexpr int GROUPS = 128 / CO;                       // vertical taps per accumulator
  static constexpr int NACC = (3 + GROUPS - 1) / GROUPS;
  static constexpr uint32_t COLUMNS = tmem_columns(NACC * BN);
  // A box that a group reads past (the unused fourth tap) ends inside the stage.
  static constexpr int STAGES = 3 * STAGE + 2048 <= TC_SMEM - 2048 ? (4 * STAGE <= TC_SMEM / 2 ? 4 : 3) : 2;
  static constexpr int BYTES = STAGES * STAGE + (2 * STAGES + 1) * 8 + 16 + 1024;
};

// f32 accumulator, bf16 A and B, both MN-major, M = 128, N.
__host__ __device__ constexpr uint32_t instr_desc_mn(int n) {
  return instr_desc(n) | (1u << 15) | (1u << 16);
}

template <int CO, int CB, int BN>
__global__ void __launch_bounds__(128, 1)
    k_conv3_dw_tc(const __grid_constant__ CUtensorMap tdz, const __grid_constant__ CUtensorMap tin,
                  const TcDwArgs a) {
  using L = TcDw<CO, CB, BN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::STAGES * L::STAGE);
  uint64_t* empty = full + L::STAGES;
  uint64_t* done = empty + L::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* bad = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int dx = blockIdx.z;  // the horizontal tap
  const int ci_tiles = a.Cin / BN;
  const int co0 = (blockIdx.y / ci_tiles) * CO, ci0 = (blockIdx.y % ci_tiles) * BN;
  const int tiles_x = (a.W + TC_TW - 1) / TC_TW, tiles_y = (a.H + TC_TH - 1) / TC_TH;
  const int64_t q0 = (int64_t)blockIdx.x * a.patches_per_block;
  const int64_t q1 = q0 + a.patches_per_block < a.patches ? q0 + a.patches_per_block : a.patches;
  const int nk = (int)(q1 - q0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < L::STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(done, 1);
    *bad = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                 "r"(L::COLUMNS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {  // loader
    int issued = 0;
    for (int kb = 0; kb < nk; kb++) {
      const int s = kb % L::STAGES;
      if (kb >= L::STAGES && !mbar_wait(&empty[s], ((kb / L::STAGES) - 1) & 1)) {
        *bad = 1;
        break;
      }
      const PatchAt q = patch_at((int)(q0 + kb), tiles_x, tiles_y);
      unsigned char* st = smem + s * L::STAGE;
      mbar_expect_tx(&full[s], (uint32_t)L::STAGE);
#pragma unroll
      for (int h = 0; h < CO / L::CA; h++)
        tma_load_4d(st + h * L::A_BOX, &tdz, &full[s], co0 + L::CA * h, q.x0 + 1 - dx, q.y0 - 1, q.img);
#pragma unroll
      for (int h = 0; h < BN / CB; h++)
        tma_load_4d(st + L::A_BYTES + h * L::B_BOX, &tin, &full[s], ci0 + CB * h, q.x0, q.y0, q.img);
      issued = kb + 1;
    }
    for (int kb = issued > L::STAGES ? issued - L::STAGES : 0; kb < issued; kb++)
      if (!mbar_wait(&full[kb % L::STAGES], (kb / L::STAGES) & 1)) *bad = 1;
  } else if (warp == 1) {  // MMA issuer: the warp waits, one lane issues
    constexpr uint32_t idesc = instr_desc_mn(BN);
    constexpr uint32_t IMG_ROW = 16u * L::CA;  // eight pixels of dz
    const bool leader = elect_one();
    int s = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < nk; kb++) {
      if (!mbar_wait(&full[s], phase)) {
        *bad = 1;
        break;
      }
      tc_fence_after();
      if (leader) {
        const uint32_t sa = saddr(smem + s * L::STAGE);
        const uint32_t alo = desc_lo(sa, CO == 128 ? (uint32_t)L::A_BOX : IMG_ROW);
        const uint32_t blo = desc_lo(sa + L::A_BYTES, (uint32_t)L::B_BOX);
#pragma unroll
        for (int t = 0; t < L::NACC; t++)
#pragma unroll
          for (int k = 0; k < TC_M / 16; k++)  // 16 pixels (two image rows) per MMA
            umma(tmem + (uint32_t)(t * BN), alo + (uint32_t)(t * L::GROUPS + 2 * k) * (IMG_ROW / 16),
                 desc_hi(2 * L::CA), blo + (uint32_t)(2 * CB * k), desc_hi(2 * CB), idesc, (kb | k) != 0);
        umma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == L::STAGES) {
        s = 0;
        phase ^= 1;
      }
    }
    if (leader) umma_commit(done);
  }
  __syncwarp();
  const bool ok = mbar_wait(done, 0);
  tc_fence_after();

  // Epilogue: thread (warp, lane) owns TMEM lane 32 warp + lane: output channel
  // co of the group's vertical tap. Group j starts j rows into the box, a row
  // above the patch, so it holds dz[q - (1 - j) rows]: tap row 2 - j.
  const int r = warp * 32 + lane, co = co0 + r % CO;
#pragma unroll 1
  for (int t = 0; t < L::NACC; t++) {
    const int ty = 2 - (t * L::GROUPS + r / CO);
#pragma unroll 1
    for (int c = 0; c < BN; c += 32) {
      float v[32];
      __syncwarp();
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(t * BN + c), v);
      if (!ok || nk <= 0 || co >= a.Cout || ty < 0) continue;
      float* row = a.dw + ((int64_t)co * 9 + 3 * ty + dx) * a.Cin + ci0 + c;
#pragma unroll
      for (int j = 0; j < 8; j++)
        atomicAdd(reinterpret_cast<float4*>(row + 4 * j), make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::COLUMNS));
  }
  if (threadIdx.x == 0 && (*bad || !ok)) atomicExch(&g_conv_tc_error, 1);
}

PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// A 4-D map of an NHWC bf16 tensor, box (C channels, 8, rows, 1), 2C-byte swizzle.
bool nhwc_map(CUtensorMap* m, const bf16* base, int channels, int ld, int W, int H, int64_t batch, int C, int rows) {
  const cuuint64_t px = (cuuint64_t)ld * 2;
  cuuint64_t dims[4] = {(cuuint64_t)channels, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)batch};
  cuuint64_t strides[3] = {px, px * (cuuint64_t)W, px * (cuuint64_t)W * (cuuint64_t)H};
  cuuint32_t box[4] = {(cuuint32_t)C, (cuuint32_t)TC_TW, (cuuint32_t)rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, C == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same with the columns split by their remainder mod s (W a multiple of
// s): dimensions (channel, column mod s, column / s, row, image), whose strides
// ascend, each a multiple of the one before; box (C, 1, 8, rows, 1).
bool nhwc_map_split(CUtensorMap* m, const bf16* base, int channels, int ld, int W, int H, int64_t batch, int C, int rows,
                    int s) {
  const cuuint64_t px = (cuuint64_t)ld * 2;
  cuuint64_t dims[5] = {(cuuint64_t)channels, (cuuint64_t)s, (cuuint64_t)(W / s), (cuuint64_t)H, (cuuint64_t)batch};
  cuuint64_t strides[4] = {px, px * (cuuint64_t)s, px * (cuuint64_t)W, px * (cuuint64_t)W * (cuuint64_t)H};
  cuuint32_t box[5] = {(cuuint32_t)C, 1, (cuuint32_t)TC_TW, (cuuint32_t)rows, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, C == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int KC, int BN>
int launch(const TcConvArgs& a, cudaStream_t s) {
  using L = TcConv<KC, BN>;
  if (!encoder()) return 2;
  CUtensorMap tin, tw;
  cuuint64_t wdims[2] = {(cuuint64_t)9 * a.Cin, (cuuint64_t)a.Cout};
  cuuint64_t wstrides[1] = {(cuuint64_t)9 * a.Cin * 2};
  cuuint32_t wbox[2] = {(cuuint32_t)KC, (cuuint32_t)BN};
  cuuint32_t westr[2] = {1, 1};
  if (encoder()(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(a.w), wdims, wstrides, wbox, westr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, KC == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return 1;
  const int sms = sm_count();
  TcConvRun run{};
  run.tiles_x = (a.W + TC_TW - 1) / TC_TW;
  run.tiles_y = (a.H + TC_TH - 1) / TC_TH;
  run.nt = a.Cout / BN;
  run.wide = ((uintptr_t)a.out & 31u) == 0 && a.ld_out % 16 == 0;
  const int64_t patches = a.batch * run.tiles_x * run.tiles_y;
  // Patches at a time: fewer where a small call would leave SMs without work, one
  // only where that is a single round over the SMs (162 patches of 32 channels:
  // two rounds of one patch took 8.3 us, one round of two 6.6).
  run.mt = L::MT;
  while (run.mt > 2 && (patches + run.mt - 1) / run.mt * run.nt < sms) run.mt /= 2;
  if (patches * run.nt <= sms) run.mt = 1;
  run.groups = (int)((patches + run.mt - 1) / run.mt);
  // The weights stay in shared memory where two stages fit beside them.
  const int budget = TC_SMEM - TC_CONTROL - 1024;
  const int64_t wbytes = (int64_t)9 * a.Cin * BN * 2;
  run.resident = wbytes + 2 * run.mt * L::A_PATCH <= budget;
  // Shared boxes: s columns apart, where the weights are resident beside two
  // stages, s divides the width, the groups (8 s columns wide) overhang it by an
  // eighth at most and every SM has one. Where the driver refuses the 5-D map each
  // patch has its own (the same sums in the same order).
  for (int s = L::MT; s >= 2 && a.share && !run.share; s /= 2) {
    const int tx = (a.W + TC_TW * s - 1) / (TC_TW * s);
    const int64_t groups = a.batch * tx * run.tiles_y;
    if (wbytes + 2 * (s + 2) * L::A_PATCH > budget || a.W % s || 8 * tx * TC_TW * s > 9 * a.W || groups * run.nt < sms)
      continue;
    if (!nhwc_map_split(&tin, a.in, a.Cin, a.ld_in, a.W, a.H, a.batch, KC, TC_ROWS, s)) break;
    run.share = 1;
    run.resident = 1;
    run.mt = s;
    run.tiles_x = tx;
    run.groups = (int)groups;
  }
  if (!run.share && !nhwc_map(&tin, a.in, a.Cin, a.ld_in, a.W, a.H, a.batch, KC, TC_ROWS)) return 1;
  const int stage = (run.share ? run.mt + 2 : run.mt) * L::A_PATCH + (run.resident ? 0 : 3 * L::B_TAP);
  run.stages = (int)((budget - (run.resident ? wbytes : 0)) / stage);
  if (run.stages > TC_MAX_STAGES) run.stages = TC_MAX_STAGES;
  const int bytes = run.stages * stage + (run.resident ? (int)wbytes : 0) + TC_CONTROL + 1024;
  // per launch: the attribute belongs to the current device's context
  if (cudaFuncSetAttribute(k_conv3_tc<KC, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
    return 2;
  int per = sms / run.nt < 1 ? 1 : sms / run.nt;  // blocks of one output-channel tile
  if (per > run.groups) per = run.groups;
  k_conv3_tc<KC, BN><<<(unsigned)(per * run.nt), TC_THREADS, bytes, s>>>(tin, tw, a, run);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

template <int KC>
int launch_kc(const TcConvArgs& a, cudaStream_t s) {
  if (a.Cout % 128 == 0) return launch<KC, 128>(a, s);
  if (a.Cout % 96 == 0) return launch<KC, 96>(a, s);
  if (a.Cout % 64 == 0) return launch<KC, 64>(a, s);
  return launch<KC, 32>(a, s);
}

template <int CO, int CB, int BN>
int launch_dw(TcDwArgs a, cudaStream_t s) {
  using L = TcDw<CO, CB, BN>;
  if (!encoder()) return 2;
  CUtensorMap tdz, tin;
  if (!nhwc_map(&tdz, a.dz, a.Cout, a.ld_dz, a.W, a.H, a.batch, L::CA, TC_ROWS) ||
      !nhwc_map(&tin, a.in, a.Cin, a.ld_in, a.W, a.H, a.batch, CB, TC_TH))
    return 1;
  if (cudaFuncSetAttribute(k_conv3_dw_tc<CO, CB, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES) !=
      cudaSuccess)
    return 2;
  a.patches = a.batch * ((a.W + TC_TW - 1) / TC_TW) * ((a.H + TC_TH - 1) / TC_TH);
  const int tiles = ((a.Cout + CO - 1) / CO) * (a.Cin / BN);
  // about one block per SM over the horizontal taps and tiles, at least 4 patches each
  int64_t splits = sm_count() / (3 * tiles);
  const int64_t max_splits = (a.patches + 3) / 4;
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  a.patches_per_block = (a.patches + splits - 1) / splits;
  splits = (a.patches + a.patches_per_block - 1) / a.patches_per_block;
  k_conv3_dw_tc<CO, CB, BN><<<dim3((unsigned)splits, tiles, 3), 128, L::BYTES, s>>>(tdz, tin, a);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// Input channels per block: the widest tile that divides them.
int dw_tile(int cin) { return cin % 128 == 0 ? 128 : cin % 96 == 0 ? 96 : cin % 64 == 0 ? 64 : 32; }

template <int CO>
int launch_dw_co(const TcDwArgs& a, cudaStream_t s) {
  if (a.Cin % 128 == 0) return launch_dw<CO, 64, 128>(a, s);
  if (a.Cin % 96 == 0) return launch_dw<CO, 32, 96>(a, s);
  if (a.Cin % 64 == 0) return launch_dw<CO, 64, 64>(a, s);
  return launch_dw<CO, 32, 32>(a, s);
}

bool a16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

int64_t patch_count(int64_t batch, int W, int H) {
  return batch * ((W + TC_TW - 1) / TC_TW) * ((H + TC_TH - 1) / TC_TH);
}

}  // namespace

bool conv3_dw_tc_supported(const TcDwArgs& a) {
  return a.Cin % 32 == 0 && a.Cout % 32 == 0 && a.ld_in % 8 == 0 && a.ld_dz % 8 == 0 && a16(a.in) && a16(a.dz) &&
         a16(a.dw) && patch_count(a.batch, a.W, a.H) < (1ll << 30) && encoder() != nullptr;
}

// Images much smaller than a patch leave most of its pixels empty, and the
// mma.sync kernel, whose blocks of 128 pixels run across images, is faster once
// enough patches follow each other: 4096 images of 1 x 1 at 32 channels 5.6 us
// against 27.8, at 384 to 128 50 against 257; 2048 of 4 x 4 at 32 channels 8.9
// against 18.1, at 128 56 against 52; 512 of 1 x 16 6.3 against 9.8.
bool conv3_tc_preferred(const TcConvArgs& a) {
  const int64_t patches = patch_count(a.batch, a.W, a.H), pixels = a.batch * a.H * a.W;
  return patches < (a.Cin == 32 ? 512 : 1024) || pixels * (a.Cout % 128 == 0 ? 16 : 8) > patches * TC_M;
}

// The weight gradient: also where one block's pixels are all there are (one
// image of 1 x 1, 128 to 128 channels: 3.4 us against 5.0), else from emptier
// patches (4096 images of 2 x 2: 13.1 us against 31 at 32 channels, 64 against
// 90 at 128; of 4 x 4 it is the other way round from 64 channels on).
bool conv3_dw_tc_preferred(const TcDwArgs& a) {
  const int64_t patches = patch_count(a.batch, a.W, a.H), pixels = a.batch * a.H * a.W;
  return pixels > 64 && (patches < 1024 || pixels * 32 > patches * TC_M);
}

int conv3_dw_tc(const TcDwArgs& a, cudaStream_t s) {
  // Output channels per block: the most with which there are blocks enough (at
  // least 4 patches each) for every SM a few times. A block ends by adding
  // 3 x CO x BN sums to dw, most of a small call: 128 to 128 channels over 32
  // patches 13.4 us at 128, 6.4 at 32; over 128 patches 17.3, 13.9 and 10.3 at 128,
  // 64 and 32; over 512 28.6 and 23.4 at 128 and 64; 32 to 64 channels over 512
  // patches 9.7 at 64, 11.1 at 32.
  const int64_t blocks = (patch_count(a.batch, a.W, a.H) + 3) / 4 * 3 * (a.Cin / dw_tile(a.Cin)), sms = sm_count();
  if (a.Cout % 128 == 0 && blocks * (a.Cout / 128) >= 3 * sms) return launch_dw_co<128>(a, s);
  if (a.Cout % 64 == 0 && blocks * (a.Cout / 64) >= 2 * sms) return launch_dw_co<64>(a, s);
  return launch_dw_co<32>(a, s);
}

bool conv3_tc_supported(const TcConvArgs& a) {
  return a.Cin % 32 == 0 && a.Cout % 32 == 0 && a.ld_in % 8 == 0 && a.ld_out % 8 == 0 &&
         (!a.mask || (a.ld_mask % 8 == 0 && a16(a.mask))) && a16(a.in) && a16(a.w) && a16(a.out) &&
         patch_count(a.batch, a.W, a.H) < (1ll << 30) && encoder() != nullptr;
}

int conv3_tc(const TcConvArgs& a, cudaStream_t s) {
  return a.Cin % 64 == 0 ? launch_kc<64>(a, s) : launch_kc<32>(a, s);
}

// The timeout path of the convolutions' waits, exercised: a block holds TMEM
// as a convolution does, waits on an mbarrier on which nothing arrives until
// the wait gives up after limit_ns, sets the flag, frees its TMEM and
// returns. Nothing else runs in the block, so nothing is left in flight.
__global__ void __launch_bounds__(128) k_wait_probe(unsigned long long limit_ns) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int gave_up;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_slot)),
                 "r"(32u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (threadIdx.x == 0 && !mbar_wait_for(&bar, 0, limit_ns)) gave_up = 1;
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32u));
  }
  if (threadIdx.x == 0 && gave_up) atomicExch(&g_conv_tc_error, 1);
}

int conv3_tc_wait_probe(unsigned long long limit_ns, cudaStream_t s) {
  k_wait_probe<<<1, 128, 0, s>>>(limit_ns);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int conv3_tc_status(cudaStream_t s) {
  int v = 0;
  if (cudaStreamSynchronize(s) != cudaSuccess) return 2;
  if (cudaMemcpyFromSymbol(&v, g_conv_tc_error, sizeof(int)) != cudaSuccess) return 2;
  const int zero = 0;
  if (v && cudaMemcpyToSymbol(g_conv_tc_error, &zero, sizeof(int)) != cudaSuccess) return 2;
  return v ? 3 : 0;
}
