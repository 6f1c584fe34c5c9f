// Two-body network on the 5th-generation tensor cores (tcgen05, TMEM), 128 evaluations per tile.
//
// Layer 1 (3 -> 128) runs on the CUDA cores in FP32 (three FMAs per hidden unit); layers 2 and 3 are
// tcgen05 MMAs with the A operand in tensor memory and FP32 accumulation:
//   layer 2 (128 -> 512): four quarters of N = 128, K = 128, FP16 operands;
//   layer 3 (512 -> 9): N = 16, K = 512, FP16 operands (W3 rows 0-8, rows 9-15 zero).
// FP16 rather than BF16 for layers 2 and 3: their operands are tanh outputs in [-1, 1] and
// weights well inside FP16's range, so the 11-bit significand costs no range and rounds 8x finer.
// The epilogue warps read a layer-2 quarter (tcgen05.ld), round it to FP16 pairs, add the
// bias as FP16 pairs, apply tanh.approx.f16x2 and write the pairs back into tensor memory as
// layer 3's A operand; layer 1's tanh'd pairs go the same way into layer 2's A operand.
//
// The bound is the MUFU: 640 tanh per evaluation at 16 tanh per clock per SM (tanh.approx.f16x2
// issues at half the rate of tanh.approx.f32, measured on B200: packing saves issue slots, not
// MUFU time), i.e. 5,120 clocks per tile per SM, against 2,600 of the tensor pipe (an MMA with A in
// tensor memory takes 67 cycles at N = 128, 35 at N = 64, 12.4 at N = 16). What keeps the MUFU fed:
//   * two independent streams of tiles per CTA, eight epilogue warps each, two warps of either
//     stream per SM sub-partition: while one stream waits for an accumulator, loads or stores, the
//     other one's tanh fill the pipe;
//   * an issuing warp per stream, run warp-uniformly with one elected lane (a lane that branches
//     off by itself needs ~130 cycles per MMA, because its operands are not in uniform registers);
//   * a quarter's accumulator is taken into registers whole and released before its tanh are
//     computed, so that the next quarter's MMAs run under them;
//   * everything else in a tile-server warp per stream (below): MUFU instructions share an in-order
//     queue with shared-memory accesses and shuffles, so chains of those in an epilogue warp
//     wait behind its neighbours' tanh;
//   * 16-lane tensor-memory shapes (16x256b loads, 16x128b stores), which give a thread two rows and
//     every fourth column pair: weights and biases are read from shared memory a quarter as often as with one
//     row per thread.
// Measured (one B200, N = 65,536 clustered near field, 1.85e8 evaluations): 5.36e9 evaluations/s, 78 %
// of the MUFU's rate at the clock of the run (1.83 GHz), against 4.16e9 of one stream of 16 warps with
// layer-1 rows per thread, an MMA lane branching off its warp and the contraction in the epilogue warps; the
// stand-alone evaluation of a million features 222 against 261 us. Per tile and stream, with the MUFU
// stubbed out, the same chain of waits, loads and stores still takes 80 % of that time: what is left is the latency
// between the tensor core and the epilogue, four warps per sub-partition deep. Slower variants (near
// field, same case): layer 3 on mma.sync fragments in registers 4.3-4.7e9 (the legacy MMAs wait while a
// tcgen05 MMA holds the tensor core); eight N = 64 chunks 5.2e9; A2 for a whole quarter, half of
// A1 in shared memory, 5.0e9 (coarser phases leave the streams in step); the same with A2 halves 5.3e9.
// CTA = 20 warps:
//   warps 0-15  epilogue; stream w / 8; warp w reaches TMEM lanes 32 (w % 4) .. + 31. Of layer 1 it
//               computes, for the 32 rows 32 (w % 4) .. of its stream's tile, the hidden units
//               64 h .. 64 h + 63 (h = (w / 4) % 2); of layers 2 and 3 all columns of the 16
//               rows 32 (w % 4) + 16 h ..;
//   warps 16-17 issue the MMAs of streams 0 and 1 (warp 16 allocates tensor memory);
//   warps 18-19 the tile servers of streams 0 and 1: they put the features of the stream's tiles into
//               shared memory and take the nine outputs of every row from there (gathers, output
//               wrapper, contraction, stores: what the kernels differ in).
// Tensor memory (512 columns allocated, 256 per stream):
//   [0, 64)     A1: tanh(layer 1) as packed FP16 pairs (A of layer 2)
//   [64, 192)   layer-2 accumulator of a quarter (FP32)
//   [192, 224)  A2: the tanh'd FP16 pairs of half a quarter (A of layer 3)
//   [224, 240), [240, 256)  layer-3 accumulators of even / odd tiles (outputs in columns 0-8)
// Shared memory: W2 (512 x 128) and W3 (16 x 512) as FP16, canonical K-major 128-byte-swizzle
// layout, brought in by bulk copies behind the first tile's layer 1; (W1, b1) per pair of
// hidden units; b2 as FP16 pairs in load order; b3; mbarriers. Every wait is
// bounded (about two seconds of clock): on a timeout the CTA records an error, every later wait
// of the CTA returns at once, and the CTA drains its MMAs and frees its tensor memory. The warps
// use no barrier but these, so a warp that gave up leaves nobody waiting.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"

namespace hignn {
namespace tc {

using hignn::TcWeights;

constexpr int kTile = 128;
constexpr int kStreams = 2;
constexpr int kStreamWarps = 8;
constexpr int kStreamThreads = 32 * kStreamWarps;
constexpr int kMmaWarp = kStreams * kStreamWarps, kServerWarp = kMmaWarp + kStreams;
constexpr int kThreads = 32 * (kServerWarp + kStreams);
constexpr uint32_t kStreamCols = 256, kQuarter = 128;
constexpr uint32_t kOffA1 = 0, kOffD2 = 64, kOffA2 = 192, kOffD3 = 224;
constexpr int kW2Bytes = kH2 * kH1 * 2;  // 131072
constexpr int kW3Rows = 16;
constexpr int kW3Bytes = kW3Rows * kH2 * 2;  // 16384
constexpr int kOutStride = 12;  // floats per row of outputs (9 used; 16-byte reads of 8 rows hit 32 banks)
constexpr long long kWaitCycles = 4000000000LL;  // ~2 s at 1.9 GHz
// Wait profile (TcWeights::prof non-null): slot c - 13 sums the cycles that lane 0 of every warp
// spent in bounded waits with code c (the MMA warps: 13 the weights, 14 a layer-2 accumulator read and
// A1 written, 15 half a quarter in A2; the epilogue warps: 21 features, 22 a layer-2 accumulator, 24 A2
// free; the servers: 23 outputs); slot 12 the cycles of warp 0's whole epilogue; slot 13 the tiles
// processed. (Keeping it slows the engine by a quarter.)
constexpr int kProfSlots = 16, kProfTotal = 12, kProfTiles = 13;

struct alignas(1024) Smem {
  uint8_t w2[kW2Bytes];
  uint8_t w3[kW3Bytes];
  float4 w1p[kH1];             // hidden units 2k, 2k + 1: [2k] = (x, x', y, y'), [2k + 1] = (z, z', b, b')
  uint4 b2f[kH2 / 32][4];      // bias pairs of 32 columns for lane % 4: columns 2c + {0, 8, 16, 24}
  float b3[16];
  float4 feat[kStreams][2][kTile];         // features and output scale of each row, by tile parity
  float out[kStreams][kTile * kOutStride];  // layer-3 accumulators of each row
  uint64_t w_full, feat_full[kStreams], out_full[kStreams], d2_full[kStreams], d2_read[kStreams], a2_full[kStreams],
      a2_free[kStreams], drain[kStreams];
  uint32_t tmem_base;
  uint32_t end_tile[kStreams];  // tiles of the stream, once its end is known
  int abort_flag;
  unsigned long long* prof;          // optional wait profile (global, kProfSlots counters) or null
  unsigned long long wprof[16];      // per-CTA wait cycles by barrier code (lane 0 of each warp)
};

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(saddr(b)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(saddr(b)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// As mbar_try, but the thread may stay suspended in hardware for up to hint_ns while the phase is
// incomplete (it resumes as soon as the phase completes): waiting warps then issue nothing, and
// in particular do not fill the MIO queue that the MUFU instructions of the working warps share.
__device__ __forceinline__ bool mbar_try_sleep(uint64_t* b, uint32_t parity, uint32_t hint_ns) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity), "r"(hint_ns)
      : "memory");
  return ok != 0;
}
// Bounded wait: returns false (and raises the CTA abort flag) if the phase never completes.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, int* abort_flag, int* err, int code) {
  const long long t0 = clock64();
  while (!mbar_try_sleep(b, parity, 20000u)) {
    if (*(volatile int*)abort_flag) return false;
    if (clock64() - t0 > kWaitCycles) {
      atomicExch(abort_flag, 1);
      atomicCAS(err, 0, code);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(dst)), "r"(ncols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols));
}

// D[tmem] (+)= A[tmem] * B[smem desc]^T, kind::f16 (16-bit inputs, FP32 accumulate)
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(saddr(bar))
               : "memory");
}

// 32 consecutive 32-bit TMEM columns of this thread's lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
      "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
      "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
      "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}

// 16 consecutive 32-bit TMEM columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t tanh_f16x2(uint32_t x) {
  uint32_t y;
  asm("tanh.approx.f16x2 %0, %1;\n" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ uint32_t add_f16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr_bytes & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused by swizzled K-major): 16 B
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;            // descriptor version of sm_100
  d |= (uint64_t)2 << 61;            // SWIZZLE_128B
  return d;
}
// Instruction descriptor: FP16 x FP16 -> FP32, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_f16x(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// 16 consecutive 32-bit TMEM columns of this thread's lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// 16 rows x 64 accumulator columns of the 16 lanes at taddr: register 4 g + 2 i + j of lane l is row
// l / 4 + 8 i, column 8 g + 2 (l % 4) + j.
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
// The same for 16 columns.
__device__ __forceinline__ void tmem_ld_frag16(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
// wait::ld that the uses of v cannot be moved ahead of
__device__ __forceinline__ void tmem_wait_ld_of(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                 "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]),
                 "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]),
                 "+r"(v[30]), "+r"(v[31])::"memory");
}
__device__ __forceinline__ void tmem_wait_ld_of(uint32_t (&v)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])::"memory");
}
// 16 rows x 32 columns (32-bit) of the 16 lanes at taddr: register 2 g + i of lane l is row l / 4 + 8 i,
// column 4 g + l % 4.
__device__ __forceinline__ void tmem_st_frag32(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// Two FP32 fused multiply-adds in one instruction (each rounded as fmaf)
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// FP32 pair -> FP16 pair
__device__ __forceinline__ uint32_t pack_f16(uint64_t v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
  return pack_f16(lo, hi);
}

// ------------------------------------------------------------------ per-CTA setup / teardown
__device__ __forceinline__ void cta_setup(Smem& s, const TcWeights& w) {
  const int t = threadIdx.x;
  if (t == 0) {
    s.prof = w.prof;
    mbar_init(&s.w_full, 1);
    for (int i = 0; i < kStreams; i++) {
      mbar_init(&s.feat_full[i], 1);
      mbar_init(&s.out_full[i], kStreamWarps);
      mbar_init(&s.d2_full[i], 1);
      mbar_init(&s.d2_read[i], kStreamWarps);
      mbar_init(&s.a2_full[i], kStreamWarps);
      mbar_init(&s.a2_free[i], 1);
      mbar_init(&s.drain[i], 1);
      s.end_tile[i] = ~0u;
    }
    s.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    // W2 and W3 behind the rest of the setup and the first tile's layer 1 (the MMA warps wait for them)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(&s.w_full)),
                 "r"(kW2Bytes + kW3Bytes)
                 : "memory");
    auto bulk = [&](void* dst, const void* src, int bytes) {
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(saddr(dst)),
          "l"(src), "r"(bytes), "r"(saddr(&s.w_full))
          : "memory");
    };
    constexpr int kPart = kW2Bytes / 4;
    for (int q = 0; q < 4; q++) bulk(s.w2 + q * kPart, reinterpret_cast<const uint8_t*>(w.w2img) + q * kPart, kPart);
    bulk(s.w3, w.w3img, kW3Bytes);
  }
  for (int i = t; i < kH1 / 2; i += blockDim.x) {
    const float4 a = w.w1b1[2 * i], b = w.w1b1[2 * i + 1];
    s.w1p[2 * i] = make_float4(a.x, b.x, a.y, b.y);
    s.w1p[2 * i + 1] = make_float4(a.z, b.z, a.w, b.w);
  }
  for (int i = t; i < kH2 / 32 * 4; i += blockDim.x) {
    const float* b = w.b2 + 32 * (i >> 2) + 2 * (i & 3);
    s.b2f[i >> 2][i & 3] = make_uint4(pack_f16(b[0], b[1]), pack_f16(b[8], b[9]), pack_f16(b[16], b[17]),
                                      pack_f16(b[24], b[25]));
  }
  if (t < 16) s.b3[t] = t < kOut ? w.b3[t] : 0.f;
  if (t < 16) s.wprof[t] = 0ull;
  if ((t >> 5) == kMmaWarp) tmem_alloc(&s.tmem_base, 512);
  fence_before();
  __syncthreads();
  fence_after();
}

__device__ __forceinline__ void cta_teardown(Smem& s) {
  fence_before();
  __syncthreads();
  fence_after();
  if (s.prof && threadIdx.x < kProfSlots) atomicAdd(&s.prof[threadIdx.x], s.wprof[threadIdx.x]);
  if ((threadIdx.x >> 5) == kMmaWarp) tmem_dealloc(s.tmem_base, 512);
}

// Bounded wait of a whole warp: every lane gets the same answer. The first try reads no clock: a wait that
// is already over costs ~90 cycles of the warp's chain this way, ~200 with the timeout set up first.
// prof: the warp's copy of "a wait profile is kept".
__device__ __forceinline__ bool warp_wait(Smem& s, int* err, uint64_t* b, uint32_t parity, int code, bool prof) {
  const long long t0 = prof ? clock64() : 0;
  bool ok = __all_sync(0xffffffffu, mbar_try(b, parity));
  if (!ok) ok = __all_sync(0xffffffffu, mbar_wait(b, parity, &s.abort_flag, err, code));
  if (prof && (threadIdx.x & 31) == 0) atomicAdd(&s.wprof[code - 13], (unsigned long long)(clock64() - t0));
  return ok;
}
// One arrival per warp, after every lane's part.
__device__ __forceinline__ void warp_arrive(uint64_t* b) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(b);
}
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}

// ------------------------------------------------------------------ MMA warps
// Per quarter q of a tile of the stream, in order:
//   L2(q + 1)                      once quarter q's accumulator has been read (for q = 3: quarter 0 of the
//                                  next tile, whose layer 1 every warp writes to A1 before that)
//   L3 of the two halves of q      each once its tanh'd pairs are in A2; its commit frees A2, and the last one
//                                  of a tile completes the tile's layer-3 accumulator
// The first tile's layer 1 counts as one more reading ahead of quarter 0, so d2_read is in phase Q + 1
// after quarter Q. The whole warp runs the loop, so that addresses and descriptors are
// warp-uniform, and one elected lane issues.
struct MmaWarp {
  Smem& s;
  int* err;
  uint32_t stream, tb, w2, w3;
  bool prof;

  __device__ __forceinline__ bool wait(uint64_t* b, uint32_t parity, int code) {
    const bool ok = warp_wait(s, err, b, parity, code, prof);
    fence_after();
    return ok;
  }
  // layer-2 quarter q of the tile whose layer 1 is in A1
  __device__ __forceinline__ void l2(uint32_t q) {
    const uint64_t b0 = sdesc(w2 + q * (kQuarter * 128));
#pragma unroll
    for (uint32_t kk = 0; kk < 8; kk++)
      mma_ts(tb + kOffD2, tb + kOffA1 + 8 * kk, b0 + (((kk >> 2) * (kH2 * 128) + (kk & 3) * 32) >> 4),
             idesc_f16x(128, kQuarter), kk > 0);
    mma_commit(&s.d2_full[stream]);
  }
  // layer 3 of half quarter p (0 .. 7) of tile t
  __device__ __forceinline__ void l3(uint32_t t, uint32_t p) {
    const uint32_t d = tb + kOffD3 + 16 * (t & 1);
    const uint64_t b0 = sdesc(w3 + p * (kW3Rows * 128));
#pragma unroll
    for (uint32_t kk = 0; kk < 4; kk++)
      mma_ts(d, tb + kOffA2 + 8 * kk, b0 + 2 * kk, idesc_f16x(128, kW3Rows), (p > 0 || kk > 0) ? 1u : 0u);
    mma_commit(&s.a2_free[stream]);
  }
  __device__ __forceinline__ bool more(uint32_t tile) {
    return tile < __shfl_sync(0xffffffffu, *(volatile uint32_t*)&s.end_tile[stream], 0);
  }
  __device__ __forceinline__ void run() {
    if (!wait(&s.w_full, 0, 13) || !wait(&s.d2_read[stream], 0, 14) || !more(0)) return;
    if (elect_one()) l2(0);
    __syncwarp();
    bool next = true;
    for (uint32_t t = 0; next; t++)
      for (uint32_t q = 0; q < 4; q++) {
        if (!wait(&s.d2_read[stream], (q + 1) & 1, 14)) return;
        if (q == 3) next = more(t + 1);
        if (elect_one() && next) l2((q + 1) & 3);
        __syncwarp();
        for (uint32_t h = 0; h < 2; h++) {
          if (!wait(&s.a2_full[stream], h, 15)) return;
          if (elect_one()) l3(t, 2 * q + h);
          __syncwarp();
        }
      }
  }
};

__device__ __forceinline__ void mma_loop(Smem& s, int* err) {
  const uint32_t stream = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0) - kMmaWarp;
  MmaWarp w{s, err, stream, __shfl_sync(0xffffffffu, s.tmem_base, 0) + kStreamCols * stream, saddr(s.w2), saddr(s.w3),
            s.prof != nullptr};
  w.run();
  // drain: the weights have landed and every MMA issued so far completes before the CTA's memory is released
  if (elect_one()) {
    mma_commit(&s.drain[stream]);
    const long long t0 = clock64();
    while ((!mbar_try(&s.w_full, 0) || !mbar_try(&s.drain[stream], 0)) && clock64() - t0 < kWaitCycles) {
    }
  }
  __syncwarp();
}

// ------------------------------------------------------------------ epilogue side
// An epilogue warp: layer 1 of each tile of its stream from the features in shared memory, the tanh of
// its layer-2 quarters, and the tile's layer-3 accumulators into shared memory, one tile late. Ends
// with the stream, or at once when a wait fails.
struct Epi {
  Smem& s;
  int* err;
  uint32_t stream, half, lane;
  bool prof;
  uint32_t a1, rows;  // TMEM addresses: A1 of the warp's 32 rows and 64 units; column 0 of its 16 rows

  __device__ __forceinline__ Epi(Smem& sm, int* e) : s(sm), err(e) {
    const uint32_t w = threadIdx.x >> 5;
    stream = w >> 3;
    half = (w >> 2) & 1;
    lane = threadIdx.x & 31;
    prof = sm.prof != nullptr;
    const uint32_t tl = sm.tmem_base + kStreamCols * stream + ((32 * (w & 3)) << 16);
    a1 = tl + kOffA1 + 32 * half;
    rows = tl + ((16 * half) << 16);
  }
  // Whatever the warp does in tensor memory after a wait is ordered behind what the wait is for: the reading
  // of an accumulator behind the MMAs that filled it, the writing of A1 and A2 behind those that read them.
  __device__ __forceinline__ bool wait(uint64_t* b, uint32_t parity, int code) {
    const bool ok = warp_wait(s, err, b, parity, code, prof);
    fence_after();
    return ok;
  }

  // A1 <- tanh(W1 r + b1) of the warp's 32 rows and 64 hidden units as FP16 pairs (FP32 FMAs, bias
  // first). A thread takes four rows and every fourth pair of units, so that a pair's weights are
  // read once per four rows.
  __device__ __forceinline__ void layer1(uint32_t tile) {
    const float4* f = s.feat[stream][tile & 1] + 32 * ((threadIdx.x >> 5) & 3) + (lane >> 2);
    const ulonglong2* w = reinterpret_cast<const ulonglong2*>(s.w1p + 64 * half) + 2 * (lane & 3);
    uint64_t x[4], y[4], z[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float4 r = f[8 * i];
      x[i] = pack_f32x2(r.x, r.x);
      y[i] = pack_f32x2(r.y, r.y);
      z[i] = pack_f32x2(r.z, r.z);
    }
    uint32_t out[2][16];
#pragma unroll
    for (int g = 0; g < 8; g++) {
      const ulonglong2 xy = w[8 * g], zb = w[8 * g + 1];
#pragma unroll
      for (int i = 0; i < 4; i++)
        out[i >> 1][2 * g + (i & 1)] = tanh_f16x2(
            pack_f16(fma_f32x2(zb.x, z[i], fma_f32x2(xy.y, y[i], fma_f32x2(xy.x, x[i], zb.y)))));
    }
    tmem_st_frag32(a1, out[0]);
    tmem_st_frag32(a1 + (16u << 16), out[1]);
    tmem_wait_st();
  }

  // Half quarter p (values in v): one rounding to FP16 pairs, the FP16 bias added to the pairs, tanh, and
  // into A2 once layer 3 of the half before has read it (which, for p = 0, also completes tile t - 1).
  __device__ __forceinline__ bool half_quarter(uint32_t t, uint32_t p, const uint32_t (&v)[32]) {
    const uint4 b0 = s.b2f[2 * p][lane & 3], b1 = s.b2f[2 * p + 1][lane & 3];
    const uint32_t bias[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    uint32_t out[16];
#pragma unroll
    for (int g = 0; g < 8; g++)
#pragma unroll
      for (int i = 0; i < 2; i++)
        out[2 * g + i] = tanh_f16x2(add_f16x2(
            pack_f16(__uint_as_float(v[4 * g + 2 * i]), __uint_as_float(v[4 * g + 2 * i + 1])), bias[g]));
    if ((t > 0 || p > 0) && !wait(&s.a2_free[stream], (p + 1) & 1, 24)) return false;
    tmem_st_frag32(rows + kOffA2, out);
    tmem_wait_st();
    fence_before();
    warp_arrive(&s.a2_full[stream]);
    return true;
  }

  // Layer-3 accumulators of the warp's rows of tile t, complete, into shared memory. The server has
  // taken the outputs of tile t - 1: the features of t + 1, which it sent after that, are here.
  __device__ __forceinline__ void retire(uint32_t t) {
    uint32_t v[8];
    tmem_ld_frag16(rows + kOffD3 + 16 * (t & 1), v);
    tmem_wait_ld_of(v);
    fence_before();  // the accumulator's reuse follows this warp's later arrivals
    const uint32_t c = lane & 3;
    float* o = s.out[stream] + kOutStride * (32 * ((threadIdx.x >> 5) & 3) + 16 * half + (lane >> 2));
    *reinterpret_cast<uint2*>(o + 2 * c) = make_uint2(v[0], v[1]);
    *reinterpret_cast<uint2*>(o + 8 * kOutStride + 2 * c) = make_uint2(v[2], v[3]);
    if (c == 0) {
      o[8] = __uint_as_float(v[4]);
      o[8 * kOutStride + 8] = __uint_as_float(v[6]);
    }
    warp_arrive(&s.out_full[stream]);
  }

  __device__ __forceinline__ void run() {
    if (!wait(&s.feat_full[stream], 0, 21)) return;
    bool have = 0 < *(volatile uint32_t*)&s.end_tile[stream];
    if (have) layer1(0);
    fence_before();
    warp_arrive(&s.d2_read[stream]);
    uint32_t t = 0;
    for (; have; t++) {
#pragma unroll 1
      for (uint32_t q = 0; q < 4; q++) {
        if (!wait(&s.d2_full[stream], q & 1, 22)) return;
        if (q == 3) {  // the last quarter is complete: every layer-2 MMA of this tile has read A1
          if (!wait(&s.feat_full[stream], (t + 1) & 1, 21)) return;
          have = t + 1 < *(volatile uint32_t*)&s.end_tile[stream];
          if (have) layer1(t + 1);
        }
        uint32_t v0[32], v1[32];
        tmem_ld_frag64(rows + kOffD2, v0);
        tmem_ld_frag64(rows + kOffD2 + 64, v1);
        tmem_wait_ld_of(v0);
        tmem_wait_ld_of(v1);
        fence_before();
        warp_arrive(&s.d2_read[stream]);
        if (!half_quarter(t, 2 * q, v0)) return;
        if (q == 0 && t > 0) retire(t - 1);
        if (!half_quarter(t, 2 * q + 1, v1)) return;
      }
      if (prof && threadIdx.x % kStreamThreads == 0) atomicAdd(&s.wprof[kProfTiles], 1ull);
    }
    if (t == 0 || !wait(&s.a2_free[stream], 1, 24)) return;
    retire(t - 1);
  }
};

// ------------------------------------------------------------------ tile servers
// Of every tile t of a stream, in order: put() its 128 rows and ready(); then, one tile later (so that
// the epilogue finds the next tile's features in time), take() its outputs after wait(t). end(tiles)
// instead of ready() ends the stream. Row of lane l, part k: 32 k + l. The feature buffer of tile t is
// rewritten by tile t + 2, after wait(t): every epilogue warp has read it by then. The outputs of tile
// t must all be taken before ready() or end() of tile t + 2.
struct Server {
  Smem& s;
  int* err;
  int stream, lane;

  __device__ __forceinline__ Server(Smem& sm, int* e)
      : s(sm), err(e), stream((threadIdx.x >> 5) - kServerWarp), lane(threadIdx.x & 31) {}
  __device__ __forceinline__ bool aborted() const { return *(volatile int*)&s.abort_flag; }

  // features of one row; kept with the scale of the output wrapper: 1 / |r|, or -1 where |r| < 1e-5
  // (there M = I)
  __device__ __forceinline__ void put(uint32_t tile, int row, float rx, float ry, float rz) {
    const float nr = sqrtf(fmaf(rz, rz, fmaf(ry, ry, __fmul_rn(rx, rx))));
    s.feat[stream][tile & 1][row] = make_float4(rx, ry, rz, nr < 1e-5f ? -1.f : __frcp_rn(nr));
  }
  __device__ __forceinline__ void ready() { warp_arrive(&s.feat_full[stream]); }
  __device__ __forceinline__ void end(uint32_t tiles) {
    if (lane == 0) *(volatile uint32_t*)&s.end_tile[stream] = tiles;  // released by the arrival
    warp_arrive(&s.feat_full[stream]);
  }
  __device__ __forceinline__ bool wait(uint32_t tile) {
    return warp_wait(s, err, &s.out_full[stream], tile & 1, 23, s.prof != nullptr);
  }

  // M (row-major 3x3) of a row of the tile waited for. Every operation is rounded by itself (no
  // contraction with what the caller does with M): the ACA pivot search compares determinants of these
  // entries, and a last-bit difference can choose another, equally valid pivot.
  __device__ __forceinline__ void take(uint32_t tile, int row, float (&M)[9]) const {
    const float4* o = reinterpret_cast<const float4*>(s.out[stream] + kOutStride * row);
    const float inv = s.feat[stream][tile & 1][row].w;
    const float4 p = o[0], q = o[1];
    const float y[9] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w, reinterpret_cast<const float*>(o)[8]};
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const bool dg = k % 4 == 0;
      float v = __fadd_rn(y[k], s.b3[k]);
      if (dg) v = __fadd_rn(v, 1.0f);
      v = __fmul_rn(v, inv);
      M[k] = inv < 0.f ? (dg ? 1.0f : 0.0f) : v;
    }
  }
};

// Roles of the CTA's warps; `serve` runs in the two tile-server warps.
template <class Serve>
__device__ __forceinline__ void run_cta(Smem& s, const TcWeights& w, int* err, Serve&& serve) {
  cta_setup(s, w);
  const int warp = threadIdx.x >> 5;
  if (warp < kMmaWarp) {
    const long long t0 = clock64();
    Epi(s, err).run();
    if (s.prof && threadIdx.x == 0) s.wprof[kProfTotal] += (unsigned long long)(clock64() - t0);
  } else if (warp < kServerWarp) {
    mma_loop(s, err);
  } else {
    serve(Server(s, err));
  }
  cta_teardown(s);
}

}  // namespace tc
}  // namespace hignn
