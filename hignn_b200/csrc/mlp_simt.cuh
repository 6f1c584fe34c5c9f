// FP32 SIMT evaluation of the two-body network, 64 evaluations per tile.
//
// This is the "plain FP32" form: every layer in FP32 on the CUDA cores, the same
// arithmetic class as the reference's libtorch FP32 forward (src/CloseDot.cpp:233).
// Layer widths 3 -> 128 -> 512 -> 9. Every operation is a single correctly rounded
// FP32 operation in a fixed order (explicit fused multiply-adds, _rn intrinsics,
// the tanh of tanh_f32.cuh), so each output is a function of its feature alone:
//   h1[k] = tanh(fma(W1[k][2], r_z, fma(W1[k][1], r_y, fma(W1[k][0], r_x, b1[k]))))
//   h2[n] = tanh((sum_k fma(h1[k], W2[n][k], .), k ascending from 0) + b2[n])
//   y[o]  = (sum_n fma(h2[n], W3[o][n], .), n ascending from 0) + b3[o] (+ 1 on the
//           diagonal), divided by |r| = sqrt(fma(r_z, r_z, fma(r_y, r_y, r_x r_x))).
//
// The bound is the FP32 pipe: 70,528 FMA per evaluation (551 clocks per SM) and 640 tanh of about 24
// FMA-pipe slots each. Two CTAs of four warps share an SM, so that one's tanh and layer 3 run under
// the other's layer 2. A warp owns 16 evaluations from features to outputs; only the W2 slices are shared:
//   layer 2 in two chunks of 256 units, 16 evaluations x 8 units per thread as packed FMAs (fma.rn.f32x2
//   over evaluation pairs: half the issue slots, the same rounding); per k a thread reads
//   16 h1 values (broadcast) and 8 weights, 24 clocks of shared-memory return for 128 of the
//   warp's FMA pipe; W2 comes in slices of 8 k x 256 units, double-buffered with cp.async;
//   each chunk's sums go through tanh and layer 3 in four pieces of 64 units by way of 5 KB of the
//   warp's shared memory; in layer 3 a lane takes two evaluations and three outputs (W3 read through the
//   constant bank instead was four times slower: its loads do not pipeline).
// Measured (one B200, 1.0M separations): 2.22e8 evaluations/s, against 1.54e8 of one CTA of eight warps per SM
// with 8 x 4 scalar FMAs per thread, branching tanh and one weight read per FMA in layer 3. Layer 2 alone
// runs at 3.4e8 (62 % of the FP32 pipe; the packed FMA itself reaches 77 % of it with two warps per
// sub-partition, and scalar FMAs in the same tile are 5 % slower), layer 2 and tanh at 2.4e8.
#pragma once

#include <cuda_runtime.h>

#include "common.h"
#include "tanh_f32.cuh"
#include "tanh_f32x2.cuh"

namespace hignn {
namespace simt {

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kRows = 16;               // evaluations per warp
constexpr int kTile = kRows * kWarps;   // per CTA
constexpr int kCtasPerSm = 2;
constexpr int kChunk = 256;             // layer-2 units per pass over k
constexpr int kSlice = 8;               // k per staged W2 slice
constexpr int kSlices = kH1 / kSlice;
constexpr int kPiece = 64;              // units per tanh / layer-3 piece
constexpr int kPieceStride = kRows + 4; // floats per unit: 16-byte stores of consecutive units hit 32 banks

struct Smem {
  float h1[kH1][kTile];                          // 32 KB, [k][e]
  float w2[2][kSlice][kChunk];                   // 16 KB, W2^T slices [k][n]
  float h2[kWarps][kPiece][kPieceStride];        // 20 KB, [n][e] of each warp
  float w3[kOut][kH2];                           // 18 KB
  float b2[kH2];                                 // 2 KB
  float4 w1b1[kH1];                              // 2 KB
  float b3[16];
  float4 r[kTile];                               // features (x, y, z, unused)
  float y[kTile][kOut + 1];                      // network outputs after the wrapper
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }

// Per-CTA weight staging (once per kernel).
__device__ __forceinline__ void load_weights(Smem& s, const MlpF32& w) {
  const int t = threadIdx.x;
  for (int i = t; i < kH2; i += kThreads) s.b2[i] = w.b2[i];
  for (int i = t; i < kH1; i += kThreads) s.w1b1[i] = w.w1b1[i];
  for (int i = t; i < kOut * kH2; i += kThreads) (&s.w3[0][0])[i] = w.w3[i];
  if (t < 16) s.b3[t] = t < kOut ? w.b3[t] : 0.f;
}

// Slice q of a tile (chunk q / kSlices, k from kSlice (q % kSlices)) into buffer q % 2.
__device__ __forceinline__ void load_w2_slice(Smem& s, const MlpF32& w, int q) {
  const float* src = w.w2t + (size_t)(q % kSlices) * kSlice * kH2 + (q / kSlices) * kChunk;
  float* dst = &s.w2[q & 1][0][0];
#pragma unroll
  for (int i = threadIdx.x; i < kSlice * kChunk / 4; i += kThreads)
    cp_async16(dst + 4 * i, src + (size_t)(i / (kChunk / 4)) * kH2 + 4 * (i % (kChunk / 4)));
  cp_async_commit();
}

// Evaluations per warp for n of them over `slots` CTAs: the smallest tile that takes them all at once. A
// tile takes 65 us at 16 evaluations per warp, 43 at 8, 30 at 4 (92, 59 and 40 with two CTAs on the SM): the
// weights and their slices cost the same for each. So fewer per warp is the better only
// while it adds no second round (9,473 evaluations over 296 slots: 102 us at 8, 92 at 16).
__host__ __device__ inline int rows_per_warp(int64_t n, int64_t slots) {
  return n <= kTile / 4 * slots ? kRows / 4 : n <= kTile / 2 * slots ? kRows / 2 : kRows;
}

// Evaluates M(r) for s.r[0 .. kWarps * Rows - 1] (caller has written them and synchronized), Rows (16, 8 or 4) per
// warp; the same operations in the same order per evaluation.
// On return s.y[e][0..8] holds M row-major and the block is synchronized.
template <int Rows = kRows>
__device__ __forceinline__ void mlp_tile(Smem& s, const MlpF32& w) {
  static_assert(Rows <= kRows && Rows % 4 == 0, "whole float4 of evaluations");
  constexpr int kQuads = Rows / 4, kPairs = Rows / 2;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, e0 = Rows * wid;
  load_w2_slice(s, w, 0);
  {  // layer 1 of the warp's evaluations: four of them and every 32 / kQuads-th unit per thread
    const int e = e0 + 4 * (lane % kQuads);
    const float4 r0 = s.r[e], r1 = s.r[e + 1], r2 = s.r[e + 2], r3 = s.r[e + 3];
    const f2 x0 = f2_make(r0.x, r1.x), y0 = f2_make(r0.y, r1.y), z0 = f2_make(r0.z, r1.z);
    const f2 x1 = f2_make(r2.x, r3.x), y1 = f2_make(r2.y, r3.y), z1 = f2_make(r2.z, r3.z);
#pragma unroll 2
    for (int k = lane / kQuads; k < kH1; k += 32 / kQuads) {
      const float4 c = s.w1b1[k];
      const f2 cx = f2_dup(c.x), cy = f2_dup(c.y), cz = f2_dup(c.z), cb = f2_dup(c.w);
      const f2 a = tanh_f32x2(f2_fma(cz, z0, f2_fma(cy, y0, f2_fma(cx, x0, cb))));
      const f2 b = tanh_f32x2(f2_fma(cz, z1, f2_fma(cy, y1, f2_fma(cx, x1, cb))));
      *reinterpret_cast<ulonglong2*>(&s.h1[k][e]) = make_ulonglong2(a.v, b.v);
    }
    __syncwarp();
  }
  // layer 3: lanes 0 .. 3 kPairs - 1 take two evaluations (e3, e3 + 1 of the warp's) and three outputs (o3 ..) each
  const int e3 = 2 * (lane % kPairs), o3 = lane < 3 * kPairs ? 3 * (lane / kPairs) : 0;
  f2 y3[3] = {f2_dup(0.f), f2_dup(0.f), f2_dup(0.f)};
  float(*h2)[kPieceStride] = s.h2[wid];
#pragma unroll 1
  for (int c = 0; c < kH2 / kChunk; c++) {
    f2 acc[kPairs][8];  // evaluation pairs x units lane + 32 j of the chunk
#pragma unroll
    for (int i = 0; i < kPairs; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[i][j] = f2_dup(0.f);
#pragma unroll 1
    for (int q = 0; q < kSlices; q++) {
      cp_async_wait_all();
      __syncthreads();  // slice visible; every warp is done with the other buffer
      const int sl = c * kSlices + q;
      if (sl + 1 < kSlices * (kH2 / kChunk)) load_w2_slice(s, w, sl + 1);
      const float* wk = &s.w2[sl & 1][0][lane];
      const ulonglong2* hk = reinterpret_cast<const ulonglong2*>(&s.h1[q * kSlice][e0]);
#pragma unroll 4
      for (int k = 0; k < kSlice; k++) {
        f2 a[kPairs];
#pragma unroll
        for (int i = 0; i < kQuads; i++) {
          const ulonglong2 v = hk[(size_t)k * (kTile / 4) + i];
          a[2 * i].v = v.x;
          a[2 * i + 1].v = v.y;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const f2 b = f2_dup(wk[k * kChunk + 32 * j]);
#pragma unroll
          for (int i = 0; i < kPairs; i++) acc[i][j] = f2_fma(a[i], b, acc[i][j]);
        }
      }
    }
#pragma unroll
    for (int p = 0; p < kChunk / kPiece; p++) {  // units 64 p .. of the chunk: j = 2 p, 2 p + 1
      const int n0 = c * kChunk + p * kPiece;
      __syncwarp();  // the piece before has been read
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const f2 bias = f2_dup(s.b2[n0 + 32 * j + lane]);
#pragma unroll
        for (int i = 0; i < kQuads; i++)
          *reinterpret_cast<ulonglong2*>(&h2[32 * j + lane][4 * i]) =
              make_ulonglong2(f2_add(acc[2 * i][2 * p + j], bias).v, f2_add(acc[2 * i + 1][2 * p + j], bias).v);
      }
      __syncwarp();
#pragma unroll 2
      for (int i = lane; i < kPiece * kQuads; i += 32) {  // tanh in place, four evaluations of a unit at a time
        ulonglong2* v = reinterpret_cast<ulonglong2*>(&h2[i / kQuads][4 * (i % kQuads)]);
        const ulonglong2 x = *v;
        *v = make_ulonglong2(tanh_f32x2(f2{x.x}).v, tanh_f32x2(f2{x.y}).v);
      }
      __syncwarp();
#pragma unroll 4
      for (int n = 0; n < kPiece; n += 4) {
        const float4 w0 = *reinterpret_cast<const float4*>(&s.w3[o3][n0 + n]);
        const float4 w1 = *reinterpret_cast<const float4*>(&s.w3[o3 + 1][n0 + n]);
        const float4 w2 = *reinterpret_cast<const float4*>(&s.w3[o3 + 2][n0 + n]);
        const float wv[3][4] = {{w0.x, w0.y, w0.z, w0.w}, {w1.x, w1.y, w1.z, w1.w}, {w2.x, w2.y, w2.z, w2.w}};
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const f2 h = f2{*reinterpret_cast<const uint64_t*>(&h2[n + m][e3])};
#pragma unroll
          for (int o = 0; o < 3; o++) y3[o] = f2_fma(h, f2_dup(wv[o][m]), y3[o]);
        }
      }
    }
  }
  if (lane < 3 * kPairs) {  // wrapper of python/convert.py:11-20: (y + b3 + I) / |r|, identity for |r| < 1e-5
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int e = e0 + e3 + q;
      const float4 r = s.r[e];
      const float nr = __fsqrt_rn(__fmaf_rn(r.z, r.z, __fmaf_rn(r.y, r.y, __fmul_rn(r.x, r.x))));
#pragma unroll
      for (int o = 0; o < 3; o++) {
        const bool dg = (o3 + o) % 4 == 0;
        float v = __fadd_rn(q ? f2_hi(y3[o]) : f2_lo(y3[o]), s.b3[o3 + o]);
        if (dg) v = __fadd_rn(v, 1.0f);
        v = __fdiv_rn(v, nr);
        if (nr < 1e-5f) v = dg ? 1.0f : 0.0f;
        s.y[e][o3 + o] = v;
      }
    }
  }
  __syncthreads();
}

}  // namespace simt
}  // namespace hignn
