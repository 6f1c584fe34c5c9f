// FP64 dense rows: u_i = sum_j 0.5 (M + M^T)(x_j - x_i) f_j with the two-body network evaluated
// in FP64 (weights promoted from their FP32 values), FP64 sums over all sources.
//
// This is the dense FP64 evaluation the H-matrix product's error is measured against
// (src/PostCheckDot.cpp:351-376 compares against a dense product; here the network itself runs
// in FP64 so that the reference point carries no FP32 network rounding). It takes the same work
// list as the FP32 dense rows (PairWork items flagged kPairSymmetrize: up to 128 gathered target
// rows against one source leaf of up to kMaxLeaf particles).
//
// One persistent CTA of sixteen warps per SM, tiles of 128 evaluations. Layers 2 and 3 are FP64
// mma.sync (m8n8k4), which reach the FP64 pipe's 64 FMA per clock per SM with 12 clocks of shared-memory
// reads per 128 of the pipe; register-tiled scalar FMAs need three times the reads.
//   layer 1: h1[k][e] = tanh(W1[k] . r_e + b1[k]) (128 x 128 doubles in shared memory);
//   layer 2: eight chunks of 64 hidden units, 32 evaluations x 16 units per warp, on one W2^T chunk
//            staged in shared memory as doubles (the next chunk's values are fetched meanwhile);
//            the chunk buffer then receives tanh(acc + b2) as [unit][evaluation];
//   layer 3: warp w accumulates the outputs of evaluations 8 w .. 8 w + 7 (columns 0-8 of 16),
//            W3 read through the read-only cache;
//   wrapper: (y + b3 + I) / |r|, identity below |r| = 1e-5 (python/convert.py:11-20).
// Both shared arrays have row strides of 4 mod 16 doubles: a fragment's 4 k x 8 rows then hit every bank once
// per half warp. The bound is the FP64 pipe: 70,528 FMA and 640 tanh per evaluation (1,100 clocks of FMA, about 440
// of tanh with sixteen warps). Measured (one B200, 100 rows x 65,536 sources): 54.0 ms, against 94.4 ms of 8 x 4
// scalar FMAs per thread in eight warps and whole (rows, leaf) items.
#include "common.h"
#include "kernels.h"

namespace hignn {

namespace {

constexpr int kF64Warps = 16;
constexpr int kF64Threads = 32 * kF64Warps;
constexpr int kF64Tile = 128;
constexpr int kF64Chunk = 64;
constexpr int kH1Stride = kF64Tile + 4, kH2Stride = kF64Tile + 4, kW2Stride = kF64Chunk + 4;
constexpr int kF64Out = 10;
static_assert(kF64Tile == 8 * kF64Warps, "layer 3 gives a warp eight evaluations");

struct F64Smem {
  double h1[kH1 * kH1Stride];   // 132 KB, [k][e]
  double buf[kH1 * kW2Stride];  // 68 KB: W2^T chunk [k][n], then h2 [n][e]
  double r[kF64Tile][3];
  double y[kF64Tile][kF64Out];
  double uI[kF64Tile][3];
  int item;
};
static_assert(sizeof(F64Smem) <= 232448, "FP64 dense-rows shared memory exceeds 227 KB per CTA");
static_assert(kF64Chunk * kH2Stride <= kH1 * kW2Stride, "h2 does not fit the chunk buffer");

// D += A B: lane l holds A[l / 4][l % 4], B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

__device__ __forceinline__ void f64_tile(F64Smem& s, const MlpF32& w) {
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int fr = lane >> 2, fk = lane & 3;  // a fragment's row (or column) and k of this lane
  constexpr int kFetch = kH1 * kF64Chunk / kF64Threads;
  float pre[kFetch];  // the next W2^T chunk
  auto fetch = [&](int c) {
#pragma unroll
    for (int q = 0; q < kFetch; q++) {
      const int idx = t + q * kF64Threads;
      pre[q] = __ldg(&w.w2t[(size_t)(idx / kF64Chunk) * kH2 + c * kF64Chunk + idx % kF64Chunk]);
    }
  };
  fetch(0);
  for (int idx = t; idx < kH1 * kF64Tile; idx += kF64Threads) {  // layer 1
    const int k = idx / kF64Tile, e = idx % kF64Tile;
    const float4 wk = __ldg(&w.w1b1[k]);
    const double z = (double)wk.w + (double)wk.x * s.r[e][0] + (double)wk.y * s.r[e][1] + (double)wk.z * s.r[e][2];
    s.h1[k * kH1Stride + e] = tanh(z);
  }
  const int em = 32 * (wid & 3), un = 16 * (wid >> 2);  // layer 2: the warp's evaluations and units of a chunk
  double y3[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 1
  for (int c = 0; c < kH2 / kF64Chunk; c++) {
    __syncthreads();  // layer 1 done / previous chunk's h2 readers done
#pragma unroll
    for (int q = 0; q < kFetch; q++) {
      const int idx = t + q * kF64Threads;
      s.buf[idx / kF64Chunk * kW2Stride + idx % kF64Chunk] = (double)pre[q];
    }
    __syncthreads();
    if (c + 1 < kH2 / kF64Chunk) fetch(c + 1);
    double acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    const double* ap = s.h1 + fk * kH1Stride + em + fr;
    const double* bp = s.buf + fk * kW2Stride + un + fr;
#pragma unroll 4
    for (int k = 0; k < kH1; k += 4) {
      double a[4], b[2];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = ap[k * kH1Stride + 8 * i];
#pragma unroll
      for (int j = 0; j < 2; j++) b[j] = bp[k * kW2Stride + 8 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) dmma(acc[i][j], a[i], b[j]);
    }
    __syncthreads();  // every warp is done with the W2 chunk: the buffer takes h2
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int n = un + 8 * j + 2 * fk + h;
        const double bias = (double)__ldg(&w.b2[c * kF64Chunk + n]);
#pragma unroll
        for (int i = 0; i < 4; i++) s.buf[n * kH2Stride + em + 8 * i + fr] = tanh(acc[i][j][h] + bias);
      }
    __syncthreads();
    const double* hp = s.buf + fk * kH2Stride + 8 * wid + fr;
#pragma unroll 4
    for (int n = 0; n < kF64Chunk; n += 4) {
      const double a = hp[n * kH2Stride];
      const int col = c * kF64Chunk + n + fk;
      dmma(y3[0], a, (double)__ldg(&w.w3[fr * kH2 + col]));
      dmma(y3[1], a, fr == 0 ? (double)__ldg(&w.w3[8 * kH2 + col]) : 0.0);
    }
  }
  s.y[8 * wid + fr][2 * fk] = y3[0][0];
  s.y[8 * wid + fr][2 * fk + 1] = y3[0][1];
  if (fk == 0) s.y[8 * wid + fr][8] = y3[1][0];
  __syncthreads();
  for (int e = t; e < kF64Tile; e += kF64Threads) {
    const double rx = s.r[e][0], ry = s.r[e][1], rz = s.r[e][2];
    const double nr = sqrt(rx * rx + ry * ry + rz * rz);
#pragma unroll
    for (int o = 0; o < kOut; o++) {
      double v = s.y[e][o] + (double)__ldg(&w.b3[o]);
      const bool dg = o % 4 == 0;
      if (dg) v += 1.0;
      v = v / nr;
      if (nr < 1e-5) v = dg ? 1.0 : 0.0;
      s.y[e][o] = v;
    }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kF64Threads, 1) k_dense_rows_f64(NearArgs a, MlpF32 w, int* counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  F64Smem& s = *reinterpret_cast<F64Smem*>(smem_raw);
  const int t = threadIdx.x;
  for (;;) {
    __syncthreads();
    if (t == 0) s.item = atomicAdd(counter, 1);
    __syncthreads();
    const int item = s.item;
    if (item >= a.nwork) break;
    const PairWork pw = a.work[item];
    const int end = pair_end(pw);
    const int i0 = pw.first / pw.nJ, i1 = (end - 1) / pw.nJ;  // targets of the item
    for (int i = i0 + t; i <= i1; i += kF64Threads) s.uI[i][0] = s.uI[i][1] = s.uI[i][2] = 0.0;
    for (int t0 = pw.first; t0 < end; t0 += kF64Tile) {
      const int flat = t0 + t;
      const bool valid = t < kF64Tile && flat < end;
      const int i = valid ? flat / pw.nJ : 0, j = valid ? flat - i * pw.nJ : 0;
      if (t < kF64Tile) {
        const float4 xi = __ldg(&a.xI[pw.sI + i]), xj = __ldg(&a.xJ[pw.sJ + j]);
        s.r[t][0] = valid ? (double)xj.x - (double)xi.x : 1.0;
        s.r[t][1] = valid ? (double)xj.y - (double)xi.y : 0.0;
        s.r[t][2] = valid ? (double)xj.z - (double)xi.z : 0.0;
      }
      __syncthreads();
      f64_tile(s, w);
      if (valid) {
        double M[9];
#pragma unroll
        for (int q = 0; q < 9; q++) M[q] = s.y[t][q];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
          for (int c = r + 1; c < 3; c++) {
            const double v = 0.5 * (M[3 * r + c] + M[3 * c + r]);
            M[3 * r + c] = v;
            M[3 * c + r] = v;
          }
        const float4 fj = __ldg(&a.fJ[pw.sJ + j]);
        const double fx = fj.x, fy = fj.y, fz = fj.z;
        atomicAdd(&s.uI[i][0], M[0] * fx + M[1] * fy + M[2] * fz);
        atomicAdd(&s.uI[i][1], M[3] * fx + M[4] * fy + M[5] * fz);
        atomicAdd(&s.uI[i][2], M[6] * fx + M[7] * fy + M[8] * fz);
      }
    }
    __syncthreads();
    for (int q = 3 * i0 + t; q < 3 * (i1 + 1); q += kF64Threads)
      atomicAdd(&a.uI[3 * (size_t)pw.sI + q], (&s.uI[0][0])[q]);
  }
}

}  // namespace

void launch_dense_f64(const NearArgs& a, const MlpF32& w, int* work_counter, int num_sms, cudaStream_t s) {
  if (a.nwork <= 0) return;
  const size_t smem = sizeof(F64Smem);
  HIGNN_CUDA(cudaFuncSetAttribute(k_dense_rows_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  HIGNN_CUDA(cudaMemsetAsync(work_counter, 0, sizeof(int), s));
  const int grid = a.nwork < num_sms ? a.nwork : num_sms;
  k_dense_rows_f64<<<grid, kF64Threads, smem, s>>>(a, w, work_counter);
  HIGNN_CHECK_LAUNCH();
}

}  // namespace hignn
