// Plain FP32 near field: fused pair features -> two-body network -> 3x3 contraction.
//
// Restates HignnModel::CloseDot (src/CloseDot.cpp:177-299): for every close
// leaf pair (I, J), u_I[i] += M(x_J[j] - x_I[i]) f_J[j], and when J > I with
// symmetry on, u_J[j] += (the same M) f_I[i] (not transposed, not
// re-evaluated). The reference writes the features to HBM, runs libtorch and
// scatters with one FP64 atomic per evaluation; here one CTA owns a pair (or a run of a pair's
// evaluations, where there are few pairs), evaluates 64 at a time, reduces
// the contributions per particle in shared memory and issues one FP64 atomic
// per particle and component per work item. With kSymmetrize the 3x3 is replaced by
// 0.5 (M + M^T) and only u_I is updated: DenseDot's contraction
// (src/DenseDot.cpp:227-243).
#include "common.h"
#include "kernels.h"
#include "mlp_simt.cuh"

namespace hignn {

namespace {

struct NearSmem {
  simt::Smem mlp;
  float uI[kMaxLeaf][3], uJ[kMaxLeaf][3];
  int item;
};

template <int Rows>
__global__ void __launch_bounds__(simt::kThreads, simt::kCtasPerSm)
    k_near_simt(NearArgs a, MlpF32 w, int* work_counter) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  NearSmem& s = *reinterpret_cast<NearSmem*>(smem_raw);
  const int t = threadIdx.x, lane = t & 31;
  const int row = Rows * (t >> 5) + lane;  // lanes 0 .. Rows - 1 of a warp: its evaluations of a tile
  simt::load_weights(s.mlp, w);
  for (;;) {
    __syncthreads();
    if (t == 0) s.item = atomicAdd(work_counter, 1);
    __syncthreads();
    const int item = s.item;
    if (item >= a.nwork) break;
    const PairWork pw = a.work[item];
    const bool trans = (pw.flags & kPairTransposed) != 0;
    const bool symm = (pw.flags & kPairSymmetrize) != 0;
    const int end = pair_end(pw);
    const int i0 = pw.first / pw.nJ, i1 = (end - 1) / pw.nJ;  // targets of the item
    for (int q = 3 * i0 + t; q < 3 * (i1 + 1); q += simt::kThreads) (&s.uI[0][0])[q] = 0.f;
    for (int q = t; q < 3 * pw.nJ; q += simt::kThreads) (&s.uJ[0][0])[q] = 0.f;
    for (int t0 = pw.first; t0 < end; t0 += simt::kWarps * Rows) {
      const int flat = t0 + row;
      const bool valid = lane < Rows && flat < end;
      const int i = valid ? flat / pw.nJ : 0, j = valid ? flat - i * pw.nJ : 0;
      if (lane < Rows) {
        const float4 xi = __ldg(&a.xI[pw.sI + i]), xj = __ldg(&a.xJ[pw.sJ + j]);
        s.mlp.r[row] = valid ? make_float4(xj.x - xi.x, xj.y - xi.y, xj.z - xi.z, 0.f) : make_float4(1.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
      simt::mlp_tile<Rows>(s.mlp, w);
      if (valid) {
        float M[9];
#pragma unroll
        for (int q = 0; q < 9; q++) M[q] = s.mlp.y[row][q];
        if (symm) {
#pragma unroll
          for (int r = 0; r < 3; r++)
#pragma unroll
            for (int c = r + 1; c < 3; c++) {
              const float v = 0.5f * (M[3 * r + c] + M[3 * c + r]);
              M[3 * r + c] = v;
              M[3 * c + r] = v;
            }
        }
        const float4 fj = __ldg(&a.fJ[pw.sJ + j]);
        atomicAdd(&s.uI[i][0], M[0] * fj.x + M[1] * fj.y + M[2] * fj.z);
        atomicAdd(&s.uI[i][1], M[3] * fj.x + M[4] * fj.y + M[5] * fj.z);
        atomicAdd(&s.uI[i][2], M[6] * fj.x + M[7] * fj.y + M[8] * fj.z);
        if (trans) {
          const float4 fi = __ldg(&a.fI[pw.sI + i]);
          atomicAdd(&s.uJ[j][0], M[0] * fi.x + M[1] * fi.y + M[2] * fi.z);
          atomicAdd(&s.uJ[j][1], M[3] * fi.x + M[4] * fi.y + M[5] * fi.z);
          atomicAdd(&s.uJ[j][2], M[6] * fi.x + M[7] * fi.y + M[8] * fi.z);
        }
      }
    }
    __syncthreads();
    for (int q = 3 * i0 + t; q < 3 * (i1 + 1); q += simt::kThreads)
      atomicAdd(&a.uI[3 * (size_t)pw.sI + q], (double)(&s.uI[0][0])[q]);
    if (trans)
      for (int q = t; q < 3 * pw.nJ; q += simt::kThreads)
        atomicAdd(&a.uJ[3 * (size_t)pw.sJ + q], (double)(&s.uJ[0][0])[q]);
  }
}

template <int Rows>
void near_simt(const NearArgs& a, const MlpF32& w, int* work_counter, int num_sms, cudaStream_t stream) {
  const size_t smem = sizeof(NearSmem);
  set_max_dynamic_smem(k_near_simt<Rows>, smem, stream);
  HIGNN_CUDA(cudaMemsetAsync(work_counter, 0, sizeof(int), stream));
  const int ctas = simt::kCtasPerSm * num_sms;
  const int grid = a.nwork < ctas ? a.nwork : ctas;
  k_near_simt<Rows><<<grid, simt::kThreads, smem, stream>>>(a, w, work_counter);
  HIGNN_CHECK_LAUNCH();
}

}  // namespace

int plain_tile(int64_t evals, int num_sms) {
  return simt::kWarps * simt::rows_per_warp(evals, (int64_t)simt::kCtasPerSm * num_sms);
}

void launch_near_simt(const NearArgs& a, const MlpF32& w, int* work_counter, int num_sms,
                      cudaStream_t stream) {
  if (a.nwork <= 0) return;
  const int tile = a.evals > 0 ? plain_tile(a.evals, num_sms) : simt::kTile;
  if (tile == simt::kTile / 4)
    near_simt<simt::kRows / 4>(a, w, work_counter, num_sms, stream);
  else if (tile == simt::kTile / 2)
    near_simt<simt::kRows / 2>(a, w, work_counter, num_sms, stream);
  else
    near_simt<simt::kRows>(a, w, work_counter, num_sms, stream);
}

}  // namespace hignn
