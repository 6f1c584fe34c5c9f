// Tensor-core (tcgen05) forms of the near field, the ACA queries and the stand-alone evaluation.
//
// All three kernels are persistent (one CTA per SM, up to ~227 KB shared
// memory, 512 TMEM columns) and drive the tile engine of tc_mlp.cuh with two
// streams of 128-evaluation tiles; a server warp per stream supplies the features of
// the next tile while the engine runs the current one, and takes its outputs:
//   k_near_tc : close pairs (I, J) fetched from a global counter by each stream,
//               flattened into tiles; the contraction u_I += M f_J
//               (and u_J += M f_I for J > I) is reduced per particle in shared memory
//               and flushed with one FP64 atomic per particle and component per
//               pair (src/CloseDot.cpp:245-299).
//   k_far_tc  : column / row queries of all active ACA blocks, symmetrised into
//               the C / Q pools (src/FarDot.cpp:348-458, 672-781).
//   k_eval_tc : M(r) for an array of features.
#include "common.h"
#include "kernels.h"
#include "tc_mlp.cuh"

namespace hignn {

namespace {

__device__ __forceinline__ uint8_t* align1k(uint8_t* p) {
  const uint32_t a = tc::saddr(p);
  return p + ((1024u - (a & 1023u)) & 1023u);
}

// Leaves up to kTcLeaf particles (the tensor-core forms need block_size <= 128).
constexpr int kTcLeaf = kTcMaxLeaf;

struct NearStage {
  float uI[kTcLeaf][3], uJ[kTcLeaf][3];
};

// Velocity accumulators, two per stream: of the pair of the current tile and of the next one. (Positions and
// forces are read through L1: the two leaves of a pair are at most 8 KB.)
struct NearTcSmem {
  tc::Smem tcs;
  NearStage st[tc::kStreams][2];
};
static_assert(sizeof(NearTcSmem) + 1024 <= 232448, "near-field shared memory exceeds 227 KB per CTA");

constexpr int kParts = tc::kTile / 32;  // rows of a tile per server lane

// A stream's position in the near-field work: tile [t0, t0 + 128) of a pair with accumulators buf, and
// this lane's rows of it as (i, j). Consecutive tiles advance a row by 128 = di nJ + dj.
struct NearTile {
  PairWork pw;
  int buf, t0, end, di, dj;
  int i[kParts], j[kParts];
  __device__ __forceinline__ bool last() const { return t0 + tc::kTile >= end; }
  __device__ __forceinline__ bool valid(int k, int lane) const { return t0 + 32 * k + lane < end; }
};

// The stream's next close pair (work item `item`) with cleared accumulators b; false at the end of the list.
// `item` becomes the following item of the counter, drawn ahead of its use.
__device__ __forceinline__ bool near_fetch(tc::Server& sv, NearStage& G, const NearArgs& a, int* counter, int b,
                                           int& item, NearTile& c) {
  const int lane = sv.lane;
  if (item >= a.nwork || __any_sync(0xffffffffu, sv.aborted())) return false;
  const PairWork pw = a.work[item];
  if (lane == 0) item = gridDim.x + atomicAdd(counter, 1);
  __syncwarp();  // every lane is done with the pair that last used accumulators b
  c.pw = pw;
  c.buf = b;
  c.t0 = pw.first;
  c.end = pair_end(pw);
  for (int q = 3 * (pw.first / pw.nJ) + lane; q < 3 * ((c.end - 1) / pw.nJ + 1); q += 32) (&G.uI[0][0])[q] = 0.f;
  for (int q = lane; q < 3 * pw.nJ; q += 32) (&G.uJ[0][0])[q] = 0.f;
  item = __shfl_sync(0xffffffffu, item, 0);
  c.di = tc::kTile / pw.nJ;
  c.dj = tc::kTile - c.di * pw.nJ;
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    const int flat = pw.first + 32 * k + lane;
    c.i[k] = flat / pw.nJ;
    c.j[k] = flat - c.i[k] * pw.nJ;
  }
  __syncwarp();
  return true;
}

__device__ __forceinline__ void near_advance(NearTile& c) {
  c.t0 += tc::kTile;
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    c.i[k] += c.di;
    c.j[k] += c.dj;
    if (c.j[k] >= c.pw.nJ) {
      c.j[k] -= c.pw.nJ;
      c.i[k]++;
    }
  }
}

// Features r = x_j - x_i of tile t (a dummy for padding rows).
__device__ __forceinline__ void near_put(tc::Server& sv, const NearArgs& a, const NearTile& c, uint32_t t) {
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    float r[3] = {1.f, 0.f, 0.f};
    if (c.valid(k, sv.lane)) {
      const float4 xi = __ldg(&a.xI[c.pw.sI + c.i[k]]), xj = __ldg(&a.xJ[c.pw.sJ + c.j[k]]);
      r[0] = xj.x - xi.x;
      r[1] = xj.y - xi.y;
      r[2] = xj.z - xi.z;
    }
    sv.put(t, 32 * k + sv.lane, r[0], r[1], r[2]);
  }
  sv.ready();
}

// Contraction of tile t into the pair's shared-memory accumulators: u_I += M f_J and for J > I
// u_J += M f_I (the same M, not transposed; src/CloseDot.cpp:245-299). One warp owns the stream's
// accumulators. The rows of a part are consecutive in j, so its lanes hold distinct j when nJ >= 32.
__device__ __forceinline__ void near_take(tc::Server& sv, NearStage& G, const NearArgs& a, const NearTile& c, uint32_t t) {
  float v[kParts][3];
  const bool distinct = c.pw.nJ >= 32;
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    v[k][0] = v[k][1] = v[k][2] = 0.f;
    if (c.valid(k, sv.lane)) {
      float M[9];
      sv.take(t, 32 * k + sv.lane, M);
      const float4 fj = __ldg(&a.fJ[c.pw.sJ + c.j[k]]);
#pragma unroll
      for (int q = 0; q < 3; q++) v[k][q] = M[3 * q] * fj.x + M[3 * q + 1] * fj.y + M[3 * q + 2] * fj.z;
      if (c.pw.flags & kPairTransposed) {
        const float4 fi = __ldg(&a.fI[c.pw.sI + c.i[k]]);
        float* u = G.uJ[c.j[k]];
#pragma unroll
        for (int q = 0; q < 3; q++) {
          const float w = M[3 * q] * fi.x + M[3 * q + 1] * fi.y + M[3 * q + 2] * fi.z;
          if (distinct)
            u[q] += w;
          else
            atomicAdd(&u[q], w);
        }
      }
    }
    __syncwarp();  // the next part's lanes may hold the same j
  }
  // u_I: the tile's rows cover the targets i0 .. i1; each one's rows are summed over lanes
  const int i0 = c.t0 / c.pw.nJ;
  const int i1 = (min(c.t0 + tc::kTile, c.end) - 1) / c.pw.nJ;
  for (int i = i0; i <= i1; i++) {
    float w[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < kParts; k++)
      if (c.i[k] == i)
#pragma unroll
        for (int q = 0; q < 3; q++) w[q] += v[k][q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < 3; q++) w[q] += __shfl_xor_sync(0xffffffffu, w[q], o);
    if (sv.lane < 3) G.uI[i][sv.lane] += sv.lane == 0 ? w[0] : sv.lane == 1 ? w[1] : w[2];
  }
}

// A finished pair's velocities: one FP64 atomic per particle and component.
__device__ __forceinline__ void near_flush(const tc::Server& sv, const NearStage& G, const NearArgs& a,
                                           const PairWork& pw) {
  __syncwarp();
  const int i0 = pw.first / pw.nJ, i1 = (pair_end(pw) - 1) / pw.nJ;  // targets of the item
  for (int q = 3 * i0 + sv.lane; q < 3 * (i1 + 1); q += 32)
    atomicAdd(&a.uI[3 * (size_t)pw.sI + q], (double)(&G.uI[0][0])[q]);
  if (pw.flags & kPairTransposed)
    for (int q = sv.lane; q < 3 * pw.nJ; q += 32) atomicAdd(&a.uJ[3 * (size_t)pw.sJ + q], (double)(&G.uJ[0][0])[q]);
}

__global__ void __launch_bounds__(tc::kThreads, 1)
    k_near_tc(NearArgs a, TcWeights w, int* work_counter, int* err) {
  extern __shared__ uint8_t smem_raw[];
  NearTcSmem& S = *reinterpret_cast<NearTcSmem*>(align1k(smem_raw));
  tc::run_cta(S.tcs, w, err, [&](tc::Server sv) {
    NearStage* G = S.st[sv.stream];
    // stream 0 of every CTA starts with the item of its block index, the rest come from the counter
    int item = blockIdx.x;
    if (sv.stream != 0) {
      if (sv.lane == 0) item = gridDim.x + atomicAdd(work_counter, 1);
      item = __shfl_sync(0xffffffffu, item, 0);
    }
    NearTile cur{};
    bool have = near_fetch(sv, G[0], a, work_counter, 0, item, cur);
    if (have)
      near_put(sv, a, cur, 0);
    else
      sv.end(0);
    for (uint32_t t = 0; have; t++) {
      // the next tile: the rest of this pair, or the next pair with the other accumulators
      NearTile nxt = cur;
      bool has_next = true;
      if (cur.last())
        has_next = near_fetch(sv, G[cur.buf ^ 1], a, work_counter, cur.buf ^ 1, item, nxt);
      else
        near_advance(nxt);
      if (has_next)
        near_put(sv, a, nxt, t + 1);
      else
        sv.end(t + 1);
      if (!sv.wait(t)) return;  // the launch reports an error
      near_take(sv, G[cur.buf], a, cur, t);
      if (cur.last()) near_flush(sv, G[cur.buf], a, cur.pw);
      cur = nxt;
      have = has_next;
    }
  });
}

struct FarTcSmem {
  tc::Smem tcs;
};

// This lane's rows of a far tile: their entries in the C / Q pool (-1: none).
struct FarTile {
  long long dst[kParts];
};

__device__ __forceinline__ void far_put(tc::Server& sv, const FarArgs& a, int which, int nact, int tot, int tile,
                                        uint32_t t, FarTile& c) {
  const int32_t* pre = which ? a.preJ : a.preI;
  // the block of the tile's first row: 32-way search of the active blocks' prefix
  const int g0 = tile * tc::kTile;
  int lo = 0, hi = nact;  // pre[lo] <= g0 < pre[hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32, p = lo + sv.lane * step;
    const unsigned m = __ballot_sync(0xffffffffu, sv.lane > 0 && p < hi && pre[p] <= g0);
    lo += __popc(m) * step;
    hi = min(hi, lo + step);
  }
  // The rows' loads depend on one another (block, its state, the pivot, positions): taken step by step for all
  // of the lane's rows, so that the four chains run at once (700 spheres, one tile per launch: 16.4 instead of 18.2 us,
  // 131,072 spheres: queries 49.0 instead of 52.0 ms).
  int b[kParts], loc[kParts];
  bool in[kParts];
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    const int g = g0 + 32 * k + sv.lane;
    in[k] = g < tot;
    while (in[k] && pre[lo + 1] <= g) lo++;
    b[k] = a.act[lo];
    loc[k] = g - pre[lo];
  }
  float4 xi[kParts], xj[kParts];
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    const FarBlock& bk = a.blocks[b[k]];
    const int it = a.state[b[k]].k;
    const int pivot = (which == 0 ? a.cols : a.rows)[(size_t)b[k] * a.ldr + it];
    const int own = in[k] ? loc[k] : 0;  // padding rows repeat the block's first
    xj[k] = a.x[bk.sJ + (which == 0 ? pivot : own)];
    xi[k] = a.x[bk.sI + (which == 0 ? own : pivot)];
    c.dst[k] = !in[k] ? -1 : which == 0 ? bk.cOff + (int64_t)it * bk.nI + own : bk.qOff + (int64_t)it * bk.nJ + own;
  }
#pragma unroll
  for (int k = 0; k < kParts; k++) {
    float r[3] = {1.f, 0.f, 0.f};
    if (in[k]) {
      r[0] = xj[k].x - xi[k].x;
      r[1] = xj[k].y - xi[k].y;
      r[2] = xj[k].z - xi[k].z;
    }
    sv.put(t, 32 * k + sv.lane, r[0], r[1], r[2]);
  }
  sv.ready();
}

// symmetrised 3x3 of each row into the C / Q pool (src/FarDot.cpp:445-456: diagonal copied,
// off-diagonal halved sum)
__device__ __forceinline__ void far_take(tc::Server& sv, pool_t* pool, const FarTile& c, uint32_t t) {
#pragma unroll
  for (int k = 0; k < kParts; k++)
    if (c.dst[k] >= 0) {
      float M[9];
      sv.take(t, 32 * k + sv.lane, M);
      pool_t* dst = pool + 9 * c.dst[k];
#pragma unroll
      for (int q = 0; q < 9; q++) {
        const int rr = q / 3, cc = q % 3;
        dst[q] = rr == cc ? M[q] : 0.5f * __fadd_rn(M[3 * rr + cc], M[3 * cc + rr]);  // the FP32 half-sum is exact in FP64 too
      }
    }
}

__global__ void __launch_bounds__(tc::kThreads, 1)
    k_far_tc(FarArgs a, TcWeights w, int which, int* err) {
  extern __shared__ uint8_t smem_raw[];
  FarTcSmem& S = *reinterpret_cast<FarTcSmem*>(align1k(smem_raw));
  const int nact = a.ctr[kCtrActive];
  const int tot = which ? a.ctr[kCtrTotJ] : a.ctr[kCtrTotI];
  if ((int)blockIdx.x * tc::kTile >= tot) return;  // uniform: before any setup
  tc::run_cta(S.tcs, w, err, [&](tc::Server sv) {
    pool_t* pool = which ? a.Q : a.C;
    int tile = blockIdx.x + gridDim.x * sv.stream;
    FarTile cur{};
    bool have = tile * tc::kTile < tot;
    if (have)
      far_put(sv, a, which, nact, tot, tile, 0, cur);
    else
      sv.end(0);
    for (uint32_t t = 0; have; t++) {
      tile += tc::kStreams * gridDim.x;
      const bool has_next = tile * tc::kTile < tot;
      FarTile nxt{};
      if (has_next)
        far_put(sv, a, which, nact, tot, tile, t + 1, nxt);
      else
        sv.end(t + 1);
      if (!sv.wait(t)) return;
      far_take(sv, pool, cur, t);
      cur = nxt;
      have = has_next;
    }
  });
  if (threadIdx.x == 0 && blockIdx.x == 0) atomicAdd(a.evals, (unsigned long long)tot);
}

struct EvalTcSmem {
  tc::Smem tcs;
};

__global__ void __launch_bounds__(tc::kThreads, 1)
    k_eval_tc(const float* __restrict__ r, float* __restrict__ y, int64_t n, TcWeights w, int* err) {
  extern __shared__ uint8_t smem_raw[];
  EvalTcSmem& S = *reinterpret_cast<EvalTcSmem*>(align1k(smem_raw));
  tc::run_cta(S.tcs, w, err, [&](tc::Server sv) {
    auto put = [&](int64_t tile, uint32_t t) {
#pragma unroll
      for (int k = 0; k < kParts; k++) {
        const int64_t g = tile * tc::kTile + 32 * k + sv.lane;
        const bool in = g < n;
        sv.put(t, 32 * k + sv.lane, in ? r[3 * g] : 1.f, in ? r[3 * g + 1] : 0.f, in ? r[3 * g + 2] : 0.f);
      }
      sv.ready();
    };
    int64_t tile = blockIdx.x + (int64_t)gridDim.x * sv.stream;
    bool have = tile * tc::kTile < n;
    if (have)
      put(tile, 0);
    else
      sv.end(0);
    for (uint32_t t = 0; have; t++) {
      const int64_t nt = tile + tc::kStreams * (int64_t)gridDim.x;
      const bool has_next = nt * tc::kTile < n;
      if (has_next)
        put(nt, t + 1);
      else
        sv.end(t + 1);
      if (!sv.wait(t)) return;
#pragma unroll
      for (int k = 0; k < kParts; k++) {
        const int64_t g = tile * tc::kTile + 32 * k + sv.lane;
        if (g < n) {
          float M[9];
          sv.take(t, 32 * k + sv.lane, M);
#pragma unroll
          for (int q = 0; q < 9; q++) y[9 * g + q] = M[q];
        }
      }
      tile = nt;
      have = has_next;
    }
  });
}

template <class K>
void set_smem(K kernel, size_t bytes, cudaStream_t s) {
  set_max_dynamic_smem(kernel, bytes, s);
}

}  // namespace

size_t near_tc_smem_bytes() { return sizeof(NearTcSmem) + 1024; }

void launch_near_tc(const NearArgs& a, const TcWeights& w, int* work_counter, int* err, int num_sms,
                    cudaStream_t s) {
  if (a.nwork <= 0) return;
  const size_t smem = sizeof(NearTcSmem) + 1024;
  set_smem(k_near_tc, smem, s);
  HIGNN_CUDA(cudaMemsetAsync(work_counter, 0, sizeof(int), s));
  const int grid = a.nwork < num_sms ? a.nwork : num_sms;
  k_near_tc<<<grid, tc::kThreads, smem, s>>>(a, w, work_counter, err);
  HIGNN_CHECK_LAUNCH();
}

void launch_far_tc(const FarArgs& a, const TcWeights& w, int which, int* err, int num_sms, cudaStream_t s) {
  const size_t smem = sizeof(FarTcSmem) + 1024;
  set_smem(k_far_tc, smem, s);
  k_far_tc<<<num_sms, tc::kThreads, smem, s>>>(a, w, which, err);
  HIGNN_CHECK_LAUNCH();
}

void launch_eval_tc(const float* r, float* y, int64_t n, const TcWeights& w, int* err, int num_sms,
                    cudaStream_t s) {
  if (n <= 0) return;
  const size_t smem = sizeof(EvalTcSmem) + 1024;
  set_smem(k_eval_tc, smem, s);
  const int64_t tiles = (n + tc::kTile - 1) / tc::kTile;
  const int grid = (int)(tiles < num_sms ? tiles : num_sms);
  k_eval_tc<<<grid, tc::kThreads, smem, s>>>(r, y, n, w, err);
  HIGNN_CHECK_LAUNCH();
}

}  // namespace hignn
