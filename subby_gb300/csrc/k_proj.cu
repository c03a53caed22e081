// Eigenbasis projections of the walk's raw staging (k_qwalk) at A = 16, 20,
// 32 (subby/oracle/oracle.py:966-1003): in place, one row of A floats per
// (branch, column),
//   stage_a: D~ = Vd^T (s D),   stage_b: U~ = Vu^T U, a leaf's from the table
//   Ut by its token (the walk leaves those rows unwritten).
//
// One thread per row.  Vd and Vu are kernel parameters and every index into
// them is a compile-time constant, so the multiply-adds take them from the
// constant bank and no matrix element passes through the load unit.  Tiles
// of 128 rows go through shared memory by bulk copies.  Rows of A = 16 and
// 32 floats keep their 16-byte chunk k at position (k + rot) mod (A / 4)
// (stage_rot), as the walk writes and k_acc reads them: the lanes of a
// quarter-warp, a row each, then touch different banks.
//
// Bound by memory: A = 20, R = 199, C = 20011 moves 1.05 GB in 183 us (5.8
// TB/s, 0.85 of the measured copy rate) while the multiply-adds run at 13e12
// per second; A = 16, R = 99, C = 4003 takes 19 us.  Projecting inside the
// accumulation instead (rows through its shared-memory ring) measured 730 us
// against 183 + 312 us here: eight warps per SM did not cover the latency of
// its row passes.
#include <algorithm>

#include "common.cuh"
#include "walk.cuh"

namespace subby {
namespace {

template <int A>
struct ProjV {
  float d[A * A], u[A * A];
};
constexpr int kPRows = 128;

template <int A>
__global__ void __launch_bounds__(kPRows)
    k_proj(const __grid_constant__ ProjV<A> W, const KParams P, float *__restrict__ stage_a,
           float *__restrict__ stage_b, int c_base, int c_count) {
  extern __shared__ __align__(128) float sm[];   // the tile's rows, then Ut
  __shared__ __align__(8) uint64_t mbar;
  __shared__ int s_err;
  float *Uts = sm + kPRows * A;
  const int t = threadIdx.x;
  const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar);
  const uint32_t srow = (uint32_t)__cvta_generic_to_shared(sm);
  const long long nrows = (long long)(P.R - 1) * c_count;
  const long long ntiles = (nrows + kPRows - 1) / kPRows;
  for (int i = t; i < (A + 1) * A; i += kPRows) Uts[i] = __ldg(P.tab + P.off.Ut + i);
  if (t == 0) {
    s_err = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  __syncthreads();
  uint32_t phase = 0;
  for (long long it = blockIdx.x; it < 2 * ntiles; it += gridDim.x) {
    const bool up = it >= ntiles;
    const long long r0 = (up ? it - ntiles : it) * kPRows;
    const int rows = (int)min((long long)kPRows, nrows - r0);
    float *g = (up ? stage_b : stage_a) + r0 * A;
    const long long r = min(r0 + t, nrows - 1);
    const int n = 1 + (int)(r / c_count), c = (int)(r % c_count);
    const bool leaf = up && __ldg(P.leaf + n) != 0;
    const int code = leaf ? btcode(__ldg(P.aln + (size_t)n * P.C + c_base + c), A) : 0;
    // a tile of leaf rows only has nothing to load
    const bool load = __syncthreads_or(!leaf) != 0;
    if (load) {
      if (t == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(rows * A * 4) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(srow),
                     "l"(g), "r"(rows * A * 4), "r"(mb) : "memory");
      }
      __syncwarp();
      if (!mbar_wait(mb, phase & 1)) s_err = 1;
      ++phase;
    }
    float *row = sm + t * A;
    const int rot = stage_rot(A, c);
    if (leaf) {
#pragma unroll
      for (int k = 0; k < A / 4; ++k)
        *reinterpret_cast<float4 *>(row + stage_chunk<A>(k, rot)) = *reinterpret_cast<const float4 *>(Uts + code * A + 4 * k);
    } else {
      float x[A], y[A];
#pragma unroll
      for (int k = 0; k < A / 4; ++k) {
        const float4 v = *reinterpret_cast<const float4 *>(row + stage_chunk<A>(k, rot));
        x[4 * k] = v.x, x[4 * k + 1] = v.y, x[4 * k + 2] = v.z, x[4 * k + 3] = v.w;
      }
#pragma unroll
      for (int o = 0; o < A; ++o) y[o] = 0.f;
      if (up) {
#pragma unroll
        for (int k = 0; k < A; ++k)
#pragma unroll
          for (int o = 0; o < A; ++o) y[o] = fmaf(x[k], W.u[k * A + o], y[o]);
      } else {
#pragma unroll
        for (int k = 0; k < A; ++k)
#pragma unroll
          for (int o = 0; o < A; ++o) y[o] = fmaf(x[k], W.d[k * A + o], y[o]);
      }
#pragma unroll
      for (int k = 0; k < A / 4; ++k)
        *reinterpret_cast<float4 *>(row + stage_chunk<A>(k, rot)) =
            make_float4(y[4 * k], y[4 * k + 1], y[4 * k + 2], y[4 * k + 3]);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t == 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(g), "r"(srow), "r"(rows * A * 4)
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      // the rows are read out before the next tile's copy or stores
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    __syncwarp();
    // (every thread passes the next tile's barrier before it writes a row)
  }
  if (t == 0) {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (s_err && P.err) atomicAdd(P.err, 1);
  }
}

template <int A>
int proj_launch(const KParams &p, const float *vd, const float *vu, float *sa, float *sb, int c_base, int c_count,
                int nsm, cudaStream_t s) {
  ProjV<A> W;
  for (int i = 0; i < A * A; ++i) W.d[i] = vd[i], W.u[i] = vu[i];
  const long long tiles = 2 * (((long long)(p.R - 1) * c_count + kPRows - 1) / kPRows);
  const int grid = (int)std::max<long long>(1, std::min<long long>(tiles, (long long)nsm * (A == 32 ? 6 : 8)));
  const size_t smem = (size_t)(kPRows + A + 1) * A * sizeof(float);
  k_proj<A><<<grid, kPRows, smem, s>>>(W, p, sa, sb, c_base, c_count);
  return (int)cudaGetLastError();
}

}  // namespace

bool proj_supported(int A) { return A == 16 || A == 20 || A == 32; }

int launch_proj(const KParams &p, int A, const float *vd, const float *vu, float *sa, float *sb, int c_base,
                int c_count, int nsm, cudaStream_t s) {
  switch (A) {
    case 16: return proj_launch<16>(p, vd, vu, sa, sb, c_base, c_count, nsm, s);
    case 20: return proj_launch<20>(p, vd, vu, sa, sb, c_base, c_count, nsm, s);
    case 32: return proj_launch<32>(p, vd, vu, sa, sb, c_base, c_count, nsm, s);
    default: return -1;
  }
}

}  // namespace subby
