// Gradient of sum_c g_c logL_c for reversible models from the walk's eigen
// staging (D~ = s Vd^T D, U~ = Vu^T U per branch and column, unmasked).  Both
// gradients of subby/jax/vjp.py:62-133 and the exchangeability gradient are
// functions of one A x A matrix per branch,
//   X_n = sum_c g_c D~_nc (x) U~_nc :
//   d/dt_n = sum_k mu_k e^{mu_k t_n} X_n[k][k],  d/dS~ = V (sum_n J_n o X_n) V^T
// (k_xform contracts X_n with the branch's coefficients, k_xsum adds the
// branches up, in FP64).
// k_xgram: per (branch, block of 4096 columns) each thread owns a 4 x 4 block
// of (k, l) for a subset of the columns (two 16-byte loads and 16 FMAs per
// column), the column subsets are reduced in shared memory and the block's
// sum is added to X_n in FP64 (one atomic per entry per block).
#include <algorithm>

#include "common.cuh"
#include "walk.cuh"

namespace subby {
namespace {

constexpr int kXThreads = 256;
constexpr int kXCols = 4096;

template <int A>
__global__ void __launch_bounds__(kXThreads) k_xgram(const float *__restrict__ sa, const float *__restrict__ sb,
                                                     const float *__restrict__ g, int c_base, int c_count, int R,
                                                     double *__restrict__ X) {
  constexpr int KB = A / 4, NB = KB * KB;
  constexpr int GROUPS = (kXThreads / NB) > 0 ? kXThreads / NB : 1;
  constexpr int THREADS = NB * GROUPS;
  static_assert(NB <= kXThreads, "A too large");
  __shared__ float s_part[THREADS * 16];
  const int t = threadIdx.x;
  const bool busy = t < THREADS;
  const int grp = busy ? t / NB : 0, b = busy ? t % NB : 0;
  const int kb = b / KB, lb = b % KB;
  const int nblk = (c_count + kXCols - 1) / kXCols;
  const long long items = (long long)(R - 1) * nblk;
  for (long long it = blockIdx.x; it < items; it += gridDim.x) {
    const int n = 1 + (int)(it / nblk);
    const int c0 = (int)(it % nblk) * kXCols, c1 = min(c_count, c0 + kXCols);
    float acc[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = 0.f;
    auto add = [&](float4 d, const float4 u, float w) {
      d.x *= w, d.y *= w, d.z *= w, d.w *= w;
      const float dv[4] = {d.x, d.y, d.z, d.w}, uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[4 * i + j] = fmaf(dv[i], uv[j], acc[4 * i + j]);
    };
    auto ld = [&](const float *base, int c, int blk) {
      return __ldg(reinterpret_cast<const float4 *>(base + ((size_t)(n - 1) * c_count + c) * A) + blk);
    };
    if (busy) {
      int c = c0 + grp;
      // four columns' loads in flight before their FMAs (the pass is load-latency-bound)
      for (; c + 3 * GROUPS < c1; c += 4 * GROUPS) {
        float4 d[4], u[4];
        float w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          d[q] = ld(sa, c + q * GROUPS, kb);
          u[q] = ld(sb, c + q * GROUPS, lb);
          w[q] = g ? __ldg(g + c_base + c + q * GROUPS) : 1.f;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) add(d[q], u[q], w[q]);
      }
      for (; c < c1; c += GROUPS) add(ld(sa, c, kb), ld(sb, c, lb), g ? __ldg(g + c_base + c) : 1.f);
    }
    __syncthreads();  // the previous item's reads of s_part are done
    if (busy)
#pragma unroll
      for (int q = 0; q < 16; ++q) s_part[(grp * NB + b) * 16 + q] = acc[q];
    __syncthreads();
    for (int e = t; e < NB * 16; e += blockDim.x) {
      double s = 0.0;
      for (int gi = 0; gi < GROUPS; ++gi) s += (double)s_part[gi * NB * 16 + e];
      const int bb = e / 16, q = e % 16;
      const int k = 4 * (bb / KB) + q / 4, l = 4 * (bb % KB) + q % 4;
      atomicAdd(X + ((size_t)n * A + k) * A + l, s);
    }
  }
}

// The same sums at A = 16, 20, 32, addition by addition (a column subset's
// FP32 sum runs over every GROUPS-th column of a block of 4096): k_xgram's
// 4 x 4 blocks load 8 floats for 16 multiply-adds, which left it bound by the
// load pipe at 1.7 TB/s.  Here a lane owns a 4 x LW block (LW = A, at A = 32
// half a row): 4 + LW floats for 4 LW multiply-adds, and a CTA takes NB
// branches of the same columns, whose rows come through a ring of bulk
// copies.  The subsets are added in their order, as k_xgram does, so that the
// gradients of up to 4096 columns are the same in every call (A = 20, R = 399,
// 50000 columns, 3.2 GB: 735 us; with an FP64 atomic per entry and subset 823).
template <int A>
struct XG {
  static constexpr int LW = A == 32 ? 16 : A;
  static constexpr int NT = (A / 4) * (A / LW);                 // blocks of X
  static constexpr int GROUPS = kXThreads / ((A / 4) * (A / 4)); // column subsets
  static constexpr int TPB = NT * GROUPS;                       // threads per branch
  static constexpr int NB = kXThreads / TPB;                    // branches per CTA
  static constexpr int IT = A == 32 ? 8 : A == 16 ? 2 : 4;      // columns per lane and ring stage
  static constexpr int TC = GROUPS * IT;                        // columns per ring stage
  static constexpr int NS = 3;
  static constexpr int ROWS = TC * A;                           // floats of a stage's rows of one vector and branch
  static constexpr int STAGE = NB * 2 * ROWS;
  static constexpr int FLOATS = NS * STAGE;
  static constexpr int OUT = NT * LW;                           // a branch's entries of one of the four rows of every block
  static_assert(NB * GROUPS * OUT <= STAGE, "the subsets' sums take a ring stage");
};

template <int A>
__global__ void __launch_bounds__(kXThreads, 2)
    k_xgram_wide(const float *__restrict__ sa, const float *__restrict__ sb, const float *__restrict__ g, int c_base,
                 int c_count, int R, double *__restrict__ X, int *err) {
  using G = XG<A>;
  constexpr int LW = G::LW, TC = G::TC;
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(8) uint64_t mbar[G::NS];
  __shared__ int s_err;
  const int t = threadIdx.x;
  const int br = t / G::TPB, r = t % G::TPB, grp = r / G::NT, tile = r % G::NT;
  const int kt = tile / (A / LW), lt = tile % (A / LW);
  if (t == 0) {
    s_err = 0;
    for (int i = 0; i < G::NS; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&mbar[i]))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  __syncthreads();
  const int nblk = (c_count + kXCols - 1) / kXCols;
  const int nbg = (R - 1 + G::NB - 1) / G::NB;   // groups of NB branches
  const int items = nbg * nblk;
  int pit = blockIdx.x, pc = -1;   // the ring's next load (thread 0)
  uint32_t pos = 0, ppos = 0;
  auto load = [&]() {
    if (pit >= items) return;
    const int n0 = pit / nblk * G::NB, b0 = (pit % nblk) * kXCols, b1 = min(c_count, b0 + kXCols);
    if (pc < 0) pc = b0;
    const uint32_t bytes = (uint32_t)min(TC, b1 - pc) * A * 4;
    const int nb = min(G::NB, R - 1 - n0);
    float *d = sm + (ppos % G::NS) * G::STAGE;
    const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar[ppos % G::NS]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(2 * nb * bytes) : "memory");
    for (int i = 0; i < nb; ++i) {
      const size_t off = ((size_t)(n0 + i) * c_count + pc) * A;
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(d + 2 * i * G::ROWS)), "l"(sa + off), "r"(bytes), "r"(mb)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(d + (2 * i + 1) * G::ROWS)), "l"(sb + off), "r"(bytes),
                   "r"(mb) : "memory");
    }
    ++ppos;
    pc += TC;
    if (pc >= b1) {
      pc = -1;
      pit += gridDim.x;
    }
  };
  if (t == 0)
    for (int i = 0; i < G::NS - 1; ++i) load();
  __syncwarp();
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int n = it / nblk * G::NB + br;   // branch - 1
    const int b0 = (it % nblk) * kXCols, b1 = min(c_count, b0 + kXCols);
    const bool busy = br < G::NB && n < R - 1;
    float2 acc[4][LW / 2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < LW / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
    for (int c = b0; c < b1; c += TC, ++pos) {
      const int cnt = min(TC, b1 - c);
      auto weight = [&](int x) { return g && x < cnt ? __ldg(g + c_base + c + x) : 1.f; };
      float w = weight(grp);   // of the lane's next column, a column ahead of its use
      // every warp is past the stage that this refills
      __syncthreads();
      if (t == 0) load();
      __syncwarp();
      if (!mbar_wait((uint32_t)__cvta_generic_to_shared(&mbar[pos % G::NS]), (pos / G::NS) & 1)) s_err = 1;
      const float *st = sm + (pos % G::NS) * G::STAGE + 2 * br * G::ROWS;
      if (busy)
#pragma unroll 1
        for (int x = grp; x < cnt; x += G::GROUPS) {
          const float wx = w;
          w = weight(x + G::GROUPS);
          const int rot = stage_rot(A, x);   // (the block starts at rotation 0)
          const float4 av = *reinterpret_cast<const float4 *>(st + x * A + stage_chunk<A>(kt, rot));
          const float a[4] = {av.x * wx, av.y * wx, av.z * wx, av.w * wx};
          const float *ur = st + G::ROWS + x * A;
#pragma unroll
          for (int j = 0; j < LW / 4; ++j) {
            const float4 u = *reinterpret_cast<const float4 *>(ur + stage_chunk<A>(lt * (LW / 4) + j, rot));
            const float2 u0 = make_float2(u.x, u.y), u1 = make_float2(u.z, u.w);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float2 aa = make_float2(a[q], a[q]);
              acc[q][2 * j] = __ffma2_rn(aa, u0, acc[q][2 * j]);
              acc[q][2 * j + 1] = __ffma2_rn(aa, u1, acc[q][2 * j + 1]);
            }
          }
        }
    }
    // The subsets' sums through the ring stage just read, which the next
    // item's first barrier hands to the bulk copies: one row of the 4 x LW
    // blocks at a time, [branch][subset][block][LW].
    float *part = sm + ((pos + G::NS - 1) % G::NS) * G::STAGE;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      __syncthreads();
      if (busy)
#pragma unroll
        for (int j = 0; j < LW / 4; ++j)
          *reinterpret_cast<float4 *>(part + ((br * G::GROUPS + grp) * G::NT + tile) * LW + 4 * j) =
              make_float4(acc[q][2 * j].x, acc[q][2 * j].y, acc[q][2 * j + 1].x, acc[q][2 * j + 1].y);
      __syncthreads();
      for (int e = t; e < G::NB * G::OUT; e += kXThreads) {
        const int b = e / G::OUT, r2 = e % G::OUT, b2 = it / nblk * G::NB + b;
        if (b2 >= R - 1) break;
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < G::GROUPS; ++i) s += (double)part[(b * G::GROUPS + i) * G::OUT + r2];
        const int tl = r2 / LW;   // its block
        atomicAdd(X + ((size_t)(b2 + 1) * A + 4 * (tl / (A / LW)) + q) * A + (tl % (A / LW)) * LW + r2 % LW, s);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (t == 0 && s_err && err) atomicAdd(err, 1);
}

// One CTA per branch, FP64: grad_t[n] = sum_k mu_k e^{mu_k t_n} X_n[k][k], and
// X_n becomes J_n o X_n with the 1e-8 degeneracy rule of J
// (subby/oracle/oracle.py:931-959).  tab64: V, S, mu, t, pi.
__global__ void k_xform(double *__restrict__ X, const double *__restrict__ tab64, int R, int A,
                        double *__restrict__ grad_t) {
  extern __shared__ double sd[];
  double *x = sd, *ek = sd + A * A;   // X_n, e^{mu t_n}
  const double *mu = tab64 + 2 * A * A, *tt = mu + A;
  const int n = 1 + blockIdx.x;
  const double t = tt[n];
  for (int k = threadIdx.x; k < A; k += blockDim.x) ek[k] = exp(mu[k] * t);
  for (int e = threadIdx.x; e < A * A; e += blockDim.x) x[e] = X[(size_t)n * A * A + e];
  __syncthreads();
  for (int e = threadIdx.x; e < A * A; e += blockDim.x) {
    const int k = e / A, l = e % A;
    const double d = mu[k] - mu[l];
    const double J = fabs(d) < 1e-8 ? t * ek[k] : (ek[k] - ek[l]) / d;
    X[(size_t)n * A * A + e] = J * x[e];
  }
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < A; ++k) s += mu[k] * ek[k] * x[k * A + k];
    grad_t[n] = s;
  }
}

// Cg = sum_n of k_xform's matrices, in a fixed order: a lane per entry, each
// warp every kSumWarps-th branch, then the warps in turn.  Behind Cg goes the
// status word of the kernels before, for the host's one readback.
constexpr int kSumWarps = 8;
__global__ void __launch_bounds__(32 * kSumWarps) k_xsum(const double *__restrict__ X, int R, int AA,
                                                         double *__restrict__ Cg, const int *__restrict__ err) {
  __shared__ double part[kSumWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  double s = 0.0;
  if (e < AA)
#pragma unroll 8
    for (int n = 1 + w; n < R; n += kSumWarps) s += X[(size_t)n * AA + e];
  part[w][lane] = s;
  __syncthreads();
  if (w == 0 && e < AA) {
    for (int i = 1; i < kSumWarps; ++i) s += part[i][lane];
    Cg[e] = s;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<int *>(Cg + AA) = *err;
}

template <int A>
int xgram_wide(const KParams &p, const float *sa, const float *sb, const float *g, int c_base, int c_count, double *X,
               int nsm, cudaStream_t s) {
  using G = XG<A>;
  const size_t smem = (size_t)G::FLOATS * sizeof(float);
  cudaError_t e = allow_smem<k_xgram_wide<A>>();
  if (e != cudaSuccess) return (int)e;
  const int items = ((p.R - 1 + G::NB - 1) / G::NB) * ((c_count + kXCols - 1) / kXCols);
  k_xgram_wide<A><<<std::max(1, std::min(items, 2 * nsm)), kXThreads, smem, s>>>(sa, sb, g, c_base, c_count, p.R, X,
                                                                               p.err);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_xform(double *X, const double *tab64, int R, int A, double *grad_t, double *Cg, const int *err,
                 cudaStream_t s) {
  const size_t smem = (size_t)(A * A + A) * sizeof(double);
  cudaError_t e = allow_smem<k_xform>();
  if (e != cudaSuccess) return (int)e;
  k_xform<<<R - 1, 256, smem, s>>>(X, tab64, R, A, grad_t);
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  k_xsum<<<(A * A + 31) / 32, 32 * kSumWarps, 0, s>>>(X, R, A * A, Cg, err);
  return (int)cudaGetLastError();
}

int launch_xgram(const KParams &p, int A, const float *sa, const float *sb, const float *g, int c_base, int c_count,
                 double *X, int nsm, cudaStream_t s) {
  switch (A) {
    case 16: return xgram_wide<16>(p, sa, sb, g, c_base, c_count, X, nsm, s);
    case 20: return xgram_wide<20>(p, sa, sb, g, c_base, c_count, X, nsm, s);
    case 32: return xgram_wide<32>(p, sa, sb, g, c_base, c_count, X, nsm, s);
    case 64: {
      const long long items = (long long)(p.R - 1) * ((c_count + kXCols - 1) / kXCols);
      k_xgram<64><<<(int)std::max<long long>(1, std::min<long long>(items, nsm * 4)), kXThreads, 0, s>>>(
          sa, sb, g, c_base, c_count, p.R, X);
      return (int)cudaGetLastError();
    }
    default: return -1;
  }
}

}  // namespace subby
