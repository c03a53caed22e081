// Inside pass only, A = 4: LogLike and RootProb without an outside pass
// (subby/oracle/oracle.py:784-838, 1571-1595), one thread per column.
//
// k_tree4 keeps every stored node's vector for the outside pass (tensor
// memory, one CTA of 8 warps per SM) and runs its inside half at that
// occupancy.  Without an outside pass a vector is dead as soon as its parent
// has read it: the program is a postorder that enters the deeper child first,
// the child just finished stays in registers, and the others wait on a stack
// of at most log2(leaves) shared-memory slots.  So 24 to 32 warps share an
// SM, and tokens are fetched three steps ahead.  The arithmetic is k_tree4's
// in its order, so the results are too.  R = 199, 200003 columns (GB300): 233
// -> 71 us; bound by issue (60 % active) and the load pipe (56 %: a product's
// four matrix rows are 16 cycles of it per warp).
#include <limits.h>

#include <algorithm>

#include "a4.cuh"
#include "common.cuh"

namespace subby {
namespace {

// Program step: x the node p; y, z its children — a leaf's node index,
// kPrev: the vector of the step before, else ~slot; w: the slot that takes
// p's own vector, -1 when the next step reads it from registers (or p is the
// root: the last step).
constexpr int kPrev = INT_MIN;

// N columns per thread (c0 + lane, c0 + lane + 32): the program, the slots'
// addresses and a product's matrix rows are read once for all of them.
template <int N>
__global__ void __launch_bounds__(256, N == 1 ? 4 : 3) k_inside4(const KParams P) {
  extern __shared__ __align__(16) float sm[];
  const int nb = blockDim.x, t = threadIdx.x, R = P.R, C = P.C, nst = P.nsteps;
  float *MT = sm;                                             // R x 5 x 4
  int4 *prog = reinterpret_cast<int4 *>(MT + R * 20);
  float *LV = reinterpret_cast<float *>(prog + max(nst, 1));  // 5 x 4
  float4 *vec = reinterpret_cast<float4 *>(LV + 20);          // [slot][column][thread]
  int *word = reinterpret_cast<int *>(vec + (size_t)P.nslots * N * nb);
  for (int i = t; i < R * 5; i += nb)
    reinterpret_cast<float4 *>(MT)[i] = __ldg(reinterpret_cast<const float4 *>(P.tab + P.off.MT) + i);
  for (int i = t; i < nst; i += nb) prog[i] = P.prog[i];
  if (t < 20) LV[t] = (t / 4 == 4 || t / 4 == t % 4) ? 1.f : 0.f;
  __syncthreads();
  const int lane = t & 31;
  for (int c0 = (blockIdx.x * nb + t - lane) * N; c0 < C; c0 += gridDim.x * nb * N) {
    int col[N];
#pragma unroll
    for (int q = 0; q < N; ++q) col[q] = min(c0 + lane + 32 * q, C - 1);
    // tokens of a step: p, and its leaf children
    struct Tk {
      int p[N], l[N], r[N];
    };
    auto tok = [&](int (&o)[N], int n) {
      const int32_t *row = P.aln + (size_t)n * C;
#pragma unroll
      for (int q = 0; q < N; ++q) o[q] = __ldg(row + col[q]);
    };
    auto fetch = [&](Tk &o, int i) {
      const int4 s = prog[min(i, nst - 1)];
      tok(o.p, s.x);
      if (s.y >= 0) tok(o.l, s.y);
      if (s.z >= 0) tok(o.r, s.z);
    };
    F4 prev[N];
    int pe[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      prev[q] = F4{make_float2(1.f, 1.f), make_float2(1.f, 1.f)};   // the root's own vector after the last step
      pe[q] = 0;
    }
    auto step = [&](int i, const Tk &k) {
      const int4 s = prog[i];
      F4 u[N];
      int e[N];
      // the children, one after the other into u
      auto child = [&](int c, const int (&tk)[N], bool first) {
        auto join = [&](int q, const F4 &x, int ex) {
          u[q] = first ? x : mul4(u[q], x);
          e[q] = first ? ex : e[q] + ex;
        };
        if (c >= 0) {
#pragma unroll
          for (int q = 0; q < N; ++q) join(q, ld4s(MT + (c * 5 + tcode4(tk[q])) * 4), 0);
        } else if (c == kPrev) {
#pragma unroll
          for (int q = 0; q < N; ++q) join(q, prev[q], pe[q]);
        } else {
#pragma unroll
          for (int q = 0; q < N; ++q) {
            const int at = (~c * N + q) * nb + t;
            join(q, ld4s(reinterpret_cast<const float *>(vec + at)), word[at]);
          }
        }
      };
      child(s.y, k.l, true);
      child(s.z, k.r, false);
      bool any = false;   // an observed internal node (its row of ones otherwise)
#pragma unroll
      for (int q = 0; q < N; ++q) any |= (unsigned)k.p[q] < 4u;
      if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int q = 0; q < N; ++q) u[q] = mul4(u[q], ld4s(LV + tcode4(k.p[q]) * 4));
      }
#pragma unroll
      for (int q = 0; q < N; ++q) pe[q] = e[q] + rescale4(u[q]);
      if (i == nst - 1) {
#pragma unroll
        for (int q = 0; q < N; ++q) prev[q] = u[q];
        return;
      }
      const float *M = MT + s.x * 20;
      const F4 m0 = ld4s(M), m1 = ld4s(M + 4), m2 = ld4s(M + 8), m3 = ld4s(M + 12);
#pragma unroll
      for (int q = 0; q < N; ++q) {   // (matvec4's order)
        F4 y = scale4(m0, u[q].a.x);
        y = fma4(u[q].a.y, m1, y);
        y = fma4(u[q].b.x, m2, y);
        prev[q] = fma4(u[q].b.y, m3, y);
      }
      if (s.w >= 0) {
#pragma unroll
        for (int q = 0; q < N; ++q) {
          const int at = (s.w * N + q) * nb + t;
          vec[at] = make_float4(prev[q].a.x, prev[q].a.y, prev[q].b.x, prev[q].b.y);
          word[at] = pe[q];
        }
      }
    };
    if (nst == 0) {
      int k[N];
      tok(k, 0);
#pragma unroll
      for (int q = 0; q < N; ++q) prev[q] = ld4s(LV + tcode4(k[q]) * 4);
    } else {
      // tokens three steps ahead, in three register sets
      Tk k0, k1, k2;
      fetch(k0, 0);
      fetch(k1, 1);
      fetch(k2, 2);
      int i = 0;
      for (; i + 3 <= nst; i += 3) {
        step(i, k0);
        fetch(k0, i + 3);
        step(i + 1, k1);
        fetch(k1, i + 4);
        step(i + 2, k2);
        fetch(k2, i + 5);
      }
      if (i < nst) step(i, k0);
      if (i + 1 < nst) step(i + 1, k1);
    }
    const F4 pr0 = ld4s(P.tab + P.off.pi0);
#pragma unroll
    for (int q = 0; q < N; ++q) {
      if (c0 + lane + 32 * q >= C) continue;
      const float Pp = dot4(pr0, prev[q]);
      if (P.mode & kModeLogLike) P.logL[col[q]] = (float)((double)pe[q] * kLn2q + (double)logf(Pp));
      if (P.mode & kModeRootProb) {
        const F4 r = scale4(mul4(pr0, prev[q]), 1.0f / Pp);
        P.rootp[col[q]] = r.a.x;
        P.rootp[(size_t)C + col[q]] = r.a.y;
        P.rootp[(size_t)2 * C + col[q]] = r.b.x;
        P.rootp[(size_t)3 * C + col[q]] = r.b.y;
      }
    }
  }
}

}  // namespace

size_t inside4_smem(int R, int nsteps, int nslots, int block, int per) {
  return (size_t)R * 80 + (size_t)std::max(nsteps, 1) * 16 + 80 + (size_t)nslots * block * per * 20;
}

int launch_inside4(const KParams &p, int per, int grid, int block, size_t smem, cudaStream_t s) {
  auto fn = per == 2 ? k_inside4<2> : k_inside4<1>;
  cudaError_t e = per == 2 ? allow_smem<k_inside4<2>>() : allow_smem<k_inside4<1>>();
  if (e != cudaSuccess) return (int)e;
  fn<<<grid, block, smem, s>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace subby
