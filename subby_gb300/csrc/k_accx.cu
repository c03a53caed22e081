// Counts of irreversible models at A = 16, 20, 32 (one system for all
// branches) from the walk's raw staging (subby/oracle/oracle.py:537-693).
//
// The eigensystem of a real rate matrix comes in conjugate pairs, so
// D~_k = sum_a D_a Vinv[k][a] and U~_l = sum_b U_b V[b][l] hold A real numbers
// each, and C_k'l' = conj(C_kl) for conjugate k', l'.  A UNIT is a conjugate
// pair or a real eigenvalue; a vector is (Re, Im) of each unit's
// representative.  With d of unit k and u, conj(u) of unit l,
//   C_kl += J_kl d u,   C_kl' += J_kl' d conj(u)
// for the representatives k only (a real l has no partner: J_kl' = 0), and
//   counts_ij = sum_k w_k Re(V_ik (C Vinv)_kj), w = 2 for a pair, 1 for a real
// (off the diagonal times Q_ij).  That is half the complex products of the
// full C.  Plans whose eigensystem does not pair up, or is ill-conditioned (kCxCond),
// keep k_acc_cx.
//
// k_acc_cx forms a column's D~, U~ one dot product per thread from strided
// rows and shares no load between columns.  Here k_projx projects with the
// matrices in the constant bank (as k_proj), and a thread of k_accx owns 2 x
// 2 units for 8 columns, in column pairs for the packed multiply-adds: 16
// loaded floats feed 112 of them, and J is loaded once for the 8 columns.
// Bound by the load pipe (64 % active: the units' rows of a vector block
// still meet on banks two at a time).  A = 20, R = 99, C = 8001 (GB300):
// k_acc_cx 2336 us; k_projx 59 + k_accx 165 us.  The sums run in registers
// over 32 branches at a time and the groups' sums in shared memory (13 us of
// the 165), which halves the error of one long FP32 sum: counts 2.2e-6 from
// FP64 against 3.2e-6.
#include <algorithm>

#include "common.cuh"
#include "walk.cuh"

namespace subby {
namespace {

constexpr int kPxRows = 128;

template <int A>
struct ProjX {
  float d[A * A], u[A * A];   // real-form projections, [state][output]
  uint8_t slot[A];            // output -> (Re or Im of a unit): row of the projected block
};

// Projections of the raw rows (chunks rotated by stage_rot) into blocks
// [branch - 1][column block][2 UP][accx_stride(G)]: one thread per row, the matrices in
// the constant bank (as k_proj); the stores of a warp are contiguous.
template <int A>
__global__ void __launch_bounds__(kPxRows)
    k_projx(const __grid_constant__ ProjX<A> W, const KParams P, const CxUnits cu, const float *__restrict__ stage_a,
            const float *__restrict__ stage_b, float *__restrict__ pa, float *__restrict__ pb, int c_base,
            int c_count) {
  extern __shared__ __align__(128) float sm[];   // the tile's rows, then the leaves' U~ by token
  __shared__ __align__(8) uint64_t mbar;
  __shared__ int s_err;
  float *Lt = sm + kPxRows * A;
  const int t = threadIdx.x;
  const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar);
  const uint32_t srow = (uint32_t)__cvta_generic_to_shared(sm);
  // tiles of one branch each, so that a tile's columns are consecutive
  const int ctiles = (c_count + kPxRows - 1) / kPxRows;
  const int nblk = (c_count + cu.G - 1) / cu.G;
  const int half = (P.R - 1) * ctiles;
  for (int i = t; i < (A + 1) * A; i += kPxRows) Lt[i] = __ldg(cu.leafU + i);
  if (t == 0) {
    s_err = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  __syncthreads();
  uint32_t phase = 0;
  for (int it = blockIdx.x; it < 2 * half; it += gridDim.x) {
    const bool up = it >= half;
    const int i2 = up ? it - half : it, n = 1 + i2 / ctiles, c0 = (i2 % ctiles) * kPxRows;
    const int rows = min(kPxRows, c_count - c0), c = c0 + t;
    const bool leaf = up && __ldg(P.leaf + n) != 0;
    __syncthreads();   // the previous tile's rows are read
    if (!leaf) {
      if (t == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(rows * A * 4) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(srow),
                     "l"((up ? stage_b : stage_a) + ((size_t)(n - 1) * c_count + c0) * A), "r"(rows * A * 4), "r"(mb)
                     : "memory");
      }
      __syncwarp();
      if (!mbar_wait(mb, phase & 1)) s_err = 1;
      ++phase;
    }
    if (t >= rows) continue;
    float y[A];
    if (leaf) {
      const int code = btcode(__ldg(P.aln + (size_t)n * P.C + c_base + c), A);
#pragma unroll
      for (int o = 0; o < A; ++o) y[o] = Lt[code * A + o];
    } else {
      const float *row = sm + t * A;
      const int rot = stage_rot(A, c);
      float x[A];
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
    }
    const int GP = accx_stride(cu.G);
    float *out = (up ? pb : pa) + ((size_t)(n - 1) * nblk + c / cu.G) * 2 * cu.UP * GP + c % cu.G;
#pragma unroll
    for (int o = 0; o < A; ++o) out[(int)W.slot[o] * GP] = y[o];
    for (int u = cu.pairs; u < cu.UP; ++u) {   // imaginary parts of reals; padding units
      out[(2 * u + 1) * GP] = 0.f;
      if (u >= cu.U) out[2 * u * GP] = 0.f;
    }
  }
  __syncthreads();
  if (t == 0 && s_err && P.err) atomicAdd(P.err, 1);
}

constexpr int kAxStages = 3;
constexpr int kAxRun = 32;       // branches summed in registers
constexpr int kAxRow = 258;      // threads' stride (float2) of the C sums: a column's pairs on different banks

// Thread: 2 x 2 units of (k, l) for 8 columns; KT^2 threads per 8 columns.
template <int A>
__global__ void __launch_bounds__(256, 1)
    k_accx(const KParams P, const CxUnits cu, const float *__restrict__ pa, const float *__restrict__ pb, int c_base,
           int c_count) {
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(8) uint64_t mbar[kAxStages];
  __shared__ int s_err;
  const int t = threadIdx.x;
  const int G = cu.G, UP = cu.UP, KT = UP / 2, NB = KT * KT;
  const int grp = t / NB, blk = t % NB;
  const bool active = grp < G / 8;
  const int k0 = 2 * (blk / KT), l0 = 2 * (blk % KT);   // first units
  const int GP = accx_stride(G);
  const int vec = 2 * UP * GP, jn = 4 * UP * UP;         // floats of a vector block, of a branch's J
  const int stage = jn + 2 * vec;
  const int nblk = (c_count + G - 1) / G, nbr = P.R - 1, C = P.C;
  // C, thread by thread ([(a, l, component, column pair)][thread] float2),
  // then the ring, later T
  float2 *Cs = reinterpret_cast<float2 *>(sm);
  float *ring = sm + 64 * 2 * kAxRow, *Ts = ring;
  const size_t mainf = 64 * 2 * kAxRow + max((size_t)kAxStages * stage, (size_t)2 * UP * A * 16);
  float2 *Vs = reinterpret_cast<float2 *>(sm + mainf);   // [i][unit]: w V
  float2 *Vis = Vs + A * UP;                             // [unit][2][j]: Vinv of the representative, of its partner
  float *Rs = reinterpret_cast<float *>(Vis + 2 * UP * A);
  for (int i = t; i < A * UP; i += 256) Vs[i] = cu.V[i];
  for (int i = t; i < 2 * UP * A; i += 256) Vis[i] = cu.Vi[i];
  for (int i = t; i < A * A; i += 256) Rs[i] = cu.rate[i];
  if (t == 0) {
    s_err = 0;
    for (int i = 0; i < kAxStages; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&mbar[i]))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  __syncthreads();
  uint32_t it0 = 0;   // ring position of the block's first branch
  for (int b = blockIdx.x; b < nblk; b += gridDim.x, it0 += nbr) {
    auto load = [&](int i) {   // branch i (node i + 1)
      float *d = ring + (size_t)((it0 + i) % kAxStages) * stage;
      const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar[(it0 + i) % kAxStages]);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(stage * 4) : "memory");
      auto copy = [&](float *dst, const float *src, int n) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n * 4), "r"(mb) : "memory");
      };
      const size_t off = ((size_t)i * nblk + b) * vec;
      copy(d, cu.J + (size_t)(i + 1) * jn, jn);
      copy(d + jn, pa + off, vec);
      copy(d + jn + vec, pb + off, vec);
    };
    float2 c1r[2][2][4], c1i[2][2][4], c2r[2][2][4], c2i[2][2][4];   // [k][l][column pair]
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int l = 0; l < 2; ++l)
#pragma unroll
        for (int p = 0; p < 4; ++p)
          c1r[a][l][p] = c1i[a][l][p] = c2r[a][l][p] = c2i[a][l][p] = make_float2(0.f, 0.f);
    // this thread's entries: the registers' sums over kAxRun branches are
    // added to C, so that no FP32 sum runs over more terms than that many
    // branches plus their groups
    auto flush = [&](bool first) {
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            float2 *o = Cs + (size_t)(16 * (2 * a + l) + p) * kAxRow + t;
            auto put = [&](float2 *q, float2 &c) {
              float2 v = c;
              if (!first) {
                const float2 old = *q;
                v.x += old.x, v.y += old.y;
              }
              *q = v;
              c = make_float2(0.f, 0.f);
            };
            put(o, c1r[a][l][p]);
            put(o + 4 * kAxRow, c1i[a][l][p]);
            put(o + 8 * kAxRow, c2r[a][l][p]);
            put(o + 12 * kAxRow, c2i[a][l][p]);
          }
    };
    // the previous block's epilogue is past C and the ring; its generic
    // writes come before the bulk copies
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t == 0)
      for (int i = 0; i < kAxStages - 1 && i < nbr; ++i) load(i);
    __syncwarp();
    for (int i = 0; i < nbr; ++i) {
      __syncthreads();   // every thread is done with the stage that this refills
      if (t == 0 && i + kAxStages - 1 < nbr) load(i + kAxStages - 1);
      __syncwarp();
      const uint32_t pos = it0 + i;
      if (!mbar_wait((uint32_t)__cvta_generic_to_shared(&mbar[pos % kAxStages]), (pos / kAxStages) & 1)) s_err = 1;
      if (!active) continue;
      const float *S = ring + (size_t)(pos % kAxStages) * stage;
      // (J_kl, J_kl'), both columns of a pair
      float2 ar[2][2], ai[2][2], br[2][2], bi[2][2];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          const float4 j = *reinterpret_cast<const float4 *>(S + 4 * ((k0 + a) * UP + l0 + l));
          ar[a][l] = make_float2(j.x, j.x), ai[a][l] = make_float2(j.y, j.y);
          br[a][l] = make_float2(j.z, j.z), bi[a][l] = make_float2(j.w, j.w);
        }
      const float *da = S + jn + 2 * k0 * GP + 8 * grp, *ub = S + jn + vec + 2 * l0 * GP + 8 * grp;
      auto neg = [](float2 x) { return make_float2(-x.x, -x.y); };
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float2 d[4], u[4];   // (Re, Im) of two units
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          d[q] = *reinterpret_cast<const float2 *>(da + q * GP + 2 * p);
          u[q] = *reinterpret_cast<const float2 *>(ub + q * GP + 2 * p);
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int l = 0; l < 2; ++l) {
            const float2 dr = d[2 * a], di = d[2 * a + 1], ur = u[2 * l], ui = u[2 * l + 1];
            const float2 m1 = __fmul2_rn(dr, ur), m2 = __fmul2_rn(dr, ui);
            const float2 z1r = __ffma2_rn(neg(di), ui, m1), z2r = __ffma2_rn(di, ui, m1);
            const float2 z1i = __ffma2_rn(di, ur, m2), z2i = __ffma2_rn(di, ur, neg(m2));
            c1r[a][l][p] = __ffma2_rn(neg(ai[a][l]), z1i, __ffma2_rn(ar[a][l], z1r, c1r[a][l][p]));
            c1i[a][l][p] = __ffma2_rn(ai[a][l], z1r, __ffma2_rn(ar[a][l], z1i, c1i[a][l][p]));
            c2r[a][l][p] = __ffma2_rn(neg(bi[a][l]), z2i, __ffma2_rn(br[a][l], z2r, c2r[a][l][p]));
            c2i[a][l][p] = __ffma2_rn(bi[a][l], z2r, __ffma2_rn(br[a][l], z2i, c2i[a][l][p]));
          }
      }
      if (i % kAxRun == kAxRun - 1 || i == nbr - 1) flush(i < kAxRun);
    }
    __syncthreads();
    // ------------------------------------------------------------- epilogue
    // 16 columns at a time: T = C Vinv ([k][j], complex), then the output
    const int gcols = min(G, c_count - b * G);
    for (int s0 = 0; s0 < gcols; s0 += 16) {
      __syncthreads();   // C complete; the previous batch's T is read
      const int x = t & 15;   // column of the batch
      const int cg = (s0 + x) >> 3, cp = ((s0 + x) & 7) >> 1;   // its group, its pair
      if (s0 + x < G)
        for (int e = t >> 4; e < cu.U * A; e += 16) {
          const int k = e / A, j = e % A;
          float sr = 0.f, si = 0.f;
          for (int l = 0; l < cu.U; ++l) {
            const float *c = reinterpret_cast<const float *>(
                                 Cs + (size_t)(16 * (2 * (k & 1) + (l & 1)) + cp) * kAxRow + cg * NB +
                                 (k >> 1) * KT + (l >> 1)) + (x & 1);
            const float2 v = Vis[2 * l * A + j], v2 = Vis[(2 * l + 1) * A + j];
            const float r1 = c[0], i1 = c[8 * kAxRow], r2 = c[16 * kAxRow], i2 = c[24 * kAxRow];
            sr = fmaf(r1, v.x, fmaf(-i1, v.y, sr)), si = fmaf(r1, v.y, fmaf(i1, v.x, si));
            sr = fmaf(r2, v2.x, fmaf(-i2, v2.y, sr)), si = fmaf(r2, v2.y, fmaf(i2, v2.x, si));
          }
          Ts[(2 * e) * 16 + x] = sr;
          Ts[(2 * e + 1) * 16 + x] = si;
        }
      __syncthreads();
      if (s0 + x < gcols)
        for (int e = t >> 4; e < A * A; e += 16) {
          const int i = e / A, j = e % A;
          float s = 0.f;
          for (int k = 0; k < cu.U; ++k) {
            const float2 v = Vs[i * UP + k];
            s = fmaf(v.x, Ts[(2 * (k * A + j)) * 16 + x], fmaf(-v.y, Ts[(2 * (k * A + j) + 1) * 16 + x], s));
          }
          P.counts[(size_t)e * C + c_base + b * G + s0 + x] = (i == j) ? s : Rs[e] * s;
        }
    }
  }
  __syncthreads();
  if (t == 0 && s_err && P.err) atomicAdd(P.err, 1);
}

size_t accx_floats(int A, int UP, int G) {
  const size_t stage = (size_t)4 * UP * UP + 4 * (size_t)UP * accx_stride(G);
  const size_t mainf = 64 * 2 * kAxRow + std::max(kAxStages * stage, (size_t)2 * UP * A * 16);
  return mainf + 2 * ((size_t)A * UP + 2 * (size_t)UP * A) + (size_t)A * A;
}

template <int A>
int accx(const KParams &p, const CxUnits &cu, const CxHost &h, const float *sa, const float *sb, float *pa, float *pb,
         int c_base, int c_count, int nsm, cudaStream_t s) {
  ProjX<A> W;
  for (int i = 0; i < A * A; ++i) W.d[i] = h.d[i], W.u[i] = h.u[i];
  for (int i = 0; i < A; ++i) W.slot[i] = h.slot[i];
  const long long tiles = 2LL * (p.R - 1) * ((c_count + kPxRows - 1) / kPxRows);
  const size_t ps = (size_t)(kPxRows + A + 1) * A * sizeof(float);
  k_projx<A><<<(int)std::max<long long>(1, std::min<long long>(tiles, (long long)nsm * (A == 32 ? 6 : 8))), kPxRows, ps,
               s>>>(W, p, cu, sa, sb, pa, pb, c_base, c_count);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  const size_t smem = accx_floats(A, cu.UP, cu.G) * sizeof(float);
  e = allow_smem<k_accx<A>>();
  if (e != cudaSuccess) return (int)e;
  const int nblk = (c_count + cu.G - 1) / cu.G;
  k_accx<A><<<std::max(1, std::min(nblk, nsm)), 256, smem, s>>>(p, cu, pa, pb, c_base, c_count);
  return (int)cudaGetLastError();
}

}  // namespace

bool accx_supported(int A) { return A == 16 || A == 20 || A == 32; }

// Columns per CTA: eight per group of (UP / 2)^2 threads, as many groups as
// fit in 256 threads and shared memory.
int accx_group(int A, int UP) {
  const int nb = (UP / 2) * (UP / 2);
  if (nb < 1 || nb > 256) return 0;
  int groups = 256 / nb;
  while (groups > 0 && accx_floats(A, UP, 8 * groups) * sizeof(float) > 220 * 1024) --groups;
  return 8 * groups;
}

// Few columns: blocks small enough for every SM to have one, as a block's
// back-transform takes as long as its columns (R = 3, A = 20, 500 columns:
// blocks of 56 103 us a call, of 16 60 us).  A block's columns do not depend on one
// another, so the results are the same.
int accx_columns(int G, int C, int nsm) {
  return std::min(G, std::max(16, ((C + nsm - 1) / nsm + 7) / 8 * 8));
}

int launch_accx(const KParams &p, int A, const CxUnits &cu, const CxHost &h, const float *sa, const float *sb,
                float *pa, float *pb, int c_base, int c_count, int nsm, cudaStream_t s) {
  switch (A) {
    case 16: return accx<16>(p, cu, h, sa, sb, pa, pb, c_base, c_count, nsm, s);
    case 20: return accx<20>(p, cu, h, sa, sb, pa, pb, c_base, c_count, nsm, s);
    case 32: return accx<32>(p, cu, h, sa, sb, pa, pb, c_base, c_count, nsm, s);
    default: return -1;
  }
}

}  // namespace subby
