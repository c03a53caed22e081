// Tree walk with four lanes per column (A = 16, 20, 32; any of them and
// A = 64 for F81 / JC models): inside pass, LogLike / RootProb, outside pass
// staging every branch's vectors in the original basis
//   stage_a[n-1][c][a] = s D_n(c, a),  stage_b[n-1][c][b] = U_n(c, b)
// (s = 2^(eD + eU - eRoot) / P, zero for masked branches;
// subby/oracle/oracle.py:784-924).  Same results as k_walk's raw staging.
//
// Lane (sg, cg) = (lane / 8, lane % 8) of a warp holds the states
// {16 k + 4 sg .. + 3} (A = 20: and 16 + sg) of the CPL columns
// CPL cg .. CPL cg + CPL - 1, so a warp walks 8 CPL columns on its own.
//
// What bounds it, and the layout that follows: one thread per column
// (k_walk) reads every matrix element as a broadcast 16-byte load for four
// multiply-adds, four cycles of the SM's load pipe each, and it waits for L2
// whenever a step's matrix is new (each matrix is used once per tile).  Here
// a load of SPL matrix elements and CPL column values feeds SPL * CPL
// multiply-adds (A = 20, CPL = 2: 7 cycles of the load pipe per 16 columns
// instead of 10), the matrices of the coming steps arrive in shared memory
// by bulk copies (a ring of kQS steps), tokens and slots are fetched a step
// ahead, and the vector that the next step needs (the child just finished,
// or the child about to be entered) stays in registers.  The projections
// into the eigenbasis, two thirds of the products of a Counts walk, do not
// depend on the tree order and are left to k_proj.
// Measured (GB300; walk with the raw staging, against k_walk's eigen
// staging): A = 20, R = 199, C = 20011 1515 -> 414 us; A = 20, R = 399,
// C = 50000 5490 -> 1683 us; A = 16, R = 99, C = 4003 368 -> 72 us; A = 32,
// R = 127, C = 16000 1724 -> 430 us; F81 at A = 64, R = 127, C = 20011 1617
// -> 484 us.  The product's loop is unrolled whole: by fours it measured 432,
// 1740 and 82 us (no spills either way).  What is left is latency at 8 to 12 warps per SM (issue 40 %
// active, load pipe 48 %).  Four columns per lane (255 registers, 8 warps
// per SM) measured 2074 us at R = 399, C = 50000, 128 registers with two
// columns per lane 2229 us (spills).

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "walk.cuh"

namespace subby {
namespace {

constexpr int kQW = 4;   // column warps per CTA
constexpr int kQS = 4;   // ring stages

template <int A, int CPL>
struct QG {
  static constexpr int SPL = A / 4;                               // states per lane
  static constexpr int N = SPL * CPL;                             // floats per lane and vector
  static constexpr int W = 8 * CPL;                               // columns per warp
  static constexpr int TILE = W * kQW;                            // columns per CTA
  static constexpr int XS = CPL == 2 ? 20 : 10;                   // x rows: conflict-free strides
  static constexpr int BLK = (A + 1) * A;                         // floats of a ring block
  static constexpr int SLOT4 = (N + 3) / 4 * 32;                  // float4s of a warp's slot vector
  static constexpr size_t smem(bool f81m) {
    return f81m ? 0 : (size_t)(kQS * 3 * BLK + kQW * 2 * A * XS) * sizeof(float);
  }
};

// This lane's states of its CPL columns, in pairs for the packed FP32x2
// instructions (A = 20: two pairs and a single).
template <int A, int CPL>
struct QV {
  static constexpr int SPL = A / 4, NP = SPL / 2;
  static constexpr bool ODD = SPL % 2 != 0;
  float2 p[CPL][NP];
  float s[CPL];   // ODD only
  __device__ __forceinline__ float &at(int q, int i) {
    return (ODD && i == SPL - 1) ? s[q] : (i & 1) ? p[q][i >> 1].y : p[q][i >> 1].x;
  }
  __device__ __forceinline__ float get(int q, int i) const {
    return (ODD && i == SPL - 1) ? s[q] : (i & 1) ? p[q][i >> 1].y : p[q][i >> 1].x;
  }
  __device__ __forceinline__ void fill(int q, float x) {
#pragma unroll
    for (int i = 0; i < NP; ++i) p[q][i] = make_float2(x, x);
    if constexpr (ODD) s[q] = x;
  }
  __device__ __forceinline__ void scale(int q, float x) {
    const float2 xx = make_float2(x, x);
#pragma unroll
    for (int i = 0; i < NP; ++i) p[q][i] = __fmul2_rn(p[q][i], xx);
    if constexpr (ODD) s[q] *= x;
  }
  __device__ __forceinline__ void mul(const QV &a, const QV &b) {
#pragma unroll
    for (int q = 0; q < CPL; ++q) {
#pragma unroll
      for (int i = 0; i < NP; ++i) p[q][i] = __fmul2_rn(a.p[q][i], b.p[q][i]);
      if constexpr (ODD) s[q] = a.s[q] * b.s[q];
    }
  }
  // this lane's states of a row of A floats (16-byte aligned)
  __device__ __forceinline__ void row(int q, const float *r, int sg) {
#pragma unroll
    for (int k = 0; k < A / 16; ++k) {
      const float4 t = *reinterpret_cast<const float4 *>(r + 16 * k + 4 * sg);
      p[q][2 * k] = make_float2(t.x, t.y), p[q][2 * k + 1] = make_float2(t.z, t.w);
    }
    if constexpr (ODD) s[q] = r[16 + sg];
  }
  // x times column q into a row (its 16-byte chunks rotated by rot)
  __device__ __forceinline__ void put(int q, float x, float *r, int sg, int rot) const {
    const float2 xx = make_float2(x, x);
#pragma unroll
    for (int k = 0; k < A / 16; ++k) {
      const float2 u = __fmul2_rn(p[q][2 * k], xx), v = __fmul2_rn(p[q][2 * k + 1], xx);
      *reinterpret_cast<float4 *>(r + stage_chunk<A>(4 * k + sg, rot)) = make_float4(u.x, u.y, v.x, v.y);
    }
    if constexpr (ODD) r[16 + sg] = s[q] * x;
  }
};

template <int A>
__device__ __forceinline__ int qstate(int i, int sg) {
  return (A == 20 && i == 4) ? 16 + sg : (i / 4) * 16 + 4 * sg + (i & 3);
}
// sum / max over the four lanes of a column
__device__ __forceinline__ float qsum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 8);
  return x + __shfl_xor_sync(0xffffffffu, x, 16);
}
__device__ __forceinline__ float qmax(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 8));
  return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 16));
}

struct QStep {
  int p, sp, l, kl, r, kr;   // node, its slot (-1: root), children and their slots (-1: leaf)
};

// MODE: 0 inside pass only, 1 with the outside pass and the staging.
template <int CPL, bool F81M>
__host__ __device__ constexpr bool q_producer() { return !F81M && CPL == 1; }
template <int CPL, bool F81M>
__host__ __device__ constexpr int q_threads() { return (kQW + (q_producer<CPL, F81M>() ? 1 : 0)) * 32; }

template <int A, int CPL, bool F81M, int MODE, int MINB>
__global__ void __launch_bounds__((q_threads<CPL, F81M>()), MINB)
    k_qwalk(const KParams P, float *__restrict__ stage_a, float *__restrict__ stage_b, int flags, int c_base,
            int c_count) {
  using G = QG<A, CPL>;
  constexpr int SPL = G::SPL;
  using V = QV<A, CPL>;
  extern __shared__ __align__(128) float sm[];
  __shared__ __align__(8) uint64_t s_full[kQS], s_empty[kQS];
  __shared__ int s_err, s_skip;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sg = lane >> 3, cg = lane & 7;
  const float *MT = P.tab + P.off.MT;
  const float *MN = P.tab + P.off.MN;
  const float *EF = P.tab + P.off.EF;
  const float *pig = P.tab + P.off.pi;
  const float *pr0g = P.tab + P.off.pi0;
  const int nst = P.nsteps, C = P.C;
  const int ntiles = (c_count + G::TILE - 1) / G::TILE;
  auto prog = [&](int i) {
    const int4 s0 = __ldg(P.prog + 4 * i);
    const int2 s1 = __ldg(reinterpret_cast<const int2 *>(P.prog + 4 * i + 1));
    const int2 s2 = __ldg(reinterpret_cast<const int2 *>(P.prog + 4 * i + 2));
    return QStep{s0.x, s0.z ? -1 : s0.y, s1.x, s1.y, s2.x, s2.y};
  };
  if (threadIdx.x == 0) {
    s_err = 0;
    for (int i = 0; i < kQS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&s_full[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&s_empty[i])),
                   "r"(kQW));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // Test hook of the failure path: a wait for the first step's matrices,
    // which nothing has requested yet (no copy is in flight), for a few polls;
    // it gives up and the CTA skips its work.
    s_skip = !F81M && P.dbg_wait_polls > 0 &&
             !mbar_wait((uint32_t)__cvta_generic_to_shared(&s_full[0]), 0, P.dbg_wait_polls);
  }
  __syncwarp();
  __syncthreads();
  if (!F81M && s_skip) {
    if (threadIdx.x == 0 && P.err) atomicAdd(P.err, 1);
    return;
  }

  // Ring of the steps' matrices in the order of their use (every tile: the
  // steps forwards, then backwards).  One thread refills it: with one column
  // per lane a warp of its own, which never makes the column warps wait for
  // an issue slot; otherwise thread 0, one step at a time, into the stage of
  // the step kQS - 2 ahead (its previous use is two steps back, which every
  // warp has mostly left).
  const uint32_t per_tile = (MODE == 0 ? 1 : 2) * (uint32_t)nst;
  const uint32_t nring =
      F81M || (int)blockIdx.x >= ntiles ? 0 : per_tile * (uint32_t)((ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1);
  uint32_t k = 0, kf = 0;   // ring positions: this warp's step, the next refill (thread 0)
  uint32_t kr = 0;          // kf within its tile
  QStep rs = nst > 0 ? prog(0) : QStep{};   // the step of kf (loaded one refill ahead)
  auto refill = [&](uint32_t upto) {
    for (; kf < upto && kf < nring; ++kf) {
      const bool outside = kr >= (uint32_t)nst;
      const QStep s = rs;
      kr = kr + 1 == per_tile ? 0 : kr + 1;
      rs = prog(kr >= (uint32_t)nst ? 2 * nst - 1 - (int)kr : (int)kr);
      const int st = kf % kQS;
      if (kf >= kQS && !mbar_wait((uint32_t)__cvta_generic_to_shared(&s_empty[st]), (kf / kQS - 1) & 1)) s_err = 1;
      const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&s_full[st]);
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(sm) + (uint32_t)st * 3 * G::BLK * 4;
      constexpr uint32_t leafb = G::BLK * 4, ownb = A * A * 4;
      const uint32_t bytes = (s.kl < 0 ? leafb : 0) + (s.kr < 0 ? leafb : 0) + (s.sp >= 0 ? ownb : 0);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
      auto copy = [&](uint32_t dst, const float *src, uint32_t n) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         dst), "l"(src), "r"(n), "r"(mb) : "memory");
      };
      if (s.kl < 0) copy(d, MT + (size_t)s.l * G::BLK, leafb);
      if (s.kr < 0) copy(d + leafb, MT + (size_t)s.r * G::BLK, leafb);
      if (s.sp >= 0) copy(d + 2 * leafb, outside ? MN + (size_t)s.p * A * A : MT + (size_t)s.p * G::BLK, ownb);
    }
  };
  constexpr bool PW = q_producer<CPL, F81M>();
  if (PW && warp == kQW) {
    if (lane == 0) refill(nring);
    __syncwarp();
  } else {
    if (!F81M && !PW && threadIdx.x == 0) refill(kQS - 2);
    __syncwarp();
    float *xs = sm + kQS * 3 * G::BLK + warp * 2 * A * G::XS;
    int xbuf = 0;
    const size_t wslot = (size_t)blockIdx.x * kQW + warp;
    float4 *svec = reinterpret_cast<float4 *>(P.scrV) + wslot * (size_t)P.nslots * G::SLOT4 + lane;
    int *sword = P.scrW + (wslot * (size_t)P.nslots * 4 + sg) * G::W + CPL * cg;
    auto slot_ld = [&](V &x, int (&w)[CPL], int s) {
      const float4 *q = svec + (size_t)s * G::SLOT4;
      float t[(G::N + 3) / 4 * 4];
#pragma unroll
      for (int i = 0; i < (G::N + 3) / 4; ++i) *reinterpret_cast<float4 *>(t + 4 * i) = q[32 * i];
#pragma unroll
      for (int i = 0; i < G::N; ++i) x.at(i / SPL, i % SPL) = t[i];
      const int *u = sword + (size_t)s * 4 * G::W;
#pragma unroll
      for (int i = 0; i < CPL; ++i) w[i] = u[i];
    };
    auto slot_st = [&](const V &x, const int (&w)[CPL], int s) {
      float4 *q = svec + (size_t)s * G::SLOT4;
      float t[(G::N + 3) / 4 * 4];
#pragma unroll
      for (int i = 0; i < (G::N + 3) / 4 * 4; ++i) t[i] = i < G::N ? x.get((i < G::N ? i : 0) / SPL, i % SPL) : 0.f;
#pragma unroll
      for (int i = 0; i < (G::N + 3) / 4; ++i) q[32 * i] = *reinterpret_cast<float4 *>(t + 4 * i);
      int *u = sword + (size_t)s * 4 * G::W;
#pragma unroll
      for (int i = 0; i < CPL; ++i) u[i] = w[i];
    };
    auto ring_wait = [&]() {
      if constexpr (!F81M) {
        if (!PW && threadIdx.x == 0) refill(k + kQS - 1);
        __syncwarp();
        if (!mbar_wait((uint32_t)__cvta_generic_to_shared(&s_full[k % kQS]), (k / kQS) & 1)) s_err = 1;
      }
    };
    auto ring_free = [&]() {
      if constexpr (!F81M) {
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                           (uint32_t)__cvta_generic_to_shared(&s_empty[k % kQS])) : "memory");
        ++k;
      }
    };
    V piv;   // F81: pi
    if constexpr (F81M) {
#pragma unroll
      for (int q = 0; q < CPL; ++q) piv.row(q, pig, sg);
    }
    // y_b = sum_j T[j][b] x_j, T the ring's third block (rows of A floats)
    auto matvec = [&](V &y, const V &x) {
      const float *T = sm + (k % kQS) * 3 * G::BLK + 2 * G::BLK;
      float *xb = xs + xbuf * A * G::XS;
      xbuf ^= 1;
#pragma unroll
      for (int i = 0; i < SPL; ++i) {
        float *d = xb + qstate<A>(i, sg) * G::XS + CPL * cg;
        if constexpr (CPL == 2) *reinterpret_cast<float2 *>(d) = make_float2(x.get(0, i), x.get(1, i));
        else *d = x.get(0, i);
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < CPL; ++q) y.fill(q, 0.f);
#pragma unroll
      for (int j = 0; j < A; ++j) {
        V m;   // column 0 only
        m.row(0, T + j * A, sg);
        float xj[CPL];
        const float *xp = xb + j * G::XS + CPL * cg;
        if constexpr (CPL == 2) {
          const float2 t = *reinterpret_cast<const float2 *>(xp);
          xj[0] = t.x, xj[1] = t.y;
        } else {
          xj[0] = *xp;
        }
#pragma unroll
        for (int q = 0; q < CPL; ++q)
#pragma unroll
          for (int i = 0; i < SPL; ++i) y.at(q, i) = fmaf(m.get(0, i), xj[q], y.at(q, i));
      }
    };
    // F81 closed form: y = e x + (1 - e) (pi . x) 1, or its transpose
    auto f81prod = [&](V &y, const V &x, int n, bool trans) {
      const float2 ef = __ldg(reinterpret_cast<const float2 *>(EF) + n);
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        float sd = 0.f;
#pragma unroll
        for (int i = 0; i < SPL; ++i) sd = trans ? sd + x.get(q, i) : fmaf(piv.get(q, i), x.get(q, i), sd);
        const float w = ef.y * qsum(sd);
#pragma unroll
        for (int i = 0; i < SPL; ++i) y.at(q, i) = fmaf(ef.x, x.get(q, i), trans ? w * piv.get(q, i) : w);
      }
    };
    auto mprod = [&](V &y, const V &x, int n, bool trans) {
      if constexpr (F81M) f81prod(y, x, n, trans);
      else matvec(y, x);
    };
    // M_n L(code): the leaf's contribution to its parent, from the ring's
    // block (side) or in closed form
    auto leaf = [&](V &x, int (&w)[CPL], const int (&tk)[CPL], int n, int side) {
      float2 ef = make_float2(0.f, 0.f);
      if constexpr (F81M) ef = __ldg(reinterpret_cast<const float2 *>(EF) + n);
      const float *T = sm + (k % kQS) * 3 * G::BLK + side * G::BLK;
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        const int code = btcode(tk[q], A);
        if constexpr (F81M) {
          const float pc = code < A ? ef.y * __ldg(pig + min(code, A - 1)) : 1.f;
#pragma unroll
          for (int i = 0; i < SPL; ++i) x.at(q, i) = qstate<A>(i, sg) == code ? ef.x + pc : pc;
        } else {
          x.row(q, T + code * A, sg);
        }
        const int u = btung(tk[q], A);
        w[q] = (u << 1) | u;
      }
    };
    // an observed internal node keeps its state only (rare: one vote skips it)
    auto obs = [&](V &x, const int (&tk)[CPL]) {
      bool any = false;
#pragma unroll
      for (int q = 0; q < CPL; ++q) any |= (unsigned)tk[q] < (unsigned)A;
      if (!__any_sync(0xffffffffu, any)) return;
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        const int code = btcode(tk[q], A);
#pragma unroll
        for (int i = 0; i < SPL; ++i) x.at(q, i) = (code >= A || qstate<A>(i, sg) == code) ? x.get(q, i) : 0.f;
      }
    };
    // multiply each column by 2^-e, e = floor(log2 max) (zero vector: -127)
    auto rescale = [&](V &x, int (&e)[CPL]) {
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        float m = x.get(q, 0);
#pragma unroll
        for (int i = 1; i < SPL; ++i) m = fmaxf(m, x.get(q, i));
        const int E = __float_as_int(qmax(m)) >> 23;
        x.scale(q, __int_as_float((254 - E) << 23));
        e[q] = E - 127;
      }
    };

    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const int cc0 = tile * G::TILE + warp * G::W + CPL * cg;   // first column within the chunk
      int co[CPL];   // columns (clamped: the surplus ones repeat the last)
#pragma unroll
      for (int q = 0; q < CPL; ++q) co[q] = c_base + min(cc0 + q, c_count - 1);
      auto tok = [&](int (&t)[CPL], int n) {
        const int32_t *r = P.aln + (size_t)n * C;
#pragma unroll
        for (int q = 0; q < CPL; ++q) t[q] = __ldg(r + co[q]);
      };
      V nl, nr, keep;   // children; keep: the vector handed to the next step in registers
      int wl[CPL], wr[CPL], wk[CPL], keep_s = -2;
      int tp[CPL], tl[CPL], tr[CPL];
      // tokens and stored children of step s (keep_s: in registers)
      auto fetch = [&](const QStep &s) {
        tok(tp, s.p);
        if (s.kl < 0) tok(tl, s.l);
        else if (s.kl != keep_s) slot_ld(nl, wl, s.kl);
        if (s.kr < 0) tok(tr, s.r);
        else if (s.kr != keep_s) slot_ld(nr, wr, s.kr);
      };
      auto take = [&](V &x, int (&w)[CPL]) {
        x = keep;
#pragma unroll
        for (int q = 0; q < CPL; ++q) w[q] = wk[q];
      };
      // -------------------------------------------------------------- inside
      V ur;
      int eR[CPL], iR[CPL];
      QStep cur{}, nxt{};
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        eR[q] = iR[q] = 0;
        ur.fill(q, 1.f);
      }
      if (nst == 0) {
        tok(tp, 0);
        obs(ur, tp);
      } else {
        cur = prog(0);
        nxt = prog(min(1, nst - 1));
        fetch(cur);
      }
      for (int i = 0; i < nst; ++i) {
        const QStep nn = prog(min(i + 2, nst - 1));
        ring_wait();
        if (cur.kl < 0) leaf(nl, wl, tl, cur.l, 0);
        else if (cur.kl == keep_s) take(nl, wl);
        if (cur.kr < 0) leaf(nr, wr, tr, cur.r, 1);
        else if (cur.kr == keep_s) take(nr, wr);
        V u;
        int e[CPL], w[CPL];
        u.mul(nl, nr);
        obs(u, tp);
        rescale(u, e);
#pragma unroll
        for (int q = 0; q < CPL; ++q) {
          e[q] += (wl[q] >> 2) + (wr[q] >> 2);
          w[q] = (e[q] << 2) | ((wl[q] | wr[q]) & 2) | (wl[q] & wr[q] & 2) >> 1;
        }
        // the next step's loads run under this one's product
        keep_s = cur.sp;
        if (i + 1 < nst) fetch(nxt);
        if (cur.sp < 0) {
          ur = u;
#pragma unroll
          for (int q = 0; q < CPL; ++q) eR[q] = e[q], iR[q] = w[q] & 1;
          ring_free();
        } else {
          mprod(keep, u, cur.p, false);
          ring_free();
          slot_st(keep, w, cur.sp);
#pragma unroll
          for (int q = 0; q < CPL; ++q) wk[q] = w[q];
        }
        cur = nxt;
        nxt = nn;
      }
      // P = pi . U_root
      float invP[CPL];
      V O;
#pragma unroll
      for (int q = 0; q < CPL; ++q) O.row(q, pr0g, sg);
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        // one sum over the states in their order, as the other walks form it
        float pp = 0.f;
#pragma unroll
        for (int j = 0; j < A; ++j) {
          const int i = (A == 20 && j >= 16) ? 4 : (j / 16) * 4 + (j & 3);
          const int from = ((A == 20 && j >= 16) ? j - 16 : (j % 16) / 4) * 8 + cg;
          pp = fmaf(__shfl_sync(0xffffffffu, O.get(q, i), from), __shfl_sync(0xffffffffu, ur.get(q, i), from), pp);
        }
        invP[q] = 1.0f / pp;
        if (cc0 + q < c_count) {
          const size_t col = (size_t)c_base + cc0 + q;
          if ((P.mode & kModeLogLike) && sg == 0) P.logL[col] = (float)((double)eR[q] * kLn2b + (double)logf(pp));
          if (P.mode & kModeRootProb)
#pragma unroll
            for (int i = 0; i < SPL; ++i)
              P.rootp[(size_t)qstate<A>(i, sg) * C + col] = O.get(q, i) * ur.get(q, i) * invP[q];
        }
      }
      if (MODE == 0 || nst == 0) continue;

      // ------------------------------------------------------------- outside
      // branch n's rows of the staging (and its scalars for the F81 path)
      const size_t row0 = (size_t)cc0 * A, rowN = (size_t)c_count * A;
      auto emit = [&](int n, const V &D, const V *U, const int (&tk)[CPL], const int (&eDU)[CPL],
                      const int (&act)[CPL]) {
        float *pa = stage_a + (size_t)(n - 1) * rowN + row0, *pb = stage_b + (size_t)(n - 1) * rowN + row0;
#pragma unroll
        for (int q = 0; q < CPL; ++q) {
          float s = invP[q] * __int_as_float((max(-127, min(127, eDU[q] - eR[q])) + 127) << 23);
          s = act[q] ? s : 0.f;
          const bool ok = cc0 + q < c_count;
          const int code = btcode(tk[q], A);
          if (ok) {
            const int rot = flags & kQRotate ? stage_rot(A, cc0 + q) : 0;
            D.put(q, s, pa + q * A, sg, rot);
            if (U) {
              U->put(q, 1.f, pb + q * A, sg, rot);
            } else if (flags & kQLeafU) {
              V L;
#pragma unroll
              for (int i = 0; i < SPL; ++i) L.at(0, i) = (code >= A || code == qstate<A>(i, sg)) ? 1.f : 0.f;
              L.put(0, 1.f, pb + q * A, sg, rot);
            }
          }
          if constexpr (F81M) {
            if (P.stage_c) {
              float pu = 0.f, ds = 0.f;
#pragma unroll
              for (int i = 0; i < SPL; ++i) {
                const float x = U ? U->get(q, i) : (code >= A || code == qstate<A>(i, sg)) ? 1.f : 0.f;
                pu = fmaf(piv.get(q, i), x, pu);
                ds += D.get(q, i) * s;
              }
              pu = qsum(pu), ds = qsum(ds);
              if (ok && sg == 0) P.stage_c[(size_t)(n - 1) * c_count + cc0 + q] = make_float2(pu, ds);
            }
          }
        }
      };
      auto act_of = [&](int n, int q, int stn, int stp) -> int {
        if (P.mask_mode == kMaskAuto) return stn & stp;
        if (P.mask_mode == kMaskGiven) return P.mask[(size_t)n * C + co[q]] != 0;
        return 1;
      };
      cur = prog(nst - 1);
      nxt = prog(max(nst - 2, 0));
      keep_s = -2;
      fetch(cur);
      for (int i = nst - 1; i >= 0; --i) {
        const QStep nn = prog(max(i - 2, 0));
        ring_wait();
        if (cur.kl < 0) leaf(nl, wl, tl, cur.l, 0);
        if (cur.kr < 0) leaf(nr, wr, tr, cur.r, 1);
        int eO[CPL], stp[CPL];
        if (cur.sp < 0) {
          // O is the root prior here
          obs(O, tp);
#pragma unroll
          for (int q = 0; q < CPL; ++q) eO[q] = 0, stp[q] = iR[q];
        } else {
          // keep: the node's D
          int act[CPL], eU[CPL], e[CPL];
          V U;
          U.mul(nl, nr);
          obs(U, tp);
          rescale(U, eU);
#pragma unroll
          for (int q = 0; q < CPL; ++q) {
            eU[q] += (wl[q] >> 2) + (wr[q] >> 2) + (wk[q] >> 2);
            stp[q] = (wk[q] >> 1) & 1;
            act[q] = wk[q] & 1;
          }
          emit(cur.p, keep, &U, tp, eU, act);
          mprod(O, keep, cur.p, true);
          obs(O, tp);
          rescale(O, e);
#pragma unroll
          for (int q = 0; q < CPL; ++q) eO[q] = (wk[q] >> 2) + e[q];
        }
        ring_free();
        V Dl, Dr;
        int el[CPL], er[CPL], sl[CPL], sr[CPL], al[CPL], ar[CPL];
        Dl.mul(O, nr);
        Dr.mul(O, nl);
#pragma unroll
        for (int q = 0; q < CPL; ++q) {
          el[q] = eO[q] + (wr[q] >> 2);
          er[q] = eO[q] + (wl[q] >> 2);
          sl[q] = (wl[q] & 1) | (stp[q] & (wl[q] >> 1) & 1);
          sr[q] = (wr[q] & 1) | (stp[q] & (wr[q] >> 1) & 1);
          al[q] = act_of(cur.l, q, sl[q], stp[q]);
          ar[q] = act_of(cur.r, q, sr[q], stp[q]);
        }
        int cl[CPL], cr[CPL];
#pragma unroll
        for (int q = 0; q < CPL; ++q) cl[q] = tl[q], cr[q] = tr[q];
        // nl and nr are free: the next step's loads run under the stores.
        // Its D: the child whose step comes next (reverse postorder: the
        // right one when it is internal) stays in registers.
        const int fwd = cur.kr >= 0 ? cur.kr : cur.kl;
        if (i > 0) {
          fetch(nxt);
          if (nxt.sp != fwd) slot_ld(keep, wk, nxt.sp);
        }
        if (cur.kl < 0) {
          emit(cur.l, Dl, nullptr, cl, el, al);
        } else {
          int w[CPL];
#pragma unroll
          for (int q = 0; q < CPL; ++q) w[q] = (el[q] << 2) | (sl[q] << 1) | al[q];
          if (cur.kl == fwd) {
            keep = Dl;
#pragma unroll
            for (int q = 0; q < CPL; ++q) wk[q] = w[q];
          } else {
            slot_st(Dl, w, cur.kl);
          }
        }
        if (cur.kr < 0) {
          emit(cur.r, Dr, nullptr, cr, er, ar);
        } else {
          keep = Dr;
#pragma unroll
          for (int q = 0; q < CPL; ++q) wk[q] = (er[q] << 2) | (sr[q] << 1) | ar[q];
        }
        cur = nxt;
        nxt = nn;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_err && P.err) atomicAdd(P.err, 1);
}

// CTAs of an instance that fit on an SM.
template <int A, int CPL, bool F, int M, int MINB>
int qocc() {
  static std::atomic<int> cached{0};
  int nb = cached.load();
  if (nb) return nb;
  const size_t smem = QG<A, CPL>::smem(F);
  auto fn = k_qwalk<A, CPL, F, M, MINB>;
  if (allow_smem<k_qwalk<A, CPL, F, M, MINB>>() != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, q_threads<CPL, F>(), smem) != cudaSuccess || nb < 1)
    return 1;
  cached.store(nb);
  return nb;
}

template <int A, int CPL, bool F, int M, int MINB>
int qlaunch(const KParams &p, float *sa, float *sb, int flags, int c_base, int c_count, int grid, cudaStream_t s) {
  const size_t smem = QG<A, CPL>::smem(F);
  cudaError_t e = allow_smem<k_qwalk<A, CPL, F, M, MINB>>();
  if (e != cudaSuccess) return (int)e;
  k_qwalk<A, CPL, F, M, MINB><<<grid, q_threads<CPL, F>(), smem, s>>>(p, sa, sb, flags, c_base, c_count);
  return (int)cudaGetLastError();
}

// f(Int<A>, Int<CPL>, Int<F81>, Int<MODE>, Int<MINB>) for the instance of a call
template <int N>
struct QI {
  static constexpr int value = N;
};
template <class Fn>
int qdispatch(int A, int cpl, bool f81, bool outside, Fn &&f) {
  auto mode = [&](auto a, auto c, auto fm, auto b) {
    return outside ? f(a, c, fm, QI<1>{}, b) : f(a, c, fm, QI<0>{}, b);
  };
  if (f81) {
    switch (A) {
      case 16: return cpl == 1 ? mode(QI<16>{}, QI<1>{}, QI<1>{}, QI<4>{}) : mode(QI<16>{}, QI<2>{}, QI<1>{}, QI<3>{});
      case 20: return cpl == 1 ? mode(QI<20>{}, QI<1>{}, QI<1>{}, QI<4>{}) : mode(QI<20>{}, QI<2>{}, QI<1>{}, QI<3>{});
      case 32: return cpl == 1 ? mode(QI<32>{}, QI<1>{}, QI<1>{}, QI<4>{}) : mode(QI<32>{}, QI<2>{}, QI<1>{}, QI<2>{});
      case 64: return mode(QI<64>{}, QI<1>{}, QI<1>{}, QI<3>{});
    }
    return -1;
  }
  switch (A) {
    case 16: return cpl == 1 ? mode(QI<16>{}, QI<1>{}, QI<0>{}, QI<3>{}) : mode(QI<16>{}, QI<2>{}, QI<0>{}, QI<3>{});
    case 20: return cpl == 1 ? mode(QI<20>{}, QI<1>{}, QI<0>{}, QI<3>{}) : mode(QI<20>{}, QI<2>{}, QI<0>{}, QI<3>{});
    case 32: return cpl == 1 ? mode(QI<32>{}, QI<1>{}, QI<0>{}, QI<2>{}) : mode(QI<32>{}, QI<2>{}, QI<0>{}, QI<2>{});
  }
  return -1;
}

}  // namespace

bool qwalk_supported(int A, bool f81) { return A == 16 || A == 20 || A == 32 || (f81 && A == 64); }

int qwalk_grid(int A, bool f81, bool outside, int C, int nslots, int nsm, QGrid *g) {
  // One column per lane while that leaves at most 12 warps per SM: a call
  // of few columns is bound by a warp's latency per step, and half the
  // columns per warp are twice the warps (A = 16, R = 99, C = 4003: 76 us
  // against 108 us); with the SMs full, two columns per lane share each
  // matrix load (A = 20, R = 199, C = 20011: 450 against 487 us).  A = 64
  // has 16 states per lane and no registers for a second column (548
  // against 744 us).
  g->variant = (A == 64 || C <= nsm * 12 * 8) ? 1 : 2;
  return qdispatch(A, g->variant, f81, outside, [&](auto a, auto c, auto fm, auto m, auto b) {
    using G = QG<decltype(a)::value, decltype(c)::value>;
    const int occ = qocc<decltype(a)::value, decltype(c)::value, decltype(fm)::value != 0, decltype(m)::value,
                         decltype(b)::value>();
    g->grid = std::max(1, std::min((C + G::TILE - 1) / G::TILE, nsm * occ));
    const size_t warps = (size_t)g->grid * kQW * nslots;
    g->vec_bytes = warps * G::SLOT4 * sizeof(float4);
    g->slot_bytes = g->vec_bytes + warps * 4 * G::W * sizeof(int);
    return 0;
  });
}

int launch_qwalk(const KParams &p, int A, bool f81, bool outside, float *sa, float *sb, int flags, int c_base,
                 int c_count, const QGrid &g, cudaStream_t s) {
  return qdispatch(A, g.variant, f81, outside, [&](auto a, auto c, auto fm, auto m, auto b) {
    return qlaunch<decltype(a)::value, decltype(c)::value, decltype(fm)::value != 0, decltype(m)::value,
                   decltype(b)::value>(p, sa, sb, flags, c_base, c_count, g.grid, s);
  });
}

}  // namespace subby
