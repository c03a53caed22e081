// A = 4: inside pass, outside pass and count accumulation (or node / branch
// posteriors) with the nodes' vectors in global memory (subby/oracle/
// oracle.py:784-1256, 1372-1435, 1755-1905).  The arithmetic of k_tree4, one
// or two columns per thread.
//
// k_tree4 keeps a column's vectors in tensor memory, which allows 256 columns
// and 8 warps per SM: 34 % of the issue slots.  Here a node's contribution
// M_n U_n goes to global memory as it is formed (16 + 4 bytes) and comes back
// once, in the outside step of its parent, loaded a step ahead; what the next
// step needs stays in registers, and a child that waits sits on a short
// shared-memory stack (the program enters the deeper child first, k_inside4).
// 12 warps of two columns share an SM, the columns share the program's words
// and every matrix row, and Vd, Vu and pi are constant-bank operands.  The
// tokens are read once: their codes travel in the words beside the vectors.
// R = 255, 2^20 columns (GB300): 3227 -> 2097 us; R = 1023, 50001 columns
// 1530 -> 549 us; node posteriors R = 127, 100001 columns 224 -> 132 us.
// What bounds it: issue (60 %; 38 % of the instructions are integer work) and
// the L2 / HBM latency of the node slots (294 MB for the resident columns,
// 2.6 GB each way per 2^20 columns).  On the way there: without the codes in
// the words 2675 us (the outside pass waited for the second read of the
// tokens), and 2532 us with an L2 prefetch of it.
#include <limits.h>

#include <algorithm>

#include "a4.cuh"
#include "common.cuh"

namespace subby {
namespace {

constexpr int kHint = 8;   // steps of lead of the token rows' L2 prefetch
constexpr int kPrev = INT_MIN;   // the program's mark of a child in registers (k_inside4)

// The program (p, children, own stack slot; the step of the child that waits
// on the stack) as a kernel parameter: read with uniform indices, its words
// stay in uniform registers, so that the branches on them need no
// convergence bookkeeping and the addresses built from them no vector
// instructions.
constexpr int kPass4Steps = 1024;
template <int S>
struct A4Prog {
  int4 step[S];
  int other[S];
};

// Vd, Vu, the FP32 pi: with compile-time indices their elements are operands
// from the constant bank.
struct A4Const {
  float vd[16], vu[16], pi[4];
};

// A CTA's shared memory: tables, then the stack.  TBN: floats per branch of
// the second table (J 16, F81 coefficients 4, posteriors none).
struct P4Smem {
  float *MT, *TB, *LV, *Ut, *piL;
  float4 *vec;   // stack [slot][column][thread]
  int *word;
};
template <int TBN>
__device__ __forceinline__ P4Smem p4_layout(float *sm, int R, int stack) {
  P4Smem m;
  m.MT = sm;                    // R x 5 x 4
  m.TB = m.MT + R * 20;         // R x TBN
  m.LV = m.TB + R * TBN;        // L(code): 5 x 4
  m.Ut = m.LV + 20;             // U~(code): 5 x 4
  m.piL = m.Ut + 20;            // pi . L(code): 5
  m.vec = reinterpret_cast<float4 *>(m.piL + 8);
  m.word = reinterpret_cast<int *>(m.vec + stack);
  return m;
}
// fill the tables (all threads; the caller synchronises)
template <int TBN>
__device__ __forceinline__ void p4_load(const KParams &P, const P4Smem &m) {
  const int t = threadIdx.x, nb = blockDim.x;
  for (int i = t; i < P.R * 5; i += nb)
    reinterpret_cast<float4 *>(m.MT)[i] = __ldg(reinterpret_cast<const float4 *>(P.tab + P.off.MT) + i);
  if constexpr (TBN > 0)
    for (int i = t; i < P.R * TBN / 4; i += nb)
      reinterpret_cast<float4 *>(m.TB)[i] =
          __ldg(reinterpret_cast<const float4 *>(P.tab + (TBN == 4 ? P.off.F81 : P.off.J)) + i);
  if (t < 20) {
    m.LV[t] = (t / 4 == 4 || t / 4 == t % 4) ? 1.f : 0.f;
    m.Ut[t] = __ldg(P.tab + P.off.Ut + t);
  }
  if (t < 5) {
    float s = 0.f;
#pragma unroll
    for (int a = 0; a < 4; ++a) s = fmaf(__ldg(P.tab + P.off.pi + a), (t == 4 || t == a) ? 1.f : 0.f, s);
    m.piL[t] = s;
  }
}

// One tile: the columns c0 + lane + 32 q of each warp (c0 the warp's first).
// gv, gw: this thread's place in the CTA's global slots [step][column][thread].
// W, T: A4Const and A4Prog, or structs of pointers with the same members.
template <bool F81, int MASK, int OUT, int N, class Consts, class Prog>
__device__ __forceinline__ void p4_tile(const KParams &P, const Consts &W, const Prog &T, const P4Smem &M4,
                                        float4 *gv, int *gw, const int c0) {
  const int nb = blockDim.x, t = threadIdx.x, C = P.C, nst = P.nsteps, lane = t & 31;
  const float *MT = M4.MT, *TB = M4.TB, *LV = M4.LV, *Ut = M4.Ut, *piL = M4.piL;
  float4 *vec = M4.vec;
  int *word = M4.word;
  const F4 pr0 = ld4s(P.tab + P.off.pi0);
  const float mu81 = P.f81_mu;
  // w: exponent << 11 | token codes of the node's step << 2 | two mask flags
  // (inside: h, init; outside: in the Steiner tree, branch active).  A code is
  // min(token, 5), three bits each for the node, its left and its right child
  // (leaves): the outside pass takes them from here and reads no tokens.
  struct Vec {
    F4 v[N];
    int w[N];
  };
  constexpr int kE = 11, kCodes = 0x7fc;

  auto gload = [&](Vec &x, int st) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const float4 f = __ldcg(gv + (size_t)(st * N + q) * nb);
      x.v[q] = F4{make_float2(f.x, f.y), make_float2(f.z, f.w)};
      x.w[q] = __ldcg(gw + (size_t)(st * N + q) * nb);
    }
  };
  auto push = [&](const Vec &x, int slot) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int at = (slot * N + q) * nb + t;
      vec[at] = make_float4(x.v[q].a.x, x.v[q].a.y, x.v[q].b.x, x.v[q].b.y);
      word[at] = x.w[q];
    }
  };
  auto pop = [&](Vec &x, int slot) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int at = (slot * N + q) * nb + t;
      x.v[q] = ld4s(reinterpret_cast<const float *>(vec + at));
      x.w[q] = word[at];
    }
  };

  {
    int col[N];
    bool valid[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      valid[q] = c0 + lane + 32 * q < C;
      col[q] = min(c0 + lane + 32 * q, C - 1);
    }
    struct Tk {
      int p[N], l[N], r[N];
    };
    auto tok = [&](int (&o)[N], int n) {
      const int32_t *row = P.aln + (size_t)n * C;
#pragma unroll
      for (int q = 0; q < N; ++q) o[q] = __ldg(row + col[q]);
    };
    auto fetch = [&](Tk &o, int i) {
      const int4 s = T.step[i];
      tok(o.p, s.x);
      if (s.y >= 0) tok(o.l, s.y);
      if (s.z >= 0) tok(o.r, s.z);
    };
    // a step's tokens into L2, some steps before `fetch` loads them
    auto hint = [&](int i) {
      const int4 s = T.step[i];
      auto row = [&](int n) {
        const int32_t *r = P.aln + (size_t)n * C;
#pragma unroll
        for (int q = 0; q < N; ++q) asm volatile("prefetch.global.L2 [%0];" ::"l"(r + col[q]));
      };
      row(s.x);
      if (s.y >= 0) row(s.y);
      if (s.z >= 0) row(s.z);
    };
    // contribution of leaf n: its row of M_n; code 4 (unobserved) counts as
    // ungapped, 5 (a gap) does not
    auto leaf = [&](Vec &x, int n, const int (&code)[N]) {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        x.v[q] = ld4s(MT + (n * 5 + min(code[q], 4)) * 4);
        x.w[q] = code[q] <= 4 ? 3 : 0;
      }
    };
    // observed internal node: a row of ones otherwise, which one vote skips
    auto any_obs = [&](const int (&code)[N]) {
      bool any = false;
#pragma unroll
      for (int q = 0; q < N; ++q) any |= code[q] < 4;
      return __any_sync(0xffffffffu, any) != 0;
    };
    auto obs = [&](F4 (&x)[N], const int (&code)[N]) {
#pragma unroll
      for (int q = 0; q < N; ++q) x[q] = mul4(x[q], ld4s(LV + min(code[q], 4) * 4));
    };
    // ---------------------------------------------------------------- inside
    Vec keep;   // the vector handed to the next step in registers
    F4 ur[N];
    int eR[N];
    {
      Tk k0, k1;
      fetch(k0, 0);
      fetch(k1, min(1, nst - 1));
      auto step = [&](int i, const Tk &k) {
        const int4 s = T.step[i];
        Vec a, b;
        Tk c;
#pragma unroll
        for (int q = 0; q < N; ++q) {
          c.p[q] = (int)min((unsigned)k.p[q], 5u);
          c.l[q] = s.y >= 0 ? (int)min((unsigned)k.l[q], 5u) : 0;
          c.r[q] = s.z >= 0 ? (int)min((unsigned)k.r[q], 5u) : 0;
        }
        if (s.y >= 0) leaf(a, s.y, c.l);
        else if (s.y == kPrev) a = keep;
        else pop(a, ~s.y);
        if (s.z >= 0) leaf(b, s.z, c.r);
        else if (s.z == kPrev) b = keep;
        else pop(b, ~s.z);
        F4 u[N];
#pragma unroll
        for (int q = 0; q < N; ++q) u[q] = mul4(a.v[q], b.v[q]);
        if (any_obs(c.p)) obs(u, c.p);
#pragma unroll
        for (int q = 0; q < N; ++q) {
          const int e = (a.w[q] >> kE) + (b.w[q] >> kE) + rescale4(u[q]);
          keep.w[q] = (e << kE) | (c.p[q] << 2) | (c.l[q] << 5) | (c.r[q] << 8) | ((a.w[q] | b.w[q]) & 2) |
                      ((a.w[q] & b.w[q] & 2) >> 1);
        }
        if (i == nst - 1) {
#pragma unroll
          for (int q = 0; q < N; ++q) ur[q] = u[q], eR[q] = keep.w[q] >> kE;
          return;
        }
        const float *M = MT + s.x * 20;
        const F4 m0 = ld4s(M), m1 = ld4s(M + 4), m2 = ld4s(M + 8), m3 = ld4s(M + 12);
#pragma unroll
        for (int q = 0; q < N; ++q) {
          F4 y = scale4(m0, u[q].a.x);
          y = fma4(u[q].a.y, m1, y);
          y = fma4(u[q].b.x, m2, y);
          keep.v[q] = fma4(u[q].b.y, m3, y);
          __stcg(gv + (size_t)(i * N + q) * nb,
                 make_float4(keep.v[q].a.x, keep.v[q].a.y, keep.v[q].b.x, keep.v[q].b.y));
          __stcg(gw + (size_t)(i * N + q) * nb, keep.w[q]);
        }
        if (s.w >= 0) push(keep, s.w);
      };
      // two token sets, so that no register is copied
      int i = 0;
      for (int j = 2; j < min(kHint, nst); ++j) hint(j);
      for (; i + 2 <= nst; i += 2) {
        hint(min(i + kHint, nst - 1));
        hint(min(i + kHint + 1, nst - 1));
        step(i, k0);
        fetch(k0, min(i + 2, nst - 1));
        step(i + 1, k1);
        fetch(k1, min(i + 3, nst - 1));
      }
      if (i < nst) step(i, k0);
    }
    float invP[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const float Pp = dot4(pr0, ur[q]);
      invP[q] = 1.0f / Pp;
      if (valid[q] && (P.mode & kModeLogLike))
        P.logL[col[q]] = (float)((double)eR[q] * kLn2q + (double)logf(Pp));
      if (valid[q] && (P.mode & kModeRootProb)) {
        const F4 r = scale4(mul4(pr0, ur[q]), invP[q]);
        P.rootp[col[q]] = r.a.x;
        P.rootp[(size_t)C + col[q]] = r.a.y;
        P.rootp[(size_t)2 * C + col[q]] = r.b.x;
        P.rootp[(size_t)3 * C + col[q]] = r.b.y;
      }
    }
    if (OUT == kOutSum && !(P.mode & kModeCounts)) return;
    // --------------------------------------------------------------- outside
    F4 acc[N][4], hacc[N], gacc[N];   // eigen C rows / F81 G rows; F81 h, g, z
    float zacc[N];
    const F4 zero = F4{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
    for (int q = 0; q < N; ++q) {
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[q][k] = zero;
      hacc[q] = gacc[q] = zero;
      zacc[q] = 0.f;
    }
    // branch above node n; code (leaves): its table rows, null for internal n
    auto branch = [&](int n, const F4 (&D)[N], const F4 (&U)[N], const int *code, const int (&eDU)[N],
                      const int (&act)[N]) {
      if constexpr (OUT == kOutPost) {
        // y = D^T M_n; node posterior y o U / Z, branch joint D_i M_n[i][j] U_j / Z
        if (P.npost_node >= 0 && n != P.npost_node) return;
        const float *Mn = MT + n * 20;
        const size_t row = P.npost_node < 0 ? (size_t)n : 0;
#pragma unroll
        for (int q = 0; q < N; ++q) {
          const F4 p = mul4(vecmat4(Mn, D[q]), U[q]);
          const float z = sum4(p);
          const float inv = z > 0.f ? 1.0f / z : 1.0f;
          if (!valid[q]) continue;
          if (P.npost) {
            // streamed stores: written once, not re-read here
            float *o = P.npost + row * 4 * C + col[q];
            __stcs(o, p.a.x * inv);
            __stcs(o + C, p.a.y * inv);
            __stcs(o + (size_t)2 * C, p.b.x * inv);
            __stcs(o + (size_t)3 * C, p.b.y * inv);
          }
          if (P.bpost) {
            float *o = P.bpost + row * 16 * C + col[q];
            const F4 ui = scale4(U[q], inv);
            const float dk[4] = {D[q].a.x, D[q].a.y, D[q].b.x, D[q].b.y};
#pragma unroll
            for (int i2 = 0; i2 < 4; ++i2) {
              // row i of M_n is column i of the MT rows: M_n[i][j] = MT[n][j][i]
              const F4 mi = F4{make_float2(Mn[i2], Mn[4 + i2]), make_float2(Mn[8 + i2], Mn[12 + i2])};
              const F4 r = scale4(mul4(mi, ui), dk[i2]);
              __stcs(o + (size_t)(4 * i2) * C, r.a.x);
              __stcs(o + (size_t)(4 * i2 + 1) * C, r.a.y);
              __stcs(o + (size_t)(4 * i2 + 2) * C, r.b.x);
              __stcs(o + (size_t)(4 * i2 + 3) * C, r.b.y);
            }
          }
        }
        return;
      } else {
        F4 Ds[N];
#pragma unroll
        for (int q = 0; q < N; ++q) {
          float s = invP[q] * __int_as_float((max(-127, min(127, eDU[q] - eR[q])) + 127) << 23);
          if (MASK != kMaskNone) s = act[q] ? s : 0.f;
          Ds[q] = scale4(D[q], s);
        }
        if constexpr (F81) {
          const float4 abg = *reinterpret_cast<const float4 *>(TB + n * 4);
          const F4 piv = F4{make_float2(W.pi[0], W.pi[1]), make_float2(W.pi[2], W.pi[3])};
#pragma unroll
          for (int q = 0; q < N; ++q) {
            const float piU = code ? piL[code[q]] : dot4(piv, U[q]);
            const float dsum = sum4(Ds[q]);
            const float bh = abg.y * piU, bg = abg.y * dsum;
            const F4 aD = scale4(Ds[q], abg.x);
            acc[q][0] = fma4(aD.a.x, U[q], acc[q][0]);
            acc[q][1] = fma4(aD.a.y, U[q], acc[q][1]);
            acc[q][2] = fma4(aD.b.x, U[q], acc[q][2]);
            acc[q][3] = fma4(aD.b.y, U[q], acc[q][3]);
            hacc[q] = fma4(bh, Ds[q], hacc[q]);
            gacc[q] = fma4(bg, U[q], gacc[q]);
            zacc[q] = fmaf(abg.z * dsum, piU, zacc[q]);
          }
        } else {
          // D~_k = sum_a Ds_a Vd[a][k], U~_l = sum_b U_b Vu[b][l]
          auto proj = [](const auto &m, const F4 &x) {
            const float v[4] = {x.a.x, x.a.y, x.b.x, x.b.y};
            float y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              y[k] = m[k] * v[0];
#pragma unroll
              for (int a = 1; a < 4; ++a) y[k] = fmaf(v[a], m[4 * a + k], y[k]);
            }
            return F4{make_float2(y[0], y[1]), make_float2(y[2], y[3])};
          };
          F4 dt[N], ut[N];
#pragma unroll
          for (int q = 0; q < N; ++q) {
            dt[q] = proj(W.vd, Ds[q]);
            ut[q] = code ? ld4s(Ut + code[q] * 4) : proj(W.vu, U[q]);
          }
          const float *Jn = TB + n * 16;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const F4 j = ld4s(Jn + 4 * k);
#pragma unroll
            for (int q = 0; q < N; ++q) {
              const float d = k == 0 ? dt[q].a.x : k == 1 ? dt[q].a.y : k == 2 ? dt[q].b.x : dt[q].b.y;
              acc[q][k] = fma4(d, mul4(j, ut[q]), acc[q][k]);
            }
          }
        }
      }
    };
    auto act_of = [&](int n, int q, int stn, int stpar) -> int {
      if constexpr (MASK == kMaskAuto) return stn & stpar;
      else if constexpr (MASK == kMaskGiven) return P.mask[(size_t)n * C + col[q]] != 0;
      else return 1;
    };
    Vec pl, pr;   // the internal children's contributions, loaded a step ahead
    auto gfetch = [&](int i) {
      const int4 s = T.step[i];
      if (s.y < 0) gload(pl, s.y == kPrev ? i - 1 : T.other[i]);
      if (s.z < 0) gload(pr, s.z == kPrev ? i - 1 : T.other[i]);
    };
    gfetch(nst - 1);
#pragma unroll 1
    for (int i = nst - 1; i >= 0; --i) {
      const int4 s = T.step[i];
      // keep: D of this node, handed over by its parent's step or from the
      // stack (the root: only its word, from the inside pass)
      if (s.w >= 0) pop(keep, s.w);
      Tk k;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        k.p[q] = (keep.w[q] >> 2) & 7;
        k.l[q] = (keep.w[q] >> 5) & 7;
        k.r[q] = (keep.w[q] >> 8) & 7;
      }
      const bool seen = any_obs(k.p);
      Vec nl, nr;
      if (s.y >= 0) leaf(nl, s.y, k.l);
      else nl = pl;
      if (s.z >= 0) leaf(nr, s.z, k.r);
      else nr = pr;
      if (i > 0) gfetch(i - 1);
      F4 O[N];
      int eO[N], stp[N];
      if (i == nst - 1) {
#pragma unroll
        for (int q = 0; q < N; ++q) O[q] = pr0, eO[q] = 0, stp[q] = keep.w[q] & 1;
        if (seen) obs(O, k.p);
      } else {
        F4 U[N];
        int eDU[N], act[N];
#pragma unroll
        for (int q = 0; q < N; ++q) U[q] = mul4(nl.v[q], nr.v[q]);
        if (seen) obs(U, k.p);
#pragma unroll
        for (int q = 0; q < N; ++q) {
          eDU[q] = (keep.w[q] >> kE) + (nl.w[q] >> kE) + (nr.w[q] >> kE) + rescale4(U[q]);
          stp[q] = (keep.w[q] >> 1) & 1;
          act[q] = keep.w[q] & 1;
        }
        branch(s.x, keep.v, U, nullptr, eDU, act);
        const float *M = MT + s.x * 20;
        const F4 m0 = ld4s(M), m1 = ld4s(M + 4), m2 = ld4s(M + 8), m3 = ld4s(M + 12);
#pragma unroll
        for (int q = 0; q < N; ++q)
          O[q] = F4{make_float2(dot4(m0, keep.v[q]), dot4(m1, keep.v[q])),
                    make_float2(dot4(m2, keep.v[q]), dot4(m3, keep.v[q]))};
        if (seen) obs(O, k.p);
#pragma unroll
        for (int q = 0; q < N; ++q) eO[q] = (keep.w[q] >> kE) + rescale4(O[q]);
      }
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const int c = side ? s.z : s.y;
        const Vec &me = side ? nr : nl, &sib = side ? nl : nr;
        const int n = c >= 0 ? c : T.step[c == kPrev ? i - 1 : T.other[i]].x;
        Vec d;
        int e[N], act[N];
#pragma unroll
        for (int q = 0; q < N; ++q) {
          d.v[q] = mul4(O[q], sib.v[q]);
          e[q] = eO[q] + (sib.w[q] >> kE);
          const int st = (me.w[q] & 1) | (stp[q] & (me.w[q] >> 1) & 1);
          act[q] = act_of(n, q, st, stp[q]);
          d.w[q] = (e[q] << kE) | (me.w[q] & kCodes) | (st << 1) | act[q];
        }
        if (c >= 0) {
          F4 L[N];
          int code[N];
#pragma unroll
          for (int q = 0; q < N; ++q) {
            code[q] = min(side ? k.r[q] : k.l[q], 4);
            L[q] = (F81 || OUT == kOutPost) ? ld4s(LV + code[q] * 4) : zero;
          }
          branch(n, d.v, L, code, e, act);
        } else if (c == kPrev) {
          keep = d;
        } else {
          push(d, ~c);
        }
      }
    }
    // -------------------------------------------------------------- epilogue
    if constexpr (OUT == kOutSum) {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        if (!valid[q]) continue;
        float *out = P.counts + col[q];
        if constexpr (F81) {
          const float pi_[4] = {W.pi[0], W.pi[1], W.pi[2], W.pi[3]};
          const float hh[4] = {hacc[q].a.x, hacc[q].a.y, hacc[q].b.x, hacc[q].b.y};
          const float gg[4] = {gacc[q].a.x, gacc[q].a.y, gacc[q].b.x, gacc[q].b.y};
#pragma unroll
          for (int i2 = 0; i2 < 4; ++i2) {
            const float cr[4] = {acc[q][i2].a.x, acc[q][i2].a.y, acc[q][i2].b.x, acc[q][i2].b.y};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float I = cr[j] + hh[i2] + pi_[i2] * (gg[j] + zacc[q]);
              out[(size_t)(i2 * 4 + j) * C] = (i2 == j) ? I : mu81 * pi_[j] * I;
            }
          }
        } else if (P.mode & kModeBT64) {
          const double *Vg = P.tab64;
          const double *Sg = P.tab64 + 16;
          double T[4][4];
#pragma unroll
          for (int k2 = 0; k2 < 4; ++k2) {
            const float cr[4] = {acc[q][k2].a.x, acc[q][k2].a.y, acc[q][k2].b.x, acc[q][k2].b.y};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              double v = 0.0;
#pragma unroll
              for (int l = 0; l < 4; ++l) v = fma((double)cr[l], __ldg(Vg + j * 4 + l), v);
              T[k2][j] = v;
            }
          }
#pragma unroll
          for (int i2 = 0; i2 < 4; ++i2)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              double v = 0.0;
#pragma unroll
              for (int k2 = 0; k2 < 4; ++k2) v = fma(__ldg(Vg + i2 * 4 + k2), T[k2][j], v);
              out[(size_t)(i2 * 4 + j) * C] = (float)((i2 == j) ? v : __ldg(Sg + i2 * 4 + j) * v);
            }
        } else {
          const float *V32 = P.tab + P.off.V, *S32 = P.tab + P.off.S;
          float T[4][4];
#pragma unroll
          for (int k2 = 0; k2 < 4; ++k2) {
            const float cr[4] = {acc[q][k2].a.x, acc[q][k2].a.y, acc[q][k2].b.x, acc[q][k2].b.y};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float v = 0.f;
#pragma unroll
              for (int l = 0; l < 4; ++l) v = fmaf(cr[l], __ldg(V32 + j * 4 + l), v);
              T[k2][j] = v;
            }
          }
#pragma unroll
          for (int i2 = 0; i2 < 4; ++i2)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float v = 0.f;
#pragma unroll
              for (int k2 = 0; k2 < 4; ++k2) v = fmaf(__ldg(V32 + i2 * 4 + k2), T[k2][j], v);
              out[(size_t)(i2 * 4 + j) * C] = (i2 == j) ? v : __ldg(S32 + i2 * 4 + j) * v;
            }
        }
      }
    }
  }
}

template <bool F81, int MASK, int OUT, int N, int S>
__global__ void __launch_bounds__(384, 1)
    k_pass4(const __grid_constant__ KParams P, const __grid_constant__ A4Const W, const __grid_constant__ A4Prog<S> T) {
  extern __shared__ __align__(16) float sm[];
  constexpr int TBN = OUT == kOutPost ? 0 : F81 ? 4 : 16;
  const int nb = blockDim.x, t = threadIdx.x;
  const P4Smem m = p4_layout<TBN>(sm, P.R, P.nslots * N * nb);
  p4_load<TBN>(P, m);
  __syncthreads();
  const size_t slots = (size_t)blockIdx.x * P.nsteps * N * nb + t;
  // (a loop of the whole CTA: its condition is uniform, so that the compiler
  // may keep the program's words in uniform registers)
  const int ntiles = (P.C + nb * N - 1) / (nb * N);
#pragma unroll 1
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    p4_tile<F81, MASK, OUT, N>(P, W, T, m, reinterpret_cast<float4 *>(P.scrV) + slots, P.scrW + slots,
                               (tile * nb + t - (t & 31)) * N);
}

// Persistent serving kernel over a flattened (job, column-range) queue: the
// columns of many small A = 4 jobs in one launch.  Each CTA claims work items
// one at a time, reloads the tables when the claimed item belongs to another
// job than the previous one, and runs the same per-column code as k_pass4, so
// every column's result equals that of a separate call.  A claim past the
// published items waits (bounded) for more until the queue is closed.
__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.sys.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
struct P4Consts {
  const float *vd, *vu, *pi;
};
struct P4Prog {
  const int4 *step;
  const int *other;
};

template <bool F81, int MASK>
__global__ void __launch_bounds__(kPackBlock, 2) k_pass4_packed(const P4Queue Q) {
  extern __shared__ __align__(16) float sm[];
  __shared__ int s_item;
  __shared__ float s_const[36];   // Vu, Vd, pi
  constexpr int TBN = F81 ? 4 : 16;
  const int nb = blockDim.x, t = threadIdx.x;
  const size_t slots = (size_t)blockIdx.x * Q.max_steps * nb + t;
  float4 *gv = Q.scrV + slots;
  int *gw = Q.scrW + slots;
  int loaded = -1;
  for (;;) {
    if (t == 0) {
      const int it = atomicAdd(Q.head, 1);
      int avail = ld_acquire(Q.published);
      for (int polls = 0; it >= avail && !ld_acquire(Q.closed) && polls < Q.wait_polls; ++polls) {
        __nanosleep(256);
        avail = ld_acquire(Q.published);
      }
      if (it < avail) {
        s_item = it;
      } else {
        // closed and drained: done; still open after the bounded wait: the
        // wait gave up, which the status word records
        if (!ld_acquire(Q.closed) && Q.err) atomicAdd(Q.err, 1);
        s_item = -1;
      }
    }
    __syncwarp();
    __syncthreads();
    const int it = s_item;
    if (it < 0) break;
    const int4 w = Q.items[it];
    const KParams &P = Q.jobs[w.x];
    // the program behind the stack
    const P4Smem m = p4_layout<TBN>(sm, P.R, P.nslots * nb);
    int4 *prog = reinterpret_cast<int4 *>(m.word + P.nslots * nb);
    int *other = reinterpret_cast<int *>(prog + P.nsteps);
    if (w.x != loaded) {
      // every thread is past the previous item (barrier above)
      p4_load<TBN>(P, m);
      for (int i = t; i < P.nsteps; i += nb) {
        prog[i] = P.prog[i];
        other[i] = P.prog_other[i];
      }
      if (t < 36) s_const[t] = __ldg(P.tab + (t < 32 ? P.off.Vu + t : P.off.pi + t - 32));
      __syncthreads();
      loaded = w.x;
    }
    for (int c0 = w.y; c0 < w.z; c0 += nb)
      p4_tile<F81, MASK, kOutSum, 1>(P, P4Consts{s_const + 16, s_const, s_const + 32}, P4Prog{prog, other}, m, gv, gw,
                                     c0 + t - (t & 31));
    __syncthreads();  // s_item and, on a job change, the tables are rewritten next
  }
}

template <bool F, int M>
int packed(const P4Queue &q, int grid, size_t smem, cudaStream_t s) {
  cudaError_t e = allow_smem<k_pass4_packed<F, M>>();
  if (e != cudaSuccess) return (int)e;
  k_pass4_packed<F, M><<<grid, kPackBlock, smem, s>>>(q);
  return (int)cudaGetLastError();
}

template <bool F81, int MASK, int OUT, int S>
int pass4_s(const KParams &p, const A4Const &w, const int4 *prog, const int *other, int per, int grid, int block,
            size_t smem, cudaStream_t s) {
  A4Prog<S> T;
  std::copy(prog, prog + p.nsteps, T.step);
  std::copy(other, other + p.nsteps, T.other);
  auto fn = per == 2 ? k_pass4<F81, MASK, OUT, 2, S> : k_pass4<F81, MASK, OUT, 1, S>;
  cudaError_t e = per == 2 ? allow_smem<k_pass4<F81, MASK, OUT, 2, S>>() : allow_smem<k_pass4<F81, MASK, OUT, 1, S>>();
  if (e != cudaSuccess) return (int)e;
  fn<<<grid, block, smem, s>>>(p, w, T);
  return (int)cudaGetLastError();
}
template <bool F81, int MASK, int OUT>
int pass4(const KParams &p, const A4Const &w, const int4 *prog, const int *other, int per, int grid, int block,
          size_t smem, cudaStream_t s) {
  return p.nsteps <= 128 ? pass4_s<F81, MASK, OUT, 128>(p, w, prog, other, per, grid, block, smem, s)
                         : pass4_s<F81, MASK, OUT, kPass4Steps>(p, w, prog, other, per, grid, block, smem, s);
}

}  // namespace

int pass4_steps() { return kPass4Steps; }

// One column per thread: tables, stack, then the program.
size_t pass4_packed_smem(int R, int nsteps, int nslots, bool f81) {
  return pass4_smem(R, nslots, kPackBlock, 1, f81, false) + (size_t)nsteps * 20;
}

int launch_pass4_packed(const P4Queue &q, bool f81, int mask_mode, int grid, size_t smem, cudaStream_t s) {
  if (f81) return mask_mode == kMaskAuto ? packed<true, kMaskAuto>(q, grid, smem, s) : packed<true, kMaskNone>(q, grid, smem, s);
  return mask_mode == kMaskAuto ? packed<false, kMaskAuto>(q, grid, smem, s) : packed<false, kMaskNone>(q, grid, smem, s);
}

size_t pass4_smem(int R, int nslots, int block, int per, bool f81, bool post) {
  return (size_t)R * 80 + (size_t)R * (post ? 0 : f81 ? 16 : 64) + 80 + 80 + 32 + (size_t)nslots * block * per * 20;
}

int launch_pass4(const KParams &p, const int4 *prog, const int *other, const float *vd, const float *vu, const float *pi, bool f81, int mask_mode, bool post,
                 int per, int grid, int block, size_t smem, cudaStream_t s) {
  A4Const w;
  for (int i = 0; i < 16; ++i) w.vd[i] = vd[i], w.vu[i] = vu[i];
  for (int i = 0; i < 4; ++i) w.pi[i] = pi[i];
  if (post) return pass4<false, kMaskNone, kOutPost>(p, w, prog, other, per, grid, block, smem, s);
  if (f81) {
    if (mask_mode == kMaskAuto) return pass4<true, kMaskAuto, kOutSum>(p, w, prog, other, per, grid, block, smem, s);
    if (mask_mode == kMaskGiven) return pass4<true, kMaskGiven, kOutSum>(p, w, prog, other, per, grid, block, smem, s);
    return pass4<true, kMaskNone, kOutSum>(p, w, prog, other, per, grid, block, smem, s);
  }
  if (mask_mode == kMaskAuto) return pass4<false, kMaskAuto, kOutSum>(p, w, prog, other, per, grid, block, smem, s);
  if (mask_mode == kMaskGiven) return pass4<false, kMaskGiven, kOutSum>(p, w, prog, other, per, grid, block, smem, s);
  return pass4<false, kMaskNone, kOutSum>(p, w, prog, other, per, grid, block, smem, s);
}

}  // namespace subby
