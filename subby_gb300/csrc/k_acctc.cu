// F81 fast-path accumulation at A = 64.
//
// The F81 counts of one column (subby/oracle/oracle.py:1190-1256) are
//   I_ij = G_ij + h_i + pi_i (g_j + z),
//   G = sum_n alpha_n (s D_n) (x) U_n,  h = sum_n beta_n (pi . U_n) s D_n,
//   g = sum_n beta_n sum(s D_n) U_n,    z = sum_n gamma_n sum(s D_n) (pi . U_n),
// with dwell = I_ii and substitutions mu pi_j I_ij.
//
// A leaf's U is one-hot (all ones for an unobserved token), so its outer
// product is one row added to G^T: half of the branches cost 64 additions
// instead of 4096 multiply-adds, and their U rows are not read.  Per CTA a
// group of 8 columns: the internal branches' products in registers (thread:
// 8 x 8 block of two columns, 16 loaded floats for 64 multiply-adds), the
// leaves' rows and the result in shared memory, [column][j][i].  Warp c also
// keeps column c's h, g, z (lane: two states) from the scalars (pi . U, sum
// s D) that the walk staged.
//
// Bound by latency at 16 warps per SM (issue 48 %, load pipe 51 % active): four
// branches per barrier.  R = 127, 20011 columns (GB300): 846 us; one branch
// per barrier 1133 us, 256 threads of two columns so 1045 us.  Products on the
// tensor cores (split-BF16 operands of two columns, 16 branches per K step)
// took 1245 us, most of it splitting and storing every branch's operands,
// with 7e-7 of error against 2e-7 here.
#include "common.cuh"

namespace subby {
namespace {

constexpr int kFA = 64;    // alphabet
constexpr int kFG = 8;     // columns per group
constexpr int kFN = 4;     // branches per ring stage (and barrier)
constexpr int kFS = 3;     // ring stages: the branches' s D and U rows
constexpr int kFRow = 68;  // floats between the rows [column][j] of the result: 8 rows on different banks
constexpr int kFBrn = 2 * kFG * kFA;        // one branch's rows
constexpr int kFStage = kFN * kFBrn;
constexpr int kFCol = kFA * kFRow + 4;   // and between columns: 8 columns x 4 rows on different banks
constexpr int kFRes = kFG * kFCol;
constexpr size_t kFBytes = (size_t)(kFRes + kFS * kFStage) * sizeof(float);
constexpr int kFT = 512;   // threads
constexpr int kFBr = kFT / kFG;   // branches whose scalars and tokens are loaded together: one (branch, column) per thread

constexpr int kWaitLimitT = 1 << 24;   // bounded mbarrier waits

__device__ __forceinline__ bool mbar_wait_t(uint32_t mb, uint32_t phase) {
  for (int it = 0; it < kWaitLimitT; ++it) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(mb), "r"(phase)
                 : "memory");
    if (done) return true;
  }
  return false;
}

__global__ void __launch_bounds__(kFT, 1)
    k_acc_f81(const KParams P, const float *__restrict__ sa, const float *__restrict__ sb,
              const float2 *__restrict__ sc, int c_base, int c_count) {
  extern __shared__ __align__(128) float sm[];
  float *res = sm, *ring = sm + kFRes;
  __shared__ __align__(8) uint64_t mbar[kFS];
  __shared__ int s_err;
  __shared__ __align__(16) float Hs[kFG][kFA], Gv[kFG][kFA], Os[kFG][kFA];
  __shared__ float Zs[kFG], pis[kFA];
  __shared__ __align__(16) float4 cf[2][kFBr];        // alpha, beta, gamma
  __shared__ __align__(8) float2 scl[2][kFBr][kFG];   // pi . U, sum s D
  __shared__ int tok[2][kFBr][kFG];                   // leaves: token code; -1: internal
  const int t = threadIdx.x;
  const int C = P.C, nbr = P.R - 1;
  const int ngroups = (c_count + kFG - 1) / kFG;
  const float4 *F8 = reinterpret_cast<const float4 *>(P.tab + P.off.F81);
  const float mu = P.f81_mu;
  // products: block (k0, l0) of column `cq`; h, g, the leaves' rows: state st
  const int cq = t >> 6, blk = t & 63, k0 = 8 * (blk & 7), l0 = 8 * (blk >> 3), st = t & 63;
  if (t == 0) {
    s_err = 0;
    for (int i = 0; i < kFS; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&mbar[i]))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (t < kFA) pis[t] = __ldg(P.tab + P.off.pi + t);
  __syncwarp();
  __syncthreads();
  const int nst = (nbr + kFN - 1) / kFN;   // ring stages per group
  uint32_t pos = 0;   // ring position of the group's first stage
  for (int gi = blockIdx.x; gi < ngroups; gi += gridDim.x, pos += nst) {
    const int g0 = gi * kFG, gcols = min(kFG, c_count - g0);
    const uint32_t bytes = (uint32_t)gcols * kFA * 4;
    // the branches kFN k .. of stage k (branch i: node i + 1), one per lane of warp 0
    auto load = [&](int k) {
      const int i = k * kFN + t;
      const bool on = t < kFN && i < nbr, up = on && __ldg(P.leaf + i + 1) == 0;
      const uint32_t rows = __popc(__ballot_sync(0xffffffffu, on)) + __popc(__ballot_sync(0xffffffffu, up));
      const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&mbar[(pos + k) % kFS]);
      if (t == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(rows * bytes) : "memory");
      __syncwarp();
      float *d = ring + (size_t)((pos + k) % kFS) * kFStage + t * kFBrn;
      const size_t off = ((size_t)i * c_count + g0) * kFA;
      if (on)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(d)), "l"(sa + off), "r"(bytes), "r"(mb) : "memory");
      if (up)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(d + kFG * kFA)), "l"(sb + off), "r"(bytes), "r"(mb)
                     : "memory");
      __syncwarp();
    };
    // the previous group's readers are past res and the ring
    __syncthreads();
    for (int i = t; i < kFRes; i += kFT) res[i] = 0.f;
    if (gcols < kFG)   // unused rows of a short group: finite values
      for (int i = t; i < kFS * kFN * 2 * (kFG - gcols) * kFA; i += kFT) {
        const int half = i / ((kFG - gcols) * kFA), e = i % ((kFG - gcols) * kFA);
        ring[half * kFG * kFA + gcols * kFA + e] = 0.f;
      }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (t < 32)
      for (int k = 0; k < kFS - 1 && k < nst; ++k) load(k);
    float2 acc[8][4];   // [k][l pair]
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int l = 0; l < 4; ++l) acc[k][l] = make_float2(0.f, 0.f);
    // h, g, z, and the rows of unobserved leaves (added to every j)
    float h = 0.f, g = 0.f, ones = 0.f, z = 0.f;
    // scalars, tokens and coefficients of kFBr branches at a time, loaded a block
    // ahead of their use
    float2 n_s;
    float4 n_cf = make_float4(0.f, 0.f, 0.f, 0.f);
    int n_tok;
    auto ahead = [&](int i0) {
      const int i = min(i0 + (t >> 3), nbr - 1), c = min(t & 7, gcols - 1);
      n_s = __ldg(sc + (size_t)i * c_count + g0 + c);
      n_tok = __ldg(P.leaf + i + 1)
                  ? (int)min((unsigned)__ldg(P.aln + (size_t)(i + 1) * C + c_base + g0 + c), (unsigned)kFA)
                  : -1;
      if (t < kFBr) n_cf = __ldg(F8 + min(i0 + t, nbr - 1) + 1);
    };
    auto put = [&](int b) {
      scl[b][t >> 3][t & 7] = n_s;
      tok[b][t >> 3][t & 7] = n_tok;
      if (t < kFBr) cf[b][t] = n_cf;
    };
    ahead(0);
    put(0);
    ahead(kFBr);
    for (int k = 0; k < nst; ++k) {
      const int i0 = k * kFN, ib = (i0 / kFBr) & 1;
      __syncthreads();   // every thread is done with the stage that this refills
      if (i0 % kFBr == 0) {   // (the other block's last readers are past the barrier)
        put(ib ^ 1);
        ahead(i0 + 2 * kFBr);
      }
      if (t < 32 && k + kFS - 1 < nst) load(k + kFS - 1);
      const uint32_t at = pos + k;
      if (!mbar_wait_t((uint32_t)__cvta_generic_to_shared(&mbar[at % kFS]), (at / kFS) & 1)) s_err = 1;
      const float *Ds = ring + (size_t)(at % kFS) * kFStage;
#pragma unroll 2
      for (int x = 0; x < kFN; ++x) {
        if (i0 + x >= nbr) break;
        const int ii = (i0 + x) % kFBr;
        const float *D = Ds + x * kFBrn, *U = D + kFG * kFA;
        const float d = D[cq * kFA + st];
        const float4 abg = cf[ib][ii];
        const float2 sv = scl[ib][ii][cq];
        const int code = tok[ib][ii][cq];
        const float bg = abg.y * sv.y;
        h = fmaf(abg.y * sv.x, d, h);
        z = fmaf(abg.z * sv.y, sv.x, z);
        if (code >= 0) {
          if (code < kFA) {
            float *r = res + cq * kFCol + code * kFRow + st;
            *r = fmaf(abg.x, d, *r);
            if (st == code) g += bg;
          } else {
            ones = fmaf(abg.x, d, ones);
            g += bg;
          }
          continue;
        }
        g = fmaf(bg, U[cq * kFA + st], g);
        const float *dq = D + cq * kFA + k0, *uq = U + cq * kFA + l0;
        const float4 d0 = *reinterpret_cast<const float4 *>(dq), d1 = *reinterpret_cast<const float4 *>(dq + 4);
        const float4 u0 = *reinterpret_cast<const float4 *>(uq), u1 = *reinterpret_cast<const float4 *>(uq + 4);
        const float dk[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
        const float2 ul[4] = {make_float2(u0.x, u0.y), make_float2(u0.z, u0.w), make_float2(u1.x, u1.y),
                              make_float2(u1.z, u1.w)};
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float ad = abg.x * dk[r];
          const float2 aa = make_float2(ad, ad);
#pragma unroll
          for (int l = 0; l < 4; ++l) acc[r][l] = __ffma2_rn(aa, ul[l], acc[r][l]);
        }
      }
    }
    // ------------------------------------------------------------- epilogue
    Hs[cq][st] = h;
    Gv[cq][st] = g;
    Os[cq][st] = ones;
    if (st == 0) Zs[cq] = z;
    __syncthreads();   // the leaves' rows are complete
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      float4 *r = reinterpret_cast<float4 *>(res + cq * kFCol + (l0 + l) * kFRow + k0);
      auto el = [&](int k) { return (l & 1) ? acc[k][l >> 1].y : acc[k][l >> 1].x; };
      const float4 a = r[0], b = r[1];
      r[0] = make_float4(a.x + el(0), a.y + el(1), a.z + el(2), a.w + el(3));
      r[1] = make_float4(b.x + el(4), b.y + el(5), b.z + el(6), b.w + el(7));
    }
    __syncthreads();
    // eight lanes write a row's eight columns (rows start at any alignment)
    const int c = t & 7;
    if (c < gcols) {
      const float *rc = res + c * kFCol;
      float *o = P.counts + c_base + g0 + c;
      for (int e = t >> 3; e < kFA * kFA; e += kFT / 8) {
        const int i = e & 63, j = e >> 6;
        const float I = rc[j * kFRow + i] + Os[c][i] + Hs[c][i] + pis[i] * (Gv[c][j] + Zs[c]);
        o[(size_t)(i * kFA + j) * C] = (i == j) ? I : mu * pis[j] * I;
      }
    }
  }
  __syncthreads();
  if (t == 0 && s_err && P.err) atomicAdd(P.err, 1);
}

}  // namespace

int launch_acc_f81_64(const KParams &p, const float *sa, const float *sb, const float2 *sc, int c_base, int c_count,
                      int grid, cudaStream_t s) {
  cudaError_t e = allow_smem<k_acc_f81>();
  if (e != cudaSuccess) return (int)e;
  k_acc_f81<<<grid, kFT, kFBytes, s>>>(p, sa, sb, sc, c_base, c_count);
  return (int)cudaGetLastError();
}

}  // namespace subby
