// Discrete adjoint of the FP64 plane-Couette step (the reverse-mode
// derivative that jax.grad takes through KMM.solve in
// examples/pcf_minimal_seed_jax.py:111-150).
//
// Inner products: coefficient arrays pair as Re sum conj(a) b over the full
// (Hermitian) spectrum, physical samples as sum a b.  In the half-spectrum
// storage of the step (kz >= 0) the full-spectrum weights (1 at kz = 0, 2 at
// kz > 0) sit on both sides of every per-pencil operator, so a per-pencil
// adjoint is the conjugate transpose of the pencil's operator, and the adjoint
// of the padded periodic-axis chain y_b -> z_b -> product -> z_f -> y_f is the
// same chain with the product replaced by its transpose: the transposes of the
// unnormalised inverse transforms are the forward transforms times My (Mz),
// those of the 1/My (1/Mz) scaled forward transforms the inverse transforms
// over My (Mz), and the factors cancel.
//
// Kernels:
//   adj_stage_kernel     every per-pencil operation of one reverse stage in one
//                        launch (adjoint of the x-operators, of the mass rows
//                        and of the solves), on the FP64 tensor cores
//   z_adjoint_warp_kernel / z_adjoint_kernel
//                        transposed rotational product: with w the adjoint of
//                        n = -(u_t x omega_t), adj u = w x omega_t and
//                        adj omega = u_t x w
//   pencil_terms_kernel  dst[:, p] (+)= sum_t c_t(ky, kz) Op_t src_t[:, p],
//                        Op_t a real x-matrix, its transpose or the identity
//                        (energy gradients, once per call)
#pragma once

#include "jfb_kmm_split.cuh"
#include "jfb_kmm_warpk.cuh"

namespace jfb {

// One term: coefficient (cre + i cim) ky^a kz^b (k^2)^c, c = -1 meaning 1/k^2
// (zero on the mean pencil).  mat == nullptr is the identity.
struct PTerm {
  const c64* src;
  const double* mat;  // row-major; forward operator of shape (dst_rows x src_rows),
                      // or (src_rows x dst_rows) when trans
  int src_rows;
  int trans;
  double cre, cim;
  int a, b, c;
};

constexpr int kMaxTerms = 8;

struct PTermList {
  c64* dst;
  int dst_rows;
  int accumulate;
  int n;
  PTerm t[kMaxTerms];
};

// block: 32 pencils (lanes) x 8 warps, each thread kTermRows consecutive
// destination rows of one pencil (every source value it loads serves all of
// them); grid (ceil(P / 32), ceil(dst_rows / (8 kTermRows)))
constexpr int kTermRows = 8;
__global__ void __launch_bounds__(256) pencil_terms_kernel(Dims d, PTermList L) {
  const int p = blockIdx.x * 32 + (threadIdx.x & 31);
  const int r0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * kTermRows;
  if (p >= d.P || r0 >= L.dst_rows) return;
  const size_t P = (size_t)d.P;
  const int nr = min(kTermRows, L.dst_rows - r0);
  const int row = p / d.Kz, kzi = p % d.Kz;
  c64 acc[kTermRows];
#pragma unroll
  for (int q = 0; q < kTermRows; ++q) acc[q] = cmk(0.0, 0.0);
  if (row != d.Ny / 2) {  // the y Nyquist row stays zero
    const double ky = ((row < d.Ny / 2) ? row : row - d.Ny) * d.dfy;
    const double kz = kzi * d.dfz;
    const double k2 = ky * ky + kz * kz;
    const bool mean = (p == 0);
    for (int t = 0; t < L.n; ++t) {
      const PTerm& T = L.t[t];
      double s = 1.0;
      for (int e = 0; e < T.a; ++e) s *= ky;
      for (int e = 0; e < T.b; ++e) s *= kz;
      if (T.c < 0) {
        if (mean) continue;
        s /= k2;
      } else {
        for (int e = 0; e < T.c; ++e) s *= k2;
      }
      c64 v[kTermRows];
#pragma unroll
      for (int q = 0; q < kTermRows; ++q) v[q] = cmk(0.0, 0.0);
      if (!T.mat) {
#pragma unroll
        for (int q = 0; q < kTermRows; ++q)
          if (q < nr) v[q] = T.src[(size_t)(r0 + q) * P + p];
      } else if (T.trans) {
        for (int k = 0; k < T.src_rows; ++k) {
          const c64 x = T.src[(size_t)k * P + p];
          const double* m = T.mat + (size_t)k * L.dst_rows + r0;
#pragma unroll
          for (int q = 0; q < kTermRows; ++q)
            if (q < nr) v[q] = v[q] + __ldg(m + q) * x;
        }
      } else {
        for (int k = 0; k < T.src_rows; ++k) {
          const c64 x = T.src[(size_t)k * P + p];
#pragma unroll
          for (int q = 0; q < kTermRows; ++q)
            if (q < nr) v[q] = v[q] + __ldg(T.mat + (size_t)(r0 + q) * T.src_rows + k) * x;
        }
      }
      const c64 cf = cmk(T.cre * s, T.cim * s);
#pragma unroll
      for (int q = 0; q < kTermRows; ++q) {
        acc[q] = acc[q] + cf * v[q];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kTermRows; ++q) {
    if (q >= nr) break;
    c64* out = L.dst + (size_t)(r0 + q) * P + p;
    *out = L.accumulate ? *out + acc[q] : acc[q];
  }
}

// ---------------------------------------------------------------------------
// One reverse stage.  With mu_k the solution of the stage's transposed system,
// the adjoint of a state and of its nonlinear term are sums over the stages
// that read them,
//   s = sum_i (M + gl_i L)^T cm_i mu_i + recon^H pro^H ax [+ add],
//   nu = sum_i cn_i mu_i + cn_new mu,   mu = S^-T s,
// (SBDF3: mu of the three following steps; IMEXRK3: of the following stages),
// so no adjoint state is kept or updated in memory: a stage reads the few mu
// it needs and AX (the adjoint of the x-physical fields of its linearisation
// point, from the y and z stages), and writes its mu and AH = R^H nu, the next
// linearisation point's input of the y and z stages.
//
// A CTA owns a tile of 16 pencils (+ky / -ky x 8 kz).  All x-operators are
// split by parity into half matrices and applied as FP64 tensor-core products
// on operand rows in shared memory (gemm_sw); S^-T is the product with the
// transposed inverse upper factor, then the substitution with the transposed
// unit lower factor.  At 65x64x64 one launch of 106 us replaces 21 launches
// of 39 us (one thread per pencil and eight rows, dense products on FMA pipes)
// and four banded solves of 43 us.  Bound by latency: six dependent phases at
// eight warps per SM.
// ---------------------------------------------------------------------------
enum AdjSub {  // rows x columns
  qA0E, qA0O, qB1E, qB1O, qB2E, qB2O,  // transposed velocity operators, by coefficient parity
  qFE, qFO,                            // F^T
  qK0E, qK0O, qK2E, qK2O, qK4E, qK4O,  // transposed Galerkin matrices of u
  qD0E, qD0O, qD2E, qD2O,              // and of g
  qR0E, qR0O, qR1E, qR1O, qR2E, qR2O,  // transposed nonlinear rows (nodes x parity)
  qNum
};
struct AdjStageOps {
  const double* frag;
  const int* krange;
  SubDesc sub[qNum];
  int Jh, Jl, nBe, nBo, nDe, nDo;
  const double *R3, *XD0, *XD2;  // mean flow: S_D Q (nD x N), Dirichlet Galerkin matrices
};
constexpr int kAdjMu = 4;
struct AdjMu {
  const c64 *u, *g, *vw;
  double cm, gl;  // weight of (M + gl L)^T mu in s
  double cn;      // weight in nu
};
struct AdjStageArgs {
  const c64* AX;                          // 6 x [Nx][P] or null
  const c64 *add_u, *add_g, *add_vw;      // added to s (null: none)
  int nmu;
  AdjMu mu[kAdjMu];
  int solve;                              // 0: out = s
  const double *su, *sg, *s00inv;
  int su_rec, sg_rec, blocks;
  c64 *out_u, *out_g, *out_vw;            // mu (or s); null: EU only
  c64* EU[3];                             // leaf: pro^H ax itself, nothing else
  double cn_new;
  c64* AH;                                // 3 x [Nx][P] or null
};

__host__ __device__ inline int adj_rows(int N, int nB, int nD) {
  const int in = 5 * (N + 4), sv = 2 * split_solve_rows(nB, nD) + round4((nD + 1) / 2) + round4(nD / 2);
  return in > sv ? in : sv;
}
inline size_t adj_smem(int N, int nB, int nD) {
  return ((size_t)adj_rows(N, nB, nD) * kSLd + 6 * nD) * sizeof(double);
}

__global__ void __launch_bounds__(kSThreads, 1)
    adj_stage_kernel(const __grid_constant__ Dims d, const __grid_constant__ AdjStageOps G,
                     const __grid_constant__ AdjStageArgs a) {
  extern __shared__ __align__(128) double sm[];
  __shared__ TileCols tc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int nKc = (d.Kz + 7) / 8, bid = blockIdx.x;
  const int kyi = bid / nKc, kz0 = (bid % nKc) * 8;
  const int nkz = min(8, d.Kz - kz0);
  const int N = d.Nx, Jh = G.Jh, nB = d.nB, nD = d.nD;
  const size_t P = (size_t)d.P;
  const double* __restrict__ frag = G.frag;
  const bool mean_cta = bid == 0;
  double* mean = sm + (size_t)adj_rows(N, nB, nD) * kSLd;  // (v, w): s, mu, nu
  c64* m_s = reinterpret_cast<c64*>(mean);
  c64* m_mu = m_s + nD;
  c64* m_nu = m_mu + nD;
  tile_columns(d, kyi, kz0, tc);
  __syncthreads();
  const int hw = tid >> 4, hc = tid & 15;
  const bool col_ok = (hc >> 3) < (kyi == 0 ? 1 : 2) && (hc & 7) < nkz;
  const size_t so = (size_t)((hc >> 3) ? d.Ny - kyi : kyi) * d.Kz + kz0 + (hc & 7);
  const int ib = (N + 3) & ~3;  // rows between input blocks
  if (mean_cta)
    for (int i = tid; i < nD; i += kSThreads) m_s[i] = a.add_vw ? a.add_vw[i] : cmk(0.0, 0.0);

  // this warp's row tiles of u and of g: tile t < mtE even rows, else odd
  constexpr int kQ = 2;
  struct Tile {
    int half, mt, nh;
  };
  auto tile_of = [&](int q, bool isg, Tile& t) {
    const int mtE = ((isg ? G.nDe : G.nBe) + 7) / 8, mtO = ((isg ? G.nDo : G.nBo) + 7) / 8;
    t.mt = warp + q * kSWarps;
    if (t.mt >= mtE + mtO) return false;
    t.half = t.mt >= mtE;
    if (t.half) t.mt -= mtE;
    t.nh = isg ? (t.half ? G.nDo : G.nDe) : (t.half ? G.nBo : G.nBe);
    return true;
  };
  auto prod = [&](int id, int mt, int base, double (&acc)[4][2]) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
    const SubDesc s = G.sub[id];
    const int* kr = G.krange + s.kr + 2 * mt;
    gemm_sw<4, 8>(frag + s.off + (size_t)mt * s.kt * 32, kr[0], kr[1], sm, base, 0, lane, acc);
  };
  auto cv = [](const double (&v)[4][2], int nt) { return cmk(v[nt][0], v[nt][1]); };

  // ---- 1. pro^H: inputs as mirror sums (row j < Jl, the middle node) and
  // differences (row N-1-j), five blocks ----
  double sU[kQ][4][2], sG[kQ][4][2];  // s of this warp's tiles
#pragma unroll
  for (int q = 0; q < kQ; ++q)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) sU[q][nt][0] = sU[q][nt][1] = sG[q][nt][0] = sG[q][nt][1] = 0.0;
  // rows of the later phases: F^T input, mass inputs (or s), linear inputs
  const int oF[2] = {0, round4(G.nDe)};  // even, odd D rows
  const int oV = oF[1] + round4(G.nDo);
  const int rU[2] = {0, round4(G.nBe)};
  const int rG[2] = {rU[1] + round4(G.nBo), rU[1] + round4(G.nBo) + round4(G.nDe)};
  const int oL = oV + split_solve_rows(nB, nD);
  if (a.AX) {
    for (int idx = tid; idx < Jh * kGW; idx += kSThreads) {
      const int j = idx / kGW, w = idx % kGW, jm = N - 1 - j, p = tc.p[w];
      const double ky = tc.ky[w], kz = tc.kz[w];
      c64 v[2][5];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        c64 x[6];
#pragma unroll
        for (int f = 0; f < 6; ++f)
          x[f] = p >= 0 && (s == 0 || jm != j) ? ldg_c(a.AX + ((size_t)f * N + (s ? jm : j)) * P + p)
                                               : cmk(0.0, 0.0);
        v[s][0] = x[0] + mul_i(ky * x[5] - kz * x[4]);
        v[s][1] = x[1] + mul_i(kz * x[3]);
        v[s][2] = x[5];
        v[s][3] = x[2] - mul_i(ky * x[3]);
        v[s][4] = x[4];
      }
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        *sat(sm, b * ib + j, w) = v[0][b] + v[1][b];
        if (jm != j) *sat(sm, b * ib + jm, w) = v[0][b] - v[1][b];
      }
    }
    for (int e = tid; e < 5 * (ib - N) * kSLd; e += kSThreads) {
      const int b = e / ((ib - N) * kSLd);
      sm[(size_t)(b * ib + N) * kSLd + e - b * (ib - N) * kSLd] = 0.0;
    }
    for (int e = tid; e < 4 * kSLd; e += kSThreads) sm[(size_t)5 * ib * kSLd + e] = 0.0;
    __syncthreads();
    double fin[kQ][4][2];
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      Tile t;
      if (tile_of(q, false, t))
        prod(t.half ? qA0O : qA0E, t.mt, t.half ? Jh : 0, sU[q]);
      if (!tile_of(q, true, t)) continue;
      double e1[4][2], e2[4][2], acc[4][2];
      const int b1 = t.half ? qB1O : qB1E, b2 = t.half ? qB2O : qB2E;
      // B1 has its column's parity about the mid-plane, B2 the opposite one
      const int o1 = t.half ? Jh : 0, o2 = t.half ? 0 : Jh;
      prod(b1, t.mt, ib + o1, e1);
      prod(b2, t.mt, 2 * ib + o2, acc);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) e1[nt][0] += acc[nt][0], e1[nt][1] += acc[nt][1];
      prod(b1, t.mt, 3 * ib + o1, e2);
      prod(b2, t.mt, 4 * ib + o2, acc);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) e2[nt][0] -= acc[nt][0], e2[nt][1] -= acc[nt][1];
      const int r = t.mt * 8 + g, i = 2 * r + t.half;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int w = nt * 4 + t4, p = tc.p[w];
        const double ky = tc.ky[w], kz = tc.kz[w], k2 = ky * ky + kz * kz;
        const c64 x1 = cv(e1, nt), x2 = cv(e2, nt);
        c64 f = cmk(0.0, 0.0), sg = f;
        if (k2 != 0.0) {
          const double y = ky / k2, z = kz / k2;
          f = cmk(0.0, 0.0) - mul_i(y * x1 + z * x2);
          sg = mul_i(y * x2 - z * x1);
        }
        fin[q][nt][0] = f.re, fin[q][nt][1] = f.im;
        sG[q][nt][0] = sg.re, sG[q][nt][1] = sg.im;
        if (p >= 0 && r < t.nh) {
          if (a.EU[1]) {
            a.EU[1][(size_t)i * P + p] = x1;
            a.EU[2][(size_t)i * P + p] = x2;
          } else if (p == 0) {  // mean flow: the real parts
            m_s[i] = m_s[i] + cmk(x1.re, x2.re);
          }
        }
      }
    }
    if (a.EU[0]) {
#pragma unroll
      for (int q = 0; q < kQ; ++q) {
        Tile t;
        if (!tile_of(q, false, t)) continue;
        const int r = t.mt * 8 + g;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const int p = tc.p[nt * 4 + t4];
          if (p >= 0 && r < t.nh) a.EU[0][(size_t)(2 * r + t.half) * P + p] = cv(sU[q], nt);
        }
      }
      return;  // whole grid: leaf mode
    }
    __syncthreads();  // the inputs are dead
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      Tile t;
      if (!tile_of(q, true, t)) continue;
      const int r = t.mt * 8 + g;
      if (r < round4(t.nh))
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
          *sat(sm, oF[t.half] + r, nt * 4 + t4) = r < t.nh ? cv(fin[q], nt) : cmk(0.0, 0.0);
    }
  }
  // ---- 2. mass inputs sum_i cm_i mu_i (and gl cm mu of the linear one) ----
  bool lin = false;
#pragma unroll
  for (int k = 0; k < kAdjMu; ++k) lin |= k < a.nmu && a.mu[k].gl != 0.0;
  for (int r = hw; r < nB + nD; r += kSThreads / 16) {
    const bool isg = r >= nB;
    const int i = isg ? r - nB : r;
    c64 c = cmk(0.0, 0.0), l = c;
    if (col_ok) {
#pragma unroll
      for (int k = 0; k < kAdjMu; ++k) {
        if (k >= a.nmu || a.mu[k].cm == 0.0) continue;
        const c64 v = a.mu[k].cm * ldg_c((isg ? a.mu[k].g : a.mu[k].u) + (size_t)i * P + so);
        c = c + v;
        l = l + a.mu[k].gl * v;
      }
    }
    const int row = (isg ? rG[i & 1] : rU[i & 1]) + (i >> 1);
    *sat(sm, oV + row, hc) = c;
    if (lin) *sat(sm, oL + row, hc) = l;
  }
  for (int q = 0; q < 4; ++q) {  // k padding
    const int n = q == 0 ? G.nBe : q == 1 ? G.nBo : q == 2 ? G.nDe : G.nDo;
    const int row = oV + (q < 2 ? rU[q] : rG[q - 2]) + n, cnt = round4(n) - n;
    for (int e = tid; e < cnt * kSLd; e += kSThreads) {
      sm[(size_t)row * kSLd + e] = 0.0;
      if (lin) sm[(size_t)(row + oL - oV) * kSLd + e] = 0.0;
    }
  }
  __syncthreads();
  // ---- 3. s = EU0 + F^T fin + mass rows ----
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
    Tile t;
    double x0[4][2], x2[4][2];
    if (tile_of(q, false, t)) {
      if (a.AX) {
        prod(t.half ? qFO : qFE, t.mt, oF[1 - t.half], x0);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) sU[q][nt][0] += x0[nt][0], sU[q][nt][1] += x0[nt][1];
      }
      prod(t.half ? qK0O : qK0E, t.mt, oV + rU[t.half], x0);
      prod(t.half ? qK2O : qK2E, t.mt, oV + rU[t.half], x2);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const double ky = tc.ky[nt * 4 + t4], kz = tc.kz[nt * 4 + t4], k2 = ky * ky + kz * kz;
        sU[q][nt][0] += d.Myz * (x2[nt][0] - k2 * x0[nt][0]);
        sU[q][nt][1] += d.Myz * (x2[nt][1] - k2 * x0[nt][1]);
      }
      if (lin) {
        double x4[4][2];
        prod(t.half ? qK0O : qK0E, t.mt, oL + rU[t.half], x0);
        prod(t.half ? qK2O : qK2E, t.mt, oL + rU[t.half], x2);
        prod(t.half ? qK4O : qK4E, t.mt, oL + rU[t.half], x4);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const double ky = tc.ky[nt * 4 + t4], kz = tc.kz[nt * 4 + t4], k2 = ky * ky + kz * kz;
#pragma unroll
          for (int c = 0; c < 2; ++c)
            sU[q][nt][c] += d.Myz * (k2 * k2 * x0[nt][c] - 2.0 * k2 * x2[nt][c] + x4[nt][c]);
        }
      }
    }
    if (tile_of(q, true, t)) {
      prod(t.half ? qD0O : qD0E, t.mt, oV + rG[t.half], x0);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) sG[q][nt][0] += d.Myz * x0[nt][0], sG[q][nt][1] += d.Myz * x0[nt][1];
      if (lin) {
        prod(t.half ? qD0O : qD0E, t.mt, oL + rG[t.half], x0);
        prod(t.half ? qD2O : qD2E, t.mt, oL + rG[t.half], x2);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const double ky = tc.ky[nt * 4 + t4], kz = tc.kz[nt * 4 + t4], k2 = ky * ky + kz * kz;
          sG[q][nt][0] += d.Myz * (x2[nt][0] - k2 * x0[nt][0]);
          sG[q][nt][1] += d.Myz * (x2[nt][1] - k2 * x0[nt][1]);
        }
      }
    }
  }
  if (mean_cta) {  // (M00 + gl L00)^T of the mean flow (the g slot of pencil 0 holds nothing)
    for (int i = tid; i < nD; i += kSThreads) {
      c64 v = m_s[i];
      for (int q = 0; q < a.nmu; ++q) {
        if (a.mu[q].cm == 0.0) continue;
        c64 x = cmk(0.0, 0.0);
        for (int k = i & 1; k < nD; k += 2) {
          const double m = __ldg(G.XD0 + (size_t)k * nD + i) +
                           (a.mu[q].gl != 0.0 ? a.mu[q].gl * __ldg(G.XD2 + (size_t)k * nD + i) : 0.0);
          x = x + m * a.mu[q].vw[k];
        }
        v = v + a.mu[q].cm * x;
      }
      m_s[i] = v;
    }
  }
  __syncthreads();  // all products done: the rows are free
#pragma unroll
  for (int q = 0; q < kQ; ++q) {
#pragma unroll
    for (int isg = 0; isg < 2; ++isg) {
      Tile t;
      if (!tile_of(q, isg, t)) continue;
      const int r = t.mt * 8 + g;
      if (r >= t.nh) continue;
      const c64* add = isg ? a.add_g : a.add_u;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int w = nt * 4 + t4, p = tc.p[w];
        c64 v = isg ? cv(sG[q], nt) : cv(sU[q], nt);
        if (add && p >= 0) v = v + add[(size_t)(2 * r + t.half) * P + p];
        *sat(sm, (isg ? rG[t.half] : rU[t.half]) + r, w) = p >= 0 ? v : cmk(0.0, 0.0);
      }
    }
  }
  __syncthreads();
  // ---- 4. mu = S^-T s ----
  if (a.solve) {
    // the tile's multipliers, used after the product
    double* Ls = sm + (size_t)split_solve_rows(nB, nD) * kSLd;
    const int per = 2 * (nB + nD);
    for (int e = tid; e < nkz * per; e += kSThreads) {
      const int md = e / per, k = e - md * per;
      const size_t mode = (size_t)kyi * d.Kz + kz0 + md;
      cp_async8(Ls + e, (k < 2 * nB) ? a.su + mode * a.su_rec + k
                                     : a.sg + mode * a.sg_rec + (k - 2 * nB));
    }
    cp_async_commit();
    // z = U^-T s: tiles of the transposed inverse (row c of z, column r of s),
    // row tiles from the last so that z may replace s
    for (int task = warp; task < 4 * (kGW / 2); task += kSWarps) {
      const int ms = task & 7, sys = (task >> 3) & 1, par = task >> 4;
      if (tc.p[ms] < 0) continue;
      const int n = sys ? nD : nB, m0 = (n + 1) / 2, m = par ? n / 2 : m0;
      const double* __restrict__ tri =
          (sys ? a.sg + (size_t)tc.mode[ms] * a.sg_rec : a.su + (size_t)tc.mode[ms] * a.su_rec) +
          2 * n + (par ? inv_class_size(m0, a.blocks) : 0);
      double* rows = sm + (size_t)(sys ? rG[par] : rU[par]) * kSLd;
      const int wb = ms + 8;
      const int col = 2 * ((g & 2) ? wb : ms) + (g & 1);
      const double* b = rows + (size_t)t4 * kSLd + (col ^ (t4 << 2));
      const int wx = 2 * ((t4 & 1) ? wb : ms);
      for (int ct = (m + 7) / 8 - 1; ct >= 0; --ct) {
        const int c = 8 * ct + g;
        double c0 = 0.0, c1 = 0.0, e0 = 0.0, e1 = 0.0;
#pragma unroll 4
        for (int kt = 0; kt < 2 * ct + 2; kt += 2) {
          const int r0 = 4 * kt + t4, r1 = r0 + 4;
          const double a0 = c < m && r0 <= c ? __ldg(tri + inv_entry(r0, c, a.blocks)) : 0.0;
          const double a1 = c < m && r1 <= c ? __ldg(tri + inv_entry(r1, c, a.blocks)) : 0.0;
          const double b0 = r0 < m ? b[(size_t)kt * 4 * kSLd] : 0.0;
          const double b1 = r1 < m ? b[(size_t)(kt + 1) * 4 * kSLd] : 0.0;
          dmma_8x8x4(c0, c1, a0, b0);
          dmma_8x8x4(e0, e1, a1, b1);
        }
        __syncwarp();
        if (t4 < 2 && c < m)
          *reinterpret_cast<double2*>(rows + (size_t)c * kSLd + (wx ^ ((c & 3) << 2))) =
              make_double2(c0 + e0, c1 + e1);
        __syncwarp();
      }
    }
    cp_async_wait_all();
    __syncthreads();
    // L^T mu = z from the last row, one thread per (pencil, system, parity)
    if (tid < 4 * kGW) {
      const int w = tid & 15, sys = (tid >> 4) & 1, par = tid >> 5;
      if (tc.p[w] >= 0) {
        const int n = sys ? nD : nB, m = par ? n / 2 : (n + 1) / 2, r0 = sys ? rG[par] : rU[par];
        const double* rec = Ls + (w & 7) * per + (sys ? 2 * nB : 0);
        c64 x1 = cmk(0.0, 0.0), x2 = x1;  // x_{r+1}, x_{r+2}
        double l1 = 0.0, l2 = 0.0;        // L[r+1, r], L[r+2, r] (class rows)
        for (int r = m - 1; r >= 0; --r) {
          c64 v = *sat(sm, r0 + r, w);
          v = v - l1 * x1;
          v = v - l2 * x2;
          *sat(sm, r0 + r, w) = v;
          x2 = x1;
          x1 = v;
          const int i = 2 * r + par;  // next: L[i, i-2] and L[i+2, i-2]
          l1 = rec[2 * i];
          l2 = r + 1 < m ? rec[2 * (i + 2) + 1] : 0.0;
        }
      }
    } else if (mean_cta) {
      for (int i = tid - 4 * kGW; i < nD; i += kSThreads - 4 * kGW) {
        c64 x = cmk(0.0, 0.0);
        for (int k = i & 1; k < nD; k += 2) x = x + __ldg(a.s00inv + (size_t)k * nD + i) * m_s[k];
        m_mu[i] = x;
      }
    }
    __syncthreads();
  } else if (mean_cta) {
    for (int i = tid; i < nD; i += kSThreads) m_mu[i] = m_s[i];
    __syncthreads();
  }
  // ---- 5. mu out, nu in place ----
  for (int r = hw; r < nB + nD; r += kSThreads / 16) {
    const bool isg = r >= nB;
    const int i = isg ? r - nB : r;
    c64* x = sat(sm, (isg ? rG[i & 1] : rU[i & 1]) + (i >> 1), hc);
    const c64 v = *x;
    if (col_ok) {
      const size_t e = (size_t)i * P + so;
      (isg ? a.out_g : a.out_u)[e] = v;
      if (a.AH) {
        c64 nu = a.cn_new * v;
#pragma unroll
        for (int k = 0; k < kAdjMu; ++k)
          if (k < a.nmu && a.mu[k].cn != 0.0)
            nu = nu + a.mu[k].cn * ldg_c((isg ? a.mu[k].g : a.mu[k].u) + e);
        *x = nu;
      }
    }
  }
  if (mean_cta)
    for (int i = tid; i < nD; i += kSThreads) {
      const c64 v = m_mu[i];
      a.out_vw[i] = v;
      c64 nu = a.cn_new * v;
      for (int k = 0; k < a.nmu; ++k)
        if (a.mu[k].cn != 0.0) nu = nu + a.mu[k].cn * a.mu[k].vw[i];
      m_nu[i] = nu;
    }
  if (!a.AH) return;
  for (int q = 0; q < 4; ++q) {  // k padding
    const int n = q == 0 ? G.nBe : q == 1 ? G.nBo : q == 2 ? G.nDe : G.nDo;
    const int row = (q < 2 ? rU[q] : rG[q - 2]) + n, cnt = round4(n) - n;
    for (int e = tid; e < cnt * kSLd; e += kSThreads) sm[(size_t)row * kSLd + e] = 0.0;
  }
  __syncthreads();
  // ---- 6. AH = R^H nu: nodes j and N-1-j from the even and odd halves ----
  const int MT = (Jh + 7) / 8;
  for (int task = warp; task < 2 * MT; task += kSWarps) {
    const int jt = task >> 1, col0 = (task & 1) * 16;
    double e0[2][2], o0[2][2], e1[2][2], o1[2][2], e2[2][2], o2[2][2];
    auto rp = [&](int id, int base, double (&acc)[2][2]) {
      acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = 0.0;
      const SubDesc s = G.sub[id];
      gemm_sw<2, 8>(frag + s.off + (size_t)jt * s.kt * 32, 0, s.kt, sm, base, col0, lane, acc);
    };
    rp(qR0E, rU[0], e0);
    rp(qR0O, rU[1], o0);
    rp(qR1E, rU[0], e1);
    rp(qR1O, rU[1], o1);
    rp(qR2E, rG[0], e2);
    rp(qR2O, rG[1], o2);
    const int j = jt * 8 + g, jm = N - 1 - j;
    if (j >= Jh) continue;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int w = (col0 >> 1) + nt * 4 + t4, p = tc.p[w];
      if (p < 0) continue;
      const double ky = tc.ky[w], kz = tc.kz[w], k2 = ky * ky + kz * kz;
      auto c2v = [&](const double (&v)[2][2]) { return cmk(v[nt][0], v[nt][1]); };
      // at j: E + O; at the mirror node E - O (R0, R2), O - E (R1)
      auto put = [&](int jj, c64 r0, c64 r1, c64 r2) {
        c64* A = a.AH + (size_t)jj * P + p;
        const size_t f = (size_t)N * P;
        c64 h1 = cmk(0.0, 0.0) - mul_i(d.Myz * (ky * r1 + kz * r2));
        c64 h2 = mul_i(d.Myz * (ky * r2 - kz * r1));
        if (p == 0) {
          double v = 0.0, q = 0.0;
          for (int i = 0; i < nD; ++i) {
            const double m = __ldg(G.R3 + (size_t)i * N + jj);
            v += m * m_nu[i].re;
            q += m * m_nu[i].im;
          }
          h1 = cmk(-v, 0.0);
          h2 = cmk(-q, 0.0);
        }
        A[0] = (d.Myz * k2) * r0;
        A[f] = h1;
        A[2 * f] = h2;
      };
      put(j, c2v(e0) + c2v(o0), c2v(e1) + c2v(o1), c2v(e2) + c2v(o2));
      if (jm != j) put(jm, c2v(e0) - c2v(o0), c2v(o1) - c2v(e1), c2v(e2) - c2v(o2));
    }
  }
}

// The transposed z stage (z_adjoint_kernel) with warp-shuffle transforms
// (Mz = 32 P, Kz <= 32 QK), one warp per (x, y) row, everything in registers:
// 71 -> 35 us at 65x64x64 against the shared-memory form, whose radix passes
// wait on barriers.
template <int P, int QK>
__global__ void __launch_bounds__(256) z_adjoint_warp_kernel(DevOps o, Dims d,
                                                             const c64* __restrict__ tw,
                                                             const c64* __restrict__ Y,
                                                             const c64* __restrict__ Wa,
                                                             c64* __restrict__ HZ) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (row >= d.Nx * d.My) return;
  WarpTw<P, double> w;
  load_warp_tw<P, double>(w, tw, lane);
  const size_t plane = (size_t)d.Nx * d.My * d.Kz;
  c64 ph[5][P];
#pragma unroll
  for (int pr = 0; pr < 5; ++pr) {
    c64 A[QK], B[QK];
#pragma unroll
    for (int q = 0; q < QK; ++q) {
      const int k = 32 * q + lane;
      auto get = [&](int f) {  // 0..5 forward u, omega; 6..8 adjoint w; 9 none
        if (k >= d.Kz || f > 8) return cmk(0.0, 0.0);
        return (f < 6 ? Y + (size_t)f * plane : Wa + (size_t)(f - 6) * plane)[(size_t)row * d.Kz + k];
      };
      A[q] = get(2 * pr);
      B[q] = get(2 * pr + 1);
    }
    build_packed<P, QK, double>(A, B, d.Kz, lane, ph[pr]);
    warp_fft_inverse<P, double>(ph[pr], w, lane);
  }
  const double ub = d.uwall * o.xphys[row / d.My];
  c64 F[3][P];
#pragma unroll
  for (int r = 0; r < P; ++r) {
    const double u0 = ph[0][r].re, u1 = ph[0][r].im + ub, u2 = ph[1][r].re;
    const double w0 = ph[1][r].im, w1 = ph[2][r].re, w2 = ph[2][r].im + d.uwall;
    const double a0 = ph[3][r].re, a1 = ph[3][r].im, a2 = ph[4][r].re;
    F[0][r] = cmk(a1 * w2 - a2 * w1, a2 * w0 - a0 * w2);
    F[1][r] = cmk(a0 * w1 - a1 * w0, u1 * a2 - u2 * a1);
    F[2][r] = cmk(u2 * a0 - u0 * a2, u0 * a1 - u1 * a0);
  }
  const double scale = 1.0 / (32 * P);
#pragma unroll
  for (int pr = 0; pr < 3; ++pr) {
    warp_fft_forward<P, double>(F[pr], w, lane);
    c64 X[QK], Z[QK];
    unpack_pair<P, QK, double>(F[pr], lane, X, Z);
#pragma unroll
    for (int q = 0; q < QK; ++q) {
      const int k = 32 * q + lane;
      if (k >= d.Kz) continue;
      HZ[(size_t)(2 * pr) * plane + (size_t)row * d.Kz + k] = scale * X[q];
      HZ[(size_t)(2 * pr + 1) * plane + (size_t)row * d.Kz + k] = scale * Z[q];
    }
  }
}

// Transposed z stage, per group of kZRows (x, y) rows: the forward u, omega
// (six half spectra, padded in y) and the adjoint w of the product (three)
// -> five packed complex inverse FFTs, adj u = w x omega_t, adj omega =
// u_t x w with u_t = u + U_b e_y, omega_t = omega + U_wall e_z, then three
// packed forward transforms into six half spectra (adj u, adj omega).
__global__ void __launch_bounds__(256) z_adjoint_kernel(DevOps o, Dims d, FFTPlan plan,
                                                        const c64* __restrict__ tw,
                                                        const c64* __restrict__ Y,
                                                        const c64* __restrict__ Wa,
                                                        c64* __restrict__ HZ) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NP = 5;              // packed input pairs per row
  constexpr int NC = kZRows * NP;    // packed input columns
  constexpr int NCf = kZRows * 3;    // packed output columns
  c64* A = reinterpret_cast<c64*>(smem_raw);
  c64* B = A + d.Mz * NC;
  const int row0 = blockIdx.x * kZRows;
  const int nrows = d.Nx * d.My;
  const size_t plane = (size_t)d.Nx * d.My * d.Kz;
  auto field = [&](int f) -> const c64* {  // 0..5 forward u, omega; 6..8 adjoint w; 9 none
    return (f < 6) ? Y + (size_t)f * plane : (f < 9) ? Wa + (size_t)(f - 6) * plane : nullptr;
  };
  // k fastest: a warp reads consecutive spectral values of one row and field
  for (int idx = threadIdx.x; idx < d.Mz * NC; idx += blockDim.x) {
    const int k = idx % d.Mz, c = idx / d.Mz;
    const int rl = c / NP, pr = c % NP;
    const int row = row0 + rl;
    c64 z = cmk(0.0, 0.0);
    if (row < nrows) {
      const c64* fa = field(2 * pr);
      const c64* fb = field(2 * pr + 1);
      auto get = [&](const c64* f, int kk) {
        return f ? f[(size_t)row * d.Kz + kk] : cmk(0.0, 0.0);
      };
      if (k == 0) {
        z = cmk(get(fa, 0).re, get(fb, 0).re);
      } else if (k < d.Kz) {
        const c64 xa = get(fa, k), xb = get(fb, k);
        z = cmk(xa.re - xb.im, xa.im + xb.re);
      } else if (k > d.Mz - d.Kz) {
        const int kk = d.Mz - k;
        const c64 xa = get(fa, kk), xb = get(fb, kk);
        z = cmk(xa.re + xb.im, -xa.im + xb.re);
      }
    }
    A[k * NC + c] = z;
  }
  __syncthreads();
  c64* phys = fft_columns<double>(A, B, plan, NC, NC, tw, +1);
  c64* other = (phys == A) ? B : A;
  for (int idx = threadIdx.x; idx < d.Mz * kZRows; idx += blockDim.x) {
    const int rl = idx % kZRows, n = idx / kZRows;
    const int row = row0 + rl;
    const int j = (row < nrows) ? row / d.My : 0;
    const c64* z = phys + n * NC + rl * NP;
    const double ub = d.uwall * o.xphys[j];
    const double u0 = z[0].re, u1 = z[0].im + ub, u2 = z[1].re;
    const double w0 = z[1].im, w1 = z[2].re, w2 = z[2].im + d.uwall;
    const double a0 = z[3].re, a1 = z[3].im, a2 = z[4].re;
    c64* out = other + n * NCf + rl * 3;
    out[0] = cmk(a1 * w2 - a2 * w1, a2 * w0 - a0 * w2);
    out[1] = cmk(a0 * w1 - a1 * w0, u1 * a2 - u2 * a1);
    out[2] = cmk(u2 * a0 - u0 * a2, u0 * a1 - u1 * a0);
  }
  __syncthreads();
  c64* spec = fft_columns<double>(other, phys, plan, NCf, NCf, tw, -1);
  const double scale = 1.0 / d.Mz;
  for (int idx = threadIdx.x; idx < d.Kz * kZRows * 6; idx += blockDim.x) {
    const int k = idx % d.Kz;
    const int rf = idx / d.Kz;
    const int f = rf % 6, rl = rf / 6;
    const int row = row0 + rl;
    if (row >= nrows) continue;
    const int col = rl * 3 + f / 2;
    const c64 Zk = spec[k * NCf + col];
    const c64 Zm = spec[((d.Mz - k) % d.Mz) * NCf + col];
    c64 v;
    if ((f & 1) == 0) v = cmk(0.5 * (Zk.re + Zm.re), 0.5 * (Zk.im - Zm.im));
    else v = cmk(0.5 * (Zk.im + Zm.im), -0.5 * (Zk.re - Zm.re));
    HZ[(size_t)f * plane + (size_t)row * d.Kz + k] = scale * v;
  }
}

// Mean flow (v, w) added to the (0, 0) column of two half-spectrum arrays.
__global__ void add_mean_kernel(const c64* __restrict__ vw, int n, size_t P, c64* __restrict__ u1,
                                c64* __restrict__ u2) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    u1[(size_t)i * P].re += vw[i].re;
    u2[(size_t)i * P].re += vw[i].im;
  }
}

// y += a x on half-spectrum arrays.
__global__ void axpy_kernel(c64* __restrict__ y, const c64* __restrict__ x, double a, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    y[i] = y[i] + a * x[i];
}

}  // namespace jfb
