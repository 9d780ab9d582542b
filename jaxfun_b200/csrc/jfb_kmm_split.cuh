// Pencil stage of the KMM step for 65 < Nx <= 129, as two kernels of FP64
// tensor-core products (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind).
//
// The one-kernel stage (pencil_gemm_kernel) keeps every operand of a tile and
// the velocity operators in one CTA's shared memory, which ends at Nx = 65.
// Above, one warp per pencil ran recurrences and small products at 8 warps
// per SM (22 % issue, 7 % of the FP64 tensor pipe).  Here a CTA of eight
// warps owns the same tile of 16 pencils ((+ky, -ky) x 8 kz, so a
// wavenumber's factors serve two pencils) and the stage is cut where the
// operands change:
//   pencil_rhs_kernel       stages the mirror sums of H, forms Nu and Ng in
//                           registers, stages the mass-row inputs over the
//                           dead H rows, completes the right-hand sides,
//                           solves Su and Sg (forward elimination, then the
//                           inverse upper factors) and writes u0, g;
//   pencil_velocity_kernel  forms u, omega (or u and its gradients) at the x
//                           nodes from u0, g.
// Each needs at most half of an SM's shared memory and 128 registers per
// thread, so two CTAs share an SM.  The operators are the folded ones of
// build_gemm_operators, read from L2 as fragments by every CTA (copy
// b % nrep), eight in flight per warp.  Operand rows hold 16 complex values =
// 32 doubles without padding; groups of four doubles are XOR-swizzled by the
// row, so that the four rows x eight columns of a B fragment fall in distinct
// banks (a padded stride of 36 doubles would not leave room for two CTAs at
// Nx = 129).
//
// FP64 plans only: the mixed form keeps the warp-per-pencil stage.  Its
// velocities are rounded to FP32 for the transforms, and where two FP64
// evaluations fall on either side of a rounding boundary the nonlinear rows
// differ by up to 1e-7 (seen at 129x128x128 in one of four seeds), so a stage
// that sums in another order would not reproduce the form's results.
//
// Measured (steady SBDF3 stage, both kernels together, events around the
// launches): 97x96x96 434 -> 138 us, 129x128x128 1033 -> 331 us against the warp
// stage with one warp per pencil.  What a CTA spends its time on at 129x128x128:
// of 118 us in pencil_rhs_kernel the inverse factors from memory 36 (300 MB per
// stage), Nu and Ng on the FP64 tensor pipe 25, the level and history rows 15, the
// mass products 11; of 48 in pencil_velocity_kernel the products and stores 40.
#pragma once

#include "jfb_kmm_gemm.cuh"

namespace jfb {

constexpr int kSThreads = 256;
constexpr int kSWarps = kSThreads / 32;
constexpr int kSLd = 2 * kGW;  // doubles per operand row
constexpr int kSMaxN = 129;
constexpr int kSSlots = 4;     // row tiles of a product per warp

__host__ __device__ inline int split_hb(int N) {  // rows of one H block
  const int Jh = (N + 1) / 2, a = round4(N), b = Jh + round4(N / 2);
  return a > b ? a : b;
}
// Operand rows of the right-hand-side kernel (lin: the stage has a linear term).
__host__ __device__ inline int split_mass_rows(int nB, int nD, bool lin) {
  const int su = lin ? 3 : 2, sg = lin ? 2 : 1;
  return round4(su * ((nB + 1) / 2)) + round4(su * (nB / 2)) + round4(sg * ((nD + 1) / 2)) +
         round4(sg * (nD / 2));
}
// Rows of the right-hand sides: four blocks (system, parity), each a multiple of 4.
__host__ __device__ inline int split_solve_rows(int nB, int nD) {
  return round4((nB + 1) / 2) + round4(nB / 2) + round4((nD + 1) / 2) + round4(nD / 2);
}
inline size_t split_rhs_smem(int N, int nB, int nD, bool lin) {
  const size_t h = (size_t)3 * split_hb(N), m = split_mass_rows(nB, nD, lin);
  const size_t rows = (h > m ? h : m) * kSLd * sizeof(double);
  // the right-hand sides and their factors' multipliers reuse the rows
  const size_t solve =
      ((size_t)split_solve_rows(nB, nD) * kSLd + (size_t)(nB + nD) * 16) * sizeof(double);
  return (rows > solve ? rows : solve) + (size_t)(2 * N + 6 * nD) * sizeof(double);
}
inline size_t split_vel_smem(int nB, int nD) {
  const int rows = round4((nB + 1) / 2) + round4(nB / 2) + round4((nD + 1) / 2) + round4(nD / 2);
  return ((size_t)rows * kSLd + 6 * kSLd) * sizeof(double);
}

// Element (row, pencil w) of an operand block that starts at row 0 of sm.
__device__ __forceinline__ c64* sat(double* sm, int row, int w) {
  return reinterpret_cast<c64*>(sm) + row * kGW + (w ^ ((row & 3) << 1));
}

// acc += A(8-row tile) * B(rows from `base`, columns col0 + 8 nt ..), k tiles
// [kb, ke); CH fragments of A always in flight (a register ring).
template <int NT, int CH>
__device__ __forceinline__ void gemm_sw(const double* __restrict__ A, int kb, int ke,
                                        const double* sm, int base, int col0, int lane,
                                        double (&acc)[NT][2]) {
  const int g = lane >> 2, t4 = lane & 3;
  const int swz = ((base + t4) & 3) << 2;
  const double* b[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
    b[nt] = sm + (size_t)(base + 4 * kb + t4) * kSLd + ((col0 + nt * 8 + g) ^ swz);
  A += kb * 32 + lane;
  const int n = ke - kb;
  double a[CH];
#pragma unroll
  for (int k = 0; k < CH; ++k) a[k] = k < n ? __ldg(A + k * 32) : 0.0;
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += CH) {
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      if (k0 + k >= n) break;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        dmma_8x8x4(acc[nt][0], acc[nt][1], a[k], b[nt][k * 4 * kSLd]);
      if (k0 + k + CH < n) a[k] = __ldg(A + (k + CH) * 32);
    }
    A += CH * 32;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) b[nt] += CH * 4 * kSLd;
  }
}

// x = U^-1 y for one parity class of m <= 8 MTX rows of two pencils wa, wb
// (columns of operand rows of LD doubles), one warp: the inverse's 8x8 blocks
// (inv_entry) as A fragments against the pencils' four real columns; the
// other four columns of the product repeat them.  Block columns run from the
// last, the next one's loads in flight; one accumulator pair per row tile, so
// the MTX chains are independent and x is written once at the end (x == y
// allowed).  SWZ: groups of four doubles XOR-swizzled by the row (the blocks
// start on a multiple of four rows).
template <int MTX>
struct InvColumn {  // fragments of one block column
  double2 a[MTX];
};
template <int MTX>
__device__ __forceinline__ void inv_load(InvColumn<MTX>& col, const double* __restrict__ tri, int j,
                                         int lane) {
  const double2* p = reinterpret_cast<const double2*>(tri + j * (j + 1) / 2 * 64) + lane;
#pragma unroll
  for (int mt = 0; mt < MTX; ++mt)
    if (mt <= j) col.a[mt] = __ldg(p + mt * 32);
}
template <int LD, bool SWZ, int MTX>
__device__ __forceinline__ void inv_product(const double* __restrict__ tri, int m, const double* y,
                                            double* x, int wa, int wb, int lane,
                                            InvColumn<MTX>& next) {
  const int g = lane >> 2, t4 = lane & 3;
  const int col = 2 * ((g & 2) ? wb : wa) + (g & 1);  // B column g & 3: re, im of wa, of wb
  const double* b = y + (size_t)t4 * LD + (SWZ ? col ^ (t4 << 2) : col);
  double acc[MTX][2];
#pragma unroll
  for (int mt = 0; mt < MTX; ++mt) acc[mt][0] = acc[mt][1] = 0.0;
#pragma unroll 1
  for (int j = (m + 7) / 8 - 1; j >= 0; --j) {
    const InvColumn<MTX> cur = next;
    if (j > 0) inv_load(next, tri, j - 1, lane);
    const double b0 = 8 * j + t4 < m ? b[(size_t)8 * j * LD] : 0.0;
    const double b1 = 8 * j + 4 + t4 < m ? b[(size_t)(8 * j + 4) * LD] : 0.0;
#pragma unroll
    for (int mt = 0; mt < MTX; ++mt)
      if (mt <= j) {
        dmma_8x8x4(acc[mt][0], acc[mt][1], cur.a[mt].x, b0);
        dmma_8x8x4(acc[mt][0], acc[mt][1], cur.a[mt].y, b1);
      }
  }
  __syncwarp();
  const int wx = 2 * ((t4 & 1) ? wb : wa);  // lanes t4 < 2: columns 2 t4, 2 t4 + 1 are a pencil
#pragma unroll
  for (int mt = 0; mt < MTX; ++mt) {
    const int r = mt * 8 + g;
    if (t4 < 2 && r < m)
      *reinterpret_cast<double2*>(x + (size_t)r * LD + (SWZ ? wx ^ ((r & 3) << 2) : wx)) =
          make_double2(acc[mt][0], acc[mt][1]);
  }
}

// Pencils of tile `bid`: index, mode and wavenumbers per column (p < 0: none).
struct TileCols {
  int p[kGW], mode[kGW];
  double ky[kGW], kz[kGW];
};
__device__ __forceinline__ void tile_columns(const Dims& d, int kyi, int kz0, TileCols& t) {
  if (threadIdx.x < kGW) {
    const int c = threadIdx.x, side = c >> 3, kz = kz0 + (c & 7);
    const bool ok = kz < d.Kz && !(side == 1 && kyi == 0);
    t.p[c] = ok ? (side ? d.Ny - kyi : kyi) * d.Kz + kz : -1;
    t.mode[c] = ok ? kyi * d.Kz + kz : 0;
    t.ky[c] = ok ? (side ? -kyi : kyi) * d.dfy : 0.0;
    t.kz[c] = ok ? kz * d.dfz : 0.0;
  }
}

__global__ void __launch_bounds__(kSThreads, 2)
    pencil_rhs_kernel(const __grid_constant__ Dims d, const __grid_constant__ DevOps o,
                      const __grid_constant__ GemmOps G, const __grid_constant__ GemmStageArgs a) {
  extern __shared__ __align__(128) double sm[];
  __shared__ TileCols tc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int nKc = (d.Kz + 7) / 8, bid = blockIdx.x;
  const int kyi = bid / nKc, kz0 = (bid % nKc) * 8;
  const int nkz = min(8, d.Kz - kz0);
  const bool mean_cta = bid == 0;
  const int N = d.Nx, Jh = G.Jh, nB = d.nB, nD = d.nD;
  const size_t P = (size_t)d.P;
  const double* __restrict__ frag = G.frag + (size_t)(bid % G.nrep) * G.nfrag;
  const double sl = a.slin;
  const bool lin = sl != 0.0;
  const int hb = split_hb(N);
  const size_t mean_at = [&] {  // first double of the mean-flow scratch
    const int h = 3 * hb, m = split_mass_rows(nB, nD, lin);
    const size_t rows = (size_t)(h > m ? h : m) * kSLd,
                 solve = (size_t)split_solve_rows(nB, nD) * kSLd + (size_t)(nB + nD) * 16;
    return rows > solve ? rows : solve;
  }();
  double* mean = sm + mean_at;
  JFB_STAMP(2, 0);
  pdl_trigger();
  tile_columns(d, kyi, kz0, tc);
  __syncthreads();
  pdl_wait();

  // ------------------------------------------------------------------ A --
  // H_f row j -> block f row j, one half-warp per row (16 pencils)
  const int hw = tid >> 4, hc = tid & 15;
  const bool col_ok = (hc >> 3) < (kyi == 0 ? 1 : 2) && (hc & 7) < nkz;
  const size_t so = (size_t)((hc >> 3) ? d.Ny - kyi : kyi) * d.Kz + kz0 + (hc & 7);
  if (col_ok)
    for (int r = hw; r < 3 * N; r += kSThreads / 16) {
      const int f = r >= 2 * N ? 2 : r >= N ? 1 : 0;
      cp_async16(sat(sm, f * hb + r - f * N, hc), a.HX + (size_t)r * P + so);
    }
  cp_async_commit();
  // history and level rows of this tile into L2 while H arrives (each row is
  // one 128-byte line per side)
  {
    const c64* src[10] = {a.u0a, a.c1 != 0.0 ? a.u0b : nullptr, a.c2 != 0.0 ? a.u0c : nullptr,
                          a.d1 != 0.0 ? a.Nup : nullptr, a.d2 != 0.0 ? a.Nuq : nullptr,
                          a.ga, a.c1 != 0.0 ? a.gb : nullptr, a.c2 != 0.0 ? a.gc : nullptr,
                          a.d1 != 0.0 ? a.Ngp : nullptr, a.d2 != 0.0 ? a.Ngq : nullptr};
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      if (!src[q]) continue;
      for (int e = tid; e < 2 * (q < 5 ? nB : nD); e += kSThreads) {
        const int side = e & 1, i = e >> 1;
        if (side && kyi == 0) continue;
        const c64* ptr = src[q] + (size_t)i * P + (size_t)(side ? d.Ny - kyi : kyi) * d.Kz + kz0;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();
  JFB_STAMP(2, 1);
  // in place: mirror sums / differences with the (i ky, i kz, k^2) weights
  for (int idx = tid; idx < Jh * kGW; idx += kSThreads) {
    const int j = idx / kGW, w = idx % kGW, jm = N - 1 - j, p = tc.p[w];
    const bool ok = p >= 0;
    c64 h[2][3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      h[0][f] = ok ? *sat(sm, f * hb + j, w) : cmk(0.0, 0.0);
      h[1][f] = (ok && jm != j) ? *sat(sm, f * hb + jm, w) : cmk(0.0, 0.0);
    }
    if (mean_cta && w == 0) {
      mean[j] = h[0][1].re;
      mean[N + j] = h[0][2].re;
      if (jm != j) {
        mean[jm] = h[1][1].re;
        mean[N + jm] = h[1][2].re;
      }
    }
    const double ky = tc.ky[w], kz = tc.kz[w], k2 = ky * ky + kz * kz;
    c64 h12[2], k2h0[2], hg[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      h12[s] = mul_i(ky * h[s][1] + kz * h[s][2]);
      k2h0[s] = k2 * h[s][0];
      hg[s] = mul_i(kz * h[s][1] - ky * h[s][2]);
    }
    if (jm != j) {
      *sat(sm, j, w) = h12[0] - h12[1];
      *sat(sm, jm, w) = k2h0[0] + k2h0[1];
      *sat(sm, hb + j, w) = h12[0] + h12[1];
      *sat(sm, hb + jm, w) = k2h0[0] - k2h0[1];
      *sat(sm, 2 * hb + j, w) = hg[0] + hg[1];
      *sat(sm, 2 * hb + jm, w) = hg[0] - hg[1];
    } else {
      *sat(sm, j, w) = k2h0[0];
      *sat(sm, hb + j, w) = h12[0];
      *sat(sm, 2 * hb + j, w) = hg[0];
    }
  }
  for (int e = tid; e < 3 * (hb - N) * kSLd; e += kSThreads) {
    const int q = e / ((hb - N) * kSLd);
    sm[(size_t)(q * hb + N) * kSLd + e - q * (hb - N) * kSLd] = 0.0;
  }
  __syncthreads();

  JFB_STAMP(2, 2);
  // ------------------------------------------------------------------ B --
  // The row tiles of Nu (even rows, then odd) and Ng are one task list, heavy
  // first, dealt to the warps in a snake.  nl holds dt times the nonlinear
  // combination while the mass inputs replace H.
  const int nNu = G.sub[gNuE].mt + G.sub[gNuO].mt, nT = nNu + G.sub[gNgE].mt + G.sub[gNgO].mt;
  struct Task {
    int kind, half, mt, nh;  // Nu / Ng, parity, row tile, rows of the parity
  };
  auto task_of = [&](int q, Task& t) {
    int k = kSWarps * q + ((q & 1) ? kSWarps - 1 - warp : warp);
    if (k >= nT) return false;
    t.kind = k >= nNu;
    t.mt = t.kind ? k - nNu : k;
    const int mtE = G.sub[t.kind ? gNgE : gNuE].mt;
    t.half = t.mt >= mtE;
    if (t.half) t.mt -= mtE;
    t.nh = t.kind ? (t.half ? G.nDo : G.nDe) : (t.half ? G.nBo : G.nBe);
    return true;
  };
  double nl[kSSlots][4][2];
#pragma unroll
  for (int q = 0; q < kSSlots; ++q) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) nl[q][nt][0] = nl[q][nt][1] = 0.0;
    Task t;
    if (!task_of(q, t)) continue;  // whole warp
    const int id = t.kind ? (t.half ? gNgO : gNgE) : (t.half ? gNuO : gNuE);
    const SubDesc s = G.sub[id];
    const int2 kr = sub_krange(G, id, t.mt);
    const int base = t.kind ? 2 * hb + (t.half ? Jh : 0) : t.half * hb;
    gemm_sw<4, 8>(frag + s.off + (size_t)t.mt * s.kt * 32, kr.x, kr.y, sm, base, 0, lane, nl[q]);
    const int r = t.mt * 8 + g, i = 2 * r + t.half;
    const c64* Np = t.kind ? a.Ngp : a.Nup;
    const c64* Nq = t.kind ? a.Ngq : a.Nuq;
    c64* Nout = t.kind ? a.Ng_out : a.Nu_out;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int p = tc.p[nt * 4 + t4];
      if (p < 0 || r >= t.nh) continue;
      const size_t gi = (size_t)i * P + p;
      const c64 n0 = cmk(d.Myz * nl[q][nt][0], d.Myz * nl[q][nt][1]);
      if (Nout) Nout[gi] = n0;
      c64 v = a.d0 * n0;
      if (a.d1 != 0.0) v = v + a.d1 * ldg_c(Np + gi);
      if (a.d2 != 0.0) v = v + a.d2 * ldg_c(Nq + gi);
      nl[q][nt][0] = d.dt * v.re;
      nl[q][nt][1] = d.dt * v.im;
    }
  }
  __syncthreads();
  JFB_STAMP(2, 3);
  // mass-row inputs: u levels -> (v1, v2[, v3]), g levels -> (w1[, w2])
  const int nsu = lin ? 3 : 2, nsg = lin ? 2 : 1;
  int oM[4];  // Mu even, odd, Mg even, odd
  oM[0] = 0;
  oM[1] = round4(nsu * G.nBe);
  oM[2] = oM[1] + round4(nsu * G.nBo);
  oM[3] = oM[2] + round4(nsg * G.nDe);
  {
    const double ky = tc.ky[hc], kz = tc.kz[hc], k2 = ky * ky + kz * kz;
    const int p = tc.p[hc];
    constexpr int RS = kSThreads / 16, UB = 4;
    for (int r0 = hw; r0 < nB + nD; r0 += RS * UB) {
      c64 va[UB], vb[UB], vc[UB];
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int r = r0 + RS * u;
        const bool ok = p >= 0 && r < nB + nD, isg = r >= nB;
        const size_t e = (size_t)(isg ? r - nB : r) * P + (ok ? p : 0);
        va[u] = ok ? ldg_c((isg ? a.ga : a.u0a) + e) : cmk(0.0, 0.0);
        vb[u] = ok && a.c1 != 0.0 ? ldg_c((isg ? a.gb : a.u0b) + e) : cmk(0.0, 0.0);
        vc[u] = ok && a.c2 != 0.0 ? ldg_c((isg ? a.gc : a.u0c) + e) : cmk(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int r = r0 + RS * u;
        if (r >= nB + nD) continue;
        c64 cu = a.c0 * va[u];
        if (a.c1 != 0.0) cu = cu + a.c1 * vb[u];
        if (a.c2 != 0.0) cu = cu + a.c2 * vc[u];
        if (r < nB) {
          const int nh = (r & 1) ? G.nBo : G.nBe, row = oM[r & 1] + (r >> 1);
          if (!lin) {
            *sat(sm, row, hc) = cu;
            *sat(sm, row + nh, hc) = cmk(0.0, 0.0) - k2 * cu;
          } else {
            *sat(sm, row, hc) = cu - (2.0 * sl * k2) * va[u];
            *sat(sm, row + nh, hc) = (sl * k2 * k2) * va[u] - k2 * cu;
            *sat(sm, row + 2 * nh, hc) = sl * va[u];
          }
        } else {
          const int i = r - nB, nh = (i & 1) ? G.nDo : G.nDe, row = oM[2 + (i & 1)] + (i >> 1);
          *sat(sm, row, hc) = lin ? cu - (sl * k2) * va[u] : cu;
          if (lin) *sat(sm, row + nh, hc) = sl * va[u];
        }
      }
    }
    const int rows[4] = {nsu * G.nBe, nsu * G.nBo, nsg * G.nDe, nsg * G.nDo};
    for (int q = 0; q < 4; ++q)  // k padding
      for (int e = tid; e < (round4(rows[q]) - rows[q]) * kSLd; e += kSThreads)
        sm[(size_t)(oM[q] + rows[q]) * kSLd + e] = 0.0;
  }
  __syncthreads();
  JFB_STAMP(2, 4);
#pragma unroll
  for (int q = 0; q < kSSlots; ++q) {
    Task t;
    if (!task_of(q, t)) continue;
    const int id = t.kind ? (t.half ? gMgO : gMgE) : (t.half ? gMuO : gMuE);
    const SubDesc s = G.sub[id];
    int2 kr = sub_krange(G, id, t.mt);
    if (!lin) kr.y = min(kr.y, t.kind ? G.kt_mg_lin[t.half] : G.kt_mu_lin[t.half]);
    double acc[4][2];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
    gemm_sw<4, 8>(frag + s.off + (size_t)t.mt * s.kt * 32, kr.x, max(kr.x, kr.y), sm,
                  oM[2 * t.kind + t.half], 0, lane, acc);
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      nl[q][nt][0] += d.Myz * acc[nt][0];
      nl[q][nt][1] += d.Myz * acc[nt][1];
    }
  }
  __syncthreads();
  JFB_STAMP(2, 5);
  // right-hand sides to shared memory: Su rows by parity, then Sg rows, each
  // block on a multiple of four rows (the swizzle's period)
  const int oR[5] = {0, round4(G.nBe), round4(G.nBe) + round4(G.nBo),
                     round4(G.nBe) + round4(G.nBo) + round4(G.nDe), split_solve_rows(nB, nD)};
#pragma unroll
  for (int q = 0; q < kSSlots; ++q) {
    Task t;
    if (!task_of(q, t)) continue;
    const int r = t.mt * 8 + g;
    if (r >= t.nh) continue;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int w = nt * 4 + t4;
      *sat(sm, oR[2 * t.kind + t.half] + r, w) =
          tc.p[w] >= 0 ? cmk(nl[q][nt][0], nl[q][nt][1]) : cmk(0.0, 0.0);
    }
  }

  // ------------------------------------------------------------------ C --
  // forward-elimination multipliers of the tile's wavenumbers
  double* Ls = sm + (size_t)oR[4] * kSLd;
  const int per = 2 * (nB + nD);
  for (int e = tid; e < nkz * per; e += kSThreads) {
    const int md = e / per, k = e - md * per;
    const size_t mode = (size_t)kyi * d.Kz + kz0 + md;
    cp_async8(Ls + e, (k < 2 * nB) ? a.su + mode * a.su_rec + k
                                   : a.sg + mode * a.sg_rec + (k - 2 * nB));
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  JFB_STAMP(2, 6);
  c64* m_nvw = reinterpret_cast<c64*>(mean + 2 * N);
  c64* m_vw = reinterpret_cast<c64*>(mean + 2 * N + 2 * nD);
  c64* m_x = reinterpret_cast<c64*>(mean + 2 * N + 4 * nD);
  // (below) x = U^-1 y for both pencils of a wavenumber, one warp per
  // (wavenumber, system, parity), in place; the first loads start here.  On
  // FMA pipes with the inverse by columns this phase issued ten times the
  // instructions (51 us per CTA at Nx = 129).
  auto inverse_of = [&](int task, int& m) {
    const int ms = task & 7, sys = (task >> 3) & 1, par = task >> 4;
    const int n = sys ? nD : nB, m0 = (n + 1) / 2;
    m = par ? n / 2 : m0;
    return (sys ? a.sg + (size_t)tc.mode[ms] * a.sg_rec : a.su + (size_t)tc.mode[ms] * a.su_rec) +
           2 * n + (par ? inv_class_size(m0, true) : 0);
  };
  InvColumn<kSWarps> inv;
  {
    int m;
    const double* tri = inverse_of(warp, m);
    inv_load(inv, tri, (m + 7) / 8 - 1, lane);
  }
  if (tid < 4 * kGW) {  // one thread per (pencil, system, parity)
    const int w = tid & 15, sys = (tid >> 4) & 1, par = tid >> 5;
    if (tc.p[w] >= 0) {
      const int n = sys ? nD : nB, m = par ? n / 2 : (n + 1) / 2, r0 = oR[2 * sys + par];
      const double* ls = Ls + (w & 7) * per + (sys ? 2 * nB : 0) + 2 * par;
      c64 y1 = cmk(0.0, 0.0), y2 = y1, v = *sat(sm, r0, w);
      for (int r = 0; r < m; ++r) {
        const c64 nx = r + 1 < m ? *sat(sm, r0 + r + 1, w) : cmk(0.0, 0.0);
        v = v - ls[4 * r] * y1;
        v = v - ls[4 * r + 1] * y2;
        *sat(sm, r0 + r, w) = v;
        y2 = y1;
        y1 = v;
        v = nx;
      }
    }
  } else if (mean_cta) {
    // mean_flow's named barrier counts kMeanThreads threads
    static_assert(kSThreads - 4 * kGW == kMeanThreads);
    mean_flow(d, o, G, a, mean, m_nvw, m_vw, m_x, tid - 4 * kGW);
  }
  __syncthreads();
  JFB_STAMP(2, 7);
#pragma unroll 1
  for (int task = warp; task < 4 * (kGW / 2); task += kSWarps) {
    const int ms = task & 7, sys = (task >> 3) & 1, par = task >> 4;
    int m;
    const double* tri = inverse_of(task, m);
    if (task != warp) inv_load(inv, tri, (m + 7) / 8 - 1, lane);
    if (tc.p[ms] < 0) continue;
    double* rows = sm + (size_t)oR[2 * sys + par] * kSLd;
    inv_product<kSLd, true>(tri, m, rows, rows, ms, ms + 8, lane, inv);
  }
  __syncthreads();
  JFB_STAMP(2, 8);
  // solved coefficients to global memory, a half-warp per row
  if (col_ok) {
    bool bad = false;
    for (int r = hw; r < nB + nD; r += kSThreads / 16) {
      const bool isg = r >= nB;
      const int i = isg ? r - nB : r;
      const c64 v = *sat(sm, oR[(isg ? 2 : 0) + (i & 1)] + (i >> 1), hc);
      bad |= !finite_c(v);
      (isg ? a.g_out : a.u0_out)[(size_t)i * P + so] = v;
    }
    flag_nonfinite(G.status, bad);
  }
  JFB_STAMP(2, 9);
}

template <int kForm>
__global__ void __launch_bounds__(kSThreads, 2)
    pencil_velocity_kernel(const __grid_constant__ Dims d, const __grid_constant__ GemmOps G,
                           const __grid_constant__ GemmStageArgs a) {
  constexpr bool grad = kForm == 1;
  extern __shared__ __align__(128) double sm[];
  __shared__ TileCols tc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int nKc = (d.Kz + 7) / 8, bid = blockIdx.x;
  const int kyi = bid / nKc, kz0 = (bid % nKc) * 8;
  const int nkz = min(8, d.Kz - kz0);
  const int N = d.Nx, Jh = G.Jh, Jl = G.Jl, nB = d.nB, nD = d.nD;
  const size_t P = (size_t)d.P;
  const double* __restrict__ frag = G.frag + (size_t)(bid % G.nrep) * G.nfrag;
  const int oUE = 0, oUO = round4(G.nBe), oGE = oUO + round4(G.nBo), oGO = oGE + round4(G.nDe);
  double* mid = sm + (size_t)(oGO + round4(G.nDo)) * kSLd;
  JFB_STAMP(3, 0);
  pdl_trigger();
  tile_columns(d, kyi, kz0, tc);
  __syncthreads();
  pdl_wait();
  const int hw = tid >> 4, hc = tid & 15;
  const bool col_ok = (hc >> 3) < (kyi == 0 ? 1 : 2) && (hc & 7) < nkz;
  const size_t so = (size_t)((hc >> 3) ? d.Ny - kyi : kyi) * d.Kz + kz0 + (hc & 7);
  for (int r = hw; r < nB + nD; r += kSThreads / 16) {
    const bool isg = r >= nB;
    const int i = isg ? r - nB : r;
    c64* dst = sat(sm, (isg ? ((i & 1) ? oGO : oGE) : ((i & 1) ? oUO : oUE)) + (i >> 1), hc);
    if (!col_ok) *dst = cmk(0.0, 0.0);
    else if (isg && bid == 0 && hc == 0) *dst = ldg_c(a.vw_out + i);  // mean flow v + i w
    else cp_async16(dst, (isg ? a.g_out : a.u0_out) + (size_t)i * P + so);
  }
  const int pads[4][2] = {{oUE + G.nBe, round4(G.nBe) - G.nBe},
                          {oUO + G.nBo, round4(G.nBo) - G.nBo},
                          {oGE + G.nDe, round4(G.nDe) - G.nDe},
                          {oGO + G.nDo, round4(G.nDo) - G.nDo}};
  for (int q = 0; q < 4; ++q)
    for (int e = tid; e < pads[q][1] * kSLd; e += kSThreads) sm[(size_t)pads[q][0] * kSLd + e] = 0.0;
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();

  JFB_STAMP(3, 1);
  // unit of work: 8 nodes (and their mirror nodes) x 8 pencils
  const int MTv = G.sub[gA0Ee].mt;
  for (int task = warp; task < 2 * MTv; task += kSWarps) {
    const int jt = task >> 1, col0 = (task & 1) * 16;
    auto prod = [&](int sub, int base, double (&acc)[2][2]) {
      acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = 0.0;
      const SubDesc s = G.sub[sub];
      gemm_sw<2, 8>(frag + s.off + (size_t)jt * s.kt * 32, 0, s.kt, sm, base, col0, lane, acc);
    };
    const int j = jt * 8 + g, jm = N - 1 - j;
    auto cv = [&](const double (&v)[2][2], int nt) { return cmk(v[nt][0], v[nt][1]); };
    auto put = [&](int q, int p, const c64 fe, const c64 fo) {
      const c64 vp = fe + fo, vm = fe - fo;
      c64* X = a.X + (size_t)q * N * P + p;
      X[(size_t)j * P] = vp;
      X[(size_t)jm * P] = vm;
    };
    // even (E) and odd (O) halves of A0 u0, P1 u0, B1 g, then P2 u0, B2 g
    double aE[2][2], aO[2][2], vE[2][2], vO[2][2], wE[2][2], wO[2][2];
    prod(gA0Ee, oUE, aE);
    prod(gP1Oe, oUE, vO);
    prod(gA0Oo, oUO, aO);
    prod(gP1Eo, oUO, vE);
    prod(gB1Ee, oGE, wE);
    prod(gB1Oo, oGO, wO);
    if (j < Jl) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int w = (col0 >> 1) + nt * 4 + t4, p = tc.p[w];
        if (p < 0) continue;
        const double ky = tc.ky[w], kz = tc.kz[w], k2 = ky * ky + kz * kz;
        const c64 c1e = cv(wE, nt), c1o = cv(wO, nt);
        c64 f1e, f1o, f2e, f2o, f3e = c1e, f3o = c1o;
        if (k2 == 0.0) {
          f1e = cmk(c1e.re, 0.0), f1o = cmk(c1o.re, 0.0);
          f2e = cmk(c1e.im, 0.0), f2o = cmk(c1o.im, 0.0);
          f3e = f3o = cmk(0.0, 0.0);
        } else {
          const double inv = 1.0 / k2, y = ky * inv, z = kz * inv;
          f1e = mul_i(y * cv(vE, nt) + z * c1e), f1o = mul_i(y * cv(vO, nt) + z * c1o);
          f2e = mul_i(z * cv(vE, nt) - y * c1e), f2o = mul_i(z * cv(vO, nt) - y * c1o);
        }
        put(0, p, cv(aE, nt), cv(aO, nt));
        put(1, p, f1e, f1o);
        put(2, p, f2e, f2o);
        if (grad) {
          put(6, p, mul_i(ky * cv(aE, nt)), mul_i(ky * cv(aO, nt)));
          put(7, p, mul_i(ky * f1e), mul_i(ky * f1o));
          put(8, p, mul_i(ky * f2e), mul_i(ky * f2o));
        } else {
          put(3, p, f3e, f3o);
        }
      }
    }
    prod(gP2Ee, oUE, vE);
    prod(gP2Oo, oUO, vO);
    prod(gB2Oe, oGE, wO);
    prod(gB2Eo, oGO, wE);
    if (j < Jl) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int w = (col0 >> 1) + nt * 4 + t4, p = tc.p[w];
        if (p < 0) continue;
        const double ky = tc.ky[w], kz = tc.kz[w], k2 = ky * ky + kz * kz;
        // d/dx u1, d/dx u2 (gradient form), or omega_1, omega_2
        auto pair = [&](const c64 av, const c64 b2, const c64 c2, c64& f4, c64& f5) {
          if (k2 == 0.0) {
            f4 = grad ? cmk(c2.re, 0.0) : cmk(-c2.im, 0.0);
            f5 = grad ? cmk(c2.im, 0.0) : cmk(c2.re, 0.0);
            return;
          }
          const double inv = 1.0 / k2, y = ky * inv, z = kz * inv;
          const c64 dx1 = mul_i(y * b2 + z * c2), dx2 = mul_i(z * b2 - y * c2);
          f4 = grad ? dx1 : mul_i(kz * av) - dx2;
          f5 = grad ? dx2 : dx1 - mul_i(ky * av);
        };
        c64 f4e, f4o, f5e, f5o;
        pair(cv(aE, nt), cv(vE, nt), cv(wE, nt), f4e, f5e);
        pair(cv(aO, nt), cv(vO, nt), cv(wO, nt), f4o, f5o);
        put(4, p, f4e, f4o);
        put(5, p, f5e, f5o);
      }
    }
    if (grad) {  // d/dx u0
      prod(gA1Oe, oUE, vO);
      prod(gA1Eo, oUO, vE);
      if (j < Jl) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const int p = tc.p[(col0 >> 1) + nt * 4 + t4];
          if (p >= 0) put(3, p, cv(vE, nt), cv(vO, nt));
        }
      }
    }
  }
  JFB_STAMP(3, 2);
  if (Jh > Jl) {  // middle node of an odd N
    for (int e = tid; e < (grad ? 6 : 5) * kSLd; e += kSThreads) {
      const int col = e % kSLd, op = e / kSLd;
      const int oB = (op <= 1) ? oUE : (op == 2 || op == 5) ? oUO : (op == 3) ? oGE : oGO;
      const int K = (op <= 1) ? G.nBe : (op == 2 || op == 5) ? G.nBo : (op == 3) ? G.nDe : G.nDo;
      const double* row = G.mid + op * G.mid_stride;
      double s = 0.0;
#pragma unroll 4
      for (int k = 0; k < K; ++k)
        s += __ldg(row + k) * sm[(size_t)(oB + k) * kSLd + (col ^ (((oB + k) & 3) << 2))];
      mid[e] = s;
    }
    __syncthreads();
    if (tid < kGW) mid_store(grad, a, mid, tc.p, tc.ky, tc.kz, tid, N, Jl, P);
  }
  JFB_STAMP(3, 3);
}

}  // namespace jfb
