// Standalone tensor-product transforms: TensorProductSpace.backward / forward /
// scalar_product (src/jaxfun/galerkin/tensorproductspace.py:253-551) for a
// Chebyshev axis (orthogonal, Dirichlet or biharmonic basis) times one or two
// Fourier axes, on full complex spectra in the reference layout, with the 3/2
// padding of the Fourier axes (Fourier.py:128-184: zero padding in the middle,
// unnormalised inverse, forward scaled 1/M and truncated to the modes
// wavenumbers() keeps, Nyquist included).
//
//   x axis:       dense real operator per axis-0 line (x_apply_kernel, FP64
//                 tensor cores)
//   middle axis:  the step's y kernels (warp-shuffle FFT, or Stockham)
//   last axis:    fft_rows_warp_kernel / fft_rows_kernel (contiguous lines)
//
// Included at the end of jfb_kmm.cu (one translation unit with the step).
#pragma once

#include "jfb_kmm_split.cuh"
#include "jfb_kmm_warpk.cuh"

namespace jfb {

// Per-mode Fourier weight of the separable maps: scale * prod over the
// periodic axes of (i m df)^k, m the FFT-ordered wavenumber, with the Nyquist
// mode zeroed for odd k (Fourier.py:210-223).
struct FourierWeight {
  int n1, n2, k1, k2;
  double df1, df2, scale;
};

__device__ __forceinline__ c64 ipow_times(c64 w, int idx, int n, int k, double df) {
  if (k == 0) return w;
  if ((k & 1) && 2 * idx == n) return cmk(0.0, 0.0);
  const int m = (idx < (n + 1) / 2) ? idx : idx - n;
  double a = 1.0;
  for (int t = 0; t < k; ++t) a *= (double)m * df;
  w = a * w;
  for (int t = 0; t < (k & 3); ++t) w = mul_i(w);  // i^k
  return w;
}

// out[i][m] = w(m) sum_k A[i][k] in[k][m], A real (rows x cols) in 8x4 mma
// fragment tiles, w a per-mode Fourier weight (m = i1 n2 + i2 over the
// periodic axes).  A block stages 16 columns of the field as B-operand rows
// (swizzled as in gemm_sw) and its warps take the row tiles of A: the field is
// read once, where one thread per output read every column once per row from
// L2 (23 -> 7 us for 65 x 63 on 4096 columns).  Bound by latency: load, product
// and store of a block follow one another.
constexpr int kXThreads = 256;  // at most: a warp per row tile
__global__ void __launch_bounds__(kXThreads)
    x_apply_kernel(const double* __restrict__ frag, int rows, int cols, const c64* __restrict__ in,
                   c64* __restrict__ out, const __grid_constant__ FourierWeight fw) {
  extern __shared__ __align__(128) double sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t M = (int64_t)fw.n1 * fw.n2, m0 = (int64_t)blockIdx.x * kGW;
  const int c = tid & 15, nc = (int)min((int64_t)kGW, M - m0);
  const int KT = (cols + 3) / 4;
  const bool wide = (reinterpret_cast<uintptr_t>(in) & 15) == 0;
  if (c < nc)
    for (int k = tid >> 4; k < cols; k += blockDim.x / 16) {
      if (wide) {
        cp_async16(sat(sm, k, c), in + (size_t)k * M + m0 + c);
      } else {  // a caller's field on an 8-byte boundary
        const double* v = &in[(size_t)k * M + m0 + c].re;
        cp_async8(sat(sm, k, c), v);
        cp_async8(&sat(sm, k, c)->im, v + 1);
      }
    }
  else
    for (int k = tid >> 4; k < cols; k += blockDim.x / 16) *sat(sm, k, c) = cmk(0.0, 0.0);
  for (int e = tid; e < (4 * KT - cols) * kSLd; e += blockDim.x) sm[(size_t)cols * kSLd + e] = 0.0;
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  const int g = lane >> 2, t4 = lane & 3;
  c64 w[4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int64_t m = m0 + nt * 4 + t4;
    w[nt] = cmk(fw.scale, 0.0);
    if (m < M && fw.k1 + fw.k2) {
      w[nt] = ipow_times(w[nt], (int)m / fw.n2, fw.n1, fw.k1, fw.df1);
      w[nt] = ipow_times(w[nt], (int)m % fw.n2, fw.n2, fw.k2, fw.df2);
    }
  }
  for (int mt = warp + blockIdx.y * (blockDim.x / 32); mt * 8 < rows;
       mt += gridDim.y * (blockDim.x / 32)) {
    double acc[4][2];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
    gemm_sw<4, 8>(frag + (size_t)mt * KT * 32, 0, KT, sm, 0, 0, lane, acc);
    const int i = mt * 8 + g;
    if (i >= rows) continue;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int64_t m = m0 + nt * 4 + t4;
      if (m < M) out[(size_t)i * M + m] = w[nt] * cmk(acc[nt][0], acc[nt][1]);
    }
  }
}

// A real (rows x cols) matrix as 8x4 mma fragment tiles (zero padded).
static std::vector<double> fragment_tiles(const std::vector<double>& A, int rows, int cols) {
  const int MT = (rows + 7) / 8, KT = (cols + 3) / 4;
  std::vector<double> f((size_t)MT * KT * 32, 0.0);
  for (int i = 0; i < rows; ++i)
    for (int k = 0; k < cols; ++k)
      f[((size_t)(i >> 3) * KT + (k >> 2)) * 32 + (i & 7) * 4 + (k & 3)] = A[(size_t)i * cols + k];
  return f;
}

// Complex FFT along contiguous lines: `lines` rows of length nin -> nout.
// Inverse (sign +1, transform length nout): pad nin -> nout in the middle,
// unnormalised.  Forward (sign -1, transform length nin): scaled 1/nin,
// truncated to nout modes in FFT order (k < nout/2 and the last nout/2 of
// the spectrum, the -nout/2 mode included).  2^lr lines per block.
constexpr int kTpsLogRows = 3;
__global__ void __launch_bounds__(256) fft_rows_kernel(FFTPlan plan, const c64* __restrict__ tw,
                                                       int sign, const c64* in, c64* out,
                                                       int64_t lines, int nin, int nout, int lr) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = plan.n, R = 1 << lr;
  c64* A = reinterpret_cast<c64*>(smem_raw);
  c64* B = A + (size_t)n * R;
  const int64_t l0 = blockIdx.x * (int64_t)R;
  for (int idx = threadIdx.x; idx < n * R; idx += blockDim.x) {
    const int c = idx & (R - 1), k = idx >> lr;
    const int64_t line = l0 + c;
    c64 v = cmk(0.0, 0.0);
    if (line < lines) {
      if (sign > 0) {
        const int h = nin / 2;
        if (k < h) v = in[line * nin + k];
        else if (k >= n - (nin - h)) v = in[line * nin + (k - n + nin)];
      } else {
        v = in[line * nin + k];
      }
    }
    A[k * R + c] = v;
  }
  __syncthreads();
  c64* res = fft_columns<double>(A, B, plan, R, R, tw, sign);
  const double scale = sign > 0 ? 1.0 : 1.0 / n;
  const int h = nout / 2;
  for (int idx = threadIdx.x; idx < nout * R; idx += blockDim.x) {
    const int c = idx & (R - 1), k = idx >> lr;
    const int64_t line = l0 + c;
    if (line >= lines) continue;
    int src = k;
    if (sign < 0 && k >= h) src = k - nout + n;
    out[line * nout + k] = scale * res[src * R + c];
  }
}

// The same with warp-shuffle transforms for lengths 32 P: a warp per line,
// natural order on the global side (coalesced), the transform's scrambled
// order through the warp's shared-memory row.  In place allowed when
// nin == nout (a warp reads its whole line first).  16 -> 8 us for 6240 lines
// of 64 -> 96 points against the shared-memory form, whose radix passes wait
// on block barriers.
template <int P>
__global__ void __launch_bounds__(256) fft_rows_warp_kernel(const c64* __restrict__ tw, int sign,
                                                            const c64* in, c64* out, int64_t lines,
                                                            int nin, int nout) {
  constexpr int n = 32 * P;
  __shared__ c64 rowbuf[8][n];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t line = blockIdx.x * (int64_t)8 + warp;
  if (line >= lines) return;
  c64* row = rowbuf[warp];
  const int br = bitrev5(lane);
  WarpTw<P, double> w;
  load_warp_tw<P, double>(w, tw, lane);
  c64 v[P];
  if (sign > 0) {
    const int h = nin / 2;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int k = 32 * r + lane;
      v[r] = k < h ? in[line * nin + k]
                   : k >= n - (nin - h) ? in[line * nin + (k - n + nin)] : cmk(0.0, 0.0);
    }
    warp_fft_inverse<P, double>(v, w, lane);
#pragma unroll
    for (int r = 0; r < P; ++r) row[r + P * br] = v[r];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < P; ++r) out[line * n + 32 * r + lane] = row[32 * r + lane];
  } else {
#pragma unroll
    for (int r = 0; r < P; ++r) row[32 * r + lane] = in[line * n + 32 * r + lane];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < P; ++r) v[r] = row[r + P * br];
    warp_fft_forward<P, double>(v, w, lane);
    const int h = nout / 2;
    const double scale = 1.0 / n;
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int k = 32 * r + lane;
      if (k < h) out[line * nout + k] = scale * v[r];
      else if (k >= n - (nout - h)) out[line * nout + (k - n + nout)] = scale * v[r];
    }
  }
}

// ---------------------------------------------------------------------------
// 2-D Helmholtz solve (la/solvers.py:22-61 with the per-wavenumber solve of
// tpmatrix.py:1550-1677), one CTA per Fourier mode, then the y transform of
// the rows.  The backward transform of f and its scalar products cancel up to
// the norms: the y transforms are inverse to each other, and the Gauss
// quadrature is exact for products of degree 2 N - 2, so
//   rhs_r = scale sum_n S_D[r, n] (P_n, P_n) f_n
// is two terms per row.  A CTA forms its mode's right-hand side, solves and
// evaluates the solution at the nodes; the launch pair replaces one cluster of
// eight CTAs that held the whole problem and worked through four transforms
// between cluster barriers (64 x 64: 38 us, now 5.4 + 2.1).  Bound by latency:
// the column of f, the recurrence, two products of which a thread takes a
// quarter of a row (9.4 us with a thread per row and no loads ahead).
// ---------------------------------------------------------------------------
constexpr int kHelmMaxDiag = 256;
constexpr int kHelmCTAs = 8;  // parts of the size range's formula (jfb_helmholtz2d_solve)
constexpr int kHelmRows = 128, kHelmSplit = 4;  // thread = (row, every 4th column)
constexpr int kHelmThreads = kHelmRows * kHelmSplit;
constexpr int kHelmCols = 16;  // matrix entries a thread loads ahead
struct Helm2DArgs {
  const double* ns;    // (P_n, P_n) / df
  const double* BDT;   // Dirichlet backward, transposed (nb x N)
  const double *L, *U;  // (n1, nL, nb), (n1, nU, nb)
  const double* Uinv;   // optional (n1, nb, nb): U^-1 per mode, entry (r, c) at c nb + r
  int nL, nU, umain;
  int l2, l4;  // indices of the L offsets -2 / -4 (-1: absent) when those are all of L
  int loff[kHelmMaxDiag], uoff[kHelmMaxDiag];
  int staged;  // general form: the mode's factors in shared memory, rows of nb | 1
  int N, nb, M;
  double scale;  // Fourier scalar-product weight / fourier_mass
  const c64* f;
  c64* u;
};

__global__ void __launch_bounds__(kHelmThreads)
    helmholtz2d_kernel(const __grid_constant__ Helm2DArgs h) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = h.N, M = h.M, nb = h.nb, k = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31;
  c64* F = reinterpret_cast<c64*>(smem_raw);  // N: the mode's column of f
  c64* x = F + N;                             // nb: right-hand side, then y
  c64* z = x + nb;                            // nb: solution
  c64* part = z + nb;                         // kHelmThreads: partial sums
  // nb each: L[r, r-2], L[r, r-4], or U[r, r] and its reciprocal
  double* l2s = reinterpret_cast<double*>(part + kHelmThreads);
  double* l4s = l2s + nb;
  const double* Lk = h.L + (size_t)k * h.nL * nb;
  const double* Uk = h.U + (size_t)k * h.nU * nb;
  const bool fast = h.Uinv && h.l2 + h.l4 > -2;
  const int row = tid & (kHelmRows - 1), grp = tid / kHelmRows;
  for (int n = tid; n < N; n += kHelmThreads) F[n] = h.f[(size_t)n * M + k];
  for (int r = tid; r < nb; r += kHelmThreads) {
    if (fast) {
      l2s[r] = (h.l2 >= 0 && r >= 2) ? __ldg(Lk + (size_t)h.l2 * nb + r - 2) : 0.0;
      l4s[r] = (h.l4 >= 0 && r >= 4) ? __ldg(Lk + (size_t)h.l4 * nb + r - 4) : 0.0;
    } else {
      l2s[r] = __ldg(Uk + (size_t)h.umain * nb + r);
      l4s[r] = 1.0 / l2s[r];
    }
  }
  __shared__ int offs[2 * kHelmMaxDiag];
  double *Ls = l4s + nb, *Us = Ls + (size_t)h.nL * (nb | 1);
  if (!fast)
    for (int d = tid; d < h.nL + h.nU; d += kHelmThreads)
      offs[d] = d < h.nL ? h.loff[d] : h.uoff[d - h.nL];
  if (h.staged) {
    for (int e = tid; e < (h.nL + h.nU) * nb; e += kHelmThreads) {
      const int d = e / nb, c = e - d * nb;
      cp_async8(Ls + (size_t)d * (nb | 1) + c, d < h.nL ? Lk + e : Uk + e - h.nL * nb);
    }
    cp_async_commit();
    cp_async_wait_all();
  }
  // the matrix entries of the two products do not depend on f: on their way
  // while the right-hand side and the recurrence run
  const double* Ui = h.Uinv + (size_t)k * nb * nb + row;
  double u[kHelmCols], b[kHelmCols];
#pragma unroll
  for (int q = 0; q < kHelmCols; ++q) {
    const int c = grp + kHelmSplit * q;
    u[q] = fast && c < nb && row <= c ? __ldg(Ui + (size_t)c * nb) : 0.0;
    b[q] = c < nb && row < N ? __ldg(h.BDT + (size_t)c * N + row) : 0.0;
  }
  __syncthreads();
  for (int r = tid; r < nb; r += kHelmThreads)
    x[r] = h.scale * (h.ns[r] * F[r] - h.ns[r + 2] * F[r + 2]);
  __syncthreads();
  // this thread's columns of row i of a matrix (entry (i, c) at m[c * ld]),
  // c >= first, against v; the first kHelmCols of them are in registers
  auto dot = [&](const double (&reg)[kHelmCols], const double* m, int ld, int first, const c64* v) {
    c64 s0 = cmk(0.0, 0.0), s1 = s0;
#pragma unroll
    for (int q = 0; q < kHelmCols; q += 2) {
      const int c = grp + kHelmSplit * q;
      if (c < nb) s0 = s0 + reg[q] * v[c];
      if (c + kHelmSplit < nb) s1 = s1 + reg[q + 1] * v[c + kHelmSplit];
    }
#pragma unroll 8
    for (int c = grp + kHelmSplit * kHelmCols; c < nb; c += kHelmSplit)
      if (c >= first) s0 = s0 + __ldg(m + (size_t)c * ld) * v[c];
    return s0 + s1;
  };
  auto total = [&](int i) {
    return (part[i] + part[i + kHelmRows]) + (part[i + 2 * kHelmRows] + part[i + 3 * kHelmRows]);
  };
  if (fast) {
    // two independent recurrences (one per parity class), then x = U^-1 y as a
    // product with the mode's explicit inverse
    if (tid < 2) {
      c64 ym2 = cmk(0.0, 0.0), ym4 = cmk(0.0, 0.0);  // y_{r-2}, y_{r-4}
#pragma unroll 4
      for (int r = tid; r < nb; r += 2) {
        const c64 v = x[r] - l4s[r] * ym4 - l2s[r] * ym2;
        x[r] = v;
        ym4 = ym2;
        ym2 = v;
      }
    }
    __syncthreads();
    part[tid] = row < nb ? dot(u, Ui, nb, row, x) : cmk(0.0, 0.0);
    __syncthreads();
    if (tid < nb) z[tid] = total(tid);
  } else if (tid < 32) {
    // column-oriented substitution: once x_c is final each lane applies its
    // diagonals' entries of column c to their rows (distinct per diagonal), from
    // shared memory (a lane's diagonals are lines apart in memory, and argument
    // words indexed by lane are read one by one).
    // Called without explicit inverses, 62 / 98 / 148 unknowns on 64 / 16 / 16
    // modes: 62 / 112 / 191 -> 36 / 58 / 91 us.
    const int ld = h.staged ? nb | 1 : nb;
    const double *Lf = h.staged ? Ls : Lk, *Uf = h.staged ? Us : Uk;
    for (int c = 0; c < nb; ++c) {
      const c64 y = x[c];
      for (int d = lane; d < h.nL; d += 32) {
        const int r = c - offs[d];
        if (r < nb) x[r] = x[r] - Lf[(size_t)d * ld + c] * y;
      }
      __syncwarp();
    }
    for (int c = nb - 1; c >= 0; --c) {
      const double dg = l2s[c], rd = l4s[c];
      const c64 y = x[c];
      c64 xc = cmk(quotient(y.re, dg, rd), quotient(y.im, dg, rd));
      if (!finite_c(xc)) xc = cmk(y.re / dg, y.im / dg);
      if (lane == 0) z[c] = xc;
      for (int d = lane; d < h.nU; d += 32) {
        const int sft = offs[h.nL + d], r = c - sft;
        if (sft > 0 && r >= 0) x[r] = x[r] - Uf[(size_t)d * ld + c] * xc;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  for (int j0 = 0; j0 < N; j0 += kHelmRows) {
    const int j = j0 + row;
    if (j0 > 0) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kHelmCols; ++q) {
        const int c = grp + kHelmSplit * q;
        b[q] = c < nb && j < N ? __ldg(h.BDT + (size_t)c * N + j) : 0.0;
      }
    }
    part[tid] = j < N ? dot(b, h.BDT + j, N, 0, z) : cmk(0.0, 0.0);
    __syncthreads();
    if (grp == 0 && j < N) h.u[(size_t)j * M + k] = total(row);
  }
}

}  // namespace jfb

struct jfb_tps {
  jfb_tps_config cfg;
  jfb::XBasis xb;  // 1-D wall-normal basis data (long double)
  std::map<int64_t, std::pair<double*, std::pair<int, int>>> xmaps;  // (map, k) -> device matrix
  int nb = 0, N = 0;
  int n1 = 1, n2 = 1, m1 = 1, m2 = 1;  // Fourier modes and padded counts
  double *B = nullptr, *F = nullptr, *Sq = nullptr;  // mma fragment tiles
  double *BT = nullptr, *ns = nullptr;               // B transposed (nb x N), norms
  std::vector<double> G0, G2;
  c64 *tw1n = nullptr, *tw1m = nullptr, *tw2n = nullptr, *tw2m = nullptr;
  FFTPlan f1n, f1m, f2n, f2m;
  c64 *w0 = nullptr, *w1 = nullptr;  // work buffers
  std::vector<void*> allocs;
};

extern "C" int jfb_tps_destroy(jfb_tps* t) {
  if (!t) return JFB_OK;
  for (auto& kv : t->xmaps) cudaFree(kv.second.first);
  for (void* p : t->allocs) cudaFree(p);
  delete t;
  return JFB_OK;
}

extern "C" int jfb_tps_create(const jfb_tps_config* cfg, jfb_tps** out) {
  JFB_REQUIRE(cfg && out, "null pointer");
  *out = nullptr;
  JFB_REQUIRE(cfg->ndim == 2 || cfg->ndim == 3, "ndim must be 2 or 3");
  JFB_REQUIRE(cfg->basis >= 0 && cfg->basis <= 2, "unknown basis");
  JFB_REQUIRE(cfg->family == JFB_FAMILY_CHEBYSHEV || cfg->family == JFB_FAMILY_LEGENDRE,
              "family must be JFB_FAMILY_CHEBYSHEV or JFB_FAMILY_LEGENDRE");
  JFB_REQUIRE(cfg->n[0] >= 8 && cfg->n[0] <= 513, "n[0] out of range [8, 513]");
  for (int a = 1; a < cfg->ndim; ++a)
    JFB_REQUIRE(cfg->n[a] >= 2 && cfg->n[a] % 2 == 0, "Fourier sizes must be even");
  JFB_REQUIRE(cfg->x_hi > cfg->x_lo, "bad domain");
  jfb_tps* t = new jfb_tps();
  t->cfg = *cfg;
  auto fail = [&](int code) {
    jfb_tps_destroy(t);
    return code;
  };
  jfb_kmm_config kc;
  std::memset(&kc, 0, sizeof(kc));
  kc.nx = cfg->n[0];
  kc.ny = 4;
  kc.nz = 4;
  kc.x_lo = cfg->x_lo;
  kc.x_hi = cfg->x_hi;
  kc.ly = kc.lz = 2.0 * M_PI;
  build_x_basis(cfg->family, cfg->basis, cfg->n[0], cfg->x_lo, cfg->x_hi, t->xb);
  TpsX x;
  if (cfg->family == JFB_FAMILY_CHEBYSHEV) {
    HostOperators op;
    build_host_operators(kc, op);
    build_tps_x_operators(op, cfg->basis, x);
  } else {
    // Legendre: backward V S^T, forward M^-1 S Q, scalar product S Q and the
    // Galerkin matrices, all from the Gauss-Legendre Vandermonde matrix
    int r, c;
    x.N = t->xb.N;
    x.nb = t->xb.nb;
    x.B = x_map_matrix(t->xb, kXBackward, 0, &r, &c);
    x.F = x_map_matrix(t->xb, kXForward, 0, &r, &c);
    x.Sq = x_map_matrix(t->xb, kXScalarProd, 0, &r, &c);
    x.G0 = x_map_matrix(t->xb, kXGalerkin, 0, &r, &c);
    x.G2 = x_map_matrix(t->xb, kXGalerkin, 2, &r, &c);
  }
  t->N = x.N;
  t->nb = x.nb;
  t->G0 = x.G0;
  t->G2 = x.G2;
  t->n1 = cfg->n[1];
  t->n2 = cfg->ndim == 3 ? cfg->n[2] : 1;
  t->m1 = std::max(t->n1, (int)(cfg->pad[0] * t->n1));
  t->m2 = cfg->ndim == 3 ? std::max(t->n2, (int)(cfg->pad[1] * t->n2)) : 1;
  if (!make_fft_plan(t->n1, t->f1n) || !make_fft_plan(t->m1, t->f1m) ||
      (cfg->ndim == 3 && (!make_fft_plan(t->n2, t->f2n) || !make_fft_plan(t->m2, t->f2m)))) {
    set_error("Fourier sizes (and padded sizes) must be of the form 2^a 3^b");
    return fail(JFB_ERR_ARG);
  }
  auto up = [&](auto** dst, const auto& v) -> int {
    using E = typename std::decay_t<decltype(v)>::value_type;
    cudaError_t e = cudaMalloc((void**)dst, std::max<size_t>(1, v.size()) * sizeof(E));
    if (e != cudaSuccess) {
      set_error(std::string("cudaMalloc: ") + cudaGetErrorString(e));
      return JFB_ERR_CUDA;
    }
    t->allocs.push_back(*dst);
    e = cudaMemcpy(*dst, v.data(), v.size() * sizeof(E), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      set_error(std::string("cudaMemcpy: ") + cudaGetErrorString(e));
      return JFB_ERR_CUDA;
    }
    return JFB_OK;
  };
  int st;
  if ((st = up(&t->B, fragment_tiles(x.B, t->N, t->nb))) ||
      (st = up(&t->F, fragment_tiles(x.F, t->nb, t->N))) ||
      (st = up(&t->Sq, fragment_tiles(x.Sq, t->nb, t->N))))
    return fail(st);
  {
    std::vector<double> bt((size_t)t->nb * t->N), ns(t->N);
    for (int j = 0; j < t->N; ++j)
      for (int r = 0; r < t->nb; ++r) bt[(size_t)r * t->N + j] = x.B[(size_t)j * t->nb + r];
    for (int n = 0; n < t->N; ++n) ns[n] = (double)t->xb.ns[n];
    if ((st = up(&t->BT, bt)) || (st = up(&t->ns, ns))) return fail(st);
  }
  if ((st = up(&t->tw1n, twiddles(t->n1))) || (st = up(&t->tw1m, twiddles(t->m1))))
    return fail(st);
  if (cfg->ndim == 3 &&
      ((st = up(&t->tw2n, twiddles(t->n2))) || (st = up(&t->tw2m, twiddles(t->m2)))))
    return fail(st);
  const size_t big = (size_t)std::max(t->N, t->nb) * t->m1 * t->m2;
  for (c64** w : {&t->w0, &t->w1}) {
    cudaError_t e = cudaMalloc((void**)w, big * sizeof(c64));
    if (e != cudaSuccess) {
      set_error(std::string("cudaMalloc: ") + cudaGetErrorString(e));
      return fail(JFB_ERR_CUDA);
    }
    t->allocs.push_back(*w);
  }
#define JFB_YW(P)                                                       \
  for (const void* fn : {(const void*)y_backward_warp_kernel<P, double>, \
                         (const void*)y_forward_warp_kernel<P, double, true>}) \
    if (allow_smem(fn) != cudaSuccess) {                                \
      set_error("cannot configure the transform kernels");              \
      return fail(JFB_ERR_CUDA);                                        \
    }
  JFB_YW(2) JFB_YW(3) JFB_YW(4) JFB_YW(6)
#undef JFB_YW
  if (allow_smem((const void*)y_backward_kernel<double>) != cudaSuccess ||
      allow_smem((const void*)y_forward_kernel<double>) != cudaSuccess ||
      allow_smem((const void*)fft_rows_kernel) != cudaSuccess ||
      allow_smem((const void*)x_apply_kernel) != cudaSuccess ||
      cudaStreamSynchronize(nullptr) != cudaSuccess) {  // the uploads have arrived
    set_error("cannot configure the transform kernels");
    return fail(JFB_ERR_CUDA);
  }
  *out = t;
  return JFB_OK;
}

namespace jfb {

// Device copy of one separable x-axis map in fragment tiles (built and
// uploaded on first use).
static int tps_xmap(jfb_tps* t, int map, int k, const double** A, int* rows, int* cols) {
  const int64_t key = (int64_t)map * 64 + k;
  auto it = t->xmaps.find(key);
  if (it == t->xmaps.end()) {
    int r = 0, c = 0;
    const std::vector<double> A0 = x_map_matrix(t->xb, map, k, &r, &c);
    const std::vector<double> h = fragment_tiles(A0, r, c);
    double* d = nullptr;
    JFB_CHECK_CUDA(cudaMalloc((void**)&d, h.size() * sizeof(double)));
    cudaError_t e = cudaMemcpy(d, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice);
    // (a copy from pageable memory may return before it has arrived)
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
    if (e != cudaSuccess) {
      cudaFree(d);
      JFB_CHECK_CUDA(e);
    }
    it = t->xmaps.emplace(key, std::make_pair(d, std::make_pair(r, c))).first;
  }
  *A = it->second.first;
  *rows = it->second.second.first;
  *cols = it->second.second.second;
  return JFB_OK;
}

static double fourier_df(const jfb_tps* t, int a) {
  const double L = t->cfg.l[a];
  return std::fabs(L - 2.0 * M_PI) < 1e-12 ? 1.0 : 2.0 * M_PI / L;
}

static int tps_x(const double* A, int rows, int cols, const c64* in, c64* out,
                 const FourierWeight& fw, cudaStream_t s) {
  const int64_t M = (int64_t)fw.n1 * fw.n2;
  // few columns (2-D spaces): the row tiles over several blocks
  const unsigned gx = (unsigned)((M + kGW - 1) / kGW);
  const unsigned gy = gx >= 148 ? 1 : std::min<unsigned>(148 / gx + 1, (rows + 63) / 64);
  // few rows: fewer warps a block, so that more blocks load at once
  const int threads = std::min(kXThreads, 32 * std::max(2, (rows + 7) / 8));
  x_apply_kernel<<<dim3(gx, gy), threads, (size_t)(cols + 3) / 4 * 4 * kSLd * sizeof(double), s>>>(
      A, rows, cols, in, out, fw);
  JFB_CHECK_LAUNCH();
  return JFB_OK;
}
static FourierWeight no_weight(const jfb_tps* t, double scale) {
  return FourierWeight{t->n1, t->n2, 0, 0, 1.0, 1.0, scale};
}

// out = w * (map_k along x) in, w the Fourier weights of orders k1, k2.
static int tps_xw(jfb_tps* t, int map, int kx, int k1, int k2, double scale, const c64* in,
                  c64* out, cudaStream_t s) {
  const double* A;
  int rows, cols;
  int st = tps_xmap(t, map, kx, &A, &rows, &cols);
  if (st) return st;
  FourierWeight fw;
  fw.n1 = t->n1;
  fw.n2 = t->n2;
  fw.k1 = k1;
  fw.k2 = t->cfg.ndim == 3 ? k2 : 0;
  fw.df1 = fourier_df(t, 0);
  fw.df2 = t->cfg.ndim == 3 ? fourier_df(t, 1) : 1.0;
  fw.scale = scale;
  return tps_x(A, rows, cols, in, out, fw, s);
}

static int check_orders(const jfb_tps* t, const int32_t* k) {
  JFB_REQUIRE(k, "null derivative orders");
  for (int a = 0; a < t->cfg.ndim; ++a)
    JFB_REQUIRE(k[a] >= 0 && k[a] < 32, "derivative orders must be in [0, 32)");
  return JFB_OK;
}

// contiguous lines: padded inverse (sign +1, n -> m) or truncated forward (m -> n)
static int tps_lines(const FFTPlan& plan, const c64* tw, int sign, int64_t lines, int n, int m,
                     const c64* in, c64* out, cudaStream_t s) {
  const int nin = sign > 0 ? n : m, nout = sign > 0 ? m : n;
  switch (warp_radix(m)) {
#define JFB_FR(P) \
  case P:                                                                                        \
    fft_rows_warp_kernel<P><<<(unsigned)((lines + 7) / 8), 256, 0, s>>>(tw, sign, in, out, lines, nin, nout); \
    break;
    JFB_FR(2) JFB_FR(3) JFB_FR(4) JFB_FR(6)
#undef JFB_FR
    default: {
      // 8 lines per block, fewer where that would leave SMs idle or not fit
      int lr = kTpsLogRows;
      while (lr > 0 && ((lines >> lr) < 148 || ((size_t)2 * m << lr) * sizeof(c64) > 200 * 1024)) --lr;
      const size_t sm = ((size_t)2 * m << lr) * sizeof(c64);
      JFB_REQUIRE(sm <= 200 * 1024, "Fourier axis too long");
      const unsigned blocks = (unsigned)((lines + (1 << lr) - 1) >> lr);
      fft_rows_kernel<<<blocks, 256, sm, s>>>(plan, tw, sign, in, out, lines, nin, nout, lr);
    }
  }
  JFB_CHECK_LAUNCH();
  return JFB_OK;
}

// middle axis of an array (rows, len, inner): the y kernels with Kz = inner
static int tps_y(jfb_tps* t, int sign, int rows, int inner, const c64* in, c64* out,
                 bool padded, cudaStream_t s) {
  const FFTPlan& plan = padded ? t->f1m : t->f1n;
  const c64* tw = padded ? t->tw1m : t->tw1n;
  const int m = padded ? t->m1 : t->n1;
  if (inner == 1) return tps_lines(plan, tw, sign, rows, t->n1, m, in, out, s);
  Dims d;
  std::memset(&d, 0, sizeof(d));
  d.Nx = rows;
  d.Ny = t->n1;
  d.Kz = inner;
  d.P = t->n1 * inner;
  d.My = m;
  if (warp_radix(m) && inner >= 8) {
    const int kc = std::min(16, inner);
    const dim3 g(rows, 1, ceil_div(inner, kc));
    const size_t sm = (size_t)(d.Ny + d.My) * (kc + 1) * sizeof(c64);
    if (sm <= 200 * 1024) {
      switch (warp_radix(m)) {
#define JFB_YW(P)                                                                            \
  case P:                                                                                    \
    if (sign > 0) y_backward_warp_kernel<P, double><<<g, 256, sm, s>>>(d, kc, tw, in, out);   \
    else y_forward_warp_kernel<P, double, true><<<g, 256, sm, s>>>(d, kc, tw, in, out, nullptr); \
    break;
        JFB_YW(2) JFB_YW(3) JFB_YW(4) JFB_YW(6)
#undef JFB_YW
      }
      JFB_CHECK_LAUNCH();
      return JFB_OK;
    }
  }
  int KC = inner;
  while ((size_t)2 * d.My * KC * sizeof(c64) > 96 * 1024 && KC % 2 == 0) KC /= 2;
  JFB_REQUIRE((size_t)2 * d.My * KC * sizeof(c64) <= 200 * 1024, "Fourier axis too long");
  dim3 g(rows, 1, inner / KC);
  const size_t sm = (size_t)2 * d.My * KC * sizeof(c64);
  if (sign > 0) y_backward_kernel<double><<<g, 256, sm, s>>>(d, plan, KC, tw, in, out);
  else y_forward_kernel<double><<<g, 256, sm, s>>>(d, plan, KC, tw, in, out, nullptr, 1);
  JFB_CHECK_LAUNCH();
  return JFB_OK;
}

static int tps_z(jfb_tps* t, int sign, int64_t lines, const c64* in, c64* out, bool padded,
                 cudaStream_t s) {
  JFB_REQUIRE(((size_t)2 * (padded ? t->m2 : t->n2) << kTpsLogRows) * sizeof(c64) <= 200 * 1024,
              "Fourier axis too long");
  return tps_lines(padded ? t->f2m : t->f2n, padded ? t->tw2m : t->tw2n, sign, lines, t->n2,
                   padded ? t->m2 : t->n2, in, out, s);
}

}  // namespace jfb

extern "C" int jfb_tps_backward(jfb_tps* t, const void* coeffs, void* phys, int padded,
                                void* stream) {
  JFB_REQUIRE(t && coeffs && phys, "null pointer");
  cudaStream_t s = (cudaStream_t)stream;
  const bool pad = padded != 0;
  const int m1 = pad ? t->m1 : t->n1;
  int st;
  if (t->cfg.ndim == 2) {
    // x: (nb, n1) -> (N, n1); y: -> (N, m1)
    if ((st = tps_x(t->B, t->N, t->nb, (const c64*)coeffs, t->w0, no_weight(t, 1.0), s))) return st;
    return tps_y(t, +1, t->N, 1, t->w0, (c64*)phys, pad, s);
  }
  if ((st = tps_x(t->B, t->N, t->nb, (const c64*)coeffs, t->w0, no_weight(t, 1.0), s))) return st;
  if ((st = tps_y(t, +1, t->N, t->n2, t->w0, t->w1, pad, s))) return st;
  return tps_z(t, +1, (int64_t)t->N * m1, t->w1, (c64*)phys, pad, s);
}

extern "C" int jfb_tps_forward(jfb_tps* t, const void* phys, void* coeffs, int padded, int kind,
                               void* stream) {
  JFB_REQUIRE(t && phys && coeffs, "null pointer");
  JFB_REQUIRE(kind == 0 || kind == 1, "kind must be 0 (forward) or 1 (scalar product)");
  cudaStream_t s = (cudaStream_t)stream;
  const bool pad = padded != 0;
  const int m1 = pad ? t->m1 : t->n1;
  const double* X = kind ? t->Sq : t->F;
  // scalar products carry the Fourier weight 2 pi / df per periodic axis
  // (Fourier.py:152-167); the forward transform does not
  double w = 1.0;
  if (kind == 1)
    for (int a = 0; a + 1 < t->cfg.ndim; ++a) w *= 2.0 * M_PI / fourier_df(t, a);
  int st;
  if (t->cfg.ndim == 2) {
    if ((st = tps_y(t, -1, t->N, 1, (const c64*)phys, t->w0, pad, s))) return st;
    return tps_x(X, t->nb, t->N, t->w0, (c64*)coeffs, no_weight(t, w), s);
  }
  if ((st = tps_z(t, -1, (int64_t)t->N * m1, (const c64*)phys, t->w0, pad, s))) return st;
  if ((st = tps_y(t, -1, t->N, t->n2, t->w0, t->w1, pad, s))) return st;
  return tps_x(X, t->nb, t->N, t->w1, (c64*)coeffs, no_weight(t, w), s);
}

extern "C" int jfb_tps_backward_primitive(jfb_tps* t, const void* coeffs, void* phys,
                                          const int32_t* k, int padded, void* stream) {
  JFB_REQUIRE(t && coeffs && phys, "null pointer");
  int st = check_orders(t, k);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const bool pad = padded != 0;
  const int m1 = pad ? t->m1 : t->n1;
  const int k2 = t->cfg.ndim == 3 ? k[2] : 0;
  if ((st = tps_xw(t, kXBackward, k[0], k[1], k2, 1.0, (const c64*)coeffs, t->w0, s))) return st;
  if (t->cfg.ndim == 2) return tps_y(t, +1, t->N, 1, t->w0, (c64*)phys, pad, s);
  if ((st = tps_y(t, +1, t->N, t->n2, t->w0, t->w1, pad, s))) return st;
  return tps_z(t, +1, (int64_t)t->N * m1, t->w1, (c64*)phys, pad, s);
}

extern "C" int jfb_tps_to_orthogonal(jfb_tps* t, const void* coeffs, void* orth, void* stream) {
  JFB_REQUIRE(t && coeffs && orth, "null pointer");
  return tps_xw(t, kXToOrth, 0, 0, 0, 1.0, (const c64*)coeffs, (c64*)orth,
                (cudaStream_t)stream);
}

extern "C" int jfb_tps_differentiate_orthogonal(jfb_tps* t, const void* orth, void* out,
                                                const int32_t* k, void* stream) {
  JFB_REQUIRE(t && orth && out, "null pointer");
  int st = check_orders(t, k);
  if (st) return st;
  return tps_xw(t, kXDiffOrth, k[0], k[1], t->cfg.ndim == 3 ? k[2] : 0, 1.0, (const c64*)orth,
                (c64*)out, (cudaStream_t)stream);
}

extern "C" int jfb_tps_project_from_orthogonal(jfb_tps* t, const void* orth, void* coeffs,
                                               void* stream) {
  JFB_REQUIRE(t && orth && coeffs, "null pointer");
  return tps_xw(t, kXProjectOrth, 0, 0, 0, 1.0, (const c64*)orth, (c64*)coeffs,
                (cudaStream_t)stream);
}

extern "C" int jfb_tps_scalar_product_from_orthogonal(jfb_tps* t, const void* orth, void* out,
                                                      void* stream) {
  JFB_REQUIRE(t && orth && out, "null pointer");
  double w = 1.0;  // Fourier mass 2 pi / df per periodic axis
  for (int a = 0; a + 1 < t->cfg.ndim; ++a) w *= 2.0 * M_PI / fourier_df(t, a);
  return tps_xw(t, kXSpFromOrth, 0, 0, 0, w, (const c64*)orth, (c64*)out, (cudaStream_t)stream);
}

extern "C" int jfb_tps_galerkin(const jfb_tps* t, int order, double* out) {
  JFB_REQUIRE(t && out, "null pointer");
  JFB_REQUIRE(order == 0 || order == 2, "order must be 0 or 2");
  const std::vector<double>& G = order ? t->G2 : t->G0;
  std::copy(G.begin(), G.end(), out);
  return JFB_OK;
}

extern "C" int jfb_tps_get_sizes(const jfb_tps* t, int32_t* out4) {
  JFB_REQUIRE(t && out4, "null pointer");
  out4[0] = t->nb;
  out4[1] = t->N;
  out4[2] = t->m1;
  out4[3] = t->m2;
  return JFB_OK;
}

extern "C" int jfb_helmholtz2d_solve(const jfb_tps* tc, const jfb_tps* td, const double* L,
                                     const int64_t* L_offsets, int64_t n_L, const double* U,
                                     const int64_t* U_offsets, int64_t n_U, const double* U_inv,
                                     double fourier_mass, const void* f_hat, void* u,
                                     void* stream) {
  JFB_REQUIRE(tc && td && U && U_offsets && f_hat && u, "null pointer");
  JFB_REQUIRE(n_L == 0 || (L && L_offsets), "null L factor");
  JFB_REQUIRE(tc->cfg.ndim == 2 && td->cfg.ndim == 2, "2-D spaces only");
  JFB_REQUIRE(tc->cfg.basis == JFB_BASIS_ORTHOGONAL && td->cfg.basis == JFB_BASIS_DIRICHLET,
              "tc must be orthogonal, td Dirichlet");
  JFB_REQUIRE(tc->N == td->N && tc->n1 == td->n1 && tc->nb == tc->N, "tc, td sizes differ");
  JFB_REQUIRE(tc->cfg.family == td->cfg.family, "tc, td families differ");
  JFB_REQUIRE(fourier_mass != 0.0, "fourier_mass must be nonzero");
  JFB_REQUIRE(n_L >= 0 && n_L <= kHelmMaxDiag && n_U >= 1 && n_U <= kHelmMaxDiag,
              "too many diagonals");
  const int N = td->N, nb = td->nb, M = td->n1;
  const int KC = (M + kHelmCTAs - 1) / kHelmCTAs, JR = (N + kHelmCTAs - 1) / kHelmCTAs;
  // the size range of this call, unchanged since the solve was one cluster's: 2 N c
  // + N q + 2 n1 ceil(N/8) complex values and the x operator in one CTA's shared
  // memory.  What it refuses goes through the separate launches.
  const int QS = KC + ((5 - KC % 4) % 4);
  const size_t smem = ((size_t)2 * N * KC + (size_t)N * QS + (size_t)2 * M * JR) * sizeof(c64) +
                      (size_t)nb * N * sizeof(double);
  int dev = 0, optin = 0;
  JFB_CHECK_CUDA(cudaGetDevice(&dev));
  JFB_CHECK_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  if (smem > (size_t)optin) {
    set_error("problem too large for the fused Helmholtz solve");
    return JFB_ERR_ARG;
  }
  Helm2DArgs h;
  std::memset(&h, 0, sizeof(h));
  h.nL = (int)n_L;
  h.nU = (int)n_U;
  h.umain = -1;
  for (int d = 0; d < h.nL; ++d) {
    h.loff[d] = (int)L_offsets[d];
    JFB_REQUIRE(h.loff[d] < 0, "L offsets must be < 0");
  }
  for (int d = 0; d < h.nU; ++d) {
    h.uoff[d] = (int)U_offsets[d];
    JFB_REQUIRE(h.uoff[d] >= 0, "U offsets must be >= 0");
    if (h.uoff[d] == 0) h.umain = d;
  }
  JFB_REQUIRE(h.umain >= 0, "U offsets must contain the main diagonal");
  JFB_REQUIRE(!U_inv || td->nb <= 128, "U_inv form: at most 128 unknowns per mode");
  h.Uinv = U_inv;
  h.l2 = h.l4 = -1;
  bool two_four = true;
  for (int d = 0; d < h.nL; ++d) {
    if (h.loff[d] == -2) h.l2 = d;
    else if (h.loff[d] == -4) h.l4 = d;
    else two_four = false;
  }
  if (!two_four) h.l2 = h.l4 = -1;  // the general column-oriented form
  // the column updates of one step write one row per diagonal
  for (int a = 0; a < h.nU; ++a)
    for (int b = a + 1; b < h.nU; ++b) JFB_REQUIRE(h.uoff[a] != h.uoff[b], "repeated U offset");
  for (int a = 0; a < h.nL; ++a)
    for (int b = a + 1; b < h.nL; ++b) JFB_REQUIRE(h.loff[a] != h.loff[b], "repeated L offset");
  h.ns = td->ns;
  h.BDT = td->BT;
  h.L = L;
  h.U = U;
  h.N = N;
  h.nb = nb;
  h.M = M;
  // Fourier scalar-product weight 2 pi / df (Fourier.py:152-167) and the
  // caller's division by the Fourier mass
  const double Ly = td->cfg.l[0];
  const double df = std::fabs(Ly - 2.0 * M_PI) < 1e-12 ? 1.0 : 2.0 * M_PI / Ly;
  h.scale = (2.0 * M_PI / df) / fourier_mass;
  h.f = (const c64*)f_hat;
  h.u = (c64*)u;
  cudaStream_t cs = (cudaStream_t)stream;
  size_t sm = (size_t)(N + 2 * nb + kHelmThreads) * sizeof(c64) + (size_t)2 * nb * sizeof(double);
  const size_t factors = (size_t)(h.nL + h.nU) * (nb | 1) * sizeof(double);
  h.staged = !(U_inv && h.l2 + h.l4 > -2) && sm + factors <= 200 * 1024;
  if (h.staged) sm += factors;
  // (the kernel holds 2 KB besides)
  if (sm > 46 * 1024) JFB_CHECK_CUDA(allow_smem((const void*)helmholtz2d_kernel));
  helmholtz2d_kernel<<<M, kHelmThreads, sm, cs>>>(h);
  JFB_CHECK_LAUNCH();
  // y: inverse transform of the rows, in place
  return tps_lines(td->f1n, td->tw1n, +1, N, M, M, h.u, h.u, cs);
}
