// jaxfun.la replacements: DIA matvec / rmatvec, batched no-pivot banded LU and
// the per-wavenumber banded solve, as standalone C-ABI entry points.
//
// Reference semantics:
//   DiaMatrix storage / matvec / rmatvec   src/jaxfun/la/diamatrix.py:100-348
//   no-pivot banded LU kernel              src/jaxfun/la/diamatrix.py:1936-1973
//   batched wavenumber solve               src/jaxfun/la/tpmatrix.py:686-799
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "jfb_common.cuh"

namespace jfb {

static thread_local std::string g_last_error;
void set_error(const std::string& msg) { g_last_error = msg; }
const char* last_error() { return g_last_error.c_str(); }

constexpr int kMaxOffsets = 512;

struct OffsetTable {
  int n;
  int off[kMaxOffsets];
};

// ---------------------------------------------------------------------------
// DIA matvec:  y[o, i, t] = sum_d data[d, i + k_d] * x[o, i + k_d, t]
// DIA rmatvec: y[o, j, t] = sum_d data[d, j] * x[o, j - k_d, t]
// One thread per output element; t (inner) is the fastest index so that a
// warp reads contiguous x and writes contiguous y.
// ---------------------------------------------------------------------------
template <typename V>
__global__ void dia_matvec_kernel(const double* __restrict__ data, OffsetTable offs,
                                  int64_t n_rows, int64_t n_cols,
                                  const V* __restrict__ x, V* __restrict__ y,
                                  int64_t outer, int64_t inner, int transpose) {
  const int64_t n_out = transpose ? n_cols : n_rows;
  const int64_t n_in = transpose ? n_rows : n_cols;
  const int64_t total = outer * n_out * inner;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx % inner;
    const int64_t i = (idx / inner) % n_out;
    const int64_t o = idx / (inner * n_out);
    const V* xo = x + o * n_in * inner;
    double acc_re = 0.0, acc_im = 0.0;
    for (int d = 0; d < offs.n; ++d) {
      const int64_t k = offs.off[d];
      int64_t col, xi;
      if (!transpose) {
        col = i + k;  // A[i, i+k] stored at data[d, i+k]
        xi = col;
        if (col < 0 || col >= n_cols || i >= n_rows) continue;
      } else {
        col = i;      // (x @ A)[j] = sum_d data[d, j] x[j - k]
        xi = i - k;
        if (xi < 0 || xi >= n_rows) continue;
      }
      const double a = data[d * n_cols + col];
      const V xv = xo[xi * inner + t];
      if constexpr (sizeof(V) == sizeof(double)) {
        acc_re += a * (double)xv;
      } else {
        acc_re += a * xv.re;
        acc_im += a * xv.im;
      }
    }
    if constexpr (sizeof(V) == sizeof(double)) {
      y[idx] = acc_re;
    } else {
      y[idx] = cmk(acc_re, acc_im);
    }
  }
}

// ---------------------------------------------------------------------------
// Batched banded LU without pivoting.  One warp per matrix: for each column
// k and each sub-diagonal s the lanes update the trailing row segment in
// parallel (the elimination order per entry is identical to the reference's
// sequential loop: every entry receives its updates in increasing k).
// band[b][p + off][j] = A_b[j - off, j].
// ---------------------------------------------------------------------------
__global__ void banded_lu_kernel(double* __restrict__ band, int64_t n_batch, int p,
                                 int q, int n, int* __restrict__ bad) {
  const int lane = threadIdx.x & 31;
  const int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (b >= n_batch) return;
  const int bw = p + q + 1;
  double* A = band + b * (int64_t)bw * n;
  auto at = [&](int row, int col) -> double& { return A[(int64_t)row * n + col]; };
  const int c = p;
  for (int k = 0; k < n; ++k) {
    const double pivot = at(c, k);
    if (lane == 0 && (!(fabs(pivot) > 0.0) || !isfinite(pivot))) atomicExch(bad, 1);
    for (int s = 1; s <= p; ++s) {
      if (k + s >= n) break;
      const double f = at(c - s, k) / pivot;
      __syncwarp();
      if (lane == 0) at(c - s, k) = f;
      for (int u = 1 + lane; u <= q; u += 32) {
        const int j = k + u;
        if (j < n) at(c + u - s, j) -= f * at(c + u, j);
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------
// Wavenumber solve.  One thread per (rhs r, Fourier mode f): forward
// elimination with the unit-lower factor, then back substitution.
// rhs/out layout (n_rhs, outer, n_P, inner); mode f = o * inner + t.
// ---------------------------------------------------------------------------
template <typename V>
__global__ void wavenumber_solve_kernel(const double* __restrict__ L, OffsetTable loff,
                                        const double* __restrict__ U, OffsetTable uoff,
                                        int main_idx, int n_P, int64_t outer,
                                        int64_t inner, int64_t n_rhs,
                                        const V* __restrict__ rhs, V* __restrict__ out) {
  const int64_t n_F = outer * inner;
  const int64_t gid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (gid >= n_F * n_rhs) return;
  const int64_t t = gid % inner;
  const int64_t o = (gid / inner) % outer;
  const int64_t r = gid / n_F;
  const int64_t f = o * inner + t;
  const int64_t base = (r * outer + o) * (int64_t)n_P * inner + t;
  const double* Lf = L + f * (int64_t)loff.n * n_P;
  const double* Uf = U + f * (int64_t)uoff.n * n_P;
  const V* b = rhs + base;
  V* x = out + base;
  constexpr bool kCplx = sizeof(V) != sizeof(double);
  // forward: y_i = b_i - sum_s L[i, i-s] y_{i-s};  L[i, i-s] = Ldata[d][i-s]
  for (int i = 0; i < n_P; ++i) {
    double yr, yi = 0.0;
    if constexpr (kCplx) {
      yr = b[(int64_t)i * inner].re;
      yi = b[(int64_t)i * inner].im;
    } else {
      yr = b[(int64_t)i * inner];
    }
    double ar = 0.0, ai = 0.0;
    for (int d = 0; d < loff.n; ++d) {
      const int j = i + loff.off[d];
      if (j < 0) continue;
      const double l = Lf[(int64_t)d * n_P + j];
      if constexpr (kCplx) {
        const V yj = x[(int64_t)j * inner];
        ar += l * yj.re;
        ai += l * yj.im;
      } else {
        ar += l * x[(int64_t)j * inner];
      }
    }
    if constexpr (kCplx) {
      x[(int64_t)i * inner] = cmk(yr - ar, yi - ai);
    } else {
      x[(int64_t)i * inner] = yr - ar;
    }
  }
  // backward: x_i = (y_i - sum_s U[i, i+s] x_{i+s}) / U[i, i]
  for (int i = n_P - 1; i >= 0; --i) {
    double ar = 0.0, ai = 0.0;
    for (int d = 0; d < uoff.n; ++d) {
      const int s = uoff.off[d];
      if (s == 0) continue;
      const int j = i + s;
      if (j >= n_P) continue;
      const double u = Uf[(int64_t)d * n_P + j];
      if constexpr (kCplx) {
        const V xj = x[(int64_t)j * inner];
        ar += u * xj.re;
        ai += u * xj.im;
      } else {
        ar += u * x[(int64_t)j * inner];
      }
    }
    const double diag = Uf[(int64_t)main_idx * n_P + i];
    if constexpr (kCplx) {
      const V yi = x[(int64_t)i * inner];
      x[(int64_t)i * inner] = cmk((yi.re - ar) / diag, (yi.im - ai) / diag);
    } else {
      x[(int64_t)i * inner] = (x[(int64_t)i * inner] - ar) / diag;
    }
  }
}

// Same solve, one warp per (rhs r, Fourier mode f), for factors with many
// diagonals (the dense upper triangles of Chebyshev stiffness matrices).
// Column-oriented substitution on the system's vector in shared memory: once
// x_c is final, lane t applies the column-c entry of diagonal t to that
// diagonal's row (distinct diagonals hit distinct rows, so the updates of one
// column are independent).  The dependent chain is one shared read, (for U)
// a division and one update per column; the factor entries of the next
// column are loaded while the current one is applied.  Reads rhs, writes out
// (in place allowed: a warp reads its whole vector before it writes).
template <typename V>
__global__ void wavenumber_solve_warp_kernel(const double* __restrict__ L, OffsetTable loff,
                                             const double* __restrict__ U, OffsetTable uoff,
                                             int main_idx, int n_P, int64_t outer,
                                             int64_t inner, int64_t n_rhs, const V* rhs,
                                             V* out) {
  extern __shared__ double wsm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double* xr = wsm + (size_t)wib * 2 * n_P;
  double* xi = xr + n_P;
  const int64_t n_F = outer * inner;
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (gid >= n_F * n_rhs) return;
  const int64_t t = gid % inner;
  const int64_t o = (gid / inner) % outer;
  const int64_t r = gid / n_F;
  const int64_t f = o * inner + t;
  const int64_t base = (r * outer + o) * (int64_t)n_P * inner + t;
  const double* Lf = L + f * (int64_t)loff.n * n_P;
  const double* Uf = U + f * (int64_t)uoff.n * n_P;
  constexpr bool kCplx = sizeof(V) != sizeof(double);
  for (int i = lane; i < n_P; i += 32) {
    if constexpr (kCplx) {
      const V v = rhs[base + (int64_t)i * inner];
      xr[i] = v.re;
      xi[i] = v.im;
    } else {
      xr[i] = rhs[base + (int64_t)i * inner];
      xi[i] = 0.0;
    }
  }
  __syncwarp();
  // forward: L[i, i + s] (s < 0) sits at column c = i + s, Lf[d * n_P + c]
  const int lrow = (lane < loff.n) ? -loff.off[lane] : n_P;  // row = c + lrow
  double lnext = (lrow < n_P) ? Lf[(int64_t)lane * n_P] : 0.0;
  for (int c = 0; c < n_P; ++c) {
    const double l = lnext;
    if (c + 1 + lrow < n_P) lnext = Lf[(int64_t)lane * n_P + c + 1];
    const double yr = xr[c], yi = xi[c];
    if (c + lrow < n_P) {
      xr[c + lrow] -= l * yr;
      xi[c + lrow] -= l * yi;
    }
    for (int d = lane + 32; d < loff.n; d += 32) {
      const int i = c - loff.off[d];
      if (i >= n_P) continue;
      const double ld = Lf[(int64_t)d * n_P + c];
      xr[i] -= ld * yr;
      xi[i] -= ld * yi;
    }
    __syncwarp();
  }
  // backward: U[i, i + s] (s > 0) sits at column c = i + s, Uf[d * n_P + c]
  const int urow = (lane < uoff.n && uoff.off[lane] != 0) ? uoff.off[lane] : -1;  // row = c - urow
  const double* Ud = Uf + (int64_t)main_idx * n_P;
  double unext = (urow > 0 && n_P - 1 - urow >= 0) ? Uf[(int64_t)lane * n_P + n_P - 1] : 0.0;
  double dnext = Ud[n_P - 1];
  for (int c = n_P - 1; c >= 0; --c) {
    const double u = unext, dg = dnext;
    if (c > 0) {
      dnext = Ud[c - 1];
      if (urow > 0 && c - 1 - urow >= 0) unext = Uf[(int64_t)lane * n_P + c - 1];
    }
    const double x_r = xr[c] / dg, x_i = xi[c] / dg;
    if (lane == (c & 31)) {
      if constexpr (kCplx) out[base + (int64_t)c * inner] = cmk(x_r, x_i);
      else out[base + (int64_t)c * inner] = x_r;
    }
    if (urow > 0 && c - urow >= 0) {
      xr[c - urow] -= u * x_r;
      xi[c - urow] -= u * x_i;
    }
    for (int d = lane + 32; d < uoff.n; d += 32) {
      const int sft = uoff.off[d];
      const int i = c - sft;
      if (sft == 0 || i < 0) continue;
      const double ud = Uf[(int64_t)d * n_P + c];
      xr[i] -= ud * x_r;
      xi[i] -= ud * x_i;
    }
    __syncwarp();
  }
}

// The same solve with the factors staged in shared memory.  A block owns M
// consecutive modes (neighbours along `inner`, so that neighbouring vectors
// share their memory sectors) and RB right-hand sides of each, and loads only
// the entries a factor has (column c of diagonal s >= 0 from c = s on: half
// the bytes of a full triangle), once for all right-hand sides.  When every
// offset is even the two parity classes are independent systems.
//   wide factors    (wavenumber_solve_tri_kernel) a warp per mode with the
//                   unknowns in registers, lane = row of a class; U (and L,
//                   when it has more than kTriFewL diagonals) as packed dense
//                   triangles, so a column update is one shared-memory read
//                   and one multiply-add per row.  A column of U is divided by
//                   U[c, c] as it is read, off the chain of the y_c, and x_c =
//                   y_c / U[c, c] on output: the roundings of a division per
//                   column (products with 1 / U[c, c] have one more, 6 % more
//                   error).
//                   Up to four right-hand sides share a warp and its factor
//                   reads.  Bound by issue.
//   narrow factors  (wavenumber_solve_narrow_kernel) a thread per vector and
//                   class, rows in order, vectors in shared memory.
// n_P = 63, 4096 modes, three complex right-hand sides (one class of 32 and
// one of 31 rows): 80 us.  A warp per system reading strided vectors and the
// factors once per right-hand side took 201 us; with the vectors in shared
// memory instead of registers 279 us (two read-modify-writes of 16 bytes per
// lane and column); one right-hand side per warp 84 us.
struct StagedTable {
  int n;
  int off[kMaxOffsets];
  int start[kMaxOffsets];  // first staged entry of the diagonal within the mode's record
};
struct StagedSolve {
  StagedTable L, U;
  int main, n, rec, ldx, M, RB, even, denseL, zero;
  int oL, oD, m0;  // tri form: L part and reciprocal diagonal within the record, class 0 rows
  unsigned outer, inner;
  int64_t n_F, n_rhs;
};
constexpr int kStagedNarrow = 8;  // diagonals a single thread walks
constexpr int kTriFewL = 4;       // diagonals of L kept as diagonals in the tri form

// Element i of right-hand side r of mode f = o inner + t.
__device__ __forceinline__ size_t staged_addr(const StagedSolve& q, unsigned f, int64_t r, int i) {
  const unsigned o = f / q.inner, t = f - o * q.inner;
  return ((size_t)(r * q.outer + o) * q.n + i) * q.inner + t;
}

template <typename V>
__global__ void wavenumber_solve_narrow_kernel(const __grid_constant__ StagedSolve q,
                                               const double* __restrict__ L,
                                               const double* __restrict__ U, const V* rhs,
                                               V* out) {
  constexpr bool kCplx = sizeof(V) != sizeof(double);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = q.n, nv = q.M * q.RB, tid = threadIdx.x, nt = blockDim.x;
  V* xs = reinterpret_cast<V*>(smem_raw);                       // [nv][ldx]
  double* fac = reinterpret_cast<double*>(xs + (size_t)nv * q.ldx);  // [M][rec]
  const int64_t f0 = (int64_t)blockIdx.x * q.M, r0 = (int64_t)blockIdx.y * q.RB;
  const int mv = (int)min((int64_t)q.M, q.n_F - f0), rv = (int)min((int64_t)q.RB, q.n_rhs - r0);
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  // factors: one warp per (mode, diagonal), lanes over its columns, all copies
  // in flight together
  for (int u = warp; u < mv * (q.L.n + q.U.n); u += nw) {
    const int m = u / (q.L.n + q.U.n), dd = u - m * (q.L.n + q.U.n);
    const bool up = dd >= q.L.n;
    const int d = up ? dd - q.L.n : dd;
    const int s = up ? q.U.off[d] : -q.L.off[d];
    const double* src = up ? U + ((f0 + m) * q.U.n + d) * n + s : L + ((f0 + m) * q.L.n + d) * n;
    double* dst = fac + (size_t)m * q.rec + (up ? q.U.start[d] : q.L.start[d]);
    for (int c = lane; c < n - s; c += 32) cp_async8(dst + c, src + c);
  }
  auto each = [&](auto&& fn) {  // all elements, the contiguous index fastest
    for (int e = tid; e < nv * n; e += nt) {
      int m, r, i;
      if (q.inner == 1) {
        i = e % n;
        m = (e / n) % q.M;
        r = e / (n * q.M);
      } else {
        m = e % q.M;
        i = (e / q.M) % n;
        r = e / (n * q.M);
      }
      if (m < mv && r < rv) fn(staged_addr(q, (unsigned)f0 + m, r0 + r, i), (r * q.M + m) * q.ldx + i);
    }
  };
  each([&](size_t g, int k) {
    const double* v = reinterpret_cast<const double*>(rhs + g);
    double* w = reinterpret_cast<double*>(xs + k);
    cp_async8(w, v);
    if constexpr (kCplx) cp_async8(w + 1, v + 1);
  });
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  const int step = q.even ? 2 : 1;
  const int v = tid / step, cls = tid - v * step;
  const int m = v % q.M, r = v / q.M;
  if (v < nv && m < mv && r < rv && cls < n) {  // (n = 1: class 1 has no rows)
    V* x = xs + (size_t)v * q.ldx;
    const double* fm = fac + (size_t)m * q.rec;
    for (int i = cls; i < n; i += step) {
      V y = x[i], acc = V();
      for (int d = 0; d < q.L.n; ++d) {
        const int j = i + q.L.off[d];
        if (j >= 0) acc = acc + fm[q.L.start[d] + j] * x[j];
      }
      x[i] = y - acc;
    }
    for (int i = n - 1 - ((n - 1 - cls) % step); i >= 0; i -= step) {
      V y = x[i], acc = V();
      for (int d = 0; d < q.U.n; ++d) {
        const int sft = q.U.off[d], j = i + sft;
        if (sft != 0 && j < n) acc = acc + fm[q.U.start[d] + i] * x[j];
      }
      const double dg = fm[q.U.start[q.main] + i];
      y = y - acc;
      if constexpr (kCplx) x[i] = cmk(y.re / dg, y.im / dg);
      else x[i] = y / dg;
    }
  }
  __syncthreads();
  each([&](size_t g, int k) { out[g] = xs[k]; });
}

// S: rows per lane and class; R: right-hand sides per warp (they share every
// factor read and keep R independent chains in flight).
template <typename V, int S, int R>
__global__ void wavenumber_solve_tri_kernel(const __grid_constant__ StagedSolve q,
                                            const double* __restrict__ L,
                                            const double* __restrict__ U, const V* rhs, V* out) {
  constexpr bool kCplx = sizeof(V) != sizeof(double);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* fac = reinterpret_cast<double*>(smem_raw);  // [M][rec]
  const int n = q.n, tid = threadIdx.x, nt = blockDim.x;
  const int64_t f0 = (int64_t)blockIdx.x * q.M, r0 = (int64_t)blockIdx.y * q.RB;
  const int mv = (int)min((int64_t)q.M, q.n_F - f0);
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  const int ncls = q.even ? 2 : 1, sh = q.even ? 1 : 0;
  const int tri1 = q.m0 * (q.m0 + 1) / 2;  // first entry of class 1's triangle
  // this warp's mode and right-hand sides, loaded first (lane + 32 s = row of
  // the class)
  const int m = warp % q.M;
  const int64_t rw = r0 + (int64_t)(warp / q.M) * R;
  const int rv = (int)min((int64_t)R, min(q.n_rhs, r0 + q.RB) - rw);
  const bool live = m < mv && rv > 0;
  V y[R][2][S];
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int cl = 0; cl < 2; ++cl)
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const int i = ((lane + 32 * s) << sh) + cl;
        y[k][cl][s] = live && k < rv && cl < ncls && i < n
                          ? rhs[staged_addr(q, (unsigned)f0 + m, rw + k, i)]
                          : V();
      }
  // absent diagonals read as zero
  if (q.zero)
    for (int e = tid; e < q.M * q.rec; e += nt) fac[e] = 0.0;
  __syncthreads();
  // factors: one warp per (mode, diagonal), lanes over its columns, all
  // copies in flight together
  auto copy8 = [](double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
  };
  for (int u = warp; u < mv * (q.L.n + q.U.n); u += nw) {
    const int mm = u / (q.L.n + q.U.n), dd = u - mm * (q.L.n + q.U.n);
    const bool up = dd >= q.L.n;
    const int d = up ? dd - q.L.n : dd;
    const int s = up ? q.U.off[d] : -q.L.off[d];
    const double* src = up ? U + ((f0 + mm) * q.U.n + d) * n : L + ((f0 + mm) * q.L.n + d) * n;
    double* F = fac + (size_t)mm * q.rec;
    if (up && d == q.main) {
      for (int c = lane; c < n; c += 32) copy8(F + q.oD + c, src + c);
    } else if (up) {
      for (int c = s + lane; c < n; c += 32) {  // entry (c - s, c)
        const int cc = c >> sh, rr = (c - s) >> sh;
        copy8(F + (sh && (c & 1) ? tri1 : 0) + cc * (cc + 1) / 2 + rr, src + c);
      }
    } else {
      for (int c = lane; c < n - s; c += 32) {  // entry (c + s, c)
        const int cc = c >> sh, rr = (c + s) >> sh;
        copy8(F + q.oL + (q.denseL ? (sh && (c & 1) ? tri1 : 0) + rr * (rr + 1) / 2 + cc : d * n + c),
              src + c);
      }
    }
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // reciprocal diagonals in the triangles' own diagonal entries
  for (int e = tid; e < mv * n; e += nt) {
    double* Fm = fac + (size_t)(e / n) * q.rec;
    const int i = e % n, c = i >> sh;
    Fm[(sh && (i & 1) ? tri1 : 0) + c * (c + 1) / 2 + c] = 1.0 / Fm[q.oD + i];
  }
  __syncthreads();
  if (!live) return;  // no barrier below
  const double* F = fac + (size_t)m * q.rec;
  const int mc[2] = {q.even ? q.m0 : n, q.even ? n / 2 : 0};
  auto bcast = [&](const V (&v)[S], int c) {
    V a = v[0];
#pragma unroll
    for (int s = 1; s < S; ++s)
      if (c >= 32 * s) a = v[s];
    if constexpr (kCplx)
      return cmk(__shfl_sync(0xffffffffu, a.re, c & 31), __shfl_sync(0xffffffffu, a.im, c & 31));
    else
      return __shfl_sync(0xffffffffu, a, c & 31);
  };
  // forward, unit lower: column c of both classes per step
  const int steps = mc[0];
  if (q.L.n) {
    const int s1 = q.denseL || q.L.n != 1 ? 0 : (-q.L.off[0]) >> sh;  // the only diagonal's row shift
#pragma unroll 1
    for (int c = 0; c < steps - 1; ++c) {
#pragma unroll
      for (int cl = 0; cl < 2; ++cl) {
        if (c >= mc[cl]) continue;  // whole warp
        double l[S];                // this lane's entries of column c
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const int rr = lane + 32 * s;
          l[s] = 0.0;
          if (q.denseL) {
            if (rr > c && rr < mc[cl]) l[s] = F[q.oL + (cl ? tri1 : 0) + rr * (rr + 1) / 2 + c];
          } else if (s1) {
            if (rr == c + s1 && rr < mc[cl]) l[s] = F[q.oL + (c << sh) + cl];
          } else {
            for (int d = 0; d < q.L.n; ++d)
              if (rr == c + ((-q.L.off[d]) >> sh) && rr < mc[cl])
                l[s] = F[q.oL + d * n + (c << sh) + cl];
          }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const V yc = bcast(y[k][cl], c);
#pragma unroll
          for (int s = 0; s < S; ++s)
            if (l[s] != 0.0) y[k][cl][s] = y[k][cl][s] - l[s] * yc;
        }
      }
    }
  }
  // backward with the upper factor
#pragma unroll 2
  for (int c = steps - 1; c > 0; --c) {
#pragma unroll
    for (int cl = 0; cl < 2; ++cl) {
      if (c >= mc[cl]) continue;
      const double* T = F + (cl ? tri1 : 0) + c * (c + 1) / 2;
      const double dg = F[q.oD + (c << sh) + cl], rd = T[c];
      double u[S];
#pragma unroll
      for (int s = 0; s < S; ++s)
        u[s] = lane + 32 * s < c ? quotient(T[lane + 32 * s], dg, rd) : 0.0;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const V yc = bcast(y[k][cl], c);
#pragma unroll
        for (int s = 0; s < S; ++s)
          if (lane + 32 * s < c) y[k][cl][s] = y[k][cl][s] - u[s] * yc;
      }
    }
  }
#pragma unroll
  for (int cl = 0; cl < 2; ++cl)
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int i = ((lane + 32 * s) << sh) + cl;
      if (cl >= ncls || i >= n) continue;
      const int c = lane + 32 * s;
      const double dg = F[q.oD + i], rd = F[(cl ? tri1 : 0) + c * (c + 1) / 2 + c];
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (k >= rv) continue;
        // (infinities and NaN: the product alone)
        auto result = [&](double v) {
          const double x = quotient(v, dg, rd);
          return isfinite(x) ? x : v * rd;
        };
        V x = y[k][cl][s];
        if constexpr (kCplx) x = cmk(result(x.re), result(x.im));
        else x = result(x);
        out[staged_addr(q, (unsigned)f0 + m, rw + k, i)] = x;
      }
    }
}

// Whether the staged form is the faster one, `waves` being its blocks over
// those resident at once.  A block lasts as long as its chains, so the staged
// time is that of a chain times the waves, while the unstaged kernels keep
// every vector in flight until memory bounds them.  Measured (complex, n
// unknowns, F modes, r right-hand sides; unstaged -> staged, us):
//   narrow, two classes: n = 129, F = 4096: r = 1 (0.9 waves) 179 -> 70, r = 3
//     (1.4) 228 -> 138, r = 8 (2.8) 323 -> 230; n = 255, F = 4096, r = 8 (5.5)
//     684 -> 782; n = 2000, F = 4096, r = 3 (28) 3736 -> 21431.  Short chains
//     keep their lead over more waves: n = 48, F = 4096, r = 64 (9.2) 499 ->
//     392, n = 63 (11) 638 -> 590, (25) 951 -> 1314, n = 97 (18) 1005 -> 1270.  The smallest pay
//     only by sharing factors: n = 16, F = 64: r = 2 21 -> 25, r = 8 22 -> 18;
//     n = 8 14 -> 19.
//   narrow, one class (a chain twice as long): n = 129, F = 4096: r = 1 (0.7)
//     130 -> 93, r = 2 (1.2) 134 -> 191; n = 48, F = 64, r = 2 42 -> 50, n = 63
//     59 -> 62, n = 97 92 -> 74.
//   wide, F = 4096: n = 129, r = 1 (4.6) 210 -> 312, r = 3 600 -> 432; n = 255
//     (28): r = 1 866 -> 2441, r = 3 2556 -> 2919, r = 8 6754 -> 2648.  With a
//     smooth field's coefficients, whose smallest underflow, the unstaged
//     divisions take their slow path: n = 95, r = 1 (2.8) 173 -> 130, n = 127
//     (4.6) 275 -> 235, against 111 and 200 for random numbers.
static bool staged_pays(bool narrow, bool even, int n, int64_t n_rhs, double waves) {
  const int rows = even ? (n + 1) / 2 : n;  // of a class
  if (!narrow) return n_rhs >= 4 || waves <= (rows <= 64 ? 8.0 : 2.5) * n_rhs;
  if (!even) return n >= 64 && waves <= 1.0;
  if (n < 24) return n >= 12 && n_rhs >= 8;
  return n <= 48 || waves <= (n <= 64 ? 12.0 : 3.0);
}

// Launch of the staged solve, or false when one mode's factors and vector do
// not fit a CTA's shared memory (or, wide, more than four rows per lane), or
// the unstaged kernels are faster: those take it then.
template <typename V>
static bool staged_solve(const double* L, const OffsetTable& lt, const double* U,
                         const OffsetTable& ut, int main_idx, int n, int64_t outer, int64_t inner,
                         int64_t n_rhs, const V* rhs, V* out, cudaStream_t s, cudaError_t* err) {
  *err = cudaSuccess;
  StagedSolve q;
  std::memset(&q, 0, sizeof(q));
  q.main = main_idx;
  q.n = n;
  q.n_F = outer * inner;
  if (q.n_F > INT_MAX) return false;
  q.outer = (unsigned)outer;
  q.inner = (unsigned)inner;
  q.n_rhs = n_rhs;
  const bool narrow = lt.n + ut.n <= kStagedNarrow;
  q.even = 1;
  int64_t rec = 0;
  auto fill = [&](StagedTable& t, const OffsetTable& o) {
    t.n = o.n;
    for (int d = 0; d < o.n; ++d) {
      t.off[d] = o.off[d];
      t.start[d] = (int)rec;
      rec += std::max(0, n - std::abs(o.off[d]));
      if (o.off[d] & 1) q.even = 0;
    }
  };
  fill(q.L, lt);
  fill(q.U, ut);
  q.m0 = q.even ? (n + 1) / 2 : n;
  int S = 0;
  if (!narrow) {
    const int64_t m1 = q.even ? n / 2 : 0, tri = (int64_t)q.m0 * (q.m0 + 1) / 2 + m1 * (m1 + 1) / 2;
    if (q.m0 > 128) return false;
    S = q.m0 <= 32 ? 1 : q.m0 <= 64 ? 2 : 4;
    q.denseL = lt.n > kTriFewL;
    q.oL = (int)tri;
    q.oD = (int)(tri + (q.denseL ? tri : (int64_t)lt.n * n));
    rec = q.oD + n;
    int in_range = 0;
    for (int d = 0; d < ut.n; ++d) in_range += ut.off[d] < n;
    q.zero = in_range < q.m0 || q.denseL;
  }
  rec |= 1;  // consecutive modes' records in different banks
  q.ldx = narrow ? (n | 1) : 0;
  constexpr size_t kMost = 200 * 1024, kGood = 64 * 1024;
  auto bytes = [&](int M, int RB) {
    return (size_t)M * rec * sizeof(double) + (size_t)M * RB * q.ldx * sizeof(V);
  };
  if (bytes(1, 1) > kMost) return false;
  q.rec = (int)rec;
  // up to 16 vectors per block (a warp each; narrow: 128, one or two threads
  // each): right-hand sides first, then modes, as long as the records leave
  // about three blocks per SM
  const int most = narrow ? 128 : 16, mmax = narrow ? 16 : 4;
  q.M = 1;
  q.RB = (int)std::min<int64_t>(n_rhs, 8);
  const int R = narrow ? 1 : (int)std::min<int64_t>(S == 4 ? 2 : 4, n_rhs);
  while (q.RB > 1 && bytes(1, q.RB) > kMost) q.RB = (q.RB + 1) / 2;
  while (q.M * 2 <= mmax && q.M * 2 * q.RB <= most && q.M < q.n_F && bytes(q.M * 2, q.RB) <= kGood)
    q.M *= 2;
  const int vecs = q.M * ((q.RB + R - 1) / R);  // warps (narrow: vectors)
  const int threads = narrow ? std::max(64, (vecs * (q.even ? 2 : 1) + 31) / 32 * 32)
                             : std::max(2, vecs) * 32;
  const int64_t gx = (q.n_F + q.M - 1) / q.M, gy = (n_rhs + q.RB - 1) / q.RB;
  if (gy > 65535) return false;
  const int64_t resident = std::min<int64_t>(
      {228 * 1024 / (int64_t)(bytes(q.M, q.RB) + 1024), 2048 / threads, 32});
  if (!staged_pays(narrow, q.even, n, n_rhs, (double)gx * gy / (148.0 * resident)))
    return false;
  auto* k = wavenumber_solve_narrow_kernel<V>;
  switch (10 * S + R) {
#define JFB_TRI(SS, RR) \
  case 10 * SS + RR: k = wavenumber_solve_tri_kernel<V, SS, RR>; break;
    JFB_TRI(1, 1) JFB_TRI(1, 2) JFB_TRI(1, 3) JFB_TRI(1, 4)
    JFB_TRI(2, 1) JFB_TRI(2, 2) JFB_TRI(2, 3) JFB_TRI(2, 4)
    JFB_TRI(4, 1) JFB_TRI(4, 2)
#undef JFB_TRI
    default: break;  // narrow (S = 0)
  }
  *err = cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(kMost + 1024));
  if (*err != cudaSuccess) return true;
  k<<<dim3((unsigned)gx, (unsigned)gy), threads, bytes(q.M, q.RB), s>>>(q, L, U, rhs, out);
  *err = cudaGetLastError();
  return true;
}

// ---------------------------------------------------------------------------
// Sum of Kronecker terms with one polynomial axis (TPMatrices @ x,
// tpmatrix.py:300-428, for Fourier x polynomial operators):
//   y[o, i, t] = sum_k c_k w_k(f) sum_d data_k[d, i + off] x[o, i + off, t],
// f = o inner + t the flattened Fourier index, w_k the product of the term's
// diagonal matrices.  A block stages kTpCols columns of x in shared memory
// and forms all their rows: x is read and y written once, where one launch
// per factor of each term moved the field nine times for three terms (48 us
// of device time at 63 x 4096 complex in nine launches, plus the sums'; now
// 20 us in one).  Bound by the latency of its operator reads.
// ---------------------------------------------------------------------------
constexpr int kTpTerms = 8, kTpCols = 16, kTpThreads = 256, kTpRows = 4;
struct TpTerm {
  const double* data;   // (n_diags, n) DIA
  const double* w[2];   // Fourier diagonals (null: absent)
  double coef;
  int first, nd;        // its offsets in TpArgs::off
};
struct TpArgs {
  TpTerm t[kTpTerms];
  int off[kMaxOffsets];
  int nt, n;
  unsigned n_F, inner, size2;  // size2: length of the last Fourier axis
};

template <typename V>
__global__ void __launch_bounds__(kTpThreads)
    tp_matvec_kernel(const __grid_constant__ TpArgs a, const V* __restrict__ x, V* __restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double ws[kTpTerms * kTpCols];  // weights of the block's columns per term
  V* xs = reinterpret_cast<V*>(smem_raw);    // [n][kTpCols + 1]
  constexpr int LD = kTpCols + 1;
  const int n = a.n, tid = threadIdx.x;
  const unsigned f0 = blockIdx.x * kTpCols;
  const int nc = (int)min((unsigned)kTpCols, a.n_F - f0);
  auto addr = [&](int c, int i) {
    const unsigned f = f0 + c, o = f / a.inner, t = f - o * a.inner;
    return ((size_t)o * n + i) * a.inner + t;
  };
  for (int e = tid; e < n * kTpCols; e += kTpThreads) {
    const int c = a.inner == 1 ? e / n : e % kTpCols, i = a.inner == 1 ? e % n : e / kTpCols;
    if (c < nc) xs[i * LD + c] = x[addr(c, i)];
  }
  if (tid < kTpTerms * kTpCols && tid / kTpCols < a.nt) {
    const TpTerm& t = a.t[tid / kTpCols];
    const unsigned f = f0 + min(tid % kTpCols, nc - 1), i1 = f / a.size2, i2 = f - i1 * a.size2;
    double w = t.coef;
    if (t.w[0]) w *= __ldg(t.w[0] + i1);
    if (t.w[1]) w *= __ldg(t.w[1] + i2);
    ws[tid] = w;
  }
  __syncthreads();
  const int c = tid % kTpCols;
  // kTpRows rows per thread: independent chains over the diagonals
  constexpr int RG = kTpThreads / kTpCols;
  for (int i0 = tid / kTpCols; i0 < n; i0 += RG * kTpRows) {
    V sum[kTpRows];
#pragma unroll
    for (int r = 0; r < kTpRows; ++r) sum[r] = V();
#pragma unroll 1
    for (int k = 0; k < a.nt; ++k) {
      const TpTerm& t = a.t[k];
      V acc[kTpRows];
#pragma unroll
      for (int r = 0; r < kTpRows; ++r) acc[r] = V();
#pragma unroll 2
      for (int d = 0; d < t.nd; ++d) {
        const int off = a.off[t.first + d];
        const double* row = t.data + (size_t)d * n;
#pragma unroll
        for (int r = 0; r < kTpRows; ++r) {
          const int i = i0 + RG * r, col = i + off;
          if (i < n && col >= 0 && col < n) acc[r] = acc[r] + __ldg(row + col) * xs[col * LD + c];
        }
      }
      const double wk = ws[k * kTpCols + c];
#pragma unroll
      for (int r = 0; r < kTpRows; ++r) sum[r] = sum[r] + wk * acc[r];
    }
#pragma unroll
    for (int r = 0; r < kTpRows; ++r) {
      const int i = i0 + RG * r;
      if (c < nc && i < n) y[addr(c, i)] = sum[r];
    }
  }
}

static int fill_offsets(OffsetTable& t, const int64_t* offs, int64_t n) {
  if (n < 0 || n > kMaxOffsets) {
    set_error("too many DIA offsets (max 512)");
    return JFB_ERR_ARG;
  }
  t.n = (int)n;
  for (int64_t i = 0; i < n; ++i) t.off[i] = (int)offs[i];
  return JFB_OK;
}

}  // namespace jfb

using namespace jfb;

extern "C" int jfb_version(void) { return 1; }

extern "C" const char* jfb_last_error(void) { return jfb::last_error(); }

extern "C" int jfb_dia_matvec(const double* data, const int64_t* offsets,
                              int64_t n_diags, int64_t n_rows, int64_t n_cols,
                              const double* x, double* y, int64_t outer, int64_t inner,
                              int is_complex, int transpose, void* stream) {
  JFB_REQUIRE(data && offsets && x && y, "null pointer");
  JFB_REQUIRE(n_rows > 0 && n_cols > 0 && outer > 0 && inner > 0, "bad shape");
  OffsetTable t;
  int st = fill_offsets(t, offsets, n_diags);
  if (st) return st;
  const int64_t n_out = transpose ? n_cols : n_rows;
  const int64_t total = outer * n_out * inner;
  const int threads = 256;
  const int blocks = (int)std::min<int64_t>((total + threads - 1) / threads, 148 * 64);
  cudaStream_t s = (cudaStream_t)stream;
  if (is_complex) {
    dia_matvec_kernel<c64><<<blocks, threads, 0, s>>>(
        data, t, n_rows, n_cols, (const c64*)x, (c64*)y, outer, inner, transpose);
  } else {
    dia_matvec_kernel<double><<<blocks, threads, 0, s>>>(
        data, t, n_rows, n_cols, x, y, outer, inner, transpose);
  }
  JFB_CHECK_LAUNCH();
  return JFB_OK;
}

extern "C" int jfb_tp_matvec(int64_t n_terms, const double* const* data, const int64_t* n_diags,
                             const int64_t* offsets, const double* const* weights,
                             int64_t n_fourier, const int64_t* fourier_sizes, const double* coefs,
                             int64_t n_P, int64_t outer, int64_t inner, const double* x,
                             double* y, int is_complex, void* stream) {
  JFB_REQUIRE(data && n_diags && offsets && weights && fourier_sizes && coefs && x && y,
              "null pointer");
  JFB_REQUIRE(n_terms >= 1 && n_terms <= kTpTerms, "between 1 and 8 terms");
  JFB_REQUIRE(n_fourier >= 1 && n_fourier <= 2, "one or two Fourier axes");
  JFB_REQUIRE(n_P > 0 && n_P <= 4096 && outer > 0 && inner > 0, "bad shape");
  JFB_REQUIRE(outer <= INT_MAX / inner, "bad shape");
  int64_t nf = 1;
  for (int64_t k = 0; k < n_fourier; ++k) {
    JFB_REQUIRE(fourier_sizes[k] > 0 && fourier_sizes[k] <= INT_MAX, "bad shape");
    nf *= fourier_sizes[k];
  }
  JFB_REQUIRE(nf == outer * inner, "Fourier sizes do not match the field");
  TpArgs a;
  std::memset(&a, 0, sizeof(a));
  a.nt = (int)n_terms;
  a.n = (int)n_P;
  a.n_F = (unsigned)nf;
  a.inner = (unsigned)inner;
  a.size2 = n_fourier == 2 ? (unsigned)fourier_sizes[1] : 1u;
  int64_t at = 0;
  for (int k = 0; k < a.nt; ++k) {
    JFB_REQUIRE(data[k] && n_diags[k] >= 0 && at + n_diags[k] <= kMaxOffsets, "too many DIA offsets");
    TpTerm& t = a.t[k];
    t.data = data[k];
    t.coef = coefs[k];
    t.first = (int)at;
    t.nd = (int)n_diags[k];
    for (int64_t j = 0; j < n_fourier; ++j) t.w[j] = weights[k * n_fourier + j];
    for (int d = 0; d < t.nd; ++d) a.off[at + d] = (int)offsets[at + d];
    at += t.nd;
  }
  const size_t sm = (size_t)n_P * (kTpCols + 1) * (is_complex ? 16 : 8);
  JFB_REQUIRE(sm <= 200 * 1024, "polynomial axis too long for the fused product");
  const void* fn = is_complex ? (const void*)tp_matvec_kernel<c64>
                              : (const void*)tp_matvec_kernel<double>;
  JFB_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  const unsigned blocks = (a.n_F + kTpCols - 1) / kTpCols;
  cudaStream_t s = (cudaStream_t)stream;
  if (is_complex)
    tp_matvec_kernel<c64><<<blocks, kTpThreads, sm, s>>>(a, (const c64*)x, (c64*)y);
  else
    tp_matvec_kernel<double><<<blocks, kTpThreads, sm, s>>>(a, x, y);
  JFB_CHECK_LAUNCH();
  return JFB_OK;
}

extern "C" int jfb_banded_lu_factor(double* band, int64_t n_batch, int64_t p, int64_t q,
                                    int64_t n, void* stream) {
  JFB_REQUIRE(band, "null pointer");
  JFB_REQUIRE(n_batch > 0 && p >= 0 && q >= 0 && n > 0, "bad shape");
  cudaStream_t s = (cudaStream_t)stream;
  int* d_bad = nullptr;
  JFB_CHECK_CUDA(cudaMallocAsync((void**)&d_bad, sizeof(int), s));
  JFB_CHECK_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(int), s));
  const int threads = 128;
  const int64_t warps = n_batch;
  const int blocks = (int)((warps * 32 + threads - 1) / threads);
  banded_lu_kernel<<<blocks, threads, 0, s>>>(band, n_batch, (int)p, (int)q, (int)n,
                                              d_bad);
  JFB_CHECK_LAUNCH();
  int h_bad = 0;
  JFB_CHECK_CUDA(cudaMemcpyAsync(&h_bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, s));
  JFB_CHECK_CUDA(cudaFreeAsync(d_bad, s));
  JFB_CHECK_CUDA(cudaStreamSynchronize(s));
  if (h_bad) {
    set_error(
        "Matrix is singular or has a zero/non-finite pivot in LU factorisation "
        "without pivoting");
    return JFB_ERR_SINGULAR;
  }
  return JFB_OK;
}

extern "C" int jfb_wavenumber_solve(const double* L, const int64_t* L_offsets, int64_t n_L,
                                    const double* U, const int64_t* U_offsets, int64_t n_U,
                                    int64_t n_P, int64_t outer, int64_t inner,
                                    int64_t n_rhs, const double* rhs, double* out,
                                    int is_complex, void* stream) {
  JFB_REQUIRE(U && U_offsets && rhs && out, "null pointer");
  JFB_REQUIRE(n_L == 0 || (L && L_offsets), "null L factor");
  JFB_REQUIRE(n_P > 0 && outer > 0 && inner > 0 && n_rhs > 0, "bad shape");
  OffsetTable lt, ut;
  int st = fill_offsets(lt, L_offsets ? L_offsets : (const int64_t*)nullptr, n_L);
  if (st) return st;
  st = fill_offsets(ut, U_offsets, n_U);
  if (st) return st;
  int main_idx = -1;
  for (int d = 0; d < ut.n; ++d) {
    JFB_REQUIRE(ut.off[d] >= 0, "U offsets must be >= 0");
    if (ut.off[d] == 0) main_idx = d;
  }
  for (int d = 0; d < lt.n; ++d) JFB_REQUIRE(lt.off[d] < 0, "L offsets must be < 0");
  JFB_REQUIRE(main_idx >= 0, "U offsets must contain the main diagonal");
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t total = n_rhs * outer * inner;
  const int threads = 128;
  if (lt.n + ut.n > 8) {  // wide factors: a warp per system
    // the column updates of one step write one row per diagonal
    for (int a = 0; a < ut.n; ++a)
      for (int b = a + 1; b < ut.n; ++b) JFB_REQUIRE(ut.off[a] != ut.off[b], "repeated U offset");
    for (int a = 0; a < lt.n; ++a)
      for (int b = a + 1; b < lt.n; ++b) JFB_REQUIRE(lt.off[a] != lt.off[b], "repeated L offset");
    const size_t sm = (size_t)(threads / 32) * 2 * n_P * sizeof(double);
    JFB_REQUIRE(sm <= 48 * 1024, "n_P too large for the warp solve (max 768)");
  }
  {
    cudaError_t e;
    const bool done =
        is_complex ? staged_solve<c64>(L, lt, U, ut, main_idx, (int)n_P, outer, inner, n_rhs,
                                       (const c64*)rhs, (c64*)out, s, &e)
                   : staged_solve<double>(L, lt, U, ut, main_idx, (int)n_P, outer, inner, n_rhs,
                                          rhs, out, s, &e);
    if (done) {
      JFB_CHECK_CUDA(e);
      return JFB_OK;
    }
  }
  if (lt.n + ut.n > 8) {
    const int64_t wblocks = (total * 32 + threads - 1) / threads;
    const size_t sm = (size_t)(threads / 32) * 2 * n_P * sizeof(double);
    if (is_complex)
      wavenumber_solve_warp_kernel<c64><<<(unsigned)wblocks, threads, sm, s>>>(
          L, lt, U, ut, main_idx, (int)n_P, outer, inner, n_rhs, (const c64*)rhs, (c64*)out);
    else
      wavenumber_solve_warp_kernel<double><<<(unsigned)wblocks, threads, sm, s>>>(
          L, lt, U, ut, main_idx, (int)n_P, outer, inner, n_rhs, rhs, out);
    JFB_CHECK_LAUNCH();
    return JFB_OK;
  }
  if (rhs != out) {
    const int64_t elems = n_rhs * outer * n_P * inner * (is_complex ? 2 : 1);
    JFB_CHECK_CUDA(cudaMemcpyAsync(out, rhs, elems * sizeof(double),
                                   cudaMemcpyDeviceToDevice, s));
  }
  const int blocks = (int)((total + threads - 1) / threads);
  if (is_complex) {
    wavenumber_solve_kernel<c64><<<blocks, threads, 0, s>>>(
        L, lt, U, ut, main_idx, (int)n_P, outer, inner, n_rhs, (const c64*)out,
        (c64*)out);
  } else {
    wavenumber_solve_kernel<double><<<blocks, threads, 0, s>>>(
        L, lt, U, ut, main_idx, (int)n_P, outer, inner, n_rhs, out, out);
  }
  JFB_CHECK_LAUNCH();
  return JFB_OK;
}

// ===========================================================================
// Allocation-free variant of the batched banded LU.
//
// Some callers cannot call cudaMalloc at all: an XLA custom call or another
// framework's operator, whose device memory belongs to that framework's
// allocator, or a process whose caching pool already holds all of the GPU's
// memory.  jfb_banded_lu_factor above allocates its pivot-status word with
// cudaMallocAsync; this entry point keeps the pivot status of every matrix in
// a fixed file-scope device array instead, so it allocates nothing.  The
// array holds JFB_NOALLOC_LU_MAX_BATCH per-matrix flags plus one slot for the
// index of the first singular matrix; every GPU that loads the library holds
// it (256 KiB) until the process exits.  The call reads that index back to
// the host, so it synchronises its stream.
// ===========================================================================

static __device__ __align__(256) int g_noalloc_lu_status[JFB_NOALLOC_LU_MAX_BATCH + 1];

namespace jfb {

// Zero the per-matrix flags of this call and reset the first-singular slot.
__global__ void noalloc_lu_clear_kernel(int* status, int64_t n_batch) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_batch;
       i += (int64_t)gridDim.x * blockDim.x)
    status[i] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) status[JFB_NOALLOC_LU_MAX_BATCH] = INT_MAX;
}

// Same elimination as banded_lu_kernel (one warp per matrix, identical
// operation order); a zero or non-finite pivot sets status[b].
__global__ void noalloc_lu_kernel(double* __restrict__ band, int64_t n_batch, int p, int q,
                                  int n, int* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (b >= n_batch) return;
  double* A = band + b * (int64_t)(p + q + 1) * n;
  auto at = [&](int row, int col) -> double& { return A[(int64_t)row * n + col]; };
  const int c = p;
  for (int k = 0; k < n; ++k) {
    const double pivot = at(c, k);
    if (lane == 0 && (!(fabs(pivot) > 0.0) || !isfinite(pivot))) status[b] = 1;
    for (int s = 1; s <= p; ++s) {
      if (k + s >= n) break;
      const double f = at(c - s, k) / pivot;
      __syncwarp();
      if (lane == 0) at(c - s, k) = f;
      for (int u = 1 + lane; u <= q; u += 32) {
        const int j = k + u;
        if (j < n) at(c + u - s, j) -= f * at(c + u, j);
      }
      __syncwarp();
    }
  }
}

// Lowest index of a singular matrix into the last slot.
__global__ void noalloc_lu_first_kernel(int* status, int64_t n_batch) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_batch;
       i += (int64_t)gridDim.x * blockDim.x)
    if (status[i]) atomicMin(&status[JFB_NOALLOC_LU_MAX_BATCH], (int)i);
}

// Device address of the status array, looked up once per device with that
// device current (the host-side symbol is only a stand-in, not a device
// address, so it must never be passed to a kernel).  The address is kept for
// the life of the process: it is not valid after cudaDeviceReset.
static int noalloc_status_address(int** out) {
  static std::mutex mu;
  static int* addr[128] = {nullptr};
  int dev = 0;
  JFB_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 128) {
    set_error("device ordinal out of range");
    return JFB_ERR_ARG;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    int* p = nullptr;
    JFB_CHECK_CUDA(cudaGetSymbolAddress((void**)&p, g_noalloc_lu_status));
    addr[dev] = p;
  }
  *out = addr[dev];
  return JFB_OK;
}

}  // namespace jfb

extern "C" int jfb_banded_lu_factor_noalloc(double* band, int64_t n_batch, int64_t p,
                                            int64_t q, int64_t n, int32_t* first_singular,
                                            void* stream) {
  JFB_REQUIRE(band, "null pointer");
  JFB_REQUIRE(n_batch > 0 && p >= 0 && q >= 0 && n > 0, "bad shape");
  if (n_batch > JFB_NOALLOC_LU_MAX_BATCH) {
    set_error("n_batch exceeds JFB_NOALLOC_LU_MAX_BATCH (65536) of the allocation-free LU");
    return JFB_ERR_ARG;
  }
  int* status = nullptr;
  int st = noalloc_status_address(&status);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const int cblocks = (int)std::min<int64_t>((n_batch + 255) / 256, 1024);
  noalloc_lu_clear_kernel<<<cblocks, 256, 0, s>>>(status, n_batch);
  JFB_CHECK_LAUNCH();
  const int threads = 128;
  const int blocks = (int)((n_batch * 32 + threads - 1) / threads);
  noalloc_lu_kernel<<<blocks, threads, 0, s>>>(band, n_batch, (int)p, (int)q, (int)n, status);
  JFB_CHECK_LAUNCH();
  noalloc_lu_first_kernel<<<cblocks, 256, 0, s>>>(status, n_batch);
  JFB_CHECK_LAUNCH();
  int first = INT_MAX;
  JFB_CHECK_CUDA(cudaMemcpyAsync(&first, status + JFB_NOALLOC_LU_MAX_BATCH, sizeof(int),
                                 cudaMemcpyDeviceToHost, s));
  JFB_CHECK_CUDA(cudaStreamSynchronize(s));
  if (first_singular) *first_singular = (first == INT_MAX) ? -1 : first;
  if (first != INT_MAX) {
    set_error("Matrix " + std::to_string(first) +
              " of the batch is singular or has a zero/non-finite pivot in LU "
              "factorisation without pivoting");
    return JFB_ERR_SINGULAR;
  }
  return JFB_OK;
}
