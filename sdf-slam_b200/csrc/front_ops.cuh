// Dense building blocks shared by the front factorization kernels: the
// Newton reciprocal of a pivot and the LDL^T of a diagonal block of up to 32
// columns by four warps.
#pragma once

#include <cuda_runtime.h>

namespace sdfgpu {

/// Columns of a panel (and rows of a diagonal block).
constexpr int kPanel = 32;

/// 1 / d by Newton-Raphson iteration x <- x + x (1 - d x), seeded with the
/// hardware's approximate reciprocal (two steps square its ~2^-23 error
/// below FP64 precision). Much shorter latency than a correctly rounded
/// division on the pivot chain; the result may differ from 1.0 / d in the
/// last bit.
__device__ __forceinline__ double Recip(double d) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
  double e = fma(-d, x, 1.0);
  x = fma(x, e, x);
  e = fma(-d, x, 1.0);
  return fma(x, e, x);
}
__device__ __forceinline__ float Recip(float d) { return 1.0f / d; }

/// c += A B for an 8 x 8 block by one warp on the FP64 tensor cores: lane l
/// holds A(l / 4, l % 4), B(l % 4, l / 4) and C(l / 4, 2 (l % 4) + {0, 1}).
__device__ __forceinline__ void Dmma884(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

/// LDL^T of the w x w (w <= 32) diagonal block at B (row r, column c at
/// B[r * ld + c], lower triangle) by the block's first four warps (threads
/// 0..127): lane i owns row i, warp q owns columns 8q..8q+7 in registers. At
/// pivot j the owning warp inverts d_j (Newton reciprocal) and publishes
/// W(:, j) and L(:, j) in shared memory (two buffers, alternating with j),
/// one named barrier (id 1, 128 threads) later every warp subtracts
/// W(i, j) L(c, j) from its columns; lanes that must not change a column
/// subtract zero (a per-column branch costs more than the multiply-add).
/// Measured on B200 for a 32x32 block: 10.7k cycles against 28k for one warp
/// holding whole rows. Writes L below the diagonal and D on it; returns true
/// when a pivot is exactly zero (in the four warps).
template <typename T>
__device__ __forceinline__ bool DiagonalBlockLdlt(T* B, int ld, int w, T (*lbuf)[kPanel], T (*wbuf)[kPanel]) {
  const int lane = threadIdx.x & 31;
  const int q = threadIdx.x >> 5;
  T col[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int c = 8 * q + t;
    col[t] = (lane < w && c <= lane) ? B[lane * ld + c] : (c == lane ? T(1) : T(0));
  }
  bool zero = false;
  for (int jb = 0; jb < 4; ++jb) {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int j = 8 * jb + t;
      if (j < w) {
        const int b = j & 1;
        if (q == jb) {
          const T dj = __shfl_sync(0xffffffffu, col[t], j);
          const T wij = col[t];
          const T lij = wij * Recip(dj);
          lbuf[b][lane] = lij;
          wbuf[b][lane] = wij;
          if (lane < w && lane >= j) {
            B[lane * ld + j] = lane == j ? dj : lij;
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        zero = zero || (wbuf[b][j] == T(0));
        const T m = lane > j ? wbuf[b][lane] : T(0);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int c = 8 * q + u;
          const T mu = (c > j && c <= lane) ? m : T(0);
          col[u] = fma(-mu, lbuf[b][c], col[u]);
        }
      }
    }
  }
  return zero;
}

/// Shared-memory layout of BlockLdlt: the trapezoid column major with pitch
/// LdltPitch(R) and, behind its kp columns, a panel buffer of 8 columns with
/// pitch LdltPanelPitch(R) and kLdltDiag doubles of the diagonal block.
/// The pitches put the addresses a warp's tensor-core fragments touch at once
/// into different banks.
__host__ __device__ constexpr int LdltPitch(int R) { return (R + 13) / 16 * 16 + 2; }
__host__ __device__ constexpr int LdltPanelPitch(int R) { return (R + 11) / 16 * 16 + 4; }
constexpr int kLdltDiag = 8 * 8 + 2 * 8;  // L row major, 1 / D, D (two of them, alternating by panel)
__host__ __device__ constexpr size_t LdltSmemDoubles(int kp, int R) {
  return static_cast<size_t>(kp) * LdltPitch(R) + 8 * static_cast<size_t>(LdltPanelPitch(R)) + 2 * kLdltDiag;
}

/// Copies one element of a front into shared memory (asynchronously where no
/// conversion is needed; the destination is read after WaitElements and a
/// barrier, which order the accesses around them, so that the copies
/// themselves need not keep the compiler from moving other accesses).
__device__ __forceinline__ void LoadElement(double* dst, const double* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void LoadElement(double* dst, const float* src) { *dst = static_cast<double>(*src); }
__device__ __forceinline__ void LoadElement(float* dst, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src));
}
__device__ __forceinline__ void WaitElements() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

/// LDL^T of the 8 x 8 diagonal block at B (column major, pitch pm, lower
/// part), by one warp, every lane alike: no exchange between lanes, one
/// reciprocal, product and multiply-add per pivot on the chain. L row major,
/// then 1 / D and D into diag. Returns whether a pivot was exactly zero.
__device__ __forceinline__ bool DiagonalLdlt8(const double* B, int pm, double* diag) {
  double a[8][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int i = j; i < 8; ++i) {
      a[i][j] = B[j * pm + i];
    }
  }
  bool zero = false;
  double inv[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    zero = zero || a[t][t] == 0.0;
    inv[t] = Recip(a[t][t]);
    double w[8];
#pragma unroll
    for (int i = t + 1; i < 8; ++i) {
      w[i] = a[i][t];
      a[i][t] *= inv[t];
    }
#pragma unroll
    for (int j = t + 1; j < 8; ++j) {
#pragma unroll
      for (int i = j; i < 8; ++i) {
        a[i][j] = fma(-a[i][t], w[j], a[i][j]);
      }
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int j = 0; j < i; ++j) {
        diag[8 * i + j] = a[i][j];
      }
      diag[64 + i] = inv[i];
      diag[72 + i] = a[i][i];
    }
  }
  return zero;
}

/// C(r0.., c0..) -= W D^-1 W^T for the 8 x 8 tiles at rows r0 and columns c0,
/// c0 + 8, ... below cend (four at a time), rank 8, one warp; inv = 1 / D. The
/// eight products of an entry are summed before it is read: added to it one by
/// one, each would be rounded to its last bit (and the products would wait for
/// it: KFactorFront over a 10-frame room's levels 88 -> 81 us, a 331-pose room's
/// 207 -> 198).
__device__ __forceinline__ void LdltTiles(double* M, int pm, const double* Wp, int pp, const double* inv, int r0,
                                          int c0, int cend) {
  const int q = threadIdx.x & 3;
  const int g = (threadIdx.x & 31) >> 2;
  const double a0 = -Wp[q * pp + r0 + g] * inv[q];
  const double a1 = -Wp[(q + 4) * pp + r0 + g] * inv[q + 4];
  for (; c0 < cend; c0 += 32) {
    double p[4][2];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      p[u][0] = p[u][1] = 0.0;
      if (c0 + 8 * u < cend) {
        Dmma884(p[u], a0, Wp[q * pp + c0 + 8 * u + g]);
        Dmma884(p[u], a1, Wp[(q + 4) * pp + c0 + 8 * u + g]);
      }
    }
    double* C = M + (c0 + 2 * q) * pm + r0 + g;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (c0 + 8 * u < cend) {
        C[8 * u * pm] += p[u][0];
        C[(8 * u + 1) * pm] += p[u][1];
      }
    }
  }
}

/// LDL^T of a trapezoid of kp pivot columns and R >= kp rows (both multiples
/// of 8) in shared memory (entry (r, c) at M[c * pm + r], lower part) by the
/// whole block of Threads >= R threads; M is overwritten. Right-looking by
/// 8-column panels, two block barriers each:
///  * a thread per row below the panel's diagonal block forms the row's W =
///    A L11^-T and L = W D^-1 (28 multiply-adds);
///  * the rows and columns behind the panel take the rank-8 update on the FP64
///    tensor cores, a warp per row of 8 x 8 tiles, while warp 0 updates the
///    next diagonal block first and factors it (DiagonalLdlt8): the pivot
///    chain runs beside the update instead of before it.
/// row(r, p0, l) receives row r's L for the panel at p0; pivots(p0, diag, lane)
/// is called by warp 0 with the factored diagonal block. The caller
/// synchronises before; returns whether a pivot was exactly zero (in warp 0).
template <int Threads, typename Row, typename Pivots>
__device__ __forceinline__ bool BlockLdlt(double* M, int pm, int kp, int R, Row&& row, Pivots&& pivots) {
  const int pp = LdltPanelPitch(R);
  double* Wp = M + kp * pm;   // W = L D of the panel: (r, t) at Wp[t * pp + r]
  double* diag = Wp + 8 * pp;  // of the panel; the next panel's goes to the other half
  const int r = threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  bool zero = false;
  if (warp == 0) {
    zero = DiagonalLdlt8(M, pm, diag);
    __syncwarp();
    pivots(0, diag, lane);
  }
  __syncthreads();
  for (int p0 = 0;; p0 += 8) {
    const int c1 = p0 + 8;
    const double* dg = diag + (p0 & 8) * (kLdltDiag / 8);
    if (r >= c1 && r < R) {
      double x[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        x[t] = M[(p0 + t) * pm + r];
      }
#pragma unroll
      for (int j = 1; j < 8; ++j) {
#pragma unroll
        for (int t = 0; t < j; t += 2) {
          const double2 l = *reinterpret_cast<const double2*>(dg + 8 * j + t);
          x[j] = fma(-x[t], l.x, x[j]);
          if (t + 1 < j) {
            x[j] = fma(-x[t + 1], l.y, x[j]);
          }
        }
      }
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        Wp[t * pp + r] = x[t];
      }
#pragma unroll
      for (int t = 0; t < 8; t += 2) {
        const double2 inv = *reinterpret_cast<const double2*>(dg + 64 + t);
        x[t] *= inv.x;
        x[t + 1] *= inv.y;
      }
      row(r, p0, x);
    }
    if (c1 >= kp) {
      return zero;
    }
    __syncthreads();
    if (warp == 0) {
      double* next = diag + (c1 & 8) * (kLdltDiag / 8);
      LdltTiles(M, pm, Wp, pp, dg + 64, c1, c1, c1 + 8);
      __syncwarp();
      zero = DiagonalLdlt8(M + c1 * pm + c1, pm, next) || zero;
      __syncwarp();
      pivots(c1, next, lane);
    } else if (warp != 4) {
      // (warp 4 shares warp 0's FP64 unit and would stretch the pivot chain)
      const int w = warp < 4 ? warp : warp - 1;
      for (int r0 = c1 + 8 * w; r0 < R; r0 += Threads / 4 - 16) {
        LdltTiles(M, pm, Wp, pp, dg + 64, r0, c1, min(r0 + 8, kp));
      }
    }
    __syncthreads();
  }
}

}  // namespace sdfgpu
