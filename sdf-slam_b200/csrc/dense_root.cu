// Tiled LDL^T of the dense pose roots: one persistent launch per level.
//
// A pose root is the dense block of an instance's pose variables with no
// rows below it (the last front of the assembly tree; its LDL^T is the
// final, and for many poses the largest, step of the reference's
// factorization: src/solvers/parallel_ldlt.hpp:150-244). Factored panel by
// panel, its ceil(n / 32) panels form a chain of dependent launches. Here
// the front is cut into 64 x 64 tiles and factored right-looking as a task
// graph that every block of one launch works through:
//
//   FACTOR(k)      LDL^T of diagonal tile k (BlockLdlt), D into dvec; for
//                  k >= 1 it first does SOLVE(k, k - 1) and
//                  UPDATE(k, k, k - 1) itself (the critical path: no hand-over
//                  between those three). Once the tile is published it also
//                  forms the tile's L^-1 for the triangular solve;
//   SOLVE(i, k)    L(i, k) = A(i, k) L(k, k)^-T D(k)^-1 by 8-column block
//                  substitution, every warp on eight rows of its own
//                  (i >= k + 2);
//   UPDATE(i,j,k)  A(i, j) -= L(i, k) D(k) L(j, k)^T, j <= i (lower part;
//                  not (k + 1, k + 1, k)); a tile's early steps in groups.
//
// The products run on the FP64 tensor cores. Bound by the chain of the FACTOR
// tasks where the root is small, by the updates where it is large.
//
// Each tile (i, j) has a counter: the updates applied to it (k of them before
// step k), plus one once it is factored (i == j) or solved (i > j); FACTOR(k)
// publishes tile (k, k - 1) as solved before it goes on. A task
// waits (one thread polling with acquire loads, bounded) until its inputs'
// counters reach their values and publishes its own with a release store
// after the block's writes; updates of a tile are applied in ascending k, so
// every entry is a fixed sequence of operations and the factor is the same
// bits from run to run. Blocks take tasks from a counter in an order sorted
// by bottom level (the longest path of task weights to the end of the
// graph), which lists every task after the tasks it waits for, so a waiting
// task's inputs are already taken by running blocks: the launch cannot
// deadlock whatever number of its blocks is resident. A wait that runs out
// marks the instance (kStatusWaitTimeout) and raises the abort flag, after
// which every remaining task is skipped.
//
// Output layout (what the solve and the diagonal-block inversion read, the
// same as the panel path's): L below each 32 x 32 diagonal block in the
// lower triangle, the strictly lower part of each 32 x 32 diagonal block of L
// transposed into its upper triangle, D in dvec.
#include "dense_root.h"

#include <algorithm>
#include <mutex>

#include "engine.h"
#include "front_ops.cuh"

namespace sdfgpu {
namespace {

constexpr int kDT = kDenseTileCols;
constexpr int kDThreads = 256;
constexpr int kWarps = kDThreads / 32;
constexpr int kDLd = kDT + 4;  // pitch of a staged tile (column major): the four columns a
                               // tensor-core fragment reads at once fall into different banks
constexpr int kTLd = kDT + 1;  // pitch of the row-major tile of the inverse
constexpr int kHLd = 33;
constexpr int kTileDoubles = kDT * kDLd;
// Shared memory: a staged tile, then a region for a second tile or FACTOR's
// trapezoid, then D, 1 / D and the inverses of eight 8 x 8 diagonal blocks,
// then the second pair of tiles of a grouped update.
// The inverse of a factored tile reuses both (its rows of L in the first, three
// 32 x 33 blocks in the second).
constexpr int kRegion2 = 64 * LdltPitch(64) + 8 * LdltPanelPitch(64) + 2 * kLdltDiag;
static_assert(kRegion2 >= kTileDoubles && kRegion2 >= 3 * 32 * kHLd && kTileDoubles >= kDT * kTLd);
constexpr int kDiagInv = kWarps * 64;
constexpr size_t kDenseSmem =
    static_cast<size_t>(kTileDoubles + kRegion2 + 2 * kDT + kDiagInv + 2 * kTileDoubles) * sizeof(double);

__device__ __forceinline__ bool WaitTile(const int32_t* word, int32_t expected, const int32_t* abort,
                                         uint32_t limit) {
  for (uint32_t it = 0; it < limit; ++it) {
    int32_t v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
    if (v >= expected) {
      return true;
    }
    if (*reinterpret_cast<const volatile int32_t*>(abort) != 0) {
      return false;
    }
    __nanosleep(20);
  }
  return false;
}

__device__ __forceinline__ void PublishTile(int32_t* word, int32_t value) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(word), "r"(value) : "memory");
}

/// Stages an h x 64 tile at src (column major, ld) into shared memory, rows
/// from h on as zeros.
__device__ __forceinline__ void StageTile(double* dst, const double* src, int64_t ld, int h) {
  const int r = threadIdx.x & (kDT - 1);
  for (int c = threadIdx.x >> 6; c < kDT; c += kDThreads / kDT) {
    if (r < h) {
      LoadElement(dst + c * kDLd + r, src + c * ld + r);
    } else {
      dst[c * kDLd + r] = 0.0;
    }
  }
}

/// acc += X S Y^T for 64 x 64 tiles staged column major, S = diag(s): a warp
/// owns 16 x 32 entries, C(wr + 8 i + lane / 4, wc + 8 j + 2 (lane % 4) + e) in
/// acc[i][j][e]. between(l) runs once per four columns l: copies issued there
/// overlap the products (issued at once before them they hold the warps for a
/// third of the product's time).
template <typename Between>
__device__ __forceinline__ void TileProduct(const double* X, const double* Y, const double* s, int wr, int wc,
                                            double (&acc)[2][4][2], Between&& between) {
  const int q = threadIdx.x & 3;
  const int g = (threadIdx.x & 31) >> 2;
#pragma unroll 4
  for (int l0 = 0; l0 < kDT; l0 += 4) {
    const int l = l0 + q;
    between(l0);
    const double d = s[l];
    const double a0 = X[l * kDLd + wr + g] * d;
    const double a1 = X[l * kDLd + wr + 8 + g] * d;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double b = Y[l * kDLd + wc + 8 * j + g];
      Dmma884(acc[0][j], a0, b);
      Dmma884(acc[1][j], a1, b);
    }
  }
}

/// Stages the unit lower triangle L of factored diagonal tile k (of full
/// width), D and 1 / D.
__device__ __forceinline__ void StageFactor(const SupernodeRec& S, const double* Fs, int k, const DenseArgs& A,
                                            double* L, double* d) {
  const int64_t F = S.F;
  const int c0 = k * kDT;
  const double* dv = A.dvec + S.first_col + c0;
  // within the 32 x 32 diagonal blocks L is stored transposed in the upper
  // triangle: threads along the contiguous index
  const int x = threadIdx.x & 31;
  for (int y = threadIdx.x >> 5; y < kDT; y += kWarps) {
    const int b = y & 32;
    if (b + x < y) {
      LoadElement(L + (b + x) * kDLd + y, Fs + (c0 + y) * F + c0 + b + x);  // L(y, b + x)
    }
    if (y < 32) {
      LoadElement(L + y * kDLd + 32 + x, Fs + (c0 + y) * F + c0 + 32 + x);  // L(32 + x, y)
    }
  }
  if (threadIdx.x < kDT) {
    const double v = __ldcg(dv + threadIdx.x);
    d[threadIdx.x] = v;
    d[kDT + threadIdx.x] = Recip(v);
  }
}

/// The A fragments (columns 4 h + lane % 4, h = 0, 1) of an 8 x 8 block held
/// as a C fragment (columns 2 (lane % 4) + {0, 1}): an exchange among the four
/// lanes of a row.
__device__ __forceinline__ void BlockAsA(const double (&c)[2], double (&a)[2]) {
  const int lane = threadIdx.x & 31;
  const int from = (lane & ~3) + ((lane & 3) >> 1);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double even = __shfl_sync(0xffffffffu, c[0], from + 2 * h);
    const double odd = __shfl_sync(0xffffffffu, c[1], from + 2 * h);
    a[h] = (lane & 1) != 0 ? odd : even;
  }
}

/// Column blocks P.. of SubstituteRows (a template per block: every register
/// index is a constant): W_P = (A_P + C_P) L_PP^-T, then the later blocks' sums C_p
/// less W_P L_pP^T (summed on their own, see LdltTiles; X: the lane's entries of A).
template <int P>
__device__ __forceinline__ void SubstituteFrom(double (&C)[8][2], const double* X, const double* L,
                                               const double* minv) {
  if constexpr (P < 8) {
    const int q = threadIdx.x & 3;
    const int g = (threadIdx.x & 31) >> 2;
    C[P][0] += X[8 * P * kDLd];
    C[P][1] += X[(8 * P + 1) * kDLd];
    double a[2];
    BlockAsA(C[P], a);
    // B(k, n) = L_PP^-1(n, k)
    double w[2] = {0.0, 0.0};
    Dmma884(w, a[0], minv[64 * P + 8 * q + g]);
    Dmma884(w, a[1], minv[64 * P + 8 * (q + 4) + g]);
    C[P][0] = w[0];
    C[P][1] = w[1];
    if constexpr (P < 7) {
      BlockAsA(w, a);
      const double* L0 = L + (8 * P + q) * kDLd + g;
#pragma unroll
      for (int p = P + 1; p < 8; ++p) {
        Dmma884(C[p], -a[0], L0[8 * p]);
        Dmma884(C[p], -a[1], L0[4 * kDLd + 8 * p]);
      }
    }
    SubstituteFrom<P + 1>(C, X, L, minv);
  }
}

/// W = A L^-T in place for the 64 x 64 tile A staged at X (column major) and
/// the staged unit lower triangle L, eight rows per warp with no exchange
/// between warps; their sums stay in registers as C fragments (the inverses of
/// the 8 x 8 diagonal blocks, warp p the p-th, go to minv). L(i, k) = W D^-1 also
/// goes to dst (rows below h). Starts and ends with a block barrier.
__device__ __forceinline__ void SubstituteRows(double* X, const double* L, double* minv, const double* dinv,
                                               double* dst, int64_t ld, int h) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int q = lane & 3;
  const int g = lane >> 2;
  __syncthreads();
  if (lane < 8) {
    // column `lane` of the inverse of diagonal block `warp`: (i, lane) at
    // minv[64 * warp + 8 * lane + i]
    const double* B = L + 8 * warp * kDLd + 8 * warp;
    double m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      m[i] = i == lane ? 1.0 : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 7; ++j) {
#pragma unroll
      for (int i = j + 1; i < 8; ++i) {
        m[i] = fma(-B[j * kDLd + i], m[j], m[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      minv[64 * warp + 8 * lane + i] = m[i];
    }
  }
  const int r = 8 * warp + g;
  double C[8][2] = {};
  __syncthreads();
  SubstituteFrom<0>(C, X + 2 * q * kDLd + r, L, minv);
#pragma unroll
  for (int p = 0; p < 8; ++p) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = 8 * p + 2 * q + e;
      X[c * kDLd + r] = C[p][e];
      if (r < h) {
        dst[c * ld + r] = C[p][e] * dinv[c];
      }
    }
  }
  __syncthreads();
}

/// Columns c of M = L^-1 for the unit lower 32 x 32 triangle at T
/// (row-major, ld kTLd, L(i, j) = T[i][j] for i > j), one warp: lane c
/// solves L m = e_c by forward substitution (unrolled: a loop over the
/// pivots with the register vector indexed at run time measured three
/// times slower). M(i, c) -> Mo[i * kHLd + c].
__device__ __forceinline__ void InvertUnitLower32(const double* T, double* Mo) {
  const int lane = threadIdx.x & 31;
  double m[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    m[i] = i == lane ? 1.0 : 0.0;
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) {
#pragma unroll
    for (int i = j + 1; i < 32; ++i) {
      m[i] = fma(-T[i * kTLd + j], m[j], m[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    Mo[i * kHLd + lane] = m[i];
  }
}

/// L^-1 = [M1 0; -M2 L21 M1  M2] of a factored tile whose L stands row major
/// in T (the identity beyond w), column major 64 x 64 into the workspace: the
/// triangular solve's 64-row panels multiply by it. H: three 32 x 33 blocks.
__device__ void InvertTile(double (*T)[kTLd], double* H, double* Mo) {
  double* M1 = H;
  double* Y = M1 + 32 * kHLd;
  double* M2 = Y + 32 * kHLd;
  const int tid = threadIdx.x;
  if (tid < 32) {
    InvertUnitLower32(&T[0][0], M1);
  } else if (tid >= 64 && tid < 96) {
    InvertUnitLower32(&T[32][32], M2);
  }
  __syncthreads();
  const int r = tid & 31;
  const int cb = tid >> 5;
  // Y = L21 M1
  double p[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int l = 0; l < 32; ++l) {
    const double x = T[32 + r][l];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      p[q] = fma(x, M1[l * kHLd + cb + 8 * q], p[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    Y[r * kHLd + cb + 8 * q] = p[q];
  }
  __syncthreads();
  double m[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int l = 0; l < 32; ++l) {
    const double x = M2[r * kHLd + l];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      m[q] = fma(x, Y[l * kHLd + cb + 8 * q], m[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int c = cb + 8 * q;
    Mo[static_cast<int64_t>(c) * kDT + 32 + r] = -m[q];
    Mo[static_cast<int64_t>(c) * kDT + r] = M1[r * kHLd + c];
    Mo[static_cast<int64_t>(32 + c) * kDT + 32 + r] = M2[r * kHLd + c];
    Mo[static_cast<int64_t>(32 + c) * kDT + r] = 0.0;
  }
}

/// SOLVE(i, k): L(i, k) = A(i, k) L(k, k)^-T D(k)^-1.
__device__ void SolveTile(const DeviceView& V, const SupernodeRec& S, int i, int k, const DenseArgs& A,
                          double* sm) {
  const int64_t F = S.F;
  double* Fs = V.fronts + S.front_off;
  double* tile = Fs + static_cast<int64_t>(k) * kDT * F + i * kDT;
  const int h = min(kDT, S.ncols - i * kDT);
  double* X = sm;
  double* L = sm + kTileDoubles;
  double* d = L + kRegion2;
  StageTile(X, tile, F, h);
  StageFactor(S, Fs, k, A, L, d);
  WaitElements();
  SubstituteRows(X, L, d + 2 * kDT, d + kDT, tile, F, h);
}

/// The entries of tile (i, j) that a thread owns in TileProduct's layout,
/// read before the product so that their latency hides behind it, and written
/// back less the product (lower part).
struct OwnedTile {
  double* base;
  int64_t ld;
  int r0, c0, h, w;
  bool diagonal;
  double old[2][4][2];
  __device__ __forceinline__ bool In(int i, int j, int e) const {
    const int r = r0 + 8 * i;
    const int c = c0 + 8 * j + e;
    return r < h && c < w && (!diagonal || r >= c);
  }
  __device__ __forceinline__ void Read(const SupernodeRec& S, double* Fs, int ti, int tj, int wr, int wc) {
    const int lane = threadIdx.x & 31;
    ld = S.F;
    base = Fs + static_cast<int64_t>(tj) * kDT * ld + ti * kDT;
    r0 = wr + (lane >> 2);
    c0 = wc + 2 * (lane & 3);
    h = min(kDT, S.ncols - ti * kDT);
    w = min(kDT, S.ncols - tj * kDT);
    diagonal = ti == tj;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          old[i][j][e] = In(i, j, e) ? __ldcg(base + (c0 + 8 * j + e) * ld + r0 + 8 * i) : 0.0;
        }
      }
    }
  }
  __device__ __forceinline__ void WriteLess(const double (&acc)[2][4][2]) const {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (In(i, j, e)) {
            base[(c0 + 8 * j + e) * ld + r0 + 8 * i] = old[i][j][e] - acc[i][j][e];
          }
        }
      }
    }
  }
};

/// UPDATE(i, j, [k, k + len)): A(i, j) -= sum of L(i, l) D(l) L(j, l)^T over the
/// steps l, lower part; the next step's tiles are staged while the current
/// ones are multiplied.
__device__ void UpdateTile(const DeviceView& V, const SupernodeRec& S, int i, int j, int k, int len,
                           const DenseArgs& A, double* sm) {
  const int64_t F = S.F;
  double* Fs = V.fronts + S.front_off;
  // two pairs of staged tiles and two copies of D
  // (offsets, not an array of pointers: those would be generic addresses)
  constexpr int kSecond = kTileDoubles + kRegion2 + 2 * kDT + kDiagInv;
  double* const d = sm + kTileDoubles + kRegion2;
  const int hi = min(kDT, S.ncols - i * kDT);
  // four columns from c0 of step l's tiles (a thread stages one row of one)
  const int r = threadIdx.x & (kDT - 1);
  auto stage = [&](int l, int c0) {
    const int c = c0 + static_cast<int>(threadIdx.x >> 6);
    const double* col = Fs + (static_cast<int64_t>(k + l) * kDT + c) * F + r;
    double* x = sm + (l & 1) * kSecond + c * kDLd + r;
    if (r < hi) {
      LoadElement(x, col + i * kDT);
    } else {
      *x = 0.0;
    }
    if (i != j) {
      LoadElement(x + kTileDoubles, col + j * kDT);  // (j < i: a full tile)
    }
    if (c0 == 0 && threadIdx.x < kDT) {
      LoadElement(d + (l & 1) * kDT + threadIdx.x, A.dvec + S.first_col + (k + l) * kDT + threadIdx.x);
    }
  };
  for (int c0 = 0; c0 < kDT; c0 += 4) {
    stage(0, c0);
  }
  const int warp = threadIdx.x >> 5;
  const int wr = 16 * (warp & 3);
  const int wc = 32 * (warp >> 2);
  OwnedTile C;
  C.Read(S, Fs, i, j, wr, wc);
  const bool mine = i != j || wc < wr + 16;
  double acc[2][4][2] = {};
  for (int l = 0; l < len; ++l) {
    WaitElements();
    __syncthreads();
    const bool more = l + 1 < len;
    if (mine) {
      const double* X = sm + (l & 1) * kSecond;
      TileProduct(X, X + (i != j ? kTileDoubles : 0), d + (l & 1) * kDT, wr, wc, acc, [&](int c0) {
        if (more) {
          stage(l + 1, c0);
        }
      });
    } else if (more) {
      for (int c0 = 0; c0 < kDT; c0 += 4) {
        stage(l + 1, c0);
      }
    }
  }
  if (mine) {
    C.WriteLess(acc);
  }
}

/// FACTOR(k). For k >= 1 the task first does the two steps that feed it:
/// SOLVE(k, k - 1) (published as soon as it is written, for the other
/// updates of step k - 1) and UPDATE(k, k, k - 1), whose result goes
/// straight into the shared-memory trapezoid instead of the front. Returns
/// false when a wait ran out.
__device__ bool FactorTask(const DeviceView& V, const SupernodeRec& S, int k, int nt, const DenseArgs& A,
                           int32_t* cnt, double* sm, int* factored) {
  const int64_t F = S.F;
  double* Fs = V.fronts + S.front_off;
  const int c0 = k * kDT;
  const int w = min(kDT, S.ncols - c0);
  const int kp = (w + 7) & ~7;
  double* X = sm;
  double* M = sm + kTileDoubles;
  double* d = M + kRegion2;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int pm = LdltPitch(kp);
  // the lower triangle's 36 blocks of 8 x 8, five or four per warp: warps v and
  // v + 4 share the block rows v (v + 1 blocks) and 7 - v (8 - v blocks)
  const int v = warp & 3;
  const int b0 = warp < 4 ? 0 : 5;
  const int nb = warp < 4 ? 5 : 4;
  auto block = [&](int x, int* br, int* bc) {
    const int e = b0 + x;  // 0..8: row 7 - v first
    *br = e < 8 - v ? 7 - v : v;
    *bc = e < 8 - v ? e : e - (8 - v);
  };
  const int q = lane & 3;
  const int g = lane >> 2;
  double old[5][2];
  double acc[5][2] = {};
#pragma unroll
  for (int x = 0; x < 5; ++x) {
    int br;
    int bc;
    block(x, &br, &bc);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 8 * br + g;
      const int c = 8 * bc + 2 * q + e;
      old[x][e] = x < nb && r < w && r >= c ? __ldcg(Fs + (c0 + c) * F + c0 + r) : (r == c ? 1.0 : 0.0);
    }
  }
  if (k > 0) {
    // the tile to solve and the one to update wait for the earlier steps only:
    // they are on their way while tile k - 1 is still being factored
    double* tile = Fs + static_cast<int64_t>(k - 1) * kDT * F + c0;
    StageTile(X, tile, F, w);
    if (tid == 0) {
      *factored = WaitTile(cnt + (k - 1) * nt + (k - 1), k, A.abort, A.wait_limit) ? 1 : 0;
    }
    __syncthreads();
    if (*factored == 0) {
      WaitElements();
      return false;
    }
    StageFactor(S, Fs, k - 1, A, M, d);
    WaitElements();
    SubstituteRows(X, M, d + 2 * kDT, d + kDT, tile, F, w);
    if (tid == 0) {
      __threadfence();
      PublishTile(cnt + k * nt + (k - 1), k);
    }
    int br[5];
    int bc[5];
#pragma unroll
    for (int x = 0; x < 5; ++x) {
      block(x, &br[x], &bc[x]);
    }
#pragma unroll 4
    for (int l = q; l < kDT; l += 4) {
      const double* col = X + l * kDLd + g;
      const double inv = d[kDT + l];
#pragma unroll
      for (int x = 0; x < 5; ++x) {
        if (x < nb) {
          Dmma884(acc[x], col[8 * br[x]] * inv, col[8 * bc[x]]);
        }
      }
    }
  }
  __syncthreads();
  // the updated tile (the identity on the padding pivots)
#pragma unroll
  for (int x = 0; x < 5; ++x) {
    int br;
    int bc;
    block(x, &br, &bc);
    if (x < nb && 8 * br < kp) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        M[(8 * bc + 2 * q + e) * pm + 8 * br + g] = old[x][e] - acc[x][e];
      }
    }
  }
  // rows of L of the tile, row major, for the inverse (the identity beyond w)
  double(*T)[kTLd] = reinterpret_cast<double(*)[kTLd]>(X);
  for (int e = tid; e < kDT * kDT; e += kDThreads) {
    T[e >> 6][e & 63] = 0.0;
  }
  __syncthreads();
  const bool zero = BlockLdlt<kDThreads>(
      M, pm, kp, kp,
      [&](int r, int p0, const double(&l)[8]) {
        if (r < w) {
          // within a 32 x 32 diagonal block transposed into its upper triangle
          const bool upper = (r ^ p0) < 32;
          double* dst = upper ? Fs + (c0 + r) * F + c0 + p0 : Fs + (c0 + p0) * F + c0 + r;
          const int64_t step = upper ? 1 : F;
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            dst[t * step] = l[t];
            T[r][p0 + t] = l[t];
          }
        }
      },
      [&](int p0, const double* diag, int lane_) {
        const int i = lane_ >> 2;
        if (p0 + i < w) {
          for (int t = lane_ & 3; t < i; t += 4) {
            Fs[(c0 + p0 + i) * F + c0 + p0 + t] = diag[8 * i + t];
            T[p0 + i][p0 + t] = diag[8 * i + t];
          }
          if ((lane_ & 3) == 0) {
            A.dvec[S.first_col + c0 + p0 + i] = diag[72 + i];
          }
        }
      });
  if (zero && lane == 0) {
    atomicOr(V.status + S.instance, kStatusZeroPivot);
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    PublishTile(cnt + k * nt + k, k + 1);
  }
  InvertTile(T, M, A.inv + S.dense_inv + static_cast<int64_t>(k) * kDT * kDT);
  return true;
}

/// Bound by the chain of FACTOR steps (about 14 us each behind one another) and,
/// in the largest roots, by the updates' products and staging. One block per SM:
/// the registers of the product and substitution fragments. Measured on B200
/// against 32-column halves by four warps with the inverse on the chain and one
/// step per UPDATE: a step of the chain 35 -> 14 us; 225 columns 140 -> 64 us, 990
/// columns 550 -> 240, 2,727 columns 1650 -> 839, roots of a 32-instance batch 330 ->
/// 145.
__global__ void __launch_bounds__(kDThreads, 1) KDenseRoot(DeviceView V, DenseArgs A) {
  extern __shared__ double dense_sm[];
  __shared__ int task;
  __shared__ int go;
  __shared__ int factored;  // FACTOR's own wait
  const int tid = threadIdx.x;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      task = atomicAdd(A.claim, 1);
    }
    __syncthreads();
    const int64_t t = task;
    if (t >= A.count) {
      return;
    }
    const int32_t* q = A.tasks + 4 * t;
    const int s = q[0];
    const int i = q[1];
    const int j = q[2];
    const int k = q[3] & 0xffff;
    const int len = (q[3] >> 16) + 1;
    const SupernodeRec S = V.sn[s];
    if (V.active[S.instance] == 0) {
      continue;
    }
    const int nt = (S.ncols + kDT - 1) / kDT;
    int32_t* cnt = A.cnt + S.dense_cnt;
    if (tid == 0) {
      bool ok;
      if (i == k) {
        // FACTOR(k) with SOLVE(k, k - 1) and UPDATE(k, k, k - 1) folded in; it
        // waits for tile (k - 1, k - 1) itself
        ok = k == 0 || (WaitTile(cnt + k * nt + (k - 1), k - 1, A.abort, A.wait_limit) &&
                        WaitTile(cnt + k * nt + k, k - 1, A.abort, A.wait_limit));
      } else if (j == k) {
        ok = WaitTile(cnt + k * nt + k, k + 1, A.abort, A.wait_limit) &&
             WaitTile(cnt + i * nt + k, k, A.abort, A.wait_limit);
      } else {
        // (tile (i, l) is solved after (i, l - 1): the last step's are enough)
        const int l = k + len - 1;
        ok = WaitTile(cnt + i * nt + l, l + 1, A.abort, A.wait_limit) &&
             (i == j || WaitTile(cnt + j * nt + l, l + 1, A.abort, A.wait_limit)) &&
             WaitTile(cnt + i * nt + j, k, A.abort, A.wait_limit);
      }
      if (!ok) {
        atomicOr(V.status + S.instance, kStatusWaitTimeout);
        atomicExch(A.abort, 1);
      }
      go = ok ? 1 : 0;
    }
    __syncthreads();
    if (go == 0) {
      continue;
    }
    if (i == k) {
      // (publishes its tile itself, before the inverse)
      if (!FactorTask(V, S, k, nt, A, cnt, dense_sm, &factored) && tid == 0) {
        atomicOr(V.status + S.instance, kStatusWaitTimeout);
        atomicExch(A.abort, 1);
      }
      continue;
    }
    if (j == k) {
      SolveTile(V, S, i, k, A, dense_sm);
    } else {
      UpdateTile(V, S, i, j, k, len, A, dense_sm);
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      PublishTile(cnt + i * nt + j, k + len);
    }
  }
}

}  // namespace

int LaunchDenseRoots(const DeviceView& V, const DenseArgs& args, cudaStream_t stream) {
  if (args.count <= 0) {
    return 0;
  }
  static std::mutex mu;
  static int blocks_per_sm[64] = {};
  static int sms[64] = {};
  int dev = 0;
  CudaCheck(cudaGetDevice(&dev), "device");
  if (dev < 0 || dev >= 64) {
    Fail(SDFGPU_ERR_CUDA, "device index out of range");
  }
  const std::lock_guard<std::mutex> lock(mu);
  if (blocks_per_sm[dev] == 0) {
    CudaCheck(cudaFuncSetAttribute(KDenseRoot, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(kDenseSmem)),
              "dense root smem attr");
    int per_sm = 0;
    CudaCheck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KDenseRoot, kDThreads, kDenseSmem),
              "dense root occupancy");
    CudaCheck(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev), "sm count");
    blocks_per_sm[dev] = per_sm > 0 ? per_sm : 1;
  }
  const int64_t grid = std::min<int64_t>(args.count, static_cast<int64_t>(blocks_per_sm[dev]) * sms[dev]);
  KDenseRoot<<<static_cast<unsigned>(grid), kDThreads, kDenseSmem, stream>>>(V, args);
  CudaCheck(cudaGetLastError(), "dense root launch");
  return 1;
}

}  // namespace sdfgpu
