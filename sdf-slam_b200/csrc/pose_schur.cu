// Pose Schur complement: root -= sum over the grid fronts s of
// L_s D_s L_s^T, L_s the pose rows of front s (its rows in the pose root).
//
// A grid front couples its pivots to the poses that see them: in a 910-pose
// office 340 rows below a leaf's 42 pivots, 310 of them pose rows. Carried up
// the assembly tree, the pose-pose part of every update matrix is added into
// the parent and again into its parent up to the root (164 of 196 million
// update entries per factorization, 24 bytes each); but a pose row is a pivot
// only in the root, so the products can be summed there at once. Each block
// owns one 64 x 64 tile of the root (or a part of its fronts) and takes the
// fronts that have rows in both of the tile's row blocks in a fixed order:
// accumulators stay in registers, the root's entries are read and written
// once, and no two blocks add into one entry, so the sums are the same from
// run to run.
//
// A front's rows of one block are consecutive in the front (rows ascend) but
// need not cover it: a 64-bit mask per (front, block) places them, absent rows
// are staged as zeros, and the 8 x 8 products whose rows or columns are all
// absent are skipped. The products run on the FP64 tensor cores
// (mma.m8n8k4.f64: on B200 36.6 TF/s measured from four warps per SM on,
// against 28 to 33 TF/s for independent DFMA chains, and fewer shared-memory
// reads per multiply-add than 4 x 4 register tiles). FP32 fronts of a mixed
// solve are converted when they are read: their pose products are accumulated
// in FP64 like the root itself.
#include "pose_schur.h"

#include <mutex>

#include "engine.h"
#include "front_ops.cuh"

namespace sdfgpu {
namespace {

constexpr int kT = kPoseTile;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kK = 16;         // pivots per stage
constexpr int kLd = kT + 4;    // doubles per staged pivot: the four pivots a warp reads at once
                               // fall into different banks
constexpr int kStages = 3;
constexpr int kScan = kThreads;  // fronts looked at per scan
constexpr int kBlocksPerSm = 3;
constexpr int kChildScan = 16;  // children looked at per scan

/// One front of the current scan that has rows in both blocks.
struct Match {
  int64_t base_a, base_b;  // first element of the front's rows of blocks I and J
  uint64_t ma, mb;         // the rows' positions in the blocks
  int32_t F;
  int32_t k;
  int32_t first;           // first pivot column (D)
  int32_t leaf;            // a child: without an update matrix
  int32_t update;          // a child: front column of the first of its columns of block J
  uint32_t groups;         // 8-row groups with a row present: block I, then block J
};

template <typename T>
struct Smem {
  T a[kStages][kK][kLd];
  T b[kStages][kK][kLd];
  double d[kStages][kK];
  Match match[kScan];
  int warp_count[kWarps];
  int last;
};

/// KChildSchur: what the products are subtracted from besides, sixteen entries
/// per thread.
struct ChildSmem {
  Smem<double> stage;
  double sum[16][kThreads];
};

/// Asynchronous copy of one element; size 0 writes zero and reads nothing.
__device__ __forceinline__ void CopyZfill(double* dst, const double* src, int size) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(size) : "memory");
}
__device__ __forceinline__ void CopyZfill(float* dst, const float* src, int size) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(size) : "memory");
}

template <typename T>
__device__ __forceinline__ const T* Fronts(const DeviceView& V);
template <>
__device__ __forceinline__ const double* Fronts<double>(const DeviceView& V) {
  return V.fronts;
}
template <>
__device__ __forceinline__ const float* Fronts<float>(const DeviceView& V) {
  return V.fronts32;
}

/// Bits (one per 8-row group) of the groups of `m` with a row present.
__device__ __forceinline__ uint32_t Groups(uint64_t m) {
  uint32_t g = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    g |= ((m >> (8 * q)) & 0xffull) != 0 ? 1u << q : 0u;
  }
  return g;
}

/// acc += sum over the matches of A D B^T, A and B the match's rows of the
/// tile's two blocks at their positions: stages of kK pivots by asynchronous
/// copies, kStages in flight, one match's stages behind another's. wr, wc: the
/// warp's first row and column of the tile; matches > 0, sm.match behind a
/// barrier. started(): called once the first stages are on their way.
template <typename T, typename Started>
__device__ __forceinline__ void MultiplyMatches(Smem<T>& sm, int matches, const T* fronts, const double* dvec,
                                                bool diagonal, int wr, int wc, double (&acc)[2][4][2], Started started) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  // staging: the first four warps copy block I's rows, the others block J's;
  // a thread copies row pos of half a stage's pivots
  const bool side = tid >= kThreads / 2;
  const int pos = tid & (kT - 1);
  const int l0 = ((tid >> 6) & 1) * (kK / 2);
  const uint64_t below = (uint64_t{1} << pos) - 1;
  T* const dst = side ? &sm.b[0][l0][pos] : &sm.a[0][l0][pos];
  // producer position: match pm, `left` of its pivots still to stage; the
  // thread's sources advance by one stage (or to the next match) per issue
  int pm = -1;
  int left = 0;
  const T* src = nullptr;
  const double* src_d = nullptr;
  int64_t F = 0;
  int size = 0;
  auto issue = [&](int stage) {
    if (left <= 0 && pm < matches) {
      if (++pm < matches) {
        const Match& m = sm.match[pm];
        const uint64_t mask = side ? m.mb : m.ma;
        left = m.k;
        F = m.F;
        src = fronts + (side ? m.base_b : m.base_a) + l0 * F + __popcll(mask & below);
        // absent rows are staged as zeros
        size = ((mask >> pos) & 1) != 0 ? static_cast<int>(sizeof(T)) : 0;
        src_d = dvec + m.first + tid;
      }
    }
    if (left > 0) {
      if (!(side && diagonal)) {
        T* to = dst + stage * (kK * kLd);
        if (left >= kK) {
#pragma unroll
          for (int l = 0; l < kK / 2; ++l) {
            CopyZfill(to + l * kLd, src + l * F, size);
          }
        } else {
          // pivots past the last are staged as zeros
#pragma unroll
          for (int l = 0; l < kK / 2; ++l) {
            CopyZfill(to + l * kLd, src + l * F, l0 + l < left ? size : 0);
          }
        }
        src += kK * F;
      }
      if (tid < kK) {
        CopyZfill(&sm.d[stage][tid], src_d, tid < left ? 8 : 0);
        src_d += kK;
      }
      left -= kK;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    issue(s);
  }
  started();
  int stage = 0;
  int ahead = kStages - 1;
  for (int cm = 0; cm < matches; ++cm) {
    const int k = sm.match[cm].k;
    const uint32_t ga = (sm.match[cm].groups >> (wr / 8)) & 3u;
    const uint32_t gb = (sm.match[cm].groups >> (8 + wc / 8)) & 15u;
    // on the diagonal tile only the lower part is used
    const bool work = ga != 0 && gb != 0 && !(diagonal && wc >= wr + 16);
    for (int ck = 0; ck < k; ck += kK) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncthreads();
      issue(ahead);
      ahead = ahead + 1 == kStages ? 0 : ahead + 1;
      if (work) {
        const T* as = &sm.a[stage][lane & 3][wr + (lane >> 2)];
        const T* bs = (diagonal ? &sm.a[stage][lane & 3][0] : &sm.b[stage][lane & 3][0]) + wc + (lane >> 2);
        double a0[kK / 4];
        double a1[kK / 4];
#pragma unroll
        for (int ks = 0; ks < kK / 4; ++ks) {
          const double d = sm.d[stage][4 * ks + (lane & 3)];
          a0[ks] = static_cast<double>(as[4 * ks * kLd]) * d;
          a1[ks] = static_cast<double>(as[4 * ks * kLd + 8]) * d;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if ((gb >> j) & 1u) {
            double bv[kK / 4];
#pragma unroll
            for (int ks = 0; ks < kK / 4; ++ks) {
              bv[ks] = static_cast<double>(bs[4 * ks * kLd + 8 * j]);
            }
            if (ga == 3u) {
#pragma unroll
              for (int ks = 0; ks < kK / 4; ++ks) {
                Dmma884(acc[0][j], a0[ks], bv[ks]);
                Dmma884(acc[1][j], a1[ks], bv[ks]);
              }
            } else if (ga == 1u) {
#pragma unroll
              for (int ks = 0; ks < kK / 4; ++ks) {
                Dmma884(acc[0][j], a0[ks], bv[ks]);
              }
            } else {
#pragma unroll
              for (int ks = 0; ks < kK / 4; ++ks) {
                Dmma884(acc[1][j], a1[ks], bv[ks]);
              }
            }
          }
        }
      }
      stage = stage + 1 == kStages ? 0 : stage + 1;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
}

/// Bound by the FP64 tensor cores and the barriers between stages, three
/// blocks per SM. A warp owns 16 x 32 entries of the tile. Measured on B200
/// (910-pose office, 1,672 tasks): 1.31 ms against 1.63 ms for the same products
/// on the packed rows with a shared-memory tile (the scatter) and 1.43 ms for
/// warps mapped without the row shuffle; 1.02 ms in an iteration as it is now
/// (1,668 tasks), tensor cores busy 42 %. The whole Schur
/// phase with its parents' updates went from 2.72 to 2.10 ms, clearing the
/// (now 0.5 instead of 3.5 GB of) fronts from 0.29 to 0.07 ms.
template <typename T>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm) KPoseSchur(DeviceView V, PoseSchurArgs A) {
  extern __shared__ __align__(16) unsigned char pose_smem[];
  Smem<T>& sm = *reinterpret_cast<Smem<T>*>(pose_smem);
  const PoseTask t = A.tasks[blockIdx.x];
  const SupernodeRec R = V.sn[t.root];
  const int inst = R.instance;
  const bool mixed = V.fronts32 != nullptr && V.inst[inst].mixed != 0;
  if (V.active[inst] == 0 || mixed != (sizeof(T) == sizeof(float))) {
    return;
  }
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const T* fronts = Fronts<T>(V);
  // the warp's rows and columns of the tile: warps w and w + 4, which share an
  // SM sub-partition, take different row quarters, so that fronts with rows
  // in a part of the block still occupy all four tensor cores
  const int wr = 16 * ((warp + 2 * (warp >> 2)) & 3);
  const int wc = 32 * (warp >> 2);
  double acc[2][4][2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[i][j][0] = acc[i][j][1] = 0.0;
    }
  }
  const uint64_t* mask_i = A.mask + t.mask + static_cast<int64_t>(t.I) * t.len;
  const uint64_t* mask_j = A.mask + t.mask + static_cast<int64_t>(t.J) * t.len;
  const int32_t* start_i = A.start + t.mask + static_cast<int64_t>(t.I) * t.len;
  const int32_t* start_j = A.start + t.mask + static_cast<int64_t>(t.J) * t.len;
  const bool diagonal = t.I == t.J;
  for (int q0 = t.q0; q0 < t.q1; q0 += kScan) {
    // the fronts of this scan with rows in both blocks, in list order
    const int q = q0 + tid;
    uint64_t ma = 0;
    uint64_t mb = 0;
    if (q < t.q1) {
      ma = mask_i[q];
      mb = mask_j[q];
    }
    const bool hit = ma != 0 && mb != 0;
    const unsigned votes = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) {
      sm.warp_count[warp] = __popc(votes);
    }
    __syncthreads();
    int at = __popc(votes & ((1u << lane) - 1u));
    int matches = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      at += w < warp ? sm.warp_count[w] : 0;
      matches += sm.warp_count[w];
    }
    if (hit) {
      const SupernodeRec S = V.sn[A.fronts[t.list + q]];
      Match& m = sm.match[at];
      m.base_a = S.front_off + S.ncols + start_i[q];
      m.base_b = S.front_off + S.ncols + start_j[q];
      m.ma = ma;
      m.mb = mb;
      m.F = S.F;
      m.k = S.ncols;
      m.first = S.first_col;
      m.groups = Groups(ma) | (Groups(mb) << 8);
    }
    __syncthreads();
    if (matches == 0) {
      continue;
    }
    MultiplyMatches<T>(sm, matches, fronts, A.dvec, diagonal, wr, wc, acc, [] {});
  }
  if (t.parts > 1) {
    // the part's sums into its slot, thread by thread; the last part to
    // arrive adds all of them in part order
    double* out = A.parts + static_cast<int64_t>(t.slot + t.part) * kT * kT + tid;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      __stcg(out + e * kThreads, acc[e >> 3][(e >> 1) & 3][e & 1]);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      sm.last = atomicAdd(A.counters + t.counter, 1) == t.parts - 1 ? 1 : 0;
    }
    __syncthreads();
    if (sm.last == 0) {
      return;
    }
    __threadfence();
    if (tid == 0) {
      A.counters[t.counter] = 0;
    }
    const double* in = A.parts + static_cast<int64_t>(t.slot) * kT * kT + tid;
    double s[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      s[e] = 0.0;
    }
    for (int p = 0; p < t.parts; ++p) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        s[e] += __ldcg(in + static_cast<int64_t>(p) * kT * kT + e * kThreads);
      }
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      acc[e >> 3][(e >> 1) & 3][e & 1] = s[e];
    }
  }
  const int n = R.ncols;
  const int64_t ld = R.F;
  double* root = V.fronts + R.front_off;
  const int r0 = t.I * kT + wr + (lane >> 2);
  const int c0 = t.J * kT + wc + 2 * (lane & 3);
  // all reads before the writes (the entries are distinct)
  double old[2][4][2];
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int r = r0 + 8 * (e >> 3);
    const int c = c0 + 8 * ((e >> 1) & 3) + (e & 1);
    old[e >> 3][(e >> 1) & 3][e & 1] = r < n && c <= r ? root[c * ld + r] : 0.0;
  }
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int r = r0 + 8 * (e >> 3);
    const int c = c0 + 8 * ((e >> 1) & 3) + (e & 1);
    if (r < n && c <= r) {
      root[c * ld + r] = old[e >> 3][(e >> 1) & 3][e & 1] - acc[e >> 3][(e >> 1) & 3][e & 1];
    }
  }
}

/// Schur complements of a level's children, pulled into their parents' fronts:
/// a block owns one 64 x 64 tile (I, J) of a parent's stored columns and takes
/// its children with rows in both blocks, in order: the tile becomes its
/// assembled values (pivot columns; the others hold nothing yet) plus the
/// children's update matrices minus L D L^T of their rows. One launch per
/// level, one read and one write per entry and no clearing of the trailing
/// columns; pushed by the children, two that share a parent needed a launch
/// each (three times the reads, and half the launches nearly empty). Bound by
/// the chain from the task to the store (task, entries, values, products) and,
/// at the wide levels, by staging. Two blocks per SM, which keep their registers.
/// The products are summed on their own (the entry and the update matrices wait in
/// shared memory): added to the entry one by one, each is rounded to the entry's
/// last bit, which made the step's error against its exact value 1.2 to 1.5 times
/// that of products summed first.
/// Measured on B200, the factorization with a pushing launch per sibling -> this:
/// 10-frame room 158 -> 105 us, 76-frame floor plan 430 -> 345, 331-pose room 1095
/// -> 985 (of which the sums on their own, here and in LdltTiles, 117 -> 105, 358
/// -> 345, 1007 -> 985), 32 instances 2070 -> 1842.
__global__ void __launch_bounds__(kThreads, 2) KChildSchur(DeviceView V, const ChildTask* tasks,
                                                                      const ChildEntry* entries, const double* dvec) {
  extern __shared__ __align__(16) unsigned char pose_smem[];
  ChildSmem& cs = *reinterpret_cast<ChildSmem*>(pose_smem);
  Smem<double>& sm = cs.stage;
  const ChildTask t = tasks[blockIdx.x];
  if (V.active[t.instance] == 0 || (V.fronts32 != nullptr && V.inst[t.instance].mixed != 0)) {
    return;
  }
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int wr = 16 * ((warp + 2 * (warp >> 2)) & 3);
  const int wc = 32 * (warp >> 2);
  const bool diagonal = t.I == t.J;
  double* out = V.fronts + t.front;
  const int r0 = wr + (lane >> 2);
  const int c0 = wc + 2 * (lane & 3);
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int r = t.I * kT + r0 + 8 * (e >> 3);
    const int c = t.J * kT + c0 + 8 * ((e >> 1) & 3) + (e & 1);
    cs.sum[e][tid] = c < t.k && r < t.F && c <= r ? out[static_cast<int64_t>(c) * t.F + r] : 0.0;
  }
  double acc[2][4][2] = {};
  for (int q0 = 0; q0 < t.count; q0 += kChildScan) {
    const int n = min(kChildScan, t.count - q0);
    if (q0 > 0) {
      __syncthreads();
    }
    if (tid < n) {
      const ChildEntry E = entries[t.begin + q0 + tid];
      Match& m = sm.match[tid];
      m.base_a = E.front + E.k + E.ra;
      m.base_b = E.front + E.k + E.ca;
      m.ma = E.rows;
      m.mb = E.cols;
      m.F = E.F;
      m.k = E.k;
      m.first = E.first;
      m.leaf = E.leaf;
      m.update = E.k + E.ca;
      m.groups = Groups(E.rows) | (Groups(E.cols) << 8);
    }
    __syncthreads();
    MultiplyMatches<double>(sm, n, V.fronts, dvec, diagonal, wr, wc, acc, [&] {
      // the children's own update matrices, while the first stages arrive
      for (int q = 0; q < n; ++q) {
        const Match& m = sm.match[q];
        if (m.leaf != 0) {
          continue;
        }
        // rows r0 and r0 + 8, four pairs of neighbouring columns
        const uint64_t ma = m.ma >> r0;
        const uint64_t mb = m.mb >> c0;
        const int64_t F = m.F;
        const int row = __popcll(m.ma & ((uint64_t{1} << r0) - 1));
        const int row8 = row + __popc(static_cast<uint32_t>(ma) & 0xffu);
        int col = __popcll(m.mb & ((uint64_t{1} << c0) - 1));
        const double* C = V.fronts + m.base_a + m.update * F;
        double v[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const int c = c0 + 8 * j + b;
            const bool in_c = ((mb >> (8 * j + b)) & 1) != 0 && t.J * kT + c < t.fcols;
            const double* Cc = C + col * F;
            const int below = t.J * kT + c - t.I * kT;
            v[2 * j + b] = in_c && (ma & 1) != 0 && below <= r0 ? Cc[row] : 0.0;
            v[8 + 2 * j + b] = in_c && ((ma >> 8) & 1) != 0 && below <= r0 + 8 ? Cc[row8] : 0.0;
            if (b == 0) {
              col += static_cast<int>((mb >> (8 * j)) & 1);
            } else {
              col += __popc(static_cast<uint32_t>(mb >> (8 * j + 1)) & 0x7fu);
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          cs.sum[e][tid] += v[e];
        }
      }
    });
  }
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int r = t.I * kT + r0 + 8 * (e >> 3);
    const int c = t.J * kT + c0 + 8 * ((e >> 1) & 3) + (e & 1);
    if (r < t.F && c <= r && c < t.fcols) {
      out[static_cast<int64_t>(c) * t.F + r] = cs.sum[e][tid] - acc[e >> 3][(e >> 1) & 3][e & 1];
    }
  }
}

template <auto kKernel>
void Configure(size_t smem) {
  static std::mutex mu;
  static bool configured[64] = {};
  int dev = 0;
  CudaCheck(cudaGetDevice(&dev), "device");
  const std::lock_guard<std::mutex> lock(mu);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    CudaCheck(cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
              "schur smem attr");
    if (dev >= 0 && dev < 64) {
      configured[dev] = true;
    }
  }
}

}  // namespace

int LaunchPoseSchur(const DeviceView& V, const PoseSchurArgs& args, bool fp32, cudaStream_t stream) {
  if (args.count <= 0) {
    return 0;
  }
  const auto grid = static_cast<unsigned>(args.count);
  Configure<KPoseSchur<double>>(sizeof(Smem<double>));
  KPoseSchur<double><<<grid, kThreads, sizeof(Smem<double>), stream>>>(V, args);
  if (fp32) {
    Configure<KPoseSchur<float>>(sizeof(Smem<float>));
    KPoseSchur<float><<<grid, kThreads, sizeof(Smem<float>), stream>>>(V, args);
  }
  CudaCheck(cudaGetLastError(), "pose schur launch");
  return fp32 ? 2 : 1;
}

void LaunchChildSchur(const DeviceView& V, const ChildTask* tasks, int64_t count, const ChildEntry* entries,
                      const double* dvec, cudaStream_t stream) {
  Configure<KChildSchur>(sizeof(ChildSmem));
  KChildSchur<<<static_cast<unsigned>(count), kThreads, sizeof(ChildSmem), stream>>>(V, tasks, entries, dvec);
  CudaCheck(cudaGetLastError(), "child schur launch");
}

}  // namespace sdfgpu
