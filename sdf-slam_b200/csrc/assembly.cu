// Residual / Jacobian assembly, J^T J and -J^T r accumulation, step and cost
// kernels of the FP64 LM path.
//
// This translation unit is compiled with --fmad=false: every product and sum
// is rounded separately, in the association order of the reference's C++
// (src/core/pose.hpp, src/core/grid_map.hpp, src/problem/residual_math.hpp,
// src/solvers/lm_solver.cpp), so cells are assigned bit-exactly and the
// Jacobian entries, J^T J and -J^T r agree with a plain FP64 evaluation of the
// reference's expressions. J^T J entries are accumulated per entry in
// ascending row order with the first product assigned (ParallelAtA,
// lm_solver.cpp:113-172); -J^T r alternates two accumulators over each
// column's entries (ParallelNegAtb, lm_solver.cpp:178-197).
#include <cuda_runtime.h>

#include <climits>

#include "device.cuh"
#include "trig.cuh"

namespace sdfgpu {

namespace {

struct PointEval {
  bool valid;
  int w, h;
  double residual;
  double wts[4];
  double d_pose[3];
};

__device__ __forceinline__ double MapValue(const DeviceView& V, const InstDev& I, int w, int h) {
  return V.map[I.node_off + static_cast<int64_t>(h) * I.nx + w];
}

/// GridMap::Interpolate for cell (w, h) with bilinear weights
/// (grid_map.hpp:86-93, FillCell :109-115).
__device__ __forceinline__ double Interp(const DeviceView& V, const InstDev& I, int w, int h, double a,
                                         double b, double* wts) {
  wts[0] = (1.0 - a) * (1.0 - b);
  wts[1] = a * (1.0 - b);
  wts[2] = (1.0 - a) * b;
  wts[3] = a * b;
  const int64_t n0 = I.node_off + static_cast<int64_t>(h) * I.nx + w;
  double value = 0.0;
  value += wts[0] * V.map[n0];
  value += wts[1] * V.map[n0 + 1];
  value += wts[2] * V.map[n0 + I.nx];
  value += wts[3] * V.map[n0 + I.nx + 1];
  return value;
}

/// LocateClamped + Interpolate (grid_map.hpp:75-93).
__device__ double ClampedValue(const DeviceView& V, const InstDev& I, double x, double y) {
  const double fx = (x - I.min_x) / I.dx;
  const double fy = (y - I.min_y) / I.dy;
  const int w = min(max(static_cast<int>(fx), 0), I.nx - 2);
  const int h = min(max(static_cast<int>(fy), 0), I.ny - 2);
  double wts[4];
  return Interp(V, I, w, h, fx - w, fy - h, wts);
}

/// EvalPointResidual (residual_math.hpp:75-106); gradient mode 0 exact
/// patch gradient (grid_map.hpp:98-106), 1 node central differences
/// (SmoothGradient :40-57), 2 metric finite differences (:63-73).
__device__ void EvalPoint(const DeviceView& V, const InstDev& I, double c, double s, const double* pose,
                          double px, double py, double delta, int mode, bool jac, PointEval& out) {
  const double gx = (c * px + (-s) * py) + pose[0];
  const double gy = (s * px + c * py) + pose[1];
  const double fx = (gx - I.min_x) / I.dx;
  const double fy = (gy - I.min_y) / I.dy;
  // the reference's bounds test, written so that a NaN coordinate (a pose
  // driven to NaN by a failed step) is outside too instead of reaching the
  // integer conversion
  if (!(fx >= 0.0) || !(fy >= 0.0) || !(fx <= I.nx - 1) || !(fy <= I.ny - 1)) {
    out.valid = false;
    out.residual = -delta;
    return;
  }
  out.valid = true;
  const int w = min(static_cast<int>(fx), I.nx - 2);
  const int h = min(static_cast<int>(fy), I.ny - 2);
  out.w = w;
  out.h = h;
  const double a = fx - w;
  const double b = fy - h;
  out.residual = Interp(V, I, w, h, a, b, out.wts) - delta;
  if (!jac) {
    return;
  }
  double grx;
  double gry;
  if (mode == 2) {
    const double st = I.smooth_gradient_step;
    grx = (ClampedValue(V, I, gx + st, gy) - ClampedValue(V, I, gx - st, gy)) / (2.0 * st);
    gry = (ClampedValue(V, I, gx, gy + st) - ClampedValue(V, I, gx, gy - st)) / (2.0 * st);
  } else if (mode == 1) {
    double g[4][2];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int ww = w + (q & 1);
      const int hh = h + (q >> 1);
      const int w_lo = max(ww - 1, 0);
      const int w_hi = min(ww + 1, I.nx - 1);
      const int h_lo = max(hh - 1, 0);
      const int h_hi = min(hh + 1, I.ny - 1);
      g[q][0] = (MapValue(V, I, w_hi, hh) - MapValue(V, I, w_lo, hh)) / (static_cast<double>(w_hi - w_lo) * I.dx);
      g[q][1] = (MapValue(V, I, ww, h_hi) - MapValue(V, I, ww, h_lo)) / (static_cast<double>(h_hi - h_lo) * I.dy);
    }
    const double s00 = (1.0 - a) * (1.0 - b);
    const double s10 = a * (1.0 - b);
    const double s01 = (1.0 - a) * b;
    const double s11 = a * b;
    grx = ((s00 * g[0][0] + s10 * g[1][0]) + s01 * g[2][0]) + s11 * g[3][0];
    gry = ((s00 * g[0][1] + s10 * g[1][1]) + s01 * g[2][1]) + s11 * g[3][1];
  } else {
    const int64_t n0 = I.node_off + static_cast<int64_t>(h) * I.nx + w;
    const double d00 = V.map[n0];
    const double d10 = V.map[n0 + 1];
    const double d01 = V.map[n0 + I.nx];
    const double d11 = V.map[n0 + I.nx + 1];
    grx = ((1.0 - b) * (d10 - d00) + b * (d11 - d01)) / I.dx;
    gry = ((1.0 - a) * (d01 - d00) + a * (d11 - d10)) / I.dy;
  }
  const double dx_dtheta = (-s) * px - c * py;
  const double dy_dtheta = c * px - s * py;
  out.d_pose[0] = grx;
  out.d_pose[1] = gry;
  out.d_pose[2] = grx * dx_dtheta + gry * dy_dtheta;
}

__device__ __forceinline__ int GradientMode(const InstDev& I) {
  if (I.smooth_gradient != 0 && I.smooth_gradient_step > 0.0) {
    return 2;
  }
  return I.smooth_gradient != 0 ? 1 : 0;
}

/// WrapAngle (src/core/pose.hpp:9) of the odometry residual's angle:
/// atan2(sin a, cos a) with correctly rounded sin and cos.
__device__ __forceinline__ double WrapAngle(double a) {
  double s;
  double c;
  SinCosRn(a, &s, &c);
  return atan2(s, c);
}

}  // namespace

/// Offsets of the (pose var (frame, 0), node column) entries in the front for
/// the four corner nodes of a cell (lower-left node n0, row length nx), -1
/// where the frame is not in the node's analysed coupling set. The four
/// lower-bound searches over the nodes' ascending frames advance in lock
/// step, so every step's four loads are in flight together.
__device__ __forceinline__ void PoseOffsets4(const DeviceView& V, int64_t n0, int nx, int frame_local,
                                             int64_t off[4]) {
  int col[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    col[q] = V.node_col[n0 + (q >> 1) * nx + (q & 1)];
  }
  int64_t base[4];
  int64_t end[4];
  int64_t len[4];
  int64_t longest = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    base[q] = col[q] >= 0 ? V.mp_ptr[col[q]] : 0;
    end[q] = col[q] >= 0 ? V.mp_ptr[col[q] + 1] : 0;
    len[q] = end[q] - base[q];
    longest = max(longest, len[q]);
  }
  // lower bound of frame_local in mp_frame[base, end)
  while (longest > 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (len[q] > 0) {
        const int64_t half = len[q] >> 1;
        if (V.mp_frame[base[q] + half] < frame_local) {
          base[q] += half + 1;
          len[q] -= half + 1;
        } else {
          len[q] = half;
        }
      }
    }
    longest >>= 1;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const bool hit = col[q] >= 0 && base[q] < end[q] && V.mp_frame[base[q]] == frame_local;
    off[q] = hit ? V.mp_off[base[q]] : -1;
  }
}

/// Point rows: AssemblePointRows (lm_solver.cpp:30-61) with HuberWeight
/// (problem.hpp:115-121). Writes the row record and the row's cell, and flags
/// a point whose cell lies outside its pose's analysed coupling set.
__device__ __forceinline__ void PointRow(const DeviceView& V, int64_t k) {
  if (k >= V.total_points) {
    return;
  }
  const int f = V.pt_frame[k];
  const int i = V.frame_inst[f];
  const InstDev& I = V.inst[i];
  if (V.active[i] == 0) {
    return;
  }
  const double* pose = V.poses + 3 * static_cast<int64_t>(f);
  const double2 cs = V.pose_cs[f];
  const double c = cs.x;
  const double s = cs.y;
  const double2 p = V.pt_xy[k];
  const double delta = V.pt_exp[k];
  const double sqrt_w = V.pt_sw[k];
  PointEval ev;
  EvalPoint(V, I, c, s, pose, p.x, p.y, delta, GradientMode(I), true, ev);
  const double weighted = sqrt_w * ev.residual;
  double hw = 1.0;
  if (I.huber_delta > 0.0) {
    const double ar = fabs(weighted);
    hw = ar <= I.huber_delta ? 1.0 : I.huber_delta / ar;
  }
  const double sw = sqrt(hw);
  double* rec = V.pt_rec + k * kPointRec;
  rec[7] = sw * weighted;
  if (!ev.valid) {
    V.pt_cell[k] = -1;
    return;
  }
  const double scale = sw * sqrt_w;
  double2* r2 = reinterpret_cast<double2*>(rec);
  r2[0] = make_double2(scale * ev.wts[0], scale * ev.wts[1]);
  r2[1] = make_double2(scale * ev.wts[2], scale * ev.wts[3]);
  r2[2] = make_double2(scale * ev.d_pose[0], scale * ev.d_pose[1]);
  rec[6] = scale * ev.d_pose[2];
  const int cell = ev.h * (I.nx - 1) + ev.w;
  V.pt_cell[k] = static_cast<int32_t>(I.cell_off + cell);
  const int local = f - I.frame_off;
  if (local >= 1) {
    const uint32_t word = V.allow_bits[I.allow_off + static_cast<int64_t>(local) * I.allow_words + (cell >> 5)];
    if (((word >> (cell & 31)) & 1u) == 0u) {
      atomicOr(V.status + i, kStatusPatternOverflow);
    }
    // front offsets of the (pose, corner node) blocks this row adds to; the
    // lookups run here, one thread per row, so that the cell passes read them
    // instead of searching
    const int64_t n0 = I.node_off + static_cast<int64_t>(ev.h) * I.nx + ev.w;
    int64_t off[4];
    PoseOffsets4(V, n0, I.nx, local, off);
    longlong2* po = reinterpret_cast<longlong2*>(V.pt_poff + 4 * k);
    po[0] = make_longlong2(off[0], off[1]);
    po[1] = make_longlong2(off[2], off[3]);
  }
}

/// Eikonal rows: EvalEikonalResidual (residual_math.hpp:158-171) scaled as in
/// AssembleEikonalRows (lm_solver.cpp:67-82).
__device__ __forceinline__ void EikonalRow(const DeviceView& V, int64_t e) {
  if (e >= V.total_eik) {
    return;
  }
  const int64_t node = V.eik_node[e];
  const int i = V.col_inst[V.node_col[node]];
  const InstDev& I = V.inst[i];
  if (V.active[i] == 0) {
    return;
  }
  const double d00 = V.map[node];
  const double d10 = V.map[node + 1];
  const double d01 = V.map[node + I.nx];
  const double gx = (d10 - d00) / I.dx;
  const double gy = (d01 - d00) / I.dy;
  const double2 n = V.eik_n[e];
  const double r = 1.0 - (n.x * gx + n.y * gy);
  const double sw = V.eik_sw[e];
  double* rec = V.eik_rec + e * kEikRec;
  rec[0] = sw * (n.x / I.dx + n.y / I.dy);
  rec[1] = sw * (-n.x / I.dx);
  rec[2] = sw * (-n.y / I.dy);
  rec[3] = sw * r;
}

/// Odometry / relation rows: EvalOdomResidual (residual_math.hpp:182-205)
/// scaled by sqrt_weight (lm_solver.cpp:275-296).
__device__ __forceinline__ void OdomRow(const DeviceView& V, int64_t o) {
  if (o >= V.total_odom) {
    return;
  }
  const int fi = V.odom_fi[o];
  const int fj = V.odom_fj[o];
  if (V.active[V.frame_inst[fi]] == 0) {
    return;
  }
  const double* pi = V.poses + 3 * static_cast<int64_t>(fi);
  const double* pj = V.poses + 3 * static_cast<int64_t>(fj);
  const double* m = V.odom_meas + 3 * o;
  const double sw = V.odom_sw[o];
  const double2 cs = V.pose_cs[fi];
  const double c = cs.x;
  const double s = cs.y;
  const double dtx = pj[0] - pi[0];
  const double dty = pj[1] - pi[1];
  const double rx = c * dtx + s * dty;
  const double ry = (-s) * dtx + c * dty;
  double* rec = V.odom_rec + o * kOdomRec;
  rec[0] = sw * (rx - m[0]);
  rec[1] = sw * (ry - m[1]);
  rec[2] = sw * WrapAngle(pj[2] - pi[2] - m[2]);
  // d_pose_i rows: [-c, -s, -s dtx + c dty], [s, -c, -c dtx - s dty], [0, 0, -1]
  rec[3] = sw * (-c);
  rec[4] = sw * (-s);
  rec[5] = sw * ((-s) * dtx + c * dty);
  rec[6] = sw * s;
  rec[7] = sw * (-c);
  rec[8] = sw * ((-c) * dtx + (-s) * dty);
  rec[9] = sw * 0.0;
  rec[10] = sw * 0.0;
  rec[11] = sw * -1.0;
  // d_pose_j rows: [c, s, 0], [-s, c, 0], [0, 0, 1]
  rec[12] = sw * c;
  rec[13] = sw * s;
  rec[14] = sw * 0.0;
  rec[15] = sw * (-s);
  rec[16] = sw * c;
  rec[17] = sw * 0.0;
  rec[18] = sw * 0.0;
  rec[19] = sw * 0.0;
  rec[20] = sw * 1.0;
}

/// All rows in one launch: the first blocks take the odometry rows, the next the
/// Eikonal rows, the others the point rows (which bound it: reads of the map and
/// of the coupling lists). Measured on B200 against a launch each, with the
/// cell sort: 10-frame room 36 -> 31 us, 76-frame floor plan 67 -> 61.
__global__ void __launch_bounds__(256) KRows(DeviceView V, int odom_blocks, int eik_blocks) {
  const int b = static_cast<int>(blockIdx.x);
  if (b < odom_blocks) {
    OdomRow(V, static_cast<int64_t>(b) * 256 + threadIdx.x);
  } else if (b < odom_blocks + eik_blocks) {
    EikonalRow(V, static_cast<int64_t>(b - odom_blocks) * 256 + threadIdx.x);
  } else {
    PointRow(V, static_cast<int64_t>(b - odom_blocks - eik_blocks) * 256 + threadIdx.x);
  }
}

/// cell_start[c] = first position of cell c in the sorted keys.
__global__ void KCellStart(const int32_t* keys, int64_t n, int64_t num_cells, int32_t* cell_start) {
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c > num_cells) {
    return;
  }
  int64_t lo = 0;
  int64_t hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (keys[mid] < c) {
      lo = mid + 1;
    } else {
      hi = mid;
    }
  }
  cell_start[c] = static_cast<int32_t>(lo);
}

namespace {

__device__ __forceinline__ double WarpSum(double v) {
  // xor butterfly: every lane ends with the same, fixed-order sum
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    v += __shfl_xor_sync(0xffffffffu, v, m);
  }
  return v;
}

/// Front offset of the J^T J entry between the cell corners a and b of a cell,
/// their columns ca and cb, or -1 when one corner is constant.
__device__ __forceinline__ int64_t PairOffset(const DeviceView& V, int ca, int cb, int a, int b) {
  if (ca < 0 || cb < 0) {
    return -1;
  }
  const int dw = (b & 1) - (a & 1);
  const int dh = (b >> 1) - (a >> 1);
  const int64_t off = V.mm_off[static_cast<int64_t>(ca) * 9 + (dh + 1) * 3 + (dw + 1)];
  if (off >= 0) {
    return off;
  }
  return V.mm_off[static_cast<int64_t>(cb) * 9 + (1 - dh) * 3 + (1 - dw)];
}

/// One step of a reduction that halves the values a lane holds: lanes a
/// distance kD apart exchange halves of their kN values.
template <int kN, int kD>
__device__ __forceinline__ void HalveStep(double* v, int lane) {
  const bool upper = (lane & kD) != 0;
#pragma unroll
  for (int q = 0; q < kN / 2; ++q) {
    const double send = upper ? v[q] : v[q + kN / 2];
    const double keep = upper ? v[q + kN / 2] : v[q];
    v[q] = keep + __shfl_xor_sync(0xffffffffu, send, kD);
  }
}

/// Sum over the warp of sixteen values per lane, in a fixed order: value q in
/// lanes 2 q and 2 q + 1 (16 exchanges; a butterfly per value takes 80).
__device__ __forceinline__ double WarpSum16(double (&v)[16], int lane) {
  HalveStep<16, 16>(v, lane);
  HalveStep<8, 8>(v, lane);
  HalveStep<4, 4>(v, lane);
  HalveStep<2, 2>(v, lane);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

/// Waits until the cells that share a node with this one and come before it
/// (a lower colour) are done, one lane per neighbour; a wait that runs out
/// marks the instance.
__device__ __forceinline__ void WaitForNeighbours(const DeviceView& V, int i, const CellSync& sync, int64_t cell,
                                                  int cx, int cy, int cw, int ch, int lane) {
  if (lane < 8) {
    const int at = lane < 4 ? lane : lane + 1;
    const int x = cx + at % 3 - 1;
    const int y = cy + at / 3 - 1;
    const int own = (cx & 1) | ((cy & 1) << 1);
    const int colour = (x & 1) | ((y & 1) << 1);
    if (x >= 0 && x < cw && y >= 0 && y < ch && colour < own) {
      const uint32_t* word = sync.done + cell + static_cast<int64_t>(y - cy) * cw + (x - cx);
      uint32_t it = 0;
      for (; it < sync.limit; ++it) {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
        if (v != 0) {
          break;
        }
        if (it > 64) {
          __nanosleep(100);
        }
      }
      if (it == sync.limit) {
        atomicOr(V.status + i, kStatusWaitTimeout);
      }
    }
  }
  __syncwarp();
}

}  // namespace

/// One cell, one warp: the 4x4 map block and the corner gradients are
/// lane-strided sums over the cell's point rows reduced in a fixed order; the
/// map-pose blocks are segmented sums over runs of rows of one frame (rows of a
/// cell are sorted, so frames are contiguous); the cell's Eikonal row (spec at
/// its lower-left node) is added to them. Cells that share a node add in the
/// order of their colours (cx % 2, cy % 2) = (colour & 1, colour >> 1), with plain
/// read-modify-writes, so every entry is a deterministic sum. kWait: the
/// launch holds all colours, and a cell waits for its neighbours of lower
/// colours before its first write; everything before that runs ahead of the
/// wait.
template <bool kWait>
__device__ __forceinline__ void CellPassOne(const DeviceView& V, int64_t entry, const CellSync& sync, int lane) {
  const int i = static_cast<int>(entry >> kCellBits);
  const int64_t cell = entry & ((int64_t{1} << kCellBits) - 1);
  const InstDev& I = V.inst[i];
  if (V.active[i] == 0) {
    return;  // as every cell it shares a node with
  }
  const int cw = I.nx - 1;
  const int ch = I.ny - 1;
  const int local = static_cast<int>(cell - I.cell_off);
  const int cx = local % cw;
  const int cy = local / cw;
  const int64_t n0 = I.node_off + static_cast<int64_t>(cy) * I.nx + cx;
  int col[4];
  col[0] = V.node_col[n0];
  col[1] = V.node_col[n0 + 1];
  col[2] = V.node_col[n0 + I.nx];
  col[3] = V.node_col[n0 + I.nx + 1];
  const int rb = V.cell_start[cell];
  const int re = V.cell_start[cell + 1];
  const int eik = V.eik_index[n0];
  if (rb == re && eik < 0) {
    if (kWait && lane == 0 && cell != sync.withhold) {
      __stcg(sync.done + cell, 1u);
    }
    return;
  }
  // what lanes 2 q and 2 q + 1 add in the end: pair q of corners (a, b), a <= b,
  // or the gradient of corner q - 10; the Eikonal row's part of it (nodes (cx,
  // cy), (cx + 1, cy), (cx, cy + 1) = corners 0, 1, 2)
  const int q = lane >> 1;
  const int ca = q < 10 ? (q < 4 ? 0 : q < 7 ? 1 : q < 9 ? 2 : 3) : q - 10;
  const int cb = q < 4 ? q : q < 7 ? q - 3 : q < 9 ? q - 5 : 3;
  const int col_a = ca == 0 ? col[0] : ca == 1 ? col[1] : ca == 2 ? col[2] : col[3];
  const int col_b = cb == 0 ? col[0] : cb == 1 ? col[1] : cb == 2 ? col[2] : col[3];
  const bool eik_part = eik >= 0 && ca < 3 && (q < 10 ? cb < 3 : q < 13);
  double* target = nullptr;
  double eik_add = 0.0;
  if ((lane & 1) == 0 && q < 14 && (rb < re || eik_part)) {
    if (q < 10) {
      const int64_t off = PairOffset(V, col_a, col_b, ca, cb);
      target = off >= 0 ? V.asm_fronts + off : nullptr;
    } else {
      target = col_a >= 0 ? V.rhs + col_a : nullptr;
    }
    if (eik_part) {
      const double* r = V.eik_rec + static_cast<int64_t>(eik) * kEikRec;
      eik_add = r[ca] * r[q < 10 ? cb : 3];
    }
  }
  bool waited = false;
  // One pass over the cell's rows in chunks of 32 (lane l takes rows
  // rb + l + 32 t): the 4x4 map block and corner gradients accumulate per
  // lane and are reduced by a fixed butterfly at the end; the map-pose
  // blocks are segmented sums over runs of one frame inside each chunk. A
  // chunk's records, frames and front offsets are loaded while the previous
  // chunk is scanned and written (the row indices one chunk further ahead).
  double sums[16];  // pairs, gradients, two unused
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    sums[e] = 0.0;
  }
  bool overflow = false;
  struct ChunkRow {
    double2 a01, a23, p01, p2r;
    longlong2 o01, o23;
    int f;
  };
  auto fetch = [&](int kk, ChunkRow& R) {
    if (kk >= 0) {
      const double2* r2 = reinterpret_cast<const double2*>(V.pt_rec + static_cast<int64_t>(kk) * kPointRec);
      const longlong2* po = reinterpret_cast<const longlong2*>(V.pt_poff + 4 * static_cast<int64_t>(kk));
      R.a01 = r2[0];
      R.a23 = r2[1];
      R.p01 = r2[2];
      R.p2r = r2[3];
      R.o01 = po[0];
      R.o23 = po[1];
      R.f = V.pt_frame[kk];
    } else {
      R.a01 = R.a23 = R.p01 = R.p2r = make_double2(0.0, 0.0);
      R.o01 = R.o23 = make_longlong2(-1, -1);
      R.f = -1;
    }
  };
  int k = (rb + lane < re) ? V.cell_rows[rb + lane] : -1;
  ChunkRow cur;
  fetch(k, cur);
  int k_next = (rb + 32 + lane < re) ? V.cell_rows[rb + 32 + lane] : -1;
  for (int base = rb; base < re; base += 32) {
    ChunkRow nxt;
    int k_after = -1;
    if (base + 32 < re) {
      fetch(k_next, nxt);
      k_after = (base + 64 + lane < re) ? V.cell_rows[base + 64 + lane] : -1;
    } else {
      fetch(-1, nxt);
    }
    const bool in = k >= 0;
    const int f = in ? cur.f : -1;
    double J[4] = {cur.a01.x, cur.a01.y, cur.a23.x, cur.a23.y};
    const double jp[3] = {cur.p01.x, cur.p01.y, cur.p2r.x};
    const double r = cur.p2r.y;
    if (in) {
      int e = 0;
#pragma unroll
      for (int aa = 0; aa < 4; ++aa) {
#pragma unroll
        for (int bb = aa; bb < 4; ++bb) {
          sums[e] = sums[e] + J[aa] * J[bb];
          ++e;
        }
        sums[10 + aa] = sums[10 + aa] + J[aa] * r;
      }
    }
    double v[12];
    const bool posed = in && (f - I.frame_off >= 1);
#pragma unroll
    for (int aa = 0; aa < 4; ++aa) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        v[3 * aa + c] = posed ? J[aa] * jp[c] : 0.0;
      }
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int fu = __shfl_up_sync(0xffffffffu, f, d);
#pragma unroll
      for (int e = 0; e < 12; ++e) {
        const double vu = __shfl_up_sync(0xffffffffu, v[e], d);
        if (lane >= d && fu == f) {
          v[e] = vu + v[e];
        }
      }
    }
    const int fn = __shfl_down_sync(0xffffffffu, f, 1);
    const int p = base + lane;
    const bool tail = in && (lane == 31 || p + 1 >= re || fn != f);
    const int fl = f - I.frame_off;
    if (kWait && !waited) {
      WaitForNeighbours(V, i, sync, cell, cx, cy, cw, ch, lane);
      waited = true;
    }
    if (tail && fl >= 1) {
      // the (up to 12) entries are distinct: all loads first, then the
      // stores, so their latencies overlap
      const int64_t offs[4] = {cur.o01.x, cur.o01.y, cur.o23.x, cur.o23.y};
      double old[12];
#pragma unroll
      for (int aa = 0; aa < 4; ++aa) {
        if (col[aa] >= 0 && offs[aa] >= 0) {
          old[3 * aa] = __ldcg(V.asm_fronts + offs[aa]);
          old[3 * aa + 1] = __ldcg(V.asm_fronts + offs[aa] + 1);
          old[3 * aa + 2] = __ldcg(V.asm_fronts + offs[aa] + 2);
        } else {
          old[3 * aa] = old[3 * aa + 1] = old[3 * aa + 2] = 0.0;
        }
      }
#pragma unroll
      for (int aa = 0; aa < 4; ++aa) {
        if (col[aa] >= 0) {
          const int64_t off = offs[aa];
          if (off >= 0) {
            V.asm_fronts[off] = old[3 * aa] + v[3 * aa];
            V.asm_fronts[off + 1] = old[3 * aa + 1] + v[3 * aa + 1];
            V.asm_fronts[off + 2] = old[3 * aa + 2] + v[3 * aa + 2];
          } else {
            overflow = true;
          }
        }
      }
    }
    __syncwarp();
    cur = nxt;
    k = k_next;
    k_next = k_after;
  }
  if (kWait && !waited) {
    WaitForNeighbours(V, i, sync, cell, cx, cy, cw, ch, lane);
  }
  const double sum = WarpSum16(sums, lane);
  if (target != nullptr) {
    *target = __ldcg(target) + (sum + eik_add);
  }
  if (overflow) {
    atomicOr(V.status + i, kStatusPatternOverflow);
  }
  if (kWait) {
    // every lane's writes before the flag
    __syncwarp();
    if (lane == 0 && cell != sync.withhold) {
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(sync.done + cell), "r"(1u) : "memory");
    }
  }
}

/// Cells of one colour, with a grid stride (the launch holds as many blocks as
/// are resident, so no cell waits for a second wave behind a busy one), or with
/// kWait all cells, colour by colour, in one launch: warps take a cell at a time
/// from a counter, in order, the next one while they work on the current, so
/// the cells a cell waits for are done or being worked on. cells: (instance,
/// cell), kCellBits bits of cell. Bound by the chain of reads behind a cell's
/// rows and, in large problems, by the segmented sums. Measured on B200 against
/// four launches with a butterfly per sum and the offsets read behind the sums:
/// 1,600 cells 48 -> 20 us, 9,900 cells 100 -> 90 (four launches), 39,600 cells
/// 324 -> 294, 32 instances 608 -> 496.
template <bool kWait>
__global__ void __launch_bounds__(256, 2) KCellPass(DeviceView V, const int64_t* cells, int64_t count,
                                                    CellSync sync) {
  const int lane = threadIdx.x & 31;
  if (!kWait) {
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t w = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < count; w += warps) {
      CellPassOne<false>(V, cells[w], sync, lane);
    }
    return;
  }
  uint32_t taken = 0;
  if (lane == 0) {
    taken = atomicAdd(sync.ticket, 1u);
  }
  for (;;) {
    const int64_t w = __shfl_sync(0xffffffffu, taken, 0);
    if (w >= count) {
      return;
    }
    uint32_t ahead = 0;
    if (lane == 0) {
      ahead = atomicAdd(sync.ticket, 1u);
    }
    CellPassOne<true>(V, cells[w], sync, lane);
    taken = ahead;
  }
}
template __global__ void KCellPass<false>(DeviceView V, const int64_t* cells, int64_t count, CellSync sync);
template __global__ void KCellPass<true>(DeviceView V, const int64_t* cells, int64_t count, CellSync sync);

/// Cross-frame pose blocks of frame pairs linked by odometry / relation rows.
__device__ __forceinline__ void PosePairEntry(const DeviceView& V, int64_t t) {
  const int p = static_cast<int>(t / 9);
  if (p >= V.num_pairs) {
    return;
  }
  const int a = static_cast<int>(t % 9) / 3;  // row var of the larger frame g
  const int b = static_cast<int>(t % 9) % 3;  // column var of the smaller frame f
  const int f = V.pair_f[p];
  const int g = V.pair_g[p];
  const int i = V.frame_inst[f];
  if (V.active[i] == 0) {
    return;
  }
  const InstDev& I = V.inst[i];
  double acc = -0.0;
  for (int64_t q = V.pair_ptr[p]; q < V.pair_ptr[p + 1]; ++q) {
    const int code = V.pair_spec[q];
    const double* rec = V.odom_rec + static_cast<int64_t>(code >> 1) * kOdomRec;
    // code bit 0 set: the spec's frame_i is the larger frame g
    const double* bg = rec + ((code & 1) ? 3 : 12);
    const double* bf = rec + ((code & 1) ? 12 : 3);
    for (int r = 0; r < 3; ++r) {
      acc = acc + bg[3 * r + a] * bf[3 * r + b];
    }
  }
  const int fl = f - I.frame_off;
  const int gl = g - I.frame_off;
  const int colf = I.pp_first + 3 * (fl - 1) + b;
  const int rowg = I.pp_first + 3 * (gl - 1) + a;
  V.asm_fronts[I.pp_base + static_cast<int64_t>(colf) * I.pp_ld + rowg] = acc;
}

/// Same-frame pose blocks and the pose columns of J^T r: one block of 256
/// threads per frame, thread-strided over the frame's point rows, a fixed
/// butterfly per warp and a fixed order over warps, then the frame's odometry
/// / relation rows in spec order.
__global__ void __launch_bounds__(256) KPoseFrames(DeviceView V) {
  __shared__ double part[8][9];
  const int64_t f = blockIdx.x;
  if (f >= V.total_frames) {
    PosePairEntry(V, (f - V.total_frames) * 256 + threadIdx.x);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int i = V.frame_inst[f];
  const InstDev& I = V.inst[i];
  const int fl = static_cast<int>(f) - I.frame_off;
  if (fl < 1 || V.active[i] == 0) {
    return;
  }
  double acc[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    acc[q] = 0.0;
  }
  const int64_t rb = V.frame_rows_ptr[f];
  const int64_t re = V.frame_rows_ptr[f + 1];
  // four rows per thread per pass, their loads issued together; a thread's
  // rows are still added in ascending order
  const int64_t stride = blockDim.x;
  for (int64_t q0 = rb + threadIdx.x; q0 < re; q0 += 4 * stride) {
    int kk[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t q = q0 + u * stride;
      kk[u] = q < re ? V.frame_rows[q] : -1;
    }
    int cellv[4];
    double2 j01[4];
    double2 j2r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (kk[u] >= 0) {
        const double2* r2 = reinterpret_cast<const double2*>(V.pt_rec + static_cast<int64_t>(kk[u]) * kPointRec);
        cellv[u] = V.pt_cell[kk[u]];
        j01[u] = r2[2];
        j2r[u] = r2[3];
      } else {
        cellv[u] = -1;
        j01[u] = make_double2(0.0, 0.0);
        j2r[u] = make_double2(0.0, 0.0);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (cellv[u] < 0) {
        continue;
      }
      const double j0 = j01[u].x;
      const double j1 = j01[u].y;
      const double j2 = j2r[u].x;
      const double r = j2r[u].y;
      acc[0] = acc[0] + j0 * j0;
      acc[1] = acc[1] + j1 * j0;
      acc[2] = acc[2] + j2 * j0;
      acc[3] = acc[3] + j1 * j1;
      acc[4] = acc[4] + j2 * j1;
      acc[5] = acc[5] + j2 * j2;
      acc[6] = acc[6] + j0 * r;
      acc[7] = acc[7] + j1 * r;
      acc[8] = acc[8] + j2 * r;
    }
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    acc[q] = WarpSum(acc[q]);
  }
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      part[warp][q] = acc[q];
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) {
    return;
  }
  for (int q = 0; q < 9; ++q) {
    double v = part[0][q];
    for (int w = 1; w < 8; ++w) {
      v = v + part[w][q];
    }
    acc[q] = v;
  }
  const int aa[6] = {0, 1, 2, 1, 2, 2};
  const int bb[6] = {0, 0, 0, 1, 1, 2};
  for (int64_t q = V.frame_odom_ptr[f]; q < V.frame_odom_ptr[f + 1]; ++q) {
    const int code = V.frame_odom[q];
    const double* rec = V.odom_rec + static_cast<int64_t>(code >> 1) * kOdomRec;
    const double* blk = rec + ((code & 1) ? 12 : 3);
    for (int r = 0; r < 3; ++r) {
      for (int e = 0; e < 6; ++e) {
        acc[e] = acc[e] + blk[3 * r + aa[e]] * blk[3 * r + bb[e]];
      }
      for (int a = 0; a < 3; ++a) {
        acc[6 + a] = acc[6 + a] + blk[3 * r + a] * rec[r];
      }
    }
  }
  const int base = I.pp_first + 3 * (fl - 1);
  for (int e = 0; e < 6; ++e) {
    V.asm_fronts[I.pp_base + static_cast<int64_t>(base + bb[e]) * I.pp_ld + (base + aa[e])] = acc[e];
  }
  const int c0 = V.frame_col[f];
  V.rhs[c0] = acc[6];
  V.rhs[c0 + 1] = acc[7];
  V.rhs[c0 + 2] = acc[8];
}

/// Zeroes the lower triangle of the assembly fronts before the row kernels
/// add into them: one warp per column c, rows c..F-1 (coalesced); task (sn,
/// first of kZeroCols columns). Also J^T r and the cell pass's counter and
/// flags. The upper triangles are never read before
/// the factorization writes them, so they are left as they are (half the
/// bytes of clearing the whole buffer).
__global__ void KZeroFronts(DeviceView V, const int32_t* tasks, int64_t count, uint32_t* words, int64_t num_words,
                            uint64_t* stamp) {
  StampPhase(stamp);
  const int64_t threads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int64_t me = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (int64_t e = me; e < V.n; e += threads) {
    V.rhs[e] = 0.0;
  }
  for (int64_t e = me; e < num_words; e += threads) {
    words[e] = 0;
  }
  if (blockIdx.x >= count) {
    return;
  }
  const int32_t* t = tasks + 2 * static_cast<int64_t>(blockIdx.x);
  const SupernodeRec S = V.sn[t[0]];
  const int c = t[1] + static_cast<int>(threadIdx.x >> 5);
  const int lane = static_cast<int>(threadIdx.x & 31);
  if (c >= S.fcols) {
    return;
  }
  double* col = V.asm_fronts + S.front_off + static_cast<int64_t>(c) * S.F;
  for (int r = c + lane; r < S.F; r += 32) {
    col[r] = 0.0;
  }
}

/// Turns the accumulated J^T r into -J^T r and applies the damping of
/// lm_solver.cpp:321-330 to every diagonal entry (lambda, or lambda times
/// max(diag, 1e-12) under Marquardt scaling).
__global__ void KFinalizeNormal(DeviceView V) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= V.n) {
    return;
  }
  const int i = V.col_inst[col];
  if (V.active[i] == 0) {
    return;
  }
  V.rhs[col] = -V.rhs[col];
  int64_t off;
  if (V.col_node[col] >= 0) {
    off = V.mm_off[static_cast<int64_t>(col) * 9 + 4];
  } else {
    const InstDev& I = V.inst[i];
    const int rel = I.pp_first + (col - I.col_off - I.num_active);
    off = I.pp_base + static_cast<int64_t>(rel) * I.pp_ld + rel;
  }
  const double d = V.asm_fronts[off];
  const double lam = V.lam[i];
  V.asm_fronts[off] = V.marquardt[i] != 0 ? d + lam * fmax(d, 1e-12) : d + lam;
}
/// Saves or restores the state of active instances (backup for revert,
/// lm_solver.cpp:366-372, 405-423). dir 0: save, 1: restore where
/// revert_mask[i] != 0.
__global__ void KBackup(DeviceView V, int dir, const int32_t* revert_mask) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < V.total_nodes) {
    const int col = V.node_col[t];
    // nodes of an instance: find instance through the column when active,
    // otherwise leave untouched (constant nodes never change)
    if (col >= 0) {
      const int i = V.col_inst[col];
      if (dir == 0 ? V.active[i] != 0 : revert_mask[i] != 0) {
        if (dir == 0) {
          V.map_backup[t] = V.map[t];
        } else {
          V.map[t] = V.map_backup[t];
        }
      }
    }
  }
  if (t < 3 * static_cast<int64_t>(V.total_frames)) {
    const int i = V.frame_inst[t / 3];
    if (dir == 0 ? V.active[i] != 0 : revert_mask[i] != 0) {
      if (dir == 0) {
        V.poses_backup[t] = V.poses[t];
      } else {
        V.poses[t] = V.poses_backup[t];
      }
    }
  }
  if (t < V.total_frames) {
    const int i = V.frame_inst[t];
    if (dir == 0 ? V.active[i] != 0 : revert_mask[i] != 0) {
      if (dir == 0) {
        V.pose_cs_backup[t] = V.pose_cs[t];
      } else {
        V.pose_cs[t] = V.pose_cs_backup[t];
      }
    }
  }
}

/// Problem::ApplyStep (problem.cpp:117-130): map values and positions; each
/// moved frame's angle theta + delta goes to theta_pre, and the pose gets a
/// provisional wrapped angle with correctly rounded cos and sin, which the
/// cost of the candidate state uses. Once the LM step is decided, the host
/// replaces the accepted angles and their cos / sin by the platform libm's
/// (KCommitPoses), so that the next linearization rotates with the
/// reference's bits.
__global__ void KApplyStep(DeviceView V, uint64_t* stamp) {
  StampPhase(stamp);
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= V.n) {
    return;
  }
  const int i = V.col_inst[col];
  // a failed factorization, a solve whose wait ran out or a stale pattern
  // leaves the state untouched
  if (V.active[i] == 0 ||
      (V.status[i] & (kStatusPatternOverflow | kStatusZeroPivot | kStatusWaitTimeout)) != 0) {
    return;
  }
  const int node = V.col_node[col];
  if (node >= 0) {
    V.map[node] += V.step[col];
    return;
  }
  const InstDev& I = V.inst[i];
  const int rel = col - I.col_off - I.num_active;
  if (rel % 3 != 0) {
    return;
  }
  const int f = I.frame_off + 1 + rel / 3;
  double* p = V.poses + 3 * static_cast<int64_t>(f);
  p[0] += V.step[col];
  p[1] += V.step[col + 1];
  const double t = p[2] + V.step[col + 2];
  V.theta_pre[f] = t;
  V.theta_upd[f] = 1;
  const double th = WrapAngle(t);
  p[2] = th;
  double sn;
  double cs;
  SinCosRn(th, &sn, &cs);
  V.pose_cs[f] = make_double2(cs, sn);
}

/// The accepted angles of the moved frames and their cos and sin, as the
/// host computed them with the platform's libm (WrapAngle, pose.hpp:9):
/// theta_out holds (theta, cos, sin, flag) per frame, flag 1 to commit.
__device__ __forceinline__ void CommitPose(const DeviceView& V, int f) {
  if (f >= V.total_frames || V.theta_out[4 * f + 3] == 0.0) {
    return;
  }
  V.poses[3 * static_cast<int64_t>(f) + 2] = V.theta_out[4 * f];
  V.pose_cs[f] = make_double2(V.theta_out[4 * f + 1], V.theta_out[4 * f + 2]);
}
__global__ void KCommitPoses(DeviceView V) { CommitPose(V, blockIdx.x * blockDim.x + threadIdx.x); }

/// Start of an iteration: its parameters from pinned host memory (read in
/// place: three copies of a few bytes cost about 12 us of copy-engine gaps per
/// iteration on B200, this kernel 4), cleared status words, and with *commit
/// the last accepted step's angles (as KCommitPoses).
__global__ void KBeginIteration(DeviceView V, const int32_t* active, const double* lam, const int32_t* marquardt,
                                const int32_t* commit, uint64_t* stamp) {
  StampPhase(stamp);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < V.num_inst) {
    V.active[t] = active[t];
    V.lam[t] = lam[t];
    V.marquardt[t] = marquardt[t];
    V.status[t] = 0;
  }
  if (*commit != 0) {
    CommitPose(V, t);
  }
}

/// Clears a few words (a kernel between kernels starts at once; a memset of
/// this size goes through the copy engine, with gaps of about 2 us).
__global__ void KClearWords(uint32_t* words, int64_t count, uint64_t* stamp) {
  StampPhase(stamp);
  for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < count;
       q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    words[q] = 0u;
  }
}

/// Per-row cost terms of Problem::Cost (problem.cpp:132-156): point rows with
/// the exact (non-smooth) evaluation and the Huber loss, Eikonal rows,
/// odometry rows. Terms are laid out points, then Eikonal, then odometry; with
/// `step` the per-column terms of the step norm and of the trust-region
/// prediction follow (lm_solver.cpp:378, 389-391): delta^2 of every column,
/// then delta * (lambda delta + rhs).
__global__ void KCostTerms(DeviceView V, double* terms, int step) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t < V.total_points) {
    const int f = V.pt_frame[t];
    const int i = V.frame_inst[f];
    const InstDev& I = V.inst[i];
    const double* pose = V.poses + 3 * static_cast<int64_t>(f);
    const double2 cs = V.pose_cs[f];
    const double c = cs.x;
    const double s = cs.y;
    const double2 p = V.pt_xy[t];
    PointEval ev;
    EvalPoint(V, I, c, s, pose, p.x, p.y, V.pt_exp[t], 0, false, ev);
    const int local = f - I.frame_off;
    if (ev.valid && local >= 1) {
      const uint32_t* allow = V.allow_bits + I.allow_off + static_cast<int64_t>(local) * I.allow_words;
      const int cw = I.nx - 1;
      const int cell = ev.h * cw + ev.w;
      if (((allow[cell >> 5] >> (cell & 31)) & 1u) == 0u) {
        atomicOr(V.status + i, kStatusNextOverflow);
      } else if (I.near_cells > 0 && (V.status[i] & kStatusNearEdge) == 0) {
        // the eight cells near_cells away (along the axes and the diagonals,
        // those inside the grid): one outside the set marks the instance
        const int g = I.near_cells;
        bool near = false;
#pragma unroll
        for (int q = 0; q < 9; ++q) {
          const int w = ev.w + g * (q % 3 - 1);
          const int h = ev.h + g * (q / 3 - 1);
          if (q != 4 && w >= 0 && w < cw && h >= 0 && h < I.ny - 1) {
            const int c = h * cw + w;
            near = near || ((allow[c >> 5] >> (c & 31)) & 1u) == 0u;
          }
        }
        if (near) {
          atomicOr(V.status + i, kStatusNearEdge);
        }
      }
    }
    const double r = V.pt_sw[t] * ev.residual;
    double term;
    if (I.huber_delta > 0.0 && fabs(r) > I.huber_delta) {
      term = I.huber_delta * (2.0 * fabs(r) - I.huber_delta);
    } else {
      term = r * r;
    }
    terms[t] = term;
    return;
  }
  const int64_t e = t - V.total_points;
  if (e < V.total_eik) {
    const int64_t node = V.eik_node[e];
    const int i = V.col_inst[V.node_col[node]];
    const InstDev& I = V.inst[i];
    const double d00 = V.map[node];
    const double d10 = V.map[node + 1];
    const double d01 = V.map[node + I.nx];
    const double gx = (d10 - d00) / I.dx;
    const double gy = (d01 - d00) / I.dy;
    const double2 n = V.eik_n[e];
    const double r = V.eik_sw[e] * (1.0 - (n.x * gx + n.y * gy));
    terms[t] = r * r;
    return;
  }
  const int64_t o = e - V.total_eik;
  if (o < V.total_odom) {
    const double* pi = V.poses + 3 * static_cast<int64_t>(V.odom_fi[o]);
    const double* pj = V.poses + 3 * static_cast<int64_t>(V.odom_fj[o]);
    const double* m = V.odom_meas + 3 * o;
    const double sw = V.odom_sw[o];
    const double2 cs = V.pose_cs[V.odom_fi[o]];
    const double c = cs.x;
    const double s = cs.y;
    const double dtx = pj[0] - pi[0];
    const double dty = pj[1] - pi[1];
    const double e0 = sw * ((c * dtx + s * dty) - m[0]);
    const double e1 = sw * (((-s) * dtx + c * dty) - m[1]);
    const double e2 = sw * WrapAngle(pj[2] - pi[2] - m[2]);
    terms[t] = (e0 * e0 + e1 * e1) + e2 * e2;
    return;
  }
  const int64_t col = o - V.total_odom;
  if (step != 0 && col < V.n) {
    const double d = V.step[col];
    terms[t] = d * d;
    terms[t + V.n] = d * (V.lam[V.col_inst[col]] * d + V.rhs[col]);
  }
}

/// Deterministic segmented sum, first level: block (seg, part) sums the
/// part-th of kSegParts equal slices of segment seg with a fixed per-thread
/// stride and a fixed tree.
constexpr int kSegParts = 32;

__global__ void __launch_bounds__(256) KSegmentPartial(const double* x, const int64_t* seg_begin,
                                                       const int64_t* seg_end, double* partial) {
  __shared__ double red[256];
  const int seg = blockIdx.x / kSegParts;
  const int part = blockIdx.x % kSegParts;
  const int64_t b = seg_begin[seg];
  const int64_t e = seg_end[seg];
  const int64_t len = (e - b + kSegParts - 1) / kSegParts;
  const int64_t pb = b + part * len;
  const int64_t pe = min(e, pb + len);
  double s = 0.0;
  for (int64_t q = pb + threadIdx.x; q < pe; q += blockDim.x) {
    s += x[q];
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[threadIdx.x] += red[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = red[0];
  }
}

/// Second level: one warp per segment adds its kSegParts partials with a
/// fixed butterfly; the sums and the instances' status words go straight to
/// pinned host memory.
__global__ void KSegmentFinal(DeviceView V, const double* partial, int num_segments, double* out,
                              int32_t* status_out, uint64_t* stamp) {
  StampPhase(stamp);
  const int thread = blockIdx.x * blockDim.x + threadIdx.x;
  for (int i = thread; i < V.num_inst; i += gridDim.x * blockDim.x) {
    status_out[i] = V.status[i];
  }
  const int seg = thread >> 5;
  const int lane = threadIdx.x & 31;
  if (seg >= num_segments) {
    return;
  }
  const double v = WarpSum(partial[static_cast<int64_t>(seg) * kSegParts + lane]);
  if (lane == 0) {
    out[seg] = v;
  }
}

}  // namespace sdfgpu
