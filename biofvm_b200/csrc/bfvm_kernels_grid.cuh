// Whole steps of a small microenvironment in one cooperative launch.
//
// A field of up to 2^19 voxel-densities with at most 64 points per axis costs
// more in kernel start-up than in work when every phase of a step is its own
// launch.  Here every step runs inside one launch, as two phases (or three,
// below) separated by grid-wide barriers of a cooperative launch (all blocks are
// resident, so each barrier completes):
//   xy: an item is one xy plane (of sg of its densities), held in shared
//       memory.  As it is loaded, its voxels take the bulk update
//       (BioFVM_microenvironment.cpp:603-609), then their agents in list order
//       (BioFVM_basic_agent.cpp:234-235), then the Dirichlet values
//       (BioFVM_microenvironment.cpp:192-197).  The x lines are solved in
//       shared memory, the y lines from there to the field.  A node's value
//       stays in its place through both: the x lines do not overwrite it, and
//       the y lines pass it on, so that it is set before each axis
//       (BioFVM_solvers.cpp:177, 207, 241).
//   z:  tiles of columns, straight from and to the field.
// Lines are solved as in bfvm_kernels_closed.cuh, in chunks of 8 points, one
// per thread: sg is the most densities whose x lines and y lines are at most
// one chunk per thread each.
//
// The steps are bound by latency: barriers, and the chains of a line.  A
// grid barrier also empties L1, so that anything read again after it costs an
// L2 round trip: the lines' constants are copied to shared memory once, and a
// plane's loads are two rounds (the field with the maps, then what they point
// to).  One block per SM: with two, the registers spill.  Steps with 1000
// agents and a fixed boundary, 100 in a call, in us (in brackets with three
// phases x, y, z through memory and the elimination's per-point tables): 50^3 x
// 1 13.1 (16.8), of three solvers at once 6.7 a step (9.9); 24^3 x 20 14.0
// (18.3), 32^3 x 8 13.1 (14.9), 64^3 x 2 16.0 (22.4), 64 x 64 x 16 x 1 15.9
// (15.3; of three at once 5.7, 6.2).  Three solvers at once with planes for 75
// to 148 blocks each find no SMs beside one another: 32^3 x 3, calls of one
// step, 8.9 -> 11.7 a step, where one alone takes 21.4 -> 15.3.
#pragma once

#include <cooperative_groups.h>

#include "bfvm_kernels_closed.cuh"

namespace bfvm {

constexpr int kGridThreads = 512;
constexpr int kGridChunk = 8;

// what a voxel has (a byte each)
enum : int { kVoxDirichlet = 1, kVoxBulk = 2, kVoxAgents = 4, kVoxMoreAgents = 8 };

struct GridStepArgs {
  double* p;  // [nz][ny][nx][S]
  int nx, ny, nz, S;
  int nsteps;
  double dt;
  int on;               // kVox* bits that take part
  const double* cst[3]; // constants of the axes (ClosedCoef) for 8-point chunks
  int cst_count[3];     // their lengths; copied to shared memory when staged
  bool staged;
  int sg, groups;       // densities per item, items per plane
  int pitch;            // shared-memory elements between an item's rows
  int tw;               // columns of a z tile: tw x chunks of nz <= kGridThreads
  uint64_t m_sg, m_last, m_nx;  // quot() of sg, of the last item's, of nx,
  uint64_t m_lx, m_ly, m_lx_last, m_ly_last, m_tw;  // of an item's x and y lines, of tw
  // a phase per axis: its columns, the columns of a tile; quot() of those, S, nx S
  bool first;  // the first step's sources in a pass of their own
  int pcols[3], ptw[3];
  uint64_t m_ptw[3], m_S, m_rowS;
  const unsigned char* flags;   // [N]
  // per flagged voxel: its bulk entry; its first agent's place in the sorted
  // list and in the agent list
  const int* bulk_map;
  const int2* ag_map;
  // Dirichlet nodes: per x and y line a mask of the points that are nodes
  // (lines numbered x: k*ny + j, y: k*nx + i), and the node values at their
  // places in a field-shaped array [N][S]
  const unsigned long long* dir_mask_x;
  const unsigned long long* dir_mask_y;
  const double* dir_field;
  const double* bulk_st;    // [E][S] S*T
  const double* bulk_su;    // [E][S] U+S
  int64_t nagents;
  const uint64_t* ag_key;  // sorted voxel keys (stable in list order)
  const int* ag_idx;       // list position of each sorted entry
  const double* ag_t1;     // [A][S] in list order
  const double* ag_t2;
};

// A chunk in registers through the block's fold: L columns, NC (at most 8)
// chunks each, thread (col, c); threads without a chunk (c >= NC) only meet
// the barrier.  cst: the axis's constants, in shared or global memory.
__device__ __forceinline__ void grid_chunk(double (&v)[kGridChunk], int len, const double* cst,
                                           int S, int s, double* sU, double* sW, int L, int NC,
                                           int c, int col) {
  const double2* k = reinterpret_cast<const double2*>(cst) + s * 4;
  const double2 rs = k[0];
  const double r = rs.x;
  if (c < NC) closed_sums<double, kGridChunk, false>(v, len, r, sU[c * L + col], sW[c * L + col]);
  __syncthreads();
  if (c >= NC) return;
  const double2 hrc = k[1], rlrn = k[2];
  double u[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) u[i] = i < NC ? sU[i * L + col] : 0.0;
  double TU = 0.0, q0 = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i == c) q0 = TU;
    if (i < NC) TU = fma(i == NC - 1 ? rlrn.x : hrc.y, TU, u[i]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) u[i] = i < NC ? sW[i * L + col] : 0.0;
  double TW = 0.0, w0 = 0.0;
#pragma unroll
  for (int i = 7; i >= 0; --i) {
    if (i == c) w0 = TW;
    TW = fma(hrc.y, TW, u[i]);
  }
  const double2 pw = reinterpret_cast<const double2*>(cst + (size_t)S * 8)[c * S + s];
  const double inv = k[3].x;
  const double qin = fma(pw.x, fma(rlrn.y, TU, TW) * inv, q0);
  const double vin = fma(pw.y, fma(rlrn.y, TW, TU) * inv, w0);
  closed_solve<double, kGridChunk, false>(v, len, r, {rs.y, 0.0}, {hrc.x, 0.0}, qin, vin);
}

// A plane's values as the x sweep finds them, into shared memory: sources,
// then Dirichlet values, a plane of up to 4096 in one round.  The field,
// which other blocks wrote, is read past L1.
__device__ __forceinline__ void grid_load(const GridStepArgs& a, int64_t vox0, int s0, int sg,
                                          double* plane) {
  constexpr int kMost = 8;
  const int width = a.nx * sg, count = width * a.ny;
  const uint64_t m_sg = sg == a.sg ? a.m_sg : a.m_last;
  for (int first = threadIdx.x; first < count; first += kMost * kGridThreads) {
    double x[kMost];
    int f[kMost], be[kMost];
    int2 ag[kMost];
#pragma unroll
    for (int q = 0; q < kMost; ++q) {
      const int u = first + q * kGridThreads;
      f[q] = 0;
      if (u < count) {
        const int vs = (int)quot(u, m_sg);  // voxel in the plane
        const int64_t vox = vox0 + vs;
        x[q] = __ldcg(a.p + vox * a.S + s0 + (u - vs * sg));
        if (a.on) f[q] = __ldg(a.flags + vox);
        if (a.on & kVoxBulk) be[q] = __ldg(a.bulk_map + vox);
        if (a.on & kVoxAgents) ag[q] = __ldg(a.ag_map + vox);
      }
    }
#pragma unroll
    for (int q = 0; q < kMost; ++q) {
      const int u = first + q * kGridThreads;
      if (u < count) {
        const int vs = (int)quot(u, m_sg), j = (int)quot(vs, a.m_nx);
        const int64_t vox = vox0 + vs;
        const int s = s0 + (u - vs * sg), flags = f[q] & a.on;
        if (flags) {
          if (flags & kVoxBulk) {
            const int64_t e = (int64_t)be[q] * a.S + s;
            x[q] = bulk_update(x[q], __ldg(a.bulk_st + e), __ldg(a.bulk_su + e), a.dt);
          }
          if (flags & kVoxAgents) {
            int64_t e = (int64_t)ag[q].y * a.S + s;
            x[q] = cell_update(x[q], __ldg(a.ag_t1 + e), __ldg(a.ag_t2 + e));
            if (f[q] & kVoxMoreAgents) {
              for (int r = ag[q].x + 1; r < a.nagents && __ldg(a.ag_key + r) == (uint64_t)vox;
                   ++r) {
                e = (int64_t)__ldg(a.ag_idx + r) * a.S + s;
                x[q] = cell_update(x[q], __ldg(a.ag_t1 + e), __ldg(a.ag_t2 + e));
              }
            }
          }
          if (flags & kVoxDirichlet) x[q] = __ldg(a.dir_field + vox * a.S + s);
        }
        plane[j * a.pitch + (u - j * width)] = x[q];
      }
    }
  }
}

// One item of the xy phase.
__device__ __forceinline__ void grid_xy(const GridStepArgs& a, int item, const double* cx,
                                        const double* cy, double* plane, double* sU, double* sW) {
  const int S = a.S, nx = a.nx, ny = a.ny;
  const int k = item / a.groups, s0 = (item - k * a.groups) * a.sg;
  const int sg = min(a.sg, S - s0);
  const uint64_t m_sg = sg == a.sg ? a.m_sg : a.m_last;
  const int64_t vox0 = (int64_t)k * nx * ny;
  const int tid = threadIdx.x;
  // x lines: columns (j, s), which meet distinct banks (pitch = sg mod 16);
  // y lines: columns (i, s)
  const int Lx = ny * sg, NCx = (nx + kGridChunk - 1) / kGridChunk;
  const int Ly = nx * sg, NCy = (ny + kGridChunk - 1) / kGridChunk;
  const int xc = (int)quot(tid, sg == a.sg ? a.m_lx : a.m_lx_last), xcol = tid - xc * Lx, xj = (int)quot(xcol, m_sg);
  const int yc = (int)quot(tid, sg == a.sg ? a.m_ly : a.m_ly_last), ycol = tid - yc * Ly, yi = (int)quot(ycol, m_sg);
  const int xlen = xc < NCx ? min(kGridChunk, nx - xc * kGridChunk) : 0;
  const int ylen = yc < NCy ? min(kGridChunk, ny - yc * kGridChunk) : 0;
  unsigned xnodes = 0, ynodes = 0;
  if (a.on & kVoxDirichlet) {
    if (xlen > 0)
      xnodes = (unsigned)(__ldg(a.dir_mask_x + (int64_t)k * ny + xj) >> (xc * kGridChunk)) & 0xffu;
    if (ylen > 0)
      ynodes = (unsigned)(__ldg(a.dir_mask_y + (int64_t)k * nx + yi) >> (yc * kGridChunk)) & 0xffu;
  }
  grid_load(a, vox0, s0, sg, plane);
  __syncthreads();
  double v[kGridChunk];
  {
    const int s = xcol - xj * sg;
    double* q = plane + xj * a.pitch + xc * kGridChunk * sg + s;
#pragma unroll
    for (int m = 0; m < kGridChunk; ++m) v[m] = m < xlen ? q[m * sg] : 0.0;
    grid_chunk(v, xlen, cx, S, s0 + s, sU, sW, Lx, NCx, xc, xcol);
#pragma unroll
    for (int m = 0; m < kGridChunk; ++m)
      if (m < xlen && !(xnodes >> m & 1u)) q[m * sg] = v[m];
  }
  __syncthreads();
  {
    const int s = ycol - yi * sg;
    const double* q = plane + yc * kGridChunk * a.pitch + ycol;
    double* o = a.p + (vox0 + (int64_t)yc * kGridChunk * nx + yi) * S + s0 + s;
#pragma unroll
    for (int m = 0; m < kGridChunk; ++m) v[m] = m < ylen ? q[m * a.pitch] : 0.0;
    grid_chunk(v, ylen, cy, S, s0 + s, sU, sW, Ly, NCy, yc, ycol);
#pragma unroll
    for (int m = 0; m < kGridChunk; ++m)
      if (m < ylen) o[(int64_t)m * nx * S] = ynodes >> m & 1u ? q[m * a.pitch] : v[m];
  }
}

// One tile of the z phase: TW columns.
__device__ __forceinline__ void grid_z(const GridStepArgs& a, int tile, int TW, const double* cz,
                                       double* sU, double* sW) {
  const int S = a.S, ncols = a.nx * a.ny * S;
  const int NC = (a.nz + kGridChunk - 1) / kGridChunk;
  const int c = (int)quot(threadIdx.x, a.m_tw), tx = threadIdx.x - c * TW;
  const int col = tile * TW + tx;
  const int len = c < NC && col < ncols ? min(kGridChunk, a.nz - c * kGridChunk) : 0;
  const int s = min(col, ncols - 1) % S;
  double* q = a.p + (int64_t)c * kGridChunk * ncols + col;
  double v[kGridChunk];
#pragma unroll
  for (int m = 0; m < kGridChunk; ++m) v[m] = m < len ? __ldcg(q + (int64_t)m * ncols) : 0.0;
  grid_chunk(v, len, cz, S, s, sU, sW, TW, NC, c, tx);
#pragma unroll
  for (int m = 0; m < kGridChunk; ++m)
    if (m < len) q[(int64_t)m * ncols] = v[m];
}

// Doubles of dynamic shared memory before the staged constants: the fold's
// two sums, and the plane.
__host__ __device__ constexpr int grid_smem_doubles(int ny, int pitch) {
  return (2 * kGridThreads + ny * pitch + 1) / 2 * 2;
}

// nsteps whole steps; launched cooperatively (every block resident).
static __global__ void __launch_bounds__(kGridThreads, 1) grid_steps_kernel(const GridStepArgs a) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) double grid_smem[];
  double* sU = grid_smem;
  double* sW = sU + kGridThreads;
  double* plane = sW + kGridThreads;
  const double* cst[3] = {a.cst[0], a.cst[1], a.cst[2]};
  if (a.staged) {
    double* t = grid_smem + grid_smem_doubles(a.ny, a.pitch);
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      for (int i = threadIdx.x; i < a.cst_count[ax]; i += kGridThreads) t[i] = __ldg(cst[ax] + i);
      cst[ax] = t;
      t += a.cst_count[ax];  // an even number
    }
  }
  const int items = a.nz * a.groups;
  const int TW = a.tw;
  const int tiles = (a.nx * a.ny * a.S + TW - 1) / TW;
  for (int step = 0; step < a.nsteps; ++step) {
    // (the barrier after a plane's load also completes the staging above)
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
      grid_xy(a, i, cst[0], cst[1], plane, sU, sW);
      __syncthreads();  // the fold and the plane are free again
    }
    grid.sync();
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      grid_z(a, t, TW, cst[2], sU, sW);
      __syncthreads();
    }
    if (step + 1 < a.nsteps) grid.sync();
  }
}

// ---------------------------------------------------------------------------
// The same steps with a phase per axis, every line straight from and to the
// field: a block takes tw columns x chunks of the axis.  The sources and
// Dirichlet values of a step are applied as the z phase before it stores its
// points, the first step's as its x lines load.  At a node the x and y lines
// store nothing, so its value stays through both.  UPD: the steps have any of
// them.
//
// A barrier more a step, but the work splits finer than whole planes: for few
// wide planes, where a thread of the planes' blocks takes up to eight voxels'
// source chains (64 x 64 x 1 with 1000 agents and bulk rates 21.6 -> 13.6 us a
// step), and for more planes than SMs, whose second wave is mostly empty
// (50^3 x 4 with the same sources 28.2 -> 17.8, without 19.5 -> 13.6).  With
// 1000 agents and a fixed boundary, 100 steps in a call: 50^3 x 4 23.6 -> 15.1
// (22.7 with the three phases and tables mentioned above), 43^3 x 6 22.6 -> 15.2
// (22.1), 64 x 64 x 2 x 20 24.8 -> 14.8 (17.8), 64 x 64 x 1 x 1 18.7 -> 12.7 (12.4).
// bfvm_solver.cu's grid_phases_better has the rule.

constexpr int kPhaseThreads = 256;
template <int AX>
struct Axis3 {
  static constexpr int value = AX;
};

// Sources and Dirichlet values of a thread's points of one line: vox0 the voxel
// of its first point, vstep between points.  The points' maps come in one
// round trip.  Agents after a voxel's first one follow in a loop of their own,
// in which a lane goes on to its next such point without waiting for the
// warp's others.  (Fetching every constant of four points at once spills, and
// is slower everywhere: 64 x 64 x 2 x 4 14.1 -> 15.7 us a step.)
__device__ __forceinline__ void grid_update(const GridStepArgs& a, double (&x)[kGridChunk], int len,
                                            int vox0, int vstep, int s) {
  int f[kGridChunk], be[kGridChunk], ag[kGridChunk];
#pragma unroll
  for (int m = 0; m < kGridChunk; ++m) {
    const int vox = vox0 + m * vstep;
    f[m] = m < len ? __ldg(a.flags + vox) : 0;
    if (m < len && (a.on & kVoxBulk)) be[m] = __ldg(a.bulk_map + vox);
    if (m < len && (a.on & kVoxAgents)) ag[m] = __ldg(&a.ag_map[vox].y);
  }
  unsigned more = 0;
#pragma unroll
  for (int m = 0; m < kGridChunk; ++m) {
    const int flags = f[m] & a.on;
    if (flags & kVoxDirichlet) {
      x[m] = __ldg(a.dir_field + (int64_t)(vox0 + m * vstep) * a.S + s);
    } else if (flags) {
      if (flags & kVoxBulk) {
        const int64_t e = (int64_t)be[m] * a.S + s;
        x[m] = bulk_update(x[m], __ldg(a.bulk_st + e), __ldg(a.bulk_su + e), a.dt);
      }
      if (flags & kVoxAgents) {
        const int64_t e = (int64_t)ag[m] * a.S + s;
        x[m] = cell_update(x[m], __ldg(a.ag_t1 + e), __ldg(a.ag_t2 + e));
        if (f[m] & kVoxMoreAgents) more |= 1u << m;
      }
    }
  }
  int m = -1, r = 0;
  uint64_t vox = 0;
  double v = 0.0;
  while (m >= 0 || more) {
    if (m < 0) {
      m = __ffs(more) - 1;
      more &= more - 1;
      vox = (uint64_t)(vox0 + m * vstep);
      r = __ldg(&a.ag_map[vox].x) + 1;
      v = reg_get<double, kGridChunk>(x, m);
    }
    const int64_t e = (int64_t)__ldg(a.ag_idx + r) * a.S + s;
    const bool last = r + 1 >= a.nagents || __ldg(a.ag_key + r + 1) != vox;
    v = cell_update(v, __ldg(a.ag_t1 + e), __ldg(a.ag_t2 + e));
    ++r;
    if (last) {
      reg_set<double, kGridChunk>(x, m, v);
      m = -1;
    }
  }
}

// The same for the whole field, an element per thread: with few elements to a
// thread shorter than eight in a row, though it takes a barrier more.
__device__ __forceinline__ void grid_update_first(const GridStepArgs& a) {
  const int count = a.nx * a.ny * a.nz * a.S;
  for (int w = blockIdx.x * kPhaseThreads + threadIdx.x; w < count;
       w += gridDim.x * kPhaseThreads) {
    const int vox = (int)quot(w, a.m_S), s = w - vox * a.S;
    const int flags = __ldg(a.flags + vox) & (a.on | kVoxMoreAgents);
    if (!(flags & a.on)) continue;
    double x = a.p[w];
    if (flags & kVoxDirichlet) {
      x = __ldg(a.dir_field + w);
    } else {
      if (flags & kVoxBulk) {
        const int64_t e = (int64_t)__ldg(a.bulk_map + vox) * a.S + s;
        x = bulk_update(x, __ldg(a.bulk_st + e), __ldg(a.bulk_su + e), a.dt);
      }
      if (flags & kVoxAgents) {
        const int2 first = __ldg(a.ag_map + vox);
        int64_t e = (int64_t)first.y * a.S + s;
        x = cell_update(x, __ldg(a.ag_t1 + e), __ldg(a.ag_t2 + e));
        if (flags & kVoxMoreAgents)
          for (int r = first.x + 1; r < a.nagents && __ldg(a.ag_key + r) == (uint64_t)vox; ++r) {
            e = (int64_t)__ldg(a.ag_idx + r) * a.S + s;
            x = cell_update(x, __ldg(a.ag_t1 + e), __ldg(a.ag_t2 + e));
          }
      }
    }
    a.p[w] = x;
  }
}

template <int AX, bool UPD>
__device__ __forceinline__ void grid_lines(const GridStepArgs& a, int tile, const double* cst,
                                           bool update, double* sU, double* sW) {
  const int S = a.S, plane = a.nx * a.ny, n = AX == 0 ? a.nx : (AX == 1 ? a.ny : a.nz);
  const int ncols = a.pcols[AX], TW = a.ptw[AX], NC = (n + kGridChunk - 1) / kGridChunk;
  const int c = (int)quot(threadIdx.x, a.m_ptw[AX]), tx = threadIdx.x - c * TW;
  const int col = tile * TW + tx, vcol = min(col, ncols - 1);
  const int len = c < NC && col < ncols ? min(kGridChunk, n - c * kGridChunk) : 0;
  const int l = (int)quot(vcol, a.m_S), s = vcol - l * S;  // line (k, j), (k, i) or (j, i)
  int64_t off;     // of the line's first point
  int ls;          // between its points
  int vox0, vstep; // voxels likewise
  if (AX == 0) {
    off = (int64_t)l * a.nx * S + s, ls = S, vox0 = l * a.nx, vstep = 1;
  } else if (AX == 1) {
    const int k = (int)quot(vcol, a.m_rowS), in = vcol - k * a.nx * S;
    off = (int64_t)k * plane * S + in, ls = a.nx * S, vox0 = 0, vstep = 0;
  } else {
    off = vcol, ls = plane * S, vox0 = l, vstep = plane;
  }
  const int k0 = c * kGridChunk;
  unsigned nodes = 0;
  if (UPD && AX < 2 && (a.on & kVoxDirichlet) && len > 0)
    nodes = (unsigned)(__ldg((AX == 0 ? a.dir_mask_x : a.dir_mask_y) + l) >> k0) & 0xffu;
  double* q = a.p + off + (int64_t)k0 * ls;
  double v[kGridChunk];
#pragma unroll
  for (int m = 0; m < kGridChunk; ++m)
    v[m] = m < len ? (AX == 0 ? q[m * ls] : __ldcg(q + m * ls)) : 0.0;
  if (UPD && AX == 0 && update) {
    grid_update(a, v, len, vox0 + k0 * vstep, vstep, s);
#pragma unroll
    for (int m = 0; m < kGridChunk; ++m)
      if (nodes >> m & 1u) q[m * ls] = v[m];
  }
  grid_chunk(v, len, cst, S, s, sU, sW, TW, NC, c, tx);
  if (UPD && AX == 2 && update) grid_update(a, v, len, vox0 + k0 * vstep, vstep, s);
#pragma unroll
  for (int m = 0; m < kGridChunk; ++m)
    if (m < len && !(nodes >> m & 1u)) q[m * ls] = v[m];
}

template <bool UPD>
__global__ void __launch_bounds__(kPhaseThreads, 2)
    grid_phases_kernel(const GridStepArgs a) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) double grid_smem[];
  double* sU = grid_smem;
  double* sW = sU + kPhaseThreads;
  const double* cst[3] = {a.cst[0], a.cst[1], a.cst[2]};
  if (a.staged) {
    double* t = grid_smem + 2 * kPhaseThreads;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      for (int i = threadIdx.x; i < a.cst_count[ax]; i += kPhaseThreads) t[i] = __ldg(cst[ax] + i);
      cst[ax] = t;
      t += a.cst_count[ax];
    }
    __syncthreads();
  }
  auto phase = [&](auto ax, bool update) {
    constexpr int AX = decltype(ax)::value;
    const int tiles = (a.pcols[AX] + a.ptw[AX] - 1) / a.ptw[AX];
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
      grid_lines<AX, UPD>(a, t, cst[AX], update, sU, sW);
      __syncthreads();  // the fold is free again
    }
  };
  if (UPD && a.first) {
    grid_update_first(a);
    grid.sync();
  }
  for (int step = 0; step < a.nsteps; ++step) {
    const bool more = step + 1 < a.nsteps;
    phase(Axis3<0>(), a.on && step == 0 && !a.first);
    grid.sync();
    phase(Axis3<1>(), false);
    grid.sync();
    phase(Axis3<2>(), a.on && more);
    if (more) grid.sync();
  }
}

// Dense voxel maps of the bulk entries and of the first agent of each voxel
// in the sorted list, the voxels' flags, and the Dirichlet nodes' line masks
// (flags and masks 0 beforehand) and values at their places in the field.
// Entries of the maps that no flag points to are not written.
static __global__ void grid_maps_kernel(int* __restrict__ bulk_map, int2* __restrict__ ag_map,
                                        unsigned* __restrict__ flag_words, int64_t nbulk,
                                        const int64_t* __restrict__ bulk_vox, int64_t nagents,
                                        const uint64_t* __restrict__ ag_key,
                                        const int* __restrict__ ag_idx, int64_t ndir,
                                        const int64_t* __restrict__ dir_vox,
                                        const double* __restrict__ dir_val,
                                        unsigned long long* __restrict__ mx,
                                        unsigned long long* __restrict__ my,
                                        double* __restrict__ dir_field, int nx, int ny, int S) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  auto flag = [&](int64_t v, int bits) {
    atomicOr(flag_words + (v >> 2), (unsigned)bits << (8 * (v & 3)));
  };
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
       i < nbulk || i < nagents || i < ndir; i += stride) {
    if (i < nbulk) {
      bulk_map[bulk_vox[i]] = (int)i;
      flag(bulk_vox[i], kVoxBulk);
    }
    if (i < nagents && (i == 0 || ag_key[i] != ag_key[i - 1])) {
      const uint64_t v = ag_key[i];
      ag_map[v] = make_int2((int)i, ag_idx[i]);
      flag((int64_t)v,
           i + 1 < nagents && ag_key[i + 1] == v ? kVoxAgents | kVoxMoreAgents : kVoxAgents);
    }
    if (i < ndir) {
      const int64_t v = dir_vox[i];
      const int64_t plane = (int64_t)nx * ny;
      const int64_t k = v / plane, ij = v - k * plane, j = ij / nx, ii = ij - j * nx;
      flag(v, kVoxDirichlet);
      atomicOr(mx + k * ny + j, 1ull << ii);
      atomicOr(my + k * nx + ii, 1ull << j);
      for (int s = 0; s < S; ++s) dir_field[v * S + s] = dir_val[i * S + s];
    }
  }
}

}  // namespace bfvm
