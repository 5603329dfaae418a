// Kernels of the adjoint (reverse-mode derivative) of the transport step.
//
// One forward step (FP64) is  p1 = bulk(p0);  p2 = cells(p1);
// p3 = D(p2), y_x = A_x^-1 p3;  p5 = D(y_x), y_y = A_y^-1 p5;
// p7 = D(y_y), y_z = A_z^-1 p7  (BioFVM_solvers.cpp:175-273), where D
// overwrites the Dirichlet nodes and A_a = (1 + c2) I + c1 L_a with L_a the
// Neumann Laplacian along axis a (diagonal 2, 1 at the line ends, -1 off the
// diagonal; 0 for a one-point line), c1 = dt D / dx^2, c2 = dt decay / 3
// (BioFVM_solvers.cpp:105-142).  A_a is symmetric, so the adjoint of a solve
// is the same solve, and the derivative of the loss with respect to c1 (c2)
// through one solve y = A^-1 x is -abar . (L y)  (-abar . y), abar = A^-1 ybar.
#pragma once

#include "bfvm_kernels_closed.cuh"

namespace bfvm {

// Adds a block's sums of a*(L y) and a*y to part[block][2S]: blockDim.x is a
// multiple of S and thread t holds density t % S.  part accumulates over every
// solve of a backward run (zeroed at its start, reduced once at its end); the
// order of every sum is fixed.
static __device__ __forceinline__ void adj_add_part(double accL, double accI, int S,
                                                    double* __restrict__ part) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double* sL = reinterpret_cast<double*>(smem_raw);  // [blockDim.x]
  double* sI = sL + blockDim.x;
  const int t = threadIdx.x;
  sL[t] = accL;
  sI[t] = accI;
  for (int g = blockDim.x / S; g > 1;) {  // threads S apart, halved
    const int half = (g + 1) / 2;
    __syncthreads();
    if (t < (g - half) * S) {
      sL[t] += sL[t + half * S];
      sI[t] += sI[t + half * S];
    }
    g = half;
  }
  if (t < S) {
    part[(int64_t)blockIdx.x * 2 * S + t] += sL[t];
    part[(int64_t)blockIdx.x * 2 * S + S + t] += sI[t];
  }
}

// Per-substrate sums over the field of a*(L_x y) and a*y.  Blocks take whole
// rows (fixed y, z: nx*S contiguous elements), block b the rows b, b +
// gridDim.x, ...; thread t steps through x = t / S, t / S + blockDim.x / S, ...
// of each row.  The neighbours' loads hit L1, and threads, not loads per
// thread, keep memory busy: 27.2 us at 128^3 x 4, against 30.4 with four rows
// a thread at half the resident threads.
static __global__ void adj_x_dot_kernel(const double* __restrict__ a, const double* __restrict__ y,
                                        int nx, int64_t rows, int S, double* __restrict__ part) {
  const int t = threadIdx.x, s = t % S, xstep = blockDim.x / S;
  double accL = 0.0, accI = 0.0;
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const double* yr = y + r * nx * S;
    const double* ar = a + r * nx * S;
    for (int x = t / S; x < nx; x += xstep) {
      const int64_t c = (int64_t)x * S + s;
      const double yv = yr[c];
      double ly = 0.0;
      if (x > 0) ly += yv - yr[c - S];
      if (x < nx - 1) ly += yv - yr[c + S];
      const double av = ar[c];
      accL += av * ly;
      accI += av * yv;
    }
  }
  adj_add_part(accL, accI, S, part);
}

// The y or z axis's layout for its dot products: columns of n points, `ls`
// apart, cut into segments of kDotPoints; an item is one segment of one
// column, columns innermost.  (An adjoint run holds six fields, so a field and
// its items count below 2^32.)
struct DotAxis {
  uint32_t C, items;  // columns per outer index; segments in all
  uint64_t mC, mSeg;  // quot() of C, of the segments per column
  int nseg, n;
  int64_t ls, os;
};
constexpr int kDotPoints = 8;

// The same sums along y or z.  C is a multiple of S, so a thread keeps the
// density threadIdx.x % S.  Bound by memory: y comes from HBM, a from the sweep
// before it.  A point at a time, with its neighbours, leaves four loads in
// flight per thread and reads y three times through L2; a segment's 18 loads
// go out together and a neighbour is the segment's own next point: 29.5 (y)
// and 30.6 (z) -> 25.2 us at 128^3 x 4.
static __global__ void __launch_bounds__(256, 4)
    adj_axis_dot_kernel(const double* __restrict__ a, const double* __restrict__ y, DotAxis d,
                        int S, double* __restrict__ part) {
  constexpr int K = kDotPoints;
  const int t = threadIdx.x, B = blockDim.x;
  double accL = 0.0, accI = 0.0;
  for (uint64_t w = (uint64_t)blockIdx.x * B + t; w < d.items; w += (uint64_t)gridDim.x * B) {
    const uint32_t id = (uint32_t)w, rest = quot(id, d.mC), col = id - rest * d.C;
    const uint32_t outer = quot(rest, d.mSeg);
    const int k0 = (int)(rest - outer * d.nseg) * K;
    const int64_t off = (int64_t)outer * d.os + (int64_t)k0 * d.ls + col;
    const int len = d.n - k0;  // points left in the column
    double yv[K], av[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int64_t q = off + k * d.ls;
      yv[k] = k < len ? y[q] : 0.0;
      av[k] = k < len ? a[q] : 0.0;
    }
    const double before = k0 > 0 ? y[off - d.ls] : 0.0;
    const double after = len > K ? y[off + K * d.ls] : 0.0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double ly = 0.0;
      if (k > 0 || k0 > 0) ly += yv[k] - (k > 0 ? yv[k - 1] : before);
      if (k + 1 < len) ly += yv[k] - (k + 1 < K ? yv[k + 1] : after);
      if (k < len) {
        accL += av[k] * ly;
        accI += av[k] * yv[k];
      }
    }
  }
  adj_add_part(accL, accI, S, part);
}

// acc[j] -= sum over blocks of part[.][j], one block of kAdjReduceThreads
// per output j in [0, 2S) (thread i sums blocks i, i + kAdjReduceThreads, ...,
// then a fixed tree): the solves' contributions -a.(L y) and -a.y.
constexpr int kAdjReduceThreads = 256;
static __global__ void __launch_bounds__(kAdjReduceThreads)
    adj_reduce_parts_kernel(const double* __restrict__ part, int blocks, int S,
                            double* __restrict__ acc) {
  __shared__ double sm[kAdjReduceThreads];
  const int j = blockIdx.x, i = threadIdx.x;
  double sum = 0.0;
  for (int b = i; b < blocks; b += kAdjReduceThreads) sum += part[(int64_t)b * 2 * S + j];
  sm[i] = sum;
  __syncthreads();
  for (int w = kAdjReduceThreads / 2; w > 0; w >>= 1) {
    if (i < w) sm[i] += sm[i + w];
    __syncthreads();
  }
  if (i == 0) acc[j] -= sm[0];
}

// a = 0 at the Dirichlet nodes (the adjoint of the overwrite).
static __global__ void adj_zero_nodes_kernel(double* __restrict__ a, int S, int64_t E,
                                      const int64_t* __restrict__ voxel) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  a[voxel[e] * S + s] = 0.0;
}

// Adjoint of the bulk update p1 = (p0 + dt S T) / ((U + S) dt + 1): a /= the
// same denominator, on the listed voxels.
static __global__ void adj_bulk_kernel(double* __restrict__ a, int S, int64_t E,
                                const int64_t* __restrict__ voxel, const double* __restrict__ su,
                                double dt) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  const int64_t q = voxel[e] * S + s;
  a[q] = __ddiv_rn(a[q], __dadd_rn(__dmul_rn(su[t], dt), 1.0));
}

// brow[r] = the bulk list's entry (sorted by voxel) of sorted agent r's voxel,
// -1 where it is not listed.
static __global__ void adj_bulk_rows_kernel(int64_t A, const uint64_t* __restrict__ key,
                                            int64_t nbulk, const int64_t* __restrict__ bulk_vox,
                                            int64_t* __restrict__ brow) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= A) return;
  const uint64_t v = key[r];
  int64_t lo = 0, hi = nbulk - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((uint64_t)bulk_vox[mid] < v)
      lo = mid + 1;
    else
      hi = mid;
  }
  brow[r] = (uint64_t)bulk_vox[lo] == v ? lo : -1;
}

// Adjoint of the cell updates of one voxel (agents in list order,
// x_j = (x_{j-1} + t1_j) / t2_j, BioFVM_basic_agent.cpp:234-235): the
// thread of the first sorted agent of a voxel recomputes the chain from the
// step input (after the bulk update when bulk ran: brow is not null), then
// walks it backwards:
//   gt1_j += g / t2_j,  gt2_j -= g x_j / t2_j,  g /= t2_j,
// recovering x_{j-1} = x_j t2_j - t1_j.  gt1/gt2 are [A][S] in list order.
//
// Bound by latency: the keys, the list position and the bulk entry come in one
// round trip and every operand of the voxel's first agent in a second, where a
// search of the bulk list per step took up to 20 dependent loads: 14.8 -> 7.3
// us for 20,000 agents x 4 among 113,000 bulk voxels.
static __global__ void adj_cells_kernel(double* __restrict__ a, const double* __restrict__ p_in, int S,
                                 int64_t A, const uint64_t* __restrict__ key,
                                 const int* __restrict__ idx, const double* __restrict__ t1,
                                 const double* __restrict__ t2, const int64_t* __restrict__ brow,
                                 const double* __restrict__ bulk_st,
                                 const double* __restrict__ bulk_su, double dt,
                                 double* __restrict__ gt1, double* __restrict__ gt2) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A * S) return;
  const int64_t r = t / S;
  const int s = (int)(t - r * S);
  const uint64_t none = ~(uint64_t)0;  // no voxel's key
  const uint64_t v = key[r], before = r > 0 ? key[r - 1] : none,
                 after = r + 1 < A ? key[r + 1] : none;
  const int64_t i0 = (int64_t)idx[r] * S + s, b = brow ? brow[r] : -1;
  if (before == v) return;
  const int64_t q = (int64_t)v * S + s;
  double x = p_in[q], g = a[q];
  const double f1 = t1[i0], f2 = t2[i0], h1 = gt1[i0], h2 = gt2[i0];
  if (b >= 0) x = bulk_update(x, bulk_st[b * S + s], bulk_su[b * S + s], dt);
  x = cell_update(x, f1, f2);
  if (after == v) {
    int64_t end = r + 1;
    while (end < A && key[end] == v) {
      const int64_t i = idx[end];
      x = cell_update(x, t1[i * S + s], t2[i * S + s]);
      ++end;
    }
    for (int64_t e = end - 1; e > r; --e) {
      const int64_t i = idx[e];
      const double b1 = t1[i * S + s], b2 = t2[i * S + s];
      gt1[i * S + s] += g / b2;
      gt2[i * S + s] -= g * x / b2;
      g = g / b2;
      x = x * b2 - b1;
    }
  }
  gt1[i0] = h1 + g / f2;
  gt2[i0] = h2 - g * x / f2;
  a[q] = g / f2;
}

}  // namespace bfvm
