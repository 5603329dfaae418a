// Device kernels of the B200 transport path.
//
// Density field: one array [nz][ny][nx][S] (substrate innermost), the
// reference's logical [voxel][substrate] order made contiguous.
//
// LOD sweep (BioFVM_solvers.cpp:175-273).  Along one axis every (line,
// substrate) pair is an independent tridiagonal system solved by the Thomas
// algorithm with precomputed coefficients:
//   forward   q_0 = p_0/d_0,  q_k = (p_k + c1*q_{k-1})/d_k     (:186-194)
//   backward  x_{n-1} = q_{n-1},  x_k = q_k - cx_k*x_{k+1}       (:196-200)
// Both are first-order linear recurrences, so a line is cut into chunks of
// CH points, one chunk per thread, held in registers:
//   1. each thread runs the recurrence over its chunk with carry-in 0 and
//      records the chunk's transfer (end value, product of slopes);
//   2. the transfers of the chunks of one line are folded through shared
//      memory to give every chunk its true carry-in;
//   3. each thread corrects its chunk: value += (running slope product)*carry.
// Every density element is read once and written once per sweep.
//
// A thread block is TW columns x NC chunks (blockDim = (TW, NC)); a
// "column" is one (line, substrate) pair and consecutive columns are
// consecutive addresses for the y and z sweeps, so every warp load/store is a
// contiguous TW*sizeof(T) run.  For the x sweep the S substrates of a row are
// the contiguous run.
//
// The x sweep also carries the rest of the step in its prologue: bulk
// sources/sinks, then cell sources/sinks (agents in reference order), then
// the Dirichlet overwrite; its epilogue is the Dirichlet overwrite that the
// reference does before the y sweep, and the y sweep's epilogue is the one
// before the z sweep.  These per-voxel updates use the same IEEE operations
// in the same order as the reference (no FMA contraction), so they are
// bit-exact; only the sweeps' rounding differs.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace bfvm {

enum : int {
  kFuseBulk = 1,
  kFuseCells = 2,
  kFuseDirPro = 4,   // Dirichlet before the sweep
  kFuseDirEpi = 8,   // Dirichlet after the sweep (= before the next axis)
};

// Coefficients of one axis, [n][S] each, in the sweep's precision.
template <typename T>
struct AxisCoef {
  const T* inv_den;  // 1 / thomas_denom
  const T* fwd;      // c1 / thomas_denom: slope of the forward recurrence
  const T* bwd;      // -thomas_c: slope of the back substitution
  const T* c1;       // [S] dt*D/dx^2
};

// Entries grouped by (line, chunk) segment: off[line*NC + c] .. off[+1].
// pos = point index along the line; a/b = per-substrate payload [E][S].
struct SegList {
  const int* off = nullptr;
  const int* pos = nullptr;
  const double* a = nullptr;
  const double* b = nullptr;
};

// T: the field's element type; CT: the type the sweep computes in (CT = T,
// or double over a float field).
template <typename T, typename CT = T>
struct SweepArgs {
  T* p;
  T* out;                // where the solved lines go (p: in place)
  int64_t col0;          // first column of this launch (a slab of planes)
  int64_t ncols;         // end of the launch's columns (all (line, substrate) columns)
  int64_t C;             // columns per outer block
  int64_t outer_stride;  // elements between outer blocks
  int64_t line_stride;   // elements between consecutive points of a line
  int n;                 // points per line
  int nchunks;           // NC = ceil(n / CH)
  int S;
  AxisCoef<CT> coef;
  SegList bulk, cells, dir_pro, dir_epi;
  double dt;
  int fuse;
};

template <typename T, int CH>
__device__ __forceinline__ T reg_get(const T (&v)[CH], int m) {
  T r = v[0];
#pragma unroll
  for (int q = 1; q < CH; ++q) r = (q == m) ? v[q] : r;
  return r;
}

template <typename T, int CH>
__device__ __forceinline__ void reg_set(T (&v)[CH], int m, T x) {
#pragma unroll
  for (int q = 0; q < CH; ++q) v[q] = (q == m) ? x : v[q];
}

// Bulk update of one voxel-substrate (BioFVM_microenvironment.cpp:603-609):
// p += dt*(S*T); p /= (U+S)*dt + 1.  st = S*T and su = U+S are stored.
__device__ __forceinline__ double bulk_update(double x, double st, double su, double dt) {
  x = __dadd_rn(x, __dmul_rn(dt, st));
  return __ddiv_rn(x, __dadd_rn(__dmul_rn(su, dt), 1.0));
}

// One agent's update (BioFVM_basic_agent.cpp:234-235): p += temp1; p /= temp2.
__device__ __forceinline__ double cell_update(double x, double t1, double t2) {
  return __ddiv_rn(__dadd_rn(x, t1), t2);
}

template <typename T, int CH>
__device__ __forceinline__ void apply_dirichlet_seg(T (&v)[CH], const SegList& L, int64_t seg,
                                                    int k0, int S, int s) {
  const int e0 = __ldg(L.off + seg), e1 = __ldg(L.off + seg + 1);
  for (int e = e0; e < e1; ++e) {
    const int m = __ldg(L.pos + e) - k0;
    reg_set<T, CH>(v, m, (T)__ldg(L.a + (int64_t)e * S + s));
  }
}

// MODE selects the fused work: kSweepPlain (z), kSweepDirEpi (y: Dirichlet
// after the sweep), kSweepFull (x: bulk/cells/Dirichlet prologue + Dirichlet
// epilogue, each switched by SweepArgs::fuse).  Separate instantiations keep
// the plain sweeps free of the prologue's registers.
enum : int { kSweepPlain = 0, kSweepDirEpi = 1, kSweepFull = 2 };

// MINB = minimum resident blocks per SM requested from the compiler (1 or 2):
// 2 caps registers at 64 per thread so two 512-thread blocks fit an SM.
// Largest block of lod_sweep_kernel for a chunk length: 32-point chunks keep
// 256 threads so that each thread has the registers for its chunk.
constexpr int sweep_max_threads(int ch) { return ch >= 32 ? 256 : 512; }

template <typename T, int CH, int MODE, int MINB, typename CT = T>
__global__ void __launch_bounds__(sweep_max_threads(CH), MINB)
    lod_sweep_kernel(const SweepArgs<T, CT> a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int TW = blockDim.x;
  const int NC = blockDim.y;
  CT* sQ = reinterpret_cast<CT*>(smem_raw);  // [NC][TW] forward chunk end values
  CT* sP = sQ + NC * TW;                    // forward chunk slope products
  CT* sX = sP + NC * TW;                    // backward chunk start values
  CT* sR = sX + NC * TW;                    // backward chunk slope products

  const int tx = threadIdx.x;
  const int c = threadIdx.y;
  const int64_t vcol = a.col0 + (int64_t)blockIdx.x * TW + tx;
  const bool active = vcol < a.ncols;
  const int S = a.S;
  const int k0 = c * CH;
  // points of this chunk that exist (partial last chunk, empty chunks)
  const int len = active ? max(0, min(CH, a.n - k0)) : 0;

  T* ptr = a.p;
  int s = 0;
  int64_t seg = 0;
  if (active) {
    const int64_t outer = vcol / a.C;
    const int64_t col = vcol - outer * a.C;
    ptr = a.p + outer * a.outer_stride + col + (int64_t)k0 * a.line_stride;
    s = (int)(col % S);
    seg = (vcol / S) * a.nchunks + c;
  }
  const int64_t ls = a.line_stride;

  CT v[CH];
#pragma unroll
  for (int m = 0; m < CH; ++m) v[m] = (m < len) ? (CT)ptr[m * ls] : CT(0);

  if (MODE == kSweepFull && active) {
    if (a.fuse & kFuseBulk) {
      const int e0 = __ldg(a.bulk.off + seg), e1 = __ldg(a.bulk.off + seg + 1);
      for (int e = e0; e < e1; ++e) {
        const int m = __ldg(a.bulk.pos + e) - k0;
        const int64_t q = (int64_t)e * S + s;
        double x = (double)reg_get<CT, CH>(v, m);
        x = bulk_update(x, __ldg(a.bulk.a + q), __ldg(a.bulk.b + q), a.dt);
        reg_set<CT, CH>(v, m, (CT)x);
      }
    }
    if (a.fuse & kFuseCells) {
      // Agents of this chunk sorted by (voxel, list order): applying them in
      // sequence keeps the reference's order for agents sharing a voxel.
      // Consecutive agents of one voxel accumulate in FP64 before rounding.
      const int e0 = __ldg(a.cells.off + seg), e1 = __ldg(a.cells.off + seg + 1);
      int e = e0;
      while (e < e1) {
        const int pos = __ldg(a.cells.pos + e);
        const int m = pos - k0;
        double x = (double)reg_get<CT, CH>(v, m);
        do {
          const int64_t q = (int64_t)e * S + s;
          x = cell_update(x, __ldg(a.cells.a + q), __ldg(a.cells.b + q));
          ++e;
        } while (e < e1 && __ldg(a.cells.pos + e) == pos);
        reg_set<CT, CH>(v, m, (CT)x);
      }
    }
    if (a.fuse & kFuseDirPro) apply_dirichlet_seg<CT, CH>(v, a.dir_pro, seg, k0, S, s);
  }

  // Coefficient rows of this chunk: [k][S] tables, stride S along the line.
  const CT* c_inv = a.coef.inv_den + (int64_t)k0 * S + s;
  const CT* c_fwd = a.coef.fwd + (int64_t)k0 * S + s;
  const CT* c_bwd = a.coef.bwd + (int64_t)k0 * S + s;

  // ---- forward elimination, chunk-local with carry-in 0 ----
  const CT c1 = active ? __ldg(a.coef.c1 + s) : CT(0);
  CT q = CT(0), P = CT(1);
#pragma unroll
  for (int m = 0; m < CH; ++m) {
    if (m < len) {
      q = (v[m] + c1 * q) * __ldg(c_inv + m * S);
      P = P * __ldg(c_fwd + m * S);
      v[m] = q;
    }
  }
  sQ[c * TW + tx] = q;
  sP[c * TW + tx] = P;
  __syncthreads();
  if (c > 0 && len > 0) {
    CT carry = CT(0);
    for (int cc = 0; cc < c; ++cc) carry = sP[cc * TW + tx] * carry + sQ[cc * TW + tx];
    CT Pm = CT(1);
#pragma unroll
    for (int m = 0; m < CH; ++m) {
      if (m < len) {
        Pm = Pm * __ldg(c_fwd + m * S);
        v[m] = v[m] + Pm * carry;
      }
    }
  }

  // ---- back substitution, chunk-local with carry-in 0 ----
  CT x = CT(0), R = CT(1);
#pragma unroll
  for (int m = CH - 1; m >= 0; --m) {
    if (m < len) {
      const CT b = __ldg(c_bwd + m * S);
      x = v[m] + b * x;
      R = R * b;
      v[m] = x;
    }
  }
  sX[c * TW + tx] = x;
  sR[c * TW + tx] = R;
  __syncthreads();
  if (c < NC - 1 && len > 0) {
    CT carry = CT(0);
    for (int cc = NC - 1; cc > c; --cc) carry = sR[cc * TW + tx] * carry + sX[cc * TW + tx];
    CT Rm = CT(1);
#pragma unroll
    for (int m = CH - 1; m >= 0; --m) {
      if (m < len) {
        Rm = Rm * __ldg(c_bwd + m * S);
        v[m] = v[m] + Rm * carry;
      }
    }
  }

  if (MODE != kSweepPlain && active && (a.fuse & kFuseDirEpi))
    apply_dirichlet_seg<CT, CH>(v, a.dir_epi, seg, k0, S, s);

  T* dst = a.out + (ptr - a.p);
#pragma unroll
  for (int m = 0; m < CH; ++m)
    if (m < len) dst[m * ls] = (T)v[m];
}

// ---------------------------------------------------------------------------
// Stand-alone per-voxel kernels (the individual simulate_* / apply_* calls).

// simulate_bulk_sources_and_sinks over the stored (non-identity) voxels.
template <typename T>
__global__ void bulk_kernel(T* __restrict__ p, int S, int64_t E, const int64_t* __restrict__ voxel,
                            const double* __restrict__ st, const double* __restrict__ su,
                            double dt) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  const int64_t q = voxel[e] * S + s;
  p[q] = (T)bulk_update((double)p[q], st[t], su[t], dt);
}

// The same update with the coefficient rows shared between voxels: voxel
// e's (S*T, U+S) for density s are tab[(row[e]*S + s)*2 + {0,1}] (the table
// is small and stays in L1), so the stream is the density itself plus 8 B
// per listed voxel.
template <typename T>
__global__ void bulk_rows_kernel(T* __restrict__ p, int S, int64_t E,
                                 const int* __restrict__ voxel, const int* __restrict__ row,
                                 const double* __restrict__ tab, double dt) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  const int64_t q = (int64_t)__ldg(voxel + e) * S + s;
  const double* c = tab + ((int64_t)__ldg(row + e) * S + s) * 2;
  p[q] = (T)bulk_update((double)p[q], __ldg(c), __ldg(c + 1), dt);
}

// x / d, correctly rounded, for a divisor used many times: with y = 1/d
// rounded to nearest, one step from x y gives a faithful quotient q, and a
// second one, q + y (x - d q) with the exact remainder, rounds it correctly
// (Markstein, IBM J. Res. Dev. 34, 1990).  The proof needs no over- or
// underflow on the way: the exponent of x within +-900 (and d within 2^+-66,
// which the callers see to); other x take the general division.
struct Divisor {
  double d, y;
};
__device__ __forceinline__ double div_fast(double x, const Divisor& v) {
  double q = x * v.y;
  q = fma(fma(-q, v.d, x), v.y, q);
  return fma(fma(-q, v.d, x), v.y, q);
}
__device__ __forceinline__ bool div_safe(double x) {
  const uint32_t e = ((uint32_t)__double2hiint(x) >> 20) & 0x7ffu;
  return e - 123u <= 1800u;
}

// The same update over runs: consecutive listed voxels with one coefficient
// row, {first voxel, voxels, row, 0} each, at most kBulkPerLane elements a
// lane.  A warp takes a run; of its lanes as many work as whole voxels fit
// (32 / S * S), so that a lane keeps its density and its division a fixed
// divisor, and every load of the run is in flight at once.  With a thread per
// (voxel, density) the chain index - field - store ran in seven waves of
// blocks (0.5M voxels: x 4 FP64 13.8 -> 9.4 us, x 10 30.1 -> 16.6).
constexpr int kBulkPerLane = 8;
// The run a warp takes, eight warps to a block (at most 2^31 runs).  2^27 of
// them make 2^32 threads, whose numbers do not fit 32 bits.
__host__ __device__ constexpr uint32_t bulk_run(uint32_t block, uint32_t thread) {
  return block * 8u + (thread >> 5);
}
template <typename T>
__global__ void __launch_bounds__(256)
    bulk_runs_kernel(T* __restrict__ p, int S, int lanes, int nruns, const int4* __restrict__ runs,
                     const double* __restrict__ tab, double dt) {
  const uint32_t w = bulk_run(blockIdx.x, threadIdx.x);
  const int lane = threadIdx.x & 31;
  if (w >= (uint32_t)nruns || lane >= lanes) return;
  const int4 run = __ldg(runs + w);
  const int count = run.y * S;
  T* q = p + (int64_t)run.x * S + lane;
  T x[kBulkPerLane];
#pragma unroll
  for (int i = 0; i < kBulkPerLane; ++i)
    if (lane + i * lanes < count) x[i] = q[i * lanes];
  const double* c = tab + ((int64_t)run.z * S + lane % S) * 2;
  const double add = __dmul_rn(dt, __ldg(c));
  Divisor by{__dadd_rn(__dmul_rn(__ldg(c + 1), dt), 1.0), 0.0};
  by.y = __drcp_rn(by.d);
  const bool moderate = fabs(by.d) > 1e-18 && fabs(by.d) < 1e18;
#pragma unroll
  for (int i = 0; i < kBulkPerLane; ++i)
    if (lane + i * lanes < count) {
      const double v = __dadd_rn((double)x[i], add);
      q[i * lanes] = (T)(moderate && div_safe(v) ? div_fast(v, by) : __ddiv_rn(v, by.d));
    }
}

// simulate_cell_sources_and_sinks over the agents sorted by voxel (key[r] =
// voxel of the r-th sorted agent, idx[r] = its position in the agent list;
// the sort is stable).  One thread per (sorted agent, substrate): the thread
// of the first agent of each voxel applies all agents of that voxel in list
// order, the others return.  t1/t2 are [A][S] in list order.  The keys around
// an agent and its list position are fetched together, then its constants
// and the field: two round trips, where the loop over a voxel's agents had
// three (1M agents x 8 on 512^3 FP32 with the bulk runs above: 137 -> 113 us).
// Four agents a thread, a grid apart, were slower (80 -> 107 us): neighbours
// in the sorted list share DRAM rows.
template <typename T>
__global__ void cells_kernel(T* __restrict__ p, int S, uint64_t m_S, int64_t A,
                             const uint64_t* __restrict__ key, const int* __restrict__ idx,
                             const double* __restrict__ t1, const double* __restrict__ t2) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= A * S) return;
  // t / S as quot() has it (t S < 2^64)
  const int64_t r = m_S ? (int64_t)__umul64hi((uint64_t)t, m_S) : t;
  const int s = (int)(t - r * S);
  const uint64_t v = __ldg(key + r);
  const uint64_t before = r > 0 ? __ldg(key + r - 1) : ~v;
  const uint64_t after = r + 1 < A ? __ldg(key + r + 1) : ~v;
  int64_t a = (int64_t)__ldg(idx + r) * S + s;
  if (before == v) return;
  const int64_t q = (int64_t)v * S + s;
  const double b1 = __ldg(t1 + a), b2 = __ldg(t2 + a);
  double x = cell_update((double)p[q], b1, b2);
  if (after == v) {
    for (int64_t e = r + 1; e < A && __ldg(key + e) == v; ++e) {
      a = (int64_t)__ldg(idx + e) * S + s;
      x = cell_update(x, __ldg(t1 + a), __ldg(t2 + a));
    }
  }
  p[q] = (T)x;
}

static __global__ void iota_kernel(int* __restrict__ out, int64_t n) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[t] = (int)t;
}

// a[r][col] = v for r < rows (row pitch `pitch` elements)
static __global__ void fill_column_kernel(double* __restrict__ a, int64_t rows, int pitch, int col,
                                   double v) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < rows) a[t * pitch + col] = v;
}

// apply_dirichlet_conditions over the de-duplicated node list.
template <typename T>
__global__ void dirichlet_kernel(T* __restrict__ p, int S, int64_t E, const int64_t* __restrict__ voxel,
                                 const double* __restrict__ val) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  p[voxel[e] * S + s] = (T)val[t];
}

// out[e][s] = p[voxel[e]][s]
template <typename T>
__global__ void gather_kernel(const T* __restrict__ p, int S, int64_t E, const int64_t* __restrict__ voxel,
                              double* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  out[t] = (double)p[voxel[e] * S + s];
}

// p[voxel[e]][s] = in[e][s]
template <typename T>
__global__ void scatter_kernel(T* __restrict__ p, int S, int64_t E, const int64_t* __restrict__ voxel,
                               const double* __restrict__ in) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= E * S) return;
  const int64_t e = t / S;
  const int s = (int)(t - e * S);
  p[voxel[e] * S + s] = (T)in[t];
}

// Microenvironment::compute_all_gradient_vectors (BioFVM_microenvironment.cpp:
// 702-787): central differences along each axis at the points with a
// neighbour on both sides, g = (p[n + jump] - p[n - jump]) / (2 d); the
// components of points at an axis end are left as they are.  g is
// [N][S][3] FP64.
//
// A warp covers 32 (i, s) elements of kGradRows rows of plane k, a thread the
// same element of each row, every load issued before the first use; a row's
// 32 x 3 results are staged in shared memory and written as one run of 768
// bytes (components at an axis end keep their old value, read back only
// there).  Warps inside the mesh run a body without guards (INNER).  The warps
// of a block share nothing but L1.  FAST: the divisors take div_fast.
//
// 256^3 x 4 FP64: 493 us (4.4 TB/s of the 32 B an element takes).  One row per
// block with the general division was bound by instructions (255 an element
// at 80 % of the issue slots: 617 us); with div_fast alone 622, four rows with
// guards 569, without them 493, 131 instructions an element.  Walking through
// z with the planes in registers moves a third of the L2 reads, but left too
// few loads in flight (591, and 739 with the planes fetched ahead).
constexpr int kGradRows = 4;
struct GradArgs {
  int64_t RS;  // elements of a row
  int ny, nz, S;
  Divisor dx, dy, dz;
  double* g;
};
template <typename T, bool FAST, bool INNER>
__device__ __forceinline__ void gradient_rows_body(const GradArgs& a, const T* __restrict__ p,
                                                   double* buf, int64_t e0, int lane, int k,
                                                   int j0) {
  const int64_t RS = a.RS, jz = RS * a.ny, e = e0 + lane;
  const bool mine = INNER || e < RS;
  const bool has_x = INNER || (mine && e >= a.S && e + a.S < RS);
  const bool has_z = INNER || (mine && k > 0 && k < a.nz - 1);
  const int rows = INNER ? kGradRows : min(kGradRows, a.ny - j0);
  const T* q = p + ((int64_t)k * a.ny + j0) * RS + e;
  double* out = a.g + 3 * (q - p - lane);  // the warp's run of the first row
  T row[kGradRows + 2], lo[kGradRows], hi[kGradRows], dn[kGradRows], up[kGradRows];
  {
    const T* c = q - RS;
#pragma unroll
    for (int r = 0; r < kGradRows + 2; ++r, c += RS)
      row[r] = INNER || (mine && j0 + r > 0 && j0 + r <= a.ny) ? __ldg(c) : T(0);
    const T *xl = q - a.S, *xh = q + a.S, *zl = q - jz, *zh = q + jz;
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      const bool in = r < rows;
      lo[r] = INNER || (has_x && in) ? __ldg(xl) : T(0);
      hi[r] = INNER || (has_x && in) ? __ldg(xh) : T(1);
      dn[r] = INNER || (has_z && in) ? __ldg(zl) : T(0);
      up[r] = INNER || (has_z && in) ? __ldg(zh) : T(1);
      xl += RS, xh += RS, zl += RS, zh += RS;
    }
  }
#pragma unroll
  for (int r = 0; r < kGradRows; ++r, out += 3 * RS) {
    if (!INNER && r >= rows) break;
    const bool has_y = INNER || (mine && j0 + r > 0 && j0 + r < a.ny - 1);
    // a missing difference is replaced by the old component below
    double x = __dsub_rn((double)hi[r], (double)lo[r]);
    double y = has_y ? __dsub_rn((double)row[r + 2], (double)row[r]) : 1.0;
    double z = __dsub_rn((double)up[r], (double)dn[r]);
    if (FAST && div_safe(x) && div_safe(y) && div_safe(z)) {
      x = div_fast(x, a.dx), y = div_fast(y, a.dy), z = div_fast(z, a.dz);
    } else {
      x = __ddiv_rn(x, a.dx.d), y = __ddiv_rn(y, a.dy.d), z = __ddiv_rn(z, a.dz.d);
    }
    if (!INNER && mine && !(has_x && has_y && has_z)) {
      const double* old = out + 3 * lane;
      if (!has_x) x = old[0];
      if (!has_y) y = old[1];
      if (!has_z) z = old[2];
    }
    buf[3 * lane] = x;
    buf[3 * lane + 1] = y;
    buf[3 * lane + 2] = z;
    __syncwarp();
    if ((INNER || e0 + 32 <= RS) && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
      const double2* s2 = reinterpret_cast<const double2*>(buf);
      double2* o2 = reinterpret_cast<double2*>(out);
      o2[lane] = s2[lane];
      if (lane < 16) o2[32 + lane] = s2[32 + lane];
    } else {
      const int count = 3 * (int)min((int64_t)32, RS - e0);
      for (int c = lane; c < count; c += 32) out[c] = buf[c];
    }
    __syncwarp();
  }
}

// The same differences a row at a time, for meshes with too few rows to keep
// the device busy four at a time: block (bx, j, k) covers 256 consecutive (i, s)
// elements of row (j, k), whose results are staged in shared memory.
template <typename T>
__global__ void __launch_bounds__(256)
    gradient_row_kernel(const T* __restrict__ p, const GradArgs a) {
  __shared__ double buf[3 * 256];
  const int64_t RS = a.RS, e0 = (int64_t)blockIdx.x * 256, e = e0 + threadIdx.x;
  const int count = (int)min((int64_t)256, RS - e0), j = blockIdx.y, k = blockIdx.z;
  const int64_t row0 = ((int64_t)k * a.ny + j) * RS, jz = RS * a.ny;
  double* out = a.g + 3 * (row0 + e0);
  if (threadIdx.x < count) {
    const T* q = p + row0 + e;
    const double* old = out + 3 * threadIdx.x;
    double* b = buf + 3 * threadIdx.x;
    b[0] = e >= a.S && e + a.S < RS
               ? __ddiv_rn(__dsub_rn((double)q[a.S], (double)q[-a.S]), a.dx.d)
               : old[0];
    b[1] = j > 0 && j < a.ny - 1 ? __ddiv_rn(__dsub_rn((double)q[RS], (double)q[-RS]), a.dy.d)
                                 : old[1];
    b[2] = k > 0 && k < a.nz - 1 ? __ddiv_rn(__dsub_rn((double)q[jz], (double)q[-jz]), a.dz.d)
                                 : old[2];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < 3 * count; c += 256) out[c] = buf[c];
}

template <typename T, bool FAST>
__global__ void __launch_bounds__(256, 4) gradient_rows_kernel(const T* __restrict__ p,
                                                               const GradArgs a) {
  __shared__ __align__(16) double staged[8][96];
  const int lane = threadIdx.x & 31;
  double* buf = staged[threadIdx.x >> 5];
  const int64_t e0 = (int64_t)blockIdx.x * 256 + (threadIdx.x & ~31);
  if (e0 >= a.RS) return;
  const bool inner_x = e0 >= a.S && e0 + 32 + a.S <= a.RS;
  for (int k = blockIdx.z; k < a.nz; k += gridDim.z)
    for (int j0 = blockIdx.y * kGradRows; j0 < a.ny; j0 += gridDim.y * kGradRows) {
      if (inner_x && k > 0 && k < a.nz - 1 && j0 > 0 && j0 + kGradRows < a.ny)
        gradient_rows_body<T, FAST, true>(a, p, buf, e0, lane, k, j0);
      else
        gradient_rows_body<T, FAST, false>(a, p, buf, e0, lane, k, j0);
    }
}

// Lines longer than the chunked kernels take (more than 1024 points): one
// thread per (line, density) column runs the reference's Thomas sequence
// (BioFVM_solvers.cpp:186-200: p_0 /= d_0; p_k = (p_k + c1 p_{k-1}) / d_k;
// then p_k -= cx_k p_{k+1}), each operation rounded on its own, so the
// result equals the reference's for an FP64 field.  Consecutive columns are
// consecutive addresses for the y and z axes (the S densities of consecutive
// rows for x).  The forward values are stored and read back by the backward
// pass: two reads and two writes per element.  den, cx: [n][S]; c1: [S].
template <typename T>
__global__ void long_line_kernel(T* __restrict__ p, T* __restrict__ out, int64_t col0,
                                 int64_t ncols, int64_t C, int64_t outer_stride,
                                 int64_t line_stride, int n, int S,
                                 const double* __restrict__ den, const double* __restrict__ cx,
                                 const double* __restrict__ c1v) {
  const int64_t vcol = col0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (vcol >= ncols) return;
  const int64_t outer = vcol / C;
  const int64_t col = vcol - outer * C;
  const int s = (int)(col % S);
  const int64_t off = outer * outer_stride + col;
  const T* q = p + off;
  T* o = out + off;
  const double c1 = __ldg(c1v + s);
  double prev = __ddiv_rn((double)q[0], __ldg(den + s));
  o[0] = (T)prev;
  for (int k = 1; k < n; ++k) {
    prev = __ddiv_rn(__dadd_rn((double)q[k * line_stride], __dmul_rn(c1, prev)),
                     __ldg(den + (int64_t)k * S + s));
    o[k * line_stride] = (T)prev;
  }
  double next = prev;
  for (int k = n - 2; k >= 0; --k) {
    next = __dsub_rn((double)o[k * line_stride], __dmul_rn(__ldg(cx + (int64_t)k * S + s), next));
    o[k * line_stride] = (T)next;
  }
}

// Joins the z slabs of a field split by planes over several solvers, after
// each slab's z sweep ran with zero carries at its ends (x').  One thread
// per (i, j, density) column of this slab.  planes [R][2][C]: every slab's
// first and last local plane after its sweep (C = nx*ny*S values each);
// cst [R][S][3] {P, Gs, R} per slab; pt [nz][S][2] {G, Rk} of this slab's
// planes.  The forward value entering slab r folds the slabs before it
// (Q = P Q + last), the solution on the first plane after this slab folds
// the slabs after it from the far end (X = first + C Gs + R X); then
// x_k = x'_k + C G_k + X Rk_k on every plane of this slab.
template <int MAXR>
__global__ void zslab_fixup_kernel(double* __restrict__ p, int64_t C, int S, int nz, int R,
                                   int rank, const double* __restrict__ planes,
                                   const double* __restrict__ cst,
                                   const double* __restrict__ pt) {
  const int64_t col = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= C) return;
  const int s = (int)(col % S);
  double carry_in[MAXR];
  double Q = 0.0;
#pragma unroll
  for (int r = 0; r < MAXR; ++r) {
    if (r < R) {
      carry_in[r] = Q;
      Q = __ldg(cst + ((int64_t)r * S + s) * 3) * Q + __ldg(planes + ((int64_t)r * 2 + 1) * C + col);
    }
  }
  double X = 0.0;
#pragma unroll
  for (int r = MAXR - 1; r >= 0; --r) {
    if (r < R && r > rank) {
      const double* k = cst + ((int64_t)r * S + s) * 3;
      X = __ldg(planes + (int64_t)r * 2 * C + col) + carry_in[r] * __ldg(k + 1) + __ldg(k + 2) * X;
    }
  }
  double Cr = 0.0;
#pragma unroll
  for (int r = 0; r < MAXR; ++r)
    if (r == rank) Cr = carry_in[r];
  for (int k = 0; k < nz; ++k) {
    const double* g = pt + ((int64_t)k * S + s) * 2;
    double* q = p + (int64_t)k * C + col;
    *q = *q + Cr * __ldg(g) + X * __ldg(g + 1);
  }
}

template <typename Dst, typename Src>
__global__ void convert_kernel(Dst* __restrict__ dst, const Src* __restrict__ src, int64_t count) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < count) dst[t] = (Dst)src[t];
}

}  // namespace bfvm
