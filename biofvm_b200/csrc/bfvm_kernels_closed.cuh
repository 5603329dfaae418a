// Closed-form LOD sweeps: the Thomas solve of one line with constant slopes.
//
// Along one axis every line solves (BioFVM_solvers.cpp:105-142, 186-200)
//   (1 + c2) x_k + c1 (2 x_k - x_{k-1} - x_{k+1}) = p_k,
// the end rows with one neighbour, which is the interior row with the ghost
// values x_{-1} = x_0 and x_n = x_{n-1}.  With r the root below 1 of
// c1 (r + 1/r) = 1 + 2 c1 + c2 the operator is (c1/r) (1 - r E^-1) (1 - r E)
// (E the shift along the line), so the line is solved by two recurrences
// whose slope r and scale s = r/c1 are the same at every point:
//   q_k = r q_{k-1} + p_k,   x_k = r x_{k+1} + s q_k.
// The ends only set the first carries: continuing p past both ends by
// reflection gives, with TU = sum r^(n-1-k) p_k and TW = sum r^k p_k,
//   q_{-1} = (TW + r^n TU) / (1 - r^(2n)),
//   w_n    = (TU + r^n TW) / (1 - r^(2n))   (w_k = r w_{k+1} + p_k),
//   x_k    = (r q_{k-1} + w_k) / (1 - r^2) s,  used where a chunk ends.
// Nothing is tabulated per point: a thread keeps r and a few products of it
// in registers, where the elimination tables cost five shared-memory loads
// per point (and their address arithmetic), which, not HBM, bounded the
// tabulated kernels: 35 thread instructions a point, 14 here.  Sweeps x, y, z
// in us, tabulated -> closed form: 511, 480, 549 -> 459, 395, 443 at 256^3 x
// 10 FP64 (y at 6.8 TB/s, an in-place copy's rate); 33, 38, 37 -> 23, 20, 20
// at 128^3 x 4; 49, 41, 33 -> 31, 23, 20 at 161 x 97 x 123 x 3; 2290, 1487,
// 1745 -> 1386, 1401, 1469 at 512^3 x 8 FP32.
//
// A line is cut into chunks of CH points, one per thread, held in registers:
//   1. U = sum r^(len-1-m) v_m and W = sum r^m v_m of the chunk (two
//      independent chains);
//   2. each thread passes over its column's chunks through shared memory,
//      forward and backward, for the carries that enter its chunk;
//   3. forward with the true carry, then backward with the true carry.
// Five multiply-adds per point, one load and one store of it.  T is the
// field's element type, CT the type the recurrences run in (the precision
// modes' arithmetic).
//
// Rounding: s is set on the host to (1 - r)^2 / (1 + c2) for the rounded r,
// so that a constant field keeps its sum exactly in the mean; an error of r
// in the last place then acts as a relative change of D by about 2 eps/(1-r).
// In FP32 every other constant, s among them, is a pair of floats (high and
// low part): a single float s would scale the field by the same slightly
// wrong factor in every sweep.
#pragma once

#include "bfvm_kernels.cuh"
#include "bfvm_tma.cuh"

namespace bfvm {

// A constant as a sum of two CTs (FP64: the low part is zero and not read).
template <typename CT>
struct Const2 {
  CT hi, lo;
};
__device__ __forceinline__ double cmul(const Const2<double>& k, double x) { return k.hi * x; }
__device__ __forceinline__ float cmul(const Const2<float>& k, float x) {
  return fma(k.hi, x, k.lo * x);
}
__device__ __forceinline__ double cfma(const Const2<double>& k, double x, double y) {
  return fma(k.hi, x, y);
}
__device__ __forceinline__ float cfma(const Const2<float>& k, float x, float y) {
  return fma(k.hi, x, fma(k.lo, x, y));
}

// Constants of one axis, two to a 16-byte load: cst [S][4][2] holds {r, s},
// {1/(1-r^2), r^CH}, {r^(length of the last chunk), r^n}, {1/(1-r^(2n)), 0};
// pw [chunks][S][2] {r^(points before the chunk), r^(points after it)}.  In
// FP32 each of them is its {high, low} pair.
enum : int { kCrS, kChRc, kCrlRn, kCinv };
template <typename CT>
struct ClosedCoef {
  const CT* cst;
  const CT* pw;
};
template <typename CT>
struct Const2x2 {
  Const2<CT> a, b;
};
__device__ __forceinline__ Const2x2<double> ld_const(const double* base, size_t i) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(base) + i);
  return {{v.x, 0.0}, {v.y, 0.0}};
}
__device__ __forceinline__ Const2x2<float> ld_const(const float* base, size_t i) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(base) + i);
  return {{v.x, v.y}, {v.z, v.w}};
}
template <typename CT>
__device__ __forceinline__ Const2x2<CT> closed_const(const ClosedCoef<CT>& cc, int s, int which) {
  return ld_const(cc.cst, (size_t)s * 4 + which);
}

template <typename T, typename CT>
struct ClosedArgs {
  T* p;
  T* out;          // where the solved lines go (p: in place)
  uint32_t col0;   // first column of this launch (a slab of planes)
  uint32_t ncols;  // end of the launch's (line, density) columns
  uint32_t C;      // columns per outer block
  uint64_t mC, mS; // quot() of C and S
  int64_t os;      // element stride between outer blocks
  int64_t ls;      // element stride between points of a line
  int n;
  int S;
  ClosedCoef<CT> cc;
  SegList dir;     // (line, chunk) segments of the axis's Dirichlet nodes
  int fuse;        // kFuseDirPro | kFuseDirEpi
};

// The same stride, unknown to the compiler: the stores of a chunk then form
// their own addresses instead of keeping those of its loads (a register pair
// per point) live across the solve.
__device__ __forceinline__ int64_t fresh(int64_t stride) {
  asm volatile("" : "+l"(stride));
  return stride;
}
__device__ __forceinline__ int fresh(int stride) {
  asm volatile("" : "+r"(stride));
  return stride;
}

// U and W of a chunk of len points (FULL: len == CH).
template <typename CT, int CH, bool FULL>
__device__ __forceinline__ void closed_sums(const CT (&v)[CH], int len, CT r, CT& U, CT& W) {
  // the points past len are zero: W need not leave them out
  CT u = CT(0), w = CT(0);
  const int lu = fresh(len);
#pragma unroll
  for (int m = 0; m < CH; ++m) {
    if (FULL || m < lu) u = fma(r, u, v[m]);
    w = fma(r, w, v[CH - 1 - m]);
  }
  U = u;
  W = w;
}

// The solve of a chunk from its true carries: qin = q before it, vin = w
// after it.
template <typename CT, int CH, bool FULL>
__device__ __forceinline__ void closed_solve(CT (&v)[CH], int len, CT r, const Const2<CT>& scale,
                                             const Const2<CT>& h, CT qin, CT vin) {
  CT q = qin;
  const int lq = fresh(len), lx = fresh(len);
#pragma unroll
  for (int m = 0; m < CH; ++m) {
    if (FULL || m < lq) {
      q = fma(r, q, v[m]);
      v[m] = q;
    }
  }
  CT x = cmul(h, fma(r, q, vin));
#pragma unroll
  for (int m = CH - 1; m >= 0; --m) {
    if (FULL || m < lx) {
      x = fma(r, x, v[m]);
      v[m] = cmul(scale, x);
    }
  }
}

// A barrier over the whole block that warps may reach from different places
// of the program (the bodies for full and for partial chunks below; a warp
// takes one of them as a whole).
__device__ __forceinline__ void block_barrier() {
  __syncwarp();
  asm volatile("bar.sync 0;" ::: "memory");
}

// Whether every chunk of this thread's warp has CH points: the last chunk
// the warp holds ends within the line.  From indices alone, so that it is the
// same for the whole warp (a vote could be taken by part of a warp after a
// loop its lanes left at different times, and the parts would then meet the
// block's barriers separately).
__device__ __forceinline__ bool warp_full(int tid, int W, int NC, int CH, int n) {
  const int last = min((tid | 31) / W, NC - 1);
  return (last + 1) * CH <= n;
}

// The rest of a chunk's solve, from every chunk's sums in shared memory (sU,
// sW: [NC][W], stored before a block barrier): each thread runs over the
// chunks of its column forward and backward, which gives the carries entering
// its chunk from zero line ends and the whole line's sums TU and TW, adds the
// line ends' share, then makes the two passes.  (One thread per column and
// direction doing this for the others needs a second barrier, at which most
// of the block waits: 31 instructions per point and 40 % of issue slots at
// 256^3 x 4 FP32.)  The constants are read here, not before the sums, to keep
// them out of the registers the chunk needs.
template <typename CT, int CH, bool FULL>
__device__ __forceinline__ void closed_finish(CT (&v)[CH], int len, CT r, const ClosedCoef<CT>& cc,
                                              int S, const CT* sU, const CT* sW, int W, int NC,
                                              int c, int col, int s) {
  const Const2x2<CT> hrc = closed_const(cc, s, kChRc), rlrn = closed_const(cc, s, kCrlRn);
  const Const2<CT>& rc = hrc.b;
  const CT *u = sU + col, *w = sW + (NC - 1) * W + col;
  CT TU = CT(0), TW = CT(0);
  int i = 0;
#pragma unroll 4
  for (; i < c; ++i, u += W) TU = cfma(rc, TU, *u);
  const CT q0 = TU;  // the sum entering chunk c
#pragma unroll 4
  for (; i < NC - 1; ++i, u += W) TU = cfma(rc, TU, *u);
  TU = cfma(rlrn.a, TU, *u);
  // (the last chunk starts from a zero carry, so that its length is no matter)
  i = NC - 1;
#pragma unroll 4
  for (; i > c; --i, w -= W) TW = cfma(rc, TW, *w);
  const CT w0 = TW;
#pragma unroll 4
  for (; i >= 0; --i, w -= W) TW = cfma(rc, TW, *w);
  const Const2x2<CT> pw = ld_const(cc.pw, (size_t)c * S + s);
  const Const2<CT> inv = closed_const(cc, s, kCinv).a;
  const CT qin = cfma(pw.a, cmul(inv, cfma(rlrn.b, TU, TW)), q0);
  const CT vin = cfma(pw.b, cmul(inv, cfma(rlrn.b, TW, TU)), w0);
  closed_solve<CT, CH, FULL>(v, len, r, closed_const(cc, s, kCrS).b, hrc.a, qin, vin);
}

// Blocks per SM the kernels are compiled for, from the registers a chunk of
// CH points takes: FP64 64 of 65,536 / (512 x 2) up to 16 points and 128 at 32;
// FP32 80 (three blocks of 256 threads) or 64 (two of 512) at 32 points.
template <typename CT>
constexpr int closed_min_blocks(int ch, int maxt) {
  return sizeof(CT) == 4 ? (maxt <= 256 ? 3 : 2) : (ch <= 16 ? 1024 : 512) / maxt;
}

// Quotients by a number d fixed per launch: v / d = __umul64hi(v, m) with m =
// floor(2^64 / d) + 1, exact for 32-bit v (v times the excess of m over 2^64/d
// stays below 2^64); m = 0 stands for d = 1.
__device__ __forceinline__ uint32_t quot(uint32_t v, uint64_t m) {
  return m ? (uint32_t)__umul64hi((uint64_t)v, m) : v;
}

template <typename T, typename CT, int CH, bool DIR, bool FULL, bool CA>
__device__ __forceinline__ void closed_lines_body(const ClosedArgs<T, CT>& a, CT* smem, int len,
                                                  uint32_t line, bool mine, int64_t off, int s) {
  const int W = blockDim.x, NC = blockDim.y;
  CT* sU = smem;
  CT* sW = sU + NC * W;
  const int tx = threadIdx.x, c = threadIdx.y;
  CT v[CH];
  {
    const T* q = a.p + off;
#pragma unroll
    for (int m = 0; m < CH; ++m, q += a.ls)
      v[m] = FULL || m < len ? (CT)(CA ? *q : __ldcg(q)) : CT(0);
  }
  const CT r = closed_const(a.cc, s, kCrS).a.hi;
  const int64_t seg = (int64_t)line * NC + c;
  if (DIR && (a.fuse & kFuseDirPro))
    apply_dirichlet_seg<CT, CH>(v, a.dir, seg, c * CH, a.S, s);
  CT U, Wd;
  closed_sums<CT, CH, FULL>(v, len, r, U, Wd);
  sU[c * W + tx] = U;
  sW[c * W + tx] = Wd;
  block_barrier();
  closed_finish<CT, CH, FULL>(v, len, r, a.cc, a.S, sU, sW, W, NC, c, tx, s);
  if (DIR && (a.fuse & kFuseDirEpi))
    apply_dirichlet_seg<CT, CH>(v, a.dir, seg, c * CH, a.S, s);
  if (!mine) return;
  T* o = a.out + off;
  const int64_t ls = fresh(a.ls);
  const int lo = fresh(len);
#pragma unroll
  for (int m = 0; m < CH; ++m, o += ls)
    if (FULL || m < lo) *o = (T)v[m];
}

// Blocks of W consecutive columns x NC chunks, the columns read and written
// straight between registers and memory, W elements at a time.  Warps whose
// chunks all have CH points run a body without bounds checks.  Columns past
// the end repeat the last one's loads and store nothing.  CA: loads through
// L1 (x lines, where a chunk's neighbouring points share sectors).
template <typename T, typename CT, int CH, int MAXT, bool DIR, bool CA, bool EXACT>
__global__ void __launch_bounds__(MAXT, closed_min_blocks<CT>(CH, MAXT))
    closed_lines_kernel(const ClosedArgs<T, CT> a) {
  extern __shared__ __align__(128) unsigned char closed_smem[];
  CT* sums = reinterpret_cast<CT*>(closed_smem);
  const int W = blockDim.x;
  const uint32_t first = a.col0 + blockIdx.x * (uint32_t)W;
  const bool mine = first + threadIdx.x < a.ncols;
  const uint32_t vcol = mine ? first + threadIdx.x : a.ncols - 1;
  const int k0 = threadIdx.y * CH;
  const int len = min(CH, a.n - k0);
  const uint32_t outer = quot(vcol, a.mC), line = quot(vcol, a.mS);
  const uint32_t col = vcol - outer * a.C;
  const int s = (int)(vcol - line * (uint32_t)a.S);
  const int64_t off = (int64_t)outer * a.os + col + (int64_t)k0 * a.ls;
  if (EXACT || warp_full(threadIdx.y * W + threadIdx.x, W, blockDim.y, CH, a.n))
    closed_lines_body<T, CT, CH, DIR, true, CA>(a, sums, CH, line, mine, off, s);
  else
    closed_lines_body<T, CT, CH, DIR, false, CA>(a, sums, len, line, mine, off, s);
}

// ---------------------------------------------------------------------------
// Tiles by TMA, persistent blocks.  A block keeps a ring of tiles in shared
// memory: as soon as its threads hold a tile in registers, the next one is
// fetched into the freed stage, so that a block loads while it solves and
// stores.
//   LINES: y and z; a tile is W consecutive columns x n points, one tensor
//     box of [n][W] (two from 257 points).
//   ROWS: x; a tile is R whole rows by bulk copies, R*S of the block's W
//     columns, at a row pitch of S modulo 16 elements (FP32: 32) so that the
//     lanes of a chunk, which read consecutive columns of one point, meet
//     distinct banks.  Rows that are not 16-byte multiples come as one
//     contiguous copy of R rows (R even, for FP32 a multiple of 4, as their
//     start needs).  Lanes past the tile's rows repeat other lanes' columns.

template <typename T, typename CT>
struct ClosedTileArgs {
  const T* p;
  T* out;
  uint32_t tile0, ntiles;  // tiles tile0 .. ntiles-1
  int n, S, stages;
  int stage_elems;         // a multiple of 128 bytes
  ClosedCoef<CT> cc;
  SegList dir;             // (line, chunk) segments
  int fuse;
  int* status;
  uint64_t mS;             // quot() of S
  // LINES
  uint32_t C, ctiles;      // columns per outer block, tiles of them
  uint64_t mT;             // quot() of ctiles
  int64_t os, ls;
  int box_n, nboxes;
  // ROWS
  int64_t row0, rows;      // rows row0 .. rows-1, tile 0 at row0
  int R, row_elems, pitch;
};

// One tile from shared memory to the output; `read` is called by every thread
// once the block holds the tile in registers, and ends the block's work when
// it returns false; `place` gives where the thread's chunk goes (null:
// nowhere) and the stride of its points, worked out anew after the solve.
template <typename T, typename CT, int CH, int W, bool DIR, bool FULL, bool ROWS, typename F,
          typename G>
__device__ __forceinline__ bool closed_tile_body(const ClosedTileArgs<T, CT>& a, const T* q,
                                                 CT* fold, int len, int64_t line, int s,
                                                 F&& read, G&& place) {
  const int NC = blockDim.y;
  CT* sU = fold;
  CT* sW = sU + NC * W;
  const int tx = threadIdx.x, c = threadIdx.y;
  const int step = ROWS ? a.S : W;
  CT v[CH];
#pragma unroll
  for (int m = 0; m < CH; ++m, q += step) v[m] = FULL || m < len ? (CT)*q : CT(0);
  const CT r = closed_const(a.cc, s, kCrS).a.hi;
  if (DIR && (a.fuse & kFuseDirPro))
    apply_dirichlet_seg<CT, CH>(v, a.dir, line * NC + c, c * CH, a.S, s);
  CT U, Wd;
  closed_sums<CT, CH, FULL>(v, len, r, U, Wd);
  sU[c * W + tx] = U;
  sW[c * W + tx] = Wd;
  block_barrier();
  if (!read()) return false;
  closed_finish<CT, CH, FULL>(v, len, r, a.cc, a.S, sU, sW, W, NC, c, tx, s);
  if (DIR && (a.fuse & kFuseDirEpi))
    apply_dirichlet_seg<CT, CH>(v, a.dir, line * NC + c, c * CH, a.S, s);
  int64_t ls;
  T* o = place(ls);
  if (o == nullptr) return true;
  const int lo = fresh(len);
#pragma unroll
  for (int m = 0; m < CH; ++m, o += ls)
    if (FULL || m < lo) *o = (T)v[m];
  return true;
}

template <typename T, typename CT, int CH, int W, bool DIR, bool ROWS, int MAXT, bool EXACT>
__global__ void __launch_bounds__(MAXT, closed_min_blocks<CT>(CH, MAXT))
    closed_tile_kernel(const __grid_constant__ CUtensorMap map, const ClosedTileArgs<T, CT> a) {
  extern __shared__ __align__(128) unsigned char closed_smem[];
  __shared__ __align__(8) uint64_t full[4];
  __shared__ int bad;
  const int NC = blockDim.y;
  const int tid = threadIdx.y * W + threadIdx.x;
  // tensor copies need 128-byte aligned destinations
  T* tiles = reinterpret_cast<T*>(
      closed_smem + ((128u - ((uint32_t)__cvta_generic_to_shared(closed_smem) & 127u)) & 127u));
  CT* folds = reinterpret_cast<CT*>(tiles + (size_t)a.stages * a.stage_elems);
  if (tid == 0) {
    if (!ROWS) tma::prefetch_map(&map);
    for (int i = 0; i < a.stages; ++i) tma::mbar_init(&full[i], 1);
    tma::fence_barrier_init();
    bad = 0;
  }
  __syncthreads();

  auto issue = [&](int st, uint32_t tile) {
    T* dst = tiles + (size_t)st * a.stage_elems;
    if (ROWS) {
      const int64_t first = a.row0 + (int64_t)tile * a.R;
      const int nr = (int)min((int64_t)a.R, a.rows - first);
      const T* src = a.p + first * a.row_elems;
      const uint32_t rb = (uint32_t)(a.row_elems * sizeof(T));
      if (a.pitch == a.row_elems) {  // one run (its end rounded up inside the allocation)
        const uint32_t bytes = (rb * nr + 15u) & ~15u;
        tma::mbar_arrive_expect_tx(&full[st], bytes);
        tma::load_bulk(dst, src, bytes, &full[st]);
      } else {
        tma::mbar_arrive_expect_tx(&full[st], rb * nr);
        for (int i = 0; i < nr; ++i)
          tma::load_bulk(dst + i * a.pitch, src + (int64_t)i * a.row_elems, rb, &full[st]);
      }
    } else {
      const uint32_t outer = quot(tile, a.mT);
      const int col0 = (int)((tile - outer * a.ctiles) * W);
      tma::mbar_arrive_expect_tx(&full[st],
                                 (uint32_t)(a.box_n * a.nboxes * W * (int)sizeof(T)));
      for (int b = 0; b < a.nboxes; ++b)
        tma::load_tile_3d(dst + b * a.box_n * W, &map, &full[st], col0, b * a.box_n, (int)outer);
    }
  };
  int issued = 0;  // tiles issued (thread 0)
  if (tid == 0) {
    for (int i = 0; i < a.stages; ++i) {
      const uint32_t t = a.tile0 + blockIdx.x + (uint32_t)i * gridDim.x;
      if (t < a.ntiles) {
        issue(i, t);
        ++issued;
      }
    }
  }

  const int S = a.S;
  const int c = threadIdx.y, tx = threadIdx.x;
  const int len = min(CH, a.n - c * CH);
  const bool whole = EXACT || warp_full(tid, W, NC, CH, a.n);
  int st = 0, i = 0;
  uint32_t parity = 0;
  for (uint32_t tile = a.tile0 + blockIdx.x; tile < a.ntiles; tile += gridDim.x, ++i) {
    if (!tma::mbar_wait(&full[st], parity)) bad = 1;
    const T* q = tiles + (size_t)st * a.stage_elems;
    int s;
    int64_t line;
    if (ROWS) {
      const int64_t first = a.row0 + (int64_t)tile * a.R;
      const int nr = (int)min((int64_t)a.R, a.rows - first);
      const int r0 = (int)quot(tx, a.mS);
      s = tx - r0 * S;
      const int r = r0 < a.R ? min(r0, nr - 1) : 0;
      line = first + r;
      q += r * a.pitch + c * CH * S + s;
    } else {
      const uint32_t outer = quot(tile, a.mT);
      const uint32_t col0 = (tile - outer * a.ctiles) * W;
      // columns past the end hold the box's fill value
      const uint32_t vcol = outer * a.C + min(col0 + tx, a.C - 1);
      const uint32_t l = quot(vcol, a.mS);
      s = (int)(vcol - l * (uint32_t)S);
      line = l;
      q += c * CH * W + tx;
    }
    auto place = [&](int64_t& ls) -> T* {
      const uint32_t t = (uint32_t)fresh((int)tile);
      const int k0 = fresh(c * CH);
      if (ROWS) {
        const int64_t first = a.row0 + (int64_t)t * a.R;
        const int r = (int)quot(tx, a.mS);
        ls = S;
        if (r >= min((int64_t)a.R, a.rows - first)) return nullptr;
        return a.out + (first + r) * a.row_elems + (int64_t)k0 * S + (tx - r * S);
      }
      const uint32_t outer = quot(t, a.mT);
      const uint32_t col = (t - outer * a.ctiles) * W + tx;
      ls = a.ls;
      if (col >= a.C) return nullptr;
      return a.out + (int64_t)outer * a.os + col + (int64_t)k0 * a.ls;
    };
    CT* fold = folds + (i & 1) * 2 * NC * W;
    auto read = [&]() -> bool {
      if (*(volatile int*)&bad) {
        if (tid == 0) {
          // copies still in flight are waited for (bounded) before the block ends
          int ws = st, wp = (int)parity;
          for (int j = i; j < issued; ++j) {
            tma::mbar_wait(&full[ws], (uint32_t)wp);
            if (++ws == a.stages) ws = 0, wp ^= 1;
          }
          atomicExch(a.status, 1);
        }
        return false;
      }
      if (tid == 0) {
        const uint32_t nt = tile + (uint32_t)a.stages * gridDim.x;
        if (nt < a.ntiles) {
          issue(st, nt);
          ++issued;
        }
      }
      return true;
    };
    const bool go =
        whole ? closed_tile_body<T, CT, CH, W, DIR, true, ROWS>(a, q, fold, CH, line, s, read, place)
              : closed_tile_body<T, CT, CH, W, DIR, false, ROWS>(a, q, fold, len, line, s, read, place);
    if (!go) return;
    if (++st == a.stages) st = 0, parity ^= 1;
  }
}

}  // namespace bfvm
