// Host side of the closed-form sweeps (bfvm_kernels_closed.cuh): their
// constants, and the launches bfvm_solver.cu's sweep() makes under
// BFVM_PATH_AUTO.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "bfvm.h"
#include "bfvm_kernels_closed.cuh"
#include "bfvm_state.h"

namespace bfvm_rt {

namespace {

int axis_points(const bfvm_solver* m, int a) { return a == 0 ? m->nx : (a == 1 ? m->ny : m->nz); }

// Whether a short line takes chunks of 8 points: a thread's passes are unrolled
// over its chunk, and along x, where a chunk's loads touch a few bytes of each
// sector, fewer of them help by themselves.  Sweeps of 12M elements in us, with
// 16-point chunks -> with 8: lines of 3, FP64 x of one density 42 -> 22, FP32 y of
// four 80 -> 51; of 12, x of one FP64 79 -> 62, FP32 60 -> 32, y FP64 38.9 -> 38.6,
// FP32 24.5 -> 29.6 (16 kept); of 9, y FP64 34.8 -> 37.4 (16 kept), x of ten FP32
// 31.4 -> 39.3 (16 kept from three on); of 16, y FP64 26.6 -> 28.6 (16 kept); of
// 20, x of one FP64 88 -> 76, FP32 62 -> 44; of 30, x FP64 of one 81 -> 76, of two
// 43 -> 46 (16 kept).
bool closed_short(const bfvm_solver* m, int a) {
  const int n = axis_points(m, a);
  if (n <= 8) return true;
  if (n == 16 || (m->math_elem() == 4 && (a != 0 || m->S > 2))) return false;
  return n <= 24 ? a == 0 || n >= 12 : a == 0 && n < 32 && m->S == 1;
}

// Points per thread: 8 for short lines (above); 32 where the line is whole
// 32-point chunks or has at least six of them; else 16.  A 32-point chunk
// spreads the per-thread work (indices, carries) over twice the points (y at
// 256^3 x 10 FP64 415 -> 396 us, at 256^3 x 4 FP32 132 -> 98), but a line's last,
// partial chunk runs the body with bounds checks, a quarter of the threads of a
// 123-point line (z at 161 x 97 x 123 x 3: 20.2 us at 16 points, 22.9 at 32).
// Fields of few columns take 16 as well, to have 128 threads on every SM
// (twelve domains of 32 to 128 points a side, 20 steps: 4.19 -> 4.07 ms).  The
// columns are counted over the whole mesh, also where LOD_2D sweeps one plane
// of a mesh with several: the constants are laid out for one chunk length,
// which may not change between a 3-D and a 2-D step.
int closed_chunk(const bfvm_solver* m, int a) {
  const int n = axis_points(m, a);
  if (closed_short(m, a)) return 8;
  if (n > 512) return 32;
  if (m->NS() / n * ((n + 31) / 32) < 128 * (int64_t)m->num_sms) return 16;
  return n % 32 == 0 || n > 160 ? 32 : 16;
}

}  // namespace

// Whether the closed-form kernels sweep this axis: the default choice
// (BFVM_PATH_AUTO, no configuration set on the axis), coefficients that have
// the closed form (closed_coefficients), lines the chunked kernels take, whole
// lines (a z slab's carries come from the other slabs).
bool closed_axis(const bfvm_solver* m, int ax) {
  if (m->path != BFVM_PATH_AUTO || m->axis[ax].user || !m->closed_ok) return false;
  if (ax == 2 && m->zs_ranks > 0) return false;
  if (ax == 0 && m->fuse_sources) return false;
  const int n = axis_points(m, ax);
  return n <= 1024 && m->NS() / n < ((int64_t)1 << 31);
}

int closed_axis_chunk(const bfvm_solver* m, int ax) { return closed_chunk(m, ax); }

namespace {

// c1 = dt D / dx^2 and c2 = dt decay / 3 (/ 2 for LOD_2D) of density s as the
// Thomas setup has them (BioFVM_solvers.cpp:105-126; dx on every axis), and
// the slope r = c1 / d, d the larger root of d^2 - (1 + 2 c1 + c2) d + c1^2,
// rounded to the arithmetic type.
struct Slope {
  long double c1, c2, r;
};
Slope closed_slope(const bfvm_solver* m, int s) {
  Slope k;
  k.c1 = (long double)m->h_c1[0][s];
  k.c2 = (long double)m->setup_decay[s] * m->setup_dt / (m->setup_dims == 2 ? 2 : 3);
  const long double b = 1 + 2 * k.c1 + k.c2;
  const long double d = (b + std::sqrt((1 + k.c2) * (1 + k.c2 + 4 * k.c1))) / 2;
  const long double r = k.c1 / d;
  k.r = m->math_elem() == 4 ? (long double)(float)r : (long double)(double)r;
  return k;
}

// Whether every density of the setup has the closed form: c1 >= 0 and
// 1 + c2 > 0, which give a real slope in [0, 1), and a slope that is still
// below 1 when rounded (FP32: c1 up to about 1e15).  Others (a negative
// diffusion coefficient, a negative decay rate of 3 / dt or more) are solved
// by elimination, which has a result wherever its divisors are not zero.
// Written so that a NaN answers false.
bool closed_coefficients(const bfvm_solver* m) {
  for (int s = 0; s < m->S; ++s) {
    const Slope k = closed_slope(m, s);
    if (!(k.c1 >= 0 && 1 + k.c2 > 0 && k.r >= 0 && k.r < 1)) return false;
  }
  return true;
}

}  // namespace

// Constants of the axes for ch[a]-point chunks (ClosedCoef: cst, then pw; none
// where ch[a] is 0), one after another from off[a], from the slopes of the
// Thomas setup, in extended precision and rounded once: to t, in FP32 to the
// pairs tf (from 2 off[a]).  The powers of a chunk's r^ch are multiplied up: at
// most 31 products and the power's own rounding, 2^-58 of the value together,
// where a power per entry cost the first step 0.36 ms at 1000 points x 16.
void closed_constants(const bfvm_solver* m, const int (&ch)[3], std::vector<double>& t,
                      std::vector<float>& tf, size_t (&off)[3]) {
  const int S = m->S;
  const bool fp32 = m->math_elem() == 4;
  size_t count = 0;
  for (int a = 0; a < 3; ++a) {
    off[a] = count;
    if (ch[a] > 0) count += (size_t)S * 8 + (size_t)((axis_points(m, a) + ch[a] - 1) / ch[a]) * S * 2;
  }
  t.assign(count, 0.0);
  tf.assign(fp32 ? 2 * count : 0, 0.0f);
  auto put = [&](size_t i, long double x) {
    t[i] = (double)x;
    if (fp32) {
      tf[2 * i] = (float)x;
      tf[2 * i + 1] = (float)(x - tf[2 * i]);
    }
  };
  std::vector<long double> before;  // r^(c ch)
  for (int s = 0; s < S; ++s) {
    const Slope slope = closed_slope(m, s);
    const long double r = slope.r;
    for (int a = 0; a < 3; ++a) {
      if (ch[a] == 0) continue;
      const int n = axis_points(m, a), nc = (n + ch[a] - 1) / ch[a];
      const long double rc = std::pow(r, (long double)ch[a]);
      const long double rl = std::pow(r, (long double)(n - (nc - 1) * ch[a]));
      const long double rn = std::pow(r, (long double)n);
      const long double k[7] = {r, (1 - r) * (1 - r) / (1 + slope.c2), 1 / ((1 - r) * (1 + r)),
                                rc, rl, rn, 1 / (1 - rn * rn)};
      for (int i = 0; i < 7; ++i) put(off[a] + (size_t)s * 8 + i, k[i]);
      before.assign(1, 1.0L);
      for (int c = 1; c < nc; ++c) before.push_back(before.back() * rc);
      for (int c = 0; c < nc; ++c) {
        const size_t i = off[a] + (size_t)S * 8 + ((size_t)c * S + s) * 2;
        put(i, before[c]);
        put(i + 1, c == nc - 1 ? 1.0L : rl * before[nc - 2 - c]);
      }
    }
  }
}

void closed_setup(bfvm_solver* m) {
  std::vector<double> t;
  std::vector<float> tf;
  m->closed_ok = closed_coefficients(m);
  if (!m->closed_ok) return;
  int ch[3];
  for (int a = 0; a < 3; ++a) ch[a] = axis_points(m, a) > 1024 ? 0 : closed_chunk(m, a);
  closed_constants(m, ch, t, tf, m->closed_off);
  if (m->math_elem() == 4)
    upload(m->closed_tab, tf, m->stream);
  else
    upload(m->closed_tab, t, m->stream);
}

namespace {

template <typename CT>
bfvm::ClosedCoef<CT> closed_view(const bfvm_solver* m, int a) {
  constexpr size_t k = sizeof(CT) == 4 ? 2 : 1;  // numbers to an entry
  const CT* t = m->closed_tab.as<CT>() + k * m->closed_off[a];
  return {t, t + k * (size_t)m->S * 8};
}

// Calls f with each of the flags as a compile-time constant.
template <typename F, typename... B>
void with_flags(F&& f, bool b, B... rest) {
  auto one = [&](auto c) {
    if constexpr (sizeof...(rest) == 0)
      f(c);
    else
      with_flags([&](auto... cs) { f(c, cs...); }, rest...);
  };
  if (b)
    one(std::true_type());
  else
    one(std::false_type());
}

template <typename T, typename CT, int CH, int MAXT>
void lines(bfvm_solver* m, const bfvm::ClosedArgs<T, CT>& a, bool ca, dim3 grid, dim3 block,
           size_t smem) {
  with_flags(
      [&](auto dir, auto l1, auto exact) {
        bfvm::closed_lines_kernel<T, CT, CH, MAXT, decltype(dir)::value, decltype(l1)::value,
                                  decltype(exact)::value><<<grid, block, smem, m->stream>>>(a);
      },
      a.fuse != 0, ca, a.n % CH == 0);
  check_launch(m);
}

template <typename T, typename CT>
void sweep_lines(bfvm_solver* m, int ax, int fuse, int64_t z0, int64_t z1) {
  const int64_t nx = m->nx, ny = m->ny, nz = m->nz, S = m->S;
  const int64_t nzp = m->lod_dims == 2 ? 1 : nz;  // planes swept
  bfvm::ClosedArgs<T, CT> a{};
  a.p = m->p.as<T>();
  a.out = m->sweep_out ? static_cast<T*>(m->sweep_out) : a.p;
  int64_t per_plane = 0;
  if (ax == 0) {
    a.n = (int)nx, a.C = (uint32_t)S, a.os = nx * S, a.ls = S, per_plane = ny * S;
  } else if (ax == 1) {
    a.n = (int)ny, a.C = (uint32_t)(nx * S), a.os = nx * ny * S, a.ls = nx * S;
    per_plane = nx * S;
  } else {
    a.n = (int)nz, a.C = (uint32_t)(nx * ny * S), a.os = 0, a.ls = nx * ny * S;
  }
  a.ncols = (uint32_t)(ax == 2 ? nx * ny * S : per_plane * nzp);
  if (z1 >= 0 && ax < 2) {  // columns of planes z0 .. z1-1
    a.col0 = (uint32_t)(z0 * per_plane);
    a.ncols = (uint32_t)(z1 * per_plane);
  }
  a.mC = quot_of(a.C);
  a.mS = quot_of(S);
  a.S = (int)S;
  const int ch = closed_chunk(m, ax), nc = (a.n + ch - 1) / ch;
  a.cc = closed_view<CT>(m, ax);
  const DevSegList& dseg = ax == 0 ? m->seg_dir_x : m->seg_dir_y;
  if (ax == 2 || !dseg.present) fuse = 0;
  a.fuse = fuse & (bfvm::kFuseDirPro | bfvm::kFuseDirEpi);
  a.dir = dseg.view();
  // short lines: blocks of 64 threads, FP32 fields 128 (lines of 8 points, FP64
  // y of one density 24.6 -> 20.3 us, FP32 24.4 -> 15.3; of 30, FP64 32.8 -> 34.5
  // with 128, FP32 22.5 -> 21)
  int W = nc <= 16 ? 32 : 16;
  while (W * nc <= (sizeof(T) == 8 ? 32 : 64) &&
         blocks_for(a.ncols - a.col0, 2 * W) >= 8 * m->num_sms)
    W *= 2;
  const dim3 block(W, nc), grid((unsigned)blocks_for(a.ncols - a.col0, W));
  const size_t smem = (size_t)2 * nc * W * sizeof(CT);
  const bool ca = ax == 0 && S * (int)sizeof(T) < 256;
  if (ch == 8)
    lines<T, CT, 8, 512>(m, a, ca, grid, block, smem);
  else if (ch == 16)
    lines<T, CT, 16, 512>(m, a, ca, grid, block, smem);
  else if (W * nc <= 256)
    lines<T, CT, 32, 256>(m, a, ca, grid, block, smem);
  else
    lines<T, CT, 32, 512>(m, a, ca, grid, block, smem);
}

constexpr size_t kTileSmem = 224 * 1024;  // of the 227 KB a block may use

struct TilePlan {
  bool ok = false;
  int ch = 0, nc = 0, w = 0, maxt = 0, stages = 0;
  int box_n = 0, nboxes = 0;     // lines
  int R = 0, pitch = 0;          // rows
  int stage_elems = 0;
  size_t smem = 0;
  uint32_t tile0 = 0, ntiles = 0;
};

// The ring of an axis's tiles: 32 columns by n points each, 16 from 257 points
// on, which keeps two blocks of 256 threads per SM up to 512 points; FP32
// fields' y and z from 513 points on, where 32 columns of 32-point chunks are
// more than a block's threads (mixed, 12M elements in lines of 700: 42 -> 31 us
// with tiles, FP32 28 -> 26.6).
template <typename T, typename CT>
TilePlan plan_tiles(const bfvm_solver* m, int ax, int64_t z0, int64_t z1) {
  TilePlan P;
  const int64_t nx = m->nx, ny = m->ny, nz = m->nz, S = m->S, es = sizeof(T);
  const int64_t nzp = m->lod_dims == 2 ? 1 : nz;
  const int n = axis_points(m, ax);
  P.ch = closed_chunk(m, ax);
  P.nc = (n + P.ch - 1) / P.ch;
  if (P.ch == 8) return P;  // the line kernel's
  const int W = P.w =
      P.ch == 32 && ((P.nc > 8 && (es == 8 || ax == 0)) || P.nc > 16) ? 16 : 32;
  P.maxt = P.ch == 16 || W * P.nc > 256 ? 512 : 256;
  if (W * P.nc > P.maxt) return P;
  if (ax == 0) {
    if (S > W) return P;
    P.R = (int)(W / S);
    const int64_t row = nx * S, rb = row * es;
    const int mod = es == 8 ? 16 : 32;
    int64_t pitch = row + ((S - row) % mod + mod) % mod;
    if (rb % 16) {  // one copy of R rows
      const int64_t g = rb % 8 ? 4 : 2;  // rows between 16-byte boundaries
      P.R = (int)(P.R / g * g);
      pitch = row;
      if (P.R == 0 || (z1 >= 0 && (z0 * ny * rb) % 16)) return P;
    } else {
      while ((pitch * es) % 16) ++pitch;
    }
    if (P.R * S * 3 < W * 2) return P;  // too many lanes would repeat others' work
    P.pitch = (int)pitch;
    const int64_t rows = (z1 >= 0 ? (z1 - z0) : nzp) * ny;
    P.ntiles = (uint32_t)((rows + P.R - 1) / P.R);
    P.stage_elems = (int)((P.R * pitch + P.ch * S + 127) / 128 * 128);
  } else {
    const int64_t ls = ax == 1 ? nx * S : nx * ny * S, os = nx * ny * S * (ax == 1 ? 1 : nz);
    const int64_t C = ls, outer = ax == 1 ? nzp : 1;
    if ((ls * es) % 16 || (os * es) % 16 || C >= ((int64_t)1 << 31)) return P;
    P.nboxes = (n + 255) / 256;
    P.box_n = (n + P.nboxes - 1) / P.nboxes;
    P.box_n += (P.box_n * W * es) % 128 ? 1 : 0;  // each box starts on a 128-byte boundary
    const int64_t ct = (C + W - 1) / W;
    P.ntiles = (uint32_t)(ct * outer);
    if (z1 >= 0 && ax == 1) {
      P.tile0 = (uint32_t)(ct * z0);
      P.ntiles = (uint32_t)(ct * z1);
    }
    P.stage_elems = P.box_n * P.nboxes * W;
  }
  const size_t fold = 4 * (size_t)P.nc * W * sizeof(CT);  // two parities of U and W
  const size_t stage = (size_t)P.stage_elems * es;
  if (stage + fold + 1024 > kTileSmem) return P;
  const int blocks =
      std::max(1, bfvm::closed_min_blocks<CT>(P.ch, P.maxt) * P.maxt / (W * P.nc));
  const size_t budget = std::max(kTileSmem / blocks - 1024, stage + fold);  // 1 KB: system, pad
  P.stages = (int)std::min<size_t>(3, (budget - fold) / stage);
  P.smem = P.stages * stage + fold + 128;
  P.ok = true;
  return P;
}

template <typename T, typename CT, int CH, int W, bool DIR, bool ROWS, int MAXT, bool EXACT>
void tile_kernel(bfvm_solver* m, const CUtensorMap& map, const bfvm::ClosedTileArgs<T, CT>& a,
                 dim3 block, size_t smem) {
  auto k = bfvm::closed_tile_kernel<T, CT, CH, W, DIR, ROWS, MAXT, EXACT>;
  allow_smem((const void*)k, m->device, smem);
  int per_sm = 0;
  BFVM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, block.x * block.y, smem));
  require(per_sm > 0, "sweep kernel does not fit on an SM", BFVM_ERR_STATE);
  // One block per place on the device, except for rows where a place gets many
  // tiles: there several blocks, of a dozen tiles each, follow one another, so
  // that no SM is left with the slow ones at the end.  x alone on the device, time
  // with one block a place over time with several, at 28, 37, 48, 60 and 72 tiles
  // a place: FP64 256 points x 10 1.03, 1.03, 1.04, 1.05, 1.07, 192 x 4 1.01, 1.02,
  // 1.04, 1.06, 1.06; FP32 512 x 8 1.00, 0.99, 0.99, 0.98, 1.00, then at 110, 160,
  // 240 and 400 1.00, 1.00, 1.01, 1.02; FP32 in FP64 arithmetic 256 x 4 0.98 from
  // 28 to 110, 1.00, 1.00, 1.01 after.  y and z do not gain.
  const uint32_t tiles = a.ntiles - a.tile0, places = (uint32_t)per_sm * m->num_sms;
  const uint32_t each = tiles / places, many = sizeof(T) == 8 ? 36 : 160;
  const dim3 grid(std::min(tiles, places * (ROWS && each >= many ? std::min(8u, each / 12) : 1)));
  k<<<grid, block, smem, m->stream>>>(map, a);
  check_launch(m);
}

template <typename T, typename CT>
void sweep_tiles(bfvm_solver* m, int ax, int fuse, int64_t z0, int64_t z1, const TilePlan& P) {
  const int64_t nx = m->nx, ny = m->ny, nz = m->nz, S = m->S;
  bfvm::ClosedTileArgs<T, CT> a{};
  a.p = m->p.as<T>();
  a.out = m->sweep_out ? static_cast<T*>(m->sweep_out) : m->p.as<T>();
  a.tile0 = P.tile0;
  a.ntiles = P.ntiles;
  a.n = axis_points(m, ax);
  a.S = (int)S;
  a.mS = quot_of(S);
  a.stages = P.stages;
  a.stage_elems = P.stage_elems;
  a.cc = closed_view<CT>(m, ax);
  const DevSegList& dseg = ax == 0 ? m->seg_dir_x : m->seg_dir_y;
  if (ax == 2 || !dseg.present) fuse = 0;
  a.fuse = fuse & (bfvm::kFuseDirPro | bfvm::kFuseDirEpi);
  a.dir = dseg.view();
  a.status = m->d_status.as<int>();
  if (ax == 0) {
    a.row0 = z1 >= 0 ? z0 * ny : 0;
    a.rows = z1 >= 0 ? z1 * ny : ny * (m->lod_dims == 2 ? 1 : nz);
    a.R = P.R;
    a.row_elems = (int)(nx * S);
    a.pitch = P.pitch;
  } else {
    a.ls = ax == 1 ? nx * S : nx * ny * S;
    a.os = nx * ny * S * (ax == 1 ? 1 : nz);
    a.C = (uint32_t)a.ls;
    a.ctiles = (a.C + P.w - 1) / P.w;
    a.mT = quot_of(a.ctiles);
    a.box_n = P.box_n;
    a.nboxes = P.nboxes;
    encode_lines_map(m, ax, sizeof(T), a.C, a.n, ax == 1 ? (m->lod_dims == 2 ? 1 : nz) : 1, a.ls,
                     a.os, P.w, P.box_n);
  }
  const dim3 block(P.w, P.nc);
  auto go = [&](auto ch, auto w, auto maxt) {
    constexpr int CH = decltype(ch)::value, W = decltype(w)::value, MAXT = decltype(maxt)::value;
    with_flags(
        [&](auto dir, auto rows, auto exact) {
          tile_kernel<T, CT, CH, W, decltype(dir)::value, decltype(rows)::value, MAXT,
                      decltype(exact)::value>(m, m->maps[ax], a, block, P.smem);
        },
        a.fuse != 0, ax == 0, a.n % CH == 0);
  };
  using std::integral_constant;
  if (P.ch == 16)
    go(integral_constant<int, 16>(), integral_constant<int, 32>(), integral_constant<int, 512>());
  else if (P.w == 32 && P.maxt == 256)
    go(integral_constant<int, 32>(), integral_constant<int, 32>(), integral_constant<int, 256>());
  else if (P.w == 32)
    go(integral_constant<int, 32>(), integral_constant<int, 32>(), integral_constant<int, 512>());
  else if (P.maxt == 256)
    go(integral_constant<int, 32>(), integral_constant<int, 16>(), integral_constant<int, 256>());
  else
    go(integral_constant<int, 32>(), integral_constant<int, 16>(), integral_constant<int, 512>());
}

// Whether the tile kernel sweeps the axis rather than the line kernel (us, line
// -> tile):
//   x: 26.4 -> 22.9 at 128^3 x 4, 95.7 -> 79.3 at 192^3 x 4, 25.9 -> 22.4 at
//     128^3 x 1, 460 either way at 256^3 x 10 (FP64), 1716 -> 1386 at 512^3 x
//     8 FP32: rows arrive whole, where the line kernel's loads touch a few
//     bytes of each sector.  At 16-point chunks only for one or two densities
//     (30.2 -> 34.2 at 101^3 x 7).
//   y and z: columns are contiguous and the line kernel, with more blocks per
//     SM to hide its loads, is ahead (y 395 -> 458 at 256^3 x 10, FP32 1401 ->
//     1837 at 512^3 x 8), except with an FP32 field in FP64 arithmetic (113 ->
//     95 at 256^3 x 4: the conversions lengthen the solve), from 257 points
//     on in FP64 (206 -> 189 at 400^3 x 1: one block per SM either way), and
//     where 32-point chunks leave a partial one (FP32 70 -> 52 at 200^3 x 4).
template <typename T, typename CT>
bool tiles_better(const bfvm_solver* m, int ax, int ch) {
  if (ax == 0) return ch == 32 || m->S <= 2;
  if (ch == 16) return false;
  const int n = axis_points(m, ax);
  return sizeof(T) != sizeof(CT) || n % 32 != 0 || (sizeof(CT) == 8 && n > 256);
}

}  // namespace

// One sweep of axis ax (planes [z0, z1) of the x and y axes, z1 < 0: all),
// with the Dirichlet overwrites of `fuse` before and after it.
void closed_sweep(bfvm_solver* m, int ax, int fuse, int64_t z0, int64_t z1) {
  auto go = [&](auto t, auto ct) {
    using T = decltype(t);
    using CT = decltype(ct);
    const TilePlan P = plan_tiles<T, CT>(m, ax, z0, z1);
    if (P.ok && tiles_better<T, CT>(m, ax, P.ch))
      sweep_tiles<T, CT>(m, ax, fuse, z0, z1, P);
    else
      sweep_lines<T, CT>(m, ax, fuse, z0, z1);
  };
  if (m->precision == BFVM_FP64)
    go(double(), double());
  else if (m->precision == BFVM_FP32_FP64MATH)
    go(float(), double());
  else
    go(float(), float());
}

}  // namespace bfvm_rt
