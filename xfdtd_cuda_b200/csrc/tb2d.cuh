// Temporally blocked 2-D TMz step: S time steps per launch, the tile in
// registers.
//
// The 2-D grids of the benchmarks sit in L2 (1044^2 cells: 13 MB of FP32
// fields), so a launch per step is bound by launch and memory latency.  Here a
// CTA loads a tile with a halo of S cells, advances it S steps and writes back
// its interior; every step the region whose values are exact shrinks by one
// cell per side (H needs Ez one cell up, E needs H one cell down).
// Neighbouring tiles recompute each other's halo, so no CTA waits for another.
//
// Layout.  A warp owns R rows (i) of the tile's 32 C columns (j): a lane holds
// an R x C block of Ez, Hx and Hy in registers, C consecutive columns of a
// row, so a global access is C elements per lane and a row of the tile is one
// coalesced run.  Neighbours along j are the lane's own registers or one
// shuffle per row, neighbours along i its own registers; only the first Ez row
// and the last Hy row of a warp pass through shared memory (16 bytes per lane
// each), with one CTA barrier per half-step.  The former tile in shared memory
// (fields, material ids and 18-entry coefficients read per cell) issued about
// 230 instructions per cell update, this one about 13 in warps without walls,
// TFSF lines or CPML cells.  Measured (us per step, before and after, as the plan
// runs them): 1044^2 cylinder FP32 14.0 and 6.5, FP64 21.7 and 12.3; 1519 x 751
// FP64 23.1 and 13.2; 2020 x 1720 FP32 (after) 11.6.  What bounds it: the tiles
// along the CPML, whose warps all run the special rows below, take three times the
// others' time, and at 1044^2 the tiles make barely two waves; in FP64 also the
// register spills of those rows (424 bytes of loads per thread at the 128 registers
// of 16 warps; FP32 12).
//
// A warp whose cells share one material keeps its coefficients in registers,
// the others look them up per cell; what else its cells need (PEC walls, TFSF
// lines, CPML slabs) is a flag per warp or lane tested once per row.  The CPML
// psi of the slab rows and columns sit in shared memory, and so do the TFSF
// increments, which the CTA tabulates for all S steps when it starts.  Halo
// cells outside the exact region carry finite garbage that never reaches the
// interior.
//
// Field and psi buffers alternate between launches: a launch reads set p and
// writes set 1-p (the E-side psi too, which the one-launch-per-step kernel
// keeps in place), so S is odd and the set holding step t is t & 1, as for
// the per-step kernels.  The per-cell arithmetic, the TFSF and CPML
// corrections and their order are those of k_step2 (and so of k_h2/k_e2 and
// the CPU restatement), FP64 results are bit-identical; the FP32 rounding is
// spelled out (mad), so it does not depend on the form of the kernel.
#pragma once

#include "fused3d.cuh"

namespace xfb {

constexpr int kTbC = 4;             // columns of a lane's block
constexpr int kTbCols = 32 * kTbC;  // columns of a tile's region
template <typename T>
constexpr int kTbRows = sizeof(T) == 4 ? 4 : 3;  // rows of a lane's block
// warps of a CTA, at most: a thread's block takes 48 (FP32) or 72 (FP64)
// registers, and at 128 per thread the update does not spill in FP32 (20 warps
// at 96 registers measured 8.3 us per step on the 1044^2 cylinder, 24 at 80 12,
// 16 at 128 6.8; 5, 6 and 8 rows in 16 or 12 warps spill: 9 to 11)
template <typename T>
constexpr int kTbMaxWarps = 16;

// Cost model of a launch (us): its fixed part, load and store of a tile, one
// step of one warp (of the slowest tiles, those along the CPML).
constexpr double kTbFixed = 2.0, kTbLoad = 5.0;
template <typename T>
constexpr double kTbWarpStep = sizeof(T) == 4 ? 0.2 : 0.36;

// Region of a launch of S steps by a CTA of nw warps: rows, interior rows and
// columns, and the columns of the left halo (rounded up to a whole lane block,
// so a lane's columns are one aligned vector).
template <typename T>
struct TbGeom {
  int xi, ti, tj, hl;
  __host__ __device__ TbGeom(int nw, int S) {
    xi = nw * kTbRows<T>;
    hl = (S + kTbC - 1) / kTbC * kTbC;
    ti = xi - 2 * S - 1;
    tj = (kTbCols - hl - S - 1) / kTbC * kTbC;
  }
};

// Shared memory of a CTA: the exchange rows [nw][kTbCols] of Ez and Hy, the
// coefficients per material {c9, c11, c12, c13} and {c6, c7, c8, 0}, the psi of
// the region's x-slab rows [2][nsx][kTbCols] (Hy, Ez) and of the lane blocks
// that hold y-slab columns [2][nsy][kTbC][xi] (Hx, Ez; zero in their other
// columns, whose profiles are zero), the y profiles (ah, bh, ae, be) of the region's
// columns and the x profiles of its slab rows, and the incident fields of S steps on the TFSF lines
// the region holds: per column, E at is and ie and H at is-1 and ie; per row,
// E at js and je and H at js-1, je.
template <typename T>
struct TbLayout {
  size_t ex, hy, lut, px, py, yp, xp, inc, bytes;
  __host__ __device__ TbLayout(int nw, int S, int n_mat, int nsx, int nsy) {
    const int xi = nw * kTbRows<T>;
    ex = 0;
    hy = ex + static_cast<size_t>(nw) * kTbCols * sizeof(T);
    lut = hy + static_cast<size_t>(nw) * kTbCols * sizeof(T);
    px = lut + static_cast<size_t>(n_mat) * 8 * sizeof(T);
    py = px + 2ull * nsx * kTbCols * sizeof(T);
    yp = (py + 2ull * nsy * kTbC * xi * sizeof(T) + 15) / 16 * 16;
    xp = yp + (nsy ? 4ull * kTbCols * sizeof(T) : 0);
    inc = (xp + 4ull * nsx * sizeof(T) + 15) / 16 * 16;
    bytes = inc + static_cast<size_t>(S) * 4 * (kTbCols + xi) * sizeof(double);
  }
};

// Slab rows of the region [b, b + n) along an axis of N cells with slabs of lo
// and hi cells: slot of coordinate q (rows of both slabs numbered in order), or -1.
struct TbSlab {
  int l0, l1, h0, h1;  // region rows of the low and of the high slab: [l0, l1), [h0, h1)
  __host__ __device__ TbSlab(int b, int n, int N, int lo, int hi) {
    l0 = b > 0 ? b : 0;
    l1 = lo < b + n ? lo : b + n;
    if (l1 < l0) l1 = l0;
    h0 = N - hi > l1 ? N - hi : l1;
    if (h0 < b) h0 = b;
    h1 = N < b + n ? N : b + n;
    if (h1 < h0) h1 = h0;
  }
  __host__ __device__ int count() const { return l1 - l0 + h1 - h0; }
  __device__ int slot(int q) const { return q >= l0 && q < l1 ? q - l0 : q >= h0 && q < h1 ? l1 - l0 + q - h0 : -1; }
};

// Lane blocks of the region that hold y-slab columns, numbered in order.
struct TbBlocks {
  int a0, a1, b0, b1;
  __host__ __device__ TbBlocks(const TbSlab& y, int jb) {
    a0 = (y.l0 - jb) / kTbC;
    a1 = y.l1 > y.l0 ? (y.l1 - jb + kTbC - 1) / kTbC : a0;
    b0 = (y.h0 - jb) / kTbC;
    if (b0 < a1) b0 = a1;
    b1 = y.h1 > y.h0 ? (y.h1 - jb + kTbC - 1) / kTbC : b0;
    if (b1 < b0) b1 = b0;
  }
  __host__ __device__ int count() const { return a1 - a0 + b1 - b0; }
  __device__ int rank(int lane) const {
    return lane >= a0 && lane < a1 ? lane - a0 : lane >= b0 && lane < b1 ? a1 - a0 + lane - b0 : -1;
  }
  __device__ int lane(int rank) const { return rank < a1 - a0 ? a0 + rank : b0 + rank - (a1 - a0); }
};

// C elements of one row (16-byte accesses).
template <typename T>
__device__ __forceinline__ void tb_ld(T (&o)[kTbC], const T* p) {
  constexpr int W = 16 / sizeof(T);
#pragma unroll
  for (int q = 0; q < kTbC / W; ++q) {
    Vec16<T> v;
    v.ld(p + q * W);
#pragma unroll
    for (int e = 0; e < W; ++e) o[q * W + e] = v.a[e];
  }
}
template <typename T>
__device__ __forceinline__ void tb_st(T* p, const T (&o)[kTbC]) {
  constexpr int W = 16 / sizeof(T);
#pragma unroll
  for (int q = 0; q < kTbC / W; ++q) {
    Vec16<T> v;
#pragma unroll
    for (int e = 0; e < W; ++e) v.a[e] = o[q * W + e];
    v.st(p + q * W);
  }
}

// R values of consecutive rows of a column table.
template <typename T, int R>
__device__ __forceinline__ void tb_ldr(T (&o)[R], const T* p) {
  if constexpr (R == kTbC) {
    tb_ld(o, p);
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) o[r] = p[r];
  }
}
template <typename T, int R>
__device__ __forceinline__ void tb_str(T* p, const T (&o)[R]) {
  if constexpr (R == kTbC) {
    tb_st(p, o);
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) p[r] = o[r];
  }
}

// Barrier of the whole CTA that warps may reach at different places of the code.
__device__ __forceinline__ void tb_sync(int threads) { asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory"); }

// add_inc on column c (of the lane's C) of a row.
template <typename T>
__device__ __forceinline__ void tb_add_col(T (&f)[kTbC], int c, double inc, double coef) {
  T v = f[0];
#pragma unroll
  for (int q = 1; q < kTbC; ++q)
    if (q == c) v = f[q];
  add_inc(v, inc, coef);
#pragma unroll
  for (int q = 0; q < kTbC; ++q)
    if (q == c) f[q] = v;
}

template <typename T>
__global__ void __launch_bounds__(32 * kTbMaxWarps<T>, 1)
    k_step2_tb(GridP<T> s, GridP<T> d, PmlP<T> pm, PsiH<T> ps, PsiH<T> pd, const T* ezx_r, const T* ezy_r, T* ezx_w,
               T* ezy_w, TfsfP tf_in, TimeP tp, ProbeP pr, int2* link, int S, int n_mat, int nsx, int nsy) {
  constexpr int R = kTbRows<T>, C = kTbC;
  extern __shared__ __align__(16) unsigned char tb_smem[];
  const int nw = blockDim.x >> 5, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const TbGeom<T> geo(nw, S);
  const TbLayout<T> lay(nw, S, n_mat, nsx, nsy);
  T* xe = reinterpret_cast<T*>(tb_smem + lay.ex);
  T* xh = reinterpret_cast<T*>(tb_smem + lay.hy);
  T* lut = reinterpret_cast<T*>(tb_smem + lay.lut);
  T* PX = reinterpret_cast<T*>(tb_smem + lay.px);
  T* PY = reinterpret_cast<T*>(tb_smem + lay.py);
  T* YP = reinterpret_cast<T*>(tb_smem + lay.yp);  // [4][kTbCols]
  T* XP = reinterpret_cast<T*>(tb_smem + lay.xp);  // [nsx][4]
  double* incc = reinterpret_cast<double*>(tb_smem + lay.inc);  // [S][4][kTbCols]: E(is), E(ie), H(is-1), H(ie)
  double* incr = incc + static_cast<size_t>(S) * 4 * kTbCols;   // [S][4][xi]: E(js), E(je), H(js-1), H(je)

  const int I0 = blockIdx.y * geo.ti, J0 = blockIdx.x * geo.tj;
  const int ib = I0 - S, jb = J0 - geo.hl;  // global index of row / column 0 of the region
  const int nx = s.nx, ny = s.ny;
  const long long sx = s.sx;
  const int i0 = ib + warp * R, j0 = jb + lane * C;  // first row and column of this lane's block
  const long long t0 = cur_step(tp);

  // ---- load: every row of the block in one vector per field ------------------
  const bool jin = j0 >= 0 && j0 < sx;  // the vector lies inside the padded row
  T E[R][C], HX[R][C], HY[R][C];
  unsigned mid[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = i0 + r;
    mid[r] = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) E[r][c] = HX[r][c] = HY[r][c] = T(0);
    if (jin && i >= 0 && i <= nx) {
      const long long g = i * sx + j0;
      tb_ld(E[r], s.ez + g);
      tb_ld(HX[r], s.hx + g);
      tb_ld(HY[r], s.hy + g);
      mid[r] = *reinterpret_cast<const unsigned*>(s.mid + g);
    }
  }
  for (int q = tid; q < n_mat * 8; q += blockDim.x) {
    const int m = q >> 3, e = q & 7;
    const int src[8] = {9, 11, 12, 13, 6, 7, 8, 8};
    lut[q] = s.lut[18 * m + src[e]];
  }
  const TbSlab sx_(ib, geo.xi, nx, pm.L[0], pm.L[1]), sy_(jb, kTbCols, ny, pm.L[2], pm.L[3]);
  for (int q = tid; q < sx_.count() * kTbCols; q += blockDim.x) {  // psi of the x-slab rows
    const int w = q / kTbCols, c = q - w * kTbCols, j = jb + c;
    const int i = w < sx_.l1 - sx_.l0 ? sx_.l0 + w : sx_.h0 + w - (sx_.l1 - sx_.l0);
    const bool in = j >= 0 && j < ny;
    const long long p = in ? slab(i, nx, pm.L[0], pm.L[1]) * sx + j : 0;
    PX[w * kTbCols + c] = in ? ps.hy_x[p] : T(0);
    PX[(nsx + w) * kTbCols + c] = in ? ezx_r[p] : T(0);
  }
  for (int w = tid; w < sx_.count(); w += blockDim.x) {
    const int i = w < sx_.l1 - sx_.l0 ? sx_.l0 + w : sx_.h0 + w - (sx_.l1 - sx_.l0);
    XP[4 * w] = pm.ah[0][i]; XP[4 * w + 1] = pm.bh[0][i];
    XP[4 * w + 2] = pm.ae[0][i]; XP[4 * w + 3] = pm.be[0][i];
  }
  const TbBlocks yb(sy_, jb);
  const int nyb = yb.count();
  for (int q = tid; q < nyb * C * geo.xi; q += blockDim.x) {  // psi of the y-slab lane blocks
    const int w = q / geo.xi, r = q - w * geo.xi, i = ib + r, j = jb + yb.lane(w / C) * C + w % C;
    const bool in = i >= 0 && i < nx && sy_.slot(j) >= 0;
    const long long p = in ? i * pm.ysx + slab(j, ny, pm.L[2], pm.L[3]) : 0;
    PY[q] = in ? ps.hx_y[p] : T(0);
    PY[nsy * C * geo.xi + q] = in ? ezy_r[p] : T(0);
  }
  if (nyb > 0)
    for (int q = tid; q < kTbCols; q += blockDim.x) {
      const int j = jb + q;
      const bool in = sy_.slot(j) >= 0, ine = in && j >= 1;  // (Ez on the wall j = 0 is not updated)
      YP[q] = in ? pm.ah[1][j] : T(0);
      YP[kTbCols + q] = in ? pm.bh[1][j] : T(0);
      YP[2 * kTbCols + q] = ine ? pm.ae[1][j] : T(0);
      YP[3 * kTbCols + q] = ine ? pm.be[1][j] : T(0);
    }

  // ---- TFSF lines inside the region, their incident values of all S steps ----
  const int ie_ = ib + geo.xi, je_ = jb + kTbCols;
  auto in_rows = [&](int i) { return i >= ib && i < ie_; };
  auto in_cols = [&](int j) { return j >= jb && j < je_; };
  const bool tf_cols = tf_in.on && (in_rows(tf_in.is - 1) || in_rows(tf_in.is) || in_rows(tf_in.ie));
  const bool tf_rows = tf_in.on && (in_cols(tf_in.js - 1) || in_cols(tf_in.js) || in_cols(tf_in.je));
  // lines of the low (js, is) and the high face (je, ie) the region holds: bit 0, 1
  const int fcols = tf_cols ? (in_rows(tf_in.is - 1) || in_rows(tf_in.is) ? 1 : 0) | (in_rows(tf_in.ie) ? 2 : 0) : 0;
  const int frows = tf_rows ? (in_cols(tf_in.js - 1) || in_cols(tf_in.js) ? 1 : 0) | (in_cols(tf_in.je) ? 2 : 0) : 0;
  for (int face = 0; face < 2; ++face) {
    if ((fcols >> face) & 1) {
#pragma unroll 2
      for (int q = tid; q < S * 2 * kTbCols; q += blockDim.x) {
        const int st = q / (2 * kTbCols), h = q / kTbCols & 1, c = q % kTbCols, j = jb + c;
        const TfsfP tf = tfsf_at_step(tf_in, t0 + st);
        double v = 0;
        if (j >= tf.js && j <= tf.je)
          v = h ? hy_inc(tf, face ? tf.ie : tf.is - 1, j, 0) : ez_inc(tf, face ? tf.ie : tf.is, j, 0);
        incc[(st * 4 + 2 * h + face) * kTbCols + c] = v;
      }
    }
    if ((frows >> face) & 1) {
#pragma unroll 2
      for (int q = tid; q < S * 2 * geo.xi; q += blockDim.x) {
        const int st = q / (2 * geo.xi), w = q - st * 2 * geo.xi, h = w >= geo.xi ? 1 : 0, r = w - h * geo.xi, i = ib + r;
        const TfsfP tf = tfsf_at_step(tf_in, t0 + st);
        double v = 0;
        if (i >= tf.is && i <= tf.ie)
          v = h ? hx_inc(tf, i, face ? tf.je : tf.js - 1, 0) : ez_inc(tf, i, face ? tf.je : tf.js, 0);
        incr[(st * 4 + 2 * h + face) * geo.xi + r] = v;
      }
    }
  }

  // ---- what this warp's cells need -------------------------------------------
  const TfsfP& tf = tf_in;
  const int m0 = __shfl_sync(0xffffffffu, static_cast<int>(mid[0] & 0xffu), 0);
  bool one = true;  // one material in the warp
#pragma unroll
  for (int r = 0; r < R; ++r) one = one && mid[r] == 0x01010101u * static_cast<unsigned>(m0);
  one = __all_sync(0xffffffffu, one);
  const int il = i0 + R - 1;  // last row of the warp
  // E kept on the PEC walls and outside the grid (H there feeds no cell of the
  // grid, so it needs no such care): bits of the lane's rows and columns to update
  const bool wall = i0 < 1 || il > nx - 1 || jb < 1 || je_ > ny;
  unsigned okr = 0, okc = 0;
#pragma unroll
  for (int q = 0; q < R; ++q) okr |= i0 + q >= 1 && i0 + q < nx ? 1u << q : 0u;
#pragma unroll
  for (int q = 0; q < C; ++q) okc |= j0 + q >= 1 && j0 + q < ny ? 1u << q : 0u;
  const bool pxw = (i0 < sx_.l1 && il >= sx_.l0) || (i0 < sx_.h1 && il >= sx_.h0);  // x-slab rows
  // TFSF rows is-1, is, ie and columns js-1, js, je among the warp's cells
  const bool tfr = tf_cols && tf.js < je_ && tf.je >= jb &&
                   ((i0 <= tf.is && il >= tf.is - 1) || (i0 <= tf.ie && il >= tf.ie));
  const bool tfc = tf_rows && i0 <= tf.ie && il >= tf.is;
  // Probes of the interior (and of the wall nodes past the last tiles): every
  // thread looks through its share of the list once per launch and puts the
  // tile's probes on the chains of the lanes that hold them, {next, node and
  // component} in `link`, heads in shared memory; at every step a lane walks its
  // own chain.  With every lane searching the whole list, 600 probes on 320 x 220
  // cells took 163 us per step (FP32; now 5.2, none 4.4) and 8 took 5.6 (4.6); on
  // 1044^2 cells 600 took 184 (6.9).
  int* heads = reinterpret_cast<int*>(tb_smem + lay.bytes);
  if (pr.n > 0) {
    heads[tid] = -1;
    __syncthreads();
    for (int p = tid; p < pr.n; p += blockDim.x) {
      const int i = static_cast<int>(pr.idx[p] / sx), j = static_cast<int>(pr.idx[p] - i * sx), fld = pr.field[p];
      const bool own_i = i >= I0 && (i < I0 + geo.ti || I0 + geo.ti >= nx);
      const bool own_j = j >= J0 && (j < J0 + geo.tj || J0 + geo.tj >= ny);
      if (fld < 0 || !own_i || !own_j) continue;
      // H on the upper walls, which no step writes (the lanes' goes past the grid)
      if (fld != XFB_EZ && (i >= nx || j >= ny)) {
        const double v = static_cast<double>((fld == XFB_HX ? s.hx : s.hy)[pr.idx[p]]);
        for (int st = 0; st < S; ++st) pr.out[p * pr.total_steps + t0 + st] = v;
        continue;
      }
      const int w = (i - ib) / R, l = (j - jb) / C, o = (i - ib - w * R) * C + j - jb - l * C;
      link[p] = make_int2(atomicExch(heads + 32 * w + l, p), o * 8 + fld);
    }
  }

  const int yr = yb.rank(lane);  // the lane's y-slab block, or -1
  // the lane's TFSF columns: js-1 and je for Hx, js and je for Ez
  int th0 = -1, th1 = -1, te0 = -1;
  if (tfc) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (j0 + c == tf.js - 1) th0 = c;
      if (j0 + c == tf.js) te0 = c;
      if (j0 + c == tf.je) th1 = c;
    }
  }
  tb_st(xe + warp * kTbCols + lane * C, E[0]);
  __syncthreads();
  const T h0 = lut[8 * m0], h1 = lut[8 * m0 + 1], h2 = lut[8 * m0 + 2], h3 = lut[8 * m0 + 3];
  const T e0 = lut[8 * m0 + 4], e1 = lut[8 * m0 + 5], e2 = lut[8 * m0 + 6];
  T nb[C];  // the neighbour row of the other warp

  // warps without special cells: the plain update alone (their barriers are the
  // same CTA barrier as the other warps', so it is named)
  const bool special = wall || pxw || tfr || tfc || !one || nyb > 0 || (pr.n > 0 && __any_sync(0xffffffffu, heads[tid] >= 0));
  if (!special) {
    const int nt = blockDim.x;
    const T* xe_n = xe + min(warp + 1, nw - 1) * kTbCols + lane * C;  // (the last warp's rows past the region are not exact)
    const T* xh_p = xh + max(warp - 1, 0) * kTbCols + lane * C;
    // (two steps per turn, the shuffles ahead of the barrier: in place, FP64 takes
    // 18 register moves a step less; 2520^2 without probes 33.5 -> 32.6 us)
#pragma unroll 2
    for (int st = 0; st < S; ++st) {
      tb_ld(nb, xe_n);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const T er = __shfl_down_sync(0xffffffffu, E[r][0], 1);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const T ez = E[r][c];
          HX[r][c] = mad(h0, HX[r][c], mul(h1, (c + 1 < C ? E[r][(c + 1) % C] : er) - ez));
          HY[r][c] = mad(h2, HY[r][c], mul(h3, (r + 1 < R ? E[(r + 1) % R][c] : nb[c]) - ez));
        }
      }
      tb_st(xh + warp * kTbCols + lane * C, HY[R - 1]);
      T sd[R];
#pragma unroll
      for (int r = 0; r < R; ++r) sd[r] = __shfl_up_sync(0xffffffffu, HX[r][C - 1], 1);
      tb_sync(nt);
      tb_ld(nb, xh_p);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const T hl = sd[r];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const T da = HX[r][c] - (c > 0 ? HX[r][(c + C - 1) % C] : hl);
          const T db = HY[r][c] - (r > 0 ? HY[(r + R - 1) % R][c] : nb[c]);
          E[r][c] = mad(e2, db, mad(e0, E[r][c], mul(e1, da)));
        }
      }
      tb_st(xe + warp * kTbCols + lane * C, E[0]);
      tb_sync(nt);
    }
  } else {
  // E coefficients per column of a one-material warp: 1, 0, 0 keeps E on the
  // walls along y and outside the grid
  T w0[C], w1[C], w2[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const bool ok = (okc >> c) & 1u;
    w0[c] = ok ? e0 : T(1); w1[c] = ok ? e1 : T(0); w2[c] = ok ? e2 : T(0);
  }
  for (int st = 0; st < S; ++st) {
    // ---- H: Ez one column and one row up --------------------------------------
    if (warp + 1 < nw) {
      tb_ld(nb, xe + (warp + 1) * kTbCols + lane * C);
    } else {
#pragma unroll
      for (int c = 0; c < C; ++c) nb[c] = E[R - 1][c];  // past the region: not exact from here on
    }
    T side[R];  // the neighbour column of the next lane
#pragma unroll
    for (int r = 0; r < R; ++r) side[r] = __shfl_down_sync(0xffffffffu, E[r][0], 1);
    // differences of Ez: along y (for Hx), along x (for Hy)
    auto ey = [&](int r, int c) { return (c + 1 < C ? E[r][(c + 1) % C] : side[r]) - E[r][c]; };
    auto ex = [&](int r, int c) { return (r + 1 < R ? E[(r + 1) % R][c] : nb[c]) - E[r][c]; };
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (one) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          HX[r][c] = mad(h0, HX[r][c], mul(h1, ey(r, c)));
          HY[r][c] = mad(h2, HY[r][c], mul(h3, ex(r, c)));
        }
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const C4<T> cf = ld_c4(lut + 8 * ((mid[r] >> (8 * c)) & 0xffu));
          HX[r][c] = mad(cf.c, HX[r][c], mul(cf.x, ey(r, c)));
          HY[r][c] = mad(cf.y, HY[r][c], mul(cf.z, ex(r, c)));
        }
      }
    }
    if (tfr) {  // rows is-1, ie (incc is zero beyond [js, je])
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = i0 + r;
        if (i != tf.is - 1 && i != tf.ie) continue;
        const double* in = incc + (st * 4 + (i == tf.ie ? 1 : 0)) * kTbCols + lane * C;
#pragma unroll
        for (int c = 0; c < C; ++c) add_inc(HY[r][c], in[c], i == tf.ie ? tf.cb[0] : -tf.cb[0]);
      }
    }
    if (th0 >= 0) {  // (incr is zero beyond [is, ie])
      const double* in = incr + st * 4 * geo.xi + warp * R;
#pragma unroll
      for (int r = 0; r < R; ++r) tb_add_col(HX[r], th0, in[r], tf.cb[1]);
    }
    if (th1 >= 0) {
      const double* in = incr + (st * 4 + 1) * geo.xi + warp * R;
#pragma unroll
      for (int r = 0; r < R; ++r) tb_add_col(HX[r], th1, in[r], -tf.cb[1]);
    }
    if (pxw) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = i0 + r, w = sx_.slot(i);
        if (w < 0) continue;
        const T ca = XP[4 * w], cb = XP[4 * w + 1];
        T p[C];
        tb_ld(p, PX + w * kTbCols + lane * C);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          p[c] = psi_next_yz(cb, p[c], ca, ex(r, c));
          HY[r][c] = mad(one ? h3 : lut[8 * ((mid[r] >> (8 * c)) & 0xffu) + 3], p[c], HY[r][c]);
        }
        tb_st(PX + w * kTbCols + lane * C, p);
      }
    }
    if (yr >= 0) {
      T ca[C], cb[C];
      tb_ld(ca, YP + lane * C);
      tb_ld(cb, YP + kTbCols + lane * C);
      T* col = PY + yr * C * geo.xi + warp * R;
#pragma unroll
      for (int c0 = 0; c0 < C; c0 += 2, col += 2 * geo.xi) {  // (both loads first: the stores may alias them)
        T p[2][R];
        tb_ldr(p[0], col);
        tb_ldr(p[1], col + geo.xi);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int c = c0 + d;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            p[d][r] = psi_next_yz(cb[c], p[d][r], ca[c], ey(r, c));
            HX[r][c] = mad(one ? h1 : lut[8 * ((mid[r] >> (8 * c)) & 0xffu) + 1], p[d][r], HX[r][c]);
          }
        }
        tb_str(col, p[0]);
        tb_str(col + geo.xi, p[1]);
      }
    }
    tb_st(xh + warp * kTbCols + lane * C, HY[R - 1]);
    tb_sync(blockDim.x);
    // ---- E: Hx one column and Hy one row down -----------------------------------
    if (warp > 0) {
      tb_ld(nb, xh + (warp - 1) * kTbCols + lane * C);
    } else {
#pragma unroll
      for (int c = 0; c < C; ++c) nb[c] = HY[0][c];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) side[r] = __shfl_up_sync(0xffffffffu, HX[r][C - 1], 1);
    // differences of Hx along y, of Hy along x
    auto hy = [&](int r, int c) { return HX[r][c] - (c > 0 ? HX[r][(c + C - 1) % C] : side[r]); };
    auto hx = [&](int r, int c) { return HY[r][c] - (r > 0 ? HY[(r + R - 1) % R][c] : nb[c]); };
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!((okr >> r) & 1u)) continue;  // PEC wall (or outside): kept
#pragma unroll
      for (int c = 0; c < C; ++c) {
        T a0 = w0[c], a1 = w1[c], a2 = w2[c];
        if (!one && ((okc >> c) & 1u)) {
          const C4<T> cf = ld_c4(lut + 8 * ((mid[r] >> (8 * c)) & 0xffu) + 4);
          a0 = cf.c; a1 = cf.x; a2 = cf.y;
        }
        E[r][c] = mad(a2, hx(r, c), mad(a0, E[r][c], mul(a1, hy(r, c))));
      }
    }
    if (tfr) {  // rows is, ie
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = i0 + r;
        if (i != tf.is && i != tf.ie) continue;
        const double* in = incc + (st * 4 + (i == tf.ie ? 3 : 2)) * kTbCols + lane * C;
#pragma unroll
        for (int c = 0; c < C; ++c) add_inc(E[r][c], in[c], i == tf.ie ? tf.ca[0] : -tf.ca[0]);
      }
    }
    if (te0 >= 0) {
      const double* in = incr + (st * 4 + 2) * geo.xi + warp * R;
#pragma unroll
      for (int r = 0; r < R; ++r) tb_add_col(E[r], te0, in[r], tf.ca[1]);
    }
    if (th1 >= 0) {
      const double* in = incr + (st * 4 + 3) * geo.xi + warp * R;
#pragma unroll
      for (int r = 0; r < R; ++r) tb_add_col(E[r], th1, in[r], -tf.ca[1]);
    }
    if (pxw) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = i0 + r, w = sx_.slot(i);
        if (w < 0 || !((okr >> r) & 1u)) continue;
        const T ca = XP[4 * w + 2], cb = XP[4 * w + 3];
        T p[C];
        tb_ld(p, PX + (nsx + w) * kTbCols + lane * C);
#pragma unroll
        for (int c = 0; c < C; ++c)
          if ((okc >> c) & 1u) {
            p[c] = psi_next_yz(cb, p[c], ca, hx(r, c));
            E[r][c] = mad(one ? e2 : lut[8 * ((mid[r] >> (8 * c)) & 0xffu) + 6], p[c], E[r][c]);
          }
        tb_st(PX + (nsx + w) * kTbCols + lane * C, p);
      }
    }
    if (yr >= 0) {
      T ca[C], cb[C];
      tb_ld(ca, YP + 2 * kTbCols + lane * C);
      tb_ld(cb, YP + 3 * kTbCols + lane * C);
      T* col = PY + (nsy + yr) * C * geo.xi + warp * R;
#pragma unroll
      for (int c0 = 0; c0 < C; c0 += 2, col += 2 * geo.xi) {
        T p[2][R];
        tb_ldr(p[0], col);
        tb_ldr(p[1], col + geo.xi);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          const int c = c0 + d;
#pragma unroll
          for (int r = 0; r < R; ++r)
            if ((okr >> r) & 1u) {
              p[d][r] = psi_next_yz(cb[c], p[d][r], ca[c], hy(r, c));
              E[r][c] = mad(one ? e1 : lut[8 * ((mid[r] >> (8 * c)) & 0xffu) + 5], p[d][r], E[r][c]);
            }
        }
        tb_str(col, p[0]);
        tb_str(col + geo.xi, p[1]);
      }
    }
    if (pr.n > 0) {
      for (int p = heads[tid]; p >= 0;) {  // record this lane's probes
        const int2 l = link[p];
        const int o = l.y >> 3, fld = l.y & 7;
        T v = T(0);
#pragma unroll
        for (int q = 0; q < R * C; ++q)
          if (q == o) v = fld == XFB_EZ ? E[q / C][q % C] : fld == XFB_HX ? HX[q / C][q % C] : HY[q / C][q % C];
        pr.out[p * pr.total_steps + t0 + st] = static_cast<double>(v);
        p = l.x;
      }
    }
    tb_st(xe + warp * kTbCols + lane * C, E[0]);
    tb_sync(blockDim.x);
  }
  }
  // ---- write back the interior (what the per-step kernel writes) --------------
  if (j0 >= J0 && j0 < J0 + geo.tj && j0 < ny) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = i0 + r;
      if (i < I0 || i >= I0 + geo.ti || i >= nx) continue;
      const long long g = i * sx + j0;
      const int sxs = sx_.slot(i);
      const long long px = sxs >= 0 ? slab(i, nx, pm.L[0], pm.L[1]) * sx : 0;
      if (j0 + C <= ny) {
        tb_st(d.hx + g, HX[r]);
        tb_st(d.hy + g, HY[r]);
        if (i >= 1 && j0 >= 1) tb_st(d.ez + g, E[r]);
      }
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int j = j0 + c;
        if (j >= ny) continue;
        const bool e_upd = i >= 1 && j >= 1;
        if (j0 + C > ny) {
          d.hx[g + c] = HX[r][c];
          d.hy[g + c] = HY[r][c];
        }
        if (e_upd && (j0 + C > ny || j0 < 1)) d.ez[g + c] = E[r][c];
        if (sxs >= 0) {
          pd.hy_x[px + j] = PX[sxs * kTbCols + lane * C + c];
          if (e_upd) ezx_w[px + j] = PX[(nsx + sxs) * kTbCols + lane * C + c];
        }
        if (yr >= 0 && sy_.slot(j) >= 0) {
          const long long p = i * pm.ysx + slab(j, ny, pm.L[2], pm.L[3]);
          pd.hx_y[p] = PY[(yr * C + c) * geo.xi + i - ib];
          if (e_upd) ezy_w[p] = PY[((nsy + yr) * C + c) * geo.xi + i - ib];
        }
      }
    }
  }
}

}  // namespace xfb
