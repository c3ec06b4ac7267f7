// Two-pass 3-D time step: an H pass and an E pass over the whole grid, in
// place on one field set, 16 bytes of every row per thread and no marching.
//
// The one-sweep step (k_step3) moves fewer bytes per cell (12 T + 1 against
// 18 T + 2) but walks plane after plane: a CTA holds two planes of a 16 x 32
// tile in flight, its CPML and TFSF items add dependent loads to every plane,
// and nothing hides them (two CTAs, 18 warps, per SM).  Here a thread owns V
// consecutive cells of one row (V = 4 FP32, 2 FP64): every operand is one
// 16-byte load, all loads of a pass are independent and issued first, up to 24
// warps per SM cover their latency, and the CPML and TFSF corrections run in the
// few warps that hold such cells.  Updating in place keeps one field set
// live, and the passes sweep the planes in opposite directions, so grids up to
// the L2's size stay there from pass to pass.
//
// In-place order: H^{n+1/2} of a cell needs its own old H and E^n of its upper
// neighbours, so the H pass writes only H and reads only E; E^{n+1} likewise
// writes only E and reads only H.  The polarisation currents of dispersive
// cells are advanced by blocks of the E pass or by k_tp_ade, which update E of
// those cells entirely (the pass's vectors leave them as E^n), one warp per run
// of cells; when a
// dispersive cell also takes a TFSF or CPML correction the E pass does the
// recursion itself.  The arithmetic and its order are those of k_h3 / k_e3 and
// of the one-sweep bodies: FP64 results are bit-identical, FP32 results equal
// those of the one-sweep step.
//
// What bounds it, measured on a B200 (us per step, with NF2FF and probes; the
// one-sweep step before): 156^3 FP32 65 (149), FP64 118 (240); 80x72x88 FP32 18.6
// (66); 36x32x40 FP64 14.9 (81); 128x152x136 Debye FP64 97 (244); 408^3
// Drude-Lorentz FP32 1183 (1356).  At 408^3 the H pass moves 2.69 GB in 0.43 ms
// and the E pass 2.64 in 0.42, 96 % of the copy bandwidth; at 280^3, with the
// dispersive runs in the E pass, 5.9 and 5.0 TB/s with 47 % L2 hits and 21 warps
// per SM (80 registers), where load latency shows; below that it dominates, and
// below 0.5 M cells the launches do.  Scenes without a CPML stay on the one-sweep
// step, whose lean interior body reaches 82 % of its 12 T + 1 bytes (384^3: 0.52 ms).
#pragma once

#include "fused3d.cuh"

namespace xfb {

template <typename T>
using Vec = Vec16<T>;

constexpr int kTpThreads = 128;  // threads of a CTA
// CTAs per SM the register budget is sized for (80 registers).  5, 6, 7 and 8
// measured 73, 69, 69 and 73 us per step on a 156^3 FP32 scene, 1248, 1191,
// 1190 and 1250 on a 408^3 one: more warps against spills.
constexpr int kTpBlocks = 6;

// Columns (vectors of a row) that hold a z-slab cell, a cell of a TFSF line at
// ks or ke, the wall k = 0 or cells past nz: the first `lo`, `n1` from c1,
// `n2` from c2, and the `hi` last.  Every row has them, so the warps of a
// plane take the plain columns of all rows first and the special ones apart:
// a warp of consecutive vectors would almost always hold a special one and run
// its code for a lane or two.
struct TpCols {
  int kv;              // vectors per row
  int lo, c1, n1, c2, n2, hi;
  int np, ns;          // plain and special columns
  unsigned mp, ms;     // ceil(2^32 / np), ceil(2^32 / ns)
  unsigned bp;         // CTAs of a plane that take the plain columns
};

template <typename T>
struct TpArgs {
  // the live field set, read and written: components Ex .. Hz and material
  // ids, shifted down by a plane and a row so that every byte offset of a
  // pass is a positive 32-bit number
  char* f[6];
  const uint8_t* mid;
  int nx, ny, nz;
  unsigned sxb, syb;  // plane and row strides in bytes
  long long sx, sy;   // ... in elements
  TpCols c;
  PmlP<T> pm;      // E-side psi
  PsiH<T> ps;      // H-side psi of the live set
  TfsfP tf;
  TimeP tp;
  AdeP<T> ad;      // kind kAdeNone unless the E pass does the recursion itself
  const T* lut8;   // [n_mat][8]
  int zvec;        // z-slab psi rows hold whole aligned vectors
  unsigned disp[8];  // materials of the dispersive cells outside the E pass's vectors (bit per id)
  // those cells' runs, the first run of each plane, the planes that have any,
  // and the blocks of a plane: its vectors' and (E pass with runs) its runs'
  AdeP<T> ar;
  GridP<T> g;
  const int2* runs;
  const int* run_first;
  int run_lo, run_hi;
  unsigned nblk, nade;
};

template <typename T>
__device__ __forceinline__ T& tp_at(const TpArgs<T>& a, int f, unsigned off) {
  return *reinterpret_cast<T*>(a.f[f] + off);
}

// Row and column of this thread's vector (false: none); bx: the CTA's block
// among its plane's.  The H pass walks the planes up and the E pass down, so each pass
// starts on the planes the last one left in L2.
template <typename T>
__device__ __forceinline__ bool tp_cell(const TpArgs<T>& a, unsigned bx, int& j, int& k0) {
  const TpCols& c = a.c;
  int q;
  if (bx < c.bp) {
    const unsigned t = bx * kTpThreads + threadIdx.x;
    if (t >= static_cast<unsigned>(a.ny) * static_cast<unsigned>(c.np)) return false;
    j = static_cast<int>(c.np > 1 ? __umulhi(t, c.mp) : t);
    q = c.lo + static_cast<int>(t) - j * c.np;
    if (q >= c.c1) q += c.n1;
    if (q >= c.c2) q += c.n2;
  } else {
    const unsigned t = (bx - c.bp) * kTpThreads + threadIdx.x;
    if (t >= static_cast<unsigned>(a.ny) * static_cast<unsigned>(c.ns)) return false;
    j = static_cast<int>(c.ns > 1 ? __umulhi(t, c.ms) : t);
    q = static_cast<int>(t) - j * c.ns;
    if (q >= c.lo) {
      if (q < c.lo + c.n1) q += c.c1 - c.lo;
      else if (q < c.lo + c.n1 + c.n2) q += c.c2 - c.lo - c.n1;
      else q += c.kv - c.ns;
    }
  }
  k0 = q * Vec<T>::V;
  return true;
}

// Byte offset of element (i, j, k) from the shifted component bases.
template <typename T>
__device__ __forceinline__ unsigned tp_off(const TpArgs<T>& a, int i, int j, int k) {
  return static_cast<unsigned>(i + 1) * a.sxb + static_cast<unsigned>(j + 1) * a.syb +
         static_cast<unsigned>(k) * static_cast<unsigned>(sizeof(T));
}

// The V material ids of a vector in one load, id of cell v in byte v; `same`
// when they are equal.
template <typename T>
__device__ __forceinline__ unsigned tp_mids(const TpArgs<T>& a, unsigned off, bool& same) {
  const uint8_t* p = a.mid + off / sizeof(T);
  if (Vec<T>::V == 4) {
    const unsigned m = *reinterpret_cast<const unsigned*>(p);
    same = m == (m & 0xffu) * 0x01010101u;
    return m;
  }
  const unsigned m = *reinterpret_cast<const unsigned short*>(p);
  same = (m & 0xffu) == (m >> 8);
  return m;
}

// TFSF corrections of a vector.  `add` puts tr * (incident value at projection
// p) * coef on one cell; the row forms run over the cells k in [lo, hi] with p =
// base + line[k] (- off).  Every term and its order are those of tfsf_h and
// tfsf_e.
template <typename T>
struct TpInc {
  const double* row;  // auxiliary row of the step
  double off;         // 0 (E), 0.5 (H)
  __device__ __forceinline__ void add(T& f, double p, double tr, double coef) const {
    add_inc(f, tr * aux_lerp(row, off != 0 ? p - off : p), coef);
  }
  __device__ __forceinline__ void run(Vec<T>& f, int k0, int lo, int hi, double base, const double* line, double tr,
                                      double coef) const {
#pragma unroll
    for (int v = 0; v < Vec<T>::V; ++v)
      if (k0 + v >= lo && k0 + v <= hi) add(f.a[v], base + line[k0 + v], tr, coef);
  }
};

template <typename T>
__device__ __forceinline__ void tp_tfsf_h(const TpArgs<T>& a, int i, int j, int k0, Vec<T>& hx, Vec<T>& hy, Vec<T>& hz) {
  const TfsfP& t = a.tf;
  const TpInc<T> in{t.e_tab + cur_step(a.tp) * (t.nl + 1), 0.0};
  const bool iin = i >= t.is && i <= t.ie, jin = j >= t.js && j <= t.je;
  const double* pk = t.pi2 - t.ks;      // projections at node k
  const double* hk = t.ph2 - t.ks + 1;  // ... at half node k
#pragma unroll
  for (int v = 0; v < Vec<T>::V; ++v) {  // columns ks-1, ke
    const int k = k0 + v;
    if (k != t.ks - 1 && k != t.ke) continue;
    const int fk = k == t.ke ? t.ke : t.ks;
    const double c = k == t.ke ? t.cb[2] : -t.cb[2];
    if (iin && jin && j < t.je) in.add(hx.a[v], t.pi0[i - t.is] + t.ph1[j - t.js + 1] + pk[fk], t.tre[1], c);
    if (iin && i < t.ie && jin) in.add(hy.a[v], t.ph0[i - t.is + 1] + t.pi1[j - t.js] + pk[fk], t.tre[0], -c);
  }
  if (i == t.is - 1 || i == t.ie) {
    const int fi = i == t.ie ? t.ie : t.is;
    const double c = i == t.ie ? -t.cb[0] : t.cb[0];
    if (jin && j < t.je) in.run(hz, k0, t.ks, t.ke, t.pi0[fi - t.is] + t.ph1[j - t.js + 1], pk, t.tre[1], c);
    if (jin) in.run(hy, k0, t.ks, t.ke - 1, t.pi0[fi - t.is] + t.pi1[j - t.js], hk, t.tre[2], -c);
  }
  if (j == t.js - 1 || j == t.je) {
    const int fj = j == t.je ? t.je : t.js;
    const double c = j == t.je ? t.cb[1] : -t.cb[1];
    if (iin && i < t.ie) in.run(hz, k0, t.ks, t.ke, t.ph0[i - t.is + 1] + t.pi1[fj - t.js], pk, t.tre[0], c);
    if (iin) in.run(hx, k0, t.ks, t.ke - 1, t.pi0[i - t.is] + t.pi1[fj - t.js], hk, t.tre[2], -c);
  }
}

template <typename T>
__device__ __forceinline__ void tp_tfsf_e(const TpArgs<T>& a, int i, int j, int k0, Vec<T>& ex, Vec<T>& ey, Vec<T>& ez) {
  const TfsfP& t = a.tf;
  const TpInc<T> in{t.h_tab + cur_step(a.tp) * t.nl, 0.5};
  const bool iin = i >= t.is && i <= t.ie, jin = j >= t.js && j <= t.je;
  const double* pk = t.pi2 - t.ks;
  const double* hk = t.ph2 - t.ks + 1;
#pragma unroll
  for (int v = 0; v < Vec<T>::V; ++v) {  // columns ks, ke
    const int k = k0 + v;
    if (k != t.ks && k != t.ke) continue;
    const int fk = k == t.ke ? t.ke : t.ks - 1;
    const double c = k == t.ke ? -t.ca[2] : t.ca[2];
    if (iin && i < t.ie && jin) in.add(ex.a[v], t.ph0[i - t.is + 1] + t.pi1[j - t.js] + hk[fk], t.trh[1], c);
    if (iin && jin && j < t.je) in.add(ey.a[v], t.pi0[i - t.is] + t.ph1[j - t.js + 1] + hk[fk], t.trh[0], -c);
  }
  if (i == t.is || i == t.ie) {
    const int fi = i == t.ie ? t.ie : t.is - 1;
    const double c = i == t.ie ? t.ca[0] : -t.ca[0];
    if (jin) in.run(ez, k0, t.ks, t.ke - 1, t.ph0[fi - t.is + 1] + t.pi1[j - t.js], hk, t.trh[1], c);
    if (jin && j < t.je) in.run(ey, k0, t.ks, t.ke, t.ph0[fi - t.is + 1] + t.ph1[j - t.js + 1], pk, t.trh[2], -c);
  }
  if (j == t.js || j == t.je) {
    const int fj = j == t.je ? t.je : t.js - 1;
    const double c = j == t.je ? -t.ca[1] : t.ca[1];
    if (iin) in.run(ez, k0, t.ks, t.ke - 1, t.pi0[i - t.is] + t.ph1[fj - t.js + 1], hk, t.trh[0], c);
    if (iin && i < t.ie) in.run(ex, k0, t.ks, t.ke, t.ph0[i - t.is + 1] + t.ph1[fj - t.js + 1], pk, t.trh[2], -c);
  }
}

// H pass of one vector cell by cell, out of line: the rare vectors that mix
// materials or TFSF cells with CPML cells.
template <typename T>
__device__ __noinline__ void tp_h_cells(const TpArgs<T>& a, int i, int j, int k0) {
  const TfsfP tf = a.tf.on ? tfsf_at_step(a.tf, cur_step(a.tp)) : a.tf;
  const PmlP<T>& pm = a.pm;
  const int sxp = slab(i, a.nx, pm.L[0], pm.L[1]), syp = slab(j, a.ny, pm.L[2], pm.L[3]);
  for (int k = k0; k < min(k0 + Vec<T>::V, a.nz); ++k) {
    const unsigned o = tp_off(a, i, j, k), ox = o + a.sxb, oy = o + a.syb, oz = o + sizeof(T);
    const C4<T> cf = ld_c4(a.lut8 + 8 * a.mid[o / sizeof(T)] + 4);
    const T ex = tp_at(a, 0, o), ey = tp_at(a, 1, o), ez = tp_at(a, 2, o);
    const T d_hx_a = tp_at(a, 1, oz) - ey, d_hx_b = tp_at(a, 2, oy) - ez;
    const T d_hy_a = tp_at(a, 2, ox) - ez, d_hy_b = tp_at(a, 0, oz) - ex;
    const T d_hz_a = tp_at(a, 0, oy) - ex, d_hz_b = tp_at(a, 1, ox) - ey;
    T hx = h_next(cf.c, tp_at(a, 3, o), cf.z, d_hx_a, cf.y, d_hx_b);
    T hy = h_next(cf.c, tp_at(a, 4, o), cf.x, d_hy_a, cf.z, d_hy_b);
    T hz = h_next(cf.c, tp_at(a, 5, o), cf.y, d_hz_a, cf.x, d_hz_b);
    if (tf.on) tfsf_h(tf, IncTables{tf}, i, j, k, hx, hy, hz);
    if (sxp >= 0) {
      const long long p = sxp * a.sx + j * a.sy + k;
      const T ca = pm.ah[0][i], cb = pm.bh[0][i];
      const T qy = psi_next_x(cb, a.ps.hy_x[p], ca, d_hy_a), qz = psi_next_x(cb, a.ps.hz_x[p], ca, d_hz_b);
      a.ps.hy_x[p] = qy; a.ps.hz_x[p] = qz;
      hy = mad(cf.x, qy, hy);   // chyez
      hz = mad(-cf.x, qz, hz);   // chzey
    }
    if (syp >= 0) {
      const long long p = i * pm.ysx + syp * a.sy + k;
      const T ca = pm.ah[1][j], cb = pm.bh[1][j];
      const T qz = psi_next_yz(cb, a.ps.hz_y[p], ca, d_hz_a), qx = psi_next_yz(cb, a.ps.hx_y[p], ca, d_hx_b);
      a.ps.hz_y[p] = qz; a.ps.hx_y[p] = qx;
      hz = mad(cf.y, qz, hz);   // chzex
      hx = mad(-cf.y, qx, hx);   // chxez
    }
    const int szp = slab(k, a.nz, pm.L[4], pm.L[5]);
    if (szp >= 0) {
      const long long p = i * pm.zsx + j * pm.zsy + szp;
      const T ca = pm.ah[2][k], cb = pm.bh[2][k];
      const T qx = psi_next_yz(cb, a.ps.hx_z[p], ca, d_hx_a), qy = psi_next_yz(cb, a.ps.hy_z[p], ca, d_hy_b);
      a.ps.hx_z[p] = qx; a.ps.hy_z[p] = qy;
      hx = mad(cf.z, qx, hx);   // chxey
      hy = mad(-cf.z, qy, hy);   // chyex
    }
    tp_at(a, 3, o) = hx; tp_at(a, 4, o) = hy; tp_at(a, 5, o) = hz;
  }
}

// E pass of one vector cell by cell: as tp_h_cells, and (FP64) dispersive vectors
// when no separate pass does the ADE recursion.
template <typename T>
__device__ __noinline__ void tp_e_cells(const TpArgs<T>& a, int i, int j, int k0) {
  const TfsfP tf = a.tf.on ? tfsf_at_step(a.tf, cur_step(a.tp)) : a.tf;
  const PmlP<T>& pm = a.pm;
  const AdeP<T>& ad = a.ad;
  const int sxp = slab(i, a.nx, pm.L[0], pm.L[1]), syp = slab(j, a.ny, pm.L[2], pm.L[3]);
  for (int k = k0; k < min(k0 + Vec<T>::V, a.nz); ++k) {
    const unsigned o = tp_off(a, i, j, k), ox = o - a.sxb, oy = o - a.syb, oz = o - sizeof(T);
    const int m = a.mid[o / sizeof(T)];
    if ((a.disp[m >> 5] >> (m & 31)) & 1u) continue;  // a run's cell
    const bool upd_x = j > 0 && k > 0, upd_y = i > 0 && k > 0, upd_z = i > 0 && j > 0;
    const C4<T> cf = ld_c4(a.lut8 + 8 * m);
    const T hx = tp_at(a, 3, o), hy = tp_at(a, 4, o), hz = tp_at(a, 5, o);
    const T d_ex_a = hy - tp_at(a, 4, oz), d_ex_b = hz - tp_at(a, 5, oy);
    const T d_ey_a = hz - tp_at(a, 5, ox), d_ey_b = hx - tp_at(a, 3, oz);
    const T d_ez_a = hx - tp_at(a, 3, oy), d_ez_b = hy - tp_at(a, 4, ox);
    const T ex_o = tp_at(a, 0, o), ey_o = tp_at(a, 1, o), ez_o = tp_at(a, 2, o);
    T ex = e_next(cf.c, ex_o, cf.z, d_ex_a, cf.y, d_ex_b);
    T ey = e_next(cf.c, ey_o, cf.x, d_ey_a, cf.z, d_ey_b);
    T ez = e_next(cf.c, ez_o, cf.y, d_ez_a, cf.x, d_ez_b);
    if constexpr (sizeof(T) == 8) {  // (such FP32 scenes stay on the one-sweep step: tp_mixed_rounding)
      if (ad.kind != kAdeNone && ad.mat[3 * m] != T(0)) {
        const long long bi = static_cast<long long>(i - ad.b0) * ad.bsx + static_cast<long long>(j - ad.b2) * ad.bsy + (k - ad.b4);
        if (upd_x) ex = ade_e(ad, 0, bi, m, ex_o, ex);
        if (upd_y) ey = ade_e(ad, 1, bi, m, ey_o, ey);
        if (upd_z) ez = ade_e(ad, 2, bi, m, ez_o, ez);
      }
    }
    if (tf.on) tfsf_e(tf, IncTables{tf}, i, j, k, ex, ey, ez);
    if (sxp >= 0) {
      const long long p = sxp * a.sx + j * a.sy + k;
      const T ca = pm.ae[0][i], cb = pm.be[0][i];
      if (upd_y) { const T q = psi_next_x(cb, pm.ey_x[p], ca, d_ey_a); pm.ey_x[p] = q; ey = mad(-cf.x, q, ey); }  // ceyhz
      if (upd_z) { const T q = psi_next_x(cb, pm.ez_x[p], ca, d_ez_b); pm.ez_x[p] = q; ez = mad(cf.x, q, ez); }  // cezhy
    }
    if (syp >= 0) {
      const long long p = i * pm.ysx + syp * a.sy + k;
      const T ca = pm.ae[1][j], cb = pm.be[1][j];
      if (upd_z) { const T q = psi_next_yz(cb, pm.ez_y[p], ca, d_ez_a); pm.ez_y[p] = q; ez = mad(-cf.y, q, ez); }  // cezhx
      if (upd_x) { const T q = psi_next_yz(cb, pm.ex_y[p], ca, d_ex_b); pm.ex_y[p] = q; ex = mad(cf.y, q, ex); }  // cexhz
    }
    const int szp = slab(k, a.nz, pm.L[4], pm.L[5]);
    if (szp >= 0) {
      const long long p = i * pm.zsx + j * pm.zsy + szp;
      const T ca = pm.ae[2][k], cb = pm.be[2][k];
      if (upd_x) { const T q = psi_next_yz(cb, pm.ex_z[p], ca, d_ex_a); pm.ex_z[p] = q; ex = mad(-cf.z, q, ex); }  // cexhy
      if (upd_y) { const T q = psi_next_yz(cb, pm.ey_z[p], ca, d_ey_b); pm.ey_z[p] = q; ey = mad(cf.z, q, ey); }  // ceyhx
    }
    if (upd_x) tp_at(a, 0, o) = ex;
    if (upd_y) tp_at(a, 1, o) = ey;
    if (upd_z) tp_at(a, 2, o) = ez;
  }
}

template <typename T>
__global__ void __launch_bounds__(kTpThreads, kTpBlocks) k_tp_h(const __grid_constant__ TpArgs<T> a) {
  constexpr int V = Vec<T>::V;
  const int i = blockIdx.y;
  int j, k0;
  if (!tp_cell(a, blockIdx.x, j, k0)) return;
  const unsigned o = tp_off(a, i, j, k0), ox = o + a.sxb, oy = o + a.syb;
  Vec<T> ex, ey, ez, eyn, ezn, exj, ezj, hx, hy, hz;
  ex.ld(a.f[0] + o); ey.ld(a.f[1] + o); ez.ld(a.f[2] + o);
  eyn.ld(a.f[1] + ox); ezn.ld(a.f[2] + ox);
  exj.ld(a.f[0] + oy); ezj.ld(a.f[2] + oy);
  const T exk = tp_at(a, 0, o + 16), eyk = tp_at(a, 1, o + 16);
  hx.ld(a.f[3] + o); hy.ld(a.f[4] + o); hz.ld(a.f[5] + o);
  bool same;
  const unsigned mids = tp_mids(a, o, same);
  const int m = static_cast<int>(mids & 0xffu);
  const TfsfP& tf = a.tf;
  const bool tfc = tf.on && (i == tf.is - 1 || i == tf.ie || j == tf.js - 1 || j == tf.je ||
                             (tf.ks > k0 && tf.ks - 1 < k0 + V) || (tf.ke >= k0 && tf.ke < k0 + V)) &&
                   i >= tf.is - 1 && i <= tf.ie && j >= tf.js - 1 && j <= tf.je && k0 + V >= tf.ks && k0 <= tf.ke;
  const PmlP<T>& pm = a.pm;
  const int sxp = slab(i, a.nx, pm.L[0], pm.L[1]);
  const int syp = slab(j, a.ny, pm.L[2], pm.L[3]);
  const bool zsl = k0 < pm.L[4] || k0 + V > a.nz - pm.L[5];
  if ((!same && (sxp >= 0 || syp >= 0 || zsl)) || (tfc && zsl)) {
    tp_h_cells(a, i, j, k0);
    return;
  }
  C4<T> cf = ld_c4(a.lut8 + 8 * m + 4);  // ch, db/dx, db/dy, db/dz
  // derivatives along z (the upper neighbour of the last cell is a scalar)
  auto dz = [&](const Vec<T>& e, T ek, int v) { return (v + 1 < V ? e.a[(v + 1) % V] : ek) - e.a[v]; };
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (v > 0 && !same) cf = ld_c4(a.lut8 + 8 * ((mids >> (8 * v)) & 0xffu) + 4);
    hx.a[v] = h_next(cf.c, hx.a[v], cf.z, dz(ey, eyk, v), cf.y, ezj.a[v] - ez.a[v]);
    hy.a[v] = h_next(cf.c, hy.a[v], cf.x, ezn.a[v] - ez.a[v], cf.z, dz(ex, exk, v));
    hz.a[v] = h_next(cf.c, hz.a[v], cf.y, exj.a[v] - ex.a[v], cf.x, eyn.a[v] - ey.a[v]);
  }
  if (tfc) tp_tfsf_h(a, i, j, k0, hx, hy, hz);
  if (sxp >= 0) {
    const long long p = sxp * a.sx + j * a.sy + k0;
    const T ca = pm.ah[0][i], cb = pm.bh[0][i];
    Vec<T> py, pz;
    py.ld(a.ps.hy_x + p); pz.ld(a.ps.hz_x + p);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      py.a[v] = psi_next_x(cb, py.a[v], ca, (ezn.a[v] - ez.a[v]));
      hy.a[v] = mad(cf.x, py.a[v], hy.a[v]);   // chyez
      pz.a[v] = psi_next_x(cb, pz.a[v], ca, (eyn.a[v] - ey.a[v]));
      hz.a[v] = mad(-cf.x, pz.a[v], hz.a[v]);   // chzey
    }
    py.st(a.ps.hy_x + p); pz.st(a.ps.hz_x + p);
  }
  if (syp >= 0) {
    const long long p = i * pm.ysx + syp * a.sy + k0;
    const T ca = pm.ah[1][j], cb = pm.bh[1][j];
    Vec<T> pz, px;
    pz.ld(a.ps.hz_y + p); px.ld(a.ps.hx_y + p);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      pz.a[v] = psi_next_yz(cb, pz.a[v], ca, (exj.a[v] - ex.a[v]));
      hz.a[v] = mad(cf.y, pz.a[v], hz.a[v]);   // chzex
      px.a[v] = psi_next_yz(cb, px.a[v], ca, (ezj.a[v] - ez.a[v]));
      hx.a[v] = mad(-cf.y, px.a[v], hx.a[v]);   // chxez
    }
    pz.st(a.ps.hz_y + p); px.st(a.ps.hx_y + p);
  }
  if (zsl) {
    const long long pr = i * pm.zsx + j * pm.zsy;
    if (a.zvec) {
      const long long p = pr + slab(k0, a.nz, pm.L[4], pm.L[5]);
      Vec<T> px, py, ca, cb;
      px.ld(a.ps.hx_z + p); py.ld(a.ps.hy_z + p);
      ca.ld(pm.ah[2] + k0); cb.ld(pm.bh[2] + k0);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        px.a[v] = psi_next_yz(cb.a[v], px.a[v], ca.a[v], dz(ey, eyk, v));
        hx.a[v] = mad(cf.z, px.a[v], hx.a[v]);   // chxey
        py.a[v] = psi_next_yz(cb.a[v], py.a[v], ca.a[v], dz(ex, exk, v));
        hy.a[v] = mad(-cf.z, py.a[v], hy.a[v]);   // chyex
      }
      px.st(a.ps.hx_z + p); py.st(a.ps.hy_z + p);
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int s = k0 + v < a.nz ? slab(k0 + v, a.nz, pm.L[4], pm.L[5]) : -1;
        if (s < 0) continue;
        const T ca = pm.ah[2][k0 + v], cb = pm.bh[2][k0 + v];
        const T qx = psi_next_yz(cb, a.ps.hx_z[pr + s], ca, dz(ey, eyk, v));
        hx.a[v] = mad(cf.z, qx, hx.a[v]);   // chxey
        const T qy = psi_next_yz(cb, a.ps.hy_z[pr + s], ca, dz(ex, exk, v));
        hy.a[v] = mad(-cf.z, qy, hy.a[v]);   // chyex
        a.ps.hx_z[pr + s] = qx;
        a.ps.hy_z[pr + s] = qy;
      }
    }
  }
  if (k0 + V > a.nz) {  // entries past the last cell keep their value
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (k0 + v >= a.nz) {
        const unsigned ov = o + v * static_cast<unsigned>(sizeof(T));
        hx.a[v] = tp_at(a, 3, ov); hy.a[v] = tp_at(a, 4, ov); hz.a[v] = tp_at(a, 5, ov);
      }
  }
  hx.st(a.f[3] + o); hy.st(a.f[4] + o); hz.st(a.f[5] + o);
}

// E update of the dispersive cells of a run (E pass of the other cells leaves
// them, and they read only H and their own E): the plain eNext value from
// H^{n+1/2} and the ADE recursion of ade_box_cell on it, one warp per run of
// at most 32 cells inside a 32-aligned k segment (the runs of k_ade_runs).
template <typename T, int MP>
__device__ __forceinline__ void tp_ade_run(const TpArgs<T>& a, int q) {
  const int lane = threadIdx.x & 31;
  const int2 r = a.runs[q];
  const int lo = (r.y >> 16) & 0xff, hi = static_cast<int>(static_cast<unsigned>(r.y) >> 24);
  if (lane < lo || lane >= hi) return;
  const int i = r.x & 0xffff, j = static_cast<int>(static_cast<unsigned>(r.x) >> 16), k = (r.y & 0xffff) + lane;
  const unsigned o = tp_off(a, i, j, k), ox = o - a.sxb, oy = o - a.syb, oz = o - sizeof(T);
  const int m = a.mid[o / sizeof(T)];
  const T hx = tp_at(a, 3, o), hy = tp_at(a, 4, o), hz = tp_at(a, 5, o);
  const T hx_km = tp_at(a, 3, oz), hy_km = tp_at(a, 4, oz), hx_jm = tp_at(a, 3, oy), hz_jm = tp_at(a, 5, oy);
  const T hy_p = tp_at(a, 4, ox), hz_p = tp_at(a, 5, ox);
  const T ec[3] = {tp_at(a, 0, o), tp_at(a, 1, o), tp_at(a, 2, o)};
  const C4<T> cf = ld_c4(a.lut8 + 8 * m);
  T pl[3];
  pl[0] = e_next(cf.c, ec[0], cf.z, hy - hy_km, cf.y, hz - hz_jm);
  pl[1] = e_next(cf.c, ec[1], cf.x, hz - hz_p, cf.z, hx - hx_km);
  pl[2] = e_next(cf.c, ec[2], cf.y, hx - hx_jm, cf.x, hy - hy_p);
  ade_cell<T, MP>(a.g, a.ar, i, j, k, i * a.g.sx + j * a.g.sy + k, m, ec, pl);
}

// All runs, a pass of its own where tp_ade_inside says so.
template <typename T>
__global__ void __launch_bounds__(128) k_tp_ade(const __grid_constant__ TpArgs<T> a, int n_runs) {
  const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (q < n_runs) tp_ade_run<T, 4>(a, q);
}

// kRuns: the grid is one row of blocks, and every plane that has dispersive
// runs has nade blocks for them (a warp per run) after its vectors' blocks.
// Beside the vectors of their plane the runs find the H that these read in L2,
// and the two kinds of loads overlap (tp_ade_inside).
template <typename T, bool kRuns>
__global__ void __launch_bounds__(kTpThreads, kTpBlocks) k_tp_e(const __grid_constant__ TpArgs<T> a) {
  constexpr int V = Vec<T>::V;
  int y = static_cast<int>(blockIdx.y);
  unsigned bx = blockIdx.x;
  if constexpr (kRuns) {
    const unsigned top = (a.nx - a.run_hi) * a.nblk, mid = (a.run_hi - a.run_lo) * (a.nblk + a.nade);
    unsigned per = a.nblk;
    if (bx >= top + mid) { y = a.nx - a.run_lo; bx -= top + mid; }
    else if (bx >= top) { y = a.nx - a.run_hi; bx -= top; per += a.nade; }
    const unsigned q = bx / per;
    y += static_cast<int>(q);
    bx -= q * per;
  }
  const int i = a.nx - 1 - y;
  if constexpr (kRuns) {
    if (bx >= a.nblk) {
      const int q = a.run_first[i] + static_cast<int>((bx - a.nblk) * (kTpThreads / 32) + (threadIdx.x >> 5));
      if (q < a.run_first[i + 1]) tp_ade_run<T, kTpAdePoles>(a, q);
      return;
    }
  }
  int j, k0;
  if (!tp_cell(a, bx, j, k0)) return;
  const unsigned o = tp_off(a, i, j, k0), ox = o - a.sxb, oy = o - a.syb;
  Vec<T> hx, hy, hz, hxj, hzj, hyi, hzi, ex, ey, ez;
  hx.ld(a.f[3] + o); hy.ld(a.f[4] + o); hz.ld(a.f[5] + o);
  hxj.ld(a.f[3] + oy); hzj.ld(a.f[5] + oy);
  hyi.ld(a.f[4] + ox); hzi.ld(a.f[5] + ox);
  const T hxk = tp_at(a, 3, o - static_cast<unsigned>(sizeof(T))), hyk = tp_at(a, 4, o - static_cast<unsigned>(sizeof(T)));
  ex.ld(a.f[0] + o); ey.ld(a.f[1] + o); ez.ld(a.f[2] + o);
  bool same;
  const unsigned mids = tp_mids(a, o, same);
  const int m = static_cast<int>(mids & 0xffu);
  const TfsfP& tf = a.tf;
  const bool tfc = tf.on && (i == tf.is || i == tf.ie || j == tf.js || j == tf.je || (tf.ks >= k0 && tf.ks < k0 + V) ||
                             (tf.ke >= k0 && tf.ke < k0 + V)) &&
                   i >= tf.is && i <= tf.ie && j >= tf.js && j <= tf.je && k0 + V > tf.ks && k0 <= tf.ke;
  const PmlP<T>& pm = a.pm;
  const int sxp = slab(i, a.nx, pm.L[0], pm.L[1]);
  const int syp = slab(j, a.ny, pm.L[2], pm.L[3]);
  const bool zsl = k0 < pm.L[4] || k0 + V > a.nz - pm.L[5];
  // cells to leave as they are: dispersive ones of the runs (a.ad: FP64 only, see tp_e_cells)
  unsigned keep = 0;
  bool inline_ade = false;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const unsigned mv = (mids >> (8 * v)) & 0xffu;
    keep |= ((a.disp[mv >> 5] >> (mv & 31)) & 1u) << v;
    if (a.ad.kind != kAdeNone) inline_ade = inline_ade || a.ad.mat[3 * mv] != T(0);
  }
  if (inline_ade || (!same && (sxp >= 0 || syp >= 0 || zsl)) || (tfc && zsl)) {
    tp_e_cells(a, i, j, k0);
    return;
  }
  if (keep == (1u << V) - 1u) return;
  C4<T> cf = ld_c4(a.lut8 + 8 * m);  // ce, cb/dx, cb/dy, cb/dz
  auto dz = [&](const Vec<T>& h, T hk, int v) { return h.a[v] - (v > 0 ? h.a[(v + V - 1) % V] : hk); };
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (v > 0 && !same) cf = ld_c4(a.lut8 + 8 * ((mids >> (8 * v)) & 0xffu));
    ex.a[v] = e_next(cf.c, ex.a[v], cf.z, dz(hy, hyk, v), cf.y, hz.a[v] - hzj.a[v]);
    ey.a[v] = e_next(cf.c, ey.a[v], cf.x, hz.a[v] - hzi.a[v], cf.z, dz(hx, hxk, v));
    ez.a[v] = e_next(cf.c, ez.a[v], cf.y, hx.a[v] - hxj.a[v], cf.x, hy.a[v] - hyi.a[v]);
  }
  if (tfc) tp_tfsf_e(a, i, j, k0, ex, ey, ez);
  // (the psi of components on PEC walls, which are never updated, is not read)
  if (sxp >= 0 && i > 0) {
    const long long p = sxp * a.sx + j * a.sy + k0;
    const T ca = pm.ae[0][i], cb = pm.be[0][i];
    Vec<T> py, pz;
    py.ld(pm.ey_x + p); pz.ld(pm.ez_x + p);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      py.a[v] = psi_next_x(cb, py.a[v], ca, (hz.a[v] - hzi.a[v]));
      ey.a[v] = mad(-cf.x, py.a[v], ey.a[v]);   // ceyhz
      pz.a[v] = psi_next_x(cb, pz.a[v], ca, (hy.a[v] - hyi.a[v]));
      ez.a[v] = mad(cf.x, pz.a[v], ez.a[v]);   // cezhy
    }
    py.st(pm.ey_x + p); pz.st(pm.ez_x + p);
  }
  if (syp >= 0 && j > 0) {
    const long long p = i * pm.ysx + syp * a.sy + k0;
    const T ca = pm.ae[1][j], cb = pm.be[1][j];
    Vec<T> pz, px;
    pz.ld(pm.ez_y + p); px.ld(pm.ex_y + p);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      pz.a[v] = psi_next_yz(cb, pz.a[v], ca, (hx.a[v] - hxj.a[v]));
      ez.a[v] = mad(-cf.y, pz.a[v], ez.a[v]);   // cezhx
      px.a[v] = psi_next_yz(cb, px.a[v], ca, (hz.a[v] - hzj.a[v]));
      ex.a[v] = mad(cf.y, px.a[v], ex.a[v]);   // cexhz
    }
    pz.st(pm.ez_y + p); px.st(pm.ex_y + p);
  }
  if (zsl) {
    const long long pr = i * pm.zsx + j * pm.zsy;
    if (a.zvec) {
      const long long p = pr + slab(k0, a.nz, pm.L[4], pm.L[5]);
      Vec<T> px, py, ca, cb;
      px.ld(pm.ex_z + p); py.ld(pm.ey_z + p);
      ca.ld(pm.ae[2] + k0); cb.ld(pm.be[2] + k0);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        px.a[v] = psi_next_yz(cb.a[v], px.a[v], ca.a[v], dz(hy, hyk, v));
        ex.a[v] = mad(-cf.z, px.a[v], ex.a[v]);   // cexhy
        py.a[v] = psi_next_yz(cb.a[v], py.a[v], ca.a[v], dz(hx, hxk, v));
        ey.a[v] = mad(cf.z, py.a[v], ey.a[v]);   // ceyhx
      }
      px.st(pm.ex_z + p); py.st(pm.ey_z + p);
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int s = k0 + v < a.nz ? slab(k0 + v, a.nz, pm.L[4], pm.L[5]) : -1;
        if (s < 0) continue;
        const T ca = pm.ae[2][k0 + v], cb = pm.be[2][k0 + v];
        const T qx = psi_next_yz(cb, pm.ex_z[pr + s], ca, dz(hy, hyk, v));
        ex.a[v] = mad(-cf.z, qx, ex.a[v]);   // cexhy
        const T qy = psi_next_yz(cb, pm.ey_z[pr + s], ca, dz(hx, hxk, v));
        ey.a[v] = mad(cf.z, qy, ey.a[v]);   // ceyhx
        pm.ex_z[pr + s] = qx;
        pm.ey_z[pr + s] = qy;
      }
    }
  }
  // components on PEC walls and entries past the last cell keep their value
  if (i == 0 || j == 0) {
    if (i == 0) { ey.ld(a.f[1] + o); ez.ld(a.f[2] + o); }
    if (j == 0) { ex.ld(a.f[0] + o); ez.ld(a.f[2] + o); }
  }
  if (k0 == 0) { ex.a[0] = tp_at(a, 0, o); ey.a[0] = tp_at(a, 1, o); }
  if (k0 + V > a.nz) {
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (k0 + v >= a.nz) {
        const unsigned ov = o + v * static_cast<unsigned>(sizeof(T));
        ex.a[v] = tp_at(a, 0, ov); ey.a[v] = tp_at(a, 1, ov); ez.a[v] = tp_at(a, 2, ov);
      }
  }
  if (keep) {  // the vector also holds cells of runs
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (!((keep >> v) & 1u)) {
        const unsigned ov = o + v * static_cast<unsigned>(sizeof(T));
        tp_at(a, 0, ov) = ex.a[v]; tp_at(a, 1, ov) = ey.a[v]; tp_at(a, 2, ov) = ez.a[v];
      }
    return;
  }
  ex.st(a.f[0] + o); ey.st(a.f[1] + o); ez.st(a.f[2] + o);
}

}  // namespace xfb
