// Host side of the blocked 2-D step: its tile plan and launches.  Included by
// tb2d_f32.cu (FMA contraction) and tb2d_f64.cu (--fmad=false).
#pragma once

#include "engine.cuh"
#include "tb2d.cuh"

namespace xfb {

// Shared-memory limit of a CTA.
constexpr size_t kTbSmem = 227u * 1024u;

// Largest CPML slab row and lane-block counts of any tile's region.
template <typename T>
void tb2d_slabs(const Compiled& c, int nw, int S, int& nsx, int& nsy) {
  const TbGeom<T> g(nw, S);
  nsx = nsy = 0;
  for (int i0 = 0; i0 < c.nx; i0 += g.ti) nsx = std::max(nsx, TbSlab(i0 - S, g.xi, c.nx, c.pml[0], c.pml[1]).count());
  for (int j0 = 0; j0 < c.ny; j0 += g.tj)
    nsy = std::max(nsy, TbBlocks(TbSlab(j0 - g.hl, kTbCols, c.ny, c.pml[2], c.pml[3]), j0 - g.hl).count());
}

template <typename T>
size_t tb2d_bytes(const Compiled& c, int nw, int S, int& nsx, int& nsy) {
  tb2d_slabs<T>(c, nw, S, nsx, nsy);
  return TbLayout<T>(nw, S, c.n_mat, nsx, nsy).bytes + (c.probes.empty() ? 0 : 32 * nw * sizeof(int));  // the probes' heads
}

// Whether a scene takes the blocked step.  The second set of the E-side psi it
// alternates with is part of a checkpoint, so the rule is kept as it was for
// the former tile (96 columns of which 2 S + 1 were halo, psi of at most 16
// slab rows and columns, 227 KB): states saved by either load into the other.
template <typename T>
bool tb2d_has_set(const xfb_handle* h) {
  const Compiled& c = h->c;
  const int S = h->tb_steps;
  if (c.dim != 2 || S <= 0 || !c.movies.empty()) return false;
  constexpr int kPitch = 96, kSlab = 16;
  const int TJ = kPitch - 1 - 2 * S;
  if (TJ < 16) return false;
  auto bytes = [&](int ti) {
    const size_t xi = ti + 2 * S + 1;
    const size_t px = (3 * xi * kPitch * sizeof(T) + xi * kPitch + 15) / 16 * 16;
    const size_t slots = px + 2ull * kSlab * kPitch * sizeof(T) + 2 * xi * kSlab * sizeof(T) + c.n_mat * 18ull * sizeof(T);
    return (slots + (xi + kPitch) * sizeof(int) + 15) / 16 * 16 + (4ull * kPitch + 4 * xi) * sizeof(double);
  };
  const int per = std::max(1, 296 / ((c.ny + TJ - 1) / TJ));
  int TI = std::min(64, std::max(16, (c.nx + per - 1) / per));
  while (TI > 16 && bytes(TI) > kTbSmem) --TI;
  if (bytes(TI) > kTbSmem) return false;
  auto fits = [&](int n, int tile, int lo, int hi) {
    for (int a0 = 0; a0 < n; a0 += tile) {
      int cnt = 0;
      for (int q = std::max(0, a0 - S); q <= std::min(n - 1, a0 + tile + S); ++q) cnt += (q < lo || q >= n - hi) ? 1 : 0;
      if (cnt > kSlab) return false;
    }
    return true;
  };
  return fits(c.nx, TI, c.pml[0], c.pml[1]) && fits(c.ny, TJ, c.pml[2], c.pml[3]);
}

// Warps per CTA (tile rows) and steps per launch of the blocked 2-D step, at
// most the caller's.  False (one launch per step) when blocking is off or the
// scene does not take it.
template <typename T>
bool tb2d_plan(xfb_handle* h) {
  const Compiled& c = h->c;
  h->tb_warps = 0;
  if (!tb2d_has_set<T>(h)) return false;
  // A grid that fills the GPU with the largest tiles takes them: its launches
  // are bound by issue slots, and the longest blocks lose more to their halo
  // than they save.  us per step with 16 warps and S = 5 / 7 / 9 / 11: FP32
  // 1044^2 7.5 / 6.5 / 6.6 / 6.7, 1521 x 753 7.7 / 6.9 / 7.0 / 7.5, 2020 x 1720
  // 13.1 / 11.9 / 11.6 / 11.4; FP64 1044^2 12.8 / 12.3 / 12.8 / 13.9, 1521 x 753
  // 13.7 / 13.3 / 13.8 / 14.7, 2020 x 1720 24.7 / 23.1 / 23.4 / 24.9.  Where the
  // last wave of the 7-step tiles is nearly empty, longer blocks are better than
  // this rule: FP32 900^2 6.5 at 7, 5.7 at 11, 1400 x 800 7.2 and 6.7, 1200^2 7.6
  // and 7.4; FP64 900^2 11.4 and (9) 10.8.
  auto tiles_of = [&](const TbGeom<T>& g) {
    return std::ceil(static_cast<double>(c.nx) / g.ti) * std::ceil(static_cast<double>(c.ny) / g.tj);
  };
  const double fill = tiles_of(TbGeom<T>(kTbMaxWarps<T>, 7)) / 148.0;
  int nw_lo = 4, S_hi = 11;
  if (fill >= 1) {
    nw_lo = kTbMaxWarps<T>;
    S_hi = sizeof(T) == 4 && fill >= 3 ? 9 : 7;
  }
  // Smaller grids: the cheapest pair by the cost model.
  double best = 0;
  for (int S = h->tb_given ? h->tb_steps : S_hi; S >= 1 && !(h->tb_warps && (h->tb_given || nw_lo > 4)); S -= 2)
    for (int nw = nw_lo; nw <= kTbMaxWarps<T>; nw += 2) {
      const TbGeom<T> g(nw, S);
      if (g.ti < kTbRows<T> || g.tj < kTbC) continue;
      int nsx, nsy;
      const size_t smem = tb2d_bytes<T>(c, nw, S, nsx, nsy);
      if (smem > kTbSmem) continue;
      const double tiles = tiles_of(g);
      const int per_sm = std::max(1, std::min<int>(kTbMaxWarps<T> / nw, static_cast<int>(228u * 1024u / (smem + 1024u))));
      // per wave, a tile's load and store and the steps of the CTAs that share an SM
      const double cost = (kTbFixed + std::ceil(tiles / (148.0 * per_sm)) * (kTbLoad + S * per_sm * nw * kTbWarpStep<T>)) / S;
      if (!h->tb_warps || cost < best) {
        best = cost;
        h->tb_warps = nw;
        h->tb_max = S;
      }
    }
  return h->tb_warps > 0;
}

// The kernel's shared-memory limit, set (and the kernel loaded) outside any
// stream capture of the step loop.
template <typename T>
int tb2d_prepare(xfb_handle* h) {
  XFB_CUDA(h, cudaFuncSetAttribute(k_step2_tb<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTbSmem)));
  return XFB_OK;
}

// One blocked 2-D launch: steps [off, off + S) of the chunk (S odd), read
// set and E-side psi buffer (step & 1), write the others.
template <typename T>
void launch_tb2d(xfb_handle* h, int off, int S) {
  const Compiled& c = h->c;
  const int parity = static_cast<int>((h->step + off) & 1), nw = h->tb_warps;
  int nsx, nsy;
  const size_t smem = tb2d_bytes<T>(c, nw, S, nsx, nsy);
  const TbGeom<T> g(nw, S);
  T* ez_x[2] = {as<T>(h->psi[1]), as<T>(h->psi_e1[0])};
  T* ez_y[2] = {as<T>(h->psi[2]), as<T>(h->psi_e1[1])};
  ProbeP pr{static_cast<int>(c.probes.size()), h->probe_idx, h->probe_field, h->probe_out, c.total_steps};
  const dim3 grid((c.ny + g.tj - 1) / g.tj, (c.nx + g.ti - 1) / g.ti);
  k_step2_tb<T><<<grid, 32 * nw, smem, h->stream>>>(
      grid_params<T>(h, parity), grid_params<T>(h, 1 - parity), pml_params<T>(h), psi_h_set<T>(h, parity),
      psi_h_set<T>(h, 1 - parity), ez_x[parity], ez_y[parity], ez_x[1 - parity], ez_y[1 - parity], tfsf_params(h),
      TimeP{h->t_dev, off}, pr, static_cast<int2*>(h->probe_link), S, c.n_mat, nsx, nsy);
}

// n steps as launches of odd step counts (each flips the sets once), as equal
// as they can be: a launch costs the same for few steps as for many.
template <typename T>
void tb2d_chunk(xfb_handle* h, int n) {
  int launches = (n + h->tb_max - 1) / h->tb_max;
  launches += (launches ^ n) & 1;
  int S = n / launches;
  S -= 1 - (S & 1);
  int longer = (n - S * launches) / 2;  // launches of S + 2 steps
  for (int off = 0; off < n;) {
    const int s = longer-- > 0 ? S + 2 : S;
    launch_tb2d<T>(h, off, s);
    off += s;
  }
}

}  // namespace xfb

#define XFB_INSTANTIATE_TB2D(T)                          \
  namespace xfb {                                        \
  template bool tb2d_plan<T>(xfb_handle*);               \
  template int tb2d_prepare<T>(xfb_handle*);             \
  template void launch_tb2d<T>(xfb_handle*, int, int);   \
  template void tb2d_chunk<T>(xfb_handle*, int);         \
  }
