// Host side of the blocked 2-D step: its tile plan and launches.  Included by
// tb2d_f32.cu (FMA contraction) and tb2d_f64.cu (--fmad=false).
#pragma once

#include "engine.cuh"
#include "tb2d.cuh"

namespace xfb {

// Tile of the blocked 2-D step: TJ + 2 S + 1 columns fill a shared row of
// kTbPitch, TI rows keep the tile count within two CTAs per SM when it can
// and the tile's shared memory within a CTA's 227 KB.
// False (one launch per step) when blocking is off, the scene has movie
// monitors (recorded between steps), or a tile's region would hold more CPML
// rows or columns than its psi tables.
template <typename T>
bool tb2d_plan(xfb_handle* h) {
  const Compiled& c = h->c;
  const int S = h->tb_steps;
  if (c.dim != 2 || S <= 0 || !c.movies.empty()) return false;
  const int TJ = kTbPitch - 1 - 2 * S;
  if (TJ < 16) return false;
  const int ntj = (c.ny + TJ - 1) / TJ;
  int TI = (c.nx + std::max(1, 296 / ntj) - 1) / std::max(1, 296 / ntj);
  TI = std::min(64, std::max(16, TI));
  // the tile's shared memory within the 227 KB a CTA may use
  while (TI > 16 && TbLayout<T>(TI + 2 * S + 1, c.n_mat).bytes > 227u * 1024u) --TI;
  if (TbLayout<T>(TI + 2 * S + 1, c.n_mat).bytes > 227u * 1024u) return false;
  auto fits = [&](int n, int tile, int lo, int hi) {  // slab cells of every tile's region along one axis
    for (int a0 = 0; a0 < n; a0 += tile) {
      int cnt = 0;
      for (int q = std::max(0, a0 - S); q <= std::min(n - 1, a0 + tile + S); ++q) cnt += (q < lo || q >= n - hi) ? 1 : 0;
      if (cnt > kTbSlab) return false;
    }
    return true;
  };
  if (!fits(c.nx, TI, c.pml[0], c.pml[1]) || !fits(c.ny, TJ, c.pml[2], c.pml[3])) return false;
  h->tb_ti = TI;
  h->tb_tj = TJ;
  return true;
}

// The kernel's shared-memory limit, set (and the kernel loaded) outside any
// stream capture of the step loop.
template <typename T>
int tb2d_prepare(xfb_handle* h) {
  const TbLayout<T> lay(h->tb_ti + 2 * h->tb_steps + 1, h->c.n_mat);
  XFB_CUDA(h, cudaFuncSetAttribute(k_step2_tb<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(lay.bytes)));
  return XFB_OK;
}

// One blocked 2-D launch: steps [off, off + S) of the chunk (S odd), read
// set and E-side psi buffer (step & 1), write the others.
template <typename T>
void launch_tb2d(xfb_handle* h, int off, int S) {
  const Compiled& c = h->c;
  const int parity = static_cast<int>((h->step + off) & 1);
  const TbLayout<T> lay(h->tb_ti + 2 * S + 1, c.n_mat);
  T* ez_x[2] = {as<T>(h->psi[1]), as<T>(h->psi_e1[0])};
  T* ez_y[2] = {as<T>(h->psi[2]), as<T>(h->psi_e1[1])};
  ProbeP pr{static_cast<int>(c.probes.size()), h->probe_idx, h->probe_field, h->probe_out, c.total_steps};
  const dim3 grid((c.ny + h->tb_tj - 1) / h->tb_tj, (c.nx + h->tb_ti - 1) / h->tb_ti);
  k_step2_tb<T><<<grid, kTbThreads, lay.bytes, h->stream>>>(
      grid_params<T>(h, parity), grid_params<T>(h, 1 - parity), pml_params<T>(h), psi_h_set<T>(h, parity),
      psi_h_set<T>(h, 1 - parity), ez_x[parity], ez_y[parity], ez_x[1 - parity], ez_y[1 - parity], tfsf_params(h),
      TimeP{h->t_dev, off}, pr, S, h->tb_ti, h->tb_tj, c.n_mat, h->scratch_err);
}

}  // namespace xfb

#define XFB_INSTANTIATE_TB2D(T)                          \
  namespace xfb {                                        \
  template bool tb2d_plan<T>(xfb_handle*);               \
  template int tb2d_prepare<T>(xfb_handle*);             \
  template void launch_tb2d<T>(xfb_handle*, int, int);   \
  }
