// Host side of the two-pass 3-D step: the rule that picks it and its launches.
// Included by twopass_f32.cu (FMA contraction) and twopass_f64.cu
// (--fmad=false), so the engine units need not be rebuilt for these kernels.
#pragma once

#include "engine.cuh"
#include "twopass.cuh"

namespace xfb {

// FP32: the one-sweep step's general body, which takes CPML columns that meet
// both faces of a thin TFSF box or dispersive cells, contracts the y and z psi
// update the other way round than its bulk-copy bodies.  The two-pass step
// rounds as the latter, so a scene with such columns stays on the one-sweep
// step and no scene's FP32 results depend on the choice.
inline bool tp_mixed_rounding(const xfb_handle* h, int TJ) {
  const Compiled& c = h->c;
  if (c.ade_kind != XFB_ADE_NONE && c.ade_box[1] > c.ade_box[0] && !h->ade_deferred) return true;
  if (!c.tfsf_on) return false;
  for (int j0 = 0; j0 < c.ny; j0 += TJ)
    for (int k0 = 0; k0 < c.nz; k0 += 32)
      if (tfsf_line_face(c.tf[2], c.tf[3], j0, TJ) == 2 || tfsf_line_face(c.tf[4], c.tf[5], k0, 32) == 2) return true;
  return false;
}

// Whether the automatic path takes the two-pass step: scenes with a CPML whose
// byte offsets fit 32 bits, thread indices the reciprocals of tp_cell and the
// plane count the launch grid; deferred ADE cells need their run list.
template <typename T>
bool tp_plan(const xfb_handle* h) {
  const Compiled& c = h->c;
  if (!h->path_auto || c.dim != 3 || is_slab(h)) return false;
  const double kv = (c.nz + Vec<T>::V - 1) / Vec<T>::V;
  if (c.nx > 65535 || c.ny * kv * kv >= 4294967296.0) return false;
  if ((c.nx + 3.0) * h->sx * sizeof(T) >= 4294967296.0) return false;
  if (h->ade_deferred && h->n_ade_runs < 0) return false;
  if (sizeof(T) == 4 && tp_mixed_rounding(h, kStepTileRows[step_tile_index(h->tj)])) return false;
  // a TFSF layer inside a CPML slab takes its corrections before the CPML's,
  // which the passes' vectors do only along z (tp_h_cells)
  if (c.tfsf_on)
    for (int ax = 0; ax < 2; ++ax)
      if (c.tf[2 * ax] - 1 < c.pml[2 * ax] || c.tf[2 * ax + 1] >= (ax ? c.ny : c.nx) - c.pml[2 * ax + 1]) return false;
  for (int f = 0; f < 6; ++f)
    if (c.pml[f]) return true;
  return false;
}

// Whether a batch left to the library takes the two-pass step for its scenes.
// All of them must (and in FP32 round alike whichever tile the one-sweep
// autotune would have picked).  Before and after, us per step: FP32 4 scenes of
// 48..64 cells a side 129 -> 30, 16 of 60..120 950 -> 447, 64 of 64..256 11870
// -> 8215 (4.9 TB/s); FP64 16 of 24..40 344 -> 100, 16 of 60..120 1618 -> 781.
template <typename T>
bool tp_batch_plan(const xfb_batch* b) {
  if (b->tile_req != 0 || b->launch_req != XFB_BATCH_AUTO) return false;
  for (const xfb_handle* h : b->hs) {
    if (!h->two_pass) return false;
    for (int t = 0; sizeof(T) == 4 && t < kStepTileCount; ++t)
      if (tp_mixed_rounding(h, kStepTileRows[t])) return false;
  }
  return true;
}

template <typename T>
TpCols tp_columns(const Compiled& c) {
  constexpr int V = Vec<T>::V;
  TpCols t{};
  t.kv = (c.nz + V - 1) / V;
  std::vector<char> special(t.kv, 0);
  auto mark = [&](int k) { if (k >= 0 && k < t.kv * V) special[k / V] = 1; };
  mark(0);
  for (int k = 0; k < c.pml[4]; ++k) mark(k);
  for (int k = c.nz - c.pml[5]; k < t.kv * V; ++k) mark(k);
  // the special columns as runs: the first and (if any) last of the row, and
  // up to two between them
  if (c.tfsf_on)
    for (int k : {c.tf[4] - 1, c.tf[4], c.tf[5]}) mark(k);
  int q = 0;
  while (q < t.kv && special[q]) ++q;
  t.lo = q;
  int e = t.kv;
  while (e > t.lo && special[e - 1]) --e;
  t.hi = t.kv - e;
  t.c1 = t.c2 = t.kv;
  while (q < e && !special[q]) ++q;
  if (q < e) {
    t.c1 = q;
    while (q < e && special[q]) ++q;
    t.n1 = q - t.c1;
    while (q < e && !special[q]) ++q;
    if (q < e) {
      t.c2 = q;
      while (q < e && special[q]) ++q;
      t.n2 = q - t.c2;
    }
  }
  t.ns = t.lo + t.n1 + t.n2 + t.hi;
  t.np = t.kv - t.ns;
  auto magic = [](int d) { return d > 1 ? static_cast<unsigned>((4294967296ULL + d - 1) / d) : 0u; };
  t.mp = magic(t.np);
  t.ms = magic(t.ns);
  t.bp = static_cast<unsigned>((static_cast<long long>(c.ny) * t.np + kTpThreads - 1) / kTpThreads);
  return t;
}

template <typename T>
TpArgs<T> tp_args(xfb_handle* h, TimeP tp) {
  constexpr int V = Vec<T>::V;
  const Compiled& c = h->c;
  TpArgs<T> a;
  const long long shift = h->sx + h->sy;
  for (int q = 0; q < 6; ++q) a.f[q] = reinterpret_cast<char*>(as<T>(field_ptr(h, h->live, q)) - shift);
  a.mid = h->mid - shift;
  a.nx = c.nx; a.ny = c.ny; a.nz = c.nz;
  a.sx = h->sx; a.sy = h->sy;
  a.sxb = static_cast<unsigned>(h->sx * sizeof(T));
  a.syb = static_cast<unsigned>(h->sy * sizeof(T));
  a.c = tp_columns<T>(c);
  a.pm = pml_params<T>(h);
  a.ps = psi_h_set<T>(h, h->live);
  a.tf = tfsf_params(h);
  a.tp = tp;
  a.ad = ade_params<T>(h);
  a.lut8 = as<const T>(h->lut8);
  a.zvec = c.pml[4] % V == 0 && c.pml[5] % V == 0 && c.nz % V == 0;
  for (unsigned& d : a.disp) d = 0;
  if (h->ade_deferred) {
    a.ad.kind = kAdeNone;
    for (size_t m = 0; m < c.mat_disp.size(); ++m)
      if (c.mat_disp[m]) a.disp[m >> 5] |= 1u << (m & 31);
  }
  a.ar = ade_params<T>(h);
  a.g = grid_params<T>(h, h->live);
  a.runs = static_cast<const int2*>(h->ade_runs);
  a.run_first = static_cast<const int*>(h->ade_planes);
  a.run_lo = h->ade_plane[0];
  a.run_hi = h->ade_plane[1];
  a.nblk = a.c.bp + (c.ny * a.c.ns + kTpThreads - 1) / kTpThreads;
  a.nade = (h->ade_plane_max + kTpThreads / 32 - 1) / (kTpThreads / 32);
  return a;
}

template <typename T>
void tp_update(xfb_handle* h, TimeP tp, cudaStream_t st, Prof* pf) {
  const Compiled& c = h->c;
  const TpArgs<T> a = tp_args<T>(h, tp);
  const dim3 grid(a.nblk, c.nx);
  prof_begin(h, pf, XFB_K_UPDATE_H);
  k_tp_h<T><<<grid, kTpThreads, 0, st>>>(a);
  prof_end(h, pf);
  prof_begin(h, pf, XFB_K_UPDATE_E);
  const bool runs = h->ade_deferred && h->n_ade_runs > 0;
  if (runs && tp_ade_inside(h)) {
    const long long row = static_cast<long long>(c.nx) * a.nblk + static_cast<long long>(a.run_hi - a.run_lo) * a.nade;
    k_tp_e<T, true><<<static_cast<unsigned>(row), kTpThreads, 0, st>>>(a);
  } else {
    k_tp_e<T, false><<<grid, kTpThreads, 0, st>>>(a);
    if (runs) k_tp_ade<T><<<(h->n_ade_runs + 3) / 4, 128, 0, st>>>(a, h->n_ade_runs);
  }
  prof_end(h, pf);
}

// The live set's fields and H-side psi into the set that holds step h->step on
// the one-sweep path (step & 1), which is live from then on.
template <typename T>
int tp_normalise(xfb_handle* h) {
  const int want = static_cast<int>(h->step & 1);
  if (!h->two_pass || h->live == want) return XFB_OK;
  cudaStream_t s = h->batch ? h->batch->stream : h->stream;
  for (int q = 0; q < 6; ++q) {
    XFB_CUDA(h, cudaMemcpyAsync(field_ptr(h, want, q), field_ptr(h, h->live, q), h->elems * sizeof(T),
                                cudaMemcpyDeviceToDevice, s));
    const size_t ax = q < 2 ? static_cast<size_t>(h->c.pml[0] + h->c.pml[1]) * h->sx
                    : q < 4 ? static_cast<size_t>(h->c.nx + 1) * h->ysx
                            : static_cast<size_t>(h->c.nx + 1) * h->zsx;
    void* const src = h->live ? h->psi_h1[q] : h->psi[6 + q];
    void* const dst = want ? h->psi_h1[q] : h->psi[6 + q];
    if (ax) XFB_CUDA(h, cudaMemcpyAsync(dst, src, ax * sizeof(T), cudaMemcpyDeviceToDevice, s));
  }
  XFB_CUDA(h, cudaStreamSynchronize(s));
  h->live = want;
  if (h->batch) {  // its step graphs name the set
    for (auto& kv : h->batch->graphs) cudaGraphExecDestroy(kv.second);
    h->batch->graphs.clear();
  }
  return XFB_OK;
}

}  // namespace xfb

#define XFB_INSTANTIATE_TWOPASS(T)                                                  \
  namespace xfb {                                                                   \
  template bool tp_plan<T>(const xfb_handle*);                                      \
  template void tp_update<T>(xfb_handle*, TimeP, cudaStream_t, Prof*);              \
  template int tp_normalise<T>(xfb_handle*);                                        \
  template bool tp_batch_plan<T>(const xfb_batch*);                                 \
  }
