// Engine handle shared by the C-ABI (api.cu) and the per-precision engine
// translation units (engine_f32.cu, engine_f64.cu).
#pragma once

#include <cuda.h>  // CUtensorMap
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "xfb_internal.h"

namespace xfb {
struct Buf {
  void* p = nullptr;
  size_t bytes = 0;
  bool state = false;  // part of the checkpoint state
  bool owner = true;   // p is a cudaMalloc base (freed with the handle's device state)
  size_t block = 0;    // an owner's allocation size
};

// Pinned staging buffers of the read-backs, shared by the handles of the
// process: a read takes two and gives them back.  Two sizes: pinning costs 0.5 ms
// per MB, so a pair per handle of 16 MB (FP32) or 32 MB (FP64) buffers cost 17 and
// 35 ms per run, and once more 4 or 7 ms to unpin, while every chunk costs some
// 65 us beside its copy (75 us for 4 MB): wake-up, host threads, their last one.
// Handles whose fields are of kPinLarge bytes or more, whose runs hide the
// pinning, take the large ones.  Reads into faulted memory with 16 / 32 MB, with
// 4 and with 16 MB chunks (ms; 12 host threads): FP32 20 MB 1.2, 1.3, 1.2, 40 MB
// 1.6, 2.0, 1.9, 271 MB 7.4, 9.8, 7.7; FP64 40 MB 1.5, 1.9, 1.5, 160 MB 4.3, 6.2,
// 4.4, 512 MB 11.2, 18.1, 12.8.  Buffers are made when none is idle, so there are
// as many as reads ran at once; at most two per handle that reads back are kept
// idle, none once the last such handle is destroyed.  (With four kept in all, 4 and
// 8 threads reading a handle each pinned and unpinned buffers at every read: 1 MB
// fields 7 and 16 ms a round instead of 0.7 and 1, 52 MB 17 and 36 instead of 9 and
// 15.)
constexpr size_t kPinBytes[2] = {4u << 20, 16u << 20};
constexpr size_t kPinLarge = 32u << 20;
void pin_warm(int size);  // have two unused buffers, as far as they can be had
struct PinnedPair {
  int size;
  void* p[2];
  explicit PinnedPair(int size);
  ~PinnedPair();
  PinnedPair(const PinnedPair&) = delete;
  PinnedPair& operator=(const PinnedPair&) = delete;
  bool ok() const { return p[0] && p[1]; }
};

}  // namespace xfb

struct xfb_batch;
struct xfb_handle {
  using Buf = xfb::Buf;
  xfb::Compiled c;
  std::string err;
  // xfb_host_prefault: ranges (64 MiB parts) queued for a pool of host
  // threads (three quarters of the cores, at most 12) that fault them in;
  // every call that writes caller memory joins the pool first
  std::vector<std::thread> prefault;
  mutable long long n_disp_cells = -1;  // cells of dispersive materials (grid info), once counted
  std::vector<std::pair<char*, char*>> pf_queue;
  std::mutex pf_mu;
  int pf_active = 0;
  int device = -1;
  cudaStream_t stream = nullptr;
  bool inited = false;
  long long step = 0;
  unsigned hint_grid[3] = {1, 1, 1}, hint_block[3] = {1, 1, 1};
  int tk = 32, tj = 16;
  int path = XFB_PATH_AUTO;  // resolved at init: XFB_PATH_SPLIT or XFB_PATH_FUSED
  bool path_auto = true;     // the path was left to the library
  // two-pass 3-D step (twopass.cuh): steps in place on field set `live` (0 or
  // 1) instead of alternating between the sets; the automatic path only
  bool two_pass = false;
  int live = 0;
  int graph_on = 1, graph_steps = 64;
  int coeff_storage = XFB_COEFF_NATIVE;  // rounding of the update-coefficient LUT (xfb_set_coeff_storage)
  // 2-D temporal blocking (k_step2_tb): steps per launch (odd; 0: one launch
  // per step), whether init enabled it, its plan, and the second set of the E-side psi (ez_x, ez_y) it alternates with psi[1], psi[2]
  int tb_steps = 9;
  bool tb_given = false;  // tb_steps set by the caller, else the plan chooses
  bool tb_on = false;
  int tb_warps = 0, tb_max = 0;  // the plan: warps of a CTA, steps of a launch at most
  void* psi_e1[2] = {};
  std::map<int, cudaGraphExec_t> graphs;
  std::vector<Buf> bufs;
  size_t bytes = 0;
  // device buffers up to kArenaMax bytes are carved from chunks of one
  // cudaMalloc each (fewer driver calls at init): the free part of the last chunk
  char* arena = nullptr;
  size_t arena_left = 0;
  int esize = 4;
  // field layout
  long long sx = 0, sy = 0, nzp = 0, elems = 0, guard = 0;
  void* f[6] = {};    // field set 0
  void* f1[6] = {};   // field set 1 (one-sweep path: step t reads set t&1, writes the other)
  uint8_t* mid = nullptr;
  void* lut8 = nullptr;       // [n_mat][8] compact coefficients (one-sweep path)
  uint8_t* mat_disp = nullptr;
  void* lut = nullptr;
  // CPML
  void* prof[12] = {};  // ae0 ae1 ae2 be0 be1 be2 ah0 ah1 ah2 bh0 bh1 bh2
  void* psi[12] = {};   // ey_x ez_x ez_y ex_y ex_z ey_z hy_x hz_x hz_y hx_y hx_z hy_z
  void* psi_h1[6] = {}; // H-side psi of field set 1 (one-sweep path)
  long long ysx = 0, zsx = 0, zsy = 0;
  // TFSF
  double* proj[6] = {};
  double* e_aux = nullptr;   // [total_steps + 1][nl + 1] incident E of every step
  double* h_aux = nullptr;   // [total_steps][nl] incident H of every half step
  double* src = nullptr;
  // ADE
  void* ade_mat = nullptr;
  void* ade_pole = nullptr;
  void* J = nullptr;
  void* Jp = nullptr;
  void* Ep = nullptr;
  long long bsx = 0, bsy = 0, bn = 0;
  // NF2FF
  double2* nf_acc = nullptr;
  double* nf_ring = nullptr;     // [kNfRing][4][npts] surface samples not yet accumulated
  long long* nf_done = nullptr;  // steps accumulated by the last flush
  double2* te = nullptr;
  double2* th = nullptr;
  int nf_off[7] = {};
  long long nf_npts = 0;
  // time-domain NF2FF (k_records / k_nftd_bins)
  void* td_ent = nullptr;     // int4 per point
  double* td_tsd = nullptr;   // delay in steps per point
  double* td_prev = nullptr;  // [2][td_n]
  long long td_n = 0;
  void* td_chunk = nullptr;   // int4 per chunk
  int td_nchunks = 0;
  double* td_part = nullptr;  // [td_nchunks][6]
  int* td_offs = nullptr;
  int* td_list = nullptr;
  double* td_pot = nullptr;   // [6][td_bins]
  // monitors
  long long* probe_idx = nullptr;
  int* probe_field = nullptr;
  double* probe_out = nullptr;
  void* probe_link = nullptr;  // int2 per probe: scratch of the blocked 2-D kernel
  std::vector<double*> movie_out;
  std::vector<long long> movie_frames;
  long long* t_dev = nullptr;
  unsigned long long* scratch_u64 = nullptr;
  void* plain_c[18] = {};  // per-cell coefficient arrays of the plain path
  // one-sweep step work items per tile configuration
  // (int4: k tile | region kind << 16, j tile, first plane, end plane)
  void* step_items[2] = {};
  int n_step_items[2] = {};
  // staging tensor maps of the one-sweep kernel per tile configuration and
  // read set (six field components, then the material ids), the bulk-store
  // maps of its lean interior items per tile configuration and write set
  // (Ex Ey Ez Hx Hy Hz), and its error flag (1: a staging wait ran out)
  CUtensorMap stage_maps[3][2][7];
  CUtensorMap store_maps[3][2][6];
  int* step_err = nullptr;
  // TFSF line tables of the one-sweep step, filled every step by
  // k_tfsf_lines (or, in a batch, k_tfsf_lines_batch; yh, ye: rows of pitch
  // line_ykp; zh, ze: rows of pitch line_zjp), and their tensor maps per tile
  // configuration.  Off without a TFSF source.
  bool lines_on = false;
  void* line_tab[4] = {};
  long long line_ykp = 0, line_zjp = 0;
  CUtensorMap line_maps[3][4];
  // ADE applied by k_ade_box after the one-sweep step (no dispersive cell
  // takes a TFSF or CPML correction)
  bool ade_deferred = false;
  // its work list: runs of dispersive cells (k_ade_runs); -1: no list (k_ade_box)
  void* ade_runs = nullptr;
  int n_ade_runs = -1;
  // the two-pass step's view of it: the first run of every plane (int[nx + 1]),
  // the planes that have runs, and the most runs of one plane
  void* ade_planes = nullptr;
  int ade_plane[2] = {}, ade_plane_max = 0;
  // set while a batch steps this handle (xfb_batch_*)
  xfb_batch* batch = nullptr;
  // learned absorbing boundary (xfb_set_learned_abc): BF16 weights and the
  // E(w, n-1), E(w+s, n-1) history planes of every wall
  bool labc_on = false;
  void* labc_w = nullptr;
  float* labc_hist = nullptr;
  // field read-back (read_field_t): a device gather buffer of the handle's pinned buffers' size and
  // the events that mark each pinned buffer's chunk as copied (chunk c lands in
  // buffer c & 1 while the host widens chunk c - 1 to double); pin_user: the
  // handle counts among the staging pool's users
  void* rb_dev = nullptr;
  cudaEvent_t rb_ev[2] = {};
  bool pin_user = false;
  // cudaMalloc blocks of the previous init, offered to the next one
  std::vector<Buf> spare;
  // bytes this handle has copied host -> device and device -> host
  long long h2d_bytes = 0, d2h_bytes = 0;
  // x-slab decomposition (xfb_set_slab): the handle updates cells
  // [slab_i0, slab_i1) along x of the full grid; planes slab_i0 - 1 and
  // slab_i1 are halos, refilled between xfb_slab_update and xfb_slab_record
  // (xfb_slab_exchange, or the host's own collective); -1: the whole grid
  int slab_i0 = 0, slab_i1 = -1;
  bool slab_pending = false;  // an update awaits its record
};

// A batch of scenes stepped together: one launch of the one-sweep kernel per
// step over the work items of every scene, or one persistent launch for a
// chunk of steps (k_step3_persist).  The handles stay owned by the caller;
// the batch owns only its tables, stream, counters and graphs.
constexpr int kBatchChains = 16;  // parallel chains of a batch's two-pass step, at most
// Steps of one graph of a batch's two-pass step: at most kBatchGraphLaunches
// kernels, or one step's where that has more.  (Longer graphs save nothing, and the
// device waits for the first one's capture: 64 scenes, the first 30 steps, 16 at a
// time and all in one graph 8.0 and 8.7 ms per step.)
constexpr long long kBatchGraphLaunches = 2048;
inline int batch_graph_steps(int graph_steps, long long launches_of_a_step) {
  return static_cast<int>(std::max(1LL, std::min<long long>(graph_steps, kBatchGraphLaunches / std::max(1LL, launches_of_a_step))));
}

struct xfb_batch {
  std::vector<xfb_handle*> hs;
  std::string err;
  int device = 0;
  int prec = XFB_FP32;
  cudaStream_t stream = nullptr;
  bool inited = false;
  long long step = 0, total = 0, cells = 0;
  int tile_req = 0;   // 0: autotune, else 8, 14 or 16 rows
  int tile = -1;      // tile configuration in use (-1 until chosen)
  int graph_steps = 64;
  void* scenes = nullptr;   // BatchScene<T>[n]
  void* maps = nullptr;     // BatchMaps[n]: tensor maps of every scene
  int* err_dev = nullptr;   // 1: a staging wait of the step kernel ran out
  void* items[3] = {};      // per tile configuration
  int n_items[3] = {};
  long long* t_dev = nullptr;
  std::map<int, cudaGraphExec_t> graphs;
  // persistent launches (XFB_BATCH_PERSISTENT): work lists (the per-step
  // lists, aliased), items per scene, and the queue (ticket counter, then one
  // finished-item counter per scene)
  int launch_req = XFB_BATCH_AUTO;  // xfb_batch_set_launch
  int launch = -1;                  // XFB_BATCH_PER_STEP or XFB_BATCH_PERSISTENT (-1 until chosen)
  bool persist_ok = false;          // no scene records monitors or runs a separate ADE pass
  void* pitems[3] = {};
  void* pscene_items[3] = {};
  unsigned* queue = nullptr;
  long long lines_work = 0;  // TFSF line entries of the largest scene (0: no scene has a TFSF source)
  // two-pass step of every scene (batch_chains): a captured stream per chain
  // of scenes, the fork and the chains' join events
  bool two_pass = false;
  std::vector<cudaStream_t> chains;
  std::vector<cudaEvent_t> chain_ev;
};

namespace xfb {

// ---- helpers (api.cu) ----------------------------------------------------
int set_err(xfb_handle* h, int code, const std::string& m);
int cuda_err(xfb_handle* h, cudaError_t e, const char* what);

#define XFB_CUDA(h, call)                                   \
  do {                                                      \
    cudaError_t e_ = (call);                                \
    if (e_ != cudaSuccess) return cuda_err((h), e_, #call); \
  } while (0)

template <typename T>
T* as(void* p) { return static_cast<T*>(p); }

void free_device(xfb_handle* h);
void keep_blocks(xfb_handle* h);
void pin_use(xfb_handle* h);  // count the handle among the staging pool's users
inline int pin_size(const xfb_handle* h) {
  return static_cast<size_t>(h->elems) * h->esize >= kPinLarge ? 1 : 0;
}
void free_spare(xfb_handle* h);
int alloc(xfb_handle* h, void** out, size_t bytes, bool state);
// n zeroed buffers of `bytes` each (256-byte aligned) from one cudaMalloc.
int alloc_block(xfb_handle* h, void** out, int n, size_t bytes, bool state);
// Every host<->device copy of the library goes through this: it is issued on
// the handle's stream (a non-blocking stream, which the legacy default stream
// does not order against) and waited for, so it lands after the zero-fill of
// alloc() and after every kernel already queued, and the host buffer may be
// released on return.
int copy(xfb_handle* h, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind);

template <typename T>
int upload(xfb_handle* h, void** out, const std::vector<double>& v, bool state = false) {
  std::vector<T> tmp(v.begin(), v.end());
  int rc = alloc(h, out, tmp.size() * sizeof(T), state);
  if (rc) return rc;
  if (!tmp.empty()) return copy(h, *out, tmp.data(), tmp.size() * sizeof(T), cudaMemcpyHostToDevice);
  return XFB_OK;
}

long long roundup(long long v, long long m);
bool fused(const xfb_handle* h);
// tile configuration of the one-sweep kernel picked by the launch hint's rows
inline int step_tile_index(int tj) { return tj <= 8 ? 0 : 1; }
// tile rows of the one-sweep kernel's configurations; single scenes use the
// first two, a batch autotunes over all three
constexpr int kStepTileCount = 3;
constexpr int kStepTileRows[kStepTileCount] = {8, 16, 14};
bool plain(const xfb_handle* h);
inline bool is_slab(const xfb_handle* h) { return h->slab_i1 >= 0; }
// planes i whose cells and monitors this handle owns (the last slab also owns
// the node plane i = nx of the E components)
inline int own_lo(const xfb_handle* h) { return is_slab(h) ? h->slab_i0 : 0; }
inline int own_hi(const xfb_handle* h) {
  return is_slab(h) && h->slab_i1 < h->c.nx ? h->slab_i1 : h->c.nx + 1;
}
int cur_set(const xfb_handle* h);
// field set the step that reads set `parity` leaves its result in
inline int out_set(const xfb_handle* h, int parity) { return h->two_pass ? h->live : fused(h) ? 1 - parity : 0; }
void* field_ptr(const xfb_handle* h, int set, int q);
long long off3(const xfb_handle* h, int i, int j, int k);
void comp_shape(const Compiled& c, int f, int s[3]);
int nf_face_points(const Compiled& c, int face);
int launches_per_step(const xfb_handle* h);
int check_handle(xfb_handle* h, bool need_init);

// ---- engine (engine.cuh, instantiated for float and double) -------------
template <typename T> int init_device(xfb_handle* h);
template <typename T> int run_steps(xfb_handle* h, long long n);
template <typename T> int slab_update(xfb_handle* h);
template <typename T> int slab_record(xfb_handle* h);
template <typename T> int profile_steps(xfb_handle* h, long long n, double* ms, long long* launches);
template <typename T> int read_field_t(xfb_handle* h, int f, double* dst);
template <typename T> int read_bytes_t(xfb_handle* h, void* dst, const void* src, size_t bytes);
template <typename T> int write_field_t(xfb_handle* h, int f, const double* src);
template <typename T> void launch_nonfinite(xfb_handle* h);
// two-pass 3-D step (twopass_f32.cu, twopass_f64.cu)
// Whether the two-pass step's E pass takes the dispersive cells in blocks of
// its own instead of leaving them to k_tp_ade: up to kTpAdePoles poles (more
// spill in its registers), and fields of at most 600 MB: where the 126 MB L2
// holds a good part of them the overlap pays.  us per step apart and inside:
// 128x152x136 Debye FP64 (153 MB) 105 and 97; Drude-Lorentz FP32 284^3 (600 MB)
// 520 and 515, 408^3 (1.7 GB) 1188 and 1204, where DRAM serves one access
// pattern better than two at once.
constexpr int kTpAdePoles = 2;
inline bool tp_ade_inside(const xfb_handle* h) {
  return h->c.ade_poles <= kTpAdePoles && 6.0 * h->elems * h->esize <= 600e6;
}
template <typename T> bool tp_plan(const xfb_handle* h);
template <typename T> int tp_normalise(xfb_handle* h);
template <typename T> bool tp_batch_plan(const xfb_batch* b);
// Back to the one-sweep kernels from the current state (monitor reads, state
// and results are unaffected).
int tp_leave(xfb_handle* h);
template <typename T> int batch_init(xfb_batch* b);
template <typename T> int batch_run(xfb_batch* b, long long n);
void batch_free(xfb_batch* b);
int batch_err(xfb_batch* b, int code, const std::string& m);

}  // namespace xfb
