// lbx_internal.h -- the domain handle's layout, shared by the library's
// translation units (not part of the ABI).
#pragma once

#include "lbx.h"

#include <cuda_runtime.h>

#include <vector>

// A division of a small 2D lattice into tiles for one part of the GPU (level
// l: at most one of its 2^l equal parts), and its tables on the device.
struct TiledPlan {
  static constexpr int kLevels = 5;
  int state = 0;                         // 0: not planned, 1: planned, -1: no tiles fit
  double us = 0.0;                       // modelled time per step (0: not looked for)
  int K = 0;                             // steps per round, at most
  int ntiles = 0;
  size_t nodes = 0;                      // region nodes of all tiles
  int base = 0;                          // counter value the next launch starts from
  void* own = nullptr;                   // its memory, where it has its own
  void* tiles = nullptr;
  int* nbrs = nullptr;                   // per tile: the tiles its halo reads
  int* flags = nullptr;                  // per-tile round counters
  int* gidx = nullptr;                   // per tile: population slots of its region's nodes
  unsigned short* list = nullptr;        // per tile: its node list; then the flags words, the halo list
};

struct lbx_domain {
  lbx_params p;
  int Q = 0, D = 0;
  long long N = 0;
  size_t real_size = 0;
  void* f = nullptr;          // [nsubs][Q][N] dense (the exchange format)
  void* fc = nullptr;         // [nsubs][Q][P] compact layout
  int* fidx = nullptr;        // [N] dense -> compact (-1 solid)
  int* fnode = nullptr;       // [F] compact -> dense
  uint2* frm = nullptr;       // [ceil(N/32) + 2] fluid bitmask with word ranks, guard word each end
  long long P = 0;            // compact plane stride: fluid rounded up to 32
  int layout = LBX_LAYOUT_DENSE;
  bool dense_stale = false;   // compact state newer than the dense array
  void* mv = nullptr;         // [nsubs][1+D][N]
  uint8_t* solids = nullptr;  // [N] as given (device rule: == 1)
  uint8_t* cls = nullptr;     // [N]
  uint32_t* nbm = nullptr;    // [N]
  void* red = nullptr;        // reduction partials
  int red_blocks = 0;
  cudaStream_t stream = nullptr;      // stream all work is queued on
  cudaStream_t own_stream = nullptr;  // the library's stream
  // with z faces in the compact layout: the face planes' launch runs on
  // `side` beside the interior launches, forked from and joined back into
  // `stream` by the two events
  cudaStream_t side = nullptr;
  cudaEvent_t side_fork = nullptr, side_join = nullptr;
  std::vector<double> n_table, s_table;
  long long fluid = 0;
  bool faces_active = false;  // any 2D face boundary configured
  bool faces_fused = false;   // fused into the step kernels
  bool faces3_active = false; // any 3D z-face boundary configured
  bool faces3_fuse_odd = false;  // z faces exact inside odd compact steps (fluid upstream)
  std::vector<long long> plane_fluid;  // fluid nodes per plane (k in 3D, j in 2D)
  void* ubuf = nullptr;        // [3][P or N] flow velocity for the solute launch
  void* prof_t = nullptr;      // [LX*LY] constant-concentration profiles (real)
  void* prof_b = nullptr;
  void* ns = nullptr;        // Walsh fraction per node, [N] in the run's precision
  // plane record (lbx_btc_*)
  double* btc_vals = nullptr;  // [2][plane nodes]: C and u_x this step
  double* btc_rec = nullptr;   // [btc_cap][2] means
  int* btc_slot = nullptr;     // steps recorded
  double* btc_part = nullptr;  // [kBtcMaxBlocks][2] block partials of one step
  unsigned* btc_ticket = nullptr;  // blocks done this step (reset by the last)
  int btc_cap = 0;
  int btc_lo = 0, btc_hi = 0;  // node (dense) or slot (compact) range
  int btc_plane = 0;
  void* fout = nullptr;        // set only while recomputing states (OOP step)
  void* adj = nullptr;         // adjoint checkpoints and objective (lbx_adjoint.cu)
  void* frames = nullptr;      // frame statistics and snapshots (lbx_frames.cu)
  void* pest = nullptr;        // PEST point samples (lbx_pest.cu)
  int parity = 0;             // 0: natural order (next step odd); 1: swapped
  long long launches = 0;
  // graph replay of frame-free, time-invariant runs: one captured AA pair
  cudaGraphExec_t graph = nullptr;
  cudaGraphExec_t graph_multi = nullptr;   // the same pair repeated (replay_pairs)
  cudaStream_t graph_stream = nullptr;   // stream the pair was captured on
  unsigned char graph_key[2 * 640];      // keys of the odd and the even step
  size_t graph_key_len = 0;
  long long graph_launches = 0;          // kernels one replay of the graph runs
  // the last stretch launched directly, and the pairs so far with its arguments
  cudaStream_t direct_stream = nullptr;
  unsigned char direct_key[2 * 640];
  size_t direct_key_len = 0;
  long long direct_pairs = 0;
  // temporal blocking of small 2D lattices (lbx_tiled.cu)
  int run_mode = LBX_RUN_AUTO;
  std::vector<uint8_t> host_solids;      // 2D lattices the tiles may fit: the mask, for the plan
  TiledPlan tiled[TiledPlan::kLevels];
  void* tiled_room = nullptr;            // memory for what follows, behind the population array
  void* tiled_own = nullptr;             // or allocated when first needed
  void* tiled_scratch = nullptr;         // a second population array for its rounds
  int* tiled_status = nullptr;           // set by a launch whose wait ran out
  void* tiled_tables = nullptr;          // room for the first plan's tables
  int tiled_level = 0;                   // the plan of the next launch, -1: a launch per step
  bool tiled_record = false;             // the stretch's launches are to be seen by other domains'
  // its last launch, for other domains' (guarded by the mutex in lbx_tiled.cu,
  // but for the event itself)
  cudaEvent_t tiled_done = nullptr;
  cudaStream_t tiled_stream = nullptr;
  unsigned long long tiled_turn = 0;
  bool tiled_listed = false, tiled_busy = false;
  int tiled_company = 0;                 // others' runs seen beside it
  bool tiled_attr = false;               // the kernel's shared-memory limit is raised
};

namespace lbx { template <typename T> struct StepArgs; }

// Hidden helpers of the library's translation units (not exported).
#define LBX_HIDDEN __attribute__((visibility("hidden")))
LBX_HIDDEN lbx_status lbx_internal_fail(lbx_status code, const char* msg);
LBX_HIDDEN lbx_status lbx_internal_step_into(lbx_domain* d, int t, void* src, void* dst);
LBX_HIDDEN void lbx_internal_adjoint_free(lbx_domain* d);
LBX_HIDDEN void lbx_internal_frames_free(lbx_domain* d);
LBX_HIDDEN void lbx_internal_drop_graphs(lbx_domain* d);
// Copies between device memory and the caller's host buffers, ordered after
// the stream's earlier work (lbx_copy.cu): staged through page-locked chunks
// and waited for where that is faster, else queued on the stream.  Each
// domain and batch registers as a user (copy_user, add = 1, -1) of its
// device's chunks.
LBX_HIDDEN cudaError_t lbx_internal_copy_out(int device, cudaStream_t stream, void* dst,
                                             const void* src, size_t bytes);
LBX_HIDDEN cudaError_t lbx_internal_copy_in(int device, cudaStream_t stream, void* dst,
                                            const void* src, size_t bytes);
// Planes that lie behind one another at src to dst[c] each (NULL: left out).
// Planes that lie so on the host too are one copy where their memory is
// pageable: a copy must not reach from page-locked memory into other.
LBX_HIDDEN cudaError_t lbx_internal_copy_planes_out(int device, cudaStream_t stream,
                                                    void* const* dst, int count, const void* src,
                                                    size_t plane);
LBX_HIDDEN void lbx_internal_copy_user(int device, int add);
// PEST sampling: whether a sample is due at time t (the step then writes
// the macro variables), the gather after that step, and the release.
LBX_HIDDEN bool lbx_internal_pest_due(const lbx_domain* d, int t);
LBX_HIDDEN lbx_status lbx_internal_pest_after(lbx_domain* d, int t);
LBX_HIDDEN void lbx_internal_pest_free(lbx_domain* d);
// Temporal blocking.  At creation: bytes the tiled run of this lattice would
// like behind the population array (0: it would not be taken).  Then whether
// the domain's run mode takes it for the stretch to be launched, the tiles
// planned on first use; then `pairs` AA pairs (two or more) with the launch
// arguments A from the state after an even step, the last step writing the
// macro variables if asked; and after the stretch's launches, tiled or not,
// tiled_launched.
LBX_HIDDEN size_t lbx_internal_tiled_room(lbx_domain* d);
// Whether the caller is capturing `stream` into a graph of its own.
LBX_HIDDEN bool lbx_internal_capturing(cudaStream_t stream);
LBX_HIDDEN lbx_status lbx_internal_tiled_plan(lbx_domain* d, bool* yes);
template <typename T>
LBX_HIDDEN lbx_status lbx_internal_tiled_run(lbx_domain* d, const lbx::StepArgs<T>& A, int pairs,
                                             bool write_mv);
LBX_HIDDEN void lbx_internal_tiled_launched(lbx_domain* d);
LBX_HIDDEN void lbx_internal_tiled_free(lbx_domain* d);
// LBX_OK, or the error of a tiled launch whose bounded wait ran out (then
// cleared); synchronous.
LBX_HIDDEN lbx_status lbx_internal_tiled_status(lbx_domain* d);
