// Host-side state of a solver handle, shared by the C-ABI files (api.cu, batch.cu).
#pragma once
#include <string>
#include <vector>

#include "ausm.h"
#include "ausm_internal.h"

struct ausm_solver {
  int M = 0, N = 0, dev = 0;
  int engine = AUSM_ENGINE_FUSED;
  AusmParams p{};
  double speed_now = 0.0;  // current inflow speed (ramped when p.ramp > 0)
  ausm::Consts c{};
  ausm::ex::ConstsR<double> cd{};  // the same constants in FP64 (F64 engine)
  ausm::F64Engine* f64 = nullptr;  // buffers of the F64 engine, once selected
  cudaStream_t st = nullptr;      // the stream calls run on (the batch's while a member)
  cudaStream_t own_st = nullptr;  // the handle's own stream
  ausm_batch* batch = nullptr;    // batch this solver belongs to, if any
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  std::vector<double> body, outer;  // M x 2
  bool has_body = false, has_outer = false, has_grid = false, has_state = false;
  double stretch = 0.0;
  char* block = nullptr;  // the device memory of the arrays from V to Q and of wave, dt, parts, move and err_flag:
                          // a new mapping and its release cost 0.6 ms each
  float2* V = nullptr;    // vertices, FP32 (reference layout, API, reference engine)
  double2* Vd = nullptr;  // vertices, FP64 (multicolor generator, metrics, forces)
  float4* Mi = nullptr;   // FP64-computed face records, i-faces [N][M]
  float4* Mj = nullptr;   // ... j-faces [N+1][M]
  float4* Q[3] = {nullptr, nullptr, nullptr};
  int cur = 0;
  float4* S[3] = {nullptr, nullptr, nullptr};
  float4 *fx = nullptr, *fy = nullptr, *res = nullptr, *flen = nullptr;
  float* area = nullptr;
  float4* staging = nullptr;
  double* cp = nullptr;
  uint32_t* wave = nullptr;    // [0] max wave speed bits; [1..2] the resident kernel's (kernels_resident.cu); [3] the
                               // finished blocks of a reduction (sum_parts_last)
  float* dt = nullptr;
  double* parts = nullptr;  // 2 * kMaxParts per-block partial sums
  uint32_t* move = nullptr;
  int* err_flag = nullptr;  // set by a kernel whose bounded wait gave up
  bool err_read_queued = false;  // a copy of *err_flag to h_wave[2] is queued on st (api.cu)
  ausm::TmaMaps tma[3];  // per tile height kTileHeights[k]
  bool counted = false;   // a user of the device's exchange buffers (resident_user)
  int tile_rows = 0;      // tile height of the TMA stage kernel; 0 until tuned
  float* h_dt = nullptr;
  uint32_t* h_wave = nullptr;
  double* h_acc = nullptr;  // pinned; sums of forces and norms, written by the kernels
  std::string err;
};

namespace ausm {
// Reference-order f32 uniforms of h's parameters and current inflow speed (api.cu).
void make_consts(ausm_solver* h);
// Inflow speed update of a ramped start after n steps (main.js:779), api.cu.
void ramp_after_steps(ausm_solver* h, int n);
void set_thread_error(const std::string& msg);
// Tile height for h's fused steps: AUSM_TILE_ROWS, the process-wide tuning cache for
// (M, N, scheme), or a tuning run (api.cu).  Enqueues work on h's stream; must not run
// inside a stream capture.
// The tile height AUSM_TILE_ROWS fixes for the stage kernels (8, 16 or 32), or 0.  A fixed
// height also keeps small grids on the stage kernels.
int forced_tile_rows();
// may_measure false: 16 rows where a tuning run would be needed.
int tuned_tile_rows(ausm_solver* h, bool force, bool may_measure, int* rows);
inline int tile_index(int rows) { return rows == 8 ? 0 : (rows == 32 ? 2 : 1); }
}  // namespace ausm
