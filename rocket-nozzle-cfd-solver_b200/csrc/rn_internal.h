// rn_internal.h -- the solver handle and helpers shared by the C-ABI sources
// (rn_api.cu, rn_batch.cu). Not part of the public interface.
#pragma once
#include <cuda_runtime.h>
#include <string>
#include <utility>
#include <vector>
#include "rn.h"
#include "rn_kernels.cuh"

// `steps` consecutive steps of a handle as a CUDA graph, and what they were
// captured with (rn_step replays them only while all of that still holds).
struct StepGraph {
  cudaGraphExec_t exec = nullptr;
  const void *K = nullptr, *base = nullptr, *xhead = nullptr;
  int tile = -1, maxX = -1, nHeavy = -1;
  int cur = -1, stepIdx = -1, wslot = -1, scur = -1;
  int steps = 0;
  long long launches = 0;
  unsigned long long used = 0;
  rn_params P = {};
};

// The state-ring slots of a step from slot cur: s1 takes the stage-1 state, s2
// the step's result. The ring turns forwards and backwards in turn with the
// step-info parity, so cur is back where it was, and the launches repeat,
// every two steps.
inline void ring_slots(int cur, int stepIdx, int& s1, int& s2) {
  const int d = stepIdx ? 2 : 1;
  s1 = (cur + d) % 3;
  s2 = (cur + 2 * d) % 3;
}

// One solver instance: all of its device memory and its stream. The layout in
// HBM is the reference's texture layout as plain arrays (see rn_api.cu).
struct rn_solver {
  int Nx = 0, Nr = 0, device = 0;
  cudaStream_t stream = nullptr;
  float4* SA[3] = {nullptr, nullptr, nullptr};
  float4* SB[3] = {nullptr, nullptr, nullptr};
  int cur = 0;
  float4 *geoA = nullptr, *geoG = nullptr, *geoM = nullptr, *jw = nullptr, *wallRow = nullptr;
  uint8_t* mask = nullptr;
  // the cells' classes (CellClass), rows padded to 16 bytes (a tensor map's row
  // stride must be a multiple of 16 bytes), rebuilt whenever the mask or the
  // geometry changes
  uint8_t* maskP = nullptr;
  int maskPitch = 0;
  // tensor maps of the stage kernels' halo copies, one TileMaps per tile shape
  rn::TileMaps* dMaps = nullptr;
  unsigned* errFlag = nullptr;    // set by a stage kernel whose halo copy did not complete in time
  float4* stepTex = nullptr;      // [2]
  unsigned* wmax = nullptr;       // [2]
  unsigned* depFlag = nullptr;    // set when a fast deposit left the fixed-point range
  unsigned* depBound = nullptr;   // [2 step parities] x (largest parcel mass, speed) of the ring, float bits
  unsigned long long* liveSteps = nullptr;   // live parcels summed over the spray steps since the ring was set
  int stepIdx = 0, wslot = 0;
  bool wvalid = false;
  long long stepCount = 0, launches = 0;
  // spray
  float4 *PA[2] = {nullptr, nullptr}, *PB[2] = {nullptr, nullptr}, *PC[2] = {nullptr, nullptr};
  float4 *src = nullptr, *tab = nullptr, *dep = nullptr;
  unsigned *key = nullptr, *val = nullptr, *keyS = nullptr, *valS = nullptr;
  void* sortTemp = nullptr;
  size_t sortTempBytes = 0;
  int scur = 0;
  uint32_t head = 0, seed = 1;
  // asynchronous read-back
  float* pinned = nullptr;
  size_t pinnedCap = 0, asyncFloats = 0;
  cudaEvent_t asyncEv = nullptr;
  unsigned long long* acc = nullptr;   // 2 x N x 4 fixed-point spray deposit sums (by step parity scur)
  float4* asyncDev = nullptr;      // device staging of the gathered rectangles
  size_t asyncDevCap = 0;          // float4 capacity of asyncDev
  cudaStream_t copyStream = nullptr;   // the staging buffer's copy to the host
  cudaEvent_t evGathered = nullptr;
  bool asyncBusy = false;
  int asyncTag = 0;
  double* dInt = nullptr;
  // per-kernel event timing: prof = 1 launch by launch, 2 inside replays of
  // the step graph (profCapture while that graph is captured; its event
  // pairs, read after every replay, in profGraphEv)
  int prof = 0;
  bool profCapture = false;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> profGraphEv;
  std::vector<cudaEvent_t> evPool;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> evPending;
  double profMs[RN_NKERNELS] = {0};
  long long profN[RN_NKERNELS] = {0};
  // tile shape of the stage/physics kernels and, per tile, the out-of-tile
  // members of its cut-cell groups (built from host copies of the topology)
  // (tile: the public name; shape: what its kernels run, TILE_TX/TILE_TY's index.
  // They differ only while autoShape, i.e. until a caller sets the tile shape, in
  // a batch whose shape nobody set, and from leaving one to the next step)
  int tile = RN_TILE_16x15, shape = RN_TILE_16x15;
  bool autoShape = true;
  rn::MemberHead* xhead = nullptr;
  int* xcell = nullptr;
  int maxX = 1;
  std::vector<int> hostXoff;
  // tiles listing more than XSMALL out-of-tile members (own fused launch)
  int* heavy = nullptr;
  int nHeavy = 0;
  int numSMs = 148;
  cudaStream_t side = nullptr;          // runs the heavy tiles' launch beside the main one
  cudaEvent_t evFork = nullptr, evJoin = nullptr;
  // whole runs of steps as CUDA graphs, the least recently used one replaced
  StepGraph graphs[2];
  unsigned long long graphClock = 0;
  int lastN = 0;             // the previous rn_step call's step count and parameters
  rn_params lastP = {};
  unsigned* dHS = nullptr;   // the spray ring's (head, seed) on the device, for graph-replayed spray steps
  bool hsOnDevice = false;   // step_once launches read and advance dHS (while capturing)
  cudaStream_t sprayStream = nullptr;   // runs the parcel step beside stage 2 + the split step
  cudaEvent_t evSprayFork = nullptr, evSprayJoin = nullptr;
  std::vector<uint8_t> hostMask;
  std::vector<float> hostGeoM;
  // kernels of the selected precision (rn_set_precision)
  const rn::KernelSet* K = &rn::kernels_fast;
  // residual snapshot (A plane + step info) and FP64 scratch (rn_readout.cu)
  float4* mark = nullptr;
  float4* markSt = nullptr;
  double* dRes = nullptr;
  // per-column wall slope, hypot(1, slope) and radius for rn_wall_separation
  double* wallProf = nullptr;
  // derived-field buffer (rn_derived) and the ring slot of the last step's
  // stage-1 state (-1 when no step has run since the state was set)
  float4* derived = nullptr;
  int s1last = -1;
  // the batch this handle is stepped by, if any (rn_batch.cu)
  struct rn_batch_t* batch = nullptr;

  rn::Grid grid() const { return rn::Grid{Nx, Nr, mask, geoA, geoG, geoM}; }
};

// (Re)encode the tensor maps of h's state ring and pitched mask (rn_api.cu).
int rn_build_tile_maps(rn_solver* h);
// Destroy h's step graphs (their launches name its buffers and lists).
void rn_drop_step_graphs(rn_solver* h);
// Rebuild h's cell classes from its mask and geometry (queued on h->stream).
int rn_classes_refresh(rn_solver* h);
// Record an error for rn_last_error() and return `code`.
int rn_record_error(int code, const std::string& msg);
int rn_record_cuda(cudaError_t e, const char* what);
// The shape a handle with an Nx x Nr grid runs when no caller set one.
int rn_auto_shape(int Nx, int Nr, int numSMs);
// Makes `shape` the one that h's kernels run and rebuilds its member lists.
int rn_use_shape(rn_solver* h, int shape);
// (Re)build the per-tile member lists of `h` for its current tile shape.
int rn_build_member_lists(rn_solver* h);
// Takes a new topology (solid mask, geoM) as h's host copy, chooses the shape
// for it and builds its member lists; on failure h keeps the one it had.
int rn_set_topology(rn_solver* h, std::vector<uint8_t> mask, std::vector<float> geoM);
// Make h->wmax[h->wslot] the wave-speed max of the current state if it is not.
int rn_ensure_wave_speed(rn_solver* h);
// Member lists of batch member h's new topology for the batch's shape; a batch
// whose shape nobody set goes back to 16x15 where they are too long for 16x16
// (rn_batch.cu).
int rn_batch_fit_member_lists(rn_solver* h);
// Takes h out of its batch, if any (rn_batch.cu).
void rn_batch_detach(rn_solver* h);
// Residual of the current state against the mark, into h->dRes[0..5], and the
// mark itself, queued on `stream` (rn_readout.cu); device bytes they hold.
int rn_residual_launch(rn_solver* h, cudaStream_t stream);
// One rectangle (x, y, w, h) of a W-wide float4 plane, gathered row by row to
// dst + off (rn_readout.cu). Up to RN_GATHER_RECTS per launch.
struct RectCopy {
  const float4* src;
  int W, x, y, w, h;
  long long off;
};
constexpr int RN_GATHER_RECTS = 8;
int rn_gather_rects(const RectCopy* r, int n, float4* dst, cudaStream_t stream);
int rn_residual_mark_on(rn_solver* h, cudaStream_t stream);
size_t rn_residual_bytes(int Nx, int Nr);

#define RN_CK(call)                                            \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return rn_record_cuda(e_, #call);   \
  } while (0)
