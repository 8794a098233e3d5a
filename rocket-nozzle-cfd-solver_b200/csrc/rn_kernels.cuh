// rn_kernels.cuh -- kernel argument blocks and the kernel sets shared by the
// step kernels (rn_step.cu), the spray kernels (rn_spray.cu) and the C-ABI
// (rn_api.cu, rn_batch.cu).
#pragma once
#include <cuda_runtime.h>
#include "rn_math.cuh"
#include "rn_tma.cuh"

namespace rn {

// Tile shapes of the stage/physics blocks: TX x TY cells on TILE_NT threads,
// a thread per cell (threads beyond TX*TY idle in the cell phases). 16x15 on
// 256 threads (the default) has 511 faces, so its face phase is exactly two
// passes of the block, where 16x16's 544 faces need a third pass for one warp
// while the other seven wait at the barrier. Measured on B200 (fast
// precision, G cell-updates/s, 16x16 / 16x8 / 16x15 / 32x15): viscous
// 512x192 2.43 / 2.31 / 2.47 / 2.26, viscous 1024x384 3.67 / 3.26 / 4.00 /
// 3.99, plain 4096x1536 5.51 / 5.49 / 5.73 / 5.51, 64 batched instances
// 3.59 / 3.07 / 4.05 / 3.98. (16x16 itself beat 32x8 by 4.5-17 %.) The
// autotuner picks per handle or batch.
// 14x16 spreads a 512x192 grid over 37 x 12 = 444 tiles, 3 per SM on 148 SMs,
// and is compiled for those 3 blocks (24 warps: 80 registers, no spills); the
// others for 32 resident warps (64 registers).
// The last shape has no public name: a handle whose tile shape nobody set runs
// it on small grids (auto_shape). 10x10 cells on 256 threads fill each phase in
// one pass (196 primitives, 220 faces, 100 updates beside 144 vcell slots),
// where 14x16 takes two: with one or two blocks an SM a block's latency is the
// kernel's time.
constexpr int NTILES = 5, NSHAPES = 6;   // public shapes (RN_TILE_*), all compiled shapes
constexpr int TILE_TX[NSHAPES] = {16, 16, 16, 32, 14, 10};
constexpr int TILE_TY[NSHAPES] = {16, 8, 15, 15, 16, 10};
constexpr int TILE_NT[NSHAPES] = {256, 128, 256, 512, 256, 256};
constexpr int TILE_WARPS[NSHAPES] = {32, 32, 32, 32, 24, 24};
constexpr int SHAPE_SMALL = 5;
inline int tile_count(int shape, int Nx, int Nr) {
  return ((Nx + TILE_TX[shape] - 1) / TILE_TX[shape]) * ((Nr + TILE_TY[shape] - 1) / TILE_TY[shape]);
}
// 16x16 in place of 16x15. A 16x16 tile costs 1.1 to 1.2 of a 16x15 one for 7 %
// more cells (its 272 faces a direction take two passes of 256 threads), so it
// has to save tiles or waves of resident blocks (4 an SM, 592 on 148 SMs):
//   a wave of at most three. us per step, 16x15 / 16x16: viscous 640x224 (600 /
//     560 tiles) 29.8 / 27.8, plain 22.9 / 20.6; presets of 1024x287 (1280 / 1152)
//     47.6 / 45.5; 24 batched 128x48 (768 / 576) 48.2 / 38.0. At worst viscous
//     1184x256 (1332 / 1184) 48.5 / 49.3. Of four: viscous 1400x320 (1936 / 1760)
//     65.5 / 65.9, plain 50.1 / 50.9.
//   a seventh of the tiles, beyond one wave: 64 batched 128x48 (2048 / 1536) 98.8 /
//     88.5, 32 of 256x96 (3584 / 3072) 161 / 154, 32 of 203x77 (2496 / 2080) 116 /
//     110. With less to save: viscous 640x288 (800 / 720) 33.3 / 36.3, 2048x512
//     (4480 / 4096) 145 / 148, 24 batched mixed grids (13344 / 12240) 535 / 592;
//     in one wave: viscous 512x256 (576 / 512) 25.4 / 27.4, 4 batched 128x48 (128 /
//     96) 24.1 / 25.7.
inline bool prefer_16x16(long long tiles16x16, long long tiles16x15, int numSMs) {
  const long long resident = 4LL * numSMs;
  const long long waves16 = (tiles16x16 + resident - 1) / resident, waves15 = (tiles16x15 + resident - 1) / resident;
  return (waves16 < waves15 && waves15 <= 3) || (waves15 > 1 && 7 * tiles16x16 <= 6 * tiles16x15);
}
// A cell's class byte, in the row-pitched plane that the step kernels copy with
// the halo (0 outside the grid). Almost all cells are uncut (99 % of the plume
// and engine grids): their geometry is that of the grid, so the kernels form it
// from the row instead of reading geoA, geoG and geoM (49 of the 113 bytes a
// cell that stage 1 needs otherwise).
enum CellClass : unsigned char {
  CELL_SOLID = 1,
  CELL_PLAIN = 2,     // fluid, its own group alone, geoG = (j + 1/2, 1, 0, 0): no wall, whole cell
  CELL_NO_BAND = 4,   // not in the boundary-layer band (geoM.z bit 16)
  CELL_L0 = 8,        // turbulence length TURB_L0
  CELL_FACES = 16,    // west and south face fully open: areas j + 1/2 and j, second order
  CELL_BOX = 32       // all four faces of the size of the grid's, whatever their sign
};
constexpr float TURB_L0 = 0.17f;
// Most out-of-tile group members one tile may list (set_geometry rejects more).
constexpr int MAXX = 64;
// Tiles listing more out-of-tile members than this run the fused stage-2 +
// split-step kernel in a launch of their own, sized for them, so that the
// shared memory of every other block stays within 4 blocks per SM (a 1024x384
// bell has a wall tile with 16; it cost the whole launch a quarter of its
// occupancy).
constexpr int XSMALL = 4;
// The split (a side-stream launch joined back) pays only on grids of many
// waves: more tiles than SPLIT_BLOCKS_PER_SM x SMs. Measured with 16x16 tiles:
// 64 batched instances (36,400 blocks) 3.59 -> 3.97 G cell-updates/s; a lone
// 1024x384 grid (1,536 blocks) 3.67 -> 3.60, so it is not split.
constexpr int SPLIT_BLOCKS_PER_SM = 16;

// A tile's out-of-tile group members: how many, the first of them (most tiles
// have fewer), and where the others are in the handle's cell list. One aligned
// record, so that a block has its list after one round of loads.
constexpr int HEAD_CELLS = 6;
struct alignas(32) MemberHead {
  int first, count;
  int cell[HEAD_CELLS];
};

struct StageArgs {
  Grid g;
  const float4* A;  const float4* B;    // stage input state
  const float4* A0; const float4* B0;   // state at t^n (stage 2)
  float4* oA; float4* oB;               // stage output
  const float4* stPrev;                 // stage 1: step info of the previous step
  float4* stNew;                        // stage 1 writes it, later kernels read it
  const unsigned* wIn;                  // stage 1: max wave speed of the step's input state
  unsigned* wOut;                       // cleared by stage 1, accumulated by the step's last kernel
  int finalCfl;                         // this kernel writes the step's final state
  const MemberHead* xhead;              // per tile: out-of-tile members of its cut-cell groups
  const int* xcell;                     // all tiles' lists
  int maxX;                             // largest per-tile list (sizes the dynamic shared memory)
  int slotIn;                           // ring slot of (A, B): selects the tensor maps of the halo copy
  const TileMaps* tm;                   // the handle's tensor maps, one TileMaps per tile shape
  unsigned* err;                        // set when a halo copy did not complete in time
  int pdl;                              // launch with programmatic dependence on the kernel before it
};

struct PhysArgs {
  Grid g;
  const float4* A1; const float4* B1;   // stage-1 result (its primitives feed the viscous terms)
  const float4* A2; const float4* B2;   // stage-2 result (slot; the fused kernel keeps it on chip)
  float4* oA; float4* oB;
  const float4* st;
  unsigned* wOut;
  int finalCfl;
};

struct SprayArgs {
  Grid g;
  const float4* A1; const float4* B1;   // stage-1 state: the gas the parcels see
  const float4* PA; const float4* PB;   // parcels before the step
  float4* oPA; float4* oPB; float4* oPC;
  const uint8_t* cls;                   // cell classes, rows of clsPitch bytes
  int clsPitch;
  const float4* tab;                    // 256 x 3 injector table
  const float4* st;
  unsigned* key; unsigned* val; float4* dep;   // deposit records (cell key, parcel index, source)
  unsigned long long* acc;              // fixed-point deposit sums of this step, 4 per cell (fast variant)
  unsigned* depFlag;                    // set when a deposit left the fixed-point range (fast variant)
  const unsigned* boundIn;              // (mass, speed) bounds of the ring this step reads (float bits)
  unsigned* boundOut;                   // the same for the ring it writes: max of boundIn and its parcels
  unsigned long long* liveSteps;        // += live parcels this step writes (parcel-steps counter)
  int head, seed;
  const unsigned* hs;                   // if set: (head, seed) read here instead (graph replay)
};

struct ApplyArgs {
  Grid g;
  const float4* A; const float4* B;
  const float4* src;
  const uint8_t* cls;                   // cell classes, rows of clsPitch bytes
  int clsPitch;
  const unsigned long long* acc;        // this step's fixed-point deposit sums (fast variant)
  const unsigned* boundIn;              // the (mass, speed) bounds its deposits were scaled by
  unsigned long long* accNext;          // the next step's, cleared here cell by cell
  float4* oA; float4* oB;
  unsigned* wOut;
  int finalCfl;
  unsigned* hsNext;                     // if set: (head, seed) advanced by one step here (graph replay)
};

// One instance of a batch: its buffers, where it stood in its state ring and
// step-info ping-pong when the batch was (re)built, its first block in the
// batch grid, and its parameter block. The kernels derive the slots of step k
// from (cur0, stepIdx0, wslot0) and the step's BatchPhase (batch_ring).
struct BatchInst {
  Grid g;
  float4* SA[3];
  float4* SB[3];
  float4* stepTex;                      // 2 float4
  unsigned* wmax;                       // 2 slots
  const MemberHead* xhead;
  const int* xcell;
  const TileMaps* tm;                   // the member's tensor maps, one TileMaps per tile shape
  unsigned* err;                        // the member's error word (halo copy timeout)
  int cur0, stepIdx0, wslot0;
  int firstBlock, tilesX;
  int pad_;
  rn_params P;
};
struct BatchPhase {
  int par;                              // step parity: stepIdx = stepIdx0 ^ par, wslot = wslot0 ^ par
  int turn;                             // the ring has turned since parity 0 (not with sprays, whose steps end where they began)
  int finalCfl;                         // the launched kernel writes the step's final state
  int maxX;
  const int* active;                    // if set: per member, 0 = stopped (its blocks return at once)
};

// State-ring slots of member d in phase ph: s0 the step's base state, s1 its
// stage-1 state, s2 its result. The ring turns by one slot pair forwards on even
// step-info parity and back on odd (ring_slots in rn_internal.h).
__host__ __device__ inline void batch_ring(const BatchInst& d, const BatchPhase& ph, int& s0, int& s1, int& s2) {
  const int d0 = d.stepIdx0 ? 2 : 1, dk = (d.stepIdx0 ^ ph.par) ? 2 : 1;
  s0 = (d.cur0 + (ph.turn ? 2 * d0 : 0)) % 3;
  s1 = (s0 + dk) % 3;
  s2 = (s0 + 2 * dk) % 3;
}

// The kernels are compiled twice from the same sources (rn_variant.cu):
//   exact -- IEEE division and square root: every float operation rounds as
//            written, so the state matches the CPU oracle bit for bit wherever
//            pow/exp/log/sin/cos agree with the host's libm;
//   fast  -- the hardware's approximate reciprocal and square root
//            (within 2 ulp, the latitude GLSL highp gives the reference's
//            shaders); agrees with the oracle to ~1e-6 relative L2.
// A solver handle launches through one of the two sets; `tile` selects the
// tile shape (index into TILE_TX/TILE_TY).
struct KernelSet {
  const char* name;
  void (*stage1)(const StageArgs& a, const rn_params& P, int tile, cudaStream_t s);
  void (*stage2)(const StageArgs& a, const rn_params& P, int tile, cudaStream_t s);
  // stage 2 + the viscous/wall/reaction split step in one kernel
  // heavy != nullptr: launch the tiles listing more than XSMALL out-of-tile
  // members (nHeavy of them); else all tiles, skipping those when `skip`
  void (*stage2phys)(const StageArgs& a, const PhysArgs& p, const rn_params& P, int tile, const int* heavy,
                     int nHeavy, bool skip, cudaStream_t s);
  void (*batchStage1)(const BatchInst* d, const int* blockInst, int nblocks, BatchPhase ph, int tile, cudaStream_t s);
  void (*batchStage2)(const BatchInst* d, const int* blockInst, int nblocks, BatchPhase ph, int tile, cudaStream_t s);
  void (*batchStage2Phys)(const BatchInst* d, const int* blockInst, int nblocks, BatchPhase ph, int tile,
                          const int2* heavy, int nHeavy, bool skip, cudaStream_t s);
  void (*reduce)(const Grid& g, const float4* A, const float4* B, unsigned* w, cudaStream_t s);
  void (*rescale)(const Grid& g, const float4* A, const float4* B, float4* oA, float4* oB, float fp, float fT,
                  float du, const rn_params& P, cudaStream_t s);
  void (*wallrow)(const Grid& g, const float4* A, const float4* B, const float4* jw, float4* row, cudaStream_t s);
  void (*integrals)(const Grid& g, const float4* A, const float4* B, const float4* geoAx,
                    const rn_integral_spec& spec, const float4* st, double* out, cudaStream_t s);
  int (*spray)(const SprayArgs& a, const rn_params& P, void* sortTemp, size_t sortTempBytes, unsigned* keyOut,
               unsigned* valOut, float4* src, cudaStream_t s, int* launches);
  void (*apply)(const ApplyArgs& a, const rn_params& P, cudaStream_t s);
  size_t (*sortTempBytes)(int Ncells);
  int (*init)();                    // opts the kernels into the dynamic shared memory they need
};
extern const KernelSet kernels_exact;
extern const KernelSet kernels_fast;

}  // namespace rn
