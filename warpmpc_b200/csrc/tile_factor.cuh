// Factorization of a 32-instance tile by all warps of a CTA (sm_100a): tables and
// host interface.  Kernel in tile_factor.cu, host scheduler in
// tile_factor_schedule.cu.
#pragma once

#include <string>
#include <vector>

#include "common.cuh"
#include "stream.cuh"

namespace wmpc {

// The up-looking LDL^T factorization as a program of small operations, one list
// per warp, cut into ticks that end at a barrier.  Operation kinds:
//   load  raw KKT inputs of a row, copied into the row's slots;
//   init  a row's slots from them (the pattern's scales, 0 for fill-in);
//   step  one step of a row's program (reference order): y = slot of the column,
//         subtract L' y from the slots of the column's earlier rows, L = y D^-1,
//         d -= y L; the last step of a row also inverts d.  L' = y' D^-1 is formed
//         again from the earlier row's y' (the same product, the same bits): y' is
//         final a step before that row stores L', so a column of the chain takes
//         one tick, where waiting for L' takes two.
// All values in flight -- rows being formed, and every y and D^-1 that a later
// step still reads -- live in shared-memory slots of [32] floats, assigned by the
// scheduler; an operation reads only what an earlier tick, or an earlier
// operation of its own warp, has written.  L and D^-1 go to memory besides.
//
// A list is read as int4 words, in pieces of 32; an operation lies within one
// piece.  Slots are named by their byte offset, 128 slot: the low field F of a word
// is bits 7-17, the high field G bits 18-28.  Operation header x: kind | end of
// tick << 3 | last of its row << 4 | count << 5 (6 bits) and
//   step   x: slot of d << 21; y: F slot, G D^-1 slot of the column; z, w: L's
//          offsets in the backward and the forward stream; last: one more word
//          {D^-1 offset}; then `count` words of 4 updates {F slot, G slot of y'};
//          fillers name slot 0
//   inputs `count` words {F slot, scale, add, 0}: raw scale + add
//   zeros  `count` words of 4 slots set to 0 (fillers: slot 0)
//   consts `count` words {F slot, value, F slot, value} (filler: slot 0)
//   pivot  y: F slot of d; z: D^-1 offset (a row without steps)
//   load   y: array (0 P, 1 A, 2 1/rho rows); `count` words of 4 inputs, index | slot <<
//          20 (fillers: input 0 into slot 0)
//   ticks  y: barriers
//   piece  go on at the next piece; with y set the list ends
enum { kTfStep = 0, kTfInputs = 1, kTfZeros = 2, kTfConsts = 3, kTfPivot = 4, kTfLoad = 5, kTfTicks = 6, kTfPiece = 7 };
constexpr unsigned kTfF = 2047u << 7;  // the low field
constexpr int kTfWarps = 16;    // warps per CTA
constexpr int kTfDelay = 4;     // ticks between a load and its use
constexpr int kTfTick = 400;    // a warp's work per tick, in cycles as the scheduler estimates them
constexpr int kTfSlots = 1536;  // slots, at most (0 is a dummy): one CTA per SM
constexpr int kTfSlots2 = 624;  // for two

// A list goes on at a piece that was asked for `ago` ticks earlier.  Copies become
// a group when their tick ends: how many groups may still be under way, or -1 where
// all copies have to land, those of this tick, no group yet, among them (rows of a
// hundred inputs and more fill several pieces within a tick).
__host__ __device__ constexpr int tf_piece_wait(int ago) { return ago >= kTfDelay ? kTfDelay - 1 : -1; }

struct TileFactor {
  const int4* prog = nullptr;  // null: not available
  const int* warp_off = nullptr;  // [kTfWarps] first word of each list
  int slots = 0;
};

// The schedule of a pattern: which warp does what in which tick, and the slots.
struct HostTileSchedule {
  struct Op {
    int tick, task;  // task: step, nnz_l + row: init, nnz_l + n + row: load
  };
  std::vector<std::vector<Op>> ops;  // by warp
  std::vector<int> slot;             // by step (its row's entry), then by row (d, then D^-1)
  std::vector<std::vector<std::pair<int, int>>> upd;  // by step: {slot index in the row, the earlier row's step}
  int slots = 0, ticks = 0;
};

bool schedule_tile_factor(const HostPattern& hp, const std::vector<int>& init_slot, HostTileSchedule* out,
                          std::string* why);

struct HostTileFactor {
  std::vector<int> prog, warp_off;
  std::vector<int> step_at, row_at;  // words of prog that hold a step's L offsets (two), a row's D^-1 offset
  int slots = 0, ticks = 0;
};

// The lists, without the places of the results.  kin: [n + inputs] {source or -1,
// kind, scale, add} in row-program order, sources: np P values, na A values, then
// 1/rho rows.
bool emit_tile_factor(const HostTileSchedule& sched, const HostPattern& hp, const std::vector<int>& init_slot,
                      const int* kin, int np, int na, HostTileFactor* out, std::string* why);

// The places: boff, foff [nnz_l] by program step, doff [n].
void place_tile_factor(const int* boff, const int* foff, const int* doff, HostTileFactor* t);

// Runs it over a batch, into the streams of `sp`.
struct TileFactorInputs {
  const float *p, *a, *r;  // P, A values, 1/rho rows: [index][ld] with batch stride sb
  long long ldp, lda, ldr;
  int sbp, sba, np, na;
};
int tile_factor_stream(const TileFactor& tf, const StreamPlan& sp, const TileFactorInputs& in, float* bstream,
                       float* fstream, int* status, int batch, int num_sms, const int* only, cudaStream_t s);

// Runs it over a batch of KKT values ([nnz][ld], batch stride sb), into lx [nnz_l][batch],
// d and dinv [n][batch] (only: just the instances marked in it).
int tile_factor_planes(const TileFactor& tf, const float* values, long long ld, int sb, float* lx, float* d,
                       float* dinv, int batch, int num_sms, const int* only, cudaStream_t s);

size_t tile_factor_smem(int slots);

}  // namespace wmpc
