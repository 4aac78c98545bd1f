// Band form of the persistent ADMM solve (sm_100a): tables, layout and host
// interface.  Kernels in band.cu, host tables in band_schedule.cu.
//
// MPC KKT matrices ordered by minimum degree factor into three parts.  The
// *head*: elimination subtrees of depth at most two -- a root column, which
// reads only leaf columns ("children") whose one entry lies in its row.  The
// *chain*: one long run of columns that reach only a few columns further (a
// band), the serial part of both sweeps.  And where the ordering starts a
// second, short run at the horizon's other end, the *pre-chain*: columns that
// come before head columns adding to the same rows.  The band form gives the
// chain to one warp that keeps a window of rows in registers, and everything
// else -- the head's columns, the ADMM updates, the head's contributions to the
// chain's rows -- to the other warps of the CTA, which need no order among
// themselves; the pre-chain goes to one of them.
#pragma once

#include <string>
#include <vector>

#include "stream.cuh"

namespace wmpc {

constexpr int kBandStages = 3;         // chain chunks in flight
constexpr int kBandWarps = 18;         // item warps of a CTA that has its SM alone
constexpr int kBandWideWarps = 14;     // the same for a 16-row window, whose chain needs more registers
constexpr int kBandChildren = 2;       // children of a root, at most
constexpr int kBandUsesPre = 1 << 15;  // item word flag: reads pre-chain values

// Everything a tile of 32 instances needs is one stream of blen floats; L
// entries in units of 4 ([unit][lane][4]), D^-1, parameters (q, or (l, u)) and
// iterates (x, or (z, y)) as [lane] records:
//   chain chunks, read with one bulk copy each: the columns' window entries
//     (rows c+1 ..; every column units - 1 or units units), the chunk's far
//     entries, then D^-1 of its columns;
//   items, each copied by the warp that works on it: its record (128-byte rows,
//     the pattern's; it travels in the stream so that an item is one run of
//     bytes) and
//     a B item (one subtree): the root's units -- child 0's entry in the last
//       slot, child 1's in the one before --, then D^-1, parameters and iterate
//       of the root and of each child; before the subtrees the pre-chain's
//       columns (units and D^-1);
//     an F item (one chain or pre-chain row): its head and pre-chain entries by
//       ascending column, its parameters and iterate.
struct BandPlan {
  int n, n_prim, n_pre, T, T4;  // KKT dimension, primal indices, pre-chain and chain columns, T to a multiple of 4
  int units;                    // window units of a chain column (2 or 4): rows up to 4 units past it
  int n_chunks, chunk_cols;     // chain chunks, columns per chunk (a multiple of 4)
  int n_yr;                     // roots and pre-chain columns (rows of the forward-result vector; row n_yr is zero)
  int nb;                       // B items (subtrees)
  int blen;                     // floats per tile
  int chunk_bytes;              // the largest chunk
  int item_bytes;               // the largest item
  int n_rows;                   // 128-byte rows of records
  const int* col_word;   // [T4] 1: the last unit is there too | first unit in the chunk << 1
  const int4* chunk;     // [n_chunks] {float offset, bytes before D^-1, columns | far entries << 8, chain rows
                         // that its forward pass needs}
  const int* far_ptr;    // [n_chunks] first far entry
  const int4* far;       // {column in its chunk, work-vector byte offset of its row, byte offset in the chunk, 0}
  const int* item;       // [2 n_pre + nb + T] stream offset in 128-byte rows | rows << 22
  const int* rec;        // [n_rows][32] records, and where each row lies in the stream
  const int* rec_off;    // [n_rows]
  const int* iter_off;   // [n] by original KKT index: stream offset of its iterate record
  const int* param_off;  // [n] by original KKT index: stream offset of its parameter record
};
// Items: pre-chain columns (last first), subtrees, pre-chain rows, chain rows.  A
// record (32-bit words) of a pre-chain column or subtree: {units | children << 4 |
// kinds << 8, 12, 16 (root, children) | record rows << 27, forward-result byte
// offset, chunks needed | kBandUsesPre, solution byte offset of a pre-chain column,
// or stream offset of the root's D^-1}, {rho, 1/rho, unscale, residual offset} of
// the root and of two children, then the work-vector byte offset of every entry.  Of
// a row: {units | kind << 8 | kBandUsesPre | record rows << 27, work-vector byte
// offset, forward-result byte offset of a pre-chain row or -1, stream offset of its
// parameters}, {rho, 1/rho, unscale, residual offset}, then the forward-result byte
// offset of every entry.  A kind: bit 0 constraint, bits 1-2 its rho class + 1.
constexpr int kBandRecB = 16, kBandRecF = 8;  // words before the entries' offsets

struct HostBand {
  int n = 0, n_prim = 0, n_pre = 0, T = 0, T4 = 0, units = 0, n_chunks = 0, chunk_cols = 0, n_yr = 0, nb = 0;
  int blen = 0, chunk_bytes = 0, item_bytes = 0;
  std::vector<int> col_word, chunk, far_ptr, far, item, rec, rec_off, iter_off, param_off;
  // where the factorization writes: per L entry (CSC order) its position and
  // its copy's (a scratch unit where there is none), per column D^-1's; L
  // positions have lane stride 4, D^-1 lane stride 1; padding to be zeroed
  std::vector<int> lpos, lpos2, dpos, pad;
};

// False (and *why) where the pattern has no such form: few columns outside the
// head reach past the window, and the work vectors fit shared memory.
bool build_band_tables(const HostPattern& hp, const float* rho, const float* rhoinv, const int* rho_type, int n_primal,
                       const float* unscale_by_index, HostBand* out, std::string* why);

// Rows of the work vector: the chain's (to a multiple of 4), the window's
// overhang, a zero row, the pre-chain's solution.
__host__ __device__ inline int band_vzero(int t4, int units) { return t4 + 4 * units; }
__host__ __device__ inline int band_vrows(int t4, int units, int n_pre) { return t4 + 4 * units + 1 + n_pre; }

// One class of a band launch.
struct BandJobDesc {
  BandPlan bp;
  float* stream = nullptr;
  float* pres = nullptr;  // scaled primal residuals [tile][m][32] (termination checks)
  int* iters = nullptr;
  const float* rho_b = nullptr;
  const int* rho_count = nullptr;
  int n_tiles = 0, max_iter = 0, batch = 0, check_every = 0, ctas_limit = 2;
  float chg_eps = 0.0f, sigma = 0.0f, alpha = 0.0f, one_minus_alpha = 0.0f;
};

// A solve's buffers: per tile the stream, the residuals.
struct BandWork {
  float *stream, *pres;
  int tiles;
};

struct Osqp;
size_t band_workspace_floats(const BandPlan& bp, int batch);
BandWork band_work(const BandPlan& bp, int batch, float* work);
int band_state_in(const BandPlan& bp, const Osqp& o, const float* aT, long long lda, int sba, bool track, bool warm,
                  const float* x, const float* z, const float* y, const float* qs, const float* ls, const float* us,
                  const BandWork& w, int batch, cudaStream_t s);
int band_state_out(const BandPlan& bp, const BandWork& w, float* x, float* z, float* y, int batch, cudaStream_t s);
// whether one launch can hold these classes
bool band_fits(const BandPlan* const* plans, int n);
int band_run(const BandJobDesc* jobs, int n_jobs, int* error, int num_sms, cudaStream_t s);
// items of an iteration in item warp 0's list (the longest)
inline int band_items(int n_pre, int nb, int T, int warps) {
  return 2 * n_pre + (nb + warps - 1) / warps + (T + warps - 1) / warps;
}

// An item warp's copies ahead.  An item's copy for the next iteration starts when the
// item kBandAhead places before it in the warp's list (B items, then F items) is
// released.  Its iterate was stored a few items before; where the warp has at least
// kBandAhead items in each phase the end of a phase, with its fence, lies between.
// Else every item has a fence of its own.
constexpr int kBandAhead = 4;
__host__ __device__ constexpr bool band_item_fence(int mb, int mf) { return mb < kBandAhead || mf < kBandAhead; }

// Sets of per-warp maxima a CTA needs.  A warp with a chain row writes its maxima in
// the F phase, once every warp has read those of the iteration before.  One without
// (a chain of fewer rows than item warps) writes them at the end of its B phase,
// which waits for no other item warp's decision: two sets, by iteration parity, put
// an F phase between a set's last read and its next write.
inline int band_maxima_sets(int T, int warps) { return T < warps ? 2 : 1; }

// bytes of shared memory a CTA of `warps` item warps, `stages` chain stages and
// `maxima_sets` sets of maxima takes
size_t band_smem_bytes(int vrows, int yrows, int t4, int n_chunks, int n_items, int chunk_bytes, int ring_bytes,
                       int warps, int stages, int maxima_sets);

}  // namespace wmpc
