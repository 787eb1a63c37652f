// Interface of the integer tensor-core screening pass (see screen_i8.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace certex_b200 {

constexpr int kMaxSegs   = 4;  // segments (query panel, base-tile range) one CTA may be given
constexpr int kMaxStages = 8;  // upper bound of the base-tile ring

constexpr int kQueryTile = 128;  // queries per accumulator unit (TMEM lanes)
constexpr int kBaseTile  = 256;  // stored rows per accumulator unit (TMEM columns, N of one MMA instruction)
constexpr int kGroupRows = 64;   // rows per group maximum (one epilogue warp's piece of a unit)

// kModeRate issues the loads and MMAs of every unit back to back with no epilogue (tensor-pipe rate probe).
// kModeGroupBound is the threshold stage at the screen's price: a tile's 16 chains are 16 adjacent anchors each (the
// 4-D anchor map below), e is taken per chain (its minimum, in `cmax`), and gmax receives per group of 64 columns
//   max over its four chains of (max of <q, x> over the chain + min of e over the chain),
// a value some row of the group reaches (the row with the chain's largest product has at least the chain's smallest e),
// so the k-th largest of them is still reached by k distinct rows. kModeGroupMax is the exact maximum of <q, x> + e.
enum : int { kModeScreen = 0, kModeGroupMax = 1, kModeRate = 2, kModeGroupBound = 3 };

/// Init value of a column that must never pass a threshold (removed rows, padding beyond the last row).
constexpr int32_t kNeverInit = -(1 << 30);

constexpr int kChainRows = 16;  // rows per chain: the unit of the conservative threshold test

/// One contiguous piece of work of a CTA: query tiles [q_tile0, q_tile0 + n_qtiles) against base tiles [t0, t1)
/// (query tiles of 128 queries, base tiles of 256 rows).
struct ScreenSeg {
  int q_tile0;
  int n_qtiles;
  int t0;
  int t1;
};

/// An entry of a query's candidate list: the rows of one chain that reached the query's threshold (or, with rows of more than two
/// K blocks, one of them).
struct __align__(16) Candidate {
  uint32_t chain;   // rows 16 chain .. 16 chain + 15 of the code rows the pass read
  uint32_t mask;    // one bit per row of the chain
  int32_t product;  // the largest <q, x> of the chain (int32, or the bits of a float): a row in the mask has it
  uint32_t unused;
};

struct ScreenArgs {
  const int32_t* init;            // [n_tiles * 256] per-row term e[x] added to <q, x> (kNeverInit: removed / padding)
  const int32_t* cmax;            // SCREEN: [n_tiles * 16] maximum of e over every chain of 16 rows; GROUPBOUND: minimum
  const int32_t* thr;             // SCREEN: [nq] keep iff <q, x> + e[x] >= thr[q]
  int32_t* gmax;                  // GROUPMAX: [nq, ld_gmax] maximum of <q, x> + e[x] over every group of 64 rows
  int64_t ld_gmax;
  Candidate* cand;                // SCREEN: [nq, ld_cand] the chains kept per query, in no order
  uint32_t* cnt;                  // SCREEN: [nq] chains kept (may exceed cap: overflow, the excess is not written)
  uint32_t cap;
  uint32_t ld_cand;
  int nq;
  int kb;                         // K blocks of 128 bytes per row
  int panel_tiles;                // query tiles resident in shared memory
  int n_stages;                   // base-tile ring depth
  int mode;
  int f16;                        // 1: fp16 codes, fp32 accumulators; init / cmax / thr hold float bits, gmax float keys
  uint32_t q_signed;              // 0 = uint8 codes, 1 = int8 codes
  uint32_t x_signed;
  const ScreenSeg* segs;          // [grid, kMaxSegs]; unused entries have t1 <= t0. With seg_begin: one list
  const int* seg_begin;           // optional [grid + 1]: CTA b works on segs[seg_begin[b] .. seg_begin[b + 1])
  const int* seg_col0;            // optional, per segment: the tile whose groups are columns 0..3 of gmax (else tile 0)
  const int* seg_step;            // optional, GROUPMAX: tile t of a segment stands for tile col0 + (t - col0) * step
  int wide;                       // 1: rows of more than two K blocks; a segment then has at most two query tiles
  int plain_tiles;                // GROUPMAX: tile t is rows [256 t, 256 t + 256) of a 2-D map (else the 3-D anchor map)
  int fine_groups;                // GROUPMAX: one maximum per 16 rows (16 columns of gmax per tile) instead of per 64 (4)
  int wide_groups;                // GROUPBOUND: one value per 128 rows (2 columns of gmax per tile)
  int* err;                       // set to a non-zero code when a bounded wait gave up
  long long* trace;               // trace builds only (see screen_set_trace): [trace_units, 12] clock stamps of CTA 0
  int trace_units;
};

constexpr size_t kMaxSmem = 227 * 1024;  // dynamic shared memory a block may have

/// What a launch needs of it.
size_t screen_smem_bytes(int kb, int panel_tiles, int n_stages);

/// Profiling aid, effective only in a library built with -DCERTEX_SCREEN_TRACE=1 (make trace): CTA 0 of every later
/// pass writes SM clock stamps of its first `units` accumulator units to the device buffer `trace` ([units, 12] int64;
/// nullptr: off). The stamps cost time themselves (every instruction on the MMA-issuing thread's and the epilogue's
/// path does): a trace shows where a unit's round trip goes, not how fast the untraced pass is. Process-wide.
void screen_set_trace(long long* trace, int units);
bool screen_trace_compiled();

cudaError_t screen_i8_launch(const CUtensorMap& tm_q, const CUtensorMap& tm_x, const ScreenArgs& args, int grid, cudaStream_t stream);

}  // namespace certex_b200
