// Tiled pipeline schedule of a sparse triangular sweep (forward over the
// entries left of the diagonal, or backward over those right of it).
//
// The rows are cut into dependency chains (each row continues the chain of
// its most recent dependency, so on a naturally ordered structured mesh the
// chains are the grid lines along the fastest index), the chains are grouped
// into tiles of about n/T rows by cuts along the axes (or, without
// coordinates, by growing regions over the chain graph), and every tile is
// given to one thread block.  A block walks its rows level by
// level: rows of one level are independent, values produced inside the tile
// in the last R steps are read from a shared-memory ring, everything else
// from global memory after the producing tile has published enough progress.
#pragma once
#include <string>
#include <vector>

struct SweepSchedule {
  int n = 0;
  int ntiles = 0;
  int nlev = 0;                    // levels of the sweep (0..nlev-1)
  int R = 4;                       // shared-memory ring depth in steps
  int max_slots = 0;               // widest tile (rows of one tile in one level)
  int cut_axes = 0;                // axes that the tiles were cut along
  std::vector<int> tile_step_ptr;  // tile t owns global steps [ptr[t], ptr[t+1])
  std::vector<int> step_level;     // level of each global step
  std::vector<int> tile_slots;     // rows per step (padded width) of each tile
  std::vector<int> step_row_ptr;   // offset of each global step's padded row list
  std::vector<int> rows;           // padded row ids, -1 = empty slot
  std::vector<int> wait_ptr;       // per global step: waits [ptr[s], ptr[s+1])
  std::vector<int> wait_tile;      // producer tile of a wait
  std::vector<int> wait_level;     // producer must have published progress >= this level
  // per CSR entry of the swept part: >= 0 ring index (step%R)*slots+slot of
  // the producing row in the same tile, < 0 global row -(code)-2
  std::vector<int> code;           // size nnz, entries of the other part untouched
  long long cross_tile_entries = 0, ring_entries = 0, global_same_tile_entries = 0;
};

// ia, ja, dg: 0-based CSR (sorted rows) and diagonal positions; lev: level of
// every row for the direction (forward: from the lower part, backward: from
// the upper part); code must have nnz entries (shared between directions).
// xyz (optional, 3*n: x,y,z of every row, e.g. the cell centroids) lets the
// tiles be cut along the axes by the chain centroids: dependencies along the
// mesh then run one way between tiles, so tiles pipeline instead of waiting
// on each other at every level.  Without
// coordinates the tiles are grown over the chain graph.  with_waits false
// stops after the layout (tiles, steps, rows): code, the waits and the entry
// counts are left empty.  nocut: an axis (0, 1, 2) not to cut along, -1: none,
// FC_CUT_UNLESS_3: none, and where all three axes would be cut S.cut_axes alone
// is filled in.
#define FC_CUT_UNLESS_3 (-2)
void build_sweep_schedule(int n, const int* ia, const int* ja, const int* dg, const std::vector<int>& lev, int nlev,
                          bool forward, int ntiles, const double* xyz, SweepSchedule& S, std::vector<int>& code,
                          bool with_waits = true, int nocut = -1);

// Critical-path estimate (microseconds) of a schedule: per level of a tile
// tau0 per FC_STEP_ROWS rows begun + per_row * rows, cross-tile waits delayed
// by hop after publication.
#define FC_STEP_ROWS 128  // rows of a step of the sweeps (fc_sweep.cuh)
double estimate_sweep_us(const SweepSchedule& S, double tau0, double per_row, double hop);

// ---------------------------------------------------------------------------
// Schedule-ordered sweep structure.
//
// The rows are renumbered in schedule order: tile by tile, step by step, so
// that every step of every tile is a contiguous range of new row indices and
// a thread block walks consecutive memory.  The forward sweep runs the steps
// of a tile in order, the backward sweep runs them in reverse; this is valid
// for both triangles because the levels are taken over the symmetrised
// pattern (row i waits for every j < i with a_ij != 0 or a_ji != 0).
//
// Per new row and per triangle the first FC_ELL entries (in the row's CSR
// order) are stored column-major (entry e of row q at e*nE + q, nE = n
// rounded up to a multiple of 4 so that every column starts 16-byte
// aligned), the rest in an overflow list.  A dependency produced in the same tile within the last
// R-1 steps is read from the block's shared-memory ring (code >= 0: ring
// index (local step % R) * W + position); every other dependency is pushed:
// its producer stores the value into the consumer's own slot of an exchange
// array xv.  The slots of a step's rows form one contiguous block of xv (in
// row order, entries in CSR order); the producer's targets likewise form one
// block per producing step.
//
// With chunk > 0 a level of a tile wider than chunk rows becomes several
// consecutive steps of at most chunk rows (their rows are independent, so
// the tiling, the levels and the values stay the same).  The dependencies of
// a level then lie up to two levels' worth of steps back, so the ring gets
// that many times its depth (as far as FC_RING_BYTES allows).
#define FC_ELL 4
#define FC_RING_BYTES (64 * 1024)  // most shared memory of a value ring deepened for chunked levels

// Last word of a row record: the row's entries, the exchanged ones among the
// first FC_ELL of them, its first exchanged value in the step's block.  A row
// served by the ring may have as many entries as the ring has values; in 8 bits
// rows of more than 255 were solved with a truncated count.
#define FC_REC_MAX_ENTRIES 8191
#define FC_REC_PACK(entries, exchanged, offset) ((entries) | ((exchanged) << 13) | (int)((unsigned)(offset) << 16))
#define FC_REC_ENTRIES(w) ((w) & FC_REC_MAX_ENTRIES)
#define FC_REC_EXCHANGED(w) (((w) >> 13) & 7)
#define FC_REC_OFFSET(w) ((unsigned)(w) >> 16)

struct OrderedDir {
  std::vector<int> ne;        // [nE] entries of this triangle in the row
  // For checks only (the kernels read rec and the slices): the original CSR
  // slots of the first FC_ELL entries, -1 past ne, the new indices of their
  // columns, [FC_ELL*nE], and [4*nE] a row record with the codes themselves, for
  // rows of up to 255 entries:
  std::vector<int> slot;
  std::vector<int> col;
  //   [0] ne | np << 8 | xoff << 16   (np: pushes of the row's value; xoff:
  //       first exchange slot of the row in its step's exchange block)
  //   [1] poff: first push target of the row in its step's push block
  //   [2], [3] codes of entries 0..3, 16 bits each, stored as code + 1
  //       (0: the value arrives through the exchange block)
  std::vector<int> srec;
  // [4*nE] the row record as the kernels read it, one 16-byte load per row:
  //   [0] np | poff << 8
  //   [1], [2] places of the values of entries 0..3, 16 bits each: a ring
  //       index (below R * W of the tile), R * W: a zero (past the row's
  //       entries), R * W + 1 + j: value j of the step's exchange block
  //   [3] FC_REC_ENTRIES, FC_REC_EXCHANGED, FC_REC_OFFSET above
  std::vector<int> rec;
  std::vector<int> xv_ptr;    // [nsteps+1] exchange block of each step
  std::vector<int> push_ptr;  // [nsteps+1] push block of each step (multiples of 4)
  std::vector<int> push;      // absolute exchange positions the values are pushed to
  std::vector<int> ovf_ptr;   // [n+1] entries e >= FC_ELL
  std::vector<int> ovf_slot, ovf_code, ovf_col;
  long long ring_entries = 0, pushed_entries = 0, cross_tile_entries = 0;
};

struct OrderedSweep {
  int n = 0, nE = 0, ntiles = 0, nsteps = 0, nlev = 0, R = 4, maxW = 0, max_tile_steps = 0;
  int max_level_rows = 0;          // rows of a tile in its widest level (maxW: in its widest step)
  int max_entries = 0;             // entries of the fullest row of a triangle
  std::vector<int> perm, iperm;    // new -> old, old -> new
  std::vector<int> tile_step_ptr;  // [ntiles+1]
  std::vector<int> step_ptr;       // [nsteps+1] first new row of each step
  std::vector<int> rp_ptr;         // [nsteps+1] the same with every step's rows padded to a multiple of 4
  std::vector<int> tile_W;         // widest step of each tile (ring / staging width)
  OrderedDir dir[2];               // 0: left of the diagonal (forward), 1: right (backward)
  std::vector<int> lo_tslot;       // [FC_ELL*nE] transpose slot of each lower entry (DILU)
  std::vector<int> lo_ovf_tslot;
  std::vector<int> dslot;          // [nE] original diagonal slot, 0 in the padding (for checks only)
  std::vector<int> p_ptr, p_col, p_slot;  // the matrix in new numbering, entries in original order
};

// levels over the symmetrised lower triangle: lev(i) = 1 + max lev(j) over
// j < i with a_ij != 0 or a_ji != 0; returns the number of levels
int symmetric_levels(int n, const int* ia, const int* ja, const int* dg, std::vector<int>& lev);

// The tile count among cand whose forward schedule has the smallest
// critical-path estimate, worked out from the tiles alone (large systems: on
// as many threads as there are cores; ties go to the earlier candidate,
// duplicates and counts < 1 are skipped).  best_est (optional) receives that
// estimate.  With nocut, and where the chains spread along all three axes,
// every second count is tried with each axis left out of the cuts (and the
// first two with all of them), and *nocut receives the best one (-1: none): on
// tetrahedra a cut along one of the axes can separate chains that depend on
// each other both ways, which makes the tiles wait for each other at every
// level (750k tetrahedra, 150 tiles: 250 such pairs of tiles and an
// estimate of 152 us with all axes cut, none and 55 us without one of them).
int pick_sweep_tiles(int n, const int* ia, const int* ja, const int* dg, const double* xyz, const std::vector<int>& cand,
                     double tau0, double per_row, double hop, double* best_est, int* nocut = nullptr);

// ia, ja, dg 0-based; ts (optional) the transpose slot of every entry;
// ntiles the tile target; xyz (optional) row coordinates for the tiling; R
// the ring depth; wmax > 0 caps the rows of a level in a tile by splitting
// levels (and cutting the tiles again); chunk > 0 caps the rows of a step as
// described above; nocut as above; checks fills in the arrays kept for checks
// alone.  S receives the underlying tiled schedule (for the critical-path
// estimate).  Returns false with a message if a consistency check fails.
bool build_ordered_sweep(int n, const int* ia, const int* ja, const int* dg, const int* ts, int ntiles,
                         const double* xyz, int R, OrderedSweep& O, SweepSchedule& S, std::string& err,
                         int wmax = 0, int chunk = 0, int nocut = -1, bool checks = true);
