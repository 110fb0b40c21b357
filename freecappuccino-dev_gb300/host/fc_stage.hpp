// Staging of the schedule-ordered sweeps (csrc/fc_sweep.cuh), as far as host
// and device share it: the warp roles, the stage buffers of the modes, the
// groups of steps that a buffer holds, and the importers' rule for taking a
// buffer again.
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

#include "fc_schedule.hpp"

#if defined(__CUDACC__)
#define FC_STAGE_HD __host__ __device__ inline
#else
#define FC_STAGE_HD inline
#endif

// Warp roles of a block: FC_SETS x FC_SET_WARPS compute warps, the importers,
// the stager.  A set is one warp per SM sub-partition and covers a step of
// FC_SET_ROWS rows with one row per thread: four warps issue their FMAs in
// about the 64 cycles one FMA takes, so more rows per step would lengthen the
// step in proportion.  20 warps leave 96 registers a thread (21 would leave 80).
#define FC_SETS 4
#define FC_SET_WARPS 4
#define FC_IMP_WARPS 3
#define FC_SET_ROWS (32 * FC_SET_WARPS)
static_assert(FC_SET_ROWS == FC_STEP_ROWS, "the schedule's cost model counts these steps");

#define FC_MAX_STAGES 16
#define FC_SMEM_HDR (2 * FC_MAX_STAGES * 8)  // full and empty mbarriers at the start of the dynamic area
#define FC_SWEEP_SMEM (200 * 1024)           // dynamic shared memory budget of a sweep kernel

// Named barriers 1..FC_STEP_BARS: the barrier of step k releases the set of
// step k once the set of step k-1 and the importer of step k have arrived.  The
// importers stay less than FC_STEP_BARS steps ahead, so that none arrives twice.
#define FC_STEP_BARS (FC_IMP_WARPS * FC_SETS)

namespace fcdev {

// the form of the applications (see the header of fc_sweep.cuh)
template <class T> struct ScaledApply { static constexpr bool value = sizeof(T) == 8; };
// values per row of a step's block
template <class T>
FC_STAGE_HD int blob_fields(int nc, int dirn) { return nc + dirn + (ScaledApply<T>::value ? 0 : 1); }
// byte offset of the block of a step: rp padded rows and pp push targets precede it
template <class T>
FC_STAGE_HD size_t blob_offset(int rp, int pp, int fields) {
  return (size_t)rp * (16 + sizeof(T) * fields) + 4 * (size_t)pp;
}

enum { OS_SETUP_DIC = 0, OS_SETUP_DILU, OS_FWD, OS_BWD, OS_BWD_DOT, OS_GS };

// One stage buffer of a sweep mode, for a group of steps: the blocks, the a_ii
// and transposes of the setups, for Gauss-Seidel a_ii and the blocks of the
// upper triangle, the q and e windows (rows widened to 16-byte bounds) and the
// exchanged values.  View: the group's sizes, OrdView or StepGroups.
struct StageLayout {
  int oX, oT, oU, oQ, oE, oI, bytes;
  template <class T, class View>
  FC_STAGE_HD static StageLayout of(const View& O, int mode) {
    StageLayout L;
    const int sz = (int)sizeof(T), dirn = mode == OS_BWD || mode == OS_BWD_DOT;
    const bool setup = mode == OS_SETUP_DIC || mode == OS_SETUP_DILU, gs = mode == OS_GS;
    int o = 0;
    auto take = [&](bool used, int b) { const int r = o; if (used) o += (b + 15) & ~15; return r; };
    take(true, 4 * O.g_push + (16 + blob_fields<T>(O.nc, dirn) * sz) * O.g_padded);
    L.oX = take(setup || gs, sz * O.g_padded);
    L.oT = take(mode == OS_SETUP_DILU, sz * O.g_padded * O.nc);
    L.oU = take(gs, 4 * O.g_push + (16 + blob_fields<T>(O.nc, 1) * sz) * O.g_padded);
    L.oQ = take(!setup, sz * (O.g_rows + 8));
    L.oE = take(mode == OS_BWD_DOT || gs, sz * (O.g_rows + 8));
    L.oI = take(true, sz * O.g_x);
    L.bytes = o;
    return L;
  }
};

// stage buffers of one mode within a stage area of `area` bytes: the largest
// power of two (at most FC_MAX_STAGES) whose buffers fit
FC_STAGE_HD int stages_in(size_t area, int buffer_bytes) {
  int K = 1;
  while (2 * K <= FC_MAX_STAGES && (size_t)(2 * K) * (size_t)buffer_bytes <= area) K *= 2;
  return K;
}

// dynamic shared memory of an ordered-sweep kernel: mbarriers, ring (and the
// zero past its end), the stage area (cut by every sweep mode into its own
// buffers), the abort flag and the stager's word
template <class T>
inline size_t osweep_fixed_bytes(int R, int maxW) {
  size_t ring = (((size_t)R * maxW + 1) * sizeof(T) + 15) & ~(size_t)15;
  return FC_SMEM_HDR + ring + 16;
}

// The importer of group g fills the exchanged values of the buffer that group
// g - K used, and releases steps whose named barriers the steps FC_STEP_BARS
// before used: both are free once group g - import_ahead is done.
// (Both functions run at the start of every sweep, where a division costs a
// hundredth of a short one; G is FC_SETS, 2 or 1.)
FC_STAGE_HD int import_ahead(int K, int G) {
  const int most = G == FC_SETS ? FC_STEP_BARS / FC_SETS : G == 2 ? FC_STEP_BARS / 2 : FC_STEP_BARS;
  return K < most ? K : most;
}

// How it learns that.  By the parity of that group's `empty` barrier, the use
// before must be known to be complete (else the test answers for the phase
// before).  The importer knows group h = g - ahead - FC_IMP_WARPS from its wait
// before, and with it the groups up to h - FC_SETS / G: a set releases the next
// step before it stores and gives its buffer back, so steps complete out of
// order, but every set has given back the ones before its own.  The use before
// is group g - ahead - K, so the parity tells for K >= FC_IMP_WARPS +
// FC_SETS / G.  Below (four buffers of one or two steps) ahead is K, and the
// stager, which waits for all groups in order, says how far it has come.
FC_STAGE_HD bool import_by_parity(int K, int G) { return K * G >= FC_IMP_WARPS * G + FC_SETS; }

// A structure's steps in groups of G, one stage buffer each: the largest group
// and, with desc, the descriptors of the steps (OrdView::desc).
struct StepGroups {
  int G = 0, nc = 3, gen = 0;
  int g_rows = 0, g_padded = 0, g_push = 0, g_x = 0;
};

// false if a descriptor's 16-bit fields do not hold a group
bool group_steps(const OrderedSweep& O, int G, StepGroups& V, std::vector<int>* desc);

// the stage area of the ordered sweeps: the shared memory the fixed parts
// leave (the sweep modes cut it into as many buffers as fit, at most
// FC_MAX_STAGES); 0 when nothing is left
inline size_t ordered_stage_area(int R, int maxW) {
  const size_t fixed = osweep_fixed_bytes<double>(R, maxW);
  return fixed >= (size_t)FC_SWEEP_SMEM ? 0 : ((size_t)FC_SWEEP_SMEM - fixed) & ~(size_t)15;
}

// The most steps of a stage buffer with which every mode (gs: Gauss-Seidel,
// else the setups and applications) gets the FC_SETS buffers the sweeps need
// (see fc_sweep.cuh); 0 if none.
int steps_per_buffer(const OrderedSweep& O, bool gs);

// The most rows of a step to try next when steps of at most `chunk` rows leave
// a mode too few stage buffers; 0: none.  Exchanged values and push targets
// are staged, up to 255 of each a row, so that wide steps of densely coupled
// rows do not fit; four rows always do (4 x 255 x (8 + 2 x 4) bytes a buffer).
inline int narrower_steps(int chunk) {
  if (chunk > FC_SET_ROWS) return std::max(FC_SET_ROWS, (3 * chunk / 4) & ~31);
  if (chunk > 32) return 32;
  return chunk > 4 ? std::max(4, chunk / 2) : 0;
}

}  // namespace fcdev
