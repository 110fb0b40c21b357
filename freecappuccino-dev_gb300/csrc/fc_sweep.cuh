// Schedule-ordered triangular sweeps of the DIC/DILU preconditioners
// (linear_solvers.f90:439-475, :613-683) and of Gauss-Seidel (:96-201).
//
// The system is renumbered in schedule order (fc_schedule.hpp): tile t is
// block t, and every step of a tile is a contiguous range of new rows.  What
// bounds a sweep is the chain of its levels: on a 128^3 hex mesh 382 levels
// follow each other, each with three dependent FP64 FMAs (64 cycles each on
// this part).  Everything else a step needs is therefore taken off that
// chain, by warps of three kinds:
//
//  - stager (one warp): per group of steps (four, fewer where the rows are
//    many) two or three bulk asynchronous copies (cp.async.bulk, the TMA
//    engine): the packed records of the group's steps (see below), the
//    right-hand-side window and, where the mode has one, the extra row
//    value, into a ring of K stage buffers.  Copies step by step, issued by
//    one thread, took longer than the steps themselves (520-580 cycles).
//  - importers (FC_IMP_WARPS warps, group g by warp g mod FC_IMP_WARPS): poll
//    the exchanged values of the group's steps in global memory until their
//    producers have stored them, put them into the stage buffer and the
//    sentinel back into the slots, and release each step once it has all of
//    its values.  A poll takes an L2 round trip, three to four steps; with a
//    whole group to a poll and three groups polled at once it delays a tile
//    once and not at every step.
//  - compute warps, FC_SETS sets of FC_SET_WARPS warps, one row per thread;
//    set s runs the steps s, s + FC_SETS, ...  A set loads its next step
//    (record, coefficients, right-hand side, where each dependency's value
//    will be) into registers while the other sets run theirs.  What remains
//    between two steps is: a named barrier (the set of step k-1 and the
//    importer of step k arrive, the set of step k waits), the ring loads, the
//    FMAs, the ring store.  The pushes to other tiles and the stores to memory
//    follow after the next set has been released.
//
// A stage buffer is handed over with two mbarriers: full (copies landed) and
// empty (the compute warps are done with its steps).  A wait names a phase by
// its parity, so it must come after the phase before it has completed and
// before the one after it does.  With at least FC_SETS buffers that holds for
// the sets (a set looks for step k after its own step k - FC_SETS and nobody
// refills the buffer without it) and for the stager, which waits for every
// group in order.  An importer of group g looks for group g - ahead (ahead <=
// K); what comes after cannot pass before it, as group g needs it, but what
// was before is only known to be complete with enough buffers.  With fewer,
// importers go by a word in which the stager counts the groups whose buffer it
// has found free (import_ahead and import_by_parity in fc_stage.hpp).
//
// Measured on a GB300, FP64, per level of one tile: 350 cycles forward with 30
// rows a level, 400 forward and 500 backward with 108 rows (the FP64 pipe
// takes 16-19 cycles per warp instruction: 4 x 3 FMAs forward, 4 x 5
// operations backward).  A one-role block that polled, staged and computed in
// turn took 1,950 cycles a step at every width; the forward sweep at 128^3
// went from 456 to 177 us on the same 152 tiles, ICCG to 1e-10 from 384 to
// 201 ms (157 with tiles cut at shared places, 132 with the passes below).
//
// Exchange: a value a row needs from another tile (or from more than R-1
// steps back) is pushed by its producer into the consumer's slot of the
// exchange array xv, whose slots start every sweep at a sentinel NaN.
//
// Arithmetic.  The setups (factors d_i, inverted as the reference does)
// and Gauss-Seidel use the reference's operations in its order.  The FP64
// applications solve the same triangular systems in scaled form: forward
// t_i = q_i - sum (a_ij d_j) t_j, where the reference's y_i is t_i d_i, and
// backward z_i = (d_i / (d_i + small)) d_i t_i - sum (a_ij d_i) z_j, with the
// bracketed factors formed once per solve.  That leaves three FMAs (the
// entries of a row) on a level's chain and no multiplication by d_i.  FP32
// FMAs take 4 cycles, so the FP32 applications keep the plain form.
#pragma once
#include <type_traits>
#include "fc_krylov.cuh"
#include "fc_stage.hpp"

static_assert(FC_SWEEP_BLOCK == 32 * (FC_SETS * FC_SET_WARPS + FC_IMP_WARPS + 1), "warp roles fill the block");

namespace fcdev {

// ------------------------------------------------- bulk copies, mbarriers
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned mb, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mb), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(unsigned mb, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned mb, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(mb), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(unsigned mb, unsigned count = 1) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(count) : "memory");
}
// global -> shared bulk copy of bytes (multiple of 16, both addresses
// 16-byte aligned), completion reported to mbarrier mb
__device__ __forceinline__ void bulk_g2s(unsigned dst, const void* src, unsigned bytes, unsigned mb) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mb)
               : "memory");
}
#define FC_MBAR_SPIN_LIMIT (1u << 22)
// bounded wait for the completion of phase `parity`; false if it ran out or
// the block is leaving.  backoff_ns > 0 sleeps between polls (a thread that
// is expected to wait long, so that it does not load the shared-memory pipe
// of the workers)
__device__ __forceinline__ bool mbar_wait(unsigned mb, unsigned parity, volatile int* abort_flag,
                                          unsigned backoff_ns = 0) {
  unsigned spins = 0;
  while (!mbar_try_wait(mb, parity)) {
    if (++spins > FC_MBAR_SPIN_LIMIT || ((spins & 15u) == 0 && abort_flag && *abort_flag)) return false;
    if (backoff_ns) __nanosleep(backoff_ns);
  }
  return true;
}
// the same for a whole warp: one lane polls (32 lanes polling one word take
// turns on it), the others wait for it
__device__ __forceinline__ bool mbar_wait_warp(unsigned mb, unsigned parity, volatile int* abort_flag) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait(mb, parity, abort_flag);
  ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
  __syncwarp();  // orders what follows in all lanes after lane 0's wait: the shuffle does not
  return ok;
}
// The word in which the stager counts the groups of a sweep whose buffer it
// has found free: written by one lane at a time, in order; a warp waits until it
// reaches count (bounded; false also if the block is leaving).  Sweeps take two
// words in turn, and the stager clears the other one, which nobody reads then.
__device__ __forceinline__ void word_publish(unsigned a, int count) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ bool word_wait_warp(unsigned a, int count, volatile int* abort_flag) {
  bool ok = true;
  if ((threadIdx.x & 31) == 0) {
    int v;
    unsigned spins = 0;
    for (;;) {
      asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
      if (v >= count) break;
      if (++spins > FC_MBAR_SPIN_LIMIT || ((spins & 15u) == 0 && *abort_flag)) { ok = false; break; }
      __nanosleep(20);
    }
  }
  ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
  __syncwarp();  // orders what follows in all lanes after lane 0's wait
  return ok;
}
__device__ __forceinline__ void bar_wait(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void bar_release(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// Shared memory by 32-bit address.  Volatile, so that they keep their place
// with respect to the barriers above.
__device__ __forceinline__ double lds(unsigned a, double) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float lds(unsigned a, float) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ int lds(unsigned a, int) {
  int v;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ int4 lds4(unsigned a) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// a value pushed to another tile: single-copy atomic, so that a poll sees the
// sentinel or the value
__device__ __forceinline__ void st_push(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void st_push(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// ------------------------------------------------------------------ views
// device copy of an OrderedSweep (fc_schedule.hpp)
struct OrdView {
  int n, nE, ntiles, R, novf0, novf1, nsteps;
  int nc;                                // coefficients of a record: 3, or FC_ELL where a row has more
  int gen;                               // rows of more than FC_ELL entries, or steps wider than FC_SET_ROWS
  int G;                                 // steps of a group (stage buffer): FC_SETS, 2 or 1
  int g_rows, g_padded, g_push, g_x;     // a group's most rows, padded rows, push targets, exchanged values
  // desc[d]: per step, where it lies in the stage buffer of its group (the
  // groups run downwards from the tile's last step backward): first row;
  // rows | push targets << 16; padded rows | push targets << 16 of the group's
  // steps before it in memory; its row in the windows | its first exchanged
  // value << 16
  int stage_area;                        // bytes of the stage area (multiple of 16)
  const int* __restrict__ tile_step_ptr;
  const int* __restrict__ step_ptr;
  const int* __restrict__ rp_ptr;
  const int* __restrict__ tile_W;
  const int* __restrict__ perm;
  const int4* __restrict__ rec[2];
  const int4* __restrict__ desc[2];
  const int* __restrict__ xv_ptr[2];
  const int* __restrict__ push_ptr[2];
  const int* __restrict__ ovf_ptr[2];
  const int* __restrict__ ovf_code[2];
  const int* __restrict__ ovf_col[2];
  const int* __restrict__ ovf_slot[2];
  const int* __restrict__ lo_tslot;
  const int* __restrict__ lo_ovf_tslot;
  // the matrix in slices of FC_SLICE rows: entry k (in the row's original
  // order) of row q at sell_ptr[q / FC_SLICE] + k FC_SLICE + q % FC_SLICE,
  // column and original slot -1 past the row's entries
  const int* __restrict__ sell_ptr;
  const int* __restrict__ sell_col;
  const int* __restrict__ sell_slot;
};
#define FC_SLICE 32
__device__ __forceinline__ int sell_at(const OrdView& O, int q, int k) {
  return __ldg(O.sell_ptr + q / FC_SLICE) + k * FC_SLICE + q % FC_SLICE;
}

// Per-solve values in the new numbering (gathered by the kernel from the
// caller's CSR values) and the exchange arrays; every vector of n rows is
// allocated with nE entries (the padding is read by the staging windows and
// never used).
//
// blob[d]: one block per step, the blocks of a tile's steps one after the
// other, so that a group of steps is copied in one piece.  A block holds the
// row records (16 bytes a row), the push targets, then the row values field
// by field (coefficients of entries 0..nc-1, then scaled: backward the factor
// of the right-hand side; plain: d_i and, backward, 1/(d_i + small)), the rows
// padded to a multiple of 4.  Records and targets are written when the array
// is allocated, the values by every solve.  Field by field because a warp
// then reads 32 consecutive values of a field without bank conflicts.
// sx, tx: per step (rows padded as in the blocks) a_ii, and the DILU
// transposes a_(j,i) of entries 0..nc-1.
template <class T>
struct OrdVals {
  unsigned char* blob[2];
  T* sx;
  T* tx;
  T* aovf[2];  // coefficients of the overflow entries
  T* tovf;     // DILU transposes of the lower overflow entries
  T* adiag;    // [nE]
  T* ap;       // matrix values in the slices of OrdView (0 past a row's entries)
  T* xv[2];    // exchange arrays (per-step blocks)
};

template <class T>
inline size_t osweep_smem_bytes(int R, size_t stage_area, int maxW) {
  return osweep_fixed_bytes<T>(R, maxW) + stage_area;
}

struct OsCtx {
  unsigned full, empty;       // shared addresses of the mbarriers, [FC_MAX_STAGES] each
  unsigned ring, stage;       // shared addresses
  int W, ncw;                 // the tile's widest step; compute warps of a set
  int s0, ns;                 // the tile's first step, its steps
  int* abort_flag;            // the stager's words after it
  unsigned parity;            // bit b: parity of the next use of stage buffer b; bit 31: of the next sweep
};

template <class T>
__device__ __forceinline__ OsCtx osweep_ctx(const OrdView& O, unsigned char* smem, int t) {
  OsCtx X;
  X.W = 1;
  X.s0 = X.ns = 0;
  if (t < O.ntiles) {
    X.W = __ldg(O.tile_W + t);
    X.s0 = __ldg(O.tile_step_ptr + t);
    X.ns = __ldg(O.tile_step_ptr + t + 1) - X.s0;
  }
  X.ncw = min(FC_SET_WARPS, (X.W + 31) >> 5);
  X.full = smem_addr(smem);
  X.empty = X.full + 8 * FC_MAX_STAGES;
  // carve with this tile's width; the host sized the area for the widest
  size_t off = FC_SMEM_HDR;
  X.ring = smem_addr(smem + off);
  off += (((size_t)O.R * X.W + 1) * sizeof(T) + 15) & ~(size_t)15;
  X.stage = smem_addr(smem + off);
  off += (size_t)O.stage_area;
  X.abort_flag = (int*)(smem + off);
  X.parity = 0;
  if (threadIdx.x == 0) {
    *X.abort_flag = 0;
    X.abort_flag[1] = X.abort_flag[2] = 0;
    for (int b = 0; b < FC_MAX_STAGES; ++b) {
      mbar_init(X.full + 8 * b, 1);
      mbar_init(X.empty + 8 * b, O.G * X.ncw);  // every step's warps
    }
    sts(X.ring + O.R * X.W * (unsigned)sizeof(T), T(0));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  return X;
}

// Row sources of a sweep.  q: the right-hand side (forward, backward,
// Gauss-Seidel), e: an extra row value (the dot partner of OS_BWD_DOT, the
// previous iterate of Gauss-Seidel), out: where the row values go.
template <class T>
struct OsIO {
  const T* q;
  const T* e;
  T* out;
};

// One row of a step between its loads and its result
template <class T>
struct OsRow {
  unsigned at[FC_ELL];  // shared address of each dependency's value
  T c[FC_ELL];          // coefficients (DIC: their squares)
  T x[FC_ELL];          // DILU: transposes; Gauss-Seidel: products of the upper entries
  T acc;                // right-hand side (setups: a_ii)
  T aii, xo;            // Gauss-Seidel: diagonal, previous iterate
  T di;                 // plain applications: d_i
  int push;             // push targets | place of the first << 8
  int ovf;              // last word of the record
};

// One ordered sweep of tile vg_bid(C).  Directions: forward over the lower
// triangle, backward over the upper one.  red (MODE OS_BWD_DOT: red[0] +=
// e*value; OS_GS: red[0] += |residual|, red[1] += |a_ii x_i|) accumulates
// per thread.  NC: values of a record's coefficients, GEN: the structure has
// rows of more than FC_ELL entries or steps wider than a set's threads.  Both
// are template parameters because every branch that is left on the chain
// counts: with the entry count, the overflow loop and the wide rows decided
// at run time a step took 490-560 cycles instead of 350-400 (a tile of 30 and
// one of 108 chains, forward), and more with the overflow loop inside.
// Every thread of the block calls it; it ends with a block barrier but no
// grid barrier, and returns false if a wait ran out.  A backward sweep may
// follow its forward sweep directly: it reads the forward values of its own
// tile only.  Not inlined: the solvers keep more state across a sweep than
// the sweep's own loop leaves registers for.
template <class T, int MODE, int NC, bool GEN, class TracerT>
__device__ __noinline__ bool osweep_tile(const GridCtl& C, const OrdView& O, const OrdVals<T>& V, const OsIO<T> io,
                                         OsCtx& Xr, double* red_out, TracerT* tr) {
  constexpr int dirn = (MODE == OS_BWD || MODE == OS_BWD_DOT) ? 1 : 0;
  constexpr bool kSetup = MODE == OS_SETUP_DIC || MODE == OS_SETUP_DILU;
  constexpr bool kE = MODE == OS_BWD_DOT || MODE == OS_GS;
  constexpr bool kGS = MODE == OS_GS;
  constexpr bool kScaled = ScaledApply<T>::value;
  constexpr int SZ = (int)sizeof(T);
  const OsCtx X = Xr;
  constexpr int nc = NC;
  const int ns = X.ns, R = O.R, G = O.G;
  const StageLayout L = StageLayout::of<T>(O, MODE);
  const int K = stages_in((size_t)O.stage_area, L.bytes);
  const int kshift = __ffs(K) - 1, gshift = __ffs(G) - 1;  // both powers of two
  T* const xv = V.xv[dirn];
  volatile int* const abort_flag = X.abort_flag;
  const unsigned free_word = smem_addr(X.abort_flag + 1 + (X.parity >> 31));
  const int lane = (int)threadIdx.x & 31, wid = (int)threadIdx.x >> 5;
  double red[2] = {0.0, 0.0};
  auto step_of = [&](int k) { return dirn ? ns - 1 - k : k; };
  // parity of the use of its buffer by group g
  auto use_parity = [&](int g) { return ((X.parity >> (g & (K - 1))) ^ (unsigned)(g >> kshift)) & 1u; };
  const int nth = 32 * X.ncw;  // threads of a set
  auto step_bar = [&](int k) { return 1 + k % FC_STEP_BARS; };
  auto step_bar_threads = [&](int k) { return (k > 0 ? 2 : 1) * nth + 32; };
  auto fail = [&]() {
    atomicCAS(C.status, 0, FC_ERR_TIMEOUT);
    *abort_flag = 1;
  };

  if (wid < FC_SETS * FC_SET_WARPS) {
    // ------------------------------------------------------------ compute
    const int set = wid / FC_SET_WARPS, sw = wid % FC_SET_WARPS;
    if (sw < X.ncw && set < ns) {
      // only the warps that the tile's widest step needs take part
      const int row0 = 32 * sw + lane;
      const int4* const desc = O.desc[dirn] + X.s0;
      const unsigned rw = (unsigned)(R * X.W);  // place of the zero
      constexpr int kStride = 16;               // bytes of a record
      const int rec_bytes = kStride + SZ * blob_fields<T>(nc, dirn);
      int4 next = __ldg(desc + step_of(set));
      int k = set;
      for (; k < ns; k += FC_SETS) {
        if (tr) tr->step(k);
        const int4 d = next;
        if (k + FC_SETS < ns) next = __ldg(desc + step_of(k + FC_SETS));
        const int g = k >> gshift, b = g & (K - 1);
        const int base = d.x, cnt = d.y & 0xFFFF, cp = (cnt + 3) & ~3, woff = d.w & 0xFFFF;
        const int rpo = d.z & 0xFFFF, ppo = (int)((unsigned)d.z >> 16);
        const unsigned S = X.stage + (unsigned)(b * L.bytes), B = S + (unsigned)(rpo * rec_bytes + 4 * ppo);
        const unsigned PS = B + kStride * cp;
        const unsigned CF = PS + 4 * ((unsigned)d.y >> 16);  // the step's values
        const unsigned I = S + L.oI + ((unsigned)d.w >> 16) * SZ - (rw + 1) * SZ;
        const unsigned ring_out = X.ring + (unsigned)((k & (R - 1)) * X.W * SZ);
        if (!mbar_wait_warp(X.full + 8 * b, use_parity(g), abort_flag)) break;
        if (tr) tr->waited(k);
        auto load = [&](int sl, OsRow<T>& w) {
          const int4 sr = lds4(B + kStride * sl);
          const unsigned cf = CF + (unsigned)(sl * SZ), cs = (unsigned)(cp * SZ);
#pragma unroll
          for (int e = 0; e < NC; ++e) w.c[e] = lds(cf + e * cs, T());
          w.push = sr.x;
          w.ovf = sr.w;
          const unsigned p01 = (unsigned)sr.y, p23 = (unsigned)sr.z;
          const unsigned place[FC_ELL] = {p01 & 0xFFFFu, p01 >> 16, p23 & 0xFFFFu, p23 >> 16};
#pragma unroll
          for (int e = 0; e < NC; ++e) w.at[e] = (place[e] <= rw ? X.ring : I) + place[e] * SZ;
          if constexpr (kSetup) {
            w.acc = lds(S + L.oX + (rpo + sl) * SZ, T());
#pragma unroll
            for (int e = 0; e < NC; ++e) {
              if (MODE == OS_SETUP_DILU) w.x[e] = lds(S + L.oT + (unsigned)((rpo * nc + e * cp + sl) * SZ), T());
              else w.c[e] = mul_rn(w.c[e], w.c[e]);
            }
          } else if constexpr (kGS) {
            w.acc = lds(S + L.oQ + (woff + sl) * SZ, T());
            w.aii = lds(S + L.oX + (rpo + sl) * SZ, T());
            w.xo = lds(S + L.oE + (woff + sl) * SZ, T());
            // the upper triangle's block of the same step
            const int s = X.s0 + k, p1 = __ldg(O.push_ptr[1] + s), p0 = __ldg(O.push_ptr[1] + X.s0 + (k & ~(G - 1)));
            const unsigned U = S + L.oU + (unsigned)(rpo * (kStride + SZ * blob_fields<T>(nc, 1)) + 4 * (p1 - p0));
            const unsigned UC = U + kStride * cp + 4 * (__ldg(O.push_ptr[1] + s + 1) - p1);
            const int nu = FC_REC_ENTRIES(lds(U + kStride * sl + 12, int())),
                      k0 = sell_at(O, base + sl, FC_REC_ENTRIES(w.ovf) + 1);
#pragma unroll
            for (int e = 0; e < NC; ++e)
              w.x[e] = e < nu ? mul_rn(lds(UC + (unsigned)((e * cp + sl) * SZ), T()), ldcg(io.e + __ldg(O.sell_col + k0 + FC_SLICE * e)))
                              : T(0);
          } else {
            w.acc = lds(S + L.oQ + (woff + sl) * SZ, T());
            if constexpr (!kScaled) w.di = lds(cf + nc * cs, T());
            if constexpr (dirn == 1) w.acc = w.acc * lds(cf + (nc + (kScaled ? 0 : 1)) * cs, T());
          }
        };
        // overflow entry e >= FC_ELL of a row: its value and coefficient; m
        // counts the row's exchanged entries
        auto dep_ovf = [&](const OsRow<T>& w, int q, int e, int& m, T& a) -> T {
          const int o = __ldg(O.ovf_ptr[dirn] + q) + e - FC_ELL;
          a = ldcg(V.aovf[dirn] + o);
          const int c = __ldg(O.ovf_code[dirn] + o);
          return lds(c >= 0 ? X.ring + c * SZ : I + (rw + 1 + FC_REC_OFFSET(w.ovf) + m++) * SZ, T());
        };
        // the row's value from its dependencies
        auto value = [&](int sl, OsRow<T>& w) {
          T v[NC];
#pragma unroll
          for (int e = 0; e < NC; ++e) v[e] = lds(w.at[e], T());
          int m = FC_REC_EXCHANGED(w.ovf);
          const int ne = GEN ? FC_REC_ENTRIES(w.ovf) : 0, q = base + sl;
          T val = w.acc;
          if constexpr (kSetup) {
            // d_i = a_ii - sum a_k^2 d_j (DIC) or a_k d_j a_(j,i) (DILU), then
            // 1/d_i; entries past the row's subtract an exact zero
#pragma unroll
            for (int e = 0; e < NC; ++e)
              val = MODE == OS_SETUP_DILU ? sub_rn(val, mul_rn(mul_rn(w.c[e], v[e]), w.x[e]))
                                          : sub_rn(val, mul_rn(w.c[e], v[e]));
            for (int e = FC_ELL; e < ne; ++e) {
              T a;
              const T dj = dep_ovf(w, q, e, m, a);
              const T at = MODE == OS_SETUP_DILU ? ldcg(V.tovf + __ldg(O.ovf_ptr[0] + q) + e - FC_ELL) : a;
              val = MODE == OS_SETUP_DILU ? sub_rn(val, mul_rn(mul_rn(a, dj), at)) : sub_rn(val, mul_rn(mul_rn(a, a), dj));
            }
            val = div_rn(T(1), val);
          }
          if constexpr (kGS) {
            // s = b - sum_{k<kd} a x_new - a_ii x_old_i - sum_{k>kd} a x_old;
            // x_i = x_old_i + s / (a_ii + small)   (exact arithmetic)
#pragma unroll
            for (int e = 0; e < NC; ++e) val = sub_rn(val, mul_rn(w.c[e], v[e]));
            for (int e = FC_ELL; e < ne; ++e) {
              T a;
              const T xj = dep_ovf(w, q, e, m, a);
              val = sub_rn(val, mul_rn(a, xj));
            }
            val = sub_rn(val, mul_rn(w.aii, w.xo));
#pragma unroll
            for (int e = 0; e < NC; ++e) val = sub_rn(val, w.x[e]);
            const int nu = GEN ? FC_REC_ENTRIES(__ldg(&O.rec[1][q].w)) : 0;
            for (int e = FC_ELL; e < nu; ++e) {
              const int o = __ldg(O.ovf_ptr[1] + q) + e - FC_ELL;
              val = sub_rn(val, mul_rn(ldcg(V.aovf[1] + o), ldcg(io.e + __ldg(O.ovf_col[1] + o))));
            }
            w.acc = val;
            val = add_rn(w.xo, div_rn(val, add_rn(w.aii, (T)FC_SMALL)));
          }
          if constexpr (!kSetup && !kGS) {
            // scaled: the nearest row's entry last (the last one forward, the
            // first one backward); plain: in the row's order
            if constexpr (dirn == 0 || !kScaled) {
#pragma unroll
              for (int e = 0; e < NC; ++e) val = fma(-w.c[e], v[e], val);
            }
            for (int e = FC_ELL; e < ne; ++e) {
              T a;
              const T x = dep_ovf(w, q, e, m, a);
              val = fma(-a, x, val);
            }
            if constexpr (dirn == 1 && kScaled) {
#pragma unroll
              for (int e = NC - 1; e >= 0; --e) val = fma(-w.c[e], v[e], val);
            }
            if constexpr (!kScaled) val = val * w.di;
          }
          return val;
        };
        // pushes, the result vector, the reductions
        auto store = [&](int sl, const OsRow<T>& w, T val) {
          const int np = w.push & 255;
          const unsigned ps = PS + 4 * ((unsigned)w.push >> 8);
          for (int m = 0; m < np; ++m) st_push(xv + lds(ps + 4 * m, int()), val);
          io.out[base + sl] = val;
          if constexpr (MODE == OS_BWD_DOT) red[0] += (double)lds(S + L.oE + (woff + sl) * SZ, T()) * (double)val;
          if constexpr (kGS) {
            red[0] += fabs((double)w.acc);
            red[1] += fabs((double)w.aii * (double)val);
          }
        };
        // threads past the step's rows repeat its last row up to the ring
        // store, so that nothing on the chain branches
        const int sl = min(row0, cnt - 1);
        OsRow<T> w;
        load(sl, w);
        if (tr) tr->at(k, 4, 0);
        const int bar = step_bar(k), bar1 = bar == FC_STEP_BARS ? 1 : bar + 1;
        __syncwarp();
        bar_wait(bar, step_bar_threads(k));
        if (tr) tr->at(k, 5, 0);
        T val = value(sl, w);
        if (row0 < cnt) sts(ring_out + row0 * SZ, val);
        if constexpr (GEN && !kGS) {
          if (cnt > nth)  // a step wider than a set's threads (forced widths only)
            for (int s2 = row0 + nth; s2 < cnt; s2 += nth) {
              OsRow<T> w2;
              load(s2, w2);
              const T v2 = value(s2, w2);
              sts(ring_out + s2 * SZ, v2);
              store(s2, w2, v2);
            }
        }
        if (tr) tr->at(k, 6, __double_as_longlong((double)val));
        __syncwarp();
        if (k + 1 < ns) bar_release(bar1, step_bar_threads(k + 1));
        if (row0 < cnt) store(row0, w, val);
        if (tr) tr->at(k, 7, 0);
        __syncwarp();
        if (lane == 0) mbar_arrive(X.empty + 8 * b);
      }
      if (k < ns) {
        // a wait for records ran out: only the barriers are kept up
        if (lane == 0) fail();
        for (; k < ns; k += FC_SETS) {
          __syncwarp();
          bar_wait(step_bar(k), step_bar_threads(k));
          if (k + 1 < ns) bar_release(step_bar(k + 1), step_bar_threads(k + 1));
        }
      }
    }
  } else if (wid < FC_SETS * FC_SET_WARPS + FC_IMP_WARPS) {
    // ----------------------------------------------------------- importers
    constexpr int U = 4;  // polls in flight per lane
    const int* const xp = O.xv_ptr[dirn] + X.s0;
    const int ng = (ns + G - 1) >> gshift, ahead = import_ahead(K, G);  // groups
    const bool by_parity = import_by_parity(K, G);
    bool ok = true;   // false: only the barriers are kept up
    for (int g = wid - FC_SETS * FC_SET_WARPS; g < ng; g += FC_IMP_WARPS) {
      const int k0 = g << gshift, k1 = min(k0 + G, ns), b = g & (K - 1);
      const int lo = dirn ? ns - k1 : k0, hi = dirn ? ns - k0 : k1;
      const int x0 = __ldg(xp + lo), nx = __ldg(xp + hi) - x0;
      const unsigned I = X.stage + (unsigned)(b * L.bytes + L.oI);
      // the values in the order of the steps: value i lies at place(i)
      auto place = [&](int i) { return dirn ? nx - 1 - i : i; };
      int rel = k0;  // next step to release
      // lane j: the values of step k0 + j end before value my_end
      int my_end = 0x7FFFFFFF;
      if (k0 + lane < k1) my_end = dirn ? nx - (__ldg(xp + ns - 1 - k0 - lane) - x0) : __ldg(xp + k0 + lane + 1) - x0;
      auto release = [&](int have) {  // the steps whose values are all among the first `have`
        while (rel < k1 && __shfl_sync(0xffffffffu, my_end, rel - k0) <= have) {
          bar_release(step_bar(rel), step_bar_threads(rel));
          ++rel;
        }
      };
      // the place of the values, and the barriers of the steps, are free once
      // group g - ahead is done
      if (ok && g >= ahead)
        ok = by_parity ? mbar_wait_warp(X.empty + 8 * ((g - ahead) & (K - 1)), use_parity(g - ahead), abort_flag)
                       : word_wait_warp(free_word, g + 1, abort_flag);
      if (ok) release(0);
      for (int c0 = 0; c0 < nx && ok; c0 += 32 * U) {
        unsigned pending = 0, spins = 0;
#pragma unroll
        for (int j = 0; j < U; ++j) pending |= (c0 + 32 * j + lane < nx ? 1u : 0u) << j;
        for (;;) {
          T v[U];
#pragma unroll
          for (int j = 0; j < U; ++j)
            v[j] = (pending >> j) & 1u ? Sentinel<T>::poll(xv + x0 + place(c0 + 32 * j + lane)) : Sentinel<T>::value();
#pragma unroll
          for (int j = 0; j < U; ++j) {
            if (Sentinel<T>::is(v[j])) continue;
            const int at = place(c0 + 32 * j + lane);
            sts(I + at * SZ, v[j]);
            st_push(xv + x0 + at, Sentinel<T>::value());
            pending &= ~(1u << j);
          }
          const unsigned first = pending ? (unsigned)(c0 + 32 * (__ffs(pending) - 1) + lane) : 0xFFFFFFFFu;
          const unsigned have = __reduce_min_sync(0xffffffffu, first);
          release(have == 0xFFFFFFFFu ? min(c0 + 32 * U, nx) : (int)have);
          if (have == 0xFFFFFFFFu) break;
          // the status word is in global memory: another block's failure is
          // looked for every 256 polls only
          if (++spins > FC_SPIN_LIMIT || *abort_flag || ((spins & 255u) == 0 && *((volatile int*)C.status) != 0)) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        // missing values only spoil numbers that an error status goes with
        if (lane == 0) fail();
        for (; rel < k1; ++rel) {
          __syncwarp();
          bar_wait(step_bar(rel), step_bar_threads(rel));
        }
      }
    }
  } else {
    // -------------------------------------------------------------- stager
    // each lane works out the copies of one group of the next 32 and issues
    // them in its turn.  The vectors were written by ordinary stores, the
    // copies are not ordinary loads.
    asm volatile("fence.proxy.async;" ::: "memory");
    const int ng = (ns + G - 1) >> gshift;
    const bool by_parity = import_by_parity(K, G);
    // also where this sweep does not use its own word: the next one may be of
    // another mode
    if (lane == 0) X.abort_flag[1 + ((X.parity >> 31) ^ 1u)] = 0;
    int issued = 0;
    bool ok = true;
    for (int g0 = 0; g0 < ng && ok; g0 += 32) {
      const int g = min(g0 + lane, ng - 1), k0 = g << gshift, k1 = min(k0 + G, ns);  // steps k0 .. k1-1
      const int lo = X.s0 + (dirn ? ns - k1 : k0), hi = X.s0 + (dirn ? ns - k0 : k1);
      const int r0 = __ldg(O.step_ptr + lo), r1 = __ldg(O.step_ptr + hi), b0 = r0 & ~3, nw = ((r1 + 3) & ~3) - b0;
      const int rp0 = __ldg(O.rp_ptr + lo), nr = __ldg(O.rp_ptr + hi) - rp0;
      const int p0 = __ldg(O.push_ptr[dirn] + lo), np = __ldg(O.push_ptr[dirn] + hi) - p0;
      const int nf = blob_fields<T>(nc, dirn);
      const unsigned S = X.stage + (unsigned)((g & (K - 1)) * L.bytes), mb = X.full + 8 * (g & (K - 1));
      const unsigned nB = (16 + SZ * nf) * nr + 4 * np, nX = SZ * nr, nT = SZ * nc * nr, nQ = SZ * nw;
      const unsigned char* const from = V.blob[dirn] + blob_offset<T>(rp0, p0, nf);
      unsigned bytes = nB;
      if (kSetup || kGS) bytes += nX;
      if (MODE == OS_SETUP_DILU) bytes += nT;
      if (!kSetup) bytes += nQ;
      if (kE) bytes += nQ;
      unsigned nU = 0;
      const unsigned char* fromU = nullptr;
      if constexpr (kGS) {
        const int u0 = __ldg(O.push_ptr[1] + lo), nu = __ldg(O.push_ptr[1] + hi) - u0;
        nU = (16 + SZ * blob_fields<T>(nc, 1)) * nr + 4 * nu;
        fromU = V.blob[1] + blob_offset<T>(rp0, u0, blob_fields<T>(nc, 1));
        bytes += nU;
      }
      const int turns = min(32, ng - g0);
      for (int j = 0; j < turns && ok; ++j) {
        if (lane == j) {
          if (g >= K && !mbar_wait(X.empty + 8 * (g & (K - 1)), use_parity(g) ^ 1u, abort_flag)) {
            fail();
            ok = false;
          } else {
            if (!by_parity) word_publish(free_word, g + 1);
            if (tr) tr->staged(k0);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive_tx(mb, bytes);
            bulk_g2s(S, from, nB, mb);
            if (kSetup || kGS) bulk_g2s(S + L.oX, V.sx + rp0, nX, mb);
            if (MODE == OS_SETUP_DILU) bulk_g2s(S + L.oT, V.tx + (size_t)rp0 * nc, nT, mb);
            if constexpr (kGS) bulk_g2s(S + L.oU, fromU, nU, mb);
            if (!kSetup) bulk_g2s(S + L.oQ, io.q + b0, nQ, mb);
            if (kE) bulk_g2s(S + L.oE, io.e + b0, nQ, mb);
            // the arrivals of the steps that the last group lacks
            if (k1 - k0 < G) mbar_arrive(X.empty + 8 * (g & (K - 1)), (G - (k1 - k0)) * X.ncw);
          }
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, j) != 0;
        if (!by_parity) __syncwarp();  // the next lane's word comes after this one's
        issued += ok ? 1 : 0;
      }
    }
    // after a failure, let the copies that nobody waits for land (bounded)
    // before the block leaves
    if (lane == 0 && *abort_flag)
      for (int g = max(0, issued - K); g < issued; ++g) mbar_wait(X.full + 8 * (g & (K - 1)), use_parity(g), nullptr);
  }
  __syncwarp();
  // the values written here may be read by the next sweep's copies
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  // every group used its buffer once
  {
    const int ng = (ns + G - 1) >> gshift, rounds = ng >> kshift, rest = ng & (K - 1);
    const unsigned all = (1u << K) - 1u, first = (1u << rest) - 1u;
    Xr.parity = X.parity ^ first ^ (rounds & 1 ? all : 0u) ^ 0x80000000u;
  }
  if (MODE == OS_BWD_DOT || kGS) red_out[0] += red[0];
  if (kGS) red_out[1] += red[1];
  if (*abort_flag) return false;
  if (tr) tr->step(ns);
  return true;
}

template <class T, int MODE, class TracerT = NoTrace>
__device__ __forceinline__ bool osweep(const GridCtl& C, const OrdView& O, const OrdVals<T>& V, const OsIO<T>& io,
                                       OsCtx& X, double* red, TracerT* tr = nullptr) {
  if (tr) tr->sweep();
  if (vg_bid(C) >= O.ntiles) return true;
  if (O.gen && O.nc == FC_ELL) return osweep_tile<T, MODE, FC_ELL, true, TracerT>(C, O, V, io, X, red, tr);
  if (O.gen) return osweep_tile<T, MODE, 3, true, TracerT>(C, O, V, io, X, red, tr);
  if (O.nc == FC_ELL) return osweep_tile<T, MODE, FC_ELL, false, TracerT>(C, O, V, io, X, red, tr);
  return osweep_tile<T, MODE, 3, false, TracerT>(C, O, V, io, X, red, tr);
}

// ------------------------------------------------------ gather / scatter
// Per-solve values in the new numbering from the caller's CSR values a
// (original entry slots), exchange arrays filled with the sentinel.  The
// blocks of the sweeps hold the plain coefficients of the lower triangle
// afterwards (gs: of both triangles).  A warp per step, so that a field of
// the step's rows is written in one piece; the caller ends the phase with a
// grid barrier.  A row's first FC_ROW_LOADS entries are read together, slots and
// then values, and serve the slices and the sweeps' fields: one entry after
// the other, and a second pass over all entries for the slices, left a warp
// waiting for one access at a time (128^3, FP64: 286 us, now 183).
#define FC_ROW_LOADS 8
template <class T>
__device__ void ord_gather_values(const GridCtl& C, const OrdView& O, const OrdVals<T>& V, const T* __restrict__ a,
                                  bool dilu, bool gs) {
  const int gt = vg_gt(C), G = vg_G(C), nc = O.nc, lane = threadIdx.x & 31;
  for (int s = gt >> 5; s < O.nsteps; s += G >> 5) {
    const int base = __ldg(O.step_ptr + s), cnt = __ldg(O.step_ptr + s + 1) - base, cp = (cnt + 3) & ~3;
    const int rp = __ldg(O.rp_ptr + s);
    T* cf[2];
    for (int d = 0; d < 2; ++d) {
      const int pp = __ldg(O.push_ptr[d] + s), np = __ldg(O.push_ptr[d] + s + 1) - pp;
      cf[d] = (T*)(V.blob[d] + blob_offset<T>(rp, pp, blob_fields<T>(nc, d)) + 16 * cp + 4 * np);
    }
    T *sx = V.sx + rp, *tx = V.tx + (size_t)rp * nc;
    for (int sl = lane; sl < cnt; sl += 32) {
      const int q = base + sl, slice = q / FC_SLICE, off = __ldg(O.sell_ptr + slice), k0 = off + q % FC_SLICE;
      const int w = (__ldg(O.sell_ptr + slice + 1) - off) / FC_SLICE;
      const int ne = FC_REC_ENTRIES(__ldg(&O.rec[0][q].w));
      auto slot_of = [&](int k) { return __ldg(O.sell_slot + k0 + FC_SLICE * k); };
      auto value_of = [&](int slot) { return slot >= 0 ? __ldg(a + slot) : T(0); };
      int slot[FC_ROW_LOADS], tslot[FC_ELL];
      T v[FC_ROW_LOADS], t[FC_ELL];
#pragma unroll
      for (int k = 0; k < FC_ROW_LOADS; ++k) slot[k] = k < w ? slot_of(k) : -1;
#pragma unroll
      for (int e = 0; e < FC_ELL; ++e)
        tslot[e] = dilu && e < nc && e < ne ? __ldg(O.lo_tslot + (size_t)e * O.nE + q) : -1;
#pragma unroll
      for (int k = 0; k < FC_ROW_LOADS; ++k) v[k] = value_of(slot[k]);
#pragma unroll
      for (int e = 0; e < FC_ELL; ++e) t[e] = value_of(tslot[e]);
      T aii = T(0);
#pragma unroll
      for (int k = 0; k < FC_ROW_LOADS; ++k) {
        if (k < w) V.ap[k0 + FC_SLICE * k] = v[k];
        if (k == ne) aii = v[k];
      }
      for (int k = FC_ROW_LOADS; k < w; ++k) {
        const T vk = value_of(slot_of(k));
        V.ap[k0 + FC_SLICE * k] = vk;
        if (k == ne) aii = vk;
      }
      V.adiag[q] = aii;
      sx[sl] = aii;
#pragma unroll
      for (int e = 0; e < FC_ELL; ++e)
        if (e < nc) {
          cf[0][e * cp + sl] = e < ne ? v[e] : T(0);
          if (dilu) tx[e * cp + sl] = t[e];
        }
      if (gs) {
        const int nu = FC_REC_ENTRIES(__ldg(&O.rec[1][q].w));
        for (int e = 0; e < nc; ++e) cf[1][e * cp + sl] = e < nu ? value_of(slot_of(ne + 1 + e)) : T(0);
      }
    }
  }
  for (int d = 0; d < 2; ++d) {
    const int novf = d ? O.novf1 : O.novf0;
    for (int o = gt; o < novf; o += G) {
      V.aovf[d][o] = __ldg(a + __ldg(O.ovf_slot[d] + o));
      if (d == 0 && dilu) V.tovf[o] = __ldg(a + __ldg(O.lo_ovf_tslot + o));
    }
  }
}

// exchange slots to the sentinel (every solve: an earlier one may have been cut short)
template <class T>
__device__ __forceinline__ void ord_reset_exchange(const GridCtl& C, const OrdView& O, const OrdVals<T>& V) {
  for (int d = 0; d < 2; ++d) {
    const int nx = __ldg(O.xv_ptr[d] + O.nsteps);
    for (int p = vg_gt(C); p < nx; p += vg_G(C)) V.xv[d][p] = Sentinel<T>::value();
  }
}

// The row values of the applications from the factors d (see the file
// header).  Scaled: forward a_ij d_j, backward a_ij d_i and the factor
// (d_i / (d_i + small)) d_i of the right-hand side.  Plain: d_i in both
// directions, backward a_ij and 1/(d_i + small).  Once per setup; the caller
// ends the phase with a grid barrier.  All loads of a row are issued before its
// first use, and d_i / (d_i + small) is divided only where small counts (else
// it is 1; the FP64 pipe takes 12 instructions for a division): 128^3 142 us,
// now 86.
template <class T>
__device__ void ord_apply_values(const GridCtl& C, const OrdView& O, const OrdVals<T>& V, const T* d) {
  const int gt = vg_gt(C), G = vg_G(C), nc = O.nc, lane = threadIdx.x & 31;
  for (int s = gt >> 5; s < O.nsteps; s += G >> 5) {
    const int base = __ldg(O.step_ptr + s), cnt = __ldg(O.step_ptr + s + 1) - base, cp = (cnt + 3) & ~3;
    const int rp = __ldg(O.rp_ptr + s);
    T* cf[2];
    for (int r = 0; r < 2; ++r) {
      const int pp = __ldg(O.push_ptr[r] + s), np = __ldg(O.push_ptr[r] + s + 1) - pp;
      cf[r] = (T*)(V.blob[r] + blob_offset<T>(rp, pp, blob_fields<T>(nc, r)) + 16 * cp + 4 * np);
    }
    for (int sl = lane; sl < cnt; sl += 32) {
      const int q = base + sl, k0 = sell_at(O, q, 0);
      auto entry = [&](int k) { return ldcg(V.ap + k0 + FC_SLICE * k); };
      auto column = [&](int k) { return __ldg(O.sell_col + k0 + FC_SLICE * k); };
      const int ne = FC_REC_ENTRIES(__ldg(&O.rec[0][q].w)), nu = FC_REC_ENTRIES(__ldg(&O.rec[1][q].w));
      const T di = ldcg(d + q);
      T lo[FC_ELL], up[FC_ELL], dj[FC_ELL];
      int col[FC_ELL];
#pragma unroll
      for (int e = 0; e < FC_ELL; ++e) {
        const bool l = ScaledApply<T>::value && e < nc && e < ne;
        lo[e] = l ? entry(e) : T(0);
        col[e] = l ? column(e) : -1;
        up[e] = e < nc && e < nu ? entry(ne + 1 + e) : T(0);
      }
#pragma unroll
      for (int e = 0; e < FC_ELL; ++e) dj[e] = col[e] >= 0 ? ldcg(d + col[e]) : T(0);
      if constexpr (ScaledApply<T>::value) {
#pragma unroll
        for (int e = 0; e < FC_ELL; ++e)
          if (e < nc) {
            cf[0][e * cp + sl] = col[e] >= 0 ? lo[e] * dj[e] : T(0);
            cf[1][e * cp + sl] = e < nu ? up[e] * di : T(0);
          }
        const T ds = di + (T)FC_SMALL;
        cf[1][nc * cp + sl] = ds == di && !isinf(di) ? di : di / ds * di;
        for (int e = FC_ELL; e < ne; ++e)
          V.aovf[0][__ldg(O.ovf_ptr[0] + q) + e - FC_ELL] = entry(e) * ldcg(d + column(e));
        for (int e = FC_ELL; e < nu; ++e)
          V.aovf[1][__ldg(O.ovf_ptr[1] + q) + e - FC_ELL] = entry(ne + 1 + e) * di;
      } else {
        cf[0][nc * cp + sl] = di;
#pragma unroll
        for (int e = 0; e < FC_ELL; ++e)
          if (e < nc) cf[1][e * cp + sl] = up[e];
        cf[1][nc * cp + sl] = di;
        cf[1][(nc + 1) * cp + sl] = T(1) / (di + (T)FC_SMALL);
      }
    }
  }
}

// y[q] = src[perm[q]] (into the new numbering) / dst[perm[q]] = y[q]
template <class T, class U>
__device__ __forceinline__ void ord_gather_vec(const GridCtl& C, const OrdView& O, const U* __restrict__ src, T* y) {
  for (int q = vg_gt(C); q < O.n; q += vg_G(C))
    y[q] = (T)ldcg(src + __ldg(O.perm + q));
}
template <class T, class U>
__device__ __forceinline__ void ord_scatter_vec(const GridCtl& C, const OrdView& O, const T* y, U* dst) {
  for (int q = vg_gt(C); q < O.n; q += vg_G(C))
    dst[__ldg(O.perm + q)] = (U)ldcg(y + q);
}

// Row products in the new numbering, FMA accumulation in the row's original
// entry order (as ax_cr / the residual loops of the reference): done(q, s, w_q)
// gets s = sum a_k x_k of every row, or NEG w_q - sum a_k x_k.  A warp per slice:
// columns and values of all entries are loaded before any is used, then the
// gathers, then the FMAs, so that a warp waits for memory twice and not once
// per entry; the next slice's place and the row's own value are loaded
// ahead.  x is read through L1 (the three neighbours of one level share lines),
// the matrix past it.  W: the slice's width (hexes 7, tetrahedra 5), 0: any.
// Bound by the latency of the loads at 20 warps an SM: 128^3 in natural order
// 56 us, with the loads ahead 50, on twice the warps 40; the traffic alone 34.
template <class T, bool NEG, int W>
__device__ __forceinline__ T sell_row(const OrdView& O, const T* __restrict__ ap, const T* x, int at, int w, T s) {
  if constexpr (W > 0) {
    int c[W];
    T a[W], v[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      c[k] = ldcg(O.sell_col + at + FC_SLICE * k);
      a[k] = ldcg(ap + at + FC_SLICE * k);
    }
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] = c[k] >= 0 ? x[c[k]] : T(0);
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (c[k] >= 0) s = fma(NEG ? -a[k] : a[k], v[k], s);
  } else {
    for (int k = 0; k < w; ++k) {
      const int c = ldcg(O.sell_col + at + FC_SLICE * k);
      if (c < 0) break;
      const T a = ldcg(ap + at + FC_SLICE * k);
      s = fma(NEG ? -a : a, x[c], s);
    }
  }
  return s;
}
template <class T, bool NEG, class Done>
__device__ __forceinline__ void ord_rows(const GridCtl& C, const OrdView& O, const T* __restrict__ ap, const T* x,
                                         const T* w, Done done) {
  const int lane = threadIdx.x & 31, ns = (O.n + FC_SLICE - 1) / FC_SLICE, step = vg_G(C) >> 5;
  int sl = vg_gt(C) >> 5, off = 0, end = 0;
  if (sl < ns) { off = __ldg(O.sell_ptr + sl); end = __ldg(O.sell_ptr + sl + 1); }
  for (; sl < ns; sl += step) {
    int off1 = 0, end1 = 0;
    if (sl + step < ns) { off1 = __ldg(O.sell_ptr + sl + step); end1 = __ldg(O.sell_ptr + sl + step + 1); }
    const int width = (end - off) / FC_SLICE, q = sl * FC_SLICE + lane, at = off + lane;
    const T own = q < O.n ? ldcg(w + q) : T(0);
    T s = NEG ? own : T(0);
    if (width == 7) s = sell_row<T, NEG, 7>(O, ap, x, at, width, s);
    else if (width == 5) s = sell_row<T, NEG, 5>(O, ap, x, at, width, s);
    else s = sell_row<T, NEG, 0>(O, ap, x, at, width, s);
    if (q < O.n) done(q, s, own);
    off = off1;
    end = end1;
  }
}

// Element-wise passes over vectors of n values (16-byte aligned): f(e, i) gets
// the values e[0..NV) of element i and may change them; bit j of STORE: v[j]
// is written back.  16-byte accesses, two of them per vector in flight a
// thread: with one 8-byte access each the 20 warps of an SM do not have
// enough bytes under way for the HBM bandwidth.
template <class T>
struct alignas(16) VecPack {
  static constexpr int N = 16 / sizeof(T);
  T v[N];
};
template <unsigned STORE, class T, int NV, class F>
__device__ __forceinline__ void vec_map(const GridCtl& C, int n, T* const (&v)[NV], F f) {
  using P = VecPack<T>;
  const int gt = vg_gt(C), G = vg_G(C), np = n / P::N;
  for (int i = gt; i < np; i += 2 * G) {
    P a[2][NV];
    const bool two = i + G < np;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const float4 t = __ldcg((const float4*)v[j] + i);
      a[0][j] = *(const P*)&t;
    }
    if (two)
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const float4 t = __ldcg((const float4*)v[j] + i + G);
        a[1][j] = *(const P*)&t;
      }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 && !two) break;
#pragma unroll
      for (int m = 0; m < P::N; ++m) {
        T e[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) e[j] = a[u][j].v[m];
        f(e, (i + u * G) * P::N + m);
#pragma unroll
        for (int j = 0; j < NV; ++j)
          if ((STORE >> j) & 1u) a[u][j].v[m] = e[j];
      }
#pragma unroll
      for (int j = 0; j < NV; ++j)
        if ((STORE >> j) & 1u) ((float4*)v[j])[i + u * G] = *(const float4*)&a[u][j];
    }
  }
  for (int i = np * P::N + gt; i < n; i += G) {
    T e[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) e[j] = ldcg(v[j] + i);
    f(e, i);
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if ((STORE >> j) & 1u) v[j][i] = e[j];
  }
}

}  // namespace fcdev
