// Device building blocks of the persistent Krylov kernels: a bounded grid
// barrier, deterministic grid reductions, exact-rounding arithmetic, the
// sentinel used by the sweeps' value exchange and CSR row products.  The
// triangular sweeps themselves are in fc_sweep.cuh.  Kernels using these are launched cooperatively (one grid of
// co-resident blocks), so the barrier cannot deadlock; every wait is still
// bounded and reports FC_ERR_TIMEOUT instead of hanging.
//
// Memory rule inside these kernels: immutable inputs (ia, ja, a, level
// lists) go through the read-only path; vectors written during the kernel by
// other blocks are read with ld.global.cg (L2, coherent across SMs).
#pragma once
#include <cuda_runtime.h>

#include "fc_internal.hpp"

#define FC_BLOCK 512
// block of the kernels with ordered sweeps: 16 compute, 3 import and 1 staging
// warp (fc_sweep.cuh)
#define FC_SWEEP_BLOCK 640
#define FC_SPIN_LIMIT (1u << 24)

namespace fcdev {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// p = p >= limit ? 0 : p + 1; returns the old value
__device__ __forceinline__ unsigned atom_inc_acqrel_u32(unsigned* p, unsigned limit) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.inc.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(limit) : "memory");
  return old;
}

template <class T> __device__ __forceinline__ T ldcg(const T* p) { return __ldcg(p); }

// Block index, block count and grid-stride start/step within the group of
// blocks the kernel runs on (the launch grid unless GridCtl names a group).
__device__ __forceinline__ int vg_bid(const GridCtl& C) { return (int)blockIdx.x - C.base; }
__device__ __forceinline__ int vg_nb(const GridCtl& C) { return C.nb > 0 ? C.nb : (int)gridDim.x; }
__device__ __forceinline__ int vg_gt(const GridCtl& C) { return vg_bid(C) * (int)blockDim.x + (int)threadIdx.x; }
__device__ __forceinline__ int vg_G(const GridCtl& C) { return vg_nb(C) * (int)blockDim.x; }

// Barrier over all blocks of the (cooperative) grid or group.  Returns false
// if the wait ran out or another block already failed; the caller then leaves
// the kernel.  One counter: the arrivals of a round take it from a multiple of
// nb to the next (it wraps at a multiple, so the difference to the round's
// start tells).  A block arrives and polls with one atomic and then loads of
// one word; a separate generation word, read before the arrival, and fences
// around the acquire-release operations cost another round trip each
// (2.8 us a barrier with 152 blocks, now 1.3).  The counter is zeroed before
// the launch.
__device__ __forceinline__ bool grid_sync(const GridCtl& C) {
  __shared__ int s_ok;
  __syncthreads();
  const unsigned nb = (unsigned)vg_nb(C);
  if (nb == 1) return true;
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned old = atom_inc_acqrel_u32(C.bar, nb * (1u << 16) - 1u), start = old - old % nb;
    unsigned spins = 0;
    while (ld_acquire_u32(C.bar) - start < nb) {
      if (++spins > FC_SPIN_LIMIT || ((spins & 63u) == 0 && *((volatile int*)C.status) != 0)) {
        atomicCAS(C.status, 0, FC_ERR_TIMEOUT);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum NV values over the grid.  Deterministic: each block sums in a fixed
// order and writes one partial per value; after the barrier every block sums
// the partials in the same fixed order, so all blocks hold identical totals.
// Partials alternate between two slot sets (ph), so a block still reading
// the previous reduction never sees slots of the next one being rewritten.
//
// A block's threads leave their values in shared memory and one warp per value
// sums them, four chains a lane, then a tree: the FP64 pipe takes a warp's
// addition each ~17 cycles, and a shuffle tree in each of 20 warps was 100
// of them per value (2 values on 152 blocks: 5.8 us with the trees, now 3.4;
// the barrier alone 1.3).
__device__ __forceinline__ double* red_buf() {
  __shared__ double sm[FC_NPART * FC_SWEEP_BLOCK];
  return sm;
}
template <int NV>
__device__ __forceinline__ bool grid_reduce(const GridCtl& C, int& ph, double (&v)[NV]) {
  static_assert(NV <= FC_NPART, "partial slots");
  __shared__ double tot[NV];
  const int tid = threadIdx.x, lane = tid & 31, j = tid >> 5, bd = blockDim.x;
  const int nb = vg_nb(C), bid = vg_bid(C);
  double* sm = red_buf();
  double* part = C.part + (size_t)(ph & 1) * FC_NPART * nb;
  ++ph;
#pragma unroll
  for (int k = 0; k < NV; ++k) sm[k * bd + tid] = v[k];
  __syncthreads();
  if (j < NV) {
    double e[4] = {0.0, 0.0, 0.0, 0.0};
    for (int t = lane; t < bd; t += 128)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (t + 32 * k < bd) e[k] += sm[j * bd + t + 32 * k];
    const double s = warp_sum((e[0] + e[1]) + (e[2] + e[3]));
    if (lane == 0) {
      if (nb == 1) tot[j] = s;
      else part[j * nb + bid] = s;
    }
  }
  if (nb > 1) {
    if (!grid_sync(C)) return false;
    if (j < NV) {
      double e[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) e[k] = lane + 32 * k < nb ? __ldcg(part + j * nb + lane + 32 * k) : 0.0;
      double s = ((e[0] + e[1]) + (e[2] + e[3])) + e[4];
      for (int b = lane + 160; b < nb; b += 32) s += __ldcg(part + j * nb + b);
      s = warp_sum(s);
      if (lane == 0) tot[j] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = tot[k];
  return true;
}

// exact-rounding arithmetic for the recurrences (no FMA contraction), so the
// DIC/DILU factors and sweeps reproduce the reference bit for bit in FP64
template <class T> __device__ __forceinline__ T mul_rn(T a, T b);
template <class T> __device__ __forceinline__ T sub_rn(T a, T b);
template <class T> __device__ __forceinline__ T add_rn(T a, T b);
template <class T> __device__ __forceinline__ T div_rn(T a, T b);
template <> __device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
template <> __device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }
template <> __device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
template <> __device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }

// Original-order CSR view (DPCG, residuals, the ILU(0) kernels of GMRES)
template <class T>
struct CsrView {
  int n;
  const int* __restrict__ ia;
  const int* __restrict__ ja;
  const int* __restrict__ dg;
  const int* __restrict__ ts;    // transpose slot (DILU)
  const T* __restrict__ a;
  const int* __restrict__ lfp;   // level sets (used by the ILU(0) kernels)
  const int* __restrict__ lfr;
  int nlf;
  const int* __restrict__ lbp;
  const int* __restrict__ lbr;
  int nlb;
};

// Exchange slots of the sweeps start filled with a sentinel NaN (a payload no
// arithmetic produces); a value pushed by another tile is read by polling the
// slot until the sentinel is gone.  A 64-bit (32-bit) store is single-copy
// atomic, so the reader sees either the sentinel or the final value and no
// fence or progress flag is needed between tiles.
template <class T> struct Sentinel;
template <> struct Sentinel<double> {
  static __device__ __forceinline__ double value() { return __longlong_as_double(0x7FF4DEADBEEF0001LL); }
  static __device__ __forceinline__ bool is(double v) { return __double_as_longlong(v) == 0x7FF4DEADBEEF0001LL; }
  static __device__ __forceinline__ double poll(const double* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double((long long)v);
  }
};
template <> struct Sentinel<float> {
  static __device__ __forceinline__ float value() { return __int_as_float(0x7FA5DEAD); }
  static __device__ __forceinline__ bool is(float v) { return __float_as_int(v) == 0x7FA5DEAD; }
  static __device__ __forceinline__ float poll(const float* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return __int_as_float((int)v);
  }
};

// Cycle tracing hooks (no-ops unless a kernel is instantiated with a real
// tracer): mark(phase) closes a phase, sweep() opens a sweep, step(k) stamps
// the start of the tile's k-th step.
struct NoTrace {
  __device__ __forceinline__ void mark(int) {}
  __device__ __forceinline__ void sweep() {}
  __device__ __forceinline__ void step(int) {}
  __device__ __forceinline__ void waited(int) {}
  __device__ __forceinline__ void staged(int) {}
  template <class V> __device__ __forceinline__ void at(int, int, V) {}
};

// sum_k a_k x_j over row i (FMA accumulation, CSR order)
template <class T>
__device__ __forceinline__ T row_dot(const CsrView<T>& S, const T* x, int i) {
  const int k0 = __ldg(S.ia + i), k1 = __ldg(S.ia + i + 1);
  T s = T(0);
  for (int k = k0; k < k1; ++k) s = fma(__ldg(S.a + k), ldcg(x + __ldg(S.ja + k)), s);
  return s;
}

// rhs_i - sum_k a_k x_j over row i (the reference's residual loop order)
template <class T>
__device__ __forceinline__ T row_residual(const CsrView<T>& S, const T* x, T bi, int i) {
  const int k0 = __ldg(S.ia + i), k1 = __ldg(S.ia + i + 1);
  T s = bi;
  for (int k = k0; k < k1; ++k) s = fma(-__ldg(S.a + k), ldcg(x + __ldg(S.ja + k)), s);
  return s;
}

}  // namespace fcdev
