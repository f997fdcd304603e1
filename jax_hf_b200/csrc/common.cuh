// Shared device/host helpers for the hf_b200 CUDA library (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include <string>

#include "../../include/hf_b200.h"

namespace hf {

// ---------------------------------------------------------------- errors ----
void set_error(const std::string& msg);
int fail(int status, const std::string& msg);
int cuda_check(cudaError_t e, const char* what);
int allow_max_dynamic_smem(const void* fn);
int context_id(unsigned long long* id);
int resident_ctas(const void* fn, int threads, size_t smem, int csize, int* out);
// Slot-indexed DIIS steps for the device-resident SCF loop (ops.cu): the history slot is
// a device int, so one captured iteration serves every slot
int scf_residuals_slot(void* stream, int nk, int nb, const void* F, const void* P, const void* Pn, const double* w,
                       void* R, size_t stride, const int* slot, void* delta, double* sums3, void* ws);
int copy_to_slot(void* stream, size_t n, const void* x, void* hist, const int* slot);
// n <= 4 inner products of hf_jdot's form in one pass, each equal to hf_jdot's (ops.cu)
int jdot_multi(void* stream, size_t nk, int nb, int n, const void* const* aX, const void* const* bX,
               const double* const* wX, const double* const* ap, const double* const* bp, const double* const* wp,
               double* out, void* ws);
int gram_row_slot(void* stream, int n, const int* slot, size_t stride, int nk, int nb, const void* R,
                  const double* w, double* b_out, void* ws);
// eigh of herm(A) (mode 0) or herm(i A) (mode 1), nb <= 16, ascending, by
// tridiagonalisation and QR (eigh.cu); eps and V in A's precision
int eigh_tri(void* stream, int dtype, int nk, int nb, const void* A, void* eps, void* V, int mode);
// P = herm(Q diag(p) Q^H), complex128, nb <= 8, lane-per-column kernel (solver_cg.cu)
int rows_density(void* stream, int nk, int nb, const void* Q, const double* p, void* P);
int symbol_address(const void* symbol, void** out);

#define HF_SMEM_CAP(...)                                              \
  do {                                                                \
    const int _st = ::hf::allow_max_dynamic_smem((const void*)(__VA_ARGS__));  \
    if (_st) return _st;                                              \
  } while (0)

#define HF_CUDA(call)                                            \
  do {                                                           \
    cudaError_t _e = (call);                                     \
    if (_e != cudaSuccess) return ::hf::cuda_check(_e, #call);   \
  } while (0)

#define HF_LAUNCH_CHECK(what)                                    \
  do {                                                           \
    cudaError_t _e = cudaGetLastError();                         \
    if (_e != cudaSuccess) return ::hf::cuda_check(_e, what);    \
  } while (0)

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// --------------------------------------------------------------- complex ----
template <typename T> struct Cpx;
template <> struct Cpx<double> { using type = double2; };
template <> struct Cpx<float> { using type = float2; };
template <typename T> using cpx_t = typename Cpx<T>::type;

template <typename C> __host__ __device__ __forceinline__ C mk(double x, double y) {
  C r; r.x = x; r.y = y; return r;
}
template <typename C, typename T> __host__ __device__ __forceinline__ C make_c(T x, T y) {
  C r; r.x = x; r.y = y; return r;
}
__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__host__ __device__ __forceinline__ double2 cmulc(double2 a, double2 b) {
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__host__ __device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__host__ __device__ __forceinline__ double2 conj(double2 a) { return make_double2(a.x, -a.y); }
__host__ __device__ __forceinline__ float2 conj(float2 a) { return make_float2(a.x, -a.y); }
__host__ __device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// multiply by -i (forward) / +i
__host__ __device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }
__host__ __device__ __forceinline__ float2 mul_mi(float2 a) { return make_float2(a.y, -a.x); }
__host__ __device__ __forceinline__ double2 mul_pi(double2 a) { return make_double2(-a.y, a.x); }
__host__ __device__ __forceinline__ float2 mul_pi(float2 a) { return make_float2(-a.y, a.x); }

// acc + a*b, acc + conj(a)*b, acc + a*conj(b)
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 acc) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
  return acc;
}
__device__ __forceinline__ double2 cfma_cj(double2 a, double2 b, double2 acc) {
  acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
  return acc;
}
__device__ __forceinline__ double2 cfma_c(double2 a, double2 b, double2 acc) {
  acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(a.y, b.x, fma(-a.x, b.y, acc.y));
  return acc;
}

// 1 / sqrt(x) and 1 / x for serial chains, for arguments well inside the range of normal
// numbers: the hardware's approximate seed and one step of third order
// (Householder's iteration), four and three dependent FP64 operations, errors of about
// one ulp.
__device__ __forceinline__ double rsqrt_seeded(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double recip_seeded(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
template <typename To, typename From> __device__ __forceinline__ To cvt(From a) {
  To r; r.x = a.x; r.y = a.y; return r;
}

// ------------------------------------------------- compensated summation ----
// Neumaier (1974) running sum: s + c carries the exact sum of the added terms
// to within O(eps^2) relative error, independent of the number of terms.
struct KSum {
  double s, c;
  __device__ __forceinline__ KSum() : s(0.0), c(0.0) {}
  __device__ __forceinline__ void add(double x) {
    double t = s + x;
    if (fabs(s) >= fabs(x)) c += (s - t) + x; else c += (x - t) + s;
    s = t;
  }
  __device__ __forceinline__ void merge(const KSum& o) { add(o.s); add(o.c); }
  __device__ __forceinline__ double value() const { return s + c; }
};

__device__ __forceinline__ KSum warp_reduce(KSum v) {
  for (int off = 16; off > 0; off >>= 1) {
    KSum o;
    o.s = __shfl_xor_sync(0xffffffffu, v.s, off);
    o.c = __shfl_xor_sync(0xffffffffu, v.c, off);
    v.merge(o);
  }
  return v;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// Block-wide compensated reduction; result valid in thread 0.  `sm` needs
// 2*32 doubles.  Deterministic for a fixed launch shape.
__device__ __forceinline__ KSum block_reduce(KSum v, double* sm) {
  v = warp_reduce(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) { sm[2 * wid] = v.s; sm[2 * wid + 1] = v.c; }
  __syncthreads();
  KSum r;
  if (wid == 0) {
    if (lane < nw) { r.s = sm[2 * lane]; r.c = sm[2 * lane + 1]; }
    r = warp_reduce(r);
  }
  return r;
}

// Block-wide compensated sums of NS quantities (block_reduce on each, the same trees), side by
// side: a compensated merge is a chain of ten dependent additions, so one quantity after the
// other left the block waiting 2 NS times.  The warps' results go through shared memory once,
// and warp w finishes quantities w, w + nw, ...  sink(q, sums of quantity q) runs in lane 0 of
// warp q % nw; call with every thread of a block of at most 256.
template <int NS, class Sink>
__device__ __forceinline__ void block_reduce_all(KSum (&acc)[NS], Sink&& sink) {
  constexpr int MW = 8;  // warps per block at most (256 threads)
  __shared__ double2 part[NS][MW];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      KSum o;
      o.s = __shfl_xor_sync(0xffffffffu, acc[q].s, off);
      o.c = __shfl_xor_sync(0xffffffffu, acc[q].c, off);
      acc[q].merge(o);
    }
  }
  __syncthreads();  // the previous use of part
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NS; ++q) part[q][wid] = make_double2(acc[q].s, acc[q].c);
  }
  __syncthreads();
  for (int q = wid; q < NS; q += nw) {
    KSum r;
    if (lane < nw) {
      r.s = part[q][lane].x;
      r.c = part[q][lane].y;
    }
    for (int off = MW / 2; off > 0; off >>= 1) {  // the lanes from 8 on hold zeros, which change nothing
      KSum o;
      o.s = __shfl_xor_sync(0xffffffffu, r.s, off);
      o.c = __shfl_xor_sync(0xffffffffu, r.c, off);
      r.merge(o);
    }
    if (lane == 0) sink(q, r);
  }
}

// ------------------------------------------------ programmatic dependent launch ----
// griddepcontrol.wait: the grids before this one have completed and their writes are
// visible (without the launch attribute it returns at once); launch_dependents lets the
// next grid take its place on the SMs once every CTA of this one has got here.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// First statement of every kernel that launch_pdl launches, ahead of any early return: a grid that
// ended without waiting would let its successor start before its predecessor ended.  No parameter
// of such a kernel is __restrict__, since its predecessor may still be at that memory.
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_launch_dependents();
}

// Launches a kernel that starts with pdl_begin() so that its launch overlaps the end of the
// one before it: the loops of the solvers are chains of kernels of a few microseconds, and
// a plain launch in such a chain costs 1 to 1.5 us of idle GPU.  Errors are left for
// HF_LAUNCH_CHECK.
template <typename... P, typename... A>
inline void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace hf
