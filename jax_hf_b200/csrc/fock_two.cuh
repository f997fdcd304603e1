// Fock-build passes for mesh sides that are a product of two factors of at most 16
// (every composite side up to 256 without a prime factor above 13; 25, 49, 75, 90, 100,
// 120, ...) and have no compile-time line shape of their own, and for 96 and 192 on the tile
// plan, where they are faster than the register passes (launch_fock has the figures).
//
// A line of N = N1 N2 points is transformed in two register DFTs with one exchange through
// shared memory, as in the register engine (fft_reg.cuh), but N1 and N2 are run-time
// values: every phase switches on its radix (uniform over the grid) into an unrolled DFT,
// so three kernels serve all sides.  16 slot lanes x T line parts, T = max(N1, N2):
// thread t takes column n2 = t of the first step and row k1 = t of the second; where the
// factors differ the surplus threads sit one step out.  No thread holds data across a
// phase, so that two CTAs of up to 256 threads fill an SM at 128 registers.  FP32 transforms and the
// forward pass fit them; of the FP64 ones the inverse row pass spills (2.0 KB of stores and
// 2.5 KB of loads over its sixteen cases: the epilogue holds h across the IDFT) and the column pass
// 92 and 372 B.
//
// What bounds it: the passes move the same bytes as the register engine's (each pass reads
// and writes the spectrum once) and their DFTs are a few hundred FP64 operations per
// thread between the copies; against the Stockham stages of the generic engine (radix 8,
// 5, 3, ... with a shared-memory round trip each and 2 N entries per line) a line has one
// exchange instead of three to five.
#pragma once

#include <type_traits>

#include "fft_reg.cuh"
#include "fock_fast.cuh"
#include "fock_params.cuh"

namespace hf {

constexpr int kTwoRadix = 16;

// Calls f(integral_constant<int, r>) for the run-time radix r (1 .. kTwoRadix).
template <class F>
__device__ __forceinline__ void two_switch(int r, F&& f) {
  switch (r) {
#define HF_CASE(R) case R: f(std::integral_constant<int, R>{}); break;
    HF_CASE(1) HF_CASE(2) HF_CASE(3) HF_CASE(4) HF_CASE(5) HF_CASE(6) HF_CASE(7) HF_CASE(8)
    HF_CASE(9) HF_CASE(10) HF_CASE(11) HF_CASE(12) HF_CASE(13) HF_CASE(14) HF_CASE(15) HF_CASE(16)
#undef HF_CASE
    default: break;
  }
}

// Keeps what is computed from v inside the loop that calls this: the addresses of all
// sixteen unrolled cases, taken out of the item loop, would not fit in registers.
__device__ __forceinline__ int in_loop(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

template <int R, bool INV, typename C>
__device__ __forceinline__ void two_dft(C* x) {
  rdft<R, R, INV>(x, static_cast<const C*>(nullptr));
}

// DFT of column t (R = N1 points, stride N2), twiddle W_N^{t k} and into buf (the caller
// synchronises before the second step reads it).
template <int R, typename FC>
__device__ __forceinline__ void two_first(FC* x, FC* buf, const FC* tw, int t, int s, int n2) {
  two_dft<R, false>(x);
#pragma unroll
  for (int k = 0; k < R; ++k) buf[(k * n2 + t) * 16 + s] = k ? cmul(x[k], tw[t * k]) : x[k];
}
// Inverse counterpart of the second step: IDFT of row t (R = N2 points), conjugate twiddle, into buf.
template <int R, typename FC>
__device__ __forceinline__ void two_first_inv(FC* x, FC* buf, const FC* tw, int t, int s) {
  two_dft<R, true>(x);
#pragma unroll
  for (int m = 0; m < R; ++m) buf[(t * R + m) * 16 + s] = m ? cmulc(x[m], tw[t * m]) : x[m];
}

template <typename ST, typename FT>
__global__ void __launch_bounds__(16 * kTwoRadix, 2) k_two_row_fwd(const __grid_constant__ FockParams p) {
  using SC = cpx_t<ST>;
  using FC = cpx_t<FT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FC* tw = reinterpret_cast<FC*>(smem_raw);
  const int N = p.nk2, LS = p.LS;
  FC* buf = tw + N;
  const int s = threadIdx.x & 15;
  build_twiddles<FT>(tw, N);
  pdl_begin();  // an earlier build on the stream may still read the scratch
  if (p.active && !*p.active) return;
  zero_h<SC>(p);
  const bool has_ref = (p.flags & HF_FOCK_HAS_REFP) != 0;
  __syncthreads();
  for (int item = blockIdx.x; item < p.ngroups * p.nk1; item += gridDim.x) {
    const int t = in_loop(threadIdx.x >> 4), N1 = in_loop(p.two_row & 31), N2 = in_loop(p.two_row >> 5);
    const int g = item % p.ngroups, k1 = item / p.ngroups;
    const int c = s < LS ? p.chan[g * LS + s] : -1;
    if (t < N2) {
      const size_t at = ((size_t)k1 * N + t) * p.nb2 + (c < 0 ? 0 : c), st = (size_t)N2 * p.nb2;
      const SC* P = static_cast<const SC*>(p.P) + at;
      const SC* ref = static_cast<const SC*>(p.refP) + at;
      two_switch(N1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = c >= 0 ? cvt<FC>(ld_stream(P + i * st)) : mk<FC>(0.0, 0.0);
        if (has_ref && c >= 0) {
#pragma unroll
          for (int i = 0; i < R; ++i) {
            // the difference at the storage precision, then converted (mixed precision)
            if constexpr (sizeof(SC) == sizeof(FC)) x[i] = csub(x[i], cvt<FC>(ld_stream(ref + i * st)));
            else x[i] = cvt<FC>(csub(ld_stream(P + i * st), ld_stream(ref + i * st)));
          }
        }
        two_first<R>(x, buf, tw, t, s, N2);
      });
    }
    __syncthreads();
    if (t < N1) {
      FC* out = static_cast<FC*>(p.scratch) + (((size_t)g * p.nk1 + k1) * N + t) * LS + s;
      const int st = N1 * LS;
      two_switch(N2, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = buf[(t * R + i) * 16 + s];
        two_dft<R, false>(x);
        if (s < LS) {
#pragma unroll
          for (int i = 0; i < R; ++i) __stcg(out + i * st, x[i]);
        }
      });
    }
    __syncthreads();  // buf is rewritten by the next item
  }
}

template <typename ST, typename FT, bool VREAL>
__global__ void __launch_bounds__(16 * kTwoRadix, 2) k_two_col(const __grid_constant__ FockParams p) {
  pdl_launch_dependents();
  using SC = cpx_t<ST>;
  using FC = cpx_t<FT>;
  using VT = std::conditional_t<VREAL, ST, SC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FC* tw = reinterpret_cast<FC*>(smem_raw);
  const int N = p.nk1, LS = p.LS;
  FC* buf = tw + N;
  const int s = threadIdx.x & 15;
  build_twiddles<FT>(tw, N);
  const bool vr_scalar = (p.flags & HF_FOCK_VR_SCALAR) != 0;
  const size_t vstride = (vr_scalar ? 1 : (size_t)p.nb2) * p.nk2;
  pdl_wait();  // the row pass has finished writing the scratch
  if (p.active && !*p.active) return;
  __syncthreads();
  for (int item = blockIdx.x; item < p.ngroups * p.nk2; item += gridDim.x) {
    const int t = in_loop(threadIdx.x >> 4), N1 = in_loop(p.two_col & 31), N2 = in_loop(p.two_col >> 5);
    const int g = item % p.ngroups, k2c = item / p.ngroups;
    const int c = s < LS ? p.chan[g * LS + s] : -1;
    FC* col = static_cast<FC*>(p.scratch) + ((size_t)g * p.nk1 * p.nk2 + k2c) * LS + (s < LS ? s : 0);
    const size_t rs = (size_t)p.nk2 * LS;
    if (t < N2) {
      two_switch(N1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = c >= 0 ? __ldcg(col + (t + i * N2) * rs) : mk<FC>(0.0, 0.0);
        two_first<R>(x, buf, tw, t, s, N2);
      });
    }
    __syncthreads();
    if (t < N1) {
      const VT* V = static_cast<const VT*>(p.VR) + (vr_scalar ? k2c : (size_t)k2c * p.nb2 + (c < 0 ? 0 : c));
      two_switch(N2, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        VT v[R];  // V-hat, in flight across the reads and the transform
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = ld_stream(V + (t + i * N1) * vstride);
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = buf[(t * R + i) * 16 + s];
        two_dft<R, false>(x);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if constexpr (VREAL) {
            const FT w = (FT)((double)v[i] * p.scale);
            x[i] = make_c<FC>(x[i].x * w, x[i].y * w);
          } else {
            x[i] = cmul(x[i], mk<FC>((double)v[i].x * p.scale, (double)v[i].y * p.scale));
          }
        }
        two_first_inv<R>(x, buf, tw, t, s);  // row t of buf is this thread's own: no barrier between
      });
    }
    __syncthreads();
    if (t < N2) {
      two_switch(N1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = buf[(i * N2 + t) * 16 + s];
        two_dft<R, true>(x);
        if (s < LS) {
#pragma unroll
          for (int i = 0; i < R; ++i) __stcg(col + (t + i * N2) * rs, x[i]);
        }
      });
    }
    __syncthreads();
  }
}

// Column t of an inverse row (N1 points at t, t + N2, ... in buf): the last register IDFT and
// the outputs of its k-points (contact sigma, Hartree diagonal, herm with the transposed
// channel, + h).  The 16 slot lanes of a line part call it together.
template <typename ST, typename FT>
__device__ __forceinline__ void two_epilogue(const FockParams& p, const cpx_t<FT>* buf, bool exch, int g, int k1,
                                             int t, int s, int N1, int N2) {
  using SC = cpx_t<ST>;
  using FC = cpx_t<FT>;
  const int LS = p.LS, nb = p.nb;
  const unsigned half = 0xffffu << (threadIdx.x & 16);  // these 16 lanes
  const bool packing = (p.flags & HF_FOCK_PACKING) != 0;
  const int c = s < LS ? p.chan[g * LS + s] : -1, pl = s < LS ? p.partner[g * LS + s] : s;
  const int a = c >= 0 ? c / nb : 0, b = c >= 0 ? c - a * nb : 0, cab = a * nb + b, cba = b * nb + a;
  const size_t at = ((size_t)k1 * N1 * N2 + t) * p.nb2, st = (size_t)N2 * p.nb2;
  const SC* h = static_cast<const SC*>(p.h) + at;
  SC* Sg = static_cast<SC*>(p.Sigma) + at;
  SC* F = static_cast<SC*>(p.F) + at;
  SC zab = mk<SC>(0.0, 0.0), zba = mk<SC>(0.0, 0.0);
  double hd = 0.0;
  if (p.sigc != nullptr && c >= 0) {
    zab = cvt<SC>(p.sigc[cab]);
    zba = cvt<SC>(p.sigc[cba]);
    if (a == b) hd = p.hdiag[a];
  }
  two_switch(N1, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    SC hv[R];
#pragma unroll
    for (int i = 0; i < R; ++i) hv[i] = c >= 0 ? ld_stream(h + i * st + cab) : mk<SC>(0.0, 0.0);
    FC x[R];
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = exch ? buf[((size_t)i * N2 + t) * 16 + s] : mk<FC>(0.0, 0.0);
    if (exch) two_dft<R, true>(x);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      SC sab = cvt<SC>(x[i]), sba, hba;
      if (packing) {
        sba = a == b ? sab : conj(sab);
        hba = c >= 0 ? ld_stream(h + i * st + cba) : mk<SC>(0.0, 0.0);
      } else {  // the transposed channel is another slot lane of the same k-point
        sba.x = __shfl_sync(half, sab.x, pl, 16);
        sba.y = __shfl_sync(half, sab.y, pl, 16);
        hba.x = __shfl_sync(half, hv[i].x, pl, 16);
        hba.y = __shfl_sync(half, hv[i].y, pl, 16);
      }
      if (c < 0) continue;
      sab = cadd(sab, zab);
      sba = cadd(sba, zba);
      SC f = mk<SC>(0.5 * ((double)hv[i].x + (double)hba.x) + 0.5 * ((double)sab.x + (double)sba.x),
                    0.5 * ((double)hv[i].y - (double)hba.y) + 0.5 * ((double)sab.y - (double)sba.y));
      f.x += (ST)hd;
      st_stream(Sg + i * st + cab, sab);
      st_stream(F + i * st + cab, f);
      if (packing && a != b) {
        st_stream(Sg + i * st + cba, sba);
        st_stream(F + i * st + cba, conj(f));
      }
    }
  });
}

template <typename ST, typename FT>
__global__ void __launch_bounds__(16 * kTwoRadix, 2) k_two_row_inv(const __grid_constant__ FockParams p) {
  using FC = cpx_t<FT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FC* tw = reinterpret_cast<FC*>(smem_raw);
  const int N = p.nk2, LS = p.LS;
  FC* buf = tw + N;
  const int s = threadIdx.x & 15;
  const bool exch = (p.flags & HF_FOCK_EXCHANGE) != 0;
  if (exch) build_twiddles<FT>(tw, N);
  pdl_wait();  // the column pass has finished writing the scratch
  if (p.active && !*p.active) return;
  __syncthreads();
  for (int item = blockIdx.x; item < p.ngroups * p.nk1; item += gridDim.x) {
    const int t = in_loop(threadIdx.x >> 4), N1 = in_loop(p.two_row & 31), N2 = in_loop(p.two_row >> 5);
    const int g = item % p.ngroups, k1 = item / p.ngroups;
    if (exch) {
      if (t < N1) {
        const FC* row = static_cast<const FC*>(p.scratch) + (((size_t)g * p.nk1 + k1) * N + t) * LS + (s < LS ? s : 0);
        const int st = N1 * LS;
        two_switch(N2, [&](auto rc) {
          constexpr int R = decltype(rc)::value;
          FC x[R];
#pragma unroll
          for (int i = 0; i < R; ++i) x[i] = __ldcg(row + i * st);
          two_first_inv<R>(x, buf, tw, t, s);
        });
      }
      __syncthreads();
    }
    if (t < N2) two_epilogue<ST, FT>(p, buf, exch, g, k1, t, s, N1, N2);
    __syncthreads();  // buf is rewritten by the next item
  }
}

}  // namespace hf
