// Line transforms of the two-factor passes (fock_two.cuh) for sides N = N1 N2 whose N2 is
// too long for a register DFT: a prime factor of 17 or more (17, 34, 37, 61, 97, 191, ...).
//
// The N2-point DFTs are direct sums, with the terms j and N2 - j of an output sharing
// their products: p_j = x_j + x_{N2-j}, m_j = x_j - x_{N2-j},
//   X_k, X_{N2-k} = (x_0 + sum_j p_j cos) -+ i (sum_j m_j sin),
// so an output costs N2 real-by-complex products.  A worker (16 slot lanes) keeps K output
// pairs in registers and walks j once: two elements and K twiddles (one broadcast each)
// are read from shared memory for 4 K fused multiply-adds, which makes the sums FP64-bound
// from K = 4 on; the Stockham stage it replaces read two operands per product and formed
// every output by itself.  Measured on a B200 (builds of complex128, nb = 8, back to back,
// before in brackets): 17 x 17 in 14 us (62), 37 x 37 in 20 (199), 61 x 61 in 35 (486),
// 97 x 97 in 104 (1188), 191 x 191 in 369 (12914).
// 16 slot lanes x 16 workers, two line buffers and one twiddle table in shared memory.
#pragma once

#include "fock_two.cuh"

namespace hf {

constexpr int kDenseWorkers = 16;

// Calls f(integral_constant<int, K>) for the output pairs per worker and walk.
template <class F>
__device__ __forceinline__ void dense_switch(int k, F&& f) {
  switch (k) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 6: f(std::integral_constant<int, 6>{}); break;
    default: f(std::integral_constant<int, 8>{}); break;
  }
}

// All N2-point DFTs of the N1 rows of `in` (row k1: [x_0, p_1 .. p_H, (x_mid), m_H .. m_1], 16
// slots each); sink(k1, k, X_k, X_{N2-k}) for k = 0 .. N2 / 2 (the two agree where k = N2 - k mod N2).
template <bool INV, typename FC, class Sink>
__device__ __forceinline__ void dense_rows(const FC* in, const FC* tw, int N, int N1, int N2, int kk, int wk, int s,
                                           Sink&& sink) {
  using T = decltype(in->x);
  using U = std::remove_cv_t<std::remove_reference_t<T>>;
  const int H = (N2 - 1) / 2, KT = N2 / 2 + 1, tiles = (KT + kk - 1) / kk;
  for (int tile = wk; tile < N1 * tiles; tile += kDenseWorkers) {
    const int k1 = tile / tiles, k0 = (tile - k1 * tiles) * kk;
    const FC* row = in + (size_t)k1 * N2 * 16 + s;
    dense_switch(kk, [&](auto kc) {
      constexpr int K = decltype(kc)::value;
      FC r[K], q[K];
      int idx[K], step[K];
      const FC x0 = row[0];
      const FC xm = (N2 & 1) ? mk<FC>(0.0, 0.0) : row[(N2 / 2) * 16];
#pragma unroll
      for (int u = 0; u < K; ++u) {
        const int k = k0 + u < KT ? k0 + u : KT - 1;
        r[u] = (k & 1) ? csub(x0, xm) : cadd(x0, xm);
        q[u] = mk<FC>(0.0, 0.0);
        idx[u] = 0;
        step[u] = N1 * k;
      }
      const FC* pp = row;
      const FC* pm = row + (size_t)N2 * 16;
      for (int j = 1; j <= H; ++j) {
        pp += 16;
        pm -= 16;
        const FC a = *pp, b = *pm;
#pragma unroll
        for (int u = 0; u < K; ++u) {
          idx[u] += step[u];
          if (idx[u] >= N) idx[u] -= N;
          const FC w = tw[idx[u]];  // (cos, -sin)
          r[u].x = fma((U)w.x, a.x, r[u].x);
          r[u].y = fma((U)w.x, a.y, r[u].y);
          q[u].x = fma((U)w.y, b.x, q[u].x);
          q[u].y = fma((U)w.y, b.y, q[u].y);
        }
      }
#pragma unroll
      for (int u = 0; u < K; ++u) {
        if (k0 + u >= KT) break;
        const FC i = INV ? mul_mi(q[u]) : mul_pi(q[u]);
        sink(k1, k0 + u, cadd(r[u], i), csub(r[u], i));
      }
    });
  }
}

// p and m of every row of buf in place.
template <typename FC>
__device__ __forceinline__ void dense_pairs(FC* buf, int N1, int N2, int wk, int s) {
  const int H = (N2 - 1) / 2;
  for (int it = wk; it < N1 * H; it += kDenseWorkers) {
    const int k1 = it / H, j = it - k1 * H + 1;
    FC* a = buf + ((size_t)k1 * N2 + j) * 16 + s;
    FC* b = buf + ((size_t)k1 * N2 + N2 - j) * 16 + s;
    const FC x = *a, y = *b;
    *a = cadd(x, y);
    *b = csub(x, y);
  }
}

template <typename ST, typename FT>
__global__ void __launch_bounds__(16 * kDenseWorkers, 2) k_dense_row_fwd(const __grid_constant__ FockParams p) {
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
    const int wk = in_loop(threadIdx.x >> 4), N1 = in_loop(p.two_row & 31), N2 = in_loop(p.two_row >> 5);
    const int g = item % p.ngroups, k1 = item / p.ngroups;
    const int c = s < LS ? p.chan[g * LS + s] : -1;
    for (int n2 = wk; n2 < N2; n2 += kDenseWorkers) {
      const size_t at = ((size_t)k1 * N + n2) * p.nb2 + (c < 0 ? 0 : c), st = (size_t)N2 * p.nb2;
      const SC* P = static_cast<const SC*>(p.P) + at;
      const SC* ref = static_cast<const SC*>(p.refP) + at;
      two_switch(N1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          SC v = c >= 0 ? ld_stream(P + i * st) : mk<SC>(0.0, 0.0);
          if (has_ref && c >= 0) v = csub(v, ld_stream(ref + i * st));
          x[i] = cvt<FC>(v);
        }
        two_first<R>(x, buf, tw, n2, s, N2);
      });
    }
    __syncthreads();
    dense_pairs(buf, N1, N2, wk, s);
    __syncthreads();
    FC* out = static_cast<FC*>(p.scratch) + ((size_t)g * p.nk1 + k1) * N * LS + s;
    dense_rows<false>(buf, tw, N, N1, N2, p.dense_row, wk, s, [&](int q1, int k, FC a, FC b) {
      if (s >= LS) return;
      __stcg(out + (q1 + N1 * k) * LS, a);
      if (k > 0 && 2 * k != N2) __stcg(out + (q1 + N1 * (N2 - k)) * LS, b);
    });
    __syncthreads();  // buf is rewritten by the next item
  }
}

template <typename ST, typename FT, bool VREAL>
__global__ void __launch_bounds__(16 * kDenseWorkers, 2) k_dense_col(const __grid_constant__ FockParams p) {
  pdl_launch_dependents();
  using SC = cpx_t<ST>;
  using FC = cpx_t<FT>;
  using VT = std::conditional_t<VREAL, ST, SC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FC* tw = reinterpret_cast<FC*>(smem_raw);
  const int N = p.nk1, LS = p.LS;
  FC* buf = tw + N;
  FC* buf2 = buf + (size_t)N * 16;
  const int s = threadIdx.x & 15;
  build_twiddles<FT>(tw, N);
  const bool vr_scalar = (p.flags & HF_FOCK_VR_SCALAR) != 0;
  const size_t vstride = (vr_scalar ? 1 : (size_t)p.nb2) * p.nk2;
  pdl_wait();  // the row pass has finished writing the scratch
  if (p.active && !*p.active) return;
  __syncthreads();
  for (int item = blockIdx.x; item < p.ngroups * p.nk2; item += gridDim.x) {
    const int wk = in_loop(threadIdx.x >> 4), N1 = in_loop(p.two_col & 31), N2 = in_loop(p.two_col >> 5);
    const int g = item % p.ngroups, k2c = item / p.ngroups;
    const int c = s < LS ? p.chan[g * LS + s] : -1;
    FC* col = static_cast<FC*>(p.scratch) + ((size_t)g * p.nk1 * p.nk2 + k2c) * LS + (s < LS ? s : 0);
    const size_t rs = (size_t)p.nk2 * LS;
    for (int n2 = wk; n2 < N2; n2 += kDenseWorkers)
      two_switch(N1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = c >= 0 ? __ldcg(col + (n2 + i * N2) * rs) : mk<FC>(0.0, 0.0);
        two_first<R>(x, buf, tw, n2, s, N2);
      });
    __syncthreads();
    dense_pairs(buf, N1, N2, wk, s);
    __syncthreads();
    const VT* V = static_cast<const VT*>(p.VR) + (vr_scalar ? k2c : (size_t)k2c * p.nb2 + (c < 0 ? 0 : c));
    auto times_v = [&](FC x, int f) {
      const VT v = ld_stream(V + f * vstride);
      if constexpr (VREAL) {
        const FT w = (FT)((double)v * p.scale);
        return make_c<FC>(x.x * w, x.y * w);
      } else {
        return cmul(x, mk<FC>((double)v.x * p.scale, (double)v.y * p.scale));
      }
    };
    // the products with V-hat go back as the pairs of the inverse sums
    dense_rows<false>(buf, tw, N, N1, N2, p.dense_col, wk, s, [&](int q1, int k, FC a, FC b) {
      FC* row = buf2 + (size_t)q1 * N2 * 16 + s;
      a = times_v(a, q1 + N1 * k);
      if (k == 0 || 2 * k == N2) {
        row[k * 16] = a;
      } else {
        b = times_v(b, q1 + N1 * (N2 - k));
        row[k * 16] = cadd(a, b);
        row[(N2 - k) * 16] = csub(a, b);
      }
    });
    __syncthreads();
    dense_rows<true>(buf2, tw, N, N1, N2, p.dense_col, wk, s, [&](int q1, int m, FC a, FC b) {
      FC* row = buf + (size_t)q1 * N2 * 16 + s;
      row[m * 16] = q1 ? cmulc(a, tw[q1 * m]) : a;
      if (m > 0 && 2 * m != N2) row[(N2 - m) * 16] = q1 ? cmulc(b, tw[q1 * (N2 - m)]) : b;
    });
    __syncthreads();
    for (int m2 = wk; m2 < N2; m2 += kDenseWorkers)
      two_switch(N1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        FC x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = buf[((size_t)i * N2 + m2) * 16 + s];
        two_dft<R, true>(x);
        if (s < LS) {
#pragma unroll
          for (int i = 0; i < R; ++i) __stcg(col + (m2 + i * N2) * rs, x[i]);
        }
      });
    __syncthreads();
  }
}

template <typename ST, typename FT>
__global__ void __launch_bounds__(16 * kDenseWorkers, 2) k_dense_row_inv(const __grid_constant__ FockParams p) {
  using FC = cpx_t<FT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FC* tw = reinterpret_cast<FC*>(smem_raw);
  const int N = p.nk2, LS = p.LS;
  FC* buf = tw + N;
  FC* buf2 = buf + (size_t)N * 16;
  const int s = threadIdx.x & 15;
  const bool exch = (p.flags & HF_FOCK_EXCHANGE) != 0;
  if (exch) build_twiddles<FT>(tw, N);
  pdl_wait();  // the column pass has finished writing the scratch
  if (p.active && !*p.active) return;
  __syncthreads();
  for (int item = blockIdx.x; item < p.ngroups * p.nk1; item += gridDim.x) {
    const int wk = in_loop(threadIdx.x >> 4), N1 = in_loop(p.two_row & 31), N2 = in_loop(p.two_row >> 5);
    const int g = item % p.ngroups, k1 = item / p.ngroups;
    if (exch) {
      const FC* in = static_cast<const FC*>(p.scratch) + ((size_t)g * p.nk1 + k1) * N * LS + (s < LS ? s : 0);
      for (int f = wk; f < N; f += kDenseWorkers)  // frequency q1 + N1 k2 to row q1, column k2
        buf[((size_t)(f % N1) * N2 + f / N1) * 16 + s] = __ldcg(in + f * LS);
      __syncthreads();
      dense_pairs(buf, N1, N2, wk, s);
      __syncthreads();
      dense_rows<true>(buf, tw, N, N1, N2, p.dense_row, wk, s, [&](int q1, int m, FC a, FC b) {
        FC* row = buf2 + (size_t)q1 * N2 * 16 + s;
        row[m * 16] = q1 ? cmulc(a, tw[q1 * m]) : a;
        if (m > 0 && 2 * m != N2) row[(N2 - m) * 16] = q1 ? cmulc(b, tw[q1 * (N2 - m)]) : b;
      });
      __syncthreads();
    }
    for (int m2 = wk; m2 < N2; m2 += kDenseWorkers)
      two_epilogue<ST, FT>(p, buf2, exch, g, k1, m2, s, N1, N2);
    __syncthreads();  // the buffers are rewritten by the next item
  }
}

}  // namespace hf
