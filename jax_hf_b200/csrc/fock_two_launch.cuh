// Launch of the two-factor passes: each side takes its register or its dense line transforms.
#pragma once

#include "fock_dense.cuh"
#include "fock_two.cuh"

namespace hf {

// Output pairs per worker and walk of the dense sums: the count that leaves the fewest
// products on the busiest of the 16 workers (4 products per pair and step, 4 for the walk).
inline int dense_pairs_per_walk(int f) {
  const int N1 = f & 31, KT = (f >> 5) / 2 + 1;
  int best = 2, cost = 1 << 30;
  for (int k : {2, 4, 6, 8}) {
    const int tiles = N1 * ((KT + k - 1) / k), c = ((tiles + kDenseWorkers - 1) / kDenseWorkers) * (4 * k + 4);
    if (c <= cost) { cost = c; best = k; }
  }
  return best;
}

// Launches the three passes when both sides have line factors; sets *handled.
template <typename ST, typename FT>
int two_fock(FockParams& p, cudaStream_t stream, bool* handled) {
  *handled = false;
  const int fr = line_factors(p.nk2), fc = line_factors(p.nk1);
  if (p.LS > 16 || p.rows_plan || !fr || !fc) return HF_OK;
  p.two_row = fr;
  p.two_col = fc;
  const bool exch = (p.flags & HF_FOCK_EXCHANGE) != 0;
  auto dense = [](int f) { return (f >> 5) > kTwoRadix; };
  if (dense(fr)) p.dense_row = dense_pairs_per_walk(fr);
  if (dense(fc)) p.dense_col = dense_pairs_per_walk(fc);
  auto pass = [&](auto kern, int f, int n, int items, const char* what) -> int {
    const int threads = dense(f) ? 16 * kDenseWorkers : 16 * ((f & 31) > (f >> 5) ? (f & 31) : (f >> 5));
    // twiddles and one or two buffers of 16 lines
    const size_t smem = (size_t)(dense(f) ? 33 : 17) * n * sizeof(cpx_t<FT>);
    int grid = 0;
    if (int e = persistent_grid(kern, threads, smem, items, &grid)) return e;
    const cudaError_t e = launch_pass(kern, grid, threads, smem, stream, p);
    return e == cudaSuccess ? HF_OK : cuda_check(e, what);
  };
  int st;
  if (exch) {
    st = pass(dense(fr) ? k_dense_row_fwd<ST, FT> : k_two_row_fwd<ST, FT>, fr, p.nk2, p.ngroups * p.nk1,
              "k_two_row_fwd");
    if (st) return st;
    auto col = (p.flags & HF_FOCK_VR_REAL) ? (dense(fc) ? k_dense_col<ST, FT, true> : k_two_col<ST, FT, true>)
                                           : (dense(fc) ? k_dense_col<ST, FT, false> : k_two_col<ST, FT, false>);
    if ((st = pass(col, fc, p.nk1, p.ngroups * p.nk2, "k_two_col"))) return st;
  }
  st = pass(dense(fr) ? k_dense_row_inv<ST, FT> : k_two_row_inv<ST, FT>, fr, p.nk2, p.ngroups * p.nk1,
            "k_two_row_inv");
  if (st) return st;
  *handled = true;
  return HF_OK;
}

}  // namespace hf
