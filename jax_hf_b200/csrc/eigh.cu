// Batched eigh of small Hermitian matrices, nb <= 16: for nb >= 2 tridiagonalisation and
// implicit-shift QR (Golub & Van Loan, Matrix Computations, secs. 8.3.1-8.3.5).
//
// What bounds it: a matrix is one k-point (1 KiB at nb = 8), the bytes are nothing, and
// the arithmetic is a serial chain per matrix.  A Jacobi sweep pays that chain (divide,
// square root, reciprocal) in every lane for 7 sweeps x 7 rounds and rotates both A and
// V; here the split is by what is parallel:
//   * a group of G lanes (4, 8 or 16) owns a matrix, one column per lane in registers,
//     for the Householder reduction and its back-accumulation (O(nb^3), all parallel);
//   * the QR iteration is scalar and serial, so ONE thread runs it per matrix: lane m of
//     the CTA's warp 0 takes matrix m with d and e in registers (a sweep is unrolled, so
//     the indices are compile-time), and only writes its rotations (c, s) to shared
//     memory; MPC (up to 32) chains run side by side in the lanes of that warp, and
//     other CTAs of the SM fill the pipes meanwhile;
//   * the group then applies the recorded rotations to the eigenvectors, lane r holding
//     row r in registers: 8 FP64 operations per rotation and lane, no reduction.
// Measured on a B200 (kernel, complex128; before: cyclic Jacobi, lane per column for nb <= 8
// and warp per matrix above): 20736 matrices of nb = 8 in 76 us (291 before), of nb = 4 in
// 14 us (40 with the call), 2401 of nb = 16 in 108 us (991 before).  It stays below 10% of
// the FP64 rate: what is left is the latency of the QR chain.
//
// Convergence: an off-diagonal is dropped at 2^-53 (|d_k| + |d_k+1|) or 2^-56 of the
// largest entry, Wilkinson shifts, at most 30 nb sweeps.  The matrix is scaled by a power
// of two first, so squares neither overflow nor underflow.  A matrix with a non-finite
// entry gives NaN eigenvalues and eigenvectors.
#include "common.cuh"

namespace hf {

namespace {

constexpr double kHalfUlp = 0x1p-53;

constexpr double kTiny2 = 1e-36;  // squares below this are zero next to entries of order one

template <int NB>
struct TriShape {
  static constexpr int G = NB <= 4 ? 4 : NB <= 8 ? 8 : 16;  // lanes per matrix
  static constexpr int LP = NB + 1;
  // odd strides in 16-byte units: the groups of a warp read the same element of their own
  // matrices from different banks
  static constexpr int MAT = NB * LP + 1;
  static constexpr int WL = NB | 1;
  // Matrices per CTA at most, and CTAs per SM (the register cap).  A QR chain costs its warp
  // the same issue slots for 1 lane as for 32, but a CTA of 32 matrices holds registers for
  // all its columns meanwhile.  Kernel times in us on a B200, complex128, (matrices, CTAs):
  // nb = 4, 20736 matrices: (32, 3) 13.7, (16, 4) 18.2;  nb = 8, 20736: (32, 2) 89, (32, 3) 77,
  // (16, 4) 87, (16, 5) 74, (16, 6) 76;  nb = 16, 2401: (16, 2) 129, (8, 2) 163, (8, 3) 106, (8, 4) 110.
  static constexpr int MAXM = NB <= 4 ? 32 : NB <= 8 ? 16 : 8;
  static constexpr int CTAS = NB <= 4 ? 4 : NB <= 8 ? 5 : 3;
  static constexpr int SWEEPS = NB <= 8 ? 6 : 8;              // sweeps per chunk of rotations
  static constexpr size_t BYTES = (size_t)(MAT + WL + SWEEPS * (NB - 1)) * 16 + 3 * NB * 8 + 8;  // per matrix
};

// One implicit-shift QR sweep of every lane's own tridiagonal (d, e), on the unreduced block
// that ends at its last nonzero off-diagonal; the rotations go to rot[k * stride],
// identities where the block does not reach.  Returns whether this lane had a block; all
// 32 lanes call it together (the steps that no lane needs are skipped by a uniform branch).
//
// A step applies c = x / r, s = z / r, r^2 = x^2 + z^2, to columns k, k + 1.  Written on the
// unnormalised x, z,
//   d_k' = (x (x d_k + z e_k) + z (x e_k + z d_k+1)) / r^2,   e_k' = (x (x e_k + z d_k+1) - z (x d_k + z e_k)) / r^2,
// and the next r^2 is e_k'^2 + (z e_k+1)^2 / r^2, so the chain from one r^2 to the next is one
// reciprocal, a product and an fma; the square root of c, s and z' runs beside it.
template <int NB>
__device__ __forceinline__ bool qr_sweep(double (&d)[NB], double (&e)[NB], double small, double2* rot, int stride,
                                         bool store) {
  unsigned nz = 0;
#pragma unroll
  for (int k = 0; k < NB - 1; ++k) {
    const bool drop = fabs(e[k]) <= fmax(kHalfUlp * (fabs(d[k]) + fabs(d[k + 1])), small);
    e[k] = drop ? 0.0 : e[k];
    nz |= drop ? 0u : 1u << k;
  }
  const int last = 31 - __clz(nz);  // the block is columns first .. last + 1; -1: no block
  const unsigned gaps = ~nz & ((1u << (last < 0 ? 0 : last)) - 1u);
  const int first = last < 0 ? NB : 32 - __clz(gaps);
  if (!__any_sync(0xffffffffu, nz != 0)) return false;
  double dq = 0.0, dp = 0.0, eq = 0.0, x = 0.0, z = 0.0;
#pragma unroll
  for (int k = 0; k < NB - 1; ++k) {
    if (k == last) { dp = d[k]; dq = d[k + 1]; eq = e[k]; }
    if (k == first) { x = d[k]; z = e[k]; }
  }
  {  // Wilkinson shift: the eigenvalue of the trailing 2 x 2 nearer to dq
    const double g = 0.5 * (dp - dq), q2 = fmax(fma(g, g, eq * eq), kTiny2);
    const double t = g + copysign(q2 * rsqrt_seeded(q2), g);
    x -= fma(-eq, eq * recip_seeded(t), dq);
  }
  double r2 = fma(x, x, z * z);
#pragma unroll
  for (int k = 0; k < NB - 1; ++k) {
    double2 cs = make_double2(1.0, 0.0);
    if (k >= first && k <= last) {
      // nothing left to chase: an entry below the dropping threshold in its place, c = 1
      if (!(r2 > kTiny2)) { x = 1e-17; z = 0.0; r2 = 1e-34; }
      const double iv = rsqrt_seeded(r2), i2 = recip_seeded(r2);
      const double ek = e[k], d0 = d[k], d1 = d[k + 1];
      const double en = k + 1 < NB - 1 ? e[k + 1 < NB - 1 ? k + 1 : 0] : 0.0;
      const double u = fma(x, d0, z * ek), w = fma(x, ek, z * d1), t = z * en;
      const double dn = fma(x, u, z * w) * i2, xn = fma(x, w, -z * u) * i2;
      cs = make_double2(x * iv, z * iv);
      {  // unit length to rounding (off the chain): iv carries an error common to c and s
        const double f = -0.5 * fma(cs.x, cs.x, fma(cs.y, cs.y, -1.0));
        cs = make_double2(fma(f, cs.x, cs.x), fma(f, cs.y, cs.y));
      }
      if (k > 0) {
        if (k > first) e[k > 0 ? k - 1 : 0] = r2 * iv;
      }
      d[k] = dn;
      d[k + 1] = d1 + (d0 - dn);
      e[k] = x = xn;
      if (k + 1 < NB - 1) {
        r2 = fma(x, x, (t * t) * i2);
        z = cs.y * en;
        if (k < last) e[k + 1 < NB - 1 ? k + 1 : 0] = cs.x * en;
      }
    }
    if (store) rot[k * stride] = cs;
  }
  return nz != 0;
}

// V diag(eps) V^H = herm(A) (mode 0) or herm(i A) (mode 1) for nk matrices, ascending.
template <typename RT, int NB>
__global__ void __launch_bounds__(TriShape<NB>::MAXM * TriShape<NB>::G, TriShape<NB>::CTAS)
    k_eigh_tri(int nk, int mode, const cpx_t<RT>* A, RT* eps, cpx_t<RT>* V) {
  pdl_begin();
  using S = TriShape<NB>;
  constexpr int G = S::G, LP = S::LP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int mpc = blockDim.x / G;
  double2* mat = reinterpret_cast<double2*>(smem_raw);
  double2* wbuf = mat + mpc * S::MAT;
  double2* rot = wbuf + mpc * S::WL;  // rotations of a chunk: [sweep][k][matrix]
  double* sD = reinterpret_cast<double*>(rot + mpc * S::SWEEPS * (NB - 1));
  double* sE = sD + mpc * NB;
  double* sT = sE + mpc * NB;
  int* sCnt = reinterpret_cast<int*>(sT + mpc * NB);
  const int g = threadIdx.x / G, c = threadIdx.x % G, k0 = blockIdx.x * mpc + g;
  const bool on = k0 < nk && c < NB;
  double2* SM = mat + g * S::MAT;
  double2* SW = wbuf + g * S::WL;
  const size_t base = (size_t)k0 * NB * NB + c;

  // ---- this lane's column of herm(A), scaled to entries of order one
  double2 a[NB];
#pragma unroll
  for (int r = 0; r < NB; ++r) {
    double2 x = on ? cvt<double2>(A[base + (size_t)r * NB]) : make_double2(0.0, 0.0);
    if (mode == 1) x = mul_pi(x);
    a[r] = x;
    if (c < NB) SM[r * LP + c] = x;
  }
  __syncwarp();
  double big = 0.0;
  bool fin = true;
  if (c < NB) {
#pragma unroll
    for (int r = 0; r < NB; ++r) {
      const double2 y = SM[c * LP + r];
      // halves first: the sum of two large entries must not overflow
      a[r] = make_double2(0.5 * a[r].x + 0.5 * y.x, r == c ? 0.0 : 0.5 * a[r].y - 0.5 * y.y);
      fin = fin && isfinite(a[r].x) && isfinite(a[r].y);
      big = fmax(big, fmax(fabs(a[r].x), fabs(a[r].y)));
    }
  }
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) {
    big = fmax(big, __shfl_xor_sync(0xffffffffu, big, off));
    fin = __shfl_xor_sync(0xffffffffu, (int)fin, off) && fin;
  }
  const int ex = (big > 0.0 && fin) ? max(-1000, min(1000, ilogb(big))) : 0;
  const double down = ldexp(1.0, -ex), up = ldexp(1.0, ex);
#pragma unroll
  for (int r = 0; r < NB; ++r) a[r] = fin ? cscale(a[r], down) : make_double2(0.0, 0.0);
  __syncwarp();

  // ---- Householder: columns k = 0 .. NB - 3, H_k = I - tau v v^H with v = x + (x_1/|x_1|) |x| e_1,
  // v kept in row k of SM.  The subdiagonals come out complex; the phases that make them
  // positive are collected in ph and go into the start of the accumulation.
  double2 ph = make_double2(1.0, 0.0), myph = ph;
#pragma unroll
  for (int k = 0; k < NB - 2; ++k) {
    if (c == k) {
#pragma unroll
      for (int i = k + 1; i < NB; ++i) SM[k * LP + i] = a[i];
    }
    __syncwarp();
    double2 v[NB];
    double n2 = 0.0;
#pragma unroll
    for (int i = k + 1; i < NB; ++i) {
      v[i] = SM[k * LP + i];
      n2 = fma(v[i].x, v[i].x, fma(v[i].y, v[i].y, n2));
    }
    double2 vc = c > k && c < NB ? SM[k * LP + c] : make_double2(0.0, 0.0);
    double nr = 0.0, tau = 0.0;
    if (n2 > kTiny2) {
      const double x2 = fma(v[k + 1].x, v[k + 1].x, v[k + 1].y * v[k + 1].y);
      const double ix = x2 > kTiny2 ? rsqrt_seeded(x2) : 0.0;
      const double2 th = x2 > kTiny2 ? cscale(v[k + 1], ix) : make_double2(1.0, 0.0);
      nr = n2 * rsqrt_seeded(n2);
      tau = recip_seeded(nr * (nr + x2 * ix));
      v[k + 1].x = fma(th.x, nr, v[k + 1].x);
      v[k + 1].y = fma(th.y, nr, v[k + 1].y);
      const double2 t = cmul(ph, th);
      ph = make_double2(-t.x, -t.y);
    }
    if (c == k + 1) { myph = ph; vc = v[k + 1]; }
    double2 p0 = make_double2(0.0, 0.0), p1 = p0;  // column c of A: (A v)_c = sum_i conj(A_ic) v_i
#pragma unroll
    for (int i = k + 1; i < NB; ++i) {
      if ((i - k) & 1) p0 = cfma_cj(a[i], v[i], p0);
      else p1 = cfma_cj(a[i], v[i], p1);
    }
    const double2 p = cscale(cadd(p0, p1), tau);
    double kp = fma(vc.x, p.x, vc.y * p.y);  // zero in the lanes outside the block (vc = 0)
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) kp += __shfl_xor_sync(0xffffffffu, kp, off);
    const double kk = 0.5 * tau * kp;
    const double2 w = make_double2(fma(-kk, vc.x, p.x), fma(-kk, vc.y, p.y));
    if (c > k && c < NB) SW[c] = w;
    __syncwarp();
    if (c == k + 1) SM[k * LP + k + 1] = v[k + 1];
    if (c == k) {
      sD[k * mpc + g] = a[k].x;
      sE[k * mpc + g] = nr;
      sT[k * mpc + g] = tau;
    }
#pragma unroll
    for (int i = k + 1; i < NB; ++i) {  // A -= v w^H + w v^H
      const double2 wi = SW[i];
      a[i].x = fma(-v[i].x, w.x, fma(-v[i].y, w.y, fma(-wi.x, vc.x, fma(-wi.y, vc.y, a[i].x))));
      a[i].y = fma(-v[i].y, w.x, fma(v[i].x, w.y, fma(-wi.y, vc.x, fma(wi.x, vc.y, a[i].y))));
    }
  }
  if (c == NB - 2) {
    SM[(NB - 2) * LP + NB - 1] = a[NB - 1];
    sD[(NB - 2) * mpc + g] = a[NB - 2].x;
  }
  if (c == NB - 1) sD[(NB - 1) * mpc + g] = a[NB - 1].x;
  __syncwarp();
  {
    const double2 zl = SM[(NB - 2) * LP + NB - 1];
    const double z2 = fma(zl.x, zl.x, zl.y * zl.y);
    const double iz = z2 > kTiny2 ? rsqrt_seeded(z2) : 0.0;
    if (c == NB - 1) {
      sE[(NB - 2) * mpc + g] = z2 * iz;
      myph = z2 > kTiny2 ? cmul(ph, cscale(zl, iz)) : ph;
    }
  }

  // ---- Q = H_0 H_1 ... diag(phases), this lane's column; then its row
  double2 q[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i) q[i] = i == c ? myph : make_double2(0.0, 0.0);
#pragma unroll
  for (int k = NB - 3; k >= 0; --k) {
    const double tau = sT[k * mpc + g];
    double2 s0 = make_double2(0.0, 0.0), s1 = s0;
#pragma unroll
    for (int i = k + 1; i < NB; ++i) {
      if ((i - k) & 1) s0 = cfma_cj(SM[k * LP + i], q[i], s0);
      else s1 = cfma_cj(SM[k * LP + i], q[i], s1);
    }
    const double2 s = cscale(cadd(s0, s1), -tau);
#pragma unroll
    for (int i = k + 1; i < NB; ++i) q[i] = cfma(SM[k * LP + i], s, q[i]);
  }
  __syncwarp();
  if (c < NB) {
#pragma unroll
    for (int i = 0; i < NB; ++i) SM[i * LP + c] = q[i];
  }
  __syncthreads();

  // ---- chunks of QR sweeps (one thread per matrix) and their rotations (every lane)
  int total = 0;
  for (;;) {
    int more = 0;
    if (threadIdx.x < 32) {  // the whole warp runs the sweeps; lanes from mpc on idle along
      const bool mine = threadIdx.x < mpc;
      const int m = mine ? threadIdx.x : 0;
      double d[NB], e[NB];
      double an = 0.0;
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        d[i] = sD[i * mpc + m];
        e[i] = i < NB - 1 ? sE[i * mpc + m] : 0.0;
        an = fmax(an, fmax(fabs(d[i]), fabs(e[i])));
      }
      if (!mine) {
#pragma unroll
        for (int i = 0; i < NB; ++i) e[i] = 0.0;
      }
      int n = 0;  // sweeps that found a block: the first n of the chunk
      for (int w = 0; w < S::SWEEPS; ++w) {
        const bool had = qr_sweep<NB>(d, e, an * 0x1p-56, rot + (w * (NB - 1)) * mpc + m, mpc, mine);
        if (!__any_sync(0xffffffffu, had)) break;
        n += had;
      }
      total += n;
      more = n == S::SWEEPS && total < 30 * NB;
      if (mine) {
        sCnt[m] = n;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          sD[i * mpc + m] = d[i];
          if (i < NB - 1) sE[i * mpc + m] = e[i];
        }
      }
    }
    const int any = __syncthreads_or(more);
    // row c of the eigenvectors comes from shared memory for each chunk, so that no lane
    // holds it across the QR sweeps
    const int n = sCnt[g];
    if (c < NB) {
#pragma unroll
      for (int i = 0; i < NB; ++i) q[i] = SM[c * LP + i];
    }
    for (int w = 0; w < n; ++w) {
#pragma unroll
      for (int k = 0; k < NB - 1; ++k) {
        const double2 cs = rot[(w * (NB - 1) + k) * mpc + g];
        if (cs.y != 0.0 || cs.x != 1.0) {
          const double2 x = q[k], y = q[k + 1];
          q[k] = make_double2(fma(cs.x, x.x, cs.y * y.x), fma(cs.x, x.y, cs.y * y.y));
          q[k + 1] = make_double2(fma(cs.x, y.x, -cs.y * x.x), fma(cs.x, y.y, -cs.y * x.y));
        }
      }
    }
    if (!any) break;
    if (c < NB) {
#pragma unroll
      for (int i = 0; i < NB; ++i) SM[c * LP + i] = q[i];
    }
    __syncthreads();  // the rotations are overwritten by the next chunk
  }
  __syncwarp();

  // ---- ascending order, eigenvectors as columns
  if (c < NB) {
    const double wc = sD[c * mpc + g];
    int rk = 0;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const double wj = sD[j * mpc + g];
      rk += (wj < wc) || (wj == wc && j < c);
    }
    if (on) eps[(size_t)k0 * NB + rk] = (RT)(fin ? wc * up : NAN);
    sT[c * mpc + g] = __longlong_as_double((long long)rk);
  }
  __syncwarp();
  if (c < NB) {
#pragma unroll
    for (int i = 0; i < NB; ++i) SM[c * LP + (int)__double_as_longlong(sT[i * mpc + g])] = q[i];
  }
  __syncwarp();
  if (on) {
#pragma unroll
    for (int r = 0; r < NB; ++r)
      V[base + (size_t)r * NB] = fin ? cvt<cpx_t<RT>>(SM[r * LP + c]) : mk<cpx_t<RT>>(NAN, NAN);
  }
}

// nb = 1: the eigenvalue is the entry's real part (mode 1: of i A), the eigenvector 1.
template <typename RT>
__global__ void k_eigh_one(int nk, int mode, const cpx_t<RT>* A, RT* eps, cpx_t<RT>* V) {
  pdl_begin();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x) {
    const cpx_t<RT> a = A[k];
    eps[k] = mode == 1 ? -a.y : a.x;
    V[k] = mk<cpx_t<RT>>(1.0, 0.0);
  }
}

template <typename RT>
int launch_one(cudaStream_t s, int nk, int mode, const void* A, void* eps, void* V) {
  const int blocks = (nk + 255) / 256;
  launch_pdl(k_eigh_one<RT>, blocks < 148 * 8 ? blocks : 148 * 8, 256, 0, s, nk, mode,
             static_cast<const cpx_t<RT>*>(A), static_cast<RT*>(eps), static_cast<cpx_t<RT>*>(V));
  HF_LAUNCH_CHECK("k_eigh_one");
  return HF_OK;
}

template <typename RT, int NB>
int launch_tri(cudaStream_t s, int nk, int mode, const void* A, void* eps, void* V) {
  using S = TriShape<NB>;
  // a CTA takes up to MAXM matrices (one warp runs their QR chains); fewer while that
  // leaves SMs without a CTA, down to one warp per CTA
  int mpc = S::MAXM;
  while (mpc > 32 / S::G && (nk + mpc - 1) / mpc < 148) mpc >>= 1;
  const size_t smem = (size_t)mpc * S::BYTES;
  HF_SMEM_CAP(k_eigh_tri<RT, NB>);
  launch_pdl(k_eigh_tri<RT, NB>, (nk + mpc - 1) / mpc, mpc * S::G, smem, s, nk, mode, static_cast<const cpx_t<RT>*>(A),
                                                                   static_cast<RT*>(eps), static_cast<cpx_t<RT>*>(V));
  HF_LAUNCH_CHECK("k_eigh_tri");
  return HF_OK;
}

}  // namespace

// nb <= 16: beyond that a column no longer fits a lane's registers (perk.cu's warp-per-matrix
// Jacobi takes nb = 17 .. 32).
int eigh_tri(void* stream, int dtype, int nk, int nb, const void* A, void* eps, void* V, int mode) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (nb == 1) return dtype == HF_C128 ? launch_one<double>(s, nk, mode, A, eps, V) : launch_one<float>(s, nk, mode, A, eps, V);
  switch (nb) {
#define HF_NB_CASE(N)                                                                \
  case N:                                                                            \
    return dtype == HF_C128 ? launch_tri<double, N>(s, nk, mode, A, eps, V) : launch_tri<float, N>(s, nk, mode, A, eps, V);
    HF_NB_CASE(2) HF_NB_CASE(3) HF_NB_CASE(4) HF_NB_CASE(5) HF_NB_CASE(6) HF_NB_CASE(7) HF_NB_CASE(8)
    HF_NB_CASE(9) HF_NB_CASE(10) HF_NB_CASE(11) HF_NB_CASE(12) HF_NB_CASE(13) HF_NB_CASE(14) HF_NB_CASE(15)
    HF_NB_CASE(16)
#undef HF_NB_CASE
    default: break;
  }
  return fail(HF_ERR_UNSUPPORTED, "eigh_tri: needs nb <= 16");
}

}  // namespace hf
