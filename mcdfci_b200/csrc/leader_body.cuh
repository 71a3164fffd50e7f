// Device code of the leader: the serial part of one mCDFCI iteration, run by
// one CTA of 512 threads (leader_body), with its helpers; included by the
// leader kernels (leader_kernel.cu).
//
//   finish iteration t-1   z[D_c] = new_z_c for the picked D_c (the exact
//                          recompute that overwrites the accumulated z,
//                          src/wavefunction.h:557-565); xz += sum_c dot_c
//                          (src/wavefunction.h:583); occupancy check
//                          (src/wavefunction.h:594-599)
//   refetch                (x, z) of every column's candidates from the table
//                          (src/wavefunction.h:567-575)
//   pick                   the k distinct determinants with the largest
//                          |x*xx*scale^2 + z|, ties to the larger determinant
//                          in the reference order (CoordinatePickGcdGrad,
//                          src/solver.h:118-143,196-224)
//   H_sub                  k x k sub-matrix (CDFCI::get_hamiltonian_submatrix,
//                          src/solver.h:637-670): upper triangle from
//                          get_off_diagonal(det_i, det_j) for i < j, diagonal
//                          from get_diagonal (src/hamiltonian.h:252-328)
//   eig update             dx, scale and xx (CoordinateUpdateEig,
//                          src/solver.h:333-609)
//   update_x               x[D_c] += dx_c, xz += z[D_c] * dx_c
//                          (WaveFunctionCuckoo::update_x, src/wavefunction.h:425-451)
//   publish                the k picked determinants, dx, H_cc, xx*scale^2
//                          and scale for the column kernel.
//
// What bounds it: a serial chain on one SM, so the cycles of its phases, and
// of those the instructions that 16 warps issue on four schedulers as much as
// the loads they wait for.  The candidate and H_sub phases keep four to
// sixteen loads per thread in flight, and nothing of the iteration state that
// is not needed is copied.  Cycles per iteration before and after (12 orbitals
// 6a5b, k = 32, m = 64): candidates and scores 16,900 and 10,100, selection
// 10,100 and 5,700, H_sub 9,800 and 6,500, eig update 34,300 and 14,500, all
// 86,700 and 46,500; 24 orbitals, k = 96, m = 128: the update by the bordered
// form instead of the full reduction, 380 us and 107 us for the whole kernel.
#pragma once

#include "eig.cuh"
#include "device_common.cuh"
#include "kernels.h"
#include "select.cuh"

namespace mcd {
namespace {


constexpr int kLT = kEigThreads;  // 512
constexpr int kLW = kLT / 32;     // warps

// ---------------------------------------------------------------------------
// Matrix elements between two determinants.

__device__ __forceinline__ int lowest_bit(uint64_t x) { return __ffsll(static_cast<long long>(x)) - 1; }

// Single p->r of spin s summed over the occupied spin-orbitals of (a, b) in
// interleaved order, sixteen loads in flight.
__device__ __forceinline__ double single_value_det(const HamDev& h, int s, int p, int r, uint64_t a, uint64_t b) {
  const size_t base = (static_cast<size_t>(s) * h.norb + p) * h.norb + r;
  const double* st = h.st + base * h.nso;
  double v = __ldg(h.sh + base);
#pragma unroll 1
  while (a | b) {
    double t[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      t[j] = 0.0;
      const uint64_t u = a | b, bit = u & (0ull - u);
      if (u == 0ull) continue;
      const bool alpha = (a & bit) != 0ull;
      t[j] = __ldg(st + 2 * lowest_bit(u) + (alpha ? 0 : 1));
      if (alpha)
        a ^= bit;
      else
        b ^= bit;
    }
    // Adding 0.0 past the last orbital changes nothing but the sign of a zero.
#pragma unroll
    for (int j = 0; j < 16; ++j) v += t[j];
  }
  return v;
}

// <d2|H|d1> computed from d1's side, as HamiltonianMolecule::get_off_diagonal(d1, d2).
__device__ __forceinline__ double off_diagonal(const HamDev& h, Det d1, Det d2) {
  const uint64_t da = d1.a ^ d2.a, db = d1.b ^ d2.b;
  const int na = __popcll(da), nb = __popcll(db);
  const bool single = na + nb == 2;
  if ((!single && na + nb != 4) || (na & 1)) return 0.0;
  // The excitation p -> r, and q -> s for a double: alpha before beta, lower
  // orbitals first; beta1 and beta2 are their spins.
  const bool beta1 = na == 0, beta2 = na != 4;
  uint64_t o1 = beta1 ? db & d1.b : da & d1.a, v1 = beta1 ? db & d2.b : da & d2.a;
  const int p = lowest_bit(o1), r = lowest_bit(v1);
  int q = 0, s = 0;
  const int n = h.norb;
  double val;
  if (single) {
    const uint64_t stored = __ldg(h.spres + (beta1 ? n : 0) + p);
    val = single_value_det(h, beta1 ? 1 : 0, p, r, d1.a, d1.b);
    if (!((stored >> r) & 1ull)) return 0.0;
  } else {
    const size_t np = static_cast<size_t>(h.npair);
    const double* at;
    if (na == 2) {
      q = lowest_bit(db & d1.b);
      s = lowest_bit(db & d2.b);
      at = h.wab + ((static_cast<size_t>(p) * n + q) * n + r) * n + s;
    } else {
      q = lowest_bit(o1 & (o1 - 1));
      s = lowest_bit(v1 & (v1 - 1));
      at = h.vss + ((beta1 ? np : 0) + pair_index(p, q)) * np + pair_index(r, s);
    }
    val = __ldg(at);
  }
  uint64_t a = d1.a, b = d1.b;
  unsigned neg = sign_one(beta1, a, b, p, r);
  (beta1 ? b : a) ^= (1ull << p) ^ (1ull << r);
  if (!single) neg ^= sign_one(beta2, a, b, q, s);
  return neg ? -val : val;
}

// Diagonal element of d by half a warp (16 lanes, the whole warp calling; d
// may differ between the halves): <i|h|i> over the occupied i and <ij||ij>
// over the occupied pairs i < j, row x of the pairs on lane x mod 16 with
// eight loads in flight, then a fixed reduction order.  occ: 128 bytes of
// scratch for each half.
__device__ __forceinline__ double diagonal_half(const HamDev& h, Det d, unsigned char* occ) {
  const int sub = threadIdx.x & 15;
  const int nocc = __popcll(d.a) + __popcll(d.b);
  // The occupied spin-orbitals in interleaved order, each at its rank.
  for (int s = sub; s < h.nso; s += 16) {
    const int p = s >> 1;
    const uint64_t below = (1ull << p) - 1ull;
    if ((((s & 1) ? d.b : d.a) >> p) & 1ull) {
      const int rank = __popcll(d.a & below) + __popcll(d.b & below) + ((s & 1) ? static_cast<int>((d.a >> p) & 1ull) : 0);
      occ[rank] = static_cast<unsigned char>(s);
    }
  }
  __syncwarp();
  double v = 0.0;
#pragma unroll 1
  for (int x = sub; x < nocc; x += 16) {
    const double* row = h.d2 + static_cast<size_t>(occ[x]) * h.nso;
    v += __ldg(h.hdiag + occ[x]);
#pragma unroll 1
    for (int y0 = x + 1; y0 < nocc; y0 += 8) {
      double t[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) t[j] = y0 + j < nocc ? __ldg(row + occ[y0 + j]) : 0.0;
      v += ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
    }
  }
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) v += __shfl_xor_sync(~0u, v, o);
  __syncwarp();
  return v + h.ecore;
}

// ---------------------------------------------------------------------------
// Eig update.  Inputs x[k], z[k] in shared memory; H (row-major k x k,
// symmetric: dsyevr with UPLO='L' on the row-major array reads its upper
// triangle, and callers fill the lower one from it) in shared or global
// memory; `work` is shared scratch of eig_work_doubles(k) doubles.  Outputs
// dx[k] (shared), new xx and scale.

struct EigResult {
  dd xx, scale;
  dd rq;              // the eigenvalue (Rayleigh quotient of the vector)
  int branch;
  bool ok;
  double resid;
  double lambda;     // rq rounded
  double max_evec;   // max |v_i| over i >= 1 (branch 1) or i >= 0 (branch 2)
  int shift_steps;   // steps of the shifted solver, 0 when the reduction ran
  double shift_diff; // change made by its last refinement step
  bool fallback;     // the shifted solver was tried and the reduction ran instead
};

constexpr int kEigVecs = 18;

// Shared scratch of eig_update: B (lda), 18 vectors, and for k + 1 <=
// kShiftMaxN the explicit inverse of the shifted solver's Cholesky factor
// and the inverse of B - sigma I formed from it.
__host__ __device__ constexpr size_t eig_work_doubles(int k) {
  return static_cast<size_t>(k + 1) * eig_lda(k + 1) + kEigVecs * static_cast<size_t>(k + 1) +
         (k + 1 <= kShiftMaxN ? 2 * static_cast<size_t>(k + 1) * eig_lda(k + 1) : 0) + 64;
}

// drop: the last update's energy drop E - lambda (0 = unknown).  When it is
// known and B has at most kShiftMaxN rows, the shifted solver runs first with
// sigma = E - max(16 drop, 1e-9 (1 + |E|)) below the current energy E = xz/xx
// (an upper bound of lambda_1: the current vector lies in the subspace, and
// its Rayleigh quotient there is xz/xx) and the current vector as the start;
// the reduction runs when that fails or its residual is not below 1e-11
// (1 + |lambda|).  Out of line, with the reduction itself: the usual update
// takes eig_update_bordered, and its code should be what the instruction
// cache holds.  x, z, dx and work are in shared memory.
__device__ __noinline__ EigResult eig_update_full(const double* H, int k, const double* x, const double* z, dd xx,
                                                  dd xz, double* dx, double* work, SectionClock& clk, double drop) {
  // (a function of its own does not see where its callers' arrays are)
  __builtin_assume(__isShared(x));
  __builtin_assume(__isShared(z));
  __builtin_assume(__isShared(dx));
  __builtin_assume(__isShared(work));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ double s_b00, s_y1, s_res;
  __shared__ dd s_sum3[3];
  __shared__ double s_sgn;
  __shared__ int s_branch;
  __shared__ dd s_rq;
  EigResult res;
  res.shift_steps = 0;
  res.shift_diff = 0.0;
  res.fallback = false;

  // B = [[b00, b'], [b, H]] in A (leading dimension lda); H's block at (1, 1)
  // also serves the first-iteration k x k problem.
  const int lda = eig_lda(k + 1);
  double* A = work;
  double* vec = work + static_cast<size_t>(k + 1) * lda;
  const int vs = k + 1;
  EigVecs V;
  V.d = vec;
  V.e = vec + vs;
  V.e2 = vec + 2 * vs;
  V.u0 = vec + 3 * vs;
  V.tau = vec + 4 * vs;
  V.num = vec + 5 * vs;
  V.den = vec + 6 * vs;
  V.ru = vec + 7 * vs;
  V.l = vec + 8 * vs;
  V.y = vec + 9 * vs;
  V.c = vec + 10 * vs;
  V.g = vec + 11 * vs;
  double* Hx = vec + 12 * vs;    // [k]
  double* bvec = vec + 13 * vs;  // [k+1] first row of B (branch 1)
  double* Bv = vec + 14 * vs;
  double* vhi = vec + 15 * vs;   // normalised eigenvector, hi part
  double* vlo = vec + 16 * vs;   // lo part

  double* Li = vec + kEigVecs * vs;   // [(k+1) x lda] when k + 1 <= kShiftMaxN
  double* Ci = Li + vs * lda;          // [(k+1) x lda] likewise
  auto fill_h = [&]() {
    for (int idx = tid; idx < k * k; idx += blockDim.x) {
      const int i = idx / k, j = idx - i * k;
      if (i <= j) {
        const double v = H[idx];
        A[(i + 1) * lda + (j + 1)] = v;
        A[(j + 1) * lda + (i + 1)] = v;
      }
    }
  };
  fill_h();
  __syncthreads();
  clk.mark(21);
  // H x in double (dsymv, src/solver.h:355); x'x, x'z, x'Hx in double-double,
  // rounded where the reference works in double.
  for (int r = warp; r < k; r += kLW) {
    const double* row = A + (r + 1) * lda + 1;
    double s = 0.0;
    for (int c = lane; c < k; c += 32) s = fma(row[c], x[c], s);
    s = warp_sum(s);
    if (lane == 0) Hx[r] = s;
  }
  __syncthreads();
  clk.mark(22);
  if (warp == 0) {
    dd sxx{0, 0}, sxz{0, 0}, sxhx{0, 0};
    for (int i = lane; i < k; i += 32) {
      sxx = dd_add(sxx, dd_two_prod(x[i], x[i]));
      sxz = dd_add(sxz, dd_two_prod(x[i], z[i]));
      sxhx = dd_add(sxhx, dd_two_prod(x[i], Hx[i]));
    }
    sxx = warp_sum_dd(sxx);
    sxz = warp_sum_dd(sxz);
    sxhx = warp_sum_dd(sxhx);
    if (lane == 0) {
      const double xTx = dd_to_d(sxx), xTz = dd_to_d(sxz), xTHx = dd_to_d(sxhx);
      const double yy = dd_to_d(dd_add_d(xx, -xTx));
      s_branch = fabs(yy) > 1e-14 ? 1 : 2;
      if (s_branch == 1) {
        const double y1 = sqrt(yy);
        dd num = dd_add_d(dd_add_d(xz, -2.0 * xTz), xTHx);
        s_b00 = dd_to_d(dd_div_d(num, yy));
        s_y1 = y1;
      }
    }
  }
  __syncthreads();
  clk.mark(23);
  const int branch = s_branch;
  const int n = branch == 1 ? k + 1 : k;
  const double y1 = s_y1;
  if (branch == 1) {
    // b = (z - Hx) / y1 (src/solver.h:378-383).
    for (int i = tid; i <= k; i += blockDim.x) {
      const double v = i == 0 ? s_b00 : (z[i - 1] - Hx[i - 1]) / y1;
      A[i] = v;
      A[i * lda] = v;
      bvec[i] = v;
    }
  }
  __syncthreads();
  clk.mark(9);

  double* Ae = branch == 1 ? A : A + lda + 1;
  bool shifted = false;
  if (branch == 1 && n <= kShiftMaxN && drop > 0.0) {
    const double e_cur = dd_to_d(dd_div(xz, xx));
    const double delta = fmax(16.0 * drop, 1e-9 * (1.0 + fabs(e_cur)));
    for (int i = tid; i < n; i += blockDim.x) V.y[i] = i == 0 ? y1 : x[i - 1];
    __syncthreads();
    int steps = 0;
    double diff = 0.0;
    shifted = eig_lowest_shifted_warp(A, lda, n, V, e_cur - delta, Li, Ci, &steps, &diff, clk);
    res.shift_steps = shifted ? steps : 0;
    res.shift_diff = shifted ? diff : 0.0;
    if (!shifted) {
      res.fallback = true;
      fill_h();
      for (int i = tid; i <= k; i += blockDim.x) {
        A[i] = bvec[i];
        A[i * lda] = bvec[i];
      }
      __syncthreads();
    }
  }
  clk.mark(16);

  bool reduce = !shifted;
#pragma unroll 1
  for (int attempt = 0; attempt < 2; ++attempt) {
  if (reduce) eig_lowest(Ae, lda, n, V, clk);
  clk.mark(13);
  // B v in double, one row per warp (H is symmetric, so its rows are read).
  const double* y = V.y;
  for (int r = warp; r < n; r += kLW) {
    double s = 0.0;
    if (branch == 1) {
      const double* hr = H + (r - 1) * k - 1;  // hr[c] = H[r-1][c-1]
      for (int c = lane; c < n; c += 32) {
        const double brc = (r == 0) ? bvec[c] : (c == 0 ? bvec[r] : hr[c]);
        s = fma(brc, y[c], s);
      }
    } else {
      const double* hr = H + r * k;
      for (int c = lane; c < n; c += 32) s = fma(hr[c], y[c], s);
    }
    s = warp_sum(s);
    if (lane == 0) Bv[r] = s;
  }
  __syncthreads();
  clk.mark(24);
  // Rayleigh quotient y'By / y'y, normalisation in double-double, sign fix,
  // residual ||B v - lambda v||: y'y on warp 0, y'Bv on warp 1 and, for the
  // first iteration's sign, y'x on warp 2; then warp 0 normalises while warp 1
  // forms the quotient and the residual.
  if (warp < 3) {
    dd acc{0, 0};
    double sgn = 0.0;
    for (int i = lane; i < n; i += 32) {
      if (warp == 2)
        sgn = branch == 2 ? fma(y[i], x[i], sgn) : 0.0;
      else
        acc = dd_add(acc, dd_two_prod(y[i], warp == 0 ? y[i] : Bv[i]));
    }
    if (warp == 2) {
      sgn = warp_sum(sgn);
      if (lane == 0) s_sgn = sgn;
    } else {
      acc = warp_sum_dd(acc);
      if (lane == 0) s_sum3[warp] = acc;
    }
  }
  __syncthreads();
  if (warp == 0) {
    const dd nrm = s_sum3[0];
    const double flip = (branch == 1) ? (y[0] < 0.0 ? -1.0 : 1.0) : (s_sgn < 0.0 ? -1.0 : 1.0);
    const dd inv = dd_div(dd{flip, 0.0}, dd_sqrt(nrm));
    for (int i = lane; i < n; i += 32) {
      const dd vi = dd_mul_d(inv, y[i]);
      vhi[i] = vi.hi;
      vlo[i] = vi.lo;
    }
  } else if (warp == 1) {
    const dd nrm = s_sum3[0];
    const dd rq = dd_div(s_sum3[1], nrm);
    const double lam = dd_to_d(rq);
    double acc = 0.0;
    for (int i = lane; i < n; i += 32) {
      const double t = fma(-lam, y[i], Bv[i]);
      acc = fma(t, t, acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      s_rq = rq;
      s_res = sqrt(acc / dd_to_d(nrm));
    }
  }
  __syncthreads();
  // A shifted solve whose residual is not small runs the reduction instead.
  if (!shifted || s_res <= 1e-11 * (1.0 + fabs(dd_to_d(s_rq)))) break;
  shifted = false;
  reduce = true;
  res.shift_steps = 0;
  res.shift_diff = 0.0;
  res.fallback = true;
  fill_h();
  for (int i = tid; i <= k; i += blockDim.x) {
    A[i] = bvec[i];
    A[i * lda] = bvec[i];
  }
  __syncthreads();
  }
  clk.mark(14);
  const dd rq = s_rq;
  const double lam = dd_to_d(rq);
  res.resid = s_res;
  res.branch = branch;
  res.ok = true;
  res.lambda = lam;
  res.rq = rq;
  {
    double mv = 0.0;
    if (warp == 0)
      for (int i = lane + (branch == 1 ? 1 : 0); i < n; i += 32) mv = fmax(mv, fabs(vhi[i]));
    for (int o = 16; o > 0; o >>= 1) mv = fmax(mv, __shfl_xor_sync(~0u, mv, o));
    res.max_evec = mv;  // warp 0's value; thread 0 publishes it
  }

  if (branch == 1) {
    // lambda_q = -rq, gamma = v0 / y1, scale = gamma sqrt(lambda_q),
    // xx = lambda_q / scale^2, dx_i = v_{i+1} / gamma - x_i (src/solver.h:516-538).
    const dd lq = dd_neg(rq);
    const dd v0{vhi[0], vlo[0]};
    const dd gamma = dd_div_d(v0, y1);
    res.ok = lq.hi > 0.0 && gamma.hi != 0.0 && isfinite(lq.hi) && isfinite(gamma.hi);
    const dd sc = dd_mul(gamma, dd_sqrt(lq));
    res.scale = sc;
    res.xx = dd_div(lq, dd_mul(sc, sc));
    for (int i = tid; i < k; i += blockDim.x) {
      const dd q = dd_div(dd{vhi[i + 1], vlo[i + 1]}, gamma);
      dx[i] = dd_to_d(dd_add_d(q, -x[i]));
    }
  } else {
    // First iteration: xx = -lambda, scale = 1, dx = v sqrt(-lambda) - x (src/solver.h:552-598).
    res.ok = lam < 0.0 && isfinite(lam);
    const double sq = sqrt(-lam);
    res.xx = dd{-lam, 0.0};
    res.scale = dd{1.0, 0.0};
    for (int i = tid; i < k; i += blockDim.x) dx[i] = (vhi[i] + vlo[i]) * sq - x[i];
  }
  __syncthreads();
  for (int i = tid; i < k; i += blockDim.x)
    if (!isfinite(dx[i])) res.ok = false;
  res.ok = __syncthreads_and(res.ok ? 1 : 0) != 0;
  return res;
}

// ---------------------------------------------------------------------------
// The eig update by the bordered fixed point, for every k: the lowest
// eigenpair of B = [[a, b'], [b, C]] (C = H, n = k + 1 rows) when it lies
// below the Gershgorin bound of C, g = min_i (C_ii - sum_{j != i} |C_ij|).  By
// Cauchy interlacing B has exactly one eigenvalue below lambda_1(C) >= g, so an
// approximate eigenpair (lambda, v) with lambda + ||B v - lambda v|| / ||v|| < g
// belongs to the lowest eigenvalue (some eigenvalue lies within the residual
// norm of lambda).  With v = (1, y), D the diagonal of C and E the rest, the
// last k rows of (B - lambda I) v = 0 read (D - lambda I) y = -(b + E y), and
// the first row lambda = a + b'y.  A step is
//     y <- -(b + E y) / (d - lambda),   lambda <- a + b'y,
// which contracts by about max_i sum_j |E_ij| / (d_i - lambda), less than 1
// whenever lambda < g (C is strongly diagonal in a subspace of picked
// determinants, most of which are not connected by a single or double
// excitation).  The product E y also gives the residual of the current
// iterate, r_i = (b + E y)_i + (d_i - lambda) y_i (row 0's is zero by the choice
// of lambda).  The start is the current vector, y = x / y1, which is within
// the update itself of the solution.  The reciprocal of d_i - lambda is a
// Newton-Raphson step from the last one, r <- r + r e with e = 1 - (d_i -
// lambda) r, while |e| < 1e-3, and a division otherwise; an inexact r changes
// only the step, not the fixed point.  The iteration stops when ||r|| / ||v||
// reaches 1e-15 max_i sum_j |B_ij| (or stalls within 16 times that), and gives
// up when it stops contracting or lambda is not below g.
//
// Bound by the latency of a step's chain.  One warp issues a shared-memory load
// about every ten cycles and a shuffle every six, so the row products are
// spread: row i of E is held in registers by four lanes (NJ values each), and
// ceil(k/8) warps take part.  A step has one named barrier, after the new y is
// in shared memory (two buffers in turn); then every warp forms b'y over all
// rows itself, from one load per 32 rows, beside the product for the step
// after.  The residual is tested at every second step, from successive y
// (r = (d - lambda) (y_t - y_{t+1}) but for the error of the reciprocal, at
// most 1e-3); the one that certifies is taken from the exact r.
// Cycles per step at k = 32: one warp over packed nonzeros 1,500; a row per
// lane and y read uniformly 1,340; four lanes per row with per-warp sums of
// b'y, rr and yy exchanged at every step 900; this form 700.
//
// With y_0 = 1 the update's formulas (src/solver.h:516-538: gamma = v_0 / y1,
// scale = gamma sqrt(-rq), xx = -rq / scale^2, dx_i = v_{i+1} / gamma - x_i,
// for the normalised v) become dx_i = y_i y1 - x_i, xx = |v|^2 y1^2 and
// scale = sqrt(-rq / xx), with rq = v'Bv / v'v; |v|^2 and v'Bv are summed in
// double-double, the rows of B v taken from the last step's products.

constexpr int kBorderIters = 64;

constexpr int kBorderWarps = kMaxK / 8;

struct BorderShared {
  double y[2][kMaxK];
  double b[kMaxK], d[kMaxK];
  double part[kBorderWarps][4];
  dd vv[kBorderWarps], vbv[kBorderWarps];  // (vv holds x'Hx before)
  dd xtx, xtz;
  double ymax[kBorderWarps];
  double lam, y1, resid;
  int ok, steps;
};

// Two double-double sums over the lanes whose numbers differ in the bits
// from `first` up to, not including, `last`, side by side: the high parts by
// exact two-sums, their errors and the low parts in one running sum, put
// together at the end (half the chain of normalised additions; the low sum's
// own rounding is 2^-53 of it).
__device__ __forceinline__ void lanes_sum_dd(dd& v, dd& w, int first, int last) {
#pragma unroll 1
  for (int o = first; o < last; o <<= 1) {
    const dd v2{__shfl_xor_sync(~0u, v.hi, o), __shfl_xor_sync(~0u, v.lo, o)};
    const dd w2{__shfl_xor_sync(~0u, w.hi, o), __shfl_xor_sync(~0u, w.lo, o)};
    const dd vs = dd_two_sum(v.hi, v2.hi), ws = dd_two_sum(w.hi, w2.hi);
    v = dd{vs.hi, (v.lo + v2.lo) + vs.lo};
    w = dd{ws.hi, (w.lo + w2.lo) + ws.lo};
  }
  v = dd_fast_two_sum(v.hi, v.lo);
  w = dd_fast_two_sum(w.hi, w.lo);
}

// x'x and x'z by one warp.
__device__ __forceinline__ void dots_dd(const double* x, const double* z, int k, dd& xtx, dd& xtz) {
  xtx = xtz = dd{0.0, 0.0};
#pragma unroll 1
  for (int i = threadIdx.x & 31; i < k; i += 32) {
    xtx = dd_add(xtx, dd_two_prod(x[i], x[i]));
    xtz = dd_add(xtz, dd_two_prod(x[i], z[i]));
  }
  lanes_sum_dd(xtx, xtz, 1, 32);
}

// A sum over the rows of a warp (a row's four lanes hold the same value).
__device__ __forceinline__ double rows_sum(double v) {
  v += __shfl_xor_sync(~0u, v, 4);
  v += __shfl_xor_sync(~0u, v, 8);
  return v + __shfl_xor_sync(~0u, v, 16);
}

// The sum of the four lanes of a row.
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(~0u, v, 1);
  return v + __shfl_xor_sync(~0u, v, 2);
}

// Threads [0, 32 ceil(k/8)), k <= 4 NJ.  S.xtx and S.xtz hold x'x and x'z.
// Leaves dx, the partial sums for bordered_scalars and S.ok: 1, 0 when the
// pair is not certified, -1 when its eigenvalue is not negative.
template <int NJ>
__device__ __forceinline__ void eig_bordered(BorderShared& S, const double* H, int k, const double* x, const double* z,
                                             dd xx, dd xz, double* dx) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = tid >> 2, q = tid & 3;
  const int nw = (k + 7) >> 3, T = 32 * nw;
  const bool own = row < k;
  // Columns q, q + 4, ...; H is symmetric: element (j, row) of row-major H.
  double e[NJ], d = 0.0, off = 0.0, hx = 0.0;
#pragma unroll
  for (int jj = 0; jj < NJ; ++jj) {
    const int j = q + 4 * jj;
    const double v = own && j < k ? H[static_cast<size_t>(j) * k + row] : 0.0;
    hx = fma(v, j < k ? x[j] : 0.0, hx);
    if (j == row) d = v;
    e[jj] = j == row ? 0.0 : v;
    off += fabs(e[jj]);
  }
  for (int i = tid; i < 2 * kMaxK; i += T) (&S.y[0][0])[i] = 0.0;  // rows that no thread has stay zero
  d = quad_sum(d);
  off = quad_sum(off);
  hx = quad_sum(hx);
  const double xi = own ? x[row] : 0.0;
  {
    dd part = dd_two_prod(xi, hx), none{0.0, 0.0};
    lanes_sum_dd(part, none, 4, 32);
    if (lane == 0) S.vv[warp] = part;
  }
  bar_named(1, T);
  // x'Hx, |rest|^2 and B's first row; x'Hx, x'z and x'x rounded to double
  // where the reference works in double.
  dd sum = lane < nw ? S.vv[lane] : dd{0.0, 0.0}, none{0.0, 0.0};
  lanes_sum_dd(sum, none, 1, nw);
  const double xtx = dd_to_d(S.xtx), xtz = dd_to_d(S.xtz);
  const double xthx = __shfl_sync(~0u, dd_to_d(sum), 0);
  const double yy0 = dd_to_d(dd_add_d(xx, -xtx));
  if (!(yy0 > 1e-14)) {  // no rest vector to border with
    if (tid == 0) S.ok = 0;
    return;
  }
  const double y1 = sqrt(yy0);
  // The quotient of a double-double and a double, rounded once: a double
  // quotient and its remainder.
  const dd num = dd_add_d(dd_add_d(xz, -2.0 * xtz), xthx);
  const double q0 = num.hi / yy0;
  const double a = q0 + (fma(-q0, yy0, num.hi) + num.lo) / yy0;
  const double b = own ? (z[row] - hx) / y1 : 0.0;

  // The start, and the sums and bounds over all rows that the tests need.
  double y = own ? xi / y1 : 0.0;
  double gl = own ? d - off : 1e300, nb = own ? fabs(d) + off + fabs(b) : 0.0;
  {
    const double by = rows_sum(b * y), babs = rows_sum(fabs(b));
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      const double g2 = __shfl_xor_sync(~0u, gl, o), n2 = __shfl_xor_sync(~0u, nb, o);
      gl = g2 < gl ? g2 : gl;
      nb = n2 > nb ? n2 : nb;
    }
    if (lane == 0) {
      S.part[warp][0] = by;
      S.part[warp][1] = babs;
      S.part[warp][2] = gl;
      S.part[warp][3] = nb;
    }
    if (q == 0) {
      S.y[0][row] = y;
      S.b[row] = b;
      S.d[row] = d;
    }
  }
  bar_named(1, T);
  double babs = 0.0, lam = a;
  gl = 1e300;
  nb = 0.0;
#pragma unroll 1
  for (int w = 0; w < nw; ++w) {
    lam += S.part[w][0];
    babs += S.part[w][1];
    const double g2 = S.part[w][2], n2 = S.part[w][3];
    gl = g2 < gl ? g2 : gl;
    nb = n2 > nb ? n2 : nb;
  }
  const double top = fabs(a) + babs, tol = 1e-15 * (nb > top ? nb : top), tol2 = tol * tol;
  const bool cold = !(lam < gl);
  if (cold) {  // a start from below instead; lambda is then not yet a + b'y
    bar_named(1, T);
    y = 0.0;
    if (q == 0) S.y[0][row] = 0.0;
    lam = (a < gl ? a : gl) - 1e-3 * (1.0 + fabs(a));
    bar_named(1, T);
  }
  // Rows lane, lane + 32, ... for the sums over all rows.
  constexpr int R = NJ <= 8 ? 1 : NJ / 8;
  double bl[R], dl[R], yl[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int j = lane + 32 * i;
    bl[i] = j < k ? S.b[j] : 0.0;
    dl[i] = j < k ? S.d[j] : 0.0;
    yl[i] = j < k ? S.y[0][j] : 0.0;
  }
  // E y over this thread's columns, then the row.
  auto product = [&](int buf) {
    const double* ys = S.y[buf] + q;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int jj = 0; jj < NJ; jj += 2) {
      s0 = fma(e[jj], ys[4 * jj], s0);
      s1 = fma(e[jj + 1], ys[4 * jj + 4], s1);
    }
    return b + quad_sum(s0 + s1);
  };
  double rcp = own ? 1.0 / (d - lam) : 0.0;
  double rrp = 1e300, vvp = 1.0;  // |r|^2 and |v|^2 at the previous test
  double s = product(0);
  int done = 0, t = 0;
  // y_t -> y_{t+1}: s, lambda and the reciprocal follow; with `test`, whether
  // (lambda_t, y_t) ends the iteration (1 converged, -1 given up), before
  // anything of it is replaced.
  auto step = [&](int buf, bool test) {
    const double yn = -s * rcp;  // rows beyond k: rcp = 0
    if (q == 0) S.y[buf ^ 1][row] = yn;
    bar_named(1, T);
    double by = 0.0, rr = 0.0, vv = 0.0, yn_l[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      yn_l[i] = lane + 32 * i < k ? S.y[buf ^ 1][lane + 32 * i] : 0.0;
      by = fma(bl[i], yn_l[i], by);
      const double ri = (dl[i] - lam) * (yl[i] - yn_l[i]);
      rr = fma(ri, ri, rr);
      vv = fma(yl[i], yl[i], vv);
    }
    const double sn = product(buf ^ 1);
    by = warp_sum(by);
    if (test) {
      rr = warp_sum(rr);
      vv = 1.0 + warp_sum(vv);
      // rn <= tol, or rn > rn_prev / 4 (two steps before) and rn <= 16 tol
      // (stalled at rounding); squared norms cross-multiplied, no division
      const bool small = rr <= tol2 * vv || (t >= 2 && rr * vvp > 0.0625 * rrp * vv && rr <= 256.0 * tol2 * vv);
      if (small && !(cold && t == 0)) {
        done = 1;
        return;
      }
      // not finite, not contracting (rn > 0.8 rn_prev), or lambda not below g
      if (!(rr < 1e290 && vv < 1e290) || (t >= 8 && rr * vvp > 0.64 * rrp * vv) || (t >= 4 && !(lam < gl))) {
        done = -1;
        return;
      }
      rrp = rr;
      vvp = vv;
    }
    y = yn;
    s = sn;
    lam = a + by;
#pragma unroll
    for (int i = 0; i < R; ++i) yl[i] = yn_l[i];
    const double den = d - lam, err = fma(-den, rcp, 1.0);  // relative error of rcp as 1 / den
    if (__any_sync(~0u, own && fabs(err) >= 1e-3))
      rcp = own ? 1.0 / den : 0.0;
    else
      rcp = fma(rcp, err, rcp);
  };
#pragma unroll 1
  for (; t < kBorderIters; t += 2) {
    step(0, true);
    if (done != 0) break;
    step(1, false);
  }
  int ok = 0;
  double rn = 0.0;
  if (done == 1) {  // (uniform over the threads: all sums are formed the same way)
    const double ri = own && q == 0 ? fma(d - lam, y, s) : 0.0, yi = q == 0 ? y : 0.0;
    const double rr = rows_sum(quad_sum(ri * ri)), vv = rows_sum(quad_sum(yi * yi));
    if (lane == 0) {
      S.part[warp][0] = rr;
      S.part[warp][1] = vv;
    }
    bar_named(1, T);
    double rrs = 0.0, vvs = 1.0;
#pragma unroll 1
    for (int w = 0; w < nw; ++w) {
      rrs += S.part[w][0];
      vvs += S.part[w][1];
    }
    rn = sqrt(rrs / vvs);
    ok = rn <= 16.0 * tol && lam + rn < gl ? 1 : 0;
  }
  if (!ok) {
    if (tid == 0) S.ok = 0;
    return;
  }
  // dx, and |v|^2 and v'Bv over the rows; row 0 of B v is lambda.
  if (own && q == 0) dx[row] = dd_to_d(dd_add_d(dd_two_prod(y, y1), -xi));
  dd vv = dd_two_prod(y, y), vbv = dd_two_prod(y, own ? fma(d, y, s) : 0.0);
  lanes_sum_dd(vv, vbv, 4, 32);
  double ym = fabs(y);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    const double m2 = __shfl_xor_sync(~0u, ym, o);
    ym = m2 > ym ? m2 : ym;
  }
  if (lane == 0) {
    S.vv[warp] = vv;
    S.vbv[warp] = vbv;
    S.ymax[warp] = ym;
  }
  if (tid == 0) {
    S.ok = lam < 0.0 ? 1 : -1;
    S.steps = t + 1;
    S.resid = rn;
    S.lam = lam;
    S.y1 = y1;
  }
}

// The update's scalars from what eig_bordered left in S, by one warp, after a
// barrier: lane 0 returns them.
__device__ __forceinline__ EigResult bordered_scalars(const BorderShared& S, int k) {
  const int lane = threadIdx.x & 31, nw = (k + 7) >> 3;
  dd vv = lane < nw ? S.vv[lane] : dd{0.0, 0.0}, vbv = lane < nw ? S.vbv[lane] : dd{0.0, 0.0};
  lanes_sum_dd(vv, vbv, 1, nw < 2 ? 2 : nw);  // lanes 0 and 1 both
  double ym = 0.0;
#pragma unroll 1
  for (int w = 0; w < nw; ++w) ym = S.ymax[w] > ym ? S.ymax[w] : ym;
  const dd nrm = dd_add_d(vv, 1.0), num = dd_add_d(vbv, S.lam);
  const dd nxx = dd_mul(nrm, dd_two_prod(S.y1, S.y1));
  // Lane 0: rq = num / nrm.  Lane 1: the root of -rq / xx = -num / (nrm xx).
  const dd quo = dd_div(lane == 0 ? num : dd_neg(num), lane == 0 ? nrm : dd_mul(nrm, nxx));
  const dd root = dd_sqrt(dd_abs(quo));
  EigResult r;
  r.xx = nxx;
  r.scale = dd{__shfl_sync(~0u, root.hi, 1), __shfl_sync(~0u, root.lo, 1)};
  r.rq = quo;
  r.lambda = dd_to_d(quo);
  r.branch = 1;
  r.ok = true;
  r.resid = S.resid;
  r.max_evec = ym * rsqrt(nrm.hi);
  r.shift_steps = S.steps;
  r.shift_diff = S.resid;
  r.fallback = false;
  return r;
}

// The bordered update of a whole CTA; S.xtx and S.xtz are set, after a
// barrier.  Returns S.ok, in every thread.
__device__ __forceinline__ int eig_update_bordered(BorderShared& S, const double* H, int k, const double* x,
                                                   const double* z, dd xx, dd xz, double* dx) {
  if (static_cast<int>(threadIdx.x >> 5) < (k + 7) >> 3) {
    if (k <= 16)
      eig_bordered<4>(S, H, k, x, z, xx, xz, dx);
    else if (k <= 32)
      eig_bordered<8>(S, H, k, x, z, xx, xz, dx);
    else if (k <= 64)
      eig_bordered<16>(S, H, k, x, z, xx, xz, dx);
    else
      eig_bordered<32>(S, H, k, x, z, xx, xz, dx);
  }
  __syncthreads();
  return S.ok;
}

// The eig update on its own (the debug entry points): the bordered fixed
// point first with method 2, eig_update_full otherwise or when it does not
// certify its result (and for the first iteration, which has no bordering
// row).  Block-wide; every thread gets the result.
__device__ __forceinline__ EigResult eig_update(const double* H, int k, const double* x, const double* z, dd xx, dd xz,
                                                double* dx, double* work, SectionClock& clk, double drop, int method) {
  __shared__ BorderShared S;
  __shared__ EigResult s_res;
  bool tried = false;
  if (method == 2) {
    if (threadIdx.x < 32) {
      dd xtx, xtz;
      dots_dd(x, z, k, xtx, xtz);
      if (threadIdx.x == 0) {
        S.xtx = xtx;
        S.xtz = xtz;
      }
    }
    __syncthreads();
    const int ok = eig_update_bordered(S, H, k, x, z, xx, xz, dx);
    if (ok != 0) {
      if (threadIdx.x < 32) {
        EigResult r = bordered_scalars(S, k);
        r.ok = ok > 0;
        if (threadIdx.x == 0) s_res = r;
      }
      __syncthreads();
      return s_res;
    }
    tried = true;
  }
  EigResult res = eig_update_full(H, k, x, z, xx, xz, dx, work, clk, drop);
  if (tried && res.branch == 1) res.fallback = true;
  return res;
}

// ---------------------------------------------------------------------------
// End of iteration t (src/wavefunction.h:557-565,583): z[D_c] = new_z_c for
// the picked determinants, then xz += sum_c dot_c.  Block-wide, on a state
// copy `S` (shared or global); table stores go to global memory.
__device__ void finish_iteration(IterState* S, const TableDev& T) {
  if (!S->pending) return;
  const int k = S->k_cur;
  if (static_cast<int>(threadIdx.x) < k) {
    Slot* sp = T.slots + S->slot[threadIdx.x];
    sp->z = S->newz[threadIdx.x];
  }
  __syncthreads();  // orders the stores for this CTA; the next launch sees them anyway
  if (threadIdx.x < 32) {
    dd acc{0.0, 0.0};
    for (int c = threadIdx.x; c < k; c += 32) acc = dd_add_d(acc, S->dot[c]);
    acc = warp_sum_dd(acc);
    if (threadIdx.x == 0) {
      S->xz = dd_add(S->xz, acc);
      S->pending = 0;
    }
  }
  __syncthreads();
}

__global__ void finish_kernel(LeaderLaunch L) { finish_iteration(L.st, L.tab); }

__device__ __forceinline__ unsigned hash32(unsigned x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// The candidates of one iteration, in dynamic shared memory: the slots of up
// to PR candidates (kNoSlot for one seen before), and a hash set of 2 PR words
// that the candidates' keys replace once it has served.
struct Candidates {
  unsigned* slot;
  unsigned* set;
  unsigned long long* key;
  int n;   // entries in use
  int pr;  // a power of two
};

// Full sort by decreasing key, equal keys in the reference's determinant
// order (rare: the k-th and (k+1)-th keys are equal); the first k slots to out.
// Where that is no order of all determinants (norb >= 32, det_ref_compare) the
// outcome depends on the candidates' places, which differ from run to run: a
// pass before puts equal keys by their larger occupation strings.
__device__ __noinline__ void sort_candidates(const Candidates& C, int k, const Slot* slots, int nwords, int norb,
                                             unsigned* out) {
  int P = 1;
  while (P < C.n) P <<= 1;
  for (int u = C.n + threadIdx.x; u < P; u += kLT) {
    C.key[u] = 0ull;
    C.slot[u] = kNoSlot;
  }
  __syncthreads();
#pragma unroll 1
  for (int pass = norb < 32 ? 1 : 0; pass < 2; ++pass) {
    for (int size = 2; size <= P; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int t = threadIdx.x; t < (P >> 1); t += kLT) {
          const int i = 2 * stride * (t / stride) + (t % stride);
          const int j = i + stride;
          const unsigned long long ki = C.key[i], kj = C.key[j];
          bool jfirst = kj > ki;
          if (ki == kj && ki != 0ull) {
            uint64_t ia, ib, ja, jb;
            load_key(slots + C.slot[i], ia, ib);
            load_key(slots + C.slot[j], ja, jb);
            jfirst = pass == 0 ? ja > ia || (ja == ia && jb > ib) : det_ref_compare(ja, jb, ia, ib, nwords) > 0;
          }
          const bool up = (i & size) == 0;
          if (jfirst == up && (ki != kj || ki != 0ull)) {
            C.key[i] = kj;
            C.key[j] = ki;
            const unsigned tmp = C.slot[i];
            C.slot[i] = C.slot[j];
            C.slot[j] = tmp;
          }
        }
        __syncthreads();
      }
    }
  }
  if (threadIdx.x < k) out[threadIdx.x] = C.slot[threadIdx.x];
  __syncthreads();
}

// The ranks of k picked keys once more, for equal ones that det_ref_compare
// leaves in a circle (two of them then have the same number of determinants
// sorted before them, and a place stays empty): by that number, and where it is
// equal by the larger occupation strings.
__device__ __noinline__ void rank_circular(const unsigned long long* key, const unsigned* slot, int k, const Slot* slots,
                                           int nwords, unsigned* out) {
  __shared__ unsigned char s_before[kMaxK];
  const int i = threadIdx.x;
  const unsigned long long mine = i < k ? key[i] : 0ull;
  uint64_t ia = 0, ib = 0;
  int before = 0;
  if (i < k) {
    load_key(slots + slot[i], ia, ib);
    for (int j = 0; j < k; ++j) {
      if (j == i || key[j] != mine) continue;
      uint64_t ja, jb;
      load_key(slots + slot[j], ja, jb);
      before += det_ref_compare(ja, jb, ia, ib, nwords) > 0;
    }
    s_before[i] = static_cast<unsigned char>(before);
  }
  __syncthreads();
  if (i < k) {
    int rank = 0;
    for (int j = 0; j < k; ++j) {
      rank += key[j] > mine;
      if (j == i || key[j] != mine) continue;
      uint64_t ja, jb;
      load_key(slots + slot[j], ja, jb);
      const int bj = s_before[j];
      rank += bj < before || (bj == before && (ja > ia || (ja == ia && jb > ib)));
    }
    out[rank] = slot[i];
  }
  __syncthreads();
}

__device__ __forceinline__ void leader_body(const LeaderLaunch& L) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) IterState sS;  // the scalars; the per-column arrays stay in global memory
  __shared__ SelectScratch s_sel;
  __shared__ unsigned s_err, s_out, s_newx;
  __shared__ dd s_xz;
  __shared__ unsigned s_slot[kMaxK], s_sel_slot[kMaxK];
  __shared__ unsigned long long s_sel_key[kMaxK];
  __shared__ Det s_det[kMaxK];
  __shared__ double s_x[kMaxK], s_z[kMaxK], s_dx[kMaxK];
  __shared__ unsigned char s_occ[2 * kLW][128];
  __shared__ BorderShared s_border;

  IterState* G = L.st;
  const TableDev& T = L.tab;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = L.m;
  SectionClock clk{L.sect, 0};
  clk.start();

  Candidates C;
  C.pr = 4;
  while (C.pr < L.k_req * m) C.pr <<= 1;
  C.slot = reinterpret_cast<unsigned*>(smem);
  C.set = C.slot + C.pr;
  C.key = reinterpret_cast<unsigned long long*>(C.set);
  for (int i = tid; i < C.pr / 2; i += kLT)
    reinterpret_cast<uint4*>(C.set)[i] = make_uint4(kNoSlot, kNoSlot, kNoSlot, kNoSlot);
  if (tid == 0) s_out = s_newx = 0u;
  if (tid < kMaxK) s_slot[tid] = kNoSlot;

  pdl_wait();  // for the column kernel

  // 1. The scalars into shared memory, and the end of the previous iteration
  //    (src/wavefunction.h:557-565,583; unless finish_kernel already did):
  //    z[D_c] = new_z_c for the picked determinants, xz += sum_c dot_c.
  const int kprev = __ldcg(&G->k_cur);
  const int pending = __ldcg(&G->pending);
  unsigned cand[4];  // the first candidates, whatever kprev is
#pragma unroll
  for (int j = 0; j < 4; ++j) cand[j] = tid + j * kLT < L.k_req * m ? __ldcg(L.cand_slot + tid + j * kLT) : kNoSlot;
  {
    constexpr int kHead = offsetof(IterState, k_cur) / 8, kTail = offsetof(IterState, x_size) / 8;
    constexpr int kWords = sizeof(IterState) / 8;
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(G);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sS);
    const int i = tid < kHead ? tid : kTail + tid - kHead;
    if (i < kWords) dst[i] = src[i];
  }
  if (tid == kLT - 1) {
    s_err = *reinterpret_cast<volatile unsigned*>(T.err);
    if (*T.n_occupied > L.st->occupancy_limit) {
      atomicOr(T.err, kErrOverflow);
      s_err |= kErrOverflow;
    }
  }
  if (pending && tid < kprev) T.slots[__ldcg(&G->slot[tid])].z = __ldcg(&G->newz[tid]);
  C.n = kprev * m;
  __syncthreads();
  clk.mark(0);

  // 2. Candidate slots, with duplicates (one determinant in several columns)
  //    removed through a shared-memory hash set: the first copy stays.
  if (warp == kLW - 1) {
    dd acc{0.0, 0.0}, none{0.0, 0.0};
    if (pending)
      for (int c = lane; c < kprev; c += 32) acc = dd_add_d(acc, __ldcg(&G->dot[c]));
    lanes_sum_dd(acc, none, 1, 32);
    if (lane == 0) s_xz = dd_add(sS.xz, acc);
  }
#pragma unroll 1
  for (int r0 = tid; r0 < C.n; r0 += 4 * kLT) {
    if (r0 != tid) {
#pragma unroll
      for (int j = 0; j < 4; ++j) cand[j] = r0 + j * kLT < C.n ? __ldcg(L.cand_slot + r0 + j * kLT) : kNoSlot;
    }
    const unsigned mask = static_cast<unsigned>(2 * C.pr - 1);
    unsigned old[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (r0 + j * kLT >= C.n) cand[j] = kNoSlot;
      old[j] = kNoSlot;
      if (cand[j] != kNoSlot) old[j] = atomicCAS(&C.set[hash32(cand[j]) & mask], kNoSlot, cand[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      unsigned h = hash32(cand[j]);
#pragma unroll 1
      while (old[j] != kNoSlot && old[j] != cand[j]) old[j] = atomicCAS(&C.set[++h & mask], kNoSlot, cand[j]);
      if (r0 + j * kLT < C.n) C.slot[r0 + j * kLT] = old[j] == kNoSlot ? cand[j] : kNoSlot;
    }
  }
  __syncthreads();
  clk.mark(1);

  // 3. Their scores |x*xx*scale^2 + z|, refetched from the table
  //    (src/wavefunction.h:567-575), and the k largest by radix selection.
  {
    const dd xss = sS.xss;
#pragma unroll 1
    for (int r0 = tid; r0 < C.n; r0 += 4 * kLT) {
      double x[4], z[4];
      bool some[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned s = r0 + j * kLT < C.n ? C.slot[r0 + j * kLT] : kNoSlot;
        some[j] = s != kNoSlot;
        x[j] = z[j] = 0.0;
        if (some[j]) load_xz(T.slots + s, x[j], z[j]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double g = score_of(x[j], z[j], xss);
        // (a non-finite gradient must not reorder the rest)
        if (r0 + j * kLT < C.n) C.key[r0 + j * kLT] = some[j] ? score_key(g >= 0.0 ? g : 0.0) : 0ull;
      }
    }
  }
  __syncthreads();
  clk.mark(2);
  const SelectEdge E = select_edge(s_sel, static_cast<unsigned>(L.k_req), [&](auto f) {
#pragma unroll 1
    for (int r0 = tid; r0 < C.n; r0 += 4 * kLT) {
      unsigned long long key[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) key[j] = r0 + j * kLT < C.n ? C.key[r0 + j * kLT] : 0ull;
#pragma unroll
      for (int j = 0; j < 4; ++j) f(key[j]);
    }
  });
  if (s_err != 0u || E.total == 0u) {
    if (tid == 0) {
      if (E.total == 0u && s_err == 0u) atomicOr(T.err, kErrCandidates);
      G->xz = s_xz;
      G->pending = 0;
      G->k_cur = 0;
    }
    return;
  }
  const int k = static_cast<int>(min(E.total, static_cast<unsigned>(L.k_req)));

  // 4. In decreasing score, equal scores in the reference's determinant order
  //    (detComp_global, src/wavefunction.h:30-36).
  if (!E.tied) {
#pragma unroll 4
    for (int r = tid; r < C.n; r += kLT) {
      const unsigned long long key = C.key[r];
      if (key < E.edge) continue;
      const unsigned pos = atomicAdd(&s_out, 1u);
      s_sel_key[pos] = key;
      s_sel_slot[pos] = C.slot[r];
    }
    __syncthreads();
    clk.mark(3);
    // Ranks by counting, 16 lanes per key; a place that two keys claim shows
    // equal keys without an order of their own.
    const int part = tid & 15;
    bool claimed = false;
#pragma unroll 1
    for (int i0 = 0; i0 < k; i0 += kLT / 16) {
      const int i = i0 + (tid >> 4);
      const unsigned long long mine = i < k ? s_sel_key[i] : 0ull;
      unsigned rank = 0, equal = 0;
      for (int j = part; j < k; j += 16) {
        const unsigned long long o = s_sel_key[j];
        rank += o > mine ? 1u : 0u;
        equal += o == mine ? 1u : 0u;
      }
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        rank += __shfl_xor_sync(~0u, rank, o);
        equal += __shfl_xor_sync(~0u, equal, o);
      }
      if (part == 0 && i < k) {
        const unsigned slot = s_sel_slot[i];
        if (equal > 1u) {
          uint64_t ia, ib;
          load_key(T.slots + slot, ia, ib);
          for (int j = 0; j < k; ++j) {
            if (j == i || s_sel_key[j] != mine) continue;
            uint64_t ja, jb;
            load_key(T.slots + s_sel_slot[j], ja, jb);
            rank += det_ref_compare(ja, jb, ia, ib, sS.n_words) > 0 ? 1u : 0u;
          }
        }
        claimed |= atomicExch(&s_slot[rank], slot) != kNoSlot;
      }
    }
    if (__syncthreads_or(claimed)) rank_circular(s_sel_key, s_sel_slot, k, T.slots, sS.n_words, s_slot);
  } else {
    __syncthreads();
    sort_candidates(C, k, T.slots, sS.n_words, L.ham.norb, s_slot);
  }
  clk.mark(4);
  if (tid < k) {
    const Slot* sp = T.slots + s_slot[tid];
    uint64_t a, b;
    load_key(sp, a, b);
    s_det[tid] = Det{a, b};
    load_xz(sp, s_x[tid], s_z[tid]);
    // The picks go out now, so that the column kernel can enumerate and probe
    // their columns while the subspace problem is solved here.
    G->det[tid] = s_det[tid];
    G->slot[tid] = s_slot[tid];
    if (tid == 0) G->k_cur = k;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) pdl_trigger();
  clk.mark(5);

  // 5. H_sub: in shared memory when it fits beside the eig scratch, else in
  //    the global copy (which is written either way for inspection).
  const bool h_in_smem = k <= 64;
  double* Hs = h_in_smem ? reinterpret_cast<double*>(smem) : L.hsub_out;
  double* work = h_in_smem ? Hs + k * k : reinterpret_cast<double*>(smem);
  // One thread per pair i < j (pair t = j(j-1)/2 + i).
#pragma unroll 1
  for (int t = tid; t < k * (k - 1) / 2; t += kLT) {
    int j = static_cast<int>((1.0f + sqrtf(1.0f + 8.0f * static_cast<float>(t))) * 0.5f);
    if (j * (j - 1) / 2 > t) --j;
    if (j * (j + 1) / 2 <= t) ++j;
    const int i = t - j * (j - 1) / 2;
    const double v = off_diagonal(L.ham, s_det[i], s_det[j]);
    Hs[i * k + j] = v;
    Hs[j * k + i] = v;
  }
#pragma unroll 1
  for (int i0 = 0; i0 < k; i0 += 2 * kLW) {
    const int i = i0 + (tid >> 4);
    const double v = diagonal_half(L.ham, s_det[min(i, k - 1)], s_occ[tid >> 4]);
    if ((tid & 15) == 0 && i < k) Hs[i * k + i] = v;
  }
  if (warp == kLW - 1) {
    dd xtx, xtz;
    dots_dd(s_x, s_z, k, xtx, xtz);
    if (lane == 0) {
      s_border.xtx = xtx;
      s_border.xtz = xtz;
    }
  }
  __threadfence_block();
  __syncthreads();
  clk.mark(6);
  if (h_in_smem)
    for (int t = tid; t < k * k; t += kLT) L.hsub_out[t] = Hs[t];
  {
    double* in = L.hsub_out + kMaxK * kMaxK;
    if (tid < k) {
      in[tid] = s_x[tid];
      in[kMaxK + tid] = s_z[tid];
    }
    if (tid == 0) {
      in[2 * kMaxK] = sS.xx.hi;
      in[2 * kMaxK + 1] = sS.xx.lo;
      in[2 * kMaxK + 2] = s_xz.hi;
      in[2 * kMaxK + 3] = s_xz.lo;
    }
  }

  // 6. Eig update: the bordered fixed point with method 2, the full solver
  //    otherwise or when it does not certify its result (and for the first
  //    iteration, which has no bordering row).
  int fast = 0;
  EigResult er;
  if (L.eig_method == 2) {
    fast = eig_update_bordered(s_border, Hs, k, s_x, s_z, sS.xx, s_xz, s_dx);
    clk.mark(16);
  }
  if (fast == 0) {
    er = eig_update_full(Hs, k, s_x, s_z, sS.xx, s_xz, s_dx, work, clk, L.eig_method == 1 ? sS.eig_drop : 0.0);
    if (L.eig_method == 2 && er.branch == 1) er.fallback = true;
  }
  clk.mark(15);
  if (fast < 0 || (fast == 0 && !er.ok)) {
    if (tid == 0) {
      atomicOr(T.err, kErrEig);
      G->xz = s_xz;
      G->pending = 0;
      G->k_cur = 0;
    }
    return;
  }

  // 7. update_x: x[D_i] += dx_i; xz += z_i dx_i; x_size counts dets whose x was 0.
  if (tid < k) {
    T.slots[s_slot[tid]].x = s_x[tid] + s_dx[tid];
    if (s_x[tid] == 0.0) atomicAdd(&s_newx, 1u);
    G->dx[tid] = s_dx[tid];
    G->hdiag[tid] = Hs[tid * k + tid];
  }
  __syncthreads();
  clk.mark(7);

  // 8. Publish the next iteration: the eigenvalue's part on warp 0, the sums
  //    over the picks on warp 1.
  if (warp == 1) {
    dd zdx{0.0, 0.0}, none{0.0, 0.0};
    double mx = 0.0;
#pragma unroll 1
    for (int i = lane; i < k; i += 32) {
      zdx = dd_add_d(zdx, s_z[i] * s_dx[i]);
      mx = fmax(mx, fabs(s_dx[i]));
    }
    lanes_sum_dd(zdx, none, 1, 32);
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(~0u, mx, o));
    if (lane == 0) {
      G->xz = dd_add(s_xz, zdx);
      G->dx_max = mx;
    }
  } else if (warp == 0) {
    if (fast > 0) er = bordered_scalars(s_border, k);
    if (tid != 0) return;
    G->xx = er.xx;
    G->scale = er.scale;
    G->xss = fast > 0 ? dd_neg(er.rq) : dd_mul(er.xx, dd_mul(er.scale, er.scale));
    G->x_size = sS.x_size + s_newx;
    G->eig_residual_max = fmax(sS.eig_residual_max, er.resid);
    G->last_branch = er.branch;
    // Energy drop of this update, for the next one's shift: the current
    // energy xz/xx minus the eigenvalue (the energy after the update).
    // (only the shifted solver, eig_method 1, uses it)
    double drop = 0.0;
    if (L.eig_method == 1 && er.branch == 1) drop = fmax(dd_to_d(dd_div(s_xz, sS.xx)) - er.lambda, 1e-300);
    G->eig_drop = drop;
    G->max_abs_evec = er.max_evec;
    G->inv_steps_curr = er.shift_steps;
    G->inv_diff_curr = er.shift_diff;
    if (er.shift_steps > 0) {
      G->inv_updates = sS.inv_updates + 1;
      G->inv_steps = sS.inv_steps + er.shift_steps;
      G->inv_diff_sum = sS.inv_diff_sum + er.shift_diff;
      G->inv_diff_max = fmax(sS.inv_diff_max, er.shift_diff);
    }
    if (er.fallback) G->eig_fallbacks = sS.eig_fallbacks + 1;
    G->emitted = 0;
    G->updates = 0;
    G->iter = sS.iter + 1;
    G->pending = 1;
    clk.mark(8);
  }
}

}  // namespace
}  // namespace mcd
