// Small dense FP64 (generalized) symmetric eigenproblems on the device.
//
// Replaces the host LAPACKE dsyev/dsygv wrappers of the reference (CPP/linalg/blas/mvops.cu:1601-1664)
// and MATLAB eig(VAV, VV + tau I) inside eig_rr.m:50-54 / svd_rr.m:58-77.
// Algorithm: Cholesky M = L L' (right-looking), C = L^-1 G L^-T (two forward substitutions), cyclic
// Jacobi on C with round-robin parallel ordering (n/2 disjoint rotations per round, Golub & Van Loan
// sym.Schur2 rotation), eigenvalue sort, U = L^-T W.
// The eigenvectors are M-orthonormal (U' M U = I), the LAPACK sygv / MATLAB 'chol' normalisation.
// Orders up to kGeigClusterMaxN (144: what the Cholesky and substitution kernels hold in one CTA's shared
// memory) run the Jacobi sweeps on a thread-block cluster (k_jacobi_cluster); larger ones run the whole
// algorithm on one CTA in a global workspace (k_geig_sym).
#include <atomic>

#include "f64_ops.cuh"
#include "ofrr_internal.cuh"

namespace ofrr {

// ======================================================================================
// Jacobi sweeps on a cluster
// ======================================================================================
// GB300 runs FP64 at 1/64 of its FP32 rate (a warp instruction occupies an SM sub-partition for about 64
// cycles), so the sweeps are bound by the FP64 pipe of the SMs they run on and, between two barriers, by
// the dependent chain that turns (a_pp, a_qq, a_pq) into a rotation (measured on 16 CTAs at n = 64, cycles
// per round: rotations ~1700, C 1100, handing over 100, barrier 1180).  The rotations of a round are
// independent, so they are spread over a cluster: CTA c owns the seats of PP = ceil(N / 2 / NC) pairs of
// the round-robin schedule, i.e. 2 PP columns of C and of W.  Rows and columns of a 2 x 2 block only
// depend on that block, so a round is one pass over the CTA's columns; the new columns go straight to the
// CTA that holds their seat in the next round (every seat moves by one), into the other of two buffers
// through distributed shared memory, and the three entries each next rotation needs go to every CTA.  So
// a round costs one cluster barrier, and every CTA computes all rotations itself (N / 2 threads; the
// chain's latency does not depend on how many warps run it, up to one per sub-partition).
constexpr int kJacT = 512;
constexpr int kGeigClusterMaxN = 144;  // Cholesky, substitutions and L beside 32 columns in one CTA's 227 KB

// The rotation of sym.Schur2 (t the root of smaller magnitude of t^2 + 2 tau t - 1 = 0, t = 1 for tau = 0).
// The chain's divisions and square roots (560 and 630 cycles each as plain operations) were the largest part of a
// round, 3260 cycles; in their short forms (f64_ops.cuh) it takes half of that.  They stay undecided between neighbours
// (1/2 + 2^-33 units in the last place instead of 1/2; another value than the plain operation's once in 2^33 random ones):
// a rotation needs c^2 + s^2 = 1 to a few units, and the five decisions take 400 cycles of a round's 6,000 (4 % of a
// 64-order solve).  Taking the angle in FP32 and normalising (c, s) in FP64 would shorten the chain as much, but on the
// SVD pencil [[0, K], [K', 0]] of a block U ~ A V the matrix K is triangular up to rounding, equal diagonal entries
// meet entries of rounding size, and which of the two roots is taken (the sign of the vectors) then hangs on the
// last bits: the quotients keep results what the one-CTA form gives.
__device__ __forceinline__ bool jac_nonzero(double x) {  // an FP64 compare costs ~100 cycles
  return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) != 0;
}
__device__ __forceinline__ void jac_rotation(double app, double aqq, double apq, double* c, double* s) {
  *c = 1.0;
  *s = 0.0;
  if (!jac_nonzero(apq)) return;
  const double tau = f64::div<false>(aqq - app, 2.0 * apq);
  const double t = f64::rcp<false>(fabs(tau) + f64::sqrt<false>(__fma_rn(tau, tau, 1.0)));
  *c = f64::rcp<false>(f64::sqrt<false>(__fma_rn(t, t, 1.0)));
  const double sa = t * *c;
  *s = (__double2hiint(tau) < 0 && jac_nonzero(tau)) ? -sa : sa;
}
// c a - s b and s a + c b, one product rounded before the sum (the contraction k_geig_sym's expressions get)
__device__ __forceinline__ double jac_diff(double c, double a, double s, double b) {
  return __fma_rn(c, a, -__dmul_rn(s, b));
}
__device__ __forceinline__ double jac_sum(double s, double a, double c, double b) {
  return __fma_rn(s, a, __dmul_rn(c, b));
}

__device__ __forceinline__ void jac_st(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
// The index at a seat in round 0 of a sweep is the seat itself; every round all seats but seat 0 (step 0)
// advance by one through 1 .. N - 1.
__device__ __forceinline__ int jac_next(int i, int step, int N) {
  i += step;
  return i == N ? 1 : i;
}
// the seat a column sits at in the next round
__device__ __forceinline__ int jac_next_seat(int s, int N) { return (s == 0) ? 0 : (s == 1) ? N - 1 : s - 1; }

// C (n x n, symmetric, ld n) -> eigenvalues w (sorted) and the matching orthonormal eigenvectors Wout
// (ld n); hit[r] = 1 for the ranks that were written (all of them, but for eigenvalues that are NaN).
// Grid = one cluster of NC CTAs.  Every thread owns up to IT items of C (one row pair of one of the
// CTA's columns; adjacent lanes the two columns of a 2 x 2 block) and IT items of W (one row of one of the
// CTA's column pairs), and at most one remote entry of the next rotations: their seats never change, so only
// the indices at the seats are stepped from round to round.  W trails by one round: W <- W J runs beside
// the next round's rotations, which keep one or a few warps in a dependent FP64 chain.
template <int IT>
__global__ void __launch_bounds__(kJacT) k_jacobi_cluster(int n, int NC, int PP, const double* __restrict__ Cin,
                                                          double* __restrict__ w, double* __restrict__ Wout,
                                                          int* __restrict__ hit, int descending, int max_sweeps) {
  extern __shared__ double jsm[];
  const int N = n + (n & 1), npair = N / 2, S = 2 * PP;
  const int rank = (int)cluster_rank();
  const int tid = threadIdx.x;
  double* cb = jsm;                          // [2][S][n]
  double* wb = cb + (size_t)2 * S * n;       // [2][S][n]
  double* sD = wb + (size_t)2 * S * n;       // [2][npair][3]: a_pp, a_qq, a_pq of every pair
  double2* s_cs = reinterpret_cast<double2*>(sD + (size_t)2 * npair * 3);  // [2][npair]: c, s of every pair
  double* s_stage = reinterpret_cast<double*>(s_cs + (size_t)2 * npair);   // [S][2]: the next rotations' entries of this CTA's columns
  double* s_diag = s_stage + 2 * S;          // n: the final diagonal
  double* s_part = s_diag + n;               // [NC][2]: off and total sums of squares
  __shared__ double s_red[2][kJacT / 32];
  const int k0 = rank * PP;                  // this CTA's first pair
  // slot 2 l + side holds seat k0 + l (side 0) or N - 1 - (k0 + l) (side 1)
  auto seat_of = [&](int slot) {
    const int k = k0 + (slot >> 1);
    return (slot & 1) ? N - 1 - k : k;
  };
  // where the column at slot `slot` goes: CTA, and slot there
  auto dest = [&](int slot, int* cta) {
    const int s2 = jac_next_seat(seat_of(slot), N), kk = (s2 < npair) ? s2 : N - 1 - s2;
    *cta = kk / PP;
    return 2 * (kk % PP) + (s2 >= npair ? 1 : 0);
  };
  auto barrier = [&]() {
    if (NC > 1) {
      cluster_arrive();
      cluster_wait();
    } else {
      __syncthreads();
    }
  };
  // items of C: row pair (seats ck, N - 1 - ck), column slot; indices at the seats
  int c_slot[IT], c_k[IT], c_p[IT], c_q[IT], c_j[IT], c_jp[IT], c_j2[IT];
  int c_s0[IT], c_s2[IT];  // steps of the column's and of the next partner's seat
  unsigned c_dst[IT];
#pragma unroll
  for (int u = 0; u < IT; ++u) {
    const int e = tid + u * kJacT, l = (e >> 1) / npair;
    c_k[u] = (e >> 1) - l * npair;
    c_slot[u] = (l < PP && k0 + l < npair) ? 2 * l + (e & 1) : -1;
    c_p[u] = c_k[u];
    c_q[u] = N - 1 - c_k[u];
    c_j[u] = c_jp[u] = c_j2[u] = n;
    c_dst[u] = 0;
    c_s0[u] = c_s2[u] = 1;
    if (c_slot[u] >= 0) {
      int cta;
      const int ds = dest(c_slot[u], &cta);
      c_dst[u] = cluster_map(cb + (size_t)ds * n, cta);
      c_j[u] = seat_of(c_slot[u]);
      c_jp[u] = seat_of(c_slot[u] ^ 1);
      c_j2[u] = N - 1 - jac_next_seat(c_j[u], N);  // index at the next partner's seat, this round
      c_s0[u] = c_j[u] != 0;
      c_s2[u] = c_j2[u] != 0;
    }
  }
  // what an item does in the coming round, from the indices at its seats: offsets of its rows p < q and a code
  // (1 active, 2 row q exists, 4 column p of its pair, 8 / 16 its vq / vp is the rotated entry, 32 / 64 vp / vq
  // is the column's diagonal entry, 128 / 256 vp / vq is the entry (next partner, column)).  Computed between
  // arriving at the round's barrier and waiting for it.
  int c_po[IT], c_qo[IT], c_code[IT];
  auto plan_c = [&]() {
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int p = min(c_p[u], c_q[u]), q = max(c_p[u], c_q[u]), j = c_j[u];
      c_po[u] = p;
      c_qo[u] = q;
      int code = 0;
      if (j < n) {
        const int j2 = jac_next(c_j2[u], c_s2[u], N);
        code = 1 | (q < n ? 2 : 0) | (j < c_jp[u] ? 4 : 0);
        if (c_k[u] == k0 + (c_slot[u] >> 1)) code |= (j == p) ? 8 : 16;
        code |= (p == j ? 32 : 0) | (q == j ? 64 : 0);
        if (j2 < j) code |= (p == j2 ? 128 : 0) | (q == j2 ? 256 : 0);
      }
      c_code[u] = code;
    }
  };
  auto step_c = [&]() {
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      if (c_slot[u] < 0) continue;
      // seat 0 is only ever a pair's side 0: the other side's seat always steps
      c_j[u] = jac_next(c_j[u], c_s0[u], N);
      c_jp[u] = jac_next(c_jp[u], (c_slot[u] & 1) ? (k0 + (c_slot[u] >> 1)) != 0 : 1, N);
      c_j2[u] = jac_next(c_j2[u], c_s2[u], N);
      c_p[u] = jac_next(c_p[u], c_k[u] != 0, N);
      c_q[u] = jac_next(c_q[u], 1, N);
    }
    plan_c();
  };
  plan_c();
  // items of W: the first ones go to the warps that compute no rotations
  const int rot_warps = (npair + 31) / 32;
  const int wt = (tid + kJacT - 32 * rot_warps) % kJacT;
  int w_l[IT], w_i[IT], w_a[IT], w_b[IT];
  unsigned w_da[IT], w_db[IT];
#pragma unroll
  for (int u = 0; u < IT; ++u) {
    const int e = wt + u * kJacT, l = e / n;
    w_i[u] = e - l * n;
    w_l[u] = (l < PP && k0 + l < npair) ? l : -1;
    w_a[u] = w_b[u] = n;
    w_da[u] = w_db[u] = 0;
    if (w_l[u] >= 0) {
      int cta;
      int ds = dest(2 * l, &cta);
      w_da[u] = cluster_map(wb + (size_t)ds * n + w_i[u], cta);
      ds = dest(2 * l + 1, &cta);
      w_db[u] = cluster_map(wb + (size_t)ds * n + w_i[u], cta);
      w_a[u] = k0 + l;
      w_b[u] = N - 1 - (k0 + l);
    }
  }
  // the remote entry this thread pushes: (slot, diagonal or off-diagonal) to CTA e_cta
  int e_slot = -1, e_j = n, e_j2 = n, e_s = 1, e_s2 = 1;
  unsigned e_dst = 0;
  if (tid < 2 * S * NC) {
    const int sl = (tid >> 1) % S, cta = (tid >> 1) / S;
    if (k0 + (sl >> 1) < npair) {
      const int s2 = jac_next_seat(seat_of(sl), N), k2 = (s2 < npair) ? s2 : N - 1 - s2;
      e_slot = sl;
      e_j = seat_of(sl);
      e_j2 = N - 1 - s2;
      e_s = e_j != 0;
      e_s2 = e_j2 != 0;
      e_dst = cluster_map(sD + (size_t)k2 * 3, cta);
    }
  }
  // byte offset of this thread's entry among its pair's three (-1: nothing to push this round)
  int e_off = -1;
  auto plan_e = [&]() {
    e_off = -1;
    if (e_slot < 0 || e_j >= n) return;
    const int j2 = jac_next(e_j2, e_s2, N);
    if (tid & 1) e_off = (j2 < e_j) ? 16 : -1;
    else e_off = (e_j < j2) ? 0 : 8;
  };
  auto step_e = [&]() {
    if (e_slot < 0) return;
    e_j = jac_next(e_j, e_s, N);
    e_j2 = jac_next(e_j2, e_s2, N);
    plan_e();
  };
  plan_e();
  if (rank == 0)
    for (int i = tid; i < n; i += kJacT) hit[i] = 0;
  int r_x = tid, r_y = N - 1 - tid;  // indices of the pair whose rotation this thread computes (tid < npair)

  for (int e = tid; e < S * n; e += kJacT) {
    const int sl = e / n, i = e - sl * n;
    const int j = (k0 + (sl >> 1) < npair) ? seat_of(sl) : n;
    if (j < n) {
      cb[e] = Cin[i + (size_t)j * n];
      wb[e] = (i == j) ? 1.0 : 0.0;
    }
  }
  for (int k = tid; k < npair; k += kJacT) {
    const int p = k, q = N - 1 - k;
    sD[3 * k] = Cin[p + (size_t)p * n];
    sD[3 * k + 1] = (q < n) ? Cin[q + (size_t)q * n] : 0.0;
    sD[3 * k + 2] = (q < n) ? Cin[p + (size_t)q * n] : 0.0;
  }
  __syncthreads();
  barrier();

  const unsigned bufbytes = (unsigned)((size_t)S * n * sizeof(double));
  const unsigned dbytes = (unsigned)((size_t)npair * 3 * sizeof(double));
  int b = 0;
  bool pending = false;
  // W <- W J with the rotations of the round before (parity b ^ 1), into buffer b
  auto update_w = [&]() {
    const double2* cs = s_cs + (size_t)(b ^ 1) * npair;
    const unsigned nxt = b ? bufbytes : 0u;
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      if (w_l[u] < 0) continue;
      const int kg = k0 + w_l[u];
      const double* W0 = wb + ((size_t)(b ^ 1) * S + 2 * w_l[u]) * n + w_i[u];
      double wa = W0[0], wv = W0[n];
      const double c = cs[kg].x, s = cs[kg].y;
      const bool ab = w_a[u] < w_b[u];
      if (jac_nonzero(s)) {
        const double ap = ab ? wa : wv, aq = ab ? wv : wa;
        const double vp = jac_diff(c, ap, s, aq), vq = jac_sum(s, ap, c, aq);
        wa = ab ? vp : vq;
        wv = ab ? vq : vp;
      }
      if (w_a[u] < n) jac_st(w_da[u] + nxt, wa);
      if (w_b[u] < n) jac_st(w_db[u] + nxt, wv);
      w_a[u] = jac_next(w_a[u], kg != 0, N);
      w_b[u] = jac_next(w_b[u], 1, N);
    }
  };
  for (int sweep = 0; sweep < max_sweeps && n > 1; ++sweep) {
    {  // converged when off(C)^2 <= eps^2 ||C||_F^2
      double off = 0.0, tot = 0.0;
      for (int e = tid; e < S * n; e += kJacT) {
        const int sl = e / n, i = e - sl * n;
        const int j = (k0 + (sl >> 1) < npair) ? seat_of(sl) : n;  // a sweep starts with seat s holding index s
        if (j < n) {
          const double x = cb[(size_t)b * S * n + e], v = x * x;
          tot += v;
          if (i != j) off += v;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        off += __shfl_down_sync(0xffffffffu, off, o);
        tot += __shfl_down_sync(0xffffffffu, tot, o);
      }
      if ((tid & 31) == 0) {
        s_red[0][tid >> 5] = off;
        s_red[1][tid >> 5] = tot;
      }
      __syncthreads();
      if (tid < 2 * NC) {
        double a = 0.0;
        for (int x = 0; x < kJacT / 32; ++x) a += s_red[tid & 1][x];
        jac_st(cluster_map(s_part + 2 * rank + (tid & 1), (unsigned)(tid >> 1)), a);
      }
      barrier();
      double so = 0.0, sa = 0.0;
      for (int c = 0; c < NC; ++c) {
        so += s_part[2 * c];
        sa += s_part[2 * c + 1];
      }
      if (so <= 1.0e-32 * sa) break;  // every thread of every CTA sees the same sums
    }
    for (int r = 0; r < N - 1; ++r) {
      double2* cs = s_cs + (size_t)b * npair;
      const double* cur = cb + (size_t)b * S * n;
      double xp[IT], xq[IT];  // this round's entries, read before the rotations are known
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const double* col = cur + (size_t)max(c_slot[u], 0) * n;
        xp[u] = (c_code[u] & 1) ? col[c_po[u]] : 0.0;
        xq[u] = (c_code[u] & 2) ? col[c_qo[u]] : 0.0;
      }
      if (tid < npair) {
        const double* D = sD + ((size_t)b * npair + tid) * 3;
        double c = 1.0, s = 0.0;
        if (max(r_x, r_y) < n) jac_rotation(D[0], D[1], D[2], &c, &s);
        cs[tid] = make_double2(c, s);
      }
      if (pending) update_w();
      __syncthreads();
      // C <- J' C J on this CTA's columns
      const unsigned nxt = b ? 0u : bufbytes;
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        // a warp without items leaves as a whole: a predicated-off FP64 instruction still occupies the pipe
        const int code = c_code[u];
        if (!__any_sync(0xffffffffu, code)) continue;
        const double2 ck = cs[c_k[u]], cg = cs[min(k0 + (max(c_slot[u], 0) >> 1), npair - 1)];
        double vp = xp[u], vq = xq[u];
        if ((code & 1) && jac_nonzero(ck.y)) {
          vp = jac_diff(ck.x, xp[u], ck.y, xq[u]);
          vq = jac_sum(ck.y, xp[u], ck.x, xq[u]);
        }
        const double zp = __shfl_xor_sync(0xffffffffu, vp, 1), zq = __shfl_xor_sync(0xffffffffu, vq, 1);
        if (code & 1) {
          if (jac_nonzero(cg.y)) {
            // column p of its pair: fma(c, a_p, -(s a_q)); column q: fma(s, a_p, c a_q)
            const bool cp = code & 4;
            const double m1 = cp ? cg.x : cg.y, m2 = cp ? -cg.y : cg.x;
            const double ap_ = cp ? vp : zp, aq_ = cp ? zp : vp, bp_ = cp ? vq : zq, bq_ = cp ? zq : vq;
            vp = __fma_rn(m1, ap_, __dmul_rn(m2, aq_));
            vq = __fma_rn(m1, bp_, __dmul_rn(m2, bq_));
            if (code & 8) vq = 0.0;
            if (code & 16) vp = 0.0;
          }
          jac_st(c_dst[u] + nxt + 8u * (unsigned)c_po[u], vp);
          if (code & 2) jac_st(c_dst[u] + nxt + 8u * (unsigned)c_qo[u], vq);
          // entries of the next round's rotations
          if (code & 96) s_stage[2 * c_slot[u]] = (code & 32) ? vp : vq;
          if (code & 384) s_stage[2 * c_slot[u] + 1] = (code & 128) ? vp : vq;
        }
      }
      __syncthreads();
      // this CTA's entries of the next rotations, to every CTA
      if (e_off >= 0) jac_st(e_dst + (b ? 0u : dbytes) + (unsigned)e_off, s_stage[2 * e_slot + (tid & 1)]);
      if (NC > 1) cluster_arrive();
      step_c();
      step_e();
      if (tid < npair) {
        r_x = jac_next(r_x, tid != 0, N);
        r_y = jac_next(r_y, 1, N);
      }
      if (NC > 1) cluster_wait();
      else __syncthreads();
      b ^= 1;
      pending = true;
    }
  }
  if (pending) update_w();
  // the diagonal to every CTA, then each CTA writes its columns at their rank (ties by index)
  for (int e = tid; e < S * NC; e += kJacT) {
    const int slot = e % S, c = e / S;
    const int j = (k0 + (slot >> 1) < npair) ? seat_of(slot) : n;
    if (j < n) jac_st(cluster_map(s_diag + j, c), cb[((size_t)b * S + slot) * n + j]);
  }
  barrier();  // after this barrier no CTA reads or writes another's shared memory
  for (int slot = tid >> 5; slot < S; slot += kJacT / 32) {
    const int j = (k0 + (slot >> 1) < npair) ? seat_of(slot) : n;
    if (j >= n) continue;
    const double dj = s_diag[j];
    int rk = 0;
    for (int i = tid & 31; i < n; i += 32) {
      const double di = s_diag[i];
      const bool before = descending ? (di > dj || (di == dj && i < j)) : (di < dj || (di == dj && i < j));
      rk += before ? 1 : 0;
    }
    rk = __reduce_add_sync(0xffffffffu, rk);
    if ((tid & 31) == 0) {
      w[rk] = dj;
      hit[rk] = 1;
    }
    for (int i = tid & 31; i < n; i += 32) Wout[i + (size_t)rk * n] = wb[((size_t)b * S + slot) * n + i];
  }
}

// U = L^-T W (n x n, ld n; U with ld ldu): u_r = (w_r - sum_{k > r} L(k, r) u_k) / L(r, r), the sum in ascending k, so
// that the bits are the one-CTA form's -- where M is nearly singular (pivots clamped) another order of the sum gives
// other vectors altogether.  The first term of a row is the value found last, so a column is a chain of n^2 / 2
// dependent FMAs whatever the schedule (n = 64: 62 us); one lane per column, one warp per CTA, L in shared memory
// where it fits.
__global__ void __launch_bounds__(32) k_back_subst(int n, const double* __restrict__ L, const double* __restrict__ W,
                                                   const int* __restrict__ hit, double* __restrict__ U, int ldu) {
  extern __shared__ double bsm[];  // L (column-major), then the CTA's 32 columns of U (row-major)
  double* sL = bsm;
  double* sU = bsm + (size_t)n * n;
  const int lane = threadIdx.x, j = blockIdx.x * 32 + lane;
  for (int e = lane; e < n * n; e += 32) sL[e] = L[e];
  __syncwarp();
  const bool store = j < n && hit[j];
  for (int r = n - 1; r >= 0; --r) {
    double s = (j < n) ? W[r + (size_t)j * n] : 0.0;
    const double* l = sL + (size_t)r * n;
    int k = r + 1;
    for (; k + 8 <= n; k += 8) {
      double a[8], b[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        a[u] = l[k + u];
        b[u] = sU[(k + u) * 32 + lane];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) s = __fma_rn(-a[u], b[u], s);
    }
    for (; k < n; ++k) s = __fma_rn(-l[k], sU[k * 32 + lane], s);
    s = f64::div(s, l[r]);
    sU[r * 32 + lane] = s;
    if (store) U[r + (size_t)j * ldu] = s;
  }
}

// C = (G + G') / 2 (or G itself)
__global__ void k_sym_copy(int n, const double* __restrict__ G, int ldg, int symmetrize, double* __restrict__ C) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * n; e += gridDim.x * blockDim.x) {
    const int i = e % n, j = e / n;
    const double g = G[i + (size_t)j * ldg];
    C[e] = symmetrize ? 0.5 * (g + G[j + (size_t)i * ldg]) : g;
  }
}

struct GeigParams {
  int n;
  const double* G;
  int ldg;
  const double* M;  // may be null (standard problem)
  int ldm;
  int symmetrize;
  int descending;
  double* w;   // out, n
  double* U;   // out, n x n (ldu)
  int ldu;
  double* gws;  // global workspace (3 n^2)
  int* flag;    // out: 1 if the Cholesky factor needed a clamp (near-singular M)
  int max_sweeps;
};

__device__ __forceinline__ int rr_index(int i, int r, int N) { return i == 0 ? 0 : ((i - 1 + r) % (N - 1)) + 1; }

__global__ void __launch_bounds__(512) k_geig_sym(GeigParams P) {
  const int n = P.n, tid = threadIdx.x, nt = blockDim.x;
  double* C = P.gws;
  double* W = C + (size_t)n * n;
  double* L = W + (size_t)n * n;
  __shared__ double s_c[160], s_s[160];
  __shared__ int s_p[160], s_q[160];
  __shared__ double s_red[32];
  __shared__ int s_stop;
  __shared__ double s_maxdiag;

  // ---- Cholesky of M (lower) ------------------------------------------------------
  const bool gen = (P.M != nullptr);
  if (gen) {
    for (int e = tid; e < n * n; e += nt) {
      int i = e % n, j = e / n;
      L[e] = (i >= j) ? P.M[i + (size_t)j * P.ldm] : 0.0;
    }
    __syncthreads();
    if (tid == 0) {
      double md = 0.0;
      for (int k = 0; k < n; ++k) md = fmax(md, fabs(L[k + (size_t)k * n]));
      s_maxdiag = md;
    }
    __syncthreads();
    for (int k = 0; k < n; ++k) {
      if (tid == 0) {
        double d = L[k + (size_t)k * n];
        const double floor_d = s_maxdiag * 1e-15 + 1e-300;
        if (!(d > floor_d)) {
          d = floor_d;
          if (P.flag) *P.flag = 1;
        }
        L[k + (size_t)k * n] = sqrt(d);
      }
      __syncthreads();
      const double dk = L[k + (size_t)k * n];
      for (int i = k + 1 + tid; i < n; i += nt) L[i + (size_t)k * n] /= dk;
      __syncthreads();
      const int rem = n - k - 1;
      for (int e = tid; e < rem * rem; e += nt) {
        int i = k + 1 + e % rem, j = k + 1 + e / rem;
        if (i >= j) L[i + (size_t)j * n] -= L[i + (size_t)k * n] * L[j + (size_t)k * n];
      }
      __syncthreads();
    }
  }

  // ---- C = G (symmetrised), reduced by L when generalized -------------------------
  for (int e = tid; e < n * n; e += nt) {
    int i = e % n, j = e / n;
    double g = P.G[i + (size_t)j * P.ldg];
    if (P.symmetrize) g = 0.5 * (g + P.G[j + (size_t)i * P.ldg]);
    C[e] = g;
  }
  __syncthreads();
  if (gen) {
    // W <- L^-1 C   (column j solved by one thread)
    for (int j = tid; j < n; j += nt) {
      for (int i = 0; i < n; ++i) {
        double s = C[i + (size_t)j * n];
        for (int k = 0; k < i; ++k) s -= L[i + (size_t)k * n] * W[k + (size_t)j * n];
        W[i + (size_t)j * n] = s / L[i + (size_t)i * n];
      }
    }
    __syncthreads();
    // C <- L^-1 W'   (right-hand side j is row j of W)
    for (int j = tid; j < n; j += nt) {
      for (int i = 0; i < n; ++i) {
        double s = W[j + (size_t)i * n];
        for (int k = 0; k < i; ++k) s -= L[i + (size_t)k * n] * C[k + (size_t)j * n];
        C[i + (size_t)j * n] = s / L[i + (size_t)i * n];
      }
    }
    __syncthreads();
    for (int e = tid; e < n * n; e += nt) {
      int i = e % n, j = e / n;
      if (i < j) {
        double a = 0.5 * (C[i + (size_t)j * n] + C[j + (size_t)i * n]);
        C[i + (size_t)j * n] = a;
        C[j + (size_t)i * n] = a;
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < n * n; e += nt) W[e] = ((e % n) == (e / n)) ? 1.0 : 0.0;
  __syncthreads();

  // ---- cyclic Jacobi, round-robin ordering ------------------------------------------
  const int N = n + (n & 1);
  const int npair = N / 2;
  for (int sweep = 0; sweep < P.max_sweeps && n > 1; ++sweep) {
    // convergence test: off(C)^2 <= eps^2 * ||C||_F^2
    double off = 0.0, tot = 0.0;
    for (int e = tid; e < n * n; e += nt) {
      double v = C[e] * C[e];
      tot += v;
      if ((e % n) != (e / n)) off += v;
    }
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_down_sync(0xffffffffu, off, o);
      tot += __shfl_down_sync(0xffffffffu, tot, o);
    }
    if ((tid & 31) == 0) s_red[tid >> 5] = off;
    __syncthreads();
    if (tid == 0) {
      double a = 0.0;
      for (int w = 0; w < (nt >> 5); ++w) a += s_red[w];
      s_red[0] = a;
    }
    __syncthreads();
    off = s_red[0];
    __syncthreads();
    if ((tid & 31) == 0) s_red[tid >> 5] = tot;
    __syncthreads();
    if (tid == 0) {
      double a = 0.0;
      for (int w = 0; w < (nt >> 5); ++w) a += s_red[w];
      s_stop = (off <= 1.0e-32 * a) ? 1 : 0;
    }
    __syncthreads();
    if (s_stop) break;
    for (int r = 0; r < N - 1; ++r) {
      for (int k = tid; k < npair; k += nt) {
        int p = rr_index(k, r, N), q = rr_index(N - 1 - k, r, N);
        if (p > q) {
          int t = p;
          p = q;
          q = t;
        }
        double c = 1.0, s = 0.0;
        if (q < n) {
          const double apq = C[p + (size_t)q * n];
          if (apq != 0.0) {
            const double app = C[p + (size_t)p * n], aqq = C[q + (size_t)q * n];
            const double tau = (aqq - app) / (2.0 * apq);
            const double t = (tau >= 0.0) ? 1.0 / (tau + sqrt(1.0 + tau * tau)) : -1.0 / (-tau + sqrt(1.0 + tau * tau));
            c = 1.0 / sqrt(1.0 + t * t);
            s = t * c;
          }
        }
        s_p[k] = p;
        s_q[k] = (q < n) ? q : -1;
        s_c[k] = c;
        s_s[k] = s;
      }
      __syncthreads();
      // rows: C <- J' C
      for (int e = tid; e < npair * n; e += nt) {
        const int k = e / n, j = e % n;
        const int q = s_q[k];
        if (q < 0 || s_s[k] == 0.0) continue;
        const int p = s_p[k];
        const double c = s_c[k], s = s_s[k];
        const double ap = C[p + (size_t)j * n], aq = C[q + (size_t)j * n];
        C[p + (size_t)j * n] = c * ap - s * aq;
        C[q + (size_t)j * n] = s * ap + c * aq;
      }
      __syncthreads();
      // columns: C <- C J, W <- W J
      for (int e = tid; e < npair * n; e += nt) {
        const int k = e / n, i = e % n;
        const int q = s_q[k];
        if (q < 0 || s_s[k] == 0.0) continue;
        const int p = s_p[k];
        const double c = s_c[k], s = s_s[k];
        double ap = C[i + (size_t)p * n], aq = C[i + (size_t)q * n];
        C[i + (size_t)p * n] = c * ap - s * aq;
        C[i + (size_t)q * n] = s * ap + c * aq;
        ap = W[i + (size_t)p * n];
        aq = W[i + (size_t)q * n];
        W[i + (size_t)p * n] = c * ap - s * aq;
        W[i + (size_t)q * n] = s * ap + c * aq;
      }
      __syncthreads();
      for (int k = tid; k < npair; k += nt) {
        const int q = s_q[k];
        if (q >= 0 && s_s[k] != 0.0) {
          const int p = s_p[k];
          C[p + (size_t)q * n] = 0.0;
          C[q + (size_t)p * n] = 0.0;
        }
      }
      __syncthreads();
    }
  }

  // ---- sort and back-transform --------------------------------------------------------
  // rank of each eigenvalue (stable): descending or ascending
  for (int i = tid; i < n; i += nt) {
    const double di = C[i + (size_t)i * n];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = C[j + (size_t)j * n];
      const bool before = P.descending ? (dj > di || (dj == di && j < i)) : (dj < di || (dj == di && j < i));
      rank += before ? 1 : 0;
    }
    P.w[rank] = di;
    // U(:, rank) = L^-T W(:, i)  (back substitution) or W(:, i)
    if (gen) {
      for (int r = n - 1; r >= 0; --r) {
        double s = W[r + (size_t)i * n];
        for (int k = r + 1; k < n; ++k) s -= L[k + (size_t)r * n] * P.U[k + (size_t)rank * P.ldu];
        P.U[r + (size_t)rank * P.ldu] = s / L[r + (size_t)r * n];
      }
    } else {
      for (int r = 0; r < n; ++r) P.U[r + (size_t)rank * P.ldu] = W[r + (size_t)i * n];
    }
  }
}

static size_t jacobi_smem(int n, int NC) {
  const int N = n + (n & 1), npair = N / 2, PP = (npair + NC - 1) / NC, S = 2 * PP;
  return sizeof(double) * ((size_t)4 * S * n + 6 * npair + 4 * npair + 2 * S + n + 2 * NC);
}

// CTAs of the Jacobi cluster.  A round costs the rotation chain and a barrier on any cluster (about 2.6 us
// on one CTA, 2.9 us on sixteen) plus 6 n^2 FP64 operations shared by the CTAs (one warp instruction per 64
// cycles and SM sub-partition).  Whole syev calls, random matrices, us for 1 / 4 / 8 / 16 CTAs:
//   n = 16: 258 / 277 / 289 / 307    n = 32: 1028 / 715 / 716 / 758   n = 48: - / 1279 / 1125 / 1109
//   n = 64: - / 2148 / 1627 / 1511   n = 96: - / - / 4057 / 3061      n = 128: - / - / 7137 / 5069
// (the one-CTA kernel below: 363, 1332, 3234, 6146, 23418 and 49327 us).  Sixteen CTAs are beyond the
// portable cluster size: 0 when the device cannot place them and eight cannot hold the items either.
static int jacobi_cluster_size(int n) {
  if (n <= 20) return 1;
  if (n <= 40) return 4;
  if (n <= 56) return 8;
  static std::atomic<int> max_cluster[64];  // per device: 0 not asked yet, else 8 or 16
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return n <= 128 ? 8 : 0;
  int mc = max_cluster[dev].load(std::memory_order_relaxed);
  if (mc == 0) {
    mc = 8;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kJacT);
    cfg.dynamicSmemBytes = jacobi_smem(kGeigClusterMaxN, 16);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(k_jacobi_cluster<2>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        allow_smem(k_jacobi_cluster<2>) == OFRR_SUCCESS &&
        cudaOccupancyMaxActiveClusters(&clusters, k_jacobi_cluster<2>, &cfg) == cudaSuccess && clusters >= 1)
      mc = 16;
    (void)cudaGetLastError();  // a refused query leaves the portable size
    max_cluster[dev].store(mc, std::memory_order_relaxed);
  }
  return mc == 16 ? 16 : n <= 128 ? 8 : 0;
}

template <int IT>
static int jacobi_launch(ofrr_ctx* ctx, int n, int NC, const double* C, double* w, double* W, int* hit, int descending,
                         int max_sweeps) {
  OFRR_TRY(allow_smem(k_jacobi_cluster<IT>));
  if (NC > 8)
    OFRR_CUDA(cudaFuncSetAttribute(k_jacobi_cluster<IT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)NC;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)NC);
  cfg.blockDim = dim3(kJacT);
  cfg.dynamicSmemBytes = jacobi_smem(n, NC);
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int PP = ((n + 1) / 2 + NC - 1) / NC;
  OFRR_CUDA(cudaLaunchKernelEx(&cfg, k_jacobi_cluster<IT>, n, NC, PP, C, w, W, hit, descending, max_sweeps));
  OFRR_LAUNCHED(ctx, "k_jacobi_cluster");
  return OFRR_SUCCESS;
}

// The cluster form: Cholesky, two substitutions, the Jacobi sweeps, and the back substitution.
static int geig_cluster(ofrr_ctx* ctx, const GeigParams& P, int NC) {
  int st = OFRR_SUCCESS;
  const int n = P.n;
  const size_t nn = (size_t)n * n;
  double *C = ws_get<double>(ctx, nn, &st), *W = ws_get<double>(ctx, nn, &st);
  int* hit = ws_get<int>(ctx, (size_t)n, &st);
  if (!C || !W || !hit) return st;
  const unsigned g = (unsigned)std::min<size_t>((nn + 255) / 256, 152);
  double *L = nullptr, *Y = nullptr;
  if (P.M) {
    L = ws_get<double>(ctx, nn, &st);
    Y = ws_get<double>(ctx, nn, &st);
    if (!L || !Y) return st;
    k_sym_copy<<<g, 256, 0, ctx->stream>>>(n, P.G, P.ldg, P.symmetrize, W);
    OFRR_LAUNCHED(ctx, "k_sym_copy");
    OFRR_TRY(small_chol(ctx, n, P.M, P.ldm, L));
    OFRR_TRY(small_trsm(ctx, n, L, W, 0, Y));  // Y = L^-1 G
    OFRR_TRY(small_trsm(ctx, n, L, Y, 1, W));  // W = L^-1 Y' = L^-1 G L^-T
    k_sym_copy<<<g, 256, 0, ctx->stream>>>(n, W, n, 1, C);
    OFRR_LAUNCHED(ctx, "k_sym_copy");
  } else {
    k_sym_copy<<<g, 256, 0, ctx->stream>>>(n, P.G, P.ldg, P.symmetrize, C);
    OFRR_LAUNCHED(ctx, "k_sym_copy");
  }
  double* Wj = (!P.M && P.ldu == n) ? P.U : W;
  // items of C and of W per thread: (N / 2) 2 PP and n PP over kJacT threads
  const int PP = ((n + 1) / 2 + NC - 1) / NC, items = (n + (n & 1)) * PP;
  if (items > 2 * kJacT || 4 * PP * NC > kJacT) return OFRR_ERR_INTERNAL;
  if (items <= kJacT)
    OFRR_TRY(jacobi_launch<1>(ctx, n, NC, C, P.w, Wj, hit, P.descending, P.max_sweeps));
  else
    OFRR_TRY(jacobi_launch<2>(ctx, n, NC, C, P.w, Wj, hit, P.descending, P.max_sweeps));
  if (P.M) {
    const size_t smem = sizeof(double) * (nn + (size_t)32 * n);
    OFRR_TRY(allow_smem(k_back_subst));
    k_back_subst<<<(unsigned)((n + 31) / 32), 32, smem, ctx->stream>>>(n, L, W, hit, P.U, P.ldu);  // U = L^-T W
    OFRR_LAUNCHED(ctx, "k_back_subst");
  } else if (Wj != P.U) {
    OFRR_CUDA(cudaMemcpy2DAsync(P.U, P.ldu * sizeof(double), Wj, n * sizeof(double), n * sizeof(double), n,
                                cudaMemcpyDeviceToDevice, ctx->stream));
  }
  return OFRR_SUCCESS;
}

static int geig_launch(ofrr_ctx* ctx, GeigParams P) {
  const int NC = (P.n <= kGeigClusterMaxN) ? jacobi_cluster_size(P.n) : 0;
  if (NC > 0) return geig_cluster(ctx, P, NC);
  int st = OFRR_SUCCESS;
  P.gws = ws_get<double>(ctx, (size_t)3 * P.n * P.n, &st);
  if (!P.gws) return st;
  k_geig_sym<<<1, 512, 0, ctx->stream>>>(P);
  OFRR_LAUNCHED(ctx, "k_geig_sym");
  return OFRR_SUCCESS;
}

int geig_dev(ofrr_ctx* ctx, int n, const double* G, int ldg, const double* M, int ldm, int symmetric, double* w,
             double* U, int ldu) {
  if (n <= 0) return OFRR_SUCCESS;
  if (n > 300) return OFRR_ERR_BLAS_INVALID_SIZE;
  if (!symmetric) return OFRR_ERR_NOT_IMPLEMENTED;
  WsScope scope(ctx);
  GeigParams P{};
  P.n = n;
  P.G = G;
  P.ldg = ldg;
  P.M = M;
  P.ldm = ldm;
  P.symmetrize = 1;
  P.descending = 1;
  P.w = w;
  P.U = U;
  P.ldu = ldu;
  P.flag = ctx->dev_flags + 1;
  P.max_sweeps = 30;
  return geig_launch(ctx, P);
}

int syev_dev(ofrr_ctx* ctx, int n, double* A, int lda, double* w) {
  if (n <= 0) return OFRR_SUCCESS;
  if (n > 300) return OFRR_ERR_BLAS_INVALID_SIZE;
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  double* U = ws_get<double>(ctx, (size_t)n * n, &st);
  if (!U) return st;
  GeigParams P{};
  P.n = n;
  P.G = A;
  P.ldg = lda;
  P.M = nullptr;
  P.symmetrize = 1;
  P.descending = 0;
  P.w = w;
  P.U = U;
  P.ldu = n;
  P.flag = ctx->dev_flags + 1;
  P.max_sweeps = 30;
  OFRR_TRY(geig_launch(ctx, P));
  OFRR_CUDA(cudaMemcpy2DAsync(A, lda * sizeof(double), U, n * sizeof(double), n * sizeof(double), n,
                              cudaMemcpyDeviceToDevice, ctx->stream));
  return OFRR_SUCCESS;
}

int sygv_dev(ofrr_ctx* ctx, int n, double* A, int lda, double* B, int ldb, double* w) {
  if (n <= 0) return OFRR_SUCCESS;
  if (n > 300) return OFRR_ERR_BLAS_INVALID_SIZE;
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  double* U = ws_get<double>(ctx, (size_t)n * n, &st);
  if (!U) return st;
  GeigParams P{};
  P.n = n;
  P.G = A;
  P.ldg = lda;
  P.M = B;
  P.ldm = ldb;
  P.symmetrize = 1;
  P.descending = 0;
  P.w = w;
  P.U = U;
  P.ldu = n;
  P.flag = ctx->dev_flags + 1;
  P.max_sweeps = 30;
  OFRR_TRY(geig_launch(ctx, P));
  OFRR_CUDA(cudaMemcpy2DAsync(A, lda * sizeof(double), U, n * sizeof(double), n * sizeof(double), n,
                              cudaMemcpyDeviceToDevice, ctx->stream));
  return OFRR_SUCCESS;
}

}  // namespace ofrr

using namespace ofrr;

extern "C" int ofrr_syev(ofrr_ctx* ctx, int n, double* A, int lda, double* w) {
  if (!ctx || n < 0 || (n > 0 && (!A || !w || lda < n))) return OFRR_ERR_INVALID_ARGUMENT;
  return syev_dev(ctx, n, A, lda, w);
}

extern "C" int ofrr_sygv(ofrr_ctx* ctx, int n, double* A, int lda, double* B, int ldb, double* w) {
  if (!ctx || n < 0 || (n > 0 && (!A || !B || !w || lda < n || ldb < n))) return OFRR_ERR_INVALID_ARGUMENT;
  return sygv_dev(ctx, n, A, lda, B, ldb, w);
}

namespace ofrr {
namespace {
__global__ void k_f64_ops(int op, int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                          double* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = op == 0 ? f64::rcp(a[i]) : op == 1 ? f64::div(a[i], b[i]) : f64::sqrt(a[i]);
}
}  // namespace
}  // namespace ofrr

// Self-test of the short FP64 operations (f64_ops.cuh): out[i] = 1 / a[i] (op 0), a[i] / b[i] (1), sqrt(a[i]) (2)
extern "C" int ofrr_debug_f64_ops(ofrr_ctx* ctx, int op, int64_t n, const double* a, const double* b, double* out) {
  if (!ctx || op < 0 || op > 2 || n < 1 || !a || !out || (op == 1 && !b)) return OFRR_ERR_INVALID_ARGUMENT;
  k_f64_ops<<<grid_for(n, 256, 152 * 8), 256, 0, ctx->stream>>>(op, n, a, b, out);
  OFRR_LAUNCHED(ctx, "k_f64_ops");
  return sync_and_check(ctx);
}
