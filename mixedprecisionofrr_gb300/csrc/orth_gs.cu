// Orthogonal comparison bases for subspace iteration: modified (MATLAB/+src/+qr/mgs.m:49-101) and
// classical (MATLAB/+src/+qr/cgs.m:49-110) Gram-Schmidt with the reference's adaptive
// re-orthogonalisation.  mgs.m is the default `function_orth` of subspace_iter_eig.m:114-115; the
// orthogonalization-free runs pass hessenberg instead.  For column i of A (m x n, tall):
//   normv = norm2(a_i); normv < select_tol -> column dropped
//   projection pass over the selected earlier columns j (in order):
//     MGS: r_j = dot(v, q_j), v = po(pc(v) - pc(r_j) pc(q_j)) one j at a time
//     CGS: all r_j = dot(v, q_j) first, then the same updates in j order
//   t = norm2(v); while t >= orth_tol and t < reorth_tol normv: normv = t, another pass with
//   R(j,i) = po(pc(R(j,i)) + pc(r_j)), t = norm2(v)
//   t < select_tol -> dropped; else q_i = po(pc(v) / pc(t)), R(i,i) = t.
// Bases in FP64 throughout are built in one cooperative launch (k_gs_coop).  With a narrower storage type, and for
// MGS without effective re-orthogonalisation, the column loop runs: dots and norms are grid reductions in the
// compute type (per-CTA partial sums, the last CTA adds them in a fixed order: deterministic); the updates are
// row-parallel and apply the j terms in order with one rounding to the output type per term, as the MATLAB code
// does; the while-loop decisions need t on the host, one synchronisation per column and pass.
// Q keeps the input's column positions (dropped columns zero) with select flags, like the Hessenberg
// basis, so the solvers compact both the same way.
#include <cmath>
#include <vector>

#include "grid_barrier.cuh"
#include "ofrr_internal.cuh"

namespace ofrr {
namespace {

constexpr int GS_T = 256;
constexpr int GS_G = 152;  // CTAs per reduction

// host-side conversions of the storage types
inline double host_double(double x) { return x; }
inline double host_double(float x) { return (double)x; }
inline double host_double(__half x) { return (double)__half2float(x); }
inline double host_double(__nv_bfloat16 x) { return (double)__bfloat162float(x); }
// x rounded to the storage type t (a tolerance compared in the output precision)
inline double round_to(ofrr_dtype t, double x) {
  switch (t) {
    case OFRR_F32: return (double)(float)x;
    case OFRR_F16: return (double)__half2float(__double2half(x));
    case OFRR_BF16: return (double)__bfloat162float(__double2bfloat16(x));
    default: return x;
  }
}

// out[c] = po(sum_i pc(v_i) pc(Q[i, cols[c]])) for c = blockIdx.y; Q == nullptr: out[0] = po(sqrt(sum pc(v_i)^2))
template <class TO, class TC>
__global__ void __launch_bounds__(GS_T) k_gs_reduce(int64_t m, const TO* __restrict__ v, const TO* __restrict__ Q,
                                                    int64_t ldq, const int* __restrict__ cols, TC* __restrict__ partial,
                                                    unsigned int* __restrict__ counters, TO* __restrict__ out) {
  __shared__ TC red[GS_T / 32];
  __shared__ bool last;
  const int c = blockIdx.y;
  const TO* q = Q ? Q + (int64_t)cols[c] * ldq : nullptr;
  TC s = TC(0);
  for (int64_t i = blockIdx.x * (int64_t)GS_T + threadIdx.x; i < m; i += (int64_t)gridDim.x * GS_T) {
    const TC a = to_c<TC, TO>(v[i]);
    s += a * (q ? to_c<TC, TO>(q[i]) : a);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    TC b = TC(0);
    for (int w = 0; w < GS_T / 32; ++w) b += red[w];
    partial[(size_t)c * gridDim.x + blockIdx.x] = b;
    __threadfence();
    last = (atomicAdd(counters + c, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  const volatile TC* vp = partial + (size_t)c * gridDim.x;
  TC tot = TC(0);
  for (unsigned int b = 0; b < gridDim.x; ++b) tot += vp[b];
  counters[c] = 0;  // self-resetting for the next reduction
  out[c] = q ? from_c<TO, TC>(tot) : from_c<TO, TC>(sqrt(tot));
}

// v_i <- po(pc(v_i) - pc(r_c) pc(Q[i, cols[c]])) for c = 0..ncols-1 in order (one rounding to po per
// term, no fused multiply-add: the MATLAB arithmetic); one thread also records R(cols[c], i) = r_c
// (acc: po(pc(R) + pc(r_c))) in the FP64 copy of R (column Rcol)
template <class TO, class TC>
__global__ void __launch_bounds__(GS_T) k_gs_update(int64_t m, TO* __restrict__ v, const TO* __restrict__ Q,
                                                    int64_t ldq, const int* __restrict__ cols, int ncols,
                                                    const TO* __restrict__ r, double* __restrict__ Rcol, int acc) {
  for (int64_t i = blockIdx.x * (int64_t)GS_T + threadIdx.x; i < m; i += (int64_t)gridDim.x * GS_T) {
    TC x = to_c<TC, TO>(v[i]);
    for (int c = 0; c < ncols; ++c) {
      const TC p = mul_rn(to_c<TC, TO>(r[c]), to_c<TC, TO>(Q[i + (int64_t)cols[c] * ldq]));
      x = to_c<TC, TO>(from_c<TO, TC>(sub_rn(x, p)));
    }
    v[i] = from_c<TO, TC>(x);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (int c = 0; c < ncols; ++c) {
      const int j = cols[c];
      const TC rc = to_c<TC, TO>(r[c]);
      Rcol[j] = acc ? (double)to_c<TC, TO>(from_c<TO, TC>(add_rn(to_c<TC, double>(Rcol[j]), rc))) : (double)rc;
    }
  }
}

// q = po(pc(v) / pc(t)), R(i,i) = t
template <class TO, class TC>
__global__ void __launch_bounds__(GS_T) k_gs_scale(int64_t m, const TO* __restrict__ v, const TO* __restrict__ t,
                                                   TO* __restrict__ q, double* __restrict__ Rii) {
  const TC tc = to_c<TC, TO>(*t);
  for (int64_t i = blockIdx.x * (int64_t)GS_T + threadIdx.x; i < m; i += (int64_t)gridDim.x * GS_T)
    q[i] = from_c<TO, TC>(div_rn(to_c<TC, TO>(v[i]), tc));
  if (blockIdx.x == 0 && threadIdx.x == 0) *Rii = (double)to_c<TC, TO>(*t);
}

// ---- FP64 bases in one cooperative launch ------------------------------------------------------------
// The column loop above costs two launches per projection and a host synchronisation per column and pass:
// 80.8 ms for 64 correlated columns of 8192 rows (4000 dependent dots).  Here one launch does the whole basis.
//  * The rows are split over the CTAs of a resident grid; all of a column's decisions are taken by every CTA
//    from the same reduced sums, so nothing returns to the host.
//  * MGS's dots of one pass depend on each other only through Q'Q: r_j = q_j'v - sum_{l<j} (q_j'q_l) r_l, that is
//    r = T Q'v with T = (I + strict lower(Q'Q))^-1, the inverse compact form of MGS (K. Swirydowicz, J. Langou,
//    S. Ananthan, U. Yang, S. Thomas, "Low synchronization Gram-Schmidt and generalized minimal residual
//    algorithms", Numer. Linear Algebra Appl. 28, 2021), which has MGS's error bounds.  T grows by one row per
//    column.  So a pass needs one reduction instead of one per earlier column; CGS has r = Q'v.
//  * One reduction after a pass gives v'v (the norm), Q'v (the next pass's dots, or the new row of Q'Q) and
//    v'a_c for the columns still to come (their first dots, once divided by the norm): a column costs as many
//    reductions as it takes passes.
// Sums are in a fixed order (rows of a CTA, then CTAs), so results do not depend on the schedule.  The terms of
// an update are summed by FMA before they are subtracted: fewer roundings than one per term.
// A reduction takes two rounds through L2: every CTA writes its partial sums, value k is summed by one warp of
// CTA k mod G, and all CTAs read the totals.
// What bounds it: for 8192 x 64 (122 passes) a pass takes about 21,000 cycles: the dots, the update and T's
// product 3,000 to 3,400 each (every FP64 warp instruction takes its sub-partition 64 cycles), the two rounds of
// the reduction 7,000, and norm, scaling and the new row of T the rest.
// Measured, call included, correlated columns: 8192 x 64 MGS 80.8 -> 1.43 ms, CGS -> 1.17 ms; 100000 x 80 MGS 5.7 ms
// (its dots, read from L2, then take two thirds); 300 x 20 0.49 ms.
constexpr int GC_T = 512;
constexpr int GC_W = GC_T / 32;
constexpr int GC_MAXN = 128;
constexpr int GC_MAXG = 160;  // CTAs at most (152 SMs, rounded up to whole warps)

struct GsCoop {
  int64_t m, lda, ldq;
  int n, classical, rows;  // rows per CTA
  const double* A;
  double* Q;
  double* R;
  int* sel;
  double stol, otol, rtol;
  double* partial;  // [G][n + 1]
  double* total;    // [n + 1]
  unsigned* ctr;    // two counters
  int* err;
};

// XS: this CTA's rows of [Q(:, < i), A(:, >= i)] stay in shared memory (row-major); otherwise they are read
// from global memory
template <bool XS>
__global__ void __launch_bounds__(GC_T) k_gs_coop(GsCoop P) {
  extern __shared__ double gsm[];
  const int n = P.n, K = n + 1, LD = n | 1, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int G = gridDim.x;
  const int64_t row0 = (int64_t)blockIdx.x * P.rows;
  const int nr = (int)max((int64_t)0, min((int64_t)P.rows, P.m - row0));
  double* TH = gsm;                        // lower triangle: T; strict upper (l, c): q_l'a_c
  double* s_v = TH + (size_t)n * LD;       // the CTA's rows of v
  double* s_r = s_v + P.rows;              // projection coefficients
  double* s_h = s_r + n;                   // dots of the pass
  double* s_tot = s_h + n;                 // totals of the reduction
  double* s_norm = s_tot + K;              // norms of the original columns
  double* s_red = s_norm + n;              // scratch: max(16 n, 1024)
  double* X = s_red + max(GC_W * n, 1024);  // XS: nr x n, row-major, leading dimension LD
  __shared__ int s_sel[GC_MAXN];
  __shared__ int s_ok;
  __shared__ double s_vv, s_t;
  // decisions are taken by one thread: an FP64 square root or compare on every warp would queue on the pipe
  __shared__ int s_skip[GC_MAXN], s_dec;
  const double* A = P.A + row0;
  double* Q = P.Q + row0;

  for (int e = tid; e < n * LD; e += GC_T) TH[e] = 0.0;
  for (int c = tid; c < n; c += GC_T) s_sel[c] = 0;
  if (XS)
    for (int c = wid; c < n; c += GC_W)
      for (int r = lane; r < nr; r += 32) X[(size_t)r * LD + c] = A[r + (int64_t)c * P.lda];
  __syncthreads();

  unsigned step = 0;
  const int owners = min(K, G);
  // s_red[0 .. K) -> s_tot[0 .. K), summed over the CTAs
  auto reduce = [&]() -> bool {
    ++step;
    for (int k = tid; k < K; k += GC_T) __stcg(P.partial + (size_t)blockIdx.x * K + k, s_red[k]);
    grid_arrive(P.ctr);
    if ((int)blockIdx.x < owners) {
      if (!grid_wait(P.ctr, (unsigned)G * step, &s_ok, P.err, 51)) return false;
      for (int k = blockIdx.x + G * wid; k < K; k += G * GC_W) {
        double v[GC_MAXG / 32], s = 0.0;  // all loads in flight together: one L2 latency
#pragma unroll
        for (int u = 0; u < GC_MAXG / 32; ++u)
          v[u] = (lane + 32 * u < G) ? __ldcg(P.partial + (size_t)(lane + 32 * u) * K + k) : 0.0;
#pragma unroll
        for (int u = 0; u < GC_MAXG / 32; ++u) s += v[u];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) __stcg(P.total + k, s);
      }
      grid_arrive(P.ctr + 1);
    }
    if (!grid_wait(P.ctr + 1, (unsigned)owners * step, &s_ok, P.err, 52)) return false;
    for (int k = tid; k < K; k += GC_T) s_tot[k] = __ldcg(P.total + k);
    __syncthreads();
    return true;
  };
  // s_red[c] = this CTA's part of x_c'v (x_c'x_c with self) for every column c, x_c = q_c for c < i and a_c
  // otherwise; s_red[n] = v'v
  auto dots = [&](int i, bool self) {
    if (XS) {
      // lanes over columns, row groups over warps; the last warp takes v'v
      const int cg = (n + 31) / 32, rg = (GC_W - 1) / cg, g = wid / cg, c = (wid % cg) * 32 + lane;
      double acc = 0.0;
      if (wid < rg * cg) {
        const int per = (nr + rg - 1) / rg, ra = g * per, rb = min(nr, ra + per);
        if (c < n)
          for (int r = ra; r < rb; ++r) {
            const double x = X[(size_t)r * LD + c];
            acc = fma(x, self ? x : s_v[r], acc);
          }
      } else if (wid == GC_W - 1 && !self) {
        for (int r = lane; r < nr; r += 32) acc = fma(s_v[r], s_v[r], acc);
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (lane == 0) s_vv = acc;
      }
      __syncthreads();  // the scratch may still hold an update's partial sums
      if (wid < rg * cg && c < n) s_red[g * n + c] = acc;
      __syncthreads();
      double s = 0.0;
      if (tid < n)
        for (int x = 0; x < rg; ++x) s += s_red[x * n + tid];
      __syncthreads();
      if (tid < n) s_red[tid] = s;
      if (tid == 0) s_red[n] = self ? 0.0 : s_vv;
    } else {
      __syncthreads();
      for (int c = wid; c < K; c += GC_W) {
        double acc = 0.0;
        if (c == n) {
          if (!self)
            for (int r = lane; r < nr; r += 32) acc = fma(s_v[r], s_v[r], acc);
        } else if (self || c > i || s_sel[c]) {
          const double* x = (c < i) ? Q + (int64_t)c * P.ldq : A + (int64_t)c * P.lda;
          double a1 = 0.0;
          int r = lane;
          for (; r + 96 < nr; r += 128) {
            const double x0 = x[r], x1 = x[r + 32], x2 = x[r + 64], x3 = x[r + 96];
            acc = fma(x0, self ? x0 : s_v[r], acc);
            a1 = fma(x1, self ? x1 : s_v[r + 32], a1);
            acc = fma(x2, self ? x2 : s_v[r + 64], acc);
            a1 = fma(x3, self ? x3 : s_v[r + 96], a1);
          }
          for (; r < nr; r += 32) {
            const double x0 = x[r];
            acc = fma(x0, self ? x0 : s_v[r], acc);
          }
          acc += a1;
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (lane == 0) s_red[c] = acc;
      }
    }
    __syncthreads();
  };
  // out[j] = sum over k of rows j0 .. of TH, j < i: columns of the lower triangle (mode 0: s_r = T s_h) or
  // its rows (mode 1: s_r(l) = sum_k s_h(k) T(k, l))
  auto apply_t = [&](int i, int mode) {
    const int jg = (i + 31) / 32, lg = GC_W / jg, g = wid / jg, j = (wid % jg) * 32 + lane;
    double acc = 0.0;
    if (wid < lg * jg) {
      const int per = (i + lg - 1) / lg, la = g * per, lb = min(i, la + per);
      if (j < i)
        for (int l = la; l < lb; ++l) {
          if (mode == 0 ? l <= j : l >= j) acc = fma(TH[mode == 0 ? j * LD + l : l * LD + j], s_h[l], acc);
        }
      if (j < i) s_red[g * i + j] = acc;
    }
    __syncthreads();
    for (int x = tid; x < i; x += GC_T) {
      double s = 0.0;
      for (int y = 0; y < lg; ++y) s += s_red[y * i + x];
      s_r[x] = s_sel[x] ? s : 0.0;
    }
    __syncthreads();
  };
  // v -= sum_{j < i} r_j q_j
  auto update = [&](int i) {
    if (XS) {
      const int rgs = (nr + 31) / 32, jgs = max(1, GC_W / max(rgs, 1));
      for (int item = wid; item < rgs * jgs; item += GC_W) {
        const int g = item / max(rgs, 1), r = (item % max(rgs, 1)) * 32 + lane;
        const int per = (i + jgs - 1) / jgs, ja = g * per, jb = min(i, ja + per);
        double acc = 0.0;
        if (r < nr)
          for (int j = ja; j < jb; ++j) acc = fma(s_r[j], X[(size_t)r * LD + j], acc);
        if (jgs == 1) {
          if (r < nr) s_v[r] -= acc;
        } else if (r < nr) {
          s_red[g * nr + r] = acc;
        }
      }
      __syncthreads();
      if (jgs > 1) {
        for (int r = tid; r < nr; r += GC_T) {
          double s = 0.0;
          for (int g = 0; g < jgs; ++g) s += s_red[g * nr + r];
          s_v[r] -= s;
        }
        __syncthreads();
      }
    } else {
      for (int r = tid; r < nr; r += GC_T) {
        double acc = 0.0;
        int j = 0;
        for (; j + 8 <= i; j += 8) {
          double q[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) q[u] = s_sel[j + u] ? Q[r + (int64_t)(j + u) * P.ldq] : 0.0;
#pragma unroll
          for (int u = 0; u < 8; ++u) acc = fma(s_r[j + u], q[u], acc);
        }
        for (; j < i; ++j) acc = fma(s_r[j], s_sel[j] ? Q[r + (int64_t)j * P.ldq] : 0.0, acc);
        s_v[r] -= acc;
      }
      __syncthreads();
    }
  };
  auto drop = [&](int i) {  // column i leaves the basis
    for (int r = tid; r < nr; r += GC_T) {
      Q[r + (int64_t)i * P.ldq] = 0.0;
      if (XS) X[(size_t)r * LD + i] = 0.0;
    }
    if (blockIdx.x == 0 && tid == 0) P.sel[i] = 0;
    __syncthreads();
  };

  dots(0, true);
  if (!reduce()) return;
  for (int c = tid; c < n; c += GC_T) {
    s_norm[c] = sqrt(s_tot[c]);
    s_skip[c] = s_norm[c] < P.stol;
  }
  __syncthreads();
  int nsel = 0;
  for (int i = 0; i < n; ++i) {
    double normv = s_norm[i];  // thread 0's copy decides
    if (s_skip[i]) {
      drop(i);
      continue;
    }
    for (int r = tid; r < nr; r += GC_T) s_v[r] = XS ? X[(size_t)r * LD + i] : A[r + (int64_t)i * P.lda];
    for (int l = tid; l < i; l += GC_T) s_h[l] = TH[l * LD + i];  // q_l'a_i (0 for dropped columns)
    __syncthreads();
    // (at most 64 further passes: the reference loops until the norm stops dropping, which takes 1-2)
    for (int pass = 0; pass <= 64; ++pass) {
      if (nsel > 0) {
        if (P.classical) {
          for (int l = tid; l < i; l += GC_T) s_r[l] = s_h[l];
          __syncthreads();
        } else {
          apply_t(i, 0);
        }
        update(i);
        if (blockIdx.x == 0)
          for (int j = tid; j < i; j += GC_T)
            if (s_sel[j]) P.R[j + (int64_t)i * n] = pass ? P.R[j + (int64_t)i * n] + s_r[j] : s_r[j];
      }
      dots(i, false);
      if (!reduce()) return;
      if (tid == 0) {
        const double t = sqrt(s_tot[n]);
        const bool again = pass < 64 && P.rtol >= 0 && t >= P.otol && t < P.rtol * normv;
        s_dec = again ? 2 : (t < P.stol ? 1 : 0);
        s_t = t;
        normv = t;
      }
      for (int l = tid; l < i; l += GC_T) s_h[l] = s_sel[l] ? s_tot[l] : 0.0;
      __syncthreads();
      if (s_dec != 2) break;
    }
    const double t = s_t;
    if (s_dec == 1) {
      drop(i);
      continue;
    }
    for (int r = tid; r < nr; r += GC_T) {
      const double q = s_v[r] / t;
      Q[r + (int64_t)i * P.ldq] = q;
      if (XS) X[(size_t)r * LD + i] = q;
    }
    if (blockIdx.x == 0 && tid == 0) {
      P.sel[i] = 1;
      P.R[i + (int64_t)i * n] = t;
    }
    // the first dots of the columns to come, and the new row of T: T(i, l) = -sum_k (q_i'q_k) T(k, l)
    for (int c = tid; c < n; c += GC_T) {
      if (c > i) TH[i * LD + c] = s_tot[c] / t;
      if (c < i) s_h[c] /= t;
    }
    __syncthreads();
    if (!P.classical && nsel > 0) {
      apply_t(i, 1);
      for (int l = tid; l < i; l += GC_T) TH[i * LD + l] = -s_r[l];
    }
    if (tid == 0) {
      TH[i * LD + i] = 1.0;
      s_sel[i] = 1;
    }
    ++nsel;
    __syncthreads();
  }
}

// shared memory of k_gs_coop
size_t gs_coop_smem(int n, int rows, bool xs) {
  const int LD = n | 1;
  return sizeof(double) * ((size_t)n * LD + rows + 4 * (size_t)n + 1 + std::max(GC_W * n, 1024) +
                           (xs ? (size_t)rows * LD : 0));
}

// *done = false: the shape does not fit (or the grid cannot be resident at once), the column loop takes it
int gs_coop(ofrr_ctx* ctx, bool classical, int64_t m, int64_t n, const double* A, int64_t lda, double* Q, int64_t ldq,
            double stol, double otol, double rtol, double* R, int* select_dev, bool* done) {
  *done = false;
  if (n > GC_MAXN) return OFRR_SUCCESS;
  // 32 rows or more per CTA; one CTA per SM
  const int G = (int)std::min<int64_t>(152, (m + 31) / 32);
  const int64_t rows = (m + G - 1) / G;
  constexpr size_t kMax = 220 * 1024;
  if (rows > 16384) return OFRR_SUCCESS;
  const bool xs = gs_coop_smem((int)n, (int)rows, true) <= kMax;
  const size_t smem = gs_coop_smem((int)n, (int)rows, xs);
  if (smem > kMax) return OFRR_SUCCESS;
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  GsCoop P{};
  P.partial = ws_get<double>(ctx, (size_t)G * (n + 1), &st);
  P.total = ws_get<double>(ctx, (size_t)n + 1, &st);
  P.ctr = ws_get<unsigned>(ctx, 2, &st);
  if (!P.partial || !P.total || !P.ctr) return st;  // the column loop needs more (152 n sums and a column of m)
  P.m = m;
  P.n = (int)n;
  P.lda = lda;
  P.ldq = ldq;
  P.classical = classical ? 1 : 0;
  P.rows = (int)rows;
  P.A = A;
  P.Q = Q;
  P.R = R;
  P.sel = select_dev;
  P.stol = stol;
  P.otol = otol;
  P.rtol = rtol;
  P.err = ctx->dev_flags + kFlagHessWait;
  OFRR_CUDA(cudaMemsetAsync(P.ctr, 0, 2 * sizeof(unsigned), ctx->stream));
  OFRR_CUDA(cudaMemsetAsync(R, 0, sizeof(double) * n * n, ctx->stream));
  void* args[] = {&P};
  const void* f = xs ? (const void*)k_gs_coop<true> : (const void*)k_gs_coop<false>;
  OFRR_TRY(allow_dynamic_smem(f));
  const cudaError_t e = cudaLaunchCooperativeKernel(f, dim3((unsigned)G), dim3(GC_T), args, smem, ctx->stream);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    (void)cudaGetLastError();
    return OFRR_SUCCESS;
  }
  OFRR_CUDA(e);
  OFRR_LAUNCHED(ctx, "k_gs_coop");
  *done = true;
  return OFRR_SUCCESS;
}

template <class TO, class TC>
int gs_run(ofrr_ctx* ctx, bool classical, int64_t m, int64_t n, const TO* A, int64_t lda, TO* Q, int64_t ldq,
           double stol, double otol, double rtol, double* R, int* select_dev) {
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  TO* v = ws_get<TO>(ctx, (size_t)m, &st);
  TO* rr = ws_get<TO>(ctx, (size_t)n + 2, &st);  // r_0..r_{n-1}, then norm scratch
  TC* partial = ws_get<TC>(ctx, (size_t)GS_G * n, &st);
  unsigned int* counters = ws_get<unsigned int>(ctx, (size_t)n, &st);
  int* cols = ws_get<int>(ctx, (size_t)n, &st);
  TO* norms = ws_get<TO>(ctx, (size_t)n, &st);
  if (!v || !rr || !partial || !counters || !cols || !norms) return st;
  OFRR_CUDA(cudaMemsetAsync(counters, 0, sizeof(unsigned int) * n, ctx->stream));
  OFRR_CUDA(cudaMemsetAsync(R, 0, sizeof(double) * n * n, ctx->stream));
  for (int64_t j = 0; j < n; ++j)
    OFRR_CUDA(cudaMemsetAsync(Q + j * ldq, 0, sizeof(TO) * m, ctx->stream));
  const unsigned gu = (unsigned)std::min<int64_t>((m + GS_T - 1) / GS_T, 4 * 152);
  auto norm_of = [&](const TO* x, TO* out) -> int {
    k_gs_reduce<TO, TC><<<dim3(GS_G, 1), GS_T, 0, ctx->stream>>>(m, x, nullptr, 0, nullptr, partial, counters, out);
    OFRR_LAUNCHED(ctx, "k_gs_reduce");
    return OFRR_SUCCESS;
  };
  // the norms of the original columns (column i is untouched until its turn)
  for (int64_t i = 0; i < n; ++i) OFRR_TRY(norm_of(A + i * lda, norms + i));
  std::vector<TO> hn((size_t)n);
  OFRR_TRY(fetch(ctx, hn.data(), norms, sizeof(TO) * n));
  std::vector<int> sel((size_t)n, 0), hcols;
  // one projection pass of v against the selected columns hcols (R column i; acc: accumulate)
  auto pass = [&](int64_t i, int acc) -> int {
    const int nc = (int)hcols.size();
    if (nc == 0) return OFRR_SUCCESS;
    double* Rcol = R + i * n;
    if (classical) {
      k_gs_reduce<TO, TC><<<dim3(GS_G, nc), GS_T, 0, ctx->stream>>>(m, v, Q, ldq, cols, partial, counters, rr);
      OFRR_LAUNCHED(ctx, "k_gs_reduce");
      k_gs_update<TO, TC><<<gu, GS_T, 0, ctx->stream>>>(m, v, Q, ldq, cols, nc, rr, Rcol, acc);
      OFRR_LAUNCHED(ctx, "k_gs_update");
    } else {
      for (int c = 0; c < nc; ++c) {
        k_gs_reduce<TO, TC><<<dim3(GS_G, 1), GS_T, 0, ctx->stream>>>(m, v, Q, ldq, cols + c, partial, counters, rr);
        OFRR_LAUNCHED(ctx, "k_gs_reduce");
        k_gs_update<TO, TC><<<gu, GS_T, 0, ctx->stream>>>(m, v, Q, ldq, cols + c, 1, rr, Rcol, acc);
        OFRR_LAUNCHED(ctx, "k_gs_update");
      }
    }
    return OFRR_SUCCESS;
  };
  for (int64_t i = 0; i < n; ++i) {
    double normv = host_double(hn[(size_t)i]);
    if (normv < stol) continue;
    OFRR_CUDA(cudaMemcpyAsync(v, A + i * lda, sizeof(TO) * m, cudaMemcpyDeviceToDevice, ctx->stream));
    OFRR_TRY(pass(i, 0));
    TO ht;
    OFRR_TRY(norm_of(v, rr + n));
    OFRR_TRY(fetch(ctx, &ht, rr + n, sizeof(TO)));
    double t = host_double(ht);
    // (at most 64 passes: the reference loops until the norm stops dropping, which takes 1-2)
    for (int guard = 0; rtol >= 0 && t >= otol && t < rtol * normv && guard < 64; ++guard) {
      normv = t;
      OFRR_TRY(pass(i, 1));
      OFRR_TRY(norm_of(v, rr + n));
      OFRR_TRY(fetch(ctx, &ht, rr + n, sizeof(TO)));
      t = host_double(ht);
    }
    if (t < stol) continue;
    k_gs_scale<TO, TC><<<gu, GS_T, 0, ctx->stream>>>(m, v, rr + n, Q + i * ldq, R + i * n + i);
    OFRR_LAUNCHED(ctx, "k_gs_scale");
    sel[(size_t)i] = 1;
    hcols.push_back((int)i);
    OFRR_CUDA(cudaMemcpyAsync(cols + hcols.size() - 1, &hcols.back(), sizeof(int), cudaMemcpyHostToDevice,
                              ctx->stream));
    OFRR_TRY(sync_and_check(ctx));  // the pageable source of the index copy stays valid until here
  }
  OFRR_CUDA(cudaMemcpyAsync(select_dev, sel.data(), sizeof(int) * n, cudaMemcpyHostToDevice, ctx->stream));
  return sync_and_check(ctx);
}

}  // namespace

int gs_basis_impl(ofrr_ctx* ctx, bool classical, ofrr_dtype tin, ofrr_dtype tout, ofrr_dtype tc, int64_t m,
                  int64_t n, const void* A, int64_t lda, void* Q, int64_t ldq, double select_tol, double* R_dev,
                  int* select_dev, double orth_tol, double reorth_tol) {
  if (n <= 0 || m <= 0) return OFRR_SUCCESS;
  if (m < n) return OFRR_ERR_BLAS_INVALID_SIZE;  // mgs.m:50 / cgs.m:50 assert a tall-thin A
  const double e = dtype_eps(tout);
  const double stol = select_tol < 0 ? e : select_tol;
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  const void* Ain = A;
  int64_t ldin = lda;
  const char* qb = (const char*)Q;
  const char* ab = (const char*)A;
  const bool alias = ab < qb + (size_t)ldq * n * dtype_size(tout) && qb < ab + (size_t)lda * n * dtype_size(tin);
  if (tin != tout || alias) {  // A = precision_output(A), in a copy when it overlaps Q
    void* w = ws_alloc(ctx, (size_t)m * n * dtype_size(tout), &st);
    if (!w) return st;
    OFRR_TRY(cast_impl(ctx, tin, tout, m, n, A, lda, w, m));
    Ain = w;
    ldin = m;
  }
  // the tolerances are compared in the output precision, as mgs.m:141-152 casts them
  const double s_t = round_to(tout, stol), o_t = round_to(tout, std::isnan(orth_tol) ? e : orth_tol),
               r_t = round_to(tout, std::isnan(reorth_tol) ? 1.0 / std::sqrt(2.0) : reorth_tol);
  // FP64 throughout: one cooperative launch.  With a narrower storage type every term of an update is rounded
  // to it and the next dot sees that rounding, so those bases keep the column loop's order of operations.  So does
  // MGS without re-orthogonalisation: its one pass takes out what a dot against the already updated vector sees, the
  // inverse compact form only what the first dots saw, and of columns dependent to working precision (a Hilbert block
  // of 1000 x 64) 62 stay above select_tol = eps where the sequential pass leaves 47.  With re-orthogonalisation both
  // end at the same residuals, up to rounding: it is effective when a column that loses half its norm is projected
  // again, down to the norms that are dropped.
  const bool again = r_t >= 0.5 && o_t <= std::max(s_t, e);
  if (tout == OFRR_F64 && tc == OFRR_F64 && (classical || again)) {
    bool done = false;
    OFRR_TRY(gs_coop(ctx, classical, m, n, (const double*)Ain, ldin, (double*)Q, ldq, s_t, o_t, r_t, R_dev,
                     select_dev, &done));
    if (done) return OFRR_SUCCESS;
  }
  OFRR_DISPATCH_STORAGE(tout, TO, OFRR_DISPATCH_COMPUTE(tc, TC, {
    OFRR_TRY((gs_run<TO, TC>(ctx, classical, m, n, (const TO*)Ain, ldin, (TO*)Q, ldq, s_t, o_t, r_t, R_dev,
                             select_dev)));
  }));
  return OFRR_SUCCESS;
}

}  // namespace ofrr

using namespace ofrr;

extern "C" int ofrr_gs_basis(ofrr_ctx* ctx, int classical, ofrr_dtype tin, ofrr_dtype tout, ofrr_dtype tcompute,
                             int64_t m, int64_t n, const void* A, int64_t lda, void* Q, int64_t ldq, double select_tol,
                             double orth_tol, double reorth_tol, double* R_host, int* skip_host) {
  if (!ctx || m < 0 || n < 0 || !dtype_valid(tin) || !dtype_valid(tout)) return OFRR_ERR_INVALID_ARGUMENT;
  if (tcompute != OFRR_F64 && tcompute != OFRR_F32) return OFRR_ERR_BLAS_UNSUPPORTED_TYPE;
  if (m < n) return OFRR_ERR_BLAS_INVALID_SIZE;
  if (n == 0) return OFRR_SUCCESS;
  if (!A || !Q || lda < m || ldq < m) return OFRR_ERR_INVALID_ARGUMENT;
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  // R, then the flags: adjacent, for one copy to the host
  double* R = (double*)ws_alloc(ctx, sizeof(double) * n * n + sizeof(int) * n, &st);
  if (!R) return st;
  int* sel = (int*)(R + n * n);
  OFRR_TRY(gs_basis_impl(ctx, classical != 0, tin, tout, tcompute, m, n, A, lda, Q, ldq, select_tol, R, sel,
                         orth_tol, reorth_tol));
  std::vector<int> hsel((size_t)n);
  OFRR_TRY(fetch_parts(ctx, R, {{R_host, sizeof(double) * n * n}, {hsel.data(), sizeof(int) * n}}));
  if (skip_host)
    for (int64_t j = 0; j < n; ++j) skip_host[j] = hsel[(size_t)j] ? 0 : 1;
  return OFRR_SUCCESS;
}
