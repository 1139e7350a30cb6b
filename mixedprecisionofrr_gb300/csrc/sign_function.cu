// Matrix sign function and the basis of its invariant subspace (the thick restart of the Krylov eigensolver),
// FP64, n <= 96.
//
// S = sign(X) by Newton's iteration X <- (mu X + (mu X)^-1) / 2 with determinant scaling mu in the first steps, the
// inverse by Gauss-Jordan elimination with partial pivoting [N. J. Higham, Functions of Matrices, SIAM 2008, ch. 5].
//
// GB300 runs an FP64 warp instruction in 64 cycles of an SM sub-partition, so one elimination step of an n = 64 matrix
// on one SM takes 2048 cycles, and the chain pivot search -> reciprocal -> next column about 1000 more.  Here the
// columns are spread over a cluster of 8 CTAs and held in registers (a warp owns one column, two above n = 64; a lane
// one row of 32), and a step is pure dataflow: the warp that owns column k + 1 applies step k to it first, finds its
// pivot (integer comparisons: an FP64 compare costs 105 cycles) and its reciprocal, and pushes (pivot row, reciprocal,
// column) to every CTA's shared memory, where one mbarrier per step completes; all other warps follow.  A Newton step
// ends in two cluster barriers: the columns of the inverse go to their places (row interchanges undone), and the
// convergence sums are exchanged.  Every entry meets the same operations in the same order as in a plain sequential
// elimination.  A restart of the
// 64-column solver (n = 65): 721 us, against 3.36 ms on one CTA with the matrix in shared memory (a division, a
// logarithm and block barriers in every step's chain).
#include <algorithm>

#include "f64_ops.cuh"
#include "ofrr_internal.cuh"
#include "tcgen05.cuh"

namespace ofrr {
namespace {

constexpr int kSignMaxN = 96;
constexpr int kSignCtas = 8;
constexpr int kSignWarps = 8;
constexpr int kSignHead = 3;  // per step, ahead of the column: pivot row, pivot, its reciprocal

__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, int* err) {
  auto done = [&]() {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(tc::smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
  };
  if (done()) return true;
  const uint64_t t0 = tc::globaltimer();
  for (int i = 0;; ++i) {
    if (done()) return true;
    if ((i & 63) == 63 && tc::globaltimer() - t0 > 2000000000ull) {
      atomicCAS(err, 0, 31);
      return false;
    }
  }
}
// one 8-byte word into another CTA's shared memory; its arrival counts on that CTA's barrier
__device__ __forceinline__ void push_f64(unsigned dst, unsigned bar, double v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void arrive_local(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// row r of a column spread over a warp (row 32 q + lane in v[q]); r is the same in every lane
template <int SL>
__device__ __forceinline__ double row_of(const double (&v)[SL], int r) {
  double x = v[0];
#pragma unroll
  for (int q = 1; q < SL; ++q)
    if ((r >> 5) == q) x = v[q];
  return __shfl_sync(0xffffffffu, x, r & 31);
}

// SL = ceil(n / 32) rows per lane, CW columns per warp
template <int SL, int CW>
__global__ void __launch_bounds__(32 * kSignWarps, 1) k_sign_cluster(int n, double* __restrict__ Xg, int maxit, double tol,
                                                                  int* __restrict__ flag, int* __restrict__ err) {
  extern __shared__ __align__(16) double sg[];
  const int me = (int)cluster_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int PC = (n + kSignCtas - 1) / kSignCtas;  // columns per CTA
  const int stride = n + kSignHead;
  double* info = sg;                               // n steps x (head, column)
  double* recv = info + (size_t)n * stride;        // PC columns of the inverse, in place
  uint64_t* bars = reinterpret_cast<uint64_t*>(recv + (size_t)PC * n);
  __shared__ double s_log[kSignMaxN], s_part[2][kSignWarps], s_all[2][kSignCtas];
  __shared__ double s_mu;
  __shared__ int s_bad;  // this CTA met a zero or NaN pivot
  if (tid < n) tc::mbar_init(&bars[tid], 1);
  if (tid == 0) s_bad = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  // this warp's columns and its entries of X
  int col[CW];
  double x[CW][SL];
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const int l = warp + kSignWarps * c;
    col[c] = (l < PC && me * PC + l < n) ? me * PC + l : -1;
#pragma unroll
    for (int q = 0; q < SL; ++q) {
      const int i = 32 * q + lane;
      x[c][q] = (col[c] >= 0 && i < n) ? Xg[i + (size_t)col[c] * n] : 0.0;
    }
  }
  const bool earlier = *flag != 0;  // an earlier stage met a singular matrix
  cluster_arrive();
  cluster_wait();
  bool singular = earlier, late = false;
  auto pivot_row = [&](int k) {
    const unsigned p = (unsigned)__double_as_longlong(info[(size_t)k * stride]);
    return p < (unsigned)n ? (int)p : k;  // always in range, but after a wait that ran out
  };

  for (int it = 0; it < maxit && !singular; ++it) {
    const uint32_t parity = it & 1;
    if (tid < n && tid / PC != me) tc::mbar_expect_tx(&bars[tid], (uint32_t)stride * 8);
    double y[CW][SL];
#pragma unroll
    for (int c = 0; c < CW; ++c)
#pragma unroll
      for (int q = 0; q < SL; ++q) y[c][q] = x[c][q];

    // pivot of column k (first largest |entry| of rows >= k; NaN never), its reciprocal, and the column with rows k
    // and p exchanged and row k cleared, to every CTA
    auto publish = [&](int k, const double (&v)[SL]) {
      long long best = -1;
      int bi = k;
#pragma unroll
      for (int q = 0; q < SL; ++q) {
        const int i = 32 * q + lane;
        const long long a = __double_as_longlong(v[q]) & 0x7fffffffffffffffLL;
        if (i >= k && i < n && a <= 0x7ff0000000000000LL && a > best) {
          best = a;
          bi = i;
        }
      }
      const int hi = (int)(best >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
      const unsigned lo = (hi == mh) ? (unsigned)best : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
      const int p = __reduce_min_sync(0xffffffffu, (hi == mh && lo == ml) ? bi : 0x7fffffff);
      const double d = row_of<SL>(v, p), vk = row_of<SL>(v, k);
      const long long ad = __double_as_longlong(d) & 0x7fffffffffffffffLL;
      const bool bad = ad == 0 || ad > 0x7ff0000000000000LL;  // zero or NaN
      double* mine = info + (size_t)k * stride;
      const unsigned off = tc::smem_u32(mine), boff = tc::smem_u32(&bars[k]);
      unsigned base[kSignCtas - 1], rbar[kSignCtas - 1];
#pragma unroll
      for (int t = 0; t < kSignCtas - 1; ++t) {
        const unsigned r = (unsigned)(me + 1 + t) % kSignCtas;  // the next CTA first
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[t]) : "r"(off), "r"(r));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbar[t]) : "r"(boff), "r"(r));
      }
#pragma unroll
      for (int q = 0; q < SL; ++q) {
        const int i = 32 * q + lane;
        if (i < n) {
          const double s = (i == k) ? 0.0 : (i == p) ? vk : v[q];
          mine[kSignHead + i] = s;
#pragma unroll
          for (int t = 0; t < kSignCtas - 1; ++t) push_f64(base[t] + (kSignHead + i) * 8, rbar[t], s);
        }
      }
      const double dinv = f64::rcp(d);
      if (lane < kSignHead) {
        const double h = (lane == 0) ? __longlong_as_double((long long)p) : (lane == 1) ? d : dinv;
        mine[lane] = h;
#pragma unroll
        for (int t = 0; t < kSignCtas - 1; ++t) push_f64(base[t] + lane * 8, rbar[t], h);
      }
      if (bad && lane == 0) s_bad = 1;  // the step goes on: the cluster stops together, after it
      __syncwarp();
      if (lane == 0) arrive_local(&bars[k]);
    };
    if (col[0] == 0) publish(0, y[0]);

    for (int k = 0; k < n; ++k) {
      if (!late && !__all_sync(0xffffffffu, wait_cluster(&bars[k], parity, err))) late = true;
      const double* in = info + (size_t)k * stride;
      const int p = pivot_row(k);
      const double dinv = in[2];
      double s[SL];
#pragma unroll
      for (int q = 0; q < SL; ++q) {
        const int i = 32 * q + lane;
        s[q] = (i < n) ? in[kSignHead + i] : 0.0;
      }
      auto apply = [&](int j, double (&v)[SL]) {
        if (j == k) {  // becomes a column of the inverse: dinv in row k, 0 - s dinv elsewhere
#pragma unroll
          for (int q = 0; q < SL; ++q) v[q] = (32 * q + lane == k) ? dinv : fma(-s[q], dinv, 0.0);
        } else {
          const double vk = row_of<SL>(v, k), rk = __dmul_rn(row_of<SL>(v, p), dinv);
#pragma unroll
          for (int q = 0; q < SL; ++q) {
            const int i = 32 * q + lane;
            const double t = fma(-s[q], rk, (i == p) ? vk : v[q]);
            v[q] = (i == k) ? rk : t;
          }
        }
      };
      int first = -1;  // the warp's column k + 1, if it has it, goes ahead
#pragma unroll
      for (int c = 0; c < CW; ++c)
        if (col[c] == k + 1) {
          first = c;
          apply(col[c], y[c]);
          publish(k + 1, y[c]);
        }
#pragma unroll
      for (int c = 0; c < CW; ++c)
        if (col[c] >= 0 && c != first) apply(col[c], y[c]);
    }
    // place of every computed column once the row interchanges are undone as column interchanges
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      if (col[c] < 0) continue;
      int d = col[c];
#pragma unroll 8
      for (int k = n - 1; k >= 0; --k) {
        const int p = pivot_row(k);
        d = (d == k) ? p : (d == p) ? k : d;
      }
      const unsigned dst = cluster_map(recv + (size_t)(d % PC) * n, (unsigned)(d / PC));
#pragma unroll
      for (int q = 0; q < SL; ++q) {
        const int i = 32 * q + lane;
        if (i < n) asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(dst + i * 8), "d"(y[c][q]) : "memory");
      }
    }
    if (it < 4) {  // determinant scaling in the first steps
      if (tid < n) s_log[tid] = log(fabs(info[(size_t)tid * stride + 1]));
      __syncthreads();
      if (tid == 0) {
        double ld = 0.0;
        for (int k = 0; k < n; ++k) ld += s_log[k];
        s_mu = exp(-ld / n);
      }
    }
    cluster_arrive();
    cluster_wait();
    const double mu = (it < 4) ? s_mu : 1.0;
    double num = 0.0, den = 0.0;
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      if (col[c] < 0) continue;
#pragma unroll
      for (int q = 0; q < SL; ++q) {
        const int i = 32 * q + lane;
        if (i < n) {
          const double v = recv[(size_t)(col[c] - me * PC) * n + i];
          const double xn = (it < 4) ? 0.5 * (mu * x[c][q] + v / mu) : 0.5 * (x[c][q] + v);
          num += (xn - x[c][q]) * (xn - x[c][q]);
          den += xn * xn;
          x[c][q] = xn;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      num += __shfl_xor_sync(0xffffffffu, num, o);
      den += __shfl_xor_sync(0xffffffffu, den, o);
    }
    if (lane == 0) {
      s_part[0][warp] = num;
      s_part[1][warp] = den;
    }
    __syncthreads();
    if (tid < 2 * kSignCtas) {  // this CTA's sums to every CTA
      const int w = tid & 1;
      double t = 0.0;
      for (int k = 0; k < kSignWarps; ++k) t += s_part[w][k];
      if (s_bad) t = -1.0;
      asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_map(&s_all[w][me], (unsigned)(tid >> 1))), "d"(t)
                   : "memory");
    }
    cluster_arrive();
    cluster_wait();
    double sn = 0.0, sd = 0.0;
    for (int r = 0; r < kSignCtas; ++r) {
      singular = singular || s_all[0][r] == -1.0;
      sn += s_all[0][r];
      sd += s_all[1][r];
    }
    if (sn <= tol * tol * sd && it >= 1) break;
  }
  // no CTA leaves while another may still write to it
  cluster_arrive();
  cluster_wait();
  if (singular) {
    if (!earlier && me == 0 && tid == 0) *flag = 1;
    return;
  }
#pragma unroll
  for (int c = 0; c < CW; ++c)
#pragma unroll
    for (int q = 0; q < SL; ++q) {
      const int i = 32 * q + lane;
      if (col[c] >= 0 && i < n) Xg[i + (size_t)col[c] * n] = x[c][q];
    }
}

// Q (n x p) = orthonormal basis of range((I + S) / 2): the projector applied to a fixed pseudo-random
// block (splitmix64 hashes), then modified Gram-Schmidt twice, on one CTA.  A warp owns whole columns (in shared
// memory; lanes hold rows 32 q + lane); as soon as column c is final every warp takes it out of its own later
// columns, and only the second pass of the next column is serial: p^2 / 2 dependent inner products instead of p^2,
// each one warp wide (no block reduction).  n = 65: 324 us
// against 672 us with block reductions and the hash of the block computed for every product.
constexpr int kProjWarps = 16;

template <int SL>
__global__ void __launch_bounds__(32 * kProjWarps) k_proj_basis(int n, int p, const double* __restrict__ S,
                                                                double* __restrict__ Q, int* __restrict__ err) {
  extern __shared__ __align__(16) double pb[];
  double* Qs = pb;                        // n x p
  double* Om = Qs + (size_t)n * p;        // n x p
  double* P = Om + (size_t)n * p;         // n x n
  __shared__ uint64_t bars[kSignMaxN];
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
  if (tid < p) tc::mbar_init(&bars[tid], 1);
  for (int e = tid; e < n * p; e += nthr) {
    const int k = e % n, c = e / n;
    unsigned long long h = 0x9e3779b97f4a7c15ULL * (unsigned long long)(k + 1) + 0xbf58476d1ce4e5b9ULL * (c + 1);
    h ^= h >> 31;
    h *= 0x94d049bb133111ebULL;
    h ^= h >> 29;
    Om[e] = (double)(h >> 11) * (1.0 / 9007199254740992.0) - 0.5;
  }
  for (int e = tid; e < n * n; e += nthr) P[e] = 0.5 * (S[e] + ((e % n == e / n) ? 1.0 : 0.0));
  __syncthreads();
  for (int e = tid; e < n * p; e += nthr) {
    const int i = e % n, c = e / n;
    double acc = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; ++k) acc = fma(P[i + (size_t)k * n], Om[k + (size_t)c * n], acc);
    Qs[e] = acc;
  }
  __syncthreads();
  // sum over the rows of a column: one 32-row tree per q, then the partial sums in the order of q
  auto rows_sum = [&](double (&v)[SL]) -> double {
#pragma unroll
    for (int q = 0; q < SL; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], 16);
    // after the first level 16 lanes hold all that is left of a tree: two trees share the warp from here
    double a = v[0];
    if constexpr (SL > 1) a = (lane & 16) ? v[1] : v[0];
    double b = (SL > 2) ? v[SL - 1] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      if (SL > 2) b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    double t = 0.0 + __shfl_sync(0xffffffffu, a, 0);
    if (SL > 1) t += __shfl_sync(0xffffffffu, a, 16);
    if (SL > 2) t += b;
    return t;
  };
  auto load = [&](int c, double (&v)[SL]) {
#pragma unroll
    for (int q = 0; q < SL; ++q) v[q] = (32 * q + lane < n) ? Qs[(size_t)c * n + 32 * q + lane] : 0.0;
  };
  auto store = [&](int c, const double (&v)[SL]) {
#pragma unroll
    for (int q = 0; q < SL; ++q)
      if (32 * q + lane < n) Qs[(size_t)c * n + 32 * q + lane] = v[q];
  };
  auto project = [&](const double (&q2)[SL], double (&v)[SL]) {
    double t[SL];
#pragma unroll
    for (int q = 0; q < SL; ++q) t[q] = __dmul_rn(q2[q], v[q]);
    const double dt = rows_sum(t);
#pragma unroll
    for (int q = 0; q < SL; ++q) v[q] = fma(-dt, q2[q], v[q]);
  };
  auto finish = [&](int c, double (&v)[SL]) {  // second pass against the final columns, unit norm
    for (int c2 = 0; c2 < c; ++c2) {
      double q2[SL];
      load(c2, q2);
      project(q2, v);
    }
    double t[SL];
#pragma unroll
    for (int q = 0; q < SL; ++q) t[q] = __dmul_rn(v[q], v[q]);
    const double s = rows_sum(t);
    const double sc = (s > 0.0) ? 1.0 / sqrt(s) : 0.0;
#pragma unroll
    for (int q = 0; q < SL; ++q) v[q] *= sc;
    store(c, v);
    __syncwarp();
    if (lane == 0) arrive_local(&bars[c]);
  };
  if (warp == 0 && p > 0) {
    double v[SL];
    load(0, v);
    finish(0, v);
  }
  bool late = false;
  for (int c2 = 0; c2 + 1 < p; ++c2) {
    if (!late && !__all_sync(0xffffffffu, wait_cluster(&bars[c2], 0, err))) late = true;
    double q2[SL];
    load(c2, q2);
    if ((c2 + 1) % kProjWarps == warp) {
      double v[SL];
      load(c2 + 1, v);
      project(q2, v);
      finish(c2 + 1, v);
    }
    for (int c = warp; c < p; c += kProjWarps)
      if (c > c2 + 1) {
        double v[SL];
        load(c, v);
        project(q2, v);
        store(c, v);
        __syncwarp();
      }
  }
  __syncthreads();
  for (int e = tid; e < n * p; e += nthr) Q[e] = Qs[e];
}

template <int SL, int CW>
int launch_sign(ofrr_ctx* ctx, int n, double* X, int maxit, double tol, int* flag) {
  const int PC = (n + kSignCtas - 1) / kSignCtas;
  const size_t smem = ((size_t)n * (n + kSignHead) + (size_t)PC * n + n) * sizeof(double);
  OFRR_TRY(allow_smem(k_sign_cluster<SL, CW>));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kSignCtas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(kSignCtas);
  cfg.blockDim = dim3(32 * kSignWarps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  OFRR_CUDA(cudaLaunchKernelEx(&cfg, k_sign_cluster<SL, CW>, n, X, maxit, tol, flag, ctx->dev_flags + kFlagTcWait));
  OFRR_LAUNCHED(ctx, "k_sign_cluster");
  return OFRR_SUCCESS;
}

template <int SL>
int launch_proj(ofrr_ctx* ctx, int n, int p, const double* S, double* Q) {
  OFRR_TRY(allow_smem(k_proj_basis<SL>));
  const size_t smem = (2 * (size_t)n * p + (size_t)n * n) * sizeof(double);
  k_proj_basis<SL><<<1, 32 * kProjWarps, smem, ctx->stream>>>(n, p, S, Q, ctx->dev_flags + kFlagTcWait);
  OFRR_LAUNCHED(ctx, "k_proj_basis");
  return OFRR_SUCCESS;
}

}  // namespace

// X (n x n, ld n) <- sign(X); *flag = 1 (X unchanged) when a step meets a singular matrix
int sign_newton(ofrr_ctx* ctx, int n, double* X, int maxit, double tol, int* flag) {
  if (n < 1 || n > kSignMaxN) return OFRR_ERR_BLAS_INVALID_SIZE;
  if (n <= 32) return launch_sign<1, 1>(ctx, n, X, maxit, tol, flag);
  if (n <= 64) return launch_sign<2, 1>(ctx, n, X, maxit, tol, flag);
  return launch_sign<3, 2>(ctx, n, X, maxit, tol, flag);
}

// Q (n x p, ld n): orthonormal basis of range((I + S) / 2), p its rank
int sign_basis(ofrr_ctx* ctx, int n, int p, const double* S, double* Q) {
  if (n < 1 || n > kSignMaxN || p < 1 || p > n) return OFRR_ERR_BLAS_INVALID_SIZE;
  if (n <= 32) return launch_proj<1>(ctx, n, p, S, Q);
  if (n <= 64) return launch_proj<2>(ctx, n, p, S, Q);
  return launch_proj<3>(ctx, n, p, S, Q);
}

}  // namespace ofrr
