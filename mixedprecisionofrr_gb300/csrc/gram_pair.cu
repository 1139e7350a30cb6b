// G = V' W and M = V' V of a Rayleigh-Ritz step in one pass over FP64 V and W (K x b, column-major, b <= 128).
//
// FP64 runs at ~594 GFMA/s on this part (64 cycles of an SM sub-partition per warp instruction; the FP64 mma.sync gives
// 522), so a Gram matrix of many rows is bound by its multiply-adds, and one of few rows by launches.  Two library
// products cost 2 K b^2 multiply-adds and two launches each with their split-K sums.  Here M's upper triangle is not
// formed (1.5 K b^2 plus the diagonal), the rows of V are staged once for both, and one kernel sums the chunks of both.
// A thread owns one 4 x 4 block of G or of M's lower triangle (blocks of one CTA: `per`), and for few blocks one of KS
// row slices of the slab, added in slice order at the end.  K is cut into chunks of kc rows over the grid; their partial
// sums are added in a fixed order, so results do not depend on the schedule.  117600 rows, b = 64: 1.34 ms for both (two library
// products 1.79 ms; the multiply-adds alone 1.24 ms); 4160 rows, b = 32: about half of the 76 us of two products with
// their split-K sums.
#include <algorithm>

#include "ofrr_internal.cuh"

namespace ofrr {
namespace {

constexpr int kGpSlab = 32;      // rows staged at a time
constexpr int kGpThreads = 512;  // at most

__host__ __device__ inline int gp_items(int T) { return T * T + T * (T + 1) / 2; }

// block e: V column block i against column block j of W (lower = false) or of V (lower = true, i >= j)
__device__ __forceinline__ void gp_decode(int e, int T, int* i, int* j, bool* lower) {
  if (e < T * T) {
    *i = e / T;
    *j = e % T;
    *lower = false;
  } else {
    const int t = e - T * T;
    int r = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= t) ++r;
    while (r * (r + 1) / 2 > t) --r;
    *i = r;
    *j = t - r * (r + 1) / 2;
    *lower = true;
  }
}

__global__ void __launch_bounds__(kGpThreads) k_gram_pair(int64_t K, int b, const double* __restrict__ V, int64_t ldv,
                                                          const double* __restrict__ W, int64_t ldw, int64_t kc, int per,
                                                          int KS, double* __restrict__ partial) {
  extern __shared__ double sm[];
  const int T = (b + 3) / 4, items = gp_items(T), bp = 4 * T, S = 2 * bp + 1;  // slab row: V then W, odd stride
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int e = blockIdx.y * per + tid % per, ks = tid / per;
  const bool on = ks < KS && e < items;
  int i = 0, j = 0;
  bool lower = false;
  if (on) gp_decode(e, T, &i, &j, &lower);
  const double* pa = sm + 4 * i;
  const double* pb = sm + (lower ? 4 * j : bp + 4 * j);
  const int64_t k0 = (int64_t)blockIdx.x * kc, k1 = min(K, k0 + kc);
  double acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0.0;
  for (int64_t kb = k0; kb < k1; kb += kGpSlab) {
    const int rows = (int)min((int64_t)kGpSlab, k1 - kb);
    for (int x = tid; x < kGpSlab * 2 * bp; x += nthr) {
      const int r = x % kGpSlab, c = x / kGpSlab, cc = c < bp ? c : c - bp;
      double v = 0.0;
      if (r < rows && cc < b) v = c < bp ? V[kb + r + (int64_t)cc * ldv] : W[kb + r + (int64_t)cc * ldw];
      sm[r * S + c] = v;
    }
    __syncthreads();
    if (on) {
#pragma unroll 2
      for (int r = ks; r < rows; r += KS) {
        double a[4], c[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = pa[r * S + u];
          c[u] = pb[r * S + u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], c[v], acc[u][v]);
      }
    }
    __syncthreads();
  }
  if (KS > 1) {
    if (on && ks > 0)
#pragma unroll
      for (int x = 0; x < 16; ++x) sm[(size_t)x * nthr + tid] = acc[x >> 2][x & 3];
    __syncthreads();
    if (on && ks == 0)
      for (int s = 1; s < KS; ++s)
#pragma unroll
        for (int x = 0; x < 16; ++x) acc[x >> 2][x & 3] += sm[(size_t)x * nthr + s * per + tid];
  }
  if (on && ks == 0) {
    double* P = partial + (size_t)blockIdx.x * items * 16 + (size_t)e;
#pragma unroll
    for (int x = 0; x < 16; ++x) P[(size_t)x * items] = acc[x >> 2][x & 3];
  }
}

// sums over the chunks: 32 entries per block, eight slices of the chunks each, then the slices in order
__global__ void __launch_bounds__(256) k_gram_pair_sum(int b, int chunks, const double* __restrict__ partial,
                                                       double* __restrict__ G, double* __restrict__ M) {
  __shared__ double red[8][33];
  const int T = (b + 3) / 4, items = gp_items(T), total = items * 16;
  const int o = threadIdx.x & 31, sl = threadIdx.x >> 5, x = blockIdx.x * 32 + o;
  double s = 0.0;
  if (x < total)
#pragma unroll 4
    for (int c = sl; c < chunks; c += 8) s += partial[(size_t)c * total + x];
  red[sl][o] = s;
  __syncthreads();
  if (sl != 0 || x >= total) return;
#pragma unroll
  for (int q = 1; q < 8; ++q) s += red[q][o];
  int i, j;
  bool lower;
  gp_decode(x % items, T, &i, &j, &lower);
  const int m = 4 * i + ((x / items) >> 2), n = 4 * j + ((x / items) & 3);
  if (m >= b || n >= b) return;
  if (!lower) {
    G[m + (size_t)n * b] = s;
  } else {
    M[m + (size_t)n * b] = s;
    if (i != j) M[n + (size_t)m * b] = s;  // (a diagonal block is formed whole)
  }
}

}  // namespace

// G = V' W, M = V' V (b x b, ld b, FP64) for V, W of K rows, 1 <= b <= 128
int gram_pair_f64(ofrr_ctx* ctx, int64_t K, int b, const double* V, int64_t ldv, const double* W, int64_t ldw, double* G,
                  double* M) {
  if (b < 1 || b > 128 || K < 1) return OFRR_ERR_BLAS_INVALID_SIZE;
  const int T = (b + 3) / 4, items = gp_items(T);
  const int ny = (items + kGpThreads - 1) / kGpThreads, per = (items + ny - 1) / ny;
  const int KS = std::max(1, std::min(kGpSlab / 2, kGpThreads / per));
  const int threads = (per * KS + 31) / 32 * 32;
  // one chunk per SM, two where that leaves at least a slab per slice of it
  const int64_t want = (K >= (int64_t)152 * 2 * kGpSlab) ? 2 * 152 / ny : 152 / ny;
  const int64_t chunks0 = std::max<int64_t>(1, std::min<int64_t>(std::max<int64_t>(want, 1), (K + KS - 1) / KS));
  const int64_t kc = (K + chunks0 - 1) / chunks0;
  const int chunks = (int)((K + kc - 1) / kc);
  int st = OFRR_SUCCESS;
  WsScope scope(ctx);
  double* partial = ws_get<double>(ctx, (size_t)chunks * items * 16, &st);
  if (!partial) return st;
  const size_t slab = (size_t)kGpSlab * (8 * T + 1), red = KS > 1 ? (size_t)threads * 16 : 0;
  OFRR_TRY(allow_smem(k_gram_pair));
  k_gram_pair<<<dim3((unsigned)chunks, (unsigned)ny), threads, std::max(slab, red) * sizeof(double), ctx->stream>>>(
      K, b, V, ldv, W, ldw, kc, per, KS, partial);
  OFRR_LAUNCHED(ctx, "k_gram_pair");
  k_gram_pair_sum<<<(unsigned)((items * 16 + 31) / 32), 256, 0, ctx->stream>>>(b, chunks, partial, G, M);
  OFRR_LAUNCHED(ctx, "k_gram_pair_sum");
  return OFRR_SUCCESS;
}

}  // namespace ofrr
