// CSR operator applications: Y = op(A) X for a block of right-hand sides.
//
// Behaviour: MATLAB/+src/+csr/csrmv.m:27-78 -- the value copy of the compute precision is used
// (sparse2csr.m:48-49), products are accumulated in that precision and the result is stored in
// the output type.
//
// Layout ('N'): a CTA owns 256 consecutive rows, one per thread.  The CTA's nonzeros (a contiguous
// range of the value and index arrays) are first copied into shared memory with coalesced loads, so
// the CSR arrays are read from HBM once for all right-hand sides; each thread then walks its row in
// shared memory for every chunk of RC columns.  For stencil operators consecutive rows touch
// consecutive columns, so a warp's gathers of X are coalesced.  CTAs whose nonzeros exceed the staging
// capacity read them from global memory instead (same arithmetic, same order).
// 'T' applies the 'N' kernel to the transpose, built once per call (or once per solve, Op::prepare_csr_t)
// with a deterministic counting sort, so results never depend on the schedule (no floating-point
// atomics).
#include "ofrr_internal.cuh"

namespace ofrr {

template <class TC> struct CsrVals;
template <> struct CsrVals<double> {
  static const double* get(const ofrr_csr* A) { return A->a_double; }
  using T = double;
};
template <> struct CsrVals<float> {
  static const float* get(const ofrr_csr* A) { return A->a_single; }
  using T = float;
};

constexpr int kSpmmRows = 256;
constexpr int kSpmmCap = 2048;  // staged nonzeros per CTA (8 per row on average)

// Products of one row with RC columns of X, nonzeros in order.  U nonzeros' entries of X are loaded ahead of the
// dependent sums, so that U RC loads of a thread are in flight.  Offsets of up to 32 bits (OFF32) leave the columns'
// bases in uniform registers: one instruction per load instead of three.
template <class TX, class TC, int RC, int U, bool OFF32, bool FULL, class IDX, class VAL>
__device__ __forceinline__ void csrmm_row(int32_t p0, int32_t p1, IDX idx, VAL val, const TX* __restrict__ Xc,
                                          int64_t ldx, int nr, TC (&acc)[RC]) {
  for (int32_t p = p0; __any_sync(0xffffffffu, p < p1); p += U) {
    TX x[U][RC];
    TC a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool ok = p + u < p1;
      const int32_t col = ok ? idx(p + u) : 0;  // past the row: column 0, read and not used
      a[u] = ok ? val(p + u) : TC(0);
#pragma unroll
      for (int r = 0; r < RC; ++r) {
        const TX* base = Xc + r * ldx;
        const TX* at = OFF32 ? reinterpret_cast<const TX*>(reinterpret_cast<const char*>(base) +
                                                           (uint32_t)col * (uint32_t)sizeof(TX))
                             : base + col;
        x[u][r] = (FULL || r < nr) ? __ldg(at) : TX(0);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      // an FP64 FMA occupies its 1/64-rate pipe even where it is predicated off: leave with the whole warp
      if (u > 0 && !__any_sync(0xffffffffu, p + u < p1)) break;
      if (p + u < p1) {
#pragma unroll
        for (int r = 0; r < RC; ++r) acc[r] = fma(a[u], to_c<TC, TX>(x[u][r]), acc[r]);
      }
    }
  }
}

template <class TX, class TC, class TY, int RC, int U, int MB, bool OFF32>
__global__ void __launch_bounds__(kSpmmRows, MB) k_csrmm_n(int64_t nrows, const int32_t* __restrict__ indptr,
                                                       const int32_t* __restrict__ indices,
                                                       const TC* __restrict__ vals, int64_t nrhs,
                                                       const TX* __restrict__ X, int64_t ldx, TY* __restrict__ Y,
                                                       int64_t ldy, int nsplit, int64_t per) {
  __shared__ TC s_val[kSpmmCap];
  __shared__ int32_t s_idx[kSpmmCap];
  // CTA b: row block b / nsplit, right-hand sides [per (b % nsplit), ...) -- the CTAs of one row block are
  // adjacent, so the block's nonzeros are read from HBM once and from L2 by the others
  const int64_t r0 = (int64_t)(blockIdx.x / nsplit) * kSpmmRows;
  const int64_t cbeg = (int64_t)(blockIdx.x % nsplit) * per;
  const int64_t cend = min(nrhs, cbeg + per);
  if (r0 >= nrows) return;
  const int64_t rend = min(nrows, r0 + kSpmmRows);
  const int64_t row = r0 + threadIdx.x;
  const bool have = row < rend;
  const int32_t pbase = __ldg(indptr + r0), pend = __ldg(indptr + rend);
  const int32_t p0 = have ? __ldg(indptr + row) : 0, p1 = have ? __ldg(indptr + row + 1) : 0;
  const bool staged = (pend - pbase) <= kSpmmCap;
  if (staged) {
    for (int32_t e = threadIdx.x; e < pend - pbase; e += kSpmmRows) {
      s_val[e] = __ldg(vals + pbase + e);
      s_idx[e] = __ldg(indices + pbase + e);
    }
  }
  __syncthreads();
  for (int64_t c0 = cbeg; c0 < cend; c0 += RC) {
    TC acc[RC];
#pragma unroll
    for (int r = 0; r < RC; ++r) acc[r] = TC(0);
    const int nr = (int)min((int64_t)RC, cend - c0);
    const TX* Xc = X + c0 * ldx;
    auto si = [&](int32_t p) { return s_idx[p - pbase]; };
    auto sv = [&](int32_t p) { return s_val[p - pbase]; };
    auto gi = [&](int32_t p) { return __ldg(indices + p); };
    auto gv = [&](int32_t p) { return __ldg(vals + p); };
    if (staged && nr == RC) csrmm_row<TX, TC, RC, U, OFF32, true>(p0, p1, si, sv, Xc, ldx, nr, acc);
    else if (staged) csrmm_row<TX, TC, RC, U, OFF32, false>(p0, p1, si, sv, Xc, ldx, nr, acc);
    else csrmm_row<TX, TC, RC, 1, OFF32, false>(p0, p1, gi, gv, Xc, ldx, nr, acc);
    if (have) {
#pragma unroll
      for (int r = 0; r < RC; ++r)
        if (r < nr) Y[row + (c0 + r) * ldy] = from_c<TY, TC>(acc[r]);
    }
  }
}

// ---- deterministic CSR transpose -------------------------------------------------------------
// A counting sort by column: count (each nonzero keeps the place it got in its column), an exclusive scan of
// the counts, the row indices written in arrival order, and a last pass in which every nonzero finds its rank
// in its column (rows ascending; duplicates of one entry in the order of the input) and writes its row index
// and values there.  Only integers are exchanged through atomics, and the ranks do not depend on the arrival
// order, so the transpose is the same whatever the schedule.
__global__ void k_csrt_count(int64_t nnz, const int32_t* __restrict__ indices, int32_t* __restrict__ cnt,
                             int32_t* __restrict__ place) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x)
    place[p] = atomicAdd(&cnt[indices[p]], 1);
}

// Exclusive scan of n counts into out (n + 1 entries) over CTAs of 1024 threads x SCAN_U counts.  Pass 1: each
// CTA's sum; pass 2: each CTA adds the sums before it (a few hundred at two million counts) and scans its own.
// Measured, 262,144 counts: 409 us with one CTA walking the array in chunks, 6 us in two passes.
constexpr int SCAN_U = 4;
constexpr int SCAN_CHUNK = 1024 * SCAN_U;

__device__ __forceinline__ int32_t warp_scan_incl(int32_t v) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, v, off);
    if ((int)(threadIdx.x & 31) >= off) v += t;
  }
  return v;
}

__global__ void __launch_bounds__(1024) k_csrt_sums(int64_t n, const int32_t* __restrict__ cnt,
                                                    int32_t* __restrict__ sums) {
  __shared__ int32_t red[32];
  const int64_t base = (int64_t)blockIdx.x * SCAN_CHUNK;
  int32_t s = 0;
#pragma unroll
  for (int u = 0; u < SCAN_U; ++u) {
    const int64_t i = base + u * 1024 + threadIdx.x;
    if (i < n) s += cnt[i];
  }
  s = __reduce_add_sync(0xffffffffu, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = __reduce_add_sync(0xffffffffu, red[threadIdx.x]);
    if (threadIdx.x == 0) sums[blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(1024) k_csrt_scan(int64_t n, const int32_t* __restrict__ cnt,
                                                    const int32_t* __restrict__ sums, int32_t* __restrict__ out) {
  __shared__ int32_t red[32], s_base;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // the sums of the CTAs before this one
  int32_t before = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += 1024) before += sums[b];
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) red[wid] = before;
  __syncthreads();
  if (wid == 0) {
    const int32_t t = __reduce_add_sync(0xffffffffu, red[lane]);
    if (lane == 0) s_base = t;
  }
  __syncthreads();
  // thread t scans counts SCAN_U t .. SCAN_U t + SCAN_U - 1 of the chunk
  const int64_t i0 = (int64_t)blockIdx.x * SCAN_CHUNK + (int64_t)threadIdx.x * SCAN_U;
  int32_t v[SCAN_U], tot = 0;
#pragma unroll
  for (int u = 0; u < SCAN_U; ++u) {
    v[u] = (i0 + u < n) ? cnt[i0 + u] : 0;
    tot += v[u];
  }
  const int32_t incl = warp_scan_incl(tot);
  if (lane == 31) red[wid] = incl;
  __syncthreads();
  if (wid == 0) red[lane] = warp_scan_incl(red[lane]);
  __syncthreads();
  int32_t x = s_base + (wid ? red[wid - 1] : 0) + incl - tot;
#pragma unroll
  for (int u = 0; u < SCAN_U; ++u) {
    if (i0 + u < n) out[i0 + u] = x;
    x += v[u];
    if (i0 + u == n - 1) out[n] = x;
  }
}

// row index of every nonzero at its place (arrival order) in its column
__global__ void k_csrt_fill(int64_t nrows, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                            const int32_t* __restrict__ colptr, const int32_t* __restrict__ place,
                            int32_t* __restrict__ rows) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x) {
    for (int32_t p = indptr[r]; p < indptr[r + 1]; ++p) rows[colptr[indices[p]] + place[p]] = (int32_t)r;
  }
}

// every nonzero to its rank in its column, with the value copies present (null: absent).  A column of k nonzeros costs
// k^2 reads, all its nonzeros at once and each warp the same addresses: with one dense column in a sparse matrix the whole
// transposed product takes 0.80 ms at k = 2000, 5.9 ms at 16,000 and 453 ms at 10^6 (17.1 and 1025 ms at the first two
// with one thread's insertion sort per column), most of it the product's own serial row.
__global__ void k_csrt_place(int64_t nrows, const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                             const int32_t* __restrict__ colptr, const int32_t* __restrict__ rows,
                             int32_t* __restrict__ rowidx, const double* __restrict__ vd, double* __restrict__ td,
                             const float* __restrict__ vf, float* __restrict__ tf, const __half* __restrict__ vh,
                             __half* __restrict__ th) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t p0 = indptr[r], p1 = indptr[r + 1];
    for (int32_t p = p0; p < p1; ++p) {
      const int32_t j = indices[p], b = colptr[j], e = colptr[j + 1];
      int32_t rank = 0, same = 0;
      for (int32_t q = b; q < e; ++q) {
        const int32_t rr = rows[q];
        rank += rr < (int32_t)r;
        same += rr == (int32_t)r;
      }
      if (same > 1)  // duplicates of (r, j): in the input's order
        for (int32_t q = p0; q < p; ++q) rank += indices[q] == j;
      const int32_t o = b + rank;
      rowidx[o] = (int32_t)r;
      if (vd) td[o] = vd[p];
      if (vf) tf[o] = vf[p];
      if (vh) th[o] = vh[p];
    }
  }
}

// want: bit mask of the value copies to carry (1 FP64, 2 FP32, 4 FP16), those present in A
int csr_transpose_impl(ofrr_ctx* ctx, const ofrr_csr* A, ofrr_csr* At, int want) {
  int st = OFRR_SUCCESS;
  const int64_t m = A->nrows, n = A->ncols, nnz = A->nnz;
  *At = ofrr_csr{};
  At->nrows = n;
  At->ncols = m;
  At->nnz = nnz;
  const size_t nz = (size_t)std::max<int64_t>(nnz, 1);
  int32_t* colptr = ws_get<int32_t>(ctx, (size_t)n + 1, &st);
  int32_t* rowidx = ws_get<int32_t>(ctx, nz, &st);
  double* td = (A->a_double && (want & 1)) ? ws_get<double>(ctx, nz, &st) : nullptr;
  float* tf = (A->a_single && (want & 2)) ? ws_get<float>(ctx, nz, &st) : nullptr;
  __half* th = (A->a_half && (want & 4)) ? ws_get<__half>(ctx, nz, &st) : nullptr;
  if (st != OFRR_SUCCESS) return st;
  At->indptr = colptr;
  At->indices = rowidx;
  At->a_double = td;
  At->a_single = tf;
  At->a_half = th;
  WsScope scope(ctx);  // what follows is only needed while the transpose is built
  const unsigned chunks = (unsigned)((n + SCAN_CHUNK - 1) / SCAN_CHUNK);
  int32_t* cnt = ws_get<int32_t>(ctx, (size_t)std::max<int64_t>(n, 1), &st);
  int32_t* sums = ws_get<int32_t>(ctx, std::max(chunks, 1u), &st);
  int32_t* place = ws_get<int32_t>(ctx, nz, &st);
  int32_t* rows = ws_get<int32_t>(ctx, nz, &st);
  if (!cnt || !sums || !place || !rows) return st;
  if (n == 0 || nnz == 0) return fill_zero(ctx, colptr, sizeof(int32_t) * ((size_t)n + 1));
  OFRR_TRY(fill_zero(ctx, cnt, sizeof(int32_t) * (size_t)n));
  k_csrt_count<<<grid_for(nnz, 256, 152 * 16), 256, 0, ctx->stream>>>(nnz, A->indices, cnt, place);
  OFRR_LAUNCHED(ctx, "k_csrt_count");
  k_csrt_sums<<<chunks, 1024, 0, ctx->stream>>>(n, cnt, sums);
  OFRR_LAUNCHED(ctx, "k_csrt_sums");
  k_csrt_scan<<<chunks, 1024, 0, ctx->stream>>>(n, cnt, sums, colptr);
  OFRR_LAUNCHED(ctx, "k_csrt_scan");
  const int gr = grid_for(m, 256, 152 * 16);
  k_csrt_fill<<<gr, 256, 0, ctx->stream>>>(m, A->indptr, A->indices, colptr, place, rows);
  OFRR_LAUNCHED(ctx, "k_csrt_fill");
  k_csrt_place<<<gr, 256, 0, ctx->stream>>>(m, A->indptr, A->indices, colptr, rows, rowidx,
                                            td ? A->a_double : nullptr, td, tf ? A->a_single : nullptr, tf,
                                            th ? (const __half*)A->a_half : nullptr, th);
  OFRR_LAUNCHED(ctx, "k_csrt_place");
  return OFRR_SUCCESS;
}

static int csrmm_n(ofrr_ctx* ctx, const ofrr_csr* A, ofrr_dtype tx, ofrr_dtype tc, ofrr_dtype ty, int64_t nrhs,
                   const void* X, int64_t ldx, void* Y, int64_t ldy) {
  const int64_t blocks = (A->nrows + kSpmmRows - 1) / kSpmmRows;
  const bool off32 = A->ncols * (int64_t)dtype_size(tx) <= 0xffffffffLL;
  const int rc = !off32 ? 8 : nrhs == 1 ? 1 : nrhs <= 4 ? 4 : 8;
  // a CTA takes as many column chunks as leave the device about 16 CTAs per SM
  const int64_t nchunks = (nrhs + rc - 1) / rc;
  const int64_t split = std::min<int64_t>(nchunks, std::max<int64_t>(1, (152 * 16 + blocks - 1) / blocks));
  const int64_t per = (nchunks + split - 1) / split * rc;
  const int nsplit = (int)((nrhs + per - 1) / per);
  if (blocks * nsplit > 0x7fffffffLL) return OFRR_ERR_BLAS_INVALID_SIZE;
  const unsigned grid = (unsigned)(blocks * nsplit);
  OFRR_DISPATCH_COMPUTE(tc, TC, {
    const TC* vals = CsrVals<TC>::get(A);
    if (!vals) return OFRR_ERR_INVALID_ARGUMENT;
    // CTAs per SM the registers are kept to: FP64 is bound by its pipe and keeps more of a row in registers
    constexpr int MB = sizeof(TC) == 8 ? 6 : 8;
    OFRR_DISPATCH_STORAGE(tx, TX, OFRR_DISPATCH_STORAGE(ty, TY, {
      auto k = off32 ? (rc == 1   ? k_csrmm_n<TX, TC, TY, 1, 4, 8, true>
                        : rc == 4 ? k_csrmm_n<TX, TC, TY, 4, 1, MB, true>
                                  : k_csrmm_n<TX, TC, TY, 8, 1, MB, true>)
                     : k_csrmm_n<TX, TC, TY, 8, 1, MB, false>;
      k<<<grid, kSpmmRows, 0, ctx->stream>>>(A->nrows, A->indptr, A->indices, vals, nrhs, (const TX*)X, ldx, (TY*)Y, ldy,
                                             nsplit, per);
      OFRR_LAUNCHED(ctx, "k_csrmm_n");
    }));
  });
  return OFRR_SUCCESS;
}

int csrmm_impl(ofrr_ctx* ctx, const ofrr_csr* A, int trans, ofrr_dtype tx, ofrr_dtype tc, ofrr_dtype ty,
               int64_t nrhs, const void* X, int64_t ldx, void* Y, int64_t ldy) {
  if (nrhs <= 0) return OFRR_SUCCESS;
  const int64_t nout = trans ? A->ncols : A->nrows;
  if (nout <= 0) return OFRR_SUCCESS;
  if (!trans) return csrmm_n(ctx, A, tx, tc, ty, nrhs, X, ldx, Y, ldy);
  // transposed: the 'N' product of the transpose (same arithmetic per output entry in a fixed order)
  WsScope scope(ctx);
  ofrr_csr At;
  // only the value copy of the compute type
  OFRR_TRY(csr_transpose_impl(ctx, A, &At, tc == OFRR_F64 ? 1 : 2));
  return csrmm_n(ctx, &At, tx, tc, ty, nrhs, X, ldx, Y, ldy);
}

}  // namespace ofrr

using namespace ofrr;

extern "C" int ofrr_csrmm(ofrr_ctx* ctx, const ofrr_csr* A, int trans, ofrr_dtype tx, ofrr_dtype tcompute,
                          ofrr_dtype ty, int64_t nrhs, const void* X, int64_t ldx, void* Y, int64_t ldy) {
  if (!ctx || !A || nrhs < 0 || A->nrows < 0 || A->ncols < 0) return OFRR_ERR_INVALID_ARGUMENT;
  if (!dtype_valid(tx) || !dtype_valid(ty)) return OFRR_ERR_BLAS_UNSUPPORTED_TYPE;
  if (tcompute != OFRR_F64 && tcompute != OFRR_F32) return OFRR_ERR_BLAS_UNSUPPORTED_TYPE;
  const int64_t nin = trans ? A->nrows : A->ncols, nout = trans ? A->ncols : A->nrows;
  if (nrhs > 0 && nout > 0 && (!X || !Y || !A->indptr || (A->nnz > 0 && !A->indices) || ldx < nin || ldy < nout))
    return OFRR_ERR_INVALID_ARGUMENT;
  return csrmm_impl(ctx, A, trans, tx, tcompute, ty, nrhs, X, ldx, Y, ldy);
}
