// Hessenberg process in one cooperative launch.
//
// Same arithmetic as the per-column kernel in hessenberg.cu (MATLAB/+src/+qr/hessenberg.m:45-85, MGS order, one
// rounding to the output type per elimination), so results are bit-identical; only the schedule changes.
// Right-looking: when column t's pivot row k is known, the coefficients of the later columns are their current
// values in row k, and every element still sees its eliminations in the order j = 0, 1, ... with the same operands.
//
// The rows are split over the CTAs of a resident grid; a CTA keeps its rows of all columns in shared memory.  Per
// column there is one exchange through L2: every CTA publishes its candidate (argmax key, row and the row's values
// of the columns still to come) and reads all candidates' keys and the winner's values.
//  * Everything that travels carries the column's number in its own 64-bit word, so the words are their own
//    flags: a CTA polls the 2 G words of the keys and rows, then reads the winner's values; no counter, no fence
//    between values and keys (800 cycles), no second trip for the keys.
//  * Look-ahead: a CTA scales column t, eliminates column t + 1 alone, finds and publishes its candidate for
//    t + 1, and only then eliminates the columns after t + 1, while the candidates travel.
// What bounds it, cycles per column of 8192 x 64 in FP64 (10,300 in all): waiting for the candidates 2,000 and for the
// winner's values with the pivot's reciprocal 2,900 (one trip through L2 is about 900), the correctly rounded
// quotients and column t + 1 1,100, the argmax 700, publishing 1,650, the remaining eliminations 1,900 (every FP64
// instruction takes its sub-partition 64 cycles).
#include <cstdlib>
#include <type_traits>

#include "grid_barrier.cuh"
#include "ofrr_internal.cuh"

namespace ofrr {

constexpr int HC_T = 512;
constexpr int HC_W = HC_T / 32;
constexpr int HC_MAXG = 152;  // one CTA per SM
constexpr int HC_MAXN = 256;
constexpr int HC_REP = 4;  // copies of a candidate's values: the whole grid reads the winner's at once
constexpr size_t HC_SMEM_MAX = 200 * 1024;

template <class TC> __device__ __forceinline__ TC hc_elim(TC v, TC r, TC q) { return sub_rn(v, mul_rn(r, q)); }

struct HcPair {
  unsigned long long a, b;
};
__device__ __forceinline__ HcPair hc_ld2(const unsigned long long* p) {
  HcPair v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long hc_ld1(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void hc_st2(unsigned long long* p, unsigned long long x, unsigned long long y) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void hc_st1(unsigned long long* p, unsigned long long x) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(x) : "memory");
}
// A value in tagged words: 32 bits of it below 32 bits of tag (one word; two for FP64)
template <class TO>
struct HcVal {
  static constexpr int W = sizeof(TO) == 8 ? 2 : 1;
  __device__ static unsigned bits(float v) { return __float_as_uint(v); }
  __device__ static unsigned bits(__half v) { return __half_as_ushort(v); }
  __device__ static unsigned bits(__nv_bfloat16 v) { return __bfloat16_as_ushort(v); }
  __device__ static void put(unsigned long long* p, TO v, unsigned long long tag) {
    if constexpr (W == 2) {
      const unsigned long long x = (unsigned long long)__double_as_longlong(v);
      hc_st2(p, tag | (x >> 32), tag | (x & 0xffffffffull));
    } else {
      hc_st1(p, tag | bits(v));
    }
  }
  __device__ static bool get(const unsigned long long* p, TO* v, unsigned long long tag) {
    if constexpr (W == 2) {
      const HcPair x = hc_ld2(p);
      *v = __longlong_as_double((long long)((x.a << 32) | (x.b & 0xffffffffull)));
      return (x.a >> 32) == (tag >> 32) && (x.b >> 32) == (tag >> 32);
    } else {
      const unsigned long long x = hc_ld1(p);
      if constexpr (std::is_same<TO, float>::value) *v = __uint_as_float((unsigned)x);
      else if constexpr (std::is_same<TO, __half>::value) *v = __ushort_as_half((unsigned short)x);
      else *v = __ushort_as_bfloat16((unsigned short)x);
      return (x >> 32) == (tag >> 32);
    }
  }
};
// A wait bounded by the global timer, looked at every 64 polls
struct HcWait {
  uint64_t t0 = 0;
  unsigned polls = 0;
  __device__ bool give_up() {
    if ((++polls & 63u) != 0) return false;
    const uint64_t now = tc::globaltimer();
    if (t0 == 0) t0 = now;
    return now - t0 > 2000000000ull;
  }
};

// words: [2][G][2] keys and rows; vals: [2][HC_REP][G][n] tagged values (copies: the whole grid reads one row)
template <class TO, class TC>
__global__ void __launch_bounds__(HC_T) k_hess_coop(int64_t m, int n, int rows, TO* __restrict__ Q, int64_t ldq,
                                                    int* __restrict__ select, int* __restrict__ perm,
                                                    double* __restrict__ R, double select_tol,
                                                    unsigned long long* __restrict__ words,
                                                    unsigned long long* __restrict__ vals,
                                                    int* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char hc_raw[];
  const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int RR = rows | 1;  // odd: a row's values lie in different banks
  const int64_t row0 = (int64_t)cta * rows;
  const int nr = (int)max((int64_t)0, min((int64_t)rows, m - row0));
  TO* X = reinterpret_cast<TO*>(hc_raw);  // n columns of RR rows
  TC* s_q = reinterpret_cast<TC*>(hc_raw + (((size_t)n * RR * sizeof(TO) + 15) & ~(size_t)15));  // column t, scaled
  TC* s_pr = s_q + RR;                                                                          // the pivot row
  __shared__ ArgMaxK red[HC_W], red_in[HC_W];
  __shared__ int s_src[HC_W];
  __shared__ TC s_y;
  __shared__ bool s_pf;
  __shared__ int s_abort;

  if (tid == 0) s_abort = 0;
  for (int c = wid; c < n; c += HC_W)
    for (int r = lane; r < nr; r += 32) X[(size_t)c * RR + r] = Q[row0 + r + (int64_t)c * ldq];
  __syncthreads();

  const double tol_o = to_c<double, TO>(from_c<TO, double>(select_tol));
  // argmax over all threads' a: key and local row, the same in every warp
  auto cta_argmax = [&](ArgMaxK a) -> ArgMaxK {
    a = warp_argmaxk_all(a);
    if (lane == 0) red[wid] = a;
    __syncthreads();
    ArgMaxK b = (lane < HC_W) ? red[lane] : ArgMaxK{-1, 0x7fffffffffffffffLL};
    return warp_argmaxk_all(b);
  };
  // candidate of column t: loc's row, its values of columns t .. n - 1 read (and, for columns after t, first
  // eliminated against the column before: elim_prev) by warp 0
  auto publish = [&](int t, ArgMaxK loc, bool elim_prev) {
    const int b = t & 1;
    constexpr int W = HcVal<TO>::W;
    unsigned long long* dst = vals + ((size_t)(b * HC_REP) * G + cta) * n * W;
    const size_t copy = (size_t)G * n * W;
    if (loc.key >= 0) {
      const int lr = (int)loc.i;
      const TC q = elim_prev ? s_q[lr] : TC(0);
      for (int u = t + lane; u < n; u += 32) {
        TO v = X[(size_t)u * RR + lr];
        if (elim_prev && u > t) {
          v = from_c<TO, TC>(hc_elim(to_c<TC, TO>(v), s_pr[u], q));
          X[(size_t)u * RR + lr] = v;
        }
#pragma unroll
        for (int x = 0; x < HC_REP; ++x) HcVal<TO>::put(dst + x * copy + (size_t)u * W, v, (unsigned long long)(t + 1) << 32);
      }
    }
    if (lane == 0) {
      const unsigned long long key = (unsigned long long)loc.key;  // -1: no rows
      const unsigned long long tag = (unsigned long long)(unsigned)(t + 1) << 48;
      const unsigned row = (loc.key >= 0) ? (unsigned)(row0 + loc.i) : 0xffffffffu;
      unsigned long long* w = words + ((size_t)b * G + cta) * 2;
      hc_st2(w, tag | (key >> 16), tag | ((key & 0xffffull) << 32) | row);
    }
  };

  {
    ArgMaxK a{-1, 0x7fffffffffffffffLL};
    for (int r = tid; r < nr; r += HC_T) {
      const long long key = amax_key(X[r]);
      if (key > a.key) a = ArgMaxK{key, r};
    }
    const ArgMaxK loc = cta_argmax(a);
    if (wid == 0) publish(0, loc, false);
  }

  for (int t = 0; t < n; ++t) {
    const int b = t & 1;
    // (1) all candidates of column t; the winner is the largest key, the lowest row among equal ones
    ArgMaxK w{-1, 0x7fffffffffffffffLL};
    if (tid < G) {
      const unsigned long long* p = words + ((size_t)b * G + tid) * 2;
      const unsigned tag = (unsigned)(t + 1);
      HcPair x = hc_ld2(p);
      HcWait wait;
      while ((unsigned)(x.a >> 48) != tag || (unsigned)(x.b >> 48) != tag) {
        if (wait.give_up()) {
          atomicCAS(err, 0, 53);
          s_abort = 1;
          break;
        }
        x = hc_ld2(p);
      }
      const unsigned long long w0 = x.a, w1 = x.b;
      const unsigned long long k48 = w0 & 0xffffffffffffull;
      // the key's upper 48 bits; -1 (no rows) has them all set
      w.key = (k48 == 0xffffffffffffull) ? -1 : (long long)((k48 << 16) | ((w1 >> 32) & 0xffffull));
      w.i = (w.key >= 0) ? (long long)(unsigned)w1 : 0x7fffffffffffffffLL;
    }
    const ArgMaxK mine = w;
    w = warp_argmaxk_all(w);
    const unsigned hit = __ballot_sync(0xffffffffu, mine.key >= 0 && mine.key == w.key && mine.i == w.i);
    if (lane == 0) {
      red_in[wid] = w;
      s_src[wid] = hit ? (wid * 32 + __ffs(hit) - 1) : 0;
    }
    __syncthreads();  // also: the eliminations of the column before are complete
    if (s_abort) return;  // a peer stopped answering: the status word is set
    ArgMaxK f = (lane < HC_W) ? red_in[lane] : ArgMaxK{-1, 0x7fffffffffffffffLL};
    const ArgMaxK mf = f;
    f = warp_argmaxk_all(f);
    const unsigned fh = __ballot_sync(0xffffffffu, lane < HC_W && mf.key == f.key && mf.i == f.i);
    const int src = s_src[fh ? __ffs(fh) - 1 : 0];
    const long long k = (f.key < 0) ? 0 : f.i;
    // (2) the pivot row's values of columns t .. n - 1
    for (int u = t + tid; u < n; u += HC_T) {
      constexpr int W = HcVal<TO>::W;
      const unsigned long long* p = vals + (((size_t)(b * HC_REP + cta % HC_REP) * G + src) * n + u) * W;
      TO v;
      HcWait wait;
      // (a candidate without rows published no values: with no rows anywhere there is nothing to wait for)
      while (!HcVal<TO>::get(p, &v, (unsigned long long)(t + 1) << 32)) {
        if (wait.give_up()) {
          atomicCAS(err, 0, 54);
          s_abort = 1;
          break;
        }
      }
      s_pr[u] = to_c<TC, TO>(v);
      if (u == t) {
        const TC pc = to_c<TC, TO>(v);
        s_y = pivot_recip(pc);
        s_pf = pivot_fast(pc);
      }
    }
    __syncthreads();
    if (s_abort) return;
    const TC pc = s_pr[t], y = s_y;
    const bool pf = s_pf;
    const bool keep = !(fabs((double)pc) < tol_o);  // a NaN pivot keeps the column (hessenberg.m)
    if (cta == 0) {
      if (tid == 0) {
        select[t] = keep ? 1 : 0;
        perm[t] = keep ? (int)k : -1;
      }
      for (int u = t + tid; u < n; u += HC_T)
        R[t + (int64_t)u * n] = (u == t || keep) ? to_c<double, TC>(s_pr[u]) : 0.0;
    }
    // (3) scale (or zero) column t, eliminate column t + 1, its argmax
    const bool has_next = t + 1 < n;
    ArgMaxK a{-1, 0x7fffffffffffffffLL};
    for (int r = tid; r < nr; r += HC_T) {
      TO nv = has_next ? X[(size_t)(t + 1) * RR + r] : TO(0);
      if (keep) {
        const TC q = to_c<TC, TO>(X[(size_t)t * RR + r]);
        const TO so = from_c<TO, TC>(pivot_div(q, pc, y, pf));
        X[(size_t)t * RR + r] = so;
        const TC qs = to_c<TC, TO>(so);
        s_q[r] = qs;
        if (has_next) {
          nv = from_c<TO, TC>(hc_elim(to_c<TC, TO>(nv), s_pr[t + 1], qs));
          X[(size_t)(t + 1) * RR + r] = nv;
        }
      } else {
        X[(size_t)t * RR + r] = TO(0);
      }
      if (has_next) {
        const long long key = amax_key(nv);
        if (key > a.key) a = ArgMaxK{key, r};
      }
    }
    if (!has_next) break;
    const ArgMaxK loc = cta_argmax(a);
    if (wid == 0) publish(t + 1, loc, keep);
    // (4) the columns after t + 1; the candidate's row is warp 0's
    if (keep) {
      const int rg = (nr + 31) / 32, lc = (loc.key >= 0) ? (int)loc.i : -1;
      const int items = rg * (n - t - 2);
      // warp 0 joins last: it has published
      for (int it = (wid + HC_W - 1) % HC_W; it < items; it += HC_W) {
        const int u = t + 2 + it / rg, r = (it % rg) * 32 + lane;
        if (r < nr && r != lc) {
          TO* e = X + (size_t)u * RR + r;
          *e = from_c<TO, TC>(hc_elim(to_c<TC, TO>(*e), s_pr[u], s_q[r]));
        }
      }
    }
  }
  __syncthreads();
  for (int c = wid; c < n; c += HC_W)
    for (int r = lane; r < nr; r += 32) Q[row0 + r + (int64_t)c * ldq] = X[(size_t)c * RR + r];
}

bool hess_blocked_fits(int64_t m, int64_t n, size_t es);

template <class TO, class TC>
static int hess_coop_t(ofrr_ctx* ctx, int64_t m, int n, int rows, int G, size_t smem, TO* Q, int64_t ldq,
                       double select_tol, double* R, int* select, int* perm, bool* done) {
  WsScope scope(ctx);
  int st = OFRR_SUCCESS;
  unsigned long long* words = ws_get<unsigned long long>(ctx, (size_t)4 * G, &st);
  const size_t nvals = (size_t)2 * HC_REP * G * n * HcVal<TO>::W;
  unsigned long long* vals = ws_get<unsigned long long>(ctx, nvals, &st);
  if (!words || !vals) return st == OFRR_ERR_OUT_OF_MEMORY ? OFRR_SUCCESS : st;  // the other schedules need less
  OFRR_CUDA(cudaMemsetAsync(words, 0, sizeof(unsigned long long) * 4 * G, ctx->stream));
  OFRR_CUDA(cudaMemsetAsync(vals, 0, sizeof(unsigned long long) * nvals, ctx->stream));
  OFRR_TRY(fill_zero(ctx, R, sizeof(double) * (size_t)n * n));
  int* err = ctx->dev_flags + kFlagHessWait;
  void* args[] = {&m, &n, &rows, &Q, &ldq, &select, &perm, &R, &select_tol, &words, &vals, &err};
  const void* f = (const void*)k_hess_coop<TO, TC>;
  OFRR_TRY(allow_dynamic_smem(f));
  const cudaError_t e = cudaLaunchCooperativeKernel(f, dim3((unsigned)G), dim3(HC_T), args, smem, ctx->stream);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // the grid cannot be resident at once on this device
    (void)cudaGetLastError();
    return OFRR_SUCCESS;
  }
  OFRR_CUDA(e);
  OFRR_LAUNCHED(ctx, "k_hess_coop");
  *done = true;
  return OFRR_SUCCESS;
}

// One cooperative launch when the CTAs' rows of all columns fit their shared memory and the blocked schedules (cluster
// blocks, register panels) are not the better ones; *done = false otherwise.  Measured, whole ofrr_hessenberg calls, us,
// this / blocked:
//   FP64            n = 16     32         64         96         128
//     600 rows      176 / 158  244 / 236  383 / 416  559 / 671  762 / 1017
//     2048          188 / 160  244 / 233  401 / 429  570 / 684  787 / 1028
//     4160          199 / 172  260 / 270  403 / 500  592 / 824  811 / 1228
//     8192          202 / 196  257 / 321  433 / 619  657 / 1016 940 / 1542
//     12000         193 / 223  256 / 375  459 / 756  725 / 1270 1057 / 1882
//     25000         197 / 312  288 / 571  574 / 1240 984 / 2002 1515 / 2972
//   FP32 arithmetic, half storage (single: within 5 %)
//     8192          198 / 140  218 / 170  328 / 248  460 / 353  625 / 475
//     16384         179 / 147  215 / 211  352 / 355  526 / 513  735 / 716
//     20000         172 / 156  221 / 227  363 / 382  551 / 579  791 / 795
//     40000         171 / 176  231 / 268  425 / 469  700 / 706  1069 / 988
//     80000         179 / 220  271 / 359  574 / 670  1023 / 1036 1632 / 1441
// Hence: FP64 but for few columns (16 up to 8192 rows, 32 up to 4096); FP32 arithmetic above 32768 rows and up to 80
// columns (between 16384 and 32768 the two are within 5 %, and in a solve, where two bases are built side by side, the
// blocked one is ahead).  Heights that the blocked schedules do not hold: 30000 x 64 in FP64 697 against 1988 us per
// column, 100000 x 40 half 378 against 518.
// The FMA arithmetic of the refinement phases (`fast`) stays with the blocked schedule: it runs two bases side by side,
// and a grid over all SMs waits for the other's cluster (mixed SVD 16384 x 4000, 40 columns: 36.4 ms with this schedule,
// 35.0 ms blocked).  Heights that the blocked schedule does not hold are built in the exact arithmetic, whatever `fast`.
int hess_run_coop(ofrr_ctx* ctx, ofrr_dtype tout, ofrr_dtype tc, int64_t m, int64_t n, void* Q, int64_t ldq,
                  double select_tol, double* R, int* select, int* perm, bool fast, bool* done) {
  *done = false;
  if (n > HC_MAXN || m < 1 || m >= 0xffffffffLL || getenv("OFRR_HESS_PER_COLUMN")) return OFRR_SUCCESS;
  if (hess_blocked_fits(m, n, dtype_size(tout))) {
    const bool here = (tc == OFRR_F32) ? m > 32768 && n <= 80 : !fast && n > (m <= 4096 ? 32 : m <= 8192 ? 16 : 0);
    if (!here) return OFRR_SUCCESS;
  }
  const int G = (int)std::min<int64_t>(HC_MAXG, (m + 31) / 32);
  const int64_t rows = (m + G - 1) / G;
  const size_t es = dtype_size(tout), cs = dtype_size(tc);
  const size_t smem = (((size_t)n * (rows | 1) * es + 15) & ~(size_t)15) + ((rows | 1) + n) * cs;
  if (smem > HC_SMEM_MAX) return OFRR_SUCCESS;
  OFRR_DISPATCH_STORAGE(tout, TO, OFRR_DISPATCH_COMPUTE(tc, TC, {
    OFRR_TRY((hess_coop_t<TO, TC>(ctx, m, (int)n, (int)rows, G, smem, (TO*)Q, ldq, select_tol, R, select, perm, done)));
  }));
  return OFRR_SUCCESS;
}

}  // namespace ofrr
