// FP64-accurate tensor-product contractions on the integer multiply-add pipe.
//
// GB300 retires 2 FP64 FMAs per clock per SM and 32 integer multiply-adds
// (32 x 32 -> 64 bits with a 64-bit addend), so an FP64 contraction
// sum_m D[p][m] v_m is cheaper in block fixed point.  The NQ values of a line
// share the exponent of the largest of them and become integers V_m of up to 60
// bits, seven more than an FP64 mantissa; each row of the matrix likewise.  Both
// are split into a signed high and a signed low 32-bit word, and
//   sum_m D_m V_m = 2^64 sum dh vh + 2^32 (sum dh vl + sum dl vh) + sum dl vl
// is formed in 64-bit accumulators; the last sum is at most 2^-56 NQ (even-odd form from
// NQ = 11 on: 2^-55 NQ) of max|D| max|v| and is dropped.
//
// Even-odd form (EO).  For nodes symmetric about the element centre (GLL,
// Gauss) D is centro-antisymmetric, D[p'][m'] = -D[p][m] (p' = NQ-1-p).  With
// e_m = v_m + v_m' and o_m = v_m - v_m' (m < H = NQ/2; e_H = v_H for odd NQ)
// both outputs of a pair come from two half-length sums,
//   (Dv)_p = s_p + d_p, (Dv)_p' = s_p - d_p,
//   s_p = sum_{m<H} (D[p][m] + D[p'][m])/2 o_m,
//   d_p = sum_{m<H} (D[p][m] - D[p'][m])/2 e_m (+ D[p][H] e_H, NQ odd),
// which halves the multiplications; the additions are 64-bit integer ones.  D^T
// has the same structure.
//
// No accumulator can overflow.  |dh| <= 2^28 and |dl|, |vl| <= 2^31; |vh| <= 2^28
// (EO: 2^29, and 2^28 from NQ = 11 on, where kVUp is 6).  The two middle sums share
// one accumulator where their bound, NQ 2^60 (EO: HM (2^59 + 2^60), HM = (NQ+1)/2,
// and HM 2^60 from NQ = 11 on), does not exceed 2^63; otherwise they have one
// each.  kGuard bits of the middle sums are kept below 2^64 in the result, as
// many as leave it below 2^63 for any line.
//
// The exponents are those of the line and of the row, so a line of small values
// next to a line of large ones keeps its own precision, and multiplying a line by
// a power of two multiplies the result by it bit for bit.
//
// Rounding is unbiased.  Values are truncated towards zero.  A result stands for
// r + 1/2: its low bits are cut off downwards (of the two halves of an even-odd
// result, one is cut and one rounded), so that the complement of a negative
// result is its mirror image and a rounded shift of it never meets a tie.
// (With every cut downwards, 100 iterations of a singular problem drifted along its
// null space by 5e-14.)
//
// What has no place in this form is reported to the caller, who evaluates
// that element in FP64 instead: a line whose largest exponent is outside
// [kExpLo, kExpHi] (Inf and NaN among them; a line of zeros is fine), and a
// matrix with a row or column of such a maximum, or of zeros.
//
// Precision.  A result is within (N + 2) 2^-54 of max|D| max|v| of its row and line, where
// FP64 sums are within N 2^-53 of their own terms, sum_m |D_m| |v_m|.  That makes it the
// less exact one where the terms are far below max|D| max|v|: where a zero of D (its
// diagonal) meets a value that dominates its line.  The full-length form therefore refuses
// a line with a row whose terms are below 2^-kReach max|D| max|v| (out_of_reach, looked at only
// where one value is 2^lone(N) above all others), and a matrix with an entry beside its
// diagonal (N = 2: any entry, and no line is looked at) that is more than 2^kDense below its
// row's or column's largest.  (GLL nodes, N=2..4,
// one node's lambda 1e12 times the others: 6e-7 to 6e-6 of the terms without the rule, 3.4e-16 to
// 3.8e-16 with it.)  The even-odd form has no such rule: it adds v_m and v_m' before the
// products, as the even-odd sums in FP64 that it stands for did, and they lose 2^-53 of the
// line's largest value there (steep lines, exp(-20 x), N=5..13: 1.3e-15 to 2.9e-15 of the terms, this form
// 2.8e-16 to 1.5e-15).
#pragma once

#include <cuda_runtime.h>

namespace nekb {
namespace fx {

constexpr int kExpLo = 400, kExpHi = 1646;    // biased exponents a line's maximum may have
constexpr int kDExpLo = 823, kDExpHi = 1223;  // and a row or column of the matrix
constexpr int kDense = 6, kReach = 9;

// Binary orders by which one value of a line of N may exceed all others before its rows are
// looked at (one in 2^14 lines of uniformly random values)
__host__ __device__ constexpr int lone(int N) { return N >= 5 ? 4 : (14 + N - 2) / (N - 1); }

// the largest and the second largest of magnitudes (high words) so far
__device__ __forceinline__ void top_two(unsigned v, unsigned& first, unsigned& second)
{
  second = max(second, min(first, v));
  first = max(first, v);
}

template <int NQ, bool EO>
struct Form {
  static constexpr int H = NQ / 2, HM = (NQ + 1) / 2;
  static constexpr int kDUp = 7;                       // bits a 53-bit mantissa is shifted up by
  static constexpr int kVUp = (EO && NQ >= 11) ? 6 : 7;
  static constexpr bool kOneMid = EO || NQ <= 8;
  // |result| < 2^(56 + kGuard) * (EO: 4 HM, or 2 HM from NQ = 11 on; else NQ) <= 2^63
  static constexpr int kTerms = EO ? (NQ >= 11 ? 2 * HM : 4 * HM) : NQ;
  static constexpr int guard() { return kTerms < 4 ? 5 : kTerms < 8 ? 4 : kTerms < 16 ? 3 : kTerms < 32 ? 2 : 1; }
  static constexpr int kGuard = guard();
  // a result stands for result * 2^(line exponent + row exponent + kScale)
  static constexpr int kScale = 64 - kGuard - 2 * (1023 + 52) - kDUp - kVUp;
};

__device__ __forceinline__ unsigned hi_abs(double v)
{
  return (unsigned)__double2hiint(v) & 0x7fffffffu;
}

// The block integer of v for the block's biased exponent e (>= v's own): its
// mantissa shifted up by UP and down by the difference of the exponents.
template <int UP>
__device__ __forceinline__ long long to_fixed(double v, int e)
{
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int sh = e - (int)((hi & 0x7fffffffu) >> 20);
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  m <<= UP;
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(sh));  // amounts above 63 give 0
  const long long s = (long long)(int)hi >> 63;
  return ((long long)m ^ s) - s;
}

// signed high and low words, v = hi 2^32 + lo
__device__ __forceinline__ void words(long long v, int& hi, int& lo)
{
  lo = (int)(unsigned)v;
  hi = (int)(v >> 32) + (int)((unsigned)v >> 31);
}

// A line of NQ values as block integers; EO: e_m in entry m < HM and o_m in
// entry NQ-1-m
template <int NQ, bool EO>
struct Line {
  int h[NQ], l[NQ];
  int e;         // biased exponent of the block
  unsigned gap;  // the largest value's high word less the second largest's, 0 if that is a zero (full-length form)

  // returns whether the line can be held in fixed point
  __device__ __forceinline__ bool set(const double (&v)[NQ])
  {
    using F = Form<NQ, EO>;
    unsigned mx = 0, second = 0;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      if constexpr (EO || NQ == 2)
        mx = max(mx, hi_abs(v[m]));
      else
        top_two(hi_abs(v[m]), mx, second);
    }
    e = (int)(mx >> 20);
    bool ok = e >= kExpLo && e <= kExpHi;
    gap = second != 0u ? mx - second : 0u;
    if (e == 0) {  // a line of zeros is fine, a subnormal maximum is not
      unsigned any = mx;
#pragma unroll
      for (int m = 0; m < NQ; ++m) any |= (unsigned)__double2loint(v[m]);
      ok = any == 0u;
      e = 200;  // every value is shifted out
    }
    if constexpr (EO) {
#pragma unroll
      for (int m = 0; m < F::H; ++m) {
        const long long a = to_fixed<F::kVUp>(v[m], e), b = to_fixed<F::kVUp>(v[NQ - 1 - m], e);
        words(a + b, h[m], l[m]);
        words(a - b, h[NQ - 1 - m], l[NQ - 1 - m]);
      }
      if constexpr (F::HM > F::H) words(to_fixed<F::kVUp>(v[F::H], e), h[F::H], l[F::H]);
    } else {
#pragma unroll
      for (int m = 0; m < NQ; ++m) words(to_fixed<F::kVUp>(v[m], e), h[m], l[m]);
    }
    return ok;
  }
};

// Shape of the tables: rows of (high, low) word pairs, padded to an even length so
// that they are read 16 bytes at a time.  EO: row p < HM holds the s coefficients
// of pair p (H) and then its d coefficients (HM); the middle row of odd NQ has no d.
template <int NQ, bool EO>
struct Table {
  using F = Form<NQ, EO>;
  static constexpr int rows = EO ? F::HM : NQ;
  static constexpr int part = EO ? ((F::HM + 1) & ~1) : 0;  // offset of the d coefficients
  static constexpr int stride = EO ? 2 * part : ((NQ + 1) & ~1);
  static constexpr int size = rows * stride;  // word pairs
};

// sum over N entries of a table row times line entries FIRST, FIRST + STEP, ...;
// rounded to nearest (NEAREST) or down
template <int NQ, bool EO, int N, int FIRST, int STEP, bool NEAREST>
__device__ __forceinline__ long long dot_part(const int2* row, const Line<NQ, EO>& v)
{
  using F = Form<NQ, EO>;
  constexpr long long kHalf = 1ll << (31 - F::kGuard);
  // two cuts below: one of them to nearest
  long long hh = 0, mid = NEAREST ? kHalf : 0, mid2 = kHalf;
  const int4* r4 = reinterpret_cast<const int4*>(row);
#pragma unroll
  for (int n = 0; n < N; n += 2) {
    const int4 d = r4[n / 2];
    const int a = FIRST + STEP * n;
    hh += (long long)d.x * v.h[a];
    mid += (long long)d.x * v.l[a];
    if (F::kOneMid)
      mid += (long long)d.y * v.h[a];
    else
      mid2 += (long long)d.y * v.h[a];
    if (n + 1 < N) {
      constexpr int kS = STEP;
      const int b = a + kS;
      hh += (long long)d.z * v.h[b];
      mid += (long long)d.z * v.l[b];
      if (F::kOneMid)
        mid += (long long)d.w * v.h[b];
      else
        mid2 += (long long)d.w * v.h[b];
    }
  }
  long long r = (hh << F::kGuard) + (mid >> (32 - F::kGuard));
  if (!F::kOneMid) r += mid2 >> (32 - F::kGuard);
  return r;
}

// whether some row of a table has too small terms for a line to be held (see above), looked at
// where one value is more than 2^orders above all others
template <int N>
__device__ __forceinline__ bool out_of_reach(const int2* tab, int rows, int stride, const Line<N, false>& v, int orders)
{
  if (v.gap <= (unsigned)orders << 20) return false;
  float top = 0.f;
#pragma unroll
  for (int m = 0; m < N; ++m) top = fmaxf(top, fabsf((float)v.h[m]));
  bool out = false;
#pragma unroll 1
  for (int p = 0; p < rows; ++p) {
    float sum = 0.f, big = 0.f;
#pragma unroll
    for (int m = 0; m < N; ++m) {
      const float d = fabsf((float)tab[p * stride + m].x);
      big = fmaxf(big, d);
      sum = fmaf(d, fabsf((float)v.h[m]), sum);
    }
    out = out || sum < big * top * (1.f / (1 << kReach));
  }
  return out;
}

// EO: the results of rows p and NQ-1-p (equal for the middle row); else row p
template <int NQ, bool EO>
__device__ __forceinline__ void dot_rows(const int2* tab, int p, const Line<NQ, EO>& v, long long& r,
                                         long long& r2)
{
  using F = Form<NQ, EO>;
  using T = Table<NQ, EO>;
  const int2* row = tab + p * T::stride;
  if constexpr (EO) {
    const long long s = dot_part<NQ, EO, F::H, NQ - 1, -1, false>(row, v);
    const long long d = dot_part<NQ, EO, F::HM, 0, 1, true>(row + T::part, v);
    r = s + d;
    r2 = s - d;
  } else {
    r = dot_part<NQ, EO, NQ, 0, 1, false>(row, v);
    r2 = 0;
  }
}

// r * 2^scale as a double, rounded to nearest (the caller keeps it in the normal
// range); r stands for r + 1/2, whose magnitude is r's or, if negative, its complement's
__device__ __forceinline__ double to_double(long long r, int scale)
{
  const unsigned s = (unsigned)((int)(r >> 32) >> 31);
  unsigned hi = (unsigned)(r >> 32) ^ s, lo = (unsigned)r ^ s;
  if (hi == 0u) {  // below 2^32
    if (r == 0) return 0.0;
    hi = lo;
    lo = 0u;
    scale -= 32;
    if (hi == 0u) hi = 1u;  // r = -1
  }
  const int lz = __clz((int)hi);
  hi = __funnelshift_l(lo, hi, lz);
  lo <<= lz;
  // leading bit at 63: biased exponent scale - lz + 63 + 1023, less one for the implicit bit
  unsigned long long m = ((unsigned long long)hi << 32) | lo;
  m = (m >> 11) + ((lo >> 10) & 1u);
  const unsigned ex = ((unsigned)(scale - lz + 1085) << 20) | (s & 0x80000000u);
  return __hiloint2double((int)((unsigned)(m >> 32) + ex), (int)(unsigned)m);
}

// r 2^-n to nearest (r stands for r + 1/2, the result for itself)
__device__ __forceinline__ long long shift_nearest(long long r, int n)
{
  asm("shr.s64 %0, %0, %1;" : "+l"(r) : "r"(n - 1));  // amounts above 63 leave the sign
  return (r + 1) >> 1;
}
// r 2^-n cut downwards (both stand for a half more)
__device__ __forceinline__ long long shift_down(long long r, int n)
{
  asm("shr.s64 %0, %0, %1;" : "+l"(r) : "r"(n));
  return r;
}

// Exponents of the rows and columns of a NQ x NQ row-major matrix, NQ <= 16:
// lane r holds row r's, lane 16 + c column c's; also stored to de and dte (NQ each)
// by the first warp.  ok: the matrix can be held.  eo: it is centro-antisymmetric to
// 2^-46 of its largest entry.  dense: no entry beside the diagonal is far below its row's or
// column's largest.  All are the same in every thread of the block, whose warps are whole.
template <int NQ>
__device__ __forceinline__ int matrix_exponents(const double* __restrict__ D, int* de, int* dte, bool& ok,
                                                bool& eo, bool& dense)
{
  const int lane = threadIdx.x & 31;
  const int rc = lane & 15;
  unsigned mx = 0, least = 0x7fffffffu, asym = 0;
  if (rc < NQ) {
    const int base = lane < 16 ? rc * NQ : rc, step = lane < 16 ? 1 : NQ;
#pragma unroll
    for (int m = 0; m < NQ; ++m) {
      const double v = D[base + m * step];
      mx = max(mx, hi_abs(v));
      if (NQ == 2 || m != rc) least = min(least, hi_abs(v));
      if (lane < 16) asym = max(asym, hi_abs(v + D[NQ * NQ - 1 - (base + m)]));
    }
  }
  int e = (int)(mx >> 20);
  ok = __all_sync(0xffffffffu, rc >= NQ || (e >= kDExpLo && e <= kDExpHi));
  dense = __all_sync(0xffffffffu, rc >= NQ || least + ((unsigned)kDense << 20) >= mx);
  const unsigned big = __reduce_max_sync(0xffffffffu, mx), off = __reduce_max_sync(0xffffffffu, asym);
  eo = off + (46u << 20) <= big;
  // mirror rows are equal up to rounding: one exponent for both
  const int em = __shfl_sync(0xffffffffu, e, rc < NQ ? lane - rc + NQ - 1 - rc : lane);
  if (eo) e = max(e, em);
  if (threadIdx.x < 32 && rc < NQ) (lane < 16 ? de : dte)[rc] = e;
  return e;
}

// Fills the table of D (transpose = false) or D^T; every thread of the block
// calls it with matrix_exponents' result.  The caller synchronises before it is read.
template <int NQ, bool EO>
__device__ __forceinline__ void fill_table(const double* __restrict__ D, int e, bool transpose, int2* t)
{
  using F = Form<NQ, EO>;
  using T = Table<NQ, EO>;
  const int lane = threadIdx.x & 31;
  for (int n0 = (int)threadIdx.x - lane; n0 < T::size; n0 += blockDim.x) {
    const int n = min(n0 + lane, T::size - 1);
    const int p = n / T::stride, c = n - p * T::stride;
    const int m = (EO && c >= T::part) ? c - T::part : c;  // coefficient of entry m of the line
    const bool second = EO && c >= T::part;
    const bool used = EO ? (second ? m < F::HM && p < F::H : m < F::H) : m < NQ;
    const int mm = used ? m : 0;
    const double a = transpose ? D[mm * NQ + p] : D[p * NQ + mm];
    const int ex = __shfl_sync(0xffffffffu, e, transpose ? 16 + p : p);
    long long w = 0;
    if constexpr (EO) {
      const int q = NQ - 1 - p;
      const double b = transpose ? D[mm * NQ + q] : D[q * NQ + mm];
      const long long x = to_fixed<F::kDUp>(a, ex), y = to_fixed<F::kDUp>(b, ex);
      if (p == q || (second && m == F::H))
        w = x;  // middle row: s alone; middle column: d alone
      else
        w = second ? (x - y) >> 1 : (x + y) >> 1;
    } else {
      w = to_fixed<F::kDUp>(a, ex);
    }
    if (used)
      words(w, t[n].x, t[n].y);
    else
      t[n] = make_int2(0, 0);
  }
}

}  // namespace fx
}  // namespace nekb
