// The FP64 advection operator (adv_impl.cuh states it) with its contractions in block
// fixed point (fixedpt.cuh).
//
// With FP64 FMAs the operator is bound by GB300's FP64 pipe (2 per clock and SM): 0.39 M
// FP64 operations per element at N=7, cubN=11, of which all but 21 per cubature node
// are interpolation, derivative and projection sums.  Those run on the integer
// multiply-add pipe here.  A thread owns a whole line of every contraction.  Between the
// three steps of an interpolation or projection the results stay integers, each with
// the exponent of its line; a line of the next step normalises them, takes the
// largest exponent and rounds (no conversion to FP64 and back).  Only the cubature
// values and their derivatives become FP64, for the pointwise terms.
//
// One CTA per element at a time, three groups of cubNq^2 threads (one per velocity
// component), persistent over elements, so that the matrices are converted once.
// Arrays, in units of 3 cubNq^3 padded words: A and B hold the cubature values and become
// the r and s derivatives in place, the t derivative comes from a column in
// registers; H holds the contravariant velocity.  Everything before and after is
// overlaid on them.
//
// E = 8192, us: N=7, cubN=11 FP64 FMAs 6060, double-float 3800, this 2966 (the integer multiply-add
// pipe active 50 % of the time at 34 % of its instruction rate, FP64 17 %; one CTA per SM, whose
// passes alternate between the two); Gauss nodes, N=7, cubN=7 792; the element's own nodes 1670,
// 1050, 334; N=2, cubN=2, 155,344 elements, own nodes 2700, 1600, 291.  Requesting the next element's metric terms into L2 and unrolling the
// pointwise passes changed nothing.
//
// An element with values that have no fixed-point form, and all elements when a matrix
// has none, are evaluated with FP64 sums (direct).  A line shares one exponent, so where a
// zero of a matrix meets a value far above the others the result would be short of bits
// (fixedpt.cuh).  Nodes that the cubature grid shares with the element's (the centre, and the
// ends of Gauss-Lobatto grids) are such places: their rows of the interpolation have one entry,
// and the derivative has zeros on its diagonal.  An element with a line to be derived or
// projected that has too small terms there takes the FP64 sums too; an interpolated value short
// of bits is one term among larger ones of the projection, as long as some row is full.
// Where the grids are the same, the interpolation is the identity, no row is full and every
// value counts: then U is taken as it is, and the advection terms are the result.
#pragma once
#include "adv_impl.cuh"
#include "fixedpt.cuh"

namespace nekb {
namespace adv_fx {

using namespace adv;

// exponents (biased) of the largest entry of a line of U and of a matrix row: three
// interpolations, the metric terms and three projections stay in the normal range
constexpr int kULo = 500, kUHi = 1546, kMLo = 983, kMHi = 1063;
// binary orders below its row's largest from which an entry counts as a zero (Gauss-Lobatto
// to Gauss interpolation has entries 10 orders below)
constexpr int kZero = 12;
// binary orders by which one value of a line of N may exceed all others before its rows are
// looked at
__host__ __device__ constexpr int far(int N) { return N >= 8 ? 6 : N >= 6 ? 7 : N >= 4 ? 8 : 10; }

template <int NQ, int CQ>
struct Shape {
  static constexpr int Np = NQ * NQ * NQ, Cp = CQ * CQ * CQ, CQ2 = CQ * CQ;
  static constexpr int THREADS = (3 * CQ2 + 31) / 32 * 32;
  static constexpr int LQ = CQ | 1, PS = CQ * LQ, AS = CQ * PS;  // padded cubature array
  static constexpr int LN = NQ | 1;
  static constexpr int RN = (NQ + 1) & ~1, RQ = (CQ + 1) & ~1;   // table rows of NQ and of CQ entries
  static constexpr int TAB = CQ * RN + NQ * RQ + CQ * RQ;        // I, I^T, D
  static constexpr int EXPS = 3 * 3 * CQ2 + 2 * CQ + NQ + 2;  // and the matrices' rows with zeros
  static constexpr int SMEM = (TAB + 9 * AS) * 8 + EXPS * 4;
  // CTAs per SM: as many as shared memory holds and registers of this number.  More CTAs
  // beat fewer spills, most on small grids (500,000 nodes, us at 128 / 80 / 64 registers: N=2,
  // cubN=4 334 / 294 / 286; N=4, cubN=7 363 / 313 / 271; N=5, cubN=8 313 / 264 / 272; N=6, cubN=10 407 / 337
  // / 337; N=7, cubN=7 116 / 104 / 100; N=5, cubN=5 99 / 88 / 94)
  static constexpr int REGS = CQ <= 4 || CQ == 8 || (CQ < 8 && CQ > NQ) ? 64 : 80;
  static constexpr int FIT = (228 * 1024) / (SMEM + 1024) < 1 ? 1 : (228 * 1024) / (SMEM + 1024);
  static constexpr int RFIT = 65536 / (REGS * THREADS) < 1 ? 1 : 65536 / (REGS * THREADS);
  static constexpr int PER_SM = FIT < RFIT ? FIT : RFIT < 32 ? RFIT : 32;
};

// one line: integers with value = V 2^x
template <int N>
struct Ln : fx::Line<N, false> {
  using F = fx::Form<N, false>;
  int x;
  // from doubles; whether they fit
  __device__ __forceinline__ bool from(const double (&v)[N], int lo, int hi)
  {
    const bool ok = this->set(v);
    x = this->e - 1075 - F::kVUp;
    return ok && (this->e == 200 || (this->e >= lo && this->e <= hi));
  }
  // the same for a line to be projected: gap is to the largest of the entries in full rows
  __device__ __forceinline__ bool from(const double (&v)[N], int lo, int hi, unsigned full)
  {
    const bool ok = from(v, lo, hi);
    unsigned top = 0, next = 0;
#pragma unroll
    for (int a = 0; a < N; ++a) {
      top = max(top, fx::hi_abs(v[a]));
      if (full >> a & 1u) next = max(next, fx::hi_abs(v[a]));
    }
    this->gap = next != 0u ? top - next : 0u;
    return ok;
  }
  // from results r[m] 2^e[m] (each standing for r + 1/2): normalised, aligned, rounded; PROJECT:
  // gap to the entries in full rows, else to the second largest
  template <bool PROJECT = false>
  __device__ __forceinline__ void from(const long long (&r)[N], const int (&e)[N], unsigned full = 0)
  {
    long long m[N];
    int ex[N], top = -100000, second = -100000;
#pragma unroll
    for (int a = 0; a < N; ++a) {
      const int lz = __clzll(r[a] ^ (r[a] >> 63));  // 1..64
      ex[a] = lz == 64 ? -100000 : e[a] - (lz - 1);
      m[a] = lz == 64 ? 0 : r[a];
      asm("shl.b64 %0, %0, %1;" : "+l"(m[a]) : "r"(lz - 1));
      if (PROJECT)
        second = full >> a & 1u ? max(second, ex[a]) : second;
      else if (N > 2)
        second = max(second, min(top, ex[a]));
      top = max(top, ex[a]);
    }
    constexpr int down = 10 - F::kVUp;  // 63-bit magnitudes to 53 + kVUp bits
#pragma unroll
    for (int a = 0; a < N; ++a) fx::words(fx::shift_nearest(m[a], min(top - ex[a], 1000) + down), this->h[a], this->l[a]);
    x = max(top, -50000) + down;
    this->gap = second == -100000 ? 0u : (unsigned)(top - second) << 20;
  }
  // whether every row of a table has terms for which the line can be held
  __device__ __forceinline__ bool fits(const int2* tab, int rows, int stride) const
  {
    return !fx::out_of_reach<N>(tab, rows, stride, *this, far(N));
  }
  // row of a table times the line; result exponent: x + row exponent + kOut
  __device__ __forceinline__ long long dot(const int2* row) const
  {
    return fx::dot_part<N, false, N, 0, 1, false>(row, *this);
  }
  static constexpr int kOut = 64 - F::kGuard;
};

// Rows (stride RS) of a matrix of ROWS x COLS entries at M[p ps + m ms], with the exponents
// of their entries (value = entry 2^ex) in ex; whether every row has a fixed-point form, in
// every thread.  rows, if given: bit p is set for a row with zeros (kZero; DIAG: beside the
// diagonal; two columns: anywhere), bit 31 if every row is the identity's.  The block synchronises here.
template <int ROWS, int COLS, int RS, bool DIAG = false>
__device__ __forceinline__ bool fill(const double* __restrict__ M, int ps, int ms, int2* t, int* ex,
                                     unsigned* rows = nullptr)
{
  static_assert(ROWS <= 31, "one row per thread of a warp");
  bool ok = true, zeros = false, unit = true;
  if (threadIdx.x < ROWS) {
    const int p = threadIdx.x;
    unsigned mx = 0, least = 0x7fffffffu;
    for (int m = 0; m < COLS; ++m) {
      const double v = M[p * ps + m * ms];
      mx = max(mx, fx::hi_abs(v));
      if (!DIAG || COLS == 2 || m != p) least = min(least, fx::hi_abs(v));
      unit = unit && v == (m == p ? 1.0 : 0.0);
    }
    const int e = (int)(mx >> 20);
    ok = e >= kMLo && e <= kMHi;
    zeros = least + ((unsigned)kZero << 20) < mx;
    ex[p] = e;
  }
  if (rows != nullptr && threadIdx.x < 32) {
    const unsigned z = __ballot_sync(0xffffffffu, zeros), u = __all_sync(0xffffffffu, unit);
    if (threadIdx.x == 0) *rows = z | (u && ROWS == COLS ? 1u << 31 : 0u);
  }
  const bool all = !__syncthreads_or(!ok);
  for (int n = threadIdx.x; n < ROWS * RS; n += blockDim.x) {
    const int p = n / RS, m = n - p * RS;
    int2 w = make_int2(0, 0);
    if (m < COLS) fx::words(fx::to_fixed<7>(M[p * ps + m * ms], ex[p]), w.x, w.y);
    t[n] = w;
  }
  __syncthreads();
  if (threadIdx.x < ROWS) ex[threadIdx.x] -= 1075 + 7;
  return all;
}

// the element with FP64 sums, matrices from global memory, arrays of AS words each
template <int NQ, int CQ>
__device__ __noinline__ void direct(const double* __restrict__ vg, const double* __restrict__ cg,
                                    const double* __restrict__ D, const double* __restrict__ It,
                                    int64_t offset, const double* __restrict__ U, double* __restrict__ NU,
                                    double* A, double* B, double* H)
{
  using S = Shape<NQ, CQ>;
  constexpr int Np = S::Np, Cp = S::Cp;
  const int tid = threadIdx.x, nt = blockDim.x;
  __syncthreads();
  for (int n = tid; n < 3 * NQ * NQ * CQ; n += nt) {  // B: X[f][c][b][i]
    const int i = n % CQ, fcb = n / CQ, f = fcb / (NQ * NQ);
    double s = 0;
#pragma unroll 1
    for (int a = 0; a < NQ; ++a) s = fma(It[a * CQ + i], U[f * offset + (fcb - f * NQ * NQ) * NQ + a], s);
    B[n] = s;
  }
  __syncthreads();
  for (int n = tid; n < 3 * NQ * CQ * CQ; n += nt) {  // H: Y[f][c][j][i]
    const int i = n % CQ, j = n / CQ % CQ, fc = n / (CQ * CQ);
    double s = 0;
#pragma unroll 1
    for (int b = 0; b < NQ; ++b) s = fma(It[b * CQ + j], B[(fc * NQ + b) * CQ + i], s);
    H[n] = s;
  }
  __syncthreads();
  for (int n = tid; n < 3 * Cp; n += nt) {  // A: cubature values [f][k][j][i]
    const int ji = n % (CQ * CQ), k = n / (CQ * CQ) % CQ, f = n / Cp;
    double s = 0;
#pragma unroll 1
    for (int c = 0; c < NQ; ++c) s = fma(It[c * CQ + k], H[(f * NQ + c) * CQ * CQ + ji], s);
    A[n] = s;
  }
  __syncthreads();
  for (int n = tid; n < 3 * Cp; n += nt) {  // B: advection terms
    const int m = n % Cp, f = n / Cp, i = m % CQ, j = m / CQ % CQ, k = m / (CQ * CQ);
    const double* c = A + f * Cp;
    double dr = 0, ds = 0, dt = 0;
#pragma unroll 1
    for (int a = 0; a < CQ; ++a) {
      dr = fma(D[i * CQ + a], c[(k * CQ + j) * CQ + a], dr);
      ds = fma(D[j * CQ + a], c[(k * CQ + a) * CQ + i], ds);
      dt = fma(D[k * CQ + a], c[(a * CQ + j) * CQ + i], dt);
    }
    const double u = A[m], v = A[Cp + m], w = A[2 * Cp + m], JW = cg[kJW * Cp + m];
    const double hr = JW * fma(w, cg[kRZ * Cp + m], fma(v, cg[kRY * Cp + m], u * cg[kRX * Cp + m]));
    const double hs = JW * fma(w, cg[kSZ * Cp + m], fma(v, cg[kSY * Cp + m], u * cg[kSX * Cp + m]));
    const double ht = JW * fma(w, cg[kTZ * Cp + m], fma(v, cg[kTY * Cp + m], u * cg[kTX * Cp + m]));
    B[n] = fma(ht, dt, fma(hs, ds, hr * dr));
  }
  __syncthreads();
  for (int n = tid; n < 3 * NQ * CQ * CQ; n += nt) {  // H: [f][c][j][i]
    const int ji = n % (CQ * CQ), c = n / (CQ * CQ) % NQ, f = n / (CQ * CQ * NQ);
    double s = 0;
#pragma unroll 1
    for (int k = 0; k < CQ; ++k) s = fma(It[c * CQ + k], B[f * Cp + k * CQ * CQ + ji], s);
    H[n] = s;
  }
  __syncthreads();
  for (int n = tid; n < 3 * NQ * NQ * CQ; n += nt) {  // A: [f][c][b][i]
    const int i = n % CQ, b = n / CQ % NQ, fc = n / (CQ * NQ);
    double s = 0;
#pragma unroll 1
    for (int j = 0; j < CQ; ++j) s = fma(It[b * CQ + j], H[(fc * CQ + j) * CQ + i], s);
    A[n] = s;
  }
  __syncthreads();
  for (int n = tid; n < 3 * Np; n += nt) {
    const int f = n / Np, m = n - f * Np, a = m % NQ;
    double s = 0;
#pragma unroll 1
    for (int i = 0; i < CQ; ++i) s = fma(It[a * CQ + i], A[(n / NQ) * CQ + i], s);
    NU[f * offset + m] = vg[kIJW * Np + m] * s;
  }
}

template <int NQ, int CQ>
__global__ void __launch_bounds__(Shape<NQ, CQ>::THREADS, Shape<NQ, CQ>::PER_SM)
k_adv_fx(int64_t E, const double* __restrict__ vgeo, const double* __restrict__ cubvgeo,
         const double* __restrict__ cubD, const double* __restrict__ cubInterpT, int64_t offset,
         const double* __restrict__ U, double* __restrict__ NU)
{
  using S = Shape<NQ, CQ>;
  constexpr int Np = S::Np, Cp = S::Cp, CQ2 = S::CQ2, LQ = S::LQ, PS = S::PS, AS = S::AS, LN = S::LN;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  int2* tI = reinterpret_cast<int2*>(sm_raw);  // rows i over a
  int2* tIt = tI + CQ * S::RN;                 // rows a over i
  int2* tD = tIt + NQ * S::RQ;                 // rows i over n
  double* A = reinterpret_cast<double*>(tD + CQ * S::RQ);
  double* B = A + 3 * AS;
  double* H = B + 3 * AS;
  int* e1 = reinterpret_cast<int*>(H + 3 * AS);  // line exponents, three sets of 3 CQ^2
  int* e2 = e1 + 3 * CQ2;
  int* e3 = e2 + 3 * CQ2;
  int* xI = e3 + 3 * CQ2;                        // row exponents of the matrices
  int* xIt = xI + CQ;
  int* xD = xIt + NQ;
  long long* Ai = reinterpret_cast<long long*>(A);
  long long* Bi = reinterpret_cast<long long*>(B);
  long long* Hi = reinterpret_cast<long long*>(H);

  const int tid = threadIdx.x;
  unsigned* rows = reinterpret_cast<unsigned*>(xD + CQ);
  bool m_ok = fill<CQ, NQ, S::RN>(cubInterpT, 1, CQ, tI, xI, rows);
  m_ok = fill<NQ, CQ, S::RQ>(cubInterpT, CQ, 1, tIt, xIt) && m_ok;
  m_ok = fill<CQ, CQ, S::RQ, true>(cubD, CQ, 1, tD, xD, rows + 1) && m_ok;
  const bool same = NQ == CQ && rows[0] >> 31;  // the cubature nodes are the element's own
  const unsigned full = ~rows[0] & ((1u << CQ) - 1u);  // full rows of the interpolation
  m_ok = m_ok && (same || full != 0u) && __popc(rows[1] & 0x7fffffffu) <= (CQ == 2 ? 0 : 1);

  // the thread's component and column (i, j); also the numbers of its lines
  const bool act = tid < 3 * CQ2;
  const int f = act ? tid / CQ2 : 0, ij = act ? tid - f * CQ2 : 0, i = ij % CQ, j = ij / CQ;
  const int col = f * AS + j * LQ + i;

  // cubature values: A and B [f][k][j][i], exponent e3[(f,j,i)] + xI[k]; whether U has a fixed-point form
  auto interpolate = [&](const double* Ue) {
    bool ok = true;
    for (int n = tid; n < 3 * Np; n += S::THREADS) {
      const int ff = n / Np, m = n - ff * Np;
      A[(n / NQ) * LN + n % NQ] = Ue[ff * offset + m];
    }
    __syncthreads();
    // interpolate in r: line (f,c,b) of A -> B[(f,c,b)][i], exponent e1[(f,c,b)] + xI[i]
    if (tid < 3 * NQ * NQ) {
      double v[NQ];
#pragma unroll
      for (int a = 0; a < NQ; ++a) v[a] = A[tid * LN + a];
      Ln<NQ> l;
      ok = l.from(v, kULo, kUHi) && ok;
      e1[tid] = l.x + l.kOut;
#pragma unroll 2
      for (int p = 0; p < CQ; ++p) Bi[tid * LQ + p] = l.dot(tI + p * S::RN);
    }
    __syncthreads();
    // in s: line (f,c,i) -> H[(f,c,j)][i], exponent e2[(f,c,i)] + xI[j]
    if (tid < 3 * NQ * CQ) {
      const int fc = tid / CQ, ii = tid - fc * CQ;
      long long r[NQ];
      int x[NQ];
#pragma unroll
      for (int b = 0; b < NQ; ++b) {
        r[b] = Bi[(fc * NQ + b) * LQ + ii];
        x[b] = e1[fc * NQ + b] + xI[ii];
      }
      Ln<NQ> l;
      l.from(r, x);
      e2[tid] = l.x + l.kOut;
#pragma unroll 2
      for (int p = 0; p < CQ; ++p) Hi[(fc * CQ + p) * LQ + ii] = l.dot(tI + p * S::RN);
    }
    __syncthreads();
    // in t: line (f,j,i) -> A and B
    if (act) {
      long long r[NQ];
      int x[NQ];
#pragma unroll
      for (int c = 0; c < NQ; ++c) {
        r[c] = Hi[((f * NQ + c) * CQ + j) * LQ + i];
        x[c] = e2[(f * NQ + c) * CQ + i] + xI[j];
      }
      Ln<NQ> l;
      l.from(r, x);
      e3[tid] = l.x + l.kOut;
#pragma unroll 2
      for (int p = 0; p < CQ; ++p) {
        const long long v = l.dot(tI + p * S::RN);
        Ai[col + p * PS] = v;
        Bi[col + p * PS] = v;
      }
    }
    return ok;
  };

  for (int64_t e = blockIdx.x; e < E; e += gridDim.x) {
    const double* Ue = U + e * Np;
    const double* cg = cubvgeo + e * (int64_t)Cp * kNvgeo;
    const double* vg = vgeo + e * (int64_t)Np * kNvgeo;
    double* NUe = NU + e * Np;
    bool ok = m_ok;
    __syncthreads();  // exponents written; the previous element's last reads
    if (same) {  // cubature values are U: A and B [f][k][j][i] as FP64
      for (int n = tid; n < 3 * Np; n += S::THREADS) {
        const int ff = n / Np, m = n - ff * Np, at = ff * AS + (m / (NQ * NQ)) * PS + (m / NQ % NQ) * LQ + m % NQ;
        A[at] = B[at] = Ue[ff * offset + m];
      }
    } else {
      ok = interpolate(Ue) && ok;
    }
    __syncthreads();
    // contravariant velocity into H, a third of the planes per group; the column for the t derivative
    Ln<CQ> t;
    if (act) {
      if (same) {
        double v[CQ];
#pragma unroll
        for (int k = 0; k < CQ; ++k) v[k] = A[col + k * PS];
        ok = t.from(v, kULo, kUHi) && ok;
      } else {
        long long r[CQ];
        int x[CQ];
#pragma unroll
        for (int k = 0; k < CQ; ++k) {
          r[k] = Ai[col + k * PS];
          x[k] = e3[tid] + xI[k];
        }
        t.from(r, x);
      }
      ok = t.fits(tD, CQ, S::RQ) && ok;
#pragma unroll 1
      for (int k = f; k < CQ; k += 3) {
        const int n = k * PS + j * LQ + i;
        const double* g = cg + k * CQ2 + ij;
        double u[3];
#pragma unroll
        for (int ff = 0; ff < 3; ++ff)
          u[ff] = same ? A[ff * AS + n] : fx::to_double(Ai[ff * AS + n], e3[ff * CQ2 + ij] + xI[k]);
        const double JW = g[kJW * Cp];
        H[n] = JW * fma(u[2], g[kRZ * Cp], fma(u[1], g[kRY * Cp], u[0] * g[kRX * Cp]));
        H[AS + n] = JW * fma(u[2], g[kSZ * Cp], fma(u[1], g[kSY * Cp], u[0] * g[kSX * Cp]));
        H[2 * AS + n] = JW * fma(u[2], g[kTZ * Cp], fma(u[1], g[kTY * Cp], u[0] * g[kTX * Cp]));
      }
    }
    __syncthreads();
    // derivatives in place: r line (j,k) = (i, j) of the thread, s line (i,k); node n of either has
    // the exponent of column (i,j) = (n, i) or (i, n)
    if (act) {
      auto derive = [&](long long* line, int stride, int from, int step, int* ex) {
        Ln<CQ> l;
        if (same) {
          double v[CQ];
#pragma unroll
          for (int n = 0; n < CQ; ++n) v[n] = __longlong_as_double(line[n * stride]);
          ok = l.from(v, kULo, kUHi) && ok;
        } else {
          long long r[CQ];
          int x[CQ];
#pragma unroll
          for (int n = 0; n < CQ; ++n) {
            r[n] = line[n * stride];
            x[n] = e3[from + n * step] + xI[j];
          }
          l.from(r, x);
        }
        ok = l.fits(tD, CQ, S::RQ) && ok;
        ex[tid] = l.x + l.kOut;
#pragma unroll 2
        for (int p = 0; p < CQ; ++p) line[p * stride] = l.dot(tD + p * S::RQ);
      };
      derive(Ai + f * AS + j * PS + i * LQ, 1, f * CQ2 + i * CQ, 1, e1);
      derive(Bi + f * AS + j * PS + i, LQ, f * CQ2 + i, CQ, e2);
    }
    __syncthreads();
    // advection term of the column, then its projection in t: A[f][c][j][i], exponent e3[(f,j,i)] + xIt[c]
    if (act) {
      const int di = xD[i], dj = xD[j], xt = t.x + t.kOut;
#pragma unroll 1
      for (int k = 0; k < CQ; ++k) {
        const int n = k * PS + j * LQ + i;
        const double dr = fx::to_double(Ai[f * AS + n], e1[f * CQ2 + k * CQ + j] + di);
        const double ds = fx::to_double(Bi[f * AS + n], e2[f * CQ2 + k * CQ + i] + dj);
        const double dt = fx::to_double(t.dot(tD + k * S::RQ), xt + xD[k]);
        A[f * AS + n] = fma(H[2 * AS + n], dt, fma(H[AS + n], ds, H[n] * dr));
      }
      if (!same) {
        double v[CQ];
#pragma unroll
        for (int k = 0; k < CQ; ++k) v[k] = A[col + k * PS];
        Ln<CQ> l;
        ok = l.from(v, fx::kExpLo, fx::kExpHi, full) && l.fits(tIt, NQ, S::RQ) && ok;
        e3[tid] = l.x + l.kOut;
#pragma unroll 2
        for (int c = 0; c < NQ; ++c) Ai[col + c * PS] = l.dot(tIt + c * S::RQ);
      }
    }
    if (__syncthreads_or(!ok)) {
      direct<NQ, CQ>(vg, cg, cubD, cubInterpT, offset, Ue, NUe, A, B, H);
      continue;
    }
    if (same) {
      if (act)
        for (int k = 0; k < CQ; ++k)
          NUe[f * offset + k * CQ2 + ij] = vg[kIJW * Np + k * CQ2 + ij] * A[col + k * PS];
      continue;
    }
    // in s: line (f,c,i) in place, exponent e1[(f,c,i)] + xIt[b]
    if (tid < 3 * NQ * CQ) {
      const int fc = tid / CQ, ii = tid - fc * CQ, ff = fc / NQ, c = fc - ff * NQ;
      long long* line = Ai + ff * AS + c * PS + ii;
      long long r[CQ];
      int x[CQ];
#pragma unroll
      for (int jj = 0; jj < CQ; ++jj) {
        r[jj] = line[jj * LQ];
        x[jj] = e3[ff * CQ2 + jj * CQ + ii] + xIt[c];
      }
      Ln<CQ> l;
      l.template from<true>(r, x, full);
      ok = l.fits(tIt, NQ, S::RQ) && ok;
      e1[tid] = l.x + l.kOut;
#pragma unroll 2
      for (int b = 0; b < NQ; ++b) line[b * LQ] = l.dot(tIt + b * S::RQ);
    }
    __syncthreads();
    // in r: line (f,c,b) in place, as FP64
    if (tid < 3 * NQ * NQ) {
      const int ff = tid / (NQ * NQ), c = tid / NQ % NQ, b = tid % NQ;
      long long* line = Ai + ff * AS + c * PS + b * LQ;
      long long r[CQ];
      int x[CQ];
#pragma unroll
      for (int ii = 0; ii < CQ; ++ii) {
        r[ii] = line[ii];
        x[ii] = e1[(ff * NQ + c) * CQ + ii] + xIt[b];
      }
      Ln<CQ> l;
      l.template from<true>(r, x, full);
      ok = l.fits(tIt, NQ, S::RQ) && ok;
#pragma unroll 2
      for (int a = 0; a < NQ; ++a)
        reinterpret_cast<double*>(line)[a] = fx::to_double(l.dot(tIt + a * S::RQ), l.x + l.kOut + xIt[a]);
    }
    if (__syncthreads_or(!ok)) {
      direct<NQ, CQ>(vg, cg, cubD, cubInterpT, offset, Ue, NUe, A, B, H);
      continue;
    }
    for (int n = tid; n < 3 * Np; n += S::THREADS) {
      const int ff = n / Np, m = n - ff * Np;
      NUe[ff * offset + m] = vg[kIJW * Np + m] * A[ff * AS + (m / (NQ * NQ)) * PS + (m / NQ % NQ) * LQ + m % NQ];
    }
  }
}

template <int NQ, int CQ>
int launch(int64_t E, const double* vgeo, const double* cubvgeo, const double* cubD,
           const double* cubInterpT, int64_t offset, const double* U, double* NU, cudaStream_t s)
{
  using S = Shape<NQ, CQ>;
  static_assert(S::SMEM <= 227 * 1024, "adv: shared memory plan exceeds 227 KB");
  static SmemOptIn smem_opt;
  NEKB_TRY(smem_opt.ensure(k_adv_fx<NQ, CQ>, S::SMEM));
  const int64_t resident = 152 * S::PER_SM;
  k_adv_fx<NQ, CQ><<<(unsigned)(E < resident ? E : resident), S::THREADS, S::SMEM, s>>>(
      E, vgeo, cubvgeo, cubD, cubInterpT, offset, U, NU);
  NEKB_CUDA(cudaGetLastError());
  return NEKB_OK;
}

}  // namespace adv_fx
}  // namespace nekb
