// FP64 axhelm with the contractions in block fixed point (fixedpt.cuh).
//
// GB300 executes FP64 at two FMAs per clock per SM, so an operator evaluated with
// FP64 FMAs is bound by that pipe (N=7 BK: 59 FP64 operations per node, 47 with
// even-odd contractions).  Here the six contractions run on the integer
// multiply-add pipe and FP64 carries only the geometric factors: 9 operations per
// node (BK), 14 with lambda.
//
// Element data live in shared memory as node arrays whose lines are NQ|1 words
// apart (neither row nor column lines meet bank conflicts at NQ = 8).  A thread
// owns a whole line: it converts each value once, forms all NQ outputs and
// replaces the line in place, first by the derivative (integers with one exponent
// per line), later, after the geometric factors, by the D^T contraction.  The three
// D^T contributions of a node are aligned to the largest of their exponents, added
// as integers and rounded to FP64 once.  Four barriers per element and field.
//
// An element whose values cannot be held in fixed point (Inf, NaN, extreme exponents, in
// the full-length form a line with too far a dominating value; see fixedpt.cuh) is evaluated
// with FP64 sums (direct_field), as is every element when D cannot.  The other elements of
// its CTA go on, so that an element's bits do not depend on those beside it.
#pragma once

#include "fixedpt.cuh"
#include "internal.h"

#include <climits>

namespace nekb {
namespace ax_fx {

// G: groups of NQ^2 threads per element.  G = 1: a thread takes the r, the s and
// the t line of its number in turn, the t line in registers.  G = 3: each group
// takes one direction, and a third of the planes in the node passes.
template <int NQ, int G>
struct CfgFX {
  static constexpr int NQ2 = NQ * NQ;
  static constexpr int NP = NQ2 * NQ;
  static constexpr int LS = NQ | 1;        // line stride
  static constexpr int PS = NQ * LS;       // plane stride
  static constexpr int AS = NQ * PS;       // one node array
  // Elements per CTA (G = 1, NQ < 8): the fewest that fill at least 94 % of two or
  // more warps (N=5, 16.8 M nodes: one element in 64 threads 675 us, five in 192 449)
  static constexpr int rounded(int n) { return (n * NQ2 + 31) / 32 * 32; }
  static constexpr int fit(int n) { return 100 * n * NQ2 >= 94 * rounded(n) && rounded(n) >= 64 ? n : fit(n + 1); }
  static constexpr int NEL = (G == 3 || NQ >= 8) ? 1 : fit(1);
  static constexpr int THREADS = ((NEL * G * NQ2 + 31) / 32) * 32;
  // Even-odd contractions from NQ = 6 on; below, they save nothing, and the direct
  // sums do not depend on how symmetric D is
  static constexpr bool EO = NQ >= 6;
  static constexpr int TAB = fx::Table<NQ, false>::size;  // the larger of the two forms' tables
  // two matrix tables, three node arrays per element, line exponents of three
  // directions, row exponents of the tables, a flag per element
  static constexpr int SMEM = (2 * TAB + NEL * 3 * AS) * 8 + (NEL * 3 * NQ2 + 2 * NQ + NEL) * 4;
  // registers per thread the launch bounds aim at, by measurement (16.8 M nodes, BK;
  // N=7: 80 registers 414 us, 72: 430, 96: 440; N=12: 96 registers 846 us, 128: 903)
  static constexpr int REGS = G == 3 || NQ <= 7 ? 64 : NQ == 8 ? 80 : 96;
  static constexpr int MINB = 65536 / (REGS * THREADS) > 0 ? 65536 / (REGS * THREADS) : 1;
};

// the plain FP64 sums of one field: q in A, Gr in B, Gs in C
template <int NQ, bool BK>
__device__ __noinline__ void direct_field(const AxArgs& a, int f, int64_t element, int i, int j,
                                          bool active, double* A, double* B, double* C)
{
  constexpr int NQ2 = NQ * NQ, NP = NQ2 * NQ;
  const int ij = j * NQ + i;
  const double* D = static_cast<const double*>(a.D);
  const double* ge = static_cast<const double*>(a.ggeo) + element * 7 * NP + ij;
  const double* lam = static_cast<const double*>(a.lambda);
  const double* qe = static_cast<const double*>(a.q) + f * a.offset + element * NP + ij;
  constexpr int U = NQ <= 5 ? NQ : 1;  // few elements of a mesh come here: a short chain at the low orders
  double r_q[NQ], r_Gt[NQ];
  __syncthreads();  // the arrays were in use
  if (active) {
#pragma unroll U
    for (int k = 0; k < NQ; ++k) {
      r_q[k] = qe[k * NQ2];
      A[k * NQ2 + ij] = r_q[k];
    }
  }
  __syncthreads();
  if (active) {
#pragma unroll U
    for (int k = 0; k < NQ; ++k) {
      const int n = k * NQ2 + ij;
      double qr = 0, qs = 0, qt = 0;
#pragma unroll U
      for (int m = 0; m < NQ; ++m) {
        qr += D[i * NQ + m] * A[k * NQ2 + j * NQ + m];
        qs += D[j * NQ + m] * A[k * NQ2 + m * NQ + i];
        qt += D[k * NQ + m] * r_q[m];
      }
      const double G00 = ge[1 * NP + k * NQ2], G01 = ge[2 * NP + k * NQ2];
      const double G02 = ge[3 * NP + k * NQ2], G11 = ge[4 * NP + k * NQ2];
      const double G12 = ge[5 * NP + k * NQ2], G22 = ge[6 * NP + k * NQ2];
      double gr = G00 * qr + G01 * qs + G02 * qt;
      double gs = G01 * qr + G11 * qs + G12 * qt;
      double gt = G02 * qr + G12 * qs + G22 * qt;
      if (!BK) {
        const double lam0 = lam[element * NP + n];
        gr *= lam0;
        gs *= lam0;
        gt *= lam0;
      }
      B[n] = gr;
      C[n] = gs;
      r_Gt[k] = gt;
    }
  }
  __syncthreads();
  if (active) {
    double* Aqe = static_cast<double*>(a.Aq) + f * a.offset + element * NP + ij;
#pragma unroll U
    for (int k = 0; k < NQ; ++k) {
      double ar = 0, as = 0, at = 0;
#pragma unroll U
      for (int m = 0; m < NQ; ++m) {
        ar += D[m * NQ + i] * B[k * NQ2 + j * NQ + m];
        as += D[m * NQ + j] * C[k * NQ2 + m * NQ + i];
        at += D[m * NQ + k] * r_Gt[m];
      }
      double out = ar + as + at;
      if (!BK) out += (ge[k * NQ2] * lam[element * NP + k * NQ2 + ij + a.offset]) * r_q[k];
      Aqe[k * NQ2] = out;
    }
  }
}

// replaces a line of doubles by its contraction with the matrix and leaves the
// exponent of the results, but for the row's
template <int NQ, bool EO>
__device__ __forceinline__ bool contract_line(double* line, int stride, const int2* tab, int& e)
{
  using F = fx::Form<NQ, EO>;
  fx::Line<NQ, EO> v;
  double raw[NQ];
#pragma unroll
  for (int m = 0; m < NQ; ++m) raw[m] = line[m * stride];
  bool ok = v.set(raw);
  if constexpr (!EO) ok = ok && !fx::out_of_reach<NQ>(tab, NQ, fx::Table<NQ, EO>::stride, v, fx::lone(NQ));
  e = v.e + F::kScale;
  long long* out = reinterpret_cast<long long*>(line);
#pragma unroll 2
  for (int p = 0; p < fx::Table<NQ, EO>::rows; ++p) {
    long long r, r2;
    fx::dot_rows<NQ, EO>(tab, p, v, r, r2);
    out[p * stride] = r;
    if (EO) out[(NQ - 1 - p) * stride] = r2;  // the same node and value for the middle row
  }
  return ok;
}

// the matrix in fixed point: tables of D and D^T and their row exponents
struct Tables {
  const int2 *d, *dt;
  const int *de, *dte;
};

// what a thread works on
template <int NQ, int G>
struct Place {
  using Cf = CfgFX<NQ, G>;
  double* A;           // node arrays A, B, C of the element
  int* flag;           // whether the element has no fixed-point form
  int* ex;             // exponents of r line (j,k) at k NQ + j, s line (i,k) at NQ^2 + k NQ + i, t line (i,j)
  int i, j, ij, group;  // column of the node passes, number of its lines
  bool active;

  __device__ __forceinline__ double* node() const { return A + j * Cf::LS + i; }  // node (i,j,0)
  // line number ij of a direction: (j,k), (i,k) or (i,j) = (ij % NQ, ij / NQ)
  __device__ __forceinline__ double* line(int dir) const
  {
    return A + dir * Cf::AS + (dir == 0 ? ij * Cf::LS : dir == 1 ? j * Cf::PS + i : j * Cf::LS + i);
  }
  static __device__ __forceinline__ int stride(int dir) { return dir == 0 ? 1 : dir == 1 ? Cf::LS : Cf::PS; }
};

// geometric factors of node (i,j,k) on the three derivatives; qt as its fixed-point result
template <int NQ, int G, bool BK>
__device__ __forceinline__ void geometry(const Place<NQ, G>& w, int k, const double* ge, const double* lam,
                                         int di, int dj, long long rt, int et)
{
  using Cf = CfgFX<NQ, G>;
  constexpr int NQ2 = Cf::NQ2, NP = Cf::NP, AS = Cf::AS;
  const double* g = ge + k * NQ2;
  const double G00 = g[1 * NP], G01 = g[2 * NP], G02 = g[3 * NP];
  const double G11 = g[4 * NP], G12 = g[5 * NP], G22 = g[6 * NP];
  double lam0 = 1.0;
  if (!BK) lam0 = lam[k * NQ2];
  double* n = w.node() + k * Cf::PS;
  const double qt = fx::to_double(rt, et);
  const double qr = fx::to_double(__double_as_longlong(n[0]), w.ex[k * NQ + w.j] + di);
  const double qs = fx::to_double(__double_as_longlong(n[AS]), w.ex[NQ2 + k * NQ + w.i] + dj);
  double gr = G00 * qr + G01 * qs + G02 * qt;
  double gs = G01 * qr + G11 * qs + G12 * qt;
  double gt = G02 * qr + G12 * qs + G22 * qt;
  if (!BK) {
    gr *= lam0;
    gs *= lam0;
    gt *= lam0;
  }
  n[0] = gr;
  n[AS] = gs;
  n[2 * AS] = gt;
}

// output of node (i,j,k); the t contribution as its fixed-point result
template <int NQ, int G, bool BK>
__device__ __forceinline__ void output(const Place<NQ, G>& w, int k, const double* ge, const double* lam1,
                                       const double* qe, double* Aqe, int di, int dj, long long rt, int st)
{
  using Cf = CfgFX<NQ, G>;
  constexpr int NQ2 = Cf::NQ2, AS = Cf::AS;
  const double* n = w.node() + k * Cf::PS;
  double wl1 = 0.0, qk = 0.0;
  if (!BK) {
    wl1 = ge[k * NQ2] * lam1[k * NQ2];
    qk = qe[k * NQ2];
  }
  // aligned to two bits above the largest exponent: the sum stays below 2^63
  const int sr = w.ex[k * NQ + w.j] + di, ss = w.ex[NQ2 + k * NQ + w.i] + dj;
  const int sm = max(st, max(sr, ss)) + 2;
  const long long sum = fx::shift_down(rt, sm - st) +
                        fx::shift_nearest(__double_as_longlong(n[0]), sm - sr) +
                        fx::shift_nearest(__double_as_longlong(n[AS]), sm - ss);
  double out = fx::to_double(sum, sm);
  if (!BK) out += wl1 * qk;
  Aqe[k * NQ2] = out;
}

// elements that have to be evaluated in FP64: any of the CTA's (the same in every thread),
// the thread's own
struct Refused {
  bool any, own;
};

// one field of the CTA's elements
template <int NQ, int G, bool BK, bool EO>
__device__ __forceinline__ Refused fixed_field(const AxArgs& a, int f, int64_t element, const Place<NQ, G>& w,
                                            const Tables& tab)
{
  using Cf = CfgFX<NQ, G>;
  using F = fx::Form<NQ, EO>;
  constexpr int NQ2 = Cf::NQ2, NP = Cf::NP, PS = Cf::PS, AS = Cf::AS;
  constexpr int rows = fx::Table<NQ, EO>::rows;
  const double* ge = static_cast<const double*>(a.ggeo) + element * 7 * NP + w.ij;
  const double* lam = static_cast<const double*>(a.lambda) + element * NP + w.ij;
  const double* qe = static_cast<const double*>(a.q) + f * a.offset + element * NP + w.ij;
  double* Aqe = static_cast<double*>(a.Aq) + f * a.offset + element * NP + w.ij;
  double* node = w.node();
  bool ok = true, on = w.active;
  Refused refused{false, false};
  fx::Line<NQ, EO> t;  // G = 1: the thread's t line

  // barrier, after which the elements with a line that is not ok drop out
  auto agree = [&]() {
    if (__syncthreads_or(!ok)) {
      refused = {true, true};
      if constexpr (Cf::NEL > 1) {
        if (!ok) *w.flag = 1;
        __syncthreads();
        refused.own = *w.flag != 0;
      }
      on = on && !refused.own;
    }
  };

  auto set_t = [&](const double (&v)[NQ], const int2* tb) {
    bool fine = t.set(v);
    if constexpr (!EO) fine = fine && !fx::out_of_reach<NQ>(tb, NQ, fx::Table<NQ, EO>::stride, t, fx::lone(NQ));
    return fine;
  };
  // the contractions of the lines in shared memory (all of the element's, G = 3)
  auto lines = [&](const int2* tb) {
    if constexpr (G == 1) {
      ok = contract_line<NQ, EO>(w.line(0), w.stride(0), tb, w.ex[w.ij]) && ok;
      ok = contract_line<NQ, EO>(w.line(1), w.stride(1), tb, w.ex[NQ2 + w.ij]) && ok;
    } else {
      ok = contract_line<NQ, EO>(w.line(w.group), w.stride(w.group), tb, w.ex[w.group * NQ2 + w.ij]);
    }
  };
  // every node of the thread with its t result (and that result's exponent, but for the row's)
  auto nodes = [&](const int2* tb, auto&& visit) {
    if constexpr (G == 1) {
      const int te = t.e + F::kScale;
#pragma unroll 1
      for (int p = 0; p < rows; ++p) {
        long long r, r2;
        fx::dot_rows<NQ, EO>(tb, p, t, r, r2);
        visit(p, r, te);
        if (EO && (!(NQ & 1) || p < NQ / 2)) visit(NQ - 1 - p, r2, te);
      }
    } else {
      const int te = w.ex[2 * NQ2 + w.ij];
#pragma unroll
      for (int k0 = 0; k0 < NQ; k0 += G) {
        const int k = k0 + w.group;
        if (k < NQ) visit(k, __double_as_longlong(node[k * PS + 2 * AS]), te);
      }
    }
  };

  if (on) {
    if constexpr (G == 1) {
      double r_q[NQ];
#pragma unroll
      for (int k = 0; k < NQ; ++k) r_q[k] = qe[k * NQ2];
#pragma unroll
      for (int k = 0; k < NQ; ++k) {
        node[k * PS] = r_q[k];
        node[k * PS + AS] = r_q[k];
      }
      ok = set_t(r_q, tab.d);
    } else {
#pragma unroll
      for (int k0 = 0; k0 < NQ; k0 += G) {
        const int k = k0 + w.group;
        if (k < NQ) {
          const double v = qe[k * NQ2];
          node[k * PS] = v;
          node[k * PS + AS] = v;
          node[k * PS + 2 * AS] = v;
        }
      }
    }
  }
  __syncthreads();
  if (on) lines(tab.d);
  agree();
  if (Cf::NEL == 1 && refused.any) return refused;
  if (on) {
    const int di = tab.de[w.i], dj = tab.de[w.j];
    nodes(tab.d, [&](int k, long long rt, int te) {
      geometry<NQ, G, BK>(w, k, ge, lam, di, dj, rt, te + tab.de[k]);
    });
  }
  __syncthreads();
  if (on) {
    lines(tab.dt);
    if constexpr (G == 1) {
      double gt[NQ];
#pragma unroll
      for (int k = 0; k < NQ; ++k) gt[k] = node[k * PS + 2 * AS];
      ok = set_t(gt, tab.dt) && ok;
    }
  }
  agree();
  if (Cf::NEL == 1 && refused.any) return refused;
  if (on) {
    const int di = tab.dte[w.i], dj = tab.dte[w.j];
    nodes(tab.dt, [&](int k, long long rt, int te) {
      output<NQ, G, BK>(w, k, ge, lam + a.offset, qe, Aqe, di, dj, rt, te + tab.dte[k]);
    });
  }
  return refused;
}

template <int NQ, int NF, bool BK, bool PARTIAL, int G>
__global__ void __launch_bounds__(CfgFX<NQ, G>::THREADS, CfgFX<NQ, G>::MINB)
k_axhelm_fx(const AxArgs a, int64_t groups)
{
  using Cf = CfgFX<NQ, G>;
  constexpr int NQ2 = Cf::NQ2, NEL = Cf::NEL;
  if (a.skip != nullptr && *a.skip != 0) return;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  int2* s_D = reinterpret_cast<int2*>(smem_raw);
  int2* s_Dt = s_D + Cf::TAB;
  double* s_all = reinterpret_cast<double*>(s_Dt + Cf::TAB);
  int* s_exp = reinterpret_cast<int*>(s_all + NEL * 3 * Cf::AS);
  int* s_de = s_exp + NEL * 3 * NQ2;  // row exponents of D and of D^T
  int* s_dte = s_de + NQ;
  int* s_flag = s_dte + NQ;

  const int tid = threadIdx.x;
  if (tid < NEL) s_flag[tid] = 0;
  const double* D = static_cast<const double*>(a.D);
  bool d_ok, sym, dense;
  const int de = fx::matrix_exponents<NQ>(D, s_de, s_dte, d_ok, sym, dense);
  d_ok = d_ok && ((Cf::EO && sym) || dense);
  if (Cf::EO && sym) {
    fx::fill_table<NQ, Cf::EO>(D, de, false, s_D);
    fx::fill_table<NQ, Cf::EO>(D, de, true, s_Dt);
  } else {
    fx::fill_table<NQ, false>(D, de, false, s_D);
    fx::fill_table<NQ, false>(D, de, true, s_Dt);
  }
  const Tables tab{s_D, s_Dt, s_de, s_dte};

  const int el = tid / (G * NQ2);
  const int elc = el < NEL ? el : 0;  // keep shared pointers in range for idle threads
  Place<NQ, G> w;
  w.ij = tid - el * (G * NQ2);
  w.group = w.ij / NQ2;
  w.ij -= w.group * NQ2;
  w.i = w.ij % NQ;
  w.j = w.ij / NQ;
  w.A = s_all + elc * 3 * Cf::AS;
  w.ex = s_exp + elc * 3 * NQ2;
  w.flag = s_flag + elc;

  for (int64_t g = blockIdx.x; g < groups; g += gridDim.x) {
    const int64_t eidx = g * NEL + el;
    w.active = (el < NEL) && (eidx < a.Nelements);
    int64_t element = eidx;
    if (PARTIAL && w.active) element = a.elementList[eidx];
#pragma unroll 1
    for (int f = 0; f < NF; ++f) {
      __syncthreads();  // the tables are written; the previous element's or field's last reads
      Refused refused{true, true};
      if (d_ok) {
        if (Cf::EO && sym)
          refused = fixed_field<NQ, G, BK, Cf::EO>(a, f, element, w, tab);
        else
          refused = fixed_field<NQ, G, BK, false>(a, f, element, w, tab);
      }
      if (refused.any) {
        direct_field<NQ, BK>(a, f, element, w.i, w.j, w.active && refused.own && w.group == 0, w.A,
                             w.A + Cf::AS, w.A + 2 * Cf::AS);
        if (tid < NEL) s_flag[tid] = 0;  // read before direct_field's barriers
      }
    }
  }
}

template <int NQ, int NF, bool BK, bool PARTIAL, int G>
int launch(const AxArgs& a, cudaStream_t s)
{
  using Cf = CfgFX<NQ, G>;
  static_assert(Cf::SMEM <= 227 * 1024, "fixed-point axhelm: shared memory plan exceeds 227 KB");
  auto kern = k_axhelm_fx<NQ, NF, BK, PARTIAL, G>;
  static SmemOptIn smem_opt;
  NEKB_TRY(smem_opt.ensure(kern, Cf::SMEM));
  const int64_t groups = (a.Nelements + Cf::NEL - 1) / Cf::NEL;
  if (groups == 0) return NEKB_OK;
  if (groups > INT_MAX) return fail(NEKB_ERR_INVALID, "axhelm: too many elements");
  const int64_t grid = groups < 152 * 64 ? groups : 152 * 64;
  kern<<<(unsigned)grid, Cf::THREADS, Cf::SMEM, s>>>(a, groups);
  NEKB_CUDA(cudaGetLastError());
  return NEKB_OK;
}

// Three groups of threads per element when there are few elements: they shorten the
// chain of one element, where one group per element keeps more elements in flight.  N=7
// BK: 78 elements 10.3 against 16.4 us, 512 elements 17.0 against 18.5, 1024 elements 26.7
// against 24.7; N=10: 197 elements 22.6 against 29.1, 394 elements 34.9 against 35.6.  Below
// NQ = 5 an element has too few lines for it.
template <int NQ, int NF, bool BK, bool PARTIAL>
int run(const AxArgs& a, cudaStream_t s)
{
  if constexpr (NQ >= 5) {
    if (a.Nelements * (NQ * NQ) <= 152 * 320) return launch<NQ, NF, BK, PARTIAL, 3>(a, s);
  }
  return launch<NQ, NF, BK, PARTIAL, 1>(a, s);
}

// all FP64 variants of one order (Partial forms included)
template <int NQ>
int run_flags(int flags, const AxArgs& a, cudaStream_t s)
{
  const bool bk = flags & NEKB_AX_BK, n3 = flags & NEKB_AX_N3, part = flags & NEKB_AX_PARTIAL;
  if (part) {
    if (n3) return bk ? run<NQ, 3, true, true>(a, s) : run<NQ, 3, false, true>(a, s);
    return bk ? run<NQ, 1, true, true>(a, s) : run<NQ, 1, false, true>(a, s);
  }
  if (n3) return bk ? run<NQ, 3, true, false>(a, s) : run<NQ, 3, false, false>(a, s);
  return bk ? run<NQ, 1, true, false>(a, s) : run<NQ, 1, false, false>(a, s);
}

}  // namespace ax_fx
}  // namespace nekb
