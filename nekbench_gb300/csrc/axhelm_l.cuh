// FP32 axhelm (FP32, BF16 storage, trilinear geometry) by whole lines, two elements
// at a time in packed FP32 pairs.
//
// The column form of this operator (axhelm_impl.cuh: thread (i,j) reads, for every node,
// the r and the s line of the node and the matrix from shared memory) is bound by those
// reads: the load path returns 128 bytes per clock and SM, so a value read once per
// multiplication costs a clock per warp, also when all threads read the same one.  Here
// a thread owns a whole line: it loads the NQ values once, forms all NQ outputs in
// registers and replaces the line in place.  Its values are those of two elements side
// by side, for packed FMAs (fma.rn.f32x2: two per issue slot), and of all fields, so that
// a matrix coefficient read from shared memory serves two or six multiplications and the
// geometric factors of a node are read once for all fields.  Thread (i,j) also owns
// the k-column of its nodes: the t direction runs in its registers.  Geometry and
// lambda are read between the two contractions; they are requested into L2 at the start
// of the CTA, without which the node passes wait for HBM (N=9, three fields: 500 against
// 388 us in an early form).
//
// Every sum runs in the column form's order: the results are the same bits.  Even-odd
// contractions were another 10 % faster but 7-11 % further from the exact result.
//
// Measured, 16.8 M nodes, column form -> this one (us): N=7 FP32 BK 110.7 -> 96.6 (6.3 TB/s),
// lambda 135.4 -> 125.5, three fields 328 -> 240; BF16 three fields 319 -> 229;
// trilinear 143 -> 96; N=9 FP32 BK 166 -> 124, lambda 187 -> 162, three fields 528 -> 339;
// N=11 three fields 737 -> 405.  Slower: four elements per thread (registers), the fields in
// separate thread groups (the factors are then read per field), persistent CTAs that
// request the next pair (N=7 lambda 198, the CTAs' passes fall into step).
#pragma once

#include "axhelm_impl.cuh"

namespace nekb {
namespace ax {

// two floats, operated on together
struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 pack(float a, float b)
{
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack(f2 x)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x.v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

// W fields of two elements
template <int W>
struct __align__(8) fw {
  f2 x[W];
};
template <int W>
__device__ __forceinline__ fw<W> fmaw(f2 a, const fw<W>& b, const fw<W>& c)
{
  fw<W> r;
#pragma unroll
  for (int w = 0; w < W; ++w) r.x[w] = fma2(a, b.x[w], c.x[w]);
  return r;
}
template <int W>
__device__ __forceinline__ fw<W> fmaw(const fw<W>& a, const fw<W>& b, const fw<W>& c)
{
  fw<W> r;
#pragma unroll
  for (int w = 0; w < W; ++w) r.x[w] = fma2(a.x[w], b.x[w], c.x[w]);
  return r;
}
template <int W>
__device__ __forceinline__ fw<W> mulw(f2 a, const fw<W>& b)
{
  fw<W> r;
#pragma unroll
  for (int w = 0; w < W; ++w) r.x[w] = mul2(a, b.x[w]);
  return r;
}
template <int W>
__device__ __forceinline__ fw<W> mulw(const fw<W>& a, const fw<W>& b)
{
  fw<W> r;
#pragma unroll
  for (int w = 0; w < W; ++w) r.x[w] = mul2(a.x[w], b.x[w]);
  return r;
}
template <int W>
__device__ __forceinline__ fw<W> addw(const fw<W>& a, const fw<W>& b)
{
  fw<W> r;
#pragma unroll
  for (int w = 0; w < W; ++w) r.x[w] = add2(a.x[w], b.x[w]);
  return r;
}
template <int NQ, int NF, int PREC>
struct CfgL {
  static constexpr int NQ2 = NQ * NQ;
  static constexpr int NP = NQ2 * NQ;
  static constexpr int LS = NQ | 1;       // line stride
  static constexpr int PS = NQ * LS;      // plane stride
  static constexpr int AS = NQ * PS;      // one node array
  static constexpr int rounded(int n) { return (n * NQ2 + 31) / 32 * 32; }
  static constexpr int fit(int n) { return 100 * n * NQ2 >= 90 * rounded(n) && rounded(n) >= 64 ? n : fit(n + 1); }
  static constexpr int NSET = NQ >= 8 ? 1 : fit(1);  // pairs of elements per CTA
  static constexpr int THREADS = rounded(NSET);
  static constexpr int RS = (NQ + 3) & ~3;      // table row
  static constexpr int TAB = NQ * RS;
  static constexpr bool TRI = (PREC == NEKB_FP32_TRILINEAR);
  static constexpr int SMEM = 2 * TAB * 4 + NSET * 2 * AS * 8 * NF + (TRI ? NSET * 24 * 8 + 2 * NQ * 4 : 0);
  // registers per thread the launch bounds aim at, by measurement (16.8 M nodes, lambda, us:
  // N=7, one field, 80 / 96 / 168: 130 / 125 / 143; three fields 386 / 317 / 240)
  static constexpr int REGS = NF == 1 ? (NQ <= 5 ? 64 : 96) : (NQ <= 7 ? 112 : 168);
  static constexpr int MINB = 65536 / (REGS * THREADS) > 0 ? 65536 / (REGS * THREADS) : 1;
};

// output p of a line; table rows are padded to RS coefficients, a multiple of 4
template <int NQ, int W>
__device__ __forceinline__ fw<W> row_dot(const float* tab, int p, const fw<W> (&v)[NQ])
{
  constexpr int RS = (NQ + 3) & ~3;
  float c[RS];  // the row, four coefficients per load, the same for all threads
#pragma unroll
  for (int m = 0; m < RS; m += 4) {
    const float4 x = *reinterpret_cast<const float4*>(tab + p * RS + m);
    c[m] = x.x;
    c[m + 1] = x.y;
    c[m + 2] = x.z;
    c[m + 3] = x.w;
  }
  fw<W> acc = mulw<W>(pack(c[0], c[0]), v[0]);
#pragma unroll
  for (int m = 1; m < NQ; ++m) acc = fmaw<W>(pack(c[m], c[m]), v[m], acc);
  return acc;
}

template <int NQ, int W>
__device__ __forceinline__ void line_dot(fw<W>* line, int stride, const float* tab)
{
  fw<W> v[NQ];
#pragma unroll
  for (int m = 0; m < NQ; ++m) v[m] = line[m * stride];
#pragma unroll(NQ <= 4 ? NQ : NQ % 4 == 0 ? 4 : 2)
  for (int p = 0; p < NQ; ++p) line[p * stride] = row_dot<NQ, W>(tab, p, v);
}

template <int NQ, int W>
__device__ __forceinline__ void column_dot(fw<W> (&t)[NQ], const float* tab)
{
  fw<W> v[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) v[k] = t[k];
#pragma unroll
  for (int p = 0; p < NQ; ++p) t[p] = row_dot<NQ, W>(tab, p, v);
}

// trilinear_G (axhelm_impl.cuh) of two elements, operation for operation
__device__ __forceinline__ void trilinear_G2(const f2* c, float r, float s, float t, float wijk, f2 (&G)[7])
{
  const f2 r2 = pack(r, r), s2 = pack(s, s), t2 = pack(t, t), w2 = pack(wijk, wijk);
  const f2 rs = mul2(r2, s2), rt = mul2(r2, t2), st = mul2(s2, t2), neg = pack(-1.f, -1.f);
  f2 d[3][3], nd[3][3];  // d[comp][dir], and minus it
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) {
    const f2* a = c + comp * 8;
    d[comp][0] = fma2(a[7], st, fma2(a[5], t2, fma2(a[4], s2, a[1])));
    d[comp][1] = fma2(a[7], rt, fma2(a[6], t2, fma2(a[4], r2, a[2])));
    d[comp][2] = fma2(a[7], rs, fma2(a[6], s2, fma2(a[5], r2, a[3])));
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) nd[comp][dir] = mul2(neg, d[comp][dir]);
  }
  f2 cr[3][3];  // cr[dir][comp]: cofactors, J grad of the direction
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    const int p = dir == 0 ? 1 : 0, q = dir == 2 ? 1 : 2;
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      const int u = comp == 0 ? 1 : 0, v = comp == 2 ? 1 : 2;
      cr[dir][comp] = (dir + comp) & 1 ? fma2(nd[u][p], d[v][q], mul2(d[v][p], d[u][q]))
                                       : fma2(d[u][p], d[v][q], mul2(nd[v][p], d[u][q]));
    }
  }
  const f2 J = fma2(d[2][0], cr[0][2], fma2(d[0][0], cr[0][0], mul2(d[1][0], cr[0][1])));
  const float2 Js = unpack(J);
  const f2 wi = pack(__fdividef(wijk, Js.x), __fdividef(wijk, Js.y));  // J > 0 and O(h^3)
  auto dot = [&](int a, int b) {
    return mul2(wi, fma2(cr[a][2], cr[b][2], fma2(cr[a][0], cr[b][0], mul2(cr[a][1], cr[b][1]))));
  };
  G[0] = mul2(J, w2);
  G[1] = dot(0, 0);
  G[2] = dot(0, 1);
  G[3] = dot(0, 2);
  G[4] = dot(1, 1);
  G[5] = dot(1, 2);
  G[6] = dot(2, 2);
}

template <int NQ, int NF, bool BK, int PREC>
__global__ void __launch_bounds__(CfgL<NQ, NF, PREC>::THREADS, CfgL<NQ, NF, PREC>::MINB)
k_axhelm_l(const AxArgs a)
{
  using C = CfgL<NQ, NF, PREC>;
  using TG = typename Prec<PREC>::TG;
  constexpr int W = NF;
  constexpr int NQ2 = C::NQ2, NP = C::NP, LS = C::LS, PS = C::PS, AS = C::AS;
  using V = fw<W>;
  if (skipped(a)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* s_D = reinterpret_cast<float*>(smem_raw);
  float* s_Dt = s_D + C::TAB;
  V* s_all = reinterpret_cast<V*>(s_Dt + C::TAB);
  f2* s_coef = reinterpret_cast<f2*>(s_all + C::NSET * 2 * AS);  // trilinear coefficients of the pairs
  float* s_r = reinterpret_cast<float*>(s_coef + C::NSET * 24);
  float* s_w = s_r + NQ;

  const int tid = threadIdx.x;
  const int st = tid / NQ2;                  // pair of the CTA
  const int ij = tid - st * NQ2;             // node column; also the number of the thread's lines
  const int i = ij % NQ, j = ij / NQ;
  V* A = s_all + (st < C::NSET ? st : 0) * 2 * AS;
  V* B = A + AS;
  const int col = j * LS + i;                // node (i,j,0)
  auto both = [](const auto* at, int step) { return pack(to_c(at[0]), to_c(at[step])); };
  const TG* geo = static_cast<const TG*>(a.ggeo);
  const TG* lam = static_cast<const TG*>(a.lambda);

  const int64_t e0 = ((int64_t)blockIdx.x * C::NSET + st) * 2;
  const bool active = st < C::NSET && e0 < a.Nelements;
  const bool two = e0 + 1 < a.Nelements;               // else the last element stands in for its partner
  const int eq = two ? NP : 0, eg = two ? 7 * NP : 0;  // to the partner's values
  const float* qe = static_cast<const float*>(a.q) + e0 * NP + ij;
  const TG* ge = geo + e0 * 7 * NP + ij;
  const TG* le = lam + e0 * NP + ij;
  auto fields = [&](int k) {                           // q of plane k
    V r;
#pragma unroll
    for (int f = 0; f < NF; ++f) r.x[f] = both(qe + f * a.offset + k * NQ2, eq);
    return r;
  };
  V t[NQ];  // the column: q, then the t derivative, its factor, its contribution
  if (active) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) t[k] = fields(k);
    if (a.z != nullptr) {  // the new direction z + beta q
      const float b1 = (float)*a.beta;
      const f2 beta = pack(b1, b1);
      const float* ze = static_cast<const float*>(a.z) + e0 * NP + ij;
      float* qw = const_cast<float*>(qe);
#pragma unroll
      for (int k = 0; k < NQ; ++k)
#pragma unroll
        for (int f = 0; f < NF; ++f) t[k].x[f] = fma2(beta, t[k].x[f], both(ze + f * a.offset + k * NQ2, eq));
#pragma unroll
      for (int k = 0; k < NQ; ++k)
#pragma unroll
        for (int f = 0; f < NF; ++f) {  // after every load: a store would hold the next ones back
          const int64_t n = f * a.offset + k * NQ2;
          const float2 v = unpack(t[k].x[f]);
          qw[n] = v.x;
          if (two) qw[n + NP] = v.y;
        }
    }
    // geometry and lambda of the node passes, on their way to L2 meanwhile
    auto request = [&](const TG* at, int n) {
      constexpr int per = 128 / (int)sizeof(TG);
      for (int x = ij * per; x < n; x += NQ2 * per) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + x));
    };
    const int ne = two ? 2 : 1;
    if (!C::TRI) request(ge - ij + (BK ? NP : 0), ne * 7 * NP - (BK ? NP : 0));
    if (!BK) {
      request(le - ij, ne * NP);
      request(le - ij + a.offset, ne * NP);
    }
  }

  const float* Dg = static_cast<const float*>(a.D);
  for (int n = tid; n < C::TAB; n += C::THREADS) {
    const int p = n / C::RS, m = n - p * C::RS;
    s_D[n] = m < NQ ? Dg[p * NQ + m] : 0.f;
    s_Dt[n] = m < NQ ? Dg[m * NQ + p] : 0.f;
  }
  if (C::TRI) {
    for (int n = tid; n < NQ; n += C::THREADS) {
      s_r[n] = a.r1d[n];
      s_w[n] = a.w1d[n];
    }
  }
  if (C::TRI) {
    const float* coef = reinterpret_cast<const float*>(geo);
    for (int n = tid; n < C::NSET * 24; n += C::THREADS) {
      const int64_t e = ((int64_t)blockIdx.x * C::NSET + n / 24) * 2;
      if (e < a.Nelements)
        s_coef[n] = pack(coef[e * 24 + n % 24], coef[min(e + 1, a.Nelements - 1) * 24 + n % 24]);
    }
  }
  if (active) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) A[k * PS + col] = B[k * PS + col] = t[k];
  }
  auto contract = [&](const float* tab) {
    line_dot<NQ, W>(A + ij * LS, 1, tab);
    line_dot<NQ, W>(B + j * PS + i, LS, tab);
    column_dot<NQ, W>(t, tab);
  };
  // slots first..6 of the geometric factors at plane k
  auto factors = [&](int k, int first, f2 (&G)[7]) {
    if constexpr (C::TRI) {
      trilinear_G2(s_coef + st * 24, s_r[i], s_r[j], s_r[k], s_w[i] * s_w[j] * s_w[k], G);
    } else {
#pragma unroll
      for (int sl = 0; sl < 7; ++sl)
        if (sl >= first) G[sl] = both(ge + sl * NP + k * NQ2, eg);
    }
  };
  __syncthreads();
  if (active) contract(s_D);
  __syncthreads();
  if (active) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int n = k * PS + col;
      f2 G[7];
      factors(k, 1, G);
      // the order of the column form's sums
      const V qr = A[n], qs = B[n], qt = t[k];
      V gr = fmaw<W>(G[3], qt, fmaw<W>(G[1], qr, mulw<W>(G[2], qs)));
      V gs = fmaw<W>(G[5], qt, fmaw<W>(G[2], qr, mulw<W>(G[4], qs)));
      V gt = fmaw<W>(G[6], qt, fmaw<W>(G[3], qr, mulw<W>(G[5], qs)));
      if (!BK) {
        const f2 lam0 = both(le + k * NQ2, eq);
        gr = mulw<W>(lam0, gr);
        gs = mulw<W>(lam0, gs);
        gt = mulw<W>(lam0, gt);
      }
      A[n] = gr;
      B[n] = gs;
      t[k] = gt;
    }
  }
  __syncthreads();
  if (active) contract(s_Dt);
  __syncthreads();
  V qaq;  // this thread's share of q . Aq (when asked for)
#pragma unroll
  for (int f = 0; f < NF; ++f) qaq.x[f] = pack(0.f, 0.f);
  if (active) {
    float* oe = static_cast<float*>(a.Aq) + e0 * NP + ij;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int n = k * PS + col;
      V out = addw<W>(addw<W>(A[n], B[n]), t[k]);
      V q2;
      if (!BK || a.dot_partials != nullptr) q2 = fields(k);
      if (!BK) {
        f2 G[7];
        if (C::TRI)
          factors(k, 0, G);
        else
          G[0] = both(ge + k * NQ2, eg);
        out = fmaw<W>(mul2(G[0], both(le + a.offset + k * NQ2, eq)), q2, out);
      }
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const float2 o = unpack(out.x[f]);
        oe[f * a.offset + k * NQ2] = o.x;
        if (two) oe[f * a.offset + NP + k * NQ2] = o.y;
      }
      if (a.dot_partials != nullptr) qaq = fmaw<W>(q2, out, qaq);
    }
  }
  if (a.dot_partials != nullptr) {  // block sum in a fixed order
    __shared__ double s_red[32];
    double v = 0.0;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const float2 x = unpack(qaq.x[f]);
      v += (double)x.x + (two ? (double)x.y : 0.0);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) s_red[tid >> 5] = v;
    __syncthreads();
    if (tid == 0) {
      double sum = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += s_red[w];
      a.dot_partials[blockIdx.x] = sum;
      if (blockIdx.x == 0) *a.dot_count = (int)gridDim.x;
    }
  }
}

template <int NQ, int NF, bool BK, int PREC>
int run_l(const AxArgs& a, cudaStream_t s)
{
  using C = CfgL<NQ, NF, PREC>;
  static_assert(C::SMEM <= 227 * 1024, "axhelm by lines: shared memory plan exceeds 227 KB");
  auto kern = k_axhelm_l<NQ, NF, BK, PREC>;
  static SmemOptIn smem_opt;
  NEKB_TRY(smem_opt.ensure(kern, C::SMEM));
  const int64_t sets = (a.Nelements + 2 * C::NSET - 1) / (2 * C::NSET);
  if (sets == 0) return NEKB_OK;
  if (sets > INT_MAX) return fail(NEKB_ERR_INVALID, "axhelm: too many elements");
  kern<<<(unsigned)sets, C::THREADS, C::SMEM, s>>>(a);
  NEKB_CUDA(cudaGetLastError());
  return NEKB_OK;
}

// Lines from 600,000 nodes on (line_nodes); fewer leave SMs without a CTA (two elements per
// thread): N=7, lambda: 1 M nodes 11.3 -> 10.3 us, 400,000 nodes 8.2 and 8.3, 131,000 nodes 6.2
// and 8.2.  One field with lambda gains least, and about the size of L2 the column form
// is ahead at some orders (column / lines, us; FP32: N=5 10,648 elements 24.0 / 28.6, 27,900
// 59.4 / 59.4; N=7 4352 21.8 / 24.6, 8000 39.0 / 41.1, 12,167 55.4 / 55.6; N=8 4352 40.8 / 43.1,
// 8400 69.8 / 68.1; BF16 N=5 18,928 36.9 / 39.2; trilinear N=8 891 10.3 / 14.4, 2000
// equal); N=3 with lambda, three fields: 9702 elements 10.3 / 12.3, 34,848 equal.
// Below NQ = 4 (trilinear 3) a line is too short: NQ = 3 BK 127 -> 119, three fields 285
// and 287 us, NQ = 2 slower throughout.
template <int NQ, int NF, bool BK, int PREC>
int run_any(const AxArgs& a, cudaStream_t s)
{
  constexpr int64_t from = line_nodes(NQ, NF, BK, PREC);
  if constexpr (from < INT64_MAX) {
    if (a.Nelements * (NQ * NQ * NQ) >= from) return run_l<NQ, NF, BK, PREC>(a, s);
  }
  return run<NQ, NF, BK, PREC>(a, s);
}

// all variants of one order and precision; Partial forms are built for FP64 only
template <int NQ, int PREC>
int run_flags(int flags, const AxArgs& a, cudaStream_t s)
{
  const bool bk = flags & NEKB_AX_BK, n3 = flags & NEKB_AX_N3;
  if (flags & NEKB_AX_PARTIAL)
    return fail(NEKB_ERR_UNSUPPORTED, "axhelm: Partial variants are built for FP64 only");
  if (n3) return bk ? run_any<NQ, 3, true, PREC>(a, s) : run_any<NQ, 3, false, PREC>(a, s);
  return bk ? run_any<NQ, 1, true, PREC>(a, s) : run_any<NQ, 1, false, PREC>(a, s);
}

}  // namespace ax
}  // namespace nekb
