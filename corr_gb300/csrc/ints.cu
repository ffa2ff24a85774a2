// Gaussian integrals of the RI path on the GPU: the 2-index metric
// J[P][Q] = (P|Q) and the 3-index integrals (P|mu nu), the inputs the
// reference computes with libint inside calculate_ri (src/POSTHF/ri.cc:25-47,
// 70-100) or the psi4 plugin writes (syshfwplug/plugin.cc:478-503).
//
// Method: McMurchie-Davidson (Helgaker, Joergensen, Olsen, "Molecular
// Electronic-Structure Theory", ch. 9): Hermite expansion coefficients E of
// each orbital Gaussian product, Hermite Coulomb integrals R_tuv from the Boys
// function F_n by the vertical recursion, then real solid harmonics
// (m = -l..l) normalised to one.  Cartesian components are ordered lx = l..0,
// ly = l-lx..0.  FP64 throughout.
//
// The auxiliary side is one Gaussian, for which a solid harmonic is a pure
// derivative, S_lm(r - A) e^(-g |r-A|^2) = (2g)^-l S_lm(d/dA) e^(-g |r-A|^2)
// (S_lm is harmonic: no lower orders appear; same text, ch. 9), so only the
// Hermite orders t + u + v = l enter and there is no expansion on that side.
//
// Work decomposition: one kernel per angular-momentum class (aux l, and the
// two orbital l's), templated so every table has a compile-time size; one
// thread per (aux shell, orbital shell pair c >= d), both triangles of
// (P|mu nu) written.  The products E_t E_u E_v of an orbital primitive pair are
// the same for every auxiliary shell: a first launch tabulates them.  (P|Q) runs
// through the same kernel with an s function of exponent 0 as the partner of Q.
//
// Bound by the FP64 pipe, two FMAs per clock per SM: what counts is FP64
// instructions per primitive triple, and loads, index arithmetic and local
// memory run beside them.  20-water cluster: 12.3 ms a call, 2 ms of it the host's
// screening (25.5 ms with expansions of the auxiliary Gaussians and per-thread E
// tables).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "abi_internal.h"
#include "common.cuh"
#include "fp64_approx.cuh"

namespace corr {

namespace {

constexpr int kLmax = 3;

struct ShellD {
  double x, y, z;
  int l, nprim, poff, bf;  // bf: index of the shell's first function
};

// Spherical <- Cartesian, every row scaled so that all functions of a shell have
// the norm of its m = 0 (rows of s and p hold a single 1).
__constant__ double c_sph[kLmax + 1][2 * kLmax + 1][10];
__constant__ int c_cexp[kLmax + 1][10][3];                   // Cartesian exponents
constexpr int kTmax = 2 * kLmax + 2;                         // Hermite orders < kTmax
__constant__ int c_tuv[kTmax][kTmax][kTmax];                  // tuv_index table

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }

// Cartesian exponent of component k of shell l along dim (0 x, 1 y, 2 z)
__host__ __device__ constexpr int cexp(int l, int k, int dim) {
  int idx = 0;
  for (int x = l; x >= 0; --x)
    for (int y = l - x; y >= 0; --y) {
      if (idx == k) return dim == 0 ? x : (dim == 1 ? y : l - x - y);
      ++idx;
    }
  return 0;
}

// The Cartesian components that S_lm (m = -l .. l as 0 .. 2l) contains, one bit
// each, so that the transforms spend nothing on zeros (a table rather than the
// rule: every use is unrolled, and the rule's loops took minutes to compile).
__host__ __device__ constexpr unsigned sph_mask(int l, int m) {
  constexpr unsigned d[5] = {0x002, 0x010, 0x029, 0x004, 0x009};
  constexpr unsigned f[7] = {0x042, 0x010, 0x142, 0x284, 0x029, 0x084, 0x009};
  return l == 2 ? d[m] : (l == 3 ? f[m] : 0u);
}

// (t, u, v) with t + u + v <= L: index in a compact table of binom(L+3, 3) entries
__host__ __device__ constexpr int tuv_count(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ constexpr int tuv_index(int t, int u, int v) {
  // orders m = t + u + v in increasing order, within an order the (u, v) pairs
  return tuv_count(t + u + v - 1 >= 0 ? t + u + v - 1 : -1) + ((u + v) * (u + v + 1)) / 2 + v;
}

// Boys function F_n(T), n <= NMAX: for T < kBoysTmax an 8-term Taylor
// expansion of F_NMAX about the nearest point of a tabulated grid (spacing
// 1/16, |dT| <= 1/32, truncation below 2^-55 relative) and downward
// recursion F_n = (2T F_{n+1} + e^-T) / (2n + 1), with e^-T from the grid
// point's and an 8-term exponential series of the offset (below 2^-55); above,
// the asymptotic F_0 = sqrt(pi/T) / 2 and upward recursion without the e^-T term:
// what they leave out, e^-T / (2T) (1 + (2n+1) / (2T) + ...), is below 7e-20 (at
// T = 40, 4e-19 of F_0 and 7e-11 of F_7, which is 9e-10 there).  The tables hold
// the Taylor coefficients F_{n+k} / k!, one FMA per term.
constexpr int kBoysOrders = 16;                // tabulated n = 0..15
constexpr int kBoysTerms = 8;
constexpr int kBoysMax = kBoysOrders - kBoysTerms;  // highest NMAX
constexpr int kBoysPerUnit = 16;               // grid points per unit of T
constexpr double kBoysTmax = 40.0;
constexpr int kBoysPoints = (int)kBoysTmax * kBoysPerUnit + 1;
__device__ double d_boys[kBoysMax + 1][kBoysPoints][kBoysTerms];
__device__ double d_boys_exp[kBoysPoints];     // e^-T_i

template <int NMAX>
__device__ __forceinline__ void boys(double T, double* F) {
  static_assert(NMAX <= kBoysMax, "Boys table orders");
  // (compared as integers: T >= 0, and an FP64 compare is an FP64 instruction;
  // unsigned, so that a NaN of either sign stays out of the table)
  if ((unsigned long long)__double_as_longlong(T) <
      (unsigned long long)__double_as_longlong(kBoysTmax)) {
    // T * 16 to the nearest integer: 2^52 + 2^51 leaves it in the low word
    const double y = fma(T, (double)kBoysPerUnit, 6755399441055744.0);
    const int i = __double2loint(y);
    const double x = fma(y - 6755399441055744.0, 1.0 / kBoysPerUnit, -T);  // -dT
    const double* f = d_boys[NMAX][i];
    double s = f[kBoysTerms - 1];
#pragma unroll
    for (int k = kBoysTerms - 2; k >= 0; --k) s = fma(s, x, f[k]);
    F[NMAX] = s;
    if (NMAX > 0) {
      double e = 1.0 / 5040.0;
      e = fma(e, x, 1.0 / 720.0);
      e = fma(e, x, 1.0 / 120.0);
      e = fma(e, x, 1.0 / 24.0);
      e = fma(e, x, 1.0 / 6.0);
      e = fma(e, x, 0.5);
      e = fma(e, x, 1.0);
      e = fma(e, x, 1.0);
      const double et = e * d_boys_exp[i], t2 = 2.0 * T;
#pragma unroll
      for (int n = NMAX - 1; n >= 0; --n) {
        F[n] = fma(t2, F[n + 1], et);
        if (n > 0) F[n] *= 1.0 / (2 * n + 1);
      }
    }
    return;
  }
  const double rt = 1.0 / T;
  F[0] = 0.886226925452758 * sqrt(rt);  // sqrt(pi) / 2
#pragma unroll
  for (int n = 0; n < NMAX; ++n) F[n + 1] = F[n] * ((n + 0.5) * rt);
}

// pref R^0_{tuv}(alpha, X, Y, Z), t + u + v <= L, into buf[0][tuv_index].
// Ping-pong over the auxiliary order n between buf[0] and buf[1]: level n holds
// the orders <= L - n.  Each entry steps down the index that is one, where
// there is one (a single product), else the first that is not zero.
template <int L>
__device__ __forceinline__ void hermite_r(double pref, double alpha, double X, double Y, double Z,
                                          double (&buf)[2][tuv_count(L)]) {
  double F[L + 1];
  boys<L>(alpha * fma(X, X, fma(Y, Y, Z * Z)), F);
  double fn[L + 1];
  const double m2a = -2.0 * alpha;
#pragma unroll
  for (int n = 0; n <= L; ++n) {
    fn[n] = pref * F[n];
    if (n < L) pref *= m2a;
  }
  buf[L & 1][0] = fn[L];
#pragma unroll
  for (int n = L - 1; n >= 0; --n) {
    const double* up = buf[(n + 1) & 1];
    double* cur = buf[n & 1];
    cur[0] = fn[n];
#pragma unroll
    for (int m = 1; m <= L - n; ++m)
#pragma unroll
      for (int t = m; t >= 0; --t)
#pragma unroll
        for (int u = m - t; u >= 0; --u) {
          const int v = m - t - u;
          double r;
          if (t == 1) {
            r = X * up[tuv_index(0, u, v)];
          } else if (u == 1) {
            r = Y * up[tuv_index(t, 0, v)];
          } else if (v == 1) {
            r = Z * up[tuv_index(t, u, 0)];
          } else if (t > 1) {
            r = fma(X, up[tuv_index(t - 1, u, v)], (t - 1) * up[tuv_index(t - 2, u, v)]);
          } else if (u > 1) {
            r = fma(Y, up[tuv_index(t, u - 1, v)], (u - 1) * up[tuv_index(t, u - 2, v)]);
          } else {
            r = fma(Z, up[tuv_index(t, u, v - 1)], (v - 1) * up[tuv_index(t, u, v - 2)]);
          }
          cur[tuv_index(t, u, v)] = r;
        }
  }
}

// Hermite coefficients E[i][j][t] (i <= LA, j <= LB, t <= i + j) of the 1-D
// product of two Gaussians, flattened, from the pair's quantities: e0 =
// exp(-ab/p X^2) in this dimension, Xpa = P - A, Xpb = P - B, h = 1/(2p).
template <int LA, int LB>
__device__ __forceinline__ void hermite_e(double e0, double Xpa, double Xpb, double h,
                                          double* E) {
  constexpr int NT = LA + LB + 1;
#define EIDX(i, j, t) (((i) * (LB + 1) + (j)) * NT + (t))
#pragma unroll
  for (int k = 0; k < (LA + 1) * (LB + 1) * NT; ++k) E[k] = 0.0;
  E[EIDX(0, 0, 0)] = e0;
#pragma unroll
  for (int i = 0; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) {
      if (i == 0 && j == 0) continue;
#pragma unroll
      for (int t = 0; t <= i + j; ++t) {
        double v;
        if (i > 0) {
          v = Xpa * E[EIDX(i - 1, j, t)];
          if (t > 0) v += h * E[EIDX(i - 1, j, t - 1)];
          if (t + 1 <= i - 1 + j) v += (t + 1) * E[EIDX(i - 1, j, t + 1)];
        } else {
          v = Xpb * E[EIDX(i, j - 1, t)];
          if (t > 0) v += h * E[EIDX(i, j - 1, t - 1)];
          if (t + 1 <= i + j - 1) v += (t + 1) * E[EIDX(i, j - 1, t + 1)];
        }
        E[EIDX(i, j, t)] = v;
      }
    }
#undef EIDX
}

// Per orbital primitive pair (e_table_kernel): p = a + b, the centre P,
// c_a c_b / p with the norms of both shells, and where its products
// E_t E_u E_v start in the table.
struct PairData {
  double p, px, py, pz, cdp;
  long long eoff;
};

// Products of one primitive pair of class (LC, LD): for every Cartesian pair
// (kc, kd) the (cx + 1)(cy + 1)(cz + 1) orders tau <= cx, nu <= cy, phi <= cz.
__host__ __device__ constexpr int e_terms(int lc, int ld) {
  int n = 0;
  for (int kc = 0; kc < ncart(lc); ++kc)
    for (int kd = 0; kd < ncart(ld); ++kd) {
      int f = 1;
      for (int dim = 0; dim < 3; ++dim) f *= cexp(lc, kc, dim) + cexp(ld, kd, dim) + 1;
      n += f;
    }
  return n;
}

struct Basis3 {
  const ShellD* aux;   // bra shells (the auxiliary basis)
  const int* alist;    // bra shells of this class
  int nalist;
  const ShellD* obs;   // ket shells
  const int2* plist;   // ket shell pairs (c, d) of this class; d < 0: exponent-0 s partner
  const int2* prange;  // per ket pair: its primitive pairs pp[x .. y)
  const long long* eoff;  // per ket pair: the first of its products in etab
  const ushort2* pp;   // (primitive of c, primitive of d) that pass the screening
  PairData* ppd;       // their data (same index)
  double* etab;        // products E_t E_u E_v of the ket primitive pairs
  int nplist;
  // For every ket primitive pair and type of bra primitive (ntype of them, 0: not
  // tabulated): gamma p / (gamma + p) and the prefactor of the integrals.
  const double2* ap;
  const int* atype;    // per bra primitive
  int ntype;
  const double* aexp;  // bra primitives: exponent gamma and
  const double* arq;   // 2 pi^(5/2) norm c / gamma / (2 gamma)^l
  const double* oexp;  // ket primitives (coefficients include the primitive
  const double* ocof;  // normalisation) and the norms of the ket shells
  const double* onorm;
  double* out;          // (P|mu nu) [X][N][N], or J [X][X] (two_center)
  int N;                // ket functions (leading dimension of out)
  int two_center;
};

// The pair data and E table of a ket class: one thread per ket pair, its
// primitive pairs in turn, the sign (-1)^(tau+nu+phi) of the ket's derivatives
// included.
template <int LC, int LD>
__global__ void __launch_bounds__(128) e_table_kernel(Basis3 g) {
  constexpr int LCD = LC + LD, NC = ncart(LC), ND = ncart(LD);
  constexpr int NE = (LC + 1) * (LD + 1) * (LCD + 1);
  for (int ki = blockIdx.x * blockDim.x + threadIdx.x; ki < g.nplist;
       ki += gridDim.x * blockDim.x) {
    const int2 cd = g.plist[ki];
    const ShellD sc = g.obs[cd.x];
    const ShellD sd = cd.y >= 0 ? g.obs[cd.y] : sc;
    const bool two = cd.y >= 0;
    const double nrm = g.onorm[cd.x] * (two ? g.onorm[cd.y] : 1.0);
    const double dx = sc.x - sd.x, dy = sc.y - sd.y, dz = sc.z - sd.z;
    double* out = g.etab + g.eoff[ki];
    const int2 rg = g.prange[ki];
    for (int q = rg.x; q < rg.y; ++q) {
      const ushort2 pr = g.pp[q];
      const double a = g.oexp[sc.poff + pr.x], b = two ? g.oexp[sd.poff + pr.y] : 0.0;
      const double p = a + b, mu = a * b / p;
      const double cc = g.ocof[sc.poff + pr.x] * (two ? g.ocof[sd.poff + pr.y] : 1.0);
      PairData pd;
      pd.p = p;
      pd.px = two ? (a * sc.x + b * sd.x) / p : sc.x;
      pd.py = two ? (a * sc.y + b * sd.y) / p : sc.y;
      pd.pz = two ? (a * sc.z + b * sd.z) / p : sc.z;
      pd.cdp = nrm * cc / p;
      pd.eoff = out - g.etab;
      g.ppd[q] = pd;
      const double h = 0.5 / p;
      double Ex[NE], Ey[NE], Ez[NE];
      hermite_e<LC, LD>(exp(-mu * dx * dx), pd.px - sc.x, pd.px - sd.x, h, Ex);
      hermite_e<LC, LD>(exp(-mu * dy * dy), pd.py - sc.y, pd.py - sd.y, h, Ey);
      hermite_e<LC, LD>(exp(-mu * dz * dz), pd.pz - sc.z, pd.pz - sd.z, h, Ez);
#pragma unroll 1
      for (int kc = 0; kc < NC; ++kc)
#pragma unroll 1
        for (int kd = 0; kd < ND; ++kd) {
          const int* ec = c_cexp[LC][kc];
          const int* ed = c_cexp[LD][kd];
          const double* ex = Ex + (ec[0] * (LD + 1) + ed[0]) * (LCD + 1);
          const double* ey = Ey + (ec[1] * (LD + 1) + ed[1]) * (LCD + 1);
          const double* ez = Ez + (ec[2] * (LD + 1) + ed[2]) * (LCD + 1);
#pragma unroll 1
          for (int ta = 0; ta <= ec[0] + ed[0]; ++ta)
#pragma unroll 1
            for (int nu = 0; nu <= ec[1] + ed[1]; ++nu) {
              const double exy = (ta + nu) & 1 ? -ex[ta] * ey[nu] : ex[ta] * ey[nu];
#pragma unroll 1
              for (int ph = 0; ph <= ec[2] + ed[2]; ++ph)
                *out++ = ph & 1 ? -exy * ez[ph] : exy * ez[ph];
            }
        }
    }
  }
}

// gamma p / (gamma + p), and 2 pi^(5/2) / (p gamma sqrt(p + gamma)) times the
// contraction coefficients and norms, for every pair and type.
__device__ __forceinline__ double2 pair_factors(double gq, double arq, const PairData& pd) {
  const double rs = rsqrt64(gq + pd.p);
  return make_double2(gq * pd.p * (rs * rs), arq * pd.cdp * rs);
}

// The same for every ket pair and type of auxiliary primitive: atoms of one kind
// share them, and computing them per integral is 11 of its 30 or more FP64
// instructions.
__global__ void ap_table_kernel(const PairData* __restrict__ ppd, long long npair,
                                const double2* __restrict__ types, int ntype,
                                double2* __restrict__ ap) {
  for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < npair * ntype;
       x += (long long)gridDim.x * blockDim.x) {
    const double2 t = types[x % ntype];
    ap[x] = pair_factors(t.x, t.y, ppd[x / ntype]);
  }
}

// Component m of shell l from its Cartesian components x[k stride].
template <int L>
__device__ __forceinline__ double spherical(int m, const double* x, int stride) {
  if (L == 0) return x[0];
  if (L == 1) return x[(m == 2 ? 0 : m + 1) * stride];  // y, z, x of x, y, z
  double s = 0.0;
  bool first = true;
#pragma unroll
  for (int k = 0; k < ncart(L); ++k) {
    if (!((sph_mask(L, m) >> k) & 1u)) continue;
    s = first ? c_sph[L][m][k] * x[k * stride] : fma(c_sph[L][m][k], x[k * stride], s);
    first = false;
  }
  return s;
}

// Contracted (P| c d) block for one bra shell and one ket pair of class
// (LP, LC, LD); spherical, normalised, written to out.  cart[kp][kc][kd]: the
// bra's derivatives of order LP, component kp = (t, u, v), of the Cartesian ket.
template <int LP, int LC, int LD>
__global__ void __launch_bounds__(128) eri3_kernel(Basis3 g) {
  constexpr int L = LP + LC + LD;
  constexpr int NP = ncart(LP), NC = ncart(LC), ND = ncart(LD);
  const long long total = (long long)g.nalist * g.nplist;
  for (long long w = blockIdx.x * (long long)blockDim.x + threadIdx.x; w < total;
       w += (long long)gridDim.x * blockDim.x) {
    const int pi = (int)(w % g.nalist);
    const int ki = (int)(w / g.nalist);
    const ShellD sp = g.aux[g.alist[pi]];
    const int2 cd = g.plist[ki];
    const ShellD sc = g.obs[cd.x];
    const bool has_d = cd.y >= 0;
    const ShellD sd = has_d ? g.obs[cd.y] : sc;
    double cart[NP * NC * ND];
#pragma unroll
    for (int k = 0; k < NP * NC * ND; ++k) cart[k] = 0.0;
    const int2 rg = g.prange[ki];
    for (int q = rg.x; q < rg.y; ++q) {
      const PairData pd = g.ppd[q];
      for (int ip = 0; ip < sp.nprim; ++ip) {
        const int k = sp.poff + ip;
        const double2 f = g.ntype ? g.ap[(size_t)q * g.ntype + g.atype[k]]
                                  : pair_factors(g.aexp[k], g.arq[k], pd);
        double Rbuf[2][tuv_count(L)];  // R^0_tuv ends in Rbuf[0]
        hermite_r<L>(f.y, f.x, sp.x - pd.px, sp.y - pd.py, sp.z - pd.pz, Rbuf);
        const double* R = Rbuf[0];
        // Run-time loops over the ket's components and orders (uniform over the
        // warp: one class per launch), index tables in constant memory.
        const double* et = g.etab + pd.eoff;
        double* out = cart;
#pragma unroll 1
        for (int kc = 0; kc < NC; ++kc)
#pragma unroll 1
          for (int kd = 0; kd < ND; ++kd, ++out) {
            const int cx = c_cexp[LC][kc][0] + c_cexp[LD][kd][0];
            const int cy = c_cexp[LC][kc][1] + c_cexp[LD][kd][1];
            const int cz = c_cexp[LC][kc][2] + c_cexp[LD][kd][2];
            double G[NP];
#pragma unroll
            for (int k = 0; k < NP; ++k) G[k] = out[k * NC * ND];
#pragma unroll 1
            for (int ta = 0; ta <= cx; ++ta)
#pragma unroll 1
              for (int nu = 0; nu <= cy; ++nu)
#pragma unroll 1
                for (int ph = 0; ph <= cz; ++ph) {
                  const double e = *et++;
#pragma unroll
                  for (int k = 0; k < NP; ++k)
                    G[k] = fma(e,
                               R[c_tuv[cexp(LP, k, 0) + ta][cexp(LP, k, 1) + nu]
                                      [cexp(LP, k, 2) + ph]],
                               G[k]);
                }
#pragma unroll
            for (int k = 0; k < NP; ++k) out[k * NC * ND] = G[k];
          }
      }
    }
    // spherical transforms (norms are in the primitives' factors), stores
    constexpr int SP = 2 * LP + 1, SC = 2 * LC + 1, SD = 2 * LD + 1;
#pragma unroll
    for (int mp = 0; mp < SP; ++mp) {
      double t1[NC * ND];
#pragma unroll
      for (int k = 0; k < NC * ND; ++k) t1[k] = spherical<LP>(mp, cart + k, NC * ND);
#pragma unroll
      for (int mc = 0; mc < SC; ++mc) {
        double t2[ND];
#pragma unroll
        for (int kd = 0; kd < ND; ++kd) t2[kd] = spherical<LC>(mc, t1 + kd, ND);
        const int fp = sp.bf + mp, fc = sc.bf + mc;
#pragma unroll
        for (int md = 0; md < SD; ++md) {
          const double v = spherical<LD>(md, t2, 1);
          if (g.two_center) {
            g.out[(size_t)fp * g.N + fc] = v;
          } else {
            const int fd = sd.bf + md;
            const size_t base = (size_t)fp * g.N * g.N;
            g.out[base + (size_t)fc * g.N + fd] = v;
            g.out[base + (size_t)fd * g.N + fc] = v;
          }
        }
      }
    }
  }
}

// ---- host side -------------------------------------------------------------
double binom(int n, int k) {
  if (k < 0 || k > n) return 0.0;
  double r = 1.0;
  for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
  return r;
}

double dfact(int n) {  // n!!, 1 for n <= 0
  double r = 1.0;
  for (int k = n; k > 1; k -= 2) r *= k;
  return r;
}

// Real regular solid harmonics S_lm (m = -l..l) as Cartesian polynomials,
// (Helgaker, Joergensen, Olsen eq. 6.4.47-6.4.50):
// S_lm = sum_{t=0}^{(l-|m|)/2} sum_{u=0}^{t} sum_{v} C_tuv x^(2t+|m|-2(u+v)) y^(2(u+v)) z^(l-2t-|m|),
// C_tuv = (-1)^(t+v-vm) (1/4)^t binom(l,t) binom(l-t,|m|+t) binom(t,u) binom(|m|,2v),
// v = vm, vm+1, ..., with vm = 0 for m >= 0 and 1/2 for m < 0.
void build_sph(double sph[kLmax + 1][2 * kLmax + 1][10]) {
  std::memset(sph, 0, sizeof(double) * (kLmax + 1) * (2 * kLmax + 1) * 10);
  for (int l = 0; l <= kLmax; ++l)
    for (int m = -l; m <= l; ++m) {
      const int am = m < 0 ? -m : m;
      const int twovm = m < 0 ? 1 : 0;  // 2 vm
      for (int t = 0; t <= (l - am) / 2; ++t)
        for (int u = 0; u <= t; ++u)
          for (int twov = twovm; twov <= am; twov += 2) {
            const int sgn = ((t + (twov - twovm) / 2) & 1) ? -1 : 1;
            const double c = sgn * std::pow(0.25, t) * binom(l, t) * binom(l - t, am + t) *
                             binom(t, u) * binom(am, twov);
            const int lx = 2 * t + am - 2 * u - twov, ly = 2 * u + twov, lz = l - 2 * t - am;
            if (lx < 0 || lz < 0) continue;
            int k = 0;  // Cartesian index of (lx, ly, lz)
            for (int x = l; x > lx; --x) k += l - x + 1;
            k += l - lx - ly;
            sph[l][m + l][k] += c;
          }
    }
  // scale every row to the norm of m = 0 (overlaps of one Gaussian: the moments
  // prod_dim (n_dim - 1)!! over even n = e_i + e_j, up to a factor of the shell)
  for (int l = 0; l <= kLmax; ++l) {
    double ov[2 * kLmax + 1] = {};
    for (int m = 0; m < 2 * l + 1; ++m)
      for (int i = 0; i < ncart(l); ++i)
        for (int j = 0; j < ncart(l); ++j) {
          double f = sph[l][m][i] * sph[l][m][j];
          for (int dim = 0; dim < 3; ++dim) {
            const int n = cexp(l, i, dim) + cexp(l, j, dim);
            f *= n & 1 ? 0.0 : dfact(n - 1);
          }
          ov[m] += f;
        }
    for (int m = 0; m < 2 * l + 1; ++m)
      for (int k = 0; k < 10; ++k) sph[l][m][k] *= std::sqrt(ov[l] / ov[m]);
  }
}

// Taylor coefficients F_{n+k}(T_i) / k!, T_i = i / kBoysPerUnit, and e^-T_i, by
// the series F_N(T) = e^-T sum_k (2T)^k / ((2N+1)(2N+3)...(2N+2k+1)) for the
// highest order (all terms positive) and downward recursion, in long double.
void build_boys(double* tab, double* etab) {
  for (int i = 0; i < kBoysPoints; ++i) {
    const long double T = (long double)i / kBoysPerUnit;
    const int N = kBoysOrders - 1;
    long double term = 1.0L / (2 * N + 1), sum = term;
    for (int k = 1; k < 2000; ++k) {
      term *= 2.0L * T / (2 * N + 2 * k + 1);
      sum += term;
      if (term < 1e-22L * sum) break;
    }
    const long double et = expl(-T);
    long double f[kBoysOrders];
    f[N] = et * sum;
    for (int n = N - 1; n >= 0; --n) f[n] = (2.0L * T * f[n + 1] + et) / (2 * n + 1);
    etab[i] = (double)et;
    for (int n = 0; n <= kBoysMax; ++n) {
      long double fact = 1.0L;
      for (int k = 0; k < kBoysTerms && n + k < kBoysOrders; ++k) {
        if (k) fact *= k;
        tab[((size_t)n * kBoysPoints + i) * kBoysTerms + k] = (double)(f[n + k] / fact);
      }
    }
  }
}

// Host copy of a basis: primitive-normalised coefficients and, per function,
// the factor that normalises its contracted spherical function.
struct HostBasis {
  std::vector<ShellD> sh;
  std::vector<double> exps, cofs;
  std::vector<double> norm;  // per shell: its m = 0 function's
  std::vector<double2> least;  // per shell: smallest exponent, largest |coefficient|
  int nbf = 0;
  int maxl = 0;
};

int make_basis(const corr_basis* b, const double sph[kLmax + 1][2 * kLmax + 1][10],
               HostBasis* out, const char* what) {
  CORR_CHECK_ARG(b && b->nsh >= 1 && b->l && b->nprim && b->poff && b->center && b->exps &&
                     b->coefs,
                 "corr_ri_integrals: bad %s basis", what);
  out->sh.resize(b->nsh);
  for (int s = 0; s < b->nsh; ++s) {
    CORR_CHECK_ARG(b->l[s] >= 0 && b->l[s] <= kLmax,
                   "corr_ri_integrals: %s shell %d has l = %d (supported: 0..%d)", what, s,
                   b->l[s], kLmax);
    CORR_CHECK_ARG(b->nprim[s] >= 1 && b->poff[s] >= 0,
                   "corr_ri_integrals: %s shell %d: bad primitives", what, s);
  }
  // Every shell gets primitives of its own: their coefficients carry its angular
  // momentum's norm and, on the auxiliary side, the shell's, while the caller's
  // shells may share a range or overlap in it.
  int bf = 0;
  for (int s = 0; s < b->nsh; ++s) {
    const int l = b->l[s];
    ShellD& d = out->sh[s];
    d.x = b->center[3 * s];
    d.y = b->center[3 * s + 1];
    d.z = b->center[3 * s + 2];
    d.l = l;
    d.nprim = b->nprim[s];
    d.poff = (int)out->exps.size();
    d.bf = bf;
    out->maxl = std::max(out->maxl, l);
    for (int k = b->poff[s]; k < b->poff[s] + d.nprim; ++k) {
      const double a = b->exps[k];
      CORR_CHECK_ARG(a > 0.0, "corr_ri_integrals: %s shell %d: exponent must be positive", what, s);
      // x^l exp(-a r^2) normalised: (2a/pi)^(3/4) (4a)^(l/2) / sqrt((2l-1)!!)
      out->exps.push_back(a);
      out->cofs.push_back(b->coefs[k] * std::pow(2.0 * a / M_PI, 0.75) *
                          std::pow(4.0 * a, 0.5 * l) / std::sqrt(dfact(2 * l - 1)));
    }
    // self-overlap of the contracted spherical functions (one centre):
    // S_ij = sum_pq c_p c_q prod_dim m(e_i + e_j, a_p + a_q),
    // m(n, s) = (n-1)!! / (2s)^(n/2) sqrt(pi/s) for even n, 0 for odd n
    const int nc = ncart(l);
    std::vector<double> Sc(nc * nc, 0.0);
    for (int i = 0; i < nc; ++i)
      for (int j = 0; j < nc; ++j) {
        double s = 0.0;
        for (int p = 0; p < d.nprim; ++p)
          for (int q = 0; q < d.nprim; ++q) {
            const double sa = out->exps[d.poff + p] + out->exps[d.poff + q];
            double f = out->cofs[d.poff + p] * out->cofs[d.poff + q];
            for (int dim = 0; dim < 3; ++dim) {
              const int n = cexp(l, i, dim) + cexp(l, j, dim);
              if (n & 1) {
                f = 0.0;
                break;
              }
              f *= dfact(n - 1) / std::pow(2.0 * sa, 0.5 * n) * std::sqrt(M_PI / sa);
            }
            s += f;
          }
        Sc[i * nc + j] = s;
      }
    double ov = 0.0;  // of m = 0; the rows of sph give the other m the same norm
    for (int i = 0; i < nc; ++i)
      for (int j = 0; j < nc; ++j) ov += sph[l][l][i] * Sc[i * nc + j] * sph[l][l][j];
    CORR_CHECK_ARG(ov > 0.0, "corr_ri_integrals: %s shell %d has a null function", what, s);
    out->norm.push_back(1.0 / std::sqrt(ov));
    double2 ext = make_double2(out->exps[d.poff], 0.0);
    for (int k = d.poff; k < d.poff + d.nprim; ++k) {
      ext.x = std::min(ext.x, out->exps[k]);
      ext.y = std::max(ext.y, std::fabs(out->cofs[k]));
    }
    out->least.push_back(ext);
    bf += 2 * l + 1;
  }
  out->nbf = bf;
  return CORR_OK;
}

// Primitive screening of the 3-index integrals.  For primitive Gaussians
// (exponents a, b on centres A, B; coefficients with their normalisation)
// the Schwarz inequality |(P|ab)| <= (P|P)^1/2 (ab|ab)^1/2 with, for s
// functions, (ab|ab) = 2 pi^(5/2) / (p^2 sqrt(2p)) K_ab^2, p = a + b,
// K_ab = exp(-ab/p |AB|^2); the factor (1 + |AB|)^(la+lb) (1 + 1/sqrt p)^(la+lb)
// covers the polynomial parts of higher angular momenta.  A primitive pair
// whose bound times the largest auxiliary factor stays below kScreen is
// skipped (its contributions lie below 1e-15 of the unit-normalised
// integrals); a shell pair left with none is zero.
constexpr double kScreen = 1e-15;

double aux_schwarz_max(const HostBasis& hb) {
  double m = 0.0;
  for (const ShellD& sh : hb.sh)
    for (int k = 0; k < sh.nprim; ++k) {
      const double q = hb.exps[sh.poff + k];
      const double f = std::fabs(hb.cofs[sh.poff + k]) *
                       std::sqrt(2.0 * std::pow(M_PI, 2.5) / (q * q * std::sqrt(2.0 * q))) *
                       std::pow(1.0 + 1.0 / std::sqrt(q), sh.l);
      m = std::max(m, f);
    }
  return m;
}

double power(double x, int n) {
  double r = 1.0;
  for (; n > 0; --n) r *= x;
  return r;
}

// Shells of the same kind (angular momentum, exponents, coefficients) and, per
// pair of kinds, the distance beyond which screen_pairs finds nothing.
struct ShellKinds {
  std::vector<int> kind;      // per shell
  std::vector<int> first;     // a shell of each kind
  std::vector<double> reach;  // squared distance, per pair of kinds; NaN: not known yet
  static constexpr int kMaxKinds = 48;

  explicit ShellKinds(const HostBasis& hb) : kind(hb.sh.size()) {
    for (size_t s = 0; s < hb.sh.size(); ++s) {
      const ShellD& a = hb.sh[s];
      size_t k = 0;
      for (; k < first.size(); ++k) {
        const ShellD& b = hb.sh[first[k]];
        if (a.l == b.l && a.nprim == b.nprim &&
            std::equal(&hb.exps[a.poff], &hb.exps[a.poff] + a.nprim, &hb.exps[b.poff]) &&
            std::equal(&hb.cofs[a.poff], &hb.cofs[a.poff] + a.nprim, &hb.cofs[b.poff]))
          break;
      }
      if (k == first.size()) {
        if (k == (size_t)kMaxKinds) {  // too many kinds: no distances
          first.clear();
          kind.clear();
          return;
        }
        first.push_back((int)s);
      }
      kind[s] = (int)k;
    }
    reach.assign(first.size() * first.size(), std::nan(""));
  }
};

// Exponent below which exp(-m) leaves the bound of screen_pairs under kScreen for
// every primitive pair of two shells r apart: without the exponential the bound
// falls with p, so its value at the smallest p and the largest coefficients.
double screen_exponent(const HostBasis& hb, int x, int y, double saux, double r) {
  const double pmin = hb.least[x].x + hb.least[y].x;
  const double k0 = std::sqrt(2.0 * std::pow(M_PI, 2.5) / std::sqrt(2.0)) * saux;
  const double top = hb.least[x].y * hb.least[y].y * k0 / (pmin * std::sqrt(std::sqrt(pmin))) *
                     power((1.0 + r) * (1.0 + 1.0 / std::sqrt(pmin)), hb.sh[x].l + hb.sh[y].l);
  return std::log(top / kScreen) + 1e-6;
}

// Squared distance from which on mu r^2 exceeds that exponent, mu of the two
// smallest exponents: their difference is concave in r, so its largest root.
double screen_reach(const HostBasis& hb, int x, int y, double saux) {
  const double a = hb.least[x].x, b = hb.least[y].x, mu = a * b / (a + b);
  const int lsum = hb.sh[x].l + hb.sh[y].l;
  auto f = [&](double r) { return screen_exponent(hb, x, y, saux, r) - mu * r * r; };
  double lo = 0.5 * (std::sqrt(1.0 + 2.0 * lsum / mu) - 1.0);  // its maximum
  if (f(lo) < 0.0) return -1.0;
  double hi = lo + 1.0;
  while (f(hi) >= 0.0) hi *= 2.0;
  for (int k = 0; k < 40; ++k) (f(0.5 * (lo + hi)) >= 0.0 ? lo : hi) = 0.5 * (lo + hi);
  return hi * hi;
}

void screen_pairs(const HostBasis& hb, ShellKinds& kinds, int x, int y, double saux,
                  std::vector<ushort2>* pp) {
  const ShellD& A = hb.sh[x];
  const ShellD& B = hb.sh[y];
  const double dx = A.x - B.x, dy = A.y - B.y, dz = A.z - B.z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  if (!kinds.kind.empty()) {
    double& reach = kinds.reach[kinds.kind[x] * kinds.first.size() + kinds.kind[y]];
    if (std::isnan(reach)) reach = screen_reach(hb, x, y, saux);
    if (r2 > reach) return;
  }
  const double r = std::sqrt(r2), far = screen_exponent(hb, x, y, saux, r);
  const int lsum = A.l + B.l;
  const double k0 = std::sqrt(2.0 * std::pow(M_PI, 2.5) / std::sqrt(2.0)) * saux;
  for (int i = 0; i < A.nprim; ++i)
    for (int j = 0; j < B.nprim; ++j) {
      const double a = hb.exps[A.poff + i], b = hb.exps[B.poff + j], p = a + b;
      const double m = a * b / p * r2;
      if (m > far) continue;
      const double sp = std::sqrt(p);
      const double bound = std::fabs(hb.cofs[A.poff + i] * hb.cofs[B.poff + j]) * std::exp(-m) *
                           k0 / (p * std::sqrt(sp)) *
                           power((1.0 + r) * (1.0 + 1.0 / sp), lsum);
      if (bound >= kScreen) pp->push_back(make_ushort2((unsigned short)i, (unsigned short)j));
    }
}

using Kern = void (*)(Basis3);

template <int LP, int LC, int LD>
Kern kern() {
  return eri3_kernel<LP, LC, LD>;
}

// class table: ket classes (LC, LD) used by the 3-index (LD <= LC <= 2) and
// the 2-index (LD = 0, LC <= 3) integrals
Kern class_kernel(int lp, int lc, int ld) {
#define KC(LP)                                                     \
  if (lp == LP) {                                                  \
    if (lc == 0 && ld == 0) return kern<LP, 0, 0>();               \
    if (lc == 1 && ld == 0) return kern<LP, 1, 0>();               \
    if (lc == 1 && ld == 1) return kern<LP, 1, 1>();               \
    if (lc == 2 && ld == 0) return kern<LP, 2, 0>();               \
    if (lc == 2 && ld == 1) return kern<LP, 2, 1>();               \
    if (lc == 2 && ld == 2) return kern<LP, 2, 2>();               \
    if (lc == 3 && ld == 0) return kern<LP, 3, 0>();               \
  }
  KC(0)
  KC(1)
  KC(2)
  KC(3)
#undef KC
  return nullptr;
}

Kern table_kernel(int lc, int ld) {
  if (lc == 0 && ld == 0) return e_table_kernel<0, 0>;
  if (lc == 1 && ld == 0) return e_table_kernel<1, 0>;
  if (lc == 1 && ld == 1) return e_table_kernel<1, 1>;
  if (lc == 2 && ld == 0) return e_table_kernel<2, 0>;
  if (lc == 2 && ld == 1) return e_table_kernel<2, 1>;
  if (lc == 2 && ld == 2) return e_table_kernel<2, 2>;
  if (lc == 3 && ld == 0) return e_table_kernel<3, 0>;
  return nullptr;
}

}  // namespace

}  // namespace corr

using namespace corr;

extern "C" int corr_ri_integrals(corr_context* c, const corr_basis* obs, const corr_basis* aux,
                                 double* J, double* pmn) {
  CORR_CHECK_ARG(c != nullptr, "null context");
  CORR_CHECK_ARG(J || pmn, "corr_ri_integrals: nothing to compute (J and pmn both NULL)");
  CORR_CHECK_ARG(aux != nullptr && (obs != nullptr || !pmn),
                 "corr_ri_integrals: null basis argument");
  CORR_CUDA(cudaSetDevice(c->device));
  double sph[kLmax + 1][2 * kLmax + 1][10];
  build_sph(sph);
  HostBasis ha, ho;
  CORR_TRY(make_basis(aux, sph, &ha, "auxiliary"));
  if (pmn) {
    CORR_TRY(make_basis(obs, sph, &ho, "orbital"));
    CORR_CHECK_ARG(ho.maxl <= 2, "corr_ri_integrals: orbital shells up to d are supported");
  }
  const int X = ha.nbf, N = pmn ? ho.nbf : 0;
  std::vector<double> arq(ha.exps.size());
  for (size_t q = 0; q < ha.sh.size(); ++q) {
    const ShellD& sh = ha.sh[q];
    for (int k = sh.poff; k < sh.poff + sh.nprim; ++k)
      arq[k] = 34.986836655249725 * ha.norm[q] * ha.cofs[k] / ha.exps[k] *
               std::pow(0.5 / ha.exps[k], sh.l);
  }
  // types of auxiliary primitives (the same on every atom of a kind)
  std::vector<double2> types;
  std::vector<int> atype(ha.exps.size(), 0);
  {
    std::map<std::pair<double, double>, int> known;
    for (size_t k = 0; k < ha.exps.size(); ++k) {
      const auto it = known.emplace(std::make_pair(ha.exps[k], arq[k]), (int)types.size());
      if (it.second) types.push_back(make_double2(ha.exps[k], arq[k]));
      atype[k] = it.first->second;
    }
  }
  // shell lists by angular momentum, ket pairs by class
  std::vector<std::vector<int>> alist(kLmax + 1);
  for (int s = 0; s < (int)ha.sh.size(); ++s) alist[ha.sh[s].l].push_back(s);
  std::vector<std::vector<int2>> plist3(9), plist2(kLmax + 1);  // 3c: lc*3 + ld ; 2c: lc
  // primitive pairs of every ket pair: all of them for (P|Q); for (P|cd) the
  // pairs whose Schwarz factor can reach kScreen (see screen_pairs)
  std::vector<std::vector<int2>> prange3(9), prange2(kLmax + 1);
  std::vector<ushort2> pp;
  std::vector<std::vector<long long>> eoff3(9), eoff2(kLmax + 1);
  long long etot = 0;
  for (int s = 0; s < (int)ha.sh.size(); ++s) {
    const ShellD& A = ha.sh[s];
    const int b = (int)pp.size();
    for (int k = 0; k < A.nprim; ++k) pp.push_back(make_ushort2((unsigned short)k, 0));
    plist2[A.l].push_back(make_int2(s, -1));
    prange2[A.l].push_back(make_int2(b, (int)pp.size()));
    eoff2[A.l].push_back(etot);
    etot += (long long)A.nprim * e_terms(A.l, 0);
  }
  if (pmn) {
    const double saux = aux_schwarz_max(ha);
    ShellKinds kinds(ho);
    int terms[9] = {};
    for (int lc = 0; lc <= 2; ++lc)
      for (int ld = 0; ld <= lc; ++ld) terms[lc * 3 + ld] = e_terms(lc, ld);
    for (int cs = 0; cs < (int)ho.sh.size(); ++cs)
      for (int ds = 0; ds <= cs; ++ds) {
        int x = cs, y = ds;
        if (ho.sh[x].l < ho.sh[y].l) std::swap(x, y);  // lc >= ld
        const int b = (int)pp.size();
        screen_pairs(ho, kinds, x, y, saux, &pp);
        const int n = (int)pp.size() - b;
        if (n == 0) continue;  // every integral of the pair is below the threshold
        const int k = ho.sh[x].l * 3 + ho.sh[y].l;
        plist3[k].push_back(make_int2(x, y));
        prange3[k].push_back(make_int2(b, b + n));
        eoff3[k].push_back(etot);
        etot += (long long)n * terms[k];
      }
  }
  // tabulated while the table stays small (molecules of a few kinds of atoms)
  const int ntype = pp.size() * types.size() * 16 <= ((size_t)1 << 29) ? (int)types.size() : 0;
  // device copies (workspace): shells, primitives, norms, lists, staged outputs
  auto bytes_of = [](size_t n, size_t e) { return n * e; };
  size_t nal = 0, np3 = 0, np2 = 0;
  for (auto& v : alist) nal += v.size();
  for (auto& v : plist3) np3 += v.size();
  for (auto& v : plist2) np2 += v.size();
  const bool jdev = J && is_device_ptr(J), pdev = pmn && is_device_ptr(pmn);
  auto plan = [&](Carver& w, void** p) {
    p[0] = w.take(bytes_of(ha.sh.size(), sizeof(ShellD)));
    p[1] = w.take(bytes_of(ha.exps.size(), 8));
    p[2] = w.take(bytes_of(ha.cofs.size(), 8));
    p[3] = w.take(bytes_of(ha.norm.size(), 8));
    p[4] = w.take(bytes_of(nal, 4));
    p[5] = w.take(bytes_of(np2, 8));
    p[6] = pmn ? w.take(bytes_of(ho.sh.size(), sizeof(ShellD))) : nullptr;
    p[7] = pmn ? w.take(bytes_of(ho.exps.size(), 8)) : nullptr;
    p[8] = pmn ? w.take(bytes_of(ho.cofs.size(), 8)) : nullptr;
    p[9] = pmn ? w.take(bytes_of(ho.norm.size(), 8)) : nullptr;
    p[10] = pmn ? w.take(bytes_of(np3, 8)) : nullptr;
    p[11] = (J && !jdev) ? w.take((size_t)X * X * 8) : nullptr;
    p[12] = (pmn && !pdev) ? w.take((size_t)X * N * N * 8) : nullptr;
    p[13] = w.take(bytes_of(np2, 8));
    p[14] = pmn ? w.take(bytes_of(np3, 8)) : nullptr;
    p[15] = w.take(bytes_of(pp.size(), 4));
    p[16] = w.take(bytes_of(pp.size(), sizeof(PairData)));
    p[17] = w.take(bytes_of(ha.exps.size(), 8));
    p[18] = w.take(bytes_of((size_t)etot, 8));
    p[19] = w.take(bytes_of(np2, 8));
    p[20] = pmn ? w.take(bytes_of(np3, 8)) : nullptr;
    p[21] = w.take(bytes_of(types.size(), 16));
    p[22] = w.take(bytes_of(atype.size(), 4));
    p[23] = w.take(bytes_of(pp.size() * ntype, 16));
  };
  void* p[24];
  Carver cv{nullptr, 0};
  plan(cv, p);
  CORR_TRY(c->ws.reserve(cv.used));
  Carver w{c->ws.ptr, 0};
  plan(w, p);
  // host-side packing of the lists (contiguous per class)
  std::vector<int> aflat;
  std::vector<int> aoff(kLmax + 2, 0);
  for (int l = 0; l <= kLmax; ++l) {
    aoff[l] = (int)aflat.size();
    aflat.insert(aflat.end(), alist[l].begin(), alist[l].end());
  }
  aoff[kLmax + 1] = (int)aflat.size();
  std::vector<int2> p2flat, p3flat, r2flat, r3flat;
  std::vector<long long> e2flat, e3flat;
  std::vector<int> p2off(kLmax + 2, 0), p3off(10, 0);
  for (int l = 0; l <= kLmax; ++l) {
    p2off[l] = (int)p2flat.size();
    p2flat.insert(p2flat.end(), plist2[l].begin(), plist2[l].end());
    r2flat.insert(r2flat.end(), prange2[l].begin(), prange2[l].end());
    e2flat.insert(e2flat.end(), eoff2[l].begin(), eoff2[l].end());
  }
  p2off[kLmax + 1] = (int)p2flat.size();
  for (int k = 0; k < 9; ++k) {
    p3off[k] = (int)p3flat.size();
    p3flat.insert(p3flat.end(), plist3[k].begin(), plist3[k].end());
    r3flat.insert(r3flat.end(), prange3[k].begin(), prange3[k].end());
    e3flat.insert(e3flat.end(), eoff3[k].begin(), eoff3[k].end());
  }
  p3off[9] = (int)p3flat.size();
  auto up = [&](void* dst, const void* src, size_t n) -> int {
    if (n) CORR_CUDA(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, c->stream));
    return CORR_OK;
  };
  CORR_TRY(up(p[0], ha.sh.data(), ha.sh.size() * sizeof(ShellD)));
  CORR_TRY(up(p[1], ha.exps.data(), ha.exps.size() * 8));
  CORR_TRY(up(p[2], ha.cofs.data(), ha.cofs.size() * 8));
  CORR_TRY(up(p[3], ha.norm.data(), ha.norm.size() * 8));
  CORR_TRY(up(p[4], aflat.data(), aflat.size() * 4));
  CORR_TRY(up(p[5], p2flat.data(), p2flat.size() * 8));
  CORR_TRY(up(p[13], r2flat.data(), r2flat.size() * 8));
  CORR_TRY(up(p[15], pp.data(), pp.size() * 4));
  CORR_TRY(up(p[19], e2flat.data(), e2flat.size() * 8));
  CORR_TRY(up(p[17], arq.data(), arq.size() * 8));
  CORR_TRY(up(p[21], types.data(), types.size() * 16));
  CORR_TRY(up(p[22], atype.data(), atype.size() * 4));
  if (pmn) {
    CORR_TRY(up(p[14], r3flat.data(), r3flat.size() * 8));
    CORR_TRY(up(p[6], ho.sh.data(), ho.sh.size() * sizeof(ShellD)));
    CORR_TRY(up(p[7], ho.exps.data(), ho.exps.size() * 8));
    CORR_TRY(up(p[8], ho.cofs.data(), ho.cofs.size() * 8));
    CORR_TRY(up(p[9], ho.norm.data(), ho.norm.size() * 8));
    CORR_TRY(up(p[10], p3flat.data(), p3flat.size() * 8));
    CORR_TRY(up(p[20], e3flat.data(), e3flat.size() * 8));
  }
  CORR_CUDA(cudaMemcpyToSymbolAsync(c_sph, sph, sizeof(sph), 0, cudaMemcpyHostToDevice, c->stream));
  {
    // built and uploaded once; a second thread's first call waits for that
    static std::mutex boys_mutex;
    std::lock_guard<std::mutex> lock(boys_mutex);
    static std::vector<double> boys_tab, boys_exp;
    static bool boys_done[64] = {};
    if (boys_tab.empty()) {
      boys_exp.resize(kBoysPoints);
      boys_tab.resize((size_t)(kBoysMax + 1) * kBoysPoints * kBoysTerms);
      build_boys(boys_tab.data(), boys_exp.data());
    }
    if (c->device < 0 || c->device >= 64 || !boys_done[c->device]) {
      CORR_CUDA(cudaMemcpyToSymbol(d_boys, boys_tab.data(), boys_tab.size() * 8));
      CORR_CUDA(cudaMemcpyToSymbol(d_boys_exp, boys_exp.data(), boys_exp.size() * 8));
      if (c->device >= 0 && c->device < 64) boys_done[c->device] = true;
    }
  }
  {
    static int ce[kLmax + 1][10][3], tv[kTmax][kTmax][kTmax];  // constant tables
    for (int l = 0; l <= kLmax; ++l)
      for (int k = 0; k < 10; ++k)
        for (int d = 0; d < 3; ++d) ce[l][k][d] = k < ncart(l) ? cexp(l, k, d) : 0;
    for (int t = 0; t < kTmax; ++t)
      for (int u = 0; u < kTmax; ++u)
        for (int v = 0; v < kTmax; ++v) tv[t][u][v] = tuv_index(t, u, v);
    CORR_CUDA(cudaMemcpyToSymbolAsync(c_cexp, ce, sizeof(ce), 0, cudaMemcpyHostToDevice,
                                      c->stream));
    CORR_CUDA(cudaMemcpyToSymbolAsync(c_tuv, tv, sizeof(tv), 0, cudaMemcpyHostToDevice,
                                      c->stream));
  }
  CORR_CUDA(cudaMemsetAsync(c->dres, 0, sizeof(ResultBlock), c->stream));
  mark(c, 0);
  mark(c, 1);
  CORR_CUDA(cudaGetLastError());
  // The largest classes keep their Cartesian block and Hermite tables in
  // local memory (up to ~8 KB per thread): raise this context's per-thread
  // stack limit to what the kernels of this call need, if it is lower.
  {
    size_t need = 0;
    for (int lp = 0; lp <= kLmax; ++lp)
      for (int lc = 0; lc <= kLmax; ++lc)
        for (int ld = 0; ld <= 2; ++ld) {
          Kern k = class_kernel(lp, lc, ld);
          if (!k) continue;
          cudaFuncAttributes fa{};
          CORR_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(k)));
          need = std::max(need, fa.localSizeBytes);
          if (lp == 0) {
            CORR_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(table_kernel(lc, ld))));
            need = std::max(need, fa.localSizeBytes);
          }
        }
    size_t have = 0;
    CORR_CUDA(cudaDeviceGetLimit(&have, cudaLimitStackSize));
    need = (need + 1023) / 1024 * 1024 + 1024;
    if (have < need) CORR_CUDA(cudaDeviceSetLimit(cudaLimitStackSize, need));
  }
  // The classes write disjoint blocks of J and (P|mu nu): they run on eight
  // side streams forked from (and joined back into) the context stream, so
  // the tails of the large classes overlap the small ones.
  constexpr int kSide = corr_context::kPreStreams;
  if (!c->pre_stream[0]) {
    for (int k = 0; k < kSide; ++k)
      CORR_CUDA(cudaStreamCreateWithFlags(&c->pre_stream[k], cudaStreamNonBlocking));
    for (int k = 0; k <= kSide; ++k)
      CORR_CUDA(cudaEventCreateWithFlags(&c->pre_ev[k], cudaEventDisableTiming));
  }
  int next_stream = 0;
  auto launch = [&](Kern k, Basis3 g, int lp, int lc, int ld) -> int {
    const long long work = (long long)g.nalist * g.nplist;
    if (work <= 0) return CORR_OK;
    const int grid = (int)std::min<long long>((work + 127) / 128, (long long)c->sms * 32);
    k<<<grid, 128, 0, c->pre_stream[next_stream]>>>(g);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      cudaFuncAttributes fa{};
      cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(k));
      cudaGetLastError();
      size_t lim = 0;
      cudaDeviceGetLimit(&lim, cudaLimitStackSize);
      cudaGetLastError();
      set_error("corr_ri_integrals: launch of class (%d|%d %d) failed: %s (local %zu B, "
                "max threads per block %d, registers %d, stack limit %zu, grid %d)",
                lp, lc, ld, cudaGetErrorString(e), fa.localSizeBytes, fa.maxThreadsPerBlock,
                fa.numRegs, lim, grid);
      return CORR_ERR_CUDA;
    }
    c->launches += 1;
    return CORR_OK;
  };
  const ShellD* dA = static_cast<const ShellD*>(p[0]);
  double* Jout = J ? (jdev ? J : static_cast<double*>(p[11])) : nullptr;
  double* Pout = pmn ? (pdev ? pmn : static_cast<double*>(p[12])) : nullptr;
  if (Pout) CORR_CUDA(cudaMemsetAsync(Pout, 0, (size_t)X * N * N * 8, c->stream));
  // every class launch with a cost estimate (auxiliary primitives x orbital
  // primitive pairs x Cartesian components); launched largest first, each on
  // the side stream with the least estimated work so far
  struct Job {
    Kern k;
    Basis3 g;
    int lp, lc, ld;
    double cost;
  };
  std::vector<Job> jobs;
  auto pairs_of = [](const std::vector<int2>& r) {
    double n = 0.0;
    for (const int2& x : r) n += x.y - x.x;
    return n;
  };
  for (int lp = 0; lp <= kLmax; ++lp) {
    const int na = aoff[lp + 1] - aoff[lp];
    if (na == 0) continue;
    double aprim = 0.0;
    for (int sidx : alist[lp]) aprim += ha.sh[sidx].nprim;
    Basis3 g{};
    g.aux = dA;
    g.alist = static_cast<const int*>(p[4]) + aoff[lp];
    g.nalist = na;
    g.aexp = static_cast<const double*>(p[1]);
    g.ppd = static_cast<PairData*>(p[16]);
    g.arq = static_cast<const double*>(p[17]);
    g.etab = static_cast<double*>(p[18]);
    g.ap = static_cast<const double2*>(p[23]);
    g.atype = static_cast<const int*>(p[22]);
    g.ntype = ntype;
    if (J) {  // (P|Q): the ket is the auxiliary basis with an exponent-0 s partner
      for (int lc = 0; lc <= kLmax; ++lc) {
        Basis3 h = g;
        h.obs = dA;
        h.plist = static_cast<const int2*>(p[5]) + p2off[lc];
        h.prange = static_cast<const int2*>(p[13]) + p2off[lc];
        h.pp = static_cast<const ushort2*>(p[15]);
        h.nplist = p2off[lc + 1] - p2off[lc];
        h.eoff = static_cast<const long long*>(p[19]) + p2off[lc];
        h.oexp = h.aexp;
        h.ocof = static_cast<const double*>(p[2]);
        h.onorm = static_cast<const double*>(p[3]);
        h.out = Jout;
        h.N = X;
        h.two_center = 1;
        jobs.push_back({class_kernel(lp, lc, 0), h, lp, lc, 0,
                        aprim * pairs_of(prange2[lc]) * ncart(lp) * ncart(lc)});
      }
    }
    if (pmn) {
      for (int lc = 0; lc <= 2; ++lc)
        for (int ld = 0; ld <= lc; ++ld) {
          Basis3 h = g;
          h.obs = static_cast<const ShellD*>(p[6]);
          h.plist = static_cast<const int2*>(p[10]) + p3off[lc * 3 + ld];
          h.prange = static_cast<const int2*>(p[14]) + p3off[lc * 3 + ld];
          h.pp = static_cast<const ushort2*>(p[15]);
          h.nplist = p3off[lc * 3 + ld + 1] - p3off[lc * 3 + ld];
          h.oexp = static_cast<const double*>(p[7]);
          h.ocof = static_cast<const double*>(p[8]);
          h.onorm = static_cast<const double*>(p[9]);
          h.eoff = static_cast<const long long*>(p[20]) + p3off[lc * 3 + ld];
          h.out = Pout;
          h.N = N;
          h.two_center = 0;
          jobs.push_back({class_kernel(lp, lc, ld), h, lp, lc, ld,
                          aprim * pairs_of(prange3[lc * 3 + ld]) * ncart(lp) * ncart(lc) *
                              ncart(ld)});
        }
    }
  }
  // the E tables of the ket classes, ahead of the class launches
  {
    bool done[2][9] = {};
    for (const Job& jb : jobs) {
      bool& d = jb.g.two_center ? done[0][jb.lc] : done[1][jb.lc * 3 + jb.ld];
      if (d || jb.g.nplist <= 0) continue;
      d = true;
      table_kernel(jb.lc, jb.ld)<<<std::min((jb.g.nplist + 127) / 128, c->sms * 16), 128, 0,
                                   c->stream>>>(jb.g);
      CORR_CUDA(cudaGetLastError());
      c->launches += 1;
    }
  }
  if (ntype) {
    const long long n = (long long)pp.size() * ntype;
    ap_table_kernel<<<(int)std::min<long long>((n + 255) / 256, c->sms * 16), 256, 0, c->stream>>>(
        static_cast<const PairData*>(p[16]), (long long)pp.size(),
        static_cast<const double2*>(p[21]), ntype, static_cast<double2*>(p[23]));
    CORR_CUDA(cudaGetLastError());
    c->launches += 1;
  }
  CORR_CUDA(cudaEventRecord(c->pre_ev[kSide], c->stream));
  for (int k = 0; k < kSide; ++k)
    CORR_CUDA(cudaStreamWaitEvent(c->pre_stream[k], c->pre_ev[kSide], 0));
  std::stable_sort(jobs.begin(), jobs.end(),
                   [](const Job& a, const Job& b) { return a.cost > b.cost; });
  double load[kSide] = {};
  for (const Job& jb : jobs) {
    int k = 0;
    for (int q = 1; q < kSide; ++q)
      if (load[q] < load[k]) k = q;
    load[k] += jb.cost;
    next_stream = k;
    CORR_TRY(launch(jb.k, jb.g, jb.lp, jb.lc, jb.ld));
  }
  for (int k = 0; k < kSide; ++k) {
    CORR_CUDA(cudaEventRecord(c->pre_ev[k], c->pre_stream[k]));
    CORR_CUDA(cudaStreamWaitEvent(c->stream, c->pre_ev[k], 0));
  }
  mark(c, 2);
  if (J && !jdev) CORR_TRY(stage_out(c, J, Jout, (size_t)X * X * 8));
  if (pmn && !pdev) CORR_TRY(stage_out(c, pmn, Pout, (size_t)X * N * N * 8));
  return finish_results(c, 0);
}
