// predictor_fix.cuh -- the FP64 predictor with its linear algebra in 60-bit
// fixed point on the integer multiply-add pipe.
//
// Why: the FP64 pipe issues one warp instruction per 20 SM cycles (1.6 lanes
// per clock, measured), the 32x32+64-bit multiply-add (IMAD.WIDE) one per 1.6.
// Most of the predictor's FP64 instructions are products with constant
// matrices: flux derivatives (Kxi), time update (T), time averages, volume
// integral and face extrapolation.  A product of two 60-bit numbers in 31-bit
// limbs takes three IMAD.WIDE (the low x low product is below the last bit
// kept), or one and two IMAD.HI (the cross products' upper halves) = 4.9 or 3.8
// cycles instead of 20, and the pipes overlap: the FP64 pipe keeps the
// pointwise fluxes and one conversion per result.  Measured (FP64 mode, all in
// registers and FP64 before): Euler vortex N = 4, 256^2 5.02 -> 2.05 ms, Riemann
// problem N = 3, 257 x 193 1.32 -> 0.56 ms, Baer-Nunziato cylinder N = 3, 200^2
// 3.28 -> 1.83 ms.  With IMAD.HI throughout the vortex takes 1.91 ms, but the
// average flux then loses up to a factor 6 of its accuracy; with IMAD.WIDE
// throughout 2.29 ms.  N >= 3: below, the Picard iterations between the first and
// the last, which this is for, are at most one.
//
// Accuracy: each operand line takes its own power-of-two scale from its
// largest magnitude, so a value's error is at most 2^-60 of that magnitude, and
// the constants are formed to twice FP64 and rounded to 2^-60 of the matrix's
// largest row sum (the FP64 ones miss the exact sums by up to 4e-15).  Against
// the predictor evaluated in 80-bit arithmetic (Euler and Baer-Nunziato, N = 3..5,
// smooth and discontinuous states, with and without noise: 27 configurations) the
// root mean square error is that of the FP64 chain times, geometric mean and
// largest: time-averaged state 0.36 and 0.99, its face values 0.25 and 0.78,
// time-averaged fluxes 0.35 and 0.74, theirs 0.32 and 0.71.
// Lines holding infinities or NaNs, or whose largest magnitude is beyond 2^900
// or below 2^-823, are contracted in FP64 and their nodes take the FP64 time
// update.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "physics.cuh"

namespace aderdg {

constexpr int kFixMin = 200;           // lines whose largest biased exponent lies below (2^-823)
constexpr int kFixMax = 1023 + 900;    // or from here on take FP64
constexpr int kFixOut = 1 << 20;       // "exponent" of a line contracted in FP64

// Numbers are (h, l) with value h 2^31 + l, l >= 0 in 31 bits.  A sum of n
// products in units of 2^62: h*h exactly (IMAD.WIDE, into s); of the two cross
// products (units of 2^31), with kFine the whole (IMAD.WIDE into 64 bits), else
// the upper 32 bits (IMAD.HI into 32 bits: two units each, half of them rounded
// away on average).  The start value holds the mean of what is left out (and,
// with kFine, the rounding half), unless all operands are 0: zeros stay exact.
template <bool kFine>
struct FixSum {
  using M = typename std::conditional<kFine, long long, int>::type;
  long long s = 0;
  M m;
  __device__ __forceinline__ FixSum(bool any, int n) {
    if constexpr (kFine) m = any ? ((long long)n << 29) + (1ll << 30) : 0;
    else m = any ? n : 0;
  }
  __device__ __forceinline__ void madd(int ah, int al, int bh, int bl) {
    s += (long long)ah * bh;
    if constexpr (kFine) {
      m += (long long)ah * bl;
      m += (long long)al * bh;
    } else {
      asm("mad.hi.s32 %0, %1, %2, %0;" : "+r"(m) : "r"(ah), "r"(bl));
      asm("mad.hi.s32 %0, %1, %2, %0;" : "+r"(m) : "r"(al), "r"(bh));
    }
  }
  __device__ __forceinline__ long long sum() const {
    if constexpr (kFine) return s + (m >> 31);
    else return s + 2 * (long long)m;
  }
};
__device__ __forceinline__ int fix_hi(long long x) { return (int)(x >> 31); }
__device__ __forceinline__ int fix_lo(long long x) { return (int)x & 0x7fffffff; }
// x >> d, 0 <= d, floor; everything beyond 63 is the sign
__device__ __forceinline__ long long fix_shift(long long x, int d) { return x >> (d < 63 ? d : 63); }
// signed integer X, |X| < 2^(53 + kUp), of the finite double (hi, lo) relative
// to a biased exponent E >= its own: x = X 2^(E - 1023 - 52 - kUp)
template <int kUp = 7>
__device__ __forceinline__ long long fix_int(int hi, int lo, int E) {
  const int d = E - ((hi >> 20) & 0x7ff);
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const unsigned long long x =
      (((unsigned long long)__funnelshift_l((unsigned)lo, mh, kUp) << 32) | ((unsigned)lo << kUp)) >> (d < 63 ? d : 63);
  const long long s = hi >> 31;
  return ((long long)x ^ s) - s;
}
// x 2^e, -1000 < e < 900 (one conversion; the exponent is added as an integer)
__device__ __forceinline__ double fix_double(long long x, int e) {
  const double r = (double)x;
  return __hiloint2double(__double2hiint(r) + (x != 0 ? e << 20 : 0), __double2loint(r));
}
// a positive factor c = C 2^(e - 1023 - 61), C = (h, l) in [2^61, 2^62)
struct FixFactor {
  int h, l, e;
  __device__ explicit FixFactor(double c) {
    const int hi = __double2hiint(c), lo = __double2loint(c);
    e = (hi >> 20) & 0x7ff;
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const long long x = (long long)(((unsigned long long)__funnelshift_l((unsigned)lo, mh, 9) << 32) | ((unsigned)lo << 9));
    h = fix_hi(x);
    l = fix_lo(x);
  }
  __device__ __forceinline__ long long times(long long r) const {  // r C / 2^62
    FixSum<true> s(r != 0, 1);
    s.madd(fix_hi(r), fix_lo(r), h, l);
    return s.sum();
  }
};
// value of a contracted entry with matrix scale 2^sh, out of line (rare): the
// bits of a double where E says so, else in fixed point
static __device__ __noinline__ double fix_value(double bits, int E, int sh) {
  return E == kFixOut ? bits : scalbn((double)__double_as_longlong(bits), E - 1020 - sh);
}

// P values p[0], p[stride], .. as limbs relative to their largest exponent E.
template <int P>
struct FixLine {
  int hi[P], lo[P], E;
  bool any;
  // false where the values need FP64
  __device__ __forceinline__ bool load(const double* __restrict__ p, int stride) {
    int top = 0;
#pragma unroll
    for (int k = 0; k < P; ++k) {
      const double f = p[k * stride];
      hi[k] = __double2hiint(f);
      lo[k] = __double2loint(f);
      const int m = hi[k] & 0x7fffffff;
      top = top > m ? top : m;
    }
    any = top != 0;
    E = any ? top >> 20 : kFixMin;
    return E >= kFixMin && E < kFixMax;
  }
  __device__ __forceinline__ double value(int k) const { return __hiloint2double(hi[k], lo[k]); }
  __device__ __forceinline__ void limbs() {
#pragma unroll
    for (int k = 0; k < P; ++k) {
      const long long x = fix_int(hi[k], lo[k], E);
      hi[k] = fix_hi(x);
      lo[k] = fix_lo(x);
    }
  }
  // the values' differences from value 0 (k >= 1), exactly; E as for values
  // twice as large
  __device__ __forceinline__ void deviations() {
    const long long x0 = fix_int<6>(hi[0], lo[0], E);
    any = false;
#pragma unroll
    for (int k = 1; k < P; ++k) {
      const long long x = fix_int<6>(hi[k], lo[k], E) - x0;
      hi[k] = fix_hi(x);
      lo[k] = fix_lo(x);
      any = any || x != 0;
    }
    ++E;
  }
  // sum over k >= kFirst of M[k * st] x_k, in units of 2^(E - 1020 - scale of M)
  template <bool kFine, int kFirst = 0>
  __device__ __forceinline__ long long dot(const int* Mh, const int* Ml, int st) const {
    FixSum<kFine> s(any, P - kFirst);
#pragma unroll
    for (int k = kFirst; k < P; ++k) s.madd(hi[k], lo[k], Mh[k * st], Ml[k * st]);
    return s.sum();
  }
};

// The derivative of one line in place, p[o] <- sum_k Kxi(k, o) p[k] as the
// integer R and the line's exponent.  The derivative of a constant is 0 (the
// 60-bit columns of Kxi sum to 0), so the line's differences from its first value
// are contracted: one product less an output, and 0 for a constant line.
template <int P, bool kFine, class Ops>
__device__ __forceinline__ void fix_line(double* __restrict__ p, int stride, int* __restrict__ ex, const Ops& op) {
  FixLine<P> x;
  if (!x.load(p, stride)) {
#pragma unroll 1
    for (int o = 0; o < P; ++o) {
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < P; ++k) s = fma(op.Kxi[k + P * o], x.value(k), s);
      p[o * stride] = s;
    }
    *ex = kFixOut;
    return;
  }
  x.deviations();
#pragma unroll
  for (int o = 0; o < P; ++o)
    p[o * stride] = __longlong_as_double(x.template dot<kFine, 1>(op.Kh + P * o, op.Kl + P * o, 1));
  *ex = x.E;
}

// Euler and Baer-Nunziato.  Shared memory of a cell: the flux planes [VF][x
// levels, y levels] (PredCfg::XL, YL, Y0), the line exponents [VF][2][P
// levels][P lines], Baer-Nunziato's volume fraction [P][P2]; sG: dudx, per
// CTA.  A node's time column q(l, v) lives in its own x-plane entries (the
// volume fraction in its own plane) between the update that forms it and the
// flux evaluation that replaces it, so no thread holds it in registers and the
// loops over the variables stay rolled: with the column in registers
// Baer-Nunziato N = 3 took 218 registers and two CTAs of 128 threads per SM, and
// waited on latency and instruction fetch (2.32 ms against 1.91 ms).  On return qh, Fh, Sh hold the node's time averages.
// un: the node's state at the start of the step; live: false in the lanes past
// the CTA's last cell, which take part in the barriers only.
template <class Sys, int N, class C, class PC>
__device__ __forceinline__ void picard_fix(double* __restrict__ cs, const double* __restrict__ sG,
                                           const PredOps<N, double>& op, const PC& pc, const double* __restrict__ un,
                                           bool act, int i, int j, double cxw, double cyw, double idx, double idy,
                                           double dt, double* qh, double (*Fh)[Sys::V], double* Sh, bool live) {
  constexpr int P = N + 1, P2 = P * P, V = Sys::V, VF = C::VF;
  constexpr bool BN = Sys::ID == kSysBN;
  const int node = i + P * j;
  int* ex = reinterpret_cast<int*>(cs + C::FLUX_ELEMS);
  double* as = cs + C::FLUX_ELEMS + C::EXP_ELEMS;
  double pg[BN ? P : 1], us[BN ? P : 1], vs[BN ? P : 1];
  auto fx = [&](int v, int l) -> double& { return cs[v * C::PLANE + l * C::XL + node]; };
  auto fy = [&](int v, int l) -> double& { return cs[v * C::PLANE + C::Y0 + l * C::YL + node]; };
  auto col = [&](int v, int l) -> double& { return BN && v == 8 ? as[l * P2 + node] : fx(v, l); };
  auto u = [&](int v) -> double { return act ? un[v] : 1.0; };
  // the gradients are formed from the volume fraction's differences from the cell's
  // first value (node 0, start of the step): 0 for a constant one, whose products
  // with dudx left 1e-16 of p_g in the momenta (face fluxes of a piecewise-constant
  // state, N = 4: relative error 5.9e-16 from the fraction itself, 4.3e-16 in the
  // FP64 chain, 1.6e-16 so)
  const double aref = BN && act ? un[8 - node * V] : 1.0;
  // exponents of the x row and the y column of level l through this node
  auto exx = [&](int v, int l) -> int { return ex[(2 * v * P + l) * P + j]; };
  auto exy = [&](int v, int l) -> int { return ex[((2 * v + 1) * P + l) * P + i]; };
  const FixFactor cx(cxw), cy(cyw);
  // the fluxes of state Q at level l into the planes
  auto flux = [&](int l, const double* Q) {
    double Fx[V], Fy[V];
    if constexpr (BN) {
      Sys::template pflux<double, true>(pc, Q, Fx, Fy, pg[l], us[l], vs[l]);
      if (live) as[l * P2 + node] = Q[8] - aref;
    } else {
      Sys::template pflux<double, true>(pc, Q, Fx, Fy);
    }
    if (live) {
#pragma unroll
      for (int v = 0; v < VF; ++v) {
        fx(v, l) = Fx[v];
        fy(v, l) = Fy[v];
      }
    }
  };
  constexpr int kLevels = BN ? P : 1;  // unrolled where the NCP's scalars stay in registers
  auto fluxes = [&]() {  // of the column
#pragma unroll kLevels
    for (int l = 0; l < P; ++l) {
      double Q[V];
#pragma unroll
      for (int v = 0; v < V; ++v) Q[v] = live ? col(v, l) : 1.0;
      flux(l, Q);
    }
  };
  // gradient of the volume fraction at level l
  auto grad = [&](int l, double& ax, double& ay) {
    ax = ay = 0.0;
#pragma unroll
    for (int k = 0; k < P; ++k) {
      ax = fma(sG[i + P * k], as[l * P2 + k + P * j], ax);
      ay = fma(sG[j + P * k], as[l * P2 + i + P * k], ay);
    }
    ax *= idx;
    ay *= idy;
  };
  // dt * NCP of a level: pncp's products (0: variable 8, 1..3: variables 5..7
  // and, negated, 1..3)
  double nc[4][BN ? P : 1];
  auto ncp_level = [&](int l) {
    if constexpr (BN) {
      double ax, ay;
      grad(l, ax, ay);
      const double un_ = us[l] * ax + vs[l] * ay, p = dt * pg[l];
      nc[0][l] = dt * un_;
      nc[1][l] = p * ax;
      nc[2][l] = p * ay;
      nc[3][l] = p * un_;
    }
  };
  auto ncp = [&](int l, int v) -> double {
    const int k = v & 3;
    const double n = k == 1 ? nc[1][l] : k == 2 ? nc[2][l] : k == 3 ? nc[3][l] : nc[0][l];
    return __hiloint2double(__double2hiint(n) ^ (v < 4 ? 0x80000000 : 0), __double2loint(n));
  };
  // every line of level 0 (the first and last iterations contract one level),
  // spread over the cell's threads
  auto lines0 = [&]() {
#pragma unroll 1
    for (int q0 = live ? node : 2 * P * VF; q0 < 2 * P * VF; q0 += P2) {
      const int v = q0 / (2 * P), r = q0 - v * (2 * P), d = r / P, ln = r - d * P;
      fix_line<P, true>(cs + v * C::PLANE + (d ? C::Y0 + ln : P * ln), d ? P : 1, ex + (2 * v + d) * P2 + ln, op);
    }
  };
  // dt (dFx/dx + dFy/dy) of variable v at level l: b = value 2^-(A - 2042 - sK) for A at
  // least the exponents' maximum; |b| < 2^59
  auto divergence = [&](int v, int l, int A) -> long long {
    const long long x = fix_shift(cx.times(__double_as_longlong(fx(v, l))), A - exx(v, l) - cx.e);
    const long long y = fix_shift(cy.times(__double_as_longlong(fy(v, l))), A - exy(v, l) - cy.e);
    return x + y;
  };
  auto divergence64 = [&](int v, int l) -> double {  // the same in FP64 (rare)
    return fma(cxw, fix_value(fx(v, l), exx(v, l), op.sK), cyw * fix_value(fy(v, l), exy(v, l), op.sK));
  };
  // level 0 in FP64
  auto divergence0 = [&](int v) -> double {
    const int A = max(exx(v, 0) + cx.e, exy(v, 0) + cy.e), e = A - 2042 - op.sK;
    return e > -1000 && e < 900 ? fix_double(divergence(v, 0, A), e) : divergence64(v, 0);
  };

  // iteration 1: the state is constant in time; g = iK1 F0 = 1 exactly
  {
    double Q[V];
#pragma unroll
    for (int v = 0; v < V; ++v) Q[v] = u(v);
    flux(0, Q);
  }
  __syncthreads();
  lines0();
  if constexpr (BN) ncp_level(0);
  __syncthreads();
#pragma unroll 1
  for (int v = 0; v < (live ? V : 0); ++v) {
    double b = v < VF ? divergence0(v) : 0.0;
    if (BN && (v & 3 || v == 8)) b += ncp(0, v);
    const double u0 = u(v);
#pragma unroll
    for (int l = 0; l < P; ++l) col(v, l) = fma(-op.tsx[l], b, u0);
  }

  // iterations 2 .. P-1
#pragma unroll 1
  for (int it = 2; it < P; ++it) {
    fluxes();
    __syncthreads();
    // this thread's lines: x row j and y column j of level i, every variable
#pragma unroll 1
    for (int r = 0; r < (live ? 2 * VF : 0); ++r) {
      const int v = r >> 1, d = r & 1;
      fix_line<P, false>(cs + v * C::PLANE + (d ? C::Y0 + i * C::YL + j : i * C::XL + P * j), d ? P : 1,
                         ex + (r * P + i) * P + j, op);
    }
    if constexpr (BN) {
#pragma unroll
      for (int l = 0; l < P; ++l) ncp_level(l);
    }
    __syncthreads();
#pragma unroll 1
    for (int v = 0; v < (live ? V : 0); ++v) {
      const bool has_f = !BN || v < VF, has_n = BN && (v & 3 || v == 8);
      // common exponent of the level's contracted values (and the NCP)
      int A = 0;
      int nh[P], nl[P];
#pragma unroll
      for (int l = 0; l < P; ++l) {
        if (has_f) A = max(A, max(exx(v, l) + cx.e, exy(v, l) + cy.e));
        if (has_n) {
          const double n = ncp(l, v);
          nh[l] = __double2hiint(n);
          nl[l] = __double2loint(n);
          int e = (nh[l] >> 20) & 0x7ff;
          e = e > kFixMin ? e : kFixMin;
          A = max(A, e >= kFixMax ? kFixOut : e + 962 + op.sK);
        }
      }
      const int sc = A - 1980 - op.sT - op.sK;  // the update is W 2^sc
      const double u0 = u(v);
      const int uh = __double2hiint(u0), ul = __double2loint(u0);
      const int ue = u0 == 0.0 ? kFixMin : (uh >> 20) & 0x7ff;
      if (sc > -1000 && sc < 900 && ue >= kFixMin && ue < kFixMax) {
        int bh[P], bl[P];
        bool any = false;
#pragma unroll
        for (int l = 0; l < P; ++l) {
          long long b = has_f ? divergence(v, l, A) : 0;
          if (has_n) b += fix_int<5>(nh[l], nl[l], A - 962 - op.sK);
          bh[l] = fix_hi(b);
          bl[l] = fix_lo(b);
          any = any || b != 0;
        }
        // u itself where nothing changes it (in the unit below, which differs from
        // node to node, it may lose its last bits)
        if (!any) {
#pragma unroll
          for (int lp = 0; lp < P; ++lp) col(v, lp) = u0;
          continue;
        }
        // q = u - W 2^sc as one integer in the coarser of the two units, 2^(ue - 1083) and 2^sc
        const int unit = max(ue - 1083, sc);
        const long long U = fix_int<8>(uh, ul, unit + 1083);
        const int dw = unit - sc;
#pragma unroll
        for (int lp = 0; lp < P; ++lp) {
          FixSum<true> s(true, P);
#pragma unroll
          for (int l = 0; l < P; ++l) s.madd(bh[l], bl[l], op.Th[lp + P * l], op.Tl[lp + P * l]);
          col(v, lp) = fix_double(U - fix_shift(s.sum(), dw), unit);
        }
      } else {
        double b[P];
#pragma unroll
        for (int l = 0; l < P; ++l) {
          b[l] = has_f ? divergence64(v, l) : 0.0;
          if (has_n) b[l] += __hiloint2double(nh[l], nl[l]);
        }
#pragma unroll
        for (int lp = 0; lp < P; ++lp) {
          double s = u0;
#pragma unroll
          for (int l = 0; l < P; ++l) s = fma(-op.T[lp + P * l], b[l], s);
          col(v, lp) = s;
        }
      }
    }
    // no barrier: each thread reads only its own column before the next one
  }

  // last iteration: the time averages of the fluxes (Fh = sum_l w_l F_l), and
  // their combination H = sum_l tw_l F_l, contracted once
  fluxes();
#pragma unroll
  for (int d = 0; d < 2; ++d)
#pragma unroll
    for (int v = 0; v < VF; ++v) {
      double* p = d == 0 ? &fx(v, 0) : &fy(v, 0);  // the node's own column: no barrier
      FixLine<P> x;
      double h = 0.0;
      Fh[d][v] = 0.0;
      if (!live) continue;
      if (x.load(p, d == 0 ? C::XL : C::YL)) {
        x.limbs();
        const int e = x.E - 1020 - op.sW;
        Fh[d][v] = fix_double(x.template dot<true>(op.Wh, op.Wl, 1), e);
        h = fix_double(x.template dot<true>(op.TWh, op.TWl, 1), e);
      } else {
#pragma unroll
        for (int l = 0; l < P; ++l) {
          Fh[d][v] = fma(op.w[l], x.value(l), Fh[d][v]);
          h = fma(op.tw[l], x.value(l), h);
        }
      }
      *p = h;
    }
#pragma unroll
  for (int v = VF; v < V; ++v) Fh[0][v] = Fh[1][v] = 0.0;
  __syncthreads();
  lines0();
  __syncthreads();
#pragma unroll
  for (int v = 0; v < V; ++v) {
    qh[v] = v < VF ? u(v) - divergence0(v) : u(v);
    Sh[v] = 0.0;
  }
  if constexpr (BN) {
#pragma unroll
    for (int l = 0; l < P; ++l) {
      double ax, ay, n[9];
      grad(l, ax, ay);
      BNSys::pncp<double>(pg[l], us[l], vs[l], ax, ay, n);
      const double c = op.tw[l] * dt;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        Sh[v] = fma(-op.w[l], n[v], Sh[v]);
        qh[v] = fma(-c, n[v], qh[v]);
      }
    }
  }
  __syncthreads();
}

// Volume integral (duh; kVolume) and face extrapolation (qbnd, fbnd) of a cell
// from its time averages Q, FX, FY ([V][P2] each at cs), whose lines are spread
// over the cell's threads; ex: room for their exponents.  All threads of the
// CTA call it (one barrier); only those of active cells (act) do work.
template <class Sys, int N, bool kVolume>
__device__ __forceinline__ void outputs_fix(const BatchArgs& a, const PredOps<N, double>& op, double rdx, double rdy,
                                            double* __restrict__ cs, int* __restrict__ ex, long long cell, int node,
                                            int i, int j, const double* Sh, bool act) {
  constexpr int P = N + 1, P2 = P * P, V = Sys::V;
  double* qb = reinterpret_cast<double*>(a.qbnd);
  double* fb = reinterpret_cast<double*>(a.fbnd);
  // items: (field: 0 Q along x, 1 FX along x, 2 Q along y, 3 FY along y; line; variable)
#pragma unroll 1
  for (int it = act ? node : 4 * P * V; it < 4 * P * V; it += P2) {
    const int v = it % V, r = it / V, ln = r % P, f = r / P, d = f >> 1;
    const bool flux = f & 1;
    double* p = cs + ((flux ? 1 + d : 0) * V + v) * P2 + (d ? ln : P * ln);
    const int st = d ? P : 1;
    FixLine<P> x;
    double lo, hi;
    const bool fix = x.load(p, st);
    if (fix) {
      x.limbs();
      const int e = x.E - 1020 - op.sE;
      lo = fix_double(x.template dot<true>(op.Eh, op.El, 1), e);
      hi = fix_double(x.template dot<true>(op.Eh + P, op.El + P, 1), e);
    } else {
      lo = hi = 0.0;
#pragma unroll
      for (int k = 0; k < P; ++k) {
        lo = fma(op.FL[k], x.value(k), lo);
        hi = fma(op.FR[k], x.value(k), hi);
      }
    }
    double* o = (flux ? fb : qb) + (((size_t)cell * 4 + 2 * d) * P + ln) * V + v;  // [cell][face][point][v]
    o[0] = lo;
    o[P * V] = hi;
    if (kVolume && flux) {
      if (fix) {
#pragma unroll
        for (int k = 0; k < P; ++k) p[k * st] = __longlong_as_double(x.template dot<true>(op.Kh + k, op.Kl + k, P));
      } else {
#pragma unroll 1
        for (int k = 0; k < P; ++k) {
          double s = 0.0;
#pragma unroll
          for (int m = 0; m < P; ++m) s = fma(op.Kxi[k + P * m], x.value(m), s);
          p[k * st] = s;
        }
      }
      ex[(d * V + v) * P + ln] = fix ? x.E : kFixOut;
    }
  }
  if constexpr (kVolume) {
    __syncthreads();
    if (act) {
      // duh = (w_j/dx) sum_k Kxi(i,k) Fhi_x(k,j) + (w_i/dy) sum_k Kxi(j,k) Fhi_y(i,k) [+ w_i w_j Shi]
      const double vx = op.w[j] * rdx, vy = op.w[i] * rdy;
      double* dst = a.duh + ((size_t)cell * P2 + node) * V;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const double bx = cs[(V + v) * P2 + node], by = cs[(2 * V + v) * P2 + node];
        const int ex_ = ex[v * P + j], ey_ = ex[(V + v) * P + i];
        const double sx = ex_ == kFixOut ? bx : fix_double(__double_as_longlong(bx), ex_ - 1020 - op.sK);
        const double sy = ey_ == kFixOut ? by : fix_double(__double_as_longlong(by), ey_ - 1020 - op.sK);
        double s = sx * vx + sy * vy;
        if constexpr (Sys::ID == kSysBN) s = fma(op.w[i] * op.w[j], Sh[v], s);
        dst[v] = s;
      }
    }
  }
}

}  // namespace aderdg
