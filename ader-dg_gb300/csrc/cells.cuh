// cells.cuh -- K3: surface integral + element update + DMP / positivity
// detection + CFL partials, one thread per spatial node, CPB cells per CTA.
//
// Reference: surface_integral.f90:8-39, element_update.f90:8-30, the DMP of
// Euler/limiter.f90:179-245 (called from Euler/main.f90:74-88), the per-cell
// part of get_min_max (Euler/limiter.f90:115-143) for the next step, and the
// node loop of calc_time_step.f90.  Compiled with --fmad=false: the phase API's
// values follow the reference's FP64 operation order; the fused step's variants
// (kFast) name their fused multiply-adds.
//
// Modes (BatchArgs::mode):
//   kCellFused   surface + update + [DMP, next min/max] + CFL partials
//   kCellSurface surface integral only (phase API)
//   kCellUpdate  update + [DMP, next min/max] + CFL partials (phase API)
//   kCellPrime   min/max of the current state for the DMP neighbourhood
//                (get_min_max step 1) + CFL denominators; no update
//   kCellInitDmp initial limiter: DMP with argmax 0.1 against the cell's own
//                nodal min/max; failing cells take the initial subcell data
//   kCellCfl     CFL denominators of the current state only
//   kCellPrimeLimited  kCellPrime for the limited cells only (their min/max
//                come from Lh), no CFL: after the initial limiter, where the
//                other cells' min/max and the CFL are those of kCellPrime
#pragma once

#include <type_traits>

#include "common.cuh"
#include "faces.cuh"
#include "physics.cuh"

namespace aderdg {

#define kInf __longlong_as_double(0x7ff0000000000000LL)

// Doubles mapped to integers of the same order (negative values have their
// magnitude bits flipped), so min/max run on the integer pipe instead of the
// FP64 pipe; the value returned is one of the inputs, as with fmin/fmax.
__device__ __forceinline__ long long okey(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double okey_inv(long long k) {
  return __longlong_as_double(k >= 0 ? k : (k ^ 0x7fffffffffffffffLL));
}

// Subcell / Gauss-Lobatto projections of one cell (get_subcell_data and
// get_lobatto_data, Euler/limiter.f90:12-68), sum-factorised y then x with
// the reference's summation order.  A "team" of nr threads with rank r works
// on one cell; the caller synchronises between the two passes.  The operators
// come from shared memory: lim = uh2lim (s,k) at [s + S*k], lob = uh2lob (q,k)
// at [q + P*k].  T = double: exact-order mul then add, or one fused
// multiply-add per term (kFast); T = float: fused multiply-adds (the FP32 modes).
template <int N, int V, class T>
struct Proj {
  static constexpr int P = N + 1, P2 = P * P, S = 2 * N + 1;
  template <bool kFast>
  __device__ __forceinline__ static T madd(T acc, T a, T b) {
    if constexpr (kFast) return fma(a, b, acc);
    // reference order: a rounded product, then a rounded sum, also in the
    // translation units compiled with fused multiply-adds
    else if constexpr (sizeof(T) == 8) return __dadd_rn(acc, __dmul_rn(a, b));
    else return acc + a * b;
  }
  // T = float: U, LY and LB hold items of V values, four to a float4 in a plane
  // of its own, the rest one to a plane (bases on 16 bytes): a load or store per
  // four values, where one word each made the passes wait on shared memory.
  // Rows of LY and LB are PS = P | 1 items apart, which leaves no bank conflict.
  static constexpr int PS = P | 1, NU = P2, NLY = S * PS, NLB = P * PS;
  static constexpr int UF = (V * NU + 3) / 4 * 4, LYF = (V * NLY + 3) / 4 * 4, LBF = (V * NLB + 3) / 4 * 4;
  template <int n>
  __device__ __forceinline__ static void ld(const float* b, int item, float* o) {
#pragma unroll
    for (int q = 0; q < V / 4; ++q) load_v<4>(b + 4 * (q * n + item), o + 4 * q);
#pragma unroll
    for (int v = V / 4 * 4; v < V; ++v) o[v] = b[v * n + item];
  }
  template <int n>
  __device__ __forceinline__ static void st(float* b, int item, const float* x) {
#pragma unroll
    for (int q = 0; q < V / 4; ++q) store_v<4>(b + 4 * (q * n + item), x + 4 * q);
#pragma unroll
    for (int v = V / 4 * 4; v < V; ++v) b[v * n + item] = x[v];
  }
  // y pass: LY[v][s][i] = sum_k U[v][i + P k] uh2lim(s,k); LB[v][s][i] likewise with uh2lob
  template <bool kFast = false>
  __device__ static void ypass(const T* U, T* LY, T* LB, const T* lim, const T* lob, int r, int nr) {
    if constexpr (sizeof(T) == 4) {
      for (int idx = r; idx < P * (S + P); idx += nr) {
        const int ii = idx % P, s = idx / P;
        float acc[V];
#pragma unroll
        for (int v = 0; v < V; ++v) acc[v] = 0.0f;
#pragma unroll
        for (int k = 0; k < P; ++k) {
          const float c = s < S ? lim[s + S * k] : lob[s - S + P * k];
          float x[V];
          ld<NU>(U, ii + P * k, x);
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] = fmaf(x[v], c, acc[v]);
        }
        if (s < S) st<NLY>(LY, s * PS + ii, acc);
        else st<NLB>(LB, (s - S) * PS + ii, acc);
      }
    } else {
      for (int idx = r; idx < P * S; idx += nr) {
        const int ii = idx % P, s = idx / P;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          T acc = 0;
#pragma unroll
          for (int k = 0; k < P; ++k) acc = madd<kFast>(acc, U[v * P2 + ii + P * k], lim[s + S * k]);
          LY[(v * S + s) * P + ii] = acc;
        }
      }
      for (int idx = r; idx < P * P; idx += nr) {
        const int ii = idx % P, s = idx / P;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          T acc = 0;
#pragma unroll
          for (int k = 0; k < P; ++k) acc = madd<kFast>(acc, U[v * P2 + ii + P * k], lob[s + P * k]);
          LB[(v * P + s) * P + ii] = acc;
        }
      }
    }
  }
  // T = float: sum over k of item (s2, k) times c[k * stride]
  template <int n>
  __device__ __forceinline__ static void row(const float* L, const float* c, int stride, int s2, float* out) {
#pragma unroll
    for (int v = 0; v < V; ++v) out[v] = 0.0f;
#pragma unroll
    for (int k = 0; k < P; ++k) {
      const float ck = c[stride * k];
      float x[V];
      ld<n>(L, s2 * PS + k, x);
#pragma unroll
      for (int v = 0; v < V; ++v) out[v] = fmaf(x[v], ck, out[v]);
    }
  }
  // subcell value (s1, s2) from the y pass
  template <bool kFast = false>
  __device__ static void subcell(const T* LY, const T* lim, int s1, int s2, T* out) {
    if constexpr (sizeof(T) == 4) {
      row<NLY>(LY, lim + s1, S, s2, out);
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        T acc = 0;
#pragma unroll
        for (int k = 0; k < P; ++k) acc = madd<kFast>(acc, LY[(v * S + s2) * P + k], lim[s1 + S * k]);
        out[v] = acc;
      }
    }
  }
  template <bool kFast = false>
  __device__ static void lobatto(const T* LB, const T* lob, int s1, int s2, T* out) {
    if constexpr (sizeof(T) == 4) {
      row<NLB>(LB, lob + s1, P, s2, out);
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        T acc = 0;
#pragma unroll
        for (int k = 0; k < P; ++k) acc = madd<kFast>(acc, LB[(v * P + s2) * P + k], lob[s1 + P * k]);
        out[v] = acc;
      }
    }
  }
  // x pass fused with min/max (integer keys) and the positivity test of every subcell (FP64)
  template <class Sys, bool kFast = false>
  __device__ static void xpass_minmax(const T* U, const T* LY, const T* LB, const T* lim, const T* lob,
                                      const Phys& ph, int r, int nr, T* mn, T* mx, bool& posfail) {
    T val[V];
    long long kmn[V], kmx[V];
#pragma unroll
    for (int v = 0; v < V; ++v) { kmn[v] = okey(mn[v]); kmx[v] = okey(mx[v]); }
    for (int idx = r; idx < S * S; idx += nr) {
      subcell<kFast>(LY, lim, idx % S, idx / S, val);
#pragma unroll
      for (int v = 0; v < V; ++v) { const long long k = okey(val[v]); kmn[v] = min(kmn[v], k); kmx[v] = max(kmx[v], k); }
      if constexpr (Sys::ID != kSysAD) {
        if (!Sys::positive_fast(ph, val)) posfail = true;
      }
    }
    for (int idx = r; idx < P * P; idx += nr) {
      lobatto<kFast>(LB, lob, idx % P, idx / P, val);
#pragma unroll
      for (int v = 0; v < V; ++v) { const long long k = okey(val[v]); kmn[v] = min(kmn[v], k); kmx[v] = max(kmx[v], k); }
    }
    for (int idx = r; idx < P2; idx += nr) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const long long k = okey(U[v * P2 + idx]);
        kmn[v] = min(kmn[v], k);
        kmx[v] = max(kmx[v], k);
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) { mn[v] = okey_inv(kmn[v]); mx[v] = okey_inv(kmx[v]); }
  }
  // FP32 x pass fused with min/max and the admissibility test.  The y pass
  // ran on the deviations d = uh - ubar from a reference state ubar of the
  // cell (the projections reproduce constants, so proj(uh) = ubar + proj(d));
  // min/max are of the projected deviations.  A subcell whose FP32 value
  // ubar + proj(d) is not clearly admissible (err = the error bound of
  // proj(d), plus the rounding of ubar to FP32) is projected again in FP64
  // from U64, in the reference's order (y pass, then x), and tested exactly:
  // the value and the decision are those of the FP64 path bit for bit.
  template <class Sys>
  __device__ static void xpass_minmax_f32(const float* LY, const float* LB, const float* lim, const float* lob,
                                          const double* U64, const double* lim64,
                                          const typename Sys::FConst& fc, const float* err, const float* ubf,
                                          const Phys& ph, int r, int nr, float* mn, float* mx, bool& posfail) {
    float val[V], q[V], e[V];
#pragma unroll
    for (int v = 0; v < V; ++v) e[v] = err[v] + 2.5e-7f * fabsf(ubf[v]);
    unsigned open = 0u;  // bit it: the it-th subcell of this thread needs the FP64 test
    int it = 0;
    for (int idx = r; idx < S * S; idx += nr, ++it) {
      subcell<true>(LY, lim, idx % S, idx / S, val);
#pragma unroll
      for (int v = 0; v < V; ++v) { mn[v] = fminf(mn[v], val[v]); mx[v] = fmaxf(mx[v], val[v]); }
      if constexpr (Sys::ID != kSysAD) {
#pragma unroll
        for (int v = 0; v < V; ++v) q[v] = ubf[v] + val[v];
        if (!Sys::admissible_box_f32(fc, q, e)) open |= 1u << it;
      }
    }
    for (int idx = r; idx < P * P; idx += nr) {
      lobatto<true>(LB, lob, idx % P, idx / P, val);
#pragma unroll
      for (int v = 0; v < V; ++v) { mn[v] = fminf(mn[v], val[v]); mx[v] = fmaxf(mx[v], val[v]); }
    }
    if constexpr (Sys::ID != kSysAD)
      while (open) {
        const int idx = r + (__ffs(open) - 1) * nr;
        open &= open - 1u;
        if (!positive64<Sys>(U64, lim64, ph, idx % S, idx / S)) posfail = true;
      }
  }
  // a subcell left open, in FP64 in the reference's order (the y pass of
  // get_subcell_data, then x; lim64 = uh2lim (s,k) at [s + S*k]): the FP64 path's
  // value and decision bit for bit
  template <class Sys>
  __device__ static bool positive64(const double* U64, const double* lim64, const Phys& ph, int s1, int s2) {
    double qd[V];
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
      double acc = 0.0;
#pragma unroll 1
      for (int k = 0; k < P; ++k) {
        double ly = 0.0;
        for (int m = 0; m < P; ++m) ly = __dadd_rn(ly, __dmul_rn(U64[v * P2 + k + P * m], lim64[s2 + S * m]));
        acc = __dadd_rn(acc, __dmul_rn(ly, lim64[s1 + S * k]));
      }
      qd[v] = acc;
    }
    return Sys::positive(ph, qd);
  }
  // The FP32 passes of a team of P2 threads (the cell kernel), each thread
  // taking several outputs that share operands: the y pass column ii = r % P
  // and the outputs r / P, + P, .. of the S subcell and P Lobatto rows; the x
  // pass row s2 and a chunk of its subcells.  One output at a time read 2P (V +
  // 1) shared-memory words for every V P products, and the kernel waited on
  // them.  Same sums in the same order.
  __device__ static void ypass_team(const float* U, float* LY, float* LB, const float* lim, const float* lob, int r) {
    constexpr int NO = (S + P + P - 1) / P;  // outputs of a thread
    const int ii = r % P, o0 = r / P;
    float c[NO][P];
#pragma unroll
    for (int q = 0; q < NO; ++q) {
      const int o = o0 + q * P;
#pragma unroll
      for (int k = 0; k < P; ++k) c[q][k] = o < S ? lim[o + S * k] : o < S + P ? lob[o - S + P * k] : 0.0f;
    }
    float x[P][V];
#pragma unroll
    for (int k = 0; k < P; ++k) ld<NU>(U, ii + P * k, x[k]);
#pragma unroll
    for (int q = 0; q < NO; ++q) {
      const int o = o0 + q * P;
      float acc[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        acc[v] = 0.0f;
#pragma unroll
        for (int k = 0; k < P; ++k) acc[v] = fmaf(x[k][v], c[q][k], acc[v]);
      }
      if (o < S) st<NLY>(LY, o * PS + ii, acc);
      else if (o < S + P) st<NLB>(LB, (o - S) * PS + ii, acc);
    }
  }
  template <class Sys>
  __device__ static void xpass_team(const float* LY, const float* LB, const float* lim, const float* lob,
                                    const double* U64, const double* lim64, const typename Sys::FConst& fc,
                                    const float* err, const float* ubf, const Phys& ph, int r, float* mn, float* mx,
                                    bool& posfail) {
    constexpr int C = P2 / S;             // chunks of a row
    constexpr int CH = (S + C - 1) / C;   // subcells of a chunk
    float val[V];
    if (r < C * S) {
      const int s2 = r / C, c0 = r - s2 * C;
      float e[V], ly[P][V];
#pragma unroll
      for (int v = 0; v < V; ++v) e[v] = err[v] + 2.5e-7f * fabsf(ubf[v]);
#pragma unroll
      for (int k = 0; k < P; ++k) ld<NLY>(LY, s2 * PS + k, ly[k]);
      unsigned open = 0u;  // bit q: the chunk's q-th subcell needs the FP64 test
#pragma unroll 1
      for (int q = 0; q < CH; ++q) {
        const int s1 = c0 + q * C;
        if (s1 >= S) break;
        float c[P], qv[V];
#pragma unroll
        for (int k = 0; k < P; ++k) c[k] = lim[s1 + S * k];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          float acc = 0.0f;
#pragma unroll
          for (int k = 0; k < P; ++k) acc = fmaf(ly[k][v], c[k], acc);
          mn[v] = fminf(mn[v], acc);
          mx[v] = fmaxf(mx[v], acc);
          qv[v] = ubf[v] + acc;
        }
        if constexpr (Sys::ID != kSysAD)
          if (!Sys::admissible_box_f32(fc, qv, e)) open |= 1u << q;
      }
      if constexpr (Sys::ID != kSysAD)
        while (open) {
          const int q = __ffs(open) - 1;
          open &= open - 1u;
          if (!positive64<Sys>(U64, lim64, ph, c0 + q * C, s2)) posfail = true;
        }
    }
    lobatto<true>(LB, lob, r % P, r / P, val);
#pragma unroll
    for (int v = 0; v < V; ++v) { mn[v] = fminf(mn[v], val[v]); mx[v] = fmaxf(mx[v], val[v]); }
  }
};

// Voronoi neighbour index along one axis (Euler/initialize.f90:219-258):
// periodic sides wrap, all others clamp.
__device__ __forceinline__ int nb_index(int x, int d, int n, int bc_lo, int bc_hi) {
  int y = x + d;
  if (y < 0) y = (bc_lo == 3) ? n - 1 : 0;
  if (y > n - 1) y = (bc_hi == 3) ? 0 : n - 1;
  return y;
}

// a / b, correctly rounded, for a constant b with y = 1/b correctly rounded
// (Markstein: a faithful quotient plus one exact-remainder correction is the
// rounded quotient; the first step makes it faithful): 5 FP64 instructions in
// place of the division's sequence.  Outside 2^-700 .. 2^700, where the
// remainders could leave the normal range, the division itself.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const unsigned e = ((unsigned)__double2hiint(a) >> 20) & 0x7ff;
  if (e - 323u >= 1400u && a != 0.0) return a / b;
  const double q0 = __dmul_rn(a, y);
  const double q1 = __fma_rn(__fma_rn(-q0, b, a), y, q0);
  return __fma_rn(__fma_rn(-q1, b, a), y, q1);
}

// CFL denominator at one node (calc_time_step.f90: Euler/BN :31-45, AD :37-50)
template <class Sys, int N>
__device__ __forceinline__ double cfl_denom(const InstDesc& in, const double* Q) {
  if constexpr (Sys::ID == kSysAD) {
    // (|c_x| + 2 a (2N+1)/dx)/dx + (|c_y| + 2 a (2N+1)/dy)/dy, the same at every
    // node: formed on the host in this order
    return in.ad_denom;
  } else {
    double ex, ey;
    Sys::max_eig2(in.ph, Q, ex, ey);
    double denom = 0.0;
    denom = denom + ex / in.dx;
    denom = denom + ey / in.dy;
    return denom;
  }
}
// out of line, for kernels whose registers it would raise (the priming pass of the
// FP64 fused step's kernel)
template <class Sys, int N>
static __device__ __noinline__ double cfl_denom_call(const InstDesc& in, const double* Q) {
  return cfl_denom<Sys, N>(in, Q);
}
// FP64 fused step: bounds on a node's denominator from FP32 (hi in the upper half,
// lo in the lower: the maximum of keys is that of hi).  The time step is the
// reference's, bit for bit, from the one maximum over all nodes, so that nearly
// all nodes need no FP64 evaluation: k_cfl evaluates the cells whose hi reaches the
// largest lo, and restarts, host steps and the phase API's calc_time_step give the
// time steps of an uninterrupted run.
template <class Sys>
__device__ __forceinline__ unsigned long long cfl_key(const InstDesc& in, const float* q) {
  float lo, hi;
  Sys::cfl_bounds(typename Sys::FConst(in.ph), q, in.idxf, in.idyf, lo, hi);
  return (unsigned long long)__float_as_uint(hi) << 32 | __float_as_uint(lo);
}

// FP32-mixed: eigenvalues and the node's denominator in FP32 (the maximum
// over nodes, and dt, in FP64); states whose FP32 pressure is not settled
// take the FP64 evaluation on Qd
template <class Sys, int N>
__device__ __forceinline__ double cfl_denom_f32(const InstDesc& in, const typename Sys::FConst& fc, const float* q,
                                                const double* Qd) {
  if constexpr (Sys::ID == kSysAD) {
    return cfl_denom<Sys, N>(in, nullptr);
  } else {
    float ex, ey;
    if (Sys::max_eig2_f32(fc, q, ex, ey)) return (double)(ex * in.idxf + ey * in.idyf);
    return cfl_denom<Sys, N>(in, Qd);
  }
}

// Maximum over the P2 lanes of a cell when every cell is an aligned segment
// of a warp (P2 = 4 or 16): xor shuffles within the segment; every lane of the
// warp must call it.
template <int P2>
__device__ __forceinline__ unsigned seg_max(unsigned x) {
#pragma unroll
  for (int o = P2 / 2; o > 0; o >>= 1) {
    const unsigned y = __shfl_xor_sync(0xffffffffu, x, o, P2);
    x = x > y ? x : y;
  }
  return x;
}
template <int P2>
__device__ __forceinline__ unsigned long long seg_max(unsigned long long x) {
#pragma unroll
  for (int o = P2 / 2; o > 0; o >>= 1) {
    const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o, P2);
    x = x > y ? x : y;
  }
  return x;
}

// VAR: the CTA size the tuner (aderdg/tuner.py) picks for the FP32 modes: 0
// the default below, 1 twice, 2 half of it
constexpr int kCellVariants = 3;
template <class Sys, int N, int VAR = 0>
struct CellCfg {
  static constexpr int P = N + 1, P2 = P * P, S = 2 * N + 1, V = Sys::V;
  // small CTAs (the kernel waits on latency and barriers: smaller CTAs, more
  // of them per SM, wait on fewer warps per barrier): 64 threads up to N = 3,
  // 128 at N = 4 and 256 at N = 5, where the 25- and 36-thread cells fill
  // smaller CTAs badly (measured: BN cylinder 0.559 -> 0.508 -> 0.487 ms,
  // Riemann problem 0.344 -> 0.330 -> 0.324 ms for 256 -> 128 -> 64 threads)
  static constexpr int CTA0 = N == 5 ? 256 : N == 4 ? 128 : 64;
  static constexpr int CTA = VAR == 1 ? 2 * CTA0 : VAR == 2 ? (CTA0 / 2 < 32 ? 32 : CTA0 / 2) : CTA0;
  static constexpr int CPB = (CTA / P2) < 1 ? 1 : (CTA / P2);
  static constexpr int THREADS = ((CPB * P2 + 31) / 32) * 32;
  // per cell: U [V][P2], LY [V][S][P], LB [V][P][P], red [2][V][P2] (FP64);
  // the FP32 projections: U64 [V][P2] then FP32 U, LY, LB (Proj's items) and red
  // [P2][2 V] in the same room, every part on 16 bytes.  Cells of a warp
  // segment start 64 bytes apart modulo the banks' 128, so that the segments'
  // accesses do not meet.
  using PF = Proj<N, V, float>;
  static constexpr int U_DBL = (V * P2 + 1) / 2 * 2, RED_F = U_DBL * 2 + PF::UF + PF::LYF + PF::LBF;
  static constexpr int CELL_RAW = U_DBL + V * S * P + V * P * P + 2 * V * P2;
  static constexpr int CELL_DBL = P2 == 16 ? (CELL_RAW + 7) / 16 * 16 + 8 : (CELL_RAW + 1) / 2 * 2;
  static_assert(CELL_DBL >= CELL_RAW && 4 * (RED_F + 2 * V * P2) <= 8 * CELL_DBL, "FP32 cell layout");
  static constexpr int OPS_DBL = S * P + P * P;  // uh2lim, uh2lob (FP64, then FP32 in the FP32 modes)
  static constexpr int SMEM_BYTES = CPB * CELL_DBL * 8 + OPS_DBL * 12 + CPB * 8 /*cell max*/ + CPB * 4 /*flags*/ +
                                    CPB * V * 4 /*|U| max*/ + CPB * V * 4 /*FP32 reference state*/ +
                                    CPB * 4 /*instances*/ + 16;
  // The DMP comparisons, (cell, variable) pairs on consecutive threads, so that
  // they fill whole warps (with the pairs of a cell on its own first V threads
  // every warp issued the comparison's FP64 instructions for a few lanes: 2.5 of
  // 6.8 FP64 slots per DOF).  Euler, whose pairs leave lanes of a warp idle: the
  // minimum and the maximum of a pair on neighbouring lanes (LPP = 2), which
  // halves the serial part between barriers: N = 3 313 -> 281 us (Riemann problem
  // 512^2), N = 4 144 -> 138 us, N = 5 291 -> 271 us; Baer-Nunziato's fill them:
  // 410 -> 455 us (cylinder N = 3 400^2), so LPP = 1.
  static constexpr int LPP = Sys::ID == kSysBN ? 1 : 2;          // lanes of a pair
  static constexpr int SPL = 2 / LPP;                            // sides of a lane
  static constexpr int NITEM = (LPP * CPB * V + THREADS - 1) / THREADS;
  // blocks per SM the register allocation aims at, in 256-thread units:
  // Euler's FP32-mixed cell kernel is latency-bound and gains from a fourth;
  // the other variants keep the allocation they reach unconstrained
  static constexpr int min_blocks(bool fast) {
    return (Sys::ID == kSysEuler ? (fast ? 4 : 3) : (Sys::ID == kSysBN ? 2 : 4)) * 256 / CTA < 1
               ? 1
               : (Sys::ID == kSysEuler ? (fast ? 4 : 3) : (Sys::ID == kSysBN ? 2 : 4)) * 256 / CTA;
  }
};

// the operators of a cell-kernel variant: 1/(w_i w_j) in FP64 for the FP64 updates
template <int N, bool kFast, bool kExact>
using CellOps = typename std::conditional<kExact || !kFast, ExactOps<N>, DevOps<N, double>>::type;

// kFast: DMP projections in FP32 with an error bound (settled from FP64 where
// the bound leaves a decision open) and, without kExact, the FP32 modes'
// storage and surface integral.  kExact: FP64 storage, surface integral and update
// beside those projections: the FP64 mode's fused step, whose decisions are those of
// the FP64 projections of its state.  Its surface integral and update are fused
// multiply-adds (7 roundings a value in place of 12; the FP64 pipe bounds the kernel:
// 365 -> 255 us on the Euler vortex N = 4 256^2, 345 -> 248 us on Baer-Nunziato N = 3
// 200^2), its CFL denominators FP32 bounds (cfl_key: 255 -> 196 and 248 -> 198 us); the
// phase API keeps the reference's order.
template <class Sys, int N, bool kFast, int VAR = 0, bool kExact = false>
__global__ void __launch_bounds__(CellCfg<Sys, N, VAR>::THREADS, CellCfg<Sys, N, VAR>::min_blocks(kFast && !kExact))
    k_cells(BatchArgs a, CellOps<N, kFast, kExact> op) {
  using C = CellCfg<Sys, N, VAR>;
  constexpr int P = N + 1, P2 = P * P, S = 2 * N + 1, V = Sys::V, CPB = C::CPB;
  constexpr bool kF32 = kFast && !kExact;  // FP32 storage and update
  // the team passes where they are faster (measured): Euler N = 3, 344 -> 328 us
  // on the Riemann problem 512^2; at N = 4 their chunks leave a quarter of the
  // lanes idle (156 -> 170 us on the vortex), at N = 5 and 2 they cost 7% and 6%.
  // Baer-Nunziato N = 3 gains 2% on the 400^2 cylinder, but a chunk's subcells
  // that need the FP64 test follow one another on one thread: 92 -> 137 us on a
  // 281 x 103 cylinder in its first steps
  constexpr bool kTeam = P == 4 && V == 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* opsm = sm + CPB * C::CELL_DBL;
  float* opsf = reinterpret_cast<float*>(opsm + C::OPS_DBL);
  unsigned long long* cmax = reinterpret_cast<unsigned long long*>(opsf + C::OPS_DBL + (C::OPS_DBL & 1));
  int* cflag = reinterpret_cast<int*>(cmax + CPB);
  unsigned* amax_all = reinterpret_cast<unsigned*>(cflag + CPB);  // [CPB][V]
  float* ubs_all = reinterpret_cast<float*>(amax_all + CPB * V);  // [CPB][V]
  int* cinst = reinterpret_cast<int*>(ubs_all + CPB * V);  // instance of each active cell, else -1

  const int mode = a.mode;
  const int t = threadIdx.x;
  const int lc = t / P2;
  const int node = t - lc * P2;
  const int i = node % P, j = node / P;
  const long long cell = a.cell0 + (long long)blockIdx.x * CPB + lc;
  const bool in_cta = lc < CPB;
  const int k_found = (in_cta && cell < a.ncells) ? find_inst_cell(a.inst, a.ninst, cell) : -1;
  const bool valid = k_found >= 0;
  const int kc = valid ? k_found : 0;
  const InstDesc& in = a.inst[kc];
  const InstState& st = a.st[kc];
  const bool priming = mode == kCellPrime || mode == kCellInitDmp || mode == kCellCfl || mode == kCellPrimeLimited;
  const bool act = valid && (priming ? (a.only_inst < 0 || kc == a.only_inst) : st.active != 0) &&
                   (mode != kCellPrimeLimited || a.status[parity(st)][cell] != 0);
  if (in_cta && node == 0) cinst[lc] = act ? kc : -1;
  if (!__syncthreads_or(act)) return;  // nothing to do in this CTA
  const int par = parity(st);
  const long long lcell = cell - in.cell_base;
  const int ci = valid ? (int)((unsigned)lcell % (unsigned)in.imax) : 0, cj = valid ? (int)((unsigned)lcell / (unsigned)in.imax) : 0;
  const bool limiter = Sys::ID != kSysAD && a.mm[0] != nullptr;
  double* U = sm + (size_t)(in_cta ? lc : 0) * C::CELL_DBL;
  double* LY = U + C::U_DBL;
  double* LB = LY + V * S * P;
  double* RED = LB + V * P * P;
  // FP32 views of the same room
  using PF = typename C::PF;
  float* Uf = reinterpret_cast<float*>(U + C::U_DBL);
  float* LYf = Uf + PF::UF;
  float* LBf = LYf + PF::LYF;
  float* REDf = LBf + PF::LBF;
  unsigned* amax = amax_all + (in_cta ? lc : 0) * V;
  float* ubs = ubs_all + (in_cta ? lc : 0) * V;

  // DMP neighbourhood bounds (get_min_max step 2, Euler/limiter.f90:147-167): the
  // threads of a (cell, variable) pair fold the minimum (side 0) and the maximum
  // (side 1) over the cell's 3x3 Voronoi neighbourhood now, so the global loads
  // overlap the update and the projections
  constexpr int LPP = C::LPP, SPL = C::SPL;
  double nbound[C::NITEM][SPL];
  float nen[C::NITEM];  // largest error bound of the folded min/max
  if (limiter && (mode == kCellFused || mode == kCellUpdate)) {
#pragma unroll
    for (int q = 0; q < C::NITEM; ++q) {
      const int it = t + q * C::THREADS, pr = it / LPP, lc2 = pr / V, v = pr - lc2 * V;
#pragma unroll
      for (int s = 0; s < SPL; ++s) nbound[q][s] = 0.0;
      nen[q] = 0.0f;
      const int k2 = pr < CPB * V ? cinst[lc2] : -1;
      if (k2 < 0) continue;
      const InstDesc& in2 = a.inst[k2];
      const int par2 = parity(a.st[k2]);
      const long long cell2 = a.cell0 + (long long)blockIdx.x * CPB + lc2;
      const unsigned l2 = (unsigned)(cell2 - in2.cell_base);  // an instance has below 2^31 cells
      const int ci2 = (int)(l2 % (unsigned)in2.imax), cj2 = (int)(l2 / (unsigned)in2.imax);
      const int side0 = LPP == 2 ? it & 1 : 0;
      const double* mmi = a.mm[par2] + side0 * V + v;
      const float* mei = a.mme[par2];
      // the maximum as the minimum of the negated values (fast kernels: of the
      // complemented integer keys, on the integer pipe, not FP64; FP64: a NaN is
      // the largest key on either side, left out as fmin and fmax leave it out)
      auto key = [](double x, long long flip) -> long long {
        if (kExact && is_nan_bits(x)) return 0x7fffffffffffffffLL;
        return okey(x) ^ flip;
      };
      double b[SPL];
      long long kb[SPL], kx[SPL];
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        kx[s] = -(long long)(side0 + s);
        const double x = mmi[(size_t)cell2 * 2 * V + s * V];
        b[s] = kx[s] ? -x : x;
        kb[s] = key(x, kx[s]);
      }
      float en = 0.0f;
#pragma unroll
      for (int jj = -1; jj <= 1; ++jj)
#pragma unroll
        for (int ii = -1; ii <= 1; ++ii) {
          const int in_ = nb_index(ci2, ii, in2.imax, in2.bc[0], in2.bc[1]);
          const int jn_ = nb_index(cj2, jj, in2.jmax, in2.bc[2], in2.bc[3]);
          const long long nc = in2.cell_base + in_ + (long long)in2.imax * jn_;
#pragma unroll
          for (int s = 0; s < SPL; ++s) {
            const double x = mmi[(size_t)nc * 2 * V + s * V];
            if constexpr (kFast) kb[s] = min(kb[s], key(x, kx[s]));
            else b[s] = fmin(b[s], kx[s] ? -x : x);
          }
          if (mei) en = fmaxf(en, mei[(size_t)nc * V + v]);
        }
#pragma unroll
      for (int s = 0; s < SPL; ++s) nbound[q][s] = kFast ? okey_inv(kb[s] ^ kx[s]) : (kx[s] ? -b[s] : b[s]);
      nen[q] = en;
    }
  }

  // projection operators into shared memory (lanes index them by subcell)
  if constexpr (Sys::ID != kSysAD) for (int k = t; k < C::OPS_DBL; k += C::THREADS) {
    opsm[k] = k < S * P ? op.uh2lim[k] : op.uh2lob[k - S * P];
    if constexpr (kFast) opsf[k] = k < S * P ? op.uh2limf[k] : op.uh2lobf[k - S * P];
  }
  if (in_cta && node == 0) {
    cmax[lc] = 0ull;
    cflag[lc] = 0;
  }
  if constexpr (kFast && Sys::ID != kSysAD) {
    // a cell's FP32 reference state ubar: its start-of-step state at node 0, rounded to FP32
    for (int pr = t; pr < CPB * V; pr += C::THREADS) {
      const int lc2 = pr / V, v = pr - lc2 * V, k2 = cinst[lc2];
      const long long cell2 = a.cell0 + (long long)blockIdx.x * CPB + lc2;
      amax_all[pr] = 0u;
      ubs_all[pr] = k2 >= 0 ? (float)a.uh[parity(a.st[k2])][(size_t)cell2 * P2 * V + v] : 0.0f;
    }
  }
  __syncthreads();

  // ---------------------------------------------------------------- update
  double u[V];
  const size_t off = ((size_t)(valid ? cell : 0) * P2 + node) * V;
  // Advection-diffusion, fused step on small grids (faces_in_cells): the cell's
  // face fluxes [4][P] from the predictor's face states; a cell stores those of its
  // left and bottom faces, the last ones of a row or column also the others
  using FR_ = typename std::conditional<kF32, float, double>::type;
  FR_* sF = reinterpret_cast<FR_*>(U);
  const bool own_faces = Sys::ID == kSysAD && mode == kCellFused && faces_in_cells(a, P2, kF32);
  if constexpr (Sys::ID == kSysAD) {
    if (own_faces) {
      if (act) {
        for (int idx = node; idx < 4 * P; idx += P2) {
          const int f = idx / P, l = idx - f * P, fi = ci + (f == 1), fj = cj + (f == 3);
          const bool xdir = f < 2;
          const FR_ x = ad_face_flux<FR_, FR_>(a, in, in.ad_pi, op.xid[l], xdir, fi, fj, l, P);
          sF[idx] = x;
          if (f == 0 || f == 2 || (f == 1 ? fi == in.imax : fj == in.jmax)) {
            const long long face = xdir ? in.fx_base + fi + (long long)(in.imax + 1) * fj : in.fy_base + fi + (long long)in.imax * fj;
            reinterpret_cast<FR_*>(xdir ? a.fu : a.gu)[(size_t)face * P + l] = x;
          }
        }
      }
      __syncthreads();
    }
  }
  if (act) {
    if (mode == kCellFused || mode == kCellSurface || mode == kCellUpdate) {
      const long long fxl = in.fx_base + ci + (long long)(in.imax + 1) * cj;
      const long long fyb = in.fy_base + ci + (long long)in.imax * cj;
      const long long fyt = fyb + in.imax;
      if constexpr (kF32) {
        // FP32-mixed: duh and the face fluxes are stored in FP32; the surface
        // contraction and the scaling by 1/(w_i w_j) in FP32, the update of
        // the FP64 state in FP64
        const float* D32 = reinterpret_cast<const float*>(a.duh);
        const float* XL = reinterpret_cast<const float*>(a.fu);
        const float* XR = reinterpret_cast<const float*>((Sys::ID == kSysBN) ? a.fp : a.fu);
        const float* YB = reinterpret_cast<const float*>(a.gu);
        const float* YT = reinterpret_cast<const float*>((Sys::ID == kSysBN) ? a.gp : a.gu);
        float d[V];
        load_v<V>(D32 + off, d);
        if (mode != kCellUpdate) {
          const float cxf = op.wf[j] * in.idxf, cyf = op.wf[i] * in.idyf;
          float fl[V], fr[V], gb[V], gt[V];
          if (own_faces) {
            fl[0] = sF[j];
            fr[0] = sF[P + j];
            gb[0] = sF[2 * P + i];
            gt[0] = sF[3 * P + i];
          } else {
            load_v<V>(XL + ((size_t)fxl * P + j) * V, fl);
            load_v<V>(XR + ((size_t)(fxl + 1) * P + j) * V, fr);
            load_v<V>(YB + ((size_t)fyb * P + i) * V, gb);
            load_v<V>(YT + ((size_t)fyt * P + i) * V, gt);
          }
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const float sx = fr[v] * op.FRf[i] - fl[v] * op.FLf[i];
            const float sy = gt[v] * op.FRf[j] - gb[v] * op.FLf[j];
            d[v] = d[v] - (cxf * sx + cyf * sy);
          }
        }
        if (mode == kCellSurface) {
          float* D32w = reinterpret_cast<float*>(a.duh);
          store_v<V>(D32w + off, d);
        } else {
          const double dt = st.dt;
          const double* uo = a.uh[par] + off;
          double* un = a.uh[par ^ 1] + off;
          const float iw = op.iwwf[i + P * j];
          load_v<V>(uo, u);
#pragma unroll
          for (int v = 0; v < V; ++v) u[v] = fma(dt, (double)(d[v] * iw), u[v]);
          store_v<V>(un, u);
        }
      } else {
        double d[V], p[V], q[V];
        load_v<V>(a.duh + off, d);
        if (mode != kCellUpdate) {
          // surface_integral.f90:20-35: x faces then y faces
          const double* XL = a.fu;
          const double* XR = (Sys::ID == kSysBN) ? a.fp : a.fu;
          const double* YB = a.gu;
          const double* YT = (Sys::ID == kSysBN) ? a.gp : a.gu;
          const double cx = in.wdx[j], cy = in.wdy[i];  // w_j / dx, w_i / dy
          if (own_faces) {
            p[0] = sF[j];
            q[0] = sF[P + j];
          } else {
            load_v<V>(XL + ((size_t)fxl * P + j) * V, p);
            load_v<V>(XR + ((size_t)(fxl + 1) * P + j) * V, q);
          }
#pragma unroll
          for (int v = 0; v < V; ++v) {
            if constexpr (kExact) d[v] = fma(-cx, fma(-p[v], op.FLd[i], q[v] * op.FRd[i]), d[v]);
            else d[v] = d[v] - cx * (q[v] * op.FRd[i] - p[v] * op.FLd[i]);
          }
          if (own_faces) {
            p[0] = sF[2 * P + i];
            q[0] = sF[3 * P + i];
          } else {
            load_v<V>(YB + ((size_t)fyb * P + i) * V, p);
            load_v<V>(YT + ((size_t)fyt * P + i) * V, q);
          }
#pragma unroll
          for (int v = 0; v < V; ++v) {
            if constexpr (kExact) d[v] = fma(-cy, fma(-p[v], op.FLd[j], q[v] * op.FRd[j]), d[v]);
            else d[v] = d[v] - cy * (q[v] * op.FRd[j] - p[v] * op.FLd[j]);
          }
        }
        if (mode == kCellSurface) {
          store_v<V>(a.duh + off, d);
        } else {
          // element_update.f90:18-26
          const double dt = st.dt;
          const double* uo = a.uh[par] + off;
          double* un = a.uh[par ^ 1] + off;
          load_v<V>(uo, p);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            if constexpr (kExact) {
              u[v] = fma(dt, quot<true>(d[v], op.wd[i] * op.wd[j], op.iwwd[i + P * j]), p[v]);
            } else {
              d[v] = div_by(d[v], op.wd[i] * op.wd[j], op.iwwd[i + P * j]);
              u[v] = p[v] + dt * d[v];
            }
          }
          store_v<V>(un, u);
        }
      }
    } else {
      load_v<V>(a.uh[par] + off, u);
    }
  }
  if (mode == kCellSurface) return;  // uniform per launch: no barrier follows

  // kFast: the node's state in FP32, and its deviation from the cell's
  // FP32 reference state ubar, formed in FP32 (one conversion per value)
  float uf[V], du[V], ubf[V];
  if constexpr (kFast && Sys::ID != kSysAD) {
#pragma unroll
    for (int v = 0; v < V; ++v) {
      ubf[v] = ubs[v];
      // on the integer pipe where the FP64 pipe bounds the kernel (504 -> 492 us on
      // the FP64 vortex; the FP32 modes wait on latency: 328 -> 344 us)
      uf[v] = !act ? 0.0f : kExact ? narrow_bits(u[v]) : (float)u[v];
      du[v] = act ? uf[v] - ubf[v] : 0.0f;
    }
  }

  // ------------------------------------------------------------- CFL part
  const bool want_cfl = mode != kCellInitDmp && mode != kCellPrimeLimited;
  auto cfl_bits = [&]() -> unsigned long long {
    double dn;
    if constexpr (kExact && Sys::ID != kSysAD) {
      if (mode == kCellFused) return cfl_key<Sys>(in, uf);
      dn = cfl_denom_call<Sys, N>(in, u);
    } else if constexpr (kF32) {
      dn = cfl_denom_f32<Sys, N>(in, typename Sys::FConst(in.ph), uf, u);
    } else {
      dn = cfl_denom<Sys, N>(in, u);
    }
    return (unsigned long long)__double_as_longlong(dn);
  };
  // cells as aligned warp segments: per-cell maxima by shuffles, one store per
  // cell instead of P2 atomics on one shared address
  // warp reductions ahead of the atomics on |du|: Euler N = 4 150 -> 144 us (vortex
  // 256^2), N = 5 301 -> 291 us; Baer-Nunziato N = 2 342 -> 379 us (nine reductions
  // of four groups each)
  constexpr bool kRedux = P2 > 16 && V <= 4;
  // (advection-diffusion's denominator is the instance's constant, folded below)
  constexpr bool kSeg = (32 % P2) == 0 && (C::THREADS % 32) == 0 && C::CPB * P2 == C::THREADS;
  if constexpr (kSeg && Sys::ID != kSysAD) {
    if (want_cfl) {
      unsigned long long bits = 0ull;
      if (act) {
        bits = cfl_bits();
      }
      bits = seg_max<P2>(bits);
      if (act && node == 0) cmax[lc] = bits;
    }
  } else if constexpr (Sys::ID != kSysAD) {
    if (want_cfl) {
      unsigned long long bits = 0ull;
      if (act) {
        bits = cfl_bits();
      }
      // the lanes of a cell within this warp by shuffles, then one atomic per
      // cell and warp (every lane on its cell's address took turns)
      const int lane = t & 31, rest = min(31 - lane, P2 - 1 - node);
#pragma unroll
      for (int o = 1; o < 32 && o < P2; o <<= 1) {
        const unsigned long long y = __shfl_down_sync(0xffffffffu, bits, o);
        if (o <= rest && y > bits) bits = y;
      }
      if (act && (lane == 0 || node == 0)) atomicMax(&cmax[lc], bits);
    }
  }

  // ------------------------------------------------------------- DMP part
  const bool want_dmp = limiter && mode != kCellCfl;
  if (want_dmp) {
    // Cells whose limiter is active keep their min/max from the subcell data
    // (get_min_max, Euler/limiter.f90:134-139) in the priming pass.
    const bool from_lh = act && (mode == kCellPrime || mode == kCellPrimeLimited) && a.status[par][valid ? cell : 0] != 0;
    if constexpr (kFast) {
      if (act) {
#pragma unroll
        for (int v = 0; v < V; ++v) U[v * P2 + node] = u[v];
        if constexpr (kRedux) {
          // the lanes of a cell within this warp, then one atomic
          const int lane = t & 31, first = max(lane - node, 0), last = min(lane + P2 - 1 - node, 31);
          const unsigned m = (0xffffffffu >> (31 - last)) & (0xffffffffu << first);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const unsigned x = __reduce_max_sync(m, __float_as_uint(fabsf(du[v])));
            if (lane == first) atomicMax(&amax[v], x);
          }
        } else if constexpr (!kSeg) {
#pragma unroll
          for (int v = 0; v < V; ++v) atomicMax(&amax[v], __float_as_uint(fabsf(du[v])));
        }
        PF::template st<PF::NU>(Uf, node, du);
      }
      if constexpr (kSeg) {
        // du = 0 in lanes of inactive cells
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const unsigned m = seg_max<P2>(__float_as_uint(fabsf(du[v])));
          if (act && node == 0) amax[v] = m;
        }
      }
      __syncthreads();
      // FP32 projections of the deviations when their error bound stays
      // within the DMP's absolute tolerance (1e-4) for every variable;
      // otherwise this cell takes the FP64 projections in the reference's
      // order (the FP64 path's values bit for bit).
      float err[V];
      bool f32ok = true;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const float am = __uint_as_float(amax[v]);
        err[v] = op.perr * am + op.pdev * (fabsf(ubf[v]) + 2.0f * am);
        f32ok = f32ok && err[v] <= 1.0e-4f;
      }
      if (act && !from_lh) {
        if (f32ok) {
          if constexpr (kTeam) Proj<N, V, float>::ypass_team(Uf, LYf, LBf, opsf, opsf + S * P, node);
          else Proj<N, V, float>::template ypass<true>(Uf, LYf, LBf, opsf, opsf + S * P, node, P2);
        }
        else Proj<N, V, double>::template ypass<false>(U, LY, LB, opsm, opsm + S * P, node, P2);
      }
      __syncthreads();
      bool posfail = false;
      if (act) {
        if (from_lh) {
          double mn[V], mx[V];
#pragma unroll
          for (int v = 0; v < V; ++v) { mn[v] = kInf; mx[v] = -kInf; }
          const double* L = a.lh[par] + (size_t)cell * S * S * V;
          for (int idx = node; idx < S * S; idx += P2)
#pragma unroll
            for (int v = 0; v < V; ++v) { mn[v] = fmin(mn[v], L[idx * V + v]); mx[v] = fmax(mx[v], L[idx * V + v]); }
#pragma unroll
          for (int v = 0; v < V; ++v) {
            RED[v * P2 + node] = mn[v];
            RED[(V + v) * P2 + node] = mx[v];
          }
        } else if (f32ok) {
          float mn[V], mx[V];
#pragma unroll
          for (int v = 0; v < V; ++v) { mn[v] = du[v]; mx[v] = du[v]; }
          if constexpr (kTeam)
            Proj<N, V, float>::template xpass_team<Sys>(LYf, LBf, opsf, opsf + S * P, U, opsm,
                                                        typename Sys::FConst(in.ph), err, ubf, in.ph, node, mn, mx,
                                                        posfail);
          else
            Proj<N, V, float>::template xpass_minmax_f32<Sys>(LYf, LBf, opsf, opsf + S * P, U, opsm,
                                                              typename Sys::FConst(in.ph), err, ubf, in.ph, node, P2,
                                                              mn, mx, posfail);
          store_v<V>(REDf + node * 2 * V, mn);
          store_v<V>(REDf + node * 2 * V + V, mx);
        } else {
          double mn[V], mx[V];
#pragma unroll
          for (int v = 0; v < V; ++v) { mn[v] = kInf; mx[v] = -kInf; }
          Proj<N, V, double>::template xpass_minmax<Sys, false>(U, LY, LB, opsm, opsm + S * P, in.ph, node, P2, mn, mx,
                                                                posfail);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            RED[v * P2 + node] = mn[v];
            RED[(V + v) * P2 + node] = mx[v];
          }
        }
        if (posfail) atomicOr(&cflag[lc], 1);
      }
      if (act && node == 0 && f32ok && !from_lh) atomicOr(&cflag[lc], 8);  // the cell's partial min/max are in REDf (FP32)
    } else {
      if (act) {
#pragma unroll
        for (int v = 0; v < V; ++v) U[v * P2 + node] = u[v];
      }
      __syncthreads();
      const double* lim = opsm;
      const double* lob = opsm + S * P;
      if (act && !from_lh) Proj<N, V, double>::template ypass<false>(U, LY, LB, lim, lob, node, P2);
      __syncthreads();
      double mn[V], mx[V];
      bool posfail = false;
#pragma unroll
      for (int v = 0; v < V; ++v) { mn[v] = kInf; mx[v] = -kInf; }
      if (act) {
        if (from_lh) {
          const double* L = a.lh[par] + (size_t)cell * S * S * V;
          for (int idx = node; idx < S * S; idx += P2)
#pragma unroll
            for (int v = 0; v < V; ++v) { mn[v] = fmin(mn[v], L[idx * V + v]); mx[v] = fmax(mx[v], L[idx * V + v]); }
        } else {
          Proj<N, V, double>::template xpass_minmax<Sys, false>(U, LY, LB, lim, lob, in.ph, node, P2, mn, mx, posfail);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          RED[v * P2 + node] = mn[v];
          RED[(V + v) * P2 + node] = mx[v];
        }
        if (posfail) atomicOr(&cflag[lc], 1);
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < C::NITEM; ++q) {
      const int it = t + q * C::THREADS, pr = it / LPP, lc2 = pr / V, v = pr - lc2 * V;
      const int k2 = pr < CPB * V ? cinst[lc2] : -1;
      const bool on = k2 >= 0;
      // LPP = 2: the lanes of a pair exchange their bounds, so the warp stays together
      if (LPP == 2 ? !__any_sync(0xffffffffu, on) : !on) continue;
      const int lcs = on ? lc2 : 0, prs = on ? pr : 0, side0 = LPP == 2 ? it & 1 : 0;
      const long long cell2 = a.cell0 + (long long)blockIdx.x * CPB + lcs;
      const int par2 = on ? parity(a.st[k2]) : 0;
      const double* U2 = sm + (size_t)lcs * C::CELL_DBL;
      const bool f32red = (cflag[lcs] & 8) != 0;
      const float am = kFast ? __uint_as_float(amax_all[prs]) : 0.0f, ub32 = kFast ? ubs_all[prs] : 0.0f;
      const double ubar = kFast ? (double)ub32 : 0.0;  // the cell's FP32 reference state
      // the cell's minimum and maximum.  FP32 projections: their deviations fx
      // from the cell's FP32 reference state ubar, and a bound on |ubar + fx -
      // FP64 value|: the projections' bound as formed above (rounded up), plus
      // the FP64 roundings of the reference-order values (generously 1e-12
      // relative)
      double cm[SPL], bound[SPL];  // own value; lmin or lmax
      float fx[SPL], en = 0.0f;
      const float ecell = !f32red ? 0.0f
                                  : (op.perr * am + op.pdev * (fabsf(ub32) + 2.0f * am)) * 1.0001f +
                                        1.0e-12f * (fabsf(ub32) + am);
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        cm[s] = 0.0;
        fx[s] = 0.0f;
      }
      if (on && f32red) {
        const float* r = reinterpret_cast<const float*>(U2) + C::RED_F + side0 * V + v;
#pragma unroll
        for (int k = 0; k < P2; ++k)
#pragma unroll
          for (int s = 0; s < SPL; ++s) {
            const float x = side0 + s ? -r[k * 2 * V + s * V] : r[k * 2 * V + s * V];
            fx[s] = k == 0 ? x : fminf(fx[s], x);
          }
#pragma unroll
        for (int s = 0; s < SPL; ++s) {
          fx[s] = side0 + s ? -fx[s] : fx[s];
          cm[s] = ubar + (double)fx[s];
        }
      } else if (on) {
#pragma unroll
        for (int s = 0; s < SPL; ++s) {
          const double* r = U2 + C::U_DBL + V * S * P + V * P * P + ((side0 + s) * V + v) * P2;
          double x = side0 + s ? -r[0] : r[0];
#pragma unroll
          for (int k = 1; k < P2; ++k) x = fmin(x, side0 + s ? -r[k] : r[k]);
          cm[s] = side0 + s ? -x : x;
        }
      }
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        const int side = side0 + s;
        bound[s] = 0.0;
        if (mode == kCellPrime || mode == kCellPrimeLimited) {
          if (on) {
            a.mm[par2][((size_t)cell2 * 2 + side) * V + v] = cm[s];
            if (a.mme[0] && side == 0) a.mme[par2][(size_t)cell2 * V + v] = ecell;
          }
        } else if (mode == kCellInitDmp) {
          // Euler/initialize.f90:291-294: the cell's own nodal min/max
          const double* Uv = U2 + v * P2;
          double x = side ? -Uv[0] : Uv[0];
          for (int k = 1; k < P2; ++k) x = fmin(x, side ? -Uv[k] : Uv[k]);
          bound[s] = side ? -x : x;
        } else {
          // get_min_max step 2: the neighbourhood bounds folded at the start
          bound[s] = nbound[q][s];
          en = nen[q];
          if (on) {
            if (a.lminmax) a.lminmax[((size_t)cell2 * 2 + side) * V + v] = bound[s];
            // candidate min/max for the next step (status 0)
            a.mm[par2 ^ 1][((size_t)cell2 * 2 + side) * V + v] = cm[s];
            if (a.mme[0] && side == 0) a.mme[par2 ^ 1][(size_t)cell2 * V + v] = ecell;
          }
        }
      }
      if (mode == kCellPrime || mode == kCellPrimeLimited) continue;
      const bool in64 = a.mme[0] == nullptr || (!f32red && en == 0.0f);
      // (no warp vote where the mode decides)
      if (a.mme[0] == nullptr || (LPP == 2 ? __any_sync(0xffffffffu, on && in64) : in64)) {
        // FP64 values (FP32-wide mode: FP32 projections taken as they are);
        // Euler/limiter.f90:210-220
        double other = bound[SPL - 1];
        if constexpr (LPP == 2) other = __shfl_xor_sync(0xffffffffu, bound[0], 1);
        if (on && in64) {
          const double lmin = side0 ? other : bound[0], lmax = side0 ? bound[0] : other;
          const double ldiff = fmax(fmax(1.0e-4, 1.0e-3 * (lmax - lmin)), mode == kCellInitDmp ? 1.0e-1 : 0.0);
#pragma unroll
          for (int s = 0; s < SPL; ++s)
            if (side0 + s ? cm[s] > lmax + ldiff : cm[s] < lmin - ldiff) atomicOr(&cflag[lc2], 2);
        }
      }
      if (LPP == 2 ? a.mme[0] != nullptr : !in64) {
        // FP64 and FP32-mixed: the same comparisons in FP32, in the deviation space
        // of the cell's FP32 reference state ub (FP64 work is the costly
        // part of this kernel).  |own - FP64 value| <= ecell; |lmin - its
        // FP64 value| <= en and likewise lmax, so the thresholds move by at
        // most en (1 + 2e-3); the FP32 forms of lmin - ub, lmax - ub, ldiff,
        // the thresholds and the differences add at most 2.5e-7 of the
        // magnitudes involved, and the FP32 constants 1e-4 and 0.1 differ
        // from their FP64 values by less than 1e-11 and 1e-8 of themselves.
        // A comparison decides here only when it holds by that margin;
        // otherwise k_settle decides the cell from FP64 values (bit 4).
        float L[SPL];
#pragma unroll
        for (int s = 0; s < SPL; ++s) L[s] = (float)(bound[s] - ubar);
        float other = L[SPL - 1];
        if constexpr (LPP == 2) other = __shfl_xor_sync(0xffffffffu, L[0], 1);
        const float ld = fmaxf(fmaxf(1.0e-4f, 1.0e-3f * (side0 ? L[0] - other : other - L[0])),
                               mode == kCellInitDmp ? 0.1f : 0.0f);
        const float e = ecell + 1.002f * en + 2.5e-7f * (fabsf(L[0]) + fabsf(other) + ld) + 1.0e-11f +
                        1.0e-12f * fabsf(ub32);
#pragma unroll
        for (int s = 0; s < SPL; ++s) {
          const float sg = side0 + s ? -1.0f : 1.0f;
          const float x = f32red ? fx[s] : (float)(cm[s] - ubar);
          const float m = e + 1.2e-7f * fabsf(x);
          const float g = sg * (x - (L[s] - sg * ld));  // >= 0: not below lmin - ldiff / not above lmax + ldiff
          if (LPP == 1 || (on && !in64)) {
            if (g < -m) atomicOr(&cflag[lc2], 2);
            else if (!(g >= m)) atomicOr(&cflag[lc2], 4);
          }
        }
      }
    }
    __syncthreads();
    {
      // a cell whose DMP the error bounds left open (bit 4) and that nothing
      // else marked goes on the list k_settle decides from FP64 values; here it
      // counts as not troubled
      if (act && node == 0 && a.settle && (cflag[lc] & 7) == 4 &&
          (mode == kCellFused || mode == kCellUpdate || mode == kCellInitDmp))
        a.settle[atomicAdd(&a.list_count[1], 1)] = (int)cell;
    }
    if (act && mode != kCellPrime && mode != kCellPrimeLimited) {
      const bool bad = (cflag[lc] & 3) != 0;
      if (mode == kCellInitDmp) {
        if (bad) {
          // Euler/initialize.f90:296-317: status 1, Lh = NewLh = initial subcell data
          if (node == 0) {
            a.status[0][cell] = 1;
            a.status[1][cell] = 1;
            atomicAdd(&a.st[kc].n_recompute, 1);
          }
          if (a.lh_ic) {
            const size_t o = (size_t)cell * S * S * V;
            for (int idx = node; idx < S * S * V; idx += P2) {
              a.lh[0][o + idx] = a.lh_ic[o + idx];
              a.lh[1][o + idx] = a.lh_ic[o + idx];
            }
          }
        }
      } else if (node == 0) {
        a.troubled[cell] = bad ? 1 : 0;
        if (bad) atomicAdd(&a.st[kc].n_recompute, 1);
      }
    }
  } else {
    __syncthreads();
  }

  // ------------------------------------------------ CFL per cell / instance
  if (!want_cfl) return;
  if (limiter && (mode == kCellFused || mode == kCellUpdate)) {
    if (act && node == 0) a.denom[cell] = __longlong_as_double((long long)cmax[lc]);
    return;
  }
  // fold the CTA's cells per instance: the node-0 thread of the first cell of
  // each instance in this CTA folds that instance's cells (a contiguous run)
  // and issues one atomic
  if (act && node == 0 && (lc == 0 || cell - 1 < in.cell_base)) {
    unsigned long long m = 0ull;
    if constexpr (Sys::ID == kSysAD) {
      m = (unsigned long long)__double_as_longlong(in.ad_denom);
    } else {
      const long long end = in.cell_base + (long long)in.imax * in.jmax;
      for (int c = lc; c < CPB && cell + (c - lc) < end; ++c) m = m > cmax[c] ? m : cmax[c];
    }
    atomicMax(&a.st[kc].denom_next, m);
  }
}


}  // namespace aderdg
