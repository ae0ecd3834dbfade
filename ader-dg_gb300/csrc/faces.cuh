// faces.cuh -- K2: numerical fluxes once per face quadrature point, with the
// boundary conditions inlined.
//
// Reference: Euler/riemann_problem.f90:10-116 (Rusanov, double Mach
// reflection boundaries), Baer-Nunziato/riemann_problem.f90:9-80
// (path-conservative Rusanov fluctuations Dm/Dp), and
// Advection-Diffusion/riemann_problem.f90:8-113 (viscous LLF).  One thread per
// (face, point); the x faces of all instances come first, then the y faces.
// R is the storage type of the face states and fluxes, CT the compute type.
// FP64 (R = CT = double) is compiled with --fmad=false for the phase API: every
// value agrees bit for bit with the reference expression evaluated in FP64 from
// the same face states; the fused step takes the kRec form.  The FP32 modes store states and fluxes in FP32; Euler and
// advection-diffusion compute in FP32, and Baer-Nunziato computes its
// path-conservative flux (Roe-matrix path integral included) in FP64 in the
// FP32-mixed mode (CT = double, instantiated with fused multiply-adds in
// predictor_tu.cu) and in FP32 in the FP32-wide mode.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "physics.cuh"

namespace aderdg {

// instance owning an x / y face, or -1 (faces between instances of a batch)
__device__ __forceinline__ int find_inst_fx(const InstDesc* inst, int n, long long f) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (inst[mid].fx_base <= f) lo = mid; else hi = mid - 1;
  }
  const InstDesc& d = inst[lo];
  if (f < d.fx_base || f - d.fx_base >= (long long)(d.imax + 1) * d.jmax) return -1;
  return lo;
}
__device__ __forceinline__ int find_inst_fy(const InstDesc* inst, int n, long long f) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (inst[mid].fy_base <= f) lo = mid; else hi = mid - 1;
  }
  const InstDesc& d = inst[lo];
  if (f < d.fy_base || f - d.fy_base >= (long long)d.imax * (d.jmax + 1)) return -1;
  return lo;
}

template <int V, class R, class T>
__device__ __forceinline__ void load_face_state(const R* qb, const R* fb, long long cell, int P, int l, int f, T* Q, T* F) {
  const size_t o = (((size_t)cell * 4 + f) * P + l) * V;  // [cell][face][point][v]
  R q[V], g[V];
  load_v<V>(qb + o, q);
  if (F) load_v<V>(fb + o, g);
#pragma unroll
  for (int v = 0; v < V; ++v) {
    Q[v] = widen<T>(q[v]);
    if (F) F[v] = widen<T>(g[v]);
  }
}

// Euler double Mach reflection boundary state: Q = prim2cons(Vp), F = flux(Q)
// along axis d (matmul(Fbc, nv) of Euler/riemann_problem.f90:43-46).
template <class T>
__device__ __forceinline__ void dmr_state(const PhysC<T>& pc, const double* Vpd, int d, T* Q, T* F) {
  T Fb[8], Vp[4];
  for (int v = 0; v < 4; ++v) Vp[v] = (T)Vpd[v];
  EulerSys::prim2cons(pc, Vp, Q);
  EulerSys::flux(pc, Q, Fb);
  for (int v = 0; v < 4; ++v) F[v] = Fb[d * 4 + v];
}

// Euler Rusanov pieces in the compute type T (FP32 in the FP32 modes)
template <class T>
__device__ __forceinline__ T euler_max_eig_t(T gamma, const T* Q, int d) {
  const T u = (d == 0 ? Q[1] : Q[2]) / Q[0];
  const T p = (gamma - T(1)) * (Q[3] - T(0.5) * (Q[1] * Q[1] + Q[2] * Q[2]) / Q[0]);
  const T c = sqrt(gamma * p / Q[0]);
  return fmax(fmax(fabs(u - c), fabs(u)), fabs(u + c));
}
template <class T>
__device__ __forceinline__ void euler_bc_state_t(T gamma, const double* Vp, int d, T* Q, T* F) {
  Q[0] = T(Vp[0]);
  Q[1] = T(Vp[0] * Vp[1]);
  Q[2] = T(Vp[0] * Vp[2]);
  Q[3] = T(Vp[3] / (double(gamma) - 1) + 0.5 * Vp[0] * (Vp[1] * Vp[1] + Vp[2] * Vp[2]));
  const T irho = T(1) / Q[0];
  const T p = (gamma - T(1)) * (Q[3] - T(0.5) * (Q[1] * Q[1] + Q[2] * Q[2]) * irho);
  const T un = (d == 0 ? Q[1] : Q[2]);
  F[0] = un;
  F[1] = irho * un * Q[1] + (d == 0 ? p : T(0));
  F[2] = irho * un * Q[2] + (d == 1 ? p : T(0));
  F[3] = irho * un * (Q[3] + p);
}

// FP32-mixed faces for Euler: boundary logic as in k_faces, arithmetic in FP32
template <int N>
__device__ void faces_euler_fp32(const BatchArgs& a, const FaceConst& fc, const InstDesc& in, int k, bool xdir, int i,
                                 int j, int l, long long face) {
  constexpr int P = N + 1, V = 4;
  const float* qb = reinterpret_cast<const float*>(a.qbnd);
  const float* fb = reinterpret_cast<const float*>(a.fbnd);
  const int I = in.imax, J = in.jmax;
  auto cid = [&](int ci, int cj) { return in.cell_base + (long long)ci + (long long)I * cj; };
  auto load = [&](long long c, int f, float* Q, float* F) {
    const size_t o = (((size_t)c * 4 + f) * P + l) * V;
    load_v<V>(qb + o, Q);
    load_v<V>(fb + o, F);
  };
  const float gamma = (float)in.ph.gamma;
  const int d = xdir ? 0 : 1, pos = xdir ? i : j, last = xdir ? I : J;
  const int bcl = in.bc[xdir ? 0 : 2], bcr = in.bc[xdir ? 1 : 3];
  const int fl = xdir ? 0 : 2, fr = xdir ? 1 : 3;
  const bool is_dmr = in.bc_mode == 1;
  float QL[V], QR[V], FL[V], FR[V];
  const long long cR = cid(i, j);
  if (pos == 0) {
    if (is_dmr && xdir) {
      euler_bc_state_t<float>(gamma, fc.Va, 0, QL, FL);
      load(cR, fl, QR, FR);
    } else if (is_dmr) {
      load(cR, fl, QL, FL);
      if (!((double)(i + 1) * in.dx <= 1.0 / 6.0)) {
        QL[2] = -QL[2];
        FL[0] = -FL[0];
        FL[1] = -FL[1];
        FL[3] = -FL[3];
      }
      load(cR, fl, QR, FR);
    } else if (bcl == 3) {
      load(xdir ? cid(I - 1, j) : cid(i, J - 1), fr, QL, FL);
      load(cR, fl, QR, FR);
    } else {
      load(cR, fl, QL, FL);
      load(cR, fl, QR, FR);
    }
  } else if (pos == last) {
    const long long cLast = xdir ? cid(I - 1, j) : cid(i, J - 1);
    load(cLast, fr, QL, FL);
    if (is_dmr && !xdir) {
      const double x_sw = fc.xsw0 + fc.xsw1 * a.st[k].time;
      euler_bc_state_t<float>(gamma, ((double)(i + 1) * in.dx <= x_sw) ? fc.Va : fc.Vb, 1, QR, FR);
    } else if (!is_dmr && bcr == 3) {
      load(xdir ? cid(0, j) : cid(i, 0), fl, QR, FR);
    } else {
      load(cLast, fr, QR, FR);
    }
  } else {
    load(xdir ? cid(i - 1, j) : cid(i, j - 1), fr, QL, FL);
    load(cR, fl, QR, FR);
  }
  const float smax = fmaxf(euler_max_eig_t<float>(gamma, QL, d), euler_max_eig_t<float>(gamma, QR, d));
  float* dst = reinterpret_cast<float*>(xdir ? a.fu : a.gu) + ((size_t)face * P + l) * V;
  float out[V];
#pragma unroll
  for (int v = 0; v < V; ++v) out[v] = 0.5f * (FL[v] + FR[v]) - 0.5f * smax * (QR[v] - QL[v]);
  store_v<V>(dst, out);
}

// Advection-diffusion's numerical flux at point l of face (i, j) along x (xdir)
// or y, as stored: Advection-Diffusion/riemann_problem.f90 with
// PDEViscLLFRiemannSolver (pde.f90:121-152); compute type CT: FP64 (reference
// order), FP32 in the FP32 modes.  xi = the point's coordinate in its face, P the
// points of a face.  On small grids the fused step's cell kernel forms its cells'
// face fluxes from it, too.
template <class R, class CT>
__device__ __forceinline__ R ad_face_flux(const BatchArgs& a, const InstDesc& in, double pi, double xi, bool xdir, int i,
                                          int j, int l, int P) {
  const R* qb = reinterpret_cast<const R*>(a.qbnd);
  const R* fb = reinterpret_cast<const R*>(a.fbnd);
  const int I = in.imax, J = in.jmax;
  auto cid = [&](int ci, int cj) { return in.cell_base + (long long)ci + (long long)I * cj; };
  const int pos = xdir ? i : j, last = xdir ? I : J;
  const int bcl = in.bc[xdir ? 0 : 2], bcr = in.bc[xdir ? 1 : 3];
  const int fl = xdir ? 0 : 2, fr = xdir ? 1 : 3;  // left/bottom and right/top face ids
  CT QL[1], QR[1], gL[2], gR[2];
  auto get = [&](long long c, int f, CT* Q, CT* gq) {
    const size_t o = (((size_t)c * 4 + f) * P + l);
    Q[0] = (CT)qb[o];
    gq[0] = (CT)fb[o * 2 + 0];
    gq[1] = (CT)fb[o * 2 + 1];
  };
  const long long cL = xdir ? cid(i - 1, j) : cid(i, j - 1);
  const long long cR = cid(i, j);
  if (pos == 0) {
    if (bcl == 1) {
      get(cR, fl, QL, gL);
      get(cR, fl, QR, gR);
    } else if (bcl == 2) {
      if (xdir) {
        // QR from the right face of cell IMAX, QL = -QR + 2 sin(pi y),
        // y = (j-1 + xi_l) dy (Advection-Diffusion/riemann_problem.f90:37-40)
        get(cid(I - 1, j), 1, QR, gR);
        const double y = ((double)j + xi) * in.dy;
        QL[0] = -QR[0] + (CT)(2.0 * sin(pi * y));
      } else {
        get(cR, fl, QR, gR);
        QL[0] = -QR[0];
      }
      gL[0] = gR[0];
      gL[1] = gR[1];
    } else {
      get(xdir ? cid(I - 1, j) : cid(i, J - 1), fr, QL, gL);
      get(cR, fl, QR, gR);
    }
  } else if (pos == last) {
    const long long cLast = xdir ? cid(I - 1, j) : cid(i, J - 1);
    if (bcr == 1) {
      get(cLast, fr, QL, gL);
      get(cLast, fr, QR, gR);
    } else if (bcr == 2) {
      get(cLast, fr, QL, gL);
      QR[0] = -QL[0];
      gR[0] = gL[0];
      gR[1] = gL[1];
    } else {
      get(cLast, fr, QL, gL);
      get(xdir ? cid(0, j) : cid(i, 0), fl, QR, gR);
    }
  } else {
    get(cL, fr, QL, gL);
    get(cR, fl, QR, gR);
  }
  const CT nv0 = xdir ? CT(1) : CT(0), nv1 = xdir ? CT(0) : CT(1);
  // smax = max(|c.n|) + 2 eta a, eta = (2N+1) / (dx sqrt(pi/2)): formed on the host
  const CT smax = (CT)in.ad_smax[xdir ? 0 : 1];
  const CT cx = (CT)in.ph.cx, cy = (CT)in.ph.cy, ca = (CT)in.ph.a;
  const CT FL0 = cx * QL[0] + -ca * gL[0], FL1 = cy * QL[0] + -ca * gL[1];
  const CT FR0 = cx * QR[0] + -ca * gR[0], FR1 = cy * QR[0] + -ca * gR[1];
  return (R)(CT(0.5) * ((FL0 + FR0) * nv0 + (FL1 + FR1) * nv1) - CT(0.5) * smax * (QR[0] - QL[0]));
}

// Baer-Nunziato's path-conservative face fluxes F-, F+ (pde.f90:326-353) in the
// reference's order
template <class CT>
__device__ __forceinline__ void bn_face(const PhysC<CT>& pc, const CT* QL, const CT* QR, const CT* FL, const CT* FR, int d,
                                        CT* fm, CT* fp) {
  const CT smax = tmax(BNSys::max_eig(pc, QL, d), BNSys::max_eig(pc, QR, d));
  CT D[9];
  BNSys::roe_times_jump(pc, QL, QR, d, D);
#pragma unroll
  for (int v = 0; v < 9; ++v) {
    const CT base = CT(0.5) * (FL[v] + FR[v]) - CT(0.5) * smax * (QR[v] - QL[v]);
    fm[v] = base - CT(0.5) * D[v];
    fp[v] = base + CT(0.5) * D[v];
  }
}
// out of line, for the states of the FP64 fused step's faces that are not ordinary:
// q holds QL, QR, FL, FR, then F- and F+
static __device__ __noinline__ void face_reference(const Phys& ph, int d, double* q) {
  double fm[9], fp[9];
  bn_face(PhysC<double>(ph), q, q + 9, q + 18, q + 27, d, fm, fp);
  for (int v = 0; v < 9; ++v) {
    q[v] = fm[v];
    q[9 + v] = fp[v];
  }
}
static __device__ __noinline__ double max_eig_call(const Phys& ph, double q0, double q1, double q2, double q3, int d) {
  const double Q[4] = {q0, q1, q2, q3};
  return EulerSys::max_eig(ph, Q, d);
}

// kRec (FP64): the reciprocal-sharing forms, for the fused step (the phase API, and
// states that are not ordinary, take the reference's operation order): Euler N = 4
// 256^2 139 -> 96 us, Baer-Nunziato N = 3 200^2 432 -> 143 us.  FP32-mixed
// Baer-Nunziato: three CTAs an SM (80 registers, 16 bytes spilled) and the rounding
// on the integer pipe: 462 -> 405 us, cylinder N = 3 400^2
template <class Sys, int N, class R, class CT, bool kRec = false>
__global__ void __launch_bounds__(256, Sys::ID == kSysBN && sizeof(R) == 4 && sizeof(CT) == 8 ? 3 : 1) k_faces(BatchArgs a, FaceConst fc) {
  constexpr int P = N + 1, V = Sys::V;
  const long long nx = a.nfx * P, ny = a.nfy * P;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nx + ny) return;
  const R* qb = reinterpret_cast<const R*>(a.qbnd);
  const R* fb = reinterpret_cast<const R*>(a.fbnd);
  // x and y face points interleave warp by warp, so that the x faces and the
  // y faces of the same cells run at the same time: a cell's face states lie
  // side by side ([cell][P][4 faces][V]) and each DRAM burst then serves both
  // directions instead of being fetched once per direction
  const long long mw = (nx < ny ? nx : ny) >> 5;  // interleaved warp pairs
  bool xdir;
  long long g;
  if (gid < 64 * mw) {
    const long long w = gid >> 5;
    xdir = (w & 1) == 0;
    g = (w >> 1) * 32 + (gid & 31);
  } else {
    // the rest: x points [32 mw, nx), then y points [32 mw, ny)
    const long long r = gid - 64 * mw, rx = nx - 32 * mw;
    xdir = r < rx;
    g = 32 * mw + (xdir ? r : r - rx);
  }
  const long long face = g / P;
  const int l = (int)(g - face * P);
  const int k = xdir ? find_inst_fx(a.inst, a.ninst, face) : find_inst_fy(a.inst, a.ninst, face);
  if (k < 0) return;
  const InstDesc& in = a.inst[k];
  if (!a.st[k].active) return;
  const Phys ph = in.ph;
  const int I = in.imax, J = in.jmax;
  const long long lf = face - (xdir ? in.fx_base : in.fy_base);
  int i, j;
  const unsigned n1 = (unsigned)(xdir ? I + 1 : I);  // below 2^31 faces an instance
  j = (int)((unsigned)lf / n1);
  i = (int)((unsigned)lf % n1);
  auto cid = [&](int ci, int cj) { return in.cell_base + (long long)ci + (long long)I * cj; };
  const int d = xdir ? 0 : 1;
  const int nfaces_side = xdir ? I : J;  // index of the last face along d is nfaces_side
  const int pos = xdir ? i : j;
  const int bcl = in.bc[xdir ? 0 : 2], bcr = in.bc[xdir ? 1 : 3];
  const int fl = xdir ? 0 : 2, fr = xdir ? 1 : 3;  // left/bottom and right/top face ids
  const size_t out = ((size_t)face * P + l) * V;
  if constexpr (Sys::ID == kSysEuler && sizeof(R) == 4) {
    static_assert(sizeof(CT) == 4, "Euler's FP32-storage faces compute in FP32");
    faces_euler_fp32<N>(a, fc, in, k, xdir, i, j, l, face);
    return;
  }

  if constexpr (Sys::ID == kSysAD) {
    reinterpret_cast<R*>(xdir ? a.fu : a.gu)[out] = ad_face_flux<R, CT>(a, in, fc.pi, fc.xi[l], xdir, i, j, l, P);
  } else {
    // Euler (FP64) and Baer-Nunziato (FP64 or FP32 compute, see above); FP32-mixed
    // Baer-Nunziato (kRcp) keeps the FP32 states and widens them where it uses them
    constexpr bool kRcp = sizeof(R) == 4 && sizeof(CT) == 8;
    using LT = typename std::conditional<kRcp, float, CT>::type;
    const PhysC<CT> pc(ph);
    LT QL[V], QR[V], FL[V], FR[V];
    const bool is_dmr = (Sys::ID == kSysEuler) && in.bc_mode == 1;
    const long long cL = xdir ? cid(i - 1, j) : cid(i, j - 1);
    const long long cR = cid(i, j);
    if (pos == 0) {
      if (is_dmr) {
        if (xdir) {  // inflow, Euler/riemann_problem.f90:41-48
          if constexpr (Sys::ID == kSysEuler) dmr_state(pc, fc.Va, 0, QL, FL);
          load_face_state<V, R>(qb, fb, cR, P, l, fl, QR, FR);
        } else {     // transmissive / reflective wall, :76-86
          load_face_state<V, R>(qb, fb, cR, P, l, fl, QL, FL);
          if (!((double)(i + 1) * in.dx <= 1.0 / 6.0)) {
            QL[2] = -QL[2];
            FL[0] = -FL[0];
            FL[1] = -FL[1];
            FL[3] = -FL[3];
          }
          load_face_state<V, R>(qb, fb, cR, P, l, fl, QR, FR);
        }
      } else if (bcl == 3) {
        load_face_state<V, R>(qb, fb, xdir ? cid(I - 1, j) : cid(i, J - 1), P, l, fr, QL, FL);
        load_face_state<V, R>(qb, fb, cR, P, l, fl, QR, FR);
      } else {
        load_face_state<V, R>(qb, fb, cR, P, l, fl, QL, FL);
        load_face_state<V, R>(qb, fb, cR, P, l, fl, QR, FR);
      }
    } else if (pos == nfaces_side) {
      const long long cLast = xdir ? cid(I - 1, j) : cid(i, J - 1);
      load_face_state<V, R>(qb, fb, cLast, P, l, fr, QL, FL);
      if (is_dmr && !xdir) {  // time-dependent top boundary, :88-100
        const double x_sw = fc.xsw0 + fc.xsw1 * a.st[k].time;
        if constexpr (Sys::ID == kSysEuler) dmr_state(pc, ((double)(i + 1) * in.dx <= x_sw) ? fc.Va : fc.Vb, 1, QR, FR);
      } else if (!is_dmr && bcr == 3) {
        load_face_state<V, R>(qb, fb, xdir ? cid(0, j) : cid(i, 0), P, l, fl, QR, FR);
      } else {
        load_face_state<V, R>(qb, fb, cLast, P, l, fr, QR, FR);
      }
    } else {
      load_face_state<V, R>(qb, fb, cL, P, l, fr, QL, FL);
      load_face_state<V, R>(qb, fb, cR, P, l, fl, QR, FR);
    }
    if constexpr (kRcp) {
      float fm[V], fp[V];
      BNSys::face_mixed(pc, BNSys::FConst(ph), QL, QR, FL, FR, d, fm, fp);
      R* dm = reinterpret_cast<R*>(xdir ? a.fu : a.gu);
      R* dp = reinterpret_cast<R*>(xdir ? a.fp : a.gp);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        dm[out + v] = fm[v];
        dp[out + v] = fp[v];
      }
    } else {
      if constexpr (kRec && Sys::ID == kSysBN) {
        double fm[V], fp[V];
        if (ordinary<Sys>(QL) && ordinary<Sys>(QR)) {
          BNSys::face_r(pc, BNSys::FConst(ph), QL, QR, FL, FR, d, fm, fp);
        } else {
          double q[4 * V];  // (a copy: the call's arguments lie in memory)
#pragma unroll
          for (int v = 0; v < V; ++v) {
            q[v] = QL[v];
            q[V + v] = QR[v];
            q[2 * V + v] = FL[v];
            q[3 * V + v] = FR[v];
          }
          face_reference(in.ph, d, q);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            fm[v] = q[v];
            fp[v] = q[V + v];
          }
        }
        double* dm = xdir ? a.fu : a.gu;
        double* dp = xdir ? a.fp : a.gp;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          dm[out + v] = fm[v];
          dp[out + v] = fp[v];
        }
        return;
      }
      // Rusanov: smax from both sides' eigenvalues (Euler/pde.f90:97-114)
      CT smax;
      if constexpr (kRec && Sys::ID == kSysEuler) {
        if (ordinary<Sys>(QL) && ordinary<Sys>(QR)) smax = max_nonneg(Sys::max_speed_r(pc, QL, d), Sys::max_speed_r(pc, QR, d));
        else smax = tmax(max_eig_call(in.ph, QL[0], QL[1], QL[2], QL[3], d), max_eig_call(in.ph, QR[0], QR[1], QR[2], QR[3], d));
      } else if constexpr (Sys::ID == kSysEuler) {
        smax = tmax(Sys::max_eig(pc, QL, d), Sys::max_eig(pc, QR, d));
      }
      if constexpr (Sys::ID == kSysBN) {
        R* dm = reinterpret_cast<R*>(xdir ? a.fu : a.gu);
        R* dp = reinterpret_cast<R*>(xdir ? a.fp : a.gp);
        CT fm[V], fp[V];
        bn_face(pc, QL, QR, FL, FR, d, fm, fp);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          dm[out + v] = (R)fm[v];
          dp[out + v] = (R)fp[v];
        }
      } else {
        R r[V];
#pragma unroll
        for (int v = 0; v < V; ++v) r[v] = (R)(CT(0.5) * (FL[v] + FR[v]) - CT(0.5) * smax * (QR[v] - QL[v]));
        store_v<V>(reinterpret_cast<R*>(xdir ? a.fu : a.gu) + out, r);
      }
    }
  }
}

}  // namespace aderdg
