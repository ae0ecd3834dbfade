// fv_update.cuh -- the finite-volume step of one cell in the subcell re-solve:
// MUSCL-Hancock reconstruction of the gathered subcells, edge fluxes and update.
// Included in the bodies of k_subcell and of fv_update_reference (limiter.cuh),
// with their template arguments and names: as an inlined function the same text
// cost the FP32-mixed re-solve 2.6% (other registers spilled: 648 -> 666 us on the
// Baer-Nunziato cylinder N = 3 400^2, 321 -> 330 us on the Riemann problem 512^2).

  auto divx = [&](T q) -> T { if constexpr (kRcp) return q * ix0; else return q / ldx0; };
  auto divy = [&](T q) -> T { if constexpr (kRcp) return q * ix1; else return q / ldx1; };
  // the flux of Q into F[d * V + v]; kRcp: along d only (the MUSCL half step
  // uses the x flux of the x-reconstructed states and the y flux of the
  // y-reconstructed ones), otherwise both directions as the reference
  auto flux = [&](const T* Q, int d, T* F) {
    if constexpr (kRcp) {
      T e;
      Sys::template flux_dir_eig_r<kRcp == 2>(pc, Q, d, F + d * V, e);
    } else {
      Sys::flux(pc, Q, F);
    }
  };
  auto ncp = [&](const T* Q, T ax, T ay, T* Sr) {
    if constexpr (Sys::ID == kSysBN) {
      if constexpr (kRcp) BNSys::src_ncp_r<kRcp == 2>(pc, Q, ax, ay, Sr);
      else BNSys::src_ncp(pc, Q, ax, ay, Sr);
    }
  };

  // ---- MUSCL-Hancock reconstruction on subcells 0..S+1; the slopes of
  // one direction at a time in registers.  The S*S interior subcells come
  // first, then the ring of halo subcells, so that the interior ones fill
  // whole warps: Euler's halo subcells have zero slopes (Euler/limiter.f90:
  // 529-536), so their two face states per direction are the subcell value,
  // the half-step flux differences vanish exactly and their evolved face
  // states are the subcell value itself; they are copied, and only the
  // warps holding interior subcells evaluate fluxes.
  for (int p = t; p < H * H; p += NT) {
    int ii, jj;
    if (p < S * S) {
      ii = 1 + p % S;
      jj = 1 + p / S;
    } else {
      const int r = p - S * S;  // the ring: bottom row, top row, left column, right column
      if (r < H) { ii = r; jj = 0; }
      else if (r < 2 * H) { ii = r - H; jj = H - 1; }
      else if (r < 2 * H + S) { ii = 0; jj = 1 + (r - 2 * H); }
      else { ii = H - 1; jj = 1 + (r - 2 * H - S); }
    }
    const bool interior = p < S * S;
    // the corners of the ring feed no edge (Euler does not gather them)
    if (!interior && (ii == 0 || ii == H - 1) && (jj == 0 || jj == H - 1)) continue;
    if (!BN && !interior) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const T q = SU(v, ii, jj);
        wLx[hx(v, ii, jj)] = q;
        wRx[hx(v, ii, jj)] = q;
        wLy[hx(v, ii, jj)] = q;
        wRy[hx(v, ii, jj)] = q;
      }
      continue;
    }
    T Qt[V], FL[2 * V], FR[2 * V];
    // Euler computes slopes for interior subcells only (halo slopes stay 0,
    // Euler/limiter.f90:529-536); BN also on the halo (BN :486-492)
    // kRcp (FP64 re-solve): minmod on the bit patterns
    auto mm = [](T a, T b) -> T {
      if constexpr (kRcp && sizeof(T) == 8) return minmod_bits(a, b);
      else return minmod(a, b);
    };
    auto slope_x = [&](int v) -> T {
      return (BN || interior) ? mm(SU(v, ii + 1, jj) - SU(v, ii, jj), SU(v, ii, jj) - SU(v, ii - 1, jj)) : T(0);
    };
    auto slope_y = [&](int v) -> T {
      return (BN || interior) ? mm(SU(v, ii, jj + 1) - SU(v, ii, jj), SU(v, ii, jj) - SU(v, ii, jj - 1)) : T(0);
    };
    T q0[V], wl[V], wr[V], sl[V];
#pragma unroll
    for (int v = 0; v < V; ++v) q0[v] = SU(v, ii, jj);
    T src[V];
    if constexpr (BN) {
      // Baer-Nunziato/limiter.f90:494-497
      const T ax = slope_x(8), ay = slope_y(8);
      sa8[ii + H * jj] = ax;
      sa8[H * H + ii + H * jj] = ay;
      ncp(q0, divx(ax), divy(ay), src);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) sl[v] = slope_x(v);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      wl[v] = q0[v] - T(0.5) * sl[v];
      wr[v] = q0[v] + T(0.5) * sl[v];
    }
    flux(wl, 0, FL);
    flux(wr, 0, FR);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (kRcp && BN && v == 8) Qt[v] = src[v];  // the volume fraction has no flux
      else if constexpr (BN) Qt[v] = src[v] - divx(FR[v] - FL[v]);
      else Qt[v] = -divx(FR[v] - FL[v]);
      wLx[hx(v, ii, jj)] = wl[v];
      wRx[hx(v, ii, jj)] = wr[v];
    }
#pragma unroll
    for (int v = 0; v < V; ++v) sl[v] = slope_y(v);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      wl[v] = q0[v] - T(0.5) * sl[v];
      wr[v] = q0[v] + T(0.5) * sl[v];
    }
    flux(wl, 1, FL);
    flux(wr, 1, FR);
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (!(kRcp && BN && v == 8)) Qt[v] = Qt[v] - divy(FR[V + v] - FL[V + v]);
      if constexpr (BN) slt[hx(v, ii, jj)] = Qt[v];
      wLx[hx(v, ii, jj)] = wLx[hx(v, ii, jj)] + T(0.5) * dt * Qt[v];
      wRx[hx(v, ii, jj)] = wRx[hx(v, ii, jj)] + T(0.5) * dt * Qt[v];
      wLy[hx(v, ii, jj)] = wl[v] + T(0.5) * dt * Qt[v];
      wRy[hx(v, ii, jj)] = wr[v] + T(0.5) * dt * Qt[v];
    }
  }
  __syncthreads();

  // ---- edge fluxes Fx(1..S+1, 1..S), Fy(1..S, 1..S+1) (Euler/limiter.f90:571-588);
  // BN's four Rusanov fluxes per subcell (Baer-Nunziato/limiter.f90:526-545)
  // are those of its edges, each formed once here from the same states
  {
    T* EX = EF;
    T* EY = EF + (BN ? 2 : 1) * V * NE;
    for (int p = t; p < 2 * NE; p += NT) {
      const bool xd = p < NE;
      const int q = xd ? p : p - NE;
      T QL[V], QR[V], F[V], Dd[V];
      int ii, jj;
      if (xd) { ii = q % (S + 1) + 1; jj = q / (S + 1) + 1; }
      else { ii = q % S + 1; jj = q / S + 1; }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        QL[v] = xd ? wRx[hx(v, ii - 1, jj)] : wRy[hx(v, ii, jj - 1)];
        QR[v] = xd ? wLx[hx(v, ii, jj)] : wLy[hx(v, ii, jj)];
      }
      rusanov_s<Sys, T, kRcp>(pc, fcs, QL, QR, xd ? 0 : 1, F, Dd);
      T* dst = xd ? EX : EY;
#pragma unroll
      for (int v = 0; v < V; ++v) dst[v * NE + q] = F[v];
      if constexpr (BN) {
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (!kRcp || (v != 0 && v != 4)) dst[(V + v) * NE + q] = Dd[v];
      }
    }
    __syncthreads();
    for (int p = t; p < S * S; p += NT) {
      const int ii = p % S + 1, jj = p / S + 1;
      const int xp = ii + (S + 1) * (jj - 1), xm = (ii - 1) + (S + 1) * (jj - 1);
      const int yp = (ii - 1) + S * jj, ym = (ii - 1) + S * (jj - 1);
      // kRcp: EX, EY hold twice the flux
      const T fX = kRcp ? T(0.5) * divx(dt) : divx(dt), fY = kRcp ? T(0.5) * divy(dt) : divy(dt);
      if constexpr (!BN) {
        // first-order FV update, Euler/limiter.f90:592-597
#pragma unroll
        for (int v = 0; v < V; ++v)
          sub1[v * S * S + p] = SU(v, ii, jj) - fX * (EX[v * NE + xp] - EX[v * NE + xm]) -
                                fY * (EY[v * NE + yp] - EY[v * NE + ym]);
      } else {
        T qh[V], src[V];
#pragma unroll
        for (int v = 0; v < V; ++v) qh[v] = SU(v, ii, jj) + T(0.5) * dt * slt[hx(v, ii, jj)];
        ncp(qh, divx(sa8[ii + H * jj]), divy(sa8[H * H + ii + H * jj]), src);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if constexpr (kRcp) {
            // the fluctuation of an x (y) edge has no component along y (x),
            // nor in the two densities
            T q = SU(v, ii, jj) - fX * (EX[v * NE + xp] - EX[v * NE + xm]) - fY * (EY[v * NE + yp] - EY[v * NE + ym]);
            if (v != 0 && v != 2 && v != 4 && v != 6) q = q - fX * (EX[(V + v) * NE + xp] + EX[(V + v) * NE + xm]);
            if (v != 0 && v != 1 && v != 4 && v != 5) q = q - fY * (EY[(V + v) * NE + yp] + EY[(V + v) * NE + ym]);
            sub1[v * S * S + p] = v != 0 && v != 4 ? q + dt * src[v] : q;
          } else {
            sub1[v * S * S + p] = SU(v, ii, jj) - divx(dt) * (EX[v * NE + xp] - EX[v * NE + xm]) -
                                  divy(dt) * (EY[v * NE + yp] - EY[v * NE + ym]) -
                                  divx(dt) * T(0.5) * (EX[(V + v) * NE + xp] + EX[(V + v) * NE + xm]) -
                                  divy(dt) * T(0.5) * (EY[(V + v) * NE + yp] + EY[(V + v) * NE + ym]) +
                                  dt * src[v];
          }
        }
      }
    }
  }
