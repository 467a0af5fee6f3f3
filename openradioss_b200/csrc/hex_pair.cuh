// hex_pair.cuh -- the SFORC3 chain of two 8-node 1-point hexas at once in the split form,
// for the persistent cycle.
//
// A thread computes two hexas of a patch, one in each half of the packed FP32 type F2
// (sm_100 add/mul/fma.f32x2): a packed instruction does both elements' arithmetic in one
// issue slot at the same lane throughput (measured 126 lane-operations per clock and SM
// against 122 scalar), and a CTA holds twice the hexas of one per thread.  Each half rounds
// exactly like the scalar instruction.  Against hex_element the sums over corners and the
// face areas are arranged in fewer operations (below), so the two agree to rounding.
#pragma once

namespace orb {

// ---------------------------------------------------------------------------
// two floats in one 64-bit register pair
// ---------------------------------------------------------------------------
struct F2 { unsigned long long u; };
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float f2_get(F2 a, int i) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.u));
  return i ? y : x;
}
// ORB_IEEE: the parity build, without contraction and with denormals
#ifdef ORB_IEEE
#define ORB_F2(op) op ".f32x2 "
#else
#define ORB_F2(op) op ".ftz.f32x2 "
#endif
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm(ORB_F2("add.rn") "%0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm(ORB_F2("mul.rn") "%0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ F2 fma_(F2 a, F2 b, F2 c) {
#ifdef ORB_IEEE
  return a * b + c;
#else
  F2 r;
  asm(ORB_F2("fma.rn") "%0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
  return r;
#endif
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm(ORB_F2("sub.rn") "%0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
// a b - c d (a packed negation costs two instructions, a subtraction one)
__device__ __forceinline__ F2 mul_sub(F2 a, F2 b, F2 c, F2 d) { return a * b - c * d; }

// the values of a thread's two hexas
struct Pair {
  typedef F2 W;
  static constexpr int N = 2;
  static __device__ __forceinline__ F2 of(const float (&a)[2]) { return f2(a[0], a[1]); }
  static __device__ __forceinline__ F2 all(float a) { return f2(a, a); }
  static __device__ __forceinline__ float get(F2 a, int i) { return f2_get(a, i); }
  template <class F> static __device__ __forceinline__ F2 map(F f) { return f2(f(0), f(1)); }
};

// SCOOR3 / SRCOOR3 and the FP64 part of SDERI3 (sderi3.F:103-149, 264-298) of one hexa:
// the corner differences of the pairs 1-7, 2-8, 3-5, 4-6 and the coordinates relative to
// corner 1 are taken in FP64, then rounded to R: beyond the determinant nothing needs
// FP64, as in the reference's -prec=sp build, which forms the inverse Jacobian, the
// hourglass vectors and SDLEN3 in my_real.
struct HexGeom {
  typedef float R;
  R x[8][3];        // relative to corner 1 (x[0] = 0)
  R j[9];           // Jacobian terms
  R c[3];           // first cofactors
  double det;       // volume
  R fr[9];          // convected frame, columns e1 e2 e3 (CORO)
};
template <int CORO, class IO>
__device__ __forceinline__ void hex_geometry(const IO& io, const int i, const bool corot, HexGeom& g) {
  typedef float R;
  double X17, X28, X35, X46, Y17, Y28, Y35, Y46, Z17, Z28, Z35, Z46;
  if (CORO && corot) {
    double XD[8], YD[8], ZD[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double q[3];
      io.x(i, k, q);
      XD[k] = q[0]; YD[k] = q[1]; ZD[k] = q[2];
    }
    // SRCOOR3 (srcoor3.F, JCVT /= 0, ISORTH = 0): convected frame R = [e1 e2 e3] of
    // SREPISO3 (FP64 differences, r, s, t in R) and SORTHO3 (three symmetric
    // corrections, then Gram-Schmidt); coordinates (FP64) and velocities in it
    const R x17 = R(XD[6] - XD[0]), x28 = R(XD[7] - XD[1]), x35 = R(XD[4] - XD[2]), x46 = R(XD[5] - XD[3]);
    const R y17 = R(YD[6] - YD[0]), y28 = R(YD[7] - YD[1]), y35 = R(YD[4] - YD[2]), y46 = R(YD[5] - YD[3]);
    const R z17 = R(ZD[6] - ZD[0]), z28 = R(ZD[7] - ZD[1]), z35 = R(ZD[4] - ZD[2]), z46 = R(ZD[5] - ZD[3]);
    const R a17 = x17 + x46, a28 = x28 + x35, b17 = y17 + y46, b28 = y28 + y35, c17 = z17 + z46, c28 = z28 + z35;
    R Ux = x17 + x28 - x35 - x46, Uy = y17 + y28 - y35 - y46, Uz = z17 + z28 - z35 - z46;
    R Vx = a17 + a28, Vy = b17 + b28, Vz = c17 + c28;
    R Wx = a17 - a28, Wy = b17 - b28, Wz = c17 - c28;
    auto unit = [](R& x, R& y, R& z) {
      R aa = ssqrt(x * x + y * y + z * z);
      if (aa != R(0)) aa = R(1) / aa;
      x *= aa; y *= aa; z *= aa;
    };
    unit(Ux, Uy, Uz); unit(Vx, Vy, Vz); unit(Wx, Wy, Wz);
#pragma unroll
    for (int it = 0; it < 3; ++it) {
      R e1x = Vy * Wz - Vz * Wy + Ux, e1y = Vz * Wx - Vx * Wz + Uy, e1z = Vx * Wy - Vy * Wx + Uz;
      R e2x = Wy * Uz - Wz * Uy + Vx, e2y = Wz * Ux - Wx * Uz + Vy, e2z = Wx * Uy - Wy * Ux + Vz;
      R e3x = Uy * Vz - Uz * Vy + Wx, e3y = Uz * Vx - Ux * Vz + Wy, e3z = Ux * Vy - Uy * Vx + Wz;
      unit(e1x, e1y, e1z); unit(e2x, e2y, e2z); unit(e3x, e3y, e3z);
      Ux = e1x; Uy = e1y; Uz = e1z; Vx = e2x; Vy = e2y; Vz = e2z; Wx = e3x; Wy = e3y; Wz = e3z;
    }
    R e3x = Uy * Vz - Uz * Vy, e3y = Uz * Vx - Ux * Vz, e3z = Ux * Vy - Uy * Vx;
    unit(e3x, e3y, e3z);
    const R R11 = Ux, R21 = Uy, R31 = Uz;
    const R R12 = e3y * Uz - e3z * Uy, R22 = e3z * Ux - e3x * Uz, R32 = e3x * Uy - e3y * Ux;
    const R R13 = e3x, R23 = e3y, R33 = e3z;
    g.fr[0] = R11; g.fr[1] = R21; g.fr[2] = R31; g.fr[3] = R12; g.fr[4] = R22; g.fr[5] = R32;
    g.fr[6] = R13; g.fr[7] = R23; g.fr[8] = R33;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double xl = (double)R11 * XD[k] + (double)R21 * YD[k] + (double)R31 * ZD[k];
      const double yl = (double)R12 * XD[k] + (double)R22 * YD[k] + (double)R32 * ZD[k];
      const double zl = (double)R13 * XD[k] + (double)R23 * YD[k] + (double)R33 * ZD[k];
      XD[k] = xl; YD[k] = yl; ZD[k] = zl;
    }
    X17 = XD[6] - XD[0]; X28 = XD[7] - XD[1]; X35 = XD[4] - XD[2]; X46 = XD[5] - XD[3];
    Y17 = YD[6] - YD[0]; Y28 = YD[7] - YD[1]; Y35 = YD[4] - YD[2]; Y46 = YD[5] - YD[3];
    Z17 = ZD[6] - ZD[0]; Z28 = ZD[7] - ZD[1]; Z35 = ZD[4] - ZD[2]; Z46 = ZD[5] - ZD[3];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      g.x[k][0] = R(XD[k] - XD[0]); g.x[k][1] = R(YD[k] - YD[0]); g.x[k][2] = R(ZD[k] - ZD[0]);
    }
  } else {
    // corner 1 first, then the pairs, so that at most two corners are held in FP64
    double q0[3];
    io.x(i, 0, q0);
    const double x0 = q0[0], y0 = q0[1], z0 = q0[2];
    g.x[0][0] = R(0); g.x[0][1] = R(0); g.x[0][2] = R(0);
    auto ld = [&](int k, double& x, double& y, double& z) {
      double q[3];
      io.x(i, k, q);
      x = q[0]; y = q[1]; z = q[2];
      g.x[k][0] = R(x - x0); g.x[k][1] = R(y - y0); g.x[k][2] = R(z - z0);
    };
    double xk, yk, zk, xm, ym, zm;
    ld(6, xk, yk, zk);
    X17 = xk - x0; Y17 = yk - y0; Z17 = zk - z0;
    ld(1, xm, ym, zm); ld(7, xk, yk, zk);
    X28 = xk - xm; Y28 = yk - ym; Z28 = zk - zm;
    ld(2, xm, ym, zm); ld(4, xk, yk, zk);
    X35 = xk - xm; Y35 = yk - ym; Z35 = zk - zm;
    ld(3, xm, ym, zm); ld(5, xk, yk, zk);
    X46 = xk - xm; Y46 = yk - ym; Z46 = zk - zm;
  }
  const double J1 = X17 + X28 - X35 - X46, J2 = Y17 + Y28 - Y35 - Y46, J3 = Z17 + Z28 - Z35 - Z46;
  const double xa = X17 + X46, xb = X28 + X35, ya = Y17 + Y46, yb = Y28 + Y35, za = Z17 + Z46, zb = Z28 + Z35;
  const double J4 = xa + xb, J5 = ya + yb, J6 = za + zb, J7 = xa - xb, J8 = ya - yb, J9 = za - zb;
  const double C1 = J5 * J9 - J6 * J8, C4 = J6 * J7 - J4 * J9, C7 = J4 * J8 - J5 * J7;
  g.det = (1.0 / 64.0) * (J1 * C1 + J2 * C4 + J3 * C7);
  g.j[0] = R(J1); g.j[1] = R(J2); g.j[2] = R(J3); g.j[3] = R(J4); g.j[4] = R(J5); g.j[5] = R(J6);
  g.j[6] = R(J7); g.j[7] = R(J8); g.j[8] = R(J9);
  g.c[0] = R(C1); g.c[1] = R(C4); g.c[2] = R(C7);
}

// M2LAW's yield stress and hardening slope at plastic strain e (m2law.F:204-226)
__device__ __forceinline__ void hex_yield(const float e, const float CA, const float CB, const float CN, const float sigmax, const float epsmax,
                                          float& AK, float& QH, float& SIGY) {
  typedef float R;
  if (CN == R(1)) { AK = CA + CB * e; QH = CB; }
  else if (e > R(0)) {
    AK = CA + CB * pow_(e, CN);
    QH = (CN > R(1)) ? CB * CN * pow_(e, CN - R(1)) : CB * CN / pow_(e, R(1) - CN);
  } else { AK = CA; QH = R(0); }
  if (sigmax < AK) { AK = sigmax; QH = R(0); }
  SIGY = AK;
  if (e > epsmax) { AK = R(0); QH = R(0); }
}

// The corner pairs (1,7) (2,8) (3,5) (4,6) share a row of PX up to its sign.  With
// p_q = a_k1 + a_k2 and d_q = a_k1 - a_k2 of a quantity a, the four hourglass modes
// (+-+-+-+-), (++----++), (+--+-++-), (+-+--+-+) are
//   m1 = (p0 - p1) + (p2 - p3)   m2 = (p0 + p1) - (p2 + p3)
//   m3 = (p0 - p1) - (p2 - p3)   m4 = (d0 - d1) + (d2 - d3)
// and the pair's part of  sum_j s_jk H_j  (j = 1..3) over both its corners is
//   b0 = (H1 + H3) + H2   b1 = H2 - (H1 + H3)   b2 = (H1 - H3) - H2   b3 = -((H1 - H3) + H2)
// Against the sums written out corner by corner this takes 11 operations for three modes
// of a component instead of 21, and 18 for a component's forces instead of 36.
//
// SFORC3 of a thread's two hexas: SDERI3, SDLEN3, SDEFO3, SRHO3, SROTA3, M1LAW / M2LAW,
// MQVISCB, SHVIS3, SFINT3.  IO gives the state and takes the new state and the corner
// forces; act[i]: whether hexa i exists (the others' arithmetic is carried along unused).
// io.early(key, bits) hands in the thread's time step minimum as soon as it is known, every
// calling thread once.
template <int CORO, class IO>
__device__ __forceinline__ void hex_pair(const HexGroupDesc& gd, const bool (&act)[2], const float DT1, IO& io,
                                         ErrorWord* err, double& my_ehou, double& my_wpla) {
  typedef float R;
  typedef Pair K;
  typedef F2 W;
  constexpr int N = K::N;
  const bool corot = CORO && gd.jcvt;
  auto all = [](R a) { return K::all(a); };
  constexpr int pk1[4] = {0, 1, 2, 3}, pk2[4] = {6, 7, 4, 5};
  W x[8][3], fr[9];
  W PX[4], PY[4], PZ[4];
  W VOLN;
  double vold[N];
  {
    HexGeom g[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      hex_geometry<CORO>(io, i, corot, g[i]);
      if (!(g[i].det > 0.0)) {   // SCHKJABT3: zero or negative volume stops the run
        if (act[i]) raise_error(err, 4, io.eid(i));
        g[i].det = 1.0;
      }
      vold[i] = g[i].det;
    }
#pragma unroll
    for (int k = 1; k < 8; ++k)
#pragma unroll
      for (int c = 0; c < 3; ++c) x[k][c] = K::map([&](int i) { return g[i].x[k][c]; });
    if (CORO) {
#pragma unroll
      for (int k = 0; k < 9; ++k) fr[k] = K::map([&](int i) { return g[i].fr[k]; });
    }
    VOLN = K::map([&](int i) { return R(g[i].det); });
    const W dett = K::map([&](int i) { return R(1.0 / 64.0) / R(g[i].det); });
    W j[9], c[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) j[k] = K::map([&](int i) { return g[i].j[k]; });
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = K::map([&](int i) { return g[i].c[k]; });
    auto minor = [&](int a, int b, int p, int q) { return mul_sub(j[a], j[b], j[p], j[q]); };
    const W I1 = dett * c[0], I4 = dett * c[1], I7 = dett * c[2];
    const W I2 = dett * minor(2, 7, 1, 8), I5 = dett * minor(0, 8, 2, 6), I8 = dett * minor(1, 6, 0, 7);
    const W I3 = dett * minor(1, 5, 2, 4), I6 = dett * minor(2, 3, 0, 5), I9 = dett * minor(0, 4, 1, 3);
    const W a12 = I1 + I2, a45 = I4 + I5, a78 = I7 + I8;
    const W b12 = I1 - I2, b45 = I4 - I5, b78 = I7 - I8;
    const W zero = all(R(0));
    PX[0] = (zero - a12) - I3; PY[0] = (zero - a45) - I6; PZ[0] = (zero - a78) - I9;
    PX[1] = I3 - a12; PY[1] = I6 - a45; PZ[1] = I9 - a78;
    PX[2] = b12 + I3; PY[2] = b45 + I6; PZ[2] = b78 + I9;
    PX[3] = b12 - I3; PY[3] = b45 - I6; PZ[3] = b78 - I9;
  }
  // hourglass projections PXiHj (sderi3.F:302-333); the mode vectors sum to zero, so
  // relative coordinates give the same products
  W PXH[4][3];
  {
    W h[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const W p0 = x[6][c], p1 = x[1][c] + x[7][c], p2 = x[2][c] + x[4][c], p3 = x[3][c] + x[5][c];
      const W m = p0 - p1, n = p2 - p3;
      h[0][c] = m + n;
      h[1][c] = (p0 + p1) - (p2 + p3);
      h[2][c] = m - n;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int jj = 0; jj < 3; ++jj) PXH[q][jj] = fma_(PZ[q], h[jj][2], fma_(PY[q], h[jj][1], PX[q] * h[jj][0]));
  }
  // ---- SDLEN3 / SLEN (sdlen3.F:110-166): 4 V / sqrt(max face (E G - F^2)).  With the
  // face's diagonals a, b the reference's E, F, G belong to a - b and a + b, so that
  // E G - F^2 = |(a - b) x (a + b)|^2 = 4 |a x b|^2 ----
  W DELTAX;
  {
    constexpr int FC[6][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {0, 1, 5, 4}, {1, 2, 6, 5}, {2, 3, 7, 6}, {3, 0, 4, 7}};
    R am[N];
#pragma unroll
    for (int i = 0; i < N; ++i) am[i] = R(EM20) * R(0.25);
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      W a[3], b[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        a[c] = FC[f][0] == 0 ? x[FC[f][2]][c] : x[FC[f][2]][c] - x[FC[f][0]][c];
        b[c] = FC[f][1] == 0 ? x[FC[f][3]][c] : x[FC[f][3]][c] - x[FC[f][1]][c];
      }
      const W n0 = mul_sub(a[1], b[2], a[2], b[1]), n1 = mul_sub(a[2], b[0], a[0], b[2]),
              n2 = mul_sub(a[0], b[1], a[1], b[0]);
      const W ar = fma_(n0, n0, fma_(n1, n1, n2 * n2));
#pragma unroll
      for (int i = 0; i < N; ++i) { const R v = K::get(ar, i); am[i] = v > am[i] ? v : am[i]; }
    }
    DELTAX = K::map([&](int i) { return R(2) * K::get(VOLN, i) / ssqrt(am[i]); });
  }
  // ---- SDEFO3 (sdefo3.F:114-170, JHBE=1) and the hourglass velocity modes of SHVIS3:
  // sum_k g_jk v_k  with g_jk = s_jk -+ PXH is the mode of v less  sum_q PXH[q][j] d_q ----
  W DXX, DYY, DZZ, DXY, DXZ, DYX, DYZ, DZX, DZY;
  W HG[3][4];                     // component, mode
  {
    W s01[3], m01[3], pp[3];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      W u1[3], u2[3];
      {
        R v1[N][3], v2[N][3];
#pragma unroll
        for (int i = 0; i < N; ++i) { io.v(i, pk1[q], v1[i]); io.v(i, pk2[q], v2[i]); }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          u1[c] = K::map([&](int i) { return v1[i][c]; });
          u2[c] = K::map([&](int i) { return v2[i][c]; });
        }
      }
      if (CORO && corot) {
        W a[3], b[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          a[c] = fma_(fr[3 * c + 2], u1[2], fma_(fr[3 * c + 1], u1[1], fr[3 * c] * u1[0]));
          b[c] = fma_(fr[3 * c + 2], u2[2], fma_(fr[3 * c + 1], u2[1], fr[3 * c] * u2[0]));
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) { u1[c] = a[c]; u2[c] = b[c]; }
      }
      const W dx = u1[0] - u2[0], dy = u1[1] - u2[1], dz = u1[2] - u2[2];
      if (q == 0) {
        DXX = PX[0] * dx; DYY = PY[0] * dy; DZZ = PZ[0] * dz;
        DXY = PY[0] * dx; DXZ = PZ[0] * dx; DYX = PX[0] * dy;
        DYZ = PZ[0] * dy; DZX = PX[0] * dz; DZY = PY[0] * dz;
      } else {
        DXX = fma_(PX[q], dx, DXX); DYY = fma_(PY[q], dy, DYY); DZZ = fma_(PZ[q], dz, DZZ);
        DXY = fma_(PY[q], dx, DXY); DXZ = fma_(PZ[q], dx, DXZ); DYX = fma_(PX[q], dy, DYX);
        DYZ = fma_(PZ[q], dy, DYZ); DZX = fma_(PX[q], dz, DZX); DZY = fma_(PY[q], dz, DZY);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const W p = u1[c] + u2[c], d = c == 0 ? dx : c == 1 ? dy : dz;
        if (q == 0) {
          pp[c] = p;
          HG[c][3] = d;
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) HG[c][jj] = PXH[0][jj] * d;
        } else {
          HG[c][3] = (q & 1) ? HG[c][3] - d : HG[c][3] + d;
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) HG[c][jj] = fma_(PXH[q][jj], d, HG[c][jj]);
          if (q == 1) { s01[c] = pp[c] + p; m01[c] = pp[c] - p; }
          else if (q == 2) pp[c] = p;
          else {
            const W s23 = pp[c] + p, m23 = pp[c] - p;
            HG[c][0] = (m01[c] + m23) - HG[c][0];
            HG[c][1] = (s01[c] - s23) - HG[c][1];
            HG[c][2] = (m01[c] - m23) - HG[c][2];
          }
        }
      }
    }
  }
  const W D4 = DXY + DYX, D5 = DYZ + DZY, D6 = DXZ + DZX;
  const W half = all(R(0.5) * DT1);
  const W WZZ = half * (DYX - DXY), WYY = half * (DXZ - DZX), WXX = half * (DZY - DYZ);
  // ---- SRHO3 (srho3.F:122-156; FP64 volume ratios, srho3.F:230-245) ----
  const R RHO0 = R(gd.rho0);
  const W rho_old = io.rho();
  const W VOLO = io.vol0();
  W DVOL, RHON, AMU;
  {
    R dv[N], rn[N], mu[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const double v0 = io.vol0dp(i);
      dv[i] = R(vold[i] - ((double)RHO0 / (double)K::get(rho_old, i)) * v0);
      const double ratio = v0 / vold[i];
      rn[i] = R((double)RHO0 * ratio);
      mu[i] = R(ratio - 1.0);
    }
    DVOL = K::of(dv); RHON = K::of(rn); AMU = K::of(mu);
  }
  W EINT = io.eint() * VOLO;
  // ---- SROTA3 Jaumann rotation (srota3.F:81-91) ----
  const W S1 = io.sig(0), S2 = io.sig(1), S3 = io.sig(2), S4 = io.sig(3), S5 = io.sig(4), S6 = io.sig(5);
  W SG[6];
  if (CORO && corot) {          // SRMALLA3 (srmall3.F): convected-frame stress, not rotated
    SG[0] = S1; SG[1] = S2; SG[2] = S3; SG[3] = S4; SG[4] = S5; SG[5] = S6;
  } else {
    const W two = all(R(2));
    const W q1 = two * S4 * WZZ, q2 = two * S6 * WYY, q3 = two * S5 * WXX;
    SG[0] = S1 - q1 + q2;
    SG[1] = S2 + q1 - q3;
    SG[2] = S3 - q2 + q3;
    SG[3] = fma_(WYY, S5, fma_(WZZ, S1 - S2, S4)) - WXX * S6;
    SG[4] = fma_(WZZ, S6, fma_(WXX, S2 - S3, S5)) - WYY * S4;
    SG[5] = fma_(WXX, S4, fma_(WYY, S3 - S1, S6)) - WZZ * S5;
  }
  const W VOL_AVG = fma_(all(R(-0.5)), DVOL, VOLN);
  const W QOLD = io.qvis();
  const W EPXE = io.pla();
  // ---- elastic predictor (m1law.F:124-140 / m2law.F:187-200) ----
  const R Gs = R(gd.shear);
  const R G1 = DT1 * Gs;
  const R SSP = ssqrt((R(1.333) * Gs + R(gd.bulk)) / RHO0);
  {
    const W third = all(-R(1.0 / 3.0)), g1 = all(G1), g2 = all(R(2) * G1);
    const W P = third * (SG[0] + SG[1] + SG[2]);
    const W DAV = third * (DXX + DYY + DZZ);
    SG[0] = fma_(g2, DXX + DAV, SG[0] + P);
    SG[1] = fma_(g2, DYY + DAV, SG[1] + P);
    SG[2] = fma_(g2, DZZ + DAV, SG[2] + P);
    SG[3] = fma_(g1, D4, SG[3]);
    SG[4] = fma_(g1, D5, SG[4]);
    SG[5] = fma_(g1, D6, SG[5]);
  }
  W DPLA = all(R(0)), SIGY = all(R(0));
  if (gd.law == 2) {
    // ---- M2LAW radial return (m2law.F:197-352), CC=0, FISOKIN=0 ----
    W AJ2 = fma_(all(R(0.5)), fma_(SG[2], SG[2], fma_(SG[1], SG[1], SG[0] * SG[0])),
                 fma_(SG[5], SG[5], fma_(SG[4], SG[4], SG[3] * SG[3])));
    AJ2 = K::map([&](int i) { return ssqrt(R(3) * K::get(AJ2, i)); });
    {   // MSTRAIN_RATE, ISRATE = 0, total strain rate
      const W e2 = fma_(D6, D6, fma_(D5, D5, D4 * D4));
      const W ee = fma_(all(R(0.5)), e2, fma_(DZZ, DZZ, fma_(DYY, DYY, DXX * DXX)));
      io.put_epsd(K::map([&](int i) { return ssqrt(K::get(ee, i)); }));
    }
    R ak[N], qh[N], sy[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
      hex_yield(K::get(EPXE, i), R(gd.jc_a), R(gd.jc_b), R(gd.jc_n), R(gd.sigmax), R(gd.epsmax), ak[i], qh[i], sy[i]);
    W AK = K::of(ak);
    const W QH = K::of(qh);
    auto ratio = [&](const W& a) {       // min(1, a / AJ2)
      return K::map([&](int i) {
        const R aj = K::get(AJ2, i);
        const R s = K::get(a, i) / (aj > R(EM15) ? aj : R(EM15));
        return s < R(1) ? s : R(1);
      });
    };
    W SCALE = ratio(AK);
    const W num = (all(R(1)) - SCALE) * AJ2;
    DPLA = K::map([&](int i) {
      const R den = R(3) * Gs + qh[i];
      return K::get(num, i) / (den > R(EM15) ? den : R(EM15));
    });
    AK = fma_(DPLA, QH, AK);
    SCALE = ratio(AK);
#pragma unroll
    for (int c = 0; c < 6; ++c) SG[c] = SCALE * SG[c];
    io.put_pla(EPXE + DPLA);
    SIGY = K::map([&](int i) { const R a = K::get(AK, i); return sy[i] > a ? sy[i] : a; });
  }
  // ---- MQVISCB (mqviscb.F:139-354) ----
  const W AL = K::map([&](int i) { const R v = K::get(VOLN, i); return v > R(0) ? cbrt_(v) : R(0); });
  W QNEW;
  {
    const W div = DXX + DYY + DZZ;
    const W AD = K::map([&](int i) { const R d = -K::get(div, i); return d > R(0) ? d : R(0); });
    const R QA = R(gd.qa), QB = R(gd.qb);
    const W QAA = all(QA * QA) * AD;
    const W qs = all(QB * SSP);
    const W QX = fma_(AL, QAA, qs);
    QNEW = RHON * AD * AL * fma_(QAA, AL, qs);
    const W r2 = fma_(QX, QX, all(SSP * SSP));
    unsigned long long mykey = ~0ull, mybits = ~0ull;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      R eq = K::get(QX, i) + ssqrt(K::get(r2, i));
      eq = eq > R(EM20) ? eq : R(EM20);
      const R DTX = R(gd.dtfac) * (K::get(DELTAX, i) / eq);
      if (!act[i]) continue;
      if ((double)DTX <= gd.dtmin) raise_error(err, 5, io.eid(i));
      const double dtd = (double)DTX;
      const unsigned long long key = dt_key(dtd, 1, io.eid(i)), bits = (unsigned long long)__double_as_longlong(dtd);
      mykey = key < mykey ? key : mykey;
      mybits = bits < mybits ? bits : mybits;
    }
    io.early(mykey, mybits);
  }
  // ---- pressure and internal energy (m1law.F:172-190 / m2law.F:434-461) ----
  {
    const W PNEW = all(R(gd.bulk)) * AMU;
    SG[0] = SG[0] - PNEW; SG[1] = SG[1] - PNEW; SG[2] = SG[2] - PNEW;
    W t1 = S1 + SG[0], t2 = S2 + SG[1], t3 = S3 + SG[2];
    W visc = QOLD + QNEW;
    if (gd.law == 1) {
      const W P2 = all(-R(1.0 / 3.0)) * (t1 + t2 + t3);
      t1 = t1 + P2; t2 = t2 + P2; t3 = t3 + P2;
      visc = visc + P2;
    }
    W EINC = fma_(D6, S6 + SG[5], fma_(D5, S5 + SG[4], fma_(D4, S4 + SG[3], fma_(DZZ, t3, fma_(DYY, t2, DXX * t1)))));
    EINC = fma_(VOL_AVG * EINC, half, all(R(-0.5)) * DVOL * visc);
    EINT = EINT + EINC;
    io.put_eint(K::map([&](int i) {
      const R vo = K::get(VOLO, i);
      return K::get(EINT, i) / (vo > R(EM15) ? vo : R(EM15));
    }));
    if (gd.law != 1) {
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (act[i]) my_wpla += (double)K::get(SIGY, i) * (double)K::get(DPLA, i) * (double)K::get(VOLN, i);
    }
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) io.put_sig(c, SG[c]);
  io.put_rho(RHON);
  io.put_qvis(QNEW);
  // ---- SHVIS3 Flanagan-Belytschko viscous hourglass (shvis3.F:156-424, JHBE>=1): HG
  // becomes the mode forces ----
  {
    const W caq = all(R(0.25) * R(gd.qh));
    W FCL = caq * RHON * (AL * AL);   // VOL**TWO_THIRD
    const W FCQ = FCL * caq * all(R(100));
    FCL = FCL * all(SSP);
    W ehou = all(R(0));
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const W g = HG[c][jj];
        const W ab = K::map([&](int i) { return R(fabs(K::get(g, i))); });
        const W f = g * fma_(ab, FCQ, FCL);
        ehou = fma_(f, g, ehou);
        HG[c][jj] = f;
      }
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (act[i]) my_ehou += (double)(DT1 * K::get(ehou, i));
  }
  // ---- SFINT3 (sfint3.F:256-321): corner k1 of a pair gets -f_q, corner k2 +f_q, added
  // to the hourglass force  -sum_j g_jk H_j - h4_k H_4 ----
  const W s1 = (SG[0] - QNEW) * VOLN, s2 = (SG[1] - QNEW) * VOLN, s3 = (SG[2] - QNEW) * VOLN;
  const W s4 = SG[3] * VOLN, s5 = SG[4] * VOLN, s6 = SG[5] * VOLN;
  W base[3][2];
#pragma unroll
  for (int c = 0; c < 3; ++c) { base[c][0] = HG[c][0] + HG[c][2]; base[c][1] = HG[c][0] - HG[c][2]; }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k1 = pk1[q], k2 = pk2[q];
    W f1[3], f2_[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const W ta = c == 0 ? s1 : c == 1 ? s4 : s6, tb = c == 0 ? s4 : c == 1 ? s2 : s5, tc = c == 0 ? s6 : c == 1 ? s5 : s3;
      const W st = fma_(tc, PZ[q], fma_(tb, PY[q], ta * PX[q]));
      // antisymmetric part: PXH . H, the 4th mode and the stress term
      W u = fma_(PXH[q][2], HG[c][2], fma_(PXH[q][1], HG[c][1], PXH[q][0] * HG[c][0])) - st;
      u = (q & 1) ? u + HG[c][3] : u - HG[c][3];
      const W b = q == 0 ? (all(R(0)) - base[c][0]) - HG[c][1] : q == 1 ? base[c][0] - HG[c][1]
                  : q == 2 ? HG[c][1] - base[c][1] : base[c][1] + HG[c][1];
      f1[c] = b + u;
      f2_[c] = b - u;
    }
    if (CORO && corot) {        // SRROTA3 with R transposed (sforc3.F:1603-1614): back to global axes
      W a[3], b[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        a[c] = fma_(fr[6 + c], f1[2], fma_(fr[3 + c], f1[1], fr[c] * f1[0]));
        b[c] = fma_(fr[6 + c], f2_[2], fma_(fr[3 + c], f2_[1], fr[c] * f2_[0]));
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) { f1[c] = a[c]; f2_[c] = b[c]; }
    }
    io.corner(k1, f1);
    io.corner(k2, f2_);
  }
}

}  // namespace orb
