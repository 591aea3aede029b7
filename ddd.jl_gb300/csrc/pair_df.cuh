// General branch of the non-singular segment-segment force in df64 arithmetic
// (double-float on the FP32 pipes).  Same formulas and evaluation order as the
// FP64 kernel (pair_f64.cuh), i.e. as DislocationForces.jl:879-1165 and
// SegSegInteg :1480-1561, with every scalar a df64.
#pragma once
#include "df64.cuh"

namespace ddd {

struct DV3 {
  df64 x, y, z;
};
DF_HD DV3 operator+(DV3 a, DV3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
DF_HD DV3 operator-(DV3 a, DV3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
DF_HD DV3 operator-(DV3 a) { return {-a.x, -a.y, -a.z}; }
DF_HD DV3 operator*(df64 s, DV3 a) { return {s * a.x, s * a.y, s * a.z}; }
DF_HD DV3 operator*(DV3 a, df64 s) { return {a.x * s, a.y * s, a.z * s}; }
DF_HD df64 dot(DV3 a, DV3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
DF_HD DV3 cross(DV3 a, DV3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }

struct KConstsDF {
  df64 aSq, mu4pi, mu4pinu, mu8piaSq, mu4pinuaSq;
};

// The integration domain of a general pair and its 19 integrals,
// ((I(x1,y1) - I(x1,y2)) - I(x2,y1)) + I(x2,y2) (SegSegInteg,
// DislocationForces.jl:1480-1561), in two loops of packed df64:
//   * Ra, 1/Ra and the arctangent integral, two corners per iteration (lanes
//     (x, y1) and (x, y2));
//   * the rest, one corner per iteration, with the mirrored quantities of the
//     formulas in the lanes: R_t1 | R_t2, x | y, integ2 | integ3, integ6 | integ5,
//     integ 7 | 8, 10 | 11, 12 | 13, 15 | 16 and 17 | 18 (0-based, as stored).
// Each lane does the scalar formula's operations, so the bits are the scalar's.
//
// Why two loops: a warp runs ~8,000 instructions per pair.  An SM's sub-core
// holds 2,048 of them (32 KB); past that all four share 1.5 fetched instructions
// per cycle (both measured), and one straight body for two whole corners ran at
// exactly that (ncu: 33 % of the warp cycles without an instruction).  These
// bodies are ~400 and ~1,000 instructions, fetched once per pair and run two and
// four times.
struct PairDF {
  df64 c, d, x1, x2, y1, y2, integ[19];
};
DF_HD void pair_integrals_df(df64 aSq, DV3 t1, DV3 n11, DV3 n12, DV3 t2, DV3 n21, DV3 n22, df64 c, PairDF& out) {
  const df64 cSq = c * c;
  const df64 omcSq = df(1.0f) - cSq;
  const df64 omcSqI = df_recip(omcSq);
  // Lanes: R1 = n21 - n11 and R2 = n22 - n12.
  auto two = [](df64 a, df64 b) { return df2_make(a, b); };
  const df2 Rx = two(n21.x, n22.x) - two(n11.x, n12.x), Ry = two(n21.y, n22.y) - two(n11.y, n12.y),
            Rz = two(n21.z, n22.z) - two(n11.z, n12.z);
  const df2 lim1 = Rx * df2_dup(t1.x) + Ry * df2_dup(t1.y) + Rz * df2_dup(t1.z);
  const df2 lim2 = Rx * df2_dup(t2.x) + Ry * df2_dup(t2.y) + Rz * df2_dup(t2.z);
  const df2 C = df2_dup(c), CSq = df2_dup(cSq), Q = df2_dup(omcSqI);
  const df2 xs = (lim2 - C * lim1) * Q, ys = (lim1 - C * lim2) * Q;
  const DV3 t2ct1 = cross(t2, t1);
  struct {
    df64 d, x1, x2, y1, y2;
  } g;
  g.d = (df2_y(Rx) * t2ct1.x + df2_y(Ry) * t2ct1.y + df2_y(Rz) * t2ct1.z) * omcSqI;
  g.x1 = df2_x(xs);
  g.x2 = df2_y(xs);
  g.y1 = df2_x(ys);
  g.y2 = df2_y(ys);
  const df64 aSq_dSq = aSq + g.d * g.d * omcSq;
  const df64 aSq_dSqI = df_recip(aSq_dSq);
  const df64 den = df_recip(df_sqrt(omcSq * aSq_dSq));

  df2 Ras[2], RaIs[2], ats[2];
  {
    const df2 A = df2_dup(aSq_dSq), D = df2_dup(den), M = df2_dup(df_scale(-den, 2.0f)), C1 = df2_dup(df(1.0f) + c);
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int q = 0; q < 2; ++q) {
      const df2 x = df2_dup(q ? g.x2 : g.x1);
      const df2 R = df_sqrt(A + x * x + ys * ys + df_scale(x, 2.0f) * ys * C);
      const df2 RI = df_recip(R), at = M * df_atan(C1 * (R + x + ys) * D);
      if (q == 0) {
        Ras[0] = R;
        RaIs[0] = RI;
        ats[0] = at;
      } else {
        Ras[1] = R;
        RaIs[1] = RI;
        ats[1] = at;
      }
    }
  }

  df64 s0 = df(0.0f), s3 = s0, s6 = s0, s9 = s0, s14 = s0;
  const df2 zero = {f2_dup(0.0f), f2_dup(0.0f)};
  df2 s12 = zero, s54 = zero, s78 = zero, sab = zero, scd = zero, sfg = zero, shi = zero;
#ifdef __CUDACC__
#pragma unroll 1
#endif
  for (int q = 0; q < 4; ++q) {
    auto pick = [&](const df2* v) {
      const df2 w = q & 2 ? v[1] : v[0];
      return q & 1 ? df2_y(w) : df2_x(w);
    };
    const df64 Ra = pick(Ras), RaInv = pick(RaIs), integ1 = pick(ats);
    const df2 X = df2_make(q & 2 ? g.x2 : g.x1, q & 1 ? g.y2 : g.y1), Y = df2_swap(X);
    const df2 RI = df2_dup(RaInv);
    const df2 Rt = df2_dup(Ra) + Y + X * C;  // Ra_Rd_t1 | t2
    const df2 L = df_log(Rt);
    const df2 XL = X * L;
    const df2 S = RI / Rt;  // RaSq_R_t1_I | t2
    const df2 XS = X * S, XXS = X * XS;

    const df64 c_1 = aSq_dSq * integ1;
    const df2 c56i4 = (C * df2_make(Ra, c_1) - df2_make(c_1, Ra)) * Q;  // c_5_6 | integ4
    const df64 integ4 = df2_y(c56i4);
    const df2 i23 = (C * df2_swap(L) - L) * Q;         // integ2 | integ3
    const df2 i65 = XL + df2_dup(df2_x(c56i4));        // integ6 | integ5
    const df2 C11 = df2_dup(integ1 - c * RaInv);       // c_11_12
    const df2 K = C * XS - RI;                         // c_15_18 | c_19
    const df2 D = L - (Y - C * X) * RI - CSq * XXS;    // c_17_19 | c_16
    const df2 XD = X * D;                              // x c_17_19 | z_15_18
    const df2 T = df2_dup(df_scale(integ4, 2.0f));     // c15_18_19
    const df2 XSs = df2_swap(XS);

    const df64 v6 = (integ1 - df2_x(XS) - df2_y(XS)) * aSq_dSqI;
    const df2 v78 = (S - C * df2_swap(S)) * Q;
    const df64 v9 = (RaInv - c * (df2_x(XS) + df2_y(XS) + integ1)) * omcSqI;
    const df2 vab = (XS + CSq * XSs + C11) * Q;
    const df2 W = df2_swap(i23) - X * K;  // integ3 - x_13_14 | integ2 - y_13_14
    const df2 vcd = (W - C * df2_swap(W)) * Q;
    const df2 G = T - X * X * K;          // c15_18_19 - xSq c_15_18 | ... - ySq c_19
    const df2 H = XD - i65;               // x c_17_19 - integ6 | z_15_18 - integ5
    const df2 vhi = (G + C * df2_swap(H)) * Q;
    const df64 v14 = (df2_y(H) + c * df2_x(G)) * omcSqI;  // -integ 14
    const df2 vfg = (XXS + C * df2_swap(D) + df_scale(i23, 2.0f)) * Q;

    // The corners' signs (+, -, -, +) as a factor: one body for all.
    const float sg = q == 1 || q == 2 ? -1.0f : 1.0f;
    const f2 sg2 = f2_dup(sg);
    auto add1 = [&](df64& a, df64 v) { a = a + df_scale(v, sg); };
    auto add2 = [&](df2& a, df2 v) { a = a + df2{v.hi * sg2, v.lo * sg2}; };
    add1(s0, integ1);
    add1(s3, integ4);
    add1(s6, v6);
    add1(s9, v9);
    add1(s14, -v14);
    add2(s12, i23);
    add2(s54, i65);
    add2(s78, v78);
    add2(sab, vab);
    add2(scd, vcd);
    add2(sfg, vfg);
    add2(shi, vhi);
  }
  out.c = c;
  out.d = g.d;
  out.x1 = g.x1;
  out.x2 = g.x2;
  out.y1 = g.y1;
  out.y2 = g.y2;
  const df64 all[19] = {s0,         df2_x(s12), df2_y(s12), s3,         df2_y(s54), df2_x(s54), s6,
                        df2_x(s78), df2_y(s78), s9,         df2_x(sab), df2_y(sab), df2_x(scd), df2_y(scd),
                        s14,        df2_x(sfg), df2_y(sfg), df2_x(shi), df2_y(shi)};
#pragma unroll
  for (int k = 0; k < 19; ++k) out.integ[k] = all[k];
}

DF_HD DV3 fsum11_df(const DV3* V, const df64* F) {
  DV3 s = V[0] * F[0] + V[1] * F[1];
#pragma unroll
  for (int k = 2; k < 11; ++k) s = s + V[k] * F[k];
  return s;
}

// The node forces of the general branch from its integrals, in df64 (forces on
// seg 1 if NEED12, seg 2 if NEED34).
template <bool NEED12, bool NEED34>
DF_HD void assemble_df(const KConstsDF& K, const PairDF& g, DV3 b1, DV3 t1, df64 t1N, DV3 b2, DV3 t2, df64 t2N, DV3& F1,
                       DV3& F2, DV3& F3, DV3& F4) {
  const df64 c = g.c, d = g.d, x1 = g.x1, x2 = g.x2, y1 = g.y1, y2 = g.y2;
  const df64* integ = g.integ;
  const df64 mu4pi = K.mu4pi, mu4pinu = K.mu4pinu, mu8piaSq = K.mu8piaSq, mu4pinuaSq = K.mu4pinuaSq;
  DV3 t2ct1 = cross(t2, t1);
  DV3 t1ct2 = -t2ct1;
  DV3 b2ct2 = cross(b2, t2);
  DV3 b1ct1 = cross(b1, t1);

  df64 t2db2 = dot(t2, b2);
  df64 t2db1 = dot(t2, b1);
  df64 t1db2 = dot(t1, b2);
  df64 t1db1 = dot(t1, b1);

  df64 t2ct1db2 = dot(t2ct1, b2);
  df64 t1ct2db1 = dot(t1ct2, b1);
  df64 b1ct1db2 = dot(b1ct1, b2);
  df64 b2ct2db1 = dot(b2ct2, b1);

  DV3 t2ct1ct2 = t1 - c * t2;
  DV3 t1ct2ct1 = t2 - c * t1;
  DV3 t2cb1ct2 = b1 - t2db1 * t2;
  DV3 t1cb2ct1 = b2 - t1db2 * t1;
  DV3 b1ct1ct2 = t2db1 * t1 - c * b1;
  DV3 b2ct2ct1 = t1db2 * t2 - c * b2;

  df64 t2ct1cb1dt1 = t2db1 - t1db1 * c;
  df64 t1ct2cb2dt2 = t1db2 - t2db2 * c;
  df64 t2ct1cb1db2 = t2db1 * t1db2 - t1db1 * t2db2;

  df64 mu4pid = mu4pi * d;
  df64 mu4pinud = mu4pinu * d;
  df64 mu4pinudSq = mu4pinud * d;
  df64 mu4pinudCu = mu4pinudSq * d;
  df64 mu4pinuaSqd = mu4pinuaSq * d;
  df64 mu8piaSqd = mu8piaSq * d;

  DV3 V[11];
  df64 Fi[11];
  df64 tmp1, tmp2;
  if (NEED12) {
    tmp1 = t1db2 * t2db1 + t2ct1cb1db2;
    DV3 V1 = tmp1 * t2ct1;
    DV3 V2 = b1ct1 * t1ct2cb2dt2;
    DV3 V3 = t1ct2 * b1ct1db2 - t1cb2ct1 * t2db1;
    DV3 V4 = -b1ct1 * t2ct1db2;
    DV3 V5 = b2ct2ct1 * t2db1 - t1ct2 * b2ct2db1;

    tmp1 = mu4pinud * t1ct2db1;
    tmp2 = mu4pinud * b2ct2db1;
    V[0] = mu4pid * V1 - mu4pinud * V2 + tmp1 * b2ct2ct1 + tmp2 * t1ct2ct1;
    tmp1 = mu4pinu * t2db1;
    tmp2 = mu4pinu * b2ct2db1;
    V[1] = mu4pi * V5 - tmp1 * b2ct2ct1 + tmp2 * t1ct2;
    tmp1 = mu4pinu * t1db1;
    V[2] = -tmp1 * b2ct2ct1 + mu4pi * V3 - mu4pinu * V4;
    tmp1 = mu4pinudCu * t1ct2cb2dt2 * t1ct2db1;
    V[3] = mu8piaSqd * V1 - mu4pinuaSqd * V2 - tmp1 * t1ct2ct1;
    tmp1 = mu4pinudSq * t1ct2cb2dt2 * t2db1;
    tmp2 = mu4pinudSq * t1ct2cb2dt2 * t1ct2db1;
    V[4] = mu8piaSq * V5 + tmp1 * t1ct2ct1 - tmp2 * t1ct2;
    tmp1 = mu4pinudSq * (t2ct1db2 * t1ct2db1 + t1ct2cb2dt2 * t1db1);
    V[5] = mu8piaSq * V3 - mu4pinuaSq * V4 + tmp1 * t1ct2ct1;
    tmp1 = mu4pinud * (t1ct2cb2dt2 * t1db1 + t2ct1db2 * t1ct2db1);
    tmp2 = mu4pinud * t2ct1db2 * t2db1;
    V[6] = tmp1 * t1ct2 - tmp2 * t1ct2ct1;
    tmp1 = mu4pinud * t1ct2cb2dt2 * t2db1;
    V[7] = tmp1 * t1ct2;
    tmp1 = mu4pinud * t2ct1db2 * t1db1;
    V[8] = -tmp1 * t1ct2ct1;
    DV3 tv = mu4pinu * t2ct1db2 * t1ct2;
    V[9] = -tv * t2db1;
    V[10] = -tv * t1db1;

    Fi[0] = integ[2] - y2 * integ[0];
    Fi[1] = integ[3] - y2 * integ[1];
    Fi[2] = integ[5] - y2 * integ[2];
    Fi[3] = integ[8] - y2 * integ[6];
    Fi[4] = integ[9] - y2 * integ[7];
    Fi[5] = integ[11] - y2 * integ[8];
    Fi[6] = integ[13] - y2 * integ[9];
    Fi[7] = integ[12] - y2 * integ[10];
    Fi[8] = integ[16] - y2 * integ[11];
    Fi[9] = integ[14] - y2 * integ[12];
    Fi[10] = integ[18] - y2 * integ[13];
    F1 = fsum11_df(V, Fi) * t1N;

    Fi[0] = y1 * integ[0] - integ[2];
    Fi[1] = y1 * integ[1] - integ[3];
    Fi[2] = y1 * integ[2] - integ[5];
    Fi[3] = y1 * integ[6] - integ[8];
    Fi[4] = y1 * integ[7] - integ[9];
    Fi[5] = y1 * integ[8] - integ[11];
    Fi[6] = y1 * integ[9] - integ[13];
    Fi[7] = y1 * integ[10] - integ[12];
    Fi[8] = y1 * integ[11] - integ[16];
    Fi[9] = y1 * integ[12] - integ[14];
    Fi[10] = y1 * integ[13] - integ[18];
    F2 = fsum11_df(V, Fi) * t1N;
  }
  if (NEED34) {
    tmp1 = t2db1 * t1db2 + t2ct1cb1db2;
    DV3 V1 = tmp1 * t1ct2;
    DV3 V2 = b2ct2 * t2ct1cb1dt1;
    DV3 V3 = t2ct1 * b1ct1db2 - b1ct1ct2 * t1db2;
    DV3 V5 = t2cb1ct2 * t1db2 - t2ct1 * b2ct2db1;
    DV3 V6 = b2ct2 * t1ct2db1;

    tmp1 = mu4pinud * t2ct1db2;
    tmp2 = mu4pinud * b1ct1db2;
    V[0] = mu4pid * V1 - mu4pinud * V2 + tmp1 * b1ct1ct2 + tmp2 * t2ct1ct2;
    tmp1 = mu4pinu * t2db2;
    V[1] = tmp1 * b1ct1ct2 + mu4pi * V5 - mu4pinu * V6;
    tmp1 = mu4pinu * t1db2;
    tmp2 = mu4pinu * b1ct1db2;
    V[2] = mu4pi * V3 + tmp1 * b1ct1ct2 - tmp2 * t2ct1;
    tmp1 = mu4pinudCu * t2ct1cb1dt1 * t2ct1db2;
    V[3] = mu8piaSqd * V1 - mu4pinuaSqd * V2 - tmp1 * t2ct1ct2;
    tmp1 = mu4pinudSq * (t1ct2db1 * t2ct1db2 + t2ct1cb1dt1 * t2db2);
    V[4] = mu8piaSq * V5 - mu4pinuaSq * V6 - tmp1 * t2ct1ct2;
    tmp1 = mu4pinudSq * t2ct1cb1dt1 * t1db2;
    tmp2 = mu4pinudSq * t2ct1cb1dt1 * t2ct1db2;
    V[5] = mu8piaSq * V3 - tmp1 * t2ct1ct2 + tmp2 * t2ct1;
    tmp1 = mu4pinud * (t2ct1cb1dt1 * t2db2 + t1ct2db1 * t2ct1db2);
    tmp2 = mu4pinud * t1ct2db1 * t1db2;
    V[6] = tmp1 * t2ct1 - tmp2 * t2ct1ct2;
    tmp1 = mu4pinud * t1ct2db1 * t2db2;
    V[7] = -tmp1 * t2ct1ct2;
    tmp1 = mu4pinud * t2ct1cb1dt1 * t1db2;
    V[8] = tmp1 * t2ct1;
    DV3 tv = mu4pinu * t1ct2db1 * t2ct1;
    V[9] = tv * t2db2;
    V[10] = tv * t1db2;

    Fi[0] = x2 * integ[0] - integ[1];
    Fi[1] = x2 * integ[1] - integ[4];
    Fi[2] = x2 * integ[2] - integ[3];
    Fi[3] = x2 * integ[6] - integ[7];
    Fi[4] = x2 * integ[7] - integ[10];
    Fi[5] = x2 * integ[8] - integ[9];
    Fi[6] = x2 * integ[9] - integ[12];
    Fi[7] = x2 * integ[10] - integ[15];
    Fi[8] = x2 * integ[11] - integ[13];
    Fi[9] = x2 * integ[12] - integ[17];
    Fi[10] = x2 * integ[13] - integ[14];
    F3 = fsum11_df(V, Fi) * t2N;

    Fi[0] = integ[1] - x1 * integ[0];
    Fi[1] = integ[4] - x1 * integ[1];
    Fi[2] = integ[3] - x1 * integ[2];
    Fi[3] = integ[7] - x1 * integ[6];
    Fi[4] = integ[10] - x1 * integ[7];
    Fi[5] = integ[9] - x1 * integ[8];
    Fi[6] = integ[12] - x1 * integ[9];
    Fi[7] = integ[15] - x1 * integ[10];
    Fi[8] = integ[13] - x1 * integ[11];
    Fi[9] = integ[17] - x1 * integ[12];
    Fi[10] = integ[14] - x1 * integ[13];
    F4 = fsum11_df(V, Fi) * t2N;
  }
}

}  // namespace ddd

namespace ddd {

struct F3 {
  float x, y, z;
};
DF_HD F3 operator+(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
DF_HD F3 operator-(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
DF_HD F3 operator-(F3 a) { return {-a.x, -a.y, -a.z}; }
DF_HD F3 operator*(float s, F3 a) { return {s * a.x, s * a.y, s * a.z}; }
DF_HD F3 operator*(F3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
DF_HD float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
DF_HD F3 cross(F3 a, F3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
DF_HD F3 f3(DV3 v) { return {v.x.hi, v.y.hi, v.z.hi}; }

struct KConstsF {
  float mu4pi, mu4pinu, mu8piaSq, mu4pinuaSq;
};

// Mixed form of the general branch: the integration-domain geometry (c, d,
// x1..y2), the four corner antiderivatives and their first moments (Fint) in
// df64 — the cancellation-prone part, whose terms cancel by up to (R/L)^3 for
// a pair at distance R — and the V-vector assembly (products of unit vectors,
// Burgers vectors and powers of d, no cancellation of that order) in FP32.
// The 11-term node sums are taken in df64 from FP32 V and df64 Fint.
template <bool NEED12, bool NEED34, bool SUM32 = false>
DF_HD void assemble_mixed(const KConstsF& KF, const PairDF& g, F3 b1, F3 ft1, float t1N, F3 b2, F3 ft2, float t2N,
                          DV3& F1, DV3& F2, DV3& F3_, DV3& F4) {
  const df64 c = g.c, d = g.d, x1 = g.x1, x2 = g.x2, y1 = g.y1, y2 = g.y2;
  const df64* integ = g.integ;
  // FP32 geometry of the V vectors.
  const float mu4pi = KF.mu4pi, mu4pinu = KF.mu4pinu, mu8piaSq = KF.mu8piaSq, mu4pinuaSq = KF.mu4pinuaSq;
  const float cf = c.hi;
  const float dfl = d.hi;
  F3 t2ct1 = cross(ft2, ft1);
  F3 t1ct2 = -t2ct1;
  F3 b2ct2 = cross(b2, ft2);
  F3 b1ct1 = cross(b1, ft1);
  float t2db2 = dot(ft2, b2), t2db1 = dot(ft2, b1), t1db2 = dot(ft1, b2), t1db1 = dot(ft1, b1);
  float t2ct1db2 = dot(t2ct1, b2), t1ct2db1 = dot(t1ct2, b1), b1ct1db2 = dot(b1ct1, b2), b2ct2db1 = dot(b2ct2, b1);
  F3 t2ct1ct2 = ft1 - cf * ft2;
  F3 t1ct2ct1 = ft2 - cf * ft1;
  F3 t2cb1ct2 = b1 - t2db1 * ft2;
  F3 t1cb2ct1 = b2 - t1db2 * ft1;
  F3 b1ct1ct2 = t2db1 * ft1 - cf * b1;
  F3 b2ct2ct1 = t1db2 * ft2 - cf * b2;
  float t2ct1cb1dt1 = t2db1 - t1db1 * cf;
  float t1ct2cb2dt2 = t1db2 - t2db2 * cf;
  float t2ct1cb1db2 = t2db1 * t1db2 - t1db1 * t2db2;
  float mu4pid = mu4pi * dfl;
  float mu4pinud = mu4pinu * dfl;
  float mu4pinudSq = mu4pinud * dfl;
  float mu4pinudCu = mu4pinudSq * dfl;
  float mu4pinuaSqd = mu4pinuaSq * dfl;
  float mu8piaSqd = mu8piaSq * dfl;

  F3 V[11];
  float tmp1, tmp2;
  // First moments of both nodes of a segment in the lanes: A + Y b with A = +-a
  // and Y = (-y2, y1) or (x2, -x1), then the 11-term node sums.
  df2 Fi[11];
  auto node = [&](float tN, auto lane) {
    if (SUM32) {
      F3 s = {0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 11; ++k) {
        const df64 f = lane(Fi[k]);
        s = s + V[k] * (f.hi + f.lo);
      }
      return DV3{df(s.x * tN), df(s.y * tN), df(s.z * tN)};
    }
    DV3 s = {df(0.f), df(0.f), df(0.f)};
#pragma unroll
    for (int k = 0; k < 11; ++k) {
      const df64 f = lane(Fi[k]);
      s.x = s.x + f * V[k].x;
      s.y = s.y + f * V[k].y;
      s.z = s.z + f * V[k].z;
    }
    return DV3{s.x * tN, s.y * tN, s.z * tN};
  };
  auto first = [](df2 v) { return df2_x(v); };
  auto second = [](df2 v) { return df2_y(v); };
  if (NEED12) {
    tmp1 = t1db2 * t2db1 + t2ct1cb1db2;
    F3 V1 = tmp1 * t2ct1;
    F3 V2 = b1ct1 * t1ct2cb2dt2;
    F3 V3 = t1ct2 * b1ct1db2 - t1cb2ct1 * t2db1;
    F3 V4 = -b1ct1 * t2ct1db2;
    F3 V5 = b2ct2ct1 * t2db1 - t1ct2 * b2ct2db1;
    tmp1 = mu4pinud * t1ct2db1;
    tmp2 = mu4pinud * b2ct2db1;
    V[0] = mu4pid * V1 - mu4pinud * V2 + tmp1 * b2ct2ct1 + tmp2 * t1ct2ct1;
    tmp1 = mu4pinu * t2db1;
    tmp2 = mu4pinu * b2ct2db1;
    V[1] = mu4pi * V5 - tmp1 * b2ct2ct1 + tmp2 * t1ct2;
    tmp1 = mu4pinu * t1db1;
    V[2] = -tmp1 * b2ct2ct1 + mu4pi * V3 - mu4pinu * V4;
    tmp1 = mu4pinudCu * t1ct2cb2dt2 * t1ct2db1;
    V[3] = mu8piaSqd * V1 - mu4pinuaSqd * V2 - tmp1 * t1ct2ct1;
    tmp1 = mu4pinudSq * t1ct2cb2dt2 * t2db1;
    tmp2 = mu4pinudSq * t1ct2cb2dt2 * t1ct2db1;
    V[4] = mu8piaSq * V5 + tmp1 * t1ct2ct1 - tmp2 * t1ct2;
    tmp1 = mu4pinudSq * (t2ct1db2 * t1ct2db1 + t1ct2cb2dt2 * t1db1);
    V[5] = mu8piaSq * V3 - mu4pinuaSq * V4 + tmp1 * t1ct2ct1;
    tmp1 = mu4pinud * (t1ct2cb2dt2 * t1db1 + t2ct1db2 * t1ct2db1);
    tmp2 = mu4pinud * t2ct1db2 * t2db1;
    V[6] = tmp1 * t1ct2 - tmp2 * t1ct2ct1;
    tmp1 = mu4pinud * t1ct2cb2dt2 * t2db1;
    V[7] = tmp1 * t1ct2;
    tmp1 = mu4pinud * t2ct1db2 * t1db1;
    V[8] = -tmp1 * t1ct2ct1;
    F3 tv = mu4pinu * t2ct1db2 * t1ct2;
    V[9] = -tv * t2db1;
    V[10] = -tv * t1db1;

    const df2 Y = df2_make(-y2, y1);
    Fi[0] = df2_make(integ[2], -integ[2]) + Y * df2_dup(integ[0]);
    Fi[1] = df2_make(integ[3], -integ[3]) + Y * df2_dup(integ[1]);
    Fi[2] = df2_make(integ[5], -integ[5]) + Y * df2_dup(integ[2]);
    Fi[3] = df2_make(integ[8], -integ[8]) + Y * df2_dup(integ[6]);
    Fi[4] = df2_make(integ[9], -integ[9]) + Y * df2_dup(integ[7]);
    Fi[5] = df2_make(integ[11], -integ[11]) + Y * df2_dup(integ[8]);
    Fi[6] = df2_make(integ[13], -integ[13]) + Y * df2_dup(integ[9]);
    Fi[7] = df2_make(integ[12], -integ[12]) + Y * df2_dup(integ[10]);
    Fi[8] = df2_make(integ[16], -integ[16]) + Y * df2_dup(integ[11]);
    Fi[9] = df2_make(integ[14], -integ[14]) + Y * df2_dup(integ[12]);
    Fi[10] = df2_make(integ[18], -integ[18]) + Y * df2_dup(integ[13]);
    F1 = node(t1N, first);
    F2 = node(t1N, second);
  }
  if (NEED34) {
    tmp1 = t2db1 * t1db2 + t2ct1cb1db2;
    F3 V1 = tmp1 * t1ct2;
    F3 V2 = b2ct2 * t2ct1cb1dt1;
    F3 V3 = t2ct1 * b1ct1db2 - b1ct1ct2 * t1db2;
    F3 V5 = t2cb1ct2 * t1db2 - t2ct1 * b2ct2db1;
    F3 V6 = b2ct2 * t1ct2db1;
    tmp1 = mu4pinud * t2ct1db2;
    tmp2 = mu4pinud * b1ct1db2;
    V[0] = mu4pid * V1 - mu4pinud * V2 + tmp1 * b1ct1ct2 + tmp2 * t2ct1ct2;
    tmp1 = mu4pinu * t2db2;
    V[1] = tmp1 * b1ct1ct2 + mu4pi * V5 - mu4pinu * V6;
    tmp1 = mu4pinu * t1db2;
    tmp2 = mu4pinu * b1ct1db2;
    V[2] = mu4pi * V3 + tmp1 * b1ct1ct2 - tmp2 * t2ct1;
    tmp1 = mu4pinudCu * t2ct1cb1dt1 * t2ct1db2;
    V[3] = mu8piaSqd * V1 - mu4pinuaSqd * V2 - tmp1 * t2ct1ct2;
    tmp1 = mu4pinudSq * (t1ct2db1 * t2ct1db2 + t2ct1cb1dt1 * t2db2);
    V[4] = mu8piaSq * V5 - mu4pinuaSq * V6 - tmp1 * t2ct1ct2;
    tmp1 = mu4pinudSq * t2ct1cb1dt1 * t1db2;
    tmp2 = mu4pinudSq * t2ct1cb1dt1 * t2ct1db2;
    V[5] = mu8piaSq * V3 - tmp1 * t2ct1ct2 + tmp2 * t2ct1;
    tmp1 = mu4pinud * (t2ct1cb1dt1 * t2db2 + t1ct2db1 * t2ct1db2);
    tmp2 = mu4pinud * t1ct2db1 * t1db2;
    V[6] = tmp1 * t2ct1 - tmp2 * t2ct1ct2;
    tmp1 = mu4pinud * t1ct2db1 * t2db2;
    V[7] = -tmp1 * t2ct1ct2;
    tmp1 = mu4pinud * t2ct1cb1dt1 * t1db2;
    V[8] = tmp1 * t2ct1;
    F3 tv = mu4pinu * t1ct2db1 * t2ct1;
    V[9] = tv * t2db2;
    V[10] = tv * t1db2;

    const df2 Y = df2_make(x2, -x1);
    Fi[0] = df2_make(-integ[1], integ[1]) + Y * df2_dup(integ[0]);
    Fi[1] = df2_make(-integ[4], integ[4]) + Y * df2_dup(integ[1]);
    Fi[2] = df2_make(-integ[3], integ[3]) + Y * df2_dup(integ[2]);
    Fi[3] = df2_make(-integ[7], integ[7]) + Y * df2_dup(integ[6]);
    Fi[4] = df2_make(-integ[10], integ[10]) + Y * df2_dup(integ[7]);
    Fi[5] = df2_make(-integ[9], integ[9]) + Y * df2_dup(integ[8]);
    Fi[6] = df2_make(-integ[12], integ[12]) + Y * df2_dup(integ[9]);
    Fi[7] = df2_make(-integ[15], integ[15]) + Y * df2_dup(integ[10]);
    Fi[8] = df2_make(-integ[13], integ[13]) + Y * df2_dup(integ[11]);
    Fi[9] = df2_make(-integ[17], integ[17]) + Y * df2_dup(integ[12]);
    Fi[10] = df2_make(-integ[14], integ[14]) + Y * df2_dup(integ[13]);
    F3_ = node(t2N, first);
    F4 = node(t2N, second);
  }
}

// General branch of calcSegSegForce in df64 and in the mixed form.
template <bool NEED12, bool NEED34>
DF_HD void general_pair_df(const KConstsDF& K, DV3 b1, DV3 n11, DV3 n12, DV3 t1, df64 t1N, DV3 b2, DV3 n21, DV3 n22,
                           DV3 t2, df64 t2N, df64 c, DV3& F1, DV3& F2, DV3& F3, DV3& F4) {
  PairDF g;
  pair_integrals_df(K.aSq, t1, n11, n12, t2, n21, n22, c, g);
  assemble_df<NEED12, NEED34>(K, g, b1, t1, t1N, b2, t2, t2N, F1, F2, F3, F4);
}
template <bool NEED12, bool NEED34, bool SUM32 = false>
DF_HD void general_pair_mixed(const KConstsDF& K, const KConstsF& KF, F3 b1, DV3 n11, DV3 n12, DV3 t1, float t1N,
                              F3 b2, DV3 n21, DV3 n22, DV3 t2, float t2N, df64 c, DV3& F1, DV3& F2, DV3& F3_,
                              DV3& F4) {
  PairDF g;
  pair_integrals_df(K.aSq, t1, n11, n12, t2, n21, n22, c, g);
  assemble_mixed<NEED12, NEED34, SUM32>(KF, g, b1, f3(t1), t1N, b2, f3(t2), t2N, F1, F2, F3_, F4);
}

// Constants of the mixed σ̃ form.
struct KConstsSig {
  df64 aSq;
  float mu4pi, mu4pinu, nuMu4pinu, aSq32, aSqMu8pi;
};

// σ̃ contribution of one segment (n1, n2, unit direction t, Burgers vector b)
// at the point x, added into six df64 accumulators (xx, yy, zz, xy, xz, yz):
// the reference's formulas (DislocationFEM.jl:135-299, sigma_point in
// pair_f64.cuh), with the geometry (R, d, s1, s2), the endpoint terms and their
// differences s_03 ... s_25 in df64 — where the two endpoints cancel — and the
// coefficient assembly (t, d, t x b, d x b products) and the five-term sum in
// FP32.
DF_HD void sigma_point_mixed(const KConstsSig& K, F3 b, DV3 n1, DV3 n2, DV3 t, DV3 x, df64* sig) {
  const DV3 R = x - n1;
  const df64 Rdt = dot(R, t);
  const DV3 nd = R - Rdt * t;
  const df64 d2 = dot(nd, nd);
  const df64 s1 = -Rdt;
  const df64 s2 = -dot(x - n2, t);
  const df64 a2_d2 = K.aSq + d2;
  const df64 a2d2inv = df_recip(a2_d2);
  df64 S[5];
  {
    df64 Ra = df_sqrt(a2_d2 + s1 * s1);
    df64 Rainv = df_recip(Ra);
    df64 Ra3inv = Rainv * Rainv * Rainv;
    df64 sRa3inv = s1 * Ra3inv;
    const df64 s_03a = s1 * Rainv * a2d2inv;
    const df64 s_13a = -Rainv;
    const df64 s_05a = (df_scale(s_03a, 2.0f) + sRa3inv) * a2d2inv;
    const df64 s_15a = -Ra3inv;
    const df64 s_25a = s_03a - sRa3inv;
    Ra = df_sqrt(a2_d2 + s2 * s2);
    Rainv = df_recip(Ra);
    Ra3inv = Rainv * Rainv * Rainv;
    sRa3inv = s2 * Ra3inv;
    const df64 s_03b = s2 * Rainv * a2d2inv;
    const df64 s_13b = -Rainv;
    const df64 s_05b = (df_scale(s_03b, 2.0f) + sRa3inv) * a2d2inv;
    const df64 s_15b = -Ra3inv;
    const df64 s_25b = s_03b - sRa3inv;
    S[0] = s_03b - s_03a;
    S[1] = s_13b - s_13a;
    S[2] = s_05b - s_05a;
    S[3] = s_15b - s_15a;
    S[4] = s_25b - s_25a;
  }
  float Sf[5];
  for (int i = 0; i < 5; ++i) Sf[i] = S[i].hi + S[i].lo;
  const F3 tf = f3(t), dv = f3(nd);
  const F3 txb = cross(tf, b), dxb = cross(dv, b);
  const float common = K.mu4pinu * dot(dxb, tf);
  const float tt[3] = {tf.x, tf.y, tf.z}, dd[3] = {dv.x, dv.y, dv.z};
  const float tb_[3] = {txb.x, txb.y, txb.z}, db_[3] = {dxb.x, dxb.y, dxb.z};
  for (int c = 0; c < 6; ++c) {
    const int p = (c < 3) ? c : (c == 3 ? 0 : (c == 4 ? 0 : 1));
    const int q = (c < 3) ? c : (c == 3 ? 1 : 2);
    float dmd, tmt, tmd, tmtxb, dmtxb, tmdxb;
    if (c < 3) {
      dmd = dd[p] * dd[p];
      tmt = tt[p] * tt[p];
      tmd = 2.0f * tt[p] * dd[p];
      tmtxb = 2.0f * tt[p] * tb_[p];
      dmtxb = 2.0f * dd[p] * tb_[p];
      tmdxb = 2.0f * tt[p] * db_[p];
    } else {
      dmd = dd[p] * dd[q];
      tmt = tt[p] * tt[q];
      tmd = tt[p] * dd[q] + tt[q] * dd[p];
      tmtxb = tt[p] * tb_[q] + tt[q] * tb_[p];
      dmtxb = dd[p] * tb_[q] + dd[q] * tb_[p];
      tmdxb = tt[p] * db_[q] + tt[q] * db_[p];
    }
    const float I03 = (c < 3) ? (common + K.mu4pinu * dmtxb - K.mu4pi * tmdxb) : (K.mu4pinu * dmtxb - K.mu4pi * tmdxb);
    const float I13 = -K.nuMu4pinu * tmtxb;
    const float I05 = (c < 3) ? (common * (K.aSq32 + dmd) - K.aSqMu8pi * tmdxb) : (common * dmd - K.aSqMu8pi * tmdxb);
    const float I15 = K.aSqMu8pi * tmtxb - common * tmd;
    const float I25 = common * tmt;
    sig[c] = sig[c] + (I03 * Sf[0] + I13 * Sf[1] + I05 * Sf[2] + I15 * Sf[3] + I25 * Sf[4]);
  }
}

}  // namespace ddd
