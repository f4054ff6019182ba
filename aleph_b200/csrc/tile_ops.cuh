// tile_ops.cuh — gate ops on amplitudes held in registers: 2^R per thread, bit j
// of the register index is a qubit of the pass (kernels_tile.cu, kernels_wide.cu).
#pragma once

#include "common.cuh"

namespace ab {

template <int R>
__device__ __forceinline__ uint64_t roff(int r, const uint64_t (&hb)[5]) {
  uint64_t o = 0;
#pragma unroll
  for (int j = 0; j < R; ++j)
    if ((r >> j) & 1) o |= hb[j];
  return o;
}

#define AB_ON(r) (thr && (((r) & creg) == creg))

// ---- register-qubit ops -----------------------------------------------------
template <typename Real, int R, int J>
__device__ __forceinline__ void reg_1q(V2<Real> (&v)[1 << R], const V2<Real>* m, bool thr, uint32_t creg) {
  const V2<Real> m0 = ld_coef<Real>(m), m1 = ld_coef<Real>(m + 1), m2 = ld_coef<Real>(m + 2),
                 m3 = ld_coef<Real>(m + 3);
  if (thr && creg == 0) {  // no register-part controls: every pair, no per-pair predicate
#pragma unroll
    for (int r = 0; r < (1 << R); ++r) {
      if (r & (1 << J)) continue;
      const int r1 = r | (1 << J);
      const V2<Real> a = v[r], b = v[r1];
      v[r] = cmul2<Real>(m0, a, m1, b);
      v[r1] = cmul2<Real>(m2, a, m3, b);
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & (1 << J)) continue;
    const int r1 = r | (1 << J);
    if (!AB_ON(r)) continue;
    const V2<Real> a = v[r], b = v[r1];
    v[r] = cmul2<Real>(m0, a, m1, b);
    v[r1] = cmul2<Real>(m2, a, m3, b);
  }
}

// Two one-qubit gates in a row, U1 on register bit J1 then U2 on register bit
// J2 != J1, neither controlled: one sweep over quartets. U1 writes four
// temporaries and U2 writes straight back into the loop-carried registers,
// so no amplitude moves between the two gates (a lone gate must park three
// of every four results while its inputs are still live).
template <typename Real, int R, int J1, int J2>
__device__ __forceinline__ void reg_1q_pair(V2<Real> (&v)[1 << R], const V2<Real>* m, const V2<Real>* u) {
  const V2<Real> m0 = ld_coef<Real>(m), m1 = ld_coef<Real>(m + 1), m2 = ld_coef<Real>(m + 2),
                 m3 = ld_coef<Real>(m + 3);
  const V2<Real> u0 = ld_coef<Real>(u), u1 = ld_coef<Real>(u + 1), u2 = ld_coef<Real>(u + 2),
                 u3 = ld_coef<Real>(u + 3);
  constexpr int B1 = 1 << J1, B2 = 1 << J2;
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & (B1 | B2)) continue;
    const V2<Real> x00 = v[r], x01 = v[r | B1], x10 = v[r | B2], x11 = v[r | B1 | B2];
    const V2<Real> t00 = cmul2<Real>(m0, x00, m1, x01), t01 = cmul2<Real>(m2, x00, m3, x01);
    const V2<Real> t10 = cmul2<Real>(m0, x10, m1, x11), t11 = cmul2<Real>(m2, x10, m3, x11);
    v[r] = cmul2<Real>(u0, t00, u1, t10);
    v[r | B2] = cmul2<Real>(u2, t00, u3, t10);
    v[r | B1] = cmul2<Real>(u0, t01, u1, t11);
    v[r | B1 | B2] = cmul2<Real>(u2, t01, u3, t11);
  }
}

// Sign flip of the registers r with (r & K) == K: a CZ-like op whose
// register part K is known at compile time runs without per-amplitude tests.
template <typename Real, int R, uint32_t K>
__device__ __forceinline__ void reg_neg(V2<Real> (&v)[1 << R]) {
#pragma unroll
  for (int r = 0; r < (1 << R); ++r)
    if (((uint32_t)r & K) == K) v[r] = cneg<Real>(v[r]);
}

template <typename Real, int R>
__device__ __forceinline__ void dispatch_neg(V2<Real> (&v)[1 << R], uint32_t creg) {
#define AB_NEG(k) \
  case k:         \
    if constexpr ((k) < (1u << R)) reg_neg<Real, R, k>(v); \
    break;
  switch (creg) {
    AB_NEG(0) AB_NEG(1) AB_NEG(2) AB_NEG(3) AB_NEG(4) AB_NEG(5) AB_NEG(6) AB_NEG(7)
    AB_NEG(8) AB_NEG(9) AB_NEG(10) AB_NEG(11) AB_NEG(12) AB_NEG(13) AB_NEG(14) AB_NEG(15)
    AB_NEG(16) AB_NEG(17) AB_NEG(18) AB_NEG(19) AB_NEG(20) AB_NEG(21) AB_NEG(22) AB_NEG(23)
    AB_NEG(24) AB_NEG(25) AB_NEG(26) AB_NEG(27) AB_NEG(28) AB_NEG(29) AB_NEG(30) AB_NEG(31)
  }
#undef AB_NEG
}

template <typename Real, int R, int J>
__device__ __forceinline__ void reg_x(V2<Real> (&v)[1 << R], bool thr, uint32_t creg) {
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & (1 << J)) continue;
    const int r1 = r | (1 << J);
    if (!AB_ON(r)) continue;
    const V2<Real> t = v[r];
    v[r] = v[r1];
    v[r1] = t;
  }
}

// 4x4 on register bits JA (matrix MSB) > JB (matrix LSB).
template <typename Real, int R, int JA, int JB>
__device__ __forceinline__ void reg_2q(V2<Real> (&v)[1 << R], const V2<Real>* m, bool thr, uint32_t creg) {
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & ((1 << JA) | (1 << JB))) continue;
    if (!AB_ON(r)) continue;
    const int i0 = r, i1 = r | (1 << JB), i2 = r | (1 << JA), i3 = r | (1 << JA) | (1 << JB);
    const V2<Real> x0 = v[i0], x1 = v[i1], x2 = v[i2], x3 = v[i3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const V2<Real> acc = cadd<Real>(cmul2<Real>(ld_coef<Real>(m + 4 * k), x0, ld_coef<Real>(m + 4 * k + 1), x1),
                                      cmul2<Real>(ld_coef<Real>(m + 4 * k + 2), x2, ld_coef<Real>(m + 4 * k + 3), x3));
      const int dst = k == 0 ? i0 : k == 1 ? i1 : k == 2 ? i2 : i3;
      v[dst] = acc;
    }
  }
}

// The q-th register index with bits JA and JB clear (q's bits deposited in order).
template <int R, int JA, int JB>
__device__ constexpr int quartet_base(int q) {
  int r = 0, bit = 0;
  for (int j = 0; j < R; ++j) {
    if (j == JA || j == JB) continue;
    if ((q >> bit) & 1) r |= 1 << j;
    ++bit;
  }
  return r;
}

// One row of a 4x4: c0 x0 + c1 x1 + c2 x2 + c3 x3 as one multiply-add chain
// per component (1 multiply + 7 fused multiply-adds).
template <typename Real>
__device__ __forceinline__ V2<Real> mac4(V2<Real> c0, V2<Real> x0, V2<Real> c1, V2<Real> x1, V2<Real> c2, V2<Real> x2,
                                         V2<Real> c3, V2<Real> x3) {
  Real re = c0.x * x0.x, im = c0.x * x0.y;
  re = fma(-c0.y, x0.y, re);
  im = fma(c0.y, x0.x, im);
  re = fma(c1.x, x1.x, re);
  im = fma(c1.x, x1.y, im);
  re = fma(-c1.y, x1.y, re);
  im = fma(c1.y, x1.x, im);
  re = fma(c2.x, x2.x, re);
  im = fma(c2.x, x2.y, im);
  re = fma(-c2.y, x2.y, re);
  im = fma(c2.y, x2.x, im);
  re = fma(c3.x, x3.x, re);
  im = fma(c3.x, x3.y, im);
  re = fma(-c3.y, x3.y, re);
  im = fma(c3.y, x3.x, im);
  return mk<Real>(re, im);
}

// Uncontrolled 4x4 on register bits JA (matrix MSB) > JB, QB quartets at a
// time: each row of coefficients is loaded once per QB quartets and the
// block's outputs wait in registers until its inputs are spent. The
// coefficients are uniform across the warp, and with the tile in registers
// they cannot all stay live; loaded per quartet, they were most of the pass's
// L1 traffic.
template <typename Real, int R, int JA, int JB, int QB>
__device__ __forceinline__ void reg_2q_blocked(V2<Real> (&v)[1 << R], const V2<Real>* m) {
  constexpr int NQ = 1 << (R - 2);
  constexpr int A = 1 << JA, B = 1 << JB;
#pragma unroll
  for (int q0 = 0; q0 < NQ; q0 += QB) {
    V2<Real> o[QB][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const V2<Real> c0 = ld_coef<Real>(m + 4 * k), c1 = ld_coef<Real>(m + 4 * k + 1),
                     c2 = ld_coef<Real>(m + 4 * k + 2), c3 = ld_coef<Real>(m + 4 * k + 3);
#pragma unroll
      for (int j = 0; j < QB; ++j) {
        const int r = quartet_base<R, JA, JB>(q0 + j);
        o[j][k] = mac4<Real>(c0, v[r], c1, v[r | B], c2, v[r | A], c3, v[r | A | B]);
      }
    }
#pragma unroll
    for (int j = 0; j < QB; ++j) {
      const int r = quartet_base<R, JA, JB>(q0 + j);
      v[r] = o[j][0];
      v[r | B] = o[j][1];
      v[r | A] = o[j][2];
      v[r | A | B] = o[j][3];
    }
  }
}

// ---- real matrices (Ry, H, and the 4x4s they fuse to with CNOTs and CZs) -----
// Half the multiply-adds of the complex forms: both components of an amplitude
// see the same real matrix. Uncontrolled, coefficients as complex numbers with
// zero imaginary parts.
template <typename Real, int R, int J>
__device__ __forceinline__ void reg_1q_real(V2<Real> (&v)[1 << R], const V2<Real>* m) {
  const Real m0 = ld_coef<Real>(m).x, m1 = ld_coef<Real>(m + 1).x, m2 = ld_coef<Real>(m + 2).x,
             m3 = ld_coef<Real>(m + 3).x;
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & (1 << J)) continue;
    const int r1 = r | (1 << J);
    const V2<Real> a = v[r], b = v[r1];
    v[r] = mk<Real>(fma(m1, b.x, m0 * a.x), fma(m1, b.y, m0 * a.y));
    v[r1] = mk<Real>(fma(m3, b.x, m2 * a.x), fma(m3, b.y, m2 * a.y));
  }
}

template <typename Real, int R>
__device__ __forceinline__ void dispatch_reg_real(int j, V2<Real> (&v)[1 << R], const V2<Real>* m) {
  switch (j) {
    case 0: if constexpr (R > 0) reg_1q_real<Real, R, 0>(v, m); break;
    case 1: if constexpr (R > 1) reg_1q_real<Real, R, 1>(v, m); break;
    case 2: if constexpr (R > 2) reg_1q_real<Real, R, 2>(v, m); break;
    case 3: if constexpr (R > 3) reg_1q_real<Real, R, 3>(v, m); break;
    case 4: if constexpr (R > 4) reg_1q_real<Real, R, 4>(v, m); break;
  }
}

// A real 4x4 on register bits JA > JB, QB quartets per coefficient row (see reg_2q_blocked).
template <typename Real, int R, int JA, int JB, int QB>
__device__ __forceinline__ void reg_2q_real(V2<Real> (&v)[1 << R], const V2<Real>* m) {
  constexpr int NQ = 1 << (R - 2);
  constexpr int A = 1 << JA, B = 1 << JB;
#pragma unroll
  for (int q0 = 0; q0 < NQ; q0 += QB) {
    V2<Real> o[QB][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const Real c0 = ld_coef<Real>(m + 4 * k).x, c1 = ld_coef<Real>(m + 4 * k + 1).x,
                 c2 = ld_coef<Real>(m + 4 * k + 2).x, c3 = ld_coef<Real>(m + 4 * k + 3).x;
#pragma unroll
      for (int j = 0; j < QB; ++j) {
        const int r = quartet_base<R, JA, JB>(q0 + j);
        o[j][k].x = fma(c3, v[r | A | B].x, fma(c2, v[r | A].x, fma(c1, v[r | B].x, c0 * v[r].x)));
        o[j][k].y = fma(c3, v[r | A | B].y, fma(c2, v[r | A].y, fma(c1, v[r | B].y, c0 * v[r].y)));
      }
    }
#pragma unroll
    for (int j = 0; j < QB; ++j) {
      const int r = quartet_base<R, JA, JB>(q0 + j);
      v[r] = o[j][0];
      v[r | B] = o[j][1];
      v[r | A] = o[j][2];
      v[r | A | B] = o[j][3];
    }
  }
}

template <typename Real, int R, int QB>
__device__ __forceinline__ void dispatch_reg_2q_real(int ja, int jb, V2<Real> (&v)[1 << R], const V2<Real>* m) {
#define AB_RR(a, b)                                                    \
  case (a)*8 + (b):                                                    \
    if constexpr (R > (a)) reg_2q_real<Real, R, (a), (b), QB>(v, m);   \
    break;
  switch (ja * 8 + jb) {
    AB_RR(1, 0) AB_RR(2, 0) AB_RR(2, 1) AB_RR(3, 0) AB_RR(3, 1)
    AB_RR(3, 2) AB_RR(4, 0) AB_RR(4, 1) AB_RR(4, 2) AB_RR(4, 3)
  }
#undef AB_RR
}

// ---- paired FP32 arithmetic ----------------------------------------------------
// An FP32 amplitude is one register pair, and a matrix entry c acts on it as
// (cx, cx) * (re, im) + (cy, cy) * (-im, re): two paired multiply-adds for both
// components, half the instructions of the scalar form. The coefficients come
// duplicated, (cx, cx) then (cy, cy) per entry; a real matrix has (cx, cx) only.
__device__ __forceinline__ float2 times_i(float2 x) { return make_float2(-x.y, x.x); }

template <int R, int J, bool REAL>
__device__ __forceinline__ void reg_1q_f32x2(float2 (&v)[1 << R], const float2* m) {
  constexpr int S = REAL ? 1 : 2;
  float2 c[4 * S];
#pragma unroll
  for (int k = 0; k < 4 * S; ++k) c[k] = ld_coef<float>(m + k);
#pragma unroll
  for (int r = 0; r < (1 << R); ++r) {
    if (r & (1 << J)) continue;
    const int r1 = r | (1 << J);
    const float2 a = v[r], b = v[r1];
    float2 o0 = __fmul2_rn(c[0], a), o1 = __fmul2_rn(c[2 * S], a);
    if constexpr (!REAL) {
      const float2 ia = times_i(a), ib = times_i(b);
      o0 = __ffma2_rn(c[1], ia, o0);
      o1 = __ffma2_rn(c[2 * S + 1], ia, o1);
      o0 = __ffma2_rn(c[S + 1], ib, o0);
      o1 = __ffma2_rn(c[3 * S + 1], ib, o1);
    }
    v[r] = __ffma2_rn(c[S], b, o0);
    v[r1] = __ffma2_rn(c[3 * S], b, o1);
  }
}

template <int R, bool REAL>
__device__ __forceinline__ void dispatch_1q_f32x2(int j, float2 (&v)[1 << R], const float2* m) {
  switch (j) {
    case 0: if constexpr (R > 0) reg_1q_f32x2<R, 0, REAL>(v, m); break;
    case 1: if constexpr (R > 1) reg_1q_f32x2<R, 1, REAL>(v, m); break;
    case 2: if constexpr (R > 2) reg_1q_f32x2<R, 2, REAL>(v, m); break;
    case 3: if constexpr (R > 3) reg_1q_f32x2<R, 3, REAL>(v, m); break;
    case 4: if constexpr (R > 4) reg_1q_f32x2<R, 4, REAL>(v, m); break;
  }
}

// A 4x4 on register bits JA > JB, QB quartets per coefficient row (see reg_2q_blocked).
template <int R, int JA, int JB, int QB, bool REAL>
__device__ __forceinline__ void reg_2q_f32x2(float2 (&v)[1 << R], const float2* m) {
  constexpr int NQ = 1 << (R - 2), S = REAL ? 1 : 2;
  constexpr int A = 1 << JA, B = 1 << JB;
#pragma unroll
  for (int q0 = 0; q0 < NQ; q0 += QB) {
    float2 o[QB][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 c[4 * S];
#pragma unroll
      for (int e = 0; e < 4 * S; ++e) c[e] = ld_coef<float>(m + 4 * S * k + e);
#pragma unroll
      for (int j = 0; j < QB; ++j) {
        const int r = quartet_base<R, JA, JB>(q0 + j);
        const float2 x[4] = {v[r], v[r | B], v[r | A], v[r | A | B]};
        float2 t = __fmul2_rn(c[0], x[0]);
#pragma unroll
        for (int e = 1; e < 4; ++e) t = __ffma2_rn(c[S * e], x[e], t);
        if constexpr (!REAL)
#pragma unroll
          for (int e = 0; e < 4; ++e) t = __ffma2_rn(c[S * e + 1], times_i(x[e]), t);
        o[j][k] = t;
      }
    }
#pragma unroll
    for (int j = 0; j < QB; ++j) {
      const int r = quartet_base<R, JA, JB>(q0 + j);
      v[r] = o[j][0];
      v[r | B] = o[j][1];
      v[r | A] = o[j][2];
      v[r | A | B] = o[j][3];
    }
  }
}

template <int R, int QB, bool REAL>
__device__ __forceinline__ void dispatch_2q_f32x2(int ja, int jb, float2 (&v)[1 << R], const float2* m) {
#define AB_RR(a, b)                                                       \
  case (a)*8 + (b):                                                       \
    if constexpr (R > (a)) reg_2q_f32x2<R, (a), (b), QB, REAL>(v, m);     \
    break;
  switch (ja * 8 + jb) {
    AB_RR(1, 0) AB_RR(2, 0) AB_RR(2, 1) AB_RR(3, 0) AB_RR(3, 1)
    AB_RR(3, 2) AB_RR(4, 0) AB_RR(4, 1) AB_RR(4, 2) AB_RR(4, 3)
  }
#undef AB_RR
}

// ---- diagonal ops -------------------------------------------------------------
template <typename Real, int R>
__device__ __forceinline__ void diag_ops(const Op& op, V2<Real> (&v)[1 << R], uint64_t gl, const uint64_t (&hb)[5],
                                         const V2<Real>* coef, const PolyTables& poly) {
  const uint32_t creg = op.creg;
  switch (op.type) {
    case OP_NEG:
      if ((gl & op.mask) == op.mask) dispatch_neg<Real, R>(v, creg);
      break;
    case OP_CPHASE: {
      const bool thr = (gl & op.mask) == op.mask;
      const V2<Real> c = ld_coef<Real>(coef + op.coef);
#pragma unroll
      for (int r = 0; r < (1 << R); ++r)
        if (AB_ON(r)) v[r] = cmul<Real>(c, v[r]);
      break;
    }
    case OP_DIAG: {
      const bool thr = (gl & op.ctrl) == op.ctrl;
      const int nq = op.nq;
      uint32_t tidx = 0;  // table-index bits taken from thread-constant qubits
#pragma unroll
      for (int i = 0; i < 3; ++i)
        if (i < nq && !((op.dsrc >> i) & 1)) tidx |= (uint32_t)((gl >> op.q[i]) & 1) << (nq - 1 - i);
      const uint32_t s0 = op.q[3], s1 = op.q[4], s2 = op.q[5];
      const uint32_t d0 = (op.dsrc >> 0) & 1, d1 = (op.dsrc >> 1) & 1, d2 = (op.dsrc >> 2) & 1;
      const V2<Real>* tab = coef + op.coef;
#pragma unroll
      for (int r = 0; r < (1 << R); ++r) {
        if (!AB_ON(r)) continue;
        uint32_t idx = tidx;
        if (d0) idx |= ((r >> s0) & 1) << (nq - 1);
        if (d1) idx |= ((r >> s1) & 1) << (nq - 2);
        if (d2) idx |= ((r >> s2) & 1) << (nq - 3);
        v[r] = cmul<Real>(ld_coef<Real>(tab + idx), v[r]);
      }
      break;
    }
    case OP_POLY: {
#pragma unroll
      for (int r = 0; r < (1 << R); ++r) v[r] = apply_diag_op<Real>(op, v[r], gl | roff<R>(r, hb), coef, poly);
      break;
    }
  }
}

template <typename Real, int R>
__device__ __forceinline__ void dispatch_reg(const Op& op, V2<Real> (&v)[1 << R], const V2<Real>* m, bool thr) {
  const uint32_t creg = op.creg;
  const int J = op.a - 5;
  if (op.type == OP_X) {
    switch (J) {
      case 0: if constexpr (R > 0) reg_x<Real, R, 0>(v, thr, creg); break;
      case 1: if constexpr (R > 1) reg_x<Real, R, 1>(v, thr, creg); break;
      case 2: if constexpr (R > 2) reg_x<Real, R, 2>(v, thr, creg); break;
      case 3: if constexpr (R > 3) reg_x<Real, R, 3>(v, thr, creg); break;
      case 4: if constexpr (R > 4) reg_x<Real, R, 4>(v, thr, creg); break;
    }
    return;
  }
  switch (J) {
    case 0: if constexpr (R > 0) reg_1q<Real, R, 0>(v, m, thr, creg); break;
    case 1: if constexpr (R > 1) reg_1q<Real, R, 1>(v, m, thr, creg); break;
    case 2: if constexpr (R > 2) reg_1q<Real, R, 2>(v, m, thr, creg); break;
    case 3: if constexpr (R > 3) reg_1q<Real, R, 3>(v, m, thr, creg); break;
    case 4: if constexpr (R > 4) reg_1q<Real, R, 4>(v, m, thr, creg); break;
  }
}

// Two uncontrolled one-qubit gates on register bits j1 != j2 (in that order).
template <typename Real, int R>
__device__ __forceinline__ void dispatch_pair(int j1, int j2, V2<Real> (&v)[1 << R], const V2<Real>* m,
                                              const V2<Real>* u) {
#define AB_PR(a, b)                                                      \
  case (a)*8 + (b):                                                      \
    if constexpr (R > (a) && R > (b)) reg_1q_pair<Real, R, (a), (b)>(v, m, u); \
    break;
  switch (j1 * 8 + j2) {
    AB_PR(0, 1) AB_PR(0, 2) AB_PR(0, 3) AB_PR(0, 4) AB_PR(1, 0) AB_PR(1, 2) AB_PR(1, 3) AB_PR(1, 4)
    AB_PR(2, 0) AB_PR(2, 1) AB_PR(2, 3) AB_PR(2, 4) AB_PR(3, 0) AB_PR(3, 1) AB_PR(3, 2) AB_PR(3, 4)
    AB_PR(4, 0) AB_PR(4, 1) AB_PR(4, 2) AB_PR(4, 3)
  }
#undef AB_PR
}

// Uncontrolled or controlled 4x4 on register bits ja (matrix MSB) > jb, QB quartets per coefficient load.
template <typename Real, int R, int QB>
__device__ __forceinline__ void dispatch_reg_2q(int ja, int jb, V2<Real> (&v)[1 << R], const V2<Real>* m, bool thr,
                                                uint32_t creg) {
  constexpr int kQB = QB > (1 << (R >= 2 ? R - 2 : 0)) ? (1 << (R >= 2 ? R - 2 : 0)) : QB;
#define AB_RR(a, b)                                                           \
  case (a)*8 + (b):                                                           \
    if constexpr (R > (a)) {                                                  \
      if (kQB > 1 && thr && creg == 0) reg_2q_blocked<Real, R, (a), (b), kQB>(v, m); \
      else reg_2q<Real, R, (a), (b)>(v, m, thr, creg);                        \
    }                                                                         \
    break;
  switch (ja * 8 + jb) {
    AB_RR(1, 0) AB_RR(2, 0) AB_RR(2, 1) AB_RR(3, 0) AB_RR(3, 1)
    AB_RR(3, 2) AB_RR(4, 0) AB_RR(4, 1) AB_RR(4, 2) AB_RR(4, 3)
  }
#undef AB_RR
}

}  // namespace ab
