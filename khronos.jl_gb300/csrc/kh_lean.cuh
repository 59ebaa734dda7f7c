// Per-cell arithmetic of the reduced-state CPML update (kh_lean.cu).
//
// The CUDA-path CPML stages of component c (n = next axis, p = previous axis)
//   u' = ((1-σn)·u + K)/(1+σn),  t' = ((1-σp)·t + (u'-u))/(1+σp),
//   O' = O + (1+σc)·m·t' - (1-σc)·m·t
// keep three auxiliaries (T = B|D, U, W = m·T).  m is constant in time and
// everything starts from zero, so most of them follow from the others:
//  * W = m·T always;
//  * outside the own-axis CPML O = m·T, so T follows from O: the t stage runs
//    on O itself;
//  * with σp = 0, T = U: one of them is enough; with σn = 0 U is not used.
// What is left is T where the cell lies in the CPML of its own axis and U where
// it lies in those of both other axes: one auxiliary in a face slab instead of
// five, three instead of seven along an edge, six instead of nine in a corner.
//
// The operations are written with explicit roundings (no contraction left to
// the compiler).  A damped O is fma(A, O, m·(B·d)): one rounding at the size of O a
// step (fma(m, B·d, A·O) has two; FP32 fluxes of 64³ runs of 173 steps were then up to
// 1.3e-6 off instead of 4.7e-7).  A plain O is fma(m, d, O) in every kernel and every
// form of a row, so they give the same bits, but for one: FP64 rows beside the x-CPML
// (row_o).
#pragma once

#include "kh_cell.cuh"

namespace kh {

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// One component of the scaled curl: ca·(a1 - a0) - cb·(b1 - b0).
template <typename T>
__device__ __forceinline__ T curl_rn(T ca, T a1, T a0, T cb, T b1, T b0) {
  return fma_rn(ca, sub_rn(a1, a0), -mul_rn(cb, sub_rn(b1, b0)));
}

// T as it follows from O outside the own-axis CPML, and how far O may be from m·T (o)
// by the rounding of both.
template <typename T>
__device__ __forceinline__ T derived_t(T O, T m) {
  return m != T(0) ? O / m : T(0);
}
template <typename T>
__device__ __forceinline__ T derived_tol(T o) {
  constexpr T eps = sizeof(T) == 4 ? T(1.1920929e-7) : T(2.220446049250313e-16);
  constexpr T tiny = sizeof(T) == 4 ? T(1.17549435e-38) : T(2.2250738585072014e-308);
  return T(8) * (eps * fabs(o) + tiny);
}

// CPML factors of a cell along one axis; f false: outside that axis's CPML.
template <typename T>
struct RedAxis {
  bool f;
  T a;   // (1-σ)/(1+σ)
  T b;   // 1/(1+σ)
  T om;  // 1-σ
  T op;  // 1+σ
};

template <typename T>
__device__ __forceinline__ RedAxis<T> red_axis(const AxisCoef<T>& x, bool f) {
  return f ? RedAxis<T>{true, mul_rn(x.om, x.ir), x.ir, x.om, x.op} : RedAxis<T>{false, T(1), T(1), T(1), T(1)};
}

// Component with own axis o, next axis n, previous axis p.  t is used iff o.f,
// u iff n.f and p.f.
template <typename T>
__device__ __forceinline__ void red_component(const RedAxis<T>& o, const RedAxis<T>& n, const RedAxis<T>& p, T K, T m,
                                              T& O, T& t, T& u) {
  T d = K;
  if (n.f && p.f) {
    const T un = fma_rn(n.a, u, mul_rn(n.b, K));
    d = sub_rn(un, u);
    u = un;
  }
  if (n.f || p.f) {
    const T A = p.f ? p.a : n.a, B = p.f ? p.b : n.b;
    const T x = mul_rn(B, d);
    if (o.f) {
      const T tn = fma_rn(A, t, x);
      O = fma_rn(m, fma_rn(o.op, tn, -mul_rn(o.om, t)), O);
      t = tn;
    } else {
      O = fma_rn(A, O, mul_rn(m, x));
    }
  } else if (o.f) {
    const T tn = add_rn(t, d);
    O = fma_rn(m, fma_rn(o.op, tn, -mul_rn(o.om, t)), O);
    t = tn;
  } else {
    O = fma_rn(m, d, O);
  }
}

// The cells of one thread: VN consecutive cells of a row.
template <typename T, int VN>
struct alignas(sizeof(T) * VN) Pack {
  T v[VN];
};
template <typename T, int VN>
struct Cells {
  Pack<T, VN> c[3];
};

// Update of VN cells without special ones.  Straight-line code for the three
// common kinds of row (plain; x-CPML alone; y and/or z), the per-cell form
// where the x-CPML meets another.  All give red_component's bits.
template <typename T, int VN>
__device__ __forceinline__ void update_cells(const bool (&fx)[VN], bool anyfx, const AxisCoef<T>* xt,
                                             const RedAxis<T>& ry, const RedAxis<T>& rz, const Cells<T, VN>& K,
                                             const Cells<T, VN>& m, Cells<T, VN>& O, Cells<T, VN>& t,
                                             Cells<T, VN>& u) {
  if (!(anyfx || ry.f || rz.f)) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int v = 0; v < VN; ++v) O.c[c].v[v] = fma_rn(m.c[c].v[v], K.c[c].v[v], O.c[c].v[v]);
  } else if (!anyfx) {
    if (ry.f && rz.f) {
#pragma unroll
      for (int v = 0; v < VN; ++v) {
        const T un = fma_rn(ry.a, u.c[0].v[v], mul_rn(ry.b, K.c[0].v[v]));
        const T d = sub_rn(un, u.c[0].v[v]);
        u.c[0].v[v] = un;
        O.c[0].v[v] = fma_rn(rz.a, O.c[0].v[v], mul_rn(m.c[0].v[v], mul_rn(rz.b, d)));
      }
    } else {
      const T A = ry.f ? ry.a : rz.a, B = ry.f ? ry.b : rz.b;
#pragma unroll
      for (int v = 0; v < VN; ++v)
        O.c[0].v[v] = fma_rn(A, O.c[0].v[v], mul_rn(m.c[0].v[v], mul_rn(B, K.c[0].v[v])));
    }
    // component y: own axis y, damped along z; component z the other way
#pragma unroll
    for (int c = 1; c < 3; ++c) {
      const RedAxis<T>& o = c == 1 ? ry : rz;
      const RedAxis<T>& d = c == 1 ? rz : ry;  // factors 1 outside its CPML
      if (o.f) {
#pragma unroll
        for (int v = 0; v < VN; ++v) {
          const T tn = fma_rn(d.a, t.c[c].v[v], mul_rn(d.b, K.c[c].v[v]));
          O.c[c].v[v] = fma_rn(m.c[c].v[v], fma_rn(o.op, tn, -mul_rn(o.om, t.c[c].v[v])), O.c[c].v[v]);
          t.c[c].v[v] = tn;
        }
      } else {
#pragma unroll
        for (int v = 0; v < VN; ++v)
          O.c[c].v[v] = fma_rn(d.a, O.c[c].v[v], mul_rn(m.c[c].v[v], mul_rn(d.b, K.c[c].v[v])));
      }
    }
  } else if (!(ry.f || rz.f)) {
#pragma unroll
    for (int v = 0; v < VN; ++v) {
      const AxisCoef<T> x = xt[v];  // a, b, 1-σ, 1+σ
      const T tn = add_rn(t.c[0].v[v], K.c[0].v[v]);
      const T o0 = fma_rn(m.c[0].v[v], fma_rn(x.op, tn, -mul_rn(x.ir, t.c[0].v[v])), O.c[0].v[v]);
      const T o1 = fma_rn(x.s, O.c[1].v[v], mul_rn(m.c[1].v[v], mul_rn(x.om, K.c[1].v[v])));
      const T o2 = fma_rn(x.s, O.c[2].v[v], mul_rn(m.c[2].v[v], mul_rn(x.om, K.c[2].v[v])));
      O.c[0].v[v] = fx[v] ? o0 : fma_rn(m.c[0].v[v], K.c[0].v[v], O.c[0].v[v]);
      O.c[1].v[v] = fx[v] ? o1 : fma_rn(m.c[1].v[v], K.c[1].v[v], O.c[1].v[v]);
      O.c[2].v[v] = fx[v] ? o2 : fma_rn(m.c[2].v[v], K.c[2].v[v], O.c[2].v[v]);
      t.c[0].v[v] = fx[v] ? tn : t.c[0].v[v];
    }
  } else {
#pragma unroll
    for (int v = 0; v < VN; ++v) {
      RedAxis<T> rx{false, T(1), T(1), T(1), T(1)};
      if (fx[v]) rx = {true, xt[v].s, xt[v].om, xt[v].ir, xt[v].op};
      red_component(rx, ry, rz, K.c[0].v[v], m.c[0].v[v], O.c[0].v[v], t.c[0].v[v], u.c[0].v[v]);
      red_component(ry, rz, rx, K.c[1].v[v], m.c[1].v[v], O.c[1].v[v], t.c[1].v[v], u.c[1].v[v]);
      red_component(rz, rx, ry, K.c[2].v[v], m.c[2].v[v], O.c[2].v[v], t.c[2].v[v], u.c[2].v[v]);
    }
  }
}

// O of a cell that only the x-CPML may damp (f; w = B·d, and A = 1, w = d outside it).
// FP32 selects the operands of one multiply-add (160×160×96 with uniform materials 64.2 to
// 64.5 µs a step; selecting the result 64.8).  FP64, bound by arithmetic, leaves plain cells
// fma(1, O, m·d), one rounding more at 2⁻⁵³ (with selects 128×96×96 145.8 to 150.5 µs).
template <bool WX, typename T>
__device__ __forceinline__ T row_o(bool f, T A, T O, T m, T w) {
  if constexpr (!WX) return fma_rn(m, w, O);
  else if constexpr (sizeof(T) == 8) return fma_rn(A, O, mul_rn(m, w));
  else return fma_rn(f ? A : m, f ? O : w, f ? mul_rn(m, w) : O);
}

// Update of VN cells of a row without special cells, compiled for the CPMLs the
// row can meet: WX its tile touches the x-CPML (fx[v]: cell v is in it, xt its
// factors a, b, 1-σ, 1+σ, all 1 outside), FY and FZ the row or plane is in the y- or
// z-CPML.  Straight-line: the cells of a row that differ only in fx[v] take both
// forms and select, which costs a few operations; branching on fx cost both sides'
// instructions and their registers.  t and u of cells that have none are read as
// finite values and come back unchanged.
template <bool WX, bool FY, bool FZ, typename T, int VN>
__device__ __forceinline__ void update_row(const bool (&fx)[VN], const AxisCoef<T>* xt, const RedAxis<T>& ry,
                                           const AxisCoef<T>& zt, const Cells<T, VN>& K, const Cells<T, VN>& m,
                                           Cells<T, VN>& O, Cells<T, VN>& t, Cells<T, VN>& u) {
  const T za = zt.s, zb = zt.om, zom = zt.ir, zop = zt.op;  // a, b, 1-σ, 1+σ
#pragma unroll
  for (int v = 0; v < VN; ++v) {
    AxisCoef<T> x{T(1), T(1), T(1), T(1)};
    bool f = false;
    if constexpr (WX) {
      x = xt[v];
      f = fx[v];
    }
    const T xa = x.s, xb = x.om;
    {  // component x: own axis x, next y, previous z
      T d = K.c[0].v[v];
      if constexpr (FY && FZ) {
        const T un = fma_rn(ry.a, u.c[0].v[v], mul_rn(ry.b, d));
        d = sub_rn(un, u.c[0].v[v]);
        u.c[0].v[v] = un;
      }
      const T A = FZ ? za : ry.a, B = FZ ? zb : ry.b;
      const T w = FY || FZ ? mul_rn(B, d) : d;
      const T o = O.c[0].v[v], mm = m.c[0].v[v], tt = t.c[0].v[v];
      T r = FY || FZ ? fma_rn(A, o, mul_rn(mm, w)) : fma_rn(mm, w, o);
      if constexpr (WX) {
        const T tn = FY || FZ ? fma_rn(A, tt, w) : add_rn(tt, w);
        const T rt = fma_rn(mm, fma_rn(x.op, tn, -mul_rn(x.ir, tt)), o);
        r = f ? rt : r;
        t.c[0].v[v] = f ? tn : tt;
      }
      O.c[0].v[v] = r;
    }
    {  // component y: own axis y, next z, previous x
      T d = K.c[1].v[v], A = za, B = zb;
      if constexpr (WX && FZ) {
        const T un = fma_rn(za, u.c[1].v[v], mul_rn(zb, d));
        d = f ? sub_rn(un, u.c[1].v[v]) : d;
        u.c[1].v[v] = f ? un : u.c[1].v[v];
        A = f ? xa : za;
        B = f ? xb : zb;
      } else if constexpr (WX) {
        A = xa;
        B = xb;
      }
      constexpr bool damp = WX || FZ;
      const T w = damp ? mul_rn(B, d) : d;
      const T o = O.c[1].v[v], mm = m.c[1].v[v], tt = t.c[1].v[v];
      if constexpr (FY) {
        const T tn = damp ? fma_rn(A, tt, w) : add_rn(tt, w);
        O.c[1].v[v] = fma_rn(mm, fma_rn(ry.op, tn, -mul_rn(ry.om, tt)), o);
        t.c[1].v[v] = tn;
      } else {
        O.c[1].v[v] = FZ ? fma_rn(A, o, mul_rn(mm, w)) : row_o<WX>(f, A, o, mm, w);
      }
    }
    {  // component z: own axis z, next x, previous y
      T d = K.c[2].v[v], A = xa, B = xb;
      if constexpr (WX && FY) {
        const T un = fma_rn(xa, u.c[2].v[v], mul_rn(xb, d));
        d = f ? sub_rn(un, u.c[2].v[v]) : d;
        u.c[2].v[v] = f ? un : u.c[2].v[v];
      }
      if constexpr (FY) {
        A = ry.a;
        B = ry.b;
      }
      constexpr bool damp = WX || FY;
      const T w = damp ? mul_rn(B, d) : d;
      const T o = O.c[2].v[v], mm = m.c[2].v[v], tt = t.c[2].v[v];
      if constexpr (FZ) {
        const T tn = damp ? fma_rn(A, tt, w) : add_rn(tt, w);
        O.c[2].v[v] = fma_rn(mm, fma_rn(zop, tn, -mul_rn(zom, tt)), o);
        t.c[2].v[v] = tn;
      } else {
        O.c[2].v[v] = FY ? fma_rn(A, o, mul_rn(mm, w)) : row_o<WX>(f, A, o, mm, w);
      }
    }
  }
}

// Component of a special cell (source, χ3, pole): the complete state, T always,
// U and W where its CPML stages have them.  has_w: own-axis CPML with σ ≠ 0, the
// condition under which the sparse passes go through W (not to be read off the
// factors, which are 1 for a σ below the rounding).
template <typename T>
__device__ __forceinline__ void special_component(bool has_w, const RedAxis<T>& o, const RedAxis<T>& n,
                                                  const RedAxis<T>& p, T K, T m, T& O, T& t, T& u, T& w) {
  T d = K;
  if (n.f) {
    const T un = fma_rn(n.a, u, mul_rn(n.b, K));
    d = sub_rn(un, u);
    u = un;
  }
  t = p.f ? fma_rn(p.a, t, mul_rn(p.b, d)) : add_rn(t, d);
  if (has_w) {
    const T wn = mul_rn(m, t);
    O = fma_rn(-o.om, w, fma_rn(o.op, wn, O));
    w = wn;
  } else {
    O = mul_rn(m, t);
  }
}

// VN cells from x0 on of which sp[v] are special ones (w: their W, where they
// have it; sx, sy, sz: σ of the cells along each axis, read where flagged).
template <typename T, int VN>
__device__ __forceinline__ void update_special_cells(const bool (&sp)[VN], const bool (&fx)[VN],
                                                     const AxisCoef<T>* sx, const AxisCoef<T>* sy, T sz,
                                                     const AxisCoef<T>* xt, const RedAxis<T>& ry,
                                                     const RedAxis<T>& rz, const Cells<T, VN>& K,
                                                     const Cells<T, VN>& m, Cells<T, VN>& O, Cells<T, VN>& t,
                                                     Cells<T, VN>& u, Cells<T, VN>& w) {
#pragma unroll
  for (int v = 0; v < VN; ++v) {
    RedAxis<T> rx{false, T(1), T(1), T(1), T(1)};
    if (fx[v]) rx = {true, xt[v].s, xt[v].om, xt[v].ir, xt[v].op};
    const RedAxis<T>* r[3] = {&rx, &ry, &rz};
    const bool has_w[3] = {fx[v] && sx[v].s != T(0), ry.f && sy->s != T(0), rz.f && sz != T(0)};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (sp[v])
        special_component(has_w[c], *r[c], *r[(c + 1) % 3], *r[(c + 2) % 3], K.c[c].v[v], m.c[c].v[v], O.c[c].v[v],
                          t.c[c].v[v], u.c[c].v[v], w.c[c].v[v]);
      else
        red_component(*r[c], *r[(c + 1) % 3], *r[(c + 2) % 3], K.c[c].v[v], m.c[c].v[v], O.c[c].v[v], t.c[c].v[v],
                      u.c[c].v[v]);
    }
  }
}

}  // namespace kh
