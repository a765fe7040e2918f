// Two values side by side in one operation.  sm_103a multiplies and adds pairs
// of FP32 numbers with one instruction (.f32x2): the FP32 pipe does the same
// work, but an instruction-bound kernel issues half as much for it.  Every
// component is rounded as by the scalar operation, so a packed computation gives
// the bits of two scalar ones.
//
// The products take an addend z = (-0, -0) that the compiler must not know (a
// kernel argument): ptxas contracts a packed product and the sum that follows it
// into one operation even where each asks for its own rounding (and sees through a
// constant zero), which would break the error-free transformations.
//
// Pk<real>::P is a pair of values (FP32, double-float or FP64) and also the
// memory image of one: {v0, v1}, for double-floats {hi0, hi1, lo0, lo1}.
#pragma once

#include "df64.cuh"

namespace ouranos {

using f2 = unsigned long long;  // two FP32 numbers

__device__ __forceinline__ f2 f2_make(float a, float b) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float f2_get(f2 a, int r) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return r ? y : x;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) { return f2_fma(b, f2_make(-1.f, -1.f), a); }  // a - b, one rounding

template <typename real>
struct Pk;

template <>
struct Pk<float> {
  using P = f2;
  using Acc = f2;
  using Op = f2;  // the second factor of products
  static __device__ __forceinline__ Op op(P v) { return v; }
  static __device__ __forceinline__ P make(float a, float b) { return f2_make(a, b); }
  static __device__ __forceinline__ float get(P v, int r) { return f2_get(v, r); }
  static __device__ __forceinline__ Acc from(P v) { return v; }
  static __device__ __forceinline__ Acc prod(P a, Op b, f2 z) { return f2_fma(a, b, z); }
  static __device__ __forceinline__ void fma(Acc& s, P a, Op b, f2) { s = f2_fma(a, b, s); }
  static __device__ __forceinline__ P raw(Acc s) { return s; }
  static __device__ __forceinline__ P result(Acc s) { return s; }
  static __device__ __forceinline__ P load(const void* p) { return *static_cast<const f2*>(p); }
  static __device__ __forceinline__ void store(void* p, P v) { *static_cast<f2*>(p) = v; }
  // 16 bytes hold the images of two pairs
  static __device__ __forceinline__ void from16(const uint4& u, P* o) {
    o[0] = f2_make(__uint_as_float(u.x), __uint_as_float(u.y));
    o[1] = f2_make(__uint_as_float(u.z), __uint_as_float(u.w));
  }
  // two neighbouring values {v0, v1} of an array
  static __device__ __forceinline__ P array_load(const unsigned char* p) { return *reinterpret_cast<const f2*>(p); }
  static __device__ __forceinline__ void array_put(unsigned char* p, P v) { *reinterpret_cast<f2*>(p) = v; }
  static __device__ __forceinline__ void array_store(float* p, P v) {
    __stcs(reinterpret_cast<float2*>(p), make_float2(f2_get(v, 0), f2_get(v, 1)));
  }
  static __device__ __forceinline__ P swap_if(P v, bool s) {
    const float a = f2_get(v, 0), b = f2_get(v, 1);
    return f2_make(s ? b : a, s ? a : b);
  }
};

template <>
struct Pk<df64> {
  struct P {
    f2 h, l;
  };
  struct Acc {
    f2 s, c;
  };
  static __device__ __forceinline__ P make(df64 a, df64 b) { return {f2_make(a.hi, b.hi), f2_make(a.lo, b.lo)}; }
  static __device__ __forceinline__ df64 get(P v, int r) { return df64(f2_get(v.h, r), f2_get(v.l, r)); }
  static __device__ __forceinline__ Acc from(P v) { return {v.h, v.l}; }
  struct Op {
    f2 h, l, nh;  // (nh = -h: the packed operations take no negated operands)
  };
  static __device__ __forceinline__ Op op(P v) { return {v.h, v.l, f2_sub(f2_make(-0.f, -0.f), v.h)}; }
  // the operations of acc_prod, acc_fma and acc_result (df64.cuh), two at a time
  static __device__ __forceinline__ Acc prod(P a, Op b, f2 z) {
    const f2 np = f2_fma(a.h, b.nh, z);
    f2 e = f2_fma(a.h, b.h, np);
    e = f2_fma(a.h, b.l, e);
    e = f2_fma(a.l, b.h, e);
    return {f2_sub(f2_make(-0.f, -0.f), np), e};
  }
  static __device__ __forceinline__ void fma(Acc& acc, P a, Op b, f2 z) {
    const f2 np = f2_fma(a.h, b.nh, z);  // -p
    f2 e = f2_fma(a.h, b.h, np);
    e = f2_fma(a.h, b.l, e);
    e = f2_fma(a.l, b.h, e);
    const f2 s = f2_sub(acc.s, np);
    const f2 bb = f2_sub(s, acc.s);
    const f2 t = f2_sub(f2_sub(acc.s, f2_sub(s, bb)), f2_add(np, bb));
    acc.s = s;
    acc.c = f2_add(acc.c, f2_add(t, e));
  }
  static __device__ __forceinline__ P raw(Acc s) { return {s.s, s.c}; }
  static __device__ __forceinline__ P result(Acc a) {
    const f2 hi = f2_add(a.s, a.c);
    return {hi, f2_add(a.c, f2_sub(a.s, hi))};
  }
  static __device__ __forceinline__ P load(const void* p) {
    P v;
    from16(*static_cast<const uint4*>(p), &v);
    return v;
  }
  static __device__ __forceinline__ void store(void* p, P v) {
    ulonglong2 u;
    u.x = v.h;
    u.y = v.l;
    *static_cast<ulonglong2*>(p) = u;
  }
  static __device__ __forceinline__ void from16(const uint4& u, P* o) {
    o->h = f2_make(__uint_as_float(u.x), __uint_as_float(u.y));
    o->l = f2_make(__uint_as_float(u.z), __uint_as_float(u.w));
  }
  static __device__ __forceinline__ P array_load(const unsigned char* p) {
    const float4 u = *reinterpret_cast<const float4*>(p);
    return {f2_make(u.x, u.z), f2_make(u.y, u.w)};
  }
  static __device__ __forceinline__ void array_put(unsigned char* p, P v) {
    *reinterpret_cast<float4*>(p) = make_float4(f2_get(v.h, 0), f2_get(v.l, 0), f2_get(v.h, 1), f2_get(v.l, 1));
  }
  static __device__ __forceinline__ void array_store(df64* p, P v) {
    __stcs(reinterpret_cast<float4*>(p),
           make_float4(f2_get(v.h, 0), f2_get(v.l, 0), f2_get(v.h, 1), f2_get(v.l, 1)));
  }
  static __device__ __forceinline__ P swap_if(P v, bool s) {
    return {Pk<float>::swap_if(v.h, s), Pk<float>::swap_if(v.l, s)};
  }
};

template <>
struct Pk<double> {
  struct P {
    double a, b;
  };
  using Acc = P;
  using Op = P;
  static __device__ __forceinline__ Op op(P v) { return v; }
  static __device__ __forceinline__ P make(double a, double b) { return {a, b}; }
  static __device__ __forceinline__ double get(P v, int r) { return r ? v.b : v.a; }
  static __device__ __forceinline__ Acc from(P v) { return v; }
  static __device__ __forceinline__ Acc prod(P x, Op y, f2) { return {__dmul_rn(x.a, y.a), __dmul_rn(x.b, y.b)}; }
  static __device__ __forceinline__ void fma(Acc& s, P x, Op y, f2) {
    s.a = __fma_rn(x.a, y.a, s.a);
    s.b = __fma_rn(x.b, y.b, s.b);
  }
  static __device__ __forceinline__ P raw(Acc s) { return s; }
  static __device__ __forceinline__ P result(Acc s) { return s; }
  static __device__ __forceinline__ P load(const void* p) {
    const double2 u = *static_cast<const double2*>(p);
    return {u.x, u.y};
  }
  static __device__ __forceinline__ void store(void* p, P v) { *static_cast<double2*>(p) = make_double2(v.a, v.b); }
  static __device__ __forceinline__ void from16(const uint4& u, P* o) {
    o->a = __hiloint2double((int)u.y, (int)u.x);
    o->b = __hiloint2double((int)u.w, (int)u.z);
  }
  static __device__ __forceinline__ P array_load(const unsigned char* p) { return load(p); }
  static __device__ __forceinline__ void array_put(unsigned char* p, P v) { store(p, v); }
  static __device__ __forceinline__ void array_store(double* p, P v) {
    __stcs(reinterpret_cast<double2*>(p), make_double2(v.a, v.b));
  }
  static __device__ __forceinline__ P swap_if(P v, bool s) { return {s ? v.b : v.a, s ? v.a : v.b}; }
};

}  // namespace ouranos
