// Forward-mode dual numbers (value + one tangent) for the adjoint pass.
//
// Instantiating the translated formula code with T = Dual<S> carries the
// directional derivative of every intermediate along one tangent: seeding the
// position with dp/dtheta and the parameters with dparams/dtheta yields dDE/dtheta in
// one evaluation.  Functions follow their derivative rules; piecewise-constant ones
// (floor, round, sign, comparisons) have a zero tangent, and min/max/select follow
// the branch the value takes.  S is float (Dual1, the FP32 adjoint) or double.
#pragma once

#include "nd_wgsl.h"

namespace ndw {

template <class S> struct Dual {
  S v, d;
  ND_HD_INLINE Dual() : v(S(0)), d(S(0)) {}
  ND_HD_INLINE Dual(float x) : v(S(x)), d(S(0)) {}
  ND_HD_INLINE Dual(double x) : v(S(x)), d(S(0)) {}
  ND_HD_INLINE Dual(int x) : v(S(x)), d(S(0)) {}
  ND_HD_INLINE Dual(unsigned x) : v(S(x)), d(S(0)) {}
  ND_HD_INLINE Dual(S x, S t, int) : v(x), d(t) {}
  ND_HD_INLINE explicit operator float() const { return float(v); }
  ND_HD_INLINE explicit operator double() const { return double(v); }
  ND_HD_INLINE Dual& operator+=(Dual o) { v += o.v; d += o.d; return *this; }
  ND_HD_INLINE Dual& operator-=(Dual o) { v -= o.v; d -= o.d; return *this; }
  ND_HD_INLINE Dual& operator*=(Dual o) { d = d * o.v + v * o.d; v *= o.v; return *this; }
  ND_HD_INLINE Dual& operator/=(Dual o) {
    const S q = v / o.v;
    d = (d - q * o.d) / o.v;
    v = q;
    return *this;
  }
};
typedef Dual<float> Dual1;

template <class S> ND_HD_INLINE Dual<S> mkd(S v, S d) { return Dual<S>(v, d, 0); }

template <class S> ND_HD_INLINE Dual<S> operator+(Dual<S> a, Dual<S> b) { return mkd(a.v + b.v, a.d + b.d); }
template <class S> ND_HD_INLINE Dual<S> operator-(Dual<S> a, Dual<S> b) { return mkd(a.v - b.v, a.d - b.d); }
template <class S> ND_HD_INLINE Dual<S> operator*(Dual<S> a, Dual<S> b) { return mkd(a.v * b.v, a.d * b.v + a.v * b.d); }
template <class S> ND_HD_INLINE Dual<S> operator/(Dual<S> a, Dual<S> b) {
  const S q = a.v / b.v;
  return mkd(q, (a.d - q * b.d) / b.v);
}
template <class S> ND_HD_INLINE Dual<S> operator-(Dual<S> a) { return mkd(-a.v, -a.d); }
template <class S> ND_HD_INLINE bool operator<(Dual<S> a, Dual<S> b) { return a.v < b.v; }
template <class S> ND_HD_INLINE bool operator>(Dual<S> a, Dual<S> b) { return a.v > b.v; }
template <class S> ND_HD_INLINE bool operator<=(Dual<S> a, Dual<S> b) { return a.v <= b.v; }
template <class S> ND_HD_INLINE bool operator>=(Dual<S> a, Dual<S> b) { return a.v >= b.v; }
template <class S> ND_HD_INLINE bool operator==(Dual<S> a, Dual<S> b) { return a.v == b.v; }
template <class S> ND_HD_INLINE bool operator!=(Dual<S> a, Dual<S> b) { return a.v != b.v; }

template <class S> ND_HD_INLINE Dual<S> sin(Dual<S> a) { return mkd(sin(a.v), cos(a.v) * a.d); }
template <class S> ND_HD_INLINE Dual<S> cos(Dual<S> a) { return mkd(cos(a.v), -sin(a.v) * a.d); }
template <class S> ND_HD_INLINE Dual<S> tan(Dual<S> a) {
  const S t = tan(a.v);
  return mkd(t, (S(1) + t * t) * a.d);
}
template <class S> ND_HD_INLINE Dual<S> asin(Dual<S> a) {
  return mkd(asin(a.v), a.d / sqrt(max(S(1) - a.v * a.v, S(1e-30))));
}
template <class S> ND_HD_INLINE Dual<S> acos(Dual<S> a) {
  return mkd(acos(a.v), -a.d / sqrt(max(S(1) - a.v * a.v, S(1e-30))));
}
template <class S> ND_HD_INLINE Dual<S> atan(Dual<S> a) { return mkd(atan(a.v), a.d / (S(1) + a.v * a.v)); }
template <class S> ND_HD_INLINE Dual<S> atan2(Dual<S> y, Dual<S> x) {
  const S r2 = x.v * x.v + y.v * y.v;
  return mkd(atan2(y.v, x.v), r2 > S(0) ? (x.v * y.d - y.v * x.d) / r2 : S(0));
}
template <class S> ND_HD_INLINE Dual<S> sinh(Dual<S> a) { return mkd(sinh(a.v), cosh(a.v) * a.d); }
template <class S> ND_HD_INLINE Dual<S> cosh(Dual<S> a) { return mkd(cosh(a.v), sinh(a.v) * a.d); }
template <class S> ND_HD_INLINE Dual<S> tanh(Dual<S> a) {
  const S t = tanh(a.v);
  return mkd(t, (S(1) - t * t) * a.d);
}
template <class S> ND_HD_INLINE Dual<S> exp(Dual<S> a) {
  const S e = exp(a.v);
  return mkd(e, e * a.d);
}
template <class S> ND_HD_INLINE Dual<S> exp2(Dual<S> a) {
  const S e = exp2(a.v);
  return mkd(e, e * S(0.6931471805599453) * a.d);
}
template <class S> ND_HD_INLINE Dual<S> log(Dual<S> a) { return mkd(log(a.v), a.d / a.v); }
template <class S> ND_HD_INLINE Dual<S> log2(Dual<S> a) { return mkd(log2(a.v), a.d / (a.v * S(0.6931471805599453))); }
template <class S> ND_HD_INLINE Dual<S> sqrt(Dual<S> a) {
  const S s = sqrt(a.v);
  return mkd(s, s > S(0) ? a.d / (S(2) * s) : S(0));
}
template <class S> ND_HD_INLINE Dual<S> inverseSqrt(Dual<S> a) {
  const S r = S(1) / sqrt(a.v);
  return mkd(r, S(-0.5) * r * r * r * a.d);
}
template <class S> ND_HD_INLINE Dual<S> pow(Dual<S> x, Dual<S> y) {
  if (x.v < S(0)) return mkd(S(0) / S(0), S(0));
  const S p = pow(x.v, y.v);
  S dp = S(0);
  if (x.d != S(0)) dp += y.v * pow(x.v, y.v - S(1)) * x.d;
  if (y.d != S(0) && x.v > S(0)) dp += p * log(x.v) * y.d;
  return mkd(p, dp);
}
template <class S> ND_HD_INLINE Dual<S> floor(Dual<S> a) { return mkd(floor(a.v), S(0)); }
template <class S> ND_HD_INLINE Dual<S> ceil(Dual<S> a) { return mkd(ceil(a.v), S(0)); }
template <class S> ND_HD_INLINE Dual<S> trunc(Dual<S> a) { return mkd(trunc(a.v), S(0)); }
template <class S> ND_HD_INLINE Dual<S> round(Dual<S> a) { return mkd(round(a.v), S(0)); }
template <class S> ND_HD_INLINE Dual<S> abs(Dual<S> a) { return a.v < S(0) ? -a : a; }
template <class S> ND_HD_INLINE Dual<S> sign(Dual<S> a) {
  return mkd(a.v > S(0) ? S(1) : (a.v < S(0) ? S(-1) : S(0)), S(0));
}
template <class S> ND_HD_INLINE Dual<S> min(Dual<S> a, Dual<S> b) { return b.v < a.v ? b : a; }
template <class S> ND_HD_INLINE Dual<S> max(Dual<S> a, Dual<S> b) { return b.v > a.v ? b : a; }
template <class S> ND_HD_INLINE Dual<S> fma(Dual<S> a, Dual<S> b, Dual<S> c) { return a * b + c; }
template <class S> ND_HD_INLINE Dual<S> radians(Dual<S> a) {
  return mkd(a.v * S(0.017453292519943295), a.d * S(0.017453292519943295));
}
template <class S> ND_HD_INLINE Dual<S> degrees(Dual<S> a) {
  return mkd(a.v * S(57.29577951308232), a.d * S(57.29577951308232));
}
template <class S> ND_HD_INLINE Dual<S> select(Dual<S> f, Dual<S> t, bool c) { return c ? t : f; }
template <class S> ND_HD_INLINE void sin_cos(Dual<S> x, Dual<S>& s, Dual<S>& c) {
  const S sv = sin(x.v), cv = cos(x.v);
  s = mkd(sv, cv * x.d);
  c = mkd(cv, -sv * x.d);
}

template <class S, int N> struct Duals {
  S v;
  S d[N];
  ND_HD_INLINE Duals() : Duals(S(0), 0) {}
  ND_HD_INLINE Duals(float x) : Duals(S(x), 0) {}
  ND_HD_INLINE Duals(double x) : Duals(S(x), 0) {}
  ND_HD_INLINE Duals(int x) : Duals(S(x), 0) {}
  ND_HD_INLINE Duals(unsigned x) : Duals(S(x), 0) {}
  ND_HD_INLINE Duals(S x, int) : v(x) {
    for (int i = 0; i < N; ++i) d[i] = S(0);
  }
  ND_HD_INLINE explicit operator float() const { return float(v); }
  ND_HD_INLINE explicit operator double() const { return double(v); }
  ND_HD_INLINE Duals& operator+=(Duals o) { return *this = *this + o; }
  ND_HD_INLINE Duals& operator-=(Duals o) { return *this = *this - o; }
  ND_HD_INLINE Duals& operator*=(Duals o) { return *this = *this * o; }
  ND_HD_INLINE Duals& operator/=(Duals o) { return *this = *this / o; }
};

// A dual with value v and the tangents f(0), ..., f(N - 1).
template <int N, class S, class F> ND_HD_INLINE Duals<S, N> mkds(S v, F f) {
  Duals<S, N> r(v, 0);
#pragma unroll
  for (int i = 0; i < N; ++i) r.d[i] = f(i);
  return r;
}
// Divides tangents by x.
template <class S> struct Divisor {
  S x;
  ND_HD_INLINE explicit Divisor(S a) : x(std::is_same<S, double>::value ? S(1) / a : a) {}
  ND_HD_INLINE S operator()(S a) const { return std::is_same<S, double>::value ? a * x : a / x; }
};

#define ND_DUAL template <class S, int N> ND_HD_INLINE
#define ND_DUAL1 ND_DUAL Duals<S, N>
ND_DUAL1 operator+(Duals<S, N> a, Duals<S, N> b) {
  return mkds<N>(a.v + b.v, [&](int i) { return a.d[i] + b.d[i]; });
}
ND_DUAL1 operator-(Duals<S, N> a, Duals<S, N> b) {
  return mkds<N>(a.v - b.v, [&](int i) { return a.d[i] - b.d[i]; });
}
ND_DUAL1 operator*(Duals<S, N> a, Duals<S, N> b) {
  return mkds<N>(a.v * b.v, [&](int i) { return a.d[i] * b.v + a.v * b.d[i]; });
}
ND_DUAL1 operator/(Duals<S, N> a, Duals<S, N> b) {
  const S q = a.v / b.v;
  const Divisor<S> by(b.v);
  return mkds<N>(q, [&](int i) { return by(a.d[i] - q * b.d[i]); });
}
ND_DUAL1 operator-(Duals<S, N> a) {
  return mkds<N>(-a.v, [&](int i) { return -a.d[i]; });
}
ND_DUAL bool operator<(Duals<S, N> a, Duals<S, N> b) { return a.v < b.v; }
ND_DUAL bool operator>(Duals<S, N> a, Duals<S, N> b) { return a.v > b.v; }
ND_DUAL bool operator<=(Duals<S, N> a, Duals<S, N> b) { return a.v <= b.v; }
ND_DUAL bool operator>=(Duals<S, N> a, Duals<S, N> b) { return a.v >= b.v; }
ND_DUAL bool operator==(Duals<S, N> a, Duals<S, N> b) { return a.v == b.v; }
ND_DUAL bool operator!=(Duals<S, N> a, Duals<S, N> b) { return a.v != b.v; }

// A function of one argument with value f and derivative g there.
ND_DUAL1 chain(S f, S g, const Duals<S, N>& a) {
  return mkds<N>(f, [&](int i) { return g * a.d[i]; });
}
ND_DUAL1 sin(Duals<S, N> a) { return chain(sin(a.v), cos(a.v), a); }
ND_DUAL1 cos(Duals<S, N> a) { return chain(cos(a.v), -sin(a.v), a); }
ND_DUAL1 tan(Duals<S, N> a) {
  const S t = tan(a.v);
  return chain(t, S(1) + t * t, a);
}
ND_DUAL1 asin(Duals<S, N> a) {
  const Divisor<S> by(sqrt(max(S(1) - a.v * a.v, S(1e-30))));
  return mkds<N>(asin(a.v), [&](int i) { return by(a.d[i]); });
}
ND_DUAL1 acos(Duals<S, N> a) {
  const Divisor<S> by(sqrt(max(S(1) - a.v * a.v, S(1e-30))));
  return mkds<N>(acos(a.v), [&](int i) { return by(-a.d[i]); });
}
ND_DUAL1 atan(Duals<S, N> a) {
  const Divisor<S> by(S(1) + a.v * a.v);
  return mkds<N>(atan(a.v), [&](int i) { return by(a.d[i]); });
}
ND_DUAL1 atan2(Duals<S, N> y, Duals<S, N> x) {
  const S r2 = x.v * x.v + y.v * y.v;
  const Divisor<S> by(r2);
  return mkds<N>(atan2(y.v, x.v), [&](int i) { return r2 > S(0) ? by(x.v * y.d[i] - y.v * x.d[i]) : S(0); });
}
ND_DUAL1 sinh(Duals<S, N> a) { return chain(sinh(a.v), cosh(a.v), a); }
ND_DUAL1 cosh(Duals<S, N> a) { return chain(cosh(a.v), sinh(a.v), a); }
ND_DUAL1 tanh(Duals<S, N> a) {
  const S t = tanh(a.v);
  return chain(t, S(1) - t * t, a);
}
ND_DUAL1 exp(Duals<S, N> a) {
  const S e = exp(a.v);
  return chain(e, e, a);
}
ND_DUAL1 exp2(Duals<S, N> a) {
  const S e = exp2(a.v);
  return chain(e, e * S(0.6931471805599453), a);
}
ND_DUAL1 log(Duals<S, N> a) {
  const Divisor<S> by(a.v);
  return mkds<N>(log(a.v), [&](int i) { return by(a.d[i]); });
}
ND_DUAL1 log2(Duals<S, N> a) {
  const Divisor<S> by(a.v * S(0.6931471805599453));
  return mkds<N>(log2(a.v), [&](int i) { return by(a.d[i]); });
}
ND_DUAL1 sqrt(Duals<S, N> a) {
  const S s = sqrt(a.v);
  const Divisor<S> by(S(2) * s);
  return mkds<N>(s, [&](int i) { return s > S(0) ? by(a.d[i]) : S(0); });
}
ND_DUAL1 inverseSqrt(Duals<S, N> a) {
  const S r = S(1) / sqrt(a.v);
  return chain(r, S(-0.5) * r * r * r, a);
}
ND_DUAL1 pow(Duals<S, N> x, Duals<S, N> y) {
  if (x.v < S(0)) return Duals<S, N>(S(0) / S(0), 0);
  const S p = pow(x.v, y.v);
  // y x^(y - 1): FP64 duals take the power from p, in place of a second 64-bit power
  const S g = y.v * (std::is_same<S, double>::value && x.v > S(0) && p > S(0) ? p / x.v : pow(x.v, y.v - S(1)));
  return mkds<N>(p, [&](int i) {
    S dp = S(0);
    if (x.d[i] != S(0)) dp += g * x.d[i];
    if (y.d[i] != S(0) && x.v > S(0)) dp += p * log(x.v) * y.d[i];
    return dp;
  });
}
ND_DUAL1 floor(Duals<S, N> a) { return Duals<S, N>(floor(a.v), 0); }
ND_DUAL1 ceil(Duals<S, N> a) { return Duals<S, N>(ceil(a.v), 0); }
ND_DUAL1 trunc(Duals<S, N> a) { return Duals<S, N>(trunc(a.v), 0); }
ND_DUAL1 round(Duals<S, N> a) { return Duals<S, N>(round(a.v), 0); }
ND_DUAL1 abs(Duals<S, N> a) { return a.v < S(0) ? -a : a; }
ND_DUAL1 sign(Duals<S, N> a) {
  return Duals<S, N>(a.v > S(0) ? S(1) : (a.v < S(0) ? S(-1) : S(0)), 0);
}
ND_DUAL1 min(Duals<S, N> a, Duals<S, N> b) { return b.v < a.v ? b : a; }
ND_DUAL1 max(Duals<S, N> a, Duals<S, N> b) { return b.v > a.v ? b : a; }
ND_DUAL1 fma(Duals<S, N> a, Duals<S, N> b, Duals<S, N> c) { return a * b + c; }
ND_DUAL1 radians(Duals<S, N> a) { return chain(a.v * S(0.017453292519943295), S(0.017453292519943295), a); }
ND_DUAL1 degrees(Duals<S, N> a) { return chain(a.v * S(57.29577951308232), S(57.29577951308232), a); }
ND_DUAL1 select(Duals<S, N> f, Duals<S, N> t, bool c) { return c ? t : f; }
ND_DUAL void sin_cos(Duals<S, N> x, Duals<S, N>& s, Duals<S, N>& c) {
  const S sv = sin(x.v), cv = cos(x.v);
  s = chain(sv, cv, x);
  c = chain(cv, -sv, x);
}
#undef ND_DUAL1
#undef ND_DUAL

}  // namespace ndw
