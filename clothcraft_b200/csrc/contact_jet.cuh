// OGC contact energy by forward differentiation (Jet3), for the FP32-assembly
// sweep. The FP64 sweep uses the closed forms of sweep_terms.cuh, which agree
// with these to ~1e-13; the FP32 form keeps this evaluation because its blocks are
// rounded to FP32 afterwards: a last-bit change of an FP64 term now and then
// changes an FP32 rounding, and the 100-step runs that its energy bar is checked
// on (a sheet sliding on a sphere) do not return to within that bar once two
// trajectories differ at all.
#pragma once
#include "sweep_terms.cuh"

namespace cc {
namespace jet {

// ----------------------------------------------- contact: forward-mode AD
// Jet3 with a symmetric Hessian: the second-order chain rules of
// src/math.rs:46-122, restricted to one vertex's three coordinates.
struct J3 {
    double v;
    double g0, g1, g2;
    double h00, h01, h02, h11, h12, h22;
};
__device__ __forceinline__ J3 jc(double v) { return {v, 0, 0, 0, 0, 0, 0, 0, 0, 0}; }
__device__ __forceinline__ J3 operator+(const J3& a, const J3& b) {
    return {a.v + b.v,     a.g0 + b.g0,   a.g1 + b.g1,   a.g2 + b.g2,   a.h00 + b.h00,
            a.h01 + b.h01, a.h02 + b.h02, a.h11 + b.h11, a.h12 + b.h12, a.h22 + b.h22};
}
__device__ __forceinline__ J3 operator-(const J3& a, const J3& b) {
    return {a.v - b.v,     a.g0 - b.g0,   a.g1 - b.g1,   a.g2 - b.g2,   a.h00 - b.h00,
            a.h01 - b.h01, a.h02 - b.h02, a.h11 - b.h11, a.h12 - b.h12, a.h22 - b.h22};
}
__device__ __forceinline__ J3 operator-(const J3& a) {
    return {-a.v, -a.g0, -a.g1, -a.g2, -a.h00, -a.h01, -a.h02, -a.h11, -a.h12, -a.h22};
}
__device__ __forceinline__ J3 operator*(const J3& a, const J3& b) {
    J3 r;
    r.v = a.v * b.v;
    r.g0 = a.g0 * b.v + a.v * b.g0;
    r.g1 = a.g1 * b.v + a.v * b.g1;
    r.g2 = a.g2 * b.v + a.v * b.g2;
    r.h00 = a.h00 * b.v + a.v * b.h00 + 2.0 * a.g0 * b.g0;
    r.h01 = a.h01 * b.v + a.v * b.h01 + a.g0 * b.g1 + b.g0 * a.g1;
    r.h02 = a.h02 * b.v + a.v * b.h02 + a.g0 * b.g2 + b.g0 * a.g2;
    r.h11 = a.h11 * b.v + a.v * b.h11 + 2.0 * a.g1 * b.g1;
    r.h12 = a.h12 * b.v + a.v * b.h12 + a.g1 * b.g2 + b.g1 * a.g2;
    r.h22 = a.h22 * b.v + a.v * b.h22 + 2.0 * a.g2 * b.g2;
    return r;
}
__device__ __forceinline__ J3 chain(const J3& a, double value, double f1, double f2) {
    J3 r;
    r.v = value;
    r.g0 = f1 * a.g0;
    r.g1 = f1 * a.g1;
    r.g2 = f1 * a.g2;
    r.h00 = f1 * a.h00 + f2 * a.g0 * a.g0;
    r.h01 = f1 * a.h01 + f2 * a.g0 * a.g1;
    r.h02 = f1 * a.h02 + f2 * a.g0 * a.g2;
    r.h11 = f1 * a.h11 + f2 * a.g1 * a.g1;
    r.h12 = f1 * a.h12 + f2 * a.g1 * a.g2;
    r.h22 = f1 * a.h22 + f2 * a.g2 * a.g2;
    return r;
}
__device__ __forceinline__ J3 operator/(const J3& a, const J3& b) {
    return a * chain(b, 1.0 / b.v, -1.0 / (b.v * b.v), 2.0 / (b.v * b.v * b.v));
}
__device__ __forceinline__ J3 ssqrt(const J3& a) {
    double r = sqrt(a.v);
    return chain(a, r, 0.5 / r, -0.25 / (r * r * r));
}
__device__ __forceinline__ J3 sln(const J3& a) { return chain(a, log(a.v), 1.0 / a.v, -1.0 / (a.v * a.v)); }
__device__ __forceinline__ double ssqrt(double x) { return sqrt(x); }
__device__ __forceinline__ double sln(double x) { return log(x); }
__device__ __forceinline__ double sval(double x) { return x; }
__device__ __forceinline__ double sval(const J3& x) { return x.v; }
template <class S>
__device__ __forceinline__ S scst(double v);
template <>
__device__ __forceinline__ double scst<double>(double v) {
    return v;
}
template <>
__device__ __forceinline__ J3 scst<J3>(double v) {
    return jc(v);
}

template <class S>
struct V {
    S x, y, z;
};
template <class S>
__device__ __forceinline__ V<S> vsub(const V<S>& a, const V<S>& b) {
    return {a.x - b.x, a.y - b.y, a.z - b.z};
}
template <class S>
__device__ __forceinline__ S vdot(const V<S>& a, const V<S>& b) {
    return a.x * b.x + a.y * b.y + a.z * b.z;
}
template <class S>
__device__ __forceinline__ V<S> vcross(const V<S>& a, const V<S>& b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// activation (src/ogc/potential.rs:8-22)
template <class S>
__device__ __forceinline__ S activation(const S& d, double r, double k) {
    if (sval(d) >= r) return scst<S>(0.0);
    if (sval(d) <= 0.0) return scst<S>(__longlong_as_double(0x7ff0000000000000ll));
    double tau = 0.5 * r;
    if (sval(d) >= tau) {
        S gg = scst<S>(r) - d;
        return scst<S>(0.5 * k) * gg * gg;
    }
    return scst<S>(0.5 * k * tau * tau) - scst<S>(k * tau * tau) * sln(d / scst<S>(tau));
}

// Contact distance of Contact::energy (src/ogc/potential.rs:39-65) on four
// named points; `degenerate` is set for an EE pair with |n|^2 < 1e-30 (energy 0).
template <class S>
__device__ __forceinline__ S contact_distance(uint32_t kind, const V<S>& p0, const V<S>& p1, const V<S>& p2,
                                              const V<S>& p3, bool& degenerate) {
    degenerate = false;
    if (kind == 0) {
        V<S> v = vsub(p0, p1);
        return ssqrt(vdot(v, v));
    }
    if (kind == 1) {
        V<S> u = vsub(p2, p1);
        V<S> w = vsub(p0, p1);
        S q = vdot(w, u) / vdot(u, u);
        V<S> dd = {w.x - q * u.x, w.y - q * u.y, w.z - q * u.z};
        return ssqrt(vdot(dd, dd));
    }
    if (kind == 2) {
        V<S> n = vcross(vsub(p2, p1), vsub(p3, p1));
        S h = vdot(vsub(p0, p1), n) / ssqrt(vdot(n, n));
        return sval(h) < 0.0 ? -h : h;
    }
    V<S> n = vcross(vsub(p1, p0), vsub(p3, p2));
    if (sval(vdot(n, n)) < 1e-30) {
        degenerate = true;
        return scst<S>(0.0);
    }
    S h = vdot(vsub(p0, p2), n) / ssqrt(vdot(n, n));
    return sval(h) < 0.0 ? -h : h;
}

// Contact::energy (src/ogc/potential.rs:39-65) on four named points.
template <class S>
__device__ __forceinline__ S contact_energy_t(uint32_t kind, double eps, const V<S>& p0, const V<S>& p1,
                                              const V<S>& p2, const V<S>& p3, double r, double k) {
    bool degenerate;
    S d = contact_distance<S>(kind, p0, p1, p2, p3, degenerate);
    if (degenerate) return scst<S>(0.0);
    S e = activation(d, r, k);
    if (kind == 3) {
        V<S> n = vcross(vsub(p1, p0), vsub(p3, p2));
        S q = vdot(n, n) / scst<S>(eps);
        if (sval(q) < 1.0) e = e * q * (scst<S>(2.0) - q);
    }
    return e;
}

// ---- mixed Jet/constant arithmetic: only the moving vertex carries derivatives
__device__ __forceinline__ J3 operator+(const J3& a, double b) {
    J3 r = a;
    r.v += b;
    return r;
}
__device__ __forceinline__ J3 operator+(double a, const J3& b) { return b + a; }
__device__ __forceinline__ J3 operator-(const J3& a, double b) {
    J3 r = a;
    r.v -= b;
    return r;
}
__device__ __forceinline__ J3 operator-(double a, const J3& b) {
    J3 r = -b;
    r.v += a;
    return r;
}
__device__ __forceinline__ J3 operator*(const J3& a, double b) {
    return {a.v * b, a.g0 * b, a.g1 * b, a.g2 * b, a.h00 * b, a.h01 * b, a.h02 * b, a.h11 * b, a.h12 * b, a.h22 * b};
}
__device__ __forceinline__ J3 operator*(double a, const J3& b) { return b * a; }
__device__ __forceinline__ J3 operator/(const J3& a, double b) { return a * (1.0 / b); }
__device__ __forceinline__ J3 operator/(double a, const J3& b) {
    return chain(b, 1.0 / b.v, -1.0 / (b.v * b.v), 2.0 / (b.v * b.v * b.v)) * a;
}
__device__ __forceinline__ J3 to_j3(const J3& a) { return a; }
__device__ __forceinline__ J3 to_j3(double a) { return jc(a); }

template <class A, class B>
struct Pro {
    using T = J3;
};
template <>
struct Pro<double, double> {
    using T = double;
};
template <class A, class B>
__device__ __forceinline__ V<typename Pro<A, B>::T> msub(const V<A>& a, const V<B>& b) {
    return {a.x - b.x, a.y - b.y, a.z - b.z};
}
template <class A, class B>
__device__ __forceinline__ typename Pro<A, B>::T mdot(const V<A>& a, const V<B>& b) {
    return a.x * b.x + a.y * b.y + a.z * b.z;
}
template <class A, class B>
__device__ __forceinline__ V<typename Pro<A, B>::T> mcross(const V<A>& a, const V<B>& b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// Contact::energy (src/ogc/potential.rs:39-65) with per-point types.
template <class S0, class S1, class S2, class S3>
__device__ __forceinline__ J3 contact_jet(uint32_t kind, double eps, const V<S0>& p0, const V<S1>& p1,
                                          const V<S2>& p2, const V<S3>& p3, double r, double k) {
    if (kind == 0) {
        auto v = msub(p0, p1);
        return to_j3(activation(ssqrt(mdot(v, v)), r, k));
    }
    if (kind == 1) {
        auto u = msub(p2, p1);
        auto w = msub(p0, p1);
        auto q = mdot(w, u) / mdot(u, u);
        auto dx = w.x - q * u.x;
        auto dy = w.y - q * u.y;
        auto dz = w.z - q * u.z;
        return to_j3(activation(ssqrt(dx * dx + dy * dy + dz * dz), r, k));
    }
    if (kind == 2) {
        auto n = mcross(msub(p2, p1), msub(p3, p1));
        auto h = mdot(msub(p0, p1), n) / ssqrt(mdot(n, n));
        auto d = sval(h) < 0.0 ? -h : h;
        return to_j3(activation(d, r, k));
    }
    auto n = mcross(msub(p1, p0), msub(p3, p2));
    auto nn = mdot(n, n);
    if (sval(nn) < 1e-30) return jc(0.0);
    auto h = mdot(msub(p0, p2), n) / ssqrt(nn);
    auto d = sval(h) < 0.0 ? -h : h;
    J3 e = to_j3(activation(d, r, k));
    J3 q = to_j3(nn / eps);
    if (q.v < 1.0) e = e * q * (2.0 - q);
    return e;
}

__device__ __forceinline__ V<J3> var_point(d3 p) {
    J3 a = jc(p.x), b = jc(p.y), c = jc(p.z);
    a.g0 = 1.0;
    b.g1 = 1.0;
    c.g2 = 1.0;
    return {a, b, c};
}
__device__ __forceinline__ V<double> cst_point(const SweepView& s, uint32_t id) {
    d3 x = ld3(s.x, id);
    return {x.x, x.y, x.z};
}
__device__ __forceinline__ V<double> dpoint(const SweepView& s, uint32_t id, uint32_t v, d3 p) {
    d3 x = pos(s, id, v, p);
    return {x.x, x.y, x.z};
}

template <bool D>
__device__ __forceinline__ double contact_term(const SweepView& s, uint32_t c, uint32_t v, d3 p, d3& g, Sym& H) {
    uint32_t kind = s.contacts.kind[c];
    uint4 cv = s.contacts.verts[c];
    double eps = s.contacts.eps[c];
    if (D) {
        // Inactive term (d >= r): the activation is the constant 0, so the term
        // adds nothing to e, g or H; skip its derivative evaluation.
        bool degenerate;
        double d0 = contact_distance<double>(kind, dpoint(s, cv.x, v, p), dpoint(s, cv.y, v, p),
                                             dpoint(s, cv.z, v, p), dpoint(s, cv.w, v, p), degenerate);
        if (degenerate || d0 >= s.contact_r) return 0.0;
        // the moving vertex's slot among the used ones (unused slots hold 0)
        uint32_t cnt = kind == 0 ? 2u : (kind == 1 ? 3u : 4u);
        int slot = cv.x == v ? 0 : (cv.y == v ? 1 : ((cnt > 2 && cv.z == v) ? 2 : 3));
        double r = s.contact_r, k = s.contact_k;
        J3 e;
        if (slot == 0)
            e = contact_jet(kind, eps, var_point(p), cst_point(s, cv.y), cst_point(s, cv.z), cst_point(s, cv.w), r, k);
        else if (slot == 1)
            e = contact_jet(kind, eps, cst_point(s, cv.x), var_point(p), cst_point(s, cv.z), cst_point(s, cv.w), r, k);
        else if (slot == 2)
            e = contact_jet(kind, eps, cst_point(s, cv.x), cst_point(s, cv.y), var_point(p), cst_point(s, cv.w), r, k);
        else
            e = contact_jet(kind, eps, cst_point(s, cv.x), cst_point(s, cv.y), cst_point(s, cv.z), var_point(p), r, k);
        g = g + mk(e.g0, e.g1, e.g2);
        H.a[0] += e.h00;
        H.a[1] += e.h01;
        H.a[2] += e.h02;
        H.a[3] += e.h11;
        H.a[4] += e.h12;
        H.a[5] += e.h22;
        return e.v;
    }
    return contact_energy_t<double>(kind, eps, dpoint(s, cv.x, v, p), dpoint(s, cv.y, v, p), dpoint(s, cv.z, v, p),
                                    dpoint(s, cv.w, v, p), s.contact_r, s.contact_k);
}

}  // namespace jet
}  // namespace cc
