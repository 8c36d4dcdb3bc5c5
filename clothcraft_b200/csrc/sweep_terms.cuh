// Device-side terms of the VBD local solve shared by the FP64 sweep
// (sweep.cu) and the FP32-assembly sweep (sweep32.cu): 3x3 symmetric blocks,
// the FP64 membrane and bending terms, stitches, the grab and the OGC contact
// energy, all with exact derivatives in closed form.
#pragma once
#include "sweep.cuh"

namespace cc {

// --------------------------------------------------------------- 3x3 sym
struct Sym {  // xx xy xz yy yz zz
    double a[6];
};
__device__ __forceinline__ void sym_zero(Sym& h) {
#pragma unroll
    for (int i = 0; i < 6; ++i) h.a[i] = 0.0;
}
__device__ __forceinline__ void sym_add_outer(Sym& h, d3 u, double s) {  // h += s u u^T
    h.a[0] += s * u.x * u.x;
    h.a[1] += s * u.x * u.y;
    h.a[2] += s * u.x * u.z;
    h.a[3] += s * u.y * u.y;
    h.a[4] += s * u.y * u.z;
    h.a[5] += s * u.z * u.z;
}
__device__ __forceinline__ void sym_add_outer2(Sym& h, d3 u, d3 v, double s) {  // h += s (u v^T + v u^T)
    h.a[0] += s * 2.0 * u.x * v.x;
    h.a[1] += s * (u.x * v.y + v.x * u.y);
    h.a[2] += s * (u.x * v.z + v.x * u.z);
    h.a[3] += s * 2.0 * u.y * v.y;
    h.a[4] += s * (u.y * v.z + v.y * u.z);
    h.a[5] += s * 2.0 * u.z * v.z;
}
__device__ __forceinline__ void sym_add_diag(Sym& h, double s) {
    h.a[0] += s;
    h.a[3] += s;
    h.a[5] += s;
}

// ----------------------------------------------------------------- terms
// axial (src/energy.rs:10-16) with its first and second derivative. With
// c == 1 (the pure quadratic law, e.g. StVK mapped with compression ratio 1)
// every (1 - c) term is exactly zero, so the square root and the reciprocal
// of the compression branch are skipped; the results are the same bits.
__device__ __forceinline__ void axial3(double s, double k, double c, double delta, double& f, double& f1, double& f2) {
    if (c == 1.0) {
        f = 0.5 * k * (c * s * s);
        f1 = k * (c * s);
        f2 = k * c;
        return;
    }
    double r = sqrt(s * s + delta * delta);
    double ir = 1.0 / r;
    double p = (s + r - delta) * 0.5;
    f = 0.5 * k * (c * s * s + (1.0 - c) * p * p);
    double p1 = 0.5 * (1.0 + s * ir);
    double p2 = 0.5 * delta * delta * (ir * ir * ir);
    f1 = k * (c * s + (1.0 - c) * p * p1);
    f2 = k * (c + (1.0 - c) * (p1 * p1 + p * p2));
}
__device__ __forceinline__ double axial1(double s, double k, double c, double delta) {
    if (c == 1.0) return 0.5 * k * (c * s * s);
    double r = sqrt(s * s + delta * delta);
    double p = (s + r - delta) * 0.5;
    return 0.5 * k * (c * s * s + (1.0 - c) * p * p);
}

__device__ __forceinline__ d3 pos(const SweepView& s, uint32_t i, uint32_t v, d3 p) {
    return i == v ? p : ld3(s.x, i);
}

// membrane (src/energy.rs:17-29) with one vertex at p; dj, dk: the other two
// vertices less p; b, k as VertexTerms has them. D: derivatives; HS: also the
// Hessian (a gradient-only evaluation skips it)
template <bool D, bool HS = D>
__device__ __forceinline__ double membrane(const SweepView& s, double4 b, double4 k, uint32_t mat, d3 dj, d3 dk, d3& g,
                                           Sym& H) {
    const d3 w = dj * b.x + dk * b.y, v = dj * b.z + dk * b.w;
    const double ew = (dot(w, w) - 1.0) * 0.5, ev = (dot(v, v) - 1.0) * 0.5, sh = dot(w, v);
    const double delta = k.w == 1.0 ? 0.0 : s.mats[mat].delta;  // unused by the pure quadratic law
    if (!D) return axial1(ew, k.x, k.w, delta) + axial1(ev, k.y, k.w, delta) + 0.5 * k.z * sh * sh;
    double fw, fw1, fw2, fv, fv1, fv2;
    axial3(ew, k.x, k.w, delta, fw, fw1, fw2);
    axial3(ev, k.y, k.w, delta, fv, fv1, fv2);
    const double aw = -(b.x + b.y), av = -(b.z + b.w);  // the rates of w and v in p
    const d3 q = v * aw + w * av;
    g = g + w * (fw1 * aw) + v * (fv1 * av) + q * (k.z * sh);
    if (HS) {
        sym_add_outer(H, w, fw2 * aw * aw);
        sym_add_outer(H, v, fv2 * av * av);
        sym_add_outer(H, q, k.z);
        sym_add_diag(H, fw1 * aw * aw + fv1 * av * av + 2.0 * k.z * sh * aw * av);
    }
    return fw + fv + 0.5 * k.z * sh * sh;
}

// energy of triangle t alone
__device__ __forceinline__ double membrane_energy(const SweepView& s, uint32_t t) {
    const int4 tv = s.tri_v[t];
    const double4 c = s.tri_coef[t];
    const double A = s.tri_area[t];
    const MatParams M = s.mats[tv.w];
    const d3 p = ld3(s.x, (uint32_t)tv.x);
    d3 g;
    Sym H;
    return membrane<false>(s, c, make_double4(A * M.warp, A * M.weft, A * M.shear, M.c), (uint32_t)tv.w,
                           ld3(s.x, (uint32_t)tv.y) - p, ld3(s.x, (uint32_t)tv.z) - p, g, H);
}

// bending (src/energy.rs:31-46): K |h1 - h2|^2 of a hinge's unit normals, which
// is 2K (1 - cos t) of the dihedral angle t. With sin t = S and cos t = h1.h2
// the derivatives in one vertex are 2K S grad t and 2K (cos t grad t grad t^T +
// S Hess t). A vertex is either an end of the shared edge or a wing (the corner
// of one triangle opposite the edge), and the two have their own closed forms
// (bending_edge, bending_wing); a hinge's corners in the order that the form
// needs are hinge_points. Generic second derivatives of both normals (skew
// matrices and projections) took ~250 FP64 operations for either role; these
// take ~70 (wing) and ~130 (edge).

// Corners of hinge (x0 x1 the edge, x2 and x3 the wings) as seen from slot:
// edge ends: {other end, wing A, wing B} with nA = (o - A) x (o - p) and
// nB = (o - p) x (o - B); wings: {edge, edge, other wing} with n1 = e x (p - x0).
// Renaming (x0, x1, x2, x3) -> (x1, x0, x3, x2) keeps both normals, so slots 1
// and 3 are slots 0 and 2 of the renamed hinge.
__device__ __forceinline__ uint3 hinge_points(uint4 hv, uint32_t slot) {
    switch (slot) {
        case 0: return make_uint3(hv.y, hv.z, hv.w);
        case 1: return make_uint3(hv.x, hv.w, hv.z);
        case 2: return make_uint3(hv.x, hv.y, hv.w);
        default: return make_uint3(hv.y, hv.x, hv.z);
    }
}

// An end p of the shared edge. grad t = -(fA + fB) with f = (a.e) n / (|e| |n|^2),
// a from the wing to the other end and e = o - p; Hess t is the symmetric part of
// sum n (df/de)^T.
template <bool D, bool HS = D>
__device__ __forceinline__ double bending_edge(double K, d3 o, d3 xa, d3 xb, d3 p, d3& g, Sym& H) {
    const d3 e = o - p, a = o - xa, b = o - xb;
    const d3 na = cross(a, e), nb = cross(e, b);
    const double la = rsqrt(dot(na, na)), lb = rsqrt(dot(nb, nb));
    const d3 ha = na * la, hb = nb * lb;
    const d3 d = ha - hb;
    const double energy = K * dot(d, d);
    if (!D) return energy;
    const double ie = 1.0 / dot(e, e);
    const double ae = dot(a, e), be = dot(b, e);
    const d3 f = ha * (ae * la) + hb * (be * lb);            // |e| (fA + fB)
    const double q = 2.0 * K * ie * dot(e, cross(hb, ha));  // 2K S / |e|
    g = g - f * q;
    if (!HS) return energy;
    sym_add_outer(H, f, 2.0 * K * ie * dot(ha, hb));
    const d3 va = a - e * (ae * ie) - cross(ha, a) * (2.0 * ae * la);
    const d3 vb = b - e * (be * ie) - cross(b, hb) * (2.0 * be * lb);
    sym_add_outer2(H, ha, va, 0.5 * q * la);
    sym_add_outer2(H, hb, vb, 0.5 * q * lb);
    return energy;
}

// A wing p: only its own normal moves, turning about the edge e with p:
// grad t = h |e| / |n|, Hess t = -(|e|^2 / |n|^2) (t h^T + h t^T), t = h x e / |e|.
template <bool D, bool HS = D>
__device__ __forceinline__ double bending_wing(double K, d3 x0, d3 x1, d3 x3, d3 p, d3& g, Sym& H) {
    const d3 e = x1 - x0;
    const d3 n1 = cross(e, p - x0), n2 = cross(x3 - x0, e);
    const double l1 = rsqrt(dot(n1, n1)), l2 = rsqrt(dot(n2, n2));
    const d3 h1 = n1 * l1, h2 = n2 * l2;
    const d3 d = h1 - h2;
    const double energy = K * dot(d, d);
    if (!D) return energy;
    const double q = 2.0 * K * l1 * dot(e, cross(h2, h1));  // 2K S |e| / |n1|
    g = g + h1 * q;
    if (!HS) return energy;
    sym_add_outer(H, h1, 2.0 * K * l1 * l1 * dot(h1, h2) * dot(e, e));
    sym_add_outer2(H, cross(h1, e), h1, -q * l1);
    return energy;
}

// energy of hinge h alone
__device__ __forceinline__ double bending_energy(const SweepView& s, uint32_t h) {
    const uint4 v = s.hinge_v[h];
    d3 g;
    Sym H;
    return bending_wing<false>(s.hinge_k[h], ld3(s.x, v.x), ld3(s.x, v.y), ld3(s.x, v.w), ld3(s.x, v.z), g, H);
}

// stitch 0.5 k |sum w_j x_j|^2 (src/vbd.rs:217-227)
template <bool D>
__device__ __forceinline__ double stitch_term(const SweepView& s, uint32_t st, uint32_t v, d3 p, d3& g, Sym& H) {
    d3 d = mk(0, 0, 0);
    double wv = 0.0;
    for (uint32_t k = s.st_off[st]; k < s.st_off[st + 1]; ++k) {
        uint32_t j = s.st_v[k];
        double w = s.st_w[k];
        d = d + pos(s, j, v, p) * w;
        if (j == v) wv += w;
    }
    double K = s.st_k[st];
    if (D) {
        g = g + d * (K * wv);
        sym_add_diag(H, K * wv * wv);
    }
    return 0.5 * K * dot(d, d);
}

// ---------------------------------------------------------------- contact
// Contact::energy (src/ogc/potential.rs:39-65): an activation of the distance d
// of two features, for edge pairs times a mollifier of |n|^2. One vertex p of
// the contact moves; its derivatives are closed forms (second-order forward
// differentiation of the same expressions, ten components a value, took ~8 times
// the operations). The vertex's part in the contact is c.w (ContactRole) and the
// other points are c.x, c.y, c.z. For the last three roles d = |w.n| with
// n = g x f / |g x f|.

// activation (src/ogc/potential.rs:8-22) with its derivatives, d < r
__device__ __forceinline__ double activation(double d, double r, double k, double& f1, double& f2) {
    const double tau = 0.5 * r;
    if (d >= tau) {
        f1 = -k * (r - d);
        f2 = k;
        return 0.5 * k * (r - d) * (r - d);
    }
    f1 = f2 = 0.0;
    if (d <= 0.0) return __longlong_as_double(0x7ff0000000000000ll);
    const double kt = k * tau * tau, id = 1.0 / d;
    f1 = -kt * id;
    f2 = kt * id * id;
    return 0.5 * kt - kt * log(d / tau);
}

// Energy of the term with p at the moving vertex, and its gradient and Hessian.
// A term at d >= r adds nothing.
template <bool D, bool HS = D>
__device__ __forceinline__ double contact_rec(const SweepView& s, uint4 c, double eps, d3 p, d3& g, Sym& H) {
    const double r = s.contact_r, k = s.contact_k;
    double f1, f2;
    if (c.w <= ON_LINE) {
        d3 n;
        double d, t = -1.0, iu = 0.0;  // the gradient of d is -t n
        d3 u = mk(0, 0, 0);
        const d3 a = ld3(s.x, c.x);
        if (c.w == POINT) {
            n = p - a;
        } else {
            const d3 b = ld3(s.x, c.y);
            const d3 w = (c.w == FROM_LINE ? p : b) - a;
            u = (c.w == FROM_LINE ? b : p) - a;
            iu = 1.0 / dot(u, u);
            const double q = dot(w, u) * iu;
            if (c.w == ON_LINE) t = q;
            n = w - u * q;
        }
        d = sqrt(dot(n, n));
        if (d >= r) return 0.0;
        const double e = activation(d, r, k, f1, f2);
        if (!D || d <= 0.0) return e;
        const double id = 1.0 / d;
        n = n * id;
        g = g - n * (f1 * t);
        if (!HS) return e;
        // f2 t^2 n n^T + f1 Hess d, Hess d = (t^2 / d)(I - n n^T - u u^T / u^2)
        //   [ON_LINE: - (d / u^2) n n^T + (t / u^2)(n u^T + u n^T)]
        const double h = f1 * t * t * id;
        const bool end = c.w == ON_LINE;
        sym_add_diag(H, h);
        sym_add_outer(H, n, f2 * t * t - h - (end ? f1 * d * iu : 0.0));
        if (c.w != POINT) sym_add_outer(H, u, -h * iu);
        if (end) sym_add_outer2(H, n, u, f1 * t * iu);
        return e;
    }
    const d3 a = ld3(s.x, c.x), b = ld3(s.x, c.y), o = ld3(s.x, c.z);
    const bool edges = c.w == EDGES;
    const d3 f = edges ? o - b : b - a;
    const d3 e1 = c.w == FROM_PLANE ? o - a : p - a;
    const d3 w = c.w == FROM_PLANE ? p - a : (edges ? a - b : o - a);
    const d3 N = cross(e1, f);
    const double NN = dot(N, N);
    if (edges && NN < 1e-30) return 0.0;
    const double il = rsqrt(NN);
    const double h = dot(w, N) * il, d = fabs(h);
    if (d >= r) return 0.0;
    double e = activation(d, r, k, f1, f2);
    double psi = 1.0, psi1 = 0.0;
    const double qm = edges ? NN / eps : 1.0;
    if (qm < 1.0) {
        psi = qm * (2.0 - qm);
        psi1 = 2.0 - 2.0 * qm;
    }
    const double energy = e * psi;
    if (!D) return energy;
    if (d <= 0.0) {
        // touching features have infinite energy and no direction; mollified, no finite derivative either
        if (qm < 1.0) g.x = __longlong_as_double(0x7ff8000000000000ll);
        return energy;
    }
    const double sg = h < 0.0 ? -1.0 : 1.0;
    const d3 n = N * il;
    // n turns about f as p leaves the plane: grad h = -l n, Hess h = -h |m|^2 n n^T + l (m n^T + n m^T),
    // m = f x n / |N|, l = w.m; from the plane's point grad h = n
    const bool from = c.w == FROM_PLANE;
    const d3 m = cross(f, n) * il;
    const double l = from ? -1.0 : dot(w, m);
    d3 gh = n * (-l * sg * f1);  // gradient of the activation
    if (HS) {
        double on = psi * f2 * l * l;
        if (!from) {
            on -= psi * f1 * d * dot(m, m);
            sym_add_outer2(H, m, n, psi * f1 * sg * l);
        }
        sym_add_outer(H, n, on);
    }
    if (qm < 1.0) {
        // q = |N|^2 / eps: grad q = 2 f x N / eps, Hess q = 2 (f^2 I - f f^T) / eps
        const d3 gq = cross(f, N) * (2.0 / eps);
        if (HS) {
            sym_add_outer2(H, gh, gq, psi1);
            sym_add_outer(H, gq, -2.0 * e);
            const double hq = e * psi1 * 2.0 / eps;
            sym_add_diag(H, hq * dot(f, f));
            sym_add_outer(H, f, -hq);
        }
        gh = gh * psi + gq * (e * psi1);
    }
    g = g + gh;
    return energy;
}

// energy of contact c alone
__device__ __forceinline__ double contact_energy(const SweepView& s, uint32_t c) {
    const uint4 v = s.contacts.verts[c];
    d3 g;
    Sym H;
    return contact_rec<false>(s, contact_ref(s.contacts.kind[c], v, v.x), s.contacts.eps[c], ld3(s.x, v.x), g, H);
}

// grab 0.5 k |sum w_j x_j - target|^2 (src/vbd.rs:237-246)
template <bool D>
__device__ __forceinline__ double grab_term(const SweepView& s, uint32_t v, d3 p, d3& g, Sym& H) {
    const GrabDev& G = s.grab;
    d3 d = mk(-G.target[0], -G.target[1], -G.target[2]);
    double wv = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        d = d + pos(s, G.v[j], v, p) * G.w[j];
        if (G.v[j] == v) wv += G.w[j];
    }
    if (D) {
        g = g + d * (G.k * wv);
        sym_add_diag(H, G.k * wv * wv);
    }
    return 0.5 * G.k * dot(d, d);
}

// A vertex's terms with its neighbours' positions staged in shared memory, one
// column of kSlots positions per group of G lanes (an interior grid vertex has 12
// neighbours; further ones are read from global memory). A position is read
// once, by one lane, and all the terms of the derivative pass and of every
// line-search trial take it from there.
// FAR: the corners' and materials' ids come from far_tri and far_hinge, the
// positions from global memory. LEAN: nothing is loaded ahead (few registers).
template <int G, bool FAR = false, bool LEAN = false>
struct Near {
    static constexpr uint32_t kSlots = G >= 4 ? 24 : (LEAN ? 4 * G : 8 * G);
    static constexpr uint32_t kDoubles = 3 * kSlots;  // per group
    uint32_t v, nb0, n_nb, t0, nt, h0, ne, nw, ns, c0, c1;
    double* at;  // x, y and z of the staged positions

    // A lane's first record of each kind, loaded while the neighbours' ids and
    // positions are on their way; the loops of local_part load the next round's
    // records before they evaluate the present one.
    struct First {
        unsigned long long t;
        double4 tb, tk;
        ulonglong2 edge, wing;
        uint4 c;
        double eps;
    };

    __device__ __forceinline__ void head(const SweepView& s, uint32_t vertex) {
        v = vertex;
        const uint4 a = s.vt.head[2 * (size_t)v], b = s.vt.head[2 * (size_t)v + 1];
        nb0 = a.x, n_nb = a.y, t0 = a.z, nt = a.w;
        h0 = b.x, ne = b.y, nw = b.z, ns = b.w;
        c0 = s.contacts.inc_off[v];
        c1 = s.contacts.inc_off[v + 1];
    }
    // head i of the colour (k_color_heads)
    __device__ __forceinline__ void head_of_color(const SweepView& s, uint32_t i) {
        const uint4 a = s.heads[3 * (size_t)i], b = s.heads[3 * (size_t)i + 1], c = s.heads[3 * (size_t)i + 2];
        v = a.x, nb0 = a.y, n_nb = a.z, t0 = a.w;
        nt = b.x, h0 = b.y, ne = b.z, nw = b.w;
        ns = c.x, c0 = c.y, c1 = c.z;
    }
    __device__ __forceinline__ void tri(const SweepView& s, uint32_t i, First& f) const {
        if (i < nt) {
            f.t = s.vt.tri[t0 + i];
            f.tb = s.vt.tri_b[t0 + i];
            f.tk = s.vt.tri_k[t0 + i];
        }
    }
    __device__ __forceinline__ void contact(const SweepView& s, uint32_t k, First& f) const {
        if (k < c1) {
            f.c = s.contacts.ref[k];
            f.eps = s.contacts.ref_eps[k];
        }
    }
    __device__ __forceinline__ First first(const SweepView& s, uint32_t lane) const {
        First f{};
        if (LEAN) return f;
        tri(s, lane, f);
        if (lane < ne) f.edge = s.vt.hinge[h0 + lane];
        if (lane < nw) f.wing = s.vt.hinge[h0 + ne + lane];
        contact(s, c0 + lane, f);
        return f;
    }
    // The lane's neighbours, and their positions into shared memory (the whole
    // group calls it).
    static constexpr int kPer = (kSlots + G - 1) / G;
    struct Ids {
        uint32_t id[kPer];
    };
    __device__ __forceinline__ Ids ids(const SweepView& s, uint32_t lane) const {
        Ids r{};
        if (LEAN) return r;
        const uint32_t m = min(n_nb, kSlots);
#pragma unroll
        for (int j = 0; j < kPer; ++j) r.id[j] = lane + j * G < m ? s.vt.nb[nb0 + lane + j * G] : 0u;
        return r;
    }
    __device__ __forceinline__ void stage(const SweepView& s, const Ids& r, uint32_t lane, unsigned mask, double* smem) {
        at = smem;
        const uint32_t m = min(n_nb, kSlots);
        if (LEAN) {
            __syncwarp(mask);
#pragma unroll 1
            for (uint32_t k = lane; k < m; k += G) {
                const d3 q = ld3(s.x, s.vt.nb[nb0 + k]);
                at[k] = q.x;
                at[kSlots + k] = q.y;
                at[2 * kSlots + k] = q.z;
            }
            __syncwarp(mask);
            return;
        }
        d3 q[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (lane + j * G < m) q[j] = ld3(s.x, r.id[j]);
        __syncwarp(mask);  // the column's last reads are done
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const uint32_t k = lane + j * G;
            if (k < m) {
                at[k] = q[j].x;
                at[kSlots + k] = q[j].y;
                at[2 * kSlots + k] = q[j].z;
            }
        }
        __syncwarp(mask);
    }
    __device__ __forceinline__ First load(const SweepView& s, uint32_t lane, unsigned mask, double* smem) {
        const Ids r = ids(s, lane);
        const First f = first(s, lane);
        stage(s, r, lane, mask, smem);
        return f;
    }
    // the corner at place i of the list, or of id far[j]
    __device__ __forceinline__ d3 pos(const SweepView& s, uint32_t i, const uint32_t* far, size_t j) const {
        if (FAR) return ld3(s.x, far[j]);
        if (i < kSlots) return mk(at[i], at[kSlots + i], at[2 * kSlots + i]);
        return ld3(s.x, s.vt.nb[nb0 + i]);
    }
};

// Partial sum of the incident terms dealt to `lane` of a group of G
// (VbdSolver::local, src/vbd.rs:196-248), with the vertex at p; f holds the
// lane's first records.
template <bool D, int G, bool HS = D, bool FAR, bool LEAN>
__device__ __forceinline__ double local_part(const SweepView& s, const Near<G, FAR, LEAN>& T,
                                             typename Near<G, FAR, LEAN>::First f, d3 p, uint32_t lane, d3& g,
                                             Sym& H) {
    constexpr uint32_t kId = (1u << 21) - 1u;
    double e = 0.0;
    for (uint32_t i = lane; i < T.nt; i += G) {
        if (LEAN) T.tri(s, i, f);
        const unsigned long long t = f.t;
        const double4 b = f.tb, k = f.tk;
        if (!LEAN) T.tri(s, i + G, f);
        const size_t far = 3 * (size_t)(T.t0 + i);
        e += membrane<D, HS>(s, b, k, FAR ? s.vt.far_tri[far + 2] : (uint32_t)(t >> 42),
                             T.pos(s, (uint32_t)t & kId, s.vt.far_tri, far) - p,
                             T.pos(s, (uint32_t)(t >> 21) & kId, s.vt.far_tri, far + 1) - p, g, H);
    }
    // edge ends, then wings: the lanes of a round take the same form
    for (uint32_t i = lane; i < T.ne; i += G) {
        const ulonglong2 h = LEAN ? s.vt.hinge[T.h0 + i] : f.edge;
        if (!LEAN && i + G < T.ne) f.edge = s.vt.hinge[T.h0 + i + G];
        const size_t far = 3 * (size_t)(T.h0 + i);
        e += bending_edge<D, HS>(__longlong_as_double((long long)h.y), T.pos(s, (uint32_t)h.x & kId, s.vt.far_hinge, far),
                                 T.pos(s, (uint32_t)(h.x >> 21) & kId, s.vt.far_hinge, far + 1),
                                 T.pos(s, (uint32_t)(h.x >> 42), s.vt.far_hinge, far + 2), p, g, H);
    }
    for (uint32_t i = lane; i < T.nw; i += G) {
        const ulonglong2 h = LEAN ? s.vt.hinge[T.h0 + T.ne + i] : f.wing;
        if (!LEAN && i + G < T.nw) f.wing = s.vt.hinge[T.h0 + T.ne + i + G];
        const size_t far = 3 * (size_t)(T.h0 + T.ne + i);
        e += bending_wing<D, HS>(__longlong_as_double((long long)h.y), T.pos(s, (uint32_t)h.x & kId, s.vt.far_hinge, far),
                                 T.pos(s, (uint32_t)(h.x >> 21) & kId, s.vt.far_hinge, far + 1),
                                 T.pos(s, (uint32_t)(h.x >> 42), s.vt.far_hinge, far + 2), p, g, H);
    }
    if (T.ns) {
        const uint32_t b1 = s.inc_off[T.v + 1];
        for (uint32_t k = b1 - T.ns + lane; k < b1; k += G)
            e += stitch_term<D>(s, s.inc[k] & 0x0fffffffu, T.v, p, g, H);
    }
    for (uint32_t k = T.c0 + lane; k < T.c1; k += G) {
        if (LEAN) T.contact(s, k, f);
        const uint4 c = f.c;
        const double eps = f.eps;
        if (!LEAN) T.contact(s, k + G, f);
        e += contact_rec<D, HS>(s, c, eps, p, g, H);
    }
    if (lane == 0 && s.grab.active && (s.grab.v[0] == T.v || s.grab.v[1] == T.v || s.grab.v[2] == T.v))
        e += grab_term<D>(s, T.v, p, g, H);
    return e;
}

template <int G>
__device__ __forceinline__ double group_sum(double x, unsigned mask) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) x += __shfl_xor_sync(mask, x, o, G);
    return x;
}

__device__ __forceinline__ d3 truncate_ball(const SweepView& s, uint32_t v, d3 proposed, bool& clipped) {  // world.rs:91-100
    d3 c = ld3(s.contacts.centers, v);
    d3 d = proposed - c;
    double l = len(d);
    double b = s.contacts.radii[v];
    if (l > b) {
        clipped = true;
        return c + d * (b / l);
    }
    clipped = false;
    return proposed;
}

}  // namespace cc
