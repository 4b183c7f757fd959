// ftb_kernels.cu -- sm_100a wavefront kernels of the forward pinhole light tracer.
//
// Up to W photon paths are in flight at once, traced with four kernels:
//   k_emit    seed the per-photon PCG32 stream, pick emitter / point / direction /
//             wavelength, book `emitted`, queue the emitter's direct camera connection
//             (reference: Renderer::tracePhoton emission, render.h:1827-1984)
//   k_extend  closest hit of every queued path over the 8-wide BVH (Scene::closestHit,
//             scene.h:2194-2242)
//   k_shade   media, interior absorption and the material interaction of one bounce;
//             queues camera connections and copies the surviving paths into the other
//             path buffer (render.h:2013-2238)
//   k_shadow  any-hit test of the queued connections (Scene::occluded, scene.h:2249) and
//             the splat into the 64-bit fixed-point film (Film::add, scene_film.h:12)
//
// Path state is compacted (a queue of n paths is entries 0..n-1 of structure-of-arrays
// buffers, no index lists) and two-ended (paths inside a dielectric grow from the top
// entry down, so each end holds paths of similar traversal cost).  The queue kernels hand
// out work to warps 32 entries at a time from a per-launch counter.  A streaming pass
// (launch_stream) refills the room freed by finished paths with the next photons every
// half-iteration and runs as one CUDA graph with a device-driven while loop; a wave
// (launch_wave) traces W photons to their last bounce.  Small passes and renders, and the last
// paths of larger passes, are traced to their ends by one launch (k_trace, k_trace_hero).
//
// Variants: k_emit_hero / k_shade_hero / k_shadow_hero trace hero-wavelength bundles (one
// path carries up to kHeroMax wavelengths), and the kernels are templated on whether the
// scenes have instances, participating media or spheres/curves, so a launch runs only the
// code its scenes need.  k_sort_queue and k_sort_connections order the rays of large scenes.
//
// Numerics.  Everything that decides a path -- triangle/sphere/curve tests, hit points,
// normals, BSDF sampling, Russian roulette, the camera projection -- is computed in fp64
// in the reference's operation order, and this file is compiled with -fmad=false so no
// product is fused.  Only the BVH culling runs in fp32, against boxes that were rounded
// outward (see bvh_build.cpp) and with the ray interval widened by 1.25 x 2^-20, so it never
// drops a primitive the fp64 test would accept.  Paths therefore follow the reference CPU
// tracer photon for photon; the remaining differences are last-bit ones from CUDA's
// exp/log/sin/cos/pow, and exact ties in t.
#include <cooperative_groups.h>
#include <algorithm>
#include <vector>
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <stdint.h>

#include "ftb_kernels.h"

namespace cg = cooperative_groups;

// Resident blocks per SM each kernel is compiled for (register budget 65536 / (128 x minB)),
// chosen by measurement on B200: latency hiding beats the spills the smaller budget costs.
#ifndef FTB_EMIT_MINB
#define FTB_EMIT_MINB 8
#endif
#ifndef FTB_TRAV_MINB
#define FTB_TRAV_MINB 8
#endif
#ifndef FTB_EXTEND_TRI_MINB    // closest hit of triangles only, 72 registers (glass 126.5 ms at 7
                               // blocks against 129.7 at 8 and at 6; curves 59.4 at 8, 61.1 at 7)
#define FTB_EXTEND_TRI_MINB 7
#endif
#ifndef FTB_SHADE_MINB
#define FTB_SHADE_MINB 8
#endif
#ifndef FTB_SHADE_HERO_MINB    // bundles: their wavelength arrays want the registers (Cornell 1.62 ms
                               // at 6 blocks, 1.77 at 8, 1.72 at 5)
#define FTB_SHADE_HERO_MINB 6
#endif
#ifndef FTB_TRACE_MINB         // whole paths: registers for traversal and shading at once
#define FTB_TRACE_MINB 4
#endif
#ifndef FTB_SHADE_MEDIA_MINB   // shading with participating media: more registers pay off (fog +
                               // strands 22.5 ms at 5 blocks, 23.6 at 4)
#define FTB_SHADE_MEDIA_MINB 5
#endif

namespace ftb {

#define PI_D 3.141592653589793
#define LAMBDA_MIN 360.0
#define LAMBDA_MAX 830.0
#define EPS_RAY 1e-6

// ------------------------------------------------------------------ vectors (fp64) -----
struct D3 { double x, y, z; };
__device__ __forceinline__ D3 mk(double x, double y, double z) { D3 r; r.x = x; r.y = y; r.z = z; return r; }
__device__ __forceinline__ D3 operator+(D3 a, D3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ D3 operator-(D3 a, D3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ D3 operator*(D3 a, double s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ D3 operator/(D3 a, double s) { return mk(a.x / s, a.y / s, a.z / s); }
__device__ __forceinline__ D3 neg(D3 a) { return mk(-a.x, -a.y, -a.z); }
__device__ __forceinline__ double dot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 cross(D3 a, D3 b) {
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double len(D3 a) { return sqrt(dot(a, a)); }
__device__ __forceinline__ D3 normalize(D3 a) { return a / len(a); }
__device__ __forceinline__ double comp(D3 a, int i) { return i == 0 ? a.x : (i == 1 ? a.y : a.z); }
__device__ __forceinline__ D3 ld3(const double* p) { return mk(p[0], p[1], p[2]); }
// reflect (linalg.h:82)
__device__ __forceinline__ D3 reflect(D3 d, D3 n) { return d - n * (2.0 * dot(d, n)); }
// onb (linalg.h:85-91)
__device__ __forceinline__ void onb(D3 n, D3& t, D3& b) {
    double sign = copysign(1.0, n.z);
    double a = -1.0 / (sign + n.z);
    double d = n.x * n.y * a;
    t = mk(1.0 + sign * n.x * n.x * a, sign * d, -sign * n.x);
    b = mk(d, sign + n.y * n.y * a, -n.y);
}

// ------------------------------------------------------------------ RNG (rng.h) --------
struct Pcg { uint64_t s, inc; };
__device__ __forceinline__ uint32_t pcg_next(Pcg& r) {
    uint64_t old = r.s;
    r.s = old * 6364136223846793005ULL + r.inc;
    uint32_t xs = (uint32_t)(((old >> 18u) ^ old) >> 27u);
    uint32_t rot = (uint32_t)(old >> 59u);
    return (xs >> rot) | (xs << ((~rot + 1u) & 31));
}
__device__ __forceinline__ double uniform(Pcg& r) { return (pcg_next(r) >> 8) * (1.0 / 16777216.0); }
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ULL;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
    return x ^ (x >> 31);
}
// seedUnit (rng.h:40) with the forward-tracer salt (main.cpp:11326)
__device__ __forceinline__ Pcg seed_photon(uint64_t k) {
    const uint64_t salt = 0x9E3779B97F4A7C15ULL;
    Pcg r;
    r.s = 0; r.inc = (mix64(k ^ salt) << 1u) | 1u;
    pcg_next(r);
    r.s += mix64(k + salt);
    pcg_next(r);
    return r;
}

// cosineHemisphere (rng.h:45-52)
__device__ D3 cosine_hemisphere(D3 n, Pcg& rng) {
    double u1 = uniform(rng), u2 = uniform(rng);
    double r = sqrt(u1);
    double phi = 6.283185307179586 * u2;
    double lx = r * cos(phi), ly = r * sin(phi), lz = sqrt(1.0 - u1);
    D3 t, b; onb(n, t, b);
    return normalize(t * lx + b * ly + n * lz);
}
// glossyDirUV / sampleGlossy (render.h:46-64)
__device__ D3 sample_glossy(D3 mdir, double roughness, Pcg& rng) {
    double u1 = uniform(rng), u2 = uniform(rng);
    if (u1 >= 1.0) return mdir;
    double rr = roughness < 1e-3 ? 1e-3 : roughness;
    double e = 2.0 / (rr * rr) - 2.0; if (e < 0) e = 0;
    double cos_t = pow(u1, 1.0 / (e + 1.0));
    double s = 1.0 - cos_t * cos_t;
    double sin_t = sqrt(s > 0.0 ? s : 0.0);
    double phi = 2.0 * PI_D * u2;
    D3 t, b; onb(mdir, t, b);
    return normalize(t * (sin_t * cos(phi)) + b * (sin_t * sin(phi)) + mdir * cos_t);
}
// hgPhase / sampleHG (phase.h:18-40)
__device__ __forceinline__ double hg_phase(double cos_t, double g) {
    double d = 1.0 + g * g - 2.0 * g * cos_t;
    if (d < 1e-9) d = 1e-9;
    return (1.0 - g * g) / (4.0 * PI_D * d * sqrt(d));
}
__device__ D3 sample_hg(D3 wi, double g, Pcg& rng) {
    double u1 = uniform(rng), u2 = uniform(rng);
    double cos_t;
    if (fabs(g) < 1e-3) cos_t = 1.0 - 2.0 * u1;
    else {
        double sq = (1.0 - g * g) / (1.0 + g - 2.0 * g * u1);
        cos_t = (1.0 + g * g - sq * sq) / (2.0 * g);
    }
    double s = 1.0 - cos_t * cos_t;
    double sin_t = sqrt(s > 0.0 ? s : 0.0);
    double phi = 2.0 * PI_D * u2;
    D3 t, b; onb(wi, t, b);
    return normalize(t * (sin_t * cos(phi)) + b * (sin_t * sin(phi)) + wi * cos_t);
}

// ------------------------------------------------------------------ spectra ------------
__device__ double spec_eval(const DevScene& sc, int idx, double w) {
    const DevSpec& s = sc.spec[idx];
    switch (s.kind) {
    case FTB_SPEC_CONST: return s.p[0];
    case FTB_SPEC_TABLE: {   // tabulatedSpectrum (spectrum.h:264-281)
        const double* x = sc.tw + s.offset;
        const double* y = sc.tv + s.offset;
        int n = s.n;
        if (w <= x[0]) return y[0];
        if (w >= x[n - 1]) return y[n - 1];
        int lo = 0, hi = n - 1;
        while (lo + 1 < hi) { int mid = (lo + hi) / 2; if (x[mid] <= w) lo = mid; else hi = mid; }
        double w0 = x[lo], w1 = x[lo + 1], v0 = y[lo], v1 = y[lo + 1];
        double f = (w1 > w0) ? (w - w0) / (w1 - w0) : 0.0;
        return v0 + (v1 - v0) * f;
    }
    case FTB_SPEC_CAUCHY: { double um = w * 1e-3; return s.p[0] + s.p[1] / (um * um); }
    case FTB_SPEC_SELLMEIER: {
        double l2 = (w * 1e-3) * (w * 1e-3);
        double n2 = 1.0 + s.p[0] * l2 / (l2 - s.p[3]) + s.p[1] * l2 / (l2 - s.p[4]) +
                    s.p[2] * l2 / (l2 - s.p[5]);
        return sqrt(n2 > 1.0 ? n2 : 1.0);
    }
    default: return 0.0;
    }
}
__device__ __forceinline__ double spec_slot(const DevScene& sc, int s, double w, double dflt) {
    return s >= 0 ? spec_eval(sc, s, w) : dflt;
}
__device__ __forceinline__ double clamp01(double x) { return x < 0 ? 0 : (x > 1 ? 1 : x); }

// CIE 1931 multi-Gaussian fit (color.h:8-24)
__device__ __forceinline__ double gauss_piece(double x, double mu, double s1, double s2) {
    double t = (x - mu) * ((x < mu) ? s1 : s2);
    return exp(-0.5 * t * t);
}
__device__ __forceinline__ double cie_x(double w) {
    return 0.362 * gauss_piece(w, 442.0, 0.0624, 0.0374) + 1.056 * gauss_piece(w, 599.8, 0.0264, 0.0323) -
           0.065 * gauss_piece(w, 501.1, 0.0490, 0.0382);
}
__device__ __forceinline__ double cie_y(double w) {
    return 0.821 * gauss_piece(w, 568.8, 0.0213, 0.0247) + 0.286 * gauss_piece(w, 530.9, 0.0613, 0.0322);
}
__device__ __forceinline__ double cie_z(double w) {
    return 1.217 * gauss_piece(w, 437.0, 0.0845, 0.0278) + 0.681 * gauss_piece(w, 459.0, 0.0385, 0.0725);
}

// ------------------------------------------------------------------ exact prim tests ---
struct Shear { int kx, ky, kz; double sx, sy, sz; };
// makeTriShear (geometry.h:261-276)
__device__ __forceinline__ Shear make_shear(D3 d) {
    Shear s;
    double ax = fabs(d.x), ay = fabs(d.y), az = fabs(d.z);
    if (ax >= ay && ax >= az) s.kz = 0; else if (ay >= az) s.kz = 1; else s.kz = 2;
    s.kx = s.kz + 1; if (s.kx == 3) s.kx = 0;
    s.ky = s.kx + 1; if (s.ky == 3) s.ky = 0;
    if (comp(d, s.kz) < 0.0) { int t = s.kx; s.kx = s.ky; s.ky = t; }
    s.sx = comp(d, s.kx) / comp(d, s.kz);
    s.sy = comp(d, s.ky) / comp(d, s.kz);
    s.sz = 1.0 / comp(d, s.kz);
    return s;
}
// The reference recomputes an exactly-zero edge function in long double (x87, 64-bit
// mantissa).  The device has no extended type: a*b - c*d is formed from exact products
// (two FMA residuals), which has the same sign whenever the extended-precision result is
// nonzero.  Reached only when a ray meets an edge line exactly.
__device__ __forceinline__ double zero_fallback(double a, double b, double c, double d) {
    double ph = a * b, qh = c * d;
    double pl = fma(a, b, -ph), ql = fma(c, d, -qh);
    return (ph - qh) + (pl - ql);
}
struct TriHitW { double u, v, w, inv_det; };
// A row of a record: one coordinate of the three vertices, and the record's tail.
struct RecRow { double a, b, c; uint32_t prim, info; };
// intersectTri acceptance (geometry.h:280-324) on the vertex rows of the ray's axes kx, ky, kz
// and the origin's components ox, oy, oz on those axes; returns t or rejects.
__device__ __forceinline__ bool tri_test(double sx, double sy, double sz, double ox, double oy, double oz,
                                         const RecRow& X, const RecRow& Y, const RecRow& Z, double tmin, double tbest,
                                         double& t_out, TriHitW* bw) {
    const double Akz = Z.a - oz, Bkz = Z.b - oz, Ckz = Z.c - oz;
    const double Ax = (X.a - ox) - sx * Akz, Ay = (Y.a - oy) - sy * Akz;
    const double Bx = (X.b - ox) - sx * Bkz, By = (Y.b - oy) - sy * Bkz;
    const double Cx = (X.c - ox) - sx * Ckz, Cy = (Y.c - oy) - sy * Ckz;
    double U = Cx * By - Cy * Bx;
    double V = Ax * Cy - Ay * Cx;
    double W = Bx * Ay - By * Ax;
    if (U == 0.0 || V == 0.0 || W == 0.0) {
        if (U == 0.0) U = zero_fallback(Cx, By, Cy, Bx);
        if (V == 0.0) V = zero_fallback(Ax, Cy, Ay, Cx);
        if (W == 0.0) W = zero_fallback(Bx, Ay, By, Ax);
    }
    if ((U < 0.0 || V < 0.0 || W < 0.0) && (U > 0.0 || V > 0.0 || W > 0.0)) return false;
    double det = U + V + W;
    if (det == 0.0) return false;
    double T = U * (sz * Akz) + V * (sz * Bkz) + W * (sz * Ckz);
    double inv_det = 1.0 / det;
    double t = T * inv_det;
    if (t < tmin || t >= tbest) return false;
    t_out = t;
    if (bw) { bw->u = U; bw->v = V; bw->w = W; bw->inv_det = inv_det; }
    return true;
}
// intersectSphere acceptance (geometry.h:377-387)
__device__ __forceinline__ bool sphere_test(D3 ro, D3 rd, const double* s, double tmin, double tbest,
                                            double& t_out) {
    D3 oc = ro - mk(s[0], s[1], s[2]);
    double r = s[3];
    double a = dot(rd, rd);
    double b = 2.0 * dot(oc, rd);
    double c = dot(oc, oc) - r * r;
    double disc = b * b - 4.0 * a * c;
    if (disc < 0.0) return false;
    double sq = sqrt(disc);
    double t = (-b - sq) / (2.0 * a);
    if (t < tmin) t = (-b + sq) / (2.0 * a);
    if (t < tmin || t >= tbest) return false;
    t_out = t;
    return true;
}
// makeCurveRay (curve.h:126-135)
struct CurveRay { D3 dn; double inv_len; };
__device__ __forceinline__ CurveRay make_curve_ray(D3 d) {
    CurveRay c; c.dn = mk(0, 0, 1); c.inv_len = 1.0;
    double l2 = dot(d, d);
    if (l2 > 0.0) { double l = sqrt(l2); c.inv_len = 1.0 / l; c.dn = d * c.inv_len; }
    return c;
}
struct CurveWin { double tn, y, shift; int piece; };
__device__ __forceinline__ void offer(CurveWin& a, double inv_len, double tmin, double tbest, double tn,
                                      int w, double y) {
    if (tn >= a.tn) return;
    double t = (tn + a.shift) * inv_len;
    if (t < tmin || t >= tbest) return;
    a.tn = tn; a.piece = w; a.y = y;
}
// curveSegCrossings<double> + intersectCurveSeg acceptance (curve.h:199-309)
__device__ bool curve_test(const CurveRay& cr, D3 ro, const double* s, double tmin, double tbest,
                           double& t_out, CurveWin* win) {
    D3 rd = cr.dn;
    D3 p0 = mk(s[0], s[1], s[2]), p1 = mk(s[3], s[4], s[5]);
    double r0 = s[6], r1 = s[7];
    CurveWin a; a.tn = DBL_MAX; a.y = 0.0; a.piece = -1;
    D3 ba = p1 - p0;
    double m0 = dot(ba, ba);
    if (!(m0 > 0.0)) return false;
    a.shift = dot(p0 - ro, rd);
    D3 o = mk(ro.x + rd.x * a.shift, ro.y + rd.y * a.shift, ro.z + rd.z * a.shift);
    D3 oa = o - p0, ob = o - p1;
    double rr = r0 - r1;
    double m1 = dot(ba, oa), m2 = dot(ba, rd), m3 = dot(rd, oa), m5 = dot(oa, oa);
    double m6 = dot(ob, rd), m7 = dot(ob, ob);
    double d2 = m0 - rr * rr;
    const double il = cr.inv_len;
    if (d2 > 0.0) {
        double k2 = d2 - m2 * m2;
        double k1 = d2 * m3 - m1 * m2 + m2 * rr * r0;
        double k0 = d2 * m5 - m1 * m1 + m1 * rr * r0 * 2.0 - m0 * r0 * r0;
        double h = k1 * k1 - k0 * k2;
        if (h >= 0.0 && k2 != 0.0) {
            double sq = sqrt(h);
            double ta = (-sq - k1) / k2, tb = (sq - k1) / k2;
            if (ta > tb) { double tmp = ta; ta = tb; tb = tmp; }
            double base = m1 - r0 * rr;
            double ya = base + ta * m2, yb = base + tb * m2;
            if (ya > 0.0 && ya < d2) offer(a, il, tmin, tbest, ta, 0, ya);
            if (yb > 0.0 && yb < d2) offer(a, il, tmin, tbest, tb, 0, yb);
        }
        double h1 = m3 * m3 - m5 + r0 * r0;
        if (h1 > 0.0) {
            double q = sqrt(h1), base = m1 - r0 * rr;
            double ta = -m3 - q, tb = -m3 + q;
            if (base + ta * m2 <= 0.0) offer(a, il, tmin, tbest, ta, 1, 0.0);
            if (base + tb * m2 <= 0.0) offer(a, il, tmin, tbest, tb, 1, 0.0);
        }
        double h2 = m6 * m6 - m7 + r1 * r1;
        if (h2 > 0.0) {
            double q = sqrt(h2), base = m1 - r0 * rr;
            double ta = -m6 - q, tb = -m6 + q;
            if (base + ta * m2 >= d2) offer(a, il, tmin, tbest, ta, 2, d2);
            if (base + tb * m2 >= d2) offer(a, il, tmin, tbest, tb, 2, d2);
        }
    } else {
        bool use_p0 = (r0 >= r1);
        double rc = use_p0 ? r0 : r1, mm = use_p0 ? m3 : m6, mq = use_p0 ? m5 : m7;
        double hh = mm * mm - mq + rc * rc;
        if (hh > 0.0) {
            double q = sqrt(hh);
            offer(a, il, tmin, tbest, -mm - q, use_p0 ? 1 : 2, use_p0 ? 0.0 : d2);
            offer(a, il, tmin, tbest, -mm + q, use_p0 ? 1 : 2, use_p0 ? 0.0 : d2);
        }
    }
    if (a.piece < 0) return false;
    t_out = (a.tn + a.shift) * il;
    if (win) *win = a;
    return true;
}

// A record's rows in natural order: d[3 * row + k].
struct Rec {
    double d[9];
    int32_t prim, info;
};
__device__ __forceinline__ int rec_type(uint32_t info) { return (info >> 24) & 3; }
__device__ __forceinline__ int rec_type(const Rec& r) { return rec_type((uint32_t)r.info); }
__device__ __forceinline__ int rec_mat(const Rec& r) { return r.info & 0xffffff; }
__device__ __forceinline__ bool rec_smooth(const Rec& r) { return (r.info >> 30) & 1; }

// Row `off` / 32 (a byte offset) of record i, in one 32-byte load.  Bound: a record test is
// instruction issue; loading the rows in the ray's axis order takes the place of the selects
// that permuted each vertex (36 of ~130 instructions) and of two of the five loads.  Closest
// hit of a frame against 80-byte vertex records (B200): Cornell 3.29 -> 2.88 ms, glass 135.7
// -> 130.0, fog + strands 66.4 -> 60.8; occlusion 2.85 -> 2.71, 32.3 -> 31.2, 30.4 -> 31.3
// (a curve reloads its rows in natural order there).
__device__ __forceinline__ RecRow ld_rec_row(const PrimRec* recs, int i, uint32_t off) {
    RecRow r;
    const char* p = reinterpret_cast<const char*>(recs + i) + off;
    double tail;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.a), "=d"(r.b), "=d"(r.c), "=d"(tail) : "l"(p));
    r.prim = (uint32_t)__double2loint(tail);
    r.info = (uint32_t)__double2hiint(tail);
    return r;
}
__device__ __forceinline__ void load_rec(const PrimRec* recs, int i, Rec& r) {
    const RecRow a = ld_rec_row(recs, i, 0), b = ld_rec_row(recs, i, 32), c = ld_rec_row(recs, i, 64);
    r.d[0] = a.a; r.d[1] = a.b; r.d[2] = a.c; r.d[3] = b.a; r.d[4] = b.b; r.d[5] = b.c;
    r.d[6] = c.a; r.d[7] = c.b; r.d[8] = c.c;
    r.prim = (int32_t)a.prim;
    r.info = (int32_t)a.info;
}

struct RayCtx {
    D3 o, d;
    Shear sh;
    CurveRay cr;
};
// A ray as the triangle test reads it: the shear, the origin's components on the axes kx, ky,
// kz, and the byte offsets of those axes' rows in a record.
struct TriRay {
    double sx, sy, sz, ox, oy, oz;
    uint32_t rx, ry, rz;
};
__device__ __forceinline__ TriRay tri_ray(const Shear& sh, D3 o) {
    TriRay r;
    r.sx = sh.sx; r.sy = sh.sy; r.sz = sh.sz;
    r.ox = comp(o, sh.kx); r.oy = comp(o, sh.ky); r.oz = comp(o, sh.kz);
    r.rx = 32u * sh.kx; r.ry = 32u * sh.ky; r.rz = 32u * sh.kz;
    return r;
}
// Test of record i of a kind that is not a triangle.
__device__ __forceinline__ bool shape_test(const RayCtx& R, const PrimRec* recs, int i, double tmin, double tbest,
                                           double& t) {
    Rec r;
    load_rec(recs, i, r);
    if (rec_type(r) == REC_SPHERE) return sphere_test(R.o, R.d, r.d, tmin, tbest, t);
    return curve_test(R.cr, R.o, r.d, tmin, tbest, t, nullptr);
}

// Hit attributes of the winning record (geometry.h:325-368, :388-396, curve.h:310-335)
struct Hit {
    double t;
    D3 p, n, ng;
    int mat, prim;
};
template <bool SHAPES>
__device__ void hit_attributes(const double* __restrict__ tri_n, const RayCtx& R, const PrimRec* recs, int i,
                               const Rec& r, Hit& h) {
    int ty = SHAPES ? rec_type(r) : REC_TRI;
    h.mat = rec_mat(r);
    h.prim = r.prim;
    double t = 0.0;
    if (ty == REC_TRI) {
        TriHitW w;
        const TriRay T = tri_ray(R.sh, R.o);
        tri_test(T.sx, T.sy, T.sz, T.ox, T.oy, T.oz, ld_rec_row(recs, i, T.rx), ld_rec_row(recs, i, T.ry),
                 ld_rec_row(recs, i, T.rz), EPS_RAY, DBL_MAX, t, &w);
        double b0 = w.u * w.inv_det, b1 = w.v * w.inv_det, b2 = w.w * w.inv_det;
        D3 v0 = mk(r.d[0], r.d[3], r.d[6]), v1 = mk(r.d[1], r.d[4], r.d[7]), v2 = mk(r.d[2], r.d[5], r.d[8]);
        D3 tgn = normalize(cross(v1 - v0, v2 - v0));     // Tri::finalize (geometry.h:52)
        D3 n0 = tgn, n1 = tgn, n2 = tgn;
        if (rec_smooth(r)) {
            const double* nn = tri_n + 9 * (size_t)r.prim;
            D3 a = ld3(nn), b = ld3(nn + 3), c = ld3(nn + 6);
            if (!(dot(a, a) < 1e-12)) n0 = a;
            if (!(dot(b, b) < 1e-12)) n1 = b;
            if (!(dot(c, c) < 1e-12)) n2 = c;
        }
        h.t = t;
        h.p = R.o + R.d * t;
        D3 ns = n0 * b0 + n1 * b1 + n2 * b2;
        double nl = dot(ns, ns);
        ns = (nl > 1e-18) ? ns * (1.0 / sqrt(nl)) : tgn;
        D3 gn = (dot(tgn, ns) < 0.0) ? neg(tgn) : tgn;
        bool flipped = !(dot(R.d, gn) < 0.0);
        h.ng = gn;
        h.n = flipped ? neg(ns) : ns;
    } else if (ty == REC_SPHERE) {
        sphere_test(R.o, R.d, r.d, EPS_RAY, DBL_MAX, t);
        h.t = t;
        h.p = R.o + R.d * t;
        D3 ng = normalize(h.p - mk(r.d[0], r.d[1], r.d[2]));
        h.ng = ng;
        h.n = (!(dot(R.d, ng) < 0.0)) ? neg(ng) : ng;
    } else {
        CurveWin win;
        curve_test(R.cr, R.o, r.d, EPS_RAY, DBL_MAX, t, &win);
        h.t = t;
        D3 rd = R.cr.dn;
        D3 p0 = mk(r.d[0], r.d[1], r.d[2]), p1 = mk(r.d[3], r.d[4], r.d[5]);
        D3 ba = p1 - p0;
        double rr = r.d[6] - r.d[7];
        double d2 = dot(ba, ba) - rr * rr;
        D3 ro = R.o + rd * win.shift;
        D3 oa = ro - p0, ob = ro - p1;
        h.p = R.o + R.d * t;
        D3 ng;
        if (win.piece == 0) ng = (oa + rd * win.tn) * d2 - ba * win.y;
        else if (win.piece == 1) ng = oa + rd * win.tn;
        else ng = ob + rd * win.tn;
        double nl = sqrt(dot(ng, ng));
        ng = (nl > 1e-18) ? ng * (1.0 / nl) : normalize(ba);
        h.ng = ng;
        h.n = (dot(R.d, ng) < 0.0) ? ng : neg(ng);
    }
}

// ------------------------------------------------------------------ traversal (fp32) ---
// Culling is conservative by construction.  Child planes are floats that enclose the child's
// box grown by 2^-18 x the scene's largest coordinate M (the builders check each against the
// exact box), and a plane x is entered at t = fma(x, ix, cx) with ix = 1/d and cx = -o*ix
// rounded to float.  The rounding of o, of cx and of the fma move t by at most ~2^-23 M |ix|
// (far inside the box growth, 2^-18 M |ix|); the rounding of d, of 1/d and of the fma's result
// (2^-24 each) scale t by less than 1 +- 2^-22 on either side of the interval, inside its
// widening by 1.25 x 2^-20 (T_WIDE).  So no ray culls a child whose primitives the exact fp64
// test would hit.
struct RayF {
    float ix, iy, iz;
    float cx, cy, cz;       // -o * ix per axis
    uint32_t nx, ny, nz;    // byte offset in a node of the axis' near planes
};
// Rows of planes in a node: lo x, y, z at 32, 64, 96 and hi x, y, z at 128, 160, 192, so an
// axis' near and far offsets add up to kRowSum + 64 * axis.
constexpr uint32_t kRowLo = 32, kRowSide = 96, kRowSum = 2 * kRowLo + kRowSide;
// 1 / x of a normal x with a normal 1 / x: the approximate reciprocal (1 ulp) and one step of
// Newton's iteration for the root of 1 / r - x.  Compared on a B200 with the correctly rounded
// reciprocal over every mantissa at the exponents -66 .. 3: equal in all of them (the
// approximation alone in 87 %).  The rounded reciprocal itself branches for subnormals, which
// a ray's direction (make_rayf) never is: renders bound by one path's latency take 1.5 % longer
// with it (preview of 2^16 photons 0.257 against 0.254 ms), small ones with planar mirrors 4 %.
__device__ __forceinline__ float reciprocal(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return __fmaf_rn(r, __fmaf_rn(-x, r, 1.0f), r);
}
__device__ __forceinline__ RayF make_rayf(D3 o, D3 d) {
    RayF r;
    float dx = (float)d.x, dy = (float)d.y, dz = (float)d.z;
    // a zero component is replaced by +-1e-20: the ray moves by at most 1e-20*t, far below
    // the box margin, and the reciprocals stay finite (no inf*0 NaNs in the slab test)
    dx = fabsf(dx) > 1e-20f ? dx : copysignf(1e-20f, dx);
    dy = fabsf(dy) > 1e-20f ? dy : copysignf(1e-20f, dy);
    dz = fabsf(dz) > 1e-20f ? dz : copysignf(1e-20f, dz);
    r.ix = reciprocal(dx); r.iy = reciprocal(dy); r.iz = reciprocal(dz);
    r.cx = -(float)o.x * r.ix; r.cy = -(float)o.y * r.iy; r.cz = -(float)o.z * r.iz;
    r.nx = kRowLo + (dx < 0.0f ? kRowSide : 0u);   // near is the hi side where d is negative
    r.ny = kRowLo + 32 + (dy < 0.0f ? kRowSide : 0u);
    r.nz = kRowLo + 64 + (dz < 0.0f ? kRowSide : 0u);
    return r;
}

#define T_WIDE (1.0f + 1.1920928955078125e-6f)   // 1 + 1.25 * 2^-20
#define T_CULL (1.0f + 1.9073486328125e-6f)      // 1 + 2^-19: covers an entry key's slot bits (< 8 ulps)
                                                 // and the scale error of its distance

// Two floats in a register pair, and the packed arithmetic of sm_100 on them (each half is
// rounded like the scalar operation).
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2_dup(float x) {
    F2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float2 f2_get(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
struct Row { F2 p[4]; };   // eight planes
__device__ __forceinline__ Row ld_row(const char* p) {
    Row r;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(r.p[0]), "=l"(r.p[1]), "=l"(r.p[2]), "=l"(r.p[3]) : "l"(p));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }
__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }

// Entry distances of the eight children of node i as sort keys -- the float's bits with the
// child's slot in the low three, all ones for a child the ray misses -- and the node's
// header (child_base, prim_base, codes).
// Bound: instruction issue and the latency of the node loads.  A visit reads 208 of the node's
// bytes in seven loads and runs the 48 plane distances as 24 packed multiply-adds; the
// interval is widened on its far side only.  Against 16-byte loads, scalar multiply-adds and
// meta bytes decoded by shifts (B200, closest hit of a frame): glass, 2^27 photons, 146.5 ->
// 135.9 ms; fog + 250k strands, 2^25 photons, 71.7 -> 66.3 ms; occlusion 36.1 -> 33.7 and
// 33.7 -> 30.7 ms; 11 % fewer warp instructions per ray.
__device__ __forceinline__ void node_keys(const FNode* __restrict__ nodes, uint32_t i, const RayF& R,
                                          float tmin_f, float tmax_f, uint32_t (&k)[8], uint4& hdr) {
    const char* n = reinterpret_cast<const char*>(nodes + i);
    const Row ax = ld_row(n + R.nx), bx = ld_row(n + (kRowSum - R.nx));
    const Row ay = ld_row(n + R.ny), by = ld_row(n + (kRowSum + 64 - R.ny));
    const Row az = ld_row(n + R.nz), bz = ld_row(n + (kRowSum + 128 - R.nz));
    hdr = __ldg(reinterpret_cast<const uint4*>(n));
    const F2 ix = f2_dup(R.ix), iy = f2_dup(R.iy), iz = f2_dup(R.iz);
    const F2 cx = f2_dup(R.cx), cy = f2_dup(R.cy), cz = f2_dup(R.cz);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const float2 nx = f2_get(f2_fma(ax.p[h], ix, cx)), fx = f2_get(f2_fma(bx.p[h], ix, cx));
        const float2 ny = f2_get(f2_fma(ay.p[h], iy, cy)), fy = f2_get(f2_fma(by.p[h], iy, cy));
        const float2 nz = f2_get(f2_fma(az.p[h], iz, cz)), fz = f2_get(f2_fma(bz.p[h], iz, cz));
        const float a0 = fmaxf(max3(nx.x, ny.x, nz.x), tmin_f), b0 = fminf(min3(fx.x, fy.x, fz.x), tmax_f);
        const float a1 = fmaxf(max3(nx.y, ny.y, nz.y), tmin_f), b1 = fminf(min3(fx.y, fy.y, fz.y), tmax_f);
        const uint32_t k0 = (__float_as_uint(a0) & ~7u) | (uint32_t)(2 * h);
        const uint32_t k1 = (__float_as_uint(a1) & ~7u) | (uint32_t)(2 * h + 1);
        k[2 * h] = a0 <= b0 * T_WIDE ? k0 : 0xffffffffu;
        k[2 * h + 1] = a1 <= b1 * T_WIDE ? k1 : 0xffffffffu;
    }
}

struct TravCount { unsigned long long nodes, recs, exact; };


// Stack entry: a node index, or (bit 31) a leaf: first record << 2 | (count - 1).  A child's
// entry is its code byte added to the node's base for its kind.
#define LEAF_BIT 0x80000000u
__device__ __forceinline__ uint32_t child_entry(uint4 hdr, uint32_t slot) {
    const uint32_t c = __byte_perm(hdr.z, hdr.w, slot);
    return ((c & 0x80u) ? (LEAF_BIT | (hdr.y << 2)) : hdr.x) + (c & 0x7fu);
}

#define CSWAP(a, b) { uint32_t lo_ = min(a, b); b = max(a, b); a = lo_; }

// A traversal stack in local memory.  (Keeping the top entries in shared memory measured
// slower on B200: the L1 serves this stack well, and shared memory takes L1 capacity.)
template <class E>
struct LocalStack {
    E loc[FTB_STACK + FTB_WIDTH];   // a node's children are pushed before the depth is checked
    __device__ __forceinline__ void put(int i, E v) { loc[i] = v; }
    __device__ __forceinline__ E get(int i) const { return loc[i]; }
};

// Closest-hit walk of one wide BVH.  Children of a node are visited near to far (leaves and
// inner nodes alike, keys sorted by an 8-input network in registers); entries farther than
// the current hit are culled when popped.  The loop is "while-while": a lane steps through
// inner nodes until it holds a leaf, so the lanes of a warp run the expensive leaf tests
// together rather than interleaved with node steps.  leaf(first, count, tmax_f) tests a
// leaf's records and returns the (possibly lowered) fp32 bound on t.
template <bool COUNT, class Stack, class Leaf>
__device__ __forceinline__ float walk_closest(const FNode* __restrict__ nodes, const RayF& F, float tmin_f,
                                              float tmax_f, Stack& st, Leaf& leaf, int32_t* status, TravCount& cnt,
                                              uint32_t root = 0) {
    int sp = 0;
    uint32_t cur = root;
    bool live = true;
    while (live) {
        while (!(cur & LEAF_BIT)) {
            uint32_t k[8];
            uint4 hdr;
            node_keys(nodes, cur, F, tmin_f, tmax_f, k, hdr);
            if (COUNT) cnt.nodes++;
            CSWAP(k[0], k[2]); CSWAP(k[1], k[3]); CSWAP(k[4], k[6]); CSWAP(k[5], k[7]);
            CSWAP(k[0], k[4]); CSWAP(k[1], k[5]); CSWAP(k[2], k[6]); CSWAP(k[3], k[7]);
            CSWAP(k[0], k[1]); CSWAP(k[2], k[3]); CSWAP(k[4], k[5]); CSWAP(k[6], k[7]);
            CSWAP(k[2], k[4]); CSWAP(k[3], k[5]);
            CSWAP(k[1], k[4]); CSWAP(k[3], k[6]);
            CSWAP(k[1], k[2]); CSWAP(k[3], k[4]); CSWAP(k[5], k[6]);
#pragma unroll
            for (int i = 7; i >= 1; --i) {
                if (k[i] != 0xffffffffu) {
                    st.put(sp, make_uint2(child_entry(hdr, k[i] & 7u), k[i]));
                    ++sp;
                }
            }
            if (sp > FTB_STACK) { atomicOr(status, ST_STACK_OVERFLOW); return tmax_f; }
            if (k[0] != 0xffffffffu) {
                cur = child_entry(hdr, k[0] & 7u);
                continue;
            }
            bool found = false;
            while (sp > 0) {
                --sp;
                const uint2 v = st.get(sp);
                if (__uint_as_float(v.y) <= tmax_f * T_CULL) { cur = v.x; found = true; break; }
            }
            if (!found) { live = false; break; }
        }
        if (!live) break;
        tmax_f = leaf((int)((cur & ~LEAF_BIT) >> 2), (int)(cur & 3u) + 1, tmax_f);
        bool found = false;
        while (sp > 0) {
            --sp;
            const uint2 v = st.get(sp);
            if (__uint_as_float(v.y) <= tmax_f * T_CULL) { cur = v.x; found = true; break; }
        }
        if (!found) break;
    }
    return tmax_f;
}

// Any-hit walk: order does not change the answer, so children are taken in slot order,
// leaves first; leaf(first, count) returns true on a hit, which ends the walk.
template <bool COUNT, class Stack, class Leaf>
__device__ __forceinline__ bool walk_any(const FNode* __restrict__ nodes, const RayF& F, float tmin_f, float tmax_f,
                                         Stack& st, Leaf& leaf, int32_t* status, TravCount& cnt,
                                         uint32_t root = 0) {
    int sp = 0;
    uint32_t cur = root;
    bool live = true;
    while (live) {
        while (!(cur & LEAF_BIT)) {
            uint32_t k[8];
            uint4 hdr;
            node_keys(nodes, cur, F, tmin_f, tmax_f, k, hdr);
            if (COUNT) cnt.nodes++;
            uint32_t hit = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (k[i] != 0xffffffffu) hit |= 1u << i;
            // bit 7 of each code byte marks a leaf: gathered to one bit per slot
            const uint32_t l0 = (hdr.z >> 7) & 0x01010101u, l1 = (hdr.w >> 7) & 0x01010101u;
            const uint32_t leaves = ((l0 * 0x10204080u) >> 28) | (((l1 * 0x10204080u) >> 28) << 4);
            uint32_t order = (hit & leaves) | ((hit & ~leaves) << 8);
            bool have_next = false;
            uint32_t next = 0;
            while (order) {
                int b = __ffs(order) - 1;
                order &= order - 1;
                uint32_t e = child_entry(hdr, (uint32_t)b & 7u);
                if (!have_next) { next = e; have_next = true; continue; }
                st.put(sp++, e);
            }
            if (sp > FTB_STACK) { atomicOr(status, ST_STACK_OVERFLOW); return false; }
            if (have_next) { cur = next; continue; }
            if (sp == 0) { live = false; break; }
            cur = st.get(--sp);
        }
        if (!live) break;
        if (leaf((int)((cur & ~LEAF_BIT) >> 2), (int)(cur & 3u) + 1)) return true;
        if (sp == 0) break;
        cur = st.get(--sp);
    }
    return false;
}

// Affine::apply / applyDir (linalg.h:105-114) of a 12-double map (3x3 row-major, then t)
__device__ __forceinline__ D3 xf_point(const double* m, D3 p) {
    return mk(m[0] * p.x + m[1] * p.y + m[2] * p.z + m[9],
              m[3] * p.x + m[4] * p.y + m[5] * p.z + m[10],
              m[6] * p.x + m[7] * p.y + m[8] * p.z + m[11]);
}
__device__ __forceinline__ D3 xf_dir(const double* m, D3 v) {
    return mk(m[0] * v.x + m[1] * v.y + m[2] * v.z,
              m[3] * v.x + m[4] * v.y + m[5] * v.z,
              m[6] * v.x + m[7] * v.y + m[8] * v.z);
}
// Affine::applyNormal of toWorld (linalg.h:161-167): toWorld.inverse() is toLocal, read
// transposed.
__device__ __forceinline__ D3 xf_normal(const double* il, D3 n) {
    return mk(il[0] * n.x + il[3] * n.y + il[6] * n.z,
              il[1] * n.x + il[4] * n.y + il[7] * n.z,
              il[2] * n.x + il[5] * n.y + il[8] * n.z);
}
__device__ __forceinline__ int rec_inst(const Rec& r) { return (int)__double_as_longlong(r.d[0]); }

// The world ray mapped into an instance's local space (Scene::closestHit instance leaf,
// scene.h:2226-2228): local t equals world t, the direction is not renormalized.
struct LocalRay { D3 o, d; };
__device__ __forceinline__ LocalRay to_local(const DevInst& I, D3 o, D3 d) {
    LocalRay L;
    L.o = xf_point(I.xl, o);
    L.d = xf_dir(I.xl, d);
    return L;
}

// The next double above a positive t (DBL_MAX -> +inf): record tests given this bound accept
// t <= best, so that an exact tie can be settled by primitive index.
__device__ __forceinline__ double next_up(double t) { return __longlong_as_double(__double_as_longlong(t) + 1); }

// Exact ties in t go to the lower primitive index (world index first, then the index within
// the BLAS).  The reference takes the first tied primitive its own hierarchy happens to
// test; with the index rule a closest hit does not depend on the hierarchy at all, and the
// oracle applies the same rule.
struct BestHit { int prim, sub_prim; };

// Blas::intersectLocal (scene.h:1017-1026): nearest BLAS triangle with t <= best_t that wins
// against the current best (ties by index); updates best_t / tmax_f / bh and returns the BLAS
// record, or -1.  `inst_prim` is the instance's world primitive index.
template <bool COUNT>
__device__ __noinline__ int blas_closest(const DevInst& I, D3 wo, D3 wd, double tmin, double& best_t,
                                         float& tmax_f, int inst_prim, BestHit& bh, int32_t* status,
                                         TravCount& cnt) {
    const LocalRay L = to_local(I, wo, wd);
    const TriRay T = tri_ray(make_shear(L.d), L.o);
    const RayF F = make_rayf(L.o, L.d);
    const PrimRec* __restrict__ recs = I.recs;
    int best = -1;
    auto leaf = [&](int first, int count, float tm) -> float {
        for (int k = 0; k < count; ++k) {
            if (COUNT) { cnt.recs++; cnt.exact++; }
            const RecRow X = ld_rec_row(recs, first + k, T.rx), Y = ld_rec_row(recs, first + k, T.ry);
            const RecRow Z = ld_rec_row(recs, first + k, T.rz);
            double t;
            if (tri_test(T.sx, T.sy, T.sz, T.ox, T.oy, T.oz, X, Y, Z, tmin, next_up(best_t), t, nullptr) &&
                (t < best_t || inst_prim < bh.prim || (inst_prim == bh.prim && (int)X.prim < bh.sub_prim))) {
                best_t = t; best = first + k; tm = __double2float_ru(t);
                bh.prim = inst_prim; bh.sub_prim = (int)X.prim;
            }
        }
        return tm;
    };
    LocalStack<uint2> st;
    tmax_f = walk_closest<COUNT>(I.nodes, F, __double2float_rd(tmin), tmax_f, st, leaf, status, cnt);
    return best;
}

// Blas::occludedLocal (scene.h:1027-1033)
template <bool COUNT>
__device__ __noinline__ bool blas_any(const DevInst& I, D3 wo, D3 wd, double tmin, double seg, float tmax_f,
                                      int32_t* status, TravCount& cnt) {
    const LocalRay L = to_local(I, wo, wd);
    const TriRay T = tri_ray(make_shear(L.d), L.o);
    const RayF F = make_rayf(L.o, L.d);
    const PrimRec* __restrict__ recs = I.recs;
    auto leaf = [&](int first, int count) -> bool {
        for (int k = 0; k < count; ++k) {
            if (COUNT) { cnt.recs++; cnt.exact++; }
            const RecRow X = ld_rec_row(recs, first + k, T.rx), Y = ld_rec_row(recs, first + k, T.ry);
            const RecRow Z = ld_rec_row(recs, first + k, T.rz);
            double t;
            if (tri_test(T.sx, T.sy, T.sz, T.ox, T.oy, T.oz, X, Y, Z, tmin, seg, t, nullptr)) return true;
        }
        return false;
    };
    LocalStack<uint32_t> st;
    return walk_any<COUNT>(I.nodes, F, __double2float_rd(tmin), tmax_f, st, leaf, status, cnt);
}

// Closest hit (Scene::closestHit, scene.h:2194-2242): returns the world record (or -1) and
// t; for an instance record, *sub receives the BLAS record.  INST selects the variant that
// can meet instance records (scenes with instances); the plain variant has no such branch.
template <bool COUNT, bool INST, bool SHAPES>
__device__ int traverse_closest(const DevScene& sc, const RayCtx& R, double tmin, double& best_t, int* sub,
                                int32_t* status, TravCount& cnt) {
    const RayF F = make_rayf(R.o, R.d);
    const TriRay T = tri_ray(R.sh, R.o);
    best_t = DBL_MAX;
    int best = -1;
    BestHit bh{INT_MAX, INT_MAX};
    const PrimRec* __restrict__ recs = sc.recs;
    // t <= best_t from a record test; a tie goes to the lower index
    auto take = [&](bool hit, double t, int rec, int prim, float& tm) {
        if (hit && (t < best_t || prim < bh.prim)) {
            best_t = t; best = rec; tm = __double2float_ru(t);
            bh.prim = prim; bh.sub_prim = INT_MAX;
        }
    };
    auto leaf = [&](int first, int count, float tm) -> float {
        for (int k = 0; k < count; ++k) {
            if (COUNT) cnt.recs++;
            const RecRow X = ld_rec_row(recs, first + k, T.rx), Y = ld_rec_row(recs, first + k, T.ry);
            const RecRow Z = ld_rec_row(recs, first + k, T.rz);
            if (INST && rec_type(X.info) == REC_INST) {
                Rec r;
                load_rec(recs, first + k, r);
                int s = blas_closest<COUNT>(sc.inst[rec_inst(r)], R.o, R.d, tmin, best_t, tm, r.prim, bh, status, cnt);
                if (s >= 0) { best = first + k; *sub = s; }
                continue;
            }
            if (COUNT) cnt.exact++;
            double t;
            const bool hit = !SHAPES || rec_type(X.info) == REC_TRI
                                 ? tri_test(T.sx, T.sy, T.sz, T.ox, T.oy, T.oz, X, Y, Z, tmin, next_up(best_t), t, nullptr)
                                 : shape_test(R, recs, first + k, tmin, next_up(best_t), t);
            take(hit, t, first + k, (int)X.prim, tm);
        }
        return tm;
    };
    LocalStack<uint2> st;
    const float tm = walk_closest<COUNT>(sc.nodes, F, __double2float_rd(tmin), FLT_MAX, st, leaf, status, cnt);
    if (SHAPES && sc.root2 > 0) {   // the curves' hierarchy, under the bound the first walk left
        auto curves = [&](int first, int count, float tm2) -> float {
            for (int k = 0; k < count; ++k) {
                if (COUNT) { cnt.recs++; cnt.exact++; }
                Rec r;
                load_rec(recs, first + k, r);
                double t;
                const bool hit = curve_test(R.cr, R.o, r.d, tmin, next_up(best_t), t, nullptr);
                take(hit, t, first + k, r.prim, tm2);
            }
            return tm2;
        };
        walk_closest<COUNT>(sc.nodes, F, __double2float_rd(tmin), tm, st, curves, status, cnt, (uint32_t)sc.root2);
    }
    return best;
}

// Any hit with t in [tmin, seg) (Scene::occluded, scene.h:2249-2271).
template <bool COUNT, bool INST, bool SHAPES>
__device__ bool traverse_any(const DevScene& sc, const RayCtx& R, double tmin, double seg, int32_t* status,
                             TravCount& cnt) {
    const RayF F = make_rayf(R.o, R.d);
    const float tmin_f = __double2float_rd(tmin), tmax_f = __double2float_ru(seg);
    const TriRay T = tri_ray(R.sh, R.o);
    const PrimRec* __restrict__ recs = sc.recs;
    auto leaf = [&](int first, int count) -> bool {
        for (int k = 0; k < count; ++k) {
            if (COUNT) cnt.recs++;
            const RecRow X = ld_rec_row(recs, first + k, T.rx), Y = ld_rec_row(recs, first + k, T.ry);
            const RecRow Z = ld_rec_row(recs, first + k, T.rz);
            if (INST && rec_type(X.info) == REC_INST) {
                Rec r;
                load_rec(recs, first + k, r);
                if (blas_any<COUNT>(sc.inst[rec_inst(r)], R.o, R.d, tmin, seg, tmax_f, status, cnt)) return true;
                continue;
            }
            if (COUNT) cnt.exact++;
            double t;
            if (!SHAPES || rec_type(X.info) == REC_TRI) {
                if (tri_test(T.sx, T.sy, T.sz, T.ox, T.oy, T.oz, X, Y, Z, tmin, seg, t, nullptr)) return true;
            } else if (shape_test(R, recs, first + k, tmin, seg, t)) {
                return true;
            }
        }
        return false;
    };
    LocalStack<uint32_t> st;
    // a scene with two hierarchies keeps a top node over both in its last three nodes
    const uint32_t root = (SHAPES && sc.root2 > 0) ? (uint32_t)(sc.n_nodes - 3) : 0u;
    return walk_any<COUNT>(sc.nodes, F, tmin_f, tmax_f, st, leaf, status, cnt, root);
}

// Hit on BLAS record `sub` of instance I, in world terms: the local hit's attributes
// (intersectTri on the local ray) mapped like Scene::instanceHitToWorld (scene.h:2139-2162).
__device__ void instance_hit(const DevInst& I, int sub, D3 ro, D3 rd, Hit& h) {
    const LocalRay L = to_local(I, ro, rd);
    RayCtx R;
    R.o = L.o; R.d = L.d;
    R.sh = make_shear(L.d);
    Rec br;
    load_rec(I.recs, sub, br);
    hit_attributes<false>(I.tri_n, R, I.recs, sub, br, h);   // BLAS records are triangles
    h.p = ro + rd * h.t;                        // world t == local t
    D3 wn = normalize(xf_normal(I.xl, h.n));
    D3 wng = normalize(xf_normal(I.xl, h.ng));
    h.ng = wng;
    h.n = (dot(rd, wn) < 0.0) ? wn : neg(wn);
    if (I.mat_override >= 0) h.mat = I.mat_override;
}

__device__ __forceinline__ RayCtx make_ray(D3 o, D3 d) {
    RayCtx R;
    R.o = o; R.d = d;
    R.sh = make_shear(d);
    R.cr = make_curve_ray(d);
    return R;
}

// ------------------------------------------------------------------ media --------------
__device__ __forceinline__ double med_sigma_t(const DevScene& sc, const DevMed& m, double lam) {
    double v = spec_eval(sc, m.sa, lam) + spec_eval(sc, m.ss, lam);
    return v > 0.0 ? v : 0.0;
}
__device__ __forceinline__ double med_albedo(const DevScene& sc, const DevMed& m, double lam) {
    double s = spec_eval(sc, m.ss, lam); s = s > 0.0 ? s : 0.0;
    double a = spec_eval(sc, m.sa, lam);
    double t = s + (a > 0.0 ? a : 0.0);
    return t > 0.0 ? s / t : 0.0;
}
// Medium::clipToBounds (scene.h:655-685)
__device__ bool clip_to_bounds(const DevMed& m, D3 o, D3 d, double t0, double t1, double& ta, double& tb) {
    if (m.bound == FTB_BOUND_NONE) { ta = t0; tb = t1; return t1 > t0; }
    if (m.bound == FTB_BOUND_SPHERE) {
        D3 oc = o - ld3(m.center);
        double A = dot(d, d);
        double B = 2.0 * dot(oc, d);
        double C = dot(oc, oc) - m.radius * m.radius;
        double disc = B * B - 4.0 * A * C;
        if (disc <= 0.0 || A <= 0.0) return false;
        double sd = sqrt(disc);
        double s0 = (-B - sd) / (2.0 * A), s1 = (-B + sd) / (2.0 * A);
        double lo = t0 > s0 ? t0 : s0, hi = t1 < s1 ? t1 : s1;
        if (lo > hi) return false;
        ta = lo; tb = hi; return tb > ta;
    }
    double lo = t0, hi = t1;
    for (int a = 0; a < 3; ++a) {
        double oa = comp(o, a), da = comp(d, a);
        double mn = m.bmin[a], mx = m.bmax[a];
        if (fabs(da) < 1e-12) { if (oa < mn || oa > mx) return false; continue; }
        double inv = 1.0 / da;
        double s0 = (mn - oa) * inv, s1 = (mx - oa) * inv;
        if (s0 > s1) { double t = s0; s0 = s1; s1 = t; }
        lo = (lo < s0) ? s0 : lo;
        hi = (s1 < hi) ? s1 : hi;
        if (lo > hi) return false;
    }
    ta = lo; tb = hi; return tb > ta;
}
// sampleMediaCollision, homogeneous (render.h:377-398, 444-458)
__device__ bool sample_media_collision(const DevScene& sc, D3 o, D3 d, double dmax, double lam, Pcg& rng,
                                       double& thit, int& which) {
    double best = dmax; int w = -1;
    for (int i = 0; i < sc.n_med; ++i) {
        const DevMed& m = sc.med[i];
        double st = med_sigma_t(sc, m, lam);
        if (st <= 0.0) continue;
        double ta, tb;
        if (!clip_to_bounds(m, o, d, 0.0, dmax, ta, tb)) continue;
        double t = ta - log(1.0 - uniform(rng)) / st;
        if (t < tb && t < best) { best = t; w = i; }
    }
    if (w < 0) return false;
    thit = best; which = w; return true;
}
// mediaTransmittance, homogeneous (render.h:403-421, 461-469)
__device__ double media_transmittance(const DevScene& sc, D3 o, D3 d, double dist, double lam) {
    double tr = 1.0;
    for (int i = 0; i < sc.n_med; ++i) {
        const DevMed& m = sc.med[i];
        double st = med_sigma_t(sc, m, lam);
        double mt = 1.0;
        if (st > 0.0) {
            double ta, tb;
            if (clip_to_bounds(m, o, d, 0.0, dist, ta, tb)) mt = exp(-st * (tb - ta));
        }
        tr *= mt;
        if (tr <= 0.0) break;
    }
    return tr;
}

// ------------------------------------------------------------------ camera -------------
// Camera::project, rectilinear (camera.h:137-151)
__device__ __forceinline__ bool cam_project(const DevCam& c, D3 p, int& px, int& py, double& cos_cam,
                                            double& dist2) {
    D3 d = p - ld3(c.eye);
    double cz = dot(d, ld3(c.w));
    if (cz <= 1e-9) return false;
    double cx = dot(d, ld3(c.u)), cy = dot(d, ld3(c.v));
    double ix = (cx / cz) / c.thx - 0.0;
    double iy = (cy / cz) / c.thy;
    if (ix < -1 || ix >= 1 || iy < -1 || iy >= 1) return false;
    px = (int)((ix * 0.5 + 0.5) * c.rx);
    py = (int)((iy * 0.5 + 0.5) * c.ry);
    dist2 = dot(d, d);
    cos_cam = cz / sqrt(dist2);
    return true;
}
__device__ __forceinline__ double cam_pixel_solid_angle(const DevCam& c, double cos_cam) {
    return c.ppa * cos_cam * cos_cam * cos_cam;
}
// The connection p -> eye (connectGeom, render.h:499-520): unit direction, distance and, if
// the point projects into the image, its pixel and cosine.  Camera::project works on
// p - eye, the exact negative of eye - p, so its squared length and distance are those of the
// connection: one square root and four divisions fewer per connection than projecting afresh
// (shading, B200: Cornell 4.19 -> 4.00 ms, glass 51.0 -> 49.2, showroom 15.6 -> 15.2).
struct EyeRay { D3 to, dir; double dist2, dist; };
__device__ __forceinline__ EyeRay eye_ray(const DevCam& c, D3 p) {
    EyeRay e;
    e.to = ld3(c.eye) - p;
    e.dist2 = dot(e.to, e.to);
    e.dist = sqrt(e.dist2);
    e.dir = e.to / e.dist;
    return e;
}
__device__ __forceinline__ bool eye_project(const DevCam& c, const EyeRay& e, int& px, int& py, double& cos_cam) {
    const D3 d = neg(e.to);
    const double cz = dot(d, ld3(c.w));
    if (cz <= 1e-9) return false;
    const double cx = dot(d, ld3(c.u)), cy = dot(d, ld3(c.v));
    const double ix = (cx / cz) / c.thx - 0.0;
    const double iy = (cy / cz) / c.thy;
    if (ix < -1 || ix >= 1 || iy < -1 || iy >= 1) return false;
    px = (int)((ix * 0.5 + 0.5) * c.rx);
    py = (int)((iy * 0.5 + 0.5) * c.ry);
    cos_cam = cz / e.dist;
    return true;
}

// geometry.h:174-242
__device__ __forceinline__ D3 oriented_geo_n(const Hit& h) { return (dot(h.ng, h.n) >= 0.0) ? h.ng : neg(h.ng); }
__device__ __forceinline__ double shading_adjoint_corr(D3 wi, D3 wo, D3 ns, D3 ng) {
    double denom = fabs(dot(wi, ng)) * fabs(dot(wo, ns));
    if (denom <= 1e-8) return 1.0;
    double num = fabs(dot(wi, ns)) * fabs(dot(wo, ng));
    return num / denom;
}
__device__ __forceinline__ double shadow_terminator_g(D3 wi, D3 ns, D3 ng) {
    double cos_ng_ns = dot(ng, ns);
    if (cos_ng_ns >= 1.0 - 1e-7) return (dot(ng, wi) > 0.0) ? 1.0 : 0.0;
    double cos_ng_wi = dot(ng, wi);
    if (cos_ng_wi <= 0.0) return 0.0;
    double denom = dot(ns, wi) * cos_ng_ns;
    if (denom <= 1e-8) return 1.0;
    double g = cos_ng_wi / denom;
    if (g >= 1.0) return 1.0;
    return g * g * (1.0 - g) + g;
}

// ------------------------------------------------------------------ shadow queue -------
__device__ __forceinline__ int agg_inc(int32_t* ctr) {
    cg::coalesced_group g = cg::coalesced_threads();
    int base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(ctr, (int)g.size());
    return g.shfl(base, 0) + (int)g.thread_rank();
}

// A queue of paths is two-ended: paths outside every dielectric grow from entry 0 up
// (count q[0]), paths inside one -- or leaving a curve, among the strands -- grow from entry
// W-1 down (count q[1]), so each end holds paths of similar traversal cost (inside a closed
// mesh a ray crosses it; outside most rays meet a wall after a few nodes) and warps diverge
// less.  Queue position p < q[0] is entry
// p; position q[0] + k is entry W-1-k.
__device__ __forceinline__ int queue_len(const int32_t* q) { return q[0] + q[1]; }

// Dynamic work distribution over a queue: a warp takes the next 32 positions from a
// per-launch counter in Wave::counts whenever it is done, so warps that drew short paths
// take more and a launch ends with fewer idle SMs than a fixed grid-stride split.  Every
// lane of the warp calls warp_fetch; the loop ends for the whole warp at once.
__device__ __forceinline__ int warp_fetch(int32_t* ctr) {
    int base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(ctr, 32);
    return __shfl_sync(0xffffffffu, base, 0);
}
#define FTB_FOR_WARP_CHUNKS(var, n, ctr)                                                      \
    for (int var##_base = warp_fetch(ctr); var##_base < (n); var##_base = warp_fetch(ctr))   \
        if (const int var = var##_base + (int)(threadIdx.x & 31); var < (n))
__device__ __forceinline__ int queue_entry(const Wave& w, int front, int p) {
    return p < front ? p : w.W - 1 - (p - front);
}

// A place in the connection queue, or -1 when it is full.  A place that was not there is given
// back, so the count stays at most the queue plus one per lane in flight however many
// connections a whole-path launch makes, and never falls below the places taken.
__device__ __forceinline__ int queue_slot(const Wave& w) {
    const int i = agg_inc(&w.counts[kShadowCount]);
    if (i < w.S) return i;
    atomicSub(&w.counts[kShadowCount], 1);
    return -1;
}

// A one-wavelength connection: the film increments cieX/Y/Z(lambda) * contribution in the
// order Film::add forms them (scene_film.h:12), from the matching functions evaluated once
// per path at emission.  Returns false when the connection queue is full.
__device__ __forceinline__ bool queue_shadow(const Wave& w, int job, int view, D3 o, D3 d, double tmax, double val,
                                             const double* cie, int pix) {
    const int i = queue_slot(w);
    if (i < 0) return false;
    w.sox[i] = o.x; w.soy[i] = o.y; w.soz[i] = o.z;
    w.sdx[i] = d.x; w.sdy[i] = d.y; w.sdz[i] = d.z;
    w.smax[i] = tmax; w.spix[i] = pix;
    w.sxyz[i] = cie[0] * val; w.sxyz[w.S + i] = cie[1] * val; w.sxyz[2 * (size_t)w.S + i] = cie[2] * val;
    w.sjob[i] = job; w.sview[i] = view;
    return true;
}

// Where a kernel's connections go.  WaveQueue: the wave's connection queue, sized so that a
// launch cannot overfill it (else a status bit fails the render).  PathQueue: the same queue,
// but a path traced to its end in one launch may queue any number of connections, so one that
// finds the queue full is tested and splatted on the spot.
struct WaveQueue {
    const Wave& w;
};
template <bool INST, bool SHAPES>
struct PathQueue {
    const Wave& w;
};
template <bool INST, bool SHAPES>
__device__ __noinline__ void connect_now(const DevJob& J, const Frame& f, int view, D3 o, D3 d, double tmax, double X,
                                         double Y, double Z, int pix);
__device__ __forceinline__ void push_shadow(const WaveQueue& q, const DevJob&, const Frame& f, int job, int view, D3 o,
                                            D3 d, double tmax, double val, const double* cie, int pix) {
    if (!queue_shadow(q.w, job, view, o, d, tmax, val, cie, pix)) atomicOr(f.status, ST_QUEUE_OVERFLOW);
}
template <bool INST, bool SHAPES>
__device__ __forceinline__ void push_shadow(const PathQueue<INST, SHAPES>& q, const DevJob& J, const Frame& f, int job,
                                            int view, D3 o, D3 d, double tmax, double val, const double* cie, int pix) {
    if (!queue_shadow(q.w, job, view, o, d, tmax, val, cie, pix))
        connect_now<INST, SHAPES>(J, f, view, o, d, tmax, cie[0] * val, cie[1] * val, cie[2] * val, pix);
}

// The views a job's vertices connect to: its own camera, or every view of a multi-camera job.
__device__ __forceinline__ int view_count(const DevJob& J) { return J.n_views > 1 ? J.n_views : 1; }
__device__ __forceinline__ const DevCam& view_cam(const DevJob& J, int v) {
    return J.n_views > 1 ? J.views[v].cam : J.cam;
}
__device__ __forceinline__ int64_t* view_film(const DevJob& J, int v) {
    return J.n_views > 1 ? J.views[v].film : J.film;
}

// connectGeom + connect, model B (render.h:499-559); the occlusion test is deferred to
// k_shadow, the rest of the contribution is formed here in the reference's order.
template <bool MEDIA, class Q>
__device__ void connect_surface(const DevScene& sc, const DevJob& J, const Q& w, const Frame& f, int job,
                                D3 p, D3 n, D3 ng, D3 wi, double lam, const double* cie, double beta, double rho) {
    for (int v = 0; v < view_count(J); ++v) {
        const DevCam& cam = view_cam(J, v);
        const EyeRay er = eye_ray(cam, p);
        const D3 wdir = er.dir;
        const double dist = er.dist, dist2 = er.dist2;
        double cos_surf = dot(n, wdir);
        if (cos_surf <= 0) continue;
        double stg = shadow_terminator_g(wdir, n, ng);
        if (stg <= 0.0) continue;
        int px, py; double cos_cam;
        if (!eye_project(cam, er, px, py, cos_cam)) continue;
        double omega = cam_pixel_solid_angle(cam, cos_cam);
        double corr = shading_adjoint_corr(wi, wdir, n, ng);
        double denom = dist2 * omega;
        double fr = rho / PI_D;
        double contrib = beta * fr * cos_surf * corr / denom * stg;
        if (MEDIA && sc.n_med > 0) contrib *= media_transmittance(sc, p, wdir, dist, lam);
        push_shadow(w, J, f, job, v, p + ng * 1e-6, wdir, dist - 2e-6, contrib, cie, py * cam.rx + px);
    }
}
// connectVolume (render.h:584-600)
template <class Q>
__device__ void connect_volume(const DevScene& sc, const DevJob& J, const Q& w, const Frame& f, int job,
                               const DevMed& m, D3 p, D3 win, double lam, const double* cie, double beta) {
    for (int v = 0; v < view_count(J); ++v) {
        const DevCam& cam = view_cam(J, v);
        const EyeRay er = eye_ray(cam, p);
        const D3 wdir = er.dir;
        const double dist = er.dist, dist2 = er.dist2;
        int px, py; double cos_cam;
        if (!eye_project(cam, er, px, py, cos_cam)) continue;
        double ph = hg_phase(dot(win, wdir), m.g);
        double alb = med_albedo(sc, m, lam);
        double omega = cam_pixel_solid_angle(cam, cos_cam);
        double contrib = beta * alb * ph / (dist2 * omega);
        contrib *= media_transmittance(sc, p, wdir, dist, lam);
        push_shadow(w, J, f, job, v, p + wdir * 1e-6, wdir, dist - 2e-6, contrib, cie, py * cam.rx + px);
    }
}

// ------------------------------------------------------------------ planar mirrors -----
// A mirror connection in the shadow queue (marked by a negative pixel, ~pixel): vertex p,
// the direction wP toward the eye's mirror image and the distance dP to the mirror point in
// the origin / direction / max fields, view | plane << 16, the wavelength, the vertex factor
// beta * (weight * shape) and cieX/Y/Z(lambda) in place of the film increments -- the
// mirror's reflectance is known only once k_shadow has seen which mirror the eye meets.
__device__ __forceinline__ bool queue_mirror(const Wave& w, int job, int view, int plane, D3 p, D3 wP, double dP,
                                             double a, double lam, const double* cie, int pix) {
    const int i = queue_slot(w);
    if (i < 0) return false;
    w.sox[i] = p.x; w.soy[i] = p.y; w.soz[i] = p.z;
    w.sdx[i] = wP.x; w.sdy[i] = wP.y; w.sdz[i] = wP.z;
    w.smax[i] = dP; w.spix[i] = ~pix;
    w.sval[i] = a; w.slam[i] = lam;
    w.sxyz[i] = cie[0]; w.sxyz[w.S + i] = cie[1]; w.sxyz[2 * (size_t)w.S + i] = cie[2];
    w.sjob[i] = job; w.sview[i] = view | (plane << 16);
    return true;
}
template <bool INST, bool SHAPES>
__device__ __noinline__ void mirror_now(const DevJob& J, const Frame& f, int view, int plane, D3 p, D3 wP, double dP,
                                        double a, double lam, double X, double Y, double Z, int pix);
__device__ __forceinline__ void push_mirror(const WaveQueue& q, const DevJob&, const Frame& f, int job, int view,
                                            int plane, D3 p, D3 wP, double dP, double a, double lam, const double* cie,
                                            int pix) {
    if (!queue_mirror(q.w, job, view, plane, p, wP, dP, a, lam, cie, pix)) atomicOr(f.status, ST_QUEUE_OVERFLOW);
}
template <bool INST, bool SHAPES>
__device__ __forceinline__ void push_mirror(const PathQueue<INST, SHAPES>& q, const DevJob& J, const Frame& f, int job,
                                            int view, int plane, D3 p, D3 wP, double dP, double a, double lam,
                                            const double* cie, int pix) {
    if (!queue_mirror(q.w, job, view, plane, p, wP, dP, a, lam, cie, pix))
        mirror_now<INST, SHAPES>(J, f, view, plane, p, wP, dP, a, lam, cie[0], cie[1], cie[2], pix);
}

// connectSpecularPlane's geometry (render.h:1334-1366) for one plane and view: the vertex and
// the eye on the same side of the plane, the path unfolded through the eye's mirror image,
// the vertex factor (SpecVtx::shape, render.h:897-901), the mirror point inside the plane's
// box and in the image.  false when the connection is culled; else the direction wP to the
// mirrored eye, the distance dP to the mirror, `shape` and the pixel.  `volume`: a medium
// scatter with incoming direction nw and HG g; otherwise a surface with normal nw.
__device__ __forceinline__ bool mirror_geometry(const DevPlane& mp, const DevCam& cam, D3 p, bool volume, D3 nw,
                                                double g, D3& wP, double& dP, double& shape, int& pix) {
    const D3 pn = ld3(mp.n);
    const D3 eye = ld3(cam.eye);
    const double se = dot(pn, eye) - mp.d;
    const double sp = dot(pn, p) - mp.d;
    if (!(se * sp > 0.0)) return false;
    const D3 eye_m = eye - pn * (2.0 * se);
    wP = eye_m - p;
    const double D = len(wP);
    if (D < 1e-9) return false;
    wP = wP * (1.0 / D);
    if (volume) {
        shape = hg_phase(dot(nw, wP), g);
    } else {
        const double cs = dot(nw, wP);
        shape = cs <= 0.0 ? -1.0 : cs / PI_D;
    }
    if (shape < 0.0) return false;
    const double denom = dot(pn, wP);
    if (fabs(denom) < 1e-12) return false;
    dP = (mp.d - dot(pn, p)) / denom;
    if (dP <= 1e-7 || dP >= D - 1e-7) return false;
    const D3 R = p + wP * dP;
    if (R.x < mp.lo[0] || R.x > mp.hi[0] || R.y < mp.lo[1] || R.y > mp.hi[1] || R.z < mp.lo[2] || R.z > mp.hi[2])
        return false;
    int px, py; double cos_cam, dist2e;
    if (!cam_project(cam, R, px, py, cos_cam, dist2e)) return false;
    if (cam_pixel_solid_angle(cam, cos_cam) <= 0.0) return false;
    pix = py * cam.rx + px;
    return true;
}

// camSpecularSplatAll / camSpecularSplatVolumeAll (render.h:1515-1585) over the planar
// mirrors: a mirror record for k_shadow per plane and view that the geometry lets through.
// `weight`: the vertex's albedo.
template <class Q>
__device__ __noinline__ void connect_mirrors(const DevScene& sc, const DevJob& J, const Q& w, const Frame& f,
                                             int job, D3 p, bool volume, D3 nw, double g, double lam,
                                             const double* cie, double beta, double weight) {
    for (int k = 0; k < sc.n_planes; ++k) {
        for (int v = 0; v < view_count(J); ++v) {
            D3 wP; double dP, shape; int pix;
            if (!mirror_geometry(sc.planes[k], view_cam(J, v), p, volume, nw, g, wP, dP, shape, pix)) continue;
            push_mirror(w, J, f, job, v, k, p, wP, dP, beta * (weight * shape), lam, cie, pix);
        }
    }
}

// isPlanarMirrorMat (scene.h:356-360)
__device__ __forceinline__ bool planar_mirror(const DevMat& m) {
    return m.type == FTB_MAT_MIRROR || m.type == FTB_MAT_HALF_MIRROR ||
           (m.type == FTB_MAT_GLOSSY && m.roughness <= 0.0);
}

// ------------------------------------------------------------------ tallies ------------
__device__ __forceinline__ long long to_fixed(double v, double scale_inv, int32_t* status) {
    double s = v * scale_inv;
    if (!(fabs(s) < 4.611686018427388e18)) {   // 2^62
        atomicOr(status, ST_FILM_SATURATED);
        return 0;
    }
    return __double2ll_rn(s);
}

// Sum a per-thread value over the block and add it to a global tally once per block.
__device__ void block_tally(unsigned long long* dst, long long v) {
    __shared__ long long red[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        int nw = (blockDim.x + 31) >> 5;
        long long s = lane < nw ? red[lane] : 0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0 && s != 0) atomicAdd(dst, (unsigned long long)s);
    }
}

enum { T_EMIT = 0, T_ABS = 1, T_SENSOR = 2, T_ESC = 3, T_RES = 4 };

// Per-thread energy tallies.  A single-job launch reduces them over the block once at the
// end of the kernel.  In a multi-job launch a thread moves its sums into a per-block table
// in shared memory (one row of five per job of the table) whenever the job of the path it
// books changes -- often, in a streaming pass, where the paths of neighbouring jobs share
// the queues -- and the block adds the table's nonzero entries to the jobs' tallies once
// at the end, so the global atomics per launch do not grow with the job changes.  The table
// is dynamic shared memory of table_rows() rows: eight blocks' full tables take 82 KB of the
// SM's storage from the L1 that holds these kernels' spills (shading of a frame of one job with
// the full table / without one, B200: Cornell 4.67 / 4.34 ms, glass 54.7 / 52.4, Cornell
// bundles 1.92 / 1.82).
constexpr size_t kTallyRow = sizeof(unsigned long long) * 5;
struct TallyAcc {
    int job;
    bool multi;
    long long v[5];
};
__device__ __forceinline__ unsigned long long* tally_table() {
    extern __shared__ unsigned long long dyn_tally[];   // a row per job, launches of many jobs only
    return dyn_tally;
}
// Called by every thread of the block at the start of the kernel.
__device__ __forceinline__ void tally_init(TallyAcc& a, bool multi, int n_jobs) {
    a.job = 0;
    a.multi = multi;
#pragma unroll
    for (int k = 0; k < 5; ++k) a.v[k] = 0;
    if (multi) {
        unsigned long long* tab = tally_table();
        for (int e = threadIdx.x; e < n_jobs * 5; e += blockDim.x) tab[e] = 0ull;
        __syncthreads();
    }
}
__device__ __forceinline__ void tally_flush(TallyAcc& a) {
    unsigned long long* row = tally_table() + 5 * a.job;
#pragma unroll
    for (int k = 0; k < 5; ++k)
        if (a.v[k]) { atomicAdd(row + k, (unsigned long long)a.v[k]); a.v[k] = 0; }
}
__device__ __forceinline__ void tally_add(TallyAcc& a, const DevJob* jobs, bool multi, int job, int k,
                                          long long x) {
    if (multi && job != a.job) { tally_flush(a); a.job = job; }
    a.v[k] += x;
}
__device__ void block_tally(unsigned long long* dst, long long v);
// Called by every thread of the block at the end of the kernel.
__device__ __forceinline__ void tally_finish(TallyAcc& a, const DevJob* jobs, bool multi, int n_jobs = 1) {
    if (multi) {
        tally_flush(a);
        __syncthreads();
        const unsigned long long* tab = tally_table();
        for (int e = threadIdx.x; e < n_jobs * 5; e += blockDim.x)
            if (tab[e]) atomicAdd(jobs[e / 5].tally + e % 5, tab[e]);
        return;
    }
    unsigned long long* t = jobs[0].tally;
#pragma unroll
    for (int k = 0; k < 5; ++k) block_tally(t + k, a.v[k]);
}

__device__ __forceinline__ uint64_t fnv_i32(uint64_t h, int32_t v) {
    uint32_t u = (uint32_t)v;
#pragma unroll
    for (int i = 0; i < 4; ++i) { h ^= (u >> (8 * i)) & 0xffu; h *= 1099511628211ULL; }
    return h;
}

// Per-path instrumentation (parity tests only).
__device__ __forceinline__ void log_finish(const Wave& w, const PathState& ps, int i, int fate, double beta) {
    if (!w.logs) return;
    ftb_photon_log& L = w.logs[ps.pid[i] - (uint64_t)w.log_base];
    L.n_hits = ps.lnh[i];
    L.fate = fate;
    L.prim_hash = ps.lhash[i];
    L.beta = beta;
    for (int k = 0; k < 8; ++k) L.prims[k] = ps.lprims[k * w.W + i];
}
// The log of a photon that ends at emission (it never enters a queue).
__device__ __forceinline__ void log_emitted(const Wave& w, uint64_t photon, int fate, double beta) {
    if (!w.logs) return;
    ftb_photon_log& L = w.logs[photon - (uint64_t)w.log_base];
    L.n_hits = 0;
    L.fate = fate;
    L.prim_hash = 1469598103934665603ULL;
    L.beta = beta;
    for (int k = 0; k < 8; ++k) L.prims[k] = -2;
}
__device__ __forceinline__ void log_start(const Wave& w, const PathState& ps, int i, uint64_t photon) {
    if (!w.logs) return;
    ps.pid[i] = photon;
    ps.lhash[i] = 1469598103934665603ULL; ps.lnh[i] = 0;
    for (int q = 0; q < 8; ++q) ps.lprims[q * w.W + i] = -2;
}
// A hit joins the log of path i (in place), before shading decides its fate.
template <bool INST>
__device__ __forceinline__ void log_hit(const Wave& w, const PathState& ps, int i, const DevScene& sc, int rec) {
    if (!w.logs) return;
    const int nh = ps.lnh[i];
    Rec r;
    r.prim = -1; r.info = 0;
    if (rec >= 0) load_rec(sc.recs, rec, r);
    const int prim = r.prim;
    uint64_t hsh = fnv_i32(ps.lhash[i], prim);
    if (INST && rec >= 0 && rec_type(r) == REC_INST)   // and the BLAS triangle
        hsh = fnv_i32(hsh, (int32_t)ld_rec_row(sc.inst[rec_inst(r)].recs, w.hit_sub[i], 0).prim);
    ps.lhash[i] = hsh;
    if (nh < 8) ps.lprims[nh * w.W + i] = prim;
    ps.lnh[i] = nh + 1;
}
// A surviving path's log moves with it.
__device__ __forceinline__ void log_move(const Wave& w, const PathState& in, int i, const PathState& out, int o) {
    if (!w.logs) return;
    out.pid[o] = in.pid[i];
    out.lhash[o] = in.lhash[i];
    out.lnh[o] = in.lnh[i];
    for (int q = 0; q < 8; ++q) out.lprims[q * w.W + o] = in.lprims[q * w.W + i];
}

// Photon sources of the emission kernels.  A wave emits photon photon0 + (t - g0) of the
// table range holding t, for t < params[1]; a streaming pass's refill emits stream indices
// next .. next+F-1, F = the free places (slots less the survivors already queued, at most the
// photons left), each mapped to its range's photon.
struct PhotonSource {
    int64_t n;           // photons this launch emits
    int64_t next;        // streaming: first stream index
    int32_t have;        // streaming: survivors already in the output queue
};
template <bool STREAM>
__device__ __forceinline__ PhotonSource photon_source(const Wave& w, const int32_t* out_count) {
    PhotonSource p;
    if (STREAM) {
        const int64_t total = reinterpret_cast<const int64_t*>(w.params)[1];
        p.next = w.ctl->next;
        p.have = out_count[0];   // the refill appends through ctl->taken, so this stays put
        const int64_t room = (int64_t)w.params[1] - p.have - out_count[1], left = total - p.next;
        p.n = left < room ? left : room;
    } else {
        p.n = w.params[1];
        p.next = 0;
        p.have = 0;
    }
    return p;
}
// Job and photon index of the t-th photon of this launch.
template <bool STREAM>
__device__ __forceinline__ int photon_job(const DevJob* __restrict__ jobs, int n_jobs, const PhotonSource& p,
                                          int64_t t, uint64_t& photon) {
    int j = 0;
    if (STREAM) {
        const int64_t g = p.next + t;
        if (n_jobs > 1) {
            int lo = 0, hi = n_jobs - 1;
            while (lo < hi) { int mid = (lo + hi + 1) / 2; if (jobs[mid].g0 <= g) lo = mid; else hi = mid - 1; }
            j = lo;
        }
        photon = jobs[j].photon0 + (uint64_t)(g - jobs[j].g0);
    } else {
        const int slot = (int)t;
        if (n_jobs > 1) {
            int lo = 0, hi = n_jobs - 1;
            while (lo < hi) { int mid = (lo + hi + 1) / 2; if (jobs[mid].g0 <= slot) lo = mid; else hi = mid - 1; }
            j = lo;
        }
        photon = jobs[j].photon0 + (uint64_t)(slot - jobs[j].g0);
    }
    return j;
}
// Queue position of a photon that survives emission, with its job, bounce count and log set.
template <bool STREAM>
__device__ __forceinline__ int photon_enqueue(const Wave& w, const PathState& out, int32_t* out_count,
                                              const PhotonSource& p, int j, bool multi, uint64_t photon) {
    const int o = STREAM ? p.have + agg_inc(&w.ctl->taken) : agg_inc(out_count);
    out.nbounce[o] = 0;
    if (multi) out.job[o] = j;
    log_start(w, out, o, photon);
    return o;
}

// ------------------------------------------------------------------ emission -----------
// Scene::selectEmitter (scene.h:1851-1857): no draw with one emitter.
__device__ __forceinline__ int select_emitter(const DevScene& sc, Pcg& rng) {
    if (sc.n_emit <= 1) return 0;
    double u = uniform(rng);
    int lo = 0, hi = sc.n_emit - 1;
    while (lo < hi) { int mid = (lo + hi) / 2; if (sc.emit_cdf[mid] < u) lo = mid + 1; else hi = mid; }
    return lo;
}
// Emitter::samplePoint (scene.h:815-880) and the emission direction (render.h:1938-1941)
__device__ __forceinline__ void emit_sample(const DevEmit& em, Pcg& rng, D3& origin, D3& emit_n, D3& dir) {
    double u1 = uniform(rng), u2 = uniform(rng);
    if (em.shape == FTB_EMIT_SPHERE) {
        double z = 1.0 - 2.0 * u1;
        double s = 1.0 - z * z;
        double r = sqrt(s > 0.0 ? s : 0.0);
        double phi = 2.0 * PI_D * u2;
        D3 d = mk(r * cos(phi), r * sin(phi), z);
        emit_n = d;
        origin = ld3(em.origin) + d * em.radius;
    } else {
        origin = ld3(em.origin) + ld3(em.u) * u1 + ld3(em.v) * u2;
        emit_n = ld3(em.normal);
    }
    dir = em.collimated ? ld3(em.beam) : cosine_hemisphere(emit_n, rng);
}
// EmissionSampler::sampleAt (spectrum.h:374-383)
__device__ __forceinline__ double sample_at(const DevEmit& em, double u, double& pdf) {
    int lo = 0, hi = em.n;
    while (lo + 1 < hi) { int mid = (lo + hi) / 2; if (em.cdf[mid] <= u) lo = mid; else hi = mid; }
    double c0 = em.cdf[lo], c1 = em.cdf[lo + 1];
    double frac = (c1 > c0) ? (u - c0) / (c1 - c0) : 0.5;
    pdf = (c1 - c0) / em.step;
    return LAMBDA_MIN + (lo + frac) * em.step;
}

// FTB_LAMBDA_UNIFORM_380_780 (no counterpart in the reference): lambda uniform over
// [380, 780) nm from the variate u, and the weight pdf_SPD(lambda) / (1/400 nm) with the
// emitter's binned SPD pdf, so the photon's power times the weight is unbiased for the band.
__device__ __forceinline__ double sample_uniform_band(const DevEmit& em, double u, double& weight) {
    const double lam = 380.0 + 400.0 * u;
    int b = (int)((lam - LAMBDA_MIN) / em.step);
    if (b < 0) b = 0;
    if (b > em.n - 1) b = em.n - 1;
    weight = (em.cdf[b + 1] - em.cdf[b]) / em.step * 400.0;
    return lam;
}

// ------------------------------------------------------------------ kernels ------------
template <bool MEDIA, bool STREAM, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_EMIT_MINB) k_emit(Wave w, const DevJob* __restrict__ jobs, Frame f, PathState out,
                                              int32_t* out_count) {
    const int32_t n_jobs = w.params[0];
    const bool multi = n_jobs > 1;
    const PhotonSource src = photon_source<STREAM>(w, out_count);
    TallyAcc acc;
    tally_init(acc, multi, n_jobs);
    for (int64_t t = blockIdx.x * blockDim.x + threadIdx.x; t < src.n; t += gridDim.x * blockDim.x) {
        uint64_t k;
        const int j = photon_job<STREAM>(jobs, n_jobs, src, t, k);
        const DevJob& J = jobs[j];
        const DevScene& sc = J.sc;
        Pcg rng = seed_photon(k);
        if (sc.total_power <= 0.0 || sc.n_emit == 0) { log_emitted(w, k, 4, 0.0); continue; }
        const int ei = select_emitter(sc, rng);
        const DevEmit& em = sc.emit[ei];
        D3 origin, emit_n, dir;
        emit_sample(em, rng, origin, emit_n, dir);
        double pdf = 0.0, wl = 1.0;
        const double ul = uniform(rng);
        double lam;
        if (J.lambda_mode == FTB_LAMBDA_UNIFORM_380_780) {
            lam = sample_uniform_band(em, ul, wl);
            pdf = wl;
        } else {
            lam = sample_at(em, ul, pdf);
        }
        if (pdf <= 0) { log_emitted(w, k, 4, 0.0); continue; }
        double beta = (sc.n_emit == 1) ? em.power : sc.total_power;
        beta *= 1.0;
        if (J.lambda_mode == FTB_LAMBDA_UNIFORM_380_780) beta *= wl;
        tally_add(acc, jobs, multi, j, T_EMIT, to_fixed(beta, J.tally_scale_inv, f.status));
        const double cie[3] = {cie_x(lam), cie_y(lam), cie_z(lam)};
        connect_surface<MEDIA>(sc, J, WaveQueue{w}, f, j, origin, emit_n, emit_n, emit_n, lam, cie, beta, 1.0);
        if (MIRROR && sc.n_planes > 0) connect_mirrors(sc, J, WaveQueue{w}, f, j, origin, false, emit_n, 0.0, lam, cie, beta, 1.0);
        D3 ro = origin + dir * 1e-6;
        if (J.max_bounce <= 0) {
            tally_add(acc, jobs, multi, j, T_RES, to_fixed(beta, J.tally_scale_inv, f.status));
            log_emitted(w, k, 2, beta);
            continue;
        }
        const int o = photon_enqueue<STREAM>(w, out, out_count, src, j, multi, k);
        out.rng_s[o] = rng.s; out.rng_i[o] = rng.inc;
        out.ox[o] = ro.x; out.oy[o] = ro.y; out.oz[o] = ro.z;
        out.dx[o] = dir.x; out.dy[o] = dir.y; out.dz[o] = dir.z;
        out.lam[o] = lam; out.beta[o] = beta;
        out.cie[o] = cie[0]; out.cie[w.W + o] = cie[1]; out.cie[2 * (size_t)w.W + o] = cie[2];
        out.stk_n[o] = 0;
    }
    tally_finish(acc, jobs, multi, n_jobs);
}

__device__ void block_add3(unsigned long long* dst, unsigned long long a, unsigned long long b,
                           unsigned long long c) {
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
        c += __shfl_down_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0 && (a | b | c)) {
        atomicAdd(dst, a); atomicAdd(dst + 1, b); atomicAdd(dst + 2, c);
    }
}

__device__ void block_add1(unsigned long long* dst, unsigned long long a) {
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0 && a) atomicAdd(dst, a);
}


template <bool COUNT, bool INST, bool SHAPES>
__global__ void __launch_bounds__(128, INST || SHAPES ? FTB_TRAV_MINB : FTB_EXTEND_TRI_MINB) k_extend(Wave w, const DevJob* __restrict__ jobs,
                                                              PathState in, const int32_t* qcount,
                                                              const int32_t* __restrict__ order, Frame f) {
    const int32_t n_jobs = w.params[0];
    const int front = qcount[0], nq = queue_len(qcount);
    TravCount cnt{0, 0, 0};
    unsigned long long rays = 0;
    FTB_FOR_WARP_CHUNKS(q, nq, &w.counts[kFetchExtend]) {
        const int i = order ? order[q] : queue_entry(w, front, q);
        const DevScene& sc = jobs[n_jobs > 1 ? in.job[i] : 0].sc;
        RayCtx R = make_ray(mk(in.ox[i], in.oy[i], in.oz[i]), mk(in.dx[i], in.dy[i], in.dz[i]));
        double t;
        int sub = -1;
        int rec = traverse_closest<COUNT, INST, SHAPES>(sc, R, EPS_RAY, t, &sub, f.status, cnt);
        w.hit_t[i] = t;
        w.hit_rec[i] = rec;
        if (INST) w.hit_sub[i] = sub;
        if (COUNT) rays++;
    }
    if (COUNT) {
        block_add3(f.stats, rays, cnt.nodes, cnt.recs);
        block_add1(f.stats + 6, cnt.exact);
    }
}

// Reordering of a closest-hit queue or of the connections before traversal (large scenes, or
// when the tuning asks): the order of rays does not change any result.

// 8-bit Morton code of two 4-bit coordinates.
__device__ __forceinline__ uint32_t morton4(uint32_t u, uint32_t v) {
    u = (u | (u << 2)) & 0x33u; u = (u | (u << 1)) & 0x55u;
    v = (v | (v << 2)) & 0x33u; v = (v | (v << 1)) & 0x55u;
    return u | (v << 1);
}

__device__ __forceinline__ uint32_t direction_key(D3 d) {
    float x = (float)d.x, y = (float)d.y, z = (float)d.z;
    const float s = fabsf(x) + fabsf(y) + fabsf(z);
    x /= s; y /= s; z /= s;
    if (z < 0.0f) {   // fold the lower hemisphere onto the octahedron's outer triangles
        const float fx = (1.0f - fabsf(y)) * copysignf(1.0f, x);
        const float fy = (1.0f - fabsf(x)) * copysignf(1.0f, y);
        x = fx; y = fy;
    }
    uint32_t u = (uint32_t)min(15, max(0, (int)((x * 0.5f + 0.5f) * 16.0f)));
    uint32_t v = (uint32_t)min(15, max(0, (int)((y * 0.5f + 0.5f) * 16.0f)));
    return morton4(u, v);
}

// The order of positions 0 .. n-1 in which each piece of CHUNK of them is bucketed by key in
// [0, KEYS) (counting sort in shared memory, one piece per block at a time): order[q] =
// entry_of(p) for the q-th position p of its piece.
template <int CHUNK, int THREADS, int KEYS, class Key, class Entry>
__device__ __forceinline__ void bucket_pieces(int n, int32_t* order, const Key& key_of, const Entry& entry_of) {
    constexpr int kPer = CHUNK / THREADS, kSlice = KEYS / THREADS, kWarps = THREADS / 32;
    static_assert(CHUNK % THREADS == 0 && KEYS % THREADS == 0 && kWarps <= 32, "whole rows");
    __shared__ int32_t hist[KEYS];
    __shared__ int32_t warp_sum[kWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int base = blockIdx.x * CHUNK; base < n; base += gridDim.x * CHUNK) {
        for (int t = threadIdx.x; t < KEYS; t += THREADS) hist[t] = 0;
        __syncthreads();
        int key[kPer], off[kPer];
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const int p = base + r * THREADS + threadIdx.x;
            key[r] = p < n ? key_of(p) : -1;
            off[r] = p < n ? atomicAdd(&hist[key[r]], 1) : 0;
        }
        __syncthreads();
        // exclusive scan of the bucket counts: a slice per thread, then over threads and warps
        int slice[kSlice], run = 0;
#pragma unroll
        for (int k = 0; k < kSlice; ++k) { slice[k] = hist[threadIdx.x * kSlice + k]; run += slice[k]; }
        int incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sum[wid] = incl;
        __syncthreads();
        int acc = incl - run;
        for (int k = 0; k < wid; ++k) acc += warp_sum[k];
#pragma unroll
        for (int k = 0; k < kSlice; ++k) { hist[threadIdx.x * kSlice + k] = acc; acc += slice[k]; }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPer; ++r)
            if (key[r] >= 0) order[base + hist[key[r]] + off[r]] = entry_of(base + r * THREADS + threadIdx.x);
        __syncthreads();   // before the next piece reuses the histogram
    }
}

// Traversal order of a queue: order[q] is the entry of the path the closest-hit kernel's q-th
// lane takes.  Pieces of 8192 paths are bucketed by the cell of the ray's origin on a 4 x 4 x 4
// grid over the scene's root box, then by its direction on an 8 x 8 octahedral grid, so a
// warp's 32 lanes start near each other and head the same way.  Closest hit of a frame (B200),
// against pieces of 1024 by direction alone (16 x 16): glass 117.0 -> 112.5 ms, fog + strands
// 55.7 -> 51.9, animation batch 34.9 -> 33.2; a sort of the whole queue by 9 bits of cell and
// 8 of direction gains as much again in traversal and costs more than that.
constexpr int kRayChunk = 8192, kRayThreads = 512, kRayKeys = 4096;
__global__ void __launch_bounds__(kRayThreads) k_sort_queue(Wave w, const DevJob* __restrict__ jobs, PathState in,
                                                            const int32_t* qcount, int32_t* order) {
    __shared__ float grid[kWaveJobs][6];   // per job: the root box's low corner, cells per unit
    const int32_t n_jobs = w.params[0];
    for (int t = threadIdx.x; t < 3 * n_jobs; t += kRayThreads) {
        const int j = t / 3, a = t % 3;
        const FNode& root = jobs[j].sc.nodes[0];
        float lo = root.lo[a][0], hi = root.hi[a][0];
        for (int k = 1; k < FTB_WIDTH; ++k) { lo = fminf(lo, root.lo[a][k]); hi = fmaxf(hi, root.hi[a][k]); }
        const float ext = hi - lo;   // not positive in an empty scene
        grid[j][a] = lo;
        grid[j][3 + a] = ext > 0.0f && ext < FLT_MAX ? 4.0f / ext : 0.0f;
    }
    __syncthreads();
    const int front = qcount[0];
    bucket_pieces<kRayChunk, kRayThreads, kRayKeys>(
        queue_len(qcount), order,
        [&](int p) {
            const int i = queue_entry(w, front, p);
            const float* g = grid[n_jobs > 1 ? in.job[i] : 0];
            const int cx = min(3, max(0, (int)(((float)in.ox[i] - g[0]) * g[3])));
            const int cy = min(3, max(0, (int)(((float)in.oy[i] - g[1]) * g[4])));
            const int cz = min(3, max(0, (int)(((float)in.oz[i] - g[2]) * g[5])));
            const uint32_t d = direction_key(mk(in.dx[i], in.dy[i], in.dz[i]));
            return ((cx | (cy << 2) | (cz << 4)) << 6) | (int)(d >> 2);
        },
        [&](int p) { return queue_entry(w, front, p); });
}

// Traversal order of the queued connections: all of a view's rays end at its eye, so those of
// one tile of the image (a 16 x 16 grid in Morton order) cross the same nodes.  Where it runs:
// ray_order.  Whole frames (B200), beside ordered closest-hit rays: fog + strands 107.4 ->
// 100.2 ms, glass 200.8 -> 197.8, animation batch 65.8 -> 64.3, served jobs 79.7 -> 75.9;
// Cornell, where it does not run, would take 0.4 ms more.  The launches themselves, order
// included and nothing beside them: strands 14 % shorter, triangles 3 to 7 % longer with one
// view and 5 to 9 % with four, whose rays end at four eyes and share tiles; with the
// closest-hit launch beside them their frames are shorter all the same.  Pieces of 4096 gain
// 1 ms more on the strands and lose 1.2 on glass.
constexpr int kConnChunk = 1024, kConnThreads = 128, kConnKeys = 256;
__global__ void __launch_bounds__(kConnThreads) k_sort_connections(Wave w, const DevJob* __restrict__ jobs,
                                                                   int32_t* order) {
    const int32_t n_jobs = w.params[0];
    int n = w.counts[kShadowCount];
    if (n > w.S) n = w.S;
    bucket_pieces<kConnChunk, kConnThreads, kConnKeys>(
        n, order,
        [&](int p) {
            const DevCam& c = view_cam(jobs[n_jobs > 1 ? w.sjob[p] : 0], w.sview[p]);
            const int pix = w.spix[p];
            const int py = pix / c.rx, px = pix - py * c.rx;
            return (int)morton4((uint32_t)((int64_t)px * 16 / c.rx), (uint32_t)((int64_t)py * 16 / c.ry));
        },
        [&](int p) { return p; });
}

struct Stk { int n; int2 e[kStkCap]; };
__device__ __forceinline__ int stk_top_pri(const Stk& s) {
    int bp = INT_MIN;
    for (int i = 0; i < s.n; ++i) if (s.e[i].y > bp) bp = s.e[i].y;
    return s.n ? bp : INT_MIN;
}
__device__ __forceinline__ int stk_top_mat(const Stk& s) {
    int bp = INT_MIN, bm = -1;
    for (int i = 0; i < s.n; ++i) if (s.e[i].y >= bp) { bp = s.e[i].y; bm = s.e[i].x; }
    return bm;
}
__device__ __forceinline__ void stk_push(Stk& s, int mi, int p, int32_t* status) {
    if (s.n < kStkCap) { s.e[s.n] = make_int2(mi, p); ++s.n; }
    else atomicOr(status, ST_MEDIUM_STACK);
}
__device__ __forceinline__ void stk_pop_mat(Stk& s, int mi) {
    for (int i = s.n - 1; i >= 0; --i)
        if (s.e[i].x == mi) {
            for (int j = i; j < s.n - 1; ++j) s.e[j] = s.e[j + 1];
            --s.n; return;
        }
}

__device__ __forceinline__ double mat_ior(const DevScene& sc, const DevMat& m, double lam) {
    return m.ior >= 0 ? spec_eval(sc, m.ior, lam) : 1.5;
}

// refractOrReflect, stochastic branch (render.h:2657-2697)
__device__ void refract_or_reflect(const DevScene& sc, const DevMat& m, const Hit& h, D3 d, double lam,
                                   Pcg& rng, bool& transmitted, double ext_ior, D3& o_out, D3& d_out) {
    double ngi = mat_ior(sc, m, lam);
    bool entering = dot(d, h.ng) < 0.0;
    D3 nl = entering ? h.ng : neg(h.ng);
    double n1 = entering ? ext_ior : ngi;
    double n2 = entering ? ngi : ext_ior;
    double eta = n1 / n2;
    double cos_i = -dot(d, nl);
    double sin2t = eta * eta * (1.0 - cos_i * cos_i);
    D3 out;
    bool refracted = false;
    if (sin2t > 1.0) out = reflect(d, nl);
    else {
        double cos_t = sqrt(1.0 - sin2t);
        double rs = (n1 * cos_i - n2 * cos_t) / (n1 * cos_i + n2 * cos_t);
        double rp = (n1 * cos_t - n2 * cos_i) / (n1 * cos_t + n2 * cos_i);
        double R = 0.5 * (rs * rs + rp * rp);
        if (uniform(rng) < R) out = reflect(d, nl);
        else { out = d * eta + nl * (eta * cos_i - cos_t); refracted = true; }
    }
    out = normalize(out);
    if (m.roughness > 1e-3) {
        D3 pert = sample_glossy(out, m.roughness, rng);
        bool ok = refracted ? (dot(pert, nl) < 0.0) : (dot(pert, nl) > 0.0);
        if (ok) out = pert;
    }
    transmitted = refracted;
    o_out = h.p + out * 1e-6;
    d_out = out;
}

// One bounce of Renderer::tracePhoton's loop body (render.h:2013-2238): media, interior
// absorption and the interaction at the closest hit (record rec at distance ht, BLAS record
// sub), connections queued.  Returns -1 when the path goes on from (no, nd), 0 absorbed, 1
// escaped; `costly`: the next ray starts among curves.  cie() yields the path's CIE values.
template <bool MEDIA, bool INST, bool SHAPES, bool MIRROR, class Q, class Cie>
__device__ __forceinline__ int shade_bounce(const DevScene& sc, const DevJob& J, const Q& w, const Frame& f, int j,
                                            Pcg& rng, D3 ro, D3 rd, double lam, double& beta, Stk& stk, double ht,
                                            int rec, int sub, const Cie& cie, D3& no, D3& nd, bool& costly) {
    int fate = -1;
    bool valid = rec >= 0;
    double d_surf = valid ? ht : 1e30;
    double d_event = d_surf;
    bool medium_event = false;
    int scatter_med = -1;
    D3 mp = mk(0, 0, 0);
    if (MEDIA && sc.n_med > 0) {
        double tm; int which;
        if (sample_media_collision(sc, ro, rd, d_surf, lam, rng, tm, which)) {
            d_event = tm; medium_event = true; scatter_med = which; mp = ro + rd * tm;
        }
    }
    {   // Beer-Lambert inside the current dielectric (render.h:2063-2066)
        int mi = stk_top_mat(stk);
        double a = (mi >= 0) ? spec_slot(sc, sc.mats[mi].absorb, lam, 0.0) : 0.0;
        if (a > 0.0) beta *= exp(-a * d_event);
    }
    no = ro; nd = rd;
    if (medium_event) {   // render.h:2105-2115
        const DevMed& sm = sc.med[scatter_med];
        connect_volume(sc, J, w, f, j, sm, mp, rd, lam, cie(), beta);
        if (MIRROR && sc.n_planes > 0)
            connect_mirrors(sc, J, w, f, j, mp, true, rd, sm.g, lam, cie(), beta, med_albedo(sc, sm, lam));
        if (uniform(rng) >= med_albedo(sc, sm, lam)) fate = 0;
        else { nd = sample_hg(rd, sm.g, rng); no = mp; }
    } else if (!valid) {
        fate = 1;
    } else {
        Rec r;
        load_rec(sc.recs, rec, r);
        if (SHAPES && rec_type(r) == REC_CURVE) costly = true;
        Hit h;
        if (INST && rec_type(r) == REC_INST) {
            instance_hit(sc.inst[rec_inst(r)], sub, ro, rd, h);
            h.prim = r.prim;
        } else {
            RayCtx R = make_ray(ro, rd);
            hit_attributes<SHAPES>(sc.tri_n, R, sc.recs, rec, r, h);
        }
        const DevMat& m = sc.mats[h.mat];
        switch (m.type) {
        case FTB_MAT_DIELECTRIC: {   // render.h:1612-1660
            bool entering = dot(rd, h.ng) < 0.0;
            int mi = h.mat, pr = m.priority;
            bool has_pri = pr != INT_MIN;
            bool transmitted = false;
            if (entering) {
                int out_mat = stk_top_mat(stk), out_pri = stk_top_pri(stk);
                bool ranked = has_pri && (stk.n == 0 || (out_mat >= 0 && sc.mats[out_mat].priority != INT_MIN));
                if (ranked && stk.n != 0 && pr <= out_pri) {
                    stk_push(stk, mi, pr, f.status);
                    no = h.p + rd * 1e-6;
                } else {
                    double ext = (ranked && out_mat >= 0) ? mat_ior(sc, sc.mats[out_mat], lam) : 1.0;
                    refract_or_reflect(sc, m, h, rd, lam, rng, transmitted, ext, no, nd);
                    if (transmitted) stk_push(stk, mi, pr, f.status);
                }
            } else {
                Stk after = stk;
                stk_pop_mat(after, mi);
                int new_mat = stk_top_mat(after), new_pri = stk_top_pri(after);
                bool ranked = has_pri && (after.n == 0 || (new_mat >= 0 && sc.mats[new_mat].priority != INT_MIN));
                if (ranked && new_mat >= 0 && pr <= new_pri) {
                    stk_pop_mat(stk, mi);
                    no = h.p + rd * 1e-6;
                } else {
                    double ext = (ranked && new_mat >= 0) ? mat_ior(sc, sc.mats[new_mat], lam) : 1.0;
                    refract_or_reflect(sc, m, h, rd, lam, rng, transmitted, ext, no, nd);
                    if (transmitted) stk_pop_mat(stk, mi);
                }
            }
            break;
        }
        case FTB_MAT_GLOSSY: {   // render.h:1725-1733
            double rr = clamp01(spec_slot(sc, m.reflect, lam, 0.5));
            if (uniform(rng) >= rr) { fate = 0; break; }
            D3 o = sample_glossy(reflect(rd, h.n), m.roughness, rng);
            if (dot(o, h.n) <= 0) { fate = 0; break; }
            no = h.p + h.n * 1e-6; nd = o;
            break;
        }
        case FTB_MAT_MIRROR: {   // render.h:1680-1688
            double rr = clamp01(spec_slot(sc, m.reflect, lam, 0.5));
            if (uniform(rng) >= rr) { fate = 0; break; }
            nd = reflect(rd, h.n);
            no = h.p + h.n * 1e-6;
            break;
        }
        case FTB_MAT_HALF_MIRROR: {   // render.h:1702-1711
            double rr = clamp01(spec_slot(sc, m.reflect, lam, 0.5));
            if (uniform(rng) < rr) {
                nd = reflect(rd, h.n);
                no = h.p + h.n * 1e-6;
            } else {
                no = h.p + rd * 1e-6;
            }
            break;
        }
        case FTB_MAT_FILTER: {   // render.h:1711-1723
            double tt = clamp01(spec_slot(sc, m.transmit, lam, 0.0));
            if (uniform(rng) >= tt) { fate = 0; break; }
            no = h.p + rd * 1e-6;
            break;
        }
        case FTB_MAT_DIFFUSE_TRANSMIT: {   // render.h:2180-2212
            double rr = clamp01(spec_slot(sc, m.reflect, lam, 0.5));
            double rt = clamp01(spec_slot(sc, m.transmit, lam, 0.0));
            double sum = rr + rt;
            if (sum > 1.0) { rr /= sum; rt /= sum; sum = 1.0; }
            D3 ngo = oriented_geo_n(h);
            D3 wi = mk(-rd.x, -rd.y, -rd.z);
            connect_surface<MEDIA>(sc, J, w, f, j, h.p, h.n, ngo, wi, lam, cie(), beta, rr);
            connect_surface<MEDIA>(sc, J, w, f, j, h.p, neg(h.n), neg(ngo), wi, lam, cie(), beta, rt);
            if (MIRROR && sc.n_planes > 0) {
                connect_mirrors(sc, J, w, f, j, h.p, false, h.n, 0.0, lam, cie(), beta, rr);
                connect_mirrors(sc, J, w, f, j, h.p, false, neg(h.n), 0.0, lam, cie(), beta, rt);
            }
            double u = uniform(rng);
            if (u < rr) {
                D3 wo = cosine_hemisphere(h.n, rng);
                beta *= shading_adjoint_corr(wi, wo, h.n, ngo);
                no = h.p + h.n * 1e-6; nd = wo;
            } else if (u < sum) {
                D3 wo = cosine_hemisphere(mk(-h.n.x, -h.n.y, -h.n.z), rng);
                beta *= shading_adjoint_corr(wi, wo, h.n, ngo);
                no = h.p - h.n * 1e-6; nd = wo;
            } else fate = 0;
            break;
        }
        default: {   // Diffuse (render.h:2215-2236)
            double rho = clamp01(spec_slot(sc, m.reflect, lam, 0.5));
            D3 ngo = oriented_geo_n(h);
            D3 wi = mk(-rd.x, -rd.y, -rd.z);
            connect_surface<MEDIA>(sc, J, w, f, j, h.p, h.n, ngo, wi, lam, cie(), beta, rho);
            if (MIRROR && sc.n_planes > 0) connect_mirrors(sc, J, w, f, j, h.p, false, h.n, 0.0, lam, cie(), beta, rho);
            if (uniform(rng) >= rho) { fate = 0; break; }
            D3 wo = cosine_hemisphere(h.n, rng);
            beta *= shading_adjoint_corr(wi, wo, h.n, ngo);
            no = h.p + h.n * 1e-6; nd = wo;
            break;
        }
        }
    }
    return fate;
}

// One bounce of every queued path; the survivors are copied into the other path buffer.
template <bool MEDIA, bool INST, bool SHAPES, bool MIRROR>
__global__ void __launch_bounds__(128, MEDIA ? FTB_SHADE_MEDIA_MINB : FTB_SHADE_MINB) k_shade(Wave w, const DevJob* __restrict__ jobs,
                                                               Frame f, PathState in, const int32_t* in_count,
                                                               PathState out, int32_t* out_count) {
    const int32_t n_jobs = w.params[0];
    const bool multi = n_jobs > 1;
    TallyAcc acc;
    tally_init(acc, multi, n_jobs);
    const int front = in_count[0], nq = queue_len(in_count);
    FTB_FOR_WARP_CHUNKS(q, nq, &w.counts[kFetchShade]) {
        const int i = queue_entry(w, front, q);
        const int j = multi ? in.job[i] : 0;
        const DevJob& J = jobs[j];
        const DevScene& sc = J.sc;
        Pcg rng; rng.s = in.rng_s[i]; rng.inc = in.rng_i[i];
        D3 ro = mk(in.ox[i], in.oy[i], in.oz[i]), rd = mk(in.dx[i], in.dy[i], in.dz[i]);
        double lam = in.lam[i], beta = in.beta[i];
        double cie[3];   // read by the paths that connect or survive
        bool have_cie = false;
        auto load_cie = [&]() -> const double* {
            if (have_cie) return cie;
            cie[0] = in.cie[i]; cie[1] = in.cie[w.W + i]; cie[2] = in.cie[2 * (size_t)w.W + i];
            have_cie = true;
            return cie;
        };
        double ht = w.hit_t[i];
        int rec = w.hit_rec[i];
        Stk stk; stk.n = in.stk_n[i];
        for (int k = 0; k < stk.n; ++k) stk.e[k] = in.stk[k * w.W + i];
        log_hit<INST>(w, in, i, sc, rec);
        bool costly = false;
        D3 no, nd;
        const int fate = shade_bounce<MEDIA, INST, SHAPES, MIRROR>(sc, J, WaveQueue{w}, f, j, rng, ro, rd, lam, beta, stk, ht, rec,
                                                                   INST ? w.hit_sub[i] : -1, load_cie, no, nd, costly);
        if (fate == 0) {
            tally_add(acc, jobs, multi, j, T_ABS, to_fixed(beta, J.tally_scale_inv, f.status));
            log_finish(w, in, i, 0, beta);
            continue;
        }
        if (fate == 1) {
            tally_add(acc, jobs, multi, j, T_ESC, to_fixed(beta, J.tally_scale_inv, f.status));
            log_finish(w, in, i, 1, beta);
            continue;
        }
        const int32_t b = in.nbounce[i];
        if (b + 1 >= J.max_bounce) {
            tally_add(acc, jobs, multi, j, T_RES, to_fixed(beta, J.tally_scale_inv, f.status));
            log_finish(w, in, i, 2, beta);
            continue;
        }
        load_cie();
        const int o = (stk.n > 0 || costly) ? w.W - 1 - agg_inc(out_count + 1) : agg_inc(out_count);
        out.rng_s[o] = rng.s; out.rng_i[o] = rng.inc;
        out.ox[o] = no.x; out.oy[o] = no.y; out.oz[o] = no.z;
        out.dx[o] = nd.x; out.dy[o] = nd.y; out.dz[o] = nd.z;
        out.lam[o] = lam; out.beta[o] = beta;
        out.cie[o] = cie[0]; out.cie[w.W + o] = cie[1]; out.cie[2 * (size_t)w.W + o] = cie[2];
        out.stk_n[o] = stk.n;
        for (int k = 0; k < stk.n; ++k) out.stk[k * w.W + o] = stk.e[k];
        out.nbounce[o] = b + 1;
        if (multi) out.job[o] = j;
        log_move(w, in, i, out, o);
    }
    tally_finish(acc, jobs, multi, n_jobs);
}

// Add a splat's four words to a pixel: one 32-byte bulk reduction (sm_90+ cp.reduce of u64
// sums) from a shared-memory slot of the thread's own, or four atomics where the caller's film
// is not 16-byte aligned, which the bulk operation requires.  Both are exact integer sums in
// any order.  The four separate atomics bounded the connection kernel: Cornell, 256^2, 2^24
// photons (40 M connections): 5.1 ms with them, 2.8 ms with the bulk reduction, 2.4 ms with
// no film update at all; glass, 1024^2, 2^27 photons: 33.5 and 32.0 ms.
__device__ __forceinline__ void film_add(int64_t* film, int pix, long long x, long long y, long long z, long long n) {
    __shared__ alignas(32) long long slot[128][4];   // blocks are of 128 threads
    long long* px = reinterpret_cast<long long*>(film) + 4 * (size_t)pix;
    if ((reinterpret_cast<uintptr_t>(film) & 15) == 0) {
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the slot's last reduction has read it
        long long* sp = slot[threadIdx.x];
        sp[0] = x; sp[1] = y; sp[2] = z; sp[3] = n;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.u64 [%0], [%1], 32;"
                     :: "l"(px), "r"((uint32_t)__cvta_generic_to_shared(sp)) : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        return;
    }
    atomicAdd(reinterpret_cast<unsigned long long*>(px), (unsigned long long)x);
    atomicAdd(reinterpret_cast<unsigned long long*>(px + 1), (unsigned long long)y);
    atomicAdd(reinterpret_cast<unsigned long long*>(px + 2), (unsigned long long)z);
    atomicAdd(reinterpret_cast<unsigned long long*>(px + 3), (unsigned long long)n);
}
// Every thread of a kernel that splats, before it ends: its reductions are complete.
__device__ __forceinline__ void film_finish() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void splat(const DevJob& J, int view, int pix, double X, double Y, double Z,
                                      int32_t* status) {
    film_add(view_film(J, view), pix, to_fixed(X, J.film_scale_inv, status), to_fixed(Y, J.film_scale_inv, status),
             to_fixed(Z, J.film_scale_inv, status), 1);
}

// A mirror record's tests, in connectSpecularPlane's order (render.h:1366-1379): the light
// leg p -> R, stopping short of the mirror, must be clear; a closest hit from the eye toward
// R must land on a planar mirror within 1e-4 (1 + dE) of R (mirrorSeenAt, render.h:
// 1294-1308).  On success: the mirror's material, the unfolded length D, the mirror point
// R, the leg R -> eye (wRE, dE) and the pixel's solid angle, recomputed from the record
// with the push's arithmetic.
struct MirrorSeen {
    int mat;
    double D, dE, omega;
    D3 R, wRE;
};
template <bool COUNT, bool INST, bool SHAPES>
__device__ __forceinline__ bool mirror_seen(const DevJob& J, const Frame& f, int view, int plane, D3 p, D3 wP,
                                            double dP, TravCount& cnt, MirrorSeen& ms) {
    const DevScene& sc = J.sc;
    const DevPlane& mp = sc.planes[plane];
    const D3 pn = ld3(mp.n);
    {
        const RayCtx L = make_ray(p + wP * 1e-6, wP);
        if (traverse_any<COUNT, INST, SHAPES>(sc, L, EPS_RAY, (dP - 2e-6) - EPS_RAY, f.status, cnt)) return false;
    }
    const DevCam& cam = view_cam(J, view);
    const D3 eye = ld3(cam.eye);
    const double se = dot(pn, eye) - mp.d;
    const D3 eye_m = eye - pn * (2.0 * se);
    ms.D = len(eye_m - p);
    ms.R = p + wP * dP;
    ms.dE = ms.D - dP;
    ms.wRE = (eye - ms.R) * (1.0 / ms.dE);
    const D3 wE = neg(ms.wRE);
    double t;
    int sub = -1;
    const int rec = traverse_closest<COUNT, INST, SHAPES>(sc, make_ray(eye, wE), EPS_RAY, t, &sub, f.status, cnt);
    if (rec < 0) return false;
    if (fabs(t - ms.dE) > 1e-4 * (1.0 + ms.dE)) return false;
    Rec r;
    load_rec(sc.recs, rec, r);
    ms.mat = rec_mat(r);
    if (INST && rec_type(r) == REC_INST) {
        Hit h;
        instance_hit(sc.inst[rec_inst(r)], sub, eye, wE, h);
        ms.mat = h.mat;
    }
    if (ms.mat < 0 || ms.mat >= sc.n_mats || !planar_mirror(sc.mats[ms.mat])) return false;
    int px, py; double cos_cam, dist2e;
    cam_project(cam, ms.R, px, py, cos_cam, dist2e);
    ms.omega = cam_pixel_solid_angle(cam, cos_cam);
    return true;
}

// One-wavelength mirror record: splatMirrorLegs (render.h:1315-1331) with the reflectance of
// the mirror the eye sees: (beta * (weight * shape)) * refl / (D^2 Omega), times the two legs'
// transmittance in media.
template <bool COUNT, bool INST, bool SHAPES>
__device__ __forceinline__ void mirror_splat(const DevJob& J, const Frame& f, int view, int plane, D3 p, D3 wP, double dP,
                                             double a, double lam, double X, double Y, double Z, int pix,
                                             TravCount& cnt) {
    MirrorSeen ms;
    if (!mirror_seen<COUNT, INST, SHAPES>(J, f, view, plane, p, wP, dP, cnt, ms)) return;
    const DevScene& sc = J.sc;
    const double inv_d2_omega = 1.0 / (ms.D * ms.D * ms.omega);
    const double refl = clamp01(spec_slot(sc, sc.mats[ms.mat].reflect, lam, 0.5));
    double contrib = a * refl * inv_d2_omega;
    if (contrib <= 0.0) return;
    if (sc.n_med > 0) {
        contrib *= media_transmittance(sc, p, wP, dP, lam);
        contrib *= media_transmittance(sc, ms.R, ms.wRE, ms.dE, lam);
    }
    splat(J, view, pix, X * contrib, Y * contrib, Z * contrib, f.status);
}
template <bool COUNT, bool INST, bool SHAPES>
__device__ __noinline__ void mirror_record(const DevJob& J, const Wave& w, const Frame& f, int i, TravCount& cnt) {
    mirror_splat<COUNT, INST, SHAPES>(J, f, w.sview[i] & 0xffff, w.sview[i] >> 16, mk(w.sox[i], w.soy[i], w.soz[i]),
                                      mk(w.sdx[i], w.sdy[i], w.sdz[i]), w.smax[i], w.sval[i], w.slam[i], w.sxyz[i],
                                      w.sxyz[w.S + i], w.sxyz[2 * (size_t)w.S + i], ~w.spix[i], cnt);
}

// A connection that found the queue full: the same test and splat, by the lane that made it.
template <bool INST, bool SHAPES>
__device__ __noinline__ void connect_now(const DevJob& J, const Frame& f, int view, D3 o, D3 d, double tmax, double X,
                                         double Y, double Z, int pix) {
    TravCount cnt{0, 0, 0};
    const RayCtx R = make_ray(o, d);
    if (traverse_any<false, INST, SHAPES>(J.sc, R, EPS_RAY, tmax - EPS_RAY, f.status, cnt)) return;
    splat(J, view, pix, X, Y, Z, f.status);
}
template <bool INST, bool SHAPES>
__device__ __noinline__ void mirror_now(const DevJob& J, const Frame& f, int view, int plane, D3 p, D3 wP, double dP,
                                        double a, double lam, double X, double Y, double Z, int pix) {
    TravCount cnt{0, 0, 0};
    mirror_splat<false, INST, SHAPES>(J, f, view, plane, p, wP, dP, a, lam, X, Y, Z, pix, cnt);
}

// Camera connections: occlusion (Scene::occluded, default tmin 1e-6) then Film::add.
// MIRROR: the queue may also hold mirror connections (scenes with planar mirrors).
template <bool COUNT, bool INST, bool SHAPES, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_TRAV_MINB) k_shadow(Wave w, const DevJob* __restrict__ jobs,
                                                              Frame f, const int32_t* __restrict__ order) {
    const int32_t n_jobs = w.params[0];
    int n = w.counts[kShadowCount];
    if (n > w.S) n = w.S;
    TravCount cnt{0, 0, 0};
    unsigned long long rays = 0;
    FTB_FOR_WARP_CHUNKS(q, n, &w.counts[kFetchShadow]) {
        const int i = order ? order[q] : q;
        const DevJob& J = jobs[n_jobs > 1 ? w.sjob[i] : 0];
        const DevScene& sc = J.sc;
        if (COUNT) rays++;
        if (MIRROR && w.spix[i] < 0) {
            mirror_record<COUNT, INST, SHAPES>(J, w, f, i, cnt);
            continue;
        }
        D3 o = mk(w.sox[i], w.soy[i], w.soz[i]), d = mk(w.sdx[i], w.sdy[i], w.sdz[i]);
        double max_dist = w.smax[i];
        RayCtx R = make_ray(o, d);
        if (traverse_any<COUNT, INST, SHAPES>(sc, R, EPS_RAY, max_dist - EPS_RAY, f.status, cnt)) continue;
        splat(J, w.sview[i], w.spix[i], w.sxyz[i], w.sxyz[w.S + i], w.sxyz[2 * (size_t)w.S + i], f.status);
    }
    film_finish();
    if (COUNT) {
        block_add3(f.stats + 3, rays, cnt.nodes, cnt.recs);
        block_add1(f.stats + 7, cnt.exact);
    }
}

// ------------------------------------------------------------------ hero bundles -------
// Hero-wavelength sampling (Renderer::tracePhotonHero / tracePhotonHeroLoop, render.h:
// 2252-2631; the policies of hero.h:28-70): a photon carries C wavelengths drawn from one
// stratified variate; the hero decides the geometry, analog Russian roulette uses the
// maximum over the live wavelengths with the bounded reweights booked as absorption, and a
// dielectric de-heroes (the hero goes on alone, its beta times C).  A camera connection
// tests occlusion once and splats every live wavelength.  The reference runs bundles only
// in scenes without media, and so does this path (the host sends such jobs to the scalar
// kernels).

// A bundle's connection, plain (pix >= 0: val per wavelength is the contribution) or through
// mirror `view >> 16` (pix < 0).  Returns false when the queue is full.
__device__ __forceinline__ bool queue_hero(const Wave& w, int job, int view, D3 o, D3 d, double tmax, int nup,
                                           const double* lam, const double* val, int pix) {
    const int i = queue_slot(w);
    if (i < 0) return false;
    w.sox[i] = o.x; w.soy[i] = o.y; w.soz[i] = o.z;
    w.sdx[i] = d.x; w.sdy[i] = d.y; w.sdz[i] = d.z;
    w.smax[i] = tmax; w.spix[i] = pix; w.sjob[i] = job; w.sview[i] = view;
    w.slam[i] = lam[0]; w.sval[i] = val[0];
    for (int k = 1; k < nup; ++k) {
        w.xlam[(size_t)(k - 1) * w.S + i] = lam[k];
        w.xval[(size_t)(k - 1) * w.S + i] = val[k];
    }
    w.snup[i] = nup;
    return true;
}
template <bool INST, bool SHAPES>
__device__ __noinline__ void connect_now_hero(const DevJob& J, const Frame& f, int view, D3 o, D3 d, double tmax,
                                              int nup, const double* lam, const double* val, int pix);
__device__ __forceinline__ void push_hero(const WaveQueue& q, const DevJob&, const Frame& f, int job, int view, D3 o,
                                          D3 d, double tmax, int nup, const double* lam, const double* val, int pix) {
    if (!queue_hero(q.w, job, view, o, d, tmax, nup, lam, val, pix)) atomicOr(f.status, ST_QUEUE_OVERFLOW);
}
template <bool INST, bool SHAPES>
__device__ __forceinline__ void push_hero(const PathQueue<INST, SHAPES>& q, const DevJob& J, const Frame& f, int job,
                                          int view, D3 o, D3 d, double tmax, int nup, const double* lam,
                                          const double* val, int pix) {
    if (!queue_hero(q.w, job, view, o, d, tmax, nup, lam, val, pix))
        connect_now_hero<INST, SHAPES>(J, f, view, o, d, tmax, nup, lam, val, pix);
}

// connectHero (render.h:564-577): one connectGeom, a contribution per live wavelength
template <class Q>
__device__ void connect_surface_hero(const DevJob& J, const Q& w, const Frame& f, int job, D3 p, D3 n,
                                     D3 ng, D3 wi, const double* lam, const double* beta, const double* rho,
                                     int nup) {
    for (int v = 0; v < view_count(J); ++v) {
        const DevCam& cam = view_cam(J, v);
        const EyeRay er = eye_ray(cam, p);
        const D3 wdir = er.dir;
        const double dist = er.dist, dist2 = er.dist2;
        double cos_surf = dot(n, wdir);
        if (cos_surf <= 0) continue;
        double stg = shadow_terminator_g(wdir, n, ng);
        if (stg <= 0.0) continue;
        int px, py; double cos_cam;
        if (!eye_project(cam, er, px, py, cos_cam)) continue;
        double omega = cam_pixel_solid_angle(cam, cos_cam);
        double corr = shading_adjoint_corr(wi, wdir, n, ng);
        double denom = dist2 * omega;
        double val[kHeroMax];
        for (int i = 0; i < nup; ++i) {
            double fr = rho[i] / PI_D;
            val[i] = beta[i] * fr * cos_surf * corr / denom * stg;
        }
        push_hero(w, J, f, job, v, p + ng * 1e-6, wdir, dist - 2e-6, nup, lam, val, py * cam.rx + px);
    }
}

// connect_mirrors for a bundle's live wavelengths (camSpecularSplatAllHero, render.h:
// 1570-1576): a record carries (lambda_i, beta_i x (rho_i x shape)) per wavelength, as the
// bundle's camera connections do; k_shadow_hero evaluates the mirror's reflectance for each.
template <class Q>
__device__ __noinline__ void connect_mirrors_hero(const DevScene& sc, const DevJob& J, const Q& w, const Frame& f,
                                                  int job, D3 p, D3 n, const double* lam, const double* beta,
                                                  const double* rho, int nup) {
    for (int k = 0; k < sc.n_planes; ++k) {
        for (int v = 0; v < view_count(J); ++v) {
            D3 wP; double dP, shape; int pix;
            if (!mirror_geometry(sc.planes[k], view_cam(J, v), p, false, n, 0.0, wP, dP, shape, pix)) continue;
            double val[kHeroMax];
            for (int q = 0; q < nup; ++q) val[q] = beta[q] * (rho[q] * shape);
            push_hero(w, J, f, job, v | (k << 16), p, wP, dP, nup, lam, val, ~pix);
        }
    }
}

__device__ __forceinline__ double sum_of(const double* a, int n) {   // activeSum (render.h:2324)
    double s = 0.0;
    for (int i = 0; i < n; ++i) s += a[i];
    return s;
}
__device__ __forceinline__ double max_of(const double* a, int n) {   // hero::maxOf (hero.h:120-126)
    double m = a[0];
    for (int i = 1; i < n; ++i) if (a[i] > m) m = a[i];
    return m;
}

template <bool STREAM, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_EMIT_MINB) k_emit_hero(Wave w, const DevJob* __restrict__ jobs, Frame f, PathState out,
                                                   int32_t* out_count) {
    const int32_t n_jobs = w.params[0];
    const bool multi = n_jobs > 1;
    const PhotonSource src = photon_source<STREAM>(w, out_count);
    TallyAcc acc;
    tally_init(acc, multi, n_jobs);
    for (int64_t t = blockIdx.x * blockDim.x + threadIdx.x; t < src.n; t += gridDim.x * blockDim.x) {
        uint64_t k;
        const int j = photon_job<STREAM>(jobs, n_jobs, src, t, k);
        const DevJob& J = jobs[j];
        const DevScene& sc = J.sc;
        const int C = J.hero_c;
        Pcg rng = seed_photon(k);
        if (sc.total_power <= 0.0 || sc.n_emit == 0) { log_emitted(w, k, 4, 0.0); continue; }
        const DevEmit& em = sc.emit[select_emitter(sc, rng)];
        D3 origin, emit_n, dir;
        emit_sample(em, rng, origin, emit_n, dir);
        // hero::sampleBundle (hero.h:100-113): one variate, strata u + i/C wrapped into [0,1)
        double lam[kHeroMax], beta[kHeroMax], one[kHeroMax], wl[kHeroMax];
        const bool band = J.lambda_mode == FTB_LAMBDA_UNIFORM_380_780;
        double u = uniform(rng), pdf;
        if (band) { lam[0] = sample_uniform_band(em, u, wl[0]); pdf = wl[0]; }
        else lam[0] = sample_at(em, u, pdf);
        if (pdf <= 0) { log_emitted(w, k, 4, 0.0); continue; }
        for (int i = 1; i < C; ++i) {
            double uu = u + (double)i / (double)C;
            if (uu >= 1.0) uu -= 1.0;
            double p2;
            if (band) lam[i] = sample_uniform_band(em, uu, wl[i]);
            else lam[i] = sample_at(em, uu, p2);
        }
        double base = (sc.n_emit == 1) ? em.power : sc.total_power;
        base *= 1.0;   // spotW
        for (int i = 0; i < C; ++i) {
            beta[i] = base / C;
            if (band) beta[i] *= wl[i];
            one[i] = 1.0;
        }
        tally_add(acc, jobs, multi, j, T_EMIT, to_fixed(sum_of(beta, C), J.tally_scale_inv, f.status));
        connect_surface_hero(J, WaveQueue{w}, f, j, origin, emit_n, emit_n, emit_n, lam, beta, one, C);
        if (MIRROR && sc.n_planes > 0) connect_mirrors_hero(sc, J, WaveQueue{w}, f, j, origin, emit_n, lam, beta, one, C);
        D3 ro = origin + dir * 1e-6;
        if (J.max_bounce <= 0) {
            tally_add(acc, jobs, multi, j, T_RES, to_fixed(sum_of(beta, C), J.tally_scale_inv, f.status));
            log_emitted(w, k, 2, beta[0]);
            continue;
        }
        const int o = photon_enqueue<STREAM>(w, out, out_count, src, j, multi, k);
        out.rng_s[o] = rng.s; out.rng_i[o] = rng.inc;
        out.ox[o] = ro.x; out.oy[o] = ro.y; out.oz[o] = ro.z;
        out.dx[o] = dir.x; out.dy[o] = dir.y; out.dz[o] = dir.z;
        for (int i = 0; i < C; ++i) {
            out.hlam[(size_t)i * w.W + o] = lam[i];
            out.hbeta[(size_t)i * w.W + o] = beta[i];
        }
        out.hlive[o] = C;
        out.stk_n[o] = 0;
    }
    tally_finish(acc, jobs, multi, n_jobs);
}

// One bounce of a bundle (tracePhotonHeroLoop): as shade_bounce, over the nup live
// wavelengths; `absorbed`: the reweights booked as absorption (fixed point, per add).
template <bool INST, bool SHAPES, bool MIRROR, class Q>
__device__ __forceinline__ int shade_bounce_hero(const DevScene& sc, const DevJob& J, const Q& w, const Frame& f, int j,
                                                 Pcg& rng, D3 ro, D3 rd, double (&lam)[kHeroMax],
                                                 double (&beta)[kHeroMax], int& nup, Stk& stk, double ht, int rec,
                                                 int sub, D3& no, D3& nd, bool& costly, long long& absorbed) {
    const int C = J.hero_c;
    const bool valid = rec >= 0;
    const double d_event = valid ? ht : 1e30;
    {   // Beer-Lambert per live wavelength (render.h:2389-2398)
        int mi = stk_top_mat(stk);
        if (mi >= 0)
            for (int i = 0; i < nup; ++i) {
                double a = spec_slot(sc, sc.mats[mi].absorb, lam[i], 0.0);
                if (a > 0.0) beta[i] *= exp(-a * d_event);
            }
    }
    int fate = -1;
    no = ro; nd = rd;
    absorbed = 0;
    if (!valid) {
        fate = 1;
    } else {
        Rec r;
        load_rec(sc.recs, rec, r);
        if (SHAPES && rec_type(r) == REC_CURVE) costly = true;
        Hit h;
        if (INST && rec_type(r) == REC_INST) {
            instance_hit(sc.inst[rec_inst(r)], sub, ro, rd, h);
            h.prim = r.prim;
        } else {
            RayCtx R = make_ray(ro, rd);
            hit_attributes<SHAPES>(sc.tri_n, R, sc.recs, rec, r, h);
        }
        const DevMat& m = sc.mats[h.mat];
        switch (m.type) {
        case FTB_MAT_DIFFUSE_TRANSMIT: {   // render.h:2454-2503
            double rr[kHeroMax], rt[kHeroMax];
            for (int i = 0; i < nup; ++i) {
                double a = clamp01(spec_slot(sc, m.reflect, lam[i], 0.5));
                double b = clamp01(spec_slot(sc, m.transmit, lam[i], 0.0));
                double s = a + b;
                if (s > 1.0) { a /= s; b /= s; }
                rr[i] = a; rt[i] = b;
            }
            D3 ngo = oriented_geo_n(h);
            D3 wi = mk(-rd.x, -rd.y, -rd.z);
            connect_surface_hero(J, w, f, j, h.p, h.n, ngo, wi, lam, beta, rr, nup);
            connect_surface_hero(J, w, f, j, h.p, neg(h.n), neg(ngo), wi, lam, beta, rt, nup);
            if (MIRROR && sc.n_planes > 0) {
                connect_mirrors_hero(sc, J, w, f, j, h.p, h.n, lam, beta, rr, nup);
                connect_mirrors_hero(sc, J, w, f, j, h.p, neg(h.n), lam, beta, rt, nup);
            }
            double q_r = max_of(rr, nup), q_t = max_of(rt, nup);
            double sum_h = q_r + q_t;
            if (nup > 1 && sum_h > 1.0) { q_r /= sum_h; q_t /= sum_h; sum_h = q_r + q_t; }
            double uu = uniform(rng);
            if (uu < q_r || uu < sum_h) {
                const bool front = uu < q_r;
                for (int i = 0; i < nup; ++i) {
                    double wgt = (front ? rr[i] : rt[i]) / (front ? q_r : q_t);
                    absorbed += to_fixed(beta[i] * (1.0 - wgt), J.tally_scale_inv, f.status);
                    beta[i] *= wgt;
                }
                D3 wo = cosine_hemisphere(front ? h.n : mk(-h.n.x, -h.n.y, -h.n.z), rng);
                double corr = shading_adjoint_corr(wi, wo, h.n, ngo);
                for (int i = 0; i < nup; ++i) beta[i] *= corr;
                no = front ? h.p + h.n * 1e-6 : h.p - h.n * 1e-6;
                nd = wo;
            } else {
                fate = 0;
            }
            break;
        }
        case FTB_MAT_MIRROR:
        case FTB_MAT_FILTER:
        case FTB_MAT_GLOSSY: {   // achromatic lobes (render.h:2509-2537)
            double cc[kHeroMax];
            for (int i = 0; i < nup; ++i)
                cc[i] = (m.type == FTB_MAT_FILTER) ? clamp01(spec_slot(sc, m.transmit, lam[i], 0.0))
                                                   : clamp01(spec_slot(sc, m.reflect, lam[i], 0.5));
            double q = max_of(cc, nup);
            if (uniform(rng) >= q) { fate = 0; break; }
            for (int i = 0; i < nup; ++i) {
                double wgt = cc[i] / q;
                absorbed += to_fixed(beta[i] * (1.0 - wgt), J.tally_scale_inv, f.status);
                beta[i] *= wgt;
            }
            if (m.type == FTB_MAT_MIRROR) {
                no = h.p + h.n * 1e-6; nd = reflect(rd, h.n);
            } else if (m.type == FTB_MAT_FILTER) {
                no = h.p + rd * 1e-6;
            } else {
                D3 o = sample_glossy(reflect(rd, h.n), m.roughness, rng);
                if (dot(o, h.n) <= 0) { fate = 0; break; }
                no = h.p + h.n * 1e-6; nd = o;
            }
            break;
        }
        case FTB_MAT_HALF_MIRROR: {   // de-hero, then the scalar half mirror (render.h:2546-2589, 1702-1711)
            if (nup > 1) { beta[0] *= (double)C; nup = 1; }
            const double rr = clamp01(spec_slot(sc, m.reflect, lam[0], 0.5));
            if (uniform(rng) < rr) {
                nd = reflect(rd, h.n);
                no = h.p + h.n * 1e-6;
            } else {
                no = h.p + rd * 1e-6;
            }
            break;
        }
        case FTB_MAT_DIELECTRIC: {   // de-hero, then the scalar interaction (render.h:2539-2589)
            if (nup > 1) { beta[0] *= (double)C; nup = 1; }
            const double lam0 = lam[0];
            bool entering = dot(rd, h.ng) < 0.0;
            int mi = h.mat, pr = m.priority;
            bool has_pri = pr != INT_MIN;
            bool transmitted = false;
            if (entering) {
                int out_mat = stk_top_mat(stk), out_pri = stk_top_pri(stk);
                bool ranked = has_pri && (stk.n == 0 || (out_mat >= 0 && sc.mats[out_mat].priority != INT_MIN));
                if (ranked && stk.n != 0 && pr <= out_pri) {
                    stk_push(stk, mi, pr, f.status);
                    no = h.p + rd * 1e-6;
                } else {
                    double ext = (ranked && out_mat >= 0) ? mat_ior(sc, sc.mats[out_mat], lam0) : 1.0;
                    refract_or_reflect(sc, m, h, rd, lam0, rng, transmitted, ext, no, nd);
                    if (transmitted) stk_push(stk, mi, pr, f.status);
                }
            } else {
                Stk after = stk;
                stk_pop_mat(after, mi);
                int new_mat = stk_top_mat(after), new_pri = stk_top_pri(after);
                bool ranked = has_pri && (after.n == 0 || (new_mat >= 0 && sc.mats[new_mat].priority != INT_MIN));
                if (ranked && new_mat >= 0 && pr <= new_pri) {
                    stk_pop_mat(stk, mi);
                    no = h.p + rd * 1e-6;
                } else {
                    double ext = (ranked && new_mat >= 0) ? mat_ior(sc, sc.mats[new_mat], lam0) : 1.0;
                    refract_or_reflect(sc, m, h, rd, lam0, rng, transmitted, ext, no, nd);
                    if (transmitted) stk_pop_mat(stk, mi);
                }
            }
            break;
        }
        default: {   // Diffuse (render.h:2591-2625)
            double rho[kHeroMax];
            for (int i = 0; i < nup; ++i) rho[i] = clamp01(spec_slot(sc, m.reflect, lam[i], 0.5));
            D3 ngo = oriented_geo_n(h);
            D3 wi = mk(-rd.x, -rd.y, -rd.z);
            connect_surface_hero(J, w, f, j, h.p, h.n, ngo, wi, lam, beta, rho, nup);
            if (MIRROR && sc.n_planes > 0) connect_mirrors_hero(sc, J, w, f, j, h.p, h.n, lam, beta, rho, nup);
            double q = max_of(rho, nup);
            if (uniform(rng) >= q) { fate = 0; break; }
            for (int i = 0; i < nup; ++i) {
                double wgt = rho[i] / q;
                absorbed += to_fixed(beta[i] * (1.0 - wgt), J.tally_scale_inv, f.status);
                beta[i] *= wgt;
            }
            D3 wo = cosine_hemisphere(h.n, rng);
            double corr = shading_adjoint_corr(wi, wo, h.n, ngo);
            for (int i = 0; i < nup; ++i) beta[i] *= corr;
            no = h.p + h.n * 1e-6; nd = wo;
            break;
        }
        }
    }
    return fate;
}

template <bool INST, bool SHAPES, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_SHADE_HERO_MINB) k_shade_hero(Wave w, const DevJob* __restrict__ jobs,
                                                                    Frame f, PathState in, const int32_t* in_count,
                                                                    PathState out, int32_t* out_count) {
    const int32_t n_jobs = w.params[0];
    const bool multi = n_jobs > 1;
    TallyAcc acc;
    tally_init(acc, multi, n_jobs);
    const int front = in_count[0], nq = queue_len(in_count);
    FTB_FOR_WARP_CHUNKS(q, nq, &w.counts[kFetchShade]) {
        const int p = queue_entry(w, front, q);
        const int j = multi ? in.job[p] : 0;
        const DevJob& J = jobs[j];
        const DevScene& sc = J.sc;
        Pcg rng; rng.s = in.rng_s[p]; rng.inc = in.rng_i[p];
        D3 ro = mk(in.ox[p], in.oy[p], in.oz[p]), rd = mk(in.dx[p], in.dy[p], in.dz[p]);
        int nup = in.hlive[p];
        double lam[kHeroMax], beta[kHeroMax];
        for (int k = 0; k < nup; ++k) {
            lam[k] = in.hlam[(size_t)k * w.W + p];
            beta[k] = in.hbeta[(size_t)k * w.W + p];
        }
        double ht = w.hit_t[p];
        int rec = w.hit_rec[p];
        Stk stk; stk.n = in.stk_n[p];
        for (int k = 0; k < stk.n; ++k) stk.e[k] = in.stk[k * w.W + p];
        log_hit<INST>(w, in, p, sc, rec);
        bool costly = false;
        D3 no, nd;
        long long absorbed;
        const int fate = shade_bounce_hero<INST, SHAPES, MIRROR>(sc, J, WaveQueue{w}, f, j, rng, ro, rd, lam, beta, nup,
                                                                 stk, ht, rec, INST ? w.hit_sub[p] : -1, no, nd, costly,
                                                                 absorbed);
        if (absorbed) tally_add(acc, jobs, multi, j, T_ABS, absorbed);
        if (fate >= 0) {
            tally_add(acc, jobs, multi, j, fate == 0 ? T_ABS : T_ESC,
                      to_fixed(sum_of(beta, nup), J.tally_scale_inv, f.status));
            log_finish(w, in, p, fate, beta[0]);
            continue;
        }
        const int32_t b = in.nbounce[p];
        if (b + 1 >= J.max_bounce) {
            tally_add(acc, jobs, multi, j, T_RES, to_fixed(sum_of(beta, nup), J.tally_scale_inv, f.status));
            log_finish(w, in, p, 2, beta[0]);
            continue;
        }
        const int o = (stk.n > 0 || costly) ? w.W - 1 - agg_inc(out_count + 1) : agg_inc(out_count);
        out.rng_s[o] = rng.s; out.rng_i[o] = rng.inc;
        out.ox[o] = no.x; out.oy[o] = no.y; out.oz[o] = no.z;
        out.dx[o] = nd.x; out.dy[o] = nd.y; out.dz[o] = nd.z;
        for (int k = 0; k < nup; ++k) {
            out.hlam[(size_t)k * w.W + o] = lam[k];
            out.hbeta[(size_t)k * w.W + o] = beta[k];
        }
        out.hlive[o] = nup;
        out.stk_n[o] = stk.n;
        for (int k = 0; k < stk.n; ++k) out.stk[k * w.W + o] = stk.e[k];
        out.nbounce[o] = b + 1;
        if (multi) out.job[o] = j;
        log_move(w, in, p, out, o);
    }
    tally_finish(acc, jobs, multi, n_jobs);
}

// A bundle's mirror record: every live wavelength is its own splat with its own reflectance
// (splatMirrorLegs, render.h:1321-1330; bundles run without media); a wavelength whose
// contribution is not positive adds nothing, not even to the hit count.
template <bool COUNT, bool INST, bool SHAPES, class Lam, class Val>
__device__ __forceinline__ void mirror_splat_hero(const DevJob& J, const Frame& f, int view, int plane, D3 p, D3 wP,
                                                  double dP, int nup, const Lam& lam_of, const Val& val_of, int pix,
                                                  TravCount& cnt) {
    MirrorSeen ms;
    if (!mirror_seen<COUNT, INST, SHAPES>(J, f, view, plane, p, wP, dP, cnt, ms)) return;
    const DevScene& sc = J.sc;
    const double inv_d2_omega = 1.0 / (ms.D * ms.D * ms.omega);
    long long sx = 0, sy = 0, sz = 0, hits = 0;
    for (int k = 0; k < nup; ++k) {
        const double lam = lam_of(k);
        const double refl = clamp01(spec_slot(sc, sc.mats[ms.mat].reflect, lam, 0.5));
        const double contrib = val_of(k) * refl * inv_d2_omega;
        if (contrib <= 0.0) continue;
        sx += to_fixed(cie_x(lam) * contrib, J.film_scale_inv, f.status);
        sy += to_fixed(cie_y(lam) * contrib, J.film_scale_inv, f.status);
        sz += to_fixed(cie_z(lam) * contrib, J.film_scale_inv, f.status);
        ++hits;
    }
    if (!hits) return;
    film_add(view_film(J, view), pix, sx, sy, sz, hits);
}
template <bool COUNT, bool INST, bool SHAPES>
__device__ __noinline__ void mirror_record_hero(const DevJob& J, const Wave& w, const Frame& f, int i, TravCount& cnt) {
    auto lam_of = [&](int k) { return k == 0 ? w.slam[i] : w.xlam[(size_t)(k - 1) * w.S + i]; };
    auto val_of = [&](int k) { return k == 0 ? w.sval[i] : w.xval[(size_t)(k - 1) * w.S + i]; };
    mirror_splat_hero<COUNT, INST, SHAPES>(J, f, w.sview[i] & 0xffff, w.sview[i] >> 16,
                                           mk(w.sox[i], w.soy[i], w.soz[i]), mk(w.sdx[i], w.sdy[i], w.sdz[i]), w.smax[i],
                                           w.snup[i], lam_of, val_of, ~w.spix[i], cnt);
}

// A bundle's connection that was not occluded: every wavelength is one Film::add, each rounded
// to fixed point on its own; their integer sum goes to the pixel at once (integer sums are
// exact).
template <class Lam, class Val>
__device__ __forceinline__ void splat_hero(const DevJob& J, const Frame& f, int view, int pix, int nup,
                                           const Lam& lam_of, const Val& val_of) {
    long long sx = 0, sy = 0, sz = 0;
    for (int k = 0; k < nup; ++k) {
        const double lam = lam_of(k), c = val_of(k);
        double X = cie_x(lam) * c, Y = cie_y(lam) * c, Z = cie_z(lam) * c;
        sx += to_fixed(X, J.film_scale_inv, f.status);
        sy += to_fixed(Y, J.film_scale_inv, f.status);
        sz += to_fixed(Z, J.film_scale_inv, f.status);
    }
    film_add(view_film(J, view), pix, sx, sy, sz, nup);
}
// A bundle's connection that found the queue full: the same test and splat at once.
template <bool INST, bool SHAPES>
__device__ __noinline__ void connect_now_hero(const DevJob& J, const Frame& f, int view, D3 o, D3 d, double tmax,
                                              int nup, const double* lam, const double* val, int pix) {
    TravCount cnt{0, 0, 0};
    auto lam_of = [&](int k) { return lam[k]; };
    auto val_of = [&](int k) { return val[k]; };
    if (pix < 0) {
        mirror_splat_hero<false, INST, SHAPES>(J, f, view & 0xffff, view >> 16, o, d, tmax, nup, lam_of, val_of, ~pix, cnt);
        return;
    }
    const RayCtx R = make_ray(o, d);
    if (traverse_any<false, INST, SHAPES>(J.sc, R, EPS_RAY, tmax - EPS_RAY, f.status, cnt)) return;
    splat_hero(J, f, view, pix, nup, lam_of, val_of);
}

// Connections of bundles: one occlusion test, then a splat per wavelength.  MIRROR: the queue
// may also hold mirror records (scenes with planar mirrors).
template <bool COUNT, bool INST, bool SHAPES, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_TRAV_MINB) k_shadow_hero(Wave w, const DevJob* __restrict__ jobs,
                                                                   Frame f) {
    const int32_t n_jobs = w.params[0];
    int n = w.counts[kShadowCount];
    if (n > w.S) n = w.S;
    TravCount cnt{0, 0, 0};
    unsigned long long rays = 0;
    FTB_FOR_WARP_CHUNKS(i, n, &w.counts[kFetchShadow]) {
        const DevJob& J = jobs[n_jobs > 1 ? w.sjob[i] : 0];
        const DevScene& sc = J.sc;
        if (COUNT) rays++;
        if (MIRROR && w.spix[i] < 0) {
            mirror_record_hero<COUNT, INST, SHAPES>(J, w, f, i, cnt);
            continue;
        }
        D3 o = mk(w.sox[i], w.soy[i], w.soz[i]), d = mk(w.sdx[i], w.sdy[i], w.sdz[i]);
        double max_dist = w.smax[i];
        RayCtx R = make_ray(o, d);
        if (traverse_any<COUNT, INST, SHAPES>(sc, R, EPS_RAY, max_dist - EPS_RAY, f.status, cnt)) continue;
        splat_hero(J, f, w.sview[i], w.spix[i], w.snup[i],
                   [&](int k) { return k == 0 ? w.slam[i] : w.xlam[(size_t)(k - 1) * w.S + i]; },
                   [&](int k) { return k == 0 ? w.sval[i] : w.xval[(size_t)(k - 1) * w.S + i]; });
    }
    film_finish();
    if (COUNT) {
        block_add3(f.stats + 3, rays, cnt.nodes, cnt.recs);
        block_add1(f.stats + 7, cnt.exact);
    }
}

// ------------------------------------------------------------------ whole paths --------
// The queue's paths, each traced to its end by one lane: closest hit and shading alternate
// until the path ends, its state stays in the lane, and the connections are queued for
// k_shadow.  For queues of at most trace_limit() paths -- the tail of a streaming pass, and
// passes and renders that small from the start -- where launches per bounce mostly wait for
// the slowest warp of each: bound by the latency of one path's chain of bounces, not by
// throughput, so with fewer paths than lanes they are spread over all warps (a warp of few
// paths diverges less).  B200: preview of 2^16 photons 0.45 -> 0.26 ms, three renders of
// 23,334 photons through glass without allocation 5.06 -> 1.62 ms, fog + strands frame (32
// bounces) 117.2 -> 116.1, session of 4 views 23.6 -> 22.5.  The line lies at one path per
// resident lane: tails of 50,000, 150,000 and 500,000 paths took the same time on whole
// frames, and above it the kernel loses to the launches per bounce (all of a Cornell frame
// traced this way: 16.1 against 13.6 ms; glass 580-650 against 235 ms), since its warps run
// closest hits and materials of all kinds side by side at half the resident warps.
template <class Load, class Step>
__device__ __forceinline__ void trace_lanes(const Wave& w, int n, const Load& load, const Step& step) {
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    const int share = (n + warps - 1) / warps;
    bool more = lane < share, alive = false;   // this lane takes paths; it has one
    for (;;) {
        const unsigned want = __ballot_sync(0xffffffffu, more && !alive);
        if (want) {
            int base = 0;
            if (lane == 0) base = atomicAdd(&w.counts[kFetchExtend], __popc(want));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (more && !alive) {
                const int q = base + __popc(want & ((1u << lane) - 1u));
                if (q < n) { load(q); alive = true; }
                else more = false;
            }
        }
        if (!__any_sync(0xffffffffu, alive)) return;
        if (alive) alive = step();
    }
}

template <bool MEDIA, bool INST, bool SHAPES, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_TRACE_MINB) k_trace(Wave w, const DevJob* __restrict__ jobs, Frame f,
                                                              PathState in, const int32_t* in_count) {
    const int32_t n_jobs = w.params[0];
    const bool multi = n_jobs > 1;
    TallyAcc acc;
    tally_init(acc, multi, n_jobs);
    const int front = in_count[0];
    const PathQueue<INST, SHAPES> queue{w};
    TravCount cnt{0, 0, 0};
    int i = 0, j = 0, bounce = 0;
    Pcg rng{0, 0};
    D3 ro = mk(0, 0, 0), rd = mk(0, 0, 1);
    double lam = 0.0, beta = 0.0, cie[3] = {0.0, 0.0, 0.0};
    Stk stk;
    stk.n = 0;
    auto load = [&](int q) {
        i = queue_entry(w, front, q);
        j = multi ? in.job[i] : 0;
        rng.s = in.rng_s[i]; rng.inc = in.rng_i[i];
        ro = mk(in.ox[i], in.oy[i], in.oz[i]); rd = mk(in.dx[i], in.dy[i], in.dz[i]);
        lam = in.lam[i]; beta = in.beta[i];
        cie[0] = in.cie[i]; cie[1] = in.cie[w.W + i]; cie[2] = in.cie[2 * (size_t)w.W + i];
        stk.n = in.stk_n[i];
        for (int e = 0; e < stk.n; ++e) stk.e[e] = in.stk[e * w.W + i];
        bounce = in.nbounce[i];
    };
    auto step = [&]() -> bool {
        const DevJob& J = jobs[j];
        const DevScene& sc = J.sc;
        double t;
        int sub = -1;
        const int rec = traverse_closest<false, INST, SHAPES>(sc, make_ray(ro, rd), EPS_RAY, t, &sub, f.status, cnt);
        if (w.logs) {
            if (INST) w.hit_sub[i] = sub;
            log_hit<INST>(w, in, i, sc, rec);
        }
        bool costly = false;
        D3 no, nd;
        int fate = shade_bounce<MEDIA, INST, SHAPES, MIRROR>(sc, J, queue, f, j, rng, ro, rd, lam, beta, stk, t, rec,
                                                            sub, [&]() -> const double* { return cie; }, no, nd, costly);
        if (fate < 0 && ++bounce >= J.max_bounce) fate = 2;
        ro = no; rd = nd;
        if (fate < 0) return true;
        tally_add(acc, jobs, multi, j, fate == 0 ? T_ABS : (fate == 1 ? T_ESC : T_RES),
                  to_fixed(beta, J.tally_scale_inv, f.status));
        log_finish(w, in, i, fate, beta);
        return false;
    };
    trace_lanes(w, queue_len(in_count), load, step);
    film_finish();
    tally_finish(acc, jobs, multi, n_jobs);
}

template <bool INST, bool SHAPES, bool MIRROR>
__global__ void __launch_bounds__(128, FTB_TRACE_MINB) k_trace_hero(Wave w, const DevJob* __restrict__ jobs, Frame f,
                                                                   PathState in, const int32_t* in_count) {
    const int32_t n_jobs = w.params[0];
    const bool multi = n_jobs > 1;
    TallyAcc acc;
    tally_init(acc, multi, n_jobs);
    const int front = in_count[0];
    const PathQueue<INST, SHAPES> queue{w};
    TravCount cnt{0, 0, 0};
    int i = 0, j = 0, bounce = 0, nup = 0;
    Pcg rng{0, 0};
    D3 ro = mk(0, 0, 0), rd = mk(0, 0, 1);
    double lam[kHeroMax], beta[kHeroMax];
    Stk stk;
    stk.n = 0;
    auto load = [&](int q) {
        i = queue_entry(w, front, q);
        j = multi ? in.job[i] : 0;
        rng.s = in.rng_s[i]; rng.inc = in.rng_i[i];
        ro = mk(in.ox[i], in.oy[i], in.oz[i]); rd = mk(in.dx[i], in.dy[i], in.dz[i]);
        nup = in.hlive[i];
        for (int k = 0; k < nup; ++k) {
            lam[k] = in.hlam[(size_t)k * w.W + i];
            beta[k] = in.hbeta[(size_t)k * w.W + i];
        }
        stk.n = in.stk_n[i];
        for (int e = 0; e < stk.n; ++e) stk.e[e] = in.stk[e * w.W + i];
        bounce = in.nbounce[i];
    };
    auto step = [&]() -> bool {
        const DevJob& J = jobs[j];
        const DevScene& sc = J.sc;
        double t;
        int sub = -1;
        const int rec = traverse_closest<false, INST, SHAPES>(sc, make_ray(ro, rd), EPS_RAY, t, &sub, f.status, cnt);
        if (w.logs) {
            if (INST) w.hit_sub[i] = sub;
            log_hit<INST>(w, in, i, sc, rec);
        }
        bool costly = false;
        D3 no, nd;
        long long absorbed;
        int fate = shade_bounce_hero<INST, SHAPES, MIRROR>(sc, J, queue, f, j, rng, ro, rd, lam, beta, nup, stk, t, rec,
                                                          sub, no, nd, costly, absorbed);
        if (absorbed) tally_add(acc, jobs, multi, j, T_ABS, absorbed);
        if (fate < 0 && ++bounce >= J.max_bounce) fate = 2;
        ro = no; rd = nd;
        if (fate < 0) return true;
        tally_add(acc, jobs, multi, j, fate == 0 ? T_ABS : (fate == 1 ? T_ESC : T_RES),
                  to_fixed(sum_of(beta, nup), J.tally_scale_inv, f.status));
        log_finish(w, in, i, fate, beta[0]);
        return false;
    };
    trace_lanes(w, queue_len(in_count), load, step);
    film_finish();
    tally_finish(acc, jobs, multi, n_jobs);
}

// ------------------------------------------------------------------ host side ----------
void wave_carve(Wave& w, void* block, int32_t W, bool log, int32_t hero) {
    w = Wave{};
    w.W = W;
    w.S = kShadowPerSlot * W;
    w.hero = hero > 1 ? hero : 1;
    w.bytes = wave_bytes(W, log, hero);
    w.block = block;
    char* p = (char*)block;
    auto take = [&](size_t n) { void* r = p; p += wave_align(n); return r; };
    size_t wn = (size_t)W, sn = (size_t)w.S;
    for (PathState& ps : w.ps) {   // path_state_bytes order
        ps.rng_s = (uint64_t*)take(8 * wn); ps.rng_i = (uint64_t*)take(8 * wn);
        ps.ox = (double*)take(8 * wn); ps.oy = (double*)take(8 * wn); ps.oz = (double*)take(8 * wn);
        ps.dx = (double*)take(8 * wn); ps.dy = (double*)take(8 * wn); ps.dz = (double*)take(8 * wn);
        ps.lam = (double*)take(8 * wn); ps.beta = (double*)take(8 * wn); ps.cie = (double*)take(24 * wn);
        ps.stk_n = (int32_t*)take(4 * wn); ps.stk = (int2*)take(8 * wn * kStkCap);
        ps.nbounce = (int32_t*)take(4 * wn); ps.job = (int32_t*)take(4 * wn);
        if (hero > 1) {
            const size_t h = (size_t)hero;
            ps.hlam = (double*)take(8 * wn * h); ps.hbeta = (double*)take(8 * wn * h); ps.hlive = (int32_t*)take(4 * wn);
        }
        if (log) {
            ps.pid = (uint64_t*)take(8 * wn); ps.lhash = (uint64_t*)take(8 * wn);
            ps.lnh = (int32_t*)take(4 * wn); ps.lprims = (int32_t*)take(4 * wn * 8);
        }
    }
    w.hit_t = (double*)take(8 * wn); w.hit_rec = (int32_t*)take(4 * wn); w.hit_sub = (int32_t*)take(4 * wn);
    w.perm = (int32_t*)take(4 * wn);
    w.counts = (int32_t*)take(64);
    w.sjob = (int32_t*)take(4 * sn);
    w.jobs = (DevJob*)take(sizeof(DevJob) * kWaveJobs);
    w.params = (int32_t*)take(64);
    w.ctl = (StreamCtl*)take(64);
    w.sox = (double*)take(8 * sn); w.soy = (double*)take(8 * sn); w.soz = (double*)take(8 * sn);
    w.sdx = (double*)take(8 * sn); w.sdy = (double*)take(8 * sn); w.sdz = (double*)take(8 * sn);
    w.smax = (double*)take(8 * sn); w.sval = (double*)take(8 * sn); w.slam = (double*)take(8 * sn);
    w.sxyz = (double*)take(24 * sn);
    w.spix = (int32_t*)take(4 * sn);
    w.sview = (int32_t*)take(4 * sn);
    if (hero > 1) {
        const size_t h = (size_t)hero;
        w.xlam = (double*)take(8 * sn * (h - 1)); w.xval = (double*)take(8 * sn * (h - 1));
        w.snup = (int32_t*)take(4 * sn);
    }
}

cudaError_t wave_alloc(Wave& w, int32_t W, bool log, int32_t hero) {
    void* block = nullptr;
    cudaError_t e = cudaMalloc(&block, wave_bytes(W, log, hero));
    if (e != cudaSuccess) { w = Wave{}; return e; }
    wave_carve(w, block, W, log, hero);
    return cudaSuccess;
}

void wave_free(Wave& w) {
    if (w.block) cudaFree(w.block);
    w.block = nullptr;
}

// Streaming-pass bookkeeping: both queues and the connection queue empty, nothing handed out.
__global__ void k_stream_init(Wave w) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    StreamCtl& c = *w.ctl;
    c.next = 0; c.taken = 0; c.half = 0; c.more = 1;
    for (int k = 0; k < 16; ++k) w.counts[k] = 0;
}

// End of a half-iteration (one thread): the refill's photons are booked and its paths join
// the queue for the next half-iteration, the consumed queue is emptied (the connection queue
// is by the launch that traces it), and whether work is left for another half-iteration --
// photons not yet handed out, or more than `tail` paths queued -- goes to the progress word
// and, inside a graph, to the loop condition.  A pass that reaches its half-iteration cap
// with such work left stops with ST_LOOP_CAP.
__global__ void k_stream_advance(Wave w, Frame f, int32_t* consumed, int32_t* next_q,
                                 int32_t tail, cudaGraphConditionalHandle loop, int32_t set_loop) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    StreamCtl& c = *w.ctl;
    const int64_t total = reinterpret_cast<const int64_t*>(w.params)[1];
    const int64_t cap = reinterpret_cast<const int64_t*>(w.params)[2];
    const int32_t have = next_q[0];   // survivors at the front; the refill filled the room above them
    const int64_t room = (int64_t)w.params[1] - have - next_q[1], left = total - c.next;
    c.next += left < room ? left : room;
    next_q[0] = have + c.taken;
    c.taken = 0;
    c.half += 1;
    consumed[0] = 0;
    consumed[1] = 0;
    w.counts[kFetchExtend] = 0;
    w.counts[kFetchShade] = 0;
    int32_t more = (queue_len(next_q) > tail || c.next < total) ? 1 : 0;
    if (more && c.half >= cap) {
        atomicOr(f.status, ST_LOOP_CAP);
        more = 0;
    }
    c.more = more;
    if (set_loop) cudaGraphSetConditional(loop, (unsigned)more);
}

// Launchers of the traversal kernels' variants (template template arguments of Issue::trav).
template <bool C, bool I, bool S>
struct LaunchExtend {
    static void go(int grid, cudaStream_t st, Wave w, const DevJob* jobs, PathState in, const int32_t* c,
                   const int32_t* order, Frame f) {
        k_extend<C, I, S><<<grid, 128, 0, st>>>(w, jobs, in, c, order, f);
    }
};
template <bool C, bool I, bool S>
struct LaunchShadow {
    static void go(int grid, cudaStream_t st, Wave w, const DevJob* jobs, Frame f, const int32_t* order) {
        k_shadow<C, I, S, false><<<grid, 128, 0, st>>>(w, jobs, f, order);
    }
};
template <bool C, bool I, bool S>
struct LaunchShadowMirror {
    static void go(int grid, cudaStream_t st, Wave w, const DevJob* jobs, Frame f) {
        k_shadow<C, I, S, true><<<grid, 128, 0, st>>>(w, jobs, f, nullptr);
    }
};
template <bool C, bool I, bool S>
struct LaunchShadowHero {
    static void go(int grid, cudaStream_t st, Wave w, const DevJob* jobs, Frame f) {
        k_shadow_hero<C, I, S, false><<<grid, 128, 0, st>>>(w, jobs, f);
    }
};
template <bool C, bool I, bool S>
struct LaunchShadowHeroMirror {
    static void go(int grid, cudaStream_t st, Wave w, const DevJob* jobs, Frame f) {
        k_shadow_hero<C, I, S, true><<<grid, 128, 0, st>>>(w, jobs, f);
    }
};

namespace {
// Kernel launches of one wave buffer with the variants its WaveKind selects.
struct Issue {
    Wave& w;
    const WaveKind& kind;
    const Frame& f;
    int grid;
    cudaStream_t st;
    LaunchSink* sink;
    int32_t sms;
    static constexpr int T = 128;

    int sort_grid(int entries, int chunk, int per_sm) const {
        return std::max(1, std::min(sms * per_sm, (entries + chunk - 1) / chunk));
    }
    size_t tally() const {   // dynamic shared memory of the tally kernels
        return kTallyRow * (size_t)kind.rows;
    }
    // paths left to the whole-path kernels, which have no counting variant
    int32_t tail() const { return f.stats ? 0 : trace_limit(sms); }

    void mark(int k, bool end) { if (sink) sink->mark(k, end, st); }
    void emit(bool stream, const PathState& out, int32_t* co) {
        mark(K_EMIT, false);
        const DevJob* jobs = w.jobs;
#define FTB_EMIT_HERO(S) \
    (kind.mirrors ? k_emit_hero<S, true><<<grid, T, tally(), st>>>(w, jobs, f, out, co) \
                  : k_emit_hero<S, false><<<grid, T, tally(), st>>>(w, jobs, f, out, co))
#define FTB_EMIT(M, S) \
    (kind.mirrors ? k_emit<M, S, true><<<grid, T, tally(), st>>>(w, jobs, f, out, co) \
                  : k_emit<M, S, false><<<grid, T, tally(), st>>>(w, jobs, f, out, co))
        if (stream) {
            if (kind.bundles) FTB_EMIT_HERO(true);
            else if (kind.media) FTB_EMIT(true, true);
            else FTB_EMIT(false, true);
        } else {
            if (kind.bundles) FTB_EMIT_HERO(false);
            else if (kind.media) FTB_EMIT(true, false);
            else FTB_EMIT(false, false);
        }
#undef FTB_EMIT
#undef FTB_EMIT_HERO
        mark(K_EMIT, true);
    }
    template <template <bool, bool, bool> class K, class... A>
    void trav(A... args) {   // a traversal kernel with the counting / instance / shape variant
        const bool count = f.stats != nullptr, inst = kind.instances, shp = kind.shapes;
        if (count) {
            if (inst) { if (shp) K<true, true, true>::go(grid, st, args...); else K<true, true, false>::go(grid, st, args...); }
            else { if (shp) K<true, false, true>::go(grid, st, args...); else K<true, false, false>::go(grid, st, args...); }
        } else {
            if (inst) { if (shp) K<false, true, true>::go(grid, st, args...); else K<false, true, false>::go(grid, st, args...); }
            else { if (shp) K<false, false, true>::go(grid, st, args...); else K<false, false, false>::go(grid, st, args...); }
        }
    }
    void shadow() {
        mark(K_SHADOW, false);
        if (kind.bundles && kind.mirrors) trav<LaunchShadowHeroMirror>(w, (const DevJob*)w.jobs, f);
        else if (kind.bundles) trav<LaunchShadowHero>(w, (const DevJob*)w.jobs, f);
        else if (kind.mirrors) trav<LaunchShadowMirror>(w, (const DevJob*)w.jobs, f);
        else {
            const int32_t* order = nullptr;
            if (kind.order.connections) {
                // 4-byte positions in an array of 8-byte values that only bundles and mirror
                // connections use
                int32_t* o = reinterpret_cast<int32_t*>(w.slam);
                k_sort_connections<<<sort_grid(w.S, kConnChunk, 16), kConnThreads, 0, st>>>(w, w.jobs, o);
                order = o;
            }
            trav<LaunchShadow>(w, (const DevJob*)w.jobs, f, order);
        }
        mark(K_SHADOW, true);
    }
    void trace(const PathState& in, const int32_t* c) {   // whole paths (booked with closest hit)
        const bool inst = kind.instances, shp = kind.shapes;
        const DevJob* jobs = w.jobs;
        const int g = sms * FTB_TRACE_MINB;
        mark(K_EXTEND, false);
#define FTB_TRACE(...) __VA_ARGS__<<<g, T, tally(), st>>>(w, jobs, f, in, c)
#define FTB_TRACE_SET(...) \
    if (inst) { if (shp) FTB_TRACE(__VA_ARGS__ true, true, false>); else FTB_TRACE(__VA_ARGS__ true, false, false>); } \
    else { if (shp) FTB_TRACE(__VA_ARGS__ false, true, false>); else FTB_TRACE(__VA_ARGS__ false, false, false>); }
        // scenes with planar mirrors share one variant for every kind of record (three builds
        // of the heaviest kernels rather than twelve); the others' exact variants are 15-20 %
        // faster than it on a preview of 2^16 photons (0.26 against 0.31 ms)
        if (kind.mirrors) {
            if (kind.bundles) FTB_TRACE(k_trace_hero<true, true, true>);
            else if (kind.media) FTB_TRACE(k_trace<true, true, true, true>);
            else FTB_TRACE(k_trace<false, true, true, true>);
        } else if (kind.bundles) { FTB_TRACE_SET(k_trace_hero<) }
        else if (kind.media) { FTB_TRACE_SET(k_trace<true,) }
        else { FTB_TRACE_SET(k_trace<false,) }
#undef FTB_TRACE_SET
#undef FTB_TRACE
        mark(K_EXTEND, true);
    }
    void extend(const PathState& in, int32_t* c) {
        mark(K_EXTEND, false);
        const int32_t* order = nullptr;
        if (kind.order.rays) {
            k_sort_queue<<<sort_grid(w.W, kRayChunk, 4), kRayThreads, 0, st>>>(w, w.jobs, in, c, w.perm);
            order = w.perm;
        }
        trav<LaunchExtend>(w, (const DevJob*)w.jobs, in, (const int32_t*)c, order, f);
        mark(K_EXTEND, true);
    }
    void shade(const PathState& in, const int32_t* ci, const PathState& out, int32_t* co) {
        const bool inst = kind.instances, shp = kind.shapes;
        const DevJob* jobs = w.jobs;
        mark(K_SHADE, false);
#define FTB_SHADE(...) __VA_ARGS__<<<grid, T, tally(), st>>>(w, jobs, f, in, ci, out, co)
        if (kind.bundles && kind.mirrors) {
            if (inst) { if (shp) FTB_SHADE(k_shade_hero<true, true, true>); else FTB_SHADE(k_shade_hero<true, false, true>); }
            else { if (shp) FTB_SHADE(k_shade_hero<false, true, true>); else FTB_SHADE(k_shade_hero<false, false, true>); }
        } else if (kind.bundles) {
            if (inst) { if (shp) FTB_SHADE(k_shade_hero<true, true, false>); else FTB_SHADE(k_shade_hero<true, false, false>); }
            else { if (shp) FTB_SHADE(k_shade_hero<false, true, false>); else FTB_SHADE(k_shade_hero<false, false, false>); }
        } else if (kind.mirrors) {
            if (kind.media) {
                if (inst) { if (shp) FTB_SHADE(k_shade<true, true, true, true>); else FTB_SHADE(k_shade<true, true, false, true>); }
                else { if (shp) FTB_SHADE(k_shade<true, false, true, true>); else FTB_SHADE(k_shade<true, false, false, true>); }
            } else {
                if (inst) { if (shp) FTB_SHADE(k_shade<false, true, true, true>); else FTB_SHADE(k_shade<false, true, false, true>); }
                else { if (shp) FTB_SHADE(k_shade<false, false, true, true>); else FTB_SHADE(k_shade<false, false, false, true>); }
            }
        } else if (kind.media) {
            if (inst) { if (shp) FTB_SHADE(k_shade<true, true, true, false>); else FTB_SHADE(k_shade<true, true, false, false>); }
            else { if (shp) FTB_SHADE(k_shade<true, false, true, false>); else FTB_SHADE(k_shade<true, false, false, false>); }
        } else {
            if (inst) { if (shp) FTB_SHADE(k_shade<false, true, true, false>); else FTB_SHADE(k_shade<false, true, false, false>); }
            else { if (shp) FTB_SHADE(k_shade<false, false, true, false>); else FTB_SHADE(k_shade<false, false, false, false>); }
        }
#undef FTB_SHADE
        mark(K_SHADE, true);
    }
};

// The launch sequence of one wave: emit, its connections, then per bounce closest hit,
// shading (survivors compacted into the other path buffer) and the connections it queued.
// Every launch reads the wave's job count and slot count from w.params, so the same
// sequence serves any table (and one captured graph serves every wave of its shape).
void issue_wave(Issue& I, int32_t max_bounce) {
    Wave& w = I.w;
    cudaStream_t st = I.st;
    cudaMemsetAsync(w.counts, 0, 64, st);
    I.emit(false, w.ps[0], queue_counts(w, 0));
    I.shadow();
    cudaMemsetAsync(&w.counts[kShadowCount], 0, 4 * kCountWords, st);
    for (int b = 0; b < max_bounce; ++b) {
        const int a = b & 1;
        I.extend(w.ps[a], queue_counts(w, a));
        cudaMemsetAsync(queue_counts(w, a ^ 1), 0, 8, st);
        I.shade(w.ps[a], queue_counts(w, a), w.ps[a ^ 1], queue_counts(w, a ^ 1));
        I.shadow();
        cudaMemsetAsync(&w.counts[kShadowCount], 0, 4 * kCountWords, st);
    }
}

// A wave of at most trace_limit() slots: emission, then every path to its end.
void issue_wave_paths(Issue& I) {
    Wave& w = I.w;
    cudaMemsetAsync(w.counts, 0, 64, I.st);
    I.emit(false, w.ps[0], queue_counts(w, 0));
    I.trace(w.ps[0], queue_counts(w, 0));
    I.shadow();
}

// A streaming pass: the prologue fills the first queue (ps[0]); a half-iteration traces queue
// `a` and leaves the next one in queue a ^ 1 (the survivors of shading, then the refill).  The
// connections a half-iteration queues are traced by the next one, beside its closest-hit
// launch (on `side` when a graph is captured): neither reads what the other writes, and the
// second launch fills the SMs that the first one's last warps leave idle.  Shading waits for
// both, since it queues connections again.  Against one after the other (B200): preview of
// 2^16 photons 0.495 -> 0.448 ms, fog + strands 119.2 -> 117.3, showroom 28.8 -> 28.1, glass
// bundles 27.4 -> 27.0, served jobs 88.7 -> 85.9.
void stream_prologue(Issue& I) {
    Wave& w = I.w;
    k_stream_init<<<1, 32, 0, I.st>>>(w);
    I.emit(true, w.ps[0], queue_counts(w, 0));
    k_stream_advance<<<1, 32, 0, I.st>>>(w, I.f, queue_counts(w, 1), queue_counts(w, 0), I.tail(), 0, 0);
}
void stream_connections(Issue& I) {
    I.shadow();
    cudaMemsetAsync(&I.w.counts[kShadowCount], 0, 4 * kShadowWords, I.st);
}
struct SideStream {   // a second stream and the events that fork to it and join it
    cudaStream_t st = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    cudaError_t init() {
        if (st) return cudaSuccess;
        cudaError_t e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        return e;
    }
    ~SideStream() {
        if (st) cudaStreamDestroy(st);
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
    }
};
void stream_half(Issue& I, int a, cudaGraphConditionalHandle loop, int32_t set_loop, SideStream* side) {
    Wave& w = I.w;
    if (side) {
        cudaStream_t main = I.st;
        cudaEventRecord(side->fork, main);
        cudaStreamWaitEvent(side->st, side->fork, 0);
        I.st = side->st;
        stream_connections(I);
        I.st = main;
        cudaEventRecord(side->join, side->st);
    } else {
        stream_connections(I);
    }
    I.extend(w.ps[a], queue_counts(w, a));
    if (side) cudaStreamWaitEvent(I.st, side->join, 0);
    I.shade(w.ps[a], queue_counts(w, a), w.ps[a ^ 1], queue_counts(w, a ^ 1));
    I.emit(true, w.ps[a ^ 1], queue_counts(w, a ^ 1));
    k_stream_advance<<<1, 32, 0, I.st>>>(w, I.f, queue_counts(w, a), queue_counts(w, a ^ 1), I.tail(), loop, set_loop);
}
// After the loop: the last half-iteration's connections, the paths still queued (in ps[0]) to
// their ends, and the connections those made.
void stream_tail(Issue& I) {
    stream_connections(I);
    I.trace(I.w.ps[0], queue_counts(I.w, 0));
    I.shadow();
}
// A pass of few photons: all of them emitted (their stream positions are the queue's), then
// every path to its end.
void stream_paths(Issue& I) {
    Wave& w = I.w;
    k_stream_init<<<1, 32, 0, I.st>>>(w);
    I.emit(true, w.ps[0], queue_counts(w, 0));
    k_stream_advance<<<1, 32, 0, I.st>>>(w, I.f, queue_counts(w, 1), queue_counts(w, 0), I.tail(), 0, 0);
    I.trace(w.ps[0], queue_counts(w, 0));
    I.shadow();
}
}  // namespace

struct WaveGraphs {
    struct Entry {
        int32_t max_bounce, grid;   // max_bounce -1: a streaming pass, -2: one of few photons
        WaveKind kind;
        int32_t* status;
        cudaGraphExec_t exec;
    };
    std::vector<Entry> entries;
    SideStream side;            // used while a graph is captured
    ~WaveGraphs() {
        for (auto& e : entries) cudaGraphExecDestroy(e.exec);
    }
    cudaGraphExec_t find(int32_t max_bounce, int32_t grid, const WaveKind& kind, int32_t* status) const {
        for (auto& e : entries)
            if (e.max_bounce == max_bounce && e.grid == grid && e.kind == kind && e.status == status)
                return e.exec;
        return nullptr;
    }
};

WaveGraphs* wave_graphs_create() { return new WaveGraphs(); }
void wave_graphs_destroy(WaveGraphs* g) { delete g; }

namespace {
int launch_grid(const Wave& w, int32_t sms, const LaunchShape& shape) {
    const int T = Issue::T;
    int grid = sms * std::max(1, shape.grid_mult);
    const int gw = (w.W + T - 1) / T;   // enough blocks to give every slot a thread
    if (gw < grid) grid = gw < 1 ? 1 : gw;
    return grid;
}
}  // namespace

int32_t trace_limit(int32_t sms) { return sms * FTB_TRACE_MINB * Issue::T; }

cudaError_t launch_wave(Wave& w, int32_t max_bounce, const WaveKind& kind, const Frame& f, int32_t sms,
                        const LaunchShape& shape, cudaStream_t st, LaunchSink* sink, WaveGraphs* graphs,
                        bool whole_paths) {
    if (kind.bundles && w.hero < 2) return cudaErrorInvalidValue;   // the buffer carries no bundles
    const int grid = launch_grid(w, sms, shape);
    // A graph bakes the kernel arguments: the wave's buffers and status word are fixed for the
    // life of its cache, but a log buffer changes per call, so logging waves launch directly, and
    // so do whole paths (few launches, for a caller without a cache).
    if (!(shape.graph && graphs) || sink || f.stats || w.logs || whole_paths) {
        Issue I{w, kind, f, grid, st, sink, sms};
        if (whole_paths) issue_wave_paths(I);
        else issue_wave(I, max_bounce);
        return cudaGetLastError();
    }
    if (cudaGraphExec_t ex = graphs->find(max_bounce, grid, kind, f.status))
        return cudaGraphLaunch(ex, st);
    cudaGraph_t g = nullptr;
    cudaError_t err = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (err != cudaSuccess) return err;
    Issue I{w, kind, f, grid, st, nullptr, sms};
    issue_wave(I, max_bounce);
    err = cudaStreamEndCapture(st, &g);
    if (err != cudaSuccess) return err;
    WaveGraphs::Entry e{max_bounce, grid, kind, f.status, nullptr};
    err = cudaGraphInstantiate(&e.exec, g, 0);
    cudaGraphDestroy(g);
    if (err != cudaSuccess) return err;
    graphs->entries.push_back(e);
    return cudaGraphLaunch(e.exec, st);
}

cudaError_t launch_stream(Wave& w, int64_t photons, int32_t slots, const WaveKind& kind, const Frame& f, int32_t sms,
                          const LaunchShape& shape, cudaStream_t st, LaunchSink* sink, WaveGraphs* graphs) {
    if (kind.bundles && w.hero < 2) return cudaErrorInvalidValue;
    const int grid = launch_grid(w, sms, shape);
    const bool few = !f.stats && photons <= std::min(slots, trace_limit(sms));
    if (!(shape.graph && graphs) || sink || f.stats || w.logs) {
        // host-driven: the graph's loop body (two half-iterations) at a time, the progress
        // word read after each, so the launches are the ones a graph replay makes
        Issue I{w, kind, f, grid, st, sink, sms};
        if (few) {
            stream_paths(I);
            return cudaGetLastError();
        }
        stream_prologue(I);
        for (;;) {
            cudaError_t e = cudaGetLastError();
            int32_t more = 0;
            if (e == cudaSuccess) e = cudaMemcpyAsync(&more, &w.ctl->more, sizeof more, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return e;
            if (!more) {
                stream_tail(I);
                return cudaGetLastError();
            }
            stream_half(I, 0, 0, 0, nullptr);
            stream_half(I, 1, 0, 0, nullptr);
        }
    }
    const int32_t key = few ? -2 : -1;
    if (cudaGraphExec_t ex = graphs->find(key, grid, kind, f.status)) return cudaGraphLaunch(ex, st);
    // prologue, then a conditional while node whose body is two half-iterations (the queues
    // swap roles between them; the last advance of the body sets the loop condition), then the
    // paths still queued and the connections
    Issue I{w, kind, f, grid, st, nullptr, sms};
    WaveGraphs::Entry entry{key, grid, kind, f.status, nullptr};
    cudaGraph_t g = nullptr;
    cudaError_t err = graphs->side.init();
    if (err != cudaSuccess) return err;
    err = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (err != cudaSuccess) return err;
    if (few) {
        stream_paths(I);
        err = cudaStreamEndCapture(st, &g);
        if (err == cudaSuccess) err = cudaGraphInstantiate(&entry.exec, g, 0);
        if (g) cudaGraphDestroy(g);
        if (err != cudaSuccess) return err;
        graphs->entries.push_back(entry);
        return cudaGraphLaunch(entry.exec, st);
    }
    stream_prologue(I);
    cudaStreamCaptureStatus cs;
    const cudaGraphNode_t* deps = nullptr;
    size_t n_deps = 0;
    cudaGraphConditionalHandle loop = 0;
    cudaGraphNode_t node = nullptr;
    cudaGraphNodeParams p{};
    err = cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &n_deps);
    if (err == cudaSuccess) err = cudaGraphConditionalHandleCreate(&loop, g, 1, cudaGraphCondAssignDefault);
    if (err == cudaSuccess) {
        p.type = cudaGraphNodeTypeConditional;
        p.conditional.handle = loop;
        p.conditional.type = cudaGraphCondTypeWhile;
        p.conditional.size = 1;
        err = cudaGraphAddNode(&node, g, deps, n_deps, &p);
    }
    if (err == cudaSuccess) err = cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies);
    if (err == cudaSuccess) stream_tail(I);
    cudaGraph_t captured = nullptr;
    cudaError_t end = cudaStreamEndCapture(st, &captured);
    if (err == cudaSuccess) err = end;
    if (err != cudaSuccess) {
        if (captured) cudaGraphDestroy(captured);
        return err;
    }
    cudaGraph_t body = p.conditional.phGraph_out[0];
    err = cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    if (err == cudaSuccess) {
        stream_half(I, 0, loop, 0, &graphs->side);
        stream_half(I, 1, loop, 1, &graphs->side);
        cudaGraph_t b2 = nullptr;
        err = cudaStreamEndCapture(st, &b2);
    }
    if (err == cudaSuccess) err = cudaGraphInstantiate(&entry.exec, captured, 0);
    cudaGraphDestroy(captured);
    if (err != cudaSuccess) return err;
    graphs->entries.push_back(entry);
    return cudaGraphLaunch(entry.exec, st);
}

}  // namespace ftb
