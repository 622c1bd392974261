// traverse.cuh - two-level compressed-BVH8 traversal with the watertight triangle test.
//
// Replaces the driver ray query used by ray_hit (src/path_tracing/general.wesl:1053-1078):
// RayDesc(flags 0, cull mask 0xFF, T_MIN, T_MAX, origin, direction), committed closest hit.
// Contract (identical to the CPU oracle's):
//   * hit iff tmin < t < tmax; no face culling; opaque geometry commits without a callback;
//     non-opaque geometry runs the reference's alpha test (general.wesl:1059-1067);
//   * per triangle: Woop-Benthin-Wald watertight test in f32 with this exact operation order
//     (explicit __f*_rn intrinsics, never contracted) and an FP64 recomputation of the three
//     edge functions when any is exactly zero;
//   * ties in t go to the lowest (instance, primitive) pair;
//   * instances are entered with the f32 object-space ray o' = M^-1 o, d' = M^-1 d (fixed fma order).
// The box test evaluates each slab plane as one FMA against the node's quantization grid; the
// far distance is scaled by (1 + 2^-20) and child boxes carry one grid step of outward padding,
// which together cover the f32 rounding of the slab distances.
#pragma once
#include "device_math.cuh"
#include "scene.h"

namespace lam {

constexpr int TRAVERSAL_STACK = 32;
constexpr uint32_t NO_HIT = 0xFFFFFFFFu;
enum : uint32_t { ERR_STACK_OVERFLOW = 1u };

// A ray in the space of one BLAS, as the triangle test reads it.
struct TriRay {
    float3 o;
    int kx, ky, kz;
    float Sx, Sy, Sz;
};

LAM_DEV float sel3(int k, float x, float y, float z) { return k == 0 ? x : (k == 1 ? y : z); }

LAM_DEV float safe_rcp(float x) {
    float y = fabsf(x) < 1e-30f ? copysignf(1e-30f, x) : x;
    // approximate reciprocal (<= 1 ulp): the slab distances only need to be conservative, which the
    // 2^-20 far-distance margin and the one-step box padding guarantee
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    return r;
}

// The dominant axis kz of a direction, and kx, ky chosen so that the winding is kept.
LAM_DEV void dominant_axis(float3 d, int* kx, int* ky, int* kz) {
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    *kz = 0;
    float m = ax;
    if (ay > m) { *kz = 1; m = ay; }
    if (az > m) *kz = 2;
    *kx = *kz + 1 == 3 ? 0 : *kz + 1;
    *ky = *kx + 1 == 3 ? 0 : *kx + 1;
    if (sel3(*kz, d.x, d.y, d.z) < 0.0f) { int t = *kx; *kx = *ky; *ky = t; }
}

LAM_DEV void setup_tri_ray(TriRay& r, float3 o, float3 d) {
    r.o = o;
    dominant_axis(d, &r.kx, &r.ky, &r.kz);
    // shear constants from one IEEE reciprocal (the oracle uses the same three operations); any
    // constants serve, as long as every triangle a ray meets is tested with the same ones
    r.Sz = __fdiv_rn(1.0f, sel3(r.kz, d.x, d.y, d.z));
    r.Sx = __fmul_rn(sel3(r.kx, d.x, d.y, d.z), r.Sz);
    r.Sy = __fmul_rn(sel3(r.ky, d.x, d.y, d.z), r.Sz);
}

LAM_DEV void object_ray(const float* m, float3 o, float3 d, float3* oo, float3* od) {
    oo->x = __fmaf_rn(m[0], o.x, __fmaf_rn(m[1], o.y, __fmaf_rn(m[2], o.z, m[3])));
    oo->y = __fmaf_rn(m[4], o.x, __fmaf_rn(m[5], o.y, __fmaf_rn(m[6], o.z, m[7])));
    oo->z = __fmaf_rn(m[8], o.x, __fmaf_rn(m[9], o.y, __fmaf_rn(m[10], o.z, m[11])));
    od->x = __fmaf_rn(m[0], d.x, __fmaf_rn(m[1], d.y, __fmul_rn(m[2], d.z)));
    od->y = __fmaf_rn(m[4], d.x, __fmaf_rn(m[5], d.y, __fmul_rn(m[6], d.z)));
    od->z = __fmaf_rn(m[8], d.x, __fmaf_rn(m[9], d.y, __fmul_rn(m[10], d.z)));
}

// Watertight test (f32).  Returns true with the IEEE quotient t = T / det when the ray crosses
// the triangle and t could beat `limit` (callers apply the exact tmin / limit / tie rules).
LAM_DEV bool wbw_f32(const TriRay& r, float4 a, float4 b, float4 c, float limit, float* t_out) {
    float Ax0 = __fsub_rn(a.x, r.o.x), Ay0 = __fsub_rn(a.y, r.o.y), Az0 = __fsub_rn(a.z, r.o.z);
    float Bx0 = __fsub_rn(b.x, r.o.x), By0 = __fsub_rn(b.y, r.o.y), Bz0 = __fsub_rn(b.z, r.o.z);
    float Cx0 = __fsub_rn(c.x, r.o.x), Cy0 = __fsub_rn(c.y, r.o.y), Cz0 = __fsub_rn(c.z, r.o.z);
    float Akx = sel3(r.kx, Ax0, Ay0, Az0), Aky = sel3(r.ky, Ax0, Ay0, Az0), Akz = sel3(r.kz, Ax0, Ay0, Az0);
    float Bkx = sel3(r.kx, Bx0, By0, Bz0), Bky = sel3(r.ky, Bx0, By0, Bz0), Bkz = sel3(r.kz, Bx0, By0, Bz0);
    float Ckx = sel3(r.kx, Cx0, Cy0, Cz0), Cky = sel3(r.ky, Cx0, Cy0, Cz0), Ckz = sel3(r.kz, Cx0, Cy0, Cz0);
    float Ax = __fmaf_rn(-r.Sx, Akz, Akx), Ay = __fmaf_rn(-r.Sy, Akz, Aky);
    float Bx = __fmaf_rn(-r.Sx, Bkz, Bkx), By = __fmaf_rn(-r.Sy, Bkz, Bky);
    float Cx = __fmaf_rn(-r.Sx, Ckz, Ckx), Cy = __fmaf_rn(-r.Sy, Ckz, Cky);
    float U = __fmaf_rn(Cx, By, -__fmul_rn(Cy, Bx));
    float V = __fmaf_rn(Ax, Cy, -__fmul_rn(Ay, Cx));
    float W = __fmaf_rn(Bx, Ay, -__fmul_rn(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = __double2float_rn(__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx)));
        V = __double2float_rn(__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx)));
        W = __double2float_rn(__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax)));
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    float Az = __fmul_rn(r.Sz, Akz), Bz = __fmul_rn(r.Sz, Bkz), Cz = __fmul_rn(r.Sz, Ckz);
    float T = __fmaf_rn(U, Az, __fmaf_rn(V, Bz, __fmul_rn(W, Cz)));
    // conservative early out: |T / det| certainly above the current limit
    if (fabsf(T) > __fmul_rn(fabsf(det), limit) * 1.00000095367431640625f) return false;
    *t_out = __fdiv_rn(T, det);
    return true;
}

// a / b rounded to nearest from b's rounded reciprocal: the quotient estimate is corrected twice by its
// exact residual (P. Markstein, IBM J. R&D 34, 1990).  For |a| <= |b| that came from f32, whose quotients
// and residuals stay far inside the FP64 range; a zero keeps the sign that the first product gives, and so
// does the zero over an infinite b, whose residual is taken with 0 for b (with b it would be NaN).
LAM_DEV double quotient_f64(double a, double b, double rcp_b) {
    const int hi = __double2hiint(b);
    const double br = __hiloint2double((hi & 0x7FF00000) == 0x7FF00000 ? 0 : hi, __double2loint(b));
    const double q0 = __dmul_rn(a, rcp_b);
    const double q1 = __fma_rn(__fma_rn(-br, q0, a), rcp_b, q0);
    const double q2 = __fma_rn(__fma_rn(-br, q1, a), rcp_b, q1);
    return a == 0.0 ? q0 : q2;
}

// FP64 re-evaluation of the committed hit (same formulas as the oracle, never contracted).
LAM_DEV void wbw_f64(float3 of, float3 df, float4 p0, float4 p1, float4 p2, float* t, float* u, float* v,
                     bool* front) {
    int kx, ky, kz;
    dominant_axis(df, &kx, &ky, &kz);
    double o[3] = {of.x, of.y, of.z}, d[3] = {df.x, df.y, df.z};
    double P0[3] = {p0.x, p0.y, p0.z}, P1[3] = {p1.x, p1.y, p1.z}, P2[3] = {p2.x, p2.y, p2.z};
    double a[3], b[3], c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a[k] = __dsub_rn(P0[k], o[k]);
        b[k] = __dsub_rn(P1[k], o[k]);
        c[k] = __dsub_rn(P2[k], o[k]);
    }
    double dkx = kx == 0 ? d[0] : (kx == 1 ? d[1] : d[2]);
    double dky = ky == 0 ? d[0] : (ky == 1 ? d[1] : d[2]);
    double dkz = kz == 0 ? d[0] : (kz == 1 ? d[1] : d[2]);
    auto pick = [&](const double* q, int k) { return k == 0 ? q[0] : (k == 1 ? q[1] : q[2]); };
    const double Sz = __ddiv_rn(1.0, dkz), Sx = quotient_f64(dkx, dkz, Sz), Sy = quotient_f64(dky, dkz, Sz);
    double Ax = __dsub_rn(pick(a, kx), __dmul_rn(Sx, pick(a, kz))), Ay = __dsub_rn(pick(a, ky), __dmul_rn(Sy, pick(a, kz)));
    double Bx = __dsub_rn(pick(b, kx), __dmul_rn(Sx, pick(b, kz))), By = __dsub_rn(pick(b, ky), __dmul_rn(Sy, pick(b, kz)));
    double Cx = __dsub_rn(pick(c, kx), __dmul_rn(Sx, pick(c, kz))), Cy = __dsub_rn(pick(c, ky), __dmul_rn(Sy, pick(c, kz)));
    double U = __dsub_rn(__dmul_rn(Cx, By), __dmul_rn(Cy, Bx));
    double V = __dsub_rn(__dmul_rn(Ax, Cy), __dmul_rn(Ay, Cx));
    double W = __dsub_rn(__dmul_rn(Bx, Ay), __dmul_rn(By, Ax));
    double det = __dadd_rn(__dadd_rn(U, V), W);
    double Az = __dmul_rn(Sz, pick(a, kz)), Bz = __dmul_rn(Sz, pick(b, kz)), Cz = __dmul_rn(Sz, pick(c, kz));
    double T = __dadd_rn(__dadd_rn(__dmul_rn(U, Az), __dmul_rn(V, Bz)), __dmul_rn(W, Cz));
    *t = __double2float_rn(__ddiv_rn(T, det));
    *u = __double2float_rn(__ddiv_rn(V, det));
    *v = __double2float_rn(__ddiv_rn(W, det));
    double e1[3] = {__dsub_rn(P1[0], P0[0]), __dsub_rn(P1[1], P0[1]), __dsub_rn(P1[2], P0[2])};
    double e2[3] = {__dsub_rn(P2[0], P0[0]), __dsub_rn(P2[1], P0[1]), __dsub_rn(P2[2], P0[2])};
    double n0 = __dsub_rn(__dmul_rn(e1[1], e2[2]), __dmul_rn(e1[2], e2[1]));
    double n1 = __dsub_rn(__dmul_rn(e1[2], e2[0]), __dmul_rn(e1[0], e2[2]));
    double n2 = __dsub_rn(__dmul_rn(e1[0], e2[1]), __dmul_rn(e1[1], e2[0]));
    double nd = __dadd_rn(__dadd_rn(__dmul_rn(n0, d[0]), __dmul_rn(n1, d[1])), __dmul_rn(n2, d[2]));
    *front = nd < 0.0;
}

// Byte k of w as the float 1 + byte * 2^-15 (the byte in mantissa bits 8..15 of 1.0f): one byte
// permute turns a quantized child coordinate into an exact float.
LAM_DEV float qone(uint32_t w, uint32_t k) {
    return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u + (k << 4)));
}

// Pairs of floats for the packed FMA.
LAM_DEV uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
LAM_DEV uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
LAM_DEV float half2f(uint64_t v, uint32_t e) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return e ? b : a;
}

// Intersects the 8 children of one node.  Outputs the node group (child_base, internal hits in
// bits 24..31 in octant order | imask) and the leaf group (leaf_base, item hits in bits 0..23).
LAM_DEV void intersect_node(const uint4* __restrict__ np, float3 o, float3 inv, uint32_t oct, float tmin, float tmax,
                            uint2& ng, uint2& tg) {
    const uint4 n0 = ld_keep(np), n1 = ld_keep(np + 1), n2 = ld_keep(np + 2), n3 = ld_keep(np + 3), n4 = ld_keep(np + 4);
    const float px = __uint_as_float(n0.x), py = __uint_as_float(n0.y), pz = __uint_as_float(n0.z);
    const uint32_t imask = n0.w >> 24;
    const float sx = __uint_as_float((n0.w & 0xFFu) << 23);
    const float sy = __uint_as_float(((n0.w >> 8) & 0xFFu) << 23);
    const float sz = __uint_as_float(((n0.w >> 16) & 0xFFu) << 23);
    const float adx = __fmul_rn(sx, inv.x), ady = __fmul_rn(sy, inv.y), adz = __fmul_rn(sz, inv.z);
    const float aox = __fmul_rn(__fsub_rn(px, o.x), inv.x);
    const float aoy = __fmul_rn(__fsub_rn(py, o.y), inv.y);
    const float aoz = __fmul_rn(__fsub_rn(pz, o.z), inv.z);
    // near plane = lo plane when the inverse direction is positive
    const bool fx = inv.x < 0.0f, fy = inv.y < 0.0f, fz = inv.z < 0.0f;
    const uint32_t nx0 = fx ? n3.z : n2.x, nx1 = fx ? n3.w : n2.y, fx0 = fx ? n2.x : n3.z, fx1 = fx ? n2.y : n3.w;
    const uint32_t ny0 = fy ? n4.x : n2.z, ny1 = fy ? n4.y : n2.w, fy0 = fy ? n2.z : n4.x, fy1 = fy ? n2.w : n4.y;
    const uint32_t nz0 = fz ? n4.z : n3.x, nz1 = fz ? n4.w : n3.y, fz0 = fz ? n3.x : n4.z, fz1 = fz ? n3.y : n4.w;
    // Hit-mask contribution of each slot, four slots per word: bits (bits 5..7 of meta, unary) at
    // position `at` (bits 0..4; internal children sit at 24 + slot, which is XORed with the octant).
    // A byte is internal when its position is 24..31 (bits 3 and 4 set); bit 0 of each byte of
    // inner_* flags it, so inner_* * oct holds the octant in exactly the internal bytes.
    const uint32_t ma = n1.z, mb = n1.w;
    const uint32_t inner_a = ((ma & (ma << 1)) >> 4) & 0x01010101u, inner_b = ((mb & (mb << 1)) >> 4) & 0x01010101u;
    const uint32_t at_a = (ma ^ (inner_a * oct)) & 0x1F1F1F1Fu, at_b = (mb ^ (inner_b * oct)) & 0x1F1F1F1Fu;
    const uint32_t bits_a = (ma >> 5) & 0x07070707u, bits_b = (mb >> 5) & 0x07070707u;
    uint32_t hits = 0u;
    // t = q * adx + aox with q read as 1 + q * 2^-15: t = (1 + q * 2^-15) * (2^15 adx) + (aox - 2^15 adx).
    // Rounding B adds at most 2^-9 of a grid step (plus 2^-24 |aox|) to each plane distance, far inside
    // the builder's one-step outward padding and the 2^-20 far-plane margin.  This saves the
    // subtraction of an integer-to-float conversion per plane.  Should 2^15 adx overflow, the plane
    // distance is NaN, which fmaxf / fminf ignore: the test only becomes more permissive.
    const float Ax = 32768.0f * adx, Ay = 32768.0f * ady, Az = 32768.0f * adz;
    const float Bx = __fmaf_rn(-32768.0f, adx, aox), By = __fmaf_rn(-32768.0f, ady, aoy),
                Bz = __fmaf_rn(-32768.0f, adz, aoz);
    // two children per packed FMA: the loop is bound by issue (icosphere field 78.0 -> 74.9 ms a frame)
    const uint64_t A2x = pack2(Ax, Ax), A2y = pack2(Ay, Ay), A2z = pack2(Az, Az);
    const uint64_t B2x = pack2(Bx, Bx), B2y = pack2(By, By), B2z = pack2(Bz, Bz);
#pragma unroll
    for (uint32_t i = 0; i < 8; i += 2) {
        const uint32_t k = i & 3u;
        const uint64_t nx2 = fma2(pack2(qone(i < 4 ? nx0 : nx1, k), qone(i < 4 ? nx0 : nx1, k + 1)), A2x, B2x);
        const uint64_t ny2 = fma2(pack2(qone(i < 4 ? ny0 : ny1, k), qone(i < 4 ? ny0 : ny1, k + 1)), A2y, B2y);
        const uint64_t nz2 = fma2(pack2(qone(i < 4 ? nz0 : nz1, k), qone(i < 4 ? nz0 : nz1, k + 1)), A2z, B2z);
        const uint64_t fx2 = fma2(pack2(qone(i < 4 ? fx0 : fx1, k), qone(i < 4 ? fx0 : fx1, k + 1)), A2x, B2x);
        const uint64_t fy2 = fma2(pack2(qone(i < 4 ? fy0 : fy1, k), qone(i < 4 ? fy0 : fy1, k + 1)), A2y, B2y);
        const uint64_t fz2 = fma2(pack2(qone(i < 4 ? fz0 : fz1, k), qone(i < 4 ? fz0 : fz1, k + 1)), A2z, B2z);
#pragma unroll
        for (uint32_t e = 0; e < 2; ++e) {
            const float tn = fmaxf(fmaxf(half2f(nx2, e), half2f(ny2, e)), fmaxf(half2f(nz2, e), tmin));
            const float tf = fminf(fminf(half2f(fx2, e), half2f(fy2, e)), fminf(half2f(fz2, e), tmax));
            if (tn <= tf * 1.00000095367431640625f)
                hits |= __byte_perm(i < 4 ? bits_a : bits_b, 0u, 0x4440u + k + e) << __byte_perm(i < 4 ? at_a : at_b, 0u, 0x4440u + k + e);
        }
    }
    ng = make_uint2(n1.x, (hits & 0xFF000000u) | imask);
    tg = make_uint2(n1.y, hits & 0x00FFFFFFu);
}

struct TraceResult {
    uint32_t tri;   // global triangle slot, NO_HIT if none
    uint32_t inst;
    float t;        // f32 watertight distance
#ifdef LAM_HAVE_HANDLER
    float3 pn, ptg; // normal and tangent of a committed procedural hit (from the handler)
#endif
};

}  // namespace lam
#ifdef LAM_HAVE_HANDLER
// The intersection handler, linked in at run time (lam_tracer_set_intersection_handler).
extern "C" __device__ lam_aabb_intersection lam_user_intersect(const lam_ray_intersection& i);
#endif
namespace lam {

// Conservative ray / box test in the ray's own space (procedural candidates reach the handler only
// when the ray crosses their box inside (tmin, limit), as the driver's AABB candidates do).
LAM_DEV bool ray_box(float3 o, float3 inv, float4 lo, float4 hi, float tmin, float limit) {
    const float tx0 = (lo.x - o.x) * inv.x, tx1 = (hi.x - o.x) * inv.x;
    const float ty0 = (lo.y - o.y) * inv.y, ty1 = (hi.y - o.y) * inv.y;
    const float tz0 = (lo.z - o.z) * inv.z, tz1 = (hi.z - o.z) * inv.z;
    const float tn = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fmaxf(fminf(tz0, tz1), tmin));
    const float tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fminf(fmaxf(tz0, tz1), limit));
    return tn <= tf * 1.00000095367431640625f;
}

enum : int { STEP_MORE = 0, STEP_DONE = 1, STEP_COOP = 2 };

// Per-warp shared memory of a traversal, one slot per lane.  The loop is bound by instruction issue, of
// which the triangle phase and the instance entries and exits took more than half.  So a ray's world
// form is written once and its form in the space of a BLAS when an instance is entered, instead of by
// all 32 lanes in every phase; an exit reads the former back; neither is held in registers (72 instead
// of 80: seven CTAs per SM); and the owners list their triangles instead of every tester searching for
// its owner.  Icosphere field, 1080p, 16 spp: 87.1 -> 78.3 ms a frame.
constexpr uint32_t COOP_LIST = 256;
template <bool MULTI>
struct CoopScenes {
    const DevScene* scene[32];  // lanes of one warp trace different scenes
};
template <>
struct CoopScenes<false> {};
template <bool MULTI>
struct CoopScratch : CoopScenes<MULTI> {
    float4 world_o[32];         // origin, tmin
    float4 world_d[32];         // direction
    float4 ray_o[32];           // origin in the instance's space, Sx
    float4 ray_s[32];           // Sy, Sz, kx | ky << 2 | kz << 4, distance limit of the phase
    unsigned long long key[32];
    uint32_t base[32], inst[32], item[32];
    uint32_t total;
    uint16_t list[COOP_LIST];   // tests of the phase: owner lane | triangle's bit << 5
};

// Alpha-test callback for non-opaque geometry: candidate accepted unless the diffuse texel's
// alpha is near zero, transparent materials always accepted (general.wesl:1059-1067).
LAM_DEV bool alpha_accept(const DevScene& S, uint32_t inst, uint32_t prim, float bu, float bv, bool transparent_passes);

// Resumable traversal: init() then step() until it returns false.  One step intersects one node
// and tests the leaf items it exposes, so a warp can refill lanes whose rays have finished
// (after Aila and Laine, "Understanding the Efficiency of Ray Traversal on GPUs", HPG 2009).
template <bool ANY, bool ALPHA, bool MULTI = false>
struct Traverser {
    typedef CoopScratch<MULTI> Scratch;
    // the ray of the current level, as box tests read it: world space in the TLAS, object space in a
    // BLAS.  (Shear constants are only computed for the latter: the TLAS holds no triangles.)
    float3 o, inv;
    uint32_t oct;
    float tmin, best_t;
    uint2 ng, tg;
    int sp, blas_base;
    uint32_t cur_inst, cur_flags;
    TraceResult res;
    bool transparent_passes = true;  // transparent materials pass the alpha test (path shaders)

    LAM_DEV void set_ray(float3 org, float3 d) {
        o = org;
        inv = make_float3(safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z));
        oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    }

    LAM_DEV void init(const DevScene& S, Scratch& ws, float3 org, float3 d, float t0, float t1) {
        const uint32_t lane = threadIdx.x & 31u;
        ws.world_o[lane] = make_float4(org.x, org.y, org.z, t0);
        ws.world_d[lane] = make_float4(d.x, d.y, d.z, 0.0f);
        tmin = t0;
        best_t = t1;
        res.tri = NO_HIT;
        res.inst = NO_HIT;
        sp = 0;
        blas_base = -1;
        cur_inst = 0u;
        cur_flags = 0u;
        set_ray(org, d);
        ng = S.tlas_node_count ? make_uint2(S.tlas_root, (1u << (24u + oct)) | 1u) : make_uint2(0u, 0u);
        tg = make_uint2(0u, 0u);
    }

    LAM_DEV void push(uint2* stack, uint2 g, uint32_t& err) {
        if (sp < TRAVERSAL_STACK) stack[sp++] = g;
        else err |= ERR_STACK_OVERFLOW;
    }

    // Whether a candidate (t, primitive of the current instance) replaces the committed hit: closer, or
    // as close with a lower (instance, primitive).  The committed primitive is only read on a tie.
    LAM_DEV bool replaces(const float4* tris, float t, uint32_t prim) const {
        if (t < best_t) return true;
        if (!(t == best_t) || res.tri == NO_HIT || cur_inst > res.inst) return false;
        return cur_inst < res.inst || prim < __float_as_uint(ld_keep(tris + 3u * res.tri).w);
    }

    // One traversal step: one node, then the leaf items it exposes.  Returns STEP_MORE, STEP_DONE
    // (res is final), or, with COOP, STEP_COOP when the exposed items are triangles: they are left in
    // tg for the warp's shared triangle phase (coop_triangles), after which finish_coop() completes
    // the step.  `stack` holds TRAVERSAL_STACK entries owned by this lane (kept outside the struct so
    // that the struct itself stays in registers).
    template <bool COOP>
    LAM_DEV int step_impl(const DevScene& S, const DevInstance* __restrict__ insts, uint2* stack, Scratch& ws,
                          uint32_t& err) {
        const uint32_t lane = threadIdx.x & 31u;
        if (ng.y > 0x00FFFFFFu) {
            const uint32_t k = __ffs(ng.y >> 24) - 1u;
            ng.y &= ~(1u << (24u + k));
            const uint32_t slot = k ^ oct;
            const uint32_t child = ng.x + __popc(ng.y & ((1u << slot) - 1u) & 0xFFu);
            if (ng.y > 0x00FFFFFFu) push(stack, ng, err);
            // one call site and one array for TLAS and BLAS nodes: lanes of a warp on either level share
            // one test (two call sites run the 8-wide test twice whenever a warp straddles the levels)
            intersect_node(S.nodes + 5u * child, o, inv, oct, tmin, best_t, ng, tg);
        } else {
            tg = ng;
            ng = make_uint2(0u, 0u);
        }
        if (COOP && blas_base >= 0 && tg.y != 0u && !(cur_flags & INST_PROCEDURAL)) return STEP_COOP;
        while (tg.y != 0u) {
            const uint32_t k = __ffs(tg.y) - 1u;
            tg.y &= tg.y - 1u;
            const uint32_t item = tg.x + k;
            if (blas_base < 0) {
                const uint32_t id = __ldg(S.tlas_items + item);
                const DevInstance& I = insts[id];
                const uint32_t flags = I.flags;
                const uint32_t root = I.blas_root;
                if (!(flags & INST_VISIBLE) || root == NO_HIT) continue;
                if (tg.y != 0u) push(stack, tg, err);
                if (ng.y > 0x00FFFFFFu) push(stack, ng, err);
                blas_base = sp;
                cur_inst = id;
                cur_flags = flags;
                float m[12];
#pragma unroll
                for (int q = 0; q < 12; ++q) m[q] = I.inv[q];
                const float4 w_o = ws.world_o[lane], w_d = ws.world_d[lane];
                float3 oo, od;
                object_ray(m, make_float3(w_o.x, w_o.y, w_o.z), make_float3(w_d.x, w_d.y, w_d.z), &oo, &od);
                set_ray(oo, od);
                TriRay r;
                setup_tri_ray(r, oo, od);
                ws.ray_o[lane] = make_float4(oo.x, oo.y, oo.z, r.Sx);
                ws.ray_s[lane] = make_float4(
                    r.Sy, r.Sz, __uint_as_float((uint32_t)r.kx | ((uint32_t)r.ky << 2) | ((uint32_t)r.kz << 4)), 0.0f);
                if (ALPHA) ws.inst[lane] = (flags & INST_OPAQUE) ? NO_HIT : id;  // the alpha test's instance
                ng = make_uint2(root, (1u << (24u + oct)) | 1u);
                tg = make_uint2(0u, 0u);
                return STEP_MORE;
            }
            const float4* tp = S.tris + 3u * item;
            if (cur_flags & INST_PROCEDURAL) {
#ifdef LAM_HAVE_HANDLER
                const float4 lo = __ldg(tp), hi = __ldg(tp + 1);
                if (!ray_box(o, inv, lo, hi, tmin, best_t)) continue;
                const uint32_t prim = __float_as_uint(lo.w);
                const float4 w_o = ws.world_o[lane], w_d = ws.world_d[lane];
                float3 oo, od;
                object_ray(insts[cur_inst].inv, make_float3(w_o.x, w_o.y, w_o.z), make_float3(w_d.x, w_d.y, w_d.z), &oo, &od);
                lam_ray_intersection ri;
                ri.kind = LAM_INTERSECTION_AABB;
                ri.t = best_t;
                const float* fw = S.inst_fwd + 16u * cur_inst;
                ri.instance_custom_data = __float_as_uint(fw[12]);
                ri.instance_index = cur_inst;
                ri.sbt_record_offset = 0u;
                ri.geometry_index = 0u;
                ri.primitive_index = prim;
                ri.barycentrics[0] = 0.0f;
                ri.barycentrics[1] = 0.0f;
                ri.front_face = 0u;
#pragma unroll
                for (int q = 0; q < 12; ++q) {
                    ri.object_to_world[q] = fw[q];
                    ri.world_to_object[q] = insts[cur_inst].inv[q];
                }
                ri.world_origin[0] = w_o.x; ri.world_origin[1] = w_o.y; ri.world_origin[2] = w_o.z;
                ri.world_direction[0] = w_d.x; ri.world_direction[1] = w_d.y; ri.world_direction[2] = w_d.z;
                ri.object_origin[0] = oo.x; ri.object_origin[1] = oo.y; ri.object_origin[2] = oo.z;
                ri.object_direction[0] = od.x; ri.object_direction[1] = od.y; ri.object_direction[2] = od.z;
                ri.tmin = tmin;
                ri.aabb_min[0] = lo.x; ri.aabb_min[1] = lo.y; ri.aabb_min[2] = lo.z;
                ri.aabb_max[0] = hi.x; ri.aabb_max[1] = hi.y; ri.aabb_max[2] = hi.z;
                const lam_aabb_intersection ai = lam_user_intersect(ri);
                const float t = ai.t;
                if (!(ai.hit && t > tmin && replaces(S.tris, t, prim))) continue;
                best_t = t;
                res.tri = item;
                res.inst = cur_inst;
                res.pn = make_float3(ai.normal[0], ai.normal[1], ai.normal[2]);
                res.ptg = make_float3(ai.tangent[0], ai.tangent[1], ai.tangent[2]);
                if (ANY) {
                    res.t = best_t;
                    return STEP_DONE;
                }
#endif
                continue;
            }
            if (COOP) continue;  // not reached: triangles go to the cooperative phase
            const float4 a = ld_keep(tp), b = ld_keep(tp + 1), c = ld_keep(tp + 2);
            float t;
            if (!wbw_f32(tri_ray(ws, lane), a, b, c, best_t, &t)) continue;
            const uint32_t prim = __float_as_uint(a.w);
            if (!(t > tmin && replaces(S.tris, t, prim))) continue;
            if (ALPHA && !(cur_flags & INST_OPAQUE) &&
                !passes_alpha(S, insts, ws, lane, cur_inst, prim, a, b, c, transparent_passes))
                continue;
            best_t = t;
            res.tri = item;
            res.inst = cur_inst;
            if (ANY) {
                res.t = best_t;
                return STEP_DONE;
            }
        }
        return tail(stack, ws) ? STEP_MORE : STEP_DONE;
    }

    // Returns false once the traversal has finished (res is final).
    LAM_DEV bool step(const DevScene& S, const DevInstance* __restrict__ insts, uint2* stack, Scratch& ws, uint32_t& err) {
        return step_impl<false>(S, insts, stack, ws, err) == STEP_MORE;
    }

    // End of a step: leave a finished instance, pop the next group; false when the ray is done.
    LAM_DEV bool tail(uint2* stack, Scratch& ws) {
        if (ng.y <= 0x00FFFFFFu) {
            if (blas_base >= 0 && sp == blas_base) {
                blas_base = -1;
                const uint32_t lane = threadIdx.x & 31u;
                const float4 w_o = ws.world_o[lane], w_d = ws.world_d[lane];
                set_ray(make_float3(w_o.x, w_o.y, w_o.z), make_float3(w_d.x, w_d.y, w_d.z));
            }
            if (sp == 0) {
                res.t = best_t;
                return false;
            }
            ng = stack[--sp];
        }
        return true;
    }

    // Completes a STEP_COOP step once the warp has tested this lane's triangles.
    LAM_DEV bool finish_coop(uint2* stack, Scratch& ws, bool hit_now) {
        if (ANY && hit_now) {
            res.t = best_t;
            return false;
        }
        return tail(stack, ws);
    }

    LAM_DEV static TriRay tri_ray(const Scratch& ws, uint32_t owner) {
        const float4 a = ws.ray_o[owner], b = ws.ray_s[owner];
        const uint32_t pm = __float_as_uint(b.z);
        TriRay r;
        r.o = make_float3(a.x, a.y, a.z);
        r.Sx = a.w;
        r.Sy = b.x;
        r.Sz = b.y;
        r.kx = (int)(pm & 3u);
        r.ky = (int)((pm >> 2) & 3u);
        r.kz = (int)(pm >> 4);
        return r;
    }

    // The alpha test of lane `owner`'s candidate, at its FP64 barycentrics.
    LAM_DEV static bool passes_alpha(const DevScene& S, const DevInstance* insts, const Scratch& ws, uint32_t owner,
                                     uint32_t inst, uint32_t prim, float4 a, float4 b, float4 c, bool transparent_passes) {
        const float4 w_o = ws.world_o[owner], w_d = ws.world_d[owner];
        float m[12];
#pragma unroll
        for (int q = 0; q < 12; ++q) m[q] = insts[inst].inv[q];
        float3 oo, od;
        object_ray(m, make_float3(w_o.x, w_o.y, w_o.z), make_float3(w_d.x, w_d.y, w_d.z), &oo, &od);
        float t, u, v;
        bool front;
        wbw_f64(oo, od, a, b, c, &t, &u, &v, &front);
        return alpha_accept(S, inst, prim, u, v, transparent_passes);
    }

    // The warp's shared triangle phase: every lane of the warp takes part.  The pending triangles
    // (tg) of the lanes with `want` are listed in shared memory and dealt out over all 32 lanes; each
    // tester runs the watertight test against its owner's ray, and the alpha test of a triangle that
    // is not opaque, and folds (t, primitive) into the owner's slot with a 64-bit shared-memory
    // atomic minimum.  The owner then commits the minimum under the same rules as the serial loop
    // (closest, ties to the lowest (instance, primitive)), so results are bit-identical.  An any-hit
    // query of an instance that is not opaque takes the first accepted triangle in order, as the
    // serial loop does.  (617x349, 4 spp of a box of cutouts: 1.39 ms with alpha-tested triangles in the
    // per-lane loop, 1.09 here.)  Returns whether this lane committed a new hit.
    LAM_DEV bool coop_triangles(bool want, const DevScene& S0, const DevInstance* insts0, Scratch& ws) {
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t todo = 0u;
        if (want) {
            todo = tg.y;
            ws.base[lane] = tg.x;
            ws.ray_s[lane].w = best_t;
            ws.key[lane] = ~0ull;
        }
        for (;;) {
            if (todo) {
                uint32_t pos = atomicAdd(&ws.total, (uint32_t)__popc(todo));
                while (todo && pos < COOP_LIST) {
                    ws.list[pos++] = (uint16_t)(lane | ((__ffs(todo) - 1u) << 5));
                    todo &= todo - 1u;
                }
            }
            __syncwarp();
            const uint32_t total = min(ws.total, COOP_LIST);
            for (uint32_t j = lane; j - lane < total; j += 32u) {
                bool has = false;
                unsigned long long key = 0ull;
                uint32_t owner = 0u, item = 0u;
                if (j < total) {
                    const uint32_t e = ws.list[j];
                    owner = e & 31u;
                    item = ws.base[owner] + (e >> 5);
                    const float4* tris = S0.tris;
                    if constexpr (MULTI) tris = ws.scene[owner]->tris;
                    const float4* tp = tris + 3u * item;
                    const float4 a = ld_keep(tp), b = ld_keep(tp + 1), c = ld_keep(tp + 2);
                    float t;
                    if (wbw_f32(tri_ray(ws, owner), a, b, c, ws.ray_s[owner].w, &t) && t > ws.world_o[owner].w) {
                        const uint32_t u = __float_as_uint(t);
                        const uint32_t ord = (u & 0x80000000u) ? ~u : (u | 0x80000000u);  // float order as unsigned
                        key = ((unsigned long long)ord << 32) | __float_as_uint(a.w);
                        has = true;
                        if (ALPHA) {
                            const uint32_t inst = ws.inst[owner];
                            if (inst != NO_HIT) {
                                if constexpr (MULTI)
                                    has = passes_alpha(*ws.scene[owner], ws.scene[owner]->inst, ws, owner, inst,
                                                       __float_as_uint(a.w), a, b, c, true);
                                else
                                    has = passes_alpha(S0, insts0, ws, owner, inst, __float_as_uint(a.w), a, b, c, true);
                                // any hit: only a candidate within the limit counts, and the order decides
                                if (ANY) {
                                    has = has && t < ws.ray_s[owner].w;
                                    key = ((unsigned long long)(e >> 5) << 32) | u;
                                }
                            }
                        }
                        if (has) atomicMin(&ws.key[owner], key);
                    }
                }
                __syncwarp();
                if (has && key == ws.key[owner]) ws.item[owner] = item;  // (t, primitive) names one triangle
                __syncwarp();
            }
            if (lane == 0u) ws.total = 0u;
            __syncwarp();
            if (!__any_sync(0xFFFFFFFFu, todo != 0u)) break;
        }
        bool hit_now = false;
        if (want) {
            const unsigned long long key = ws.key[lane];
            if (key != ~0ull) {
                const uint32_t ord = (uint32_t)(key >> 32);
                float t = __uint_as_float((ord & 0x80000000u) ? (ord & 0x7FFFFFFFu) : ~ord);
                const float4* tris = S0.tris;
                if constexpr (MULTI) tris = ws.scene[lane]->tris;
                bool better;
                if (ALPHA && ANY && !(cur_flags & INST_OPAQUE)) {
                    t = __uint_as_float((uint32_t)key);
                    better = true;
                } else {
                    better = replaces(tris, t, (uint32_t)key);
                }
                if (better) {
                    best_t = t;
                    res.tri = ws.item[lane];
                    res.inst = cur_inst;
                    hit_now = true;
                }
            }
            tg.y = 0u;
        }
        __syncwarp();
        return hit_now;
    }
};

// Lanes below this many active rays trigger a refill of the idle lanes from the work queue.
constexpr int REFILL_THRESHOLD = 26;  // 24..30 within 2%: 26 / 28 / 30 take 1,773 / 1,801 / 1,868 us for 4.2M rays
constexpr uint32_t SMALL_WARPS = 8;  // per SM, see trace_persistent

// Persistent warp loop over work items [0, n) claimed with a global counter.  `load(i, o, d, t0, t1)`
// fetches item i; `store(i, res)` consumes a finished traversal.  Every lane of the warp must call it,
// in blocks of 128 threads.  Triangle tests are dealt out over the whole warp
// (Traverser::coop_triangles): with one ray per lane, a step exposes 0 to 24 triangles per lane, and
// a per-lane loop would run as long as the busiest lane.
// With MULTI the items belong to different scenes: `load(i, o, d, t0, t1, sp)` also returns the item's
// scene, whose TLAS and instances are read from global memory.
template <bool ANY, bool ALPHA, bool MULTI = false, class Load, class Store>
LAM_DEV void trace_persistent(const DevScene& S0, const DevInstance* __restrict__ in, uint32_t n,
                              uint32_t* __restrict__ work, uint32_t& err, Load load, Store store) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    __shared__ CoopScratch<MULTI> coop_ws[4];  // one per warp of a 128-thread block
    CoopScratch<MULTI>& ws = coop_ws[(threadIdx.x >> 5) & 3u];
    if (lane == 0u) ws.total = 0u;
    __syncwarp();
    // A queue that cannot fill the chip is spread over SMALL_WARPS warps per SM: a warp runs as long as its
    // longest ray, and fewer rays a warp diverge less.  (More warps with fewer rays each issue more in total:
    // 1,000 rays of the icosphere field take 102 us with 32 a warp, 80 with 8, 72 with 1; a 128x128 render of
    // the Cornell box 246 us with 32, 245 with 4, 232 with 8, 229.5 with 14.)
    uint32_t sms;
    asm("mov.u32 %0, %%nsmid;" : "=r"(sms));
    const uint32_t warps = min(gridDim.x * (blockDim.x >> 5), sms * SMALL_WARPS);
    const uint32_t cap = min(32u, (n + warps - 1u) / warps);
    Traverser<ANY, ALPHA, MULTI> T;
    uint2 stack[TRAVERSAL_STACK];
    const DevScene* sp = nullptr;
    bool active = false, exhausted = false;
    uint32_t item = 0;
    for (;;) {
        const uint32_t act = __ballot_sync(0xFFFFFFFFu, active);
        const uint32_t held = __popc(act);
        if (!exhausted && held < min(cap, (uint32_t)REFILL_THRESHOLD)) {
            const uint32_t need = cap - held;
            uint32_t base = 0;
            if (lane == 0u) base = atomicAdd(work, need);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            const uint32_t rank = __popc(~act & lt_mask);
            if (!active && rank < need) {
                const uint32_t i = base + rank;
                if (i < n) {
                    float3 o, d;
                    float t0, t1;
                    if constexpr (MULTI) {
                        load(i, o, d, t0, t1, sp);
                        ws.scene[lane] = sp;
                        T.init(*sp, ws, o, d, t0, t1);
                    } else {
                        load(i, o, d, t0, t1);
                        T.init(S0, ws, o, d, t0, t1);
                    }
                    item = i;
                    active = true;
                }
            }
            if (base + need >= n) exhausted = true;
        }
        if (!__any_sync(0xFFFFFFFFu, active)) break;
        int code = STEP_MORE;
        if (active) {
            if constexpr (MULTI) code = T.template step_impl<true>(*sp, sp->inst, stack, ws, err);
            else code = T.template step_impl<true>(S0, in, stack, ws, err);
        }
        const bool want = active && code == STEP_COOP;
        if (__any_sync(0xFFFFFFFFu, want)) {  // warp-uniform: triangle tests dealt out over all lanes
            const bool hit_now = T.coop_triangles(want, S0, in, ws);
            if (want) code = T.finish_coop(stack, ws, hit_now) ? STEP_MORE : STEP_DONE;
        }
        if (active && code == STEP_DONE) {
            store(item, T.res);
            active = false;
        }
    }
}

// End of a ray-query kernel: the last block to finish clears the work counter words[0] and the
// finished-block count words[1] for the next query that uses them.
LAM_DEV void trace_done(uint32_t* words) {
    __syncthreads();
    if (threadIdx.x == 0u) {
        __threadfence();
        if (atomicAdd(words + 1, 1u) + 1u == gridDim.x) words[0] = words[1] = 0u;
    }
}

constexpr int TRACE_BLOCK = 128;
constexpr uint32_t SMEM_INSTANCES = 128;

// Bytes of dynamic shared memory that a traversal kernel of this scene is launched with: its instance
// records, if they are few enough (every instance entry reads one).  Sized by the scene, so that a small
// one leaves the rest to L1 (64 instances: 17 instead of 21 KB a CTA, icosphere field 74.9 -> 74.6 ms).
inline uint32_t instance_smem(const DevScene& S) {
    return S.instance_count <= SMEM_INSTANCES ? S.instance_count * (uint32_t)sizeof(DevInstance) : 0u;
}

// Copies the instance records into shared memory when they fit; returns where the traversal finds them.
// The nodes stay in global memory, where the TLAS is L1-resident: one node-test call site then loads TLAS
// and BLAS nodes alike through the read-only path (staging the TLAS in shared memory made those loads
// generic: 1104 against 1118 Mrays/s).
LAM_DEV const DevInstance* stage_instances(const DevScene& S) {
    extern __shared__ uint4 staged_instances[];
    if (S.instance_count > SMEM_INSTANCES) return S.inst;
    const uint4* src = reinterpret_cast<const uint4*>(S.inst);
    for (uint32_t i = threadIdx.x; i < S.instance_count * 4u; i += blockDim.x) staged_instances[i] = src[i];
    __syncthreads();
    return reinterpret_cast<const DevInstance*>(staged_instances);
}

}  // namespace lam
