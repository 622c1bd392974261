// reservoir.cuh - a lam_reservoir (Reservoir, src/bindings.wesl:158-169; 64 bytes, 16-byte aligned in every
// buffer) as four 16-byte words.
#pragma once
#include "../../include/lambent.h"
#include "device_math.cuh"

namespace lam {

// A reservoir as four 16-byte words: (visible point, normal), (sample point, normal), (radiance, type),
// (roughness, w, confidence, W).  Field by field it is sixteen 4-byte accesses 64 bytes apart, each of
// which touches as many sectors as one of these (at 1280x720: temporal pass 74 -> 26 us).
LAM_DEV lam_reservoir res_unpack(uint4 a, uint4 b, uint4 c, uint4 d) {
    lam_reservoir r;
    r.visible_point[0] = __uint_as_float(a.x); r.visible_point[1] = __uint_as_float(a.y);
    r.visible_point[2] = __uint_as_float(a.z); r.visible_normal = a.w;
    r.sample_point[0] = __uint_as_float(b.x); r.sample_point[1] = __uint_as_float(b.y);
    r.sample_point[2] = __uint_as_float(b.z); r.sample_normal = b.w;
    r.out_radiance[0] = __uint_as_float(c.x); r.out_radiance[1] = __uint_as_float(c.y);
    r.out_radiance[2] = __uint_as_float(c.z); r.ty = c.w;
    r.roughness = __uint_as_float(d.x); r.w = __uint_as_float(d.y);
    r.packed_confidence_valid = d.z; r.W = __uint_as_float(d.w);
    return r;
}
LAM_DEV lam_reservoir res_load(const lam_reservoir* p) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    return res_unpack(q[0], q[1], q[2], q[3]);
}

LAM_DEV void res_store(lam_reservoir* p, const lam_reservoir& r) {
    uint4* q = reinterpret_cast<uint4*>(p);
    q[0] = make_uint4(__float_as_uint(r.visible_point[0]), __float_as_uint(r.visible_point[1]),
                      __float_as_uint(r.visible_point[2]), r.visible_normal);
    q[1] = make_uint4(__float_as_uint(r.sample_point[0]), __float_as_uint(r.sample_point[1]),
                      __float_as_uint(r.sample_point[2]), r.sample_normal);
    q[2] = make_uint4(__float_as_uint(r.out_radiance[0]), __float_as_uint(r.out_radiance[1]),
                      __float_as_uint(r.out_radiance[2]), r.ty);
    q[3] = make_uint4(__float_as_uint(r.roughness), __float_as_uint(r.w), r.packed_confidence_valid, __float_as_uint(r.W));
}

}  // namespace lam
