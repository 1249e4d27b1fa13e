// Two-box responses with few instructions, for lanes that keep one pixel and take many features (pass 1 of the
// staged split search) or many tree nodes (prediction). The decisions are those of feature_bin (eval_fast.cuh):
//   - depth scaling: trunc(RN(v / d)) is floor(v i) for a float i that checked_reciprocal has tried for every
//     magnitude v in use; v i + 2^23 rounded toward zero is one instruction for two values;
//   - corner offsets are floats whose bits are the integer (multiples of the smallest denormal), so they need
//     no conversions;
//   - depth means are estimated in float with a bound on the error; colour sums are exact in double.
#pragma once

#include "eval_fast.cuh"

namespace cf {

using u64 = unsigned long long;

// ---- two floats per instruction -----------------------------------------------------------------
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 fma2_rz(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(u64 v) {
    float2 r;
    unpack_f2(v, r.x, r.y);
    return r;
}

// A float i with floor(v i) = trunc(RN(v / d)) for v = 1 .. most (RN(1 / d) or the next float), or 0. One of the
// two serves 99.9 % of the depths d = RN(mm / 1000) with most = 60, 99.8 % with most = 127.
__device__ __forceinline__ float checked_reciprocal(float d, int most) {
    float inv = __frcp_rn(d);
    for (int k = 0; k < 2; k++) {
        bool same = true;
        for (int v = 1; v <= most && same; v++) {
            const float f = __uint2float_rn(v);
            same = __fmaf_rz(f, inv, 8388608.0f) == __fadd_rz(__fdiv_rn(f, d), 8388608.0f);
        }
        if (same) return inv;
        inv = __uint_as_float(__float_as_uint(inv) + 1u);
    }
    return 0.0f;
}

// What a lane holds of its pixel.
struct BoxLane {
    u64 pos;        // (x, y)
    u64 inv;        // the checked reciprocal of its depth, twice
    u64 side;       // (1 or -1 for a flipped response, 1)
};

// Last column and row of the frame, and bytes of an element and of a row and the first bytes of the planes of
// box 1 and box 2, as multiples of the smallest denormal: such a float's bits are the integer, up to 2^24.
struct FrameView {
    float xmax, ymax, size, pitch, base1, base2;
};
constexpr long long kMaxBoxPlane = (1ll << 24) / 12;   // pixels of a frame whose offsets stay below 2^24

// trunc(RN(v / d)) of two parameters; big = 2^23 with each value's sign
__device__ __forceinline__ u64 scale2(u64 v, const BoxLane& l, u64 big) {
    return sub2(fma2_rz(v, l.inv, big), big);
}

// The two boxes of one feature, and whether both lie inside the frame.
struct Boxes {
    float2 lo1, hi1, lo2, hi2;
    bool in;
};

// (o1, o2, r1, r2: the feature's parameter pairs as floats; b1, b2: 2^23 with the offsets' signs)
__device__ __forceinline__ Boxes boxes(const BoxLane& l, u64 o1, u64 o2, u64 r1, u64 r2, u64 b1, u64 b2, float xmax,
                                       float ymax) {
    const u64 big = pack_f2(8388608.0f, 8388608.0f);
    const u64 c1 = fma2(scale2(o1, l, b1), l.side, l.pos);
    const u64 c2 = fma2(scale2(o2, l, b2), l.side, l.pos);
    const float2 g1 = unpack2(scale2(r1, l, big)), g2 = unpack2(scale2(r2, l, big));
    const float w1 = fmaxf(g1.x, 1.0f), h1 = fmaxf(g1.y, 1.0f), w2 = fmaxf(g2.x, 1.0f), h2 = fmaxf(g2.y, 1.0f);
    const u64 s1 = pack_f2(w1, h1), s2 = pack_f2(w2, h2);
    Boxes b;
    b.lo1 = unpack2(sub2(c1, s1));
    b.hi1 = unpack2(add2(c1, s1));
    b.lo2 = unpack2(sub2(c2, s2));
    b.hi2 = unpack2(add2(c2, s2));
    b.in = fminf(fminf(b.lo1.x, b.lo1.y), fminf(b.lo2.x, b.lo2.y)) >= 0.0f && fmaxf(b.hi1.x, b.hi2.x) <= xmax &&
           fmaxf(b.hi1.y, b.hi2.y) <= ymax;
    return b;
}

// Offsets of the corners: bytes in the sample's frame (corners), or elements of a plane (wide_corners).
struct Corners {
    int ul1, ur1, ll1, lr1, ul2, ur2, ll2, lr2;
    bool in;
};

__device__ __forceinline__ Corners corners(const BoxLane& l, u64 o1, u64 o2, u64 r1, u64 r2, u64 b1, u64 b2,
                                           const FrameView& p) {
    const Boxes b = boxes(l, o1, o2, r1, r2, b1, b2, p.xmax, p.ymax);
    Corners k;
    k.in = b.in;
    const float x1l = fmaf(b.lo1.x, p.size, p.base1), x1r = fmaf(b.hi1.x, p.size, p.base1);
    const float x2l = fmaf(b.lo2.x, p.size, p.base2), x2r = fmaf(b.hi2.x, p.size, p.base2);
    k.ul1 = __float_as_int(fmaf(b.lo1.y, p.pitch, x1l));
    k.ur1 = __float_as_int(fmaf(b.lo1.y, p.pitch, x1r));
    k.ll1 = __float_as_int(fmaf(b.hi1.y, p.pitch, x1l));
    k.lr1 = __float_as_int(fmaf(b.hi1.y, p.pitch, x1r));
    k.ul2 = __float_as_int(fmaf(b.lo2.y, p.pitch, x2l));
    k.ur2 = __float_as_int(fmaf(b.lo2.y, p.pitch, x2r));
    k.ll2 = __float_as_int(fmaf(b.hi2.y, p.pitch, x2l));
    k.lr2 = __float_as_int(fmaf(b.hi2.y, p.pitch, x2r));
    return k;
}

// Frames whose byte offsets do not stay below 2^24: element indices in integers. A coordinate v of less than 2^22
// plus 1.5 * 2^23 is the float with the bits kIntegerBits + v; the bits' excess cancels modulo 2^32.
constexpr int kMaxWideSide = 1 << 21;   // a corner of a box inside the frame is below it
__device__ __forceinline__ Corners wide_corners(const BoxLane& l, u64 o1, u64 o2, u64 r1, u64 r2, u64 b1, u64 b2,
                                                float xmax, float ymax, int width) {
    constexpr uint32_t kIntegerBits = 0x4B400000u;
    const Boxes b = boxes(l, o1, o2, r1, r2, b1, b2, xmax, ymax);
    const u64 big = pack_f2(12582912.0f, 12582912.0f);
    const uint32_t w = static_cast<uint32_t>(width), excess = kIntegerBits * (w + 1u);
    auto bits = [&](float2 v) {
        const float2 t = unpack2(add2(pack_f2(v.x, v.y), big));
        return make_uint2(__float_as_uint(t.x) - excess, __float_as_uint(t.y));
    };
    const uint2 lo1 = bits(b.lo1), hi1 = bits(b.hi1), lo2 = bits(b.lo2), hi2 = bits(b.hi2);
    Corners k;
    k.in = b.in;
    k.ul1 = static_cast<int>(lo1.y * w + lo1.x);
    k.ur1 = static_cast<int>(lo1.y * w + hi1.x);
    k.ll1 = static_cast<int>(hi1.y * w + lo1.x);
    k.lr1 = static_cast<int>(hi1.y * w + hi1.x);
    k.ul2 = static_cast<int>(lo2.y * w + lo2.x);
    k.ur2 = static_cast<int>(lo2.y * w + hi2.x);
    k.ll2 = static_cast<int>(hi2.y * w + lo2.x);
    k.lr2 = static_cast<int>(hi2.y * w + hi2.x);
    return k;
}

template <typename V>
__device__ __forceinline__ V frame_at(const unsigned char* frame, int offset) {
    return __ldg(reinterpret_cast<const V*>(frame + offset));
}

// The box sums (mm) and counts of a depth feature.
struct DepthBoxes {
    int s1, n1, s2, n2;
};

// (at: the value at a corner's offset)
template <typename At>
__device__ __forceinline__ DepthBoxes depth_boxes_at(const Corners& k, const At& at) {
    int2 ul1 = make_int2(0, 0), ur1 = ul1, ll1 = ul1, lr1 = ul1, ul2 = ul1, ur2 = ul1, ll2 = ul1, lr2 = ul1;
    if (k.in) {
        ul1 = at(k.ul1), ur1 = at(k.ur1);
        ll1 = at(k.ll1), lr1 = at(k.lr1);
        ul2 = at(k.ul2), ur2 = at(k.ur2);
        ll2 = at(k.ll2), lr2 = at(k.lr2);
    }
    auto box = [](int lr, int ur, int ul, int ll) {
        return static_cast<int>(static_cast<uint32_t>(lr) - static_cast<uint32_t>(ur) + static_cast<uint32_t>(ul) -
                                static_cast<uint32_t>(ll));
    };
    DepthBoxes b;
    b.s1 = box(lr1.x, ur1.x, ul1.x, ll1.x);
    b.n1 = box(lr1.y, ur1.y, ul1.y, ll1.y);
    b.s2 = box(lr2.x, ur2.x, ul2.x, ll2.x);
    b.n2 = box(lr2.y, ur2.y, ul2.y, ll2.y);
    return b;
}

__device__ __forceinline__ DepthBoxes depth_boxes(const Corners& k, const unsigned char* frame) {
    return depth_boxes_at(k, [=](int offset) { return frame_at<int2>(frame, offset); });
}

// Bounds of the exact response of a depth feature in metres, where both counts lie in [1, 2^23) (`plain`).
// Means in mm: the conversion is within 2^-24, the reciprocal within 2^-23, the products, the difference,
// 0.001f and the last rounding within 2^-24 each: the response is within 4.1e-10 (|a| + |b|) of the exact one,
// and 5e-10 (|a| + |b|) bounds it.
struct DepthBounds {
    float lo, hi;
    bool plain;
};

__device__ __forceinline__ DepthBounds depth_bounds(const DepthBoxes& x) {
    const float n1 = __int_as_float(0x4B000000 + x.n1) - 8388608.0f;
    const float n2 = __int_as_float(0x4B000000 + x.n2) - 8388608.0f;
    float i1, i2;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(i1) : "f"(n1));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(i2) : "f"(n2));
    const float a = static_cast<float>(x.s1) * i1, b = static_cast<float>(x.s2) * i2;
    const float delta = fmaf(fabsf(a) + fabsf(b), 5e-10f, 1e-30f);
    const float r = a - b;
    DepthBounds d;
    d.lo = fmaf(r, 0.001f, -delta);
    d.hi = fmaf(r, 0.001f, delta);
    d.plain = (static_cast<uint32_t>(x.n1 - 1) | static_cast<uint32_t>(x.n2 - 1)) < 0x7FFFFFu;
    return d;
}

// The exact response of a colour feature (NaN if a corner is); at1, at2: the value at a corner's offset for each box.
template <typename At1, typename At2>
__device__ __forceinline__ double color_response_at(const Corners& k, const At1& at1, const At2& at2) {
    float ul1 = 0, ur1 = 0, ll1 = 0, lr1 = 0, ul2 = 0, ur2 = 0, ll2 = 0, lr2 = 0;
    if (k.in) {
        ul1 = at1(k.ul1), ur1 = at1(k.ur1);
        ll1 = at1(k.ll1), lr1 = at1(k.lr1);
        ul2 = at2(k.ul2), ur2 = at2(k.ur2);
        ll2 = at2(k.ll2), lr2 = at2(k.lr2);
    }
    const double A = __dadd_rn(__dsub_rn(lr1, ur1), __dsub_rn(ul1, ll1));
    const double B = __dadd_rn(__dsub_rn(lr2, ur2), __dsub_rn(ul2, ll2));
    return __dsub_rn(A, B);
}

__device__ __forceinline__ double color_response(const Corners& k, const unsigned char* frame) {
    const auto at = [=](int offset) { return frame_at<float>(frame, offset); };
    return color_response_at(k, at, at);
}

}  // namespace cf
