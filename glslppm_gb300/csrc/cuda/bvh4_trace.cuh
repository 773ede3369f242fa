// Single-ray traversal of the mixed path's 4-wide quantised BVH (shared by the eye pass of the
// mixed path and the photon kernels of kernels_mixed.cu).
//
// Node4Dev: w[0] = origin xyz, exponent bytes x|y|z|child count; w[1] = the four child links (>= 0
// node, < 0 ~triangle, INT32_MIN empty); w[2] = lower box bytes x,y,z and upper x; w[3] = upper
// y,z.  A child box is origin + byte * 2^(exponent-127) per axis, rounded outward when the tree
// was built; the slab distances are widened by a bound on their rounding, and triangles are
// tested with the exact path's arithmetic (device_common.cuh), so the closest hit -- triangle, t and
// barycentrics -- is the exact traversal's; where two triangles give the same t, the leaf ranks of
// the exact walk's ordering (DevScene::tri_rank) pick the one it meets first.
#pragma once

#include "device_common.cuh"

namespace sppm_dev {

constexpr int kStack = 196;  // >= 3 * kBvh4MaxDepth + 1 (kBvh4MaxDepth = 64)

struct Hit4 {
    float t;
    int32_t tri;
    float bu, bv, bw;  // (v, w, u) as the plain path stores them
};

__device__ __forceinline__ float node_scale(uint8_t e) { return __uint_as_float((uint32_t)e << 23); }

// direction component used for the slab reciprocals: a zero (or tiny) component is replaced by
// +-1e-26 so that the slab of that axis is +-huge instead of NaN (a NaN slab would be ignored by
// fminf/fmaxf and the ray would enter every box the other axes allow)
__device__ __forceinline__ float slab_dir(float d) { return fabsf(d) < 1e-26f ? copysignf(1e-26f, d) : d; }

// ---- conservative slab tests over the quantised boxes ------------------------------------------
// A child plane is P = origin + q * 2^e (q a byte).  One byte permutation places the byte in the
// mantissa of 0.5: f = 0.5 + q * 2^-16, and the plane's distance along the ray is
//     fma(f, A, B - A/2 -+ E),  A = 2^(e+16) * r (exact scaling of r = fl(1/d)),
//     B = fma(origin, r, n),  n = fl(-o * r),
// the two planes of a child and axis in one two-lane operation (near with -E, far with +E): half the
// instructions of q made a float of its own (permutation and subtraction) and two scalar fmas.
// Against the exact distance (P' - o) / d to the enclosing plane P' = fl(origin + q 2^e) that the
// builder checked, the roundings of r, n, B, B - A/2, -+ E, the fma and P' add at most
// 8 u S + 2^-8 * 2^e |r| (1 + O(u)), u = 2^-24, with S = (|origin| + |o| + 255 * 2^e) / |d| (each
// rounding's error is u times a term bounded by S, and those of B - A/2 and -+ E u times |A/2| more).
// E = 16 u S' + 2^-7 * 2^e |r|, S' the same sum computed from |r|, |n| and |A| (relative error a few
// u), exceeds that bound, so the near distance is never above the exact entry and the far distance
// never below the exact exit: a box the exact arithmetic enters is never culled (Ize, "Robust BVH Ray
// Traversal", JCGT 2013, applies the same argument to the plain slab test).  Where A overflows, the
// distances become NaN, which the minimum and maximum drop: the box is entered.  Where A does not,
// |A/2| is at most half the largest float, so B - A/2 overflows only with |B| above that half, and a plane
// is at most 0.0078 |A/2| from B: the infinite distance has the side that the plane is on.  (With the byte
// under 1.0 and A half as large, B - A overflowed where B was next to nothing, and entered boxes were
// culled.)  The near plane of each axis is chosen by the sign of the direction once per node, so a child
// needs no per-axis min/max.
constexpr float kSlabErr = 9.5367431640625e-07f;  // 16 * 2^-24
// E's part in |A|: 255 * 2^-16 of S', and 2^-7 of a step (2^-23 of A)
constexpr float kSlabErrA = 255.0f * kSlabErr / 65536.0f + 1.1920928955078125e-07f;
// a box entered later than the closest hit so far by less than this relative margin is still
// visited: the exact triangle test's own rounding may put the winner's t just below its box entry
constexpr float kCullMargin = 1.000244140625f;    // 1 + 2^-12

// a * b + c in two single-precision lanes
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// (r < 0 selects the upper bound as the near plane)
struct Ray4 {
    float ox, oy, oz, dx, dy, dz;
    float rx, ry, rz, nx, ny, nz;     // r = 1/slab_dir(d), n = -o * r
};

__device__ __forceinline__ void ray4_setup(Ray4& R, float ox, float oy, float oz, float dx, float dy, float dz) {
    R.ox = ox, R.oy = oy, R.oz = oz, R.dx = dx, R.dy = dy, R.dz = dz;
    R.rx = 1.0f / slab_dir(dx), R.ry = 1.0f / slab_dir(dy), R.rz = 1.0f / slab_dir(dz);
    R.nx = -ox * R.rx, R.ny = -oy * R.ry, R.nz = -oz * R.rz;
}

// one axis of a node for one ray
struct Slab4 {
    unsigned long long A, B;  // A twice; B - A/2 - E (near planes) and B - A/2 + E (far planes)
    uint32_t near, far;       // words holding the near-plane and far-plane bytes of the four children
};

// e: the axis' exponent byte; lo, hi: the words of its lower and upper bytes
__device__ __forceinline__ Slab4 slab4(uint32_t e, float origin, float lo, float hi, float r, float n) {
    Slab4 s;
    const float A = (node_scale(e) * r) * 65536.0f;
    const float C = fmaf(-0.5f, A, fmaf(origin, r, n));
    const float E = fmaf(kSlabErrA, fabsf(A), kSlabErr * fmaf(fabsf(origin), fabsf(r), fabsf(n)));
    s.A = pack2(A, A);
    s.B = pack2(C - E, C + E);
    const bool neg = r < 0.0f;
    s.near = __float_as_uint(neg ? hi : lo);
    s.far = __float_as_uint(neg ? lo : hi);
    return s;
}

// near and far distance of child K along one axis
template <int K>
__device__ __forceinline__ void slab4_child(const Slab4& s, float& near, float& far) {
    constexpr uint32_t sel = 0x7604u | ((uint32_t)K << 4);  // byte K under the exponent of 0.5
    const float fn = __uint_as_float(__byte_perm(s.near, 0x3F000000u, sel));
    const float ff = __uint_as_float(__byte_perm(s.far, 0x3F000000u, sel));
    unpack2(fma2(pack2(fn, ff), s.A, s.B), near, far);
}

// conservative entry distance of child K (clamped at 0) and whether the ray may hit its box before
// tcull (the closest hit so far times kCullMargin)
template <int K>
__device__ __forceinline__ void child_box(const Slab4& X, const Slab4& Y, const Slab4& Z, float tcull, float& tn,
                                          bool& hit) {
    float nx, ny, nz, fx, fy, fz;
    slab4_child<K>(X, nx, fx);
    slab4_child<K>(Y, ny, fy);
    slab4_child<K>(Z, nz, fz);
    const float t0 = fmaxf(fmax3(nx, ny, nz), 0.0f);
    const float t1 = fmin3(fx, fy, fz);
    tn = t0;
    hit = t0 <= t1 && t0 <= tcull;
}

__device__ __forceinline__ void cswap(float& ta, int32_t& ca, float& tb, int32_t& cb) {
    if (tb < ta) {
        const float t = ta;
        ta = tb;
        tb = t;
        const int32_t c = ca;
        ca = cb;
        cb = c;
    }
}

// closest hit through the 4-wide BVH; PHOTON rays skip emitters, eye rays of the first bounce
// cull back faces (eyeraytrace.fs:130)
// The triangle test is the exact walk's, ended at the first coordinate that fails (u > 1 leaves w < 0), a
// stack entry one 64-bit word, and the loops end without jumps, as in k_trace_photons4.  Us a pass with
// an eye pass in each, environment scene: 274 -> 265 at 133x234 pixels, 203 -> 199 at 872x96; 1024^2 and
// larger images the same.
// rank: the leaf positions of the ordering the exact walk would take for this ray (tri_rank of
// its cube face) or null; at an equal t the triangle the exact walk meets first wins, as there
template <bool PHOTON>
__device__ __forceinline__ Hit4 trace4(const Node4Dev* __restrict__ nodes, const float4* __restrict__ tri_isect, f3 org,
                                       f3 dir, bool cull, float tmax0, uint32_t& err,
                                       const int32_t* __restrict__ rank = nullptr) {
    Hit4 h;
    h.t = tmax0;
    h.tri = -1;
    h.bu = h.bv = h.bw = 0.0f;
    Ray4 R;
    ray4_setup(R, org.x, org.y, org.z, dir.x, dir.y, dir.z);
    int2 stack[kStack];  // node, entry distance
    bool found = true;
    int sp = 0;
    int32_t cur = 0;
    uint32_t visits = 0;
    while (found) {
        if (++visits > 4u * (1u << 20)) {  // bounded: no tree here has this many nodes
            err |= kErrWatchdogTraverse;
            break;
        }
        const float4* np = reinterpret_cast<const float4*>(nodes + cur);
        float4 w0, w1, w2, w3;
        ldg32(np, w0, w1);
        ldg32(np + 2, w2, w3);
        const int cnt = (int)(__float_as_uint(w0.w) >> 24);
        int32_t ch[4] = {__float_as_int(w1.x), __float_as_int(w1.y), __float_as_int(w1.z), __float_as_int(w1.w)};
        // conservative slab test of the (up to) four children
        float tnear[4];
        bool hit[4];
        const uint32_t eb = __float_as_uint(w0.w);
        const Slab4 X = slab4(eb & 0xFF, w0.x, w2.x, w2.w, R.rx, R.nx);
        const Slab4 Y = slab4((eb >> 8) & 0xFF, w0.y, w2.y, w3.x, R.ry, R.ny);
        const Slab4 Z = slab4((eb >> 16) & 0xFF, w0.z, w2.z, w3.y, R.rz, R.nz);
        const float tcull = h.t * kCullMargin;
        child_box<0>(X, Y, Z, tcull, tnear[0], hit[0]);
        child_box<1>(X, Y, Z, tcull, tnear[1], hit[1]);
        child_box<2>(X, Y, Z, tcull, tnear[2], hit[2]);
        child_box<3>(X, Y, Z, tcull, tnear[3], hit[3]);
        // leaf children: their triangles in child order (a closer hit shrinks the search), one copy
        // of the test in a loop over the leaves
        uint32_t leaves = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            hit[k] = hit[k] && k < cnt;
            if (!hit[k] || ch[k] >= 0) continue;
            hit[k] = false;
            if (!(PHOTON && (~ch[k] & kEmitterBit))) leaves |= 1u << k;
        }
        while (leaves) {
            const int k = __ffs(leaves) - 1;
            leaves &= leaves - 1;
            const int32_t ck = k == 0 ? ch[0] : (k == 1 ? ch[1] : (k == 2 ? ch[2] : ch[3]));
            const int32_t tri = ~ck & kTriMask;
            const float4 a = __ldg(&tri_isect[(size_t)tri * 3 + 0]);
            const float4 b = __ldg(&tri_isect[(size_t)tri * 3 + 1]);
            const float4 c = __ldg(&tri_isect[(size_t)tri * 3 + 2]);
            const f3 e0 = mk(a.w, b.x, b.y), e1 = mk(b.z, b.w, c.x);
            const f3 pv = cross(dir, e1);
            const float det = dot(e0, pv);
            const f3 tv = sub(org, mk(a.x, a.y, a.z));
            const f3 qv = cross(tv, e0);
            const float u = xdiv(dot(tv, pv), det);
            if (u >= 0.0f && u <= 1.0f && (PHOTON || !cull || det > 1e-10f)) {
                const float v = xdiv(dot(dir, qv), det);
                const float w = xsub(xsub(1.0f, u), v);
                if (v >= 0.0f && w >= 0.0f) {
                    const float tt = xdiv(dot(e1, qv), det);
                    if (tt >= 0.0f &&
                        (tt < h.t || (rank && tt == h.t && h.tri >= 0 && __ldg(&rank[tri]) < __ldg(&rank[h.tri])))) {
                        h.t = tt;
                        h.tri = tri;
                        h.bu = v;
                        h.bv = w;
                        h.bw = u;
                    }
                }
            }
        }
        // internal children hit before the closest hit so far, sorted near to far: the nearest
        // is next, the others go on the stack farthest first
        const float inf = __int_as_float(0x7f800000);
        const float tcull2 = h.t * kCullMargin;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (!hit[k]) tnear[k] = inf;
        cswap(tnear[0], ch[0], tnear[1], ch[1]);
        cswap(tnear[2], ch[2], tnear[3], ch[3]);
        cswap(tnear[0], ch[0], tnear[2], ch[2]);
        cswap(tnear[1], ch[1], tnear[3], ch[3]);
        cswap(tnear[1], ch[1], tnear[2], ch[2]);
        found = tnear[0] <= tcull2;
        if (found) {
            const int pushes = (tnear[1] <= tcull2) + (tnear[2] <= tcull2) + (tnear[3] <= tcull2);
            if (sp + pushes > kStack) {
                err |= kErrWatchdogTraverse;
                found = false;
                sp = 0;
            } else {
                if (tnear[3] <= tcull2) stack[sp++] = make_int2(ch[3], __float_as_int(tnear[3]));
                if (tnear[2] <= tcull2) stack[sp++] = make_int2(ch[2], __float_as_int(tnear[2]));
                if (tnear[1] <= tcull2) stack[sp++] = make_int2(ch[1], __float_as_int(tnear[1]));
                cur = ch[0];
            }
        }
        while (!found && sp > 0) {
            const int2 e = stack[--sp];
            cur = e.x;
            found = __int_as_float(e.y) <= h.t * kCullMargin;
        }
    }
    return h;
}


}  // namespace sppm_dev
