// Plain-FP32 SPPM kernels for sm_103a: every operation of the reference shaders in IEEE single
// precision, in the order the shaders write it (see device_common.cuh for the pinned helpers),
// so each per-pixel and per-photon value is bit-identical to the CPU restatement.  This
// translation unit is also compiled with -fmad=false.
//
// One SPPM frame (m_display, glslppm.cpp:214-536) is one launch per stage over all jobs of a
// batch:
//   k_frame_begin        hash-slot clear + per-job frame bookkeeping (AA offset of the eye pass)
//   k_eye                eyeraytrace.fs, fused with the max/min reductions (warp shuffles + one
//                        atomic per warp) that replace ReduceTexture's 2x2 passes and 18 readbacks
//   k_grid               InitialRadius / grid (glslppm.cpp:294-311), on the device
//   k_photon_gen         photontrace.fs emission / bounce / Russian roulette + the sum reduction;
//                        queues each live photon's ray (with its bin for the counting sort)
//   k_ray_bins_*         counting sort of the queued rays by direction class and origin cell
//   k_trace_photons      persistent traversal of the queued rays (dynamic fetch); rays with a zero
//                        direction component are set aside for k_trace_photons_coop (one warp each)
//   k_photon_store       store rule + hash.fs + scatter.vs (depth test = atomicMin of the photon
//                        index) + correction.vs (additive blend = atomicAdd), warp-aggregated
//   k_gather             progressive.fs
//   k_resolve            re.fs (on demand)
// k_photon is the single-kernel form of gen + trace + store (SPPM_FLAG_FUSED_PHOTON).
#include <cstddef>
#include <cstdint>

#include "bvh4_trace.cuh"
#include "device_common.cuh"
#include "kernels.h"
#include "photon_grid.cuh"

namespace sppm_dev {

// ----------------------------------------------------------------------------------------------
// traversal: the threaded BVH walk of raytrace() (eyeraytrace.fs:67-290, photontrace.fs:123-255)
// ----------------------------------------------------------------------------------------------
struct Hit {
    float t;
    int32_t tri;
    int32_t mat;
    float bu, bv, bw;  // Barycentric = (v, w, u)
};

// bin of a queued ray: direction class (cube face x signs of the two minor components) and the
// Morton index of its origin's cell in a grid over the scene's bounding cube
__device__ __forceinline__ uint32_t spread_bits4(uint32_t v) {  // bits 0..3 -> 0, 3, 6, 9
    v = (v | (v << 4)) & 0x0C3u;
    return (v | (v << 2)) & 0x249u;
}
__device__ __forceinline__ uint32_t ray_bin(const DevScene& s, f3 o, f3 d) {
    const float* bs = s.bsphere;
    const float half = (float)(1u << (kRayCellBits - 1));
    const float sc = half / fmaxf(bs[3], 1e-30f);
    const float top = 2.0f * half - 1.0f;
    const uint32_t cx = (uint32_t)fminf(fmaxf((o.x - bs[0]) * sc + half, 0.0f), top);
    const uint32_t cy = (uint32_t)fminf(fmaxf((o.y - bs[1]) * sc + half, 0.0f), top);
    const uint32_t cz = (uint32_t)fminf(fmaxf((o.z - bs[2]) * sc + half, 0.0f), top);
    const int face = cube_face(d);
    const int axis = face >> 1;
    const float m1 = axis == 0 ? d.y : d.x, m2 = axis == 2 ? d.y : d.z;
    const uint32_t cls = (uint32_t)face * 4u + (m1 < 0.0f ? 2u : 0u) + (m2 < 0.0f ? 1u : 0u);
    return (cls << (3 * kRayCellBits)) | (spread_bits4(cx) << 2) | (spread_bits4(cy) << 1) | spread_bits4(cz);
}

struct TraversalCount {
    uint32_t nodes = 0, tris = 0;
};

// The walk of one ray by one thread.  The divisions of the triangle test follow one
// another's tests, as few lanes need all three, and the loop ends in one place, so that a warp's lanes
// meet before the next node (u > 1 leaves w < 0 whatever v is).  AHEAD: both nodes that may come next
// are loaded before this one is tested (k_trace_photons).
template <bool PHOTON, bool COUNT = false, bool AHEAD = false>
__device__ __forceinline__ Hit trace_exact(const DevScene& s, f3 org, f3 dir, bool cull, uint32_t& err,
                                           TraversalCount* cnt = nullptr) {
    Hit h;
    h.t = PHOTON ? 1.0e30f : 1.0e20f;
    h.tri = -1;
    h.mat = -1;
    h.bu = h.bv = h.bw = 0.0f;
    const int face = cube_face(dir);
    const NodeX* nodes = s.nodes + (size_t)face * s.num_nodes;
    const RayX R = ray_x(org, dir, face);
    const int32_t nn = (int32_t)s.num_nodes;
    int32_t i = 0;
    unsigned long long lo, hi, near_far, links;
    if (AHEAD) ldg32q(nodes, lo, hi, near_far, links);
    int32_t steps = 0;
    do {
        unsigned long long next_lo, next_hi, next_near_far, next_links, miss_lo, miss_hi, miss_near_far, miss_links;
        if (AHEAD) {
            const uint32_t last = (uint32_t)nn - 1u;
            ldg32q(nodes + min((uint32_t)i + 1u, last), next_lo, next_hi, next_near_far, next_links);
            ldg32q(nodes + min((uint32_t)node_miss(links), last), miss_lo, miss_hi, miss_near_far, miss_links);
        } else {
            ldg32q(nodes + i, lo, hi, near_far, links);
        }
        if (COUNT) cnt->nodes++;
        float tmin, tmax;
        slab_x<false>(R, lo, hi, near_far, tmin, tmax);
        const bool hit = (tmin <= tmax) && (tmin <= h.t) && (tmax >= 0.0f);
        const int32_t tri = node_tri(links);
        if (hit && tri >= 0 && (!PHOTON || !(tri & kEmitterBit))) {
            const int32_t t = tri & kTriMask;
            if (COUNT) cnt->tris++;
            const float4 a = __ldg(&s.tri_isect[(size_t)t * 3 + 0]);
            const float4 b = __ldg(&s.tri_isect[(size_t)t * 3 + 1]);
            const float4 c = __ldg(&s.tri_isect[(size_t)t * 3 + 2]);
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
                    if (tt >= 0.0f && tt < h.t) {
                        h.t = tt;
                        h.tri = t;
                        h.mat = __float_as_int(c.y);
                        h.bu = v;
                        h.bv = w;
                        h.bw = u;
                    }
                }
            }
        }
        i = hit ? i + 1 : node_miss(links);
        if (AHEAD) {
            lo = hit ? next_lo : miss_lo;
            hi = hit ? next_hi : miss_hi;
            near_far = hit ? next_near_far : miss_near_far;
            links = hit ? next_links : miss_links;
        }
        steps++;
    } while ((uint32_t)i < (uint32_t)nn && steps <= nn);
    if ((uint32_t)i < (uint32_t)nn) err |= kErrWatchdogTraverse;
    return h;
}

// A ray with a zero (or denormal-small) direction component has an infinite reciprocal, and
// 0 * inf or inf - inf turn that axis' slab into NaN, which fminf/fmaxf then ignore: the box test
// passes for every box the other axes allow (for a photon leaving the light straight down,
// every box), and the walk visits nearly the whole tree.  Such rays are rare (a few per 10^7)
// but each costs thousands of dependent node fetches, so they are traced by coop_trace_exact.
__device__ __forceinline__ bool slab_degenerate(f3 d) {
    return fabsf(d.x) < 1e-30f || fabsf(d.y) < 1e-30f || fabsf(d.z) < 1e-30f;
}

// Warp-cooperative form of trace_exact for one ray (all 32 lanes call it with the same
// arguments and get the same result).  The lanes evaluate the box and triangle tests of 32
// consecutive nodes at once; the walk itself -- which nodes are visited, in which order, and
// which triangle hit replaces the current one -- is then resolved with ballots in exactly the
// order of the scalar loop, so the result is the same bit for bit.  A node is visited as a hit
// when its box passes with the t of the closest hit so far; a visited leaf replaces the closest
// hit when its triangle test passes with that t; the walk goes to node + 1 after a hit and to
// the miss link otherwise.
// The walk may also be resumed where a scalar walk stopped: at node `start` with the closest hit
// `h0` after `steps0` steps (coop_trace_exact_from); the result is the scalar walk's all the same.
template <bool PHOTON, bool COUNT>
__device__ __forceinline__ Hit coop_trace_exact_from(const DevScene& s, f3 org, f3 dir, bool cull, uint32_t& err,
                                                  TraversalCount* cnt, int32_t start, Hit h0, uint32_t steps0) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const int lane = (int)(threadIdx.x & 31);
    Hit h = h0;
    const int face = cube_face(dir);
    const NodeX* nodes = s.nodes + (size_t)face * s.num_nodes;
    const RayX R = ray_x(org, dir, face);
    const int32_t nn = (int32_t)s.num_nodes;
    int32_t cur = start;
    uint32_t steps = steps0;
    bool done = start < 0 || start >= nn;
    while (!done) {
        const int32_t base = cur;
        const int32_t j = base + lane;
        bool box = false, leaf = false, ok = false;
        float tmin = 0.0f, tt = 0.0f, bu = 0.0f, bv = 0.0f, bw = 0.0f;
        int32_t miss = -1, tri = -1, mat = -1;
        if (j < nn) {
            unsigned long long lo, hi, near_far, links;
            ldg32q(nodes + j, lo, hi, near_far, links);
            float tmax;
            slab_x<false>(R, lo, hi, near_far, tmin, tmax);
            box = (tmin <= tmax) && (tmax >= 0.0f);
            miss = node_miss(links);
            const int32_t raw = node_tri(links);
            leaf = raw >= 0 && (!PHOTON || !(raw & kEmitterBit));
            if (leaf && box) {
                tri = raw & kTriMask;
                const float4 a = __ldg(&s.tri_isect[(size_t)tri * 3 + 0]);
                const float4 b = __ldg(&s.tri_isect[(size_t)tri * 3 + 1]);
                const float4 c = __ldg(&s.tri_isect[(size_t)tri * 3 + 2]);
                const f3 v0 = mk(a.x, a.y, a.z), e0 = mk(a.w, b.x, b.y), e1 = mk(b.z, b.w, c.x);
                const f3 pv = cross(dir, e1);
                const float det = dot(e0, pv);
                if (PHOTON || !cull || det > 1e-10f) {
                    const f3 tv = sub(org, v0);
                    const f3 qv = cross(tv, e0);
                    const float u = xdiv(dot(tv, pv), det);
                    const float v = xdiv(dot(dir, qv), det);
                    tt = xdiv(dot(e1, qv), det);
                    const float w = xsub(xsub(1.0f, u), v);
                    ok = u >= 0.0f && v >= 0.0f && tt >= 0.0f && w >= 0.0f;
                    mat = __float_as_int(c.y);
                    bu = v;
                    bv = w;
                    bw = u;
                }
            }
        }
        const unsigned inwin = __ballot_sync(kFull, j < nn);
        const unsigned leaves = __ballot_sync(kFull, leaf);
        int pos = 0;
        for (;;) {
            const unsigned ge = kFull << pos;
            const unsigned M = __ballot_sync(kFull, box && tmin <= h.t) & ge & inwin;  // hits with the current t
            const unsigned U = __ballot_sync(kFull, ok && tt < h.t) & M;               // hits that replace it
            const unsigned notM = ~M & ge;
            const int stop = notM ? __ffs(notM) - 1 : 32;  // first lane >= pos that is not a hit
            const unsigned run = (stop == 32 ? kFull : ((1u << stop) - 1u)) & ge;
            const unsigned ur = U & run;
            if (ur) {
                const int p = __ffs(ur) - 1;  // visits pos..p, the leaf at p replaces the hit
                const unsigned vis = run & (p == 31 ? kFull : ((2u << p) - 1u));
                steps += __popc(vis);
                if (COUNT) {
                    cnt->nodes += __popc(vis);
                    cnt->tris += __popc(vis & leaves);
                }
                h.t = __shfl_sync(kFull, tt, p);
                h.tri = __shfl_sync(kFull, tri, p);
                h.mat = __shfl_sync(kFull, mat, p);
                h.bu = __shfl_sync(kFull, bu, p);
                h.bv = __shfl_sync(kFull, bv, p);
                h.bw = __shfl_sync(kFull, bw, p);
                if (p == 31) {
                    cur = base + 32;
                    done = cur >= nn;
                    break;
                }
                pos = p + 1;
                if (base + pos >= nn) {
                    done = true;
                    break;
                }
                continue;
            }
            steps += __popc(run);  // pos..stop-1 visited as hits, none replaces the hit
            if (COUNT) {
                cnt->nodes += __popc(run);
                cnt->tris += __popc(run & leaves);
            }
            if (stop == 32) {
                cur = base + 32;
                done = cur >= nn;
                break;
            }
            if (!((inwin >> stop) & 1u)) {  // the walk stepped past the last node
                done = true;
                break;
            }
            steps += 1;  // lane `stop` is visited and missed: follow its miss link
            if (COUNT) cnt->nodes += 1;
            const int32_t nx = __shfl_sync(kFull, miss, stop);
            if (nx < 0 || nx >= nn) {
                done = true;
                break;
            }
            if (nx > base + stop && nx < base + 32) {
                pos = nx - base;
                continue;
            }
            cur = nx;
            break;
        }
        if (steps > (uint32_t)nn + 1u) {
            err |= kErrWatchdogTraverse;
            done = true;
        }
    }
    return h;
}

template <bool PHOTON, bool COUNT>
__device__ __forceinline__ Hit coop_trace_exact(const DevScene& s, f3 org, f3 dir, bool cull, uint32_t& err,
                                                TraversalCount* cnt) {
    Hit h;
    h.t = PHOTON ? 1.0e30f : 1.0e20f;
    h.tri = -1;
    h.mat = -1;
    h.bu = h.bv = h.bw = 0.0f;
    return coop_trace_exact_from<PHOTON, COUNT>(s, org, dir, cull, err, cnt, 0, h, 0u);
}

// Block-wide form of the same walk (1024 threads, one ray, the same result bit for bit): the
// threads evaluate the box and triangle tests of 1024 consecutive nodes into shared memory; one
// warp then resolves the walk with 32-bit masks of the window -- M = nodes whose box passes with
// the current closest t, U = those of M whose triangle would replace the closest hit -- jumping
// straight to the next "event" (first node at or after the walk's position that is not in M, or
// is in U).  All nodes before an event are visited as hits without effect, so a window costs a
// few mask operations per event instead of a step per node; M and U are recomputed only when the
// closest hit changes.
constexpr int kBlockWalk = 1024;
constexpr int kBlockWords = kBlockWalk / 32;

struct BlockWalkShared {
    float tmin[kBlockWalk], tt[kBlockWalk], bu[kBlockWalk], bv[kBlockWalk], bw[kBlockWalk];
    int32_t miss[kBlockWalk], tri[kBlockWalk], mat[kBlockWalk];
    uint32_t box[kBlockWords], leaf[kBlockWords], ok[kBlockWords], inwin[kBlockWords];
    uint32_t M[kBlockWords], U[kBlockWords];  // with the closest t at the window's start
    // the walk's state, broadcast to the block between windows
    Hit h;
    int32_t cur;
    uint32_t steps, nodes, tris;
    int done;
};

template <bool PHOTON, bool COUNT>
__device__ __noinline__ Hit block_trace_exact(const DevScene& s, f3 org, f3 dir, bool cull, uint32_t& err,
                                              TraversalCount* cnt, BlockWalkShared& sh) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const int t = (int)threadIdx.x;
    const int lane = t & 31;
    const int face = cube_face(dir);
    const NodeX* nodes = s.nodes + (size_t)face * s.num_nodes;
    const RayX R = ray_x(org, dir, face);
    const int32_t nn = (int32_t)s.num_nodes;
    if (t == 0) {
        sh.h.t = PHOTON ? 1.0e30f : 1.0e20f;
        sh.h.tri = -1;
        sh.h.mat = -1;
        sh.h.bu = sh.h.bv = sh.h.bw = 0.0f;
        sh.cur = 0;
        sh.steps = sh.nodes = sh.tris = 0;
        sh.done = 0;
    }
    __syncthreads();
    while (!sh.done) {
        const int32_t base = sh.cur;
        // ---- evaluate the window's nodes (every thread one node) ----
        {
            const int32_t j = base + t;
            bool box = false, leaf = false, ok = false;
            float tmin = 0.0f, tt = 0.0f, bu = 0.0f, bv = 0.0f, bw = 0.0f;
            int32_t miss = -1, tri = -1, mat = -1;
            if (j < nn) {
                // two 16-byte loads: this toolkit's ptxas fails on the 256-bit form in this function
                const ulonglong2 A = __ldg(reinterpret_cast<const ulonglong2*>(nodes + j));
                const ulonglong2 B = __ldg(reinterpret_cast<const ulonglong2*>(nodes + j) + 1);
                float tmax;
                slab_x<false>(R, A.x, A.y, B.x, tmin, tmax);
                box = (tmin <= tmax) && (tmax >= 0.0f);
                miss = node_miss(B.y);
                const int32_t raw = node_tri(B.y);
                leaf = raw >= 0 && (!PHOTON || !(raw & kEmitterBit));
                if (leaf && box) {
                    tri = raw & kTriMask;
                    const float4 a = __ldg(&s.tri_isect[(size_t)tri * 3 + 0]);
                    const float4 b = __ldg(&s.tri_isect[(size_t)tri * 3 + 1]);
                    const float4 c = __ldg(&s.tri_isect[(size_t)tri * 3 + 2]);
                    const f3 v0 = mk(a.x, a.y, a.z), e0 = mk(a.w, b.x, b.y), e1 = mk(b.z, b.w, c.x);
                    const f3 pv = cross(dir, e1);
                    const float det = dot(e0, pv);
                    if (PHOTON || !cull || det > 1e-10f) {
                        const f3 tv = sub(org, v0);
                        const f3 qv = cross(tv, e0);
                        const float u = xdiv(dot(tv, pv), det);
                        const float v = xdiv(dot(dir, qv), det);
                        tt = xdiv(dot(e1, qv), det);
                        const float w = xsub(xsub(1.0f, u), v);
                        ok = u >= 0.0f && v >= 0.0f && tt >= 0.0f && w >= 0.0f;
                        mat = __float_as_int(c.y);
                        bu = v;
                        bv = w;
                        bw = u;
                    }
                }
            }
            sh.tmin[t] = tmin;
            sh.tt[t] = tt;
            sh.bu[t] = bu;
            sh.bv[t] = bv;
            sh.bw[t] = bw;
            sh.miss[t] = miss;
            sh.tri[t] = tri;
            sh.mat[t] = mat;
            const float ht = sh.h.t;
            const bool m = box && j < nn && tmin <= ht;
            const unsigned bx = __ballot_sync(kFull, box), lf = __ballot_sync(kFull, leaf),
                           okm = __ballot_sync(kFull, ok), in = __ballot_sync(kFull, j < nn),
                           mm = __ballot_sync(kFull, m), um = __ballot_sync(kFull, m && ok && tt < ht);
            if (lane == 0) {
                sh.box[t >> 5] = bx;
                sh.leaf[t >> 5] = lf;
                sh.ok[t >> 5] = okm;
                sh.inwin[t >> 5] = in;
                sh.M[t >> 5] = mm;
                sh.U[t >> 5] = um;
            }
        }
        __syncthreads();
        // ---- one warp resolves the walk through the window ----
        if (t < 32) {
            const int w = lane;  // this lane's 32-node word
            Hit h = sh.h;
            uint32_t steps = sh.steps, cn = 0, ct = 0;
            int32_t next_window = -1;
            bool done = false;
            // M and U of words from..31 for the current closest t: word k from node k*32 + lane of
            // every lane (conflict-free shared reads), kept by lane k
            auto masks = [&](uint32_t& M, uint32_t& U, int from) {
                for (int k = from; k < kBlockWords; k++) {
                    const int n = k * 32 + lane;
                    const bool in = (sh.inwin[k] >> lane) & 1u, bx = (sh.box[k] >> lane) & 1u;
                    const bool m = in && bx && sh.tmin[n] <= h.t;
                    const bool u = m && ((sh.ok[k] >> lane) & 1u) && sh.tt[n] < h.t;
                    const unsigned bm = __ballot_sync(kFull, m), bu = __ballot_sync(kFull, u);
                    if (lane == k) {
                        M = bm;
                        U = bu;
                    }
                }
            };
            uint32_t M = sh.M[w], U = sh.U[w];
            const uint32_t leafw = sh.leaf[w], inw = sh.inwin[w];
            int pos = 0;
            for (;;) {
                // nodes at or after pos in this lane's word
                const int pw = pos >> 5;
                const uint32_t ge = w < pw ? 0u : (w > pw ? kFull : (kFull << (pos & 31)));
                const uint32_t ev = (~M | U) & ge;
                const unsigned has = __ballot_sync(kFull, ev != 0u);
                int e = kBlockWalk;  // event position (window end when none)
                if (has) {
                    const int fw = __ffs(has) - 1;
                    const uint32_t evw = __shfl_sync(kFull, ev, fw);
                    e = fw * 32 + __ffs(evw) - 1;
                }
                // nodes pos .. e-1 are visited as hits that change nothing
                {
                    const uint32_t lo = ge;
                    const uint32_t hi = (e >> 5) > w ? kFull : ((e >> 5) < w ? 0u : ((1u << (e & 31)) - 1u));
                    const uint32_t vis = lo & hi;
                    const uint32_t nv = __reduce_add_sync(kFull, __popc(vis));
                    steps += nv;
                    if (COUNT) {
                        cn += nv;
                        ct += __reduce_add_sync(kFull, __popc(vis & leafw));
                    }
                }
                if (e == kBlockWalk) {  // ran off the window's end: continue at the next node
                    next_window = base + kBlockWalk;
                    done = next_window >= nn;
                    break;
                }
                const int ew = e >> 5, eb = e & 31;
                const bool e_in = (__shfl_sync(kFull, inw, ew) >> eb) & 1u;
                if (!e_in) {  // the walk stepped past the last node
                    done = true;
                    break;
                }
                const bool e_upd = (__shfl_sync(kFull, U, ew) >> eb) & 1u;
                steps += 1;
                if (COUNT) cn += 1;
                if (e_upd) {  // a hit whose triangle replaces the closest hit
                    if (COUNT) ct += 1;
                    h.t = sh.tt[e];
                    h.tri = sh.tri[e];
                    h.mat = sh.mat[e];
                    h.bu = sh.bu[e];
                    h.bv = sh.bv[e];
                    h.bw = sh.bw[e];
                    pos = e + 1;
                    if (base + pos >= nn) {
                        done = true;
                        break;
                    }
                    if (pos == kBlockWalk) {
                        next_window = base + kBlockWalk;
                        break;
                    }
                    masks(M, U, pos >> 5);
                    continue;
                }
                // a node whose box misses: follow its miss link
                const int32_t nx = sh.miss[e];
                if (nx < 0 || nx >= nn) {
                    done = true;
                    break;
                }
                if (nx > base + e && nx < base + kBlockWalk) {
                    pos = nx - base;
                    continue;
                }
                next_window = nx;
                break;
            }
            if (lane == 0) {
                sh.h = h;
                sh.steps = steps;
                if (COUNT) {
                    sh.nodes += cn;
                    sh.tris += ct;
                }
                sh.cur = next_window;
                sh.done = done || steps > (uint32_t)nn + 1u;
                if (steps > (uint32_t)nn + 1u) sh.steps = 0xFFFFFFFFu;
            }
        }
        __syncthreads();
    }
    const Hit out = sh.h;
    if (sh.steps == 0xFFFFFFFFu) err |= kErrWatchdogTraverse;
    if (COUNT) {
        cnt->nodes += sh.nodes;
        cnt->tris += sh.tris;
    }
    __syncthreads();  // the shared state is read by every thread before a next ray reuses it
    return out;
}

struct Shade {
    f3 pos, nrm, gnrm, col;
    int brdf;
    float eta, g;
};

// Result of raytrace() for a hit (eyeraytrace.fs:256-287)
__device__ __forceinline__ Shade shade_hit(const DevScene& s, const Hit& h) {
    const float4* ts = s.tri_shade + (size_t)h.tri * 6;
    float4 r0, r1, r2, r3, r4, r5;
    ldg32(ts, r0, r1);
    ldg32(ts + 2, r2, r3);
    ldg32(ts + 4, r4, r5);
    const f3 V0 = mk(r1.x, r1.y, r1.z), V1 = mk(r1.w, r2.x, r2.y), V2 = mk(r2.z, r2.w, r3.x);
    const f3 N0 = mk(r3.y, r3.z, r3.w), N1 = mk(r4.x, r4.y, r4.z), N2 = mk(r4.w, r5.x, r5.y);
    Shade o;
    o.pos = add(add(scl(V2, h.bu), scl(V0, h.bv)), scl(V1, h.bw));
    o.nrm = normalize(add(add(scl(N2, h.bu), scl(N0, h.bv)), scl(N1, h.bw)));
    o.gnrm = mk(r0.x, r0.y, r0.z);
    const DevMaterial& m = s.mats[__float_as_int(r0.w)];
    o.col = mk(m.color[0], m.color[1], m.color[2]);
    o.brdf = m.brdf;
    o.eta = m.eta;
    o.g = m.g;
    return o;
}

// col *= texture3D(VolumeTextureTextures, vec3(tex, r)).rgb when |tex.x| < 1e10 (eyeraytrace.fs:
// 443-446, photontrace.fs:418-422, 562-565), tex = T2 * b0 + T0 * b1 + T1 * b2 of the triangle's
// texture coordinates (eyeraytrace.fs:280); sampling as include/sppm_texture.h pins it
__device__ __forceinline__ f3 textured(const DevScene& S, int32_t tri, float b0, float b1, float b2, float r, f3 col) {
    const float2 T0 = __ldg(&S.tri_tex[(size_t)tri * 3]), T1 = __ldg(&S.tri_tex[(size_t)tri * 3 + 1]),
                 T2 = __ldg(&S.tri_tex[(size_t)tri * 3 + 2]);
    const float tu = xadd(xadd(xmul(T2.x, b0), xmul(T0.x, b1)), xmul(T1.x, b2));
    const float tv = xadd(xadd(xmul(T2.y, b0), xmul(T0.y, b1)), xmul(T1.y, b2));
    if (!(fabsf(tu) < 1e+10f)) return col;
    float t[3];
    sppm_tex_sample(S.tex, S.mat_layer, S.num_mats, tu, tv, r, t);
    return mk(xmul(col.x, t[0]), xmul(col.y, t[1]), xmul(col.z, t[2]));
}

// a photon bounce's colour: the hit's barycentrics from the stored position (photontrace.fs:
// 521-545), then the texture at layer (material + 0.5 + 0.25) / materials (:562-565)
__device__ __forceinline__ f3 textured_bounce(const DevScene& S, int32_t tri, f3 ipos, int32_t mat, f3 icol) {
    const float4* ts = S.tri_shade + (size_t)tri * 6;
    const float4 r1 = __ldg(ts + 1), r2 = __ldg(ts + 2), r3 = __ldg(ts + 3);
    const f3 V0 = mk(r1.x, r1.y, r1.z), V1 = mk(r1.w, r2.x, r2.y), V2 = mk(r2.z, r2.w, r3.x);
    const float bx = length(cross(sub(V1, V0), sub(ipos, V0)));
    const float by = length(cross(sub(V2, V1), sub(ipos, V1)));
    const float bz = length(cross(sub(V0, V2), sub(ipos, V2)));
    const float bs = xadd(xadd(bx, by), bz);
    return textured(S, tri, xdiv(bx, bs), xdiv(by, bs), xdiv(bz, bs),
                    xmul(S.mat_rcp, xadd(xadd((float)mat, 0.5f), 0.25f)), icol);
}

// ----------------------------------------------------------------------------------------------
// BRDF helpers (eyeraytrace.fs:293-392, photontrace.fs:60-89, 258-280, 443-461)
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ f3 onb(f3 x, f3 n) {
    if (n.z < -0.9999999f) return sub(scl(n, x.y), mk(x.z, x.x, 0.0f));
    const float a = xdiv(1.0f, xadd(1.0f, n.z));
    const float b = xmul(xmul(-n.x, n.y), a);
    const f3 u = mk(xsub(1.0f, xmul(xmul(n.x, n.x), a)), b, -n.x);
    const f3 w = mk(b, xsub(1.0f, xmul(xmul(n.y, n.y), a)), -n.y);
    return add(add(scl(u, x.x), scl(n, x.y)), scl(w, x.z));
}

__device__ __forceinline__ float fresnel(f3 incom, f3 normal, float ii, float ie) {
    const float eta = xdiv(ii, ie);
    const float c1 = dot(incom, normal);
    float c2 = xsub(1.0f, xmul(xmul(eta, eta), xsub(1.0f, xmul(c1, c1))));
    if (c2 < 0.0f) return 1.0f;
    c2 = xsqrt(c2);
    const float rs = xdiv(xsub(xmul(ii, c1), xmul(ie, c2)), xadd(xmul(ii, c1), xmul(ie, c2)));
    const float rp = xdiv(xsub(xmul(ii, c2), xmul(ie, c1)), xadd(xmul(ii, c2), xmul(ie, c1)));
    return xmul(xadd(xmul(rs, rs), xmul(rp, rp)), 0.5f);
}

__device__ __forceinline__ f3 glossy_reflect(f3 d, f3 n, float g, float4& rndv) {
    const f3 r = normalize(add(scl(reflect(d, n), xsub(xsub(1.0f, g), g)), scl(n, xadd(g, g))));
    const float rnd1 = gpu_rnd(rndv);
    const float rnd2 = gpu_rnd(rndv);
    const float temp1 = xmul(6.283184f, rnd1);
    const float temp2_ = sppm_fpow(rnd2, g);
    const float temp2 = xsqrt(xsub(1.0f, xmul(temp2_, temp2_)));
    float sn, cs;
    fsincos(temp1, sn, cs);
    const f3 v = mk(xmul(sn, temp2), temp2_, xmul(cs, temp2));
    f3 result = normalize(onb(v, r));
    if (dot(result, n) < 0.0f) result = reflect(result, n);
    return result;
}

__device__ __forceinline__ uint32_t grid_tid() { return blockIdx.x * blockDim.x + threadIdx.x; }

// ----------------------------------------------------------------------------------------------
// k_frame_begin: clear the hashed grid of every job; per-job bookkeeping by the job's slot 0
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ float xorshift_frand(uint32_t* s) {
    const uint32_t t = s[0] ^ (s[0] << 11);
    s[0] = s[1];
    s[1] = s[2];
    s[2] = s[3];
    s[3] = (s[3] ^ (s[3] >> 19)) ^ (t ^ (t >> 8));
    return xmul(__uint2float_rn(s[3]), 1.0f / 4294967295.0f);
}

// a job's state at the start of a frame
__device__ __forceinline__ void begin_job(const JobDesc& J) {
    JobState* st = J.state;
    const uint32_t f = st->frames_started;
    st->frame = f;
    st->frames_started = f + 1;
    st->emitted_frame = 0;
    st->segments_frame = 0;
    const uint32_t interval = J.eye_interval ? J.eye_interval : 1u;
    st->is_eye_frame = (f % interval) == 0;
    if (st->is_eye_frame) {
        // AAOffset (glslppm.cpp:276-277)
        st->aa[0] = xmul(xsub(xorshift_frand(st->xs), 0.5f), 1.25f);
        st->aa[1] = xmul(xsub(xorshift_frand(st->xs), 0.5f), 1.25f);
        st->eye_samples += 1;
        for (int c = 0; c < 3; c++) {
            st->bbmax_key[c] = 0u;           // below every float
            st->bbmin_key[c] = 0xFFFFFFFFu;  // above every float
        }
    }
}
// (four hash slots and four bins a thread: one search for the job and two wide stores)
__global__ void k_frame_begin(LaunchSet ls, RayQueue q) {
    const uint32_t t = grid_tid();
    if (t == 0 && q.counters) {
        q.counters[0] = 0;
        q.counters[1] = 0;
        q.counters[2] = 0;
        q.counters[3] = 0;
        q.counters[4] = 0;
        q.counters[7] += 1u;  // frames since the bins were last reordered
    }
    static_assert(kBinCounters * kRayBins % 4 == 0, "bins must split into uint4");
    if (q.bins && t < kBinCounters * kRayBins / 4) reinterpret_cast<uint4*>(q.bins)[t] = make_uint4(0u, 0u, 0u, 0u);
    if (t > (ls.total - 1u) / 4u) return;
    const uint32_t g = 4u * t, n = min(ls.total - g, 4u);
    const int k = find_job(ls, g);
    const JobDesc& J = job_of(ls, k);
    const uint32_t local = g - first_item(ls, k);
    if (n == 4u && local + 4u <= J.hash_num && local % 4u == 0u) {
        *reinterpret_cast<uint4*>(J.winner + local) = make_uint4(kEmptySlot, kEmptySlot, kEmptySlot, kEmptySlot);
        *reinterpret_cast<uint4*>(J.count + local) = make_uint4(0u, 0u, 0u, 0u);
        if (local == 0) begin_job(J);
        return;
    }
    for (uint32_t i = g; i < g + n; i++) {
        const int ki = find_job(ls, i);
        const JobDesc& Ji = job_of(ls, ki);
        const uint32_t li = i - first_item(ls, ki);
        Ji.winner[li] = kEmptySlot;
        Ji.count[li] = 0;
        if (li == 0) begin_job(Ji);
    }
}

// the photon ray queue emptied for the next wave of the photon pass (the eye pass's deferred
// pixel count, counters[3], belongs to the eye branch running beside the waves and is kept)
__global__ void k_queue_reset(RayQueue q) {
    const uint32_t g = grid_tid();
    if (g == 0) {
        q.counters[0] = 0;
        q.counters[1] = 0;
        q.counters[2] = 0;
        q.counters[4] = 0;
    }
    if (q.bins && g < kBinCounters * kRayBins) q.bins[g] = 0u;
}

// ----------------------------------------------------------------------------------------------
// k_eye: eyeraytrace.fs main (:396-554) + max/min reduction of the hit positions
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void warp_bbox_atomics(JobState* st, f3 p, int job_k) {
    // lanes of the same job combine with warp reductions; the leader issues one atomic per
    // component; a NaN component is ignored, as fminf/fmaxf ignore it
    const unsigned mask = __match_any_sync(__activemask(), job_k);
    const float v[3] = {p.x, p.y, p.z};
    for (int c = 0; c < 3; c++) {
        const bool ok = v[c] == v[c];
        uint32_t kmx = ok ? float_key(v[c]) : 0u;
        uint32_t kmn = ok ? float_key(v[c]) : 0xFFFFFFFFu;
        kmx = __reduce_max_sync(mask, kmx);
        kmn = __reduce_min_sync(mask, kmn);
        // An add to one address takes the GPU 0.7 ns, so six per warp were 137 us of the eye pass at
        // 1024^2.  The bounds only grow: one read earlier (also a stale one, from L1) that already holds
        // the warp's bounds makes the atomic unnecessary, as for nearly all warps.
        if ((threadIdx.x & 31) == (__ffs(mask) - 1)) {
            if (kmx > __ldca(&st->bbmax_key[c])) atomicMax(&st->bbmax_key[c], kmx);
            if (kmn < __ldca(&st->bbmin_key[c])) atomicMin(&st->bbmin_key[c], kmn);
        }
    }
}

// eye rays of the mixed path walk the 4-wide quantised BVH (the material comes from the triangle)
__device__ __forceinline__ Hit trace_eye4(const DevScene& s, f3 org, f3 dir, bool cull, uint32_t& err) {
    const Hit4 h4 = trace4<false>(s.nodes4, s.tri_isect, org, dir, cull, 1.0e20f, err,
                                  s.tri_rank ? s.tri_rank + (size_t)cube_face(dir) * s.num_tris : nullptr);
    Hit h;
    h.t = h4.t;
    h.tri = h4.tri;
    h.mat = h4.tri >= 0 ? __float_as_int(__ldg(&s.tri_isect[(size_t)h4.tri * 3 + 2]).y) : -1;
    h.bu = h4.bu;
    h.bv = h4.bv;
    h.bw = h4.bw;
    return h;
}

// the eye path of one pixel (eyeraytrace.fs main :396-554) up to its outputs; `trace(org, dir,
// cull, hit)` finds the closest hit and may decline (returns false), which abandons the path
// without side effects so that it can be rerun from its stored state
struct EyeOut {
    f3 pos, col, nrm, rdir, emi;
    float4 rndv;
    Hit last;
    uint32_t segs;
};

// TEX: the launch may hold a job whose scene has texture coordinates (texture lookups compiled in)
template <bool TEX, class Trace>
__device__ __forceinline__ bool eye_path(const JobDesc& J, const JobState* st, uint32_t p, Trace&& trace, EyeOut& out) {
    const uint32_t px = p % J.W, py = p / J.W;
    const DevScene& S = J.scene;
    float4 rndv = J.px.rng[p];
    const float eps = 1e-5f;
    const f3 U = mk(J.cam_u[0], J.cam_u[1], J.cam_u[2]);
    const f3 V = mk(J.cam_v[0], J.cam_v[1], J.cam_v[2]);
    const f3 Wd = mk(J.cam_w[0], J.cam_w[1], J.cam_w[2]);
    const f3 CP = mk(J.cam_pos[0], J.cam_pos[1], J.cam_pos[2]);
    const float aax = st->aa[0], aay = st->aa[1];
    const float ppx = xsub(xadd(xadd((float)px, 0.5f), aax), J.cam_cx);
    const float ppy = xsub(xadd(xadd((float)py, 0.5f), aay), J.cam_cy);
    f3 rdir = normalize(add(add(scl(U, ppx), scl(V, ppy)), scl(Wd, J.cam_dist)));
    f3 rorg;
    const float filter = xmul(xsub(1.0f, xdiv(fabsf(aax), 1.5f)), xsub(1.0f, xdiv(fabsf(aay), 1.5f)));
    {
        const f3 fp = add(CP, scl(rdir, J.focal));
        const float radius = xmul(xsqrt(gpu_rnd(rndv)), J.aperture);
        const float theta = xmul(6.283184f, gpu_rnd(rndv));
        float sn, cs;
        fsincos(theta, sn, cs);
        const f3 lens = add(CP, scl(add(scl(U, cs), scl(V, sn)), radius));
        rdir = normalize(sub(fp, lens));
        rorg = lens;
    }
    f3 col = mk(filter, filter, filter);
    f3 nrm = mk(0, 0, 0), pos = mk(0, 0, 0), emi = mk(0, 0, 0);
    Hit last;
    last.tri = -1;
    last.t = 1.0e20f;
    uint32_t segs = 0;
    for (uint32_t j = 0; j < J.max_path; j++) {
        Hit h;
        if (!trace(rorg, rdir, j == 0, h)) return false;  // deferred to the block-wide pass
        last = h;
        segs++;
        if (h.tri < 0) {
            nrm = mk(0, 0, 0);
            if (S.light_area == 0.0f) emi = mul(mk(0.7f, 0.7f, 1.0f), col);
            break;
        }
        Shade i = shade_hit(S, h);
        pos = i.pos;
        nrm = i.nrm;
        if (TEX && S.tri_tex)
            i.col = textured(S, h.tri, h.bu, h.bv, h.bw, xmul(S.mat_rcp, xadd((float)h.mat, 0.5f)), i.col);
        if (i.brdf == -1) {
            nrm = mk(0, 0, 0);
            emi = mul(col, i.col);
            break;
        } else if (i.brdf == 0) {
            col = mul(col, i.col);
            break;
        } else if (i.brdf == 1 || i.brdf == 4) {
            rorg = add(pos, scl(i.gnrm, eps));
            if (i.brdf == 4) nrm = glossy_reflect(nrm, nrm, i.g, rndv);
            rdir = reflect(rdir, nrm);
            if (dot(rdir, i.gnrm) < 0.0f) rdir = neg(rdir);
            col = mul(col, i.col);
        } else if (i.brdf == 2 || i.brdf == 5) {
            if (i.brdf == 5) nrm = glossy_reflect(nrm, nrm, i.g, rndv);
            const float ln = dot(nrm, rdir);
            if (ln < 0.0f) {
                const float re = fresnel(neg(rdir), nrm, 1.0f, i.eta);
                if (gpu_rnd(rndv) < re) {
                    rorg = add(pos, scl(i.gnrm, eps));
                    rdir = reflect(rdir, nrm);
                    if (dot(rdir, i.gnrm) < 0.0f) rdir = neg(rdir);
                } else {
                    col = mul(col, i.col);
                    rorg = sub(pos, scl(i.gnrm, eps));
                    rdir = refract(rdir, nrm, xdiv(1.0f, i.eta));
                    if (dot(rdir, i.gnrm) > 0.0f) rdir = neg(rdir);
                }
            } else {
                const float re = fresnel(neg(rdir), neg(nrm), i.eta, 1.0f);
                col = mul(col, i.col);
                if (gpu_rnd(rndv) < re) {
                    rorg = sub(pos, scl(i.gnrm, eps));
                    rdir = reflect(rdir, neg(nrm));
                    if (dot(rdir, neg(i.gnrm)) < 0.0f) rdir = neg(rdir);
                } else {
                    rorg = add(pos, scl(i.gnrm, eps));
                    rdir = refract(rdir, neg(nrm), i.eta);
                    if (dot(rdir, neg(i.gnrm)) > 0.0f) rdir = neg(rdir);
                }
            }
        } else if (i.brdf == 3 || i.brdf == 6) {
            if (i.brdf == 6) nrm = glossy_reflect(nrm, nrm, i.g, rndv);
            const float re = fresnel(neg(rdir), nrm, 1.0f, i.eta);
            if (gpu_rnd(rndv) < re) {
                rorg = add(pos, scl(i.gnrm, eps));
                rdir = reflect(rdir, nrm);
                if (dot(rdir, i.gnrm) < 0.0f) rdir = neg(rdir);
            } else {
                col = mul(col, i.col);
                break;
            }
        }
    }
    out.pos = pos;
    out.col = col;
    out.nrm = nrm;
    out.rdir = rdir;
    out.emi = emi;
    out.rndv = rndv;
    out.last = last;
    out.segs = segs;
    return true;
}

// the pixel outputs of a finished eye path (the running emission mean of :543-545)
__device__ __forceinline__ void eye_write(const JobDesc& J, const JobState* st, uint32_t p, const EyeOut& o) {
    float4 qe = J.px.emi_n[p];
    const float a = xdiv(1.0f, (float)st->eye_samples);
    const float oma = xsub(1.0f, a);
    qe.x = xadd(xmul(qe.x, oma), xmul(o.emi.x, a));
    qe.y = xadd(xmul(qe.y, oma), xmul(o.emi.y, a));
    qe.z = xadd(xmul(qe.z, oma), xmul(o.emi.z, a));
    J.px.pos[p] = f4(o.pos, o.rdir.x);
    J.px.refl[p] = f4(o.col, o.rdir.y);
    J.px.nrm[p] = f4(o.nrm, o.rdir.z);
    J.px.rng[p] = o.rndv;
    J.px.tri[p] = o.last.tri;
    J.px.t[p] = o.last.t;
    J.px.emi_n[p] = qe;
}

// the pixel of item `item` of a job whose pixels a launch covers in 8x4 tiles (a warp's worth of items
// each); false: the tile reaches over the image's edge there
__device__ __forceinline__ bool tile_pixel(const JobDesc& J, uint32_t item, uint32_t& p) {
    const uint32_t tw = (J.W + 7u) >> 3, tile = item >> 5, lane = item & 31u, ty = tile / tw;
    const uint32_t px = (tile - ty * tw) * 8u + (lane & 7u), py = ty * 4u + (lane >> 3);
    p = py * J.W + px;
    return px < J.W && py < J.H;
}

// eye pass, one thread per pixel.  A ray with a zero direction component (slab_degenerate)
// would walk most of the tree in one lane: the exact path defers such pixels to k_eye_coop
// (their whole path is rerun there with block-wide walks); the mixed path's slab tests do not
// degenerate.
//
// Bound by the divergence of a warp's paths and by the node loads' latency.  A warp takes an 8x4 tile: its
// rays spread less than a row of 32 pixels does, so they share more nodes and end closer together.  Us a
// pass of ten with one eye frame, rows -> tiles: a 1024^2 frame of a 1M-triangle mesh 1057 -> 1049, sixteen
// 512^2 frames 1043 -> 1029, the Cornell box at 1024^2 302 -> 301; and 8 resident blocks (64 registers;
// spills of 44 bytes stored, 28 loaded) 1049 -> 1044, 1029 -> 1025, 301 -> 301.  The textured path gets 6
// (80 registers): us a pass of the textured box with an eye pass in each and 1024^2 photons, 5 / 6 / 8
// blocks, plain 505 / 489 / 475 at 1024^2 pixels and 697 / 666 / 636 at 1536^2, mixed 514 / 502 / 500 and
// 715 / 691 / 684; with 512^2 photons 179.4 / 178.5 / 184.6 and 181.5 / 180.0 / 181.2 at 512^2, with 256^2
// 126.0 / 126.2 / 127.5 and 102.5 / 102.8 / 103.9 at 256^2.
// FEW (untextured launches of few items): the exact path walks a step ahead, the mixed one has more
// registers.
//
// Up to kEyeAheadItems the exact path's walk loads a step ahead: with few warps the paths' chains decide.
// Us a pass without / with it, an eye pass in each, 1024x512 photons: glass and glossy spheres 433 / 366 at
// 256^2 pixels, 465 / 407 at 512^2, 514 / 479 at 768^2, 604 / 597 at 1024^2, 901 / 937 at 1536^2; Cornell
// box 172 / 174, 192 / 198, 232 / 243, 289 / 307, 422 / 463; 102k-triangle mesh 282 / 266, 308 / 321, 369 / 400,
// 449 / 500, 654 / 754.  Up to 2^18 the long paths gain more than the short ones lose (with an eye pass in
// ten: glass 232 / 225 at 256^2, 243 / 237 at 512^2, box 164 / 164, 169 / 170, mesh 244 / 245, 252 / 253).
constexpr uint32_t kEyeAheadItems = 1u << 18;
// The mixed path's walk has no such chain to shorten, but at 8 blocks it spills (112 bytes stored, 280
// loaded): up to kEyeMixedItems it runs with all 91 registers (5 blocks).  Us a pass, 8 / 5 blocks, as above:
// glass and glossy spheres 368 / 356 at 256^2, 443 / 406 at 512^2, 474 / 436 at 640x600, 526 / 492 at 768^2,
// 661 / 631 at 1024^2, 1022 / 1041 at 1536^2; Cornell box 175 / 173, 202 / 201, 216 / 217, 242 / 247, 298 / 311,
// 459 / 483; 102k-triangle mesh 262 / 259, 315 / 315, 341 / 344, 389 / 394, 483 / 499, 738 / 780.
constexpr uint32_t kEyeMixedItems = 1u << 19;
template <bool MIXED, bool TEX, bool FEW = false>
__global__ void __launch_bounds__(128, TEX ? 6 : FEW ? (MIXED ? 5 : 6) : 8)
    k_eye(LaunchSet ls, uint32_t* deferred_n, uint32_t* deferred, uint32_t deferred_cap) {
    // the block's segment count for the job of its first item: one global add per block, made by the
    // last of its threads to get there (no barrier: the others' registers are free when their paths
    // have ended; lanes of one warp may get there apart)
    __shared__ uint32_t s_segs, s_threads;
    if (threadIdx.x == 0) s_segs = s_threads = 0u;
    __syncthreads();
    const uint32_t g = grid_tid();
    if (g >= ls.total) return;
    const int k = find_job(ls, g);
    const JobDesc& J = job_of(ls, k);
    JobState* st = J.state;
    uint32_t p, err = 0;
    EyeOut o;
    const bool live = tile_pixel(J, g - first_item(ls, k), p);
    const bool done = live && eye_path<TEX>(J, st, p, [&](f3 org, f3 dir, bool cull, Hit& h) {
        if (MIXED) {
            h = trace_eye4(J.scene, org, dir, cull, err);
            return true;
        }
        if (slab_degenerate(dir)) {
            const uint32_t slot = atomicAdd(deferred_n, 1u);
            if (slot < deferred_cap) {
                deferred[slot] = g;
                return false;
            }
        }
        h = trace_exact<false, false, FEW>(J.scene, org, dir, cull, err);
        return true;
    }, o);
    if (done) eye_write(J, st, p, o);
    const f3 bpos = done ? o.pos : mk(__int_as_float(0x7FC00000), __int_as_float(0x7FC00000), __int_as_float(0x7FC00000));
    warp_bbox_atomics(st, bpos, k);  // a deferred pixel contributes nothing (NaN is ignored)
    // segment count and errors: one add per warp and job
    const unsigned active = __activemask();
    const unsigned mask = __match_any_sync(active, k);
    const uint32_t wsegs = __reduce_add_sync(mask, done ? o.segs : 0u);
    const uint32_t werr = __reduce_or_sync(mask, err);
    const uint32_t first = blockIdx.x * blockDim.x;
    const int block_k = find_job(ls, first);
    if ((threadIdx.x & 31) == (__ffs(mask) - 1)) {
        if (k == block_k) atomicAdd(&s_segs, wsegs);
        else atomicAdd(&st->eye_segments, (unsigned long long)wsegs);
        if (werr) atomicOr(&st->err, werr);
    }
    __syncwarp(active);
    if ((threadIdx.x & 31) == (__ffs(active) - 1)) {
        __threadfence_block();
        const uint32_t n_active = __popc(active);
        if (atomicAdd(&s_threads, n_active) + n_active == min(blockDim.x, ls.total - first)) {
            __threadfence_block();
            const uint32_t n = atomicAdd(&s_segs, 0u);
            if (n) atomicAdd(&job_of(ls, block_k).state->eye_segments, (unsigned long long)n);
        }
    }
}

// the deferred pixels of k_eye<false>, one block of 1024 threads per pixel: every thread runs
// the same path (identical values), each trace is block_trace_exact, thread 0 writes
template <bool TEX>
__global__ void __launch_bounds__(kBlockWalk) k_eye_coop(LaunchSet ls, const uint32_t* deferred_n,
                                                         const uint32_t* deferred, uint32_t deferred_cap) {
    __shared__ BlockWalkShared sh;
    const uint32_t n = min(*deferred_n, deferred_cap);
    for (uint32_t w = blockIdx.x; w < n; w += gridDim.x) {
        const uint32_t g = deferred[w];
        const int k = find_job(ls, g);
        const JobDesc& J = job_of(ls, k);
        JobState* st = J.state;
        uint32_t p, err = 0;
        tile_pixel(J, g - first_item(ls, k), p);
        EyeOut o;
        eye_path<TEX>(J, st, p, [&](f3 org, f3 dir, bool cull, Hit& h) {
            TraversalCount ct;
            h = block_trace_exact<false, false>(J.scene, org, dir, cull, err, &ct, sh);
            return true;
        }, o);
        if (threadIdx.x == 0) {
            eye_write(J, st, p, o);
            const float v[3] = {o.pos.x, o.pos.y, o.pos.z};
            for (int c = 0; c < 3; c++) {
                if (!(v[c] == v[c])) continue;
                atomicMax(&st->bbmax_key[c], float_key(v[c]));
                atomicMin(&st->bbmin_key[c], float_key(v[c]));
            }
            atomicAdd(&st->eye_segments, (unsigned long long)o.segs);
            if (err) atomicOr(&st->err, err);
        }
        __syncthreads();
    }
}

// ----------------------------------------------------------------------------------------------
// k_grid: glslppm.cpp:292-311 for every job in an eye frame (one thread per job)
// ----------------------------------------------------------------------------------------------
__global__ void k_grid(const JobDesc* jobs, const uint32_t* job_ids, uint32_t njobs) {
    const uint32_t k = grid_tid();
    if (k >= njobs) return;
    const JobDesc& J = jobs[job_ids[k]];
    JobState* st = J.state;
    float mx[3], mn[3];
    for (int c = 0; c < 3; c++) {
        mx[c] = key_float(st->bbmax_key[c]);
        mn[c] = key_float(st->bbmin_key[c]);
    }
    float r0;
    if (J.radius_rule == SPPM_RADIUS_DIAGONAL) {
        r0 = J.fixed_radius;
    } else {
        float bbsize = 0.0f;
        for (int c = 0; c < 3; c++) bbsize = xadd(bbsize, xsub(mx[c], mn[c]));
        r0 = xmul(xdiv(xdiv(bbsize, 3.0f), (float)J.W), J.footprint);
    }
    st->initial_radius = r0;
    for (int c = 0; c < 3; c++) {
        st->bbmin[c] = xsub(mn[c], r0);
        st->bbmax[c] = xadd(mx[c], r0);
    }
    st->grid_scale = xdiv(0.5f, r0);
    st->hash_scale1 = xdiv(4194304.0f, st->grid_scale);
    if (st->frame == 0) st->r0 = r0;
}

// k_cell_bounds: the in-cell test's bounds (progressive.fs:79-81: cell / GridScale + BBMin, with the
// test's own correctly rounded division and addition) for every integer cell coordinate of the
// grid k_grid has just set, a block per job of the eye phase
__global__ void __launch_bounds__(256) k_cell_bounds(const JobDesc* jobs, const uint32_t* job_ids) {
    const JobDesc& J = jobs[job_ids[blockIdx.x]];
    if (!J.cell_bounds) return;
    JobState* st = J.state;
    const float G = st->grid_scale;
    uint32_t n = 0;
    for (int a = 0; a < 3; a++) {
        const float e = xmul(xsub(st->bbmax[a], st->bbmin[a]), G);  // cells along the axis
        const uint32_t na = e >= 0.0f && e < (float)kCellTable ? (uint32_t)e + 3u : kCellTable;
        n = max(n, na);
    }
    n = min(n, kCellTable);
    for (uint32_t i = threadIdx.x; i < 3 * n; i += blockDim.x) {
        const uint32_t a = i / n, c = i - a * n;
        J.cell_bounds[a * kCellTable + c] = xadd(xdiv((float)c, G), st->bbmin[a]);
    }
    if (threadIdx.x == 0) st->cell_table_n = n;
}

// ----------------------------------------------------------------------------------------------
// k_photon: photontrace.fs main (:464-720), sum.fs, hash.fs + scatter.vs + correction.vs
// ----------------------------------------------------------------------------------------------
// GenerateLightSourceSample (photontrace.fs:345-440) up to its cosine lobe: the origin, the flux and
// the lobe's normal (the lobe itself is cosine_lobe, drawn right after, shared with the bounces)
template <bool TEX>
__device__ __forceinline__ void light_sample(const JobDesc& J, float4& rndv, f3& flux, f3& lobe_n, f3& org,
                                             uint32_t& err) {
    const DevScene& S = J.scene;
    const float rnd = gpu_rnd(rndv);
    int low = 0;
    int high = (int)xadd(xdiv(1.0f, S.light_stride), 0.5f);
    const int nl = (int)S.num_lights;
    // texel of search step `mid` at texcoord (mid - 0.5)*stride: index mid-1, clamped
    int guard = 0;
    while (low < high) {
        if (++guard > 64) {
            err |= kErrWatchdogLight;
            break;
        }
        const int mid = low + ((high - low) / 2);
        const int kk = min(max(mid - 1, 0), nl - 1);
        if (__ldg(&S.light_cdf[kk]) < rnd) low = mid + 1;
        else high = mid;
    }
    const int32_t lt = __ldg(&S.light_tri[min(max(high - 1, 0), nl - 1)]);
    const float rndv2 = gpu_rnd(rndv);
    const float t = xsqrt(xsub(1.0f, rndv2));
    const float sv = gpu_rnd(rndv);
    const float a = xsub(1.0f, t);
    const float c = xmul(sv, t);
    const float b = xsub(t, c);
    const float4* ts = S.tri_shade + (size_t)lt * 6;
    const float4 r0 = __ldg(ts + 0), r1 = __ldg(ts + 1), r2 = __ldg(ts + 2);
    const float4 r3 = __ldg(ts + 3), r4 = __ldg(ts + 4), r5 = __ldg(ts + 5);
    const f3 V0 = mk(r1.x, r1.y, r1.z), V1 = mk(r1.w, r2.x, r2.y), V2 = mk(r2.z, r2.w, r3.x);
    const f3 N0 = mk(r3.y, r3.z, r3.w), N1 = mk(r4.x, r4.y, r4.z), N2 = mk(r4.w, r5.x, r5.y);
    const DevMaterial& m = S.mats[__float_as_int(r0.w)];
    flux = scl(mk(m.color[0], m.color[1], m.color[2]), xmul(S.light_area, 3.141592f));
    if (TEX && S.tri_tex)  // T = T2 * c + T0 * a + T1 * b (photontrace.fs:413-422)
        flux = textured(S, lt, c, a, b, xmul(S.mat_rcp, xadd((float)__float_as_int(r0.w), 0.75f)), flux);
    f3 o = add(add(scl(V0, a), scl(V1, b)), scl(V2, c));
    const f3 nrm = normalize(add(add(scl(N0, a), scl(N1, b)), scl(N2, c)));
    const f3 gnrm = mk(r0.x, r0.y, r0.z);
    o = add(o, scl(gnrm, 1.0e-5f));
    lobe_n = nrm;
    org = o;
}

// cosine lobe around n (photontrace.fs:432-439 for emission, :567-578 for matte bounces): two draws
__device__ __forceinline__ f3 cosine_lobe(float4& rndv, f3 n) {
    const float r0 = xmul(6.283184f, gpu_rnd(rndv));
    const float r1 = xsqrt(gpu_rnd(rndv));
    float sn, cs;
    fsincos(r0, sn, cs);
    return onb(mk(xmul(sn, r1), xsqrt(xsub(1.0f, xmul(r1, r1))), xmul(cs, r1)), n);
}

__device__ __forceinline__ void ibl_sample(const JobDesc& J, float4& rndv, f3& flux, f3& dir, f3& org) {
    const float* bs = J.scene.bsphere;
    const float area = xmul(xmul(12.566368f, bs[3]), bs[3]);
    const float temp2 = xmul(6.283184f, gpu_rnd(rndv));
    const float aaa = xsqrt(xsub(1.0f, gpu_rnd(rndv)));
    const float sinA = sppm_fsin(aaa);
    const float sinTemp1 = xmul(xadd(sinA, sinA), sppm_fcos(aaa));
    f3 d = mk(xmul(sinTemp1, sppm_fcos(temp2)), xsub(1.0f, xmul(xadd(sinA, sinA), sinA)), xmul(sinTemp1, sppm_fsin(temp2)));
    if (gpu_rnd(rndv) > 0.5f) {
        d = mk(1.0f, 1.0f, 1.0f);
        d.y = xadd(d.y, d.y);
        d.z = -d.z;
        d = normalize(d);
        flux = scl(mk(1.0f, 1.0f, 0.7f), area);
    } else {
        flux = scl(mk(0.7f, 0.7f, 1.0f), area);
    }
    const float radius = xsqrt(gpu_rnd(rndv));
    const float theta = xmul(6.283184f, gpu_rnd(rndv));
    const f3 temp = mk(xmul(radius, sppm_fcos(theta)), 0.0f, xmul(radius, sppm_fsin(theta)));
    org = add(add(onb(scl(temp, bs[3]), d), scl(d, bs[3])), mk(bs[0], bs[1], bs[2]));
    dir = neg(d);
}

// emit a photon or bounce the stored one (photontrace.fs main :464-686): the ray of this pass
struct PhotonRay {
    f3 org, dir, flux;
    float depth;
    bool cont;
    uint32_t emitted;
};

// hitin: the previous segment's (triangle, depth), (-1, 0) before the first; PP, PF, PD: its
// record (position, flux, direction, with the normal in the w components)
template <bool TEX>
__device__ __forceinline__ PhotonRay photon_generate(const JobDesc& J, int2 hitin, float4 PP, float4 PF, float4 PD,
                                                     float4& rndv, uint32_t& err) {
    // Emission and the diffuse bounces end in the same cosine lobe: each path sets up its lobe
    // (normal, origin; the draws before the lobe stay in the path) and the lanes draw the lobe
    // together, then finish their path (the flip against the geometric normal, Russian roulette).
    const DevScene& S = J.scene;
    const float eps = 1e-6f;
    PhotonRay R;
    R.org = mk(0, 0, 0);
    R.dir = mk(0, 0, 0);
    R.depth = xadd((float)hitin.y, 1.0f);
    const bool emit = hitin.x < 0 || R.depth >= (float)J.max_path;
    bool lobe = false, flip = false;
    f3 lobe_n = mk(0, 0, 0), gnrm = mk(0, 0, 0), icol = mk(0, 0, 0), flux = mk(0, 0, 0);
    f3 rorg = mk(0, 0, 0), rdir = mk(0, 0, 0);
    if (emit) {
        if (S.light_area != 0.0f) {
            light_sample<TEX>(J, rndv, R.flux, lobe_n, rorg, err);
            lobe = true;
        } else {
            ibl_sample(J, rndv, R.flux, rdir, rorg);
        }
    } else {
        flux = mk(fabsf(PF.x), fabsf(PF.y), fabsf(PF.z));
        const f3 ipos = xyz(PP);
        f3 inrm = mk(PP.w, PF.w, PD.w);
        const f3 pd = xyz(PD);
        const float4 r0 = __ldg(S.tri_shade + (size_t)hitin.x * 6);
        gnrm = mk(r0.x, r0.y, r0.z);
        const DevMaterial& m = S.mats[__float_as_int(r0.w)];
        icol = mk(m.color[0], m.color[1], m.color[2]);
        if (TEX && S.tri_tex) icol = textured_bounce(S, hitin.x, ipos, __float_as_int(r0.w), icol);
        const int brdf = m.brdf;
        if (brdf == 0) {
            rorg = add(ipos, scl(gnrm, eps));  // matte_bounce
            lobe_n = inrm;
            lobe = flip = true;
        } else if (brdf == 1 || brdf == 4) {
            rorg = add(ipos, scl(gnrm, eps));
            if (brdf == 4) inrm = glossy_reflect(inrm, inrm, m.g, rndv);
            rdir = reflect(pd, inrm);
            if (dot(rdir, gnrm) < 0.0f) rdir = neg(rdir);
        } else if (brdf == 2 || brdf == 5) {
            if (brdf == 5) inrm = glossy_reflect(inrm, inrm, m.g, rndv);
            const float ln = dot(inrm, pd);
            if (ln < 0.0f) {
                const float re = fresnel(neg(pd), inrm, 1.0f, m.eta);
                if (gpu_rnd(rndv) < re) {
                    rorg = add(ipos, scl(gnrm, eps));
                    rdir = reflect(pd, inrm);
                    icol = mk(1.0f, 1.0f, 1.0f);
                    if (dot(rdir, gnrm) < 0.0f) rdir = neg(rdir);
                } else {
                    rorg = sub(ipos, scl(gnrm, eps));
                    rdir = refract(pd, inrm, xdiv(1.0f, m.eta));
                    if (dot(rdir, gnrm) > 0.0f) rdir = neg(rdir);
                }
            } else {
                const float re = fresnel(neg(pd), neg(inrm), m.eta, 1.0f);
                if (gpu_rnd(rndv) < re) {
                    rorg = sub(ipos, scl(gnrm, eps));
                    rdir = reflect(pd, neg(inrm));
                    if (dot(rdir, neg(gnrm)) < 0.0f) rdir = neg(rdir);
                } else {
                    rorg = add(ipos, scl(gnrm, eps));
                    rdir = refract(pd, neg(inrm), m.eta);
                    if (dot(rdir, neg(gnrm)) > 0.0f) rdir = neg(rdir);
                }
            }
        } else if (brdf == 3 || brdf == 6) {
            if (brdf == 6) inrm = glossy_reflect(inrm, inrm, m.g, rndv);
            const float re = fresnel(neg(pd), inrm, 1.0f, m.eta);
            if (gpu_rnd(rndv) < re) {
                rorg = add(ipos, scl(gnrm, eps));
                rdir = reflect(pd, inrm);
                icol = mk(1.0f, 1.0f, 1.0f);
                if (dot(rdir, gnrm) < 0.0f) rdir = neg(rdir);
            } else {
                rorg = add(ipos, scl(gnrm, eps));  // matte_bounce
                lobe_n = inrm;
                lobe = flip = true;
            }
        }
    }
    if (lobe) {
        rdir = cosine_lobe(rndv, lobe_n);
        if (flip && dot(rdir, gnrm) < 0.0f) rdir = neg(rdir);
    }
    R.org = rorg;
    R.dir = rdir;
    if (emit) {
        R.emitted = 1;
        R.depth = 0.0f;
        R.cont = true;
        return R;
    }
    // Russian roulette (:671-685)
    const float pmax = fmaxf(fmaxf(icol.x, icol.y), icol.z);
    if (pmax < gpu_rnd(rndv)) {
        R.cont = false;
    } else {
        R.cont = true;
        icol = mk(xdiv(icol.x, pmax), xdiv(icol.y, pmax), xdiv(icol.z, pmax));
        flux = mul(flux, icol);
    }
    R.emitted = 0;
    R.flux = flux;
    return R;
}

template <bool TEX>
__device__ __forceinline__ PhotonRay photon_generate(const JobDesc& J, uint32_t sidx, uint32_t frame, float4& rndv,
                                                     uint32_t& err) {
    const int2 hitin = frame == 0 ? make_int2(-1, 0) : J.ph.hit[sidx];
    return photon_generate<TEX>(J, hitin, J.ph.pos[sidx], J.ph.flux[sidx], J.ph.dir[sidx], rndv, err);
}

__device__ __forceinline__ void photon_terminate(const JobDesc& J, uint32_t sidx) {
    J.ph.pos[sidx] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    J.ph.flux[sidx] = make_float4(-1.0f, -1.0f, -1.0f, 0.0f);
    J.ph.dir[sidx] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    J.ph.hit[sidx] = make_int2(-1, 0);
}

// store the traced photon (photontrace.fs :692-709); returns the hash slot or 0xFFFFFFFF
// (jobs with SPPM_FLAG_PHOTON_GRID: the slot of the counting-sort grid's cell, split grid_shift
// times, or 0xFFFFFFFF for a photon outside the grid)
__device__ __forceinline__ uint32_t photon_store(const JobDesc& J, const JobState* st, uint32_t sidx, const Hit& h,
                                                 f3 rdir, f3 flux, float depth, uint32_t grid_shift = 0) {
    const DevScene& S = J.scene;
    f3 ppos = mk(0, 0, 0), pnrm = mk(0, 0, 0), pg = mk(0, 0, 0);
    int brdf = 0;
    if (h.tri >= 0) {
        const Shade i = shade_hit(S, h);
        ppos = i.pos;
        pnrm = i.nrm;
        pg = i.gnrm;
        brdf = i.brdf;
    }
    if (h.tri < 0 || (brdf != 0 && brdf != 6 && brdf != 3)) flux = neg(flux);
    const float gf = fminf(fabsf(xdiv(dot(rdir, pnrm), dot(rdir, pg))), 2.236068010e+00f);
    flux = scl(flux, gf);
    J.ph.pos[sidx] = f4(ppos, pnrm.x);
    J.ph.flux[sidx] = f4(flux, pnrm.y);
    J.ph.dir[sidx] = f4(rdir, pnrm.z);
    J.ph.hit[sidx] = make_int2(h.tri, (int)depth);
    if (flux.x < 0.0f) return 0xFFFFFFFFu;
    if (J.flags & SPPM_FLAG_PHOTON_GRID) return grid_photon_slot(J, st, grid_shift, ppos.x, ppos.y, ppos.z);
    // hash.fs main (:51-68): cell = floor((p - BBoxMin) * GridScale), slot = hash(cell)
    const f3 cell = mk(floorf(xmul(xsub(ppos.x, st->bbmin[0]), st->grid_scale)),
                       floorf(xmul(xsub(ppos.y, st->bbmin[1]), st->grid_scale)),
                       floorf(xmul(xsub(ppos.z, st->bbmin[2]), st->grid_scale)));
    return hash_cell(cell, st->grid_scale, st->hash_scale1, (float)J.hash_num);
}

// scatter.vs + depth test and correction.vs + blend, one atomic pair per warp and slot.
//
// A warp's photons mostly fall into slots of their own.  A reduction whose mask is each lane's peers
// runs once per distinct mask, so those lanes add and compare for themselves, together, and only lanes
// with peers reduce.  Us of the store, a reduction for every slot -> this: the Cornell box at 1024^2
// 45.8 -> 37.4, sixteen jobs 115 -> 93, a 1M-triangle mesh with 2^21 photons 83 -> 71 (about 2, 6 and 5
// of it from a write per ray that nothing read).  Without looking for peers at all the store is no
// faster, and a slot that all photons reach is an address with one atomic at a time.
__device__ __forceinline__ void hash_insert(const JobDesc& J, int k, uint32_t sidx, uint32_t slot, unsigned active) {
    const bool store = slot != 0xFFFFFFFFu;
    // photon index order = depth order; photons of the last row with i >= w/2 have z >= 1 and are
    // clipped by the scatter draw (counted by the correction draw all the same).  A clipped photon
    // offers P (the photon count) to the minimum: a slot that only clipped photons reach keeps P,
    // which the gather reads as the cleared texel -- photon 0 -- weighted by the slot's count.
    const bool clipped = (J.flags & SPPM_FLAG_GL_DEPTH_CLIP) && sidx >= (J.PH - 1) * J.PW + (J.PW + 1) / 2;
    const unsigned long long key = store ? ((unsigned long long)k << 32) | slot : ~0ull;
    const unsigned peers = __match_any_sync(active, key);
    const uint32_t n = __popc(peers), lane = threadIdx.x & 31u;
    const int leader = __ffs(peers) - 1;
    const bool grid = store && (J.flags & SPPM_FLAG_PHOTON_GRID);
    if (__any_sync(active, grid)) {
        // counting-sort grid: the count, and each photon's rank among its slot's photons (the
        // order of the ranks within a slot is arbitrary: the gather's sums do not depend on it)
        uint32_t base = 0;
        if (grid && (int)lane == leader) base = atomicAdd(&J.count[slot], n);
        base = __shfl_sync(active, base, leader);
        if (grid) J.grid_key[sidx] = make_uint2(slot, base + __popc(peers & ((1u << lane) - 1u)));
    }
    if (store && !grid) {
        const uint32_t cand = clipped ? J.PW * J.PH : sidx;
        if (n == 1u) {
            atomicAdd(&J.count[slot], 1u);
            atomicMin(&J.winner[slot], cand);
        } else {
            const uint32_t wmin = __reduce_min_sync(peers, cand);
            if ((int)lane == leader) {
                atomicAdd(&J.count[slot], n);
                if (wmin != 0xFFFFFFFFu) atomicMin(&J.winner[slot], wmin);
            }
        }
    }
}

// sum.fs (emitted photons), traced segments and errors: one atomic per warp and job
__device__ __forceinline__ void photon_counters(JobState* st, int k, unsigned active, uint32_t emitted, uint32_t segs,
                                                uint32_t err) {
    const unsigned jm = __match_any_sync(active, k);
    const uint32_t we = __reduce_add_sync(jm, emitted);
    const uint32_t ws = __reduce_add_sync(jm, segs);
    const uint32_t wr = __reduce_or_sync(jm, err);
    if ((threadIdx.x & 31) == (__ffs(jm) - 1)) {
        if (we) atomicAdd(&st->emitted_frame, we);
        if (ws) atomicAdd(&st->segments_frame, ws);
        if (wr) atomicOr(&st->err, wr);
    }
}

// fused photon pass: one thread per photon slot, generate + trace + store + hash insert
template <bool COUNT, bool TEX>
__global__ void __launch_bounds__(128) k_photon(LaunchSet ls) {
    const uint32_t g = grid_tid();
    if (g >= ls.total) return;
    const int k = find_job(ls, g);
    const JobDesc& J = job_of(ls, k);
    JobState* st = J.state;
    const uint32_t sidx = g - first_item(ls, k);
    uint32_t err = 0;
    float4 rndv = J.ph.rng[sidx];
    const PhotonRay R = photon_generate<TEX>(J, sidx, st->frame, rndv, err);
    uint32_t slot = 0xFFFFFFFFu;
    TraversalCount tc;
    if (R.cont) {
        const Hit h = trace_exact<true, COUNT>(J.scene, R.org, R.dir, false, err, &tc);
        slot = photon_store(J, st, sidx, h, R.dir, R.flux, R.depth);
    } else {
        photon_terminate(J, sidx);
    }
    J.ph.rng[sidx] = rndv;
    const unsigned active = __activemask();
    hash_insert(J, k, sidx, slot, active);
    photon_counters(st, k, active, R.emitted, R.cont ? 1u : 0u, err);
    if (COUNT) {
        const unsigned jm = __match_any_sync(active, k);
        const uint32_t wn = __reduce_add_sync(jm, tc.nodes);
        const uint32_t wt = __reduce_add_sync(jm, tc.tris);
        const uint32_t ws = __reduce_add_sync(jm, R.cont ? 1u : 0u);
        if ((threadIdx.x & 31) == (__ffs(jm) - 1)) {
            atomicAdd(&st->count_nodes, (unsigned long long)wn);
            atomicAdd(&st->count_tris, (unsigned long long)wt);
            atomicAdd(&st->count_segments, (unsigned long long)ws);
        }
    }
}

// ----------------------------------------------------------------------------------------------
// wavefront photon pass: generate -> trace (persistent, dynamic ray fetch) -> store
// ----------------------------------------------------------------------------------------------
// generate: emit/bounce every slot; RR-terminated photons are finished here, the others append
// their ray to the queue (warp-aggregated append)
//
// The block's slots are first reordered so that the emissions (a photon with no previous hit or
// at the bounce limit) come before the bounces: each warp then runs one of the two paths (the
// state written is per slot, so the order of work changes nothing).  Only the 8-byte hit decides
// the order, so only it goes through shared memory: the rest of the record is read by the lane that
// works on it (within the block's lines; an emission reads none of it but the generator).
//
// Bound by the instructions of the two paths and the latency of these loads: 10 blocks per SM (48
// registers; spills of 20 bytes stored, 28 loaded).  Us a pass against the whole record staged through
// shared memory at 9 blocks (56 registers) -> this: the Cornell box at 1024^2 297.1 -> 290.8, sixteen jobs
// 1013 -> 1002, glass and glossy spheres with 517x389 photons 163.9 -> 159.4, a 1M-triangle mesh with 2^21
// photons 1039 -> 1036.  Blocks of 64 threads (twice the adds to the queue's counter): 297.5, 1024, 162.7,
// 1059 where these read 293.2, 1008, 160.3, 1046; of 512: 306, 1035, 159.6, 1043.
// Textured, 6 blocks (80 registers): us a pass of the textured box, an eye pass in each, 5 / 6 / 8 blocks,
// 504 / 489 / 480 with 1024^2 photons and pixels, 179.0 / 177.5 / 177.0 with 512^2 (mixed 515 / 500 / 492 and
// 181.8 / 177.6 / 177.9), 125.8 / 126.2 / 126.4 with 256^2; 8 blocks spill 156 bytes and take the small
// launches' generation 4 to 9 % longer (20.0 -> 21.5 us with 128^2, 24.9 -> 27.3 with 256^2).
template <bool TEX>
__global__ void __launch_bounds__(128, TEX ? 6 : 10) k_photon_gen(LaunchSet ls, RayQueue q) {
    // the slots and their previous hits in processing order
    __shared__ uint32_t order[128];
    __shared__ int2 rec_hit[128];
    __shared__ uint32_t warp_emit[4], warp_valid[4], warp_rays[4], block_base;
    __shared__ int block_job;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        const uint32_t g0 = ls.first + grid_tid();
        const bool valid = g0 < ls.total;
        bool emit = false;
        int2 h = make_int2(-1, 0);
        if (valid) {
            const int k0 = find_job(ls, g0);
            if (threadIdx.x == 0) block_job = k0;
            const JobDesc& J0 = job_of(ls, k0);
            const JobState* st0 = J0.state;
            const uint32_t s0 = g0 - first_item(ls, k0);
            if (st0->frame != 0) h = J0.ph.hit[s0];
            emit = h.x < 0 || xadd((float)h.y, 1.0f) >= (float)J0.max_path;
        }
        const unsigned em = __ballot_sync(0xFFFFFFFFu, emit), vm = __ballot_sync(0xFFFFFFFFu, valid);
        if (lane == 0) {
            warp_emit[warp] = __popc(em);
            warp_valid[warp] = __popc(vm);
        }
        __syncthreads();
        uint32_t e_before = 0, v_before = 0, e_total = 0;
        for (uint32_t w = 0; w < 4; w++) {
            if (w < warp) {
                e_before += warp_emit[w];
                v_before += warp_valid[w];
            }
            e_total += warp_emit[w];
        }
        const unsigned below = (1u << lane) - 1u;
        if (valid) {
            // emissions at [0, e_total), bounces after them
            const uint32_t dst = emit ? e_before + __popc(em & below)
                                      : e_total + (v_before - e_before) + __popc(vm & ~em & below);
            order[dst] = g0;
            rec_hit[dst] = h;
        }
        __syncthreads();
    }
    // Every count of the pass is one address for all warps, and the GPU adds to one address once in 0.7 ns:
    // with a ray count, an emission count and a segment count per warp, 2^20 slots took 46 to 69 us of
    // the kernel's 75.  So a block adds once to the queue and once to its job's two counts.
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const uint32_t t = threadIdx.x;
    const bool on = t < warp_valid[0] + warp_valid[1] + warp_valid[2] + warp_valid[3];
    const uint32_t g = on ? order[t] : 0u;
    const int k = on ? find_job(ls, g) : block_job;
    const JobDesc& J = job_of(ls, k);
    JobState* st = J.state;
    uint32_t err = 0;
    PhotonRay R;
    R.cont = false;
    R.emitted = 0;
    uint32_t bin = 0, rank = 0;
    if (on) {
        const uint32_t sidx = g - first_item(ls, k);
        float4 rndv = J.ph.rng[sidx];
        R = photon_generate<TEX>(J, rec_hit[t], J.ph.pos[sidx], J.ph.flux[sidx], J.ph.dir[sidx], rndv, err);
        J.ph.rng[sidx] = rndv;
        if (R.cont) {
            J.ph.flux[sidx] = f4(R.flux, 0.0f);  // flux before the segment, read back by k_photon_store
            J.ph.hit[sidx] = make_int2(-1, (int)R.depth);
        } else {
            photon_terminate(J, sidx);
        }
    }
    const unsigned live = __ballot_sync(kFull, R.cont);
    if (lane == 0) warp_rays[warp] = __popc(live);
    const uint32_t emitted = __popc(__ballot_sync(kFull, R.emitted != 0));
    if (lane == 0) warp_emit[warp] = emitted;
    if (q.key && R.cont) {
        // lanes with the same bin take consecutive ranks from one atomic
        bin = q.bin_rank[ray_bin(J.scene, R.org, R.dir)];
        const unsigned same = __match_any_sync(live, bin);
        const int lead = __ffs(same) - 1;
        const uint32_t counter = blockIdx.x % kBinCounters;
        if ((int)lane == lead) rank = atomicAdd(&q.bins[counter * kRayBins + bin], __popc(same));
        rank = __shfl_sync(live, rank, lead) + __popc(same & ((1u << lane) - 1u));
        bin |= counter << 16;
    }
    const bool one_job = __syncthreads_and(!on || k == block_job) != 0;
    if (t == 0) {
        const uint32_t rays = warp_rays[0] + warp_rays[1] + warp_rays[2] + warp_rays[3];
        block_base = rays ? atomicAdd(&q.counters[0], rays) : 0u;
        if (one_job) {
            // emitted_frame in the low word, segments_frame in the high one
            static_assert(offsetof(JobState, emitted_frame) % 8 == 0 &&
                          offsetof(JobState, segments_frame) == offsetof(JobState, emitted_frame) + 4, "one 64-bit add");
            const unsigned long long n = (unsigned long long)rays << 32 | (warp_emit[0] + warp_emit[1] + warp_emit[2] + warp_emit[3]);
            if (n) atomicAdd(reinterpret_cast<unsigned long long*>(&st->emitted_frame), n);
        }
    }
    if (err) atomicOr(&st->err, err);
    __syncthreads();
    if (R.cont) {
        uint32_t qi = block_base + __popc(live & ((1u << lane) - 1u));
        for (uint32_t w = 0; w < warp; w++) qi += warp_rays[w];
        q.org[qi] = make_float4(R.org.x, R.org.y, R.org.z, __uint_as_float(g));
        q.dir[qi] = make_float4(R.dir.x, R.dir.y, R.dir.z, 0.0f);
        if (q.key) q.key[qi] = make_uint2(bin, rank);
    }
    if (!one_job && on) photon_counters(st, k, __activemask(), R.emitted, R.cont ? 1u : 0u, 0u);
}

// exclusive scan of the bin counts in place, a bin's counters one after the other: one block of 1024
// threads, each with four consecutive bins of every 4096, so that a warp's accesses are consecutive (twelve
// consecutive bins a thread: 7.4 us, bound by the loads' and stores' wavefronts; this 5.1)
__global__ void __launch_bounds__(1024) k_ray_bins_scan(uint32_t* bins) {
    constexpr uint32_t kChunks = kRayBins / 4096;
    static_assert(kRayBins % 4096 == 0 && kChunks <= 32, "bins must split into chunks of a uint4 per thread");
    __shared__ uint32_t warp_sums[kChunks][32], totals[kChunks];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4 v[kBinCounters][kChunks];
#pragma unroll
    for (uint32_t c = 0; c < kBinCounters; c++)
#pragma unroll
        for (uint32_t i = 0; i < kChunks; i++)
            v[c][i] = reinterpret_cast<const uint4*>(bins + c * kRayBins)[i * 1024 + threadIdx.x];
    auto warp_scan = [&](uint32_t x) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        return x;
    };
    uint32_t run[kChunks];
#pragma unroll
    for (uint32_t i = 0; i < kChunks; i++) {
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t c = 0; c < kBinCounters; c++) sum += v[c][i].x + v[c][i].y + v[c][i].z + v[c][i].w;
        const uint32_t incl = warp_scan(sum);
        if (lane == 31) warp_sums[i][warp] = incl;
        run[i] = incl - sum;
    }
    __syncthreads();
    if (warp < kChunks) {
        const uint32_t w = warp_sums[warp][lane], wi = warp_scan(w);
        warp_sums[warp][lane] = wi - w;
        if (lane == 31) totals[warp] = wi;
    }
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (uint32_t i = 0; i < kChunks; i++) {
        uint32_t r = run[i] + before + warp_sums[i][warp];
        before += totals[i];
        auto take = [&](uint32_t& x) {
            const uint32_t n = x;
            x = r;
            r += n;
        };
#pragma unroll
        for (uint32_t c = 0; c < kBinCounters; c++) take(v[c][i].x);
#pragma unroll
        for (uint32_t c = 0; c < kBinCounters; c++) take(v[c][i].y);
#pragma unroll
        for (uint32_t c = 0; c < kBinCounters; c++) take(v[c][i].z);
#pragma unroll
        for (uint32_t c = 0; c < kBinCounters; c++) take(v[c][i].w);
    }
#pragma unroll
    for (uint32_t c = 0; c < kBinCounters; c++)
#pragma unroll
        for (uint32_t i = 0; i < kChunks; i++)
            reinterpret_cast<uint4*>(bins + c * kRayBins)[i * 1024 + threadIdx.x] = v[c][i];
}

// the bins' traversal order, from the mean walk of their rays since the last reorder (at most once
// per 8 frames; the frame kernel counts them): the longest first, so that the persistent traversal
// starts its longest walks early and its drain (lanes idle while the last walks finish) is short
// -- a longest-processing-time-first schedule.  One
// block: the means quantised to 256 keys (0: no ray since the last reorder, placed last); a
// stable counting sort by descending key, rounds of 1024 bins in bin order, each lane's place
// among equal keys from the warp histograms of the round.  Any order gives the same results (the
// rays are independent); this one is deterministic.
__global__ void __launch_bounds__(1024) k_ray_bins_order(RayQueue q) {
    constexpr uint32_t kKeys = 256, kRounds = kRayBins / 1024;
    static_assert(kRayBins % 1024 == 0, "bins must split into rounds of 1024");
    __shared__ uint32_t base[kKeys], cursor[kKeys];
    __shared__ uint32_t hist[32][kKeys];  // [warp][key]: counts of the round, then offsets
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // at most once per 8 frames (with an eye pass every frame the sort would cost a few percent)
    if (q.counters[7] < 8u) return;
    if (t < kKeys) {
        base[t] = 0;
        cursor[t] = 0;
    }
    __syncthreads();
    if (t == 0) q.counters[7] = 0;
    uint32_t key[kRounds];
#pragma unroll
    for (uint32_t r = 0; r < kRounds; r++) {
        const uint32_t at = q.bin_rank[r * 1024 + t];
        unsigned long long c = 0;
#pragma unroll
        for (uint32_t k = 0; k < kBinCosts; k++) c += q.bin_cost[k * kRayBins + at];
        const uint32_t n = (uint32_t)c, mean = n ? (uint32_t)(c >> 32) / n : 0u;
        const uint32_t k = n ? 1u + min(254u, mean < 128u ? mean : 128u + (mean - 128u) / 8u) : 0u;
        key[r] = kKeys - 1u - k;  // descending mean
        atomicAdd(&base[key[r]], 1u);
    }
    __syncthreads();
    if (warp == 0) {  // exclusive scan of the key totals, 8 keys per lane
        uint32_t v[kKeys / 32], s = 0;
#pragma unroll
        for (uint32_t i = 0; i < kKeys / 32; i++) {
            v[i] = base[lane * (kKeys / 32) + i];
            s += v[i];
        }
        uint32_t incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane >= o) incl += y;
        }
        uint32_t run = incl - s;
#pragma unroll
        for (uint32_t i = 0; i < kKeys / 32; i++) {
            base[lane * (kKeys / 32) + i] = run;
            run += v[i];
        }
    }
    for (uint32_t i = t; i < kBinCosts * kRayBins; i += 1024) q.bin_cost[i] = 0ull;  // every cost was read above
    uint32_t rank[kRounds];
#pragma unroll
    for (uint32_t r = 0; r < kRounds; r++) {
        for (uint32_t i = t; i < 32 * kKeys; i += 1024) (&hist[0][0])[i] = 0u;
        __syncthreads();
        const uint32_t k = key[r];
        const unsigned same = __match_any_sync(0xFFFFFFFFu, k);
        if ((int)lane == __ffs(same) - 1) hist[warp][k] = __popc(same);
        __syncthreads();
        if (t < kKeys) {  // offsets of each warp's lanes among the key's bins so far
            uint32_t run = cursor[t];
            for (uint32_t w = 0; w < 32; w++) {
                const uint32_t c = hist[w][t];
                hist[w][t] = run;
                run += c;
            }
            cursor[t] = run;
        }
        __syncthreads();
        rank[r] = base[k] + hist[warp][k] + __popc(same & ((1u << lane) - 1u));
        __syncthreads();
    }
#pragma unroll
    for (uint32_t r = 0; r < kRounds; r++) q.bin_rank[r * 1024 + t] = rank[r];
}

// perm[offset of the bin + rank] = queue index
__global__ void __launch_bounds__(256) k_ray_bins_scatter(RayQueue q) {
    const uint32_t qi = grid_tid();
    if (qi >= q.counters[0]) return;
    const uint2 kr = q.key[qi];
    q.perm[q.bins[(kr.x >> 16) * kRayBins + (kr.x & 0xFFFFu)] + kr.y] = qi;
}

// trace: persistent warps; a lane whose ray finished fetches the next one from the queue, so
// lanes stay busy while their neighbours walk longer paths (dynamic fetch).
// Bound by instruction issue and L1 wavefronts at 13 to 14 active lanes (a quarter of a step's
// issue slots test a box, a third a triangle for 3 to 4 lanes), on large meshes by the node loads.
// So a step does as little as it can: the box test in two-lane arithmetic, the major axis without
// minimum and maximum (slab_x), one comparison each for the walk's end and for a leaf to test, no
// step counter of its own: 142.5 -> 126.7 us a launch on the Cornell box (2^20 slots), 744 -> 697 on
// a 1M-triangle mesh (2^21), 610 -> 568 over 16 jobs.  With fewer rays than lanes the longest walk
// decides, and what its step waits for: spread over the warps, 2^14 rays take 51 us instead of 70,
// 2^16 63 instead of 74.
// AHEAD (launches of up to kTraceAheadSlots): a step loads both nodes that the next one may need before
// it tests its own box, so the chain of a walk holds the loads alone and not the test between them; twice
// the loads and 75 registers (6 blocks per SM) that larger launches have no room for.
template <bool COUNT, bool AHEAD>
__global__ void __launch_bounds__(128, AHEAD ? 6 : 9) k_trace_photons(LaunchSet ls, RayQueue q) {
    const uint32_t total = q.counters[0];
    const int refill = q.refill_steps ? (int)q.refill_steps : 32;
    const unsigned lane = threadIdx.x & 31;
    // a lane's ray, or: it needs one, it has found none left, it takes none (with fewer rays than lanes
    // they are spread over all warps, spread_lanes)
    const uint32_t kNeed = 0xFFFFFFFDu, kDone = 0xFFFFFFFEu, kIdle = 0xFFFFFFFFu;
    uint32_t idx = lane < spread_lanes(total) ? kNeed : kIdle;
    const NodeX* nodes = nullptr;
    const float4* tri_isect = nullptr;
    int32_t nn = 0;
    f3 org = mk(0, 0, 0), dir = mk(0, 0, 0);
    RayX R{};
    Hit h;
    int32_t node = 0, steps = 0;
    uint32_t err = 0;
    int job_k = 0;
    // traversal counters: summed per lane, added to the job's totals when the lane moves to
    // another job's rays and at the end (three 64-bit atomics per ray would serialise the kernel)
    TraversalCount tc;
    uint32_t tc_segs = 0;
    int tc_job = -1;
    auto flush_counts = [&]() {
        if (tc_job >= 0 && tc_segs) {
            JobState* st = job_of(ls, tc_job).state;
            atomicAdd(&st->count_nodes, (unsigned long long)tc.nodes);
            atomicAdd(&st->count_tris, (unsigned long long)tc.tris);
            atomicAdd(&st->count_segments, (unsigned long long)tc_segs);
        }
        tc.nodes = tc.tris = 0;
        tc_segs = 0;
    };
    for (;;) {
        const bool need = idx == kNeed;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, need);
        if (m) {
            const int leader = __ffs(m) - 1;
            uint32_t base = 0;
            if ((int)lane == leader) base = atomicAdd(&q.counters[1], __popc(m));
            base = __shfl_sync(0xFFFFFFFFu, base, leader);
            if (need) {
                idx = base + __popc(m & ((1u << lane) - 1));
                if (idx >= total) {
                    idx = kDone;
                } else {
                    if (q.perm) idx = q.perm[idx];
                    const float4 o = q.org[idx], d = q.dir[idx];
                    const uint32_t g = __float_as_uint(o.w);
                    const int nk = find_job(ls, g);
                    if (err && nk != job_k) {  // an error belongs to the job whose ray raised it
                        atomicOr(&job_of(ls, job_k).state->err, err);
                        err = 0;
                    }
                    job_k = nk;
                    if (COUNT && job_k != tc_job) {
                        flush_counts();
                        tc_job = job_k;
                    }
                    const DevScene& S = job_of(ls, job_k).scene;
                    org = mk(o.x, o.y, o.z);
                    dir = mk(d.x, d.y, d.z);
                    nn = (int32_t)S.num_nodes;
                    const int face = cube_face(dir);
                    nodes = S.nodes + (size_t)face * nn;
                    tri_isect = S.tri_isect;
                    R = ray_x(org, dir, face);
                    h.t = 1.0e30f;
                    h.tri = -1;
                    h.mat = -1;
                    h.bu = h.bv = h.bw = 0.0f;
                    node = 0;
                    steps = 0;
                    if (slab_degenerate(dir)) {
                        // walks most of the tree: left to k_trace_photons_coop
                        q.slow[atomicAdd(&q.counters[2], 1u)] = idx;
                        idx = kNeed;
                    }
                }
            }
        }
        if (__all_sync(0xFFFFFFFFu, idx >= kDone)) break;
        // the tail: once the queue is drained, a warp left with a few long walks hands them to
        // k_trace_photons_tail, which finishes each with all 32 lanes of a warp, resumed where the
        // lane stands (coop_trace_exact_from, the same result bit for bit): a walk's chain of
        // dependent node loads becomes windows of 32 loads in flight
        if (q.tail_lanes) {
            const unsigned act = __ballot_sync(0xFFFFFFFFu, idx < kNeed);
            const unsigned drained = __ballot_sync(0xFFFFFFFFu, idx == kDone);
            if (drained && act && (uint32_t)__popc(act) <= q.tail_lanes) {
                if (idx < kNeed) {
                    const int32_t mat = h.tri >= 0 ? __float_as_int(__ldg(&tri_isect[(size_t)h.tri * 3 + 2]).y) : -1;
                    q.hit[idx] = make_float4(__int_as_float(h.tri), h.bu, h.bv, h.bw);
                    q.tail_state[idx] = make_float4(h.t, __int_as_float(mat), __int_as_float(node),
                                                    __int_as_float(steps));
                    q.tail_list[atomicAdd(&q.counters[4], 1u)] = idx;
                    idx = kDone;
                }
                continue;  // every walk of the warp is handed over; the next iteration leaves the loop
            }
        }
        if (idx >= kNeed) continue;
        bool finished = false;
        int it = 0;
        unsigned long long lo, hi, near_far, links;
        if (AHEAD) ldg32q(nodes + node, lo, hi, near_far, links);
#pragma unroll 1
        do {
            unsigned long long next_lo, next_hi, next_near_far, next_links;  // the node after a hit
            unsigned long long miss_lo, miss_hi, miss_near_far, miss_links;  // and after a miss
            if (AHEAD) {
                const uint32_t last = (uint32_t)nn - 1u;  // (past the end: a node, not used)
                ldg32q(nodes + min((uint32_t)node + 1u, last), next_lo, next_hi, next_near_far, next_links);
                ldg32q(nodes + min((uint32_t)node_miss(links), last), miss_lo, miss_hi, miss_near_far, miss_links);
            } else {
                ldg32q(nodes + node, lo, hi, near_far, links);
            }
            if (COUNT) tc.nodes++;
            float tmin, tmax;
            slab_x<true>(R, lo, hi, near_far, tmin, tmax);
            const bool hit = (tmin <= tmax) && (tmin <= h.t) && (tmax >= 0.0f);
            const int32_t tri = node_tri(links);
            // a leaf that is no emitter's: neither -1 nor the emitter bit
            if (hit && (uint32_t)tri < (uint32_t)kEmitterBit) {
                if (COUNT) tc.tris++;
                const float4 a = __ldg(&tri_isect[(size_t)tri * 3 + 0]);
                const float4 b = __ldg(&tri_isect[(size_t)tri * 3 + 1]);
                const float4 c = __ldg(&tri_isect[(size_t)tri * 3 + 2]);
                // the triangle test with the divisions one after the other's test: few lanes get here at a
                // time (3 to 4 of a warp), and often none needs the next one
                const f3 v0 = mk(a.x, a.y, a.z), e0 = mk(a.w, b.x, b.y), e1 = mk(b.z, b.w, c.x);
                const f3 pv = cross(dir, e1);
                const float det = dot(e0, pv);
                const f3 tv = sub(org, v0);
                const f3 qv = cross(tv, e0);
                const float u = xdiv(dot(tv, pv), det);
                if (u >= 0.0f) {
                    const float v = xdiv(dot(dir, qv), det);
                    const float w = xsub(xsub(1.0f, u), v);
                    if (v >= 0.0f && w >= 0.0f) {
                        const float tt = xdiv(dot(e1, qv), det);
                        if (tt >= 0.0f && tt < h.t) {
                            h.t = tt;
                            h.tri = tri;
                            h.bu = v;
                            h.bv = w;
                            h.bw = u;
                        }
                    }
                }
            }
            node = hit ? node + 1 : node_miss(links);
            if (AHEAD) {
                lo = hit ? next_lo : miss_lo;
                hi = hit ? next_hi : miss_hi;
                near_far = hit ? next_near_far : miss_near_far;
                links = hit ? next_links : miss_links;
            }
            it++;
            finished = (uint32_t)node >= (uint32_t)nn;
        } while (!finished && it < refill);
        steps += it;
        if (!finished && steps > nn) {
            err |= kErrWatchdogTraverse;
            finished = true;
        }
        if (finished) {
            q.hit[idx] = make_float4(__int_as_float(h.tri), h.bu, h.bv, h.bw);
            if (q.perm) bin_cost_add(q, q.key[idx].x & 0xFFFFu, (uint32_t)steps);
            if (COUNT) tc_segs++;
            idx = kNeed;
        }
    }
    if (COUNT) flush_counts();
    if (err) atomicOr(&job_of(ls, job_k).state->err, err);
}

// the walks k_trace_photons handed over once its queue was drained: one warp per walk, resumed at
// the node, closest hit and step count where its lane stopped
template <bool COUNT>
__global__ void __launch_bounds__(128) k_trace_photons_tail(LaunchSet ls, RayQueue q) {
    const uint32_t n = q.counters[4];
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const unsigned lane = threadIdx.x & 31;
    for (uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n; w += warps) {
        const uint32_t idx = q.tail_list[w];
        const float4 o = q.org[idx], d = q.dir[idx], hr = q.hit[idx], ts = q.tail_state[idx];
        const int job_k = find_job(ls, __float_as_uint(o.w));
        const JobDesc& J = job_of(ls, job_k);
        Hit h0;
        h0.t = ts.x;
        h0.mat = __float_as_int(ts.y);
        h0.tri = __float_as_int(hr.x);
        h0.bu = hr.y;
        h0.bv = hr.z;
        h0.bw = hr.w;
        uint32_t err = 0;
        TraversalCount ct;
        const Hit h = coop_trace_exact_from<true, COUNT>(J.scene, mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), false, err,
                                                         &ct, __float_as_int(ts.z), h0, (uint32_t)__float_as_int(ts.w));
        if (lane == 0) {
            q.hit[idx] = make_float4(__int_as_float(h.tri), h.bu, h.bv, h.bw);
            if (err) atomicOr(&J.state->err, err);
            if (COUNT) {
                atomicAdd(&J.state->count_nodes, (unsigned long long)ct.nodes);
                atomicAdd(&J.state->count_tris, (unsigned long long)ct.tris);
                atomicAdd(&J.state->count_segments, 1ull);
            }
        }
    }
}

// the rays k_trace_photons set aside (slab_degenerate directions), one block of 1024 threads per
// ray (block_trace_exact)
template <bool COUNT>
__global__ void __launch_bounds__(kBlockWalk) k_trace_photons_coop(LaunchSet ls, RayQueue q) {
    __shared__ BlockWalkShared sh;
    const uint32_t n = q.counters[2];
    for (uint32_t w = blockIdx.x; w < n; w += gridDim.x) {
        const uint32_t idx = q.slow[w];
        const float4 o = q.org[idx], d = q.dir[idx];
        const int job_k = find_job(ls, __float_as_uint(o.w));
        const JobDesc& J = job_of(ls, job_k);
        uint32_t err = 0;
        TraversalCount ct;
        const Hit h = block_trace_exact<true, COUNT>(J.scene, mk(o.x, o.y, o.z), mk(d.x, d.y, d.z), false, err, &ct,
                                                     sh);
        if (threadIdx.x == 0) {
            q.hit[idx] = make_float4(__int_as_float(h.tri), h.bu, h.bv, h.bw);
            atomicAdd(&J.state->coop_segments, 1ull);
            if (err) atomicOr(&J.state->err, err);
            if (COUNT) {
                atomicAdd(&J.state->count_nodes, (unsigned long long)ct.nodes);
                atomicAdd(&J.state->count_tris, (unsigned long long)ct.tris);
                atomicAdd(&J.state->count_segments, 1ull);
            }
        }
    }
}

// store: shade the hit of each queued ray, write the photon record, insert it into the grid
__global__ void __launch_bounds__(128) k_photon_store(LaunchSet ls, RayQueue q, uint32_t grid_shift) {
    const uint32_t qi = grid_tid();
    if (qi >= q.counters[0]) return;
    const float4 o = q.org[qi], d = q.dir[qi], hr = q.hit[qi];
    const uint32_t g = __float_as_uint(o.w);
    const int k = find_job(ls, g);
    const JobDesc& J = job_of(ls, k);
    const JobState* st = J.state;
    const uint32_t sidx = g - first_item(ls, k);
    Hit h;
    h.tri = __float_as_int(hr.x);
    h.bu = hr.y;
    h.bv = hr.z;
    h.bw = hr.w;
    const float4 f = J.ph.flux[sidx];
    const int depth = J.ph.hit[sidx].y;
    const uint32_t slot = photon_store(J, st, sidx, h, mk(d.x, d.y, d.z), mk(f.x, f.y, f.z), (float)depth, grid_shift);
    hash_insert(J, k, sidx, slot, __activemask());
}

// ----------------------------------------------------------------------------------------------
// k_gather: progressive.fs (:98-142, AccumulatePhotons :65-95)
// ----------------------------------------------------------------------------------------------
// A warp takes an 8x4-pixel tile (neighbouring hit points read the same slots).  Bound by its chain of
// loads -- pixel state, the eight cells' winners, their photons -- at 32 warps per SM (64 registers);
// the bounds of the in-cell test are nine planes per pixel, loaded once, not six per cell: 57.8 -> 52.1
// us on the Cornell box (1024^2), 189 -> 171 over 16 jobs.
// BLOCKS per SM: 5 (48 registers; spills of 52 bytes stored, 72 loaded) where a launch has waves of blocks
// to fill them.  Us a pass with 1024x512 photons, 4 / 5 blocks: Cornell box 168.1 / 171.4 at 512^2 pixels,
// 186.9 / 189.2 at 768^2, 210.1 / 209.2 at 1024^2, 216.2 / 214.7 at 1280x1024, 343.8 / 332.9 at 2048^2;
// 102k-triangle mesh 256.3 / 254.8, 269.0 / 268.9, 288.5 / 285.7, 297.5 / 295.2, 407.0 / 397.5; sixteen
// jobs 978 / 968.
constexpr uint32_t kGatherWideItems = 1u << 20;
template <int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS) k_gather(LaunchSet ls) {
    const uint32_t g = grid_tid();
    if (g >= ls.total) return;
    const int k = find_job(ls, g);
    const JobDesc& J = job_of(ls, k);
    JobState* st = J.state;
    const uint32_t item = g - first_item(ls, k);
    uint32_t p;
    if (!tile_pixel(J, item, p)) return;
    const uint32_t frame = st->frame;
    if (p == 0) {
        // NumPhotons += int(sum) (glslppm.cpp:397) once the photon pass of this frame is done
        const uint32_t e = st->emitted_frame;
        st->num_photons_f32 = xadd(st->num_photons_f32, (float)(int)e);
        st->num_photons += e;
        st->photon_segments += st->segments_frame;
    }
    float4 qfr = frame == 0 ? make_float4(0.0f, 0.0f, 0.0f, st->r0) : J.px.flux_r[p];
    float4 qe = J.px.emi_n[p];
    const int32_t tri = J.px.tri[p];
    // (loaded whether or not the pixel has a hit point: one wait instead of two; read once a pass)
    const float4 pos4 = __ldcs(&J.px.pos[p]), nrm4 = __ldcs(&J.px.nrm[p]), refl4 = __ldcs(&J.px.refl[p]);
    if (tri >= 0) {
        const float G = st->grid_scale;
        const float hs1 = st->hash_scale1;
        const float hn = (float)J.hash_num;
        const float alpha = J.alpha;
        const f3 bbmin = mk(st->bbmin[0], st->bbmin[1], st->bbmin[2]);
        const f3 qp = xyz(pos4), qn = xyz(nrm4), qr = xyz(refl4);
        float N = qe.w, R = qfr.w;
        f3 tau = xyz(qfr);
        const f3 ii = mk(floorf(xsub(xmul(fabsf(xsub(qp.x, bbmin.x)), G), 0.5f)),
                         floorf(xsub(xmul(fabsf(xsub(qp.y, bbmin.y)), G), 0.5f)),
                         floorf(xsub(xmul(fabsf(xsub(qp.z, bbmin.z)), G), 0.5f)));
        f3 flux = mk(0, 0, 0);
        float M = 0.0f;
        // the eight cells' slots and winners first (independent loads in flight together), then
        // the candidate photons' positions, then the accumulation in cell order (the sum's order
        // is progressive.fs's)
        uint32_t slot[8], win[8];
        hash_cells8(ii, G, hs1, hn, slot);
        const uint32_t clipped_only = J.PW * J.PH;  // every photon of the slot clipped: photon 0
#pragma unroll
        for (int c = 0; c < 8; c++) {
            win[c] = __ldg(&J.winner[slot[c]]);
            if (win[c] == clipped_only) win[c] = 0u;
        }
        uint32_t inside = 0;
        // the cells' bounds from the table k_cell_bounds made for this grid (the same values as
        // the division below), when the 2x2x2 block lies inside it
        const float tn = (float)st->cell_table_n;
        const bool table = J.cell_bounds && ii.x >= 0.0f && ii.y >= 0.0f && ii.z >= 0.0f && ii.x + 2.0f < tn &&
                           ii.y + 2.0f < tn && ii.z + 2.0f < tn;
        // the three planes per axis that bound the two cells of each
        float X[3], Y[3], Z[3];
        if (table) {
            const float* T = J.cell_bounds;
            const uint32_t tx = (uint32_t)ii.x, ty = (uint32_t)ii.y, tz = (uint32_t)ii.z;
#pragma unroll
            for (int o = 0; o < 3; o++) {
                X[o] = __ldg(&T[tx + o]);
                Y[o] = __ldg(&T[kCellTable + ty + o]);
                Z[o] = __ldg(&T[2 * kCellTable + tz + o]);
            }
        } else {
            f3 e = ii;
#pragma unroll
            for (int o = 0; o < 3; o++) {
                X[o] = xadd(xdiv(e.x, G), bbmin.x);
                Y[o] = xadd(xdiv(e.y, G), bbmin.y);
                Z[o] = xadd(xdiv(e.z, G), bbmin.z);
                e = mk(xadd(e.x, 1.0f), xadd(e.y, 1.0f), xadd(e.z, 1.0f));
            }
        }
#pragma unroll
        for (int c = 0; c < 8; c++) {
            if (win[c] == kEmptySlot) continue;  // the cleared texel: photon 0 weighted by count 0
            const float4 pp = __ldg(&J.ph.pos[win[c]]);
            const int cx = c & 1, cy = (c >> 1) & 1, cz = c >> 2;
            const f3 rmin = mk(X[cx], Y[cy], Z[cz]), rmax = mk(X[cx + 1], Y[cy + 1], Z[cz + 1]);
            if (pp.x > rmin.x && pp.y > rmin.y && pp.z > rmin.z && pp.x < rmax.x && pp.y < rmax.y && pp.z < rmax.z &&
                length(sub(xyz(pp), qp)) < R)
                inside |= 1u << c;
        }
#pragma unroll
        for (int c = 0; c < 8; c++) {
            if (!((inside >> c) & 1u)) continue;
            const float4 pd = __ldg(&J.ph.dir[win[c]]);
            if (dot(qn, neg(xyz(pd))) > 0.0f) {
                const float4 pf = __ldg(&J.ph.flux[win[c]]);
                const float cnt = (float)__ldg(&J.count[slot[c]]);
                flux = add(flux, scl(xyz(pf), cnt));
                M = xadd(M, cnt);
            }
        }
        flux = mul(flux, scl(qr, 3.183099627e-01f));
        const float gg = fminf(xdiv(xadd(N, xmul(alpha, M)), xadd(N, M)), 1.0f);
        R = xmul(R, xsqrt(gg));
        N = xadd(N, xmul(M, alpha));
        tau = scl(add(tau, flux), gg);
        qfr = f4(tau, R);
        qe.w = N;
        J.px.emi_n[p] = qe;
    }
    J.px.flux_r[p] = qfr;
}

// ----------------------------------------------------------------------------------------------
// k_resolve: re.fs
// ----------------------------------------------------------------------------------------------
__global__ void k_resolve(LaunchSet ls, uint32_t display) {
    const uint32_t g = grid_tid();
    if (g >= ls.total) return;
    const int k = find_job(ls, g);
    const JobDesc& J = job_of(ls, k);
    const uint32_t p = g - first_item(ls, k);
    const float4 fr = J.px.flux_r[p];
    const float4 qe = J.px.emi_n[p];
    const float total = J.state->num_photons_f32;
    const float den = xmul(xmul(xmul(fr.w, fr.w), 3.141592f), total);
    float L[3] = {xadd(xdiv(fr.x, den), qe.x), xadd(xdiv(fr.y, den), qe.y), xadd(xdiv(fr.z, den), qe.z)};
    for (int c = 0; c < 3; c++) {
        float v = L[c];
        if (display) {
            v = xsub(1.0f, sppm_fexp(xmul(-v, 60000.0f)));
            if (v < 0.0031308f) v = xmul(12.92f, v);
            else v = xsub(xmul(xadd(1.0f, 0.055f), sppm_fpow(v, 0.416666666667f)), 0.055f);
        }
        J.image[(size_t)p * 3 + c] = v;
    }
}

// ----------------------------------------------------------------------------------------------
// stage-level hash build on caller arrays (sppm_hash_build)
// ----------------------------------------------------------------------------------------------
// (four slots a thread where the arrays allow it; a table may have up to 2^32 - 1)
__global__ void k_hash_clear(uint32_t* winner, uint32_t* count, uint32_t n) {
    const uint32_t g = grid_tid() * 4u;
    if (g >= n) return;
    if (n - g >= 4u && ((reinterpret_cast<uintptr_t>(winner) | reinterpret_cast<uintptr_t>(count)) & 15) == 0) {
        *reinterpret_cast<uint4*>(winner + g) = make_uint4(kEmptySlot, kEmptySlot, kEmptySlot, kEmptySlot);
        *reinterpret_cast<uint4*>(count + g) = make_uint4(0u, 0u, 0u, 0u);
    } else {
        for (uint32_t i = 0; i < 4u && i < n - g; i++) {
            winner[g + i] = kEmptySlot;
            count[g + i] = 0;
        }
    }
}

__global__ void k_hash_build(const float4* pos, const float4* flux, uint32_t pw, uint32_t ph, uint32_t hash_num,
                             float bx, float by, float bz, float G, uint32_t flags, uint32_t* winner, uint32_t* count) {
    const uint32_t id = grid_tid();
    if (id >= pw * ph) return;
    const float hs1 = xdiv(4194304.0f, G);
    const float4 f = flux[id];
    const bool store = !(f.x < 0.0f);
    uint32_t slot = 0;
    if (store) {
        const float4 pp = pos[id];
        const f3 cell = mk(floorf(xmul(xsub(pp.x, bx), G)), floorf(xmul(xsub(pp.y, by), G)), floorf(xmul(xsub(pp.z, bz), G)));
        slot = hash_cell(cell, G, hs1, (float)hash_num);
    }
    const bool clipped = (flags & SPPM_FLAG_GL_DEPTH_CLIP) && id >= (ph - 1) * pw + (pw + 1) / 2;
    // (as hash_insert; 2^20 photons into 2^20 slots, clear included: 27.9 -> 21.8 us)
    const unsigned peers = __match_any_sync(__activemask(), store ? slot : 0xFFFFFFFFu);
    if (store) {
        const uint32_t n = __popc(peers), cand = clipped ? 0xFFFFFFFFu : id;
        if (n == 1u) {
            atomicAdd(&count[slot], 1u);
            if (!clipped) atomicMin(&winner[slot], cand);
        } else {
            const uint32_t wmin = __reduce_min_sync(peers, cand);
            if ((threadIdx.x & 31) == (__ffs(peers) - 1)) {
                atomicAdd(&count[slot], n);
                if (wmin != 0xFFFFFFFFu) atomicMin(&winner[slot], wmin);
            }
        }
    }
}

// pinned math on the device, for the accuracy / determinism tests
__global__ void k_fpmath(int fn, const float* x, const float* y, float* out, uint32_t n) {
    const uint32_t i = grid_tid();
    if (i >= n) return;
    float r;
    switch (fn) {
        case 0: r = sppm_fsin(x[i]); break;
        case 1: r = sppm_fcos(x[i]); break;
        case 2: r = sppm_fpow(x[i], y[i]); break;
        case 3: r = sppm_fexp(x[i]); break;
        case 4: r = sppm_flog2(x[i]); break;
        default: r = sppm_fexp2(x[i]); break;
    }
    out[i] = r;
}

// single rays through the exact traversal: mode 0 one thread per ray (trace_exact), mode 1 one
// warp per ray (coop_trace_exact), mode 2 one block per ray (block_trace_exact), mode 3 the mixed
// path's 4-wide quantised traversal one per thread (trace4); photon rays skip emitters, eye rays
// may cull back faces
template <bool PHOTON>
__global__ void __launch_bounds__(1024) k_debug_trace(DevScene s, const float* org, const float* dir, uint32_t n,
                                                     int cull, int mode, int32_t* tri, float* t, uint32_t* err) {
    uint32_t e = 0;
    if (mode == 2) {
        __shared__ BlockWalkShared sh;
        for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
            TraversalCount ct;
            const Hit h = block_trace_exact<PHOTON, false>(s, mk(org[3 * i], org[3 * i + 1], org[3 * i + 2]),
                                                           mk(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]), cull != 0, e,
                                                           &ct, sh);
            if (threadIdx.x == 0) {
                tri[i] = h.tri;
                t[i] = h.t;
            }
        }
    } else if (mode == 0) {
        const uint32_t i = grid_tid();
        if (i >= n) return;
        const Hit h = trace_exact<PHOTON>(s, mk(org[3 * i], org[3 * i + 1], org[3 * i + 2]),
                                          mk(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]), cull != 0, e);
        tri[i] = h.tri;
        t[i] = h.t;
    } else if (mode == 3) {
        // the mixed path's 4-wide quantised traversal (the eye pass's trace4)
        const uint32_t i = grid_tid();
        if (i >= n) return;
        const f3 d3 = mk(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]);
        const Hit4 h = trace4<PHOTON>(s.nodes4, s.tri_isect, mk(org[3 * i], org[3 * i + 1], org[3 * i + 2]), d3,
                                      cull != 0, PHOTON ? 1.0e30f : 1.0e20f, e,
                                      s.tri_rank ? s.tri_rank + (size_t)cube_face(d3) * s.num_tris : nullptr);
        tri[i] = h.tri;
        t[i] = h.t;
    } else {
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
            TraversalCount ct;
            const Hit h = coop_trace_exact<PHOTON, false>(s, mk(org[3 * i], org[3 * i + 1], org[3 * i + 2]),
                                                          mk(dir[3 * i], dir[3 * i + 1], dir[3 * i + 2]), cull != 0,
                                                          e, &ct);
            if ((threadIdx.x & 31) == 0) {
                tri[i] = h.tri;
                t[i] = h.t;
            }
        }
    }
    if (e) atomicOr(err, e);
}

__global__ void k_copy_from_host(unsigned long long* dst, const unsigned long long* src, uint32_t words) {
    for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) dst[w] = src[w];
}

__global__ void k_copy_descs(DescCopy list) {
    static_assert(sizeof(JobDesc) % 8 == 0, "JobDesc is copied in 8-byte words");
    if (blockIdx.x >= list.n) return;
    auto* dst = reinterpret_cast<unsigned long long*>(list.dst[blockIdx.x]);
    const auto* src = reinterpret_cast<const unsigned long long*>(list.src[blockIdx.x]);
    for (uint32_t w = threadIdx.x; w < sizeof(JobDesc) / 8; w += blockDim.x) dst[w] = src[w];
}

// one block per listed job: its JobState word by word
__global__ void k_gather_states(const JobDesc* jobs, StateGather list, JobState* out) {
    static_assert(sizeof(JobState) % 4 == 0, "JobState is copied in 32-bit words");
    if (blockIdx.x >= list.n) return;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(jobs[list.slot[blockIdx.x]].state);
    uint32_t* dst = reinterpret_cast<uint32_t*>(out + blockIdx.x);
    for (uint32_t w = threadIdx.x; w < sizeof(JobState) / 4; w += blockDim.x) dst[w] = src[w];
}

// ----------------------------------------------------------------------------------------------
// launchers
// ----------------------------------------------------------------------------------------------
static inline uint32_t blocks_for(uint32_t n, uint32_t b) { return (n + b - 1) / b; }

void launch_copy_from_host(void* dst, const void* src_mapped, size_t bytes, cudaStream_t s) {
    k_copy_from_host<<<1, 64, 0, s>>>(static_cast<unsigned long long*>(dst),
                                       static_cast<const unsigned long long*>(src_mapped), (uint32_t)(bytes / 8));
}
void launch_copy_descs(const DescCopy& list, cudaStream_t s) {
    if (list.n) k_copy_descs<<<list.n, 64, 0, s>>>(list);
}
void launch_gather_states(const JobDesc* jobs, const StateGather& list, JobState* out, cudaStream_t s) {
    if (list.n) k_gather_states<<<list.n, 64, 0, s>>>(jobs, list, out);
}
void launch_frame_begin(const LaunchSet& ls, const RayQueue& q, cudaStream_t s) {
    if (!ls.total) return;
    const uint32_t items = (ls.total - 1) / 4 + 1, bins = q.bins ? kBinCounters * kRayBins / 4 : 0;
    k_frame_begin<<<blocks_for(items > bins ? items : bins, 256), 256, 0, s>>>(ls, q);
}
// block sizes: a multiple of 32 up to the kernel's launch bound (0 or anything else: the bound)
static uint32_t block_or(uint32_t block, uint32_t bound) {
    return block >= 32 && block <= bound && block % 32 == 0 ? block : bound;
}

template <bool TEX>
static void launch_eye_t(const LaunchSet& ls, const RayQueue& q, bool mixed, uint32_t block, cudaStream_t s) {
    const uint32_t b = block_or(block, 128);
    if (mixed) {
        if (!TEX && ls.total <= kEyeMixedItems) k_eye<true, false, true><<<blocks_for(ls.total, b), b, 0, s>>>(ls, nullptr, nullptr, 0);
        else k_eye<true, TEX><<<blocks_for(ls.total, b), b, 0, s>>>(ls, nullptr, nullptr, 0);
        return;
    }
    if (!TEX && ls.total <= kEyeAheadItems)
        k_eye<false, false, true><<<blocks_for(ls.total, b), b, 0, s>>>(ls, q.counters + 3, q.eye_deferred, kEyeDeferred);
    else
        k_eye<false, TEX><<<blocks_for(ls.total, b), b, 0, s>>>(ls, q.counters + 3, q.eye_deferred, kEyeDeferred);
    // a fixed grid (the count is on the device): blocks beyond the deferred pixels exit at once
    k_eye_coop<TEX><<<32, kBlockWalk, 0, s>>>(ls, q.counters + 3, q.eye_deferred, kEyeDeferred);
}
void launch_eye(const LaunchSet& ls, const RayQueue& q, bool mixed, bool textured, uint32_t block, cudaStream_t s) {
    if (!ls.total) return;
    if (textured) launch_eye_t<true>(ls, q, mixed, block, s);
    else launch_eye_t<false>(ls, q, mixed, block, s);
}
void launch_grid(const JobDesc* jobs, const uint32_t* job_ids, uint32_t njobs, cudaStream_t s) {
    if (njobs) k_grid<<<blocks_for(njobs, 64), 64, 0, s>>>(jobs, job_ids, njobs);
}
void launch_cell_bounds(const JobDesc* jobs, const uint32_t* job_ids, uint32_t njobs, cudaStream_t s) {
    if (njobs) k_cell_bounds<<<njobs, 256, 0, s>>>(jobs, job_ids);
}
void launch_photon_fp32(const LaunchSet& ls, bool count, bool textured, cudaStream_t s) {
    if (!ls.total) return;
    const uint32_t b = blocks_for(ls.total, 128);
    if (count && textured) k_photon<true, true><<<b, 128, 0, s>>>(ls);
    else if (count) k_photon<true, false><<<b, 128, 0, s>>>(ls);
    else if (textured) k_photon<false, true><<<b, 128, 0, s>>>(ls);
    else k_photon<false, false><<<b, 128, 0, s>>>(ls);
}

void launch_photon_gen_fp32(const LaunchSet& ls, const RayQueue& q, bool textured, cudaStream_t s) {
    if (ls.total <= ls.first) return;
    const uint32_t n = ls.total - ls.first;
    if (textured) k_photon_gen<true><<<blocks_for(n, 128), 128, 0, s>>>(ls, q);
    else k_photon_gen<false><<<blocks_for(n, 128), 128, 0, s>>>(ls, q);
}
void launch_queue_reset(const RayQueue& q, cudaStream_t s) {
    if (q.counters) k_queue_reset<<<blocks_for(kBinCounters * kRayBins, 256), 256, 0, s>>>(q);
}
void launch_ray_bins_order(const RayQueue& q, cudaStream_t s) {
    if (q.key && q.bin_rank && q.bin_cost) k_ray_bins_order<<<1, 1024, 0, s>>>(q);
}
void launch_ray_bins(const RayQueue& q, cudaStream_t s) {
    if (!q.key || !q.capacity) return;
    k_ray_bins_scan<<<1, 1024, 0, s>>>(q.bins);
    k_ray_bins_scatter<<<blocks_for(q.capacity, 256), 256, 0, s>>>(q);
}

void launch_trace_photons_fp32(const LaunchSet& ls, const RayQueue& q, bool count, uint32_t persistent_blocks,
                               bool ahead, cudaStream_t s) {
    if (!ls.total) return;
    if (count) k_trace_photons<true, false><<<persistent_blocks, 128, 0, s>>>(ls, q);
    else if (ahead) k_trace_photons<false, true><<<persistent_blocks, 128, 0, s>>>(ls, q);
    else k_trace_photons<false, false><<<persistent_blocks, 128, 0, s>>>(ls, q);
    if (q.tail_lanes && q.tail_list) {
        // one warp per handed-over walk: enough warps for every SM
        if (count) k_trace_photons_tail<true><<<persistent_blocks, 128, 0, s>>>(ls, q);
        else k_trace_photons_tail<false><<<persistent_blocks, 128, 0, s>>>(ls, q);
    }
    launch_trace_photons_coop(ls, q, count, s);
}
void launch_trace_photons_coop(const LaunchSet& ls, const RayQueue& q, bool count, cudaStream_t s) {
    if (!ls.total || !q.slow) return;
    if (count) k_trace_photons_coop<true><<<64, kBlockWalk, 0, s>>>(ls, q);
    else k_trace_photons_coop<false><<<64, kBlockWalk, 0, s>>>(ls, q);
}

void launch_photon_store_fp32(const LaunchSet& ls, const RayQueue& q, uint32_t block, uint32_t grid_shift,
                              cudaStream_t s) {
    const uint32_t b = block_or(block, 128);
    if (ls.total) k_photon_store<<<blocks_for(q.capacity, b), b, 0, s>>>(ls, q, grid_shift);
}

template <bool AHEAD>
static uint32_t trace_photons_fit() {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_trace_photons<false, AHEAD>, 128, 0) != cudaSuccess) n = 4;
    return n > 0 ? (uint32_t)n : 1u;
}
uint32_t trace_photons_blocks_per_sm(bool ahead) {
    return ahead ? trace_photons_fit<true>() : trace_photons_fit<false>();
}
void launch_gather_fp32(const LaunchSet& ls, uint32_t block, cudaStream_t s) {
    const uint32_t b = block_or(block, 256);
    if (ls.total >= kGatherWideItems) k_gather<5><<<blocks_for(ls.total, b), b, 0, s>>>(ls);
    else if (ls.total) k_gather<4><<<blocks_for(ls.total, b), b, 0, s>>>(ls);
}
void launch_resolve_fp32(const LaunchSet& ls, uint32_t display, cudaStream_t s) {
    if (ls.total) k_resolve<<<blocks_for(ls.total, 256), 256, 0, s>>>(ls, display);
}
void launch_hash_build(const float4* pos, const float4* flux, uint32_t pw, uint32_t ph, uint32_t hash_num,
                       const float bbmin[3], float G, uint32_t flags, uint32_t* winner, uint32_t* count, cudaStream_t s) {
    k_hash_clear<<<blocks_for((hash_num - 1) / 4 + 1, 256), 256, 0, s>>>(winner, count, hash_num);
    const uint32_t n = pw * ph;
    if (n) k_hash_build<<<blocks_for(n, 256), 256, 0, s>>>(pos, flux, pw, ph, hash_num, bbmin[0], bbmin[1], bbmin[2], G, flags, winner, count);
}
void launch_fpmath(int fn, const float* x, const float* y, float* out, uint32_t n, cudaStream_t s) {
    if (n) k_fpmath<<<blocks_for(n, 256), 256, 0, s>>>(fn, x, y, out, n);
}

void launch_debug_trace(const DevScene& sc, const float* org, const float* dir, uint32_t n, bool photon, bool cull,
                        int mode, int32_t* tri, float* t, uint32_t* err, cudaStream_t s) {
    if (!n) return;
    const uint32_t threads = mode == 2 ? kBlockWalk : 128;
    const uint32_t blocks =
        (mode == 0 || mode == 3) ? blocks_for(n, 128) : (mode == 1 ? blocks_for(n, 4) : (n < 256 ? n : 256u));
    if (photon) k_debug_trace<true><<<blocks, threads, 0, s>>>(sc, org, dir, n, cull, mode, tri, t, err);
    else k_debug_trace<false><<<blocks, threads, 0, s>>>(sc, org, dir, n, cull, mode, tri, t, err);
}

}  // namespace sppm_dev
