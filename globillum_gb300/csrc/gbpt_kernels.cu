// gbpt_kernels.cu -- sm_103a kernels of the GB300 path-tracing hot path.
//
// The progressive frame runs as a wavefront over a pool of path slots.  The
// paths of a chunk (samples p0..p1-1 of every pixel) are handed out to the
// slots in path order; a slot whose path ends stores the path's sample and
// takes the next path, so every iteration works on a full queue until the
// chunk runs dry.  One iteration is two launches:
//   k_rays   traces the extension rays (closest hit) and the shadow rays of
//            the previous vertices (any hit) in one persistent grid
//   k_shade  adds the previous vertex's light sample if its shadow ray was
//            free; a miss adds handle_no_hit's contribution
//            (hybrid-pt.cpp:196-206) and ends the path; a hit draws the
//            bounce's uniforms, takes the area-light sample
//            (arealight-sampler-cpu.cpp:25-143), the BRDF sample and eval,
//            throughput and next ray of
//            compute_path_contribution_and_bounce (hybrid-pt.cpp:450-584)
// then k_combine folds the chunk's samples into the image with new_path's
// moving average (util-kernels.cu:17-25), in path order per pixel, so the
// image equals the reference's pixel-sequential one bit for bit.
// Tracing both ray kinds together halves the launches that end in a tail of
// a few long rays, and a traced ray leaves only its hit behind, so the
// traversal kernel carries no shading code (registers, refill cost).
//
// Traversal: compressed 8-wide BVH (80 B nodes, 8-bit quantised child
// boxes), node-group stack of 32 entries, octant-ordered child visits,
// conservative slab tests (relative slack 2e-5 on top of outward-rounded
// boxes), so the result equals the (t, id)-minimum over all triangles.
#include "gbpt_kernels.h"

#include <curand_kernel.h>

#include <algorithm>

namespace gb {

namespace {

constexpr int kBlock = 128;
// Resident 128-thread blocks per SM the traversal kernels are compiled for: 7
// (72 registers; 8 B of spills in the variants for several scenes, none in those
// for one).  1M-triangle frame, 64 spp, at 6 / 7 / 8 blocks: 35.7 / 34.0 / 33.9
// ms; 12 mixed scenes 3.19 / 3.09 / 3.01 ms; 262 K closest hits in 64 K triangles
// 95 / 94 / 96 us; 2 M shadow rays 319 / 297 / 290 us.
#ifndef GB_TRAV_MIN_BLOCKS
#define GB_TRAV_MIN_BLOCKS 7
#endif
constexpr int kStack = 32;
constexpr int kIterLimit = 1 << 22;
// Experimental build option, off by default (slower: the nodes are L2 hits): L2
// prefetch of hit child nodes.
#ifndef GB_PREFETCH
#define GB_PREFETCH 0
#endif
#ifndef GB_SHADE_MIN_BLOCKS
#define GB_SHADE_MIN_BLOCKS 7  // resident k_shade blocks per SM (72 registers)
#endif

__device__ __forceinline__ v3 ld3(const float4 a) { return mk(a.x, a.y, a.z); }

struct RayInv {
    v3 o, d, idir;
    uint32_t oxor;
};

__device__ __forceinline__ RayInv make_ray(v3 o, v3 d) {
    RayInv r;
    r.o = o; r.d = d;
    const float ooeps = 8.271806125530277e-25f;  // 2^-80 (tracers.cu:48-51)
    r.idir.x = 1.0f / (fabsf(d.x) > ooeps ? d.x : copysignf(ooeps, d.x));
    r.idir.y = 1.0f / (fabsf(d.y) > ooeps ? d.y : copysignf(ooeps, d.y));
    r.idir.z = 1.0f / (fabsf(d.z) > ooeps ? d.z : copysignf(ooeps, d.z));
    uint32_t oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
    r.oxor = oct ^ 7u;
    return r;
}

// Read-only 16-byte loads of the tree with cache hints: triangles without L1
// allocation (GB_TRI_NOALLOC), nodes with a 128-byte L2 fetch (GB_NODE_L2_128);
// plain __ldg otherwise.
#ifndef GB_TRI_NOALLOC
#define GB_TRI_NOALLOC 0
#endif
#ifndef GB_NODE_L2_128
#define GB_NODE_L2_128 0
#endif
__device__ __forceinline__ float4 ld_tri(const float4* p) {
#if GB_TRI_NOALLOC
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
#else
    return __ldg(p);
#endif
}
__device__ __forceinline__ float4 ld_node(const float4* p) {
#if GB_NODE_L2_128
    float4 v;
    asm("ld.global.nc.L2::128B.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
#else
    return __ldg(p);
#endif
}

// Packed FP32 (two lanes per 64-bit register) and 3-input min/max of sm_100+.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// The visit order of a node's hit children is a permutation of its 8-bit hit
// mask by the ray's octant: a 2 KB table in shared memory (2 instructions)
// instead of three conditional swaps (15): 38.0 -> 37.1 ms on the 1M-triangle
// 64-spp frame, 333 -> 321 us on 2 M shadow rays.
__device__ __forceinline__ uint8_t* order_table() {
    __shared__ __align__(4) uint8_t t[2048];  // [octant][mask]
    return t;
}
// Every bit of an 8-bit mask three times over: a hit leaf's triangles are
// those of the node's leaf bits that survive this mask.  Taken from a table
// and without asking which hit children are leaves, instead of a loop over the
// hit leaves (about 30 of a visit's 200 instructions): 36.7 -> 35.5 ms on the
// 1M-triangle 64-spp frame, 3.25 -> 3.18 ms on 12 mixed scenes.
__device__ __forceinline__ uint32_t* leaf_table() {
    __shared__ uint32_t t[256];
    return t;
}
// Bits of an 8-bit mask moved from position i to i ^ x (x in 0..7).
__device__ __forceinline__ uint32_t xor_permute8(uint32_t m, uint32_t x) {
    if (x & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (x & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (x & 4u) m = ((m & 0x0fu) << 4) | ((m >> 4) & 0x0fu);
    return m;
}

// Fills the tables: all threads of the block call it before they traverse.
__device__ __forceinline__ void fill_tables() {
    for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x) {
        uint32_t x = (i | (i << 8)) & 0x00f00fu;
        x = (x | (x << 4)) & 0x0c30c3u;
        leaf_table()[i] = ((x | (x << 2)) & 0x249249u) * 7u;
    }
    uint32_t* t = reinterpret_cast<uint32_t*>(order_table());
    for (uint32_t i = threadIdx.x; i < 512u; i += blockDim.x) {
        const uint32_t x = i >> 6, m = (i & 63u) << 2, w = xor_permute8(m, x), b0 = 1u << x, b1 = 1u << (x ^ 1u);
        t[i] = w | (w | b0) << 8 | (w | b1) << 16 | (w | b0 | b1) << 24;
    }
    __syncthreads();
}

// Intersects the 8 children of node `ni`; returns the node group (child
// base, hit bits 24-31 in visit order | imask) and the triangle group.
// Per axis the near and far planes are chosen once per node from the sign
// of the inverse direction (fma is monotonic in the plane index, so this
// equals taking min/max of the two plane distances per child); children are
// tested two at a time with packed FP32.  The test is conservative: a child
// is hit when lo * (1 - 2e-5) <= min(hi, bound), on top of outward-rounded
// boxes.  Empty slots (no leaf bits, imask bit 0) may test positive; they add
// neither a node nor a triangle.
//
// The ALU pipe (byte permutes, min/max, compares, selects; half rate) bounds
// this function, not FMA: 65-70 % against 17 % busy before, 64-69 % against
// 30 % with what follows.
//  - one PRMT places two plane bytes in the mantissas of two FP16 subnormals
//    (q 2^-24, exact), which the FMA pipe widens to FP32 (cvt.f32.f16), so
//    distances are in units of 2^24 (exact, and no plane step overflows that
//    did not before).  A PRMT per byte and an FADD to take the
//    magic number off again: 41.5 against 40.1 ms on the 1M-triangle 64-spp
//    frame, 566 against 530 us on 2 M shadow rays.
//  - the hit bits are the signs of min(hi, bound) - lo (1 - 2e-5), one packed
//    FMA per pair, shifted into the mask by a funnel shift each, instead of
//    two slack multiplications, a compare and a predicated OR: 40.1 -> 39.4 ms
//    and 530 -> 505 us.
// Loading each axis's near and far words by sign instead of selecting them
// (six 8-byte loads for three of 16 bytes, 12 selects less) changes nothing.
__device__ __forceinline__ uint64_t half_pair(uint32_t h) {
    uint64_t r;
    asm("{.reg .f16 a, b; .reg .f32 x, y; mov.b32 {a, b}, %1; cvt.f32.f16 x, a; cvt.f32.f16 y, b; mov.b64 %0, {x, y};}"
        : "=l"(r) : "r"(h));
    return r;
}
__device__ __forceinline__ void intersect_node(const float4* __restrict__ nodes, uint32_t ni, const RayInv& r,
                                               float bound, uint2* ng, uint2* tg, uint32_t* tv) {
    const float4* n = nodes + 5 * (size_t)ni;
    float4 n0 = ld_node(n + 0), n1 = ld_node(n + 1), n2 = ld_node(n + 2), n3 = ld_node(n + 3), n4 = ld_node(n + 4);
    const bool fx = r.idir.x < 0.0f, fy = r.idir.y < 0.0f, fz = r.idir.z < 0.0f;
    uint32_t ew = __float_as_uint(n0.w);
    float sx = __uint_as_float((ew & 0xffu) << 23);
    float sy = __uint_as_float(((ew >> 8) & 0xffu) << 23);
    float sz = __uint_as_float(((ew >> 16) & 0xffu) << 23);
    const uint32_t imask = ew >> 24;
    const float aix = sx * r.idir.x, aiy = sy * r.idir.y, aiz = sz * r.idir.z;
    const uint64_t AX = pack2(aix, aix), AY = pack2(aiy, aiy), AZ = pack2(aiz, aiz);
    const float k24 = 5.9604644775390625e-08f;  // 2^-24
    const float aox = (n0.x - r.o.x) * r.idir.x * k24, aoy = (n0.y - r.o.y) * r.idir.y * k24,
                aoz = (n0.z - r.o.z) * r.idir.z * k24;
    bound *= k24;
    const uint64_t OX = pack2(aox, aox), OY = pack2(aoy, aoy), OZ = pack2(aoz, aoz);
    const uint64_t KN = pack2(-0.99998f, -0.99998f);
    uint32_t hm = 0;  // children missed, by slot
#pragma unroll
    for (int half = 1; half >= 0; --half) {
        uint32_t qlx = __float_as_uint(half ? n2.y : n2.x), qly = __float_as_uint(half ? n2.w : n2.z);
        uint32_t qlz = __float_as_uint(half ? n3.y : n3.x), qhx = __float_as_uint(half ? n3.w : n3.z);
        uint32_t qhy = __float_as_uint(half ? n4.y : n4.x), qhz = __float_as_uint(half ? n4.w : n4.z);
        uint32_t nx = fx ? qhx : qlx, fxw = fx ? qlx : qhx;
        uint32_t ny = fy ? qhy : qly, fyw = fy ? qly : qhy;
        uint32_t nz = fz ? qhz : qlz, fzw = fz ? qlz : qhz;
#pragma unroll
        for (int j = 2; j >= 0; j -= 2) {
            // plane distances q * a + o of children j, j + 1 of this half
#define GB_PLANES(w, A, O) fma2(half_pair(__byte_perm(w, 0u, j ? 0x4342u : 0x4140u)), A, O)
            float tnx0, tnx1, tny0, tny1, tnz0, tnz1, tfx0, tfx1, tfy0, tfy1, tfz0, tfz1;
            unpack2(GB_PLANES(nx, AX, OX), tnx0, tnx1);
            unpack2(GB_PLANES(ny, AY, OY), tny0, tny1);
            unpack2(GB_PLANES(nz, AZ, OZ), tnz0, tnz1);
            unpack2(GB_PLANES(fxw, AX, OX), tfx0, tfx1);
            unpack2(GB_PLANES(fyw, AY, OY), tfy0, tfy1);
            unpack2(GB_PLANES(fzw, AZ, OZ), tfz0, tfz1);
#undef GB_PLANES
            const uint64_t lo = pack2(max3(tnx0, tny0, fmaxf(tnz0, 0.0f)), max3(tnx1, tny1, fmaxf(tnz1, 0.0f)));
            const uint64_t hi = pack2(min3(tfx0, tfy0, fminf(tfz0, bound)), min3(tfx1, tfy1, fminf(tfz1, bound)));
            float d0, d1;
            unpack2(fma2(lo, KN, hi), d0, d1);
            hm = __funnelshift_l(__float_as_uint(d1), hm, 1);
            hm = __funnelshift_l(__float_as_uint(d0), hm, 1);
        }
    }
    hm = ~hm & 0xffu;
    const uint32_t inner = hm & imask;
#if GB_PREFETCH
    // the hit inner children will be visited: start their fetch into L2 now
    for (uint32_t m = inner; m; m &= m - 1u) {
        const uint32_t s = (uint32_t)__ffs(m) - 1u;
        const float4* cp = nodes + 5 * (size_t)(__float_as_uint(n1.x) + (uint32_t)__popc(imask & ((1u << s) - 1u)));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(cp)));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(cp + 4)));
    }
#endif
    *ng = make_uint2(__float_as_uint(n1.x), ((uint32_t)order_table()[(r.oxor << 8) | inner] << 24) | imask);
    // the triangles of the hit leaves, and what all their bits are counted
    // against (n1.z, zero for inner and empty slots)
    *tg = make_uint2(__float_as_uint(n1.y), leaf_table()[hm] & __float_as_uint(n1.z));
    *tv = __float_as_uint(n1.z);
}

// Resumable traversal state of one ray (the node-group stack lives beside it).
struct Trav {
    uint2 ng;
    uint2 tg;         // pending triangles: the node's first, and leaf bits still to test
    uint32_t tv;      // the node's leaf bits: triangle of bit b = first + bits of tv below b
    uint2 nt;         // second pending group (policy 0)
    uint32_t nv;
    int sp;
    float best_t, bb, bg;
    uint32_t best_id;
};

// best_t starts at t_max (at most FLT_MAX, so that an infinite distance is
// never a hit): a hit at t_max exactly is taken, as closer() prefers any id to
// none, and one test serves both limits.
__device__ __forceinline__ void trav_init(Trav& s, const RayInv& r, float tmax) {
    s.ng = make_uint2(0u, 0x80000000u | (1u << (r.oxor ^ 7u)));
    s.tg = make_uint2(0u, 0u);
    s.nt = make_uint2(0u, 0u);
    s.sp = 0;
    s.best_t = fminf(tmax, FLT_MAX);
    s.best_id = 0xffffffffu;
    s.bb = 0.0f;
    s.bg = 0.0f;
}

// Traversal steps.  The stack holds node groups (hit bits 24-31 set) and
// postponed triangle groups (24-bit triangle mask, bits 24-31 clear).
//
// tri_step: one triangle of the current triangle group.  Returns true when
// an any-hit query has found its hit.
template <bool INSTR>
__device__ __forceinline__ bool tri_step(const float4* __restrict__ tris, const RayInv& r, bool any, Trav& s,
                                         uint32_t* ntri) {
    const uint32_t below = s.tg.y - 1u;  // bits below the lowest one, and the others less it
    const float4* tp = tris + 3 * (size_t)(s.tg.x + (uint32_t)__popc(s.tv & below & ~s.tg.y));
    s.tg.y &= below;
    float4 a0 = ld_tri(tp + 0), a1 = ld_tri(tp + 1), a2 = ld_tri(tp + 2);
    if (INSTR) ++*ntri;
    // intersect_tri with its conditions joined at the end (the same operations;
    // det = 0 gives u = inf or NaN, which is no hit either): no branch to
    // reconverge between the steps, 38.4 -> 37.8 ms on the 1M-triangle frame
    const v3 e1 = ld3(a1), e2 = ld3(a2);
    const v3 p = fcross(r.d, e2);
    const float inv = 1.0f / fdot(e1, p);
    const v3 w = r.o - ld3(a0);
    const float u = fdot(w, p) * inv;
    const v3 q = fcross(w, e1);
    const float v = fdot(r.d, q) * inv, t = fdot(e2, q) * inv;
    const uint32_t id = __float_as_uint(a0.w);
    if (u >= 0.0f && u <= 1.0f && v >= 0.0f && u + v <= 1.0f && t > 0.0f && closer(t, id, s.best_t, s.best_id)) {
        s.best_t = t; s.best_id = id; s.bb = u; s.bg = v;
        return any;
    }
    return false;
}

// visit_node: the next node of the current node group (not empty).  Returns
// true when the stack overflows.
template <bool INSTR, int STACK = kStack>
__device__ __forceinline__ bool visit_node(const float4* __restrict__ nodes, const RayInv& r, Trav& s,
                                           uint2* stack, uint32_t* status, uint32_t* nvis, uint2* tg,
                                           uint32_t* tv) {
    const uint32_t k = 31u - (uint32_t)__clz(s.ng.y);
    s.ng.y &= ~(1u << k);
    const uint32_t slot = (k - 24u) ^ r.oxor;
    const uint32_t imask = s.ng.y & 0xffu;
    const uint32_t child = s.ng.x + (uint32_t)__popc(imask & ((1u << slot) - 1u));
    if (s.ng.y > 0x00ffffffu) {
        if (s.sp >= STACK) { atomicOr(status, ST_STACK_OVERFLOW); return true; }
        stack[s.sp++] = s.ng;
    }
    if (INSTR) ++*nvis;
    intersect_node(nodes, child, r, s.best_t, &s.ng, tg, tv);
    return false;
}

// node_step (current triangle group empty): one node of the current node
// group, or a stack pop.  Returns true when the ray is finished; the result
// is the (t, id)-minimum in s (any-hit: best_id != none when found).
template <bool INSTR, int STACK = kStack>
__device__ __forceinline__ bool node_step(const float4* __restrict__ nodes, const RayInv& r, Trav& s,
                                          uint2* stack, uint32_t* status, uint32_t* nvis) {
    if (s.ng.y > 0x00ffffffu) {
        const bool over = visit_node<INSTR, STACK>(nodes, r, s, stack, status, nvis, &s.tg, &s.tv);
        // these policies stack groups and hand them to other lanes: bits without gaps, for any tv
        uint32_t m = 0;
        for (uint32_t left = s.tg.y; left; left &= left - 1u) m |= 1u << __popc(s.tv & (left - 1u) & ~left);
        s.tg.y = m;
        s.tv = 0xffffffffu;
        return over;
    }
    if (s.sp > 0) {
        uint2 g = stack[--s.sp];
        if (g.y > 0x00ffffffu) s.ng = g;
        else s.tg = g;
        return false;
    }
    return true;
}

// warp_step: triangle policy 0, called by the whole warp.  The warp either
// visits a node with every lane that can, or tests one triangle with every
// lane that has some pending, whichever keeps more lanes busy: a node visit
// of a closest-hit ray yields triangles one time in eight, so testing them
// as they come runs the test with two or three lanes after nearly every
// visit.  A lane with a pending group goes on visiting nodes until it has a
// second one (nt), which it cannot store further.  A pop and the visit it
// leads to are one step, and a lane whose last group is empty is finished at
// the end of the step.  GB_TRI_RATIO (triangle lanes times this >= node lanes
// tests triangles) on the 1M-triangle frame at 64 spp / 1 spp / the 256x256
// 16-spp room: 34.3 34.0 34.1 34.3 ms / 896 893 904 909 us / 822 833 847 848 us
// for 1 / 2 / 3 / 4; every pending triangle after each visit, with pops as steps
// of their own, was slower by a tenth when the vote was introduced.  A lane is
// finished when it has neither, so the two votes of the step also tell which
// lanes are idle.
#ifndef GB_TRI_RATIO
#define GB_TRI_RATIO 2
#endif
__device__ __forceinline__ bool has_tri(const Trav& s) { return s.tg.y != 0u; }
__device__ __forceinline__ bool has_node(const Trav& s) { return s.nt.y == 0u && (s.ng.y > 0x00ffffffu || s.sp > 0); }
// A lane without a ray, or whose any-hit query is answered, has neither.
__device__ __forceinline__ void trav_stop(Trav& s) {
    s.tg.y = s.nt.y = s.ng.y = 0u;
    s.sp = 0;
}
template <bool INSTR, int STACK>
__device__ __forceinline__ void warp_step(bool tri, bool node, uint32_t mt, uint32_t mn,
                                          const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                          const RayInv& r, bool any, Trav& s, uint2* stack,
                                          uint32_t* status, uint32_t* nvis, uint32_t* ntri) {
    if (__popc(mt) * GB_TRI_RATIO >= __popc(mn)) {
        if (tri) {
            const bool found = tri_step<INSTR>(tris, r, any, s, ntri);
            if (s.tg.y == 0u) {
                s.tg = s.nt;
                s.tv = s.nv;
                s.nt.y = 0u;
            }
            if (found) trav_stop(s);
        }
    } else if (node) {
        if (s.ng.y <= 0x00ffffffu) s.ng = stack[--s.sp];
        uint2 tg = make_uint2(0u, 0u);
        uint32_t tv = 0u;
        const bool over = visit_node<INSTR, STACK>(nodes, r, s, stack, status, nvis, &tg, &tv);
        if (s.tg.y == 0u) {
            s.tg = tg;
            s.tv = tv;
        } else {
            s.nt = tg;
            s.nv = tv;
        }
        if (over) trav_stop(s);
    }
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ void add_stats(unsigned long long* s, uint32_t v) {
    uint32_t w = __reduce_add_sync(0xffffffffu, v);
    if (lane_id() == 0u && w) atomicAdd(s, (unsigned long long)w);
}

// ----------------------------------------------------------------- kernels

__device__ __forceinline__ MrgState mrg_pack(const curandStateMRG32k3a& st) {
    MrgState m;
    for (int k = 0; k < 3; ++k) { m.s1[k] = st.s1[k]; m.s2[k] = st.s2[k]; }
    return m;
}
// 24-byte states as three 8-byte accesses.
__device__ __forceinline__ MrgState ld_mrg(const MrgState* base, size_t i) {
    const uint2* q = reinterpret_cast<const uint2*>(base + i);
    uint2 a = rec_ld(q), b = rec_ld(q + 1), c = rec_ld(q + 2);
    MrgState m;
    m.s1[0] = a.x; m.s1[1] = a.y; m.s1[2] = b.x; m.s2[0] = b.y; m.s2[1] = c.x; m.s2[2] = c.y;
    return m;
}
__device__ __forceinline__ void st_mrg(MrgState* base, size_t i, const MrgState& m) {
    uint2* q = reinterpret_cast<uint2*>(base + i);
    rec_st(q, make_uint2(m.s1[0], m.s1[1]));
    rec_st(q + 1, make_uint2(m.s1[2], m.s2[0]));
    rec_st(q + 2, make_uint2(m.s2[1], m.s2[2]));
}
// Three uniforms of a stream: the numbers curand_uniform gives (equal for all
// 2^32 - 209 values of z and for four draws from each of 2^30 pseudo-random
// states), with the recurrences in integers and three double operations a
// draw (an SM does two double operations a clock): k_jitter_pool of the 256x256
// 16-spp room 43 -> 25 us (with mrg_apply reducing rows), of 12 mixed scenes
// 262 -> 163 us.
__device__ __forceinline__ v3 draw3(MrgState* m) {
    const float x = mrg_uniform(mrg_next(m->s1, m->s2));
    const float y = mrg_uniform(mrg_next(m->s1, m->s2));
    const float z = mrg_uniform(mrg_next(m->s1, m->s2));
    return mk(x, y, z);
}

// The state curand_init(seed, sub, 0) leaves: curand_init of subsequence 0
// (no skip-ahead) advanced by sub * 2^76 steps with the table's jumps, one
// 3x3 matrix product per component for each set bit of sub, in exact
// integer arithmetic mod m1 / m2.
__device__ __forceinline__ MrgState mrg_stream(const MrgSubseqTable& T, uint32_t seed, uint32_t sub) {
    curandStateMRG32k3a s;
    curand_init((unsigned long long)seed, 0ull, 0ull, &s);
    MrgState m = mrg_pack(s);
    for (int k = 0; sub != 0u; ++k, sub >>= 1)
        if (sub & 1u) {
            mrg_apply(m.s1, T.j1[k], 209u, kMrgM1);
            mrg_apply(m.s2, T.j2[k], 22853u, kMrgM2);
        }
    return m;
}

// curand states right after curand_init(seed, pixel, 0) (util-kernels.cu:277-285)
// for every pixel of every scene of the frame (pixel = index within its scene).
__global__ void k_rng_init_frame(Frame F, const MrgSubseqTable T) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= F.ntot) return;
    const SceneRec& R = F.scenes[F.pscene[g]];
    st_mrg(F.pristine, (size_t)g, mrg_stream(T, R.seed, (uint32_t)(g - (int)R.pixel_base)));
}

// States of curand_init(seed, sub[i], 0): method 0 by curand_init itself,
// 1 by mrg_stream.
__global__ void k_mrg_states(const MrgSubseqTable T, uint32_t seed, const uint32_t* sub, int n, int method,
                             uint32_t* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    MrgState m;
    if (method == 0) {
        curandStateMRG32k3a s;
        curand_init((unsigned long long)seed, (unsigned long long)sub[i], 0ull, &s);
        m = mrg_pack(s);
    } else {
        m = mrg_stream(T, seed, sub[i]);
    }
    for (int k = 0; k < 3; ++k) { out[6 * i + k] = m.s1[k]; out[6 * i + 3 + k] = m.s2[k]; }
}

// Scene and Halton light draw of every global pixel.
__global__ void k_fill_pscene(Frame F) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= F.ntot) return;
    int lo = 0, hi = F.nscenes - 1;
    while (lo < hi) {  // last scene whose pixel_base <= g
        int mid = (lo + hi + 1) >> 1;
        if ((int)F.scenes[mid].pixel_base <= g) lo = mid;
        else hi = mid - 1;
    }
    F.pscene[g] = (uint32_t)lo;
    // the pixel's light draw of GB_RNG_HALTON_LIGHT, the same for all its
    // paths and bounces: about 650 instructions of digit loops and divisions,
    // against 1100 for the rest of a hit's shading (256x256 room at 16 spp:
    // 1.045 -> 1.007 ms)
    if (F.halton) {
        const int pid = g - (int)F.scenes[lo].pixel_base + 1;
        F.halton[g] = make_float2(halton(pid, 2), halton(pid, 3));
    }
}

// ------------------------------------------------------------ path slots --
// A slot carries one path (scene, pixel, sample p) at a time.  The frame's
// pixels are laid out scene after scene with scenes sorted by spp (largest
// first), so the pixels that still take a sample in round p form the prefix
// [0, N_p) and a chunk's paths enumerate without holes: path l of the chunk
// is (p0 + r, l - round_start[r]) for the round r holding l.  The
// reference's three identically seeded per-pixel pools
// (hybrid-pt.cpp:83-95, util-kernels.cu:284) become:
//   camera jitter  = update p of the pixel's stream, read from the chunk's
//                    jitter pool (k_jitter_pool walks each pixel's stream)
//   lens sample    = update p of pixel (pixel+17)%n (raygen.cu:100-106)
//   light/path     = updates pL, pL+1, ... one per bounce (hybrid-pt.h:229-233):
//                    k_jitter_pool walks the pixel's stream cursor over the
//                    chunk's paths (a jump of L updates, 3L generator steps,
//                    mrg_jump, per path) and leaves each path's start state
//                    in the chunk's stream pool.
// A path's stream therefore depends only on (pixel, p): a launch may start
// several paths of one pixel, in any order, on any slots.
// The state n jumps on.
__device__ __forceinline__ MrgState mrg_skip(MrgState s, const MrgPowers& T, uint32_t n) {
    for (int k = 0; n != 0u; ++k, n >>= 1)
        if (n & 1u) mrg_jump(s.s1, s.s2, T.j1[k], T.j2[k]);
    return s;
}
// A pixel's camera-jitter and light/path streams `r` paths after the chunk's
// start: a frame starts at curand_init(seed, pixel, 0), a later chunk where the
// last one ended.  J: jumps by the three draws of a jitter update.
__device__ __forceinline__ MrgState jitter_stream(const Frame& F, const RenderParams& P, const MrgPowers& J,
                                                  uint32_t pix, uint32_t r) {
    return mrg_skip(ld_mrg(P.p0 == 0 ? F.pristine : F.jcursor, (size_t)pix), J, r);
}
__device__ __forceinline__ MrgState path_stream(const Frame& F, const RenderParams& P, const SceneRec& R,
                                                uint32_t pix, uint32_t r) {
    return mrg_skip(ld_mrg(P.p0 == 0 ? F.pristine : F.cursor, (size_t)pix), R.jump, r);
}

// Per pixel, for the paths p of the pixel in the chunk from round pool_round
// on (path l = round_start[p - p0] + pixel): its camera jitter (update p of the
// pixel's jitter stream) and the state of its light/path stream (L updates per
// path: one jump of 3 L generator steps from the previous path's).  Paths that
// restart on a slot take these entries, in any order and several per pixel at
// once; the first paths (k_start, k_paths) jump to their own states instead,
// which saves 80 B of pool traffic per path and most of this kernel.  Both
// streams' cursors then move on to the next chunk.
__global__ void k_jitter_pool(Frame F, RenderParams P, const MrgPowers J) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= F.ntot) return;
    const SceneRec& R = F.scenes[F.nscenes == 1 ? 0u : F.pscene[g]];
    const int rounds = min(P.rounds, R.spp - P.p0);
    const int r0 = min(P.pool_round, rounds);
    if (rounds <= 0) return;
    MrgState s = jitter_stream(F, P, J, (uint32_t)g, (uint32_t)r0);
    MrgState c = path_stream(F, P, R, (uint32_t)g, (uint32_t)r0);
    for (int r = r0; r < rounds; ++r) {
        const uint32_t l = P.round_start[r] + (uint32_t)g;
        v3 j = draw3(&s);
        rec_st(&F.jpool[l], make_float4(j.x, j.y, j.z, 0.0f));
        st_mrg(F.spool, l, c);
        mrg_jump(c.s1, c.s2, R.jump.j1[0], R.jump.j2[0]);  // = L draw3 calls
    }
    if (P.more) {
        st_mrg(F.jcursor, (size_t)g, s);
        st_mrg(F.cursor, (size_t)g, c);
    }
}

// Ray differentials of a slot, 12 floats in 3 planes of nslots float4.
__device__ __forceinline__ RayDiff ld_rdiff(const Frame& F, uint32_t slot) {
    const size_t n = (size_t)F.nslots;
    const float4 a = F.rdiff[slot], b = F.rdiff[n + slot], c = F.rdiff[2 * n + slot];
    RayDiff r;
    r.uo = mk(a.x, a.y, a.z);
    r.ud = mk(a.w, b.x, b.y);
    r.ro = mk(b.z, b.w, c.x);
    r.rd = mk(c.y, c.z, c.w);
    return r;
}
__device__ __forceinline__ void st_rdiff(const Frame& F, uint32_t slot, const RayDiff& r) {
    const size_t n = (size_t)F.nslots;
    F.rdiff[slot] = make_float4(r.uo.x, r.uo.y, r.uo.z, r.ud.x);
    F.rdiff[n + slot] = make_float4(r.ud.y, r.ud.z, r.ro.x, r.ro.y);
    F.rdiff[2 * n + slot] = make_float4(r.ro.z, r.rd.x, r.rd.y, r.rd.z);
}

__device__ __forceinline__ Sector pack_sector(v3 a, v3 b, uint32_t c, uint32_t d) {
    return Sector{{__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z), __float_as_uint(b.x),
                   __float_as_uint(b.y), __float_as_uint(b.z), c, d}};
}
__device__ __forceinline__ v3 sec3(const Sector& s, int k) {
    return mk(__uint_as_float(s.w[k]), __uint_as_float(s.w[k + 1]), __uint_as_float(s.w[k + 2]));
}
// The `path` and `strm` sectors of a slot: throughput, accumulation, stream
// and pending light sample.
__device__ __forceinline__ void st_path(const Frame& F, uint32_t slot, v3 tp, v3 acc, const MrgState& m, v3 pend) {
    rec_st(&F.path[slot], pack_sector(tp, acc, __float_as_uint(pend.x), __float_as_uint(pend.y)));
    rec_st(&F.strm[slot], Sector{{m.s1[0], m.s1[1], m.s1[2], m.s2[0], m.s2[1], m.s2[2], __float_as_uint(pend.z), 0u}});
}

// Path l of the chunk: its pixel, scene, sample index, camera ray and stream.
struct PathStart {
    uint32_t pix, sc, path;
    int x, y;
    v3 o, d;
    MrgState st;
};
// J: jump to the path's streams; null: they are in the chunk's pool.
__device__ __forceinline__ PathStart path_start(const Frame& F, const RenderParams& P, uint32_t l,
                                                const MrgPowers* J) {
    int lo = 0, hi = P.rounds - 1;
    while (lo < hi) {  // round holding path l
        int mid = (lo + hi + 1) >> 1;
        if (P.round_start[mid] <= l) lo = mid;
        else hi = mid - 1;
    }
    PathStart s;
    s.pix = l - P.round_start[lo];
    s.sc = F.nscenes == 1 ? 0u : F.pscene[s.pix];
    s.path = (uint32_t)P.p0 + (uint32_t)lo;
    const SceneRec& R = F.scenes[s.sc];
    const uint32_t lp = s.pix - R.pixel_base, lens = R.pixel_base + (lp + 17u) % (uint32_t)R.n;
    const bool aperture = R.cam.aperture != 0.0f;
    v3 j, lj = mk(0.0f, 0.5f, 0.5f);
    if (J) {
        MrgState js = jitter_stream(F, P, *J, s.pix, (uint32_t)lo);
        j = draw3(&js);
        if (aperture) {
            js = jitter_stream(F, P, *J, lens, (uint32_t)lo);
            lj = draw3(&js);
        }
        s.st = path_stream(F, P, R, s.pix, (uint32_t)lo);
    } else {
        const float4* jp = F.jpool + P.round_start[lo];
        j = ld3(rec_ld(&jp[s.pix]));
        if (aperture) lj = ld3(rec_ld(&jp[lens]));
        s.st = ld_mrg(F.spool, l);
    }
    const float lx = aperture ? lj.z - 0.5f : 0.0f, ly = aperture ? lj.y - 0.5f : 0.0f;
    s.x = (int)(lp % (uint32_t)R.w);
    s.y = (int)(lp / (uint32_t)R.w);
    camera_ray(R.cam, s.x, s.y, j.x, j.y, lx, ly, &s.o, &s.d);
    return s;
}

// Path s on a slot.
__device__ __forceinline__ void put_path(const Frame& F, const RenderParams& P, uint32_t slot, const PathStart& s) {
    rec_st(&F.ray[slot], pack_sector(s.o, s.d, s.path << 10, s.pix));
    st_path(F, slot, mk(1.0f, 1.0f, 1.0f), mk(0.0f, 0.0f, 0.0f), s.st, mk(0.0f, 0.0f, 0.0f));
    if (P.mode == MODE_FROZEN) F.tp0[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    if (P.textured && F.scenes[s.sc].S.texcoord) st_rdiff(F, slot, camera_diff(F.scenes[s.sc].cam, s.x, s.y));
}
// Path l of the chunk, from the pool, on a slot.
__device__ __forceinline__ void start_path(const Frame& F, const RenderParams& P, uint32_t slot, uint32_t l) {
    put_path(F, P, slot, path_start(F, P, l, nullptr));
}

// The scene of a pixel's paths; a frame of one scene needs no load.
__device__ __forceinline__ uint32_t scene_of(const Frame& F, uint32_t pix) {
    return F.nscenes == 1 ? 0u : F.pscene[pix];
}

// The iteration index lives in F.iter (device), so an iteration's launches
// are the same every time (graph-capturable).
__device__ __forceinline__ uint32_t* ctr_set(const Frame& F, int it) { return F.ctr + 8 * (it % 3); }

// The sample of a path that ended (new_path's input to the moving average):
// path p's colour at sample index round_start[p - p0] + pixel.
__device__ __forceinline__ void store_sample(const Frame& F, const RenderParams& P, uint32_t pix, uint32_t pbv,
                                             v3 acc) {
    rec_st(&F.samples[P.round_start[(pbv >> 10) - (uint32_t)P.p0] + pix], make_float4(acc.x, acc.y, acc.z, 0.0f));
}

// Adjoint mode: starts the next paths of the chunk on the slots whose paths
// k_adjoint has swept, appending them to the next extension queue.
__global__ void __launch_bounds__(kBlock) k_regen(Frame F, RenderParams P) {
    uint32_t* cn = ctr_set(F, F.iter[1] + 1);
    const uint32_t count = cn[CTR_DONE];
    uint32_t* qout = F.q[(F.iter[1] + 1) & 1];
    __shared__ uint32_t s_l, s_q;
    for (uint32_t base = blockIdx.x * kBlock; base < count; base += gridDim.x * kBlock) {
        if (threadIdx.x == 0) {
            const uint32_t n = min(count - base, (uint32_t)kBlock);
            const uint32_t l = atomicAdd(F.path_ctr, n);
            const uint32_t go = l < P.chunk_paths ? min(n, P.chunk_paths - l) : 0u;
            s_l = l;
            s_q = go ? atomicAdd(&cn[CTR_EXT], go) : 0u;
            if (go) atomicAdd(&cn[CTR_STARTED], go);
        }
        __syncthreads();
        const uint32_t i = base + threadIdx.x, l = s_l + threadIdx.x;
        if (i < count && l < P.chunk_paths) {
            const uint32_t slot = F.q[5][i];
            start_path(F, P, slot, l);
            qout[s_q + threadIdx.x] = slot;
        }
        __syncthreads();
    }
}

// First paths of a chunk: slot s takes path s.  A thread starts the paths of
// one pixel in `group` rounds one after the other, from where the pixel's
// streams are then.  Sets the queue of iteration 0 (the counters are zero) and
// the iteration index.
__global__ void __launch_bounds__(kBlock) k_start(Frame F, RenderParams P, int nstart, int group, const MrgPowers J) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const int r0 = (int)blockIdx.y * group;
    if (g == 0 && r0 == 0) {
        *F.path_ctr = (uint32_t)nstart;
        F.iter[0] = 0;
        F.ctr[CTR_EXT] = (uint32_t)nstart;
        F.ctr[CTR_STARTED] = (uint32_t)nstart;
    }
    if (g >= (uint32_t)F.ntot || P.round_start[r0] + g >= (uint32_t)nstart) return;
    PathStart s;
    s.pix = g;
    s.sc = F.nscenes == 1 ? 0u : F.pscene[g];
    const SceneRec& R = F.scenes[s.sc];
    const int r1 = min(min(r0 + group, P.rounds), R.spp - P.p0);
    if (r0 >= r1) return;
    const uint32_t lp = g - R.pixel_base;
    s.x = (int)(lp % (uint32_t)R.w);
    s.y = (int)(lp / (uint32_t)R.w);
    const bool aperture = R.cam.aperture != 0.0f;
    MrgState js = jitter_stream(F, P, J, g, (uint32_t)r0), ls = js;
    if (aperture) ls = jitter_stream(F, P, J, R.pixel_base + (lp + 17u) % (uint32_t)R.n, (uint32_t)r0);
    s.st = path_stream(F, P, R, g, (uint32_t)r0);
    for (int r = r0; r < r1; ++r) {
        const uint32_t l = P.round_start[r] + g;
        if (l >= (uint32_t)nstart) break;
        const v3 j = draw3(&js);
        float lx = 0.0f, ly = 0.0f;
        if (aperture) {
            const v3 lj = draw3(&ls);
            lx = lj.z - 0.5f;
            ly = lj.y - 0.5f;
        }
        s.path = (uint32_t)(P.p0 + r);
        camera_ray(R.cam, s.x, s.y, j.x, j.y, lx, ly, &s.o, &s.d);
        put_path(F, P, l, s);
        F.q[0][l] = l;
        mrg_jump(s.st.s1, s.st.s2, R.jump.j1[0], R.jump.j2[0]);  // = L draw3 calls
    }
}

// (t, canonical id) as one 64-bit key whose unsigned order is the
// lexicographic closest-hit order: t > 0, so its bits order like its value.
__device__ __forceinline__ unsigned long long hit_key(float t, uint32_t id) {
    return ((unsigned long long)__float_as_uint(t) << 32) | id;
}

// Warp-cooperative triangle phase (triangle policy 3): the pending triangles
// of all active lanes are tested by the whole warp, 32 at a time.  A warp
// scan of the per-lane counts numbers the (lane, triangle) pairs; tester
// lane g finds its owner (the last lane whose exclusive count is <= g), the
// owner's k-th pending triangle, and the owner's ray through shuffles.  Hits
// resolve per owner by an atomicMin of hit_key in shared memory, so the
// result is the same lexicographic minimum as testing sequentially.  A new
// closest hit's barycentrics are recomputed by its owner from the shading
// record with the same (v0, v1 - v0, v2 - v0) arithmetic as the triangle
// layout, so they are bit-identical too.  All 32 lanes must call this.
template <bool INSTR>
__device__ __forceinline__ bool coop_triangles(bool act, const float4* tris, const float4* shade, const RayInv& r,
                                               bool any, Trav& s, unsigned long long* skey, uint32_t* ntri) {
    const uint32_t lane = lane_id();
    const uint32_t cnt = act ? (uint32_t)__popc(s.tg.y) : 0u;
    uint32_t incl = cnt;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (total == 0u) return false;
    const uint32_t excl = incl - cnt;
    const unsigned long long mine = act ? hit_key(s.best_t, s.best_id) : ~0ull;
    skey[lane] = mine;
    __syncwarp();
    for (uint32_t base = 0; base < total; base += 32u) {
        const uint32_t g = base + lane;
        uint32_t o = 0;
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1) {
            uint32_t c = o + step;
            if (__shfl_sync(0xffffffffu, excl, (int)c) <= g) o = c;
        }
        const uint32_t om = __shfl_sync(0xffffffffu, s.tg.y, (int)o);
        const uint32_t ob = __shfl_sync(0xffffffffu, s.tg.x, (int)o);
        const uint32_t oe = __shfl_sync(0xffffffffu, excl, (int)o);
        const v3 ro = mk(__shfl_sync(0xffffffffu, r.o.x, (int)o), __shfl_sync(0xffffffffu, r.o.y, (int)o),
                         __shfl_sync(0xffffffffu, r.o.z, (int)o));
        const v3 rd = mk(__shfl_sync(0xffffffffu, r.d.x, (int)o), __shfl_sync(0xffffffffu, r.d.y, (int)o),
                         __shfl_sync(0xffffffffu, r.d.z, (int)o));
        const float4* otris = (const float4*)__shfl_sync(0xffffffffu, (unsigned long long)tris, (int)o);
        if (g < total) {
            const uint32_t bit = __fns(om, 0u, (int)(g - oe) + 1);
            if (bit < 32u && ((om >> bit) & 1u)) {
                const float4* tp = otris + 3 * (size_t)(ob + bit);
                float4 a0 = ld_tri(tp + 0), a1 = ld_tri(tp + 1), a2 = ld_tri(tp + 2);
                if (INSTR) ++*ntri;
                float t, u, v;
                if (intersect_tri(ro, rd, ld3(a0), ld3(a1), ld3(a2), &t, &u, &v))
                    atomicMin(skey + o, hit_key(t, __float_as_uint(a0.w)));
            }
        }
    }
    __syncwarp();
    bool found = false;
    if (act) {
        const unsigned long long k = skey[lane];
        s.tg.y = 0u;
        if (k != mine) {
            const float t = __uint_as_float((uint32_t)(k >> 32));
            const uint32_t id = (uint32_t)k;
            s.best_t = t;
            s.best_id = id;
            found = true;
            if (!any) {
                const float4* sh = shade + 6 * (size_t)id;
                const v3 a = ld3(__ldg(sh + 0)), b = ld3(__ldg(sh + 1)), c = ld3(__ldg(sh + 2));
                float tt, u, v;
                if (intersect_tri(r.o, r.d, a, b - a, c - a, &tt, &u, &v)) { s.bb = u; s.bg = v; }
            }
        }
    }
    __syncwarp();
    return found;
}

// Persistent-warp ray loop of the traversal kernels: lanes whose ray has
// finished run `finish` together, idle lanes are refilled from the queue as
// soon as `refill` lanes are idle (all lanes once the queue is exhausted),
// and traversal resumes where each lane stopped.  The first wave is assigned
// by warp index (warp w takes entries [32w, 32w+32)); later fetches take one
// atomic per warp on `head`.  Each lane carries the geometry of its own
// scene.  fetch(q, &handle, ...) loads queue entry q's ray; bit 31 of the
// handle says any-hit; finish(handle, trav) gets it back when the ray is
// done.  A warp that makes kIterLimit steps without a refill gives up.
constexpr uint32_t kAnyHit = 0x80000000u;

// nodes0, tris0: the tree every lane starts with (fetch may change it).
template <bool INSTR, int MODE, int STACK, int BT, typename Fetch, typename Finish>
__device__ __forceinline__ void ray_loop(uint32_t count, uint32_t* head, int refill, uint32_t* status,
                                         const float4* nodes0, const float4* tris0, Fetch fetch, Finish finish,
                                         uint32_t* nvis, uint32_t* ntri) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const uint32_t dyn0 = nwarps * 32u;
    const uint32_t gwarp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    bool act = false, fin = false, exhausted = false, first = true;
    uint32_t hd = 0;  // the lane's handle for finish, as fetch sets it
    RayInv r;
    Trav s;
    trav_stop(s);
    uint2 stack[STACK];
    const float4* nodes = nodes0;
    const float4* tris = tris0;
    const float4* shade = nullptr;
    __shared__ unsigned long long s_key[MODE == 3 ? BT : 1];
    unsigned long long* skey = s_key + (MODE == 3 ? (threadIdx.x & ~31u) : 0u);
    while (true) {
        if (fin) finish(hd, s);
        fin = false;
        uint32_t idle = __ballot_sync(0xffffffffu, !act);
        if (!exhausted && idle) {
            uint32_t n = (uint32_t)__popc(idle);
            uint32_t base;
            if (first) {
                base = gwarp * 32u;
                first = false;
                if (dyn0 >= count) exhausted = true;
            } else {
                uint32_t leader = (uint32_t)__ffs(idle) - 1u;
                base = 0;
                if (lane == leader) base = atomicAdd(head, n);
                base = dyn0 + __shfl_sync(0xffffffffu, base, (int)leader);
                if (base + n >= count) exhausted = true;
            }
            if (!act) {
                uint32_t q = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                if (q < count) {
                    v3 o, d;
                    float tmax;
                    fetch(q, &hd, &o, &d, &tmax, &nodes, &tris, &shade);
                    r = make_ray(o, d);
                    trav_init(s, r, tmax);
                    act = true;
                }
            }
        }
        if (!__any_sync(0xffffffffu, act)) break;
        const bool any = (hd & kAnyHit) != 0u;
        int steps = 0;
        if (MODE == 0) {
            bool tri, node;
            while (true) {
                tri = has_tri(s);
                node = has_node(s);
                const uint32_t mt = __ballot_sync(0xffffffffu, tri), mn = __ballot_sync(0xffffffffu, node);
                const int live = __popc(mt | mn);
                if (live == 0 || (!exhausted && live <= 32 - refill)) break;
                if (++steps > kIterLimit) {
                    if (act) atomicOr(status, ST_ITER_LIMIT);
                    trav_stop(s);
                    continue;
                }
                warp_step<INSTR, STACK>(tri, node, mt, mn, nodes, tris, r, any, s, stack, status, nvis, ntri);
            }
            fin = act && !tri && !node;
            act = tri || node;
            continue;
        }
        while (true) {
            bool done = false;
            if (MODE == 3) {
                // the warp tests every lane's pending triangles together, then
                // each lane visits one node
                const bool hit = coop_triangles<INSTR>(act, tris, shade, r, any, s, skey, ntri);
                if (act) done = (any && hit) || node_step<INSTR, STACK>(nodes, r, s, stack, status, nvis);
            } else {
                // triangle postponing: when fewer than a fifth of the active
                // lanes have triangles pending, those lanes stack their
                // triangle group and keep traversing nodes with the rest of
                // the warp; otherwise they test one (MODE 1) or all (MODE 2)
                // of their pending triangles
                const bool want_tri = act && s.tg.y != 0u;
                const uint32_t mt = __ballot_sync(0xffffffffu, want_tri);
                const uint32_t ma = __ballot_sync(0xffffffffu, act);
                bool do_tri = want_tri;
                if (want_tri && 5u * (uint32_t)__popc(mt) < (uint32_t)__popc(ma) && s.sp < STACK) {
                    stack[s.sp++] = s.tg;
                    s.tg.y = 0u;
                    do_tri = false;
                }
                if (act) {
                    if (do_tri) {
                        if (MODE == 1) done = tri_step<INSTR>(tris, r, any, s, ntri);
                        else
                            while (s.tg.y != 0u && !done) done = tri_step<INSTR>(tris, r, any, s, ntri);
                    } else {
                        done = node_step<INSTR, STACK>(nodes, r, s, stack, status, nvis);
                    }
                }
            }
            if (++steps > kIterLimit) {
                if (act) atomicOr(status, ST_ITER_LIMIT);
                done = act;
            }
            if (done) { act = false; fin = true; }
            uint32_t nidle = (uint32_t)__popc(__ballot_sync(0xffffffffu, !act));
            if (nidle == 32u || (!exhausted && nidle >= (uint32_t)refill)) break;
        }
    }
}

// gb_trace_closest / gb_trace_any: the caller's rays through the persistent
// ray loop.  head: the queue head (zero), read only when there are more rays
// than lanes in the grid.  A negative or NaN max_t traces nothing.  Refilled at
// 4 / 8 / 12 / 16 / 20 idle lanes: 2 M shadow rays 342 / 306 / 297 / 298 / 307 us,
// 262 K closest hits 96 / 93 / 94 / 94 / 93.
constexpr int kTraceRefill = 12;
__global__ void __launch_bounds__(kBlock, GB_TRAV_MIN_BLOCKS) k_trace(DevScene S, uint32_t n,
                                                                      const float* __restrict__ orig,
                                                                      const float* __restrict__ dir,
                                                                      const float* __restrict__ tmaxv, float4* hits,
                                                                      uint8_t* occluded, int any, uint32_t* head,
                                                                      uint32_t* status) {
    fill_tables();
    uint32_t nvis = 0, ntri = 0;
    const uint32_t flag = any ? kAnyHit : 0u;
    auto fetch = [&](uint32_t q, uint32_t* handle, v3* o, v3* d, float* tmax, const float4** nodes,
                     const float4** tris, const float4** shade) {
        *handle = q | flag;
        const float *po = orig + 3 * (size_t)q, *pd = dir + 3 * (size_t)q;
        *o = mk(po[0], po[1], po[2]);
        *d = mk(pd[0], pd[1], pd[2]);
        const float t = tmaxv[q];
        *tmax = t >= 0.0f ? t : -1.0f;
    };
    auto finish = [&](uint32_t handle, const Trav& h) {
        const uint32_t i = handle & ~kAnyHit;
        const bool hit = h.best_id != 0xffffffffu;
        if (any) occluded[i] = hit ? 1 : 0;
        else hits[i] = make_float4(hit ? h.best_t : FLT_MAX, h.bb, h.bg, __uint_as_float(h.best_id));
    };
    ray_loop<false, 0, kStack, kBlock>(n, head, kTraceRefill, status, S.nodes, S.tris, fetch, finish, &nvis, &ntri);
}

// The same with every lane on its own: all pending triangles, then a node, with no
// vote.  A vote pays where other rays refill the lanes that have finished; a
// warp that gets no more rays only becomes as slow as its slowest lane at every
// step instead of at the end, and in a tree of a few levels there is little to
// vote on.  At most two waves of blocks, since each fills the tables (2 M rays, 3.8 K
// triangles: 95 against 108 us with a block per 128 rays).
__global__ void __launch_bounds__(kBlock, GB_TRAV_MIN_BLOCKS) k_trace_alone(DevScene S, uint32_t n,
                                                                            const float* __restrict__ orig,
                                                                            const float* __restrict__ dir,
                                                                            const float* __restrict__ tmaxv,
                                                                            float4* hits, uint8_t* occluded, int any,
                                                                            uint32_t* status) {
    fill_tables();
    uint32_t nvis = 0, ntri = 0;
    uint2 stack[kStack];
    for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
        const float *po = orig + 3 * (size_t)i, *pd = dir + 3 * (size_t)i;
        const RayInv r = make_ray(mk(po[0], po[1], po[2]), mk(pd[0], pd[1], pd[2]));
        const float t = tmaxv[i];
        Trav s;
        trav_init(s, r, t >= 0.0f ? t : -1.0f);
        for (int steps = 0;; ++steps) {
            bool done = false;
            while (s.tg.y != 0u && !done) done = tri_step<false>(S.tris, r, any != 0, s, &ntri);
            if (done) break;
            if (s.ng.y <= 0x00ffffffu) {
                if (s.sp == 0) break;
                s.ng = stack[--s.sp];
            }
            if (steps > kIterLimit) { atomicOr(status, (uint32_t)ST_ITER_LIMIT); break; }
            if (visit_node<false>(S.nodes, r, s, stack, status, &nvis, &s.tg, &s.tv)) break;
        }
        const bool hit = s.best_id != 0xffffffffu;
        if (any) occluded[i] = hit ? 1 : 0;
        else hits[i] = make_float4(hit ? s.best_t : FLT_MAX, s.bb, s.bg, __uint_as_float(s.best_id));
    }
}

// Whether the chunk's loop stops before iteration `it` and leaves its queues
// to k_finish: every path has started and few are alive.  k_rays decides and
// notes it in F.iter[2]: path_ctr moves while k_shade runs.
__device__ __forceinline__ bool left_to_finish(const Frame& F, const RenderParams& P, const uint32_t* cs) {
    return P.finish_max > 0 && *F.path_ctr >= P.chunk_paths &&
           cs[CTR_EXT] + cs[CTR_ENDED] <= (uint32_t)P.finish_max;
}

// The rays of one iteration: the closest hit of every extension ray (to
// F.hit), then whether anything blocks every shadow ray (to F.occl).  Block 0
// keeps the loop: it hands the iteration index to the kernels after it,
// clears the counter set after next (nobody reads it now), accounts the rays
// and paths of this iteration and tells the graph's loop (when there is one)
// to go on, so the loop ends with one iteration on empty queues.
// STACK: traversal stack entries; BT: threads per block (the register budget
// is that of GB_TRAV_MIN_BLOCKS blocks of 128 threads).
template <bool INSTR, int MODE, int STACK, int BT, bool MULTI>
__global__ void __launch_bounds__(BT, GB_TRAV_MIN_BLOCKS * 128 / BT) k_rays(Frame F, RenderParams P,
                                                                            unsigned long long cond, int has_cond) {
    const int it = F.iter[0];
    uint32_t* cs = ctr_set(F, it);
    const uint32_t next = cs[CTR_EXT], nsh = cs[CTR_SHADOW];
    const bool leave = left_to_finish(F, P, cs);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const uint32_t work = next | nsh | cs[CTR_ENDED], started = cs[CTR_STARTED];
        F.iter[1] = it;
        F.iter[2] = leave ? 1 : 0;
        uint32_t* c2 = ctr_set(F, it + 2);
        for (int k = 0; k < 8; ++k) c2[k] = 0u;
        F.stats[0] += started;
        F.stats[1] += next - started;
        F.stats[2] += nsh;
        if (leave) {
            if (has_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, 0u);
            return;
        }
        if (work) F.stats[7] += 1ull;
        if (work && it >= P.max_iters) atomicOr(F.status, (uint32_t)ST_ITER_LIMIT);
        if (has_cond) cudaGraphSetConditional((cudaGraphConditionalHandle)cond, work && it < P.max_iters ? 1u : 0u);
    }
    if (leave) return;
    fill_tables();
    const uint32_t *qe = F.q[it & 1], *qs = F.q[2];
    uint32_t nvis = 0, ntri = 0, nvis_any = 0, ntri_any = 0;
    auto fetch = [&](uint32_t q, uint32_t* handle, v3* o, v3* d, float* tmax, const float4** nodes,
                     const float4** tris, const float4** shade) {
        Sector r;
        uint32_t sc;
        if (q < next) {
            const uint32_t slot = qe[q];
            *handle = slot;
            r = rec_ld(&F.ray[slot]);
            *tmax = FLT_MAX;
            sc = MULTI ? scene_of(F, r.w[7]) : 0u;
        } else {
            const uint32_t slot = qs[q - next];
            *handle = slot | kAnyHit;
            r = rec_ld(&F.shray[slot]);
            *tmax = __uint_as_float(r.w[6]);
            sc = r.w[7];
        }
        if (MULTI) {
            const SceneRec& R = F.scenes[sc];
            *nodes = R.S.nodes;
            *tris = R.S.tris;
            *shade = R.S.shade;
        }
        *o = sec3(r, 0);
        *d = sec3(r, 3);
    };
    auto finish = [&](uint32_t handle, const Trav& h) {
        const uint32_t slot = handle & ~kAnyHit;
        if (handle & kAnyHit) F.occl[slot] = h.best_id != 0xffffffffu ? 1 : 0;
        else rec_st(&F.hit[slot], make_float4(h.bb, h.bg, __uint_as_float(h.best_id), 0.0f));
        if (INSTR) {
            if (handle & kAnyHit) { nvis_any += nvis; ntri_any += ntri; }
            else { atomicAdd(&F.stats[3], (unsigned long long)nvis); atomicAdd(&F.stats[4], (unsigned long long)ntri); }
            nvis = 0;
            ntri = 0;
        }
    };
    ray_loop<INSTR, MODE, STACK, BT>(next + nsh, cs + CTR_HEAD, P.refill, F.status, MULTI ? nullptr : P.nodes,
                                     MULTI ? nullptr : P.tris, fetch, finish, &nvis, &ntri);
    if (INSTR) {
        add_stats(&F.stats[5], nvis_any);
        add_stats(&F.stats[6], ntri_any);
    }
}

// Material record of index mi; the texture fields (last float4) only when
// the scene has textures.
__device__ __forceinline__ MaterialRec load_material(const float* mats, uint32_t mi, bool textured = false) {
    float mf[kMaterialFloats];
    const float4* mp = (const float4*)(mats + (size_t)kMaterialFloats * mi);
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        float4 q = __ldg(mp + k);
        mf[4 * k] = q.x; mf[4 * k + 1] = q.y; mf[4 * k + 2] = q.z; mf[4 * k + 3] = q.w;
    }
    float4 q = textured ? __ldg(mp + 7) : make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    mf[28] = q.x; mf[29] = q.y; mf[30] = q.z; mf[31] = q.w;
    return unpack_material(mf);
}

// Hit of a path in a textured scene: the ray differentials move to the hit
// (computeRayDiffs, hybrid-pt.cpp:518-519) and a diffuse texture scales the
// material's base colour.
__device__ __noinline__ void texture_hit(const SceneRec& R, uint32_t tid, float bb, float bg, v3 Nr, RayDiff* df,
                                         MaterialRec* m) {
    const float4* sh = R.S.shade + 6 * (size_t)tid;
    const v3 a = ld3(__ldg(sh)), b = ld3(__ldg(sh + 1)), c = ld3(__ldg(sh + 2));
    const float* tcs = R.S.texcoord + 6 * (size_t)tid;
    float ts, tt;
    bary2(bb, bg, tcs, &ts, &tt);
    const float diff = ray_diff_hit(df, a, b, c, tcs, ts, tt, normalize_div(Nr));
    if (m->dtex >= 0 && m->dtex < R.S.n_tex)
        *m = textured_material(*m, tex_sample_bilin_lod(R.S.tex[m->dtex], ts, tt, diff));
}

// The light sample of a hit (generate_arealight_sample,
// arealight-sampler-cpu.cpp:25-143) on the bounce's light draw.
struct LightSample {
    v3 so, sd, psc;      // shadow ray (to_light), potential_sample_contribution
    float smax, scale;   // max_t (negative: no light), geometry term over the pick probability
    int light;
};
__device__ __forceinline__ LightSample light_sample(const Frame& F, const SceneRec& R, uint32_t pix, v3 Pp, v3 Nr,
                                                    v3 rnd) {
    const DevScene& S = R.S;
    v3 lr = rnd;
    if (R.rng_mode == 1) {
        const float2 h = __ldg(&F.halton[pix]);
        lr = mk(h.x, h.y, h.y);
    }
    LightSample s;
    s.so = s.sd = s.psc = mk(0.0f, 0.0f, 0.0f);
    s.smax = -1.0f;
    s.scale = 0.0f;
    s.light = 0;
    if (S.n_lights > 0) {
        s.light = pick_light(S.lights, S.n_lights, S.overall_power, lr.z);
        LightRec L = S.lights[s.light];
        if (L.type == 1)
            sky_light_sample(S.sky, L.power, S.overall_power, Pp, Nr, lr.x, lr.y, R.sp.shadow_offset, &s.so, &s.sd,
                             &s.smax, &s.psc);
        else
            rect_light_sample(L, S.lights_eval[s.light].col, S.overall_power, Pp, Nr, lr.x, lr.y,
                              R.sp.shadow_offset, &s.so, &s.sd, &s.smax, &s.psc, &s.scale);
    }
    return s;
}

// Shading of every traced path (compute_path_contribution_and_bounce for the
// hits, handle_no_hit for the misses).  A block takes tiles of kShadeTile queue
// entries, sorts each into hits and paths that end here (misses, and ended
// paths whose last shadow ray has now been traced) and works on them in rounds
// of 32 of one kind, which warps take as they get to them, the hits' first (hits
// cost several times what ends do; every fourth round a warp instead: 35.3
// against 34.8 ms on the 1M-triangle 64-spp frame, 3.15 against 3.10 ms on 12
// mixed scenes, 684 against 664 us on a textured frame).  The outcome is gathered in
// lists in shared memory, which take their places in the global queues with
// one atomic per list.  A path that ends stores its sample and restarts on its
// slot with the chunk's next path; in MODE_ADJOINT it goes to the done queue
// instead, for k_adjoint and k_regen.
//
// What bounds it: latency of the scattered sector, triangle and material loads,
// of the ~1100 dependent instructions of a hit and of fetching them (the code is
// larger than the instruction cache), at 28 warps per SM.  Tiles of one entry per
// thread sorted by a block scan, and a warp on its own with tiles of 128, were
// slower by 3 to 6 % when rounds of one kind were introduced.  1M-triangle 64-spp frame
// / 1 spp / 256x256 room: tiles of 256 / 384 / 512 / 640 / 768 36.7 35.4 34.0
// 34.0 34.3 ms (room 856 849 831 834 846 us); 5 / 6 / 7 / 8 / 10 blocks per SM
// (96 / 80 / 72 / 64 / 48 registers) 34.7 34.1 34.0 34.2 35.4 ms, 917 896 890
// 900 925 us and 862 842 831 884 945 us, spills of 110 to 230 B at 7 among them.
// Fetching a tile's sectors to L2 ahead changes nothing, triangles as well slows
// small scenes by a quarter.
//
// A vertex's light sample adds bl * (tp * psc) to the accumulation if its
// shadow ray is free.  The contribution is formed here and kept pending; the
// next iteration's k_rays traces the ray and the next k_shade adds it before
// anything else, so the sums and their order are those of the reference.  No
// ray is traced for a contribution of exactly zero (the light or the surface
// faces away, no lobe towards the light): adding +-0 to an accumulation that
// is never -0 leaves its bits as they are.  The adjoint leaves out samples of
// scale zero only: a black light still has a gradient.
//
// MODE_FROZEN evaluates the BRDF with the scene's eval records and carries
// the sampling throughput in tp0; MODE_ADJOINT writes the vertex record of
// the path-replay adjoint and leaves pb's bounce field = the number of
// vertices the path shaded.
// What shading a hit needs beside the path's state.
struct Vertex {
    v3 P, N;          // hit point, interpolated (unnormalised) normal
    uint32_t mi;      // material
    MaterialRec m;
    LightSample ls;
    v3 rnd;           // the bounce's draw
};
// Loads a hit's triangle, draws the bounce's uniforms, takes its light sample
// and loads its material (df: the path's ray differentials, TEX only).
template <bool TEX>
__device__ __forceinline__ Vertex make_vertex(const Frame& F, const SceneRec& R, uint32_t pix, float bb, float bg,
                                              uint32_t id, MrgState& st, RayDiff* df) {
    Vertex v;
    v.rnd = draw3(&st);
    const float4* sh = R.S.shade + 6 * (size_t)id;
    const float4 a = __ldg(sh), b = __ldg(sh + 1), c = __ldg(sh + 2);
    v.P = bary(bb, bg, ld3(a), ld3(b), ld3(c));
    v.N = bary(bb, bg, ld3(__ldg(sh + 3)), ld3(__ldg(sh + 4)), ld3(__ldg(sh + 5)));
    v.ls = light_sample(F, R, pix, v.P, v.N, v.rnd);
    v.mi = __float_as_uint(a.w);
    const bool textured = TEX && R.S.texcoord != nullptr;
    v.m = load_material(R.S.mats, v.mi, textured);
    if (textured) texture_hit(R, id, bb, bg, v.N, df, &v.m);
    return v;
}

// A vertex record of the adjoint: two sectors (throughput, wo, pdf, roulette
// probability; wi, normal, light sample's scale, material) and 16 bytes (light
// direction, flags), each in a plane of its own per bounce.  Whole sectors
// take one 32 B access where five 16 B planes took a half-used sector each:
// gradient of a 509x511 16-spp frame 2.747 -> 2.706 ms.
__device__ __forceinline__ size_t adj_slots(const Frame& F) {  // even, so that every bounce's sectors are aligned
    return ((size_t)F.nslots + 1) & ~(size_t)1;
}
__device__ __forceinline__ Sector* adj_sector(const Frame& F, int bounce, uint32_t slot) {
    return reinterpret_cast<Sector*>(F.adj + (size_t)bounce * kAdjPlanes * adj_slots(F)) + slot;
}
__device__ __forceinline__ float4* adj_tail(const Frame& F, int bounce, uint32_t slot) {
    return F.adj + ((size_t)bounce * kAdjPlanes + 4) * adj_slots(F) + slot;
}

// Shared memory of a shading block: the tile's entries and what became of
// them.
constexpr uint32_t kShadeTile = 512;
enum { L_CONT = 0, L_SHADOW = 1, L_ENDED = 2, L_FIN = 3, L_HIT = 4, L_END = 5, L_ROUND = 6 };
struct ShadeTile {
    float4 entry[kShadeTile];  // beta, gamma, triangle id, slot: hits from the front, the others from the back
    uint32_t list[4][kShadeTile];
    uint32_t n[7];             // entries of the lists, hits, others; rounds taken
    uint32_t base[4];          // places taken in the global queues
};

// Tile of a launch with `count` entries: as few entries as give every block
// one tile (at least one per thread), or, where that is more than kShadeTile,
// each block's share in equal tiles, so that no wave of tiles is nearly empty
// (whole tiles of 512 instead: 256x256 16-spp room 866 against 838 us, textured
// frame 664 against 647; equal tiles in steps of 32 for single tiles as well:
// 12 mixed scenes 3.10 against 3.15 ms).
__device__ __forceinline__ uint32_t shade_tile(uint32_t count) {
    const uint32_t per = count / gridDim.x;
    if (count <= gridDim.x * kShadeTile) return min(max((per + 127u) & ~127u, (uint32_t)kBlock), kShadeTile);
    const uint32_t tiles = (per + kShadeTile) / kShadeTile;
    return min((per / tiles + 32u) & ~31u, kShadeTile);
}

// Appends `v` of the flagged lanes to a list of the block.
__device__ __forceinline__ void append(bool pred, uint32_t v, ShadeTile& T, int k) {
    const uint32_t m = __ballot_sync(0xffffffffu, pred);
    if (m == 0u) return;
    uint32_t b = 0;
    if (lane_id() == 0u) b = atomicAdd(&T.n[k], (uint32_t)__popc(m));
    b = __shfl_sync(0xffffffffu, b, 0);
    if (pred) T.list[k][b + (uint32_t)__popc(m & ((1u << lane_id()) - 1u))] = v;
}

template <int MODE, bool TEX>
__global__ void __launch_bounds__(kBlock, GB_SHADE_MIN_BLOCKS) k_shade(Frame F, RenderParams P) {
    __shared__ ShadeTile T;
    const int it = F.iter[1];
    const uint32_t *cs = ctr_set(F, it), *qe = F.q[it & 1], *qc = F.q[3 + (it & 1)];
    uint32_t *cn = ctr_set(F, it + 1), *qout = F.q[(it + 1) & 1], *qcout = F.q[3 + ((it + 1) & 1)];
    const uint32_t ne = cs[CTR_EXT], count = ne + cs[CTR_ENDED];
    const uint32_t tid = threadIdx.x, lane = lane_id(), lt = (1u << lane) - 1u;
    const uint32_t tile = shade_tile(count);
    if (F.iter[2]) return;  // the loop is over: k_finish takes the queues
    if (blockIdx.x == 0 && tid == 0) F.iter[0] = it + 1;
    for (uint32_t base = blockIdx.x * tile; base < count; base += gridDim.x * tile) {
        if (tid < 7) T.n[tid] = 0;
        __syncthreads();
        const uint32_t n = min(count - base, tile);
        for (uint32_t k = tid & ~31u; k < n; k += kBlock) {
            const uint32_t i = base + k + lane;
            const bool valid = k + lane < n;
            uint32_t slot = 0u;
            float4 hit = make_float4(0.0f, 0.0f, __uint_as_float(0xffffffffu), 0.0f);
            if (valid && i < ne) {
                slot = qe[i];
                hit = rec_ld(&F.hit[slot]);
            } else if (valid) {
                slot = qc[i - ne] | kAnyHit;  // marks an ended path
            }
            const bool ishit = __float_as_uint(hit.z) != 0xffffffffu;
            const uint32_t mh = __ballot_sync(0xffffffffu, ishit), md = __ballot_sync(0xffffffffu, valid && !ishit);
            uint32_t b = 0;
            if (lane < 2) b = atomicAdd(&T.n[L_HIT + lane], (uint32_t)__popc(lane ? md : mh));
            const uint32_t bh = __shfl_sync(0xffffffffu, b, 0), bd = __shfl_sync(0xffffffffu, b, 1);
            if (valid) {
                hit.w = __uint_as_float(slot);
                T.entry[ishit ? bh + (uint32_t)__popc(mh & lt) : n - 1u - bd - (uint32_t)__popc(md & lt)] = hit;
            }
        }
        __syncthreads();
        const uint32_t nh = T.n[L_HIT], rounds = ((nh + 31u) >> 5) + ((n - nh + 31u) >> 5);
        while (true) {  // warps take rounds as they get to them, the hits' first
            uint32_t round = 0;
            if (lane == 0) round = atomicAdd(&T.n[L_ROUND], 1u);
            round = __shfl_sync(0xffffffffu, round, 0);
            if (round >= rounds) break;
            const bool hits = round < ((nh + 31u) >> 5);  // this round shades hits
            const uint32_t e = (hits ? 0u : nh) + (round - (hits ? 0u : (nh + 31u) >> 5)) * 32u + lane;
            const bool valid = e < (hits ? nh : n);
            float4 hit = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (valid) hit = T.entry[e];
            uint32_t slot = __float_as_uint(hit.w);
            const bool dead = (slot & kAnyHit) != 0u;
            slot &= ~kAnyHit;

            bool cont = false, fin = false, shadow = false, ended = false;
            if (valid) {
                const Sector rs = rec_ld(&F.ray[slot]), ps = rec_ld(&F.path[slot]), ss = rec_ld(&F.strm[slot]);
                const uint32_t pbv = rs.w[6], pix = rs.w[7];
                const int bounce = (int)(pbv & 1023u);
                v3 acc = sec3(ps, 3);
                const v3 tp = sec3(ps, 0), rd = sec3(rs, 3);
                const bool occl = F.occl[slot] != 0;
                if (!occl)
                    acc = acc + mk(__uint_as_float(ps.w[6]), __uint_as_float(ps.w[7]), __uint_as_float(ss.w[6]));
                else if (MODE == MODE_ADJOINT && bounce > 0)  // the last vertex's light sample did not count
                    atomicAnd(reinterpret_cast<uint32_t*>(adj_tail(F, bounce - 1, slot)) + 3, ~(1u << 23));
                const uint32_t sc = scene_of(F, pix);
                const SceneRec& R = F.scenes[sc];
                if (hits) {
                    MrgState st{{ss.w[0], ss.w[1], ss.w[2]}, {ss.w[3], ss.w[4], ss.w[5]}};
                    RayDiff df;
                    const bool textured = TEX && R.S.texcoord != nullptr;
                    if (textured) df = ld_rdiff(F, slot);
                    const Vertex v = make_vertex<TEX>(F, R, pix, hit.x, hit.y, __float_as_uint(hit.z), st, &df);
                    if (textured) st_rdiff(F, slot, df);
                    const LightSample& ls = v.ls;
                    const uint32_t path = pbv >> 10, lp = pix - R.pixel_base;
                    ShadeOut o;
                    if (MODE == MODE_FROZEN) {
                        MaterialRec me = load_material(R.S.mats_eval, v.mi);
                        v3 t0 = ld3(F.tp0[slot]);
                        o = shade_hit(v.m, v.P, v.N, rd, tp, v.rnd, ls.smax >= 0.0f, ls.sd, ls.psc, R.sp, lp, path,
                                      bounce, &me, &t0);
                        F.tp0[slot] = make_float4(t0.x, t0.y, t0.z, 0.0f);
                    } else if (MODE == MODE_ADJOINT) {
                        ShadeTrace tr;
                        o = shade_hit(v.m, v.P, v.N, rd, tp, v.rnd, ls.smax >= 0.0f, ls.sd, ls.psc, R.sp, lp, path,
                                      bounce, nullptr, nullptr, &tr);
                        // a sample of scale zero adds nothing to the value or the gradient: it counts as blocked
                        shadow = tr.nee && ls.scale != 0.0f;
                        uint32_t info = (uint32_t)ls.light | ((uint32_t)tr.lobe << 16) | (tr.clamp_mask << 20) |
                                        (shadow ? (1u << 23) : 0u) | ((tr.flags & 7u) << 24);
                        Sector* rec = adj_sector(F, bounce, slot);
                        rec_st(rec, pack_sector(tp, tr.wo, __float_as_uint(tr.pdf), __float_as_uint(tr.q)));
                        rec_st(rec + adj_slots(F), pack_sector(tr.wi, tr.N, __float_as_uint(ls.scale), v.mi));
                        rec_st(adj_tail(F, bounce, slot), make_float4(tr.ld.x, tr.ld.y, tr.ld.z, __uint_as_float(info)));
                    } else {
                        o = shade_hit(v.m, v.P, v.N, rd, tp, v.rnd, ls.smax >= 0.0f, ls.sd, ls.psc, R.sp, lp, path,
                                      bounce);
                    }
                    const v3 pend = o.accum_add;
                    if (MODE != MODE_ADJOINT) shadow = pend.x != 0.0f || pend.y != 0.0f || pend.z != 0.0f;
                    if (shadow) rec_st(&F.shray[slot], pack_sector(ls.so, ls.sd, __float_as_uint(ls.smax), sc));
                    cont = o.alive && bounce + 1 < R.L;
                    if (cont) rec_st(&F.ray[slot], pack_sector(o.org, o.dir, pbv + 1u, pix));
                    else if (MODE == MODE_ADJOINT) F.ray[slot].w[6] = pbv + 1u;  // the path's vertices, for k_adjoint
                    ended = !cont && shadow;
                    fin = !cont && !shadow;
                    if (!fin) st_path(F, slot, o.tp, acc, st, pend);
                } else {
                    if (!dead) acc = acc + miss_contribution(tp, rd, R.sp, &R.S.sky);
                    fin = true;
                }
                if (fin) store_sample(F, P, pix, pbv, acc);
            }
            append(cont, slot, T, L_CONT);
            append(shadow, slot, T, L_SHADOW);
            append(ended, slot, T, L_ENDED);
            append(fin, slot, T, L_FIN);
        }
        __syncthreads();
        // places in the queues; finished paths take the chunk's next paths and
        // queue places after the continuing ones
        const uint32_t n_cont = T.n[L_CONT], n_shadow = T.n[L_SHADOW], n_ended = T.n[L_ENDED], n_fin = T.n[L_FIN];
        if (tid == 0) {
            uint32_t go = 0;
            if (MODE == MODE_ADJOINT) {
                if (n_fin) T.base[L_FIN] = atomicAdd(&cn[CTR_DONE], n_fin);
            } else if (n_fin) {
                const uint32_t l = atomicAdd(F.path_ctr, n_fin);
                T.base[L_FIN] = l;
                go = l < P.chunk_paths ? min(n_fin, P.chunk_paths - l) : 0u;
                if (go) atomicAdd(&cn[CTR_STARTED], go);
            }
            if (n_cont + go) T.base[L_CONT] = atomicAdd(&cn[CTR_EXT], n_cont + go);
        }
        if (tid == 32 && n_shadow) T.base[L_SHADOW] = atomicAdd(&cn[CTR_SHADOW], n_shadow);
        if (tid == 64 && n_ended) T.base[L_ENDED] = atomicAdd(&cn[CTR_ENDED], n_ended);
        if (tid == 96 && nh) atomicAdd(&F.stats[8], (unsigned long long)nh);
        __syncthreads();
        const uint32_t b0 = T.base[L_CONT], b1 = T.base[L_SHADOW], b2 = T.base[L_ENDED], b3 = T.base[L_FIN];
        for (uint32_t j = tid; j < n_cont; j += kBlock) qout[b0 + j] = T.list[L_CONT][j];
        for (uint32_t j = tid; j < n_shadow; j += kBlock) F.q[2][b1 + j] = T.list[L_SHADOW][j];
        for (uint32_t j = tid; j < n_ended; j += kBlock) qcout[b2 + j] = T.list[L_ENDED][j];
        for (uint32_t j = tid; j < n_fin; j += kBlock) {
            const uint32_t slot = T.list[L_FIN][j];
            if (MODE == MODE_ADJOINT) {
                F.q[5][b3 + j] = slot;
            } else if (b3 + j < P.chunk_paths) {
                start_path(F, P, slot, b3 + j);
                qout[b0 + n_cont + j] = slot;
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------- whole paths --
// Paths followed to their end by one thread each, with the operations of the
// slot-pool loop in the same order per path: k_paths takes a small chunk from
// the camera on, k_finish the paths a chunk has left when few are alive.
// After a vertex the warp traces the lanes' shadow rays and next extension
// rays together and meets again to shade: a lane goes on to its extension ray
// as soon as its shadow ray is done, or, in warps of at most 16 paths, leaves
// it to the lane 16 further on.
//
// A queue that does not fill the chip is bound by latency: each bounce costs
// the loop two launches, a tail of long rays and a round trip of the path
// state, whatever the work.  Wall time of a frame, the loop with k_finish for its
// last paths against k_paths (us, paths in thousands):
//   room      4K 122 / 102   48K 156 / 131   128K 232 / 225   196K 282 / 263   256K 320 / 341   512K 478 / 633
//   64 K tri  6K 169 / 150   48K 213 / 189   144K 301 / 258   192K 312 / 323   250K 327 / 351
//   512 K tri               48K 228 / 200   144K 335 / 364   192K 378 / 426   225K 390 / 478
// hence k_paths up to 3 * 2^16 paths: past the crossing of the largest trees, short
// of that of small ones.  The last paths of a chunk at 0 / 2^14 /
// 2^15 / 2^16 / 2^17 / 2^18 alive: 1 spp of the 1M-triangle frame 1090 / 935 /
// 938 / 887 / 965 / 966, textured sky 712 / 651 / 628 / 642 / 639 / 641, 12 mixed
// scenes 3160 / 3086 / 3088 / 3086 / 3086 / 3089: 2^16.
// 10 blocks of 64 per SM (96 registers, 270 to 310 B of spills) against as many
// registers as it likes: room 1K 102 / 99, 128K 225 / 212, 196K 263 / 280; 64 K
// triangles 48K 189 / 181, 192K 323 / 311; 512 K triangles 48K 200 / 227, 225K
// 387 / 376: neither is better everywhere.
constexpr int kPathsBlock = 64;
constexpr int kPathsMinBlocks = 10;
constexpr uint32_t kPathsWarps8 = 1216;
constexpr uint32_t kPathsWarps16 = 3040;
struct PathState {
    v3 o, d, tp, acc, pend;  // extension ray, throughput, accumulation, pending light sample
    v3 so, sd;               // shadow ray of the pending light sample
    float smax;
    bool ext, shadow;        // rays to trace
    int bounce;
    uint32_t path, pix;
    MrgState st;
};

__device__ __forceinline__ v3 shfl3(v3 v, uint32_t lane) {
    return mk(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane),
              __shfl_sync(0xffffffffu, v.z, lane));
}

// All 32 lanes call this; `alive` lanes have a path.  The sample goes to
// *sample.  helpers: paths are in lanes 0 .. 15 at most, and lane l + 16 traces
// the extension ray of lane l's path while lane l traces its shadow ray.
template <bool TEX>
__device__ __forceinline__ void follow_paths(const Frame& F, const SceneRec& R, bool alive, PathState& p, RayDiff& df,
                                             float4* sample, bool helpers) {
    uint32_t n_ext = 0, n_shadow = 0, n_hit = 0, nvis = 0, ntri = 0;
    uint2 stack[kStack];
    RayInv r;
    Trav s;
    // a helper traces in its path's scene, which need not be this lane's
    const float4 *nodes = R.S.nodes, *tris = R.S.tris;
    if (helpers) {
        nodes = (const float4*)__shfl_sync(0xffffffffu, (unsigned long long)nodes, lane_id() & 15u);
        tris = (const float4*)__shfl_sync(0xffffffffu, (unsigned long long)tris, lane_id() & 15u);
    }
    while (__any_sync(0xffffffffu, alive)) {
        bool any = alive && p.shadow, occl = false;
        bool ext = alive && p.ext;  // an extension ray this lane traces
        v3 eo = p.o, ed = p.d;
        if (helpers) {
            eo = shfl3(eo, lane_id() & 15u);
            ed = shfl3(ed, lane_id() & 15u);
            ext = __shfl_sync(0xffffffffu, (int)ext, lane_id() & 15u) != 0 && lane_id() >= 16u;
        }
        if (any || ext) {
            r = any ? make_ray(p.so, p.sd) : make_ray(eo, ed);
            trav_init(s, r, any ? p.smax : FLT_MAX);
        }
        else trav_stop(s);
        int steps = 0;
        while (true) {
            const bool tri = has_tri(s);
            bool node = has_node(s);
            if (any && !tri && !node) {  // the shadow ray is done
                occl = s.best_id != 0xffffffffu;
                any = false;
                if (ext) {
                    r = make_ray(eo, ed);
                    trav_init(s, r, FLT_MAX);
                    node = true;
                }
            }
            const uint32_t mt = __ballot_sync(0xffffffffu, tri), mn = __ballot_sync(0xffffffffu, node);
            if ((mt | mn) == 0u) break;
            if (++steps > kIterLimit) {
                if (tri || node) atomicOr(F.status, (uint32_t)ST_ITER_LIMIT);
                any = false;
                trav_stop(s);
                continue;
            }
            warp_step<false, kStack>(tri, node, mt, mn, nodes, tris, r, any, s, stack, F.status, &nvis, &ntri);
        }
        if (helpers) {
            s.best_id = __shfl_sync(0xffffffffu, s.best_id, lane_id() | 16u);
            s.bb = __shfl_sync(0xffffffffu, s.bb, lane_id() | 16u);
            s.bg = __shfl_sync(0xffffffffu, s.bg, lane_id() | 16u);
        }
        if (alive) {
            if (p.shadow && !occl) p.acc = p.acc + p.pend;
            p.shadow = false;
            bool end = true;
            if (p.ext && s.best_id != 0xffffffffu) {
                ++n_hit;
                const Vertex v = make_vertex<TEX>(F, R, p.pix, s.bb, s.bg, s.best_id, p.st, &df);
                const ShadeOut o = shade_hit(v.m, v.P, v.N, p.d, p.tp, v.rnd, v.ls.smax >= 0.0f, v.ls.sd, v.ls.psc,
                                             R.sp, p.pix - R.pixel_base, p.path, p.bounce);
                p.pend = o.accum_add;
                p.shadow = p.pend.x != 0.0f || p.pend.y != 0.0f || p.pend.z != 0.0f;
                p.so = v.ls.so;
                p.sd = v.ls.sd;
                p.smax = v.ls.smax;
                p.ext = o.alive && p.bounce + 1 < R.L;
                p.o = o.org;
                p.d = o.dir;
                p.tp = o.tp;
                ++p.bounce;
                n_ext += p.ext ? 1u : 0u;
                n_shadow += p.shadow ? 1u : 0u;
                end = !p.ext && !p.shadow;
            } else if (p.ext) {
                p.acc = p.acc + miss_contribution(p.tp, p.d, R.sp, &R.S.sky);
            }
            if (end) {
                rec_st(sample, make_float4(p.acc.x, p.acc.y, p.acc.z, 0.0f));
                alive = false;
                p.ext = false;
            }
        }
    }
    add_stats(&F.stats[1], n_ext);
    add_stats(&F.stats[2], n_shadow);
    add_stats(&F.stats[8], n_hit);
}

// Paths a warp follows when there are n: 16 while all their warps are resident
// together (10 blocks of 2 on 152 SMs), 8 up to two warps per scheduler, else
// 32.  The chip is then far from full whatever the split; fewer paths make
// fewer turns of the vote between nodes and triangles, fewer lobes one after
// the other, and leave lanes for the second ray.  32 always / this rule (us,
// paths in thousands): room 1K 115 / 102, 16K 117 / 106, 48K 129 / 131; 64 K
// triangles 6K 175 / 150, 48K 199 / 189; 512 K triangles 48K 224 / 200; last
// paths of 225K there 416 / 387.
__host__ __device__ __forceinline__ uint32_t paths_per_warp(uint32_t n) {
    return n <= 8u * kPathsWarps8 ? 8u : n <= 16u * kPathsWarps16 ? 16u : 32u;
}

template <bool TEX>
__global__ void __launch_bounds__(kPathsBlock, kPathsMinBlocks) k_paths(Frame F, RenderParams P, const MrgPowers J) {
    fill_tables();
    const uint32_t lanes = paths_per_warp(P.chunk_paths);
    const uint32_t l = (blockIdx.x * kPathsBlock + threadIdx.x) / 32u * lanes + lane_id();
    const bool alive = lane_id() < lanes && l < P.chunk_paths;
    const PathStart ps = path_start(F, P, alive ? l : 0u, &J);
    const SceneRec& R = F.scenes[ps.sc];
    const v3 z = mk(0.0f, 0.0f, 0.0f);
    PathState p{ps.o, ps.d, mk(1.0f, 1.0f, 1.0f), z, z, z, z, 0.0f, alive, false, 0, ps.path, ps.pix,
                ps.st};
    RayDiff df;
    if (TEX && R.S.texcoord) df = camera_diff(R.cam, ps.x, ps.y);
    add_stats(&F.stats[0], alive ? 1u : 0u);
    follow_paths<TEX>(F, R, alive, p, df, F.samples + (alive ? l : 0u), lanes <= 16u);
}

template <bool TEX>
__global__ void __launch_bounds__(kPathsBlock, kPathsMinBlocks) k_finish(Frame F, RenderParams P) {
    const int it = F.iter[0];
    const uint32_t* cs = ctr_set(F, it);
    const uint32_t ne = cs[CTR_EXT], count = ne + cs[CTR_ENDED];
    const uint32_t lanes = paths_per_warp(count);
    if (blockIdx.x * (kPathsBlock / 32) * lanes >= count) return;
    fill_tables();
    const uint32_t first = (blockIdx.x * kPathsBlock + threadIdx.x) / 32u * lanes, i = first + lane_id();
    if (first >= count) return;
    const bool alive = lane_id() < lanes && i < count;
    const uint32_t k = alive ? i : 0u;
    const uint32_t slot = k < ne ? F.q[it & 1][k] : F.q[3 + (it & 1)][k - ne];
    const Sector rs = rec_ld(&F.ray[slot]), ps = rec_ld(&F.path[slot]), ss = rec_ld(&F.strm[slot]);
    const SceneRec& R = F.scenes[scene_of(F, rs.w[7])];
    PathState p;
    p.o = sec3(rs, 0);
    p.d = sec3(rs, 3);
    p.tp = sec3(ps, 0);
    p.acc = sec3(ps, 3);
    p.pend = mk(__uint_as_float(ps.w[6]), __uint_as_float(ps.w[7]), __uint_as_float(ss.w[6]));
    p.ext = alive && k < ne;
    p.shadow = alive && (p.pend.x != 0.0f || p.pend.y != 0.0f || p.pend.z != 0.0f);
    p.bounce = (int)(rs.w[6] & 1023u);
    p.path = rs.w[6] >> 10;
    p.pix = rs.w[7];
    p.st = MrgState{{ss.w[0], ss.w[1], ss.w[2]}, {ss.w[3], ss.w[4], ss.w[5]}};
    if (p.shadow) {
        const Sector sh = rec_ld(&F.shray[slot]);
        p.so = sec3(sh, 0);
        p.sd = sec3(sh, 3);
        p.smax = __uint_as_float(sh.w[6]);
    }
    RayDiff df;
    if (TEX && R.S.texcoord) df = ld_rdiff(F, slot);
    follow_paths<TEX>(F, R, alive, p, df, F.samples + P.round_start[p.path - (uint32_t)P.p0] + p.pix, lanes <= 16u);
}

// Path-replay adjoint of every path that finished this iteration (done queue,
// before k_regen reuses the slots).  The path's value is
//   C = sum_k T_k * bl_k * col_l(k) * s_k,  T_{k+1} = clamp1(T_k * brdf_k / pdf_k) / q_k
// with pdf, q, the clamp pattern and all directions held at their recorded
// values; the reverse sweep k = K-1 .. 0 carries a = dLoss/dT_{k+1} and adds
// the BRDF vector-Jacobian products and the emission gradient to this
// block's gradient replica.  g = dLoss/dI(pixel) / spp.
// A copy per block keeps a float sum to the terms of one block (they are summed
// in double), whatever the number of parameters.  A fifth of the copies would
// cost less to clear and sum (8 scenes of 3.6 K floats: 3.71 against 3.75 ms a
// fitting step), but each sum would take five times as many terms: a step's
// gradient moved by 2e-7 with them, where two runs differ by 1e-8.  5 blocks per
// SM (96 registers; 104 and 4 blocks without the bound) for the same reason.
__global__ void __launch_bounds__(kBlock, 5) k_adjoint(Frame F, RenderParams P) {
    const uint32_t count = ctr_set(F, F.iter[1] + 1)[CTR_DONE];
    float* grad = F.grad + (size_t)(blockIdx.x % (uint32_t)F.grad_replicas) * (size_t)F.grad_stride;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t slot = F.q[5][i];
        const uint32_t pbv = F.ray[slot].w[6], pix = F.ray[slot].w[7];
        const int K = (int)(pbv & 1023u);
        const float4 g4 = F.dimg[pix];
        if (K == 0 || (g4.x == 0.0f && g4.y == 0.0f && g4.z == 0.0f)) continue;
        const SceneRec& R = F.scenes[scene_of(F, pix)];
        const v3 g = ld3(g4);
        float* gm_base = grad + R.grad_base;
        float* gl_base = gm_base + (size_t)kMatGradFloats * (size_t)R.n_mats;
        v3 an = mk(0.0f, 0.0f, 0.0f);  // dLoss / dT_{k+1}
        // sampling terms: gsuf = g . (light-sample terms of the vertices
        // after k); each vertex's scores are kept for the path's final miss
        // term, known once every light-sample term has been seen
        const bool st = P.sampling_terms != 0;
        float gsuf = 0.0f;
        uint32_t smi[kMaxAdjBounces];
        float ssm[kMaxAdjBounces], ssr[kMaxAdjBounces];
        int nsc = 0;
        for (int k = K - 1; k >= 0; --k) {
            const Sector r0 = rec_ld(adj_sector(F, k, slot)), r1 = rec_ld(adj_sector(F, k, slot) + adj_slots(F));
            const float4 r2 = rec_ld(adj_tail(F, k, slot));
            const v3 T = sec3(r0, 0), wo = sec3(r0, 3), wi = sec3(r1, 0), N = sec3(r1, 3), ld = ld3(r2);
            const float pdf = __uint_as_float(r0.w[6]), q = __uint_as_float(r0.w[7]), sc = __uint_as_float(r1.w[6]);
            const uint32_t mi = r1.w[7], info = __float_as_uint(r2.w);
            const int light = (int)(info & 0xffffu), lobe = (int)((info >> 16) & 15u);
            const uint32_t cmask = (info >> 20) & 7u;
            const bool nee = (info >> 23) & 1u;
            const uint32_t sflags = (info >> 24) & 7u;
            const MaterialRec m = load_material(R.S.mats, mi);
            MatGrad mg;
            matgrad_zero(&mg);
            v3 ak = mk(0.0f, 0.0f, 0.0f);
            float gw = 0.0f;  // dLoss / d log w of this vertex's Walter weight (through T_{k+1})
            if (an.x != 0.0f || an.y != 0.0f || an.z != 0.0f) {
                const v3 brdf = material_eval(m, lobe, wo, wi, N);
                const float inv = 1.0f / (pdf * q);
                const v3 c = mk((cmask & 1u) ? 0.0f : 1.0f, (cmask & 2u) ? 0.0f : 1.0f, (cmask & 4u) ? 0.0f : 1.0f);
                const v3 db = (c * T * an) * inv;  // dLoss / d brdf
                material_eval_vjp(m, lobe, wo, wi, N, db, &mg);
                ak = (c * brdf * an) * inv;
                gw = -dot(db, brdf);
            }
            float gnee = 0.0f;  // g . this vertex's light-sample term
            if (nee) {
                const v3 col = R.S.lights[light].col;
                const v3 psc = col * sc;
                const v3 bl = material_eval(m, lobe, wo, ld, N);
                material_eval_vjp(m, lobe, wo, ld, N, g * T * psc, &mg);
                const v3 acol = (g * T * bl) * sc;
                float* gl = gl_base + 3 * light;
                if (acol.x != 0.0f) atomicAdd(gl + 0, acol.x);
                if (acol.y != 0.0f) atomicAdd(gl + 1, acol.y);
                if (acol.z != 0.0f) atomicAdd(gl + 2, acol.z);
                ak = ak + g * bl * psc;
                gnee = dot(g, T * (bl * psc));
            }
            if (st) {
                // the branch decision moves this vertex's light-sample term
                // and everything after it; the sampled direction moves what
                // comes after this vertex; the Walter weight divides T_{k+1}
                float sm, sr, wr, zlo = 0.0f, zhi = 1.0f;
                if (R.rng_mode == 0 && R.S.n_lights > 0)
                    light_pick_interval(R.S.lights, R.S.n_lights, R.S.overall_power, light, &zlo, &zhi);
                sampling_scores(m, lobe, sflags, wo, wi, N, pdf, zlo, zhi, &sm, &sr, &wr);
                mg.metallic += sm * (gnee + gsuf);
                mg.roughness += sr * gsuf + gw * wr;
                if (sm != 0.0f || sr != 0.0f) {
                    smi[nsc] = mi;
                    ssm[nsc] = sm;
                    ssr[nsc] = sr;
                    ++nsc;
                }
            }
            gsuf += gnee;
            float* gmat = gm_base + (size_t)kMatGradFloats * mi;
            const float* mv = &mg.cdlin[0];
#pragma unroll
            for (int f = 0; f < kMatGradFloats; ++f)
                if (mv[f] != 0.0f) atomicAdd(gmat + f, mv[f]);
            an = ak;
        }
        if (st && nsc > 0) {
            // the path's final miss (the white background a throughput of
            // (1, 1, 1) adds, hybrid-pt.cpp:567-572): its sample minus the
            // light-sample terms; below rounding of the sum it is none
            const float4 sv = F.samples[P.round_start[(pbv >> 10) - (uint32_t)P.p0] + pix];
            const float gtot = dot(g, ld3(sv));
            const float gmiss = gtot - gsuf;
            if (fabsf(gmiss) > 1e-4f * fabsf(gtot)) {
                for (int i = 0; i < nsc; ++i) {
                    float* gmat = gm_base + (size_t)kMatGradFloats * smi[i];
                    if (ssm[i] != 0.0f) atomicAdd(gmat + offsetof(MatGrad, metallic) / sizeof(float), ssm[i] * gmiss);
                    if (ssr[i] != 0.0f) atomicAdd(gmat + offsetof(MatGrad, roughness) / sizeof(float), ssr[i] * gmiss);
                }
            }
        }
    }
}

// Direct lighting as the reference's gpu_area_lights integrator
// (direct-lighting.cpp:29-104, arealight-sampler.cu:156-260, :340-364), one
// pixel per thread: the pixel-centre camera ray's first hit gives the
// material colour (material_t::diffuse_color; the background for a miss,
// evaluate_material), then `samples` area-light samples of the GPU sampler
// (shadow offset as given, 0.01 there) are averaged: each adds psc * colour
// when its shadow ray is unoccluded.  Sample k uses pool update max(0, k-1)
// of the pixel's MRG32k3a stream, as the reference's update order gives
// (the pool advances after the second sample is set up).  A missed pixel's
// psc is the scaled sky texel of the direction its ray buffer holds: the
// camera ray's for the first sample, (0, 0, 0) afterwards.
//
// hybrid_area_lights (direct-lighting.cpp:203-316, direct-lighting.h:137-215):
// per pixel `cam_samples` jittered camera rays (jittered lens generator,
// jitter pool update c), the material colour of each camera hit
// (evaluate_material, material-cpu.cpp:20-80; footprint from the camera
// differentials), and `light_samples` samples of the CPU area-light sampler
// per camera sample (generate_arealight_sample, arealight-sampler-cpu.cpp:
// 25-143) folded into one moving average over sample c * L + j.  Sample j of
// a camera sample is set up before the pool's update of that step, so
// samples 0 and 1 share update c*L and sample j >= 2 takes c*L + j - 1; the
// L-th update of each camera sample goes unused.  All pools are seeded
// alike in the reference (curand_init(0, pixel, 0), util-kernels.cu:276-285),
// so the jitter and light draws are one stream read twice.
//
// Both (HYBRID: the second): a thread per pixel.  Light samples are taken
// kDirectGroup at a time: all their shadow rays are set up together, each lane
// traces its own one after the other while the warp steps together
// (warp_step), and the samples are then averaged in order, so that the warp
// waits for its slowest lane once a group and not once a ray.  A sample whose
// weight is exactly zero traces nothing (its term is zero either way while the
// colour is finite).  64 K triangles, 641x359 hybrid 2 x 8, the same 2 x 2,
// 384 K triangles 1280x720 with 16 samples, and 64 K 200x150 hybrid 2 x 8 (us with
// the image to the host):
//   groups of 4 / 8 / 16 at 14 blocks of 64 per SM   904 471 3192 497 / 893 469 3163 480 / 896 471 3150 483
//   of 8 at 10 / 12 / 16 blocks                      902 471 3198 446 / 893 469 3086 459 / 908 469 3193 493
// (14 blocks spill 290 to 430 B).  A ray at a time per thread: 641x359 1266 against
// 863, 200x150 631 against 480, 500x400 2 x 2 630 against 447.
// The loops over a group stay rolled: unrolled, the code leaves the
// instruction cache (1190 us).
constexpr int kDirectGroup = 8;
constexpr int kDirectBlock = 64;
constexpr int kDirectMinBlocks = 14;
template <bool HYBRID>
__global__ void __launch_bounds__(kDirectBlock, kDirectMinBlocks) k_direct(
    DevScene S, CameraRec cam, int w, int h, int cam_samples, int light_samples, uint32_t seed, float shadow_offset,
    v3 background, float* out, uint32_t* status, const MrgSubseqTable T) {
    fill_tables();
    const int g0 = blockIdx.x * kDirectBlock + threadIdx.x;
    const bool mine = g0 < w * h;
    const int g = mine ? g0 : 0;  // idle threads of the last block trace nothing
    const int px = g % w, py = g / w;
    MrgState js = mrg_stream(T, seed, (uint32_t)g), ls = js, lens = js;
    const bool aperture = HYBRID && cam.aperture != 0.0f;
    if (aperture) lens = mrg_stream(T, seed, (uint32_t)((g + 17) % (w * h)));
    const int L = light_samples;
    uint2 stack[kStack];
    Trav t;
    RayInv r;
    uint32_t nvis = 0, ntri = 0;
    v3 acc = mk(0.0f, 0.0f, 0.0f);
    for (int c = 0; c < cam_samples; ++c) {
        v3 o, d;
        if (HYBRID) {
            const v3 j = draw3(&js);
            float lx = 0.0f, ly = 0.0f;
            if (aperture) {
                const v3 lj = draw3(&lens);
                lx = lj.z - 0.5f;
                ly = lj.y - 0.5f;
            }
            camera_ray(cam, px, py, j.x, j.y, lx, ly, &o, &d);
        } else {
            camera_ray(cam, px, py, 0.5f, 0.5f, 0.0f, 0.0f, &o, &d);
        }
        r = make_ray(o, d);
        trav_init(t, r, FLT_MAX);
        if (!mine) trav_stop(t);
        for (int steps = 0;;) {
            const bool tri = has_tri(t), node = has_node(t);
            const uint32_t mt = __ballot_sync(0xffffffffu, tri), mn = __ballot_sync(0xffffffffu, node);
            if ((mt | mn) == 0u) break;
            if (++steps > kIterLimit) { atomicOr(status, (uint32_t)ST_ITER_LIMIT); trav_stop(t); continue; }
            warp_step<false, kStack>(tri, node, mt, mn, S.nodes, S.tris, r, false, t, stack, status, &nvis, &ntri);
        }
        const bool is_hit = mine && t.best_id != 0xffffffffu;
        v3 P = mk(0.0f, 0.0f, 0.0f), N = P, mcol = background;
        if (is_hit) {
            const float4* sh = S.shade + 6 * (size_t)t.best_id;
            const float4 a = sh[0];
            P = bary(t.bb, t.bg, ld3(a), ld3(sh[1]), ld3(sh[2]));
            N = bary(t.bb, t.bg, ld3(sh[3]), ld3(sh[4]), ld3(sh[5]));
            const float* mf = S.mats + (size_t)kMaterialFloats * __float_as_uint(a.w);
            mcol = mk(mf[25], mf[26], mf[27]);
            const int dtex = (int)mf[31];
            if (S.texcoord && dtex >= 0 && dtex < S.n_tex) {
                // pixel_evaluate_material_bilin_lod_cpu (material-cpu.cpp:36-77)
                const float* tcs = S.texcoord + 6 * (size_t)t.best_id;
                float ts, tt;
                bary2(t.bb, t.bg, tcs, &ts, &tt);
                RayDiff df = camera_diff(cam, px, py);
                const float diff = ray_diff_hit(&df, ld3(a), ld3(sh[1]), ld3(sh[2]), tcs, ts, tt, N);
                mcol = mcol * tex_sample_bilin_lod(S.tex[dtex], ts, tt, diff);
            }
        }
        const bool finite = isfinite(mcol.x) && isfinite(mcol.y) && isfinite(mcol.z);
        v3 buf_dir = d;
        v3 rnd = draw3(&ls);
        for (int k0 = 0; k0 < L; k0 += kDirectGroup) {
            const int n = min(kDirectGroup, L - k0);
            v3 so[kDirectGroup], sd[kDirectGroup], weight[kDirectGroup];
            float smax[kDirectGroup];
            uint32_t rays = 0, occluded = 0;  // by sample of the group
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
                if (k0 + i >= 2) rnd = draw3(&ls);
                weight[i] = mk(0.0f, 0.0f, 0.0f);
                if (is_hit && S.n_lights > 0) {
                    const int l = pick_light(S.lights, S.n_lights, S.overall_power, rnd.z);
                    const LightRec Lr = S.lights[l];
                    if (Lr.type == 1 && HYBRID)
                        sky_light_sample(S.sky, Lr.power, S.overall_power, P, N, rnd.x, rnd.y, shadow_offset, &so[i],
                                         &sd[i], &smax[i], &weight[i]);
                    else if (Lr.type == 1)
                        sky_light_sample_uniform(S.sky, Lr.power, S.overall_power, P, N, rnd.x, rnd.y, shadow_offset,
                                                 &so[i], &sd[i], &smax[i], &weight[i]);
                    else
                        rect_light_sample(Lr, Lr.col, S.overall_power, P, N, rnd.x, rnd.y, shadow_offset, &so[i],
                                          &sd[i], &smax[i], &weight[i], nullptr, HYBRID);
                    buf_dir = sd[i];
                    const bool zero = finite && weight[i].x == 0.0f && weight[i].y == 0.0f && weight[i].z == 0.0f;
                    if (smax[i] >= 0.0f && !zero) rays |= 1u << i;
                } else {
                    if (S.sky.light >= 0) weight[i] = S.sky.scale * sky_eval(S.sky, buf_dir);
                    buf_dir = mk(0.0f, 0.0f, 0.0f);
                }
            }
            int cur = -1;
            trav_stop(t);
            for (int steps = 0;;) {
                const bool tri = has_tri(t);
                bool node = has_node(t);
                if (!tri && !node) {  // the ray of sample `cur` is done: on to the lane's next one
                    if (cur >= 0 && t.best_id != 0xffffffffu) occluded |= 1u << cur;
                    cur = __ffs(rays) - 1;
                    if (cur >= 0) {
                        rays &= rays - 1u;
                        r = make_ray(so[cur], sd[cur]);
                        trav_init(t, r, smax[cur]);
                        node = true;
                    }
                }
                const uint32_t mt = __ballot_sync(0xffffffffu, tri), mn = __ballot_sync(0xffffffffu, node);
                if ((mt | mn) == 0u) break;
                if (++steps > kIterLimit) {
                    atomicOr(status, (uint32_t)ST_ITER_LIMIT);
                    trav_stop(t);
                    rays = 0;
                    continue;
                }
                warp_step<false, kStack>(tri, node, mt, mn, S.nodes, S.tris, r, true, t, stack, status, &nvis, &ntri);
            }
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
                const v3 mat = (occluded >> i) & 1u ? mk(0.0f, 0.0f, 0.0f) : mcol;
                const float s = float(c * L + k0 + i);
                acc = (s * acc + weight[i] * mat) / (s + 1.0f);
            }
        }
        if (HYBRID && L >= 2) draw3(&ls);
    }
    if (!mine) return;
    out[3 * g] = acc.x;
    out[3 * g + 1] = acc.y;
    out[3 * g + 2] = acc.z;
}

__global__ void k_dimg_pack(const float* __restrict__ src, int n, float scale, float4* dst) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    dst[i] = make_float4(src[3 * i] * scale, src[3 * i + 1] * scale, src[3 * i + 2] * scale, 0.0f);
}

// L2 image losses of a fitting step's scenes (blockIdx.y): loss = sum (x - t)^2
// over a scene's n pixels and the adjoint's image gradient dimg = 2 (x - t) *
// scale (scale = 1 / spp), the same float operations as k_dimg_pack applied to
// 2 (x - t); the image goes to the caller's buffer on the way.  Doubles are
// summed in a fixed order (thread, block, then k_loss_sum over the blocks), so
// the loss is the same every launch.  An SM does two double operations a
// clock, 12 of them per pixel: one block per scene took 0.2 ms for 65,536
// pixels, scene after scene.
__global__ void __launch_bounds__(kLossBlock) k_l2_loss(const FitLossItem* __restrict__ items,
                                                        const float4* __restrict__ img, float4* dimg, double* partial) {
    const FitLossItem it = items[blockIdx.y];
    __shared__ double part[kLossBlock];
    double acc = 0.0;
    for (int i = blockIdx.x * kLossBlock + threadIdx.x; i < it.n; i += gridDim.x * kLossBlock) {
        const float4 x = img[(size_t)it.base + i];
        const float c[3] = {x.x, x.y, x.z};
        float g[3];
        for (int k = 0; k < 3; ++k) {
            const float d = c[k] - it.target[3 * (size_t)i + k];
            acc += (double)d * (double)d;
            g[k] = (2.0f * d) * it.scale;
            if (it.image) it.image[3 * (size_t)i + k] = c[k];
        }
        dimg[(size_t)it.base + i] = make_float4(g[0], g[1], g[2], 0.0f);
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int s = kLossBlock / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = part[0];
}
__global__ void k_loss_sum(const double* __restrict__ partial, int blocks, int n, double* loss) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double acc = 0.0;
    for (int b = 0; b < blocks; ++b) acc += partial[(size_t)k * blocks + b];
    loss[k] = acc;
}

// Sum of the gradient replicas, in double: 32 elements per block, 16 threads
// per element take every 16th replica, their sums are added in order.  A thread
// per element alone: 75 us for 3.6 K elements of 760 replicas.
constexpr int kReduceRows = 16;
__global__ void __launch_bounds__(32 * kReduceRows) k_grad_reduce(const float* __restrict__ grad, int replicas,
                                                                  int stride, double* out) {
    __shared__ double part[kReduceRows][32];
    const int i = blockIdx.x * 32 + threadIdx.x;
    double acc = 0.0;
    if (i < stride)
        for (int r = threadIdx.y; r < replicas; r += kReduceRows)
            acc += (double)grad[(size_t)r * (size_t)stride + (size_t)i];
    part[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && i < stride) {
        for (int k = 1; k < kReduceRows; ++k) acc += part[k][threadIdx.x];
        out[i] = acc;
    }
}

// new_path's moving average (util-kernels.cu:17-25) over the chunk's paths
// p0 .. min(p0 + rounds, spp)-1 of every pixel, in path order.
__global__ void k_combine(Frame F, RenderParams P) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= F.ntot) return;
    const int p0 = P.p0;
    const int pe = min(p0 + P.rounds, F.scenes[F.pscene[g]].spp);
    if (p0 >= pe) return;
    v3 o = mk(0.0f, 0.0f, 0.0f);
    if (p0 > 0) { float4 c = F.out[g]; o = mk(c.x, c.y, c.z); }
    for (int p = p0; p < pe; ++p) {
        float4 s = F.samples[P.round_start[p - p0] + (uint32_t)g];
        o = combine_sample(o, mk(s.x, s.y, s.z), p);
    }
    F.out[g] = make_float4(o.x, o.y, o.z, 0.0f);
}

__global__ void k_pack_rgb(const float4* __restrict__ src, int n, float* dst) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = src[i];
    dst[3 * i] = v.x; dst[3 * i + 1] = v.y; dst[3 * i + 2] = v.z;
}

__global__ void k_mrg_pool(int pixel0, int npix, uint32_t seed, int first_update, int num_updates, float* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix) return;
    curandStateMRG32k3a s;
    curand_init((unsigned long long)seed, (unsigned long long)(uint32_t)(pixel0 + i), 0ull, &s);
    for (int u = 0; u < 3 * first_update; ++u) (void)curand_uniform(&s);
    for (int u = 0; u < num_updates; ++u) {
        size_t o = ((size_t)u * npix + i) * 3;
        for (int k = 0; k < 3; ++k) out[o + k] = curand_uniform(&s);
    }
}

// rta::generate_arealight_sample on a pixel grid (device buffers).
__global__ void k_nee_stage(DevScene S, int n, float shadow_offset, const float* __restrict__ rnd,
                            const float4* __restrict__ hits, float* ray_orig, float* ray_dir, float* max_t,
                            float* psc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 h = hits[i];
    uint32_t id = __float_as_uint(h.w);
    v3 r = mk(rnd[3 * i], rnd[3 * i + 1], rnd[3 * i + 2]);
    if (id != 0xffffffffu && S.n_lights > 0) {
        int l = pick_light(S.lights, S.n_lights, S.overall_power, r.z);
        const float4* sh = S.shade + 6 * (size_t)id;
        v3 Pp = bary(h.y, h.z, ld3(sh[0]), ld3(sh[1]), ld3(sh[2]));
        v3 Nr = bary(h.y, h.z, ld3(sh[3]), ld3(sh[4]), ld3(sh[5]));
        v3 so, sd, ps; float sm;
        if (S.lights[l].type == 1)
            sky_light_sample(S.sky, S.lights[l].power, S.overall_power, Pp, Nr, r.x, r.y, shadow_offset, &so, &sd,
                             &sm, &ps);
        else
            rect_light_sample(S.lights[l], S.lights[l].col, S.overall_power, Pp, Nr, r.x, r.y, shadow_offset, &so,
                              &sd, &sm, &ps);
        ray_orig[3 * i] = so.x; ray_orig[3 * i + 1] = so.y; ray_orig[3 * i + 2] = so.z;
        ray_dir[3 * i] = sd.x; ray_dir[3 * i + 1] = sd.y; ray_dir[3 * i + 2] = sd.z;
        max_t[i] = sm;
        psc[3 * i] = ps.x; psc[3 * i + 1] = ps.y; psc[3 * i + 2] = ps.z;
    } else {
        // arealight-sampler-cpu.cpp:121-142: the ray is killed and psc is the
        // (scaled) sky texel of the direction the buffer held, 0 without a sky
        v3 d = mk(ray_dir[3 * i], ray_dir[3 * i + 1], ray_dir[3 * i + 2]);
        v3 le = S.sky.light >= 0 ? S.sky.scale * sky_eval(S.sky, d) : mk(0.0f, 0.0f, 0.0f);
        ray_orig[3 * i] = FLT_MAX; ray_orig[3 * i + 1] = FLT_MAX; ray_orig[3 * i + 2] = FLT_MAX;
        ray_dir[3 * i] = 0.0f; ray_dir[3 * i + 1] = 0.0f; ray_dir[3 * i + 2] = 0.0f;
        max_t[i] = -1.0f;
        psc[3 * i] = le.x; psc[3 * i + 1] = le.y; psc[3 * i + 2] = le.z;
    }
}

// compute_path_contribution_and_bounce on a pixel grid (device buffers).
__global__ void k_shade_stage(DevScene S, int n, ShadeParams sp, float* ray_orig, float* ray_dir, float* max_t,
                              const float4* __restrict__ hits, const uint8_t* __restrict__ occl,
                              const float* __restrict__ rnd, float* tp, float* accum,
                              const float* __restrict__ to_light, const float* __restrict__ psc, int path,
                              int bounce) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 h = hits[i];
    uint32_t id = __float_as_uint(h.w);
    v3 t = mk(tp[3 * i], tp[3 * i + 1], tp[3 * i + 2]);
    v3 ac = mk(accum[3 * i], accum[3 * i + 1], accum[3 * i + 2]);
    if (id != 0xffffffffu) {
        const float4* sh = S.shade + 6 * (size_t)id;
        float4 a = sh[0];
        v3 Pp = bary(h.y, h.z, ld3(a), ld3(sh[1]), ld3(sh[2]));
        v3 Nr = bary(h.y, h.z, ld3(sh[3]), ld3(sh[4]), ld3(sh[5]));
        MaterialRec m = unpack_material(S.mats + (size_t)kMaterialFloats * __float_as_uint(a.w));
        v3 rd = mk(ray_dir[3 * i], ray_dir[3 * i + 1], ray_dir[3 * i + 2]);
        ShadeOut o = shade_hit(m, Pp, Nr, rd, t, mk(rnd[3 * i], rnd[3 * i + 1], rnd[3 * i + 2]), occl[i] == 0,
                               mk(to_light[3 * i], to_light[3 * i + 1], to_light[3 * i + 2]),
                               mk(psc[3 * i], psc[3 * i + 1], psc[3 * i + 2]), sp, (uint32_t)i, (uint32_t)path,
                               bounce);
        ac = ac + o.accum_add;
        t = o.tp;
        if (o.alive) {
            ray_orig[3 * i] = o.org.x; ray_orig[3 * i + 1] = o.org.y; ray_orig[3 * i + 2] = o.org.z;
            ray_dir[3 * i] = o.dir.x; ray_dir[3 * i + 1] = o.dir.y; ray_dir[3 * i + 2] = o.dir.z;
            max_t[i] = FLT_MAX;
        } else {
            ray_orig[3 * i] = FLT_MAX; ray_orig[3 * i + 1] = FLT_MAX; ray_orig[3 * i + 2] = FLT_MAX;
            ray_dir[3 * i] = 0.0f; ray_dir[3 * i + 1] = 0.0f; ray_dir[3 * i + 2] = 0.0f;
            max_t[i] = -1.0f;
        }
    } else {
        // handle_no_hit (hybrid-pt.cpp:196-206); dead rays (max_t == -1) add 0
        if (max_t[i] != -1.0f)
            ac = ac + miss_contribution(t, mk(ray_dir[3 * i], ray_dir[3 * i + 1], ray_dir[3 * i + 2]), sp, &S.sky);
        ray_orig[3 * i] = FLT_MAX; ray_orig[3 * i + 1] = FLT_MAX; ray_orig[3 * i + 2] = FLT_MAX;
        ray_dir[3 * i] = 0.0f; ray_dir[3 * i + 1] = 0.0f; ray_dir[3 * i + 2] = 0.0f;
        max_t[i] = -1.0f;
        t = mk(0.0f, 0.0f, 0.0f);
    }
    tp[3 * i] = t.x; tp[3 * i + 1] = t.y; tp[3 * i + 2] = t.z;
    accum[3 * i] = ac.x; accum[3 * i + 1] = ac.y; accum[3 * i + 2] = ac.z;
}

inline int blocks_for(int n) { return (n + kBlock - 1) / kBlock; }

// SMs and resident blocks per SM of a persistent kernel.
struct Grid {
    int sms, per;
};

template <typename K>
Grid persistent_grid(K kernel, int block = kBlock) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, block, 0);
    if (sms < 1) sms = 1;
    if (per < 1) per = 1;
    return Grid{sms, per};
}

template <typename K>
int persistent_blocks(K kernel) {
    Grid g = persistent_grid(kernel);
    return g.sms * g.per;
}

// Grid of a persistent traversal kernel: every SM holds min(occupancy
// limit, blocks_per_sm) blocks (all it can hold when blocks_per_sm is 0);
// blocks_per_sm counts 128-thread blocks, so blocks of bt threads scale it.
inline int traversal_grid(const Grid& g, int blocks_per_sm, int bt = kBlock) {
    const int want = blocks_per_sm > 0 ? std::max(1, blocks_per_sm * kBlock / bt) : g.per;
    return g.sms * std::min(g.per, want);
}

}  // namespace

// Whether n rays go through k_trace_alone instead of k_trace, whose grid has
// `lanes` lanes (136 K on 152 SMs).  k_trace / k_trace_alone, us a call, warm and
// after a flush of the L2:
//   no more rays than lanes   1 M triangles, 16 K and 131 K shadow rays 52 57 / 44 55, 74 79 / 68 68, closest 59 71 /
//                             57 71, 84 92 / 80 90; 64 K triangles, 131 K closest 60 58 / 55 57
//   up to two rays a lane     13 K triangles, 262 K closest 62 58 / 57 53, any 61 58 / 56 53; 23 K any 57 55 / 49 53;
//                             but 64 K, 262 K any 63 60 / 63 64, 13 K, 400 K closest 64 62 / 69 65
//   more                      1.3 K triangles, 2 M closest 101 98 / 83 80; 3.8 K closest 110 105 / 96 98; 2.6 K, 450 K
//                             any 59 55 / 50 52; but 5.1 K, 2 M closest 112 108 / 122 126, 3.8 K any 123 119 / 169 176
inline bool trace_alone(int n, int lanes, int tris, bool any) {
    if (n <= lanes) return true;
    if (n <= 2ll * lanes) return tris <= 3 << 13;
    return tris <= (any ? 2560 : 4096);
}

cudaError_t k_launch_trace(const DevScene& S, int n, const float* orig, const float* dir, const float* tmax,
                           float4* hits, uint8_t* occluded, bool any, uint32_t* head, uint32_t* status,
                           cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    static int g = persistent_blocks(k_trace);
    if (trace_alone(n, g * kBlock, S.n_tris, any)) {
        static int ga = persistent_blocks(k_trace_alone);
        k_trace_alone<<<std::min(2 * ga, blocks_for(n)), kBlock, 0, st>>>(S, (uint32_t)n, orig, dir, tmax, hits, occluded,
                                                                          any ? 1 : 0, status);
        return cudaGetLastError();
    }
    if (n > g * kBlock) {
        cudaError_t e = cudaMemsetAsync(head, 0, sizeof(uint32_t), st);
        if (e != cudaSuccess) return e;
    }
    k_trace<<<std::min(g, blocks_for(n)), kBlock, 0, st>>>(S, (uint32_t)n, orig, dir, tmax, hits, occluded,
                                                           any ? 1 : 0, head, status);
    return cudaGetLastError();
}

// The subsequence jumps, computed once per process.
const MrgSubseqTable& subseq_table() {
    static const MrgSubseqTable T = [] {
        MrgSubseqTable t;
        mrg_subsequence_table(&t);
        return t;
    }();
    return T;
}

cudaError_t k_launch_frame_init(const Frame& F, bool rng, cudaStream_t st) {
    k_fill_pscene<<<blocks_for(F.ntot), kBlock, 0, st>>>(F);
    if (rng) k_rng_init_frame<<<blocks_for(F.ntot), kBlock, 0, st>>>(F, subseq_table());
    return cudaGetLastError();
}

// Jumps by the three draws of a camera-jitter update, computed once per process.
const MrgPowers& jitter_powers() {
    static const MrgPowers T = [] {
        MrgPowers t;
        mrg_powers(3, &t);
        return t;
    }();
    return T;
}

constexpr int kStartThreads = 1 << 17;
cudaError_t k_launch_start(const Frame& F, const RenderParams& P, int nstart, cudaStream_t st) {
    // enough threads to fill the chip, at most 8 paths each (12 mixed scenes 3.43 ms with the pool for every path,
    // 3.52 with a thread per path, 3.25 so; 256x256 room 0.935 / 0.921 / 0.907); rounds beyond the first nstart
    // paths have no blocks
    const int group = std::min(8, std::max(1, nstart / kStartThreads));
    int rounds = 1;
    while (rounds < P.rounds && P.round_start[rounds] < (uint32_t)nstart) ++rounds;
    const dim3 grid((unsigned)blocks_for(F.ntot), (unsigned)((rounds + group - 1) / group));
    k_start<<<grid, kBlock, 0, st>>>(F, P, nstart, group, jitter_powers());
    return cudaGetLastError();
}

// Launch of a traversal kernel; with an L2 window in P (the scene's node
// array) the launch carries it as an access-policy attribute: node lines
// persist in the L2 set-aside, so that the per-iteration state streaming
// past does not evict them.
template <typename K, typename... Args>
void launch_traversal(K kernel, dim3 grid, int block, const RenderParams& P, cudaStream_t st, Args... args) {
    if (P.l2_nodes_bytes == 0) {
        kernel<<<grid, block, 0, st>>>(args...);
        return;
    }
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeAccessPolicyWindow;
    at[0].val.accessPolicyWindow.base_ptr = const_cast<void*>(P.l2_nodes);
    at[0].val.accessPolicyWindow.num_bytes = (size_t)P.l2_nodes_bytes;
    at[0].val.accessPolicyWindow.hitRatio = P.l2_hit_ratio;
    at[0].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    at[0].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <bool INSTR, int MODE, int STACK, int BT, bool MULTI>
void launch_rays_v(const Frame& F, const RenderParams& P, unsigned long long cond, bool has_cond, cudaStream_t st) {
    static Grid g = persistent_grid(k_rays<INSTR, MODE, STACK, BT, MULTI>, BT);
    launch_traversal(k_rays<INSTR, MODE, STACK, BT, MULTI>, traversal_grid(g, P.blocks_per_sm, BT), BT, P, st, F, P, cond,
                     has_cond ? 1 : 0);
}

// The default triangle policy has variants for two stack depths and two
// block shapes (RenderParams::trav_variant) and for frames of one scene, whose
// tree is a kernel parameter (four registers less); the other policies have
// one each.
template <bool INSTR, bool MULTI>
void launch_rays_0(const Frame& F, const RenderParams& P, unsigned long long c, bool h, cudaStream_t st) {
    if (P.trav_variant == 1) launch_rays_v<INSTR, 0, 24, 128, MULTI>(F, P, c, h, st);
    else if (P.trav_variant == 2) launch_rays_v<INSTR, 0, 32, 64, MULTI>(F, P, c, h, st);
    else if (P.trav_variant == 3) launch_rays_v<INSTR, 0, 24, 64, MULTI>(F, P, c, h, st);
    else launch_rays_v<INSTR, 0, kStack, kBlock, MULTI>(F, P, c, h, st);
}
template <bool INSTR, int MODE>
void launch_rays_t(const Frame& F, const RenderParams& P, unsigned long long c, bool h, cudaStream_t st) {
    if constexpr (MODE != 0) launch_rays_v<INSTR, MODE, kStack, kBlock, true>(F, P, c, h, st);
    else if (P.nodes) launch_rays_0<INSTR, false>(F, P, c, h, st);
    else launch_rays_0<INSTR, true>(F, P, c, h, st);
}

cudaError_t k_launch_rays(const Frame& F, const RenderParams& P, bool instrument, unsigned long long c, bool h,
                          cudaStream_t st) {
    switch (P.tri_mode * 2 + (instrument ? 1 : 0)) {
        case 0: launch_rays_t<false, 0>(F, P, c, h, st); break;
        case 1: launch_rays_t<true, 0>(F, P, c, h, st); break;
        case 2: launch_rays_t<false, 1>(F, P, c, h, st); break;
        case 3: launch_rays_t<true, 1>(F, P, c, h, st); break;
        case 4: launch_rays_t<false, 2>(F, P, c, h, st); break;
        case 5: launch_rays_t<true, 2>(F, P, c, h, st); break;
        case 6: launch_rays_t<false, 3>(F, P, c, h, st); break;
        default: launch_rays_t<true, 3>(F, P, c, h, st); break;
    }
    return cudaGetLastError();
}

// Grid of the streaming per-path kernels (k_shade, k_regen): persistent for
// pools of up to 2^20 slots, one thread per four slots above that, with a loop
// over what is left.  A block per 512 slots gives a full queue's blocks
// one whole tile each; a thread per slot makes the tiles of 128, fewer blocks
// leave a long last wave.  nslots / 1 / 4 / 16 / 64 threads: 1M-triangle 64-spp
// frame 37.2 / 34.0 / 34.8 / 34.7 ms, 12 mixed scenes 3.49 / 3.08 / 3.19 /
// 3.42 ms.
#ifndef GB_WIDE_GRID_DIV
#define GB_WIDE_GRID_DIV 4  // the wide grid has nslots / GB_WIDE_GRID_DIV threads
#endif
inline int stream_grid(int persistent, int nslots) {
    return nslots > (1 << 20) ? std::max(1, blocks_for(nslots / GB_WIDE_GRID_DIV)) : persistent;
}

template <int MODE, bool TEX>
void launch_shade_t(const Frame& F, const RenderParams& P, cudaStream_t st) {
    static int g = persistent_blocks(k_shade<MODE, TEX>);
    k_shade<MODE, TEX><<<stream_grid(g, F.nslots), kBlock, 0, st>>>(F, P);
}

// The texture path is compiled into its own variant so that frames without
// textures run the kernel without it; replay and adjoint frames have none.
cudaError_t k_launch_shade(const Frame& F, const RenderParams& P, cudaStream_t st) {
    if (P.mode == MODE_FROZEN) launch_shade_t<MODE_FROZEN, false>(F, P, st);
    else if (P.mode == MODE_ADJOINT) launch_shade_t<MODE_ADJOINT, false>(F, P, st);
    else if (P.textured) launch_shade_t<MODE_FORWARD, true>(F, P, st);
    else launch_shade_t<MODE_FORWARD, false>(F, P, st);
    return cudaGetLastError();
}

// The adjoint's blocks, each with a gradient copy of its own.
int k_adjoint_grid() {
    static int g = persistent_blocks(k_adjoint);
    return g;
}

cudaError_t k_launch_adjoint(const Frame& F, const RenderParams& P, cudaStream_t st) {
    k_adjoint<<<k_adjoint_grid(), kBlock, 0, st>>>(F, P);
    return cudaGetLastError();
}

cudaError_t k_launch_direct(const DevScene& S, const CameraRec& cam, int w, int h, int samples, uint32_t seed,
                            float shadow_offset, v3 background, float* out, uint32_t* status, cudaStream_t st) {
    if (w * h <= 0) return cudaSuccess;
    k_direct<false><<<(w * h + kDirectBlock - 1) / kDirectBlock, kDirectBlock, 0, st>>>(
        S, cam, w, h, 1, samples, seed, shadow_offset, background, out, status, subseq_table());
    return cudaGetLastError();
}

cudaError_t k_launch_direct_hybrid(const DevScene& S, const CameraRec& cam, int w, int h, int cam_samples,
                                   int light_samples, uint32_t seed, float shadow_offset, v3 background, float* out,
                                   uint32_t* status, cudaStream_t st) {
    if (w * h <= 0) return cudaSuccess;
    k_direct<true><<<(w * h + kDirectBlock - 1) / kDirectBlock, kDirectBlock, 0, st>>>(
        S, cam, w, h, cam_samples, light_samples, seed, shadow_offset, background, out, status, subseq_table());
    return cudaGetLastError();
}

cudaError_t k_launch_dimg_pack(const float* src, int n, float scale, float4* dst, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_dimg_pack<<<blocks_for(n), kBlock, 0, st>>>(src, n, scale, dst);
    return cudaGetLastError();
}

cudaError_t k_launch_l2_loss(const FitLossItem* items, int n, const float4* img, float4* dimg, double* partial,
                             double* loss, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_l2_loss<<<dim3(kLossBlocks, (unsigned)n), kLossBlock, 0, st>>>(items, img, dimg, partial);
    k_loss_sum<<<(n + 31) / 32, 32, 0, st>>>(partial, kLossBlocks, n, loss);
    return cudaGetLastError();
}

cudaError_t k_launch_grad_reduce(const float* grad, int replicas, int stride, double* out, cudaStream_t st) {
    if (stride <= 0) return cudaSuccess;
    k_grad_reduce<<<(stride + 31) / 32, dim3(32, kReduceRows), 0, st>>>(grad, replicas, stride, out);
    return cudaGetLastError();
}

int k_launches_per_iteration(int mode) {
    return mode == MODE_ADJOINT ? 4 : 2;  // rays, shade; adjoint, regen
}

cudaError_t k_launch_regen(const Frame& F, const RenderParams& P, cudaStream_t st) {
    if (P.mode != MODE_ADJOINT) return cudaSuccess;  // paths restart in k_shade
    static int g0 = persistent_blocks(k_regen);
    k_regen<<<stream_grid(g0, F.nslots), kBlock, 0, st>>>(F, P);
    return cudaGetLastError();
}

cudaError_t k_launch_paths(const Frame& F, const RenderParams& P, cudaStream_t st) {
    const unsigned per_block = kPathsBlock / 32 * paths_per_warp(P.chunk_paths);
    const unsigned grid = (P.chunk_paths + per_block - 1) / per_block;
    if (P.textured) k_paths<true><<<grid, kPathsBlock, 0, st>>>(F, P, jitter_powers());
    else k_paths<false><<<grid, kPathsBlock, 0, st>>>(F, P, jitter_powers());
    return cudaGetLastError();
}

cudaError_t k_launch_finish(const Frame& F, const RenderParams& P, cudaStream_t st) {
    if (P.finish_max <= 0) return cudaSuccess;
    // the blocks of the most paths and, for fewer at 8 or 16 a warp, of at most kPathsWarps16 warps
    const unsigned most = (unsigned)std::min(P.finish_max, F.nslots), per_block = kPathsBlock / 32;
    const unsigned warps = std::max((most + 31) / 32, std::min((most + 7) / 8, std::max(kPathsWarps16, kPathsWarps8)));
    const unsigned grid = (warps + per_block - 1) / per_block;
    if (P.textured) k_finish<true><<<grid, kPathsBlock, 0, st>>>(F, P);
    else k_finish<false><<<grid, kPathsBlock, 0, st>>>(F, P);
    return cudaGetLastError();
}

// After k_start / k_paths, which start from the cursors this moves on.
cudaError_t k_launch_jitter_pool(const Frame& F, const RenderParams& P, cudaStream_t st) {
    if (P.pool_round >= P.rounds && !P.more) return cudaSuccess;
    k_jitter_pool<<<blocks_for(F.ntot), kBlock, 0, st>>>(F, P, jitter_powers());
    return cudaGetLastError();
}

cudaError_t k_launch_combine(const Frame& F, const RenderParams& P, cudaStream_t st) {
    k_combine<<<blocks_for(F.ntot), kBlock, 0, st>>>(F, P);
    return cudaGetLastError();
}

cudaError_t k_launch_pack_rgb(const float4* src, int n, float* dst, cudaStream_t st) {
    k_pack_rgb<<<blocks_for(n), kBlock, 0, st>>>(src, n, dst);
    return cudaGetLastError();
}

cudaError_t k_launch_mrg_states(uint32_t seed, const uint32_t* sub, int n, int method, uint32_t* out,
                                cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_mrg_states<<<blocks_for(n), kBlock, 0, st>>>(subseq_table(), seed, sub, n, method, out);
    return cudaGetLastError();
}

cudaError_t k_launch_mrg_pool(int pixel0, int npix, uint32_t seed, int first_update, int num_updates, float* out,
                              cudaStream_t st) {
    k_mrg_pool<<<blocks_for(npix), kBlock, 0, st>>>(pixel0, npix, seed, first_update, num_updates, out);
    return cudaGetLastError();
}

cudaError_t k_launch_nee_stage(const DevScene& S, int n, float shadow_offset, const float* rnd, const float4* hits,
                               float* ray_orig, float* ray_dir, float* max_t, float* psc, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_nee_stage<<<blocks_for(n), kBlock, 0, st>>>(S, n, shadow_offset, rnd, hits, ray_orig, ray_dir, max_t, psc);
    return cudaGetLastError();
}

cudaError_t k_launch_shade_stage(const DevScene& S, int n, const ShadeParams& sp, float* ray_orig, float* ray_dir,
                                 float* max_t, const float4* hits, const uint8_t* occl, const float* rnd,
                                 float* tp, float* accum, const float* to_light, const float* psc, int path,
                                 int bounce, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_shade_stage<<<blocks_for(n), kBlock, 0, st>>>(S, n, sp, ray_orig, ray_dir, max_t, hits, occl, rnd, tp, accum,
                                                    to_light, psc, path, bounce);
    return cudaGetLastError();
}

}  // namespace gb
