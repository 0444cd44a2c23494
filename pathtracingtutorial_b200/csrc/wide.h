// wide.h -- four-wide tree with 8-bit boxes, collapsed from the binary tree on
// the device at upload, and its closest-hit and any-hit walks (device only).
//
// Results are those of the binary walk (traverse.h) bit for bit.  The binary
// walk tests a leaf exactly when the leaf's box passes the exact box test
// against the best distance at the time the depth-first order reaches it:
//   * a child box lies inside its parent's, and every step of the box test is
//     monotone in the box planes, so a leaf that passes has ancestors that
//     passed (at their earlier time the best distance was no smaller);
//   * so any inner test that never rejects a node with a passing leaf below
//     it, taken in the same depth-first order, reaches a superset of those
//     leaves in the same order, and a triangle found in one of them counts
//     only if its leaf's own box passes the exact test.  That test is made
//     when a triangle would be accepted (about once a ray), not per leaf.
// Containment of the boxes is checked while the tree is collapsed
// (k_wide_collapse); a scene that fails it, or whose coordinates are not
// finite or huge, keeps the binary walk.
//
// Conservative inner test.  A plane is base + D(code) * scale with scale a
// power of two; its distance is D * S + B, S = scale * inv (exact), B =
// base * inv - o * inv.  With u = 2^-24, M the scene's largest coordinate on
// the axis and |base| <= 2.4 M, D * scale <= 5.4 M, the rounding of o * inv, B
// and the sum, and of the exact test's own two operations, move the
// comparison by at most u |inv| (6 |o| + 6.4 M); the near distances are
// lowered and the far ones raised by 8 u |inv| (|o| + M) (16 u in watertight
// mode, whose exact exit is scaled by 1 + 8 u).  An axis with a zero direction
// component (inv infinite) uses a power of two that puts its pad far above
// every distance on the other axes, which keeps "inside the slab, its planes
// included" and rejects outside.  Long directions need no bound of their own: a
// product below the normal numbers is off by less than 2^-140, and pads are at
// least 2^-111.  Rays beyond what this argument needs -- denormal components,
// distances beyond about 2^117, no direction at all -- take the binary walk
// (wide_ray), out of line and lane by lane: 2M rays of length 1e8 over 512k
// triangles took 3.6 ms there and take 1.2 here.
//
// Codes: D(code) is the float with code at bits 16-23 under exponent byte
// 0x43: 128 + code below 128, 2 * code above, so one byte permute makes the
// float and the values stay exact.  The two halves of the grid have steps 1
// and 2.  Planes are rounded outwards (wide_box.h), so a stored box holds the
// exact one.
#pragma once

#include "traverse.h"
#include "wide_box.h"

namespace ptb {

// 64 bytes, two 32-byte loads.  Children are four slots (ref as in InnerNode,
// unused slots masked out by valid).  order: for direction octants 0-3, 16
// bits each: nibble c holds the slots visited after slot c.  The opposite
// octant visits in the opposite order.
struct alignas(32) WideNode {
    float    base[3];
    uint32_t exps;          // biased exponents of the three scales, byte 3: valid slots
    uint32_t qlo[3], qhi[3];   // code of slot c at byte c
    uint32_t order[2];
    uint32_t ref[4];
};
static_assert(sizeof(WideNode) == 64, "WideNode must be 64 bytes");

// Triangle record of the wide walk: the 40 bytes of TriRecord and the exact
// box of the triangle's leaf.  64 bytes: one 32-byte and one 8-byte load a
// test, the box only when a triangle would be accepted.
struct alignas(32) WideTri {
    float    v0[3], e1[3], e2xy[2];
    float    e2z;
    uint32_t flags;         // bit 0: last of its leaf
    float    lo[3], hi[3];
};
static_assert(sizeof(WideTri) == 64, "WideTri must be 64 bytes");

constexpr float kWideInvMax = 7.5557864e22f;   // 2^76
constexpr float kWidePadMin = 3.8518599e-34f, kWidePadMax = 1e29f;   // 2^-111; products far from overflow
// (distances on an axis go up to 2^21 pads; of a flat axis's pad the roundings
// leave a fifth)
constexpr float kWideFlatAbove = 16777216.0f;
constexpr uint32_t kWideLiteral = 8u;           // in WideRay::sgn: an inverse is infinite

// A ray as the wide walk holds it.
struct WideRay {
    float    ox, oy, oz, dx, dy, dz;
    float    ix, iy, iz;        // 1 / d, infinite ones replaced
    float    nx, ny, nz;        // -(o * inv + pad): near planes
    float    fx, fy, fz;        // -(o * inv - pad): far planes
    uint32_t sgn;               // direction sign bits x | y << 1 | z << 2; kWideLiteral
};

// False when the ray needs the binary walk.  NaN and infinite origins and
// directions fail by their pads.
PT_HD bool wide_ray(const DeviceScene& s, const RayInv& r, bool watertight, WideRay& w) {
    w.ox = r.ox; w.oy = r.oy; w.oz = r.oz;
    w.dx = r.dx; w.dy = r.dy; w.dz = r.dz;
    w.ix = r.ix; w.iy = r.iy; w.iz = r.iz;
    w.sgn = static_cast<uint32_t>(r.sx | (r.sy << 1) | (r.sz << 2));
    const float k = watertight ? 9.5367432e-7f : 4.7683716e-7f;   // 16 u, 8 u
    bool ok = s.wide_on != 0u;
    if (!(fmaxf(fmaxf(fabsf(r.ix), fabsf(r.iy)), fabsf(r.iz)) <= kWideInvMax)) {
        // an infinite inverse becomes the power of two that puts the pad at 2^79
        // to 2^80 (2^126 at most); the pad must then dominate the other axes
        float flat = FLT_MAX, rest = 0.0f;
        auto fix = [&](float& v, float d, float o, float most) {
            const float a = fmaf(fabsf(o), k, most * k);
            if (d == 0.0f) {
                const uint32_t e = 333u - (__float_as_uint_hd(a) >> 23);
                v = copysignf(__uint_as_float_hd((e < 253u ? e : 253u) << 23), v);
                flat = fminf(flat, a * fabsf(v));
                w.sgn |= kWideLiteral;
            } else {
                ok = ok && fabsf(v) <= kWideInvMax;   // false for NaN and for denormal components
                rest = fmaxf(rest, a * fabsf(v));
            }
        };
        fix(w.ix, r.dx, r.ox, s.coord_max[0]);
        fix(w.iy, r.dy, r.oy, s.coord_max[1]);
        fix(w.iz, r.dz, r.oz, s.coord_max[2]);
        ok = ok && rest > 0.0f && flat >= kWideFlatAbove * rest;
    }
    const float px = fmaf(fabsf(r.ox), k, s.coord_max[0] * k) * fabsf(w.ix);
    const float py = fmaf(fabsf(r.oy), k, s.coord_max[1] * k) * fabsf(w.iy);
    const float pz = fmaf(fabsf(r.oz), k, s.coord_max[2] * k) * fabsf(w.iz);
    w.nx = fmaf(-r.ox, w.ix, -px); w.ny = fmaf(-r.oy, w.iy, -py); w.nz = fmaf(-r.oz, w.iz, -pz);
    w.fx = fmaf(-r.ox, w.ix, px); w.fy = fmaf(-r.oy, w.iy, py); w.fz = fmaf(-r.oz, w.iz, pz);
    return ok && fminf(fminf(px, py), pz) >= kWidePadMin && px < kWidePadMax && py < kWidePadMax && pz < kWidePadMax;
}

// One node in registers.
struct WideRegs {
    float    bx, by, bz;
    uint32_t exps, lo[3], hi[3], o0, o1, ref[4];
};

// D(code of slot c).
template <int C>
PT_HD float wide_code(uint32_t q) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(__byte_perm(q, 0x43000000u, 0x7044u | (C << 8)));
#else
    return wide_decode((q >> (8 * C)) & 255u);
#endif
}

// Conservative entry distances of the four slots; returns the slots hit.
PT_HD uint32_t wide_boxes(const WideRegs& n, const WideRay& r, float best, float (&t)[4]) {
    const float sx = __uint_as_float_hd((n.exps & 0xffu) << 23) * r.ix;
    const float sy = __uint_as_float_hd((n.exps & 0xff00u) << 15) * r.iy;
    const float sz = __uint_as_float_hd((n.exps & 0xff0000u) << 7) * r.iz;
    const float nx = fmaf(n.bx, r.ix, r.nx), ny = fmaf(n.by, r.iy, r.ny), nz = fmaf(n.bz, r.iz, r.nz);
    const float fx = fmaf(n.bx, r.ix, r.fx), fy = fmaf(n.by, r.iy, r.fy), fz = fmaf(n.bz, r.iz, r.fz);
    const uint32_t qnx = (r.sgn & 1u) ? n.hi[0] : n.lo[0], qfx = (r.sgn & 1u) ? n.lo[0] : n.hi[0];
    const uint32_t qny = (r.sgn & 2u) ? n.hi[1] : n.lo[1], qfy = (r.sgn & 2u) ? n.lo[1] : n.hi[1];
    const uint32_t qnz = (r.sgn & 4u) ? n.hi[2] : n.lo[2], qfz = (r.sgn & 4u) ? n.lo[2] : n.hi[2];
    uint32_t h = 0;
#define PT_SLOT(C)                                                                                             \
    {                                                                                                          \
        const float a = fmaf(wide_code<C>(qnx), sx, nx), b = fmaf(wide_code<C>(qny), sy, ny),                  \
                    c = fmaf(wide_code<C>(qnz), sz, nz);                                                       \
        const float d = fmaf(wide_code<C>(qfx), sx, fx), e = fmaf(wide_code<C>(qfy), sy, fy),                  \
                    f = fmaf(wide_code<C>(qfz), sz, fz);                                                       \
        t[C] = fmaxf(fmaxf(a, b), fmaxf(c, 0.0f));                                                             \
        if (t[C] <= fminf(fminf(d, e), fminf(f, best))) h |= 1u << C;                                          \
    }
    PT_SLOT(0) PT_SLOT(1) PT_SLOT(2) PT_SLOT(3)
#undef PT_SLOT
    return h & (n.exps >> 24);
}

#if defined(__CUDACC__)

constexpr uint32_t kNoRef = 0xffffffffu;   // a lane without a ray; an unused slot

// (Volatile: a load that is free to move could move above the test that the
// lane has a node.)
__device__ __forceinline__ WideRegs load_wide(const WideNode* p) {
    WideRegs n;
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(n.bx), "=f"(n.by), "=f"(n.bz), "=r"(n.exps), "=r"(n.lo[0]), "=r"(n.lo[1]), "=r"(n.lo[2]), "=r"(n.hi[0])
        : "l"(p));
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(n.hi[1]), "=r"(n.hi[2]), "=r"(n.o0), "=r"(n.o1), "=r"(n.ref[0]), "=r"(n.ref[1]), "=r"(n.ref[2]),
          "=r"(n.ref[3])
        : "l"(reinterpret_cast<const char*>(p) + 32));
    return n;
}

// Slots visited after each slot (nibbles) in this ray's octant.
__device__ __forceinline__ uint32_t wide_after(const WideRegs& n, uint32_t sgn) {
    const uint32_t flip = (sgn & 4u) ? 0xffffu : 0u;
    const uint32_t k = (sgn ^ ((sgn & 4u) ? 7u : 0u)) & 3u;
    const uint32_t a = (k & 2u) ? n.o1 : n.o0;
    return (((k & 1u) ? a >> 16 : a) ^ flip) & 0x7bdeu;
}

// Number of bits of each nibble of x (each at most 3 of its 4 bits set).
__device__ __forceinline__ uint32_t nibble_counts(uint32_t x) {
    x -= (x >> 1) & 0x5555u;
    return (x & 0x3333u) + ((x >> 2) & 0x3333u);
}

// The literal box test of a ray with an infinite inverse, out of line.
static __device__ __noinline__ bool wide_leaf_literal(float ox, float oy, float oz, float dx, float dy, float dz,
                                                      float2 b0, float2 b1, float2 b2, float best, float xs) {
    RayInv r = make_ray_inv(ox, oy, oz, dx, dy, dz);
    r.xs = xs;
    float en, ex;
    box_span(r, b0.x, b0.y, b1.x, b1.y, b2.x, b2.y, en, ex);
    return en <= best && en <= ex;
}
// Exact box test of the leaf a triangle record belongs to.
template <bool Watertight>
__device__ __forceinline__ bool wide_leaf_passes(const WideTri* p, const WideRay& w, float best) {
    const float2* b = reinterpret_cast<const float2*>(reinterpret_cast<const char*>(p) + 40);
    const float2 b0 = __ldg(b), b1 = __ldg(b + 1), b2 = __ldg(b + 2);
    if (w.sgn & kWideLiteral)
        return wide_leaf_literal(w.ox, w.oy, w.oz, w.dx, w.dy, w.dz, b0, b1, b2, best, exit_scale(Watertight));
    RayInv r;
    r.ox = w.ox; r.oy = w.oy; r.oz = w.oz;
    r.ix = w.ix; r.iy = w.iy; r.iz = w.iz;
    r.xs = exit_scale(Watertight);
    r.nan_free = true;
    float en, ex;
    box_span(r, b0.x, b0.y, b1.x, b1.y, b2.x, b2.y, en, ex);
    return en <= best && en <= ex;
}

// Triangle ti: its distance (or -1), barycentrics and whether it ends its leaf.
template <bool Watertight>
__device__ __forceinline__ float wide_tri(const DeviceScene& s, const WideRay& w, uint32_t ti, bool shadow, float& u,
                                          float& v, bool& last) {
    const WideTri* p = s.wtris + ti;
    RayInv r;
    r.ox = w.ox; r.oy = w.oy; r.oz = w.oz;
    r.dx = w.dx; r.dy = w.dy; r.dz = w.dz;
    const uint2 c = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(p) + 32));
    last = (c.y & 1u) != 0u;
    if (Watertight) {
        const uint4 f = PT_LDGU4(s.faces + ti);
        const float4 p0 = PT_LDG4(s.vertices[f.x].position);
        const float4 p1 = PT_LDG4(s.vertices[f.y].position);
        const float4 p2 = PT_LDG4(s.vertices[f.z].position);
        const float q0[3] = {p0.x, p0.y, p0.z}, q1[3] = {p1.x, p1.y, p1.z}, q2[3] = {p2.x, p2.y, p2.z};
        return tri_watertight(r, q0, q1, q2, shadow, u, v);
    }
    float a[8];
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]), "=f"(a[7])
        : "l"(p));
    return tri_mt(r, a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], __uint_as_float(c.x), shadow, u, v);
}

// The binary walks, out of line, for rays the wide walk does not take.  Their
// scene is rebuilt from the pointers (a reference to the kernel's would put
// the whole parameter block in local memory).
struct BinaryView {
    const InnerNode* inner;
    const TriRecord* tris;
    const pt_face*   faces;
    const pt_vertex* vertices;
    uint32_t         root_ref, watertight;
    float            lo[3], hi[3];
};
__device__ __forceinline__ BinaryView binary_view(const DeviceScene& s, bool watertight) {
    return BinaryView{s.inner, s.tris, s.faces, s.vertices, s.root_ref, watertight ? 1u : 0u,
                      {s.root_lo[0], s.root_lo[1], s.root_lo[2]}, {s.root_hi[0], s.root_hi[1], s.root_hi[2]}};
}
__device__ __forceinline__ void binary_scene(const BinaryView& b, DeviceScene& s) {
    s.inner = b.inner; s.tris = b.tris; s.faces = b.faces; s.vertices = b.vertices;
    s.root_ref = b.root_ref;
    s.num_faces = 1u;
    for (int a = 0; a < 3; ++a) { s.root_lo[a] = b.lo[a]; s.root_hi[a] = b.hi[a]; }
}
struct BinaryHit { int prim; float t, u, v; uint32_t err; };
static __device__ __noinline__ BinaryHit closest_binary(BinaryView b, float ox, float oy, float oz, float dx, float dy,
                                                        float dz) {
    DeviceScene s;
    binary_scene(b, s);
    BinaryHit h;
    h.err = 0u;
    TraceCounters tc{0, 0};
    h.prim = trace_closest(s, make_ray_inv(ox, oy, oz, dx, dy, dz), b.watertight != 0u, h.t, h.u, h.v, h.err, tc);
    return h;
}
// bit 31: occluded; the rest: error bits
static __device__ __noinline__ uint32_t any_binary(BinaryView b, float ox, float oy, float oz, float dx, float dy,
                                                   float dz, float tmax) {
    DeviceScene s;
    binary_scene(b, s);
    uint32_t err = 0u;
    TraceCounters tc{0, 0};
    const bool hit = trace_any(s, make_ray_inv(ox, oy, oz, dx, dy, dz), tmax, b.watertight != 0u, err, tc);
    return err | (hit ? 0x80000000u : 0u);
}

// How a warp divides its time.  Its lanes walk different rays, so at any
// moment some stand on inner nodes, some at a leaf, some are out of work.  A
// warp keeps stepping through inner nodes while at least kWideInnerMin of its
// lanes (kWideAnyInnerMin for shadow rays) stand on one, two steps a vote;
// below that the lanes at leaves test their
// triangles.  Finished rays are stored, and new ones set up, once kWideFetchMin
// lanes are out of work.  The walks are bound by issue slots: 16.7 of 32 lanes
// active, 68 % of slots used (closed 200k-triangle room, second bounce).
// Extension / shadow stage of that room at 1024 x 1024, 64 spp, depth 16, as
// the loop was built up: binary tree, all lanes to a leaf before any tests it
// 139 / 80 ms; four-wide tree, threshold 16, refill at once 101 / 63 ms; 64
// registers 94 / 63 ms; contiguous chunks 91 / 59 ms; no order for shadow rays
// 91 / 47 ms; two steps a vote, threshold 20 90 / 46 ms.  Thresholds 8 to 24
// and refills at 1 to 12 lanes lie within 6 %.
constexpr int kWideInnerMin = 20, kWideAnyInnerMin = 16, kWideFetchMin = 4;

// A warp's share of the rays: contiguous chunks, handed out in order to the
// lanes that ask, so that a warp's rays stay neighbours in the queue (a grid
// stride per lane lets them drift apart: 4 % slower).  Chunks of 128, fewer
// where the queue is short so that every warp gets at least four.
constexpr uint32_t kWideChunk = 128;
struct RayFeed {
    uint32_t n, chunk, jump, base, next, lim;
    __device__ __forceinline__ explicit RayFeed(uint32_t n_rays) {
        const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
        n = n_rays;
        chunk = max(32u, min(kWideChunk, (n / (warps * 4u)) & ~31u));
        jump = chunk * warps;
        base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * chunk;
        next = base;
        lim = min(base + chunk, n);
    }
    __device__ __forceinline__ bool more() const { return base < n; }
    // a ray for each lane of `idle` (kNoRef: none this time)
    __device__ __forceinline__ uint32_t take(uint32_t idle) {
        const uint32_t mine = next + __popc(idle & ((1u << (threadIdx.x & 31u)) - 1u));
        const uint32_t r = mine < lim ? mine : kNoRef;
        next += __popc(idle);
        if (next >= lim) {
            base += jump;
            next = base;
            lim = min(base + chunk, n);
        }
        return r;
    }
};

// Lanes whose ref is an inner node / any lane waiting at a leaf.
__device__ __forceinline__ bool go_on(uint32_t ref, int least) {
    const uint32_t in = __ballot_sync(0xffffffffu, !(ref & kLeafBit));
    if (in == 0u) return false;
    return __popc(in) >= least || !__any_sync(0xffffffffu, (ref & kLeafBit) && ref != kNoRef);
}

// Closest hits of rays 0 .. n - 1 over the wide tree, for the whole grid.
// fetch(i, RayInv&) loads ray i; done(i, prim, t, u, v) stores its result.
// The scene has faces (wide_on).
template <int Depth, bool Watertight, class Fetch, class Done>
__device__ __forceinline__ void wide_closest_loop(const DeviceScene& s, uint32_t n, uint32_t& err, Fetch&& fetch,
                                                  Done&& done) {
    RayFeed feed(n);
    uint2 stack[Depth];   // deferred nodes and their entry distances
    WideRay w;
    float best = FLT_MAX, bu = 0.0f, bv = 0.0f;
    int prim = -1, sp = 0;
    uint32_t ref = kNoRef, i = 0;
    bool open = false;    // ray i is walked or its result not stored yet
    // next deferred node that still passes the best distance
    auto pop = [&]() {
        ref = kNoRef;
        while (sp > 0) {
            const uint2 e = stack[--sp];
            if (__uint_as_float(e.y) <= best) { ref = e.x; break; }
        }
    };
    // inner node ref: its hit slots go on the stack, farthest first, and the
    // nearest becomes ref
    auto step = [&]() {
        const WideRegs nd = load_wide(s.wide + ref);
        float t[4];
        const uint32_t h = wide_boxes(nd, w, best, t);
        if (h == 0u) { pop(); return; }
        if (sp + 3 > Depth) { err |= kErrStackOverflow; ref = kNoRef; return; }
        // slot c goes behind the hit slots visited after it; the one in front
        // of all others is next
        const uint32_t cnt = nibble_counts(wide_after(nd, w.sgn) & (h * 0x1111u));
        const uint32_t top = static_cast<uint32_t>(__popc(h)) - 1u;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t k = (cnt >> (4 * c)) & 3u;
            if (h & (1u << c)) {
                if (k == top) ref = nd.ref[c];
                else stack[sp + static_cast<int>(k)] = make_uint2(nd.ref[c], __float_as_uint(t[c]));
            }
        }
        sp += static_cast<int>(top);
    };
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, ref == kNoRef);
        if (__popc(idle) >= kWideFetchMin) {
            if (ref == kNoRef && open) { done(i, prim, best, bu, bv); open = false; }
            if (feed.more()) {
                const uint32_t mine = feed.take(idle);
                if (ref == kNoRef && mine != kNoRef) {
                    RayInv r;
                    i = mine;
                    fetch(i, r);
                    best = FLT_MAX; bu = 0.0f; bv = 0.0f; prim = -1; sp = 0;
                    if (wide_ray(s, r, Watertight, w)) {
                        ref = s.wide_root;
                        open = true;
                    } else {
                        const BinaryHit h = closest_binary(binary_view(s, Watertight), r.ox, r.oy, r.oz, r.dx, r.dy, r.dz);
                        err |= h.err;
                        done(i, h.prim, h.t, h.u, h.v);
                    }
                }
            } else if (idle == 0xffffffffu) {
                break;
            }
            __syncwarp();
        }
        while (go_on(ref, kWideInnerMin)) {
            if (!(ref & kLeafBit)) step();
            __syncwarp();
            if (!(ref & kLeafBit)) step();
            __syncwarp();
        }
        if ((ref & kLeafBit) && ref != kNoRef) {
            // the nearest triangle of the leaf; its leaf's box is tested once
            // for all lanes, against the distance before the leaf
            uint32_t ti = ref & ~kLeafBit, lp = kNoRef;
            float bt = best, lu = 0.0f, lv = 0.0f;
            for (;;) {
                float u, v; bool last;
                const float t = wide_tri<Watertight>(s, w, ti, false, u, v, last);
                if (t >= 0.0f && t < bt) { bt = t; lp = ti; lu = u; lv = v; }
                if (last) break;
                ++ti;
            }
            if (lp != kNoRef && wide_leaf_passes<Watertight>(s.wtris + lp, w, best)) {
                best = bt; prim = static_cast<int>(lp); bu = lu; bv = lv;
            }
            pop();
        }
        __syncwarp();
    }
}

// Any-hit tests of rays 0 .. n - 1 over the wide tree, for the whole grid.
// fetch(i, RayInv&) returns tmax; done(i, occluded) consumes the result.  The
// answer does not depend on the order, so the slots are taken as they come:
// without the ordering a step is a quarter shorter (59 -> 47 ms above).
template <int Depth, bool Watertight, class Fetch, class Done>
__device__ __forceinline__ void wide_any_loop(const DeviceScene& s, uint32_t n, uint32_t& err, Fetch&& fetch,
                                              Done&& done) {
    RayFeed feed(n);
    uint32_t stack[Depth];
    WideRay w;
    float tmax = 0.0f;
    int sp = 0;
    uint32_t ref = kNoRef, i = 0;
    bool open = false, hit = false;
    // one inner node: the last child hit is next, the others go on the stack
    auto step = [&] {
        const WideRegs nd = load_wide(s.wide + ref);
        float t[4];
        const uint32_t h = wide_boxes(nd, w, tmax, t);
        ref = kNoRef;
        if (sp + 3 > Depth) {
            err |= kErrStackOverflow;
            return;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (h & (1u << c)) {
                if (ref != kNoRef) stack[sp++] = ref;
                ref = nd.ref[c];
            }
        if (ref == kNoRef && sp > 0) ref = stack[--sp];
    };
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, ref == kNoRef);
        if (__popc(idle) >= kWideFetchMin) {
            if (ref == kNoRef && open) { done(i, hit); open = false; }
            if (feed.more()) {
                const uint32_t mine = feed.take(idle);
                if (ref == kNoRef && mine != kNoRef) {
                    RayInv r;
                    i = mine;
                    tmax = fetch(i, r);
                    sp = 0;
                    hit = false;
                    if (wide_ray(s, r, Watertight, w)) {
                        ref = s.wide_root;
                        open = true;
                    } else {
                        const uint32_t h = any_binary(binary_view(s, Watertight), r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, tmax);
                        err |= h & 0x7fffffffu;
                        done(i, (h & 0x80000000u) != 0u);
                    }
                }
            } else if (idle == 0xffffffffu) {
                break;
            }
            __syncwarp();
        }
        while (go_on(ref, kWideAnyInnerMin)) {
            if (!(ref & kLeafBit)) step();
            __syncwarp();
            if (!(ref & kLeafBit)) step();
            __syncwarp();
        }
        if ((ref & kLeafBit) && ref != kNoRef) {
            uint32_t ti = ref & ~kLeafBit;
            bool got = false;
            for (;;) {
                float u, v; bool last;
                const float t = wide_tri<Watertight>(s, w, ti, true, u, v, last);
                got = t > 0.0f && t < tmax;
                if (got || last) break;
                ++ti;
            }
            hit = got && wide_leaf_passes<Watertight>(s.wtris + ti, w, tmax);
            ref = !hit && sp > 0 ? stack[--sp] : kNoRef;
        }
        __syncwarp();
    }
}

#endif  // __CUDACC__

}  // namespace ptb
