// rt_traverse.cuh -- per-ray traversal of the 8-wide quantised BVH, the
// reference-exact Moller-Trumbore test, and the shading helpers shared by
// every kernel of the core.
//
// Traversal keeps node groups (child base + hit bits) on a per-ray stack:
// internal-child hits live in bits 24..31 at position slot ^ octant ^ 7 so the
// highest set bit is the child nearest the ray's origin side, the node's
// internal-child mask rides in bits 0..7, and leaf triangles of a node are
// tested as soon as the node is intersected (after Ylitie et al., HPG 2017).
#pragma once

#include "rt_internal.cuh"

namespace rtc {

struct RayState {
    float3 o, d;
};

// Reference-exact triangle test (triangle::is_intersecting,
// raytracer/triangle.h:190-235): e1 = c - a, e2 = b - a, reject
// |det| < 1e-6, u weighs c, v weighs b.  Returns t, or +inf when rejected.
__device__ __forceinline__ float mt_intersect(const float4 w0, const float4 w1, const float4 w2, const float3 o,
                                              const float3 d, float &u_out, float &v_out)
{
    const float3 a = make_float3(w0.x, w0.y, w0.z);
    const float3 b = make_float3(w0.w, w1.x, w1.y);
    const float3 c = make_float3(w1.z, w1.w, w2.x);
    const float3 e1 = xsub3(c, a);   // triangle.h:193
    const float3 e2 = xsub3(b, a);   // triangle.h:194
    const float3 P = xcross(d, e2);
    const float det = xdot(e1, P);
    const float inv_det = __frcp_rn(det);      // == 1.0f / det, correctly rounded
    const float3 T = xsub3(o, a);
    const float u = xmul(xdot(T, P), inv_det);
    const float3 Q = xcross(T, e1);
    const float v = xmul(xdot(d, Q), inv_det);
    const float t = xmul(xdot(e2, Q), inv_det);
    const bool reject = (det > -kDetEps && det < kDetEps) || (u < 0.0f) || (v < 0.0f) || (xadd(u, v) > 1.0f);
    u_out = u;
    v_out = v;
    return reject ? __int_as_float(0x7f800000) : t;
}

// Per-ray constants of the watertight test: the axis of largest |d| is z
// (kx, ky follow, swapped when d.z < 0 to keep the winding), and the shear
// that maps the ray to +z.
struct Shear {
    int kx, ky, kz;
    float sx, sy, sz;
};

__device__ __forceinline__ float comp(const float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

__device__ __forceinline__ Shear make_shear(const float3 d)
{
    Shear s;
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    s.kz = (ax > ay) ? ((ax > az) ? 0 : 2) : ((ay > az) ? 1 : 2);
    s.kx = (s.kz + 1) % 3;
    s.ky = (s.kx + 1) % 3;
    if (comp(d, s.kz) < 0.0f) { const int t = s.kx; s.kx = s.ky; s.ky = t; }
    const float dz = comp(d, s.kz);
    s.sx = comp(d, s.kx) / dz;
    s.sy = comp(d, s.ky) / dz;
    s.sz = 1.0f / dz;
    return s;
}

// Watertight ray/triangle test of Woop, Benthin and Wald (JCGT 2013): the
// three edge functions are evaluated in the ray's sheared frame from the
// exact vertex positions, so two triangles sharing an edge always agree on
// which side a ray passes (no ray leaks through a shared edge); an edge
// function that rounds to exactly zero is re-evaluated in double.  Returns
// t (accepting t > 0 here; the caller applies EPSILON), or +inf.  u weighs
// c and v weighs b, as in the reference.
__device__ __forceinline__ float wt_intersect(const float4 w0, const float4 w1, const float4 w2, const float3 o,
                                              const Shear &sh, float &u_out, float &v_out)
{
    const float3 A = make_float3(w0.x - o.x, w0.y - o.y, w0.z - o.z);
    const float3 B = make_float3(w0.w - o.x, w1.x - o.y, w1.y - o.z);
    const float3 C = make_float3(w1.z - o.x, w1.w - o.y, w2.x - o.z);
    const float Az = comp(A, sh.kz), Bz = comp(B, sh.kz), Cz = comp(C, sh.kz);
    // every vertex is sheared by the same uncontracted operations, so a
    // vertex shared by several triangles lands on the same point in all
    const float Ax = xsub(comp(A, sh.kx), xmul(sh.sx, Az)), Ay = xsub(comp(A, sh.ky), xmul(sh.sy, Az));
    const float Bx = xsub(comp(B, sh.kx), xmul(sh.sx, Bz)), By = xsub(comp(B, sh.ky), xmul(sh.sy, Bz));
    const float Cx = xsub(comp(C, sh.kx), xmul(sh.sx, Cz)), Cy = xsub(comp(C, sh.ky), xmul(sh.sy, Cz));
    // uncontracted products: an edge shared by two triangles gives exactly
    // negated edge functions in both
    float U = xsub(xmul(Cx, By), xmul(Cy, Bx));
    float V = xsub(xmul(Ax, Cy), xmul(Ay, Cx));
    float W = xsub(xmul(Bx, Ay), xmul(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
        V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
        W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    const float inf = __int_as_float(0x7f800000);
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return inf;
    const float det = U + V + W;
    if (det == 0.0f) return inf;
    const float T = (U * (sh.sz * Az) + V * (sh.sz * Bz)) + W * (sh.sz * Cz);
    const float inv = 1.0f / det;
    const float t = T * inv;
    if (!(t > 0.0f)) return inf;
    u_out = W * inv;   // weight of c
    v_out = V * inv;   // weight of b
    return t;
}

// Child-box test of one wide node: internal-hit bits (24..31, in the ray's
// order, nearest highest) | imask (0..7) in ngroup.y with child_base in
// ngroup.x; the hit leaf slots as an 8-bit mask (slot order) with the node's
// triangle base and meta bytes.
struct NodeHits {
    uint2 ngroup;
    uint32_t leaf_slots;
    uint32_t tri_base, meta_lo, meta_hi;
};

// Signed byte weights -(1 << s) of slots s = 0..3 and 4..7: the dot product
// of a byte mask (0xff = -1 per marked slot) with them is the slots' bit mask.
constexpr uint32_t kSlotWeightsLo = 0xF8FCFEFFu, kSlotWeightsHi = 0x80C0E0F0u;

// Highest set bit (one instruction; the lowest would take a bit reversal too).
__device__ __forceinline__ uint32_t top_bit(uint32_t v) { return 31u - (uint32_t)__clz((int)v); }

// prmt with its sign-replicate selectors (bit 3 of a nibble), which
// __byte_perm does not promise.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// Byte masks (0xff: sign bit set) of four floats.
__device__ __forceinline__ uint32_t sign_bytes(float a, float b, float c, float d)
{
    const uint32_t lo = prmt(__float_as_uint(a), __float_as_uint(b), 0x00FBu);
    const uint32_t hi = prmt(__float_as_uint(c), __float_as_uint(d), 0xFB00u);
    return prmt(lo, hi, 0x7610u);
}

// max / min of three floats (one instruction).
__device__ __forceinline__ float fmax3f(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmin3f(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Packed single-precision arithmetic (sm_100 family): each half rounded
// exactly as its scalar counterpart.
__device__ __forceinline__ uint64_t pack2f(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 fma2f(float a0, float a1, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pack2f(a0, a1)), "l"(b), "l"(c));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return r;
}
__device__ __forceinline__ float2 sub2f(float a0, float a1, float b0, float b1)
{
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2f(a0, a1)), "l"(pack2f(b0, b1)));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return r;
}

// One axis of a wide node for one ray.  A plane byte q becomes the float
// 1 + q * 2^-16 (kQWeight * q added to the bits of 1.0f by one byte dot
// product, whose weight picks the byte), so that plane distances are
// t = (1 + q * 2^-16) * scale + offset with scale = 2^16 * step / d and
// offset = (origin - o) / d - scale.  The offset rounds at the magnitude of
// 2^16 steps: an error below 2^-7 of one step, far inside the one-step
// padding of every box.
constexpr float kQScale = 65536.0f;
constexpr uint32_t kQWeight = 0x80u;
struct AxisPlanes {
    uint64_t scale, offset;   // the same value in both halves
    uint32_t near_w;          // weights that pick an even slot's entry plane: byte 0 (d >= 0) or 1
};
__device__ __forceinline__ AxisPlanes axis_planes(uint32_t e, float p, float o, float inv)
{
    const float s = __uint_as_float(e << 23) * inv * kQScale;
    const float off = (p - o) * inv - s;
    AxisPlanes A;
    A.scale = pack2f(s, s);
    A.offset = pack2f(off, off);
    A.near_w = kQWeight << (8 * (__float_as_uint(inv) >> 31));
    return A;
}

// Plane distances of two neighbouring slots (w: low, high, low, high).
__device__ __forceinline__ float2 plane_pair(uint32_t w, uint32_t weights, const AxisPlanes &A)
{
    const uint32_t one = 0x3F800000u;
    const uint32_t a = __dp4a(w, weights, one), b = __dp4a(w, weights << 16, one);
    return fma2f(__uint_as_float(a), __uint_as_float(b), A.scale, A.offset);
}

// What bounds it: the two half-rate arithmetic pipes (a node test alone runs
// no faster beyond two warps per scheduler).  Byte dot products run on the
// multiply pipe and byte permutes, selects, min/max and compares on the
// other, so the plane bytes go through __dp4a -- which also picks the entry
// or exit plane by its weights, where separate planes needed 12 selects --
// and the hit masks are formed from sign bits by permutes and dot products
// instead of a compare and three bit operations per slot.  Cycles per node and
// scheduler: 246; 286 with permutes and selects, 257 with permutes alone.
// Together with the watertight test in kernels of its own: 2M any-hit rays
// 718 -> 631 us, 1080p terrain frame 759 -> 695 us, AO-instances frame 4.10 ->
// 3.76 ms, glass trees 713 -> 642 us.
__device__ __forceinline__ NodeHits intersect_node(const WideNode *__restrict__ nodes, uint32_t idx, const float3 o,
                                                   const float3 inv, uint32_t w0, uint32_t w1, float tmax)
{
    const float4 *np = reinterpret_cast<const float4 *>(nodes + idx);
    const float4 n0 = __ldg(np + 0);
    const float4 n1 = __ldg(np + 1);
    const float4 n2 = __ldg(np + 2);
    const float4 n3 = __ldg(np + 3);
    const float4 n4 = __ldg(np + 4);
    const uint32_t e_imask = __float_as_uint(n0.w);
    const uint32_t meta_lo = __float_as_uint(n1.z), meta_hi = __float_as_uint(n1.w);
    const AxisPlanes X = axis_planes(e_imask & 0xffu, n0.x, o.x, inv.x);
    const AxisPlanes Y = axis_planes((e_imask >> 8) & 0xffu, n0.y, o.y, inv.y);
    const AxisPlanes Z = axis_planes((e_imask >> 16) & 0xffu, n0.z, o.z, inv.z);
    const uint32_t far_w = kQWeight | (kQWeight << 8);   // near_w ^ far_w: the exit plane's weights
    const uint32_t wx[4] = {__float_as_uint(n2.x), __float_as_uint(n2.y), __float_as_uint(n2.z), __float_as_uint(n2.w)};
    const uint32_t wy[4] = {__float_as_uint(n3.x), __float_as_uint(n3.y), __float_as_uint(n3.z), __float_as_uint(n3.w)};
    const uint32_t wz[4] = {__float_as_uint(n4.x), __float_as_uint(n4.y), __float_as_uint(n4.z), __float_as_uint(n4.w)};
    float m[8];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const float2 nx = plane_pair(wx[p], X.near_w, X), fx = plane_pair(wx[p], X.near_w ^ far_w, X);
        const float2 ny = plane_pair(wy[p], Y.near_w, Y), fy = plane_pair(wy[p], Y.near_w ^ far_w, Y);
        const float2 nz = plane_pair(wz[p], Z.near_w, Z), fz = plane_pair(wz[p], Z.near_w ^ far_w, Z);
        // the box is hit when max(near, 0) <= min(far, tmax): no sign bit in
        // the difference (a NaN, from an overflowing scale, counts as a hit)
        const float2 d = sub2f(fmin3f(fx.x, fy.x, fminf(fz.x, tmax)), fmin3f(fx.y, fy.y, fminf(fz.y, tmax)),
                               fmax3f(nx.x, ny.x, fmaxf(nz.x, 0.0f)), fmax3f(nx.y, ny.y, fmaxf(nz.y, 0.0f)));
        m[2 * p] = d.x;
        m[2 * p + 1] = d.y;
    }
    // an empty slot needs no test of its own: its box is inverted, and should
    // rounding let it "hit", it has no internal bit and no triangles
    const uint32_t miss_lo = sign_bytes(m[0], m[1], m[2], m[3]), miss_hi = sign_bytes(m[4], m[5], m[6], m[7]);
    const uint32_t int_lo = prmt(meta_lo, 0u, 0xBA98u), int_hi = prmt(meta_hi, 0u, 0xBA98u);   // sign bits of the meta bytes
    const int hits_int = __dp4a((int)(~miss_lo & int_lo), (int)w0, __dp4a((int)(~miss_hi & int_hi), (int)w1, 0));
    const int hits_leaf = __dp4a((int)~(miss_lo | int_lo), (int)kSlotWeightsLo,
                                 __dp4a((int)~(miss_hi | int_hi), (int)kSlotWeightsHi, 0));
    NodeHits h;
    // byte 3: the internal hits, byte 0: imask (bits 8..23 are not looked at)
    h.ngroup = make_uint2(__float_as_uint(n1.x), prmt((uint32_t)hits_int, e_imask, 0x0447u));
    h.leaf_slots = (uint32_t)hits_leaf;
    h.tri_base = __float_as_uint(n1.y);
    h.meta_lo = meta_lo;
    h.meta_hi = meta_hi;
    return h;
}

// The triangles of a node's hit leaf slots as bits from its triangle base.
__device__ __forceinline__ uint32_t leaf_triangles(const NodeHits &h)
{
    uint32_t bits = 0u;
    for (uint32_t ls = h.leaf_slots; ls != 0u;) {
        const uint32_t s = __ffs(ls) - 1u;
        ls &= ls - 1u;
        const uint32_t m = prmt(h.meta_lo, h.meta_hi, s) & 0xffu;
        bits |= ((1u << (m >> 5)) - 1u) << (m & 31u);
    }
    return bits;
}

__device__ __forceinline__ float3 safe_inv(float3 d)
{
    const float tiny = 1e-20f;
    const float x = (fabsf(d.x) > tiny) ? d.x : copysignf(tiny, d.x);
    const float y = (fabsf(d.y) > tiny) ? d.y : copysignf(tiny, d.y);
    const float z = (fabsf(d.z) > tiny) ? d.z : copysignf(tiny, d.z);
    return make_float3(__frcp_rn(x), __frcp_rn(y), __frcp_rn(z));
}

__device__ __forceinline__ uint32_t octant_of(float3 d)
{
    return (d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u);
}

// kSlotWeights with the slots permuted by `order`: bit s ^ order for slot s.
__device__ __forceinline__ void order_weights(uint32_t order, uint32_t &w0, uint32_t &w1)
{
    const uint32_t sel = 0x3210u ^ (0x1111u * (order & 3u));
    const uint32_t lo = prmt(kSlotWeightsLo, 0u, sel), hi = prmt(kSlotWeightsHi, 0u, sel);
    w0 = (order & 4u) ? hi : lo;
    w1 = (order & 4u) ? lo : hi;
}

struct HitRecord {
    int32_t id;
    float t, u, v;
};
struct FetchCount {
    uint32_t nodes = 0;
    uint32_t tris = 0;
};

// Resumable traversal state of one ray: trav_begin sets it up, each
// trav_step intersects one node (or resumes a stacked node group) and tests
// that node's leaf triangles.  The stack lives with the caller.
struct Trav {
    float3 o, d, inv;
    uint32_t order;    // octant ^ 7: slot s has bit 24 + (s ^ order), nearest highest
    uint32_t w0, w1;   // order_weights
    float tmax;        // any-hit limit
    float box_tmax;    // boxes beyond this are culled (closest: best t so far)
    uint2 ngroup;
    int sp;
    int steps;
    HitRecord hit;
    bool occluded;
};

__device__ __forceinline__ void trav_begin(Trav &T, const SceneView &sc, const float3 o, const float3 d, float tmax,
                                           bool any)
{
    T.o = o;
    T.d = d;
    T.inv = safe_inv(d);
    T.order = octant_of(d) ^ 7u;
    order_weights(T.order, T.w0, T.w1);
    T.tmax = tmax;
    T.box_tmax = any ? tmax : FLT_MAX;
    // a group holding only the root (as slot 0 of a virtual parent)
    T.ngroup = make_uint2((uint32_t)sc.root, sc.nnodes > 0 ? ((1u << (24 + T.order)) | 1u) : 0u);
    T.sp = 0;
    T.steps = 0;
    T.hit.id = -1;
    T.hit.t = FLT_MAX;
    T.hit.u = 0.f;
    T.hit.v = 0.f;
    T.occluded = false;
}

// One traversal step; returns true when the ray is finished.  Closest hit
// (any = false) or any hit inside (EPSILON, tmax) skipping light and
// transparent triangles (any = true).  WT: the watertight triangle test.
// Status bits go to `status`.  STACK: the stack's capacity in node groups (a
// ray holds at most one group per tree level, so any capacity above the
// tree's depth suffices).
template <bool COUNT, bool WT, int STACK = kStackSize>
__device__ __forceinline__ bool trav_step(Trav &T, uint2 *stack, const SceneView &sc, bool any, uint32_t &status,
                                          FetchCount *fc)
{
    if (++T.steps > kMaxTraversalSteps) { status |= kStatusStepLimit; return true; }
    uint32_t tri_base = 0u, tri_bits = 0u;
    if (T.ngroup.y & 0xff000000u) {
        const uint32_t bit = top_bit(T.ngroup.y);
        T.ngroup.y ^= 1u << bit;
        const uint32_t slot = (bit ^ T.order) & 7u;
        const uint32_t idx = T.ngroup.x + __popc(T.ngroup.y & ((1u << slot) - 1u));
        if (idx >= (uint32_t)sc.nnodes) { status |= kStatusBadIndex; return true; }
        if (T.ngroup.y & 0xff000000u) {
            if (T.sp >= STACK) { status |= kStatusStackOverflow; return true; }
            stack[T.sp++] = T.ngroup;
        }
        const NodeHits nh = intersect_node(any ? sc.any_nodes : sc.nodes, idx, T.o, T.inv, T.w0, T.w1, T.box_tmax);
        if (COUNT) ++fc->nodes;
        T.ngroup = nh.ngroup;
        tri_base = nh.tri_base;
        tri_bits = leaf_triangles(nh);
    }
    while (tri_bits != 0u) {
        const uint32_t k = __ffs(tri_bits) - 1u;
        tri_bits &= tri_bits - 1u;
        const uint32_t ti = tri_base + k;
        if (ti >= (uint32_t)sc.ntris) { status |= kStatusBadIndex; continue; }
        const PackedTri *tp = sc.tris + ti;
        if (COUNT) ++fc->tris;
        const float4 w0 = __ldg(&tp->w0);
        const float4 w1 = __ldg(&tp->w1);
        const float4 w2 = __ldg(&tp->w2);
        float u = 0.f, v = 0.f;
        const float t = WT ? wt_intersect(w0, w1, w2, T.o, make_shear(T.d), u, v)
                           : mt_intersect(w0, w1, w2, T.o, T.d, u, v);
        const int32_t id = __float_as_int(w2.y);
        if ((uint32_t)id >= (uint32_t)sc.ntris) { status |= kStatusBadIndex; continue; }
        if (any) {
            if ((__float_as_uint(w2.z) & (RT_TRI_LIGHT | RT_TRI_TRANSPARENT)) == 0u && t > kEpsilon && t < T.tmax) {
                T.occluded = true;
                T.hit.id = id;
                T.hit.t = t;
                return true;
            }
        } else if (t > kEpsilon && (t < T.hit.t || (t == T.hit.t && id < T.hit.id))) {
            T.hit.id = id;
            T.hit.t = t;
            T.hit.u = u;
            T.hit.v = v;
            T.box_tmax = t;
        }
    }
    if (!(T.ngroup.y & 0xff000000u)) {
        if (T.sp == 0) return true;
        T.ngroup = stack[--T.sp];
    }
    return false;
}

// Whole traversal of one ray, closest or any hit.  Returns the device status
// bits.
template <bool COUNT, int STACK = kStackSize, class SC>
__device__ __forceinline__ uint32_t traverse_ray(const SC &sc, const float3 o, const float3 d, float tmax, bool any,
                                                 HitRecord &hit, bool &occluded, FetchCount *fc = nullptr)
{
    uint2 stack[STACK];
    Trav T;
    trav_begin(T, sc, o, d, tmax, any);
    uint32_t status = 0u;
    while (!trav_step<COUNT, SC::kWatertight, STACK>(T, stack, sc, any, status, fc)) {
    }
    hit = T.hit;
    occluded = T.occluded;
    return status;
}

template <bool ANY, bool COUNT = false, int STACK = kStackSize, class SC>
__device__ __forceinline__ uint32_t traverse(const SC &sc, const float3 o, const float3 d, float tmax, HitRecord &hit,
                                             bool &occluded, FetchCount *fc = nullptr)
{
    return traverse_ray<COUNT, STACK>(sc, o, d, tmax, ANY, hit, occluded, fc);
}

// Traversal of a list of rays by a warp whose lanes take further rays once
// kIdle of them are idle (4 and 16 were slower), every lane calling it, converged.
// claim(want, base): up to `want` further rays, base on, the same for all lanes;
// 0: none are left.  fetch(take, k, o, d, tmax): ray k, for the lanes with take
// set.  done(k, trav): its result, lane by lane.
constexpr int kIdle = 8;
template <bool ANY, class SC, class Claim, class Fetch, class Done>
__device__ __forceinline__ uint32_t traverse_list(const SC &sc, Claim claim, Fetch fetch, Done done)
{
    const uint32_t full = 0xffffffffu, below = (1u << (threadIdx.x & 31u)) - 1u;
    uint2 stack[kStackSize];
    Trav T;
    int ray = -1;
    int refill = kIdle;   // 32 once no rays are left
    uint32_t status = 0u;
    for (;;) {
        const uint32_t idle = __ballot_sync(full, ray < 0);
        if (__popc(idle) >= refill) {
            int base = 0;
            const int got = claim(__popc(idle), base);
            if (got == 0) {
                if (idle == full) break;
                refill = 32;
                continue;
            }
            const int rank = __popc(idle & below);
            const bool take = ray < 0 && rank < got;
            float3 o, d;
            float tmax;
            fetch(take, base + rank, o, d, tmax);
            if (take) {
                ray = base + rank;
                trav_begin(T, sc, o, d, tmax, ANY);
            }
        }
        if (ray >= 0 && trav_step<false, SC::kWatertight>(T, stack, sc, ANY, status, nullptr)) {
            done(ray, T);
            ray = -1;
        }
    }
    return status;
}

// Traversal of a warp's rays in step, for rays that take similar paths (every
// lane of the warp calls it, converged; live: the lane has a ray).  In
// traverse a warp tests triangles after every node for the few lanes that met
// some (4.9 of 32 on the terrain frame, three tests for every two nodes).
// Here a lane holds the triangles of a node and goes on to the next nodes; one
// that can go no further without its triangles -- a second node's are held, or
// it has no node left -- waits, and once kWaiting lanes wait (or none can go
// on) the warp tests one triangle of every lane that holds some.  The same
// hits: neither kind depends on the order of the tests.
// Measured (kWaiting 3; 2 to 6 tried): terrain 1080p 0.781 -> 0.733 ms, 20k
// sphere 512^2 140 -> 131 us; rays in all directions lose (AO 3.82 -> 4.15 ms,
// 2M incoherent any-hit rays 604 -> 710 us), as a delayed test finds its ray's
// end later, so those stay with traverse.
constexpr int kWaiting = 3;
template <bool ANY, bool COUNT = false, int STACK = kStackSize, class SC>
__device__ __forceinline__ uint32_t traverse_warp(const SC &sc, bool live, const float3 o, const float3 d, float tmax,
                                                  HitRecord &hit, bool &occluded, FetchCount *fc = nullptr)
{
    const uint32_t full = 0xffffffffu, hit_bits = 0x00ffffffu;   // a group with hits is above hit_bits
    uint2 stack[STACK];
    const float3 inv = safe_inv(d);
    const uint32_t order = octant_of(d) ^ 7u;
    uint32_t w0, w1;
    order_weights(order, w0, w1);
    float best = ANY ? tmax : FLT_MAX;
    uint2 group = make_uint2((uint32_t)sc.root, live && sc.nnodes > 0 ? ((1u << (24 + order)) | 1u) : 0u);
    int sp = 0, steps = 0;
    // held triangles (base and bits): of one node, of a second one
    uint32_t base0 = 0u, bits0 = 0u, base1 = 0u, bits1 = 0u;
    uint32_t status = 0u;
    hit.id = -1;
    hit.t = FLT_MAX;
    hit.u = 0.f;
    hit.v = 0.f;
    occluded = false;
    for (;;) {
        const uint32_t holding = __ballot_sync(full, bits0 != 0u);
        const uint32_t can = __ballot_sync(full, group.y > hit_bits && bits1 == 0u);
        const uint32_t waiting = __ballot_sync(full, bits0 != 0u && (bits1 != 0u || group.y <= hit_bits));
        if (__popc(waiting) >= kWaiting || !can) {
            if (!holding && !can) break;
            if (bits0 != 0u) {
                const uint32_t k = top_bit(bits0);
                bits0 ^= 1u << k;
                const PackedTri *tp = sc.tris + (base0 + k);
                if (COUNT) ++fc->tris;
                const float4 v0 = __ldg(&tp->w0);
                const float4 v1 = __ldg(&tp->w1);
                const float4 v2 = __ldg(&tp->w2);
                if (bits0 == 0u) {
                    base0 = base1;
                    bits0 = bits1;
                    bits1 = 0u;
                }
                float u = 0.f, v = 0.f;
                const float t = SC::kWatertight ? wt_intersect(v0, v1, v2, o, make_shear(d), u, v)
                                                : mt_intersect(v0, v1, v2, o, d, u, v);
                if (ANY) {
                    if ((__float_as_uint(v2.z) & (RT_TRI_LIGHT | RT_TRI_TRANSPARENT)) == 0u && t > kEpsilon && t < tmax) {
                        occluded = true;
                        group.y = bits0 = bits1 = 0u;
                    }
                } else {
                    const int32_t id = __float_as_int(v2.y);
                    if (t > kEpsilon && (t < hit.t || (t == hit.t && id < hit.id))) {
                        hit.id = id;
                        hit.t = t;
                        hit.u = u;
                        hit.v = v;
                        best = t;
                    }
                }
            }
            continue;
        }
        if (group.y > hit_bits && bits1 == 0u) {
            const uint32_t bit = top_bit(group.y);
            group.y ^= 1u << bit;
            const uint32_t idx = group.x + __popc(group.y & ~(full << ((bit ^ order) & 7u)));
            const bool push = group.y > hit_bits;
            if (idx >= (uint32_t)sc.nnodes || ++steps > kMaxTraversalSteps || (push && sp >= STACK)) {
                status |= idx >= (uint32_t)sc.nnodes      ? kStatusBadIndex
                          : steps > kMaxTraversalSteps ? kStatusStepLimit
                                                       : kStatusStackOverflow;
                group.y = bits0 = 0u;
                sp = 0;
            } else {
                if (push) stack[sp++] = group;
                const NodeHits nh = intersect_node(ANY ? sc.any_nodes : sc.nodes, idx, o, inv, w0, w1, best);
                if (COUNT) ++fc->nodes;
                group = nh.ngroup;
                if (nh.leaf_slots) {
                    uint32_t bits = leaf_triangles(nh);
                    if (bits != 0u && nh.tri_base + top_bit(bits) >= (uint32_t)sc.ntris) {
                        status |= kStatusBadIndex;
                        bits = 0u;
                    }
                    if (bits0 == 0u) {
                        base0 = nh.tri_base;
                        bits0 = bits;
                    } else {
                        base1 = nh.tri_base;
                        bits1 = bits;
                    }
                }
                if (group.y <= hit_bits && sp > 0) group = stack[--sp];
            }
        }
    }
    if (!ANY && hit.id != -1 && (uint32_t)hit.id >= (uint32_t)sc.ntris) {
        status |= kStatusBadIndex;
        hit.id = -1;
        hit.t = FLT_MAX;
    }
    return status;
}

// ------------------------------------------------------------ shading

// ray::offset_start_point(d) (raytracer/ray.h:111-157) for d = +1 (out of
// the surface, dsign 1) or -1 (into it, the refraction start point): each
// coordinate moves by int(+-32 * n * d) units in the last place, or, when
// the coordinate is tiny, to 1e-4 * n whatever d.
__device__ __forceinline__ float offset_coord(float p, float n, float dsign = 1.0f)
{
    uint32_t x = __float_as_uint(p);
    if ((x & 0x7fffffffu) < 0x38d1b717u)   // bit pattern of 1.0e-4f
        return xadd(0.0f, xmul(1.0e-4f, n));
    const float off = ((x >> 31) & 1u) ? -32.0f : 32.0f;
    const float f = xmul(xmul(off, n), dsign);
    int32_t iv;
    if (!(f > -2147483904.0f && f < 2147483648.0f)) iv = INT32_MIN;
    else iv = __float2int_rz(f);
    x += (uint32_t)iv;
    return __uint_as_float(x);
}

__device__ __forceinline__ float3 offset_start(float3 p, float3 n)
{
    return make_float3(offset_coord(p.x, n.x), offset_coord(p.y, n.y), offset_coord(p.z, n.z));
}

__device__ __forceinline__ float3 offset_start_in(float3 p, float3 n)
{
    return make_float3(offset_coord(p.x, n.x, -1.0f), offset_coord(p.y, n.y, -1.0f), offset_coord(p.z, n.z, -1.0f));
}

// Camera ray of pixel (x, y) (camera.h:127-140, EXACT_NORMALISE).
__device__ __forceinline__ RayState camera_ray(const CameraView &cam, int x, int y)
{
    const float x_t = xadd(xmul((float)x, cam.x_inc), cam.x_m);
    const float y_t = xadd(xmul((float)y, cam.y_inc), cam.y_m);
    const float3 screen = xadd3(xadd3(xmul3(cam.X, x_t), xmul3(cam.Y, y_t)), xmul3(cam.Z, cam.t));
    RayState r;
    r.o = cam.c;
    r.d = xnorm(screen);
    return r;
}

struct SurfacePoint {
    float3 dst;       // refined hit point
    float3 sn;        // face-forwarded shading normal
    float3 geo;       // face-forwarded geometric normal
    float3 vt;        // interpolated per-vertex attribute
    bool has_attr;
    bool out_in;      // the ray meets the front face (hit_t::out_in)
};

// Hit refinement and face-forwarding (raytracer.cc:30-31,
// triangle::normal_at_point triangle.h:464-498) and the barycentric
// attribute (triangle.h:74-79).
__device__ __forceinline__ SurfacePoint surface_at(const SceneView &sc, const RayState &r, const HitRecord &h)
{
    SurfacePoint sp;
    const ShadeTri st = sc.shade[h.id];
    const float3 n = make_float3(st.n_cx.x, st.n_cx.y, st.n_cx.z);
    const float3 c = make_float3(st.n_cx.w, st.c_yz.x, st.c_yz.y);
    float3 p = xadd3(r.o, xmul3(r.d, h.t));
    const float denom = xdot(n, r.d);
    const float num = xdot(n, xsub3(c, p));
    p = xadd3(p, xmul3(r.d, xdiv(num, denom)));
    // shading normal: the triangle's corner normals interpolated by the
    // hit's barycentrics when it has them (triangle.h:473-476), else the
    // face normal; both face-forwarded with the face normal's test
    float3 sn = n;
    if (sc.cnorm) {
        const float *cn = sc.cnorm + 9 * (size_t)h.id;
        if (cn[0] != FLT_MAX) {
            const float3 A = make_float3(cn[0], cn[1], cn[2]), B = make_float3(cn[3], cn[4], cn[5]),
                         C = make_float3(cn[6], cn[7], cn[8]);
            const float w = xsub(1.0f, xadd(h.u, h.v));
            sn = xadd3(xadd3(xmul3(C, h.u), xmul3(B, h.v)), xmul3(A, w));
        }
    }
    if (denom > 0.0f) {
        sp.sn = make_float3(-sn.x, -sn.y, -sn.z);
        sp.geo = make_float3(-n.x, -n.y, -n.z);
    } else {
        sp.sn = sn;
        sp.geo = n;
    }
    sp.out_in = !(denom > 0.0f);
    sp.dst = p;
    sp.has_attr = sc.vattr != nullptr;
    if (sp.has_attr) {
        const int3 t = sc.idx[h.id];
        const float3 A = make_float3(sc.vattr[3 * t.x], sc.vattr[3 * t.x + 1], sc.vattr[3 * t.x + 2]);
        const float3 B = make_float3(sc.vattr[3 * t.y], sc.vattr[3 * t.y + 1], sc.vattr[3 * t.y + 2]);
        const float3 C = make_float3(sc.vattr[3 * t.z], sc.vattr[3 * t.z + 1], sc.vattr[3 * t.z + 2]);
        const float w = xsub(1.0f, xadd(h.u, h.v));
        sp.vt = xadd3(xadd3(xmul3(C, h.u), xmul3(B, h.v)), xmul3(A, w));
    } else {
        sp.vt = make_float3(FLT_MAX, FLT_MAX, FLT_MAX);
    }
    return sp;
}

// Diffuse colour (coloured_mapper_shader.cc:61-66 with attribute*255 samples).
__device__ __forceinline__ float3 material_kd(const MaterialView &m, const SurfacePoint &sp)
{
    if (!sp.has_attr || (m.flags & RT_MAT_NO_VERTEX_COLOUR)) return m.kd;
    const float k = 1.0f / 255.0f;
    return make_float3(xmul(xmul(sp.vt.x, 255.0f), xmul(m.kd.x, k)), xmul(xmul(sp.vt.y, 255.0f), xmul(m.kd.y, k)),
                       xmul(xmul(sp.vt.z, 255.0f), xmul(m.kd.z, k)));
}

// Shadow ray towards a light (ray::find_rays ray.cc:91-104,
// light::find_rays light.h:62-100, ray::set_up ray.h:44-54).
__device__ __forceinline__ void shadow_ray(const LightView &L, float3 start, float3 &dir, float &len)
{
    const float3 target = (L.kind == RT_LIGHT_DIRECTIONAL) ? xadd3(start, xmul3(L.dir, L.dist_sign)) : L.pos;
    const float3 dv = xsub3(target, start);
    len = xmag(dv);
    dir = xdiv3(dv, len);
}

// x^n rounded as (float)pow((double)x, (double)n) is, for x > 0.  The double
// power keeps a warp on the SM's few FP64 units.  Whole exponents from 1 to 128
// (specular exponents mostly are) go by squaring in pairs of floats: x = m 2^e
// with m in [0.70, 1.41], so no product of at most 128 m's leaves 2^-65 .. 2^64.
// With u = 2^-24 a product of pairs is off by at most 6.1 u^2 < 2^-45.3 of itself
// (two roundings of the low parts, 2 u^2 and 3 u^2, and the dropped product of
// the tails, u^2), a power of up to 127 products by less than 2^-38.3; 5 M powers
// over all exponents were off by 2^-40.7 at most.  The pair's head is the rounded
// power unless its tail, made larger by 2^-11 of itself (a tail that can matter is
// above 2^-26 of the head), carries the head to a neighbour: those (one in 2000),
// results outside the normal range and other exponents take the double power.
// 512^2 glass frames: ray trees 435 -> 401 us, diffuse sets 12.04 -> 11.17 ms;
// float terrain frames 1369 -> 1360 us, adjoint step 751 -> 738 us.
struct FloatPair { float h, l; };
__device__ __forceinline__ FloatPair pair_mul(FloatPair a, FloatPair b)
{
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    const float h = __fadd_rn(p, e);
    return {h, __fsub_rn(e, __fsub_rn(h, p))};
}
__device__ __forceinline__ float specular_power(float x, float n)
{
    const int k = (int)n;
    if ((float)k == n && k >= 1 && k <= 128 && x > 1.0e-30f && x < 1.0e30f) {
        int e = (int)(__float_as_uint(x) >> 23) - 127;
        float m = __uint_as_float((__float_as_uint(x) & 0x007fffffu) | 0x3f800000u);
        if (m > 1.41f) {
            m = __fmul_rn(m, 0.5f);
            ++e;
        }
        FloatPair b = {m, 0.f}, r = {1.f, 0.f};
        for (int q = k;;) {
            if (q & 1) r = pair_mul(r, b);
            q >>= 1;
            if (!q) break;
            b = pair_mul(b, b);
        }
        const int scale = e * k;
        const int top = (int)((__float_as_uint(r.h) >> 23) & 0xffu) + scale;   // the result's biased exponent
        if (top > 1 && top < 254 && __fadd_rn(r.h, __fmul_rn(r.l, 1.0f + 0x1p-11f)) == r.h)
            return __uint_as_float(__float_as_uint(r.h) + ((uint32_t)scale << 23));
    }
    return (float)pow((double)x, (double)n);
}

// One light's Phong term (coloured_mapper_shader.cc:76-109,
// light::get_light_intensity light.h:44-59) added into c.  EXACT = true
// takes the double power rounded once, the reference's result (specular_power);
// EXACT = false single-precision powf (a few ulp), whose pixels near a
// truncation are shaded again with the exact one.
template <bool EXACT = true>
__device__ __forceinline__ void phong_add(const LightView &L, const MaterialView &m, const float3 kd, const float3 sn,
                                          const float3 view_dir, const float3 ldir, float len, float magn, float3 &c)
{
    const float shade = xdot(ldir, sn);
    if (shade < 0.0f) return;
    const float3 ref = xsub3(ldir, xmul3(sn, xmul(2.0f, shade)));
    const float rdr = xdot(view_dir, ref);
    float3 sc = make_float3(xmul(shade, kd.x), xmul(shade, kd.y), xmul(shade, kd.z));
    if (rdr > 0.0f) {
        const float p = EXACT ? specular_power(rdr, m.ns) : powf(rdr, m.ns);
        sc = make_float3(xadd(sc.x, xmul(p, m.ks.x)), xadd(sc.y, xmul(p, m.ks.y)), xadd(sc.z, xmul(p, m.ks.z)));
    }
    const float dist = xmul(len, L.d);
    const float d_scale = xadd(xmul(dist, dist), 1.0f);
    float3 I;
    if (L.s_b != 0.0f) {
        // spot light: intensity by the angle off its axis (light.h:49-55);
        // the angle always in double, rounded once: divided by a narrow
        // cone width, a few ulp of acosf would not stay within the
        // truncation guard
        const float cosa = xdot(ldir, L.dir);
        const float a = (float)acos((double)cosa);
        const float p = xdiv(xsub(a, L.s_a), xsub(L.s_b, L.s_a));
        const float q = xsub(1.0f, p);
        const float f = (0.0f < ((q < 1.0f) ? q : 1.0f)) ? ((q < 1.0f) ? q : 1.0f) : 0.0f;   // max(0, min(1, q))
        const float fs = xdiv(f, d_scale);
        I = make_float3(xmul(L.rgb255.x, fs), xmul(L.rgb255.y, fs), xmul(L.rgb255.z, fs));
    } else {
        I = make_float3(xdiv(L.rgb255.x, d_scale), xdiv(L.rgb255.y, d_scale), xdiv(L.rgb255.z, d_scale));
    }
    c = make_float3(xadd(c.x, xmul(I.x, xmul(sc.x, magn))), xadd(c.y, xmul(I.y, xmul(sc.y, magn))),
                    xadd(c.z, xmul(I.z, xmul(sc.z, magn))));
}

// camera::clip_image_to_rgb (camera.h:312-314): clamp, then truncate.
__device__ __forceinline__ uint8_t clip8(float v)
{
    return (uint8_t)__float2uint_rz(smin(255.0f, smax(0.0f, xdiv(v, 1.0f))));
}

// The single-precision specular power differs from the exact one by a few
// ulp (<= 1e-6 relative), which moves a colour channel by far less than
// kTruncGuard; only a channel that close to an integer can truncate
// differently.
constexpr float kTruncGuard = 4e-3f;
__device__ __forceinline__ bool near_integer(float v)
{
    const float f = v - floorf(v);
    return f < kTruncGuard || f > 1.0f - kTruncGuard;
}
__device__ __forceinline__ bool near_truncation(float3 c)
{
    return near_integer(c.x) || near_integer(c.y) || near_integer(c.z);
}

// Colour of a hit pixel with the exact specular power, from the stored
// shading inputs and per-light shadow answers (bit l = light l blocked).
__device__ __forceinline__ float3 shade_lights_exact(const LightView *lights, int nl, const MaterialView &mat,
                                                     float3 kd, float3 sn, float3 view_dir, float3 start,
                                                     uint32_t blocked_bits)
{
    float3 c = make_float3(0.f, 0.f, 0.f);
    for (int l = 0; l < nl; ++l) {
        float3 ldir;
        float len;
        shadow_ray(lights[l], start, ldir, len);
        phong_add<true>(lights[l], mat, kd, sn, view_dir, ldir, len, ((blocked_bits >> l) & 1u) ? 0.0f : 1.0f, c);
    }
    return xadd3(c, mat.ka);
}

// ---------------------------------------------------------- AO sampler

// Philox4x32-10 (Salmon et al., SC'11).
__device__ __forceinline__ uint4 philox4x32(uint4 c, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

struct AOBasis {
    float3 T, B, g;
};

// Orthonormal basis of Duff et al. (JCGT 2017), IEEE-exact.
__device__ __forceinline__ AOBasis ao_basis(float3 g)
{
    const float sign = (g.z < 0.0f || (g.z == 0.0f && (__float_as_uint(g.z) >> 31))) ? -1.0f : 1.0f;
    const float a = xdiv(-1.0f, xadd(sign, g.z));
    const float b = xmul(xmul(g.x, g.y), a);
    AOBasis ob;
    ob.T = make_float3(xadd(1.0f, xmul(xmul(sign, xmul(g.x, g.x)), a)), xmul(sign, b), -xmul(sign, g.x));
    ob.B = make_float3(b, xadd(sign, xmul(xmul(g.y, g.y), a)), -g.y);
    ob.g = g;
    return ob;
}

// Direction of AO sample s for a pixel (cosine-weighted by rejection from
// the unit disk, at most 8 tries, lifted to the hemisphere).
__device__ __forceinline__ float3 ao_direction(const AOBasis &ob, uint32_t pixel, uint32_t s, uint32_t seed)
{
    float x = 0.0f, y = 0.0f;
    bool found = false;
    for (uint32_t call = 0; call < 4 && !found; ++call) {
        const uint4 r = philox4x32(make_uint4(pixel, s, call, 0x414f5259u), seed, 0x52415054u);
        const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int pair = 0; pair < 2; ++pair) {
            if (found) break;
            const float px = xsub(xmul((float)(rr[2 * pair] >> 8), 1.1920928955078125e-7f), 1.0f);
            const float py = xsub(xmul((float)(rr[2 * pair + 1] >> 8), 1.1920928955078125e-7f), 1.0f);
            if (xadd(xmul(px, px), xmul(py, py)) < 1.0f) { x = px; y = py; found = true; }
        }
    }
    const float z = __fsqrt_rn(smax(0.0f, xsub(1.0f, xadd(xmul(x, x), xmul(y, y)))));
    const float3 d = xadd3(xadd3(xmul3(ob.T, x), xmul3(ob.B, y)), xmul3(ob.g, z));
    return xnorm(d);
}

}  // namespace rtc
