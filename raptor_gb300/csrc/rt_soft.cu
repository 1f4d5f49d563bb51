// rt_soft.cu -- soft shadows as RAPTor renders them when it is built with
// SOFT_SHADOW = samples: every primary hit sends `samples` shadow rays to
// random points of each spherical (point or spot) or triangle-defined light
// and one to each directional light; a light's term is shaded with its
// first ray's direction and length and weighted by the fraction of rays that
// reach the light (ray::find_rays ray.cc:91-104, light::find_rays
// light.h:62-164, triangle::find_rays triangle.h:504-525,
// ray_trace_engine::ray_trace raytracer.cc:44-64).
//
// The random points come from the reference's own generator, one process-
// wide stream (common/common.cc:35-105) that the reference draws from in
// pixel order (x + y * xres) and, within a pixel, in light order: three
// numbers per ray of a spherical light, two per ray a triangle-defined
// light makes.  A pixel's position in that stream
// is therefore fixed by how many pixels before it hit something, so a frame
// is rendered in two passes: the camera rays first (hit records kept, one
// flag per pixel), an exclusive scan of the flags (each hit draws the same
// count), the frame's slice of the stream generated on the device (k_ref_jump,
// k_ref_stream: blocks walk the generator's states from points a jump apart), then
// the shading pass, every pixel reading its own slice.
// The cosine table the offsets go through (common/common.h:171-209) is
// built on the host the same way and kept on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include <cub/cub.cuh>

#include "rt_api_internal.cuh"
#include "rt_shade.cuh"

namespace rtc {

constexpr float kRefPi = 3.1415926535897932384626433f;   // common/common.cc:10
constexpr int kCosLutSize = 16384;                          // COS_LUT_SIZE, common/common.h:109-111

namespace {

// The reference's generator: a Mersenne twister of kMtWords words seeded with
// 5489 whose refill updates words 0..622 only, its words tempered and scaled
// to [0, 1] in binary32.  Number p is word p % 624 of the state after refill
// p / 624 (counted from 0), so the stream is kept as those states' words;
// ref_number tempers one where it is read.
constexpr int kMtWords = 624;

__device__ __forceinline__ float ref_number(uint32_t y)
{
    y ^= (y >> 11);
    y ^= ((y << 7) & 0x9d2c5680u);
    y ^= ((y << 15) & 0xefc60000u);
    y ^= (y >> 18);
    return xmul(__uint2float_rn(y), 1.0f / 4294967296.0f);
}

__device__ __forceinline__ uint32_t mt_twist(uint32_t a, uint32_t b)
{
    const uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
    return (y >> 1) ^ ((uint32_t)((int32_t)(b << 31) >> 31) & 0x9908b0dfu);
}

// Refills follow one another, so what counts is the latency of one.  A new word
// i needs old words i and i + 1 and word i + 397, which for i >= 227 is the new
// word i - 227: thread t takes words t, t + 227 and t + 454, so those chains stay
// inside a thread and a refill is one exchange of the old words through shared
// memory (two buffers, one barrier).  130 ns a refill with output, 85 without (138
// and 110 with branches around the idle threads' work; 177 on four warps of two
// words per third; a host core takes 350).
constexpr int kMtThreads = 256;
constexpr int kMtThird = kMtWords - 1 - 2 * 227;   // words 454..622
constexpr int kMtBuffer = 1024;                    // idle threads read past the words
template <bool OUT>
__device__ __forceinline__ void mt_refill(uint32_t *w, int t, int t3, bool on, bool third, uint32_t &a, uint32_t &b,
                                          uint32_t &c, uint32_t *dst)
{
    if (on) {
        w[t] = a;
        w[t + 227] = b;
    }
    if (third) w[t + 454] = c;
    __syncthreads();
    const uint32_t far = w[t + 397];
    const uint32_t fa = mt_twist(a, w[t + 1]), fb = mt_twist(b, w[t + 228]), fc = mt_twist(c, w[t3 + 455]);
    const uint32_t fbc = fb ^ fc;
    a = far ^ fa;
    b = far ^ fa ^ fb;
    c = far ^ fa ^ fbc;
    if (OUT) {
        if (on) {
            dst[t] = a;
            dst[t + 227] = b;
        }
        if (third) dst[t + 454] = c;
    }
}

// `refills` refills of a state whose words are a (t), b (t + 227), c (t + 454)
// and `last`; OUT: the words after each go to out.
template <bool OUT>
__device__ __forceinline__ void mt_refills(uint32_t *words, int32_t refills, uint32_t &a, uint32_t &b, uint32_t &c,
                                           uint32_t last, uint32_t *out)
{
    const int t = threadIdx.x;
    const bool on = t < 227, third = t < kMtThird;
    const int t3 = third ? t : kMtThird - 1;
    for (int i = t; i < 2 * kMtBuffer; i += kMtThreads) words[i] = 0u;
    __syncthreads();
    if (t < 2) words[t * kMtBuffer + kMtWords - 1] = last;
    uint32_t *dst = out;
    int32_t r = 0;
    for (; r + 1 < refills; r += 2) {
        mt_refill<OUT>(words, t, t3, on, third, a, b, c, dst);
        if (OUT) dst += kMtWords;
        mt_refill<OUT>(words + kMtBuffer, t, t3, on, third, a, b, c, dst);
        if (OUT) dst += kMtWords;
    }
    if (r < refills) mt_refill<OUT>(words, t, t3, on, third, a, b, c, dst);
    if (OUT)
        for (int32_t i = t; i < refills; i += kMtThreads) out[(size_t)i * kMtWords + kMtWords - 1] = last;
}

// `total` refills, `each` of them to a block, block k from state starts + k * kMtWords
// on; the words after every one to out (OUT), the state after the last to end.
template <bool OUT>
__global__ void __launch_bounds__(kMtThreads) k_ref_stream(const uint32_t *starts, int64_t total, int32_t each,
                                                           uint32_t *__restrict__ out, uint32_t *end)
{
    __shared__ uint32_t words[2 * kMtBuffer];
    const int t = threadIdx.x;
    const bool on = t < 227, third = t < kMtThird;
    const uint32_t *state = starts + (size_t)blockIdx.x * kMtWords;
    const int64_t first = (int64_t)blockIdx.x * each;
    uint32_t a = state[on ? t : 0], b = state[on ? t + 227 : 0], c = state[third ? t + 454 : kMtWords - 2];
    const uint32_t last = state[kMtWords - 1];
    mt_refills<OUT>(words, (int32_t)min((int64_t)each, total - first), a, b, c, last,
                    OUT ? out + (size_t)first * kMtWords : nullptr);
    if (first + each < total) return;
    if (on) {
        end[t] = a;
        end[t + 227] = b;
    }
    if (third) end[t + 454] = c;
    if (t == 0) end[kMtWords - 1] = last;
}

// A refill is linear over GF(2) in the state's bits (the twist is, and word 623
// stays), so kJump refills are one bit matrix.  Its column j, the state that
// kJump refills make of bit j alone, is walked by block j.
// With it the states kJump refills apart follow one another by one product each
// (k_ref_jump, 4 us) and a block walks the refills after each (k_ref_stream): 52,000
// refills, a 900p frame's of 16 samples, take 0.47 ms where one block takes 6.8, and
// 3,400 of a 320x200 frame 85 us for 440.  50 MB and 3 ms, made once a context has
// walked as long (kJumpWorth).  Jumps of 1024: 0.32 ms, 150 us, 6 ms to make; of 256
// 0.85 ms, 85 us.
constexpr int kJump = 512;
constexpr int kMtBits = kMtWords * 32;
__global__ void __launch_bounds__(kMtThreads) k_ref_matrix(uint32_t *__restrict__ columns)
{
    __shared__ uint32_t words[2 * kMtBuffer];
    const int t = threadIdx.x, j = blockIdx.x;
    const uint32_t bit = 1u << (j & 31);
    const int w = j >> 5;
    uint32_t a = w == t ? bit : 0u, b = w == t + 227 ? bit : 0u, c = w == t + 454 ? bit : 0u;
    const uint32_t last = w == kMtWords - 1 ? bit : 0u;
    mt_refills<false>(words, kJump, a, b, c, last, nullptr);
    uint32_t *col = columns + (size_t)j * kMtWords;
    if (t < 227) {
        col[t] = a;
        col[t + 227] = b;
    }
    if (t < kMtThird) col[t + 454] = c;
    if (t == 0) col[kMtWords - 1] = last;
}

// One jump, its state's words shared out over kJumpBlocks blocks, four each: a
// block puts its words of the state together -- from `state`, or from the parts
// that the blocks of the jump before made of theirs -- and stores them in `at`;
// then (product) its part of the next state is the sum of the columns of their
// set bits.  What counts is the latency of a jump, so all of a block's columns
// (half of 128, 16 bytes a thread) are in flight at once; together the blocks
// read half of the matrix, out of the L2, and a launch is ready while the one
// before ends: 4 us a jump (10 without any of it in the caches).
constexpr int kJumpBlocks = kMtWords / 4;
constexpr int kJumpLanes = 160;                    // a group's threads: one for four words of a column
constexpr int kJumpThreads = 4 * kJumpLanes;       // four groups, for a word's bits each
__global__ void __launch_bounds__(kJumpThreads) k_ref_jump(const uint4 *__restrict__ columns, const uint4 *state,
                                                           const uint4 *parts, uint4 *next, uint4 *at, bool product)
{
    __shared__ uint4 s_part[kJumpThreads / 32];
    __shared__ uint32_t s_word[4];
    __shared__ uint4 s_sum[3][kJumpBlocks];
    const auto add = [](uint4 p, uint4 q) { return make_uint4(p.x ^ q.x, p.y ^ q.y, p.z ^ q.z, p.w ^ q.w); };
    const int t = threadIdx.x, b = blockIdx.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint4 mine = make_uint4(0u, 0u, 0u, 0u);
    if (state) {
        if (t == 0) mine = state[b];
    } else if (t < kJumpBlocks) {
        mine = __ldcg(parts + (size_t)t * kJumpBlocks + b);
    }
    for (int o = 16; o > 0; o >>= 1)
        mine = add(mine, make_uint4(__shfl_xor_sync(0xffffffffu, mine.x, o), __shfl_xor_sync(0xffffffffu, mine.y, o),
                                    __shfl_xor_sync(0xffffffffu, mine.z, o), __shfl_xor_sync(0xffffffffu, mine.w, o)));
    if ((t & 31) == 0) s_part[t >> 5] = mine;
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < kJumpLanes / 32; ++w) mine = add(mine, s_part[w]);
        at[b] = mine;
        s_word[0] = mine.x;
        s_word[1] = mine.y;
        s_word[2] = mine.z;
        s_word[3] = mine.w;
    }
    __syncthreads();
    if (!product) return;
    const int group = t / kJumpLanes, lane = t % kJumpLanes;
    const uint32_t bits = s_word[group];
    uint4 sum = make_uint4(0u, 0u, 0u, 0u);
    if (lane < kJumpBlocks) {
        const uint4 *col = columns + (size_t)(128 * b + 32 * group) * kJumpBlocks + lane;
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if ((bits >> j) & 1u) sum = add(sum, __ldg(col + (size_t)j * kJumpBlocks));
        if (group > 0) s_sum[group - 1][lane] = sum;
    }
    __syncthreads();
    if (group == 0 && lane < kJumpBlocks)
        next[(size_t)b * kJumpBlocks + lane] = add(add(sum, s_sum[0][lane]), add(s_sum[1][lane], s_sum[2][lane]));
}

// The rays light::find_rays makes for a triangle-defined light of ntris
// triangles asked for n (light.h:129-164): n / ntris per triangle, one more
// for every triangle the binary32 stride lands on.  cnt (ntris entries,
// nullable) receives the counts; returns their sum.
int32_t area_light_rays(int32_t ntris, int32_t n, int32_t *cnt)
{
    const int32_t ppt = n / ntris;
    const int32_t extra = n - ntris * ppt;
    const float stride = (float)ntris / (float)std::max(extra, 1);
    float at = 0.0f;
    int32_t made = 0;
    for (int32_t j = 0; j < ntris; ++j) {
        int32_t k = ppt;
        if (j == (int32_t)at) {
            ++k;
            at += stride;
        }
        if (cnt) cnt[j] = k;
        made += k;
    }
    return made;
}

}  // namespace

// Per-context state of the soft-shadow path.
struct SoftState {
    DevBuf lut;                  // the cosine table
    bool lut_ready = false;
    DevBuf hits;                 // int4 per pixel: the primary hit record
    DevBuf flags, prefix;        // int per pixel: hit flag, exclusive scan of the flags
    DevBuf scan_temp;
    DevBuf area;                 // int4 per ray of a triangle-defined light: triangle, its rays, index
    DevBuf counts, prefix64;     // int64 per pixel: numbers a distributed pixel draws, their exclusive scan
    DevBuf scan64_temp;
    // distributed frames on per-pixel streams: each pixel's camera-ray node
    // (colour, material; first item, set sizes), the items (its sets' rays),
    // their subtrees' colours, the item count
    DevBuf root_c, root_sets, items, item_c, nitems;
    DevBuf nodes, node_sets, node_hits, node_over;   // nodes below them, their children, hit nodes, nodes walked whole
    int64_t item_cap = 0;
    // The stream's words on the device, in two windows: words that a window has
    // no more room behind go on in the other.  refills counts what the
    // generator's state has behind it (-1: to be seeded).
    struct Window {
        DevBuf words;
        int64_t first = 0, count = 0;      // refills [first, first + count)
    } win[2];
    int cur = 0;                           // the window the last frame read
    DevBuf rng;                            // the generator's state, then the seeded one
    int64_t refills = -1;
    DevBuf jump;                           // the jump's matrix, the states of a row of jumps, their parts
    bool jump_ready = false;
    int64_t walked = 0;                    // refills walked one after another
    int device = 0;
};

void soft_release(rt_context *ctx)
{
    if (!ctx->soft) return;
    SoftState &S = *ctx->soft;
    for (SoftState::Window &w : S.win) w.words.release();
    S.rng.release();
    S.jump.release();
    S.lut.release();
    S.hits.release();
    S.flags.release();
    S.prefix.release();
    S.scan_temp.release();
    S.area.release();
    S.counts.release();
    S.prefix64.release();
    S.scan64_temp.release();
    S.root_c.release();
    S.root_sets.release();
    S.items.release();
    S.item_c.release();
    S.nitems.release();
    S.nodes.release();
    S.node_sets.release();
    S.node_hits.release();
    S.node_over.release();
    delete ctx->soft;
    ctx->soft = nullptr;
}

namespace {

// static_cos::get_cos / get_sin (common/common.h:186-198): the index
// truncates toward zero and wraps modulo the table size (how the unsigned
// conversion of a negative angle behaves on the reference's x86-64 build).
__device__ __forceinline__ float lut_cos(const float *__restrict__ lut, float a)
{
    const float k = xmul(xdiv(1.0f, xmul(2.0f, kRefPi)), (float)kCosLutSize);
    const float v = xmul(k, a);
    long long e = 0;
    if (v > -9.2e18f && v < 9.2e18f) e = __float2ll_rz(v);
    return __ldg(lut + ((uint32_t)e & (uint32_t)(kCosLutSize - 1)));
}
__device__ __forceinline__ float lut_sin(const float *__restrict__ lut, float a)
{
    return lut_cos(lut, xsub(a, xdiv(kRefPi, 2.0f)));
}

// Shadow ray i of n to spherical light L: a random offset of the light's
// centre from the numbers u0, u1, u2 (light.h:102-128), then
// ray::set_up(start, centre + offset) (ray.h:44-54).
__device__ __forceinline__ void soft_ray(const LightView &L, const float *__restrict__ lut, float3 start, int n,
                                         int i, float u0, float u1, float u2, float3 &dir, float &len)
{
    const float a_scale = xdiv(1.0f, (float)((n >> 4) + ((n & 0xe) != 0) + 1));
    const float b_scale = xdiv(1.0f, (float)((n >> 4) + ((n & 0xc) != 0) + 1));
    const float r_scale = xdiv(1.0f, (float)((n >> 4) + ((n & 0x8) != 0) + 1));
    const int eighths = (i >> 2) & ~0x1;
    const float two_pi = xmul(2.0f, kRefPi);
    const float a_off = xmul(xmul(u0, xmul(a_scale, (float)(eighths + (i & 0x1)))), two_pi);
    const float b_off = xmul(xmul(u1, xmul(b_scale, (float)(eighths + (i & 0x2)))), two_pi);
    const float r_off = xmul(xmul(u2, xmul(r_scale, (float)(eighths + (i & 0x4)))), L.radius);
    const float sin_a = lut_sin(lut, a_off), cos_a = lut_cos(lut, a_off);
    const float sin_b = lut_sin(lut, b_off), cos_b = lut_cos(lut, b_off);
    const float3 off = make_float3(xmul(xmul(r_off, cos_a), sin_b), xmul(xmul(r_off, sin_a), sin_b), xmul(r_off, cos_b));
    const float3 dv = xsub3(xadd3(L.pos, off), start);
    len = xmag(dv);
    dir = xdiv3(dv, len);
}

// Shadow ray to triangle-defined light point e = (triangle, rays it makes,
// index of this one): barycentrics from the numbers u0, u1
// (triangle.h:504-525), then ray::set_up(start, point).
__device__ __forceinline__ void area_ray(const float *__restrict__ verts, const int3 *__restrict__ idx, int4 e,
                                         float3 start, float u0, float u1, float3 &dir, float &len)
{
    const int n = e.y, i = e.z;
    const float beta_scale = xdiv(1.0f, (float)((n >> 4) + ((n & 0xe) != 0) + 1));
    const float gamma_scale = xdiv(1.0f, (float)((n >> 4) + ((n & 0xc) != 0) + 1));
    const int eighths = (i >> 2) & ~0x1;
    const float beta = xmul(u0, xmul(beta_scale, (float)(eighths + (i & 0x1))));
    const float gamma = xmul(xmul(u1, xmul(gamma_scale, (float)(eighths + (i & 0x2)))), xsub(1.0f, beta));
    const float alpha = xsub(1.0f, xadd(beta, gamma));
    const int3 t = idx[e.x];
    const float3 a = make_float3(__ldg(verts + 3 * t.x), __ldg(verts + 3 * t.x + 1), __ldg(verts + 3 * t.x + 2));
    const float3 b = make_float3(__ldg(verts + 3 * t.y), __ldg(verts + 3 * t.y + 1), __ldg(verts + 3 * t.y + 2));
    const float3 c = make_float3(__ldg(verts + 3 * t.z), __ldg(verts + 3 * t.z + 1), __ldg(verts + 3 * t.z + 2));
    const float3 p = xadd3(xadd3(xmul3(a, alpha), xmul3(b, beta)), xmul3(c, gamma));
    const float3 dv = xsub3(p, start);
    len = xmag(dv);
    dir = xdiv3(dv, len);
}

__device__ __forceinline__ bool soft_light(const LightView &L, int samples)
{
    return samples > 1 && L.kind != RT_LIGHT_DIRECTIONAL;
}

// Per light: first entry of its rays in the ray table and the rays it
// makes (0: not triangle-defined); numbers a hit draws for it.
struct AreaSet {
    int32_t first[RT_MAX_LIGHTS];
    int32_t made[RT_MAX_LIGHTS];
    int32_t draws[RT_MAX_LIGHTS];
};

// Pass 1: the camera ray of every pixel; hit record and hit flag.
template <class SC>
__global__ void __launch_bounds__(kTraceThreads, 6) k_soft_primary(SC sc, CameraView cam,
                                                                                      int4 *__restrict__ hits,
                                                                                      int32_t *__restrict__ flags,
                                                                                      Counters *ctr)
{
    int tiles_x;
    const int items = tiles_of<8>(cam.xres, cam.yres, tiles_x) * 32;
    uint32_t status = 0;
    for (;;) {
        const int base = warp_claim(&ctr->work, 32);
        if (base >= items) break;
        int x, y;
        tile_pixel<8>(base + (threadIdx.x & 31), tiles_x, x, y);
        const bool live = (x < cam.xres) && (y < cam.yres);
        bool hit = false;
        const RayState r = camera_ray(cam, x, y);
        HitRecord h;
        bool occ;
        status |= traverse_warp<false>(sc, live, r.o, r.d, FLT_MAX, h, occ);
        if (live) {
            hit = h.t < FLT_MAX;
            const size_t pix = (size_t)x + (size_t)y * (size_t)cam.xres;
            hits[pix] = make_int4(h.id, __float_as_int(h.t), __float_as_int(h.u), __float_as_int(h.v));
            flags[pix] = hit ? 1 : 0;
        }
        warp_count(&ctr->primary, live);
        warp_count(&ctr->hits, hit);
    }
    if (status) atomicOr(&ctr->status, status);
}

// The rays from a warp's hits to one light: `n` from the lane's `start` (0: the
// lane has no hit).  32 at a time in the hits' order: the rays of one hit, which
// leave one point for one light, are on neighbouring lanes, and trace in step.
// fetch(own): what the rays of lane own's hit need (called converged);
// make(data, sample, start, dir, len): one of them.  Out: the rays that arrive,
// direction and length of the first.
// Against a ray of every hit at a time: k_soft_shade on 900p terrain, 16 samples,
// 2.27 -> 1.92 ms (27.5 lanes an instruction); k_dist_lights 13.9 -> 11.7 ms
// (11.0 -> 17.0 lanes) on the 512x512 glass frame with diffuse sets.
template <class SC, class Fetch, class Make>
__device__ __forceinline__ void trace_hit_rays(const SC &sc, const float3 start, int n, Fetch fetch, Make make,
                                               float3 &ldir, float &len, int &made, uint32_t &status)
{
    const int lane = (int)(threadIdx.x & 31u);
    int end = n;                    // the hit's rays are [first, end) of the warp's
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += t;
    }
    const int first = end - n, total = __shfl_sync(0xffffffffu, end, 31);
    made = 0;
    for (int at = 0; at < total; at += 32) {
        const int r = at + lane;
        int own = 0;                // the hit of ray r: hits whose rays end at or before it
        for (int o = 16; o > 0; o >>= 1)
            if (__shfl_sync(0xffffffffu, end, own + o - 1) <= r) own += o;
        const bool ray = r < total;
        const float3 rs = make_float3(__shfl_sync(0xffffffffu, start.x, own), __shfl_sync(0xffffffffu, start.y, own),
                                      __shfl_sync(0xffffffffu, start.z, own));
        const int sample = r - __shfl_sync(0xffffffffu, first, own);
        const auto data = fetch(own);
        float3 di = rs;
        float li = 0.f;
        if (ray) make(data, sample, rs, di, li);
        HitRecord sh;
        bool blocked;
        status |= traverse_warp<true>(sc, ray, rs, di, li, sh, blocked);
        const uint32_t lit = __ballot_sync(0xffffffffu, ray && !blocked);
        const int lo = max(first - at, 0), hi = min(end - at, 32);   // the hit's lanes
        if (lo < hi) made += __popc(lit & (0xffffffffu >> (32 - (hi - lo)) << lo));
        const int from = (first - at) & 31;
        const float3 d0 = make_float3(__shfl_sync(0xffffffffu, di.x, from), __shfl_sync(0xffffffffu, di.y, from),
                                      __shfl_sync(0xffffffffu, di.z, from));
        const float l0 = __shfl_sync(0xffffffffu, li, from);
        if (n > 0 && first >= at && first < at + 32) {
            ldir = d0;
            len = l0;
        }
    }
}

// Pass 2: shading.  rnd holds the frame's numbers (rnd[0] = the frame's
// first), nrnd of them; a hit pixel's first is prefix[pix] * per_hit.
// 6 blocks an SM for the camera rays and 7 here: a 900p frame's kernels 2.33 -> 2.27 ms
// (8 and 8; 5 and 5: 2.34).
template <class SC>
__global__ void __launch_bounds__(kTraceThreads, 7) k_soft_shade(
    SC sc, CameraView cam, LightSet lights, MaterialTable table, AreaSet areas, const int4 *__restrict__ area,
    const float *__restrict__ verts, int32_t samples, int32_t per_hit, const uint32_t *__restrict__ rnd, int64_t nrnd,
    const float *__restrict__ lut, const int4 *__restrict__ hits, const int32_t *__restrict__ prefix,
    uint8_t *__restrict__ rgb, float *__restrict__ fimg, Counters *ctr)
{
    int tiles_x;
    const int items = tiles_of<8>(cam.xres, cam.yres, tiles_x) * 32;
    uint32_t status = 0;
    for (;;) {
        const int base = warp_claim(&ctr->work, 32);
        if (base >= items) break;
        int x, y;
        tile_pixel<8>(base + (threadIdx.x & 31), tiles_x, x, y);
        const bool live = (x < cam.xres) && (y < cam.yres);
        // every lane goes through the lights and their rays, so that the warp's
        // rays to one light are traced in step
        uint32_t nsec = 0;
        const size_t pix = (size_t)x + (size_t)y * (size_t)cam.xres;
        HitRecord h;
        h.t = FLT_MAX;
        if (live) {
            const int4 hr = hits[pix];
            h.id = hr.x;
            h.t = __int_as_float(hr.y);
            h.u = __int_as_float(hr.z);
            h.v = __int_as_float(hr.w);
        }
        bool on = h.t < FLT_MAX;   // false from here on for a lane that leaves the lights' loop
        const bool hit = on;
        const RayState r = camera_ray(cam, x, y);
        SurfacePoint sp;
        float3 start = r.o, kd = r.o, c = make_float3(0.f, 0.f, 0.f);
        int32_t mi = 0;
        int64_t draw = 0;
        if (hit) {
            if (sc.mat) {
                mi = __ldg(&sc.mat[h.id - sc.tri_base]);
                if (mi < 0 || mi >= table.n) { status |= kStatusBadIndex; mi = 0; }
            }
            sp = surface_at(sc, r, h);
            start = offset_start(sp.dst, sp.geo);
            kd = material_kd(table.m[mi], sp);
            draw = (int64_t)prefix[pix] * per_hit;
        }
        const MaterialView &mat = table.m[mi];
        const int nl = __any_sync(0xffffffffu, on) ? lights.n : 0;
        for (int l = 0; l < nl; ++l) {
            const LightView &L = lights.l[l];
            float3 ldir = r.d;
            float len = 0.f;
            int n = 1, made = 0;
            if (soft_light(L, samples)) {
                n = samples;
                if (on && draw + (int64_t)areas.draws[l] > nrnd) {   // never expected: the host sized the slice
                    status |= kStatusBadIndex;
                    on = false;
                }
                const bool tri_light = areas.made[l] > 0;
                trace_hit_rays(
                    sc, start, on ? n : 0, [&](int own) { return __shfl_sync(0xffffffffu, draw, own); },
                    [&](int64_t at, int i, float3 from, float3 &di, float &li) {
                        const uint32_t *u = rnd + at + (tri_light ? 2 : 3) * i;
                        const float u0 = ref_number(__ldg(u)), u1 = ref_number(__ldg(u + 1));
                        if (tri_light)
                            area_ray(verts, sc.idx, __ldg(area + areas.first[l] + i), from, u0, u1, di, li);
                        else
                            soft_ray(L, lut, from, n, i, u0, u1, ref_number(__ldg(u + 2)), di, li);
                    },
                    ldir, len, made, status);
                draw += areas.draws[l];
            } else {
                if (on) shadow_ray(L, start, ldir, len);
                HitRecord sh;
                bool blocked;
                status |= traverse_warp<true>(sc, on, start, ldir, len, sh, blocked);
                made = blocked ? 0 : 1;
            }
            if (on) {
                nsec += (uint32_t)n;
                // made_it / nr_pending_shadows, both floats (raytracer.cc:46-61)
                phong_add<true>(L, mat, kd, sp.sn, r.d, ldir, len, xdiv((float)made, (float)n), c);
            }
        }
        if (live) {
            c = hit ? xadd3(c, mat.ka) : cam.background;
            if (rgb) store_rgb(rgb, pix, c);
            if (fimg) {
                fimg[3 * pix] = c.x;
                fimg[3 * pix + 1] = c.y;
                fimg[3 * pix + 2] = c.z;
            }
        }
        warp_add(&ctr->secondary, nsec);
    }
    if (status) atomicOr(&ctr->status, status);
}

// ------------------------------------------------ distributed ray tracing

// Frames of a pixel's ray tree: one per level below the camera ray.
constexpr int kDistDepth = RT_MAX_BOUNCES + 1;
// Componant levels with their own counts: componant 4^k for k < 4; with
// at most 64 samples every count max(samples / 4^k, 1) is 1 from k = 3 on.
constexpr int kDistLevels = 4;

// Per light and componant level: the first entry of the light's rays in
// the ray table and the rays it makes (0: not triangle-defined), and the
// numbers one hit draws for it.
struct DistLights {
    int32_t first[RT_MAX_LIGHTS][kDistLevels];
    int32_t made[RT_MAX_LIGHTS][kDistLevels];
    int32_t draws[RT_MAX_LIGHTS][kDistLevels];
};

struct DistParams {
    int32_t soft, diffuse;
    int32_t pixel_stream;        // 1: per-pixel Philox streams; 0: the frame's slice of the reference's
    uint32_t key0, key1;
    int32_t max_steps;           // frame visits per pixel (bounded by the tree's worst case)
    float rfd[RT_MAX_MATERIALS];
    float td[RT_MAX_MATERIALS];
};

// Tree nodes of a pixel's per-pixel streams: the camera ray is kTreeRoot;
// ray `index` of a node's reflection (set 0) or refraction (set 1) set is
// SplitMix64 (Steele, Lea and Flood 2014) of node + (64 set + index + 1) *
// 0x9E3779B97F4A7C15.
constexpr uint64_t kTreeRoot = 0x6A09E667F3BCC909ull;
__device__ __forceinline__ uint64_t tree_child(uint64_t parent, int set, int index)
{
    uint64_t z = parent + (uint64_t)(set * 64 + index + 1) * 0x9E3779B97F4A7C15ull + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// A pixel's random numbers: number k that tree node `node` draws from the
// pixel's Philox streams (counter (pixel, node low, node high, k / 4)), or
// number base + k of the frame's slice of the reference's stream (k the
// pixel's running index; node unused).
struct DistStream {
    const uint32_t *win;
    int64_t base, nwin;
    uint32_t pixel, key0, key1;
    bool pixel_mode;
    uint32_t blk;                // last Philox block computed, and its node
    uint64_t bnode;
    uint4 w;

    __device__ __forceinline__ float at(uint64_t node, uint32_t k, uint32_t &status)
    {
        if (pixel_mode) {
            if ((k >> 2) != blk || node != bnode) {
                blk = k >> 2;
                bnode = node;
                w = philox4x32(make_uint4(pixel, (uint32_t)node, (uint32_t)(node >> 32), blk), key0, key1);
            }
            const uint32_t u = (k & 3u) == 0u ? w.x : (k & 3u) == 1u ? w.y : (k & 3u) == 2u ? w.z : w.w;
            return xmul(__uint2float_rn(u), 2.3283064365386963e-10f);
        }
        const int64_t i = base + (int64_t)k;
        if (i < 0 || i >= nwin) {   // never expected: the host sized the slice
            status |= kStatusBadIndex;
            return 0.0f;
        }
        return ref_number(__ldg(win + i));
    }
};

// One ray of a diffuse set about direction ref (ray::reflect
// ray.cc:137-182, ray::refract ray.cc:236-280): ref + perpen * r cos a +
// cross * r sin a, with perpen = (ref.z, ref.y, -ref.x), cross = ref x
// perpen, r = spread * u0, a = 2 pi * u1 through the cosine table; the
// direction is not normalised.
__device__ __forceinline__ float3 spread_dir(float3 ref, float spread, float u0, float u1, const float *__restrict__ lut)
{
    const float3 perpen = make_float3(ref.z, ref.y, -ref.x);
    const float3 cr = xcross(ref, perpen);
    const float r_off = xmul(u0, spread);
    const float a_off = xmul(u1, xmul(2.0f, kRefPi));
    const float x_off = xmul(r_off, lut_cos(lut, a_off));
    const float y_off = xmul(r_off, lut_sin(lut, a_off));
    return xadd3(xadd3(ref, xmul3(perpen, x_off)), xmul3(cr, y_off));
}

struct DistFrame {
    float3 o;            // the ray's origin; after its hit, the refined hit point
    float3 d;            // its direction
    float3 sn, geo;      // shading and geometric normal at the hit
    float3 c;            // its colour: the lights and ka, then the sets' means
    float3 sum;          // colours of the current set's rays so far
    float magn;          // power
    int32_t level;       // componant 4^level
    uint64_t node;       // its tree node (per-pixel streams)
    int32_t mat;
    int32_t stage;
    int32_t out_in;
    int32_t nrefl, nrefr, child;
    uint32_t refl_at, refr_at;   // the pixel's number index of each set's first number
};

enum : int32_t { kDistTrace = 0, kDistRefl = 1, kDistRefr = 2, kDistDone = 3, kDistLights = 4 };

__device__ __forceinline__ int dist_count(int32_t samples, int32_t level)
{
    return max(samples >> (2 * min(level, kDistLevels - 1)), 1);
}

// Child ray i of frame f's reflection (set 0: ray::reflect ray.cc:118-182,
// power magn * rf) or refraction (set 1: ray::refract ray.cc:198-281, power
// magn * tran, ri inverted for a ray entering the front face, start point
// pushed into the surface) set, its direction spread by the set's numbers
// when the material spreads it.
__device__ __forceinline__ void spawn_child(const DistFrame &f, const MaterialView &m, const DistParams &dp, int set,
                                            int i, const float *__restrict__ lut, DistStream &S, uint32_t &status,
                                            DistFrame &C)
{
    if (set == 0) {
        const bool spread = dp.diffuse > 0 && dp.rfd[f.mat] != 0.0f;
        const float rdn = xmul(2.0f, xdot(f.d, f.sn));
        const float3 ref = xsub3(f.d, xmul3(f.sn, rdn));
        if (spread) {
            const uint32_t at = f.refl_at + 2u * (uint32_t)i;
            C.d = spread_dir(ref, dp.rfd[f.mat], S.at(f.node, at, status), S.at(f.node, at + 1, status), lut);
        } else {
            C.d = ref;
        }
        C.o = offset_start(f.o, f.geo);
        C.magn = xmul(f.magn, m.rf);
        C.level = f.level + (spread ? 1 : 0);
    } else {
        const bool spread = dp.diffuse > 0 && dp.td[f.mat] != 0.0f;
        float ri = m.ri;
        const float rdn = -xdot(f.d, f.sn);
        if (f.out_in) ri = xdiv(1.0f, ri);
        const float cos_t2 = xsub(1.0f, xmul(xmul(ri, ri), xsub(1.0f, xmul(rdn, rdn))));
        const float off = xsub(xmul(ri, rdn), __fsqrt_rn(cos_t2));
        const float3 ref = xadd3(xmul3(f.d, ri), xmul3(f.sn, off));
        if (spread) {
            const uint32_t at = f.refr_at + 2u * (uint32_t)i;
            C.d = spread_dir(ref, dp.td[f.mat], S.at(f.node, at, status), S.at(f.node, at + 1, status), lut);
        } else {
            C.d = ref;
        }
        C.o = offset_start_in(f.o, f.geo);
        C.magn = xmul(f.magn, m.tran);
        C.level = f.level + (spread ? 1 : 0);
    }
    C.node = tree_child(f.node, set, i);
    C.stage = kDistTrace;
}

// Ray `sample` of light l's n at a hit whose numbers for the light start at kb.
__device__ __forceinline__ void dist_light_ray(const LightSet &lights, const DistLights &dl,
                                               const int4 *__restrict__ area, const float *__restrict__ verts,
                                               const int3 *__restrict__ idx, const float *__restrict__ lut,
                                               DistStream &S, uint64_t node, int l, int lvl, int n, int sample,
                                               uint32_t kb, float3 start, float3 &di, float &li, uint32_t &status)
{
    const LightView &L = lights.l[l];
    if (n == 1) {
        shadow_ray(L, start, di, li);
    } else if (dl.made[l][lvl] > 0) {
        const float u0 = S.at(node, kb + 2 * sample, status);
        const float u1 = S.at(node, kb + 2 * sample + 1, status);
        area_ray(verts, idx, __ldg(area + dl.first[l][lvl] + sample), start, u0, u1, di, li);
    } else {
        const float u0 = S.at(node, kb + 3 * sample, status);
        const float u1 = S.at(node, kb + 3 * sample + 1, status);
        const float u2 = S.at(node, kb + 3 * sample + 2, status);
        soft_ray(L, lut, start, n, sample, u0, u1, u2, di, li);
    }
}

// The sets of a shaded node (f.nrefl, f.nrefr rays; 0 on entry), their
// numbers from kb on, past the lights'.
__device__ __forceinline__ void dist_sets(DistFrame &f, const MaterialView &m, const DistParams &dp, uint32_t &kb)
{
    if ((double)xmul(f.magn, m.rf) > 0.1) {
        if (dp.diffuse > 0 && dp.rfd[f.mat] != 0.0f) {
            f.nrefl = dist_count(dp.diffuse, f.level);
            f.refl_at = kb;
            kb += 2u * (uint32_t)f.nrefl;
        } else {
            f.nrefl = 1;
        }
    }
    if ((double)xmul(f.magn, m.tran) > 0.1) {
        float ri = m.ri;
        const float rdn = -xdot(f.d, f.sn);
        if (f.out_in) ri = xdiv(1.0f, ri);
        const float cos_t2 = xsub(1.0f, xmul(xmul(ri, ri), xsub(1.0f, xmul(rdn, rdn))));
        if (!(cos_t2 < 0.0f)) {
            if (dp.diffuse > 0 && dp.td[f.mat] != 0.0f) {
                f.nrefr = dist_count(dp.diffuse, f.level);
                f.refr_at = kb;
                kb += 2u * (uint32_t)f.nrefr;
            } else {
                f.nrefr = 1;
            }
        }
    }
}

// The counting pass of a reference-stream frame without diffuse rays: the
// pixel's ray tree (ray_trace_engine::ray_trace, raytracer.cc:20-87) walked
// post-order with an explicit stack, without shadow rays, counting the
// numbers the pixel draws in the reference's order (at each hit: the
// lights' rays, then the reflection set, then the refraction set; then the
// children's subtrees in order).
template <class SC>
__device__ __forceinline__ uint32_t dist_count_pixel(const SC &sc, const CameraView &cam,
                                                     const LightSet &lights, const MaterialTable &table,
                                                     const DistLights &dl, const DistParams &dp,
                                                     const float *__restrict__ lut, DistStream &S, int x, int y,
                                                     DistFrame *F, uint32_t &status)
{
    uint32_t k = 0;
    const RayState cr = camera_ray(cam, x, y);
    F[0].o = cr.o;
    F[0].d = cr.d;
    F[0].magn = 1.0f;
    F[0].level = 0;
    F[0].node = kTreeRoot;
    F[0].stage = kDistTrace;
    int sp = 1;
    for (int step = 0; sp > 0 && step < dp.max_steps; ++step) {
        DistFrame &f = F[sp - 1];
        if (f.stage == kDistTrace) {
            HitRecord h;
            bool occ;
            status |= traverse<false>(sc, f.o, f.d, FLT_MAX, h, occ);
            f.nrefl = 0;
            f.nrefr = 0;
            f.stage = kDistDone;
            if (h.t < FLT_MAX) {
                const int32_t id = h.id - sc.tri_base;
                int32_t mi = sc.mat ? __ldg(&sc.mat[id]) : 0;
                if (mi < 0 || mi >= table.n) { status |= kStatusBadIndex; mi = 0; }
                const MaterialView &m = table.m[mi];
                RayState r;
                r.o = f.o;
                r.d = f.d;
                const SurfacePoint spt = surface_at(sc, r, h);
                const int lvl = min(f.level, kDistLevels - 1);
                for (int l = 0; l < lights.n; ++l) k += (uint32_t)dl.draws[l][lvl];
                f.o = spt.dst;
                f.sn = spt.sn;
                f.geo = spt.geo;
                f.mat = mi;
                f.out_in = spt.out_in ? 1 : 0;
                if ((double)xmul(f.magn, m.rf) > 0.1) {
                    f.nrefl = (dp.diffuse > 0 && dp.rfd[mi] != 0.0f) ? dist_count(dp.diffuse, f.level) : 1;
                    if (dp.diffuse > 0 && dp.rfd[mi] != 0.0f) { f.refl_at = k; k += 2u * (uint32_t)f.nrefl; }
                }
                if ((double)xmul(f.magn, m.tran) > 0.1) {
                    float ri = m.ri;
                    const float rdn = -xdot(f.d, f.sn);
                    if (f.out_in) ri = xdiv(1.0f, ri);
                    const float cos_t2 = xsub(1.0f, xmul(xmul(ri, ri), xsub(1.0f, xmul(rdn, rdn))));
                    if (!(cos_t2 < 0.0f)) {
                        f.nrefr = (dp.diffuse > 0 && dp.td[mi] != 0.0f) ? dist_count(dp.diffuse, f.level) : 1;
                        if (dp.diffuse > 0 && dp.td[mi] != 0.0f) { f.refr_at = k; k += 2u * (uint32_t)f.nrefr; }
                    }
                }
                f.child = 0;
                f.stage = kDistRefl;
            }
        }
        if (f.stage == kDistRefl) {
            if (f.child < f.nrefl) {
                if (sp >= kDistDepth) { status |= kStatusStepLimit; f.child = f.nrefl; continue; }
                spawn_child(f, table.m[f.mat], dp, 0, f.child, lut, S, status, F[sp]);
                ++f.child;
                ++sp;
                continue;
            }
            f.child = 0;
            f.stage = kDistRefr;
        }
        if (f.stage == kDistRefr) {
            if (f.child < f.nrefr) {
                if (sp >= kDistDepth) { status |= kStatusStepLimit; f.child = f.nrefr; continue; }
                spawn_child(f, table.m[f.mat], dp, 1, f.child, lut, S, status, F[sp]);
                ++f.child;
                ++sp;
                continue;
            }
            f.stage = kDistDone;
        }
        --sp;
    }
    if (sp > 0) status |= kStatusStepLimit;
    return k;
}

// How dist_walk walks: the whole tree from the camera ray; the camera ray's
// node alone (its colour from the lights and ka, its sets left in F[0] for
// the caller to hand out); or the subtree of a ray given in F[0].
enum : int { kDistWhole = 0, kDistRoot = 1, kDistSub = 2 };

// A pixel's ray tree shaded (ray_trace_engine::ray_trace, raytracer.cc:
// 20-87): the post-order walk of dist_count_pixel with every node shaded
// -- the coloured Phong of each light with its first ray's direction and
// length, weighted by the fraction of its rays that reach it (ray::find_rays
// ray.cc:91-104, light::find_rays light.h:62-164), plus ka; then each set's
// mean colour times rf, then tran -- drawing the numbers in the reference's
// order.  The walk is resumable: walk_advance moves it to the lane's next
// ray (a node's camera, mirror, refracted or diffuse ray: closest hit; a
// light's ray: any hit), the caller traces it, walk_consume takes the
// result -- so a warp's lanes trace together at one call site whatever
// stage their trees are at.  Walk holds the state besides the frame stack;
// the top frame's lights are shaded before any child is pushed, so one set
// of light state serves every frame.
struct Walk {
    int sp, step;
    float3 start, kd, ldir, c, out;
    float len;
    int light, sample, nl, made, lvl;
    uint32_t k;            // reference stream: the pixel's next number
    uint32_t kb, k0;       // the node's next number and its first
    uint32_t drawn, nsec;
    bool hit;
};

// A walk from the camera ray of (x, y), or (kDistSub) from the ray already
// in F[0].
template <int MODE>
__device__ __forceinline__ void walk_start(Walk &w, const CameraView &cam, DistFrame *F, int x, int y)
{
    if (MODE != kDistSub) {
        const RayState cr = camera_ray(cam, x, y);
        F[0].o = cr.o;
        F[0].d = cr.d;
        F[0].magn = 1.0f;
        F[0].level = 0;
        F[0].node = kTreeRoot;
        F[0].stage = kDistTrace;
    }
    w.sp = 1;
    w.step = 0;
    w.start = w.kd = w.ldir = w.c = make_float3(0.f, 0.f, 0.f);
    w.out = cam.background;
    w.len = 0.f;
    w.light = w.sample = w.made = w.lvl = 0;
    w.nl = 1;
    w.k = w.kb = w.k0 = w.drawn = w.nsec = 0;
    w.hit = false;
}

// Moves the walk to its next ray (true: ray in ro, rd, rt, any) or to its
// end (false: colour in w.out; kDistRoot: also when the camera ray's node
// is shaded, its sets left in F[0]).
template <int MODE>
__device__ __forceinline__ bool walk_advance(Walk &w, const SceneView &sc, const LightSet &lights,
                                             const MaterialTable &table, const DistLights &dl, const DistParams &dp,
                                             const int4 *__restrict__ area, const float *__restrict__ verts,
                                             const float *__restrict__ lut, DistStream &S, DistFrame *F,
                                             float3 &ro, float3 &rd, float &rt, bool &any, uint32_t &status)
{
    if (w.sp <= 0) return false;
    if (++w.step > dp.max_steps) {
        status |= kStatusStepLimit;
        w.sp = 0;
        return false;
    }
    for (int guard = 0; w.sp > 0 && guard < 4 * kDistDepth + 2 * RT_MAX_LIGHTS + 4; ++guard) {
        DistFrame &f = F[w.sp - 1];
        if (f.stage == kDistTrace) {
            ro = f.o;
            rd = f.d;
            rt = FLT_MAX;
            any = false;
            return true;
        }
        if (f.stage == kDistLights) {
            const MaterialView &m = table.m[f.mat];
            if (w.light < lights.n) {
                const LightView &L = lights.l[w.light];
                if (w.sample < w.nl) {
                    // ray `sample` of this light
                    float3 di;
                    float li;
                    dist_light_ray(lights, dl, area, verts, sc.idx, lut, S, f.node, w.light, w.lvl, w.nl, w.sample,
                                   w.kb, w.start, di, li, status);
                    if (w.sample == 0) {
                        w.ldir = di;
                        w.len = li;
                    }
                    ro = w.start;
                    rd = di;
                    rt = li;
                    any = true;
                    return true;
                }
                w.kb += (uint32_t)dl.draws[w.light][w.lvl];
                w.nsec += (uint32_t)w.nl;
                phong_add<true>(L, m, w.kd, f.sn, f.d, w.ldir, w.len, xdiv((float)w.made, (float)w.nl), w.c);
                ++w.light;
                w.sample = 0;
                w.made = 0;
                if (w.light < lights.n)
                    w.nl = (lights.l[w.light].kind == RT_LIGHT_DIRECTIONAL) ? 1 : dist_count(dp.soft, f.level);
                continue;
            }
            // shaded: ka, then the sets (their numbers after the lights')
            f.c = xadd3(w.c, m.ka);
            dist_sets(f, m, dp, w.kb);
            w.drawn += w.kb - w.k0;
            if (!dp.pixel_stream) w.k = w.kb;
            f.child = 0;
            f.sum = make_float3(0.f, 0.f, 0.f);
            f.stage = kDistRefl;
            if (MODE == kDistRoot) {   // the camera ray's node alone: its sets stay in F[0]
                w.out = f.c;
                w.sp = 0;
                return false;
            }
            continue;
        }
        if (f.stage == kDistRefl) {
            const MaterialView &m = table.m[f.mat];
            if (f.child < f.nrefl) {
                if (w.sp >= kDistDepth) {
                    status |= kStatusStepLimit;
                    f.child = f.nrefl;
                } else {
                    spawn_child(f, m, dp, 0, f.child, lut, S, status, F[w.sp]);
                    ++f.child;
                    ++w.sp;
                }
            } else {
                if (m.rf > 0.0f && f.nrefl > 0) f.c = xadd3(f.c, xmul3(xdiv3(f.sum, (float)f.nrefl), m.rf));
                f.child = 0;
                f.sum = make_float3(0.f, 0.f, 0.f);
                f.stage = kDistRefr;
            }
            continue;
        }
        if (f.stage == kDistRefr) {
            const MaterialView &m = table.m[f.mat];
            if (f.child < f.nrefr) {
                if (w.sp >= kDistDepth) {
                    status |= kStatusStepLimit;
                    f.child = f.nrefr;
                } else {
                    spawn_child(f, m, dp, 1, f.child, lut, S, status, F[w.sp]);
                    ++f.child;
                    ++w.sp;
                }
            } else {
                if (m.tran > 0.0f && f.nrefr > 0) f.c = xadd3(f.c, xmul3(xdiv3(f.sum, (float)f.nrefr), m.tran));
                f.stage = kDistDone;
            }
            continue;
        }
        // done: the frame's colour goes to its parent's current set
        const float3 col = f.c;
        --w.sp;
        if (w.sp == 0) w.out = col;
        else F[w.sp - 1].sum = xadd3(F[w.sp - 1].sum, col);
    }
    if (w.sp > 0) {   // never expected: the guard bounds the moves between two rays
        status |= kStatusStepLimit;
        w.sp = 0;
    }
    return false;
}

// Takes the result of the ray walk_advance asked for.
template <int MODE>
__device__ __forceinline__ void walk_consume(Walk &w, const HitRecord &h, bool occluded, bool any, const SceneView &sc,
                                             const CameraView &cam, const LightSet &lights, const MaterialTable &table,
                                             const DistParams &dp, DistFrame *F, uint32_t &status)
{
    DistFrame &f = F[w.sp - 1];
    if (any) {
        if (!occluded) ++w.made;
        ++w.sample;
        return;
    }
    // the node's closest hit
    if (w.sp > 1 || MODE == kDistSub) ++w.nsec;
    f.nrefl = 0;
    f.nrefr = 0;
    if (!(h.t < FLT_MAX)) {
        f.c = cam.background;
        f.stage = kDistDone;
        if (MODE == kDistRoot) {
            w.out = f.c;
            w.sp = 0;
        }
        return;
    }
    const int32_t id = h.id - sc.tri_base;
    if (w.sp == 1 && MODE != kDistSub) w.hit = true;
    int32_t mi = sc.mat ? __ldg(&sc.mat[id]) : 0;
    if (mi < 0 || mi >= table.n) { status |= kStatusBadIndex; mi = 0; }
    const MaterialView &m = table.m[mi];
    RayState r;
    r.o = f.o;
    r.d = f.d;
    const SurfacePoint spt = surface_at(sc, r, h);
    w.start = offset_start(spt.dst, spt.geo);
    w.kd = material_kd(m, spt);
    w.c = make_float3(0.f, 0.f, 0.f);
    w.lvl = min(f.level, kDistLevels - 1);
    // this node's first number: its own stream's first, or the pixel's next
    // in the reference's stream
    w.k0 = dp.pixel_stream ? 0u : w.k;
    w.kb = w.k0;
    w.light = 0;
    w.sample = 0;
    w.made = 0;
    w.nl = (lights.n > 0 && lights.l[0].kind == RT_LIGHT_DIRECTIONAL) ? 1 : dist_count(dp.soft, f.level);
    f.o = spt.dst;
    f.sn = spt.sn;
    f.geo = spt.geo;
    f.mat = mi;
    f.out_in = spt.out_in ? 1 : 0;
    f.stage = kDistLights;
}

// The whole walk of one lane (its lanes' rays traced together while their
// walks last).
template <int MODE, class SC>
__device__ __forceinline__ uint32_t dist_walk(const SC &sc, const CameraView &cam, const LightSet &lights,
                                              const MaterialTable &table, const DistLights &dl, const DistParams &dp,
                                              const int4 *__restrict__ area, const float *__restrict__ verts,
                                              const float *__restrict__ lut, DistStream &S, int x, int y,
                                              DistFrame *F, float3 &out, bool &hit, uint32_t &nsec,
                                              uint32_t &status)
{
    Walk w;
    walk_start<MODE>(w, cam, F, x, y);
    for (;;) {
        float3 ro, rd;
        float rt;
        bool any;
        if (!walk_advance<MODE>(w, sc, lights, table, dl, dp, area, verts, lut, S, F, ro, rd, rt, any, status)) break;
        HitRecord h;
        bool occluded;
        status |= traverse_ray<false>(sc, ro, rd, rt, any, h, occluded);
        walk_consume<MODE>(w, h, occluded, any, sc, cam, lights, table, dp, F, status);
    }
    out = w.out;
    hit = w.hit;
    nsec += w.nsec;
    return w.drawn;
}

// One launch of the distributed walk: the counting pass (SHADE false:
// counts[pix] = numbers the pixel draws) or the shading pass (numbers from
// the pixels' own streams, or from rnd at prefix[pix]).  A warp walks the 32
// pixels of an 8x4 tile, its lanes' rays traced together.
// RT_DIST_MIN_BLOCKS: resident blocks per SM the register allocation must
// allow (5: 96 registers, measured fastest for the converged walk; 4 was
// for the walk that traced at three call sites).
#ifndef RT_DIST_MIN_BLOCKS
#define RT_DIST_MIN_BLOCKS 5
#endif
template <bool SHADE, class SC>
__global__ void __launch_bounds__(kTraceThreads, RT_DIST_MIN_BLOCKS) k_dist(SC sc, CameraView cam, LightSet lights,
                                                        MaterialTable table, DistLights dl, DistParams dp,
                                                        const int4 *__restrict__ area, const float *__restrict__ verts,
                                                        const float *__restrict__ lut, const uint32_t *__restrict__ rnd,
                                                        int64_t nrnd, const int64_t *__restrict__ prefix,
                                                        int64_t *__restrict__ counts, uint8_t *__restrict__ rgb,
                                                        float *__restrict__ fimg, Counters *ctr)
{
    DistFrame F[kDistDepth];
    int tiles_x;
    const int items = tiles_of<8>(cam.xres, cam.yres, tiles_x) * 32;
    uint32_t status = 0;
    for (;;) {
        const int base = warp_claim(&ctr->work, 32);
        if (base >= items) break;
        int x, y;
        tile_pixel<8>(base + (threadIdx.x & 31), tiles_x, x, y);
        const bool live = (x < cam.xres) && (y < cam.yres);
        uint32_t nsec = 0, drawn = 0;
        bool hit = false;
        if (live) {
            const size_t pix = (size_t)x + (size_t)y * (size_t)cam.xres;
            DistStream S;
            S.win = rnd;
            S.nwin = nrnd;
            S.base = (SHADE && !dp.pixel_stream) ? prefix[pix] : 0;
            S.pixel = (uint32_t)pix;
            S.key0 = dp.key0;
            S.key1 = dp.key1;
            S.pixel_mode = dp.pixel_stream != 0;
            S.blk = 0xffffffffu;
            S.bnode = 0;
            float3 c;
            if (SHADE)
                drawn = dist_walk<kDistWhole>(sc, cam, lights, table, dl, dp, area, verts, lut, S, x, y, F, c, hit,
                                              nsec, status);
            else
                drawn = dist_count_pixel(sc, cam, lights, table, dl, dp, lut, S, x, y, F, status);
            if (SHADE) {
                if (rgb) store_rgb(rgb, pix, c);
                if (fimg) {
                    fimg[3 * pix] = c.x;
                    fimg[3 * pix + 1] = c.y;
                    fimg[3 * pix + 2] = c.z;
                }
            } else {
                counts[pix] = (int64_t)drawn;
            }
        }
        if (SHADE) {
            warp_count(&ctr->primary, live);
            warp_count(&ctr->hits, hit);
            warp_add(&ctr->secondary, nsec);
            unsigned long long d = drawn;
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if ((threadIdx.x & 31) == 0 && d) atomicAdd(&ctr->drawn, d);
        }
    }
    if (status) atomicOr(&ctr->status, status);
}

// Frames of per-pixel streams with ray trees are traced in three launches:
// the camera ray's node of every pixel (k_dist_root: its colour from the
// lights and ka, its sets' rays handed out as separate items), every item's
// subtree (k_dist_sub), then every pixel's colour from its node's and its
// items' (k_dist_combine, in the walk's order of additions).  A node's
// numbers are keyed by the node, so an item's subtree draws the same numbers
// traced alone as in the pixel's walk, and neighbouring items -- the rays of
// one set -- trace together.
struct DistItem {
    float4 o_magn;       // origin, power
    float4 d_level;      // direction, componant level (int bits)
    ulonglong2 node;     // tree node, pixel
};

__device__ __forceinline__ DistStream pixel_streams(const DistParams &dp, uint32_t pix)
{
    DistStream S;
    S.win = nullptr;
    S.nwin = 0;
    S.base = 0;
    S.pixel = pix;
    S.key0 = dp.key0;
    S.key1 = dp.key1;
    S.pixel_mode = true;
    S.blk = 0xffffffffu;
    S.bnode = 0;
    return S;
}

#ifndef RT_DIST_NODE_MIN_BLOCKS
#define RT_DIST_NODE_MIN_BLOCKS 7
#endif
#ifndef RT_DIST_LIGHTS_MIN_BLOCKS
#define RT_DIST_LIGHTS_MIN_BLOCKS 8
#endif
template <class SC>
__global__ void __launch_bounds__(kTraceThreads, RT_DIST_MIN_BLOCKS) k_dist_root(
    SC sc, CameraView cam, LightSet lights, MaterialTable table, DistLights dl, DistParams dp,
    const int4 *__restrict__ area, const float *__restrict__ verts, const float *__restrict__ lut,
    float4 *__restrict__ root_c, int4 *__restrict__ root_sets, DistItem *__restrict__ items, int32_t cap,
    int32_t *__restrict__ nitems, Counters *ctr)
{
    DistFrame F[kDistDepth];   // the walk stops at F[0]
    int tiles_x;
    const int items_n = tiles_of<8>(cam.xres, cam.yres, tiles_x) * 32;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t status = 0;
    for (;;) {
        const int base = warp_claim(&ctr->work, 32);
        if (base >= items_n) break;
        int x, y;
        tile_pixel<8>(base + (int)lane, tiles_x, x, y);
        const bool live = (x < cam.xres) && (y < cam.yres);
        uint32_t nsec = 0, drawn = 0;
        bool hit = false;
        float3 c = cam.background;
        int cnt = 0;
        const size_t pix = live ? (size_t)x + (size_t)y * (size_t)cam.xres : 0;
        if (live) {
            DistStream S = pixel_streams(dp, (uint32_t)pix);
            drawn = dist_walk<kDistRoot>(sc, cam, lights, table, dl, dp, area, verts, lut, S, x, y, F, c, hit,
                                                nsec, status);
            if (F[0].stage == kDistRefl) cnt = F[0].nrefl + F[0].nrefr;
        }
        // the warp's items in lane order, reflection and refraction sets in
        // lists of their own (a warp of subtrees then holds one kind), one
        // allocation per list per warp
        const int nr = cnt > 0 ? F[0].nrefl : 0, nt = cnt > 0 ? F[0].nrefr : 0;
        int ir = nr, it_ = nt;
        for (int o = 1; o < 32; o <<= 1) {
            const int vr = __shfl_up_sync(0xffffffffu, ir, o), vt = __shfl_up_sync(0xffffffffu, it_, o);
            if ((int)lane >= o) { ir += vr; it_ += vt; }
        }
        int rbase = 0, tbase = 0;
        if (lane == 31u) {
            if (ir) rbase = atomicAdd(&nitems[0], ir);
            if (it_) tbase = atomicAdd(&nitems[1], it_);
        }
        rbase = __shfl_sync(0xffffffffu, rbase, 31) + ir - nr;
        tbase = __shfl_sync(0xffffffffu, tbase, 31) + it_ - nt;
        if (live) {
            // else the host grows the lists and runs again
            const bool fits = rbase >= 0 && rbase + nr <= cap && tbase >= 0 && tbase + nt <= cap;
            if (cnt > 0 && fits) {
                DistStream S = pixel_streams(dp, (uint32_t)pix);
                const MaterialView &m = table.m[F[0].mat];
                for (int j = 0; j < cnt; ++j) {
                    const int set = j < nr ? 0 : 1;
                    DistFrame C;
                    spawn_child(F[0], m, dp, set, set ? j - nr : j, lut, S, status, C);
                    DistItem it;
                    it.o_magn = make_float4(C.o.x, C.o.y, C.o.z, C.magn);
                    it.d_level = make_float4(C.d.x, C.d.y, C.d.z, __int_as_float(C.level));
                    it.node = make_ulonglong2(C.node, (unsigned long long)pix);
                    items[set ? (size_t)cap + tbase + (j - nr) : (size_t)rbase + j] = it;
                }
            }
            root_c[pix] = make_float4(c.x, c.y, c.z, __int_as_float(cnt > 0 ? F[0].mat : 0));
            root_sets[pix] = make_int4(rbase, nr, tbase, nt);
        }
        warp_count(&ctr->primary, live);
        warp_count(&ctr->hits, hit);
        warp_add(&ctr->secondary, nsec);
        unsigned long long d = drawn;
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane == 0u && d) atomicAdd(&ctr->drawn, d);
    }
    if (status) atomicOr(&ctr->status, status);
}

// The items of a frame: nr of the reflection sets from entry 0, nt of the
// refraction sets from entry cap, walked as [0, nr) rounded up to a warp and
// then [0, nt).  Entries 2 cap .. 2 cap + pool are the nodes below them.
struct DistLists {
    int32_t nr, nt, cap, pool;
    DistItem *items, *nodes;

    __device__ __forceinline__ DistItem *item(int slot) const
    {
        return slot < 2 * cap ? items + slot : nodes + (slot - 2 * cap);
    }

    __host__ __device__ __forceinline__ int count() const { return ((nr + 31) & ~31) + nt; }
    __device__ __forceinline__ int slot(int v) const   // -1: none
    {
        const int rw = (nr + 31) & ~31;
        return v < rw ? (v < nr ? v : -1) : (v - rw < nt ? cap + (v - rw) : -1);
    }
};

// Counts of a piece of the items' subtrees, level by level.
struct DistCounts {
    int32_t hits, over;                 // nodes to shade, nodes left to k_dist_sub
    int32_t work_lights, work_over;
    int32_t made[kDistDepth + 1];       // nodes asked for at each level below the items' (level 0)
    int32_t work[kDistDepth + 1];
};

// Entries [first, end) of the pool that hold level k's nodes.
__device__ __forceinline__ void dist_level(const DistCounts *dc, int pool, int k, int &first, int &end)
{
    int at = 0;
    end = 0;
    for (int j = 1; j <= k; ++j) {
        at = end;
        end = (int)min((int64_t)pool, (int64_t)at + dc->made[j]);
    }
    first = at;
}

// A node that hit something, for its lights.
struct DistHit {
    float4 start_slot;   // the rays' start, the node's entry (int bits)
    float4 kd_mat;       // diffuse colour, material (int bits)
    float4 sn;           // shading normal
};

constexpr float kDistNoNode = -1.0f;   // the power of an entry without a node

// The items' subtrees are traced a level of all of them at a time: every
// lane of a warp traces a closest hit (k_dist_node), then every lane the
// rays to the lights of a hit (k_dist_lights), then colours are gathered
// from the deepest level up (k_dist_gather).  A node's numbers are keyed by
// the node and follow the lights', whose count is known before they are
// traced, so children are made as soon as their parent has hit.  A node
// whose children don't fit the pool is walked whole by one lane
// (k_dist_sub), as is everything where the lists can't be had.
// The walk is bound by issue slots at 11.8 lanes an instruction: lanes stand at
// nodes and rays of different kinds.  512x512 glass frame with 16-ray diffuse
// sets and soft shadows (51.6 M rays): walked 23.9 ms, by levels 21.6, with a
// hit's rays to a light on neighbouring lanes 19.4, with 7 and 8 blocks to an SM
// for 6 and 6 18.65 ms.
template <class SC>
__global__ void __launch_bounds__(kTraceThreads, RT_DIST_NODE_MIN_BLOCKS) k_dist_node(
    SC sc, CameraView cam, LightSet lights, MaterialTable table, DistLights dl, DistParams dp,
    const float *__restrict__ lut, DistLists lists, int v0, int v1, int level, int last,
    int4 *__restrict__ sets, float4 *__restrict__ item_c, DistHit *__restrict__ hits, int32_t *__restrict__ over,
    DistCounts *dc, Counters *ctr)
{
    const uint32_t lane = threadIdx.x & 31u;
    const int pool0 = 2 * lists.cap;
    int first = v0, end = v1, next = 0;
    if (level > 0) dist_level(dc, lists.pool, level, first, end);
    if (level > 0) next = end;         // the next level's nodes follow
    uint32_t status = 0;
    uint32_t nsec = 0;
    unsigned long long drawn = 0;
    for (;;) {
        const int base = first + warp_claim(&dc->work[level], 32);
        if (base >= end) break;
        const int v = base + (int)lane;
        const int slot = v < end ? (level > 0 ? pool0 + v : lists.slot(v)) : -1;
        DistFrame f;
        f.o = f.d = make_float3(0.f, 0.f, 0.f);
        bool on = slot >= 0;
        uint32_t pix = 0;
        if (on) {
            const DistItem it = *lists.item(slot);
            f.o = make_float3(it.o_magn.x, it.o_magn.y, it.o_magn.z);
            f.magn = it.o_magn.w;
            f.d = make_float3(it.d_level.x, it.d_level.y, it.d_level.z);
            f.level = __float_as_int(it.d_level.w);
            f.node = it.node.x;
            pix = (uint32_t)it.node.y;
            on = f.magn != kDistNoNode;
        }
        HitRecord h;
        bool occ;
        status |= traverse_warp<false>(sc, on, f.o, f.d, FLT_MAX, h, occ);
        const bool hit = on && h.t < FLT_MAX;
        float3 start, kd;
        uint32_t kb = 0, nl = 0;
        f.nrefl = f.nrefr = 0;
        f.mat = 0;
        if (hit) {
            const int32_t id = h.id - sc.tri_base;
            int32_t mi = sc.mat ? __ldg(&sc.mat[id]) : 0;
            if (mi < 0 || mi >= table.n) { status |= kStatusBadIndex; mi = 0; }
            const MaterialView &m = table.m[mi];
            RayState r;
            r.o = f.o;
            r.d = f.d;
            const SurfacePoint spt = surface_at(sc, r, h);
            start = offset_start(spt.dst, spt.geo);
            kd = material_kd(m, spt);
            f.o = spt.dst;
            f.sn = spt.sn;
            f.geo = spt.geo;
            f.mat = mi;
            f.out_in = spt.out_in ? 1 : 0;
            const int lvl = min(f.level, kDistLevels - 1);
            for (int l = 0; l < lights.n; ++l) {
                kb += (uint32_t)dl.draws[l][lvl];
                nl += lights.l[l].kind == RT_LIGHT_DIRECTIONAL ? 1u : (uint32_t)dist_count(dp.soft, f.level);
            }
            dist_sets(f, m, dp, kb);
        }
        int cnt = f.nrefl + f.nrefr;
        if (last && cnt > 0) {         // never expected: the tree's bound gives the levels
            status |= kStatusStepLimit;
            f.nrefl = f.nrefr = cnt = 0;
        }
        // the warp's children in lane order, one allocation
        int sum = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, sum, o);
            if ((int)lane >= o) sum += t;
        }
        int at = 0;
        if (lane == 31u && sum) at = atomicAdd(&dc->made[level + 1], sum);
        const int64_t child = (int64_t)next + __shfl_sync(0xffffffffu, at, 31) + sum - cnt;
        const bool fits = cnt == 0 || child + cnt <= lists.pool;
        if (cnt > 0) {
            if (fits) {
                const MaterialView &m = table.m[f.mat];
                DistStream S = pixel_streams(dp, pix);
                for (int j = 0; j < cnt; ++j) {
                    const int set = j < f.nrefl ? 0 : 1;
                    DistFrame C;
                    spawn_child(f, m, dp, set, set ? j - f.nrefl : j, lut, S, status, C);
                    DistItem it;
                    it.o_magn = make_float4(C.o.x, C.o.y, C.o.z, C.magn);
                    it.d_level = make_float4(C.d.x, C.d.y, C.d.z, __int_as_float(C.level));
                    it.node = make_ulonglong2(C.node, (unsigned long long)pix);
                    lists.nodes[child + j] = it;
                }
            } else {
                for (int64_t j = child; j < lists.pool; ++j)
                    lists.nodes[j].o_magn = make_float4(0.f, 0.f, 0.f, kDistNoNode);
                over[atomicAdd(&dc->over, 1)] = slot;
            }
        }
        // the hits, in lane order
        const uint32_t hm = __ballot_sync(0xffffffffu, hit && fits);
        int hat = 0;
        if (lane == 0u && hm) hat = atomicAdd(&dc->hits, __popc(hm));
        hat = __shfl_sync(0xffffffffu, hat, 0);
        if (hit && fits) {
            DistHit H;
            H.start_slot = make_float4(start.x, start.y, start.z, __int_as_float(slot));
            H.kd_mat = make_float4(kd.x, kd.y, kd.z, __int_as_float(f.mat));
            H.sn = make_float4(f.sn.x, f.sn.y, f.sn.z, 0.f);
            hits[hat + __popc(hm & ((1u << lane) - 1u))] = H;
            nsec += nl;
            drawn += kb;
        }
        if (slot >= 0) {
            sets[slot] = cnt > 0 && fits ? make_int4(pool0 + (int)child, f.nrefl, f.nrefr, f.mat) : make_int4(0, 0, 0, 0);
            if (on && !hit) item_c[slot] = make_float4(cam.background.x, cam.background.y, cam.background.z, 0.f);
        }
        if (on && fits) ++nsec;
    }
    warp_add(&ctr->secondary, nsec);
    for (int o = 16; o > 0; o >>= 1) drawn += __shfl_xor_sync(0xffffffffu, drawn, o);
    if (lane == 0u && drawn) atomicAdd(&ctr->drawn, drawn);
    if (status) atomicOr(&ctr->status, status);
}

// The colour of every hit node from its lights and ka (the walk's sum).  A
// warp takes 32 hits, light by light.
template <class SC>
__global__ void __launch_bounds__(kTraceThreads, RT_DIST_LIGHTS_MIN_BLOCKS) k_dist_lights(
    SC sc, LightSet lights, MaterialTable table, DistLights dl, DistParams dp, const int4 *__restrict__ area,
    const float *__restrict__ verts, const float *__restrict__ lut, DistLists lists, const DistHit *__restrict__ hits,
    float4 *__restrict__ item_c, DistCounts *dc, Counters *ctr)
{
    struct Hit {
        uint64_t node;
        uint32_t pix, kb;
        int lvl, n;
    };
    const uint32_t lane = threadIdx.x & 31u;
    const int n = dc->hits;
    uint32_t status = 0;
    for (;;) {
        const int base = warp_claim(&dc->work_lights, 32);
        if (base >= n) break;
        const bool on = base + (int)lane < n;
        const DistHit H = hits[on ? base + (int)lane : base];
        const int slot = __float_as_int(H.start_slot.w);
        const DistItem it = *lists.item(slot);
        const float3 start = make_float3(H.start_slot.x, H.start_slot.y, H.start_slot.z);
        const float3 kd = make_float3(H.kd_mat.x, H.kd_mat.y, H.kd_mat.z);
        const float3 sn = make_float3(H.sn.x, H.sn.y, H.sn.z);
        const float3 d = make_float3(it.d_level.x, it.d_level.y, it.d_level.z);
        const int level = __float_as_int(it.d_level.w), lvl = min(level, kDistLevels - 1);
        const MaterialView &m = table.m[__float_as_int(H.kd_mat.w)];
        uint32_t kb = 0;
        float3 c = make_float3(0.f, 0.f, 0.f);
        for (int l = 0; l < lights.n; ++l) {
            const LightView &L = lights.l[l];
            const int nl = L.kind == RT_LIGHT_DIRECTIONAL ? 1 : dist_count(dp.soft, level);
            float3 ldir = d;
            float len = 0.f;
            int made = 0;
            trace_hit_rays(
                sc, start, on ? nl : 0,
                [&](int own) {
                    Hit q;
                    q.node = __shfl_sync(0xffffffffu, it.node.x, own);
                    q.pix = __shfl_sync(0xffffffffu, (uint32_t)it.node.y, own);
                    q.lvl = __shfl_sync(0xffffffffu, lvl, own);
                    q.n = __shfl_sync(0xffffffffu, nl, own);
                    q.kb = __shfl_sync(0xffffffffu, kb, own);
                    return q;
                },
                [&](const Hit &q, int i, float3 from, float3 &di, float &li) {
                    DistStream S = pixel_streams(dp, q.pix);
                    dist_light_ray(lights, dl, area, verts, sc.idx, lut, S, q.node, l, q.lvl, q.n, i, q.kb, from, di,
                                   li, status);
                },
                ldir, len, made, status);
            kb += (uint32_t)dl.draws[l][lvl];
            if (on) phong_add<true>(L, m, kd, sn, d, ldir, len, xdiv((float)made, (float)nl), c);
        }
        if (on) {
            c = xadd3(c, m.ka);
            item_c[slot] = make_float4(c.x, c.y, c.z, 0.f);
        }
    }
    if (status) atomicOr(&ctr->status, status);
}

// A set's mean colour times its weight, added to c.
__device__ __forceinline__ float3 add_set(float3 c, const float4 *__restrict__ set, int n, float weight)
{
    if (!(weight > 0.0f) || n <= 0) return c;
    float3 sum = make_float3(0.f, 0.f, 0.f);
    for (int j = 0; j < n; ++j) {
        const float4 q = set[j];
        sum = xadd3(sum, make_float3(q.x, q.y, q.z));
    }
    return xadd3(c, xmul3(xdiv3(sum, (float)n), weight));
}

// The nodes of a level: their sets' means added times rf, then tran.
__global__ void k_dist_gather(MaterialTable table, DistLists lists, int v0, int v1, int level,
                              const int4 *__restrict__ sets, float4 *__restrict__ item_c, const DistCounts *dc)
{
    int first = v0, end = v1;
    if (level > 0) dist_level(dc, lists.pool, level, first, end);
    for (int v = first + blockIdx.x * blockDim.x + threadIdx.x; v < end; v += gridDim.x * blockDim.x) {
        const int slot = level > 0 ? 2 * lists.cap + v : lists.slot(v);
        if (slot < 0) continue;
        const int4 s = sets[slot];
        if (s.y + s.z == 0) continue;
        const MaterialView &m = table.m[s.w];
        const float4 q = item_c[slot];
        float3 c = make_float3(q.x, q.y, q.z);
        c = add_set(c, item_c + s.x, s.y, m.rf);
        c = add_set(c, item_c + s.x + s.y, s.z, m.tran);
        item_c[slot] = make_float4(c.x, c.y, c.z, 0.f);
    }
}

// The subtrees of the items, or of the nodes of `list`, one per lane; a warp
// takes 32 consecutive ones (the rays of one or two sets) at a time.  (Lanes
// that take the next item as soon as theirs is finished were measured slower:
// 61 against 41 ms on the 512x512 glass frame with 16-ray diffuse sets, their
// rays no longer neighbours.)
// 6 resident blocks (80 registers): 34.1 ms against 41.3 at 4 and 37.1 at 5
// on the 512x512 glass frame with 16-ray diffuse sets; 7 and 8 no faster
#ifndef RT_DIST_SUB_MIN_BLOCKS
#define RT_DIST_SUB_MIN_BLOCKS 6
#endif
template <class SC>
__global__ void __launch_bounds__(kTraceThreads, RT_DIST_SUB_MIN_BLOCKS) k_dist_sub(
    SC sc, CameraView cam, LightSet lights, MaterialTable table, DistLights dl, DistParams dp,
    const int4 *__restrict__ area, const float *__restrict__ verts, const float *__restrict__ lut, DistLists lists,
    const int32_t *__restrict__ list,
    const int32_t *__restrict__ nlist, int32_t *work, float4 *__restrict__ item_c, Counters *ctr)
{
    DistFrame F[kDistDepth];
    const uint32_t lane = threadIdx.x & 31u;
    const int n = list ? *nlist : lists.count();
    uint32_t status = 0;
    for (;;) {
        const int base = warp_claim(work, 32);
        if (base >= n) break;
        const int v = base + (int)lane;
        const int i = list ? (v < n ? list[v] : -1) : lists.slot(v);
        uint32_t nsec = 0, drawn = 0;
        if (i >= 0) {
            const DistItem it = *lists.item(i);
            F[0].o = make_float3(it.o_magn.x, it.o_magn.y, it.o_magn.z);
            F[0].magn = it.o_magn.w;
            F[0].d = make_float3(it.d_level.x, it.d_level.y, it.d_level.z);
            F[0].level = __float_as_int(it.d_level.w);
            F[0].node = it.node.x;
            F[0].stage = kDistTrace;
            DistStream S = pixel_streams(dp, (uint32_t)it.node.y);
            float3 c;
            bool hit;
            drawn = dist_walk<kDistSub>(sc, cam, lights, table, dl, dp, area, verts, lut, S, 0, 0, F, c, hit, nsec,
                                        status);
            item_c[i] = make_float4(c.x, c.y, c.z, 0.f);
        }
        warp_add(&ctr->secondary, nsec);
        unsigned long long d = drawn;
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane == 0u && d) atomicAdd(&ctr->drawn, d);
    }
    if (status) atomicOr(&ctr->status, status);
}

// A pixel's colour: its node's, then each set's mean added times rf, then
// tran (the walk's additions, in its order).
__global__ void k_dist_combine(CameraView cam, MaterialTable table, const float4 *__restrict__ root_c,
                               const int4 *__restrict__ root_sets, const float4 *__restrict__ item_c, int32_t nr,
                               int32_t nt, int32_t cap, uint8_t *__restrict__ rgb, float *__restrict__ fimg,
                               Counters *ctr)
{
    const int32_t npix = cam.xres * cam.yres;
    uint32_t status = 0;
    for (int32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const float4 r = root_c[p];
        const int4 sets = root_sets[p];   // reflection list's first, count; refraction list's first, count
        float3 c = make_float3(r.x, r.y, r.z);
        if (sets.y + sets.w > 0) {
            if (sets.x < 0 || sets.x + sets.y > nr || sets.z < 0 || sets.z + sets.w > nt) {
                status |= kStatusBadIndex;
            } else {
                const MaterialView &m = table.m[__float_as_int(r.w)];
                c = add_set(c, item_c + sets.x, sets.y, m.rf);
                c = add_set(c, item_c + (size_t)cap + sets.z, sets.w, m.tran);
            }
        }
        if (rgb) store_rgb(rgb, (size_t)p, c);
        if (fimg) {
            fimg[3 * (size_t)p] = c.x;
            fimg[3 * (size_t)p + 1] = c.y;
            fimg[3 * (size_t)p + 2] = c.z;
        }
    }
    if (status) atomicOr(&ctr->status, status);
}

}  // namespace
}  // namespace rtc

using namespace rtc;

namespace {

rt_status sfail(rt_status c, const char *m) { return set_error(c, m); }

#define RT_CUDA_S(call, what)                                  \
    do {                                                       \
        cudaError_t _e = (call);                               \
        if (_e != cudaSuccess) return set_cuda_error(_e, what); \
    } while (0)

struct SGuard {
    int prev = -1;
    explicit SGuard(int dev)
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~SGuard()
    {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

rt_status check_shapes(const rt_scene *s, const rt_light *lights, int32_t nlights, const rt_light_shape *shapes,
                       const char *who);
rt_status stream_window(SoftState &S, int64_t offset, int64_t total, cudaStream_t st, const uint32_t **rnd);

template <class SC>
int soft_blocks_per_sm()
{
    static const int per_sm = [] {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_soft_shade<SC>, kTraceThreads, 0) != cudaSuccess || b < 1) {
            cudaGetLastError();
            b = 4;
        }
        return b;
    }();
    return per_sm;
}

}  // namespace

extern "C" rt_status rt_render_soft_shadows(rt_scene *s, const rt_camera *camera, const rt_light *lights,
                                            int32_t nlights, const rt_light_shape *shapes,
                                            const rt_material *materials, int32_t nmaterials, int32_t samples,
                                            int64_t stream_offset, uint8_t *rgb_out, float *rgb_f32,
                                            int64_t *stream_end, rt_render_stats *stats)
{
    if (!s || !camera || !materials || (!rgb_out && !rgb_f32))
        return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: NULL argument");
    if (camera->xres <= 0 || camera->yres <= 0 || (int64_t)camera->xres * camera->yres > (int64_t)1 << 28)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: camera resolution out of range");
    if (nlights < 0 || nlights > RT_MAX_LIGHTS || (nlights > 0 && !lights))
        return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: light count out of range");
    if (nmaterials < 1 || nmaterials > RT_MAX_MATERIALS)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: material count must be 1..RT_MAX_MATERIALS");
    if (samples < 1 || samples > RT_MAX_SOFT_SAMPLES)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: samples must be 1..RT_MAX_SOFT_SAMPLES");
    if (stream_offset < 0) return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: negative stream offset");
    for (int32_t i = 0; i < nmaterials; ++i)
        if (materials[i].rf != 0.0f || materials[i].tran != 0.0f)
            return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: mirror and refracting materials are not offered");
    {
        const rt_status st = check_shapes(s, lights, nlights, shapes, "rt_render_soft_shadows");
        if (st != RT_OK) return st;
    }
    if (!s->built) return sfail(RT_ERR_NOT_BUILT, "rt_render_soft_shadows: hierarchy not built");
    if (s->mat_max >= nmaterials)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_soft_shadows: the scene's material indices exceed the table");
    rt_context *ctx = s->ctx;
    SGuard g(ctx->device);
    if (!ctx->soft) {
        ctx->soft = new (std::nothrow) SoftState();
        if (!ctx->soft) return sfail(RT_ERR_OUT_OF_MEMORY, "rt_render_soft_shadows: state allocation");
        ctx->soft->device = ctx->device;
    }
    SoftState &S = *ctx->soft;
    cudaStream_t st = ctx->stream;
    if (!S.lut_ready) {
        // static_cos (common/common.h:174-181): angle rounded to binary32,
        // cosine in double, rounded to binary32
        std::vector<float> lut(kCosLutSize);
        for (int i = 0; i < kCosLutSize; ++i)
            lut[i] = (float)std::cos((double)((((float)i * 2.0f) * kRefPi) / (float)kCosLutSize));
        RT_CUDA_S(S.lut.reserve(kCosLutSize * sizeof(float)), "cosine table allocation");
        RT_CUDA_S(cudaMemcpy(S.lut.ptr, lut.data(), kCosLutSize * sizeof(float), cudaMemcpyHostToDevice),
                  "cosine table copy");
        S.lut_ready = true;
    }
    const size_t npix = (size_t)camera->xres * (size_t)camera->yres;
    RT_CUDA_S(S.hits.reserve(npix * sizeof(int4)), "hit record allocation");
    RT_CUDA_S(S.flags.reserve(npix * sizeof(int32_t)), "hit flag allocation");
    RT_CUDA_S(S.prefix.reserve(npix * sizeof(int32_t)), "prefix allocation");
    size_t scan_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const int32_t *)S.flags.ptr, (int32_t *)S.prefix.ptr,
                                  (int)npix, st);
    RT_CUDA_S(S.scan_temp.reserve(scan_bytes), "scan scratch allocation");
    LightSet ls;
    ls.n = nlights;
    ls.fast_pow = 0;
    AreaSet as = {};
    std::vector<int4> area_rays;
    int32_t per_hit = 0;
    for (int i = 0; i < nlights; ++i) {
        ls.l[i] = make_light_view(lights[i]);
        ls.l[i].radius = shapes ? shapes[i].radius : 0.0f;
        if (!(samples > 1 && ls.l[i].kind != RT_LIGHT_DIRECTIONAL)) continue;
        if (shapes && shapes[i].ntris > 0) {
            // the light's rays in the order find_rays makes them; the first
            // `samples` are traced, every one made draws two numbers
            const int32_t nt = shapes[i].ntris;
            std::vector<int32_t> cnt((size_t)nt);
            const int32_t made = area_light_rays(nt, samples, cnt.data());
            if (made < samples)
                return sfail(RT_ERR_INVALID_ARG,
                             "rt_render_soft_shadows: a triangle-defined light makes fewer rays than samples");
            as.first[i] = (int32_t)area_rays.size();
            as.made[i] = made;
            as.draws[i] = 2 * made;
            for (int32_t j = 0; j < nt; ++j)
                for (int32_t k = 0; k < cnt[(size_t)j]; ++k) area_rays.push_back(make_int4(shapes[i].tris[j], cnt[(size_t)j], k, 0));
        } else {
            as.draws[i] = 3 * samples;
        }
        per_hit += as.draws[i];
    }
    if (!area_rays.empty()) {
        RT_CUDA_S(S.area.reserve(area_rays.size() * sizeof(int4)), "light ray table allocation");
        RT_CUDA_S(cudaMemcpyAsync(S.area.ptr, area_rays.data(), area_rays.size() * sizeof(int4), cudaMemcpyHostToDevice,
                                  st),
                  "light ray table copy");
    }
    MaterialTable mt;
    mt.n = nmaterials;
    for (int i = 0; i < nmaterials; ++i) mt.m[i] = make_material_view(materials[i]);
    const SceneView sv = scene_view(s);
    const CameraView cv = make_camera_view(*camera);

    RT_CUDA_S(cudaMemsetAsync(ctx->d_counters, 0, sizeof(Counters), st), "counter clear");
    RT_CUDA_S(cudaEventRecord(ctx->ev0, st), "event record");
    with_scene(sv, [&](const auto &view) {
        using SC = std::decay_t<decltype(view)>;
        k_soft_primary<SC><<<soft_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
            view, cv, (int4 *)S.hits.ptr, (int32_t *)S.flags.ptr, ctx->d_counters);
    });
    RT_CUDA_S(cudaGetLastError(), "primary launch");
    cub::DeviceScan::ExclusiveSum(S.scan_temp.ptr, scan_bytes, (const int32_t *)S.flags.ptr, (int32_t *)S.prefix.ptr,
                                  (int)npix, st);
    RT_CUDA_S(cudaGetLastError(), "scan launch");
    // the frame's count of numbers: per_hit for every hit pixel
    int32_t *h = ctx->h_scratch;
    RT_CUDA_S(cudaMemcpyAsync(h, (const int32_t *)S.prefix.ptr + (npix - 1), sizeof(int32_t), cudaMemcpyDeviceToHost, st),
              "prefix read");
    RT_CUDA_S(cudaMemcpyAsync(h + 1, (const int32_t *)S.flags.ptr + (npix - 1), sizeof(int32_t),
                              cudaMemcpyDeviceToHost, st),
              "flag read");
    RT_CUDA_S(cudaStreamSynchronize(st), "synchronize");
    const int64_t nhits = (int64_t)h[0] + h[1];
    const int64_t total = nhits * per_hit;
    // the frame's slice of the reference's stream
    const uint32_t *rnd = nullptr;
    const rt_status wst = stream_window(S, stream_offset, total, st, &rnd);
    if (wst != RT_OK) return wst;

    // outputs: device pointers as given, host ones staged
    const bool rgb_host = rgb_out && !is_device_ptr(rgb_out);
    const bool f_host = rgb_f32 && !is_device_ptr(rgb_f32);
    uint8_t *d_rgb = rgb_out;
    float *d_f = rgb_f32;
    if (rgb_host) {
        RT_CUDA_S(ctx->stage_a.reserve(npix * 3), "staging allocation");
        d_rgb = (uint8_t *)ctx->stage_a.ptr;
    }
    if (f_host) {
        RT_CUDA_S(ctx->fimg.reserve(npix * 3 * sizeof(float)), "float frame allocation");
        d_f = (float *)ctx->fimg.ptr;
    }
    RT_CUDA_S(cudaMemsetAsync(&ctx->d_counters->work, 0, sizeof(int), st), "work counter clear");
    with_scene(sv, [&](const auto &view) {
        using SC = std::decay_t<decltype(view)>;
        k_soft_shade<SC><<<soft_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
            view, cv, ls, mt, as, (const int4 *)S.area.ptr, s->d_verts, samples, per_hit, rnd, total,
            (const float *)S.lut.ptr, (const int4 *)S.hits.ptr, (const int32_t *)S.prefix.ptr, d_rgb, d_f,
            ctx->d_counters);
    });
    RT_CUDA_S(cudaGetLastError(), "shade launch");
    RT_CUDA_S(cudaEventRecord(ctx->ev1, st), "event record");
    if (rgb_host) RT_CUDA_S(cudaMemcpyAsync(rgb_out, d_rgb, npix * 3, cudaMemcpyDeviceToHost, st), "rgb copy");
    if (f_host)
        RT_CUDA_S(cudaMemcpyAsync(rgb_f32, d_f, npix * 3 * sizeof(float), cudaMemcpyDeviceToHost, st), "image copy");
    Counters c;
    RT_CUDA_S(cudaMemcpyAsync(&c, ctx->d_counters, sizeof(Counters), cudaMemcpyDeviceToHost, st), "counter read");
    RT_CUDA_S(cudaStreamSynchronize(st), "synchronize");
    if (stats) {
        stats->primary_rays = (int64_t)c.primary;
        stats->secondary_rays = (int64_t)c.secondary;
        stats->primary_hits = (int64_t)c.hits;
        stats->status = (int32_t)c.status;
        stats->nodes_fetched = 0;
        stats->tris_tested = 0;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->device_ms = ms;
    }
    if (stream_end) *stream_end = stream_offset + total;
    return status_to_error(c.status);
}

namespace {

template <class K>
int resident_blocks(K kernel, int otherwise)
{
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kTraceThreads, 0) != cudaSuccess || b < 1) {
        cudaGetLastError();
        b = otherwise;
    }
    return b;
}

template <class SC>
int sub_blocks_per_sm()
{
    static const int per_sm = resident_blocks(k_dist_sub<SC>, 2);
    return per_sm;
}

template <class SC>
int node_blocks_per_sm()
{
    static const int per_sm = resident_blocks(k_dist_node<SC>, 2);
    return per_sm;
}

template <class SC>
int light_blocks_per_sm()
{
    static const int per_sm = resident_blocks(k_dist_lights<SC>, 2);
    return per_sm;
}

template <class SC>
int dist_blocks_per_sm()
{
    static const int per_sm = [] {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (k_dist<true, SC>), kTraceThreads, 0) != cudaSuccess || b < 1) {
            cudaGetLastError();
            b = 2;
        }
        return b;
    }();
    return per_sm;
}

// Worst-case ray tree of a distributed frame: a ray of power a^i * b^j
// (a, b the largest rf and tran of the table) at componant level k spawns,
// while the child's power exceeds 0.1, a reflection set -- one mirror ray,
// or max(diffuse / 4^k, 1) rays at level k + 1 where some reflective
// material spreads -- and likewise a refraction set.  rays: the largest
// tree; depth: its levels below the camera ray; levels: the deepest
// componant level.
struct TreeBound {
    double rays = 0.0;
    int depth = 0, levels = 0;
};

struct TreeBounder {
    double a, b;
    bool mirror_r, spread_r, mirror_t, spread_t;
    int diffuse;
    static constexpr int kI = 4 * RT_MAX_BOUNCES + 2, kK = 18;
    std::vector<double> memo;
    std::vector<int> deep, lev;

    TreeBounder() : memo((size_t)kI * kI * kK, -1.0), deep((size_t)kI * kI * kK, 0), lev((size_t)kI * kI * kK, 0) {}

    // rays of the worst tree below a ray of power a^i b^j at level k
    double f(int i, int j, int k)
    {
        const size_t at = ((size_t)i * kI + (size_t)j) * kK + (size_t)k;
        if (memo[at] >= 0.0) return memo[at];
        const double thr = 0.1 * (1.0 - 1.0e-5);
        double r = 1.0;
        int d = 0, l = k;
        for (int side = 0; side < 2; ++side) {
            const int ni = i + (side == 0), nj = j + (side == 1);
            if (ni + nj >= kI - 1 || !(std::pow(a, ni) * std::pow(b, nj) > thr)) continue;
            const bool mirror = side == 0 ? mirror_r : mirror_t, spread = side == 0 ? spread_r : spread_t;
            double best = 0.0;
            if (mirror) {
                best = f(ni, nj, k);
                const size_t c = ((size_t)ni * kI + (size_t)nj) * kK + (size_t)k;
                d = std::max(d, 1 + deep[c]);
                l = std::max(l, lev[c]);
            }
            if (spread) {
                const int kk = std::min(k + 1, kK - 1);
                const double nr = (double)std::max(diffuse >> (2 * std::min(k, kDistLevels - 1)), 1);
                best = std::max(best, nr * f(ni, nj, kk));
                const size_t c = ((size_t)ni * kI + (size_t)nj) * kK + (size_t)kk;
                d = std::max(d, 1 + deep[c]);
                l = std::max(l, lev[c]);
            }
            r += best;
        }
        memo[at] = r;
        deep[at] = d;
        lev[at] = l;
        return r;
    }
};

TreeBound dist_tree_bound(const rt_material *m, int32_t n, int32_t diffuse)
{
    TreeBounder tb;
    tb.a = tb.b = 0.0;
    tb.mirror_r = tb.spread_r = tb.mirror_t = tb.spread_t = false;
    tb.diffuse = diffuse;
    for (int32_t i = 0; i < n; ++i) {
        tb.a = std::max(tb.a, (double)m[i].rf);
        tb.b = std::max(tb.b, (double)m[i].tran);
        if (m[i].rf > 0.0f) {
            if (diffuse > 0 && m[i].rfd != 0.0f) tb.spread_r = true;
            else tb.mirror_r = true;
        }
        if (m[i].tran > 0.0f) {
            if (diffuse > 0 && m[i].td != 0.0f) tb.spread_t = true;
            else tb.mirror_t = true;
        }
    }
    TreeBound out;
    out.rays = tb.f(0, 0, 0);
    out.depth = tb.deep[0];
    out.levels = tb.lev[0];
    return out;
}

// Shapes of the lights (rt_light_shape): radii finite and >= 0; triangle
// lists in range on point or spot lights of radius 0.
rt_status check_shapes(const rt_scene *s, const rt_light *lights, int32_t nlights, const rt_light_shape *shapes,
                       const char *who)
{
    for (int32_t i = 0; i < nlights && shapes; ++i) {
        const rt_light_shape &sh = shapes[i];
        const std::string w(who);
        if (!(sh.radius >= 0.0f && sh.radius < 3.0e38f))
            return sfail(RT_ERR_INVALID_ARG, (w + ": light radius must be finite and >= 0").c_str());
        if (sh.ntris < 0 || (sh.ntris > 0 && !sh.tris))
            return sfail(RT_ERR_INVALID_ARG, (w + ": bad triangle list of a light").c_str());
        if (sh.ntris > 0 && (sh.radius != 0.0f || (lights[i].kind & 0xff) == RT_LIGHT_DIRECTIONAL))
            return sfail(RT_ERR_INVALID_ARG,
                         (w + ": a triangle-defined light is a point or spot light of radius 0").c_str());
        for (int32_t j = 0; j < sh.ntris; ++j)
            if (sh.tris[j] < 0 || sh.tris[j] >= s->ntris)
                return sfail(RT_ERR_INVALID_ARG, (w + ": light triangle index out of range").c_str());
    }
    return RT_OK;
}

rt_status stream_setup(SoftState &S)
{
    if (S.rng.ptr) return RT_OK;
    // the seeded state (common/common.cc:35-50)
    uint32_t mt[2 * kMtWords];
    mt[0] = 5489u;
    for (int i = 1; i < kMtWords; ++i) mt[i] = 1812433253u * (mt[i - 1] ^ (mt[i - 1] >> 30)) + (uint32_t)i;
    std::memcpy(mt + kMtWords, mt, kMtWords * sizeof(uint32_t));
    RT_CUDA_S(S.rng.reserve(sizeof(mt)), "generator allocation");
    const cudaError_t e = cudaMemcpy(S.rng.ptr, mt, sizeof(mt), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) S.rng.release();
    RT_CUDA_S(e, "generator seed");
    S.refills = 0;
    return RT_OK;
}

// Refills [a, b) are in w.
bool window_holds(const SoftState::Window &w, int64_t a, int64_t b)
{
    return w.count > 0 && a >= w.first && b <= w.first + w.count;
}

// w ends where the generator stands, and refill r is in w or the next.
bool window_leads(const SoftState &S, const SoftState::Window &w, int64_t r)
{
    return w.count > 0 && w.first + w.count == S.refills && r >= w.first && r <= S.refills;
}

size_t refill_bytes(int64_t refills) { return (size_t)refills * kMtWords * sizeof(uint32_t); }

// Window w, with room for `refills`, starts at refill r0 with the words that
// `from` (null: none) holds from there to the generator's position.  Windows
// of short frames hold many of them, so that their words are seldom moved.
constexpr int64_t kMinWindow = 128;
rt_status window_start(SoftState &S, SoftState::Window &w, int64_t r0, int64_t refills,
                       const SoftState::Window *from, cudaStream_t st)
{
    const int64_t n = from ? S.refills - r0 : 0;
    w.count = 0;
    RT_CUDA_S(w.words.reserve(refill_bytes(std::max({refills, n, kMinWindow}))), "stream allocation");
    w.first = r0;
    if (n > 0)
        RT_CUDA_S(cudaMemcpyAsync(w.words.ptr, (const uint32_t *)from->words.ptr + (r0 - from->first) * kMtWords,
                                  refill_bytes(n), cudaMemcpyDeviceToDevice, st),
                  "stream copy");
    w.count = n;
    return RT_OK;
}

// The jump's matrix, once the context has walked (or is about to) as many refills
// as it costs; without memory for it the refills are walked.
constexpr int64_t kJumpWorth = 20000;
constexpr int kJumpRow = 256;   // jumps whose states are kept at a time
constexpr size_t kMatrixWords = (size_t)kMtBits * kMtWords, kPartWords = (size_t)kJumpBlocks * kMtWords;
void jump_setup(SoftState &S, int64_t refills, cudaStream_t st)
{
    if (S.jump_ready || S.walked + refills < kJumpWorth) return;
    if (S.jump.reserve((kMatrixWords + (size_t)(kJumpRow + 1) * kMtWords + 2 * kPartWords) * sizeof(uint32_t)) !=
        cudaSuccess) {
        cudaGetLastError();
        S.walked = 0;   // tried again after as many
        return;
    }
    k_ref_matrix<<<kMtBits, kMtThreads, 0, st>>>((uint32_t *)S.jump.ptr);
    S.jump_ready = true;
}

// Jumps from the generator's state: state k, k jumps on, to states + k * kMtWords,
// k = 0 .. n - 1.
rt_status jump_states(SoftState &S, uint32_t *states, int n, cudaStream_t st)
{
    const uint4 *columns = (const uint4 *)S.jump.ptr;
    uint32_t *parts = (uint32_t *)S.jump.ptr + kMatrixWords + (size_t)(kJumpRow + 1) * kMtWords;
    cudaLaunchAttribute early;   // launched while the jump before ends
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kJumpBlocks);
    cfg.blockDim = dim3(kJumpThreads);
    cfg.stream = st;
    cfg.attrs = &early;
    for (int k = 0; k < n; ++k) {
        const uint4 *state = k == 0 ? (const uint4 *)S.rng.ptr : nullptr;
        const uint4 *from = (const uint4 *)(parts + ((k + 1) & 1) * kPartWords);
        uint4 *to = (uint4 *)(parts + (k & 1) * kPartWords), *at = (uint4 *)(states + (size_t)k * kMtWords);
        cfg.numAttrs = k > 0 ? 1 : 0;
        RT_CUDA_S(cudaLaunchKernelEx(&cfg, k_ref_jump, columns, state, from, to, at, k + 1 < n), "jump launch");
    }
    return RT_OK;
}

// The generator up to refill r1, its words to the end of w (null: skipped).
// Walks are launched at most kMtLaunch refills at a time, a few milliseconds
// each; slices from kJumpLeast on take jumps (a jump costs 4 us, a block's walk of
// kJump refills 60).
constexpr int64_t kMtLaunch = 65536, kJumpLeast = kJump + kJump / 2;
rt_status generate(SoftState &S, SoftState::Window *w, int64_t r1, cudaStream_t st)
{
    uint32_t *state = (uint32_t *)S.rng.ptr;
    int64_t pos = S.refills;
    S.refills = -1;   // whatever fails below, the next frame starts from the seed
    if (r1 - pos >= kJumpLeast) jump_setup(S, r1 - pos, st);
    uint32_t *states = (uint32_t *)S.jump.ptr + kMatrixWords;
    while (pos < r1) {
        uint32_t *out = w ? (uint32_t *)w->words.ptr + (pos - w->first) * kMtWords : nullptr;
        int64_t n = r1 - pos;
        if (!S.jump_ready || n < kJumpLeast) {
            n = std::min(n, kMtLaunch);
            S.walked += n;
            if (w) k_ref_stream<true><<<1, kMtThreads, 0, st>>>(state, n, (int32_t)n, out, state);
            else k_ref_stream<false><<<1, kMtThreads, 0, st>>>(state, n, (int32_t)n, nullptr, state);
        } else if (w) {
            n = std::min(n, (int64_t)kJumpRow * kJump);
            const int blocks = (int)((n + kJump - 1) / kJump);
            const rt_status rc = jump_states(S, states, blocks, st);
            if (rc != RT_OK) return rc;
            k_ref_stream<true><<<blocks, kMtThreads, 0, st>>>(states, n, kJump, out, state);
        } else {
            const int jumps = (int)std::min(n / kJump, (int64_t)kJumpRow);
            n = (int64_t)jumps * kJump;
            const rt_status rc = jump_states(S, states, jumps + 1, st);
            if (rc != RT_OK) return rc;
            RT_CUDA_S(cudaMemcpyAsync(state, states + (size_t)jumps * kMtWords, kMtWords * sizeof(uint32_t),
                                      cudaMemcpyDeviceToDevice, st),
                      "generator state");
        }
        pos += n;
    }
    RT_CUDA_S(cudaGetLastError(), "generator launch");
    S.refills = pos;
    if (w) w->count = pos - w->first;
    return RT_OK;
}

// The frame's numbers [offset, offset + total) of the reference's stream as
// words on the device (ref_number), kept while later frames fall inside their
// window; *rnd points at number offset.  Of frames that each start where the
// one before ended, only the first can start from the seed: one of the windows
// always leads from the last one's end on.
rt_status stream_window(SoftState &S, int64_t offset, int64_t total, cudaStream_t st, const uint32_t **rnd)
{
    *rnd = nullptr;
    if (total <= 0) return RT_OK;
    rt_status rc = stream_setup(S);
    if (rc != RT_OK) return rc;
    const int64_t r0 = offset / kMtWords, r1 = (offset + total + kMtWords - 1) / kMtWords;
    const int a = S.cur, b = S.cur ^ 1;
    int use = window_holds(S.win[a], r0, r1) ? a : window_holds(S.win[b], r0, r1) ? b : -1;
    if (use < 0) {
        const int lead = window_leads(S, S.win[a], r0) ? a : window_leads(S, S.win[b], r0) ? b : -1;
        if (lead >= 0 && refill_bytes(r1 - S.win[lead].first) <= S.win[lead].words.cap) {
            use = lead;
        } else if (lead >= 0) {
            use = lead ^ 1;
            rc = window_start(S, S.win[use], r0, r1 - r0, &S.win[lead], st);
        } else {
            use = b;
            rc = window_start(S, S.win[use], r0, r1 - r0, nullptr, st);
            if (rc == RT_OK && (S.refills < 0 || S.refills > r0)) {
                S.refills = -1;
                uint32_t *state = (uint32_t *)S.rng.ptr;
                RT_CUDA_S(cudaMemcpyAsync(state, state + kMtWords, kMtWords * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                                          st),
                          "generator reset");
                S.refills = 0;
            }
            if (rc == RT_OK) rc = generate(S, nullptr, r0, st);
        }
        if (rc == RT_OK) rc = generate(S, &S.win[use], r1, st);
        if (rc != RT_OK) return rc;
    }
    S.cur = use;
    *rnd = (const uint32_t *)S.win[use].words.ptr + (offset - S.win[use].first * kMtWords);
    return RT_OK;
}

// The subtrees of a frame's items (on the device already): a piece of at most
// kDistPiece items at a time, level by level, the nodes below them in a pool of
// one for each item and one for each ray of a set at an item, at most
// kDistPoolPerItem (frames of the glass scene make 0.92 an item with sets of 1 or
// 4 rays, 3.7 with 16): 132 bytes a node, the items' colours and sets and a
// piece's hits beside them.  They take at most half of the device's free memory;
// without room for all of them the items are walked whole.
constexpr int32_t kDistPiece = 1 << 22;
constexpr int32_t kDistPoolPerItem = 4;

rt_status trace_items(SoftState &S, rt_scene *s, const CameraView &cv, const LightSet &ls, const MaterialTable &mt,
                      const DistLights &dl, const DistParams &dp, const SceneView &sv, DistLists lists, int levels,
                      rt_context *ctx, cudaStream_t st)
{
    const int32_t n = lists.count(), piece = std::min(n, kDistPiece);
    DistCounts *dc = (DistCounts *)((int32_t *)S.nitems.ptr + 2);
    lists.items = (DistItem *)S.items.ptr;
    constexpr size_t kNode = sizeof(DistItem) + sizeof(float4) + sizeof(int4) + sizeof(DistHit) + sizeof(int32_t);
    const int64_t per_item = std::min(1 + std::max(dp.diffuse >> 2, 1), kDistPoolPerItem);
    int64_t pool = levels < 2 ? 0 : std::min(per_item * piece, ((int64_t)1 << 31) - 1 - 2 * (int64_t)lists.cap);
    const size_t held = S.nodes.cap + S.item_c.cap + S.node_sets.cap + S.node_hits.cap + S.node_over.cap;
    if ((size_t)pool * kNode > held) {   // more than these buffers were ever asked for, maybe
        size_t free_b = 0, all_b = 0;
        if (cudaMemGetInfo(&free_b, &all_b) != cudaSuccess) free_b = 0;
        pool = std::min(pool, (int64_t)((free_b + held) / 2 / (kNode + kNode / 4)));
    }
    lists.pool = (int32_t)pool;
    const size_t entries = 2 * (size_t)lists.cap + (size_t)pool;
    const size_t nodes = (size_t)piece + (size_t)pool;   // of a piece, at most
    const int4 *area = (const int4 *)S.area.ptr;
    const float *lut = (const float *)S.lut.ptr;
    const bool walk = S.nodes.reserve((size_t)pool * sizeof(DistItem)) != cudaSuccess ||
                      S.item_c.reserve(entries * sizeof(float4)) != cudaSuccess ||
                      S.node_sets.reserve(entries * sizeof(int4)) != cudaSuccess ||
                      S.node_hits.reserve(nodes * sizeof(DistHit)) != cudaSuccess ||
                      S.node_over.reserve(nodes * sizeof(int32_t)) != cudaSuccess;
    if (walk) {
        cudaGetLastError();
        for (DevBuf *b : {&S.nodes, &S.item_c, &S.node_sets, &S.node_hits, &S.node_over}) b->release();
        lists.pool = 0;
        RT_CUDA_S(S.item_c.reserve(2 * (size_t)lists.cap * sizeof(float4)), "item colour allocation");
    }
    lists.nodes = (DistItem *)S.nodes.ptr;
    float4 *item_c = (float4 *)S.item_c.ptr;
    int4 *sets = (int4 *)S.node_sets.ptr;
    DistHit *hits = (DistHit *)S.node_hits.ptr;
    int32_t *over = (int32_t *)S.node_over.ptr;
    for (int64_t at = 0; at < n; at += walk ? n : piece) {
        const int32_t v0 = (int32_t)at, v1 = (int32_t)std::min<int64_t>(n, at + piece);
        RT_CUDA_S(cudaMemsetAsync(dc, 0, sizeof(DistCounts), st), "node counter clear");
        with_scene(sv, [&](const auto &view) {
            using SC = std::decay_t<decltype(view)>;
            if (!walk) {
                for (int k = 0; k < levels; ++k)
                    k_dist_node<SC><<<node_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
                        view, cv, ls, mt, dl, dp, lut, lists, v0, v1, k, k == levels - 1, sets, item_c, hits, over,
                        dc, ctx->d_counters);
                k_dist_lights<SC><<<light_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
                    view, ls, mt, dl, dp, area, s->d_verts, lut, lists, hits, item_c, dc, ctx->d_counters);
            }
            k_dist_sub<SC><<<sub_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
                view, cv, ls, mt, dl, dp, area, s->d_verts, lut, lists, walk ? nullptr : over, &dc->over,
                &dc->work_over, item_c, ctx->d_counters);
            if (!walk)
                for (int k = levels - 1; k-- > 0;)
                    k_dist_gather<<<ctx->sm_count * 8, 256, 0, st>>>(mt, lists, v0, v1, k, sets, item_c, dc);
        });
        RT_CUDA_S(cudaGetLastError(), "subtree launch");
    }
    return RT_OK;
}

}  // namespace

extern "C" rt_status rt_render_distributed(rt_scene *s, const rt_camera *camera, const rt_light *lights,
                                           int32_t nlights, const rt_light_shape *shapes,
                                           const rt_material *materials, int32_t nmaterials,
                                           const rt_sampling *sampling, uint8_t *rgb_out, float *rgb_f32,
                                           int64_t *stream_end, rt_render_stats *stats)
{
    if (!s || !camera || !materials || !sampling || (!rgb_out && !rgb_f32))
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: NULL argument");
    if (camera->xres <= 0 || camera->yres <= 0 || (int64_t)camera->xres * camera->yres > (int64_t)1 << 28)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: camera resolution out of range");
    if (nlights < 0 || nlights > RT_MAX_LIGHTS || (nlights > 0 && !lights))
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: light count out of range");
    if (nmaterials < 1 || nmaterials > RT_MAX_MATERIALS)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: material count must be 1..RT_MAX_MATERIALS");
    const rt_sampling smp = *sampling;
    if (smp.soft_samples < 1 || smp.soft_samples > RT_MAX_SOFT_SAMPLES || smp.diffuse_samples < 0 ||
        smp.diffuse_samples > RT_MAX_SOFT_SAMPLES)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: sample counts out of range");
    if (smp.stream != RT_STREAM_REFERENCE && smp.stream != RT_STREAM_PIXEL)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: unknown stream");
    if (smp.stream == RT_STREAM_REFERENCE && smp.stream_offset < 0)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: negative stream offset");
    bool tree = false, spread = false;
    for (int32_t i = 0; i < nmaterials; ++i) {
        const rt_material &m = materials[i];
        if (!(m.rf >= 0.0f && m.rf < 1.0f) || !(m.tran >= 0.0f && m.tran < 1.0f))
            return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: reflectivity and transparency must be in [0, 1)");
        if (m.tran > 0.0f && !(m.ri > 0.0f && m.ri < 3.0e38f))
            return sfail(RT_ERR_INVALID_ARG,
                         "rt_render_distributed: a transparent material needs a finite positive refractive index");
        if (!(std::fabs(m.rfd) < 3.0e38f) || !(std::fabs(m.td) < 3.0e38f))
            return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: diffuse spreads must be finite");
        tree = tree || m.rf > 0.0f || m.tran > 0.0f;
        spread = spread || (smp.diffuse_samples > 0 && ((m.rf > 0.0f && m.rfd != 0.0f) || (m.tran > 0.0f && m.td != 0.0f)));
    }
    if (spread && smp.stream == RT_STREAM_REFERENCE)
        return sfail(RT_ERR_INVALID_ARG,
                     "rt_render_distributed: diffuse rays draw the reference's stream in an order one pass cannot "
                     "replay in parallel (a pixel's count depends on where earlier random rays landed); use "
                     "RT_STREAM_PIXEL");
    {
        const rt_status st = check_shapes(s, lights, nlights, shapes, "rt_render_distributed");
        if (st != RT_OK) return st;
    }
    if (!s->built) return sfail(RT_ERR_NOT_BUILT, "rt_render_distributed: hierarchy not built");
    if (s->mat_max >= nmaterials)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: the scene's material indices exceed the table");
    // without ray trees or diffuse rays, the reference-stream frame is the
    // soft-shadow frame
    if (!tree && smp.stream == RT_STREAM_REFERENCE)
        return rt_render_soft_shadows(s, camera, lights, nlights, shapes, materials, nmaterials, smp.soft_samples,
                                      smp.stream_offset, rgb_out, rgb_f32, stream_end, stats);
    const TreeBound tb = dist_tree_bound(materials, nmaterials, smp.diffuse_samples);
    if (tb.depth > RT_MAX_BOUNCES || tb.rays > (double)RT_MAX_TREE_RAYS || tb.levels > 15)
        return sfail(RT_ERR_INVALID_ARG, "rt_render_distributed: the materials allow more than RT_MAX_BOUNCES levels "
                                         "or RT_MAX_TREE_RAYS rays per pixel");

    rt_context *ctx = s->ctx;
    SGuard g(ctx->device);
    if (!ctx->soft) {
        ctx->soft = new (std::nothrow) SoftState();
        if (!ctx->soft) return sfail(RT_ERR_OUT_OF_MEMORY, "rt_render_distributed: state allocation");
        ctx->soft->device = ctx->device;
    }
    SoftState &S = *ctx->soft;
    cudaStream_t st = ctx->stream;
    if (!S.lut_ready) {
        std::vector<float> lut(kCosLutSize);
        for (int i = 0; i < kCosLutSize; ++i)
            lut[i] = (float)std::cos((double)((((float)i * 2.0f) * kRefPi) / (float)kCosLutSize));
        RT_CUDA_S(S.lut.reserve(kCosLutSize * sizeof(float)), "cosine table allocation");
        RT_CUDA_S(cudaMemcpy(S.lut.ptr, lut.data(), kCosLutSize * sizeof(float), cudaMemcpyHostToDevice),
                  "cosine table copy");
        S.lut_ready = true;
    }
    // lights: per componant level, the rays of every triangle-defined
    // light and the numbers a hit draws
    LightSet ls;
    ls.n = nlights;
    ls.fast_pow = 0;
    DistLights dl = {};
    std::vector<int4> area_rays;
    for (int i = 0; i < nlights; ++i) {
        ls.l[i] = make_light_view(lights[i]);
        ls.l[i].radius = shapes ? shapes[i].radius : 0.0f;
        if (ls.l[i].kind == RT_LIGHT_DIRECTIONAL) continue;
        for (int k = 0; k < kDistLevels; ++k) {
            const int32_t n = std::max(smp.soft_samples >> (2 * k), 1);
            if (n == 1) continue;
            if (shapes && shapes[i].ntris > 0) {
                const int32_t nt = shapes[i].ntris;
                std::vector<int32_t> cnt((size_t)nt);
                const int32_t made = area_light_rays(nt, n, cnt.data());
                if (made < n)
                    return sfail(RT_ERR_INVALID_ARG,
                                 "rt_render_distributed: a triangle-defined light makes fewer rays than asked");
                dl.first[i][k] = (int32_t)area_rays.size();
                dl.made[i][k] = made;
                dl.draws[i][k] = 2 * made;
                for (int32_t j = 0; j < nt; ++j)
                    for (int32_t q = 0; q < cnt[(size_t)j]; ++q)
                        area_rays.push_back(make_int4(shapes[i].tris[j], cnt[(size_t)j], q, 0));
            } else {
                dl.draws[i][k] = 3 * n;
            }
        }
    }
    if (!area_rays.empty()) {
        RT_CUDA_S(S.area.reserve(area_rays.size() * sizeof(int4)), "light ray table allocation");
        RT_CUDA_S(cudaMemcpyAsync(S.area.ptr, area_rays.data(), area_rays.size() * sizeof(int4), cudaMemcpyHostToDevice,
                                  st),
                  "light ray table copy");
    }
    MaterialTable mt;
    mt.n = nmaterials;
    DistParams dp = {};
    dp.soft = smp.soft_samples;
    dp.diffuse = smp.diffuse_samples;
    dp.pixel_stream = smp.stream == RT_STREAM_PIXEL ? 1 : 0;
    dp.key0 = (uint32_t)smp.seed;
    dp.key1 = (uint32_t)(smp.seed >> 32);
    // walk steps per pixel: every ray of the tree and every light's rays at each of its hits
    dp.max_steps = (int32_t)std::min(8.0 * tb.rays * (1.0 + (double)nlights * smp.soft_samples) + 64.0, 1.0e9);
    for (int i = 0; i < nmaterials; ++i) {
        mt.m[i] = make_material_view(materials[i]);
        dp.rfd[i] = materials[i].rfd;
        dp.td[i] = materials[i].td;
    }
    const SceneView sv = scene_view(s);
    const CameraView cv = make_camera_view(*camera);
    const size_t npix = (size_t)camera->xres * (size_t)camera->yres;

    RT_CUDA_S(cudaMemsetAsync(ctx->d_counters, 0, sizeof(Counters), st), "counter clear");
    RT_CUDA_S(cudaEventRecord(ctx->ev0, st), "event record");
    const uint32_t *rnd = nullptr;
    int64_t total = 0;
    if (smp.stream == RT_STREAM_REFERENCE) {
        // counting pass, scan, the frame's slice of the stream
        RT_CUDA_S(S.counts.reserve(npix * sizeof(int64_t)), "count allocation");
        RT_CUDA_S(S.prefix64.reserve(npix * sizeof(int64_t)), "prefix allocation");
        size_t scan_bytes = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const int64_t *)S.counts.ptr, (int64_t *)S.prefix64.ptr,
                                      (int)npix, st);
        RT_CUDA_S(S.scan64_temp.reserve(scan_bytes), "scan scratch allocation");
        with_scene(sv, [&](const auto &view) {
            using SC = std::decay_t<decltype(view)>;
            k_dist<false, SC><<<dist_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
                view, cv, ls, mt, dl, dp, (const int4 *)S.area.ptr, s->d_verts, (const float *)S.lut.ptr, nullptr, 0,
                nullptr, (int64_t *)S.counts.ptr, nullptr, nullptr, ctx->d_counters);
        });
        RT_CUDA_S(cudaGetLastError(), "counting launch");
        cub::DeviceScan::ExclusiveSum(S.scan64_temp.ptr, scan_bytes, (const int64_t *)S.counts.ptr,
                                      (int64_t *)S.prefix64.ptr, (int)npix, st);
        RT_CUDA_S(cudaGetLastError(), "scan launch");
        int64_t last[2];
        RT_CUDA_S(cudaMemcpyAsync(&last[0], (const int64_t *)S.prefix64.ptr + (npix - 1), sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, st),
                  "prefix read");
        RT_CUDA_S(cudaMemcpyAsync(&last[1], (const int64_t *)S.counts.ptr + (npix - 1), sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, st),
                  "count read");
        RT_CUDA_S(cudaStreamSynchronize(st), "synchronize");
        total = last[0] + last[1];
        const rt_status wst = stream_window(S, smp.stream_offset, total, st, &rnd);
        if (wst != RT_OK) return wst;
        RT_CUDA_S(cudaMemsetAsync(&ctx->d_counters->work, 0, sizeof(int), st), "work counter clear");
    }
    const bool rgb_host = rgb_out && !is_device_ptr(rgb_out);
    const bool f_host = rgb_f32 && !is_device_ptr(rgb_f32);
    uint8_t *d_rgb = rgb_out;
    float *d_f = rgb_f32;
    if (rgb_host) {
        RT_CUDA_S(ctx->stage_a.reserve(npix * 3), "staging allocation");
        d_rgb = (uint8_t *)ctx->stage_a.ptr;
    }
    if (f_host) {
        RT_CUDA_S(ctx->fimg.reserve(npix * 3 * sizeof(float)), "float frame allocation");
        d_f = (float *)ctx->fimg.ptr;
    }
    // per-pixel streams with ray trees: the camera rays' nodes, then their
    // sets' subtrees as separate items, then the pixels' colours
    const int64_t per_pixel = 2 * (int64_t)std::max(smp.diffuse_samples, 1);   // items a pixel can hand out
    const bool split = smp.stream == RT_STREAM_PIXEL && tree && (int64_t)npix * per_pixel < ((int64_t)1 << 31);
    if (split) {
        RT_CUDA_S(S.root_c.reserve(npix * sizeof(float4)), "node allocation");
        RT_CUDA_S(S.root_sets.reserve(npix * sizeof(int4)), "node allocation");
        RT_CUDA_S(S.nitems.reserve(2 * sizeof(int32_t) + sizeof(DistCounts)), "item counter allocation");
        // items per list (reflection sets, refraction sets)
        int64_t cap = std::min((int64_t)npix * per_pixel / 2, std::max(S.item_cap, (int64_t)npix * 2));
        int32_t n[2] = {0, 0};
        for (int attempt = 0; attempt < 2; ++attempt) {
            RT_CUDA_S(S.items.reserve(2 * (size_t)cap * sizeof(DistItem)), "item allocation");
            RT_CUDA_S(cudaMemsetAsync(ctx->d_counters, 0, sizeof(Counters), st), "counter clear");
            RT_CUDA_S(cudaMemsetAsync(S.nitems.ptr, 0, 2 * sizeof(int32_t), st), "item counter clear");
            with_scene(sv, [&](const auto &view) {
                using SC = std::decay_t<decltype(view)>;
                k_dist_root<SC><<<dist_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
                    view, cv, ls, mt, dl, dp, (const int4 *)S.area.ptr, s->d_verts, (const float *)S.lut.ptr,
                    (float4 *)S.root_c.ptr, (int4 *)S.root_sets.ptr, (DistItem *)S.items.ptr, (int32_t)cap,
                    (int32_t *)S.nitems.ptr, ctx->d_counters);
            });
            RT_CUDA_S(cudaGetLastError(), "node launch");
            RT_CUDA_S(cudaMemcpyAsync(n, S.nitems.ptr, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, st),
                      "item count read");
            RT_CUDA_S(cudaStreamSynchronize(st), "synchronize");
            if (n[0] >= 0 && n[1] >= 0 && n[0] <= cap && n[1] <= cap) break;
            if (n[0] < 0 || n[1] < 0 || attempt == 1)
                return sfail(RT_ERR_INTERNAL, "rt_render_distributed: item count out of range");
            const int64_t need = std::max(n[0], n[1]);
            cap = std::min((int64_t)npix * per_pixel / 2, need + need / 8);   // grow to fit and run again
        }
        S.item_cap = cap;
        if (n[0] + n[1] > 0) {
            const rt_status wst = trace_items(S, s, cv, ls, mt, dl, dp, sv, DistLists{n[0], n[1], (int32_t)cap, 0, nullptr, nullptr},
                                              std::max(tb.depth, 1), ctx, st);
            if (wst != RT_OK) return wst;
        }
        k_dist_combine<<<ctx->sm_count * 8, 256, 0, st>>>(cv, mt, (const float4 *)S.root_c.ptr,
                                                          (const int4 *)S.root_sets.ptr, (const float4 *)S.item_c.ptr,
                                                          n[0], n[1], (int32_t)cap, d_rgb, d_f, ctx->d_counters);
    } else {
        with_scene(sv, [&](const auto &view) {
            using SC = std::decay_t<decltype(view)>;
            k_dist<true, SC><<<dist_blocks_per_sm<SC>() * ctx->sm_count, kTraceThreads, 0, st>>>(
                view, cv, ls, mt, dl, dp, (const int4 *)S.area.ptr, s->d_verts, (const float *)S.lut.ptr, rnd, total,
                (const int64_t *)S.prefix64.ptr, nullptr, d_rgb, d_f, ctx->d_counters);
        });
    }
    RT_CUDA_S(cudaGetLastError(), "shade launch");
    RT_CUDA_S(cudaEventRecord(ctx->ev1, st), "event record");
    if (rgb_host) RT_CUDA_S(cudaMemcpyAsync(rgb_out, d_rgb, npix * 3, cudaMemcpyDeviceToHost, st), "rgb copy");
    if (f_host)
        RT_CUDA_S(cudaMemcpyAsync(rgb_f32, d_f, npix * 3 * sizeof(float), cudaMemcpyDeviceToHost, st), "image copy");
    Counters c;
    RT_CUDA_S(cudaMemcpyAsync(&c, ctx->d_counters, sizeof(Counters), cudaMemcpyDeviceToHost, st), "counter read");
    RT_CUDA_S(cudaStreamSynchronize(st), "synchronize");
    if (stats) {
        stats->primary_rays = (int64_t)c.primary;
        stats->secondary_rays = (int64_t)c.secondary;
        stats->primary_hits = (int64_t)c.hits;
        stats->status = (int32_t)c.status;
        stats->nodes_fetched = 0;
        stats->tris_tested = 0;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        stats->device_ms = ms;
    }
    if (stream_end)
        *stream_end = smp.stream == RT_STREAM_REFERENCE ? smp.stream_offset + total : (int64_t)c.drawn;
    return status_to_error(c.status);
}
