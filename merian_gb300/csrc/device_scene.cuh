// Device view of a scene in HBM and the CWBVH traversal.
//
// Traversal replaces the hardware ray query merian issues through TraceRayInline with
// RAY_FLAG_CULL_BACK_FACING_TRIANGLES (acceleration-structure.slang:59-72) on ForceOpaque
// instances (scene.cpp:1849-1850). Closest hit over triangles whose instance mask intersects the
// ray mask, back faces culled unless the geometry is TwoSided, the front face swapped by
// FlipFacing (scene.cpp:1841-1848). Ties at equal t go to the smallest (geometry, primitive), so
// the result does not depend on the BVH layout.
#pragma once

#include "device_math.cuh"

#include <type_traits>
#include "gbpt.h"
#include "runtime.h"

namespace gbpt {

struct GeomGPU {
    uint32_t first_vertex, first_triangle, material, flags;
};

// per-triangle flag word (third float4 of a triangle record)
constexpr uint32_t kTriTwoSided = 1u << 8;
constexpr uint32_t kTriFlip = 1u << 9;
constexpr uint32_t kTriAlpha = 1u << 10; // non-opaque geometry: candidate hits run the alpha test
constexpr uint32_t kTriKeyShift = 11;    // material-sort key of the geometry, 2 bits
constexpr uint32_t kTriKey = 3u << kTriKeyShift;
constexpr uint32_t kRayAny = 1u << 7;

// What a traversal looks for: every ray's closest hit, every ray's first hit, or per ray the one
// its axis word says (kRayAny).
enum TraceMode { kTraceClosest, kTraceAny, kTraceMixed };

struct DevScene {
    const uint4* __restrict__ nodes;  // 5 per CWBVH node
    const float4* __restrict__ tris;  // 3 per triangle record and copy
    uint32_t tri_stride;              // float4 from one copy of the records to the next
    const uint32_t* __restrict__ verts; // gbpt_packed_vertex as 6 words
    const uint32_t* __restrict__ idx;
    const uint4* __restrict__ tri_verts; // 5 per triangle (3 vertices, padded) or null
    const GeomGPU* __restrict__ geoms;
    const float4* __restrict__ mats;  // gbpt_material as 5 float4
    uint32_t geom_count;
    // environment
    const float4* __restrict__ env;
    uint32_t ew, eh;
    float env_m[9];
    float env_intensity;
    const float* __restrict__ env_marg; // eh + 1, normalised
    const float* __restrict__ env_cond; // eh * (ew + 1), normalised per row
    const float* __restrict__ env_func; // eh * ew
    float env_func_int;
    // emissive triangles
    const float4* __restrict__ light_tris; // 3 per light: v0 (w = geometry), v1, v2
    const float* __restrict__ light_cdf;   // n_lights, inclusive, normalised
    uint32_t n_lights;
    float light_total; // sum of area x luminance
    float p_env;       // probability of choosing the environment in NEE
    // guide tables of the light, marginal and conditional CDFs: entry k is the upper bound of
    // k / G (G a power of two), so the search for u covers [guide[k], guide[k + 1]] only
    const uint32_t* __restrict__ light_guide;
    const uint2* __restrict__ env_rows; // alias tables (GBPT_ENV_ALIAS): per row, per texel
    const uint2* __restrict__ env_cols;
    const uint32_t* __restrict__ env_marg_guide;
    const uint32_t* __restrict__ env_cond_guide; // G + 1 per row
    uint32_t light_g, env_marg_g, env_cond_g;
    // two-level scenes: instance records (7 float4 each), n_inst = 0 for single-level scenes
    const float4* __restrict__ inst;
    uint32_t n_inst;
    // RGBA8 textures: texels of all textures, (first texel, width, height, sRGB) per texture and
    // the sRGB-to-linear table
    const uchar4* __restrict__ tex;
    const uint4* __restrict__ tex_info;
    uint32_t n_tex;
    const float* __restrict__ srgb_lut;
};

struct Hit {
    float t, u, v;
    uint32_t prim, geom; // geom = 0xFFFFFFFF on miss (the scene-global geometry index)
    uint32_t inst;       // instance index of two-level scenes, 0xFFFFFFFF otherwise
};

// ---- alpha test of non-opaque geometry (material-system.slang:28-38, scene.slang:500-519) --------
// The material's alpha texture, bilinear with repeat addressing at level 0, at the candidate hit's
// interpolated uv; alpha below 0.5 (merian_alpha_test_threshold) discards the candidate. Rounded
// operations in a fixed order, shared with the oracle, so the decision is bit-identical.
constexpr float kAlphaThreshold = 0.5f;

GBPT_DI float texture_alpha(const DevScene& sc, uint32_t t, float u, float v) {
    const uint4 info = __ldg(&sc.tex_info[t]);
    const int w = (int)info.y, h = (int)info.z;
    if (!(fabsf(u) < 65536.0f)) u = 0.0f; // half uvs: only NaN / inf are out of range
    if (!(fabsf(v) < 65536.0f)) v = 0.0f;
    const float x = __fsub_rn(__fmul_rn(u, (float)w), 0.5f);
    const float y = __fsub_rn(__fmul_rn(v, (float)h), 0.5f);
    const float fx = floorf(x), fy = floorf(y);
    const float a = __fsub_rn(x, fx), b = __fsub_rn(y, fy);
    const int ix = (int)fx, iy = (int)fy;
    const int x0 = ((ix % w) + w) % w, x1 = (((ix + 1) % w) + w) % w;
    const int y0 = ((iy % h) + h) % h, y1 = (((iy + 1) % h) + h) % h;
    const uchar4* base = sc.tex + info.x;
    auto alpha = [&](int xx, int yy) {
        return __fmul_rn((float)__ldg(&base[(size_t)yy * w + xx]).w, 1.0f / 255.0f);
    };
    const float ia = __fsub_rn(1.0f, a), ib = __fsub_rn(1.0f, b);
    const float top = __fadd_rn(__fmul_rn(alpha(x0, y0), ia), __fmul_rn(alpha(x1, y0), a));
    const float bot = __fadd_rn(__fmul_rn(alpha(x0, y1), ia), __fmul_rn(alpha(x1, y1), a));
    return __fadd_rn(__fmul_rn(top, ib), __fmul_rn(bot, b));
}

// True when the candidate hit (geometry, primitive, barycentrics u, v) is transparent.
GBPT_DI bool alpha_discard(const DevScene& sc, uint32_t geom, uint32_t prim, float bu, float bv) {
    const GeomGPU g = sc.geoms[geom];
    const int tex = __float_as_int(__ldg(&sc.mats[5ull * g.material + 4]).y);
    if (tex < 0 || (uint32_t)tex >= sc.n_tex) return false;
    const uint32_t tri = g.first_triangle + prim;
    float uvx[3], uvy[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t* v =
            sc.tri_verts ? (const uint32_t*)(sc.tri_verts + 5ull * tri) + 6 * k
                         : sc.verts + 6ull * (g.first_vertex + __ldg(&sc.idx[3 * tri + k]));
        const uint32_t uv = __ldg(v + 4);
        uvx[k] = __half2float(__ushort_as_half((unsigned short)(uv & 0xFFFFu)));
        uvy[k] = __half2float(__ushort_as_half((unsigned short)(uv >> 16)));
    }
    const float b0 = __fsub_rn(__fsub_rn(1.0f, bu), bv);
    const float u = __fadd_rn(__fadd_rn(__fmul_rn(b0, uvx[0]), __fmul_rn(bu, uvx[1])),
                              __fmul_rn(bv, uvx[2]));
    const float v = __fadd_rn(__fadd_rn(__fmul_rn(b0, uvy[0]), __fmul_rn(bu, uvy[1])),
                              __fmul_rn(bv, uvy[2]));
    return texture_alpha(sc, (uint32_t)tex, u, v) < kAlphaThreshold;
}

// ---- watertight test (Woop, Benthin, Wald 2013) -------------------------------------------------
// Explicit round-to-nearest intrinsics (no FMA contraction) so the float result equals the
// host oracle's bit for bit.
struct RayPre {
    // the axes kx, ky, kz in bits 0-1, 2-3, 4-5 (kx = kz + 1, ky = kz + 2 mod 3); bit 6 when the
    // direction is negative along kz. The watertight test's paper swaps kx and ky for that sign
    // to keep the winding; keeping one frame per kz negates U, V, W, det and T instead, which
    // leaves t, u and v unchanged and flips the facing. The traversal keeps more of the ray in
    // the same register (set_ray, TraceState): 7 - the direction octant in bits 8-10, the closest
    // hit's material-sort key in bits 11-12 (kTriKey, as in the triangle's flag word), the ray's
    // instance mask in bits 16-23 and the stack depth in bits 24-31; bit 7 marks a first-hit ray
    // among closest-hit ones (kRayAny).
    uint32_t k;
    GBPT_DI int kz() const { return (int)((k >> 4) & 3u); }
    GBPT_DI uint32_t oct_inv() const { return (k >> 8) & 7u; }
    GBPT_DI uint32_t mask() const { return (k >> 16) & 0xFFu; }
};
// The rest of the test's ray: the shear, and the origin permuted to (kx, ky, kz).
struct RayShear {
    float Sx, Sy, Sz;
    float ox, oy, oz;
};
GBPT_DI float pick(float x, float y, float z, int k) { return k == 0 ? x : (k == 1 ? y : z); }
GBPT_DI RayPre ray_pre(float3 o, float3 d, RayShear& r) {
    RayPre p;
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    const int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    const int kx = kz == 2 ? 0 : kz + 1;
    const int ky = kx == 2 ? 0 : kx + 1;
    const float dkz = pick(d.x, d.y, d.z, kz);
    p.k = (uint32_t)kx | ((uint32_t)ky << 2) | ((uint32_t)kz << 4) | (dkz < 0.0f ? 64u : 0u);
    r.Sx = __fdiv_rn(pick(d.x, d.y, d.z, kx), dkz);
    r.Sy = __fdiv_rn(pick(d.x, d.y, d.z, ky), dkz);
    r.Sz = __frcp_rn(dkz);
    r.ox = pick(o.x, o.y, o.z, kx);
    r.oy = pick(o.x, o.y, o.z, ky);
    r.oz = pick(o.x, o.y, o.z, kz);
    return p;
}

// Returns true with t, u, v when hit within [tmin, tmax] on an accepted face.
// The barycentrics are returned undivided (u_out = V, v_out = W, det_out = det): the caller divides
// them once for the final hit instead of at every accepted candidate.
GBPT_DI bool intersect_tri(const RayPre& p, const RayShear& r, float4 a4, float4 b4, float4 c4,
                           uint32_t tflags, float tmin, float tmax, float& t_out, float& u_out,
                           float& v_out, float& det_out) {
    // the record copy of axis kz holds the coordinates (kx, ky, kz)
    const float Akx = __fsub_rn(a4.x, r.ox);
    const float Aky = __fsub_rn(a4.y, r.oy);
    const float Akz = __fsub_rn(a4.z, r.oz);
    const float Bkx = __fsub_rn(b4.x, r.ox);
    const float Bky = __fsub_rn(b4.y, r.oy);
    const float Bkz = __fsub_rn(b4.z, r.oz);
    const float Ckx = __fsub_rn(c4.x, r.ox);
    const float Cky = __fsub_rn(c4.y, r.oy);
    const float Ckz = __fsub_rn(c4.z, r.oz);
    const float Ax = __fsub_rn(Akx, __fmul_rn(r.Sx, Akz));
    const float Ay = __fsub_rn(Aky, __fmul_rn(r.Sy, Akz));
    const float Bx = __fsub_rn(Bkx, __fmul_rn(r.Sx, Bkz));
    const float By = __fsub_rn(Bky, __fmul_rn(r.Sy, Bkz));
    const float Cx = __fsub_rn(Ckx, __fmul_rn(r.Sx, Ckz));
    const float Cy = __fsub_rn(Cky, __fmul_rn(r.Sy, Ckz));
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = __double2float_rn(__dsub_rn(__dmul_rn((double)Cx, (double)By), __dmul_rn((double)Cy, (double)Bx)));
        V = __double2float_rn(__dsub_rn(__dmul_rn((double)Ax, (double)Cy), __dmul_rn((double)Ay, (double)Cx)));
        W = __double2float_rn(__dsub_rn(__dmul_rn((double)Bx, (double)Ay), __dmul_rn((double)By, (double)Ax)));
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    if (!(tflags & kTriTwoSided)) {
        const bool front = (det > 0.0f) != ((p.k & 64u) != 0u);
        if (front == ((tflags & kTriFlip) != 0)) return false;
    }
    const float Az = __fmul_rn(r.Sz, Akz);
    const float Bz = __fmul_rn(r.Sz, Bkz);
    const float Cz = __fmul_rn(r.Sz, Ckz);
    const float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
    const float t = __fdiv_rn(T, det);
    if (!(t >= tmin && t <= tmax)) return false;
    t_out = t;
    u_out = V;
    v_out = W;
    det_out = det;
    return true;
}

// ---- CWBVH traversal ----------------------------------------------------------------------------
// Traversal stack entries per ray. The builder bounds the tree depth (24 levels), which with
// instance entries stays below the default. A build with a smaller
// GBPT_STACK_SIZE makes deep traversals overflow: the overflow sets the kernels' error word
// (GBPT_ERR_DEVICE on the host) and finishes the ray with what it found, never a fault, so the
// error path can be exercised on purpose.
#ifndef GBPT_STACK_SIZE
#define GBPT_STACK_SIZE 48
#endif
constexpr int kStackSize = GBPT_STACK_SIZE;
static_assert(kStackSize >= 1, "the traversal needs a stack entry");
constexpr uint32_t kNoInst = 0xFFFFFFFFu;
constexpr int kTraceThreads = 128; // block of every traversal kernel

// Work of the instrumented traversal (COUNT): nodes visited and triangles tested per lane, and
// on the first active lane of each warp-wide step the step and its active lanes.
struct TraceCounters {
    uint32_t nodes, tris;
    uint32_t node_steps, node_lanes, tri_steps, tri_lanes;
};
GBPT_DI void count_step(uint32_t& steps, uint32_t& lanes) {
    const uint32_t m = __activemask();
    if ((threadIdx.x & 31u) == (uint32_t)(__ffs(m) - 1)) {
        steps++;
        lanes += __popc(m);
    }
}

GBPT_DI float safe_rcp(float d) {
    const float m = 1e-20f;
    return __frcp_rn(fabsf(d) > m ? d : copysignf(m, d));
}

// Instance records of two-level scenes, 7 float4 each: object-to-world rows (0..2), world-to-
// object rows (3..5), then (BLAS root node, mask, first geometry of the BLAS, 0) as bits. The
// transforms are evaluated with explicit round-to-nearest operations in a fixed order, as the
// oracle does, so transformed rays (and therefore hits) are bit-identical to the host's.
GBPT_DI float xform_row(float4 r, float3 p, float w) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.x, p.x), __fmul_rn(r.y, p.y)),
                               __fmul_rn(r.z, p.z)),
                     __fmul_rn(r.w, w));
}
GBPT_DI float3 xform_point(float4 r0, float4 r1, float4 r2, float3 p) {
    return f3(xform_row(r0, p, 1.0f), xform_row(r1, p, 1.0f), xform_row(r2, p, 1.0f));
}
GBPT_DI float3 xform_vector(float4 r0, float4 r1, float4 r2, float3 v) {
    return f3(xform_row(r0, v, 0.0f), xform_row(r1, v, 0.0f), xform_row(r2, v, 0.0f));
}

// ---- traversal state and loop ------------------------------------------------------------------
// One loop serves every query (trace_persistent): a node step, the triangles of the leaves it hit,
// then the next group off the stack; the warp leaves it to refill idle lanes once fewer than
// `refill_lanes` lanes are busy (a launch argument). Two-level scenes: a top-level leaf is an
// instance; entering it pushes what is left of the top level, transforms the ray to object space
// (t is unchanged: the direction is not renormalised) and continues from the BLAS root; when the
// stack drops back to the entry depth the world ray is restored. The closest hit and the tie rule
// (equal t: smallest geometry, primitive, instance) do not depend on the visit order.
// The loop is kept short: postponing triangle groups until several lanes of a warp had some to
// test, and sharing rays only every other step, each cost more instructions a step than they
// saved (1080p soup frame 251.9 ms with both, 244.7 without the first, 240.4 without either; a
// million closest hits 0.82 / 0.75 / 0.72 ms).


// What a node step does not touch, in shared memory: the closest hit (written when a candidate is
// accepted, two or three times a ray) and the triangle test's ray (read while the triangle's
// record is on its way). In registers these words made the traversal spill others, 96 to 136 bytes
// a thread at 8 and 9 blocks per SM, and what it spilled missed L1 two times in three; now it
// spills 8 to 48, in ticks of several two-level scenes up to 114 (640x360 soup frame 7.18 instead
// of 7.35 ms, 1080p 226.1 instead of 227.4, 37,003 listed pixels 1.50 instead of 1.55, a million
// closest hits 0.645 instead of 0.652).
// 13 words, an odd stride: the lanes' words fall into different banks.
struct LaneMem {
    RayShear ray;
    // u, v are V, W of the test until divided by det. kSignedZero: det has the sign of the hit's t
    // (all three may be negated, which leaves the quotients as they are)
    float u, v, det;
    uint32_t prim, geom, inst; // geom = kNoInst until a hit is found
    uint32_t pad;
};
// The world ray of two-level scenes, read when an instance is entered or left, there as well: it
// makes room for an eighth block per SM (trace_blocks).
struct WorldRay {
    float ox, oy, oz, dx, dy, dz;
    uint32_t pad;
};

// A scene's traversal data.
struct SceneRef {
    const uint4* nodes;
    const float4* tris;  // copy 0 of the records
    const float4* insts; // instance records; nullptr for single-level scenes
    uint32_t tri_stride; // float4 from one copy of the records to the next
};

struct TraceState {
    SceneRef ref;        // the ray's scene (RayScene)
    const float4* tris;  // its records (copy-major layout: the current ray's copy)
    float3 o, d, inv;    // the ray in the current space (object space inside an instance)
    float tmin;
    RayPre pre;
    uint2 ngroup, tgroup;
    LaneMem* lane;   // the rest of the closest hit and of the current ray
    float t; // the closest hit's distance, the span's end before the first
    WorldRay* world; // of two-level scenes
    uint32_t inst; // instance being traversed, kNoInst at the top level
    int inst_sp;   // stack depth at which it was entered
    // bits 24-31: the stack's first entry of this lane (those below were given to other lanes), as
    // the depth in the axis word; bits 8-12: the lane that keeps the ray's result
    uint32_t aux;
    GBPT_DI int floor() const { return (int)(aux >> 24); }
    GBPT_DI bool at_floor() const { return (pre.k ^ aux) < (1u << 24); }
    GBPT_DI uint32_t owner() const { return (aux >> 8) & 31u; }
    // the traversal stack's depth, kept in bits 24..31 of the ray's axis word
    GBPT_DI int sp() const { return (int)(pre.k >> 24); }
    GBPT_DI void push_sp() { pre.k += 1u << 24; }
    GBPT_DI void pop_sp() { pre.k -= 1u << 24; }
};

// Where a launch's rays find their scene: in each ray's state (requests of several scenes share
// ticks), or, when all rays are of one scene, in the kernel's arguments. The latter saves the
// two-level state five registers (instanced 1280x720 frame 4.09 instead of 4.25 ms; its G-buffer
// 0.86 instead of 0.90) and the ray queries' two (a million closest hits 0.81 instead of 0.86);
// the single-level wavefront is no faster with it (1080p soup frame 225.0 against 224.6 ms).
// A lane that works on another lane's ray without having loaded one (share_rays) finds OneScene's
// data there too: nothing of it is in the lane's state.
struct RayScene {
    static constexpr bool kPerRay = true;
    GBPT_DI const SceneRef& of(const TraceState& s) const { return s.ref; }
};
struct OneScene {
    static constexpr bool kPerRay = false;
    SceneRef ref;
    GBPT_DI const SceneRef& of(const TraceState&) const { return ref; }
};

template <class Scene>
GBPT_DI void set_ray(TraceState& s, const Scene& scene, float3 o, float3 d) {
    s.o = o;
    s.d = d;
    s.inv = f3(safe_rcp(d.x), safe_rcp(d.y), safe_rcp(d.z));
    const uint32_t oct = (__float_as_uint(d.x) >> 31) | ((__float_as_uint(d.y) >> 31) << 1) |
                         ((__float_as_uint(d.z) >> 31) << 2);
    // the stack, the mask and the hit outlive a change of space
    const uint32_t kept = s.pre.k & (0xFFFF0000u | kTriKey | kRayAny);
    s.pre = ray_pre(o, d, s.lane->ray);
    s.pre.k |= ((7u - oct) << 8) | kept;
    const SceneRef& ref = scene.of(s);
    s.tris = ref.tris + (size_t)s.pre.kz() * ref.tri_stride;
}

// A span's start with -0 for +0 and its end with +0 for -0, as intersect_node needs them. (Made +0
// in the box test instead, the end cost a register there: a million closest hits 640 against 626
// us.)
GBPT_DI float span_start(float tmin) { return tmin == 0.0f ? -0.0f : tmin; }
GBPT_DI float span_end(float tmax) { return __fadd_rn(tmax, 0.0f); }

// Whether a hit at -0 leaves a span that ends at +0, its sign kept in LaneMem::det: wherever a
// direction can be infinite, the caller's or one transformed into an instance. The bounce and
// shadow rays of single-level scenes are normalised; there the different registers of the
// acceptance cost 37,003 listed pixels 1.60 instead of 1.54 ms.
template <TraceMode MODE, bool TWO_LEVEL>
constexpr bool kSignedZero = MODE != kTraceMixed || TWO_LEVEL;

template <class Scene>
GBPT_DI void trace_init(TraceState& s, const Scene& scene, float3 o, float3 d, float tmin,
                        float tmax, uint32_t mask, uint32_t any = 0u) {
    s.pre.k = ((mask & 0xFFu) << 16) | any; // any: kRayAny or 0
    set_ray(s, scene, o, d);
    // a span with a NaN end holds no hit, but would make every box test one: an empty span
    const bool span = tmin == tmin && tmax == tmax;
    if (!span) tmin = 0.0f, tmax = -1.0f;
    s.ngroup = make_uint2(0u, 0x80000000u);
    s.tgroup = make_uint2(0u, 0u);
    s.tmin = span_start(tmin);
    s.t = span_end(tmax);
    s.lane->u = s.lane->v = 0.0f;
    s.lane->prim = s.lane->geom = s.lane->inst = kNoInst;
    s.inst = kNoInst;
    s.inst_sp = -1;
}

template <class Scene>
GBPT_DI void enter_instance(TraceState& s, const Scene& scene, uint32_t ii) {
    const float4* r = scene.of(s).insts + 7ull * ii;
    const float4 w0 = __ldg(r + 3), w1 = __ldg(r + 4), w2 = __ldg(r + 5);
    const WorldRay& w = *s.world;
    set_ray(s, scene, xform_point(w0, w1, w2, f3(w.ox, w.oy, w.oz)),
            xform_vector(w0, w1, w2, f3(w.dx, w.dy, w.dz)));
    s.inst = ii;
    s.inst_sp = s.sp();
    s.ngroup = make_uint2(__float_as_uint(__ldg(r + 6).x), 0x80000000u);
}

template <class Scene> GBPT_DI void exit_instance(TraceState& s, const Scene& scene) {
    const WorldRay& w = *s.world;
    set_ray(s, scene, f3(w.ox, w.oy, w.oz), f3(w.dx, w.dy, w.dz));
    s.inst = kNoInst;
    s.inst_sp = -1;
}

// Child box planes. Byte j of a plane word w is the quantised plane q of child j; the slab
// distance is t = q * a + o, a = 2^e / d and o = (p - origin) / d per node and axis.
// GBPT_BOX_BIAS (the default): one byte permute writes q into bits 8..15 of the float 32768.0,
// which makes the float 32768 + q exactly, and the per-node offsets absorb the bias
// (o' = o - 32768 a), so a plane costs a permute and an FMA. The rounding of o' is at most
// 2^-9 |a| (a 512th of a quantisation step); the slack below covers it. Without it: shift, mask
// and integer-to-float conversion, then the FMA.
#ifndef GBPT_BOX_BIAS
#define GBPT_BOX_BIAS 1
#endif
#if GBPT_BOX_BIAS
constexpr float kPlaneBias = 32768.0f;
GBPT_DI float qplane(uint32_t w, int j) {
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7504u | ((uint32_t)j << 4)));
}
#else
constexpr float kPlaneBias = 0.0f;
GBPT_DI float qplane(uint32_t w, int j) { return (float)((w >> (8 * j)) & 0xFFu); }
#endif

// GBPT_BOX_FMA2: the plane distances of two children with one paired FP32 FMA (fma.rn.f32x2).
#ifndef GBPT_BOX_FMA2
#define GBPT_BOX_FMA2 1
#endif
GBPT_DI uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
// the biased planes of children J and J + 1 of word w (as qplane), times a plus o, per lane
template <int J> GBPT_DI float2 plane_t2(uint32_t w, uint64_t a2, uint64_t o2) {
    float2 r;
    asm("{\n\t.reg .b32 q0, q1;\n\t.reg .b64 q, d;\n\t"
        "prmt.b32 q0, %2, 0x47000000, %3;\n\t"
        "prmt.b32 q1, %2, 0x47000000, %4;\n\t"
        "mov.b64 q, {q0, q1};\n\t"
        "fma.rn.f32x2 d, q, %5, %6;\n\t"
        "mov.b64 {%0, %1}, d;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "r"(w), "n"(0x7504 | (J << 4)), "n"(0x7504 | ((J + 1) << 4)), "l"(a2), "l"(o2));
    return r;
}

// The order of a node's inner children: bit s of m to bit s ^ o, o the ray's inverted octant, so
// that the highest bit is the child to visit first. One byte per (o, m), in shared memory.
struct OctantOrder {
    uint8_t bits[8 * 256];
};
GBPT_DI void octant_order_init(OctantOrder& t) {
    for (uint32_t i = threadIdx.x; i < 8u * 256u; i += blockDim.x) {
        uint32_t m = i & 255u;
        const uint32_t o = i >> 8;
        if (o & 1u) m = ((m >> 1) & 0x55u) | ((m << 1) & 0xAAu);
        if (o & 2u) m = ((m >> 2) & 0x33u) | ((m << 2) & 0xCCu);
        if (o & 4u) m = (m >> 4) | ((m << 4) & 0xF0u);
        t.bits[i] = (uint8_t)m;
    }
    __syncthreads();
}

// Bound by the ALU pipe (byte permutes, minima and maxima, at half the FMA pipe's rate), so what can
// go elsewhere does: hits are collected from the signs of differences (FMA pipe) instead of
// compares and shifted meta bytes, the visiting order comes from a table in shared memory, and only
// the leaves that are hit (one in six nodes has any) look at their meta bytes: 1080p soup frame
// 251.7 instead of 258.2 ms.
// Intersects the 8 children of node `ni`. ngroup receives the child base and the inner children
// hit in visiting order in bits 24..31, the node's imask in bits 0..7; tgroup the triangle base
// and the hit leaves' triangles in bits 0..23.
// The quantised planes are dequantised with a per-axis slack of 2^-20 of the plane distance
// magnitude (plus 2^-8 of a quantisation step for the biased planes), so rounding never loses a
// child the exact box would keep.
template <bool COUNT, bool PAIRED>
GBPT_DI void intersect_node(const TraceState& s, const uint4* nodes, uint32_t ni, const OctantOrder& order,
                            uint2& ngroup, uint2& tgroup, TraceCounters* ctr) {
    if (COUNT) ctr->nodes++;
    const uint4 n0 = __ldg(&nodes[5 * ni + 0]);
    const uint4 n1 = __ldg(&nodes[5 * ni + 1]);
    const uint4 n2 = __ldg(&nodes[5 * ni + 2]);
    const uint4 n3 = __ldg(&nodes[5 * ni + 3]);
    const uint4 n4 = __ldg(&nodes[5 * ni + 4]);
    const float kErr = 1.0f / 1048576.0f;
    const float kBiasErr = GBPT_BOX_BIAS ? 1.0f / 256.0f : 0.0f;
    // every operation rounded once in a fixed order (no contraction choices left to the
    // compiler), so a host walk of the same tree makes the same box decisions
    const float aix = __fmul_rn(__uint_as_float((n0.w & 0xFFu) << 23), s.inv.x);
    const float aiy = __fmul_rn(__uint_as_float(((n0.w >> 8) & 0xFFu) << 23), s.inv.y);
    const float aiz = __fmul_rn(__uint_as_float(((n0.w >> 16) & 0xFFu) << 23), s.inv.z);
    const float aox = __fmul_rn(__fsub_rn(__uint_as_float(n0.x), s.o.x), s.inv.x);
    const float aoy = __fmul_rn(__fsub_rn(__uint_as_float(n0.y), s.o.y), s.inv.y);
    const float aoz = __fmul_rn(__fsub_rn(__uint_as_float(n0.z), s.o.z), s.inv.z);
    const float ex = __fmaf_rn(kBiasErr, fabsf(aix),
                               __fmul_rn(__fmaf_rn(255.0f, fabsf(aix), fabsf(aox)), kErr));
    const float ey = __fmaf_rn(kBiasErr, fabsf(aiy),
                               __fmul_rn(__fmaf_rn(255.0f, fabsf(aiy), fabsf(aoy)), kErr));
    const float ez = __fmaf_rn(kBiasErr, fabsf(aiz),
                               __fmul_rn(__fmaf_rn(255.0f, fabsf(aiz), fabsf(aoz)), kErr));
    const float nox = __fmaf_rn(-kPlaneBias, aix, __fsub_rn(aox, ex));
    const float fox = __fmaf_rn(-kPlaneBias, aix, __fadd_rn(aox, ex));
    const float noy = __fmaf_rn(-kPlaneBias, aiy, __fsub_rn(aoy, ey));
    const float foy = __fmaf_rn(-kPlaneBias, aiy, __fadd_rn(aoy, ey));
    const float noz = __fmaf_rn(-kPlaneBias, aiz, __fsub_rn(aoz, ez));
    const float foz = __fmaf_rn(-kPlaneBias, aiz, __fadd_rn(aoz, ez));
    const uint32_t imask = n0.w >> 24;

    // the direction's signs from the octant (negative axis a: bit a of oct_inv clear)
    const uint32_t oct_inv = s.pre.oct_inv();
    const bool negx = (oct_inv & 1u) == 0u, negy = (oct_inv & 2u) == 0u;
    const bool negz = (oct_inv & 4u) == 0u;
    // the children missed, the first child in the highest bit: the sign of cmax - cmin is set
    // when cmin <= cmax is false. Neither is NaN (trace_init ends such rays), and inf - inf is the
    // canonical, positive NaN. It is also set for cmin = +0 and cmax = -0, though 0 <= -0
    // (-0 - +0 = -0), which must not meet: cmax is -0 only as the distance, after a hit at the
    // origin along a negative axis (span_end, kSignedZero), cmin is +0 only as a near plane
    // (span_start), and that where the box begins beyond 0, since the slack puts it before the
    // box - except along an infinite direction, whose planes are all 0.
    uint32_t miss = 0;
    auto add = [&](float cmin, float cmax) {
        miss = __funnelshift_l(__float_as_uint(__fsub_rn(cmax, cmin)), miss, 1);
    };
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t qlx = half ? n2.y : n2.x, qly = half ? n2.w : n2.z;
        const uint32_t qlz = half ? n3.y : n3.x, qhx = half ? n3.w : n3.z;
        const uint32_t qhy = half ? n4.y : n4.x, qhz = half ? n4.w : n4.z;
        const uint32_t nqx = negx ? qhx : qlx, fqx = negx ? qlx : qhx;
        const uint32_t nqy = negy ? qhy : qly, fqy = negy ? qly : qhy;
        const uint32_t nqz = negz ? qhz : qlz, fqz = negz ? qlz : qhz;
        if constexpr (PAIRED) {
            // children j and j + 1 of the half at once: the paired FP32 FMA rounds each lane like
            // __fmaf_rn, so the decisions are the scalar ones
            const uint64_t ax2 = pack2(aix, aix), ay2 = pack2(aiy, aiy), az2 = pack2(aiz, aiz);
            const uint64_t nox2 = pack2(nox, nox), noy2 = pack2(noy, noy), noz2 = pack2(noz, noz);
            const uint64_t fox2 = pack2(fox, fox), foy2 = pack2(foy, foy), foz2 = pack2(foz, foz);
            auto pair = [&](auto jc) {
                constexpr int j = decltype(jc)::value;
                const float2 tnx = plane_t2<j>(nqx, ax2, nox2), tny = plane_t2<j>(nqy, ay2, noy2);
                const float2 tnz = plane_t2<j>(nqz, az2, noz2), tfx = plane_t2<j>(fqx, ax2, fox2);
                const float2 tfy = plane_t2<j>(fqy, ay2, foy2), tfz = plane_t2<j>(fqz, az2, foz2);
                const float cmin0 = fmaxf(fmaxf(tnx.x, tny.x), fmaxf(tnz.x, s.tmin));
                const float cmax0 = fminf(fminf(tfx.x, tfy.x), fminf(tfz.x, s.t));
                const float cmin1 = fmaxf(fmaxf(tnx.y, tny.y), fmaxf(tnz.y, s.tmin));
                const float cmax1 = fminf(fminf(tfx.y, tfy.y), fminf(tfz.y, s.t));
                add(cmin0, cmax0);
                add(cmin1, cmax1);
            };
            pair(std::integral_constant<int, 0>{});
            pair(std::integral_constant<int, 2>{});
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float tnx = __fmaf_rn(qplane(nqx, j), aix, nox);
                const float tny = __fmaf_rn(qplane(nqy, j), aiy, noy);
                const float tnz = __fmaf_rn(qplane(nqz, j), aiz, noz);
                const float tfx = __fmaf_rn(qplane(fqx, j), aix, fox);
                const float tfy = __fmaf_rn(qplane(fqy, j), aiy, foy);
                const float tfz = __fmaf_rn(qplane(fqz, j), aiz, foz);
                const float cmin = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, s.tmin));
                const float cmax = fminf(fminf(tfx, tfy), fminf(tfz, s.t));
                add(cmin, cmax);
            }
        }
    }
    const uint32_t hits = (__brev(miss) >> 24) ^ 0xFFu; // by child
    const uint32_t inner = hits & imask;
    const uint32_t first = order.bits[(s.pre.k & 0x700u) | inner];
    ngroup = make_uint2(n1.x, (first << 24) | imask);
    // the leaves' triangles, from their meta bytes: unary count << 5 | first triangle
    uint32_t leaves = hits & ~imask, tri = 0u;
    while (leaves != 0u) {
        const uint32_t j = __ffs(leaves) - 1u;
        leaves &= leaves - 1u;
        const uint32_t meta = __byte_perm(n1.z, n1.w, j) & 0xFFu;
        tri |= (meta >> 5) << (meta & 31u);
    }
    tgroup = make_uint2(n1.y, tri);
}

// Runs the traversal of the ray in s until it is finished (returns true; result in s.t and *s.lane,
// geom = kNoInst on a miss; of a first-hit ray the first hit found) or until the warp should refill
// its idle lanes (returns false; s keeps the state). `st(i)` is stack entry i. A stack overflow raises *err
// and finishes the ray with what it found.
// `alpha(geom, prim, u, v)` decides the candidate hits of non-opaque triangles (true: skip).
template <TraceMode MODE, bool COUNT, bool TWO_LEVEL, class Scene, class StackRef, class Alpha>
GBPT_DI bool trace_loop(TraceState& s, const Scene& scene, StackRef&& st, const OctantOrder& order,
                        TraceCounters* ctr, uint32_t* err,
                        const Alpha& alpha, int min_lanes) {
    while (true) {
        // without instances the stack holds node groups only
        if (!TWO_LEVEL || s.ngroup.y > 0x00FFFFFFu) {
            const uint32_t hits = s.ngroup.y;
            const uint32_t bit = 31u - __clz(hits);
            s.ngroup.y = hits ^ (1u << bit);
            if (s.ngroup.y > 0x00FFFFFFu) {
                if (s.sp() >= kStackSize) {
                    atomicOr(err, 1u);
                    return true;
                }
                st(s.sp()) = s.ngroup;
                s.push_sp();
            }
            const uint32_t slot = (bit - 24u) ^ s.pre.oct_inv();
            const uint32_t ni = s.ngroup.x + __popc(hits & ((1u << slot) - 1u));
            if (COUNT) count_step(ctr->node_steps, ctr->node_lanes);
            // the paired planes hold more registers: first-hit traversal, which keeps fewer,
            // measured faster with the scalar ones
            intersect_node<COUNT, GBPT_BOX_FMA2 != 0 && MODE != kTraceAny>(
                s, scene.of(s).nodes, ni, order, s.ngroup, s.tgroup, ctr);
        } else {
            // the rest of a top-level instance group came off the stack
            s.tgroup = s.ngroup;
            s.ngroup = make_uint2(0u, 0u);
        }
        while (s.tgroup.y != 0u) {
            const uint32_t b = __ffs(s.tgroup.y) - 1u;
            s.tgroup.y &= s.tgroup.y - 1u;
            const uint32_t ti = s.tgroup.x + b;
            if (TWO_LEVEL && scene.of(s).insts != nullptr && s.inst == kNoInst) {
                // a top-level leaf: an instance (record: instance index, mask in the flag word)
                const uint32_t fl = __float_as_uint(__ldg(&s.tris[3 * ti + 2]).w);
                if ((fl & s.pre.mask()) == 0u) continue;
                if (s.sp() + 2 > kStackSize) {
                    atomicOr(err, 1u);
                    s.tgroup.y = 0u;
                    continue;
                }
                if (s.ngroup.y > 0x00FFFFFFu) {
                    st(s.sp()) = s.ngroup;
                    s.push_sp();
                }
                if (s.tgroup.y != 0u) {
                    st(s.sp()) = s.tgroup;
                    s.push_sp();
                }
                s.tgroup.y = 0u;
                enter_instance(s, scene, __float_as_uint(__ldg(&s.tris[3 * ti]).w));
                break;
            }
            const float4* rec = s.tris + 3 * ti;
            const float4 r0 = __ldg(rec + 0);
            const float4 r1 = __ldg(rec + 1);
            const float4 r2 = __ldg(rec + 2);
            const uint32_t tfl = __float_as_uint(r2.w);
            if (COUNT) {
                if ((tfl & s.pre.mask()) == 0u) continue;
                ctr->tris++;
                count_step(ctr->tri_steps, ctr->tri_lanes);
            }
            float t, u, v;
            float det;
            if (!intersect_tri(s.pre, s.lane->ray, r0, r1, r2, tfl, s.tmin, s.t, t, u, v, det))
                continue;
            // the instance mask is tested where few candidates get: before the intersection, it made
            // every triangle step wait for the flag word and branch once more (1080p soup frame
            // 235.1 instead of 227.7 ms, a million closest hits 0.72 instead of 0.65). What is
            // counted is still what passes the mask.
            if (!COUNT && (tfl & s.pre.mask()) == 0u) continue;
            const uint32_t prim = __float_as_uint(r0.w), geom = __float_as_uint(r1.w);
            if (t < s.t || geom < s.lane->geom ||
                (geom == s.lane->geom &&
                 (prim < s.lane->prim || (prim == s.lane->prim && s.inst < s.lane->inst)))) {
                if ((tfl & kTriAlpha) && alpha(geom, prim, __fdiv_rn(u, det), __fdiv_rn(v, det)))
                    continue;
                if (kSignedZero<MODE, TWO_LEVEL>) {
                    const uint32_t neg =
                        (__float_as_uint(t) ^ __float_as_uint(det)) & 0x80000000u;
                    det = __uint_as_float(__float_as_uint(det) ^ neg);
                    u = __uint_as_float(__float_as_uint(u) ^ neg);
                    v = __uint_as_float(__float_as_uint(v) ^ neg);
                    t = span_end(t);
                }
                s.lane->det = det;
                s.t = t;
                s.lane->u = u;
                s.lane->v = v;
                s.lane->prim = prim;
                s.lane->geom = geom;
                s.lane->inst = s.inst;
                if (MODE != kTraceAny) s.pre.k = (s.pre.k & ~kTriKey) | (tfl & kTriKey);
                // a first-hit ray ends with it
                if (MODE == kTraceAny || (MODE == kTraceMixed && (s.pre.k & kRayAny) != 0u))
                    return true;
            }
        }
        if (s.ngroup.y <= 0x00FFFFFFu) {
            if (TWO_LEVEL && s.inst != kNoInst && s.sp() == s.inst_sp) exit_instance(s, scene);
            if (s.at_floor()) return true;
            s.pop_sp();
            s.ngroup = st(s.sp());
        }
        if (__popc(__activemask()) < min_lanes) return false;
    }
}

// Position of the r-th set bit of m (r < popc(m)).
GBPT_DI uint32_t nth_bit(uint32_t m, uint32_t r) {
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t w = 16; w > 0; w >>= 1) {
        const uint32_t c = __popc((m >> pos) & ((1u << w) - 1u));
        if (r >= c) {
            r -= c;
            pos += w;
        }
    }
    return pos;
}

template <class T> GBPT_DI T* shfl_ptr(T* p, uint32_t src) {
    return (T*)__shfl_sync(0xFFFFFFFFu, (unsigned long long)p, src);
}

// Whether a hit comes before the lane's: nearer, or at the same distance the smaller (geometry,
// primitive, instance).
GBPT_DI bool hit_before(float t, uint32_t geom, uint32_t prim, uint32_t inst,
                        const TraceState& s) {
    const LaneMem& b = *s.lane;
    return t < s.t || (t == s.t && (geom < b.geom ||
                                    (geom == b.geom &&
                                     (prim < b.prim || (prim == b.prim && inst < b.inst)))));
}

// Once the pool is empty, the rays a warp has left are shared out: idle lanes take the oldest stack
// entries of busy ones and traverse them for the same ray (helpers). The lane that loaded the ray
// (its owner) keeps the result: helpers report hits to it and take over its distance, and it
// stores the result when no lane works on the ray any more. The closest hit and the tie rule do
// not depend on which lane finds it. Called by all 32 lanes; `active`: the lane traverses a part
// of a ray; `owns`: it keeps an unfinished ray.
// One long ray (a hundred dependent node steps of about a microsecond each) used to keep its warp,
// and with it the launch, while 31 lanes idled: without / with sharing, the instanced 1280x720
// frame of path length 16 takes 5.56 / 4.41 ms, 37,003 pixels x 8 of the 200k-triangle soup 2.17 /
// 1.79, a 64x64 frame of the room 0.30 / 0.25; where queues are long it is neutral (1080p soup
// frame 261.5 / 260.6).
template <TraceMode MODE, bool TWO_LEVEL, class Scene, class StackRef, class Store>
GBPT_DI void share_rays(TraceState& s, const Scene& scene, StackRef&& st, uint32_t& ray, bool& active, bool& owns,
                        const Store& store) {
    const uint32_t lane = threadIdx.x & 31u;
    // helpers' hits, one at a time, to their rays' owners
    const bool helper = s.owner() != lane;
    uint32_t m = __ballot_sync(0xFFFFFFFFu, helper && s.lane->geom != kNoInst);
    while (m != 0u) {
        const uint32_t h = __ffs(m) - 1u;
        m &= m - 1u;
        const uint32_t o = __shfl_sync(0xFFFFFFFFu, s.owner(), h);
        const float t = __shfl_sync(0xFFFFFFFFu, s.t, h);
        const float u = __shfl_sync(0xFFFFFFFFu, s.lane->u, h);
        const float v = __shfl_sync(0xFFFFFFFFu, s.lane->v, h);
        const float det = __shfl_sync(0xFFFFFFFFu, s.lane->det, h);
        const uint32_t prim = __shfl_sync(0xFFFFFFFFu, s.lane->prim, h);
        const uint32_t geom = __shfl_sync(0xFFFFFFFFu, s.lane->geom, h);
        const uint32_t inst = TWO_LEVEL ? __shfl_sync(0xFFFFFFFFu, s.lane->inst, h) : kNoInst;
        const uint32_t k = __shfl_sync(0xFFFFFFFFu, s.pre.k, h);
        if (lane == o && hit_before(t, geom, prim, inst, s)) {
            s.t = t;
            s.lane->u = u;
            s.lane->v = v;
            s.lane->det = det;
            s.lane->prim = prim;
            s.lane->geom = geom;
            s.lane->inst = inst;
            s.pre.k = (s.pre.k & ~kTriKey) | (k & kTriKey);
        }
        if (lane == h) s.lane->prim = s.lane->geom = s.lane->inst = kNoInst;
    }
    // the owner's distance; a first-hit ray ends with its first hit
    const float t_own = __shfl_sync(0xFFFFFFFFu, s.t, s.owner());
    const uint32_t g_own = __shfl_sync(0xFFFFFFFFu, s.lane->geom, s.owner());
    if (helper) s.t = fminf(s.t, t_own);
    const bool any =
        MODE == kTraceAny || (MODE == kTraceMixed && (s.pre.k & kRayAny) != 0u);
    if (any && g_own != kNoInst) active = false;
    // rays without a busy lane
    const uint32_t busy = __reduce_or_sync(0xFFFFFFFFu, active ? 1u << s.owner() : 0u);
    if (owns && ((busy >> lane) & 1u) == 0u) {
        store(ray, s);
        owns = false;
    }
    // idle lanes take stack entries
    const bool donor = active && s.sp() > s.floor();
    const bool idle = !active && !owns;
    const uint32_t m_donor = __ballot_sync(0xFFFFFFFFu, donor);
    const uint32_t m_idle = __ballot_sync(0xFFFFFFFFu, idle);
    const uint32_t pairs = min(__popc(m_donor), __popc(m_idle));
    if (pairs == 0u) return;
    const uint32_t below = (1u << lane) - 1u;
    uint2 e = make_uint2(0u, 0u);
    bool top = false; // the entry belongs to the top level while the donor is in an instance
    if (donor && __popc(m_donor & below) < pairs) {
        e = st(s.floor());
        top = TWO_LEVEL && s.inst != kNoInst && s.floor() < s.inst_sp;
        s.aux += 1u << 24;
    }
    const uint32_t r = __popc(m_idle & below);
    const bool take = idle && r < pairs;
    const uint32_t src = take ? nth_bit(m_donor, r) : lane;
    auto f = [&](float x) { return __shfl_sync(0xFFFFFFFFu, x, src); };
    auto w = [&](uint32_t x) { return __shfl_sync(0xFFFFFFFFu, x, src); };
    if (Scene::kPerRay) s.ref.nodes = shfl_ptr(s.ref.nodes, src);
    s.tris = shfl_ptr(s.tris, src);
    s.o = f3(f(s.o.x), f(s.o.y), f(s.o.z));
    s.inv = f3(f(s.inv.x), f(s.inv.y), f(s.inv.z));
    if (MODE != kTraceMixed) s.tmin = f(s.tmin); // bounce and shadow rays start at 0
    const RayShear q = s.lane->ray;
    const RayShear shear{f(q.Sx), f(q.Sy), f(q.Sz), f(q.ox), f(q.oy), f(q.oz)};
    s.t = f(s.t);
    ray = w(ray);
    const uint32_t k = w(s.pre.k), aux = w(s.aux);
    e.x = w(e.x);
    e.y = w(e.y);
    bool restart = false;
    if (TWO_LEVEL) {
        if (Scene::kPerRay) {
            s.ref.tris = shfl_ptr(s.ref.tris, src);
            s.ref.tri_stride = w(s.ref.tri_stride);
            s.ref.insts = shfl_ptr(s.ref.insts, src);
        }
        const WorldRay q = *s.world;
        const WorldRay wr{f(q.ox), f(q.oy), f(q.oz), f(q.dx), f(q.dy), f(q.dz), 0u};
        if (take) *s.world = wr;
        s.inst = w(s.inst);
        restart = w(top ? 1u : 0u) != 0u;
    }
    if (take) {
        active = true;
        s.lane->ray = shear;
        s.pre.k = k & ~(0xFF000000u | kTriKey); // an empty stack, no hit
        s.aux = aux & 0x1F00u;
        s.ngroup = e;
        s.tgroup = make_uint2(0u, 0u);
        s.lane->prim = s.lane->geom = s.lane->inst = kNoInst;
        s.inst_sp = TWO_LEVEL && s.inst != kNoInst ? 0 : -1;
        if (TWO_LEVEL && restart) exit_instance(s, scene);
    }
}

// Runs the traversal of every ray i < n with persistent warps that pull ray indices from *fetch
// (zero before the launch; one atomic per warp for all idle lanes). load(i, state) calls
// trace_init and, when `scene` is per ray, sets ray i's scene (s.ref) before; store(i, hit, key) receives its result
// and the material-sort key of the closest hit (0 on a miss);
// alpha(i, geom, prim, u, v) is ray i's alpha test (true: skip the candidate). Must be called by
// all 32 lanes of every warp. Fewer rays than lanes are spread over all warps, a few lanes of
// each; with SHARE the last rays are shared out within each warp (share_rays), and a first-hit ray
// may then report any of its hits. Without it the visits are those of a one-ray-at-a-time walk.
template <TraceMode MODE, bool COUNT, bool TWO_LEVEL, bool SHARE, class Scene, class Load,
          class Store, class Alpha>
__device__ __forceinline__ void trace_persistent(const Scene& scene, uint32_t n, uint32_t* fetch,
                                                 Load load,
                                                 Store store_hit, Alpha alpha, TraceCounters* ctr,
                                                 uint32_t* err, int refill_lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    __shared__ OctantOrder order;
    octant_order_init(order);
    uint2 stack[kStackSize];
    auto st_ref = [&](int i) -> uint2& { return stack[i]; };
    // the barycentrics are divided once, for the final hit
    auto store = [&](uint32_t i, TraceState& s) {
        Hit h{s.t, s.lane->u, s.lane->v, s.lane->prim, s.lane->geom, s.lane->inst};
        if (h.geom != kNoInst) {
            if (kSignedZero<MODE, TWO_LEVEL> && h.t == 0.0f) h.t = copysignf(0.0f, s.lane->det);
            h.u = __fdiv_rn(h.u, s.lane->det);
            h.v = __fdiv_rn(h.v, s.lane->det);
        }
        store_hit(i, h, (s.pre.k & kTriKey) >> kTriKeyShift);
    };
    __shared__ LaneMem lanes[kTraceThreads];
    // a lane that has not loaded a ray may help with another's, and what share_rays does not hand
    // over (tmin of bounce and shadow rays, the instance of a single-level scene) is then this
    // initial state: the values that every load sets, which keep them constants
    TraceState s{};
    s.tmin = span_start(0.0f);
    s.inst = kNoInst;
    s.inst_sp = -1;
    s.lane = &lanes[threadIdx.x];
    __shared__ WorldRay worlds[TWO_LEVEL ? kTraceThreads : 1];
    s.world = &worlds[TWO_LEVEL ? threadIdx.x : 0];
    auto load_ray = [&](uint32_t i) {
        load(i, s);
        if (TWO_LEVEL) *s.world = WorldRay{s.o.x, s.o.y, s.o.z, s.d.x, s.d.y, s.d.z, 0u};
    };
    s.lane->geom = kNoInst;
    s.aux = lane << 8;
    uint32_t ray = 0xFFFFFFFFu;
    bool active = false, owns = false, pool_empty = false;
    if (!COUNT) {
        const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
        const uint32_t lanes = n / warps + (n % warps != 0u ? 1u : 0u);
        if (lanes < 32u) { // every warp has its rays at once, and the pool is empty
            const uint32_t i = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * lanes + lane;
            if (lane < lanes && i < n) {
                ray = i;
                load_ray(ray);
                active = owns = true;
            }
            pool_empty = true;
        }
    }
    while (true) {
        __syncwarp();
        if (!SHARE || !pool_empty) {
            bool exhausted = false;
            const uint32_t want_mask = __ballot_sync(0xFFFFFFFFu, !active);
            if (want_mask && !pool_empty) {
                const uint32_t leader = __ffs(want_mask) - 1u;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(fetch, (uint32_t)__popc(want_mask));
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if (!active) {
                    const uint32_t i = base + __popc(want_mask & ((1u << lane) - 1u));
                    if (i < n) {
                        ray = i;
                        load_ray(ray);
                        active = owns = true;
                    } else {
                        exhausted = true;
                    }
                }
                pool_empty = __ballot_sync(0xFFFFFFFFu, exhausted) != 0u;
            }
        }
        if (SHARE && pool_empty) share_rays<MODE, TWO_LEVEL>(s, scene, st_ref, ray, active, owns, store);
        if (__ballot_sync(0xFFFFFFFFu, active) == 0u) {
            if (!SHARE || __ballot_sync(0xFFFFFFFFu, owns) == 0u) break;
            continue;
        }
        if (!active) continue;
        const auto ray_alpha = [&](uint32_t g, uint32_t p, float u, float v) {
            return alpha(ray, g, p, u, v);
        };
        // until few lanes are busy and the pool can refill the others; with the pool empty a step
        // between two shares, or to the end
        if (trace_loop<MODE, COUNT, TWO_LEVEL>(
                s, scene, st_ref, order, ctr, err, ray_alpha,
                pool_empty ? (SHARE ? 33 : 0) : refill_lanes)) {
            active = false;
            if (!SHARE || !pool_empty) {
                store(ray, s);
                owns = false;
                s.lane->geom = kNoInst;
            }
        }
    }
}

// ---- camera (camera.slang:29-56), bit-identical to the oracle's FP32 build ---------------------------
struct CamGPU {
    float3 pos, U, V, W;
    float near_plane, far_plane, jx, jy;
};
GBPT_DI void camera_ray(const CamGPU& c, uint32_t px, uint32_t py, uint32_t w, uint32_t h,
                        float3& o, float3& d, float& tmin, float& tmax) {
    const float x = __fdiv_rn(__fadd_rn(__fadd_rn((float)px, 0.5f), c.jx), (float)w);
    const float y = __fdiv_rn(__fadd_rn(__fadd_rn((float)py, 0.5f), c.jy), (float)h);
    const float nx = __fadd_rn(__fmul_rn(2.0f, x), -1.0f);
    const float ny = __fadd_rn(__fmul_rn(-2.0f, y), 1.0f);
    const float dx = __fadd_rn(__fadd_rn(__fmul_rn(nx, c.U.x), __fmul_rn(ny, c.V.x)), c.W.x);
    const float dy = __fadd_rn(__fadd_rn(__fmul_rn(nx, c.U.y), __fmul_rn(ny, c.V.y)), c.W.y);
    const float dz = __fadd_rn(__fadd_rn(__fmul_rn(nx, c.U.z), __fmul_rn(ny, c.V.z)), c.W.z);
    const float l = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
    d = f3(__fdiv_rn(dx, l), __fdiv_rn(dy, l), __fdiv_rn(dz, l));
    const float lw = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(c.W.x, c.W.x), __fmul_rn(c.W.y, c.W.y)),
                                          __fmul_rn(c.W.z, c.W.z)));
    const float wx = __fdiv_rn(c.W.x, lw), wy = __fdiv_rn(c.W.y, lw), wz = __fdiv_rn(c.W.z, lw);
    const float cosv = __fadd_rn(__fadd_rn(__fmul_rn(wx, d.x), __fmul_rn(wy, d.y)), __fmul_rn(wz, d.z));
    const float inv_cos = __fdiv_rn(1.0f, cosv);
    o = c.pos;
    tmin = __fmul_rn(c.near_plane, inv_cos);
    tmax = __fmul_rn(c.far_plane, inv_cos);
}

// ---- environment (environment-map.slang:23-35, utils/math.slang:243-250) -------------------------------
GBPT_DI float3 env_to_local(const DevScene& s, float3 d) {
    const float* M = s.env_m;
    return f3(M[0] * d.x + M[1] * d.y + M[2] * d.z, M[3] * d.x + M[4] * d.y + M[5] * d.z,
              M[6] * d.x + M[7] * d.y + M[8] * d.z);
}
GBPT_DI int wrapi(int i, int n) {
    const int r = i % n;
    return r < 0 ? r + n : r;
}
// The lat-long map coordinates (u, v) of a world direction (its local frame by env_to_local).
GBPT_DI void env_uv(const DevScene& s, float3 dir, float& u, float& v) {
    const float3 p = normalize(env_to_local(s, dir));
    u = atan2f(p.x, -p.z) * kInv2Pi + 0.5f;
    v = acosf(fminf(fmaxf(p.y, -1.0f), 1.0f)) * kInvPi;
}
// The environment's radiance at map coordinates (u, v): bilinear, repeating.
GBPT_DI float3 env_eval_uv(const DevScene& s, float u, float v) {
    if (!(u == u) || !(v == v)) return f3(0.f, 0.f, 0.f);
    const float x = u * (float)s.ew - 0.5f, y = v * (float)s.eh - 0.5f;
    const float fx = floorf(x), fy = floorf(y);
    const float a = x - fx, b = y - fy;
    const int ix = (int)fx, iy = (int)fy;
    const int x0 = wrapi(ix, (int)s.ew), x1 = wrapi(ix + 1, (int)s.ew);
    const int y0 = wrapi(iy, (int)s.eh), y1 = wrapi(iy + 1, (int)s.eh);
    const float4 t00 = __ldg(&s.env[(size_t)y0 * s.ew + x0]);
    const float4 t10 = __ldg(&s.env[(size_t)y0 * s.ew + x1]);
    const float4 t01 = __ldg(&s.env[(size_t)y1 * s.ew + x0]);
    const float4 t11 = __ldg(&s.env[(size_t)y1 * s.ew + x1]);
    const float3 top = f3(t00.x, t00.y, t00.z) * (1.0f - a) + f3(t10.x, t10.y, t10.z) * a;
    const float3 bot = f3(t01.x, t01.y, t01.z) * (1.0f - a) + f3(t11.x, t11.y, t11.z) * a;
    return (top * (1.0f - b) + bot * b) * s.env_intensity;
}
GBPT_DI float3 env_eval(const DevScene& s, float3 dir) {
    if (s.ew == 0u) return f3(0.f, 0.f, 0.f);
    float u, v;
    env_uv(s, dir, u, v);
    return env_eval_uv(s, u, v);
}

} // namespace gbpt
