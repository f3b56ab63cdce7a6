// The device traversal (trace_persistent of device_scene.cuh) compiled for the host: the 32 lanes
// of a warp run as coroutines that meet at every warp-wide operation, blocks of one warp run one
// after the other. Reads through __ldg are checked against the scene's arrays (counted and
// answered with zeros when outside), and -ftrivial-auto-var-init=pattern fills what the code
// leaves unset, so a use of unset lane state shows as a wrong hit or a counted read. NaNs and the
// order of signed zeros are the GPU's.
#include <ucontext.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <functional>
#include <vector>

#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace host {
constexpr int kLanes = 32;
struct Lane {
    ucontext_t ctx;
    std::vector<char> stack;
    uint64_t slot[2];
    int turn = 0;
    bool done = false;
};
Lane lanes[kLanes];
ucontext_t scheduler;
int current = 0;
uint3 thread, block;
dim3 grid_dim, block_dim;
const std::function<void()>* body;

// every lane's value of one warp-wide operation
const uint64_t* exchange(uint64_t v, uint64_t* all) {
    Lane& l = lanes[current];
    const int t = l.turn;
    l.turn ^= 1;
    l.slot[t] = v;
    swapcontext(&l.ctx, &scheduler);
    for (int i = 0; i < kLanes; ++i) all[i] = lanes[i].slot[t];
    return all;
}
void entry() {
    (*body)();
    lanes[current].done = true;
    swapcontext(&lanes[current].ctx, &scheduler);
}
void run_warp(const std::function<void()>& f) {
    body = &f;
    for (Lane& l : lanes) {
        l.stack.resize(256 << 10);
        l.turn = 0;
        l.done = false;
        getcontext(&l.ctx);
        l.ctx.uc_stack.ss_sp = l.stack.data();
        l.ctx.uc_stack.ss_size = l.stack.size();
        l.ctx.uc_link = nullptr;
        makecontext(&l.ctx, entry, 0);
    }
    for (bool any = true; any;) {
        any = false;
        for (int i = 0; i < kLanes; ++i) {
            if (lanes[i].done) continue;
            any = true;
            current = i;
            thread.x = (unsigned)i;
            swapcontext(&scheduler, &lanes[i].ctx);
        }
    }
}

struct Range {
    const char* p;
    size_t n;
};
std::vector<Range> readable;
uint64_t bad_reads = 0;
} // namespace host

#define threadIdx host::thread
#define blockIdx host::block
#define gridDim host::grid_dim
#define blockDim host::block_dim
#undef __shared__
#define __shared__ static
#undef __launch_bounds__
#define __launch_bounds__(...)

template <class T> T __ldg(const T* p) {
    T v;
    std::memset(&v, 0, sizeof(v));
    for (const host::Range& r : host::readable)
        if ((const char*)p >= r.p && (const char*)p + sizeof(T) <= r.p + r.n) {
            std::memcpy(&v, p, sizeof(v));
            return v;
        }
    ++host::bad_reads;
    return v;
}
template <class To, class From> To bits(From f) {
    To t;
    static_assert(sizeof(To) == sizeof(From), "bits");
    std::memcpy(&t, &f, sizeof(t));
    return t;
}
inline uint32_t __float_as_uint(float f) { return bits<uint32_t>(f); }
inline int __float_as_int(float f) { return bits<int>(f); }
inline float __int_as_float(int i) { return bits<float>(i); }
inline float __uint_as_float(uint32_t u) { return bits<float>(u); }
inline float canonical(float f) { return f == f ? f : bits<float>(0x7FFFFFFFu); }
inline float __fadd_rn(float a, float b) { return canonical(a + b); }
inline float __fsub_rn(float a, float b) { return canonical(a - b); }
inline float __fmul_rn(float a, float b) { return canonical(a * b); }
inline float __fdiv_rn(float a, float b) { return canonical(a / b); }
inline float __frcp_rn(float a) { return canonical(1.0f / a); }
inline float __fsqrt_rn(float a) { return canonical(std::sqrt(a)); }
inline float __fmaf_rn(float a, float b, float c) { return canonical(std::fma(a, b, c)); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline float __double2float_rn(double a) { return (float)a; }
inline int __float2int_rn(float a) { return (int)std::nearbyint(a); }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }
inline uint32_t __brev(uint32_t x) {
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= ((x >> i) & 1u) << (31 - i);
    return r;
}
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t n) {
    n &= 31u;
    return n ? (hi << n) | (lo >> (32u - n)) : hi;
}
inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
    const uint64_t w = ((uint64_t)b << 32) | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i)
        r |= (uint32_t)((w >> (8 * ((s >> (4 * i)) & 7u))) & 0xFFu) << (8 * i);
    return r;
}
template <class T> T __shfl_sync(uint32_t, T v, uint32_t src) {
    uint64_t all[host::kLanes], u = 0;
    std::memcpy(&u, &v, sizeof(v));
    host::exchange(u, all);
    std::memcpy(&v, &all[src & 31u], sizeof(v));
    return v;
}
inline uint32_t __ballot_sync(uint32_t, bool p) {
    uint64_t all[host::kLanes];
    host::exchange(p ? 1u : 0u, all);
    uint32_t r = 0;
    for (int i = 0; i < host::kLanes; ++i) r |= (uint32_t)all[i] << i;
    return r;
}
inline uint32_t __reduce_or_sync(uint32_t, uint32_t v) {
    uint64_t all[host::kLanes];
    host::exchange(v, all);
    uint32_t r = 0;
    for (int i = 0; i < host::kLanes; ++i) r |= (uint32_t)all[i];
    return r;
}
inline void __syncwarp() { __ballot_sync(0xFFFFFFFFu, true); }
inline void __syncthreads() { __ballot_sync(0xFFFFFFFFu, true); }
inline uint32_t __activemask() { return 0xFFFFFFFFu; } // lanes never leave a step together
inline uint32_t atomicAdd(uint32_t* p, uint32_t v) {
    const uint32_t old = *p;
    *p += v;
    return old;
}
inline uint32_t atomicOr(uint32_t* p, uint32_t v) {
    const uint32_t old = *p;
    *p |= v;
    return old;
}
using std::min;
// the GPU's: a NaN gives way to a number, -0 is less than +0
namespace gbpt {
inline float fmaxf(float a, float b) {
    if (a != a) return b;
    if (b != b) return a;
    return a > b || (a == b && !std::signbit(a)) ? a : b;
}
inline float fminf(float a, float b) {
    if (a != a) return b;
    if (b != b) return a;
    return a < b || (a == b && std::signbit(a)) ? a : b;
}
} // namespace gbpt

#define GBPT_BOX_FMA2 0 // the pairs round each plane as the single ones do
#include "device_scene.cuh"

using namespace gbpt;

namespace {
template <TraceMode MODE, bool TWO_LEVEL, class Scene>
void trace_all(const Scene& scene, const SceneRef& ref, const gbpt_ray* rays, const uint8_t* any,
               uint32_t n, uint32_t mask, uint32_t grid, gbpt_hit* hits, uint32_t* err) {
    uint32_t fetch = 0;
    auto load = [&](uint32_t i, TraceState& s) {
        const gbpt_ray& r = rays[i];
        if (Scene::kPerRay) s.ref = ref;
        trace_init(s, scene, f3(r.origin[0], r.origin[1], r.origin[2]),
                   f3(r.direction[0], r.direction[1], r.direction[2]),
                   MODE == kTraceMixed ? 0.0f : r.tmin, r.tmax, mask, any[i] ? kRayAny : 0u);
    };
    // the fields of gbpt_hit as the scene-global hit holds them
    auto store = [&](uint32_t i, const Hit& h, uint32_t key) {
        hits[i].instance_id = h.inst;
        hits[i].primitive_id = h.prim;
        hits[i].geometry_index = h.geom;
        hits[i].barycentrics[0] = h.u;
        hits[i].barycentrics[1] = h.v;
        hits[i].t = h.t;
        hits[i].reserved = key;
    };
    auto alpha = [](uint32_t, uint32_t, uint32_t, float, float) { return false; };
    host::grid_dim = dim3(grid);
    host::block_dim = dim3(host::kLanes);
    for (uint32_t b = 0; b < grid; ++b) {
        host::block.x = b;
        host::run_warp([&] {
            trace_persistent<MODE, false, TWO_LEVEL, true>(scene, n, &fetch, load, store, alpha,
                                                           nullptr, err, 20);
        });
    }
}
} // namespace

// The rays through `grid` warps, sharing their last rays: as ray queries (mixed = 0: closest hits,
// the scene in the kernel's arguments) or as a tick's launch (mixed = 1: any[i] asks for a first
// hit, spans start at 0; per_ray: the scene in each ray's state). `tris` is one copy of the
// records. Returns the number of reads outside the arrays, or -1 for a raised error word.
extern "C" __attribute__((visibility("default"))) int64_t
traversal_host(const void* nodes, uint64_t n_nodes, const float* tris, uint64_t n_tris,
               const float* insts, uint64_t n_inst, int mixed, int per_ray, const gbpt_ray* rays,
               const uint8_t* any, uint32_t n, uint32_t mask, uint32_t grid, gbpt_hit* hits) {
    std::vector<float4> rec(3 * 3 * n_tris); // the copies, as a scene's upload makes them
    for (uint64_t i = 0; i < n_tris; ++i)
        for (int c = 0; c < 3; ++c)
            for (int v = 0; v < 3; ++v) {
                const float* p = tris + 12 * i + 4 * v;
                rec[3 * (c * n_tris + i) + v] =
                    make_float4(p[(c + 1) % 3], p[(c + 2) % 3], p[c], p[3]);
            }
    host::readable = {{(const char*)nodes, n_nodes * 80},
                      {(const char*)rec.data(), rec.size() * sizeof(float4)},
                      {(const char*)insts, n_inst * 112}};
    host::bad_reads = 0;
    const SceneRef ref{(const uint4*)nodes, rec.data(), n_inst ? (const float4*)insts : nullptr,
                       (uint32_t)(3 * n_tris)};
    uint32_t err = 0;
    auto go = [&](auto mode, auto two_level, const auto& scene) {
        trace_all<decltype(mode)::value, decltype(two_level)::value>(scene, ref, rays, any, n, mask,
                                                                     grid, hits, &err);
    };
    using Closest = std::integral_constant<TraceMode, kTraceClosest>;
    using Mixed = std::integral_constant<TraceMode, kTraceMixed>;
    const OneScene one{ref};
    if (!mixed && n_inst) go(Closest{}, std::true_type{}, one);
    else if (!mixed) go(Closest{}, std::false_type{}, one);
    else if (per_ray && n_inst) go(Mixed{}, std::true_type{}, RayScene{});
    else if (per_ray) go(Mixed{}, std::false_type{}, RayScene{});
    else go(Mixed{}, std::true_type{}, one);
    return err ? -1 : (int64_t)host::bad_reads;
}
