// Host build of the device traversal (csrc/rtg_trace.cuh) over a flattened scene, for
// test_trace_host.py: the CUDA intrinsics it uses are given here by their documented results.
#include <vector_types.h>

#include <cmath>
#include <cstdint>
#include <string>

static inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { uint4 v; v.x = x; v.y = y; v.z = z; v.w = w; return v; }
static inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
    const uint64_t v = ((uint64_t)b << 32) | a;
    uint32_t r = 0;
    for (int k = 0; k < 4; ++k) r |= (uint32_t)((v >> (8 * ((s >> (4 * k)) & 7u))) & 0xffu) << (8 * k);
    return r;
}
static inline float __frcp_rn(float x) { return 1.0f / x; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }

#include "../repackshot_b200/csrc/rtg_scene.h"
#include "../repackshot_b200/csrc/rtg_trace.cuh"

using namespace rtg;

struct Loaded {
    HScene scene;
    Flat flat;
    SceneDev S;
};

extern "C" void* host_load(const uint8_t* bytes, uint64_t len) {
    auto* l = new Loaded;
    std::string error;
    if (!parse_rsb(bytes, len, l->scene, error) || !flatten_scene(l->scene, l->flat, error)) return nullptr;
    l->S = l->flat.scene;
    l->S.nodes = l->flat.nodes.data();
    l->S.tris = l->flat.tris.data();
    l->S.blas = l->flat.blas.data();
    l->S.leaf_boxes = l->flat.leaf_boxes.data();
    return l;
}
extern "C" void host_free(void* l) { delete static_cast<Loaded*>(l); }

// (instance, triangle, t bits) of every ray, or whether it hits; `positive`: the form for t_min > 0.
// Returns the stack overflows.
extern "C" uint32_t host_trace(void* l, const float* rays, uint64_t n, int any, int camera, int positive, uint32_t* out) {
    const SceneDev& S = static_cast<Loaded*>(l)->S;
    uint32_t overflows = 0;
    for (uint64_t i = 0; i < n; ++i) {
        const float* r = rays + 8 * i;
        const V3 o = v3(r[0], r[1], r[2]), d = v3(r[3], r[4], r[5]);
        uint64_t shared[SHORT_STACK], deep[STACK_CAP - SHORT_STACK];
        SplitStack stack{shared, deep, 1};
        uint32_t err = 0;
        TraceResult res;
        bool hit;
        if (any) hit = positive ? traverse<true, true>(S, o, d, r[6], r[7], camera != 0, res, &err, stack) : traverse<true>(S, o, d, r[6], r[7], camera != 0, res, &err, stack);
        else hit = positive ? traverse<false, true>(S, o, d, r[6], r[7], camera != 0, res, &err, stack) : traverse<false>(S, o, d, r[6], r[7], camera != 0, res, &err, stack);
        overflows += err & 1u;
        if (any) {
            out[i] = hit;
        } else {
            out[3 * i] = hit ? res.inst : 0xffffffffu;
            out[3 * i + 1] = hit ? S.tris[res.tri].tri : 0xffffffffu;
            out[3 * i + 2] = hit ? fbits(res.t) : 0u;
        }
    }
    return overflows;
}
