// trace_exact.cuh -- the FP32 cone march of voxelConeTracing.frag over a
// linear atlas in the reference's layout, generic in the atlas's texel type:
// ExactAtlas (RGBA8, the drop-in) and F4Atlas (float RGBA, the
// differentiable form).  Software trilinear filter with FP32 weights and
// REPEAT addressing; the units that include it build with -fmad=false, so
// every form runs the same arithmetic in the same order.
#pragma once

#include <cmath>

#include "trace_common.cuh"

namespace vct {

// ---------------------------------------------------------------------------
// Two floats in a 64-bit register: one packed instruction rounds each half as
// the scalar one does, in half the issue slots.
typedef unsigned long long F2;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2(float v) { return f2(v, v); }
__device__ __forceinline__ float2 f2_split(F2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// A product that an add may follow is two scalar multiplies: the assembler is
// free to contract packed ones (measured: it does, .rn and all).
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    const float2 x = f2_split(a), y = f2_split(b);
    return f2(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y));
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, f2(-1.0f), a); }  // a - b, rounded once

struct Texel2 {
    F2 rg, ba;
};
__device__ __forceinline__ float4 texel_f4(Texel2 t) {
    const float2 a = f2_split(t.rg), b = f2_split(t.ba);
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ Texel2 texel_scale(Texel2 t, F2 w) { return {f2_mul(t.rg, w), f2_mul(t.ba, w)}; }
__device__ __forceinline__ Texel2 texel_add(Texel2 p, Texel2 q) { return {f2_add(p.rg, q.rg), f2_add(p.ba, q.ba)}; }
// p + (q - p) t
__device__ __forceinline__ Texel2 texel_lerp(Texel2 p, Texel2 q, F2 t) {
    return {f2_add(p.rg, f2_mul(f2_sub(q.rg, p.rg), t)), f2_add(p.ba, f2_mul(f2_sub(q.ba, p.ba), t))};
}

// Two bytes b -> b / 255, correctly rounded.  The byte three times over as the
// bits of a float is 65793 b 2^-149 (denormals and the first binade are one
// linear range), and b / 255 = 65793 b 2^-24 (1 + 2^-24 + 2^-48 + ...): one
// fused multiply-add forms the first two terms and rounds once, which leaves
// 2^-48 relative below the quotient (the test suite checks all 256 bytes).
__device__ __forceinline__ F2 unorm8_pair(uint32_t v, int c) {
    const uint32_t lo = __byte_perm(v, 0u, c == 0 ? 0x4000 : 0x4222), hi = __byte_perm(v, 0u, c == 0 ? 0x4111 : 0x4333);
    const F2 x = f2(__uint_as_float(lo), __uint_as_float(hi));
    return f2_fma(x, f2(0x1p125f), f2_mul(x, f2(0x1p101f)));
}

// The atlas forms.  A row is the texels of one (y, z); texel(row, x) loads one
// texel raw, zero() tells that eight raw texels all decode to zero.
struct ExactAtlas {
    const uint32_t* __restrict__ p;
    AtlasDims A;
    typedef const uint32_t* Row;
    typedef uint32_t Raw;
    static constexpr bool kZeroTest = true;
    __device__ __forceinline__ Row row(int y, int z) const { return p + ((int64_t)z * A.H + y) * A.W; }
    __device__ __forceinline__ Raw texel(Row r, int x) const { return __ldg(r + x); }
    static __device__ __forceinline__ bool zero(const Raw t[8]) {
        return ((t[0] | t[1] | t[2]) | (t[3] | t[4] | t[5]) | (t[6] | t[7])) == 0u;
    }
    static __device__ __forceinline__ Texel2 decode(Raw v) { return {unorm8_pair(v, 0), unorm8_pair(v, 2)}; }
};

// The RGBA8 atlas's texels read through a radiance texture holding the same
// texels (point filter at texel centres, unnormalised coordinates): one
// texture instruction returns the four channels decoded to float by the
// texture unit, in place of the 64-bit address arithmetic, the 4-byte load
// and the four-channel decode.  The unit's unorm8 conversion gives c/255
// correctly rounded, the float unorm8_pair computes (the tests compare whole
// traces through both reads bit for bit), so the trace's arithmetic, in its
// order, is unchanged.
struct TexelAtlas {
    cudaTextureObject_t t;
    AtlasDims A;
    typedef float2 Row;
    typedef float4 Raw;
    static constexpr bool kZeroTest = false;
    __device__ __forceinline__ Row row(int y, int z) const { return make_float2((float)y + 0.5f, (float)z + 0.5f); }
    __device__ __forceinline__ Raw texel(Row r, int x) const { return tex3D<float4>(t, (float)x + 0.5f, r.x, r.y); }
    static __device__ __forceinline__ bool zero(const Raw*) { return false; }
    static __device__ __forceinline__ Texel2 decode(Raw v) { return {f2(v.x, v.y), f2(v.z, v.w)}; }
};

// Float RGBA texels (16 B each), the layout of the FP16 form widened to FP32.
struct F4Atlas {
    const float4* __restrict__ p;
    AtlasDims A;
    typedef const float4* Row;
    typedef float4 Raw;
    static constexpr bool kZeroTest = false;
    __device__ __forceinline__ Row row(int y, int z) const { return p + ((int64_t)z * A.H + y) * A.W; }
    __device__ __forceinline__ Raw texel(Row r, int x) const { return __ldg(r + x); }
    static __device__ __forceinline__ bool zero(const Raw*) { return false; }
    static __device__ __forceinline__ Texel2 decode(Raw v) { return {f2(v.x, v.y), f2(v.z, v.w)}; }
};

__device__ __forceinline__ int wrap_rep(int i, int n) {
    int m = i % n;
    return m < 0 ? m + n : m;
}

// REPEAT of a texel index that a sampler coordinate in [0, 1) produces
// (i in [-1, n]): one compare and select on that range; the general
// modulo for anything else, so no index leaves [0, n).
__device__ __forceinline__ int wrap_tap(int i, int n) {
    const int m = i < 0 ? i + n : (i >= n ? i - n : i);
    return (unsigned)m < (unsigned)n ? m : wrap_rep(i, n);
}

// Launch constants of the march that replace divisions by exact equals.
struct MarchScale {
    float dim2_hi, dim2_lo;     // 1 / (volume_dimension + 2) in two floats, where `recip`
    float min_radius, inv_r2;   // of the min level's sphere; inv_r2 = 0: the shader's expression everywhere
    float inv_uvs, inv_extent;  // 1 / voxel_size, 1 / level 0's extent
    bool recip, pow2, pow2_uvs; // powers of two: volume_dimension; it and voxel_size; voxel_size
};

inline MarchScale march_scale(const vct_cone_tracing_desc& d) {
    MarchScale C;
    const float dim = d.volume_dimension;
    int e = 0;
    C.recip = std::frexp(dim, &e) == 0.5f && dim >= 1.0f && dim <= 2048.0f;
    const float y = dim + 2.0f;
    C.dim2_hi = (float)(1.0 / (double)y);
    C.dim2_lo = (float)(1.0 / (double)y - (double)C.dim2_hi);
    C.pow2_uvs = std::frexp(d.voxel_size, &e) == 0.5f && e > -100 && e < 100;
    C.pow2 = C.recip && C.pow2_uvs;
    C.inv_uvs = 1.0f / d.voxel_size;
    C.inv_extent = 1.0f / (d.voxel_size * dim);
    C.min_radius = d.voxel_size * dim * 0.5f;
    C.inv_r2 = (float)(1.0 / ((double)C.min_radius * (double)C.min_radius));
    if (!std::isnormal(C.inv_r2)) C.inv_r2 = 0.0f;
    return C;
}

// x / y for a divisor y known beforehand, hi + lo = 1 / y in two floats
// (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", 2004): the
// correctly rounded quotient for every x away from the exponent's ends where
// y is 6 or 2 + 2^k, k = 0 .. 11 (the test suite checks every significand).
__device__ __forceinline__ float div_known(float x, float hi, float lo) {
    return __fmaf_rn(x, hi, __fmul_rn(x, lo));
}
constexpr float kSixth = (float)(1.0 / 6.0), kSixthLo = (float)(1.0 / 6.0 - (double)kSixth);

// ceil(log2(|center - pos| / min_radius)) from the squared distance: with
// t = (dist / radius)^2 up to a few ulp, ceil(log2(t) / 2) is an exponent
// unless t is next to an even power of two, where the shader's expression
// decides (its logarithm is within an ulp, which moves no other ceil).
__device__ __forceinline__ float cone_min_level(float inv_r2, float min_radius, float3 center, float3 pos) {
    const float d2 = dot3(center - pos, center - pos);
    const uint32_t bits = __float_as_uint(d2 * inv_r2);
    const int rel = (int)(bits - 0x3f800000u);  // even powers of two are multiples of 2^24
    if (((uint32_t)(rel + 128) & 0xffffffu) < 256u || bits - 0x0d800000u >= 0x64800000u)
        return ceilf(log2f(sqrtf(d2) / min_radius));
    return (float)((rel >> 24) + 1);
}

// log2(diameter / uvs), before the clamps.
__device__ __forceinline__ float cone_raw_level(const MarchScale& C, float diameter, float uvs) {
    return log2f(C.pow2_uvs ? diameter * C.inv_uvs : diameter / uvs);
}

// The sampler coordinates (in one face) of position p at a level.
__device__ __forceinline__ float3 clipmap_coords(const MarchScale& C, const vct_cone_tracing_desc& d, float3 p,
                                                 int level) {
    const float dim = d.volume_dimension;
    float q[3] = {p.x, p.y, p.z};
    if (C.pow2) {
        const float inv = C.inv_extent * __uint_as_float((uint32_t)(127 - level) << 23);  // 2^-level
#pragma unroll
        for (int a = 0; a < 3; ++a) q[a] = q[a] * inv;
    } else {
        const float extent = d.voxel_size * exp2f((float)level) * dim;
#pragma unroll
        for (int a = 0; a < 3; ++a) q[a] = q[a] / extent;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) q[a] = fractf(q[a]) * dim + 1.0f;
    if (C.recip) {
#pragma unroll
        for (int a = 0; a < 3; ++a) q[a] = div_known(q[a], C.dim2_hi, C.dim2_lo);
    } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) q[a] = q[a] / (dim + 2.0f);
    }
    static_assert(kClipLevels == 6 && kFaces == 6, "the known divisor");
    return f3(div_known(q[0], kSixth, kSixthLo), div_known(q[1] + (float)level, kSixth, kSixthLo), q[2]);
}

// sampleClipmap (voxelConeTracing.frag:313-327): three linear-filtered
// sampler3D fetches (Vulkan linear filter, REPEAT, one mip) that differ in the
// x coordinate alone, weighted.
template <class Atlas>
__device__ __forceinline__ Texel2 sample_clipmap(const Atlas& T, const MarchScale& C, const vct_cone_tracing_desc& d,
                                                 float3 p, int level, float3 fo, float3 wt) {
    const AtlasDims& A = T.A;
    const float3 s = clipmap_coords(C, d, p, level);
    const float v = s.y * (float)A.H - 0.5f, w = s.z * (float)A.D - 0.5f;
    const float fv = floorf(v), fw = floorf(w);
    const float b = v - fv, c = w - fw;
    const int j0 = wrap_tap((int)fv, A.H), j1 = wrap_tap((int)fv + 1, A.H);
    const int k0 = wrap_tap((int)fw, A.D), k1 = wrap_tap((int)fw + 1, A.D);
    const typename Atlas::Row r00 = T.row(j0, k0), r10 = T.row(j1, k0), r01 = T.row(j0, k1), r11 = T.row(j1, k1);
    Texel2 sum;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        const float u = (s.x + (f == 0 ? fo.x : (f == 1 ? fo.y : fo.z))) * (float)A.W - 0.5f;
        const float fu = floorf(u), a = u - fu;
        const int i0 = wrap_tap((int)fu, A.W), i1 = wrap_tap((int)fu + 1, A.W);
        const typename Atlas::Raw t[8] = {T.texel(r00, i0), T.texel(r00, i1), T.texel(r10, i0), T.texel(r10, i1),
                                          T.texel(r01, i0), T.texel(r01, i1), T.texel(r11, i0), T.texel(r11, i1)};
        Texel2 x;
        if (Atlas::kZeroTest && Atlas::zero(t)) {
            const float z = ((a + b) + c) * 0.0f;  // zero; NaN where a fraction is
            x.rg = x.ba = f2(z);
        } else {
            const F2 a2 = f2(a), b2 = f2(b), c2 = f2(c);
            x = texel_lerp(texel_lerp(texel_lerp(T.decode(t[0]), T.decode(t[1]), a2),
                                      texel_lerp(T.decode(t[2]), T.decode(t[3]), a2), b2),
                           texel_lerp(texel_lerp(T.decode(t[4]), T.decode(t[5]), a2),
                                      texel_lerp(T.decode(t[6]), T.decode(t[7]), a2), b2),
                           c2);
        }
        x = texel_scale(x, f2(f == 0 ? wt.x : (f == 1 ? wt.y : wt.z)));
        sum = f == 0 ? x : texel_add(sum, x);
    }
    return sum;
}

// The filtered sample at a fractional level.
template <class Atlas>
__device__ __forceinline__ float4 sample_levels(const Atlas& T, const MarchScale& C, const vct_cone_tracing_desc& d,
                                                float3 pos, float level, float3 fo, float3 wt) {
    const int lower = (int)floorf(level), upper = (int)ceilf(level);
    const float fr = fractf(level);
    Texel2 lo, hi;
    // one copy of the sampling code, looped; an integral level mixes its sample with itself at fr = 0
#pragma unroll 1
    for (int l = lower;; l = upper) {
        hi = sample_clipmap(T, C, d, pos, l, fo, wt);
        if (l == lower) lo = hi;
        if (l == upper) break;
    }
    return texel_f4(texel_add(texel_scale(lo, f2(1.0f - fr)), texel_scale(hi, f2(fr))));
}

__device__ __forceinline__ float cone_coef(float aperture) { return 2.0f * tanf(aperture * 0.5f); }

// A cone as traceCone sets it up (start already offset by half a step).
struct ConeGeo {
    float3 start, dir, fo, wt, center;
    float uvs, coef, start_level, step_factor;
};

__device__ __forceinline__ ConeGeo make_cone(const vct_cone_tracing_desc& d, float3 start, float3 dir, float coef,
                                             float start_level, float step_factor) {
    ConeGeo K;
    K.uvs = d.voxel_size;
    K.coef = coef;
    const float vs = K.uvs * exp2f(start_level);
    K.start = start + dir * (vs * d.trace_start_offset * 0.5f);
    K.dir = dir;
    K.fo = f3(dir.x > 0.0f ? 0.0f : 1.0f / 6.0f, dir.y > 0.0f ? 2.0f / 6.0f : 3.0f / 6.0f,
              dir.z > 0.0f ? 4.0f / 6.0f : 5.0f / 6.0f);
    K.wt = f3(dir.x * dir.x, dir.y * dir.y, dir.z * dir.z);
    K.center = f3(d.volume_center[0], d.volume_center[1], d.volume_center[2]);
    K.start_level = start_level;
    K.step_factor = step_factor;
    return K;
}

// The loop's schedule at one step: distance, segment length, diameter.
struct Sched {
    float step, seg, diameter;
};

__device__ __forceinline__ Sched first_sched(const ConeGeo& K) {
    return Sched{0.0f, K.uvs * exp2f(K.start_level), fmaxf(0.0f * K.coef, K.uvs)};
}

// step += max(diameter, uvs) * stepFactor (the loop's expressions and order).
__device__ __forceinline__ void sched_advance(Sched& s, const ConeGeo& K) {
    const float prev = s.step;
    s.step = s.step + fmaxf(s.diameter, K.uvs) * K.step_factor;
    s.seg = s.step - prev;
    s.diameter = s.step * K.coef;
}

// What one step adds to its cone: the corrected colour, the opacity and the
// occlusion divisor.
struct StepTerm {
    float3 c;
    float op, q;
    bool some;  // false: all of it leaves the composite as it is
};

// traceCone's loop (voxelConeTracing.frag:341-392) from the sample s of one
// step, at `level`, to the composite.
__device__ __forceinline__ StepTerm cone_term(const vct_cone_tracing_desc& d, const ConeGeo& K, float step, float seg,
                                              float level, float4 s) {
    StepTerm t;
    t.some = true;
    const float vs = K.uvs * exp2f(level);
    const float correction = seg / vs;
    t.c = f3(s.x * correction, s.y * correction, s.z * correction);
    // a filtered alpha rounded above 1 (the face weights sum to 1 + ulp) would make the base of pow
    // negative, which GLSL leaves undefined (NaN, then clamped to a transparent 0 on hardware); the
    // base is taken as 0 there: the sample is opaque
    t.op = clampf(1.0f - powf(fmaxf(1.0f - s.w, 0.0f), correction), 0.0f, 1.0f);
    t.q = 1.0f + (step + vs) * d.occlusion_decay;
    return t;
}

// The step's level (raw_level: cone_raw_level of its diameter).
__device__ __forceinline__ float clamp_level(const MarchScale& C, const ConeGeo& K, float3 pos, float raw_level) {
    const float min_level = cone_min_level(C.inv_r2, C.min_radius, K.center, pos);
    return fminf(fmaxf(fmaxf(K.start_level, raw_level), min_level), (float)(kClipLevels - 1));
}
__device__ __forceinline__ float step_level(const MarchScale& C, const ConeGeo& K, float3 pos, float diameter) {
    return clamp_level(C, K, pos, cone_raw_level(C, diameter, K.uvs));
}

// One step over a clipmap atlas.  `raw_level`: cone_raw_level of the step's diameter.
template <class Atlas>
__device__ __forceinline__ StepTerm exact_step(const Atlas& T, const MarchScale& C, const vct_cone_tracing_desc& d,
                                               const ConeGeo& K, float step, float seg, float raw_level) {
    const float3 pos = K.start + K.dir * step;
    const float level = clamp_level(C, K, pos, raw_level);
    const float4 s = sample_levels(T, C, d, pos, level, K.fo, K.wt);
    StepTerm t;
    t.some = s.x != 0.0f || s.y != 0.0f || s.z != 0.0f || s.w != 0.0f || !(d.occlusion_decay >= 0.0f);
    return t.some ? cone_term(d, K, step, seg, level, s) : t;
}

struct ConeSum {
    float4 c;
    float occlusion;
    __device__ __forceinline__ void add(float3 rc, float op, float q) {
        const float k = clampf(1.0f - c.w, 0.0f, 1.0f);
        c = make_float4(c.x + k * rc.x, c.y + k * rc.y, c.z + k * rc.z, c.w + k * op);
        occlusion = occlusion + (1.0f - occlusion) * op / q;
    }
    __device__ __forceinline__ float4 result() const { return make_float4(c.x, c.y, c.z, 1.0f - occlusion); }
};

// traceCone on one lane.  level_at[k] (k < levels): cone_raw_level of step k,
// where the caller has it.
template <class Atlas>
__device__ __forceinline__ float4 trace_cone(const Atlas& T, const MarchScale& C, const vct_cone_tracing_desc& d,
                                             const ConeGeo& K, float max_dist, const float* level_at, int levels,
                                             unsigned long long& steps) {
    ConeSum sum{make_float4(0.f, 0.f, 0.f, 0.f), 0.0f};
    Sched s = first_sched(K);
    int k = 0;
    for (; s.step < max_dist && sum.occlusion < 1.0f; ++k) {
        const float raw = k < levels ? level_at[k] : cone_raw_level(C, s.diameter, K.uvs);
        const StepTerm t = exact_step(T, C, d, K, s.step, s.seg, raw);
        if (t.some) sum.add(t.c, t.op, t.q);
        sched_advance(s, K);
    }
    steps += (unsigned)k;
    return sum.result();
}

// traceCone by `group` lanes (a power of two up to 8; the whole warp calls,
// 32 / group cones side by side): the lanes of a group take consecutive steps,
// each samples its own (`at(sched)`, a StepTerm), then all add the terms in
// step order, so the sum is the one-lane march's bit for bit and the steps
// after the occlusion stop are dropped.  Every lane returns its cone's sum and
// adds the cone's steps to `taken`.
template <class StepFn>
__device__ __forceinline__ ConeSum march_group(const ConeGeo& K, int group, bool valid, const StepFn& at,
                                               unsigned int& taken) {
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31, first = lane & ~(group - 1);
    const uint32_t firsts = group == 1 ? kFull : (group == 2 ? 0x55555555u : (group == 4 ? 0x11111111u : 0x01010101u));
    ConeSum sum{make_float4(0.f, 0.f, 0.f, 0.f), 0.0f};
    Sched s = first_sched(K);  // the group's next step, the same on its lanes
    bool running = valid && s.step < kMaxTraceDistance;
    while (__any_sync(kFull, running)) {
        Sched mine = s;
        for (int j = 0; j < group; ++j) {
            if (lane - first == j) mine = s;
            sched_advance(s, K);
        }
        const bool has = running && mine.step < kMaxTraceDistance;
        StepTerm t;
        t.some = false;
        if (has) t = at(mine);
        const uint32_t has_mask = __ballot_sync(kFull, has) >> first, some = __ballot_sync(kFull, t.some);
        if (some == 0u) {  // nothing to add in the warp
            taken += __popc(has_mask & ((2u << (group - 1)) - 1u));
        } else {
            for (int j = 0; j < group; ++j) {
                const bool on = ((has_mask >> j) & 1u) && sum.occlusion < 1.0f;
                taken += on;
                if (!((some >> j) & firsts)) continue;  // no cone of the warp adds at its step j
                const int src = first + j;
                const float3 rc = f3(__shfl_sync(kFull, t.c.x, src), __shfl_sync(kFull, t.c.y, src),
                                     __shfl_sync(kFull, t.c.z, src));
                const float op = __shfl_sync(kFull, t.op, src), q = __shfl_sync(kFull, t.q, src);
                if (on && ((some >> src) & 1u)) sum.add(rc, op, q);
            }
        }
        running = running && s.step < kMaxTraceDistance && sum.occlusion < 1.0f;
    }
    return sum;
}

// Lanes per specular cone of a list of m: a power of two up to kMaxConeGroup,
// as few as give every lane of the grid work.  Measured (whole exact trace,
// 65,536 cones on a grid of 32 warps per SM, us): two lanes 1,485, four 1,145,
// eight 1,154; every further lane repeats the additions, so larger lists take
// fewer.
constexpr int kMaxConeGroup = 8;
__device__ __forceinline__ int cone_group(int64_t m) {
    int group = 1;
    while (group < kMaxConeGroup && m * group < (int64_t)gridDim.x * blockDim.x) group <<= 1;
    return group;
}

// What one step computes for the adjoint: the filtered sample, the opacity
// correction, the raw and clamped opacity and the occlusion divisor.
struct StepDetail {
    float correction, op_raw, op, q;
    float4 smp;
};

template <class Atlas>
__device__ __forceinline__ StepDetail exact_step_detail(const Atlas& T, const MarchScale& C,
                                                        const vct_cone_tracing_desc& d, const ConeGeo& K,
                                                        const Sched& s) {
    StepDetail e;
    const float3 pos = K.start + K.dir * s.step;
    const float level = step_level(C, K, pos, s.diameter);
    e.smp = sample_levels(T, C, d, pos, level, K.fo, K.wt);
    const float vs = K.uvs * exp2f(level);
    e.correction = s.seg / vs;
    e.op_raw = 1.0f - powf(fmaxf(1.0f - e.smp.w, 0.0f), e.correction);  // base >= 0 as in cone_term
    e.op = clampf(e.op_raw, 0.0f, 1.0f);
    e.q = 1.0f + (s.step + vs) * d.occlusion_decay;
    return e;
}

// The visiting plan of the exact forms and their adjoint: the samples in the
// coherent order (normal class, then Morton) and the specular samples listed
// grouped by aperture (log-spaced buckets of max(roughness, 0.05)), each group
// in the coherent order, with their count (device).  A cone's step count is
// about proportional to 1 / aperture, so the 32 cones of a warp taken from
// one group march nearly the same number of steps.  Stream-ordered scratch:
// release it with exact_plan_free after the last kernel that reads it.
struct ExactPlan {
    const uint32_t* order;
    uint32_t* spec_list;
    unsigned int* spec_count;
    void* block;
    void* order_block;
};
int exact_plan(const vct_surface_sample* samples, int64_t n, const vct_cone_tracing_desc& d, ExactPlan* plan,
               cudaStream_t st);
void exact_plan_free(ExactPlan* plan, cudaStream_t st);

}  // namespace vct
