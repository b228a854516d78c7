// svo_trace.cu -- OctreeVoxelConeTracing pass (voxelConeTracing_Octree.frag)
// over a sparse-voxel-octree node pool.
//
// Same cone loop as the clipmap tracer, sampling the pool by point location:
// sampleSVO normalises the position by a scene box (the shader hard-codes
// Sponza's), descends from uVolumeDimension to resolution 2^level and reads
// the node's RGBA8; two levels are mixed by fract(level).  FP32 in the
// shader's order (-fmad=false), so the results track the FP32 restatement.
//
// Work layout: the exact clipmap trace's plan (samples in the coherent order;
// the diffuse cones of a warp's samples dealt to its lanes, trace_deal.cuh;
// the specular cones over a list grouped by aperture, one to eight lanes to a
// cone), instead of one thread marching a sample's 17 cones.  The march is
// bound by its own arithmetic (the pool stays in L2, and most of the box is
// empty space that a descent leaves after a node or two), so each step computes
// only what its result needs, every needed value being the shader expression's
// bit for bit:
//   * both levels' nodes come from one descent (the coarser is an ancestor),
//     child slots straight from the cell's bits, a node read as one 8 bytes;
//   * the cell is a fused multiply-add and a floor per axis, the shader's
//     divisions only where the position is within rounding of a cell border;
//   * min_level is the exponent of the squared distance, the square root,
//     division and logarithm only within 2^-16 of a power of two;
//   * the diffuse cones' level by step comes from a table (the schedule is the
//     same for all of them);
//   * a step whose two nodes are zero leaves the composite as it is (where the
//     decay is not negative or NaN), so level size, opacity power and divisions
//     run for the others alone.
// Measured: the trace of 1,000,003 samples on the 4M-triangle terrain at
// L = 9 went from 4.9 to 1.3 ms, 65,536 samples on the room at L = 7 from 0.57
// to 0.17 ms, every output unchanged.
#include <cmath>

#include "trace_deal.cuh"
#include "trace_exact.cuh"

namespace vct {

int fill_trace_params(TraceParams& P, const vct_cone_tracing_desc* desc, const vct_cam_matrix* cam,
                      const vct_shadow_map* shadow, const vct_directional_light_desc* light,
                      const vct_directional_light_shadow_desc* light_shadow);

struct SvoScene {
    const uint2* __restrict__ pool;
    uint32_t nodes;
    uint32_t dim;        // the root resolution, a power of two
    int top;             // its log2 - 1: the cell bit of the first descent step
    float c[3], ev;      // box centre and half extent
    float a, b[3];       // cell coordinate = p * a + b, up to rounding
    float ga, g0[3];     // bound of that rounding: |p| * ga + g0
    float min_radius, inv_r2, inv_uvs;
    bool uvs_pow2;       // voxel_size is a power of two: x * inv_uvs == x / voxel_size
};

// sampleSVO's cell of coordinate p on axis k, clamped to the last cell (the
// shader's cell `resolution` takes the upper child at every step, as the last
// cell does).
__device__ __forceinline__ uint32_t svo_cell(const SvoScene& S, float p, int k) {
    const float q = fmaf(p, S.a, S.b[k]), g = fmaf(fabsf(p), S.ga, S.g0[k]);
    float u = floorf(q);
    const float r = q - u;
    if (!(r > g && r < 1.0f - g)) {  // within rounding of a border (or not finite): the shader's expression
        const float s = (p - S.c[k]) / S.ev;
        u = ((s + 1.0f) * 0.5f) * (float)S.dim;
    }
    return min((uint32_t)fminf(fmaxf(u, 0.0f), 4294967040.0f), S.dim - 1u);
}

// The RGBA8 words of the nodes at levels lo <= hi around p.
__device__ __forceinline__ uint2 svo_nodes(const SvoScene& S, float3 p, uint32_t lo, uint32_t hi) {
    const uint32_t x = svo_cell(S, p.x, 0), y = svo_cell(S, p.y, 1), z = svo_cell(S, p.z, 2);
    const uint32_t target_lo = 1u << lo, target_hi = 1u << hi;
    uint32_t cur = 0, vlo = 0, vhi = 0;
    bool coarse = true;  // the coarser node not reached yet
    int b = S.top;
    for (;;) {
        const uint32_t idx = cur + (((z >> b) & 1u) | (((x >> b) & 1u) << 1) | (((y >> b) & 1u) << 2));
        if (idx >= S.nodes) {  // malformed pool: never read past it, the sample is empty
            vlo = 0;
            if (coarse) vhi = 0;
            break;
        }
        const uint2 n = __ldg(S.pool + idx);
        cur = n.x & 0x7fffffffu;
        vlo = n.y;
        if (coarse) {
            vhi = n.y;
            coarse = cur != 0u && (1u << b) > target_hi;
        }
        if (cur == 0u || (1u << b) <= target_lo) break;
        --b;
    }
    return make_uint2(vlo, vhi);
}

__device__ __forceinline__ float svo_over_uvs(const SvoScene& S, float x, float uvs) {
    return S.uvs_pow2 ? x * S.inv_uvs : x / uvs;
}

// One step of traceCone over the pool.
__device__ __forceinline__ StepTerm svo_step(const SvoScene& S, const vct_cone_tracing_desc& d, const ConeGeo& K,
                                             float step, float seg, float raw_level) {
    const float3 pos = K.start + K.dir * step;
    const float min_level = cone_min_level(S.inv_r2, S.min_radius, K.center, pos);
    const float level = fminf(fmaxf(fmaxf(K.start_level, raw_level), min_level), (float)(kClipLevels - 1));
    const uint2 v = svo_nodes(S, pos, (uint32_t)floorf(level), (uint32_t)ceilf(level));
    StepTerm t;
    // (a divisor that vanishes or is NaN turns a step of no opacity into 0 / 0, which ends the march)
    t.some = (v.x | v.y) != 0u || !(d.occlusion_decay >= 0.0f);
    if (!t.some) return t;
    const float4 a = unpack_rgba8(v.x), b = unpack_rgba8(v.y);
    const float fr = fractf(level);
    return cone_term(d, K, step, seg, level,
                     make_float4(a.x * (1.0f - fr) + b.x * fr, a.y * (1.0f - fr) + b.y * fr,
                                 a.z * (1.0f - fr) + b.z * fr, a.w * (1.0f - fr) + b.w * fr));
}

__device__ __forceinline__ float4 svo_result(const ConeSum& sum) {
    const float4 r = sum.result();
    return make_float4(clampf(r.x, 0.f, 1.f), clampf(r.y, 0.f, 1.f), clampf(r.z, 0.f, 1.f), clampf(r.w, 0.f, 1.f));
}

// traceCone on one lane.  level_at[k] (k < levels): log2(diameter / uvs) of step k, where the caller has it.
__device__ float4 svo_trace_cone(const SvoScene& S, const vct_cone_tracing_desc& d, const ConeGeo& K,
                                 const float* level_at, int levels, unsigned long long& steps) {
    ConeSum sum{make_float4(0.f, 0.f, 0.f, 0.f), 0.0f};
    Sched s = first_sched(K);
    int k = 0;
    for (; s.step < kMaxTraceDistance && sum.occlusion < 1.0f; ++k) {
        const float raw = k < levels ? level_at[k] : log2f(svo_over_uvs(S, s.diameter, K.uvs));
        const StepTerm t = svo_step(S, d, K, s.step, s.seg, raw);
        if (t.some) sum.add(t.c, t.op, t.q);
        sched_advance(s, K);
    }
    steps += (unsigned)k;
    return svo_result(sum);
}

// The rendering-mode switch of voxelConeTracing_Octree.frag, its two outputs.
__device__ __forceinline__ float4 svo_specular_out(uint32_t mode, float3 ispec) {
    if (mode == 6u || mode >= 8u) return make_float4(0.f + ispec.x, 0.f + ispec.y, 0.f + ispec.z, 1.f);
    return make_float4(0.f, 0.f, 0.f, 1.f);
}

struct SvoFinish {
    const DealArgs& A;
    __device__ __forceinline__ void operator()(const GSample& g, float min_level, float4 ind, uint32_t idx) const {
        const TraceParams& P = *A.P;
        const vct_cone_tracing_desc& d = P.d;
        const bool c32 = A.ncones == 32;
        float valid = 0.0f;
        for (int c = 0; c < A.ncones; ++c) {
            const float3 dir = c32 ? f3(c_dirs32[c][0], c_dirs32[c][1], c_dirs32[c][2])
                                   : f3(c_dirs16[c][0], c_dirs16[c][1], c_dirs16[c][2]);
            const float cos_t = dot3(g.normal, dir);
            if (!(cos_t < 0.0f)) valid = valid + cos_t;
        }
        ind = make_float4(ind.x / valid, ind.y / valid, ind.z / valid, ind.w / valid);
        ind.w = ind.w * d.ambient_occlusion_factor;
        ind.x = ind.x * (g.diffuse_color.x * d.indirect_diffuse_intensity);
        ind.y = ind.y * (g.diffuse_color.y * d.indirect_diffuse_intensity);
        ind.z = ind.z * (g.diffuse_color.z * d.indirect_diffuse_intensity);
        ind = make_float4(clampf(ind.x, 0.f, 1.f), clampf(ind.y, 0.f, 1.f), clampf(ind.z, 0.f, 1.f), clampf(ind.w, 0.f, 1.f));
        float3 direct = direct_term(P, g);
        direct = f3(clampf(direct.x, 0.f, 1.f), clampf(direct.y, 0.f, 1.f), clampf(direct.z, 0.f, 1.f));
        float4 D = make_float4(0.f, 0.f, 0.f, 1.f);
        switch (d.rendering_mode) {
            case 0: D = make_float4(g.diffuse_color.x, g.diffuse_color.y, g.diffuse_color.z, 1.f); break;
            case 1: D = make_float4(g.specular_color.x, g.specular_color.y, g.specular_color.z, 1.f); break;
            case 2:
                D = make_float4(g.normal.x * 0.5f + 0.5f, g.normal.y * 0.5f + 0.5f, g.normal.z * 0.5f + 0.5f, 1.f);
                break;
            case 3: {
                const float colors[7][4] = {{1, 0, 0, 1}, {0, 1, 0, 1}, {0, 0, 1, 1}, {1, 1, 0, 1},
                                            {0, 1, 1, 1}, {1, 0, 1, 1}, {1, 1, 1, 1}};
                float v[4] = {0.f, 0.f, 0.f, 0.f};
                for (int k = 0; k < 6; ++k)
                    if (min_level < (float)(k + 1)) {
                        const float fr = fractf(min_level);
                        for (int c = 0; c < 4; ++c) v[c] = colors[k][c] * (1.0f - fr) + colors[k + 1][c] * fr;
                        break;
                    }
                D = make_float4(v[0] * 0.5f, v[1] * 0.5f, v[2] * 0.5f, v[3] * 0.5f);
                break;
            }
            case 4:
                direct = direct * ind.w;
                D = make_float4(direct.x, direct.y, direct.z, 1.f);
                break;
            case 5: D = make_float4(D.x + ind.x, D.y + ind.y, D.z + ind.z, 1.f); break;
            case 6: break;
            case 7: D = make_float4(ind.w, ind.w, ind.w, 1.f); break;
            default:
                direct = direct * ind.w;
                D = make_float4(D.x + direct.x + ind.x, D.y + direct.y + ind.y, D.z + direct.z + ind.z, 1.f);
                break;
        }
        reinterpret_cast<float4*>(A.dout)[idx] = D;
        if (!has_specular_cone(g))
            reinterpret_cast<float4*>(A.sout)[idx] = svo_specular_out(d.rendering_mode, f3(0.f, 0.f, 0.f));
    }
};

constexpr int kSvoWarps = 4;  // warps per block of the diffuse kernel
constexpr int kSvoWarpsPerSm = 16;  // warp items per SM that deal_samples_per_warp aims at
// Warps per SM of a full specular grid, which the lanes per cone follow
// (65,536 samples on the room, us of the whole case: 16: 954, 32: 894, 40: 893, 64: 872).
constexpr int kSvoSpecWarpsPerSm = 64;
constexpr int kSvoLevels = 128;  // steps of the diffuse schedule kept as a table (default descriptors take 19 to 40)

struct SvoDiffuseMarch {
    const SvoScene* S;
    const vct_cone_tracing_desc* d;
    float coef, step_factor;
    const float* level_at;
    int levels;
    __device__ __forceinline__ float4 operator()(float3 start, float3 dir, float start_level,
                                                 unsigned long long& steps) const {
        return svo_trace_cone(*S, *d, make_cone(*d, start, dir, coef, start_level, step_factor), level_at, levels, steps);
    }
};

__global__ void __launch_bounds__(32 * kSvoWarps) k_svo_diffuse(const __grid_constant__ TraceParams P,
                                                                const __grid_constant__ SvoScene S,
                                                                const vct_surface_sample* __restrict__ samples,
                                                                int64_t n, const uint32_t* __restrict__ order,
                                                                float* __restrict__ dout, float* __restrict__ sout,
                                                                unsigned long long* __restrict__ step_counter,
                                                                unsigned int* __restrict__ ticket, int per_warp) {
    __shared__ float s_level[kSvoLevels];
    __shared__ int s_levels;
    const bool c32 = P.d.enable_32_cones != 0;
    const float uvs = P.d.voxel_size;
    const float coef = 2.0f * tanf((c32 ? kAperture32 : kAperture16) * 0.5f);
    const float sf = fmaxf(kMinTraceStepFactor, P.d.min_trace_step_factor);
    if (threadIdx.x == 0) {  // the march's own recurrence
        float step = 0.0f, diameter = fmaxf(step * coef, uvs);
        int k = 0;
        for (; k < kSvoLevels && step < kMaxTraceDistance; ++k) {
            s_level[k] = diameter;
            step = step + fmaxf(diameter, uvs) * sf;
            diameter = step * coef;
        }
        s_levels = k;
    }
    __syncthreads();
    const int levels = s_levels;
    for (int k = threadIdx.x; k < levels; k += blockDim.x) s_level[k] = log2f(svo_over_uvs(S, s_level[k], uvs));
    __syncthreads();
    DealArgs D{&P, samples, n, order, 0u, (uint32_t)n, dout, sout, c32 ? 32 : 16, true, true, per_warp};
    unsigned long long steps = 0;
    deal_cones<kSvoWarps, true>(D, SvoDiffuseMarch{&S, &P.d, coef, sf, s_level, levels}, SvoFinish{D}, steps, ticket);
    add_steps(step_counter, steps);
}

// A group of lanes (cone_group) per specular cone of the aperture-grouped
// list, a warp's worth at a time to the warps as they free up.
__global__ void __launch_bounds__(128) k_svo_specular(const __grid_constant__ TraceParams P,
                                                      const __grid_constant__ SvoScene S,
                                                      const vct_surface_sample* __restrict__ samples,
                                                      const uint32_t* __restrict__ list,
                                                      const unsigned int* __restrict__ spec_count,
                                                      float* __restrict__ sout,
                                                      unsigned long long* __restrict__ step_counter,
                                                      unsigned int* __restrict__ ticket) {
    const vct_cone_tracing_desc& d = P.d;
    const uint32_t m = *spec_count;
    const int lane = threadIdx.x & 31;
    const int group = cone_group(m), cones = 32 / group, first = lane & ~(group - 1);
    unsigned long long steps = 0;
    for (;;) {
        uint32_t c0 = 0;
        if (lane == 0) c0 = atomicAdd(ticket, (unsigned)cones);
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        if (c0 >= m) break;
        const uint32_t c = c0 + (uint32_t)(lane / group);
        const bool valid = c < m;
        const uint32_t idx = __ldg(list + (valid ? c : c0));
        const GSample g = load_sample(samples + idx, P.eye);
        const float min_level = calc_min_level(d, g.wp);
        const float vs = d.voxel_size * exp2f(min_level);
        const float3 start = g.wp + g.normal * (vs * d.trace_start_offset);
        const float3 sdir = normalize3(reflect3(f3(-g.view.x, -g.view.y, -g.view.z), g.normal));
        const ConeGeo K = make_cone(d, start, sdir, cone_coef(fmaxf(g.roughness, kMinSpecularAperture)), min_level,
                                    fmaxf(kMinTraceStepFactor, d.voxel_size));
        float4 r;
        if (group == 1) {  // the groups' ballots and shuffles cost a tenth of a long list's time
            if (!valid) continue;
            r = svo_trace_cone(S, d, K, nullptr, 0, steps);
        } else {
            unsigned int taken = 0;
            const ConeSum sum = march_group(K, group, valid, [&](const Sched& s) {
                return svo_step(S, d, K, s.step, s.seg, log2f(svo_over_uvs(S, s.diameter, K.uvs)));
            }, taken);
            if (lane != first || !valid) continue;
            steps += taken;
            r = svo_result(sum);
        }
        const float isi = d.indirect_specular_intensity;
        reinterpret_cast<float4*>(sout)[idx] = svo_specular_out(
            d.rendering_mode,
            f3(r.x * g.specular_color.x * isi, r.y * g.specular_color.y * isi, r.z * g.specular_color.z * isi));
    }
    add_steps(step_counter, steps);
}

}  // namespace vct

using namespace vct;

extern "C" int vct_svo_cone_trace(const vct_cone_tracing_desc* desc, const vct_cam_matrix* cam, const uint32_t* pool,
                                  int64_t node_count, const float bb_min[3], const float bb_max[3],
                                  const vct_shadow_map* shadow, const vct_directional_light_desc* light,
                                  const vct_directional_light_shadow_desc* light_shadow,
                                  const vct_surface_sample* samples, int64_t n, float* dout, float* sout,
                                  unsigned long long* cone_steps, void* stream) {
    VCT_CHECK_ARG(pool && node_count >= 8 && bb_min && bb_max, "vct_svo_cone_trace: bad node pool / scene box");
    VCT_CHECK_ARG(n >= 0, "vct_svo_cone_trace: negative sample count");
    if (n == 0) return VCT_OK;
    VCT_CHECK_ARG(samples && dout && sout, "vct_svo_cone_trace: null sample or output buffer");
    VCT_CHECK_ARG(((uintptr_t)samples & 15) == 0 && ((uintptr_t)dout & 15) == 0 && ((uintptr_t)sout & 15) == 0,
                  "vct_svo_cone_trace: buffers must be 16-byte aligned");
    TraceParams P;
    int rc = fill_trace_params(P, desc, cam, shadow, light, light_shadow);
    if (rc != VCT_OK) return rc;
    const uint32_t dim = (uint32_t)desc->volume_dimension;
    VCT_CHECK_ARG(dim >= 2 && (dim & (dim - 1)) == 0 && dim <= 4096,
                  "vct_svo_cone_trace: volume dimension must be a power of two (the pool's root resolution)");
    SvoScene S;
    S.pool = reinterpret_cast<const uint2*>(pool);
    VCT_CHECK_ARG(node_count < (1LL << 31), "vct_svo_cone_trace: node count out of range");
    S.nodes = (uint32_t)node_count;
    S.dim = dim;
    S.top = 30 - __builtin_clz(dim);
    float ext[3];
    for (int a = 0; a < 3; ++a) {
        ext[a] = bb_max[a] - bb_min[a];
        S.c[a] = (bb_min[a] + bb_max[a]) * 0.5f;
    }
    S.ev = fmaxf(ext[0], fmaxf(ext[1], ext[2])) * 0.5f;
    const double scale = 0.5 * (double)dim / (double)S.ev;
    S.a = (float)scale;
    S.ga = (float)(fabs(scale) * 0x1p-20);
    for (int a = 0; a < 3; ++a) {
        const double off = 0.5 * (double)dim - (double)S.c[a] * scale;
        S.b[a] = (float)off;
        S.g0[a] = (float)((fabs((double)S.c[a] * scale) + (double)dim) * 0x1p-20);
    }
    S.min_radius = desc->voxel_size * desc->volume_dimension * 0.5f;
    S.inv_r2 = (float)(1.0 / ((double)S.min_radius * (double)S.min_radius));
    if (!std::isnormal(S.inv_r2)) S.inv_r2 = 0.0f;  // the shader's expression everywhere
    S.inv_uvs = 1.0f / desc->voxel_size;
    int exponent = 0;
    S.uvs_pow2 = frexpf(desc->voxel_size, &exponent) == 0.5f && exponent > -120 && exponent < 120;
    // counts of 2^30 samples or more run in chunks (the orders are 32-bit)
    cudaStream_t st = as_stream(stream);
    constexpr int64_t kChunk = 1LL << 30;
    for (int64_t off = 0; off < n; off += kChunk) {
        const int64_t m = n - off < kChunk ? n - off : kChunk;
        const vct_surface_sample* smp = samples + off;
        ExactPlan plan;
        rc = exact_plan(smp, m, P.d, &plan, st);
        if (rc != VCT_OK) return rc;
        const int sms = sm_count(), per_warp = deal_samples_per_warp(m, (int64_t)sms * kSvoWarpsPerSm);
        const int64_t gd = (m + (int64_t)per_warp * kSvoWarps - 1) / ((int64_t)per_warp * kSvoWarps);
        k_svo_diffuse<<<(int)(gd > sms * 8 ? sms * 8 : gd), 32 * kSvoWarps, 0, st>>>(
            P, S, smp, m, plan.order, dout + 4 * off, sout + 4 * off, cone_steps, plan.spec_count + 2, per_warp);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) {
            const int64_t gs = (m * kMaxConeGroup + 127) / 128, full = (int64_t)sms * kSvoSpecWarpsPerSm / 4;
            k_svo_specular<<<(int)(gs > full ? full : gs), 128, 0, st>>>(
                P, S, smp, plan.spec_list, plan.spec_count, sout + 4 * off, cone_steps, plan.spec_count + 1);
            e = cudaGetLastError();
        }
        exact_plan_free(&plan, st);
        if (e != cudaSuccess) return cuda_fail(e, "octree cone trace");
    }
    return VCT_OK;
}
