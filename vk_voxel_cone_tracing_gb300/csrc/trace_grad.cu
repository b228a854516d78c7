// trace_grad.cu -- the adjoint of the FP32 cone trace over a float atlas
// (vct_cone_trace_f32): given dL/d(diffuse out) and dL/d(specular out) per
// sample, accumulate dL/d(texel) into a float RGBA atlas of the same layout.
//
// The march's step schedule, levels, tap positions, opacity corrections and
// occlusion divisors depend on geometry only; the number of steps depends on
// the volume through the occlusion stop and is held fixed (the derivative of
// a piecewise-smooth function away from its switches).  The clamps of the
// opacity and of 1 - alpha pass the derivative of their argument when it lies
// in [0, 1], bounds included: from an empty texel (alpha 0) the opacity's
// right derivative reaches it, which is the one inverse fitting needs.
//
// With T_i = prod_{m<i} (1 - op_m) (the weight clamp(1 - alpha) of step i),
// U_i = prod_{m<i} (1 - op_m / q_m) (1 - occlusion before step i),
// q_i = 1 + (t_i + vs_i) decay and c_i the opacity correction, the cone
// returns C = sum_i T_i c_i s_i.rgb and O = 1 - U_n, so for L = gC . C + gO O
//     dL/d(s_i.rgb) = gC T_i c_i
//     dL/d(op_i)    = -T_i R_i + gO U_i V_i / q_i,
//     R_i = sum_{j>i} prod_{i<m<j} (1 - op_m) c_j gC . s_j.rgb,
//     V_i = prod_{j>i} (1 - op_j / q_j),
//     dL/d(s_i.a)   = dL/d(op_i) c_i (1 - s_i.a)^(c_i - 1).
// g(s_i) is split over the two levels (1 - fr, fr), the three faces (the
// direction weights) and the eight texels of each trilinear tap (the products
// of the lerp fractions) and added to the gradient atlas with float4 atomics.
// Same FP32 expressions as the forward kernels (this unit is built with
// -fmad=false like them), so the recomputed steps are the forward's.
//
// A cone is walked by one lane or, where the cones are few, by a group of
// lanes that take consecutive steps (march_group's split): a march forward
// keeps a record of each of the first kStoredRounds rounds' steps (the state
// before the step, its opacity terms, its colour against gC, its distance) in
// device scratch and a checkpoint of the march every kSegRounds rounds after
// those; the walk backward, with the recurrences above in sequential form,
// reads the records, a later segment's after marching it again from its
// checkpoint.  Diffuse cones all share one step schedule; specular cones are
// taken from the exact forward's aperture-grouped list, so a warp's cones also
// march nearly the same number of steps.  Work goes to the warps as they free
// up.
//
// Bound by the scatter: up to 48 float4 atomics a step (274 M sectors of them
// in the diffuse kernel of 65,536 samples at R = 64; L1 wavefronts 61 % and L2
// 50 % of their peaks).  One lane a cone, 128 steps of 12 fields and a static
// deal took 1.78 ms for the specular cones, whose longest marches outlast the
// rest by half, and 1.64 ms for the diffuse ones, with 478 MB of records whose
// allocation cost another 1.2 ms a call; this takes 1.33 and 1.50 ms with
// 174 MB.
#include <algorithm>

#include "trace_exact.cuh"

namespace vct {

int fill_trace_params(TraceParams& P, const vct_cone_tracing_desc* desc, const vct_cam_matrix* cam,
                      const vct_shadow_map* shadow, const vct_directional_light_desc* light,
                      const vct_directional_light_shadow_desc* light_shadow);

namespace {

constexpr int kMaxSteps = 8192;  // per cone: the specular cone at R = 1024 takes ~7.1k
// Rounds (one step a lane) whose records the forward march keeps, and of a
// segment marched again: default diffuse cones take 19 to 40.
constexpr int kStoredRounds = 48, kSegRounds = 32;
constexpr int kMaxSegments = (kMaxSteps - kStoredRounds + kSegRounds - 1) / kSegRounds;

// A lane's records lie in a block of its warp (device scratch, one block per
// warp of the grid, fields outermost and lanes innermost: a warp's store or
// load of a field is one 128-byte line); the segment marched again has the
// block's last kSegRounds rounds.  What a step's level, tap positions and
// occlusion divisor take is computed again from its distance.
enum RecField { kRecAlpha, kRecOcc, kRecOp, kRecSlope, kRecColour, kRecCorr, kRecStep, kRecFields };
constexpr size_t kRecRounds = kStoredRounds + kSegRounds;
constexpr size_t kRecWarpFloats = (size_t)kRecFields * kRecRounds * 32;
__device__ __forceinline__ float& rec_at(float* rec, int field, int slot) {
    return rec[((size_t)field * kRecRounds + slot) * 32 + (threadIdx.x & 31)];
}

// Diffuse cones per warp group: 0 deals them cone-major (each cone slot over
// all samples of the coherent order in turn); T > 0 deals all slots of T
// consecutive samples before the next T.
constexpr int kDiffuseTile = 1024;

struct MarchState {
    float step, seg, diameter, alpha, occ;
};

__device__ __forceinline__ void add4(float4* p, float4 v) {
    if (v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f) atomicAdd(p, v);
}

// Adjoint of texture3d: the eight texels' shares of g.
__device__ __forceinline__ void texture3d_grad(float4* __restrict__ G, const AtlasDims& A, float ux, float uy, float uz,
                                               float4 g) {
    float u = ux * (float)A.W - 0.5f, v = uy * (float)A.H - 0.5f, w = uz * (float)A.D - 0.5f;
    float fu = floorf(u), fv = floorf(v), fw = floorf(w);
    float a = u - fu, b = v - fv, c = w - fw;
    int i0 = wrap_tap((int)fu, A.W), i1 = wrap_tap((int)fu + 1, A.W);
    int j0 = wrap_tap((int)fv, A.H), j1 = wrap_tap((int)fv + 1, A.H);
    int k0 = wrap_tap((int)fw, A.D), k1 = wrap_tap((int)fw + 1, A.D);
    const float wi[2] = {1.0f - a, a}, wj[2] = {1.0f - b, b}, wk[2] = {1.0f - c, c};
    const int ii[2] = {i0, i1}, jj[2] = {j0, j1}, kk[2] = {k0, k1};
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float wt = wi[x] * wj[y] * wk[z];
                add4(G + A.index(ii[x], jj[y], kk[z]), make_float4(g.x * wt, g.y * wt, g.z * wt, g.w * wt));
            }
}

// Adjoint of sample_clipmap: the three face taps' shares (one copy of the
// tap code, looped: the kernel is instruction-fetch bound when it is inlined
// six times per step).
__device__ __forceinline__ void sample_clipmap_grad(float4* __restrict__ G, const AtlasDims& A,
                                                    const MarchScale& C, const vct_cone_tracing_desc& d, float3 p,
                                                    int level, float3 fo,
                                                    float3 wt, float4 g) {
    const float3 s = clipmap_coords(C, d, p, level);
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
        const float off = f == 0 ? fo.x : (f == 1 ? fo.y : fo.z);
        const float w = f == 0 ? wt.x : (f == 1 ? wt.y : wt.z);
        texture3d_grad(G, A, s.x + off, s.y, s.z, make_float4(g.x * w, g.y * w, g.z * w, g.w * w));
    }
}

// g(s) of one step spread over its levels, faces and texels.
__device__ __forceinline__ void scatter_step(float4* __restrict__ G, const AtlasDims& A, const MarchScale& C,
                                             const vct_cone_tracing_desc& d,
                                             const ConeGeo& K, float3 pos, int lower, int upper, float fr, float4 gs) {
    // s = lo (1 - fr) + hi fr: the lower level's share, then the upper's (zero when fr = 0)
#pragma unroll 1
    for (int lv = 0; lv < 2; ++lv) {
        const float f = lv ? fr : 1.0f - fr;
        if (f == 0.0f) continue;
        sample_clipmap_grad(G, A, C, d, pos, lv ? upper : lower, K.fo, K.wt,
                            make_float4(gs.x * f, gs.y * f, gs.z * f, gs.w * f));
    }
}

// d(op)/d(s.a) for op = clamp(1 - (1 - s.a)^c, 0, 1), the bounds inside.
__device__ __forceinline__ float opacity_slope(const StepDetail& e) {
    const float base = 1.0f - e.smp.w;
    return (e.op_raw >= 0.0f && e.op_raw <= 1.0f && base > 0.0f) ? e.correction * powf(base, e.correction - 1.0f)
                                                                   : 0.0f;
}

// A group's cone during its walk: one value on all of the group's lanes.
struct Group {
    int size, first;  // lanes; the first of them
    __device__ __forceinline__ int at() const { return (int)(threadIdx.x & 31) - first; }
};

// One round of trace_cone (same expressions) from march state m, which it
// advances: each lane samples its step, then the states before the steps
// follow in step order.  Writes the lane's record to `slot`; false where the
// cone does not have the lane's step.
__device__ __forceinline__ bool march_round(const F4Atlas& T, const MarchScale& C, const vct_cone_tracing_desc& d,
                                            const ConeGeo& K, const Group& g, float3 gC, float max_dist, bool running,
                                            MarchState& m, float* rec, int slot) {
    constexpr unsigned kFull = 0xffffffffu;
    Sched s{m.step, m.seg, m.diameter}, mine = s;
    for (int j = 0; j < g.size; ++j) {
        if (g.at() == j) mine = s;
        sched_advance(s, K);
    }
    const bool has = running && mine.step < max_dist;
    StepDetail e;
    e.op = e.q = 0.0f;
    if (has) e = exact_step_detail(T, C, d, K, mine);
    const uint32_t has_mask = __ballot_sync(kFull, has) >> g.first;
    float alpha = m.alpha, occ = m.occ, alpha0 = 0.0f, occ0 = 0.0f;
    bool mine_on = false;
    for (int j = 0; j < g.size; ++j) {
        const bool on = ((has_mask >> j) & 1u) && occ < 1.0f;
        const float op = __shfl_sync(kFull, e.op, g.first + j), q = __shfl_sync(kFull, e.q, g.first + j);
        if (g.at() == j) {
            alpha0 = alpha;
            occ0 = occ;
            mine_on = on;
        }
        if (on) {
            const float k = clampf(1.0f - alpha, 0.0f, 1.0f);
            alpha = alpha + k * op;
            occ = occ + (1.0f - occ) * op / q;
        }
    }
    if (running) m = MarchState{s.step, s.seg, s.diameter, alpha, occ};
    if (mine_on) {
        rec_at(rec, kRecAlpha, slot) = alpha0;
        rec_at(rec, kRecOcc, slot) = occ0;
        rec_at(rec, kRecOp, slot) = e.op;
        rec_at(rec, kRecSlope, slot) = opacity_slope(e);
        rec_at(rec, kRecColour, slot) = (gC.x * e.smp.x + gC.y * e.smp.y + gC.z * e.smp.z) * e.correction;
        rec_at(rec, kRecCorr, slot) = e.correction;
        rec_at(rec, kRecStep, slot) = mine.step;
    }
    return mine_on;
}

// The adjoint of a warp's cones, g.size lanes to each: gC (rgb) and gO (d/d
// occlusion) at the end of the march.  The warp's lanes run in lock step:
// every loop runs to the warp's longest march and a lane sits out the steps
// its cone does not have (or all of them when `active` is false).
// `rec`: the warp's record block (kRecWarpFloats floats), written and read
// by each lane for its own steps only.
__device__ void cone_backward(const F4Atlas& T, float4* __restrict__ G, const MarchScale& C,
                              const vct_cone_tracing_desc& d, const ConeGeo& K, const Group& g, float3 gC, float gO,
                              bool active, float max_dist, float* rec, int* __restrict__ err) {
    constexpr unsigned kFull = 0xffffffffu;
    MarchState ckpt[kMaxSegments];
    const Sched s0 = first_sched(K);
    MarchState m{s0.step, s0.seg, s0.diameter, 0.0f, 0.0f};
    int rounds = 0, mine = 0;  // of the cone, and those in which it has the lane's step (the first ones)
    bool running = active && m.step < max_dist && m.occ < 1.0f;
    for (int j = 0; __any_sync(kFull, running); ++j) {  // j is warp-uniform
        if (j * g.size >= kMaxSteps) {
            if (running) atomicOr(err, 1);
            return;
        }
        const int past = j - kStoredRounds;
        if (past >= 0 && past % kSegRounds == 0) ckpt[past / kSegRounds] = m;
        const int slot = past < 0 ? j : kStoredRounds + past % kSegRounds;
        mine += march_round(T, C, d, K, g, gC, max_dist, running, m, rec, slot);
        rounds += running;
        running = running && m.step < max_dist && m.occ < 1.0f;
    }
    const int nmax = __reduce_max_sync(kFull, rounds);
    float gA = 0.0f;
    int kept = (nmax - 1 - kStoredRounds) / kSegRounds;  // the segment whose records the block holds
    for (int j = nmax - 1; j >= 0; --j) {
        const int past = j - kStoredRounds, seg = past / kSegRounds;
        if (past >= 0 && seg != kept) {  // march the segment again
            MarchState r = ckpt[seg];
            for (int i = 0; i < kSegRounds; ++i)
                march_round(T, C, d, K, g, gC, max_dist, kStoredRounds + seg * kSegRounds + i < rounds, r, rec,
                            kStoredRounds + i);
            kept = seg;
        }
        const int slot = past < 0 ? j : kStoredRounds + past % kSegRounds;
        const bool on = j < mine;
        float alpha = 0.0f, occ = 0.0f, op = 0.0f, slope = 0.0f, colour = 0.0f, c = 0.0f, q = 1.0f, level = 0.0f;
        float3 pos = f3(0.f, 0.f, 0.f);
        if (on) {
            alpha = rec_at(rec, kRecAlpha, slot);
            occ = rec_at(rec, kRecOcc, slot);
            op = rec_at(rec, kRecOp, slot);
            slope = rec_at(rec, kRecSlope, slot);
            colour = rec_at(rec, kRecColour, slot);
            c = rec_at(rec, kRecCorr, slot);
            const float step = rec_at(rec, kRecStep, slot);
            // exact_step_detail's expressions
            pos = K.start + K.dir * step;
            level = step_level(C, K, pos, j == 0 && g.at() == 0 ? first_sched(K).diameter : step * K.coef);
            q = 1.0f + (step + K.uvs * exp2f(level)) * d.occlusion_decay;
        }
        const float k_raw = 1.0f - alpha, k = clampf(k_raw, 0.0f, 1.0f);
        const float keep = 1.0f - op / q;
        const uint32_t on_mask = __ballot_sync(kFull, on) >> g.first;
        const uint32_t in_mask = __ballot_sync(kFull, k_raw >= 0.0f && k_raw <= 1.0f) >> g.first;
        float my_gA = 0.0f, my_gO = 0.0f;
        for (int i = g.size - 1; i >= 0; --i) {
            const int src = g.first + i;
            const float op_i = __shfl_sync(kFull, op, src), colour_i = __shfl_sync(kFull, colour, src);
            const float keep_i = __shfl_sync(kFull, keep, src);
            if (g.at() == i) {
                my_gA = gA;
                my_gO = gO;
            }
            if ((on_mask >> i) & 1u) {
                if ((in_mask >> i) & 1u) gA = gA - (colour_i + gA * op_i);
                gO = gO * keep_i;
            }
        }
        if (on) {
            float4 gs;
            gs.x = gC.x * k * c;
            gs.y = gC.y * k * c;
            gs.z = gC.z * k * c;
            const float gop = my_gA * k + my_gO * (1.0f - occ) / q;
            gs.w = gop * slope;
            scatter_step(G, T.A, C, d, K, pos, (int)floorf(level), (int)ceilf(level), fractf(level), gs);
        }
    }
}

// dL/d(indirect) -> the diffuse cones' gC and gO; false when the mode does
// not read the volume through the diffuse cones.
__device__ __forceinline__ bool diffuse_seeds(const TraceParams& P, const GSample& g, float4 GD, float cos_t, int nc,
                                              float3& gC, float& gO) {
    const vct_cone_tracing_desc& d = P.d;
    const uint32_t mode = d.rendering_mode;
    // D.rgb = direct * ind.w + ind.rgb (modes 5 and the default), direct * ind.w (4), ind.w (7)
    float3 g_ind = f3(0.f, 0.f, 0.f);
    float g_ao = 0.0f;
    const bool rgb_mode = mode == 5 || mode >= 8;
    if (rgb_mode) g_ind = f3(GD.x, GD.y, GD.z);
    if (rgb_mode || mode == 4) {
        const float3 direct = direct_term(P, g);
        g_ao = GD.x * direct.x + GD.y * direct.y + GD.z * direct.z;
    } else if (mode == 7) {
        g_ao = GD.x + GD.y + GD.z;
    }
    const float w = cos_t / (float)nc;
    gC = f3(g_ind.x * w * (g.diffuse_color.x * d.indirect_diffuse_intensity),
            g_ind.y * w * (g.diffuse_color.y * d.indirect_diffuse_intensity),
            g_ind.z * w * (g.diffuse_color.z * d.indirect_diffuse_intensity));
    gO = -(g_ao * w * d.ambient_occlusion_factor);  // the cone returns 1 - occlusion
    return !(gC.x == 0.0f && gC.y == 0.0f && gC.z == 0.0f && gO == 0.0f);
}

__global__ void __launch_bounds__(128) k_cone_backward_diffuse(const __grid_constant__ TraceParams P,
                                                               const __grid_constant__ MarchScale C, F4Atlas T,
                                                               const vct_surface_sample* __restrict__ samples,
                                                               int64_t n, const uint32_t* __restrict__ order,
                                                               const float4* __restrict__ gd, float4* __restrict__ G,
                                                               float* rec_all, int* __restrict__ err,
                                                               unsigned int* __restrict__ ticket) {
    const vct_cone_tracing_desc& d = P.d;
    float* rec = rec_all + (size_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kRecWarpFloats;
    const bool c32 = d.enable_32_cones != 0;
    const int nc = c32 ? 32 : 16;
    const int lane = threadIdx.x & 31;
    const int64_t total = n * nc;
    const Group g1{1, lane};
    for (;;) {
        unsigned int item = 0;
        if (lane == 0) item = atomicAdd(ticket, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        const int64_t t0 = (int64_t)item * 32;
        if (t0 >= total) break;
        const int64_t t = t0 + lane;
        bool active = t < total;
        // a warp's lanes march the same cone of consecutive samples in the coherent order (the same direction
        // from neighbouring points: the lanes stay in step and share texels), all cones of kDiffuseTile samples
        // before the next kDiffuseTile (the resident warps' gradient scatter then stays near one patch)
        int slot = 0;
        int64_t u = 0;
        if (active && kDiffuseTile > 0) {
            const int64_t per = (int64_t)kDiffuseTile * nc, tile = t / per, base = tile * kDiffuseTile;
            const int64_t len = min((int64_t)kDiffuseTile, n - base), r = t - tile * per;
            slot = (int)(r / len);
            u = base + (r - (int64_t)slot * len);
        } else if (active) {
            slot = (int)(t / n);
            u = t - (int64_t)slot * n;
        }
        const int64_t i = order ? (int64_t)__ldg(order + u) : u;
        const GSample g = load_sample(samples + i, P.eye);
        active = active && g.depth != 1.0f;
        const float min_level = calc_min_level(d, g.wp);
        const float vs = d.voxel_size * exp2f(min_level);
        const float3 start = g.wp + g.normal * (vs * d.trace_start_offset);
        const float3 dir = c32 ? f3(c_dirs32[slot][0], c_dirs32[slot][1], c_dirs32[slot][2])
                               : f3(c_dirs16[slot][0], c_dirs16[slot][1], c_dirs16[slot][2]);
        const float cos_t = dot3(g.normal, dir);
        active = active && cos_t >= 0.0f;
        float3 gC = f3(0.f, 0.f, 0.f);
        float gO = 0.0f;
        active = active && diffuse_seeds(P, g, gd[i], cos_t, nc, gC, gO);
        const ConeGeo K = make_cone(d, start, dir, cone_coef(P.diffuse_aperture), min_level,
                                    fmaxf(kMinTraceStepFactor, d.min_trace_step_factor));
        cone_backward(T, G, C, d, K, g1, gC, gO, active, kMaxTraceDistance, rec, err);
    }
}

// A group of lanes (cone_group) per specular cone of the aperture-grouped list
// (a warp's cones share their step schedule, so the lock-step walk keeps its
// lanes busy).
__global__ void __launch_bounds__(128) k_cone_backward_specular(
    const __grid_constant__ TraceParams P, const __grid_constant__ MarchScale C, F4Atlas T,
    const vct_surface_sample* __restrict__ samples, const uint32_t* __restrict__ list,
    const unsigned int* __restrict__ spec_count, const float4* __restrict__ gsp, float4* __restrict__ G,
    float* rec_all, int* __restrict__ err,
                                                               unsigned int* __restrict__ ticket) {
    const vct_cone_tracing_desc& d = P.d;
    float* rec = rec_all + (size_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kRecWarpFloats;
    if (!(d.rendering_mode == 6 || d.rendering_mode >= 8)) return;
    const int lane = threadIdx.x & 31;
    const int64_t m = *spec_count;
    const int group = cone_group(m), cones = 32 / group;
    const Group gr{group, lane & ~(group - 1)};
    for (;;) {
        unsigned int t0 = 0;
        if (lane == 0) t0 = atomicAdd(ticket, (unsigned)cones);
        t0 = __shfl_sync(0xffffffffu, t0, 0);
        if ((int64_t)t0 >= m) break;
        const int64_t t = (int64_t)t0 + lane / group;
        bool active = t < m;
        const uint32_t i = __ldg(list + (active ? t : (int64_t)t0));
        const GSample g = load_sample(samples + i, P.eye);
        const float4 GS = gsp[i];
        const float isi = d.indirect_specular_intensity;
        const float3 gC = f3(GS.x * g.specular_color.x * isi, GS.y * g.specular_color.y * isi,
                             GS.z * g.specular_color.z * isi);
        active = active && !(gC.x == 0.0f && gC.y == 0.0f && gC.z == 0.0f);
        const float min_level = calc_min_level(d, g.wp);
        const float vs = d.voxel_size * exp2f(min_level);
        const float3 start = g.wp + g.normal * (vs * d.trace_start_offset);
        const float3 sdir = reflect3(f3(-g.view.x, -g.view.y, -g.view.z), g.normal);
        const ConeGeo K = make_cone(d, start, sdir, cone_coef(fmaxf(g.roughness, kMinSpecularAperture)), min_level,
                                    d.voxel_size);
        cone_backward(T, G, C, d, K, gr, gC, 0.0f, active, kMaxTraceDistance, rec, err);
    }
}

}  // namespace
}  // namespace vct

using namespace vct;

extern "C" int vct_cone_trace_backward(const vct_cone_tracing_desc* desc, const vct_cam_matrix* cam,
                                       const float* atlas4, int32_t R, const vct_shadow_map* shadow,
                                       const vct_directional_light_desc* light,
                                       const vct_directional_light_shadow_desc* light_shadow,
                                       const vct_surface_sample* samples, int64_t n, const float* grad_diffuse,
                                       const float* grad_specular, float* grad_atlas4, void* stream) {
    vct::NvtxRange nvtx_range("vct_cone_trace_backward");
    VCT_CHECK_ARG(atlas4 && grad_atlas4 && valid_resolution(R), "vct_cone_trace_backward: bad atlas / resolution");
    VCT_CHECK_ARG((((uintptr_t)atlas4 | (uintptr_t)grad_atlas4) & 15) == 0,
                  "vct_cone_trace_backward: atlases must be 16-byte aligned");
    VCT_CHECK_ARG(n >= 0, "vct_cone_trace_backward: negative sample count");
    if (n == 0) return VCT_OK;
    VCT_CHECK_ARG(samples && grad_diffuse && grad_specular, "vct_cone_trace_backward: null sample or gradient buffer");
    VCT_CHECK_ARG((((uintptr_t)samples | (uintptr_t)grad_diffuse | (uintptr_t)grad_specular) & 15) == 0,
                  "vct_cone_trace_backward: sample / gradient buffers must be 16-byte aligned");
    TraceParams P;
    int rc = fill_trace_params(P, desc, cam, shadow, light, light_shadow);
    if (rc != VCT_OK) return rc;
    cudaStream_t st = as_stream(stream);
    const int nc = desc->enable_32_cones ? 32 : 16;
    // grids of resident blocks (their warps take work by tickets): the record scratch holds one block per warp
    int dev = 0, sms = 0, occ_d = 0, occ_s = 0;
    VCT_CUDA_TRY(cudaGetDevice(&dev));
    VCT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    VCT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_d, k_cone_backward_diffuse, 128, 0));
    VCT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, k_cone_backward_specular, 128, 0));
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((n * nc + 127) / 128, (int64_t)sms * std::max(occ_d, 1)));
    const int64_t lblocks = std::max<int64_t>(1, std::min<int64_t>((n * kMaxConeGroup + 127) / 128, (int64_t)sms * std::max(occ_s, 1)));
    const size_t rec_bytes = (size_t)std::max(blocks, lblocks) * (128 / 32) * kRecWarpFloats * sizeof(float);
    int* err = nullptr;
    VCT_CUDA_TRY(cudaMallocAsync(&err, sizeof(int), st));
    VCT_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
    float* rec = nullptr;
    if (cudaMallocAsync(&rec, rec_bytes, st) != cudaSuccess) {
        cudaFreeAsync(err, st);
        return fail(VCT_E_CUDA, "vct_cone_trace_backward: record scratch allocation failed");
    }
    F4Atlas T{reinterpret_cast<const float4*>(atlas4), AtlasDims(R)};
    const MarchScale C = march_scale(P.d);
    ExactPlan plan;
    rc = exact_plan(samples, n, P.d, &plan, st);
    if (rc != VCT_OK) {
        cudaFreeAsync(rec, st);
        cudaFreeAsync(err, st);
        return rc;
    }
    float4* G = reinterpret_cast<float4*>(grad_atlas4);
    k_cone_backward_diffuse<<<(int)blocks, 128, 0, st>>>(P, C, T, samples, n, plan.order,
                                                          reinterpret_cast<const float4*>(grad_diffuse), G, rec, err,
                                                          plan.spec_count + 2);
    cudaError_t le = cudaGetLastError();
    if (le == cudaSuccess) {
        k_cone_backward_specular<<<(int)lblocks, 128, 0, st>>>(P, C, T, samples, plan.spec_list, plan.spec_count,
                                                               reinterpret_cast<const float4*>(grad_specular), G, rec,
                                                               err, plan.spec_count + 1);
        le = cudaGetLastError();
    }
    int h_err = 0;
    cudaError_t ce = cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t se = cudaStreamSynchronize(st);
    cudaFreeAsync(rec, st);
    cudaFreeAsync(err, st);
    exact_plan_free(&plan, st);
    if (le != cudaSuccess) return cuda_fail(le, "vct_cone_trace_backward kernels");
    if (ce != cudaSuccess) return cuda_fail(ce, "vct_cone_trace_backward readback");
    if (se != cudaSuccess) return cuda_fail(se, "vct_cone_trace_backward");
    if (h_err) return fail(VCT_E_OVERFLOW, "vct_cone_trace_backward: a cone marched more than 8192 steps");
    return VCT_OK;
}

// ------------------------------------------------------ inverse fitting ops
namespace vct {
namespace {

constexpr int kSqErrBlocks = 152 * 4;
constexpr int kSqErrThreads = 256;

// Squared error and its gradient; one double partial sum per block, each
// thread summing its grid-stride elements in index order, the block in a
// fixed tree order: the result does not depend on scheduling.
__global__ void __launch_bounds__(kSqErrThreads) k_sq_error(const float4* __restrict__ out,
                                                            const float4* __restrict__ target, int64_t n, float scale,
                                                            float4* __restrict__ grad, double* __restrict__ partial) {
    __shared__ double red[kSqErrThreads / 32];
    const float two_scale = 2.0f * scale;
    double acc = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 o = out[i], t = target[i];
        const float dx = o.x - t.x, dy = o.y - t.y, dz = o.z - t.z, dw = o.w - t.w;
        if (grad) grad[i] = make_float4(two_scale * dx, two_scale * dy, two_scale * dz, two_scale * dw);
        acc += ((double)dx * dx + (double)dy * dy) + ((double)dz * dz + (double)dw * dw);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kSqErrThreads / 32; ++w) s += red[w];
        partial[blockIdx.x] = s;
    }
}

__global__ void k_sq_error_fold(const double* __restrict__ partial, int blocks, double scale,
                                double* __restrict__ loss) {
    // one warp, lanes over the partial sums in turn, then the lanes in a fixed tree (608 adds in a row took 19 us)
    double s = 0.0;
    for (int b = threadIdx.x; b < blocks; b += 32) s += partial[b];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *loss = s * scale;
}

struct AdamArgs {
    float lr, b1, omb1, b2, omb2, eps, c1, c2;
    float lo[4], hi[4];
    int zero_grad;
};

// One rounding per operation (the file is compiled without contraction), so
// a float32 host restatement in the same order reproduces every bit.
__device__ __forceinline__ float adam1(float& p, float g, float& m, float& v, const AdamArgs& a, int c) {
    m = a.b1 * m + a.omb1 * g;
    v = a.b2 * v + (a.omb2 * g) * g;
    const float mh = m * a.c1, vh = v * a.c2;
    const float upd = (a.lr * mh) / (__fsqrt_rn(vh) + a.eps);
    p = fminf(fmaxf(p - upd, a.lo[c]), a.hi[c]);
    return p;
}

__global__ void __launch_bounds__(256) k_adam(float4* __restrict__ p, float4* __restrict__ g, float4* __restrict__ m,
                                              float4* __restrict__ v, int64_t n4, const AdamArgs a) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        float4 P = p[i], G = g[i], M = m[i], V = v[i];
        adam1(P.x, G.x, M.x, V.x, a, 0);
        adam1(P.y, G.y, M.y, V.y, a, 1);
        adam1(P.z, G.z, M.z, V.z, a, 2);
        adam1(P.w, G.w, M.w, V.w, a, 3);
        p[i] = P;
        m[i] = M;
        v[i] = V;
        if (a.zero_grad) g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

}  // namespace
}  // namespace vct

extern "C" int vct_sq_error(const float* out4, const float* target4, int64_t n, float scale, float* grad4,
                            double* loss, void* stream) {
    vct::NvtxRange nvtx_range("vct_sq_error");
    VCT_CHECK_ARG(n >= 0 && loss, "vct_sq_error: bad size or null loss");
    VCT_CHECK_ARG(n == 0 || (out4 && target4), "vct_sq_error: null output / target");
    VCT_CHECK_ARG((((uintptr_t)out4 | (uintptr_t)target4 | (uintptr_t)grad4) & 15) == 0,
                  "vct_sq_error: buffers must be 16-byte aligned");
    cudaStream_t st = as_stream(stream);
    double* partial = nullptr;
    VCT_CUDA_TRY(cudaMallocAsync(&partial, sizeof(double) * kSqErrBlocks, st));
    int64_t blocks = (n + kSqErrThreads - 1) / kSqErrThreads;
    blocks = blocks < 1 ? 1 : (blocks > kSqErrBlocks ? kSqErrBlocks : blocks);
    k_sq_error<<<(int)blocks, kSqErrThreads, 0, st>>>(reinterpret_cast<const float4*>(out4),
                                                      reinterpret_cast<const float4*>(target4), n, scale,
                                                      reinterpret_cast<float4*>(grad4), partial);
    cudaError_t le = cudaGetLastError();
    if (le == cudaSuccess) {
        k_sq_error_fold<<<1, 32, 0, st>>>(partial, (int)blocks, (double)scale, loss);
        le = cudaGetLastError();
    }
    cudaFreeAsync(partial, st);
    if (le != cudaSuccess) return cuda_fail(le, "k_sq_error");
    return VCT_OK;
}

extern "C" int vct_adam_step(float* param, float* grad, float* m, float* v, int64_t n, const vct_adam_desc* desc,
                             void* stream) {
    vct::NvtxRange nvtx_range("vct_adam_step");
    VCT_CHECK_ARG(desc && n >= 0 && (n & 3) == 0, "vct_adam_step: null descriptor or n not a multiple of 4");
    VCT_CHECK_ARG(desc->step >= 1, "vct_adam_step: step counts from 1");
    VCT_CHECK_ARG(desc->beta1 >= 0.0f && desc->beta1 < 1.0f && desc->beta2 >= 0.0f && desc->beta2 < 1.0f &&
                      desc->eps > 0.0f,
                  "vct_adam_step: betas must lie in [0, 1) and eps be positive");
    if (n == 0) return VCT_OK;
    VCT_CHECK_ARG(param && grad && m && v, "vct_adam_step: null buffer");
    VCT_CHECK_ARG((((uintptr_t)param | (uintptr_t)grad | (uintptr_t)m | (uintptr_t)v) & 15) == 0,
                  "vct_adam_step: buffers must be 16-byte aligned");
    AdamArgs a;
    a.lr = desc->lr;
    a.b1 = desc->beta1;
    a.omb1 = 1.0f - desc->beta1;
    a.b2 = desc->beta2;
    a.omb2 = 1.0f - desc->beta2;
    a.eps = desc->eps;
    a.c1 = (float)(1.0 / (1.0 - pow((double)desc->beta1, (double)desc->step)));
    a.c2 = (float)(1.0 / (1.0 - pow((double)desc->beta2, (double)desc->step)));
    for (int c = 0; c < 3; ++c) {
        a.lo[c] = desc->rgb_lo;
        a.hi[c] = desc->rgb_hi;
    }
    a.lo[3] = desc->alpha_lo;
    a.hi[3] = desc->alpha_hi;
    a.zero_grad = desc->zero_grad;
    cudaStream_t st = as_stream(stream);
    const int64_t n4 = n / 4;
    int64_t blocks = (n4 + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    k_adam<<<(int)blocks, 256, 0, st>>>(reinterpret_cast<float4*>(param), reinterpret_cast<float4*>(grad),
                                        reinterpret_cast<float4*>(m), reinterpret_cast<float4*>(v), n4, a);
    VCT_LAUNCH_CHECK();
    return VCT_OK;
}
