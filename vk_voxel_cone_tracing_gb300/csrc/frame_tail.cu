// frame_tail.cu -- the streaming passes of a deterministic frame over bitmaps
// of its voxels: the opacity atlas written from the voxelised bits, and the due
// radiance levels' copy-alpha and mips.
//
// A frame's clipmap is mostly empty (3 % of a hall's voxels at R = 256 hold
// anything), and the passes' cost was reading that: the cleared atlas, the
// stale radiance under it, the children of empty blocks.  With one bit per
// voxel and level -- voxelised (FrameBits::opaque), lit by the injection
// (lit), nonzero after its mip (nonzero) -- the empty texels are written
// without being read.  What remains is the stores: every interior texel of a
// due level goes to the atlas and to the texture.
// Measured, R = 256 hall frame: k_opacity_fill 0.35 ms (7.0 TB/s) where a clear,
// scattered six-face stores and their write-backs were; k_radiance_fill 1.16 ms
// with the texture (4.2 TB/s), 0.72 ms without (3.4), and the five k_radiance_mip
// 0.50 ms, where copy-alpha and the fused copy-alpha + mip passes took 0.37 +
// 2.24 ms (they waited for their loads: DRAM 42 % busy).  The frame 8.59 ->
// 7.72 ms.  Texture stores of 16 bytes cost 0.44 ms a frame, the 4-byte ones
// before 0.95 ms.
// Built with -fmad=false; the mips' arithmetic is written with explicit
// rounding, as in clipmap_passes.cu.
#include "common.cuh"
#include "mip_pairs.cuh"

namespace vct {

namespace {

__device__ __forceinline__ uint32_t voxel_bit(const uint32_t* __restrict__ bits, int64_t i) {
    return (__ldg(bits + (i >> 5)) >> ((uint32_t)i & 31u)) & 1u;
}

// Four neighbouring texels of an atlas row, the g-th four of a pair of faces:
// a face is R + 2 texels wide, 2 modulo 4, so two faces hold a whole number of
// fours and the three face pairs of a row repeat the pattern -- and a voxel's
// six faces share its bits, so a thread works a four out once and writes it
// three times.  xf0 is the first texel's place in its face (texel xf holds
// voxel xf - 1, 0 and R + 1 are border); the four at xf0 == R runs from the
// first face's end into the second.
struct Four {
    int x0, xf0;
    uint32_t inner;  // interior texels
};

__device__ __forceinline__ Four four_of(int g, const AtlasDims& A) {
    const int x0 = 4 * g, xf0 = x0 >= A.rb ? x0 - A.rb : x0;
    return Four{x0, xf0, xf0 == 0 ? 14u : (xf0 == A.R ? 9u : (xf0 + 3 > A.R ? 7u : 15u))};
}

// Its texels' bits, in the row whose first voxel is bit b0.
__device__ __forceinline__ uint32_t four_bits(const uint32_t* __restrict__ bits, int64_t b0, const Four& f,
                                              const AtlasDims& A) {
    if (f.xf0 == A.R) return voxel_bit(bits, b0 + A.R - 1) | (voxel_bit(bits, b0) << 3);
    const int64_t i = b0 + max(f.xf0 - 1, 0);
    const uint32_t sh = (uint32_t)i & 31u;
    const uint32_t lo = __ldg(bits + (i >> 5)), hi = sh > 28u ? __ldg(bits + (i >> 5) + 1) : 0u;
    const uint32_t r = __funnelshift_r(lo, hi, sh);
    return (f.xf0 == 0 ? r << 1 : r) & f.inner;
}

// Work item t of a block of row pairs: lane pairs take a four of the pair's
// two rows (in the texture's block-linear layout a 32-byte sector holds 16
// bytes of each), then the next four.  rows 2 * pair and 2 * pair + 1.
struct RowFour {
    uint32_t pair;
    int row, g;
};

__device__ __forceinline__ RowFour row_four(uint32_t t, uint32_t fours) {
    const uint32_t u = t >> 1, pair = u / fours;
    return RowFour{pair, (int)(2u * pair + (t & 1u)), (int)(u - pair * fours)};
}

// Four texels of a row: one 16-byte (4-byte) store where the atlas is aligned.
__device__ __forceinline__ void store4(uint32_t* p, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, bool vec) {
    if (vec) {
        *reinterpret_cast<uint4*>(p) = make_uint4(v0, v1, v2, v3);
    } else {
        p[0] = v0;
        p[1] = v1;
        p[2] = v2;
        p[3] = v3;
    }
}
__device__ __forceinline__ void store4(uint8_t* p, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, bool vec) {
    const uint32_t w = (v0 & 0xffu) | ((v1 & 0xffu) << 8) | ((v2 & 0xffu) << 16) | (v3 << 24);
    if (vec) {
        *reinterpret_cast<uint32_t*>(p) = w;
    } else {
        for (int k = 0; k < 4; ++k) p[k] = (uint8_t)(w >> (8 * k));
    }
}

// Every texel of the opacity atlas: all ones in a voxelised voxel's six faces,
// zero elsewhere and in the borders (the clear and the voxeliser's stores in
// one pass).  blockIdx.y walks the z slices.
template <class T>
__global__ void __launch_bounds__(256) k_opacity_fill(T* __restrict__ atlas, const uint32_t* __restrict__ opaque,
                                                      AtlasDims A, bool vec) {
    const uint32_t fours = (uint32_t)A.rb / 2u, items = (uint32_t)A.H * fours;
    for (int z = blockIdx.y; z < A.D; z += gridDim.y) {
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < items; t += gridDim.x * blockDim.x) {
            const RowFour u = row_four(t, fours);
            const int level = u.row / A.rb, yl = u.row - level * A.rb;
            const Four f = four_of(u.g, A);
            uint32_t m = 0u;
            if (z >= 1 && z <= A.R && yl >= 1 && yl <= A.R)
                m = four_bits(opaque, (((int64_t)level * A.R + (z - 1)) * A.R + (yl - 1)) * A.R, f, A);
            T* p = atlas + A.index(f.x0, u.row, z);
#pragma unroll
            for (int k = 0; k < 3; ++k)
                store4(p + 2 * A.rb * k, (m & 1u) ? 0xffffffffu : 0u, (m & 2u) ? 0xffffffffu : 0u,
                       (m & 4u) ? 0xffffffffu : 0u, (m & 8u) ? 0xffffffffu : 0u, vec);
        }
    }
}

// The interior of the due radiance levels after copy-alpha: rgb as the
// injection left it where the voxel is lit and zero elsewhere (the level's
// clear), alpha from the opacity -- from the bits (BITS: the voxelised value,
// which is the final alpha outside the mips' target blocks; the mips take their
// own from the opacity atlas) or from the opacity atlas (the toroidal update).
// All due levels in one launch: none of it depends on the mips, which then
// write their blocks over it (leaving the blocks out broke up the rows: 0.74
// against 0.47 ms for the stores of a R = 256 frame without the texture).
struct FillLevels {
    int n;
    int level[VCT_CLIP_LEVEL_COUNT];
};

template <bool BITS>
__global__ void __launch_bounds__(256) k_radiance_fill(uint32_t* __restrict__ rad, const uint32_t* __restrict__ opa,
                                                       const FrameBits B, AtlasDims A, const FillLevels F,
                                                       cudaSurfaceObject_t mirror, bool vec) {
    const uint32_t fours = (uint32_t)A.rb / 2u, items = (uint32_t)A.rb * fours;
    // blockIdx.y walks the (due level, z) slices
    for (int s = blockIdx.y; s < F.n * A.R; s += gridDim.y) {
        const int li = s / A.R, z = s - li * A.R, level = F.level[li];
        for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < items; t += gridDim.x * blockDim.x) {
            const RowFour u = row_four(t, fours);
            if (u.row < 1 || u.row > A.R) continue;  // border rows
            const Four f = four_of(u.g, A);
            const int64_t b0 = (((int64_t)level * A.R + z) * A.R + (u.row - 1)) * A.R;
            const uint32_t lit = four_bits(B.lit, b0, f, A);
            const uint32_t o = BITS ? four_bits(B.opaque, b0, f, A) : 0u;
            const int y = level * A.rb + u.row;
            const int64_t i0 = A.index(f.x0, y, z + 1);
            const int step = 2 * A.rb;  // to the next pair of faces
            // every load before the first store (the compiler cannot tell the atlas's loads from its stores)
            uint32_t v[3][4];
#pragma unroll
            for (int pair = 0; pair < 3; ++pair) {
                if (BITS) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[pair][k] = ((o >> k) & 1u) ? 0xff000000u : 0u;
                } else if (vec) {
                    const uint4 a = __ldg(reinterpret_cast<const uint4*>(opa + i0 + step * pair));
                    v[pair][0] = a.x & 0xff000000u;
                    v[pair][1] = a.y & 0xff000000u;
                    v[pair][2] = a.z & 0xff000000u;
                    v[pair][3] = a.w & 0xff000000u;
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[pair][k] = __ldg(opa + i0 + step * pair + k) & 0xff000000u;
                }
            }
            if (lit) {
                uint32_t c[3][4];
#pragma unroll
                for (int pair = 0; pair < 3; ++pair)
#pragma unroll
                    for (int k = 0; k < 4; ++k) c[pair][k] = ((lit >> k) & 1u) ? rad[i0 + step * pair + k] : 0u;
#pragma unroll
                for (int pair = 0; pair < 3; ++pair)
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[pair][k] |= c[pair][k] & 0x00ffffffu;
            }
#pragma unroll
            for (int pair = 0; pair < 3; ++pair) {
                const int64_t i = i0 + step * pair;
                const int x = f.x0 + step * pair;
                if (f.inner == 15u) {
                    store4(rad + i, v[pair][0], v[pair][1], v[pair][2], v[pair][3], vec);
                    if (mirror)
                        surf3Dwrite(make_uint4(v[pair][0], v[pair][1], v[pair][2], v[pair][3]), mirror, x * 4, y, z + 1);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if ((f.inner >> k) & 1u) {
                            rad[i + k] = v[pair][k];
                            if (mirror) surf3Dwrite(v[pair][k], mirror, (x + k) * 4, y, z + 1);
                        }
                }
            }
        }
    }
}

__device__ __forceinline__ uint32_t opa_alpha(const uint32_t* __restrict__ opa, int64_t i) {
    return __ldg(opa + i) & 0xff000000u;
}
__device__ __forceinline__ uint32_t opa_alpha(const uint8_t* __restrict__ opa, int64_t i) {
    return (uint32_t)__ldg(opa + i) << 24;
}

// calculateImageCoords' wrap of the downsample shaders.
__device__ __forceinline__ int wrap_r(int p, int R) { return (p + R * (abs(p / R) + 1)) & (R - 1); }

// The target block of one level l >= 1 (radianceDownSample.comp after
// copyAlphaImage.comp): the (R/2)^3 voxels of the previous region's corner / 2
// on, toroidally, each the 2x2x2 composite of level l - 1 blended with its own
// copy-alpha value.  With SKIP (the bits cover level l - 1), a voxel whose
// eight children hold nothing on any face loads none of their 48 texels.
template <class OT, bool SKIP>
__global__ void __launch_bounds__(128, 8) k_radiance_mip(uint32_t* __restrict__ rad, const uint32_t* __restrict__ prev,
                                                         const OT* __restrict__ opa, const FrameBits B, AtlasDims A,
                                                         int3 pmin, int level, int band, int lgh,
                                                         cudaSurfaceObject_t mirror) {
    const int half = A.R >> 1;
    const int pm[3] = {pmin.x, pmin.y, pmin.z};
    const uint32_t nh = 1u << (3 * lgh), mh = (1u << lgh) - 1u;
    const float inv = 1.0f / __fadd_rn((float)band, 1.0f);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nh; t += gridDim.x * blockDim.x) {
        const int g[3] = {(int)(t & mh), (int)((t >> lgh) & mh), (int)(t >> (2 * lgh))};
        int cur[3], w[3], c[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            cur[a] = (pm[a] >> 1) + g[a];
            w[a] = wrap_r(cur[a], A.R);
            c[a] = wrap_r(cur[a] << 1, A.R);
        }
        // lerpFactor (opacityDownSample.comp:55-64)
        float dist[3];
        bool any_ge = false;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float center = __fadd_rn((float)(pm[a] >> 1), (float)(half >> 1));
            dist[a] = __fsub_rn(fabsf(__fsub_rn(__fadd_rn((float)cur[a], 0.5f), center)), 0.5f);
            any_ge |= dist[a] >= (float)((half >> 1) - band);
        }
        float lerp = 0.0f;
        if (any_ge) {
            lerp = __fadd_rn(__fsub_rn(fmaxf(dist[0], fmaxf(dist[1], dist[2])), (float)((half >> 1) - band)), 1.0f);
            lerp = __fmul_rn(lerp, inv);
        }
        uint32_t children = 1u;
        if (SKIP) {
            children = 0u;
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // c[0] is even: a row's two children share a word
                const int64_t i = (((int64_t)(level - 1) * A.R + c[2] + (k >> 1)) * A.R + c[1] + (k & 1)) * A.R + c[0];
                children |= ((__ldg(B.opaque + (i >> 5)) | __ldg(B.lit + (i >> 5)) | B.nonzero[i >> 5]) >> (i & 31)) & 3u;
            }
        }
        const int64_t bit = (((int64_t)level * A.R + w[2]) * A.R + w[1]) * A.R + w[0];
        const bool on = voxel_bit(B.lit, bit);  // rgb is zero elsewhere
        const int wy = w[1] + 1 + A.rb * level, wz = w[2] + 1;
        const int64_t w0 = A.index(w[0] + 1, wy, wz);
        uint32_t own6[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) own6[f] = opa_alpha(opa, w0 + A.rb * f);
        if (on) {
#pragma unroll
            for (int f = 0; f < 6; ++f) own6[f] |= rad[w0 + A.rb * f] & 0x00ffffffu;
        }
        const int64_t c0 = A.index(c[0] + 1, c[1] + 1 + A.rb * (level - 1), c[2] + 1);
        const int64_t dy = A.W, dz = (int64_t)A.W * A.H;
        uint32_t any = 0u;
#pragma unroll
        for (int f0 = 0; f0 < 6; f0 += 2) {  // two faces' children in flight together
            uint32_t raw2[2][8];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    raw2[h][i] = children ? __ldg(prev + c0 + A.rb * (f0 + h) + (i & 1) + ((i >> 1) & 1) * dy +
                                                  ((i >> 2) & 1) * dz)
                                          : 0u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int f = f0 + h;
                const uint32_t* raw = raw2[h];
                uint32_t out = 0;
                if (children | own6[f]) {
                    float sc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t r0 = raw[ds_pair(f, k, 0)], r1 = raw[ds_pair(f, k, 1)];
                        const float tt = __fsub_rn(1.0f, unorm8_load(r0, 3));
#pragma unroll
                        for (int ch = 0; ch < 4; ++ch) {
                            const float a0 = unorm8_load(r0, ch);
                            const float b = __fmul_rn(tt, unorm8_load(r1, ch));
                            sc[ch] = (k == 0) ? __fadd_rn(a0, b) : __fadd_rn(__fadd_rn(sc[ch], a0), b);
                        }
                    }
#pragma unroll
                    for (int ch = 0; ch < 4; ++ch) {
                        const float res = __fmul_rn(sc[ch], 0.25f);
                        out |= unorm8_store(mix_rn(res, unorm8_load(own6[f], ch), lerp)) << (8 * ch);
                    }
                }
                any |= out;
                rad[w0 + A.rb * f] = out;
                if (mirror) surf3Dwrite(out, mirror, (w[0] + 1 + A.rb * f) * 4, wy, wz);
            }
        }
        if (SKIP && any) atomicOr(B.nonzero + (bit >> 5), 1u << (bit & 31));
    }
}

int grid_for(int64_t threads, int block) {
    int64_t g = (threads + block - 1) / block;
    return (int)(g < 1 ? 1 : (g > 152 * 64 ? 152 * 64 : g));
}

// Blocks of 256 over `items` of each of `slices` slices.
dim3 slice_grid(int64_t items, int slices) {
    return dim3((unsigned)((items + 255) / 256), (unsigned)(slices < 65535 ? slices : 65535));
}

}  // namespace

size_t frame_bitmap_bytes(int R) { return ((6 * (size_t)R * R * R / 8 + 8) + 255) & ~(size_t)255; }

int frame_opacity_fill(void* atlas, bool r8, int R, const uint32_t* opaque, cudaStream_t st) {
    AtlasDims A(R);
    const bool vec = ((uintptr_t)atlas & (r8 ? 3 : 15)) == 0;
    const dim3 grid = slice_grid((int64_t)A.H * (A.rb / 2), A.D);
    if (r8) k_opacity_fill<<<grid, 256, 0, st>>>(static_cast<uint8_t*>(atlas), opaque, A, vec);
    else k_opacity_fill<<<grid, 256, 0, st>>>(static_cast<uint32_t*>(atlas), opaque, A, vec);
    VCT_LAUNCH_CHECK();
    return VCT_OK;
}

int frame_radiance_fill(uint32_t* radiance, const uint32_t* opacity, const FrameBits& B, int R, uint32_t due,
                        cudaSurfaceObject_t mirror, cudaStream_t st) {
    AtlasDims A(R);
    FillLevels F;
    F.n = 0;
    for (int l = 0; l < VCT_CLIP_LEVEL_COUNT; ++l) {
        if (!((due >> l) & 1u)) continue;
        F.level[F.n++] = l;
    }
    if (F.n == 0) return VCT_OK;
    const dim3 grid = slice_grid((int64_t)A.rb * (A.rb / 2), F.n * R);
    if (B.opaque) {
        const bool vec = ((uintptr_t)radiance & 15) == 0;
        k_radiance_fill<true><<<grid, 256, 0, st>>>(radiance, nullptr, B, A, F, mirror, vec);
    } else {
        const bool vec = (((uintptr_t)radiance | (uintptr_t)opacity) & 15) == 0;
        k_radiance_fill<false><<<grid, 256, 0, st>>>(radiance, opacity, B, A, F, mirror, vec);
    }
    VCT_LAUNCH_CHECK();
    return VCT_OK;
}

int frame_radiance_mips(uint32_t* radiance, const void* opacity, bool r8, const FrameBits& B,
                        const vct_clipmap_region regions[6], int R, uint32_t due, cudaSurfaceObject_t mirror,
                        cudaStream_t st) {
    AtlasDims A(R);
    const int lgh = 30 - __builtin_clz((unsigned)R), grid = grid_for((int64_t)1 << (3 * lgh), 128);
    const uint32_t* o32 = static_cast<const uint32_t*>(opacity);
    const uint8_t* o8 = static_cast<const uint8_t*>(opacity);
    for (int l = 1; l < VCT_CLIP_LEVEL_COUNT; ++l) {
        if (!((due >> l) & 1u)) continue;
        const int3 pm = make_int3(regions[l - 1].min_corner[0], regions[l - 1].min_corner[1], regions[l - 1].min_corner[2]);
        constexpr int band = VCT_DOWNSAMPLE_REGION_SIZE;
        if (r8) k_radiance_mip<uint8_t, true><<<grid, 128, 0, st>>>(radiance, radiance, o8, B, A, pm, l, band, lgh, mirror);
        else if (B.opaque)
            k_radiance_mip<uint32_t, true><<<grid, 128, 0, st>>>(radiance, radiance, o32, B, A, pm, l, band, lgh, mirror);
        else
            k_radiance_mip<uint32_t, false><<<grid, 128, 0, st>>>(radiance, radiance, o32, B, A, pm, l, band, lgh, mirror);
        VCT_LAUNCH_CHECK();
    }
    return VCT_OK;
}

}  // namespace vct
