// svo.cu -- sparse voxel octree build over a uint2 node pool
// (OctreeBuilder::cmdBuild, VFS/RenderPass/Octree/OctreeBuilder.cpp:205-345).
//
// Node: x = MSB flag | child block index (8 children), y = RGBA8 colour.
// VCT_SVO_ATOMIC runs the reference's way, level by level: init the window,
// flag (every fragment steps down and sets its node's MSB; atomicOr,
// order-free), allocate a child block for every flagged node (racy atomicAdd),
// then the leaf colours by CAS loops.
// VCT_SVO_DETERMINISTIC gives the canonical pool -- child blocks in
// breadth-first order, leaf colours folded in fragment order -- from one sort:
// a fragment's leaf is its path (three bits a level), breadth-first order
// within a depth is path order, and the distinct prefixes of the sorted paths
// are the pool's nodes.  Consecutive fragments mostly share their leaf (the
// samples of a pixel), so the sort runs over runs of them, and the fold reads
// each run's fragments where they lie.  What bounds it is the one pass over
// the fragments that finds the runs and the fold's chain.  Against a flag pass
// over the fragments per level and a sort of every fragment by its leaf:
// 58.4 M fragments at L = 9, fragments + build + trace 11.04 -> 7.13 ms (two
// host readbacks in the build instead of eight); the room at L = 7, 2.01 ->
// 1.43 ms.
// Mips (octreeNodeMipmapWrite.comp) are computed per node: the shader
// writes, for each power-of-two target level t <= 2^(L-1), the flagged nodes
// at resolution t; a per-node pass over those windows gives the same values
// without the shader's per-fragment redundancy.
// Compiled with -fmad=false.
#include <cstring>

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "common.cuh"

namespace vct {

__device__ inline uint3 frag_pos(uint2 f) {
    return make_uint3((f.x & 0xfffu) >> 1, ((f.x >> 12) & 0xfffu) >> 1,
                      (((f.x >> 24) & 0xffu) | ((f.y >> 20) & 0xf00u)) >> 1);
}

__global__ void k_init(uint2* pool, uint64_t begin, uint64_t num) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < num; i += (uint64_t)gridDim.x * blockDim.x)
        pool[begin + i] = make_uint2(0u, 0u);
}

// Child slot a fragment takes at descent step k (resolution 2^(L-1-k)).  The
// node shaders descend from the root subtracting the resolution where
// pos >= resolution; for the halved position p <= 2^(L-1) that is: step 0
// takes the upper child only when p == 2^(L-1) (and leaves p = 0), later
// steps take bit (L-1-k) of the remaining p.  So the node a fragment reaches
// at depth i is the depth-(i-1) node's child block plus slot(i-1): one step
// per level from a per-fragment cursor instead of a descent from the root.
__device__ inline uint32_t slot_at(uint3 p, int L, int k) {
    const uint32_t top = 1u << (L - 1);
    if (k == 0) return (p.z >= top ? 1u : 0u) | (p.x >= top ? 2u : 0u) | (p.y >= top ? 4u : 0u);
    const uint3 q = make_uint3(p.x >= top ? p.x - top : p.x, p.y >= top ? p.y - top : p.y, p.z >= top ? p.z - top : p.z);
    const int b = L - 1 - k;
    return ((q.z >> b) & 1u) | (((q.x >> b) & 1u) << 1) | (((q.y >> b) & 1u) << 2);
}

// octreeNodeFlag.comp for level i through the cursor; the flag is written
// only if not yet set (the shader's racy |= is idempotent either way).
__global__ void k_flag_level(uint2* pool, const uint2* __restrict__ frags, int64_t F, int L, int level,
                             uint32_t* __restrict__ cursor) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < F; i += (int64_t)gridDim.x * blockDim.x) {
        const uint3 p = frag_pos(__ldg(frags + i));
        const uint32_t slot = slot_at(p, L, level - 1);
        const uint32_t node = level == 1 ? slot : (pool[cursor[i]].x & 0x7fffffffu) + slot;
        cursor[i] = node;
        if (!(pool[node].x & 0x80000000u)) atomicOr(&pool[node].x, 0x80000000u);
    }
}

// octreeNodeAlloc.comp with a warp-aggregated counter increment (one atomicAdd per warp).
__global__ void k_alloc_atomic(uint2* pool, uint64_t begin, uint64_t num, unsigned int* counter) {
    const int lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); base < num; base += stride) {
        const uint64_t i = base + lane;
        const bool flagged = i < num && (pool[begin + i].x & 0x80000000u);
        const unsigned m = __ballot_sync(0xffffffffu, flagged);
        unsigned wbase = 0;
        if (lane == 0 && m) wbase = atomicAdd(counter, (unsigned)__popc(m));
        wbase = __shfl_sync(0xffffffffu, wbase, 0);
        if (flagged) {
            const unsigned c = wbase + __popc(m & ((1u << lane) - 1u));
            pool[begin + i] = make_uint2(((c + 1u) << 3) | 0x80000000u, 0u);
        }
    }
}

__device__ inline uint32_t conv_u8x4(float x, float y, float z, float w) {
    return (((uint32_t)w & 0xffu) << 24) | (((uint32_t)z & 0xffu) << 16) | (((uint32_t)y & 0xffu) << 8) |
           ((uint32_t)x & 0xffu);
}

__device__ inline uint32_t avg_fold(uint32_t cur, uint32_t v) {
    const float vr = (float)(v & 0xffu), vg = (float)((v >> 8) & 0xffu), vb = (float)((v >> 16) & 0xffu),
                va = (float)(v >> 24);
    if (cur == 0u) return conv_u8x4(vr, vg, vb, va);
    float rx = (float)(cur & 0xffu), ry = (float)((cur >> 8) & 0xffu), rz = (float)((cur >> 16) & 0xffu),
          rw = (float)(cur >> 24);
    rx = rx * rw;
    ry = ry * rw;
    rz = rz * rw;
    float cx = rx + vr, cy = ry + vg, cz = rz + vb, cw = rw + va;
    cx = cx / cw;
    cy = cy / cw;
    cz = cz / cw;
    return conv_u8x4(cx, cy, cz, cw);
}

// ------------------------------------------------ deterministic build
// A fragment's path from the root: its child slot at each of the L descent
// steps, the first step in the highest bits.  Step 0 compares the halved
// position with 2^(L-1) (slot_at), the others take its bits, so below the
// first three bits the path is the Morton interleave of L - 1 <= 10 bits.
__device__ __forceinline__ uint32_t spread_bits(uint32_t v) {
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    return (v | (v << 2)) & 0x09249249u;
}

template <class Key>
__device__ __forceinline__ Key path_key(uint2 f, int L) {
    const uint3 p = frag_pos(f);
    const uint32_t top = 1u << (L - 1), m = top - 1u;
    const uint3 q = make_uint3((p.x >= top ? p.x - top : p.x) & m, (p.y >= top ? p.y - top : p.y) & m,
                               (p.z >= top ? p.z - top : p.z) & m);
    const uint32_t low = spread_bits(q.z) | (spread_bits(q.x) << 1) | (spread_bits(q.y) << 2);
    return ((Key)slot_at(p, L, 0) << (3 * (L - 1))) | (Key)low;
}

// Starts of the runs of fragments with the same halved position over [0, n],
// n itself closing the last run.
struct FragRunHead {
    const uint2* frags;
    uint32_t n;
    __device__ bool operator()(uint32_t i) const {
        if (i == 0u || i == n) return true;
        const uint2 a = __ldg(frags + i - 1), b = __ldg(frags + i);
        return (((a.x ^ b.x) & 0xfeffeffeu) | ((a.y ^ b.y) >> 28)) != 0u;
    }
};

template <class Key>
__global__ void k_run_keys(const uint2* __restrict__ frags, const uint32_t* __restrict__ starts, uint32_t runs, int L,
                           Key* __restrict__ keys, uint32_t* __restrict__ vals) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < runs; i += gridDim.x * blockDim.x) {
        keys[i] = path_key<Key>(__ldg(frags + starts[i]), L);
        vals[i] = i;
    }
}

// Starts of the leaves' groups of runs in the sorted keys over [0, n].
template <class Key>
struct LeafHead {
    const Key* keys;
    uint32_t n;
    __device__ bool operator()(uint32_t i) const { return i == 0u || i == n || keys[i - 1] != keys[i]; }
};

// Leaf l's path shares its first `shared` slots with its predecessor's, so it
// is the first leaf below its node at every depth d > shared.
template <class Key>
__device__ __forceinline__ int shared_slots(const Key* __restrict__ keys, const uint32_t* __restrict__ heads,
                                            uint32_t l, int L) {
    if (l == 0u) return 0;
    const unsigned long long x = (unsigned long long)(keys[heads[l]] ^ keys[heads[l] - 1u]);
    return (3 * L - 1 - (63 - __clzll((long long)x))) / 3;
}

constexpr int kTreeBlock = 256;  // leaves of one chunk

// New nodes per depth 1 .. L-1 and chunk of leaves: counts[(d - 1) * stride + chunk].
template <class Key>
__global__ void __launch_bounds__(kTreeBlock) k_tree_count(const Key* __restrict__ keys,
                                                           const uint32_t* __restrict__ heads,
                                                           const uint32_t* __restrict__ nheads, int L,
                                                           uint32_t* __restrict__ counts, uint32_t stride) {
    __shared__ uint32_t s_count[12];
    const uint32_t leaves = *nheads - 1u, chunks = (leaves + kTreeBlock - 1u) / kTreeBlock;
    for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        if (threadIdx.x < 12) s_count[threadIdx.x] = 0u;
        __syncthreads();
        const uint32_t l = c * kTreeBlock + threadIdx.x;
        const int shared = l < leaves ? shared_slots(keys, heads, l, L) : L;
        for (int d = 1; d < L; ++d) {
            const unsigned b = __ballot_sync(0xffffffffu, shared < d);
            if ((threadIdx.x & 31) == 0 && b) atomicAdd(&s_count[d], (uint32_t)__popc(b));
        }
        __syncthreads();
        if (threadIdx.x >= 1 && (int)threadIdx.x < L) counts[(threadIdx.x - 1) * stride + c] = s_count[threadIdx.x];
        __syncthreads();
    }
}

// Exclusive scan of each depth's chunk counts in place, one warp a depth;
// totals[d] (1 <= d < L) the nodes of depth d with children, totals[0] the leaves.
__global__ void k_tree_scan(uint32_t* __restrict__ counts, uint32_t stride, const uint32_t* __restrict__ nheads, int L,
                            uint32_t* __restrict__ totals) {
    const int d = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t leaves = *nheads - 1u, chunks = (leaves + kTreeBlock - 1u) / kTreeBlock;
    if (d == 0) {
        if (lane == 0) totals[0] = leaves;
        return;
    }
    uint32_t* c = counts + (size_t)(d - 1) * stride;
    uint32_t sum = 0;
    for (uint32_t i0 = 0; i0 < chunks; i0 += 32u) {
        const uint32_t v = i0 + lane < chunks ? c[i0 + lane] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (i0 + lane < chunks) c[i0 + lane] = sum + incl - v;
        sum += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) totals[d] = sum;
}

// One step of the leaf average for alpha sum cw = rw + va > 0.  Every operand
// is an integer below 2^16 and cw below 2^9, so the truncated quotient is the
// integer one, and (a + 1/2) / cw is at least 1 / (2 cw) from any integer:
// far more than an approximate reciprocal's error.
__device__ __forceinline__ uint32_t avg_fold_int(uint32_t cur, uint32_t v) {
    const float rw = (float)(cur >> 24), cw = rw + (float)(v >> 24);
    if (cur == 0u || cw == 0.0f) return avg_fold(cur, v);
    const float r = __fdividef(1.0f, cw);
    const uint32_t x = (uint32_t)(((float)(cur & 0xffu) * rw + ((float)(v & 0xffu) + 0.5f)) * r);
    const uint32_t y = (uint32_t)(((float)((cur >> 8) & 0xffu) * rw + ((float)((v >> 8) & 0xffu) + 0.5f)) * r);
    const uint32_t z = (uint32_t)(((float)((cur >> 16) & 0xffu) * rw + ((float)((v >> 16) & 0xffu) + 0.5f)) * r);
    return (((uint32_t)cw & 0xffu) << 24) | ((z & 0xffu) << 16) | ((y & 0xffu) << 8) | (x & 0xffu);
}

// The same steps on a cell whose bytes stay floats: a byte of the fragment is
// the low bits of 2^23 + byte, a floor is a sum rounded down at 2^23, so no
// step converts.  A step to or from alpha 0 (the first, the one after the
// 256-count wraps, a fragment of alpha 0, whose quotient may pass 255) goes by
// the words.  The conversions bound the emission of the terrain's 57 M
// fragments: 656 -> 534 us.
struct LeafCell {
    float r, g, b, a;
};
__device__ __forceinline__ float byte_float(uint32_t v, int k) {
    return __uint_as_float(__byte_perm(v, 0x4b000000u, 0x7440 + k)) - 8388608.0f;
}
__device__ __forceinline__ LeafCell leaf_cell(uint32_t v) {
    return LeafCell{byte_float(v, 0), byte_float(v, 1), byte_float(v, 2), byte_float(v, 3)};
}
__device__ __forceinline__ uint32_t leaf_word(const LeafCell& c) {
    return ((uint32_t)c.a << 24) | ((uint32_t)c.b << 16) | ((uint32_t)c.g << 8) | (uint32_t)c.r;
}
__device__ __forceinline__ void leaf_step(LeafCell& c, uint32_t v) {
    if (c.a == 0.0f || (v >> 24) == 0u) {
        c = leaf_cell(avg_fold_int(leaf_word(c), v));
        return;
    }
    const LeafCell f = leaf_cell(v);
    const float cw = c.a + f.a, inv = __fdividef(1.0f, cw);
    c.r = __fadd_rd((c.r * c.a + (f.r + 0.5f)) * inv, 8388608.0f) - 8388608.0f;
    c.g = __fadd_rd((c.g * c.a + (f.g + 0.5f)) * inv, 8388608.0f) - 8388608.0f;
    c.b = __fadd_rd((c.b * c.a + (f.b + 0.5f)) * inv, 8388608.0f) - 8388608.0f;
    c.a = cw >= 256.0f ? cw - 256.0f : cw;
}

// A fragment the light test discarded adds (0, 0, 0, 0): that leaves a cell
// with alpha as it is and empties one without (0 / 0 stores 0).
__device__ __forceinline__ uint32_t avg_fold_zero(uint32_t cur) { return (cur >> 24) ? cur : 0u; }

constexpr uint32_t kLongLeaf = 4096;  // fragments from which a warp folds a leaf together

// A long leaf on the calling warp, 32 fragments loaded at a time: only the
// fragments with a colour cost a step (a scene's discarded fragments all lie
// at position 0, in one leaf).
__device__ inline uint32_t fold_long_leaf(const uint2* __restrict__ frags, const uint32_t* __restrict__ starts,
                                          const uint32_t* __restrict__ order, uint32_t h0, uint32_t h1) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t cell = 0u;
    for (uint32_t h = h0; h < h1; ++h) {
        const uint32_t run = order[h], e = starts[run + 1];
        for (uint32_t i = starts[run]; i < e; i += 32u) {
            const uint32_t n = min(32u, e - i);
            const uint32_t v = lane < n ? __ldg(&frags[i + lane].y) & 0xfffffffu : 0u;
            uint32_t next = 0;  // fragments of the 32 folded so far
            for (unsigned b = __ballot_sync(0xffffffffu, v != 0u); b; b &= b - 1u) {
                const uint32_t k = (uint32_t)__ffs(b) - 1u;
                if (k > next) cell = avg_fold_zero(cell);
                cell = avg_fold_int(cell, __shfl_sync(0xffffffffu, v, (int)k));
                next = k + 1u;
            }
            if (n > next) cell = avg_fold_zero(cell);
        }
    }
    return cell;
}

// Writes every node of the pool, a thread per leaf: the nodes its path is the
// first to reach, with their child blocks (the r-th node of depth d owns block
// before[d] + r + 1, before[d] the blocks of the depths above), and its leaf
// with the colours of its fragments folded in order.
struct TreeDepths {
    uint32_t before[12];
};

template <class Key>
__global__ void __launch_bounds__(kTreeBlock) k_tree_emit(uint2* __restrict__ pool, const uint2* __restrict__ frags,
                                                          const uint32_t* __restrict__ starts,
                                                          const Key* __restrict__ keys,
                                                          const uint32_t* __restrict__ order,
                                                          const uint32_t* __restrict__ heads, uint32_t leaves, int L,
                                                          const uint32_t* __restrict__ counts, uint32_t stride,
                                                          const TreeDepths T) {
    __shared__ uint32_t s_warp[12][kTreeBlock / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t chunks = (leaves + kTreeBlock - 1u) / kTreeBlock;
    for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const uint32_t l = c * kTreeBlock + threadIdx.x;
        const bool live = l < leaves;
        const int shared = live ? shared_slots(keys, heads, l, L) : L;
        for (int d = 1; d < L; ++d) {
            const unsigned b = __ballot_sync(0xffffffffu, shared < d);
            if (lane == 0) s_warp[d][w] = (uint32_t)__popc(b);
        }
        __syncthreads();
        if (threadIdx.x >= 1 && (int)threadIdx.x < L) {
            uint32_t sum = counts[(threadIdx.x - 1) * stride + c];
            for (int i = 0; i < kTreeBlock / 32; ++i) {
                const uint32_t v = s_warp[threadIdx.x][i];
                s_warp[threadIdx.x][i] = sum;
                sum += v;
            }
        }
        __syncthreads();
        const Key key = live ? keys[heads[l]] : (Key)0;
        uint32_t node = 0, block = 0;  // the path's node at depth d, and the child block it lies in
        for (int d = 1; d <= L; ++d) {
            node = block + ((uint32_t)(key >> (3 * (L - d))) & 7u);
            if (d == L) break;
            const unsigned b = __ballot_sync(0xffffffffu, shared < d);
            // the last new node of depth d up to this leaf is its own
            const uint32_t r = s_warp[d][w] + (uint32_t)__popc(b & (0xffffffffu >> (31 - lane))) - 1u;
            block = (T.before[d] + r + 1u) << 3;
            if (live && shared < d) pool[node] = make_uint2(block | 0x80000000u, 0u);
        }
        const uint32_t h0 = live ? heads[l] : 0u, h1 = live ? heads[l + 1] : 0u;
        uint32_t fragments = 0;
        for (uint32_t h = h0; h < h1 && fragments < kLongLeaf; ++h) {
            const uint32_t run = order[h];
            fragments += starts[run + 1] - starts[run];
        }
        uint32_t cell = 0u;
        if (fragments < kLongLeaf) {
            LeafCell lc{0.0f, 0.0f, 0.0f, 0.0f};
            for (uint32_t h = h0; h < h1; ++h) {
                const uint32_t run = order[h], e = starts[run + 1];
                // the fold is a serial chain; fetch four fragments ahead of it
                for (uint32_t i = starts[run]; i < e; i += 4u) {
                    uint32_t v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = i + u < e ? __ldg(&frags[i + u].y) & 0xfffffffu : 0u;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i + u < e) leaf_step(lc, v[u]);
                }
            }
            cell = leaf_word(lc);
        }
        for (unsigned b = __ballot_sync(0xffffffffu, fragments >= kLongLeaf); b; b &= b - 1u) {
            const int o = __ffs(b) - 1;
            const uint32_t v = fold_long_leaf(frags, starts, order, __shfl_sync(0xffffffffu, h0, o),
                                              __shfl_sync(0xffffffffu, h1, o));
            if (lane == o) cell = v;
        }
        if (live) pool[node] = make_uint2(0x80000000u, cell);
        __syncthreads();  // s_warp is rewritten by the next chunk
    }
}

__global__ void k_leaf_atomic(uint2* pool, const uint2* __restrict__ frags, int64_t F,
                              const uint32_t* __restrict__ cursor, int* err) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < F; i += (int64_t)gridDim.x * blockDim.x) {
        const uint2 f = __ldg(frags + i);
        const uint32_t idx = cursor[i];
        const uint32_t v = f.y & 0xfffffffu;
        uint32_t prev = 0u, newv = avg_fold(0u, v), cur;
        int guard = 0;
        while ((cur = atomicCAS(&pool[idx].y, prev, newv)) != prev) {
            prev = cur;
            newv = avg_fold(cur, v);
            if (++guard > (1 << 20)) {
                atomicExch(err, 1);
                break;
            }
        }
    }
}

// Per-node mip of one window (octreeNodeMipmapWrite.comp:50-60): y = sum(child/8).
__global__ void k_mip_nodes(uint2* pool, uint64_t begin, uint64_t num) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < num; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 n = pool[begin + i];
        if (!(n.x & 0x80000000u)) continue;
        const uint32_t child = n.x & 0x7fffffffu;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        for (int j = 0; j < 8; ++j) {
            const uint32_t v = pool[child + j].y;
#pragma unroll
            for (int c = 0; c < 4; ++c) s[c] = s[c] + (float)((v >> (8 * c)) & 0xffu) / 8.0f;
        }
        pool[begin + i].y = conv_u8x4(s[0], s[1], s[2], s[3]);
    }
}

// Canonical relabelling, one level: new window nodes read their old node via new2old.
__global__ void k_canon_flags(const uint2* __restrict__ in, const uint32_t* __restrict__ new2old, uint64_t begin,
                              uint64_t num, uint32_t* __restrict__ f) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < num; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 n = in[new2old[begin + i]];
        f[i] = (n.x >> 31) && (n.x & 0x7fffffffu) ? 1u : 0u;
    }
}

__global__ void k_canon_write(const uint2* __restrict__ in, uint2* __restrict__ out, uint32_t* __restrict__ new2old,
                              uint64_t begin, uint64_t num, const uint32_t* __restrict__ rank, uint64_t counter) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < num; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 n = in[new2old[begin + i]];
        uint32_t x = n.x & 0x80000000u;
        const uint32_t oc = n.x & 0x7fffffffu;
        if ((n.x >> 31) && oc) {
            const uint32_t nc = (uint32_t)((counter + rank[i] + 1) << 3);
            x |= nc;
            for (int c = 0; c < 8; ++c) new2old[nc + c] = oc + c;
        }
        out[begin + i] = make_uint2(x, n.y);
    }
}

static int grid_n(uint64_t n, int block = 256) {
    uint64_t g = (n + block - 1) / block;
    return (int)(g < 1 ? 1 : (g > 152 * 32 ? 152 * 32 : g));
}
static size_t a256s(size_t x) { return (x + 255) & ~size_t(255); }

// Exclusive scan of `num` 0/1 flags -> ranks; returns the number of ones (host).
static int scan_flags(const uint32_t* flags, uint32_t* rank, uint64_t num, void* tmp, size_t tmp_bytes,
                      uint32_t* d_tail, uint64_t* ones, cudaStream_t st) {
    size_t tb = tmp_bytes;
    VCT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(tmp, tb, flags, rank, (int)num, st));
    uint32_t h[2];
    VCT_CUDA_TRY(cudaMemcpyAsync(&h[0], rank + (num - 1), 4, cudaMemcpyDeviceToHost, st));
    VCT_CUDA_TRY(cudaMemcpyAsync(&h[1], flags + (num - 1), 4, cudaMemcpyDeviceToHost, st));
    VCT_CUDA_TRY(cudaStreamSynchronize(st));
    (void)d_tail;
    *ones = (uint64_t)h[0] + h[1];
    return VCT_OK;
}

}  // namespace vct

using namespace vct;

extern "C" int64_t vct_svo_pool_capacity(int64_t F) {
    if (F < 0) return -1;
    int64_t n = F * 8;
    if (n < (int64_t)VCT_MIN_OCTREE_NODE_NUM) n = VCT_MIN_OCTREE_NODE_NUM;
    if (n > (int64_t)VCT_MAX_OCTREE_NODE_NUM) n = VCT_MAX_OCTREE_NODE_NUM;
    return n;
}

namespace vct {

// Windows of the pool by depth, for the mips.
struct PoolWindows {
    uint64_t begin[12], num[12];
};

// The deterministic build into `pool`, zeroed up to the node count here.  The
// workspace holds the run starts, then (sized by the run count) the sort.
template <class Key>
static int build_sorted(const uint2* frags, uint32_t F, int L, uint2* pool, int64_t capacity, vct_workspace_s* ws,
                        uint64_t* nodes, PoolWindows* W, cudaStream_t st) {
    size_t select_bytes = 0;
    VCT_CUDA_TRY(cub::DeviceSelect::If(nullptr, select_bytes, thrust::counting_iterator<uint32_t>(0u),
                                       (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)F + 1, FragRunHead{frags, F}));
    const size_t f_arr = a256s(4 * ((size_t)F + 1)), fixed = f_arr + 512;
    int rc = workspace_reserve(ws, fixed + a256s(select_bytes));
    if (rc != VCT_OK) return rc;
    uint32_t runs = 0;
    size_t run_select = 0, sort_bytes = 0, r_arr = 0, k_arr = 0, c_arr = 0, need = 0;
    uint32_t stride = 0;
    for (;;) {
        char* b = (char*)ws->ptr;
        size_t tb = select_bytes;
        VCT_CUDA_TRY(cub::DeviceSelect::If(b + fixed, tb, thrust::counting_iterator<uint32_t>(0u), (uint32_t*)b,
                                           (uint32_t*)(b + f_arr), (int64_t)F + 1, FragRunHead{frags, F}, st));
        uint32_t nheads = 0;
        VCT_CUDA_TRY(cudaMemcpyAsync(&nheads, b + f_arr, 4, cudaMemcpyDeviceToHost, st));
        VCT_CUDA_TRY(cudaStreamSynchronize(st));
        runs = nheads - 1u;
        VCT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (Key*)nullptr, (Key*)nullptr,
                                                     (uint32_t*)nullptr, (uint32_t*)nullptr, (int)runs, 0, 3 * L));
        VCT_CUDA_TRY(cub::DeviceSelect::If(nullptr, run_select, thrust::counting_iterator<uint32_t>(0u),
                                           (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)runs + 1,
                                           LeafHead<Key>{nullptr, runs}));
        stride = (runs + kTreeBlock - 1u) / kTreeBlock;
        r_arr = a256s(4 * ((size_t)runs + 1));
        k_arr = a256s(sizeof(Key) * (size_t)runs);
        c_arr = a256s(4 * (size_t)stride * 11);
        need = fixed + 2 * k_arr + 3 * r_arr + c_arr + a256s(sort_bytes > run_select ? sort_bytes : run_select);
        if (ws->bytes >= need) break;
        if ((rc = workspace_reserve(ws, need)) != VCT_OK) return rc;  // the starts moved with the arena: select again
    }
    char* b = (char*)ws->ptr;
    const uint32_t* starts = (const uint32_t*)b;
    uint32_t* nleaf = (uint32_t*)(b + f_arr + 64);
    uint32_t* totals = (uint32_t*)(b + f_arr + 128);
    char* q = b + fixed;
    Key *kin = (Key*)q, *kout = (Key*)(q + k_arr);
    q += 2 * k_arr;
    uint32_t *vin = (uint32_t*)q, *order = (uint32_t*)(q + r_arr), *heads = (uint32_t*)(q + 2 * r_arr);
    q += 3 * r_arr;
    uint32_t* counts = (uint32_t*)q;
    void* tmp = q + c_arr;
    k_run_keys<Key><<<grid_n(runs), 256, 0, st>>>(frags, starts, runs, L, kin, vin);
    VCT_LAUNCH_CHECK();
    size_t tb = sort_bytes;
    VCT_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tb, kin, kout, vin, order, (int)runs, 0, 3 * L, st));
    tb = run_select;
    VCT_CUDA_TRY(cub::DeviceSelect::If(tmp, tb, thrust::counting_iterator<uint32_t>(0u), heads, nleaf,
                                       (int64_t)runs + 1, LeafHead<Key>{kout, runs}, st));
    const int grid = (int)(stride > 152u * 8u ? 152u * 8u : stride);
    k_tree_count<Key><<<grid, kTreeBlock, 0, st>>>(kout, heads, nleaf, L, counts, stride);
    VCT_LAUNCH_CHECK();
    k_tree_scan<<<1, 32 * L, 0, st>>>(counts, stride, nleaf, L, totals);
    VCT_LAUNCH_CHECK();
    uint32_t tot[12];
    VCT_CUDA_TRY(cudaMemcpyAsync(tot, totals, sizeof(tot), cudaMemcpyDeviceToHost, st));
    VCT_CUDA_TRY(cudaStreamSynchronize(st));
    TreeDepths T;
    uint64_t blocks = 0;
    W->begin[1] = 0;
    W->num[1] = 8;
    for (int d = 1; d < L; ++d) {
        T.before[d] = (uint32_t)blocks;
        W->begin[d + 1] = 8 + 8 * blocks;
        W->num[d + 1] = 8 * (uint64_t)tot[d];
        blocks += tot[d];
    }
    *nodes = 8 + 8 * blocks;
    if (*nodes > (uint64_t)capacity) return fail(VCT_E_OVERFLOW, "vct_svo_build: node pool capacity exceeded");
    VCT_CUDA_TRY(cudaMemsetAsync(pool, 0, 8 * (size_t)*nodes, st));
    k_tree_emit<Key><<<grid, kTreeBlock, 0, st>>>(pool, frags, starts, kout, order, heads, tot[0], L, counts, stride, T);
    VCT_LAUNCH_CHECK();
    return VCT_OK;
}

// The reference's level-by-level build with its racy allocation and averages.
static int build_atomic(const uint2* frags, int64_t F, int L, uint2* pool, int64_t capacity, vct_workspace_s* ws,
                        uint64_t* nodes, PoolWindows* W, cudaStream_t st) {
    const size_t f_arr = a256s(4 * (size_t)(F > 0 ? F : 1));
    int rc = workspace_reserve(ws, 256 + f_arr);
    if (rc != VCT_OK) return rc;
    unsigned int* counter = (unsigned int*)ws->ptr;
    int* err = (int*)ws->ptr + 1;
    uint32_t* cursor = (uint32_t*)((char*)ws->ptr + 256);
    uint64_t begin = 0, num = 8, count = 0;
    VCT_CUDA_TRY(cudaMemsetAsync(counter, 0, 8, st));
    for (int i = 1; i <= L; ++i) {
        if (begin + num > (uint64_t)capacity) return fail(VCT_E_OVERFLOW, "vct_svo_build: node pool capacity exceeded");
        W->begin[i] = begin;
        W->num[i] = num;
        k_init<<<grid_n(num), 256, 0, st>>>(pool, begin, num);
        if (F) k_flag_level<<<grid_n(F), 256, 0, st>>>(pool, frags, F, L, i, cursor);
        VCT_LAUNCH_CHECK();
        if (i != L) {
            k_alloc_atomic<<<grid_n(num), 256, 0, st>>>(pool, begin, num, counter);
            VCT_LAUNCH_CHECK();
            uint32_t c;
            VCT_CUDA_TRY(cudaMemcpyAsync(&c, counter, 4, cudaMemcpyDeviceToHost, st));
            VCT_CUDA_TRY(cudaStreamSynchronize(st));
            count = c;
            begin += num;  // octreeNodeModifyArg.comp
            num = count * 8 + 8 - begin;
        }
    }
    *nodes = count * 8 + 8;
    if (F) {
        k_leaf_atomic<<<grid_n(F), 256, 0, st>>>(pool, frags, F, cursor, err);
        VCT_LAUNCH_CHECK();
        int herr = 0;
        VCT_CUDA_TRY(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st));
        VCT_CUDA_TRY(cudaStreamSynchronize(st));
        if (herr) return fail(VCT_E_TIMEOUT, "vct_svo_build: a CAS loop gave up after 2^20 retries");
    }
    return VCT_OK;
}

}  // namespace vct

extern "C" int vct_svo_build(const uint32_t* fragments, int64_t F, int32_t L, uint32_t* pool_u32, int64_t capacity,
                             int32_t mode, int64_t* node_count, vct_workspace_s* ws, void* stream) {
    vct::NvtxRange nvtx_range("vct_svo_build");
    VCT_CHECK_ARG(node_count && ws, "vct_svo_build: null argument");
    VCT_CHECK_ARG(L >= 1 && L <= 11, "vct_svo_build: octree level must be 1..11");
    VCT_CHECK_ARG(F >= 0 && F < (1LL << 31), "vct_svo_build: fragment count out of range");
    VCT_CHECK_ARG(F == 0 || fragments, "vct_svo_build: null fragment list");
    VCT_CHECK_ARG(pool_u32 && capacity >= 8 && capacity < (1LL << 31), "vct_svo_build: bad node pool");
    VCT_CHECK_ARG(mode == VCT_SVO_DETERMINISTIC || mode == VCT_SVO_ATOMIC, "vct_svo_build: bad mode");
    *node_count = 0;
    cudaStream_t st = as_stream(stream);
    uint2* pool = reinterpret_cast<uint2*>(pool_u32);
    const uint2* frags = reinterpret_cast<const uint2*>(fragments);
    uint64_t nodes = 8;
    PoolWindows W;
    memset(&W, 0, sizeof(W));
    if (mode == VCT_SVO_ATOMIC) {
        int rc = build_atomic(frags, F, L, pool, capacity, ws, &nodes, &W, st);
        if (rc != VCT_OK) return rc;
    } else if (F == 0) {
        VCT_CUDA_TRY(cudaMemsetAsync(pool, 0, 64, st));  // the root's eight empty children
    } else {
        int rc = L <= 10 ? build_sorted<uint32_t>(frags, (uint32_t)F, L, pool, capacity, ws, &nodes, &W, st)
                         : build_sorted<unsigned long long>(frags, (uint32_t)F, L, pool, capacity, ws, &nodes, &W, st);
        if (rc != VCT_OK) return rc;
    }
    *node_count = (int64_t)nodes;
    // mips: targets t = 2, 4, 8, ... <= L and <= 2^(L-1): the window at depth L - log2(t)
    for (int k = 1; (1 << k) <= L && k <= L - 1; ++k) {
        const int depth = L - k;
        if (F) k_mip_nodes<<<grid_n(W.num[depth]), 256, 0, st>>>(pool, W.begin[depth], W.num[depth]);
        VCT_LAUNCH_CHECK();
    }
    return VCT_OK;
}

extern "C" int vct_svo_canonicalize(const uint32_t* pool_in_u32, int64_t node_count, int32_t L, uint32_t* pool_out_u32,
                                    vct_workspace_s* ws, void* stream) {
    VCT_CHECK_ARG(pool_in_u32 && pool_out_u32 && ws && pool_in_u32 != pool_out_u32, "vct_svo_canonicalize: bad argument");
    VCT_CHECK_ARG(L >= 1 && L <= 11 && node_count >= 8 && node_count < (1LL << 31), "vct_svo_canonicalize: bad size");
    cudaStream_t st = as_stream(stream);
    const uint2* in = reinterpret_cast<const uint2*>(pool_in_u32);
    uint2* out = reinterpret_cast<uint2*>(pool_out_u32);
    size_t scan_bytes = 0;
    VCT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (int)node_count));
    const size_t arr = a256s(4 * (size_t)node_count);
    int rc = workspace_reserve(ws, 3 * arr + a256s(scan_bytes));
    if (rc != VCT_OK) return rc;
    char* b = (char*)ws->ptr;
    uint32_t* new2old = (uint32_t*)b;
    uint32_t* flags = (uint32_t*)(b + arr);
    uint32_t* rank = (uint32_t*)(b + 2 * arr);
    void* tmp = b + 3 * arr;
    const uint32_t ident[8] = {0, 1, 2, 3, 4, 5, 6, 7};
    VCT_CUDA_TRY(cudaMemcpyAsync(new2old, ident, sizeof(ident), cudaMemcpyHostToDevice, st));
    uint64_t begin = 0, num = 8, count = 0;
    for (int i = 1; i <= L && num > 0; ++i) {
        if (begin + num > (uint64_t)node_count) return fail(VCT_E_BAD_ARG, "vct_svo_canonicalize: pool is not a complete build");
        k_canon_flags<<<grid_n(num), 256, 0, st>>>(in, new2old, begin, num, flags);
        VCT_LAUNCH_CHECK();
        uint64_t ones = 0;
        rc = scan_flags(flags, rank, num, tmp, scan_bytes, nullptr, &ones, st);
        if (rc != VCT_OK) return rc;
        k_canon_write<<<grid_n(num), 256, 0, st>>>(in, out, new2old, begin, num, rank, count);
        VCT_LAUNCH_CHECK();
        count += ones;
        begin += num;
        num = count * 8 + 8 - begin;
    }
    return VCT_OK;
}
