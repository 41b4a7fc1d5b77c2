// GPU LBVH construction (Karras, "Maximizing Parallelism in the Construction
// of BVHs, Octrees, and k-d Trees", HPG 2012): 63-bit Morton codes (21 bits per
// axis) of the box centroids, a radix sort of (code, primitive) pairs, one
// thread per internal node to find its range and split (equal codes are told
// apart by their sorted position, as in the paper), and a bottom-up pass that
// fills each node with the (slightly enlarged) boxes of both children.
#include <cub/cub.cuh>

#include <cfloat>

#include "az_internal.h"
#include "az_pool.h"

namespace az {
namespace {

// 21 bits spread to every third bit of a 63-bit word.
__device__ __forceinline__ unsigned long long spread3(unsigned long long v) {
    v &= 0x1FFFFFull;
    v = (v | (v << 32)) & 0x001F00000000FFFFull;
    v = (v | (v << 16)) & 0x001F0000FF0000FFull;
    v = (v | (v << 8)) & 0x100F00F00F00F00Full;
    v = (v | (v << 4)) & 0x10C30C30C30C30C3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// Bounds of the boxes' centres: kBoundsBlocks blocks, then one block over their
// results (min and max do not depend on the order).  4 M boxes: 1.2 ms in one
// block, 0.03 ms so.
constexpr uint32_t kBoundsBlocks = 592, kBoundsBlock = 256;   // four blocks a multiprocessor

__device__ __forceinline__ void block_bounds(float mn[3], float mx[3], float *out6) {
    __shared__ float s[6][kBoundsBlock / 32];
    for (int k = 0; k < 3; k++)
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xFFFFFFFFu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xFFFFFFFFu, mx[k], o));
        }
    if ((threadIdx.x & 31u) == 0)
        for (int k = 0; k < 3; k++) {
            s[k][threadIdx.x >> 5] = mn[k];
            s[3 + k][threadIdx.x >> 5] = mx[k];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        float r = s[threadIdx.x][0];
        for (uint32_t w = 1; w < kBoundsBlock / 32; w++)
            r = threadIdx.x < 3 ? fminf(r, s[threadIdx.x][w]) : fmaxf(r, s[threadIdx.x][w]);
        out6[threadIdx.x] = r;
    }
}

__global__ void __launch_bounds__(kBoundsBlock) k_bounds_part(const float4 *lo, const float4 *hi, uint32_t n,
                                                              float *part) {
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * kBoundsBlock + threadIdx.x; i < n; i += gridDim.x * kBoundsBlock) {
        const float4 a = lo[i], b = hi[i];
        const float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
        for (int k = 0; k < 3; k++) {
            mn[k] = fminf(mn[k], c[k]);
            mx[k] = fmaxf(mx[k], c[k]);
        }
    }
    block_bounds(mn, mx, part + 6 * blockIdx.x);
}

__global__ void __launch_bounds__(kBoundsBlock) k_bounds_join(const float *part, uint32_t blocks, float *out6) {
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t b = threadIdx.x; b < blocks; b += kBoundsBlock)
        for (int k = 0; k < 3; k++) {
            mn[k] = fminf(mn[k], part[6 * b + k]);
            mx[k] = fmaxf(mx[k], part[6 * b + 3 + k]);
        }
    block_bounds(mn, mx, out6);
}

// bounds: 6 floats of result, then the blocks' own
constexpr size_t kBoundsFloats = 6 + 6 * (size_t)kBoundsBlocks;
void CentreBounds(const float4 *lo, const float4 *hi, uint32_t n, float *bounds, cudaStream_t st) {
    const uint32_t blocks = std::min(kBoundsBlocks, (n + kBoundsBlock - 1) / kBoundsBlock);
    k_bounds_part<<<blocks, kBoundsBlock, 0, st>>>(lo, hi, n, bounds + 6);
    k_bounds_join<<<1, kBoundsBlock, 0, st>>>(bounds + 6, blocks, bounds);
}

__global__ void k_morton(const float4 *lo, const float4 *hi, uint32_t n, const float *bounds6,
                         unsigned long long *keys, uint32_t *vals) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 a = lo[i], b = hi[i];
    double c[3] = {0.5 * ((double)a.x + b.x), 0.5 * ((double)a.y + b.y), 0.5 * ((double)a.z + b.z)};
    unsigned long long q[3];
    for (int k = 0; k < 3; k++) {
        double ext = (double)bounds6[3 + k] - bounds6[k];
        double u = ext > 0.0 ? (c[k] - bounds6[k]) / ext : 0.5;
        u = fmin(fmax(u, 0.0), 1.0);
        q[k] = (unsigned long long)fmin(u * 2097152.0, 2097151.0);
    }
    keys[i] = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
    vals[i] = i;
}

// Common-prefix length of sorted keys i and j; equal keys continue with the
// bits of their positions (Karras 2012, section 4).
__device__ __forceinline__ int delta(const unsigned long long *k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    unsigned long long a = k[i], b = k[j];
    if (a == b) return 64 + __clz((uint32_t)(i ^ j));
    return __clzll(a ^ b);
}

// One thread per internal node i in [0, n-2]: children (internal index or
// leaf flagged with bit 31), parents, and the node's sorted primitive range.
__global__ void k_karras(const unsigned long long *k, int n, uint32_t *left, uint32_t *right, int *parent_int,
                         int *parent_leaf, uint2 *range, uint32_t leaf_base) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) > 0 ? 1 : -1;
    int dmin = delta(k, n, i, i - d);
    int lmax = 2;
    while (delta(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(k, n, i, j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    range[i] = make_uint2(leaf_base + (uint32_t)lo, (uint32_t)(hi - lo + 1));
    uint32_t lc, rc;
    if (lo == gamma) {
        lc = 0x80000000u | (uint32_t)gamma;
        parent_leaf[gamma] = i;
    } else {
        lc = (uint32_t)gamma;
        parent_int[gamma] = i;
    }
    if (hi == gamma + 1) {
        rc = 0x80000000u | (uint32_t)(gamma + 1);
        parent_leaf[gamma + 1] = i;
    } else {
        rc = (uint32_t)(gamma + 1);
        parent_int[gamma + 1] = i;
    }
    left[i] = lc;
    right[i] = rc;
}

__device__ __forceinline__ void pad_box(float4 &lo, float4 &hi) {
    // enlarge by 2^-19 of the largest magnitude so that rounding in the slab
    // test never rejects a primitive lying on a face of its box
    float m = fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(lo.z), fabsf(hi.x))),
                    fmaxf(fabsf(hi.y), fabsf(hi.z)));
    float p = m * 1.9073486328125e-06f + 1e-30f;
    lo.x -= p; lo.y -= p; lo.z -= p;
    hi.x += p; hi.y += p; hi.z += p;
}

// Bottom-up: one thread per leaf walks to the root; the second child to
// arrive at a node writes it.
__global__ void k_fill(const uint32_t *order, const float4 *plo, const float4 *phi, int n,
                       const uint32_t *left, const uint32_t *right, const int *parent_int, const int *parent_leaf,
                       float4 *ilo, float4 *ihi, unsigned int *visits, azd::BVHNode *nodes, uint32_t node_base,
                       uint32_t leaf_base) {
    int leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= n) return;
    int node = parent_leaf[leaf];
    for (int guard = 0; node >= 0 && guard < n; guard++) {
        __threadfence();
        if (atomicAdd(&visits[node], 1u) == 0) return;  // first arrival: the sibling finishes the node
        __threadfence();
        uint32_t c[2] = {left[node], right[node]};
        float4 blo[2], bhi[2];
        uint32_t ref[2], cnt[2];
        for (int s = 0; s < 2; s++) {
            if (c[s] & 0x80000000u) {
                uint32_t li = c[s] & 0x7FFFFFFFu;
                uint32_t prim = order[li];
                blo[s] = plo[prim];
                bhi[s] = phi[prim];
                ref[s] = leaf_base + li;
                cnt[s] = 1;
            } else {
                blo[s] = __ldcg(ilo + c[s]);
                bhi[s] = __ldcg(ihi + c[s]);
                ref[s] = node_base + c[s];
                cnt[s] = 0;
            }
        }
        float4 ulo = make_float4(fminf(blo[0].x, blo[1].x), fminf(blo[0].y, blo[1].y), fminf(blo[0].z, blo[1].z), 0);
        float4 uhi = make_float4(fmaxf(bhi[0].x, bhi[1].x), fmaxf(bhi[0].y, bhi[1].y), fmaxf(bhi[0].z, bhi[1].z), 0);
        __stcg(ilo + node, ulo);
        __stcg(ihi + node, uhi);
        pad_box(blo[0], bhi[0]);
        pad_box(blo[1], bhi[1]);
        azd::BVHNode out;
        out.bx = make_float4(blo[0].x, bhi[0].x, blo[1].x, bhi[1].x);
        out.by = make_float4(blo[0].y, bhi[0].y, blo[1].y, bhi[1].y);
        out.bz = make_float4(blo[0].z, bhi[0].z, blo[1].z, bhi[1].z);
        out.ch = make_uint4(ref[0], ref[1], cnt[0], cnt[1]);
        nodes[node_base + node] = out;
        node = parent_int[node];
    }
}

__global__ void k_copy_u32(const uint32_t *src, uint32_t n, uint32_t *dst) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i];
}

__global__ void k_single(const float4 *lo, const float4 *hi, azd::BVHNode *nodes, uint2 *range, uint32_t node_base,
                         uint32_t leaf_base, uint32_t *perm) {
    float4 a = lo[0], b = hi[0];
    pad_box(a, b);
    azd::BVHNode out;
    // child 1 is an empty box (lo > hi) that no ray enters
    out.bx = make_float4(a.x, b.x, FLT_MAX, -FLT_MAX);
    out.by = make_float4(a.y, b.y, FLT_MAX, -FLT_MAX);
    out.bz = make_float4(a.z, b.z, FLT_MAX, -FLT_MAX);
    out.ch = make_uint4(leaf_base, leaf_base, 1u, 1u);
    nodes[node_base] = out;
    range[node_base] = make_uint2(leaf_base, 1u);
    perm[0] = 0;
}

// ---- PLOC: parallel locally-ordered clustering (Meister, Bittner, "Parallel
// Locally-Ordered Clustering for Bounding Volume Hierarchy Construction",
// IEEE TVCG 2018).  The clusters, kept in Morton order, each find the
// neighbour within `radius` positions whose merged box has the smallest
// surface area; mutual nearest neighbours merge (the lower position keeps
// the new node), and the survivors are compacted.  Ties go to the lowest
// position, and node numbers come from scans, so the tree is the same on
// every build.

constexpr int kPlocRadius = 24;
constexpr uint32_t kLeafBit = 0x80000000u;

__device__ __forceinline__ float merged_area(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    const float dx = fmaxf(ahi.x, bhi.x) - fminf(alo.x, blo.x);
    const float dy = fmaxf(ahi.y, bhi.y) - fminf(alo.y, blo.y);
    const float dz = fmaxf(ahi.z, bhi.z) - fminf(alo.z, blo.z);
    return dx * dy + dy * dz + dz * dx;
}

// Where the rounds stand, on the device: a batch of rounds is queued without
// the host knowing the counts between them.
struct PlocState {
    uint32_t count;    // clusters
    uint32_t made;     // nodes made so far
    uint32_t side;     // which of the two cluster arrays holds them
    uint32_t pad;
};

__global__ void k_ploc_init(const uint32_t *order, const float4 *plo, const float4 *phi, uint32_t n, uint32_t *ids,
                            float4 *lo, float4 *hi, PlocState *start) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0) *start = PlocState{n, 0u, 0u, 0u};
    ids[i] = kLeafBit | i;   // leaf: its sorted position
    lo[i] = plo[order[i]];
    hi[i] = phi[order[i]];
}

__device__ __forceinline__ uint32_t cluster_count(uint32_t id, const uint32_t *node_count) {
    return (id & kLeafBit) ? 1u : node_count[id];
}

struct PlocClusters {
    uint32_t *ids[2];
    float4 *lo[2], *hi[2];
};
struct PlocNodes {
    uint32_t *left, *right, *count;
    float4 *lo, *hi;
};

// The neighbour of cluster i among 0..count-1 with the smallest merged box;
// `at` reads a cluster's box.
template <typename AT>
__device__ __forceinline__ int ploc_nearest(int i, int count, AT at) {
    float4 a0, a1;
    at(i, a0, a1);
    float best = FLT_MAX;
    int bj = i == 0 ? 1 : i - 1;
    const int j0 = max(0, i - kPlocRadius), j1 = min(count - 1, i + kPlocRadius);
    for (int j = j0; j <= j1; j++) {
        if (j == i) continue;
        float4 b0, b1;
        at(j, b0, b1);
        const float a = merged_area(a0, a1, b0, b1);
        if (a < best) {
            best = a;
            bj = j;
        }
    }
    return bj;
}

// Node `id` from clusters a and b; its box goes to ulo, uhi.
__device__ __forceinline__ void ploc_node(const PlocNodes &N, uint32_t id, uint32_t a, uint32_t b, float4 alo, float4 ahi,
                                          float4 blo, float4 bhi, float4 &ulo, float4 &uhi) {
    ulo = make_float4(fminf(alo.x, blo.x), fminf(alo.y, blo.y), fminf(alo.z, blo.z), 0.0f);
    uhi = make_float4(fmaxf(ahi.x, bhi.x), fmaxf(ahi.y, bhi.y), fmaxf(ahi.z, bhi.z), 0.0f);
    N.left[id] = a;
    N.right[id] = b;
    N.lo[id] = ulo;
    N.hi[id] = uhi;
    N.count[id] = cluster_count(a, N.count) + cluster_count(b, N.count);
}

// A round takes two launches.  k_ploc_pairs finds every cluster's neighbour
// and counts the block's new nodes and survivors (bits 32.. and 0..31 of a
// block's word).  A pair is mutual when the neighbour's neighbour is the
// cluster itself, so the block also searches for the kPlocRadius clusters on
// either side of its own, from boxes in shared memory.  k_ploc_merge adds the
// words of the blocks before its own, which replaces a scan of all clusters.
// That is quadratic in the blocks, and still less than the scan for all that a
// scene may hold: hierarchies of 21 M and 84 M triangles take 32 and 111 ms, with
// the scan 89 and 277.
// The tree of 1.3 M triangles takes 65 rounds of five launches and a wait for
// the host each when searched, flagged, scanned and merged apart.
// A count of kPlocTail or fewer is left to k_ploc_tail.
constexpr int kPlocBlock = 512;
constexpr uint32_t kPlocTail = 1024;

__global__ void __launch_bounds__(kPlocBlock) k_ploc_pairs(PlocClusters C, const PlocState *in, uint32_t *nn,
                                                           unsigned long long *words) {
    constexpr int kHalo = 2 * kPlocRadius, kSpan = kPlocBlock + 2 * kHalo;
    __shared__ float4 slo[kSpan], shi[kSpan];
    __shared__ int snn[kPlocBlock + kHalo];
    const PlocState s = *in;
    const int count = (int)s.count, first = (int)(blockIdx.x * kPlocBlock);
    if (s.count <= kPlocTail || first >= count) return;
    const float4 *lo = C.lo[s.side], *hi = C.hi[s.side];
    const int base = first - kHalo;               // cluster of slo[0]
    for (int k = threadIdx.x; k < kSpan; k += kPlocBlock) {
        const int j = base + k;
        if (j >= 0 && j < count) {
            slo[k] = lo[j];
            shi[k] = hi[j];
        }
    }
    __syncthreads();
    const int nbase = first - kPlocRadius;        // cluster of snn[0]
    for (int k = threadIdx.x; k < kPlocBlock + kHalo; k += kPlocBlock) {
        const int j = nbase + k;
        if (j >= 0 && j < count)
            snn[k] = ploc_nearest(j, count, [&](int c, float4 &l, float4 &h) {
                l = slo[c - base];
                h = shi[c - base];
            });
    }
    __syncthreads();
    const int i = first + (int)threadIdx.x;
    bool makes = false, survives = false;
    if (i < count) {
        const int j = snn[i - nbase];
        const bool mutual = snn[j - nbase] == i;
        makes = mutual && i < j;
        survives = !(mutual && i > j);
        nn[i] = (uint32_t)j | (mutual ? kLeafBit : 0u);   // the top bit: mutual
    }
    const uint32_t m = __syncthreads_count(makes), v = __syncthreads_count(survives);
    if (threadIdx.x == 0) words[blockIdx.x] = ((unsigned long long)m << 32) | v;
}

__global__ void __launch_bounds__(kPlocBlock) k_ploc_merge(PlocClusters C, PlocNodes N, const PlocState *in,
                                                           PlocState *out, const uint32_t *nn,
                                                           const unsigned long long *words) {
    const PlocState s = *in;
    if (s.count <= kPlocTail) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *out = s;
        return;
    }
    const uint32_t i = blockIdx.x * kPlocBlock + threadIdx.x;
    if (blockIdx.x * kPlocBlock >= s.count) return;
    __shared__ unsigned long long part[kPlocBlock / 32];
    __shared__ uint32_t wmakes[kPlocBlock / 32], wsurvives[kPlocBlock / 32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    // nodes and survivors of the blocks before this one
    unsigned long long before = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kPlocBlock) before += words[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
    // and of the threads before this one
    const uint32_t w = i < s.count ? nn[i] : 0u, j = w & ~kLeafBit;
    const bool mutual = i < s.count && (w & kLeafBit), makes = mutual && i < j,
               survives = i < s.count && !(mutual && i > j);
    const uint32_t mb = __ballot_sync(0xFFFFFFFFu, makes), vb = __ballot_sync(0xFFFFFFFFu, survives);
    if (lane == 0) {
        part[warp] = before;
        wmakes[warp] = __popc(mb);
        wsurvives[warp] = __popc(vb);
    }
    __syncthreads();
    before = 0;
    uint32_t id = s.made + __popc(mb & ((1u << lane) - 1u)), pos = __popc(vb & ((1u << lane) - 1u));
    for (uint32_t k = 0; k < kPlocBlock / 32; k++) {
        before += part[k];
        if (k < warp) {
            id += wmakes[k];
            pos += wsurvives[k];
        }
    }
    id += (uint32_t)(before >> 32);
    pos += (uint32_t)(before & 0xFFFFFFFFull);
    if (i == s.count - 1) {   // the last cluster: what this round made and left
        out->count = pos + (survives ? 1u : 0u);
        out->made = id + (makes ? 1u : 0u);
        out->side = s.side ^ 1u;
    }
    if (!survives) return;   // merged into its lower neighbour's node
    const uint32_t *ids = C.ids[s.side];
    const float4 *lo = C.lo[s.side], *hi = C.hi[s.side];
    uint32_t c = ids[i];
    float4 l = lo[i], h = hi[i];
    if (makes) {
        float4 ul, uh;
        ploc_node(N, id, c, ids[j], l, h, lo[j], hi[j], ul, uh);
        c = id;
        l = ul;
        h = uh;
    }
    C.ids[s.side ^ 1u][pos] = c;
    C.lo[s.side ^ 1u][pos] = l;
    C.hi[s.side ^ 1u][pos] = h;
}

// The last rounds, of at most kPlocTail clusters, by one block: a thread per
// cluster, boxes in shared memory.  Half of a large tree's rounds are here,
// and each is a few microseconds of latency instead of launches.
// rounds[0] = their number, then the nodes made before each and after the last;
// *out = the end.
__global__ void __launch_bounds__(kPlocTail) k_ploc_tail(PlocClusters C, PlocNodes N, const PlocState *in,
                                                         PlocState *out, uint32_t *rounds) {
    __shared__ float4 slo[kPlocTail], shi[kPlocTail];
    __shared__ uint32_t sid[kPlocTail];
    __shared__ uint16_t snn[kPlocTail];
    __shared__ uint32_t wmakes[kPlocTail / 32], wsurvives[kPlocTail / 32];
    const PlocState s = *in;
    const uint32_t i = threadIdx.x, warp = i >> 5, lane = i & 31u;
    uint32_t count = s.count, made = s.made, done = 0;
    if (count > kPlocTail) return;   // the host saw no progress
    uint32_t c = 0;
    float4 l = make_float4(0.0f, 0.0f, 0.0f, 0.0f), h = l;
    if (i < count) {
        c = C.ids[s.side][i];
        l = C.lo[s.side][i];
        h = C.hi[s.side][i];
    }
    while (count > 1) {
        if (i < count) {
            sid[i] = c;
            slo[i] = l;
            shi[i] = h;
        }
        __syncthreads();
        int j = 0;
        if (i < count) {
            j = ploc_nearest((int)i, (int)count, [&](int k, float4 &bl, float4 &bh) {
                bl = slo[k];
                bh = shi[k];
            });
            snn[i] = (uint16_t)j;
        }
        __syncthreads();
        const bool mutual = i < count && snn[j] == i, makes = mutual && (int)i < j,
                   survives = i < count && !(mutual && (int)i > j);
        const uint32_t mb = __ballot_sync(0xFFFFFFFFu, makes), vb = __ballot_sync(0xFFFFFFFFu, survives);
        if (lane == 0) {
            wmakes[warp] = __popc(mb);
            wsurvives[warp] = __popc(vb);
        }
        __syncthreads();
        uint32_t id = made + __popc(mb & ((1u << lane) - 1u)), pos = __popc(vb & ((1u << lane) - 1u));
        uint32_t nm = 0, nv = 0;
        for (uint32_t k = 0; k < kPlocTail / 32; k++) {
            if (k == warp) {
                id += nm;
                pos += nv;
            }
            nm += wmakes[k];
            nv += wsurvives[k];
        }
        if (makes) {
            float4 ul, uh;
            ploc_node(N, id, c, sid[j], l, h, slo[j], shi[j], ul, uh);
            c = id;
            l = ul;
            h = uh;
        }
        __syncthreads();   // every box and node of this round has been read and written
        if (i == 0) rounds[1 + done] = made;
        if (survives) {
            sid[pos] = c;
            slo[pos] = l;
            shi[pos] = h;
        }
        __syncthreads();
        done++;
        if (nm == 0) break;   // no progress: the node count tells the host
        made += nm;
        count = nv;
        if (i < count) {
            c = sid[i];
            l = slo[i];
            h = shi[i];
        }
        __syncthreads();
    }
    if (i == 0) {
        rounds[0] = done;
        rounds[1 + done] = made;
        *out = PlocState{count, made, 0u, 0u};
    }
}

// Depth-first positions, top-down one merge round at a time (a node's parent
// was made in a later round): the left child starts where its parent does,
// the right child after the left child's primitives.
__device__ __forceinline__ void ploc_first(uint32_t id, const PlocNodes &N, uint32_t *node_first, uint32_t *leaf_first) {
    const uint32_t f = node_first[id];
    const uint32_t a = N.left[id], b = N.right[id];
    const uint32_t fb = f + cluster_count(a, N.count);
    if (a & kLeafBit) leaf_first[a & ~kLeafBit] = f;
    else node_first[a] = f;
    if (b & kLeafBit) leaf_first[b & ~kLeafBit] = fb;
    else node_first[b] = fb;
}

__global__ void k_ploc_first(uint32_t node_begin, uint32_t nodes, PlocNodes N, uint32_t *node_first,
                             uint32_t *leaf_first) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nodes) ploc_first(node_begin + k, N, node_first, leaf_first);
}

// The rounds of k_ploc_tail, by one block.
__global__ void __launch_bounds__(kPlocTail) k_ploc_first_tail(const uint32_t *rounds, PlocNodes N, uint32_t *node_first,
                                                               uint32_t *leaf_first) {
    for (uint32_t r = rounds[0]; r-- > 0;) {
        const uint32_t id = rounds[1 + r] + threadIdx.x;
        if (id < rounds[2 + r]) ploc_first(id, N, node_first, leaf_first);
        __syncthreads();   // the nodes below read what this round wrote
    }
}

__global__ void k_ploc_emit(uint32_t n_nodes, const uint32_t *node_left, const uint32_t *node_right,
                            const float4 *node_lo, const float4 *node_hi, const uint32_t *node_count,
                            const uint32_t *node_first, const uint32_t *leaf_first, const float4 *plo,
                            const float4 *phi, const uint32_t *order, azd::BVHNode *nodes, uint2 *range,
                            uint32_t node_base, uint32_t leaf_base, uint32_t *err) {
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n_nodes) return;
    const uint32_t n = n_nodes + 1;
    const uint32_t c[2] = {node_left[id], node_right[id]};
    float4 blo[2], bhi[2];
    uint32_t ref[2], cnt[2];
    for (int s = 0; s < 2; s++) {
        if (c[s] & kLeafBit) {
            const uint32_t li = c[s] & ~kLeafBit;
            blo[s] = plo[order[li]];
            bhi[s] = phi[order[li]];
            uint32_t pos = leaf_first[li];
            if (pos >= n) {   // a leaf the depth-first pass did not reach: a broken tree
                atomicOr(err, 1u);
                pos = 0;
            }
            ref[s] = leaf_base + pos;
            cnt[s] = 1;
        } else {
            blo[s] = node_lo[c[s]];
            bhi[s] = node_hi[c[s]];
            ref[s] = node_base + c[s];
            cnt[s] = 0;
        }
    }
    pad_box(blo[0], bhi[0]);
    pad_box(blo[1], bhi[1]);
    azd::BVHNode out;
    out.bx = make_float4(blo[0].x, bhi[0].x, blo[1].x, bhi[1].x);
    out.by = make_float4(blo[0].y, bhi[0].y, blo[1].y, bhi[1].y);
    out.bz = make_float4(blo[0].z, bhi[0].z, blo[1].z, bhi[1].z);
    out.ch = make_uint4(ref[0], ref[1], cnt[0], cnt[1]);
    nodes[node_base + id] = out;
    uint32_t first = node_first[id], count = node_count[id];
    if ((uint64_t)first + count > n || count < 2) {
        atomicOr(err, 1u);
        first = 0;
        count = 2;
    }
    range[node_base + id] = make_uint2(leaf_base + first, count);
}

// Sorted position -> depth-first position: the primitive order the leaves' references use.
__global__ void k_ploc_perm(const uint32_t *order, const uint32_t *leaf_first, uint32_t n, uint32_t *perm) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n && leaf_first[s] < n) perm[leaf_first[s]] = order[s];   // the collapse checks it is a permutation
}

}  // namespace

int BuildPLOC(const float4 *d_lo, const float4 *d_hi, uint32_t n, azd::BVHNode *d_nodes, uint2 *d_range,
              uint32_t node_base, uint32_t leaf_base, uint32_t *d_perm, cudaStream_t stream, uint32_t *root_out) {
    if (n <= 2) return BuildLBVH(d_lo, d_hi, n, d_nodes, d_range, node_base, leaf_base, d_perm, stream, root_out);
    PoolBuf<float> bounds;
    PoolBuf<unsigned long long> keys, keys_sorted, words;
    PoolBuf<uint32_t> vals, order, ids_a, ids_b, nn, nl, nr, ncount, nfirst, lfirst, tail;
    PoolBuf<float4> lo_a, hi_a, lo_b, hi_b, nlo, nhi;
    PoolBuf<unsigned char> temp;
    PoolBuf<uint32_t> err;
    PoolBuf<PlocState> state;
    constexpr uint32_t kBatch = 8;   // rounds queued before the host looks at the count
    AZ_CUDA_TRY(err.alloc(1, stream));
    AZ_CUDA_TRY(cudaMemsetAsync(err.p, 0, sizeof(uint32_t), stream));
    AZ_CUDA_TRY(bounds.alloc(kBoundsFloats, stream));
    AZ_CUDA_TRY(keys.alloc(n, stream));
    AZ_CUDA_TRY(keys_sorted.alloc(n, stream));
    AZ_CUDA_TRY(vals.alloc(n, stream));
    AZ_CUDA_TRY(order.alloc(n, stream));
    AZ_CUDA_TRY(ids_a.alloc(n, stream));
    AZ_CUDA_TRY(ids_b.alloc(n, stream));
    AZ_CUDA_TRY(lo_a.alloc(n, stream));
    AZ_CUDA_TRY(hi_a.alloc(n, stream));
    AZ_CUDA_TRY(lo_b.alloc(n, stream));
    AZ_CUDA_TRY(hi_b.alloc(n, stream));
    AZ_CUDA_TRY(nn.alloc(n, stream));
    AZ_CUDA_TRY(words.alloc(n / kPlocBlock + 1, stream));
    AZ_CUDA_TRY(nl.alloc(n, stream));
    AZ_CUDA_TRY(nr.alloc(n, stream));
    AZ_CUDA_TRY(nlo.alloc(n, stream));
    AZ_CUDA_TRY(nhi.alloc(n, stream));
    AZ_CUDA_TRY(ncount.alloc(n, stream));
    AZ_CUDA_TRY(nfirst.alloc(n, stream));
    AZ_CUDA_TRY(lfirst.alloc(n, stream));
    AZ_CUDA_TRY(tail.alloc(kPlocTail + 2, stream));
    AZ_CUDA_TRY(state.alloc(kBatch + 1, stream));
    size_t temp_bytes = 0;
    AZ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, keys.p, keys_sorted.p, vals.p, order.p, (int)n, 0,
                                                63, stream));
    AZ_CUDA_TRY(temp.alloc(temp_bytes, stream));
    const int B = 256;
    CentreBounds(d_lo, d_hi, n, bounds.p, stream);
    k_morton<<<(n + B - 1) / B, B, 0, stream>>>(d_lo, d_hi, n, bounds.p, keys.p, vals.p);
    AZ_CUDA_TRY(cudaGetLastError());
    AZ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(temp.p, temp_bytes, keys.p, keys_sorted.p, vals.p, order.p, (int)n, 0,
                                                63, stream));
    // state[k] is where round k of a batch starts; the last round's end is the
    // next batch's start
    k_ploc_init<<<(n + B - 1) / B, B, 0, stream>>>(order.p, d_lo, d_hi, n, ids_a.p, lo_a.p, hi_a.p, state.p + kBatch);
    AZ_CUDA_TRY(cudaGetLastError());
    const PlocClusters C{{ids_a.p, ids_b.p}, {lo_a.p, lo_b.p}, {hi_a.p, hi_b.p}};
    const PlocNodes N{nl.p, nr.p, ncount.p, nlo.p, nhi.p};
    std::vector<std::pair<uint32_t, uint32_t>> rounds;   // nodes made per round: (first id, count)
    uint32_t count = n, made = 0;
    while (count > kPlocTail) {
        const uint32_t grid = (count + kPlocBlock - 1) / kPlocBlock;   // a later round's clusters are fewer
        for (uint32_t k = 0; k < kBatch; k++) {
            const PlocState *in = state.p + (k == 0 ? kBatch : k);
            k_ploc_pairs<<<grid, kPlocBlock, 0, stream>>>(C, in, nn.p, words.p);
            k_ploc_merge<<<grid, kPlocBlock, 0, stream>>>(C, N, in, state.p + k + 1, nn.p, words.p);
        }
        AZ_CUDA_TRY(cudaGetLastError());
        PlocState after[kBatch];
        AZ_CUDA_TRY(cudaMemcpyAsync(after, state.p + 1, sizeof(after), cudaMemcpyDeviceToHost, stream));
        AZ_CUDA_TRY(cudaStreamSynchronize(stream));
        for (const PlocState &a : after) {
            if (count <= kPlocTail) break;   // this round and the rest of the batch were skipped
            if (a.made <= made || a.made > n - 1 || a.count + (a.made - made) != count)
                return SetError(AZ_ERR_CUDA, "PLOC made no progress");
            rounds.push_back({made, a.made - made});
            made = a.made;
            count = a.count;
        }
    }
    k_ploc_tail<<<1, kPlocTail, 0, stream>>>(C, N, state.p + kBatch, state.p, tail.p);
    AZ_CUDA_TRY(cudaGetLastError());
    PlocState end{};
    AZ_CUDA_TRY(cudaMemcpyAsync(&end, state.p, sizeof(end), cudaMemcpyDeviceToHost, stream));
    AZ_CUDA_TRY(cudaStreamSynchronize(stream));
    if (end.count != 1 || end.made != n - 1) return SetError(AZ_ERR_CUDA, "PLOC did not build a binary tree");
    // depth-first positions from the root (the last node made) down
    const uint32_t root = n - 2;
    AZ_CUDA_TRY(cudaMemsetAsync(nfirst.p, 0, (size_t)n * sizeof(uint32_t), stream));
    AZ_CUDA_TRY(cudaMemsetAsync(lfirst.p, 0xFF, (size_t)n * sizeof(uint32_t), stream));
    k_ploc_first_tail<<<1, kPlocTail, 0, stream>>>(tail.p, N, nfirst.p, lfirst.p);
    for (size_t r = rounds.size(); r-- > 0;) {
        const uint32_t k = rounds[r].second;
        k_ploc_first<<<(k + B - 1) / B, B, 0, stream>>>(rounds[r].first, k, N, nfirst.p, lfirst.p);
    }
    AZ_CUDA_TRY(cudaGetLastError());
    k_ploc_emit<<<(n - 1 + B - 1) / B, B, 0, stream>>>(n - 1, nl.p, nr.p, nlo.p, nhi.p, ncount.p, nfirst.p, lfirst.p,
                                                       d_lo, d_hi, order.p, d_nodes, d_range, node_base, leaf_base,
                                                       err.p);
    k_ploc_perm<<<(n + B - 1) / B, B, 0, stream>>>(order.p, lfirst.p, n, d_perm);
    AZ_CUDA_TRY(cudaGetLastError());
    uint32_t err_h = 0;
    AZ_CUDA_TRY(cudaMemcpyAsync(&err_h, err.p, sizeof(err_h), cudaMemcpyDeviceToHost, stream));
    AZ_CUDA_TRY(cudaStreamSynchronize(stream));   // scratch is freed on return
    if (err_h) return SetError(AZ_ERR_CUDA, "PLOC: the depth-first numbering of the tree failed");
    *root_out = node_base + root;
    return AZ_OK;
}

int BuildLBVH(const float4 *d_lo, const float4 *d_hi, uint32_t n, azd::BVHNode *d_nodes, uint2 *d_range,
              uint32_t node_base, uint32_t leaf_base, uint32_t *d_perm, cudaStream_t stream, uint32_t *root_out) {
    if (n == 0) {
        *root_out = 0xFFFFFFFFu;
        return AZ_OK;
    }
    *root_out = node_base;
    if (n == 1) {
        k_single<<<1, 1, 0, stream>>>(d_lo, d_hi, d_nodes, d_range, node_base, leaf_base, d_perm);
        AZ_CUDA_TRY(cudaGetLastError());
        return AZ_OK;
    }
    PoolBuf<float> bounds;
    PoolBuf<unsigned long long> keys, keys_sorted;
    PoolBuf<uint32_t> vals, vals_sorted;
    PoolBuf<uint32_t> left, right;
    PoolBuf<int> parent_int, parent_leaf;
    PoolBuf<float4> ilo, ihi;
    PoolBuf<unsigned int> visits;
    PoolBuf<unsigned char> temp;
    AZ_CUDA_TRY(bounds.alloc(kBoundsFloats, stream));
    AZ_CUDA_TRY(keys.alloc(n, stream));
    AZ_CUDA_TRY(keys_sorted.alloc(n, stream));
    AZ_CUDA_TRY(vals.alloc(n, stream));
    AZ_CUDA_TRY(vals_sorted.alloc(n, stream));
    AZ_CUDA_TRY(left.alloc(n, stream));
    AZ_CUDA_TRY(right.alloc(n, stream));
    AZ_CUDA_TRY(parent_int.alloc(n, stream));
    AZ_CUDA_TRY(parent_leaf.alloc(n, stream));
    AZ_CUDA_TRY(ilo.alloc(n, stream));
    AZ_CUDA_TRY(ihi.alloc(n, stream));
    AZ_CUDA_TRY(visits.alloc(n, stream));
    size_t temp_bytes = 0;
    AZ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, keys.p, keys_sorted.p, vals.p, vals_sorted.p,
                                                (int)n, 0, 63, stream));
    AZ_CUDA_TRY(temp.alloc(temp_bytes, stream));
    const int B = 256;
    uint32_t grid = (n + B - 1) / B;
    CentreBounds(d_lo, d_hi, n, bounds.p, stream);
    k_morton<<<grid, B, 0, stream>>>(d_lo, d_hi, n, bounds.p, keys.p, vals.p);
    AZ_CUDA_TRY(cudaGetLastError());
    AZ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(temp.p, temp_bytes, keys.p, keys_sorted.p, vals.p, vals_sorted.p,
                                                (int)n, 0, 63, stream));
    AZ_CUDA_TRY(cudaMemsetAsync(parent_int.p, 0xFF, n * sizeof(int), stream));   // root's parent = -1
    AZ_CUDA_TRY(cudaMemsetAsync(visits.p, 0, n * sizeof(unsigned int), stream));
    k_karras<<<grid, B, 0, stream>>>(keys_sorted.p, (int)n, left.p, right.p, parent_int.p, parent_leaf.p,
                                     d_range + node_base, leaf_base);
    k_fill<<<grid, B, 0, stream>>>(vals_sorted.p, d_lo, d_hi, (int)n, left.p, right.p, parent_int.p, parent_leaf.p,
                                   ilo.p, ihi.p, visits.p, d_nodes, node_base, leaf_base);
    k_copy_u32<<<grid, B, 0, stream>>>(vals_sorted.p, n, d_perm);
    AZ_CUDA_TRY(cudaGetLastError());
    // scratch is freed when this returns: finish the work that uses it
    AZ_CUDA_TRY(cudaStreamSynchronize(stream));
    return AZ_OK;
}

}  // namespace az
