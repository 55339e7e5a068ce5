// rt_build.cu — the BVH built on the device: the binary SAH tree, then its
// collapse to 8-wide nodes, and the packed node arrays the traversal reads
// (full, quantised and 4-wide).
//
// The same tree as the host builder (SahBuilder in rt_host.cu), which restates
// BvhTree::sah_partition (bvh.rs:290-323): at every node the centroid bounds,
// 12 bins per axis, the prefix / suffix surface-area sweep with
// cost = 1 + (SA_l·N_l + SA_r·N_r)/SA_node, the cheapest (axis, bin) split,
// a stable counting sort of the node's primitives by bin on that axis, and a
// split at half the span when one side would be empty.  The internal node
// that splits [lo, hi) at mid is numbered mid − 1 (a bijection onto
// [0, n − 1)), so the tree does not depend on the order nodes are processed.
//
// Large nodes are split level by level: atomics (order-independent min / max
// and counts) gather the node box, centroid bounds and bin statistics, one
// thread per node chooses the split, and a stable counting sort by bin reorders
// the primitives.  Nodes below SMALL primitives are finished by one warp each.
// Compiled without FMA contraction so every comparison sees the host's values.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <vector>

#include "rt_internal.h"

namespace {

constexpr int NB = 12;           // bins per axis (bvh.rs:295)
constexpr int SMALL = 192;       // nodes below this many primitives: one warp
constexpr int CHUNK = 4096;      // primitives per block in the level kernels

struct Seg { int32_t lo, hi, parent, side; };   // side 0: parent's left child, 1: right, −1: root

// Scratch of one call: one allocation cut into 256-byte aligned parts.  A build
// made 33 scratch allocations and as many releases, driver calls of 0.1-0.3 ms
// each once they are large (327,680 triangles: 20.3 ms a build, of 4.7 ms in
// kernels; 7.2 ms with one allocation per call, one copy each way per level and
// k_scatter's sort).
struct Arena {
    void* base = nullptr;
    size_t total = 0;
    std::vector<std::pair<void**, size_t>> parts;
    template <typename T>
    void part(T** p, size_t bytes) {
        parts.push_back({(void**)p, total});
        total += (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
    }
    cudaError_t open() {
        cudaError_t e = cudaMalloc(&base, total);
        if (e != cudaSuccess) { base = nullptr; return e; }
        for (auto& q : parts) *q.first = (char*)base + q.second;
        return e;
    }
    ~Arena() { if (base) cudaFree(base); }
};

// ordered-integer images of floats for atomicMin / atomicMax
__device__ __forceinline__ int f2o(float f) { int i = __float_as_int(f); return i >= 0 ? i : i ^ 0x7FFFFFFF; }
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

__device__ __forceinline__ float area6(const float* b) {                          // aabb surface area
    float dx = b[3] - b[0], dy = b[4] - b[1], dz = b[5] - b[2];
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}
__device__ __forceinline__ void unite6(float* a, const float* b) {
    for (int k = 0; k < 3; k++) { a[k] = fminf(a[k], b[k]); a[3 + k] = fmaxf(a[3 + k], b[3 + k]); }
}
__device__ __forceinline__ int bin_of(float c, float cmn, float ext) {
    float t = (c - cmn) / ext;
    return min((int)((float)NB * t), NB - 1);
}

// ── triangles ───────────────────────────────────────────────────────────────
// The box of every triangle (triangle.rs:128-140: over v0, v0 + e1, v0 + e2,
// padded as aabb.rs:18-29), the arithmetic of the host's boxes.
__global__ void k_tri_boxes(const float* __restrict__ v, int32_t n, float* box) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* p = v + (size_t)i * 9;
        for (int a = 0; a < 3; a++) {
            float c0 = p[a], c1 = c0 + (p[3 + a] - c0), c2 = c0 + (p[6 + a] - c0);
            float mn = fminf(fminf(c0, c1), c2), mx = fmaxf(fmaxf(c0, c1), c2);
            float pd = mx - mn < 0.0001f ? 0.0001f : 0.0f;
            box[(size_t)i * 6 + a] = mn - pd;
            box[(size_t)i * 6 + 3 + a] = mx + pd;
        }
    }
}
// the union of n boxes, as ordered-integer images (initialised by k_stats_init)
__global__ void k_union_boxes(const float* __restrict__ box, int32_t n, int32_t* out) {
    float v[6];
    for (int k = 0; k < 3; k++) { v[k] = INFINITY; v[3 + k] = -INFINITY; }
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = 0; k < 3; k++) {
            v[k] = fminf(v[k], box[(size_t)i * 6 + k]);
            v[3 + k] = fmaxf(v[3 + k], box[(size_t)i * 6 + 3 + k]);
        }
    for (int k = 0; k < 6; k++)
        for (int o = 16; o > 0; o >>= 1) {
            float x = __shfl_xor_sync(0xFFFFFFFFu, v[k], o);
            v[k] = k < 3 ? fminf(v[k], x) : fmaxf(v[k], x);
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 6; k++) { if (k < 3) atomicMin(out + k, f2o(v[k])); else atomicMax(out + k, f2o(v[k])); }
}
// the triangle records in leaf order (rt_device.cuh) from the caller's arrays
__global__ void k_tri_records(const int32_t* __restrict__ order, int32_t n, rth::RawTris T, float4* tri, float4* nrm,
                              float4* uv, float4* tan) {
    for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int32_t g = order[k];
        const float* v = T.v + (size_t)g * 9;
        float e1[3], e2[3];
        for (int a = 0; a < 3; a++) { e1[a] = v[3 + a] - v[a]; e2[a] = v[6 + a] - v[a]; }
        tri[(size_t)k * 3] = make_float4(v[0], v[1], v[2], e1[0]);
        tri[(size_t)k * 3 + 1] = make_float4(e1[1], e1[2], e2[0], e2[1]);
        tri[(size_t)k * 3 + 2] = make_float4(e2[2], __int_as_float(g), __int_as_float(T.mat[g]), __int_as_float(T.n ? 1 : 0));
        if (T.n) {
            const float* q = T.n + (size_t)g * 9;
            nrm[(size_t)k * 3] = make_float4(q[0], q[1], q[2], q[3]);
            nrm[(size_t)k * 3 + 1] = make_float4(q[4], q[5], q[6], q[7]);
            nrm[(size_t)k * 3 + 2] = make_float4(q[8], 0.f, 0.f, 0.f);
        }
        if (T.uv) {
            const float* u = T.uv + (size_t)g * 6;
            const float* t = T.tan + (size_t)g * 9;
            uv[(size_t)k * 2] = make_float4(u[0], u[1], u[2], u[3]);
            uv[(size_t)k * 2 + 1] = make_float4(u[4], u[5], 0.f, 0.f);
            tan[(size_t)k * 3] = make_float4(t[0], t[1], t[2], t[3]);
            tan[(size_t)k * 3 + 1] = make_float4(t[4], t[5], t[6], t[7]);
            tan[(size_t)k * 3 + 2] = make_float4(t[8], 0.f, 0.f, 0.f);
        }
    }
}

// node statistics: box (6), centroid bounds (6), then per axis per bin a count
// and a box (7 words): 12 + 3·NB·7 ints
constexpr int ST_WORDS = 12 + 3 * NB * 7;

__global__ void k_centroids(const float* __restrict__ box, int32_t n, float* __restrict__ cen, int32_t* idx) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* b = box + (size_t)i * 6;
        for (int a = 0; a < 3; a++) cen[(size_t)i * 3 + a] = (b[a] + b[3 + a]) * 0.5f;
        idx[i] = i;
    }
}

__global__ void k_stats_init(int32_t* st, int32_t nseg) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nseg * ST_WORDS; i += gridDim.x * blockDim.x) {
        int w = i % ST_WORDS;
        bool is_min;
        if (w < 12) is_min = (w % 6) < 3;
        else {
            int r = (w - 12) % 7;
            if (r == 0) { st[i] = 0; continue; }                 // count
            is_min = r <= 3;
        }
        st[i] = is_min ? 0x7F800000 : (int)0xFF800000 ^ 0x7FFFFFFF;   // +inf / −inf images
    }
}

// pass 1: node box and centroid bounds (chunk c of segment chunk_seg[c])
__global__ void k_stats_bounds(const Seg* __restrict__ segs, const int32_t* __restrict__ chunk_seg,
                               const int32_t* __restrict__ chunk_lo, int32_t nchunks, const int32_t* __restrict__ idx,
                               const float* __restrict__ box, const float* __restrict__ cen, int32_t* st) {
    __shared__ int sh[12];
    for (int32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        if (threadIdx.x < 12) sh[threadIdx.x] = (threadIdx.x % 6) < 3 ? 0x7F800000 : (int)0xFF800000 ^ 0x7FFFFFFF;
        __syncthreads();
        const Seg s = segs[chunk_seg[c]];
        int32_t lo = chunk_lo[c], hi = min(lo + CHUNK, s.hi);
        float v[12];
        for (int k = 0; k < 3; k++) { v[k] = INFINITY; v[3 + k] = -INFINITY; v[6 + k] = INFINITY; v[9 + k] = -INFINITY; }
        for (int32_t k = lo + threadIdx.x; k < hi; k += blockDim.x) {
            int32_t o = idx[k];
            const float* b = box + (size_t)o * 6;
            for (int a = 0; a < 3; a++) {
                v[a] = fminf(v[a], b[a]); v[3 + a] = fmaxf(v[3 + a], b[3 + a]);
                float cc = cen[(size_t)o * 3 + a];
                v[6 + a] = fminf(v[6 + a], cc); v[9 + a] = fmaxf(v[9 + a], cc);
            }
        }
        for (int w = 0; w < 12; w++) {
            if ((w % 6) < 3) atomicMin(&sh[w], f2o(v[w])); else atomicMax(&sh[w], f2o(v[w]));
        }
        __syncthreads();
        if (threadIdx.x < 12) {
            int32_t* g = st + (size_t)chunk_seg[c] * ST_WORDS;
            if ((threadIdx.x % 6) < 3) atomicMin(&g[threadIdx.x], sh[threadIdx.x]);
            else atomicMax(&g[threadIdx.x], sh[threadIdx.x]);
        }
        __syncthreads();
    }
}

// pass 2: per axis with a non-degenerate centroid extent, bin counts and boxes
__global__ void k_stats_bins(const Seg* __restrict__ segs, const int32_t* __restrict__ chunk_seg,
                             const int32_t* __restrict__ chunk_lo, int32_t nchunks, const int32_t* __restrict__ idx,
                             const float* __restrict__ box, const float* __restrict__ cen, int32_t* st) {
    __shared__ int sh[3 * NB * 7];
    for (int32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        for (int w = threadIdx.x; w < 3 * NB * 7; w += blockDim.x) {
            int r = w % 7;
            sh[w] = r == 0 ? 0 : (r <= 3 ? 0x7F800000 : (int)0xFF800000 ^ 0x7FFFFFFF);
        }
        __syncthreads();
        int32_t s = chunk_seg[c];
        const int32_t* g = st + (size_t)s * ST_WORDS;
        float cmn[3], ext[3];
        for (int a = 0; a < 3; a++) { cmn[a] = o2f(g[6 + a]); ext[a] = o2f(g[9 + a]) - cmn[a]; }
        int32_t lo = chunk_lo[c], hi = min(lo + CHUNK, segs[s].hi);
        for (int32_t k = lo + threadIdx.x; k < hi; k += blockDim.x) {
            int32_t o = idx[k];
            const float* b = box + (size_t)o * 6;
            for (int a = 0; a < 3; a++) {
                if (ext[a] < 1e-6f) continue;
                int bi = bin_of(cen[(size_t)o * 3 + a], cmn[a], ext[a]);
                int* bw = sh + (a * NB + bi) * 7;
                atomicAdd(bw, 1);
                for (int q = 0; q < 3; q++) { atomicMin(bw + 1 + q, f2o(b[q])); atomicMax(bw + 4 + q, f2o(b[3 + q])); }
            }
        }
        __syncthreads();
        int32_t* gw = st + (size_t)s * ST_WORDS + 12;
        for (int w = threadIdx.x; w < 3 * NB * 7; w += blockDim.x) {
            int r = w % 7;
            if (r == 0) { if (sh[w]) atomicAdd(gw + w, sh[w]); }
            else if (r <= 3) atomicMin(gw + w, sh[w]);
            else atomicMax(gw + w, sh[w]);
        }
        __syncthreads();
    }
}

// the split of one node from its statistics (SahBuilder::partition's sweep);
// *bax, *ext_ok: the axis the primitives are binned on; returns the split
// offset within the node
__device__ int32_t choose_split(const int32_t* g, int32_t span, int* bax_out, bool* binned) {
    float nb[6];
    for (int w = 0; w < 6; w++) nb[w] = o2f(g[w]);
    float nsa = area6(nb);
    float best = INFINITY;
    int bax = 0, bsp = 0;
    for (int ax = 0; ax < 3; ax++) {
        float ext = o2f(g[9 + ax]) - o2f(g[6 + ax]);
        if (ext < 1e-6f) continue;
        const int32_t* bw = g + 12 + ax * NB * 7;
        float lsa[NB];
        uint32_t ln[NB];
        bool ah = false;
        float acc[6];
        uint32_t an = 0;
        for (int i = 0; i < NB; i++) {
            const int32_t* q = bw + i * 7;
            an += (uint32_t)q[0];
            if (q[0]) {
                float b[6];
                for (int w = 0; w < 6; w++) b[w] = o2f(q[1 + w]);
                if (ah) unite6(acc, b); else for (int w = 0; w < 6; w++) acc[w] = b[w];
                ah = true;
            }
            ln[i] = an;
            lsa[i] = ah ? area6(acc) : 0.0f;
        }
        ah = false;
        an = 0;
        for (int sp = NB - 2; sp >= 0; sp--) {
            const int32_t* q = bw + (sp + 1) * 7;
            an += (uint32_t)q[0];
            if (q[0]) {
                float b[6];
                for (int w = 0; w < 6; w++) b[w] = o2f(q[1 + w]);
                if (ah) unite6(acc, b); else for (int w = 0; w < 6; w++) acc[w] = b[w];
                ah = true;
            }
            uint32_t nl = ln[sp], nr = an;
            if (nl == 0 || nr == 0) continue;
            float rsa = ah ? area6(acc) : 0.0f;
            float cost = 1.0f + (lsa[sp] * (float)nl + rsa * (float)nr) / nsa;
            if (cost < best) { best = cost; bax = ax; bsp = sp; }
        }
    }
    float ext = o2f(g[9 + bax]) - o2f(g[6 + bax]);
    *bax_out = bax;
    *binned = !(ext < 1e-6f);
    uint32_t mid_off = 0;
    if (*binned) {
        const int32_t* bw = g + 12 + bax * NB * 7;
        for (int b = 0; b <= bsp; b++) mid_off += (uint32_t)bw[b * 7];
    } else {
        mid_off = (uint32_t)span;                            // every primitive in bin 0
    }
    return (mid_off == 0 || mid_off == (uint32_t)span) ? span / 2 : (int32_t)mid_off;
}

struct LevelOut {
    Seg* next; int32_t* n_next;          // large children
    Seg* small; int32_t* n_small;        // small children
};

__device__ void link(int32_t* bl, int32_t* br, int32_t* root, const Seg& s, int32_t ref) {
    if (s.side < 0) *root = ref;
    else if (s.side == 0) bl[s.parent] = ref;
    else br[s.parent] = ref;
}
__device__ void emit_child(const Seg& c, const float* box, const int32_t* idx, int32_t* bl, int32_t* br,
                           int32_t* root, float* bbox, LevelOut out) {
    int32_t len = c.hi - c.lo;
    if (len == 1) { link(bl, br, root, c, -c.lo - 1); return; }
    if (len < SMALL) out.small[atomicAdd(out.n_small, 1)] = c;
    else out.next[atomicAdd(out.n_next, 1)] = c;
}

// one thread per large node: choose the split, write the bin keys' axis, the
// node box, and queue the two children
__global__ void k_split(const Seg* __restrict__ segs, int32_t nseg, const int32_t* __restrict__ st, int32_t* mids,
                        int32_t* axes, int32_t* bl, int32_t* br, int32_t* root, float* bbox) {
    for (int32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) {
        const int32_t* g = st + (size_t)s * ST_WORDS;
        int bax;
        bool binned;
        int32_t span = segs[s].hi - segs[s].lo;
        int32_t mid = choose_split(g, span, &bax, &binned);
        mids[s] = segs[s].lo + mid;
        axes[s] = binned ? bax : -1;
        int32_t id = segs[s].lo + mid - 1;
        for (int w = 0; w < 6; w++) bbox[(size_t)id * 6 + w] = o2f(g[w]);
        link(bl, br, root, segs[s], id);
    }
}

__global__ void k_keys(const Seg* __restrict__ segs, const int32_t* __restrict__ chunk_seg,
                       const int32_t* __restrict__ chunk_lo, int32_t nchunks, const int32_t* __restrict__ idx,
                       const float* __restrict__ cen, const int32_t* __restrict__ st, const int32_t* __restrict__ axes,
                       uint8_t* keys, int32_t* hist) {
    __shared__ int32_t cnt[NB];
    for (int32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        if (threadIdx.x < NB) cnt[threadIdx.x] = 0;
        __syncthreads();
        int32_t s = chunk_seg[c];
        int ax = axes[s];
        const int32_t* g = st + (size_t)s * ST_WORDS;
        float cmn = ax >= 0 ? o2f(g[6 + ax]) : 0.0f, ext = ax >= 0 ? o2f(g[9 + ax]) - cmn : 1.0f;
        int32_t lo = chunk_lo[c], hi = min(lo + CHUNK, segs[s].hi);
        for (int32_t k = lo + threadIdx.x; k < hi; k += blockDim.x) {
            int b = ax >= 0 ? bin_of(cen[(size_t)idx[k] * 3 + ax], cmn, ext) : 0;
            keys[k] = (uint8_t)b;
            atomicAdd(&cnt[b], 1);
        }
        __syncthreads();
        if (threadIdx.x < NB) hist[(size_t)threadIdx.x * nchunks + c] = cnt[threadIdx.x];
        __syncthreads();
    }
}

// The stable sort of every large node's primitives by bin: k_keys counts each
// chunk's bins, k_offsets turns the counts into first positions (one block per
// node, one warp per bin, the node's chunks first[s] .. first[s + 1]), k_scatter
// places the chunk's primitives in order.  A segmented radix sort gives a node to
// one block, so the first levels ran on one, two, four ... of 148 SMs
// (327,680 triangles: 1.12 ms of sorting; 0.23 ms here).
__global__ void __launch_bounds__(NB * 32) k_offsets(const Seg* __restrict__ segs, const int32_t* __restrict__ first,
                                                     int32_t nchunks, int32_t* hist) {
    __shared__ int32_t tot[NB];
    const int32_t s = blockIdx.x, b = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int32_t c0 = first[s], c1 = first[s + 1];
    int32_t* h = hist + (size_t)b * nchunks;
    int32_t sum = 0;
    for (int32_t c = c0 + lane; c < c1; c += 32) sum += h[c];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) tot[b] = sum;
    __syncthreads();
    int32_t run = segs[s].lo;
    for (int q = 0; q < b; q++) run += tot[q];
    for (int32_t c = c0; c < c1; c += 32) {
        int32_t v = c + lane < c1 ? h[c + lane] : 0, x = v;
        for (int o = 1; o < 32; o <<= 1) {
            int32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (c + lane < c1) h[c + lane] = run + x - v;
        run += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
}
constexpr int SCATTER_WARPS = 8, SCATTER_RUN = CHUNK / SCATTER_WARPS;   // consecutive primitives per warp
__global__ void __launch_bounds__(SCATTER_WARPS * 32)
k_scatter(const Seg* __restrict__ segs, const int32_t* __restrict__ chunk_seg, const int32_t* __restrict__ chunk_lo,
          int32_t nchunks, const int32_t* __restrict__ hist, const uint8_t* __restrict__ keys,
          const int32_t* __restrict__ from, int32_t* to) {
    __shared__ int32_t at[SCATTER_WARPS][NB + 1];   // [NB]: lanes past the chunk's end
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t below = (1u << lane) - 1u;
    for (int32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        if (lane <= NB) at[w][lane] = 0;
        __syncwarp();
        const int32_t lo = chunk_lo[c] + w * SCATTER_RUN, hi = min(chunk_lo[c] + CHUNK, segs[chunk_seg[c]].hi);
        for (int i = 0; i < SCATTER_RUN; i += 32) {
            const int32_t k = lo + i + lane;
            const int b = k < hi ? keys[k] : NB;
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, b);
            if (!(peers & below)) at[w][b] += __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < NB) {
            int32_t run = hist[(size_t)threadIdx.x * nchunks + c];
            for (int q = 0; q < SCATTER_WARPS; q++) {
                int32_t v = at[q][threadIdx.x];
                at[q][threadIdx.x] = run;
                run += v;
            }
        }
        __syncthreads();
        for (int i = 0; i < SCATTER_RUN; i += 32) {
            const int32_t k = lo + i + lane;
            const int b = k < hi ? keys[k] : NB;
            const uint32_t peers = __match_any_sync(0xFFFFFFFFu, b);
            if (k < hi) to[at[w][b] + __popc(peers & below)] = from[k];
            __syncwarp();
            if (!(peers & below)) at[w][b] += __popc(peers);
            __syncwarp();
        }
        __syncthreads();
    }
}

__global__ void k_copy_back(const Seg* __restrict__ segs, const int32_t* __restrict__ chunk_seg,
                            const int32_t* __restrict__ chunk_lo, int32_t nchunks, const int32_t* __restrict__ from,
                            int32_t* to) {
    for (int32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        int32_t lo = chunk_lo[c], hi = min(lo + CHUNK, segs[chunk_seg[c]].hi);
        for (int32_t k = lo + threadIdx.x; k < hi; k += blockDim.x) to[k] = from[k];
    }
}

__global__ void k_children(const Seg* __restrict__ segs, int32_t nseg, const int32_t* __restrict__ mids,
                           const float* box, const int32_t* idx, int32_t* bl, int32_t* br, int32_t* root, float* bbox,
                           LevelOut out) {
    for (int32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) {
        int32_t id = mids[s] - 1;
        emit_child(Seg{segs[s].lo, mids[s], id, 0}, box, idx, bl, br, root, bbox, out);
        emit_child(Seg{mids[s], segs[s].hi, id, 1}, box, idx, bl, br, root, bbox, out);
    }
}

// One warp finishes a small node: the sequential partition's steps over its
// range, each by all lanes, with the range's boxes, order and pending ranges in
// shared memory.  Every step is order-independent (min, max, counts) or keeps
// the order (the stable sort ranks equal bins by position), so the tree is the
// sequential one.  A thread per node, which walked the range five times per
// split through global memory, was the longest kernel of a build (327,680
// triangles: 15.0 ms of 18.7, at 64 threads per block on 2-3 % of the GPU's lanes).
constexpr int SMALL_WARPS = 4;
struct SmallWarp {
    float box[SMALL][6];
    float cen[SMALL][3];
    int32_t bins[3 * NB * 7];            // as in the large nodes' statistics
    uint16_t ord[2][SMALL];              // the range's primitives (local ids), and the sort's output
    uint16_t off[NB];
    Seg stack[64];                       // pending right halves: the smaller side is finished first
};
__device__ __forceinline__ float wmin(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
__device__ __forceinline__ float wmax(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
__global__ void __launch_bounds__(SMALL_WARPS * 32) k_small(const Seg* __restrict__ segs, int32_t nseg,
                                                            const float* __restrict__ box,
                                                            const float* __restrict__ cen, int32_t* idx, int32_t* bl,
                                                            int32_t* br, int32_t* root, float* bbox) {
    extern __shared__ __align__(16) unsigned char small_mem[];
    SmallWarp& W = reinterpret_cast<SmallWarp*>(small_mem)[threadIdx.x >> 5];
    const uint32_t FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    for (int32_t si = blockIdx.x * SMALL_WARPS + (threadIdx.x >> 5); si < nseg; si += gridDim.x * SMALL_WARPS) {
        const Seg whole = segs[si];
        const int32_t base = whole.lo, n = whole.hi - whole.lo;
        for (int k = lane; k < n; k += 32) {
            int32_t o = idx[base + k];
            for (int w = 0; w < 6; w++) W.box[k][w] = box[(size_t)o * 6 + w];
            for (int a = 0; a < 3; a++) W.cen[k][a] = cen[(size_t)o * 3 + a];
            W.ord[0][k] = (uint16_t)k;
        }
        __syncwarp();
        int sp = 0;
        Seg s = whole;
        while (true) {
            const int lo = s.lo - base, span = s.hi - s.lo;
            if (span == 1) {
                if (lane == 0) link(bl, br, root, s, -s.lo - 1);
            } else {
                // node box and centroid bounds
                float v[12];
                for (int k = 0; k < 3; k++) { v[k] = v[6 + k] = INFINITY; v[3 + k] = v[9 + k] = -INFINITY; }
                for (int k = lane; k < span; k += 32) {
                    int o = W.ord[0][lo + k];
                    for (int a = 0; a < 3; a++) {
                        v[a] = fminf(v[a], W.box[o][a]);
                        v[3 + a] = fmaxf(v[3 + a], W.box[o][3 + a]);
                        v[6 + a] = fminf(v[6 + a], W.cen[o][a]);
                        v[9 + a] = fmaxf(v[9 + a], W.cen[o][a]);
                    }
                }
                for (int w = 0; w < 12; w++) v[w] = (w % 6) < 3 ? wmin(v[w]) : wmax(v[w]);
                const float nsa = area6(v);
                // bin counts and boxes per axis
                for (int w = lane; w < 3 * NB * 7; w += 32) {
                    int r = w % 7;
                    W.bins[w] = r == 0 ? 0 : (r <= 3 ? 0x7F800000 : (int)0xFF800000 ^ 0x7FFFFFFF);
                }
                __syncwarp();
                for (int k = lane; k < span; k += 32) {
                    int o = W.ord[0][lo + k];
                    for (int a = 0; a < 3; a++) {
                        float ext = v[9 + a] - v[6 + a];
                        if (ext < 1e-6f) continue;
                        int* bw = W.bins + (a * NB + bin_of(W.cen[o][a], v[6 + a], ext)) * 7;
                        atomicAdd(bw, 1);
                        for (int q = 0; q < 3; q++) {
                            atomicMin(bw + 1 + q, f2o(W.box[o][q]));
                            atomicMax(bw + 4 + q, f2o(W.box[o][3 + q]));
                        }
                    }
                }
                __syncwarp();
                // the cheapest split: the sequential sweep takes axes upward and splits
                // downward and keeps the first of equal costs
                float best = INFINITY;
                int bax = 0, bsp = 0, brank = 64;
                for (int c = lane; c < 3 * (NB - 1); c += 32) {
                    const int ax = c / (NB - 1), q = c % (NB - 1);
                    if (v[9 + ax] - v[6 + ax] < 1e-6f) continue;
                    float l[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY}, r[6];
                    for (int w = 0; w < 6; w++) r[w] = l[w];
                    uint32_t nl = 0, nr = 0;
                    for (int i = 0; i < NB; i++) {
                        const int32_t* bw = W.bins + (ax * NB + i) * 7;
                        uint32_t cnt = (uint32_t)bw[0];
                        if (!cnt) continue;
                        float b[6];
                        for (int w = 0; w < 6; w++) b[w] = o2f(bw[1 + w]);
                        if (i <= q) { unite6(l, b); nl += cnt; } else { unite6(r, b); nr += cnt; }
                    }
                    if (nl == 0 || nr == 0) continue;
                    float cost = 1.0f + (area6(l) * (float)nl + area6(r) * (float)nr) / nsa;
                    if (!(cost < INFINITY)) continue;
                    int rank = ax * (NB - 1) + (NB - 2 - q);
                    if (cost < best || (cost == best && rank < brank)) { best = cost; bax = ax; bsp = q; brank = rank; }
                }
                for (int o = 16; o > 0; o >>= 1) {
                    float c2 = __shfl_xor_sync(FULL, best, o);
                    int a2 = __shfl_xor_sync(FULL, bax, o), p2 = __shfl_xor_sync(FULL, bsp, o), r2 = __shfl_xor_sync(FULL, brank, o);
                    if (c2 < best || (c2 == best && r2 < brank)) { best = c2; bax = a2; bsp = p2; brank = r2; }
                }
                if (brank == 64) { bax = 0; bsp = 0; }
                const float cmn = v[6 + bax], ext = v[9 + bax] - cmn;
                // stable counting sort by bin (a degenerate axis: every primitive in bin 0)
                int mid_off = 0;
                if (ext < 1e-6f) {
                    mid_off = span;
                } else {
                    if (lane == 0) {
                        int run = 0;
                        for (int i = 0; i < NB; i++) { W.off[i] = (uint16_t)run; run += W.bins[(bax * NB + i) * 7]; }
                    }
                    __syncwarp();
                    mid_off = bsp + 1 < NB ? W.off[bsp + 1] : span;
                    __syncwarp();
                    for (int k0 = 0; k0 < span; k0 += 32) {
                        const int k = k0 + lane;
                        const int o = k < span ? W.ord[0][lo + k] : 0;
                        const int bi = k < span ? bin_of(W.cen[o][bax], cmn, ext) : NB;
                        const uint32_t same = __match_any_sync(FULL, bi);
                        if (k < span) {
                            int at = W.off[bi] + __popc(same & lt);
                            W.ord[1][lo + at] = (uint16_t)o;
                        }
                        __syncwarp();
                        if (k < span && (same & lt) == 0) W.off[bi] += (uint16_t)__popc(same);
                        __syncwarp();
                    }
                    for (int k = lane; k < span; k += 32) W.ord[0][lo + k] = W.ord[1][lo + k];
                    __syncwarp();
                }
                const int mid = (mid_off == 0 || mid_off == span) ? span / 2 : mid_off;
                const int32_t id = s.lo + mid - 1;
                if (lane < 6) {
                    float w = v[0];
                    for (int q = 1; q < 6; q++) if (lane == q) w = v[q];
                    bbox[(size_t)id * 6 + lane] = w;
                }
                if (lane == 0) link(bl, br, root, s, id);
                // the larger half waits: at most log2(SMALL) halves wait at once
                Seg L{s.lo, s.lo + mid, id, 0}, R{s.lo + mid, s.hi, id, 1};
                const bool left_first = mid <= span - mid;
                if (lane == 0) W.stack[sp] = left_first ? R : L;
                sp++;
                s = left_first ? L : R;
                __syncwarp();
                continue;
            }
            if (sp == 0) break;
            s = W.stack[--sp];
            __syncwarp();
        }
        // the range's final order, through the original ids
        for (int k0 = 0; k0 < n; k0 += 32 * 6) {
            int32_t o[6];
            for (int q = 0; q < 6; q++) { int k = k0 + q * 32 + lane; if (k < n) o[q] = idx[base + W.ord[0][k]]; }
            __syncwarp();
            for (int q = 0; q < 6; q++) { int k = k0 + q * 32 + lane; if (k < n) idx[base + k] = o[q]; }
        }
        __syncwarp();
    }
}

// ── the collapse to 8-wide nodes on the device ──────────────────────────────
// The host collapse (SahBuilder::collapse) builds a wide node from binary node
// b by opening the inner child of largest surface area (the first of equal
// ones) until 8 children (or only leaves) remain, and numbers the wide nodes
// in preorder, leaves in the order the preorder meets them.  Here: every
// binary node's opening is computed in parallel; the wide nodes are found
// level by level from the root; subtree node and leaf counts are summed
// bottom-up and the preorder indices handed down; then one thread per wide
// node writes it.

// kids of the wide node rooted at binary node b (≥ 0 binary node, < 0 leaf)
__global__ void k_wide_kids(const int32_t* __restrict__ bl, const int32_t* __restrict__ br,
                            const float* __restrict__ bbox, int32_t nn, int32_t* kids, int32_t* nk, int width) {
    for (int32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < nn; b += gridDim.x * blockDim.x) {
        int32_t k[8];
        int n = 2;
        k[0] = bl[b]; k[1] = br[b];
        for (int c = 2; c < 8; c++) k[c] = 0;
        while (n < width) {
            int best = -1;
            float ba = -1.0f;
            for (int i = 0; i < n; i++)
                if (k[i] >= 0) { float a = area6(bbox + (size_t)k[i] * 6); if (a > ba) { ba = a; best = i; } }
            if (best < 0) break;
            int32_t o = k[best];
            k[best] = bl[o];
            k[n++] = br[o];
        }
        for (int c = 0; c < 8; c++) kids[(size_t)b * 8 + c] = k[c];
        nk[b] = n;
    }
}

__global__ void k_count_inner(const int32_t* __restrict__ lvl, int32_t m, const int32_t* __restrict__ kids,
                              const int32_t* __restrict__ nk, int32_t* cnt) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int32_t b = lvl[i], c = 0;
        for (int j = 0; j < nk[b]; j++) c += kids[(size_t)b * 8 + j] >= 0;
        cnt[i] = c;
    }
}
__global__ void k_next_level(const int32_t* __restrict__ lvl, int32_t m, const int32_t* __restrict__ kids,
                             const int32_t* __restrict__ nk, const int32_t* __restrict__ pos, int32_t* next) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int32_t b = lvl[i], o = pos[i];
        for (int j = 0; j < nk[b]; j++) {
            int32_t k = kids[(size_t)b * 8 + j];
            if (k >= 0) next[o++] = k;
        }
    }
}
// wide nodes (S) and leaves (L) in the wide subtree of every node of a level
__global__ void k_subtree_sizes(const int32_t* __restrict__ lvl, int32_t m, const int32_t* __restrict__ kids,
                                const int32_t* __restrict__ nk, int32_t* S, int32_t* L) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int32_t b = lvl[i], sn = 1, sl = 0;
        for (int j = 0; j < nk[b]; j++) {
            int32_t k = kids[(size_t)b * 8 + j];
            if (k >= 0) { sn += S[k]; sl += L[k]; } else sl += 1;
        }
        S[b] = sn;
        L[b] = sl;
    }
}
// preorder index (P) and first leaf slot (LB) of every inner kid of a level's nodes
__global__ void k_preorder(const int32_t* __restrict__ lvl, int32_t m, const int32_t* __restrict__ kids,
                           const int32_t* __restrict__ nk, const int32_t* __restrict__ S,
                           const int32_t* __restrict__ L, int32_t* P, int32_t* LB) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int32_t b = lvl[i], on = P[b] + 1, ol = LB[b];
        for (int j = 0; j < nk[b]; j++) {
            int32_t k = kids[(size_t)b * 8 + j];
            if (k >= 0) { P[k] = on; LB[k] = ol; on += S[k]; ol += L[k]; } else ol += 1;
        }
    }
}
// the node of every wide root: child boxes (empty slots inverted), inner
// children by preorder index, leaves for now as RT_LEAF_BIT | leaf slot
__global__ void k_write_nodes(const int32_t* __restrict__ order, int32_t m, const int32_t* __restrict__ kids,
                              const int32_t* __restrict__ nk, const int32_t* __restrict__ P,
                              const int32_t* __restrict__ LB, const int32_t* __restrict__ L, const float* __restrict__ bbox,
                              const float* __restrict__ box, const int32_t* __restrict__ idx, float4* nodes,
                              int32_t* export_ch, int32_t* leaf_gid) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int32_t b = order[i], me = P[b], ol = LB[b];
        float f[56];
        for (int c = 0; c < 8; c++) {
            int32_t k = c < nk[b] ? kids[(size_t)b * 8 + c] : INT32_MIN;
            uint32_t ref;
            int32_t ex;
            const float* cb = nullptr;
            if (c >= nk[b]) {
                ref = RT_EMPTY_REF; ex = INT32_MIN;
            } else if (k >= 0) {
                ref = (uint32_t)P[k]; ex = P[k]; cb = bbox + (size_t)k * 6;
                ol += L[k];                                  // the inner kid's leaves come first
            } else {
                int32_t slot = ol++, prim = idx[-k - 1];
                leaf_gid[slot] = prim;
                ref = RT_LEAF_BIT | (uint32_t)slot; ex = -(slot + 1); cb = box + (size_t)prim * 6;
            }
            for (int a = 0; a < 3; a++) {
                f[a * 8 + c] = cb ? cb[a] : INFINITY;
                f[24 + a * 8 + c] = cb ? cb[3 + a] : -INFINITY;
            }
            f[48 + c] = __uint_as_float(ref);
            export_ch[(size_t)me * 8 + c] = ex;
        }
        float4* out = nodes + (size_t)me * 14;
        for (int q = 0; q < 14; q++) out[q] = make_float4(f[q * 4], f[q * 4 + 1], f[q * 4 + 2], f[q * 4 + 3]);
    }
}
// 4-wide nodes (7 float4: lower x, y, z and upper x, y, z planes of the 4
// children, then their references).  The leaves keep the 8-wide tree's leaf
// order, in which the primitive records are stored: a leaf kid's reference is
// its primitive's typed slot there (inv8: primitive → 8-wide leaf slot).
__global__ void k_write_nodes4(const int32_t* __restrict__ order, int32_t m, const int32_t* __restrict__ kids,
                               const int32_t* __restrict__ nk, const int32_t* __restrict__ P,
                               const float* __restrict__ bbox, const float* __restrict__ box,
                               const int32_t* __restrict__ idx, const int32_t* __restrict__ inv8,
                               const int32_t* __restrict__ scans, int32_t n, int64_t e0, int64_t e1, int64_t e2,
                               float4* nodes4) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        int32_t b = order[i], me = P[b];
        float f[28];
        for (int c = 0; c < 4; c++) {
            int32_t k = c < nk[b] ? kids[(size_t)b * 8 + c] : INT32_MIN;
            uint32_t ref;
            const float* cb = nullptr;
            if (c >= nk[b]) {
                ref = RT_EMPTY_REF;
            } else if (k >= 0) {
                ref = (uint32_t)P[k]; cb = bbox + (size_t)k * 6;
            } else {
                int32_t prim = idx[-k - 1], slot = inv8[prim];
                uint32_t t = prim < e0 ? RT_PRIM_TRI : prim < e1 ? RT_PRIM_QUAD : prim < e2 ? RT_PRIM_SPHERE : RT_PRIM_CONVEX;
                ref = RT_LEAF_BIT | (t << 28) | (uint32_t)scans[(size_t)t * n + slot];
                cb = box + (size_t)prim * 6;
            }
            for (int a = 0; a < 3; a++) {
                f[a * 4 + c] = cb ? cb[a] : INFINITY;
                f[12 + a * 4 + c] = cb ? cb[3 + a] : -INFINITY;
            }
            f[24 + c] = __uint_as_float(ref);
        }
        float4* out = nodes4 + (size_t)me * 7;
        for (int q = 0; q < 7; q++) out[q] = make_float4(f[q * 4], f[q * 4 + 1], f[q * 4 + 2], f[q * 4 + 3]);
    }
}
__global__ void k_invert(const int32_t* __restrict__ leaf_gid, int32_t n, int32_t* inv) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) inv[leaf_gid[i]] = i;
}
// leaf type of every slot: one flag array per type for the typed-slot scans
__global__ void k_leaf_types(const int32_t* __restrict__ leaf_gid, int32_t n, int64_t e0, int64_t e1, int64_t e2,
                             int32_t* flags) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int64_t g = leaf_gid[i];
        int t = g < e0 ? RT_PRIM_TRI : g < e1 ? RT_PRIM_QUAD : g < e2 ? RT_PRIM_SPHERE : RT_PRIM_CONVEX;
        for (int k = 0; k < 4; k++) flags[(size_t)k * n + i] = t == k;
    }
}
// leaf references: type in bits 28-30, the slot among leaves of that type
__global__ void k_fix_leaf_refs(float4* nodes, int64_t n_nodes, const int32_t* __restrict__ leaf_gid, int32_t n,
                                int64_t e0, int64_t e1, int64_t e2, const int32_t* __restrict__ scans) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_nodes * 8; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t* ch = reinterpret_cast<uint32_t*>(nodes + (size_t)(i / 8) * 14 + 12) + (i % 8);
        uint32_t v = *ch;
        if (v == RT_EMPTY_REF || !(v & RT_LEAF_BIT)) continue;
        int32_t slot = (int32_t)(v & ~RT_LEAF_BIT);
        int64_t g = leaf_gid[slot];
        uint32_t t = g < e0 ? RT_PRIM_TRI : g < e1 ? RT_PRIM_QUAD : g < e2 ? RT_PRIM_SPHERE : RT_PRIM_CONVEX;
        *ch = RT_LEAF_BIT | (t << 28) | (uint32_t)scans[(size_t)t * n + slot];
    }
}
// ── packed nodes: what the traversal reads (rt_trace.cu) ────────────────────
// From a tree in the reference layout (preorder, child references).  The scheme is
// that of Ylitie, Karras and Laine 2017 (octant slots, a base index and masks in
// place of child references); the slot choice, the header and the leaf records are
// this file's.  Every child gets a slot by octant (bit 0, 1, 2 of the slot: the
// upper side of x, y, z), so a ray finds its children roughly front to back as
// slot XOR octant without keeping distances; the inner children of a node become
// neighbours in slot order, so a node index, a slot mask and a population count
// name a child (a header instead of 8 references), and a visit's pending children
// are one 8-byte stack entry.  The leaves of a node are neighbours too, in their
// own copy of the triangle records (for other primitives only the reference), so a
// leaf's triangle is found from the header without a reference in between; the
// leaves' float boxes are a second array.
//
// Slots of one node's children, 4 bits per child: greedily the (child, free
// slot) pair with the largest projection of the child's offset from the node
// centre onto the slot's diagonal.
template <int W>
__device__ uint32_t octant_slots(const float* f, const uint32_t* ch) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int c = 0; c < W; c++) {
        if (ch[c] == RT_EMPTY_REF) continue;
        for (int a = 0; a < 3; a++) { lo[a] = fminf(lo[a], f[a * W + c]); hi[a] = fmaxf(hi[a], f[3 * W + a * W + c]); }
    }
    uint32_t slots = 0, free_slots = (1u << W) - 1u, todo = 0;
    for (int c = 0; c < W; c++) todo |= (ch[c] != RT_EMPTY_REF ? 1u : 0u) << c;
    while (todo) {
        float best = -INFINITY;
        int bc = __ffs(todo) - 1, bs = __ffs(free_slots) - 1;
        for (int c = 0; c < W; c++) {
            if (!((todo >> c) & 1u)) continue;
            float off[3];
            for (int a = 0; a < 3; a++) off[a] = (f[a * W + c] + f[3 * W + a * W + c]) - (lo[a] + hi[a]);
            for (int q = 0; q < W; q++) {
                if (!((free_slots >> q) & 1u)) continue;
                float v = ((q & 1) ? off[0] : -off[0]) + ((q & 2) ? off[1] : -off[1]);
                if (W == 8) v += (q & 4) ? off[2] : -off[2];
                if (v > best) { best = v; bc = c; bs = q; }
            }
        }
        slots |= (uint32_t)bs << (4 * bc);
        todo &= ~(1u << bc);
        free_slots &= ~(1u << bs);
    }
    return slots;
}
template <int W>
__device__ void load_ref_node(const float4* __restrict__ in, int64_t i, float* f, uint32_t* ch) {
    constexpr int F4 = W == 8 ? 14 : 7;
    const float4* N = in + (size_t)i * F4;
    for (int q = 0; q < F4; q++) {
        float4 v = N[q];
        f[q * 4] = v.x; f[q * 4 + 1] = v.y; f[q * 4 + 2] = v.z; f[q * 4 + 3] = v.w;
    }
    for (int c = 0; c < W; c++) ch[c] = __float_as_uint(f[6 * W + c]);
}
template <int W>
__global__ void k_pack_slots(const float4* __restrict__ in, int32_t n, uint32_t* slots, uint64_t* cnt) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float f[7 * W];
        uint32_t ch[W];
        load_ref_node<W>(in, i, f, ch);
        slots[i] = octant_slots<W>(f, ch);
        // inner children (low word) and leaves (high word) of the node
        uint64_t k = 0;
        for (int c = 0; c < W; c++)
            if (ch[c] != RT_EMPTY_REF) k += (ch[c] & RT_LEAF_BIT) ? 1ull << 32 : 1ull;
        cnt[i] = k;
    }
}
// slots of a node's inner children
template <int W>
__device__ uint32_t inner_slots(const uint32_t* ch, uint32_t slots) {
    uint32_t m = 0;
    for (int c = 0; c < W; c++)
        if (ch[c] != RT_EMPTY_REF && !(ch[c] & RT_LEAF_BIT)) m |= 1u << ((slots >> (4 * c)) & 7u);
    return m;
}
// packed index of every node: 1 + the inner children of the nodes before its
// parent + its rank among its siblings' slots (the root is 0)
template <int W>
__global__ void k_pack_index(const float4* __restrict__ in, int32_t n, const uint32_t* __restrict__ slots,
                             const uint64_t* __restrict__ base, int32_t* index) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t* ch = reinterpret_cast<const uint32_t*>(in + (size_t)i * (W == 8 ? 14 : 7) + (W == 8 ? 12 : 6));
        uint32_t r[W];
        for (int c = 0; c < W; c++) r[c] = ch[c];
        uint32_t im = inner_slots<W>(r, slots[i]);
        for (int c = 0; c < W; c++) {
            if (r[c] == RT_EMPTY_REF || (r[c] & RT_LEAF_BIT)) continue;
            uint32_t q = (slots[i] >> (4 * c)) & 7u;
            index[r[c]] = 1 + (int32_t)base[i] + __popc(im & ((1u << q) - 1u));
        }
        if (i == 0) index[0] = 0;
    }
}
// a leaf reference (RT_LEAF_BIT, type, typed index) as the hit record it yields
__device__ uint32_t leaf_hit_ref(const rtd::DevScene& S, uint32_t v) {
    uint32_t type = (v >> 28) & 3u, idx = v & 0x07FFFFFFu;
    float m = type == RT_PRIM_TRI ? S.tri[(size_t)idx * 3 + 2].z
            : type == RT_PRIM_QUAD ? S.quad[(size_t)idx * 5 + 4].y
            : type == RT_PRIM_SPHERE ? S.sphere[(size_t)idx * 2 + 1].y : S.cvx[(size_t)idx * 2].z;
    return RT_HIT_MAKE(v, S.mat_code[__float_as_int(m)]);
}
// the record of a leaf: a triangle's (v0, e1, e2, canonical id) with its
// reference in place of the material; of another primitive (-, -, (-, id, reference, -))
__device__ void write_leaf(const rtd::DevScene& S, uint32_t v, float4* rec) {
    uint32_t type = (v >> 28) & 3u, idx = v & 0x07FFFFFFu;
    float ref = __uint_as_float(leaf_hit_ref(S, v));
    if (type == RT_PRIM_TRI) {
        const float4* g = S.tri + (size_t)idx * 3;
        rec[0] = g[0];
        rec[1] = g[1];
        rec[2] = make_float4(g[2].x, g[2].y, ref, 0.f);
    } else {
        float gid = type == RT_PRIM_QUAD ? S.quad[(size_t)idx * 5 + 4].x
                  : type == RT_PRIM_SPHERE ? S.sphere[(size_t)idx * 2 + 1].x : S.cvx[(size_t)idx * 2 + 1].x;
        rec[0] = rec[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        rec[2] = make_float4(0.f, gid, ref, 0.f);
    }
}
// the packed node's header; its leaves go to `LS` (rec null: they are written already)
template <int W>
__device__ float4 pack_head(const rtd::DevScene& S, const float* f, const uint32_t* ch, uint32_t slots, uint64_t base,
                            rtd::LeafSet LS) {
    uint32_t lm = 0, first = (uint32_t)(base >> 32);
    for (int c = 0; c < W; c++)
        if (ch[c] != RT_EMPTY_REF && (ch[c] & RT_LEAF_BIT)) lm |= 1u << ((slots >> (4 * c)) & 7u);
    for (int c = 0; LS.rec && c < W; c++) {
        if (ch[c] == RT_EMPTY_REF || !(ch[c] & RT_LEAF_BIT)) continue;
        uint32_t q = (slots >> (4 * c)) & 7u;
        size_t k = first + __popc(lm & ((1u << q) - 1u));
        write_leaf(S, ch[c], const_cast<float4*>(LS.rec) + k * 3);
        float4* r = const_cast<float4*>(LS.box) + k * 2;
        r[0] = make_float4(f[c], f[W + c], f[2 * W + c], 0.f);
        r[1] = make_float4(f[3 * W + c], f[4 * W + c], f[5 * W + c], 0.f);
    }
    return make_float4(__uint_as_float(1u + (uint32_t)base), __uint_as_float(inner_slots<W>(ch, slots) | lm << 8),
                       __uint_as_float(first), 0.f);
}
// full nodes: RT_NODE_F4 (8-wide) or RT_NODE4_F4 (4-wide) float4
template <int W>
__global__ void k_pack_nodes(rtd::DevScene S, const float4* __restrict__ in, int32_t n,
                             const uint32_t* __restrict__ slots, const uint64_t* __restrict__ base,
                             const int32_t* __restrict__ index, float4* out, rtd::LeafSet LS) {
    constexpr int F4 = W == 8 ? RT_NODE_F4 : RT_NODE4_F4, BOX4 = W == 8 ? 12 : 6;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float f[7 * W], g[6 * W];
        uint32_t ch[W];
        load_ref_node<W>(in, i, f, ch);
        // slots without a child hold inverted boxes: their slab test fails
        for (int a = 0; a < 3; a++)
            for (int q = 0; q < W; q++) { g[a * W + q] = INFINITY; g[3 * W + a * W + q] = -INFINITY; }
        for (int c = 0; c < W; c++) {
            if (ch[c] == RT_EMPTY_REF) continue;
            int q = (slots[i] >> (4 * c)) & 7u;
            for (int a = 0; a < 3; a++) { g[a * W + q] = f[a * W + c]; g[3 * W + a * W + q] = f[3 * W + a * W + c]; }
        }
        float4* N = out + (size_t)index[i] * F4;
        for (int q = 0; q < BOX4; q++) N[q] = make_float4(g[q * 4], g[q * 4 + 1], g[q * 4 + 2], g[q * 4 + 3]);
        N[BOX4] = pack_head<W>(S, f, ch, slots[i], base[i], LS);
    }
}
// Quantised nodes (RT_QNODE_F4 float4): the child boxes as 8-bit offsets from
// the node's lower corner p in steps of s = 2^e per axis, rounded outward so
// that the real planes p + q·s contain the exact child box (Ylitie et al. 2017
// store child boxes this way; the rounding here is made conservative so the
// hits stay the brute-force ones).  Words: 0: p.x, p.y, p.z, (e_x + 127) << 23 |
// (e_y + 127) << 15 | (e_z + 127) << 7; 1-3: per axis the bytes q_lo, q_hi of
// slots 0-7 in turn; 4: header.
// A node whose extent needs a step beyond 2^60 sets *fail (steps are kept in
// [2^-60, 2^60], so with |1/d| in [2^-60, 2^60] every s/d is a normal float).
__global__ void k_pack_qnodes(rtd::DevScene S, const float4* __restrict__ nodes, int32_t n_nodes,
                              const uint32_t* __restrict__ slots, const uint64_t* __restrict__ base,
                              const int32_t* __restrict__ index, float4* qnodes, int* fail) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += gridDim.x * blockDim.x) {
        float f[56];
        uint32_t ch[8];
        load_ref_node<8>(nodes, i, f, ch);
        uint32_t valid = 0;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int c = 0; c < 8; c++) {
            if (ch[c] == RT_EMPTY_REF) continue;
            valid |= 1u << c;
            for (int a = 0; a < 3; a++) { lo[a] = fminf(lo[a], f[a * 8 + c]); hi[a] = fmaxf(hi[a], f[24 + a * 8 + c]); }
        }
        if (!valid) for (int a = 0; a < 3; a++) lo[a] = hi[a] = 0.0f;
        int e[3];
        bool flat[3];
        int e_any = -60;
        for (int a = 0; a < 3; a++) {
            float ext = __fsub_ru(hi[a], lo[a]);
            flat[a] = !(ext > 0.0f);
            if (flat[a]) continue;
            int ex;
            frexpf(ext / 255.0f, &ex);
            while (ex > -60 && ldexpf(255.0f, ex - 1) >= ext) ex--;
            while (ldexpf(255.0f, ex) < ext) ex++;
            e[a] = max(ex, -60);
            e_any = max(e_any, e[a]);
        }
        bool ok = true;
        for (int a = 0; a < 3; a++) {
            if (flat[a]) e[a] = e_any;
            if (e[a] > 60) ok = false;
        }
        if (!ok) { atomicExch(fail, 1); continue; }
        uint32_t w[3][4];
        for (int a = 0; a < 3; a++) {
            float sa = ldexpf(1.0f, e[a]);
            w[a][0] = w[a][1] = w[a][2] = w[a][3] = 0x00FF00FFu;   // slots without a child: lo 255, hi 0
            for (int c = 0; c < 8; c++) {
                if (!((valid >> c) & 1u)) continue;
                uint32_t q = (slots[i] >> (4 * c)) & 7u, sh = 16 * (q & 1u);
                float dl = __fsub_rd(f[a * 8 + c], lo[a]), dh = __fsub_ru(f[24 + a * 8 + c], lo[a]);
                uint32_t ql = (uint32_t)fminf(fmaxf(floorf(dl / sa), 0.0f), 255.0f);
                uint32_t qh = (uint32_t)fminf(fmaxf(ceilf(dh / sa), 0.0f), 255.0f);
                w[a][q >> 1] = (w[a][q >> 1] & ~(0xFFFFu << sh)) | (ql | qh << 8) << sh;
            }
        }
        uint32_t meta = (uint32_t)(e[0] + 127) << 23 | (uint32_t)(e[1] + 127) << 15 | (uint32_t)(e[2] + 127) << 7;
        float4* Q = qnodes + (size_t)index[i] * RT_QNODE_F4;
        Q[0] = make_float4(lo[0], lo[1], lo[2], __uint_as_float(meta));
        for (int a = 0; a < 3; a++)
            Q[1 + a] = make_float4(__uint_as_float(w[a][0]), __uint_as_float(w[a][1]), __uint_as_float(w[a][2]),
                                   __uint_as_float(w[a][3]));
        Q[4] = pack_head<8>(S, f, ch, slots[i], base[i], rtd::LeafSet{nullptr, nullptr});
    }
}

}  // namespace

namespace rth {

// the device collapse: bl / br / bbox / box / idx and root are the device
// arrays of the binary tree
static cudaError_t collapse_wide(const int32_t* bl, const int32_t* br, const float* bbox, const float* box,
                                 const int32_t* idx, int32_t root, int32_t n, int sms, cudaStream_t st, WideOut* W) {
    const int32_t nn = n - 1;
    int32_t *kids = nullptr, *nk = nullptr, *order = nullptr, *cnt = nullptr, *pos = nullptr;
    int32_t *S = nullptr, *L = nullptr, *P = nullptr, *LB = nullptr, *leaf_gid = nullptr, *flags = nullptr, *scans = nullptr;
    void* tmp = nullptr;
    size_t tmp_bytes = 0;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) { if (e == cudaSuccess && r != cudaSuccess) e = r; return e == cudaSuccess; };
    auto scan = [&](const int32_t* in, int32_t* out, int32_t m) {
        size_t need = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, need, in, out, m, st);
        if (need > tmp_bytes) { ok(cudaErrorMemoryAllocation); return; }   // m ≤ n: never
        ok(cub::DeviceScan::ExclusiveSum(tmp, need, in, out, m, st));
    };
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, cnt, pos, n, st);
    Arena A;
    A.part(&kids, (size_t)nn * 8 * 4); A.part(&nk, (size_t)nn * 4);
    A.part(&order, ((size_t)nn + 1) * 4); A.part(&cnt, ((size_t)nn + 1) * 4); A.part(&pos, ((size_t)nn + 1) * 4);
    A.part(&S, (size_t)nn * 4); A.part(&L, (size_t)nn * 4); A.part(&P, (size_t)nn * 4); A.part(&LB, (size_t)nn * 4);
    A.part(&leaf_gid, (size_t)n * 4); A.part(&flags, (size_t)n * 16); A.part(&scans, (size_t)n * 16);
    A.part(&tmp, tmp_bytes);
    ok(A.open());
    int grid = sms * 8;
    std::vector<int32_t> lvl_off;
    // the wide nodes of one width: each binary node's opening, the wide roots
    // level by level (in `order`), subtree sizes bottom-up and preorder indices
    // top-down; returns the node count (0 on an error) and the depth in *depth
    auto plan = [&](int width, int32_t* depth) -> int32_t {
        lvl_off.assign({0, 1});
        if (e != cudaSuccess) return 0;
        k_wide_kids<<<grid, 256, 0, st>>>(bl, br, bbox, nn, kids, nk, width);
        ok(cudaMemcpyAsync(order, &root, 4, cudaMemcpyHostToDevice, st));
        while (e == cudaSuccess) {
            int32_t off = lvl_off[lvl_off.size() - 2], m = lvl_off.back() - off;
            k_count_inner<<<std::max(1, std::min((m + 255) / 256, grid)), 256, 0, st>>>(order + off, m, kids, nk, cnt);
            scan(cnt, pos, m);
            int32_t tail[2] = {0, 0};
            ok(cudaMemcpyAsync(&tail[0], pos + m - 1, 4, cudaMemcpyDeviceToHost, st));
            ok(cudaMemcpyAsync(&tail[1], cnt + m - 1, 4, cudaMemcpyDeviceToHost, st));
            ok(cudaStreamSynchronize(st));
            int32_t nxt = tail[0] + tail[1];
            if (nxt == 0 || e != cudaSuccess) break;
            if (lvl_off.back() + nxt > nn) { e = cudaErrorUnknown; break; }
            k_next_level<<<std::max(1, std::min((m + 255) / 256, grid)), 256, 0, st>>>(order + off, m, kids, nk, pos,
                                                                                   order + lvl_off.back());
            lvl_off.push_back(lvl_off.back() + nxt);
        }
        const int nlev = (int)lvl_off.size() - 1;
        if (e != cudaSuccess) return 0;
        for (int l = nlev - 1; l >= 0; l--) {
            int32_t m = lvl_off[l + 1] - lvl_off[l];
            k_subtree_sizes<<<std::max(1, std::min((m + 255) / 256, grid)), 256, 0, st>>>(order + lvl_off[l], m, kids,
                                                                                       nk, S, L);
        }
        ok(cudaMemsetAsync(P + root, 0, 4, st));
        ok(cudaMemsetAsync(LB + root, 0, 4, st));
        for (int l = 0; l < nlev; l++) {
            int32_t m = lvl_off[l + 1] - lvl_off[l];
            k_preorder<<<std::max(1, std::min((m + 255) / 256, grid)), 256, 0, st>>>(order + lvl_off[l], m, kids, nk,
                                                                                  S, L, P, LB);
        }
        int32_t total = 0;
        ok(cudaMemcpyAsync(&total, S + root, 4, cudaMemcpyDeviceToHost, st));
        ok(cudaStreamSynchronize(st));
        if (e == cudaSuccess && total != lvl_off.back()) e = cudaErrorUnknown;   // every wide root counted once
        *depth = nlev - 1;
        return e == cudaSuccess ? total : 0;
    };
    if (e == cudaSuccess) W->n_nodes = plan(8, &W->max_depth);
    if (e == cudaSuccess) {
        ok(cudaMalloc(&W->nodes, (size_t)W->n_nodes * 14 * 16));
        ok(cudaMalloc(&W->export_ch, (size_t)W->n_nodes * 8 * 4));
    }
    if (e == cudaSuccess) {
        int32_t m = lvl_off.back();
        k_write_nodes<<<std::max(1, std::min((m + 127) / 128, grid)), 128, 0, st>>>(
            order, m, kids, nk, P, LB, L, bbox, box, idx, W->nodes, W->export_ch, leaf_gid);
        k_leaf_types<<<grid, 256, 0, st>>>(leaf_gid, n, W->type_end[0], W->type_end[1], W->type_end[2], flags);
        for (int t = 0; t < 4; t++) scan(flags + (size_t)t * n, scans + (size_t)t * n, n);
        k_fix_leaf_refs<<<grid, 256, 0, st>>>(W->nodes, W->n_nodes, leaf_gid, n, W->type_end[0], W->type_end[1],
                                             W->type_end[2], scans);
        ok(cudaMemcpyAsync(W->leaf_gids_h, leaf_gid, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
        ok(cudaStreamSynchronize(st));
        ok(cudaGetLastError());
    }
    // the 4-wide tree over the same binary tree (RT_NODES_WIDE4), its leaves
    // referring to the primitive records in the 8-wide leaf order
    if (e == cudaSuccess) {
        int32_t* inv8 = cnt;                         // n + 1 ≥ n entries, free now
        W->n_nodes4 = plan(4, &W->max_depth4);
        if (e == cudaSuccess) ok(cudaMalloc(&W->nodes4, (size_t)W->n_nodes4 * 7 * 16));
        if (e == cudaSuccess) {
            k_invert<<<grid, 256, 0, st>>>(leaf_gid, n, inv8);
            int32_t m = lvl_off.back();
            k_write_nodes4<<<std::max(1, std::min((m + 127) / 128, grid)), 128, 0, st>>>(
                order, m, kids, nk, P, bbox, box, idx, inv8, scans, n, W->type_end[0], W->type_end[1], W->type_end[2],
                W->nodes4);
            ok(cudaStreamSynchronize(st));
            ok(cudaGetLastError());
        }
    }
    if (e != cudaSuccess) {
        void* outs[] = {W->nodes, W->export_ch, W->nodes4};
        for (void* p : outs) if (p) cudaFree(p);
        W->nodes = W->nodes4 = nullptr;
        W->export_ch = nullptr;
    }
    return e;
}

// Packs the n nodes of a reference-layout tree (width 8 or 4) with n_leaves
// leaves: *out gets the packed nodes, *lout the leaves, and for width 8
// *qout the quantised nodes (left null when an extent is beyond their range).  Needs the scene's primitive records and
// material codes on the device.
cudaError_t pack_nodes(const rtd::DevScene& S, const float4* in, int64_t n_nodes, int64_t n_leaves, int width,
                       float4** out, rtd::LeafSet* lout, float4** qout, int sms, cudaStream_t st) {
    const int32_t n = (int32_t)n_nodes;
    uint32_t* slots = nullptr;
    uint64_t *cnt = nullptr, *base = nullptr;
    int32_t* index = nullptr;
    int* fail = nullptr;
    void* tmp = nullptr;
    size_t need = 0;
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) { if (e == cudaSuccess && r != cudaSuccess) e = r; return e == cudaSuccess; };
    cub::DeviceScan::ExclusiveSum(nullptr, need, cnt, base, n, st);
    Arena A;
    A.part(&slots, (size_t)n * 4); A.part(&cnt, (size_t)n * 8); A.part(&base, (size_t)n * 8);
    A.part(&index, (size_t)n * 4); A.part(&fail, 4); A.part(&tmp, need);
    ok(A.open());
    ok(cudaMalloc((void**)&lout->rec, (size_t)n_leaves * 48)); ok(cudaMalloc((void**)&lout->box, (size_t)n_leaves * 32));
    ok(cudaMalloc(out, (size_t)n * (width == 8 ? RT_NODE_F4 : RT_NODE4_F4) * 16));
    if (qout) ok(cudaMalloc(qout, (size_t)n * RT_QNODE_F4 * 16));
    if (e == cudaSuccess) {
        const int g = std::max(1, std::min((n + 127) / 128, sms * 8));
        ok(cudaMemsetAsync(fail, 0, 4, st));
        if (width == 8) k_pack_slots<8><<<g, 128, 0, st>>>(in, n, slots, cnt);
        else            k_pack_slots<4><<<g, 128, 0, st>>>(in, n, slots, cnt);
        ok(cub::DeviceScan::ExclusiveSum(tmp, need, cnt, base, n, st));
        if (width == 8) {
            k_pack_index<8><<<g, 128, 0, st>>>(in, n, slots, base, index);
            k_pack_nodes<8><<<g, 128, 0, st>>>(S, in, n, slots, base, index, *out, *lout);
        } else {
            k_pack_index<4><<<g, 128, 0, st>>>(in, n, slots, base, index);
            k_pack_nodes<4><<<g, 128, 0, st>>>(S, in, n, slots, base, index, *out, *lout);
        }
        if (qout) k_pack_qnodes<<<g, 128, 0, st>>>(S, in, n, slots, base, index, *qout, fail);
        int hfail = 0;
        ok(cudaMemcpyAsync(&hfail, fail, 4, cudaMemcpyDeviceToHost, st));
        ok(cudaStreamSynchronize(st));
        ok(cudaGetLastError());
        if (e == cudaSuccess && hfail && qout) { cudaFree(*qout); *qout = nullptr; }
    }
    if (e != cudaSuccess) {
        if (*out) cudaFree(*out);
        if (lout->rec) cudaFree((void*)lout->rec);
        if (lout->box) cudaFree((void*)lout->box);
        *out = nullptr;
        *lout = rtd::LeafSet{nullptr, nullptr};
        if (qout && *qout) { cudaFree(*qout); *qout = nullptr; }
    }
    return e;
}

void launch_tri_records(const int32_t* order, int32_t n, const RawTris& T, float4* tri, float4* nrm, float4* uv,
                        float4* tan, int sms, cudaStream_t st) {
    k_tri_records<<<std::max(1, std::min((n + 255) / 256, sms * 8)), 256, 0, st>>>(order, n, T, tri, nrm, uv, tan);
}

// Build the binary SAH tree of n primitive boxes on the device: those of the
// first n_tris from the triangles tri_v (device, 9 floats each; their union goes
// to tri_bounds), the others from boxes_h (host, 6 floats each);
// idx (n), bl / br (n − 1 child refs: ≥ 0 node, < 0 leaf −(pos + 1)) and bbox ((n − 1) × 6) are written on the host.  Returns 0 or a CUDA error.
int gpu_build_binary(const float* boxes_h, const float* tri_v, int32_t n_tris, float* tri_bounds, int32_t n,
                     int32_t* idx_h, int32_t* bl_h, int32_t* br_h, float* bbox_h, int32_t* root_h, int sms,
                     cudaStream_t st, WideOut* wide) {
    float *box = nullptr, *cen = nullptr, *bbox = nullptr;
    int32_t *idx = nullptr, *tmp = nullptr, *bl = nullptr, *br = nullptr, *root = nullptr, *cnt = nullptr;
    int32_t *stats = nullptr, *mids = nullptr, *axes = nullptr;
    uint8_t* keys = nullptr;
    Seg *nxt = nullptr, *small = nullptr;
    int32_t *lvl = nullptr, *hist = nullptr;
    int32_t nn = std::max(n - 1, 1);
    cudaError_t e = cudaSuccess;
    auto ok = [&](cudaError_t r) { if (e == cudaSuccess && r != cudaSuccess) e = r; return e == cudaSuccess; };
    size_t max_chunks = (size_t)n / CHUNK + (size_t)n / SMALL + 2;
    size_t max_segs = (size_t)n / SMALL + 2;
    Arena A;
    A.part(&box, (size_t)n * 24); A.part(&cen, (size_t)n * 12); A.part(&bbox, (size_t)nn * 24);
    A.part(&idx, (size_t)n * 4); A.part(&tmp, (size_t)n * 4);
    A.part(&bl, (size_t)nn * 4); A.part(&br, (size_t)nn * 4); A.part(&root, 4);
    A.part(&keys, (size_t)n);
    A.part(&stats, max_segs * ST_WORDS * 4); A.part(&mids, max_segs * 4); A.part(&axes, max_segs * 4);
    A.part(&lvl, (5 * max_segs + 1 + 2 * max_chunks) * 4); A.part(&hist, max_chunks * NB * 4);
    A.part(&cnt, 16 + max_segs * sizeof(Seg));
    A.part(&small, ((size_t)n / 2 + 2) * sizeof(Seg));
    ok(A.open());
    if (e == cudaSuccess) {
        if (n > n_tris)
            ok(cudaMemcpyAsync(box + (size_t)n_tris * 6, boxes_h, (size_t)(n - n_tris) * 24, cudaMemcpyHostToDevice, st));
        if (n_tris > 0) {
            const int g = std::max(1, std::min((n_tris + 255) / 256, sms * 8));
            k_tri_boxes<<<g, 256, 0, st>>>(tri_v, n_tris, box);
            k_stats_init<<<1, 256, 0, st>>>(stats, 1);
            k_union_boxes<<<g, 256, 0, st>>>(box, n_tris, stats);
            int32_t u[6];
            ok(cudaMemcpyAsync(u, stats, sizeof(u), cudaMemcpyDeviceToHost, st));
            ok(cudaStreamSynchronize(st));
            for (int k = 0; k < 6; k++) {
                int32_t b = u[k] >= 0 ? u[k] : u[k] ^ 0x7FFFFFFF;
                memcpy(tri_bounds + k, &b, 4);
            }
        }
        k_centroids<<<sms * 8, 256, 0, st>>>(box, n, cen, idx);
        ok(cudaMemsetAsync(cnt, 0, 8, st));
        ok(cudaMemsetAsync(root, 0, 4, st));
    }
    // the root: large, small or a single leaf
    std::vector<Seg> level;
    int32_t n_small = 0;
    Seg r0{0, n, -1, -1};
    if (n == 1) {
        int32_t leaf = -1;
        ok(cudaMemcpyAsync(root, &leaf, 4, cudaMemcpyHostToDevice, st));
    } else if (n < SMALL) {
        ok(cudaMemcpyAsync(small, &r0, sizeof(Seg), cudaMemcpyHostToDevice, st));
        n_small = 1;
    } else {
        level.push_back(r0);
    }
    // a level's nodes, each node's first chunk and the chunks' nodes and starts
    // go to the device in one copy; its children come back in one
    nxt = (Seg*)(cnt + 4);
    std::vector<int32_t> up, down;
    while (e == cudaSuccess && !level.empty()) {
        int32_t ns = (int32_t)level.size(), nch = 0;
        up.resize((size_t)ns * 5 + 1);
        memcpy(up.data(), level.data(), (size_t)ns * sizeof(Seg));
        for (int32_t s = 0; s < ns; s++) { up[(size_t)ns * 4 + s] = nch; nch += (level[s].hi - level[s].lo + CHUNK - 1) / CHUNK; }
        up[(size_t)ns * 5] = nch;
        up.resize((size_t)ns * 5 + 1 + 2 * (size_t)nch);
        int32_t* q = up.data() + (size_t)ns * 5 + 1;
        for (int32_t s = 0; s < ns; s++)
            for (int32_t lo = level[s].lo; lo < level[s].hi; lo += CHUNK, q++) { q[0] = s; q[nch] = lo; }
        ok(cudaMemcpyAsync(lvl, up.data(), up.size() * 4, cudaMemcpyHostToDevice, st));
        const Seg* cur = (const Seg*)lvl;
        const int32_t *first = lvl + (size_t)ns * 4, *chunk_seg = first + ns + 1, *chunk_lo = chunk_seg + nch;
        int grid = std::min(nch, sms * 16);
        k_stats_init<<<std::min((ns * ST_WORDS + 255) / 256, sms * 8), 256, 0, st>>>(stats, ns);
        k_stats_bounds<<<grid, 256, 0, st>>>(cur, chunk_seg, chunk_lo, nch, idx, box, cen, stats);
        k_stats_bins<<<grid, 256, 0, st>>>(cur, chunk_seg, chunk_lo, nch, idx, box, cen, stats);
        k_split<<<(ns + 127) / 128, 128, 0, st>>>(cur, ns, stats, mids, axes, bl, br, root, bbox);
        k_keys<<<grid, 256, 0, st>>>(cur, chunk_seg, chunk_lo, nch, idx, cen, stats, axes, keys, hist);
        k_offsets<<<ns, NB * 32, 0, st>>>(cur, first, nch, hist);
        k_scatter<<<grid, SCATTER_WARPS * 32, 0, st>>>(cur, chunk_seg, chunk_lo, nch, hist, keys, idx, tmp);
        k_copy_back<<<grid, 256, 0, st>>>(cur, chunk_seg, chunk_lo, nch, tmp, idx);
        ok(cudaMemsetAsync(cnt, 0, 8, st));
        LevelOut out{nxt, cnt, small + n_small, cnt + 1};
        k_children<<<(ns + 127) / 128, 128, 0, st>>>(cur, ns, mids, box, idx, bl, br, root, bbox, out);
        down.resize(4 + std::min(2 * (size_t)ns, max_segs) * 4);
        ok(cudaMemcpyAsync(down.data(), cnt, down.size() * 4, cudaMemcpyDeviceToHost, st));
        ok(cudaStreamSynchronize(st));
        if (e != cudaSuccess) break;
        n_small += down[1];
        level.resize(down[0]);
        memcpy(level.data(), down.data() + 4, (size_t)down[0] * sizeof(Seg));
    }
    if (e == cudaSuccess && n_small > 0)
    {
        const size_t sm = sizeof(SmallWarp) * SMALL_WARPS;
        ok(cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        k_small<<<std::min((n_small + SMALL_WARPS - 1) / SMALL_WARPS, sms * 8), SMALL_WARPS * 32, sm, st>>>(
            small, n_small, box, cen, idx, bl, br, root, bbox);
    }
    ok(cudaGetLastError());
    if (e == cudaSuccess && wide) {
        // the collapse on the device; the host gets the leaf order, not the tree
        int32_t rt = 0;
        ok(cudaMemcpyAsync(&rt, root, 4, cudaMemcpyDeviceToHost, st));
        ok(cudaStreamSynchronize(st));
        if (e == cudaSuccess) {
            if (rt < 0 || n < 2) e = cudaErrorInvalidValue;       // one primitive: the host builds that node
            else ok(collapse_wide(bl, br, bbox, box, idx, rt, n, sms, st, wide));
        }
        if (root_h) *root_h = rt;
    } else if (e == cudaSuccess) {
        ok(cudaMemcpyAsync(idx_h, idx, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
        if (n > 1) {
            ok(cudaMemcpyAsync(bl_h, bl, (size_t)(n - 1) * 4, cudaMemcpyDeviceToHost, st));
            ok(cudaMemcpyAsync(br_h, br, (size_t)(n - 1) * 4, cudaMemcpyDeviceToHost, st));
            ok(cudaMemcpyAsync(bbox_h, bbox, (size_t)(n - 1) * 24, cudaMemcpyDeviceToHost, st));
        }
        ok(cudaMemcpyAsync(root_h, root, 4, cudaMemcpyDeviceToHost, st));
        ok(cudaStreamSynchronize(st));
    }
    return (int)e;
}

}  // namespace rth
