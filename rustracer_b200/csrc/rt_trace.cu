// rt_trace.cu — 8-wide BVH traversal kernels (closest hit, any hit).
//
// Compiled with --fmad=false: the reference (Rust) never fuses a*b+c, and the
// hit ids / t values must be bit-identical to that arithmetic, so no FFMA may
// appear in the primitive tests and the leaf-box test.  The node tests, which only
// have to be conservative, use explicit FMAs: one per plane.
//
// Traversal (replaces BvhTree::hit_index, src/bvh.rs:229-288, and the AVX2
// slab test :326-364): one ray per lane in persistent warps; lanes that finish
// pull new rays as soon as enough of the warp is idle (lane refill), which keeps
// SIMD lanes busy across very uneven ray costs.
// Per visited node the thread tests all 8 child boxes, intersects the hit leaves
// at once (closest t, ties → smaller canonical id) and is left with a mask of
// hit inner children.  The children of a node are neighbours in memory and sit
// in slots by octant (octant_slots in rt_build.cu), so that mask and the index of
// the first child are the whole to-do list of the visit (a "group", 8 bytes):
// the next child is the slot nearest along the ray's octant, no distances are
// kept or sorted, and a visit pushes at most one stack entry (octant slots and
// stack entries of a first child and its pending slots: Ylitie, Karras and Laine,
// Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs, 2017).
#include <algorithm>

#include <cub/block/block_scan.cuh>

#include "rt_internal.h"
#include "rt_media.cuh"

using namespace rtd;

namespace {

struct Best { float t, b1, b2; uint32_t ref, gid; };

RT_D uint32_t f2u(float f) { return __float_as_uint(f); }

// A convex solid (convex_hit, diamond.rs:202-253): the interval inside every
// half-space, the entry for outside rays, the exit for rays inside; *plane is the
// crossing plane.  One ray by the whole warp: a brilliant has 97 planes and a
// step cut up to several hundred, one lane's serial loop over them idles the
// other 31, and the loop's result — the entry is the largest crossing of the
// planes facing the ray, the exit the smallest of the others, the first plane of
// equal ones — does not depend on the order.  Lane l takes planes l, l + 32, …; a
// −0 crossing counts as 0 in the comparison, as it does there.  Every lane calls
// it with the same arguments; all get the result.
RT_D uint32_t order_key(float t) {                  // monotone in t
    uint32_t u = __float_as_uint(t + 0.0f);
    return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
RT_D bool warp_convex(const float4* pl, int n, float3 o, float3 d, float tmin, float tmax, float* t_out, int* plane) {
    const uint32_t FULL = 0xFFFFFFFFu;
    float te = tmin, tx = tmax;
    int ie = -1, ix = -1;
    bool out = false;
    for (int i = threadIdx.x & 31u; i < n; i += 32) {
        float4 q = __ldg(pl + i);
        float nd = q.x * d.x + q.y * d.y + q.z * d.z;
        float no = q.x * o.x + q.y * o.y + q.z * o.z;
        float tf = (q.w - no) / nd;
        if (fabsf(nd) < 1e-8f) out = out || no > q.w;
        else if (nd < 0.0f) { if (tf > te) { te = tf; ie = i; } }
        else if (tf < tx || (ix < 0 && tf == tx)) { tx = tf; ix = i; }
    }
    if (__any_sync(FULL, out)) return false;
    // the entry: the largest key, then its first plane (none: t_min); the exit likewise
    uint32_t ke = ie >= 0 ? order_key(te) : 0u, me = __reduce_max_sync(FULL, ke);
    uint32_t pe = __reduce_min_sync(FULL, ie >= 0 && ke == me ? (uint32_t)ie : 0xFFFFFFFFu);
    uint32_t kx = ix >= 0 ? order_key(tx) : 0xFFFFFFFFu, mx = __reduce_min_sync(FULL, kx);
    uint32_t px = __reduce_min_sync(FULL, ix >= 0 && kx == mx ? (uint32_t)ix : 0xFFFFFFFFu);
    const bool entry = pe != 0xFFFFFFFFu, exit = px != 0xFFFFFFFFu;
    float t_enter = tmin, t_exit = tmax;
    if (entry) t_enter = __shfl_sync(FULL, te, __ffs(__ballot_sync(FULL, ie == (int)pe)) - 1);
    if (exit) t_exit = __shfl_sync(FULL, tx, __ffs(__ballot_sync(FULL, ix == (int)px)) - 1);
    if (t_enter > t_exit) return false;
    if (t_enter == t_exit && t_enter < tmax) return false;
    if (entry) { *t_out = t_enter; *plane = (int)pe; return true; }
    if (!exit || t_exit > tmax) return false;
    *t_out = t_exit; *plane = (int)px;
    return true;
}

// three-input min / max (sm_100)
RT_D float fmax3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
RT_D float fmin3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Per-ray slab constants.  Fast path (every |1/d| in [2^-60, 2^60], o/d finite,
// t_min ≥ 0): the near and far planes of each axis are chosen once per ray from
// the sign of the direction, and a plane distance is one FMA, b·inv + c with
// c = −o·inv moved outward by 2^-22·|o·inv| (more than the rounding of o·inv):
// a near distance is then at most the exact one and a far distance at least
// the exact one, but for the 3 relative roundings of inv and the FMA, which
// the exit widened by 2^-15 covers many times over.  So the culling is
// conservative and any layout returns the brute-force answer.
// General path (all other rays): both planes with min/max, a NaN slab (ray
// lying in a face plane) spanning the whole line, and the exit widened.
struct RayC {
    float3 o, inv, cn, cf;
    int nx, ny, nz;          // float4 offsets of the near-plane arrays in a full node
    uint32_t ord;            // per slot bit 2, 1, 0 (bytes 0, 1, 2): the slots nearer along the ray
    bool general;
};
constexpr float EXIT_WIDEN = 1.000031471252441f;      // 1 + 2^-15 + 2^-20

RT_D bool inv_in_range(float x) {
    float a = fabsf(x);
    return a >= 8.673617379884035e-19f && a <= 1.152921504606846976e18f;   // 2^-60 .. 2^60
}
RT_D void axis_consts(float o, float inv, float* cn, float* cf) {
    float oi = o * inv, m = fabsf(oi) * 2.384185791015625e-07f;           // 2^-22
    *cn = __fsub_rd(-oi, m);
    *cf = __fadd_ru(-oi, m);
}

RT_D RayC make_rayc(float3 o, float3 d, float tmin) {
    RayC r;
    r.o = o;
    r.inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
    axis_consts(o.x, r.inv.x, &r.cn.x, &r.cf.x);
    axis_consts(o.y, r.inv.y, &r.cn.y, &r.cf.y);
    axis_consts(o.z, r.inv.z, &r.cn.z, &r.cf.z);
    r.general = !(tmin >= 0.0f) || !inv_in_range(r.inv.x) || !inv_in_range(r.inv.y) || !inv_in_range(r.inv.z) ||
                !isfinite(r.cn.x + r.cn.y + r.cn.z);
    bool sx = signbit(r.inv.x), sy = signbit(r.inv.y), sz = signbit(r.inv.z);
    r.nx = sx ? 6 : 0;
    r.ny = sy ? 8 : 2;
    r.nz = sz ? 10 : 4;
    // slot bit 0, 1, 2 set = the child lies on the upper side of x, y, z
    r.ord = (sz ? 0xF0u : 0x0Fu) | (sy ? 0xCC00u : 0x3300u) | (sx ? 0xAA0000u : 0x550000u);
    return r;
}

// Header of a node: the index of its first inner child, the slots of its inner
// children (bits 0-7) and of its leaves (bits 8-15), and the index of its first
// leaf record; the children of a node and its leaves follow one another in slot
// order.
struct NodeHead { uint32_t child, masks, leaf; };
RT_D NodeHead load_head(const float4* p) {
    uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    return NodeHead{v.x, v.y, v.z};
}

__device__ __noinline__ uint32_t node_test_general(const float4* N, float3 o, float3 inv, float tmin, float tmax) {
    uint32_t mask = 0;
    float4 q[12];
#pragma unroll
    for (int i = 0; i < 12; i++) q[i] = __ldg(N + i);
    const float* f = reinterpret_cast<const float*>(q);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        float dax = (f[0 + c] - o.x) * inv.x, dbx = (f[24 + c] - o.x) * inv.x;
        float day = (f[8 + c] - o.y) * inv.y, dby = (f[32 + c] - o.y) * inv.y;
        float daz = (f[16 + c] - o.z) * inv.z, dbz = (f[40 + c] - o.z) * inv.z;
        float lx = fminf(dax, dbx), hx = fmaxf(dax, dbx);
        float ly = fminf(day, dby), hy = fmaxf(day, dby);
        float lz = fminf(daz, dbz), hz = fmaxf(daz, dbz);
        if (isnan(dax) || isnan(dbx)) { lx = -INFINITY; hx = INFINITY; }
        if (isnan(day) || isnan(dby)) { ly = -INFINITY; hy = INFINITY; }
        if (isnan(daz) || isnan(dbz)) { lz = -INFINITY; hz = INFINITY; }
        float t0 = fmaxf(fmaxf(fmaxf(tmin, lx), ly), lz);
        float t1 = fminf(fminf(fminf(tmax, hx), hy), hz);
        float t1w = t1 + fabsf(t1) * (EXIT_WIDEN - 1.0f);
        if (t0 <= t1w) mask |= 1u << c;
    }
    return mask;
}

// Slots of node `ni` whose box meets [tmin, tmax] along the ray (slots without
// a child may be among them: the header's masks clear those).  The sign of
// exit·widen − entry is shifted into the mask (a funnel shift per child)
// instead of a compare and a select.
RT_D uint32_t node_test(const DevScene& S, uint32_t ni, const RayC& R, float tmin, float tmax, NodeHead& h) {
    const float4* N = S.nodes + (size_t)ni * RT_NODE_F4;
    h = load_head(N + 12);
    if (R.general) return node_test_general(N, R.o, R.inv, tmin, tmax);
    float4 q[12];
    q[0] = __ldg(N + R.nx); q[1] = __ldg(N + R.nx + 1);
    q[2] = __ldg(N + R.ny); q[3] = __ldg(N + R.ny + 1);
    q[4] = __ldg(N + R.nz); q[5] = __ldg(N + R.nz + 1);
    q[6] = __ldg(N + 6 - R.nx); q[7] = __ldg(N + 7 - R.nx);
    q[8] = __ldg(N + 10 - R.ny); q[9] = __ldg(N + 11 - R.ny);
    q[10] = __ldg(N + 14 - R.nz); q[11] = __ldg(N + 15 - R.nz);
    const float* f = reinterpret_cast<const float*>(q);
    uint32_t miss = 0;
#pragma unroll
    for (int c = 7; c >= 0; c--) {
        float nx = __fmaf_rn(f[0 + c], R.inv.x, R.cn.x), fx = __fmaf_rn(f[24 + c], R.inv.x, R.cf.x);
        float ny = __fmaf_rn(f[8 + c], R.inv.y, R.cn.y), fy = __fmaf_rn(f[32 + c], R.inv.y, R.cf.y);
        float nz = __fmaf_rn(f[16 + c], R.inv.z, R.cn.z), fz = __fmaf_rn(f[40 + c], R.inv.z, R.cf.z);
        float t0 = fmax3f(fmaxf(tmin, nx), ny, nz);
        float t1 = fmin3f(fminf(tmax, fx), fy, fz);
        miss = __funnelshift_l(__float_as_uint(__fmaf_rn(t1, EXIT_WIDEN, -t0)), miss, 1);
    }
    return ~miss;
}

// ── quantised nodes (5 float4: see k_pack_qnodes in rt_build.cu) ─────────────
// Child planes are the real numbers p + q·s (s = 2^e per axis), which contain
// the exact child boxes.  Per ray and node S = s/d is exact, and with the ray's
// slab constants (c moved outward by more than the rounding of o/d)
// A = fma(p, 1/d, c), rounded down for the near planes and up for the far ones,
// bounds (p − o)/d.  The byte q enters as the float 2^15 + q (one byte permute,
// its unit 2^8 above the last mantissa bit), with 2^15·S taken off A rounded the
// same way: that loses at most 2^-8 steps (2^23 + q would lose a whole one), so
// q·S + A stays on the conservative side but for the last FMA's own rounding,
// which the widened exit covers.  The kernel issues in 63 % of the cycles on the
// first bounce and 54 % later, at 13 to 16 lanes of 32 and 4 long-scoreboard stalls
// per issue: half instructions, half the wait for the next node.  Packed two-wide
// FMAs save 14 % of the instructions and lose it again to the register pairs their
// constants need (spills; icosphere extend 50.2 against 49.7 ms).
RT_D float qbyte(uint32_t w, uint32_t sel) { return __uint_as_float(__byte_perm(w, 0x47000000u, sel)); }

__device__ __noinline__ uint32_t qnode_test_general(const float4* N, float3 o, float3 inv, float tmin, float tmax);

RT_D uint32_t qnode_test(const DevScene& S, uint32_t ni, const RayC& R, float tmin, float tmax, NodeHead& hd) {
    const float4* N = S.qnodes + (size_t)ni * RT_QNODE_F4;
    float4 h = __ldg(N);
    uint4 bq[3] = {__ldg(reinterpret_cast<const uint4*>(N + 1)), __ldg(reinterpret_cast<const uint4*>(N + 2)),
                   __ldg(reinterpret_cast<const uint4*>(N + 3))};
    hd = load_head(N + 4);
    if (R.general) return qnode_test_general(N, R.o, R.inv, tmin, tmax);
    const uint32_t meta = __float_as_uint(h.w);
    const float P[3] = {h.x, h.y, h.z}, I[3] = {R.inv.x, R.inv.y, R.inv.z};
    const float CN[3] = {R.cn.x, R.cn.y, R.cn.z}, CF[3] = {R.cf.x, R.cf.y, R.cf.z};
    float Sa[3], An[3], Af[3];
    uint32_t sn[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        // exponent fields of x, y, z: bits 30-23, 22-15, 14-7
        Sa[a] = __uint_as_float((meta << (8 * a)) & 0x7F800000u) * I[a];
        An[a] = __fmaf_rd(-32768.0f, Sa[a], __fmaf_rd(P[a], I[a], CN[a]));
        Af[a] = __fmaf_ru(-32768.0f, Sa[a], __fmaf_ru(P[a], I[a], CF[a]));
        // the bytes of a child are (lower, upper): the near one is the lower for a positive direction
        sn[a] = I[a] < 0.0f ? 0x7414u : 0x7404u;
    }
    uint32_t miss = 0;
#pragma unroll
    for (int c = 7; c >= 0; c--) {
        float n[3], f[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const uint32_t w = c < 2 ? bq[a].x : c < 4 ? bq[a].y : c < 6 ? bq[a].z : bq[a].w;
            const uint32_t sel = sn[a] + ((c & 1) ? 0x20u : 0u);
            n[a] = __fmaf_rn(qbyte(w, sel), Sa[a], An[a]);
            f[a] = __fmaf_rn(qbyte(w, sel ^ 0x10u), Sa[a], Af[a]);
        }
        float t0 = fmax3f(fmaxf(tmin, n[0]), n[1], n[2]);
        float t1 = fmin3f(fminf(tmax, f[0]), f[1], f[2]);
        miss = __funnelshift_l(__float_as_uint(__fmaf_rn(t1, EXIT_WIDEN, -t0)), miss, 1);
    }
    return ~miss;
}

// General rays (a zero, denormal or extreme direction component, or t_min < 0):
// the planes decoded with outward rounding, then the general slab test.
__device__ __noinline__ uint32_t qnode_test_general(const float4* N, float3 o, float3 inv, float tmin, float tmax) {
    float4 h = __ldg(N);
    const uint32_t meta = __float_as_uint(h.w);
    const float P[3] = {h.x, h.y, h.z};
    float lo[3][8], hi[3][8];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        uint4 b = __ldg(reinterpret_cast<const uint4*>(N + 1 + a));
        float sa = __uint_as_float((meta << (8 * a)) & 0x7F800000u);
        const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int c = 0; c < 8; c++) {
            uint32_t v = w[c >> 1] >> (16 * (c & 1));
            float ql = (float)(v & 0xFFu), qh = (float)((v >> 8) & 0xFFu);
            lo[a][c] = __fmaf_rd(ql, sa, P[a]);
            hi[a][c] = __fmaf_ru(qh, sa, P[a]);
        }
    }
    uint32_t mask = 0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        float dax = (lo[0][c] - o.x) * inv.x, dbx = (hi[0][c] - o.x) * inv.x;
        float day = (lo[1][c] - o.y) * inv.y, dby = (hi[1][c] - o.y) * inv.y;
        float daz = (lo[2][c] - o.z) * inv.z, dbz = (hi[2][c] - o.z) * inv.z;
        float lx = fminf(dax, dbx), hx = fmaxf(dax, dbx);
        float ly = fminf(day, dby), hy = fmaxf(day, dby);
        float lz = fminf(daz, dbz), hz = fmaxf(daz, dbz);
        if (isnan(dax) || isnan(dbx)) { lx = -INFINITY; hx = INFINITY; }
        if (isnan(day) || isnan(dby)) { ly = -INFINITY; hy = INFINITY; }
        if (isnan(daz) || isnan(dbz)) { lz = -INFINITY; hz = INFINITY; }
        float t0 = fmaxf(fmaxf(fmaxf(tmin, lx), ly), lz);
        float t1 = fminf(fminf(fminf(tmax, hx), hy), hz);
        float t1w = t1 + fabsf(t1) * (EXIT_WIDEN - 1.0f);
        if (t0 <= t1w) mask |= 1u << c;
    }
    return mask;
}

// ── 4-wide nodes (7 float4: lower x, y, z, upper x, y, z, header) ───────────
__device__ __noinline__ uint32_t node4_test_general(const float4* N, float3 o, float3 inv, float tmin, float tmax) {
    float4 q[6];
#pragma unroll
    for (int i = 0; i < 6; i++) q[i] = __ldg(N + i);
    const float* f = reinterpret_cast<const float*>(q);
    uint32_t mask = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float dax = (f[0 + c] - o.x) * inv.x, dbx = (f[12 + c] - o.x) * inv.x;
        float day = (f[4 + c] - o.y) * inv.y, dby = (f[16 + c] - o.y) * inv.y;
        float daz = (f[8 + c] - o.z) * inv.z, dbz = (f[20 + c] - o.z) * inv.z;
        float lx = fminf(dax, dbx), hx = fmaxf(dax, dbx);
        float ly = fminf(day, dby), hy = fmaxf(day, dby);
        float lz = fminf(daz, dbz), hz = fmaxf(daz, dbz);
        if (isnan(dax) || isnan(dbx)) { lx = -INFINITY; hx = INFINITY; }
        if (isnan(day) || isnan(dby)) { ly = -INFINITY; hy = INFINITY; }
        if (isnan(daz) || isnan(dbz)) { lz = -INFINITY; hz = INFINITY; }
        float t0 = fmaxf(fmaxf(fmaxf(tmin, lx), ly), lz);
        float t1 = fminf(fminf(fminf(tmax, hx), hy), hz);
        float t1w = t1 + fabsf(t1) * (EXIT_WIDEN - 1.0f);
        if (t0 <= t1w) mask |= 1u << c;
    }
    return mask;
}

RT_D uint32_t node4_test(const DevScene& S, uint32_t ni, const RayC& R, float tmin, float tmax, NodeHead& h) {
    const float4* N = S.nodes4 + (size_t)ni * RT_NODE4_F4;
    h = load_head(N + 6);
    if (R.general) return node4_test_general(N, R.o, R.inv, tmin, tmax);
    // the near planes of an axis are the lower ones for a positive direction
    // (R.nx / 2 is 0 or 3, R.ny / 2 is 1 or 4, R.nz / 2 is 2 or 5)
    float4 q[6];
    q[0] = __ldg(N + R.nx / 2); q[1] = __ldg(N + R.ny / 2); q[2] = __ldg(N + R.nz / 2);
    q[3] = __ldg(N + 3 - R.nx / 2); q[4] = __ldg(N + 5 - R.ny / 2); q[5] = __ldg(N + 7 - R.nz / 2);
    const float* f = reinterpret_cast<const float*>(q);
    uint32_t miss = 0;
#pragma unroll
    for (int c = 3; c >= 0; c--) {
        float nx = __fmaf_rn(f[0 + c], R.inv.x, R.cn.x), fx = __fmaf_rn(f[12 + c], R.inv.x, R.cf.x);
        float ny = __fmaf_rn(f[4 + c], R.inv.y, R.cn.y), fy = __fmaf_rn(f[16 + c], R.inv.y, R.cf.y);
        float nz = __fmaf_rn(f[8 + c], R.inv.z, R.cn.z), fz = __fmaf_rn(f[20 + c], R.inv.z, R.cf.z);
        float t0 = fmax3f(fmaxf(tmin, nx), ny, nz);
        float t1 = fmin3f(fminf(tmax, fx), fy, fz);
        miss = __funnelshift_l(__float_as_uint(__fmaf_rn(t1, EXIT_WIDEN, -t0)), miss, 1);
    }
    return ~miss;
}

// the node test of node `ni` in the layout NF (RT_NODES_FULL,
// RT_NODES_QUANTISED, RT_NODES_WIDE4) and the leaves of its tree
template <int NF>
RT_D uint32_t node_test_any(const DevScene& S, uint32_t ni, const RayC& R, float tmin, float tmax, NodeHead& h) {
    if constexpr (NF == RT_NODES_QUANTISED) return qnode_test(S, ni, R, tmin, tmax, h);
    else if constexpr (NF == RT_NODES_WIDE4) return node4_test(S, ni, R, tmin, tmax, h);
    else return node_test(S, ni, R, tmin, tmax, h);
}
template <int NF>
RT_D const LeafSet& leaf_set(const DevScene& S) { return NF == RT_NODES_WIDE4 ? S.leaves4 : S.leaves; }

// A primitive's hit counts only if the ray meets the leaf's own float box, in the
// arithmetic of the reference-layout slab test: planes (b − o)·inv, the exit
// widened by 2^-15, the bound by 2^-16 (rays with a zero direction component or
// t_min < 0: both planes with min / max, a NaN slab spanning the whole line).  The
// node tests are the looser ones in every layout.  A triangle seen edge-on at its
// box's corner can have a t far off its box, so without this the looseness would
// show in a hit (one in 10^8 camera rays of the icosphere).  The closest hit so
// far is no bound here (closest-hit rays pass an infinite t_max): whether a hit
// counts depends on the primitive and the ray, not on the order of the tests.
// (What the order still decides, as in the reference, is whether the traversal
// comes to a primitive at all whose box begins beyond the closest hit while its
// computed t lies before.)  Asked for accepted hits only: ahead of every primitive
// test it cost 12 % of the closest-hit kernel (48.3 → 54.0 ms).
__device__ __noinline__ bool leaf_box_general(float4 lo, float4 hi, float3 o, float3 inv, float tmin, float tmax) {
    const float W = 1.000030517578125f;   // 1 + 2^-15
    const float L[3] = {lo.x, lo.y, lo.z}, H[3] = {hi.x, hi.y, hi.z}, O[3] = {o.x, o.y, o.z}, I[3] = {inv.x, inv.y, inv.z};
    const bool general = isinf(inv.x) || isinf(inv.y) || isinf(inv.z) || !(tmin >= 0.0f);
    float t0 = tmin, t1 = general ? tmax : tmax + fabsf(tmax) * SLAB_WIDEN;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (general) {
            float da = (L[a] - O[a]) * I[a], db = (H[a] - O[a]) * I[a];
            float l = fminf(da, db), h = fmaxf(da, db);
            if (isnan(da) || isnan(db)) { l = -INFINITY; h = INFINITY; }
            t0 = fmaxf(t0, l);
            t1 = fminf(t1, h);
        } else {
            bool neg = signbit(I[a]);
            t0 = fmaxf(t0, ((neg ? H[a] : L[a]) - O[a]) * I[a]);
            t1 = fminf(t1, ((neg ? L[a] : H[a]) - O[a]) * (I[a] * W));
        }
    }
    return t0 <= (general ? t1 + fabsf(t1) * SLAB_WIDEN : t1);
}
RT_D bool leaf_box(const float4* box, const RayC& R, float tmin, float tmax) {
    const float4 lo = __ldg(box), hi = __ldg(box + 1);
    if (R.general) return leaf_box_general(lo, hi, R.o, R.inv, tmin, tmax);
    const float W = 1.000030517578125f;
    bool sx = R.inv.x < 0.0f, sy = R.inv.y < 0.0f, sz = R.inv.z < 0.0f;
    float nx = ((sx ? hi.x : lo.x) - R.o.x) * R.inv.x, fx = ((sx ? lo.x : hi.x) - R.o.x) * (R.inv.x * W);
    float ny = ((sy ? hi.y : lo.y) - R.o.y) * R.inv.y, fy = ((sy ? lo.y : hi.y) - R.o.y) * (R.inv.y * W);
    float nz = ((sz ? hi.z : lo.z) - R.o.z) * R.inv.z, fz = ((sz ? lo.z : hi.z) - R.o.z) * (R.inv.z * W);
    return fmax3f(fmaxf(tmin, nx), ny, nz) <= fmin3f(fminf(tmax + fabsf(tmax) * SLAB_WIDEN, fx), fy, fz);
}

// Test of leaf `k` (its index in the set's order); updates `best`.  Returns true
// for a convex solid, which is not tested here.  The leaf's triangle is its own
// record, found from the node's header alone: one round trip to the L2 where a
// reference and then the primitive would be two (icosphere extend 52.9 ms that
// way, 51.3 this way; gem 10.4 and 9.3).  The reference is a hit record already (RT_HIT_MAKE).
// ANA: the scene has convex solids or shapes; without them the type-3 branch
// is compiled out, so triangle scenes keep a lean traversal kernel.
template <bool ANA>
RT_D bool leaf_closest(const DevScene& S, const LeafSet& LS, uint32_t k, const RayC& R, float3 d, float tmin, Best& best) {
    const float3 o = R.o;
    const float4* rec = LS.rec + (size_t)k * 3;
    float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
    const uint32_t ref = f2u(c.z), type = RT_HIT_TYPE(ref), idx = RT_HIT_INDEX(ref);
    float t, b1, b2;
    uint32_t gid = f2u(c.y);
    bool h;
    if (type == RT_PRIM_TRI) {
        h = tri_test(a, b, c, o, d, tmin, best.t, &t, &b1, &b2);
    } else if (type == RT_PRIM_QUAD) {
        const float4* g = S.quad + (size_t)idx * 5;
        float4 gg[4] = {__ldg(g), __ldg(g + 1), __ldg(g + 2), __ldg(g + 3)};
        h = quad_test(gg, o, d, tmin, best.t, &t, &b1, &b2);
    } else if (type == RT_PRIM_SPHERE) {
        const float4* g = S.sphere + (size_t)idx * 2;
        h = sphere_test(__ldg(g), o, d, tmin, best.t, &t);
        b1 = b2 = 0.0f;
    } else if (!ANA) {
        return false;
    } else {                                        // a shape; b1 carries the surface
        float4 c0 = __ldg(S.cvx + (size_t)idx * 2);
        int pi = -1, cnt = __float_as_int(c0.y);
        if (cnt > 0) return true;                   // a convex solid: left to the warp (warp_convex)
        const float4* P = S.shape_par + __float_as_int(c0.x);
        float3 lo, ld;
        shape_local(P, o, d, &lo, &ld);
        h = shape_test(-1 - cnt, P, lo, ld, tmin, best.t, &t, &pi);
        b1 = __int_as_float(pi);
        b2 = 0.0f;
    }
    if (h && (t < best.t || best.ref == RT_MISS_REF || gid < best.gid) &&
        leaf_box(LS.box + (size_t)k * 2, R, tmin, INFINITY)) {
        best.t = t; best.b1 = b1; best.b2 = b2; best.ref = ref; best.gid = gid;
    }
    return false;
}

template <bool ANA>
RT_D bool leaf_any_test(const DevScene& S, const float4* rec, float3 o, float3 d, float tmin, float tmax, bool* convex) {
    float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
    const uint32_t ref = f2u(c.z), type = RT_HIT_TYPE(ref), idx = RT_HIT_INDEX(ref);
    float t, b1, b2;
    if (type == RT_PRIM_TRI) {
        return tri_test(a, b, c, o, d, tmin, tmax, &t, &b1, &b2);
    } else if (type == RT_PRIM_QUAD) {
        const float4* g = S.quad + (size_t)idx * 5;
        float4 gg[4] = {__ldg(g), __ldg(g + 1), __ldg(g + 2), __ldg(g + 3)};
        return quad_test(gg, o, d, tmin, tmax, &t, &b1, &b2);
    }
    if (type == RT_PRIM_SPHERE) return sphere_test(__ldg(S.sphere + (size_t)idx * 2), o, d, tmin, tmax, &t);
    if (!ANA) return false;
    float4 c0 = __ldg(S.cvx + (size_t)idx * 2);
    int pi, cnt = __float_as_int(c0.y);
    if (cnt > 0) { *convex = true; return false; }  // left to the warp (warp_convex)
    const float4* P = S.shape_par + __float_as_int(c0.x);
    float3 lo, ld;
    shape_local(P, o, d, &lo, &ld);
    return shape_test(-1 - cnt, P, lo, ld, tmin, tmax, &t, &pi);
}
template <bool ANA>
RT_D bool leaf_any(const DevScene& S, const LeafSet& LS, uint32_t k, const RayC& R, float3 d, float tmin, float tmax,
                   bool* convex) {
    return leaf_any_test<ANA>(S, LS.rec + (size_t)k * 3, R.o, d, tmin, tmax, convex) &&
           leaf_box(LS.box + (size_t)k * 2, R, tmin, tmax);
}

}  // namespace

namespace rtk {

// Per-thread traversal stack of groups (the reference keeps 128 nodes inline
// and spills to a heap Vec, bvh.rs:229-239).  A group is the pending children
// of one node: x = its first child's index, y = their slots (bits 0-7) and the
// slots of all its inner children (bits 8-15).  The newest RT_SHORT_STACK
// groups live in a ring: the thread's local memory (RT_STACK_LOCAL, the
// default) or shared memory laid out [entry][thread].  Entry e ≥ RT_SHORT_STACK
// of a deeper stack waits in the thread's global column, two words at
// spill[2(e − RT_SHORT_STACK) · stride] (rt_set_tuning can shrink the ring to
// fewer slots, so the tests run every traversal through the spill path).  A
// push beyond the ring first moves the ring slot's old entry to its column, a
// pop that uncovers a spilled entry brings it back.  A traversal holds at most
// one group per tree level, so S.stack_cap (what a column holds, from the tree's
// depth) is never reached in the scene's own tree; a lower one from rt_set_tuning
// makes the traversal stop with RT_ERR_CAPACITY.
constexpr int RING_STRIDE = RT_STACK_LOCAL ? 1 : RT_TRACE_BLOCK;
struct TStack {
    uint2* ring;             // ring slot k at ring[k · RING_STRIDE] (shared: &ring[threadIdx.x])
    int sp;
    bool any;                // the any-hit kernel's columns: it may run beside the closest-hit kernel

    // S.stack_cap entries at most; S.stack_ring ring slots in use (a power of two).
    // The spill column's address is formed only when an entry goes there.
    RT_D bool room(const DevScene& S) const { return sp < S.stack_cap; }
    RT_D uint32_t* column(const DevScene& S, int e) const {
        return (any ? S.stack_spill_any : S.stack_spill) + (size_t)(2 * e) * (gridDim.x * blockDim.x) + blockIdx.x * blockDim.x + threadIdx.x;
    }
    RT_D void push(const DevScene& S, uint2 v) {
        int slot = sp & (S.stack_ring - 1);
        if (sp >= S.stack_ring) {
            uint2 old = ring[slot * RING_STRIDE];
            uint32_t* e = column(S, sp - S.stack_ring);
            e[0] = old.x; e[gridDim.x * blockDim.x] = old.y;
        }
        ring[slot * RING_STRIDE] = v;
        sp++;
    }
    RT_D uint2 pop(const DevScene& S) {
        sp--;
        int slot = sp & (S.stack_ring - 1);
        uint2 v = ring[slot * RING_STRIDE];
        if (sp >= S.stack_ring) {
            const uint32_t* e = column(S, sp - S.stack_ring);
            ring[slot * RING_STRIDE] = make_uint2(e[0], e[gridDim.x * blockDim.x]);
        }
        return v;
    }
};

// the root as a group of one
RT_D uint2 root_group() { return make_uint2(0u, 0x0101u); }

// Takes the group's pending slot that is nearest along the ray's octant (the
// smallest slot XOR octant, bit by bit) and returns its node.
RT_D uint32_t take_nearest(uint2& g, uint32_t ord) {
    uint32_t m = g.y & 0xFFu, t;
    t = m & ord;         if (t) m = t;
    t = m & (ord >> 8);  if (t) m = t;
    t = m & (ord >> 16); if (t) m = t;
    g.y ^= m;
    return g.x + __popc((g.y >> 8) & (m - 1u));
}
// Takes the group's first pending slot.
RT_D uint32_t take_first(uint2& g) {
    uint32_t m = g.y & (0u - g.y);
    g.y ^= m;
    return g.x + __popc((g.y >> 8) & (m - 1u));
}
// After a visit: go on with its hit inner children, else with the rest of the
// current group, else with the newest one on the stack; false when none is left.
RT_D bool next_group(const DevScene& S, uint2& g, uint32_t child, uint32_t inner, uint32_t masks, TStack& stk,
                     bool& ok) {
    if (inner) {
        if (g.y & 0xFFu) {
            if (!stk.room(S)) { ok = false; return false; }
            stk.push(S, g);
        }
        g = make_uint2(child, inner | (masks & 0xFFu) << 8);
        return true;
    }
    if (g.y & 0xFFu) return true;
    if (stk.sp == 0) return false;
    g = stk.pop(S);
    return true;
}

// Convex solids a lane met in a visit: the node's first leaf and which of its leaves.
struct Convex { uint32_t first, which; };
__device__ __forceinline__ float3 shfl3(float3 v, int l) {
    return mk(__shfl_sync(0xFFFFFFFFu, v.x, l), __shfl_sync(0xFFFFFFFFu, v.y, l), __shfl_sync(0xFFFFFFFFu, v.z, l));
}

// One node visit of the closest-hit traversal: tests the children of the
// group's nearest node and intersects its hit leaves (convex solids are only
// noted in `cv`); `inner` gets the hit inner children.
template <bool ANA, int NF>
RT_D void closest_visit(const DevScene& S, const RayC& R, float3 d, float tmin, Best& best, uint2& grp, NodeHead& h,
                        uint32_t& inner, Convex& cv) {
    const uint32_t node = take_nearest(grp, R.ord);
    const uint32_t hits = node_test_any<NF>(S, node, R, tmin, best.t, h);
    uint32_t leaves = hits & (h.masks >> 8);
    inner = hits & h.masks & 0xFFu;
    cv.which = 0u;
    if (leaves) {
        const uint32_t all = h.masks >> 8;
        cv.first = h.leaf;
#pragma unroll 1
        while (leaves) {
            uint32_t k = __popc(all & ((leaves & (0u - leaves)) - 1u));
            leaves &= leaves - 1;
            if (leaf_closest<ANA>(S, leaf_set<NF>(S), h.leaf + k, R, d, tmin, best) && ANA) cv.which |= 1u << k;
        }
    }
}
// The noted convex solids of the warp's lanes, one test at a time (every lane calls it).
RT_D void closest_convex(const DevScene& S, const LeafSet& LS, const RayC& R, float3 d, float tmin, Best& best, Convex& cv) {
    uint32_t need = __ballot_sync(0xFFFFFFFFu, cv.which != 0u);
    while (need) {
        const int L = __ffs(need) - 1;
        const uint32_t leaf = __shfl_sync(0xFFFFFFFFu, cv.first + __ffs(cv.which) - 1u, L);
        if ((threadIdx.x & 31u) == L) cv.which &= cv.which - 1u;
        const uint32_t ref = f2u(__ldg(LS.rec + (size_t)leaf * 3 + 2).z);
        const float4* rec = S.cvx + (size_t)RT_HIT_INDEX(ref) * 2;
        float4 c0 = __ldg(rec);
        float t;
        int pi;
        bool h = warp_convex(S.cvx_planes + __float_as_int(c0.x), __float_as_int(c0.y), shfl3(R.o, L), shfl3(d, L),
                             __shfl_sync(0xFFFFFFFFu, tmin, L), __shfl_sync(0xFFFFFFFFu, best.t, L), &t, &pi);
        if (h && (threadIdx.x & 31u) == L) {
            uint32_t gid = f2u(__ldg(rec + 1).x);
            if ((t < best.t || best.ref == RT_MISS_REF || gid < best.gid) && leaf_box(LS.box + (size_t)leaf * 2, R, tmin, INFINITY)) {
                best.t = t; best.b1 = __int_as_float(pi); best.b2 = 0.0f; best.ref = ref; best.gid = gid;
            }
        }
        need = __ballot_sync(0xFFFFFFFFu, cv.which != 0u);
    }
}

// One node visit of the any-hit traversal (bvh.rs:487-530): true when a
// primitive was hit.
template <bool ANA, int NF>
RT_D bool any_visit(const DevScene& S, const RayC& R, float3 d, float tmin, float tmax, uint2& grp, NodeHead& h,
                    uint32_t& inner, Convex& cv) {
    const uint32_t node = take_first(grp);
    const uint32_t hits = node_test_any<NF>(S, node, R, tmin, tmax, h);
    uint32_t leaves = hits & (h.masks >> 8);
    inner = hits & h.masks & 0xFFu;
    cv.which = 0u;
    if (leaves) {
        const uint32_t all = h.masks >> 8;
        cv.first = h.leaf;
#pragma unroll 1
        while (leaves) {
            uint32_t k = __popc(all & ((leaves & (0u - leaves)) - 1u));
            leaves &= leaves - 1;
            bool convex = false;
            if (leaf_any<ANA>(S, leaf_set<NF>(S), h.leaf + k, R, d, tmin, tmax, &convex)) { cv.which = 0u; return true; }
            if (ANA && convex) cv.which |= 1u << k;
        }
    }
    return false;
}
// The noted convex solids of the warp's lanes (every lane calls it): true for a lane whose ray hit one.
RT_D bool any_convex(const DevScene& S, const LeafSet& LS, const RayC& R, float3 d, float tmin, float tmax, Convex& cv) {
    bool hit = false;
    uint32_t need = __ballot_sync(0xFFFFFFFFu, cv.which != 0u);
    while (need) {
        const int L = __ffs(need) - 1;
        const uint32_t leaf = __shfl_sync(0xFFFFFFFFu, cv.first + __ffs(cv.which) - 1u, L);
        if ((threadIdx.x & 31u) == L) cv.which &= cv.which - 1u;
        const uint32_t ref = f2u(__ldg(LS.rec + (size_t)leaf * 3 + 2).z);
        float4 c0 = __ldg(S.cvx + (size_t)RT_HIT_INDEX(ref) * 2);
        float t;
        int pi;
        bool h = warp_convex(S.cvx_planes + __float_as_int(c0.x), __float_as_int(c0.y), shfl3(R.o, L), shfl3(d, L),
                             __shfl_sync(0xFFFFFFFFu, tmin, L), __shfl_sync(0xFFFFFFFFu, tmax, L), &t, &pi);
        if (h && (threadIdx.x & 31u) == L && leaf_box(LS.box + (size_t)leaf * 2, R, tmin, tmax)) { hit = true; cv.which = 0u; }
        need = __ballot_sync(0xFFFFFFFFu, cv.which != 0u);
    }
    return hit;
}

RT_D bool nan_ray(float3 o, float3 d, float tmin, float tmax) {
    return isnan(o.x) || isnan(o.y) || isnan(o.z) || isnan(d.x) || isnan(d.y) || isnan(d.z) || isnan(tmin) ||
           isnan(tmax);
}

}  // namespace rtk

// ── persistent traversal with lane refill ───────────────────────────────────
// Each lane owns one ray; every loop iteration performs one node visit per
// active lane.  When at least RT_REFILL lanes of a warp are idle, they pull
// new rays from the queue together (one atomic per warp), so a warp is not held
// by its slowest ray (persistent threads with dynamic fetch, Aila & Laine 2009).
#ifndef RT_REFILL
#define RT_REFILL 12
#endif
// the closest-hit kernel refills later: its rays are longer, and fewer,
// larger refills measured faster (icosphere workload, extend 62.8 → 60.6 ms
// at 24; any-hit stays best at 12)
#ifndef RT_REFILL_CLOSEST
#define RT_REFILL_CLOSEST 24
#endif
// with split leaves (below) the idle lanes are dearer: 4M caller rays 1.42 -> 1.34
// ms at 16, 1.43 at 20, 1.48 at 28; icosphere extend 12.54 -> 12.45, 12.39, 13.09
#ifndef RT_REFILL_SPLIT
#define RT_REFILL_SPLIT 16
#endif
#define FULLMASK 0xFFFFFFFFu
// Resident blocks per SM each traversal kernel is compiled for.  Full nodes
// keep 48 box words in flight: 7 blocks (72 registers; gem extend 9.0 ms against
// 9.7 at 5, 10.0 at 6 and 10.2 at 8, where ptxas spills).  Quantised nodes need
// 12: 8 blocks (64 registers; icosphere extend 49.7 ms against 54.6, 50.9, 51.6
// at 6, 7, 9).  The closest-hit kernel with the convex solids' warp test takes 6
// (gem room extend 7.0 ms against 7.7 at 7).
template <int NF, bool ANA, bool ANY> constexpr int trace_minb() {
    return NF == RT_NODES_QUANTISED ? 8 : ANA && !ANY ? 6 : 7;
}
static_assert(RT_TRACE_MINB == 8, "the spill columns are sized for the most resident blocks");

// Lanes of a warp that take rays: all of them — but in a scene with convex
// solids, whose tests the warp runs one after the other (warp_convex), rays too
// few to fill the grid's warps are spread over them, down to 4 a warp (gem room
// 22.3 -> 21.0 ms: its 50 bounces end in many small launches).  Without such
// solids the spread only keeps more warps busy beside the shadow rays and the
// caustic lookup (gem 31.2 -> 31.9 ms).  Asked anew at each refill: no register
// is kept for it.
template <bool ANA>
RT_D uint32_t warp_lanes(uint32_t n) {
    const uint32_t warps = gridDim.x * (RT_TRACE_BLOCK / 32);
    if (!ANA || n >= warps * 31u) return FULLMASK;
    return (1u << max(4u, (n + warps - 1) / warps)) - 1u;
}

// MODE 0: wavefront extend (queue of path ids, rays in PathState, hits to PathState)
// MODE 1: API (rays n×8 in memory, hits as int4)

// Closest hit over quantised nodes, without convex solids: an iteration is at
// most one node visit and one leaf test per lane, and a lane with leaves left
// tests them in the next iterations while the others visit nodes, instead of
// holding the warp in a loop as long as its longest list.  Each lane's own order
// of visits and tests is the same, so its hits are.  Bound by issue slots at 14-17
// of 32 lanes (1,310,720 triangles, 1080p at 64 samples: extend 50.0 -> 45.2 ms;
// 4M caller rays against 327,680 triangles 1.58 -> 1.41 ms).  Waiting for 3, 6 or
// 10 lanes with leaves before testing any was slower (46.6, 48.7, 54.6 ms).  The
// loop stays for full nodes, where the list's two words spill (96 B at 72
// registers; 24 thumbnails 20.2 -> 21.1 ms, equal at 80 registers), and for
// any-hit rays, where it made no difference (14.8 ms both).
template <bool ANA, int NF> constexpr bool split_leaves() { return !ANA && NF == RT_NODES_QUANTISED; }

template <int MODE, bool ANA, int NF>
__global__ void __launch_bounds__(RT_TRACE_BLOCK, trace_minb<NF, ANA, false>()) k_closest(DevScene S, PathState P, const uint32_t* __restrict__ queue,
                                                            const float* __restrict__ rays, uint32_t n_api,
                                                            const uint32_t* count, uint32_t* next,
                                                            int4* __restrict__ out, int* err) {
    const uint32_t n = MODE == 0 ? *count : n_api;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
#if RT_STACK_LOCAL
    uint2 ring[RT_SHORT_STACK];
#else
    __shared__ uint2 ring[RT_SHORT_STACK * RT_TRACE_BLOCK];
#endif
    rtk::TStack stk{RT_STACK_LOCAL ? ring : ring + threadIdx.x, 0, false};
    bool active = false, exhausted = false, ok = true;
    uint32_t item = 0, pid = 0;
    uint2 grp = make_uint2(0u, 0u);
    float3 o = mk(0.f, 0.f, 0.f), d = o;
    RayC R = make_rayc(o, mk(1.f, 1.f, 1.f), 0.0f);
    float tmin = 0.0f;
    Best best{0.0f, 0.0f, 0.0f, RT_MISS_REF, 0xFFFFFFFFu};
    // split leaves: the pending ones of the last visited node (bits 0-7), all its
    // leaves (8-15) and whether no group is left (16); its first leaf
    uint32_t pend = 0u, first = 0u;
    while (true) {
        uint32_t idle = __ballot_sync(FULLMASK, !active);
        if (!exhausted && __popc(idle) >= (split_leaves<ANA, NF>() ? RT_REFILL_SPLIT : RT_REFILL_CLOSEST)) {
            if (ANA) idle &= warp_lanes<ANA>(n);
            uint32_t k = __popc(idle), base = 0;
            if (lane == 0 && (!ANA || k)) base = atomicAdd(next, k);
            base = __shfl_sync(FULLMASK, base, 0);
            if ((!ANA || k) && base + k >= n) exhausted = true;
            if (ANA ? (idle >> lane) & 1u : !active) {
                uint32_t i = base + __popc(idle & lt);
                if (i < n) {
                    item = i;
                    float tmax;
                    if (MODE == 0) {
                        pid = queue ? queue[i] : i;
                        float4 ro = P.ray_o[pid], rd = P.ray_d[pid];
                        o = mk(ro.x, ro.y, ro.z); d = mk(rd.x, rd.y, rd.z);
                        tmin = 0.001f; tmax = INFINITY;
                    } else {
                        const float* r = rays + (size_t)i * 8;
                        o = mk(r[0], r[1], r[2]); d = mk(r[3], r[4], r[5]);
                        tmin = r[6]; tmax = r[7];
                    }
                    R = make_rayc(o, d, tmin);
                    best = Best{tmax, 0.0f, 0.0f, RT_MISS_REF, 0xFFFFFFFFu};
                    grp = rtk::root_group(); stk.sp = 0;
                    active = !rtk::nan_ray(o, d, tmin, tmax);
                    if (!active) {
                        if (MODE == 0) P.hit[pid] = make_float4(__uint_as_float(RT_MISS_REF), 0.f, 0.f, 0.f);
                        else out[i] = make_int4(-1, 0, 0, 0);
                    }
                }
            }
        }
        if (exhausted && __ballot_sync(FULLMASK, active) == 0) break;
        auto finish = [&] {
            active = false;
            bool hit = best.ref != RT_MISS_REF;
            if (MODE == 0) {
                P.hit[pid] = make_float4(__uint_as_float(best.ref), best.t, best.b1, best.b2);
            } else {
                out[item] = make_int4(hit ? (int)best.gid : -1, __float_as_int(hit ? best.t : 0.0f),
                                      __float_as_int(hit ? best.b1 : 0.0f), __float_as_int(hit ? best.b2 : 0.0f));
            }
        };
        if constexpr (!split_leaves<ANA, NF>()) {
            NodeHead h{0u, 0u, 0u};
            uint32_t inner = 0u;
            rtk::Convex cv{0u, 0u};
            if (active) rtk::closest_visit<ANA, NF>(S, R, d, tmin, best, grp, h, inner, cv);
            if (ANA) rtk::closest_convex(S, leaf_set<NF>(S), R, d, tmin, best, cv);
            if (active) {
                bool lok = true;
                bool more = rtk::next_group(S, grp, h.child, inner, h.masks, stk, lok);
                if (!lok) ok = false;
                if (!more) finish();
            }
        } else {
            if (active && !(pend & 0xFFu)) {
                NodeHead h{0u, 0u, 0u};
                const uint32_t node = rtk::take_nearest(grp, R.ord);
                const uint32_t hits = node_test_any<NF>(S, node, R, tmin, best.t, h);
                bool lok = true;
                const bool more = rtk::next_group(S, grp, h.child, hits & h.masks & 0xFFu, h.masks, stk, lok);
                if (!lok) ok = false;
                pend = (hits & (h.masks >> 8)) | (h.masks & 0xFF00u) | (more ? 0u : 1u << 16);
                first = h.leaf;
            }
            if (pend & 0xFFu) {
                const uint32_t leaves = pend & 0xFFu;
                const uint32_t k = __popc(((pend >> 8) & 0xFFu) & ((leaves & (0u - leaves)) - 1u));
                pend &= pend - 1u;
                leaf_closest<ANA>(S, leaf_set<NF>(S), first + k, R, d, tmin, best);
            }
            if (active && (pend >> 16) && !(pend & 0xFFu)) {
                pend = 0u;
                finish();
            }
        }
    }
    if (!ok) atomicExch(err, RT_ERR_CAPACITY);
}

// MODE 0: wavefront shadow rays (an occluded ray cancels its parked contribution)
// MODE 1: API any-hit (occluded flags)
template <int MODE, bool ANA, int NF>
__global__ void __launch_bounds__(RT_TRACE_BLOCK, trace_minb<NF, ANA, true>()) k_any(DevScene S, PendTargets T, const float4* __restrict__ sq,
                                                        const float* __restrict__ rays, uint32_t n_api,
                                                        const uint32_t* count, uint32_t* next,
                                                        uint8_t* __restrict__ out, int* err) {
    const uint32_t n = MODE != 1 ? *count : n_api;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
#if RT_STACK_LOCAL
    uint2 ring[RT_SHORT_STACK];
#else
    __shared__ uint2 ring[RT_SHORT_STACK * RT_TRACE_BLOCK];
#endif
    rtk::TStack stk{RT_STACK_LOCAL ? ring : ring + threadIdx.x, 0, true};
    bool active = false, exhausted = false, ok = true;
    uint32_t item = 0, tag = 0;
    uint2 grp = make_uint2(0u, 0u);
    float3 o = mk(0.f, 0.f, 0.f), d = o;
    RayC R = make_rayc(o, mk(1.f, 1.f, 1.f), 0.0f);
    float tmin = 0.0f, tmax = 0.0f;
    bool hit = false;
    while (true) {
        uint32_t idle = __ballot_sync(FULLMASK, !active);
        if (!exhausted && __popc(idle) >= RT_REFILL) {
            if (ANA) idle &= warp_lanes<ANA>(n);
            uint32_t k = __popc(idle), base = 0;
            if (lane == 0 && (!ANA || k)) base = atomicAdd(next, k);
            base = __shfl_sync(FULLMASK, base, 0);
            if ((!ANA || k) && base + k >= n) exhausted = true;
            if (ANA ? (idle >> lane) & 1u : !active) {
                uint32_t i = base + __popc(idle & lt);
                if (i < n) {
                    item = i;
                    if (MODE != 1) {
                        float4 a = sq[(size_t)i * 2], b = sq[(size_t)i * 2 + 1];
                        o = mk(a.x, a.y, a.z); d = mk(b.x, b.y, b.z);
                        tmin = 0.001f; tmax = a.w;
                        tag = __float_as_uint(b.w);
                    } else {
                        const float* r = rays + (size_t)i * 8;
                        o = mk(r[0], r[1], r[2]); d = mk(r[3], r[4], r[5]);
                        tmin = r[6]; tmax = r[7];
                    }
                    R = make_rayc(o, d, tmin);
                    grp = rtk::root_group(); stk.sp = 0; hit = false;
                    active = !rtk::nan_ray(o, d, tmin, tmax);
                    if (!active && MODE == 1) out[i] = 0;
                }
            }
        }
        if (exhausted && __ballot_sync(FULLMASK, active) == 0) break;
        NodeHead h{0u, 0u, 0u};
        uint32_t inner = 0u;
        rtk::Convex cv{0u, 0u};
        if (active) hit = rtk::any_visit<ANA, NF>(S, R, d, tmin, tmax, grp, h, inner, cv);
        if (ANA) { if (rtk::any_convex(S, leaf_set<NF>(S), R, d, tmin, tmax, cv)) hit = true; }
        if (active) {
            bool lok = true;
            bool more = !hit && rtk::next_group(S, grp, h.child, inner, h.masks, stk, lok);
            if (!lok) ok = false;
            if (!more) {
                active = false;
                if (MODE != 1) {
                    if (hit) {
                        T.pend[tag & 3u][tag >> 2] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                } else {
                    out[item] = hit ? 1 : 0;
                }
            }
        }
    }
    if (!ok) atomicExch(err, RT_ERR_CAPACITY);
}

// ── participating media next to the traversal ───────────────────────────────
// A medium's scatter distance depends on the ray alone, so after the closest
// hit each ray takes the nearest medium event before its surface hit (media
// ids follow the primitives: a tie goes to the surface).
// MODE 0: wavefront paths (dense set, wavelength in meta.w)
// MODE 1: photons (queued, wavelength in ray_d.w)
// NOISE: a noise medium's tables in the block's shared memory
#define MEDIA_BLOCK 512
template <int MODE, bool NOISE>
__global__ void __launch_bounds__(MEDIA_BLOCK, 2) k_media(DevScene S, PathState P, const uint32_t* __restrict__ queue,
                                                          const uint32_t* count) {
    extern __shared__ __align__(16) unsigned char media_mem[];
    uint32_t n = *count;
    if (blockIdx.x * blockDim.x >= n) return;             // uniform in the block
    SharedNoise tab{nullptr, nullptr};
    if (NOISE) tab = load_noise(S.media[S.noise_medium], media_mem);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t pid = MODE == 1 ? queue[i] : i;
        float4 ro = P.ray_o[pid], rd = P.ray_d[pid], hv = P.hit[pid];
        float lam = MODE == 1 ? rd.w : __uint_as_float(P.meta[pid].w);
        float3 o = mk(ro.x, ro.y, ro.z), d = mk(rd.x, rd.y, rd.z);
        if (rtk::nan_ray(o, d, 0.001f, INFINITY)) continue;
        float tsurf = __float_as_uint(hv.x) == RT_MISS_REF ? INFINITY : hv.y;
        float tm;
        int med = media_event(S, NOISE ? &tab : nullptr, o, d, lam, 0.001f, tsurf, &tm);
        if (med >= 0) P.hit[pid] = make_float4(__uint_as_float(RT_HIT_MEDIUM_BASE | (uint32_t)med), tm, 0.f, 0.f);
    }
}

// The shadow rays of a scene with media, after the any-hit kernel: a ray whose
// parked contribution was not cancelled scales it by the media's transmittance
// (bvh.rs:532-575).  One thread per ray here; inside the traversal kernel the
// transmittance (16 points × 7 octaves of noise) ran for the one or two lanes
// that had just finished their rays while the rest of the warp waited.
template <bool NOISE>
__global__ void __launch_bounds__(MEDIA_BLOCK, 2) k_media_shadow(DevScene S, PendTargets T,
                                                                 const float4* __restrict__ sq, const uint32_t* count) {
    extern __shared__ __align__(16) unsigned char media_mem[];
    const uint32_t n = *count;
    if (blockIdx.x * blockDim.x >= n) return;             // uniform in the block
    SharedNoise tab{nullptr, nullptr};
    if (NOISE) tab = load_noise(S.media[S.noise_medium], media_mem);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = sq[(size_t)i * 2], b = sq[(size_t)i * 2 + 1];
        const uint32_t tag = __float_as_uint(b.w);
        float4* pp = T.pend[tag & 3u] + (tag >> 2);
        const float4 v = *pp;
        if (v.x == 0.0f && v.y == 0.0f && v.z == 0.0f) continue;
        const float3 o = mk(a.x, a.y, a.z), d = mk(b.x, b.y, b.z);
        if (rtk::nan_ray(o, d, 0.001f, a.w)) continue;
        const float tr = media_transmittance(S, NOISE ? &tab : nullptr, o, d, 0.001f, a.w);
        if (tr < 1.0f) *pp = make_float4(v.x * tr, v.y * tr, v.z * tr, v.w);
    }
}

// API: rays n × 8 (o, d, t_min, t_max) with closest hits already in `out`
// (fill_miss: there is no BVH, every ray starts as a miss)
__global__ void k_media_api(DevScene S, const float* __restrict__ rays, uint32_t n, int4* out, int32_t n_prims,
                            int fill_miss) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* r = rays + (size_t)i * 8;
        float3 o = mk(r[0], r[1], r[2]), d = mk(r[3], r[4], r[5]);
        if (fill_miss) out[i] = make_int4(-1, 0, 0, 0);
        if (rtk::nan_ray(o, d, r[6], r[7])) continue;
        int4 h = out[i];
        float tsurf = h.x < 0 ? r[7] : __int_as_float(h.y);
        float tm;
        int med = media_event(S, nullptr, o, d, 550.0f, r[6], tsurf, &tm);
        if (med >= 0) out[i] = make_int4(n_prims + med, __float_as_int(tm), 0, 0);
    }
}

// API: world.transmittance per ray, from the any-hit flags (NULL: no primitives)
__global__ void k_transmittance_api(DevScene S, const float* __restrict__ rays, uint32_t n,
                                    const uint8_t* __restrict__ occ, float* out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float* r = rays + (size_t)i * 8;
        float3 o = mk(r[0], r[1], r[2]), d = mk(r[3], r[4], r[5]);
        float tr = (occ && occ[i]) ? 0.0f : 1.0f;
        if (tr > 0.0f && S.n_media > 0 && !rtk::nan_ray(o, d, r[6], r[7])) tr = media_transmittance(S, nullptr, o, d, r[6], r[7]);
        out[i] = tr;
    }
}

// ── host launchers ──────────────────────────────────────────────────────────
// ── ray binning before extend (RT_RAY_BINS) ────────────────────────────────
// A counting sort of the set's rays by direction octant and a coarse cell of
// the origin: the extend kernel then takes its rays in bin order, so the lanes
// of a warp start rays that visit similar nodes in a similar order.  Each
// block sorts a contiguous chunk, so neighbours in the set stay neighbours
// within a bin.  The hits do not depend on the order.
#define BIN_BLOCK 256
#define BIN_ITEMS 8
#define BIN_CHUNK (BIN_BLOCK * BIN_ITEMS)
__device__ __forceinline__ uint32_t ray_bin(float4 ro, float4 rd, float3 lo, float3 sc) {
    uint32_t oct = (rd.x < 0.f ? 1u : 0u) | (rd.y < 0.f ? 2u : 0u) | (rd.z < 0.f ? 4u : 0u);
    int cx = min(max(__float2int_rz((ro.x - lo.x) * sc.x), 0), RT_BIN_CELLS - 1);
    int cy = min(max(__float2int_rz((ro.y - lo.y) * sc.y), 0), RT_BIN_CELLS - 1);
    int cz = min(max(__float2int_rz((ro.z - lo.z) * sc.z), 0), RT_BIN_CELLS - 1);
    return ((oct * RT_BIN_CELLS + (uint32_t)cx) * RT_BIN_CELLS + (uint32_t)cy) * RT_BIN_CELLS + (uint32_t)cz;
}
__global__ void __launch_bounds__(BIN_BLOCK) k_bin_count(PathState A, const uint32_t* __restrict__ count, float3 lo,
                                                         float3 sc, uint32_t* hist) {
    __shared__ uint32_t h[RT_NBINS];
    const uint32_t n = *count, base = blockIdx.x * BIN_CHUNK;
    if (base >= n) return;                       // uniform in the block
    for (int b = threadIdx.x; b < RT_NBINS; b += BIN_BLOCK) h[b] = 0;
    __syncthreads();
    for (int k = 0; k < BIN_ITEMS; k++) {
        uint32_t i = base + k * BIN_BLOCK + threadIdx.x;
        if (i < n) atomicAdd(&h[ray_bin(A.ray_o[i], A.ray_d[i], lo, sc)], 1u);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < RT_NBINS; b += BIN_BLOCK)
        if (h[b]) atomicAdd(hist + b, h[b]);
}
__global__ void __launch_bounds__(BIN_BLOCK) k_bin_scatter(PathState A, const uint32_t* __restrict__ count, float3 lo,
                                                           float3 sc, const uint32_t* __restrict__ hist,
                                                           uint32_t* cursor, uint32_t* out) {
    static_assert(RT_NBINS == 2 * BIN_BLOCK, "two bins per thread in the scan");
    typedef cub::BlockScan<uint32_t, BIN_BLOCK> Scan;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ uint32_t h[RT_NBINS], start[RT_NBINS];
    const uint32_t n = *count, base = blockIdx.x * BIN_CHUNK;
    if (base >= n) return;                       // uniform in the block
    // the bins' starts: exclusive prefix of the histogram
    uint32_t v[2] = {hist[2 * threadIdx.x], hist[2 * threadIdx.x + 1]};
    Scan(tmp).ExclusiveSum(v, v);
    start[2 * threadIdx.x] = v[0];
    start[2 * threadIdx.x + 1] = v[1];
    h[2 * threadIdx.x] = 0;
    h[2 * threadIdx.x + 1] = 0;
    __syncthreads();
    uint32_t key[BIN_ITEMS], rank[BIN_ITEMS];
    for (int k = 0; k < BIN_ITEMS; k++) {
        uint32_t i = base + k * BIN_BLOCK + threadIdx.x;
        key[k] = i < n ? ray_bin(A.ray_o[i], A.ray_d[i], lo, sc) : RT_NBINS;
        rank[k] = key[k] < RT_NBINS ? atomicAdd(&h[key[k]], 1u) : 0u;
    }
    __syncthreads();
    // this block's run in each bin
    for (int b = threadIdx.x; b < RT_NBINS; b += BIN_BLOCK)
        if (h[b]) h[b] = start[b] + atomicAdd(cursor + b, h[b]);
    __syncthreads();
    for (int k = 0; k < BIN_ITEMS; k++)
        if (key[k] < RT_NBINS) out[h[key[k]] + rank[k]] = base + k * BIN_BLOCK + threadIdx.x;
}

namespace rth {
// persistent kernels: one wave of resident blocks, or fewer when tuned
int trace_grid(const DevScene& S, int dev_sms, int resident) {
    return dev_sms * (S.trace_per_sm > 0 ? std::min(S.trace_per_sm, resident) : resident);
}

// The layout a launch reads.  RT_NODES_AUTO: the quantised copy where its 80 bytes
// against 208 win more in fetches than its decoding costs, and where its
// closest-hit kernel also splits the leaf tests.
// Renders without convex solids or shapes: from 640 nodes on (720p frames at 8
// samples of triangle soups of 360, 509, 635, 1,577 nodes: full 6.16, 7.15, 7.81,
// 10.23 ms, quantised 6.47, 7.35, 7.84, 9.82; icospheres of 419, 1,920, 5,950,
// 26,712 nodes: 3.53, 4.08, 4.46, 5.17 and 3.57, 4.06, 4.41, 4.98; gem with
// photons, 715 nodes, 30.3 and 29.0).
// Caller-given rays, incoherent as a rule: from 256 (4M random rays, 26, 189, 419,
// 1,920, 26,712 nodes: full 0.71, 1.65, 0.91, 1.24, 1.52 ms, quantised 0.68, 1.48,
// 0.80, 0.96, 1.13; the little it gives below is not taken).
// Renders with such solids, whose kernel does not split: from 32,768 (16-spp frames
// by the unsplit kernels: 5,776 nodes 15.6 and 16.2 ms, 26,984 17.9 and 17.8).
int trace_format(const DevScene& S, bool caller_rays) {
    const uint32_t from = caller_rays ? 256u : S.n_analytic == 0 ? 640u : 32768u;
    if (S.node_format != RT_NODES_AUTO) return S.node_format;
    return S.qnodes && S.n_nodes >= from ? RT_NODES_QUANTISED : RT_NODES_FULL;
}
// the traversal kernels with (ANA) or without analytic solids, by node layout
#define RT_TRACE_ONE(K, MODE, ANA, NF, ...)                                                          \
    K<MODE, ANA, NF><<<trace_grid(S, sms, trace_minb<NF, ANA, K##_any>()), RT_TRACE_BLOCK, 0, st>>>(__VA_ARGS__)
#define RT_TRACE_LAUNCH(K, MODE, ...)                                                                           \
    do {                                                                                                        \
        constexpr bool k_closest_any = false, k_any_any = true;                                                 \
        (void)k_closest_any; (void)k_any_any;                                                                   \
        const int f_ = trace_format(S, MODE == 1);                                                              \
        if (S.n_analytic > 0) {                                                                                 \
            if (f_ == RT_NODES_QUANTISED)  RT_TRACE_ONE(K, MODE, true, RT_NODES_QUANTISED, __VA_ARGS__);        \
            else if (f_ == RT_NODES_WIDE4) RT_TRACE_ONE(K, MODE, true, RT_NODES_WIDE4, __VA_ARGS__);            \
            else                           RT_TRACE_ONE(K, MODE, true, RT_NODES_FULL, __VA_ARGS__);             \
        } else {                                                                                                \
            if (f_ == RT_NODES_QUANTISED)  RT_TRACE_ONE(K, MODE, false, RT_NODES_QUANTISED, __VA_ARGS__);       \
            else if (f_ == RT_NODES_WIDE4) RT_TRACE_ONE(K, MODE, false, RT_NODES_WIDE4, __VA_ARGS__);           \
            else                           RT_TRACE_ONE(K, MODE, false, RT_NODES_FULL, __VA_ARGS__);            \
        }                                                                                                       \
    } while (0)
// the media kernels with (two 64 KB blocks per SM) or without shared noise tables
#define RT_COMMA ,
#define RT_MEDIA_LAUNCH(K, ARG, ...)                                                                              \
    do {                                                                                                          \
        if (S.noise_medium >= 0) {                                                                                \
            cudaFuncSetAttribute(K<ARG true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_NOISE_SMEM);        \
            K<ARG true><<<sms * 2, MEDIA_BLOCK, RT_NOISE_SMEM, st>>>(__VA_ARGS__);                                \
        } else {                                                                                                  \
            K<ARG false><<<sms * 2, MEDIA_BLOCK, 0, st>>>(__VA_ARGS__);                                           \
        }                                                                                                         \
    } while (0)
void launch_trace_closest_api(const DevScene& S, const float* rays, uint32_t n, int4* out, uint32_t* next, int* err,
                              int sms, cudaStream_t st) {
    RT_TRACE_LAUNCH(k_closest, 1, S, PathState{}, nullptr, rays, n, nullptr, next, out, err);
}
void launch_trace_any_api(const DevScene& S, const float* rays, uint32_t n, uint8_t* out, uint32_t* next, int* err,
                          int sms, cudaStream_t st) {
    RT_TRACE_LAUNCH(k_any, 1, S, PendTargets{}, nullptr, rays, n, nullptr, next, out, err);
}
void launch_bin_rays(const PathState& A, const uint32_t* count, uint32_t capacity, float3 lo, float3 scale,
                     uint32_t* bins, uint32_t* out, cudaStream_t st) {
    uint32_t grid = std::max<uint32_t>(1u, (capacity + BIN_CHUNK - 1) / BIN_CHUNK);
    cudaMemsetAsync(bins, 0, 2 * RT_NBINS * sizeof(uint32_t), st);
    k_bin_count<<<grid, BIN_BLOCK, 0, st>>>(A, count, lo, scale, bins);
    k_bin_scatter<<<grid, BIN_BLOCK, 0, st>>>(A, count, lo, scale, bins, bins + RT_NBINS, out);
}
void launch_extend(const DevScene& S, const PathState& P, const uint32_t* queue, const uint32_t* count,
                   uint32_t* next, int* err, int sms, cudaStream_t st) {
    RT_TRACE_LAUNCH(k_closest, 0, S, P, queue, nullptr, 0, count, next, nullptr, err);
}
void launch_shadow(const DevScene& S, const PendTargets& T, const float4* sq, const uint32_t* count,
                   uint32_t* next, int* err, int sms, cudaStream_t st) {
    RT_TRACE_LAUNCH(k_any, 0, S, T, sq, nullptr, 0, count, next, nullptr, err);
    if (S.n_media > 0) RT_MEDIA_LAUNCH(k_media_shadow, , S, T, sq, count);
}
#undef RT_TRACE_LAUNCH
#undef RT_TRACE_ONE
void launch_media(const DevScene& S, const PathState& P, const uint32_t* queue, const uint32_t* count, int sms,
                  cudaStream_t st) {
    if (queue) RT_MEDIA_LAUNCH(k_media, 1 RT_COMMA, S, P, queue, count);
    else       RT_MEDIA_LAUNCH(k_media, 0 RT_COMMA, S, P, nullptr, count);
}
void launch_media_api(const DevScene& S, const float* rays, uint32_t n, int4* out, int32_t n_prims, int fill_miss,
                      int sms, cudaStream_t st) {
    k_media_api<<<sms * 8, 128, 0, st>>>(S, rays, n, out, n_prims, fill_miss);
}
void launch_transmittance_api(const DevScene& S, const float* rays, uint32_t n, const uint8_t* occ, float* out,
                              int sms, cudaStream_t st) {
    k_transmittance_api<<<sms * 8, 128, 0, st>>>(S, rays, n, occ, out);
}
}  // namespace rth
