// Persistent traversal of the compressed 8-wide layout (RB2_NODE_ORDER_CW8,
// node format in rb2_cw8.cpp), after Ylitie, Karras and Laine, "Efficient
// Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs" (HPG 2017).
//
// Per lane: a node group (child_base of a visited node and a mask of its hit
// inner children, bits 24-31 in octant-permuted order, the node's inner-child
// mask in bits 0-7), a triangle group (tri_base, the node's triangle mask and
// the hit triangles among its bits) and a stack of node groups.  A node test
// yields an 8-bit mask of hit slots; a table lookup and three multiplications
// turn it into both groups (instead of the paper's per-child meta-byte decoding).  The warp walks nodes
// until every busy lane holds triangles (the counterpart of the binary
// kernel's postponed leaf) or too few lanes still want nodes, then tests
// triangles, then refills lanes from the
// ray source as the binary kernel does (same RaySource policy, same dynamic
// fetch).  Triangles are the binary layout's Woop rows with the same test
// arithmetic, so an accepted hit has the same t, u, v bits; boxes are
// conservative, so the closest hit equals the binary traversal's except for
// exact ties in t.
#pragma once

#include "rb2_traverse.cuh"

#include <string.h>

namespace rb2dev {

// Node groups on the stack: at most one per wide level.  The host refuses a
// layout deeper than this (rb2_tracer_set_node_order).
constexpr int kStackSizeCw8 = 72;
// Words of a node on the device: the layout's 20 (rb2_cw8.cpp), with the origin
// less 32768 cells (the plane bias, below) in words 0-2, then the three scales as
// floats and an unused word, so that a node is three aligned 32-byte sectors read
// with three 256-bit loads (five 128-bit loads of 80-byte nodes touch three
// sectors too).  Made from the layout by cw8_device_node.
constexpr uint32_t kCw8NodeWords = 24;

// Two quantized planes (bytes 2h and 2h + 1 of w) as floats 32768 + q: each
// byte is moved into bits 8-15 of the float 32768 (0x47000000), whose unit in
// the last place there is 1, so one byte permute yields the plane exactly.
// The 32768 cells are taken off the node's origin, so the slab offset holds
// them (the layout widens every box by 2^-14 of its node, 2^-6 cells, for the
// rounding of the biased origin and of that offset, 2^-9 cells each).
constexpr float kCw8PlaneBias = 32768.0f;

// One device node from the layout's 20 words.
inline void cw8_device_node(const uint32_t* layout, uint32_t* node)
{
    for (uint32_t k = 0; k < kCw8NodeWords; k++) node[k] = k < 20 ? layout[k] : 0u;
    for (int a = 0; a < 3; a++) {
        const uint32_t scale_bits = ((layout[3] >> (8 * a)) & 0xFFu) << 23;
        float org, scale;
        memcpy(&org, &layout[a], 4);
        memcpy(&scale, &scale_bits, 4);
        org -= kCw8PlaneBias * scale;
        memcpy(&node[a], &org, 4);
        node[20 + a] = scale_bits;
    }
}
__device__ __forceinline__ float cw8_plane(uint32_t w, int b)
{
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7504u | ((uint32_t)b << 4)));
}
__device__ __forceinline__ float2 cw8_planes(uint32_t w, int h)
{
    return make_float2(cw8_plane(w, 2 * h), cw8_plane(w, 2 * h + 1));
}

// Two IEEE single-precision FMAs in one paired instruction (sm_100 f32x2).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    unsigned long long ra, rb, rc, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(rd));
    return r;
}

// Per-thread words of a ray that only the triangle phase and the end of the ray
// need, kept in shared memory so that the node phase has their registers:
// volatile accesses, so that the compiler does not keep copies in registers.
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sts_ray(uint32_t a, float x, float y, float z, uint32_t w)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void lds_ray(uint32_t a, float& x, float& y, float& z, uint32_t& w)
{
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=f"(x), "=f"(y), "=f"(z), "=r"(w) : "r"(a) : "memory");
}
__device__ __forceinline__ void sts_ptr(uint32_t a, const float4* p)
{
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(p) : "memory");
}
__device__ __forceinline__ const float4* lds_ptr(uint32_t a)
{
    unsigned long long v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return reinterpret_cast<const float4*>(v);
}

// Woop test of one triangle (the binary leaf loop's arithmetic); shortens hitT
// and returns true when it accepts.
__device__ __forceinline__ bool cw8_triangle(const float4* wp, float ox, float oy, float oz, float dx, float dy,
                                             float dz, float tmin, float& hitT)
{
    const float4 v00 = __ldg(wp + 0);
    const float4 v11 = __ldg(wp + 1);
    const float4 v22 = __ldg(wp + 2);
    const float Oz = __fmaf_rn(-oz, v00.z, __fmaf_rn(-oy, v00.y, __fmaf_rn(-ox, v00.x, v00.w)));
    const float Dz = __fmaf_rn(dz, v00.z, __fmaf_rn(dy, v00.y, __fmul_rn(dx, v00.x)));
    const float t = __fmul_rn(Oz, __frcp_rn(Dz));  // IEEE 1 / Dz, as __fdiv_rn(1, Dz)
    if (!(t > tmin && t < hitT)) return false;
    const float Ox = __fmaf_rn(oz, v11.z, __fmaf_rn(oy, v11.y, __fmaf_rn(ox, v11.x, v11.w)));
    const float Dx = __fmaf_rn(dz, v11.z, __fmaf_rn(dy, v11.y, __fmul_rn(dx, v11.x)));
    const float u = __fmaf_rn(t, Dx, Ox);
    if (!(u >= 0.0f)) return false;
    const float Oy = __fmaf_rn(oz, v22.z, __fmaf_rn(oy, v22.y, __fmaf_rn(ox, v22.x, v22.w)));
    const float Dy = __fmaf_rn(dz, v22.z, __fmaf_rn(dy, v22.y, __fmul_rn(dx, v22.x)));
    const float v = __fmaf_rn(t, Dy, Oy);
    if (!(v >= 0.0f && __fadd_rn(u, v) <= 1.0f)) return false;
    hitT = t;
    return true;
}

// What bounds it: a node visit issues about 210 warp instructions (130 on the
// ALU pipe, at half rate), a triangle test 79, at 17 to 21 busy lanes; issue
// slots (61 %), the ALU (56 %) and the L1 data pipe (63 to 72 %) share the limit, so
// more resident warps alone do not help (a 56-register budget, 36 warps per SM,
// measured 2 % slower).  The node phase therefore keeps out of registers what
// only triangles and the ray's end need (origin, direction, job, Woop
// pointer: shared memory, 40 bytes per thread; 8 bytes spilled at 64 registers
// in the job kernel, none in the integrators'),
// reads a node with three loads, spreads leaf bits with multiplications
// (FMA pipe) instead of a second shared table, and reads each child's hit from the
// sign of a subtraction.  500k triangles, 1M incoherent rays: occlusion 263 -> 244
// us, closest hit 338 -> 312 us; batch of 16 scenes x 262,144 rays 840 -> 803 us.
// Tried and slower: testing the warp's pending (ray, triangle) pairs with all
// lanes (3 to 6 %), leaving some triangles pending to return to nodes (2 to
// 20 %), pushing a group only when the next node yields inner hits (2 %),
// loading the second and third Woop row only after the first test (4 %).
//
// node_threshold: a node phase also ends, so that pending triangle groups are
// tested, once fewer than this many lanes still want nodes while some lane
// holds triangles (0 or 1: only when no lane wants nodes).  Testing triangles
// earlier shortens the lanes' hit distances sooner and keeps more lanes busy
// in the node phases; a lane's own order of node visits and triangle tests is
// unchanged, so results do not depend on it.  It is capped at half the busy
// lanes, so that a warp with few of them does not end every node phase at its
// first leaf: 100,000 rays 87 -> 81 us, 1M closest 321 -> 317 us, AO frame 494 ->
// 485 us, BDPT 1280 x 720 x 4 18.40 -> 18.12 ms (a cap of 3/8 costs 1 % on the
// path-traced frame).  Source::kLateCap: apply the cap at the break instead of
// keeping its value across the phase; the job kernel, short of a register,
// is 0.7 % faster so on a batch, the integrators' are 1.5 to 2 % slower.
template <int BLOCK, class Source>
__device__ __forceinline__ void persistent_trace_cw8(Source& src, uint32_t fetch_threshold, uint32_t node_threshold,
                                                     unsigned int* status)
{
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    uint2 stack[kStackSizeCw8];
    int sp = 0;
    Lane L;
    L.hitIndex = -1;
    uint32_t ng_base = 0, ng_bits = 0, tg_base = 0, tg_bits = 0, tg_mask = 0;
    uint32_t tg2_base = 0, tg2_bits = 0, tg2_mask = 0;  // a second pending triangle group
    uint32_t oct_inv = 0;  // 7 xor the ray's direction octant (set when a ray is fetched)
    bool has_ray = false, retired = lane >= src.lanes();

    // Table shared by the block: s_perm[o][m] moves bit s of an 8-bit slot mask
    // to bit s ^ o (inner children in ray-octant order).
    // Each step swaps bit groups of four masks at once.
    __shared__ uint32_t s_perm_words[8 * 64];
    const uint8_t* s_perm = reinterpret_cast<const uint8_t*>(s_perm_words);
    for (uint32_t i = threadIdx.x; i < 8u * 64u; i += BLOCK) {
        uint32_t w = (i & 63u) * 0x04040404u + 0x03020100u;
        if (i & 64u) w = ((w & 0x55555555u) << 1) | ((w >> 1) & 0x55555555u);
        if (i & 128u) w = ((w & 0x33333333u) << 2) | ((w >> 2) & 0x33333333u);
        if (i & 256u) w = ((w & 0x0F0F0F0Fu) << 4) | ((w >> 4) & 0x0F0F0F0Fu);
        s_perm_words[i] = w;
    }
    // Origin and tag, direction and ray index, Woop rows of the thread's ray.
    __shared__ float4 s_org[BLOCK], s_dir[BLOCK];
    __shared__ uint2 s_woop[BLOCK];
    const uint32_t a_org = smem_addr(&s_org[threadIdx.x]), a_dir = smem_addr(&s_dir[threadIdx.x]),
                   a_woop = smem_addr(&s_woop[threadIdx.x]);
    __syncthreads();

    for (;;) {
        // ---- refill: lanes without a ray claim the next slots from the queue.
        const bool need = !has_ray && !retired;
        const unsigned needm = __ballot_sync(kFull, need);
        if (needm) {
            const int leader = __ffs(needm) - 1;
            unsigned long long b1 = 0, b2 = 0;
            unsigned n1 = 0;
            claim_slots(src, (int)lane == leader, leader, (unsigned)__popc(needm), b1, n1, b2);
            if (need) {
                const unsigned rank = (unsigned)__popc(needm & lt_mask);
                const unsigned long long slot = rank < n1 ? b1 + rank : b2 + (rank - n1);
                const int r = src.fetch(slot, L);
                if (r == 0) {
                    retired = true;
                } else if (r > 0) {
                    sts_ray(a_org, L.ox, L.oy, L.oz, L.tag);
                    sts_ray(a_dir, L.dx, L.dy, L.dz, L.ray);
                    if constexpr (!Source::kOneScene) sts_ptr(a_woop, L.woop);
                    sp = 0;
                    ng_base = 0;             // the root: node 0, reached through bit 31
                    // with an empty inner-child mask; no node for a ray without an interval,
                    // since a NaN box distance counts as a hit (below)
                    ng_bits = L.tmin == L.tmin && L.hitT == L.hitT ? 0x80000000u : 0u;
                    tg_bits = 0;
                    tg2_bits = 0;
                    oct_inv = 7u ^ ((__float_as_uint(L.idx) >> 31) | ((__float_as_uint(L.idy) >> 31) << 1) |
                                    ((__float_as_uint(L.idz) >> 31) << 2));
                    has_ray = true;
                }
            }
        }
        if (__all_sync(kFull, retired)) break;

        for (;;) {
            const unsigned busy = (unsigned)__popc(__ballot_sync(kFull, has_ray));
            if (busy == 0) break;
            const unsigned node_lanes = Source::kLateCap ? node_threshold : min(node_threshold, busy >> 1);
            // ---- nodes, until every busy lane holds triangles or is done, or
            //      fewer than node_threshold lanes want nodes while some lane
            //      holds triangles.
            for (;;) {
                const bool in = has_ray && tg2_bits == 0 && (ng_bits > 0x00FFFFFFu || sp > 0);
                const unsigned inm = __ballot_sync(kFull, in);
                if (inm == 0) break;
                if ((unsigned)__popc(inm) < node_lanes &&
                    (!Source::kLateCap ||
                     2u * (unsigned)__popc(inm) < (unsigned)__popc(__ballot_sync(kFull, has_ray))) &&
                    __any_sync(kFull, has_ray && tg_bits != 0))
                    break;
                if (in) {
                    if (ng_bits <= 0x00FFFFFFu) {
                        --sp;
                        ng_base = stack[sp].x;
                        ng_bits = stack[sp].y;
                    }
                    const uint32_t k = 31u - (uint32_t)__clz(ng_bits);
                    ng_bits &= ~(1u << k);
                    const uint32_t slot = (k - 24u) ^ oct_inv;
                    const uint32_t node = ng_base + (uint32_t)__popc(ng_bits & ((1u << slot) - 1u));
                    bool ok = true;
                    if (ng_bits > 0x00FFFFFFu) {
                        if (sp >= kStackSizeCw8) {
                            // Unreachable for layouts whose depth was validated; a corrupt
                            // layout abandons the ray and reports it.
                            atomicOr(status, kStatusStack);
                            ok = false;
                        } else {
                            stack[sp].x = ng_base;
                            stack[sp].y = ng_bits;
                            ++sp;
                        }
                    }
                    if (!ok) {
                        L.hitIndex = -1;
                        ng_bits = 0;
                        sp = 0;
                    } else {
                        const float4* np =
                            (Source::kOneScene ? src.nodes : L.nodes) + (size_t)node * (kCw8NodeWords / 4);
                        float4 h0, h1, qx, qy, qz, sc;
                        ldg_v8(np + 0, h0, h1);
                        ldg_v8(np + 2, qx, qy);
                        ldg_v8(np + 4, qz, sc);
                        const float sx = __fmul_rn(sc.x, L.idx), sy = __fmul_rn(sc.y, L.idy),
                                    sz = __fmul_rn(sc.z, L.idz);
                        // Slab offsets of the biased origin (planes arrive as 32768 + q cells).
                        const float ax = __fmaf_rn(h0.x, L.idx, -L.oodx), ay = __fmaf_rn(h0.y, L.idy, -L.oody),
                                    az = __fmaf_rn(h0.z, L.idz, -L.oodz);
                        // Near and far plane words per axis (the high plane is near for a
                        // negative direction), children 0-3 in the first word, 4-7 in the second.
                        const bool rx = L.idx < 0.0f, ry = L.idy < 0.0f, rz = L.idz < 0.0f;
                        const uint32_t nx0 = __float_as_uint(rx ? qx.z : qx.x), nx1 = __float_as_uint(rx ? qx.w : qx.y);
                        const uint32_t fx0 = __float_as_uint(rx ? qx.x : qx.z), fx1 = __float_as_uint(rx ? qx.y : qx.w);
                        const uint32_t ny0 = __float_as_uint(ry ? qy.z : qy.x), ny1 = __float_as_uint(ry ? qy.w : qy.y);
                        const uint32_t fy0 = __float_as_uint(ry ? qy.x : qy.z), fy1 = __float_as_uint(ry ? qy.y : qy.w);
                        const uint32_t nz0 = __float_as_uint(rz ? qz.z : qz.x), nz1 = __float_as_uint(rz ? qz.w : qz.y);
                        const uint32_t fz0 = __float_as_uint(rz ? qz.x : qz.z), fz1 = __float_as_uint(rz ? qz.y : qz.w);
                        // Slots whose box the ray misses: the sign bits of far less near distance
                        // (a subtraction on the FMA pipe and a shift, where a comparison and a
                        // conditional OR are two ALU instructions), the last slot first.  A NaN
                        // difference has a clear sign: equal infinities count as hits, as they
                        // compare; tmin and hitT are numbers here.
                        uint32_t miss = 0;
                        const float2 sx2 = make_float2(sx, sx), sy2 = make_float2(sy, sy), sz2 = make_float2(sz, sz);
                        const float2 ax2 = make_float2(ax, ax), ay2 = make_float2(ay, ay), az2 = make_float2(az, az);
#pragma unroll
                        for (int s = 6; s >= 0; s -= 2) {
                            const int w = s >> 2, hh = (s >> 1) & 1;
                            const float2 nx = cw8_planes(w ? nx1 : nx0, hh), fx = cw8_planes(w ? fx1 : fx0, hh);
                            const float2 ny = cw8_planes(w ? ny1 : ny0, hh), fy = cw8_planes(w ? fy1 : fy0, hh);
                            const float2 nz = cw8_planes(w ? nz1 : nz0, hh), fz = cw8_planes(w ? fz1 : fz0, hh);
                            // Slab distances of the two children, one paired FMA per plane.
                            const float2 tnx2 = fma2(nx, sx2, ax2), tfx2 = fma2(fx, sx2, ax2);
                            const float2 tny2 = fma2(ny, sy2, ay2), tfy2 = fma2(fy, sy2, ay2);
                            const float2 tnz2 = fma2(nz, sz2, az2), tfz2 = fma2(fz, sz2, az2);
#pragma unroll
                            for (int e = 1; e >= 0; e--) {
                                const float tnx = e ? tnx2.y : tnx2.x, tfx = e ? tfx2.y : tfx2.x;
                                const float tny = e ? tny2.y : tny2.x, tfy = e ? tfy2.y : tfy2.x;
                                const float tnz = e ? tnz2.y : tnz2.x, tfz = e ? tfz2.y : tfz2.x;
                                const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, L.tmin));
                                const float tf = fminf(fminf(tfx, tfy), fminf(tfz, L.hitT));
                                miss = __funnelshift_l(__float_as_uint(__fsub_rn(tf, tn)), miss, 1);
                            }
                        }
                        const uint32_t hm = ~miss & 0xFFu;
                        // Hit inner slots, octant-permuted, into bits 24-31 (above the
                        // node's inner-child mask); hit leaf slots' triangles from the
                        // node's triangle mask (inner and empty slots have no bits there).
                        const uint32_t imask = __float_as_uint(h0.w) >> 24;
                        ng_base = __float_as_uint(h1.x);
                        ng_bits = ((uint32_t)s_perm[(oct_inv << 8) | (hm & imask)] << 24) | imask;
                        // Bit s to bit 3s: doubling the gaps, each step a multiplication.
                        uint32_t spread = (hm * 0x101u) & 0x00F00Fu;
                        spread = (spread * 0x11u) & 0x0C30C3u;
                        spread = (spread * 0x5u) & 0x249249u;
                        const uint32_t tmask = __float_as_uint(h1.z), tbits = (spread * 7u) & tmask;
                        if (tbits) {
                            if (tg_bits == 0) {
                                tg_base = __float_as_uint(h1.y); tg_mask = tmask; tg_bits = tbits;
                            } else {
                                tg2_base = __float_as_uint(h1.y); tg2_mask = tmask; tg2_bits = tbits;
                            }
                        }
                    }
                }
            }

            // ---- triangles of the current group, then finish lanes with no work left.
            if (tg_bits != 0) {
                float ox, oy, oz, dx, dy, dz;
                uint32_t tag, ray;
                lds_ray(a_org, ox, oy, oz, tag);
                lds_ray(a_dir, dx, dy, dz, ray);
                const float4* woop;
                if constexpr (Source::kOneScene) woop = src.woop;
                else woop = lds_ptr(a_woop);
                for (;;) {
                    if (tg_bits == 0) {
                        if (tg2_bits == 0) break;
                        tg_base = tg2_base; tg_mask = tg2_mask; tg_bits = tg2_bits; tg2_bits = 0;
                    }
                    const int i = __ffs(tg_bits) - 1;
                    tg_bits &= tg_bits - 1u;
                    // Triangle bit i is the node's (mask bits below i)-th triangle.
                    const int row = 3 * (int)(tg_base + (uint32_t)__popc(tg_mask & ((1u << i) - 1u)));
                    if (cw8_triangle(woop + row, ox, oy, oz, dx, dy, dz, L.tmin, L.hitT)) {
                        L.hitIndex = row;
                        if ((tag >> 30) != kClosest) {
                            tg_bits = 0;
                            tg2_bits = 0;
                            ng_bits = 0;
                            sp = 0;
                        }
                    }
                }
            }
            if (has_ray && ng_bits <= 0x00FFFFFFu && sp == 0) {
                Lane F;
                lds_ray(a_org, F.ox, F.oy, F.oz, F.tag);
                lds_ray(a_dir, F.dx, F.dy, F.dz, F.ray);
                if constexpr (Source::kOneScene) F.woop = src.woop;
                else F.woop = lds_ptr(a_woop);
                F.tmin = L.tmin;
                F.hitT = L.hitT;
                F.hitIndex = L.hitIndex;
                src.finish(F);
                has_ray = false;
            }
            // Dynamic fetch (kepler_dynamic_fetch.h:308-310).
            if ((unsigned)__popc(__ballot_sync(kFull, has_ray)) < fetch_threshold) break;
        }
    }
}

}  // namespace rb2dev
