// Phase-scheduled traversal: the queries of a warp share its instruction
// stream by phases that the warp votes for.
//
// What bounds a traversal kernel here is the issue of divergent instructions:
// testing a node's primitives right after the node ran those tests with about
// 4 of 32 lanes, and the end of a query and the start of the next one with one
// or two.  Here the warp tests either nodes or primitives in a round, and
// finished lanes wait until several can write results and take new queries
// together.
//
// A lane whose node had leaf primitives keeps them and goes on to its next
// node; a second such group waits behind the first (pg2), and the lane then
// takes no further node until its primitives have been tested.  Groups are
// tested in the order in which their nodes were visited, so two primitives at
// exactly the same distance are decided as when every node's primitives are
// tested at once (the first one found stays).  At the top level, whose
// primitives are spheres and group entries that push on the stack, a lane
// waits for its primitives before it takes another node.
//
// What a lane needs in every round is in registers; what it needs now and then
// (the hit so far, the second group, the limits of a visibility query) and the
// lower part of its stack are in its column of shared memory.  The world ray is
// read again from the queue (`load`) where a query enters or leaves a group.
#pragma once
#include "az_trace.cuh"

namespace azd {

// Two floats as one 64-bit operand of the packed FMA.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The watertight kernels call the divisions out of line: inline, beside those of
// wt_setup, they spilled registers of the loop (dense mesh, 16 M samples:
// 58.4 ms a watertight frame inline, 54.4 out of line).
static __device__ __noinline__ f3 safe_inv_call(f3 d) { return safe_inv(d); }

struct WideHits2 {
    uint32_t inner;      // hit inner children, bit = slot ^ perm
    uint32_t lo, hi;     // meta bytes of the hit leaf children, slots 0-3 and 4-7
};

// wide_test with two children per FMA and without a branch per child: a hit is
// a byte of `hb`; the inner ones are permuted by byte and packed by dot
// products, the leaf ones select their meta bytes.
__device__ __forceinline__ WideHits2 wide_test2(const uint4 w0, const uint4 w1, const uint4 w2, const uint4 w3,
                                                const uint4 w4, f3 o, f3 inv, uint32_t perm, float tmax) {
    const float px = __uint_as_float(w0.x), py = __uint_as_float(w0.y), pz = __uint_as_float(w0.z);
    const uint32_t ex = w0.w & 0xFFu, ey = (w0.w >> 8) & 0xFFu, ez = (w0.w >> 16) & 0xFFu, imask = w0.w >> 24;
    const float sx = __uint_as_float(ex << 23) * inv.x, sy = __uint_as_float(ey << 23) * inv.y,
                sz = __uint_as_float(ez << 23) * inv.z;
    // the bias of qbyte_biased folded into the offsets (see wide_test)
    const float ox = __fmaf_rn(-8388608.0f, sx, (px - o.x) * inv.x);
    const float oy = __fmaf_rn(-8388608.0f, sy, (py - o.y) * inv.y);
    const float oz = __fmaf_rn(-8388608.0f, sz, (pz - o.z) * inv.z);
    const unsigned long long s2x = pack2(sx, sx), s2y = pack2(sy, sy), s2z = pack2(sz, sz), o2x = pack2(ox, ox),
                             o2y = pack2(oy, oy), o2z = pack2(oz, oz);
    const bool nx = inv.x < 0.0f, ny = inv.y < 0.0f, nz = inv.z < 0.0f;
    const uint32_t nx0 = nx ? w3.z : w2.x, nx1 = nx ? w3.w : w2.y, fx0 = nx ? w2.x : w3.z, fx1 = nx ? w2.y : w3.w;
    const uint32_t ny0 = ny ? w4.x : w2.z, ny1 = ny ? w4.y : w2.w, fy0 = ny ? w2.z : w4.x, fy1 = ny ? w2.w : w4.y;
    const uint32_t nz0 = nz ? w4.z : w3.x, nz1 = nz ? w4.w : w3.y, fz0 = nz ? w3.x : w4.z, fz1 = nz ? w3.y : w4.w;
    uint32_t hb[2] = {0u, 0u};
#pragma unroll
    for (int s = 0; s < 8; s += 2) {
        const uint32_t k = s & 3;
        auto pair = [&](uint32_t w, unsigned long long sc, unsigned long long of, float &a, float &b) {
            unpack2(fma2(pack2(qbyte_biased(w, k), qbyte_biased(w, k + 1)), sc, of), a, b);
        };
        float tn[2][3], tf[2][3];
        pair(s < 4 ? nx0 : nx1, s2x, o2x, tn[0][0], tn[1][0]);
        pair(s < 4 ? fx0 : fx1, s2x, o2x, tf[0][0], tf[1][0]);
        pair(s < 4 ? ny0 : ny1, s2y, o2y, tn[0][1], tn[1][1]);
        pair(s < 4 ? fy0 : fy1, s2y, o2y, tf[0][1], tf[1][1]);
        pair(s < 4 ? nz0 : nz1, s2z, o2z, tn[0][2], tn[1][2]);
        pair(s < 4 ? fz0 : fz1, s2z, o2z, tf[0][2], tf[1][2]);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float n = fmaxf(max3f(tn[j][0], tn[j][1], tn[j][2]), 0.0f);
            const float f = fminf(min3f(tf[j][0], tf[j][1], tf[j][2]), tmax) * 1.00000095367431640625f;
            if (n <= f) hb[s >> 2] |= 1u << (8 * (k + j));
        }
    }
    WideHits2 h;
    // imask's bits spread to the bytes 0..3
    const uint32_t in0 = hb[0] & (((imask & 15u) * 0x00204081u) & 0x01010101u);
    const uint32_t in1 = hb[1] & (((imask >> 4) * 0x00204081u) & 0x01010101u);
    const uint32_t sel = 0x3210u ^ (perm * 0x1111u);
    h.inner = __dp4a(__byte_perm(in0, in1, sel), 0x08040201u,
                     __dp4a(__byte_perm(in0, in1, sel ^ 0x4444u), 0x80402010u, 0u));
    h.lo = w1.z & (hb[0] * 255u);   // inner children and empty slots have meta 0
    h.hi = w1.w & (hb[1] * 255u);
    return h;
}

// A lane's column of the block's shared memory.
constexpr int kSharedStack = 8;   // stack entries in shared memory, the rest in local memory
enum : int { LM_PG2 = 0, LM_PG2_LO, LM_PG2_HI, LM_GROUP, LM_PRIM, LM_A, LM_B, LM_C, LM_D, LM_COUNT };
template <int BLOCK>
struct PhaseShared {
    uint2 stack[kSharedStack][BLOCK];
    uint32_t mem[LM_COUNT][BLOCK];
};

// MULTI: lanes of a warp may trace different scenes; a lane keeps the two array
// addresses it needs in every round instead of reading them from its scene's
// record each time.
template <QueryKind KIND, bool WT, bool SPH, int BLOCK, bool MULTI>
struct PhaseTracer {
    PhaseShared<BLOCK> &sh;
    uint2 *deep;                 // stack entries beyond the shared ones: an array of the caller, so that this
                                 // object's members stay in registers
    f3 o, d, inv;                // ray in the current space
    float time;
    uint32_t perm;               // a child's bit is slot ^ perm; the highest bit is visited first
    float tcur;                  // pruning distance in the current space
    float bl_t;                  // nearest local hit of this group's visit (Q_ANY: or the limit of one that counts)
    uint32_t ng_base, ng_bits;   // current node group
    uint32_t pg_base, pg_lo, pg_hi;   // primitives to test next: meta bytes of leaf children
    int sp;
    bool in_blas, pg2;
    bool stopped, occluded;      // Q_ANY: stopped at a hit to be confirmed; something lies closer than tmax
    WtRay wt;
    const WideNode *own_nodes;   // MULTI
    const float4 *own_tris;

    __device__ __forceinline__ PhaseTracer(PhaseShared<BLOCK> &s, uint2 *lower) : sh(s), deep(lower) {}
    __device__ __forceinline__ uint32_t &mem(int k) { return sh.mem[k][threadIdx.x]; }
    __device__ __forceinline__ float memf(int k) { return __uint_as_float(mem(k)); }
    __device__ __forceinline__ uint2 top() { return sp <= kSharedStack ? sh.stack[sp - 1][threadIdx.x] : deep[sp - 1 - kSharedStack]; }
    __device__ __forceinline__ void put(uint32_t x, uint32_t y) {
        if (sp < kSharedStack) sh.stack[sp][threadIdx.x] = make_uint2(x, y);
        else deep[sp - kSharedStack] = make_uint2(x, y);
        sp++;
    }
    __device__ __forceinline__ void push(uint32_t x, uint32_t y, uint32_t *err) {
        if (sp < AZD_WSTACK) put(x, y);
        else atomicOr(err, 2u);
    }
    __device__ __forceinline__ Ray ray() const {
        Ray r;
        r.o = o;
        r.d = d;
        r.time = SPH ? time : 0.0f;   // only the top-level sphere test reads it
        return r;
    }

    __device__ __forceinline__ void set_ray(const Ray &r) {
        o = r.o;
        d = r.d;
        if (SPH) time = r.time;
        inv = WT ? safe_inv_call(d) : safe_inv(d);
        perm = octant_of(d) ^ (KIND == Q_ANY ? 0u : 7u);
        if (WT) wt = wt_setup(d);
    }
    __device__ __forceinline__ void start(uint32_t root) {
        ng_base = root;
        ng_bits = root == 0xFFFFFFFFu ? 0u : ((1u << 8) | (1u << perm));
    }

    // tmax, skip: of a visibility query (Q_ANY)
    __device__ __forceinline__ void init(const DevScene &S, const Ray &wr, float tmax, uint32_t skip) {
        if (KIND == Q_ANY) {
            mem(LM_A) = __float_as_uint(tmax);
            mem(LM_B) = skip;
        } else {
            mem(LM_A) = __float_as_uint(FLT_MAX);   // best.t, tl, prim, ent
            mem(LM_B) = 0u;
            mem(LM_C) = 0xFFFFFFFFu;
            mem(LM_D) = 0xFFFFFFFFu;
        }
        if (MULTI) {
            own_nodes = S.wnodes;
            own_tris = WT ? (const float4 *)S.tri_verts : (const float4 *)S.tris;
        }
        bl_t = FLT_MAX;
        pg_base = pg_lo = pg_hi = 0u;
        ng_base = ng_bits = 0u;
        sp = 0;
        in_blas = pg2 = stopped = occluded = false;
        if (S.tlas_single_group != 0xFFFFFFFFu) {
            enter_group(S, wr, S.tlas_single_group);
        } else {
            set_ray(wr);
            tcur = KIND == Q_ANY ? tmax : FLT_MAX;
            start(S.tlas_root);
        }
    }

    __device__ __forceinline__ void enter_group(const DevScene &S, const Ray &wr, uint32_t gi) {
        const DevGroup &g = S.groups[gi];
        if (g.root == 0xFFFFFFFFu) return;
        mem(LM_GROUP) = gi;
        put(0u, AZD_E_EXIT);   // room was kept when the group's entry was pushed
        const float wlim = memf(LM_A);
        tcur = FLT_MAX;
        bl_t = FLT_MAX;
        if (g.raw) {
            set_ray(wr);
            if (wlim < FLT_MAX) tcur = wlim + 1e-30f;
        } else if (g.identity) {
            set_ray(local_ray_identity(wr));
            if (wlim < FLT_MAX) {
                tcur = wlim * group_t_scale(g, wr.d) + 1e-30f;
                if (KIND == Q_ANY) bl_t = tcur;   // hits from here on are out of a visibility query's range
            }
        } else {
            const GroupRay gr = group_ray_call(S.groups + gi, wr);
            set_ray(gr.r);
            if (wlim < FLT_MAX) tcur = wlim * gr.scale + 1e-30f;
        }
        if (KIND == Q_CLOSEST) mem(LM_PRIM) = 0xFFFFFFFFu;
        in_blas = true;
        start(g.root);
    }

    // azimuth's instance path keeps the nearest local hit of a mesh and
    // recomputes its world t (src/azimuth_main.cpp:256-276)
    __device__ __forceinline__ void take_group_hit(const DevScene &S, const Ray &wr, float eps) {
        if (KIND == Q_CLOSEST && mem(LM_PRIM) != 0xFFFFFFFFu) {
            const float w = group_world_t(S.groups[mem(LM_GROUP)], wr, ray(), bl_t);
            if (w > eps && w < memf(LM_A)) {
                mem(LM_A) = __float_as_uint(w);
                mem(LM_B) = __float_as_uint(bl_t);
                mem(LM_C) = mem(LM_PRIM);
                mem(LM_D) = S.tri_attr[mem(LM_PRIM)].entity;
            }
        }
    }

    // Q_ANY: a lane that stopped at a triangle decides whether its
    // world t is in range; returns false when the query has to go on.
    __device__ __forceinline__ bool confirm(const DevScene &S, const Ray &wr, float eps) {
        if (!stopped) return true;
        stopped = false;
        const float w = group_world_t(S.groups[mem(LM_GROUP)], wr, ray(), bl_t);
        occluded = w > eps && w < memf(LM_A);
        return occluded;
    }

    // The result of a closest-hit query as the hit queue holds it.
    __device__ __forceinline__ uint4 hit() { return make_uint4(mem(LM_A), mem(LM_B), mem(LM_C), mem(LM_D)); }

    // Ends a query that exceeded its step limit.
    __device__ __forceinline__ void abandon() {
        ng_bits = pg_lo = pg_hi = 0u;
        pg2 = false;
        sp = 0;
    }

    __device__ __forceinline__ bool has_prims() const { return (pg_lo | pg_hi) != 0u; }
    __device__ __forceinline__ bool wants_node() const {
        return (ng_bits & 0xFFu) && !pg2 && (in_blas || !has_prims());
    }

    // Gives a lane without nodes its next stack entry.  Returns true when the
    // query is finished; the exit of the last group is left to the caller.
    template <typename LOAD>
    __device__ __forceinline__ bool refill(const DevScene &S, LOAD load, float eps) {
        if ((ng_bits & 0xFFu) || pg2) return false;
        if (sp == 0) return !has_prims();
        const uint2 e = top();
        if (e.y < AZD_E_GROUP) {
            if (in_blas || !has_prims()) {
                sp--;
                ng_base = e.x;
                ng_bits = e.y;
            }
            return false;
        }
        if (has_prims()) return false;   // the ray's space changes after its primitives
        sp--;
        if (e.y == AZD_E_EXIT) {
            if (sp == 0) return true;
            const Ray wr = load();
            take_group_hit(S, wr, eps);
            in_blas = false;
            set_ray(wr);
            tcur = memf(LM_A);
        } else {
            enter_group(S, load(), e.x);
        }
        return false;
    }

    // Visits the group's next node.
    __device__ __forceinline__ void node(const DevScene &S, uint32_t *err) {
        const uint32_t key = 31u - __clz(ng_bits & 0xFFu);
        const uint32_t slot = key ^ perm, imask = ng_bits >> 8;
        const uint32_t n = ng_base + __popc(imask & ((1u << slot) - 1u));
        const uint4 *np = reinterpret_cast<const uint4 *>((MULTI ? own_nodes : S.wnodes) + n);
        const uint4 w0 = __ldg(np + 0), w1 = __ldg(np + 1), w2 = __ldg(np + 2), w3 = __ldg(np + 3),
                    w4 = __ldg(np + 4);
        ng_bits ^= 1u << key;
        if (ng_bits & 0xFFu) push(ng_base, ng_bits, err);
        const WideHits2 h = wide_test2(w0, w1, w2, w3, w4, o, inv, perm, tcur);
        ng_base = w1.x;
        ng_bits = h.inner | ((w0.w >> 24) << 8);
        if (h.lo | h.hi) {
            if (has_prims()) {
                mem(LM_PG2) = w1.y;
                mem(LM_PG2_LO) = h.lo;
                mem(LM_PG2_HI) = h.hi;
                pg2 = true;
            } else {
                pg_base = w1.y;
                pg_lo = h.lo;
                pg_hi = h.hi;
            }
        }
    }

    // Tests the next primitive.  Returns true when the lane has to stop (Q_ANY).
    template <typename LOAD>
    __device__ __forceinline__ bool prim(const DevScene &S, LOAD load, bool cull, float eps, uint32_t *err) {
        // the lowest meta byte: count << 5 | offset; one primitive less at the next offset
        const uint32_t w = pg_lo ? pg_lo : pg_hi;
        const uint32_t at = (__ffs(w) - 1u) & 24u;
        const uint32_t b = (w >> at) & 0xFFu;
        const uint32_t left = w - ((b >= 64u ? 31u : b) << at);
        if (pg_lo) pg_lo = left;
        else pg_hi = left;
        const uint32_t pi = pg_base + (b & 31u);
        if (!has_prims() && pg2) {
            pg_base = mem(LM_PG2);
            pg_lo = mem(LM_PG2_LO);
            pg_hi = mem(LM_PG2_HI);
            pg2 = false;
        }
        if (in_blas) {
            float t, bt, gm;
            bool hit;
            if (WT) hit = tri_test_wt(load_tri_verts(MULTI ? (const DevTriVerts *)own_tris : S.tri_verts, pi), ray(), wt, cull, eps, bl_t, t);
            else hit = tri_test(load_tri(MULTI ? (const DevTri *)own_tris : S.tris, pi), ray(), cull, eps, bl_t, t, bt, gm);
            if (!hit) return false;
            if (KIND == Q_ANY) {
                // a primitive of the skipped entity is ignored; its owner is
                // looked up only for the few primitives that are hit
                const uint32_t skip = mem(LM_B);
                if (skip != 0xFFFFFFFFu && __ldg(&S.tri_attr[pi].entity) == skip) return false;
            } else {
                tcur = fminf(tcur, t);
            }
            bl_t = t;
            if (KIND == Q_ANY) stopped = true;
            else mem(LM_PRIM) = pi;
            return KIND == Q_ANY;
        }
        const uint32_t p = __ldg(S.tlas_prims + pi);
        if (p & AZD_TLAS_GROUP) {
            push(p & ~AZD_TLAS_GROUP, AZD_E_GROUP, err);   // entered when popped
        } else if (SPH && (KIND != Q_ANY || p != mem(LM_B)) && S.ents[p].type == ENT_SPHERE) {
            const SphereHit s = sphere_hit(S.ents + p, ray(), eps);
            if (s.hit && s.t_world < memf(LM_A)) {
                if (KIND == Q_ANY) {
                    occluded = true;
                    return true;
                }
                mem(LM_A) = __float_as_uint(s.t_world);
                mem(LM_B) = __float_as_uint(s.t_local);
                mem(LM_C) = 0xFFFFFFFFu;
                mem(LM_D) = p;
                tcur = s.t_world;
            }
        }
        return false;
    }
};

}  // namespace azd
