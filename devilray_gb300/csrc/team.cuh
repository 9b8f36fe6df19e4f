// team.cuh -- traversal of the compressed 8-wide BVH by teams of lanes, for
// launches with too few rays to fill the chip with one ray per lane.
//
// A team of G lanes (G = 4 or 8) carries one ray: lane k of the team tests the
// 8 / G child boxes at the traversal positions k, k + G of each node (slot =
// position ^ octant, so the ballot of the hits is already in the ray's order),
// and its own slots' leaf triangles, so a node step is a chain of a few dozen
// instructions instead of the several hundred of a lane that tests 8 boxes and
// waits for 31 other rays. The rays' state is the same in every lane of the
// team. Boxes, bounds and the candidate rule are those of trace_wide.cuh (the
// slab times are the same FMAs on the same values), so hits are identical.
#pragma once

#include "team_stack.cuh"
#include "trace_kernels.cuh"
#include "trace_wide.cuh"

namespace dr {

// Lanes per ray. Public launches: 8 lanes have the shorter chain per node (2^10
// rays, 300,000 triangles, closest hit: 25 us against 27 us with 4 lanes and 41 us
// with one lane per ray; 2^14 rays 34 / 40 / 54 us); 4 lanes keep more rays in
// flight, which the path kernel wants (box room 256x256, 1 spp, before its paths
// were dealt in runs: 464 us against 593 us with 8; now 433 us).
constexpr int kTeamTrace = 8, kTeamPaths = 4;

// Public launches of up to this many rays per SM run with teams (65,664 rays
// on 152 SMs). Teams / one lane per ray, us, closest hit and any hit:
// 300,000 triangles 2^8 rays 19 / 30, 15 / 29; 2^12 27 / 55, 26 / 54; 2^16
// 63 / 74, 52 / 61; 2^17 96 / 83, 79 / 67; 5,000 triangles 2^16 32 / 35,
// 29 / 35; 2^17 45 / 49, 41 / 38. 2^20 triangles (against the kernels of one lane per
// ray before them): 2^12 35 / 61, 34 / 59; 65,600 74 / 87, 67 / 80.
constexpr uint32_t kTeamRaysPerSm = 432;

// The traversal stacks of a block of kTraceBlock threads in shared memory: 32
// S entries per warp (a column of S per lane, or 32 S / teams per team).
template <int S>
__device__ __forceinline__ uint2 *block_stacks()
{
    __shared__ uint2 s_stack[kTraceBlock / 32][S > 0 ? S : 1][32];
    return &s_stack[0][0][0];
}

// 2^15 + q as a float, for a grid plane q: with A = a and B = slab_axis(a, b)'s
// near_b or far_b, fma(grid_f(q), A, B) rounds the same real number as
// fma(byte_q(q), A / 256, B) of the node test.
__device__ __forceinline__ float grid_f(uint32_t q) { return __uint_as_float(q * 256u + 0x47000000u); }

// Hands out rays 0 .. n - 1 of a launch. The first ray of every team is its
// number in the grid (one ray per warp before any warp gets a second one);
// teams that finish take the next index from `counter`, which counts the rays
// handed out after those: with at most one ray per team there is no atomic.
template <int G>
struct GridQueue {
    uint64_t n;
    unsigned long long *counter;
    bool fresh = true;
    // Called by the whole warp; `idle` has the first lane of each team that
    // wants a ray. Returns whether rays may be left.
    __device__ __forceinline__ bool take(unsigned idle, int lane, uint64_t &idx)
    {
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        const uint64_t teams = (uint64_t)warps * (32 / G);
        if (fresh) {
            fresh = false;
            idx = (uint64_t)(lane / G) * warps + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
            return n > teams;
        }
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)__popc(idle));
        b = teams + __shfl_sync(0xffffffffu, b, 0);
        idx = b + __popc(idle & ((1u << (lane & ~(G - 1))) - 1u));
        return b + __popc(idle) < n;
    }
};

// The rays 0 .. n - 1 of one warp.
template <int G>
struct WarpQueue {
    uint32_t n;
    uint32_t next = 0;
    __device__ __forceinline__ bool take(unsigned idle, int lane, uint32_t &idx)
    {
        idx = next + __popc(idle & ((1u << (lane & ~(G - 1))) - 1u));
        next += __popc(idle);
        return next < n;
    }
};

// Traces the rays that `queue` hands out (indices of `src`).
template <int MODE, int G, int STACK, class Source, class Queue>
__device__ __forceinline__ void team_wide(const Wide8Args &a, const Source &src, Queue queue)
{
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int SL = 8 / G, DEPTH = STACK * G;
    constexpr unsigned TEAM_MASK = (1u << G) - 1u;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), shift = lane & ~(G - 1);
    uint2 *stack = block_stacks<STACK>() + (threadIdx.x >> 5) * (32 * STACK) + shift * STACK;
    uint2 over[kWideStack > DEPTH ? kWideStack - DEPTH : 1];  // entries past the shared ones, the same in every lane
    decltype(queue.n) idx = 0;
    bool exhausted = false;  // warp-uniform
    bool active = false, any = false;
    DevRay r;
    WtSetup w;
    uint32_t oct = 0, node = 0, child_base = 0, imask = 0, hits = 0;
    float best_t = 0.0f;
    int32_t best_prim = INT_MAX;
    int sp = 0;
    while (true) {
        if (!exhausted) {
            const unsigned idle = __ballot_sync(FULL, !active && sub == 0);
            if (idle != 0) {
                decltype(queue.n) i = 0;
                exhausted = !queue.take(idle, lane, i);
                if (!active && i < queue.n) {
                    uint32_t root;
                    idx = i;
                    any = src.is_any(idx);
                    if (src.load(idx, r, root) && root != kNoRoot) {
                        if (MODE == 1) w = wt_setup(r.v);
                        oct = ray_octant(r);
                        best_t = r.tmax;
                        best_prim = INT_MAX;
                        node = root;
                        sp = 0;
                        active = true;
                    } else if (sub == 0) {
                        if (any) src.any(idx, false);
                        else src.closest(idx, 0.0f, INT_MAX);
                    }
                }
            }
        }
        if (__ballot_sync(FULL, active) == 0) {
            if (exhausted) break;
            continue;
        }
        // 1. the node's boxes
        bool inner[SL];
        uint32_t tmask = 0, tbase = 0;
#pragma unroll
        for (int j = 0; j < SL; ++j) inner[j] = false;
        if (active) {
            const Bvh8Node *nd = a.nodes + node;
            const uint8_t *bytes = reinterpret_cast<const uint8_t *>(nd);
            const uint4 w0 = __ldg(&nd->w[0]);
            const uint2 base = __ldg(reinterpret_cast<const uint2 *>(&nd->w[1]));
            const float sx = exp2_bits(w0.w & 0xffu), sy = exp2_bits((w0.w >> 8) & 0xffu),
                        sz = exp2_bits((w0.w >> 16) & 0xffu);
            imask = w0.w >> 24;
            child_base = base.x;
            tbase = base.y;
            const float ax = sx * r.inv.x, ay = sy * r.inv.y, az = sz * r.inv.z;
            const SlabAxis cx = slab_axis(ax, (bits_f(w0.x) - r.o.x) * r.inv.x),
                           cy = slab_axis(ay, (bits_f(w0.y) - r.o.y) * r.inv.y),
                           cz = slab_axis(az, (bits_f(w0.z) - r.o.z) * r.inv.z);
            const int nx = r.inv.x < 0.0f ? 8 : 0, ny = r.inv.y < 0.0f ? 8 : 0, nz = r.inv.z < 0.0f ? 8 : 0;
#pragma unroll
            for (int j = 0; j < SL; ++j) {
                const uint32_t slot = (uint32_t)(sub + j * G) ^ oct;
                const uint8_t *q = bytes + 32 + slot;
                const float tnx = fmaf(grid_f(__ldg(q + nx)), ax, cx.near_b), tfx = fmaf(grid_f(__ldg(q + 8 - nx)), ax, cx.far_b);
                const float tny = fmaf(grid_f(__ldg(q + 16 + ny)), ay, cy.near_b),
                            tfy = fmaf(grid_f(__ldg(q + 24 - ny)), ay, cy.far_b);
                const float tnz = fmaf(grid_f(__ldg(q + 32 + nz)), az, cz.near_b),
                            tfz = fmaf(grid_f(__ldg(q + 40 - nz)), az, cz.far_b);
                const uint32_t meta = __ldg(bytes + 24 + slot);
                const bool hit = fmaxf(max3f(tnx, tny, tnz), 0.0f) <= fminf(min3f(tfx, tfy, tfz), best_t) * kBoxFarScale;
                inner[j] = hit && ((imask >> slot) & 1u);
                if (hit && !inner[j]) tmask |= (meta >> 5) << (meta & 31u);  // 0 for an empty slot
            }
        }
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < SL; ++j) m |= ((__ballot_sync(FULL, inner[j]) >> shift) & TEAM_MASK) << (j * G);
        hits = m;
        // 2. the hit leaf slots' triangles, each by the lane of its slot; the
        //    team keeps the smallest (t, index)
        bool done = false, found = false;
        if (__ballot_sync(FULL, tmask != 0) != 0) {
            float bt = best_t;
            int32_t bp = INT_MAX;
            while (tmask) {
                const uint32_t k = tbase + (uint32_t)(__ffs(tmask) - 1);
                tmask &= tmask - 1u;
                float t;
                const bool ok = MODE == 1 ? tri_test_wt(a.tri_wt, k, r, w, bt, t) : tri_test_ref(a.tri_ref, k, r, bt, t);
                if (ok) {
                    const int32_t prim = any ? 0 : DR_LD(a.prim + k);
                    if (any) tmask = 0;
                    if (t < bt || prim < bp) {
                        bt = t;
                        bp = prim;
                    }
                }
            }
            if (__ballot_sync(FULL, bp != INT_MAX) != 0) {
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) {
                    const float ot = __shfl_xor_sync(FULL, bt, o);
                    const int32_t op = __shfl_xor_sync(FULL, bp, o);
                    if (ot < bt || (ot == bt && op < bp)) {
                        bt = ot;
                        bp = op;
                    }
                }
                if (active && bp != INT_MAX) {
                    if (any) {
                        done = found = true;
                    } else if (bt < best_t || (bt == best_t && bp < best_prim)) {
                        best_t = bt;
                        best_prim = bp;
                    }
                }
            }
        }
        // 3. the next node, in octant order
        bool full = false;
        const bool end = team_next_node<DEPTH>(active && !done, sub == 0, oct, child_base, imask, hits, stack, over, a.stack_limit, sp,
                                               node, full, [] { __syncwarp(); });
        done = done || end;
        if (full && sub == 0) atomicOr(a.error, ERR_STACK_OVERFLOW);
        if (active && done) {
            if (sub == 0) {
                if (any) src.any(idx, found);
                else src.closest(idx, best_t, best_prim);
            }
            active = false;
        }
    }
}

}  // namespace dr
