// tmpm_grid.cuh -- the grid update of one substep (world.rs:401-417), shared by
// its own kernel and the whole-segment kernels.
#pragma once

#include "tmpm_device.cuh"

namespace tmpm {

// Grid update over all allocated blocks of `g` (thread gtid of `stride`); also
// zeroes the same blocks in the other pool `next_pool`, which receives the next
// P2G.  MULTI: each block takes its scene's parameters from the scene table
// (scene = block namespace >> kSceneShift).  Blocks have edge 2^BS cells.
// OBST: the scene has rigid obstacles (a batch never has).
//
// A chain of dependent loads on a small scene: the first node and its block's
// coordinates are read beside the block count, not after it (every index below
// max_blocks is allocated).  All grid reads go to L2: in a whole-segment kernel
// other SMs wrote these lines during this launch.
template <bool MULTI, int BS, bool OBST>
__device__ __forceinline__ void grid_nodes(const GridTable &g, float4 *next_pool, const SimParams &sp,
                                           const DevObstacle *__restrict__ obstacles,
                                           const float *__restrict__ planes, double *reactions, size_t gtid,
                                           size_t stride) {
    constexpr int kM = (1 << BS) - 1;
    const size_t most = static_cast<size_t>(g.max_blocks) << (3 * BS);
    float4 mp = make_float4(0.f, 0.f, 0.f, 0.f);
    int4 c = make_int4(0, 0, 0, 0);
    if (gtid < most) {
        mp = __ldcg(g.pool + gtid);
        c = __ldcg(g.coords + (gtid >> (3 * BS)));
    }
    const size_t nodes = static_cast<size_t>(min(__ldcg(g.count), g.max_blocks)) << (3 * BS);
    for (size_t node = gtid; node < nodes; node += stride) {
        if (node != gtid) {
            mp = __ldcg(g.pool + node);
            c = __ldcg(g.coords + (node >> (3 * BS)));
        }
        if (next_pool) next_pool[node] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mp.x <= 0.0f) {
            g.pool[node] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        int l = static_cast<int>(node) & ((1 << (3 * BS)) - 1);
        int cx = (c.x << BS) + (l >> (2 * BS)), cy = (c.y << BS) + ((l >> BS) & kM), cz = (c.z << BS) + (l & kM);
        const SceneParams *const scn = sp.scenes + (MULTI ? (static_cast<uint32_t>(c.w) >> kSceneShift) : 0u);
#define SCN(f) (MULTI ? scn->f : sp.s0.f)
        const float h = SCN(h), dt = SCN(dt);
        V3f vel = mk(mp.y / mp.x + SCN(gx) * dt, mp.z / mp.x + SCN(gy) * dt, mp.w / mp.x + SCN(gz) * dt);
        V3f pos = mk(static_cast<float>(cx) * h, static_cast<float>(cy) * h, static_cast<float>(cz) * h);
        if (SCN(has_bounds)) {
            // walls by node index (thresholds from the f64 comparisons, see SceneParams)
            const int ci[3] = {cx, cy, cz};
            if (SCN(wall_mode) == 1) {
                bool near = false;
                for (int a = 0; a < 3; ++a) near = near || ci[a] <= SCN(wall_lo[a]) || ci[a] >= SCN(wall_hi[a]);
                if (near) vel = mk(0, 0, 0);
            } else {
                for (int a = 0; a < 3; ++a) {
                    const float va = comp(vel, a);
                    if ((ci[a] <= SCN(wall_lo[a]) && va < 0.0f) || (ci[a] >= SCN(wall_hi[a]) && va > 0.0f))
                        set_comp(vel, a, 0.0f);
                }
            }
        }
#undef SCN
        for (int oi = 0; OBST && oi < sp.num_obstacles; ++oi) {
            const DevObstacle &o = obstacles[oi];
            if (!obstacle_may_contact(o, pos, h)) continue;
            V3f nrm;
            float d = obstacle_surface(o, planes, pos, nrm);
            if (d <= h * (1.0f + 1e-5f)) {
                V3f before = vel;
                vel = contact_velocity(o, pos, vel, nrm);
                if (sp.reactions)
                    add_reaction(reactions, oi, mk(o.center[0], o.center[1], o.center[2]), pos - nrm * d,
                                 (before - vel) * mp.x);
            }
        }
        g.pool[node] = make_float4(vel.x, vel.y, vel.z, mp.x);
    }
}

}  // namespace tmpm
