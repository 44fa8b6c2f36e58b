// Contact islands of at most 32 contacts, a contact per lane: the solve of the per-thread and the
// small per-warp class when the step has few islands.  Included by cc_solver.cu after
// cc_solve_block.cuh.
//
// With few islands the per-thread solve is bound by one thread's chain of memory round trips (a
// contact's rows, its bodies' velocities, inertias and flags, again for each of its visits), not
// by throughput.  Here a contact's rows stay in its lane's registers for the whole solve and the
// bodies' velocities (then poses) in shared memory.  Visit v of a contact runs when both its
// dynamic bodies have seen the contacts before it: body X has had turn[X] visits, and the contact
// is number pos of deg on X in the solve order, so its turn is v deg + pos.  Contacts of one island
// that share no body, other islands in the warp and later sweeps run side by side.
// 18 islands of a 32-body world: 250 -> 110 us; 4,489 islands of 7,470 bodies: 464 us (per-thread)
// beside 290 us (per-warp) -> 170 us.
// One contact per lane costs a warp more instructions per contact than one island per thread does, so
// above LANE_ISLANDS islands, when the SMs are full either way, the per-thread and per-warp classes
// keep them: a step of 4,096 uneven worlds (325,297 islands) takes 6.45 ms on lanes and 6.08 ms so.
// Below the line lanes win for every kind of island measured (steps of 8,000 alike: 5 contacts 0.82 and
// 1.00 ms, 12 contacts 1.74 and 2.22, 22 contacts 3.35 and 3.71), and for islands that are all alike
// also somewhat above it (32,000 of 5 contacts 1.83 and 2.29 ms, 64,000 3.12 and 3.20).
#pragma once

constexpr int LANE_ISLANDS = 16384;
constexpr int LANE_BLOCK = 64;  // two warps
constexpr int LANE_BUCKETS = SMALL_BUCKETS + 2;  // the per-thread class's buckets, the two smallest per-warp ones

struct LaneWarp {
    float state[64 * 7];  // per body: velocities (6), then the pose
    int turn[64];         // visits a dynamic body has had
    int body[64];         // -1: none
    int awake[32];        // per island: a body that may not sleep yet
};

__device__ __forceinline__ bool lanes_take(const DevWorld &w) {
    return w.ctr->num_islands <= LANE_ISLANDS && c_settings.small_island_max_cons < SMALL_BUCKETS;
}

__global__ void __launch_bounds__(LANE_BLOCK) k_solve_lanes(DevWorld w, CacheTables ct, const int *small_list, float dt,
                                                            float ratio, int phase) {
    if (islands_failed(w) || !lanes_take(w)) return;
    __shared__ LaneWarp smem[LANE_BLOCK / 32];
    LaneWarp &S = smem[threadIdx.x >> 5];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    CacheRecord *crecs = ct.recs[*ct.parity];
    // Islands by size, most contacts first: bucket rank 0 is the per-warp class's second bucket
    // (17-32 contacts), 1 its first (9-16), 2 + r the per-thread class's bucket SMALL_BUCKETS - 1 - r.
    // A warp takes one island of the first, two of the second, 32 / k islands of k contacts of the others.
    // (With one of the second as well, half the lanes had no contact: 8,000 islands of 12 contacts took
    // 1,821 us, 1,436 on the per-warp class; two to a warp 930 us.)
    const int rank = min(lane, LANE_BUCKETS - 1);
    const int small_k = SMALL_BUCKETS + 1 - rank;
    const int have = rank < 2 ? w.ctr->mid_bucket[1 - rank] : w.ctr->small_bucket[small_k];
    const int per = rank < 2 ? 1 + rank : 32 / max(small_k, 1);
    int items = lane < LANE_BUCKETS ? (have + per - 1) / per : 0;
    for (int o = 1; o < 32; o <<= 1) {  // inclusive scan: the buckets' ends
        const int v = __shfl_up_sync(FULL, items, o);
        if (lane >= o) items += v;
    }
    const int total = __shfl_sync(FULL, items, 31);
    const int nwarps = gridDim.x * (LANE_BLOCK / 32);
    for (int item = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; item < total; item += nwarps) {
        const int r = __popc(__ballot_sync(FULL, items <= item));  // the item's bucket
        const int first = r > 0 ? __shfl_sync(FULL, items, r - 1) : 0;
        const int count = __shfl_sync(FULL, have, r), group = __shfl_sync(FULL, per, r);
        const int k = r < 2 ? 32 >> r : SMALL_BUCKETS + 1 - r;  // lanes per island (0: islands without contacts)
        const int *list = r < 2 ? w.mid_list + (size_t)(1 - r) * w.cap : small_list + (size_t)k * w.cap;
        const int i0 = (item - first) * group, ni = min(group, count - i0);
        // ---- this lane's island and contact ----
        const int gi = k > 0 ? lane / k : lane, c_in = k > 0 ? lane - gi * k : 0;
        const bool in_group = gi < ni;
        const int isl = in_group ? list[i0 + gi] : -1;
        int nc = 0, nb = 0, vel_iters = 0, pos_iters = 0;
        const int *bl = nullptr;
        if (in_group) {
            nc = w.island_cons_count[isl];
            nb = w.island_body_count[isl];
            bl = w.island_bodies + w.island_body_off[isl];
            island_iterations(w, isl, c_settings.vel_iters, c_settings.pos_iters, vel_iters, pos_iters);
        }
        const bool has = k > 0 && in_group && c_in < nc;
        const int slots = r < 2 ? 64 >> r : k + 1;  // body slots per island: k contacts join at most k + 1 bodies
        const bool vel = phase != SOLVE_POSITION;
        // ---- bodies ----
        for (int i = lane; i < 64; i += 32) {
            S.turn[i] = 0;
            S.body[i] = -1;
        }
        S.awake[lane] = 0;
        __syncwarp();
        // each island's lanes (a single lane without contacts) place its bodies
        const int lanes_per = k > 0 ? k : 1;
        for (int j = c_in; in_group && j < nb; j += lanes_per) {
            const int b = bl[j], at = gi * slots + j;
            S.body[at] = b;
            w.body_local[b] = at;
            if (vel) {
                prepare_body(w, b);
                const float4 v = w.linvel[b], a = w.angvel[b];
                float *s = S.state + 7 * at;
                s[0] = v.x;
                s[1] = v.y;
                s[2] = v.z;
                s[3] = a.x;
                s[4] = a.y;
                s[5] = a.z;
            }
        }
        __syncwarp();
        // ---- the contact's rows into registers ----
        const int ci = has ? w.island_cons[w.island_cons_off[isl] + c_in] : 0;
        const float4 *c4 = (const float4 *)&w.cons[ci];
        int4 hd = make_int4(0, 0, 0, 0);
        uint32_t fa = 0, fb = 0, key = 0;
        int la = -1, lb = -1;
        bool dynA = false, dynB = false;
        if (has) {
            hd = *(const int4 *)c4;  // a, b, n, island
            key = w.cons[ci].sort_key;
            fa = w.flags[hd.x];
            fb = w.flags[hd.y];
            // a body of another island (static, or asleep and kinematic) has no slot
            const int xa = w.body_local[hd.x], xb = w.body_local[hd.y];
            if (xa >= 0 && xa < 64 && S.body[xa] == hd.x) la = xa;
            if (xb >= 0 && xb < 64 && S.body[xb] == hd.y) lb = xb;
            dynA = la >= 0 && motion_of(fa) == DYNAMIC;
            dynB = lb >= 0 && motion_of(fb) == DYNAMIC;
        }
        // ---- the contact's place on its bodies in (sortKey, idA, idB) order ----
        int degA = 0, posA = 0, degB = 0, posB = 0;
        for (int j = 0; j < k; j++) {
            const int src = min(gi * k + j, 31);
            const uint32_t ok = __shfl_sync(FULL, key, src);
            const int oa = __shfl_sync(FULL, hd.x, src), ob = __shfl_sync(FULL, hd.y, src);
            if (!has || j >= nc) continue;
            const bool before = ok != key ? ok < key : (oa != hd.x ? oa < hd.x : (ob != hd.y ? ob < hd.y : j < c_in));
            if (dynA && (oa == hd.x || ob == hd.x)) {
                degA++;
                posA += before;
            }
            if (dynB && (oa == hd.y || ob == hd.y)) {
                degB++;
                posB += before;
            }
        }
        const int n = hd.z, bits = side_bits(n, fa, fb);
        // One turn-taking pass of `visits` visits per contact: visit(v) solves the lane's contact.
        // Every round at least one waiting contact has its turn, so the rounds are bounded.  All lanes
        // read the turns before any lane visits, with a barrier of the warp between: a body passes from
        // one visit to the next, its turn and its state, over a barrier only.
        auto turns = [&](int visits, auto &&visit) {
            int v = 0, turnA = posA, turnB = posB;
            const int most = __reduce_max_sync(FULL, has ? visits : 0) * 32;
            for (int round = 0; round < most; round++) {
                const bool wait = has && v < visits;
                if (!__any_sync(FULL, wait)) break;
                const bool ready = wait && (!dynA || S.turn[la] == turnA) && (!dynB || S.turn[lb] == turnB);
                __syncwarp();
                if (ready) {
                    visit(v);
                    v++;
                    if (dynA) S.turn[la]++;
                    if (dynB) S.turn[lb]++;
                    turnA += degA;
                    turnB += degB;
                }
                __syncwarp();
            }
        };
        if (vel) {
            if (k > 0) {
                float4 n4, t14, t24;
                PointRow p[4];
                Sym3 IA{0, 0, 0, 0, 0, 0}, IB{0, 0, 0, 0, 0, 0};
                if (has) {
                    n4 = c4[1];
                    t14 = c4[2];
                    t24 = c4[3];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (j >= n) continue;
                        const float4 q0 = c4[5 + 5 * j], q1 = c4[6 + 5 * j], q3 = c4[8 + 5 * j], q4 = c4[9 + 5 * j];
                        p[j] = PointRow{f3(q0.x, q0.y, q0.z), f3(q0.w, q1.x, q1.y), q3.x, q3.y, q3.z, q3.w, q4.x, q4.y,
                                        q4.z};
                    }
                    if (motion_of(fa) == DYNAMIC) IA = load_sym(w.inv_inertia_world, hd.x);
                    if (motion_of(fb) == DYNAMIC) IB = load_sym(w.inv_inertia_world, hd.y);
                }
                float3 vA0 = f3(0.f, 0.f, 0.f), wA0 = vA0, vB0 = vA0, wB0 = vA0;  // of the bodies without a slot
                if (has && la < 0) vA0 = xyz(w.linvel[hd.x]), wA0 = xyz(w.angvel[hd.x]);
                if (has && lb < 0) vB0 = xyz(w.linvel[hd.y]), wB0 = xyz(w.angvel[hd.y]);
                const int warm = c_settings.warm_starting ? 1 : 0;
                turns(vel_iters + warm, [&](int v) {
                    // the bodies are put together here, per visit, as the other classes load them per
                    // contact: the rows' arithmetic then compiles to the same operations (bodies
                    // kept over the visits let the compiler split the loop by their motion types
                    // and fuse other multiplies and adds: differences in the last bit)
                    BodyRef A, B;
                    A.motion = (bits >> 4) & 3;
                    B.motion = (bits >> 6) & 3;
                    A.dof = (bits >> 8) & 63;
                    B.dof = (bits >> 16) & 63;
                    A.im = B.im = 0.f;
                    A.I = IA;
                    B.I = IB;
                    A.v = vA0, A.w = wA0, B.v = vB0, B.w = wB0;
                    if (la >= 0) {
                        const float *s = S.state + 7 * la;
                        A.v = f3(s[0], s[1], s[2]);
                        A.w = f3(s[3], s[4], s[5]);
                    }
                    if (lb >= 0) {
                        const float *s = S.state + 7 * lb;
                        B.v = f3(s[0], s[1], s[2]);
                        B.w = f3(s[3], s[4], s[5]);
                    }
                    const float3 nn = xyz(n4), t1 = xyz(t14), t2 = xyz(t24);
                    if (v < warm) {
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (j < n) warm_start_point(p[j], A, B, t14.w, t24.w, nn, t1, t2, ratio);
                    } else if (A.motion == DYNAMIC || B.motion == DYNAMIC) {
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (j < n) friction_point(p[j], A, B, t14.w, t24.w, t1, t2, n4.w);
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (j < n) normal_point(p[j], A, B, t14.w, t24.w, nn);
                    }
                    if (dynA) {
                        float *s = S.state + 7 * la;
                        s[0] = A.v.x;
                        s[1] = A.v.y;
                        s[2] = A.v.z;
                        s[3] = A.w.x;
                        s[4] = A.w.y;
                        s[5] = A.w.z;
                    }
                    if (dynB) {
                        float *s = S.state + 7 * lb;
                        s[0] = B.v.x;
                        s[1] = B.v.y;
                        s[2] = B.v.z;
                        s[3] = B.w.x;
                        s[4] = B.w.y;
                        s[5] = B.w.z;
                    }
                });
                if (has) {  // impulses to the contact and the cache
                    ContactConstraint &c = w.cons[ci];
                    CacheRecord *rec = crecs + c.cache_slot;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (j >= n) continue;
                        c.p[j].lam_n = rec->ln[j] = p[j].lam_n;
                        c.p[j].lam_t1 = rec->lt1[j] = p[j].lam_t1;
                        c.p[j].lam_t2 = rec->lt2[j] = p[j].lam_t2;
                    }
                }
            }
            for (int i = lane; i < 64; i += 32) {
                const int b = S.body[i];
                if (b < 0) continue;
                if (k > 0 && motion_of(w.flags[b]) == DYNAMIC) {
                    const float *s = S.state + 7 * i;
                    w.linvel[b] = make_float4(s[0], s[1], s[2], 0.f);
                    w.angvel[b] = make_float4(s[3], s[4], s[5], 0.f);
                }
                integrate_body(w, b, dt, phase == SOLVE_VELOCITY);
            }
            __syncwarp();
            if (phase == SOLVE_VELOCITY) continue;
        }
        // ---- position iterations: the reference stops after a sweep that moved nothing
        // (update.ts:218-221); a later sweep would not move anything either ----
        if (k > 0) {
            for (int i = lane; i < 64; i += 32) {
                S.turn[i] = 0;
                const int b = S.body[i];
                if (b < 0) continue;
                const float4 c = w.com[b], q = w.quat[b];
                float *s = S.state + 7 * i;
                s[0] = c.x;
                s[1] = c.y;
                s[2] = c.z;
                s[3] = q.x;
                s[4] = q.y;
                s[5] = q.z;
                s[6] = q.w;
            }
            __syncwarp();
            float4 com0A, com0B, q0A, q0B;  // of the bodies without a slot
            if (has) {
                com0A = w.com[hd.x], q0A = w.quat[hd.x];
                com0B = w.com[hd.y], q0B = w.quat[hd.y];
            }
            turns(pos_iters, [&](int) {
                PoseRef PA{xyz(com0A), q0A}, PB{xyz(com0B), q0B};
                if (la >= 0) {
                    const float *s = S.state + 7 * la;
                    PA = PoseRef{f3(s[0], s[1], s[2]), make_float4(s[3], s[4], s[5], s[6])};
                }
                if (lb >= 0) {
                    const float *s = S.state + 7 * lb;
                    PB = PoseRef{f3(s[0], s[1], s[2]), make_float4(s[3], s[4], s[5], s[6])};
                }
                if (!solve_position_con(w, w.cons[ci], PA, PB, motion_of(fa), motion_of(fb), fa, fb)) return;
                if (dynA) {
                    float *s = S.state + 7 * la;
                    s[0] = PA.com.x;
                    s[1] = PA.com.y;
                    s[2] = PA.com.z;
                    s[3] = PA.q.x;
                    s[4] = PA.q.y;
                    s[5] = PA.q.z;
                    s[6] = PA.q.w;
                }
                if (dynB) {
                    float *s = S.state + 7 * lb;
                    s[0] = PB.com.x;
                    s[1] = PB.com.y;
                    s[2] = PB.com.z;
                    s[3] = PB.q.x;
                    s[4] = PB.q.y;
                    s[5] = PB.q.z;
                    s[6] = PB.q.w;
                }
            });
        }
        for (int i = lane; i < 64; i += 32) {
            const int b = S.body[i];
            if (b < 0) continue;
            if (k > 0 && motion_of(w.flags[b]) == DYNAMIC) {
                const float *s = S.state + 7 * i;
                w.com[b] = make_float4(s[0], s[1], s[2], 0.f);
                w.quat[b] = make_float4(s[3], s[4], s[5], s[6]);
            }
            finish_body(w, b);
            if (c_settings.allow_sleeping && motion_of(w.flags[b]) == DYNAMIC && !sleep_update(w, b, dt))
                S.awake[i / slots] = 1;
        }
        __syncwarp();
        if (c_settings.allow_sleeping)
            for (int i = lane; i < 64; i += 32) {
                const int b = S.body[i];
                if (b >= 0 && !S.awake[i / slots] && motion_of(w.flags[b]) == DYNAMIC) sleep_body(w, b);
            }
        __syncwarp();
    }
}
