// Islands above the per-warp tier and up to a pile of thousands of bodies: one CTA each, the
// island's body state in shared memory.  Included by cc_solver.cu after the solver primitives.
//
// The reference sweeps an island's contacts one after another in (sortKey, idA, idB) order, sweep
// after sweep.  Only contacts that share a dynamic body depend on each other: visit p of a contact
// waits for the contact before it on either body, which for the first contact on a body is the
// body's last one in visit p - 1.  A task's (contact's visit's) level is one more than the levels
// of the two tasks it waits for; solving level by level gives the sequential sweeps' result.  The
// sort key grows with the body indices, so one sweep of a heap is a wavefront of about a hundred
// narrow levels across it (28 contacts a level for 10 x 10 x 10 boxes), and the next sweep's
// wavefront can follow a few levels behind: all sweeps of a 1,000-box heap take about twice the
// levels of one.  The work, in order:
//   - per-body lists of contacts in shared memory give each contact's predecessors; a counted
//     breadth-first pass over the tasks gives the levels, cut into chunks of at most 32 contacts;
//   - the solver rows are repacked in the first sweep's order, one coalesced float4 row per field;
//   - the chunks go to the CTA's warps in turn.  A warp loads its chunk's rows before it waits for
//     the chunk's turn: a counter of finished chunks, polled in shared memory, reaches the number
//     of chunks in the earlier levels.  No barrier separates the levels;
//   - velocities (in the position sweeps, poses) stay in shared memory, accumulated impulses in
//     the rows.
// It is bound by the latency of a level (four points' friction and normal rows in sequence, about
// 1.2 us) on narrow islands and by the issue rate of one SM on wide ones.
#pragma once

// rows of the repacked contacts: row f of slot s at rows[f * stride + s]
enum : int {
    ROW_N = 0,      // normal, friction
    ROW_T1 = 1,     // first tangent, inverse mass of A
    ROW_T2 = 2,     // second tangent, inverse mass of B
    ROW_ID = 3,     // local bodies A | B << 16, constraint, side_bits, 0
    ROW_R = 4,      // 4 per side (A, then B): moment arm of point k; w: world inverse inertia xx xy xz yy
    ROW_I = 12,     // the rest of it: A's yz zz, B's yz zz
    ROW_EFFN = 13,  // per point: effective masses of the normal and the tangent rows, bias
    ROW_EFF1 = 14,
    ROW_EFF2 = 15,
    ROW_BIAS = 16,
    ROW_LN = 17,    // per point: accumulated impulses
    ROW_L1 = 18,
    ROW_L2 = 19,
    SOLVE_ROWS = 20
};
constexpr unsigned BLOCK_NONE = 0xffffu;  // no local body / no predecessor
// bits of ROW_ID.z: point count, motion types, degrees of freedom (all, unless dynamic)
__device__ __forceinline__ int side_bits(int n, uint32_t fa, uint32_t fb) {
    const int da = motion_of(fa) == DYNAMIC ? dof_of(fa) : 63, db = motion_of(fb) == DYNAMIC ? dof_of(fb) : 63;
    return n | (motion_of(fa) << 4) | (motion_of(fb) << 6) | (da << 8) | (db << 16);
}

struct PointRow {
    float3 rA, rB;
    float eff_n, eff_t1, eff_t2, lam_n, lam_t1, lam_t2, bias_n;
};
__device__ __forceinline__ float comp(const float4 &v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w)); }

// MC contacts and MB bodies at most, W warps.  Two instances, by footprint: islands of up to 4,096
// contacts and 2,048 bodies take 65 KB of shared memory and leave the rest of it to
// the L1 cache, which keeps their rows; the larger ones take most of it.
template <int MC, int MB, int W>
struct BlockTier {
    static constexpr int CONS = MC, BODIES = MB, WARPS = W, THREADS = 32 * W;
    static constexpr size_t LIST_BYTES = sizeof(int) * (2 * MB + 4) + (sizeof(uint32_t) + sizeof(uint16_t)) * 2 * MC;
    static constexpr size_t ORDER_BYTES = sizeof(int) * MC + sizeof(uint16_t) * 5 * MC;
    static constexpr size_t STATE_BYTES = sizeof(float) * 7 * MB;
    static constexpr size_t SMEM = LIST_BYTES > ORDER_BYTES ? (LIST_BYTES > STATE_BYTES ? LIST_BYTES : STATE_BYTES)
                                                            : (ORDER_BYTES > STATE_BYTES ? ORDER_BYTES : STATE_BYTES);
    static_assert(SMEM <= 227 * 1024, "shared memory of a block");
};
using BlockTierS = BlockTier<BLOCK_S_CONS, BLOCK_S_BODIES, 12>;
using BlockTierL = BlockTier<BLOCK_L_CONS, BLOCK_L_BODIES, 12>;
static_assert(BLOCK_L_CONS < 0x8000 && BLOCK_L_BODIES < 0xffff, "16-bit local indices, a flag beside the contact");
// a chunk word: first task (18 bits), tasks - 1 (5), chunks since the level's first (9)
static_assert(BLOCK_L_CONS * SOLVE_SWEEPS < 1 << 18 && BLOCK_L_CONS / 32 < 1 << 9, "chunk word fields");
constexpr unsigned TASK_WARM = 0x8000u;  // a task that warm starts its contact
static_assert(sizeof(ContactConstraint) == 400 && sizeof(ContactPoint) == 80, "float4 loads of a contact");

// exclusive scan over the CTA of one value per thread; total: the sum
template <int W>
__device__ int block_scan(int v, int *warp_tot, int &total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += a;
    }
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    int base = 0;
    total = 0;
#pragma unroll
    for (int k = 0; k < W; k++) {
        const int t = warp_tot[k];
        if (k < wid) base += t;
        total += t;
    }
    return base + inc - v;
}
// the islands of this instance: list[0], list[step], ...
template <class T>
__global__ void __launch_bounds__(T::THREADS, 1)
    k_solve_block(DevWorld w, CacheTables ct, const int *list, int step, const int *count, float dt, float ratio,
                  int phase) {
    if (islands_failed(w)) return;
    constexpr int W = T::WARPS, THREADS = T::THREADS;
    extern __shared__ __align__(16) unsigned char block_smem[];
    __shared__ int s_scan[W];
    __shared__ int s_front[3];  // tasks found for the next level, three levels in rotation
    __shared__ int s_slots, s_any;
    __shared__ volatile int s_fail;
    __shared__ volatile int s_done;  // chunks finished of the current schedule
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned FULL = 0xffffffffu;
    CacheRecord *crecs = ct.recs[*ct.parity];
    const int nl = *count;
    const size_t stride = (size_t)w.max_manifolds;
    for (int li = blockIdx.x; li < nl; li += gridDim.x) {
        const int isl = list[(ptrdiff_t)li * step];
        int vel_iters, pos_iters;
        island_iterations(w, isl, c_settings.vel_iters, c_settings.pos_iters, vel_iters, pos_iters);
        const int nb = w.island_body_count[isl], nc = w.island_cons_count[isl];
        const int *bl = w.island_bodies + w.island_body_off[isl];
        const int *cl = w.island_cons + w.island_cons_off[isl];
        const int base = w.island_cons_off[isl];
        int *lab = w.scratch_order + base;           // per contact: dynamic local bodies A | B << 16, then successors
        int *preds = w.scratch_colour + base;        // per contact: predecessors on A | on B << 16
        int *slot_k = w.scratch_claim + w.cap + base;  // per slot: contact
        uint16_t *tasks = w.solve_tasks + (size_t)SOLVE_SWEEPS * base;
        uint32_t *chunks = w.solve_chunks + (size_t)SOLVE_SWEEPS * base;
        float4 *rows = w.solve_rows + base;
        const bool vel = phase != SOLVE_POSITION;
        // ---- bodies; contacts per dynamic body ----
        int *off = (int *)block_smem, *fill = off + T::BODIES + 2;
        uint32_t *ekey = (uint32_t *)(fill + T::BODIES + 2);
        uint16_t *ek = (uint16_t *)(ekey + 2 * T::CONS);
        for (int k = tid; k < nb; k += THREADS) {
            w.body_local[bl[k]] = k;
            if (vel) prepare_body(w, bl[k]);
            off[k] = 0;
        }
        if (tid == 0) {
            s_fail = 0;
            s_slots = 0;
        }
        __syncthreads();
        auto local_of = [&](int body) -> unsigned {
            int l = w.body_local[body];
            return l >= 0 && l < nb && bl[l] == body ? (unsigned)l : BLOCK_NONE;
        };
#pragma unroll 4
        for (int k = tid; k < nc; k += THREADS) {
            const ContactConstraint &c = w.cons[cl[k]];
            const int ca = c.a, cb = c.b;
            unsigned la = motion_of(w.flags[ca]) == DYNAMIC ? local_of(ca) : BLOCK_NONE;
            unsigned lb = motion_of(w.flags[cb]) == DYNAMIC ? local_of(cb) : BLOCK_NONE;
            lab[k] = (int)(la | (lb << 16));
            if (la != BLOCK_NONE) atomicAdd(&off[la], 1);
            if (lb != BLOCK_NONE) atomicAdd(&off[lb], 1);
        }
        __syncthreads();
        {
            const int seg = (nb + THREADS - 1) / THREADS, k0 = min(tid * seg, nb), k1 = min(k0 + seg, nb);
            int sum = 0;
            for (int k = k0; k < k1; k++) sum += off[k];
            int total, at = block_scan<W>(sum, s_scan, total);
            for (int k = k0; k < k1; k++) {
                int n = off[k];
                off[k] = fill[k] = at;
                at += n;
            }
            if (tid == 0) off[nb] = total;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = tid; k < nc; k += THREADS) {
            const uint32_t key = w.cons[cl[k]].sort_key;
            const unsigned l2 = (unsigned)lab[k];
            for (int side = 0; side < 2; side++) {
                unsigned l = side ? l2 >> 16 : l2 & 0xffffu;
                if (l == BLOCK_NONE) continue;
                int e = atomicAdd(&fill[l], 1);
                ekey[e] = key;
                ek[e] = (uint16_t)k;
            }
        }
        __syncthreads();
        // ---- each contact's predecessor on either body: the last one before it in solve order ----
        for (int k = tid; k < nc; k += THREADS) {
            const ContactConstraint &c = w.cons[cl[k]];
            const uint32_t key = c.sort_key;
            const unsigned l2 = (unsigned)lab[k];
            unsigned pred[2] = {BLOCK_NONE, BLOCK_NONE};
            for (int side = 0; side < 2; side++) {
                unsigned l = side ? l2 >> 16 : l2 & 0xffffu;
                if (l == BLOCK_NONE) continue;
                uint32_t best = 0;
                for (int e = off[l]; e < off[l + 1]; e++) {
                    const int o = ek[e];
                    if (o == k || ekey[e] > key) continue;
                    if (ekey[e] == key) {  // equal sort keys: by bodies, then by list entry
                        const ContactConstraint &co = w.cons[cl[o]];
                        if (con_less(c, co) || (!con_less(co, c) && o > k)) continue;
                    }
                    if (pred[side] != BLOCK_NONE) {
                        if (ekey[e] < best) continue;
                        if (ekey[e] == best) {
                            const ContactConstraint &co = w.cons[cl[o]], &cp = w.cons[cl[pred[side]]];
                            if (con_less(co, cp) || (!con_less(cp, co) && o < (int)pred[side])) continue;
                        }
                    }
                    pred[side] = (unsigned)o;
                    best = ekey[e];
                }
            }
            preds[k] = (int)(pred[0] | (pred[1] << 16));
        }
        __syncthreads();
        // ---- each contact's successors on its bodies; a body's last contact is followed by its first ----
        int *wait = (int *)block_smem;                  // predecessors still to come | visits begun << 8
        uint16_t *succ = (uint16_t *)(wait + T::CONS);  // next contact on body A, on body B
        uint16_t *slot_of = succ + 2 * T::CONS;
        uint16_t *front = slot_of + T::CONS;            // this level's contacts, the next one's: two of CONS
        for (int k = tid; k < nc; k += THREADS) succ[2 * k] = succ[2 * k + 1] = (uint16_t)BLOCK_NONE;
        __syncthreads();
        for (int k = tid; k < nc; k += THREADS) {
            const unsigned pp = (unsigned)preds[k], l2 = (unsigned)lab[k];
            for (int side = 0; side < 2; side++) {
                const unsigned p = side ? pp >> 16 : pp & 0xffffu, body = side ? l2 >> 16 : l2 & 0xffffu;
                if (p != BLOCK_NONE) succ[2 * p + (((unsigned)lab[p] & 0xffffu) == body ? 0 : 1)] = (uint16_t)k;
            }
        }
        __syncthreads();
        // the first contacts of the bodies follow the last ones: a body's first contact finds its
        // last by walking the chain (short: a body's contacts)
        for (int k = tid; k < nc; k += THREADS) {
            const unsigned pp = (unsigned)preds[k], l2 = (unsigned)lab[k];
            for (int side = 0; side < 2; side++) {
                const unsigned p = side ? pp >> 16 : pp & 0xffffu, body = side ? l2 >> 16 : l2 & 0xffffu;
                if (p != BLOCK_NONE || body == BLOCK_NONE) continue;
                unsigned last = (unsigned)k, at = (unsigned)side;
                while (succ[2 * last + at] != BLOCK_NONE) {
                    last = succ[2 * last + at];
                    at = ((unsigned)lab[last] & 0xffffu) == body ? 0 : 1;
                }
                front[2 * k + side] = (uint16_t)(2 * last + at);  // closed below: the chains are read here
            }
        }
        __syncthreads();
        for (int k = tid; k < nc; k += THREADS) {
            const unsigned pp = (unsigned)preds[k], l2 = (unsigned)lab[k];
            for (int side = 0; side < 2; side++) {
                const unsigned p = side ? pp >> 16 : pp & 0xffffu, body = side ? l2 >> 16 : l2 & 0xffffu;
                if (p == BLOCK_NONE && body != BLOCK_NONE) succ[front[2 * k + side]] = (uint16_t)k;
            }
            if (l2 == 0xffffffffu) succ[2 * k] = (uint16_t)k;  // no dynamic body: only its own visits follow each other
        }
        __syncthreads();
        for (int k = tid; k < nc; k += THREADS) lab[k] = (int)(succ[2 * k] | ((unsigned)succ[2 * k + 1] << 16));
        // ---- a schedule of `sweeps` visits of every contact.  The first one also numbers the
        // contacts' slots in the order of their first visit ----
        auto schedule = [&](int sweeps, bool warm, bool number) -> int {
            __syncthreads();
            for (int k = tid; k < nc; k += THREADS) {
                const unsigned pp = (unsigned)preds[k], sc = (unsigned)lab[k];
                succ[2 * k] = (uint16_t)(sc & 0xffffu);
                succ[2 * k + 1] = (uint16_t)(sc >> 16);
                wait[k] = ((pp & 0xffffu) != BLOCK_NONE) + ((pp >> 16) != BLOCK_NONE);
                if (!number) slot_of[slot_k[k]] = (uint16_t)k;
            }
            if (tid < 3) s_front[tid] = 0;
            if (tid == 0) s_done = 0;
            __syncthreads();
            // visit p of contact k joins the next level
            auto enter = [&](int k, int p, int level, int tail, uint16_t *next) {
                wait[k] = ((succ[2 * k] != BLOCK_NONE) + (succ[2 * k + 1] != BLOCK_NONE)) | ((p + 1) << 8);
                if (number && p == 0) {
                    const int slot = atomicAdd(&s_slots, 1);
                    slot_of[k] = (uint16_t)slot;
                    slot_k[slot] = k;
                }
                const int e = atomicAdd(&s_front[level % 3], 1);
                next[e] = (uint16_t)k;
                tasks[tail + e] = (uint16_t)(slot_of[k] | (warm && p == 0 ? TASK_WARM : 0u));
            };
            for (int k = tid; k < nc; k += THREADS)
                if (wait[k] == 0) enter(k, 0, 0, 0, front);
            __syncthreads();
            int nchunks = 0;
            for (int head = 0, level = 0;; level++) {
                const int n = *(volatile int *)&s_front[level % 3];
                if (n == 0) break;
                const uint16_t *cur = front + (level & 1) * T::CONS;
                uint16_t *next = front + (~level & 1) * T::CONS;
                const int tail = head + n;
                if (tid == 0) s_front[(level + 2) % 3] = 0;  // last read before the barrier just passed
                for (int j = tid; 32 * j < n; j += THREADS)
                    chunks[nchunks + j] = (uint32_t)(head + 32 * j) | (uint32_t)(min(32, n - 32 * j) - 1) << 18 |
                                          (uint32_t)j << 23;
                nchunks += (n + 31) >> 5;
                for (int e = tid; e < n; e += THREADS) {
                    const int k = cur[e];
                    for (int side = 0; side < 2; side++) {
                        const unsigned o = succ[2 * k + side];
                        if (o == BLOCK_NONE) continue;
                        const int old = atomicSub(&wait[o], 1);
                        if ((old & 0xff) == 1 && (old >> 8) < sweeps) enter((int)o, old >> 8, level + 1, tail, next);
                    }
                }
                head = tail;
                __syncthreads();
            }
            return nchunks;
        };
        const int vel_total = vel_iters + (c_settings.warm_starting ? 1 : 0);
        auto batch = [](int total, int done) {  // sweeps of the next schedule: all in equal shares of at most SOLVE_SWEEPS
            const int n = (total + SOLVE_SWEEPS - 1) / SOLVE_SWEEPS;
            return min((total + n - 1) / n, total - done);
        };
        int nchunks = 0;
        if (vel)
            nchunks = schedule(vel_total > 0 ? batch(vel_total, 0) : 1, c_settings.warm_starting != 0, true);
        else
            nchunks = schedule(pos_iters > 0 ? batch(pos_iters, 0) : 1, false, true);
        // ---- the contacts' rows in slot order ----
        for (int slot = tid; slot < nc; slot += THREADS) {
            const int ci = cl[slot_k[slot]];
            const float4 *c4 = (const float4 *)&w.cons[ci];
            const int4 hd = *(const int4 *)c4;  // a, b, n, island
            const uint32_t fa = w.flags[hd.x], fb = w.flags[hd.y];
            const unsigned la = local_of(hd.x), lb = local_of(hd.y);
            const bool da = motion_of(fa) == DYNAMIC, db = motion_of(fb) == DYNAMIC;
            float4 *r = rows + slot;
            r[ROW_ID * stride] = make_float4(__uint_as_float(la | (lb << 16)), __int_as_float(ci),
                                             __int_as_float(side_bits(hd.z, fa, fb)), 0.f);
            if (!vel) continue;  // the position passes read the contact itself
            r[ROW_N * stride] = c4[1];
            r[ROW_T1 * stride] = c4[2];
            r[ROW_T2 * stride] = c4[3];
            Sym3 IA{0, 0, 0, 0, 0, 0}, IB{0, 0, 0, 0, 0, 0};
            if (da) IA = load_sym(w.inv_inertia_world, hd.x);
            if (db) IB = load_sym(w.inv_inertia_world, hd.y);
            const float ia[4] = {IA.xx, IA.xy, IA.xz, IA.yy}, ib[4] = {IB.xx, IB.xy, IB.xz, IB.yy};
            float en[4], e1[4], e2[4], bn[4], ln[4], l1[4], l2[4];
#pragma unroll
            for (int p = 0; p < 4; p++) {
                float4 q0 = make_float4(0.f, 0.f, 0.f, 0.f), q1 = q0, q3 = q0, q4 = q0;
                if (p < hd.z) {
                    const float4 *q = c4 + 5 + 5 * p;
                    q0 = q[0];
                    q1 = q[1];
                    q3 = q[3];
                    q4 = q[4];
                }
                r[(ROW_R + p) * stride] = make_float4(q0.x, q0.y, q0.z, ia[p]);
                r[(ROW_R + 4 + p) * stride] = make_float4(q0.w, q1.x, q1.y, ib[p]);
                en[p] = q3.x;
                e1[p] = q3.y;
                e2[p] = q3.z;
                ln[p] = q3.w;
                l1[p] = q4.x;
                l2[p] = q4.y;
                bn[p] = q4.z;
            }
            r[ROW_I * stride] = make_float4(IA.yz, IA.zz, IB.yz, IB.zz);
            r[ROW_EFFN * stride] = make_float4(en[0], en[1], en[2], en[3]);
            r[ROW_EFF1 * stride] = make_float4(e1[0], e1[1], e1[2], e1[3]);
            r[ROW_EFF2 * stride] = make_float4(e2[0], e2[1], e2[2], e2[3]);
            r[ROW_BIAS * stride] = make_float4(bn[0], bn[1], bn[2], bn[3]);
            r[ROW_LN * stride] = make_float4(ln[0], ln[1], ln[2], ln[3]);
            r[ROW_L1 * stride] = make_float4(l1[0], l1[1], l1[2], l1[3]);
            r[ROW_L2 * stride] = make_float4(l2[0], l2[1], l2[2], l2[3]);
        }
        __syncthreads();  // the lists are done with: their memory takes the state
        float *state = (float *)block_smem;  // 7 per body: velocities (6), then in the position sweeps the pose
        // a chunk's turn: every chunk of the earlier levels is done.  The wait is bounded: 32 polls of
        // shared memory for each poll of the whole-grid solve's barrier, which pauses between them
        const unsigned poll_limit = min(c_settings.wait_polls, ~0u / 32) * 32;
        auto turn = [&](int want) -> bool {
            bool ok = true;
            for (unsigned polls = 0; s_done < want; polls++)
                if (s_fail || polls > poll_limit) {
                    s_fail = 1;
                    atomicOr(&w.ctr->overflow, OVF_TIMEOUT);
                    ok = false;
                    break;
                }
            __threadfence_block();
            return __all_sync(FULL, ok);  // the lanes go on, or leave, together
        };
        auto chunk_done = [&]() {
            __syncwarp();
            if (lane == 0 && !(c_settings.test_withhold_block && wid == 0)) {
                __threadfence_block();
                atomicAdd((int *)&s_done, 1);
            }
        };
        if (vel) {
            for (int done = 0; done < vel_total;) {
                if (done > 0) nchunks = schedule(batch(vel_total, done), false, false);
                done += batch(vel_total, done);
                __syncthreads();
                for (int k = tid; k < nb; k += THREADS) {
                    const float4 v = w.linvel[bl[k]], a = w.angvel[bl[k]];
                    float *s = state + 7 * k;
                    s[0] = v.x;
                    s[1] = v.y;
                    s[2] = v.z;
                    s[3] = a.x;
                    s[4] = a.y;
                    s[5] = a.z;
                }
                __syncthreads();
                // a warp has the word and the tasks of its next chunk while it solves one
                auto task_of = [&](uint32_t word) -> unsigned {
                    return tasks[(word & 0x3ffffu) + (lane <= (int)((word >> 18) & 31u) ? lane : 0)];
                };
                uint32_t word1 = wid < nchunks ? chunks[wid] : 0u;
                unsigned task1 = wid < nchunks ? task_of(word1) : 0u;
                for (int i = wid; i < nchunks; i += W) {
                    const uint32_t word = word1;
                    const int dep = i - (int)(word >> 23);
                    const bool on = lane <= (int)((word >> 18) & 31u);
                    float4 *r = rows + (task1 & ~TASK_WARM);
                    const bool warm = (task1 & TASK_WARM) != 0;
                    // everything but the velocities and impulses, ahead of the turn
                    const float4 n4 = r[ROW_N * stride], t14 = r[ROW_T1 * stride], t24 = r[ROW_T2 * stride];
                    const float4 id = r[ROW_ID * stride];
                    const float4 en4 = r[ROW_EFFN * stride], e14 = r[ROW_EFF1 * stride], e24 = r[ROW_EFF2 * stride];
                    const float4 bn4 = r[ROW_BIAS * stride], i4 = r[ROW_I * stride];
                    float4 ra[4], rb[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        ra[k] = r[(ROW_R + k) * stride];
                        rb[k] = r[(ROW_R + 4 + k) * stride];
                    }
                    if (i + W < nchunks) {
                        word1 = chunks[i + W];
                        task1 = task_of(word1);
                    }
                    const float3 nn = xyz(n4), t1 = xyz(t14), t2 = xyz(t24);
                    const int bits = __float_as_int(id.z), n = bits & 15;
                    const unsigned la = __float_as_uint(id.x) & 0xffffu, lb = __float_as_uint(id.x) >> 16;
                    BodyRef A, B;
                    A.motion = (bits >> 4) & 3;
                    B.motion = (bits >> 6) & 3;
                    A.dof = (bits >> 8) & 63;
                    B.dof = (bits >> 16) & 63;
                    A.im = B.im = 0.f;
                    A.I = Sym3{ra[0].w, ra[1].w, ra[2].w, ra[3].w, i4.x, i4.y};
                    B.I = Sym3{rb[0].w, rb[1].w, rb[2].w, rb[3].w, i4.z, i4.w};
                    A.v = A.w = B.v = B.w = f3(0.f, 0.f, 0.f);
                    // a body of no island (static, or kinematic and asleep) keeps its velocity
                    if (la == BLOCK_NONE && A.motion != STATIC) {
                        const int g = w.cons[__float_as_int(id.y)].a;
                        A.v = xyz(w.linvel[g]);
                        A.w = xyz(w.angvel[g]);
                    }
                    if (lb == BLOCK_NONE && B.motion != STATIC) {
                        const int g = w.cons[__float_as_int(id.y)].b;
                        B.v = xyz(w.linvel[g]);
                        B.w = xyz(w.angvel[g]);
                    }
                    if (!turn(dep)) break;
                    const float4 ln4 = r[ROW_LN * stride], l14 = r[ROW_L1 * stride], l24 = r[ROW_L2 * stride];
                    if (la != BLOCK_NONE) {
                        const float *s = state + 7 * la;
                        A.v = f3(s[0], s[1], s[2]);
                        A.w = f3(s[3], s[4], s[5]);
                    }
                    if (lb != BLOCK_NONE) {
                        const float *s = state + 7 * lb;
                        B.v = f3(s[0], s[1], s[2]);
                        B.w = f3(s[3], s[4], s[5]);
                    }
                    PointRow p[4];
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        p[k] = PointRow{xyz(ra[k]),    xyz(rb[k]),    comp(en4, k), comp(e14, k), comp(e24, k),
                                        comp(ln4, k), comp(l14, k), comp(l24, k), comp(bn4, k)};
                    // the rows in the functions that every tier solves them with: the same operations
                    // in the same order, so the same bits
                    if (warm) {
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (k < n) warm_start_point(p[k], A, B, t14.w, t24.w, nn, t1, t2, ratio);
                    } else if (A.motion == DYNAMIC || B.motion == DYNAMIC) {
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (k < n) friction_point(p[k], A, B, t14.w, t24.w, t1, t2, n4.w);
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            if (k < n) normal_point(p[k], A, B, t14.w, t24.w, nn);
                    }
                    if (on) {
                        if (la != BLOCK_NONE && A.motion == DYNAMIC) {
                            float *s = state + 7 * la;
                            s[0] = A.v.x;
                            s[1] = A.v.y;
                            s[2] = A.v.z;
                            s[3] = A.w.x;
                            s[4] = A.w.y;
                            s[5] = A.w.z;
                        }
                        if (lb != BLOCK_NONE && B.motion == DYNAMIC) {
                            float *s = state + 7 * lb;
                            s[0] = B.v.x;
                            s[1] = B.v.y;
                            s[2] = B.v.z;
                            s[3] = B.w.x;
                            s[4] = B.w.y;
                            s[5] = B.w.z;
                        }
                        r[ROW_LN * stride] = make_float4(p[0].lam_n, p[1].lam_n, p[2].lam_n, p[3].lam_n);
                        r[ROW_L1 * stride] = make_float4(p[0].lam_t1, p[1].lam_t1, p[2].lam_t1, p[3].lam_t1);
                        r[ROW_L2 * stride] = make_float4(p[0].lam_t2, p[1].lam_t2, p[2].lam_t2, p[3].lam_t2);
                    }
                    chunk_done();
                }
                __syncthreads();
                if (s_fail) return;
                for (int k = tid; k < nb; k += THREADS) {
                    const int i = bl[k];
                    if (motion_of(w.flags[i]) != DYNAMIC) continue;
                    const float *s = state + 7 * k;
                    w.linvel[i] = make_float4(s[0], s[1], s[2], 0.f);
                    w.angvel[i] = make_float4(s[3], s[4], s[5], 0.f);
                }
            }
            __syncthreads();
            // impulses to the contacts and the cache, then the integration
            for (int k = tid; k < nc; k += THREADS) {
                const float4 id = rows[ROW_ID * stride + k];
                const float4 ln = rows[ROW_LN * stride + k], l1 = rows[ROW_L1 * stride + k], l2 = rows[ROW_L2 * stride + k];
                ContactConstraint &c = w.cons[__float_as_int(id.y)];
                CacheRecord *rec = crecs + c.cache_slot;
                const int n = __float_as_int(id.z) & 15;
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    if (p >= n) continue;
                    c.p[p].lam_n = rec->ln[p] = comp(ln, p);
                    c.p[p].lam_t1 = rec->lt1[p] = comp(l1, p);
                    c.p[p].lam_t2 = rec->lt2[p] = comp(l2, p);
                }
            }
            for (int k = tid; k < nb; k += THREADS) integrate_body(w, bl[k], dt, phase == SOLVE_VELOCITY);
            __syncthreads();
            if (phase == SOLVE_VELOCITY) continue;
        }
        // ---- position iterations (contact-constraints.ts:1098-1216).  The reference stops after a
        // sweep that moved nothing (update.ts:218-221); so would every later sweep ----
        for (int done = 0; done < pos_iters;) {
            if (vel || done > 0) nchunks = schedule(batch(pos_iters, done), false, false);
            done += batch(pos_iters, done);
            __syncthreads();
            for (int k = tid; k < nb; k += THREADS) {
                const float4 c = w.com[bl[k]], q = w.quat[bl[k]];
                float *s = state + 7 * k;
                s[0] = c.x;
                s[1] = c.y;
                s[2] = c.z;
                s[3] = q.x;
                s[4] = q.y;
                s[5] = q.z;
                s[6] = q.w;
            }
            if (tid == 0) s_any = 0;
            __syncthreads();
            bool any = false;
            for (int i = wid; i < nchunks; i += W) {
                const uint32_t word = chunks[i];
                const int first = (int)(word & 0x3ffffu), dep = i - (int)(word >> 23);
                const bool on = lane <= (int)((word >> 18) & 31u);
                const float4 id = rows[ROW_ID * stride + tasks[first + (on ? lane : 0)]];
                const float4 *c4 = (const float4 *)&w.cons[__float_as_int(id.y)];
                const int4 hd = *(const int4 *)c4;
                const uint32_t fa = w.flags[hd.x], fb = w.flags[hd.y];
                const unsigned la = __float_as_uint(id.x) & 0xffffu, lb = __float_as_uint(id.x) >> 16;
                PoseRef PA, PB;
                if (la == BLOCK_NONE) PA = PoseRef{xyz(w.com[hd.x]), w.quat[hd.x]};
                if (lb == BLOCK_NONE) PB = PoseRef{xyz(w.com[hd.y]), w.quat[hd.y]};
                if (!turn(dep)) break;
                if (on) {
                    if (la != BLOCK_NONE) {
                        const float *s = state + 7 * la;
                        PA = PoseRef{f3(s[0], s[1], s[2]), make_float4(s[3], s[4], s[5], s[6])};
                    }
                    if (lb != BLOCK_NONE) {
                        const float *s = state + 7 * lb;
                        PB = PoseRef{f3(s[0], s[1], s[2]), make_float4(s[3], s[4], s[5], s[6])};
                    }
                    const ContactConstraint &con = w.cons[__float_as_int(id.y)];
                    if (solve_position_con(w, con, PA, PB, motion_of(fa), motion_of(fb), fa, fb)) {
                        if (la != BLOCK_NONE && motion_of(fa) == DYNAMIC) {
                            float *s = state + 7 * la;
                            s[0] = PA.com.x;
                            s[1] = PA.com.y;
                            s[2] = PA.com.z;
                            s[3] = PA.q.x;
                            s[4] = PA.q.y;
                            s[5] = PA.q.z;
                            s[6] = PA.q.w;
                        }
                        if (lb != BLOCK_NONE && motion_of(fb) == DYNAMIC) {
                            float *s = state + 7 * lb;
                            s[0] = PB.com.x;
                            s[1] = PB.com.y;
                            s[2] = PB.com.z;
                            s[3] = PB.q.x;
                            s[4] = PB.q.y;
                            s[5] = PB.q.z;
                            s[6] = PB.q.w;
                        }
                        any = true;
                    }
                }
                chunk_done();
            }
            if (any) s_any = 1;
            __syncthreads();
            if (s_fail) return;
            for (int k = tid; k < nb; k += THREADS) {
                const int i = bl[k];
                if (motion_of(w.flags[i]) != DYNAMIC) continue;
                const float *s = state + 7 * k;
                w.com[i] = make_float4(s[0], s[1], s[2], 0.f);
                w.quat[i] = make_float4(s[3], s[4], s[5], s[6]);
            }
            const bool more = s_any != 0;
            __syncthreads();
            if (!more) break;
        }
        for (int k = tid; k < nb; k += THREADS) finish_body(w, bl[k]);
        __syncthreads();
        if (c_settings.allow_sleeping) {
            int mine = 1;
            for (int k = tid; k < nb; k += THREADS) {
                const int i = bl[k];
                if (motion_of(w.flags[i]) != DYNAMIC) continue;
                if (!sleep_update(w, i, dt)) mine = 0;
            }
            const int all = __syncthreads_and(mine);
            if (all)
                for (int k = tid; k < nb; k += THREADS)
                    if (motion_of(w.flags[bl[k]]) == DYNAMIC) sleep_body(w, bl[k]);
        }
        __syncthreads();
    }
}
