// Islands above the per-warp tier and up to a pile of thousands of bodies: one CTA each, the
// island's body state in shared memory.  Included by cc_solver.cu after the solver primitives.
//
// The reference solves an island's contacts one after another in (sortKey, idA, idB) order.  Only
// contacts that share a dynamic body depend on each other, so a contact's level (one more than
// the levels of its predecessor on either body) says when it can run: the result of a sweep by
// levels is the sequential sweep's.  The levels of a heap are many and narrow (100 levels of 28
// contacts for 10 x 10 x 10 boxes), so a sweep is bound by the latency of one contact, not by
// bandwidth or arithmetic, and everything that does not depend on the velocities is taken out of
// that chain:
//   - the contacts are laid out in level order in chunks of at most 32 that one warp solves; chunk
//     i belongs to warp i mod W in every pass;
//   - the solver rows are repacked in that order, one coalesced float4 row per field, and a warp
//     loads its next chunk's rows into registers before it waits for the chunk's turn;
//   - the velocities (and in the position passes the poses) stay in shared memory;
//   - no barrier separates the levels: a counter of finished chunks is polled in shared memory,
//     and a chunk starts when every chunk of the earlier levels is counted.
// A level costs about 0.6 us (the sequential chain of four points' friction and normal rows); the
// whole-grid and barrier-per-colour solves it replaces took 10 us and more per colour.
#pragma once

// rows of the repacked contacts: row f of slot s at rows[f * stride + s]
enum : int {
    ROW_N = 0,      // normal, friction
    ROW_T1 = 1,     // first tangent, inverse mass of A
    ROW_T2 = 2,     // second tangent, inverse mass of B
    ROW_ID = 3,     // local bodies A | B << 16, constraint, SideBits, 0
    ROW_P = 4,      // 2 per point: rA, rB.x | rB.yz, bias, effective mass (normal)
    ROW_EFF1 = 12,  // effective masses of the first / second tangent rows, one component per point
    ROW_EFF2 = 13,
    ROW_LN = 14,    // accumulated impulses, one component per point
    ROW_L1 = 15,
    ROW_L2 = 16,
    ROW_I = 17,     // 3: world inverse inertias of A (6 values), then B (6)
    SOLVE_ROWS = 20
};
constexpr unsigned BLOCK_NONE = 0xffffu;  // no local body / no predecessor
// bits of ROW_ID.z: point count, motion types, degrees of freedom
__device__ __forceinline__ int side_bits(int n, uint32_t fa, uint32_t fb) {
    return n | (motion_of(fa) << 4) | (motion_of(fb) << 6) | (dof_of(fa) << 8) | (dof_of(fb) << 16);
}

struct PointRow {
    float3 rA, rB;
    float eff_n, eff_t1, eff_t2, lam_n, lam_t1, lam_t2, bias_n;
};
__device__ __forceinline__ float comp(const float4 &v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w)); }

// MC contacts and MB bodies at most, W warps.  The two instances differ in footprint: islands of
// up to 2,048 contacts and 1,024 bodies take four warps and 36 KB, so that two fit on an SM beside
// the other tiers' blocks; the larger ones take eight warps and most of an SM's shared memory.
template <int MC, int MB, int W>
struct BlockTier {
    static constexpr int CONS = MC, BODIES = MB, WARPS = W, THREADS = 32 * W;
    static constexpr size_t ORDER_BYTES = sizeof(int) * (2 * MB + 4) + (sizeof(uint32_t) + sizeof(uint16_t)) * 2 * MC;
    static constexpr size_t LEVEL_BYTES = sizeof(uint32_t) * MC + sizeof(int) * (MC + 4) + sizeof(uint16_t) * MC;
    static constexpr size_t STATE_BYTES = sizeof(float) * 7 * MB;
    static constexpr size_t SMEM = (ORDER_BYTES > LEVEL_BYTES ? (ORDER_BYTES > STATE_BYTES ? ORDER_BYTES : STATE_BYTES)
                                                              : (LEVEL_BYTES > STATE_BYTES ? LEVEL_BYTES : STATE_BYTES));
};
using BlockTierS = BlockTier<BLOCK_S_CONS, BLOCK_S_BODIES, 4>;
using BlockTierL = BlockTier<BLOCK_L_CONS, BLOCK_L_BODIES, 8>;
static_assert(BLOCK_L_CONS < 0xffff && BLOCK_L_BODIES < 0xffff, "16-bit local indices");
static_assert(sizeof(ContactConstraint) == 400 && sizeof(ContactPoint) == 80, "float4 loads of a contact");

// inclusive scan of a pair over the CTA, returned exclusive; the totals in tot
template <int W>
__device__ int2 block_scan_pair(int2 v, int2 *warp_tot, int2 &tot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int2 inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        int a = __shfl_up_sync(0xffffffffu, inc.x, o), b = __shfl_up_sync(0xffffffffu, inc.y, o);
        if (lane >= o) {
            inc.x += a;
            inc.y += b;
        }
    }
    __syncthreads();
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    int2 base = make_int2(0, 0);
    tot = make_int2(0, 0);
    for (int k = 0; k < W; k++) {
        int2 t = warp_tot[k];
        if (k < wid) {
            base.x += t.x;
            base.y += t.y;
        }
        tot.x += t.x;
        tot.y += t.y;
    }
    return make_int2(base.x + inc.x - v.x, base.y + inc.y - v.y);
}

// lists: the islands of this instance (from `first`, `step` apart)
template <class T>
__global__ void __launch_bounds__(T::THREADS, 1) k_solve_block(DevWorld w, CacheTables ct, const int *list, int step,
                                                               const int *count, float dt, float ratio, int phase) {
    if (islands_failed(w)) return;
    constexpr int W = T::WARPS, THREADS = T::THREADS;
    extern __shared__ __align__(16) unsigned char block_smem[];
    __shared__ int2 s_scan[W];
    __shared__ int s_any;
    __shared__ volatile int s_fail;
    __shared__ volatile int s_done;  // chunks finished since the pass counter was cleared
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
        int *lab = w.scratch_order + base;                 // per contact: dynamic local bodies A | B << 16
        int *chunk_x = w.scratch_colour + base;            // per chunk: first slot | contacts << 16
        int *chunk_dep = w.scratch_claim + w.cap + base;   // per chunk: chunks of the earlier levels
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
            s_done = 0;
            s_fail = 0;
        }
        __syncthreads();
        auto local_of = [&](int body) -> unsigned {
            int l = w.body_local[body];
            return l >= 0 && l < nb && bl[l] == body ? (unsigned)l : BLOCK_NONE;
        };
        for (int k = tid; k < nc; k += THREADS) {
            const ContactConstraint &c = w.cons[cl[k]];
            unsigned la = motion_of(w.flags[c.a]) == DYNAMIC ? local_of(c.a) : BLOCK_NONE;
            unsigned lb = motion_of(w.flags[c.b]) == DYNAMIC ? local_of(c.b) : BLOCK_NONE;
            lab[k] = (int)(la | (lb << 16));
            if (la != BLOCK_NONE) atomicAdd(&off[la], 1);
            if (lb != BLOCK_NONE) atomicAdd(&off[lb], 1);
        }
        __syncthreads();
        {
            const int seg = (nb + THREADS - 1) / THREADS, k0 = min(tid * seg, nb), k1 = min(k0 + seg, nb);
            int sum = 0;
            for (int k = k0; k < k1; k++) sum += off[k];
            int2 tot, ex = block_scan_pair<W>(make_int2(sum, 0), s_scan, tot);
            int at = ex.x;
            for (int k = k0; k < k1; k++) {
                int n = off[k];
                off[k] = fill[k] = at;
                at += n;
            }
            if (tid == 0) off[nb] = tot.x;
        }
        __syncthreads();
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
            chunk_x[k] = (int)(pred[0] | (pred[1] << 16));
        }
        __syncthreads();
        // ---- levels, from 1: in place until every contact has one (the values do not depend on
        // the order in which they are found) ----
        uint32_t *pred = (uint32_t *)block_smem;
        int *at = (int *)(pred + T::CONS);  // contacts per level, then the level's next slot
        uint16_t *lev = (uint16_t *)(at + T::CONS + 4);
        for (int k = tid; k < nc; k += THREADS) {
            pred[k] = (uint32_t)chunk_x[k];
            lev[k] = 0;
            at[k] = 0;
        }
        __syncthreads();
        volatile uint16_t *vlev = lev;
        int left;
        do {
            left = 0;
            for (int k = tid; k < nc; k += THREADS) {
                if (vlev[k]) continue;
                const unsigned pa = pred[k] & 0xffffu, pb = pred[k] >> 16;
                const int a = pa == BLOCK_NONE ? 0 : vlev[pa], b = pb == BLOCK_NONE ? 0 : vlev[pb];
                if ((pa == BLOCK_NONE || a) && (pb == BLOCK_NONE || b))
                    vlev[k] = (uint16_t)(max(a, b) + 1);
                else
                    left = 1;
            }
        } while (__syncthreads_or(left));
        for (int k = tid; k < nc; k += THREADS) atomicAdd(&at[lev[k] - 1], 1);
        __syncthreads();
        // ---- chunks: each level's contacts in groups of 32 ----
        int nchunks;
        {
            const int seg = (nc + THREADS - 1) / THREADS, l0 = min(tid * seg, nc), l1 = min(l0 + seg, nc);
            int2 sum = make_int2(0, 0);
            for (int l = l0; l < l1; l++) {
                sum.x += at[l];
                sum.y += (at[l] + 31) >> 5;
            }
            int2 tot, ex = block_scan_pair<W>(sum, s_scan, tot);
            nchunks = tot.y;
            for (int l = l0; l < l1; l++) {
                const int n = at[l];
                at[l] = ex.x;
                for (int j = 0; 32 * j < n; j++) {
                    chunk_x[ex.y + j] = (ex.x + 32 * j) | (min(32, n - 32 * j) << 16);
                    chunk_dep[ex.y + j] = ex.y;
                }
                ex.x += n;
                ex.y += (n + 31) >> 5;
            }
        }
        __syncthreads();
        // ---- the contacts' rows in slot order (the order inside a level is free) ----
        for (int k = tid; k < nc; k += THREADS) {
            const int ci = cl[k], slot = atomicAdd(&at[lev[k] - 1], 1);
            const float4 *c4 = (const float4 *)&w.cons[ci];
            const int4 hd = *(const int4 *)c4;  // a, b, n, island
            const uint32_t fa = w.flags[hd.x], fb = w.flags[hd.y];
            const unsigned la = local_of(hd.x), lb = local_of(hd.y);
            float4 *r = rows + slot;
            r[ROW_ID * stride] = make_float4(__uint_as_float(la | (lb << 16)), __int_as_float(ci),
                                             __int_as_float(side_bits(hd.z, fa, fb)), 0.f);
            if (!vel) continue;  // the position passes read the contact itself
            r[ROW_N * stride] = c4[1];
            r[ROW_T1 * stride] = c4[2];
            r[ROW_T2 * stride] = c4[3];
            float e1[4], e2[4], ln[4], l1[4], l2[4];
#pragma unroll
            for (int p = 0; p < 4; p++) {
                e1[p] = e2[p] = ln[p] = l1[p] = l2[p] = 0.f;
                if (p >= hd.z) continue;
                const float4 *q = c4 + 5 + 5 * p;
                const float4 q0 = q[0], q1 = q[1], q3 = q[3], q4 = q[4];
                r[(ROW_P + 2 * p) * stride] = q0;
                r[(ROW_P + 2 * p + 1) * stride] = make_float4(q1.x, q1.y, q4.z, q3.x);
                e1[p] = q3.y;
                e2[p] = q3.z;
                ln[p] = q3.w;
                l1[p] = q4.x;
                l2[p] = q4.y;
            }
            r[ROW_EFF1 * stride] = make_float4(e1[0], e1[1], e1[2], e1[3]);
            r[ROW_EFF2 * stride] = make_float4(e2[0], e2[1], e2[2], e2[3]);
            r[ROW_LN * stride] = make_float4(ln[0], ln[1], ln[2], ln[3]);
            r[ROW_L1 * stride] = make_float4(l1[0], l1[1], l1[2], l1[3]);
            r[ROW_L2 * stride] = make_float4(l2[0], l2[1], l2[2], l2[3]);
            Sym3 IA{0, 0, 0, 0, 0, 0}, IB{0, 0, 0, 0, 0, 0};
            if (motion_of(fa) == DYNAMIC) IA = load_sym(w.inv_inertia_world, hd.x);
            if (motion_of(fb) == DYNAMIC) IB = load_sym(w.inv_inertia_world, hd.y);
            r[ROW_I * stride] = make_float4(IA.xx, IA.xy, IA.xz, IA.yy);
            r[(ROW_I + 1) * stride] = make_float4(IA.yz, IA.zz, IB.xx, IB.xy);
            r[(ROW_I + 2) * stride] = make_float4(IB.xz, IB.yy, IB.yz, IB.zz);
        }
        __syncthreads();  // the order and level arrays are done with: their memory takes the state
        float *state = (float *)block_smem;  // 7 per body: velocities (6), then in the position passes the pose
        // a chunk's turn: every chunk of the earlier passes and levels is done (bounded wait)
        int passes = 0;
        auto turn = [&](int dep) -> bool {
            const int want = passes * nchunks + dep;
            bool ok = true;
            for (unsigned polls = 0; s_done < want; polls++)
                if (s_fail || polls > (1u << 26)) {
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
            if (lane == 0) {
                __threadfence_block();
                atomicAdd((int *)&s_done, 1);
            }
        };
        if (vel) {
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
            bool ok = true;
            for (int pass = c_settings.warm_starting ? -1 : 0; ok && pass < vel_iters; pass++, passes++) {
                for (int i = wid; i < nchunks; i += W) {
                    const int cx = chunk_x[i], dep = chunk_dep[i];
                    const bool on = lane < (cx >> 16);
                    const float4 *r = rows + (cx & 0xffff) + (on ? lane : 0);
                    // everything but the velocities, ahead of the turn
                    const float4 n4 = r[ROW_N * stride], t14 = r[ROW_T1 * stride], t24 = r[ROW_T2 * stride];
                    const float4 id = r[ROW_ID * stride];
                    const float4 e1 = r[ROW_EFF1 * stride], e2 = r[ROW_EFF2 * stride];
                    float4 ln = r[ROW_LN * stride], l1 = r[ROW_L1 * stride], l2 = r[ROW_L2 * stride];
                    const float4 i0 = r[ROW_I * stride], i1 = r[(ROW_I + 1) * stride], i2 = r[(ROW_I + 2) * stride];
                    const int bits = __float_as_int(id.z), n = bits & 15;
                    PointRow p[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                        if (k < n) {
                            a = r[(ROW_P + 2 * k) * stride];
                            b = r[(ROW_P + 2 * k + 1) * stride];
                        }
                        p[k].rA = f3(a.x, a.y, a.z);
                        p[k].rB = f3(a.w, b.x, b.y);
                        p[k].bias_n = b.z;
                        p[k].eff_n = b.w;
                        p[k].eff_t1 = comp(e1, k);
                        p[k].eff_t2 = comp(e2, k);
                        p[k].lam_n = comp(ln, k);
                        p[k].lam_t1 = comp(l1, k);
                        p[k].lam_t2 = comp(l2, k);
                    }
                    const unsigned la = __float_as_uint(id.x) & 0xffffu, lb = __float_as_uint(id.x) >> 16;
                    BodyRef A, B;
                    A.motion = (bits >> 4) & 3;
                    B.motion = (bits >> 6) & 3;
                    A.dof = (bits >> 8) & 63;
                    B.dof = (bits >> 16) & 63;
                    A.im = B.im = 0.f;
                    A.I = Sym3{i0.x, i0.y, i0.z, i0.w, i1.x, i1.y};
                    B.I = Sym3{i1.z, i1.w, i2.x, i2.y, i2.z, i2.w};
                    A.v = A.w = B.v = B.w = f3(0.f, 0.f, 0.f);
                    // a body of no island (static, or asleep and kinematic) keeps its velocity
                    if (on && la == BLOCK_NONE && A.motion != STATIC) {
                        const int g = w.cons[__float_as_int(id.y)].a;
                        A.v = xyz(w.linvel[g]);
                        A.w = xyz(w.angvel[g]);
                    }
                    if (on && lb == BLOCK_NONE && B.motion != STATIC) {
                        const int g = w.cons[__float_as_int(id.y)].b;
                        B.v = xyz(w.linvel[g]);
                        B.w = xyz(w.angvel[g]);
                    }
                    if (!(ok = turn(dep))) break;
                    if (on) {
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
                        const float3 nn = xyz(n4), t1 = xyz(t14), t2 = xyz(t24);
                        if (pass < 0) {
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
                    }
                    chunk_done();
                    if (on) {  // the impulses are this lane's alone: not part of the turn
                        float4 *ro = rows + (cx & 0xffff) + lane;
                        ro[ROW_LN * stride] = make_float4(p[0].lam_n, p[1].lam_n, p[2].lam_n, p[3].lam_n);
                        ro[ROW_L1 * stride] = make_float4(p[0].lam_t1, p[1].lam_t1, p[2].lam_t1, p[3].lam_t1);
                        ro[ROW_L2 * stride] = make_float4(p[0].lam_t2, p[1].lam_t2, p[2].lam_t2, p[3].lam_t2);
                    }
                }
            }
            __syncthreads();
            if (s_fail) return;
            // impulses to the contacts and the cache, velocities to the bodies, integration
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
            for (int k = tid; k < nb; k += THREADS) {
                const int i = bl[k];
                if (motion_of(w.flags[i]) == DYNAMIC) {
                    const float *s = state + 7 * k;
                    w.linvel[i] = make_float4(s[0], s[1], s[2], 0.f);
                    w.angvel[i] = make_float4(s[3], s[4], s[5], 0.f);
                }
                integrate_body(w, i, dt, phase == SOLVE_VELOCITY);
            }
            __syncthreads();
            if (phase == SOLVE_VELOCITY) continue;
        }
        // ---- position iterations (contact-constraints.ts:1098-1216), early exit as update.ts:218-221 ----
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
        if (tid == 0) s_done = 0;
        passes = 0;
        __syncthreads();
        for (int it = 0; it < pos_iters; it++, passes++) {
            if (tid == 0) s_any = 0;
            __syncthreads();
            bool any = false, ok = true;
            for (int i = wid; i < nchunks; i += W) {
                const int cx = chunk_x[i], dep = chunk_dep[i];
                const bool on = lane < (cx >> 16);
                const float4 id = rows[ROW_ID * stride + (cx & 0xffff) + (on ? lane : 0)];
                const float4 *c4 = (const float4 *)&w.cons[__float_as_int(id.y)];
                const int4 hd = *(const int4 *)c4;
                const float4 n4 = c4[1], m1 = c4[2], m2 = c4[3];
                const int bits = __float_as_int(id.z), n = bits & 15;
                float3 la3[4], lb3[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    la3[k] = lb3[k] = f3(0.f, 0.f, 0.f);
                    if (k < n) {
                        const float4 a = c4[6 + 5 * k], b = c4[7 + 5 * k];
                        la3[k] = f3(a.z, a.w, b.x);
                        lb3[k] = f3(b.y, b.z, b.w);
                    }
                }
                const unsigned la = __float_as_uint(id.x) & 0xffffu, lb = __float_as_uint(id.x) >> 16;
                PoseSide SA{(bits >> 4) & 3, (bits >> 8) & 63, w.inertia_rot[hd.x], xyz(w.inv_inertia[hd.x]), m1.w};
                PoseSide SB{(bits >> 6) & 3, (bits >> 16) & 63, w.inertia_rot[hd.y], xyz(w.inv_inertia[hd.y]), m2.w};
                PoseRef PA, PB;
                if (la == BLOCK_NONE) PA = PoseRef{xyz(w.com[hd.x]), w.quat[hd.x]};
                if (lb == BLOCK_NONE) PB = PoseRef{xyz(w.com[hd.y]), w.quat[hd.y]};
                if (!(ok = turn(dep))) break;
                if (on && (SA.motion == DYNAMIC || SB.motion == DYNAMIC)) {
                    if (la != BLOCK_NONE) {
                        const float *s = state + 7 * la;
                        PA = PoseRef{f3(s[0], s[1], s[2]), make_float4(s[3], s[4], s[5], s[6])};
                    }
                    if (lb != BLOCK_NONE) {
                        const float *s = state + 7 * lb;
                        PB = PoseRef{f3(s[0], s[1], s[2]), make_float4(s[3], s[4], s[5], s[6])};
                    }
                    const Mat3 RA = quat_to_mat(PA.q), RB = quat_to_mat(PB.q);
                    Sym3 IA{0, 0, 0, 0, 0, 0}, IB{0, 0, 0, 0, 0, 0};
                    if (SA.motion == DYNAMIC) IA = world_inv_inertia(PA.q, SA.inertia_rot, SA.inv_inertia, SA.dof);
                    if (SB.motion == DYNAMIC) IB = world_inv_inertia(PB.q, SB.inertia_rot, SB.inv_inertia, SB.dof);
                    bool applied = false;
                    for (int k = 0; k < n; k++) {
                        const float3 pa = k == 0 ? la3[0] : (k == 1 ? la3[1] : (k == 2 ? la3[2] : la3[3]));
                        const float3 pb = k == 0 ? lb3[0] : (k == 1 ? lb3[1] : (k == 2 ? lb3[2] : lb3[3]));
                        applied = position_point(pa, pb, xyz(n4), PA, PB, RA, RB, IA, IB, SA, SB) || applied;
                    }
                    if (applied) {
                        if (la != BLOCK_NONE && SA.motion == DYNAMIC) {
                            float *s = state + 7 * la;
                            s[0] = PA.com.x;
                            s[1] = PA.com.y;
                            s[2] = PA.com.z;
                            s[3] = PA.q.x;
                            s[4] = PA.q.y;
                            s[5] = PA.q.z;
                            s[6] = PA.q.w;
                        }
                        if (lb != BLOCK_NONE && SB.motion == DYNAMIC) {
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
            const bool more = s_any != 0;
            __syncthreads();
            if (!more) break;
        }
        for (int k = tid; k < nb; k += THREADS) {
            const int i = bl[k];
            if (motion_of(w.flags[i]) == DYNAMIC) {
                const float *s = state + 7 * k;
                w.com[i] = make_float4(s[0], s[1], s[2], 0.f);
                w.quat[i] = make_float4(s[3], s[4], s[5], s[6]);
            }
            finish_body(w, i);
        }
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
