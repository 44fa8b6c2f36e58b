// Stable LSD radix sort of up to SORT_SMALL (key, index) pairs by one block in shared memory.
#pragma once
#include "cc_internal.cuh"

namespace cc {

constexpr int SORT_BLOCK = 1024, SORT_WARPS = SORT_BLOCK / 32, SORT_SMALL = 9216;

struct SmallSort {
    static constexpr int ITEMS = SORT_SMALL / SORT_BLOCK;  // keys per lane at most
    static constexpr int ROW = 257;                        // digit counts of a warp, padded against bank conflicts
    unsigned long long *key[2];
    uint16_t *val[2];
    int *count;  // SORT_WARPS x ROW
    __host__ __device__ static size_t bytes(int n) {
        const size_t m = ((size_t)n + 31) / 32 * 32;
        return m * (2 * sizeof(unsigned long long) + 2 * sizeof(uint16_t)) + sizeof(int) * SORT_WARPS * ROW;
    }
    __device__ SmallSort(unsigned char *smem, int n) {
        const int m = (n + 31) / 32 * 32;
        key[0] = (unsigned long long *)smem;
        key[1] = key[0] + m;
        count = (int *)(key[1] + m);
        val[0] = (uint16_t *)(count + SORT_WARPS * ROW);
        val[1] = val[0] + m;
    }
    // Sorts key[0], val[0] (filled by any thread) by the low `bits` bits; returns the buffer that
    // holds the result.  Begins and ends with a barrier.
    __device__ int sort(int n, int bits) {
        __shared__ int warp_tot[SORT_WARPS];
        const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
        const unsigned FULL = 0xffffffffu, lt = (1u << lane) - 1u;
        const int per = ((n + SORT_BLOCK - 1) / SORT_BLOCK) * 32;  // keys per warp, a multiple of 32
        int *mine = count + wid * ROW;
        int b = 0;
        for (int shift = 0; shift < bits; shift += 8, b ^= 1) {
            for (int k = tid; k < SORT_WARPS * ROW; k += SORT_BLOCK) count[k] = 0;
            __syncthreads();
            int rank[ITEMS];
#pragma unroll
            for (int it = 0; it < ITEMS; it++) {
                const int i = wid * per + it * 32 + lane;
                rank[it] = 0;
                if (it * 32 >= per) break;  // the same for the whole block
                const bool valid = i < n;
                const int d = valid ? (int)((key[b][i] >> shift) & 255) : 256 + lane;
                const unsigned peers = __match_any_sync(FULL, d);
                const int leader = __ffs(peers) - 1;
                int base = 0;
                if (valid && lane == leader) {
                    base = mine[d];
                    mine[d] = base + __popc(peers);
                }
                rank[it] = __shfl_sync(FULL, base, leader) + __popc(peers & lt);
                __syncwarp();
            }
            __syncthreads();
            // exclusive scan over (digit, warp): thread t takes digit t / 4, warps 8 (t mod 4) .. + 8
            int c[8], sum = 0;
            const int d = tid >> 2, w0 = (tid & 3) * 8;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                c[k] = count[(w0 + k) * ROW + d];
                sum += c[k];
            }
            int inc = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += v;
            }
            if (lane == 31) warp_tot[wid] = inc;
            __syncthreads();
            if (wid == 0) {
                const int v = warp_tot[lane];
                int s = v;
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(FULL, s, o);
                    if (lane >= o) s += u;
                }
                warp_tot[lane] = s - v;
            }
            __syncthreads();
            int at = warp_tot[wid] + inc - sum;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                count[(w0 + k) * ROW + d] = at;
                at += c[k];
            }
            __syncthreads();
#pragma unroll
            for (int it = 0; it < ITEMS; it++) {
                const int i = wid * per + it * 32 + lane;
                if (it * 32 >= per) break;
                if (i >= n) continue;
                const unsigned long long k = key[b][i];
                const int to = mine[(int)((k >> shift) & 255)] + rank[it];
                key[b ^ 1][to] = k;
                val[b ^ 1][to] = val[b][i];
            }
            __syncthreads();
        }
        return b;
    }
};

}  // namespace cc
