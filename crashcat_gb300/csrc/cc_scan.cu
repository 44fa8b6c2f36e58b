// Device-wide exclusive scan and stable LSD radix sort (64-bit keys, int
// values) used by the broadphase and island construction.  Both are written
// for this project: tiles of 4096 elements per CTA, three launches per scan
// and per radix pass; few elements take one block and one launch.
#include <utility>

#include "cc_internal.cuh"
#include "cc_per_device.h"
#include "cc_sort_small.cuh"

namespace cc {

// SM count of the current device; 152 when the attribute cannot be read
int device_sm_count() {
    static PerDevice count;
    return count.get([] {
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 152;
        return v;
    });
}

constexpr int SCAN_BLOCK = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

__device__ __forceinline__ int warp_incl_scan(int v) {
    int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// exclusive block scan of one value per thread; returns exclusive prefix, writes block total
__device__ int block_excl_scan(int v, int *total) {
    __shared__ int warp_sums[32];
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = warp_incl_scan(v);
    if (lane == 31) warp_sums[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int nw = (blockDim.x + 31) >> 5;
        int s = lane < nw ? warp_sums[lane] : 0;
        int si = warp_incl_scan(s);
        if (lane < nw) warp_sums[lane] = si - s;
        if (lane == nw - 1 && total) *total = si;
    }
    __syncthreads();
    int r = warp_sums[wid] + inc - v;
    __syncthreads();
    return r;
}

__global__ void k_scan_reduce(const int *in, int n, int *block_sums) {
    int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        int i = base + k;
        if (i < n) s += in[i];
    }
    __shared__ int tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = tot;
}

__global__ void k_scan_blocks(int *block_sums, int nb, int *total) {
    // single CTA scans up to SCAN_TILE block sums
    int base = threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        v[k] = (base + k < nb) ? block_sums[base + k] : 0;
        s += v[k];
    }
    __shared__ int tot;
    int off = block_excl_scan(s, &tot);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        if (base + k < nb) block_sums[base + k] = off;
        off += v[k];
    }
    if (threadIdx.x == 0 && total) *total = tot;
}

__global__ void k_scan_apply(const int *in, int *out, int n, const int *block_offsets) {
    int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        s += v[k];
    }
    int off = block_excl_scan(s, nullptr) + block_offsets[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        if (base + k < n) out[base + k] = off;
        off += v[k];
    }
}

size_t scan_tmp_ints(int n) {
    size_t nb = (size_t)(n + SCAN_TILE - 1) / SCAN_TILE + 1;
    // radix histograms: 256 digits x blocks of 4096 keys
    size_t rb = (size_t)(n + 4095) / 4096 + 1;
    size_t need = rb * 256 + 64;
    return (nb > need ? nb : need) + 64;
}

// Scans of up to SCAN_ONE entries by one block each, tile after tile with the sum carried along:
// one launch in place of three (7,518 entries: 7 us against 11 us; at 32,000 entries one block takes
// 18 us, the three launches 13 us).
constexpr int SCAN_ONE = 16384;
struct ScanJob {
    const int *in;
    int *out, *total;
};
struct ScanJobs {
    ScanJob job[3];
};
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_one(ScanJobs jobs, int n) {
    const ScanJob j = jobs.job[blockIdx.x];
    int carry = 0;
    __shared__ int tot;
    for (int tile = 0; tile < n; tile += SCAN_TILE) {
        const int base = tile + threadIdx.x * SCAN_ITEMS;
        int v[SCAN_ITEMS], s = 0;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            v[k] = (base + k < n) ? j.in[base + k] : 0;
            s += v[k];
        }
        int off = carry + block_excl_scan(s, &tot);
        carry += tot;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            if (base + k < n) j.out[base + k] = off;
            off += v[k];
        }
        __syncthreads();  // the next tile writes tot
    }
    if (threadIdx.x == 0 && j.total) *j.total = carry;
}

// Up to three scans of the same length, side by side (in: null to leave one out)
void exclusive_scan_multi(const int *in0, int *out0, const int *in1, int *out1, const int *in2, int *out2, int n,
                          int *tmp, cudaStream_t s) {
    if (n <= 0) return;
    if (n <= SCAN_ONE) {
        ScanJobs jobs{{{in0, out0, nullptr}, {in1, out1, nullptr}, {in2, out2, nullptr}}};
        k_scan_one<<<in2 ? 3 : 2, SCAN_BLOCK, 0, s>>>(jobs, n);
        return;
    }
    exclusive_scan_int(in0, out0, n, nullptr, tmp, s);
    exclusive_scan_int(in1, out1, n, nullptr, tmp, s);
    if (in2) exclusive_scan_int(in2, out2, n, nullptr, tmp, s);
}

// out[i] = sum in[0..i-1]; *total = sum of all (device pointer, may be null)
void exclusive_scan_int(const int *in, int *out, int n, int *total, int *tmp, cudaStream_t s) {
    if (n <= 0) return;
    if (n <= SCAN_ONE) {
        ScanJobs jobs{{{in, out, total}, {}, {}}};
        k_scan_one<<<1, SCAN_BLOCK, 0, s>>>(jobs, n);
        return;
    }
    int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    k_scan_reduce<<<nb, SCAN_BLOCK, 0, s>>>(in, n, tmp);
    k_scan_blocks<<<1, SCAN_BLOCK, 0, s>>>(tmp, nb, total);
    k_scan_apply<<<nb, SCAN_BLOCK, 0, s>>>(in, out, n, tmp);
}

// ---------------------------------------------------------------------------
// radix sort
// ---------------------------------------------------------------------------
constexpr int RS_BLOCK = 512, RS_WARPS = RS_BLOCK / 32;
constexpr int RS_ITEMS = 8;
constexpr int RS_TILE = RS_BLOCK * RS_ITEMS;  // 4096 keys per CTA

__global__ void __launch_bounds__(RS_BLOCK) k_radix_hist(const unsigned long long *keys, int n, int shift, int *hist,
                                                         int nblocks) {
    __shared__ int h[256];
    if (threadIdx.x < 256) h[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * RS_TILE;
#pragma unroll
    for (int k = 0; k < RS_ITEMS; k++) {
        int i = base + k * RS_BLOCK + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255], 1);
    }
    __syncthreads();
    if (threadIdx.x < 256) hist[threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of a tile.  Each warp ranks a contiguous run of 256 keys with warp matches against
// its own digit counts (no barrier inside the run), then the counts become places: the digit's place
// of the tile plus the warps before.  A pass over chunks of 256 keys with five barriers each took 28 us
// a digit for 511,195 keys (and for 8,320: three busy CTAs), this takes 10 us.
__global__ void __launch_bounds__(RS_BLOCK) k_radix_scatter(const unsigned long long *keys, const int *vals,
                                                            unsigned long long *okeys, int *ovals, int n, int shift,
                                                            const int *hist_off, int nblocks) {
    __shared__ int count[RS_WARPS][257];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned FULL = 0xffffffffu, lt = (1u << lane) - 1u;
    for (int k = tid; k < RS_WARPS * 257; k += RS_BLOCK) (&count[0][0])[k] = 0;
    const int base = blockIdx.x * RS_TILE + wid * (32 * RS_ITEMS) + lane;
    unsigned long long key[RS_ITEMS];
    int val[RS_ITEMS], rank[RS_ITEMS];
#pragma unroll
    for (int it = 0; it < RS_ITEMS; it++) {
        const int i = base + 32 * it;
        key[it] = i < n ? keys[i] : 0ull;
        val[it] = i < n ? vals[i] : 0;
    }
    __syncthreads();
    int *mine = count[wid];
#pragma unroll
    for (int it = 0; it < RS_ITEMS; it++) {
        const bool valid = base + 32 * it < n;
        const int d = valid ? (int)((key[it] >> shift) & 255) : 256 + lane;  // invalid lanes match no valid one
        const unsigned peers = __match_any_sync(FULL, d);
        const int leader = __ffs(peers) - 1;
        int before = 0;
        if (valid && lane == leader) {
            before = mine[d];
            mine[d] = before + __popc(peers);
        }
        rank[it] = __shfl_sync(FULL, before, leader) + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();
    if (tid < 256) {
        int at = hist_off[tid * nblocks + blockIdx.x];
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) {
            const int c = count[w][tid];
            count[w][tid] = at;
            at += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < RS_ITEMS; it++) {
        if (base + 32 * it >= n) break;
        const int to = mine[(int)((key[it] >> shift) & 255)] + rank[it];
        okeys[to] = key[it];
        ovals[to] = val[it];
    }
}

// Few keys: the whole sort in one block, keys and values in shared memory (one launch in place of
// five a digit, which took 300 us on 7,518 keys of 36 bits; this takes 12).  Stable: each warp
// ranks a contiguous run of keys with warp matches against its own digit counts, and the counts
// are scanned digit by digit, warp by warp.
__global__ void __launch_bounds__(SORT_BLOCK) k_radix_sort_small(unsigned long long *keys, int *vals, int n, int bits) {
    extern __shared__ __align__(16) unsigned char sort_smem[];
    SmallSort S(sort_smem, n);
    for (int i = threadIdx.x; i < n; i += SORT_BLOCK) {
        S.key[0][i] = keys[i];
        S.val[0][i] = (uint16_t)i;
    }
    const int b = S.sort(n, bits);
    // the values move once, by their sorted places (through the other key buffer)
    int *moved = (int *)S.key[b ^ 1];
    for (int i = threadIdx.x; i < n; i += SORT_BLOCK) moved[i] = vals[S.val[b][i]];
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += SORT_BLOCK) {
        keys[i] = S.key[b][i];
        vals[i] = moved[i];
    }
}

// Sorts (keys, vals) by the low `bits` bits of the keys; result ends in keys/vals.
// ints of scratch radix_sort_pairs_u64 needs for n keys
size_t radix_tmp_ints(int n) {
    size_t nblocks = (size_t)(n + RS_TILE - 1) / RS_TILE;
    return nblocks * 256 + 32 + scan_tmp_ints((int)(nblocks * 256));
}

void radix_sort_pairs_u64(unsigned long long *keys, unsigned long long *keys_alt, int *vals, int *vals_alt, int n,
                          int bits, int *tmp, cudaStream_t s, const int *) {
    if (n <= 1) return;
    if (n <= SORT_SMALL) {
        static PerDevice shared;
        shared.get([] { return allow_shared(SmallSort::bytes(SORT_SMALL), k_radix_sort_small); });
        k_radix_sort_small<<<1, SORT_BLOCK, SmallSort::bytes(n), s>>>(keys, vals, n, bits);
        return;
    }
    int nblocks = (n + RS_TILE - 1) / RS_TILE;
    int passes = (bits + 7) / 8;
    if (passes & 1) passes++;  // even number of passes leaves the result in the primary buffers
    int *hist = tmp;
    int *scan_tmp = tmp + (size_t)nblocks * 256 + 32;
    unsigned long long *ki = keys, *ko = keys_alt;
    int *vi = vals, *vo = vals_alt;
    for (int p = 0; p < passes; p++) {
        int shift = p * 8;
        k_radix_hist<<<nblocks, RS_BLOCK, 0, s>>>(ki, n, shift, hist, nblocks);
        exclusive_scan_int(hist, hist, nblocks * 256, nullptr, scan_tmp, s);
        k_radix_scatter<<<nblocks, RS_BLOCK, 0, s>>>(ki, vi, ko, vo, n, shift, hist, nblocks);
        std::swap(ki, ko);
        std::swap(vi, vo);
    }
}

}  // namespace cc
