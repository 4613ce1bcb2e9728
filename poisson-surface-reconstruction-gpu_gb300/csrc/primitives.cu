// Hand-written radix sort (stable LSD, 8-bit digits, one look-back scatter per digit).
#include "primitives.cuh"

namespace psr {

static int g_num_sms = 0;

int scan_grid(int max_tiles, int blocks_per_sm) {
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_num_sms <= 0) g_num_sms = 148;
    }
    int g = g_num_sms * blocks_per_sm;
    return g < max_tiles ? g : (max_tiles > 0 ? max_tiles : 1);
}

// One pass: stable scatter of the tiles' keys by an 8-bit digit, tile offsets by decoupled
// look-back per digit (thread d: digit d).  A status word is a count (bits 0-29) | aggregate
// flag (30) | inclusive flag (31).  Tiles are claimed in order, so a tile only waits for tiles
// that run already.  Each thread reads kLook predecessors at once: at 200k keys all 98 tiles run
// together and a one-by-one walk over the others' aggregates would cost 97 L2 round trips.
// Within a tile, warp w owns keys [w*256, w*256+256) in striped order (item j of lane l is key
// w*256 + 32*j + l), so processing items in order and ranking equal digits with
// __match_any_sync preserves the input order.  Counting all digits once beside the encoder and
// scattering with look-back takes one launch per pass; a histogram, its size, its scan and the
// scatter took four (24 us a pass one after another at 200k keys, 7 now).
constexpr int kLook = 16;
enum : unsigned { kSortAgg = 1u << 30, kSortIncl = 1u << 31, kSortMask = kSortAgg - 1u };
__global__ void __launch_bounds__(kBlock) k_sort_pass(const unsigned* keys_in, const unsigned* vals_in,
                                                      unsigned* keys_out, unsigned* vals_out, const int* count_ptr,
                                                      int pass, SortScratch sc, unsigned* err) {
    PSR_CLOUD(keys_in, vals_in, keys_out, vals_out, count_ptr, sc, err);
    __shared__ unsigned s_cnt[kBlock / 32][kRadix];
    __shared__ unsigned s_off[kRadix];
    __shared__ int s_tile;
    const int n = *count_ptr;
    const int ntiles = (n + kSortTile - 1) / kSortTile;
    if (ntiles > sc.max_tiles) return;   // flagged by the counting kernel
    const int shift = pass * kRadixBits;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    volatile unsigned* status = sc.status + (size_t)pass * sc.max_tiles * kRadix;
    unsigned* next = sc.bins + kSortMaxPasses * kRadix + pass;
    while (true) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(next, 1u);
        for (int d = threadIdx.x; d < kRadix * (kBlock / 32); d += kBlock) (&s_cnt[0][0])[d] = 0;
        __syncthreads();
        const int t = s_tile;
        if (t >= ntiles) break;
        const int base = t * kSortTile + warp * 256;
        unsigned key[kSortItems], val[kSortItems], rank[kSortItems];
        bool ok[kSortItems];
#pragma unroll
        for (int j = 0; j < kSortItems; ++j) {
            const int i = base + 32 * j + lane;
            ok[j] = i < n;
            key[j] = ok[j] ? keys_in[i] : 0u;
            val[j] = !ok[j] ? 0u : vals_in ? vals_in[i] : (unsigned)i;
        }
#pragma unroll
        for (int j = 0; j < kSortItems; ++j) {
            const unsigned dgt = (key[j] >> shift) & (kRadix - 1);
            const unsigned act = __ballot_sync(0xffffffffu, ok[j]);
            rank[j] = 0;
            if (ok[j]) {
                const unsigned peers = __match_any_sync(act, dgt);
                const unsigned before = __popc(peers & lt_mask);
                const unsigned cur = s_cnt[warp][dgt];
                rank[j] = cur + before;
                __syncwarp(act);
                if (before == 0) s_cnt[warp][dgt] = cur + __popc(peers);
            }
            __syncwarp();
        }
        __syncthreads();
        {   // thread d: the digit's exclusive prefix over the warps (in place) and over the tiles
            const int d = threadIdx.x;
            unsigned run = 0;
#pragma unroll
            for (int w = 0; w < kBlock / 32; ++w) {
                const unsigned c = s_cnt[w][d];
                s_cnt[w][d] = run;
                run += c;
            }
            status[(size_t)t * kRadix + d] = (t == 0 ? kSortIncl : kSortAgg) | run;
            unsigned before = 0;
            bool found = t == 0, timeout = false;
            for (int p = t - 1; !found; p -= kLook) {
                unsigned s[kLook];
#pragma unroll
                for (int q = 0; q < kLook; ++q) s[q] = (p - q >= 0) ? status[(size_t)(p - q) * kRadix + d] : kSortIncl;
#pragma unroll
                for (int q = 0; q < kLook; ++q) {
                    if (found) continue;
                    for (int it = 0; !(s[q] & (kSortAgg | kSortIncl)); ++it) {
                        if (it > kSpinLimit) { timeout = true; s[q] = kSortIncl; break; }
                        __nanosleep(20);
                        s[q] = status[(size_t)(p - q) * kRadix + d];
                    }
                    before += s[q] & kSortMask;
                    found = (s[q] & kSortIncl) != 0u;
                }
            }
            if (timeout) atomicOr(err, kErrSpinTimeout);
            if (t > 0) status[(size_t)t * kRadix + d] = kSortIncl | (before + run);
            s_off[d] = sc.bins[pass * kRadix + d] + before;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kSortItems; ++j) {
            if (!ok[j]) continue;
            const unsigned dgt = (key[j] >> shift) & (kRadix - 1);
            const unsigned pos = s_off[dgt] + s_cnt[warp][dgt] + rank[j];
            if (pos < (unsigned)n) {   // always, unless a wait ran out
                keys_out[pos] = key[j];
                vals_out[pos] = val[j];
            }
        }
        __syncthreads();
    }
}

// p[0 .. n) = v, in every cloud of the launch
__global__ void __launch_bounds__(kBlock) k_fill_words(unsigned* p, unsigned v, long long n) {
    PSR_CLOUD(p);
    for (long long i = blockIdx.x * (long long)kBlock + threadIdx.x; i < n; i += (long long)gridDim.x * kBlock) p[i] = v;
}

cudaError_t fill_words(unsigned* p, unsigned v, long long n, int clouds, cudaStream_t stream) {
    const long long g = (n + kBlock - 1) / kBlock;
    const int cap = scan_grid(1 << 30, 4);
    const int gx = (int)(g < cap ? (g < 1 ? 1 : g) : cap);
    k_fill_words<<<dim3(cloud_blocks(clouds, gx), clouds), kBlock, 0, stream>>>(p, v, n);
    return cudaGetLastError();
}

cudaError_t radix_sort_pairs(unsigned* keys, unsigned* vals, const int* count_ptr, int key_bits, SortScratch sc,
                             unsigned* err, cudaStream_t stream, bool* result_in_alt) {
    const int passes = sort_passes(key_bits) < 1 ? 1 : sort_passes(key_bits);
    unsigned *ki = keys, *vi = nullptr, *ko = sc.keys_alt, *vo = sc.vals_alt;
    const dim3 grid(cloud_blocks(sc.batch, scan_grid(sc.max_tiles)), sc.batch);
    for (int p = 0; p < passes; ++p) {
        k_sort_pass<<<grid, kBlock, 0, stream>>>(ki, vi, ko, vo, count_ptr, p, sc, err);
        ki = ko;
        vi = vo;
        ko = (p & 1) ? sc.keys_alt : keys;
        vo = (p & 1) ? sc.vals_alt : vals;
    }
    *result_in_alt = (passes & 1) != 0;
    return cudaGetLastError();
}

}  // namespace psr
