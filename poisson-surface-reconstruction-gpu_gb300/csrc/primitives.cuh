// Hand-written device-wide primitives: single-pass prefix scan with fused load / store
// functors (decoupled look-back, dynamic tile ids, bounded waits) and a stable LSD radix
// sort of (32-bit key, 32-bit value) pairs.  Problem sizes are read from device memory.
#pragma once
#include "psr_common.cuh"

namespace psr {

constexpr int kScanItems = 8;                    // default items per thread
constexpr int kScanMinTile = kBlock;             // smallest tile (1 item per thread)

// Scratch of the scans: [0] tile counter, [1] blocks finished, [2] epoch, [3 + t] status
// of tile t.  A status word is value (bits 0-31) | aggregate flag (32) | inclusive flag
// (33) | epoch (34-63); only statuses of the running launch's epoch count, so nothing is
// cleared between launches: the last block of a launch resets the counters and advances
// the epoch (launches on one stream are ordered, so the next launch sees both).
struct ScanScratch {
    unsigned long long* words;
    int max_tiles;
    int batch = 1;   // clouds of the launch (host side: the grid's y extent)
    __device__ void rebase() { PSR_CLOUD(words); }   // to cloud blockIdx.y
};
constexpr int kScanHeader = 3;

// Flattens ranges over the kLanes lanes of a group (mask gmask): each lane hands in one range per call
// (cnt elements from `base`), ranges in lane order, call after call.  Only ranges with elements are
// listed: list entry j starts at flat index off[j], and element t of it is t + from[j].  After the
// last call one lane sets off[used] = 0x7fffffff, so that a walk over increasing t needs no other end.
// Every lane walks the list, which is why it is short: of 27 cells around a surface point two thirds
// are empty.
template <int kLanes>
__device__ __forceinline__ void list_range(unsigned gmask, int cnt, int base, int* off, int* from, int& used,
                                           int& running) {
    const int lane = threadIdx.x & (kLanes - 1);
    int incl = cnt;
#pragma unroll
    for (int q = 1; q < kLanes; q <<= 1) {
        const int y = __shfl_up_sync(gmask, incl, q, kLanes);
        if (lane >= q) incl += y;
    }
    const unsigned some = (__ballot_sync(gmask, cnt > 0) & gmask) >> (threadIdx.x & 31 & ~(kLanes - 1));
    if (cnt > 0) {
        const int at = used + __popc(some & ((1u << lane) - 1u));
        off[at] = running + incl - cnt;
        from[at] = base - (running + incl - cnt);
    }
    used += __popc(some);
    running += __shfl_sync(gmask, incl, kLanes - 1, kLanes);
}

// optional count written by the last tile: min(total, cap) (overflow flags kErrCapacity)
struct ScanCount {
    int* dst = nullptr;
    int cap = 0;
    __device__ void rebase() { PSR_CLOUD(dst); }   // to cloud blockIdx.y
};

// Store functors may define `void done(unsigned total) const`: the scan calls it once, after
// the last element (or at once for an empty scan), to chain counts into the next launch.
template <class S>
__device__ __forceinline__ auto scan_done(const S& s, unsigned tot, int) -> decltype(s.done(tot), void()) {
    s.done(tot);
}
template <class S>
__device__ __forceinline__ void scan_done(const S&, unsigned, long) {}

// Load functors may define `void begin(int base) const`: every thread of the block calls it before
// the loads of the tile that starts at element `base`.
template <class L>
__device__ __forceinline__ auto scan_begin(const L& l, int base, int) -> decltype(l.begin(base), void()) {
    l.begin(base);
}
template <class L>
__device__ __forceinline__ void scan_begin(const L&, int, long) {}

// Functors over plain arrays may define all(base, v): a thread's items in 16-byte accesses (its
// items are consecutive, so one by one each access of a warp would touch 32 sectors: the 2.1M-entry
// cell table took 21.8 us).
template <class L, int K>
__device__ __forceinline__ auto scan_load_all(const L& l, int base, unsigned (&v)[K], int) -> decltype(l.all(base, v)) {
    return l.all(base, v);
}
template <class L, int K>
__device__ __forceinline__ bool scan_load_all(const L&, int, unsigned (&)[K], long) { return false; }
template <class S, int K>
__device__ __forceinline__ auto scan_store_all(const S& s, int base, unsigned pre, const unsigned (&v)[K], int)
    -> decltype(s.all(base, pre, v)) {
    return s.all(base, pre, v);
}
template <class S, int K>
__device__ __forceinline__ bool scan_store_all(const S&, int, unsigned, const unsigned (&)[K], long) { return false; }

constexpr unsigned long long kFlagAgg = 1ull << 32;
constexpr unsigned long long kFlagIncl = 1ull << 33;
constexpr int kEpochShift = 34;

__device__ __forceinline__ unsigned long long load_status(const unsigned long long* p) {
    return *((volatile const unsigned long long*)p);
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned& excl, unsigned* smem_warp) {
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned w = (lane < (kBlock / 32)) ? smem_warp[lane] : 0u;
        unsigned s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= (unsigned)o) s += y;
        }
        if (lane < (kBlock / 32)) smem_warp[lane] = s - w;   // exclusive warp offsets
        if (lane == (kBlock / 32) - 1) smem_warp[kBlock / 32] = s;
    }
    __syncthreads();
    excl = smem_warp[warp] + x - v;
    unsigned total = smem_warp[kBlock / 32];
    __syncthreads();
    return total;
}

// Generic scan.  Load(i) -> unsigned value of element i; Store(i, prefix, value) gets the
// exclusive prefix of element i.  *total receives the sum of all n elements.  kItems
// elements per thread: 8 for light functors, 1 or 2 where Load / Store do enough work per
// element that more, smaller tiles (more blocks in flight) pay.
template <int kItems, class Load, class Store>
__device__ __forceinline__ void scan_body(Load load, Store store, int n, ScanScratch sc, unsigned* total, unsigned* err,
                                          ScanCount cnt) {
    constexpr int kTile = kBlock * kItems;
    __shared__ unsigned s_warp[kBlock / 32 + 1];
    __shared__ int s_tile;
    __shared__ unsigned s_prefix;
    const int ntiles = (n + kTile - 1) / kTile;
    if (n <= 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            *total = 0u;
            if (cnt.dst) *cnt.dst = 0;
            scan_done(store, 0u, 0);
        }
        return;
    }
    if (ntiles > sc.max_tiles) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, kErrCapacity);
        return;
    }
    unsigned long long* st = sc.words + kScanHeader;
    const unsigned long long epoch = load_status(sc.words + 2);
    const unsigned long long etag = epoch << kEpochShift;
    while (true) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(sc.words, 1ull);
        __syncthreads();
        const int t = s_tile;
        __syncthreads();
        if (t >= ntiles) break;
        scan_begin(load, t * kTile, 0);
        const int base = t * kTile + threadIdx.x * kItems;
        unsigned v[kItems];
        unsigned sum = 0;
        if (base + kItems <= n && scan_load_all(load, base, v, 0)) {
#pragma unroll
            for (int k = 0; k < kItems; ++k) sum += v[k];
        } else {
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                int i = base + k;
                v[k] = (i < n) ? load(i) : 0u;
                sum += v[k];
            }
        }
        unsigned excl;
        const unsigned agg = block_exclusive_scan(sum, excl, s_warp);
        // look-back by warp 0
        if (threadIdx.x < 32) {
            const unsigned lane = lane_id();
            if (t == 0) {
                if (lane == 0) {
                    atomicExch(st, etag | kFlagIncl | (unsigned long long)agg);
                    s_prefix = 0u;
                }
            } else {
                if (lane == 0) atomicExch(st + t, etag | kFlagAgg | (unsigned long long)agg);
                unsigned run = 0;
                int pred = t - 1;
                bool timeout = false;
                while (true) {
                    int idx = pred - (int)lane;
                    unsigned long long s = kFlagIncl;   // "prefix 0" past the first tile
                    if (idx >= 0) {
                        int it = 0;
                        s = load_status(st + idx);
                        while ((s >> kEpochShift) != epoch || !(s & (kFlagAgg | kFlagIncl))) {
                            if (++it > kSpinLimit) { timeout = true; s = kFlagIncl; break; }
                            __nanosleep(20);
                            s = load_status(st + idx);
                        }
                    }
                    unsigned incl_mask = __ballot_sync(0xffffffffu, (s & kFlagIncl) != 0);
                    unsigned val = (unsigned)(s & 0xffffffffull);
                    if (incl_mask) {
                        int first = __ffs(incl_mask) - 1;
                        unsigned contrib = ((int)lane <= first) ? val : 0u;
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xffffffffu, contrib, o);
                        run += contrib;
                        break;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
                    run += val;
                    pred -= 32;
                }
                if (__any_sync(0xffffffffu, timeout) && lane == 0) atomicOr(err, kErrSpinTimeout);
                if (lane == 0) {
                    atomicExch(st + t, etag | kFlagIncl | (unsigned long long)(run + agg));
                    s_prefix = run;
                }
            }
        }
        __syncthreads();
        unsigned pre = s_prefix + excl;
        if (!(base + kItems <= n && scan_store_all(store, base, pre, v, 0))) {
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                int i = base + k;
                if (i < n) store(i, pre, v[k]);
                pre += v[k];
            }
        }
        if (t == ntiles - 1 && threadIdx.x == kBlock - 1) {
            const unsigned tot = s_prefix + agg;
            *total = tot;
            if (cnt.dst) {
                int c = (int)tot;
                if (tot > (unsigned)cnt.cap) { atomicOr(err, kErrCapacity); c = cnt.cap; }
                *cnt.dst = c;
            }
            scan_done(store, tot, 0);
        }
        __syncthreads();
    }
    // every block ends here after claiming a tile past the end, i.e. after its last tile;
    // the last one to arrive resets the counters for the next launch
    if (threadIdx.x == 0) {
        const unsigned long long done = atomicAdd(sc.words + 1, 1ull);
        if (done == (unsigned long long)gridDim.x - 1) {
            atomicExch(sc.words, 0ull);
            atomicExch(sc.words + 1, 0ull);
            atomicExch(sc.words + 2, (epoch + 1) & ((1ull << (64 - kEpochShift)) - 1));
        }
    }
}

// blocks per SM the registers of a scan must leave room for (heavy functors define kMinBlocks)
template <class L>
constexpr auto scan_min_blocks(int) -> decltype(L::kMinBlocks) { return L::kMinBlocks; }
template <class L>
constexpr int scan_min_blocks(long) { return 1; }

template <int kItems, class Load, class Store>
__global__ void __launch_bounds__(kBlock, scan_min_blocks<Load>(0)) k_scan(Load load, Store store, const int* count_ptr, int count_add,
                                                 ScanScratch sc, unsigned* total, unsigned* err, ScanCount cnt) {
    PSR_CLOUD(load, store, count_ptr, sc, total, err, cnt);
    scan_body<kItems>(load, store, *count_ptr + count_add, sc, total, err, cnt);
}

// One scan of a launch of several: scans that only read what earlier launches wrote run side by
// side, blockIdx.z taking one each, with a scratch of its own.
template <int kItems, class Load, class Store>
struct ScanJob {
    Load load;
    Store store;
    const int* count_ptr;
    ScanScratch sc;
    unsigned* total;
    ScanCount cnt;
    static constexpr bool kUsed = true;
    __device__ void run(unsigned* err) {
        PSR_CLOUD(load, store, count_ptr, sc, total, cnt);
        scan_body<kItems>(load, store, *count_ptr, sc, total, err, cnt);
    }
};
struct NoScan {
    static constexpr bool kUsed = false;
    __device__ void run(unsigned*) {}
};
template <int kItems, class Load, class Store>
ScanJob<kItems, Load, Store> scan_job(Load load, Store store, const int* count_ptr, ScanScratch sc, unsigned* total,
                                      ScanCount cnt = ScanCount{}) {
    return ScanJob<kItems, Load, Store>{load, store, count_ptr, sc, total, cnt};
}
template <class A, class B, class C, class D>
__global__ void __launch_bounds__(kBlock) k_scans(A a, B b, C c, D d, unsigned* err) {
    PSR_CLOUD(err);
    if (blockIdx.z == 0) a.run(err);
    else if (blockIdx.z == 1) b.run(err);
    else if (blockIdx.z == 2) c.run(err);
    else d.run(err);
}

// blocks of a scan launch: blocks_per_sm per SM, at most max_tiles
int scan_grid(int max_tiles, int blocks_per_sm = 4);

// blocks_per_sm: 4 for scans that can be long (hundreds of tiles or more); small scans
// (per octree level, per point at a few hundred tiles) take 1 so that idle blocks do not
// occupy the GPU while other reconstructions run beside them
template <int kItems = kScanItems, class Load, class Store>
inline cudaError_t launch_scan(Load load, Store store, const int* count_ptr, int count_add, ScanScratch sc,
                               unsigned* total, unsigned* err, cudaStream_t stream, ScanCount cnt = ScanCount{},
                               int blocks_per_sm = 4) {
    const dim3 grid(cloud_blocks(sc.batch, scan_grid(sc.max_tiles, blocks_per_sm)), sc.batch);
    k_scan<kItems, Load, Store><<<grid, kBlock, 0, stream>>>(load, store, count_ptr, count_add, sc, total, err, cnt);
    return cudaGetLastError();
}

template <class A, class B, class C = NoScan, class D = NoScan>
inline cudaError_t launch_scans(A a, B b, C c, D d, unsigned* err, cudaStream_t stream, int blocks_per_sm = 4) {
    const int jobs = 2 + (C::kUsed ? 1 : 0) + (D::kUsed ? 1 : 0);
    const dim3 grid(cloud_blocks(a.sc.batch, scan_grid(a.sc.max_tiles, blocks_per_sm)), a.sc.batch, jobs);
    k_scans<A, B, C, D><<<grid, kBlock, 0, stream>>>(a, b, c, d, err);
    return cudaGetLastError();
}

// ---- common load / store functors ----------------------------------------------------
// the array starts on a 16-byte boundary (a workspace buffer)
struct LoadArray {
    const unsigned* a;
    __device__ unsigned operator()(int i) const { return a[i]; }
    __device__ bool all(int base, unsigned (&v)[8]) const {
        const uint4 p = *reinterpret_cast<const uint4*>(a + base), q = *reinterpret_cast<const uint4*>(a + base + 4);
        v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
        v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
        return true;
    }
    __device__ void rebase() { PSR_CLOUD(a); }   // to cloud blockIdx.y
};
struct StoreExclusive {
    unsigned* out;
    __device__ void operator()(int i, unsigned pre, unsigned) const { out[i] = pre; }
    __device__ bool all(int base, unsigned pre, const unsigned (&v)[8]) const {
        unsigned p[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) { p[k] = pre; pre += v[k]; }
        *reinterpret_cast<uint4*>(out + base) = make_uint4(p[0], p[1], p[2], p[3]);
        *reinterpret_cast<uint4*>(out + base + 4) = make_uint4(p[4], p[5], p[6], p[7]);
        return true;
    }
    __device__ void rebase() { PSR_CLOUD(out); }   // to cloud blockIdx.y
};

// ---- radix sort ------------------------------------------------------------------------
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kSortItems = 8;
constexpr int kSortTile = kBlock * kSortItems;   // 2048 keys per tile

constexpr int kSortMaxPasses = 4;

// Scratch of the radix sort.  bins: [kSortMaxPasses][kRadix] digit counts of the whole input, then
// their exclusive prefixes; [kSortMaxPasses * kRadix + p]: the next tile of pass p.  The caller's
// first kernel zeroes it (kSortBinWords words).  status: [pass][tile][digit] words of the passes'
// look-back, cleared by the kernel that counts the digits.
struct SortScratch {
    unsigned* bins;
    unsigned* status;
    unsigned* keys_alt;
    unsigned* vals_alt;
    int max_tiles;
    int batch = 1;   // clouds of the launch (host side: the grid's y extent)
    __device__ void rebase() { PSR_CLOUD(bins, status, keys_alt, vals_alt); }   // to cloud blockIdx.y
};
constexpr int kSortBinWords = kSortMaxPasses * (kRadix + 1);
inline int sort_passes(int key_bits) { return (key_bits + kRadixBits - 1) / kRadixBits; }

// n 32-bit words at p set to v, in each of `clouds` clouds (a memset that multi-cloud
// launches can take: every cloud's copy of the buffer)
cudaError_t fill_words(unsigned* p, unsigned v, long long n, int clouds, cudaStream_t stream);

// Counting side of the sort, inside the kernel that makes the keys (kBlock threads a block):
// count() the digits of every key of the block, then finish() in every block of the cloud.
struct SortCounter {
    unsigned (*s_h)[kRadix];   // [kSortMaxPasses][kRadix] shared
    int passes;
    __device__ void clear() const {
        for (int d = threadIdx.x; d < passes * kRadix; d += kBlock) (&s_h[0][0])[d] = 0u;
        __syncthreads();
    }
    __device__ void count(unsigned key) const {
        for (int p = 0; p < passes; ++p) atomicAdd(&s_h[p][(key >> (kRadixBits * p)) & (kRadix - 1)], 1u);
    }
    // adds the block's counts to the bins; the last block to finish turns them into exclusive
    // prefixes.  Also clears the passes' look-back words of n keys.
    __device__ void finish(const SortScratch& sc, int n, unsigned* ticket, unsigned* err) const {
        const int ntiles = (n + kSortTile - 1) / kSortTile;
        if (ntiles > sc.max_tiles) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, kErrCapacity);
            return;
        }
        for (int p = 0; p < passes; ++p) {
            unsigned* st = sc.status + (size_t)p * sc.max_tiles * kRadix;
            PSR_GRID_STRIDE(i, ntiles * kRadix) st[i] = 0u;
        }
        __syncthreads();
        for (int d = threadIdx.x; d < passes * kRadix; d += kBlock) {
            const unsigned v = (&s_h[0][0])[d];
            if (v) atomicAdd(&sc.bins[d], v);
        }
        __shared__ unsigned s_warp[kBlock / 32 + 1];
        __shared__ int s_last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        static_assert(kRadix == kBlock, "a thread per digit");
        for (int p = 0; p < passes; ++p) {
            unsigned* b = sc.bins + p * kRadix;
            unsigned excl;
            block_exclusive_scan(__ldcg(b + threadIdx.x), excl, s_warp);
            b[threadIdx.x] = excl;
        }
    }
};

// The passes: a stable sort of the n = *count_ptr (key, index) pairs whose digits were counted;
// vals_in of the first pass is the input index.  *result_in_alt: where they end.
cudaError_t radix_sort_pairs(unsigned* keys, unsigned* vals, const int* count_ptr, int key_bits, SortScratch sc,
                             unsigned* err, cudaStream_t stream, bool* result_in_alt);

}  // namespace psr
