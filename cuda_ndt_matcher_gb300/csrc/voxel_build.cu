// voxel_build.cu — GPU voxel-map build for sm_103a (the `set_target` hot path).
//
// Pipeline (one CUDA stream, no host work between kernels except the size reads that pick
// the key width and size the allocations):
//   1. cells + bounds      : cell = floor(p / res) per finite point (f32 IEEE division, the
//                            membership rule of VoxelCoord::from_point,
//                            src/ndt_cuda/src/voxel_grid/types.rs:206-212); min/max cell.
//   2. Morton keys         : the order of morton(cell - min cell), 21 bits per axis
//                            (src/ndt_cuda/src/voxel_grid/gpu/morton.rs:45-95), as a 32-bit key of
//                            the bits that the map's box has; non-finite points sort last.
//   3. LSD radix sort      : stable, digits of up to 8 bits, the key's bits shared evenly by
//                            the passes (replaces cub::DeviceRadixSort,
//                            src/cuda_ffi/csrc/radix_sort.cu); 64-bit keys from 2^30 points on.
//   4. segments            : starts of the runs of equal keys, one launch with look-back
//                            (src/cuda_ffi/csrc/segment_detect.cu:27-146; the API's
//                            ndt_detect_segments keeps flags + scan for the segment ids).
//   5. voxel statistics    : segments visited largest first; segments of 48 points or more
//                            summed by a warp each (k_segment_sums), the rest by a thread
//                            each, every voxel finished by a thread (k_voxel_stats); exact
//                            integer moments of the segment's points (the FP64
//                            running sum's mean bit for bit, the centred covariance from an
//                            exact numerator), FP64 two-pass moments where the exact bounds
//                            do not hold; eigenvector directions by an f32 Jacobi, refined
//                            in FP64; regularisation to the min-ratio and inverse in FP64,
//                            f32 outputs (Voxel::from_statistics / regularize_covariance,
//                            src/ndt_cuda/src/voxel_grid/types.rs:54-190).
//   6. compaction          : valid voxels keep their Morton order; their search records; the
//                            dense cell index when it fits, {centroid, voxel} per cell of the
//                            map's box; and hash insert: bounded linear probing with
//                            atomicCAS, displacement recorded (voxel_hash_build_kernel,
//                            src/cuda_ffi/csrc/voxel_hash.cu:69-114).
//   7. masks               : with the dense index, the neighbourhood masks (one per octant of
//                            each cell while they fit their budget, else one per cell) that
//                            list the neighbours a point there can accept.
// Bit-exact parts (cells, keys, counts, means) do not depend on FMA contraction: cells are an
// f32 quotient, means the correctly rounded FP64 quotient of an exact sum (or a running sum of
// adds); the regularised covariances, compared in f32 ULPs, use FMAs freely.
#include <algorithm>
#include <cstdio>
#include <mutex>

#include <cuda.h>

#include "ndt_internal.h"

namespace ndtgb {

constexpr int BT = 256;        // threads per block for tile kernels
constexpr int ITEMS = 16;      // items per thread
constexpr int TILE = BT * ITEMS;

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
static inline uint32_t ntiles(size_t n) { return (uint32_t)((n + TILE - 1) / TILE); }

// ---------------------------------------------------------------------------------------
// Block-wide exclusive scan of one value per thread (256 threads).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* ws,
                                                         uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (BT / 32) ? ws[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < BT / 32) ws[lane] = w;
    }
    __syncthreads();
    uint32_t pre = warp ? ws[warp - 1] : 0u;
    *total = ws[BT / 32 - 1];
    __syncthreads();
    return pre + x - v;
}

// ---------------------------------------------------------------------------------------
// Exclusive scan in three launches, none of which waits for another block: the form of the
// standalone entry points, which return before their kernels end and so could not report a wait
// that ran out, and of the 64-bit sort.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(BT) k_tile_reduce(const uint32_t* __restrict__ in, size_t n,
                                                    uint32_t* __restrict__ bsum) {
    __shared__ uint32_t ws[BT / 32];
    size_t base = (size_t)blockIdx.x * TILE;
    uint32_t s = 0;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        size_t i = base + (size_t)r * BT + threadIdx.x;
        if (i < n) s += in[i];
    }
    uint32_t tot;
    block_exclusive_scan(s, ws, &tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(BT) k_scan_bsums(uint32_t* __restrict__ bsum, uint32_t nb) {
    __shared__ uint32_t ws[BT / 32];
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nb; base += TILE) {
        uint32_t v[ITEMS];
        uint32_t s = 0;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            uint32_t i = base + threadIdx.x * ITEMS + k;
            v[k] = i < nb ? bsum[i] : 0u;
            s += v[k];
        }
        uint32_t tot;
        uint32_t run = carry + block_exclusive_scan(s, ws, &tot);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            uint32_t i = base + threadIdx.x * ITEMS + k;
            if (i < nb) bsum[i] = run;
            run += v[k];
        }
        carry += tot;
        __syncthreads();
    }
}

// exclusive scan of a tile; element order: thread t holds items t*ITEMS .. t*ITEMS+15
__global__ void __launch_bounds__(BT) k_tile_scan(const uint32_t* __restrict__ in,
                                                  uint32_t* __restrict__ out, size_t n,
                                                  const uint32_t* __restrict__ bsum) {
    __shared__ uint32_t ws[BT / 32];
    size_t base = (size_t)blockIdx.x * TILE + (size_t)threadIdx.x * ITEMS;
    uint32_t v[ITEMS];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0u;
        s += v[k];
    }
    uint32_t tot;
    uint32_t run = bsum[blockIdx.x] + block_exclusive_scan(s, ws, &tot);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
}

static size_t scan_temp_bytes(size_t n) { return align_up((size_t)ntiles(n) * 4 + 4, 256); }

// exclusive scan in -> out (may alias); temp >= scan_temp_bytes(n), 4-byte aligned
static int exclusive_scan(const uint32_t* in, uint32_t* out, size_t n, void* temp,
                          cudaStream_t s) {
    if (n == 0) return 0;
    uint32_t nb = ntiles(n);
    uint32_t* bsum = (uint32_t*)temp;
    k_tile_reduce<<<nb, BT, 0, s>>>(in, n, bsum);
    k_scan_bsums<<<1, BT, 0, s>>>(bsum, nb);
    k_tile_scan<<<nb, BT, 0, s>>>(in, out, n, bsum);
    return cuda_fail(cudaGetLastError(), "scan launch");
}

// ---------------------------------------------------------------------------------------
// Decoupled look-back (Merrill and Garland 2016): the tiles of a launch take their numbers from
// a ticket, so every earlier tile is running or done; each publishes its own sum, then walks
// back over the earlier tiles' words until it meets an inclusive prefix. A word holds state
// (top two bits: 0 not there yet, 1 the tile's sum, 2 the inclusive prefix) and value, so it
// is read and written whole and needs no fence.
// ---------------------------------------------------------------------------------------
// Where a launch's words are (one ticket, then a word per tile, all zero at the start), how
// long a wait may last, and (test hook) whether tile 0 withholds its word, so that the waits of
// the others run out. A wait that runs out sets *failed, a word of the whole build: the kernels
// behind it that would index memory with what the scan was to write leave at once, and the host
// reads it with the sizes, before it uses them.
struct LookBack {
    unsigned long long* words;
    uint32_t* failed;
    unsigned long long limit_ns;
    bool withhold;
};
// The look-back launch `stage` of a build (BuildScratch::lb_withhold)
enum { LB_SORT = 1, LB_SEGMENTS = 2, LB_SIZES = 3, LB_RANKS = 4 };
static LookBack look_back(const BuildScratch& sc, void* words, uint32_t* failed, int stage) {
    return {(unsigned long long*)words, failed, sc.lb_limit_ns, sc.lb_withhold == stage};
}
static int look_back_failed() {
    set_error("map build: a look-back wait ran out");
    return NDT_ERR_DEVICE;
}

__device__ __forceinline__ unsigned long long lb_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Exclusive prefix of tile `tile`, whose own sum is `sum`, over the earlier tiles, by one warp (32
// tiles at a time); publishes the tile's inclusive prefix. False (in every lane) when a word did
// not arrive within the limit: the warp decides together, and on words read after the time was
// taken, so a context that was paused for longer finds what has arrived meanwhile.
__device__ __forceinline__ bool lookback_warp(const LookBack& lb, uint32_t tile,
                                              unsigned long long sum, int lane,
                                              unsigned long long& excl) {
    constexpr unsigned long long ONE = 1ull << 62, TWO = 2ull << 62, VAL = ONE - 1ull;
    unsigned long long* const w = lb.words + 1;
    if (lane == 0 && !(tile == 0 && lb.withhold))
        atomicExch(w + tile, (tile == 0 ? TWO : ONE) | sum);
    excl = 0ull;
    if (tile == 0) return true;
    const unsigned long long t0 = lb_now();
    int64_t at = (int64_t)tile - 1 - lane;
    for (;;) {
        unsigned long long v = at >= 0 ? *(volatile unsigned long long*)(w + at) : TWO;
        while (__any_sync(0xffffffffu, (v >> 62) == 0ull)) {
            const int late = __any_sync(0xffffffffu, lb_now() - t0 > lb.limit_ns);
            if ((v >> 62) == 0ull) v = *(volatile unsigned long long*)(w + at);
            if (late && __any_sync(0xffffffffu, (v >> 62) == 0ull)) {
                if (lane == 0) atomicExch(lb.failed, 1u);
                return false;
            }
        }
        // the nearest inclusive prefix among these 32, and the sums after it
        const unsigned full = __ballot_sync(0xffffffffu, (v >> 62) == 2ull);
        const int stop = full ? __ffs(full) - 1 : 32;
        unsigned long long x = lane <= stop ? (v & VAL) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        excl += x;
        if (full) break;
        at -= 32;
    }
    if (lane == 0) atomicExch(w + tile, TWO | (excl + sum));
    return true;
}

// Exclusive scan in one launch, element order (thread t of a tile holds items t * ITEMS ..).
// In place allowed. total (may be null): the sum of all items.
__global__ void __launch_bounds__(BT) k_scan(const uint32_t* __restrict__ in,
                                             uint32_t* __restrict__ out, size_t n,
                                             const LookBack lb, uint32_t* __restrict__ total) {
    __shared__ uint32_t ws[BT / 32];
    __shared__ uint32_t s_tile, s_excl;
    __shared__ bool s_ok;
    if (threadIdx.x == 0) s_tile = atomicAdd((unsigned int*)lb.words, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const size_t base = (size_t)tile * TILE + (size_t)threadIdx.x * ITEMS;
    uint32_t v[ITEMS];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0u;
        s += v[k];
    }
    uint32_t tot;
    const uint32_t pre = block_exclusive_scan(s, ws, &tot);
    if (threadIdx.x < 32) {
        unsigned long long e;
        const bool ok = lookback_warp(lb, tile, tot, (int)threadIdx.x, e);
        if (threadIdx.x == 0) {
            s_excl = (uint32_t)e;
            s_ok = ok;
        }
    }
    __syncthreads();
    if (!s_ok) return;
    uint32_t run = s_excl + pre;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (total && tile == gridDim.x - 1 && threadIdx.x == 0) *total = s_excl + tot;
}

static size_t lookback_bytes(size_t n) { return align_up((size_t)ntiles(n) * 8 + 8, 256); }

// exclusive scan in -> out (may alias); lb.words: lookback_bytes(n), 8-byte aligned, all zero
static int exclusive_scan_zeroed(const uint32_t* in, uint32_t* out, size_t n, const LookBack& lb,
                                 cudaStream_t s, uint32_t* total = nullptr) {
    if (n == 0) return 0;
    k_scan<<<ntiles(n), BT, 0, s>>>(in, out, n, lb, total);
    return cuda_fail(cudaGetLastError(), "scan launch");
}

// ---------------------------------------------------------------------------------------
// Stable LSD radix sort of (u64 key, u32 value) pairs, 8-bit digits: the standalone form, and the
// build's from 2^30 points on.
// ---------------------------------------------------------------------------------------
// Digit counts of each TILE-key tile: shared-memory atomics into one counter set per warp
// (keys of one digit then queue only within their warp), summed per digit at the end.
__global__ void __launch_bounds__(BT) k_radix_hist(const uint64_t* __restrict__ keys, size_t n,
                                                   int shift, uint32_t dmask,
                                                   uint32_t* __restrict__ hist, uint32_t nb) {
    __shared__ uint32_t h[BT / 32][256];
#pragma unroll
    for (int w = 0; w < BT / 32; ++w) h[w][threadIdx.x] = 0;
    __syncthreads();
    uint32_t* const hw = h[threadIdx.x >> 5];
    const size_t base = (size_t)blockIdx.x * TILE;
    uint64_t kv[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const size_t i = base + (size_t)r * BT + threadIdx.x;
        kv[r] = i < n ? keys[i] : 0ull;
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        if (base + (size_t)r * BT + threadIdx.x < n)
            atomicAdd(&hw[(uint32_t)(kv[r] >> shift) & dmask], 1u);
    __syncthreads();
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < BT / 32; ++w) c += h[w][threadIdx.x];
    hist[(size_t)threadIdx.x * nb + blockIdx.x] = c;
}

// Lanes of the warp whose 9-bit value d (an 8-bit digit, or 0x100 for no key) equals this
// lane's: one ballot per bit, each narrowing the set to the lanes that agree on that bit.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d) {
    uint32_t m = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const bool bit = (d >> k) & 1u;
        const uint32_t b = __ballot_sync(0xffffffffu, bit);
        m &= bit ? b : ~b;
    }
    return m;
}

// One block per TILE-key tile. Warp w owns the tile's keys [w * 512, (w + 1) * 512), held in
// registers as 16 rounds of 32. Pass 1: each warp counts its digits into its own counters
// (same-digit lanes found by digit_peers). Then per digit: the tile-local start (block
// scan) plus the counts of the earlier warps give each warp's first position. Pass 2: each
// key goes to shared memory at its warp's running position of its digit plus its rank among
// the round's same-digit lanes: tile order within each digit, so the sort is stable. Last, the
// keys leave in that order: the keys of one digit as one contiguous run at base[digit] (the
// scanned histogram), so the stores coalesce.
__global__ void __launch_bounds__(BT, 3) k_radix_scatter(
    const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin,
    uint64_t* __restrict__ kout, uint32_t* __restrict__ vout, size_t n, int shift, uint32_t dmask,
    const uint32_t* __restrict__ offs, uint32_t nb) {
    constexpr int NWARP = BT / 32;
    constexpr int WROUNDS = TILE / BT;  // rounds of 32 keys per warp
    extern __shared__ __align__(16) unsigned char sc_smem[];
    uint64_t* skey = reinterpret_cast<uint64_t*>(sc_smem);
    uint32_t* sval = reinterpret_cast<uint32_t*>(sc_smem + TILE * sizeof(uint64_t));
    __shared__ uint32_t wpos[NWARP][256];  // per warp: digit counts, then running positions
    __shared__ uint32_t base[256];         // global position of the tile's first key of each digit
    __shared__ uint32_t loff[256];         // tile-local position of the first key of each digit
    __shared__ uint32_t ws[NWARP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t tbase = (size_t)blockIdx.x * TILE;
    const uint32_t tn = (uint32_t)min((size_t)TILE, n - tbase);
    const uint32_t wbase = (uint32_t)warp * (WROUNDS * 32);
#pragma unroll
    for (int w = 0; w < NWARP; ++w) wpos[w][threadIdx.x] = 0;
    __syncthreads();
    uint64_t key[WROUNDS];
#pragma unroll
    for (int r = 0; r < WROUNDS; ++r) {
        const uint32_t li = wbase + (uint32_t)r * 32 + lane;
        key[r] = li < tn ? kin[tbase + li] : 0ull;
    }
#pragma unroll
    for (int r = 0; r < WROUNDS; ++r) {
        const uint32_t li = wbase + (uint32_t)r * 32 + lane;
        const uint32_t d = li < tn ? ((uint32_t)(key[r] >> shift) & dmask) : 0x100u;
        const uint32_t peers = digit_peers(d);
        if (d != 0x100u && lane == __ffs(peers) - 1) wpos[warp][d] += (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        const uint32_t d = threadIdx.x;  // one thread per digit (BT == 256)
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < NWARP; ++w) {
            const uint32_t c = wpos[w][d];
            wpos[w][d] = run;
            run += c;
        }
        uint32_t tot;
        const uint32_t lo = block_exclusive_scan(run, ws, &tot);
        loff[d] = lo;
#pragma unroll
        for (int w = 0; w < NWARP; ++w) wpos[w][d] += lo;
        base[d] = offs[(size_t)d * nb + blockIdx.x];
    }
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < WROUNDS; ++r) {
        const uint32_t li = wbase + (uint32_t)r * 32 + lane;
        const bool valid = li < tn;
        const uint32_t d = valid ? ((uint32_t)(key[r] >> shift) & dmask) : 0x100u;
        const uint32_t peers = digit_peers(d);
        if (valid) {
            const uint32_t pos = wpos[warp][d] + (uint32_t)__popc(peers & lt);
            skey[pos] = key[r];
            sval[pos] = vin[tbase + li];
        }
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wpos[warp][d] += (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < tn; i += BT) {
        const uint64_t k = skey[i];
        const uint32_t d = (uint32_t)(k >> shift) & dmask;
        const uint32_t pos = base[d] + (i - loff[d]);
        kout[pos] = k;
        vout[pos] = sval[i];
    }
}

size_t radix_sort_temp_bytes(size_t n) {
    size_t nb = ntiles(n);
    return align_up(n * 8, 256) + align_up(n * 4, 256) + align_up(256 * nb * 4, 256) +
           scan_temp_bytes(256 * nb);
}

int radix_sort_pairs(uint64_t* keys, uint32_t* vals, size_t n, int begin_bit, int end_bit,
                     void* temp, size_t temp_bytes, cudaStream_t s) {
    if (n <= 1 || end_bit <= begin_bit) return 0;
    if (temp_bytes < radix_sort_temp_bytes(n)) {
        set_error("radix sort: temporary storage too small");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    uint32_t nb = ntiles(n);
    char* t = (char*)temp;
    uint64_t* kalt = (uint64_t*)t;
    t += align_up(n * sizeof(uint64_t), 256);
    uint32_t* valt = (uint32_t*)t;
    t += align_up(n * 4, 256);
    uint32_t* hist = (uint32_t*)t;
    t += align_up(256 * (size_t)nb * 4, 256);
    void* stemp = t;
    uint64_t* kin = keys;
    uint32_t* vin = vals;
    uint64_t* kout = kalt;
    uint32_t* vout = valt;
    int passes = 0;
    // the scatter's tile staging may exceed the default dynamic shared-memory limit (set on
    // the current device at every call: a host-side attribute, no allocation)
    constexpr int smem = TILE * (int)(sizeof(uint64_t) + 4);
    cudaFuncSetAttribute(k_radix_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    for (int shift = begin_bit; shift < end_bit; shift += 8, ++passes) {
        int width = std::min(8, end_bit - shift);
        uint32_t dmask = (1u << width) - 1u;
        k_radix_hist<<<nb, BT, 0, s>>>(kin, n, shift, dmask, hist, nb);
        int rc = exclusive_scan(hist, hist, 256 * (size_t)nb, stemp, s);
        if (rc) return rc;
        k_radix_scatter<<<nb, BT, smem, s>>>(kin, vin, kout, vout, n, shift, dmask, hist, nb);
        int e = cuda_fail(cudaGetLastError(), "radix scatter launch");
        if (e) return e;
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    if (passes & 1) {
        cudaMemcpyAsync(keys, kin, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(vals, vin, n * 4, cudaMemcpyDeviceToDevice, s);
    }
    return cuda_fail(cudaGetLastError(), "radix sort");
}

// ---------------------------------------------------------------------------------------
// Stable LSD sort of (u32 key, u32 value) pairs with digits of up to 8 bits, the map build's
// form. Against the form above: the key's bits shared evenly by the passes (fewer digits make
// longer runs), the first pass's tile counts taken while the keys are made, and one search for
// each key's peers instead of two (that form was bound by the instructions of its ballots: 58%
// issue, math pipe throttled). 50M pairs: 277 us a pass, 225 this way. Slower: 9-bit digits (460
// us a pass: a tile's runs are 32 bytes), and a one-sweep form with look-back over the earlier
// tiles instead of scanned counts (545 us: 600 tiles in flight walk over one another's sums).
// ---------------------------------------------------------------------------------------
constexpr int SP_BINS = 256;
constexpr size_t SP_MAX_PAIRS = size_t(1) << 30;

// Passes over `bits` key bits and the digit width of each
struct SortPlan {
    int passes, width;
};
static SortPlan sort_plan(int bits) {
    SortPlan o;
    o.passes = std::max(1, (bits + 7) / 8);
    o.width = std::max(1, (bits + o.passes - 1) / o.passes);
    return o;
}
// Workspace of a sort: tile counts [bins][tiles]; and look-back words of its scans, a set per
// pass, zero at the start. A build clears the look-back words of all its launches at once: a
// memset before each cost a 126k-point tile 21 us of 0.7 ms.
static size_t sort_counts(size_t n, SortPlan o) { return (size_t)ntiles(n) << o.width; }
static size_t sort_bytes(size_t n, SortPlan o) { return align_up(sort_counts(n, o) * 4, 256); }
static size_t sort_words_bytes(size_t n, SortPlan o) {
    return (size_t)o.passes * lookback_bytes(sort_counts(n, o));
}

// Digit counts of a tile: shared-memory atomics into one counter set per warp, so keys of one
// digit queue only within their warp
struct TileCounts {
    uint32_t c[BT / 32][SP_BINS];
};
__device__ __forceinline__ void tile_counts_clear(TileCounts& t, uint32_t bins) {
    for (uint32_t i = threadIdx.x; i < (BT / 32) * SP_BINS; i += BT)
        if (i % SP_BINS < bins) t.c[i / SP_BINS][i % SP_BINS] = 0;
}
__device__ __forceinline__ void tile_counts_add(TileCounts& t, uint32_t d, bool valid) {
    if (valid) atomicAdd(&t.c[threadIdx.x >> 5][d], 1u);
}
__device__ __forceinline__ void tile_counts_store(const TileCounts& t, uint32_t bins,
                                                  uint32_t* __restrict__ hist, uint32_t tile,
                                                  uint32_t nb) {
    for (uint32_t d = threadIdx.x; d < bins; d += BT) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < BT / 32; ++w) c += t.c[w][d];
        hist[(size_t)d * nb + tile] = c;
    }
}

__global__ void __launch_bounds__(BT) k_tile_digits(const uint32_t* __restrict__ keys, uint32_t n,
                                                    int shift, int width,
                                                    uint32_t* __restrict__ hist) {
    __shared__ TileCounts t;
    const uint32_t bins = 1u << width;
    tile_counts_clear(t, bins);
    const uint32_t base = blockIdx.x * (uint32_t)TILE;
    uint32_t kv[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t i = base + (uint32_t)r * BT + threadIdx.x;
        kv[r] = i < n ? keys[i] : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r)
        tile_counts_add(t, (kv[r] >> shift) & (bins - 1u),
                        base + (uint32_t)r * BT + threadIdx.x < n);
    __syncthreads();
    tile_counts_store(t, bins, hist, blockIdx.x, gridDim.x);
}

// One pass. A block takes one TILE-key tile; warp w holds the tile's keys [w * 512, (w + 1) *
// 512) as 16 rounds of 32. Each round finds every key's peers (same digit) by ballots, and its
// rank from the warp's counter: tile order within a digit, so the sort is stable. The digits'
// tile positions (scanned over the block) and global positions (the scanned tile counts, offs)
// then give each key's place; the tile leaves through shared memory as one contiguous run per
// digit. vin null: the values are the positions. Nothing moves when the scan of offs failed.
__global__ void __launch_bounds__(BT, 4) k_sort_pass(
    const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
    uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n, int shift, int width,
    const uint32_t* __restrict__ offs, const uint32_t* __restrict__ failed) {
    if (*failed) return;
    constexpr int NWARP = BT / 32, ROUNDS = TILE / BT, PER = SP_BINS / BT;
    __shared__ TileCounts wc;          // per warp: digit counts, then first positions
    __shared__ uint32_t base[SP_BINS]; // global position minus tile position of a digit
    __shared__ uint32_t skey[TILE], sval[TILE];  // the tile on its way out
    __shared__ uint32_t ws[NWARP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t bins = 1u << width, dmask = bins - 1u;
    const uint32_t tbase = blockIdx.x * (uint32_t)TILE;
    const uint32_t tn = min((uint32_t)TILE, n - tbase);
    const uint32_t wbase = (uint32_t)warp * (ROUNDS * 32);
    uint32_t key[ROUNDS];
    uint32_t rank[ROUNDS / 2];  // two 16-bit ranks a word
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const uint32_t li = wbase + (uint32_t)r * 32 + lane;
        key[r] = li < tn ? kin[tbase + li] : 0u;
    }
    tile_counts_clear(wc, bins);
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t* const wcnt = wc.c[warp];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const uint32_t li = wbase + (uint32_t)r * 32 + lane;
        const bool valid = li < tn;
        const uint32_t d = (key[r] >> shift) & dmask;
        uint32_t peers = tn == (uint32_t)TILE ? 0xffffffffu : __ballot_sync(0xffffffffu, valid);
        for (int k = 0; k < width; ++k) {
            const bool bit = (d >> k) & 1u;
            const uint32_t b = __ballot_sync(0xffffffffu, bit);
            peers &= bit ? b : ~b;
        }
        uint32_t rk = 0;
        if (valid) rk = wcnt[d];
        __syncwarp();
        if (valid && (peers & lt) == 0u) wcnt[d] = rk + (uint32_t)__popc(peers);
        __syncwarp();
        rk += (uint32_t)__popc(peers & lt);
        if (r & 1)
            rank[r / 2] |= rk << 16;
        else
            rank[r / 2] = rk;
    }
    __syncthreads();
    // thread t owns the digits t * PER .. (only the first `bins` exist)
    uint32_t cnt[PER], tot, mine = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t d = threadIdx.x * PER + j;
        uint32_t run = 0;
        if (d < bins) {
#pragma unroll
            for (int w = 0; w < NWARP; ++w) {
                const uint32_t c = wc.c[w][d];
                wc.c[w][d] = run;
                run += c;
            }
            base[d] = offs[(size_t)d * gridDim.x + blockIdx.x];
        }
        cnt[j] = run;
        mine += run;
    }
    uint32_t lo = block_exclusive_scan(mine, ws, &tot);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const uint32_t d = threadIdx.x * PER + j;
        if (d < bins) {
#pragma unroll
            for (int w = 0; w < NWARP; ++w) wc.c[w][d] += lo;
            base[d] -= lo;
        }
        lo += cnt[j];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const uint32_t li = wbase + (uint32_t)r * 32 + lane;
        if (li < tn) {
            const uint32_t rk = (rank[r / 2] >> (16 * (r & 1))) & 0xFFFFu;
            const uint32_t pos = wcnt[(key[r] >> shift) & dmask] + rk;
            skey[pos] = key[r];
            sval[pos] = vin ? vin[tbase + li] : tbase + li;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < tn; i += BT) {
        const uint32_t k = skey[i];
        const uint32_t at = base[(k >> shift) & dmask] + i;
        kout[at] = k;
        vout[at] = sval[i];
    }
}

// Sorts n pairs (keys k0, values: the positions) with the workspace `work` and zeroed look-back
// words lb.words; counted: the first pass's tile counts are in the workspace already; alternate
// buffers k1 and v1, values through v0 and v1. On return *kout and *vout
// are the buffers that hold the result: v0 after an even number of passes, else v1.
static int sort_positions(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, size_t n,
                          SortPlan o, bool counted, void* work, const LookBack& lb,
                          uint32_t** kout, uint32_t** vout, cudaStream_t s) {
    uint32_t* hist = (uint32_t*)work;
    const size_t wb = lookback_bytes(sort_counts(n, o));
    const uint32_t nb = ntiles(n);
    uint32_t *ki = k0, *vi = v0, *ko = k1, *vo = v1;
    int rc;
    for (int p = 0; p < o.passes; ++p) {
        if (p > 0 || !counted)
            k_tile_digits<<<nb, BT, 0, s>>>(ki, (uint32_t)n, p * o.width, o.width, hist);
        LookBack pass = lb;
        pass.words += p * (wb / 8);
        if ((rc = exclusive_scan_zeroed(hist, hist, sort_counts(n, o), pass, s))) return rc;
        k_sort_pass<<<nb, BT, 0, s>>>(ki, p == 0 ? nullptr : vi, ko, vo, (uint32_t)n,
                                      p * o.width, o.width, hist, lb.failed);
        std::swap(ki, ko);
        std::swap(vi, vo);
    }
    *kout = ki;
    *vout = vi;
    return cuda_fail(cudaGetLastError(), "sort");
}

// ---------------------------------------------------------------------------------------
// Allocation-free radix sort: the passes above with their scratch (alternate key/value
// buffers, digit histograms, scan block sums) in one fixed device array of this module.
// Sized for STATIC_SORT_MAX_PAIRS pairs: 8 + 4 bytes per pair + 256 counters per 4096-pair
// tile + the scan's block sums = 12,845,312 bytes. Nothing in it needs to start at zero:
// every pass writes each word of the scratch before it reads it.
// ---------------------------------------------------------------------------------------
constexpr size_t STATIC_SORT_MAX_PAIRS = size_t(1) << 20;
constexpr size_t STATIC_SORT_SCRATCH_BYTES = STATIC_SORT_MAX_PAIRS * 8 + STATIC_SORT_MAX_PAIRS * 4 +
                                             256 * (STATIC_SORT_MAX_PAIRS / TILE) * 4 + 256;
constexpr int STATIC_SORT_MAX_DEVICES = 64;

static __device__ __align__(256) unsigned char g_static_sort_scratch[STATIC_SORT_SCRATCH_BYTES];

static std::mutex g_static_sort_mu;
static void* g_static_sort_ptr[STATIC_SORT_MAX_DEVICES];
static unsigned long long g_static_sort_ctx[STATIC_SORT_MAX_DEVICES];

// Unique id of the calling thread's current CUDA context (cuCtxGetId through the runtime's
// driver entry points), 0 when it cannot be read. A device reset or a new primary context
// gives a new id, and the module (with its __device__ array) is loaded again at a new address.
static unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault,
                                             &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = (GetCurrent)p;
        p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (GetId)p;
    });
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&c) != CUDA_SUCCESS || !c) return 0;
    if (get_id(c, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Device address of the scratch array on the current device. It is resolved once per device
// and context: the first call on a device (and the first after a cudaDeviceReset, which ends
// the context the address belonged to) calls cudaGetSymbolAddress, which can load this
// module onto the device. When the context id cannot be read, the address is resolved on
// every call (a lookup, no allocation).
static int static_sort_scratch(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "static radix sort: no current device");
    if (dev < 0 || dev >= STATIC_SORT_MAX_DEVICES) {
        set_error("static radix sort: device ordinal out of range");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    // makes the device's primary context current (created if needed), so its id is readable
    e = cudaSetDevice(dev);
    if (e != cudaSuccess) return cuda_fail(e, "static radix sort: device set-up");
    const unsigned long long ctx_id = current_context_id();
    std::lock_guard<std::mutex> lock(g_static_sort_mu);
    if (!g_static_sort_ptr[dev] || ctx_id == 0 || g_static_sort_ctx[dev] != ctx_id) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_sort_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "static radix sort: scratch set-up");
        if (radix_sort_temp_bytes(STATIC_SORT_MAX_PAIRS) > STATIC_SORT_SCRATCH_BYTES) {
            set_error("static radix sort: scratch array smaller than the sort needs");
            return NDT_ERR_CAPACITY;
        }
        g_static_sort_ptr[dev] = p;
        g_static_sort_ctx[dev] = ctx_id;
    }
    *out = g_static_sort_ptr[dev];
    return NDT_OK;
}

}  // namespace ndtgb

extern "C" int ndt_radix_sort_pairs_u64_u32_static(uint64_t* d_keys, uint32_t* d_values,
                                                   uint64_t n, int32_t begin_bit,
                                                   int32_t end_bit, void* stream) {
    using namespace ndtgb;
    if (begin_bit < 0 || end_bit > 64 || begin_bit > end_bit) {
        set_error("static radix sort: bit range must satisfy 0 <= begin_bit <= end_bit <= 64");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    if (n > STATIC_SORT_MAX_PAIRS) {
        set_error("static radix sort: at most 1048576 pairs (fixed 12.25 MiB device scratch)");
        return NDT_ERR_CAPACITY;
    }
    if (n && (!d_keys || !d_values)) {
        set_error("static radix sort: null key or value pointer");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    void* scratch = nullptr;
    int rc = static_sort_scratch(&scratch);
    if (rc) return rc;
    return radix_sort_pairs(d_keys, d_values, (size_t)n, begin_bit, end_bit, scratch,
                            STATIC_SORT_SCRATCH_BYTES, (cudaStream_t)stream);
}

namespace ndtgb {

// ---------------------------------------------------------------------------------------
// Segments of sorted keys.
// ---------------------------------------------------------------------------------------
__global__ void k_seg_flags(const uint64_t* __restrict__ keys, size_t n,
                            uint32_t* __restrict__ flags) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flags[i] = (i > 0 && keys[i] != keys[i - 1]) ? 1u : 0u;
}

__global__ void k_seg_finish(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ ex,
                             size_t n, uint32_t* __restrict__ seg_ids,
                             uint32_t* __restrict__ starts, uint32_t* __restrict__ num) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t f = flags[i];
    uint32_t sid = ex[i] + f;
    if (seg_ids) seg_ids[i] = sid;
    if (i == 0 || f) starts[sid] = (uint32_t)i;
    if (i == n - 1) *num = sid + 1;
}

size_t detect_segments_temp_bytes(size_t n) {
    return 2 * align_up(n * 4 + 4, 256) + scan_temp_bytes(n);
}

// Segment starts without per-key flags (the map build's form, no segment ids), in one launch:
// a block counts its tile's segment starts (key != previous key), finds the earlier tiles'
// count by look-back and writes its starts there, in key order.
template <typename K>
__global__ void __launch_bounds__(BT) k_seg_starts(const K* __restrict__ keys, size_t n,
                                                   const LookBack lb,
                                                   uint32_t* __restrict__ starts,
                                                   uint32_t* __restrict__ num) {
    __shared__ uint32_t ws[BT / 32];
    __shared__ uint32_t s_tile, s_excl;
    __shared__ bool s_ok;
    constexpr int ROUNDS = TILE / BT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd((unsigned int*)lb.words, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    // warp w holds the tile's keys [w * 512, (w + 1) * 512) as 16 rounds of 32
    const size_t wbase = (size_t)tile * TILE + (size_t)warp * (ROUNDS * 32);
    uint32_t start[ROUNDS], mine = 0;  // a round's segment starts, by lane
    K last = lane == 0 && wbase > 0 && wbase - 1 < n ? keys[wbase - 1] : K(0);
    last = __shfl_sync(0xffffffffu, last, 0);
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const size_t i = wbase + (size_t)r * 32 + lane;
        const K key = i < n ? keys[i] : K(0);
        K prev = __shfl_up_sync(0xffffffffu, key, 1);
        if (lane == 0) prev = last;
        last = __shfl_sync(0xffffffffu, key, 31);
        start[r] = __ballot_sync(0xffffffffu, i < n && (i == 0 || key != prev));
        mine += (uint32_t)__popc(start[r]);
    }
    uint32_t tot;
    uint32_t r0 = block_exclusive_scan(lane == 0 ? mine : 0u, ws, &tot);
    r0 = __shfl_sync(0xffffffffu, r0, 0);
    if (threadIdx.x < 32) {
        unsigned long long e;
        const bool ok = lookback_warp(lb, tile, tot, (int)threadIdx.x, e);
        if (threadIdx.x == 0) {
            s_excl = (uint32_t)e;
            s_ok = ok;
        }
    }
    __syncthreads();
    if (!s_ok) return;
    r0 += s_excl;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        if (start[r] >> lane & 1u)
            starts[r0 + __popc(start[r] & ((1u << lane) - 1u))] =
                (uint32_t)(wbase + (size_t)r * 32 + lane);
        r0 += (uint32_t)__popc(start[r]);
    }
    if (tile == gridDim.x - 1 && threadIdx.x == 0) *num = s_excl + tot;
}

// starts of the runs of equal keys in sorted[0..n), their count in *num_segments (0 when a
// wait ran out); *num_segments zero at the start, lb.words: lookback_bytes(n), 8-byte
// aligned, all zero; n > 0
template <typename K>
static int segment_starts(const K* sorted, size_t n, uint32_t* seg_starts,
                          uint32_t* num_segments, const LookBack& lb, cudaStream_t s) {
    k_seg_starts<K><<<ntiles(n), BT, 0, s>>>(sorted, n, lb, seg_starts, num_segments);
    return cuda_fail(cudaGetLastError(), "segments");
}

int detect_segments(const uint64_t* sorted, size_t n, uint32_t* seg_ids, uint32_t* seg_starts,
                    uint32_t* num_segments, void* temp, size_t temp_bytes, cudaStream_t s) {
    cudaMemsetAsync(num_segments, 0, 4, s);
    if (n == 0) return cuda_fail(cudaGetLastError(), "segments");
    if (temp_bytes < detect_segments_temp_bytes(n)) {
        set_error("detect segments: temporary storage too small");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    char* t = (char*)temp;
    uint32_t* flags = (uint32_t*)t;
    t += align_up(n * 4 + 4, 256);
    uint32_t* ex = (uint32_t*)t;
    t += align_up(n * 4 + 4, 256);
    unsigned g = (unsigned)((n + BT - 1) / BT);
    k_seg_flags<<<g, BT, 0, s>>>(sorted, n, flags);
    int rc = exclusive_scan(flags, ex, n, t, s);
    if (rc) return rc;
    k_seg_finish<<<g, BT, 0, s>>>(flags, ex, n, seg_ids, seg_starts, num_segments);
    return cuda_fail(cudaGetLastError(), "segments");
}

// ---------------------------------------------------------------------------------------
// Cells, bounds and Morton keys.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ bool finite3(float x, float y, float z) {
    return isfinite(x) && isfinite(y) && isfinite(z);
}

__device__ __forceinline__ void cell_of(const float* p, float res, int32_t* c) {
    c[0] = sat_i32(floorf(p[0] / res));
    c[1] = sat_i32(floorf(p[1] / res));
    c[2] = sat_i32(floorf(p[2] / res));
}

// The same by a multiplication with inv = 1 / res where res is a power of two (inv exact, so
// the product is the quotient, rounded alike), else by the division (inv 0)
__device__ __forceinline__ void cell_of_inv(const float* p, float res, float inv, int32_t* c) {
    if (inv == 0.f) {
        cell_of(p, res, c);
        return;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) c[a] = sat_i32(floorf(__fmul_rn(p[a], inv)));
}
static float exact_inverse(float res) {
    int e = 0;
    const float f = std::frexp(res, &e);
    const float inv = 1.0f / res;
    return f == 0.5f && std::isnormal(inv) ? inv : 0.f;
}

// Point i of pts, four consecutive points (i a multiple of 4) as three 16-byte loads when `vec`
// (pts 16-byte aligned) and all four exist; returns how many of the four there are.
__device__ __forceinline__ int load4(const float* __restrict__ pts, size_t n, size_t i, bool vec,
                                     float (*p)[3]) {
    if (vec && i + 4 <= n) {
        const float4* q = reinterpret_cast<const float4*>(pts + 3 * i);
        const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
        const float v[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
#pragma unroll
        for (int k = 0; k < 12; ++k) p[k / 3][k % 3] = v[k];
        return 4;
    }
    int m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (i + k < n) {
            m = k + 1;
            for (int a = 0; a < 3; ++a) p[k][a] = pts[3 * (i + k) + a];
        }
    return m;
}

// mm: [0..2] min cell, [3..5] max cell, [6] finite count. Bound: reading the points once; a
// block adds its seven values with one atomic each (one per warp queued at seven addresses:
// 58 us on 5M points, 17 now).
__global__ void __launch_bounds__(BT) k_cells_minmax(const float* __restrict__ pts, size_t n,
                                                     float res, float inv, bool vec,
                                                     int32_t* __restrict__ mm) {
    __shared__ int32_t red[BT / 32][7];
    int32_t v[6] = {INT32_MAX, INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN, INT32_MIN};
    uint32_t cnt = 0;
    for (size_t i = 4 * ((size_t)blockIdx.x * BT + threadIdx.x); i < n;
         i += 4 * (size_t)gridDim.x * BT) {
        float p[4][3];
        const int m = load4(pts, n, i, vec, p);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k >= m || !finite3(p[k][0], p[k][1], p[k][2])) continue;
            int32_t c[3];
            cell_of_inv(p[k], res, inv, c);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                v[a] = min(v[a], c[a]);
                v[3 + a] = max(v[3 + a], c[a]);
            }
            cnt++;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[a] = __reduce_min_sync(0xffffffffu, v[a]);
        v[3 + a] = __reduce_max_sync(0xffffffffu, v[3 + a]);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
#pragma unroll
        for (int a = 0; a < 6; ++a) red[warp][a] = v[a];
        red[warp][6] = (int32_t)cnt;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int a = threadIdx.x;
        int32_t x = red[0][a];
        for (int w = 1; w < BT / 32; ++w) {
            const int32_t y = red[w][a];
            x = a < 3 ? min(x, y) : (a < 6 ? max(x, y) : x + y);
        }
        if (a < 3) atomicMin(&mm[a], x);
        else if (a < 6) atomicMax(&mm[a], x);
        else atomicAdd(&mm[6], x);
    }
}

__global__ void k_minmax_init(int32_t* mm) {
    if (threadIdx.x < 3) mm[threadIdx.x] = INT32_MAX;
    else if (threadIdx.x < 6) mm[threadIdx.x] = INT32_MIN;
    else if (threadIdx.x == 6) mm[6] = 0;
}

// Morton key of each point's cell relative to the minimum cell, all ones for a non-finite
// point (it sorts last).
__global__ void __launch_bounds__(BT) k_morton(const float* __restrict__ pts, size_t n, float res,
                                               const int32_t* __restrict__ mm,
                                               uint64_t* __restrict__ codes,
                                               uint32_t* __restrict__ idx) {
    size_t i = (size_t)blockIdx.x * BT + threadIdx.x;
    if (i >= n) return;
    float p[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
    uint64_t code = ~0ull;
    if (finite3(p[0], p[1], p[2])) {
        int32_t c[3];
        cell_of(p, res, c);
        uint32_t q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            int64_t d = (int64_t)c[a] - (int64_t)mm[a];
            q[a] = d > 0x1FFFFF ? 0x1FFFFFu : (uint32_t)d;
        }
        code = (uint64_t)morton3(q[0], q[1], q[2]);
    }
    codes[i] = code;
    idx[i] = (uint32_t)i;
}

// Order-preserving 32-bit form of the Morton key of a cell offset inside a box with b[a] bits
// per axis (b0 + b1 + b2 <= 31): the interleaved bits that can be set. Up to the shortest
// axis's bits all three interleave, above them the two longer ones, above those the longest.
struct CompactKey {
    uint32_t lo, mid;         // bits of the shortest and of the middle axis
    uint32_t ax_hi, ax_lo;    // the two longer axes, the earlier of x, y, z first
    uint32_t ax_long;         // the longest
    uint32_t total;           // key bits
};
static CompactKey compact_key(const uint32_t* b) {
    uint32_t o[3] = {0, 1, 2};  // axes by bits, ascending (stable)
    std::stable_sort(o, o + 3, [&](uint32_t x, uint32_t y) { return b[x] < b[y]; });
    CompactKey c;
    c.lo = b[o[0]];
    c.mid = b[o[1]];
    c.ax_hi = std::min(o[1], o[2]);
    c.ax_lo = std::max(o[1], o[2]);
    c.ax_long = o[2];
    c.total = b[0] + b[1] + b[2];
    return c;
}
__host__ __device__ __forceinline__ uint32_t spread16(uint32_t v) {
    v &= 0xFFFFu;
    v = (v | (v << 8)) & 0x00FF00FFu;
    v = (v | (v << 4)) & 0x0F0F0F0Fu;
    v = (v | (v << 2)) & 0x33333333u;
    return (v | (v << 1)) & 0x55555555u;
}
__host__ __device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    return (v | (v << 2)) & 0x09249249u;
}
__host__ __device__ __forceinline__ uint32_t compact_morton(const CompactKey& c,
                                                            const uint32_t* q) {
    const uint32_t lm = (1u << c.lo) - 1u;  // lo <= 10, mid - lo <= 15
    uint32_t key = (spread10(q[0] & lm) << 2) | (spread10(q[1] & lm) << 1) | spread10(q[2] & lm);
    const uint32_t qh = c.ax_hi == 0u ? q[0] : q[1], ql = c.ax_lo == 1u ? q[1] : q[2];
    const uint32_t qx = c.ax_long == 0u ? q[0] : (c.ax_long == 1u ? q[1] : q[2]);
    const uint32_t w = c.mid - c.lo, wm = (1u << w) - 1u;
    key |= ((spread16((qh >> c.lo) & wm) << 1) | spread16((ql >> c.lo) & wm)) << (3u * c.lo);
    const uint32_t up = 3u * c.lo + 2u * w;
    return up < 32u ? key | ((qx >> c.mid) << up) : key;
}

// Compact Morton key of every point (non-finite points: the first value past every cell's, so
// they sort last) and the first sort pass's tile counts. A block takes one tile, four points a
// thread at a time.
__global__ void __launch_bounds__(BT) k_compact_keys(const float* __restrict__ pts, uint32_t n,
                                                     float res, float inv, bool vec,
                                                     const int32_t* __restrict__ mm,
                                                     CompactKey ck, int width,
                                                     uint32_t* __restrict__ keys,
                                                     uint32_t* __restrict__ hist) {
    __shared__ TileCounts t;
    const uint32_t bins = 1u << width;
    tile_counts_clear(t, bins);
    __syncthreads();
    const int32_t mn[3] = {mm[0], mm[1], mm[2]};
#pragma unroll 1
    for (uint32_t r = 0; r < TILE / (4 * BT); ++r) {
        const size_t i = (size_t)blockIdx.x * TILE + 4 * (r * BT + threadIdx.x);
        float p[4][3];
        const int m = i < n ? load4(pts, n, i, vec, p) : 0;
        uint32_t key[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            key[k] = 1u << ck.total;
            if (k < m && finite3(p[k][0], p[k][1], p[k][2])) {
                int32_t c[3];
                cell_of_inv(p[k], res, inv, c);
                const uint32_t q[3] = {(uint32_t)c[0] - (uint32_t)mn[0],
                                       (uint32_t)c[1] - (uint32_t)mn[1],
                                       (uint32_t)c[2] - (uint32_t)mn[2]};
                key[k] = compact_morton(ck, q);
            }
            tile_counts_add(t, key[k] & (bins - 1u), k < m);
        }
        if (m == 4) {
            *reinterpret_cast<uint4*>(keys + i) = make_uint4(key[0], key[1], key[2], key[3]);
        } else {
            for (int k = 0; k < m; ++k) keys[i + k] = key[k];
        }
    }
    __syncthreads();
    tile_counts_store(t, bins, hist, blockIdx.x, gridDim.x);
}

// min / max cell and finite count of the points into mm
static void cell_bounds(const float* pts, size_t n, float res, int32_t* mm, cudaStream_t s) {
    k_minmax_init<<<1, 32, 0, s>>>(mm);
    if (n) {
        unsigned g = (unsigned)std::min<size_t>((n + 4 * BT - 1) / (4 * BT),
                                                  8 * (size_t)device_sms());
        k_cells_minmax<<<g, BT, 0, s>>>(pts, n, res, exact_inverse(res),
                                        ((uintptr_t)pts & 15u) == 0, mm);
    }
}

int morton_codes(const float* pts, size_t n, float res, uint64_t* codes, uint32_t* idx,
                 int32_t* mm, cudaStream_t s) {
    cell_bounds(pts, n, res, mm, s);
    if (n) k_morton<<<(unsigned)((n + BT - 1) / BT), BT, 0, s>>>(pts, n, res, mm, codes, idx);
    return cuda_fail(cudaGetLastError(), "morton codes");
}

// ---------------------------------------------------------------------------------------
// Voxel statistics (one thread per segment) and regularisation.
// ---------------------------------------------------------------------------------------

// Cyclic Jacobi for a symmetric 3x3 in f32 (row-major a, eigenvectors in the columns of v).
// It only has to find the eigenvector directions to f32 accuracy: the eigenvalues and the
// regularised covariance and inverse are then formed in FP64 (k_voxel_stats).
__device__ void jacobi3f(float* a, float* v) {
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) v[i * 3 + j] = (i == j) ? 1.f : 0.f;
#pragma unroll 1
    for (int sweep = 0; sweep < 12; ++sweep) {
        const float off = a[1] * a[1] + a[2] * a[2] + a[5] * a[5];
        const float dg = a[0] * a[0] + a[4] * a[4] + a[8] * a[8];
        if (!(off > 1e-14f * dg)) break;
#pragma unroll
        for (int pq = 0; pq < 3; ++pq) {
            const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
            const float apq = a[p * 3 + q];
            if (apq == 0.f) continue;
            const float theta = (a[q * 3 + q] - a[p * 3 + p]) / (2.f * apq);
            float t = 1.f / (fabsf(theta) + sqrtf(theta * theta + 1.f));
            if (theta < 0.f) t = -t;
            const float c = 1.f / sqrtf(t * t + 1.f);
            const float sn = t * c;
            a[p * 3 + p] -= t * apq;
            a[q * 3 + q] += t * apq;
            a[p * 3 + q] = a[q * 3 + p] = 0.f;
            const int r = 3 - p - q;
            const float arp = a[r * 3 + p], arq = a[r * 3 + q];
            a[r * 3 + p] = a[p * 3 + r] = c * arp - sn * arq;
            a[r * 3 + q] = a[q * 3 + r] = sn * arp + c * arq;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float vp = v[k * 3 + p], vq = v[k * 3 + q];
                v[k * 3 + p] = c * vp - sn * vq;
                v[k * 3 + q] = sn * vp + c * vq;
            }
        }
    }
}

// FP64 cyclic Jacobi sweeps on B = V^T A V, rotating V along (B and V row-major, V's columns
// the eigenvector estimates), until the reference's rule 2 off^2 < 1e-28 diag^2 holds or
// max_sweeps pass. Started from an orthonormalised f32 solution, B is diagonal to about 1e-7
// of its scale and one or two sweeps reach FP64 accuracy.
__device__ void jacobi3_refine(double* B, double* V, int max_sweeps) {
    for (int sweep = 0; sweep < max_sweeps; ++sweep) {
        const double off = B[1] * B[1] + B[2] * B[2] + B[5] * B[5];
        const double dg = B[0] * B[0] + B[4] * B[4] + B[8] * B[8];
        if (2.0 * off <= 1e-28 * dg) break;
        for (int pq = 0; pq < 3; ++pq) {
            const int p = pq == 2 ? 1 : 0, q = pq == 0 ? 1 : 2;
            const double bpq = B[p * 3 + q];
            if (bpq == 0.0) continue;
            const double theta = (B[q * 3 + q] - B[p * 3 + p]) / (2.0 * bpq);
            double t = 1.0 / (fabs(theta) + sqrt(theta * theta + 1.0));
            if (theta < 0.0) t = -t;
            const double c = 1.0 / sqrt(t * t + 1.0);
            const double sn = t * c;
            B[p * 3 + p] -= t * bpq;
            B[q * 3 + q] += t * bpq;
            B[p * 3 + q] = B[q * 3 + p] = 0.0;
            const int r = 3 - p - q;
            const double brp = B[r * 3 + p], brq = B[r * 3 + q];
            B[r * 3 + p] = B[p * 3 + r] = c * brp - sn * brq;
            B[r * 3 + q] = B[q * 3 + r] = sn * brp + c * brq;
            for (int k = 0; k < 3; ++k) {
                const double vp = V[k * 3 + p], vq = V[k * 3 + q];
                V[k * 3 + p] = c * vp - sn * vq;
                V[k * 3 + q] = sn * vp + c * vq;
            }
        }
    }
}

// FP64 Rayleigh quotient v^T A v / v^T v of an f32 unit vector v (|v|^2 = 1 +- 1e-7, so
// 1 / v^T v = 2 - v^T v to FP64 rounding): FP64-accurate for an eigenvalue, since its error
// is quadratic in v's direction error. *w receives 1 / v^T v.
__device__ __forceinline__ double rayleigh(const double* A, const double* v, double* w) {
    double num = 0.0;
    for (int rr = 0; rr < 3; ++rr)
        num += v[rr] * (A[rr * 3] * v[0] + A[rr * 3 + 1] * v[1] + A[rr * 3 + 2] * v[2]);
    const double vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    *w = 2.0 - vv;
    return num * *w;
}

// Inverse of a symmetric positive definite 3x3 by its adjugate (FP64); false unless det > 0.
__device__ __forceinline__ bool inverse_sym3(const double* C, float* icov6) {
    const double c00 = C[4] * C[8] - C[5] * C[5];
    const double c01 = C[2] * C[5] - C[1] * C[8];
    const double c02 = C[1] * C[5] - C[2] * C[4];
    const double c11 = C[0] * C[8] - C[2] * C[2];
    const double c12 = C[1] * C[2] - C[0] * C[5];
    const double c22 = C[0] * C[4] - C[1] * C[1];
    const double det = C[0] * c00 + C[1] * c01 + C[2] * c02;
    if (!(det > 0.0)) return false;
    const double id = 1.0 / det;
    icov6[0] = (float)(c00 * id);
    icov6[1] = (float)(c01 * id);
    icov6[2] = (float)(c02 * id);
    icov6[3] = (float)(c11 * id);
    icov6[4] = (float)(c12 * id);
    icov6[5] = (float)(c22 * id);
    return true;
}

// First-order correction of an f32 eigenvector v (eigenvalue lam) against the eigenvectors
// v_j of the set `others` (bit mask): v += sum_j (v_j^T (A v - lam v)) / (lam - lam_j) v_j
// (w_j = 1 / v_j^T v_j). The direction error drops from about 1e-7 lambda_max / gap to its
// square; the 1 / gap factors need only f32 accuracy.
__device__ __forceinline__ void refine_vector(const double* A, double* v, double lam,
                                              const double (*vs)[3], const double* lams,
                                              const double* ws, int others) {
    double r[3];
    for (int rr = 0; rr < 3; ++rr)
        r[rr] = A[rr * 3] * v[0] + A[rr * 3 + 1] * v[1] + A[rr * 3 + 2] * v[2] - lam * v[rr];
    double dv[3] = {0.0, 0.0, 0.0};
    for (int j = 0; j < 3; ++j) {
        if (!(others >> j & 1)) continue;
        const double proj = vs[j][0] * r[0] + vs[j][1] * r[1] + vs[j][2] * r[2];
        const double inv = (double)(1.f / (float)(lam - lams[j]));
        const double c = proj * ws[j] * inv;
        for (int k = 0; k < 3; ++k) dv[k] += c * vs[j][k];
    }
    for (int k = 0; k < 3; ++k) v[k] += dv[k];
}

// Regularised covariance and inverse of the FP64 covariance A (Voxel::from_statistics /
// regularize_covariance, src/ndt_cuda/src/voxel_grid/types.rs:54-190): eigenvalues below
// ratio * lambda_max are raised to it; cov' = V diag(clamped) V^T when any was, else A;
// inverse V diag(1 / clamped) V^T. a32 / V32: the f32 Jacobi's eigenvalues (diagonal) and
// eigenvectors (columns). Which eigenvalues clamp is read from the f32 eigenvalues when they
// lie clear of the threshold (1e-4 relative, against their 1e-5 error there), and the clamped
// ones lie at least lambda_max / 1000 below the others (an f32 direction error of 1e-4 at most,
// 1e-8 after the first-order refinement); then, with FP64 Rayleigh quotients as
// the eigenvalues:
//   - nothing clamps: cov' = A, inverse by the adjugate (A's condition number <= 1 / ratio);
//   - one clamps: cov' = A + (thr - lambda_c) v_c v_c^T, v_c refined against the other two;
//   - two clamp: cov' = thr I + (lambda_u - thr) v_u v_u^T, v_u refined against the other
//     two (mixing inside the clamped pair then cannot matter);
//   and the inverse by the adjugate of cov'.
// Anything else takes the full FP64 route: the f32 eigenvectors orthonormalised
// (Gram-Schmidt), Jacobi sweeps on V^T A V to the reference's stopping rule, and the
// reconstruction from the eigen-decomposition. Every route is FP64-accurate, so the f32
// outputs agree with an FP64 eigen-decomposition to f32 rounding.
__device__ bool regularize(const double* A, const float* a32, const float* V32, float ratio,
                           SegRec& r) {
    const float e32[3] = {a32[0], a32[4], a32[8]};
    const float mx32 = fmaxf(e32[0], fmaxf(e32[1], e32[2]));
    bool fast = mx32 > 0.f;
    int clamp = 0;  // bit i: eigenvalue i clamps
    if (fast) {
        const float thr32 = mx32 * ratio;
        for (int i = 0; i < 3; ++i) {
            if (e32[i] <= thr32 * 0.9999f) {
                clamp |= 1 << i;
            } else if (!(e32[i] >= thr32 * 1.0001f)) {
                fast = false;
            }
        }
        for (int i = 0; i < 3 && fast; ++i)
            for (int j = 0; j < 3; ++j)
                if ((clamp >> i & 1) && !(clamp >> j & 1) && e32[j] - e32[i] < 0.001f * mx32)
                    fast = false;
    }
    if (fast) {
        if (!clamp) {
            for (int q = 0; q < 9; ++q) r.cov[q] = (float)A[q];
            return inverse_sym3(A, r.icov);
        }
        double v[3][3], w[3], lam[3];
        for (int i = 0; i < 3; ++i) {
            for (int k = 0; k < 3; ++k) v[i][k] = (double)V32[k * 3 + i];
            lam[i] = rayleigh(A, v[i], &w[i]);
        }
        const double mx = fmax(lam[0], fmax(lam[1], lam[2]));
        if (!(mx > 0.0)) return false;
        const double thr = mx * (double)ratio;
        const int one = __popc(clamp) == 1;
        const int t = one ? __ffs(clamp) - 1 : __ffs(7 & ~clamp) - 1;  // the vector to refine
        double u[3] = {v[t][0], v[t][1], v[t][2]};
        refine_vector(A, u, lam[t], v, lam, w, 7 & ~(1 << t));
        const double wu = 2.0 - (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
        double C[9];
        const double c = one ? (thr - lam[t]) * wu : (lam[t] - thr) * wu;
        for (int rr = 0; rr < 3; ++rr)
            for (int cc = rr; cc < 3; ++cc) {  // upper triangle, mirrored: C stays symmetric
                const double base = one ? A[rr * 3 + cc] : (rr == cc ? thr : 0.0);
                C[rr * 3 + cc] = C[cc * 3 + rr] = base + c * u[rr] * u[cc];
            }
        for (int q = 0; q < 9; ++q) r.cov[q] = (float)C[q];
        return inverse_sym3(C, r.icov);
    }
    // full FP64 route: orthonormal basis from the f32 eigenvectors, Jacobi sweeps on V^T A V
    double V[9];
    for (int q = 0; q < 9; ++q) V[q] = (double)V32[q];
    for (int i = 0; i < 3; ++i) {
        for (int j = 0; j < i; ++j) {
            const double d = V[i] * V[j] + V[3 + i] * V[3 + j] + V[6 + i] * V[6 + j];
            for (int k = 0; k < 3; ++k) V[k * 3 + i] -= d * V[k * 3 + j];
        }
        const double inv = 1.0 / sqrt(V[i] * V[i] + V[3 + i] * V[3 + i] + V[6 + i] * V[6 + i]);
        for (int k = 0; k < 3; ++k) V[k * 3 + i] *= inv;
    }
    double AV[9], B[9];
    for (int rr = 0; rr < 3; ++rr)
        for (int cc = 0; cc < 3; ++cc)
            AV[rr * 3 + cc] =
                A[rr * 3] * V[cc] + A[rr * 3 + 1] * V[3 + cc] + A[rr * 3 + 2] * V[6 + cc];
    for (int rr = 0; rr < 3; ++rr)
        for (int cc = rr; cc < 3; ++cc)
            B[rr * 3 + cc] = B[cc * 3 + rr] =
                V[rr] * AV[cc] + V[3 + rr] * AV[3 + cc] + V[6 + rr] * AV[6 + cc];
    jacobi3_refine(B, V, 4);
    const double ev[3] = {B[0], B[4], B[8]};
    const double mx = fmax(ev[0], fmax(ev[1], ev[2]));
    if (!(mx > 0.0)) return false;
    const double thr = mx * (double)ratio;
    int needs = 0;
    double cl[3], icl[3];
    for (int i = 0; i < 3; ++i) {
        cl[i] = ev[i] < thr ? thr : ev[i];
        if (ev[i] < thr) needs = 1;
        icl[i] = 1.0 / cl[i];
    }
    for (int rr = 0; rr < 3; ++rr)
        for (int cc = rr; cc < 3; ++cc) {
            double sr = 0.0, si = 0.0;
            for (int k = 0; k < 3; ++k) {
                const double vv = V[rr * 3 + k] * V[cc * 3 + k];
                sr += vv * cl[k];
                si += vv * icl[k];
            }
            const float fc = (float)(needs ? sr : A[rr * 3 + cc]);
            r.cov[rr * 3 + cc] = r.cov[cc * 3 + rr] = fc;
            r.icov[rr == 0 ? cc : (rr == 1 ? 2 + cc : 5)] = (float)si;
        }
    return true;
}

// ---- Exact moments ------------------------------------------------------------------------
// Per axis, a quantum 2^e0 from the voxel's cell k: its points lie within
// B = max(|k|, |k + 1|) resolutions of zero, below 2^EB (B < 2^EB with a 1e-3 margin for the
// f32 cell rule). For a cell at least one resolution from zero every point is at least about
// B / 2, a multiple of its ulp >= 2^(EB - 26): e0 = EB - 26. A cell next to zero (k = 0 or
// -1) holds values of any size: e0 = EB - 40. Each point is then m 2^e0 with an integer
// |m| < 2^40, exact unless it is a value below 2^(e0 + 23) whose low bits fall under the
// quantum (it is rounded then, by at most 2^-41 of the cell's reach). With d = m - m_first
// (|d| < 2^41) the sums S1 = sum d (int64) and S2 = sum d d^T (128-bit) are exact for up to
// 65536 points and independent of the order of the points. From them:
//   - the mean of an axis whose points were all exact and whose sum (S1 + n m_first) has at
//     most 53 significant bits above the coarsest power of two dividing every point: every
//     partial sum of these same-sign values (one cell) is then an FP64 number, so the FP64
//     running sum in input order (build_voxel_grid_cpu, src/ndt_cuda/src/voxel_grid/cpu.rs:
//     51-75) never rounds and equals it, and fl(sum / n) is its mean bit for bit. Any other
//     axis takes that running sum in input order (moments_mean_fp64);
//   - the centred covariance (n S2 - S1 S1^T) 2^(e0a + e0b) / (n (n - 1)) from the 128-bit
//     numerator rounded once to FP64 and the FP64 reciprocal of n (n - 1): within a few
//     roundings of the exact value whatever the order of the points (a tile merge and a full
//     build of the same cell agree bit for bit).
// A value beyond the cell's reach or non-finite sends the voxel to the FP64 two-pass formula.
struct ExactMoments {
    int32_t e0[3];            // quantum exponent per axis
    int32_t tz[3];            // fewest trailing zero bits of a non-zero m (the coarse quantum)
    long long m0[3];          // the first point in quanta
    long long s1[3];
    long long s2h[6];         // xx, xy, xz, yy, yz, zz as 128-bit (hi, lo)
    unsigned long long s2l[6];
    bool rep[3];              // every point of the axis an exact multiple of 2^e0
    bool ok;                  // every point within the cell's reach
};

// m of one coordinate in quanta 2^e0 (rounded to nearest; rep cleared when inexact, ok when
// beyond 2^(e0 + 40))
__device__ __forceinline__ long long exact_units(float x, int32_t e0, bool& rep, int32_t& tz,
                                                 bool& ok) {
    const uint32_t b = __float_as_uint(x);
    const uint32_t ex = (b >> 23) & 0xFFu;
    if (ex == 0u) {  // +-0 is exact; a subnormal rounds to 0 quanta
        rep &= (b << 1) == 0u;
        return 0;
    }
    ok &= ex != 0xFFu;
    const int32_t sh = (int32_t)ex - 150 - e0;
    ok &= sh <= 16;
    const unsigned long long M = (b & 0x7FFFFFu) | 0x800000u;
    unsigned long long m;
    if (sh >= 0) {
        m = M << (sh & 63);
    } else if (sh > -25) {
        const int r = -sh;
        rep &= (M & ((1ull << r) - 1ull)) == 0ull;
        m = (M + (1ull << (r - 1))) >> r;
    } else {
        rep = false;
        m = 0;
    }
    if (m) tz = min(tz, __ffsll((long long)m) - 1);
    return (b >> 31) ? -(long long)m : (long long)m;
}

__device__ __forceinline__ void add_prod128(long long& hi, unsigned long long& lo, long long a,
                                            long long b) {
    const unsigned long long pl = (unsigned long long)a * (unsigned long long)b;
    const long long ph = __mul64hi(a, b);
    const unsigned long long s = lo + pl;
    hi += ph + (s < lo ? 1ll : 0ll);
    lo = s;
}

// quanta of the cell `coord` (the f32 cell index of the voxel) and the first point
__device__ __forceinline__ void exact_begin(ExactMoments& em, const float* p, const int32_t* coord,
                                            float res) {
    em.ok = true;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float k = (float)coord[a];
        const float reach = fmaxf(fabsf(k), fabsf(k + 1.f)) * res * 1.001f;
        int eb;
        frexpf(reach, &eb);  // reach < 2^eb
        em.e0[a] = eb - ((coord[a] == 0 || coord[a] == -1) ? 40 : 26);
        em.tz[a] = 64;
        em.rep[a] = true;
        em.s1[a] = 0;
        em.m0[a] = exact_units(p[a], em.e0[a], em.rep[a], em.tz[a], em.ok);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        em.s2h[k] = 0;
        em.s2l[k] = 0ull;
    }
}

__device__ __forceinline__ void exact_add(ExactMoments& em, const float* p) {
    long long d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        d[a] = exact_units(p[a], em.e0[a], em.rep[a], em.tz[a], em.ok) - em.m0[a];
        em.s1[a] += d[a];
    }
    add_prod128(em.s2h[0], em.s2l[0], d[0], d[0]);
    add_prod128(em.s2h[1], em.s2l[1], d[0], d[1]);
    add_prod128(em.s2h[2], em.s2l[2], d[0], d[2]);
    add_prod128(em.s2h[3], em.s2l[3], d[1], d[1]);
    add_prod128(em.s2h[4], em.s2l[4], d[1], d[2]);
    add_prod128(em.s2h[5], em.s2l[5], d[2], d[2]);
}

// 2^e as an FP64 (normal range)
__device__ __forceinline__ double pow2d(int e) {
    return __longlong_as_double((long long)(e + 1023) << 52);
}

// A signed 128-bit integer (hi, lo) rounded once to the nearest FP64 (ties to even)
__device__ __forceinline__ double i128_to_double(long long hi, unsigned long long lo) {
    const bool neg = hi < 0;
    unsigned long long uh = (unsigned long long)hi, ul = lo;
    if (neg) {
        ul = ~ul + 1ull;
        uh = ~uh + (ul == 0ull ? 1ull : 0ull);
    }
    if (uh == 0ull) {
        const double v = __ull2double_rn(ul);
        return neg ? -v : v;
    }
    const int lz = __clzll((long long)uh);
    unsigned long long top = lz ? (uh << lz) | (ul >> (64 - lz)) : uh;
    const unsigned long long rest = lz ? ul << lz : ul;
    if (rest != 0ull) top |= 1ull;  // sticky: the discarded bits decide ties and halves
    const double v = __ull2double_rn(top) * pow2d(64 - lz);
    return neg ? -v : v;
}

// Mean and covariance from exact sums over n points. Returns a mask of the axes whose mean
// the exact sums cannot give (bit a set: take the FP64 running sum of axis a).
__device__ __forceinline__ int exact_finish(const ExactMoments& em, uint32_t n, double* mean,
                                            double* A) {
    const double nn = (double)n;
    int redo = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const long long tot = em.s1[a] + (long long)n * em.m0[a];
        const unsigned long long mag = tot < 0 ? (unsigned long long)(-tot) : (unsigned long long)tot;
        const int sig = mag ? 64 - __clzll((long long)mag) - min(em.tz[a], 63) : 0;
        if (em.rep[a] && sig <= 53) {
            mean[a] = (__ll2double_rn(tot) * pow2d(em.e0[a])) / nn;
        } else {
            redo |= 1 << a;
        }
    }
    const double inv_den = 1.0 / (nn * (double)(n - 1u));
    const int ia[6] = {0, 0, 0, 1, 1, 2}, ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        // n S2 (128-bit times a small unsigned) minus S1_a S1_b (64 x 64 -> 128), exact
        const unsigned long long nl = em.s2l[k] * (unsigned long long)n;
        const long long nh = em.s2h[k] * (long long)n +
                             (long long)__umul64hi(em.s2l[k], (unsigned long long)n);
        const long long pa = em.s1[ia[k]], pb = em.s1[ib[k]];
        const unsigned long long ql = (unsigned long long)pa * (unsigned long long)pb;
        const long long qh = __mul64hi(pa, pb);
        const unsigned long long rl = nl - ql;
        const long long rh = nh - qh - (nl < ql ? 1ll : 0ll);
        const double v =
            i128_to_double(rh, rl) * pow2d(em.e0[ia[k]] + em.e0[ib[k]]) * inv_den;
        A[ia[k] * 3 + ib[k]] = A[ib[k] * 3 + ia[k]] = v;
    }
    return redo;
}

// The FP64 running sums of the axes in `axes` (bit mask) over the points in input order, the
// means fl(sum / n) (build_voxel_grid_cpu's accumulation)
template <class Each>
__device__ __noinline__ void moments_mean_fp64(Each each, uint32_t cnt, int axes, double* mean) {
    double sum[3] = {0.0, 0.0, 0.0};
    each([&](const float* p) {
        sum[0] += (double)p[0];
        sum[1] += (double)p[1];
        sum[2] += (double)p[2];
    });
    for (int a = 0; a < 3; ++a)
        if (axes >> a & 1) mean[a] = sum[a] / (double)cnt;
}

// FP64 centred two-pass moments of one voxel's points, visited in input order by each(f) (f
// called with a pointer to each point's xyz): mean = sum / n, covariance = sum of the centred
// products / (n - 1). The route for voxels the exact sums cannot take.
template <class Each>
__device__ __noinline__ void moments_two_pass(Each each, uint32_t cnt, double* mean, double* A) {
    double sum[3] = {0.0, 0.0, 0.0};
    each([&](const float* p) {
        sum[0] += (double)p[0];
        sum[1] += (double)p[1];
        sum[2] += (double)p[2];
    });
    const double nn = (double)cnt;
    for (int a = 0; a < 3; ++a) mean[a] = sum[a] / nn;
    // upper triangle xx, xy, xz, yy, yz, zz (the products are symmetric bit for bit)
    double sq[6] = {0, 0, 0, 0, 0, 0};
    each([&](const float* p) {
        const double d0 = (double)p[0] - mean[0], d1 = (double)p[1] - mean[1],
                     d2 = (double)p[2] - mean[2];
        sq[0] += d0 * d0;
        sq[1] += d0 * d1;
        sq[2] += d0 * d2;
        sq[3] += d1 * d1;
        sq[4] += d1 * d2;
        sq[5] += d2 * d2;
    });
    const double nm1 = nn - 1.0;
    A[0] = sq[0] / nm1;
    A[1] = A[3] = sq[1] / nm1;
    A[2] = A[6] = sq[2] / nm1;
    A[4] = sq[3] / nm1;
    A[5] = A[7] = sq[4] / nm1;
    A[8] = sq[5] / nm1;
}

// Regularised covariance, inverse and mean of a voxel from its FP64 mean and covariance
// A. GB300's FP64 rate is a small fraction of its FP32 rate: the eigenvector directions come
// from an f32 Jacobi, and FP64 is spent only where the outputs depend on it (regularize).
__device__ __forceinline__ bool voxel_finish(const double* mean, const double* A, float ratio,
                                             SegRec& r) {
    float a32[9], V32[9];
    for (int q = 0; q < 9; ++q) a32[q] = (float)A[q];
    jacobi3f(a32, V32);
    if (!regularize(A, a32, V32, ratio, r)) return false;
    for (int q = 0; q < 3; ++q) r.mean[q] = (float)mean[q];
    return true;
}

constexpr uint32_t SIZE_KEY_MAX = 255;

// Largest voxel whose sums stay exact (S1 below 2^57, S2 below 2^98 with |d| < 2^41)
constexpr uint32_t EXACT_MAX_POINTS = 65536;

// Statistics of one voxel by one thread: count, then exact moments (FP64 running sums for
// the axes whose mean they cannot give) when the voxel has at most EXACT_MAX_POINTS points
// within the exact bounds, else FP64 two-pass moments; then voxel_finish. each(f) visits the
// voxel's points in input order; first: its first point. r.coord (the voxel's cell) is the
// caller's.
template <class Each>
__device__ __forceinline__ bool voxel_stats(Each each, const float* first, uint32_t cnt,
                                            int min_points, float ratio, float res, SegRec& r) {
    r.count = cnt;
    if ((int)cnt < min_points) return false;
    double mean[3], A[9];
    bool exact = cnt <= EXACT_MAX_POINTS;
    ExactMoments em;
    if (exact) {
        exact_begin(em, first, r.coord, res);
        each([&](const float* p) { exact_add(em, p); });
        exact = em.ok;
    }
    if (exact) {
        const int redo = exact_finish(em, cnt, mean, A);
        if (redo) moments_mean_fp64(each, cnt, redo, mean);
    } else {
        moments_two_pass(each, cnt, mean, A);
    }
    return voxel_finish(mean, A, ratio, r);
}

// Segment sizes as 8-bit sort keys: segments visited largest first (key 255 - min(count, 255)),
// so the threads of a warp take segments of nearly equal size and the longest start first.
__global__ void k_seg_size_keys(const uint32_t* __restrict__ starts, uint32_t S, uint32_t nf,
                                uint32_t* __restrict__ keys) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const uint32_t e = s + 1 < S ? starts[s + 1] : nf;
    keys[s] = SIZE_KEY_MAX - min(e - starts[s], SIZE_KEY_MAX);
}

// Voxels of at least WARP_SEG_MIN points are summed by a whole warp (exact sums of the lanes'
// strided shares, added over the lanes in 128-bit), up to EXACT_MAX_POINTS points.
constexpr uint32_t WARP_SEG_MIN = 48;
static_assert(WARP_SEG_MIN < SIZE_KEY_MAX, "the size keys tell large segments apart");

// 128-bit (hi, lo) sum over the warp's lanes (every lane ends with the total)
__device__ __forceinline__ void warp_sum128(long long& hi, unsigned long long& lo) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ol = __shfl_xor_sync(0xffffffffu, lo, o);
        const long long oh = __shfl_xor_sync(0xffffffffu, hi, o);
        const unsigned long long s = lo + ol;
        hi = hi + oh + (s < lo ? 1ll : 0ll);
        lo = s;
    }
}

// f(point) for the points sidx[k], k = b, b + step, ... < e, in that order, with the loads of
// four points issued together (the gathers are random reads of the map: four in flight per
// thread instead of one)
template <class F>
__device__ __forceinline__ void visit_points(const float* __restrict__ pts,
                                             const uint32_t* __restrict__ sidx, uint32_t b,
                                             uint32_t e, uint32_t step, F f) {
    uint32_t k = b;
    for (; k + 3 * step < e; k += 4 * step) {
        float v[4][3];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float* q = pts + 3 * (size_t)sidx[k + j * step];
            v[j][0] = q[0];
            v[j][1] = q[1];
            v[j][2] = q[2];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) f(v[j]);
    }
    for (; k < e; k += step) f(pts + 3 * (size_t)sidx[k]);
}

// Exact sums of one large segment, as a warp leaves them for the thread that finishes it
struct SegSums {
    long long s1[3];
    long long hi[6];
    unsigned long long lo[6];
    int32_t tz[3];
    int32_t flags;  // bit 0: the exact route holds; bits 1-3: axis a's points all exact
};

// Number of visit-order segments with at least WARP_SEG_MIN points (sorted size keys ascend)
__device__ __forceinline__ uint32_t large_segments(const uint32_t* __restrict__ skey, uint32_t S) {
    uint32_t lo = 0, hi = S;
    const uint32_t lim = SIZE_KEY_MAX - WARP_SEG_MIN;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (skey[mid] <= lim) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Exact sums of the large segments (the first W in visit order, order[t], largest first),
// one warp per segment at a time (lanes take strided shares, the 128-bit sums are added over
// the lanes), into sums[t]. k_voxel_stats finishes them one per thread.
__global__ void __launch_bounds__(128) k_segment_sums(
    const float* __restrict__ pts, const uint32_t* __restrict__ sidx,
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ order,
    const uint32_t* __restrict__ skey, const uint32_t* __restrict__ failed, uint32_t S,
    uint32_t nf, float res, int min_points, SegSums* __restrict__ sums) {
    if (*failed) return;
    __shared__ uint32_t sW;
    if (threadIdx.x == 0) sW = large_segments(skey, S);
    __syncthreads();
    const uint32_t W = sW;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < W; t += warps) {
        const uint32_t s = order[t];
        const uint32_t b = starts[s];
        const uint32_t e = (s + 1 < S) ? starts[s + 1] : nf;
        const uint32_t cnt = e - b;
        if ((int)cnt < min_points) continue;
        const float* first = pts + 3 * (size_t)sidx[b];
        int32_t coord[3];
        cell_of(first, res, coord);
        ExactMoments em;
        exact_begin(em, first, coord, res);
        visit_points(pts, sidx, b + lane, e, 32u, [&](const float* p) { exact_add(em, p); });
        const bool exact = __all_sync(0xffffffffu, em.ok) && cnt <= EXACT_MAX_POINTS;
        int flags = exact ? 1 : 0;
        SegSums& o = sums[t];
        if (exact) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
#pragma unroll
                for (int k = 16; k > 0; k >>= 1) {
                    em.s1[a] += __shfl_xor_sync(0xffffffffu, em.s1[a], k);
                    em.tz[a] = min(em.tz[a], __shfl_xor_sync(0xffffffffu, em.tz[a], k));
                }
                if (__all_sync(0xffffffffu, em.rep[a])) flags |= 2 << a;
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                long long h = em.s2h[k];
                unsigned long long l = em.s2l[k];
                warp_sum128(h, l);
                if (lane == 0) {
                    o.hi[k] = h;
                    o.lo[k] = l;
                }
            }
            if (lane == 0)
                for (int a = 0; a < 3; ++a) {
                    o.s1[a] = em.s1[a];
                    o.tz[a] = em.tz[a];
                }
        }
        if (lane == 0) o.flags = flags;
    }
}

// One thread per segment in visit order (order[t], largest first; skey[t] its sorted size
// key). The first W (WARP_SEG_MIN points or more) are finished from their sums in sums[t]
// (k_segment_sums); the others are summed here. Every segment's record gets its cell and
// count (a tile merge reads them for cells shared between tiles); valid[s] marks the voxels.
__global__ void __launch_bounds__(128) k_voxel_stats(
    const float* __restrict__ pts, const uint32_t* __restrict__ sidx,
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ order,
    const uint32_t* __restrict__ skey, const uint32_t* __restrict__ failed,
    const SegSums* __restrict__ sums, uint32_t S, uint32_t nf, float res, int min_points,
    float ratio, SegRec* __restrict__ rec, uint32_t* __restrict__ valid) {
    if (*failed) return;
    __shared__ uint32_t sW;
    if (threadIdx.x == 0) sW = large_segments(skey, S);
    __syncthreads();
    const uint32_t W = sW;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= S) return;
    const uint32_t s = order[t];
    const uint32_t b = starts[s];
    const uint32_t e = (s + 1 < S) ? starts[s + 1] : nf;
    const uint32_t cnt = e - b;
    const float* first = pts + 3 * (size_t)sidx[b];
    SegRec r;
    cell_of(first, res, r.coord);
    auto each = [&](auto f) { visit_points(pts, sidx, b, e, 1u, f); };
    bool ok;
    if (t < W) {
        r.count = cnt;
        ok = false;
        if ((int)cnt >= min_points) {
            double mean[3], A[9];
            const SegSums& ss = sums[t];
            const int flags = ss.flags;
            if (flags & 1) {
                ExactMoments em;
                exact_begin(em, first, r.coord, res);
                for (int a = 0; a < 3; ++a) {
                    em.s1[a] = ss.s1[a];
                    em.tz[a] = ss.tz[a];
                    em.rep[a] = (flags >> (a + 1)) & 1;
                }
                for (int k = 0; k < 6; ++k) {
                    em.s2h[k] = ss.hi[k];
                    em.s2l[k] = ss.lo[k];
                }
                const int redo = exact_finish(em, cnt, mean, A);
                if (redo) moments_mean_fp64(each, cnt, redo, mean);
            } else {
                moments_two_pass(each, cnt, mean, A);
            }
            ok = voxel_finish(mean, A, ratio, r);
        }
    } else {
        ok = voxel_stats(each, first, cnt, min_points, ratio, res, r);
    }
    rec[s] = r;
    valid[s] = ok ? 1u : 0u;
}

// Inserts `key` into an open-addressing table of keys (stride words apart): its slot and its
// displacement from the home slot s, or -1 when the table is full.
__device__ __forceinline__ int64_t hash_claim(uint32_t* keys, uint32_t stride, uint32_t mask,
                                              uint32_t key, uint32_t s, uint32_t& disp) {
    for (uint32_t j = 0; j <= mask; ++j) {
        if (atomicCAS(keys + (size_t)s * stride, EMPTY_KEY, key) == EMPTY_KEY) {
            disp = j;
            return (int64_t)s;
        }
        s = (s + 1) & mask;
    }
    return -1;
}

// Valid voxels of the S segment records, in order, into the map's voxel arrays and the search
// records. With the dense index (grid set) the record of a voxel is written at its own index
// and its grid entry {centroid, voxel} at its cell, and only its key is inserted into a table
// of 4-byte keys: no search reads the table then, but the map's description reports its
// longest probe. Otherwise the voxel goes to its hash slot. On the 50M-point 2 m map (3.1M
// voxels) writing 52 bytes to each random slot took 607 us and filling the grid from the
// slots 112 us more; records in voxel order are written by neighbouring threads, and
// neighbouring voxels share the lines that the searches read.
// A block reads its 128 records and writes its voxels (consecutive ones: ranks are a scan)
// through shared memory, so 88-byte records and 36-byte matrices move as whole lines (a thread
// each was bound by the load-store unit's replays). Compaction, hash insert and grid of the
// 50M-point 2 m map together: 0.88 ms as three kernels, 0.36 now.
constexpr int VC = 128;
__global__ void __launch_bounds__(VC) k_voxel_compact(
    const SegRec* __restrict__ rec, const uint32_t* __restrict__ valid,
    const uint32_t* __restrict__ rank, uint32_t S, int32_t* __restrict__ coord,
    float4* __restrict__ mean4, float* __restrict__ cov, float* __restrict__ icov,
    uint32_t* __restrict__ count, MapView m, float4* __restrict__ icov8,
    float4* __restrict__ grid, uint32_t* __restrict__ keys, uint4* __restrict__ slots,
    int32_t* __restrict__ slot_vidx, uint32_t* __restrict__ max_probe,
    uint32_t* __restrict__ status) {
    constexpr int RW = sizeof(SegRec) / 4;
    static_assert(sizeof(SegRec) == RW * 4, "records move as words");
    __shared__ uint32_t in[VC * RW];
    __shared__ float o_cov[VC * 9], o_icov[VC * 9];
    __shared__ int32_t o_coord[VC * 3];
    const uint32_t s0 = blockIdx.x * VC, s = s0 + threadIdx.x, ns = min((uint32_t)VC, S - s0);
    for (uint32_t i = threadIdx.x; i < ns * RW; i += VC)
        in[i] = __ldg(reinterpret_cast<const uint32_t*>(rec + s0) + i);
    const bool ok = s < S && valid[s];
    const uint32_t v0 = rank[s0], v = s < S ? rank[s] : 0u;
    const uint32_t nv = (uint32_t)__syncthreads_count(ok);
    uint32_t disp = 0;  // this voxel's displacement from its home slot
    if (ok) {
        const SegRec& r = *reinterpret_cast<const SegRec*>(in + threadIdx.x * RW);
        const uint32_t lv = v - v0;
        const int32_t g[3] = {r.coord[0], r.coord[1], r.coord[2]};
        for (int a = 0; a < 3; ++a) o_coord[3 * lv + a] = g[a];
        const float mu[3] = {r.mean[0], r.mean[1], r.mean[2]};
        mean4[v] = make_float4(mu[0], mu[1], mu[2], __uint_as_float(r.count));
        for (int q = 0; q < 9; ++q) o_cov[9 * lv + q] = r.cov[q];
        float c[6];
        for (int q = 0; q < 6; ++q) c[q] = r.icov[q];
        const float full[9] = {c[0], c[1], c[2], c[1], c[3], c[4], c[2], c[4], c[5]};
        for (int q = 0; q < 9; ++q) o_icov[9 * lv + q] = full[q];
        count[v] = r.count;
        uint32_t key, home;
        cell_slot(m, g[0], g[1], g[2], key, home);  // every voxel lies inside the map's box
        int64_t at;
        if (grid) {
            const size_t cell = ((size_t)(g[0] - m.min_cell[0]) * m.ext[1] +
                                 (g[1] - m.min_cell[1])) * m.ext[2] + (g[2] - m.min_cell[2]);
            grid[cell] = make_float4(mu[0], mu[1], mu[2], __int_as_float((int32_t)v));
            at = hash_claim(keys, 1u, m.mask, key, home, disp) < 0 ? -1 : (int64_t)v;
        } else {
            at = hash_claim(&slots[0].w, 4u, m.mask, key, home, disp);
            if (at >= 0) {
                slots[at].x = __float_as_uint(mu[0]);
                slots[at].y = __float_as_uint(mu[1]);
                slots[at].z = __float_as_uint(mu[2]);
                slot_vidx[at] = (int32_t)v;
            }
        }
        if (at >= 0) {
            icov8[2 * at] = make_float4(c[0], c[1], c[2], c[3]);
            icov8[2 * at + 1] = make_float4(c[4], c[5], 0.f, 0.f);
        } else {
            atomicOr(status, ST_HASH_FULL);
        }
    }
    // the largest displacement: an atomic only where it grows (one per warp queued at the
    // counter's L2 slice: 90k atomics, 0.5 ms of the 50M-point build)
    disp = __reduce_max_sync(0xffffffffu, disp);
    if ((threadIdx.x & 31u) == 0 && disp > *(volatile uint32_t*)max_probe)
        atomicMax(max_probe, disp);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nv * 9; i += VC) {
        cov[9 * (size_t)v0 + i] = o_cov[i];
        icov[9 * (size_t)v0 + i] = o_icov[i];
    }
    for (uint32_t i = threadIdx.x; i < nv * 3; i += VC) coord[3 * (size_t)v0 + i] = o_coord[i];
}

// Neighbourhood masks (layout in MapView::nmask). Bit 9 (dx + 1) + 3 (dy + 1) + (dz + 1) of a
// cell's mask (or octant's) stands for the voxel in cell + d. It is set only where that voxel's
// centroid can pass the radius test from some point of the cell (of the octant): its distance
// to the cell's (octant's) box is at most the radius, widened by 1e-5 of it and by 1e-6 cell
// widths per cell of distance from the origin (the f32 rounding of a point's cell and octant
// and of the f32 distance test). A cleared bit names a neighbour no point there accepts, so
// neighbour lists are those of the full 27-cell search. On the 5M-point 400 m map at 2 m a scan
// point tests 16.3 candidates with one mask per cell and 9.0 with octant masks, of which it
// accepts 5.45.

// Distance along an axis from a voxel's centroid mu (in cell c of that axis) to the box of the
// cell at offset -d (dk = d + 1): h = 0 the lower half, 1 the upper half, or (whole) the cell
__device__ __forceinline__ float mask_gap(float mu, int32_t c, float res, uint32_t dk, uint32_t h,
                                          bool whole) {
    const float half = 0.5f * res;
    const float lo = fmaxf(mu - (float)c * res, 0.f);           // above the voxel's cell floor
    const float hi = fmaxf(((float)c + 1.f) * res - mu, 0.f);   // below its ceiling
    if (whole) return dk == 2u ? lo : (dk == 0u ? hi : 0.f);
    if (dk == 2u) return h ? lo : lo + half;  // the cell below the voxel's
    if (dk == 0u) return h ? hi + half : hi;  // the cell above
    return h ? fmaxf(hi - half, 0.f) : fmaxf(lo - half, 0.f);  // its own slab: the other half
}

// Squared limit of the distance test for a voxel in cell c. f32 evaluation: the cell corners
// and gaps carry at most a few ulps of far * res, well inside the 1e-6 far * res widening.
__device__ __forceinline__ float mask_limit2(const int32_t* c, float res) {
    float far = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) far = fmaxf(far, fabsf((float)c[a]) + 2.f);
    const float lim = res * (1.f + 1e-5f) + 1e-6f * far * res;
    return lim * lim;
}

// One mask per cell (m.msh = 0), scattered from the voxels: the voxel in local cell v is
// neighbour d of cell v - d, at grown-box position v - d + 1. One thread per voxel, in Morton
// order, so a warp's atomics fall on neighbouring words; the masks start at zero, and OR is
// order-free. The work goes with the number of voxels: these are the maps whose box is large.
__global__ void __launch_bounds__(128) k_grid_mask(MapView m, const int32_t* __restrict__ coord,
                                                   const float4* __restrict__ mean4,
                                                   uint32_t* __restrict__ nmask) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= m.num_voxels) return;
    const int32_t c[3] = {coord[3 * (size_t)s], coord[3 * (size_t)s + 1],
                          coord[3 * (size_t)s + 2]};
    const uint32_t v[3] = {(uint32_t)(c[0] - m.min_cell[0]), (uint32_t)(c[1] - m.min_cell[1]),
                           (uint32_t)(c[2] - m.min_cell[2])};
    const float4 mv = mean4[s];
    const float lim2 = mask_limit2(c, m.res);
    const uint32_t E1 = m.ext[1] + 2u, E2 = m.ext[2] + 2u;
#pragma unroll 1
    for (uint32_t b = 0; b < 27u; ++b) {
        const uint32_t dx = b / 9u, dy = b / 3u % 3u, dz = b % 3u;
        const float gx = mask_gap(mv.x, c[0], m.res, dx, 0u, true);
        const float gy = mask_gap(mv.y, c[1], m.res, dy, 0u, true);
        const float gz = mask_gap(mv.z, c[2], m.res, dz, 0u, true);
        if (fmaf(gx, gx, fmaf(gy, gy, gz * gz)) > lim2) continue;
        atomicOr(nmask + ((size_t)(v[0] + 2u - dx) * E1 + (v[1] + 2u - dy)) * E2 +
                     (v[2] + 2u - dz),
                 1u << b);
    }
}

// Octant masks (m.msh = 3), gathered: one thread per cell of the grown box tests the voxels of
// its 27 cells against its eight octants and writes the eight words. The boxes are small enough
// (256 MiB of masks), a warp's cells share columns of the grid, and every word is written: no
// atomics (about 70 words a voxel, bound by the L2's atomic rate) and no clear. Bound: the ALU
// (70% busy) on half-empty warps; 56 -> 53 us on the 5M-point map, and the clear saved.
__global__ void __launch_bounds__(128) k_grid_mask_oct(MapView m, uint4* __restrict__ nmask) {
    const uint32_t E1 = m.ext[1] + 2u, E2 = m.ext[2] + 2u;
    const size_t cells = (size_t)(m.ext[0] + 2u) * E1 * E2;
    const size_t u = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= cells) return;
    // local cell + 1 of this cell
    const uint32_t uz = (uint32_t)(u % E2), uy = (uint32_t)(u / E2 % E1),
                   ux = (uint32_t)(u / E2 / E1);
    uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
    for (uint32_t dx = 0; dx < 3u; ++dx) {
        const uint32_t x = ux + dx - 2u;
        if (x >= m.ext[0]) continue;
#pragma unroll
        for (uint32_t dy = 0; dy < 3u; ++dy) {
            const uint32_t y = uy + dy - 2u;
            if (y >= m.ext[1]) continue;
            const float4* const col = m.grid + ((size_t)x * m.ext[1] + y) * m.ext[2];
            float4 e[3];
#pragma unroll
            for (uint32_t dz = 0; dz < 3u; ++dz) {
                const uint32_t z = uz + dz - 2u;
                e[dz] = z < m.ext[2] ? __ldg(col + z)
                                     : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
            }
#pragma unroll
            for (uint32_t dz = 0; dz < 3u; ++dz) {
                if (__float_as_int(e[dz].w) < 0) continue;
                const int32_t c[3] = {(int32_t)x + m.min_cell[0], (int32_t)y + m.min_cell[1],
                                      (int32_t)(uz + dz - 2u) + m.min_cell[2]};
                const float lim2 = mask_limit2(c, m.res);
                float gx[2], gy[2], gz[2];
#pragma unroll
                for (uint32_t h = 0; h < 2u; ++h) {
                    gx[h] = mask_gap(e[dz].x, c[0], m.res, dx, h, false);
                    gy[h] = mask_gap(e[dz].y, c[1], m.res, dy, h, false);
                    gz[h] = mask_gap(e[dz].z, c[2], m.res, dz, h, false);
                }
                const uint32_t bit = 1u << (dx * 9u + dy * 3u + dz);
#pragma unroll
                for (uint32_t o = 0; o < 8u; ++o) {
                    const float x0 = gx[(o >> 2) & 1u], y0 = gy[(o >> 1) & 1u], z0 = gz[o & 1u];
                    if (!(fmaf(x0, x0, fmaf(y0, y0, z0 * z0)) > lim2)) w[o] |= bit;
                }
            }
        }
    }
    nmask[2 * u] = make_uint4(w[0], w[1], w[2], w[3]);
    nmask[2 * u + 1] = make_uint4(w[4], w[5], w[6], w[7]);
}

static uint32_t bit_width(uint32_t x) {
    uint32_t b = 0;
    while (b < 32 && (x >> b)) ++b;
    return b;
}

// Key width of a cell box: bits per axis of (max - min), checked against the key limits.
static int box_bits(const int32_t* mn, const int32_t* mx, uint32_t* bits) {
    for (int a = 0; a < 3; ++a) {
        int64_t range = (int64_t)mx[a] - (int64_t)mn[a];
        if (range > 0x1FFFFF) {
            set_error("map extent exceeds 2^21 voxels along an axis");
            return NDT_ERR_RANGE;
        }
        bits[a] = std::max<uint32_t>(1, bit_width((uint32_t)range));
    }
    if (bits[0] + bits[1] + bits[2] > 31) {
        set_error("map bounding box exceeds 2^31 voxel cells (tile the map)");
        return NDT_ERR_RANGE;
    }
    return 0;
}

// Stages 1-5 of a build: cells and bounds, Morton keys, sort, segments, per-segment
// statistics. Leaves in sc: vals (point indices in key order), seg_starts, seg_rec,
// seg_valid; returns the counts and the cell box in g. The last launches may still run, and a
// wait of theirs may run out: the caller reads *sc.failed before it uses the records.
int build_segments(BuildScratch& sc, const float* d_pts, size_t n, const ndt_config& cfg,
                   cudaStream_t s, SegGeometry& g) {
    int rc = 0;
    if ((rc = dev_reserve(sc.keys_a, n * 8)) || (rc = dev_reserve(sc.vals_a, n * 4)) ||
        (rc = dev_reserve(sc.small, 256)) || (rc = dev_reserve(sc.seg_starts, n * 4 + 4)) ||
        (rc = dev_reserve(sc.seg_valid, n * 4 + 4)) || (rc = dev_reserve(sc.seg_rank, n * 4 + 4)) ||
        (rc = dev_reserve(sc.seg_rec, n * sizeof(SegRec))) || (rc = pin_reserve(sc.host, 256)))
        return rc;
    size_t tmp = std::max(radix_sort_temp_bytes(n), detect_segments_temp_bytes(n));
    tmp = std::max(tmp, sort_bytes(n, SortPlan{1, 8}) + 2 * align_up(n * 4, 256));
    // look-back words of every launch behind it, zeroed together: the number of segments, the
    // sort's passes (at most four of 8 bits), the segment starts, the size sort
    const SortPlan oz = {1, 8};
    const size_t w_sort = 256, w_seg = w_sort + sort_words_bytes(n, SortPlan{4, 8}),
                 w_size = w_seg + lookback_bytes(n), w_end = w_size + sort_words_bytes(n, oz);
    tmp = align_up(tmp, 256);
    if ((rc = dev_reserve(sc.tmp, tmp + w_end))) return rc;
    char* const words = (char*)sc.tmp.p + tmp;
    cudaMemsetAsync(words, 0, w_end, s);
    int32_t* mm = (int32_t*)sc.small.p;
    uint32_t* nseg = (uint32_t*)words;
    sc.failed = nseg + 1;
    int32_t* hmm = (int32_t*)sc.host.p;
    uint32_t* hseg = (uint32_t*)sc.host.p + 16;

    cell_bounds(d_pts, n, cfg.resolution, mm, s);
    cudaMemcpyAsync(hmm, mm, 28, cudaMemcpyDeviceToHost, s);
    if ((rc = cuda_fail(cudaStreamSynchronize(s), "map bounds"))) return rc;
    g.nf = (size_t)(uint32_t)hmm[6];
    if (g.nf == 0) {
        set_error("Target point cloud is empty");
        return NDT_ERR_EMPTY_INPUT;
    }
    for (int a = 0; a < 3; ++a) {
        g.mn[a] = hmm[a];
        g.mx[a] = hmm[3 + a];
    }
    uint32_t bits[3];
    if ((rc = box_bits(g.mn, g.mx, bits))) return rc;
    // workspace of the sorts in front of sc.tmp, their alternate values behind it
    uint32_t* vals = (uint32_t*)sc.vals_a.p;  // ends with the point indices in key order
    const CompactKey ck = compact_key(bits);
    if (n < SP_MAX_PAIRS) {
        const SortPlan o = sort_plan((int)ck.total + (g.nf < n ? 1 : 0));
        uint32_t* k0 = (uint32_t*)sc.keys_a.p;
        uint32_t* k1 = k0 + n;
        uint32_t* v1 = (uint32_t*)((char*)sc.tmp.p + sort_bytes(n, o));
        k_compact_keys<<<ntiles(n), BT, 0, s>>>(d_pts, (uint32_t)n, cfg.resolution,
                                                exact_inverse(cfg.resolution),
                                                ((uintptr_t)d_pts & 15u) == 0, mm, ck, o.width,
                                                k0, (uint32_t*)sc.tmp.p);
        uint32_t *ks, *vs;
        // the last pass writes the values to vals_a: an even number of passes starts there
        uint32_t *va = vals, *vb = v1;
        if (o.passes & 1) std::swap(va, vb);
        if ((rc = sort_positions(k0, va, k1, vb, n, o, true, sc.tmp.p,
                                 look_back(sc, words + w_sort, sc.failed, LB_SORT), &ks, &vs, s)) ||
            (rc = segment_starts(ks, g.nf, (uint32_t*)sc.seg_starts.p, nseg,
                                 look_back(sc, words + w_seg, sc.failed, LB_SEGMENTS), s)))
            return rc;
    } else {
        const uint32_t lv = std::max(bits[0], std::max(bits[1], bits[2]));
        uint64_t* keys = (uint64_t*)sc.keys_a.p;
        k_morton<<<(unsigned)((n + BT - 1) / BT), BT, 0, s>>>(d_pts, n, cfg.resolution, mm, keys,
                                                              vals);
        if ((rc = radix_sort_pairs(keys, vals, n, 0, std::min(64, (int)(3 * lv + 1)), sc.tmp.p,
                                   tmp, s)) ||
            (rc = segment_starts(keys, g.nf, (uint32_t*)sc.seg_starts.p, nseg,
                                 look_back(sc, words + w_seg, sc.failed, LB_SEGMENTS), s)))
            return rc;
    }
    cudaMemcpyAsync(hseg, nseg, 8, cudaMemcpyDeviceToHost, s);
    if ((rc = cuda_fail(cudaStreamSynchronize(s), "segments"))) return rc;
    if (hseg[1]) return look_back_failed();
    g.S = hseg[0];
    // visit order of the segments, largest first (the keys' buffer is free again: the
    // segments are recorded by their starts)
    uint32_t* skeys = (uint32_t*)sc.keys_a.p;
    uint32_t* order = (uint32_t*)sc.seg_rank.p;
    const size_t oz_bytes = sort_bytes(g.S, oz);
    uint32_t* sorted = skeys + g.S;
    uint32_t *kz, *vz;
    k_seg_size_keys<<<(g.S + 255) / 256, 256, 0, s>>>((const uint32_t*)sc.seg_starts.p, g.S,
                                                      (uint32_t)g.nf, skeys);
    if ((rc = sort_positions(skeys, nullptr, sorted, order, g.S, oz, false, sc.tmp.p,
                             look_back(sc, words + w_size, sc.failed, LB_SIZES), &kz, &vz, s)))
        return rc;
    // the large segments' sums behind the sort's workspace: at most nf / WARP_SEG_MIN segments
    // of SegSums, well inside its 8 bytes per point
    SegSums* sums = (SegSums*)((char*)sc.tmp.p + oz_bytes);
    const uint32_t wmax = (uint32_t)std::min<size_t>(g.S, g.nf / WARP_SEG_MIN + 1);
    const unsigned gs = (unsigned)std::min<uint32_t>((wmax + 3) / 4, 64u * (uint32_t)device_sms());
    k_segment_sums<<<gs, 128, 0, s>>>(d_pts, vals, (uint32_t*)sc.seg_starts.p, order, kz,
                                      sc.failed, g.S, (uint32_t)g.nf, cfg.resolution,
                                      cfg.min_points_per_voxel, sums);
    k_voxel_stats<<<(g.S + 127) / 128, 128, 0, s>>>(
        d_pts, vals, (uint32_t*)sc.seg_starts.p, order, kz, sc.failed, sums, g.S, (uint32_t)g.nf,
        cfg.resolution, cfg.min_points_per_voxel, cfg.eigenvalue_ratio, (SegRec*)sc.seg_rec.p,
        (uint32_t*)sc.seg_valid.p);
    return cuda_fail(cudaGetLastError(), "voxel statistics");
}

// Stages 6-7: valid voxels of the S records (in Morton order of their cells) compacted into
// the map's voxel arrays, hash insert, dense cell index and neighbourhood masks.
int finish_map(Map& map, BuildScratch& sc, const SegRec* rec, const uint32_t* valid, uint32_t S,
               const SegGeometry& g, const ndt_config& cfg, uint32_t* d_status, cudaStream_t s) {
    int rc;
    if ((rc = dev_reserve(sc.seg_rank, (size_t)S * 4 + 4)) || (rc = dev_reserve(sc.small, 256)))
        return rc;
    uint32_t* mprobe = (uint32_t*)((char*)sc.small.p + 128);
    uint32_t bits[3];
    if ((rc = box_bits(g.mn, g.mx, bits))) return rc;
    // (the words in front of sc.tmp; *sc.failed and the sum behind it lie beyond)
    cudaMemsetAsync(sc.tmp.p, 0, lookback_bytes(S), s);
    if ((rc = exclusive_scan_zeroed(valid, (uint32_t*)sc.seg_rank.p, S,
                                    look_back(sc, sc.tmp.p, sc.failed, LB_RANKS), s,
                                    sc.failed + 1)) ||
        (rc = pin_reserve(sc.host, 256)))
        return rc;
    uint32_t* hs = (uint32_t*)sc.host.p + 24;
    cudaMemcpyAsync(hs, sc.failed, 8, cudaMemcpyDeviceToHost, s);
    if ((rc = cuda_fail(cudaStreamSynchronize(s), "voxel compaction"))) return rc;
    if (hs[0]) return look_back_failed();
    const uint32_t V = hs[1];
    if (V == 0) {
        set_error("No voxels created from target points (too sparse?)");
        return NDT_ERR_NO_VOXELS;
    }
    uint64_t factor = (uint64_t)std::max(2, cfg.hash_capacity_factor);
    uint64_t cap = 1;
    while (cap < factor * V) cap *= 2;
    if (cap > (1ull << 31)) {
        set_error("hash capacity exceeds 2^31 slots");
        return NDT_ERR_CAPACITY;
    }
    MapView v{};
    v.mask = (uint32_t)(cap - 1);
    v.max_probe = 0;
    uint64_t cells = 1, mcells = 1;
    for (int a = 0; a < 3; ++a) {
        v.min_cell[a] = g.mn[a];
        v.bits[a] = bits[a];
        v.ext[a] = (uint32_t)((int64_t)g.mx[a] - (int64_t)g.mn[a] + 1);
        cells *= v.ext[a];
        mcells *= (uint64_t)v.ext[a] + 2;
    }
    v.res = cfg.resolution;
    v.inv_res = 1.0f / cfg.resolution;
    v.r2 = cfg.resolution * cfg.resolution;
    v.num_voxels = V;
    {
        int ex = 0;
        float fr = frexpf(v.inv_res, &ex);
        v.exact_inv = (fr == 0.5f) ? 1 : 0;
    }
    // dense cell index over the bounding box of the map's cells, when it fits the budget, with
    // octant masks (eight words per cell of the grown box) while they fit theirs, or
    // (NDT_CELL_INDEX_OCTANT) while grid and masks fit the dense index's
    const bool dense =
        cfg.cell_index != NDT_CELL_INDEX_HASH && cells * 16 <= DENSE_GRID_MAX_BYTES;
    const bool oct = dense && (cfg.cell_index == NDT_CELL_INDEX_OCTANT
                                   ? cells * 16 + mcells * 32 <= DENSE_GRID_MAX_BYTES
                                   : mcells * 32 <= OCTANT_MASK_MAX_BYTES);
    v.msh = oct ? 3u : 0u;
    const uint64_t mwords = dense ? mcells << v.msh : 0;
    if ((rc = dev_reserve(map.vox_coord, (size_t)V * 12)) ||
        (rc = dev_reserve(map.vox_mean, (size_t)V * 16)) ||
        (rc = dev_reserve(map.vox_cov, (size_t)V * 36)) ||
        (rc = dev_reserve(map.vox_icov, (size_t)V * 36)) ||
        (rc = dev_reserve(map.vox_count, (size_t)V * 4)) ||
        (rc = dev_reserve(map.slots, cap * (dense ? 4 : 16))) ||
        (rc = dev_reserve(map.icov8, (dense ? (size_t)V : (size_t)cap) * 32)))
        return rc;
    if (dense ? (rc = dev_reserve(map.grid, (size_t)cells * 16)) ||
                    (rc = dev_reserve(map.nmask, (size_t)mwords * 4))
              : (rc = dev_reserve(map.slot_vidx, cap * 4)))
        return rc;
    v.icov8 = (const float*)map.icov8.p;
    cudaMemsetAsync(map.slots.p, 0xFF, cap * (dense ? 4 : 16), s);
    cudaMemsetAsync(mprobe, 0, 4, s);
    v.rmean = (const float4*)(dense ? map.vox_mean.p : map.slots.p);
    if (dense) {
        v.grid = (const float4*)map.grid.p;
        v.nmask = (const uint32_t*)map.nmask.p;
        cudaMemsetAsync(map.grid.p, 0xFF, (size_t)cells * 16, s);
        if (!oct) cudaMemsetAsync(map.nmask.p, 0, (size_t)mwords * 4, s);
    } else {
        v.slots = (const uint4*)map.slots.p;
        v.slot_vidx = (const int32_t*)map.slot_vidx.p;
    }
    k_voxel_compact<<<(S + VC - 1) / VC, VC, 0, s>>>(
        rec, valid, (uint32_t*)sc.seg_rank.p, S, (int32_t*)map.vox_coord.p,
        (float4*)map.vox_mean.p, (float*)map.vox_cov.p, (float*)map.vox_icov.p,
        (uint32_t*)map.vox_count.p, v, (float4*)map.icov8.p, dense ? (float4*)map.grid.p : nullptr,
        (uint32_t*)map.slots.p, (uint4*)map.slots.p, (int32_t*)map.slot_vidx.p, mprobe, d_status);
    if (oct)
        k_grid_mask_oct<<<(unsigned)((mcells + 127) / 128), 128, 0, s>>>(v, (uint4*)map.nmask.p);
    else if (dense)
        k_grid_mask<<<(V + 127) / 128, 128, 0, s>>>(v, (const int32_t*)map.vox_coord.p,
                                                    (const float4*)map.vox_mean.p,
                                                    (uint32_t*)map.nmask.p);
    cudaMemcpyAsync(&hs[2], mprobe, 4, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&hs[3], d_status, 4, cudaMemcpyDeviceToHost, s);
    if ((rc = cuda_fail(cudaStreamSynchronize(s), "hash insert"))) return rc;
    const uint32_t hprobe = hs[2];
    map.status = hs[3];
    v.max_probe = hprobe;
    map.view = v;
    ndt_map_info& info = map.info;
    info.num_points = g.nf;
    info.num_segments = S;
    info.num_voxels = V;
    info.hash_capacity = cap;
    info.max_probe = hprobe;
    for (int a = 0; a < 3; ++a) {
        info.key_bits[a] = bits[a];
        info.min_coord[a] = g.mn[a];
        info.max_coord[a] = g.mx[a];
    }
    info.dense_grid_mib =
        v.grid ? (float)(((double)cells * 16.0 + (double)mwords * 4.0) / (1024.0 * 1024.0)) : 0.f;
    info.masks_per_cell = v.grid ? 1u << v.msh : 0u;
    info.reserved = 0u;
    map.valid = true;
    return 0;
}

// ---------------------------------------------------------------------------------------
// Map tiles: segments built once per tile, merged per commit.
// ---------------------------------------------------------------------------------------
// Keys of every tile's segments for the merged map: compact Morton key of the cell in the
// merged box (the key set_target of the concatenated points would give each of its points);
// the values of the sort are the segments' indices in tile order.
__global__ void k_merge_keys(const TileSegRef* __restrict__ tiles, int nt, uint32_t total,
                             int32_t mn0, int32_t mn1, int32_t mn2, CompactKey ck,
                             uint32_t* __restrict__ keys) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int t = 0;
    while (t + 1 < nt && i >= tiles[t + 1].seg_off) ++t;
    const int32_t* c = tiles[t].rec[i - tiles[t].seg_off].coord;
    const uint32_t q[3] = {(uint32_t)c[0] - (uint32_t)mn0, (uint32_t)c[1] - (uint32_t)mn1,
                           (uint32_t)c[2] - (uint32_t)mn2};
    keys[i] = compact_morton(ck, q);
}

// One thread per cell of the merged map (a group of equal keys: the segments of that cell in
// tile order). A cell held by one tile keeps that tile's record; a cell shared by tiles is
// recomputed from all its points in tile order, then each tile's input order, which is the
// order set_target of the concatenated tiles would visit them in.
__global__ void __launch_bounds__(128) k_merge_groups(
    const TileSegRef* __restrict__ tiles, int nt, const uint32_t* __restrict__ members,
    const uint32_t* __restrict__ gstart, const uint32_t* __restrict__ num_groups,
    const uint32_t* __restrict__ failed, uint32_t n_members, int min_points, float ratio,
    float res, SegRec* __restrict__ grec, uint32_t* __restrict__ gvalid) {
    if (*failed) return;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t G = *num_groups;
    if (g >= G) return;
    const uint32_t m0 = gstart[g], m1 = g + 1 < G ? gstart[g + 1] : n_members;
    auto locate = [&](uint32_t id, int& t, uint32_t& sl) {
        t = 0;
        while (t + 1 < nt && id >= tiles[t + 1].seg_off) ++t;
        sl = id - (uint32_t)tiles[t].seg_off;
    };
    int t;
    uint32_t sl;
    locate(members[m0], t, sl);
    if (m1 - m0 == 1) {
        grec[g] = tiles[t].rec[sl];
        gvalid[g] = tiles[t].valid[sl];
        return;
    }
    SegRec r;
    for (int a = 0; a < 3; ++a) r.coord[a] = tiles[t].rec[sl].coord[a];
    uint32_t cnt = 0;
    for (uint32_t m = m0; m < m1; ++m) {
        locate(members[m], t, sl);
        cnt += tiles[t].rec[sl].count;
    }
    auto each = [&](auto f) {
        for (uint32_t m = m0; m < m1; ++m) {
            int tm;
            uint32_t sm;
            locate(members[m], tm, sm);
            const TileSegRef& T = tiles[tm];
            const uint32_t b = T.starts[sm], e = sm + 1 < T.S ? T.starts[sm + 1] : T.nf;
            for (uint32_t k = b; k < e; ++k) f(T.pts + 3 * (size_t)T.idx[k]);
        }
    };
    locate(members[m0], t, sl);
    const float* first = tiles[t].pts + 3 * (size_t)tiles[t].idx[tiles[t].starts[sl]];
    const bool ok = voxel_stats(each, first, cnt, min_points, ratio, res, r);
    grec[g] = r;
    gvalid[g] = ok ? 1u : 0u;
}

int merge_tiles(Map& map, BuildScratch& sc, const std::vector<TileSegRef>& refs,
                DevBuf& d_refs, const ndt_config& cfg, uint32_t* d_status, cudaStream_t s,
                float* build_ms) {
    SegGeometry g{};
    uint64_t total = 0;
    bool any = false;
    for (const auto& t : refs) {
        if (!t.S) continue;
        for (int a = 0; a < 3; ++a) {
            g.mn[a] = any ? std::min(g.mn[a], t.mn[a]) : t.mn[a];
            g.mx[a] = any ? std::max(g.mx[a], t.mx[a]) : t.mx[a];
        }
        any = true;
        g.nf += t.nf;
        total += t.S;
    }
    if (!any) {
        set_error("Target point cloud is empty");
        return NDT_ERR_EMPTY_INPUT;
    }
    // (the sort indexes with 32 bits, a tile past the end included; the 64-bit keys of builds from
    // SP_MAX_PAIRS points on are a matter of speed)
    if (total >= 0xFFFFFFFFull - TILE) {
        set_error("too many occupied cells in the tiles");
        return NDT_ERR_CAPACITY;
    }
    uint32_t bits[3];
    int rc = box_bits(g.mn, g.mx, bits);
    if (rc) return rc;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    std::vector<TileSegRef> used;
    for (const auto& t : refs)
        if (t.S) used.push_back(t);
    const int nt = (int)used.size();
    const CompactKey ck = compact_key(bits);
    const SortPlan o = sort_plan((int)ck.total);
    const size_t ob = sort_bytes(total, o);
    const size_t w_at = std::max(ob + align_up(total * 4, 256), lookback_bytes(total)),
                 w_seg = 256 + sort_words_bytes(total, o), w_end = w_seg + lookback_bytes(total);
    if ((rc = dev_reserve(d_refs, used.size() * sizeof(TileSegRef))) ||
        (rc = dev_reserve(sc.keys_a, total * 8)) || (rc = dev_reserve(sc.vals_a, total * 4)) ||
        (rc = dev_reserve(sc.small, 256)) || (rc = dev_reserve(sc.seg_starts, total * 4 + 4)) ||
        (rc = dev_reserve(sc.seg_valid, total * 4 + 4)) ||
        (rc = dev_reserve(sc.seg_rec, total * sizeof(SegRec))) ||
        (rc = pin_reserve(sc.host, 256)) ||
        (rc = dev_reserve(sc.tmp, w_at + w_end)))
        return rc;
    char* const words = (char*)sc.tmp.p + w_at;  // number of groups, sort, group starts: zeroed
    cudaMemsetAsync(words, 0, w_end, s);
    cudaMemcpyAsync(d_refs.p, used.data(), used.size() * sizeof(TileSegRef),
                    cudaMemcpyHostToDevice, s);
    uint32_t* keys = (uint32_t*)sc.keys_a.p;
    uint32_t* ngroups = (uint32_t*)words;
    sc.failed = ngroups + 1;
    const TileSegRef* dref = (const TileSegRef*)d_refs.p;
    k_merge_keys<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
        dref, nt, (uint32_t)total, g.mn[0], g.mn[1], g.mn[2], ck, keys);
    uint32_t *ks, *vals;
    if ((rc = sort_positions(keys, (uint32_t*)sc.vals_a.p, keys + total,
                             (uint32_t*)((char*)sc.tmp.p + ob), total, o, false, sc.tmp.p,
                             look_back(sc, words + 256, sc.failed, LB_SORT), &ks, &vals, s)) ||
        (rc = segment_starts(ks, total, (uint32_t*)sc.seg_starts.p, ngroups,
                             look_back(sc, words + w_seg, sc.failed, LB_SEGMENTS), s)))
        return rc;
    k_merge_groups<<<(unsigned)((total + 127) / 128), 128, 0, s>>>(
        dref, nt, vals, (const uint32_t*)sc.seg_starts.p, ngroups, sc.failed, (uint32_t)total,
        cfg.min_points_per_voxel, cfg.eigenvalue_ratio, cfg.resolution, (SegRec*)sc.seg_rec.p,
        (uint32_t*)sc.seg_valid.p);
    uint32_t* hseg = (uint32_t*)sc.host.p + 16;
    cudaMemcpyAsync(hseg, ngroups, 8, cudaMemcpyDeviceToHost, s);
    if ((rc = cuda_fail(cudaStreamSynchronize(s), "tile merge"))) return rc;
    if (hseg[1]) return look_back_failed();
    g.S = hseg[0];
    rc = finish_map(map, sc, (const SegRec*)sc.seg_rec.p, (const uint32_t*)sc.seg_valid.p, g.S,
                    g, cfg, d_status, s);
    cudaEventRecord(e1, s);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (build_ms) *build_ms = ms;
    map.info.build_ms = ms;
    return 0;
}

// A tile's segments, kept with the tile: the outputs of build_segments moved into the tile's
// own buffers (point indices in key order, segment starts, records, validity).
int build_tile_segments(BuildScratch& sc, const float* d_pts, size_t n, const ndt_config& cfg,
                        cudaStream_t s, TileSegs& out, float* ms_out) {
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    SegGeometry g{};
    int rc = build_segments(sc, d_pts, n, cfg, s, g);
    if (rc == NDT_ERR_EMPTY_INPUT) {  // no finite point: the tile adds no cell
        out.geo = SegGeometry{};
        rc = 0;
    } else if (!rc) {
        out.geo = g;
        if ((rc = dev_reserve(out.idx, g.nf * 4)) || (rc = dev_reserve(out.starts, (size_t)g.S * 4)) ||
            (rc = dev_reserve(out.rec, (size_t)g.S * sizeof(SegRec))) ||
            (rc = dev_reserve(out.valid, (size_t)g.S * 4)))
            return rc;
        cudaMemcpyAsync(out.idx.p, sc.vals_a.p, g.nf * 4, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(out.starts.p, sc.seg_starts.p, (size_t)g.S * 4, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(out.rec.p, sc.seg_rec.p, (size_t)g.S * sizeof(SegRec),
                        cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(out.valid.p, sc.seg_valid.p, (size_t)g.S * 4, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync((uint32_t*)sc.host.p + 17, sc.failed, 4, cudaMemcpyDeviceToHost, s);
    }
    cudaEventRecord(e1, s);
    if (!rc) rc = cuda_fail(cudaEventSynchronize(e1), "tile segments");
    if (!rc && out.geo.S && ((const uint32_t*)sc.host.p)[17]) {
        out.geo = SegGeometry{};  // the tile adds no cell: its old segments are overwritten
        rc = look_back_failed();
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (ms_out) *ms_out = ms;
    return rc;
}

int build_map(Map& map, BuildScratch& sc, const float* d_pts, size_t n, const ndt_config& cfg,
              uint32_t* d_status, cudaStream_t s, float* build_ms) {
    if (n == 0) {
        set_error("Target point cloud is empty");
        return NDT_ERR_EMPTY_INPUT;
    }
    if (n >= 0xFFFFFFF0ull) {
        set_error("target point cloud exceeds 2^32 points");
        return NDT_ERR_CAPACITY;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    SegGeometry g{};
    int rc = build_segments(sc, d_pts, n, cfg, s, g);
    if (!rc)
        rc = finish_map(map, sc, (const SegRec*)sc.seg_rec.p, (const uint32_t*)sc.seg_valid.p, g.S,
                        g, cfg, d_status, s);
    cudaEventRecord(e1, s);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (build_ms) *build_ms = ms;
    map.info.build_ms = ms;
    return 0;
}

}  // namespace ndtgb
