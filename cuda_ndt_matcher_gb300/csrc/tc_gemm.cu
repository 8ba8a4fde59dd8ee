// tc_gemm.cu — BF16 GEMM on the 5th-generation tensor cores of sm_103a (tcgen05 + TMA).
//
//   D[M x N] (f32) = A B^T over K,  A[m][k], B[n][k] in bf16
//
// Each operand is row-major either with K contiguous ([rows x K], "K-major") or with its rows
// contiguous ([K x rows], "MN-major"): the tensor cores read both from the swizzled tiles that a
// TMA box leaves, so the proposal network keeps no transposed copy of its weights, activations
// or gradients (such copies of the 36,864-wide input and of every weight cost a training step
// about 60 us).
//
// One CTA of eight warps computes a tile of D of 128 MT x BN:
//   warp 0, lane 0  TMA producer: a 128 MT x 64 tile of A and a BN x 64 tile of B per stage
//                   (128-byte swizzle) into a shared-memory ring, completion counted on a "full"
//                   mbarrier;
//   warp 1, lane 0  MMA issuer: per stage 4 MT tcgen05.mma.kind::f16 (M 128, N BN, K 16) into MT
//                   times BN f32 columns of tensor memory; tcgen05.commit arrives on the
//                   stage's "empty" mbarrier when those MMAs are done;
//   warps 0-7       epilogue: tcgen05.ld of 32 accumulator rows and half the columns each, then
//                   a plain store or the network's elementwise step (GemmEpilogue).
// A second kernel (k_gemm_adam) updates weights from the accumulator of their gradient.
// The tile's size is chosen by the number of tiles (gemm_bf16). With one CTA of four warps an SM
// and 128 x 128 tiles throughout, the hidden layers' products were bound by their epilogues (8.6 us
// for 1024 x 512 x 512, now 6.0) and the large ones by operand traffic with nothing beside the
// epilogue (4096^3 172 us, now 93; 1024 x 512 x 36864 73, now 39).
// Every mbarrier wait is bounded (about one second of the global timer); on timeout the CTA
// records an error code in *err, stops issuing work and frees its tensor memory.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "ndt_internal.h"

namespace ndtgb {

__device__ __forceinline__ float gelu_tanh(float z) {  // tanh approximation of GELU
    const float k = 0.7978845608f;                      // sqrt(2 / pi)
    const float u = k * (z + 0.044715f * z * z * z);
    return 0.5f * z * (1.f + tanhf(u));
}
__device__ __forceinline__ float gelu_tanh_grad(float z) {
    const float k = 0.7978845608f;
    const float u = k * (z + 0.044715f * z * z * z);
    const float t = tanhf(u);
    return 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * k * (1.f + 3.f * 0.044715f * z * z);
}


constexpr int GB_M = 128, GB_K = 64, GB_THREADS = 256;
constexpr int GB_ATILE = GB_M * GB_K * 2;  // 16 KB
__host__ __device__ constexpr int gb_stage_bytes(int bn, int mt) {  // a tile of 128 mt x bn
    return mt * GB_ATILE + bn * GB_K * 2;
}
__host__ __device__ constexpr int gb_smem(int bn, int mt, int st) {  // with alignment
    return st * gb_stage_bytes(bn, mt) + 1024;
}
// Tiles (us at M, N, K, split in 16 where K = 36,864; L2 flushed between launches):
//   256 x 256 for a plain store from GB_SQUARE_TILES on: half the operand traffic of 128 x 128.
//     1024, 512, 36864: 39 and 46; 640, 512, 36864 (96 tiles): 36 and 43; 512, 512, 36864 (64):
//     35 and 28; 4096^3: 93 (1.47 PFLOP/s) and 119. One CTA to an SM.
//   128 x 128, two CTAs to an SM, from a tile per SM on. 640, 512, 36864: 43, as 128
//     x 64 50; 512, 36864, 1024: 61 and 77.
//   128 x 128 with a deep ring for few tiles and a K beyond GB_DEEP_K. 256, 512, 36864: 19.1,
//     as 128 x 64 21.6.
//   128 x 64 else: twice the CTAs, half the epilogue. 1024, 512, 512: 6.0, deep 6.7.
constexpr int GB_SQUARE_TILES = 96, GB_DEEP_K = 2048;
constexpr uint64_t GB_WAIT_NS = 1000000000ull;  // bounded waits: 1 s
constexpr uint32_t GB_NAP_NS = 20000;           // a waiting thread sleeps up to this long a try

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t gb_now() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for the given phase parity of an mbarrier; false (and *err |= code) on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* err,
                                          uint32_t code) {
    const uint32_t a = smem_u32(bar);
    const uint64_t t0 = gb_now();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity), "r"(GB_NAP_NS)
            : "memory");
        if (ok) return true;
        if (gb_now() - t0 > GB_WAIT_NS) {
            atomicOr(err, code);
            return false;
        }
    }
}

// Operand tile in shared memory, 128-byte swizzle (the layout a TMA box of 64 bf16 columns with
// CU_TENSOR_MAP_SWIZZLE_128B writes): rows of 128 B in 8-row, 1024-byte atoms.
// Descriptor fields: start address >> 4 (bits 0-13), leading-dimension offset >> 4 (16-29),
// stride-dimension offset >> 4 (32-45), descriptor version 1 (46-47), base offset 0 (49-51: atoms
// 1024-B aligned), layout type 2 = 128-byte swizzle (61-63).
// K-major tile: a box of all rows; stride offset 1024 B between 8-row groups, leading offset
// unused; the MMA's 16 of K are 32 bytes along the rows.
// MN-major tile: boxes of 64 rows of K by 64 elements, one per 64 of M or N, 8 KB apart (leading
// offset); stride offset 1024 B between groups of 8 of K; 16 of K are 2048 bytes.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr, int mn_major) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(mn_major ? 8192 >> 4 : 1) << 16) |
           ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of tcgen05.mma.kind::f16: D f32 (bits 4-5 = 1), A and B bf16
// (bits 7-9 = 1, 10-12 = 1), A, B MN-major (bits 15, 16), N >> 3 (bits 17-22), M >> 4
// (bits 24-28).
__device__ __forceinline__ uint32_t mma_idesc_bf16(int m, int n, int a_mn, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// 32 consecutive accumulator columns from column `c` of the warp's 32 rows (one lane, one row)
__device__ __forceinline__ void tmem_load32(uint32_t ta, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, "
        "%9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, "
        "%25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(ta));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Epilogue of 32 rows by 32 columns of the accumulator (a warp's rows row0.., columns col0..; `r`
// holds one row a lane): through the warp's shared-memory square, so that global accesses are 16
// bytes a lane and eight lanes a row (128-byte lines; a lane per row wrote half sectors, 32 lines
// an instruction: 10 us of the 47 of the input layer's product). Columns beyond N, and all columns
// where N is no multiple of 4, go one by one.
constexpr int GB_SQ_PITCH = 36;
template <bool FUSED>
__device__ __forceinline__ void epilogue(const GemmEpilogue& epi, const uint32_t* r, float* sq,
                                         float* D, int ldd, int M, int N, int row0, int col0,
                                         int lane) {
#pragma unroll
    for (int q = 0; q < 32; q += 4)
        *reinterpret_cast<float4*>(sq + lane * GB_SQ_PITCH + q) =
            make_float4(__uint_as_float(r[q]), __uint_as_float(r[q + 1]),
                        __uint_as_float(r[q + 2]), __uint_as_float(r[q + 3]));
    __syncwarp();
    const int c = 4 * (lane & 7), n = col0 + c;
    const bool vec = n + 4 <= N && (!FUSED || (N & 3) == 0);
    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (FUSED && vec && epi.mode != GEMM_EPI_GELU_BACK)
        b4 = *reinterpret_cast<const float4*>(epi.bias + n);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rr = 4 * i + (lane >> 3), row = row0 + rr;
        if (row >= M || n >= N) continue;
        const float4 a = *reinterpret_cast<const float4*>(sq + rr * GB_SQ_PITCH + c);
        float o[4] = {a.x, a.y, a.z, a.w}, x[4];
        if (FUSED) {
            float p[4] = {b4.x, b4.y, b4.z, b4.w};
            const bool back = epi.mode == GEMM_EPI_GELU_BACK;
            const float* const src = back ? epi.zin + (size_t)row * N + n : epi.bias + n;
            if (vec && back) {
                const float4 z = *reinterpret_cast<const float4*>(src);
                p[0] = z.x, p[1] = z.y, p[2] = z.z, p[3] = z.w;
            } else if (!vec) {
                for (int u = 0; u < 4; ++u) p[u] = n + u < N ? src[u] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                o[u] = back ? o[u] * gelu_tanh_grad(p[u]) : o[u] + p[u];
                x[u] = epi.mode == GEMM_EPI_BIAS_GELU ? gelu_tanh(o[u]) : o[u];
            }
        }
        float* const dst = D + (size_t)row * ldd + n;
        __nv_bfloat16* const xd = FUSED && epi.x ? epi.x + (size_t)row * N + n : nullptr;
        if (vec) {
            *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
            if (FUSED && xd) {
                __nv_bfloat162 h[2] = {__floats2bfloat162_rn(x[0], x[1]),
                                       __floats2bfloat162_rn(x[2], x[3])};
                *reinterpret_cast<uint2*>(xd) = *reinterpret_cast<uint2*>(h);
            }
        } else {
            for (int u = 0; u < 4 && n + u < N; ++u) {
                dst[u] = o[u];
                if (FUSED && xd) xd[u] = __float2bfloat16(x[u]);
            }
        }
    }
    __syncwarp();  // the square may be overwritten
}

// The TMA boxes of one k-block of a tile, counted on the mbarrier `fb`. Innermost coordinates
// are multiples of 64 bf16 = 128 B.
template <int BN, int MT>
__device__ __forceinline__ void load_stage(uint64_t pa, uint64_t pb, uint32_t sa, uint32_t fb,
                                           int m0, int n0, int k, int a_mn, int b_mn) {
    auto load = [&](uint32_t dst, uint64_t map, int x, int y) {
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::"
            "complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
            "l"(map), "r"(x), "r"(y), "r"(fb)
            : "memory");
    };
    const uint32_t sb = sa + MT * GB_ATILE;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb),
                 "r"(gb_stage_bytes(BN, MT))
                 : "memory");
    if (a_mn) {
        for (int j = 0; j < 2 * MT; ++j) load(sa + 8192 * j, pa, m0 + 64 * j, k);
    } else {
        for (int j = 0; j < MT; ++j) load(sa + GB_ATILE * j, pa, k, m0 + GB_M * j);
    }
    if (b_mn) {
        for (int j = 0; j < BN / 64; ++j) load(sb + 8192 * j, pb, n0 + 64 * j, k);
    } else {
        load(sb, pb, k, n0);
    }
}

// The products of one k-block into the accumulator at `tmem` (MT times BN columns); the
// accumulator starts from zero with `first`
template <int BN, int MT>
__device__ __forceinline__ void mma_stage(uint32_t tmem, uint32_t sa, uint32_t idesc, int a_mn,
                                          int b_mn, bool first) {
    const uint32_t sb = sa + MT * GB_ATILE;
    const uint32_t ka = a_mn ? 2048 : 32, kbytes = b_mn ? 2048 : 32;  // 16 of K
#pragma unroll
    for (int k = 0; k < GB_K / 16; ++k) {
        const uint64_t bd = sw128_desc(sb + kbytes * k, b_mn);
        const uint32_t acc = !(first && k == 0) ? 1u : 0u;
#pragma unroll
        for (int j = 0; j < MT; ++j) {
            const uint64_t ad = sw128_desc(sa + GB_ATILE * j + ka * k, a_mn);
            asm volatile(
                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
                    tmem + (uint32_t)(j * BN)),
                "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                : "memory");
        }
    }
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
}

enum { GB_STORE, GB_FUSED };

template <int BN, int MT, int ST, int EPI>
__global__ void __launch_bounds__(GB_THREADS, gb_smem(BN, MT, ST) < 110 * 1024 ? 2 : 1)
    k_gemm_bf16(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                float* __restrict__ D, int M, int N, int K, int a_mn, int b_mn, int ldd,
                int splits, size_t split_stride, uint32_t* err, const GemmEpilogue epi) {
    constexpr int SB = gb_stage_bytes(BN, MT);
    extern __shared__ __align__(1024) uint8_t gb_smem_raw[];
    __shared__ __align__(8) uint64_t full[ST], empty[ST], done;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    uint8_t* smem = (uint8_t*)(((uintptr_t)gb_smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * GB_M * MT, n0 = blockIdx.x * BN;
    // split-K: blockIdx.z takes k-blocks [kb0, kb0 + nk) and writes its own f32 partial of D
    const int nk_all = K / GB_K, z = (int)blockIdx.z;
    const int kb0 = (int)((long long)nk_all * z / splits);
    const int nk = (int)((long long)nk_all * (z + 1) / splits) - kb0;
    D += (size_t)z * split_stride;

    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&full[s]);
            mbar_init(&empty[s]);
        }
        mbar_init(&done);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        abort_flag = 0;
    }
    if (warp == 1) {  // MT BN f32 columns x 128 lanes of tensor memory for the accumulator
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_base)),
                     "r"(MT * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    if (warp == 0 && lane == 0) {  // TMA producer
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % ST;
            if (kb >= ST && !mbar_wait(&empty[s], ((kb / ST) - 1) & 1, err, 1u)) {
                abort_flag = 1;
                break;
            }
            if (*(volatile int*)&abort_flag) break;
            load_stage<BN, MT>((uint64_t)&tmA, (uint64_t)&tmB, smem_u32(smem + s * SB),
                               smem_u32(&full[s]), m0, n0, (kb0 + kb) * GB_K, a_mn, b_mn);
        }
    } else if (warp == 1 && lane == 0) {  // MMA issuer
        const uint32_t idesc = mma_idesc_bf16(GB_M, BN, a_mn, b_mn);
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % ST;
            if (!mbar_wait(&full[s], (kb / ST) & 1, err, 2u)) {
                abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            mma_stage<BN, MT>(tmem, smem_u32(smem + s * SB), idesc, a_mn, b_mn, kb == 0);
            mma_commit(&empty[s]);
        }
        mma_commit(&done);  // accumulator complete (or abandoned): the epilogue waits for it
    }
    __syncwarp();
    // epilogue: warps w and w + 4 read accumulator lanes 32w..32w+31 (rows of the tile), half of
    // the columns each
    // (one warp polls, the others sleep at the barrier: eight polling warps slowed the producer and
    // the MMA issuer by 12%)
    if (warp == 0 && !mbar_wait(&done, 0, err, 4u)) abort_flag = 1;
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool ok = !*(volatile int*)&abort_flag;
    const int quad = warp & 3, cbeg = (warp >> 2) * (BN / 2);
    // (the ring is idle: every load has arrived and every MMA has read it)
    float* const square = reinterpret_cast<float*>(smem) + warp * 32 * GB_SQ_PITCH;
    if (ok) {
#pragma unroll 1
        for (int i = 0; i < MT * (BN / 64); ++i) {
            const int j = i / (BN / 64), c = cbeg + 32 * (i % (BN / 64));
            uint32_t r[32];
            tmem_load32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(j * BN + c), r);
            epilogue<EPI == GB_FUSED>(epi, r, square, D, ldd, M, N, m0 + j * GB_M + quad * 32,
                                      n0 + c, lane);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(MT * BN));
    }
}

// ------------------------------------------------------------------------------------
// Weight gradient and Adam update
//
// acc[M x N] = A B^T is the gradient of a weight [M x N]; its f32 master, two moments and bf16
// copy are updated from the accumulator, which never reaches memory. The update moves 26 bytes a
// weight, far more than the products' operands, so it is what must not pause: one persistent CTA
// per SM takes tiles of all layers, and its producer and MMA warps run a tile ahead (two
// accumulators in tensor memory) of the 28 warps that update. These take a tile through shared
// memory to have a warp per row and a float4 per lane (whole 512-byte rows: 128-byte pieces
// by 32 x 32 squares took 146 us), a row's loads ahead of the row they work on. The hidden layers'
// 52 tiles fill the last round of the input layer's 1,152.
// For a step of 19.7M weights: 126 us, where the product, its store, and a sweep over the gradient
// and the state took 94 + 89. The products alone take 55 us, the update alone 105 (DRAM at
// 4.7 TB/s; a plain sweep reaches 6.4): rows of a tile are 147 KB apart.
// ------------------------------------------------------------------------------------
constexpr int GA_N = 128, GA_STAGES = 4, GA_UPD = 896;    // updating threads
constexpr int GA_WP = GA_UPD / 32, GA_THREADS = GA_UPD + 64;  // producer warp; the next: MMA
constexpr int GA_PITCH = GA_N + 4;  // floats: accesses by row meet no bank conflicts
constexpr int GA_SB = gb_stage_bytes(GA_N, 1);
constexpr int GA_SMEM = GA_STAGES * GA_SB + GB_M * GA_PITCH * 4 + 1024;

struct AdamLayer {
    CUtensorMap a, b;
    AdamState st;
    int m, n, start;  // weight [m x n]; its first tile
};
struct AdamLayers {
    AdamLayer l[GEMM_ADAM_MAX];
    int layers, tiles, k;
};

__device__ __forceinline__ void update_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(GA_UPD) : "memory");
}
// the layer of tile t and the tile's origin (tiles that share columns follow one another)
__device__ __forceinline__ const AdamLayer& adam_tile(const AdamLayers& p, int t, int& m0,
                                                      int& n0) {
    int l = 0;
    while (l + 1 < p.layers && t >= p.l[l + 1].start) ++l;
    const int tm = (p.l[l].m + GB_M - 1) / GB_M, i = t - p.l[l].start;
    m0 = i % tm * GB_M;
    n0 = i / tm * GA_N;
    return p.l[l];
}

__global__ void __launch_bounds__(GA_THREADS, 1)
    k_gemm_adam(const __grid_constant__ AdamLayers p, uint32_t* err) {
    constexpr int ST = GA_STAGES;
    extern __shared__ __align__(1024) uint8_t gb_smem_raw[];
    __shared__ __align__(8) uint64_t full[ST], empty[ST], tfull[2], tempty[2];
    __shared__ uint32_t tmem_base;
    __shared__ int stop_load, stop_update;
    __shared__ float s_adam[2];
    uint8_t* smem = (uint8_t*)(((uintptr_t)gb_smem_raw + 1023) & ~(uintptr_t)1023);
    float* const tile = reinterpret_cast<float*>(smem + ST * GA_SB);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nk = p.k / GB_K;
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&full[s]);
            mbar_init(&empty[s]);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull[s]);
            mbar_init(&tempty[s]);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        stop_load = stop_update = 0;
        adam_corrections(p.l[0].st, s_adam);  // (the layers share step count and rates)
    }
    if (warp == GA_WP + 1) {  // two accumulators of GA_N f32 columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_base)),
                     "r"(2 * GA_N));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    if (warp == GA_WP) {
        if (lane == 0) {
            int g = 0;  // k-blocks so far
            bool on = true;
            for (int t = blockIdx.x; t < p.tiles && on; t += gridDim.x) {
                int m0, n0;
                const AdamLayer& L = adam_tile(p, t, m0, n0);
                for (int kb = 0; kb < nk && on; ++kb, ++g) {
                    const int s = g % ST;
                    on = (g < ST || mbar_wait(&empty[s], ((g / ST) - 1) & 1, err, 1u)) &&
                         !*(volatile int*)&stop_load;
                    if (on)
                        load_stage<GA_N, 1>((uint64_t)&L.a, (uint64_t)&L.b,
                                            smem_u32(smem + s * GA_SB), smem_u32(&full[s]), m0, n0,
                                            kb * GB_K, 1, 1);
                }
            }
        }
    } else if (warp == GA_WP + 1) {
        if (lane == 0) {
            const uint32_t idesc = mma_idesc_bf16(GB_M, GA_N, 1, 1);
            int g = 0, i = 0;
            bool on = true;
            for (int t = blockIdx.x; t < p.tiles && on; t += gridDim.x, ++i) {
                on = i < 2 || mbar_wait(&tempty[i & 1], ((i >> 1) - 1) & 1, err, 8u);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < nk && on; ++kb, ++g) {
                    const int s = g % ST;
                    if (!(on = mbar_wait(&full[s], (g / ST) & 1, err, 2u))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    mma_stage<GA_N, 1>(tmem + (uint32_t)((i & 1) * GA_N),
                                       smem_u32(smem + s * GA_SB), idesc, 1, 1, kb == 0);
                    mma_commit(&empty[s]);
                }
                if (on) mma_commit(&tfull[i & 1]);
            }
            if (!on) *(volatile int*)&stop_load = 1;  // (the update's wait for the tile runs out)
        }
    } else {
        constexpr int UA = 1, NB = (GB_M + UA * GA_WP - 1) / (UA * GA_WP);  // rows of a warp at a time; times a tile
        const int quad = warp & 3, cbeg = (warp >> 2) * (GA_N / 4);
        const float lc1 = s_adam[0], ic2 = s_adam[1];
        int i = 0;
        for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++i) {
            int m0, n0;
            const AdamLayer& L = adam_tile(p, t, m0, n0);
            const int col = n0 + 4 * lane, N = L.n;
            const int rows = col < N ? min(GB_M, L.m - m0) : 0;
            const size_t base = (size_t)(m0 + warp) * N + col, hop = (size_t)GA_WP * N;
            float* const pm = L.st.m + base;
            float* const pv = L.st.v + base;
            float* const pw = L.st.w + base;
            __nv_bfloat16* const pb = L.st.wb + base;
            float4 m4[2][UA], v4[2][UA], w4[2][UA];
            auto fetch = [&](int b) {
#pragma unroll
                for (int u = 0; u < UA; ++u) {
                    const int k = b * UA + u;
                    if (warp + k * GA_WP >= rows) continue;
                    m4[b & 1][u] = __ldcg(reinterpret_cast<const float4*>(pm + k * hop));
                    v4[b & 1][u] = __ldcg(reinterpret_cast<const float4*>(pv + k * hop));
                    w4[b & 1][u] = __ldcg(reinterpret_cast<const float4*>(pw + k * hop));
                }
            };
            fetch(0);
            if (!mbar_wait(&tfull[i & 1], (i >> 1) & 1, err, 4u)) *(volatile int*)&stop_update = 1;
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (warp < 16) {  // four warps a quadrant of rows, 32 columns each
                uint32_t r[32];
                tmem_load32(tmem + ((uint32_t)(quad * 32) << 16) +
                                (uint32_t)((i & 1) * GA_N + cbeg), r);
#pragma unroll
                for (int q = 0; q < 32; q += 4)
                    *reinterpret_cast<float4*>(tile + (quad * 32 + lane) * GA_PITCH + cbeg + q) =
                        make_float4(__uint_as_float(r[q]), __uint_as_float(r[q + 1]),
                                    __uint_as_float(r[q + 2]), __uint_as_float(r[q + 3]));
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            update_sync();  // the tile is in shared memory, the accumulator free
            // written before this barrier only, by warps that wait: the same for all of them
            if (*(volatile int*)&stop_update) break;
            if (tid == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                                 smem_u32(&tempty[i & 1]))
                             : "memory");
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                if (b + 1 < NB) fetch(b + 1);
#pragma unroll
                for (int u = 0; u < UA; ++u) {
                    const int k = b * UA + u;
                    if (warp + k * GA_WP >= rows) continue;
                    const float4 g4 = *reinterpret_cast<const float4*>(
                        tile + (warp + k * GA_WP) * GA_PITCH + 4 * lane);
                    float4 &m = m4[b & 1][u], &v = v4[b & 1][u], &w = w4[b & 1][u];
                    adam_update(L.st, g4.x, m.x, v.x, w.x, lc1, ic2);
                    adam_update(L.st, g4.y, m.y, v.y, w.y, lc1, ic2);
                    adam_update(L.st, g4.z, m.z, v.z, w.z, lc1, ic2);
                    adam_update(L.st, g4.w, m.w, v.w, w.w, lc1, ic2);
                    __stcg(reinterpret_cast<float4*>(pm + k * hop), m);
                    __stcg(reinterpret_cast<float4*>(pv + k * hop), v);
                    __stcg(reinterpret_cast<float4*>(pw + k * hop), w);
                    __nv_bfloat162 h[2] = {__floats2bfloat162_rn(w.x, w.y),
                                           __floats2bfloat162_rn(w.z, w.w)};
                    *reinterpret_cast<uint2*>(pb + k * hop) = *reinterpret_cast<uint2*>(h);
                }
            }
            update_sync();  // the tile has been read
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == GA_WP + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(2 * GA_N));
    }
}

// ------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                             cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// 2-D bf16 row-major [rows x cols] tensor map with boxes of `box_rows` x 64 and 128-byte swizzle.
static int make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols,
                    uint32_t box_rows) {
    auto enc = tensor_map_encoder();
    if (!enc) {
        set_error("cuTensorMapEncodeTiled unavailable");
        return NDT_ERR_DEVICE;
    }
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                     strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    return 0;
}

// Tensor maps of the operands for tiles of BN columns. MN-major: boxes of 64 of K by 64; K-major:
// boxes of 64 of K by a tile's rows.
template <int BN>
static int make_maps(CUtensorMap* ta, CUtensorMap* tb, const GemmOperand& A, const GemmOperand& B,
                     int M, int N, int K) {
    int rc = A.mn_major ? make_map(ta, A.p, (uint64_t)K, (uint64_t)M, GB_K)
                        : make_map(ta, A.p, (uint64_t)M, (uint64_t)K, GB_M);
    if (rc) return rc;
    return B.mn_major ? make_map(tb, B.p, (uint64_t)K, (uint64_t)N, GB_K)
                      : make_map(tb, B.p, (uint64_t)N, (uint64_t)K, BN);
}

template <int BN, int MT, int ST, int EPI>
static int launch_gemm(const GemmOperand& A, const GemmOperand& B, float* D, int M, int N, int K,
                       int ldd, uint32_t* d_err, cudaStream_t s, int splits,
                       const GemmEpilogue& e) {
    CUtensorMap ta, tb;
    int rc = make_maps<BN>(&ta, &tb, A, B, M, N, K);
    if (rc) return rc;
    auto kern = k_gemm_bf16<BN, MT, ST, EPI>;
    cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          gb_smem(BN, MT, ST));
    if (ce != cudaSuccess) return cuda_fail(ce, "gemm launch");
    dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + GB_M * MT - 1) / (GB_M * MT)),
              (unsigned)splits);
    kern<<<grid, GB_THREADS, gb_smem(BN, MT, ST), s>>>(ta, tb, D, M, N, K, A.mn_major, B.mn_major,
                                                   ldd, splits, (size_t)M * ldd, d_err, e);
    return cuda_fail(cudaGetLastError(), "gemm launch");
}

// splits > 1: split-K, partial products of k-range z at D + z * M * ldd (the caller sums)
int gemm_bf16(GemmOperand A, GemmOperand B, float* D, int M, int N, int K, int ldd,
              uint32_t* d_err, cudaStream_t s, int splits, const GemmEpilogue* epi) {
    if (M <= 0 || N <= 0 || K <= 0 || K % GB_K || ldd < N || ((uintptr_t)A.p & 15) ||
        ((uintptr_t)B.p & 15) || ((uintptr_t)D & 15) || (ldd & 3) || splits < 1 ||
        splits > K / GB_K || splits > 65535 || (A.mn_major && M % 64) || (B.mn_major && N % 64)) {
        set_error("gemm: K must be a multiple of 64, operands 16-byte aligned, ldd >= N, "
                  "1 <= splits <= K / 64");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    GemmEpilogue e{};
    if (epi) e = *epi;
    if (e.mode != GEMM_EPI_STORE &&
        (splits != 1 || ldd != N || ((uintptr_t)e.x & 15) ||
         (e.mode == GEMM_EPI_GELU_BACK ? !e.zin : !e.bias))) {
        set_error("gemm: a fused epilogue needs splits = 1, ldd = N, its bias (or input) and "
                  "16-byte aligned outputs");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    auto tiles = [&](int m, int n) {
        return (long long)((M + m - 1) / m) * ((N + n - 1) / n) * splits;
    };
    const bool wide = tiles(128, 128) >= device_sms(), deep = K / splits > GB_DEEP_K;
    if (e.mode == GEMM_EPI_STORE) {
        if (tiles(256, 256) >= GB_SQUARE_TILES)
            return launch_gemm<256, 2, 3, GB_STORE>(A, B, D, M, N, K, ldd, d_err, s, splits, e);
        return wide   ? launch_gemm<128, 1, 3, GB_STORE>(A, B, D, M, N, K, ldd, d_err, s, splits, e)
               : deep ? launch_gemm<128, 1, 6, GB_STORE>(A, B, D, M, N, K, ldd, d_err, s, splits, e)
                      : launch_gemm<64, 1, 4, GB_STORE>(A, B, D, M, N, K, ldd, d_err, s, splits, e);
    }
    return wide   ? launch_gemm<128, 1, 3, GB_FUSED>(A, B, D, M, N, K, ldd, d_err, s, splits, e)
           : deep ? launch_gemm<128, 1, 6, GB_FUSED>(A, B, D, M, N, K, ldd, d_err, s, splits, e)
                  : launch_gemm<64, 1, 4, GB_FUSED>(A, B, D, M, N, K, ldd, d_err, s, splits, e);
}

// One Adam step of the weights w[i] = [m x n] whose gradients are A B^T over k samples, A [k x m]
// and B [k x n] (MN-major).
int gemm_adam(const GemmAdam* w, int count, int k, uint32_t* d_err, cudaStream_t s) {
    AdamLayers p;
    if (count < 1 || count > GEMM_ADAM_MAX || k <= 0 || k % GB_K) {
        set_error("gemm: K must be a multiple of 64");
        return NDT_ERR_INVALID_ARGUMENT;
    }
    p.layers = count;
    p.k = k;
    p.tiles = 0;
    for (int i = 0; i < count; ++i) {
        const GemmAdam& g = w[i];
        if (g.m <= 0 || g.n <= 0 || g.m % 64 || g.n % 64 || ((uintptr_t)g.a & 15) ||
            ((uintptr_t)g.b & 15)) {
            set_error("gemm: weights must be multiples of 64, operands 16-byte aligned");
            return NDT_ERR_INVALID_ARGUMENT;
        }
        AdamLayer& l = p.l[i];
        int rc = make_maps<GA_N>(&l.a, &l.b, {g.a, 1}, {g.b, 1}, g.m, g.n, k);
        if (rc) return rc;
        l.st = g.st;
        l.m = g.m;
        l.n = g.n;
        l.start = p.tiles;
        const long long t = (long long)((g.m + GB_M - 1) / GB_M) * ((g.n + GA_N - 1) / GA_N);
        if (p.tiles + t > 0x3FFFFFFFll) {
            set_error("gemm: too many tiles");
            return NDT_ERR_CAPACITY;
        }
        p.tiles += (int)t;
    }
    cudaError_t e = cudaFuncSetAttribute(k_gemm_adam, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         GA_SMEM);
    if (e != cudaSuccess) return cuda_fail(e, "gemm launch");
    k_gemm_adam<<<std::min(p.tiles, device_sms()), GA_THREADS, GA_SMEM, s>>>(p, d_err);
    return cuda_fail(cudaGetLastError(), "gemm launch");
}

// error word of the standalone entry point (device global, no allocation)
static __device__ uint32_t g_gemm_err;

}  // namespace ndtgb

extern "C" int ndt_gemm_bf16(const void* d_a, const void* d_b, float* d_d, int32_t m, int32_t n,
                             int32_t k, int32_t splits, void* stream) {
    using namespace ndtgb;
    uint32_t* err = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&err, g_gemm_err);
    if (e != cudaSuccess) return cuda_fail(e, "gemm error word");
    cudaStream_t s = (cudaStream_t)stream;
    cudaMemsetAsync(err, 0, 4, s);
    int rc = gemm_bf16({d_a, 0}, {d_b, 0}, d_d, m, n, k, n, err, s, splits, nullptr);
    if (rc) return rc;
    uint32_t h = 0;
    cudaMemcpyAsync(&h, err, 4, cudaMemcpyDeviceToHost, s);
    if ((rc = cuda_fail(cudaStreamSynchronize(s), "gemm"))) return rc;
    if (h) {
        set_error("gemm: a pipeline wait timed out (code " + std::to_string(h) + ")");
        return NDT_ERR_DEVICE;
    }
    return NDT_OK;
}
