// ndt_score.cu — per-pose scoring and the neighbour query on sm_103a.
//
// k_score: for each (scan, pose) job, every point is transformed (compensated f32: the
// transform as hi/lo pairs, so x = q - mean keeps f32 precision), the voxels whose
// centroid lies within one resolution are found through the 27-cell hash probe (all of
// them: kiddo's `within` set, src/ndt_cuda/src/voxel_grid/search.rs:90-99), and the block
// accumulates
//   NVTL terms : max over those voxels of -d1 exp(-d2/2 x^T C x), for points with >= 1
//                voxel (compute_nvtl_simple, src/ndt_cuda/src/scoring/nvtl.rs:211-260);
//   TP terms   : the sum of the scores and the number of pairs
//                (compute_transform_probability, src/ndt_cuda/src/scoring/metrics.rs:58-121).
// The transform is either given (evaluate_*), or built from an alignment's final pose vector
// with nalgebra's from_euler_angles (Rz*Ry*Rx), the isometry the reference evaluates NVTL on
// after an alignment (src/ndt_cuda/src/optimization/types.rs:156-161, solver.rs:386,424).
// Block partials are added in a fixed order: results are deterministic.
#include <algorithm>

#include "ndt_internal.h"

namespace ndtgb {

constexpr int ST = 128;  // threads per block
constexpr uint32_t SCORE_MAX_PPT = 8;

struct ScorePartial {
    double nvtl_sum;
    double score_sum;
    uint64_t nvtl_count;
    uint64_t ncorr;
};

// Points per thread of a launch over `jobs` jobs of at most max_n points: one while the grid
// is small, so a single scan's points spread over every SM (a 20k-point scan: 157 blocks
// instead of 10; scoring it is one dependent chain of loads per point, 54 -> 16 us), then
// doubled, up to 8, while about four blocks per resident slot (8 an SM) remain: the
// block's set-up and reduction are then paid once per 8 points (filling the slots once, four
// and sixteen times measured 70, 64 and 72 us on 64 scans of 2k-40k points).
static uint32_t score_ppt(uint32_t jobs, uint32_t max_n, int sms) {
    uint32_t ppt = 1;
    while (ppt < SCORE_MAX_PPT &&
           (uint64_t)jobs * (((uint64_t)max_n + ST * 2 * ppt - 1) / (ST * 2 * ppt)) >=
               4ull * 8 * (uint32_t)sms)
        ppt *= 2;
    return ppt;
}

static uint32_t score_blocks(uint32_t jobs, uint32_t max_n, int sms) {
    const uint32_t per = ST * score_ppt(jobs, max_n, sms);
    return std::max<uint32_t>(1u, (uint32_t)(((uint64_t)max_n + per - 1) / per));
}

// Transform of one job (row-major 3x4, FP64) by the lanes of one warp, as hi/lo f32 pairs: the
// given matrix, or nalgebra's from_euler_angles (Rz*Ry*Rx) of an alignment's final pose: three
// lanes take a sine and cosine each (about 1,700 cycles of dependent FP64 apiece), twelve an
// entry each.
__device__ __forceinline__ void job_transform(const ScoreJob& job, const AlignOut* aout,
                                              double* trig, float* Th, float* Tl, int lane) {
    double v = 0.0;
    if (job.pose_src == 1) {
        const double* pose = aout[job.out_index].pose;
        if (lane < 3) {
            double s, c;
            sincos(pose[3 + lane], &s, &c);
            trig[2 * lane] = s;
            trig[2 * lane + 1] = c;
        }
        __syncwarp();
        if (lane < 12) {
            const double sr = trig[0], cr = trig[1], sp = trig[2], cp = trig[3], sy = trig[4],
                         cy = trig[5];
            const int i = lane >> 2, j = lane & 3;
            if (j == 3) {
                v = pose[i];
            } else if (i == 2) {
                v = j == 0 ? -sp : cp * (j == 1 ? sr : cr);
            } else {
                const double a = i == 0 ? cy : sy;  // the factor of the sin p terms
                const double b = i == 0 ? -sy : cy;
                v = j == 0 ? a * cp : (j == 1 ? a * sp * sr + b * cr : a * sp * cr - b * sr);
            }
        }
    } else if (lane < 12) {
        v = job.T[lane];
    }
    if (lane < 12) {
        Th[lane] = (float)v;
        Tl[lane] = (float)(v - (double)Th[lane]);
    }
}

// q = T p as an unevaluated sum qh + ql: T given as hi/lo f32 pairs, TwoProd/TwoSum
__device__ __forceinline__ void transform_comp(const float* Th, const float* Tl, float px,
                                               float py, float pz, float* qh, float* ql) {
    const float pv[3] = {px, py, pz};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float hi = Th[4 * i + 3], lo = Tl[4 * i + 3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            float r = Th[4 * i + j];
            float ph = r * pv[j];
            float pl = fmaf(r, pv[j], -ph);
            float s = hi + ph;
            float bb = s - hi;
            float e = (hi - (s - bb)) + (ph - bb);
            hi = s;
            lo += e + pl + Tl[4 * i + j] * pv[j];
        }
        float s = hi + lo;
        ql[i] = lo - (s - hi);
        qh[i] = s;
    }
}

// s + e == a + b exactly
__device__ __forceinline__ void two_sum_f(float a, float b, float& s, float& e) {
    s = a + b;
    const float bp = s - a;
    e = (a - (s - bp)) + (b - bp);
}

// hi + lo += (oh + ol), both unevaluated f32 pairs
__device__ __forceinline__ void pair_add(float& hi, float& lo, float oh, float ol) {
    float e;
    two_sum_f(hi, oh, hi, e);
    lo += ol + e;
}

// One block per `chunk` points of a job (bx blocks per job in the grid; those past the job's
// end leave at once). A point's voxels are first listed (the radius test, candidates loaded
// four at a time), then scored: the lanes of a warp stay on one instruction stream. The FP64
// unit takes 16 cycles per SM for a warp instruction, so a thread's and a block's sums are
// kept as f32 pairs (TwoSum: 48 bits, against the terms' own 24) and become FP64 once per
// block. The block that finishes a job last adds its partials in a fixed order: no second
// launch. `done` counts a job's finished blocks and is back at zero when the launch ends.
// Bound: dependent loads (mask, candidates, records) and instruction issue. One 20k-point scan
// 54 -> 16 us, 20k points at 100 poses 132 -> 112 us, 64 scans of 2k-40k 92 -> 62 us, 256 x
// 20k points 266 -> 261 us.
__global__ void __launch_bounds__(ST, 8) k_score(MapView m, const float* __restrict__ pts,
                                                 const ScoreJob* __restrict__ jobs,
                                                 const AlignOut* __restrict__ aout, float d1,
                                                 float d2, uint32_t bx, uint32_t chunk,
                                                 ScorePartial* __restrict__ part,
                                                 uint32_t* __restrict__ done,
                                                 ScoreOut* __restrict__ out) {
    __shared__ float Th[12], Tl[12];
    __shared__ double trig[6];
    __shared__ float red[ST / 32][4];
    __shared__ uint32_t redc[ST / 32][2];
    __shared__ uint32_t s_off[32];            // neighbour offsets of the dense index
    __shared__ float4 s_list[LIST_CAP][ST];   // listed voxels per thread
    __shared__ bool s_last;
    const uint32_t j = blockIdx.x / bx, blk = blockIdx.x % bx;
    const ScoreJob& job = jobs[j];
    const uint32_t n = job.n, nblk = max(1u, (n + chunk - 1u) / chunk);
    if (blk >= nblk) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    nbhd_offsets(m, s_off);
    if (warp == 0) job_transform(job, aout, trig, Th, Tl, lane);
    __syncthreads();
    float nvh = 0.f, nvl = 0.f, sch = 0.f, scl = 0.f;
    uint32_t nvc = 0, nc = 0;
    const float* P = pts + 3 * job.offset;
    const uint32_t first = blk * chunk, last = min(n, first + chunk);
    float4* const list = &s_list[0][threadIdx.x];
    for (uint32_t i = first + threadIdx.x; i < last; i += ST) {
        float px = __ldg(P + 3 * (size_t)i), py = __ldg(P + 3 * (size_t)i + 1),
              pz = __ldg(P + 3 * (size_t)i + 2);
        if (!(isfinite(px) && isfinite(py) && isfinite(pz))) continue;
        float qh[3], ql[3];
        transform_comp(Th, Tl, px, py, pz, qh, ql);
        int32_t gc[3];
        const uint32_t oct = cell_oct_of_sum(m, qh, ql, gc);
        uint32_t corner;
        uint32_t state = search_begin(m, gc, oct, corner);
        int total = 0;
        float best = -INFINITY, sum = 0.f;
        do {
            const int cnt = search_round(m, s_off, gc, qh, ql, state, corner, MAX_NB_ALL, list, ST);
            total += cnt;
#pragma unroll 1
            for (int k = 0; k < cnt; ++k) {
                const float4 x = list[k * ST];
                float C[6];
                load_icov(m, __float_as_uint(x.w), C);
                const float c0 = fmaf(C[0], x.x, fmaf(C[1], x.y, C[2] * x.z));
                const float c1 = fmaf(C[1], x.x, fmaf(C[3], x.y, C[4] * x.z));
                const float c2 = fmaf(C[2], x.x, fmaf(C[4], x.y, C[5] * x.z));
                const float md = fmaf(x.x, c0, fmaf(x.y, c1, x.z * c2));
                const float s0 = -d1 * expf(-d2 * md * 0.5f);
                best = fmaxf(best, s0);
                sum += s0;
            }
        } while (search_more(m, state));
        if (total == 0) continue;
        float e;
        two_sum_f(nvh, best, nvh, e);
        nvl += e;
        two_sum_f(sch, sum, sch, e);
        scl += e;
        nvc++;
        nc += (uint32_t)total;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        pair_add(nvh, nvl, __shfl_xor_sync(0xffffffffu, nvh, o),
                 __shfl_xor_sync(0xffffffffu, nvl, o));
        pair_add(sch, scl, __shfl_xor_sync(0xffffffffu, sch, o),
                 __shfl_xor_sync(0xffffffffu, scl, o));
    }
    nvc = __reduce_add_sync(0xffffffffu, nvc);
    nc = __reduce_add_sync(0xffffffffu, nc);
    if (lane == 0) {
        red[warp][0] = nvh;
        red[warp][1] = nvl;
        red[warp][2] = sch;
        red[warp][3] = scl;
        redc[warp][0] = nvc;
        redc[warp][1] = nc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < ST / 32; ++w) {
            pair_add(nvh, nvl, red[w][0], red[w][1]);
            pair_add(sch, scl, red[w][2], red[w][3]);
            nvc += redc[w][0];
            nc += redc[w][1];
        }
        // an infinite sum has no low part
        const ScorePartial p{(double)nvh + (isfinite(nvh) ? (double)nvl : 0.0),
                             (double)sch + (isfinite(sch) ? (double)scl : 0.0), nvc, nc};
        if (nblk == 1u) {
            out[j] = ScoreOut{p.nvtl_sum, p.score_sum, p.nvtl_count, p.ncorr};
            s_last = false;
        } else {
            part[(size_t)j * bx + blk] = p;
            __threadfence();
            s_last = atomicAdd(done + j, 1u) == nblk - 1u;
        }
    }
    __syncthreads();
    if (!s_last || warp != 0) return;
    __threadfence();  // acquire: every block's partial is visible
    // lane l adds the partials l, l + 32, ..., then the lanes in a tree
    ScorePartial t{0.0, 0.0, 0, 0};
    for (uint32_t b = lane; b < nblk; b += 32) {
        const ScorePartial* q = part + (size_t)j * bx + b;
        t.nvtl_sum += __ldcg(&q->nvtl_sum);
        t.score_sum += __ldcg(&q->score_sum);
        t.nvtl_count += __ldcg((const unsigned long long*)&q->nvtl_count);
        t.ncorr += __ldcg((const unsigned long long*)&q->ncorr);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t.nvtl_sum += __shfl_xor_sync(0xffffffffu, t.nvtl_sum, o);
        t.score_sum += __shfl_xor_sync(0xffffffffu, t.score_sum, o);
        t.nvtl_count += __shfl_xor_sync(0xffffffffu, (unsigned long long)t.nvtl_count, o);
        t.ncorr += __shfl_xor_sync(0xffffffffu, (unsigned long long)t.ncorr, o);
    }
    if (lane == 0) {
        out[j] = ScoreOut{t.nvtl_sum, t.score_sum, t.nvtl_count, t.ncorr};
        done[j] = 0u;
    }
}

size_t score_part_bytes(uint32_t num_jobs, uint32_t max_n, int sms) {
    return (size_t)score_blocks(num_jobs, max_n, sms) * num_jobs * sizeof(ScorePartial);
}

int launch_score(const MapView& map, const float* pts, const ScoreJob* jobs, uint32_t num_jobs,
                 uint32_t max_n, const AlignOut* align_out, void* part, uint32_t* done,
                 ScoreOut* out, float d1, float d2, int sms, cudaStream_t s) {
    if (num_jobs == 0) return 0;
    const uint32_t bx = score_blocks(num_jobs, max_n, sms);
    const uint64_t grid = (uint64_t)bx * num_jobs;
    if (grid > 0x7FFFFFFFull) {
        set_error("score launch: too many points times poses");
        return NDT_ERR_CAPACITY;
    }
    k_score<<<(unsigned)grid, ST, 0, s>>>(map, pts, jobs, align_out, d1, d2, bx,
                                          ST * score_ppt(num_jobs, max_n, sms), (ScorePartial*)part,
                                          done, out);
    return cuda_fail(cudaGetLastError(), "score launch");
}

// Standalone neighbour query with the graph kernel's semantics, f32 arithmetic unfused.
__global__ void k_query(MapView m, const float* __restrict__ q, size_t n, int max_nb,
                        int32_t* __restrict__ idx, int32_t* __restrict__ cnt) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float qx = q[3 * i], qy = q[3 * i + 1], qz = q[3 * i + 2];
    int32_t gx = (int32_t)floorf(__fmul_rn(qx, m.inv_res));
    int32_t gy = (int32_t)floorf(__fmul_rn(qy, m.inv_res));
    int32_t gz = (int32_t)floorf(__fmul_rn(qz, m.inv_res));
    int c = 0;
    for (int k = 0; k < 27 && c < max_nb; ++k) {
        int dx, dy, dz;
        offset27(k, dx, dy, dz);
        float mx, my, mz;
        const int32_t s = find_cell(m, (int32_t)((uint32_t)gx + (uint32_t)dx),
                                    (int32_t)((uint32_t)gy + (uint32_t)dy),
                                    (int32_t)((uint32_t)gz + (uint32_t)dz), &mx, &my, &mz);
        if (s < 0) continue;
        if (dist2_rn(qx, qy, qz, mx, my, mz) <= m.r2)
            idx[i * (size_t)max_nb + c++] = m.grid ? s : m.slot_vidx[s];
    }
    for (int k = c; k < max_nb; ++k) idx[i * (size_t)max_nb + k] = -1;
    cnt[i] = c;
}

int launch_query(const MapView& map, const float* q, size_t n, int max_nb, int32_t* idx,
                 int32_t* cnt, cudaStream_t s) {
    if (n == 0) return 0;
    k_query<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(map, q, n, max_nb, idx, cnt);
    return cuda_fail(cudaGetLastError(), "query launch");
}

}  // namespace ndtgb
