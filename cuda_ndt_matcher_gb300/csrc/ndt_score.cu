// ndt_score.cu — per-pose scoring and the neighbour query on sm_103a.
//
// k_score: for each (scan, pose) job, every point is transformed (compensated f32: the
// transform as hi/lo pairs, so x = q - mean keeps f32 precision), the voxels whose
// centroid lies within one resolution are found through the neighbourhood masks of the dense
// index, or the 27-cell hash probe (all of them: kiddo's `within` set, src/ndt_cuda/src/voxel_grid/search.rs:90-99), and the block
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

constexpr int ST = 256;  // threads per block

struct ScorePartial {
    double nvtl_sum;
    double score_sum;
    uint64_t nvtl_count;
    uint64_t ncorr;
};

// Points per thread of a launch over `jobs` jobs of `points` points in all, at most max_n each. One
// while they do not fill the GPU, so that a single scan spreads over every SM (scoring a point is
// one dependent chain of loads); more as they do, which pays the block's set-up and reduction
// once for several points. By points in all, us at 1, 2, 4, 8 points per thread (a 400 m map with
// octant masks; calls that evaluate 5,000 or 18,000 points at many poses):
//     75k 48/49/52/72, 270k 65/55/66/77, 500k 74/63/61/73, 1.1M 103/91/91/91, 1.8M
//     140/116/116/115, 3.6M 231/192/178/177, 18M 972/744/659/621.
// Scans of uneven size leave the blocks past their end empty: no more than four in five.
static uint32_t score_ppt(uint32_t jobs, uint32_t max_n, uint64_t points, int sms) {
    const uint64_t per_sm = points / (uint64_t)std::max(1, sms);
    uint32_t ppt = per_sm < 1000 ? 1 : (per_sm < 3000 ? 2 : (per_sm < 26000 ? 4 : 8));
    auto blocks = [&](uint64_t n) { return (n + ST * (uint64_t)ppt - 1) / (ST * (uint64_t)ppt); };
    while (ppt < 8 && jobs * blocks(max_n) > 4 * (blocks(points) + jobs)) ppt *= 2;
    while (jobs * blocks(max_n) > 0x7FFFFFFFull) ppt *= 2;  // (blocks of a launch)
    return ppt;
}

static uint32_t score_blocks(uint32_t max_n, uint32_t ppt) {
    const uint64_t per = (uint64_t)ST * ppt;
    return std::max<uint32_t>(1u, (uint32_t)((max_n + per - 1) / per));
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

// One block per `chunk` points of a job (bx blocks per job in the grid; those past the job's
// end leave at once). A voxel is scored as it passes the radius test; sums are FP64. The block
// that finishes a job last adds its partials in a fixed order: no second launch. `done` counts
// a job's finished blocks and is back at zero when the launch ends.
// Bound: dependent loads (mask, candidates, records) hidden by 48 warps an SM at 40 registers, and
// instruction issue. Listing a point's voxels first and scoring them in a second loop was
// slower wherever the GPU is full (128 threads, 64 registers: 18M point-poses 775 us for 621; 200
// scans of 5k points 94 for 64) and no faster elsewhere. Kernel: one 20k-point scan 52 -> 16 us,
// 18k points at 100 poses 101 -> 81, 64 scans of 2k-18k 68 -> 49, 256 x 18k 203 -> 186.
__global__ void __launch_bounds__(ST, 6) k_score(MapView m, const float* __restrict__ pts,
                                                 const ScoreJob* __restrict__ jobs,
                                                 const AlignOut* __restrict__ aout, float d1,
                                                 float d2, uint32_t bx, uint32_t chunk,
                                                 ScorePartial* __restrict__ part,
                                                 uint32_t* __restrict__ done,
                                                 ScoreOut* __restrict__ out) {
    __shared__ float Th[12], Tl[12];
    __shared__ double trig[6];
    __shared__ double red[ST / 32][2];
    __shared__ uint32_t redc[ST / 32][2];
    __shared__ uint32_t s_off[32];  // neighbour offsets of the dense index
    __shared__ bool s_last;
    const uint32_t j = blockIdx.x / bx, blk = blockIdx.x % bx;
    const ScoreJob& job = jobs[j];
    const uint32_t n = job.n, nblk = max(1u, (n + chunk - 1u) / chunk);
    if (blk >= nblk) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    nbhd_offsets(m, s_off);
    if (warp == 0) job_transform(job, aout, trig, Th, Tl, lane);
    __syncthreads();
    double nv = 0.0, sc = 0.0;
    uint32_t nvc = 0, nc = 0;  // (at most 27 pairs a point, and fewer than 2^27 points a block)
    const float* P = pts + 3 * job.offset;
    const uint32_t first = blk * chunk, last = min(n, first + chunk);
    for (uint32_t i = first + threadIdx.x; i < last; i += ST) {
        float px = __ldg(P + 3 * (size_t)i), py = __ldg(P + 3 * (size_t)i + 1),
              pz = __ldg(P + 3 * (size_t)i + 2);
        if (!(isfinite(px) && isfinite(py) && isfinite(pz))) continue;
        float qh[3], ql[3];
        transform_comp(Th, Tl, px, py, pz, qh, ql);
        int32_t gc[3];
        const uint32_t oct = cell_oct_of_sum(m, qh, ql, gc);
        int total = 0;
        float best = -INFINITY, sum = 0.f;
        // one voxel with centroid (mx, my, mz) in record r: radius test, then its score term
        auto visit = [&](float mx, float my, float mz, int32_t r) {
            const float x0 = (qh[0] - mx) + ql[0], x1 = (qh[1] - my) + ql[1],
                        x2 = (qh[2] - mz) + ql[2];
            if (fmaf(x0, x0, fmaf(x1, x1, x2 * x2)) > m.r2) return;
            float C[6];
            load_icov(m, (uint32_t)r, C);
            const float c0 = fmaf(C[0], x0, fmaf(C[1], x1, C[2] * x2));
            const float c1 = fmaf(C[1], x0, fmaf(C[3], x1, C[4] * x2));
            const float c2 = fmaf(C[2], x0, fmaf(C[4], x1, C[5] * x2));
            const float md = fmaf(x0, c0, fmaf(x1, c1, x2 * c2));
            const float s0 = -d1 * expf(-d2 * md * 0.5f);
            best = fmaxf(best, s0);
            sum += s0;
            total++;
        };
        if (m.grid) {  // occupied neighbours only, in the same order, from the mask
            uint32_t corner;
            uint32_t bits = nbhd_mask(m, gc, oct, corner);
#pragma unroll 1
            while (bits != 0u) {
                const uint32_t b = (uint32_t)(__ffs(bits) - 1);
                bits &= bits - 1u;
                const float4 e = __ldg(m.grid + (corner + s_off[b]));
                visit(e.x, e.y, e.z, __float_as_int(e.w));
            }
        } else {
#pragma unroll 1
            for (int c = 0; c < 27; ++c) {
                int dx, dy, dz;
                offset27(c, dx, dy, dz);
                float mx, my, mz;
                const int32_t r = find_cell(m, (int32_t)((uint32_t)gc[0] + (uint32_t)dx),
                                            (int32_t)((uint32_t)gc[1] + (uint32_t)dy),
                                            (int32_t)((uint32_t)gc[2] + (uint32_t)dz), &mx, &my,
                                            &mz);
                if (r >= 0) visit(mx, my, mz, r);
            }
        }
        if (total == 0) continue;
        nv += (double)best;
        sc += (double)sum;
        nvc++;
        nc += (uint32_t)total;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nv += __shfl_xor_sync(0xffffffffu, nv, o);
        sc += __shfl_xor_sync(0xffffffffu, sc, o);
    }
    nvc = __reduce_add_sync(0xffffffffu, nvc);
    nc = __reduce_add_sync(0xffffffffu, nc);
    if (lane == 0) {
        red[warp][0] = nv;
        red[warp][1] = sc;
        redc[warp][0] = nvc;
        redc[warp][1] = nc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < ST / 32; ++w) {
            nv += red[w][0];
            sc += red[w][1];
            nvc += redc[w][0];
            nc += redc[w][1];
        }
        const ScorePartial p{nv, sc, nvc, nc};
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

size_t score_part_bytes(uint32_t num_jobs, uint32_t max_n, uint64_t points, int sms) {
    return (size_t)score_blocks(max_n, score_ppt(num_jobs, max_n, points, sms)) * num_jobs *
           sizeof(ScorePartial);
}

int launch_score(const MapView& map, const float* pts, const ScoreJob* jobs, uint32_t num_jobs,
                 uint32_t max_n, uint64_t points, const AlignOut* align_out, void* part,
                 uint32_t* done, ScoreOut* out, float d1, float d2, int sms, cudaStream_t s) {
    if (num_jobs == 0) return 0;
    const uint32_t ppt = score_ppt(num_jobs, max_n, points, sms), bx = score_blocks(max_n, ppt);
    k_score<<<bx * num_jobs, ST, 0, s>>>(map, pts, jobs, align_out, d1, d2, bx, ST * ppt,
                                         (ScorePartial*)part, done, out);
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
