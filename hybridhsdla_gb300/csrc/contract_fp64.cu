// FP64 tensor-core contraction OUT = P^H diag(w) Q (complex128), batched over jobs.
//
// It carries the plain-FP64 form of
//   * kernel (b), the per-atom T application X_a = T_a [A_a; B_a]
//     (h_and_s_stripped_v2.cpp:193-231 zhemm+zgemm and :321-349 zhemm): P is the
//     Hermitian 2L x 2L block [[T_AA, T_AB],[T_AB^H, T_BB]], so P^H = P;
//   * kernel (c), the lower-triangle Hermitian contractions
//     S = C^H diag(1, ||udot||^2) C  (the two zherk calls, :158/:177) and
//     H = C^H X                      (zher2k + zherkx, :300/:362)
//     with C = [A_a; B_a] stacked per atom.
//
// and, in the structure-factor form, the real products of its rows.
//
// GB300 mapping: FP64 MMA (mma.sync m16n8k4 .f64), complex products as four real MMAs
//   Re += Pr Qr + Pi Qi,   Im += Pr Qi - Pi Qr,
// and a flat tile list over all jobs (lower-triangle tiles only for the Hermitian outputs) so that every
// atom / k-point of a call goes out in one launch.
#include <algorithm>

#include "common.cuh"

namespace hsdla {
namespace {

__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

template <typename Job>
__device__ __forceinline__ void tile_of(const Job &j, int64_t x, int64_t &ti, int64_t &tj) {
    if (j.lower) {
        ti = triangle_row(x);
        tj = x - ti * (ti + 1) / 2;
    } else {
        ti = x / j.tiles_n;
        tj = x - ti * j.tiles_n;
    }
}

// Complex DMMA products (the per-atom form, the contraction entry, the plugin), as fp64_real_kernel (below) with
// both parts of an element in one CTA: bound by GB300's FP64 rate at every shape, so fragments come straight
// from global memory and what counts is an even share of the MMAs per SM.  A tile of 32 x 32, a 16 x 16 quarter per
// warp, or of 16 x 16 with the contraction split over the warps (fp64_edge).  Lower triangle of P^H Q of n columns
// over k rows, ms, here and on the staged 64 x 64 tiles before: n 200, k 400 0.18 and 1.94; n 200, k 1200 0.42 and
// 5.69; n 700, k 1200 2.6 and 5.7; n 2200, k 1200 22.5 and 27.7; n 6000, k 1000 136 and 140.  Relative error (Frobenius,
// against extended precision, k 700) 6.5e-16 and 1.3e-15.
constexpr int kJobsU = 2;           // K steps loaded ahead

template <bool kSplit>
__device__ __forceinline__ void fp64_job_tile(const Fp64Job &j, int64_t x) {
    constexpr int kT = kSplit ? 16 : 32;
    const int64_t m = j.m, n = j.n, K = j.k;
    int64_t ti, tj;
    tile_of(j, x, ti, tj);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    const int64_t m0 = ti * kT + (kSplit ? 0 : (warp >> 1) * 16), n0 = tj * kT + (kSplit ? 0 : (warp & 1) * 16);
    double re[2][4] = {}, im[2][4] = {};
    const int64_t steps = (K + 3) / 4;
    const int64_t s0 = kSplit ? steps * warp / 4 : 0, s1 = kSplit ? steps * (warp + 1) / 4 : steps;
    if (m0 < m && n0 < n && !(j.lower && m0 + 15 < n0)) {
        // rows and columns past the ends repeat the last one (their results are not stored)
        const double2 *pa0 = j.P + j.ldp * min(m0 + gid, m - 1), *pa1 = j.P + j.ldp * min(m0 + gid + 8, m - 1);
        const double2 *pb0 = j.Q + j.ldq * min(n0 + gid, n - 1), *pb1 = j.Q + j.ldq * min(n0 + gid + 8, n - 1);
        double2 a0[2][kJobsU], a1[2][kJobsU], b0[2][kJobsU], b1[2][kJobsU];
        auto load = [&](int buf, int64_t s) {
#pragma unroll
            for (int u = 0; u < kJobsU; ++u) {
                const int64_t k = (s + u) * 4 + tig, kc = min(k, K - 1);
                const bool in = k < K && s + u < s1;
                const double2 zero = make_double2(0.0, 0.0);
                a0[buf][u] = in ? pa0[kc] : zero;
                a1[buf][u] = in ? pa1[kc] : zero;
                b0[buf][u] = in ? pb0[kc] : zero;
                b1[buf][u] = in ? pb1[kc] : zero;
                if (j.w) {
                    const double w = j.w[kc];
                    b0[buf][u].x *= w;
                    b0[buf][u].y *= w;
                    b1[buf][u].x *= w;
                    b1[buf][u].y *= w;
                }
            }
        };
        // conj(P) Q: Re += Pr Qr + Pi Qi, Im += Pr Qi - Pi Qr
        auto mma = [&](int buf, int64_t left) {
#pragma unroll
            for (int u = 0; u < kJobsU; ++u) {
                if (u >= left) break;           // no MMA for a step past the end
                const double2 x0 = a0[buf][u], x1 = a1[buf][u], y0 = b0[buf][u], y1 = b1[buf][u];
                dmma(re[0], x0.x, x1.x, y0.x);
                dmma(re[1], x0.x, x1.x, y1.x);
                dmma(im[0], x0.x, x1.x, y0.y);
                dmma(im[1], x0.x, x1.x, y1.y);
                dmma(re[0], x0.y, x1.y, y0.y);
                dmma(re[1], x0.y, x1.y, y1.y);
                dmma(im[0], x0.y, x1.y, -y0.x);
                dmma(im[1], x0.y, x1.y, -y1.x);
            }
        };
        if (s0 < s1) load(0, s0);
        for (int64_t s = s0; s < s1; s += 2 * kJobsU) {
            if (s + kJobsU < s1) load(1, s + kJobsU);
            mma(0, s1 - s);
            if (s + 2 * kJobsU < s1) load(0, s + 2 * kJobsU);
            if (s + kJobsU < s1) mma(1, s1 - s - kJobsU);
        }
    }
    if constexpr (kSplit) {
        // the warps' parts, added in warp order
        __shared__ double2 part[3][2][4][32];
        if (warp > 0)
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int c = 0; c < 4; ++c) part[warp - 1][t][c][lane] = make_double2(re[t][c], im[t][c]);
        __syncthreads();
        if (warp > 0) return;
#pragma unroll
        for (int w = 0; w < 3; ++w)
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    re[t][c] += part[w][t][c][lane].x;
                    im[t][c] += part[w][t][c][lane].y;
                }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int64_t row = m0 + gid + ((c >= 2) ? 8 : 0), col = n0 + t * 8 + tig * 2 + (c & 1);
            if (row < m && col < n && (!j.lower || row >= col)) j.out[row + j.ldo * col] = make_double2(re[t][c], im[t][c]);
        }
}

// ---------------------------------------------------------------- real products
// Real DMMA products for the structure-factor form's real rows.  GB300's FP64 rate (~1.1 TFLOP/s,
// one m16n8k4 MMA in ~300 cycles and SM) bounds every shape, so there is no staging: fragments come
// straight from global memory (L1 and L2 serve the reuse, 0.3-0.5 TB/s), four K steps ahead, and what
// counts is an even share of the MMAs per SM.  A CTA of four warps has a 32 x 32 tile (a 16 x 16
// quarter each); products with fewer than kSplitBelow of those per SM sum their contraction in four parts, on 16 x 16
// tiles with a part per warp, or, in a launch that others fill, one part after the other on 32 x 32 tiles (the
// same sums: a k-point's results keep their bits whatever it runs with.  3 k-points of 700 columns, one type, 0.345 ms
// as one sum, 0.354 in parts, 0.378 on 16 x 16 tiles).  Whole pass, complex 64 x 64 tiles before and this now: 235 columns,
// lmax 8, two types (host call) 2.98 and 0.62 ms (20 of 152 SMs were busy); 3000 columns of four types
// 55.7 and 18.5 ms (eight real products and three, each at the FP64 rate).
// The multiplications by S's row weights share the pipe, at a sixth of an MMA each: done once, by the T application
// (Fp64RealJob::wq), not for every fragment: 3001 columns of four types 19.6 and 18.4 ms, 400 columns of two 0.232 and
// 0.226.  Split tiles write diag(w) Q with the warps whose parts are handed over.
constexpr int kRealU = 4;            // K steps loaded ahead
constexpr int kSplitBelow = 8;

// kParts: the contraction in the split tile's four parts, summed in its order.
template <bool kSplit, bool kParts>
__device__ __forceinline__ void fp64_real_tile(const Fp64RealJob &j, int64_t x) {
    constexpr int kT = kSplit ? 16 : 32;
    const int64_t m = j.m, n = j.n, K = j.k;
    int64_t ti, tj;
    tile_of(j, x, ti, tj);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    const int64_t m0 = ti * kT + (kSplit ? 0 : (warp >> 1) * 16), n0 = tj * kT + (kSplit ? 0 : (warp & 1) * 16);
    double acc[2][4] = {}, sum[2][4];
    const int64_t steps = (K + 3) / 4;
    int64_t s0 = kSplit ? steps * warp / 4 : 0, s1 = kSplit ? steps * (warp + 1) / 4 : steps;
    if (m0 < m && n0 < n && !(j.lower && m0 + 15 < n0)) {
        // rows and columns past the ends repeat the last one (their results are not stored)
        const double *pa0 = j.P + j.ldp * min(m0 + gid, m - 1), *pa1 = j.P + j.ldp * min(m0 + gid + 8, m - 1);
        const double *pb0 = j.Q + j.ldq * min(n0 + gid, n - 1), *pb1 = j.Q + j.ldq * min(n0 + gid + 8, n - 1);
        double a0[2][kRealU], a1[2][kRealU], b0[2][kRealU], b1[2][kRealU];
        auto load = [&](int buf, int64_t s) {
#pragma unroll
            for (int u = 0; u < kRealU; ++u) {
                const int64_t k = (s + u) * 4 + tig, kc = min(k, K - 1);
                const bool in = k < K && s + u < s1;
                a0[buf][u] = in ? pa0[kc] : 0.0;
                a1[buf][u] = in ? pa1[kc] : 0.0;
                b0[buf][u] = pb0[kc];
                b1[buf][u] = pb1[kc];
            }
        };
        auto step = [&](int buf, int u) {
            dmma(acc[0], a0[buf][u], a1[buf][u], b0[buf][u]);
            dmma(acc[1], a0[buf][u], a1[buf][u], b1[buf][u]);
        };
        // the last steps by number: MMAs of steps past the end, even predicated off, would take their time
        // (whole pass, 235 columns 0.241 and 0.212 ms, 3000 of four types 20.4 and 19.6, 256 of three 0.368 and 0.309)
        auto mma = [&](int buf, int64_t left) {
            switch (left < kRealU ? (int)left : kRealU) {
                case 1: step(buf, 0); break;
                case 2: step(buf, 0); step(buf, 1); break;
                case 3: step(buf, 0); step(buf, 1); step(buf, 2); break;
                default: step(buf, 0); step(buf, 1); step(buf, 2); step(buf, 3);
            }
        };
        static_assert(kRealU == 4, "steps by number");
#pragma unroll 1
        for (int q = 0; q < (kParts ? 4 : 1); ++q) {
            if constexpr (kParts) {
                s0 = steps * q / 4;
                s1 = steps * (q + 1) / 4;
            }
            if (s0 < s1) load(0, s0);
            for (int64_t s = s0; s < s1; s += 2 * kRealU) {
                if (s + kRealU < s1) load(1, s + kRealU);
                mma(0, s1 - s);
                if (s + 2 * kRealU < s1) load(0, s + 2 * kRealU);
                if (s + kRealU < s1) mma(1, s1 - s - kRealU);
            }
            if constexpr (kParts) {
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        sum[t][c] = q == 0 ? acc[t][c] : sum[t][c] + acc[t][c];
                        acc[t][c] = q == 3 ? sum[t][c] : 0.0;
                    }
            }
        }
    }
    if constexpr (kSplit) {
        // the warps' parts, added in warp order
        __shared__ double part[3][2][4][32];
        if (warp > 0)
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int c = 0; c < 4; ++c) part[warp - 1][t][c][lane] = acc[t][c];
        __syncthreads();
        if (warp > 0) {
            if (j.wq)
                for (int e = threadIdx.x - 32; e < kT * kT; e += 96) {
                    const int64_t row = m0 + (e & 15), col = n0 + (e >> 4);
                    if (row < K && col < n) j.wq[row + j.ldq * col] = j.w[row] * j.Q[row + j.ldq * col];
                }
            return;
        }
#pragma unroll
        for (int w = 0; w < 3; ++w)
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[t][c] += part[w][t][c][lane];
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int64_t row = m0 + gid + ((c >= 2) ? 8 : 0), col = n0 + t * 8 + tig * 2 + (c & 1);
            if (row < m && col < n && (!j.lower || row >= col)) j.out[row + j.ldo * col] = acc[t][c];
            if (!kSplit && j.wq && row < K && col < n) j.wq[row + j.ldq * col] = j.w[row] * j.Q[row + j.ldq * col];
        }
}

// The job of a block's tile, and the tile in that job's shape.
template <typename Job>
__device__ __forceinline__ const Job &job_of(const Job *jobs, int num_jobs, int64_t tile) {
    int lo = 0, hi = num_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    return jobs[lo];
}
__global__ void __launch_bounds__(128) fp64_jobs_kernel(const Fp64Job *__restrict__ jobs, int num_jobs) {
    const Fp64Job &j = job_of(jobs, num_jobs, blockIdx.x);
    if (j.edge == 16) fp64_job_tile<true>(j, blockIdx.x - j.tile_begin);
    else fp64_job_tile<false>(j, blockIdx.x - j.tile_begin);
}
__global__ void __launch_bounds__(128) fp64_real_kernel(const Fp64RealJob *__restrict__ jobs, int num_jobs) {
    const Fp64RealJob &j = job_of(jobs, num_jobs, blockIdx.x);
    const int64_t x = blockIdx.x - j.tile_begin;
    if (j.edge == 16) fp64_real_tile<true, false>(j, x);
    else if (j.parts) fp64_real_tile<false, true>(j, x);
    else fp64_real_tile<false, false>(j, x);
}

}  // namespace

namespace {
template <typename Job>
int64_t assign(Job *jobs, int num_jobs) {
    int64_t total = 0;
    for (int i = 0; i < num_jobs; ++i) {
        Job &j = jobs[i];
        const int64_t edge = j.edge, tm = (j.m + edge - 1) / edge, tn = (j.n + edge - 1) / edge;
        j.tiles_n = (int32_t)tn;
        j.tile_begin = total;
        total += j.lower ? tm * (tm + 1) / 2 : tm * tn;
    }
    return total;
}
}  // namespace

// Tiles of 32 from kSplitBelow of them per SM on (complex products, n 2200: 22.5 ms, 22.9 on tiles of 16), else of 16
// (n 1500, k 1200: 10.8 ms, 11.3 on tiles of 32; n 200, k 1200: 0.42, 1.48).
int fp64_edge(int64_t tiles32) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return tiles32 >= (int64_t)kSplitBelow * nsm ? 32 : 16;
}
int64_t fp64_assign(Fp64Job *jobs, int num_jobs) { return assign(jobs, num_jobs); }
int64_t fp64_real_assign(Fp64RealJob *jobs, int num_jobs) {
    int64_t tiles = 0;
    for (int i = 0; i < num_jobs; ++i) {
        const int64_t tm = (jobs[i].m + 31) / 32, tn = (jobs[i].n + 31) / 32;
        tiles += jobs[i].lower ? tm * (tm + 1) / 2 : tm * tn;
    }
    const int edge = fp64_edge(tiles);
    for (int i = 0; i < num_jobs; ++i) jobs[i].edge = jobs[i].parts ? edge : 32;
    return assign(jobs, num_jobs);
}

cudaError_t launch_fp64_real(const Fp64RealJob *d_jobs, int num_jobs, int64_t tiles, cudaStream_t st) {
    if (tiles <= 0) return cudaSuccess;
    if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
    fp64_real_kernel<<<(unsigned)tiles, 128, 0, st>>>(d_jobs, num_jobs);
    return cudaGetLastError();
}

cudaError_t launch_fp64_jobs(const Fp64Job *d_jobs, int num_jobs, int64_t total_tiles, cudaStream_t st) {
    if (total_tiles <= 0) return cudaSuccess;
    if (total_tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
    fp64_jobs_kernel<<<(unsigned)total_tiles, 128, 0, st>>>(d_jobs, num_jobs);
    return cudaGetLastError();
}

}  // namespace hsdla
