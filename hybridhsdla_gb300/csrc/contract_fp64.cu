// FP64 tensor-core contraction OUT = P^H diag(w) Q (complex128), batched over jobs.
//
// This one kernel carries the plain-FP64 form of
//   * kernel (b), the per-atom T application X_a = T_a [A_a; B_a]
//     (h_and_s_stripped_v2.cpp:193-231 zhemm+zgemm and :321-349 zhemm): P is the
//     Hermitian 2L x 2L block [[T_AA, T_AB],[T_AB^H, T_BB]], so P^H = P;
//   * kernel (c), the lower-triangle Hermitian contractions
//     S = C^H diag(1, ||udot||^2) C  (the two zherk calls, :158/:177) and
//     H = C^H X                      (zher2k + zherkx, :300/:362)
//     with C = [A_a; B_a] stacked per atom.
//
// GB300 mapping: FP64 MMA (mma.sync m16n8k4 .f64) on 64x64 complex tiles, four
// warps of 32x32, complex products as four real MMAs
//   Re += Pr Qr + Pi Qi,   Im += Pr Qi - Pi Qr,
// a two-stage cp.async pipeline over K chunks of 16, and a flat tile list over
// all jobs (lower-triangle tiles only for the Hermitian outputs) so that every
// atom / k-point of a call goes out in one launch.
#include <algorithm>

#include "common.cuh"

namespace hsdla {
namespace {

constexpr int BM = kFp64Tile, BN = kFp64Tile, BK = 16;
constexpr int SROW = 66;                       // double2 per smem row (== 2 mod 8: conflict-free fragments)
constexpr int kStageElems = 2 * BK * SROW;     // P and Q tiles of one stage (double2)
constexpr int kThreads = 128;

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int sz = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void tile_of(const Fp64Job &j, int64_t x, int64_t &ti, int64_t &tj) {
    if (j.lower) {
        ti = triangle_row(x);
        tj = x - ti * (ti + 1) / 2;
    } else {
        ti = x / j.tiles_n;
        tj = x - ti * j.tiles_n;
    }
}

__global__ void __launch_bounds__(kThreads) fp64_jobs_kernel(const Fp64Job *__restrict__ jobs, int num_jobs,
                                                            int64_t total_tiles) {
    extern __shared__ __align__(16) double2 sm[];
    for (int64_t gt = blockIdx.x; gt < total_tiles; gt += gridDim.x) {
        // job lookup (jobs sorted by tile_begin)
        int lo = 0, hi = num_jobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (jobs[mid].tile_begin <= gt) lo = mid; else hi = mid - 1;
        }
        const Fp64Job j = jobs[lo];
        int64_t ti, tj;
        tile_of(j, gt - j.tile_begin, ti, tj);
        const int64_t m0 = ti * BM, n0 = tj * BN;

        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        const int gid = lane >> 2, tig = lane & 3;
        const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;

        double re[2][4][4], im[2][4][4];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int c = 0; c < 4; ++c) { re[a][b][c] = 0.0; im[a][b][c] = 0.0; }

        const int64_t nk = (j.k + BK - 1) / BK;
        auto load_stage = [&](int stage, int64_t kc) {
            double2 *Ps = sm + stage * kStageElems;
            double2 *Qs = Ps + BK * SROW;
            const int64_t k0 = kc * BK;
#pragma unroll
            for (int it = 0; it < (BK * BM) / kThreads; ++it) {
                const int idx = tid + it * kThreads;
                const int kk = idx % BK, c = idx / BK;
                const int64_t gk = k0 + kk;
                const bool vp = gk < j.k && (m0 + c) < j.m;
                const double2 *srcp = vp ? j.P + gk + j.ldp * (m0 + c) : j.P;
                cp_async16(Ps + kk * SROW + c, srcp, vp);
                const bool vq = gk < j.k && (n0 + c) < j.n;
                const double2 *srcq = vq ? j.Q + gk + j.ldq * (n0 + c) : j.Q;
                cp_async16(Qs + kk * SROW + c, srcq, vq);
            }
            cp_async_commit();
        };

        __syncthreads();   // previous tile's readers are done with the stages
        load_stage(0, 0);
        for (int64_t kc = 0; kc < nk; ++kc) {
            const int stage = (int)(kc & 1);
            if (kc + 1 < nk) {
                load_stage(stage ^ 1, kc + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
            const double2 *Ps = sm + stage * kStageElems;
            const double2 *Qs = Ps + BK * SROW;
#pragma unroll
            for (int ks = 0; ks < BK / 4; ++ks) {
                const int kk = ks * 4 + tig;
                double wk = 1.0;
                if (j.w) {
                    const int64_t gk = kc * BK + kk;
                    wk = gk < j.k ? j.w[gk] : 0.0;
                }
                double ar[2][2], ai[2][2], nai[2][2];
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const double2 v = Ps[kk * SROW + wm + mt * 16 + gid + 8 * h];
                        ar[mt][h] = v.x * wk;
                        ai[mt][h] = v.y * wk;
                        nai[mt][h] = -ai[mt][h];
                    }
                double br[4], bi[4];
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    const double2 v = Qs[kk * SROW + wn + nt * 8 + gid];
                    br[nt] = v.x;
                    bi[nt] = v.y;
                }
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 4; ++nt) {
                        dmma(re[mt][nt], ar[mt][0], ar[mt][1], br[nt]);
                        dmma(re[mt][nt], ai[mt][0], ai[mt][1], bi[nt]);
                        dmma(im[mt][nt], ar[mt][0], ar[mt][1], bi[nt]);
                        dmma(im[mt][nt], nai[mt][0], nai[mt][1], br[nt]);
                    }
            }
            __syncthreads();
        }
        // epilogue: masked store (lower triangle for Hermitian outputs)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int64_t row = m0 + wm + mt * 16 + gid + ((c >= 2) ? 8 : 0);
                    const int64_t col = n0 + wn + nt * 8 + tig * 2 + (c & 1);
                    if (row < j.m && col < j.n && (!j.lower || row >= col))
                        j.out[row + j.ldo * col] = make_double2(re[mt][nt][c], im[mt][nt][c]);
                }
    }
}

// ---------------------------------------------------------------- real products
// Real DMMA products for the structure-factor form's real rows.  GB300's FP64 rate (1.05 TFLOP/s,
// one m16n8k4 MMA in ~300 cycles and SM) bounds every shape, so there is no staging: fragments come
// straight from global memory (L1 and L2 serve the reuse, 0.3-0.5 TB/s), four K steps ahead, and what
// counts is an even share of the MMAs per SM.  A CTA of four warps has a 32 x 32 tile (a 16 x 16
// quarter each); where a launch has fewer than kSplitBelow of those per SM, a 16 x 16 tile with the
// contraction split over the warps.  Whole pass, complex 64 x 64 tiles before and this now: 235 columns,
// lmax 8, two types (host call) 2.96 and 0.64 ms (20 of 152 SMs were busy); 3000 columns of four types
// 55.7 and 20.6 ms (eight real products and three, each at the FP64 rate).
constexpr int kRealU = 4;            // K steps loaded ahead
constexpr int kSplitBelow = 8;

template <bool kSplit>
__global__ void __launch_bounds__(128) fp64_real_kernel(const Fp64RealJob *__restrict__ jobs, int num_jobs) {
    constexpr int kT = kSplit ? 16 : 32;
    const int64_t gt = blockIdx.x;
    int lo = 0, hi = num_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].tile_begin <= gt) lo = mid; else hi = mid - 1;
    }
    const Fp64RealJob &j = jobs[lo];
    const int64_t m = j.m, n = j.n, K = j.k, x = gt - j.tile_begin;
    int64_t ti, tj;
    if (j.lower) {
        ti = triangle_row(x);
        tj = x - ti * (ti + 1) / 2;
    } else {
        ti = x / j.tiles_n;
        tj = x - ti * j.tiles_n;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    const int64_t m0 = ti * kT + (kSplit ? 0 : (warp >> 1) * 16), n0 = tj * kT + (kSplit ? 0 : (warp & 1) * 16);
    double acc[2][4] = {};
    const int64_t steps = (K + 3) / 4;
    const int64_t s0 = kSplit ? steps * warp / 4 : 0, s1 = kSplit ? steps * (warp + 1) / 4 : steps;
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
                if (j.w) {
                    const double w = j.w[kc];
                    a0[buf][u] *= w;
                    a1[buf][u] *= w;
                }
            }
        };
        auto mma = [&](int buf) {
#pragma unroll
            for (int u = 0; u < kRealU; ++u) {
                dmma(acc[0], a0[buf][u], a1[buf][u], b0[buf][u]);
                dmma(acc[1], a0[buf][u], a1[buf][u], b1[buf][u]);
            }
        };
        if (s0 < s1) load(0, s0);
        for (int64_t s = s0; s < s1; s += 2 * kRealU) {
            if (s + kRealU < s1) load(1, s + kRealU);
            mma(0);
            if (s + 2 * kRealU < s1) load(0, s + 2 * kRealU);
            if (s + kRealU < s1) mma(1);
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
        if (warp > 0) return;
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
        }
}

}  // namespace

int64_t fp64_real_assign(Fp64RealJob *jobs, int num_jobs, int *edge) {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    int64_t total = 0;
    for (int e = 32; e >= 16; e /= 2) {
        total = 0;
        for (int i = 0; i < num_jobs; ++i) {
            Fp64RealJob &j = jobs[i];
            const int64_t tm = (j.m + e - 1) / e, tn = (j.n + e - 1) / e;
            j.tiles_n = (int32_t)tn;
            j.tile_begin = total;
            total += j.lower ? tm * (tm + 1) / 2 : tm * tn;
        }
        *edge = e;
        if (total >= (int64_t)kSplitBelow * nsm) break;
    }
    return total;
}

cudaError_t launch_fp64_real(const Fp64RealJob *d_jobs, int num_jobs, int64_t tiles, int edge, cudaStream_t st) {
    if (tiles <= 0) return cudaSuccess;
    if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
    if (edge == 16) fp64_real_kernel<true><<<(unsigned)tiles, 128, 0, st>>>(d_jobs, num_jobs);
    else fp64_real_kernel<false><<<(unsigned)tiles, 128, 0, st>>>(d_jobs, num_jobs);
    return cudaGetLastError();
}

int64_t fp64_job_tiles(const Fp64Job &j) {
    const int64_t tm = (j.m + BM - 1) / BM, tn = (j.n + BN - 1) / BN;
    return j.lower ? tm * (tm + 1) / 2 : tm * tn;
}

cudaError_t launch_fp64_jobs(const Fp64Job *d_jobs, int num_jobs, int64_t total_tiles, cudaStream_t st) {
    if (total_tiles <= 0) return cudaSuccess;
    const size_t smem = sizeof(double2) * 2 * kStageElems;
    cudaError_t e = cudaFuncSetAttribute(fp64_jobs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fp64_jobs_kernel, kThreads, smem);
    const int64_t grid = std::min<int64_t>(total_tiles, (int64_t)nsm * std::max(per_sm, 1));
    fp64_jobs_kernel<<<(unsigned)grid, kThreads, smem, st>>>(d_jobs, num_jobs, total_tiles);
    return cudaGetLastError();
}

}  // namespace hsdla
