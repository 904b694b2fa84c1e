// Ozaki-split complex FP64 contractions on the FP8 tensor cores of sm_103a.
//
// Emulates the FP64 BLAS-3 work of create_HS2_stripped_v2
// (flapw_opt/src/h_and_s_stripped_v2.cpp:155-368: zherk, zher2k, zherkx and the
// per-atom zhemm/zgemm T application) with exact integer products on tcgen05:
//
//  * slicing (oz_slice_kernel): every column g of an operand Z (K x n) gets a
//    power-of-two exponent e_g with max_k |Re,Im Z_kg| < 2^e_g, and the scaled
//    column z = Z 2^-e_g is rounded to an integer X = rint(z 2^(5s-1)) that is
//    split into s balanced base-32 digits
//        z ~= sum_i d_i 2^(1-5i),  d_1 in [-16,16],  d_i in [-16,15]  (i >= 2).
//    Every digit is an integer of magnitude <= 16, exactly representable in
//    e4m3; one byte plane per (digit, re/im).  The digit extraction runs in
//    64-bit integer arithmetic (one FP64 multiply per weighted value):
//    GB300's FP64 pipe delivers ~1 TFLOP/s, its integer pipes far more.
//  * products (oz_gemm_kernel): for the output tile (rows g, cols g') and each
//    diagonal t = i + j of the digit-product triangle (t = 2..s+1), the FP32
//    TMEM accumulator sums, over the contraction index and all pairs (i, t-i),
//        Re += dr_i er_j + di_i ei_j,   Im += dr_i ei_j - di_i er_j
//    as kind::f8f6f4 MMAs (e4m3 x e4m3 -> f32).  Products are integers <= 256,
//    so a K chunk of at most 2^24 / (2 * 256 * pairs) complex terms keeps every
//    partial sum an exactly representable integer; chunks are drained into the
//    FP64 output tile with weight 2^(2-5t), and the last drain applies
//    2^(e_g + e_g').
//  * the structure-factor form's products are real ones (real_products.cu); here are the complex products of
//    the per-atom form, the contraction entry and the plugin (oz_pair_kernel on CTA pairs; oz_gemm_kernel
//    where no pairs are to be used), and the groups' set-up and runs.
//
// oz_gemm_kernel: persistent CTAs (one per SM, 512 TMEM columns = two 128x(128
// re + 128 im) FP32 accumulators), warp-specialised: one TMA producer warp
// (SW128 K-major 128x128-byte boxes, 64 KB per stage, 3 stages), one MMA warp
// (single elected issuer, tcgen05.commit to release stages and publish
// accumulators), eight epilogue warps (tcgen05.ld 32x32b, FP64 recombination,
// coalesced read-modify-write of the L2-resident output tile).  Every mbarrier
// wait is bounded by a clock64 budget; on expiry the kernel records an error
// word, stops issuing work, waits (bounded) for its in-flight copies and MMAs,
// frees TMEM and returns.
#include <cuda.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <type_traits>
#include <cstdio>
#include <cstring>
#include <vector>

#include "digits.cuh"
#include "ozaki.cuh"
#include "ptx.cuh"
#include "real_products.cuh"

namespace hsdla {

// Message of the last failed Ozaki call, per host thread: contexts driven from different threads
// never see each other's messages (each context copies it into its own message at once).
static thread_local const char *g_oz_err = "";
const char *ozaki_last_error() { return g_oz_err; }

namespace {

// ------------------------------------------------------------------ constants
constexpr int kTileM = 128;          // output rows per tile (TMEM lanes)
constexpr int kTileN = 128;          // output complex columns per tile
constexpr int kKBlock = 128;         // contraction bytes (e4m3 values) per stage
constexpr int kStages = 3;
constexpr int kStageBytes = 4 * kTileM * kKBlock;   // Ar, Ai, Br, Bi boxes
constexpr int kThreads = 320;        // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
constexpr int kEpiWarps = 8;         // two per TMEM lane quadrant, each drains half the columns
constexpr int kExactTerms = 1 << 24;                // FP32 exact-integer bound
constexpr int kSyncEvery = 64;                      // stages per lockstep epoch (cooperative launches)
constexpr int kRetired = 0x7F7F7F7F;                // progress value of a CTA that has no work left
constexpr int kErrWords = 8;                        // error word + diagnostics of the first expired wait
constexpr int kErrAlloc = 16;                       // error words + the wait self-test's progress slots

struct OzJob {
    int32_t lmap, rmap;        // tensor-map index (0..3) of the left / right digit operand
    int32_t lower;             // 1: only tiles and elements with row >= col
    int32_t accum;             // 1: the first unit of a tile adds to the output instead of storing
    int64_t lplane, rplane;    // rows per digit plane in each map
    int64_t lrow0, rrow0;      // first operand row (output row / col 0) inside a plane
    int64_t lk0, rk0;          // first contraction byte (multiple of 128)
    int64_t nkb;               // contraction blocks of 128
    int64_t m, n;              // valid output rows / cols
    int64_t tiles_n;           // tile columns (full mode)
    int64_t tile_begin;        // first global tile index
    double2 *out;
    int64_t ldo;
    const int32_t *el;         // exponent of each output row (job-relative)
    const int32_t *er;         // exponent of each output col (job-relative)
};

// kind::f8f6f4, A = B = e4m3, D = f32, both K-major, M = 128, N = 128
__host__ __device__ constexpr uint32_t idesc_f8(bool negA) {
    return (1u << 4) | (0u << 7) | (0u << 10) | ((negA ? 1u : 0u) << 13) | (0u << 14) | (0u << 15) | (0u << 16) |
           ((uint32_t)(kTileN >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

// ------------------------------------------------------- work decomposition
__device__ __forceinline__ int job_of(const OzJob *jobs, int num_jobs, int64_t tile) {
    int lo = 0, hi = num_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ void tile_coords(const OzJob &j, int64_t x, int64_t &tm, int64_t &tn) {
    if (j.lower) {
        tm = triangle_row(x);
        tn = x - tm * (tm + 1) / 2;
    } else {
        tm = x / j.tiles_n;
        tn = x - tm * j.tiles_n;
    }
}
// Tile g of the launch: from the host-built schedule (job, tm, tn) when given, else the
// jobs' own row-major order.
__device__ __forceinline__ const OzJob &resolve_tile(const OzJob *jobs, int num_jobs, const int4 *tile_list,
                                                     int64_t tile, int64_t &tm, int64_t &tn) {
    if (tile_list) {
        const int4 e = tile_list[tile];
        tm = e.y;
        tn = e.z;
        return jobs[e.x];
    }
    const OzJob &j = jobs[job_of(jobs, num_jobs, tile)];
    tile_coords(j, tile - j.tile_begin, tm, tn);
    return j;
}

// k-blocks per exact accumulation chunk on diagonal t (pairs = t - 1 for t <= s + 1)
__host__ __device__ __forceinline__ int64_t chunk_kblocks(int pairs) {
    const int64_t terms_per_kb = (int64_t)2 * kKBlock * pairs * 256;   // re/im products x max |product|
    int64_t c = kExactTerms / terms_per_kb;
    return c < 1 ? 1 : c;
}

// Loose grid-wide lockstep for cooperative launches: every producer publishes its stage epoch in
// its slot (one per CTA, or per CTA pair), and may run at most one epoch ahead of the slowest.  All persistent CTAs walk
// identical stage sequences, so staying within an epoch keeps the operand panels they share
// resident in L2 (left to themselves, CTAs drift apart by far more than L2 can hold).
// Bounded: on expiry the CTA raises the abort flag and records the error word.
__device__ bool grid_lockstep(int *progress, int n, int epoch, volatile int *abort_flag, int *err, int slot,
                              int slack = 1, long long budget = kWaitCycles) {
    atomicExch(progress + slot, epoch);
    const long long t0 = clock64();
    while (true) {
        int mn = kRetired;
        for (int i = 0; i < n; i += 4) {
            const int4 v = __ldcg(reinterpret_cast<const int4 *>(progress + i));
            mn = min(mn, min(min(v.x, v.y), min(v.z, v.w)));
        }
        if (mn >= epoch - slack) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > budget) {
            *abort_flag = 1;
            atomicCAS(err, 0, kDevTimeout * 16 + 5);
            return false;
        }
    }
}

// x * 2^k as a double for an FP32 accumulator x (a multiple of 2^-5 below 2^25), built with
// integer operations: GB300's FP64 pipe is a small fraction of its integer pipes, and a drain
// converts 2^16 values per CTA.  (f & 0x7fffffff) >> 3 puts the FP32 exponent and the top 20
// mantissa bits exactly where the FP64 high word keeps them, so rebasing the exponent is one
// add of (1023 - 127 + k) << 20; the low word takes the last 3 mantissa bits.  Valid for
// k in [kPow2Lo, kPow2Hi] (the result stays normal); pow2_ok() checks that once per column.
constexpr int kPow2Lo = -1017, kPow2Hi = 997;
__device__ __forceinline__ bool pow2_ok(int k) { return k >= kPow2Lo && k <= kPow2Hi; }
__device__ __forceinline__ double f32_pow2_to_f64_fast(uint32_t f, uint32_t ebias) {
    const uint32_t a = f & 0x7fffffffu;
    // a signed zero keeps its bits (high word = f, low word = 0)
    const uint32_t hi = a ? ((f & 0x80000000u) | ((a >> 3) + ebias)) : f;
    const uint32_t lo = f << 29;
    return __hiloint2double((int)hi, (int)lo);
}
__device__ __noinline__ double f32_pow2_to_f64_slow(uint32_t f, int k) { return ldexp((double)__uint_as_float(f), k); }
__device__ __forceinline__ uint32_t pow2_ebias(int k) { return (uint32_t)(1023 - 127 + k) << 20; }

// Drain 32 accumulator columns of one output row: out = (out +) x 2^(kb + e_col) with kb =
// 2 - 5t + e_row (a plain store on the first unit of a tile).  Every unit carries its full scale,
// so an output that already holds an earlier panel's sum is accumulated correctly.  Loads are
// grouped kDrainBatch at a time ahead of the stores (the compiler cannot reorder a load past a
// store to a possibly aliasing column), so a drain costs a few L2 round trips per 32 columns.
constexpr int kDrainBatch = 8;
__device__ __forceinline__ void drain32(const OzJob &j, int64_t row, int64_t col0, const uint32_t (&vre)[32],
                                        const uint32_t (&vim)[32], int kb, bool first) {
#pragma unroll
    for (int h = 0; h < 32; h += kDrainBatch) {
        double2 o[kDrainBatch];
#pragma unroll
        for (int cc = 0; cc < kDrainBatch; ++cc) {
            const int64_t col = col0 + h + cc;
            const bool live = col < j.n && !(j.lower && row < col);
            o[cc] = (live && !first) ? __ldcg(j.out + row + j.ldo * col) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int cc = 0; cc < kDrainBatch; ++cc) {
            const int64_t col = col0 + h + cc;
            if (col >= j.n || (j.lower && row < col)) continue;
            const int k = kb + j.er[col];
            double re, im;
            if (pow2_ok(k)) {
                const uint32_t eb = pow2_ebias(k);
                re = f32_pow2_to_f64_fast(vre[h + cc], eb);
                im = f32_pow2_to_f64_fast(vim[h + cc], eb);
            } else {
                re = f32_pow2_to_f64_slow(vre[h + cc], k);
                im = f32_pow2_to_f64_slow(vim[h + cc], k);
            }
            j.out[row + j.ldo * col] = make_double2(re + o[cc].x, im + o[cc].y);
        }
    }
}

struct __align__(8) Barriers {
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t tfull[2];
    uint64_t tempty[2];
};

__global__ void __launch_bounds__(kThreads, 1)
    oz_gemm_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
                   const __grid_constant__ CUtensorMap map2, const __grid_constant__ CUtensorMap map3,
                   const OzJob *__restrict__ jobs, int num_jobs, int64_t total_tiles, int s, int *err,
                   const int4 *__restrict__ tile_list, int *progress) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1024-byte alignment of the stage buffers (SW128 atoms)
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ Barriers bars;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto map_of = [&](int i) -> const CUtensorMap * {
        return i == 0 ? &map0 : i == 1 ? &map1 : i == 2 ? &map2 : &map3;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) { mbar_init(&bars.full[i], 1); mbar_init(&bars.empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&bars.tfull[i], 1); mbar_init(&bars.tempty[i], 32 * kEpiWarps); }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int i = 0; i < 4; ++i) asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)map_of(i)) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_base_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_sh;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int64_t issued = 0;
            bool ok = true;
            for (int64_t tile = blockIdx.x; ok && tile < total_tiles; tile += gridDim.x) {
                int64_t tm, tn;
                const OzJob &j = resolve_tile(jobs, num_jobs, tile_list, tile, tm, tn);
                const CUtensorMap *lm = map_of(j.lmap), *rm = map_of(j.rmap);
                for (int t = 2; ok && t <= s + 1; ++t) {
                    const int ilo = max(1, t - s), ihi = min(s, t - 1);
                    const int64_t ck = chunk_kblocks(ihi - ilo + 1);
                    for (int64_t cb = 0; ok && cb < j.nkb; cb += ck) {
                        const int64_t ce = min(j.nkb, cb + ck);
                        for (int64_t kb = cb; ok && kb < ce; ++kb) {
                            for (int i = ilo; i <= ihi; ++i) {
                                const int jj = t - i;
                                if (progress && issued > 0 && issued % kSyncEvery == 0 &&
                                    !grid_lockstep(progress, (int)gridDim.x, (int)(issued / kSyncEvery), &abort_flag,
                                                   err, (int)blockIdx.x)) { ok = false; break; }
                                if (!mbar_wait(&bars.empty[stage], phase ^ 1, &abort_flag, err, 1)) { ok = false; break; }
                                unsigned char *st = smem + stage * kStageBytes;
                                mbar_expect_tx(&bars.full[stage], kStageBytes);
                                const int xl = (int)(j.lk0 + kb * kKBlock), xr = (int)(j.rk0 + kb * kKBlock);
                                const int64_t yl = j.lrow0 + tm * kTileM, yr = j.rrow0 + tn * kTileN;
                                tma_load_2d(st, lm, &bars.full[stage], xl, (int)((2 * (i - 1)) * j.lplane + yl));
                                tma_load_2d(st + 16384, lm, &bars.full[stage], xl, (int)((2 * (i - 1) + 1) * j.lplane + yl));
                                tma_load_2d(st + 32768, rm, &bars.full[stage], xr, (int)((2 * (jj - 1)) * j.rplane + yr));
                                tma_load_2d(st + 49152, rm, &bars.full[stage], xr, (int)((2 * (jj - 1) + 1) * j.rplane + yr));
                                ++issued;
                                if (++stage == kStages) { stage = 0; phase ^= 1; }
                            }
                        }
                    }
                }
            }
            if (progress) atomicExch(progress + blockIdx.x, kRetired);
            // drain: every issued stage must have landed before the CTA may exit
            if (!ok) {
                for (int q = 0; q < kStages; ++q) {
                    // the last kStages issued stages are the only ones possibly in flight
                    if (issued == 0) break;
                    if (--stage < 0) { stage = kStages - 1; phase ^= 1; }
                    mbar_drain_wait(&bars.full[stage], phase);
                    --issued;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int64_t unit = 0;
            bool ok = true;
            const uint32_t id_pos = idesc_f8(false), id_neg = idesc_f8(true);
            const uint32_t sbase = smem_u32(smem);
            for (int64_t tile = blockIdx.x; ok && tile < total_tiles; tile += gridDim.x) {
                int64_t tm_, tn_;
                const OzJob &j = resolve_tile(jobs, num_jobs, tile_list, tile, tm_, tn_);
                for (int t = 2; ok && t <= s + 1; ++t) {
                    const int ilo = max(1, t - s), ihi = min(s, t - 1);
                    const int64_t ck = chunk_kblocks(ihi - ilo + 1);
                    for (int64_t cb = 0; ok && cb < j.nkb; cb += ck) {
                        const int64_t ce = min(j.nkb, cb + ck);
                        const int buf = (int)(unit & 1);
                        const uint32_t uphase = (uint32_t)((unit >> 1) & 1);
                        if (!mbar_wait(&bars.tempty[buf], uphase ^ 1, &abort_flag, err, 2)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t d_re = tmem_base + buf * 256, d_im = d_re + 128;
                        bool first = true;
                        for (int64_t kb = cb; ok && kb < ce; ++kb) {
                            for (int i = ilo; i <= ihi; ++i) {
                                if (!mbar_wait(&bars.full[stage], phase, &abort_flag, err, 3)) { ok = false; break; }
                                tc_fence_after();
                                const uint32_t a_re = sbase + stage * kStageBytes, a_im = a_re + 16384;
                                const uint32_t b_re = a_re + 32768, b_im = a_re + 49152;
#pragma unroll
                                for (int kk = 0; kk < kKBlock / 32; ++kk) {
                                    const uint32_t off = kk * 32;
                                    const uint32_t acc = first ? 0u : 1u;
                                    mma_f8(d_re, sw128_desc(a_re + off), sw128_desc(b_re + off), id_pos, acc);
                                    mma_f8(d_re, sw128_desc(a_im + off), sw128_desc(b_im + off), id_pos, 1u);
                                    mma_f8(d_im, sw128_desc(a_re + off), sw128_desc(b_im + off), id_pos, acc);
                                    mma_f8(d_im, sw128_desc(a_im + off), sw128_desc(b_re + off), id_neg, 1u);
                                    first = false;
                                }
                                mma_commit(&bars.empty[stage]);
                                if (++stage == kStages) { stage = 0; phase ^= 1; }
                            }
                        }
                        if (!ok) break;
                        mma_commit(&bars.tfull[buf]);
                        ++unit;
                    }
                }
            }
            // wait for the MMAs still in flight before TMEM is freed
            if (unit > 0) {
                const int64_t u = unit - 1;
                mbar_drain_wait(&bars.tfull[u & 1], (uint32_t)((u >> 1) & 1));
            }
            if (!ok) {
                // a partially issued unit may still be running: commit and wait for it too
                mma_commit(&bars.tfull[unit & 1]);
                mbar_drain_wait(&bars.tfull[unit & 1], (uint32_t)((unit >> 1) & 1));
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..9)
        const int q = warp & 3;                      // TMEM lane quadrant of this warp
        const int cbeg = ((warp - 2) >> 2) * (kTileN / 2);   // its half of the columns
        const int r_in_tile = q * 32 + lane;
        int64_t unit = 0;
        bool ok = true;
        for (int64_t tile = blockIdx.x; ok && tile < total_tiles; tile += gridDim.x) {
            int64_t tm, tn;
            const OzJob &j = resolve_tile(jobs, num_jobs, tile_list, tile, tm, tn);
            const int64_t row = tm * kTileM + r_in_tile;
            const bool row_ok = row < j.m;
            const int erow = row_ok ? j.el[row] : 0;
            for (int t = 2; ok && t <= s + 1; ++t) {
                const int ilo = max(1, t - s), ihi = min(s, t - 1);
                const int64_t ck = chunk_kblocks(ihi - ilo + 1);
                for (int64_t cb = 0; ok && cb < j.nkb; cb += ck) {
                    const bool first = (t == 2 && cb == 0) && !j.accum;
                    const int buf = (int)(unit & 1);
                    const uint32_t uphase = (uint32_t)((unit >> 1) & 1);
                    if (!mbar_wait(&bars.tfull[buf], uphase, &abort_flag, err, 4)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256;
#pragma unroll 1
                    for (int c0 = cbeg; c0 < cbeg + kTileN / 2; c0 += 32) {
                        uint32_t vre[32], vim[32];
                        tmem_ld32(tbase + c0, vre);
                        tmem_ld32(tbase + 128 + c0, vim);
                        tmem_ld_wait();
                        if (c0 + 32 >= cbeg + kTileN / 2) {
                            tc_fence_before();
                            mbar_arrive(&bars.tempty[buf]);
                        }
                        if (row_ok) drain32(j, row, tn * kTileN + c0, vre, vim, 2 - 5 * t + erow, first);
                    }
                    ++unit;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem_base) : "memory");
    }
}

// ------------------------------------------------------- CTA-pair products
// The S/H launch on 2-CTA tiles: a cluster of two CTAs (one per SM) computes a 256 x 256
// output tile with tcgen05.mma.cta_group::2 (M = 256, N = 256).  Each CTA stages its own half
// of the left operand (128 rows) and its own half of the right operand (128 rows) per k-block,
// so an MMA of twice the 1-CTA tile's flops reads the same 8 KB of shared memory per SM, and TMA
// writes half the bytes per flop.  Each CTA's TMEM holds its 128 output rows x (256 re + 256 im)
// FP32 columns (single-buffered: an exact-accumulation unit runs ~10^5 cycles, its drain a few
// 10^3).  Roles:
//   leader (cluster rank 0): TMA for its halves, expect_tx for both CTAs' bytes on its full
//     barrier, the single MMA issuer, commits multicast to both CTAs' empty / tfull barriers;
//   peer (rank 1): TMA for its halves completing on the leader's full barrier (.cta_group::2);
//   both: eight epilogue warps drain their own TMEM rows and arrive on the leader's tempty.
// Every wait is bounded as in oz_gemm_kernel; both CTAs meet at a cluster barrier before TMEM
// is freed, so no CTA exits while its shared memory or TMEM can still be addressed by the other.
constexpr int kPairTile = 256;
// Epilogue warps of the pair kernel: four per TMEM lane quadrant (each drains a quarter of the
// columns) hide the drain's latencies twice as well as two; HSDLA_PAIR_EPI_WARPS=8 builds two.
#ifndef HSDLA_PAIR_EPI_WARPS
#define HSDLA_PAIR_EPI_WARPS 16
#endif
constexpr int kPairEpiWarps = HSDLA_PAIR_EPI_WARPS;
constexpr int kPairThreads = 64 + 32 * kPairEpiWarps;      // warp 0 TMA, warp 1 MMA, the rest epilogue
constexpr int kColsPerWarp = 4 * kPairTile / kPairEpiWarps;
constexpr int kChunksPerWarp = kColsPerWarp / 32;
static_assert(kChunksPerWarp >= 1 && kColsPerWarp % 32 == 0, "epilogue column split");
// TMEM columns per load (re and im each): 16 with four epilogue warps per quadrant (18 warps leave
// 96 registers a thread), 32 with two
constexpr int kLdColsPair() { return kPairEpiWarps > 8 ? 16 : 32; }
constexpr int kLdCols = kLdColsPair();
// Operand stages of the pair kernel and the drain staging that shares its shared memory (over the
// epilogue warps, kDrainBufs buffers each: a warp fills one while the bulk copies of the others
// read them).  The drain's throughput is bounded by the staging bytes in flight.
#ifndef HSDLA_PAIR_STAGES
#define HSDLA_PAIR_STAGES 3
#endif
#ifndef HSDLA_PAIR_STAGING_KB
#define HSDLA_PAIR_STAGING_KB 32
#endif
// Drain staging buffers per epilogue warp: one buffer of 4 columns (2 KB) per warp drains with
// half the proxy fences and read-waits of two 2-column buffers; c2's per-type S/H launches took
// 23.35-23.41 ms against 24.37-24.43 (two buffers) and 27.8 ms (four) on one GB300, builds alternating.
#ifndef HSDLA_DRAIN_BUFS
#define HSDLA_DRAIN_BUFS 1
#endif
constexpr int kPairStages = HSDLA_PAIR_STAGES;
constexpr int kDrainBufs = HSDLA_DRAIN_BUFS;
constexpr int kStageCols = HSDLA_PAIR_STAGING_KB * 1024 / kPairEpiWarps / kDrainBufs / 512;   // columns per buffer
constexpr int kStageWarpBytes = kDrainBufs * kStageCols * 32 * 16;   // buffers x columns x 32 rows x 16 B
static_assert(kStageCols >= 1 && kLdColsPair() % kStageCols == 0, "drain staging shape");

constexpr int kPairStageBytes = kPairEpiWarps * kStageWarpBytes;
// Bulk copies and f64 add-reductions shared memory -> global with an L2 eviction policy
// (createpolicy): an output tile stays resident through its units (evict_last) and leaves first
// after its last one (evict_first).
__device__ __forceinline__ void bulk_store_g(void *gdst, uint32_t ssrc, uint32_t bytes, uint64_t pol) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;\n" ::"l"(gdst),
                 "r"(ssrc), "r"(bytes), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void bulk_add_g(void *gdst, uint32_t ssrc, uint32_t bytes, uint64_t pol) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.L2::cache_hint.add.f64 [%0], [%1], %2, %3;\n" ::"l"(
                     gdst),
                 "r"(ssrc), "r"(bytes), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
    return p;
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

#ifndef HSDLA_COLLECTOR_A
#define HSDLA_COLLECTOR_A 1
#endif
struct __align__(8) PairBarriers {
    uint64_t full[kPairStages];   // leader: both CTAs' bytes of a stage landed
    uint64_t empty[kPairStages];  // each CTA: the stage's MMAs completed (multicast commit)
    uint64_t tfull;              // each CTA: the accumulator is complete (multicast commit)
    uint64_t tempty;             // leader: the epilogue warps of both CTAs drained it
};

constexpr size_t kPairSmem = (size_t)kPairStages * kStageBytes + kPairStageBytes + 1024;
static_assert(kPairSmem <= 227 * 1024, "pair kernel shared memory");
__host__ __device__ constexpr uint32_t idesc_f8_pair(bool negA) {
    return (1u << 4) | ((negA ? 1u : 0u) << 13) | ((uint32_t)(kPairTile >> 3) << 17) |
           ((uint32_t)(kPairTile >> 4) << 24);
}

__global__ void __launch_bounds__(kPairThreads, 1)
    oz_pair_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
                   const __grid_constant__ CUtensorMap map2, const __grid_constant__ CUtensorMap map3,
                   const OzJob *__restrict__ jobs, int num_jobs, int64_t total_tiles, int s, int *err,
                   const int4 *__restrict__ tile_list, int *progress, int sync_every, int slack,
                   const int4 *__restrict__ parts, double2 *slabs) {
    constexpr int kStages = kPairStages;
    constexpr int kStageB = kStageBytes;
    constexpr int kN = kPairTile;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ PairBarriers bars;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // launched as clusters of two or not at all: nothing below (the pair TMEM allocation above
    // all) is valid otherwise
    if (cluster_size() != 2) {
        if (threadIdx.x == 0) atomicCAS(err, 0, kDevBadInput * 16 + 6);
        return;
    }
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    // bounded wait that records where it expired (first failure wins)
    auto expired = [&](uint32_t parity, int stage_, int count) -> bool {
        if (atomicCAS(err + 7, 0, 1) == 0) {
            err[1] = blockIdx.x; err[2] = (int)rank; err[3] = stage_; err[4] = (int)parity; err[5] = count;
        }
        return false;
    };
    auto pwait = [&](uint64_t *bar, uint32_t parity, int where, int stage_, int count) -> bool {
        return mbar_wait(bar, parity, &abort_flag, err, where) || expired(parity, stage_, count);
    };
    auto pwait_pair = [&](uint64_t *bar, uint32_t parity, int where, int stage_, int count) -> bool {
        return mbar_wait<true>(bar, parity, &abort_flag, err, where) || expired(parity, stage_, count);
    };
    const int64_t pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    auto map_of = [&](int i) -> const CUtensorMap * {
        return i == 0 ? &map0 : i == 1 ? &map1 : i == 2 ? &map2 : &map3;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) { mbar_init(&bars.full[i], 1); mbar_init(&bars.empty[i], 1); }
        mbar_init(&bars.tfull, 1);
        mbar_init(&bars.tempty, 2 * kPairEpiWarps);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int i = 0; i < 4; ++i) asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)map_of(i)) : "memory");
    }
    if (warp == 1) {
        // collective over the pair: one warp of each CTA
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_base_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // barriers of both CTAs initialised before any remote arrival
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    const uint32_t full0_leader = mapa_rank(smem_u32(&bars.full[0]), 0);
    const uint32_t tempty_leader = mapa_rank(smem_u32(&bars.tempty), 0);
    // the steps (digit pair and k-block, in the order of the loops) [x, y) of an entry, and its slab z
    auto part_of = [&](int64_t tile) { return parts ? parts[tile] : make_int4(0, INT_MAX, -1, 0); };
    const int64_t half = (int64_t)rank * (kPairTile / 2);     // this CTA's rows of a tile, and of the right operand

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producers (both CTAs)
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int64_t issued = 0;
            bool ok = true;
            for (int64_t tile = pair; ok && tile < total_tiles; tile += npairs) {
                int64_t tm, tn;
                const OzJob &j = resolve_tile(jobs, num_jobs, tile_list, tile, tm, tn);
                const CUtensorMap *lm = map_of(j.lmap), *rm = map_of(j.rmap);
                const int4 part = part_of(tile);
                int step = 0;
                for (int t = 2; ok && t <= s + 1; ++t) {
                    const int ilo = max(1, t - s), ihi = min(s, t - 1);
                    const int64_t ck = chunk_kblocks(ihi - ilo + 1);
                    for (int64_t cb = 0; ok && cb < j.nkb; cb += ck) {
                        const int64_t ce = min(j.nkb, cb + ck);
                        const int end = step + (int)(ce - cb) * (ihi - ilo + 1);
                        if (end <= part.x || step >= part.y) { step = end; continue; }
                        for (int64_t kb = cb; ok && kb < ce; ++kb) {
                            for (int i = ilo; i <= ihi; ++i, ++step) {
                                if (step < part.x || step >= part.y) continue;
                                const int jj = t - i;
                                if (leader && progress && issued > 0 && issued % sync_every == 0 &&
                                    !grid_lockstep(progress, (int)npairs, (int)(issued / sync_every), &abort_flag, err,
                                                   (int)pair, slack)) { ok = false; break; }
                                if (!pwait(&bars.empty[stage], phase ^ 1, 1, stage, (int)issued)) { ok = false; break; }
                                unsigned char *st = smem + stage * kStageB;
                                if (leader) mbar_expect_tx(&bars.full[stage], 2 * kStageB);
                                const uint32_t fb = full0_leader + stage * 8;
                                const int xl = (int)(j.lk0 + kb * kKBlock), xr = (int)(j.rk0 + kb * kKBlock);
                                const int64_t yl = j.lrow0 + tm * kPairTile + half, yr = j.rrow0 + tn * kPairTile + half;
                                tma_load_2d_pair(st, lm, fb, xl, (int)((2 * (i - 1)) * j.lplane + yl));
                                tma_load_2d_pair(st + 16384, lm, fb, xl, (int)((2 * (i - 1) + 1) * j.lplane + yl));
                                tma_load_2d_pair(st + 32768, rm, fb, xr, (int)((2 * (jj - 1)) * j.rplane + yr));
                                tma_load_2d_pair(st + 49152, rm, fb, xr, (int)((2 * (jj - 1) + 1) * j.rplane + yr));
                                ++issued;
                                if (++stage == kStages) { stage = 0; phase ^= 1; }
                            }
                        }
                    }
                }
            }
            if (leader && progress) atomicExch(progress + pair, kRetired);
            // Before exit every stage this CTA issued must have been consumed: its bytes landed and
            // the MMA commit that frees it (multicast, possibly remote) arrived.  Normally these
            // waits return at once; after an abort they are bounded.
            for (int q = 0; q < kStages && issued > 0; ++q) {
                if (--stage < 0) { stage = kStages - 1; phase ^= 1; }
                mbar_drain_wait(&bars.empty[stage], phase);
                --issued;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        if (lane == 0 && leader) {
            int stage = 0;
            uint32_t phase = 0;
            int64_t unit = 0;            // units issued
            bool ok = true;
            const uint32_t id_pos = idesc_f8_pair(false), id_neg = idesc_f8_pair(true);
            const uint32_t sbase = smem_u32(smem);
            const uint32_t d_re = tmem_base, d_im = d_re + kN;
            for (int64_t tile = pair; ok && tile < total_tiles; tile += npairs) {
                int64_t tm_, tn_;
                const OzJob &j = resolve_tile(jobs, num_jobs, tile_list, tile, tm_, tn_);
                // the job's fields in registers: the asm statements below clobber memory, and the
                // issuer must not reload them between MMAs
                const int64_t jnkb = j.nkb;
                const int4 part = part_of(tile);
                int step = 0;
                for (int t = 2; ok && t <= s + 1; ++t) {
                    const int ilo = max(1, t - s), ihi = min(s, t - 1);
                    const int64_t ck = chunk_kblocks(ihi - ilo + 1);
                    for (int64_t cb = 0; ok && cb < jnkb; cb += ck) {
                        const int64_t ce = min(jnkb, cb + ck);
                        const int end = step + (int)(ce - cb) * (ihi - ilo + 1);
                        if (end <= part.x || step >= part.y) { step = end; continue; }
                        if (!pwait_pair(&bars.tempty, (uint32_t)((unit & 1) ^ 1), 2, stage, (int)unit)) { ok = false; break; }
                        tc_fence_after();
                        bool first = true;
                        for (int64_t kb = cb; ok && kb < ce; ++kb) {
                            for (int i = ilo; i <= ihi; ++i, ++step) {
                                if (step < part.x || step >= part.y) continue;
                                if (!pwait(&bars.full[stage], phase, 3, stage, (int)unit)) { ok = false; break; }
                                tc_fence_after();
                                const uint32_t a_re = sbase + stage * kStageB, a_im = a_re + 16384;
                                const uint32_t b_re = a_re + 32768, b_im = a_re + 49152;
                                // The stage's four descriptors once; a 32-byte step along K adds 2
                                // to the start-address field (16-byte units; shared-memory
                                // addresses stay below 2^18, so the field never carries).
                                const uint64_t dar = sw128_desc(a_re), dai = sw128_desc(a_im);
                                const uint64_t dbr = sw128_desc(b_re), dbi = sw128_desc(b_im);
#pragma unroll
                                for (int kk = 0; kk < kKBlock / 32; ++kk) {
                                    const uint64_t o = 2u * kk;
                                    const uint32_t acc = first ? 0u : 1u;
#if HSDLA_COLLECTOR_A
                                    // the two MMAs of the real left plane back to back, the
                                    // second taking A from the collector buffer.  (Not for
                                    // the imaginary plane: an MMA that reads A from the
                                    // collector does not apply the negate-A bit, measured:
                                    // the -A_im B_re term came out as +A_im B_re.)
                                    mma_f8_pair_ca<true>(d_re, dar + o, dbr + o, id_pos, acc);
                                    mma_f8_pair_ca<false>(d_im, dar + o, dbi + o, id_pos, acc);
                                    mma_f8_pair(d_re, dai + o, dbi + o, id_pos, 1u);
                                    mma_f8_pair(d_im, dai + o, dbr + o, id_neg, 1u);
#else
                                    mma_f8_pair(d_re, dar + o, dbr + o, id_pos, acc);
                                    mma_f8_pair(d_re, dai + o, dbi + o, id_pos, 1u);
                                    mma_f8_pair(d_im, dar + o, dbi + o, id_pos, acc);
                                    mma_f8_pair(d_im, dai + o, dbr + o, id_neg, 1u);
#endif
                                    first = false;
                                }
                                mma_commit_pair(&bars.empty[stage]);
                                if (++stage == kStages) { stage = 0; phase ^= 1; }
                            }
                        }
                        if (!ok) break;
                        mma_commit_pair(&bars.tfull);
                        ++unit;
                    }
                }
            }
            if (!ok) {
                // a partially issued unit may still be running: commit it and wait (bounded)
                mma_commit_pair(&bars.tfull);
                mbar_drain_wait(&bars.tfull, (uint32_t)(unit & 1));
            } else if (unit > 0) {
                // the last unit's MMAs and both CTAs' drains of it
                mbar_drain_wait(&bars.tfull, (uint32_t)((unit - 1) & 1));
                mbar_drain_wait(&bars.tempty, (uint32_t)((unit - 1) & 1));
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2.., both CTAs)
        // A unit's drain: TMEM -> registers -> FP64 with the full scale 2^(2-5t+e_row+e_col) (built
        // with integer operations) -> the output: a plain store for the tile's first unit,
        // fire-and-forget f64 reductions in L2 for the others.  Each lane owns one output row, so
        // successive updates of an element come from one thread and stay in program order; the
        // SM never waits on the output.  Only stored elements (row < m, col < n, lower: row >=
        // col) are written.
        constexpr int kCols = kColsPerWarp, kCh = kChunksPerWarp;
        const int q = warp & 3;                      // TMEM lane quadrant of this warp
        const int cbeg = ((warp - 2) >> 2) * kCols;  // its share of a buffer's columns
        unsigned char *stg = smem + kStages * kStageB + (warp - 2) * kStageWarpBytes;
        const uint32_t stg_s = smem_u32(stg);
        const uint64_t pol_last = policy_evict_last(), pol_first = policy_evict_first();
        int64_t unit = 0;
        int rd = 0;                                  // staged buffers so far (the ring position)
        bool ok = true;
        for (int64_t tile = pair; ok && tile < total_tiles; tile += npairs) {
            int64_t tm, tn;
            const OzJob &j = resolve_tile(jobs, num_jobs, tile_list, tile, tm, tn);
            const int64_t r0 = tm * kPairTile + half + q * 32, row = r0 + lane;
            const int64_t m = j.m, n = j.n;
            const int nkb = (int)j.nkb;
            const bool lower = j.lower != 0;
            const int erow = row < m ? j.el[row] : 0;
            // a later part of a tile goes to a slab of its own
            int64_t ldo = j.ldo;
            double2 *out = j.out;
            bool fresh = j.accum == 0;
            int from = 0, to = INT_MAX;
            if (parts) {
                const int4 part = parts[tile];
                from = part.x;
                to = part.y;
                if (part.z >= 0) {
                    ldo = kPairTile;
                    out = slabs + (int64_t)part.z * kPairTile * kPairTile - tm * kPairTile - tn * kPairTile * ldo;
                    fresh = true;
                }
            }
            int step = 0;
            // The tile's column exponents, loaded once for all its units: lane l holds column
            // tn*256 + cbeg + 32c + l of chunk c in ex[c], with each chunk's
            // range for the fast-path test.  The registers rotate after each chunk, so the current
            // chunk's are always in ex[0] (after a unit's chunks they are back in order).
            const int32_t *er = j.er;
            int ex[kCh], exlo[kCh], exhi[kCh];
#pragma unroll
            for (int x = 0; x < kCh; ++x) {
                const int64_t col = tn * kPairTile + cbeg + 32 * x + lane;
                ex[x] = col < n ? __ldg(er + col) : 0;
            }
#pragma unroll
            for (int x = 0; x < kCh; ++x) {
                exlo[x] = __reduce_min_sync(0xffffffffu, ex[x]);
                exhi[x] = __reduce_max_sync(0xffffffffu, ex[x]);
            }
            for (int t = 2; ok && t <= s + 1; ++t) {
                const int cnt = min(s, t - 1) - max(1, t - s) + 1;
                const int ck = (int)min((int64_t)nkb, chunk_kblocks(cnt));
                const int kb = 2 - 5 * t + erow;
                // 2^(kb + e_col) as an FP64 exponent bias: the row's part plus e_col << 20
                const uint32_t rbias = pow2_ebias(kb);
                for (int cb = 0; ok && cb < nkb; cb += ck) {
                    const int end = step + (min(nkb, cb + ck) - cb) * cnt;
                    const bool none = end <= from || step >= to;
                    step = end;
                    if (none) continue;
                    const bool first = fresh;
                    fresh = false;
                    const uint64_t pol = ((t == s + 1 && cb + ck >= nkb) || end >= to) ? pol_first : pol_last;
                    {
                        if (!pwait(&bars.tfull, (uint32_t)(unit & 1), 4, warp, (int)unit)) { ok = false; break; }
                        tc_fence_after();
                        // the previous unit's copies are complete: successive updates stay in order
                        if (lane < kStageCols) bulk_wait_all();
                        const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
                        for (int c = 0; c < kCh; ++c) {
                            const int64_t colb = tn * kPairTile + cbeg + 32 * c;
                            const bool fast = __all_sync(0xffffffffu, pow2_ok(kb + exlo[0]) && pow2_ok(kb + exhi[0]));
#pragma unroll
                            for (int hh = 0; hh < 32; hh += kLdCols) {
                                uint32_t vre[kLdCols], vim[kLdCols];
                                tmem_ld<kLdCols>(tbase + cbeg + 32 * c + hh, vre);
                                tmem_ld<kLdCols>(tbase + kN + cbeg + 32 * c + hh, vim);
                                tmem_ld_wait();
                                if (c == kCh - 1 && hh + kLdCols >= 32) {
                                    tc_fence_before();
                                    __syncwarp();
                                    if (lane == 0) mbar_arrive_pair(tempty_leader);
                                }
#pragma unroll
                                for (int g4 = 0; g4 < kLdCols; g4 += kStageCols, ++rd) {
                                    const uint32_t buf = (uint32_t)(rd % kDrainBufs) * (kStageCols * 512);
                                    if (lane < kStageCols) bulk_wait_read<kDrainBufs - 1>();
                                    __syncwarp();
#pragma unroll
                                    for (int cc = 0; cc < kStageCols; ++cc) {
                                        const int cl = g4 + cc;
                                        const int ec = __shfl_sync(0xffffffffu, ex[0], hh + cl);
                                        double re, im;
                                        if (fast) {
                                            const uint32_t eb = rbias + ((uint32_t)ec << 20);
                                            re = f32_pow2_to_f64_fast(vre[cl], eb);
                                            im = f32_pow2_to_f64_fast(vim[cl], eb);
                                        } else {
                                            re = f32_pow2_to_f64_slow(vre[cl], kb + ec);
                                            im = f32_pow2_to_f64_slow(vim[cl], kb + ec);
                                        }
                                        *reinterpret_cast<double2 *>(stg + buf + cc * 512 + lane * 16) = make_double2(re, im);
                                    }
                                    fence_async_smem();
                                    __syncwarp();
                                    // lane cc issues the copy of the group's column cc (32 rows) and commits it
                                    if (lane < kStageCols) {
                                        const int64_t col = colb + hh + g4 + lane;
                                        const int64_t lo = lower ? max(r0, col) : r0, hi = min(r0 + 32, m);
                                        if (col < n && lo < hi) {
                                            const uint32_t src = stg_s + buf + lane * 512 + (uint32_t)(lo - r0) * 16;
                                            double2 *dst = out + lo + ldo * col;
                                            if (first) bulk_store_g(dst, src, (uint32_t)(hi - lo) * 16, pol);
                                            else bulk_add_g(dst, src, (uint32_t)(hi - lo) * 16, pol);
                                        }
                                        bulk_commit();
                                    }
                                }
                            }
                            // the next chunk's exponents into ex[0]
                            const int xe = ex[0], xl = exlo[0], xh = exhi[0];
#pragma unroll
                            for (int x = 0; x + 1 < kCh; ++x) {
                                ex[x] = ex[x + 1];
                                exlo[x] = exlo[x + 1];
                                exhi[x] = exhi[x + 1];
                            }
                            ex[kCh - 1] = xe;
                            exlo[kCh - 1] = xl;
                            exhi[kCh - 1] = xh;
                        }
                    }
                    ++unit;
                }
            }
        }
        // every copy complete before the CTA may exit
        if (lane < kStageCols) bulk_wait_all();
    }
    tc_fence_before();
    __syncwarp();
    __syncthreads();
    cluster_sync_all();          // neither CTA frees TMEM or exits while the other may address it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(tmem_base) : "memory");
    }
}

// The slabs of a split tile into the output, in the order of its parts (adds: job, tile row, tile
// column, first slab; then their number).  A block per column of a tile, lanes along its rows.
__global__ void __launch_bounds__(kPairTile) oz_slab_add_kernel(const OzJob *__restrict__ jobs, const int4 *__restrict__ adds,
                                                                const double2 *__restrict__ slabs) {
    const int4 a = adds[2 * blockIdx.x];
    const int count = adds[2 * blockIdx.x + 1].x;
    const OzJob &j = jobs[a.x];
    const int64_t row = (int64_t)a.y * kPairTile + threadIdx.x;
    if (row >= j.m) return;
    const int64_t col = (int64_t)a.z * kPairTile + blockIdx.y;
    if (col >= j.n || (j.lower && row < col)) return;
    const double2 *p = slabs + ((int64_t)a.w * kPairTile + blockIdx.y) * kPairTile + threadIdx.x;
    double2 v = j.out[row + j.ldo * col];
#pragma unroll 8
    for (int q = 0; q < count; ++q, p += kPairTile * kPairTile) {
        const double2 x = __ldcs(p);
        v.x += x.x;
        v.y += x.y;
    }
    j.out[row + j.ldo * col] = v;
}

// --------------------------------------------------------------- slicing
// Digit planes of Z (Kin x ncols, column-major, ld ldz) with optional row weights v:
// padded contraction layout: source rows [b*rpb, (b+1)*rpb) land at [b*bpad, b*bpad + rpb).
//
// One CTA per plane row (= source column), 512 threads and one CTA per SM, which keeps the
// column set in flight (152 x <= 0.5 MB) inside L2: pass 1 reads the column from HBM for its
// exponent, pass 2 re-reads it from L2 and writes the digits.  Digit extraction without carries:
// with B = 16 (1 + 32 + ... + 32^(s-2)), the balanced digits d_i in [-16, 15] (i >= 2) of X are
// the 5-bit fields of U = X + B minus 16, and the top digit is U >> 5(s-1) in [-16, 16]; digits
// are encoded two at a time by the hardware f32 -> e4m3x2 conversion (exact for |d| <= 16).
// A dual table slices the same source twice in one pass (C unweighted and W = C with row
// weights), reading the source once.
constexpr int kSliceThreads = 512;
constexpr int kSliceVec = 8;       // consecutive contraction bytes per thread and plane

// One slicing launch covers an operand for every k-point of a group: the k-points' columns
// are stacked as consecutive rows of each digit plane (row0 of an entry = its first row).
struct SliceEntry {
    const double2 *Z;          // source K x ncols, column-major, ld SliceTab::ldz
    int64_t ncols;
    int64_t row0;
};
struct SliceTab {
    int nk = 0;
    int s = 0;
    int64_t ldz = 0, Kin = 0, rpb = 0, bpad = 0;
    const double *v = nullptr;          // optional per-row weights (K)
    uint8_t *digits = nullptr;
    int64_t Kpad = 0, plane_rows = 0, pitch = 0;
    int32_t *expo = nullptr;            // exponent of each plane row
    // dual: a second digit operand of the same geometry from the same source with weights v2
    const double *v2 = nullptr;
    uint8_t *digits2 = nullptr;
    int32_t *expo2 = nullptr;
    SliceEntry e[kMaxGroup];
};

// The planes of U = X + B: plane 2 i + part holds digit i of the real (part 0) or imaginary part.
template <int kVec>
__device__ __forceinline__ void write_planes(const long long (&ur)[kVec], const long long (&ui)[kVec], int s,
                                             uint8_t *row, int64_t plane) {
    write_digits<kVec>(ur, s, row, 2 * plane);
    write_digits<kVec>(ui, s, row + plane, 2 * plane);
}

// Maximum over the block of non-negative doubles given as bit patterns (which order like the
// values), with integer operations: GB300's FP64 pipe takes 16 cycles per warp instruction, and
// an FP64 max here was most of the slicing's FP64 work.
__device__ __forceinline__ unsigned long long block_max_bits(unsigned long long m, unsigned long long *red) {
    for (int o = 16; o > 0; o >>= 1) m = max(m, (unsigned long long)__shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    unsigned long long r = 0;
    for (int i = 0; i < kSliceThreads / 32; ++i) r = max(r, red[i]);
    return r;
}
// frexp's exponent of a positive finite double given as bits: x = f 2^e with f in [1/2, 1)
__device__ __forceinline__ int frexp_exp_bits(unsigned long long b) {
    const int E = (int)(b >> 52) & 0x7ff;
    if (E) return E - 1022;
    return -1010 - __clzll((long long)(b & 0xfffffffffffffull));   // subnormal: mantissa 2^-1074
}

// Integer-pipe helpers of the slicing (GB300's FP64 pipe runs ~1/64 of its integer rate).
// |x| as an ordered integer: for finite doubles the bit pattern of |x| orders like |x|.
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
// rint(x 2^k), round half to even, exactly as __double2ll_rn(x * 2^k) for |x 2^k| < 2^62: the
// mantissa shifted by the exponent, with the round bit and the sticky remainder.
__device__ __forceinline__ long long rint_pow2(double x, int k) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7ff);
    const unsigned long long mant = b & 0xfffffffffffffull;
    const unsigned long long m = E ? (mant | (1ull << 52)) : mant;
    const int sh = 1075 - (E ? E : 1) - k;          // |x 2^k| = m 2^-sh
    unsigned long long q;
    if (sh <= 0) {
        q = m << (-sh);
    } else if (sh >= 54) {
        q = 0;                                      // m 2^-sh < 1/2
    } else {
        q = m >> sh;
        const unsigned long long rem = m & ((1ull << sh) - 1), half = 1ull << (sh - 1);
        q += (rem > half) | ((rem == half) & (q & 1ull));
    }
    return (b >> 63) ? -(long long)q : (long long)q;
}
// v 2^k by an exponent add (v normal and the result normal), else ldexp
__device__ __noinline__ double ldexp_out_of_line(double v, int k) { return ldexp(v, k); }
__device__ __forceinline__ double scale_pow2(double v, int k) {
    const long long b = __double_as_longlong(v);
    const int E = (int)((b >> 52) & 0x7ff);
    if (E > 0 && E + k > 0 && E + k < 2047) return __longlong_as_double(b + ((long long)k << 52));
    return ldexp_out_of_line(v, k);    // (a call: inlined, its FP64 work was issued for every value)
}

// the weighted operand's digits of one chunk (kept out of line: inlined next to the first
// operand's, the compiler interleaves the two and spills)
template <int kV>
__device__ __noinline__ void weighted_chunk(const double2 *zc, const double *vv, int nv, int kw, long long B, int s,
                                            uint8_t *row, int64_t plane) {
    long long xr[kV], xi[kV];
#pragma unroll
    for (int u = 0; u < kV; ++u) {
        const double2 z = u < nv ? zc[u] : make_double2(0.0, 0.0);
        const double sc = u < nv ? scale_pow2(vv[u], kw) : 0.0;
        xr[u] = B + rint_pow2(z.x * sc, 0);
        xi[u] = B + rint_pow2(z.y * sc, 0);
    }
    write_planes<kV>(xr, xi, s, row, plane);
}

#ifndef HSDLA_SLICE_CTAS
#define HSDLA_SLICE_CTAS 2
#endif
template <bool kDual>
__global__ void __launch_bounds__(kSliceThreads, HSDLA_SLICE_CTAS) oz_slice_kernel(const __grid_constant__ SliceTab tab) {
    // values per thread and step of the digit pass (the dual pass keeps two operands' state)
    constexpr int kV = kDual ? 4 : kSliceVec;
    const int64_t r = blockIdx.x;           // plane row
    int k = 0;
    while (k + 1 < tab.nk && tab.e[k + 1].row0 <= r) ++k;
    const int64_t g = r - tab.e[k].row0;
    const bool live = g >= 0 && g < tab.e[k].ncols;
    const double2 *Zc = tab.e[k].Z + tab.ldz * (live ? g : 0);
    const double *v = tab.v, *v2 = tab.v2;
    const int Kin = (int)tab.Kin, rpb = (int)tab.rpb, bpad = (int)tab.bpad, Kpad = (int)tab.Kpad;
    const int64_t pitch = tab.pitch, plane_rows = tab.plane_rows;
    const int s = tab.s;
    __shared__ unsigned long long red[2][kSliceThreads / 32];
    // pass 1: column max of max(|re|, |im|) (times the row weight; the only FP64 multiply here)
    // Each thread reads 8 values per step (all loads of a step in flight together: one kept too few
    // bytes in flight to cover the memory latency), lanes on consecutive ones.
    // (the weighted and unweighted forms as separate loops: GB300 issues the FP64 multiplies of a
    // predicated-off branch all the same, at 16 cycles per warp instruction)
    unsigned long long mx = 0, mx2 = 0;
    auto pass1 = [&](auto weighted) {
        for (int k0 = threadIdx.x; k0 < Kin; k0 += kSliceThreads * kSliceVec) {
            double2 z[kSliceVec];
#pragma unroll
            for (int u = 0; u < kSliceVec; ++u) {
                const int i = k0 + u * kSliceThreads;
                z[u] = i < Kin ? Zc[i] : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < kSliceVec; ++u) {
                const unsigned long long a = max(abs_bits(z[u].x), abs_bits(z[u].y));
                const int i = k0 + u * kSliceThreads;
                if (i < Kin) {
                    if constexpr (decltype(weighted)::value) mx = max(mx, abs_bits(__longlong_as_double((long long)a) * v[i]));
                    else mx = max(mx, a);
                    if (kDual) mx2 = max(mx2, abs_bits(__longlong_as_double((long long)a) * v2[i]));
                }
            }
        }
    };
    if (live) {
        if (v) pass1(std::true_type{});
        else pass1(std::false_type{});
    }
    int e = 0, e2 = 0;
    const unsigned long long m = block_max_bits(mx, red[0]);
    if (m > 0) e = frexp_exp_bits(m);       // max < 2^e
    if (kDual) {
        const unsigned long long m2 = block_max_bits(mx2, red[1]);
        if (m2 > 0) e2 = frexp_exp_bits(m2);
    }
    if (threadIdx.x == 0) {
        tab.expo[r] = e;
        if (kDual) tab.expo2[r] = e2;
    }
    const int top = 5 * s - 1;              // X = rint(z 2^(5s-1)), |z| < 1
    const int kx = top - e, kw = top - e2;
    long long B = 0;
    for (int p = 0; p < s - 1; ++p) B |= 16ll << (5 * p);
    const int nb = Kpad / bpad;
    const int64_t plane = plane_rows * pitch;
    auto pass2 = [&](auto weighted) {
        for (int kp0 = threadIdx.x * kV; kp0 < Kpad; kp0 += kSliceThreads * kV) {
            // a chunk never straddles a contraction block (bpad is a multiple of kV)
            const int b = kp0 / bpad, rr0 = kp0 - b * bpad;
            // number of live values of this chunk (a prefix: the block tail and Kin cut it from above)
            const int nv = live && b < nb ? max(0, min(min(kV, rpb - rr0), Kin - (b * rpb + rr0))) : 0;
            const double2 *zc = Zc + b * rpb + rr0;
            long long xr[kV], xi[kV];
#pragma unroll
            for (int u = 0; u < kV; ++u) {
                const double2 z = u < nv ? zc[u] : make_double2(0.0, 0.0);
                if constexpr (decltype(weighted)::value) {
                    const double sc = u < nv ? scale_pow2(v[b * rpb + rr0 + u], kx) : 0.0;
                    xr[u] = B + rint_pow2(z.x * sc, 0);
                    xi[u] = B + rint_pow2(z.y * sc, 0);
                } else {
                    xr[u] = B + rint_pow2(z.x, kx);
                    xi[u] = B + rint_pow2(z.y, kx);
                }
            }
            write_planes<kV>(xr, xi, s, tab.digits + r * pitch + kp0, plane);
            if (kDual)      // the chunk again (an L1 hit) for the weighted operand
                weighted_chunk<kV>(zc, v2 + b * rpb + rr0, nv, kw, B, s, tab.digits2 + r * pitch + kp0, plane);
        }
    };
    if (v) pass2(std::true_type{});
    else pass2(std::false_type{});
}

// ------------------------------------------------------------ host helpers
typedef CUresult (*PFN_encodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                    const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

PFN_encodeTiled get_encode() {
    static PFN_encodeTiled fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(p);
    }
    return fn;
}

// digit operand: 2s planes of plane_rows rows; a row holds Kpad digit bytes at a row pitch of
// Kpad + pad bytes.  The pad keeps the pitch off a power of two: with a power-of-two pitch the
// 128 rows of one TMA box fall on the same L2 sets and memory channels.
struct DigitOperand {
    uint8_t *digits = nullptr;
    int32_t *expo = nullptr;
    int64_t plane_rows = 0, Kpad = 0, pitch = 0;
    CUtensorMap map;
    CUtensorMap map64;         // 64-row boxes: a right operand of the real products
};

int64_t env_int(const char *name, int64_t dflt) {
    const char *v = getenv(name);
    if (!v || !*v) return dflt;
    char *end = nullptr;
    const long long x = strtoll(v, &end, 10);
    return (end && *end == 0) ? (int64_t)x : dflt;
}

// Row pitch pad of the digit planes (bytes, multiple of 16); HSDLA_DIGIT_PITCH_PAD overrides.
int64_t pitch_pad() {
    static const int64_t p = [] {
        int64_t x = env_int("HSDLA_DIGIT_PITCH_PAD", 128);
        if (x < 0 || x > 4096) x = 128;
        return (x + 15) / 16 * 16;
    }();
    return p;
}

// box_rows: rows of a TMA box (kTileM; 64 for the right operand of the real products)
// and contraction bytes of one: 128 with the 128-byte swizzle, 64 with the 64-byte one
int make_map(DigitOperand &d, int planes, int box_rows = kTileM, CUtensorMap *dst = nullptr, int box_bytes = kKBlock) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) { g_oz_err = "cuTensorMapEncodeTiled unavailable"; return HSDLA_ERR_CUDA; }
    if (d.Kpad % 128 != 0 || d.pitch % 16 != 0 || d.pitch < d.Kpad ||
        (reinterpret_cast<uintptr_t>(d.digits) & 255) != 0) {
        g_oz_err = "digit operand misaligned";
        return HSDLA_ERR_ARG;
    }
    const int64_t rows = d.plane_rows * planes;
    if (rows > INT32_MAX || d.Kpad > INT32_MAX) { g_oz_err = "digit operand too large for TMA"; return HSDLA_ERR_UNSUPPORTED; }
    cuuint64_t dims[2] = {(cuuint64_t)d.Kpad, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)d.pitch};
    cuuint32_t box[2] = {(cuuint32_t)box_bytes, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    CUresult r = enc(dst ? dst : &d.map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, d.digits, dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE,
                     box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { g_oz_err = "cuTensorMapEncodeTiled failed"; return HSDLA_ERR_CUDA; }
    return HSDLA_OK;
}

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// Bump allocator over the caller's workspace.
struct Arena {
    char *p;
    int64_t used = 0;
    template <typename T>
    T *take(int64_t count) {
        T *r = reinterpret_cast<T *>(p + used);
        used += round_up((int64_t)sizeof(T) * count, 1024);
        return r;
    }
};

// planes: digit planes (0: 2s)
int64_t operand_bytes(int s, int64_t rows, int64_t Kpad, int planes = 0) {
    const int64_t pr = round_up(rows, kTileM) + kTileM;
    return round_up((planes ? planes : 2 * s) * pr * (Kpad + pitch_pad()), 1024) + round_up(4 * pr, 1024);
}

void carve_operand(Arena &a, DigitOperand &d, int s, int64_t rows, int64_t Kpad, int planes = 0) {
    d.plane_rows = round_up(rows, kTileM) + kTileM;
    d.Kpad = Kpad;
    d.pitch = Kpad + pitch_pad();
    d.digits = a.take<uint8_t>((planes ? planes : 2 * s) * d.plane_rows * d.pitch);
    d.expo = a.take<int32_t>(d.plane_rows);
}

SliceTab slice_table(const double2 *Z, int64_t ldz, const double *v, int64_t Kin, int64_t ncols, int64_t rpb,
                     int64_t bpad, int s, const DigitOperand &d) {
    SliceTab t;
    t.nk = 1; t.s = s; t.ldz = ldz; t.Kin = Kin; t.rpb = rpb; t.bpad = bpad; t.v = v;
    t.digits = d.digits; t.Kpad = d.Kpad; t.plane_rows = d.plane_rows; t.pitch = d.pitch; t.expo = d.expo;
    t.e[0] = SliceEntry{Z, ncols, 0};
    return t;
}

cudaError_t slice_launch(const SliceTab &t, cudaStream_t st) {
    if (t.digits2) oz_slice_kernel<true><<<(unsigned)t.plane_rows, kSliceThreads, 0, st>>>(t);
    else oz_slice_kernel<false><<<(unsigned)t.plane_rows, kSliceThreads, 0, st>>>(t);
    return cudaGetLastError();
}

cudaError_t slice(const double2 *Z, int64_t ldz, const double *v, int64_t Kin, int64_t ncols, int64_t rpb,
                  int64_t bpad, int s, DigitOperand &d, cudaStream_t st) {
    return slice_launch(slice_table(Z, ldz, v, Kin, ncols, rpb, bpad, s, d), st);
}

int64_t job_tiles(const OzJob &j, int64_t tile = kTileM) {
    const int64_t tm = (j.m + tile - 1) / tile, tn = (j.n + tile - 1) / tile;
    return j.lower ? tm * (tm + 1) / 2 : tm * tn;
}

// The S/H launch runs on CTA pairs (256 x 256 tiles) unless HSDLA_PAIR=0.
bool use_pair() {
    static const bool b = env_int("HSDLA_PAIR", 1) != 0;
    return b;
}

// Host-built tile schedule.  Persistent CTAs take tiles g, g + grid, ... so tiles that are
// close in the list run at the same time and share their operand panels in L2.  Lower-
// triangle jobs of equal size (S and H of one k-point) are walked together in square super-
// blocks of super_block() tiles, the jobs' tiles of one (tm, tn) adjacent (they share the
// left operand); full jobs (T application) go job by job, tile columns outermost.
// Super-block edge in tiles; HSDLA_SCHED_SUPERBLOCK overrides (0 = row-major over the whole
// triangle).  With the CTAs in lockstep, 8 x 8 super-blocks cut the S/H launch of the
// 8000-column FLAPW workload from 378 ms (row-major) to 355 ms: a wave then reads ~16 left and
// ~16 right panels instead of ~2 left and ~120 right ones.
// On 256 x 256 pair tiles the default edge is 4 (the same panel span).
int64_t super_block(int64_t tile) {
    static const int64_t b = env_int("HSDLA_SCHED_SUPERBLOCK", 0);
    if (b < 0) return (int64_t)1 << 30;
    if (b > 0) return b;
    return tile == kTileN ? 8 : 4;
}

void build_schedule(const std::vector<OzJob> &jobs, std::vector<int4> &list, int64_t tile = kTileN) {
    const int64_t kSuperBlock = super_block(tile);
    list.clear();
    std::vector<char> done(jobs.size(), 0);
    for (size_t a = 0; a < jobs.size(); ++a) {
        if (done[a]) continue;
        const OzJob &ja = jobs[a];
        if (ja.lower) {
            std::vector<int> group;
            for (size_t b = a; b < jobs.size(); ++b)
                if (!done[b] && jobs[b].lower && jobs[b].n == ja.n) { group.push_back((int)b); done[b] = 1; }
            const int64_t T = (ja.n + tile - 1) / tile;
            for (int64_t I = 0; I < T; I += kSuperBlock)
                for (int64_t J = 0; J <= I; J += kSuperBlock)
                    for (int64_t tm = I; tm < std::min(T, I + kSuperBlock); ++tm)
                        for (int64_t tn = J; tn < std::min(tm + 1, J + kSuperBlock); ++tn)
                            for (int g : group) list.push_back(make_int4(g, (int)tm, (int)tn, 0));
        } else {
            done[a] = 1;
            const int64_t tmn = (ja.m + tile - 1) / tile, tnn = (ja.n + tile - 1) / tile;
            for (int64_t tn = 0; tn < tnn; ++tn)
                for (int64_t tm = 0; tm < tmn; ++tm) list.push_back(make_int4((int)a, (int)tm, (int)tn, 0));
        }
    }
}

constexpr int kProgressCap = 1024;   // progress slots (>= SM count, multiple of 4)
// Streamed host output: the S/H launches of all types are cut into at most kMaxOutBlocks launches
// of whole waves of tiles; the tiles are ordered by kOutColumnBlocks column blocks (of about
// equal tile counts), so that the columns a launch completes are combined and sent to the host
// while the next launch runs.  Only the part completed by the last launch stays exposed.
constexpr int kMaxOutBlocks = 8;
constexpr int kOutColumnBlocks = 8;

int launch_gemm(std::vector<OzJob> &jobs, const CUtensorMap *maps, int s, int *d_err, OzJob *d_jobs,
                cudaStream_t st, cudaEvent_t ev0 = nullptr, cudaEvent_t ev1 = nullptr, int4 *d_list = nullptr,
                int *d_progress = nullptr) {
    int64_t total = 0;
    for (auto &j : jobs) {
        j.tiles_n = (j.n + kTileN - 1) / kTileN;
        j.tile_begin = total;
        total += job_tiles(j);
    }
    if (total == 0) return HSDLA_OK;
    cudaError_t e = cudaMemcpyAsync(d_jobs, jobs.data(), sizeof(OzJob) * jobs.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    std::vector<int4> list;
    if (d_list) {
        build_schedule(jobs, list);
        if ((int64_t)list.size() != total) { g_oz_err = "tile schedule size mismatch"; return HSDLA_ERR_ARG; }
        e = cudaMemcpyAsync(d_list, list.data(), sizeof(int4) * list.size(), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    }
    const size_t smem = (size_t)kStages * kStageBytes + 1024;
    e = cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t grid = std::min<int64_t>(total, nsm);
    // lockstep needs every CTA resident at once: cooperative launch, one CTA per SM
    const bool lockstep = d_progress != nullptr && grid > 1 && grid <= kProgressCap && env_int("HSDLA_LOCKSTEP", 1) != 0;
    if (lockstep) {
        const int64_t g4 = (grid + 3) / 4 * 4;
        e = cudaMemsetAsync(d_progress, 0, sizeof(int) * grid, st);
        if (e == cudaSuccess && g4 > grid) e = cudaMemsetAsync(d_progress + grid, 0x7F, sizeof(int) * (g4 - grid), st);
        if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    }
    if (ev0) cudaEventRecord(ev0, st);
    if (lockstep) {
        CUtensorMap m0 = maps[0], m1 = maps[1], m2 = maps[2], m3 = maps[3];
        const OzJob *pj = d_jobs;
        int nj = (int)jobs.size();
        int64_t tt = total;
        int ss = s;
        int *perr = d_err;
        const int4 *pl = d_list;
        int *pp = d_progress;
        void *args[] = {&m0, &m1, &m2, &m3, &pj, &nj, &tt, &ss, &perr, &pl, &pp};
        e = cudaLaunchCooperativeKernel((const void *)oz_gemm_kernel, dim3((unsigned)grid), dim3(kThreads), args, smem, st);
    } else {
        oz_gemm_kernel<<<(unsigned)grid, kThreads, smem, st>>>(maps[0], maps[1], maps[2], maps[3], d_jobs,
                                                                (int)jobs.size(), total, s, d_err, d_list, nullptr);
        e = cudaGetLastError();
    }
    if (ev1) cudaEventRecord(ev1, st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    // the job table is read by the kernel: keep the host copy alive until it is consumed
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    return HSDLA_OK;
}

// ------------------------------------------------------------ wait self-test
// Exercises the bounded-wait and abort path of the product kernels on a condition that never
// comes true, with a short budget: the CTA holds TMEM as the product kernels do, one thread
// waits on an mbarrier nothing arrives on (which = 0) or on a lockstep slot that never advances
// (which = 1), the wait records the error word and raises the abort flag, and the CTA frees TMEM
// and returns.  Nothing faults, traps or hangs.
__global__ void __launch_bounds__(64, 1) oz_wait_probe_kernel(int *err, int *progress, long long budget, int which) {
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int abort_flag;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;\n" ::"r"(smem_u32(&tmem_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) {
        if (which == 0) mbar_wait(&bar, 0, &abort_flag, err, 7, budget);
        else grid_lockstep(progress, 4, 3, &abort_flag, err, 0, 1, budget);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;\n" ::"r"(tmem_sh) : "memory");
    }
}

}  // namespace

int ozaki_wait_selftest(OzakiPlan &oz, int which, long long budget_cycles, cudaStream_t st) {
    if (!oz.d_error) { g_oz_err = "Ozaki plan not initialised"; return HSDLA_ERR_ARG; }
    if (which < 0 || which > 1 || budget_cycles <= 0 || budget_cycles > kWaitCycles) {
        g_oz_err = "wait self-test: which must be 0 or 1, budget in (0, 2e9] cycles";
        return HSDLA_ERR_ARG;
    }
    // progress slots for which = 1: slot 0 is this CTA, slots 1..3 stay at epoch 0
    int *progress = oz.d_error + 8;
    cudaError_t e = cudaMemsetAsync(progress, 0, 4 * sizeof(int), st);
    if (e == cudaSuccess) {
        oz_wait_probe_kernel<<<1, 64, 0, st>>>(oz.d_error, progress, budget_cycles, which);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    return ozaki_check_device_error(oz);
}

namespace {

}  // namespace

// ==================================================================== API
int ozaki_plan_init(OzakiPlan &oz, int num_slices, double target) {
    if (num_slices == 0) num_slices = kOzDefaultSlices;
    if (num_slices < 2 || num_slices > kOzMaxSlices) { g_oz_err = "num_slices outside [2, 12]"; return HSDLA_ERR_ARG; }
    oz.num_slices = num_slices;
    oz.target = target;
    if (!oz.d_error) {
        if (cudaMalloc(&oz.d_error, kErrAlloc * sizeof(int)) != cudaSuccess) { g_oz_err = "cudaMalloc"; return HSDLA_ERR_NOMEM; }
        cudaMemset(oz.d_error, 0, kErrAlloc * sizeof(int));
    }
    return HSDLA_OK;
}

void ozaki_plan_release(OzakiPlan &oz) {
    if (oz.d_error) cudaFree(oz.d_error);
    oz.d_error = nullptr;
}

int ozaki_check_device_error(OzakiPlan &oz) {
    if (!oz.d_error) return HSDLA_OK;
    int w[kErrWords] = {};
    if (cudaMemcpy(w, oz.d_error, sizeof(w), cudaMemcpyDeviceToHost) != cudaSuccess) return HSDLA_ERR_CUDA;
    const int h = w[0];
    if (h != 0) {
        static thread_local char buf[192];
        snprintf(buf, sizeof(buf),
                 "device wait expired (code %d, role %d; block %d rank %d stage %d phase %d count %d)", h / 16,
                 h % 16, w[1], w[2], w[3], w[4], w[5]);
        g_oz_err = buf;
        cudaMemset(oz.d_error, 0, sizeof(w));
        return h / 16 == kDevBadInput ? HSDLA_ERR_CUDA : HSDLA_ERR_TIMEOUT;
    }
    return HSDLA_OK;
}

int64_t schedule_capacity_lower(int64_t n) {
    const int64_t T = (n + kTileN - 1) / kTileN;
    return T * (T + 1);                                     // two lower-triangle jobs
}

int64_t ozaki_herkx_workspace(int s, int64_t K, int64_t n) {
    const int64_t Kpad = round_up(std::max<int64_t>(K, 1), kKBlock);
    return 2 * operand_bytes(s, n, Kpad) + 4096 + 4096 + round_up(sizeof(int4) * schedule_capacity_lower(n), 1024) +
           round_up(sizeof(int) * kProgressCap, 1024);
}

// ---------------------------------------------------------------- k-point groups
// A group is a set of k-points whose digit operands are resident together.  Its digit planes
// stack the k-points' columns as consecutive rows, so one tensor map per operand covers every
// k-point, one slicing launch per operand covers the group, and one oz_gemm launch runs the T
// application and one the S/H products of all k-points.  Everything but the output pointers
// is prepared once; a run only enqueues launches (it can be captured in a CUDA graph).
// One atom panel of a group: the contraction index split by atoms, each panel sliced with its own
// exponents and its S/H products accumulated into the outputs.
struct OzPanel {
    int64_t a0 = 0, a1 = 0;            // atoms [a0, a1)
    SliceTab tC, tX;                   // tC is dual: C and W
    int64_t jt_off = 0, lt_off = 0;    // this panel's T-application jobs / tiles (non-hoisted)
    int n_jobs_t = 0;
    int64_t tiles_t = 0;
};

// A split of the tiles that do not fill a wave of CTA pairs: each pair takes an equal run of their steps
// (a step: one digit pair of one k-block), so a tile is made by one pair or by several.  The part with a
// tile's first step adds into the output as an unsplit tile does, the others into slabs of their own,
// which oz_slab_add_kernel adds in the order of the parts (results repeat bit for bit).
struct PairSplit {
    int4 *list = nullptr, *parts = nullptr, *adds = nullptr;
    double2 *slabs = nullptr;
    int64_t total = 0;             // entries
    int pairs = 0, n_adds = 0;     // CTA pairs; split tiles
};
struct OzGroup {
    int s = 0, nk = 0, panels = 1;
    bool hoist = false;
    int64_t twoL = 0, na = 0, nt = 0, K = 0, bpad = 0, rows = 0;
    std::vector<OzKBufs> kb;
    std::vector<int64_t> row0;
    std::vector<OzPanel> pan;
    DigitOperand dC, dW, dX, dM, dT;
    SliceTab tM;
    CUtensorMap maps_t[4], maps_sh[4];
    OzJob *d_jobs_t = nullptr, *d_jobs_sh = nullptr, *h_jobs_sh = nullptr;
    int n_jobs_t = 0, n_jobs_sh = 0;   // hoisted T jobs; S/H jobs per panel (2 per k-point)
    int4 *d_list_t = nullptr, *d_list_sh = nullptr;
    int64_t tiles_t = 0, tiles_sh = 0;
    int *d_progress = nullptr;
    int *d_err = nullptr;
    bool pair = false;          // S/H on CTA-pair tiles
    bool pair_t = false;        // the T application on CTA-pair tiles
    PairSplit split, split_t;   // of the S/H products' and the T application's tiles
    bool sf = false;            // structure-factor form, on real rows:
    RealSliceTab rM, rX;        // the slicing of R (and R diag(w)) and of Z'
    RealJob *d_rjobs_t = nullptr, *d_rjobs_sh = nullptr;   // T application; 3 nk products per type
    RealBands bands{}, bands_t{};   // digit-pair order of the products and of the T application
    int halves = 2;             // the products' configuration (see set_sh_tiles)
    bool merged = true;
    int tbatch = 1;             // its types per combine batch
    // with one batch: the first side_types types are combined on a side stream while the S/H
    // launches of the others run (the combine is FP64-bound, the products tensor-bound)
    int side_types = 0;
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    SfTab sft{};                // its combine table (outputs patched per run)
    const void *sf_tab = nullptr;
    // Streamed host output (structure-factor form on pair tiles, every type in one combine batch):
    // the S/H products of all types in column blocks, one launch per block, each block combined
    // into the caller's page-locked outputs on blk_side while the next block's products run.
    // Block b covers tile-list entries [blk_begin[b], blk_begin[b+1]) of d_list_blk and output
    // columns [blk_col[b], blk_col[b+1]).
    int nblk = 0;
    int64_t blk_begin[kMaxOutBlocks + 1] = {};
    int64_t blk_col[kMaxOutBlocks + 1] = {};
    int4 *d_list_blk = nullptr;
    cudaStream_t blk_side = nullptr;
    cudaEvent_t ev_blk[kMaxOutBlocks] = {};
    cudaEvent_t ev_blk_join = nullptr;
};

namespace {

int64_t group_rows(const std::vector<int64_t> &G) {
    int64_t r = 0;
    for (int64_t g : G) r += round_up(std::max<int64_t>(g, 1), kTileM);
    return r + kTileM;
}

constexpr int64_t kSlabBytes = (int64_t)kPairTile * kPairTile * sizeof(double2);

// Launch of a prepared pair-tile job table: clusters of two CTAs, one per SM, as many pairs as
// can be resident (at most one per tile); cooperative when the lockstep slots are given.
// With a split (make_split) its entries run in place of the tiles, then the slabs are added up.
cudaError_t pair_config(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *at, int &max_out, cudaStream_t st) {
    const size_t smem = kPairSmem;
    cudaError_t e = cudaFuncSetAttribute(oz_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    static int max_pairs = 0;
    if (max_pairs == 0) {
        cfg.gridDim = dim3(2);
        int nc = 0;
        e = cudaOccupancyMaxActiveClusters(&nc, (const void *)oz_pair_kernel, &cfg);
        if (e != cudaSuccess) return e;
        if (nc < 1) return cudaErrorInvalidConfiguration;
        max_pairs = nc;
    }
    max_out = max_pairs;
    return cudaSuccess;
}

cudaError_t launch_pair(const CUtensorMap *maps, int s, int *d_err, const OzJob *d_jobs, int n_jobs, int64_t total,
                        const int4 *d_list, int *d_progress, cudaStream_t st, const PairSplit *split = nullptr) {
    if (total <= 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    int max_pairs = 0;
    cudaError_t e = pair_config(cfg, at, max_pairs, st);
    if (e != cudaSuccess) return e;
    const bool cut = split && split->n_adds > 0;
    if (cut) { total = split->total; d_list = split->list; }
    const int64_t pairs = cut ? split->pairs : std::min<int64_t>(total, max_pairs);
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    const bool lockstep = d_progress && pairs > 1 && pairs <= kProgressCap && env_int("HSDLA_LOCKSTEP", 1) != 0;
    if (lockstep) {
        const int64_t g4 = (pairs + 3) / 4 * 4;
        e = cudaMemsetAsync(d_progress, 0, sizeof(int) * pairs, st);
        if (e == cudaSuccess && g4 > pairs) e = cudaMemsetAsync(d_progress + pairs, 0x7F, sizeof(int) * (g4 - pairs), st);
        if (e != cudaSuccess) return e;
        // cooperative: the launch waits until every pair can be resident (the lockstep needs
        // that); HSDLA_COOPERATIVE=0 drops the attribute for profilers that cannot replay a
        // cooperative cluster launch (on an otherwise idle GPU the grid is resident anyway, and
        // the lockstep waits stay bounded)
        if (env_int("HSDLA_COOPERATIVE", 1) != 0) {
            at[1].id = cudaLaunchAttributeCooperative;
            at[1].val.cooperative = 1;
            cfg.numAttrs = 2;
        }
    }
    // lockstep epoch (stages) and how many epochs a pair may lead the slowest one
    static const int sync_every = (int)std::max<int64_t>(8, env_int("HSDLA_SYNC_EVERY", kSyncEvery));
    static const int slack = (int)std::max<int64_t>(1, env_int("HSDLA_SYNC_SLACK", 1));
    e = cudaLaunchKernelEx(&cfg, oz_pair_kernel, maps[0], maps[1], maps[2], maps[3], d_jobs, n_jobs, total,
                           s, d_err, d_list, lockstep ? d_progress : (int *)nullptr, sync_every, slack,
                           cut ? (const int4 *)split->parts : (const int4 *)nullptr, cut ? split->slabs : (double2 *)nullptr);
    if (e != cudaSuccess || !cut) return e;
    oz_slab_add_kernel<<<dim3((unsigned)split->n_adds, kPairTile), kPairTile, 0, st>>>(d_jobs, split->adds, split->slabs);
    return cudaGetLastError();
}

// The rule: of N tiles of `steps` steps (~1.3 us each) on np pairs, the R = N mod np beyond whole waves are
// cut where that shortens the last wave by at least kSplitGain steps and a quarter; below, the slabs (1 MB
// each, written and read), the additional drains and operand panels that fewer pairs share at a time take
// as much.  Whole and cut, us: 3 tiles of 66 steps (57 saved) 488 and 383 of a call, 21 of 66 (47 saved) 524 and
// 484, 78 of 66 (57 saved) 747 and 662, 21 of 726 (525 saved) 1255 and 729; but 36 of 66 (34 saved) 550 and
// 553, 66 of 528 (69 saved) 1155 and 1173.  Parts have at least kSplitMin steps.
constexpr int64_t kSplitGain = 40, kSplitMin = 8;
struct SplitRule {
    int np = 0;
    int64_t R = 0, P = 0, per = 0;       // tiles cut, over P pairs, steps of each
};
bool split_rule(int64_t N, int64_t steps, SplitRule &r) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    if (N < 1 || steps > INT_MAX || !use_pair() || pair_config(cfg, at, r.np, nullptr) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    r.R = N % r.np;
    r.P = std::min<int64_t>(r.np, r.R * steps / kSplitMin);
    if (r.R == 0 || r.P <= r.R) return false;
    r.per = (r.R * steps + r.P - 1) / r.P;
    return steps - r.per >= std::max(kSplitGain, steps / 4);
}

// Whether the T application of `jobs` runs on CTA-pair tiles (256 x 256) or on single-CTA ones (128 x 128).  Where both
// take as many waves a tile's own time decides: ~0.14-0.16 ms a wave of pair tiles of one k-block (lmax 6 and below), 0.26 of
// two, 0.33 and 0.40 of three and four, against 0.21, 0.25, 0.27 and 0.30 on single tiles, which at 40 columns take
// 0.16, 0.17, 0.19 and 0.24 and at 7 0.09 to 0.20 (pair tiles 0.14 to 0.35).  Tiles cut over the idle pairs (`cut`) always
// are pair ones: 1 atom, lmax 7, 232 columns 68 us, 184 uncut.
bool pair_t_tiles(const std::vector<OzJob> &jobs, bool cut, int64_t steps) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    int np = 0;
    if (jobs.empty() || !use_pair()) return use_pair();
    if (pair_config(cfg, at, np, nullptr) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    int64_t n1 = 0, n2 = 0, cols = 0;
    for (const OzJob &j : jobs) {
        n1 += job_tiles(j, kTileM);
        n2 += job_tiles(j, kPairTile);
        cols = std::max(cols, j.n);
    }
    SplitRule r;
    if (cut && split_rule(n2, steps, r)) return true;
    if ((n1 + 2 * np - 1) / (2 * np) > (n2 + np - 1) / np) return true;
    const int64_t kblocks = jobs[0].nkb;
    return cols > (kblocks < 2 ? 16 : kblocks < 3 ? 64 : INT64_MAX - 1);
}

// `mem`, `bytes`: as ozaki_split_bytes says, or none (no split).
int make_split(PairSplit &sp, const std::vector<int4> &list, int64_t steps, void *mem, int64_t bytes) {
    sp = PairSplit();
    SplitRule rule;
    const int64_t N = (int64_t)list.size();
    if (!mem || !split_rule(N, steps, rule)) return HSDLA_OK;
    const int64_t np = rule.np, W = N / np, R = rule.R, P = rule.P, per = rule.per;
    std::vector<std::vector<std::pair<int4, int4>>> of(P);
    std::vector<int4> adds;
    int slab = 0;
    size_t rounds = 0;
    for (int64_t p = 0; p < P; ++p) {
        int64_t a = std::min(p * per, R * steps);
        const int64_t b = std::min(a + per, R * steps);
        for (; a < b;) {
            const int64_t r = a / steps, lo = a - r * steps, hi = std::min(steps, b - r * steps);
            const int4 e = list[W * np + r];
            if (lo > 0) {
                if (adds.empty() || adds[adds.size() - 2].x != e.x || adds[adds.size() - 2].y != e.y || adds[adds.size() - 2].z != e.z) {
                    adds.push_back(make_int4(e.x, e.y, e.z, slab));
                    adds.push_back(make_int4(0, 0, 0, 0));
                }
                ++adds.back().x;
            }
            of[p].push_back({e, make_int4((int)lo, (int)hi, lo > 0 ? slab++ : -1, 0)});
            a = r * steps + hi;
        }
        rounds = std::max(rounds, of[p].size());
    }
    const int64_t G = W > 0 ? np : P, total = (W + (int64_t)rounds) * G;
    if (slab * kSlabBytes + 32 * total + 16 * (int64_t)adds.size() > bytes) return HSDLA_OK;
    std::vector<int4> up(2 * total, make_int4(0, 0, 0, 0));
    for (int64_t i = 0; i < total; ++i) up[total + i] = make_int4(0, 0, -1, 0);
    for (int64_t i = 0; i < W * np; ++i) {
        up[i] = list[i];
        up[total + i] = make_int4(0, INT_MAX, -1, 0);
    }
    for (int64_t p = 0; p < P; ++p)
        for (size_t q = 0; q < of[p].size(); ++q) {
            const int64_t i = (W + (int64_t)q) * G + p;
            up[i] = of[p][q].first;
            up[total + i] = of[p][q].second;
        }
    up.insert(up.end(), adds.begin(), adds.end());
    sp.slabs = reinterpret_cast<double2 *>(mem);
    sp.list = reinterpret_cast<int4 *>(reinterpret_cast<char *>(mem) + slab * kSlabBytes);
    sp.parts = sp.list + total;
    sp.adds = sp.parts + total;
    sp.total = total;
    sp.pairs = (int)G;
    sp.n_adds = (int)adds.size() / 2;
    const cudaError_t e = cudaMemcpy(sp.list, up.data(), sizeof(int4) * up.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    return HSDLA_OK;
}

int upload_schedule(std::vector<OzJob> &jobs, OzJob *d_jobs, int4 *d_list, int64_t &tiles, int64_t tile = kTileN,
                    PairSplit *split = nullptr, int64_t steps = 0, void *split_mem = nullptr, int64_t split_size = 0) {
    int64_t total = 0;
    for (auto &j : jobs) {
        j.tiles_n = (j.n + tile - 1) / tile;
        j.tile_begin = total;
        total += job_tiles(j, tile);
    }
    std::vector<int4> list;
    build_schedule(jobs, list, tile);
    if ((int64_t)list.size() != total) { g_oz_err = "tile schedule size mismatch"; return HSDLA_ERR_ARG; }
    cudaError_t e = cudaMemcpy(d_jobs, jobs.data(), sizeof(OzJob) * jobs.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess && total > 0)
        e = cudaMemcpy(d_list, list.data(), sizeof(int4) * list.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    tiles = total;
    return split ? make_split(*split, list, steps, split_mem, split_size) : HSDLA_OK;
}

// Launch of a prepared job table (no host synchronisation; capturable).
cudaError_t launch_prepared(const CUtensorMap *maps, int s, int *d_err, const OzJob *d_jobs, int n_jobs,
                            int64_t total, const int4 *d_list, int *d_progress, cudaStream_t st) {
    if (total <= 0) return cudaSuccess;
    const size_t smem = (size_t)kStages * kStageBytes + 1024;
    cudaError_t e = cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t grid = std::min<int64_t>(total, nsm);
    const bool lockstep = d_progress && grid > 1 && grid <= kProgressCap && env_int("HSDLA_LOCKSTEP", 1) != 0;
    if (lockstep) {
        const int64_t g4 = (grid + 3) / 4 * 4;
        e = cudaMemsetAsync(d_progress, 0, sizeof(int) * grid, st);
        if (e == cudaSuccess && g4 > grid) e = cudaMemsetAsync(d_progress + grid, 0x7F, sizeof(int) * (g4 - grid), st);
        if (e != cudaSuccess) return e;
        CUtensorMap m0 = maps[0], m1 = maps[1], m2 = maps[2], m3 = maps[3];
        const OzJob *pj = d_jobs;
        int nj = n_jobs;
        int64_t tt = total;
        int ss = s;
        int *perr = d_err;
        const int4 *pl = d_list;
        int *pp = d_progress;
        void *args[] = {&m0, &m1, &m2, &m3, &pj, &nj, &tt, &ss, &perr, &pl, &pp};
        return cudaLaunchCooperativeKernel((const void *)oz_gemm_kernel, dim3((unsigned)grid), dim3(kThreads), args,
                                           smem, st);
    }
    oz_gemm_kernel<<<(unsigned)grid, kThreads, smem, st>>>(maps[0], maps[1], maps[2], maps[3], d_jobs, n_jobs, total,
                                                            s, d_err, d_list, nullptr);
    return cudaGetLastError();
}

}  // namespace

namespace {
int64_t split_bytes(int64_t N, int64_t steps) {
    SplitRule r;
    if (!split_rule(N, steps, r)) return 0;
    // at most P - 1 parts do not begin a tile; entries of whole waves and of up to P tiles a pair in the last
    return round_up(r.P * kSlabBytes + 32 * (N + (2 + (r.R + r.P - 1) / r.P) * r.np) + 32 * r.R, 1024);
}
int64_t pair_steps(int s, int64_t K) { return round_up(std::max<int64_t>(K, 1), kKBlock) / kKBlock * s * (s + 1) / 2; }
}  // namespace

// Memory with which ozaki_herkx, or a group, splits the tiles of a partial last wave: `jobs` lower products
// of n columns over K rows (0: they would not be split).
int64_t ozaki_split_bytes(int s, int64_t K, int64_t n, int64_t jobs) {
    const int64_t T = (n + kPairTile - 1) / kPairTile;
    return split_bytes(jobs * T * (T + 1) / 2, pair_steps(s, K));
}
// ... or `jobs` T applications of m rows and n columns.
int64_t ozaki_split_bytes_t(int s, int64_t m, int64_t n, int64_t jobs) {
    const int64_t tm = (m + kPairTile - 1) / kPairTile, tn = (n + kPairTile - 1) / kPairTile;
    return split_bytes(jobs * tm * tn, pair_steps(s, m));
}

// P^H diag(w) Q (lower triangle) for one pair of K x n operands: the contraction behind
// hsdla_zherkx_lower and the BLAS-shaped plugin.
int ozaki_herkx(OzakiPlan &oz, const double2 *P, int64_t ldp, const double2 *Q, int64_t ldq, const double *w,
                int64_t K, int64_t n, double2 *out, int64_t ldo, void *ws, cudaStream_t st, int *launches, void *split,
                int64_t split_size) {
    const int s = oz.num_slices;
    const int64_t Kpad = round_up(std::max<int64_t>(K, 1), kKBlock);
    Arena ar{reinterpret_cast<char *>(ws)};
    DigitOperand dp, dq;
    carve_operand(ar, dp, s, n, Kpad);
    carve_operand(ar, dq, s, n, Kpad);
    OzJob *d_jobs = ar.take<OzJob>(4);
    int4 *d_list = ar.take<int4>(schedule_capacity_lower(n));
    cudaError_t e = slice(P, ldp, nullptr, K, n, Kpad, Kpad, s, dp, st);
    if (e == cudaSuccess) e = slice(Q, ldq, w, K, n, Kpad, Kpad, s, dq, st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    int rc = make_map(dp, 2 * s);
    if (!rc) rc = make_map(dq, 2 * s);
    if (rc) return rc;
    CUtensorMap maps[4] = {dp.map, dq.map, dp.map, dp.map};
    std::vector<OzJob> jobs(1);
    OzJob &j = jobs[0];
    memset(&j, 0, sizeof(j));
    j.lmap = 0; j.rmap = 1; j.lower = 1;
    j.lplane = dp.plane_rows; j.rplane = dq.plane_rows;
    j.nkb = Kpad / kKBlock; j.m = n; j.n = n;
    j.out = out; j.ldo = ldo; j.el = dp.expo; j.er = dq.expo;
    if (use_pair()) {
        // CTA-pair 256 x 256 tiles, one exact unit per diagonal and K chunk, pairs in lockstep
        int *d_progress = ar.take<int>(kProgressCap);
        int64_t tiles = 0;
        PairSplit sp;
        rc = upload_schedule(jobs, d_jobs, d_list, tiles, kPairTile, &sp, j.nkb * s * (s + 1) / 2, split, split_size);
        if (rc) return rc;
        const cudaError_t el = launch_pair(maps, s, oz.d_error, d_jobs, 1, tiles, d_list, d_progress, st, &sp);
        if (el != cudaSuccess) { g_oz_err = cudaGetErrorString(el); return HSDLA_ERR_CUDA; }
    } else {
        rc = launch_gemm(jobs, maps, s, oz.d_error, d_jobs, st, nullptr, nullptr, d_list);
    }
    if (launches) *launches = 3;
    return rc;
}

// Run-time scratch of a group (digit planes and exponents, rewritten by every run; groups of a
// plan share it) and its persistent part (T digits, job tables, tile schedules, lockstep slots).
static int64_t panel_atoms(int64_t na, int panels) { return (na + panels - 1) / panels; }
// Stride of one atom's 2L rows along the contraction index of the digit planes: 16 bytes keeps
// every atom's block on a TMA boundary (the T application starts its loads there).  A T job reads
// ceil(2L / 128) k-blocks from that start; the rows past 2L it covers (padding and the next atoms)
// meet T digits that are exactly zero, and reads past the operand's extent are zero-filled.
static int64_t atom_stride(int64_t twoL) { return round_up(twoL, 16); }

int64_t ozaki_group_bytes(int s, int64_t twoL, int64_t na, int64_t nt, const std::vector<int64_t> &G, int panels,
                          bool hoist, bool sf) {
    const int64_t bpad = atom_stride(twoL), rows = group_rows(G);
    if (sf) {      // digits of the real rows R, of R diag(w_t) and of Z' (two parts): each type's
                   // rows on whole k-blocks
        const int64_t KT = round_up(round_up(twoL, kRealKBlock) * nt, kKBlock);
        auto dig = [&](int64_t planes) {
            return round_up(planes * rows * (KT + pitch_pad()), 1024) + round_up(4 * rows, 1024);
        };
        return 2 * dig(s) + dig(2 * s) + 4096;
    }
    const int64_t Kp = round_up(bpad * panel_atoms(na, panels), kKBlock);
    const int64_t Kx = hoist ? std::max(Kp, round_up(bpad * nt, kKBlock)) : Kp;
    auto dig = [&](int64_t K) { return round_up(2 * s * rows * (K + pitch_pad()), 1024) + round_up(4 * rows, 1024); };
    return 2 * dig(Kp) + dig(Kx) + 4096;
}

int64_t ozaki_group_persist_bytes(int s, int64_t twoL, int64_t na, int64_t nt, const std::vector<int64_t> &G,
                                  int panels, bool sf, int64_t ntypes) {
    const int64_t bpad = round_up(atom_stride(twoL), kKBlock);    // T operand: one atom's rows per plane row
    const int64_t nk = (int64_t)G.size();
    if (sf) {
        int64_t tiles_t = 0, tiles_sh = 0;
        for (int64_t g : G) {
            const int64_t tn = (g + kRealTileN - 1) / kRealTileN, tm = (g + kRealTileM - 1) / kRealTileM;
            tiles_t += nt * ((2 * twoL + kRealTileM - 1) / kRealTileM) * tn;
            tiles_sh += 3 * nt * tm * tn;                // (more than the lower triangle's)
        }
        return operand_bytes(s, 2 * ntypes * twoL, bpad, s) + round_up(sizeof(RealJob) * nk * nt, 1024) +
               round_up(sizeof(RealJob) * 3 * nk * nt, 1024) + round_up(sizeof(int4) * (tiles_t + 1), 1024) +
               2 * round_up(sizeof(int4) * (tiles_sh + 1), 1024) + 8192;
    }
    int64_t tiles_t = 0, tiles_sh = 0;
    for (int64_t g : G) {
        const int64_t T = (g + kTileN - 1) / kTileN;
        tiles_t += std::max(na, nt) * ((twoL + kTileM - 1) / kTileM) * T;
        tiles_sh += T * (T + 1);
    }
    return operand_bytes(s, nt * twoL, bpad, 2 * s) + round_up(sizeof(OzJob) * nk * (std::max(na, nt) + 2), 1024) +
           round_up(sizeof(OzJob) * 2 * nk * panels, 1024) + round_up(sizeof(int4) * (tiles_t + panels), 1024) +
           round_up(sizeof(int4) * (tiles_sh + 1), 1024) + round_up(sizeof(int) * kProgressCap, 1024) + 8192;
}

// The streamed host output's launches.  The output columns are split into kOutColumnBlocks ranges
// (whole tile columns) of about equal lower-triangle areas; the tile list runs through them in
// order, and within a range type by type, each type in the per-type schedule's order (so that the
// pairs working at a time share few types' operands in L2).  The list is then cut into launches of
// whole waves (one tile per cluster pair of the GPU); launch b leaves columns
// [blk_col[b], blk_col[b+1]) complete (possibly none).  l0: the first type's tiles.
static int build_output_blocks(OzGroup *g, const std::vector<int4> &l0) {
    int64_t T = 0;
    for (const int4 &e : l0) T = std::max<int64_t>(T, e.z + 1);
    g->nblk = 0;
    if (T < 2) return HSDLA_OK;
    const int C = (int)std::min<int64_t>(kOutColumnBlocks, T);
    const int64_t total = T * (T + 1) / 2;
    std::vector<int64_t> cb(C + 1, T);
    cb[0] = 0;
    int64_t acc = 0, c = 0;
    for (int b = 1; b < C; ++b) {
        while (c < T && acc < total * b / C) { acc += T - c; ++c; }
        cb[b] = c;
    }
    std::vector<int4> lb;
    lb.reserve(l0.size() * g->nt);
    for (int b = 0; b < C; ++b)
        for (int t = 0; t < g->nt; ++t)
            for (const int4 &e : l0)
                if (e.z >= cb[b] && e.z < cb[b + 1]) lb.push_back(make_int4(t * g->n_jobs_sh + e.x, e.y, e.z, 0));
    const int64_t N = (int64_t)lb.size();
    if (N != (int64_t)l0.size() * g->nt) { g_oz_err = "output block schedule size mismatch"; return HSDLA_ERR_ARG; }
    // first incomplete tile column after list position i: suffix minimum of the tile columns
    std::vector<int64_t> open(N + 1, T);
    for (int64_t i = N - 1; i >= 0; --i) open[i] = std::min<int64_t>(open[i + 1], lb[i].z);
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int64_t wave = std::max(1, nsm / 2);
    const int64_t waves = (N + wave - 1) / wave;
    const int64_t per = std::max<int64_t>(1, (waves + kMaxOutBlocks - 1) / kMaxOutBlocks) * wave;
    g->blk_begin[0] = 0;
    g->blk_col[0] = 0;
    for (int64_t i0 = 0; i0 < N && g->nblk < kMaxOutBlocks; ++g->nblk) {
        const int64_t i1 = g->nblk + 1 == kMaxOutBlocks ? N : std::min(N, i0 + per);
        g->blk_begin[g->nblk + 1] = i1;
        g->blk_col[g->nblk + 1] = std::max(g->blk_col[g->nblk], open[i1] * kRealTileN);
        i0 = i1;
    }
    g->blk_col[g->nblk] = T * kRealTileN;
    const cudaError_t e = cudaMemcpy(g->d_list_blk, lb.data(), sizeof(int4) * N, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    return HSDLA_OK;
}

static void set_sh_tiles(OzGroup *g, int halves, bool merged) {
    g->halves = halves;
    g->merged = merged;
    g->bands = real_bands(g->s, merged ? 2 : 1, halves, g->twoL);
}

// Structure-factor form of a group, on the real rows (real_products.cu): digit planes of R, R
// diag(w_t) and Z' (2L rows per type, each type's rows starting on a k-block so that the per-type
// products never mix types), the T application Z'_t = T'_t R_t, and the products S, Re H, Im H of
// every type of a combine batch in one launch, followed by the combine into S and H.
static int group_prepare_sf(OzakiPlan &oz, const OzGroupDesc &d, const std::vector<OzKBufs> &kb, void *ws,
                            void *persist, cudaStream_t st, OzGroup **out) {
    auto *g = new OzGroup();
    g->sf = true;
    g->s = oz.num_slices;
    g->nk = (int)kb.size();
    g->hoist = true;
    g->twoL = d.twoL; g->na = d.na; g->nt = d.nt;
    // type stride along the contraction: whole 64-byte chunks
    g->bpad = round_up(d.twoL, kRealKBlock);
    const int64_t tkb = g->bpad / kRealKBlock, KT = round_up(g->bpad * d.nt, kKBlock);
    // K steps of 32 bytes in a type's last chunk (the contraction length is 2L per type)
    const int ksl = (int)((d.twoL - (tkb - 1) * kRealKBlock + 31) / 32);
    g->kb = kb;
    g->d_err = oz.d_error;
    g->sf_tab = d.sf_tab;
    g->tbatch = std::max(1, d.tbatch);
    // HSDLA_COMBINE_OVERLAP=1: the first half of the combine on a side stream, next to the products
    // of the other types.  Off by default: on the 8000-column workload the co-running combine slowed
    // the products by more than it saved.
    if (g->tbatch >= d.nt && d.nt >= 2 && env_int("HSDLA_COMBINE_OVERLAP", 0) != 0) {
        g->side_types = (int)(d.nt / 2);
        if (cudaStreamCreateWithFlags(&g->side, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&g->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&g->ev_join, cudaEventDisableTiming) != cudaSuccess) {
            g_oz_err = "side stream creation failed";
            ozaki_group_destroy(g);
            return HSDLA_ERR_CUDA;
        }
    }
    std::vector<int64_t> G;
    for (auto &k : kb) G.push_back(k.G);
    g->rows = group_rows(G);
    int64_t r0 = 0;
    for (int64_t x : G) { g->row0.push_back(r0); r0 += round_up(std::max<int64_t>(x, 1), kTileM); }
    const int s = g->s;
    Arena ar{reinterpret_cast<char *>(ws)};
    Arena keep{reinterpret_cast<char *>(persist)};
    auto carve_rows = [&](DigitOperand &o, int planes) {
        o.plane_rows = g->rows;
        o.Kpad = KT;
        o.pitch = KT + pitch_pad();
        o.digits = ar.take<uint8_t>(planes * o.plane_rows * o.pitch);
        o.expo = ar.take<int32_t>(o.plane_rows);
    };
    carve_rows(g->dM, s);        // R
    carve_rows(g->dW, s);        // R diag(w_t)
    carve_rows(g->dX, 2 * s);    // Z'
    carve_operand(keep, g->dT, s, 2 * d.ntypes * d.twoL, round_up(g->bpad, kKBlock), s);
    const int64_t nk = g->nk;
    auto fail = [&](int code) { ozaki_group_destroy(g); return code; };
    auto table = [&](const DigitOperand &o, int parts) {
        RealSliceTab t;
        t.nk = g->nk; t.s = s; t.parts = parts;
        t.ldz = parts * d.twoL * d.nt; t.blocks = d.nt; t.rpb = d.twoL; t.bstride = parts * d.twoL;
        t.pstride = d.twoL; t.bpad = g->bpad;
        t.digits = o.digits; t.plane_rows = o.plane_rows; t.pitch = o.pitch; t.expo = o.expo;
        for (int k = 0; k < g->nk; ++k)
            t.e[k] = RealSliceEntry{parts == 1 ? (const void *)kb[k].R : (const void *)kb[k].ZR, kb[k].G, g->row0[k]};
        return t;
    };
    g->rM = table(g->dM, 1);              // dual: R and R diag(w_t)
    g->rM.v2 = d.wt;
    g->rM.digits2 = g->dW.digits;
    g->rM.expo2 = g->dW.expo;
    g->bands_t = real_bands(s, 2, 2, d.twoL);
    g->rX = table(g->dX, 2);
    g->rX.frac = g->bands_t.frac;         // Z' in fixed point, with T's row and R's column exponents
    g->rX.el = g->dT.expo;
    g->rX.set_type = d.d_set_type;
    g->rX.er = g->dM.expo;
    g->panels = 1;
    RealSliceTab tT;
    tT.nk = 1; tT.s = s; tT.ldz = d.twoL; tT.blocks = 1; tT.rpb = d.twoL; tT.bstride = d.twoL; tT.bpad = g->bpad;
    tT.digits = g->dT.digits; tT.plane_rows = g->dT.plane_rows; tT.pitch = g->dT.pitch; tT.expo = g->dT.expo;
    tT.e[0] = RealSliceEntry{d.TR, 2 * d.ntypes * d.twoL, 0};
    cudaError_t e = launch_real_slice(tT, st);    // stream-ordered before every use of the T digits
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return fail(HSDLA_ERR_CUDA); }
    // left operands in boxes of a CTA's 128 rows, right operands of its 64 rows
    int rc = make_map(g->dM, s, kRealTileM / 2, &g->dM.map, kRealKBlock);
    if (!rc) rc = make_map(g->dT, s, kRealTileM / 2, &g->dT.map, kRealKBlock);
    if (!rc) rc = make_map(g->dM, s, kRealBRows, &g->dM.map64, kRealKBlock);
    if (!rc) rc = make_map(g->dW, s, kRealBRows, &g->dW.map64, kRealKBlock);
    if (!rc) rc = make_map(g->dX, 2 * s, kRealBRows, &g->dX.map64, kRealKBlock);
    if (rc) return fail(rc);
    // T application per type: the real and imaginary rows of Z'_t = T'_t R_t as one product
    std::vector<RealJob> jt, jsh;
    for (int k = 0; k < g->nk; ++k)
        for (int64_t t = 0; t < d.nt; ++t) {
            RealJob j;
            memset(&j, 0, sizeof(j));
            j.rmap = 0; j.rstep = 1;
            j.lplane = g->dT.plane_rows; j.rplane = g->rows;
            j.lrow0 = 2 * d.set_type[t] * d.twoL; j.rrow0 = g->row0[k];
            j.rk0 = t * g->bpad;
            j.nkb = tkb; j.ksteps_last = ksl;
            j.m = 2 * d.twoL; j.n = kb[k].G;
            j.out = kb[k].ZR + 2 * d.twoL * t; j.ldo = 2 * d.twoL * d.nt;
            jt.push_back(j);
        }
    for (int64_t t = 0; t < d.nt; ++t)                    // (place t of the combine's order)
        for (int k = 0; k < g->nk; ++k)
            for (int which = 0; which < 3; ++which) {     // S, Re H, Im H
                RealJob j;
                memset(&j, 0, sizeof(j));
                j.rmap = which == 0 ? 0 : 1; j.lower = 1;
                j.rstep = which == 0 ? 1 : 2; j.rpart = which == 2 ? 1 : 0;
                j.lplane = g->rows; j.rplane = g->rows;
                j.lrow0 = g->row0[k]; j.rrow0 = g->row0[k];
                j.lk0 = j.rk0 = d.order[t] * g->bpad;
                j.nkb = tkb; j.ksteps_last = ksl;
                j.m = kb[k].G; j.n = kb[k].G;
                j.out = (which == 0 ? kb[k].RS : which == 1 ? kb[k].RHr : kb[k].RHi) + (t % g->tbatch) * kb[k].pstride;
                j.ldo = kb[k].G;
                jsh.push_back(j);
            }
    g->n_jobs_sh = (int)(3 * nk);
    std::vector<int4> lt, lsh, l0;
    real_schedule(jt, lt);
    real_schedule(std::vector<RealJob>(jsh.begin(), jsh.begin() + g->n_jobs_sh), l0);
    for (int t = 0; t < d.nt; ++t)
        for (const int4 &x : l0) lsh.push_back(make_int4(t * g->n_jobs_sh + x.x, x.y, x.z, 0));
    g->tiles_t = (int64_t)lt.size();
    g->tiles_sh = (int64_t)l0.size();
    int64_t want_t = 0, want_sh = 0;
    for (auto &j : jt) want_t += real_job_tiles(j);
    for (int q = 0; q < g->n_jobs_sh; ++q) want_sh += real_job_tiles(jsh[q]);
    if (want_t != g->tiles_t || want_sh != g->tiles_sh) { g_oz_err = "tile schedule size mismatch"; return fail(HSDLA_ERR_ARG); }
    g->d_rjobs_t = keep.take<RealJob>((int64_t)jt.size());
    g->d_rjobs_sh = keep.take<RealJob>((int64_t)jsh.size());
    g->d_list_t = keep.take<int4>((int64_t)lt.size() + 1);
    g->d_list_sh = keep.take<int4>((int64_t)lsh.size() + 1);
    g->d_list_blk = keep.take<int4>((int64_t)lsh.size() + 1);
    e = cudaMemcpy(g->d_rjobs_t, jt.data(), sizeof(RealJob) * jt.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(g->d_rjobs_sh, jsh.data(), sizeof(RealJob) * jsh.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(g->d_list_t, lt.data(), sizeof(int4) * lt.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(g->d_list_sh, lsh.data(), sizeof(int4) * lsh.size(), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return fail(HSDLA_ERR_CUDA); }
    rc = build_output_blocks(g, l0);
    if (rc) return fail(rc);
    set_sh_tiles(g, env_int("HSDLA_PAIR_HALVES", 2) == 2 ? 2 : 1, env_int("HSDLA_MERGE", 1) != 0);
    *out = g;
    return HSDLA_OK;
}

int ozaki_group_prepare(OzakiPlan &oz, const OzGroupDesc &d, const std::vector<OzKBufs> &kb, void *ws,
                        void *persist, cudaStream_t st, OzGroup **out) {
    *out = nullptr;
    if (kb.empty() || (int)kb.size() > kMaxGroup) { g_oz_err = "group size out of range"; return HSDLA_ERR_ARG; }
    if (d.panels < 1 || d.panels > d.na) { g_oz_err = "panel count out of range"; return HSDLA_ERR_ARG; }
    if (d.sf) return group_prepare_sf(oz, d, kb, ws, persist, st, out);
    auto *g = new OzGroup();
    g->s = oz.num_slices;
    g->nk = (int)kb.size();
    g->hoist = d.hoist;
    g->twoL = d.twoL; g->na = d.na; g->nt = d.nt;
    g->K = d.twoL * d.na;
    g->bpad = atom_stride(d.twoL);
    const int64_t tkb = (d.twoL + kKBlock - 1) / kKBlock;      // k-blocks of one T application
    g->kb = kb;
    g->d_err = oz.d_error;
    // atom panels: equal sizes but the last
    const int64_t pa = panel_atoms(d.na, d.panels);
    for (int64_t a0 = 0; a0 < d.na; a0 += pa) {
        OzPanel p;
        p.a0 = a0;
        p.a1 = std::min(d.na, a0 + pa);
        g->pan.push_back(p);
    }
    g->panels = (int)g->pan.size();
    std::vector<int64_t> G;
    for (auto &k : kb) G.push_back(k.G);
    g->rows = group_rows(G);
    int64_t r0 = 0;
    for (int64_t x : G) { g->row0.push_back(r0); r0 += round_up(std::max<int64_t>(x, 1), kTileM); }
    const int s = g->s;
    Arena ar{reinterpret_cast<char *>(ws)};
    Arena keep{reinterpret_cast<char *>(persist)};
    auto carve_rows = [&](DigitOperand &o, int64_t kpad) {
        o.plane_rows = g->rows;
        o.Kpad = kpad;
        o.pitch = kpad + pitch_pad();
        o.digits = ar.take<uint8_t>(2 * s * o.plane_rows * o.pitch);
        o.expo = ar.take<int32_t>(o.plane_rows);
    };
    const int64_t Kp = round_up(g->bpad * pa, kKBlock), Km = round_up(g->bpad * d.nt, kKBlock);
    carve_rows(g->dC, Kp);
    carve_rows(g->dW, Kp);
    carve_rows(g->dX, d.hoist ? std::max(Kp, Km) : Kp);
    carve_operand(keep, g->dT, s, d.nt * d.twoL, tkb * kKBlock);
    // the M digits (per-type rows, K = bpad nt) borrow the X digit region: they are consumed by the
    // T application, which runs before any panel's X is sliced
    g->dM.plane_rows = g->rows;
    g->dM.Kpad = Km;
    g->dM.pitch = g->dM.Kpad + pitch_pad();
    g->dM.digits = g->dX.digits;
    g->dM.expo = g->dX.expo;
    const int64_t nk = g->nk;
    int64_t tiles_t = 0, tiles_sh = 0;
    for (int64_t x : G) {
        const int64_t T = (x + kTileN - 1) / kTileN;
        tiles_t += std::max(d.na, d.nt) * ((d.twoL + kTileM - 1) / kTileM) * T;
        tiles_sh += T * (T + 1);
    }
    g->d_jobs_t = keep.take<OzJob>(nk * (std::max(d.na, d.nt) + 2));
    g->d_jobs_sh = keep.take<OzJob>(2 * nk * g->panels);
    g->d_list_t = keep.take<int4>(tiles_t + g->panels);
    g->d_list_sh = keep.take<int4>(tiles_sh + 1);
    g->d_progress = keep.take<int>(kProgressCap);
    int rc = HSDLA_OK;
    auto fail = [&](int code) { ozaki_group_destroy(g); return code; };
    if (cudaHostAlloc((void **)&g->h_jobs_sh, sizeof(OzJob) * 2 * nk * g->panels, cudaHostAllocDefault) !=
        cudaSuccess) {
        g->h_jobs_sh = nullptr;
        g_oz_err = "pinned job table allocation failed";
        return fail(HSDLA_ERR_NOMEM);
    }
    // slicing tables: source rows [a0 2L, a1 2L) of every k-point's column
    auto table = [&](const DigitOperand &o, int64_t ldz, const double *v, int64_t row_off, int64_t Kin, int64_t kpad,
                     int which) {
        SliceTab t;
        t.nk = g->nk; t.s = s; t.ldz = ldz; t.Kin = Kin; t.rpb = d.twoL; t.bpad = g->bpad; t.v = v;
        t.digits = o.digits; t.Kpad = kpad; t.plane_rows = o.plane_rows; t.pitch = o.pitch; t.expo = o.expo;
        for (int k = 0; k < g->nk; ++k) {
            const double2 *src = which == 1 ? kb[k].M : kb[k].CX + row_off;
            t.e[k] = SliceEntry{src, kb[k].G, g->row0[k]};
        }
        return t;
    };
    for (OzPanel &p : g->pan) {
        const int64_t off = p.a0 * d.twoL, Kin = (p.a1 - p.a0) * d.twoL;
        const int64_t kpad = round_up((p.a1 - p.a0) * g->bpad, kKBlock);
        p.tC = table(g->dC, g->K, nullptr, off, Kin, kpad, 0);
        p.tC.v2 = d.w + off;
        p.tC.digits2 = g->dW.digits;
        p.tC.expo2 = g->dW.expo;
        p.tX = table(g->dX, g->K, nullptr, off, Kin, kpad, 0);
    }
    if (d.hoist) g->tM = table(g->dM, d.twoL * d.nt, nullptr, 0, d.twoL * d.nt, Km, 1);
    // T digits once: they do not change between runs
    cudaError_t e = slice(d.Tfull, d.twoL, nullptr, d.twoL, d.nt * d.twoL, d.twoL, g->bpad, s, g->dT, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return fail(HSDLA_ERR_CUDA); }
    rc = make_map(g->dC, 2 * s);
    if (!rc) rc = make_map(g->dW, 2 * s);
    if (!rc) rc = make_map(g->dX, 2 * s);
    if (!rc) rc = make_map(g->dT, 2 * s);
    if (!rc && d.hoist) rc = make_map(g->dM, 2 * s);
    if (rc) return fail(rc);
    // (b) T application: per type once (hoisted), or per atom of each panel
    g->pair = use_pair();
    const int64_t tile = g->pair ? kPairTile : kTileN;
    g->pair_t = true;
    if (d.hoist) {
        std::vector<OzJob> jt;
        for (int k = 0; k < g->nk; ++k)
            for (int64_t t = 0; t < d.nt; ++t) {
                OzJob j;
                memset(&j, 0, sizeof(j));
                j.lmap = 3; j.rmap = 0;
                j.lplane = g->dT.plane_rows; j.rplane = g->dM.plane_rows;
                j.lrow0 = t * d.twoL; j.rrow0 = g->row0[k];
                j.rk0 = t * g->bpad;
                j.nkb = tkb;
                j.m = d.twoL; j.n = kb[k].G;
                j.out = kb[k].Z + d.twoL * t; j.ldo = d.twoL * d.nt;
                j.el = g->dT.expo + t * d.twoL; j.er = g->dM.expo + g->row0[k];
                jt.push_back(j);
            }
        g->n_jobs_t = (int)jt.size();
        g->pair_t = pair_t_tiles(jt, false, 0);
        rc = upload_schedule(jt, g->d_jobs_t, g->d_list_t, g->tiles_t, g->pair_t ? kPairTile : kTileN);
        if (rc) return fail(rc);
    } else {
        int64_t joff = 0, loff = 0;
        for (OzPanel &p : g->pan) {
            std::vector<OzJob> jt;
            for (int k = 0; k < g->nk; ++k)
                for (int64_t a = p.a0; a < p.a1; ++a) {
                    const int64_t t = d.atom_type[a];
                    OzJob j;
                    memset(&j, 0, sizeof(j));
                    j.lmap = 3; j.rmap = 0;
                    j.lplane = g->dT.plane_rows; j.rplane = g->dC.plane_rows;
                    j.lrow0 = t * d.twoL; j.rrow0 = g->row0[k];
                    j.rk0 = (a - p.a0) * g->bpad;
                    j.nkb = tkb;
                    j.m = d.twoL; j.n = kb[k].G;
                    j.out = kb[k].CX + d.twoL * a; j.ldo = g->K;
                    j.el = g->dT.expo + t * d.twoL; j.er = g->dC.expo + g->row0[k];
                    jt.push_back(j);
                }
            p.jt_off = joff;
            p.lt_off = loff;
            p.n_jobs_t = (int)jt.size();
            // (one shape for all panels, by the first and largest)
            void *cut = g->pair && g->panels == 1 ? d.split_t : nullptr;
            if (&p == &g->pan[0]) g->pair_t = pair_t_tiles(jt, cut != nullptr, tkb * s * (s + 1) / 2);
            rc = upload_schedule(jt, g->d_jobs_t + joff, g->d_list_t + loff, p.tiles_t, g->pair_t ? kPairTile : kTileN, &g->split_t,
                                 tkb * s * (s + 1) / 2, g->pair_t ? cut : nullptr, d.split_t_bytes);
            if (rc) return fail(rc);
            joff += p.n_jobs_t;
            loff += p.tiles_t;
        }
    }
    g->maps_t[0] = d.hoist ? g->dM.map : g->dC.map;
    g->maps_t[1] = g->maps_t[0]; g->maps_t[2] = g->maps_t[0]; g->maps_t[3] = g->dT.map;
    // (c) S and H jobs of every panel; outputs are patched per run, later panels accumulate
    g->n_jobs_sh = 2 * g->nk;
    for (int pi = 0; pi < g->panels; ++pi) {
        const OzPanel &p = g->pan[pi];
        std::vector<OzJob> jsh;
        for (int k = 0; k < g->nk; ++k)
            for (int which = 0; which < 2; ++which) {
                OzJob j;
                memset(&j, 0, sizeof(j));
                j.lmap = 0; j.rmap = which == 0 ? 1 : 2; j.lower = 1;
                j.accum = pi > 0;
                j.lplane = g->dC.plane_rows; j.rplane = which == 0 ? g->dW.plane_rows : g->dX.plane_rows;
                j.lrow0 = g->row0[k]; j.rrow0 = g->row0[k];
                j.nkb = round_up((p.a1 - p.a0) * g->bpad, kKBlock) / kKBlock;
                j.m = kb[k].G; j.n = kb[k].G;
                j.el = g->dC.expo + g->row0[k];
                j.er = (which == 0 ? g->dW.expo : g->dX.expo) + g->row0[k];
                jsh.push_back(j);
            }
        // the tile list is the same for every panel: upload it once
        if (pi == 0) {
            rc = upload_schedule(jsh, g->d_jobs_sh, g->d_list_sh, g->tiles_sh, tile, &g->split, jsh[0].nkb * s * (s + 1) / 2,
                                 g->pair && g->panels == 1 ? d.split : nullptr, d.split_bytes);
            if (rc) return fail(rc);
        } else {
            int64_t total = 0;
            for (auto &j : jsh) {
                j.tiles_n = (j.n + tile - 1) / tile;
                j.tile_begin = total;
                total += job_tiles(j, tile);
            }
        }
        memcpy(g->h_jobs_sh + 2 * g->nk * pi, jsh.data(), sizeof(OzJob) * jsh.size());
    }
    g->maps_sh[0] = g->dC.map; g->maps_sh[1] = g->dW.map; g->maps_sh[2] = g->dX.map; g->maps_sh[3] = g->dC.map;
    *out = g;
    return HSDLA_OK;
}

void ozaki_group_sf_exponents(const OzGroup *g, SfTab &t) {
    t.frac = g->bands.frac;
    for (int k = 0; k < g->nk; ++k) {
        t.e[k].el = g->dM.expo + g->row0[k];
        t.e[k].ers = g->dW.expo + g->row0[k];
        t.e[k].erh = g->dX.expo + g->row0[k];
    }
}
void ozaki_group_set_sf(OzGroup *g, const SfTab &t) { g->sft = t; }
int ozaki_group_last_combine(const OzGroup *g) {
    if (g->side_types > 0) return g->side_types;
    return (g->nt - 1) / g->tbatch * g->tbatch;
}

void ozaki_group_set_outputs(OzGroup *g, double2 *const *S, double2 *const *H, const int64_t *ld) {
    for (int pi = 0; pi < g->panels; ++pi) {
        OzJob *j = g->h_jobs_sh + 2 * g->nk * pi;
        for (int k = 0; k < g->nk; ++k) {
            j[2 * k].out = S[k];
            j[2 * k].ldo = ld[k];
            j[2 * k + 1].out = H[k];
            j[2 * k + 1].ldo = ld[k];
        }
    }
}

// The T application of the complex forms, on CTA-pair tiles or single-CTA ones (pair_t_tiles): 272 us for 8 atoms, lmax 8,
// 1501 columns (507 on single-CTA tiles), 161 for 2 atoms, lmax 1, 100 columns (207), 602 for 16, lmax 10, 1500 (813).
// Cut over the idle pairs (the contraction entry): 236 us of the first; 1 atom, lmax 7, 232 columns 184 -> 68, 4 atoms,
// lmax 8, 400 columns 268 -> 91.
static cudaError_t launch_t(const OzGroup *g, const OzJob *jobs, int n_jobs, int64_t tiles, const int4 *list, cudaStream_t st) {
    return g->pair_t ? launch_pair(g->maps_t, g->s, g->d_err, jobs, n_jobs, tiles, list, nullptr, st, &g->split_t)
                     : launch_prepared(g->maps_t, g->s, g->d_err, jobs, n_jobs, tiles, list, nullptr, st);
}

// Events around the S/H launch; under stream capture they become external event-record nodes
// so that a replayed graph still times the launch.
static cudaError_t record(cudaEvent_t ev, cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cs);
    return cs == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(ev, st, cudaEventRecordExternal)
                                               : cudaEventRecord(ev, st);
}

// One run: [hoisted: M digits, Z_t = T_t M_t], then per atom panel: C and W digits, the panel's
// T application (or phase expansion), X digits, the S/H products (accumulating after the first
// panel).  With several panels the events span the panels' S/H launches and the slicing between
// them.
int ozaki_group_tapply_events(const OzGroup *g) { return (g->sf || g->hoist) ? 1 : g->panels; }

bool ozaki_group_streamable(const OzGroup *g) {
    return g && g->sf && g->nblk > 1 && g->tbatch >= g->nt && g->side_types == 0 &&
           env_int("HSDLA_STREAM_OUTPUT", 1) != 0;
}

int ozaki_group_output_blocks(const OzGroup *g) { return g ? g->nblk : 0; }

// Products of `tiles` entries of a tile list.
static cudaError_t launch_sh(const OzGroup *g, const int4 *list, int64_t tiles, cudaStream_t st) {
    return launch_real_products(g->dM.map, g->dW.map64, g->dX.map64, g->d_rjobs_sh, list, tiles, g->bands, g->d_err, st);
}

// The streamed host output's S/H part.  Per column block: one pair launch over every type's tiles
// of the block, then the block's combine on the main stream, which writes the block's diagonal
// square (rows < the block's end) into the caller's page-locked outputs in place and the rows
// below it into the device outputs; the copy engine then downloads those rows (side stream)
// while the next block's products run.  The last block's combine writes everything in place.
// The main stream waits for the last download at the end.  No SM work runs beside the products.
static cudaError_t run_sh_streamed(OzGroup *g, cudaStream_t st, const cudaEvent_t *ev, int nev, const SfTab &out,
                                   int *nl) {
    cudaError_t e = cudaSuccess;
    if (!g->blk_side) {
        e = cudaStreamCreateWithFlags(&g->blk_side, cudaStreamNonBlocking);
        for (int b = 0; b < g->nblk && e == cudaSuccess; ++b)
            e = cudaEventCreateWithFlags(&g->ev_blk[b], cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&g->ev_blk_join, cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
    }
    // the dominant-launch event pairs: pair b spans block b's S/H launch where there are enough of
    // them (the rest, and a shortfall, span nothing)
    const int npair = nev / 2;
    for (int b = 0; b < g->nblk && e == cudaSuccess; ++b) {
        const int64_t c0 = g->blk_col[b], c1 = g->blk_col[b + 1];
        const bool last = b + 1 == g->nblk;
        if (b < npair) e = record(ev[2 * b], st);
        if (e == cudaSuccess)
            e = launch_sh(g, g->d_list_blk + g->blk_begin[b], g->blk_begin[b + 1] - g->blk_begin[b], st);
        if (e == cudaSuccess && b < npair) e = record(ev[2 * b + 1], st);
        SfTab tab = out;
        tab.type = 0;
        tab.ntypes = g->nt;
        tab.slot0 = 0;
        tab.col0 = c0;
        tab.col1 = c1;
        if (!last) {
            // rows below the block's diagonal square into the device outputs (the sums Si, Hi of an
            // earlier batch are the device outputs themselves; this is the only batch)
            tab.xrow1 = c1;
            for (int q = 0; q < tab.nk; ++q) {
                SfEntry &E = tab.e[q];
                E.Sx = E.S;
                E.Hx = E.H;
                E.ldx = E.ldo;
                E.S = const_cast<double2 *>(E.Si);
                E.H = const_cast<double2 *>(E.Hi);
                E.ldo = E.ldi;
            }
        }
        if (c1 <= c0) { *nl += 1; continue; }       // no column completed by this launch
        if (e == cudaSuccess) e = launch_sf_combine(tab, g->sf_tab, true, st);
        *nl += 2;
        if (last || e != cudaSuccess) continue;
        e = cudaEventRecord(g->ev_blk[b], st);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(g->blk_side, g->ev_blk[b], 0);
        for (int q = 0; q < tab.nk && e == cudaSuccess; ++q) {
            const SfEntry &E = tab.e[q];
            if (c1 >= E.n) continue;
            const int64_t w = std::min(c1, E.n) - c0;
            for (int m = 0; m < 2 && e == cudaSuccess; ++m) {
                double2 *host = (m == 0 ? E.Sx : E.Hx) + c1 + E.ldx * c0;
                const double2 *dev = (m == 0 ? E.S : E.H) + c1 + E.ldo * c0;
                e = cudaMemcpy2DAsync(host, E.ldx * sizeof(double2), dev, E.ldo * sizeof(double2),
                                      (E.n - c1) * sizeof(double2), w, cudaMemcpyDeviceToHost, g->blk_side);
            }
        }
    }
    for (int p = g->nblk; p < npair && e == cudaSuccess; ++p) {
        e = record(ev[2 * p], st);
        if (e == cudaSuccess) e = record(ev[2 * p + 1], st);
    }
    if (e == cudaSuccess) e = cudaEventRecord(g->ev_blk_join, g->blk_side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, g->ev_blk_join, 0);
    return e;
}

int ozaki_group_run(OzGroup *g, const DevSystem &sys, const KTable &ktab, cudaStream_t st, const cudaEvent_t *ev,
                    int nev, int *launches, bool defer_last_combine, const cudaEvent_t *ev_t, int nev_t,
                    const SfTab *host_out) {
    const cudaEvent_t ev0 = nev >= 2 ? ev[0] : nullptr, ev1 = nev >= 2 ? ev[nev - 1] : nullptr;
    // T-application events: pair q around the q-th T launch (when the caller gave enough of them)
    const bool tev = ev_t && nev_t >= 2 * ozaki_group_tapply_events(g);
    int nl = 0;
    cudaError_t e = cudaSuccess;
    if (g->sf) {
        e = launch_real_slice(g->rM, st);                 // R and R diag(w_t)
        if (e == cudaSuccess && tev) e = cudaEventRecord(ev_t[0], st);
        if (e == cudaSuccess)
            e = launch_real_products(g->dT.map, g->dM.map64, g->dM.map64, g->d_rjobs_t, g->d_list_t, g->tiles_t,
                                     g->bands_t, g->d_err, st);
        if (e == cudaSuccess && tev) e = cudaEventRecord(ev_t[1], st);
        if (e == cudaSuccess) e = launch_real_slice(g->rX, st);      // Z'
        nl += 3;
        if (host_out && ozaki_group_streamable(g)) {
            if (e == cudaSuccess) e = run_sh_streamed(g, st, ev, nev, *host_out, &nl);
            if (launches) *launches = nl;
            if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
            return HSDLA_OK;
        }
        // batches of types: their products in one launch, then their combine into S and H (the
        // caller combines the group's last batch when it defers it).  With a side stream the one
        // batch runs in two parts, the first part's combine beside the second part's products.
        const int step = g->side_types > 0 ? g->side_types : g->tbatch;
        int p = 0;
        for (int t0 = 0; t0 < g->nt && e == cudaSuccess; ++p) {
            const int t1 = g->side_types > 0 && t0 > 0 ? (int)g->nt : (int)std::min<int64_t>(g->nt, t0 + step);
            const bool last = t1 == g->nt, timed = 2 * p + 1 < nev;
            if (timed) e = record(ev[2 * p], st);
            if (e == cudaSuccess) e = launch_sh(g, g->d_list_sh + t0 * g->tiles_sh, (t1 - t0) * g->tiles_sh, st);
            if (e == cudaSuccess && timed) e = record(ev[2 * p + 1], st);
            nl += 1;
            SfTab tab = g->sft;
            tab.type = t0;
            tab.ntypes = t1 - t0;
            tab.slot0 = t0 % g->tbatch;
            if (g->side_types > 0 && !last) {
                // plain records: under graph capture they fork the side stream into the graph
                // and join it back
                if (e == cudaSuccess) e = cudaEventRecord(g->ev_fork, st);
                if (e == cudaSuccess) e = cudaStreamWaitEvent(g->side, g->ev_fork, 0);
                if (e == cudaSuccess) e = launch_sf_combine(tab, g->sf_tab, true, g->side);
                if (e == cudaSuccess) e = cudaEventRecord(g->ev_join, g->side);
                nl += 1;
            } else {
                if (e == cudaSuccess && g->side_types > 0) e = cudaStreamWaitEvent(st, g->ev_join, 0);
                if (e == cudaSuccess && !(defer_last_combine && last)) {
                    e = launch_sf_combine(tab, g->sf_tab, t0 == 0, st);
                    nl += 1;
                }
            }
            t0 = t1;
        }
        // event pairs past the batches (kept for the streamed form's column blocks) span nothing,
        // after the products (the last event closes the group's products)
        for (; 2 * p + 1 < nev && e == cudaSuccess; ++p) {
            e = record(ev[2 * p], st);
            if (e == cudaSuccess) e = record(ev[2 * p + 1], st);
        }
        if (launches) *launches = nl;
        if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
        return HSDLA_OK;
    }
    if (g->hoist) {
        e = slice_launch(g->tM, st);
        if (e == cudaSuccess && tev) e = cudaEventRecord(ev_t[0], st);
        if (e == cudaSuccess)
            e = launch_t(g, g->d_jobs_t, g->n_jobs_t, g->tiles_t, g->d_list_t, st);
        if (e == cudaSuccess && tev) e = cudaEventRecord(ev_t[1], st);
        nl += 2;
    }
    // the S/H job tables travel from pinned memory in stream order (a graph replays the copy)
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(g->d_jobs_sh, g->h_jobs_sh, sizeof(OzJob) * g->n_jobs_sh * g->panels,
                            cudaMemcpyHostToDevice, st);
    for (int pi = 0; pi < g->panels && e == cudaSuccess; ++pi) {
        const OzPanel &p = g->pan[pi];
        e = slice_launch(p.tC, st);           // C and W = C diag(w) in one pass over C
        nl += 1;
        if (e == cudaSuccess) {
            if (g->hoist) {
                KTable kt = ktab;
                kt.a0 = (int)p.a0;
                kt.a1 = (int)p.a1;
                e = launch_apply_phase_multi(sys, kt, st);
            } else {
                if (tev) e = cudaEventRecord(ev_t[2 * pi], st);
                if (e == cudaSuccess)
                    e = launch_t(g, g->d_jobs_t + p.jt_off, p.n_jobs_t, p.tiles_t, g->d_list_t + p.lt_off, st);
                if (e == cudaSuccess && tev) e = cudaEventRecord(ev_t[2 * pi + 1], st);
            }
            nl += 1;
        }
        if (e == cudaSuccess) { e = slice_launch(p.tX, st); nl += 1; }
        if (e == cudaSuccess && pi == 0 && ev0) e = record(ev0, st);
        const OzJob *jobs = g->d_jobs_sh + (int64_t)g->n_jobs_sh * pi;
        if (e == cudaSuccess)
            e = g->pair ? launch_pair(g->maps_sh, g->s, g->d_err, jobs, g->n_jobs_sh, g->tiles_sh, g->d_list_sh,
                                      g->d_progress, st, &g->split)
                        : launch_prepared(g->maps_sh, g->s, g->d_err, jobs, g->n_jobs_sh, g->tiles_sh, g->d_list_sh,
                                          g->d_progress, st);
        nl += 1;
    }
    if (e == cudaSuccess && ev1) e = record(ev1, st);
    if (launches) *launches = nl;
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    return HSDLA_OK;
}

bool ozaki_group_tunable(const OzGroup *g) { return g && g->sf; }

void ozaki_group_tiles(const OzGroup *g, int *halves, int *merged) {
    *halves = g->halves;
    *merged = g->merged ? 1 : 0;
}

void ozaki_group_set_tiles(OzGroup *g, int halves, int merged) {
    if (ozaki_group_tunable(g)) set_sh_tiles(g, halves == 1 ? 1 : 2, merged != 0);
}

// Times the first type's products (every k-point of the group) in each configuration and keeps
// the fastest.  (Bands of two everywhere so far: bands of one took 1.00 to 1.56 times as long over lmax 2 to 14, 300 to 4000
// columns and 8 to 12 digits.)  The digit planes must hold a completed run's data (the launches only rewrite that
// type's product slot, which the run has combined already).  Each configuration runs twice, the
// second timed.
int ozaki_group_tune_tiles(OzGroup *g, cudaStream_t st, float *ms_best) {
    if (!ozaki_group_tunable(g)) return HSDLA_OK;
    const int cfg[2][2] = {{2, 1}, {2, 0}};
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        if (e0) cudaEventDestroy(e0);
        g_oz_err = "tile tuner: event creation failed";
        return HSDLA_ERR_CUDA;
    }
    const int h0 = g->halves;
    const bool m0 = g->merged;
    // a prefix of the tile list is enough to rank the configurations (a batched group's launch
    // covers every k-point): at most 16 waves of pair tiles
    const int64_t tiles = std::min<int64_t>(g->tiles_sh, 16 * 76);
    float best = -1.f;
    int bi = 0;
    cudaError_t e = cudaSuccess;
    for (int c = 0; c < 2 && e == cudaSuccess; ++c) {
        set_sh_tiles(g, cfg[c][0], cfg[c][1] != 0);
        // one untimed launch, then the faster of two timed ones (a launch slowed by something
        // else on the machine would otherwise fix a worse configuration for the plan)
        float ms = -1.f;
        for (int rep = 0; rep < 3 && e == cudaSuccess; ++rep) {
            if (rep > 0) e = cudaEventRecord(e0, st);
            if (e == cudaSuccess)
                e = launch_sh(g, g->d_list_sh, tiles, st);
            if (e == cudaSuccess && rep > 0) e = cudaEventRecord(e1, st);
            if (e == cudaSuccess && rep > 0) e = cudaEventSynchronize(e1);
            float t = 0.f;
            if (e == cudaSuccess && rep > 0) e = cudaEventElapsedTime(&t, e0, e1);
            if (e == cudaSuccess && rep > 0 && (ms < 0.f || t < ms)) ms = t;
        }
        if (e == cudaSuccess && (best < 0.f || ms < best)) { best = ms; bi = c; }
        if (e == cudaSuccess && env_int("HSDLA_TRACE", 0))
            fprintf(stderr, "tile tuner: bands of %d: %.3f ms\n", cfg[c][1] ? 2 : 1, ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) {
        set_sh_tiles(g, h0, m0);
        g_oz_err = cudaGetErrorString(e);
        return HSDLA_ERR_CUDA;
    }
    set_sh_tiles(g, cfg[bi][0], cfg[bi][1] != 0);
    if (ms_best) *ms_best = best;
    return HSDLA_OK;
}

void ozaki_group_destroy(OzGroup *g) {
    if (!g) return;
    if (g->h_jobs_sh) cudaFreeHost(g->h_jobs_sh);
    if (g->ev_fork) cudaEventDestroy(g->ev_fork);
    if (g->ev_join) cudaEventDestroy(g->ev_join);
    if (g->side) cudaStreamDestroy(g->side);
    for (auto &ev : g->ev_blk)
        if (ev) cudaEventDestroy(ev);
    if (g->ev_blk_join) cudaEventDestroy(g->ev_blk_join);
    if (g->blk_side) cudaStreamDestroy(g->blk_side);
    delete g;
}

// One k-point through a temporary group (the slice autotuner's probe).
int64_t ozaki_pipeline_workspace(int s, int64_t twoL, int64_t na, int64_t nt, int64_t G) {
    const std::vector<int64_t> g{G};
    return ozaki_group_bytes(s, twoL, na, nt, g, 1, true, false) + ozaki_group_persist_bytes(s, twoL, na, nt, g, 1, false, nt) +
           2048;
}

int ozaki_pipeline(OzakiPlan &oz, const OzakiInputs &in, double2 *S, double2 *H, int64_t ldo, void *ws,
                   cudaStream_t st, int *launches) {
    OzGroupDesc d;
    d.twoL = in.twoL; d.na = in.na; d.nt = in.nt; d.hoist = in.M != nullptr;
    d.w = in.w; d.Tfull = in.Tfull; d.atom_type = in.atom_type; d.ntypes = in.nt;
    std::vector<OzKBufs> kb(1);
    // the probe keeps C and X apart: C is its input, X is written by the T application
    kb[0].CX = const_cast<double2 *>(in.C);
    kb[0].M = const_cast<double2 *>(in.M);
    kb[0].Z = in.Z;
    kb[0].G = in.G;
    OzGroup *g = nullptr;
    const int64_t scratch = ozaki_group_bytes(oz.num_slices, in.twoL, in.na, in.nt, std::vector<int64_t>{in.G}, 1,
                                              d.hoist, false);
    char *persist = reinterpret_cast<char *>(ws) + (scratch + 1023) / 1024 * 1024;
    int rc = ozaki_group_prepare(oz, d, kb, ws, persist, st, &g);
    if (rc) return rc;
    double2 *Sp[1] = {S}, *Hp[1] = {H};
    int64_t ld[1] = {ldo};
    ozaki_group_set_outputs(g, Sp, Hp, ld);
    KTable kt;
    kt.nk = 1; kt.ldc = in.twoL * in.na; kt.ldm = in.twoL * in.nt; kt.total_cols = in.G;
    if (in.kp) kt.e[0] = KEntry{*in.kp, nullptr, nullptr, in.Z, kb[0].CX, 0};
    const cudaEvent_t evs[2] = {in.ev_dom0, in.ev_dom1};
    rc = ozaki_group_run(g, in.sys ? *in.sys : DevSystem{}, kt, st, evs, in.ev_dom0 ? 2 : 0, launches);
    if (rc == HSDLA_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = HSDLA_ERR_CUDA;
    ozaki_group_destroy(g);
    return rc;
}

}  // namespace hsdla

// ======================================================================
// Allocation-free variant of the Ozaki lower-triangle contraction.
//
// Some callers cannot allocate device memory: code running inside another
// framework's memory pool or under a fixed memory budget, plug-ins that may only
// touch the buffers they are handed, and processes that must not call cudaMalloc
// once their steady state has begun.  For them, hsdla_zherkx_lower_noalloc keeps
// every scratch byte of the Ozaki contraction (digit planes, exponents, the job
// table and the device error word) in one file-scope device array of
// kNoAllocScratchBytes.  That array exists on every GPU that loads this library
// and stays resident until the process exits.  The caller still passes the
// inputs and the output.
#include <mutex>

namespace hsdla {
namespace {

constexpr int64_t kNoAllocScratchBytes = int64_t(128) << 20;   // 128 MiB
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Host-side cache of the array's device address, per device.  In host code the
// symbol g_noalloc_scratch is only a stand-in for the device array, so its address
// must come from cudaGetSymbolAddress with that device current.
std::mutex g_noalloc_mu;
unsigned char *g_noalloc_ptr[kNoAllocMaxDevices] = {};

int noalloc_scratch(unsigned char **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        g_oz_err = "no current CUDA device";
        return HSDLA_ERR_DEVICE;
    }
    if (dev < 0 || dev >= kNoAllocMaxDevices) {
        g_oz_err = "device index beyond the 64 devices the static scratch table covers";
        return HSDLA_ERR_DEVICE;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || p == nullptr) {
            g_oz_err = "cudaGetSymbolAddress of the static scratch failed";
            return HSDLA_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = reinterpret_cast<unsigned char *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return HSDLA_OK;
}

// Bytes of static scratch one call needs: two digit operands, their exponents, the
// job table and the error word.
int64_t noalloc_bytes(int s, int64_t n, int64_t Kpad) {
    return 2 * operand_bytes(s, n, Kpad) + round_up(sizeof(OzJob), 1024) + 1024;
}

}  // namespace
}  // namespace hsdla

extern "C" int hsdla_zherkx_lower_noalloc(int32_t num_slices, int64_t n, int64_t k, const hsdla_cx *dP, int64_t ldp,
                                          const hsdla_cx *dQ, int64_t ldq, const double *dw, hsdla_cx *dOut,
                                          int64_t ldo, void *stream) {
    using namespace hsdla;
    const int s = num_slices == 0 ? kOzDefaultSlices : num_slices;
    if (s < 2 || s > kOzMaxSlices) {
        g_oz_err = "num_slices outside [2, 12] (0 selects 11)";
        return HSDLA_ERR_ARG;
    }
    if (n < 0 || k < 0 || !dP || !dQ || !dOut || ldp < k || ldq < k || ldo < n) {
        g_oz_err = "bad arguments: n or k negative, a NULL buffer, or a leading dimension below k (inputs) or n "
                   "(output)";
        return HSDLA_ERR_ARG;
    }
    g_oz_err = "";
    if (n == 0) return HSDLA_OK;
    const int64_t Kpad = round_up(std::max<int64_t>(k, 1), kKBlock);
    if (noalloc_bytes(s, n, Kpad) > kNoAllocScratchBytes) {
        g_oz_err = "problem exceeds the 128 MiB static scratch of hsdla_zherkx_lower_noalloc";
        return HSDLA_ERR_UNSUPPORTED;
    }
    unsigned char *scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    Arena ar{reinterpret_cast<char *>(scratch)};
    DigitOperand dp, dq;
    carve_operand(ar, dp, s, n, Kpad);
    carve_operand(ar, dq, s, n, Kpad);
    OzJob *d_job = ar.take<OzJob>(1);
    int *d_err = ar.take<int>(1);
    // the array keeps the previous call's contents: the error word must start at zero
    // (digit planes and exponents are rewritten in full by the slicing kernel)
    cudaError_t e = cudaMemsetAsync(d_err, 0, sizeof(int), st);
    if (e == cudaSuccess) e = slice(reinterpret_cast<const double2 *>(dP), ldp, nullptr, k, n, Kpad, Kpad, s, dp, st);
    if (e == cudaSuccess) e = slice(reinterpret_cast<const double2 *>(dQ), ldq, dw, k, n, Kpad, Kpad, s, dq, st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    rc = make_map(dp, 2 * s);
    if (!rc) rc = make_map(dq, 2 * s);
    if (rc) return rc;
    OzJob j;
    memset(&j, 0, sizeof(j));
    j.lmap = 0; j.rmap = 1; j.lower = 1;
    j.lplane = dp.plane_rows; j.rplane = dq.plane_rows;
    j.nkb = Kpad / kKBlock; j.m = n; j.n = n;
    j.tiles_n = (n + kTileN - 1) / kTileN;
    j.tile_begin = 0;
    j.out = reinterpret_cast<double2 *>(dOut); j.ldo = ldo;
    j.el = dp.expo; j.er = dq.expo;
    const int64_t tiles = job_tiles(j);
    e = cudaMemcpyAsync(d_job, &j, sizeof(OzJob), cudaMemcpyHostToDevice, st);
    const size_t smem = (size_t)kStages * kStageBytes + 1024;
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(oz_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int dev = 0, nsm = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    const int64_t grid = std::min<int64_t>(tiles, nsm);
    oz_gemm_kernel<<<(unsigned)grid, kThreads, smem, st>>>(dp.map, dq.map, dp.map, dp.map, d_job, 1, tiles, s, d_err,
                                                            nullptr, nullptr);
    e = cudaGetLastError();
    int herr = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { g_oz_err = cudaGetErrorString(e); return HSDLA_ERR_CUDA; }
    if (herr != 0) {
        // the error word: code * 16 + the role whose bounded wait expired (1 TMA producer, 2 MMA
        // issuer waiting for a drained accumulator, 3 MMA issuer waiting for operands, 4 epilogue)
        static thread_local char buf[160];
        snprintf(buf, sizeof(buf), "device wait expired in hsdla_zherkx_lower_noalloc (code %d, role %d)", herr / 16,
                 herr % 16);
        g_oz_err = buf;
        return herr / 16 == kDevBadInput ? HSDLA_ERR_CUDA : HSDLA_ERR_TIMEOUT;
    }
    return HSDLA_OK;
}
