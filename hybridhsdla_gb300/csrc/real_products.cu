// Real digit products of the structure-factor form on the FP8 tensor cores.
//
// The matching rows of one type come in pairs: row (l, -m) is (-1)^m times the complex conjugate
// of row (l, m) (Y_l,-m = (-1)^m conj Y_lm).  With rho = (Re, Im of the rows m > 0; the real rows
// m = 0) the rows are M = V rho with V constant per pair, so
//     S_t[g, g'] = rho(g)^T diag(w'_t) rho(g'),            w' = 2 w on the rows of m != 0,
//     H_t[g, g'] = rho(g)^T (T'_t rho(g')),                T'_t = V^H T_t V:
// one real product for S and two for H where the complex rows need four each, over the same 2L
// rows (the rows rho are the very numbers of M; T' sums four entries of T).
//
// oz_real_kernel forms these products exactly as oz_pair_kernel does the complex ones (base-32
// digits in e4m3, FP32 accumulators that hold exact integers, the triangle i + j <= s + 1), with
// the work arranged for short real contractions (K = 2L):
//  * CTA pairs, 256 x 128 tiles, tcgen05.mma.cta_group::2 (M 256, N 128, K 32).
//  * The contraction runs in chunks of 64 digits.  All digit planes of a chunk (left 8 KB, right 4
//    KB each) are in shared memory together, so each is loaded once for all its digit pairs: 132 KB
//    per 8.4k MMA cycles and SM at s = 11 (16 B per cycle), where staging the planes pair by pair
//    takes 96 B per cycle.  (128-digit chunks leave no room to load ahead.)  Planes arrive and
//    leave in batches of four: a barrier per plane kept the MMA thread at its waits and commits
//    (150 cycles per MMA of 64).
//  * The digit pairs run in bands of two diagonals (RealBands) summed in one accumulator: the products
//    of the upper diagonal carry a factor 32, as the left operand's block scale (mxf8f6f4; the scale
//    factors 1 and 32 fill TMEM columns of their own).  A band leaves 128 columns of TMEM instead of 256
//    and takes one FP32 operation less per element.  Three accumulators take the bands in turn.
//  * Two threads issue the MMAs, every other band each: one takes ~75 cycles per MMA, of which it
//    must not take more than 80 and did not keep to with the epilogue's warps on its scheduler.
//  * The sums over diagonals and chunks stay in registers as 64-bit fixed-point numbers (64 per
//    thread of the eight epilogue warps): a band's FP32 integer becomes an integer by one FMA
//    (x + 1.5 2^23 leaves it in the low mantissa bits) and adds with one multiply-add.  Each output
//    element is written once, rather than once per accumulation unit through L2 reductions.  The
//    fixed-point sum is exact down to 2^-frac of a unit of the top diagonal.
//  * A tile is stored only when the next one's first band has left its accumulator, so the MMAs run
//    four bands ahead meanwhile.
// What bounds it: the tensor pipe, 0.93 of the time (0.83 ms with neither stores nor sums).  One type of
// the 8000-column workload (lmax 10, 11 digits): 3.05 ms in the complex form, 0.863 ms here = 3.56
// PFLOP/s of e4m3, 0.93 of twice the measured bf16 rate.  On the way: two accumulators a band, summed by
// the epilogue, and one issuer 1.067; block scales 1.059; the next tile's chunk count fetched ahead
// 1.033; the delayed store 1.004; two issuers 0.863.  Measured and not kept: sixteen epilogue warps with
// half the sums each, TMEM loads ahead of the arithmetic, shifts and adds in place of the wide
// multiply-adds, large bands first in a tile, right planes a chunk at a time ahead of the left ones.
// Every wait is bounded (ptx.cuh); both CTAs meet at a cluster barrier before TMEM is freed.
#include <cuda_fp8.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "digits.cuh"
#include "ptx.cuh"
#include "real_products.cuh"

namespace hsdla {
namespace {

constexpr int kThreads = 384;              // warps 0-3: TMA, MMA, idle, MMA; 4-11 epilogue
constexpr int kEpi = 8;
constexpr int kCols = kRealTileN / 2;      // columns of an epilogue warp (two warps per lane quadrant)
constexpr int kABytes = 128 * kRealKBlock, kBBytes = kRealBRows * kRealKBlock;
// Planes move in batches of kBatch digits.  Left planes: a ring of kRing batches, one more than a
// chunk has; right planes: a bank per chunk, two banks.
constexpr int kBatch = 4, kRing = 4, kNA = kRing * kBatch, kBank = kRealMaxSlices, kNB = 2 * kBank;
static_assert((kRing - 1) * kBatch >= kRealMaxSlices, "the ring holds a chunk's planes");
constexpr int kSmem = 1024 + kNA * kABytes + kNB * kBBytes;
static_assert(kSmem <= 226 * 1024, "shared memory (the barriers are static)");
// TMEM: buffers of one FP32 accumulator, then the scale factors 1 and 32 (all bytes of 32 columns each)
constexpr int kBufs = 3;
constexpr uint32_t kScaleOne = kBufs * kRealTileN, kScale32 = kScaleOne + 32;
constexpr uint32_t kOneBytes = 0x7F7F7F7Fu, k32Bytes = 0x84848484u;    // ue8m0
// Register split: 384 threads are launched with 168 registers each (64512); the control warps keep
// 56 and the epilogue warps get 216, 62464 in all.  launch_real_products checks the 168.
constexpr int kRegsLaunch = 168, kRegsControl = 56, kRegsEpilogue = 216;
static_assert(128 * kRegsControl + 256 * kRegsEpilogue <= kThreads * kRegsLaunch, "register split");

struct __align__(8) RealBarriers {
    uint64_t full[kRing];              // a batch's left and right planes landed (both CTAs')
    uint64_t aempty[kRing], bempty[2]; // a left batch, a right bank consumed
    uint64_t tfull[kBufs], tempty[kBufs];   // a band's accumulators in each TMEM buffer
};

__host__ __device__ constexpr uint32_t idesc_real() {
    return (1u << 4) | ((uint32_t)(kRealTileN >> 3) << 17) | ((uint32_t)(kRealTileM >> 4) << 24);
}

// The same with block scales (mxf8f6f4; scale factors in ue8m0, byte 0 of each TMEM word)
__host__ __device__ constexpr uint32_t idesc_scaled() {
    return ((uint32_t)(kRealTileN >> 3) << 17) | (1u << 23) | ((uint32_t)(kRealTileM >> 4) << 24);
}

// After an abort the copies and MMAs in flight have long landed: short waits for them
constexpr long long kAbortCycles = 100000000LL;

constexpr float kMagic = 12582912.0f;                  // 1.5 2^23
constexpr uint32_t kMagicBits = 0x4B400000u;

// One band's accumulators into the sums (RealBands).  One short path per kind of fold: a path per shift
// and width, and FP64 conversions at the tile's end, overflowed the instruction cache.
template <int kFold>
__device__ __forceinline__ void add_band(unsigned long long (&acc)[kCols], const uint32_t (&v)[2][32], float f,
                                         uint32_t mul) {
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
        const uint32_t b = __float_as_uint(fmaf(__uint_as_float(v[c / 32][c % 32]), f, kMagic));
        if (kFold == kFoldHigh) {
            const uint32_t lo = (uint32_t)acc[c], hi = (uint32_t)(acc[c] >> 32) + b * mul;
            acc[c] = ((unsigned long long)hi << 32) | lo;
        } else acc[c] += (unsigned long long)b * mul;
    }
}

// MMAs of the pair with operands given by the low words of their descriptors; the high word and the
// instruction descriptor are constants (fewer registers to move to the uniform file per MMA).
constexpr uint32_t kDescHi = (512u >> 4) | (1u << 14) | (4u << 29);    // SW64 K-major, 8 rows of 64 bytes
__device__ __forceinline__ void mma_real(uint32_t d, uint32_t a, uint32_t b, uint32_t acc) {
    asm volatile(
        "{\n .reg .b64 da, db;\n .reg .pred p;\n .reg .b32 h;\n mov.b32 h, %3;\n mov.b64 da, {%1, h};\n"
        " mov.b64 db, {%2, h};\n setp.ne.b32 p, %5, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], da, db, %4, p;\n}\n" ::"r"(d),
        "r"(a), "r"(b), "n"(kDescHi), "r"(idesc_real()), "r"(acc)
        : "memory");
}
// ... with the left operand scaled by the factors at sa (those at sb are 1)
__device__ __forceinline__ void mma_scaled(uint32_t d, uint32_t a, uint32_t b, uint32_t acc, uint32_t sa, uint32_t sb) {
    asm volatile(
        "{\n .reg .b64 da, db;\n .reg .pred p;\n .reg .b32 h;\n mov.b32 h, %3;\n mov.b64 da, {%1, h};\n"
        " mov.b64 db, {%2, h};\n setp.ne.b32 p, %5, 0;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], da, db, %4, [%6], [%7], p;\n}\n" ::"r"(d),
        "r"(a), "r"(b), "n"(kDescHi), "r"(idesc_scaled()), "r"(acc), "r"(sa), "r"(sb)
        : "memory");
}
// 32 columns of this warp's lane quadrant set to one word
__device__ __forceinline__ void tmem_fill32(uint32_t taddr, uint32_t v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
        "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr),
        "r"(v)
        : "memory");
}
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFF) >> 4) | (1u << 16); }

__global__ void __launch_bounds__(kThreads, 1)
    oz_real_kernel(const __grid_constant__ CUtensorMap lmap, const __grid_constant__ CUtensorMap rmap0,
                   const __grid_constant__ CUtensorMap rmap1, const RealJob *__restrict__ jobs, int64_t total_tiles,
                   const int4 *__restrict__ tile_list, int *err, const __grid_constant__ RealBands bands) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ RealBarriers bars;
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (cluster_size() != 2) {
        if (threadIdx.x == 0) atomicCAS(err, 0, kDevBadInput * 16 + 6);
        return;
    }
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    const int s = bands.s;
    auto expired = [&](uint32_t parity, int slot, int count) -> bool {
        if (atomicCAS(err + 7, 0, 1) == 0) {
            err[1] = blockIdx.x; err[2] = (int)rank; err[3] = slot; err[4] = (int)parity; err[5] = count;
        }
        return false;
    };
    auto pwait = [&](uint64_t *bar, uint32_t parity, int where, int slot, int count) -> bool {
        return mbar_wait(bar, parity, &abort_flag, err, where) || expired(parity, slot, count);
    };
    auto pwait_pair = [&](uint64_t *bar, uint32_t parity, int where, int slot, int count) -> bool {
        return mbar_wait<true>(bar, parity, &abort_flag, err, where) || expired(parity, slot, count);
    };
    const int64_t pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    unsigned char *abuf = smem, *bbuf = smem + kNA * kABytes;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kRing; ++i) { mbar_init(&bars.full[i], 1); mbar_init(&bars.aempty[i], 2); }
        for (int i = 0; i < 2; ++i) mbar_init(&bars.bempty[i], 2);
        for (int i = 0; i < kBufs; ++i) {
            mbar_init(&bars.tfull[i], 1);
            mbar_init(&bars.tempty[i], 2 * kEpi);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)&lmap) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)&rmap0) : "memory");
        asm volatile("prefetch.tensormap [%0];\n" ::"l"((uint64_t)&rmap1) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&tmem_base_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_sh;
    if (warp >= 4 && warp < 8) {
        const uint32_t t = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        tmem_fill32(t + kScaleOne, kOneBytes);
        tmem_fill32(t + kScale32, k32Bytes);
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // barriers and scale factors of both CTAs in place
    tc_fence_after();

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kRegsControl));
        const bool one = elect_one();
        if (warp == 0 && one) {
            // ------------------------------------------------ planes, in batches
            const uint32_t full_leader = mapa_rank(smem_u32(&bars.full[0]), 0);
            uint32_t n = 0, chunk = 0;               // batches issued, chunks begun
            bool ok = true;
            for (int64_t tile = pair; ok && tile < total_tiles; tile += npairs) {
                const int4 e = tile_list[tile];
                const RealJob &j = jobs[e.x];
                const CUtensorMap *rm = j.rmap ? &rmap1 : &rmap0;
                const int64_t lstep = j.lplane, rstep = j.rstep * j.rplane, nkb = j.nkb;
                int64_t yl = j.lrow0 + (int64_t)e.y * kRealTileM + rank * (kRealTileM / 2);
                int64_t yr = j.rpart * j.rplane + j.rrow0 + (int64_t)e.z * kRealTileN + rank * kRealBRows;
                const int64_t kl = j.lk0, kr = j.rk0;
                for (int64_t kb = 0; ok && kb < nkb; ++kb, ++chunk) {
                    const int xl = (int)(kl + kb * kRealKBlock), xr = (int)(kr + kb * kRealKBlock);
                    if (!pwait(&bars.bempty[chunk & 1], ((chunk >> 1) & 1) ^ 1, 7, (int)(chunk & 1), (int)chunk)) { ok = false; break; }
                    unsigned char *bp = bbuf + (chunk & 1) * kBank * kBBytes;
                    for (int i0 = 0; i0 < s; i0 += kBatch, ++n) {
                        const int slot = n % kRing, cnt = min(kBatch, s - i0);
                        if (!pwait(&bars.aempty[slot], ((n / kRing) & 1) ^ 1, 1, slot, (int)n)) { ok = false; break; }
                        if (leader) mbar_expect_tx(&bars.full[slot], 2 * cnt * (kABytes + kBBytes));
                        const uint32_t fb = full_leader + slot * 8;
                        for (int q = 0; q < cnt; ++q) {
                            tma_load_2d_pair(abuf + (slot * kBatch + q) * kABytes, &lmap, fb, xl, (int)(yl + (i0 + q) * lstep));
                            tma_load_2d_pair(bp + (i0 + q) * kBBytes, rm, fb, xr, (int)(yr + (i0 + q) * rstep));
                        }
                    }
                }
            }
            // every batch issued has been consumed before the CTA may exit (bounded after an abort):
            // its left planes' release follows the last use of its right planes or precedes their bank's
            const long long budget = ok ? kWaitCycles : kAbortCycles;
            for (uint32_t q = n > kRing ? n - kRing : 0; q < n; ++q)
                mbar_drain_wait(&bars.aempty[q % kRing], (q / kRing) & 1, budget);
            for (uint32_t c = chunk > 2 ? chunk - 2 : 0; c < chunk; ++c)
                mbar_drain_wait(&bars.bempty[c & 1], (c >> 1) & 1, budget);
        } else if ((warp & 1) && one && leader) {
            const uint32_t me = warp >> 1;           // the bands seq = me (mod 2) are this issuer's
            // ------------------------------------------------ MMA issuers
            const uint32_t da0 = desc_lo(smem_u32(abuf)), db0 = desc_lo(smem_u32(bbuf));
            constexpr uint32_t kAStep = kABytes >> 4, kBStep = kBBytes >> 4;
            uint32_t n = 0, chunk = 0, seq = 0;      // the chunk's first batch; chunks; bands so far
            const int nbuf = bands.halves == 2 ? kBufs : 1, nbatch = (s + kBatch - 1) / kBatch, nbands = bands.n;
            const int step = nbuf == 1 ? 1 : 2;
            bool ok = true, cut = false;
            // (a tile's chunk count is fetched while the tile before runs)
            int nkb = 0, ksl = 0, nkb1 = 0, ksl1 = 0;
            if (pair < total_tiles) {
                const RealJob &j = jobs[tile_list[pair].x];
                nkb1 = (int)j.nkb;
                ksl1 = j.ksteps_last;
            }
            for (int64_t tile = pair; ok && tile < total_tiles; tile += npairs) {
                nkb = nkb1;
                ksl = ksl1;
                if (tile + npairs < total_tiles) {
                    const RealJob &j = jobs[tile_list[tile + npairs].x];
                    nkb1 = (int)j.nkb;
                    ksl1 = j.ksteps_last;
                }
                for (int kb = 0; ok && kb < nkb; ++kb, ++chunk, n += nbatch) {
                    const bool two = kb + 1 < nkb || ksl > 1;      // K steps of the chunk
                    const uint32_t db = db0 + (chunk & 1) * kBank * kBStep;
                    int ready = 0;                                 // left batches seen to have landed
                    // this issuer's bands of the chunk; the last one also frees the planes (a chunk without a
                    // band of its own is only signed off), all of them seen to have landed before, so that no
                    // barrier is signed twice in a phase.  One buffer has one issuer: the other could not tell
                    // its phases apart
                    const int b0 = nbuf == 1 ? (me ? nbands : 0) : (int)((seq ^ me) & 1);
                    const uint32_t seq0 = seq;
                    seq += b0;
                    if (b0 >= nbands) {
                        for (; ready < nbatch; ++ready)
                            if (!pwait(&bars.full[(n + ready) % kRing], ((n + ready) / kRing) & 1, 3, ready, (int)seq)) { ok = false; break; }
                        if (!ok) break;
                        for (int q = 0; q < nbatch; ++q) mma_commit_pair(&bars.aempty[(n + q) % kRing]);
                        mma_commit_pair(&bars.bempty[chunk & 1]);
                    }
                    for (int b = b0; b < nbands; b += step, seq += step) {
                        const int T = bands.T[b];
                        const bool last = b + step >= nbands, pairs = bands.w[b] == 2;
                        const uint32_t use = nbuf == 1 ? seq : seq / kBufs;
                        const int h = (int)(seq - use * nbuf);
                        if (!pwait_pair(&bars.tempty[h], (use & 1) ^ 1, 2, b, (int)seq)) { ok = false; break; }
                        for (; ready <= (last ? nbatch - 1 : (T - 2) / kBatch); ++ready)
                            if (!pwait(&bars.full[(n + ready) % kRing], ((n + ready) / kRing) & 1, 3, ready, (int)seq)) { ok = false; break; }
                        if (!ok) break;
                        tc_fence_after();
                        cut = true;
                        const uint32_t d = tmem_base + h * kRealTileN, one = tmem_base + kScaleOne, x32 = tmem_base + kScale32;
                        // left plane i with right planes T - 1 - i (diagonal T - 1, times 32) and T - i (diagonal T)
                        uint32_t dt = db + (T - 2) * kBStep;
                        for (int i0 = 1; i0 < T; i0 += kBatch) {
                            const int slot = (n + (i0 - 1) / kBatch) % kRing;
                            uint32_t da = da0 + slot * kBatch * kAStep;
                            const int i1 = min(i0 + kBatch, T);
                            if (two && i0 + kBatch < T) {
                                // a whole batch as straight-line code
                                if (pairs) {
#pragma unroll
                                    for (int q = 0; q < kBatch; ++q, da += kAStep, dt -= kBStep) {
                                        const uint32_t dl = dt - kBStep;
                                        mma_scaled(d, da, dl, q > 0 || i0 > 1 ? 1u : 0u, x32, one);
                                        mma_scaled(d, da, dt, 1u, one, one);
                                        mma_scaled(d, da + 2, dl + 2, 1u, x32, one);
                                        mma_scaled(d, da + 2, dt + 2, 1u, one, one);
                                    }
                                } else {
#pragma unroll
                                    for (int q = 0; q < kBatch; ++q, da += kAStep, dt -= kBStep) {
                                        mma_real(d, da, dt, q > 0 || i0 > 1 ? 1u : 0u);
                                        mma_real(d, da + 2, dt + 2, 1u);
                                    }
                                }
                            } else {
                                for (int i = i0; i < i1; ++i, da += kAStep, dt -= kBStep) {
                                    const uint32_t acc = i > 1 ? 1u : 0u;
                                    if (pairs) {
                                        if (i + 1 < T) {
                                            const uint32_t dl = dt - kBStep;
                                            mma_scaled(d, da, dl, acc, x32, one);
                                            if (two) mma_scaled(d, da + 2, dl + 2, 1u, x32, one);
                                        }
                                        mma_scaled(d, da, dt, i + 1 < T ? 1u : acc, one, one);
                                        if (two) mma_scaled(d, da + 2, dt + 2, 1u, one, one);
                                    } else {
                                        mma_real(d, da, dt, acc);
                                        if (two) mma_real(d, da + 2, dt + 2, 1u);
                                    }
                                }
                            }
                            if (last) mma_commit_pair(&bars.aempty[slot]);     // the batch's last use
                        }
                        if (last)
                            for (int q = (T + kBatch - 2) / kBatch; q < nbatch; ++q) mma_commit_pair(&bars.aempty[(n + q) % kRing]);
                        mma_commit_pair(&bars.tfull[h]);
                        if (last) mma_commit_pair(&bars.bempty[chunk & 1]);
                        cut = false;
                    }
                    if (ok) seq = seq0 + nbands;
                }
            }
            if (!ok) {
                // wait (bounded) for the MMAs of a band cut short: the commit tracks all of them
                if (cut) {
                    const uint32_t use = nbuf == 1 ? seq : seq / kBufs, h = seq - use * nbuf;
                    mma_commit_pair(&bars.tfull[h]);
                    mbar_drain_wait(&bars.tfull[h], use & 1);
                }
            } else {
                // both CTAs' drains of the last bands
                for (uint32_t q = seq > (uint32_t)nbuf ? seq - nbuf : 0; q < seq; ++q) {
                    const uint32_t use = nbuf == 1 ? q : q / kBufs, h = q - use * nbuf;
                    mbar_drain_wait(&bars.tfull[h], use & 1);
                    mbar_drain_wait(&bars.tempty[h], use & 1);
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------ epilogue
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kRegsEpilogue));
        const int q4 = warp & 3, cbeg = ((warp - 4) >> 2) * kCols;
        const uint32_t tempty_leader = mapa_rank(smem_u32(&bars.tempty[0]), 0);
        const uint32_t tb = tmem_base + ((uint32_t)(q4 * 32) << 16) + cbeg;
        uint32_t seq = 0;
        bool ok = true;
        const uint32_t nbuf = bands.halves == 2 ? kBufs : 1;
        unsigned long long acc[kCols];
        long long *out = nullptr;                 // the tile whose sums acc holds: where they go
        int64_t ldo = 0;
        int live = 0;
        auto store = [&]() {
#pragma unroll
            for (int c = 0; c < kCols; ++c)
                if (c < live) out[ldo * c] = (long long)acc[c];
        };
        for (int64_t tile = pair; ok && tile < total_tiles; tile += npairs) {
            const int4 te = tile_list[tile];
            const RealJob &j = jobs[te.x];
            const int nkb = (int)j.nkb;
            for (int kb = 0; ok && kb < nkb; ++kb) {
                for (int b = 0; b < bands.n; ++b, ++seq) {
                    const uint32_t use = nbuf == 1 ? seq : seq / kBufs, h = seq - use * nbuf;
                    if (!pwait(&bars.tfull[h], use & 1, 8, warp, (int)seq)) { ok = false; break; }
                    tc_fence_after();
                    const float f = bands.f[b];
                    const uint32_t mul = bands.mul[b], t = tb + h * kRealTileN;
                    uint32_t v[2][32];
                    tmem_ld32(t, v[0]);
                    tmem_ld32(t + 32, v[1]);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_pair(tempty_leader + h * 8);
                    if (kb == 0 && b == 0) {
                        // the tile before leaves only here, after this band has left its buffer: the MMAs
                        // run ahead by one more band while it is being stored
                        store();
                        const unsigned long long a0 = 0ull - bands.bias * (unsigned long long)nkb;
#pragma unroll
                        for (int c = 0; c < kCols; ++c) acc[c] = a0;
                        // lane = row, so a column's 32 values are 256 consecutive bytes
                        const int64_t row = (int64_t)te.y * kRealTileM + rank * (kRealTileM / 2) + q4 * 32 + lane;
                        const int64_t col0 = (int64_t)te.z * kRealTileN + cbeg;
                        const int64_t cend = j.lower ? min(j.n, row + 1) : j.n;
                        ldo = j.ldo;
                        out = j.out + row + ldo * col0;
                        live = row < j.m ? (int)max((int64_t)0, min((int64_t)kCols, cend - col0)) : 0;
                    }
                    if (bands.fold[b] == kFoldHigh) add_band<kFoldHigh>(acc, v, f, mul);
                    else add_band<kFoldLow>(acc, v, f, mul);
                }
            }
        }
        if (ok) store();
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // neither CTA frees TMEM or exits while the other may address it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(tmem_base) : "memory");
    }
}

// ------------------------------------------------------------------ slicing of real columns
// As oz_slice_kernel (the same digits of the same values): one CTA per plane row, first the
// column's largest magnitude (its exponent), then X = rint(z 2^(5s-1-e)) of eight consecutive
// contraction bytes per thread and their balanced base-32 digits, one 8-byte store per plane.
constexpr int kSliceThreads = 256;
constexpr int kVec = 8;

__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
// frexp's exponent of a positive finite double given as bits
__device__ __forceinline__ int frexp_exp_bits(unsigned long long b) {
    const int E = (int)(b >> 52) & 0x7ff;
    if (E) return E - 1022;
    return -1010 - __clzll((long long)(b & 0xfffffffffffffull));
}
// x 2^k rounded to nearest (halves away from zero), for |x 2^k| < 2^62
__device__ __forceinline__ long long rint_pow2(double x, int k) {
    const int hi = __double2hiint(x), E = (hi >> 20) & 0x7ff;
    const unsigned long long m = ((unsigned long long)(uint32_t)((hi & 0xfffff) | (E ? 0x100000 : 0)) << 32) | (uint32_t)__double2loint(x);
    const int sh = 1084 - max(E, 1) - k;
    // (sh < 0: a column of subnormal numbers)
    const long long q = (long long)(sh < 0 ? m << min(9 - sh, 63) : (((m << 10) >> min(sh, 63)) + 1) >> 1);
    return hi < 0 ? -q : q;
}

__device__ __forceinline__ unsigned long long block_max(unsigned long long m, unsigned long long *red) {
    for (int o = 16; o > 0; o >>= 1) m = max(m, (unsigned long long)__shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    unsigned long long r = 0;
    for (int i = 0; i < (int)blockDim.x / 32; ++i) r = max(r, red[i]);
    return r;
}

// kFixed: the source is a product's fixed-point numbers (parts rows exponents el, see RealSliceTab).
// One thread per eight contraction bytes up to kSliceThreads; a thread's first eight values (all of them up to
// 2048 bytes) stay in registers between the two passes; they and their exponents and weights come in pairs
// (launch_real_slice checks that they can).  Bound by the integer pipe.  The 8000-column workload's (8
// types, lmax 10, 12 digits) columns with their weighted copy take 167 us, its fixed-point ones 160 (both passes
// reading single values, 256 threads a column: 209 and 207; with 768 contraction bytes a column: 278 and 253
// us, now 187 and 204).
template <bool kDual, bool kFixed>
__global__ void __launch_bounds__(kSliceThreads) oz_slice_real_kernel(const __grid_constant__ RealSliceTab tab) {
    __shared__ unsigned long long red[2][kSliceThreads / 32];
    const int64_t r = blockIdx.x;
    int k = 0;
    while (k + 1 < tab.nk && tab.e[k + 1].row0 <= r) ++k;
    const int64_t g = r - tab.e[k].row0;
    const bool live = g >= 0 && g < tab.e[k].ncols;
    const long long *Z = reinterpret_cast<const long long *>(tab.e[k].Z) + tab.ldz * (live ? g : 0);
    const int rpb = live ? (int)tab.rpb : 0, bpad = (int)tab.bpad, nblk = (int)tab.blocks, parts = tab.parts, s = tab.s;
    const int bch = bpad / kVec, nch = bch * nblk;               // chunks of a block and part; of a part
    struct Place {
        int b, p, r0;
    };
    auto place = [&](int c) {
        const int p = c / nch, cc = c - p * nch, b = cc / bch;
        return Place{b, p, (cc - b * bch) * kVec};
    };
    // eight values of a chunk, and their weighted copies or row exponents (zeros past the rows)
    auto load = [&](const Place &q, long long (&z)[kVec], double (&y)[kVec], int (&el)[kVec]) {
        const longlong2 *src = reinterpret_cast<const longlong2 *>(Z + (int64_t)q.b * tab.bstride + q.p * tab.pstride + q.r0);
        const int2 *ex = kFixed ? reinterpret_cast<const int2 *>(tab.el + (int64_t)tab.set_type[q.b] * tab.bstride + q.p * tab.pstride + q.r0)
                                : nullptr;
        const double2 *w = kDual ? reinterpret_cast<const double2 *>(tab.v2 + q.b * rpb + q.r0) : nullptr;
#pragma unroll
        for (int u = 0; u < kVec; u += 2) {
            const bool in = q.r0 + u < rpb;
            const longlong2 x = in ? src[u / 2] : make_longlong2(0, 0);
            z[u] = x.x;
            z[u + 1] = x.y;
            if constexpr (kFixed) {
                const int2 e = in ? ex[u / 2] : make_int2(0, 0);
                el[u] = e.x;
                el[u + 1] = e.y;
            }
            if constexpr (kDual) {
                const double2 v = in ? w[u / 2] : make_double2(0.0, 0.0);
                y[u] = __longlong_as_double(x.x) * v.x;
                y[u + 1] = __longlong_as_double(x.y) * v.y;
            }
        }
    };
    // (a fixed-point number's bit length and row exponent, offset to stay positive, order as |value|)
    constexpr int kOff = 1 << 20;
    unsigned long long mx = 0, mx2 = 0;
    int mxf = 0;
    auto largest = [&](const long long (&z)[kVec], const double (&y)[kVec], const int (&el)[kVec]) {
#pragma unroll
        for (int u = 0; u < kVec; ++u) {
            if constexpr (kFixed) {
                if (z[u]) mxf = max(mxf, kOff + 64 - __clzll(z[u] < 0 ? -z[u] : z[u]) + el[u]);
            } else {
                mx = max(mx, (unsigned long long)z[u] & 0x7fffffffffffffffull);
                if (kDual) mx2 = max(mx2, abs_bits(y[u]));
            }
        }
    };
    long long z[kVec];
    double y[kVec];
    int el[kVec];
    const Place first = place((int)threadIdx.x);
    const bool any = threadIdx.x < nch * parts;
    if (any) {
        load(first, z, y, el);
        largest(z, y, el);
    }
    for (int c = threadIdx.x + blockDim.x; c < nch * parts; c += blockDim.x) {
        long long zc[kVec];
        double yc[kVec];
        int ec[kVec];
        load(place(c), zc, yc, ec);
        largest(zc, yc, ec);
    }
    int e = 0, e2 = 0, q = 0;
    const unsigned long long m = block_max(kFixed ? (unsigned long long)mxf : mx, red[0]);
    if constexpr (kFixed) {
        q = (live ? tab.er[r] : 0) - 8 - tab.frac;               // the column's part of the values' exponent
        if (m > 0) e = (int)m - kOff + q;
    } else if (m > 0) e = frexp_exp_bits(m);
    if (kDual) {
        const unsigned long long m2 = block_max(mx2, red[1]);
        if (m2 > 0) e2 = frexp_exp_bits(m2);
    }
    if (threadIdx.x == 0) {
        tab.expo[r] = e;
        if (kDual) tab.expo2[r] = e2;
    }
    const int top = 5 * s - 1;
    long long B = 0;
    for (int p = 0; p < s - 1; ++p) B |= 16ll << (5 * p);
    const int64_t plane = tab.plane_rows * tab.pitch;
    auto digits = [&](const Place &at, const long long (&z)[kVec], const double (&y)[kVec], const int (&el)[kVec]) {
        long long x[kVec];
#pragma unroll
        for (int u = 0; u < kVec; ++u) {
            if constexpr (kFixed) {
                // F 2^(el + q) scaled by 2^(top - e): a shift, rounded half up
                const int d = el[u] + q + top - e;
                x[u] = B + (d >= 0 ? z[u] << min(d, 63) : d < -63 ? 0 : ((z[u] >> (-d - 1)) + 1) >> 1);
            } else x[u] = B + rint_pow2(__longlong_as_double(z[u]), top - e);
        }
        const int64_t o = r * tab.pitch + (int64_t)at.b * bpad + at.r0;
        write_digits<kVec>(x, s, tab.digits + o + at.p * plane, parts * plane);
        if constexpr (kDual) {
#pragma unroll
            for (int u = 0; u < kVec; ++u) x[u] = B + rint_pow2(y[u], top - e2);
            write_digits<kVec>(x, s, tab.digits2 + o, plane);
        }
    };
    if (any) digits(first, z, y, el);
    for (int c = threadIdx.x + blockDim.x; c < nch * parts; c += blockDim.x) {
        const Place at = place(c);
        load(at, z, y, el);
        digits(at, z, y, el);
    }
}

}  // namespace

RealBands real_bands(int s, int width, int halves, int64_t kvalid) {
    RealBands b;
    memset(&b, 0, sizeof(b));
    b.s = s;
    b.halves = halves;
    width = std::max(1, std::min(width, 2));
    // |sum| <= kvalid 2^8 (operands below 2^4 in units of their top digit) stays below 2^(63 - frac)
    int kb = 0;
    while (((int64_t)1 << kb) <= kvalid) ++kb;
    b.frac = 55 - kb;
    // Pairs while the largest |32 x0 + x1| of a chunk (64 products of at most 2^8 per digit pair) stays
    // below 2^22, from the first diagonals on: theirs are the bands shorter than a drain.
    for (int t = 1, T; t < s + 1; t = T) {
        T = std::min(t + width, s + 1);
        if (T - t == 2 && (int64_t)kRealKBlock * 256 * (32 * (T - 2) + T - 1) >= 1 << 22) T = t + 1;
        const int n = b.n++, sh = b.frac - 5 * (T - 2);
        b.T[n] = (int8_t)T;
        b.w[n] = (int8_t)(T - t);
        b.fold[n] = sh >= 32 ? kFoldHigh : kFoldLow;
        b.mul[n] = sh >= 32 ? 1u << (sh - 32) : 1u << std::max(sh, 0);
        b.f[n] = std::ldexp(1.0f, std::min(sh, 0));       // below the fixed point the sums are rounded to it
        b.bias += b.fold[n] == kFoldHigh ? (unsigned long long)(kMagicBits * b.mul[n]) << 32
                                         : (unsigned long long)kMagicBits * b.mul[n];
    }
    return b;
}

int64_t real_job_tiles(const RealJob &j) {
    const int64_t tm = (j.m + kRealTileM - 1) / kRealTileM, tn = (j.n + kRealTileN - 1) / kRealTileN;
    if (!j.lower) return tm * tn;
    int64_t t = 0;
    for (int64_t i = 0; i < tm; ++i) t += std::min(tn, (i + 1) * (kRealTileM / kRealTileN));
    return t;
}

void real_schedule(const std::vector<RealJob> &jobs, std::vector<int4> &list) {
    // super-blocks of 4 x 8 tiles (1024 rows and columns) keep a wave's operand planes in L2
    constexpr int64_t kSB = 4, kRatio = kRealTileM / kRealTileN;
    list.clear();
    for (size_t a = 0; a < jobs.size();) {
        const RealJob &ja = jobs[a];
        const int64_t tm = (ja.m + kRealTileM - 1) / kRealTileM, tn = (ja.n + kRealTileN - 1) / kRealTileN;
        if (!ja.lower) {
            for (int64_t c = 0; c < tn; ++c)
                for (int64_t r = 0; r < tm; ++r) list.push_back(make_int4((int)a, (int)r, (int)c, 0));
            ++a;
            continue;
        }
        size_t b = a;
        while (b < jobs.size() && jobs[b].lower && jobs[b].n == ja.n && jobs[b].lrow0 == ja.lrow0 && jobs[b].lk0 == ja.lk0) ++b;
        for (int64_t I = 0; I < tm; I += kSB)
            for (int64_t J = 0; J <= I; J += kSB)
                for (int64_t r = I; r < std::min(tm, I + kSB); ++r)
                    for (int64_t c = J * kRatio; c < std::min(std::min(tn, (r + 1) * kRatio), (J + kSB) * kRatio); ++c)
                        for (size_t q = a; q < b; ++q) list.push_back(make_int4((int)q, (int)r, (int)c, 0));
        a = b;
    }
}

cudaError_t launch_real_products(const CUtensorMap &left, const CUtensorMap &right0, const CUtensorMap &right1,
                                 const RealJob *d_jobs, const int4 *d_list, int64_t tiles, const RealBands &bands,
                                 int *d_err, cudaStream_t st) {
    if (tiles <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(oz_real_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    static int max_pairs = 0;
    if (max_pairs == 0) {
        // the register split draws on what the block was launched with
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, oz_real_kernel);
        if (e != cudaSuccess) return e;
        if (fa.numRegs * kThreads < 128 * kRegsControl + 256 * kRegsEpilogue) return cudaErrorInvalidConfiguration;
        cfg.gridDim = dim3(2);
        int nc = 0;
        e = cudaOccupancyMaxActiveClusters(&nc, (const void *)oz_real_kernel, &cfg);
        if (e != cudaSuccess) return e;
        if (nc < 1) return cudaErrorInvalidConfiguration;
        max_pairs = nc;
    }
    cfg.gridDim = dim3((unsigned)(2 * std::min<int64_t>(tiles, max_pairs)));
    return cudaLaunchKernelEx(&cfg, oz_real_kernel, left, right0, right1, d_jobs, tiles, d_list, d_err, bands);
}

cudaError_t launch_real_slice(const RealSliceTab &t, cudaStream_t st) {
    if (t.plane_rows <= 0) return cudaSuccess;
    // pairs of values, weights and exponents: 2L rows a block and aligned arrays, as every caller has them
    if ((t.rpb | t.ldz | t.bstride | t.pstride) & 1 || reinterpret_cast<uintptr_t>(t.v2) % 16 || reinterpret_cast<uintptr_t>(t.el) % 8)
        return cudaErrorInvalidValue;
    for (int k = 0; k < t.nk; ++k)
        if (reinterpret_cast<uintptr_t>(t.e[k].Z) % 16) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)t.plane_rows;
    const unsigned threads = (unsigned)std::min<int64_t>(kSliceThreads, (t.bpad / kVec * t.blocks * t.parts + 31) / 32 * 32);
    if (t.frac) oz_slice_real_kernel<false, true><<<grid, threads, 0, st>>>(t);
    else if (t.digits2) oz_slice_real_kernel<true, false><<<grid, threads, 0, st>>>(t);
    else oz_slice_real_kernel<false, false><<<grid, threads, 0, st>>>(t);
    return cudaGetLastError();
}

}  // namespace hsdla
