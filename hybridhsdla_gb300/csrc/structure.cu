// Structure-factor form of S and H for plans whose atoms share their type's rotation.
//
// With C_a = phi_a (.) M_t(a) and X_a = phi_a (.) Z_t(a), phi_a(g) = e^{i 2pi (k+g).tau_a} (the
// per-type rows M_t and Z_t = T_t M_t of the hoisted T application), the per-atom sums of
// create_HS2_stripped_v2 (flapw_opt/src/h_and_s_stripped_v2.cpp:155-368) regroup by type:
//     S[g, g'] = sum_t SF_t(g' - g) (M_t^H diag(w_t) M_t)[g, g'],
//     H[g, g'] = sum_t SF_t(g' - g) (M_t^H Z_t)[g, g'],
//     SF_t(dG) = sum_{a of type t} e^{i 2pi dG.tau_a}          (k cancels),
// so the contractions run over 2L rows per type instead of 2L rows per atom (a factor of atoms
// per type fewer products), and the structure factors enter once per element and type.
#include <algorithm>

#include "common.cuh"

namespace hsdla {

namespace {

__device__ __forceinline__ double2 cmul_d(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}


// sf[((ix ny + iy) nz + iz) nt + t] = sum over the atoms of type t of ex[a][ix] ey[a][iy] ez[a][iz],
// the atoms listed type by type (order[type_begin[t] .. type_begin[t+1])).  One CTA per (ix, t):
// the products ex ey of a chunk of atoms go to shared memory once per block of entries, and each
// entry then costs one complex FMA per atom (FP64, the pipe that bounds this table).
constexpr int kSfChunk = 16, kSfTabThreads = 256, kSfSmem = 48 * 1024;
__global__ void __launch_bounds__(kSfTabThreads) sf_table_kernel(const double2 *__restrict__ ex,
                                                                 const double2 *__restrict__ ey,
                                                                 const double2 *__restrict__ ez,
                                                                 const int32_t *__restrict__ order,
                                                                 const int32_t *__restrict__ type_begin,
                                                                 const int32_t *__restrict__ bits, int nx, int ny, int nz,
                                                                 int chunk, void *__restrict__ sf) {
    extern __shared__ double2 pxy[];            // [chunk][ny]
    const int ix = blockIdx.x, t = blockIdx.y;
    const int64_t nyz = (int64_t)ny * nz;
    const int a0 = type_begin[t], a1 = type_begin[t + 1];
    const int nt = gridDim.y;
    for (int64_t e0 = 0; e0 < nyz; e0 += blockDim.x) {
        const int64_t e = e0 + threadIdx.x;
        const int iy = (int)(e / nz), iz = (int)(e % nz);
        double2 acc = make_double2(0.0, 0.0);
        for (int c0 = a0; c0 < a1; c0 += chunk) {
            const int nc = min(chunk, a1 - c0);
            __syncthreads();
            for (int w = threadIdx.x; w < nc * ny; w += blockDim.x) {
                const int k = w / ny, y = w - k * ny;
                const int a = order[c0 + k];
                pxy[k * ny + y] = cmul_d(ex[(int64_t)a * nx + ix], ey[(int64_t)a * ny + y]);
            }
            __syncthreads();
            if (e < nyz)
                for (int k = 0; k < nc; ++k) {
                    const double2 p = pxy[k * ny + iy], z = ez[(int64_t)order[c0 + k] * nz + iz];
                    acc.x = fma(p.x, z.x, fma(-p.y, z.y, acc.x));
                    acc.y = fma(p.x, z.y, fma(p.y, z.x, acc.y));
                }
        }
        if (e < nyz) {
            const int64_t o = ((int64_t)ix * nyz + e) * nt + t;
            if (!bits) {
                static_cast<double2 *>(sf)[o] = acc;
            } else {
                const double s = __longlong_as_double((long long)(1023 + bits[t]) << 52);
                const long long re = __double2ll_rn(acc.x * s), im = __double2ll_rn(acc.y * s);
                constexpr int kLow = (1 << 28) - 1;
                static_cast<int4 *>(sf)[o] = make_int4((int)(re >> 28), (int)(re & kLow), (int)(im >> 28), (int)(im & kLow));
            }
        }
    }
}

// Exact sums of products p f of 64-bit fixed-point products p and structure factors f of up to 59 bits, in four
// 64-bit sums of the limb products: p = p1 2^32 + p0 with p0 in [-2^31, 2^31) and |p1| < 2^31, f = f1 2^28 + f0
// with f0 in (-2^28, 2^28).  kSumTypes types of two terms each overflow no sum with f0, and a group's types
// (sf_fixed_points) none with f1, so a term is four multiply-adds and no carry.
constexpr int kSumTypes = 8;
struct Limbs {
    int hi, lo;
    __device__ __forceinline__ explicit Limbs(int2 p) : hi(p.y + (p.x < 0 ? 1 : 0)), lo(p.x) {}   // (x: the low word)
};
struct LimbSum {
    long long a11 = 0, a10 = 0, a01 = 0, a00 = 0;
    __device__ __forceinline__ void add(Limbs p, int f1, int f0) {
        a11 += (long long)p.hi * f1;
        a10 += (long long)p.hi * f0;
        a01 += (long long)p.lo * f1;
        a00 += (long long)p.lo * f0;
    }
    // the sum times 2^k as a double: the bits below 2^36 dropped (the terms' own last places are above
    // 2^50), the rest rounded on the integer pipes (the FP64 pipe, which a conversion instruction uses
    // too, takes 64 cycles per warp instruction and scheduler: with three conversions the 2 k-points of
    // the kernel's comment took 1.88 ms)
    __device__ __forceinline__ double value(int k) const {
        const long long m = (a10 >> 4) + (a01 >> 8) + (a00 >> 36), top = a11 + (m >> 24);
        const int sign = (int)(top >> 63);
        // the magnitude's 96 bits (less one place of 2^36 where negative), its leading one to the top
        uint32_t w2 = (uint32_t)(top >> 32) ^ sign, w1 = (uint32_t)top ^ sign, w0 = ((uint32_t)m << 8) ^ sign;
        k += 1022 + 36 + 24 + 63;
        if (w2 == 0) { w2 = w1; w1 = w0; w0 = 0; k -= 32; }
        const int lz = __clz((int)w2);
        const uint32_t hi = __funnelshift_l(w1, w2, lz), lo = __funnelshift_l(w0, w1, lz);
        k -= lz;
        if (w2 == 0 || k <= 0 || k >= 2046) return small_or_large(top, (uint32_t)m & 0xffffffu, k + lz);
        // 53 bits, the next one rounding; the leading one counts in the exponent
        const unsigned long long b = (((unsigned long long)hi << 32) | lo) >> 11;
        const unsigned long long r = b + ((lo >> 10) & 1u) + ((unsigned long long)(uint32_t)k << 52);
        return __longlong_as_double((long long)(r | ((unsigned long long)(uint32_t)(sign & 0x80000000) << 32)));
    }
    // sums that the exponent range or 32 leading zeros take out of the path above (`k` as there)
    static __device__ __noinline__ double small_or_large(long long top, uint32_t low, int k) {
        if (top == 0 && low == 0) return 0.0;
        return ldexp((double)top + (double)low * 5.9604644775390625e-8, k - (1022 + 63) + (k_small(top) ? 32 : 0));
    }
    static __device__ __forceinline__ bool k_small(long long top) { return ((uint32_t)((top ^ (top >> 63)) >> 32)) == 0; }
};

constexpr int kSfTile = 32;

// out (+)= sum over the batch's types t of SF_t(g_col - g_row) * P_t over the lower triangle of
// every entry (S, then H), one CTA per 32 x 32 tile, a warp per column, consecutive lanes on consecutive
// rows.  A batch of several types reads and writes S and H once.  The tiles of an entry are its tile
// columns [tc0, tc1) (a column range of the launch), each from the diagonal tile down.  S_t is real
// and H_t complex: six real products per element and type.
// The structure factors of a column's 32 elements lie in 32 places of the table, each with its types
// together; the warp fetches them with lanes side by side on an element's types and hands them over in
// shared memory (a lane fetching its own element's cost a cache line per lane and type, which bounded
// the kernel).
// A warp's work is cut into items, four types of one column: an item's structure factors and products
// arrive in one of two stages of shared memory by asynchronous copies while the item before is summed.
// kFixed: fixed-point products and structure factors, summed exactly in integers.  GB300's FP64 pipe
// (2 multiply-adds per cycle and SM) bounded this kernel at 0.95 of its rate.  8000 columns of 8 types:
// FP64 2.60 ms, integers 1.39 ms (0.77 of the measured copy rate); 2 k-points of 6300 columns and 4 types: 1.74 and 1.13
// ms.  Bound now by the wide multiply-adds (a warp's takes four cycles; 24 an element and type) on 16 warps an
// SM; 20 warps leave too little L1 beside the stages (1.67 and 1.44 ms).  Loads into registers, four types
// ahead of their use on 24 warps, took 1.59 and 1.41 ms.
constexpr int kChunk = kSfItemTypes, kSumItems = kSumTypes / kChunk;     // types of an item; items of a full sum
constexpr int kSfPitch = kChunk + 1;                             // 16-byte words of an element's structure factors
constexpr int kStageSf = kSfTile * kSfPitch * 16, kStageBytesWarp = kStageSf + 3 * kChunk * kSfTile * 8;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_but_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

template <bool kFixed>
struct Sums {
    double2 s = make_double2(0.0, 0.0), h = make_double2(0.0, 0.0);
    __device__ __forceinline__ void add(int2 a, int2 c, int2 d, int4 w) {
        auto dbl = [](int lo, int hi) { return __hiloint2double(hi, lo); };
        const double fr = dbl(w.x, w.y), fi = dbl(w.z, w.w), x = dbl(a.x, a.y), y = dbl(c.x, c.y), z = dbl(d.x, d.y);
        s.x = fma(fr, x, s.x);
        s.y = fma(fi, x, s.y);
        h.x = fma(fr, y, fma(-fi, z, h.x));
        h.y = fma(fr, z, fma(fi, y, h.y));
    }
};
template <>
struct Sums<true> {
    LimbSum sr, si, hr, hi;
    __device__ __forceinline__ void add(int2 a, int2 c, int2 d, int4 w) {
        const Limbs x(a), y(c), z(d);
        sr.add(x, w.x, w.y);
        si.add(x, w.z, w.w);
        hr.add(y, w.x, w.y);
        hr.add(z, -w.z, -w.w);
        hi.add(z, w.x, w.y);
        hi.add(y, w.z, w.w);
    }
};

// (a call: the additions that a batch does not need would issue all the same, predicated off: 1.44 ms of the
// 8000 columns above where this took 1.42)
__device__ __noinline__ double2 sum2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// kItems: the items and ends of the sums as listed (SfTab::item); else four types each (the last fewer) and every second
// item or the last, of one fixed point, SfTab::bits0 (combine and slicing of 8000 columns of 8 equal types: listed 1.84 ms,
// 1.79 here; of 1 to 33 atoms, a group of seven types and one of one: 2.23).
template <bool kFixed, int kRows, bool kItems>
__global__ void __launch_bounds__(kSfTile *kRows, 512 / (kSfTile * kRows)) sf_combine_kernel(const __grid_constant__ SfTab tab,
                                                                                     const int4 *__restrict__ sf, int first) {
    extern __shared__ __align__(16) unsigned char stages[];
    const int64_t tile = blockIdx.x;
    int k = 0;
    while (k + 1 < tab.nk && tab.e[k + 1].tile_begin <= tile) ++k;
    const SfEntry &E = tab.e[k];
    const int64_t b = tile - E.tile_begin;
    // tile column tc: the last one whose first tile is at or before b (tiles before tile column
    // c: sum_{c'=tc0}^{c-1} (T - c'))
    const int64_t T = (E.n + kSfTile - 1) / kSfTile, tc0 = tab.col0 / kSfTile;
    auto before = [&](int64_t c) { return (c - tc0) * T - (c * (c - 1) - tc0 * (tc0 - 1)) / 2; };
    int64_t lo = tc0, hi = (min(E.n, tab.col1) + kSfTile - 1) / kSfTile - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) / 2;
        if (before(mid) <= b) lo = mid;
        else hi = mid - 1;
    }
    const int64_t tc = lo, tr = tc + (b - before(tc));
    const int lane = threadIdx.x;
    const int64_t row = tr * kSfTile + lane, rowc = min(row, E.n - 1), colc = min(tc * kSfTile + lane, E.n - 1);
    // the table's place of dG = g_col - g_row is linear in both: this lane's row's and column's parts, and
    // the rows' of the elements whose structure factors it fetches
    auto place = [&](int64_t x) {
        const int32_t *g = E.g + 3 * x;
        return (((int64_t)g[0] * tab.ny + g[1]) * tab.nz + g[2]) * tab.nt;
    };
    const int64_t prow = place(rowc);
    const int64_t pcol = place(colc) + (((int64_t)tab.dx * tab.ny + tab.dy) * tab.nz + tab.dz) * tab.nt + tab.type;
    int64_t from[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) from[i] = __shfl_sync(0xffffffffu, prow, lane / 4 + 8 * i) - lane % 4;
    const int kr = kFixed ? E.el[rowc] - 8 - tab.frac - (kItems ? 0 : tab.bits0) : 0;
    const int kcs = kFixed ? E.ers[colc] : 0, kch = kFixed ? E.erh[colc] : 0;
    // the warp's columns of the tile: threadIdx.y, + kRows, ... below cend (those of the lower triangle)
    const int cend = (int)min((int64_t)kSfTile, (tr == tc ? E.n : min(E.n, tc * kSfTile + kSfTile)) - tc * kSfTile);
    const int ntypes = tab.ntypes, nitems = kItems ? tab.nitems : (ntypes + kChunk - 1) / kChunk;
    const int64_t ps = E.pstride, ldp = E.ldp, ldo = E.ldo;
    unsigned char *mem = stages + threadIdx.y * 2 * kStageBytesWarp;
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(mem);
    // the item to be fetched next: column ic, item it; its column's first product
    int ic = threadIdx.y, it = 0;
    uint32_t next = kItems ? tab.item[0] : 0;      // (loaded an item ahead of its use)
    int64_t o = rowc + tab.slot0 * ps + ldp * (tc * kSfTile + ic);
    auto fetch = [&](uint32_t st) {
        if (ic < cend) {
            const int t0 = kItems ? (int)(next & 0xff) : kChunk * it, n = kItems ? (int)((next >> 8) & 0xff) : min(kChunk, ntypes - kChunk * it);
            const int4 *base = sf + __shfl_sync(0xffffffffu, pcol, ic) + t0;
            const uint32_t ds = st + (lane / 4 * kSfPitch + lane % 4) * 16;
            if (lane % 4 < n) {
#pragma unroll
                for (int i = 0; i < 4; ++i) cp_async16(ds + i * (8 * kSfPitch * 16), base - from[i]);
            }
            const uint32_t dp = st + kStageSf + lane * 8;
            int64_t x = o + t0 * ps;
#pragma unroll
            for (int t = 0; t < kChunk; ++t, x += ps)
                if (t < n) {
                    cp_async8(dp + (3 * t) * (kSfTile * 8), static_cast<const int2 *>(E.RS) + x);
                    cp_async8(dp + (3 * t + 1) * (kSfTile * 8), static_cast<const int2 *>(E.RHr) + x);
                    cp_async8(dp + (3 * t + 2) * (kSfTile * 8), static_cast<const int2 *>(E.RHi) + x);
                }
            if (++it == nitems) {
                it = 0;
                ic += kRows;
                o += kRows * ldp;
            }
            if (kItems) next = tab.item[it];
        }
        cp_async_commit();
    };
    int stage = 0;
    uint32_t item = next, item1 = next;            // the item being summed, the one fetched last
    fetch(smem);
    int64_t oo = row + ldo * (tc * kSfTile + threadIdx.y);
#pragma unroll 1
    for (int c = threadIdx.y; c < cend; c += kRows, oo += kRows * ldo) {
        double2 vs = make_double2(0.0, 0.0), vh = make_double2(0.0, 0.0);
        Sums<kFixed> v;
        const int ks = kFixed ? kr + __shfl_sync(0xffffffffu, kcs, c) : 0, kh = kFixed ? kr + __shfl_sync(0xffffffffu, kch, c) : 0;
#pragma unroll 1
        for (int q = 0; q < nitems; ++q) {
            item = item1;
            item1 = next;
            fetch(smem + (stage ^ 1) * kStageBytesWarp);
            cp_async_wait_but_one();
            __syncwarp();
            const int n = kItems ? (int)((item >> 8) & 0xff) : min(kChunk, ntypes - kChunk * q);
            const int4 *w = reinterpret_cast<const int4 *>(mem + stage * kStageBytesWarp) + lane * kSfPitch;
            const int2 *p = reinterpret_cast<const int2 *>(mem + stage * kStageBytesWarp + kStageSf) + lane;
            if (n == kChunk) {
                // (no branch between the types: their multiply-adds interleave; 1.42 and 1.16 ms with one)
#pragma unroll
                for (int t = 0; t < kChunk; ++t) v.add(p[3 * t * kSfTile], p[(3 * t + 1) * kSfTile], p[(3 * t + 2) * kSfTile], w[t]);
            } else {
#pragma unroll 1
                for (int t = 0; t < n; ++t) v.add(p[3 * t * kSfTile], p[(3 * t + 1) * kSfTile], p[(3 * t + 2) * kSfTile], w[t]);
            }
            __syncwarp();
            stage ^= 1;
            if constexpr (kFixed) {
                const int fb = kItems ? (item >> 16) & 0xff : 0;
                if (kItems ? fb != 0 : q % kSumItems == kSumItems - 1 || q + 1 == nitems) {
                    // one power of two for the products of an element and the structure factors of these types
                    const double2 s = make_double2(v.sr.value(ks - fb), v.si.value(ks - fb));
                    const double2 h = make_double2(v.hr.value(kh - fb), v.hi.value(kh - fb));
                    if (kItems ? item >> 24 : q < kSumItems) { vs = s; vh = h; }
                    else { vs = sum2(vs, s); vh = sum2(vh, h); }
                    v = Sums<kFixed>();
                }
            }
        }
        if constexpr (!kFixed) {
            vs = v.s;
            vh = v.h;
        }
        const int64_t col = tc * kSfTile + c;
        if (row >= E.n || col > row) continue;
        const bool x = E.Sx && row < tab.xrow1;
        double2 *so = x ? E.Sx + row + E.ldx * col : E.S + oo, *ho = x ? E.Hx + row + E.ldx * col : E.H + oo;
        if (!first) {
            const double2 s0 = E.Si[row + E.ldi * col], h0 = E.Hi[row + E.ldi * col];
            vs = sum2(vs, s0);
            vh = sum2(vh, h0);
        }
        *so = vs;
        *ho = vh;
    }
}

template <bool kFixed, bool kItems>
cudaError_t combine_launch(const SfTab &t, const void *sf, bool first, int64_t tiles, cudaStream_t st) {
    // 4 columns of a tile at a time from two tiles per SM on, 8 below.  Combine and slicing, us, by 8 and by 4: 235 columns of 2
    // types (36 tiles) 42 and 47, 501 of 2 (136) 43 and 49, 1000 of 4 (528) 70 and 67, 1500 of 4 (1128) 96 and 93, 3000 of 8
    // (4465) 337 and 316
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const bool few = tiles < 2 * (int64_t)nsm;
    const void *kernel = few ? (const void *)sf_combine_kernel<kFixed, 8, kItems> : (const void *)sf_combine_kernel<kFixed, 4, kItems>;
    const int rows = few ? 8 : 4, smem = rows * 2 * kStageBytesWarp;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int4 *f = static_cast<const int4 *>(sf);
    if (few) sf_combine_kernel<kFixed, 8, kItems><<<(unsigned)tiles, dim3(kSfTile, 8), smem, st>>>(t, f, first ? 1 : 0);
    else sf_combine_kernel<kFixed, 4, kItems><<<(unsigned)tiles, dim3(kSfTile, 4), smem, st>>>(t, f, first ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sf_table(const double2 *ex, const double2 *ey, const double2 *ez, const int32_t *order,
                            const int32_t *type_begin, const int32_t *bits, int nt, int nx, int ny, int nz, void *sf,
                            cudaStream_t st) {
    const int64_t n = (int64_t)nx * ny * nz * nt;
    if (n <= 0) return cudaSuccess;
    // atoms per shared-memory chunk: kSfChunk, fewer for a long y extent
    const int chunk = std::min<int>(kSfChunk, kSfSmem / (int)sizeof(double2) / std::max(ny, 1));
    if (nx > 65535 || nt > 65535 || chunk < 1) return cudaErrorInvalidValue;
    const size_t smem = sizeof(double2) * (size_t)chunk * ny;
    sf_table_kernel<<<dim3((unsigned)nx, (unsigned)nt), kSfTabThreads, smem, st>>>(ex, ey, ez, order, type_begin,
                                                                                 bits, nx, ny, nz, chunk, sf);
    return cudaGetLastError();
}

// A set of N atoms has |Re SF| + |Im SF| <= sqrt(2) N, so the sums with f1 stay below 2^63 while the group's atoms are no
// more than 2^(59 - f), f the fixed point, and f1 fits 32 bits while N is less.  A group ends after kSumTypes types, or
// before one of which its fixed point would keep fewer bits than an FP64 number of N's magnitude has: one atom
// takes f = 53, 4000 leave 47.
void sf_fixed_points(const std::vector<int32_t> &atoms, std::vector<int32_t> &order, std::vector<int32_t> &bits,
                     std::vector<int32_t> &group) {
    const int n = (int)atoms.size();
    order.resize(n);
    bits.resize(n);
    group.resize(n);
    for (int i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) { return atoms[a] > atoms[b]; });
    auto log2_up = [](int64_t x) {            // least b with x <= 2^b
        int b = 0;
        while (((int64_t)1 << b) < x) ++b;
        return b;
    };
    for (int a = 0, g = 0; a < n; ++g) {
        int64_t sum = 0;
        int b = a, f = 0;
        for (; b < n && b - a < kSumTypes; ++b) {
            const int64_t N = atoms[order[b]];
            const int fb = std::min(56, 59 - log2_up(std::max<int64_t>(sum + N, atoms[order[a]] + 1)));
            if (b > a && N > 0 && fb < 54 - log2_up(N + 1)) break;
            sum += N;
            f = fb;
        }
        for (; a < b; ++a) {
            bits[a] = f;
            group[a] = g;
        }
    }
}

// The batch's items and the ends of its integer sums, both within the groups.
static void sf_items(SfTab &t) {
    t.nitems = 0;
    t.bits0 = t.bits ? t.bits[t.type] : 0;
    t.listed = false;
    bool first = true;
    for (int a = 0; a < t.ntypes; ++t.nitems) {
        auto same = [&](int x) { return x < t.ntypes && (!t.bits || t.group[t.type + x] == t.group[t.type + a]); };
        int b = a + 1;
        while (b - a < kSfItemTypes && same(b)) ++b;
        t.item[t.nitems] = (uint32_t)a | (uint32_t)(b - a) << 8;
        if (t.bits && !same(b)) {
            t.item[t.nitems] |= (uint32_t)t.bits[t.type + a] << 16 | (first ? 1u << 24 : 0u);
            first = false;
        }
        if (t.bits && (t.bits[t.type + a] != t.bits0 || a != kSfItemTypes * t.nitems ||
                       !same(b) != (t.nitems % kSumItems == kSumItems - 1 || b == t.ntypes)))
            t.listed = true;
        a = b;
    }
}

int64_t sf_tab_tiles(SfTab &tab) {
    int64_t total = 0;
    const int64_t tc0 = tab.col0 / kSfTile;
    for (int k = 0; k < tab.nk; ++k) {
        const int64_t T = (tab.e[k].n + kSfTile - 1) / kSfTile;
        const int64_t tc1 = (std::min(tab.e[k].n, tab.col1) + kSfTile - 1) / kSfTile;   // (col1 may be INT64_MAX)
        tab.e[k].tile_begin = total;
        // tile columns [tc0, tc1), T - c tiles each
        if (tc1 > tc0) total += (tc1 - tc0) * T - (tc1 * (tc1 - 1) - tc0 * (tc0 - 1)) / 2;
    }
    return total;
}

cudaError_t launch_sf_combine(const SfTab &tab, const void *sf, bool first, cudaStream_t st) {
    SfTab t = tab;
    for (int k = 0; k < t.nk; ++k)
        if (!t.e[k].Si) {
            t.e[k].Si = t.e[k].S;
            t.e[k].Hi = t.e[k].H;
            t.e[k].ldi = t.e[k].ldo;
        }
    const int64_t tiles = sf_tab_tiles(t);
    if (tiles <= 0) return cudaSuccess;
    if (tiles > 0x7fffffffLL || t.ntypes < 1 || t.ntypes > kMaxTypes) return cudaErrorInvalidValue;
    sf_items(t);
    if (t.nk < 1 || !t.e[0].el) return combine_launch<false, false>(t, sf, first, tiles, st);
    return t.listed ? combine_launch<true, true>(t, sf, first, tiles, st) : combine_launch<true, false>(t, sf, first, tiles, st);
}

}  // namespace hsdla
