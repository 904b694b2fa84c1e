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
                                                                 const int32_t *__restrict__ type_begin, int nx,
                                                                 int ny, int nz, int chunk, int sfbits,
                                                                 void *__restrict__ sf) {
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
            if (sfbits == 0) {
                static_cast<double2 *>(sf)[o] = acc;
            } else {
                const double s = __longlong_as_double((long long)(1023 + sfbits) << 52);
                const long long re = __double2ll_rn(acc.x * s), im = __double2ll_rn(acc.y * s);
                constexpr int kLow = (1 << 28) - 1;
                static_cast<int4 *>(sf)[o] = make_int4((int)(re >> 28), (int)(re & kLow), (int)(im >> 28), (int)(im & kLow));
            }
        }
    }
}

__device__ __noinline__ double ldexp_call(double v, int k) { return ldexp(v, k); }

// Exact sums of products p f of 64-bit fixed-point products p and 55-bit structure factors f, in four
// 64-bit sums of the limb products: p = p1 2^32 + p0 with p0 in [-2^31, 2^31), f = f1 2^28 + f0 with f0
// in (-2^28, 2^28).  With |p1| < 2^31 and |f1| <= 2^27, kSumTypes types of two terms each overflow none
// of them, so a term is four multiply-adds and no carry.
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
    // 2^50), the rest rounded on the integer pipes (the FP64 pipe, which a conversion instruction
    // uses, issues one warp instruction in 16 cycles)
    __device__ __forceinline__ double value(int k) const {
        const long long m = (a10 >> 4) + (a01 >> 8) + (a00 >> 36);
        const long long top = a11 + (m >> 24);
        const unsigned low = (unsigned)m & 0xffffffu;
        const int s = min(__clzll(top ^ (top >> 63)) - 1, 24);
        const long long x = (top << s) | (long long)(low >> (24 - s));
        // x to nearest even
        const unsigned long long sign = (unsigned long long)x & 0x8000000000000000ull;
        unsigned long long u = x < 0 ? 0ull - (unsigned long long)x : (unsigned long long)x;
        const int lz = __clzll((long long)u);
        u <<= lz & 63;
        const unsigned long long rem = u & 0x7ffull;
        unsigned long long b = ((unsigned long long)(unsigned)(1023 + 62 - lz) << 52) + (u >> 11);   // (hidden bit carries)
        b += (rem > 0x400ull) | ((rem == 0x400ull) & (b & 1ull));
        if (!x) return 0.0;
        k += 60 - s;
        const int E = (int)(b >> 52) + k;
        if (E > 0 && E < 2047) return __longlong_as_double((long long)((b + ((unsigned long long)(unsigned)k << 52)) | sign));
        return ldexp_call(__longlong_as_double((long long)(b | sign)), k);
    }
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
// kFixed: fixed-point products and structure factors, summed exactly in integers.  GB300's FP64 pipe
// (2 multiply-adds per cycle and SM) bounded this kernel at 0.95 of its rate.  8000 columns of 8 types:
// FP64 2.60 ms, integers 1.59 ms (0.57 of the DRAM rate, 24 warps an SM); 2 k-points of 6300 columns and 4
// types: 1.74 and 1.41 ms.
//
// combine_chunk: kNT types from t0 on of one element per lane into its sums.  All loads -- the lanes'
// share of the warp's structure factors and the element's 3 kNT products -- go out before the first
// use: the kernel lives on bytes in flight.  Four types at a time leave registers for 24 warps an SM;
// eight at a time on 16 warps took 1.66 and 1.60 ms.
template <bool kFixed>
struct Sums {
    double2 s = make_double2(0.0, 0.0), h = make_double2(0.0, 0.0);
};
template <>
struct Sums<true> {
    LimbSum sr, si, hr, hi;
};
template <bool kFixed, int kNT>
__device__ __forceinline__ void combine_chunk(Sums<kFixed> &v, const SfEntry &E, const int4 *__restrict__ sf, int64_t idx,
                                              int64_t off, int t0, int4 (*st)[kSumTypes]) {
    const int lane = threadIdx.x;
    const int64_t ps = E.pstride;
    int4 g[kNT];
    int2 a[kNT], c[kNT], d[kNT];
#pragma unroll
    for (int i = 0; i < kNT; ++i) {
        const int w = lane + 32 * i;
        g[i] = sf[__shfl_sync(0xffffffffu, idx, w / kNT) + t0 + w % kNT];
    }
    const int2 *pa = static_cast<const int2 *>(E.RS) + off + t0 * ps;
    const int2 *pc = static_cast<const int2 *>(E.RHr) + off + t0 * ps, *pd = static_cast<const int2 *>(E.RHi) + off + t0 * ps;
#pragma unroll
    for (int t = 0; t < kNT; ++t) {
        a[t] = __ldcs(pa + t * ps);
        c[t] = __ldcs(pc + t * ps);
        d[t] = __ldcs(pd + t * ps);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kNT; ++i) {
        const int w = lane + 32 * i, e = w / kNT, t = w % kNT;
        st[e][(t + e) % kSumTypes] = g[i];     // (rotated: rows of 128 bytes would share banks)
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kNT; ++t) {
        const int4 w = st[lane][(t + lane) % kSumTypes];
        if constexpr (kFixed) {
            const Limbs x(a[t]), y(c[t]), z(d[t]);
            v.sr.add(x, w.x, w.y);
            v.si.add(x, w.z, w.w);
            v.hr.add(y, w.x, w.y);
            v.hr.add(z, -w.z, -w.w);
            v.hi.add(z, w.x, w.y);
            v.hi.add(y, w.z, w.w);
        } else {
            auto dbl = [](int lo, int hi) { return __hiloint2double(hi, lo); };
            const double fr = dbl(w.x, w.y), fi = dbl(w.z, w.w), x = dbl(a[t].x, a[t].y), y = dbl(c[t].x, c[t].y), z = dbl(d[t].x, d[t].y);
            v.s.x = fma(fr, x, v.s.x);
            v.s.y = fma(fi, x, v.s.y);
            v.h.x = fma(fr, y, fma(-fi, z, v.h.x));
            v.h.y = fma(fr, z, fma(fi, y, v.h.y));
        }
    }
}

template <bool kFixed, int kRows>
__global__ void __launch_bounds__(kSfTile *kRows, 768 / (kSfTile * kRows)) sf_combine_kernel(const __grid_constant__ SfTab tab,
                                                                                     const void *__restrict__ sf, int first) {
    __shared__ int4 stage[kRows][kSfTile][kSumTypes];
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
    const int64_t row = tr * kSfTile + lane, rowc = min(row, E.n - 1);
    const int32_t *gr = E.g + 3 * rowc;
    const int gr0 = gr[0], gr1 = gr[1], gr2 = gr[2];
    int4 (*st)[kSumTypes] = stage[threadIdx.y];
#pragma unroll 1
    for (int q = 0; q < kSfTile; q += kRows) {
        const int64_t col = tc * kSfTile + threadIdx.y + q;
        if (col >= E.n || col > tr * kSfTile + kSfTile - 1) break;      // (warp-uniform)
        const bool live = row < E.n && col <= row;
        const int32_t *gc = E.g + 3 * col;
        const int64_t idx = (((int64_t)(gc[0] - gr0 + tab.dx) * tab.ny + (gc[1] - gr1 + tab.dy)) * tab.nz +
                             (gc[2] - gr2 + tab.dz)) * tab.nt + tab.type;
        const int64_t off = rowc + E.ldp * col + tab.slot0 * E.pstride;
        double2 vs = make_double2(0.0, 0.0), vh = make_double2(0.0, 0.0);
        for (int t0 = 0; t0 < tab.ntypes; t0 += kSumTypes) {
            const int nt = min(tab.ntypes - t0, kSumTypes);
            const int4 *f = static_cast<const int4 *>(sf);
            Sums<kFixed> v;
            if constexpr (!kFixed) { v.s = vs; v.h = vh; }
            int t = t0;
            if (nt == kSumTypes) { combine_chunk<kFixed, 4>(v, E, f, idx, off, t, st); t += 4; }
            if (nt >= 4) { combine_chunk<kFixed, 4>(v, E, f, idx, off, t, st); t += 4; }
            if (nt & 2) { combine_chunk<kFixed, 2>(v, E, f, idx, off, t, st); t += 2; }
            if (nt & 1) combine_chunk<kFixed, 1>(v, E, f, idx, off, t, st);
            if constexpr (kFixed) {
                // one power of two for every type's products of an element
                const int k0 = E.el[rowc] - 8 - tab.frac - tab.sfbits, ks = k0 + E.ers[col], kh = k0 + E.erh[col];
                const double2 s = make_double2(v.sr.value(ks), v.si.value(ks)), h = make_double2(v.hr.value(kh), v.hi.value(kh));
                if (t0 == 0) { vs = s; vh = h; }
                else { vs.x += s.x; vs.y += s.y; vh.x += h.x; vh.y += h.y; }
            } else {
                vs = v.s;
                vh = v.h;
            }
        }
        if (!live) continue;
        const bool x = E.Sx && row < tab.xrow1;
        double2 *so = x ? E.Sx + row + E.ldx * col : E.S + row + E.ldo * col;
        double2 *ho = x ? E.Hx + row + E.ldx * col : E.H + row + E.ldo * col;
        if (!first) {
            const double2 s0 = E.Si[row + E.ldi * col], h0 = E.Hi[row + E.ldi * col];
            vs.x += s0.x; vs.y += s0.y;
            vh.x += h0.x; vh.y += h0.y;
        }
        *so = vs;
        *ho = vh;
    }
}

template <bool kFixed>
void combine_launch(const SfTab &t, const void *sf, bool first, int64_t tiles, cudaStream_t st) {
    // 4 columns of a tile at a time where there are tiles enough, 8 where not
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (tiles < 8 * (int64_t)nsm) sf_combine_kernel<kFixed, 8><<<(unsigned)tiles, dim3(kSfTile, 8), 0, st>>>(t, sf, first ? 1 : 0);
    else sf_combine_kernel<kFixed, 4><<<(unsigned)tiles, dim3(kSfTile, 4), 0, st>>>(t, sf, first ? 1 : 0);
}

}  // namespace

cudaError_t launch_sf_table(const double2 *ex, const double2 *ey, const double2 *ez, const int32_t *order,
                            const int32_t *type_begin, int nt, int nx, int ny, int nz, int sfbits, void *sf,
                            cudaStream_t st) {
    const int64_t n = (int64_t)nx * ny * nz * nt;
    if (n <= 0) return cudaSuccess;
    // atoms per shared-memory chunk: kSfChunk, fewer for a long y extent
    const int chunk = std::min<int>(kSfChunk, kSfSmem / (int)sizeof(double2) / std::max(ny, 1));
    if (nx > 65535 || nt > 65535 || chunk < 1) return cudaErrorInvalidValue;
    const size_t smem = sizeof(double2) * (size_t)chunk * ny;
    sf_table_kernel<<<dim3((unsigned)nx, (unsigned)nt), kSfTabThreads, smem, st>>>(ex, ey, ez, order, type_begin, nx,
                                                                                 ny, nz, chunk, sfbits, sf);
    return cudaGetLastError();
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
    if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
    if (t.nk > 0 && t.e[0].el) combine_launch<true>(t, sf, first, tiles, st);
    else combine_launch<false>(t, sf, first, tiles, st);
    return cudaGetLastError();
}

}  // namespace hsdla
