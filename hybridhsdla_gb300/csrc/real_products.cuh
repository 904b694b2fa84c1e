// Real digit products of the structure-factor form (see real_products.cu).
#pragma once

#include <cuda.h>

#include <vector>

#include "common.cuh"

namespace hsdla {

constexpr int kRealTileM = 256;      // output rows of a tile (a CTA pair: 128 each)
constexpr int kRealTileN = 128;      // output columns
constexpr int kRealKBlock = 64;      // contraction bytes (e4m3 digits) per operand plane and chunk
constexpr int kRealBRows = kRealTileN / 2;   // right-operand rows a CTA stages
constexpr int kRealMaxSlices = 12;

// One real product sum_k left[k, r] right[k, c] of digit operands as 64-bit fixed-point numbers: the
// value of element (r, c) is out[r + ldo c] 2^(el[r] + er[c] - 8 - frac) (RealBands::frac).  Plane i
// (1-based digit) of the left operand holds its rows at (i - 1) lplane + lrow0; of the right operand
// at (rstep (j - 1) + rpart) rplane + rrow0.
struct RealJob {
    int32_t rmap;              // right tensor map (0 or 1)
    int32_t lower;             // 1: only elements with row >= col
    int32_t ksteps_last;       // K steps of 32 bytes in the last chunk (1-2)
    int32_t rstep, rpart;
    int32_t reserved;
    int64_t lplane, rplane, lrow0, rrow0;
    int64_t lk0, rk0;          // first contraction byte (multiple of 64)
    int64_t nkb;               // chunks of 64 contraction bytes
    int64_t m, n;
    long long *out;
    int64_t ldo;
};

// The order in which a chunk's digit pairs (i, j), i + j = t, run: bands of one or two adjacent
// diagonals ending at T, ascending, each summed in one FP32 accumulator x (diagonal T - 1 times 32,
// diagonal T) that enters the fixed-point sums as
//     sum += bits(x f) mul        bits(y): those of the FP32 number y + 1.5 2^23 (an integer plus a
//                                 constant, |y| < 2^22)
// (kFoldHigh: into the high word only); the constants are taken off at the start (bias per chunk).
enum { kFoldHigh = 0, kFoldLow = 1 };
struct RealBands {
    int32_t s;                         // digits per operand
    int32_t frac;                      // fraction bits of the fixed-point sums
    int32_t halves;                    // 2: the bands alternate between TMEM buffers, 1: they wait for each other
    int32_t n;                         // bands
    unsigned long long bias;
    int8_t T[kRealMaxSlices];          // last diagonal of each band
    int8_t w[kRealMaxSlices];          // its diagonals (1-2)
    int8_t fold[kRealMaxSlices];
    float f[kRealMaxSlices];
    uint32_t mul[kRealMaxSlices];
};
// Bands of at most `width` diagonals for s digits and a contraction over kvalid digits.
RealBands real_bands(int s, int width, int halves, int64_t kvalid);
int64_t real_job_tiles(const RealJob &j);
// Tile list (job, tile row, tile column) of `jobs`: consecutive lower jobs of equal size (the
// products of one k-point) interleaved per tile in super-blocks, other jobs one after another.
void real_schedule(const std::vector<RealJob> &jobs, std::vector<int4> &list);
// Left map: boxes of 64 bytes x 128 rows; right maps: 64 bytes x 64 rows (64-byte swizzle).
cudaError_t launch_real_products(const CUtensorMap &left, const CUtensorMap &right0, const CUtensorMap &right1,
                                 const RealJob *d_jobs, const int4 *d_list, int64_t tiles, const RealBands &bands,
                                 int *d_err, cudaStream_t st);

// Digit planes of real columns.  Column g of an entry holds `blocks` contraction blocks; block b's
// part p (parts: the real and imaginary rows of a complex operand) is source[b bstride + p pstride +
// r], r < rpb, and lands at contraction bytes [b bpad, b bpad + rpb) of planes parts (i - 1) + p.  One
// exponent per column over every block and part.  The source is FP64, or (fixed) a product's
// fixed-point numbers with the row exponents el (index as the source's rows) and column exponents.
struct RealSliceEntry {
    const void *Z;
    int64_t ncols;
    int64_t row0;              // first plane row
};
struct RealSliceTab {
    int nk = 0, s = 0, parts = 1;
    int64_t ldz = 0, blocks = 0, rpb = 0, bstride = 0, pstride = 0, bpad = 0;
    uint8_t *digits = nullptr;
    int64_t plane_rows = 0, pitch = 0;
    int32_t *expo = nullptr;
    int frac = 0;                      // fixed-point source: its fraction bits (0: an FP64 source),
    const int32_t *el = nullptr;       // row exponents (those of block b from set_type[b] bstride on),
    const int32_t *set_type = nullptr;
    const int32_t *er = nullptr;       // and the column exponents (per plane row)
    // a second operand of the same source with row weights v2[b rpb + r] (parts = 1)
    const double *v2 = nullptr;
    uint8_t *digits2 = nullptr;
    int32_t *expo2 = nullptr;
    RealSliceEntry e[kMaxGroup];
};
cudaError_t launch_real_slice(const RealSliceTab &t, cudaStream_t st);

}  // namespace hsdla
