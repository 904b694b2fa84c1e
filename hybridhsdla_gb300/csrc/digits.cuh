// Base-32 digits in e4m3, as the slicing kernels write them.
#pragma once

#include <cuda_fp8.h>
#include <stdint.h>

namespace hsdla {
namespace {

// The s digits of kVec (8 or 4) values X + B (B = 16 in every lower digit) to planes `step` apart (dst: the
// first digit's).  The lower digits are 5-bit fields: 15 bits of two values side by side, a field of each
// at a time into FP16 (1024 + field, less 1040) and both to e4m3 in one conversion (a field and a table
// read at a time took 237 us where this takes 207, the fixed-point columns of the 8000-column workload).
__device__ __forceinline__ uint32_t e4m3_pair(uint32_t h) {          // two FP16 numbers, low half first
    __half2_raw r;
    r.x = (unsigned short)h;
    r.y = (unsigned short)(h >> 16);
    return __nv_cvt_halfraw2_to_fp8x2(r, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ uint32_t sub_1040(uint32_t h) {
    uint32_t d;
    asm("sub.f16x2 %0, %1, %2;\n" : "=r"(d) : "r"(h), "r"(0x64106410u));
    return d;
}
template <int kVec>
__device__ __forceinline__ void put_digits(uint8_t *p, const uint32_t (&d)[kVec / 2]) {
    const uint32_t w0 = __byte_perm(d[0], d[1], 0x5410);
    if constexpr (kVec == 8) *reinterpret_cast<uint2 *>(p) = make_uint2(w0, __byte_perm(d[2], d[3], 0x5410));
    else *reinterpret_cast<uint32_t *>(p) = w0;
}
template <int kVec>
__device__ __forceinline__ void write_digits(const long long (&u)[kVec], int s, uint8_t *dst, int64_t step) {
    // the first digit: in [-16, 16] for a finite column (clamped for any)
    {
        uint32_t w[kVec / 2];
        const int sh = 5 * (s - 1);
#pragma unroll
        for (int v = 0; v < kVec; v += 2) {
            const int d0 = min(max((int)(u[v] >> sh), -16), 16), d1 = min(max((int)(u[v + 1] >> sh), -16), 16);
            w[v / 2] = e4m3_pair(sub_1040(__byte_perm(d0 + 0x6410, d1 + 0x6410, 0x5410)));
        }
        put_digits<kVec>(dst, w);
    }
    uint8_t *p = dst + (int64_t)(s - 1) * step;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (3 * c >= s - 1) break;
        uint32_t w[kVec / 2];
#pragma unroll
        for (int v = 0; v < kVec; v += 2)
            w[v / 2] = __byte_perm((uint32_t)(u[v] >> (15 * c)), (uint32_t)(u[v + 1] >> (15 * c)), 0x5410);
#pragma unroll
        for (int f = 0; f < 3; ++f, p -= step) {
            if (3 * c + f >= s - 1) break;
            uint32_t d[kVec / 2];
#pragma unroll
            for (int v = 0; v < kVec / 2; ++v) d[v] = e4m3_pair(sub_1040(((w[v] >> (5 * f)) & 0x001f001fu) | 0x64006400u));
            put_digits<kVec>(p, d);
        }
    }
}

}  // namespace
}  // namespace hsdla
