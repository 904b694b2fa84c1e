// Shared definitions of the sm_103a H/S generation library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "../../include/hsdla.h"

namespace hsdla {

// Row r of element x of a triangle stored row by row (r (r + 1) / 2 <= x), x < 2^31.  The estimate is
// FP32: a double square root takes GB300's FP64 pipe ~1000 cycles per block of 256 threads.
__device__ __forceinline__ int64_t triangle_row(int64_t x) {
    int64_t r = (int64_t)((sqrtf(8.0f * (float)x + 1.0f) - 1.0f) * 0.5f);
    while (r * (r + 1) / 2 > x) --r;
    while ((r + 1) * (r + 2) / 2 <= x) ++r;
    return r;
}


constexpr int kMaxLmax = 14;                 // (14+1)^2 = 225 lm per atom
constexpr int kMaxL = (kMaxLmax + 1) * (kMaxLmax + 1);
constexpr int kMaxTypes = 64;
constexpr int kMaxSets = 4096;               // row sets of the structure-factor form
constexpr double kPi = 3.14159265358979323846;

// Device error word: kernels with bounded waits write a code here instead of trapping.
enum DeviceError : int {
    kDevOk = 0,
    kDevTimeout = 1,
    kDevBadInput = 2,
};

// ------------------------------------------------------------------ system
// Device-resident per-run data (uploaded once per plan).
struct DevSystem {
    int num_atoms, num_types, max_lmax, L;
    double vol_prefac;          // 4 pi / sqrt(Omega)
    double bmat[9];             // row-major rows b_i
    const int32_t *atom_type;   // [a]
    const double *atom_pos;     // [a][3]
    const double *atom_rotmat;  // [a][9] or nullptr
    const double *type_rmt;     // [t]
    const int32_t *type_lmax;   // [t]
    // per (type, l), index t*(max_lmax+1)+l
    const double *u, *u_dr, *dE_u, *dE_u_dr;
    const double *inv_w;        // 1 / (udot u' - u udot')
    const double *ynorm;        // [L] Y_lm normalisation (ylm4.f:111-137)
    // The row sets of the structure-factor form: the types, or (type, rotation) classes, whose atoms
    // share the rotation.  Set q is of type set_type[q]; the sets of rotation rho (row-major mrot bmat
    // at rots[9 rho]) are [rot_begin[rho], rot_begin[rho + 1]).  num_rots = 0: every set's rows use
    // R = bmat (no atom carries its own rotation).
    int num_sets, num_rots;
    const int32_t *set_type;    // [num_sets]
    const double *rots;         // [num_rots][9]
    const int32_t *rot_begin;   // [num_rots + 1]
    // normalised Legendre recursion, [2][max_lmax + 1 (m)][max_lmax + 1 (l)]: P_l^m = a_lm (cos P_{l-1}^m -
    // b_lm P_{l-2}^m), with a_mm the factor of sin^m in P_m^m
    const double *legendre;
};

// Shared memory of the rows kernel (construct_rows_kernel) for L lm, lmax max_lmax and nt types; the
// kernel runs only where it fits (160 KB).
constexpr int kRowCols = 16;    // G columns of a CTA
constexpr int kRowRots = 16;    // rotations of a CTA at most
inline size_t rows_kernel_smem(int L, int max_lmax, int nt) {
    const int nl = max_lmax + 1, tnl = nt * nl;
    size_t b = sizeof(double) * (kRowCols * L + 2 * kRowCols * tnl + tnl + 4 * kRowCols + 4 * kRowCols * kRowRots) +
               sizeof(double *) * kRowCols + L + 16;
    return (b + 15) & ~size_t(15);
}
constexpr size_t kRowsKernelSmemMax = 160 * 1024;

struct DevKpoint {
    double k[3];
    int64_t n_g;
    const int32_t *g;           // [n_g][3]
};

// A group of k-points handled by one launch per stage (passed by value as a kernel parameter).
constexpr int kMaxGroup = 64;
struct KEntry {
    DevKpoint kp;
    double2 *C;                 // (2 L a) x n_g, ld KTable::ldc
    double2 *M;                 // (2 L nt) x n_g, ld KTable::ldm, or nullptr
    const double2 *Z;           // per-type product, ld KTable::ldm (phase expansion input)
    double2 *X;                 // per-atom output, ld KTable::ldc (phase expansion output)
    int64_t col_begin;          // first global column of this k-point
    double *R;                  // real per-type rows (2 L nt) x n_g, ld KTable::ldm, or nullptr: row
                                // (l, m >= 0) of M's real part, row (l, -m) of row (l, m)'s imaginary part
};
struct KTable {
    int nk = 0;
    int a0 = 0, a1 = -1;        // atom range of the phase expansion (a1 < 0: every atom)
    int64_t ldc = 0, ldm = 0;
    int64_t total_cols = 0;
    KEntry e[kMaxGroup];
};

// dst[2L u + i] = src[L u + i] for u < units, i < L: rows of A (or, dst + L, of B) into [A; B].
cudaError_t launch_stack_rows(const double2 *src, int L, int64_t units, double2 *dst, cudaStream_t st);

// ----------------------------------------------------------- kernels (host)
// (a) for every k-point of a table in one launch (C always; M when the entries give it)
cudaError_t launch_construct_ab_multi(const DevSystem &sys, const KTable &tab, cudaStream_t st);
// X = phase Z for every k-point of a table in one launch
cudaError_t launch_apply_phase_multi(const DevSystem &sys, const KTable &tab, cudaStream_t st);
// (a) matching tensors of one k-point into C: (2 L a) x n_g column-major, per-atom [A_a; B_a]
// Optionally also the phase-free per-type rows M ((2 L nt) x n_g, ld ldm) when no atom carries
// its own rotation (M_t = C_a e^{-i 2pi K.tau_a} for every atom a of type t).
cudaError_t launch_construct_ab(const DevSystem &sys, const DevKpoint &kp, double2 *C, int64_t ldc,
                                cudaStream_t st, double2 *M = nullptr, int64_t ldm = 0);
// The Hermitian 2L x 2L blocks [[T_AA, T_AB], [T_AB^H, T_BB]] of every type (column-major, ld 2L,
// 4 L^2 apart) into tf, from the caller's lower triangles of T_AA and T_BB and all of T_AB (each
// nt x L x L, column-major per type), with the input checks per type in stats[5 t .. 5 t + 4]
// (zeroed by the caller): bit q of [0] set when block q (0 AA, 1 AB, 2 BB) holds a non-finite
// value; [1], [2] = max |T|^2 and max |T - T^H|^2 over T_AA's lower triangle, [3], [4] the same
// for T_BB (doubles as bit patterns).  tf NULL: the checks alone.
cudaError_t launch_tfull(const double2 *aa, const double2 *ab, const double2 *bb, int nt, int L, double2 *tf,
                         unsigned long long *stats, cudaStream_t st);
// The real form of the T blocks (see real_products.cu): tr holds per type 4L columns of 2L values,
// column r the row r of Re T', column 2L + r the row r of Im T', T' = V^H T V with launch_tfull's T.
cudaError_t launch_treal(const double2 *aa, const double2 *ab, const double2 *bb, int nt, int L, double *tr,
                         cudaStream_t st);
// Per-atom structure phases along each axis, ph[o] = e^{i 2pi (i - half_c) pos[3 j + c]} with o
// running over c, then atom j, then i in [0, ext_c).
cudaError_t launch_sf_phases(const double *pos, int na, const int *half, const int *ext, double2 *ph, cudaStream_t st);
// X[2L a + r, g] = e^{i 2pi (k+g).tau_a} Z[2L t(a) + r, g]
cudaError_t launch_apply_phase(const DevSystem &sys, const DevKpoint &kp, const double2 *Z, int64_t ldz,
                               double2 *X, int64_t ldx, cudaStream_t st);

// FP64 tiled contraction OUT = P^H diag(w) Q over a batch of jobs (kernels (b) and (c) in FP64).
struct Fp64Job {
    const double2 *P; int64_t ldp;   // k x m
    const double2 *Q; int64_t ldq;   // k x n
    const double *w;                 // k weights or nullptr
    double2 *out; int64_t ldo;       // m x n
    int64_t m, n, k;
    int32_t lower;                   // 1: only elements with row >= col (m == n required)
    int32_t edge;                    // tile edge, 32 or 16 (fp64_edge)
    int32_t tiles_n;                 // tile columns of this job
    int64_t tile_begin;              // first global tile index of this job
};
// The edge of jobs that come to `tiles32` tiles of edge 32.
int fp64_edge(int64_t tiles32);
// Numbers the jobs' tiles for one launch and returns their count.
int64_t fp64_assign(Fp64Job *jobs, int num_jobs);
cudaError_t launch_fp64_jobs(const Fp64Job *d_jobs, int num_jobs, int64_t total_tiles, cudaStream_t st);

// Real FP64 contraction out = P^T Q over a batch of jobs (the structure-factor form's real rows, see
// real_products.cu): P k x m, Q k x n, out m x n, column-major.
struct Fp64RealJob {
    const double *P; int64_t ldp;
    const double *Q; int64_t ldq;
    const double *w;                 // k weights, with
    double *wq;                      // diag(w) Q, also written (ld ldq; m >= k, not lower), or nullptr
    double *out; int64_t ldo;
    int64_t m, n, k;
    int32_t lower;                   // 1: only elements with row >= col (m == n required)
    int32_t parts;                   // 1: the contraction summed in four parts (products that alone are few tiles)
    int32_t edge;                    // tile edge, 32, or 16 where a launch of such products has few tiles as well
    int32_t tiles_n;                 // tile columns of this job
    int64_t tile_begin;              // first global tile index of this job
};
// Chooses the jobs' edges and numbers their tiles for one launch.
int64_t fp64_real_assign(Fp64RealJob *jobs, int num_jobs);
cudaError_t launch_fp64_real(const Fp64RealJob *d_jobs, int num_jobs, int64_t tiles, cudaStream_t st);

// ---- structure-factor form (atoms sharing their type's rotation)
// One k-point of a combine: real per-type products (lower triangles, ld ldp) into the outputs
// S, H (ld ldo); g the k-point's G-vectors [n][3] on the device.
struct SfEntry {
    // per-type products S, Re H and Im H, type slot b at + b pstride: FP64, or (el set) fixed-point
    // numbers, element (r, c) times 2^(el[r] + er[c] - 8 - frac) with er = ers for S and erh for H
    const void *RS = nullptr, *RHr = nullptr, *RHi = nullptr;
    const int32_t *el = nullptr, *ers = nullptr, *erh = nullptr;
    double2 *S = nullptr, *H = nullptr;
    // what a combine that is not the first adds to (NULL: S and H themselves, ldo)
    const double2 *Si = nullptr, *Hi = nullptr;
    int64_t ldp = 0, ldo = 0, n = 0, pstride = 0, ldi = 0;
    const int32_t *g = nullptr;
    int64_t tile_begin = 0;
    // where rows < SfTab::xrow1 go instead of S and H (NULL: nowhere else), leading dimension ldx
    double2 *Sx = nullptr, *Hx = nullptr;
    int64_t ldx = 0;
};
constexpr int kSfItemTypes = 4;                   // types of an item, the unit of a combine's work
struct SfTab {
    int nk = 0, type = 0, ntypes = 1;             // the batch: types [type, type + ntypes) in slots
    int slot0 = 0;                                // slot0, slot0 + 1, ...
    int64_t col0 = 0, col1 = INT64_MAX;           // the columns combined (of every entry)
    int frac = 0;                                 // fixed-point products: their fraction bits
    int64_t xrow1 = 0;                            // rows below it go to the entries' Sx, Hx when set

    int dx = 0, dy = 0, dz = 0, ny = 0, nz = 0;   // box offsets (half widths) and extents
    int64_t box = 0;                              // entries
    int nt = 1;                                   // row sets of the structure-factor table
    // (the entries lie within reach of an immediate offset: behind what follows the combine took 2.5% longer)
    SfEntry e[kMaxGroup];
    const int32_t *bits = nullptr;                // host: its fixed points (launch_sf_table) [nt], NULL: FP64,
    const int32_t *group = nullptr;               // and the groups that are summed in integers
    // set by launch_sf_combine: the batch's items, each at most kSfItemTypes types of one group: its first
    // type, bits 8-15 their number, and where the integer sums end with it bits 16-23 the fixed point, bit 24
    // for the first such item
    int nitems = 0;
    uint32_t item[kMaxTypes];
    int bits0 = 0;                                // the first type's fixed point
    bool listed = false;                          // whether the items are other than four types each, in sums of two
};
// SF_t(dG) = sum_{a of type t} e^{i 2pi dG.tau_a} over the box of G-vector differences, from
// per-atom factors ex[a][dGx + dx] = e^{i 2pi dGx tau_a,x} (and y, z); atoms listed by type.  The table
// holds entry dG's types together (type fastest), 16 bytes each: FP64 (re, im), or with bits (device) each
// part as the limbs {f >> 28, f & (2^28 - 1)} of f = rint(part 2^bits[t]), |f| < 2^59.
cudaError_t launch_sf_table(const double2 *ex, const double2 *ey, const double2 *ez, const int32_t *order,
                            const int32_t *type_begin, const int32_t *bits, int nt, int nx, int ny, int nz, void *sf,
                            cudaStream_t st);
// The order in which row sets of atoms[q] atoms are combined, and by their place in it the groups of sets whose
// terms are summed in integers and the groups' fixed points.
void sf_fixed_points(const std::vector<int32_t> &atoms, std::vector<int32_t> &order, std::vector<int32_t> &bits,
                     std::vector<int32_t> &group);
// S (+)= sum_b SF_{type+b} (.) S_b and H (+)= sum_b SF_{type+b} (.) H_b over the lower triangles
// of every entry, b over the batch's type slots, in columns [tab.col0, tab.col1) (multiples of 32
// but for the end); rows below tab.xrow1 into Sx, Hx instead for entries that give them.
cudaError_t launch_sf_combine(const SfTab &tab, const void *sf, bool first, cudaStream_t st);

// BLAS-shaped plugin (blas_plugin.cu).  Operand in the 'C' layout: dst rows [r0, r0 + k) of every
// column c < n (ld ldd) = s * src[r, c] (src k x n, transpose false) or s * conj(src[c, r]) (src
// n x k, transpose true).
cudaError_t launch_plugin_operand(const double2 *src, int64_t lds, bool transpose, int64_t k, int64_t n, double2 s,
                                  double2 *dst, int64_t ldd, int64_t r0, cudaStream_t st);
// On C's uplo triangle: C = a T(R) + beta C, T(R)[i, j] = R[i, j] (lower) or conj(R[j, i]) (upper),
// R's lower triangle read (R may be NULL: C = beta C); herm: real diagonal.
cudaError_t launch_plugin_diagonal(double2 *C, int64_t ldc, int64_t n, cudaStream_t st);
cudaError_t launch_plugin_epilogue(const double2 *R, int64_t ldr, double2 *C, int64_t ldc, int64_t n, double2 a,
                                   double beta, bool upper, bool herm, cudaStream_t st);

// Fleur's packed lower triangle (row by row) of a column-major n x n matrix (device buffers).
cudaError_t launch_pack_lower(const double2 *M, int64_t ld, int64_t n, double2 *P, cudaStream_t st);

}  // namespace hsdla
