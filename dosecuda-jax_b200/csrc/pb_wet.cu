// pb_wet.cu -- HU -> RLSP conversion and the water-equivalent-thickness
// (WET) pass: ray trace toward the source and lateral smoothing.
//
//   HU -> RLSP            DoseCUDA/plan_impt.py:158-168 (numpy.interp)
//   ray trace             DoseCUDA/dose_kernels/CudaClasses.cu:180-228
//   smoothing             DoseCUDA/dose_kernels/IMPTClasses.cu:139-202
//
// Layout: every volume is x-fastest.  The ray trace takes one voxel per thread
// in bricks of 8x4x4, so that a warp covers an 8x4 patch whose rays have similar
// lengths whatever the beam direction, and each row of 8 voxels is one
// 32-byte sector; the smoothing takes runs of consecutive voxels.  Several beams
// share one launch.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <type_traits>

#include "pb_internal.h"

namespace pb {

// ------------------------------------------------------------------ HU->RLSP

struct HuCurve {
    double x[PB_MAX_CURVE];
    double y[PB_MAX_CURVE];
    double slope[PB_MAX_CURVE];
    int n;
};

// numpy.interp: left of the first point -> first value, right of the last
// -> last value, on a knot -> the knot's value, else slope*(x-x_j)+y_j in
// FP64 with no contraction; the result is rounded to FP32 as np.array(...,
// dtype=single) does.
__global__ void k_rlsp(const float *__restrict__ hu, int64_t n,
                       const __grid_constant__ HuCurve c,
                       float *__restrict__ out)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        const double x = (double)hu[q];
        double r;
        if (x != x) {
            r = x;
        } else if (x < c.x[0]) {
            r = c.y[0];
        } else if (x > c.x[c.n - 1]) {
            r = c.y[c.n - 1];
        } else {
            int j = 0;
            while (j + 1 < c.n && c.x[j + 1] <= x) ++j;
            if (j == c.n - 1 || c.x[j] == x) {
                r = c.y[j];
            } else {
                r = __dadd_rn(__dmul_rn(c.slope[j], __dsub_rn(x, c.x[j])), c.y[j]);
            }
        }
        out[q] = __double2float_rn(r);
    }
}

PbStatus launch_rlsp(const float *hu, int64_t n, const double *xh,
                     const double *yh, int m, float *out, cudaStream_t st)
{
    HuCurve c;
    c.n = m;
    for (int i = 0; i < m; ++i) {
        c.x[i] = xh[i];
        c.y[i] = yh[i];
    }
    for (int i = 0; i + 1 < m; ++i) c.slope[i] = (yh[i + 1] - yh[i]) / (xh[i + 1] - xh[i]);
    c.slope[m - 1] = 0.0;
    if (n == 0) return PB_OK;
    int blocks = (int)((n + 255) / 256);
    const int cap = 148 * 16;
    if (blocks > cap) blocks = cap;
    k_rlsp<<<blocks, 256, 0, st>>>(hu, n, c, out);
    return check_launch("k_rlsp");
}

// ----------------------------------------------------------------- ray trace

// Trilinear sample at voxel-index coordinates with 0 outside the grid
// (the reference samples a border-0 texture with linear filtering).
__device__ __forceinline__ float trilinear(const float *__restrict__ rho,
                                           int nx, int ny, int nz, float xb,
                                           float yb, float zb)
{
    const float fx = floorf(xb), fy = floorf(yb), fz = floorf(zb);
    const int i0 = (int)fx, j0 = (int)fy, k0 = (int)fz;
    const float ax = xb - fx, ay = yb - fy, az = zb - fz;
    const int64_t sy = nx, sz = (int64_t)nx * ny;
    float c000, c100, c010, c110, c001, c101, c011, c111;
    if (i0 >= 0 && j0 >= 0 && k0 >= 0 && i0 + 1 < nx && j0 + 1 < ny && k0 + 1 < nz) {
        const float *p = rho + i0 + sy * j0 + sz * k0;
        c000 = __ldg(p);
        c100 = __ldg(p + 1);
        c010 = __ldg(p + sy);
        c110 = __ldg(p + sy + 1);
        c001 = __ldg(p + sz);
        c101 = __ldg(p + sz + 1);
        c011 = __ldg(p + sz + sy);
        c111 = __ldg(p + sz + sy + 1);
    } else {
        const bool xi0 = i0 >= 0 && i0 < nx, xi1 = i0 + 1 >= 0 && i0 + 1 < nx;
        const bool yj0 = j0 >= 0 && j0 < ny, yj1 = j0 + 1 >= 0 && j0 + 1 < ny;
        const bool zk0 = k0 >= 0 && k0 < nz, zk1 = k0 + 1 >= 0 && k0 + 1 < nz;
        auto at = [&](bool ok, int i, int j, int k) -> float {
            return ok ? __ldg(rho + i + sy * j + sz * k) : 0.0f;
        };
        c000 = at(xi0 && yj0 && zk0, i0, j0, k0);
        c100 = at(xi1 && yj0 && zk0, i0 + 1, j0, k0);
        c010 = at(xi0 && yj1 && zk0, i0, j0 + 1, k0);
        c110 = at(xi1 && yj1 && zk0, i0 + 1, j0 + 1, k0);
        c001 = at(xi0 && yj0 && zk1, i0, j0, k0 + 1);
        c101 = at(xi1 && yj0 && zk1, i0 + 1, j0, k0 + 1);
        c011 = at(xi0 && yj1 && zk1, i0, j0 + 1, k0 + 1);
        c111 = at(xi1 && yj1 && zk1, i0 + 1, j0 + 1, k0 + 1);
    }
    const float c00 = fmaf(ax, c100 - c000, c000);
    const float c10 = fmaf(ax, c110 - c010, c010);
    const float c01 = fmaf(ax, c101 - c001, c001);
    const float c11 = fmaf(ax, c111 - c011, c011);
    const float c0 = fmaf(ay, c10 - c00, c00);
    const float c1 = fmaf(ay, c11 - c01, c01);
    return fmaf(az, c1 - c0, c0);
}

// Number of leading samples t = 0, 1, ... whose texture coordinates are
// certainly inside [0, n) on every axis, so the in-grid test can be skipped
// for them.  The bound is taken on the exact (real-number) coordinates
// A + B t of the FP32 formula with a margin of 4e-3 texel; the FP32
// evaluation differs from them by less than 1e-3 texel for any grid this
// library accepts, so the skipped tests would all have passed.
__device__ __forceinline__ int safe_steps(const PbGrid &g, const PbBeamGeom &B, float inv_s,
                                          float px, float py, float pz, float ux, float uy,
                                          float uz, int cap)
{
    const double margin = 4e-3;
    const float pv[3] = {px, py, pz}, uv[3] = {ux, uy, uz};
    const int nv[3] = {g.nx, g.ny, g.nz};
    double T = (double)cap;
    for (int a = 0; a < 3; ++a) {
        const double A = (double)inv_s * ((double)pv[a] + (double)B.iso[a]) + 0.5;
        const double Bt = (double)inv_s * (double)uv[a];
        const double lo = margin, hi = (double)nv[a] - margin;
        if (!(A >= lo && A <= hi) || Bt != Bt) return 0;
        if (Bt > 0.0) T = fmin(T, (hi - A) / Bt);
        else if (Bt < 0.0) T = fmin(T, (lo - A) / Bt);
    }
    if (!(T >= 0.0)) return 0;
    const double n = floor(T) + 1.0;
    return n < (double)cap ? (int)n : cap;
}

template <bool TEX>
__device__ __forceinline__ float ray_sample(const float *__restrict__ rho,
                                            cudaTextureObject_t tex, const PbGrid &g,
                                            float x, float y, float z)
{
    if (TEX) return tex3D<float>(tex, x, y, z);
    return trilinear(rho, g.nx, g.ny, g.nz, __fsub_rn(x, 0.5f), __fsub_rn(y, 0.5f),
                     __fsub_rn(z, 0.5f));
}

// Raw WET (cm) per voxel: samples every 1 mm from the voxel toward the
// source while the texture coordinate stays inside [0, n); WET = -0.05 +
// 0.1 * sum(max(RLSP, 0)).  The sum is carried in FP64 (FP32 partials of 8
// samples).  A ray that exceeds the grid-diagonal step cap stops and raises
// PB_ERR_RAY_CAP in *status.  The leading samples that are certainly inside
// the grid (safe_steps) go without the in-grid test: with cell records, as
// runs through flat cells and bursts of samples elsewhere; without them, 8
// fetches at a time.  Either way several fetches are in flight per thread.
//
// TEX = true samples RLSP through a border-0, linearly filtered 3-D texture
// and forms the ray direction with rnorm3df, as the reference does
// (CudaClasses.cuh:41-52, TextureClasses.cu:14-41), so the samples are the
// reference's own.  A ray is a chain of record loads (cell_run) with fetches
// between, and the kernel lives on occupancy; where hardly any cell is flat (image
// noise everywhere) the texture unit's rate bounds it.  There half of the samples
// can come from records of the texels with the unit's filter in FP32
// (200x188x160 CT with noise, 3 beams: 8.7 -> 6.5 ms), but they are off by a
// rounding in a third of the samples, and that decided a radius of the smoothing
// otherwise in some voxel of every tenth noisy volume.  The unit's own sum, exact
// and rounded once, makes it the slower one: 11.9 ms in FP64, 10.5 as two FP32
// sums of split texels.  So every sample is the unit's.
//
// TEX = false takes exact FP32 trilinear weights, from the records (flat_run,
// cell_sample2) or from global memory, and forms the direction in FP64, the CPU
// oracle's arithmetic.  Each sample by its eight texels from the volume is bound
// by the loads: 165x150x121, 2 beams, noise: 3.41 -> 1.8 ms by the records.

// floor(a) for -2^22 <= a < 2^22 on the FP32 adder: adding 1.5 * 2^23 with
// rounding toward -infinity leaves floor(a) in the low mantissa bits.
__device__ __forceinline__ int floor_small(float a)
{
    return __float_as_int(__fadd_rd(a, 12582912.0f)) - 0x4B400000;
}

__device__ __forceinline__ float floor_small_f(float a)
{
    return __fsub_rn(__fadd_rd(a, 12582912.0f), 12582912.0f);
}

// Row length (bytes) of the distance passes' work arrays: cells padded to a
// multiple of 4.
__host__ __device__ __forceinline__ int cell_row(int nx) { return (nx + 1 + 3) & ~3; }

// A handle's records as the ray trace reads them (texture_create below).  Cell
// (ci, cj, ck) holds the 2x2x2 texels with base (ci-1, cj-1, ck-1), with zeros
// outside the grid.
//   cell  with a texture: value and distance (of quad and dist below) of the cell,
//         (nx+1) x (ny+1) x (nz+1), x fastest
//   quad  without: (nx+1) x (ny+2) x (nz+1), x fastest: the texels (ci-1, r-1, ck-1),
//         (ci-1, r-1, ck), (ci, r-1, ck-1), (ci, r-1, ck); a cell's eight are
//         its entries at rows cj and cj + 1
//   dist  without: distance in cells to the nearest cell that is not flat, rows of
//         cell_row(nx) bytes
struct CellIndex {
    int cx, cxy;      // quad strides per row and per plane
    unsigned off;     // takes the biased integers of the float adders out
};

// Run of samples, starting with the one at (x, y, z), whose texture values
// are certainly the flat value v of the current cell.  Every cell within
// L-infinity distance r-1 of a flat cell with distance r is flat, with the
// same value (face-adjacent flat cells share four texels).  Sample m of the
// run lies within m*dmax texels of sample 0 on each axis, so its computed
// cell (floor(x-0.5)+1) is within floor(m*dmax)+1 cells of the current one,
// and the texture unit, which quantises the coordinate before taking the
// floor, may read the cell next to that one: one more.  Hence samples with
// m*dmax <= r-3 read only cells of value v, and a flat 2x2x2 neighbourhood
// filters to exactly v.  Returns 0 where no run is certain.
// `at` receives the quad that holds v (its first texel).
__device__ __forceinline__ float flat_run(const RayCells &C, const CellIndex &I, int drow, int cy,
                                          float x, float y, float z, float inv_dmax,
                                          const float4 *&at)
{
    const int i = floor_small(__fsub_rn(x, 0.5f)) + 1, j = floor_small(__fsub_rn(y, 0.5f)) + 1,
              k = floor_small(__fsub_rn(z, 0.5f)) + 1;
    // (up to 2^32 - 1 entries, twice the cells that a handle takes)
    const unsigned ui = i, uj = j, uk = k;
    const int d = __ldg(C.dist + (ui + (unsigned)drow * (uj + (unsigned)cy * uk)));
    if (d < 3) return 0.0f;
    at = C.quad + (ui + (unsigned)I.cx * uj + (unsigned)I.cxy * uk);
    // floor((r - 3) / dmax) + 1, every rounding downward so that the run
    // never exceeds the bound
    return floor_small_f(__fmul_rd((float)(d - 3), inv_dmax)) + 1.0f;
}

// The same from a texture's records: value and distance in one load.
__device__ __forceinline__ float cell_run(const float2 *__restrict__ rec, int cx, int cy,
                                            float x, float y, float z, float inv_dmax, float &v)
{
    const int i = floor_small(__fsub_rn(x, 0.5f)) + 1, j = floor_small(__fsub_rn(y, 0.5f)) + 1,
              k = floor_small(__fsub_rn(z, 0.5f)) + 1;
    const float2 r = __ldg(rec + (unsigned)(i + cx * (j + cy * k)));
    v = r.x;
    if (r.y < 3.0f) return 0.0f;
    return floor_small_f(__fmul_rd(r.y - 3.0f, inv_dmax)) + 1.0f;
}

// Samples from the quads: two 16-byte loads of 4.9 cycles each of the L1's data
// stage (exact ray trace of a 165x150x121 CT: 332 million wavefronts for 68 million
// loads of a warp); a linear 3-D FP32 fetch of a warp takes the unit 16.
//
// FILTER (pb_texture_sample): the texture unit's own filter, from its fixed-point rule: the
// coordinate to the nearest 1/256 (halves up), the cell and three 8-bit
// fractions from it, and the eight weights as whole 256ths that sum to 256,
// divided among z, then x, then y, each product to the nearest whole (halves
// to the upper texel; at the lower x, where y divides, to the lower one).
// The sum is the FP32 products', so a sample agrees with the unit's to FP32
// rounding.  Otherwise exact trilinear weights, in trilinear's operation order
// bit for bit.
constexpr float kFixMagic = 6291328.5f;    // 1.5 * 2^22 - 128 + 0.5: an ulp of 0.5,
                                           // coordinates below 8192
constexpr float kIntMagic = 12582912.0f;   // 1.5 * 2^23: an ulp of 1

template <bool FILTER>
__device__ __forceinline__ CellIndex cell_index(const PbGrid &g)
{
    CellIndex I;
    I.cx = g.nx + 1;
    I.cxy = I.cx * (g.ny + 2);
    // the integers below are cell - 1 + bias
    const unsigned bias = FILTER ? 0x256000u : 0x4B400000u;
    I.off = (bias - 1u) * (unsigned)(1 + I.cx + I.cxy);
    return I;
}

// The two samples at (X, Y, Z).x and .y; both inside the grid.
template <bool FILTER>
__device__ __forceinline__ float2 cell_sample2(const RayCells &C, const CellIndex &I, float2 X,
                                               float2 Y, float2 Z)
{
    auto bc = [](float a) { return make_float2(a, a); };
    float out[2];
    if constexpr (FILTER) {
        const float2 mx = __ffma2_rd(X, bc(256.0f), bc(kFixMagic));
        const float2 my = __ffma2_rd(Y, bc(256.0f), bc(kFixMagic));
        const float2 mz = __ffma2_rd(Z, bc(256.0f), bc(kFixMagic));
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const unsigned bx = __float_as_uint(s ? mx.y : mx.x);
            const unsigned by = __float_as_uint(s ? my.y : my.x);
            const unsigned bz = __float_as_uint(s ? mz.y : mz.x);
            const unsigned q = (bx >> 9) + (by >> 9) * (unsigned)I.cx +
                               (bz >> 9) * (unsigned)I.cxy - I.off;
            const float4 r0 = __ldg(C.quad + q), r1 = __ldg(C.quad + q + I.cx);
            // twice the 8-bit fractions, as floats 2^23 + 2 f
            const float fx = __uint_as_float((bx & 0x1FEu) | 0x4B000000u) - 8388608.0f;
            const float fy = __uint_as_float((by & 0x1FEu) | 0x4B000000u) - 8388608.0f;
            const float fz = __uint_as_float((bz & 0x1FEu) | 0x4B000000u) - 8388608.0f;
            // fractions / 256 with a bias far below 1/256 that decides halves
            constexpr float kTie = 3.814697265625e-06f;   // 2^-18
            const float ax = __fmaf_rn(fx, 1.0f / 512.0f, kTie);
            const float ayu = __fmaf_rn(fy, 1.0f / 512.0f, kTie);
            const float ayl = __fmaf_rn(fy, 1.0f / 512.0f, -kTie);
            const float g1 = __fmul_rn(fz, 0.5f);
            const float2 G = make_float2(256.0f - g1, g1);   // lower z, upper z
            const float2 M = bc(kIntMagic), nM = bc(-kIntMagic);
            const float2 A = __fadd2_rn(__ffma2_rn(G, bc(ax), M), nM);       // upper x
            const float2 B = __ffma2_rn(A, bc(-1.0f), G);                    // lower x
            const float2 C1 = __fadd2_rn(__ffma2_rn(A, bc(ayu), M), nM);     // upper x, upper y
            const float2 D1 = __fadd2_rn(__ffma2_rn(B, bc(ayl), M), nM);     // lower x, upper y
            const float2 C0 = __ffma2_rn(C1, bc(-1.0f), A);
            const float2 D0 = __ffma2_rn(D1, bc(-1.0f), B);
            float2 t = __fmul2_rn(D0, make_float2(r0.x, r0.y));
            t = __ffma2_rn(C0, make_float2(r0.z, r0.w), t);
            t = __ffma2_rn(D1, make_float2(r1.x, r1.y), t);
            t = __ffma2_rn(C1, make_float2(r1.z, r1.w), t);
            out[s] = __fmul_rn(__fadd_rn(t.x, t.y), 1.0f / 256.0f);
        }
    } else {
        const float2 xb = __fadd2_rn(X, bc(-0.5f)), yb = __fadd2_rn(Y, bc(-0.5f));
        const float2 zb = __fadd2_rn(Z, bc(-0.5f));
        const float2 mx = __fadd2_rd(xb, bc(kIntMagic)), my = __fadd2_rd(yb, bc(kIntMagic));
        const float2 mz = __fadd2_rd(zb, bc(kIntMagic));
        const float2 nM = bc(-kIntMagic), neg = bc(-1.0f);
        const float2 AX = __ffma2_rn(__fadd2_rn(mx, nM), neg, xb);
        const float2 AY = __ffma2_rn(__fadd2_rn(my, nM), neg, yb);
        const float2 AZ = __ffma2_rn(__fadd2_rn(mz, nM), neg, zb);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const unsigned q = __float_as_uint(s ? mx.y : mx.x) +
                               __float_as_uint(s ? my.y : my.x) * (unsigned)I.cx +
                               __float_as_uint(s ? mz.y : mz.x) * (unsigned)I.cxy - I.off;
            const float4 r0 = __ldg(C.quad + q), r1 = __ldg(C.quad + q + I.cx);
            const float2 ax = bc(s ? AX.y : AX.x), ay = bc(s ? AY.y : AY.x);
            const float2 l0 = make_float2(r0.x, r0.y), l1 = make_float2(r1.x, r1.y);
            const float2 c0 = __ffma2_rn(ax, __ffma2_rn(l0, neg, make_float2(r0.z, r0.w)), l0);
            const float2 c1 = __ffma2_rn(ax, __ffma2_rn(l1, neg, make_float2(r1.z, r1.w)), l1);
            const float2 c = __ffma2_rn(ay, __ffma2_rn(c0, neg, c1), c0);
            out[s] = fmaf(s ? AZ.y : AZ.x, c.y - c.x, c.x);
        }
    }
    return make_float2(out[0], out[1]);
}

// Samples of a burst, fetched together.
constexpr int kBurst = 4;
// Exact weights: after the n-th look at the records without a run, n bursts, at most
// kMaxBursts, go by until the next.
constexpr int kMaxBursts = 8;
// Resident blocks per SM (registers): texture 12 (40; they cover the latency of
// the dependent record loads: 10 took 6.77 ms against 6.52 on the 256x256x160
// phantom), exact weights 6 (80).
constexpr int kTextureBlocks = 12, kExactBlocks = 6;
// The batch's texture kernel keeps its item too and spills at 12: two plans of
// 48x52x45, 1 beam 56 us at 12 blocks, 50 at 10, 47 at 9, 46 at 8; eight of 64x68x61,
// 2 beams 220, 210, 210, 210; four of up to 1.6 million voxels, 1 beam 650, 630, 638,
// 635.
constexpr int kTextureBatchBlocks = 9;
// Up to kEachBricks a block per brick, above them kBricksPerBlock bricks a block in
// turn: us, a loop over bricks against a block each, 50x111x55, 4 beams 187 / 183;
// 96x87x68, 2 beams, noise in the body 241 / 239; 180x171x110, 3 beams (83,000
// bricks) 2587 / 2511; 256x256x160, 4 beams, phantom 3640 / 3729.  (One brick index
// in a row, divided by the three extents in the kernel, cost 8 % of a small volume's
// ray trace.)
constexpr int kBricksPerBlock = 8;
constexpr int64_t kEachBricks = 148 * 1024;

template <bool TEX>
__device__ __forceinline__ float raytrace_voxel(const float *__restrict__ rho,
                                                cudaTextureObject_t tex, const RayCells &rec,
                                                const PbGrid &g, const PbBeamGeom &B, int i, int j, int k,
                                                int cap, int *status)
{
    float px, py, pz, ux, uy, uz;
    vox_mm(B, g.spacing, i, j, k, px, py, pz);
    if (TEX) {
        ux = __fsub_rn(B.src[0], px);
        uy = __fsub_rn(B.src[1], py);
        uz = __fsub_rn(B.src[2], pz);
        const float nrm = rnorm3df(ux, uy, uz);
        ux = __fmul_rn(ux, nrm);
        uy = __fmul_rn(uy, nrm);
        uz = __fmul_rn(uz, nrm);
    } else {
        unit_to_source(B, px, py, pz, ux, uy, uz);
    }
    const float inv_s = __fdiv_rn(1.0f, g.spacing);
    const float fnx = (float)g.nx, fny = (float)g.ny, fnz = (float)g.nz;
    const float ix = B.iso[0], iy = B.iso[1], iz = B.iso[2];
    const int nsafe = safe_steps(g, B, inv_s, px, py, pz, ux, uy, uz, cap);
    double acc = 0.0;
    int n = 0;
    if (TEX ? rec.cell != nullptr : rec.quad != nullptr) {
        // runs through flat regions, samples elsewhere; the sample counter
        // is kept in FP32 (exact below 2^24).  Both filters on a flat cell
        // give exactly its value.
        const float dmax = fmaxf(fabsf(inv_s * ux), fmaxf(fabsf(inv_s * uy), fabsf(inv_s * uz))) +
                           1e-6f;
        const float inv_dmax = __frcp_rd(dmax);
        const float nsf = (float)nsafe;
        if constexpr (TEX) {
            const int cx = g.nx + 1, cy = g.ny + 1;
            float t = 0.0f;
            while (t < nsf) {
                const float x = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(ux, t, px), ix), 0.5f);
                const float y = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uy, t, py), iy), 0.5f);
                const float z = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uz, t, pz), iz), 0.5f);
                float v;
                const float run = cell_run(rec.cell, cx, cy, x, y, z, inv_dmax, v);
                if (run > 0.0f) {
                    const float m = fminf(run, nsf - t);
                    acc += (double)(m * fmaxf(v, 0.0f));
                    t += m;
                } else {
                    // not flat here: the texture unit for the next few samples
                    // before looking at the records again
                    float part = fmaxf(ray_sample<true>(rho, tex, g, x, y, z), 0.0f);
                    const float e = fminf(t + (float)kBurst, nsf);
                    {
                        // all fetches of the burst issued together; those past
                        // e (possibly outside the grid: the border reads 0) are
                        // not added, so the sum is the loop's, bit for bit
                        // (measured 7.50 -> 7.24 ms for the whole WET)
                        float sv[kBurst - 1];
#pragma unroll
                        for (int q = 1; q < kBurst; ++q) {
                            const float tq = __fadd_rn(t, (float)q);
                            const float x = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(ux, tq, px), ix), 0.5f);
                            const float y = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uy, tq, py), iy), 0.5f);
                            const float z = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uz, tq, pz), iz), 0.5f);
                            sv[q - 1] = fmaxf(tex3D<float>(tex, x, y, z), 0.0f);
                        }
#pragma unroll
                        for (int q = 1; q < kBurst; ++q)
                            part = __fadd_rn(t, (float)q) < e ? __fadd_rn(part, sv[q - 1]) : part;
                        t = fmaxf(__fadd_rn(t, 1.0f), e);
                    }
                    acc += (double)part;
                }
            }
            n = (int)t;
        } else {
            const int cy = g.ny + 1, drow = cell_row(g.nx);
            const CellIndex I = cell_index<false>(g);
            auto at2 = [&](float t0, float2 &X, float2 &Y, float2 &Z) {
                const float2 t2 = make_float2(t0, __fadd_rn(t0, 1.0f));
                auto axis = [&](float u, float p, float o) {
                    return __ffma2_rn(make_float2(inv_s, inv_s),
                                      __fadd2_rn(__ffma2_rn(make_float2(u, u), t2,
                                                            make_float2(p, p)), make_float2(o, o)),
                                      make_float2(0.5f, 0.5f));
                };
                X = axis(ux, px, ix);
                Y = axis(uy, py, iy);
                Z = axis(uz, pz, iz);
            };
            float t = 0.0f;
            float run_m = 0.0f, run_v = 0.0f;   // the last run's samples and their value
            int thick = 0;                      // looks at the records since then
            while (t < nsf) {
                float2 X, Y, Z;
                at2(t, X, Y, Z);
                const float4 *at = nullptr;
                const float run = flat_run(rec, I, drow, cy, X.x, Y.x, Z.x, inv_dmax, at);
                if (run > 0.0f) {
                    // a run's value is waited for at the next run only
                    acc += (double)(run_m * fmaxf(run_v, 0.0f));
                    run_m = fminf(run, nsf - t);
                    run_v = __ldg(&at->x);
                    t += run_m;
                    thick = 0;
                    continue;
                }
                // not flat here: the next few samples before looking at the
                // records again.  The fetches of a burst are issued together.
                if (t + (float)kBurst > nsf) {
                    float part = 0.0f;
                    for (; t < nsf; t += 1.0f) {
                        const float x = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(ux, t, px), ix), 0.5f);
                        const float y = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uy, t, py), iy), 0.5f);
                        const float z = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uz, t, pz), iz), 0.5f);
                        part += fmaxf(ray_sample<false>(rho, tex, g, x, y, z), 0.0f);
                    }
                    acc += (double)part;
                    break;
                }
                auto burst = [&](bool first) {
                    float sv[kBurst];
                    if (!first) at2(t, X, Y, Z);
#pragma unroll
                    for (int m = 0; m < kBurst; m += 2) {
                        if (m > 0) at2(t + (float)m, X, Y, Z);
                        const float2 w = cell_sample2<false>(rec, I, X, Y, Z);
                        sv[m] = w.x;
                        sv[m + 1] = w.y;
                    }
                    float part = fmaxf(sv[0], 0.0f);
#pragma unroll
                    for (int m = 1; m < kBurst; ++m) part = __fadd_rn(part, fmaxf(sv[m], 0.0f));
                    acc += (double)part;
                    t += (float)kBurst;
                };
                ++thick;
                burst(true);
#pragma unroll 1
                for (int q = 1; q < min(thick, kMaxBursts) && t + (float)kBurst <= nsf; ++q)
                    burst(false);
            }
            acc += (double)(run_m * fmaxf(run_v, 0.0f));
            n = (int)t;
        }
    } else {
        for (; n + 8 <= nsafe; n += 8) {
            float r[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const float t = (float)(n + m);
                const float x = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(ux, t, px), ix), 0.5f);
                const float y = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uy, t, py), iy), 0.5f);
                const float z = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uz, t, pz), iz), 0.5f);
                r[m] = ray_sample<TEX>(rho, tex, g, x, y, z);
            }
            float part = 0.0f;
#pragma unroll
            for (int m = 0; m < 8; ++m) part += fmaxf(r[m], 0.0f);
            acc += (double)part;
        }
    }
    float part = 0.0f;
    for (;; ++n) {
        const float t = (float)n;
        const float x = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(ux, t, px), ix), 0.5f);
        const float y = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uy, t, py), iy), 0.5f);
        const float z = __fmaf_rn(inv_s, __fadd_rn(__fmaf_rn(uz, t, pz), iz), 0.5f);
        if (n >= nsafe &&
            !(x >= 0.0f && x < fnx && y >= 0.0f && y < fny && z >= 0.0f && z < fnz))
            break;
        if (n >= cap) {
            if (status) atomicOr(status, (int)PB_ERR_RAY_CAP);
            break;
        }
        part += fmaxf(ray_sample<TEX>(rho, tex, g, x, y, z), 0.0f);
    }
    acc += (double)part;
    return __double2float_rn(fma(0.1, acc, -0.05));
}

// EACH: a block per brick.  Otherwise a block takes the bricks of its row and
// column in every gridDim.z-th plane (and, past the grid's limit, row).
template <bool TEX, bool EACH>
__global__ void __launch_bounds__(128, TEX ? kTextureBlocks : kExactBlocks)
k_raytrace(const float *__restrict__ rho, cudaTextureObject_t tex, const RayCells rec,
           PbGrid g, const __grid_constant__ BeamGeomSet bs, int n_beams, int cap,
           float *__restrict__ raw, int *status)
{
    const unsigned by = (g.ny + 3) / 4, bz = (g.nz + 3) / 4;
    const int64_t V = (int64_t)g.nx * g.ny * g.nz;
    const int i = blockIdx.x * 8 + (threadIdx.x & 7);
    if (i >= g.nx) return;
    auto brick = [&](unsigned y, unsigned z) {
        const int j = y * 4 + ((threadIdx.x >> 3) & 3);
        const int b = z / bz, k = (z - b * bz) * 4 + (threadIdx.x >> 5);
        if (j >= g.ny || k >= g.nz) return;
        const int64_t v = i + (int64_t)g.nx * (j + (int64_t)g.ny * k);
        raw[b * V + v] = raytrace_voxel<TEX>(rho, tex, rec, g, bs.b[b], i, j, k, cap, status);
    };
    if constexpr (EACH) {
        brick(blockIdx.y, blockIdx.z);
    } else {
        for (unsigned y = blockIdx.y; y < by; y += gridDim.y)
            for (unsigned z = blockIdx.z; z < bz * n_beams; z += gridDim.z) brick(y, z);
    }
}

// Samples at the coordinates of `at` (x, y, z; two per thread), through the
// texture unit and from the cell records with its filter; only those the
// records take (inside the grid by the ray trace's margin), the others 0.
__global__ void k_texture_quads(cudaTextureObject_t tex, PbGrid g, int64_t n,
                                float4 *__restrict__ quad)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int cx = g.nx + 1, rows = g.ny + 2;
    const int i = (int)(q % cx), j = (int)(q / cx % rows), k = (int)(q / cx / rows);
    // a texel's centre: weight 1 for it, border 0 outside
    auto texel = [&](int a, int c) {
        return tex3D<float>(tex, (float)(i - 1 + a) + 0.5f, (float)(j - 1) + 0.5f,
                            (float)(k - 1 + c) + 0.5f);
    };
    quad[q] = make_float4(texel(0, 0), texel(0, 1), texel(1, 0), texel(1, 1));
}

__global__ void k_texture_sample(cudaTextureObject_t tex, const RayCells rec, PbGrid g,
                                 const float *__restrict__ at, int64_t pairs,
                                 float *__restrict__ unit, float *__restrict__ cells)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= pairs) return;
    float c[3][2];
    bool in[2];
    for (int s = 0; s < 2; ++s) {
        const int n[3] = {g.nx, g.ny, g.nz};
        in[s] = true;
        for (int a = 0; a < 3; ++a) {
            c[a][s] = at[6 * q + 3 * s + a];
            in[s] = in[s] && c[a][s] >= 3e-3f && c[a][s] <= (float)n[a] - 3e-3f;
        }
        if (!in[s])
            for (int a = 0; a < 3; ++a) c[a][s] = 0.5f;
    }
    const float2 w = cell_sample2<true>(rec, cell_index<true>(g), make_float2(c[0][0], c[0][1]),
                                        make_float2(c[1][0], c[1][1]),
                                        make_float2(c[2][0], c[2][1]));
    for (int s = 0; s < 2; ++s) {
        unit[2 * q + s] = in[s] ? tex3D<float>(tex, c[0][s], c[1][s], c[2][s]) : 0.0f;
        cells[2 * q + s] = in[s] ? (s ? w.y : w.x) : 0.0f;
    }
}

// A texture's handle holds no quads, so they are made here from the texture, for the length of the call.
PbStatus launch_texture_sample(cudaTextureObject_t tex, const PbGrid &g, const float *at,
                               int64_t pairs, float *unit, float *cells, cudaStream_t st)
{
    if (pairs == 0) return PB_OK;
    const int64_t n = (int64_t)(g.nx + 1) * (g.ny + 2) * (g.nz + 1);
    float4 *quad = nullptr;
    PbStatus s = check_cuda(cudaMalloc(&quad, sizeof(float4) * n), "cudaMalloc");
    if (s != PB_OK) return s;
    k_texture_quads<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(tex, g, n, quad);
    k_texture_sample<<<(unsigned)((pairs + 127) / 128), 128, 0, st>>>(
        tex, RayCells{quad, nullptr, nullptr}, g, at, pairs, unit, cells);
    s = check_launch("k_texture_sample");
    const PbStatus w = check_cuda(cudaStreamSynchronize(st), "cudaStreamSynchronize");
    cudaFree(quad);
    return s != PB_OK ? s : w;
}

// Per-beam table of the smoothing samples.  Sample (direction dd, radius
// dr = r + 1 mm) of voxel (i, j, k) lies, along each axis a, at index
// coordinate  m_a = i_a + dr * dm_a  up to the FP32 roundings of the
// reference's sample position (the map from head to image coordinates is
// linear and the voxel's own coordinate is an integer), where dm_a is the
// index step of 1 mm along the direction.  Where the fractional part of
// dr * dm_a is farther than the rounding bound from 0.5, roundf picks
// i_a + ro, ro = round(dr * dm_a), for every voxel of the beam.  The other
// (direction, radius, axis) triples are flagged in tmask and take the
// reference-order position per voxel, which is i_a + ro or i_a + ro + 1
// with ro = floor(dr * dm_a) there.  The table holds ro + 1/2 (hh): for a
// flagged triple, the half-integer the position is compared with.
struct SmoothBeam {
    int off[6][9];            // linear-index offset when no axis is flagged
    float hh[6][9][3];        // per-axis index offset ro + 1/2: ro = round(dr * dm_a),
                              // floor where flagged
    unsigned tmask[6];        // 3 bits (x, y, z) per radius, radius 1 lowest
    int margin[3];            // interior: margin_a <= i_a <= n_a - 1 - margin_a
    float inv_s;              // 1 / spacing in FP32
    int pow2;                 // the spacing is a power of two: inv_s is exact
};

struct SmoothSet {
    SmoothBeam b[PB_MAX_BEAMS];
};

// Which (direction, radius, axis) samples can come near a half-integer.  A
// voxel's reference-order index coordinate differs from the real-number
// i_a + dr*dm_a by at most `err` (FP32 roundings of positions no larger
// than the grid's extent plus the isocentre), so where the fractional part
// of dr*dm_a is farther than tie + 2*err + 1e-4 from 0.5, every voxel's
// sample rounds to i_a + round(dr*dm_a); elsewhere the kernel takes the
// reference-order index, which is one of the two integers around it.
// (With beams along the image axes the lateral step is exactly half a
// voxel along an axis, so every other radius of two directions is flagged.)
static void smooth_table(const PbGrid &g, const PbBeamGeom &B, const float *c, const float *sn,
                         double err, double tie, SmoothBeam &T)
{
    memset(&T, 0, sizeof(T));
    const double inv_s = 1.0 / (double)g.spacing;
    int e2;
    T.pow2 = frexp((double)g.spacing, &e2) == 0.5;
    T.inv_s = (float)inv_s;
    const double sg = B.singa, cg = B.cosga, st = B.sinta, ct = B.costa;
    // head (hx, hy, hz) -> (xz, yz, zz) = (-hx, hz, hy); gantry; couch:
    // x = (xz cg - yz sg) ct + zz st ; y = xz sg + yz cg ;
    // z = -(xz cg - yz sg) st + zz ct.  Rows: image axis; columns: hx, hy.
    const double M[3][2] = {{-cg * ct, st}, {-sg, 0.0}, {cg * st, ct}};
    const double band = tie + 2.0 * err + 1e-4;
    const int64_t sy = g.nx, sz = (int64_t)g.nx * g.ny;
    for (int dd = 0; dd < 6; ++dd) {
        double dm[3];
        for (int a = 0; a < 3; ++a)
            dm[a] = (M[a][0] * (double)c[dd] + M[a][1] * (double)sn[dd]) * inv_s;
        unsigned m = 0;
        for (int r = 0; r < 9; ++r) {
            const double dr = (double)(r + 1);
            // dr is a small integer, so the FP64 product is exact and its
            // FP32 rounding is the FP32 product
            int64_t off = 0;
            for (int a = 0; a < 3; ++a) {
                const double x = dr * dm[a];
                const bool flag = fabs((x - floor(x)) - 0.5) < band;
                if (flag) m |= 1u << (3 * r + a);
                // flagged: the lower of the two candidates (exact_steps)
                const int o = (int)(flag ? floor(x) : nearbyint(x));
                T.hh[dd][r][a] = (float)o + 0.5f;
                off += (a == 0 ? 1 : a == 1 ? sy : sz) * (int64_t)o;
                T.margin[a] = std::max(T.margin[a], (int)ceil(fabs(x)) + 1);
            }
            T.off[dd][r] = (int)off;   // used only when the grid has < 2^31 voxels
        }
        T.tmask[dd] = m;
    }
}

static void smooth_set(const PbGrid &g, const PbBeamGeom *beams, int n_beams, SmoothSet &o)
{
    float c[6], sn[6];
    smooth_dirs(c, sn);
    const double inv_s = 1.0 / (double)g.spacing;
    // Bound on |FP32 reference-order index - real index|: about 8 roundings
    // of a coordinate no larger than `ext` mm, divided by the spacing, plus
    // 2e-4; the band is twice that, at least 2e-3.
    double ext = g.spacing * (double)(g.nx > g.ny ? (g.nx > g.nz ? g.nx : g.nz)
                                                  : (g.ny > g.nz ? g.ny : g.nz));
    for (int b = 0; b < n_beams; ++b)
        for (int a = 0; a < 3; ++a) ext = fmax(ext, fabs((double)beams[b].iso[a]) + ext);
    const double err = 8.0 * ldexp(ext + 16.0, -24) * inv_s + 2e-4;
    const double tie = fmax(2e-3, 2.0 * err);
    for (int b = 0; b < n_beams; ++b) smooth_table(g, beams[b], c, sn, err, tie, o.b[b]);
}

// The correctly rounded quotient, out of line: the unrolled smoothing
// loop calls it from many places.
__device__ __noinline__ float div_rn(float q, float s) { return __fdiv_rn(q, s); }

// roundf(q / s) (CudaClasses.cuh:112-116) minus lo, for a flagged sample
// whose quotient lies within half a voxel of h = lo + 1/2: 1 when the
// quotient is above h, or equal to it and positive (roundf rounds halves
// away from zero), else 0.  The quotient is the correctly rounded one;
// with a power-of-two spacing 1/s is exact, so q * (1/s) is it.
template <bool POW2>
__device__ __forceinline__ int round_up(float q, float h, float s, float inv_s)
{
    const float m = POW2 ? __fmul_rn(q, inv_s) : div_rn(q, s);
    return (m > h || (m == h && h > 0.0f)) ? 1 : 0;
}

// Sample (dd, r) along the flagged axes: the reference's FP32 position
// (head point plus dr*(c, s, 0), rotated to the image frame, plus the
// isocentre) divided by the spacing and rounded, as 0/1 steps from the
// table's lower candidates; fi, fj, fk are the voxel's indexes as floats.
// Only the flagged axes' image coordinates are formed.
// The six smoothing directions (cos, sin of i pi/3) as the reference forms
// them on the device: the FP32 angle (float)i * pi / 3 and CUDA's sincosf
// (IMPTClasses.cu:175-177).  Ties decided by the FP32 sample positions
// depend on these exact values, so they are CUDA's, not the host library's.
__device__ __forceinline__ void smooth_dir_dev(int i, float &c, float &s)
{
    sincosf(__fdiv_rn(__fmul_rn((float)i, 3.141592654f), 3.0f), &s, &c);
}

template <bool POW2>
__device__ __forceinline__ void exact_steps(const PbBeamGeom &B, const SmoothBeam &T, float s,
                                            const float *dc, const float *ds, float hx,
                                            float hy, float hz, float fi, float fj, float fk,
                                            int dd, int r, int axes, int &ui, int &uj, int &uk)
{
    // h + dr * (cos, sin), dr = r + 1 mm, each one fused multiply-add as the
    // reference's compiled code forms it (IMPTClasses.cu:180-181)
    const float dr = (float)(r + 1);
    const float hxs = __fmaf_rn(dr, dc[dd], hx);
    const float hys = __fmaf_rn(dr, ds[dd], hy);
    float qx, qy, qz;
    if (axes & 1) {
        head_to_image_ref(B, hxs, hys, hz, qx, qy, qz);
        ui = round_up<POW2>(__fadd_rn(qx, B.iso[0]), __fadd_rn(fi, T.hh[dd][r][0]), s,
                            T.inv_s);
    }
    if (axes & 2) {
        head_to_image_ref(B, hxs, hys, hz, qx, qy, qz);
        uj = round_up<POW2>(__fadd_rn(qy, B.iso[1]), __fadd_rn(fj, T.hh[dd][r][1]), s,
                            T.inv_s);
    }
    if (axes & 4) {
        head_to_image_ref(B, hxs, hys, hz, qx, qy, qz);
        uk = round_up<POW2>(__fadd_rn(qz, B.iso[2]), __fadd_rn(fk, T.hh[dd][r][2]), s,
                            T.inv_s);
    }
}

// Smoothed WET: mean of the voxel's raw WET and the in-grid nearest-voxel
// samples at 1..9 mm along six BEV-lateral directions, taking radius dr
// while dr < 10*WET(cm) (IMPTClasses.cu:166-198), summed in FP32 in the
// reference's order (direction, then radius).  A sample is the voxel at
// a fixed offset from this one (SmoothBeam), except along flagged axes,
// where the reference's FP32 position is rounded (exact_steps); the
// chosen voxels are the reference's.  POW2: the grid spacing is a power
// of two.

// Radii 1..nr of a voxel: dr < lim and dr < 10.
__device__ __forceinline__ int smooth_radii(float lim)
{
    return lim > 9.0f ? 9 : (int)ceilf(lim) - 1;
}

// One voxel near the faces: every sample is tested against the grid.
template <bool POW2>
__device__ __forceinline__ float smooth_voxel(const float *__restrict__ R, const PbGrid &g,
                                              const PbBeamGeom &B, const SmoothBeam &T,
                                              const float *dc, const float *ds, int i, int j,
                                              int k, float center)
{
    const int nr = smooth_radii(__fmul_rn(center, 10.0f));
    float px, py, pz, hx, hy, hz;
    vox_mm(B, g.spacing, i, j, k, px, py, pz);
    image_to_head_ref(B, px, py, pz, hx, hy, hz);
    const float s = g.spacing;
    const float fi = (float)i, fj = (float)j, fk = (float)k;
    float sum = center;
    int n = 1;
    for (int dd = 0; dd < 6; ++dd) {
        unsigned tm = T.tmask[dd];
#pragma unroll 1
        for (int r = 0; r < 9; ++r, tm >>= 3) {
            int ii = i + __float2int_rd(T.hh[dd][r][0]), jj = j + __float2int_rd(T.hh[dd][r][1]),
                kk = k + __float2int_rd(T.hh[dd][r][2]);
            const int axes = tm & 7u;
            if (axes) {
                int ui = 0, uj = 0, uk = 0;
                exact_steps<POW2>(B, T, s, dc, ds, hx, hy, hz, fi, fj, fk, dd, r, axes, ui, uj,
                                  uk);
                ii += ui;
                jj += uj;
                kk += uk;
            }
            const bool take = r < nr && (unsigned)ii < (unsigned)g.nx &&
                              (unsigned)jj < (unsigned)g.ny && (unsigned)kk < (unsigned)g.nz;
            if (take) {
                sum = __fadd_rn(sum, __ldg(R + ii + (int64_t)g.nx * (jj + (int64_t)g.ny * kk)));
                n += 1;
            }
        }
    }
    return __fdiv_rn(sum, (float)n);
}

// The voxels whose every sample lies in the grid (the table's margins) and the
// shell around them are different blocks of the launch.  Inside, a thread takes
// PER voxels 32 apart in memory, a warp 32 * PER consecutive ones: a
// sample's table entry, its test for a flagged axis and its address are formed
// once for them, whose loads differ by a constant, and a warp's load is one
// run of 128 bytes.  One voxel a thread in 8x4x4 bricks, interior or not, spent
// some 20 instructions on a sample that is not flagged (issue slots 87 % used) and
// four L1 wavefronts on each load.  256x256x160, 4 beams along the axes (18 of 54
// samples flagged): 2.28 -> 1.7 ms; 200x188x160, 3 oblique beams: 0.93 -> 0.46 ms.
//
// PER is 4, or 2 where fours would fill the GPU less than twice (kSmoothFew): then
// the chain of a thread's samples is the launch's length.  us, one voxel a thread /
// 2 / 4: 96x88x72, 1 beam 42 / 26 / 35; 322,000 voxels, 1 beam 36 / 27 / 46;
// 421,000, 2 beams 62 / 36 / 50; 305,000, 4 beams 93 / 82 / 91; 572,000, 2 beams
// 87 / 48 / 49; 1,351,000, 2 beams 178 / 157 / 129.

// The inner box of a grid: voxels m[a] .. n[a] - 1 - m[a] of each axis, or none;
// the blocks of the inside (over the whole volume) and of the shell.
struct SmoothBox {
    int mx, my, mz;                // half of each axis where nothing is inside
    long long inner, shell;        // blocks
};

// Largest volume with inner blocks: the index of their last thread's last voxel,
// past the volume's end in the last block, still is an int.  Larger volumes are all shell.
constexpr long long smooth_inner_max(int per) { return 0x7fffffffll - 128 * per; }
constexpr long long smooth_last_index(long long V, int per)
{
    return (V + 128 * per - 1) / (128 * per) * (128 * per) - 1;
}
static_assert(smooth_last_index(smooth_inner_max(2), 2) <= 0x7fffffffll &&
              smooth_last_index(smooth_inner_max(2) - 255, 2) <= 0x7fffffffll &&
              smooth_last_index(smooth_inner_max(4), 4) <= 0x7fffffffll &&
              smooth_last_index(smooth_inner_max(4) - 511, 4) <= 0x7fffffffll,
              "a voxel index of the smoothing's inner blocks passes INT32_MAX");

template <int PER>
__host__ __device__ __forceinline__ SmoothBox smooth_box(const PbGrid &g, const int *margin)
{
    SmoothBox X;
    const long long V = (long long)g.nx * g.ny * g.nz;
    const bool some = 2 * margin[0] < g.nx && 2 * margin[1] < g.ny && 2 * margin[2] < g.nz &&
                      V <= smooth_inner_max(PER);
    X.mx = margin[0];
    X.my = margin[1];
    // nothing inside: the shell's end planes are the whole volume
    X.mz = some ? margin[2] : g.nz;
    const long long in = some ? (long long)(g.nx - 2 * X.mx) * (g.ny - 2 * X.my) *
                                    (g.nz - 2 * X.mz) : 0;
    X.inner = some ? (V + 128 * PER - 1) / (128 * PER) : 0;
    X.shell = (V - in + 127) / 128;
    return X;
}

// The q-th voxel of the shell: the end planes, then of each other plane the end
// rows and of its other rows the ends.  False past the last.
__device__ __forceinline__ bool shell_voxel(const PbGrid &g, const SmoothBox &X, long long q,
                                            int &i, int &j, int &k)
{
    const long long plane = (long long)g.nx * g.ny;
    if (X.mz >= g.nz) {                          // all of the volume
        if (q >= plane * g.nz) return false;
        k = (int)(q / plane);
        q -= plane * k;
        j = (int)q / g.nx;
        i = (int)q - j * g.nx;
        return true;
    }
    if (q < 2 * X.mz * plane) {
        k = (int)(q / plane);
        q -= plane * k;
        if (k >= X.mz) k += g.nz - 2 * X.mz;
        j = (int)q / g.nx;
        i = (int)q - j * g.nx;
        return true;
    }
    q -= 2 * X.mz * plane;
    const int rows = 2 * X.my * g.nx, per = rows + (g.ny - 2 * X.my) * 2 * X.mx;
    if (per == 0) return false;
    k = X.mz + (int)(q / per);
    if (k >= g.nz - X.mz) return false;
    int r = (int)(q - (long long)per * (k - X.mz));
    if (r < rows) {
        j = r / g.nx;
        i = r - j * g.nx;
        if (j >= X.my) j += g.ny - 2 * X.my;
        return true;
    }
    r -= rows;
    j = X.my + r / (2 * X.mx);
    i = r % (2 * X.mx);
    if (i >= X.mx) i += g.nx - 2 * X.mx;
    return true;
}

template <bool POW2, int PER>
__device__ __forceinline__ void smooth_block(const float *__restrict__ R, const PbGrid &g,
                                             const PbBeamGeom &Bp, const SmoothBeam &T,
                                             const float *dc, const float *ds, long long block,
                                             float *__restrict__ out)
{
    const int64_t V = (int64_t)g.nx * g.ny * g.nz;
    const SmoothBox X = smooth_box<PER>(g, T.margin);
    const PbBeamGeom B = Bp;   // the rotation and isocentre in registers
    const float s = g.spacing;
    int i, j, k;
    if (block >= X.inner) {
        if (!shell_voxel(g, X, (block - X.inner) * 128 + threadIdx.x, i, j, k)) return;
        const int64_t v = i + (int64_t)g.nx * (j + (int64_t)g.ny * k);
        const float c = R[v];
        out[v] = 1.0f < __fmul_rn(c, 10.0f) ? smooth_voxel<POW2>(R, g, B, T, dc, ds, i, j, k, c)
                                            : c;
        return;
    }
    const int v0 = (int)block * (128 * PER) + (threadIdx.x >> 5) * (32 * PER) +
                   (threadIdx.x & 31);
    if (v0 >= V) return;
    {
        const unsigned row = (unsigned)v0 / (unsigned)g.nx;
        i = (int)((unsigned)v0 - row * (unsigned)g.nx);
        k = (int)(row / (unsigned)g.ny);
        j = (int)(row - (unsigned)k * (unsigned)g.ny);
    }
    // Whether every sample of the PER, at either candidate, lies in the
    // volume's memory: then the loads need no tests.  What a voxel of the shell
    // reads so is not used.
    const int64_t reach = X.mx + (int64_t)g.nx * (X.my + (int64_t)g.ny * X.mz);
    const bool whole = v0 >= reach && v0 + 32 * (PER - 1) + reach < V;
    float center[PER], sum[PER], hx[PER], hy[PER], hz[PER];
    float fi[PER], fj[PER], fk[PER];
    int nr[PER];        // radii of each voxel, -1: not inside
    bool inner = false;
#pragma unroll
    for (int m = 0; m < PER; ++m) {
        if (m > 0) {
            i += 32;
            while (i >= g.nx) {
                i -= g.nx;
                if (++j == g.ny) {
                    j = 0;
                    ++k;
                }
            }
        }
        const bool in = i >= X.mx && i < g.nx - X.mx && j >= X.my && j < g.ny - X.my &&
                        k >= X.mz && k < g.nz - X.mz;
        center[m] = in ? R[v0 + 32 * m] : 0.0f;
        sum[m] = center[m];
        const float lim = __fmul_rn(center[m], 10.0f);
        nr[m] = !in ? -1 : 1.0f < lim ? smooth_radii(lim) : 0;
        inner |= nr[m] > 0;
        float px, py, pz;
        vox_mm(B, s, i, j, k, px, py, pz);
        image_to_head_ref(B, px, py, pz, hx[m], hy[m], hz[m]);
        fi[m] = (float)i;
        fj[m] = (float)j;
        fk[m] = (float)k;
    }
    if (whole && inner) {
        const float *at = R + v0;
        const int sy = g.nx, sz = g.nx * g.ny;
        for (int dd = 0; dd < 6; ++dd) {
            const unsigned tm = T.tmask[dd];   // the same for the whole beam
            if (tm == 0) {
#pragma unroll
                for (int r = 0; r < 9; ++r) {
                    const float *q = at + T.off[dd][r];
#pragma unroll
                    for (int m = 0; m < PER; ++m) {
                        const float x = __ldg(q + 32 * m);
                        sum[m] = r < nr[m] ? __fadd_rn(sum[m], x) : sum[m];
                    }
                }
                continue;
            }
            const float c = dc[dd], sn = ds[dd];
#pragma unroll 1
            for (int r = 0; r < 9; ++r) {
                const int axes = (tm >> (3 * r)) & 7u;
                const float *q = at + T.off[dd][r];
                float x[PER] = {};
                // One flagged axis, the usual case (beams along the image
                // axes): exact_steps' operations for it alone, with what does
                // not change over the samples in registers.  The candidate is
                // inside the grid, so h > 0 and a quotient of h rounds up.
                auto one_axis = [&](auto a, const int stride) {
                    constexpr int A = decltype(a)::value;
                    const float hh = T.hh[dd][r][A], dr = (float)(r + 1);
#pragma unroll
                    for (int m = 0; m < PER; ++m) {
                        const float xz = -__fmaf_rn(dr, c, hx[m]);
                        float p;
                        if constexpr (A == 1) {
                            p = __fmaf_rn(xz, B.singa, __fmul_rn(hz[m], B.cosga));
                        } else {
                            const float xg = __fmaf_rn(xz, B.cosga, __fmul_rn(-hz[m], B.singa));
                            const float zg = __fmaf_rn(dr, sn, hy[m]);
                            p = A == 0 ? __fmaf_rn(xg, B.costa, __fmul_rn(zg, B.sinta))
                                       : __fmaf_rn(-xg, B.sinta, __fmul_rn(zg, B.costa));
                        }
                        p = __fadd_rn(p, B.iso[A]);
                        const float h = __fadd_rn(A == 0 ? fi[m] : A == 1 ? fj[m] : fk[m], hh);
                        const float quotient = POW2 ? __fmul_rn(p, T.inv_s) : div_rn(p, s);
                        x[m] = __ldg(q + 32 * m + (quotient >= h ? stride : 0));
                    }
                };
                if (axes == 1) {
                    one_axis(std::integral_constant<int, 0>{}, 1);
                } else if (axes == 2) {
                    one_axis(std::integral_constant<int, 1>{}, sy);
                } else if (axes == 4) {
                    one_axis(std::integral_constant<int, 2>{}, sz);
                } else if (axes) {
#pragma unroll 1
                    for (int m = 0; m < PER; ++m) {
                        int ui = 0, uj = 0, uk = 0;
                        auto of = [&](const float *v) {   // no indexed registers
                            float r = v[0];
#pragma unroll
                            for (int l = 1; l < PER; ++l) r = l == m ? v[l] : r;
                            return r;
                        };
                        exact_steps<POW2>(B, T, s, dc, ds, of(hx), of(hy), of(hz), of(fi), of(fj),
                                          of(fk), dd, r, axes, ui, uj, uk);
                        const float w = __ldg(q + 32 * m + (ui + sy * uj + sz * uk));
#pragma unroll
                        for (int l = 0; l < PER; ++l) x[l] = l == m ? w : x[l];
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < PER; ++m) x[m] = __ldg(q + 32 * m);
                }
#pragma unroll
                for (int m = 0; m < PER; ++m)
                    sum[m] = r < nr[m] ? __fadd_rn(sum[m], x[m]) : sum[m];
            }
        }
    }
#pragma unroll
    for (int m = 0; m < PER; ++m) {
        if (nr[m] < 0) continue;
        float r = nr[m] > 0 ? __fdiv_rn(sum[m], (float)(6 * nr[m] + 1)) : center[m];
        if (!whole && nr[m] > 0)   // the first and last rows inside
            r = smooth_voxel<POW2>(R, g, B, T, dc, ds, (int)fi[m], (int)fj[m], (int)fk[m],
                                   center[m]);
        out[v0 + 32 * m] = r;
    }
}

// Resident blocks per SM (registers): 9 of 56; 6, 7, 8 and 10 took 6.15, 5.96, 5.84
// and 5.90 ms for the whole WET of the 256x256x160 phantom against 5.80.
// For the batch, whose table is in shared memory, 10: 8.03 ms for a batch of 8 plans
// against 8.18 (6) and 8.08 (8).
constexpr int kSmoothBlocks = 9, kSmoothBatchBlocks = 10;
constexpr int64_t kSmoothFew = 2ll * 148 * kSmoothBlocks * 128 * 4;   // voxels x beams
// First block of each beam.
struct SmoothStarts {
    int n;
    unsigned start[PB_MAX_BEAMS];
};

template <bool POW2, int PER>
__global__ void __launch_bounds__(128, kSmoothBlocks)
k_smooth(const float *__restrict__ raw, PbGrid g, const __grid_constant__ BeamGeomSet bs,
         const __grid_constant__ SmoothSet st,
         const __grid_constant__ SmoothStarts at, float *__restrict__ wet)
{
    __shared__ float s_dc[6], s_ds[6];
    if (threadIdx.x < 6) smooth_dir_dev(threadIdx.x, s_dc[threadIdx.x], s_ds[threadIdx.x]);
    __syncthreads();
    int b = 0;
    while (b + 1 < at.n && blockIdx.x >= at.start[b + 1]) ++b;
    const int64_t V = (int64_t)g.nx * g.ny * g.nz;
    smooth_block<POW2, PER>(raw + b * V, g, bs.b[b], st.b[b], s_dc, s_ds, blockIdx.x - at.start[b],
                       wet + b * V);
}

// One (plan, beam) of a batched WET pass.
struct BatchWet {
    PbGrid g;
    PbBeamGeom geom;
    const float *rlsp;
    cudaTextureObject_t tex;
    RayCells rec;               // the handle's cell records (or null)
    float *raw;                 // this beam's unsmoothed WET (V)
    float *wet;                 // this beam's smoothed WET (V)
    SmoothBeam sm;              // this beam's smoothing samples
    int cap;
    int bx, by, bz;             // 8x4x4 bricks per axis
    long long brick_start;      // first brick of this item in the launches
    long long smooth_blocks;    // its blocks of the smoothing launch, no more than its bricks
};

__device__ __forceinline__ int find_wet_item(const BatchWet *__restrict__ items, int n,
                                             long long brick)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].brick_start <= brick) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Brick of 8x4x4 voxels of one (plan, beam) per block of 128 threads.
__device__ __forceinline__ bool brick_voxel(const BatchWet &W, long long brick, int &i, int &j,
                                            int &k)
{
    long long lb = brick - W.brick_start;
    const int bx = (int)(lb % W.bx);
    lb /= W.bx;
    const int by = (int)(lb % W.by);
    const int bz = (int)(lb / W.by);
    i = bx * 8 + (threadIdx.x & 7);
    j = by * 4 + ((threadIdx.x >> 3) & 3);
    k = bz * 4 + (threadIdx.x >> 5);
    return i < W.g.nx && j < W.g.ny && k < W.g.nz;
}

__global__ void __launch_bounds__(128, kTextureBatchBlocks)
k_raytrace_batch(const BatchWet *__restrict__ items, int n_items, int *status)
{
    const BatchWet &W = items[find_wet_item(items, n_items, blockIdx.x)];
    int i, j, k;
    if (!brick_voxel(W, blockIdx.x, i, j, k)) return;
    float r;
    if (W.tex)
        r = raytrace_voxel<true>(W.rlsp, W.tex, W.rec, W.g, W.geom, i, j, k, W.cap, status);
    else
        r = raytrace_voxel<false>(W.rlsp, 0, W.rec, W.g, W.geom, i, j, k, W.cap, status);
    W.raw[i + (int64_t)W.g.nx * (j + (int64_t)W.g.ny * k)] = r;
}

template <int PER>
__global__ void __launch_bounds__(128, kSmoothBatchBlocks)
k_smooth_batch(const BatchWet *__restrict__ items, int n_items)
{
    static_assert(sizeof(SmoothBeam) % 4 == 0, "the table is copied as words");
    __shared__ SmoothBeam sm;
    __shared__ float s_dc[6], s_ds[6];
    const BatchWet &W = items[find_wet_item(items, n_items, blockIdx.x)];
    const long long block = blockIdx.x - W.brick_start;
    if (block >= W.smooth_blocks) return;   // the whole block
    if (threadIdx.x < 6) smooth_dir_dev(threadIdx.x, s_dc[threadIdx.x], s_ds[threadIdx.x]);
    // the block's sample table into shared memory (one item per block)
    const int *src = reinterpret_cast<const int *>(&W.sm);
    int *dst = reinterpret_cast<int *>(&sm);
    for (int q = threadIdx.x; q < (int)(sizeof(SmoothBeam) / 4); q += blockDim.x)
        dst[q] = __ldg(src + q);
    __syncthreads();
    if (sm.pow2)
        smooth_block<true, PER>(W.raw, W.g, W.geom, sm, s_dc, s_ds, block, W.wet);
    else
        smooth_block<false, PER>(W.raw, W.g, W.geom, sm, s_dc, s_ds, block, W.wet);
}

__device__ float g_smooth_dirs[12];

__global__ void k_smooth_dirs()
{
    if (threadIdx.x < 6)
        smooth_dir_dev(threadIdx.x, g_smooth_dirs[threadIdx.x], g_smooth_dirs[6 + threadIdx.x]);
}

PbStatus device_smooth_dirs(float *c, float *s)
{
    k_smooth_dirs<<<1, 32>>>();
    PbStatus st = check_launch("k_smooth_dirs");
    float v[12];
    if (st == PB_OK)
        st = check_cuda(cudaMemcpyFromSymbol(v, g_smooth_dirs, sizeof(v)),
                        "cudaMemcpyFromSymbol(directions)");
    if (st != PB_OK) return st;
    for (int i = 0; i < 6; ++i) {
        c[i] = v[i];
        s[i] = v[6 + i];
    }
    return PB_OK;
}

int ray_step_cap(const PbGrid &g)
{
    const double diag = g.spacing * sqrt((double)g.nx * g.nx + (double)g.ny * g.ny +
                                         (double)g.nz * g.nz);
    return (int)ceil(diag) + 2;
}

PbStatus launch_wet(const float *rlsp, cudaTextureObject_t tex, const RayCells &rec,
                    const PbGrid &g, const PbBeamGeom *beams, int n_beams, float *raw,
                    float *wet, int *status, cudaStream_t st)
{
    BeamGeomSet bs;
    for (int b = 0; b < n_beams; ++b) bs.b[b] = beams[b];
    SmoothSet ss;
    smooth_set(g, beams, n_beams, ss);
    const int64_t bx = (g.nx + 7) / 8, by = (g.ny + 3) / 4;
    const int64_t planes = (int64_t)((g.nz + 3) / 4) * n_beams, bricks = bx * by * planes;
    if (bricks > INT32_MAX) return set_error(PB_ERR_INVALID, "grid too large");
    const int64_t limit = 65535;   // of a launch's y and z
    // about `blocks` blocks: all of a plane's bricks, every so many planes
    auto many = [&](int64_t blocks) {
        const int64_t z = std::min(std::max<int64_t>((blocks + bx * by - 1) / (bx * by), 1), planes);
        return dim3((unsigned)bx, (unsigned)std::min(by, limit), (unsigned)std::min(z, limit));
    };
    const bool each = bricks <= kEachBricks && by <= limit && planes <= limit;
    const dim3 all((unsigned)bx, (unsigned)by, (unsigned)planes);
    const int cap = ray_step_cap(g);
    const dim3 some = many((bricks + kBricksPerBlock - 1) / kBricksPerBlock);
    if (tex && each)
        k_raytrace<true, true><<<all, 128, 0, st>>>(rlsp, tex, rec, g, bs, n_beams, cap, raw, status);
    else if (tex)
        k_raytrace<true, false><<<some, 128, 0, st>>>(rlsp, tex, rec, g, bs, n_beams, cap, raw,
                                                      status);
    else
        k_raytrace<false, false><<<each ? all : some, 128, 0, st>>>(rlsp, tex, rec, g, bs, n_beams,
                                                                    cap, raw, status);
    PbStatus s = check_launch("k_raytrace");
    if (s != PB_OK) return s;
    SmoothStarts at;
    at.n = n_beams;
    const bool few = (int64_t)g.nx * g.ny * g.nz * n_beams < kSmoothFew;
    long long blocks = 0;
    for (int b = 0; b < n_beams; ++b) {
        at.start[b] = (unsigned)blocks;
        const SmoothBox X = few ? smooth_box<2>(g, ss.b[b].margin) : smooth_box<4>(g, ss.b[b].margin);
        blocks += X.inner + X.shell;
        if (blocks > INT32_MAX) return set_error(PB_ERR_INVALID, "grid too large");
    }
    auto kernel = ss.b[0].pow2 ? (few ? k_smooth<true, 2> : k_smooth<true, 4>)
                               : (few ? k_smooth<false, 2> : k_smooth<false, 4>);
    kernel<<<(unsigned)blocks, 128, 0, st>>>(raw, g, bs, ss, at, wet);
    return check_launch("k_smooth");
}

void smooth_table_host(const PbGrid &g, const PbBeamGeom *beams, int n_beams, int beam,
                       int *off, float *hh, unsigned *tmask, int *margin)
{
    SmoothSet ss;
    smooth_set(g, beams, n_beams, ss);
    const SmoothBeam &T = ss.b[beam];
    memcpy(off, T.off, sizeof(T.off));
    memcpy(hh, T.hh, sizeof(T.hh));
    memcpy(tmask, T.tmask, sizeof(T.tmask));
    memcpy(margin, T.margin, sizeof(T.margin));
}

size_t batch_wet_size() { return sizeof(BatchWet); }

// Bricks below which a batch's smoothing takes two voxels a thread.
long long batch_wet_few() { return kSmoothFew / 128; }

// Fills the batch records of one plan's beams; returns the bricks they use.
// few: for the smoothing with two voxels a thread.
long long fill_batch_wet(void *items_host, int first, const PbGrid &g, const PbBeamGeom *beams,
                         int n_beams, const float *rlsp, cudaTextureObject_t tex,
                         const RayCells &rec, float *raw, float *wet, long long brick_start,
                         bool few)
{
    BatchWet *W = static_cast<BatchWet *>(items_host) + first;
    SmoothSet ss;
    smooth_set(g, beams, n_beams, ss);
    const int64_t V = (int64_t)g.nx * g.ny * g.nz;
    const int bx = (g.nx + 7) / 8, by = (g.ny + 3) / 4, bz = (g.nz + 3) / 4;
    long long start = brick_start;
    for (int b = 0; b < n_beams; ++b) {
        BatchWet &w = W[b];
        w.g = g;
        w.geom = beams[b];
        w.rlsp = rlsp;
        w.tex = tex;
        w.rec = rec;
        w.raw = raw + b * V;
        w.wet = wet + b * V;
        w.sm = ss.b[b];
        w.cap = ray_step_cap(g);
        w.bx = bx;
        w.by = by;
        w.bz = bz;
        w.brick_start = start;
        const SmoothBox X = few ? smooth_box<2>(g, w.sm.margin) : smooth_box<4>(g, w.sm.margin);
        w.smooth_blocks = X.inner + X.shell;
        // both launches go by these starts
        start += std::max((long long)bx * by * bz, w.smooth_blocks);
    }
    return start - brick_start;
}

PbStatus launch_wet_batch(const void *items_dev, int n_items, long long n_bricks, int *status,
                          cudaStream_t st)
{
    if (n_bricks <= 0) return PB_OK;
    if (n_bricks > 0x7fffffffLL) return set_error(PB_ERR_INVALID, "batch too large");
    const BatchWet *I = static_cast<const BatchWet *>(items_dev);
    k_raytrace_batch<<<(unsigned)n_bricks, 128, 0, st>>>(I, n_items, status);
    PbStatus s = check_launch("k_raytrace_batch");
    if (s != PB_OK) return s;
    if (n_bricks < batch_wet_few())
        k_smooth_batch<2><<<(unsigned)n_bricks, 128, 0, st>>>(I, n_items);
    else
        k_smooth_batch<4><<<(unsigned)n_bricks, 128, 0, st>>>(I, n_items);
    return check_launch("k_smooth_batch");
}

// Cells of a volume with border 0: cell (ci, cj, ck) holds the 2x2x2
// texels with base (ci-1, cj-1, ck-1) -- the texels a linear fetch reads
// for a coordinate inside it.  A cell is flat when its eight texels are
// equal.  Two adjacent flat cells share texels, so a connected flat region
// has one value.
constexpr int kRunCap = 15;   // largest stored distance (cells)
constexpr int kFlagPad = 16;  // zero bytes before and after each row of flat flags

// Row length (bytes) of the flat flags: cell_row with kFlagPad bytes on each side.
__host__ __device__ __forceinline__ int flag_row(int nx) { return cell_row(nx) + 2 * kFlagPad; }

// Pass 0: the quads (where there are any), and the x distance pass's input:
// kRunCap where a cell is flat (its eight texels equal), else 0, in rows with
// kFlagPad zero bytes before and after (flag_row).  A thread takes kFlatRows
// rows of one (ci, ck) column and keeps each row's four texels for the next
// cell, so that a texel pair is loaded twice per row (its x and z neighbours)
// instead of eight times.  256x256x160: 56 us with the quads' 170 MB, against 117 us
// for one cell a thread and a 4-byte value per cell.
constexpr int kFlatRows = 8;
__global__ void __launch_bounds__(256)
k_cell_flat(const float *__restrict__ rho, PbGrid g, float4 *__restrict__ quad,
            unsigned char *__restrict__ flag)
{
    const int cx = g.nx + 1, cy = g.ny + 1, cz = g.nz + 1;
    const int col = blockIdx.x * 256 + threadIdx.x;   // (ci, ck)
    const bool live = col < cx * cz;
    const int ci = col % cx, ck = col / cx;
    const bool x0 = ci > 0, x1 = ci < g.nx, z0 = ck > 0, z1 = ck < g.nz;
    const int64_t plane = (int64_t)g.nx * g.ny;
    const int r0 = blockIdx.y * kFlatRows;             // first quad row
    auto row = [&](int r) {                            // quad row r: texel row r - 1
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live && r > 0 && r <= g.ny) {
            const float *p = rho + plane * (ck - 1) + (int64_t)g.nx * (r - 1) + ci - 1;
            if (x0 && z0) v.x = __ldg(p);
            if (x0 && z1) v.y = __ldg(p + plane);
            if (x1 && z0) v.z = __ldg(p + 1);
            if (x1 && z1) v.w = __ldg(p + 1 + plane);
        }
        return v;
    };
    float4 a = row(r0);
#pragma unroll
    for (int m = 0; m < kFlatRows; ++m) {
        const int r = r0 + m;
        if (r > cy) break;                             // rows 0 .. ny + 1
        if (live && quad) quad[(int64_t)cx * (r + (int64_t)(cy + 1) * ck) + ci] = a;
        if (r == cy) break;                            // the last row starts no cell
        const float4 b = row(r + 1);
        const float v = a.x;
        const bool f = a.y == v && a.z == v && a.w == v && b.x == v && b.y == v && b.z == v &&
                       b.w == v;                       // false for NaN
        if (live)
            flag[((int64_t)cy * ck + r) * flag_row(g.nx) + kFlagPad + ci] =
                f ? (unsigned char)kRunCap : 0;
        a = b;
    }
}

// Separable L-infinity distance to the nearest non-flat cell, capped at
// kRunCap: min over |k| <= kRunCap of max(|k|, d(pos + k)), a cell outside
// the grid counting as non-flat (d = 0).  The distances are bytes in rows
// padded to a multiple of 4 cells (cell_row); the x pass reads the flat flags
// (kRunCap or 0) in rows with kFlagPad zero bytes on each side (flag_row).
// A thread takes words of four cells, the even and the odd cells apart as
// 16-bit pairs, whose minimum and maximum are one instruction each (the
// byte-wise ones are a dozen; the passes were bound by them), and in y and z
// kDistRun words along the axis, which share their taps in registers.  Measured
// on the 257x257x161 cells of a 256x256x160 volume: x 69 -> 28 us, y 98 -> 26 us,
// z with a texture's records 108 + 32 -> 65 us.
__device__ __forceinline__ unsigned int dist_tap(unsigned int best, int k, unsigned int below,
                                                 unsigned int above)
{
    return __vminu2(best, __vmaxu2((unsigned int)k * 0x00010001u, __vminu2(below, above)));
}

constexpr unsigned int kEven = 0x00FF00FFu;   // the bytes of cells 0 and 2 of a word

__global__ void __launch_bounds__(256)
k_cell_dist_x(PbGrid g, const unsigned char *__restrict__ flag, unsigned int *__restrict__ dout)
{
    static_assert(kFlagPad > kRunCap && kFlagPad % 4 == 0, "every tap inside the padded row");
    constexpr int kWords = (kFlagPad + kRunCap) / 4 + 2;   // words w .. w + kWords - 1
    const int cy = g.ny + 1, cz = g.nz + 1, words = cell_row(g.nx) / 4, frow = flag_row(g.nx);
    const int64_t n = (int64_t)words * cy * cz;
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int w = (int)(c % words);
    const int64_t line = c / words;
    // cells 4w - kRunCap .. 4w + 3 + kRunCap: flag bytes from
    // 4w + kFlagPad - kRunCap on, within the row's words from w (the last
    // word read ends at most at the row's last byte)
    const unsigned int *src = reinterpret_cast<const unsigned int *>(flag + line * frow + 4 * w);
    unsigned int E[kWords], O[kWords];   // cells 4j, 4j + 2 and 4j + 1, 4j + 3
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
        const unsigned int v = __ldg(src + j);
        E[j] = v & kEven;
        O[j] = (v >> 8) & kEven;
    }
    auto pair = [&](int p) {             // cells p and p + 2 of the window
        const unsigned int *s = (p & 1) ? O : E;
        const int j = p >> 2;
        return (p & 2) ? __funnelshift_r(s[j], s[j + 1], 16) : s[j];
    };
    unsigned int even = pair(kFlagPad), odd = pair(kFlagPad + 1);
#pragma unroll
    for (int k = 1; k <= kRunCap; ++k) {
        even = dist_tap(even, k, pair(kFlagPad - k), pair(kFlagPad + k));
        odd = dist_tap(odd, k, pair(kFlagPad + 1 - k), pair(kFlagPad + 1 + k));
    }
    dout[c] = even | (odd << 8);
}

constexpr int kDistRun = 8;

// The z pass, the last, also writes a texture's records.
template <int AXIS>
__global__ void __launch_bounds__(128)
k_cell_dist4(PbGrid g, const unsigned int *__restrict__ din, unsigned int *__restrict__ dout,
             const float *__restrict__ rho = nullptr, float2 *__restrict__ cell = nullptr)
{
    static_assert(AXIS == 1 || AXIS == 2, "y or z");
    const int cy = g.ny + 1, cz = g.nz + 1, words = cell_row(g.nx) / 4;
    const int len = AXIS == 1 ? cy : cz, other = AXIS == 1 ? cz : cy;
    const int64_t stride = AXIS == 1 ? (int64_t)words : (int64_t)words * cy;
    const int64_t across = AXIS == 1 ? (int64_t)words * cy : (int64_t)words;
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int w = (int)(q % words), o = (int)(q / words % other);
    const int p0 = (int)(q / ((int64_t)words * other)) * kDistRun;
    if (p0 >= len) return;
    const int64_t base = w + across * o;
    constexpr int kTaps = kDistRun + 2 * kRunCap;
    unsigned int E[kTaps], O[kTaps];
#pragma unroll
    for (int j = 0; j < kTaps; ++j) {
        const int p = p0 + j - kRunCap;
        // outside the grid counts as non-flat (distance 0)
        const unsigned int v = p >= 0 && p < len ? __ldg(din + base + stride * p) : 0u;
        E[j] = v & kEven;
        O[j] = (v >> 8) & kEven;
    }
#pragma unroll
    for (int m = 0; m < kDistRun; ++m) {
        const int p = p0 + m, j = m + kRunCap;
        if (p >= len) break;
        unsigned int even = E[j], odd = O[j];
#pragma unroll
        for (int k = 1; k <= kRunCap; ++k) {
            even = dist_tap(even, k, E[j - k], E[j + k]);
            odd = dist_tap(odd, k, O[j - k], O[j + k]);
        }
        const unsigned int best = even | (odd << 8);
        dout[base + stride * p] = best;
        if (AXIS == 2 && cell) {
            // a flat cell's value from its texel inside the grid
            const int cx = g.nx + 1;
            const float *row = rho + (int64_t)g.nx * (min(o, g.ny - 1) +
                                                      (int64_t)g.ny * min(p, g.nz - 1));
            float2 *out = cell + (int64_t)cx * (o + (int64_t)cy * p);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int ci = 4 * w + i;
                const unsigned int d = (best >> (8 * i)) & 255u;
                if (ci < cx)
                    out[ci] = d ? make_float2(__ldg(row + min(ci, g.nx - 1)), (float)d)
                                : make_float2(0.0f, 0.0f);
            }
        }
    }
}

// 3-D texture over an RLSP volume: float channel, linear filter, border 0,
// unnormalised coordinates (TextureClasses.cu:14-41), and the cell records
// the ray trace uses to take runs of samples in flat regions at once.
struct RlspTexture {
    cudaArray_t arr = nullptr;
    cudaTextureObject_t tex = 0;
    // The cell records (RayCells) and the passes' work arrays, in one allocation,
    // or none of them: no memory.
    unsigned char *block = nullptr;
    float2 *cell = nullptr;           // with a texture
    float4 *quad = nullptr;           // without
    unsigned char *d0 = nullptr, *d1 = nullptr;  // distances, and the passes' other buffer
    unsigned char *flag = nullptr;    // work: flat flags (zero-padded rows)
    int nx = 0, ny = 0, nz = 0;
};

static PbStatus texture_fill(RlspTexture *t, const float *rlsp, cudaStream_t st)
{
    cudaMemcpy3DParms p{};
    p.srcPtr = make_cudaPitchedPtr(const_cast<float *>(rlsp), sizeof(float) * (size_t)t->nx, t->nx,
                                   t->ny);
    p.dstArray = t->arr;
    p.extent = make_cudaExtent(t->nx, t->ny, t->nz);
    p.kind = cudaMemcpyDeviceToDevice;
    if (t->arr) {
        const PbStatus s = check_cuda(cudaMemcpy3DAsync(&p, st), "cudaMemcpy3DAsync");
        if (s != PB_OK) return s;
    }
    const PbGrid g{t->nx, t->ny, t->nz, 1.0f};
    if (!t->block) return PB_OK;
    const int64_t words = cell_row(t->nx) / 4, cy = t->ny + 1, cz = t->nz + 1;
    auto blocks = [](int64_t threads, int block) { return (unsigned)((threads + block - 1) / block); };
    auto runs = [](int64_t n) { return (n + kDistRun - 1) / kDistRun; };
    const dim3 cols((unsigned)(((t->nx + 1) * (int64_t)(t->nz + 1) + 255) / 256),
                    (unsigned)((t->ny + 2 + kFlatRows - 1) / kFlatRows));
    k_cell_flat<<<cols, 256, 0, st>>>(rlsp, g, t->quad, t->flag);
    k_cell_dist_x<<<blocks(words * cy * cz, 256), 256, 0, st>>>(
        g, t->flag, reinterpret_cast<unsigned int *>(t->d0));
    k_cell_dist4<1><<<blocks(words * cz * runs(cy), 128), 128, 0, st>>>(
        g, reinterpret_cast<const unsigned int *>(t->d0),
        reinterpret_cast<unsigned int *>(t->d1));
    k_cell_dist4<2><<<blocks(words * cy * runs(cz), 128), 128, 0, st>>>(
        g, reinterpret_cast<const unsigned int *>(t->d1),
        reinterpret_cast<unsigned int *>(t->d0), rlsp, t->cell);
    return check_launch("cell records");
}

static void texture_free(RlspTexture *t)
{
    if (t->tex) cudaDestroyTextureObject(t->tex);
    if (t->arr) cudaFreeArray(t->arr);
    cudaFree(t->block);
    delete t;
}

// with_texture false: the cell records only, for exact-trilinear sampling.
PbStatus texture_create(const float *rlsp, const PbGrid &g, uint64_t *out, cudaStream_t st,
                        bool with_texture)
{
    const size_t ncell = (size_t)(g.nx + 1) * (g.ny + 1) * (g.nz + 1);
    if (ncell > (size_t)INT32_MAX)
        return set_error(PB_ERR_INVALID, "grid too large for a texture (%zu cells)", ncell);
    RlspTexture *t = new (std::nothrow) RlspTexture;
    if (!t) return set_error(PB_ERR_NOMEM, "host allocation failed");
    t->nx = g.nx;
    t->ny = g.ny;
    t->nz = g.nz;
    cudaChannelFormatDesc ch = cudaCreateChannelDesc<float>();
    cudaExtent ext = make_cudaExtent(g.nx, g.ny, g.nz);
    PbStatus s = PB_OK;
    if (with_texture)
        s = check_cuda(cudaMalloc3DArray(&t->arr, &ch, ext, cudaArrayDefault),
                       "cudaMalloc3DArray");
    // the records of a grid that leaves no memory for them are left out: the
    // ray trace then takes every sample from the texture or the volume
    const size_t nquad = (size_t)(g.nx + 1) * (g.ny + 2) * (g.nz + 1);
    // distance passes: rows padded to 4 cells (32-bit words)
    const size_t npad = (size_t)cell_row(g.nx) * (g.ny + 1) * (g.nz + 1);
    const size_t nflag = (size_t)flag_row(g.nx) * (g.ny + 1) * (g.nz + 1);
    size_t bytes = 0;
    auto part = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t at_cells = part(with_texture ? sizeof(float2) * ncell : sizeof(float4) * nquad);
    const size_t at_d0 = part(npad), at_d1 = part(npad), at_flag = part(nflag);
    if (s == PB_OK && cudaMalloc(&t->block, bytes) != cudaSuccess) {
        t->block = nullptr;
        cudaGetLastError();
    }
    if (s == PB_OK && t->block) {
        if (with_texture) t->cell = reinterpret_cast<float2 *>(t->block + at_cells);
        else t->quad = reinterpret_cast<float4 *>(t->block + at_cells);
        t->d0 = t->block + at_d0;
        t->d1 = t->block + at_d1;
        t->flag = t->block + at_flag;
        // flat flags: the padding bytes stay zero, the cells are rewritten by
        // every fill
        s = check_cuda(cudaMemsetAsync(t->flag, 0, nflag, st), "cudaMemsetAsync");
    }
    if (s == PB_OK && with_texture) {
        cudaResourceDesc rd{};
        rd.resType = cudaResourceTypeArray;
        rd.res.array.array = t->arr;
        cudaTextureDesc td{};
        td.addressMode[0] = td.addressMode[1] = td.addressMode[2] = cudaAddressModeBorder;
        td.filterMode = cudaFilterModeLinear;
        td.readMode = cudaReadModeElementType;
        td.normalizedCoords = 0;
        s = check_cuda(cudaCreateTextureObject(&t->tex, &rd, &td, nullptr),
                       "cudaCreateTextureObject");
    }
    if (s == PB_OK) s = texture_fill(t, rlsp, st);
    if (s != PB_OK) {
        texture_free(t);
        return s;
    }
    *out = reinterpret_cast<uint64_t>(t);
    return PB_OK;
}

PbStatus texture_update(uint64_t h, const float *rlsp, cudaStream_t st)
{
    return texture_fill(reinterpret_cast<RlspTexture *>(h), rlsp, st);
}

bool texture_matches(uint64_t h, const PbGrid &g)
{
    const RlspTexture *t = reinterpret_cast<const RlspTexture *>(h);
    return t && t->nx == g.nx && t->ny == g.ny && t->nz == g.nz;
}

bool texture_samples(uint64_t h)
{
    return h && reinterpret_cast<const RlspTexture *>(h)->tex != 0;
}

cudaTextureObject_t texture_object(uint64_t h)
{
    return h ? reinterpret_cast<const RlspTexture *>(h)->tex : 0;
}

RayCells texture_cells(uint64_t h)
{
    const RlspTexture *t = reinterpret_cast<const RlspTexture *>(h);
    return t && t->block ? RayCells{t->quad, t->d0, t->cell} : RayCells{};
}

void texture_destroy(uint64_t h)
{
    RlspTexture *t = reinterpret_cast<RlspTexture *>(h);
    if (t) texture_free(t);
}

}  // namespace pb
