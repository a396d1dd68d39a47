// USFFT Radon transform (tomography operator) for sm_100a.
//
// Replaces class radonusfft of the reference (src/cuda/radonusfft.cu:1-144,
// kernels src/include/kernels.cuh:5-216).  Same mathematics, different
// machinery:
//
//  forward  R f   (radonusfft.cu:54-92)
//    K1 k_fwd_rows    pad2 edge replication + circ mask + deapodisation 1/phi
//                     + centring sign, zero-pad to 2N, row FFT (the N rows
//                     that are non-zero)                       [smem FFT]
//    K2 k_fwd_cols    column FFT of length 2N (zero rows implicit) with the
//                     post-FFT centring sign folded in          [smem FFT]
//    K3a k_fwd_gather_pts  window gather at the polar points
//                     (kernels.cuh:97-126), one 8-slice lane group per point
//    K3b k_fwd_lines  1-D centred inverse FFT along the detector, crop n of N
//  adjoint  R* g  (radonusfft.cu:94-139)
//    A1 k_adj_lines     edge-replicating pad, centred 1-D FFT, written for all
//                       slices as lines[point][slice]
//    A2 k_adj_colgather one block per (grid column, 16 slices): every cell of
//                       the column sums, in a fixed order, w * g over the polar
//                       points whose kernel window covers it (cell -> (point,
//                       weight) lists built once at setobj; no float atomics,
//                       no halo, no fold), then the column inverse FFT runs in
//                       the same block and only the n rows that survive the
//                       final crop are written
//    A4 k_adj_rows      row inverse FFT + centring sign + 1/phi + circ + crop
//
// The forward processes slices in chunks of ZC = 8 with slice-minor
// intermediates ([..][ZC]) so every gather tap and every row of the column
// kernel is a contiguous 64-byte segment, and a chunk's intermediates
// (N*2N + (2N)^2 complex per slice) stay well inside L2.  The adjoint keeps
// slice-minor full-volume buffers ([..][nzp], nzp = nz rounded up to 16).
//
// Gridding window.  The reference interpolates between the 2N grid and the
// polar points with a Gaussian of half-width M = 7 (15 x 15 taps,
// kernels.cuh:97-158) and divides the slice by its transform phi; the result
// approximates the exact non-uniform DFT of the padded slice.  Here the same
// transform is evaluated with a Kaiser-Bessel window of 8 x 8 cells and its
// own transform as the deapodisation: 64 taps instead of 225.  On the same 2x
// grid its error against the exact sum is smaller than the Gaussian's (per
// axis, rms over offsets and the slice's disc: 4 to 5e-8 against 1.06e-7, at
// most 8.3e-7 against 1.05e-6), and its deapodisation amplifies rounding less
// (2.8 against 5.6 per axis at the slice's edge): on white noise at 256 wide
// the forward is 1.6e-7 from the sum in 64 bits, the Gaussian's was 7.7e-7.
// The forced half-width 4 keeps its Gaussian (9 x 9 taps): its 1.1e-5 error is
// what that option is for.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "pt_common.cuh"
#include "pt_fft.cuh"

namespace {

constexpr int ZC = 8;   // slices per chunk (slice-minor lanes)
constexpr int RSETS = 4;   // forward chunk buffer sets (chunks in flight at most)
constexpr int CK = 2;   // grid columns per block in the column kernels
constexpr int ZH = 4;   // slices per block of the forward's column kernel
constexpr double PI_REF = 3.1415926535;  // kernels.cuh:1

// circ, kernels.cuh:160-172 (r = 1.0f/N); evaluated without FMA contraction so
// that it equals the float32 expression (4x*x + 4y*y) < 1 - r exactly.
__device__ __forceinline__ float circ_keep(int tx, int ty, int N)
{
    const float x = (float)(tx - N / 2) / (float)N;
    const float y = (float)(ty - N / 2) / (float)N;
    const float lhs = __fadd_rn(__fmul_rn(__fmul_rn(4.f, x), x), __fmul_rn(__fmul_rn(4.f, y), y));
    const float r = 1.0f / (float)N;
    return lhs < 1.f - r ? 1.f : 0.f;
}

// phi, kernels.cuh:12 and :23 (same expression as the reference), for the Gaussian window
__device__ __forceinline__ float deapod(int tx, int ty, int N, float mu)
{
    return __expf(-mu * (tx - N / 2) * (tx - N / 2) - mu * (ty - N / 2) * (ty - N / 2));
}

// fac[ty][tx] = (-1)^(tx + ty) circ / (the window's transform) on the N x N
// padded slice: the factor that unpaddivphi / divphi and circ apply
// (kernels.cuh:5-37, 160-172) with the centring sign of the 2N grid
// (kernels.cuh:28-37), evaluated once per handle; the row passes multiply by it.  inv1 (Kaiser-
// Bessel): 1 / transform per axis; null (Gaussian): circ / phi / (4 N^2) with
// the expressions above.
__global__ void k_deap_table(float *__restrict__ fac, int N, float mu, const double *__restrict__ inv1)
{
    const int tx = blockIdx.x * blockDim.x + threadIdx.x, ty = blockIdx.y;
    if (tx >= N) return;
    const float den = (float)(4 * N * N);
    const float f = inv1 ? circ_keep(tx, ty, N) * (float)(inv1[tx] * inv1[ty])
                         : circ_keep(tx, ty, N) / deapod(tx, ty, N, mu) / den;
    fac[(size_t)ty * N + tx] = ((tx + ty) & 1) ? -f : f;
}

// ---- gridding window -----------------------------------------------------------
constexpr int WKB = 8, WGAUSS = 9;   // cells per axis: Kaiser-Bessel (default), Gaussian of half-width 4
template <int W>
constexpr int win_left() { return W == WKB ? WKB / 2 - 1 : WGAUSS / 2; }   // first cell: floor(2N x) - win_left
// the rms error is flat about its minimum: 3.9e-8 to 4.9e-8 from 2.30 W to 2.36 W
constexpr double KB_BETA = 2.35 * WKB;

// wtab[p][0..W-1], [W..2W-1]: the window's values in x and y at the W cells
// of point p's window (first cell floor(2N x) - win_left).  Kaiser-Bessel
// I0(beta sqrt(1 - (2 d / W)^2)) / I0(beta), d the distance in cells, in
// double; Gaussian with the reference's float expression (kernels.cuh:115-119).
template <int W>
__global__ void k_window(const float *__restrict__ xt, const float *__restrict__ yt, float *__restrict__ wtab, int npts,
                         int G, float a, double i0_beta)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= npts * 2 * W) return;
    const int p = e / (2 * W), i = e % (2 * W), j = i % W;
    const float c = i < W ? xt[p] : yt[p];
    const int first = (int)floorf((float)G * c) - win_left<W>();
    if (W == WKB) {
        const double t = ((double)(first + j) - (double)G * (double)c) * (2.0 / W);
        wtab[e] = (float)(cyl_bessel_i0(KB_BETA * sqrt(fmax(0.0, 1.0 - t * t))) / i0_beta);
    } else {
        const float w = (float)(first + j) / (float)G - c;
        wtab[e] = __expf(-a * (w * w));
    }
}

// The forward gather's record of a point, in visiting order (perm; null: in
// point order) (six float4):
// floats 0..9 the x weights of the five column pairs that cover the window (0
// for the columns outside it), 10..18 the y weights times the sample's scale
// pre, 20 the point's index, 21 and 22 its
// window's first row and column pair on the haloed grid, 23 whether the window
// needs all five pairs (an even-sized window that starts on a pair covers four).
constexpr int REC4 = 6;
constexpr int NPAIR = 5;
static_assert(WKB <= 9 && WGAUSS <= 9, "a window spans at most five column pairs and nine rows");
template <int W>
__global__ void k_point_records(const int *__restrict__ perm, const int *__restrict__ org,
                                const float *__restrict__ wtab, float *__restrict__ rec, int npts, float pre)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npts) return;
    const int p = perm ? perm[i] : i;
    const int ox = org[2 * p], oy = org[2 * p + 1], odd = ox & 1;
    const float *wx = wtab + (size_t)p * 2 * W, *wy = wx + W;
    float *r = rec + (size_t)i * REC4 * 4;
    for (int j = 0; j < 2 * NPAIR; ++j) r[j] = (j >= odd && j - odd < W) ? wx[j - odd] : 0.f;
    for (int j = 0; j < 9; ++j) r[10 + j] = j < W ? pre * wy[j] : 0.f;
    r[19] = 0.f;
    r[20] = __int_as_float(p);
    r[21] = __int_as_float(oy);
    r[22] = __int_as_float(ox / 2);
    r[23] = __int_as_float(W + odd > 2 * (NPAIR - 1));
}

// ---- geometry: takexy, kernels.cuh:84-95 (identical expression) -----------
__global__ void k_takexy(float *x, float *y, const float *theta, int N, int ntheta)
{
    const int tx = blockIdx.x * blockDim.x + threadIdx.x;
    const int ty = blockIdx.y;
    if (tx >= N || ty >= ntheta) return;
    float xv = (tx - N / 2) / (float)N * __cosf(theta[ty]);
    float yv = -(tx - N / 2) / (float)N * __sinf(theta[ty]);
    if (xv >= 0.5f) xv = 0.5f - 1e-5;
    if (yv >= 0.5f) yv = 0.5f - 1e-5;
    x[tx + ty * N] = xv;
    y[tx + ty * N] = yv;
}

// Resident blocks that the two-round kernels of length G are compiled for: 80
// registers a thread at 768 and below without spills (256^3 forward 1.42 ->
// 1.36 ms against two blocks of 128), one block at 1536 (48 x 32 values).
template <int G>
constexpr int row_blocks() { return G > 768 ? 1 : G > 384 ? 3 : 2; }

// The forward's four kernels work on up to RSETS chunks of ZC slices per
// launch, one per buffer set: the chunk is the last grid dimension, `set` the
// distance of two sets in float2.

// ---- K1: pad2 + circ + divphi + fftshiftc + row FFT ------------------------
// The block's ZC slices are interleaved transforms (lane q = slice), so the
// output rows of the slice-minor buffer are contiguous.  The non-zero inputs
// X = N/2 .. 3N/2 - 1 are the R1/2 middle rows i1 of the R1 x R2 split; the
// table tw holds W^(i2 k1) i^k1: the shift of those rows by R1/4 gives
// (-i)^k1, the centring sign of the outputs (-1)^k1.
// The object is read and the transform written by the threads that compute it,
// with one trip through shared memory between: 12.4 us for 8 slices at 256
// wide (four Stockham passes and two staging copies: 21.7 us).
template <int G>
__global__ void __launch_bounds__(ptfft::Exchange<G, ZC>::NT, row_blocks<G>())
    k_fwd_rows(const float2 *__restrict__ u, float2 *__restrict__ rbuf, size_t set, int nz, int z0,
               const float *__restrict__ fac, const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<G, ZC>;
    constexpr int N = G / 2, n = G / 3, R1 = E::R1, R2 = E::R2;
    constexpr int c0 = N / 6, c1 = 5 * N / 6 - 1;
    extern __shared__ float2 sm[];
    const int y = blockIdx.x;
    const int q = threadIdx.x % ZC, b = threadIdx.x / ZC;
    if (b < R2) {
        const int z = z0 + blockIdx.y * ZC + q;
        float2 in[R1 / 2];
        if (z < nz) {
            const float2 *src = u + ((size_t)z * n + (min(max(y, c0), c1) - c0)) * n;
            const float *f = fac + (size_t)y * N;
#pragma unroll
            for (int a = 0; a < R1 / 2; ++a) {
                const int tx = a * R2 + b;
                in[a] = __ldg(&f[tx]) * src[min(max(tx, c0), c1) - c0];
            }
        } else {
#pragma unroll
            for (int a = 0; a < R1 / 2; ++a) in[a] = czero();
        }
        float2 v[R1];
        ptfft::dft_half<R1, -1>(in, v);
        ptfft::twiddle_pairs<R1, R2>(v, b, tw);
        E::put(sm, v, b, q);
    }
    __syncthreads();
    if (b < R1) {
        float2 w[R2];
        E::get(sm, w, b, q);
        ptfft::Dft<R2, -1, true>::run(w);
        float2 *dst = rbuf + blockIdx.y * set + ((size_t)y * G + b) * ZC + q;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) dst[k2 * R1 * ZC] = w[k2];
    }
}

// The forward's Fourier grid carries a halo, like the reference's (G+2M)^2
// grid (radonusfft.cu:16, wrap in kernels.cuh:50-65): rows 0..GH_ROWS-1 are
// repeated after row G-1 and column pairs 0..GH_PAIRS-1 after pair G/2-1, so
// every gather window is a plain rectangle (no index wraps) addressed from one
// base pointer.  Layout [G + GH_ROWS][G/2 + GH_PAIRS][ZC][2].
constexpr int GH_ROWS = 8;    // the largest window (9 cells) minus one
constexpr int GH_PAIRS = NPAIR - 1;

// ---- K2: column FFT of the 2N grid ---------------------------------------------
// The block's CK columns x ZH slices are NF interleaved transforms, ordered as
// the grid's column pairs hold them (q = slice * CK + column), so both the
// row-FFT buffer and the grid are touched in whole 32- or 64-byte runs.  Rows
// outside N/2 .. 3N/2 - 1 are zero; the table is K1's.
// 17.5 us for 8 slices at 256 wide (Stockham passes: 30.6 us).
template <int G>
__global__ void __launch_bounds__(ptfft::Exchange<G, CK * ZH>::NT, row_blocks<G>())
    k_fwd_cols(const float2 *__restrict__ rbuf, float2 *__restrict__ fg, size_t set, const float4 *__restrict__ tw)
{
    constexpr int NF = CK * ZH;
    using E = ptfft::Exchange<G, NF>;
    constexpr int R1 = E::R1, R2 = E::R2;
    static_assert(CK == 2, "the grid layout pairs two columns");
    extern __shared__ float2 sm[];
    const int pr = blockIdx.x, zh = blockIdx.y * ZH;
    const int q = threadIdx.x % NF, b = threadIdx.x / NF;
    if (b < R2) {
        const float2 *src = rbuf + blockIdx.z * set + ((size_t)b * G + pr * CK + q % CK) * ZC + zh + q / CK;
        float2 in[R1 / 2];
#pragma unroll
        for (int a = 0; a < R1 / 2; ++a) in[a] = src[(size_t)a * R2 * G * ZC];
        float2 v[R1];
        ptfft::dft_half<R1, -1>(in, v);
        ptfft::twiddle_pairs<R1, R2>(v, b, tw);
        E::put(sm, v, b, q);
    }
    __syncthreads();
    if (b < R1) {
        float2 w[R2];
        E::get(sm, w, b, q);
        ptfft::Dft<R2, -1, true>::run(w);
        // column-pair layout [ky][kx/2][z][kx&1], plus the halo copies (rows <
        // GH_ROWS again at G + ky, pairs < GH_PAIRS again at G/2 + pair)
        constexpr size_t PS = G / 2 + GH_PAIRS;
        float2 *dst = fg + blockIdx.z * set + (size_t)pr * (CK * ZC) + zh * CK + q;
        const bool edge = pr < GH_PAIRS;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) {
            const int ky = b + R1 * k2;
            dst[ky * PS * (CK * ZC)] = w[k2];
            if (edge) dst[(ky * PS + G / 2) * (CK * ZC)] = w[k2];
            if (R1 * k2 < GH_ROWS && ky < GH_ROWS) {
                dst[(ky + G) * PS * (CK * ZC)] = w[k2];
                if (edge) dst[((ky + G) * PS + G / 2) * (CK * ZC)] = w[k2];
            }
        }
    }
}

// ---- K3a: gather only, many blocks --------------------------------------------
// block = GPB points x ZC slice lanes.  The grid is in column-pair layout, so
// a lane reads its slice's value at two neighbouring window columns with one
// 16-byte load (the point's 8 lanes read one 128-byte line).  The window's
// columns are covered by four or five column pairs; a covered column outside
// the window has weight 0.  Writes the gathered, 1/N-scaled
// samples to lines[(theta N + k) ZC + z].  Points are visited in the order of
// `perm` (built at setobj): sorted by the 16 x 16-cell grid tile their window
// starts in, then by the parity of its first column, so the points of a block
// read overlapping windows and a warp's four points mostly agree on the number
// of pairs.  The order changes no arithmetic.
//
// Bound by shared-memory reads: W (W + 1) / 2 16-byte loads per point and
// slice on average (36 of the 8-cell window; the 15-cell Gaussian took 120),
// against 4 multiply-adds each.  An 8-slice chunk at 256 wide and 384 angles
// takes 33 us; with the Gaussian's taps it took 88 us (1060 against 2814 us
// for the 32 chunks of 256 slices).
constexpr int GPB = 32;
constexpr int GTILE = 16;   // grid cells per tile edge of the visiting order

// One point's gather: base is the window's first pair on this lane's slice,
// `pitch` the float4 distance of two rows, r the point's record.
template <int W, typename Load>
__device__ __forceinline__ float2 window_sum(const float4 *__restrict__ base, size_t pitch, const float4 *__restrict__ r,
                                             Load load)
{
    const float4 a0 = r[0], a1 = r[1], a2 = r[2], a3 = r[3], a4 = r[4], a5 = r[5];
    const float wx[2 * NPAIR] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w, a2.x, a2.y};
    const float wy[9] = {a2.z, a2.w, a3.x, a3.y, a3.z, a3.w, a4.x, a4.y, a4.z};
    float2 acc = czero();
    auto rows = [&](auto np) {
        constexpr int NP = decltype(np)::value;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const float4 *rowp = base + (size_t)i * pitch;
            float2 rs = czero();
#pragma unroll
            for (int j = 0; j < NP; ++j) {
                const float4 v = load(rowp + j * ZC);
                rs.x = fmaf(wx[2 * j], v.x, rs.x);
                rs.y = fmaf(wx[2 * j], v.y, rs.y);
                rs.x = fmaf(wx[2 * j + 1], v.z, rs.x);
                rs.y = fmaf(wx[2 * j + 1], v.w, rs.y);
            }
            acc.x = fmaf(wy[i], rs.x, acc.x);
            acc.y = fmaf(wy[i], rs.y, acc.y);
        }
    };
    if (__float_as_int(a5.w))
        rows(std::integral_constant<int, NPAIR>{});
    else
        rows(std::integral_constant<int, NPAIR - 1>{});
    return acc;
}

template <int N, int W>
__global__ void __launch_bounds__(GPB *ZC, 4)
    k_fwd_gather_pts(const float2 *__restrict__ fg, size_t set, float2 *__restrict__ lines, const float4 *__restrict__ rec,
                     int npts)
{
    constexpr int G = 2 * N, PS = G / 2 + GH_PAIRS;
    static_assert(W - 1 <= GH_ROWS, "the grid halo must cover the window");
    const int lane = threadIdx.x % ZC;
    const int pi = blockIdx.x * GPB + threadIdx.x / ZC;
    if (pi >= npts) return;
    const float4 *r = rec + (size_t)pi * REC4;
    const float4 q = __ldg(&r[5]);
    const float4 *base =
        reinterpret_cast<const float4 *>(fg + blockIdx.y * set) + ((size_t)__float_as_int(q.y) * PS + __float_as_int(q.z)) * ZC + lane;
    lines[((size_t)blockIdx.y * npts + __float_as_int(q.x)) * ZC + lane] =
        window_sum<W>(base, (size_t)PS * ZC, r, [](const float4 *p) { return __ldg(p); });
}

// The same gather with the grid staged in shared memory.  Points were sorted
// at setobj by the 16 x 16-cell tile of their window origin; a block takes a
// chunk of at most tile_points points of one tile, loads the part of the haloed grid
// that their windows cover (rows ty0 .. ty0 + 16 + W - 2, column pairs
// tx0/2 .. tx0/2 + 11, clipped to the haloed grid) and the points' records
// once, and gathers from there.  Weights, loads and the order of the sums are
// those of k_fwd_gather_pts, so the results are bit-identical.
// points per block of the tiled gather: up to 128 wide there are too few blocks
// of 128 points to fill the GPU evenly (64 wide, 64 slices, 96 angles 56 -> 50
// us; 128^3, 128 angles 177 -> 171); at 256 wide half-empty blocks cost more than
// they balance (256^3, 384 angles 1.36 and 1.39 ms)
template <int N>
constexpr int tile_points() { return N <= 192 ? 64 : 128; }
template <int W>
constexpr int tile_rows() { return GTILE + W - 1; }
constexpr int TILE_PAIRS = GTILE / 2 - 1 + NPAIR;
template <int W>
constexpr size_t tile_bytes() { return (size_t)tile_rows<W>() * TILE_PAIRS * ZC * sizeof(float4); }
template <int N, int W>
constexpr size_t tile_smem() { return tile_bytes<W>() + (size_t)tile_points<N>() * REC4 * sizeof(float4); }

// The gather of one chunk's points from its staged tile and records (both tiled kernels).
template <int W>
__device__ __forceinline__ void tile_gather(const float4 *__restrict__ tsm, const float4 *__restrict__ rsm, int count,
                                            int ty0, int px0, float2 *__restrict__ lines)
{
    const int lane = threadIdx.x % ZC;
    for (int t = threadIdx.x / ZC; t < count; t += GPB) {
        const float4 *r = rsm + t * REC4;
        const float4 q = r[5];
        // window origin relative to the staged region (inside it by the tile sort)
        const int rr = __float_as_int(q.y) - ty0, pp = __float_as_int(q.z) - px0;
        lines[(size_t)__float_as_int(q.x) * ZC + lane] =
            window_sum<W>(tsm + (rr * TILE_PAIRS + pp) * ZC + lane, TILE_PAIRS * ZC, r,
                          [](const float4 *p) { return *p; });
    }
}

template <int N, int W>
__global__ void __launch_bounds__(GPB *ZC, 4)
    k_fwd_gather_tile(const float2 *__restrict__ fg, size_t set, float2 *__restrict__ lines,
                      const float4 *__restrict__ rec, const int4 *__restrict__ chunks, int npts)
{
    constexpr int G = 2 * N;
    constexpr int PS = G / 2 + GH_PAIRS, NROWS = G + GH_ROWS;   // the haloed grid's pair pitch and rows
    extern __shared__ float4 tsm[];
    float4 *rsm = tsm + tile_bytes<W>() / sizeof(float4);
    const int4 ch = chunks[blockIdx.x];   // (tile row, tile column, first, count)
    const int ty0 = ch.x * GTILE, px0 = ch.y * GTILE / 2;
    const int rows = min(tile_rows<W>(), NROWS - ty0), pairs = min(TILE_PAIRS, PS - px0);
    const float4 *g4 = reinterpret_cast<const float4 *>(fg + blockIdx.y * set);
    for (int e = threadIdx.x; e < rows * pairs * ZC; e += blockDim.x) {
        const int r = e / (pairs * ZC), rem = e % (pairs * ZC), pj = rem / ZC, q = rem % ZC;
        tsm[(r * TILE_PAIRS + pj) * ZC + q] = __ldg(&g4[((size_t)(ty0 + r) * PS + px0 + pj) * ZC + q]);
    }
    for (int e = threadIdx.x; e < ch.w * REC4; e += blockDim.x) rsm[e] = __ldg(&rec[(size_t)ch.z * REC4 + e]);
    __syncthreads();
    tile_gather<W>(tsm, rsm, ch.w, ty0, px0, lines + (size_t)blockIdx.y * npts * ZC);
}

// The same with the tile and the records staged by the Tensor Memory
// Accelerator: one cp.async.bulk.tensor 3-D box load (32 floats = one column
// pair of ZC slices, TILE_PAIRS pairs, tile_rows rows) of the haloed grid and
// one bulk copy of the chunk's records into shared memory, completed on an
// mbarrier.  The box lands in exactly the layout of k_fwd_gather_tile's copy
// (and is zero-filled past the grid's end, where no window reads), so the
// results are bit-identical.  The wait is bounded: after TMA_SPIN polls the
// block records the failure in *err, waits (bounded again) for its copies and
// returns without writing.  The mbarriers sit after the tile and the records
// in dynamic shared memory (no static shared memory, so the tile starts at the
// 128-byte aligned base; checked, and a misaligned base is recorded in *err
// instead of issuing the copy).
constexpr int TMA_SPIN = 1 << 24;
template <int N, int W>
constexpr size_t tma_smem() { return tile_smem<N, W>() + 16; }
struct GridMaps {
    CUtensorMap m[RSETS];   // one per buffer set
};
template <int N, int W>
__global__ void __launch_bounds__(GPB *ZC, 4)
    k_fwd_gather_tma(const __grid_constant__ GridMaps maps, int set0, float2 *__restrict__ lines,
                     const float4 *__restrict__ rec, const int4 *__restrict__ chunks, int npts, int *__restrict__ err,
                     int spin = TMA_SPIN, int check = 0)
{
    // check != 0 (the status test only): the blocks first wait on a second
    // barrier that nothing arrives at, so that wait runs out on purpose; the
    // failure path then waits for the copies themselves before returning
    constexpr unsigned TB = (unsigned)tile_bytes<W>(), END = (unsigned)tile_smem<N, W>();
    static_assert(TB % 128 == 0 && END % 16 == 0, "the records and the mbarriers follow the tile");
    extern __shared__ __align__(128) float4 tsm_tma[];
    float4 *tsm = tsm_tma, *rsm = tsm_tma + TB / sizeof(float4);
    const int4 ch = chunks[blockIdx.x];
    const int ty0 = ch.x * GTILE, px0 = ch.y * GTILE / 2;   // >= 0; the column coordinate is 0
    const unsigned dst = (unsigned)__cvta_generic_to_shared(tsm);
    const unsigned bar_a = dst + END, bar_b = dst + END + 8;
    if (dst & 127) {
        if (threadIdx.x == 0) atomicExch(err, 2);
        return;
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_b) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned rbytes = (unsigned)ch.w * (unsigned)(REC4 * sizeof(float4));   // 16-byte multiples, as the source
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_a), "r"(TB + rbytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
            "%4}], [%5];" ::"r"(dst),
            "l"(reinterpret_cast<unsigned long long>(&maps.m[set0 + blockIdx.y])), "r"(0), "r"(px0), "r"(ty0), "r"(bar_a)
            : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst + TB),
                     "l"(rec + (size_t)ch.z * REC4), "r"(rbytes), "r"(bar_a)
                     : "memory");
    }
    auto wait = [&](unsigned bar, int limit) {
        unsigned ok = 0;
        for (int it = 0; it < limit && !ok; ++it)
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                : "=r"(ok)
                : "r"(bar), "r"(0)
                : "memory");
        return ok;
    };
    if (!wait(check ? bar_b : bar_a, spin)) {
        if (threadIdx.x == 0) atomicExch(err, 1);
        wait(bar_a, TMA_SPIN);   // the copies land in this block's memory: let them finish first
        return;
    }
    tile_gather<W>(tsm, rsm, ch.w, ty0, px0, lines + (size_t)blockIdx.y * npts * ZC);
}

// ---- K3b: fftshift1c / 1-D inverse FFT / fftshift1c + crop + scale --------
// tw: W^(i2 k1) (-1)^(i2 + k1), inverse: the two sign changes of the centred
// transform.  Only the cropped outputs are formed.
template <int N>
__global__ void __launch_bounds__(ptfft::Exchange<N, ZC>::NT, N > 384 ? 2 : 4)
    k_fwd_lines(const float2 *__restrict__ lines, float2 *__restrict__ out, int nz, int z0, float scale,
                const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<N, ZC>;
    constexpr int n = 2 * N / 3, c0 = N / 6, R1 = E::R1, R2 = E::R2;
    extern __shared__ float2 sm[];
    const int th = blockIdx.x;
    const int q = threadIdx.x % ZC, b = threadIdx.x / ZC;
    if (b < R2) {
        const float2 *src = lines + (((size_t)blockIdx.y * gridDim.x + th) * N + b) * ZC + q;
        float2 v[R1];
#pragma unroll
        for (int i1 = 0; i1 < R1; ++i1) v[i1] = src[i1 * R2 * ZC];
        ptfft::Dft<R1, +1, true>::run(v);
        ptfft::twiddle_pairs<R1, R2>(v, b, tw);
        E::put(sm, v, b, q);
    }
    __syncthreads();
    const int z = z0 + blockIdx.y * ZC + q;
    if (b < R1 && z < nz) {
        float2 w[R2];
        E::get(sm, w, b, q);
        ptfft::Dft<R2, +1, true>::run(w);
        float2 *dst = out + ((size_t)th * nz + z) * n;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) {
            if (R1 * k2 + R1 <= c0 || R1 * k2 >= c0 + n) continue;   // wholly cropped
            const int j = b + R1 * k2 - c0;
            if (j >= 0 && j < n) dst[j] = scale * w[k2];
        }
    }
}

// K3a and K3b in one launch for short lines: a block gathers the N points of
// one angle through L1 into shared memory and transforms them (the same sums
// and rounds as k_fwd_gather_pts and k_fwd_lines).  rec is in point order.
// One launch and one pass over the lines buffer less, but the grid is read
// through L1.  32 wide, against the tiles in shared memory (us): 8 slices, 96
// angles 16.4 and 18.4; 256 slices, 96 angles 151 and 164.  With more than
// FUSED_POINTS polar points in the chunks that the pipelines work on at once
// (angles x N x chunks) the tiles win.  32 wide: 384 angles, 8 slices (18432
// points) 18.5 and 20.5, 16 slices 26.7 and 22.6; 16 wide: 192 angles, 32 slices
// (18432) 20.5 and 20.6, 288 angles 22.4 and 20.6; 8 wide: 288 angles, 32 slices
// (13824) 18.4 and 19.6, 768 angles 26.7 and 22.6.  64 wide the tiles take less
// time on the device at every size (25 slices, 28 angles 22 against 25 us; 64
// slices, 96 angles 50 and 59), but with few angles a caller who launches each
// call waits for their fourth launch (25 slices, 28 angles 27.5 against 25.4).
constexpr int FUSED_N = 96;   // longest line (64 wide)
constexpr int FUSED_POINTS = 18432;
template <int N, int W>
__global__ void __launch_bounds__(GPB *ZC, 4)
    k_fwd_gather_lines(const float2 *__restrict__ fg, size_t set, const float4 *__restrict__ rec,
                       float2 *__restrict__ out, int nz, int z0, float scale, const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<N, ZC>;
    constexpr int G = 2 * N, PS = G / 2 + GH_PAIRS, n = 2 * N / 3, c0 = N / 6, R1 = E::R1, R2 = E::R2;
    static_assert(W - 1 <= GH_ROWS && E::NT <= GPB * ZC, "the halo covers the window, the block the transform");
    __shared__ float2 line[N * ZC], sm[E::BYTES / sizeof(float2)];
    const int th = blockIdx.x;
    const int q = threadIdx.x % ZC, b = threadIdx.x / ZC;
    const float4 *g4 = reinterpret_cast<const float4 *>(fg + blockIdx.y * set) + q;
    for (int k = b; k < N; k += GPB) {
        const float4 *r = rec + ((size_t)th * N + k) * REC4;
        const float4 o = __ldg(&r[5]);
        line[k * ZC + q] = window_sum<W>(g4 + ((size_t)__float_as_int(o.y) * PS + __float_as_int(o.z)) * ZC,
                                         (size_t)PS * ZC, r, [](const float4 *p) { return __ldg(p); });
    }
    __syncthreads();
    if (b < R2) {
        float2 v[R1];
#pragma unroll
        for (int i1 = 0; i1 < R1; ++i1) v[i1] = line[(i1 * R2 + b) * ZC + q];
        ptfft::Dft<R1, +1, true>::run(v);
        ptfft::twiddle_pairs<R1, R2>(v, b, tw);
        E::put(sm, v, b, q);
    }
    __syncthreads();
    const int z = z0 + blockIdx.y * ZC + q;
    if (b < R1 && z < nz) {
        float2 w[R2];
        E::get(sm, w, b, q);
        ptfft::Dft<R2, +1, true>::run(w);
        float2 *dst = out + ((size_t)th * nz + z) * n;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) {
            if (R1 * k2 + R1 <= c0 || R1 * k2 >= c0 + n) continue;   // wholly cropped
            const int j = b + R1 * k2 - c0;
            if (j >= 0 && j < n) dst[j] = scale * w[k2];
        }
    }
}

// ---- A1: pad (kernels.cuh:189-206) + fftshift1c/FFT/fftshift1c -------------
// grid (ntheta, nzp / ZC); writes lines[(theta*N + k) * nzp + z].  ZP: the
// exact adjoint's zero padding (the adjoint of the forward's crop) instead
// of the reference's edge replication.  tw: W^(i2 k1) (-1)^(i2 + k1), forward.
template <int N, bool ZP = false>
__global__ void __launch_bounds__(ptfft::Exchange<N, ZC>::NT, N > 384 ? 2 : 4)
    k_adj_lines(const float2 *__restrict__ g, float2 *__restrict__ lines, int nz, int nzp, float pre,
                const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<N, ZC>;
    constexpr int n = 2 * N / 3, c0 = N / 6, c1 = 5 * N / 6 - 1, R1 = E::R1, R2 = E::R2;
    extern __shared__ float2 sm[];
    const int th = blockIdx.x, z0 = blockIdx.y * ZC;
    const int q = threadIdx.x % ZC, b = threadIdx.x / ZC;
    const int z = z0 + q;
    if (b < R2) {
        float2 v[R1];
        const float2 *src = g + ((size_t)th * nz + z) * n;
#pragma unroll
        for (int i1 = 0; i1 < R1; ++i1) {
            const int k = i1 * R2 + b;
            v[i1] = czero();
            if (z < nz && (!ZP || (k >= c0 && k <= c1))) v[i1] = src[min(max(k, c0), c1) - c0];
        }
        ptfft::Dft<R1, -1, true>::run(v);
        ptfft::twiddle_pairs<R1, R2>(v, b, tw);
        E::put(sm, v, b, q);
    }
    __syncthreads();
    if (b < R1) {
        float2 w[R2];
        E::get(sm, w, b, q);
        ptfft::Dft<R2, -1, true>::run(w);
        float2 *dst = lines + ((size_t)th * N + b) * nzp + z;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) dst[(size_t)k2 * R1 * nzp] = pre * w[k2];
    }
}

// ---- A2: column gather (transpose of the forward gather) + column IFFT ----
// grid (nzp / 16, G); block of CT threads.  A warp owns 4 consecutive
// cells (a "cell group") of the column at a time; the group's list holds every
// polar point whose kernel window covers any of the 4 cells, with the 4
// weights (0 where the window misses a cell), in increasing point order.
// A warp holds 4 entry streams x 16 slices, combined at the end in a fixed
// order -> deterministic.  Each loaded g value feeds 4 accumulators.  A point
// of the 8-cell window has 22 entries (8 columns x 2.75 groups), of the 15-cell
// Gaussian 67: at 256^3 and 384 angles 1.58 against 2.79 ms.
// The list loop takes 0.98 of the kernel's 1.34 ms, the transforms 0.27.
// Tried and slower: a list per stream (more weight lines per load), one masked
// trip per list end with the indices loaded ahead, columns as the fast grid
// dimension.
// ALL: write all N rows of the padded slice (rows N/2 .. N/2 + N - 1 of the
// grid, for the exact adjoint's fold) instead of the n rows of the crop.
constexpr int ZQ = 16;
constexpr int CG = 4;  // cells per group
template <int G>
constexpr int col_threads() { return G >= 1024 ? 1024 : G >= 96 ? 512 : 256; }   // 64^3: 40 us with 256, 36 with 512
template <int G, bool ALL = false>
__global__ void __launch_bounds__(col_threads<G>(), (G >= 1024 ? 1 : G >= 96 ? 2 : 4))
    k_adj_colgather(const float2 *__restrict__ lines, float2 *__restrict__ rbuf, const int *__restrict__ goff,
                    const int *__restrict__ gpt, const float4 *__restrict__ gw, const int *__restrict__ col_order,
                    int nzp, const float2 *__restrict__ tw1, const float2 *__restrict__ tw2)
{
    constexpr int N = G / 2, n = G / 3, NG4 = G / CG;
    constexpr int Y0 = N / 2 + N / 6;
    constexpr int U = 4;  // entries in flight per lane
    extern __shared__ float2 sm[];
    const int z0 = blockIdx.x * ZQ;
    const int kx = col_order[blockIdx.y];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // 4 entry streams per warp; a stream's 8 lanes hold 2 slices each (one
    // 16-byte load of a point's line covers 2 slices)
    const int s = lane >> 3, zl = lane & 7;
    const int nwarps = blockDim.x >> 5;
    const float4 *lz = reinterpret_cast<const float4 *>(lines + z0) + zl;
    const size_t lstride = (size_t)nzp / 2;  // float4 per point line
    for (int gi = warp; gi < NG4; gi += nwarps) {
        const int beg = goff[kx * NG4 + gi], end = goff[kx * NG4 + gi + 1];
        float4 acc[CG];  // (re, im) of slices 2 zl and 2 zl + 1, per cell
#pragma unroll
        for (int c = 0; c < CG; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        int e = beg + s;
        for (; e + 4 * (U - 1) < end; e += 4 * U) {
            int pp[U];
            float4 w[U], v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                pp[u] = __ldg(&gpt[e + 4 * u]);
                w[u] = __ldg(&gw[e + 4 * u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = __ldg(lz + (size_t)pp[u] * lstride);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float wc[CG] = {w[u].x, w[u].y, w[u].z, w[u].w};
#pragma unroll
                for (int c = 0; c < CG; ++c) {
                    acc[c].x = fmaf(wc[c], v[u].x, acc[c].x);
                    acc[c].y = fmaf(wc[c], v[u].y, acc[c].y);
                    acc[c].z = fmaf(wc[c], v[u].z, acc[c].z);
                    acc[c].w = fmaf(wc[c], v[u].w, acc[c].w);
                }
            }
        }
        for (; e < end; e += 4) {
            const int pp = __ldg(&gpt[e]);
            const float4 w = __ldg(&gw[e]);
            const float4 v = __ldg(lz + (size_t)pp * lstride);
            const float wc[CG] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int c = 0; c < CG; ++c) {
                acc[c].x = fmaf(wc[c], v.x, acc[c].x);
                acc[c].y = fmaf(wc[c], v.y, acc[c].y);
                acc[c].z = fmaf(wc[c], v.z, acc[c].z);
                acc[c].w = fmaf(wc[c], v.w, acc[c].w);
            }
        }
        // streams 0+2 and 1+3, then those two sums: each exchange hands over the
        // half that the partner keeps, so stream s ends with cell s (12 shuffles
        // instead of 32, and a store by all lanes)
        {
            const bool up2 = s & 2, up1 = s & 1;
            float4 k[2], g;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                k[j] = up2 ? acc[2 + j] : acc[j];
                g = up2 ? acc[j] : acc[2 + j];
                k[j].x += __shfl_xor_sync(0xffffffffu, g.x, 16);
                k[j].y += __shfl_xor_sync(0xffffffffu, g.y, 16);
                k[j].z += __shfl_xor_sync(0xffffffffu, g.z, 16);
                k[j].w += __shfl_xor_sync(0xffffffffu, g.w, 16);
            }
            float4 r = up1 ? k[1] : k[0];
            g = up1 ? k[0] : k[1];
            r.x += __shfl_xor_sync(0xffffffffu, g.x, 8);
            r.y += __shfl_xor_sync(0xffffffffu, g.y, 8);
            r.z += __shfl_xor_sync(0xffffffffu, g.z, 8);
            r.w += __shfl_xor_sync(0xffffffffu, g.w, 8);
            reinterpret_cast<float4 *>(sm)[(gi * CG + s) * (ZQ / 2) + zl] = r;
        }
    }
    __syncthreads();
    // the 16 slices' column transforms in place (shared row ky = element ky of
    // each; the grid's centring sign (-1)^ky is in tw2, (-1)^kx in the row
    // pass's table); the cropped rows go from the last round's registers to memory
    constexpr int ROWS = ALL ? N : n, YB = ALL ? N / 2 : Y0;
    constexpr int C = ptfft::split3_c(G), AB = G / C;
    float2 *dst = rbuf + (size_t)kx * nzp + z0;
    ptfft::fft3<G, +1, col_threads<G>(), ZQ>(sm, tw1, tw2, [&](int kk, int q, const float2 (&w)[C]) {
#pragma unroll
        for (int k3 = 0; k3 < C; ++k3) {
            if (AB * k3 + AB <= YB || AB * k3 >= YB + ROWS) continue;   // wholly cropped
            const int r = kk + AB * k3 - YB;
            if (r >= 0 && r < ROWS) dst[(size_t)r * G * nzp + q] = w[k3];
        }
    });
}

// setobj: the 4 weights of every (cell group, point) entry, wx * wy of the
// forward gather's window (kernels.cuh:115-119 written separably).
// key = point << 9 | i0 << 5 | (r0 + 3): window column i0, and the window row
// r0 in [-3, W - 1] of the group's first cell.
template <int W>
__global__ void k_make_entries(const unsigned *__restrict__ keys, int *__restrict__ gpt, float4 *__restrict__ gw,
                               size_t total, const float *__restrict__ wtab)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const unsigned key = keys[e];
    const int p = (int)(key >> 9), i0 = (int)((key >> 5) & 15), r0 = (int)(key & 31) - 3;
    const float *wy = wtab + (size_t)p * 2 * W + W;
    const float wx = wtab[(size_t)p * 2 * W + i0];
    float w[CG];
#pragma unroll
    for (int c = 0; c < CG; ++c) {
        const int i1 = r0 + c;
        w[c] = (i1 >= 0 && i1 < W) ? wx * wy[i1] : 0.f;
    }
    gpt[e] = p;
    gw[e] = make_float4(w[0], w[1], w[2], w[3]);
}

// Round 1 of the adjoint's row transforms: src is the row's first column for
// this thread's slice, columns nzp apart.
template <int G>
__device__ __forceinline__ void adj_row_round1(const float2 *__restrict__ src, int nzp, float2 *sm, int b, int q,
                                               const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<G, ZC>;
    constexpr int R1 = E::R1, R2 = E::R2;
    if (b < R2) {
        float2 v[R1];
#pragma unroll
        for (int i1 = 0; i1 < R1; ++i1) v[i1] = src[(size_t)(i1 * R2 + b) * nzp];
        ptfft::Dft<R1, +1, true>::run(v);
        ptfft::twiddle_pairs<R1, R2>(v, b, tw);
        E::put(sm, v, b, q);
    }
}

// ---- A4: row inverse FFT + fftshiftc + unpaddivphi + circ + crop -----------
// grid (n, nzp / ZC); reads rbuf[(r * G + kx) * nzp + z].  tw: W^(i2 k1)
// (-1)^i2, inverse (the sign of the grid column; that of the output is in fac).
template <int G>
__global__ void __launch_bounds__(ptfft::Exchange<G, ZC>::NT, row_blocks<G>())
    k_adj_rows(const float2 *__restrict__ rbuf, float2 *__restrict__ out, int nz, int nzp,
               const float *__restrict__ fac, float scale, const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<G, ZC>;
    constexpr int N = G / 2, n = G / 3, c0 = N / 6, R1 = E::R1, R2 = E::R2;
    extern __shared__ float2 sm[];
    const int r = blockIdx.x, z0 = blockIdx.y * ZC;
    const int q = threadIdx.x % ZC, b = threadIdx.x / ZC;
    adj_row_round1<G>(rbuf + (size_t)r * G * nzp + z0 + q, nzp, sm, b, q, tw);
    __syncthreads();
    const int z = z0 + q;
    if (b < R1 && z < nz) {
        float2 w[R2];
        E::get(sm, w, b, q);
        ptfft::Dft<R2, +1, true>::run(w);
        const float *f = fac + (size_t)(c0 + r) * N + c0;
        float2 *dst = out + ((size_t)z * n + r) * n;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) {
            if (R1 * k2 + R1 <= N / 2 + c0 || R1 * k2 >= N / 2 + c0 + n) continue;   // wholly cropped
            const int c = b + R1 * k2 - (N / 2 + c0);
            if (c >= 0 && c < n) dst[c] = scale * (__ldg(&f[c]) * w[k2]);
        }
    }
}


// ---- exact adjoint: rows of the whole padded slice, then the folds ---------
// The forward's pad2 replicates the edge pixels of f into the margins of the
// N x N slice (kernels.cuh:208-216) and its last step crops n of N detector
// samples; their adjoints are a fold (every margin pixel added onto the edge
// pixel it copies) and a zero padding.  grid (N, nzp / ZC): input row ty of
// the padded slice (rbuf row ty, written by the ALL column gather): row
// inverse FFT, sign, circ / phi / (4 N^2), and the fold along x; a row inside
// the crop goes to out, a margin row (ty <= c0 or ty >= c0 + n - 1) to its
// slot of mbuf [n/2 + 2][nz][n] for the fold along y.
template <int G>
__global__ void __launch_bounds__(ptfft::Exchange<G, ZC>::NT, row_blocks<G>())
    k_adj_rows_exact(const float2 *__restrict__ rbuf, float2 *__restrict__ out, float2 *__restrict__ mbuf, int nz,
                     int nzp, const float *__restrict__ fac, float scale, const float4 *__restrict__ tw)
{
    using E = ptfft::Exchange<G, ZC>;
    constexpr int N = G / 2, n = G / 3, c0 = N / 6, R1 = E::R1, R2 = E::R2;
    extern __shared__ float2 sm[];
    const int ty = blockIdx.x, z0 = blockIdx.y * ZC;
    {
        const int q = threadIdx.x % ZC, b = threadIdx.x / ZC;
        adj_row_round1<G>(rbuf + (size_t)ty * G * nzp + z0 + q, nzp, sm, b, q, tw);
        __syncthreads();
        float2 w[R2];
        if (b < R1) E::get(sm, w, b, q);
        __syncthreads();   // the exchange is read: the row goes back in natural order
        if (b < R1) {
            ptfft::Dft<R2, +1, true>::run(w);
#pragma unroll
            for (int k2 = 0; k2 < R2; ++k2) sm[(b + R1 * k2) * ZC + q] = w[k2];
        }
        __syncthreads();
    }
    const float *facr = fac + (size_t)ty * N;
    for (int e = threadIdx.x; e < ZC * n; e += blockDim.x) {
        const int q = e % ZC, c = e / ZC;
        const int z = z0 + q;
        if (z >= nz) continue;
        // columns tx of the padded row that copy pixel c (fixed order)
        const int lo = c == 0 ? 0 : c0 + c, hi = c == n - 1 ? N - 1 : c0 + c;
        float2 acc = czero();
        for (int tx = lo; tx <= hi; ++tx) {
            acc = acc + __ldg(&facr[tx]) * sm[(N / 2 + tx) * ZC + q];
        }
        acc = scale * acc;
        if (ty > c0 && ty < c0 + n - 1) {
            out[((size_t)z * n + (ty - c0)) * n + c] = acc;
        } else {
            const int slot = ty <= c0 ? ty : (c0 + 1) + (ty - (c0 + n - 1));
            mbuf[((size_t)slot * nz + z) * n + c] = acc;
        }
    }
}

// out row 0 = sum of margin slots 0..c0, row n-1 = the remaining slots (fixed
// order; grid y: the row).  Unrolled: eight slots' loads are in flight.
__global__ void k_adj_fold_rows(const float2 *__restrict__ mbuf, float2 *__restrict__ out, int nz, int n, int c0,
                                int nslots)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nz * n) return;
    const int z = (int)(i / n), c = (int)(i % n);
    const bool last = blockIdx.y != 0;
    const int s0 = last ? c0 + 1 : 0, s1 = last ? nslots : c0 + 1;
    float2 a = czero();
#pragma unroll 8
    for (int s = s0; s < s1; ++s) a = a + mbuf[((size_t)s * nz + z) * n + c];
    out[((size_t)z * n + (last ? n - 1 : 0)) * n + c] = a;
}

}  // namespace

// ============================================================================
// handle
// ============================================================================
struct pt_radon {
    int ntheta = 0, nz = 0, n = 0, N = 0, G = 0, M = 0, nzp = 0;
    float mu = 0.f;
    int device = -1;
    bool ready = false;
    // two allocations cut into pieces: the tables (tw_fwd ..
    // tma_err, deap, inv1, goff, col_order) and the forward's buffer sets (rbuf, fgrid)
    char *tables = nullptr, *sets = nullptr;
    // twiddles with the centring signs: the forward's rows and columns, the
    // adjoint's rows, the detector lines (twiddle_pairs layout), and the three
    // rounds of the adjoint's columns
    float4 *tw_fwd = nullptr, *tw_adj = nullptr, *tw_fwd_line = nullptr, *tw_inv_line = nullptr;
    float2 *tw_col1 = nullptr, *tw_col2 = nullptr;
    float *theta = nullptr, *x = nullptr, *y = nullptr;
    int W = 0;                // cells of the gridding window per axis (WKB or WGAUSS)
    int *org = nullptr;       // first grid column and row of each point's window
    float *wtab = nullptr;    // the window's values, [point][x: W, y: W]
    int *perm = nullptr;      // the forward gather's point order (grid tiles)
    float4 *rec = nullptr;    // each point's gather record, in that order
    float4 *rec_pt = nullptr; // the records in point order (N <= FUSED_N)
    int4 *chunks = nullptr;   // the tiled gather's blocks: (tile row, tile column, first, count)
    int nchunks = 0, chunks_cap = 0;
    int gather = 2;           // 0: gather through L1 (k_fwd_gather_pts), 1: shared-memory tiles, 2: TMA-staged tiles
    // gather 2: one 3-D tensor map per grid buffer set, and a device flag the
    // TMA kernel sets if a tile load did not complete
    GridMaps tmap;
    bool tma_ok = false;
    int *tma_err = nullptr;
    // forward: per chunk of ZC slices, a row-FFT buffer and a Fourier grid (a
    // buffer set; RSETS of them, a constant distance apart).  `streams`
    // pipelines of RSETS / streams chunks per launch: pipeline 0 on the
    // caller's stream, the others on side streams (fork/join by events), so
    // one pipeline's FFTs overlap another's gather
    float2 *rbuf[RSETS] = {}, *fgrid[RSETS] = {};
    int streams = 4;   // 1, 2 or 4 (pt_radon_autotune chooses)
    cudaStream_t side[RSETS - 1] = {};
    cudaEvent_t ev_fork = nullptr, ev_join[RSETS - 1] = {};
    // adjoint (all slices, slice-minor with nzp lanes)
    float2 *lines = nullptr, *rbuf_adj = nullptr, *mbuf = nullptr;
    int *goff = nullptr, *col_order = nullptr, *gpt = nullptr;
    float4 *gw = nullptr;
    float *deap = nullptr;  // N x N: circ / the window's transform
    double *inv1 = nullptr; // Kaiser-Bessel: 1 / the window's transform on one axis
    size_t entries_cap = 0;
};

namespace {

void radon_free(pt_radon *h)
{
    void *bufs[] = {h->tables, h->sets, h->chunks, h->lines, h->rbuf_adj, h->mbuf, h->gpt, h->gw};
    for (void *p : bufs)
        if (p) cudaFree(p);
    for (int k = 0; k < RSETS - 1; ++k) {
        if (h->side[k]) cudaStreamDestroy(h->side[k]);
        if (h->ev_join[k]) cudaEventDestroy(h->ev_join[k]);
    }
    if (h->ev_fork) cudaEventDestroy(h->ev_fork);
}

// Kernel half-width for a forced M: choose -log(eps) so that the reference's
// formula (radonusfft.cu:12) yields exactly M, then mu = -log(eps)/(2N^2).
void radon_params(int n, int m_override, int *N, int *M, float *mu)
{
    *N = n * 3 / 2;
    const size_t NN = (size_t)*N;
    if (m_override <= 0) {
        float eps = 1e-6;  // radonusfft.cu:10-12, same expressions and types
        *mu = -log(eps) / (2 * NN * NN);
        *M = (int)ceil(2 * NN * 1 / PI_REF * sqrt(-*mu * log(eps) + (*mu * NN) * (*mu * NN) / 4));
    } else {
        const double L = m_override * PI_REF / 1.5 - 1e-3;  // ceil(2/pi*0.75*L) = M
        *mu = (float)(L / (2.0 * (double)NN * (double)NN));
        *M = m_override;
    }
}

// Factor of the gathered (forward) and padded (adjoint) line samples: the 1/N
// of the 1-D transforms, times pi/mu of the Gaussian kernel (kernels.cuh:119).
float radon_pre(const pt_radon *h)
{
    const float s = h->W == WKB ? 1.f : (float)(PI_REF / std::fabs(h->mu));
    return s / (float)h->N;
}

// Tensor maps of the haloed grid buffers (RSETS) for k_fwd_gather_tma: float32,
// dims (innermost first) {ZC * 4 floats = one column pair of the chunk's
// slices, G/2 + GH_PAIRS pairs, G + GH_ROWS rows}, row-major strides
// {ZC * 16, (G/2 + GH_PAIRS) * ZC * 16} bytes, box {ZC * 4, TILE_PAIRS, tile_rows}: the
// box's inner extent is 128 bytes and its first coordinate is always 0, so
// every load starts on a 16-byte boundary.  cuTensorMapEncodeTiled comes
// from the driver through the runtime's entry-point query (no link against
// libcuda); false if it or any encode fails.
bool encode_grid_maps(pt_radon *h)
{
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || fn == nullptr) {
        cudaGetLastError();
        return false;
    }
    auto encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    const int G = h->G;
    const cuuint64_t pairs = (cuuint64_t)(G / 2 + GH_PAIRS), rows = (cuuint64_t)(G + GH_ROWS);
    const cuuint64_t dims[3] = {(cuuint64_t)ZC * 4, pairs, rows};
    const cuuint64_t strides[2] = {(cuuint64_t)ZC * 16, pairs * ZC * 16};
    const cuuint32_t tr = (cuuint32_t)(GTILE + h->W - 1), tp = (cuuint32_t)TILE_PAIRS;
    const cuuint32_t box[3] = {(cuuint32_t)ZC * 4, tp, tr};
    const cuuint32_t estr[3] = {1, 1, 1};
    for (int b = 0; b < RSETS; ++b) {
        if (((uintptr_t)h->fgrid[b] & 127) != 0) return false;
        if (encode(&h->tmap.m[b], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, h->fgrid[b], dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

template <int L>
constexpr int ex_smem() { return (int)ptfft::Exchange<L, ZC>::BYTES; }
template <int G>
constexpr int col_smem() { return ZQ * G * (int)sizeof(float2); }

template <int G>
int set_attrs()
{
    constexpr int N = G / 2;
    static_assert(CK * ZH == ZC, "ex_smem serves the column kernel too");
#define PT_ATTR(K, S) PT_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(S)))
    PT_ATTR(k_fwd_rows<G>, ex_smem<G>());
    PT_ATTR(k_fwd_cols<G>, ex_smem<G>());
    PT_ATTR(k_adj_colgather<G>, col_smem<G>());
    PT_ATTR((k_adj_colgather<G, true>), col_smem<G>());
    PT_ATTR(k_adj_rows<G>, ex_smem<G>());
    PT_ATTR(k_adj_rows_exact<G>, ex_smem<G>());
    PT_ATTR(k_fwd_lines<N>, ex_smem<N>());
    PT_ATTR(k_adj_lines<N>, ex_smem<N>());
    PT_ATTR((k_adj_lines<N, true>), ex_smem<N>());
    PT_ATTR((k_fwd_gather_tile<N, WKB>), (tile_smem<N, WKB>()));
    PT_ATTR((k_fwd_gather_tile<N, WGAUSS>), (tile_smem<N, WGAUSS>()));
    PT_ATTR((k_fwd_gather_tma<N, WKB>), (tma_smem<N, WKB>()));
    PT_ATTR((k_fwd_gather_tma<N, WGAUSS>), (tma_smem<N, WGAUSS>()));
#undef PT_ATTR
    return PT_OK;
}

template <int G, int W>
int run_fwd(pt_radon *h, float2 *g, const float2 *f, float scale, cudaStream_t st)
{
    constexpr int N = G / 2;
    using EG = ptfft::Exchange<G, ZC>;
    using EN = ptfft::Exchange<N, ZC>;
    const int nchunks = (h->nz + ZC - 1) / ZC;
    // `streams` pipelines, each with `batch` buffer sets: a launch of pipeline p
    // works on up to `batch` chunks in sets p batch ..., gathered into the same
    // blocks of the lines buffer (nzp / ZC blocks, at least the chunk count)
    const int batch = RSETS / h->streams;
    const int sets = std::min(h->streams, (nchunks + batch - 1) / batch);   // pipelines in use
    const size_t stride = h->rbuf[1] - h->rbuf[0];
    const int npts = h->ntheta * N;
    if (sets > 1) {   // fork: the side streams start after everything queued on st so far
        PT_CUDA(cudaEventRecord(h->ev_fork, st));
        for (int k = 1; k < sets; ++k) PT_CUDA(cudaStreamWaitEvent(h->side[k - 1], h->ev_fork, 0));
    }
    for (int c = 0, it = 0; c < nchunks; c += batch, ++it) {
        // pipeline it % sets reuses its buffer sets in order on its own stream
        const int p = it % sets, k = p * batch, cnt = std::min(batch, nchunks - c), z0 = c * ZC;
        cudaStream_t s = p ? h->side[p - 1] : st;
        float2 *rb = h->rbuf[k], *fg = h->fgrid[k];
        float2 *ln = h->lines + (size_t)k * npts * ZC;
        k_fwd_rows<G><<<dim3(N, cnt), EG::NT, EG::BYTES, s>>>(f, rb, stride, h->nz, z0, h->deap, h->tw_fwd);
        PT_LAUNCHED("k_fwd_rows");
        k_fwd_cols<G><<<dim3(G / CK, ZC / ZH, cnt), EG::NT, EG::BYTES, s>>>(rb, fg, stride, h->tw_fwd);
        PT_LAUNCHED("k_fwd_cols");
        if constexpr (N <= FUSED_N) {
            if (h->gather == 0) {
                k_fwd_gather_lines<N, W><<<dim3(h->ntheta, cnt), GPB * ZC, 0, s>>>(fg, stride, h->rec_pt, g, h->nz, z0,
                                                                                   scale, h->tw_inv_line);
                PT_LAUNCHED("k_fwd_gather_lines");
                continue;
            }
        }
        if (h->gather == 2) {
            k_fwd_gather_tma<N, W><<<dim3(h->nchunks, cnt), GPB * ZC, tma_smem<N, W>(), s>>>(
                h->tmap, k, ln, h->rec, h->chunks, npts, h->tma_err);
            PT_LAUNCHED("k_fwd_gather_tma");
        } else if (h->gather == 1) {
            k_fwd_gather_tile<N, W><<<dim3(h->nchunks, cnt), GPB * ZC, tile_smem<N, W>(), s>>>(fg, stride, ln, h->rec,
                                                                                           h->chunks, npts);
            PT_LAUNCHED("k_fwd_gather_tile");
        } else if constexpr (N > FUSED_N) {
            k_fwd_gather_pts<N, W><<<dim3((npts + GPB - 1) / GPB, cnt), GPB * ZC, 0, s>>>(fg, stride, ln, h->rec, npts);
            PT_LAUNCHED("k_fwd_gather_pts");
        }
        k_fwd_lines<N><<<dim3(h->ntheta, cnt), EN::NT, EN::BYTES, s>>>(ln, g, h->nz, z0, scale, h->tw_inv_line);
        PT_LAUNCHED("k_fwd_lines");
    }
    for (int k = 1; k < sets; ++k) {   // join: st continues after every side stream's chunks
        PT_CUDA(cudaEventRecord(h->ev_join[k - 1], h->side[k - 1]));
        PT_CUDA(cudaStreamWaitEvent(st, h->ev_join[k - 1], 0));
    }
    return PT_OK;
}

template <int G>
int run_adj(pt_radon *h, float2 *f, const float2 *g, float scale, cudaStream_t st, bool exact)
{
    constexpr int N = G / 2, n = G / 3;
    using EG = ptfft::Exchange<G, ZC>;
    using EN = ptfft::Exchange<N, ZC>;
    const float pre = radon_pre(h);
    const int nzp = h->nzp;
    const dim3 glines(h->ntheta, nzp / ZC), gcols(nzp / ZQ, G);
    if (exact) {
        k_adj_lines<N, true><<<glines, EN::NT, EN::BYTES, st>>>(g, h->lines, h->nz, nzp, pre, h->tw_fwd_line);
        PT_LAUNCHED("k_adj_lines");
        k_adj_colgather<G, true><<<gcols, col_threads<G>(), col_smem<G>(), st>>>(
            h->lines, h->rbuf_adj, h->goff, h->gpt, h->gw, h->col_order, nzp, h->tw_col1, h->tw_col2);
        PT_LAUNCHED("k_adj_colgather");
        k_adj_rows_exact<G><<<dim3(N, nzp / ZC), EG::NT, EG::BYTES, st>>>(h->rbuf_adj, f, h->mbuf, h->nz, nzp, h->deap,
                                                                         scale, h->tw_adj);
        PT_LAUNCHED("k_adj_rows_exact");
        const size_t cnt = (size_t)h->nz * n;
        k_adj_fold_rows<<<dim3((unsigned)((cnt + 127) / 128), 2), 128, 0, st>>>(h->mbuf, f, h->nz, n, N / 6, n / 2 + 2);
        PT_LAUNCHED("k_adj_fold_rows");
        return PT_OK;
    }
    k_adj_lines<N><<<glines, EN::NT, EN::BYTES, st>>>(g, h->lines, h->nz, nzp, pre, h->tw_fwd_line);
    PT_LAUNCHED("k_adj_lines");
    k_adj_colgather<G><<<gcols, col_threads<G>(), col_smem<G>(), st>>>(
        h->lines, h->rbuf_adj, h->goff, h->gpt, h->gw, h->col_order, nzp, h->tw_col1, h->tw_col2);
    PT_LAUNCHED("k_adj_colgather");
    k_adj_rows<G><<<dim3(n, nzp / ZC), EG::NT, EG::BYTES, st>>>(h->rbuf_adj, f, h->nz, nzp, h->deap, scale, h->tw_adj);
    PT_LAUNCHED("k_adj_rows");
    return PT_OK;
}

// Compiled grid sizes 2N = 3n (n = 8, 16, 32, 64, 128, 256, 512).
#define PT_RADON_GRIDS(X) X(24) X(48) X(96) X(192) X(384) X(768) X(1536)

bool grid_supported(int G)
{
#define PT_CASE(GG) \
    if (G == GG) return true;
    PT_RADON_GRIDS(PT_CASE)
#undef PT_CASE
    return false;
}

int radon_set_attrs(int G)
{
#define PT_CASE(GG) \
    if (G == GG) return set_attrs<GG>();
    PT_RADON_GRIDS(PT_CASE)
#undef PT_CASE
    pt::set_error("radonusfft: unsupported grid size %d", G);
    return PT_ERR_UNSUPPORTED;
}

int radon_dispatch(pt_radon *h, bool adj, float2 *out, const float2 *in, float scale, cudaStream_t st,
                   bool exact = false)
{
#define PT_CASE(GG)                                                                 \
    if (h->G == GG) {                                                               \
        if (adj) return run_adj<GG>(h, out, in, scale, st, exact);                  \
        return h->W == WKB ? run_fwd<GG, WKB>(h, out, in, scale, st)                \
                           : run_fwd<GG, WGAUSS>(h, out, in, scale, st);            \
    }
    PT_RADON_GRIDS(PT_CASE)
#undef PT_CASE
    pt::set_error("radonusfft: no kernel for grid %d", h->G);
    return PT_ERR_UNSUPPORTED;
}

// The TMA gather of the first slice chunk whose blocks first wait, 256 polls
// at most, on a barrier that nothing arrives at: every block's wait runs out,
// records code 1, waits for its own tile copy and returns without writing
// (the status test of pt_radon_check_tma_wait).
template <int G, int W>
int run_tma_wait_check(pt_radon *h, cudaStream_t st)
{
    constexpr int N = G / 2;
    k_fwd_gather_tma<N, W><<<h->nchunks, GPB * ZC, tma_smem<N, W>(), st>>>(h->tmap, 0, h->lines, h->rec, h->chunks,
                                                                        h->ntheta * N, h->tma_err, 256, 1);
    PT_LAUNCHED("k_fwd_gather_tma");
    return PT_OK;
}

int radon_tma_wait_check(pt_radon *h, cudaStream_t st)
{
#define PT_CASE(GG)                                                         \
    if (h->G == GG) {                                                       \
        return h->W == WKB ? run_tma_wait_check<GG, WKB>(h, st)             \
                           : run_tma_wait_check<GG, WGAUSS>(h, st);         \
    }
    PT_RADON_GRIDS(PT_CASE)
#undef PT_CASE
    pt::set_error("radonusfft: no kernel for grid %d", h->G);
    return PT_ERR_UNSUPPORTED;
}

template <typename T>
int dmalloc(T **p, size_t count)
{
    cudaError_t e = cudaMalloc((void **)p, count * sizeof(T) + 16);
    if (e != cudaSuccess) {
        *p = nullptr;
        pt::set_error("cudaMalloc of %zu bytes failed: %s", count * sizeof(T), cudaGetErrorString(e));
        return PT_ERR_ALLOC;
    }
    return PT_OK;
}

// exp(dir 2 pi i m / L) times (-1)^neg, in double
float2 unit_root(long long m, int L, int dir, int neg)
{
    const double a = dir * 2.0 * M_PI * (double)(m % L) / L, s = (neg & 1) ? -1.0 : 1.0;
    return make_float2((float)(s * std::cos(a)), (float)(s * std::sin(a)));
}

// The twiddle tables of the handle's lengths (see ptfft::Exchange and fft3).
cudaError_t upload_twiddles(pt_radon *h)
{
    // extra(i2, k1): quarter turns (times dir) the table adds to W^(i2 k1)
    auto pairs = [](int L, int dir, auto &&extra) {
        const int R1 = ptfft::split_r1(L), R2 = ptfft::split_r2(L);
        std::vector<float4> t((size_t)L / 2);
        for (int j = 0; j < R1 / 2; ++j)
            for (int i2 = 0; i2 < R2; ++i2) {
                float2 w[2];
                for (int o = 0; o < 2; ++o) {
                    const int k1 = 2 * j + o;
                    w[o] = unit_root((long long)i2 * k1 + (long long)extra(i2, k1) * (L / 4), L, dir, 0);
                }
                t[(size_t)j * R2 + i2] = make_float4(w[0].x, w[0].y, w[1].x, w[1].y);
            }
        return t;
    };
    const int G = h->G, N = h->N;
    // (-i)^k1 of the shifted rows times (-1)^k1, in quarter turns of exp(-2 pi i / 4): 3 k1
    const auto fwd = pairs(G, -1, [](int, int k1) { return 3 * k1; });
    const auto adj = pairs(G, +1, [](int i2, int) { return 2 * i2; });
    const auto lf = pairs(N, -1, [](int i2, int k1) { return 2 * (i2 + k1); });
    const auto li = pairs(N, +1, [](int i2, int k1) { return 2 * (i2 + k1); });
    const int A = ptfft::split3_a(G), C = ptfft::split3_c(G), B = ptfft::split3_b(G), BC = B * C;
    std::vector<float2> t1(G), t2(BC);
    for (int k1 = 0; k1 < A; ++k1)
        for (int i = 0; i < BC; ++i) t1[(size_t)k1 * BC + i] = unit_root((long long)i * k1, G, +1, 0);
    for (int k2 = 0; k2 < B; ++k2)
        for (int i3 = 0; i3 < C; ++i3) t2[(size_t)k2 * C + i3] = unit_root((long long)i3 * k2, BC, +1, i3);
    struct {
        void *dst;
        const void *src;
        size_t bytes;
    } up[] = {{h->tw_fwd, fwd.data(), fwd.size() * sizeof(float4)},    {h->tw_adj, adj.data(), adj.size() * sizeof(float4)},
              {h->tw_fwd_line, lf.data(), lf.size() * sizeof(float4)}, {h->tw_inv_line, li.data(), li.size() * sizeof(float4)},
              {h->tw_col1, t1.data(), t1.size() * sizeof(float2)},     {h->tw_col2, t2.data(), t2.size() * sizeof(float2)}};
    for (const auto &u : up) {
        const cudaError_t e = cudaMemcpy(u.dst, u.src, u.bytes, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int check_device(const pt_radon *h)
{
    int dev = -1;
    PT_CUDA(cudaGetDevice(&dev));
    if (dev != h->device) {
        pt::set_error("radonusfft handle belongs to device %d, current device is %d", h->device, dev);
        return PT_ERR_ARG;
    }
    return PT_OK;
}

}  // namespace

extern "C" int pt_radon_create_ex(size_t ntheta, size_t nz, size_t n, int m_override, pt_radon **out)
{
    pt::clear_error();
    PT_CHECK_ARG(out != nullptr, "radonusfft: null output handle");
    *out = nullptr;
    PT_CHECK_ARG(ntheta >= 1 && ntheta <= (1u << 20), "radonusfft: bad Ntheta %zu", ntheta);
    PT_CHECK_ARG(nz >= 1 && nz <= (1u << 20), "radonusfft: bad Nz %zu", nz);
    PT_CHECK_ARG(n >= 8 && n % 8 == 0, "radonusfft: n=%zu must be a positive multiple of 8", n);
    PT_CHECK_ARG(ntheta * (3 * n / 2) < ((size_t)1 << 23), "radonusfft: Ntheta*3n/2 = %zu polar points exceed 2^23",
                 ntheta * (3 * n / 2));
    PT_CHECK_ARG(m_override == 0 || m_override == 4 || m_override == 7,
                 "radonusfft: kernel half-width override %d not compiled (0, 4 or 7)", m_override);
    const int G = (int)(3 * n);
    if (!grid_supported(G)) {
        pt::set_error("radonusfft: n=%zu not compiled (supported n: 8,16,32,64,128,256,512)", n);
        return PT_ERR_UNSUPPORTED;
    }
    pt_radon *h = new pt_radon();
    h->ntheta = (int)ntheta;
    h->nz = (int)nz;
    h->n = (int)n;
    radon_params((int)n, m_override, &h->N, &h->M, &h->mu);
    h->G = G;
    if (cudaGetDevice(&h->device) != cudaSuccess) {
        delete h;
        pt::set_error("radonusfft: no CUDA device");
        return PT_ERR_CUDA;
    }
    if (h->M != 7 && h->M != 4) {
        pt::set_error("radonusfft: reference half-width M=%d has no compiled kernel", h->M);
        delete h;
        return PT_ERR_UNSUPPORTED;
    }
    h->W = h->M == 7 ? WKB : WGAUSS;
    int rc = PT_OK;
    const size_t N = h->N;
    const size_t npts = ntheta * N;
    // cuts of one allocation, each on a 256-byte boundary: the first pass adds up, the second places
    auto carve = [&](char *&base, auto &&cuts) {
        size_t used = 0;
        auto cut = [&](auto *&p, size_t count) {
            if (base) p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + used);
            used += (count * sizeof(*p) + 255) / 256 * 256;
        };
        cuts(cut);
        if (rc == PT_OK) rc = dmalloc(&base, used);
        used = 0;
        if (rc == PT_OK) cuts(cut);
    };
    carve(h->tables, [&](auto &cut) {
        cut(h->tw_fwd, (size_t)G / 2);
        cut(h->tw_adj, (size_t)G / 2);
        cut(h->tw_fwd_line, N / 2);
        cut(h->tw_inv_line, N / 2);
        cut(h->tw_col1, (size_t)G);
        cut(h->tw_col2, (size_t)G);
        cut(h->theta, ntheta);
        cut(h->x, npts);
        cut(h->y, npts);
        cut(h->org, 2 * npts);
        cut(h->wtab, 2 * (size_t)h->W * npts);
        cut(h->perm, npts);
        cut(h->rec, REC4 * npts);
        if (N <= FUSED_N) cut(h->rec_pt, REC4 * npts);
        cut(h->deap, N * N);
        if (h->W == WKB) cut(h->inv1, N);
        cut(h->goff, (size_t)G * (G / CG) + 1);
        cut(h->col_order, (size_t)G);
        cut(h->tma_err, 1);
    });
    carve(h->sets, [&](auto &cut) {
        for (int k = 0; k < RSETS; ++k) {
            cut(h->rbuf[k], N * G * ZC);
            cut(h->fgrid[k], (size_t)(G + GH_ROWS) * (G + 2 * GH_PAIRS) * ZC);
        }
    });
    if (rc == PT_OK && cudaMemset(h->tma_err, 0, sizeof(int)) == cudaSuccess)
        h->tma_ok = encode_grid_maps(h);   // gather 2 is offered only if every map encodes
    // default variant: two pipelines of two chunks per launch, TMA-staged tiles
    // (or the gather and the lines in one launch, see FUSED_N).
    // Against four pipelines of one (us): 64 wide, 64 slices, 96 angles 50 and 57;
    // 128 x 84 slices, 128 angles 123 and 124; 128^3, 128 angles 171 and 172, 192
    // angles 202 to 214 and 205; 256^3, 384 angles 1359 and 1355.  One pipeline of
    // four is slower from 64 slices up (55, 144, 205, 230, 1497)
    h->streams = 2;
    const size_t inflight = npts * std::min<size_t>((nz + ZC - 1) / ZC, RSETS);
    h->gather = N <= FUSED_N && inflight <= FUSED_POINTS ? 0 : h->tma_ok ? 2 : 1;
    if (rc == PT_OK && cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming) != cudaSuccess) rc = PT_ERR_CUDA;
    for (int k = 0; k < RSETS - 1 && rc == PT_OK; ++k)
        if (cudaStreamCreateWithFlags(&h->side[k], cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&h->ev_join[k], cudaEventDisableTiming) != cudaSuccess)
            rc = PT_ERR_CUDA;
    if (rc == PT_ERR_CUDA) pt::set_error("radonusfft: stream/event creation failed");
    h->nzp = (int)((nz + ZQ - 1) / ZQ * ZQ);
    const size_t nzp = h->nzp;
    if (rc == PT_OK) rc = dmalloc(&h->lines, ntheta * N * nzp);
    // all N rows of the padded slice (the exact adjoint's fold needs them; the
    // reference adjoint uses the first n)
    if (rc == PT_OK) rc = dmalloc(&h->rbuf_adj, N * (size_t)G * nzp);
    if (rc == PT_OK) rc = dmalloc(&h->mbuf, (n / 2 + 2) * (size_t)nz * n);
    if (rc == PT_OK) rc = radon_set_attrs(G);
    if (rc == PT_OK) {
        if (upload_twiddles(h) != cudaSuccess) rc = PT_ERR_CUDA;
        if (rc == PT_OK && h->inv1) {
            // transform of I0(beta sqrt(1 - (2 d / W)^2)) / I0(beta) (d in cells of
            // the G grid) at pixel t: W sinh(s) / s / I0(beta), s^2 = beta^2 - (pi W t / G)^2
            std::vector<double> inv(N);
            const double i0b = std::cyl_bessel_i(0.0, KB_BETA);
            for (size_t i = 0; i < N; ++i) {
                const double w = M_PI * WKB * ((double)i - (double)(N / 2)) / G;
                const double sq = std::sqrt(KB_BETA * KB_BETA - w * w);
                inv[i] = i0b * sq / (WKB * std::sinh(sq));
            }
            if (cudaMemcpy(h->inv1, inv.data(), N * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
                rc = PT_ERR_CUDA;
        }
        if (rc != PT_OK) pt::set_error("radonusfft: twiddle upload failed");
    }
    if (rc != PT_OK) {
        radon_free(h);
        delete h;
        return rc;
    }
    *out = h;
    return PT_OK;
}

extern "C" int pt_radon_create(size_t ntheta, size_t nz, size_t n, pt_radon **out)
{
    return pt_radon_create_ex(ntheta, nz, n, 0, out);
}

extern "C" int pt_radon_destroy(pt_radon *h)
{
    pt::clear_error();
    if (!h) return PT_OK;
    radon_free(h);
    delete h;
    return PT_OK;
}

extern "C" int pt_radon_setobj(pt_radon *h, const float *theta, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "radonusfft.setobj: null handle");
    PT_CHECK_ARG(theta != nullptr, "radonusfft.setobj: null theta");
    int rc = check_device(h);
    if (rc != PT_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    h->ready = false;
    const int N = h->N, G = h->G, W = h->W, left = W == WKB ? win_left<WKB>() : win_left<WGAUSS>(), ntheta = h->ntheta;
    PT_CUDA(cudaMemcpyAsync(h->theta, theta, ntheta * sizeof(float), cudaMemcpyDefault, st));
    k_takexy<<<dim3((N + 127) / 128, ntheta), 128, 0, st>>>(h->x, h->y, h->theta, N, ntheta);
    PT_LAUNCHED("k_takexy");
    k_deap_table<<<dim3((N + 127) / 128, N), 128, 0, st>>>(h->deap, N, h->mu, h->inv1);
    PT_LAUNCHED("k_deap_table");
    const size_t npts = (size_t)ntheta * N;
    std::vector<float> xs(npts), ys(npts);
    PT_CUDA(cudaMemcpyAsync(xs.data(), h->x, npts * sizeof(float), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaMemcpyAsync(ys.data(), h->y, npts * sizeof(float), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaStreamSynchronize(st));
    // window origins on the G grid, from floor(2N x) exactly as kernels.cuh:112-115 (float product)
    std::vector<int> org(2 * npts);
    for (size_t p = 0; p < npts; ++p) {
        if (!(xs[p] >= -0.5f && xs[p] < 0.5f && ys[p] >= -0.5f && ys[p] < 0.5f)) {
            pt::set_error("radonusfft.setobj: theta[%zu] is not a finite angle", p / N);
            h->ready = false;
            return PT_ERR_ARG;
        }
        org[2 * p] = ((N + (int)floorf((float)G * xs[p]) - left) % G + G) % G;
        org[2 * p + 1] = ((N + (int)floorf((float)G * ys[p]) - left) % G + G) % G;
    }
    PT_CUDA(cudaMemcpyAsync(h->org, org.data(), 2 * npts * sizeof(int), cudaMemcpyHostToDevice, st));
    {
        const float a = (float)(PI_REF * PI_REF / h->mu);
        const unsigned blocks = (unsigned)((npts * 2 * W + 255) / 256);
        const double i0b = std::cyl_bessel_i(0.0, KB_BETA);
        if (W == WKB)
            k_window<WKB><<<blocks, 256, 0, st>>>(h->x, h->y, h->wtab, (int)npts, G, a, i0b);
        else
            k_window<WGAUSS><<<blocks, 256, 0, st>>>(h->x, h->y, h->wtab, (int)npts, G, a, i0b);
        PT_LAUNCHED("k_window");
    }
    {   // the forward gather's visiting order: by the grid tile of the window origin, the parity of
        // its first column, then point index
        std::vector<int> perm(npts);
        std::vector<unsigned> tile(npts);
        const int TPR = (G + GTILE - 1) / GTILE;
        for (size_t p = 0; p < npts; ++p) {
            perm[p] = (int)p;
            tile[p] = (unsigned)((org[2 * p + 1] / GTILE) * TPR + org[2 * p] / GTILE);
        }
        auto key = [&](int i) { return 2 * tile[i] + (unsigned)(org[2 * (size_t)i] & 1); };
        std::stable_sort(perm.begin(), perm.end(), [&](int i, int j) { return key(i) < key(j); });
        PT_CUDA(cudaMemcpyAsync(h->perm, perm.data(), npts * sizeof(int), cudaMemcpyHostToDevice, st));
        const unsigned blocks = (unsigned)((npts + 255) / 256);
        auto records = [&](const int *order, float4 *rec) {
            if (W == WKB)
                k_point_records<WKB><<<blocks, 256, 0, st>>>(order, h->org, h->wtab, (float *)rec, (int)npts,
                                                             radon_pre(h));
            else
                k_point_records<WGAUSS><<<blocks, 256, 0, st>>>(order, h->org, h->wtab, (float *)rec, (int)npts,
                                                                radon_pre(h));
        };
        records(h->perm, h->rec);
        if (h->rec_pt) records(nullptr, h->rec_pt);
        PT_LAUNCHED("k_point_records");
        // the tiled gather's blocks: runs of one tile in perm order, at most tile_points points each
        std::vector<int4> chunks;
        for (size_t i = 0; i < npts;) {
            size_t j = i;
            while (j < npts && tile[perm[j]] == tile[perm[i]]) ++j;
            const int t = (int)tile[perm[i]];
            const size_t most = N <= 192 ? tile_points<192>() : tile_points<384>();
            for (size_t f = i; f < j; f += most)
                chunks.push_back(make_int4(t / TPR, t % TPR, (int)f, (int)std::min(most, j - f)));
            i = j;
        }
        if ((int)chunks.size() > h->chunks_cap) {
            if (h->chunks) cudaFree(h->chunks);
            h->chunks = nullptr;
            h->chunks_cap = 0;
            PT_CUDA(cudaMalloc(&h->chunks, chunks.size() * sizeof(int4)));
            h->chunks_cap = (int)chunks.size();
        }
        h->nchunks = (int)chunks.size();
        PT_CUDA(cudaMemcpy(h->chunks, chunks.data(), chunks.size() * sizeof(int4), cudaMemcpyHostToDevice));
    }
    // cell-group lists for the adjoint: a group is CG consecutive rows of one
    // grid column; every point is listed, in increasing point order, in each
    // group that its W x W window (mod G: the reference's halo fold,
    // kernels.cuh:67-82) touches, with the window column i0 and row offset r0.
    const int NG4 = G / CG;
    const size_t ngroups = (size_t)G * NG4;
    std::vector<int> off(ngroups + 1, 0);
    int cols[32], grp_first[8], ngrp = 0, oy = 0;
    auto window = [&](size_t p) {
        const int ox = org[2 * p];
        oy = org[2 * p + 1];
        for (int i = 0; i < W; ++i) cols[i] = (ox + i) % G;
        ngrp = 0;
        for (int i = 0; i < W; ++i) {
            const int gi = ((oy + i) % G) / CG;
            if (ngrp == 0 || grp_first[ngrp - 1] != gi) grp_first[ngrp++] = gi;
        }
    };
    for (size_t p = 0; p < npts; ++p) {
        window(p);
        for (int i0 = 0; i0 < W; ++i0)
            for (int k = 0; k < ngrp; ++k) off[(size_t)cols[i0] * NG4 + grp_first[k] + 1]++;
    }
    for (size_t c = 0; c < ngroups; ++c) off[c + 1] += off[c];
    const size_t total = (size_t)off[ngroups];
    std::vector<unsigned> keys(total);
    {
        std::vector<int> pos(off.begin(), off.end() - 1);
        for (size_t p = 0; p < npts; ++p) {
            window(p);
            for (int k = 0; k < ngrp; ++k) {
                int r0 = ((grp_first[k] * CG - oy) % G + G) % G;  // row offset of the group's first cell
                if (r0 > G - CG) r0 -= G;                          // in [-(CG-1), W-1]
                for (int i0 = 0; i0 < W; ++i0)
                    keys[pos[(size_t)cols[i0] * NG4 + grp_first[k]]++] =
                        ((unsigned)p << 9) | ((unsigned)i0 << 5) | (unsigned)(r0 + 3);
            }
        }
    }
    // columns ordered by decreasing work so the heavy centre columns start first
    std::vector<long long> colw(G, 0);
    for (int c = 0; c < G; ++c) colw[c] = off[(size_t)(c + 1) * NG4] - off[(size_t)c * NG4];
    std::vector<int> order(G);
    for (int i = 0; i < G; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int i, int j) { return colw[i] > colw[j]; });
    if (total > h->entries_cap) {
        if (h->gpt) cudaFree(h->gpt);
        if (h->gw) cudaFree(h->gw);
        h->gpt = nullptr;
        h->gw = nullptr;
        h->entries_cap = 0;
        rc = dmalloc(&h->gpt, total);
        if (rc == PT_OK) rc = dmalloc(&h->gw, total);
        if (rc != PT_OK) return rc;
        h->entries_cap = total;
    }
    unsigned *dkeys = nullptr;
    rc = dmalloc(&dkeys, total);
    if (rc != PT_OK) return rc;
    cudaError_t e1 = cudaMemcpy(dkeys, keys.data(), total * sizeof(unsigned), cudaMemcpyHostToDevice);
    if (e1 == cudaSuccess) {
        const unsigned blocks = (unsigned)((total + 255) / 256);
        if (W == WKB)
            k_make_entries<WKB><<<blocks, 256, 0, st>>>(dkeys, h->gpt, h->gw, total, h->wtab);
        else
            k_make_entries<WGAUSS><<<blocks, 256, 0, st>>>(dkeys, h->gpt, h->gw, total, h->wtab);
        e1 = cudaGetLastError();
        if (e1 == cudaSuccess) e1 = cudaStreamSynchronize(st);
    }
    cudaFree(dkeys);
    if (e1 != cudaSuccess) {
        pt::set_error("radonusfft.setobj: building the adjoint lists failed: %s", cudaGetErrorString(e1));
        return PT_ERR_CUDA;
    }
    PT_CUDA(cudaMemcpy(h->goff, off.data(), (ngroups + 1) * sizeof(int), cudaMemcpyHostToDevice));
    PT_CUDA(cudaMemcpy(h->col_order, order.data(), G * sizeof(int), cudaMemcpyHostToDevice));
    h->ready = true;
    return PT_OK;
}

namespace {
int radon_call(pt_radon *h, bool adj, void *out, const void *in, float scale, void *stream, bool exact = false)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "radonusfft: null handle");
    PT_CHECK_ARG(out != nullptr && in != nullptr, "radonusfft.%s: null array pointer", adj ? "adj" : "fwd");
    if (!h->ready) {
        pt::set_error("radonusfft.%s: setobj(theta) has not been called", adj ? "adj" : "fwd");
        return PT_ERR_STATE;
    }
    int rc = check_device(h);
    if (rc != PT_OK) return rc;
    return radon_dispatch(h, adj, (float2 *)out, (const float2 *)in, scale, (cudaStream_t)stream, exact);
}
}  // namespace

extern "C" int pt_radon_fwd(pt_radon *h, void *g, const void *f, void *stream)
{
    return radon_call(h, false, g, f, 1.0f, stream);
}
extern "C" int pt_radon_adj(pt_radon *h, void *f, const void *g, void *stream)
{
    return radon_call(h, true, f, g, 1.0f, stream);
}
extern "C" int pt_radon_fwd_scaled(pt_radon *h, void *g, const void *f, float scale, void *stream)
{
    return radon_call(h, false, g, f, scale, stream);
}
extern "C" int pt_radon_adj_scaled(pt_radon *h, void *f, const void *g, float scale, void *stream)
{
    return radon_call(h, true, f, g, scale, stream);
}

// Autotuner: times the forward with one, two and four pipelines, each with the
// three gathers, and keeps the fastest (setup-time; blocks the host).
extern "C" int pt_radon_autotune(pt_radon *h, void *g, const void *f, int trials, int *streams_out, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h && g && f && trials >= 1, "radonusfft.autotune: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    cudaEvent_t e0, e1;
    PT_CUDA(cudaEventCreate(&e0));
    PT_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    int best_s = h->streams, best_g = h->gather, rc = PT_OK;
    const int ngather = h->tma_ok ? 3 : 2;   // streams {1, 2, 4} x gather {L1, tiles, TMA tiles}
    for (int combo = 0; combo < 3 * ngather && rc == PT_OK; ++combo) {
        const int sc = 1 << (combo % 3);
        h->streams = sc;
        h->gather = combo / 3;
        std::vector<float> ts;
        for (int k = 0; k <= trials && rc == PT_OK; ++k) {
            cudaEventRecord(e0, st);
            rc = pt_radon_fwd(h, g, f, stream);
            cudaEventRecord(e1, st);
            if (rc == PT_OK && cudaEventSynchronize(e1) == cudaSuccess && k > 0) {
                float ms = 0;
                cudaEventElapsedTime(&ms, e0, e1);
                ts.push_back(ms);
            }
        }
        if (rc != PT_OK) break;
        std::sort(ts.begin(), ts.end());
        if (ts[ts.size() / 2] < best) {
            best = ts[ts.size() / 2];
            best_s = sc;
            best_g = h->gather;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    h->streams = best_s;
    h->gather = best_g;
    if (streams_out) *streams_out = best_s + 8 * best_g;
    if (rc == PT_OK && h->tma_ok) {   // a TMA tile load that never completed
        int flag = 0;
        PT_CUDA(cudaMemcpy(&flag, h->tma_err, sizeof(int), cudaMemcpyDeviceToHost));
        if (flag) {
            h->gather = 1;
            pt::set_error("radonusfft.autotune: a TMA tile load did not complete; TMA gather disabled");
            h->tma_ok = false;
            return PT_ERR_CUDA;
        }
    }
    return rc;
}

extern "C" int pt_radon_check_tma_wait(pt_radon *h, int *code, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h && code, "radonusfft.check_tma_wait: null pointer");
    if (!h->ready || !h->tma_ok) {
        pt::set_error("radonusfft.check_tma_wait: needs setobj and the TMA gather");
        return PT_ERR_STATE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    PT_CUDA(cudaMemsetAsync(h->tma_err, 0, sizeof(int), st));
    int rc = radon_tma_wait_check(h, st);
    if (rc != PT_OK) return rc;
    PT_CUDA(cudaMemcpyAsync(code, h->tma_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaStreamSynchronize(st));
    PT_CUDA(cudaMemsetAsync(h->tma_err, 0, sizeof(int), st));
    PT_CUDA(cudaStreamSynchronize(st));
    return PT_OK;
}

extern "C" int pt_radon_status(pt_radon *h, int *tma_timeouts, int *tma_available)
{
    pt::clear_error();
    PT_CHECK_ARG(h && tma_timeouts && tma_available, "radonusfft.status: null pointer");
    *tma_available = h->tma_ok ? 1 : 0;
    *tma_timeouts = 0;
    if (h->tma_err) {
        PT_CUDA(cudaMemcpy(tma_timeouts, h->tma_err, sizeof(int), cudaMemcpyDeviceToHost));
        PT_CUDA(cudaMemset(h->tma_err, 0, sizeof(int)));
    }
    return PT_OK;
}

int pt::radon_dims(const pt_radon *h, int *nz, int *ntheta)
{
    PT_CHECK_ARG(h != nullptr, "radonusfft: null handle");
    if (!h->ready) {
        pt::set_error("radonusfft: setobj(theta) has not been called");
        return PT_ERR_STATE;
    }
    *nz = h->nz;
    *ntheta = h->ntheta;
    return PT_OK;
}

extern "C" int pt_radon_set_variant(pt_radon *h, int streams, int gather)
{
    pt::clear_error();
    PT_CHECK_ARG(h && (streams == 1 || streams == 2 || streams == 4) && (gather >= 0 && gather <= 2),
                 "radonusfft.set_variant: streams 1, 2 or 4, gather 0 (L1), 1 (tiles) or 2 (TMA tiles)");
    if (gather == 2 && !h->tma_ok) {
        pt::set_error("radonusfft.set_variant: the TMA gather is not available (tensor map encoding failed)");
        return PT_ERR_UNSUPPORTED;
    }
    h->streams = streams;
    h->gather = gather;
    return PT_OK;
}

extern "C" int pt_radon_adj_exact(pt_radon *h, void *f, const void *g, float scale, void *stream)
{
    return radon_call(h, true, f, g, scale, stream, true);
}

extern "C" int pt_radon_get_params(const pt_radon *h, int *N, int *M, float *mu)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "radonusfft: null handle");
    if (N) *N = h->N;
    if (M) *M = h->M;
    if (mu) *mu = h->mu;
    return PT_OK;
}

extern "C" int pt_radon_get_xy(const pt_radon *h, float *x, float *y, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "radonusfft: null handle");
    if (!h->ready) {
        pt::set_error("radonusfft.get_xy: setobj(theta) has not been called");
        return PT_ERR_STATE;
    }
    const size_t bytes = (size_t)h->ntheta * h->N * sizeof(float);
    cudaStream_t st = (cudaStream_t)stream;
    if (x) PT_CUDA(cudaMemcpyAsync(x, h->x, bytes, cudaMemcpyDefault, st));
    if (y) PT_CUDA(cudaMemcpyAsync(y, h->y, bytes, cudaMemcpyDefault, st));
    return PT_OK;
}
