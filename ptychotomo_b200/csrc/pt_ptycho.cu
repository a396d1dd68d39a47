// Ptychography operator for sm_100a.
//
// Replaces class ptychofft of the reference (src/cuda/ptychofft.cu:1-93,
// kernels mul/mula/takeshifts/shifts/shiftsa in src/include/kernels.cuh).
//
//  forward  g = F Q psi   (ptychofft.cu:58-76): the probe-weighted patch
//    (detector row = object column, kernels.cuh:257-263) is loaded straight
//    into registers, transformed in three register rounds with two trips
//    through shared memory, and written with the per-scan phase
//    (kernels.cuh:306-336) applied.
//  adjoint  psi = Q* F* g (ptychofft.cu:78-93): the same transform in reverse;
//    block (part, angle) walks scans s = part, part + parts, ... in order and
//    accumulates conj(probe) x frame into its own slab; with parts > 1 the
//    slabs are summed in a fixed order by a second kernel.  Deterministic:
//    one block adds to a slab, and its frames' sums keep their order.
//  Detector 128x128 has its own kernels (k_ptycho_fwd128, k_ptycho_adj128): 32
//    values per thread, one 512-thread block per SM.  Few frames of 16x16 to
//    64x64 take k_ptycho_fwd_few (few_frames) and k_ptycho_adj_few (choose_split).
//  The adjoints also serve the residual-on-load and probe adjoints.
//  Detector 8x8 uses a plain shared-memory Stockham path.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <cstdint>
#include <functional>
#include <map>
#include <numeric>
#include <queue>
#include <type_traits>
#include <vector>

#include "pt_common.cuh"
#include "pt_fft.cuh"

namespace {

constexpr double PI_REF = 3.1415926535;  // kernels.cuh:1

// Residual of the ptycho data term applied to a frame value x on load
// (solver.py:220-224, D = dscale * data): RESID 0 = none (plain adjoint),
// 1 = Poisson x - D x / (|x|^2 + 1e-32), 2 = Gaussian x - sqrt(D) exp(i angle x).
template <int RESID>
__device__ __forceinline__ float2 resid_of(float2 x, float D)
{
    if constexpr (RESID == 1)
        return pt_residual_poisson(x, D);
    else if constexpr (RESID == 2)
        return pt_residual_gaussian(x, D);
    else
        return x;
}
template <int RESID>
__device__ __forceinline__ float2 resid(float2 x, const float *__restrict__ data, size_t idx, float dscale)
{
    if constexpr (RESID == 0)
        return x;
    else
        return resid_of<RESID>(x, __ldg(&data[idx]) * dscale);
}

// The hardware's 1/sqrt(x) and 1/x (relative error below 2^-22.9), for normal x.
__device__ __forceinline__ float rsqrt_normal(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float rcp_normal(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Residuals of a line of M frame values, v[m] with counts d[m] (unscaled; at
// `data` + m stride), without a branch for the ordinary values.  Poisson
// x - D x / b, b = |x|^2 + 1e-32: 1 / b is one Newton step from the hardware's
// approximation; Gaussian x (1 - sqrt(D) / |x|): sqrt(D) is one Heron step from
// D / sqrt(D), and 1 / |x| the approximation that pt_residual_gaussian takes.
// Either step gives the correctly rounded value: no difference from __frcp_rn
// for any b in [1e-32, 1e37] nor from __fsqrt_rn for any D in [1e-30, 1e37].  A
// value out of range (|x|^2 above 1e37; Poisson also D / b above 1e37; Gaussian
// also |x|^2 below 1e-30, or D not zero and outside these bounds, negative or
// not finite) makes the thread take pt_residual_* for it afterwards.  With a test and a call site per value
// and the rounded reciprocal or square root of the library, the det-128
// gradient of 45 angles with 100 to 400 scans took 1.81 ms Gaussian; it takes
// 1.48 ms.
template <int RESID, int M>
__device__ __forceinline__ void resid_line(float2 (&v)[M], float (&d)[M], float dscale, const float *__restrict__ data,
                                           int stride)
{
    if constexpr (RESID != 0) {
        unsigned rare = 0;
        float top = 0.f;   // Poisson: one maximum per value, and one test per line
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float D = d[m] * dscale;
            const float a2 = v[m].x * v[m].x + v[m].y * v[m].y;
            if constexpr (RESID == 1) {
                const float b = a2 + 1e-32f, y = rcp_normal(b);
                d[m] = D * fmaf(fmaf(-b, y, 1.f), y, y);
                top = fmaxf(top, fmaxf(b, fabsf(d[m])));   // a NaN makes its value NaN without further care
                continue;
            }
            const float z = rsqrt_normal(D), s0 = D * z;
            float s = fmaf(fmaf(-s0, s0, D), 0.5f * z, s0);
            if (D == 0.f) s = 0.f;
            if (!(a2 >= 1e-30f && a2 <= 1e37f && (D == 0.f || (D >= 1e-30f && D <= 1e37f)))) rare |= 1u << m;
            d[m] = s * rsqrt_normal(a2);
        }
        if (RESID == 1 && top > 1e37f) {
#pragma unroll
            for (int m = 0; m < M; ++m)
                if (fmaxf(v[m].x * v[m].x + v[m].y * v[m].y, fabsf(d[m])) > 1e37f) rare |= 1u << m;
        }
        if (rare) {
#pragma unroll
            for (int m = 0; m < M; ++m)
                if (rare >> m & 1) {
                    v[m] = resid_of<RESID>(v[m], __ldg(&data[m * stride]) * dscale);
                    d[m] = 0.f;
                }
        }
#pragma unroll
        for (int m = 0; m < M; ++m) v[m] = make_float2(v[m].x - d[m] * v[m].x, v[m].y - d[m] * v[m].y);
    }
}

template <int DET>
constexpr int ptycho_fft_threads() { return (512 / DET) < 4 ? 4 : ((512 / DET) > 32 ? 32 : 512 / DET); }
template <int DET>
constexpr int ptycho_block() { return DET * ptycho_fft_threads<DET>(); }

// setobj tables: integer corners (kernels.cuh:255-256) and the per-scan
// phase shiftx*shifty (takeshifts, kernels.cuh:306-317, same expressions);
// frac: the offsets s - round(s) in [-1/2, 1/2] (the sub-pixel model's shifts).
__global__ void k_ptycho_tables(const float *__restrict__ scan, int *__restrict__ corner,
                                float2 *__restrict__ phase, float *__restrict__ frac, int nframes)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nframes) return;
    const float sx = scan[i], sy = scan[nframes + i];
    corner[2 * i] = (int)roundf(sx);
    corner[2 * i + 1] = (int)roundf(sy);
    frac[2 * i] = sx - roundf(sx);
    frac[2 * i + 1] = sy - roundf(sy);
    float2 px, py;
    px.x = cosf(2 * PI_REF * (sx - roundf(sx)));
    px.y = sinf(2 * PI_REF * (sx - roundf(sx)));
    py.x = cosf(2 * PI_REF * (sy - roundf(sy)));
    py.y = sinf(2 * PI_REF * (sy - roundf(sy)));
    phase[i] = cmul(px, py);
}

template <int DET>
__global__ void __launch_bounds__(ptycho_block<DET>(), 1)
    k_ptycho_fwd_small(const float2 *__restrict__ psi, float2 *__restrict__ g, const int *__restrict__ corner,
                 const float2 *__restrict__ phase, const float2 *__restrict__ prb, int nz, int n, int nscan,
                 int P, float c, float scale, const float2 *__restrict__ tw)
{
    constexpr int T = ptycho_fft_threads<DET>(), NT = ptycho_block<DET>(), PITCH = DET + 1;
    extern __shared__ float2 fr[];
    const int s = blockIdx.x, th = blockIdx.y;
    const int fid = th * nscan + s;
    const int stx = corner[2 * fid], sty = corner[2 * fid + 1];
    float2 *out = g + (size_t)fid * DET * DET;
    if (stx < 0 || sty < 0) {  // skipped scan: the reference leaves a zero frame
        for (int e = threadIdx.x; e < DET * DET; e += NT) out[e] = czero();
        return;
    }
    if (P < DET) {
        for (int e = threadIdx.x; e < DET * DET; e += NT) fr[(e / DET) * PITCH + e % DET] = czero();
        __syncthreads();
    }
    const int off = (DET - P) / 2;
    const float2 *src = psi + ((size_t)th * nz + sty) * n + stx;
    for (int e = threadIdx.x; e < P * P; e += NT) {
        const int iy = e / P, ix = e % P;
        const float2 v = src[(size_t)iy * n + ix];
        const float2 pr = prb[ix * P + iy];
        fr[(off + ix) * PITCH + off + iy] = c * cmul(pr, v);
    }
    __syncthreads();
    const int f = threadIdx.x / T, t = threadIdx.x % T;
    ptfft::fft<DET, -1, T>(fr + f * PITCH, 1, t, tw);  // along the detector row
    ptfft::fft<DET, -1, T>(fr + f, PITCH, t, tw);      // along the detector column
    const float2 ph = scale * phase[fid];
    for (int e = threadIdx.x; e < DET * DET; e += NT) out[e] = cmul(fr[(e / DET) * PITCH + e % DET], ph);
}

template <int DET, int RESID>
__global__ void __launch_bounds__(ptycho_block<DET>(), 1)
    k_ptycho_adj_small(const float2 *__restrict__ g, float2 *__restrict__ psi, const int *__restrict__ corner,
                 const float2 *__restrict__ phase, const float2 *__restrict__ prb, int nz, int n, int nscan,
                 int P, float c, float scale, const float2 *__restrict__ tw, const float *__restrict__ data,
                 float dscale)
{
    constexpr int T = ptycho_fft_threads<DET>(), NT = ptycho_block<DET>(), PITCH = DET + 1;
    extern __shared__ float2 fr[];
    const int th = blockIdx.x;
    float2 *slab = psi + (size_t)th * nz * n;
    for (int e = threadIdx.x; e < nz * n; e += NT) slab[e] = czero();
    __syncthreads();
    const int off = (DET - P) / 2;
    const int f = threadIdx.x / T, t = threadIdx.x % T;
    const float cs = c * scale;
    for (int s = 0; s < nscan; ++s) {
        const int fid = th * nscan + s;
        const int stx = corner[2 * fid], sty = corner[2 * fid + 1];
        if (stx < 0 || sty < 0) continue;
        const float2 ph = phase[fid];
        const float2 *in = g + (size_t)fid * DET * DET;
        for (int e = threadIdx.x; e < DET * DET; e += NT)
            fr[(e / DET) * PITCH + e % DET] = cmulc(ph, resid<RESID>(in[e], data, (size_t)fid * DET * DET + e, dscale));
        __syncthreads();
        ptfft::fft<DET, +1, T>(fr + f * PITCH, 1, t, tw);
        ptfft::fft<DET, +1, T>(fr + f, PITCH, t, tw);
        float2 *dst = slab + (size_t)sty * n + stx;
        for (int e = threadIdx.x; e < P * P; e += NT) {
            const int iy = e / P, ix = e % P;
            const float2 v = cs * cmulc(prb[ix * P + iy], fr[(off + ix) * PITCH + off + iy]);
            float2 *d = dst + (size_t)iy * n + ix;
            *d = *d + v;
        }
        __syncthreads();
    }
}


// ---- frames of det x det, det = 16 to 64, in three register rounds -----------
// B[u][v] = f sum_{r,q} A[r][q] w^(DIR (u r + v q)), w = exp(2 pi i / det),
// for a det x det array A whose q runs along memory.  r = rt + RT m and
// u = k1 + 16 k2 split the r transform 16 x RT, q = qb + 16 qa and
// v = v1 + QA v2 the q transform QA x 16:
//   R1  thread (q, rt): 16-point DFT over m, times w^(rt k1)
//   R2  (k1, qb): RT-point DFT over rt (gives k2), QA-point DFT over qa
//       (gives v1), times w^(qb v1) f
//   R3  thread (u, v1): 16-point DFT over qb (gives v2)
// The forward takes A = probe x patch [y][x] and stores frame[kx = v][ky = u];
// the adjoint takes A = frame[kx][ky] and adds pixel [y = v][x = u].  Both
// touch memory in whole row segments.
//
// Between the rounds the frame sits in shared memory as rows (k1, j) of 16
// values qb, j = qa RT + rt after R1 and v1 RT + k2 after R2: R2 reads and
// writes the same slots, so it needs no barrier of its own.  The row's 16-byte
// slots are XORed with k1 & 7, so R3's 16-byte reads of eight consecutive u
// fall on eight different slots; every access takes the minimum number of
// wavefronts.
//
// 16 values per thread keep the kernels at 80 registers, so several blocks
// share an SM and one's loads and stores run under another's arithmetic; a
// row / transpose / column form with 512-thread blocks ran one block per SM
// with four barriers per frame.  A probe smaller than the detector leaves
// most of A zero (forward) or most of B unused (adjoint): R1 (R3) then runs
// on the probe's columns only, packed onto the first threads, and R2 skips
// the slots outside it.
// 192 angles x 225 scans, 64 x 64 detector, 16-pixel probe, forward: 1.04 ->
// 0.41 ms; Poisson gradient of 128 x 49 scans of a 64-pixel probe: 0.31 ->
// 0.14 ms.
template <int DET>
struct FR {
    static constexpr int QA = DET / 16, RT = DET / 16, J = QA * RT;
    static constexpr int NT = DET * QA;                  // threads per frame
    static constexpr int FPB = NT < 32 ? 32 / NT : 1;    // frames per block
    static constexpr int BLOCK = NT * FPB;
    static constexpr int R2C = 256 / NT;                 // (k1, qb) pairs per thread
    static constexpr int BPS = 768 / BLOCK;              // resident blocks per SM at 80 registers a thread
    static constexpr int BPSP = 512 / BLOCK;             // probe adjoint: 128 registers
    // Frames per trip, three barriers for both: two pay where a trip is long,
    // at 64 x 64 with a probe smaller than the detector.  Forward, where the
    // window lines of both fit the threads (P <= DET / 2) and every resident
    // block has two frames (280 x 15 scans, P 24: 53 -> 47 us; P 33 to 52
    // gain nothing, few frames lose 2 us); adjoint with the residual (70 x 341
    // scans, P 33: 468 -> 408 us; without it 178 x 66 scans, P 26: 137 ->
    // 147 us).  32 x 32 frames lose in all forms (5 x 340 scans, P 29:
    // forward 10 -> 14 us, adjoint 57 -> 79 us).
    static constexpr int nf_adj(bool full, bool resid) { return DET == 64 && !full && resid ? 2 : 1; }
    static constexpr size_t smem(int nf) { return (size_t)FPB * nf * DET * DET * sizeof(float2); }
    static_assert(DET * RT == NT, "R1 and R3 give every thread one line of 16");
};

// Byte offset of row (0, j), value qb, before the XOR of k1; row (k1, j) is
// k1 J rows of 128 bytes further on.  Written so that the compile-time index
// of each round (k1 in R1, the row j in R2, the slot in R3) is an XOR or an
// immediate offset on one register.
__device__ __forceinline__ unsigned fr_off(int j, int qb) { return ((unsigned)j << 7) + ((unsigned)qb << 3); }
__device__ __forceinline__ float2 *fr_ptr(float2 *ex, unsigned off) { return reinterpret_cast<float2 *>(reinterpret_cast<char *>(ex) + off); }

// R1 of a line v[m] = A[rt + RT m][q]; w holds exp(-2 pi i m / DET)
template <int DET, int DIR>
__device__ __forceinline__ void fr_r1(float2 (&v)[16], float2 *ex, int q, int rt, const float2 *__restrict__ w)
{
    constexpr int RT = FR<DET>::RT;
    ptfft::Dft<16, DIR, true>::run(v);
    if constexpr (RT > 1) {
#pragma unroll
        for (int k1 = 1; k1 < 16; ++k1) {
            float2 t = __ldg(&w[rt * k1]);
            if (DIR > 0) t.y = -t.y;
            v[k1] = cmul(v[k1], t);
        }
    }
    const unsigned o = fr_off((q >> 4) * RT + rt, q & 15);
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) *fr_ptr(ex, (o ^ ((k1 & 7) << 4)) + k1 * FR<DET>::J * 128) = v[k1];
}

// R2 in place.  in(q): whether R1 wrote column q (the others are zero);
// out(u): whether R3 reads row u.
template <int DET, int DIR, typename In, typename Out>
__device__ __forceinline__ void fr_r2(float2 *ex, int t, float2 f, const float2 *__restrict__ w, In in, Out out)
{
    using F = FR<DET>;
#pragma unroll
    for (int c = 0; c < F::R2C; ++c) {
        const int item = t + c * F::NT, k1 = item >> 4, qb = item & 15;
        float2 *s = fr_ptr(ex, (fr_off(0, qb) ^ ((k1 & 7) << 4)) + k1 * F::J * 128);
        float2 a[F::QA][F::RT];
#pragma unroll
        for (int qa = 0; qa < F::QA; ++qa) {
            const bool ok = in(qb + 16 * qa);
#pragma unroll
            for (int rt = 0; rt < F::RT; ++rt) a[qa][rt] = ok ? s[(qa * F::RT + rt) * 16] : czero();
            ptfft::Dft<F::RT, DIR, true>::run(a[qa]);
        }
#pragma unroll
        for (int k2 = 0; k2 < F::RT; ++k2) {
            float2 b[F::QA];
#pragma unroll
            for (int qa = 0; qa < F::QA; ++qa) b[qa] = a[qa][k2];
            ptfft::Dft<F::QA, DIR, true>::run(b);
#pragma unroll
            for (int v1 = 0; v1 < F::QA; ++v1) a[v1][k2] = b[v1];
        }
#pragma unroll
        for (int v1 = 0; v1 < F::QA; ++v1) {
            float2 t1 = f;
            if (v1 > 0) {
                t1 = __ldg(&w[qb * v1]);
                if (DIR > 0) t1.y = -t1.y;
                t1 = cmul(t1, f);
            }
#pragma unroll
            for (int k2 = 0; k2 < F::RT; ++k2)
                if (out(k1 + 16 * k2)) s[(v1 * F::RT + k2) * 16] = cmul(a[v1][k2], t1);
        }
    }
}

// R3's read of row (u, v1)
template <int DET>
__device__ __forceinline__ void fr_r3_read(float2 (&v)[16], const float2 *ex, int u, int v1)
{
    const int k1 = u & 15;
    const unsigned o = ((k1 * FR<DET>::J + v1 * FR<DET>::RT + (u >> 4)) << 7) + ((k1 & 7) << 4);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const float4 x = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(ex) + (o ^ (s << 4)));
        v[2 * s] = make_float2(x.x, x.y);
        v[2 * s + 1] = make_float2(x.z, x.w);
    }
}

// An opaque copy of a thread index: what is derived from it (slot and window
// addresses, twiddles) is formed where it is used in each frame, instead of
// being hoisted out of the frame loop into registers.
__device__ __forceinline__ int fresh(int t)
{
    asm volatile("mov.b32 %0, %0;" : "+r"(t));
    return t;
}

// *p += v in L2, without waiting for the sum: one FP32 addition per component,
// rounded as an add rounds it, but for subnormal inputs and results, which red
// flushes to zero on global memory (k_ptycho_adj_few keeps them).  Each frame
// adds to a pixel at most once and the frames of a block are separated by its
// barriers, so the order of the sums, and the result, is that of the frames.
__device__ __forceinline__ void add_l2(float2 *p, float2 v)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
}

// The lines of R1 (forward) or R3 (adjoint): RT lines of each window column,
// px + P r.  Thread t takes line t of the trip's first frame (A) and, with two
// frames per trip, a line of the second (B), on the threads that A leaves idle
// first, so a narrow probe's two frames run on different warps.
template <int DET, bool FULL, int FRAME>
__device__ __forceinline__ void fr_line(int t, int PW, int &px, int &r)
{
    const int lines = PW * FR<DET>::RT;
    const int l = FRAME == 0 ? t : (t >= lines ? t - lines : t + FR<DET>::NT - lines);
    px = l % PW;
    r = l / PW;      // valid if below RT
}

// Forward, grid-stride over frames, NF consecutive ones per trip.
template <int DET, bool FULL, bool SUB = false, int NF = 1>
__global__ void __launch_bounds__(FR<DET>::BLOCK, FR<DET>::BPS)
    k_ptycho_fwd(const float2 *__restrict__ psi, float2 *__restrict__ g, const int *__restrict__ corner,
                 const float2 *__restrict__ phase, const float2 *__restrict__ prbT, int nz, int n, int nscan,
                 int nframes, int P, float scale, const float2 *__restrict__ w, const int *__restrict__ sid = nullptr)
{
    using F = FR<DET>;
    extern __shared__ float4 sm4[];
    const int t0 = threadIdx.x % F::NT, sub = threadIdx.x / F::NT;
    float2 *ex = reinterpret_cast<float2 *>(sm4) + sub * DET * DET;
    const int PW = FULL ? DET : P, off0 = FULL ? 0 : (DET - P) / 2;
    int px0[NF], r0[NF];
    fr_line<DET, FULL, 0>(t0, PW, px0[0], r0[0]);
    if constexpr (NF == 2) fr_line<DET, FULL, 1>(t0, PW, px0[1], r0[1]);
    for (int f0 = blockIdx.x * F::FPB * NF; f0 < nframes; f0 += gridDim.x * F::FPB * NF) {
        int stx[NF], sty[NF];
        bool act[NF];
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int fid = f0 + sub + j;
            stx[j] = fid < nframes ? corner[2 * fid] : -1;
            sty[j] = fid < nframes ? corner[2 * fid + 1] : -1;
            act[j] = stx[j] >= 0 && sty[j] >= 0;
        }
        const int t = fresh(t0), off = FULL ? 0 : fresh(off0);
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            if (!act[j] || r0[j] >= F::RT) continue;
            const int fid = f0 + sub + j, px = fresh(px0[j]), rt = fresh(r0[j]);
            const float2 *src = psi + ((size_t)(fid / nscan) * nz + sty[j]) * n + stx[j] + px;
            const float2 *pr = (SUB ? prbT + (size_t)sid[fid] * P * P : prbT) + px;  // sub-pixel: the frame's shifted probe
            float2 v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                const int py = rt + F::RT * m - off;
                v[m] = FULL || (py >= 0 && py < P) ? cmul(__ldg(&pr[py * PW]), __ldg(&src[(size_t)py * n])) : czero();
            }
            fr_r1<DET, -1>(v, ex + j * DET * DET, off + px, rt, w);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NF; ++j)
            if (act[j])
                fr_r2<DET, -1>(ex + j * DET * DET, t, scale * phase[f0 + sub + j], w,
                               [&](int q) { return FULL || (q >= off && q < off + P); }, [](int) { return true; });
        __syncthreads();
        const int u = t % DET, v1 = t / DET;
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            float2 v[16];
            if (act[j]) fr_r3_read<DET>(v, ex + j * DET * DET, u, v1);
            if (j == NF - 1) __syncthreads();  // read: the next trip's R1 may write
            const int fid = f0 + sub + j;
            if (fid >= nframes) continue;
            float2 *out = g + (size_t)fid * DET * DET + v1 * DET + u;   // frame[kx = v1 + QA v2][ky = u]
            if (act[j]) {
                ptfft::Dft<16, -1, true>::run(v);
            } else {   // skipped scan: the reference leaves a zero frame
#pragma unroll
                for (int v2 = 0; v2 < 16; ++v2) v[v2] = czero();
            }
#pragma unroll
            for (int v2 = 0; v2 < 16; ++v2) __stcs(&out[F::QA * v2 * DET], v[v2]);
        }
    }
}

// Object adjoint: grid (parts, ntheta), block (part, angles[y]) owns slab
// dst[angle][part] and walks scans part, part + parts, ...  PROBE (the adjoint with respect to the
// probe): grid (blocks, 1), block b walks frames b, b + gridDim.x, ... <
// nframes and sums conj(psi patch) x frame into its P x P partial dst[b] (one
// per frame of the block); each element belongs to one thread, which keeps it
// in registers.
template <int DET, bool FULL, int RESID, bool SUB = false, bool PROBE = false>
__global__ void __launch_bounds__(FR<DET>::BLOCK, PROBE ? FR<DET>::BPSP : FR<DET>::BPS)
    k_ptycho_adj(const float2 *__restrict__ g, float2 *dst, const int *__restrict__ corner,
                 const float2 *__restrict__ phase, const float2 *prbT, int nz, int n, int nscan, int P, float scale,
                 const float2 *__restrict__ w, const float *__restrict__ data, float dscale,
                 const int *__restrict__ angles, const int *__restrict__ sid = nullptr,
                 const float2 *psi = nullptr, int nframes = 0)
{
    using F = FR<DET>;
    constexpr int NF = PROBE ? 1 : F::nf_adj(FULL, RESID != 0);
    extern __shared__ float4 sm4[];
    const int t0 = threadIdx.x % F::NT, sub = threadIdx.x / F::NT;
    float2 *ex = reinterpret_cast<float2 *>(sm4) + sub * DET * DET;
    const int part = blockIdx.x, parts = gridDim.x, th0 = PROBE ? 0 : angles[blockIdx.y];
    const int PW = FULL ? DET : P, off0 = FULL ? 0 : (DET - P) / 2;
    // R3's lines: window column px (= u - off), rows r + QA v2
    int px0[NF], r0[NF];
    fr_line<DET, FULL, 0>(t0, PW, px0[0], r0[0]);
    if constexpr (NF == 2) fr_line<DET, FULL, 1>(t0, PW, px0[1], r0[1]);
    float2 *slab = PROBE ? dst + (size_t)(part * F::FPB + sub) * P * P : dst + ((size_t)th0 * parts + part) * nz * n;
    if (!PROBE)
        for (int e = threadIdx.x; e < nz * n; e += F::BLOCK) slab[e] = czero();
    float2 acc[PROBE ? 16 : 1];
    if constexpr (PROBE) {
#pragma unroll
        for (int v2 = 0; v2 < 16; ++v2) acc[v2] = czero();
    }
    const int count = PROBE ? nframes : nscan;
    // frame j of the trip that starts at s0
    const int jstep = F::FPB > 1 ? 1 : parts;
    for (int s0 = part * F::FPB; s0 < count; s0 += parts * F::FPB * NF) {
        int stx[NF], sty[NF];
        bool act[NF];
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            const int s = s0 + sub + j * jstep, fid = PROBE ? s : th0 * nscan + s;
            stx[j] = s < count ? corner[2 * fid] : -1;
            sty[j] = s < count ? corner[2 * fid + 1] : -1;
            act[j] = stx[j] >= 0 && sty[j] >= 0;
        }
        if (F::FPB == 1 && !act[0] && !(NF == 2 && act[NF - 1])) continue;
        const int t = fresh(t0), off = FULL ? 0 : fresh(off0);
        auto frame = [&](int j) { return (PROBE ? 0 : th0 * nscan) + s0 + sub + j * jstep; };
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            if (!act[j]) continue;
            const int ky = t % DET, rt = t / DET;
            const size_t e0 = (size_t)frame(j) * DET * DET + rt * DET + ky;
            float2 v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = __ldcs(&g[e0 + m * F::RT * DET]);
            if constexpr (RESID != 0) {
                float d[16];
#pragma unroll
                for (int m = 0; m < 16; ++m) d[m] = __ldcs(&data[e0 + m * F::RT * DET]);
                resid_line<RESID>(v, d, dscale, data + e0, F::RT * DET);
            }
            fr_r1<DET, +1>(v, ex + j * DET * DET, ky, rt, w);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NF; ++j) {
            if (!act[j]) continue;
            const float2 ph = phase[frame(j)];
            fr_r2<DET, +1>(ex + j * DET * DET, t, make_float2(scale * ph.x, -scale * ph.y), w,
                           [](int) { return true; }, [&](int u) { return FULL || (u >= off && u < off + P); });
        }
        __syncthreads();
        // object: slab += conj(probe) x value; probe: sum of conj(psi) x value
        auto add = [&](int j, const float2 (&v)[16]) {
            const int px = fresh(px0[j]), v1 = fresh(r0[j]), fid = frame(j);
            const float2 *mul = (PROBE ? psi + ((size_t)(fid / nscan) * nz + sty[j]) * n + stx[j]
                                       : (SUB ? prbT + (size_t)sid[fid] * P * P : prbT)) + px;
            const size_t ms = PROBE ? n : PW;
            float2 *col = slab + (size_t)sty[j] * n + stx[j] + px;
            constexpr int RB = 8;   // multiplier loads in flight
#pragma unroll
            for (int h = 0; h < 16; h += RB) {
                float2 pv[RB];
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    const int py = v1 + F::QA * (h + i) - off;
                    pv[i] = FULL || (py >= 0 && py < P) ? __ldg(&mul[py * ms]) : czero();
                }
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    const int py = v1 + F::QA * (h + i) - off;
                    if (!FULL && (py < 0 || py >= P)) continue;
                    if constexpr (PROBE)
                        acc[h + i] = acc[h + i] + cmulc(pv[i], v[h + i]);
                    else
                        add_l2(&col[(size_t)py * n], cmulc(pv[i], v[h + i]));
                }
            }
        };
        float2 v[16];
        if constexpr (NF == 2) {
            // frame A's sums are queued before the barrier, B's after it
            if (act[0] && r0[0] < F::QA) {
                fr_r3_read<DET>(v, ex, off + fresh(px0[0]), r0[0]);
                ptfft::Dft<16, +1, true>::run(v);
                add(0, v);
            }
            const bool b = act[1] && r0[1] < F::QA;
            if (b) {
                fr_r3_read<DET>(v, ex + DET * DET, off + fresh(px0[1]), r0[1]);
                ptfft::Dft<16, +1, true>::run(v);
            }
            __syncthreads();  // read: the next trip's R1 may write
            if (b) add(1, v);
        } else {
            const bool a = act[0] && r0[0] < F::QA;
            if (a) fr_r3_read<DET>(v, ex, off + fresh(px0[0]), r0[0]);
            __syncthreads();  // read: the next trip's R1 may write
            if (a) ptfft::Dft<16, +1, true>::run(v);
            // frames of one block that share a slab add to it one after the other
#pragma unroll
            for (int o = 0; o < (PROBE ? 1 : F::FPB); ++o) {
                if (!PROBE && o > 0) __syncthreads();
                if (a && (PROBE || F::FPB == 1 || sub == o)) add(0, v);
            }
        }
    }
    if constexpr (PROBE) {
        if (r0[0] < F::QA) {
#pragma unroll
            for (int v2 = 0; v2 < 16; ++v2) {
                const int py = r0[0] + F::QA * v2 - off0;
                if (FULL || (py >= 0 && py < P)) slab[(size_t)py * P + px0[0]] = acc[v2];
            }
        }
    }
}

// ---- few frames: four or eight threads per line -------------------------------
// Where few blocks are in flight, a frame's latency counts, not the SM's
// instruction slots: the kernels above take 16 values per thread (16, 64 or 256
// threads per frame), these 4 or 8 (64, 128 or 512 threads): row transforms, a
// transpose through shared memory, column transforms.
// Adjoint: choose_split compares the modelled times.  16 x 16 frames, adjoint:
// 9 x 74 scans 18.5 -> 14.4 us, 65 x 14 scans on a 145 x 152 object 29 -> 20 us
// (more threads to clear its slabs); but 224 x 146 scans take 94 us here and
// 66 us there.
template <int DET>
struct PF {
    static constexpr int N2 = DET == 64 ? 8 : 4;           // threads per line
    static constexpr int N1 = DET / N2;                    // points per thread
    static constexpr int KPT = N1 / N2;                    // k1 values per thread after the exchange
    static constexpr int NT = DET * N2;                    // threads per block
    static constexpr int P = DET + 8;                      // frame pitch (P = 8 mod 16)
    // resident blocks of the adjoint per SM (80, 136 and 128 registers a thread)
    static constexpr int BPS = DET == 16 ? 12 : DET == 32 ? 3 : 1;
    static constexpr size_t SMEM = (size_t)(DET * P + DET) * sizeof(float2);
};

// frame swizzle: row r, column c live at r * P + (c ^ fswz(r))
template <int DET>
__device__ __forceinline__ int fswz(int r)
{
    return ((r / PF<DET>::KPT) % PF<DET>::N2) * 2;
}

// DFT of one line held as v[m] = x[t + N2 m] by the N2 threads t of a group.
// On return v[j N2 + k2] = X[t KPT + j + N1 k2].  `sc` is the group's
// scratch (DET + 1 complex), `tws` the table exp(-2 pi i m / DET).
template <int DET, int DIR>
__device__ __forceinline__ void line_dft(float2 (&v)[PF<DET>::N1], int t, float2 *sc, const float2 *tws)
{
    using F = PF<DET>;
    ptfft::Dft<F::N1, DIR>::run(v);
#pragma unroll
    for (int k1 = 1; k1 < F::N1; ++k1) {
        float2 w = tws[t * k1];
        if (DIR > 0) w.y = -w.y;
        v[k1] = cmul(v[k1], w);
    }
    __syncwarp();
#pragma unroll
    for (int k1 = 0; k1 < F::N1; ++k1) sc[t * F::N1 + ((k1 + t * F::KPT) % F::N1)] = v[k1];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < F::KPT; ++j) {
        float2 u[F::N2];
        const int k1 = t * F::KPT + j;
#pragma unroll
        for (int n2 = 0; n2 < F::N2; ++n2) u[n2] = sc[n2 * F::N1 + ((k1 + n2 * F::KPT) % F::N1)];
        ptfft::Dft<F::N2, DIR>::run(u);
#pragma unroll
        for (int k2 = 0; k2 < F::N2; ++k2) v[j * F::N2 + k2] = u[k2];
    }
}

// Forward: one frame per block, up to few_frames frames per SM.
template <int DET, bool SUB>
__global__ void __launch_bounds__(PF<DET>::NT, 1)
    k_ptycho_fwd_few(const float2 *__restrict__ psi, float2 *__restrict__ g, const int *__restrict__ corner,
                     const float2 *__restrict__ phase, const float2 *__restrict__ prbT, int nz, int n, int nscan, int P,
                     float scale, const float2 *__restrict__ tw, const int *__restrict__ sid)
{
    using F = PF<DET>;
    extern __shared__ float2 sm[];
    float2 *fr = sm;
    float2 *tws = sm + DET * F::P;
    const int fid = blockIdx.x;
    const int stx = corner[2 * fid], sty = corner[2 * fid + 1];
    float2 *out = g + (size_t)fid * DET * DET;
    if (stx < 0 || sty < 0) {   // skipped scan: the reference leaves a zero frame
        for (int e = threadIdx.x; e < DET * DET; e += F::NT) out[e] = czero();
        return;
    }
    for (int i = threadIdx.x; i < DET; i += F::NT) tws[i] = tw[i];
    const int t = threadIdx.x % F::N2, grp = threadIdx.x / F::N2;
    float2 *sc = fr + grp * (DET + 1);
    const int off = (DET - P) / 2, py = grp - off;
    const float2 *src = psi + ((size_t)(fid / nscan) * nz + sty) * n + stx;
    const float2 *pr = SUB ? prbT + (size_t)sid[fid] * P * P : prbT;  // sub-pixel: the frame's shifted probe
    // along the object row: line = detector column iy = grp, points ix = t + N2 m
    float2 v[F::N1];
#pragma unroll
    for (int m = 0; m < F::N1; ++m) {
        const int px = t + F::N2 * m - off;
        v[m] = py >= 0 && py < P && px >= 0 && px < P
                   ? cmul(__ldg(&pr[py * P + px]), __ldg(&src[(size_t)py * n + px]))
                   : czero();
    }
    __syncthreads();
    line_dft<DET, -1>(v, t, sc, tws);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < F::KPT; ++j)
#pragma unroll
        for (int k2 = 0; k2 < F::N2; ++k2) {
            const int kx = t * F::KPT + j + F::N1 * k2;
            fr[kx * F::P + (grp ^ fswz<DET>(kx))] = v[j * F::N2 + k2];
        }
    __syncthreads();
    const int sw = fswz<DET>(grp);
#pragma unroll
    for (int m = 0; m < F::N1; ++m) v[m] = fr[grp * F::P + ((t + F::N2 * m) ^ sw)];
    __syncthreads();
    const float2 ph = scale * phase[fid];
    line_dft<DET, -1>(v, t, sc, tws);
#pragma unroll
    for (int k2 = 0; k2 < F::N2; ++k2)
#pragma unroll
        for (int j = 0; j < F::KPT; ++j)
            out[grp * DET + t * F::KPT + j + F::N1 * k2] = cmul(v[j * F::N2 + k2], ph);
}

// Frames per SM up to which k_ptycho_fwd_few is the faster forward (us, this
// kernel and k_ptycho_fwd; P the probe's width; a probe smaller than the
// detector costs k_ptycho_fwd two launch steps of 1 us, this kernel nothing):
// det 16, P 16: 444 frames 4.1 and 5.7, 1776 6.2 and 6.2, 2072 7.2 and 6.2;
//         P 15: 444 frames 4.1 and 8.2, 2072 6.7 and 8.2, 2664 8.2 and 8.2;
// det 32, P 32: 148 frames 4.6 and 6.2, 296 6.2 and 6.2, 592 8.2 and 6.2;
//         P 24: 148 frames 4.1 and 8.2, 592 6.5 and 8.2, 1184 10.3 and 9.0;
// det 64, P 64: 148 frames 6.2 and 8.2, 222 9.2 and 8.2;
//         P 48: 148 frames 6.2 and 8.7, 296 8.2 and 10.2, 370 12.3 and 10.3.
constexpr int few_frames(int det, bool full)
{
    return det == 16 ? (full ? 12 : 16) : det == 32 ? (full ? 2 : 5) : (full ? 1 : 2);
}

// grid (parts, ntheta): block (part, angles[y]) owns slab dst[angle][part]
template <int DET, int RESID, bool SUB = false>
__global__ void __launch_bounds__(PF<DET>::NT, 1)
    k_ptycho_adj_few(const float2 *__restrict__ g, float2 *__restrict__ dst, const int *__restrict__ corner,
                 const float2 *__restrict__ phase, const float2 *__restrict__ prbT, int nz, int n, int nscan,
                 int P, float scale, const float2 *__restrict__ tw, const float *__restrict__ data, float dscale,
                 const int *__restrict__ angles, const int *__restrict__ sid)
{
    using F = PF<DET>;
    extern __shared__ float2 sm[];
    float2 *fr = sm;
    float2 *tws = sm + DET * F::P;
    // angles: null where all angles have the same number of scans (one load less
    // before the first frame: 1 us of 15)
    const int part = blockIdx.x, parts = gridDim.x, th = angles ? angles[blockIdx.y] : blockIdx.y;
    float2 *slab = dst + ((size_t)th * parts + part) * nz * n;
    for (int i = threadIdx.x; i < DET; i += F::NT) tws[i] = tw[i];
    for (int e = threadIdx.x; e < nz * n; e += F::NT) slab[e] = czero();
    const int t = threadIdx.x % F::N2, grp = threadIdx.x / F::N2;
    float2 *sc = fr + grp * (DET + 1);
    const int off = (DET - P) / 2;
    __syncthreads();
    for (int s = part; s < nscan; s += parts) {
        const int fid = th * nscan + s;
        const int stx = corner[2 * fid], sty = corner[2 * fid + 1];
        if (stx < 0 || sty < 0) continue;
        const float2 ph = phase[fid];
        const float2 *pr = SUB ? prbT + (size_t)sid[fid] * P * P : prbT;
        const float2 *in = g + (size_t)fid * DET * DET;
        float2 v[F::N1];
        // along the detector row: line kx = grp, points ky = t + N2 m (contiguous)
#pragma unroll
        for (int m = 0; m < F::N1; ++m) {
            const int e = grp * DET + t + F::N2 * m;
            v[m] = scale * cmulc(ph, resid<RESID>(__ldg(&in[e]), data, (size_t)fid * DET * DET + e, dscale));
        }
        line_dft<DET, +1>(v, t, sc, tws);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < F::KPT; ++j)
#pragma unroll
            for (int k2 = 0; k2 < F::N2; ++k2) {
                const int iy = t * F::KPT + j + F::N1 * k2;
                fr[iy * F::P + (grp ^ fswz<DET>(iy))] = v[j * F::N2 + k2];
            }
        __syncthreads();
        const int sw = fswz<DET>(grp);
#pragma unroll
        for (int m = 0; m < F::N1; ++m) v[m] = fr[grp * F::P + ((t + F::N2 * m) ^ sw)];
        __syncthreads();
        line_dft<DET, +1>(v, t, sc, tws);
        const int py = grp - off;
        if (py >= 0 && py < P) {
            float2 *row = slab + (size_t)(sty + py) * n + stx;
            float2 cur[F::N1];
#pragma unroll
            for (int k2 = 0; k2 < F::N2; ++k2)
#pragma unroll
                for (int j = 0; j < F::KPT; ++j) {
                    const int px = t * F::KPT + j + F::N1 * k2 - off;
                    cur[j * F::N2 + k2] = (px >= 0 && px < P) ? row[px] : czero();
                }
#pragma unroll
            for (int k2 = 0; k2 < F::N2; ++k2)
#pragma unroll
                for (int j = 0; j < F::KPT; ++j) {
                    const int px = t * F::KPT + j + F::N1 * k2 - off;
                    if (px >= 0 && px < P)
                        row[px] = cur[j * F::N2 + k2] + cmulc(__ldg(&pr[py * P + px]), v[j * F::N2 + k2]);
                }
        }
        __syncthreads();
    }
}

// ---- det = 128 ---------------------------------------------------------
// The same three rounds for a 128 x 128 frame, 32 values per thread and one
// 512-thread block per SM (the frame's exchange buffer takes 128 KB):
//   R1  thread (q = 32 g + lane, rt = w + 4 c, c = 0, 1): 16-point DFTs over m
//       of r = rt + 8 m, times w128^(rt k1)
//   R2  thread (k1 = warp, qb = lane): 8-point DFT over rt, u = k1 + 16 k2;
//       4-point DFT over qa of q = qb + 32 qa, v1; times w128^(qb v1) f
//   R3  thread (u = tid & 127, v1 = g): 32-point DFT over qb, v = v1 + 4 v2
// with g = tid >> 7 the thread's group of four warps and w its warp there.
// R1's lanes load 32 consecutive q (256 B of one row) and R3's lanes hold 32
// consecutive u, so every global access of a warp covers 256 bytes.
//
// The exchange rows (k1, j) hold 32 values qb (256 B, 16-byte slots XORed with
// k1 & 7), j = qa 8 + rt after R1 and v1 8 + k2 after R2, which works in place.
// Group g writes the rows qa = g in R1 and reads the rows v1 = g in R3: the
// same memory.  So a frame has two block-wide barriers, around R2; from R3 to
// the next frame's R1 a group waits for its own four warps only, and one
// group's loads and stores run under another's arithmetic.
//
// The probe table (128 KB) does not stay in the 100 KB of L1 that the exchange
// buffer leaves: rereading it cyclically hit 10 % (forward).  Its first 96 KB
// sit in shared memory instead, the rest is read through L2.
// 256^3, 384 angles x 169 scans on one raster: forward 3.75 -> 3.34 ms (a table
// of 64 KB costs 0.05, later patch loads 0.17 more), adjoint 4.26 -> 3.70 ms
// (jittered scans 4.4 -> 3.75 to 3.95).  The adjoint keeps 32 KB only: with 96
// KB in the table the L1 left for loads in flight is too small (4.00 ms; 16 KB
// 3.83, 48 KB 3.75).  The arithmetic and the exchange alone take 2.1 ms of the
// forward, the exchange 1.1 ms.
constexpr int P128_EX = 128 * 128 * 8;          // exchange buffer
constexpr int P128_FTAB = 96 * 1024, P128_ATAB = 32 * 1024;   // probe rows kept in shared memory: forward, adjoint
constexpr int P128_FSMEM = P128_EX + P128_FTAB, P128_ASMEM = P128_EX + P128_ATAB;

// The det-128 twiddles a thread needs, w(t k1) for k1 = 0..15, in pairs:
// entry q * 8 + t of the 64-entry float4 table holds w(2q t) and w((2q+1) t)
// (w = exp(-2 pi i / 128); DIR > 0 takes the conjugates).
template <int DIR>
__device__ __forceinline__ void twiddle16(float2 (&v)[16], float4 w, int q)
{
    float2 w0 = make_float2(w.x, w.y), w1 = make_float2(w.z, w.w);
    if (DIR > 0) {
        w0.y = -w0.y;
        w1.y = -w1.y;
    }
    if (q > 0) v[2 * q] = cmul(v[2 * q], w0);
    v[2 * q + 1] = cmul(v[2 * q + 1], w1);
}

// R1 of one line: v[m] = A[rt + 8 m][q].  tw4 is twiddle16's pair table; rt is
// the same across a warp, so its loads are broadcasts.
template <int DIR, bool PK>
__device__ __forceinline__ void f128_r1(float2 (&v)[16], float2 *ex, int q, int rt, const float4 *__restrict__ tw4)
{
    ptfft::Dft<16, DIR, PK>::run(v);
#pragma unroll
    for (int k = 0; k < 8; ++k) twiddle16<DIR>(v, __ldg(&tw4[k * 8 + rt]), k);
    const unsigned o = ((unsigned)((q >> 5) * 8 + rt) << 8) + ((unsigned)(q & 31) << 3);
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) *fr_ptr(ex, (o ^ ((k1 & 7) << 4)) + k1 * 8192) = v[k1];
}

// R2 in place for thread (k1 = warp, qb = lane).  The twiddles w128^(qb j)
// (j = 1..3, in direction DIR; w128[m] = exp(-2 pi i m / 128)) are multiplied
// by the frame factor f: the factor rides on them.
template <int DIR, bool PK>
__device__ __forceinline__ void f128_r2(float2 *ex, int t, float2 f, const float2 *__restrict__ w128)
{
    const int k1 = t >> 5, qb = t & 31;
    float2 rw1 = __ldg(&w128[qb]), rw2 = __ldg(&w128[2 * qb]), rw3 = __ldg(&w128[3 * qb]);
    if (DIR > 0) {
        rw1.y = -rw1.y;
        rw2.y = -rw2.y;
        rw3.y = -rw3.y;
    }
    float2 *s = fr_ptr(ex, (((unsigned)qb << 3) ^ ((k1 & 7) << 4)) + k1 * 8192);
    float2 a[4][8];
#pragma unroll
    for (int qa = 0; qa < 4; ++qa)
#pragma unroll
        for (int rt = 0; rt < 8; ++rt) a[qa][rt] = s[(qa * 8 + rt) * 32];
#pragma unroll
    for (int qa = 0; qa < 4; ++qa) ptfft::Dft<8, DIR, PK>::run(a[qa]);
    const float2 r1 = cmul(rw1, f), r2 = cmul(rw2, f), r3 = cmul(rw3, f);
#pragma unroll
    for (int k2 = 0; k2 < 8; ++k2) {
        ptfft::dft4<DIR, PK>(a[0][k2], a[1][k2], a[2][k2], a[3][k2]);
        s[k2 * 32] = cmul(a[0][k2], f);
        s[(8 + k2) * 32] = cmul(a[1][k2], r1);
        s[(16 + k2) * 32] = cmul(a[2][k2], r2);
        s[(24 + k2) * 32] = cmul(a[3][k2], r3);
    }
}

// R3's read of row (u, v1): w[qb], qb = 0..31.
__device__ __forceinline__ void f128_r3_read(float2 (&w)[32], const float2 *ex, int u, int v1)
{
    const int k1 = u & 15;
    const unsigned o = ((unsigned)(k1 * 32 + v1 * 8 + (u >> 4)) << 8) + ((k1 & 7) << 4);
#pragma unroll
    for (int s = 0; s < 16; ++s) {
        const float4 q = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(ex) + (o ^ (s << 4)));
        w[2 * s] = make_float2(q.x, q.y);
        w[2 * s + 1] = make_float2(q.z, q.w);
    }
}

// barrier of group g's 128 threads (named barriers 1..4; 0 is __syncthreads)
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory"); }

// Starts the copy of the first probe rows into shared memory (both 16-byte
// aligned), all of it in flight at once and under the caller's first loads;
// f128_probe_wait ends it, then the caller synchronises.  Forward of 148, 592 and
// 2220 full frames, with the copy through registers, a few loads at a time: 13.7,
// 39.1 and 132 us; so: 13.0, 38.1 and 131 (waiting inside the loop, after the
// first frame's second half of loads: 14.0, 39.8 and 134).
__device__ __forceinline__ void f128_probe_rows(float2 *tab, const float2 *__restrict__ prbT, int rows, int P)
{
    const int n = rows * P;
    for (int e = threadIdx.x; e < n / 2; e += 512)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(tab + 2 * e)),
                     "l"(prbT + 2 * e)
                     : "memory");
    if ((n & 1) && threadIdx.x == 0) tab[n - 1] = __ldg(&prbT[n - 1]);
}
__device__ __forceinline__ void f128_probe_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Loads of data read once (frames, counts, patches) that do not allocate in
// L1, so that what is reread keeps its L1 lines (at 256^3 / 384 angles: plain
// adjoint 4.39 -> 4.24 ms, Poisson residual 5.85 -> 5.52 ms, Gaussian 6.32 ->
// 5.99 ms, before the probe rows moved to shared memory).
__device__ __forceinline__ float2 ld_once(const float2 *p)
{
    float2 r;
    asm("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];\n" : "=f"(r.x), "=f"(r.y) : "l"(p));
    return r;
}
__device__ __forceinline__ float ld_once(const float *p)
{
    float r;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];\n" : "=f"(r) : "l"(p));
    return r;
}

// Asks for `bytes` (a multiple of 16) at the 16-byte aligned p to be brought
// into L2; no data moves to the SM.
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}

// Forward, grid-stride over frames, one resident block per SM.  The first half
// of the next frame's patch values (line c = 0) is requested before R3's
// arithmetic and stores, so its latency runs under them.
template <bool FULL, bool SUB = false>
__global__ void __launch_bounds__(512, 1)
    k_ptycho_fwd128(const float2 *__restrict__ psi, float2 *__restrict__ g, const int *__restrict__ corner,
                    const float2 *__restrict__ phase, const float2 *__restrict__ prbT, int nz, int n, int nscan,
                    int nframes, int P, float scale, const float4 *__restrict__ tw4,
                    const float2 *__restrict__ w128, const int *__restrict__ sid = nullptr)
{
    extern __shared__ float4 sm4[];
    float2 *ex = reinterpret_cast<float2 *>(sm4);
    float2 *tab = ex + 128 * 128;
    const int grp = threadIdx.x >> 7, q0 = threadIdx.x >> 7 << 5 | (threadIdx.x & 31), rt0 = (threadIdx.x >> 5) & 3;
    const int PS = FULL ? 128 : P;  // a constant row stride: the probe rows are immediate offsets
    const int off0 = FULL ? 0 : (128 - P) / 2;
    const int rows = SUB ? 0 : FULL ? P128_FTAB / 1024 : min(P, P128_FTAB / (P * (int)sizeof(float2)));
    f128_probe_rows(tab, prbT, rows, P);
    // patch value (row rt + 8 m, column q) of frame f; 0 outside the window
    auto patch = [&](const float2 *src, int px, int py, int off) {
        return FULL || (px >= 0 && px < P && py >= 0 && py < P) ? ld_once(&src[(ptrdiff_t)py * n]) : czero();
    };
    auto source = [&](int fid, int sx, int sy, int px) {
        return psi + ((size_t)(fid / nscan) * nz + sy) * n + sx + px;
    };
    // the thread's probe values below the table, rows rt0 + 4 c + 8 m, m >= KT,
    // the same for every frame: kept in registers (3.42 -> 3.34 ms)
    constexpr int KT = P128_FTAB / 8192;
    float2 pk[2][16 - KT];
    if (FULL && !SUB) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int m = KT; m < 16; ++m) pk[c][m - KT] = __ldg(&prbT[(rt0 + 4 * c + 8 * m) * 128 + q0]);
    }
    int fid = blockIdx.x;
    int stx = corner[2 * fid], sty = corner[2 * fid + 1];
    float2 pre[16];
    {
        const bool ok = stx >= 0 && sty >= 0;
        const int px = q0 - off0;
        const float2 *src = source(fid, max(stx, 0), max(sty, 0), px);
#pragma unroll
        for (int m = 0; m < 16; ++m) pre[m] = ok ? patch(src, px, rt0 + 8 * m - off0, off0) : czero();
    }
    f128_probe_wait();
    __syncthreads();
    while (true) {
        const int nxt = fid + gridDim.x;
        const bool more = nxt < nframes;
        const int nsx = more ? corner[2 * nxt] : -1, nsy = more ? corner[2 * nxt + 1] : -1;
        const bool act = stx >= 0 && sty >= 0, nact = nsx >= 0 && nsy >= 0;
        const int q = fresh(q0), rt = fresh(rt0), off = FULL ? 0 : fresh(off0), px = q - off;
        float2 *out = g + (size_t)fid * 128 * 128;
        float2 w[32];
        if (act) {
            const float2 *src = source(fid, stx, sty, px);
            const float2 *pr = (SUB ? prbT + (size_t)sid[fid] * P * P : prbT) + px;  // sub-pixel: the frame's shifted probe
            const float2 *ps = tab + px;
            auto probe = [&](int c, int m, int py) {
                if (FULL && !SUB && m >= KT) return pk[c][m - KT];
                if (!FULL && !(px >= 0 && px < P && py >= 0 && py < P)) return czero();
                if (!SUB && (FULL || py < rows)) return ps[py * PS];
                return __ldg(&pr[py * PS]);
            };
            float2 v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = patch(src, px, rt + 4 + 8 * m - off, off);
#pragma unroll
            for (int m = 0; m < 16; ++m) pre[m] = cmul(probe(0, m, rt + 8 * m - off), pre[m]);
            f128_r1<-1, false>(pre, ex, q, rt, tw4);
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = cmul(probe(1, m, rt + 4 + 8 * m - off), v[m]);
            f128_r1<-1, false>(v, ex, q, rt + 4, tw4);
            __syncthreads();
            f128_r2<-1, false>(ex, fresh(threadIdx.x), scale * phase[fid], w128);
            __syncthreads();
            f128_r3_read(w, ex, fresh(threadIdx.x & 127), grp);
            group_sync(grp);  // the group's rows are read: its next R1 may write
        }
        {
            const float2 *src = source(more ? nxt : fid, max(nsx, 0), max(nsy, 0), px);
#pragma unroll
            for (int m = 0; m < 16; ++m) pre[m] = nact ? patch(src, px, rt + 8 * m - off, off) : czero();
        }
        float2 *o = out + grp * 128 + fresh(threadIdx.x & 127);   // frame[kx = grp + 4 v2][ky = u]
        if (act) {
            ptfft::Dft<32, -1, false>::run(w);
#pragma unroll
            for (int v2 = 0; v2 < 32; ++v2) __stcs(&o[4 * v2 * 128], w[v2]);
        } else {   // skipped scan: the reference leaves a zero frame
#pragma unroll
            for (int v2 = 0; v2 < 32; ++v2) __stcs(&o[4 * v2 * 128], czero());
        }
        if (!more) break;
        fid = nxt;
        stx = nsx;
        sty = nsy;
    }
}

// The adjoints (see k_ptycho_fwd128).  Object adjoint: grid (parts, ntheta),
// block (part, angles[y]) owns slab dst[angle][part] and walks that angle's scans
// part, part + parts, ...  PROBE (the adjoint with respect to the probe): grid
// (blocks, 1), block b walks frames b, b + gridDim.x, ... < nframes and
// accumulates conj(psi patch) x frame into its P x P partial dst[b].  RESID
// forms the Poisson / Gaussian residual of each frame value on load.  R3's
// thread adds pixel column x = u, rows y = v1 + 4 v2, so the 32 lanes of a
// warp touch 256 consecutive bytes of one slab (or partial) row whatever the
// frame's column parity.  w128[m] = exp(-2 pi i m / 128).
template <bool FULL, int RESID, bool SUB = false, bool PROBE = false>
__global__ void __launch_bounds__(512, 1)
    k_ptycho_adj128(const float2 *__restrict__ g, float2 *dst, const int *__restrict__ corner,
                    const float2 *__restrict__ phase, const float2 *prbT, int nz, int n, int nscan,
                    int P, float scale, const float4 *__restrict__ tw4, const float2 *__restrict__ w128,
                    const float *__restrict__ data, float dscale, const int *__restrict__ angles,
                    const int *__restrict__ sid = nullptr, const float2 *psi = nullptr, int nframes = 0)
{
    extern __shared__ float4 sm4[];
    float2 *ex = reinterpret_cast<float2 *>(sm4);
    float2 *tab = ex + 128 * 128;
    const int part = blockIdx.x, parts = gridDim.x, th0 = PROBE ? 0 : angles[blockIdx.y];
    float2 *slab = PROBE ? dst + (size_t)part * P * P : dst + ((size_t)th0 * parts + part) * nz * n;
    const int grp = threadIdx.x >> 7, q0 = threadIdx.x >> 7 << 5 | (threadIdx.x & 31), rt0 = (threadIdx.x >> 5) & 3;
    const int off0 = FULL ? 0 : (128 - P) / 2;
    constexpr bool TAB = !SUB && !PROBE;
    const int rows = !TAB ? 0 : FULL ? P128_ATAB / 1024 : min(P, P128_ATAB / (P * (int)sizeof(float2)));
    if constexpr (TAB) f128_probe_rows(tab, prbT, rows, P);
    for (int e = threadIdx.x; e < (PROBE ? P * P : nz * n); e += 512) slab[e] = czero();
    if constexpr (TAB) f128_probe_wait();
    __syncthreads();
    const int count = PROBE ? nframes : nscan;
    for (int s = part; s < count; s += parts) {
        const int fid = PROBE ? s : th0 * nscan + s;
        const int th = PROBE ? fid / nscan : th0;
        // the block's next frame (and its counts) into L2 one frame ahead, in
        // 16 KB pieces: its loads then wait on L2 rather than on HBM
        // (plain adjoint 4.64 -> 4.42 ms with the earlier kernel).  Not with the
        // residual: 45 angles of 100 to 400 scans, Poisson 0.90 -> 1.00 ms.
        constexpr bool PREFETCH = RESID == 0 || PROBE;
        const bool aligned = (((uintptr_t)g | (RESID != 0 ? (uintptr_t)data : 0)) & 15) == 0;
        if (PREFETCH && aligned && threadIdx.x < 8 && s + parts < count) {
            const size_t nf = (size_t)fid + parts;
            prefetch_l2(g + (nf * 128 * 128 + threadIdx.x * 2048), 16384);
            if (RESID != 0 && threadIdx.x < 4) prefetch_l2(data + (nf * 128 * 128 + threadIdx.x * 4096), 16384);
        }
        const int stx = corner[2 * fid], sty = corner[2 * fid + 1];
        if (stx < 0 || sty < 0) continue;
        {
            const int q = fresh(q0), rt = fresh(rt0);
            const float2 *in = g + (size_t)fid * 128 * 128 + rt * 128 + q;
            const float *din = RESID ? data + (size_t)fid * 128 * 128 + rt * 128 + q : nullptr;
            // all 32 frame values (and counts) are loaded before the first
            // residual: its branches would otherwise hold each later load back
            float2 v[2][16];
            float d[2][16];
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    v[c][m] = ld_once(&in[(4 * c + 8 * m) * 128]);
                    if constexpr (RESID != 0) d[c][m] = ld_once(&din[(4 * c + 8 * m) * 128]);
                }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if constexpr (RESID != 0) resid_line<RESID>(v[c], d[c], dscale, din + 4 * c * 128, 8 * 128);
                f128_r1<+1, true>(v[c], ex, q, rt + 4 * c, tw4);
            }
        }
        __syncthreads();
        const float2 ph = phase[fid];
        f128_r2<+1, true>(ex, fresh(threadIdx.x), make_float2(scale * ph.x, -scale * ph.y), w128);
        __syncthreads();
        float2 w[32];
        const int u = fresh(threadIdx.x & 127), off = FULL ? 0 : fresh(off0);
        f128_r3_read(w, ex, u, grp);
        group_sync(grp);  // the group's rows are read: its next R1 may write
        ptfft::Dft<32, +1, true>::run(w);
        // object: slab += conj(probe) x value; probe: partial += conj(psi) x value
        const int px = u - off;
        if (!FULL && (px < 0 || px >= P)) continue;
        const float2 *mul = (PROBE ? psi + ((size_t)th * nz + sty) * n + stx
                                   : (SUB ? prbT + (size_t)sid[fid] * P * P : prbT)) + px;
        const int ms = PROBE ? n : (FULL ? 128 : P);  // row stride of mul (a constant for the probe table)
        float2 *col = PROBE ? slab + px : slab + (size_t)sty * n + stx + px;
        const size_t cs = PROBE ? P : n;              // row stride of col
        // RB rows at a time: their multiplier loads are issued before the first add
        constexpr int RB = 8;
#pragma unroll
        for (int h = 0; h < 32; h += RB) {
            float2 pv[RB];
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                const int py = grp + 4 * (h + j) - off;
                const bool ok = FULL || (py >= 0 && py < P);
                if (TAB && (FULL ? h + j < P128_ATAB / 4096 : py < rows))
                    pv[j] = ok ? tab[py * ms + px] : czero();
                else
                    pv[j] = ok ? mul[(size_t)py * ms] : czero();
            }
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                const int py = grp + 4 * (h + j) - off;
                if (FULL || (py >= 0 && py < P)) add_l2(&col[py * cs], cmulc(pv[j], w[h + j]));
            }
        }
    }
}

// out[angle] = sum over parts of dst[angle][part], fixed order
__global__ void k_ptycho_reduce(const float2 *__restrict__ part, float2 *__restrict__ out, size_t slab,
                                int parts, size_t total)
{
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t th = e / slab, i = e % slab;
        const float2 *p = part + th * parts * slab + i;
        float2 acc = p[0];
        for (int k = 1; k < parts; ++k) acc = acc + p[k * slab];
        out[e] = acc;
    }
}

// prbT[iy][ix] = c * prb[ix][iy] (the reference's mul/mula index prb[iy + ix*Nprb])
__global__ void k_probe_t(const float2 *__restrict__ prb, float2 *__restrict__ prbT, int P, float c)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P * P) return;
    const int iy = i / P, ix = i % P;
    prbT[i] = c * prb[ix * P + iy];
}

// ---- adjoint with respect to the probe (no counterpart in the reference) ----
// The forward is linear in the probe too: with c prbT[py][px] = c prb[px P + py]
// multiplying psi[th][sty + py][stx + px] (ptychofft.cu:58-76, kernels.cuh:
// 243-265), the adjoint maps frames g to
//   gprb[px P + py] = c sum_frames conj(psi[th][sty + py][stx + px]) G[py][px],
// G = scale x inverse DFT of conj(phase) g (the same transform as the object
// adjoint).  Block b walks frames b, b + gridDim.x, ... and accumulates into
// its own P x P partial part[b] (prbT layout); every (py, px) of the window
// belongs to one thread, so no atomics; k_probe_reduce sums the partials in a
// fixed order.  The kernels are the object adjoints in their PROBE mode.

// gprb[px P + py] = c sum_b part[b][py P + px].  A block takes 32 elements; its
// warps sum the partials b = warp, warp + warps, ..., then their sums are added
// in warp order, in FP64: the order then shows in the last bit at most.
// T double2: the sum as it is, for a caller that adds several.
template <typename T>
__global__ void __launch_bounds__(1024)
    k_probe_reduce(const float2 *__restrict__ part, T *__restrict__ gprb, int nblk, int P, float c)
{
    __shared__ double2 sums[32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    double2 s = make_double2(0.0, 0.0);
    if (i < P * P)
#pragma unroll 4
        for (int b = warp; b < nblk; b += warps) {
            const float2 v = part[(size_t)b * P * P + i];
            s.x += v.x;
            s.y += v.y;
        }
    sums[warp][lane] = s;
    __syncthreads();
    if (warp || i >= P * P) return;
    for (int k = 1; k < warps; ++k) {
        s.x += sums[k][lane].x;
        s.y += sums[k][lane].y;
    }
    const int py = i / P, px = i % P;
    T r;
    r.x = c * s.x;
    r.y = c * s.y;
    gprb[px * P + py] = r;
}

}  // namespace

// ---- sub-pixel scan model (no counterpart in the reference) -----------------
// The reference rounds each scan position s to the object grid and multiplies
// the frame by a constant phase (kernels.cuh:306-336), which leaves the
// intensities unchanged.  The sub-pixel model keeps the object on its grid and
// evaluates the probe at the scan's offset instead: the exit wave is
// P(r - d) psi(c + r), c = round(s), d = s - c in [-1/2, 1/2]^2, r the patch
// pixel, with P(r - d) the band-limited (trigonometric) interpolation of the
// probe's samples, separable in x and y:
//   P_d[y][x] = sum_{i,j} D(y - dy - i) P[i][j] D(x - dx - j),
//   D(t) = sin(pi t) / (P tan(pi t / P))  (even P;  P sin(pi t / P) for odd P),
// the Dirichlet kernel whose spectrum is 1 below Nyquist and cos(pi d) at it.
// Offsets are quantised to multiples of 1/quant pixel; one shifted table is
// kept per distinct offset pair and each frame indexes its own.

// tmp[s][i][x] = sum_j prbT[i][j] MxT[kx_s][j][x]   (one thread per (s, i, x))
__global__ void k_probe_shift_x(const float2 *__restrict__ prbT, const float *__restrict__ mxT,
                                const int2 *__restrict__ pairs, float2 *__restrict__ tmp, int P, int npairs)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)npairs * P * P) return;
    const int x = (int)(e % P), i = (int)((e / P) % P), sidx = (int)(e / ((size_t)P * P));
    const float *m = mxT + (size_t)pairs[sidx].x * P * P;
    double re = 0, im = 0;
    for (int j = 0; j < P; ++j) {
        const float2 v = prbT[(size_t)i * P + j];
        const double w = m[(size_t)j * P + x];
        re += w * v.x;
        im += w * v.y;
    }
    tmp[e] = make_float2((float)re, (float)im);
}

// out[s][y][x] = sum_i My[ky_s][y][i] tmp[s][i][x]
__global__ void k_probe_shift_y(const float2 *__restrict__ tmp, const float *__restrict__ my,
                                const int2 *__restrict__ pairs, float2 *__restrict__ out, int P, int npairs)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)npairs * P * P) return;
    const int x = (int)(e % P), y = (int)((e / P) % P), sidx = (int)(e / ((size_t)P * P));
    const float *m = my + (size_t)pairs[sidx].y * P * P + (size_t)y * P;
    const float2 *src = tmp + (size_t)sidx * P * P + x;
    double re = 0, im = 0;
    for (int i = 0; i < P; ++i) {
        const float2 v = src[(size_t)i * P];
        const double w = m[i];
        re += w * v.x;
        im += w * v.y;
    }
    out[e] = make_float2((float)re, (float)im);
}

__global__ void k_fill_one(float2 *__restrict__ a, size_t n)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) a[e] = make_float2(1.f, 0.f);
}

// The object adjoint's split: blocks (and slabs) per angle, and whether they run
// k_ptycho_adj_few (det 16 to 64).
struct Split {
    int parts = 1;
    bool few = false;
};

struct pt_ptycho {
    int ntheta = 0, nz = 0, n = 0, nscan = 0, det = 0, P = 0;
    Split split[3];   // the object adjoint's, by residual (none, Poisson, Gaussian)
    int device = -1, nsm = 148;
    bool ready = false;
    float c = 0.f;
    char *tables = nullptr;   // one allocation: tw, tw128, prb, prbT, prbT2, angles, phase, corner, frac
    float2 *tw = nullptr, *prb = nullptr, *prbT = nullptr, *phase = nullptr, *partial = nullptr;
    float4 *tw128 = nullptr;  // det = 128: the twiddles in twiddle16's pair layout
    int *corner = nullptr;
    // the object adjoint's order of angles: most scans first (as uploaded: order)
    int *angles = nullptr;
    std::vector<int> order;
    bool ordered = false;       // that order is not 0, 1, 2, ...
    // the scans of each angle that are not skipped, most first (none before setobj: as if all), and their sum
    std::vector<int> counts;
    double scans_all = 0;
    int parts_set = 0;          // the parts that the caller or the environment set; 0: chosen, -1: autotuned
    int few_set = -1;           // k_ptycho_adj_few: 1 always, 0 never, -1 chosen
    // slabs per angle that `partial` holds, and whether a launch has used them:
    // a captured graph may hold their address, so setobj leaves them where they are
    size_t slabs = 0;
    bool slabs_used = false;
    // probe retrieval: a second transposed probe table (forward with a given
    // probe) and one P x P partial per block of the probe adjoint
    float2 *prbT2 = nullptr, *prb_part = nullptr;
    int prb_blocks = 0;
    // sub-pixel scan model (quant > 0): frac = per-frame offsets s - round(s);
    // prbS = one shifted probe table per distinct quantised offset pair (prbT
    // layout), sid = each frame's table, ones = the unit phase the model uses
    float *frac = nullptr;
    float2 *prbS = nullptr, *ones = nullptr;
    int *sid = nullptr;
    int quant = 0, nshift = 0;
    // the tables the kernels take
    const float2 *probe_tab() const { return quant ? prbS : prbT; }
    const float2 *phase_tab() const { return quant ? ones : phase; }
    const int *shift_ids() const { return quant ? sid : nullptr; }
};

namespace {

#define PT_PTYCHO_DETS(X) X(8) X(16) X(32) X(64) X(128)

template <int DET>
int ptycho_attrs()
{
#define PT_ATTR(K, S) PT_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(S)))
    if constexpr (DET < 16) {
        const int s = DET * (DET + 1) * sizeof(float2);
        PT_ATTR(k_ptycho_fwd_small<DET>, s);
        PT_ATTR((k_ptycho_adj_small<DET, 0>), s);
        PT_ATTR((k_ptycho_adj_small<DET, 1>), s);
        PT_ATTR((k_ptycho_adj_small<DET, 2>), s);
    } else if constexpr (DET == 128) {
        PT_ATTR((k_ptycho_fwd128<true>), P128_FSMEM);
        PT_ATTR((k_ptycho_fwd128<false>), P128_FSMEM);
        PT_ATTR((k_ptycho_fwd128<true, true>), P128_FSMEM);
        PT_ATTR((k_ptycho_fwd128<false, true>), P128_FSMEM);
#define PT_ATTR_ADJ(RESID)                                                  \
    PT_ATTR((k_ptycho_adj128<true, RESID>), P128_ASMEM);                     \
    PT_ATTR((k_ptycho_adj128<false, RESID>), P128_ASMEM);                    \
    PT_ATTR((k_ptycho_adj128<true, RESID, true>), P128_ASMEM);               \
    PT_ATTR((k_ptycho_adj128<false, RESID, true>), P128_ASMEM);              \
    PT_ATTR((k_ptycho_adj128<true, RESID, false, true>), P128_ASMEM);        \
    PT_ATTR((k_ptycho_adj128<false, RESID, false, true>), P128_ASMEM);
        PT_ATTR_ADJ(0)
        PT_ATTR_ADJ(1)
        PT_ATTR_ADJ(2)
#undef PT_ATTR_ADJ
    } else if constexpr (DET == 64) {   // two frames per trip
        constexpr size_t s = FR<DET>::smem(2);
        static_assert(FR<32>::smem(2) <= 48 * 1024, "no attribute needed");
        PT_ATTR((k_ptycho_fwd<DET, false, false, 2>), s);
        PT_ATTR((k_ptycho_fwd<DET, false, true, 2>), s);
        PT_ATTR((k_ptycho_adj<DET, false, 1>), s);
        PT_ATTR((k_ptycho_adj<DET, false, 2>), s);
        PT_ATTR((k_ptycho_adj<DET, false, 1, true>), s);
        PT_ATTR((k_ptycho_adj<DET, false, 2, true>), s);
    }
#undef PT_ATTR
    return PT_OK;
}

// go(FULL, SUB) for the handle: whether the probe fills the detector, and
// whether each frame has its own shifted probe
template <typename Go>
void by_kind(const pt_ptycho *h, Go go)
{
    const bool full = h->P == h->det;
    if (h->quant)
        full ? go(std::true_type{}, std::true_type{}) : go(std::false_type{}, std::true_type{});
    else
        full ? go(std::true_type{}, std::false_type{}) : go(std::false_type{}, std::false_type{});
}

template <int DET, int RESID, bool SUB>
void launch_few(dim3 grid, pt_ptycho *h, const float2 *in, float2 *dst, float scale, const float *data, float dscale,
                cudaStream_t st)
{
    // the order of the angles matters only where blocks wait for others to end
    const bool queued = (size_t)grid.x * grid.y > (size_t)h->nsm * PF<DET>::BPS;
    if constexpr (DET <= 64)
        k_ptycho_adj_few<DET, RESID, SUB><<<grid, PF<DET>::NT, PF<DET>::SMEM, st>>>(
            in, dst, h->corner, h->phase_tab(), h->probe_tab(), h->nz, h->n, h->nscan, h->P, scale, h->tw, data, dscale,
            h->ordered && queued ? h->angles : nullptr, h->shift_ids());
}

template <int DET, int RESID>
int ptycho_adj_launch(pt_ptycho *h, float2 *out, const float2 *in, float scale, const float *data, float dscale,
                      cudaStream_t st)
{
    if constexpr (DET < 16) {
        const size_t s = DET * (DET + 1) * sizeof(float2);
        k_ptycho_adj_small<DET, RESID><<<h->ntheta, ptycho_block<DET>(), s, st>>>(
            in, out, h->corner, h->phase, h->prb, h->nz, h->n, h->nscan, h->P, h->c, scale, h->tw, data, dscale);
        PT_LAUNCHED("k_ptycho_adj_small");
        return PT_OK;
    } else {
        const Split split = h->split[RESID];
        float2 *dst = split.parts > 1 ? h->partial : out;
        h->slabs_used |= split.parts > 1;
        const dim3 grid(split.parts, h->ntheta);
        // SUB: the sub-pixel model's per-frame probe tables (a separate
        // instantiation, so the reference model's kernels are unchanged)
        auto go = [&](auto full, auto sub) {
            constexpr bool FU = decltype(full)::value, S = decltype(sub)::value;
            if constexpr (DET == 128)
                k_ptycho_adj128<FU, RESID, S><<<grid, 512, P128_ASMEM, st>>>(
                    in, dst, h->corner, h->phase_tab(), h->probe_tab(), h->nz, h->n, h->nscan, h->P, scale, h->tw128,
                    h->tw, data, dscale, h->angles, h->shift_ids());
            else if (DET <= 64 && split.few)
                launch_few<DET, RESID, S>(grid, h, in, dst, scale, data, dscale, st);
            else
                k_ptycho_adj<DET, FU, RESID, S>
                    <<<grid, FR<DET>::BLOCK, FR<DET>::smem(FR<DET>::nf_adj(FU, RESID != 0)), st>>>(
                    in, dst, h->corner, h->phase_tab(), h->probe_tab(), h->nz, h->n, h->nscan, h->P, scale, h->tw,
                    data, dscale, h->angles, h->shift_ids());
        };
        by_kind(h, go);
        PT_LAUNCHED("k_ptycho_adj");
        if (split.parts > 1) {
            const size_t slab = (size_t)h->nz * h->n, total = slab * h->ntheta;
            const unsigned blocks = (unsigned)std::min<size_t>((total + 255) / 256, 148 * 16);
            k_ptycho_reduce<<<blocks, 256, 0, st>>>(h->partial, out, slab, split.parts, total);
            PT_LAUNCHED("k_ptycho_reduce");
        }
        return PT_OK;
    }
}

template <int DET>
int ptycho_run(pt_ptycho *h, bool adj, float2 *out, const float2 *in, float scale, cudaStream_t st, int resid_mode,
               const float *data, float dscale)
{
    if (adj) {
        if (resid_mode == 1) return ptycho_adj_launch<DET, 1>(h, out, in, scale, data, dscale, st);
        if (resid_mode == 2) return ptycho_adj_launch<DET, 2>(h, out, in, scale, data, dscale, st);
        return ptycho_adj_launch<DET, 0>(h, out, in, scale, data, dscale, st);
    }
    const int nframes = h->ntheta * h->nscan;
    if constexpr (DET < 16) {
        const size_t s = DET * (DET + 1) * sizeof(float2);
        k_ptycho_fwd_small<DET><<<dim3(h->nscan, h->ntheta), ptycho_block<DET>(), s, st>>>(
            in, out, h->corner, h->phase, h->prb, h->nz, h->n, h->nscan, h->P, h->c, scale, h->tw);
    } else {
        // the resident blocks walk the frames (grid-stride); few frames, a block each
        auto go = [&](auto full, auto sub) {
            constexpr bool FU = decltype(full)::value, S = decltype(sub)::value;
            if constexpr (DET == 128) {
                k_ptycho_fwd128<FU, S><<<std::min(nframes, h->nsm), 512, S ? P128_EX : P128_FSMEM, st>>>(
                    in, out, h->corner, h->phase_tab(), h->probe_tab(), h->nz, h->n, h->nscan, nframes, h->P, scale,
                    h->tw128, h->tw, h->shift_ids());
            } else {
                using F = FR<DET>;
                if (nframes <= few_frames(DET, FU) * h->nsm) {
                    k_ptycho_fwd_few<DET, S><<<nframes, PF<DET>::NT, PF<DET>::SMEM, st>>>(
                        in, out, h->corner, h->phase_tab(), h->probe_tab(), h->nz, h->n, h->nscan, h->P, scale, h->tw,
                        h->shift_ids());
                    return;
                }
                auto trips = [&](auto frames) {
                    constexpr int NF = decltype(frames)::value;
                    const int per = F::FPB * NF, grid = std::min((nframes + per - 1) / per, h->nsm * F::BPS);
                    k_ptycho_fwd<DET, FU, S, NF><<<grid, F::BLOCK, F::smem(NF), st>>>(
                        in, out, h->corner, h->phase_tab(), h->probe_tab(), h->nz, h->n, h->nscan, nframes, h->P,
                        scale, h->tw, h->shift_ids());
                };
                if constexpr (DET == 64 && !FU) {
                    if (2 * h->P <= DET && nframes >= 2 * h->nsm * F::BPS)
                        trips(std::integral_constant<int, 2>{});
                    else
                        trips(std::integral_constant<int, 1>{});
                } else {
                    trips(std::integral_constant<int, 1>{});
                }
            }
        };
        by_kind(h, go);
    }
    PT_LAUNCHED("k_ptycho_fwd");
    return PT_OK;
}

bool det_supported(int d)
{
#define PT_CASE(D) \
    if (d == D) return true;
    PT_PTYCHO_DETS(PT_CASE)
#undef PT_CASE
    return false;
}

int ptycho_set_attrs(int d)
{
#define PT_CASE(D) \
    if (d == D) return ptycho_attrs<D>();
    PT_PTYCHO_DETS(PT_CASE)
#undef PT_CASE
    return PT_ERR_UNSUPPORTED;
}

int ptycho_dispatch(pt_ptycho *h, bool adj, float2 *out, const float2 *in, float scale, cudaStream_t st,
                    int resid_mode = 0, const float *data = nullptr, float dscale = 1.f)
{
#define PT_CASE(D) \
    if (h->det == D) return ptycho_run<D>(h, adj, out, in, scale, st, resid_mode, data, dscale);
    PT_PTYCHO_DETS(PT_CASE)
#undef PT_CASE
    pt::set_error("ptychofft: detector size %d not compiled", h->det);
    return PT_ERR_UNSUPPORTED;
}

template <int DET, int RESID>
int probe_adj_launch(pt_ptycho *h, void *gprb, bool fp64, const float2 *in, const float2 *psi, float scale,
                     const float *data, float dscale, cudaStream_t st)
{
    if constexpr (DET < 16) {
        pt::set_error("ptychofft.adj_probe: not compiled for detector %d (16 to 128)", DET);
        return PT_ERR_UNSUPPORTED;
    } else {
        const int nframes = h->ntheta * h->nscan;
        auto go = [&](auto full) {
            constexpr bool FU = decltype(full)::value;
            if constexpr (DET == 128)
                k_ptycho_adj128<FU, RESID, false, true><<<h->prb_blocks, 512, P128_ASMEM, st>>>(
                    in, h->prb_part, h->corner, h->phase, h->prbT, h->nz, h->n, h->nscan, h->P, scale, h->tw128,
                    h->tw, data, dscale, nullptr, nullptr, psi, nframes);
            else
                k_ptycho_adj<DET, FU, RESID, false, true>
                    <<<h->prb_blocks / FR<DET>::FPB, FR<DET>::BLOCK, FR<DET>::smem(1), st>>>(
                        in, h->prb_part, h->corner, h->phase, h->prbT, h->nz, h->n, h->nscan, h->P, scale, h->tw, data,
                        dscale, nullptr, nullptr, psi, nframes);
        };
        if (h->P == DET)
            go(std::true_type{});
        else
            go(std::false_type{});
        PT_LAUNCHED("k_ptycho_adj_probe");
        // many partials: 32 warps (with eight, the few blocks of a small probe waited on
        // 4736 / 8 partials a warp: 16 x 16 frames of 100 x 150 scans 156 us, now 35; 64 x
        // 64 frames of 40 x 60, 296 partials, 45 and 39); det 128 has at most 148
        const unsigned blocks = (unsigned)((h->P * h->P + 31) / 32), threads = h->prb_blocks > 256 ? 1024 : 256;
        if (fp64)
            k_probe_reduce<<<blocks, threads, 0, st>>>(h->prb_part, (double2 *)gprb, h->prb_blocks, h->P, h->c);
        else
            k_probe_reduce<<<blocks, threads, 0, st>>>(h->prb_part, (float2 *)gprb, h->prb_blocks, h->P, h->c);
        PT_LAUNCHED("k_probe_reduce");
        return PT_OK;
    }
}

int probe_adj_dispatch(pt_ptycho *h, void *gprb, bool fp64, const float2 *in, const float2 *psi, float scale,
                       int resid_mode, const float *data, float dscale, cudaStream_t st)
{
#define PT_CASE(D)                                                                                               \
    if (h->det == D) {                                                                                           \
        if (resid_mode == 1) return probe_adj_launch<D, 1>(h, gprb, fp64, in, psi, scale, data, dscale, st);      \
        if (resid_mode == 2) return probe_adj_launch<D, 2>(h, gprb, fp64, in, psi, scale, data, dscale, st);      \
        return probe_adj_launch<D, 0>(h, gprb, fp64, in, psi, scale, data, dscale, st);                          \
    }
    PT_PTYCHO_DETS(PT_CASE)
#undef PT_CASE
    pt::set_error("ptychofft: detector size %d not compiled", h->det);
    return PT_ERR_UNSUPPORTED;
}

// Times of the object adjoint's steps in microseconds, but for det 128 in frames
// of an SM (only one block runs there).
struct SplitCost {
    // one trip of a block alone on its SM, and an SM's time for a frame, by
    // residual and whether the probe is as wide as the detector
    double lone[3][2], frame[3][2];
    double clear, fixed;          // a thread's clear of a slab cell; a call
    double clear_sm = 9.5e-5;     // an SM's clear of a slab cell
    double sum = 4.3, sum_part = 0.15, sum_cell = 2e-6;   // the sum of the parts: a launch, per part, per slab cell
};
// Resident blocks per SM (of the probe adjoint, of the object adjoint), frames
// that a block works on at a time, and its threads.
struct Residency {
    int probe_blocks, frames, blocks, threads;
    SplitCost cost;
};
Residency residency(int det)
{
    switch (det) {
    case 16: return {FR<16>::BPSP, FR<16>::FPB, FR<16>::BPS, FR<16>::BLOCK,
                     {{{3.57, 1.97}, {3.86, 2.64}, {5.80, 4.27}}, {{0.107, 0.100}, {0.165, 0.176}, {0.312, 0.335}}, 2.0e-3, 0.7}};
    case 32: return {FR<32>::BPSP, FR<32>::FPB, FR<32>::BPS, FR<32>::BLOCK,
                     {{{2.25, 1.69}, {2.87, 2.52}, {4.51, 2.64}}, {{0.384, 0.393}, {0.642, 0.594}, {1.05, 0.616}}, 6.5e-4, 0}};
    case 64: return {FR<64>::BPSP, FR<64>::FPB, FR<64>::BPS, FR<64>::BLOCK,
                     {{{2.75, 2.27}, {3.81, 2.98}, {5.12, 3.58}}, {{1.06, 1.47}, {1.56, 1.80}, {1.81, 2.09}}, 2.0e-3, 0}};
    // a block clears a slab's worth of frames at 0.375 of one, and once more for the sum
    default: return {1, 1, 1, 512, {{{1, 1}, {1, 1}, {1, 1}}, {}, 0, 0, 0.375 / (128 * 128), 0, 0, 0}};
    }
}
// k_ptycho_adj_few
Residency residency_few(int det)
{
    if (det == 16)
        return {0, 1, PF<16>::BPS, PF<16>::NT,
                {{{0.85, 0.94}, {1.52, 1.60}, {1.57, 1.65}}, {{0.200, 0.233}, {0.226, 0.251}, {0.229, 0.252}}, 2.0e-3, 0.7}};
    if (det == 64)
        return {0, 1, PF<64>::BPS, PF<64>::NT,
                {{{2.85, 3.23}, {4.82, 4.95}, {4.97, 5.13}}, {{1.37, 1.72}, {2.06, 2.09}, {2.17, 2.20}}, 2.0e-3, 0}};
    return {0, 1, PF<32>::BPS, PF<32>::NT,
            {{{1.37, 1.50}, {2.86, 3.06}, {3.00, 3.19}}, {{0.733, 0.983}, {0.968, 1.27}, {0.965, 1.27}}, 1.4e-3, 0.1}};
}

// The adjoint's split of an angle's scans over blocks for one residual: the
// number of parts with the earliest end, and up to 64 pixels the kernel.
// With R the blocks on an SM:
//   a block    clears its slab, at the SM's store rate, and takes trips of
//              sqrt(lone^2 + (R frames)^2) each: a few blocks wait on latency,
//              many on the SM;
//   the sum    of more than one part reads every slab once, after a launch.
// Angles with different numbers of scans: only det 128, whose SMs take few blocks
// each, has the blocks placed one by one (45 angles: 0.3 ms of setobj; the bound
// below it costs up to 12 %: 38 x 236 scans 442 -> 494 us).  The others have the
// bound, which chooses as well as the placement on 119 calls, in constant time
// (384 angles of 400 scans, 16 x 16: setobj 4.3 -> 1.0 ms).
// No more parts than an angle has scans, or than `most`; more than 16 only while
// all blocks run at once and their slabs take at most 1 GiB.  only > 0: that
// number of parts, and the kernel for it.
// The costs are least-squares fits, of the logarithm, to 335 calls of 16- and
// 32-pixel and 70 of 64-pixel detectors, with each residual, timed at every
// split (4 to 384 angles, 9 to 400 scans, objects of 19 to 256; rms 9 to 11 %).
// Against the wave rule with k_ptycho_adj_few alone, 520 further calls with each
// residual: mean time 0.80 / 0.73 / 0.77 of it (none, Poisson, Gaussian) at 16
// pixels, 0.71 / 0.58 / 0.64 at 32 and 0.71 / 0.58 / 0.64 at 64; 61 of 1560 take
// 3 % more or worse, at most one launch step of 2 us or 1.17 times.  One choice
// for all residuals and probes had 207, up to 1.6 times.
// Det 128, one block per SM: 45 angles with 100 to 400 scans:
// 6 parts and the angles with most scans first instead of 3 parts in angle
// order, Gaussian gradient 1.48 -> 1.09 ms, Poisson 1.43 -> 0.90 ms.
Split choose_split(const pt_ptycho &h, int resid, size_t most, int only = 0)
{
    const double cells = (double)h.nz * h.n;
    const bool full = h.P == h.det;
    const int most_scans = h.counts.empty() ? h.nscan : h.counts.front(), least = h.counts.empty() ? h.nscan : h.counts.back();
    const int scans = std::max(most_scans, 1);
    const bool few_can = h.det >= 16 && h.det <= 64;
    Split best_split;
    double best = 1e300;
    auto time = [&](int p, const Residency &res) {
        const size_t slots = (size_t)h.nsm * res.blocks, blocks = (size_t)h.ntheta * p;
        const SplitCost &c = res.cost;
        const double lone = c.lone[resid][full], frame = res.frames * c.frame[resid][full], q = (double)p * res.frames;
        const int passes = h.det == 128 && p > 1 ? 2 : 1;
        auto clear = [&](size_t R) { return std::max(c.clear * cells / res.threads, passes * R * c.clear_sm * cells); };
        auto block = [&](int n, size_t R) { return clear(R) + std::ceil(n / q) * std::hypot(lone, R * frame); };
        auto sharing = [&](size_t n) { return (std::min(n, slots) + h.nsm - 1) / h.nsm; };   // blocks on an SM
        const size_t R = sharing(blocks);
        // trips of one block of each angle: every quotient rounded up, by a half on average
        const double trips = (h.scans_all + h.ntheta * (q - 1) / 2) / q;
        double end = c.fixed + (p > 1 ? c.sum + c.sum_part * p + c.sum_cell * cells * h.ntheta * (p + 1) : 0);
        if (least == most_scans) {   // whole waves of equal blocks and what is left
            const size_t rest = blocks % slots;
            end += blocks / slots * block(most_scans, res.blocks) + (rest ? block(most_scans, sharing(rest)) : 0);
        } else if (blocks <= slots) {   // all at once: the longest block, while the others end
            end += clear(R) + std::hypot(std::ceil(most_scans / q) * lone, frame * trips * R / h.ntheta);
        } else if (h.det < 128) {   // most scans first: the SMs end together, but for a part of the shortest block
            const double all = p * (h.ntheta * clear(R) + trips * std::hypot(lone, R * frame));
            end += std::max(block(most_scans, R), all / slots + 0.5 * block(least, R));
        } else {   // one block after the other goes to the SM that is free first
            std::priority_queue<double, std::vector<double>, std::greater<double>> ends;
            double last = 0;
            for (int n : h.counts)
                for (int k = 0; k < p; ++k) {
                    double start = 0;
                    if (ends.size() == slots) {
                        start = ends.top();
                        ends.pop();
                    }
                    ends.push(start + block(n, R));
                    last = std::max(last, start + block(n, R));
                }
            end += last;
        }
        return end;
    };
    for (const bool few : {false, true}) {
        if ((few && !few_can) || (few_can && h.few_set == !few)) continue;
        const Residency res = few ? residency_few(h.det) : residency(h.det);
        for (int p : {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 20, 24, 32, 48, 64}) {
            const size_t blocks = (size_t)h.ntheta * p;
            if (only)
                p = only;
            else if (p > scans || (size_t)p > most)
                break;
            else if (p > 16 && (h.det == 128 || blocks > (size_t)h.nsm * res.blocks || blocks * cells > (1u << 27)))
                break;
            const double end = time(p, res);
            if (end < best - 1e-9) {
                best = end;
                best_split.parts = p, best_split.few = few;
            }
            if (only) break;
        }
    }
    if (few_can && h.few_set != 0) {
        // a modelled gain of less than 7 % is within the model's error: then the
        // split by whole waves of a block per SM, 3 % for each further part, in
        // k_ptycho_adj_few
        double least = 1e300;
        int p0 = only ? only : 1;
        for (int p = 1; !only && p <= std::min(scans, 16) && (size_t)p <= most; ++p) {
            const double waves = std::ceil((double)h.ntheta * p / h.nsm);
            const double cost = waves * std::ceil((double)scans / p) * (1.0 + 0.03 * (p - 1));
            if (cost < least - 1e-9) {
                least = cost;
                p0 = p;
            }
        }
        const double end = time(p0, residency_few(h.det));
        if (best > 0.93 * end) best_split.parts = p0, best_split.few = true;
    }
    return best_split;
}

void release_slabs(pt_ptycho *h)
{
    if (h->partial) cudaFree(h->partial);
    h->partial = nullptr;
    h->slabs = 0;
    h->slabs_used = false;
}

// Uses these splits from now on, with slabs for them; one part if they do not fit.
bool use_splits(pt_ptycho *h, std::array<Split, 3> split)
{
    const int parts = std::max({split[0].parts, split[1].parts, split[2].parts});
    std::copy(split.begin(), split.end(), h->split);
    if (parts > 1 && (size_t)parts > h->slabs) {
        release_slabs(h);
        if (cudaMalloc((void **)&h->partial, (size_t)parts * h->ntheta * h->nz * h->n * sizeof(float2)) !=
            cudaSuccess) {
            cudaGetLastError();
            h->partial = nullptr;
            for (Split &s : h->split) s.parts = 1;
            return false;
        }
        h->slabs = parts;
    }
    return true;
}
// The same number of parts with every residual, in the kernel that suits it.
bool set_parts(pt_ptycho *h, int parts)
{
    std::array<Split, 3> split;
    for (int r = 0; r < 3; ++r) split[r] = choose_split(*h, r, SIZE_MAX, parts);
    return use_splits(h, split);
}

void ptycho_free(pt_ptycho *h)
{
    void *bufs[] = {h->tables, h->partial, h->prb_part, h->prbS, h->ones, h->sid};
    for (void *p : bufs)
        if (p) cudaFree(p);
}

// D(t) of the sub-pixel model in double: 1 at multiples of P, exactly 0 at
// the other integers (a zero offset leaves the probe unchanged)
double dirichlet(double t, int P)
{
    if (t == std::floor(t)) return std::fmod(t, (double)P) == 0.0 ? 1.0 : 0.0;
    const double a = M_PI * t / P;
    return (P % 2 == 0) ? std::sin(M_PI * t) / (P * std::tan(a)) : std::sin(M_PI * t) / (P * std::sin(a));
}

void subpixel_free(pt_ptycho *h)
{
    void *bufs[] = {h->prbS, h->ones, h->sid};
    for (void *p : bufs)
        if (p) cudaFree(p);
    h->prbS = h->ones = nullptr;
    h->sid = nullptr;
    h->quant = h->nshift = 0;
}

// Builds the shifted probe tables from the handle's offsets (setobj) and
// probe.  Set-up: allocates, blocks the host.
int subpixel_build(pt_ptycho *h, int quant, cudaStream_t st)
{
    const int nf = h->ntheta * h->nscan, P = h->P;
    std::vector<float> frac(2 * (size_t)nf);
    std::vector<int> corner(2 * (size_t)nf);
    PT_CUDA(cudaMemcpyAsync(frac.data(), h->frac, frac.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaMemcpyAsync(corner.data(), h->corner, corner.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaStreamSynchronize(st));
    std::map<int, int> ux, uy;                   // quantised offset -> axis table index
    std::map<std::pair<int, int>, int> up;       // (x index, y index) -> shifted table
    std::vector<int> sid(nf, 0);
    std::vector<int2> pairs;
    auto axis = [](std::map<int, int> &m, int q) {
        auto it = m.find(q);
        if (it != m.end()) return it->second;
        const int k = (int)m.size();
        m.emplace(q, k);
        return k;
    };
    for (int f = 0; f < nf; ++f) {
        if (corner[2 * f] < 0 || corner[2 * f + 1] < 0) continue;   // skipped scan
        const int qx = (int)std::lrint((double)frac[2 * f] * quant), qy = (int)std::lrint((double)frac[2 * f + 1] * quant);
        const int kx = axis(ux, qx), ky = axis(uy, qy);
        auto it = up.find({kx, ky});
        if (it == up.end()) {
            it = up.emplace(std::make_pair(kx, ky), (int)pairs.size()).first;
            pairs.push_back(make_int2(kx, ky));
        }
        sid[f] = it->second;
    }
    if (pairs.empty()) pairs.push_back(make_int2(axis(ux, 0), axis(uy, 0)));   // every scan skipped
    const size_t tab = (size_t)P * P * sizeof(float2);
    if (pairs.size() * tab > ((size_t)1 << 31)) {
        pt::set_error("ptychofft.set_subpixel: %zu distinct offsets need %zu MB of probe tables (limit 2048); "
                      "use a coarser quantisation",
                      pairs.size(), pairs.size() * tab >> 20);
        return PT_ERR_ARG;
    }
    // axis matrices: MxT[k][j][x] = D(x - dx_k - j), My[k][y][i] = D(y - dy_k - i)
    std::vector<float> mx(ux.size() * P * P), my(uy.size() * P * P);
    for (const auto &kv : ux)
        for (int j = 0; j < P; ++j)
            for (int x = 0; x < P; ++x)
                mx[((size_t)kv.second * P + j) * P + x] = (float)dirichlet(x - (double)kv.first / quant - j, P);
    for (const auto &kv : uy)
        for (int y = 0; y < P; ++y)
            for (int i = 0; i < P; ++i)
                my[((size_t)kv.second * P + y) * P + i] = (float)dirichlet(y - (double)kv.first / quant - i, P);
    float *dmx = nullptr, *dmy = nullptr;
    int2 *dpairs = nullptr;
    float2 *tmp = nullptr, *prbS = nullptr, *ones = nullptr;
    int *dsid = nullptr;
    const size_t np = pairs.size();
    bool ok = cudaMalloc((void **)&dmx, mx.size() * sizeof(float)) == cudaSuccess &&
              cudaMalloc((void **)&dmy, my.size() * sizeof(float)) == cudaSuccess &&
              cudaMalloc((void **)&dpairs, np * sizeof(int2)) == cudaSuccess &&
              cudaMalloc((void **)&tmp, np * tab) == cudaSuccess && cudaMalloc((void **)&prbS, np * tab) == cudaSuccess &&
              cudaMalloc((void **)&ones, (size_t)nf * sizeof(float2)) == cudaSuccess &&
              cudaMalloc((void **)&dsid, (size_t)nf * sizeof(int)) == cudaSuccess;
    int rc = PT_OK;
    if (!ok) {
        cudaGetLastError();
        pt::set_error("ptychofft.set_subpixel: device allocation failed");
        rc = PT_ERR_ALLOC;
    }
    if (rc == PT_OK &&
        (cudaMemcpyAsync(dmx, mx.data(), mx.size() * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess ||
         cudaMemcpyAsync(dmy, my.data(), my.size() * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess ||
         cudaMemcpyAsync(dpairs, pairs.data(), np * sizeof(int2), cudaMemcpyHostToDevice, st) != cudaSuccess ||
         cudaMemcpyAsync(dsid, sid.data(), (size_t)nf * sizeof(int), cudaMemcpyHostToDevice, st) != cudaSuccess)) {
        pt::set_error("ptychofft.set_subpixel: table upload failed");
        rc = PT_ERR_CUDA;
    }
    if (rc == PT_OK) {
        const size_t tot = np * P * P;
        const unsigned blocks = (unsigned)((tot + 255) / 256);
        k_probe_shift_x<<<blocks, 256, 0, st>>>(h->prbT, dmx, dpairs, tmp, P, (int)np);
        k_probe_shift_y<<<blocks, 256, 0, st>>>(tmp, dmy, dpairs, prbS, P, (int)np);
        k_fill_one<<<(unsigned)((nf + 255) / 256), 256, 0, st>>>(ones, (size_t)nf);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
            pt::set_error("ptychofft.set_subpixel: table kernels failed");
            rc = PT_ERR_CUDA;
        }
    }
    for (void *q : {(void *)dmx, (void *)dmy, (void *)dpairs, (void *)tmp})
        if (q) cudaFree(q);
    if (rc != PT_OK) {
        for (void *q : {(void *)prbS, (void *)ones, (void *)dsid})
            if (q) cudaFree(q);
        return rc;
    }
    subpixel_free(h);
    h->prbS = prbS;
    h->ones = ones;
    h->sid = dsid;
    h->quant = quant;
    h->nshift = (int)np;
    return PT_OK;
}

}  // namespace

extern "C" int pt_ptycho_create(size_t ntheta, size_t nz, size_t n, size_t ntheta0, size_t nscan, size_t detx,
                                size_t dety, size_t nprb, pt_ptycho **out)
{
    (void)ntheta0;
    pt::clear_error();
    PT_CHECK_ARG(out != nullptr, "ptychofft: null output handle");
    *out = nullptr;
    PT_CHECK_ARG(ntheta >= 1 && nz >= 1 && n >= 1 && nscan >= 1 && nprb >= 1,
                 "ptychofft: sizes must be positive (Ntheta=%zu Nz=%zu N=%zu Nscan=%zu Nprb=%zu)", ntheta, nz, n,
                 nscan, nprb);
    PT_CHECK_ARG(ntheta * nscan < (1u << 31) && ntheta * nz * n < ((size_t)1 << 40), "ptychofft: sizes too large");
    if (detx != dety || !det_supported((int)detx)) {
        pt::set_error("ptychofft: detector %zux%zu not compiled (square 8,16,32,64,128)", detx, dety);
        return PT_ERR_UNSUPPORTED;
    }
    PT_CHECK_ARG(nprb <= detx, "ptychofft: probe %zu larger than detector %zu", nprb, detx);
    PT_CHECK_ARG(nprb <= n && nprb <= nz, "ptychofft: probe %zu larger than the object %zux%zu", nprb, nz, n);
    pt_ptycho *h = new pt_ptycho();
    h->ntheta = (int)ntheta;
    h->nz = (int)nz;
    h->n = (int)n;
    h->nscan = (int)nscan;
    h->det = (int)detx;
    h->P = (int)nprb;
    h->c = 1 / sqrtf(detx * dety);  // kernels.cuh:260
    h->scans_all = (double)h->ntheta * h->nscan;
    if (cudaGetDevice(&h->device) != cudaSuccess) {
        delete h;
        pt::set_error("ptychofft: no CUDA device");
        return PT_ERR_CUDA;
    }
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
    h->nsm = nsm;
    // PT_PTYCHO_ADJ_PARTS=<k> overrides the choice of the parts, PT_PTYCHO_ADJ_FEW=0
    // or 1 that of the kernel (tuning and tests)
    const char *env_parts = getenv("PT_PTYCHO_ADJ_PARTS"), *env_few = getenv("PT_PTYCHO_ADJ_FEW");
    if (env_few) h->few_set = atoi(env_few) != 0;
    if (env_parts && atoi(env_parts) >= 1)
        h->parts_set = std::min<int>(atoi(env_parts), (int)nscan);
    else if (detx >= 16)
        h->split[0].parts = choose_split(*h, 0, SIZE_MAX).parts;   // setobj chooses, for the scans that are there
    // the small tables are cuts of one allocation, each on a 256-byte boundary
    const size_t P2 = nprb * nprb, nf = ntheta * nscan;
    size_t used = 0;
    auto cuts = [&](auto &&cut) {
        used = 0;
        cut(h->tw, detx);
        cut(h->tw128, (size_t)64);
        cut(h->prb, P2);
        cut(h->prbT, P2);
        cut(h->prbT2, P2);
        cut(h->angles, ntheta);
        cut(h->phase, nf);
        cut(h->corner, 2 * nf);
        cut(h->frac, 2 * nf);
    };
    auto place = [&](auto *&p, size_t count) {
        if (h->tables) p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(h->tables + used);
        used += (count * sizeof(*p) + 255) / 256 * 256;
    };
    cuts(place);
    bool ok = cudaMalloc((void **)&h->tables, used) == cudaSuccess && (h->parts_set == 0 || set_parts(h, h->parts_set));
    if (ok) cuts(place);
    // probe adjoint: one partial per frame in flight
    const Residency res = residency((int)detx);
    const size_t inflight = (size_t)nsm * res.probe_blocks;
    h->prb_blocks = (int)(std::min(inflight, (ntheta * nscan + res.frames - 1) / res.frames) * res.frames);
    ok = ok && cudaMalloc((void **)&h->prb_part, (size_t)h->prb_blocks * nprb * nprb * sizeof(float2)) == cudaSuccess;
    if (!ok) {
        ptycho_free(h);
        delete h;
        pt::set_error("ptychofft: device allocation failed");
        return PT_ERR_ALLOC;
    }
    std::vector<float2> tw(detx);
    pt_make_twiddles(tw.data(), (int)detx);
    int rc = ptycho_set_attrs((int)detx);
    if (rc == PT_OK && cudaMemcpy(h->tw, tw.data(), detx * sizeof(float2), cudaMemcpyHostToDevice) != cudaSuccess) {
        pt::set_error("ptychofft: twiddle upload failed");
        rc = PT_ERR_CUDA;
    }
    if (rc == PT_OK && detx == 128) {
        // entry q * 8 + t = (w(2q t), w((2q+1) t)), t k1 <= 105 < 128
        std::vector<float4> tw4(64);
        for (int q = 0; q < 8; ++q)
            for (int t = 0; t < 8; ++t) {
                const float2 a = tw[2 * q * t], b = tw[(2 * q + 1) * t];
                tw4[q * 8 + t] = make_float4(a.x, a.y, b.x, b.y);
            }
        if (cudaMemcpy(h->tw128, tw4.data(), 64 * sizeof(float4), cudaMemcpyHostToDevice) != cudaSuccess) {
            pt::set_error("ptychofft: twiddle upload failed");
            rc = PT_ERR_CUDA;
        }
    }
    if (rc != PT_OK) {
        ptycho_free(h);
        delete h;
        return rc;
    }
    *out = h;
    return PT_OK;
}

extern "C" int pt_ptycho_destroy(pt_ptycho *h)
{
    pt::clear_error();
    if (!h) return PT_OK;
    ptycho_free(h);
    delete h;
    return PT_OK;
}

extern "C" int pt_ptycho_setobj(pt_ptycho *h, const float *scan, const void *prb, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "ptychofft.setobj: null handle");
    PT_CHECK_ARG(scan != nullptr && prb != nullptr, "ptychofft.setobj: null scan or probe");
    int dev = -1;
    PT_CUDA(cudaGetDevice(&dev));
    PT_CHECK_ARG(dev == h->device, "ptychofft handle belongs to device %d, current device is %d", h->device, dev);
    cudaStream_t st = (cudaStream_t)stream;
    const int nf = h->ntheta * h->nscan;
    h->ready = false;
    PT_CUDA(cudaMemcpyAsync(h->prb, prb, (size_t)h->P * h->P * sizeof(float2), cudaMemcpyDefault, st));
    k_ptycho_tables<<<(nf + 255) / 256, 256, 0, st>>>(scan, h->corner, h->phase, h->frac, nf);
    PT_LAUNCHED("k_ptycho_tables");
    k_probe_t<<<(h->P * h->P + 255) / 256, 256, 0, st>>>(h->prb, h->prbT, h->P, h->c);
    PT_LAUNCHED("k_probe_t");
    std::vector<int> corner(2 * (size_t)nf);
    PT_CUDA(cudaMemcpyAsync(corner.data(), h->corner, corner.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    PT_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < nf; ++i) {
        const int x = corner[2 * i], y = corner[2 * i + 1];
        if (x < 0 || y < 0) continue;  // sentinel: scan skipped
        if (x + h->P > h->n || y + h->P > h->nz) {
            pt::set_error("ptychofft.setobj: scan %d of angle %d at (%d,%d) puts the %dx%d probe outside the "
                          "%dx%d object",
                          i % h->nscan, i / h->nscan, x, y, h->P, h->P, h->nz, h->n);
            return PT_ERR_ARG;
        }
    }
    // angles by decreasing number of scans, and the split for those numbers
    std::vector<int> counts(h->ntheta, 0), order(h->ntheta);
    for (int i = 0; i < nf; ++i) counts[i / h->nscan] += corner[2 * i] >= 0 && corner[2 * i + 1] >= 0;
    for (int t = 0; t < h->ntheta; ++t) order[t] = t;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return counts[a] > counts[b]; });
    h->ordered = !std::is_sorted(order.begin(), order.end());
    if (order != h->order) {
        PT_CUDA(cudaMemcpyAsync(h->angles, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice, st));
        PT_CUDA(cudaStreamSynchronize(st));
        h->order = order;
    }
    std::sort(counts.begin(), counts.end(), std::greater<int>());
    h->counts = counts;
    h->scans_all = std::accumulate(counts.begin(), counts.end(), 0.0);
    if (h->parts_set > 0) {   // the kernels for it may change with the scans
        for (int r = 0; r < 3; ++r) h->split[r].few = choose_split(*h, r, SIZE_MAX, h->split[r].parts).few;
    } else if (h->parts_set == 0 && h->det >= 16) {
        auto choose = [&](size_t most) {
            std::array<Split, 3> split;
            for (int r = 0; r < 3; ++r) split[r] = r > 0 && h->det == 128 ? split[0] : choose_split(*h, r, most);
            return use_splits(h, split);
        };
        // never more parts than slabs that a launch has used hold: those stay
        // (one part if new ones cannot be allocated)
        if (!choose(h->slabs_used ? h->slabs : SIZE_MAX)) choose(1);
    }
    h->ready = true;
    if (h->quant) {   // new offsets or probe: new shifted tables (on failure the model is switched off)
        const int rc = subpixel_build(h, h->quant, st);
        if (rc != PT_OK) subpixel_free(h);
        return rc;
    }
    return PT_OK;
}

namespace {
int ptycho_call(pt_ptycho *h, bool adj, void *out, const void *in, float scale, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "ptychofft: null handle");
    PT_CHECK_ARG(out != nullptr && in != nullptr, "ptychofft.%s: null array pointer", adj ? "adj" : "fwd");
    if (!h->ready) {
        pt::set_error("ptychofft.%s: setobj(scan, prb) has not been called", adj ? "adj" : "fwd");
        return PT_ERR_STATE;
    }
    int dev = -1;
    PT_CUDA(cudaGetDevice(&dev));
    PT_CHECK_ARG(dev == h->device, "ptychofft handle belongs to device %d, current device is %d", h->device, dev);
    return ptycho_dispatch(h, adj, (float2 *)out, (const float2 *)in, scale, (cudaStream_t)stream);
}
}  // namespace

extern "C" int pt_ptycho_fwd(pt_ptycho *h, void *g, const void *f, void *stream)
{
    return ptycho_call(h, false, g, f, 1.0f, stream);
}
// ---- autotuner: the adjoint's angle split ---------------------------------
// Times the plain object adjoint (the CG's dominant kernel) at the present split
// and at others, in both kernels where there are two, and keeps the fastest; the
// present one unless another is faster.  The residual adjoints keep their splits.
// Setup-time: allocates the partial slabs of each candidate, blocks the host.
extern "C" int pt_ptycho_autotune(pt_ptycho *h, void *f, const void *g, int trials, int *parts_out, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h && f && g && trials >= 1, "ptychofft.autotune: bad arguments");
    if (h->det < 16) {   // the small-detector kernel has no angle split
        if (parts_out) *parts_out = h->split[0].parts;
        return PT_OK;
    }
    cudaStream_t st = (cudaStream_t)stream;
    cudaEvent_t e0, e1;
    PT_CUDA(cudaEventCreate(&e0));
    PT_CUDA(cudaEventCreate(&e1));
    const Split resid[2] = {h->split[1], h->split[2]};
    auto use = [&](const Split &plain) { return use_splits(h, {plain, resid[0], resid[1]}); };
    std::vector<Split> cands = {h->split[0]};
    const bool few_can = h->det <= 64;
    for (const bool few : {false, true}) {
        if ((few && !few_can) || (few_can && h->few_set == !few)) continue;
        for (int p : {1, 2, 3, 4, 6, 8, 12, 16, h->split[0].parts})
            if (p <= h->nscan) cands.push_back({p, few});
    }
    Split best = cands.front();
    float best_t = 1e30f;
    int rc = PT_OK;
    for (const Split &c : cands) {
        if (!use(c)) continue;   // this split does not fit: skip it
        std::vector<float> ts;
        for (int k = 0; k <= trials && rc == PT_OK; ++k) {   // the first run warms up
            cudaEventRecord(e0, st);
            rc = pt_ptycho_adj(h, f, g, stream);
            cudaEventRecord(e1, st);
            if (rc == PT_OK && cudaEventSynchronize(e1) == cudaSuccess && k > 0) {
                float ms = 0;
                cudaEventElapsedTime(&ms, e0, e1);
                ts.push_back(ms);
            }
        }
        if (rc != PT_OK || ts.empty()) break;
        std::sort(ts.begin(), ts.end());
        const float med = ts[ts.size() / 2];
        if (med < best_t) {
            best_t = med;
            best = c;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    release_slabs(h);   // the largest candidate's
    h->parts_set = -1;
    if (!use(best)) {
        pt::set_error("ptychofft.autotune: the chosen split's slabs could not be allocated");
        return PT_ERR_ALLOC;
    }
    if (parts_out) *parts_out = h->split[0].parts;
    return rc;
}

extern "C" int pt_ptycho_set_parts(pt_ptycho *h, int parts)
{
    pt::clear_error();
    PT_CHECK_ARG(h && parts >= 1 && (size_t)parts <= h->nscan, "ptychofft.set_parts: parts must be in [1, nscan]");
    if (h->det < 16) {
        PT_CHECK_ARG(parts == h->split[0].parts, "ptychofft.set_parts: the small-detector kernel has no angle split");
        return PT_OK;
    }
    release_slabs(h);
    h->parts_set = parts;
    if (!set_parts(h, parts)) {
        pt::set_error("ptychofft.set_parts: the split's slabs could not be allocated");
        return PT_ERR_ALLOC;
    }
    return PT_OK;
}

extern "C" int pt_ptycho_get_parts(const pt_ptycho *h, int *parts)
{
    pt::clear_error();
    PT_CHECK_ARG(h && parts, "ptychofft: null pointer");
    *parts = h->split[0].parts;
    return PT_OK;
}

extern "C" int pt_ptycho_adj(pt_ptycho *h, void *f, const void *g, void *stream)
{
    return ptycho_call(h, true, f, g, 1.0f, stream);
}
extern "C" int pt_ptycho_fwd_scaled(pt_ptycho *h, void *g, const void *f, float scale, void *stream)
{
    return ptycho_call(h, false, g, f, scale, stream);
}
extern "C" int pt_ptycho_adj_scaled(pt_ptycho *h, void *f, const void *g, float scale, void *stream)
{
    return ptycho_call(h, true, f, g, scale, stream);
}

extern "C" int pt_ptycho_adj_resid(pt_ptycho *h, void *f, const void *fpsi, const float *data, float dscale,
                                   int model, float scale, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "ptychofft: null handle");
    PT_CHECK_ARG(f != nullptr && fpsi != nullptr && data != nullptr, "ptychofft.adj_resid: null array pointer");
    PT_CHECK_ARG(model == 0 || model == 1, "ptychofft.adj_resid: model 0 (poisson) or 1 (gaussian)");
    if (!h->ready) {
        pt::set_error("ptychofft.adj_resid: setobj(scan, prb) has not been called");
        return PT_ERR_STATE;
    }
    int dev = -1;
    PT_CUDA(cudaGetDevice(&dev));
    PT_CHECK_ARG(dev == h->device, "ptychofft handle belongs to device %d, current device is %d", h->device, dev);
    return ptycho_dispatch(h, true, (float2 *)f, (const float2 *)fpsi, scale, (cudaStream_t)stream, model + 1, data,
                           dscale);
}

// ---- probe retrieval (no counterpart in the reference) -----------------------
namespace {
int probe_checks(pt_ptycho *h, const char *what)
{
    PT_CHECK_ARG(h != nullptr, "ptychofft.%s: null handle", what);
    if (!h->ready) {
        pt::set_error("ptychofft.%s: setobj(scan, prb) has not been called", what);
        return PT_ERR_STATE;
    }
    int dev = -1;
    PT_CUDA(cudaGetDevice(&dev));
    PT_CHECK_ARG(dev == h->device, "ptychofft handle belongs to device %d, current device is %d", h->device, dev);
    if (h->quant) {
        pt::set_error("ptychofft.%s: probe retrieval is not available with the sub-pixel scan model", what);
        return PT_ERR_STATE;
    }
    return PT_OK;
}
}  // namespace

extern "C" int pt_ptycho_adj_probe(pt_ptycho *h, void *gprb, const void *g, const void *psi, float scale,
                                   void *stream)
{
    pt::clear_error();
    const int rc = probe_checks(h, "adj_probe");
    if (rc != PT_OK) return rc;
    PT_CHECK_ARG(gprb && g && psi, "ptychofft.adj_probe: null array pointer");
    return probe_adj_dispatch(h, gprb, false, (const float2 *)g, (const float2 *)psi, scale, 0, nullptr, 1.f,
                              (cudaStream_t)stream);
}

namespace {
int adj_probe_resid(pt_ptycho *h, void *gprb, bool fp64, const void *psi, const void *fpsi, const float *data,
                    float dscale, int model, float scale, void *stream)
{
    pt::clear_error();
    const int rc = probe_checks(h, "adj_probe_resid");
    if (rc != PT_OK) return rc;
    PT_CHECK_ARG(gprb && psi && fpsi && data, "ptychofft.adj_probe_resid: null array pointer");
    PT_CHECK_ARG(model == 0 || model == 1, "ptychofft.adj_probe_resid: model 0 (poisson) or 1 (gaussian)");
    return probe_adj_dispatch(h, gprb, fp64, (const float2 *)fpsi, (const float2 *)psi, scale, model + 1, data, dscale,
                              (cudaStream_t)stream);
}
}  // namespace

extern "C" int pt_ptycho_adj_probe_resid(pt_ptycho *h, void *gprb, const void *psi, const void *fpsi,
                                         const float *data, float dscale, int model, float scale, void *stream)
{
    return adj_probe_resid(h, gprb, false, psi, fpsi, data, dscale, model, scale, stream);
}

extern "C" int pt_ptycho_adj_probe_resid64(pt_ptycho *h, void *gprb, const void *psi, const void *fpsi,
                                           const float *data, float dscale, int model, float scale, void *stream)
{
    return adj_probe_resid(h, gprb, true, psi, fpsi, data, dscale, model, scale, stream);
}

extern "C" int pt_ptycho_fwd_probe(pt_ptycho *h, void *g, const void *psi, const void *prb, float scale,
                                   void *stream)
{
    pt::clear_error();
    const int rc = probe_checks(h, "fwd_probe");
    if (rc != PT_OK) return rc;
    PT_CHECK_ARG(g && psi && prb, "ptychofft.fwd_probe: null array pointer");
    cudaStream_t st = (cudaStream_t)stream;
    k_probe_t<<<(h->P * h->P + 255) / 256, 256, 0, st>>>((const float2 *)prb, h->prbT2, h->P, h->c);
    PT_LAUNCHED("k_probe_t");
    // the forward kernels read the handle's table: point it at this probe for one launch
    float2 *own = h->prbT;
    h->prbT = h->prbT2;
    const int rc2 = ptycho_dispatch(h, false, (float2 *)g, (const float2 *)psi, scale, st);
    h->prbT = own;
    return rc2;
}

extern "C" int pt_ptycho_set_subpixel(pt_ptycho *h, int quant, void *stream)
{
    pt::clear_error();
    PT_CHECK_ARG(h != nullptr, "ptychofft.set_subpixel: null handle");
    PT_CHECK_ARG(quant >= 0 && quant <= 65536, "ptychofft.set_subpixel: quant must be in [0, 65536] (0: off)");
    if (quant == 0) {
        subpixel_free(h);
        return PT_OK;
    }
    if (h->det < 16) {
        pt::set_error("ptychofft.set_subpixel: not compiled for detector %d (16 to 128)", h->det);
        return PT_ERR_UNSUPPORTED;
    }
    if (!h->ready) {
        pt::set_error("ptychofft.set_subpixel: setobj(scan, prb) has not been called");
        return PT_ERR_STATE;
    }
    int dev = -1;
    PT_CUDA(cudaGetDevice(&dev));
    PT_CHECK_ARG(dev == h->device, "ptychofft handle belongs to device %d, current device is %d", h->device, dev);
    return subpixel_build(h, quant, (cudaStream_t)stream);
}

extern "C" int pt_ptycho_get_subpixel(const pt_ptycho *h, int *quant, int *ntables)
{
    pt::clear_error();
    PT_CHECK_ARG(h && quant && ntables, "ptychofft.get_subpixel: null pointer");
    *quant = h->quant;
    *ntables = h->nshift;
    return PT_OK;
}
