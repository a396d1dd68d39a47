// Block-cooperative complex64 FFTs held in shared memory.
//
// Stockham autosort formulation (Govindaraju et al., "High performance
// discrete Fourier transforms on graphics processors", SC'08): for a pass of
// radix R on a sequence of length L whose already-transformed sub-length is
// NS, butterfly j (0 <= j < L/R) reads x[j + r L/R], multiplies input r by
// W_{NS R}^{r (j mod NS)}, runs an R-point DFT and writes
// y[(j / NS) NS R + (j mod NS) + r NS].  After the last pass the output is in
// natural order.  Lengths are L = 2^a 3^b; passes run radix-3 first, then one
// radix-2 or radix-4 pass if a is not a multiple of 3, then radix-8.
//
// Unnormalised, like cuFFT C2C: DIR = -1 is exp(-2 pi i jk/L) (forward),
// DIR = +1 is exp(+2 pi i jk/L) (inverse).  Twiddles come from a table
// tw[m] = exp(-2 pi i m / L) computed in double on the host.
#pragma once

#include "pt_common.cuh"

namespace ptfft {

__host__ __device__ constexpr int pow3_of(int L) { return (L > 1 && L % 3 == 0) ? 1 + pow3_of(L / 3) : 0; }
__host__ __device__ constexpr int pow2_of(int L) { return (L > 1 && L % 2 == 0) ? 1 + pow2_of(L / 2) : 0; }
__host__ __device__ constexpr int ipow(int b, int e) { return e == 0 ? 1 : b * ipow(b, e - 1); }
__host__ __device__ constexpr bool supported_len(int L)
{
    return L >= 2 && ipow(2, pow2_of(L)) * ipow(3, pow3_of(L)) == L;
}
__host__ __device__ constexpr int num_passes(int L)
{
    return pow3_of(L) + pow2_of(L) / 3 + (pow2_of(L) % 3 ? 1 : 0);
}
__host__ __device__ constexpr int radix_at(int L, int i)
{
    return i < pow3_of(L) ? 3
           : (pow2_of(L) % 3 && i == pow3_of(L)) ? (pow2_of(L) % 3 == 1 ? 2 : 4)
                                                  : 8;
}

// Complex sum and difference.  PK: one packed FP32 instruction (add.rn.f32x2,
// the same two IEEE sums), which halves the issue slots of a butterfly's adds.
// A sum with a value turned by i stays scalar: its halves would have to be
// swapped into a register pair first.
template <bool PK>
__device__ __forceinline__ float2 cadd(float2 a, float2 b)
{
    if constexpr (!PK) return a + b;
    float2 r;
    asm("{\n .reg .b64 p, q;\n mov.b64 p, {%2, %3};\n mov.b64 q, {%4, %5};\n add.rn.f32x2 p, p, q;\n mov.b64 {%0, %1}, p;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
template <bool PK>
__device__ __forceinline__ float2 csub(float2 a, float2 b)
{
    if constexpr (!PK) return a - b;
    float2 r;
    asm("{\n .reg .b64 p, q;\n mov.b64 p, {%2, %3};\n mov.b64 q, {%4, %5};\n sub.rn.f32x2 p, p, q;\n mov.b64 {%0, %1}, p;\n}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// multiply by DIR * i
template <int DIR>
__device__ __forceinline__ float2 mul_i(float2 z)
{
    return DIR < 0 ? make_float2(z.y, -z.x) : make_float2(-z.y, z.x);
}

template <int R, int DIR, bool PK = false>
struct Dft;

template <int DIR, bool PK>
struct Dft<2, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *v)
    {
        float2 a = v[0], b = v[1];
        v[0] = cadd<PK>(a, b);
        v[1] = csub<PK>(a, b);
    }
};

template <int DIR, bool PK>
struct Dft<3, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *v)
    {
        const float s3 = 0.86602540378443864676f;  // sin(pi/3)
        float2 t1 = cadd<PK>(v[1], v[2]);
        float2 t2 = v[0] - 0.5f * t1;
        float2 t3 = s3 * csub<PK>(v[1], v[2]);
        v[0] = cadd<PK>(v[0], t1);
        v[1] = t2 + mul_i<DIR>(t3);
        v[2] = t2 - mul_i<DIR>(t3);
    }
};

template <int DIR, bool PK = false>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d)
{
    float2 t0 = cadd<PK>(a, c), t1 = csub<PK>(a, c), t2 = cadd<PK>(b, d), t3 = mul_i<DIR>(csub<PK>(b, d));
    a = cadd<PK>(t0, t2);
    b = t1 + t3;
    c = csub<PK>(t0, t2);
    d = t1 - t3;
}

template <int DIR, bool PK>
struct Dft<4, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *v) { dft4<DIR, PK>(v[0], v[1], v[2], v[3]); }
};

template <int DIR, bool PK>
struct Dft<8, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *v)
    {
        const float h = 0.70710678118654752440f;  // sqrt(2)/2
        float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
        float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        dft4<DIR, PK>(e0, e1, e2, e3);
        dft4<DIR, PK>(o0, o1, o2, o3);
        // W8^k o_k, W8 = exp(DIR 2 pi i / 8)
        o1 = h * (o1 + mul_i<DIR>(o1));
        o2 = mul_i<DIR>(o2);
        o3 = h * (mul_i<DIR>(o3) - o3);
        v[0] = cadd<PK>(e0, o0);
        v[4] = csub<PK>(e0, o0);
        v[1] = cadd<PK>(e1, o1);
        v[5] = csub<PK>(e1, o1);
        v[2] = cadd<PK>(e2, o2);
        v[6] = csub<PK>(e2, o2);
        v[3] = cadd<PK>(e3, o3);
        v[7] = csub<PK>(e3, o3);
    }
};

// 16-point DFT as 4 x 4 (n = 4 n1 + n2, k = k1 + 4 k2), natural-order output.
template <int DIR, bool PK>
struct Dft<16, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *v)
    {
        const float c1 = 0.92387953251128675613f;  // cos(pi/8)
        const float s1 = 0.38268343236508977173f;  // sin(pi/8)
        const float h = 0.70710678118654752440f;
        const float d = (float)DIR;
        float2 a[4][4];
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
            a[n2][0] = v[n2];
            a[n2][1] = v[4 + n2];
            a[n2][2] = v[8 + n2];
            a[n2][3] = v[12 + n2];
            dft4<DIR, PK>(a[n2][0], a[n2][1], a[n2][2], a[n2][3]);
        }
        // a[n2][k1] *= W16^(n2 k1), W16 = exp(DIR 2 pi i / 16)
        a[1][1] = cmul(a[1][1], make_float2(c1, d * s1));
        a[1][2] = cmul(a[1][2], make_float2(h, d * h));
        a[1][3] = cmul(a[1][3], make_float2(s1, d * c1));
        a[2][1] = cmul(a[2][1], make_float2(h, d * h));
        a[2][2] = mul_i<DIR>(a[2][2]);
        a[2][3] = cmul(a[2][3], make_float2(-h, d * h));
        a[3][1] = cmul(a[3][1], make_float2(s1, d * c1));
        a[3][2] = cmul(a[3][2], make_float2(-h, d * h));
        a[3][3] = cmul(a[3][3], make_float2(-c1, -d * s1));
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            float2 b0 = a[0][k1], b1 = a[1][k1], b2 = a[2][k1], b3 = a[3][k1];
            dft4<DIR, PK>(b0, b1, b2, b3);
            v[k1] = b0;
            v[k1 + 4] = b1;
            v[k1 + 8] = b2;
            v[k1 + 12] = b3;
        }
    }
};

// cos(j pi / 16) for j = 0..8
__host__ __device__ constexpr float cos_pi16(int j)
{
    return j == 0   ? 1.0f
           : j == 1 ? 0.98078528040323044913f
           : j == 2 ? 0.92387953251128675613f
           : j == 3 ? 0.83146961230254523708f
           : j == 4 ? 0.70710678118654752440f
           : j == 5 ? 0.55557023301960222474f
           : j == 6 ? 0.38268343236508977173f
           : j == 7 ? 0.19509032201612826785f
                    : 0.0f;
}

// z * W32^j, W32 = exp(DIR 2 pi i / 32), for a compile-time 0 <= j < 24
template <int DIR>
__device__ __forceinline__ float2 mul_w32(float2 z, int j)
{
    if (j == 0) return z;
    if (j == 8) return mul_i<DIR>(z);
    if (j == 16) return make_float2(-z.x, -z.y);
    // angle j pi / 16 by quadrant: (cos, sin)
    const float c = j < 8 ? cos_pi16(j) : j < 16 ? -cos_pi16(16 - j) : -cos_pi16(j - 16);
    const float s = j < 8 ? cos_pi16(8 - j) : j < 16 ? cos_pi16(j - 8) : -cos_pi16(24 - j);
    return cmul(z, make_float2(c, DIR * s));
}

// 32-point DFT as 4 x 8 (n = 4 n1 + n2, k = k1 + 8 k2), natural-order output.
template <int DIR, bool PK>
struct Dft<32, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *v)
    {
        float2 a[4][8];
#pragma unroll
        for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
            for (int n1 = 0; n1 < 8; ++n1) a[n2][n1] = v[4 * n1 + n2];
            Dft<8, DIR, PK>::run(a[n2]);
        }
#pragma unroll
        for (int n2 = 1; n2 < 4; ++n2)
#pragma unroll
            for (int k1 = 1; k1 < 8; ++k1) a[n2][k1] = mul_w32<DIR>(a[n2][k1], n2 * k1);
#pragma unroll
        for (int k1 = 0; k1 < 8; ++k1) {
            dft4<DIR, PK>(a[0][k1], a[1][k1], a[2][k1], a[3][k1]);
            v[k1] = a[0][k1];
            v[k1 + 8] = a[1][k1];
            v[k1 + 16] = a[2][k1];
            v[k1 + 24] = a[3][k1];
        }
    }
};

// One Stockham pass, in place in shared memory.  `buf` is this FFT's base,
// `es` the element stride, `t` the thread's index among the T threads that
// share this FFT.  All threads of the block must call it (it synchronises).
template <int L, int R, int NS, int DIR, int T>
__device__ __forceinline__ void pass(float2 *buf, int es, int t, const float2 *__restrict__ tw)
{
    constexpr int NB = L / R;
    constexpr int PER = (NB + T - 1) / T;
    float2 v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int j = t + p * T;
        if ((NB % T == 0) || j < NB) {
#pragma unroll
            for (int r = 0; r < R; ++r) v[p][r] = buf[(j + r * NB) * es];
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int j = t + p * T;
        if ((NB % T == 0) || j < NB) {
            const int k = j % NS;
            if (NS > 1) {
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    float2 w = __ldg(&tw[r * k * (L / (NS * R))]);
                    if (DIR > 0) w.y = -w.y;
                    v[p][r] = cmul(v[p][r], w);
                }
            }
            Dft<R, DIR>::run(v[p]);
            const int base = (j / NS) * NS * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r) buf[(base + r * NS) * es] = v[p][r];
        }
    }
    __syncthreads();
}

template <int L, int DIR, int T, int I = 0, int NS = 1>
__device__ __forceinline__ void fft(float2 *buf, int es, int t, const float2 *__restrict__ tw)
{
    static_assert(supported_len(L), "FFT length must be 2^a 3^b");
    if constexpr (I < num_passes(L)) {
        constexpr int R = radix_at(L, I);
        pass<L, R, NS, DIR, T>(buf, es, t, tw);
        fft<L, DIR, T, I + 1, NS * R>(buf, es, t, tw);
    }
}

// ---- register transforms of length 3 x 2^a ----------------------------------
// Good-Thomas: R = 3 M with M a power of two (coprime), n = (M n1 + 3 n2) mod R
// and k = (M M' k1 + 3 T k2) mod R, M' = 1/M mod 3, T = 1/3 mod M, turn the
// R-point DFT into 3-point and M-point DFTs with no twiddles between them.
template <int M, int DIR, bool PK>
struct Dft3M {
    static constexpr int R = 3 * M, MI = M % 3 == 1 ? 1 : 2;
    static constexpr int inv3()
    {
        for (int t = 1; t < M; ++t)
            if (3 * t % M == 1) return t;
        return 0;
    }
    static __device__ __forceinline__ void run(float2 *v)
    {
        float2 t[3][M];
#pragma unroll
        for (int n2 = 0; n2 < M; ++n2) {
            float2 a[3] = {v[3 * n2 % R], v[(M + 3 * n2) % R], v[(2 * M + 3 * n2) % R]};
            Dft<3, DIR, PK>::run(a);
            t[0][n2] = a[0];
            t[1][n2] = a[1];
            t[2][n2] = a[2];
        }
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            Dft<M, DIR, PK>::run(t[k1]);
#pragma unroll
            for (int k2 = 0; k2 < M; ++k2) v[(M * MI * k1 + 3 * inv3() * k2) % R] = t[k1][k2];
        }
    }
};
template <int DIR, bool PK>
struct Dft<6, DIR, PK> : Dft3M<2, DIR, PK> {};
template <int DIR, bool PK>
struct Dft<12, DIR, PK> : Dft3M<4, DIR, PK> {};
template <int DIR, bool PK>
struct Dft<24, DIR, PK> : Dft3M<8, DIR, PK> {};
template <int DIR, bool PK>
struct Dft<48, DIR, PK> : Dft3M<16, DIR, PK> {};
template <int DIR, bool PK>
struct Dft<1, DIR, PK> {
    static __device__ __forceinline__ void run(float2 *) {}
};

// exp(2 pi i n / R), n < R/2, as compile-time constants: the power series of
// sine and cosine at an angle in [0, pi/4], the other octants by symmetry
constexpr double series_cos(double x)
{
    double s = 1.0, t = 1.0;
    for (int i = 1; i < 14; ++i) {
        t *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
        s += t;
    }
    return s;
}
constexpr double series_sin(double x)
{
    double s = x, t = x;
    for (int i = 1; i < 14; ++i) {
        t *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
        s += t;
    }
    return s;
}
template <int R>
struct HalfRoots {
    float c[R / 2], s[R / 2];
    constexpr HalfRoots() : c(), s()
    {
        const double turn = 6.283185307179586476925286766559;
        for (int n = 0; n < R / 2; ++n) {
            // n / R of a turn, folded into an eighth: m / R from an axis
            const bool far = 4 * n > R;                  // second quadrant: R/2 - n mirrored
            const int k = far ? R / 2 - n : n;           // [0, R/4]
            const double x = turn * k / R, y = turn * (R / 4.0 - k) / R;
            const double cs = 8 * k <= R ? series_cos(x) : series_sin(y);
            const double sn = 8 * k <= R ? series_sin(x) : series_cos(y);
            c[n] = (float)(far ? -cs : cs);
            s[n] = (float)sn;
        }
    }
};

// R-point DFT (R even) of a sequence whose second half is zero: in[0 .. R/2)
// -> v[0 .. R).  The even outputs are the R/2-point DFT of the input, the odd
// ones that of the input times W_R^n.
template <int R, int DIR>
__device__ __forceinline__ void dft_half(const float2 (&in)[R / 2], float2 (&v)[R])
{
    constexpr HalfRoots<R> w;
    float2 e[R / 2], o[R / 2];
#pragma unroll
    for (int n = 0; n < R / 2; ++n) {
        e[n] = in[n];
        o[n] = n == 0         ? in[n]
               : 4 * n == R   ? mul_i<DIR>(in[n])
                              : cmul(in[n], make_float2(w.c[n], DIR * w.s[n]));
    }
    Dft<R / 2, DIR, true>::run(e);
    Dft<R / 2, DIR, true>::run(o);
#pragma unroll
    for (int m = 0; m < R / 2; ++m) {
        v[2 * m] = e[m];
        v[2 * m + 1] = o[m];
    }
}

// ---- the USFFT's transforms: two or three rounds in registers -----------------
// L = R1 x R2, i = i1 R2 + i2, k = k1 + R1 k2.  Round 1: a thread holds the R1
// elements i1 of one i2, runs an R1-point DFT and multiplies by W_L^(i2 k1).
// One exchange through shared memory.  Round 2: a thread holds the R2 elements
// i2 of one k1, runs an R2-point DFT and has k = k1 + R1 k2.  So a transform is
// read from and written to global memory by the registers that compute it, and
// passes through shared memory once, where Stockham passes of radix at most 8
// passed through it four times, plus a staging copy on either side.
// R1 and R2 are even and, for the 2N grids (L >= 24), R1 is a multiple of 4:
// the non-zero half of the forward's rows and columns, L/4 .. 3L/4, is then
// R1/2 whole rows i1, and the signs of the centred transforms depend on i2 and
// k1 alone and sit in the twiddle table.
__host__ __device__ constexpr int split_r1(int L)
{
    return L == 12 ? 2 : L == 24 ? 4 : L <= 96 ? 8 : L <= 384 ? 16 : L == 768 ? 24 : 32;
}
__host__ __device__ constexpr int split_r2(int L) { return L / split_r1(L); }

// v[k1] *= w[k1]: tw holds the table in pairs, entry j R2 + i2 = (w(2j), w(2j+1)) of i2
template <int R1, int R2>
__device__ __forceinline__ void twiddle_pairs(float2 (&v)[R1], int i2, const float4 *__restrict__ tw)
{
#pragma unroll
    for (int j = 0; j < R1 / 2; ++j) {
        const float4 w = __ldg(&tw[j * R2 + i2]);
        v[2 * j] = cmul(v[2 * j], make_float2(w.x, w.y));
        v[2 * j + 1] = cmul(v[2 * j + 1], make_float2(w.z, w.w));
    }
}

// The exchange buffer for NQ interleaved sequences: row k1 holds R2 x NQ
// values.  With NQ = 8 a half warp's 8-byte reads in round 2 cover two rows;
// the pad of 8 values puts them on different banks.
template <int L, int NQ>
struct Exchange {
    static constexpr int R1 = split_r1(L), R2 = split_r2(L);
    static constexpr int PITCH = R2 * NQ + (NQ == 8 ? 8 : 0);
    static constexpr int NT = (R1 > R2 ? R1 : R2) * NQ;           // threads
    static constexpr size_t BYTES = (size_t)R1 * PITCH * sizeof(float2);
    static __device__ __forceinline__ void put(float2 *sm, const float2 (&v)[R1], int i2, int q)
    {
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) sm[k1 * PITCH + i2 * NQ + q] = v[k1];
    }
    static __device__ __forceinline__ void get(const float2 *sm, float2 (&w)[R2], int k1, int q)
    {
#pragma unroll
        for (int i2 = 0; i2 < R2; ++i2) w[i2] = sm[k1 * PITCH + i2 * NQ + q];
    }
};

// Three in-place rounds for a transform that is already in shared memory
// (element i of sequence q at sm[i NQ + q]) and whose registers must stay few:
// L = A B C, i = (i1 B + i2) C + i3, k = k1 + A k2 + A B k3.  Each round reads
// and writes the same slots, so only the rounds are separated by barriers.
// tw1[k1 (B C) + i] = W_L^(i k1), i = i2 C + i3, and tw2[k2 C + i3] =
// W_BC^(i3 k2) times the sign of the centred transform, both in direction DIR.
// The C-point outputs of (k1, k2, q) are handed to out(k1 + A k2, q, w).
__host__ __device__ constexpr int split3_c(int L) { return 12; }
__host__ __device__ constexpr int split3_a(int L)
{
    return L <= 48 ? 1 : L == 96 ? 2 : L <= 384 ? 4 : L == 768 ? 8 : 16;
}
__host__ __device__ constexpr int split3_b(int L) { return L / split3_a(L) / split3_c(L); }

template <int L, int DIR, int NT, int NQ, typename Out>
__device__ __forceinline__ void fft3(float2 *sm, const float2 *__restrict__ tw1, const float2 *__restrict__ tw2, Out out)
{
    constexpr int A = split3_a(L), B = split3_b(L), C = split3_c(L), BC = B * C;
    if constexpr (A > 1) {
        for (int it = threadIdx.x; it < BC * NQ; it += NT) {
            const int i = it / NQ;
            float2 v[A];
#pragma unroll
            for (int i1 = 0; i1 < A; ++i1) v[i1] = sm[i1 * BC * NQ + it];
            Dft<A, DIR, true>::run(v);
            sm[it] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < A; ++k1) sm[k1 * BC * NQ + it] = cmul(v[k1], __ldg(&tw1[k1 * BC + i]));
        }
        __syncthreads();
    }
    for (int it = threadIdx.x; it < A * C * NQ; it += NT) {
        const int k1 = it / (C * NQ), r = it % (C * NQ), i3 = r / NQ;
        float2 *s = sm + k1 * BC * NQ + r;
        float2 v[B];
#pragma unroll
        for (int i2 = 0; i2 < B; ++i2) v[i2] = s[i2 * C * NQ];
        Dft<B, DIR, true>::run(v);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) s[k2 * C * NQ] = cmul(v[k2], __ldg(&tw2[k2 * C + i3]));
    }
    __syncthreads();
    for (int it = threadIdx.x; it < A * B * NQ; it += NT) {
        const int kk = it / NQ, q = it % NQ, k2 = kk / A, k1 = kk % A;   // kk = k1 + A k2
        const float2 *s = sm + (k1 * B + k2) * C * NQ + q;
        float2 w[C];
#pragma unroll
        for (int i3 = 0; i3 < C; ++i3) w[i3] = s[i3 * NQ];
        Dft<C, DIR, true>::run(w);
        out(kk, q, w);
    }
}

}  // namespace ptfft

// Host helper: fill tw[m] = exp(-2 pi i m / L), m < L (double precision).
void pt_make_twiddles(float2 *host_tw, int L);
