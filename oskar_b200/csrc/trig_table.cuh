// Table-driven phase factors e^{i ph} for the element loops of the station
// beam (Trig<T>, below, with larger tables) and, in FP64, of the weighted DFT
// and the smearing kernel's transform, where one sincos per phase bounds the
// kernel on the FP64 pipe.
//
// Method: P. T. P. Tang's table-driven scheme ("Table-lookup algorithms for
// elementary functions and their error analysis", ARITH 1991). The loops
// carry the phase in table steps, u = ph / h with h = 2 pi / 128 (the
// per-direction factors are pre-scaled by 1 / h, so u costs the same
// multiply-adds as ph would), and
//
//   u = n + f,  n = round(u),  |f| <= 1/2 (f = u - n exactly),
//   e^{i h u} = T[n mod 128] * e^{i h f},  T[j] = e^{2 pi i j / 128},
//
// with e^{i h f} from the Taylor series of sin and cos in x = h f,
// |x| <= pi / 128, written as polynomials in f: sin to x^7 and cos - 1 to
// x^6; the first omitted terms, x^9/9! and x^8/8!, are below 4e-18. n comes
// from adding 1.5 x 2^52, which leaves round(u) in the low bits of the
// sum; the high word of that sum is one of two values exactly when
// -2^32 <= n < 2^32 (|ph| below 2.1e8 rad), which is the range the table
// path covers. Other phases, infinities and NaN are flagged for sincospi().
//
// The table sits in shared memory as 8 copies interleaved entry by entry:
// entry j of copy c is element 8 j + c. A 16-byte shared load is served a
// quarter-warp (8 lanes) at a time, and lane l reads copy l mod 8, which
// lies in bank group l mod 8 whatever the index, so the random lookups of a
// warp take four wavefronts and never conflict. 16 KB per CTA.
//
// Cost per phase factor: 15 FP64 operations (3 for the reduction, 8 for the
// polynomials, 4 to rotate the table entry), one 16-byte shared load and
// three integer operations, against one library sincos.
#pragma once

#include "f32x2.cuh"

namespace oskb {

constexpr int kTrigEntries = 128;
constexpr int kTrigCopies = 8;
constexpr int kTrigTableSize = kTrigEntries * kTrigCopies;  // double2 slots

// 1 / h = 64 / pi: multiplies a phase in radians into table steps.
constexpr double kTrigStepsPerRadian = 20.371832715762604;

// Fills the table; all threads of the CTA take part and must reach a
// __syncthreads() before the first lookup.
__device__ __forceinline__ void trig_table_fill(double2* table)
{
    for (int j = threadIdx.x; j < kTrigEntries; j += blockDim.x)
    {
        double s, c;
        sincospi((double) j / (kTrigEntries / 2), &s, &c);
        // (each lane starts at its own copy: distinct banks)
#pragma unroll
        for (int k = 0; k < kTrigCopies; ++k)
            table[j * kTrigCopies + ((k + j) & (kTrigCopies - 1))] =
                    make_double2(c, s);
    }
}

// e^{i h u} as (*c, *s) from the copy of this lane. Clears *covered when u
// is outside the table's range (the result is then wrong but the lookup
// stays inside the table): hot loops accumulate the flag and redo the rare
// uncovered case with trig_steps_exact, so the unrolled body has no branch.
__device__ __forceinline__ void trig_steps_sincos(const double2* table,
        double u, double* s, double* c, bool& covered)
{
    constexpr double kShift = 6755399441055744.0;  // 1.5 x 2^52
    constexpr double h = 3.141592653589793 / 64.0;
    constexpr double s1 = h, s3 = -h * h * h / 6.0,
            s5 = h * h * h * h * h / 120.0,
            s7 = -h * h * h * h * h * h * h / 5040.0;
    constexpr double c2 = -h * h / 2.0, c4 = h * h * h * h / 24.0,
            c6 = -h * h * h * h * h * h / 720.0;
    const double t = u + kShift;
    const int n = __double2loint(t);
    covered &= (unsigned) (__double2hiint(t) - 0x4337FFFF) <= 1u;
    const double f = u - (t - kShift);
    const double f2 = f * f;
    // sin(h f) = f (s1 + f^2 (s3 + f^2 (s5 + f^2 s7)))
    const double sr = f * fma(f2, fma(f2, fma(f2, s7, s5), s3), s1);
    // cos(h f) - 1 = f^2 (c2 + f^2 (c4 + f^2 c6))
    const double cm = f2 * fma(f2, fma(f2, c6, c4), c2);
    const double2 e = table[((n & (kTrigEntries - 1)) * kTrigCopies) |
            (threadIdx.x & (kTrigCopies - 1))];
    // (e.x + i e.y)(1 + cm + i sr), the small terms added to e last
    *c = fma(e.x, cm, fma(-e.y, sr, e.x));
    *s = fma(e.y, cm, fma(e.x, sr, e.y));
}

// e^{i h u} for any u, through the library: sincospi(u / 64) (u / 64 is
// exact).
__device__ __forceinline__ void trig_steps_exact(double u, double* s,
        double* c)
{
    sincospi(u * (1.0 / (kTrigEntries / 2)), s, c);
}

// e^{i h u} for any u: the table where it covers u, else the library.
__device__ __forceinline__ void trig_steps_checked(const double2* table,
        double u, double* s, double* c)
{
    bool covered = true;
    trig_steps_sincos(table, u, s, c, covered);
    if (!covered) trig_steps_exact(u, s, c);
}

// ---------------------------------------------------------------------------
// The station beam's larger tables, with shorter series. Entry j of copy c is
// element kCopies j + c, as above (FP32: 16 copies of 8-byte entries, for
// half-warp requests). N entries: h = 2 pi / N, |x| = |h f| <= pi / N. The
// fill takes the first quadrant's entries from the library and turns them, so
// that a small CTA has two sines to form instead of eight.
//   FP64, N = 512 (64 KB): sin to x^5 (the omitted x^7/7! < 7e-20) and
//     cos - 1 to x^4 with the x^6 term economised into the lower two
//     (Chebyshev; what is left is below 5e-18): 13 operations.
//   FP32, N = 256 (32 KB): sin to x^3 (x^5/5! < 3e-12) and cos - 1 as one
//     economised x^2 term (left: 2e-10): 11 operations.
// The caller bounds the phase: |u| < kLimit, where round(u) still sits in
// the low bits of u + 1.5 x 2^52 (FP32: 2^23).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sincos_half_turns(double x, double* s,
        double* c)
{
    sincospi(x, s, c);
}
__device__ __forceinline__ void sincos_half_turns(float x, float* s, float* c)
{
    sincospif(x, s, c);
}

// Fills COPIES copies of the N entries (cos, sin)(2 pi j / N) from those of
// the first quadrant: every thread takes one entry of it at a time and writes
// it turned by 0, 1, 2 and 3 right angles; where the CTA has more threads
// than the quadrant entries, several threads share an entry's four turns.
template <int N, int COPIES, typename T2>
__device__ __forceinline__ void trig_fill_quadrants(T2* table)
{
    constexpr int Q = N / 4;
    const int share = min(4, max(1, (int) blockDim.x / Q));  // 1, 2 or 4
    for (int i = threadIdx.x; i < Q * share; i += blockDim.x)
    {
        const int j = i % Q;
        T2 e;   // (cos, sin)
        sincos_half_turns((decltype(e.x)) j / (N / 2), &e.y, &e.x);
        for (int q = i / Q; q < 4; q += share)
        {
            T2 v = e;
            if (q & 1) { v.x = 0 - e.y; v.y = e.x; }
            if (q & 2) { v.x = 0 - v.x; v.y = 0 - v.y; }
            // (each lane starts at its own copy: distinct banks)
#pragma unroll
            for (int k = 0; k < COPIES; ++k)
                table[(j + q * Q) * COPIES + ((k + j) & (COPIES - 1))] = v;
        }
    }
}

template <typename T> struct Trig;

template <> struct Trig<double>
{
    typedef double2 Entry;
    static constexpr int kEntries = 512, kCopies = 8;
    static constexpr int kSize = kEntries * kCopies;
    static constexpr double kStepsPerRadian = 81.48733086305042;  // 256 / pi
    static constexpr double kLimit = 4294967296.0;

    static __device__ __forceinline__ void fill(Entry* table)
    {
        trig_fill_quadrants<kEntries, kCopies>(table);
    }
    static __device__ __forceinline__ void sincos(const Entry* table,
            double u, double* s, double* c)
    {
        constexpr double kShift = 6755399441055744.0;  // 1.5 x 2^52
        constexpr double h = 3.141592653589793 / (kEntries / 2);
        constexpr double h2 = h * h, h4 = h2 * h2, h6 = h4 * h2;
        constexpr double s1 = h, s3 = -h * h2 / 6.0, s5 = h * h4 / 120.0;
        // f2^3 on [0, 1/4] as 3/8 f2^2 - 9/256 f2 (+ 1/2048)
        constexpr double c4 = h4 / 24.0 - h6 / 720.0 * (3.0 / 8.0);
        constexpr double c2 = -h2 / 2.0 + h6 / 720.0 * (9.0 / 256.0);
        const double t = u + kShift;
        const int n = __double2loint(t);
        const double f = u - (t - kShift);
        const double f2 = f * f;
        const double sr = f * fma(f2, fma(f2, s5, s3), s1);
        const double cm = f2 * fma(f2, c4, c2);
        const Entry e = table[((n & (kEntries - 1)) * kCopies) |
                (threadIdx.x & (kCopies - 1))];
        *c = fma(e.x, cm, fma(-e.y, sr, e.x));
        *s = fma(e.y, cm, fma(e.x, sr, e.y));
    }
    static __device__ __forceinline__ void exact(double u, double* s,
            double* c)
    {
        sincospi(u * (1.0 / (kEntries / 2)), s, c);
    }
    static __device__ __forceinline__ void checked(const Entry* table,
            double u, double* s, double* c)
    {
        if (fabs(u) < kLimit) sincos(table, u, s, c);
        else exact(u, s, c);
    }
};

template <> struct Trig<float>
{
    typedef float2 Entry;
    static constexpr int kEntries = 256, kCopies = 16;
    static constexpr int kSize = kEntries * kCopies;
    static constexpr double kStepsPerRadian = 40.74366543152521;  // 128 / pi
    static constexpr float kLimit = 2097152.0f;
    static constexpr float kShift = 12582912.0f;  // 1.5 x 2^23
    static constexpr double h = 3.141592653589793 / (kEntries / 2);
    static constexpr float s1 = (float) h, s3 = (float) (-h * h * h / 6.0);
    // f2^2 on [0, 1/4] as f2 / 4 (- 1/128)
    static constexpr float c2 = (float) (-h * h / 2.0 + h * h * h * h / 24.0
            / 4.0);

    // The entry of round(u), in the low bits of t = u + kShift, turned by
    // the remainder's sine and cosine - 1.
    static __device__ __forceinline__ void rotate(const Entry* table, float t,
            float sr, float cm, float* s, float* c)
    {
        const int n = __float_as_int(t);
        const Entry e = table[((n & (kEntries - 1)) * kCopies) |
                (threadIdx.x & (kCopies - 1))];
        *c = fmaf(e.x, cm, fmaf(-e.y, sr, e.x));
        *s = fmaf(e.y, cm, fmaf(e.x, sr, e.y));
    }

    static __device__ __forceinline__ void fill(Entry* table)
    {
        trig_fill_quadrants<kEntries, kCopies>(table);
    }
    // One phase.
    static __device__ __forceinline__ void sincos(const Entry* table, float u,
            float* s, float* c)
    {
        const float t = u + kShift;
        const float f = u - (t - kShift);
        const float f2 = f * f;
        rotate(table, t, f * fmaf(f2, s3, s1), f2 * c2, s, c);
    }
    // Two phases as a packed pair.
    static __device__ __forceinline__ void sincos2(const Entry* table,
            f32x2 u, float* s, float* c)
    {
        const f32x2 t = add2(u, pack2(kShift, kShift));
        const f32x2 f = fma2(add2(t, pack2(-kShift, -kShift)),
                pack2(-1.0f, -1.0f), u);
        const f32x2 f2 = mul2(f, f);
        const f32x2 sr2 = mul2(f, fma2(f2, pack2(s3, s3), pack2(s1, s1)));
        const f32x2 cm2 = mul2(f2, pack2(c2, c2));
        float tt[2], sr[2], cm[2];
        unpack2(t, tt[0], tt[1]);
        unpack2(sr2, sr[0], sr[1]);
        unpack2(cm2, cm[0], cm[1]);
#pragma unroll
        for (int j = 0; j < 2; ++j)
            rotate(table, tt[j], sr[j], cm[j], &s[j], &c[j]);
    }
    static __device__ __forceinline__ void exact(float u, float* s, float* c)
    {
        sincospif(u * (1.0f / (kEntries / 2)), s, c);
    }
    static __device__ __forceinline__ void checked(const Entry* table,
            float u, float* s, float* c)
    {
        if (fabsf(u) < kLimit) sincos(table, u, s, c);
        else exact(u, s, c);
    }
};

}  // namespace oskb
