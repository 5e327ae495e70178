// Direct cross-correlation with per-baseline factors: Gaussian sources and
// bandwidth and time-average smearing, where
//     V_pq += sum_s f_pq(s) (J_p B J_q^H)(s),
// f the product of exp(-(a uu^2 + 2 b uu vv + c vv^2)) and of
// sinc(phi_p - phi_q) per smearing (define_cross_correlate.h:16-111). The
// factor depends on the baseline, so nothing separates into station terms
// and the work stays on the FP64 (FP32) pipe: per source-baseline of the
// matrix form 40 multiply-adds of the product and about 23 of two smearing
// factors.
//
// One CTA of 512 threads owns a 32 x 32 station tile, its 16 warps an 8 x 8
// station patch each, two baselines per thread (FP64: two rows p; FP32: two
// columns q, as packed pairs). Two baselines keep a thread within 128
// registers (most FP64 matrix forms at 128, spilling up to 24 bytes), so 16
// warps fit an SM: with four baselines per thread 8 warps of 248 registers
// were latency-bound (FP64 pipe 35 % active; now 58 %, and what is left is
// the latency of a source's chain of loads, reciprocal and select with four
// warps per scheduler). A warp whose patch holds no baseline
// (above the diagonal, past the last station) skips the arithmetic; the
// patches are dealt so that a diagonal tile's ten live ones spread over the
// four schedulers.
//
// Warp w also stages and transforms 4 stations (w % 8) of block w / 8 (rows
// or columns) of every chunk of 8 sources: its cp.async copies land in its
// own raw buffer, and J B, J, K E and the per-station smearing phases with
// their sines and cosines go into one of two factor buffers, so that a chunk
// needs one block barrier. Half of each scheduler's warps transform the next
// chunk before the current chunk's products and half after, so that the
// serial transform of some overlaps the products of the others.
//
// Measured on one B200, 30 % Gaussian sources, both smearings, against the
// four-baseline kernel: 256 stations x 20,000 sources x 4 channels FP64 20.1
// ms (30.5 before: 130 G source-baselines/s against 86); 211 stations x
// 9,001 sources x 6 FP32 5.8 ms (9.5).
#pragma once

#include "f32x2.cuh"
#include "trig_table.cuh"
#include "xcorr_common.cuh"

namespace oskb {
namespace {

constexpr int kSmearThreads = 512;
// Stations per source row of 16-byte and 8-byte factors, padded: a warp's
// transform writes 4 stations of 8 sources at a time, in distinct banks.
constexpr int kPad16 = kTile + 1;
constexpr int kPad8 = kTile + 2;
constexpr int kSrcWarp = 11;   // copies the per-source values

// Factors of one chunk. FP64: rows and columns [comp][source][station]
// complex; smearing phase phi and (sin, cos) per block.
template <typename T, int NC>
struct SmearFactors
{
    double2 row[NC][kChunk][kPad16];
    double2 col[NC][kChunk][kPad16];
    double phi[2][2][kChunk][kPad8];    // [bandwidth, time][block]
    double2 sc[2][2][kChunk][kPad16];
    double gauss[kChunk][4];            // a, b, c of the source
};

// FP32: packed operands. A row (p) value is stored twice {x, x}; a column
// (q) pair holds stations 2 j and 2 j + 1. The row cosine is negated, so
// that sin_p cos_q - cos_p sin_q is one multiply and one multiply-add.
template <int NC>
struct SmearFactors<float, NC>
{
    float4 row[NC][kChunk][kPad16];         // {re, re, im, im}
    float4 col[NC][kChunk][kTile / 2 + 1];  // {re0, re1, im0, im1}
    float4 row_ps[2][kChunk][kPad16];       // {phi, phi, sin, sin}
    float2 row_c[2][kChunk][kPad8];         // {-cos, -cos}
    float4 col_ps[2][kChunk][kTile / 2 + 1];    // {phi0, phi1, sin0, sin1}
    float2 col_c[2][kChunk][kTile / 2 + 1];     // {cos0, cos1}
    float gauss[kChunk][4];
};

template <typename T, bool MATRIX>
struct SmearSmem
{
    typedef Staging<T, MATRIX> G;
    static constexpr int NCOMP = MATRIX ? 4 : 1;
    // The next chunk's Jones, per warp (4 stations x 8 sources):
    // [warp][piece][element] x COPY bytes
    __align__(16) unsigned char raw[kSmearThreads / 32][G::PIECES][32]
            [G::COPY];
    SmearFactors<T, NCOMP> f[2];
    // FP64: phase factors of the fused K (trig_table.cuh)
    double2 trig[sizeof(T) == 8 ? kTrigTableSize : 1];
    T raw_src[2][kNumSrcArr][kChunk];       // per-source values of a chunk
    // Per item: station u, v, w (bandwidth phase, fused K) and the rotated
    // x, y pair (time smearing).
    T st_uvw[2][kTile][3];
    double st_xy[2][kTile][2];
    unsigned bound[2];   // longest baseline of the tile in phase units (bits)
};

// sinc(d) = sin(d) / d of a phase difference d, from the per-station sin and
// cos: sin(a - b) = sin a cos b - cos a sin b. Where d is small the identity
// loses relative accuracy (its absolute error is a few ulp of 1), so below
// |d| = tau the series of sinc is summed instead. FP64, tau = 1/16: 1 - y/6 +
// y^2/120 - y^3/5040 + y^4/362880 (y = d^2; the next term is below 3e-20)
// with the y^4 term economised into the lower ones (Chebyshev on [0, tau^2]:
// y^4 = 2 t y^3 - 5/4 t^2 y^2 + 1/4 t^3 y to within t^4/64, t = tau^2, the
// constant t^4/128 left out as well; the remainder is 1.0e-17). FP32, tau =
// 1/2: the five terms (next: 3e-11). Above tau the identity's relative error
// is below ~1e-14 (FP64; measured 3.4e-15 from 0 to 700 rad) and ~1e-6
// (FP32). Both forms are evaluated and one selected (no divergence within a
// warp), as a numerator and a denominator (sin d, d) or (series, 1), so that
// the bandwidth and time factors of a source-baseline share one reciprocal.
template <typename T>
constexpr T kSincTau = sizeof(T) == 8 ? (T) (1.0 / 16) : (T) 0.5;

__device__ __forceinline__ double sinc_series(double d)
{
    constexpr double t = 1.0 / 256, c4 = 1.0 / 362880;
    constexpr double a3 = -1.0 / 5040 + c4 * 2 * t;
    constexpr double a2 = 1.0 / 120 - c4 * 1.25 * t * t;
    constexpr double a1 = -1.0 / 6 + c4 * 0.25 * t * t * t;
    const double y = d * d;
    return fma(y, fma(y, fma(y, a3, a2), a1), 1.0);
}

__device__ __forceinline__ f32x2 sinc_series(f32x2 d)
{
    const f32x2 y = mul2(d, d);
    f32x2 s = fma2(y, pack2((float) (1.0 / 362880), (float) (1.0 / 362880)),
            pack2((float) (-1.0 / 5040), (float) (-1.0 / 5040)));
    s = fma2(y, s, pack2((float) (1.0 / 120), (float) (1.0 / 120)));
    s = fma2(y, s, pack2((float) (-1.0 / 6), (float) (-1.0 / 6)));
    return fma2(y, s, pack2(1.0f, 1.0f));
}

__device__ __forceinline__ void sinc_parts(double d, double by_identity,
        double& num, double& den)
{
    const double by_series = sinc_series(d);
    // |d| < 1/16 by its exponent (an integer comparison; false for NaN)
    const bool small = (__double2hiint(d) & 0x7fffffff) < 0x3fb00000;
    num = small ? by_series : by_identity;
    den = small ? 1.0 : d;
}

// num / den for |den| >= 1/256: the hardware's reciprocal approximation y
// (20 bits of den give 20 bits: e = 1 - den y is at most about 2^-19), and
// the quotient num y corrected by 1 / (1 - e) = 1 + e + e^2 (+ e^3 < 2^-57):
// a short dependent chain instead of the IEEE division's; within an ulp or
// two of the correctly rounded quotient (a whole call's error is that with
// the division to three digits).
__device__ __forceinline__ double quotient(double num, double den)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(den));
    const double e = fma(-den, y, 1.0);
    const double q = num * y;
    return fma(q, fma(e, e, e), q);
}

// One chunk's Jones of the warp's 4 stations, in copies of consecutive lanes:
// the 8 sources of a station are contiguous (512 bytes in FP64), so an
// instruction touches one to four short runs. (A source per warp, 64 bytes
// of each of 8 stations per instruction, measured 3 % (FP64 block) to 7 %
// (FP32) slower.) Entries outside the stations or sources are zero-filled
// without a global read.
template <typename T, bool MATRIX>
__device__ __forceinline__ void smear_issue(SmearSmem<T, MATRIX>& sm,
        const XcorrParams<T>& prm, const T* jsrc, const ItemCtx& ctx, int s0)
{
    typedef Staging<T, MATRIX> G;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (jsrc)
    {
        const unsigned char* jb = reinterpret_cast<const unsigned char*>(jsrc);
        const int st0 = (warp < 8 ? ctx.p0 : ctx.q0) + 4 * (warp & 7);
#pragma unroll
        for (int i = 0; i < G::PIECES; ++i)
        {
            const int idx = 32 * i + lane, pc = idx % G::PIECES;
            const int el = idx / G::PIECES;   // station x source
            const int st = st0 + (el >> 3), s = s0 + (el & 7);
            const bool in = st < prm.num_st && s < ctx.src_end;
            const unsigned char* src = in ? jb + ((size_t) st *
                    prm.src_stride + s) * G::ELEM + pc * G::COPY : jb;
            cp_async(sm.raw[warp][pc][el], src, in, G::COPY);
        }
    }
    cp_async_commit();
}

// The per-source values of one chunk (those this variant reads), by one
// warp, into buffer b.
template <typename T, bool MATRIX, bool GAUSS, bool LMN>
__device__ __forceinline__ void smear_issue_src(SmearSmem<T, MATRIX>& sm,
        const XcorrParams<T>& prm, const ItemCtx& ctx, int s0, int b)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < (kNumSrcArr * kChunk + 31) / 32; ++i)
    {
        const int k = (32 * i + lane) / kChunk, sl = lane % kChunk;
        const bool want = (k == kI) || (MATRIX && k <= kV) ||
                (LMN && k >= kL && k <= kN) || (GAUSS && k >= kGa &&
                k < kNumSrcArr);
        if (!want) continue;
        const T* arr = k == kI ? prm.I : k == kQ ? prm.Q : k == kU ? prm.U :
                k == kV ? prm.V : k == kL ? prm.l : k == kM ? prm.m :
                k == kN ? prm.n : k == kGa ? prm.a : k == kGb ? prm.b :
                prm.c;
        const long long off = k <= kV ? ctx.c * prm.flux_channel_stride : 0;
        const int s = s0 + sl;
        const bool in = s < ctx.src_end;
        cp_async(&sm.raw_src[b][k][sl], in ? arr + off + s : prm.I, in,
                (int) sizeof(T));
    }
    cp_async_commit();
}

// The larger value, or NaN where one is (as bits of a non-negative value).
__device__ __forceinline__ float max_or_nan(float a, float b)
{
    return __uint_as_float(max(__float_as_uint(a), __float_as_uint(b)));
}

// FP32: whether every phase difference of a chunk is below tau: reach is the
// chunk's largest |(l, m, n - 1)|, bw and ts the longest baseline in phase
// units (0 without that smearing). False for NaN. The series alone is then
// taken, as in arrays of a few km (211 stations x 9,001 sources x 6, 2 km:
// 6.2 -> 5.8 ms); in FP64 tau = 1/16 seldom holds, and a second loop cost 3
// to 5 % where it did not.
__device__ __forceinline__ bool sinc_small(float reach, float bw, float ts)
{
    return reach * bw < kSincTau<float> && reach * ts < kSincTau<float>;
}

// Stores one element's factor values.
template <int NC>
__device__ __forceinline__ void put_entry(SmearFactors<double, NC>& f,
        int blk, int k, int sl, int stl, double re, double im)
{
    (blk ? f.col : f.row)[k][sl][stl] = make_double2(re, im);
}
template <int NC>
__device__ __forceinline__ void put_entry(SmearFactors<float, NC>& f,
        int blk, int k, int sl, int stl, float re, float im)
{
    if (blk)
    {
        float* o = &f.col[k][sl][stl >> 1].x + (stl & 1);
        o[0] = re;
        o[2] = im;
    }
    else
    {
        f.row[k][sl][stl] = make_float4(re, re, im, im);
    }
}
// The station's smearing phase with its sine and cosine, by the library:
// they are those of the stored phase, as the identity above needs, whose
// error over d shows every difference between the two (through the phase in
// table steps, rounded once more, the factor was off by up to 1.4e-12 at 700
// rad). The table's sine and cosine of the unrounded steps were 1.3 times the
// library's error at the same time (197 stations x 4,001 sources: 607 us,
// 600 with the rounded steps).
template <int NC>
__device__ __forceinline__ void put_phase(SmearFactors<double, NC>& f,
        int which, int blk, int sl, int stl, double ph, bool)
{
    f.phi[which][blk][sl][stl] = ph;
    double sn, cs;
    sincos(ph, &sn, &cs);
    f.sc[which][blk][sl][stl] = make_double2(sn, cs);
}
template <int NC>
__device__ __forceinline__ void put_phase(SmearFactors<float, NC>& f,
        int which, int blk, int sl, int stl, float ph, bool small)
{
    float sn = 0.0f, cs = 1.0f;
    if (!small) sincosf(ph, &sn, &cs);
    if (blk)
    {
        float* o = &f.col_ps[which][sl][stl >> 1].x + (stl & 1);
        o[0] = ph;
        o[2] = sn;
        (&f.col_c[which][sl][stl >> 1].x)[stl & 1] = cs;
    }
    else
    {
        f.row_ps[which][sl][stl] = make_float4(ph, ph, sn, sn);
        f.row_c[which][sl][stl] = make_float2(-cs, -cs);
    }
}

// The warp's elements of a landed chunk, one per lane: station 4 (warp % 8) +
// lane / 8 of block warp / 8, source lane % 8. in_range: the source exists
// (else every factor is zero: the raw values were zero-filled).
template <typename T, bool MATRIX, bool GAUSS, bool BW, bool TS, bool CASA,
        bool FUSED>
__device__ __forceinline__ void smear_transform(SmearSmem<T, MATRIX>& sm,
        const XcorrParams<T>& prm, bool have_jones, const ItemCtx& ctx,
        T wavenumber, bool in_range, int buf, float& reach)
{
    typedef typename vec2<T>::type T2;
    typedef Staging<T, MATRIX> G;
    constexpr int NC = MATRIX ? 4 : 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int blk = warp >> 3, stl = 4 * (warp & 7) + (lane >> 3);
    const int sl = lane & 7;
    const T (*src)[kChunk] = sm.raw_src[buf];
    SmearFactors<T, NC>& f = sm.f[buf];
    T v[2 * NC];
    if (have_jones)
    {
        constexpr int PER = G::COPY / (int) sizeof(T);
#pragma unroll
        for (int pc = 0; pc < G::PIECES; ++pc)
        {
            if constexpr (G::COPY == 16)
            {
                const uint4 u = *reinterpret_cast<const uint4*>(
                        sm.raw[warp][pc][lane]);
                memcpy(&v[pc * PER], &u, 16);
            }
            else
            {
                const uint2 u = *reinterpret_cast<const uint2*>(
                        sm.raw[warp][pc][lane]);
                memcpy(&v[pc * PER], &u, 8);
            }
        }
    }
    else
    {
        // Identity E (fused mode without a station beam).
#pragma unroll
        for (int k = 0; k < 2 * NC; ++k) v[k] = (T) 0;
        v[0] = (T) 1;
        if (MATRIX) v[6] = (T) 1;
    }
    if (FUSED)
    {
        // J = K E with the reference's K
        // (oskar/interferometer/define_evaluate_jones_K.h:53-70).
        const T* u = sm.st_uvw[blk][stl];
        const T l = src[kL][sl], m = src[kM][sl], n1 = src[kN][sl] - (T) 1;
        const T flux = src[kI][sl];
        const T phase = (u[0] * l + u[1] * m + u[2] * n1) * wavenumber;
        T ks, kc;
        if constexpr (sizeof(T) == 8)
            trig_steps_checked(sm.trig, phase, &ks, &kc);
        else
            sincos(phase, &ks, &kc);
        if (!(in_range && flux > (T) prm.filter_min &&
                flux <= (T) prm.filter_max))
            ks = kc = (T) 0;
#pragma unroll
        for (int k = 0; k < NC; ++k)
        {
            const T re = v[2 * k], im = v[2 * k + 1];
            v[2 * k] = kc * re - ks * im;
            v[2 * k + 1] = kc * im + ks * re;
        }
    }
    // Left factor (J B, or I J) lives in the row block unless CASA.
    const bool left = (blk == 0) != CASA;
    if constexpr (MATRIX)
    {
        if (left)
        {
            const T I = src[kI][sl], Q = src[kQ][sl];
            const T2 buv = T2{src[kU][sl], src[kV][sl]};
            const T2 buvc = T2{buv.x, -buv.y};
            const T xx = I + Q, yy = I - Q;
#pragma unroll
            for (int r = 0; r < 4; r += 2)
            {
                const T2 j0 = T2{v[2 * r], v[2 * r + 1]};
                const T2 j1 = T2{v[2 * r + 2], v[2 * r + 3]};
                const T2 t0 = cmul<T>(j1, buvc), t1 = cmul<T>(j0, buv);
                v[2 * r] = j0.x * xx + t0.x;
                v[2 * r + 1] = j0.y * xx + t0.y;
                v[2 * r + 2] = j1.x * yy + t1.x;
                v[2 * r + 3] = j1.y * yy + t1.y;
            }
        }
    }
    else if (left)
    {
        v[0] *= src[kI][sl];
        v[1] *= src[kI][sl];
    }
#pragma unroll
    for (int k = 0; k < NC; ++k)
        put_entry(f, blk, k, sl, stl, v[2 * k], v[2 * k + 1]);
    if (BW || TS)
    {
        // Per-station source phases (phi_p - phi_q is the reference's
        // baseline argument), in FP64.
        const T* u = sm.st_uvw[blk][stl];
        const double* xy = sm.st_xy[blk][stl];
        const double l = src[kL][sl], m = src[kM][sl];
        const double n1 = (double) src[kN][sl] - 1.0;
        // the chunk's largest |(l, m, n - 1)|: times a baseline's length in
        // phase units, it bounds the phase differences of the chunk (for
        // the time smearing too: (s m - c (n - 1)) is no longer than
        // (m, n - 1))
        if (sizeof(T) == 4)
        {
            const float r = in_range ? 1.0001f * sqrtf((float) (l * l +
                    m * m + n1 * n1)) : 0.0f;
            reach = __uint_as_float(__reduce_max_sync(0xffffffffu,
                    __float_as_uint(r)));
        }
        const bool small = sizeof(T) == 4 && sinc_small(reach,
                __uint_as_float(sm.bound[0]), __uint_as_float(sm.bound[1]));
        if (BW)
            put_phase(f, 0, blk, sl, stl, (T) (((double) u[0] * l +
                    (double) u[1] * m + (double) u[2] * n1) * prm.bw_scale),
                    small);
        if (TS)
            put_phase(f, 1, blk, sl, stl, (T) ((xy[0] * l + xy[1] *
                    (prm.s_dec * m - prm.c_dec * n1)) * ctx.ts_scale), small);
    }
    if (GAUSS && warp < 3 && lane < kChunk)
        f.gauss[lane][warp] = src[kGa + warp][lane];
}

// One chunk's products, FP64: the thread's rows pr, pr + 1 and column qc.
template <bool MATRIX, bool GAUSS, bool BW, bool TS, bool CASA>
__device__ __forceinline__ void smear_products(
        const SmearFactors<double, MATRIX ? 4 : 1>& f, int ns, int pr, int qc,
        const double (&uu2)[2], const double (&vv2)[2],
        const double (&uuvv)[2], double (&acc)[2][MATRIX ? 8 : 2])
{
    constexpr int NC = MATRIX ? 4 : 1;
#pragma unroll 1
    for (int sl = 0; sl < ns; ++sl)
    {
        // ---- factors of the two baselines
        double w[2] = {1.0, 1.0};
        if (BW || TS)
        {
            double num[2], den[2];
#pragma unroll
            for (int which = BW ? 0 : 1; which < (TS ? 2 : 1); ++which)
            {
                const double pb = f.phi[which][1][sl][qc];
                const double2 b = f.sc[which][1][sl][qc];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                {
                    const double2 a = f.sc[which][0][sl][pr + i];
                    double nu, de;
                    sinc_parts(f.phi[which][0][sl][pr + i] - pb,
                            a.x * b.y - a.y * b.x, nu, de);
                    const bool first = !(BW && which == 1);
                    num[i] = first ? nu : num[i] * nu;
                    den[i] = first ? de : den[i] * de;
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) w[i] = quotient(num[i], den[i]);
        }
        if (GAUSS)
        {
            // a point source (a = b = c = 0, exp(-0) = 1 exactly) skips it
            const double ga = f.gauss[sl][0], gb = f.gauss[sl][1],
                    gc = f.gauss[sl][2];
            if (ga != 0.0 || gb != 0.0 || gc != 0.0)
            {
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    w[i] *= exp(-(ga * uu2[i] + gb * uuvv[i] + gc * vv2[i]));
            }
        }
        // ---- products: each part of L R^H, then times the factor
        double2 C[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) C[k] = f.col[k][sl][qc];
#pragma unroll
        for (int i = 0; i < 2; ++i)
        {
            double2 R[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) R[k] = f.row[k][sl][pr + i];
            const double2* L = CASA ? C : R;
            const double2* Rt = CASA ? R : C;
            double* o = acc[i];
#pragma unroll
            for (int e = 0; e < NC; ++e)
            {
                // element e = (r, c): sum_u L[2r + u] conj(Rt[2c + u])
                double re = 0, im = 0;
#pragma unroll
                for (int u = 0; u < (MATRIX ? 2 : 1); ++u)
                {
                    const double2 x = L[MATRIX ? 2 * (e >> 1) + u : 0];
                    const double2 y = Rt[MATRIX ? 2 * (e & 1) + u : 0];
                    re = u ? fma(x.x, y.x, re) : x.x * y.x;
                    im = u ? fma(x.y, y.x, im) : x.y * y.x;
                    re = fma(x.y, y.y, re);
                    im = fma(-x.x, y.y, im);
                }
                o[2 * e] = fma(re, w[i], o[2 * e]);
                o[2 * e + 1] = fma(im, w[i], o[2 * e + 1]);
            }
        }
    }
}

// One chunk's products, FP32: the thread's row pr and columns qc, qc + 1 as
// packed pairs; the chunk's sums are added to the FP64 sums at its end.
// SMALL: every phase difference of the warp's patch is below tau.
template <bool MATRIX, bool GAUSS, bool BW, bool TS, bool CASA, bool SMALL>
__device__ __forceinline__ void smear_products(
        const SmearFactors<float, MATRIX ? 4 : 1>& f, int ns, int pr, int qc,
        const float (&uu2)[2], const float (&vv2)[2],
        const float (&uuvv)[2], double (&acc)[2][MATRIX ? 8 : 2])
{
    constexpr int NC = MATRIX ? 4 : 1;
    const int qp = qc >> 1;
    f32x2 part[2 * NC];
#pragma unroll
    for (int k = 0; k < 2 * NC; ++k) part[k] = 0;
#pragma unroll 1
    for (int sl = 0; sl < ns; ++sl)
    {
        float w[2] = {1.0f, 1.0f};
        if ((BW || TS) && SMALL)
        {
            f32x2 x = 0;
#pragma unroll
            for (int which = BW ? 0 : 1; which < (TS ? 2 : 1); ++which)
            {
                const f32x2 a = *reinterpret_cast<const f32x2*>(
                        &f.row_ps[which][sl][pr]);
                const f32x2 b = *reinterpret_cast<const f32x2*>(
                        &f.col_ps[which][sl][qp]);
                const f32x2 y = sinc_series(fma2(b, pack2(-1.0f, -1.0f), a));
                x = BW && which == 1 ? mul2(x, y) : y;
            }
            unpack2(x, w[0], w[1]);
        }
        else if (BW || TS)
        {
            float num[2], den[2];
#pragma unroll
            for (int which = BW ? 0 : 1; which < (TS ? 2 : 1); ++which)
            {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(
                        &f.row_ps[which][sl][pr]);
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(
                        &f.col_ps[which][sl][qp]);
                const f32x2 nca = *reinterpret_cast<const f32x2*>(
                        &f.row_c[which][sl][pr]);
                const f32x2 cb = *reinterpret_cast<const f32x2*>(
                        &f.col_c[which][sl][qp]);
                const f32x2 d = fma2(b.x, pack2(-1.0f, -1.0f), a.x);
                const f32x2 ident = fma2(nca, b.y, mul2(a.y, cb));
                const f32x2 ser = sinc_series(d);
                float dd[2], id[2], se[2];
                unpack2(d, dd[0], dd[1]);
                unpack2(ident, id[0], id[1]);
                unpack2(ser, se[0], se[1]);
#pragma unroll
                for (int j = 0; j < 2; ++j)
                {
                    const bool small = fabsf(dd[j]) < kSincTau<float>;
                    const float nu = small ? se[j] : id[j];
                    const float de = small ? 1.0f : dd[j];
                    const bool first = !(BW && which == 1);
                    num[j] = first ? nu : num[j] * nu;
                    den[j] = first ? de : den[j] * de;
                }
            }
            // |den| >= 0.25 (each factor's d is 1 or at least tau = 0.5),
            // well inside the range where the fast division is accurate to
            // 2 ulp
#pragma unroll
            for (int j = 0; j < 2; ++j) w[j] = __fdividef(num[j], den[j]);
        }
        if (GAUSS)
        {
            const float ga = f.gauss[sl][0], gb = f.gauss[sl][1],
                    gc = f.gauss[sl][2];
            if (ga != 0.0f || gb != 0.0f || gc != 0.0f)
            {
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    w[j] *= expf(-(ga * uu2[j] + gb * uuvv[j] + gc * vv2[j]));
            }
        }
        const f32x2 ww = pack2(w[0], w[1]);
        // real and imaginary parts of the column pair and the row
        f32x2 cr[NC], ci[NC], rr[NC], ri[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k)
        {
            const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(
                    &f.col[k][sl][qp]);
            cr[k] = c.x;
            ci[k] = c.y;
            const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(
                    &f.row[k][sl][pr]);
            rr[k] = r.x;
            ri[k] = r.y;
        }
        const f32x2* xr = CASA ? cr : rr;
        const f32x2* xi = CASA ? ci : ri;
        const f32x2* yr = CASA ? rr : cr;
        const f32x2* yi = CASA ? ri : ci;
        // -y_i once per component: Im = x_i y_r - x_r y_i
        f32x2 nyi[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) nyi[k] = neg2(yi[k]);
#pragma unroll
        for (int e = 0; e < NC; ++e)
        {
            f32x2 re = 0, im = 0;
#pragma unroll
            for (int u = 0; u < (MATRIX ? 2 : 1); ++u)
            {
                const int x = MATRIX ? 2 * (e >> 1) + u : 0;
                const int y = MATRIX ? 2 * (e & 1) + u : 0;
                re = u ? fma2(xr[x], yr[y], re) : mul2(xr[x], yr[y]);
                im = u ? fma2(xi[x], yr[y], im) : mul2(xi[x], yr[y]);
                re = fma2(xi[x], yi[y], re);
                im = fma2(xr[x], nyi[y], im);
            }
            part[2 * e] = fma2(re, ww, part[2 * e]);
            part[2 * e + 1] = fma2(im, ww, part[2 * e + 1]);
        }
    }
#pragma unroll
    for (int k = 0; k < 2 * NC; ++k)
    {
        float x, y;
        unpack2(part[k], x, y);
        acc[0][k] += (double) x;
        acc[1][k] += (double) y;
    }
}

template <typename T, bool MATRIX, bool GAUSS, bool BW, bool TS, bool CASA,
        bool FUSED>
__global__ void __launch_bounds__(kSmearThreads, 1)
xcorr_smear_kernel(const XcorrParams<T> prm)
{
    typedef SmearSmem<T, MATRIX> S;
    constexpr int NC = MATRIX ? 4 : 1;
    constexpr bool LMN = BW || TS || FUSED;
    constexpr bool F64 = sizeof(T) == 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S& sm = *reinterpret_cast<S*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // products: the warp's 8 x 8 patch, and the thread's stations in it
    const int pi = warp >> 2, qi = ((warp & 3) - pi) & 3;
    const bool early = pi & 1;   // transforms before the products
    const int pr = 8 * pi + (F64 ? 2 * (lane >> 3) : lane >> 2);
    const int qc = 8 * qi + (F64 ? lane & 7 : 2 * (lane & 3));
    const int N = prm.num_st;
    const int num_items = prm.num_times * prm.num_channels * prm.tiles *
            prm.slices;

    if (F64 && FUSED) trig_table_fill(sm.trig);   // synchronised below
    for (int item = blockIdx.x; item < num_items; item += gridDim.x)
    {
    ItemCtx ctx;
    const int slice = decode_item(prm, item, TS, ctx);
    const T* su = prm.st_u + ctx.t * prm.uvw_time_stride;
    const T* sv = prm.st_v + ctx.t * prm.uvw_time_stride;
    const T* sw = prm.st_w + ctx.t * prm.uvw_time_stride;
    const T* jsrc = !FUSED ? prm.jones : (prm.jones ?
            prm.jones + ctx.t * prm.e_time_stride : nullptr);
    // radians (FP32) or table steps (FP64: 2 pi x 64 / pi = 128) per metre
    const T wavenumber = F64 ? (T) (128.0 * ctx.inv_wavelength) :
            (T) (2.0 * kPi * ctx.inv_wavelength);
    const int nchunks = ctx.src_end > ctx.src_begin ?
            (ctx.src_end - ctx.src_begin + kChunk - 1) / kChunk : 0;

    __syncthreads();  // the previous item is done with shared memory
    if (tid < 2) sm.bound[tid] = 0;
    if (nchunks > 0)
    {
        if (warp == kSrcWarp)
            smear_issue_src<T, MATRIX, GAUSS, LMN>(sm, prm, ctx,
                    ctx.src_begin, 0);
        smear_issue<T, MATRIX>(sm, prm, jsrc, ctx, ctx.src_begin);
    }
    if (LMN && tid < 2 * kTile)
    {
        const int b = tid / kTile, stl = tid % kTile;
        const int st = (b ? ctx.q0 : ctx.p0) + stl;
        T* u = sm.st_uvw[b][stl];
        double* xy = sm.st_xy[b][stl];
        u[0] = u[1] = u[2] = 0;
        xy[0] = xy[1] = 0;
        if (st < N)
        {
            u[0] = su[st]; u[1] = sv[st]; u[2] = sw[st];
            if (TS)
            {
                const double x = prm.st_x[st], y = prm.st_y[st];
                xy[0] = x * ctx.c_ha - y * ctx.s_ha;
                xy[1] = x * ctx.s_ha + y * ctx.c_ha;
            }
        }
    }

    // The thread's two baselines (p, q): FP64 (pr, qc) and (pr + 1, qc),
    // FP32 (pr, qc) and (pr, qc + 1). Terms as the reference forms them
    // (oskar/correlate/define_correlate_utils.h:5-13).
    const double uv_scale = prm.uv_filter_in_metres ? ctx.inv_wavelength :
            1.0;
    const T uv_lo = (T) (prm.uv_min * uv_scale);
    const T uv_hi = (T) (prm.uv_max * uv_scale);
    bool exists[2], valid[2];
    float longest[2] = {0.0f, 0.0f};   // baselines in phase units: bw, ts
    T uu2[2], vv2[2], uuvv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
    {
        const int p = ctx.p0 + pr + (F64 ? i : 0);
        const int q = ctx.q0 + qc + (F64 ? 0 : i);
        exists[i] = p < N && q < p;
        T uu = 0, vv = 0;
        bool ok = exists[i];
        if (ok)
        {
            uu = (su[p] - su[q]) * (T) ctx.inv_wavelength;
            vv = (sv[p] - sv[q]) * (T) ctx.inv_wavelength;
            const T len = sqrt(uu * uu + vv * vv);
            ok = !(len < uv_lo || len > uv_hi);
            if (BW && !F64)
            {
                const double du = su[p] - su[q], dv = sv[p] - sv[q],
                        dw = sw[p] - sw[q];
                longest[0] = max_or_nan(longest[0], (float) (fabs(
                        prm.bw_scale) * sqrt(du * du + dv * dv + dw * dw)));
            }
            if (TS && !F64)
            {
                const double dx = prm.st_x[p] - prm.st_x[q],
                        dy = prm.st_y[p] - prm.st_y[q];
                longest[1] = max_or_nan(longest[1], (float) (fabs(
                        ctx.ts_scale) * sqrt(dx * dx + dy * dy)));
            }
        }
        valid[i] = ok;
        uu2[i] = uu * uu;
        vv2[i] = vv * vv;
        uuvv[i] = 2 * uu * vv;
    }
    const bool active = __any_sync(0xffffffffu, valid[0] || valid[1]);
    if ((BW || TS) && !F64)
    {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            longest[k] = __uint_as_float(__reduce_max_sync(0xffffffffu,
                    __float_as_uint(longest[k])));
    }

    double acc[2][2 * NC];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 2 * NC; ++k) acc[i][k] = 0.0;

    // Transform of chunk c into buffer c & 1, then the copies of chunk
    // c + 1 into the warp's raw buffer. Returns the chunk's reach.
    const auto advance = [&](int c)
    {
        float reach = 0.0f;
        const int s0 = ctx.src_begin + c * kChunk;
        cp_async_wait_all();
        __syncwarp();   // the warp's own copies, visible to its lanes
        smear_transform<T, MATRIX, GAUSS, BW, TS, CASA, FUSED>(sm, prm,
                jsrc != nullptr, ctx, wavenumber, s0 + (lane & 7) <
                ctx.src_end, c & 1, reach);
        __syncwarp();
        if (c + 1 < nchunks)
            smear_issue<T, MATRIX>(sm, prm, jsrc, ctx, s0 + kChunk);
        return reach;
    };
    // The per-source values of chunk c + 1, in buffer (c + 1) & 1, are read
    // by chunk c's iteration: copied one iteration earlier by one warp, whose
    // own transform of that iteration (after its products) waits for them.
    const auto issue_src = [&](int c)
    {
        if (warp == kSrcWarp && c < nchunks)
            smear_issue_src<T, MATRIX, GAUSS, LMN>(sm, prm, ctx,
                    ctx.src_begin + c * kChunk, c & 1);
    };
    cp_async_wait_all();
    __syncthreads();  // per-station terms and chunk 0's values are there
    float reach = 0.0f, reach_next = 0.0f;
    if ((BW || TS) && !F64)
    {
        if (lane < 2) atomicMax(&sm.bound[lane], __float_as_uint(
                lane ? longest[1] : longest[0]));
        __syncthreads();
    }
    if (nchunks > 0)
    {
        issue_src(1);
        reach = advance(0);
    }
    __syncthreads();
#pragma unroll 1
    for (int c = 0; c < nchunks; ++c)
    {
        const int ns = min(kChunk, ctx.src_end - ctx.src_begin - c * kChunk);
        issue_src(c + 2);
#pragma unroll 1
        for (int step = 0; step < 2; ++step)
        {
            if ((step == 0) == early)
            {
                if (c + 1 < nchunks) reach_next = advance(c + 1);
            }
            else if (active)
            {
                if constexpr (F64)
                    smear_products<MATRIX, GAUSS, BW, TS, CASA>(sm.f[c & 1],
                            ns, pr, qc, uu2, vv2, uuvv, acc);
                else if ((BW || TS) && sinc_small(reach, longest[0],
                        longest[1]))
                    smear_products<MATRIX, GAUSS, BW, TS, CASA, true>(
                            sm.f[c & 1], ns, pr, qc, uu2, vv2, uuvv, acc);
                else
                    smear_products<MATRIX, GAUSS, BW, TS, CASA, false>(
                            sm.f[c & 1], ns, pr, qc, uu2, vv2, uuvv, acc);
            }
        }
        reach = reach_next;
        __syncthreads();  // chunk c consumed, chunk c + 1's factors ready
    }

#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (exists[i])
            store_baseline<T, 2 * NC>(prm, ctx, slice,
                    ctx.p0 + pr + (F64 ? i : 0), ctx.q0 + qc + (F64 ? 0 : i),
                    valid[i], acc[i]);
    }  // items
}

}  // namespace
}  // namespace oskb
