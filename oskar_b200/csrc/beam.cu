// Aperture-array station beam (Jones E) for many stations in one launch, and
// the parallactic-angle rotation (Jones R).
//
// Replaces the chain the reference runs per station and per feed
// (oskar/telescope/station/src/oskar_station_beam.c:84-182 and
// oskar_evaluate_station_beam_aperture_array.c:150-240): element pattern
// (dipole, oskar_element_evaluate.c:76-157), element weights
// (define_evaluate_element_weights_dft.h:3-16), weighted DFT
// (define_dftw_m2m.h:24-107), horizon blanking
// (define_blank_below_horizon.h:15-29) and final normalisation
// (define_mem_normalise.h:31-51). The reference runs these as six kernels
// with five round trips through a per-station signal buffer; here a thread
// owns one to four directions of a station and the pieces stay in registers.
//
// With a single element type the weighted DFT of the element signals is
// pattern(dir) x AF(dir), AF = sum_e w_e exp(i k r_e . dir): the pattern is
// evaluated once per direction and the element loop carries only the array
// factor: per element-direction one phase, which includes the weight's, one
// table lookup (trig_table.cuh, both precisions) and one real-by-complex
// multiply-add. Element terms are staged in shared memory in chunks.
// The normalisation direction's beam (one per station) is recomputed by each
// CTA cooperatively beside the staging, so there is no second launch.
#include <algorithm>
#include <climits>

#include "beam_common.cuh"
#include "trig_table.cuh"

namespace oskb {
namespace {

constexpr int kThreads = 256;
constexpr int kChunk = 512;
constexpr int kCtasPerSm = 2;
// directions per thread: most items, and those of the last round (FP32 works
// on pairs, but on one where a call's directions do not fill the chip)
template <typename T>
constexpr int dirs_big(int num_types)
{
    // FP64 sums of several element types leave no registers for more
    return sizeof(T) == 4 || num_types == 1 ? 4 : num_types == 2 ? 2 : 1;
}
template <typename T> constexpr int kDirsSmall = sizeof(T) == 8 ? 1 : 2;

struct BeamFlags
{
    int normalise_element, normalise_array, normalise_final, swap_xy;
    int scalar;  // complex beam of the pattern amplitude (Stokes-I mode)
};

// Bit pattern of |v| as a float rounded up: orders as the values do, with
// NaN above everything.
__device__ __forceinline__ unsigned abs_bits(double v)
{
    return __float_as_uint(__double2float_ru(fabs(v)));
}
__device__ __forceinline__ unsigned abs_bits(float v)
{
    return __float_as_uint(fabsf(v));
}

template <typename T>
__device__ __forceinline__ T half_frobenius(const T p[4], T ar, T ai)
{
    // |p * af|_F^2 / 2 with p real and af complex.
    const T a2 = ar * ar + ai * ai;
    return (p[0] * p[0] + p[1] * p[1] + p[2] * p[2] + p[3] * p[3]) * a2 /
            (T) 2;
}

// Up to kMaxTypes element types per station (a dipole length each).
constexpr int kMaxTypes = 4;

template <typename T>
struct TypeParams
{
    T kL[kMaxTypes];      // dipole length x pi f / c
    T cos_kL[kMaxTypes], sin_kL[kMaxTypes];
    int kind[kMaxTypes];  // 0 dipole, 1 isotropic
    int taper[kMaxTypes]; // 0 none, 1 cos(theta)^p, 2 Gaussian in theta
    T taper_param[kMaxTypes];  // p, or 4 ln 2 / FWHM^2
};

// Real pattern {a, b, c, d} of element type t in direction (X, Y, Z): the
// dipole's, or the identity for an isotropic element
// (oskar_element_evaluate.c:82-87).
template <typename T>
__device__ __forceinline__ void type_pattern(const TypeParams<T>& tp, int t,
        T X, T Y, T Z, bool pole, T dphi1, T dphi2, int swap_xy, T p[4])
{
    if (tp.kind[t] == 1)
    {
        p[0] = p[3] = (T) 1;
        p[1] = p[2] = (T) 0;
        return;
    }
    element_pattern<T>(X, Y, Z, pole, dphi1, dphi2, tp.kL[t], tp.cos_kL[t],
            swap_xy, p);
}

// The same in one of the beam's directions; rot as element_pattern_rotated
// (FP64; the FP32 pattern keeps the reference's angles, whose rounding near
// the dipole's axis its single-precision results carry).
template <typename T>
__device__ __forceinline__ void direction_pattern(const TypeParams<T>& tp,
        int t, T X, T Y, T Z, T dphi1, T dphi2, const T* rot, int swap_xy,
        T p[4])
{
    if (tp.kind[t] == 1)
    {
        p[0] = p[3] = (T) 1;
        p[1] = p[2] = (T) 0;
        return;
    }
    if constexpr (sizeof(T) == 8)
        element_pattern_rotated<T>(X, Y, Z, dphi1, dphi2, rot, tp.kL[t],
                tp.cos_kL[t], tp.sin_kL[t], swap_xy, p);
    else
        element_pattern<T>(X, Y, Z, false, dphi1, dphi2, tp.kL[t],
                tp.cos_kL[t], swap_xy, p);
}

// Element taper of type t at polar angle theta = atan2(|(X, Y)|, Z),
// applied after the pole normalisation (oskar_element_evaluate.c:159-174;
// define_apply_element_taper_{cosine,gaussian}.h).
template <typename T>
__device__ __forceinline__ T type_taper(const TypeParams<T>& tp, int t, T X,
        T Y, T Z)
{
    if (tp.taper[t] == 0) return (T) 1;
    const T theta = atan2(sqrt(X * X + Y * Y), Z);
    if (tp.taper[t] == 1) return pow(cos(theta), tp.taper_param[t]);
    return exp(-(theta * theta) * tp.taper_param[t]);
}

// Terms of one element, staged once per (station, chunk): position, gain and
// the phase of its weight in table steps (reduced to one turn). FP32 terms
// are stored twice, as packed pairs {v, v} for two directions at a time.
template <typename T, bool IS3D> struct ElementTerms;
template <bool IS3D> struct ElementTerms<double, IS3D>
{
    double2 xy[kChunk], pg[kChunk];
    double z[IS3D ? kChunk : 1];
};
template <bool IS3D> struct ElementTerms<float, IS3D>
{
    float4 xy[kChunk], pg[kChunk];
    float2 z[IS3D ? kChunk : 1];
};

template <bool IS3D>
__device__ __forceinline__ void put_element(ElementTerms<double, IS3D>& el,
        int i, double x, double y, double z, double p, double g)
{
    el.xy[i] = make_double2(x, y);
    el.pg[i] = make_double2(p, g);
    if (IS3D) el.z[i] = z;
}
template <bool IS3D>
__device__ __forceinline__ void put_element(ElementTerms<float, IS3D>& el,
        int i, float x, float y, float z, float p, float g)
{
    el.xy[i] = make_float4(x, x, y, y);
    el.pg[i] = make_float4(p, p, g, g);
    if (IS3D) el.z[i] = make_float2(z, z);
}

// Phase factors e^{i u} of element i in the thread's ND directions, u in
// table steps.
template <bool IS3D, int ND>
__device__ __forceinline__ void element_factors(
        const ElementTerms<double, IS3D>& el, const double2* table, int i,
        const double (&kX)[ND], const double (&kY)[ND],
        const double (&kZ)[ND], double (&sn)[ND], double (&cs)[ND],
        double& gain)
{
    const double2 xy = el.xy[i], pg = el.pg[i];
    gain = pg.y;
#pragma unroll
    for (int j = 0; j < ND; ++j)
    {
        double u = fma(kY[j], xy.y, pg.x);
        if (IS3D) u = fma(kZ[j], el.z[i], u);
        u = fma(kX[j], xy.x, u);
        Trig<double>::sincos(table, u, &sn[j], &cs[j]);
    }
}
template <bool IS3D, int ND>
__device__ __forceinline__ void element_factors(
        const ElementTerms<float, IS3D>& el, const float2* table, int i,
        const float (&kX)[ND], const float (&kY)[ND], const float (&kZ)[ND],
        float (&sn)[ND], float (&cs)[ND], float& gain)
{
    const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(&el.xy[i]);
    const ulonglong2 pg = *reinterpret_cast<const ulonglong2*>(&el.pg[i]);
    float g2;
    unpack2(pg.y, gain, g2);
    if constexpr (ND == 1)
    {
        const float4 p = el.xy[i];
        float u = fmaf(kY[0], p.z, el.pg[i].x);
        if (IS3D) u = fmaf(kZ[0], el.z[i].x, u);
        u = fmaf(kX[0], p.x, u);
        Trig<float>::sincos(table, u, &sn[0], &cs[0]);
        return;
    }
#pragma unroll
    for (int j = 0; j + 1 < ND; j += 2)
    {
        f32x2 u = fma2(pack2(kY[j], kY[j + 1]), xy.y, pg.x);
        if (IS3D)
            u = fma2(pack2(kZ[j], kZ[j + 1]),
                    *reinterpret_cast<const f32x2*>(&el.z[i]), u);
        u = fma2(pack2(kX[j], kX[j + 1]), xy.x, u);
        Trig<float>::sincos2(table, u, &sn[j], &cs[j]);
    }
}

// The same through the library, for phases the table does not cover.
template <typename T, bool IS3D, int ND>
__device__ __forceinline__ void element_factors_exact(
        const ElementTerms<T, IS3D>& el, int i, const T (&kX)[ND],
        const T (&kY)[ND], const T (&kZ)[ND], T (&sn)[ND], T (&cs)[ND],
        T& gain)
{
    T x, y, p;
    if constexpr (sizeof(T) == 8) { x = el.xy[i].x; y = el.xy[i].y; }
    else { x = el.xy[i].x; y = el.xy[i].z; }
    if constexpr (sizeof(T) == 8) { p = el.pg[i].x; gain = el.pg[i].y; }
    else { p = el.pg[i].x; gain = el.pg[i].z; }
    T z = 0;
    if constexpr (IS3D && sizeof(T) == 8) z = el.z[i];
    if constexpr (IS3D && sizeof(T) == 4) z = el.z[i].x;
#pragma unroll
    for (int j = 0; j < ND; ++j)
    {
        T u = fma(kY[j], y, p);
        if (IS3D) u = fma(kZ[j], z, u);
        u = fma(kX[j], x, u);
        Trig<T>::exact(u, &sn[j], &cs[j]);
    }
}

// (ar, ai)[t] += gain e^{i u} for the element's type t only: register
// selects over a compile-time number of types, so the accumulators stay in
// registers.
template <typename T, int NT>
__device__ __forceinline__ void add_term(T* ar, T* ai, T gain, int type,
        T sn, T cs)
{
#pragma unroll
    for (int t = 0; t < NT; ++t)
    {
        const T g = (NT == 1 || type == t) ? gain : (T) 0;
        ar[t] = fma(g, cs, ar[t]);
        ai[t] = fma(g, sn, ai[t]);
    }
}

template <typename T, bool IS3D, int NT>
struct BeamSmem
{
    typename Trig<T>::Entry table[Trig<T>::kSize];
    ElementTerms<T, IS3D> el;
    int type[NT > 1 ? kChunk : 1];
    T red[2][NT][kThreads / 32];
    // Of the item's station, per element type: the elements' azimuths, their
    // cosines and sines (element_pattern_rotated's), the pole normalisation
    // and the pattern and taper in the normalisation direction.
    T dphi[NT][2], rot[NT][4], pole[NT], norm_p[NT][4], norm_taper[NT];
    unsigned bound[3];   // largest |x|, |y|, |z| of the chunk, float bits
};

// Arguments of a station-beam launch (the entry points').
template <typename T>
struct BeamArgs
{
    int num_elements;
    const T *el_x, *el_y, *el_z, *meas_x, *meas_y, *meas_z, *cable;
    const T* weight_factors;
    const int* element_type;
    const double *orientation_x, *orientation_y;
    TypeParams<T> tp;
    BeamFlags flags;
    double wavenumber;
    const double *beam_enu, *norm_enu;
    int num_dir;
    const T *dir_x, *dir_y, *dir_z;
    int directions_per_station;
    // rows: 0 all four; 1 the x feed's (xx, xy); 2 the y feed's (yx, yy).
    // With one feed per launch the final normalisation needs both feeds'
    // array factors at the normalisation direction: the launch writes its
    // own to norm_af[station][type] (complex) and leaves the scaling to
    // feeds_finalise_kernel.
    int rows;
    T* norm_af;
    T* beam;
};

// Half f of the terms of element type t of station st (BeamSmem), each by one
// thread, so that the patterns of all types at the pole and in the
// normalisation direction take the time of one.
template <typename T, bool IS3D, int NT>
__device__ __forceinline__ void station_terms(BeamSmem<T, IS3D, NT>& sm,
        const BeamArgs<T>& arg, int st, int t, int f, T nX, T nY, T nZ)
{
    const T dphi1 = (T) (kPi / 2 - (arg.orientation_x[st * NT + t] + kPi / 2));
    const T dphi2 = (T) (kPi / 2 - arg.orientation_y[st * NT + t]);
    sm.dphi[t][f] = f ? dphi2 : dphi1;
    if constexpr (sizeof(T) == 8)
        sincos(f ? dphi2 : dphi1, &sm.rot[t][2 * f + 1], &sm.rot[t][2 * f]);
    // f = 0: the pole; 1: the normalisation direction
    T p[4] = {};
    if (f ? arg.flags.normalise_final : arg.flags.normalise_element)
        type_pattern<T>(arg.tp, t, f ? nX : (T) 0, f ? nY : (T) 0, f ? nZ :
                (T) 1, f == 0, dphi1, dphi2, arg.flags.swap_xy, p);
    if (f)
    {
        for (int k = 0; k < 4; ++k) sm.norm_p[t][k] = p[k];
        sm.norm_taper[t] = type_taper<T>(arg.tp, t, nX, nY, nZ);
    }
    else
        // element normalisation: 1 / |pattern at the pole|
        sm.pole[t] = arg.flags.normalise_element ? (T) 1 /
                sqrt(half_frobenius<T>(p, 1, 0)) : (T) 1;
}

// Beam of station st in directions d_first + thread + j threads, j < ND.
// The weight of an element, f e^{-i k (r_m . b + cable)}, is folded into the
// element loop as a gain |f| and a phase in table steps, so an
// element-direction is one phase (2 or 3 multiply-adds), one table phase
// factor and one real-by-complex multiply-add: in FP64 17 operations
// (planar) against 21 with a complex weight and the 128-entry table.
template <typename T, bool IS3D, int NT, int ND>
__device__ __forceinline__ void station_beam_item(BeamSmem<T, IS3D, NT>& sm,
        const BeamArgs<T>& arg, int st, unsigned d_first)
{
    typedef typename vec2<T>::type T2;
    typedef Trig<T> Tr;
    const int num_elements = arg.num_elements;
    // (unsigned: a block may reach past the largest int)
    const unsigned num_dir = arg.num_dir;
    const BeamFlags& flags = arg.flags;
    const TypeParams<T>& tp = arg.tp;
    const double* beam_enu = arg.beam_enu;
    const int rows = arg.rows;
    const unsigned d0 = d_first + threadIdx.x;
    const int threads = blockDim.x;
    const size_t el0 = (size_t) st * num_elements;
    const size_t dir0 = arg.directions_per_station ? (size_t) st * num_dir : 0;
    const int per_dir = flags.scalar ? 1 : 4;
    T2* out = reinterpret_cast<T2*>(arg.beam) + per_dir * ((size_t) st * num_dir);

    const double bx = (T) beam_enu[3 * st], by = (T) beam_enu[3 * st + 1],
            bz = (T) beam_enu[3 * st + 2];
    if (beam_enu[3 * st + 2] < 0.0)  // pointing below the horizon
    {
#pragma unroll
        for (int j = 0; j < ND; ++j)
        {
            const unsigned d = d0 + j * threads;
            if (d < num_dir)
                for (int k = 0; k < per_dir; ++k)
                    out[(size_t) per_dir * d + k] = T2{(T) 0, (T) 0};
        }
        return;
    }
    T kX[ND], kY[ND], kZ[ND];
    const double k_steps = arg.wavenumber * Tr::kStepsPerRadian;
#pragma unroll
    for (int j = 0; j < ND; ++j)
    {
        const unsigned d = d0 + j * threads;
        const bool in = d < num_dir;
        // phase per metre in table steps, rounded once
        kX[j] = (T) (in ? k_steps * (double) arg.dir_x[dir0 + d] : 0.0);
        kY[j] = (T) (in ? k_steps * (double) arg.dir_y[dir0 + d] : 0.0);
        kZ[j] = (T) (IS3D && in ? k_steps * (double) arg.dir_z[dir0 + d] :
                0.0);
    }
    T nX = 0, nY = 0, nZ = 1;
    if (flags.normalise_final)
    {
        nX = (T) arg.norm_enu[3 * st];
        nY = (T) arg.norm_enu[3 * st + 1];
        nZ = (T) arg.norm_enu[3 * st + 2];
    }
    const T knX[1] = {(T) (k_steps * (double) nX)},
            knY[1] = {(T) (k_steps * (double) nY)},
            knZ[1] = {(T) (k_steps * (double) nZ)};

    // array factors per element type: the thread's directions (ar, ai) and
    // the normalisation direction (nr, ni)
    T ar[ND][NT], ai[ND][NT], nr[NT], ni[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t)
    {
        nr[t] = ni[t] = (T) 0;
#pragma unroll
        for (int j = 0; j < ND; ++j) ar[j][t] = ai[j][t] = (T) 0;
    }
    // The station's terms, by lanes of the last warp, which has the fewest
    // elements to stage: beside the other warps' staging where the element
    // loop is short, else beside their loops (128 stations x 12,000
    // directions FP64: 564 us against 576 before the staging; the choice at
    // run time, with both copies of the code, took 1 to 8 % longer).
    const int lane = threadIdx.x & 31;
    const int term = threadIdx.x >= threads - 32 && lane < 2 * NT ? lane : -1;
    for (int e0 = 0; e0 < num_elements; e0 += kChunk)
    {
        const int ne = min(kChunk, num_elements - e0);
        __syncthreads();  // table filled; the previous chunk is consumed
        if (threadIdx.x < 3) sm.bound[threadIdx.x] = 0;
        __syncthreads();
        if (ND == 1 && e0 == 0 && term >= 0)
            station_terms<T, IS3D, NT>(sm, arg, st, term >> 1, term & 1, nX,
                    nY, nZ);
        unsigned ex = 0, ey = 0, ez = 0;
        for (int t = threadIdx.x; t < ne; t += threads)
        {
            const size_t g = el0 + e0 + t;
            const T x = arg.el_x[g], y = arg.el_y[g], z = arg.el_z ? arg.el_z[g] : (T) 0;
            const double wx = arg.meas_x ? arg.meas_x[g] : x;
            const double wy = arg.meas_y ? arg.meas_y[g] : y;
            const double wz = arg.meas_z ? arg.meas_z[g] : z;
            // the weight's phase in table steps and its gain
            double p = -k_steps * (wx * bx + wy * by + wz * bz +
                    (arg.cable ? (double) arg.cable[g] : 0.0));
            T gain = (T) 1;
            if (arg.weight_factors)
            {
                // element errors x apodisation, applied to the DFT weight
                const T2 f = reinterpret_cast<const T2*>(arg.weight_factors)[g];
                gain = hypot(f.x, f.y);
                p += atan2((double) f.y, (double) f.x) * Tr::kStepsPerRadian;
            }
            p -= Tr::kEntries * rint(p * (1.0 / Tr::kEntries));
            put_element(sm.el, t, x, y, z, (T) p, gain);
            int type = 0;
            if constexpr (NT > 1)
            {
                type = arg.element_type ? arg.element_type[g] : 0;
                sm.type[t] = type;
            }
            ex = max(ex, abs_bits(x));
            ey = max(ey, abs_bits(y));
            if (IS3D) ez = max(ez, abs_bits(z));
            // The normalisation direction: elements split across threads.
            if (flags.normalise_final)
            {
                T u = fma(knY[0], y, (T) p);
                if (IS3D) u = fma(knZ[0], z, u);
                u = fma(knX[0], x, u);
                T s2, c2;
                Tr::checked(sm.table, u, &s2, &c2);
                add_term<T, NT>(nr, ni, gain, type, s2, c2);
            }
        }
        ex = __reduce_max_sync(0xffffffffu, ex);
        ey = __reduce_max_sync(0xffffffffu, ey);
        if (IS3D) ez = __reduce_max_sync(0xffffffffu, ez);
        if ((threadIdx.x & 31) == 0)
        {
            atomicMax(&sm.bound[0], ex);
            atomicMax(&sm.bound[1], ey);
            if (IS3D) atomicMax(&sm.bound[2], ez);
        }
        __syncthreads();
        if (ND > 1 && e0 == 0 && term >= 0)
            station_terms<T, IS3D, NT>(sm, arg, st, term >> 1, term & 1, nX,
                    nY, nZ);
        if (d0 < num_dir)
        {
            // The table covers every phase of the chunk when the largest
            // possible one is covered (false for NaN); otherwise the chunk
            // goes through the library.
            bool covered = true;
#pragma unroll
            for (int j = 0; j < ND; ++j)
            {
                T bound = fabs(kX[j]) * (T) __uint_as_float(sm.bound[0]) +
                        fabs(kY[j]) * (T) __uint_as_float(sm.bound[1]) +
                        (T) Tr::kEntries;
                if (IS3D)
                    bound += fabs(kZ[j]) * (T) __uint_as_float(sm.bound[2]);
                covered &= bound < (T) Tr::kLimit;
            }
            T sn[ND], cs[ND], gain;
            if (covered)
            {
#pragma unroll 4
                for (int i = 0; i < ne; ++i)
                {
                    element_factors<IS3D, ND>(sm.el, sm.table, i, kX, kY, kZ,
                            sn, cs, gain);
#pragma unroll
                    for (int j = 0; j < ND; ++j)
                        add_term<T, NT>(ar[j], ai[j], gain,
                                NT > 1 ? sm.type[i] : 0, sn[j], cs[j]);
                }
            }
            else
            {
#pragma unroll 1
                for (int i = 0; i < ne; ++i)
                {
                    element_factors_exact<T, IS3D, ND>(sm.el, i, kX, kY, kZ,
                            sn, cs, gain);
#pragma unroll
                    for (int j = 0; j < ND; ++j)
                        add_term<T, NT>(ar[j], ai[j], gain,
                                NT > 1 ? sm.type[i] : 0, sn[j], cs[j]);
                }
            }
        }
    }

    if (ND > 1 && !flags.normalise_final)
        __syncthreads();   // (else the reduction's) the terms are there
    const T array_scale = flags.normalise_array ?
            (T) (1.0 / num_elements) : (T) 1;

    // Final normalisation: amplitude of the beam in the normalisation
    // direction (block reduction of its array factors first).
    T final_scale = (T) 1;
    if (flags.normalise_final)
    {
#pragma unroll
        for (int t = 0; t < NT; ++t)
        {
            for (int o = 16; o > 0; o >>= 1)
            {
                nr[t] += __shfl_xor_sync(0xffffffffu, nr[t], o);
                ni[t] += __shfl_xor_sync(0xffffffffu, ni[t], o);
            }
            if ((threadIdx.x & 31) == 0)
            {
                sm.red[0][t][threadIdx.x >> 5] = nr[t];
                sm.red[1][t][threadIdx.x >> 5] = ni[t];
            }
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < NT; ++t)
        {
            nr[t] = ni[t] = 0;
            for (int w = 0; w < threads / 32; ++w)
            {
                nr[t] += sm.red[0][t][w];
                ni[t] += sm.red[1][t][w];
            }
            // A normalisation direction below the horizon is blanked, as in
            // the reference, which then divides by zero.
            if (nZ < (T) 0) nr[t] = ni[t] = (T) 0;
        }
        if (rows != 0)
        {
            if (d0 == 0)
            {
#pragma unroll
                for (int t = 0; t < NT; ++t)
                {
                    arg.norm_af[2 * ((size_t) st * NT + t)] = nr[t];
                    arg.norm_af[2 * ((size_t) st * NT + t) + 1] = ni[t];
                }
            }
        }
        else if (flags.scalar)
        {
            // |sum_t amplitude_t AF_t| (define_mem_normalise.h:13-29)
            T vr = 0, vi = 0;
#pragma unroll
            for (int t = 0; t < NT; ++t)
            {
                const T a = sqrt(half_frobenius<T>(sm.norm_p[t], 1, 0)) *
                        sm.norm_taper[t] * sm.pole[t] * array_scale;
                vr += a * nr[t];
                vi += a * ni[t];
            }
            final_scale = (T) 1 / sqrt(vr * vr + vi * vi);
        }
        else if constexpr (NT == 1)
        {
            T pn[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                pn[k] = sm.norm_p[0][k] * (sm.pole[0] * sm.norm_taper[0] *
                        array_scale);
            final_scale = (T) 1 / sqrt(half_frobenius<T>(pn, nr[0], ni[0]));
        }
        else
        {
            // |sum_t pattern_t AF_t|_F^2 / 2 over the four polarisations
            T amp = 0;
            for (int k = 0; k < 4; ++k)
            {
                T vr = 0, vi = 0;
#pragma unroll
                for (int t = 0; t < NT; ++t)
                {
                    const T pk = sm.norm_p[t][k] * sm.norm_taper[t] *
                            sm.pole[t] * array_scale;
                    vr += pk * nr[t];
                    vi += pk * ni[t];
                }
                amp += vr * vr + vi * vi;
            }
            final_scale = (T) 1 / sqrt(amp / (T) 2);
        }
    }
#pragma unroll 1
    for (int j = 0; j < ND; ++j)
    {
        const unsigned d = d0 + j * threads;
        if (d >= num_dir) break;
        T2* o = out + (size_t) per_dir * d;
        // (read again: kept, they would spill from the element loop)
        const T x = arg.dir_x[dir0 + d], y = arg.dir_y[dir0 + d],
                z = arg.dir_z[dir0 + d];
        T fr[NT], fi[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t)
        {
            fr[t] = ar[0][t];
            fi[t] = ai[0][t];
        }
#pragma unroll
        for (int k = 1; k < ND; ++k)
            if (j == k)
#pragma unroll
                for (int t = 0; t < NT; ++t)
                {
                    fr[t] = ar[k][t];
                    fi[t] = ai[k][t];
                }
        const bool blank = z < (T) 0;
        // The reference's order: pattern (normalised), times the weighted
        // element sum, times the DFT norm, then the final scale. One copy of
        // the pattern's code for all types: a call of few directions waits
        // for its instructions, about 3,000 cycles per copy (FP32, 4
        // stations x 18 elements x 3,614 directions, four types, with the
        // same for the patterns of station_terms: 26.7 -> 10.8 us).
        T2 v[4] = {};
#pragma unroll 1
        for (int t = 0; t < NT; ++t)
        {
            T wr = fr[0], wi = fi[0];
#pragma unroll
            for (int k = 1; k < NT; ++k)
                if (t == k)
                {
                    wr = fr[k];
                    wi = fi[k];
                }
            T pt[4];
            direction_pattern<T>(tp, t, x, y, z, sm.dphi[t][0],
                    sm.dphi[t][1], sm.rot[t], flags.swap_xy, pt);
            const T taper = type_taper<T>(tp, t, x, y, z);
            if (flags.scalar)
            {
                // pattern amplitude sqrt(sum p_k^2 / 2)
                // (define_evaluate_dipole_pattern.h:51-75) times the array
                // factor
                const T a = sqrt(half_frobenius<T>(pt, 1, 0)) * taper *
                        sm.pole[t];
                v[0].x += a * wr * array_scale;
                v[0].y += a * wi * array_scale;
                continue;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                const T pk = pt[k] * taper * sm.pole[t];
                v[k].x += pk * wr * array_scale;
                v[k].y += pk * wi * array_scale;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            if (blank) v[k] = T2{(T) 0, (T) 0};
            v[k].x *= final_scale;
            v[k].y *= final_scale;
            if (flags.scalar ? k == 0 : rows == 0 || (rows == 1) == (k < 2))
                o[k] = v[k];
        }
    }
}

// One CTA takes items in turn, with its table filled once: first `full`
// (station, block of threads x BIG directions) items in whole rounds of the
// grid, then the rest of the directions in parts of threads x SMALL, so that
// the last round is short: at 128 stations x 12,000 directions a grid of 296
// has 5.2 rounds of 1,024 directions, and a whole sixth round would idle most
// of the chip. More directions per thread share the staged element terms
// (FP64: 629 us with four against 668 us with one on that shape, before the
// split). The parts are those of the stations from first_station on (the
// first one's from first_part), the first part of every station before the
// second and so on: none is empty, and the last ones, which are short, come
// last and spread over the CTAs. (Numbered so that a station's short or empty
// parts fell to every second CTA, 393 stations x 513 elements x 1,025
// directions FP64 took 664 us, now 391.)
template <typename T, bool IS3D, int NT, int BIG, int SMALL>
__global__ void __launch_bounds__(kThreads, BIG == 1 && sizeof(T) == 4 ? 1 :
        kCtasPerSm)
station_beam_kernel(const __grid_constant__ BeamArgs<T> arg, unsigned blocks,
        unsigned full, unsigned first_station, unsigned first_part,
        unsigned stations, unsigned total)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BeamSmem<T, IS3D, NT>& sm =
            *reinterpret_cast<BeamSmem<T, IS3D, NT>*>(smem_raw);
    Trig<T>::fill(sm.table);
    for (unsigned item = blockIdx.x; item < full; item += gridDim.x)
        station_beam_item<T, IS3D, NT, BIG>(sm, arg, item / blocks,
                item % blocks * (blockDim.x * BIG));
    for (unsigned n = blockIdx.x; n < total; n += gridDim.x)
    {
        const unsigned st = first_station + n % stations, p = n / stations;
        if (n % stations != 0 || p >= first_part)
            station_beam_item<T, IS3D, NT, SMALL>(sm, arg, st,
                    p * (blockDim.x * SMALL));
    }
}

// Final normalisation of a station beam evaluated one feed per launch:
// the beam in the normalisation direction takes its (xx, xy) row from the
// x feed's array factors and its (yx, yy) row from the y feed's
// (norm_af[feed][station][type], complex); every direction of the station
// is divided by that matrix's amplitude (define_mem_normalise.h:31-51).
template <typename T, int NT>
__global__ void __launch_bounds__(256)
feeds_finalise_kernel(int num_stations, int num_elements,
        const double* __restrict__ orientation_x,
        const double* __restrict__ orientation_y, TypeParams<T> tp,
        BeamFlags flags, const double* __restrict__ beam_enu,
        const double* __restrict__ norm_enu, int num_dir,
        const T* __restrict__ norm_af, T* __restrict__ beam)
{
    const int st = blockIdx.y;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    // a pointing below the horizon left a zero beam and no array factors
    if (d >= num_dir || beam_enu[3 * st + 2] < 0.0) return;
    const T nX = (T) norm_enu[3 * st], nY = (T) norm_enu[3 * st + 1],
            nZ = (T) norm_enu[3 * st + 2];
    const T array_scale = flags.normalise_array ?
            (T) (1.0 / num_elements) : (T) 1;
    T amp = 0;
    T pn[NT][4], pole[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t)
    {
        const T dphi1 = (T) (kPi / 2 - (orientation_x[st * NT + t] + kPi / 2));
        const T dphi2 = (T) (kPi / 2 - orientation_y[st * NT + t]);
        pole[t] = (T) 1;
        if (flags.normalise_element)
        {
            T pp[4];
            type_pattern<T>(tp, t, 0, 0, 1, true, dphi1, dphi2,
                    flags.swap_xy, pp);
            pole[t] = (T) 1 / sqrt(half_frobenius<T>(pp, 1, 0));
        }
        type_pattern<T>(tp, t, nX, nY, nZ, false, dphi1, dphi2,
                flags.swap_xy, pn[t]);
        const T taper = type_taper<T>(tp, t, nX, nY, nZ);
        for (int k = 0; k < 4; ++k) pn[t][k] *= taper;
    }
    for (int k = 0; k < 4; ++k)
    {
        const T* af = norm_af + 2 * (size_t) NT *
                ((size_t) (k < 2 ? 0 : 1) * num_stations + st);
        T vr = 0, vi = 0;
#pragma unroll
        for (int t = 0; t < NT; ++t)
        {
            const T pk = pn[t][k] * pole[t] * array_scale;
            vr += pk * af[2 * t];
            vi += pk * af[2 * t + 1];
        }
        amp += vr * vr + vi * vi;
    }
    const T scale = (T) 1 / sqrt(amp / (T) 2);
    T* b = beam + 8 * ((size_t) st * num_dir + d);
#pragma unroll
    for (int i = 0; i < 8; ++i) b[i] *= scale;
}

template <typename T>
__global__ void __launch_bounds__(256)
jones_r_kernel(int num_sources, const T* __restrict__ ra,
        const T* __restrict__ dec, const double* __restrict__ lat_rad,
        const double* __restrict__ lst_rad, T* __restrict__ jones)
{
    typedef typename vec2<T>::type T2;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int st = blockIdx.y;
    if (s >= num_sources) return;
    // (define_evaluate_jones_R.h:3-29; per-station latitude and LST as the
    // driver oskar_evaluate_jones_R.c:42-49 derives them in double.)
    const T cos_lat = (T) cos(lat_rad[st]), sin_lat = (T) sin(lat_rad[st]);
    const T lst = (T) lst_rad[st];
    T sh, ch, sd, cd, sq, cq;
    sincos(lst - ra[s], &sh, &ch);
    sincos(dec[s], &sd, &cd);
    const T q = atan2(cos_lat * sh, sin_lat * cd - cos_lat * sd * ch);
    sincos(q, &sq, &cq);
    T2* o = reinterpret_cast<T2*>(jones) + 4 * ((size_t) st * num_sources + s);
    o[0] = T2{cq, (T) 0};
    o[1] = T2{-sq, (T) 0};
    o[2] = T2{sq, (T) 0};
    o[3] = T2{cq, (T) 0};
}

}  // namespace
}  // namespace oskb

namespace oskb {
namespace {

// Per-type parameters from host arrays (NULL kinds: dipoles; NULL tapers:
// none). Returns an OSKAR status.
template <typename T>
int make_type_params(int num_types, const double* dipole_length_m,
        const int* element_kind, const int* taper_kind,
        const double* taper_param, double frequency_hz, TypeParams<T>* tp)
{
    if (num_types < 1 || !dipole_length_m) return OSKB_ERR_INVALID_ARGUMENT;
    if (num_types > kMaxTypes) return OSKB_ERR_OUT_OF_RANGE;
    const double c0 = 299792458.0;
    for (int t = 0; t < kMaxTypes; ++t)
    {
        const bool on = t < num_types;
        const double kL = on ?
                dipole_length_m[t] * (kPi * frequency_hz / c0) : 0.0;
        tp->kL[t] = (T) kL;
        tp->cos_kL[t] = (T) cos(kL);
        tp->sin_kL[t] = (T) sin(kL);
        tp->kind[t] = on && element_kind ? element_kind[t] : 0;
        tp->taper[t] = on && taper_kind ? taper_kind[t] : 0;
        if (tp->kind[t] < 0 || tp->kind[t] > 1 || tp->taper[t] < 0 ||
                tp->taper[t] > 2 || (tp->taper[t] && !taper_param))
            return OSKB_ERR_INVALID_ARGUMENT;
        double q = 0.0;
        if (tp->taper[t] == 1) q = taper_param[t];
        if (tp->taper[t] == 2)
        {
            const double fwhm = taper_param[t];
            if (!(fwhm > 0.0)) return OSKB_ERR_INVALID_ARGUMENT;
            q = 4.0 * log(2.0) / (fwhm * fwhm);
        }
        tp->taper_param[t] = (T) q;
    }
    return 0;
}

// Work items of a launch (station_beam_kernel) on `threads` threads per CTA:
// `full` items of big directions per thread in whole rounds, the rest in
// parts of small (few: of one, by the kernel that has no other).
struct BeamSplit
{
    int threads, small, few, grid;
    int blocks, full, first_station, first_part, stations;
    long long total;   // parts
};

// CTAs that an SM holds: two tables of 64 KB or four of 32 fit.
template <typename T>
int beam_ctas_per_sm(int threads)
{
    return std::min(sizeof(T) == 8 ? kCtasPerSm : 2 * kCtasPerSm,
            kCtasPerSm * kThreads / threads);
}

// The items of a call. Where its directions do not fill whole rounds of big
// items, the threads per CTA and the directions per thread of the parts are
// those of the least estimated time, in units of one element's work on an
// SM's 256 directions: the rounds of the busiest SM's CTAs (latency of the
// element loop, of the patterns and of staging the elements), the work of
// its directions and the table's filling. Constants fitted to the times of
// 694 shapes of 1 to 512 stations x 16 to 1,024 elements x 200 to 30,000
// directions x 1 to 4 element types, both precisions, with every choice
// timed: the choice is 0.5 % above the best on average. Against one direction
// per thread on 128 threads and the 128-entry table (FP64) or sincosf (FP32)
// calls of all sizes take 0.78 (FP64) and 0.63 (FP32) of the time; of 900
// shapes 22 take 1 to 9 % more, and 18 stations x 17 elements x 9,053
// directions FP32, whose time is the patterns', 26 %.
template <typename T>
BeamSplit beam_split(int num_stations, int num_elements, int num_directions,
        int num_types)
{
    const int sms = device_sm_count(), big = dirs_big<T>(num_types);
    const auto ceil_div = [](long long a, long long b)
    {
        return (a + b - 1) / b;
    };
    BeamSplit s = {kThreads, kDirsSmall<T>, 0};
    // whole rounds of big items, unless their blocks would be a quarter
    // empty or more
    const int slots = kCtasPerSm * sms;
    s.blocks = (int) ceil_div(num_directions, kThreads * big);
    const long long items = (long long) s.blocks * num_stations;
    if (4LL * num_directions >= 3LL * s.blocks * kThreads * big)
        s.full = (int) std::min<long long>(items / slots * slots, INT_MAX);
    if (s.full == 0)
    {
        double best = 0;
        for (int small = kDirsSmall<T>; small >= 1; small /= 2)
            for (int threads = kThreads; threads >= 64; threads /= 2)
            {
                const double n = num_elements, total = (double) (ceil_div(
                        num_directions, threads * small) * num_stations);
                const int per_sm = beam_ctas_per_sm<T>(threads);
                const double ctas = ceil(total / sms), rounds = ceil(ctas /
                        per_sm), all = ctas * threads;
                const double staging = (double) ceil_div(std::min(
                        num_elements, kChunk), threads) * std::max(1.0, n /
                        kChunk);
                double cost = rounds * 40.0 * staging;
                if constexpr (sizeof(T) == 8)
                {
                    // warps without directions take less; a last warp with
                    // elements stages them after the station's terms
                    const double live = std::max<double>(threads, 32.0 *
                            ceil_div(num_directions, 32) * num_stations / sms);
                    cost += (0.68 * all + 0.3 * live) / 256.0 * n + 0.17 * n *
                            std::max(1.0, total / (per_sm * sms)) + 4.0 *
                            256 / threads;
                    if (num_elements > threads - 32) cost += 12.0 * rounds;
                }
                else
                    // (one direction at a time takes 1.3 times its share of
                    // a pair)
                    cost += rounds * small * (0.4 * n + 12.0 * num_types) +
                            all * (small == 1 ? 1.3 : small) / 256.0 * n +
                            10.0 * 256 / threads;
                if (best == 0 || cost < best)
                {
                    best = cost;
                    s.threads = threads;
                    s.small = small;
                    s.few = small == 1;
                }
            }
    }
    s.first_station = s.full / s.blocks;
    s.first_part = s.full % s.blocks * (big / s.small);
    s.stations = num_stations - s.first_station;
    s.total = ceil_div(num_directions, s.threads * s.small) * s.stations;
    s.grid = s.full ? slots : (int) std::min<long long>(s.total,
            beam_ctas_per_sm<T>(s.threads) * sms);
    return s;
}

template <typename T, bool IS3D, int NT>
void launch_beam(const BeamArgs<T>& arg, const BeamSplit& s,
        cudaStream_t stream)
{
    auto k = station_beam_kernel<T, IS3D, NT, dirs_big<T>(NT), kDirsSmall<T>>;
    if (s.few)
        k = station_beam_kernel<T, IS3D, NT, 1, 1>;
    const int smem = (int) sizeof(BeamSmem<T, IS3D, NT>);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
            smem);
    k<<<s.grid, s.threads, smem, stream>>>(arg, s.blocks, s.full,
            s.first_station, s.first_part, s.stations, (unsigned) s.total);
}

template <typename T>
int station_beam_aa(int num_stations, int num_elements, const T* el_x,
        const T* el_y, const T* el_z, const T* meas_x, const T* meas_y,
        const T* meas_z, const T* cable, const T* weight_factors,
        int num_element_types, const int* element_type,
        const double* orientation_x,
        const double* orientation_y, const double* dipole_length_m,
        const int* element_kind, const int* taper_kind,
        const double* taper_param,
        int normalise_element, int normalise_array, int normalise_final,
        int swap_xy, int is_3d, double frequency_hz, const double* beam_enu,
        const double* norm_enu, int num_directions, const T* x, const T* y,
        const T* z, int directions_per_station, T* beam, void* stream,
        int rows = 0, T* norm_af = nullptr, int scalar = 0)
{
    if (num_stations < 0 || num_elements < 0 || num_directions < 0)
        return OSKB_ERR_INVALID_ARGUMENT;
    if (num_stations == 0 || num_directions == 0) return 0;
    if (num_elements == 0 || !el_x || !el_y || (is_3d && !el_z) ||
            !orientation_x || !orientation_y || !beam_enu ||
            (normalise_final && !norm_enu) || !x || !y || !z || !beam)
        return OSKB_ERR_INVALID_ARGUMENT;
    if (num_stations > 65535) return OSKB_ERR_INVALID_ARGUMENT;
    TypeParams<T> tp;
    if (int err = make_type_params<T>(num_element_types, dipole_length_m,
            element_kind, taper_kind, taper_param, frequency_hz, &tp))
        return err;
    const double c0 = 299792458.0;
    const double wavenumber = 2.0 * kPi * frequency_hz / c0;
    BeamFlags flags{normalise_element, normalise_array, normalise_final,
            swap_xy, scalar};
    const BeamSplit split = beam_split<T>(num_stations, num_elements,
            num_directions, num_element_types);
    if (split.total > INT_MAX) return OSKB_ERR_INVALID_ARGUMENT;
    const BeamArgs<T> arg = {num_elements, el_x, el_y, el_z, meas_x, meas_y,
            meas_z, cable, weight_factors, element_type, orientation_x,
            orientation_y, tp, flags, wavenumber, beam_enu, norm_enu,
            num_directions, x, y, z, directions_per_station, rows, norm_af,
            beam};
    cudaStream_t s = as_stream(stream);
#define OSKB_BEAM(D, NT)                                                     \
    launch_beam<T, D, NT>(arg, split, s);
#define OSKB_BEAM_NT(D)                                                      \
    switch (num_element_types)                                               \
    {                                                                        \
    case 1: OSKB_BEAM(D, 1) break;                                           \
    case 2: OSKB_BEAM(D, 2) break;                                           \
    case 3: OSKB_BEAM(D, 3) break;                                           \
    default: OSKB_BEAM(D, 4) break;                                          \
    }
    if (is_3d) { OSKB_BEAM_NT(true) } else { OSKB_BEAM_NT(false) }
#undef OSKB_BEAM_NT
#undef OSKB_BEAM
    return check_launch("station_beam_aa");
}

// Stations whose two feeds have their own element data (the reference's
// num_feeds = 2 when a station is not common_pol_beams,
// oskar_evaluate_station_beam_aperture_array.c:208-223): element arrays
// are [feed][station][element]; one launch per feed writes that feed's
// rows, then the final normalisation combines both feeds.
template <typename T>
int station_beam_aa_feeds(int num_feeds, int num_stations, int num_elements,
        const T* el_x, const T* el_y, const T* el_z, const T* meas_x,
        const T* meas_y, const T* meas_z, const T* cable,
        const T* weight_factors, int num_element_types,
        const int* element_type, const double* orientation_x,
        const double* orientation_y, const double* dipole_length_m,
        const int* element_kind, const int* taper_kind,
        const double* taper_param,
        int normalise_element, int normalise_array, int normalise_final,
        int swap_xy, int is_3d, double frequency_hz, const double* beam_enu,
        const double* norm_enu, int num_directions, const T* x, const T* y,
        const T* z, int directions_per_station, T* beam, void* stream)
{
    if (num_feeds == 1)
        return station_beam_aa<T>(num_stations, num_elements, el_x, el_y,
                el_z, meas_x, meas_y, meas_z, cable, weight_factors,
                num_element_types, element_type, orientation_x,
                orientation_y, dipole_length_m, element_kind, taper_kind,
                taper_param, normalise_element,
                normalise_array, normalise_final, swap_xy, is_3d,
                frequency_hz, beam_enu, norm_enu, num_directions, x, y, z,
                directions_per_station, beam, stream);
    if (num_feeds != 2) return OSKB_ERR_INVALID_ARGUMENT;
    if (num_stations <= 0 || num_directions <= 0)
        return num_stations < 0 || num_directions < 0 ?
                OSKB_ERR_INVALID_ARGUMENT : 0;
    TypeParams<T> tp;
    if (int err = make_type_params<T>(num_element_types, dipole_length_m,
            element_kind, taper_kind, taper_param, frequency_hz, &tp))
        return err;
    cudaStream_t s = as_stream(stream);
    T* norm_af = nullptr;
    const size_t af_count = (size_t) 2 * num_stations * num_element_types * 2;
    if (normalise_final)
    {
        if (scratch_alloc((void**) &norm_af, af_count * sizeof(T), s) !=
                cudaSuccess)
        {
            cudaGetLastError();
            return OSKB_ERR_MEMORY_ALLOC_FAILURE;
        }
    }
    const size_t n = (size_t) num_stations * num_elements;
    int err = 0;
    for (int f = 0; f < 2 && !err; ++f)
    {
        const size_t o = f * n;
        err = station_beam_aa<T>(num_stations, num_elements, el_x + o,
                el_y + o, el_z ? el_z + o : nullptr,
                meas_x ? meas_x + o : nullptr, meas_y ? meas_y + o : nullptr,
                meas_z ? meas_z + o : nullptr, cable ? cable + o : nullptr,
                weight_factors ? weight_factors + 2 * o : nullptr,
                num_element_types, element_type, orientation_x,
                orientation_y, dipole_length_m, element_kind, taper_kind,
                taper_param, normalise_element,
                normalise_array, normalise_final, swap_xy, is_3d,
                frequency_hz, beam_enu, norm_enu, num_directions, x, y, z,
                directions_per_station, beam, stream, 1 + f,
                norm_af ? norm_af + f * (af_count / 2) : nullptr);
    }
    if (!err && normalise_final)
    {
        BeamFlags flags{normalise_element, normalise_array, normalise_final,
                swap_xy, 0};
        dim3 grid((num_directions + 255) / 256, num_stations);
#define OSKB_FIN(NT) feeds_finalise_kernel<T, NT><<<grid, 256, 0, s>>>(       \
        num_stations, num_elements, orientation_x, orientation_y, tp, flags, \
        beam_enu, norm_enu, num_directions, norm_af, beam)
        switch (num_element_types)
        {
        case 1: OSKB_FIN(1); break;
        case 2: OSKB_FIN(2); break;
        case 3: OSKB_FIN(3); break;
        default: OSKB_FIN(4); break;
        }
#undef OSKB_FIN
        err = check_launch("station_beam_feeds_finalise");
    }
    if (norm_af) scratch_free(norm_af, s);
    return err;
}

template <typename T>
int jones_r(int num_sources, const T* ra, const T* dec, int num_stations,
        const double* lat_rad, const double* lst_rad, T* jones, void* stream)
{
    if (num_sources < 0 || num_stations < 0 || num_stations > 65535)
        return OSKB_ERR_INVALID_ARGUMENT;
    if (num_sources == 0 || num_stations == 0) return 0;
    if (!ra || !dec || !lat_rad || !lst_rad || !jones)
        return OSKB_ERR_INVALID_ARGUMENT;
    dim3 grid((num_sources + 255) / 256, num_stations);
    jones_r_kernel<T><<<grid, 256, 0, as_stream(stream)>>>(num_sources, ra,
            dec, lat_rad, lst_rad, jones);
    return check_launch("evaluate_jones_R");
}

}  // namespace
}  // namespace oskb

extern "C" {

#define OSKB_BEAM_ENTRY(T, S)                                                \
int oskb_station_beam_aa_##S(int num_stations, int num_elements,             \
        const T* el_x, const T* el_y, const T* el_z, const T* meas_x,        \
        const T* meas_y, const T* meas_z, const T* cable_length_error,       \
        const double* orientation_x_rad, const double* orientation_y_rad,    \
        double dipole_length_m, int normalise_element, int normalise_array,  \
        int normalise_final, int swap_xy, int is_3d, double frequency_hz,    \
        const double* beam_enu, const double* norm_enu, int num_directions,  \
        const T* x, const T* y, const T* z, int directions_per_station,      \
        T* beam, void* stream)                                               \
{                                                                            \
    return oskb::station_beam_aa<T>(num_stations, num_elements, el_x, el_y,  \
            el_z, meas_x, meas_y, meas_z, cable_length_error, nullptr, 1,    \
            nullptr, orientation_x_rad, orientation_y_rad, &dipole_length_m, \
            nullptr, nullptr, nullptr,                                       \
            normalise_element, normalise_array, normalise_final, swap_xy,    \
            is_3d, frequency_hz, beam_enu, norm_enu, num_directions, x, y,   \
            z, directions_per_station, beam, stream);                        \
}                                                                            \
int oskb_station_beam_aa_weighted_##S(int num_stations, int num_elements,    \
        const T* el_x, const T* el_y, const T* el_z, const T* meas_x,        \
        const T* meas_y, const T* meas_z, const T* cable_length_error,       \
        const T* element_weight_factors,                                     \
        const double* orientation_x_rad, const double* orientation_y_rad,    \
        double dipole_length_m, int normalise_element, int normalise_array,  \
        int normalise_final, int swap_xy, int is_3d, double frequency_hz,    \
        const double* beam_enu, const double* norm_enu, int num_directions,  \
        const T* x, const T* y, const T* z, int directions_per_station,      \
        T* beam, void* stream)                                               \
{                                                                            \
    return oskb::station_beam_aa<T>(num_stations, num_elements, el_x, el_y,  \
            el_z, meas_x, meas_y, meas_z, cable_length_error,                \
            element_weight_factors, 1, nullptr, orientation_x_rad,           \
            orientation_y_rad, &dipole_length_m, nullptr, nullptr, nullptr,  \
            normalise_element,                                               \
            normalise_array, normalise_final, swap_xy, is_3d, frequency_hz,  \
            beam_enu, norm_enu, num_directions, x, y, z,                     \
            directions_per_station, beam, stream);                           \
}                                                                            \
int oskb_station_beam_aa_types_##S(int num_stations, int num_elements,       \
        const T* el_x, const T* el_y, const T* el_z, const T* meas_x,        \
        const T* meas_y, const T* meas_z, const T* cable_length_error,       \
        const T* element_weight_factors, int num_element_types,              \
        const int* element_type, const double* dipole_length_m,              \
        const int* element_kind, const int* taper_kind,                      \
        const double* taper_param,                                           \
        const double* orientation_x_rad, const double* orientation_y_rad,    \
        int normalise_element, int normalise_array, int normalise_final,     \
        int swap_xy, int is_3d, double frequency_hz,                         \
        const double* beam_enu, const double* norm_enu, int num_directions,  \
        const T* x, const T* y, const T* z, int directions_per_station,      \
        T* beam, void* stream)                                               \
{                                                                            \
    return oskb::station_beam_aa<T>(num_stations, num_elements, el_x, el_y,  \
            el_z, meas_x, meas_y, meas_z, cable_length_error,                \
            element_weight_factors, num_element_types, element_type,         \
            orientation_x_rad, orientation_y_rad, dipole_length_m,           \
            element_kind, taper_kind, taper_param,                           \
            normalise_element, normalise_array, normalise_final, swap_xy,    \
            is_3d, frequency_hz, beam_enu, norm_enu, num_directions, x, y,   \
            z, directions_per_station, beam, stream);                        \
}                                                                            \
int oskb_station_beam_aa_scalar_##S(int num_stations, int num_elements,      \
        const T* el_x, const T* el_y, const T* el_z, const T* meas_x,        \
        const T* meas_y, const T* meas_z, const T* cable_length_error,       \
        const T* element_weight_factors, int num_element_types,              \
        const int* element_type, const double* dipole_length_m,              \
        const int* element_kind, const int* taper_kind,                      \
        const double* taper_param,                                           \
        const double* orientation_x_rad, const double* orientation_y_rad,    \
        int normalise_element, int normalise_array, int normalise_final,     \
        int swap_xy, int is_3d, double frequency_hz,                         \
        const double* beam_enu, const double* norm_enu, int num_directions,  \
        const T* x, const T* y, const T* z, int directions_per_station,      \
        T* beam, void* stream)                                               \
{                                                                            \
    return oskb::station_beam_aa<T>(num_stations, num_elements, el_x, el_y,  \
            el_z, meas_x, meas_y, meas_z, cable_length_error,                \
            element_weight_factors, num_element_types, element_type,         \
            orientation_x_rad, orientation_y_rad, dipole_length_m,           \
            element_kind, taper_kind, taper_param,                           \
            normalise_element, normalise_array, normalise_final, swap_xy,    \
            is_3d, frequency_hz, beam_enu, norm_enu, num_directions, x, y,   \
            z, directions_per_station, beam, stream, 0, nullptr, 1);         \
}                                                                            \
int oskb_station_beam_aa_feeds_##S(int num_feeds, int num_stations,        \
        int num_elements, const T* el_x, const T* el_y, const T* el_z,       \
        const T* meas_x, const T* meas_y, const T* meas_z,                   \
        const T* cable_length_error, const T* element_weight_factors,        \
        int num_element_types, const int* element_type,                     \
        const double* dipole_length_m, const int* element_kind,              \
        const int* taper_kind, const double* taper_param,                    \
        const double* orientation_x_rad,                                     \
        const double* orientation_y_rad, int normalise_element,              \
        int normalise_array, int normalise_final, int swap_xy, int is_3d,    \
        double frequency_hz, const double* beam_enu, const double* norm_enu, \
        int num_directions, const T* x, const T* y, const T* z,              \
        int directions_per_station, T* beam, void* stream)                   \
{                                                                            \
    return oskb::station_beam_aa_feeds<T>(num_feeds, num_stations,           \
            num_elements, el_x, el_y, el_z, meas_x, meas_y, meas_z,          \
            cable_length_error, element_weight_factors, num_element_types,   \
            element_type, orientation_x_rad, orientation_y_rad,              \
            dipole_length_m, element_kind, taper_kind, taper_param,          \
            normalise_element, normalise_array,                              \
            normalise_final, swap_xy, is_3d, frequency_hz, beam_enu,         \
            norm_enu, num_directions, x, y, z, directions_per_station, beam, \
            stream);                                                         \
}                                                                            \
int oskb_evaluate_jones_R_##S(int num_sources, const T* ra_rad,              \
        const T* dec_rad, int num_stations, const double* lat_rad,           \
        const double* lst_rad, T* jones, void* stream)                       \
{                                                                            \
    return oskb::jones_r<T>(num_sources, ra_rad, dec_rad, num_stations,      \
            lat_rad, lst_rad, jones, stream);                                \
}

OSKB_BEAM_ENTRY(double, d)
OSKB_BEAM_ENTRY(float, f)
#undef OSKB_BEAM_ENTRY

}  // extern "C"

// ---------------------------------------------------------------------------
// Hierarchical aperture-array stations of any depth: level 0 holds the leaf
// layouts (dipole arrays), each node type of level l > 0 is an array of
// children of level l - 1, and the top level is the station itself. The
// reference recurses (oskar_evaluate_station_beam_aperture_array.c:242-287):
// it evaluates every child station's beam, copying the first child's beam to
// all children when they are identical, then forms the parent's weighted DFT
// over its children with the child beams as the data. Here the recursion runs
// bottom-up over node TYPES instead of over the tree: one fused station-beam
// launch evaluates every leaf layout once, however many tiles share it, and
// each node type of each higher level is one launch of DFT weights and one
// weighted DFT whose data index is the child's type, so identical children
// (and any repeated sub-tree) cost no copies and no re-evaluation. Levels
// alternate between two beam buffers of the workspace; the top level writes
// the caller's beam.
// ---------------------------------------------------------------------------
namespace oskb {
namespace {

__global__ void hierarchy_setup_kernel(int num_types, double bx, double by,
        double bz, double* pointing, int num_zero, int* zero_idx)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x;
            i < num_types || i < num_zero; i += gridDim.x * blockDim.x)
    {
        if (i < num_types)
        {
            pointing[3 * i] = bx;
            pointing[3 * i + 1] = by;
            pointing[3 * i + 2] = bz;
        }
        if (zero_idx && i < num_zero) zero_idx[i] = 0;
    }
}

size_t align256(size_t b) { return (b + 255) & ~(size_t) 255; }

constexpr int kMaxLevels = 16;

// Checks the tree description; on success gives the most node types of the
// even and of the odd levels below the top (the two beam buffers) and the
// most children of any node (weights and the zero data index).
int hierarchy_shape(int num_levels, const int* num_types,
        const int* child_start, int& max_types_even, int& max_types_odd,
        int& max_children)
{
    if (num_levels < 2 || num_levels > kMaxLevels || !num_types ||
            !child_start)
        return OSKB_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < num_levels; ++l)
        if (num_types[l] < 1 || num_types[l] > 65535)
            return OSKB_ERR_INVALID_ARGUMENT;
    if (num_types[num_levels - 1] != 1) return OSKB_ERR_INVALID_ARGUMENT;
    max_types_even = max_types_odd = max_children = 0;
    for (int l = 0; l < num_levels - 1; ++l)
    {
        int& m = (l % 2) ? max_types_odd : max_types_even;
        if (num_types[l] > m) m = num_types[l];
    }
    if (child_start[0] != 0) return OSKB_ERR_INVALID_ARGUMENT;
    int nodes = 0;
    for (int l = 1; l < num_levels; ++l) nodes += num_types[l];
    for (int n = 0; n < nodes; ++n)
    {
        const long long c = (long long) child_start[n + 1] - child_start[n];
        if (c < 1 || c > INT_MAX / 2) return OSKB_ERR_INVALID_ARGUMENT;
        if (c > max_children) max_children = (int) c;
    }
    return 0;
}

size_t hierarchy_workspace(size_t elem, int num_directions,
        int max_types_even, int max_types_odd, int max_children,
        int num_leaf_types)
{
    return align256(elem * 8 * (size_t) max_types_even * num_directions) +
            align256(elem * 8 * (size_t) max_types_odd * num_directions) +
            align256(elem * 2 * (size_t) max_children) +
            align256(sizeof(double) * 3 * (size_t) num_leaf_types) +
            align256(sizeof(int) * (size_t) max_children);
}

template <typename T>
int station_beam_hierarchical(int num_levels, const int* num_types,
        int num_elements, const T* el_x, const T* el_y, const T* el_z,
        const double* orientation_x, const double* orientation_y,
        double dipole_length_m, int normalise_element,
        const int* normalise_array, const int* child_start,
        const T* child_x, const T* child_y, const T* child_z,
        const int* child_type, int swap_xy, int is_3d, double frequency_hz,
        const double* beam_enu, int num_directions, const T* x, const T* y,
        const T* z, void* workspace, size_t workspace_bytes, T* beam,
        void* stream)
{
    int max_even = 0, max_odd = 0, max_children = 0;
    if (int err = hierarchy_shape(num_levels, num_types, child_start,
            max_even, max_odd, max_children))
        return err;
    if (num_directions < 0 || !normalise_array || !beam_enu)
        return OSKB_ERR_INVALID_ARGUMENT;
    if (num_directions == 0) return 0;
    if (!child_x || !child_y || (is_3d && !child_z) || !workspace || !beam)
        return OSKB_ERR_INVALID_ARGUMENT;
    if (workspace_bytes < hierarchy_workspace(sizeof(T), num_directions,
            max_even, max_odd, max_children, num_types[0]))
        return OSKB_ERR_MEMORY_ALLOC_FAILURE;
    uint8_t* w = static_cast<uint8_t*>(workspace);
    T* level_beams[2];
    level_beams[0] = reinterpret_cast<T*>(w);
    w += align256(sizeof(T) * 8 * (size_t) max_even * num_directions);
    level_beams[1] = reinterpret_cast<T*>(w);
    w += align256(sizeof(T) * 8 * (size_t) max_odd * num_directions);
    T* weights = reinterpret_cast<T*>(w);
    w += align256(sizeof(T) * 2 * (size_t) max_children);
    double* pointing = reinterpret_cast<double*>(w);
    w += align256(sizeof(double) * 3 * (size_t) num_types[0]);
    int* zero_idx = child_type ? nullptr : reinterpret_cast<int*>(w);
    cudaStream_t s = as_stream(stream);
    const int n = num_types[0] > max_children ? num_types[0] : max_children;
    hierarchy_setup_kernel<<<(n + 255) / 256, 256, 0, s>>>(num_types[0],
            beam_enu[0], beam_enu[1], beam_enu[2], pointing, max_children,
            zero_idx);
    if (int err = check_launch("station_beam_hierarchical")) return err;
    // leaf beams [type][direction]: element pattern x leaf array factor,
    // blanked below the horizon, no final normalisation
    if (int err = station_beam_aa<T>(num_types[0], num_elements, el_x, el_y,
            el_z, nullptr, nullptr, nullptr, nullptr, nullptr, 1, nullptr,
            orientation_x, orientation_y, &dipole_length_m, nullptr, nullptr,
            nullptr, normalise_element, normalise_array[0], 0, swap_xy,
            is_3d, frequency_hz, pointing, nullptr, num_directions, x, y, z,
            0, level_beams[0], stream))
        return err;
    const double k = 2.0 * kPi * frequency_hz / 299792458.0;
    const T* zo = is_3d ? z : nullptr;
    const size_t beam_stride = (size_t) 8 * num_directions;
    int node = 0;
    for (int l = 1; l < num_levels; ++l)
    {
        const T* data = level_beams[(l - 1) % 2];
        const double* b = beam_enu + 3 * l;
        for (int j = 0; j < num_types[l]; ++j, ++node)
        {
            const int c0 = child_start[node];
            const int nc = child_start[node + 1] - c0;
            const T* cz = is_3d ? child_z + c0 : nullptr;
            const int* idx = child_type ? child_type + c0 : zero_idx;
            T* out = (l == num_levels - 1) ? beam :
                    level_beams[l % 2] + beam_stride * j;
            const T norm = normalise_array[l] ? (T) (1.0 / nc) : (T) 1;
            if constexpr (sizeof(T) == 8)
            {
                if (int err = oskb_evaluate_element_weights_dft_d(nc,
                        child_x + c0, child_y + c0, cz, nullptr, k, b[0],
                        b[1], is_3d ? b[2] : 0.0, weights, stream))
                    return err;
                if (int err = oskb_dftw_d(1, nc, k, weights, child_x + c0,
                        child_y + c0, cz, 0, num_directions, x, y, zo, idx,
                        data, 1, 1, 0, out, norm, stream))
                    return err;
            }
            else
            {
                if (int err = oskb_evaluate_element_weights_dft_f(nc,
                        child_x + c0, child_y + c0, cz, nullptr, (float) k,
                        (float) b[0], (float) b[1],
                        (float) (is_3d ? b[2] : 0.0), weights, stream))
                    return err;
                if (int err = oskb_dftw_f(1, nc, (float) k, weights,
                        child_x + c0, child_y + c0, cz, 0, num_directions, x,
                        y, zo, idx, data, 1, 1, 0, out, norm, stream))
                    return err;
            }
        }
    }
    return 0;
}

}  // namespace
}  // namespace oskb

extern "C" {

size_t oskb_station_beam_hierarchical_workspace_bytes(int precision_bytes,
        int num_levels, const int* num_types, const int* child_start,
        int num_directions)
{
    int max_even = 0, max_odd = 0, max_children = 0;
    if ((precision_bytes != 4 && precision_bytes != 8) ||
            num_directions < 0 || oskb::hierarchy_shape(num_levels,
                num_types, child_start, max_even, max_odd, max_children))
        return 0;
    return oskb::hierarchy_workspace((size_t) precision_bytes,
            num_directions, max_even, max_odd, max_children, num_types[0]);
}

size_t oskb_station_beam_two_level_workspace_bytes(int precision_bytes,
        int num_tile_types, int num_tiles, int num_directions)
{
    if (num_tiles < 1)
        return num_tile_types >= 1 && num_tiles == 0 &&
                num_directions >= 0 ? 256 : 0;
    const int types[2] = {num_tile_types, 1};
    const int start[2] = {0, num_tiles};
    return oskb_station_beam_hierarchical_workspace_bytes(precision_bytes,
            2, types, start, num_directions);
}

#define OSKB_HIERARCHICAL_ENTRY(T, S)                                        \
int oskb_station_beam_hierarchical_##S(int num_levels,                       \
        const int* num_types, int num_elements, const T* el_x,               \
        const T* el_y, const T* el_z, const double* orientation_x_rad,       \
        const double* orientation_y_rad, double dipole_length_m,             \
        int normalise_element, const int* normalise_array,                   \
        const int* child_start, const T* child_x, const T* child_y,          \
        const T* child_z, const int* child_type, int swap_xy, int is_3d,     \
        double frequency_hz, const double* beam_enu, int num_directions,     \
        const T* x, const T* y, const T* z, void* workspace,                 \
        size_t workspace_bytes, T* beam, void* stream)                       \
{                                                                            \
    return oskb::station_beam_hierarchical<T>(num_levels, num_types,         \
            num_elements, el_x, el_y, el_z, orientation_x_rad,               \
            orientation_y_rad, dipole_length_m, normalise_element,           \
            normalise_array, child_start, child_x, child_y, child_z,         \
            child_type, swap_xy, is_3d, frequency_hz, beam_enu,              \
            num_directions, x, y, z, workspace, workspace_bytes, beam,       \
            stream);                                                         \
}

OSKB_HIERARCHICAL_ENTRY(double, d)
OSKB_HIERARCHICAL_ENTRY(float, f)
#undef OSKB_HIERARCHICAL_ENTRY

// The two-level station is the hierarchy {tile layouts, station}.
#define OSKB_TWO_LEVEL_ENTRY(T, S)                                           \
int oskb_station_beam_two_level_##S(int num_tile_types, int num_elements,    \
        const T* el_x, const T* el_y, const T* el_z,                         \
        const double* orientation_x_rad, const double* orientation_y_rad,    \
        double dipole_length_m, int normalise_element,                       \
        int normalise_tile_array, int num_tiles, const T* tile_x,            \
        const T* tile_y, const T* tile_z, const int* tile_type,              \
        int normalise_station_array, int swap_xy, int is_3d,                 \
        double frequency_hz, double beam_x, double beam_y, double beam_z,    \
        int num_directions, const T* x, const T* y, const T* z,              \
        void* workspace, size_t workspace_bytes, T* beam, void* stream)      \
{                                                                            \
    if (num_tile_types < 1 || num_tiles < 0 || num_directions < 0)           \
        return OSKB_ERR_INVALID_ARGUMENT;                                    \
    if (num_tiles == 0 || num_directions == 0) return 0;                     \
    const int types[2] = {num_tile_types, 1};                                \
    const int start[2] = {0, num_tiles};                                     \
    const int norm[2] = {normalise_tile_array, normalise_station_array};     \
    const double b[6] = {beam_x, beam_y, beam_z, beam_x, beam_y, beam_z};    \
    return oskb::station_beam_hierarchical<T>(2, types, num_elements, el_x,  \
            el_y, el_z, orientation_x_rad, orientation_y_rad,                \
            dipole_length_m, normalise_element, norm, start, tile_x, tile_y, \
            tile_z, tile_type, swap_xy, is_3d, frequency_hz, b,              \
            num_directions, x, y, z, workspace, workspace_bytes, beam,       \
            stream);                                                         \
}

OSKB_TWO_LEVEL_ENTRY(double, d)
OSKB_TWO_LEVEL_ENTRY(float, f)
#undef OSKB_TWO_LEVEL_ENTRY

}  // extern "C"
