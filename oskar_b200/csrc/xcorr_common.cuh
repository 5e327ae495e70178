// Shared by the direct cross-correlation kernels (xcorr_direct.cu,
// xcorr_smear.cuh): the launch parameters, the work items and the cp.async
// staging helpers.
#pragma once

#include <string.h>

#include "common.cuh"

namespace oskb {
namespace {

constexpr int kTile = 32;      // stations per block edge
constexpr int kChunk = 8;      // sources per shared-memory chunk

template <typename T>
struct XcorrParams
{
    int num_src, num_st, offset_out;
    int src_stride;  // sources per station row of jones (= num_src)
    const T* jones;  // J [station][source], or E when K is fused
    const T *I, *Q, *U, *V, *l, *m, *n, *a, *b, *c;
    // Station (u, v, w) metres of dump t at st_u + t * uvw_time_stride
    // (v and w follow at +num_st and +2 num_st in block mode).
    const T *st_u, *st_v, *st_w, *st_x, *st_y;
    long long uvw_time_stride;
    double uv_min, uv_max;  // wavelengths (single call) or metres (block)
    int uv_filter_in_metres;
    double inv_wavelength;            // single call
    const double* inv_wavelength_c;   // block: [channel]
    double bw_scale;  // pi * frac_bandwidth * inv_wavelength (= pi bw / c0)
    double ts_base;   // pi * omega_earth * time_int_sec (x inv_wavelength)
    double gha0;                      // single call
    const double* gha0_t;             // block: [dump]
    double s_dec, c_dec;
    T* vis;
    // Items: num_times x num_channels x tiles x slices, in that nesting
    // (slices fastest). Source slice y covers [y * slice_len,
    // (y + 1) * slice_len). With more than one slice each CTA writes its sums to partial[y][baseline][comp] and
    // reduce_partials adds them to vis in slice order (deterministic).
    int num_times, num_channels, tiles, slices, slice_len;
    int tile_major;  // item order: tile outermost instead of innermost
    double* partial;
    // Fused Jones K (block mode): J = K E, K = exp(i 2 pi / lambda (u l +
    // v m + w (n - 1))), zero where I is outside (filter_min, filter_max].
    long long e_time_stride;  // E of dump t at jones + t * e_time_stride
    double filter_min, filter_max;
    // Brightness per channel (block mode): I, Q, U, V of channel c at
    // + c * flux_channel_stride (0: the same for every channel).
    long long flux_channel_stride;
};

template <typename T, bool MATRIX>
struct Staging
{
    // Bytes of one Jones element and the cp.async copy size used for it.
    static constexpr int ELEM = (int) sizeof(T) * (MATRIX ? 8 : 2);
    static constexpr int COPY = ELEM >= 16 ? 16 : ELEM;
    static constexpr int PIECES = ELEM / COPY;
};

// Per-source arrays staged with each chunk.
enum SrcArr { kI = 0, kQ, kU, kV, kL, kM, kN, kGa, kGb, kGc, kNumSrcArr };

// Per-item constants.
struct ItemCtx
{
    int t, c, p0, q0, src_begin, src_end;
    double inv_wavelength, ts_scale, s_ha, c_ha;
};

__device__ __forceinline__ void cp_async(void* smem, const void* gmem,
        bool in_range, int bytes)
{
    const unsigned s = (unsigned) __cvta_generic_to_shared(smem);
    const int src = in_range ? bytes : 0;  // 0: zero-fill, nothing read
    if (bytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                :: "r"(s), "l"(gmem), "r"(src) : "memory");
    else if (bytes == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n"
                :: "r"(s), "l"(gmem), "r"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n"
                :: "r"(s), "l"(gmem), "r"(src) : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Maps a linear block index to (bp, bq) with bp >= bq.
__device__ __forceinline__ void tri_block(int k, int& bp, int& bq)
{
    int p = (int) ((sqrt(8.0 * k + 1.0) - 1.0) * 0.5);
    while ((p + 1) * (p + 2) / 2 <= k) ++p;
    while (p * (p + 1) / 2 > k) --p;
    bp = p;
    bq = k - p * (p + 1) / 2;
}

// The work item's dump, channel, station tile, source slice and scales.
template <typename T>
__device__ __forceinline__ int decode_item(const XcorrParams<T>& prm,
        int item, bool time_smearing, ItemCtx& ctx)
{
    int r = item;
    const int slice = r % prm.slices; r /= prm.slices;
    int tile;
    if (prm.tile_major)
    {
        // Consecutive items share a station tile (its E rows stay in L2).
        const int tc = r % (prm.num_times * prm.num_channels);
        tile = r / (prm.num_times * prm.num_channels);
        ctx.c = tc % prm.num_channels;
        ctx.t = tc / prm.num_channels;
    }
    else
    {
        tile = r % prm.tiles;
        r /= prm.tiles;
        ctx.c = r % prm.num_channels;
        ctx.t = r / prm.num_channels;
    }
    int bp, bq;
    tri_block(tile, bp, bq);
    ctx.p0 = bp * kTile;
    ctx.q0 = bq * kTile;
    ctx.src_begin = slice * prm.slice_len;
    ctx.src_end = min(prm.num_src, ctx.src_begin + prm.slice_len);
    ctx.inv_wavelength = prm.inv_wavelength_c ?
            prm.inv_wavelength_c[ctx.c] : prm.inv_wavelength;
    ctx.ts_scale = prm.ts_base * ctx.inv_wavelength;
    ctx.s_ha = ctx.c_ha = 0;
    if (time_smearing) sincos(prm.gha0_t ? prm.gha0_t[ctx.t] : prm.gha0,
            &ctx.s_ha, &ctx.c_ha);
    return slice;
}

// Adds one baseline's sums (v, NC2 reals) to its visibility, or stores them
// as the slice's partial sums; every baseline of a slice is stored (zero
// where the uv filter drops it), so the reduction reads no stale data.
template <typename T, int NC2>
__device__ __forceinline__ void store_baseline(const XcorrParams<T>& prm,
        const ItemCtx& ctx, int slice, int p, int q, bool valid,
        const double (&v)[NC2])
{
    const int N = prm.num_st;
    const long long nbl = (long long) N * (N - 1) / 2;
    const long long bl = baseline_index(N, p, q);
    const long long tc = (long long) ctx.t * prm.num_channels + ctx.c;
    if (prm.partial)
    {
        double* out = prm.partial + (size_t) NC2 * (size_t) (((long long)
                slice * prm.num_times * prm.num_channels + tc) * nbl + bl);
#pragma unroll
        for (int k = 0; k < NC2; ++k) out[k] = valid ? v[k] : 0.0;
        return;
    }
    if (!valid) return;
    // Block layout [dump][channel][baseline] (the reference's
    // oskar_VisBlock order, private_vis_block.h:33-57).
    T* out = prm.vis + (size_t) NC2 * (size_t) (tc * nbl + bl +
            prm.offset_out);
#pragma unroll
    for (int k = 0; k < NC2; ++k) out[k] = (T) ((double) out[k] + v[k]);
}

}  // namespace
}  // namespace oskb
