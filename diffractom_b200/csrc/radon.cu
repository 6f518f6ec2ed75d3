// Parallel-beam Radon transform of a batch of channel-fastest images (the orientations of a batch are the channels),
// sm_100a, FP32. Semantics: operators/radon_kernels.cl of diffractom (ParallelRadon); tap weights as in
// dfx_common.cuh, which the CPU oracle (oracle/oracle_core.h) restates bit for bit.
//
// Work split: the 32 lanes of a warp own 8 channels each (256 channels per warp), so everything that depends on the
// geometry only (detector coordinate, tap bins and weights) is the same for the whole warp: one warp instruction
// serves 256 channels, and a zero weight skips its FMAs with a branch all lanes take.
//
// Forward (ray-driven gather, no atomics): a warp owns one bin of one angle, or four neighbouring bins (grouped table);
// it walks the pixels whose footprint reaches them, found per image row (radon_forward_v4) or listed in a table built
// once per geometry. The grid is ordered so that one channel block of the image stays in L2 while all angles and bins
// of the launch read it.
//
// Backward (pixel-driven, no atomics): a warp owns four neighbouring pixels of an image row (radon_backward_tile: whole
// images, two taps per pixel and angle), or one pixel (radon_backward_v3: pixel lists, more taps, few pixels; the
// per-angle constants are computed once per block into shared memory); per angle it evaluates the pixels' taps and
// reads 8 channels of each tap's sinogram bin per lane. A fused variant applies SPDHG's primal step in the epilogue (no
// dz array).
//
// The sinogram is float32 or, in the BF16 precision path, BF16 with its own row stride (bins of all orientation
// batches side by side): loads widen BF16 to float32 exactly, the forward rounds its float32 sums once on store.
#include <cuda_bf16.h>

#include "dfx_common.cuh"
#include "transpose.cuh"

namespace dfx {

constexpr int WARPS = 8;        // warps per block
constexpr int CPL = 8;          // channels per lane
constexpr int CPW = 32 * CPL;   // channels per warp

// The 8 channels of a lane are two runs of four, at Chan<T>::off(lane, 0) and (lane, 1) of the warp's 256, T the type
// that the inner loop loads. BF16: 8 channels side by side, one 16-byte load. float32: channels 4 lane and 128 + 4
// lane, so that each 16-byte load of the warp covers 512 contiguous bytes; with 8 channels side by side every load
// touched half of each of 8 lines, and L1 gave 64 instead of 87 or more bytes per clock and SM (measured, L1 hits).
template <typename T> struct Chan;
template <> struct Chan<float> {
    static __device__ __forceinline__ int off(int lane, int h) { return 4 * lane + h * (CPW / 2); }
};
template <> struct Chan<__nv_bfloat16> {
    static __device__ __forceinline__ int off(int lane, int h) { return CPL * lane + 4 * h; }
};

__device__ __forceinline__ void st4(float *p, const float *r)
{
    *reinterpret_cast<float4 *>(p) = make_float4(r[0], r[1], r[2], r[3]);
}

__device__ __forceinline__ void ld8(const float *p, float4 &a, float4 &b)
{
    a = __ldg(reinterpret_cast<const float4 *>(p));
    b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
}

__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

__device__ __forceinline__ void ld8(const __nv_bfloat16 *p, float4 &a, float4 &b)
{
    const uint4 u = __ldg(reinterpret_cast<const uint4 *>(p));
    a = make_float4(bf_lo(u.x), bf_hi(u.x), bf_lo(u.y), bf_hi(u.y));
    b = make_float4(bf_lo(u.z), bf_hi(u.z), bf_lo(u.w), bf_hi(u.w));
}

__device__ __forceinline__ void st8(float *p, const float (&r)[CPL])
{
    reinterpret_cast<float4 *>(p)[0] = make_float4(r[0], r[1], r[2], r[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(r[4], r[5], r[6], r[7]);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void st8(__nv_bfloat16 *p, const float (&r)[CPL])
{
    *reinterpret_cast<uint4 *>(p) = make_uint4(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]), pack_bf16(r[4], r[5]),
                                               pack_bf16(r[6], r[7]));
}

__device__ __forceinline__ void st4(__nv_bfloat16 *p, const float *r)
{
    *reinterpret_cast<uint2 *>(p) = make_uint2(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]));
}

// a += w p on 8 channels: four paired FMAs (FFMA2, sm_100), each lane of a pair rounded once as fmaf does
__device__ __forceinline__ void acc8(float (&a)[CPL], float w, const float4 &p0, const float4 &p1)
{
    const float2 ww = make_float2(w, w);
    float2 r0 = __ffma2_rn(ww, make_float2(p0.x, p0.y), make_float2(a[0], a[1]));
    float2 r1 = __ffma2_rn(ww, make_float2(p0.z, p0.w), make_float2(a[2], a[3]));
    float2 r2 = __ffma2_rn(ww, make_float2(p1.x, p1.y), make_float2(a[4], a[5]));
    float2 r3 = __ffma2_rn(ww, make_float2(p1.z, p1.w), make_float2(a[6], a[7]));
    a[0] = r0.x; a[1] = r0.y; a[2] = r1.x; a[3] = r1.y;
    a[4] = r2.x; a[5] = r2.y; a[6] = r3.x; a[7] = r3.y;
}

// bins strictly inside a pixel's footprint (t - hw, t + hw) at this angle: at most ceil(1 + |A|) for the trapezoid
// (2 for the hat), never more than the caller's bound n_taps
__device__ __forceinline__ int taps_of(const AngleGeo &g, int kernel, int n_taps)
{
    if (kernel != 1) return 2;
    const int t = max(2, (int)ceilf(1.0f + fabsf(g.A) - 1e-6f));
    return min(t, n_taps);
}

// first bin that can get a non-zero weight from a pixel at detector coordinate t
template <int KERNEL>
__device__ __forceinline__ int first_tap(const AngleGeo &g, float t)
{
    return KERNEL == 1 ? (int)floorf(__fsub_rn(t, g.hw)) + 1 : (int)floorf(t);
}

// ------------------------------------------------------------------------------------------------ forward
// Ray-driven gather: a warp owns one bin s of one angle and 256 channels. Per image row it evaluates the pixels whose
// footprint can reach s (two to four), skips zero weights (a branch the whole warp takes) and accumulates the
// weighted channels in registers: no shared memory, no atomics, a fixed summation order. The grid runs
// channel-block-major (blockIdx.z), so the columns of one channel block (npix x 256) are read from L2 by every
// angle and bin while they are resident.
template <int KERNEL, typename ST>
__global__ void __launch_bounds__(32 * WARPS) radon_forward_v4(
    const float *__restrict__ img, ST *__restrict__ sino, int64_t sld, const float4 *__restrict__ geo, int nx, int ny,
    int ns, int kstride, int kb, float scale)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = blockIdx.x * WARPS + warp;
    const int a = blockIdx.y;
    const int k = blockIdx.z * CPW + lane * CPL;
    if (s >= ns) return;                                   // whole warps
    const bool live = k < kstride;
    if (blockIdx.z * CPW >= kb) {                          // padding channels only
        const float zero[CPL] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (live) st8(sino + ((int64_t)a * ns + s) * sld + k, zero);
        return;
    }
    const bool load = k < kb;
    const AngleGeo g = load_geo(geo, a);
    const int nu = g.rows_are_y ? nx : ny, nv = g.rows_are_y ? ny : nx;
    const int64_t du = (g.rows_are_y ? 1 : (int64_t)nx) * kstride, dv = (g.rows_are_y ? (int64_t)nx : 1) * kstride;
    const float half = KERNEL == 1 ? g.hw : 1.0f;
    const float inv = __frcp_rn(g.A);
    const float fs = (float)s;
    float acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = 0.0f;
    const float *base = img + (live ? k : 0);
#pragma unroll 2
    for (int v = 0; v < nv; ++v) {
        const float c = __fmaf_rn(g.B, (float)v, g.T0);
        const float e1 = (fs - half - c) * inv, e2 = (fs + half - c) * inv;
        // a margin of 1e-3 pixel covers the rounding of e1, e2; the tap weights decide membership
        const int u0 = max((int)floorf(fminf(e1, e2) - 1e-3f), 0);
        const int u1 = min((int)ceilf(fmaxf(e1, e2) + 1e-3f), nu - 1);
        const float *row = base + (int64_t)v * dv;
        for (int u = u0; u <= u1; ++u) {
            const float w = tap_weight<KERNEL>(g, __fsub_rn(__fmaf_rn(g.A, (float)u, c), fs));
            if (w == 0.0f) continue;
            float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
            if (load) ld8(row + (int64_t)u * du, p0, p1);
            acc8(acc, w, p0, p1);
        }
    }
    if (!live) return;
    float r[CPL];
#pragma unroll
    for (int q = 0; q < CPL; ++q) r[q] = (k + q < kb) ? __fmul_rn(scale, acc[q]) : 0.0f;   // padding channels: 0
    st8(sino + ((int64_t)a * ns + s) * sld + k, r);
}

// ---- ray table: the non-zero taps of every (angle, bin) in the order radon_forward_v4 visits them (rows v, then
// pixels u ascending), as (pixel index, weight bits). The geometry of an operator is fixed, so the table is built
// once; the table-driven forward then spends its instructions on loads and FMAs only, with many taps in flight.
// supp (optional, one byte per pixel): only the taps of pixels inside the support; for images that are zero outside
// it (a solver's iterates projected onto the support) the forward through this table adds exactly the same terms
// minus zeros, so it gives the same bits.
// DERIV: the same taps with the weights K'(t - s) (tap_dweight), the table of the projections' derivative with
// respect to a detector shift of every angle.
template <int KERNEL, bool DERIV = false>
__global__ void ray_table_kernel(const float4 *__restrict__ geo, int n_angles, int nx, int ny, int ns,
                                 const uint8_t *__restrict__ supp, int32_t *__restrict__ counts,
                                 const int32_t *__restrict__ row_ptr, int2 *__restrict__ entries)
{
    const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;      // a * ns + s
    if (row >= (int64_t)n_angles * ns) return;
    const int a = (int)(row / ns), s = (int)(row % ns);
    const AngleGeo g = load_geo(geo, a);
    const int nu = g.rows_are_y ? nx : ny, nv = g.rows_are_y ? ny : nx;
    const float half = KERNEL == 1 ? g.hw : 1.0f;
    const float inv = __frcp_rn(g.A);
    const float fs = (float)s;
    int n = 0;
    int64_t pos = row_ptr ? row_ptr[row] : 0;
    for (int v = 0; v < nv; ++v) {
        const float c = __fmaf_rn(g.B, (float)v, g.T0);
        const float e1 = (fs - half - c) * inv, e2 = (fs + half - c) * inv;
        const int u0 = max((int)floorf(fminf(e1, e2) - 1e-3f), 0);
        const int u1 = min((int)ceilf(fmaxf(e1, e2) + 1e-3f), nu - 1);
        for (int u = u0; u <= u1; ++u) {
            const float d = __fsub_rn(__fmaf_rn(g.A, (float)u, c), fs);
            const float w = tap_weight<KERNEL>(g, d);
            if (w == 0.0f) continue;
            const int pix = g.rows_are_y ? u + nx * v : v + nx * u;
            if (supp && !supp[pix]) continue;
            if (row_ptr) entries[pos++] = make_int2(pix, __float_as_int(DERIV ? tap_dweight<KERNEL>(g, d) : w));
            ++n;
        }
    }
    if (!row_ptr) counts[row] = n;
}

// The lane's runs of the 256 channels from kblk on: k[h] their first channels (outputs: those below kstride), o[h] the
// offsets its loads use (runs past kb read channel kblk instead, and their sums are dropped).
template <typename T>
__device__ __forceinline__ void lane_runs(int lane, int kblk, int kb, int (&k)[2], int (&o)[2])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        o[h] = Chan<T>::off(lane, h);
        k[h] = kblk + o[h];
    }
    const bool two = sizeof(T) == 4;
    o[1] = (two ? k[1] : k[0]) < kb ? o[1] : 0;
    o[0] = k[0] < kb ? o[0] : 0;
}

// one output row of the warp's channels: scale r on channels below kb, 0 on the padding channels up to kstride
template <typename ST>
__device__ __forceinline__ void store_row(ST *row, const int (&k)[2], int kstride, int kb, float scale,
                                          const float (&r)[CPL])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (k[h] >= kstride) continue;
        float o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = k[h] + q < kb ? __fmul_rn(scale, r[4 * h + q]) : 0.0f;
        st4(row + k[h], o);
    }
}

// Raw channel loads of the table-driven forward: 8 channels kept as loaded (2 x float4, or 8 BF16 in a uint4) until
// their FMAs, so that a warp can hold many taps' loads in flight in few registers.
template <typename IT> struct Raw8;
template <> struct Raw8<float> { float4 a, b; };
template <> struct Raw8<__nv_bfloat16> { uint4 u; };

// o0, o1: the lane's two runs (Chan), those outside the row moved to channel 0 by lane_runs (their sums are dropped)
__device__ __forceinline__ void ldraw(const float *p, int o0, int o1, Raw8<float> &r)
{
    r.a = __ldg(reinterpret_cast<const float4 *>(p + o0));
    r.b = __ldg(reinterpret_cast<const float4 *>(p + o1));
}
__device__ __forceinline__ void ldraw(const __nv_bfloat16 *p, Raw8<__nv_bfloat16> &r)
{
    r.u = __ldg(reinterpret_cast<const uint4 *>(p));
}
__device__ __forceinline__ void accraw(float (&a)[CPL], float w, const Raw8<float> &r) { acc8(a, w, r.a, r.b); }
__device__ __forceinline__ void accraw(float (&a)[CPL], float w, const Raw8<__nv_bfloat16> &r)
{
    acc8(a, w, make_float4(bf_lo(r.u.x), bf_hi(r.u.x), bf_lo(r.u.y), bf_hi(r.u.y)),
         make_float4(bf_lo(r.u.z), bf_hi(r.u.z), bf_lo(r.u.w), bf_hi(r.u.w)));
}

// Table-driven forward: warp per (angle, bin, 256 channels), angle a of the launch = angles[a] of the table (angles
// NULL: a); the same taps, weights and summation order as radon_forward_v4, so the same bits. Bound by the L1 data
// path and L2 (a float32 launch of all 360 angles at 256 x 256 pixels, 1012 channels: 84 % and 80 % of their peaks);
// what it needs is loads in flight at few registers: a software pipeline over groups of U taps (60 registers; without
// it ptxas kept 40 and one tap's loads in flight). That launch went from 10.9 to 7.2 ms, 18 angles from 0.68 to 0.44 ms
// (U = 4: 8.1 and 0.46, U = 8: 11.7 and 0.64).
template <typename ST>
__global__ void __launch_bounds__(32 * WARPS) radon_forward_table(
    const float *__restrict__ img, ST *__restrict__ sino, int64_t sld, const int32_t *__restrict__ row_ptr,
    const int2 *__restrict__ entries, const int32_t *__restrict__ angles, int ns, int kstride, int kb, float scale)
{
    constexpr int U = 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = blockIdx.x * WARPS + warp;
    const int al = blockIdx.y;
    const int kblk = blockIdx.z * CPW;
    if (s >= ns) return;
    int k[2], o[2];
    lane_runs<float>(lane, kblk, kb, k, o);
    ST *out = sino + ((int64_t)al * ns + s) * sld;
    float acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = 0.0f;
    if (kblk < kb) {                                       // not padding channels only
        const int a = angles ? __ldg(angles + al) : al;
        const int64_t r = (int64_t)a * ns + s;
        int e = __ldg(row_ptr + r);
        const int e1 = __ldg(row_ptr + r + 1);
        const float *base = img + kblk;
        // software pipeline over groups of U taps: the next group's pixels are loaded while this one's FMAs run
        if (e + U <= e1) {
            int2 t[U], tn[U];
            Raw8<float> q[U];
#pragma unroll
            for (int i = 0; i < U; ++i) t[i] = __ldg(entries + e + i);
#pragma unroll
            for (int i = 0; i < U; ++i) ldraw(base + (int64_t)t[i].x * kstride, o[0], o[1], q[i]);
            e += U;
#pragma unroll 2
            for (; e + U <= e1; e += U) {
                Raw8<float> qn[U];
#pragma unroll
                for (int i = 0; i < U; ++i) tn[i] = __ldg(entries + e + i);
#pragma unroll
                for (int i = 0; i < U; ++i) ldraw(base + (int64_t)tn[i].x * kstride, o[0], o[1], qn[i]);
#pragma unroll
                for (int i = 0; i < U; ++i) accraw(acc, __int_as_float(t[i].y), q[i]);
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    t[i] = tn[i];
                    q[i] = qn[i];
                }
            }
#pragma unroll
            for (int i = 0; i < U; ++i) accraw(acc, __int_as_float(t[i].y), q[i]);
        }
        for (; e < e1; ++e) {
            const int2 t = __ldg(entries + e);
            Raw8<float> q;
            ldraw(base + (int64_t)t.x * kstride, o[0], o[1], q);
            accraw(acc, __int_as_float(t.y), q);
        }
    }
    store_row(out, k, kstride, kb, scale, acc);
}

// The table-driven forward of a BF16 image with BF16 rows: the same split, 16 taps loaded before their FMAs. A warp's tap
// is one 512-byte load, so that the wait for them counts, not L1: 0.281 ms for 18 angles at 256 x 256 pixels, 1012
// channels, 17 us for 9 at 97 x 40, 256 channels; the pipeline above with groups of 4 taps 0.285 ms and 19 us, of 6 0.288
// and 16, of 8 0.347 and 15.
__global__ void __launch_bounds__(32 * WARPS) radon_forward_table_bf16(
    const __nv_bfloat16 *__restrict__ img, __nv_bfloat16 *__restrict__ sino, int64_t sld,
    const int32_t *__restrict__ row_ptr, const int2 *__restrict__ entries, const int32_t *__restrict__ angles, int ns,
    int kstride, int kb, float scale)
{
    constexpr int U = 16;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = blockIdx.x * WARPS + warp;
    const int al = blockIdx.y;
    const int k = blockIdx.z * CPW + lane * CPL;
    if (s >= ns) return;
    const bool live = k < kstride;
    __nv_bfloat16 *out = sino + ((int64_t)al * ns + s) * sld + k;
    if (blockIdx.z * CPW >= kb) {
        const float zero[CPL] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (live) st8(out, zero);
        return;
    }
    const bool load = k < kb;
    const int a = angles ? __ldg(angles + al) : al;
    const int64_t r = (int64_t)a * ns + s;
    int e = __ldg(row_ptr + r);
    const int e1 = __ldg(row_ptr + r + 1);
    const __nv_bfloat16 *base = img + (load ? k : 0);
    float acc[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) acc[c] = 0.0f;
    for (; e + U <= e1; e += U) {
        int2 t[U];
        Raw8<__nv_bfloat16> q[U];
#pragma unroll
        for (int i = 0; i < U; ++i) t[i] = __ldg(entries + e + i);
#pragma unroll
        for (int i = 0; i < U; ++i) {
            q[i].u = make_uint4(0, 0, 0, 0);
            if (load) ldraw(base + (int64_t)t[i].x * kstride, q[i]);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) accraw(acc, __int_as_float(t[i].y), q[i]);
    }
    for (; e < e1; ++e) {
        const int2 t = __ldg(entries + e);
        Raw8<__nv_bfloat16> q;
        q.u = make_uint4(0, 0, 0, 0);
        if (load) ldraw(base + (int64_t)t.x * kstride, q);
        accraw(acc, __int_as_float(t.y), q);
    }
    if (!live) return;
    float o[CPL];
#pragma unroll
    for (int c = 0; c < CPL; ++c) o[c] = (k + c < kb) ? __fmul_rn(scale, acc[c]) : 0.0f;
    st8(out, o);
}

// ------------------------------------------------------------------------------------------------ grouped table
// The float32 forward reads each pixel of a row about twice per angle through the per-bin table: a pixel's footprint
// covers two bins (more for steep trapezoids), and every bin's warp loads it again. The grouped table lists, per
// (angle, group of GB consecutive bins), every pixel that reaches one of the group's bins, with its weight on each
// of them (0 where the per-bin row has no entry), in the per-bin rows' order (image row v, then u): one warp loads a
// pixel's channels once for the whole group, and every bin still adds exactly its per-bin row's taps in its order,
// so the sums are the per-bin forward's bits.
constexpr int GB = 4;           // bins per group

template <int KERNEL>
__global__ void ray_gtable_kernel(const float4 *__restrict__ geo, int n_angles, int nx, int ny, int ns,
                                  const uint8_t *__restrict__ supp, int32_t *__restrict__ counts,
                                  const int32_t *__restrict__ row_ptr, int32_t *__restrict__ pix_out,
                                  float4 *__restrict__ w_out)
{
    const int ng = (ns + GB - 1) / GB;
    const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;      // a * ng + g
    if (row >= (int64_t)n_angles * ng) return;
    const int a = (int)(row / ng), s0 = (int)(row % ng) * GB;
    const AngleGeo g = load_geo(geo, a);
    const int nu = g.rows_are_y ? nx : ny, nv = g.rows_are_y ? ny : nx;
    const float half = KERNEL == 1 ? g.hw : 1.0f;
    const float inv = __frcp_rn(g.A);
    int n = 0;
    int64_t pos = row_ptr ? row_ptr[row] : 0;
    for (int v = 0; v < nv; ++v) {
        const float c = __fmaf_rn(g.B, (float)v, g.T0);
        int u0[GB], u1[GB];
        int lo = nu, hi = -1;
#pragma unroll
        for (int j = 0; j < GB; ++j) {                    // each bin's candidate range, as the per-bin table's
            const float fs = (float)(s0 + j);
            const float e1 = (fs - half - c) * inv, e2 = (fs + half - c) * inv;
            u0[j] = max((int)floorf(fminf(e1, e2) - 1e-3f), 0);
            u1[j] = min((int)ceilf(fmaxf(e1, e2) + 1e-3f), nu - 1);
            if (s0 + j >= ns) u1[j] = -1;
            if (u0[j] <= u1[j]) {
                lo = min(lo, u0[j]);
                hi = max(hi, u1[j]);
            }
        }
        for (int u = lo; u <= hi; ++u) {
            float w[GB];
            bool any = false;
#pragma unroll
            for (int j = 0; j < GB; ++j) {
                w[j] = 0.0f;
                if (u < u0[j] || u > u1[j]) continue;
                const float d = __fsub_rn(__fmaf_rn(g.A, (float)u, c), (float)(s0 + j));
                w[j] = tap_weight<KERNEL>(g, d);
                any |= w[j] != 0.0f;
            }
            if (!any) continue;
            const int pix = g.rows_are_y ? u + nx * v : v + nx * u;
            if (supp && !supp[pix]) continue;
            if (row_ptr) {
                pix_out[pos] = pix;
                w_out[pos++] = make_float4(w[0], w[1], w[2], w[3]);
            }
            ++n;
        }
    }
    if (!row_ptr) counts[row] = n;
}

// Grouped-table forward of a float32 image: warp per (angle, GB bins, 256 channels); U pixels in flight, each pixel's
// FMAs into the bins whose weight is not 0 (a branch the whole warp takes). A block's warps take GA consecutive angles
// of two groups: the rays of neighbouring angles through the same bins cross nearly the same pixels, so the block
// finds them in L1 (hit rate 10 -> 64 %, L2 throughput 59 -> 28 % of its peak), which leaves the L1 data path as
// its bound (76 %). 360 angles at 256 x 256 pixels, 1012 channels: 10.2 ms with a lane's 8 channels side by side, 7.6
// with whole 512-byte loads (Chan), 6.6 with the block over angles (8 angles of one group: 6.7).
constexpr int GA = 4;           // angles per block

template <typename ST>
__global__ void __launch_bounds__(32 * WARPS) radon_forward_gtable(
    const float *__restrict__ img, ST *__restrict__ sino, int64_t sld, const int32_t *__restrict__ row_ptr,
    const int32_t *__restrict__ pix, const float4 *__restrict__ wts, const int32_t *__restrict__ angles, int n_angles,
    int ns, int kstride, int kb, float scale)
{
    constexpr int U = 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ng = (ns + GB - 1) / GB;
    const int grp = blockIdx.x * (WARPS / GA) + warp / GA;
    const int al = blockIdx.y * GA + warp % GA;
    const int kblk = blockIdx.z * CPW;
    if (grp >= ng || al >= n_angles) return;
    int k[2], o[2];
    lane_runs<float>(lane, kblk, kb, k, o);
    const int s0 = grp * GB;
    ST *out = sino + ((int64_t)al * ns + s0) * sld;
    const int nb = min(GB, ns - s0);
    float acc[GB][CPL];
#pragma unroll
    for (int j = 0; j < GB; ++j)
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[j][c] = 0.0f;
    if (kblk < kb) {                                       // not padding channels only
        const int a = angles ? __ldg(angles + al) : al;
        const int64_t r = (int64_t)a * ng + grp;
        int e = __ldg(row_ptr + r);
        const int e1 = __ldg(row_ptr + r + 1);
        const float *base = img + kblk;
        for (; e + U <= e1; e += U) {
            int p[U];
            float4 w[U];
            Raw8<float> q[U];
#pragma unroll
            for (int i = 0; i < U; ++i) {
                p[i] = __ldg(pix + e + i);
                w[i] = __ldg(wts + e + i);
            }
#pragma unroll
            for (int i = 0; i < U; ++i) ldraw(base + (int64_t)p[i] * kstride, o[0], o[1], q[i]);
#pragma unroll
            for (int i = 0; i < U; ++i) {
                if (w[i].x != 0.0f) accraw(acc[0], w[i].x, q[i]);
                if (w[i].y != 0.0f) accraw(acc[1], w[i].y, q[i]);
                if (w[i].z != 0.0f) accraw(acc[2], w[i].z, q[i]);
                if (w[i].w != 0.0f) accraw(acc[3], w[i].w, q[i]);
            }
        }
        for (; e < e1; ++e) {
            const int p = __ldg(pix + e);
            const float4 w = __ldg(wts + e);
            Raw8<float> q;
            ldraw(base + (int64_t)p * kstride, o[0], o[1], q);
            if (w.x != 0.0f) accraw(acc[0], w.x, q);
            if (w.y != 0.0f) accraw(acc[1], w.y, q);
            if (w.z != 0.0f) accraw(acc[2], w.z, q);
            if (w.w != 0.0f) accraw(acc[3], w.w, q);
        }
    }
#pragma unroll
    for (int j = 0; j < GB; ++j)
        if (j < nb) store_row(out + (int64_t)j * sld, k, kstride, kb, scale, acc[j]);
}

// ------------------------------------------------------------------------------------------------ backward
// SPDHG primal step of one coefficient: the operations of primal_update_kernel (solver.cu), bitwise
__device__ __forceinline__ void primal_step(float &x, float &z, float t, float dz, float inv_p, float lam)
{
    const float zi = __fadd_rn(z, dz);
    z = zi;
    const float zb = __fadd_rn(zi, __fmul_rn(inv_p, dz));
    x = t > 0.0f ? fmaxf(0.0f, __fsub_rn(x, __fmul_rn(t, __fadd_rn(zb, lam)))) : 0.0f;
}

// A pixel's result on the lane's run h of four channels from k on: MODE 0 writes the backprojection acc to img, MODE 1
// applies it to x (img), z with the steps T and writes the BF16 copy of x. Channels kb .. kstride-1 are padding: MODE 0
// writes 0, MODE 1 takes dz = 0 (which leaves z, and x, 0 there, unchanged); a warp with padding channels only does
// not touch MODE 1's arrays.
template <int MODE>
__device__ __forceinline__ void finish_run(float *img, float *z, const float *T, __nv_bfloat16 *xb, int64_t row, int k,
                                           int kstride, int kb, const float *acc, float inv_p, float lam)
{
    if (k >= kstride) return;
    const int64_t o = row * kstride + k;
    float r[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = k + c < kb ? acc[c] : 0.0f;
    if (MODE == 0) {
        st4(img + o, r);
        return;
    }
    float4 *xp = reinterpret_cast<float4 *>(img + o), *zp = reinterpret_cast<float4 *>(z + o);
    float4 xv = *xp, zv = *zp;
    const float4 tv = __ldg(reinterpret_cast<const float4 *>(T + o));
    primal_step(xv.x, zv.x, tv.x, r[0], inv_p, lam);
    primal_step(xv.y, zv.y, tv.y, r[1], inv_p, lam);
    primal_step(xv.z, zv.z, tv.z, r[2], inv_p, lam);
    primal_step(xv.w, zv.w, tv.w, r[3], inv_p, lam);
    *xp = xv;
    *zp = zv;
    const float xn[4] = {xv.x, xv.y, xv.z, xv.w};
    if (xb) st4(xb + o, xn);           // the BF16 copy of x the next forward projection reads
}

// 8 channels of a sinogram row in float32: the lane's two runs (o0, o1 as lane_runs gives them)
__device__ __forceinline__ void ldrow(const float *p, int o0, int o1, float4 &a, float4 &b)
{
    a = __ldg(reinterpret_cast<const float4 *>(p + o0));
    b = __ldg(reinterpret_cast<const float4 *>(p + o1));
}
__device__ __forceinline__ void ldrow(const __nv_bfloat16 *p, int o0, int, float4 &a, float4 &b) { ld8(p + o0, a, b); }

// Any tap count and any pixels: img (npix, kstride) = backprojection; plist (optional): only the pixels plist[0 ..
// n_out-1], output row r for pixel plist[r] (the same arithmetic per pixel as the whole image). MODE as finish_run.
// P channel groups of 256 per warp: the pixel's taps and weights are computed once for P x 8 channels per lane; every
// channel sums the same terms in the same order whatever P is. Whole images with two taps per pixel and angle take
// radon_backward_tile unless they have few pixels (launch_backward). Launches of few warps wait for one angle's chain
// (place, loads, FMAs) after the other: the loop over the angles is unrolled, so that the next angles' places are
// computed meanwhile (48 x 48 pixels, 180 angles, 256 channels 95 -> 62.5 us, BF16 rows 67 -> 58 us; unrolled by 4: 66
// us), and the lane's first run is folded into the row pointer. PAIRS (P = 1, more than two taps): two taps' rows loaded
// before their FMAs, 164 -> 114 us in that launch with four taps; with P = 2 it costs registers (1.02 -> 1.27 ms for 99 x
// 99 pixels, 1000 channels), with two taps code (62.5 -> 65 us).
template <int KERNEL, int MODE, typename ST, int P, bool PAIRS>
__global__ void __launch_bounds__(32 * WARPS) radon_backward_v3(
    const ST *__restrict__ sino, int64_t sld, float *__restrict__ img, const float4 *__restrict__ geo, int n_angles, int nx,
    int ny, int ns, int kstride, int kb, int n_taps, float *__restrict__ z, const float *__restrict__ T, float inv_p,
    float lam, __nv_bfloat16 *__restrict__ xb, const int32_t *__restrict__ plist, int64_t n_out)
{
    extern __shared__ AngleParams prm[];                   // the constants of every angle
    for (int i = threadIdx.x; i < n_angles; i += blockDim.x) prm[i] = pack_geo(load_geo(geo, i));
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t p = (int64_t)blockIdx.x * WARPS + warp;     // output row
    const int kblk = blockIdx.y * CPW * P;
    if (p >= n_out) return;
    int k[P][2], o[P][2];
    bool data[P];                          // not a group of padding channels only
#pragma unroll
    for (int h = 0; h < P; ++h) {
        lane_runs<ST>(lane, kblk + h * CPW, kb, k[h], o[h]);
        data[h] = kblk + h * CPW < kb;
    }
    const int64_t pix = plist ? (int64_t)__ldg(plist + p) : p;
    const int px = (int)(pix % nx), py = (int)(pix / nx);
    const float fx = (float)px, fy = (float)py;
    float acc[P][CPL];
#pragma unroll
    for (int h = 0; h < P; ++h)
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[h][c] = 0.0f;
    const ST *col = sino + kblk;
    if (P == 1) {
        col += o[0][0];
        o[0][1] -= o[0][0];
        o[0][0] = 0;
    }
    const int64_t angle_stride = (int64_t)ns * sld;
    if (data[0]) {
#pragma unroll 8
        for (int a = 0; a < n_angles; ++a, col += angle_stride) {
            const AngleGeo g = unpack_geo(prm[a]);
            const float t = __fmaf_rn(g.A, g.rows_are_y ? fx : fy, __fmaf_rn(g.B, g.rows_are_y ? fy : fx, g.T0));
            const int sf = first_tap<KERNEL>(g, t);
            const int ntap = taps_of(g, KERNEL, n_taps);
            if (ntap == 2 && sf >= 0 && sf + 1 < ns) {        // the common case: two taps inside the detector
                const float w0 = __fmul_rn(g.w, tap_weight<KERNEL>(g, __fsub_rn(t, (float)sf)));
                const float w1 = __fmul_rn(g.w, tap_weight<KERNEL>(g, __fsub_rn(t, (float)(sf + 1))));
#pragma unroll
                for (int h = 0; h < P; ++h) {
                    if (!data[h]) continue;
                    float4 a0, a1, b0, b1;
                    ldrow(col + h * CPW + (int64_t)sf * sld, o[h][0], o[h][1], a0, a1);
                    ldrow(col + h * CPW + (int64_t)(sf + 1) * sld, o[h][0], o[h][1], b0, b1);
                    acc8(acc[h], w0, a0, a1);
                    acc8(acc[h], w1, b0, b1);
                }
                continue;
            }
            if constexpr (PAIRS) {
                for (int i = 0; i < ntap; i += 2) {
                    float ww[2];
                    bool on[2];
                    float4 q[2][2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int s = sf + i + j;
                        const float w = tap_weight<KERNEL>(g, __fsub_rn(t, (float)s));
                        on[j] = i + j < ntap && s >= 0 && s < ns && w != 0.0f;
                        ww[j] = __fmul_rn(g.w, w);
                        if (on[j]) ldrow(col + (int64_t)s * sld, o[0][0], o[0][1], q[j][0], q[j][1]);
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        if (on[j]) acc8(acc[0], ww[j], q[j][0], q[j][1]);
                }
                continue;
            }
            for (int i = 0; i < ntap; ++i) {
                const int s = sf + i;
                if (s < 0 || s >= ns) continue;
                const float w = tap_weight<KERNEL>(g, __fsub_rn(t, (float)s));
                if (w == 0.0f) continue;
                const float ww = __fmul_rn(g.w, w);
#pragma unroll
                for (int h = 0; h < P; ++h) {
                    if (!data[h]) continue;
                    float4 q0, q1;
                    ldrow(col + h * CPW + (int64_t)s * sld, o[h][0], o[h][1], q0, q1);
                    acc8(acc[h], ww, q0, q1);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < P; ++h) {
        if (MODE == 1 && !data[h]) continue;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            finish_run<MODE>(img, z, T, xb, p, k[h][r], kstride, kb, acc[h] + 4 * r, inv_p, lam);
    }
}

// Whole images whose pixels have two taps per angle (bins no narrower than pixels): a warp owns TX neighbouring pixels
// of an image row and 256 channels. radon_backward_v3 is bound by the L1 data path: two bins loaded per pixel and
// angle, for 16 paired FMAs. The TX pixels of a row share bins: their first taps step by 0 or 1 bin from pixel to
// pixel, so an angle's taps cover 2 to 5 bins, 3.9 on average, each loaded once into registers. Which bins a pixel
// takes is then a choice of registers, made by one switch per angle, which the whole warp takes alike, over the
// 15 possible step patterns with straight-line code for each. The lanes compute the tap weights of BA angles in
// parallel (lane = angle and pixel) and read them back as broadcasts. The terms and their order per pixel and channel
// are radon_backward_v3's, so are the sums. BW rows below one another make a block: they share bins in L1 (65 % hits).
// 256 x 256 pixels, 1012 channels, 360 angles: 8.2 ms with a pixel per warp, 5.0 so (with 8 neighbouring channels per
// lane 10.8; BF16 rows 6.4 -> 4.1), 18 angles with SPDHG's primal step 0.49 -> 0.39 ms. Latency is what is left (24
// warps of 80 registers; L1 data path 62 %, issue 52 %): 6.2 ms at 20 warps, 7.7 ms for 4 x 2 pixels with a switch per
// pixel, 5.5 ms for 512 channels per warp.
constexpr int TX = 4;                           // pixels of a warp
constexpr int BW = 4;                           // warps per block: rows below one another
constexpr int BA = 32 / TX;                     // angles per weight batch (one lane per angle and pixel)

// first taps of a row's pixels relative to the smallest: code bit j - 1: a step of one bin between pixels j - 1 and j,
// upwards (DOWN 0) or downwards
__host__ __device__ constexpr int tap_offset(int bits, int down, int j)
{
    int n = 0;
    for (int i = 1; i < TX; ++i)
        if (down ? i > j : i <= j) n += (bits >> (i - 1)) & 1;
    return n;
}

template <typename ST>
__device__ __forceinline__ const ST *at_bytes(const ST *p, uint32_t bytes)
{
    return reinterpret_cast<const ST *>(reinterpret_cast<const char *>(p) + bytes);
}

__device__ __forceinline__ void ldrun(const float *p, uint32_t b0, uint32_t b1, float4 &a, float4 &b)
{
    a = __ldg(reinterpret_cast<const float4 *>(at_bytes(p, b0)));
    b = __ldg(reinterpret_cast<const float4 *>(at_bytes(p, b1)));
}
__device__ __forceinline__ void ldrun(const __nv_bfloat16 *p, uint32_t b0, uint32_t, float4 &a, float4 &b)
{
    ld8(at_bytes(p, b0), a, b);
}

// the taps of one angle on TX pixels of a row: the first bin's row b0 bytes into the angle's rows, bins bin_b bytes
// apart, the lane's two runs d0 and d1 bytes into a row
template <int BITS, int DOWN, typename ST>
__device__ __forceinline__ void row_taps(float (&acc)[TX][CPL], const ST *col, uint32_t b0, uint32_t bin_b,
                                         uint32_t d0, uint32_t d1, const float2 (&w)[TX])
{
    constexpr int NB = 2 + tap_offset(BITS, 0, TX - 1);   // bins under the row
    float4 va[NB], vb[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) ldrun(col, b0 + b * bin_b + d0, b0 + b * bin_b + d1, va[b], vb[b]);
#pragma unroll
    for (int j = 0; j < TX; ++j) {
        const int b = tap_offset(BITS, DOWN, j);
        acc8(acc[j], w[j].x, va[b], vb[b]);
        acc8(acc[j], w[j].y, va[b + 1], vb[b + 1]);
    }
}

template <int KERNEL, int MODE, typename ST>
__global__ void __launch_bounds__(32 * BW, 6) radon_backward_tile(
    const ST *__restrict__ sino, int64_t sld, float *__restrict__ img, const float4 *__restrict__ geo, int n_angles,
    int nx, int ny, int ns, int kstride, int kb, float *__restrict__ z, const float *__restrict__ T, float inv_p,
    float lam, __nv_bfloat16 *__restrict__ xb)
{
    __shared__ __align__(16) float2 wts[BW][BA][TX];   // the two tap weights of every pixel
    __shared__ int first[BW][BA][TX];                  // their first bins
    __shared__ int2 head[BW][BA];                      // byte offset of the row's first bin, step code
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nbx = (nx + TX - 1) / TX;
    const int x0 = (int)(blockIdx.x % nbx) * TX;
    const int y = (int)(blockIdx.x / nbx) * BW + warp;
    const int kblk = blockIdx.y * CPW;
    if (y >= ny) return;                        // whole warps; no block-wide synchronisation below
    int k[2], o[2];
    lane_runs<ST>(lane, kblk, kb, k, o);
    const uint32_t d0 = (uint32_t)(o[0] * sizeof(ST)), d1 = (uint32_t)(o[1] * sizeof(ST));
    float acc[TX][CPL];
#pragma unroll
    for (int j = 0; j < TX; ++j)
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[j][c] = 0.0f;
    const int64_t angle_stride = (int64_t)ns * sld;
    const uint32_t bin_b = (uint32_t)(sld * sizeof(ST));
    if (kblk < kb) {
        for (int a0 = 0; a0 < n_angles; a0 += BA) {
            __syncwarp();
            {
                const int i = lane / TX, j = lane % TX;
                const AngleGeo g = load_geo(geo, min(a0 + i, n_angles - 1));
                // pixels past the image's edge stand in for the last one (their sums are dropped)
                const float fx = (float)min(x0 + j, nx - 1), fy = (float)y;
                const float t = __fmaf_rn(g.A, g.rows_are_y ? fx : fy, __fmaf_rn(g.B, g.rows_are_y ? fy : fx, g.T0));
                const int sf = first_tap<KERNEL>(g, t);
                wts[warp][i][j] = make_float2(__fmul_rn(g.w, tap_weight<KERNEL>(g, __fsub_rn(t, (float)sf))),
                                              __fmul_rn(g.w, tap_weight<KERNEL>(g, __fsub_rn(t, (float)(sf + 1)))));
                int lo = sf, hi = sf;
#pragma unroll
                for (int d = 1; d < TX; d *= 2) {
                    lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, d));
                    hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, d));
                }
                // the row's code: bits 0..2 a step of one bin between neighbouring pixels, bit 3 downwards; 16: none of
                // the straight-line bodies
                const int before = __shfl_up_sync(0xFFFFFFFFu, sf, 1), step = j > 0 ? sf - before : 0;
                uint32_t code = 0;
                if (step == 1) code = 1u << (j - 1) | 32u;
                else if (step == -1) code = 1u << (j - 1) | 8u;
                else if (step != 0) code = 16u;
                if (lo < 0 || hi + 1 >= ns) code |= 16u;            // at the detector's edge
#pragma unroll
                for (int d = 1; d < TX; d *= 2) code |= __shfl_xor_sync(0xFFFFFFFFu, code, d);
                if ((code & 40u) == 40u) code |= 16u;               // up and down
                first[warp][i][j] = sf;
                if (j == 0) head[warp][i] = make_int2((int)(lo * bin_b), code & 16u ? 16 : (int)(code & 15u));
            }
            __syncwarp();
            const int na = min(BA, n_angles - a0);
            const ST *col = sino + kblk + a0 * angle_stride;
            for (int i = 0; i < na; ++i, col += angle_stride) {
                const int2 hd = head[warp][i];
                const float4 w01 = reinterpret_cast<const float4 *>(wts[warp][i])[0];
                const float4 w23 = reinterpret_cast<const float4 *>(wts[warp][i])[1];
                const float2 w[TX] = {make_float2(w01.x, w01.y), make_float2(w01.z, w01.w), make_float2(w23.x, w23.y),
                                      make_float2(w23.z, w23.w)};
#define DFX_ROW(BITS, DOWN) row_taps<BITS, DOWN, ST>(acc, col, (uint32_t)hd.x, bin_b, d0, d1, w); break
                switch (hd.y) {
                case 0: DFX_ROW(0, 0);
                case 1: DFX_ROW(1, 0);
                case 2: DFX_ROW(2, 0);
                case 3: DFX_ROW(3, 0);
                case 4: DFX_ROW(4, 0);
                case 5: DFX_ROW(5, 0);
                case 6: DFX_ROW(6, 0);
                case 7: DFX_ROW(7, 0);
                case 9: DFX_ROW(1, 1);
                case 10: DFX_ROW(2, 1);
                case 11: DFX_ROW(3, 1);
                case 12: DFX_ROW(4, 1);
                case 13: DFX_ROW(5, 1);
                case 14: DFX_ROW(6, 1);
                case 15: DFX_ROW(7, 1);
                default:
                    // each pixel's taps inside the detector
#pragma unroll
                    for (int j = 0; j < TX; ++j) {
                        const int s = first[warp][i][j];
                        const bool both = s >= 0 && s + 1 < ns;
#pragma unroll
                        for (int i2 = 0; i2 < 2; ++i2) {
                            const float wt = i2 ? w[j].y : w[j].x;
                            if (!both && (s + i2 < 0 || s + i2 >= ns || wt == 0.0f)) continue;
                            float4 q0, q1;
                            ldrun(col, (uint32_t)(s + i2) * bin_b + d0, (uint32_t)(s + i2) * bin_b + d1, q0, q1);
                            acc8(acc[j], wt, q0, q1);
                        }
                    }
                }
#undef DFX_ROW
            }
        }
    }
    if (MODE == 1 && kblk >= kb) return;
#pragma unroll
    for (int j = 0; j < TX; ++j) {
        if (x0 + j >= nx) continue;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            finish_run<MODE>(img, z, T, xb, (int64_t)y * nx + x0 + j, k[r], kstride, kb, acc[j] + 4 * r, inv_p, lam);
    }
}

// ------------------------------------------------------------------------------------------------ batch helpers
// Element-wise on channel-fastest batches (npix, kstride) whose channels kb .. kstride-1 are padding:
// mode 0: x = 1 inside the support on live channels, else 0 (support_ones); mode 1: x = 0 outside the support, on
// padding channels or where negative (project_support); mode 2: T = min(T, c / colsum) inside the support where
// colsum > 0 (tmin).
// V channels per step (4 where the stride and the arrays allow 16-byte accesses), with 32-bit indices where they reach.
// HBM bounds it: on 256 x 256 pixels x 960 channels 0.23 ms with one channel per step and 64-bit divisions, now 0.11.
template <int V, typename Index>
__global__ void __launch_bounds__(256) batch_support_kernel(float *__restrict__ x, const float *__restrict__ colsum,
                                                            const uint8_t *__restrict__ supp, int64_t npix, int kstride,
                                                            int kb, float c, int mode)
{
    const Index kv = (Index)(kstride / V), n = (Index)npix * kv;
    for (Index i = blockIdx.x * (Index)256 + threadIdx.x; i < n; i += (Index)gridDim.x * 256) {
        const Index p = i / kv;
        const int k = (int)(i - p * kv) * V;
        const bool in = supp ? __ldg(supp + p) != 0 : true;
        alignas(16) float r[V], cs[V];
        if (V == 4) {
            if (mode != 0) *reinterpret_cast<float4 *>(r) = reinterpret_cast<const float4 *>(x)[i];
            if (mode == 2) *reinterpret_cast<float4 *>(cs) = __ldg(reinterpret_cast<const float4 *>(colsum) + i);
        } else {
            if (mode != 0) r[0] = x[i];
            if (mode == 2) cs[0] = __ldg(colsum + i);
        }
#pragma unroll
        for (int q = 0; q < V; ++q) {
            const bool inside = in && k + q < kb;
            if (mode == 0) r[q] = inside ? 1.0f : 0.0f;
            else if (mode == 1) r[q] = !inside || r[q] < 0.0f ? 0.0f : r[q];
            else if (mode == 3) r[q] = inside ? r[q] : 0.0f;
            else if (inside && cs[q] > 0.0f) r[q] = fminf(r[q], __fdiv_rn(c, cs[q]));
        }
        if (V == 4) reinterpret_cast<float4 *>(x)[i] = *reinterpret_cast<const float4 *>(r);
        else x[i] = r[0];
    }
}

static int check_radon_args(const void *in, const void *out, const void *geo, int n_angles, int nx, int ny,
                            int n_det, int kstride, int kb, int kernel)
{
    DFX_REQUIRE(in && out && geo, "radon: null pointer");
    DFX_REQUIRE(n_angles >= 0 && nx > 0 && ny > 0 && n_det > 0, "radon: bad sizes (angles %d, %d x %d, %d bins)",
                n_angles, nx, ny, n_det);
    DFX_REQUIRE(kstride > 0 && kstride % CPL == 0 && kb >= 0 && kb <= kstride,
                "radon: kstride (%d) must be a positive multiple of %d and kb (%d) <= kstride", kstride, CPL, kb);
    DFX_REQUIRE(kernel == 0 || kernel == 1, "radon: kernel must be 0 (hat) or 1 (trapezoid)");
    DFX_REQUIRE(((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0 && ((uintptr_t)geo % 16) == 0,
                "radon: arrays must be 16-byte aligned");
    DFX_REQUIRE((int64_t)nx * ny * kstride < ((int64_t)1 << 40), "radon: image batch too large");
    return DFX_OK;
}

template <typename Kernel>
static int allow_smem(Kernel kernel, size_t bytes)
{
    if (bytes <= 48 * 1024) return DFX_OK;
    const cudaError_t e = allow_max_dynamic_smem(kernel);
    if (e != cudaSuccess) {
        set_error("radon: %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
        return DFX_ECUDA;
    }
    return DFX_OK;
}

template <int KERNEL, int MODE, typename ST>
static int launch_backward(const ST *sino, int64_t sld, float *img, const float *geo, int n_angles, int nx, int ny,
                           int n_det, int kstride, int kb, int n_taps, float *z, const float *T, float inv_p, float lam,
                           __nv_bfloat16 *xb, void *stream, const int32_t *plist = nullptr, int64_t n_list = 0)
{
    const int64_t npix = plist ? n_list : (int64_t)nx * ny;
    const size_t smem = sizeof(AngleParams) * (size_t)(n_angles > 0 ? n_angles : 1);
    // radon_backward_v3's limit, for both kernels alike: which one serves a launch depends on its size
    DFX_REQUIRE(smem <= 200 * 1024, "radon: %d angles exceed the shared memory of one launch", n_angles);
    // Few warps (under 28 per SM with one pixel and 256 channels each, 32 with the primal step, 24 for BF16 rows): one
    // warp per pixel and channel group, whose chain per angle is the shortest. Whole images, one pixel per warp against
    // four, 90 angles, without the primal step, with it, and BF16 rows: 48 x 48 pixels, 256 channels (16 per SM) 34 and
    // 50 us, 34 and 52, 32 and 44; 64 x 64, 64 channels (28) 44 and 52, 46 and 52, 46 and 48; 48 x 48, 400 channels (31)
    // 46 and 53, 46 and 55, 48 and 48, but at 12 angles 35.3 and 34.3 for a call without the step; 64 x 40, 400 channels
    // (35) 56 and 54, 60 and 56, 59 and 50; 80 x 80, 200 channels (43) 75 and 55, 77 and 58, 67 and 50.
    constexpr int line = sizeof(ST) == 2 ? 24 : MODE == 1 ? 32 : 28;
    const bool few = npix * cdiv(kstride, CPW) < line * 148;
    // pixels with at most two taps, an angle's rows within 32-bit byte offsets: neighbouring pixels share their bins
    if (!plist && !few && n_taps == 2 && (int64_t)n_det * sld * (int64_t)sizeof(ST) < ((int64_t)1 << 32)) {
        const dim3 tiles((unsigned)(cdiv(nx, TX) * cdiv(ny, BW)), (unsigned)cdiv(kstride, CPW));
        DFX_REQUIRE(cdiv(nx, TX) * cdiv(ny, BW) < 2147483647LL && tiles.y <= 65535u,
                    "radon: batch too large for one launch");
        radon_backward_tile<KERNEL, MODE, ST><<<tiles, 32 * BW, 0, (cudaStream_t)stream>>>(
            sino, sld, img, reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, kstride, kb, z, T, inv_p,
            lam, xb);
        return launch_status(MODE ? "radon_backward_spdhg" : "radon_backward");
    }
    // two channel groups per warp where the batch has them (the taps of a pixel are evaluated once for 16 channels per
    // lane: 5 to 14 % faster from 40 warps per SM on), one where that leaves few warps (up to 1.7 times faster)
    const bool pair = kstride > CPW && !few;
    dim3 grid((unsigned)cdiv(npix, WARPS), (unsigned)cdiv(kstride, pair ? 2 * CPW : CPW));
    DFX_REQUIRE(grid.x < 2147483647u && grid.y <= 65535u, "radon: batch too large for one launch");
    const auto kernel = pair ? radon_backward_v3<KERNEL, MODE, ST, 2, false>
                        : KERNEL == 1 && n_taps > 2 ? radon_backward_v3<KERNEL, MODE, ST, 1, KERNEL == 1>
                                                    : radon_backward_v3<KERNEL, MODE, ST, 1, false>;
    const int st = allow_smem(kernel, smem);
    if (st) return st;
    kernel<<<grid, 32 * WARPS, smem, (cudaStream_t)stream>>>(sino, sld, img, reinterpret_cast<const float4 *>(geo),
                                                             n_angles, nx, ny, n_det, kstride, kb, n_taps, z, T, inv_p,
                                                             lam, xb, plist, npix);
    return launch_status(MODE ? "radon_backward_spdhg" : "radon_backward");
}

}  // namespace dfx

using namespace dfx;

template <typename ST>
static int radon_forward_any(const float *img_k, ST *sino, int64_t sld, const float *geo, int n_angles, int nx, int ny,
                             int n_det, int kstride, int kb, int kernel, float scale, void *stream)
{
    int st = check_radon_args(img_k, sino, geo, n_angles, nx, ny, n_det, kstride, kb, kernel);
    if (st) return st;
    DFX_REQUIRE(sld >= kstride && sld % CPL == 0, "radon: sinogram row stride (%lld) must be a multiple of %d >= "
                "kstride", (long long)sld, CPL);
    if (n_angles == 0) return DFX_OK;
    DFX_REQUIRE(n_angles <= 65535, "radon: at most 65535 angles per launch");
    DFX_REQUIRE(cdiv(kstride, CPW) <= 65535, "radon: kstride too large for one launch");
    dim3 grid((unsigned)cdiv(n_det, WARPS), (unsigned)n_angles, (unsigned)cdiv(kstride, CPW));
    if (kernel == 1)
        radon_forward_v4<1, ST><<<grid, 32 * WARPS, 0, (cudaStream_t)stream>>>(
            img_k, sino, sld, reinterpret_cast<const float4 *>(geo), nx, ny, n_det, kstride, kb, scale);
    else
        radon_forward_v4<0, ST><<<grid, 32 * WARPS, 0, (cudaStream_t)stream>>>(
            img_k, sino, sld, reinterpret_cast<const float4 *>(geo), nx, ny, n_det, kstride, kb, scale);
    return launch_status("radon_forward");
}

template <typename ST, typename IT>
static int radon_forward_table_any(const IT *img_k, ST *sino, int64_t sld, const int32_t *row_ptr,
                                   const int32_t *entries, const int32_t *angles, int n_angles, int n_det,
                                   int kstride, int kb, float scale, void *stream)
{
    DFX_REQUIRE(img_k && sino && row_ptr && entries, "radon_forward_table: null pointer");
    DFX_REQUIRE(((uintptr_t)img_k % 16) == 0 && ((uintptr_t)sino % 16) == 0 && ((uintptr_t)entries % 8) == 0,
                "radon_forward_table: misaligned arrays");
    DFX_REQUIRE(n_angles >= 0 && n_angles <= 65535 && n_det > 0, "radon_forward_table: bad sizes");
    DFX_REQUIRE(kstride > 0 && kstride % CPL == 0 && kb >= 0 && kb <= kstride && cdiv(kstride, CPW) <= 65535,
                "radon_forward_table: kstride (%d) must be a positive multiple of %d and kb (%d) <= kstride",
                kstride, CPL, kb);
    DFX_REQUIRE(sld >= kstride && sld % CPL == 0, "radon_forward_table: sinogram row stride (%lld) must be a "
                "multiple of %d >= kstride", (long long)sld, CPL);
    if (n_angles == 0) return DFX_OK;
    dim3 grid((unsigned)cdiv(n_det, WARPS), (unsigned)n_angles, (unsigned)cdiv(kstride, CPW));
    const int2 *ent = reinterpret_cast<const int2 *>(entries);
    if constexpr (sizeof(IT) == 2)
        radon_forward_table_bf16<<<grid, 32 * WARPS, 0, (cudaStream_t)stream>>>(
            img_k, sino, sld, row_ptr, ent, angles, n_det, kstride, kb, scale);
    else
        radon_forward_table<ST><<<grid, 32 * WARPS, 0, (cudaStream_t)stream>>>(
            img_k, sino, sld, row_ptr, ent, angles, n_det, kstride, kb, scale);
    return launch_status("radon_forward_table");
}

template <int MODE, typename ST>
static int radon_backward_any(const ST *sino, int64_t sld, float *img_k, const float *geo, int n_angles, int nx,
                              int ny, int n_det, int kstride, int kb, int kernel, int n_taps, float *z_k,
                              const float *T_k, float inv_p, float lam, void *stream,
                              __nv_bfloat16 *xb = nullptr)
{
    int st = check_radon_args(sino, img_k, geo, n_angles, nx, ny, n_det, kstride, kb, kernel);
    if (st) return st;
    DFX_REQUIRE(sld >= kstride && sld % CPL == 0, "radon: sinogram row stride (%lld) must be a multiple of %d >= "
                "kstride", (long long)sld, CPL);
    DFX_REQUIRE(MODE == 0 || (z_k && T_k && ((uintptr_t)z_k % 16) == 0 && ((uintptr_t)T_k % 16) == 0),
                "radon_backward_spdhg: z and T must be 16-byte aligned device arrays");
    DFX_REQUIRE(n_taps >= 2 && n_taps <= 64, "radon: n_taps (%d) out of range", n_taps);
    if (kernel == 1)
        return launch_backward<1, MODE, ST>(sino, sld, img_k, geo, n_angles, nx, ny, n_det, kstride, kb, n_taps, z_k,
                                            T_k, inv_p, lam, xb, stream);
    return launch_backward<0, MODE, ST>(sino, sld, img_k, geo, n_angles, nx, ny, n_det, kstride, kb, n_taps, z_k, T_k,
                                        inv_p, lam, xb, stream);
}

extern "C" int dfx_radon_forward(const float *img_k, float *sino_k, const float *geo, int n_angles, int nx, int ny,
                                 int n_det, int kstride, int kb, int kernel, float scale, void *stream)
{
    return radon_forward_any(img_k, sino_k, (int64_t)kstride, geo, n_angles, nx, ny, n_det, kstride, kb, kernel,
                             scale, stream);
}

extern "C" int dfx_radon_forward_bf16(const float *img_k, void *sino_bf16, int64_t sino_ld, const float *geo,
                                      int n_angles, int nx, int ny, int n_det, int kstride, int kb, int kernel,
                                      float scale, void *stream)
{
    return radon_forward_any(img_k, reinterpret_cast<__nv_bfloat16 *>(sino_bf16), sino_ld, geo, n_angles, nx, ny,
                             n_det, kstride, kb, kernel, scale, stream);
}

extern "C" int dfx_radon_backward_pixels(const float *sino_k, float *img_k, const float *geo, int n_angles, int nx,
                                         int ny, int n_det, int kstride, int kb, int kernel, int n_taps,
                                         const int32_t *pixels, int64_t n_pix, void *stream)
{
    int st = check_radon_args(sino_k, img_k, geo, n_angles, nx, ny, n_det, kstride, kb, kernel);
    if (st) return st;
    DFX_REQUIRE(pixels && n_pix > 0 && n_pix <= (int64_t)nx * ny, "radon_backward_pixels: bad pixel list");
    DFX_REQUIRE(n_taps >= 2 && n_taps <= 64, "radon: n_taps (%d) out of range", n_taps);
    if (kernel == 1)
        return launch_backward<1, 0, float>(sino_k, (int64_t)kstride, img_k, geo, n_angles, nx, ny, n_det, kstride, kb,
                                            n_taps, nullptr, nullptr, 0.0f, 0.0f, nullptr, stream, pixels, n_pix);
    return launch_backward<0, 0, float>(sino_k, (int64_t)kstride, img_k, geo, n_angles, nx, ny, n_det, kstride, kb,
                                        n_taps, nullptr, nullptr, 0.0f, 0.0f, nullptr, stream, pixels, n_pix);
}

extern "C" int dfx_radon_backward(const float *sino_k, float *img_k, const float *geo, int n_angles, int nx, int ny,
                                  int n_det, int kstride, int kb, int kernel, int n_taps, void *stream)
{
    return radon_backward_any<0>(sino_k, (int64_t)kstride, img_k, geo, n_angles, nx, ny, n_det, kstride, kb, kernel,
                                 n_taps, nullptr, nullptr, 0.0f, 0.0f, stream);
}

extern "C" int dfx_radon_backward_bf16(const void *sino_bf16, int64_t sino_ld, float *img_k, const float *geo,
                                       int n_angles, int nx, int ny, int n_det, int kstride, int kb, int kernel,
                                       int n_taps, void *stream)
{
    return radon_backward_any<0>(reinterpret_cast<const __nv_bfloat16 *>(sino_bf16), sino_ld, img_k, geo, n_angles, nx,
                                 ny, n_det, kstride, kb, kernel, n_taps, nullptr, nullptr, 0.0f, 0.0f, stream);
}

extern "C" int dfx_radon_backward_spdhg(const float *sino_k, const float *geo, int n_angles, int nx, int ny, int n_det,
                                        int kstride, int kb, int kernel, int n_taps, float *x_k, float *z_k,
                                        const float *T_k, float inv_p, float lam, void *stream)
{
    return radon_backward_any<1>(sino_k, (int64_t)kstride, x_k, geo, n_angles, nx, ny, n_det, kstride, kb, kernel,
                                 n_taps, z_k, T_k, inv_p, lam, stream);
}

extern "C" int dfx_radon_backward_spdhg_bf16(const void *sino_bf16, int64_t sino_ld, const float *geo, int n_angles,
                                             int nx, int ny, int n_det, int kstride, int kb, int kernel, int n_taps,
                                             float *x_k, float *z_k, const float *T_k, float inv_p, float lam,
                                             void *x_bf16, void *stream)
{
    DFX_REQUIRE(((uintptr_t)x_bf16 % 16) == 0, "radon_backward_spdhg_bf16: x_bf16 must be 16-byte aligned");
    return radon_backward_any<1>(reinterpret_cast<const __nv_bfloat16 *>(sino_bf16), sino_ld, x_k, geo, n_angles, nx,
                                 ny, n_det, kstride, kb, kernel, n_taps, z_k, T_k, inv_p, lam, stream,
                                 reinterpret_cast<__nv_bfloat16 *>(x_bf16));
}

extern "C" int dfx_radon_table_count(const float *geo, int n_angles, int nx, int ny, int n_det, int kernel,
                                     const uint8_t *supp, int32_t *counts, void *stream)
{
    DFX_REQUIRE(geo && counts && ((uintptr_t)geo % 16) == 0, "radon_table: null or misaligned pointer");
    DFX_REQUIRE(n_angles > 0 && nx > 0 && ny > 0 && n_det > 0 && (kernel == 0 || kernel == 1),
                "radon_table: bad sizes or kernel");
    const int64_t rows = (int64_t)n_angles * n_det;
    DFX_REQUIRE(cdiv(rows, 128) < 2147483647LL, "radon_table: too many rows");
    if (kernel == 1)
        ray_table_kernel<1><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, counts, nullptr, nullptr);
    else
        ray_table_kernel<0><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, counts, nullptr, nullptr);
    return launch_status("radon_table_count");
}

extern "C" int dfx_radon_table_fill(const float *geo, int n_angles, int nx, int ny, int n_det, int kernel,
                                    const uint8_t *supp, const int32_t *row_ptr, int32_t *entries, void *stream)
{
    DFX_REQUIRE(geo && row_ptr && entries && ((uintptr_t)geo % 16) == 0 && ((uintptr_t)entries % 8) == 0,
                "radon_table: null or misaligned pointer");
    DFX_REQUIRE(n_angles > 0 && nx > 0 && ny > 0 && n_det > 0 && (kernel == 0 || kernel == 1),
                "radon_table: bad sizes or kernel");
    const int64_t rows = (int64_t)n_angles * n_det;
    int2 *e = reinterpret_cast<int2 *>(entries);
    if (kernel == 1)
        ray_table_kernel<1><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, nullptr, row_ptr, e);
    else
        ray_table_kernel<0><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, nullptr, row_ptr, e);
    return launch_status("radon_table_fill");
}

extern "C" int dfx_radon_gtable_count(const float *geo, int n_angles, int nx, int ny, int n_det, int kernel,
                                      const uint8_t *supp, int32_t *counts, void *stream)
{
    DFX_REQUIRE(geo && counts && ((uintptr_t)geo % 16) == 0, "radon_gtable: null or misaligned pointer");
    DFX_REQUIRE(n_angles > 0 && nx > 0 && ny > 0 && n_det > 0 && (kernel == 0 || kernel == 1),
                "radon_gtable: bad sizes or kernel");
    const int64_t rows = (int64_t)n_angles * cdiv(n_det, GB);
    DFX_REQUIRE(cdiv(rows, 128) < 2147483647LL, "radon_gtable: too many rows");
    if (kernel == 1)
        ray_gtable_kernel<1><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, counts, nullptr, nullptr, nullptr);
    else
        ray_gtable_kernel<0><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, counts, nullptr, nullptr, nullptr);
    return launch_status("radon_gtable_count");
}

extern "C" int dfx_radon_gtable_fill(const float *geo, int n_angles, int nx, int ny, int n_det, int kernel,
                                     const uint8_t *supp, const int32_t *row_ptr, int32_t *pixels, float *weights,
                                     void *stream)
{
    DFX_REQUIRE(geo && row_ptr && pixels && weights && ((uintptr_t)geo % 16) == 0 && ((uintptr_t)weights % 16) == 0,
                "radon_gtable: null or misaligned pointer");
    DFX_REQUIRE(n_angles > 0 && nx > 0 && ny > 0 && n_det > 0 && (kernel == 0 || kernel == 1),
                "radon_gtable: bad sizes or kernel");
    const int64_t rows = (int64_t)n_angles * cdiv(n_det, GB);
    float4 *w = reinterpret_cast<float4 *>(weights);
    if (kernel == 1)
        ray_gtable_kernel<1><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, nullptr, row_ptr, pixels, w);
    else
        ray_gtable_kernel<0><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, supp, nullptr, row_ptr, pixels, w);
    return launch_status("radon_gtable_fill");
}

template <typename ST>
static int radon_forward_gtable_any(const float *img_k, ST *sino, int64_t sld, const int32_t *row_ptr,
                                    const int32_t *pixels, const float *weights, const int32_t *angles, int n_angles,
                                    int n_det, int kstride, int kb, float scale, void *stream)
{
    DFX_REQUIRE(img_k && sino && row_ptr && pixels && weights, "radon_forward_gtable: null pointer");
    DFX_REQUIRE(((uintptr_t)img_k % 16) == 0 && ((uintptr_t)sino % 16) == 0 && ((uintptr_t)weights % 16) == 0,
                "radon_forward_gtable: misaligned arrays");
    DFX_REQUIRE(n_angles >= 0 && n_angles <= 65535 && n_det > 0, "radon_forward_gtable: bad sizes");
    DFX_REQUIRE(kstride > 0 && kstride % CPL == 0 && kb >= 0 && kb <= kstride && cdiv(kstride, CPW) <= 65535,
                "radon_forward_gtable: kstride (%d) must be a positive multiple of %d and kb (%d) <= kstride",
                kstride, CPL, kb);
    DFX_REQUIRE(sld >= kstride && sld % CPL == 0, "radon_forward_gtable: sinogram row stride (%lld) must be a "
                "multiple of %d >= kstride", (long long)sld, CPL);
    if (n_angles == 0) return DFX_OK;
    dim3 grid((unsigned)cdiv(cdiv(n_det, GB), WARPS / GA), (unsigned)cdiv(n_angles, GA), (unsigned)cdiv(kstride, CPW));
    radon_forward_gtable<ST><<<grid, 32 * WARPS, 0, (cudaStream_t)stream>>>(
        img_k, sino, sld, row_ptr, pixels, reinterpret_cast<const float4 *>(weights), angles, n_angles, n_det, kstride,
        kb, scale);
    return launch_status("radon_forward_gtable");
}

extern "C" int dfx_radon_forward_gtable(const float *img_k, float *sino_k, const int32_t *row_ptr,
                                        const int32_t *pixels, const float *weights, const int32_t *angles,
                                        int n_angles, int n_det, int kstride, int kb, float scale, void *stream)
{
    return radon_forward_gtable_any(img_k, sino_k, (int64_t)kstride, row_ptr, pixels, weights, angles, n_angles, n_det,
                                    kstride, kb, scale, stream);
}

extern "C" int dfx_radon_forward_gtable_bf16(const float *img_k, void *sino_bf16, int64_t sino_ld,
                                             const int32_t *row_ptr, const int32_t *pixels, const float *weights,
                                             const int32_t *angles, int n_angles, int n_det, int kstride, int kb,
                                             float scale, void *stream)
{
    return radon_forward_gtable_any(img_k, reinterpret_cast<__nv_bfloat16 *>(sino_bf16), sino_ld, row_ptr, pixels,
                                    weights, angles, n_angles, n_det, kstride, kb, scale, stream);
}

extern "C" int dfx_radon_dtable_fill(const float *geo, int n_angles, int nx, int ny, int n_det, int kernel,
                                     const int32_t *row_ptr, int32_t *entries, void *stream)
{
    DFX_REQUIRE(geo && row_ptr && entries && ((uintptr_t)geo % 16) == 0 && ((uintptr_t)entries % 8) == 0,
                "radon_dtable: null or misaligned pointer");
    DFX_REQUIRE(n_angles > 0 && nx > 0 && ny > 0 && n_det > 0 && (kernel == 0 || kernel == 1),
                "radon_dtable: bad sizes or kernel");
    const int64_t rows = (int64_t)n_angles * n_det;
    int2 *e = reinterpret_cast<int2 *>(entries);
    if (kernel == 1)
        ray_table_kernel<1, true><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, nullptr, nullptr, row_ptr, e);
    else
        ray_table_kernel<0, true><<<(unsigned)cdiv(rows, 128), 128, 0, (cudaStream_t)stream>>>(
            reinterpret_cast<const float4 *>(geo), n_angles, nx, ny, n_det, nullptr, nullptr, row_ptr, e);
    return launch_status("radon_dtable_fill");
}

extern "C" int dfx_radon_forward_table(const float *img_k, float *sino_k, const int32_t *row_ptr,
                                       const int32_t *entries, const int32_t *angles, int n_angles, int n_det,
                                       int kstride, int kb, float scale, void *stream)
{
    return radon_forward_table_any(img_k, sino_k, (int64_t)kstride, row_ptr, entries, angles, n_angles, n_det,
                                   kstride, kb, scale, stream);
}

extern "C" int dfx_radon_forward_table_bf16(const float *img_k, void *sino_bf16, int64_t sino_ld,
                                            const int32_t *row_ptr, const int32_t *entries, const int32_t *angles,
                                            int n_angles, int n_det, int kstride, int kb, float scale, void *stream)
{
    return radon_forward_table_any(img_k, reinterpret_cast<__nv_bfloat16 *>(sino_bf16), sino_ld, row_ptr, entries,
                                   angles, n_angles, n_det, kstride, kb, scale, stream);
}

extern "C" int dfx_radon_forward_table_bf16_bf16(const void *img_bf16, void *sino_bf16, int64_t sino_ld,
                                                 const int32_t *row_ptr, const int32_t *entries, const int32_t *angles,
                                                 int n_angles, int n_det, int kstride, int kb, float scale, void *stream)
{
    return radon_forward_table_any(reinterpret_cast<const __nv_bfloat16 *>(img_bf16),
                                   reinterpret_cast<__nv_bfloat16 *>(sino_bf16), sino_ld, row_ptr, entries, angles,
                                   n_angles, n_det, kstride, kb, scale, stream);
}

extern "C" int dfx_batch_support(float *x_k, const float *colsum_k, const uint8_t *supp, int64_t npix, int kstride,
                                 int kb, float c, int mode, void *stream)
{
    DFX_REQUIRE(x_k && npix > 0 && kstride > 0 && kb >= 0 && kb <= kstride && mode >= 0 && mode <= 3,
                "batch_support: bad arguments");
    DFX_REQUIRE(mode != 2 || colsum_k, "batch_support: tmin needs the column sums");
    const bool vec = kstride % 4 == 0 && (uintptr_t)x_k % 16 == 0 && (mode != 2 || (uintptr_t)colsum_k % 16 == 0);
    const int64_t n = npix * (vec ? kstride / 4 : kstride), blocks = cdiv(n, 256);
    const bool small = n < ((int64_t)1 << 31);
    const auto kernel = vec ? (small ? batch_support_kernel<4, uint32_t> : batch_support_kernel<4, int64_t>)
                            : (small ? batch_support_kernel<1, uint32_t> : batch_support_kernel<1, int64_t>);
    kernel<<<(unsigned)(blocks < 148 * 32 ? blocks : 148 * 32), 256, 0, (cudaStream_t)stream>>>(
        x_k, colsum_k, supp, npix, kstride, kb, c, mode);
    return launch_status("batch_support");
}

extern "C" int dfx_gather_channels(const float *coeffs, float *img_k, int64_t npix, int k0, int kb, int kstride,
                                   void *stream)
{
    DFX_REQUIRE(coeffs && img_k, "gather: null pointer");
    DFX_REQUIRE(npix > 0 && k0 >= 0 && kb >= 0 && kb <= kstride, "gather: bad sizes");
    return launch_transpose(coeffs + (int64_t)k0 * npix, npix, 0, nullptr, 0, img_k, kstride, 0, kb, kstride, npix, 1,
                            (cudaStream_t)stream);
}

extern "C" int dfx_scatter_channels(const float *img_k, float *coeffs, int64_t npix, int k0, int kb, int kstride,
                                    void *stream)
{
    DFX_REQUIRE(coeffs && img_k, "scatter: null pointer");
    DFX_REQUIRE(npix > 0 && k0 >= 0 && kb >= 0 && kb <= kstride, "scatter: bad sizes");
    if (kb == 0) return DFX_OK;
    return launch_transpose(img_k, kstride, 0, nullptr, 0, coeffs + (int64_t)k0 * npix, npix, 0, npix, npix, kb, 1,
                            (cudaStream_t)stream);
}
