// Transposes of float32 matrices between the layouts of the kernels (channels, detector lines or pixels fastest).
#pragma once
#include "dfx_common.cuh"

namespace dfx {

// out[c out_ld + r] = r < rows ? in[r in_ld + c] : 0 for c < cols, r < rows_out, for each of the matrices blockIdx.y: in
// at in + m in_m (m = list[blockIdx.y], or m0 + blockIdx.y), out at out + blockIdx.y out_m. A lane transposes 4 x 4
// elements in registers: four 16-byte loads along c, four 16-byte stores along r. The warp's 32 rows x 16 columns
// read 64 contiguous bytes per row and write 128 per column; no shared memory, no synchronisation, and 64 bytes per
// lane in flight. VI: the loads may be vectors (alignment); otherwise element by element. The output's columns are
// 16-byte aligned. HBM bounds it: 0.53 GB in and out 0.19 -> 0.09 ms against transpose_tile_kernel.
template <bool VI>
__global__ void __launch_bounds__(256) transpose_kernel(const float *__restrict__ in, int64_t in_ld, int64_t in_m,
                                                        const int32_t *__restrict__ list, int m0, float *__restrict__ out,
                                                        int64_t out_ld, int64_t out_m, int64_t rows, int64_t rows_out,
                                                        int64_t cols, int col_tiles)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tile = blockIdx.x;
    const int64_t c = (tile % col_tiles) * 128 + warp * 16 + (lane >> 3) * 4;
    const int64_t r = (tile / col_tiles) * 32 + (lane & 7) * 4;
    if (c >= cols || r >= rows_out) return;
    in += (list ? __ldg(list + blockIdx.y) : m0 + (int)blockIdx.y) * in_m + c;
    out += blockIdx.y * out_m + r;
    float v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float *p = in + (r + i) * in_ld;
        if (VI && c + 4 <= cols) {
            const float4 q = r + i < rows ? __ldg(reinterpret_cast<const float4 *>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][0] = q.x;
            v[i][1] = q.y;
            v[i][2] = q.z;
            v[i][3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = r + i < rows && c + j < cols ? __ldg(p + j) : 0.0f;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (c + j >= cols) break;
        float *p = out + (c + j) * out_ld;
        if (r + 4 <= rows_out) {
            *reinterpret_cast<float4 *>(p) = make_float4(v[0][j], v[1][j], v[2][j], v[3][j]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (r + i < rows_out) p[i] = v[i][j];
        }
    }
}

// The same for outputs whose columns are not 16-byte aligned (images of an odd number of pixels): a 32 x 32 tile through
// shared memory, 128 contiguous bytes per warp on both sides. transpose_kernel's stores would be single words 16 bytes
// apart: 9801 pixels, 1000 channels 29 us, so 21; 130 channels 10.6 and 6.5.
static __global__ void __launch_bounds__(256) transpose_tile_kernel(
    const float *__restrict__ in, int64_t in_ld, int64_t in_m, const int32_t *__restrict__ list, int m0,
    float *__restrict__ out, int64_t out_ld, int64_t out_m, int64_t rows, int64_t rows_out, int64_t cols, int row_tiles)
{
    __shared__ float tile[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t r0 = (int64_t)(blockIdx.x % row_tiles) * 32, c0 = (int64_t)(blockIdx.x / row_tiles) * 32;
    in += (list ? __ldg(list + blockIdx.y) : m0 + (int)blockIdx.y) * in_m;
    out += blockIdx.y * out_m;
    const bool cin = c0 + lane < cols, rout = r0 + lane < rows_out;
    in += (r0 + warp) * in_ld + c0 + lane;
    out += (c0 + warp) * out_ld + r0 + lane;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = cin && r0 + warp + 8 * i < rows ? __ldg(in + 8 * i * in_ld) : 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) tile[warp + 8 * i][lane] = v[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (rout && c0 + warp + 8 * i < cols) out[8 * i * out_ld] = tile[lane][warp + 8 * i];
}

inline int launch_transpose(const float *in, int64_t in_ld, int64_t in_m, const int32_t *list, int m0, float *out,
                            int64_t out_ld, int64_t out_m, int64_t rows, int64_t rows_out, int64_t cols, int n,
                            cudaStream_t st)
{
    const bool vo = (uintptr_t)out % 16 == 0 && out_ld % 4 == 0 && out_m % 4 == 0;
    const int64_t rt = cdiv(rows_out, 32), ct = cdiv(cols, vo ? 128 : 32);
    DFX_REQUIRE(rt * ct < 2147483647LL && n <= 65535, "transpose: too large for one launch");
    const dim3 grid((unsigned)(rt * ct), (unsigned)n);
    if (!vo) {
        transpose_tile_kernel<<<grid, 256, 0, st>>>(in, in_ld, in_m, list, m0, out, out_ld, out_m, rows, rows_out, cols,
                                                    (int)rt);
        return launch_status("transpose");
    }
    const bool vi = (uintptr_t)in % 16 == 0 && in_ld % 4 == 0 && in_m % 4 == 0;
    const auto kernel = vi ? transpose_kernel<true> : transpose_kernel<false>;
    kernel<<<grid, 256, 0, st>>>(in, in_ld, in_m, list, m0, out, out_ld, out_m, rows, rows_out, cols, (int)ct);
    return launch_status("transpose");
}

}  // namespace dfx
