// Copies of dense-layer operands whose rows no tensor map can address (row lengths or bases that are no multiples of 16
// bytes), or that lie transposed, into rows that it can: out[r][c] = src[r][c], or src[c][r], with a 16-byte row pitch.
// HBM-bound, one pass. The copy buys the tensor-core (16-bit) or TMA-fed FMA kernel (fp32): at 2 x 731 x 5280 fp16 it costs
// 5 us where the scalar-load kernel took 52 us for the whole layer.
#include "common.cuh"

namespace xg {
namespace {

// One 16-byte vector of a row per thread, put together from the (naturally aligned) elements.
__global__ void __launch_bounds__(256) pad_rows32_kernel(const uint32_t* __restrict__ src, int64_t rows, int64_t cols, int64_t ld,
                                                         uint32_t* __restrict__ out, int64_t out_ld) {
    pdl_sync();
    const int64_t vecs = out_ld / 4, total = rows * vecs;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const int64_t r = i / vecs, c = (i - r * vecs) * 4;
        const uint32_t* s = src + r * ld + c;
        uint4 v;
        v.x = c < cols ? s[0] : 0u;
        v.y = c + 1 < cols ? s[1] : 0u;
        v.z = c + 2 < cols ? s[2] : 0u;
        v.w = c + 3 < cols ? s[3] : 0u;
        *reinterpret_cast<uint4*>(out + r * out_ld + c) = v;
    }
}

// 16-bit elements: five aligned words hold the eight elements of a vector wherever the row starts.
__global__ void __launch_bounds__(256) pad_rows16_kernel(const uint16_t* __restrict__ src, int64_t rows, int64_t cols, int64_t ld,
                                                         uint16_t* __restrict__ out, int64_t out_ld) {
    pdl_sync();
    const int64_t vecs = out_ld / 8, total = rows * vecs;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const int64_t r = i / vecs, c = (i - r * vecs) * 8;
        const uint16_t* s = src + r * ld + c;
        const int n = (int)(cols - c < 8 ? cols - c : 8);  // elements of this vector inside the row (<= 0: padding only)
        const unsigned odd = (unsigned)(reinterpret_cast<uintptr_t>(s) >> 1) & 1u;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(s - odd);
        uint32_t x[5], v[4];
#pragma unroll
        for (int k = 0; k < 5; ++k) x[k] = 2 * k < n + (int)odd ? w[k] : 0u;  // only words with an element of the row
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = __funnelshift_r(x[k], x[k + 1], odd * 16);
            if (2 * k + 1 >= n) v[k] &= 2 * k < n ? 0xffffu : 0u;
        }
        *reinterpret_cast<uint4*>(out + r * out_ld + c) = make_uint4(v[0], v[1], v[2], v[3]);
    }
}

// out[r][c] = src[c][r] through a 32 x 32 tile of shared memory; 256 threads as 8 rows of 32. One grid dimension: the second one
// ends at 65535 tiles, which 2,097,120 columns fill.
template <typename U>
__global__ void __launch_bounds__(256) pad_transpose_kernel(const U* __restrict__ src, int64_t rows, int64_t cols, int64_t ld,
                                                            U* __restrict__ out, int64_t out_ld, unsigned row_tiles) {
    pdl_sync();
    __shared__ U tile[32][33];
    const int64_t r0 = (int64_t)(blockIdx.x % row_tiles) * 32, c0 = (int64_t)(blockIdx.x / row_tiles) * 32;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 32; k += 8)
        if (c0 + y + k < cols && r0 + x < rows) tile[y + k][x] = src[(c0 + y + k) * ld + r0 + x];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 32; k += 8)
        if (r0 + y + k < rows && c0 + x < out_ld) out[(r0 + y + k) * out_ld + c0 + x] = c0 + x < cols ? tile[x][y + k] : U(0);
}

}  // namespace
}  // namespace xg

extern "C" int xg_pad_rows(const void* src, int64_t rows, int64_t cols, int64_t ld, int transpose, void* out, int64_t out_ld,
                           int elem_size, void* stream) {
    using namespace xg;
    if (!src || !out) return fail(XG_ERR_INVALID_ARG, "xg_pad_rows: null pointer");
    if (elem_size != 2 && elem_size != 4) return fail(XG_ERR_INVALID_ARG, "xg_pad_rows: element size %d", elem_size);
    if (rows < 0 || cols <= 0 || ld < (transpose ? rows : cols) || out_ld < cols || out_ld % (16 / elem_size) != 0 || !aligned16(out) ||
        reinterpret_cast<uintptr_t>(src) % (uintptr_t)elem_size != 0)
        return fail(XG_ERR_INVALID_ARG, "xg_pad_rows: bad extents, strides or alignment");
    if (rows == 0) return XG_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (transpose) {
        const int64_t gx = (rows + 31) / 32, gy = (out_ld + 31) / 32;
        if (gx > 0x7fffffffLL / gy) return fail(XG_ERR_TOO_LARGE, "xg_pad_rows: extent too large");
        const unsigned grid = (unsigned)(gx * gy);
        if (elem_size == 4)
            launch(pad_transpose_kernel<uint32_t>, grid, 256, 0, st, reinterpret_cast<const uint32_t*>(src), rows, cols, ld,
                   reinterpret_cast<uint32_t*>(out), out_ld, (unsigned)gx);
        else
            launch(pad_transpose_kernel<uint16_t>, grid, 256, 0, st, reinterpret_cast<const uint16_t*>(src), rows, cols, ld,
                   reinterpret_cast<uint16_t*>(out), out_ld, (unsigned)gx);
    } else {
        const int64_t blocks = (rows * (out_ld * elem_size / 16) + 255) / 256, cap = 16LL * num_sms();
        const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
        if (elem_size == 4)
            launch(pad_rows32_kernel, grid, 256, 0, st, reinterpret_cast<const uint32_t*>(src), rows, cols, ld, reinterpret_cast<uint32_t*>(out), out_ld);
        else
            launch(pad_rows16_kernel, grid, 256, 0, st, reinterpret_cast<const uint16_t*>(src), rows, cols, ld, reinterpret_cast<uint16_t*>(out), out_ld);
    }
    return check_launch("xg_pad_rows");
}
