// Bit-exact copy fusions: segmented 2-D copy (slice+cat, multi-slice, split, cat/stack, optional
// row mask) and multi-table row gather (embedding lookups fused with where-mask and stack).
//
// Both are single-pass and HBM-bound: every useful byte is read once and written once, in the
// widest unit (up to 16 bytes) that the pointers, strides and lengths allow. The column -> segment
// map is a small look-up table built in shared memory from the segment list, so consecutive
// threads write consecutive output units (coalesced stores; loads are coalesced within a segment).
#include "common.cuh"

namespace xg {
namespace {

constexpr int kMaxSegs = 64;     // segments per launch (kernel parameter space)
constexpr int kLutMax = 8192;    // output units per row per launch (at most 32 KiB of shared memory)
constexpr int kCopyThreads = 256;
constexpr int kCopyUnroll = 4;
constexpr int kGatherRows = 8;    // rows per CTA in the gather kernel

struct SegDesc {
    const char* src;
    char* dst;
    int64_t src_ld;  // bytes
    int64_t dst_ld;  // bytes
    int32_t units;
    int32_t unit_start;
};

struct SegCopyParams {
    SegDesc seg[kMaxSegs];
    int32_t nseg;
    int32_t width;  // total units per row in this launch
    int32_t rows_per_cta;
    int32_t zero_when;
    int64_t rows;
    const uint8_t* mask;
};

template <typename U>
__device__ __forceinline__ U zero_unit() {
    U z;
    memset(&z, 0, sizeof(U));
    return z;
}

template <typename U>
__global__ void __launch_bounds__(kCopyThreads) seg_copy_kernel(const __grid_constant__ SegCopyParams p) {
    pdl_sync();
    __shared__ SegDesc segs[kMaxSegs];
    extern __shared__ uint32_t lut[];  // [width]: no more than the launch needs, so that eight CTAs fit an SM
    for (int k = threadIdx.x; k < p.nseg; k += kCopyThreads) segs[k] = p.seg[k];
    __syncthreads();
    // a thread looks its columns' segments up by bisection: one step of latency per doubling of the segments instead of one
    // per segment (a CTA lives for a few microseconds, and with a pass per segment the table took most of them)
    for (int c = threadIdx.x; c < p.width; c += kCopyThreads) {
        int k = 0;
        for (int step = kMaxSegs / 2; step > 0; step >>= 1)
            if (k + step < p.nseg && segs[k + step].unit_start <= c) k += step;
        lut[c] = ((uint32_t)k << 24) | (uint32_t)(c - segs[k].unit_start);
    }
    __syncthreads();

    const int64_t r0 = (int64_t)blockIdx.x * p.rows_per_cta;
    const int64_t left = p.rows - r0;
    const int nrows = (int)(left < p.rows_per_cta ? left : p.rows_per_cta);
    const int W = p.width;
    if (W >= 128) {
        // wide rows: walk the columns with stride 256 and take the same column of several rows at once
        // (no index division; 64 bytes of loads in flight per thread: 4 rows of 16-byte units, 8 of narrower ones)
        constexpr int kRowsAtOnce = sizeof(U) >= 16 ? kCopyUnroll : 2 * kCopyUnroll;
        for (int rb = 0; rb < nrows; rb += kRowsAtOnce) {
            for (int c = threadIdx.x; c < W; c += kCopyThreads) {
                const uint32_t e = lut[c];
                const SegDesc& sd = segs[e >> 24];
                const int64_t j = (int64_t)(e & 0xffffffu) * sizeof(U);
                U v[kRowsAtOnce];
#pragma unroll
                for (int k = 0; k < kRowsAtOnce; ++k) {
                    if (rb + k < nrows) {
                        const int64_t row = r0 + rb + k;
                        bool zero = false;
                        if (p.mask != nullptr) zero = ((p.mask[row] != 0) == (p.zero_when != 0));
                        v[k] = zero ? zero_unit<U>() : *reinterpret_cast<const U*>(sd.src + row * sd.src_ld + j);
                    }
                }
#pragma unroll
                for (int k = 0; k < kRowsAtOnce; ++k) {
                    if (rb + k < nrows) *reinterpret_cast<U*>(sd.dst + (r0 + rb + k) * sd.dst_ld + j) = v[k];
                }
            }
        }
        return;
    }
    const int total = nrows * W;  // host keeps rows_per_cta * width below 2^31
    for (int i0 = threadIdx.x; i0 < total; i0 += kCopyThreads * kCopyUnroll) {
        U v[kCopyUnroll];
        U* d[kCopyUnroll];
#pragma unroll
        for (int k = 0; k < kCopyUnroll; ++k) {
            const int i = i0 + k * kCopyThreads;
            if (i < total) {
                const int r = i / W;
                const int c = i - r * W;
                const uint32_t e = lut[c];
                const SegDesc& sd = segs[e >> 24];
                const int64_t j = (int64_t)(e & 0xffffffu) * sizeof(U);
                const int64_t row = r0 + r;
                bool zero = false;
                if (p.mask != nullptr) zero = ((p.mask[row] != 0) == (p.zero_when != 0));
                d[k] = reinterpret_cast<U*>(sd.dst + row * sd.dst_ld + j);
                v[k] = zero ? zero_unit<U>() : *reinterpret_cast<const U*>(sd.src + row * sd.src_ld + j);
            }
        }
#pragma unroll
        for (int k = 0; k < kCopyUnroll; ++k) {
            const int i = i0 + k * kCopyThreads;
            if (i < total) *d[k] = v[k];
        }
    }
}

template <typename U>
int launch_seg_copy(const SegCopyParams& p, cudaStream_t st) {
    const int64_t grid = (p.rows + p.rows_per_cta - 1) / p.rows_per_cta;
    if (grid > 0x7fffffffLL) return fail(XG_ERR_TOO_LARGE, "xg_seg_copy: too many row tiles");
    launch(seg_copy_kernel<U>, (unsigned)grid, kCopyThreads, (size_t)p.width * sizeof(uint32_t), st, p);
    return check_launch("xg_seg_copy");
}

int dispatch_seg_copy(int unit, const SegCopyParams& p, cudaStream_t st) {
    switch (unit) {
        case 16: return launch_seg_copy<uint4>(p, st);
        case 8: return launch_seg_copy<uint2>(p, st);
        case 4: return launch_seg_copy<uint32_t>(p, st);
        case 2: return launch_seg_copy<uint16_t>(p, st);
        default: return launch_seg_copy<uint8_t>(p, st);
    }
}

inline int pow2_align(uint64_t v) {  // largest power of two <= 16 dividing v (16 for v == 0)
    int a = 16;
    while (a > 1 && (v % (uint64_t)a) != 0) a >>= 1;
    return a;
}

// ---------------------------------------------------------------------------------------
// multi-table gather
// ---------------------------------------------------------------------------------------
struct GatherParams {
    const char* table[kMaxSegs];
    int64_t table_rows[kMaxSegs];
    int32_t F;
    int32_t f0;             // first field of this launch (offset into idx columns / out columns)
    int32_t units_per_row;  // D * elem_size / sizeof(U)
    int32_t zero_when;
    int64_t rows;
    int64_t row_bytes;  // D * elem_size
    const int64_t* idx;
    int64_t idx_rs, idx_cs;
    const uint8_t* mask;
    char* out;
    int64_t out_ld_bytes;
};

template <typename U>
__global__ void __launch_bounds__(kCopyThreads) gather_rows_kernel(const __grid_constant__ GatherParams p) {
    pdl_sync();
    __shared__ const char* tab[kMaxSegs];
    __shared__ int64_t trows[kMaxSegs];
    for (int k = threadIdx.x; k < p.F; k += kCopyThreads) {
        tab[k] = p.table[k];
        trows[k] = p.table_rows[k];
    }
    __syncthreads();
    // One CTA owns kGatherRows consecutive rows; a thread walks the (field, unit) columns of a row with stride 256
    // and takes the same column of 4 rows at once: 4 index loads, then 4 table loads in flight, 32-bit index math.
    const int upr = p.units_per_row;
    const int per_row = p.F * upr;
    const int64_t r0 = (int64_t)blockIdx.x * kGatherRows;
    for (int rb = 0; rb < kGatherRows; rb += kCopyUnroll) {
        for (int c = threadIdx.x; c < per_row; c += kCopyThreads) {
            const int f = c / upr;
            const int u = c - f * upr;
            int64_t ix[kCopyUnroll];
#pragma unroll
            for (int k = 0; k < kCopyUnroll; ++k) {
                const int64_t r = r0 + rb + k;
                ix[k] = (r < p.rows) ? p.idx[r * p.idx_rs + (int64_t)(p.f0 + f) * p.idx_cs] : -1;
            }
            U v[kCopyUnroll];
#pragma unroll
            for (int k = 0; k < kCopyUnroll; ++k) {
                const int64_t r = r0 + rb + k;
                bool zero = (ix[k] < 0) || (ix[k] >= trows[f]);
                if (r < p.rows && p.mask != nullptr) zero = zero || ((p.mask[r] != 0) == (p.zero_when != 0));
                v[k] = zero ? zero_unit<U>() : reinterpret_cast<const U*>(tab[f] + ix[k] * p.row_bytes)[u];
            }
#pragma unroll
            for (int k = 0; k < kCopyUnroll; ++k) {
                const int64_t r = r0 + rb + k;
                if (r < p.rows)
                    reinterpret_cast<U*>(p.out + r * p.out_ld_bytes + (int64_t)(p.f0 + f) * p.row_bytes)[u] = v[k];
            }
        }
    }
}

template <typename U>
int launch_gather(const GatherParams& p, cudaStream_t st) {
    const int64_t grid = (p.rows + kGatherRows - 1) / kGatherRows;
    if (grid > 0x7fffffffLL) return fail(XG_ERR_TOO_LARGE, "xg_gather_rows: too many tiles");
    launch(gather_rows_kernel<U>, (unsigned)grid, kCopyThreads, 0, st, p);
    return check_launch("xg_gather_rows");
}

// ---------------------------------------------------------------------------------------
// slices and lookups side by side, as the three bf16 planes that the fp32 tensor-core layers read
// ---------------------------------------------------------------------------------------
// out3[r][s * Kp + k], s = 0..2: columns 0..K-1 are the slices of src's row r, then the rows idx[r][f] of the tables (zeros
// where the mask hides the row or the index is outside its table), columns up to Kp are zero. A unit is four columns of one
// row; a thread takes the same unit of four rows (four index loads, then four 16-byte loads in flight). HBM-bound: reading the
// tables and writing 6 bytes per column is all the traffic. As separate copies, a gather and a split the fp32 matrix was
// written and read twice: 16384 rows of 64 + 26 x 64 took 152 us, 1.7 KB of reads and 10.4 KB of writes per row.
constexpr int kPlaneRows = 4;
constexpr int kPlaneMaxSliceUnits = 1024;
struct PlanesParams {
    const float* table[kMaxSegs];
    int32_t table_rows[kMaxSegs];
    int32_t start[kMaxSegs];       // slices: first unit in the source row ...
    int32_t unit_start[kMaxSegs];  // ... and in the output row
    const float* src;
    const int64_t* idx;
    const uint8_t* mask;
    __nv_bfloat16* out3;
    int64_t rows, src_ld, idx_rs, idx_cs, Kp;
    int32_t nslices, slice_units, F, units_per_lookup, zero_when;
};
static_assert(sizeof(PlanesParams) <= 4096, "kernel parameter space");

__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c) {
    a = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(a);
    b = __float2bfloat16_rn(r1);
    c = __float2bfloat16_rn(r1 - __bfloat162float(b));
}

__global__ void __launch_bounds__(kCopyThreads) gather_planes_kernel(const __grid_constant__ PlanesParams p) {
    pdl_sync();
    __shared__ const float* tab[kMaxSegs];
    __shared__ int trows[kMaxSegs];
    __shared__ int src_unit[kPlaneMaxSliceUnits];
    for (int f = threadIdx.x; f < p.F; f += blockDim.x) {
        tab[f] = p.table[f];
        trows[f] = p.table_rows[f];
    }
    for (int c = threadIdx.x; c < p.slice_units; c += blockDim.x) {
        int k = 0;
        for (int step = kMaxSegs / 2; step > 0; step >>= 1)
            if (k + step < p.nslices && p.unit_start[k + step] <= c) k += step;
        src_unit[c] = p.start[k] + c - p.unit_start[k];
    }
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x * kPlaneRows;
    const int units = (int)(p.Kp / 4), used = p.slice_units + p.F * p.units_per_lookup;
    bool hidden[kPlaneRows];
#pragma unroll
    for (int k = 0; k < kPlaneRows; ++k)
        hidden[k] = r0 + k >= p.rows || (p.mask != nullptr && ((p.mask[r0 + k] != 0) == (p.zero_when != 0)));
    for (int c = threadIdx.x; c < units; c += blockDim.x) {
        float4 v[kPlaneRows];
#pragma unroll
        for (int k = 0; k < kPlaneRows; ++k) v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < p.slice_units) {
            const float* s = p.src + 4 * (int64_t)src_unit[c];
#pragma unroll
            for (int k = 0; k < kPlaneRows; ++k)
                if (r0 + k < p.rows) v[k] = *reinterpret_cast<const float4*>(s + (r0 + k) * p.src_ld);
        } else if (c < used) {
            const int f = (c - p.slice_units) / p.units_per_lookup, u = c - p.slice_units - f * p.units_per_lookup;
            int64_t ix[kPlaneRows];
#pragma unroll
            for (int k = 0; k < kPlaneRows; ++k) ix[k] = hidden[k] ? -1 : p.idx[(r0 + k) * p.idx_rs + f * p.idx_cs];
#pragma unroll
            for (int k = 0; k < kPlaneRows; ++k)
                if (ix[k] >= 0 && ix[k] < trows[f])
                    v[k] = reinterpret_cast<const float4*>(tab[f])[ix[k] * p.units_per_lookup + u];
        }
#pragma unroll
        for (int k = 0; k < kPlaneRows; ++k) {
            if (r0 + k >= p.rows) break;
            const float x[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
            __align__(8) __nv_bfloat16 q[3][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) split3(x[i], q[0][i], q[1][i], q[2][i]);
            __nv_bfloat16* o = p.out3 + (r0 + k) * (3 * p.Kp) + 4 * c;
#pragma unroll
            for (int s = 0; s < 3; ++s) *reinterpret_cast<uint2*>(o + s * p.Kp) = *reinterpret_cast<const uint2*>(q[s]);
        }
    }
}

}  // namespace
}  // namespace xg

extern "C" int xg_gather_planes(const void* src, int64_t src_ld, const int64_t* starts, const int64_t* lens, int64_t nslices,
                                const void* const* tables, const int64_t* table_rows, int64_t F, const int64_t* idx,
                                int64_t idx_row_stride, int64_t idx_col_stride, const uint8_t* row_mask, int mask_zero_when,
                                void* out3, int64_t rows, int64_t D, void* stream) {
    using namespace xg;
    if (rows < 0 || nslices < 0 || F < 0 || D < 0) return fail(XG_ERR_INVALID_ARG, "xg_gather_planes: negative extent");
    if (rows == 0) return XG_OK;
    if (!out3 || (nslices > 0 && (!src || !starts || !lens)) || (F > 0 && (!tables || !table_rows || !idx)))
        return fail(XG_ERR_INVALID_ARG, "xg_gather_planes: null pointer");
    if (nslices > kMaxSegs || F > kMaxSegs) return fail(XG_ERR_UNSUPPORTED, "xg_gather_planes: more than %d slices or tables", kMaxSegs);
    if (D % 4 != 0 || !aligned16(src) || src_ld % 4 != 0 || !aligned16(out3))
        return fail(XG_ERR_UNSUPPORTED, "xg_gather_planes: rows must be 16-byte addressable");
    PlanesParams p;
    int64_t units = 0;
    p.nslices = 0;
    for (int64_t k = 0; k < nslices; ++k) {
        if (starts[k] < 0 || lens[k] < 0 || (rows > 1 && starts[k] + lens[k] > src_ld))
            return fail(XG_ERR_INVALID_ARG, "xg_gather_planes: slice %lld is outside its row", (long long)k);
        if (starts[k] % 4 != 0 || lens[k] % 4 != 0 || starts[k] > 0x7fffffffLL || units + lens[k] / 4 > kPlaneMaxSliceUnits)
            return fail(XG_ERR_UNSUPPORTED, "xg_gather_planes: slices must be whole units of four columns, %d units at most", kPlaneMaxSliceUnits);
        if (lens[k] == 0) continue;
        p.start[p.nslices] = (int32_t)(starts[k] / 4);
        p.unit_start[p.nslices++] = (int32_t)units;
        units += lens[k] / 4;
    }
    for (int64_t f = 0; f < F; ++f) {
        if (!tables[f] || table_rows[f] < 0) return fail(XG_ERR_INVALID_ARG, "xg_gather_planes: bad table %lld", (long long)f);
        if (!aligned16(tables[f]) || table_rows[f] > 0x7fffffffLL) return fail(XG_ERR_UNSUPPORTED, "xg_gather_planes: table %lld", (long long)f);
        p.table[f] = reinterpret_cast<const float*>(tables[f]);
        p.table_rows[f] = (int32_t)table_rows[f];
    }
    const int64_t K = 4 * units + F * D;
    if (K == 0) return XG_OK;
    if (D > 0x1000000LL) return fail(XG_ERR_TOO_LARGE, "xg_gather_planes: row too wide");
    p.src = reinterpret_cast<const float*>(src);
    p.src_ld = src_ld;
    p.idx = idx;
    p.idx_rs = idx_row_stride;
    p.idx_cs = idx_col_stride;
    p.mask = row_mask;
    p.zero_when = mask_zero_when;
    p.out3 = reinterpret_cast<__nv_bfloat16*>(out3);
    p.rows = rows;
    p.Kp = xg_gemm_f32x3_padded_k(K);
    p.slice_units = (int32_t)units;
    p.F = D > 0 ? (int32_t)F : 0;
    p.units_per_lookup = D > 0 ? (int32_t)(D / 4) : 1;
    const int64_t grid = (rows + kPlaneRows - 1) / kPlaneRows;
    if (grid > 0x7fffffffLL) return fail(XG_ERR_TOO_LARGE, "xg_gather_planes: too many rows");
    // a row's units in equal steps: 432 of them are two steps of 216 threads (224), not one and a half of 256
    const int64_t steps = (p.Kp / 4 + kCopyThreads - 1) / kCopyThreads;
    const unsigned threads = (unsigned)(((p.Kp / 4 + steps - 1) / steps + 31) / 32 * 32);
    launch(gather_planes_kernel, (unsigned)grid, threads, 0, reinterpret_cast<cudaStream_t>(stream), p);
    return check_launch("xg_gather_planes");
}

extern "C" int xg_seg_copy(const void* const* src_ptrs, void* const* dst_ptrs, const int64_t* src_ld_bytes,
                           const int64_t* dst_ld_bytes, const int64_t* len_bytes, int64_t nseg, int64_t rows,
                           const uint8_t* row_mask, int mask_zero_when, void* stream) {
    using namespace xg;
    if (nseg < 0 || rows < 0) return fail(XG_ERR_INVALID_ARG, "xg_seg_copy: negative extent");
    if (nseg == 0 || rows == 0) return XG_OK;
    if (!src_ptrs || !dst_ptrs || !src_ld_bytes || !dst_ld_bytes || !len_bytes)
        return fail(XG_ERR_INVALID_ARG, "xg_seg_copy: null descriptor array");
    uint64_t bits = 0;
    for (int64_t k = 0; k < nseg; ++k) {
        if (len_bytes[k] < 0 || src_ld_bytes[k] < 0 || dst_ld_bytes[k] < 0)
            return fail(XG_ERR_INVALID_ARG, "xg_seg_copy: negative length/stride in segment %lld", (long long)k);
        if (len_bytes[k] == 0) continue;
        if (!src_ptrs[k] || !dst_ptrs[k]) return fail(XG_ERR_INVALID_ARG, "xg_seg_copy: null pointer in segment %lld", (long long)k);
        if (rows > 1 && (src_ld_bytes[k] < len_bytes[k] || dst_ld_bytes[k] < len_bytes[k]))
            return fail(XG_ERR_INVALID_ARG, "xg_seg_copy: stride smaller than length in segment %lld", (long long)k);
        bits |= (uint64_t)reinterpret_cast<uintptr_t>(src_ptrs[k]) | (uint64_t)reinterpret_cast<uintptr_t>(dst_ptrs[k]) |
                (uint64_t)src_ld_bytes[k] | (uint64_t)dst_ld_bytes[k] | (uint64_t)len_bytes[k];
    }
    const int unit = pow2_align(bits & 15u ? (bits & 15u) : 16);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);

    SegCopyParams p;
    p.rows = rows;
    p.mask = row_mask;
    p.zero_when = mask_zero_when;
    auto flush = [&]() -> int {
        if (p.nseg == 0) return XG_OK;
        // Rows per CTA: every CTA first copies the segment list out of the (large) parameter block and builds the
        // look-up table, so a CTA should take many rows - about 16 CTAs per SM over the whole launch - but never
        // fewer than a thread takes at once.
        const int64_t min_rows = unit >= 16 ? kCopyUnroll : 2 * kCopyUnroll;
        const int64_t want_ctas = 16LL * num_sms();
        int64_t rpc = (rows + want_ctas - 1) / want_ctas;
        rpc = (rpc + min_rows - 1) / min_rows * min_rows;  // whole groups of the rows a thread takes at once
        if (rpc * p.width > 0x3fffffffLL) rpc = 0x3fffffffLL / p.width;  // the narrow-row path indexes rows * width in 32 bits
        if (rpc < 1) rpc = 1;
        p.rows_per_cta = (int32_t)rpc;
        int rc = dispatch_seg_copy(unit, p, st);
        p.nseg = 0;
        p.width = 0;
        return rc;
    };
    p.nseg = 0;
    p.width = 0;
    for (int64_t k = 0; k < nseg; ++k) {
        int64_t units_left = len_bytes[k] / unit;
        int64_t done = 0;
        while (units_left > 0) {
            if (p.nseg == kMaxSegs || p.width == kLutMax) {
                int rc = flush();
                if (rc != XG_OK) return rc;
            }
            int64_t take = kLutMax - p.width;
            if (take > units_left) take = units_left;
            SegDesc& sd = p.seg[p.nseg];
            sd.src = reinterpret_cast<const char*>(src_ptrs[k]) + done * unit;
            sd.dst = reinterpret_cast<char*>(dst_ptrs[k]) + done * unit;
            sd.src_ld = src_ld_bytes[k];
            sd.dst_ld = dst_ld_bytes[k];
            sd.units = (int32_t)take;
            sd.unit_start = p.width;
            p.nseg += 1;
            p.width += (int32_t)take;
            done += take;
            units_left -= take;
        }
    }
    return flush();
}

extern "C" int xg_gather_rows(const void* const* tables, const int64_t* table_rows, int64_t F, const int64_t* idx,
                              int64_t idx_row_stride, int64_t idx_col_stride, const uint8_t* row_mask,
                              int mask_zero_when, void* out, int64_t rows, int64_t D, int64_t out_ld, int elem_size,
                              void* stream) {
    using namespace xg;
    if (F < 0 || rows < 0 || D < 0) return fail(XG_ERR_INVALID_ARG, "xg_gather_rows: negative extent");
    if (elem_size != 2 && elem_size != 4 && elem_size != 8) return fail(XG_ERR_INVALID_ARG, "xg_gather_rows: elem_size must be 2, 4 or 8");
    if (F == 0 || rows == 0 || D == 0) return XG_OK;
    if (!tables || !table_rows || !idx || !out) return fail(XG_ERR_INVALID_ARG, "xg_gather_rows: null pointer");
    if (out_ld < F * D) return fail(XG_ERR_INVALID_ARG, "xg_gather_rows: out_ld smaller than F*D");
    const int64_t row_bytes = D * elem_size;
    if (row_bytes > 0x7fffffffLL) return fail(XG_ERR_TOO_LARGE, "xg_gather_rows: row too wide");
    uint64_t bits = (uint64_t)reinterpret_cast<uintptr_t>(out) | (uint64_t)(out_ld * elem_size) | (uint64_t)row_bytes;
    for (int64_t f = 0; f < F; ++f) {
        if (!tables[f]) return fail(XG_ERR_INVALID_ARG, "xg_gather_rows: null table %lld", (long long)f);
        if (table_rows[f] < 0) return fail(XG_ERR_INVALID_ARG, "xg_gather_rows: negative table size");
        bits |= (uint64_t)reinterpret_cast<uintptr_t>(tables[f]);
    }
    const int unit = pow2_align(bits & 15u ? (bits & 15u) : 16);
    if (unit < 2) return fail(XG_ERR_UNSUPPORTED, "xg_gather_rows: pointers must be at least 2-byte aligned");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    for (int64_t f0 = 0; f0 < F; f0 += kMaxSegs) {
        GatherParams p;
        p.F = (int32_t)((F - f0) < kMaxSegs ? (F - f0) : kMaxSegs);
        p.f0 = (int32_t)f0;
        for (int k = 0; k < p.F; ++k) {
            p.table[k] = reinterpret_cast<const char*>(tables[f0 + k]);
            p.table_rows[k] = table_rows[f0 + k];
        }
        p.units_per_row = (int32_t)(row_bytes / unit);
        if ((int64_t)p.F * p.units_per_row > 0x3fffffffLL) return fail(XG_ERR_TOO_LARGE, "xg_gather_rows: F * D too large");
        p.zero_when = mask_zero_when;
        p.rows = rows;
        p.row_bytes = row_bytes;
        p.idx = idx;
        p.idx_rs = idx_row_stride;
        p.idx_cs = idx_col_stride;
        p.mask = row_mask;
        p.out = reinterpret_cast<char*>(out);
        p.out_ld_bytes = out_ld * elem_size;
        int rc;
        switch (unit) {
            case 16: rc = launch_gather<uint4>(p, st); break;
            case 8: rc = launch_gather<uint2>(p, st); break;
            case 4: rc = launch_gather<uint32_t>(p, st); break;
            default: rc = launch_gather<uint16_t>(p, st); break;
        }
        if (rc != XG_OK) return rc;
    }
    return XG_OK;
}
