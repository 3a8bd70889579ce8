// True-fp32 dense layer (no TF32): out = act(A @ W + bias + residual) with FFMA accumulation.
// Shared-memory tiled SIMT kernel; used for the fp32 graphs whose tolerance (1e-5 relative) rules out
// tensor-core TF32, and - with 16-bit elements converted on the way in and out, fp32 in between - for the 16-bit
// shapes whose rows no tensor map can address (row lengths or base addresses that are not multiples of 16 bytes). W is [K, N] (trans_b = 0) or [N, K] (trans_b = 1); both tiles are stored k-major
// in shared memory so the inner product reads float4 vectors without bank conflicts.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include <cmath>
#include <cstdlib>

namespace xg {

__device__ unsigned int g_f32_status[4];  // non-zero after a bounded wait expired in gemm_fma_kernel

namespace {

struct GemmF32Params {  // element type: the kernel's template parameter
    const void* A;
    const void* B;
    const void* bias;
    const void* residual;
    void* out;
    int64_t M, N, K, lda, ldb, ldc, ldr;
    int trans_b;
    int act;
};

__device__ __forceinline__ float act_f32(float v, int act) {
    switch (act) {
        case XG_ACT_GELU: return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
        case XG_ACT_RELU: return v > 0.f ? v : 0.f;
        case XG_ACT_SILU: return v / (1.0f + expf(-v));
        case XG_ACT_SIGMOID: return 1.0f / (1.0f + expf(-v));
        default: return v;
    }
}

// 256 threads; thread (ty, tx) owns a TM x TN micro-tile; BM = 16*TM, BN = 16*TN.
template <typename T, int TM, int TN, int BK>
__device__ __forceinline__ void gemm_f32_tile(const GemmF32Params& p) {
    constexpr int BM = 16 * TM, BN = 16 * TN;
    const T* __restrict__ gA = reinterpret_cast<const T*>(p.A);
    const T* __restrict__ gB = reinterpret_cast<const T*>(p.B);
    const T* gbias = reinterpret_cast<const T*>(p.bias);
    const T* gres = reinterpret_cast<const T*>(p.residual);
    T* gout = reinterpret_cast<T*>(p.out);
    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Bs[2][BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int64_t m0 = (int64_t)blockIdx.y * BM, n0 = (int64_t)blockIdx.x * BN;

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    constexpr int A_ELEMS = BM * BK / 256;
    constexpr int B_ELEMS = BN * BK / 256;
    float a_reg[A_ELEMS], b_reg[B_ELEMS];

    auto load_global = [&](int64_t k0) {
#pragma unroll
        for (int e = 0; e < A_ELEMS; ++e) {
            const int idx = tid + e * 256;  // k fastest: consecutive threads read consecutive k of one row
            const int kk = idx % BK, mm = idx / BK;
            const int64_t gm = m0 + mm, gk = k0 + kk;
            a_reg[e] = (gm < p.M && gk < p.K) ? Cvt<T>::to_f(gA[gm * p.lda + gk]) : 0.f;
        }
#pragma unroll
        for (int e = 0; e < B_ELEMS; ++e) {
            const int idx = tid + e * 256;
            if (p.trans_b) {  // W[N, K]: k fastest
                const int kk = idx % BK, nn = idx / BK;
                const int64_t gn = n0 + nn, gk = k0 + kk;
                b_reg[e] = (gn < p.N && gk < p.K) ? Cvt<T>::to_f(gB[gn * p.ldb + gk]) : 0.f;
            } else {  // W[K, N]: n fastest
                const int nn = idx % BN, kk = idx / BN;
                const int64_t gn = n0 + nn, gk = k0 + kk;
                b_reg[e] = (gn < p.N && gk < p.K) ? Cvt<T>::to_f(gB[gk * p.ldb + gn]) : 0.f;
            }
        }
    };
    auto store_shared = [&](int buf) {
#pragma unroll
        for (int e = 0; e < A_ELEMS; ++e) {
            const int idx = tid + e * 256;
            As[buf][idx % BK][idx / BK] = a_reg[e];
        }
#pragma unroll
        for (int e = 0; e < B_ELEMS; ++e) {
            const int idx = tid + e * 256;
            if (p.trans_b) Bs[buf][idx % BK][idx / BK] = b_reg[e];
            else Bs[buf][idx / BN][idx % BN] = b_reg[e];
        }
    };

    const int64_t nk = (p.K + BK - 1) / BK;
    load_global(0);
    store_shared(0);
    __syncthreads();
    for (int64_t kt = 0; kt < nk; ++kt) {
        const int buf = (int)(kt & 1);
        if (kt + 1 < nk) load_global((kt + 1) * BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; i += 4) {
                const float4 t = *reinterpret_cast<const float4*>(&As[buf][kk][ty * TM + i]);
                a[i] = t.x; a[i + 1] = t.y; a[i + 2] = t.z; a[i + 3] = t.w;
            }
#pragma unroll
            for (int j = 0; j < TN; j += 4) {
                const float4 t = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * TN + j]);
                b[j] = t.x; b[j + 1] = t.y; b[j + 2] = t.z; b[j + 3] = t.w;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (kt + 1 < nk) {
            store_shared(buf ^ 1);
            __syncthreads();
        }
    }

#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int64_t gm = m0 + ty * TM + i;
        if (gm >= p.M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int64_t gn = n0 + tx * TN + j;
            if (gn >= p.N) continue;
            float v = acc[i][j];
            if (gbias) v += Cvt<T>::to_f(gbias[gn]);
            if (gres) v += Cvt<T>::to_f(gres[gm * p.ldr + gn]);
            gout[gm * p.ldc + gn] = Cvt<T>::from_f(act_f32(v, p.act));
        }
    }
}

template <typename T, int TM, int TN, int BK>
__global__ void __launch_bounds__(256) gemm_f32_kernel(const GemmF32Params p) {
    pdl_sync();
    gemm_f32_tile<T, TM, TN, BK>(p);
}

// Grouped form: blockIdx.z picks the entry; its five pointers come from a table in the kernel's parameter space, the
// extents, strides and activation are shared by the group.
constexpr int kF32GroupMax = 24;  // 24 x 5 pointers = 960 bytes of parameters
struct GemmF32Group {
    const void* A[kF32GroupMax];
    const void* B[kF32GroupMax];
    const void* bias[kF32GroupMax];
    const void* residual[kF32GroupMax];
    void* out[kF32GroupMax];
};
__device__ __forceinline__ GemmF32Params entry_params(const GemmF32Params& p, const GemmF32Group& g) {
    GemmF32Params pe = p;
    const int e = blockIdx.z;
    pe.A = g.A[e];
    pe.B = g.B[e];
    pe.bias = g.bias[e];
    pe.residual = g.residual[e];
    pe.out = g.out[e];
    return pe;
}

template <typename T, int TM, int TN, int BK>
__global__ void __launch_bounds__(256) gemm_f32_group_kernel(const GemmF32Params p, const __grid_constant__ GemmF32Group g) {
    pdl_sync();
    const GemmF32Params pe = entry_params(p, g);
    gemm_f32_tile<T, TM, TN, BK>(pe);
}

// Small problems (fewer 64 x 64 tiles than SMs) are latency-bound in the kernel above: every 16-wide k-tile costs a
// round trip to L2. This variant gives each CTA a small output tile and the whole K-panel of both operands, 256 k at
// a time, fetched with one burst of 16-byte asynchronous copies, so a k-chunk costs one round trip; the inner
// product reads both panels as float4 along k (A rows are shared by the 16 threads of a row group, the B rows of the
// 8 threads of a wavefront fall into distinct bank groups with the 260-float row pitch). W must be [N, K].
// 128 threads as 8 (m) x 16 (n); thread (ty, tx) owns a TM x TN micro-tile; BM = 8 TM, BN = 16 TN.
constexpr int kPanelK = 256;
constexpr int kPanelPitch = kPanelK + 4;  // floats; rows stay 16-byte aligned

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
    const int bytes = valid ? 16 : 0;  // 0 source bytes: the 16 destination bytes are zero-filled
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc), "r"(bytes) : "memory");
}

template <int TM, int TN>
__device__ __forceinline__ void gemm_f32_panel_tile(const GemmF32Params& p) {
    constexpr int BM = 8 * TM, BN = 16 * TN;
    extern __shared__ __align__(16) float panel[];
    float* As = panel;                      // [BM][kPanelPitch]
    float* Bs = panel + BM * kPanelPitch;   // [BN][kPanelPitch]
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int64_t m0 = (int64_t)blockIdx.y * BM, n0 = (int64_t)blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int64_t k0 = 0; k0 < p.K; k0 += kPanelK) {
        const int kc = (int)((p.K - k0) < kPanelK ? (p.K - k0) : kPanelK);  // multiple of 4 (host-checked)
        const int vec_per_row = kc / 4;
        if (k0 > 0) __syncthreads();  // the previous chunk has been consumed
        for (int idx = tid; idx < BM * vec_per_row; idx += 128) {
            const int r = idx / vec_per_row, v = idx - r * vec_per_row;
            const int64_t gm = m0 + r;
            cp_async16(As + r * kPanelPitch + 4 * v, reinterpret_cast<const float*>(p.A) + (gm < p.M ? gm : 0) * p.lda + k0 + 4 * v, gm < p.M);
        }
        for (int idx = tid; idx < BN * vec_per_row; idx += 128) {
            const int r = idx / vec_per_row, v = idx - r * vec_per_row;
            const int64_t gn = n0 + r;
            cp_async16(Bs + r * kPanelPitch + 4 * v, reinterpret_cast<const float*>(p.B) + (gn < p.N ? gn : 0) * p.ldb + k0 + 4 * v, gn < p.N);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // unrolled: with two or three warps per scheduler the shared-memory loads of several k-steps have to be in
        // flight together (one k-step per iteration ran at 7.9 cycles per issued instruction)
#pragma unroll 4
        for (int k = 0; k < kc; k += 4) {
            float4 a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(As + (ty * TM + i) * kPanelPitch + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(Bs + (tx * TN + j) * kPanelPitch + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float c = acc[i][j];
                    c = fmaf(a[i].x, b[j].x, c);
                    c = fmaf(a[i].y, b[j].y, c);
                    c = fmaf(a[i].z, b[j].z, c);
                    c = fmaf(a[i].w, b[j].w, c);
                    acc[i][j] = c;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int64_t gm = m0 + ty * TM + i;
        if (gm >= p.M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int64_t gn = n0 + tx * TN + j;
            if (gn >= p.N) continue;
            float v = acc[i][j];
            if (p.bias) v += reinterpret_cast<const float*>(p.bias)[gn];
            if (p.residual) v += reinterpret_cast<const float*>(p.residual)[gm * p.ldr + gn];
            reinterpret_cast<float*>(p.out)[gm * p.ldc + gn] = act_f32(v, p.act);
        }
    }
}

template <int TM, int TN>
__global__ void __launch_bounds__(128) gemm_f32_panel_group_kernel(const GemmF32Params p, const __grid_constant__ GemmF32Group g) {
    pdl_sync();
    const GemmF32Params pe = entry_params(p, g);
    gemm_f32_panel_tile<TM, TN>(pe);
}

template <int TM, int TN>
int launch_panel_group(const GemmF32Params& p, const GemmF32Group& g, int count, cudaStream_t st) {
    constexpr int BM = 8 * TM, BN = 16 * TN;
    constexpr int smem = (BM + BN) * kPanelPitch * (int)sizeof(float);
    auto kern = gemm_f32_panel_group_kernel<TM, TN>;
    static std::atomic<uint64_t> reserved{0};
    if (!reserve_smem(kern, smem, reserved)) return fail(XG_ERR_LAUNCH, "xg_gemm_group_bias_act(f32): cannot reserve %d bytes of shared memory", smem);
    dim3 grid((unsigned)((p.N + BN - 1) / BN), (unsigned)((p.M + BM - 1) / BM), (unsigned)count);
    launch_with({.early = false}, kern, grid, 128, smem, st, p, g);
    return check_launch("xg_gemm_group_bias_act(f32)");
}

// ---------------------------------------------------------------------------------------------------------
// Tiled FMA kernel with K split twice: over the eight warps of a CTA, and over the CTAs of a cluster.
//
// What bounds these problems is latency, not the FMA pipe: a 256 x 768 x 256 layer is 1.4 us of FMAs spread over the chip
// but only 24 tiles of 64 x 128. So tiles are small (32 or 64 wide), a tile's K range is dealt to 8 / (WM WN) groups of
// warps in slices of 32, and where the tiles still do not fill the chip to S CTAs of a cluster; the partial tiles are added
// in a fixed order through shared memory (and the cluster's distributed shared memory), so results do not depend on timing.
//
// A slice is one TMA box of [rows x 32 floats] per operand with the 128-byte swizzle: rows stay K-contiguous as they are in
// memory, the 16-byte chunk c of row r lies at c ^ (r & 7), and the eight (four) rows that a warp reads together fall into
// different banks. Both operands are read as float4 along K and multiplied as packed pairs (fma.rn.f32x2: even and odd k
// accumulate separately), 64 packed FMAs per 12 shared-memory loads. Operands TMA cannot address are left
// to the kernel above (the torch operators copy them into rows it can address first: pad_rows.cu).
// ---------------------------------------------------------------------------------------------------------
constexpr int kSliceK = 32;
constexpr int kFmaWarps = 8;
constexpr int kFmaThreads = kFmaWarps * 32 + 32;  // + the TMA warp
constexpr int kFmaStages = 3;

template <int TM, int WN>
struct FmaCfg {
    static constexpr int BM = 4 * TM, BN = 32 * WN;
    static constexpr int KW = kFmaWarps / WN;                 // warp groups along K
    static constexpr int KC = KW * kSliceK;                   // K per stage
    static constexpr int A_BYTES = BM * kSliceK * 4, W_BYTES = BN * kSliceK * 4;
    static constexpr int STAGE_BYTES = KW * (A_BYTES + W_BYTES);
    static constexpr int PITCH = BN + 8;                      // floats per row of a partial tile: conflict-free writes
    static constexpr int PART_BYTES = KW * BM * PITCH * 4;
    static constexpr int smem(int stages) {
        return (stages * STAGE_BYTES > PART_BYTES ? stages * STAGE_BYTES : PART_BYTES) + 1024 /*alignment*/ + 512 /*barriers*/;
    }
};

struct FmaParams {
    GemmF32Params g;
    int stages;
    int S;       // CTAs of a cluster = k-splits
    int vec_ok;  // rows of out, residual and bias can be accessed four elements at a time
};

// chunk c (16 bytes) of row r of a slice
__device__ __forceinline__ int slice_off(int r, int c) { return r * (kSliceK * 4) + ((c ^ (r & 7)) << 4); }

__device__ __forceinline__ void fma_pair(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void ld_pairs(uint64_t& x, uint64_t& y, uint32_t addr) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(addr));
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t cluster_addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
    return v;
}

// One slice of K: TM x 4 outputs per thread, rows i * 4 + ty and columns j * 8 + tx of the warp's tile. `a_base`, `w_base`:
// multiples of 128 bytes, so that the swizzle of chunk c is an exclusive-or of the row's address with c << 4.
template <int TM>
__device__ __forceinline__ void fma_slice(uint64_t (&acc)[TM][4], uint32_t a_base, uint32_t w_base, int ty, int tx) {
    // rows 4 i + ty: the swizzle sees ty for even i and ty + 4 for odd i
    const uint32_t a_even = a_base + (uint32_t)slice_off(ty, 0), a_odd = a_base + (uint32_t)slice_off(ty + 4, 0);
    const uint32_t w_row = w_base + (uint32_t)slice_off(tx, 0);
#pragma unroll
    for (int c = 0; c < kSliceK / 4; ++c) {
        const uint32_t swz = (uint32_t)c << 4;
        uint64_t b[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j) ld_pairs(b[j][0], b[j][1], (w_row ^ swz) + (uint32_t)(j * 8 * kSliceK * 4));
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            uint64_t a0, a1;
            ld_pairs(a0, a1, (((i & 1) ? a_odd : a_even) ^ swz) + (uint32_t)((i >> 1) * 8 * kSliceK * 4));
#pragma unroll
            for (int j = 0; j < 4; ++j) fma_pair(acc[i][j], a0, b[j][0]);
#pragma unroll
            for (int j = 0; j < 4; ++j) fma_pair(acc[i][j], a1, b[j][1]);
        }
    }
}

template <int TM, int WN>
__global__ void __launch_bounds__(kFmaThreads, 2)
gemm_fma_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const FmaParams fp) {
    using Cfg = FmaCfg<TM, WN>;
    constexpr int BM = Cfg::BM, BN = Cfg::BN, KW = Cfg::KW, KC = Cfg::KC;
    const GemmF32Params& p = fp.g;
    const int S = fp.S, stages = fp.stages;
    extern __shared__ uint8_t smem_raw[];
    // the same offset in every CTA of a cluster: addresses mapped into a peer name the same object there
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int area = stages * Cfg::STAGE_BYTES > Cfg::PART_BYTES ? stages * Cfg::STAGE_BYTES : Cfg::PART_BYTES;
    // a barrier pair per stage and warp group along K: every group runs down its own slices
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + area);  // [kFmaStages][KW]
    uint64_t* empty_bar = full_bar + kFmaStages * KW;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty_bar + kFmaStages * KW);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int s = (int)(blockIdx.x % (unsigned)S);
    const int64_t n0 = (int64_t)(blockIdx.x / (unsigned)S) * BN, m0 = (int64_t)blockIdx.y * BM;
    const int nch = (int)((p.K + KC - 1) / KC);
    const int ch0 = (int)((int64_t)nch * s / S), ch1 = (int)((int64_t)nch * (s + 1) / S);  // this CTA's share of the stages

    if (tid == 0) {
        for (int i = 0; i < stages * KW; ++i) {
            ptx::mbar_init(&full_bar[i], 1);
            ptx::mbar_init(&empty_bar[i], WN);
        }
        *abort_flag = 0;
        ptx::fence_mbar_init();
        ptx::fence_proxy_async();
    }
    __syncthreads();
    pdl_sync();

    const int kw = warp / WN, wn = warp % WN;  // of the eight multiplying warps
    const int ty = lane >> 3, tx = lane & 7;
    uint64_t acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    bool ok = true;

    auto compute = [&](const uint8_t* stage) {
        const uint32_t base = ptx::smem_u32(stage + kw * (Cfg::A_BYTES + Cfg::W_BYTES));
        fma_slice<TM>(acc, base, base + (uint32_t)(Cfg::A_BYTES + wn * 32 * kSliceK * 4), ty, tx);
    };

    if (warp == kFmaWarps) {
        if (ptx::elect_one()) {
            ptx::prefetch_tensormap(&tmap_a);
            ptx::prefetch_tensormap(&tmap_w);
            for (int ch = ch0; ch < ch1 && ok; ++ch) {
                const int i = (ch - ch0) % stages;
                const uint32_t par = (uint32_t)((ch - ch0) / stages) & 1u;
                for (int q = 0; q < KW; ++q) {
                    const int64_t k0 = (int64_t)ch * KC + q * kSliceK;
                    if (k0 >= p.K) break;
                    uint64_t* full = &full_bar[i * KW + q];
                    if (!ptx::mbar_wait_bounded(&empty_bar[i * KW + q], par ^ 1u, abort_flag)) { ok = false; break; }
                    ptx::mbar_arrive_expect_tx(full, (uint32_t)(Cfg::A_BYTES + Cfg::W_BYTES));
                    uint8_t* st = smem + i * Cfg::STAGE_BYTES + q * (Cfg::A_BYTES + Cfg::W_BYTES);
                    ptx::tma_load_2d(st, &tmap_a, full, (int)k0, (int)m0);
                    ptx::tma_load_2d(st + Cfg::A_BYTES, &tmap_w, full, (int)k0, (int)n0);
                }
            }
            if (!ok) {  // unwinding: give the copies in flight a bounded time to land before shared memory is given up
                atomicOr(&g_f32_status[0], 1u);
                const uint64_t t0 = ptx::globaltimer_ns();
                while (ptx::globaltimer_ns() - t0 < 20000ull) {
                }
            }
        }
    } else {
        for (int ch = ch0; ch < ch1; ++ch) {
            const int i = (ch - ch0) % stages;
            if ((int64_t)ch * KC + kw * kSliceK >= p.K) break;  // only the last stage lacks slices
            ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded(&full_bar[i * KW + kw], (uint32_t)((ch - ch0) / stages) & 1u, abort_flag));
            if (!ok) break;
            compute(smem + i * Cfg::STAGE_BYTES);
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&empty_bar[i * KW + kw]);
        }
        if (!ok && lane == 0) atomicOr(&g_f32_status[0], 2u);
    }

    // ---- partial tiles: added over the warp groups, then over the cluster, in a fixed order ----
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem);  // [KW][BM][PITCH]
    if (warp < kFmaWarps) {
        float* mine = part + kw * BM * Cfg::PITCH + wn * 32;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mine[(i * 4 + ty) * Cfg::PITCH + j * 8 + tx] =
                    __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
    }
    __syncthreads();
    auto finish = [&](const float4& v4, int r, int c) {
        const int64_t gm = m0 + r, gn = n0 + c;
        if (gm >= p.M || gn >= p.N) return;
        float v[4] = {v4.x, v4.y, v4.z, v4.w};
        const float* bias = reinterpret_cast<const float*>(p.bias) + gn;
        const float* res = reinterpret_cast<const float*>(p.residual) + gm * p.ldr + gn;
        float* out = reinterpret_cast<float*>(p.out) + gm * p.ldc + gn;
        struct alignas(16) Quad {
            float e[4];
        };
        if (fp.vec_ok && gn + 4 <= p.N) {
            Quad q;
            if (p.bias) {
                q = *reinterpret_cast<const Quad*>(bias);
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] += q.e[u];
            }
            if (p.residual) {
                q = *reinterpret_cast<const Quad*>(res);
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] += q.e[u];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) q.e[u] = act_f32(v[u], p.act);
            *reinterpret_cast<Quad*>(out) = q;
        } else {
            for (int u = 0; u < 4 && gn + u < p.N; ++u) {
                float x = v[u];
                if (p.bias) x += bias[u];
                if (p.residual) x += res[u];
                out[u] = act_f32(x, p.act);
            }
        }
    };
    for (int e = tid; e < BM * BN / 4; e += kFmaThreads) {
        const int r = e / (BN / 4), c = e % (BN / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int q = 0; q < KW; ++q) {
            const float4 t = *reinterpret_cast<const float4*>(part + (q * BM + r) * Cfg::PITCH + c);
            v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
        }
        if (S == 1) finish(v, r, c);
        else *reinterpret_cast<float4*>(part + r * Cfg::PITCH + c) = v;
    }
    if (S > 1) {
        __syncthreads();      // (the cluster barrier below is warp-aligned: the warps are converged here)
        ptx::cluster_sync();  // every CTA's share is in its shared memory
        constexpr int kUnits = BM * (BN / 4) / 32;  // warp-sized pieces of the tile, dealt to the CTAs
        const int e_lo = kUnits * s / S * 32, e_hi = kUnits * (s + 1) / S * 32;
        for (int e = e_lo + tid; e < e_hi; e += kFmaThreads) {
            const int r = e / (BN / 4), c = e % (BN / 4) * 4;
            // nothing is loaded that is not stored: a remote load without a consumer could still be under way when its owner leaves
            if (m0 + r >= p.M || n0 + c >= p.N) continue;
            const uint32_t at = ptx::smem_u32(part + r * Cfg::PITCH + c);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int q = 0; q < S; ++q) {
                const float4 t = ld_cluster_f32x4(ptx::map_to_cta(at, (uint32_t)q));
                v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
            }
            finish(v, r, c);
        }
        __syncthreads();
        ptx::cluster_sync();  // no CTA leaves while a peer still reads its shared memory
    }
}

bool make_tmap_2d_f32(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    PFN_encodeTiled enc = get_encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * 4};
    cuuint32_t box[2] = {(cuuint32_t)kSliceK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TM, int WN>
int launch_fma(const GemmF32Params& g, int S, cudaStream_t st) {
    using Cfg = FmaCfg<TM, WN>;
    auto kern = gemm_fma_kernel<TM, WN>;
    static std::atomic<uint64_t> reserved{0};
    if (!reserve_smem(kern, Cfg::smem(kFmaStages), reserved))
        return fail(XG_ERR_LAUNCH, "xg_gemm_bias_act(f32): cannot reserve %d bytes of shared memory", Cfg::smem(kFmaStages));
    CUtensorMap ta, tw;
    if (!make_tmap_2d_f32(&ta, g.A, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda, Cfg::BM) ||
        !make_tmap_2d_f32(&tw, g.B, (uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.ldb, Cfg::BN))
        return fail(XG_ERR_UNSUPPORTED, "xg_gemm_bias_act(f32): tensor-map encoding failed");
    FmaParams p;
    p.g = g;
    p.S = S;
    p.vec_ok = g.ldc % 4 == 0 && aligned16(g.out) && aligned16(g.bias) && (!g.residual || (g.ldr % 4 == 0 && aligned16(g.residual)));
    const int64_t per_cta = ((g.K + Cfg::KC - 1) / Cfg::KC + S - 1) / S;
    p.stages = (int)(per_cta < kFmaStages ? per_cta : kFmaStages);
    const dim3 grid((unsigned)((g.N + Cfg::BN - 1) / Cfg::BN * S), (unsigned)((g.M + Cfg::BM - 1) / Cfg::BM));
    // Placed early only above one CTA per SM (see LaunchOptions). Clusters never are: an early one of eight raised a
    // misaligned-address error behind another launch of itself. What reading excludes: the row pitch of a partial tile (160, 288
    // or 544 bytes) and the column offsets are multiples of 16 bytes and end inside the partial tiles, the area starts at one
    // offset in all CTAs, peers have started before the first remote access (cluster barrier) and are there until the last one
    // (second barrier). What it leaves open: whether the form that faulted still read rows past M from the peers and dropped
    // them; a load without a consumer can be under way when its owner's shared memory goes to the next kernel. The kernel has no
    // such loads (see the `continue` above); that they were the cause is not shown.
    launch_with({.cluster = S > 1 ? (unsigned)S : 0u, .early = (int64_t)grid.x * grid.y > num_sms()}, kern, grid, kFmaThreads,
                Cfg::smem(p.stages), st, ta, tw, p);
    return check_launch("xg_gemm_bias_act(f32)");
}

// Tile shape (TM x 4 rows by WN x 32 columns) and K split over the CTAs of a cluster: the cheapest by a cost model in
// microseconds fitted to a sweep on B200 (26 shapes, M = 1..8192, N = 64..11008, K = 64..11008, every choice below; the model's
// choice is within 0.8 % of the best one on average):
//   stage  : an SM multiplies a stage in 0.166 us per unit of TM (0.138 us at the packed-FMA rate) or takes it in at
//            0.0051 us per KB, whichever is longer, for every CTA it gets;
//   CTA    : 1.44 us to set up, reduce and store, and 0.49 us of latency per stage, per round of resident CTAs;
//   split  : 1.6 us, and 0.24 us per CTA of the cluster, to add the partial tiles through distributed shared memory.
struct FmaChoice {
    int TM, WN, S;
};
FmaChoice plan_fma(int64_t M, int64_t N, int64_t K) {
    const double sms = num_sms();
    FmaChoice best{4, 1, 1};
    double best_cost = 1e30;
    for (int TM = 2; TM <= 4; TM += 2) {
        for (int WN = 1; WN <= 4; WN *= 2) {
            const int BM = 4 * TM, BN = 32 * WN, KW = kFmaWarps / WN, KC = KW * kSliceK;
            const double tiles = (double)((M + BM - 1) / BM) * (double)((N + BN - 1) / BN);
            const int64_t chunks = (K + KC - 1) / KC;
            const double kb = KW * (BM + BN) * 0.128;
            for (int S : {1, 2, 3, 4, 6, 8}) {
                if (S > 1 && chunks < S) break;
                const double stages = (double)((chunks + S - 1) / S);
                const double smem = (stages < kFmaStages ? stages : kFmaStages) * kb + 2.5;
                const double resident = 2 * smem <= 233.0 ? 2 : 1;
                const double per_sm = std::ceil(tiles * S / sms), rounds = std::ceil(tiles * S / (sms * resident));
                const double fma = 0.166 * TM, in = 0.0051 * kb;
                const double cost = per_sm * stages * (fma > in ? fma : in) + rounds * (1.44 + 0.49 * stages + (S > 1 ? 1.6 + 0.24 * S : 0.0));
                if (cost < best_cost) {
                    best_cost = cost;
                    best = {TM, WN, S};
                }
            }
        }
    }
    return best;
}

bool fma_addressable(const GemmF32Params& g) {
    return g.trans_b && g.lda % 4 == 0 && g.ldb % 4 == 0 && aligned16(g.A) && aligned16(g.B) && g.K <= 0x7fffffff && g.N <= 0x7fffffff &&
           (g.M + 7) / 8 <= 65535;
}

int dispatch_fma(const GemmF32Params& g, cudaStream_t st) {
    const FmaChoice c = plan_fma(g.M, g.N, g.K);
    if (c.TM == 2) {
        switch (c.WN) {
            case 1: return launch_fma<2, 1>(g, c.S, st);
            case 2: return launch_fma<2, 2>(g, c.S, st);
            default: return launch_fma<2, 4>(g, c.S, st);
        }
    }
    switch (c.WN) {
        case 1: return launch_fma<4, 1>(g, c.S, st);
        case 2: return launch_fma<4, 2>(g, c.S, st);
        default: return launch_fma<4, 4>(g, c.S, st);
    }
}

}  // namespace

int gemm_f32_entry(const void* A, const void* B, const void* bias, const void* residual, void* out, int64_t M, int64_t N,
                   int64_t K, int64_t lda, int64_t ldb, int64_t ldc, int64_t ldr, int trans_b, int act, cudaStream_t st) {
    if (M * N == 0) return XG_OK;
    GemmF32Params p{A, B, bias, residual, out, M, N, K, lda, ldb, ldc, ldr, trans_b, act};
    if (fma_addressable(p)) return dispatch_fma(p, st);
    const int64_t big_tiles = ((M + 127) / 128) * ((N + 127) / 128);
    if (big_tiles >= 2LL * num_sms()) {
        dim3 grid((unsigned)((N + 127) / 128), (unsigned)((M + 127) / 128));
        if ((M + 127) / 128 > 65535) return fail(XG_ERR_TOO_LARGE, "xg_gemm_bias_act(f32): M too large");
        launch_with({.early = false}, gemm_f32_kernel<float, 8, 8, 16>, grid, 256, 0, st, p);
    } else {
        dim3 grid((unsigned)((N + 63) / 64), (unsigned)((M + 63) / 64));
        if ((M + 63) / 64 > 65535) return fail(XG_ERR_TOO_LARGE, "xg_gemm_bias_act(f32): M too large");
        launch_with({.early = false}, gemm_f32_kernel<float, 4, 4, 16>, grid, 256, 0, st, p);
    }
    return check_launch("xg_gemm_bias_act(f32)");
}

// 16-bit operands the tensor-core kernels cannot address (rows or base addresses that are not multiples of 16 bytes):
// the same tiled FMA kernel, elements converted on the way in and out, fp32 accumulation.
int gemm_simt16_entry(const void* A, const void* B, const void* bias, const void* residual, void* out, int64_t M, int64_t N,
                      int64_t K, int64_t lda, int64_t ldb, int64_t ldc, int64_t ldr, int trans_b, int act, int dtype,
                      cudaStream_t st) {
    if (M * N == 0) return XG_OK;
    GemmF32Params p{A, B, bias, residual, out, M, N, K, lda, ldb, ldc, ldr, trans_b, act};
    const bool big = ((M + 127) / 128) * ((N + 127) / 128) >= 2LL * num_sms();
    const int64_t bm = big ? 128 : 64;
    if ((M + bm - 1) / bm > 65535) return fail(XG_ERR_TOO_LARGE, "xg_gemm_bias_act: M too large for the unaligned 16-bit path");
    dim3 grid((unsigned)((N + bm - 1) / bm), (unsigned)((M + bm - 1) / bm));
    if (dtype == XG_BF16) {
        if (big) launch_with({.early = false}, gemm_f32_kernel<__nv_bfloat16, 8, 8, 16>, grid, 256, 0, st, p);
        else launch_with({.early = false}, gemm_f32_kernel<__nv_bfloat16, 4, 4, 16>, grid, 256, 0, st, p);
    } else {
        if (big) launch_with({.early = false}, gemm_f32_kernel<__half, 8, 8, 16>, grid, 256, 0, st, p);
        else launch_with({.early = false}, gemm_f32_kernel<__half, 4, 4, 16>, grid, 256, 0, st, p);
    }
    return check_launch("xg_gemm_bias_act (16-bit, FMA path)");
}

// out[e] = act(A[e] @ W[e] + bias[e] + residual[e]) for `count` fp32 problems of one shape; the operands stay where
// they are (a pointer per entry). One launch per 24 entries; the kernel is chosen as for a single problem with `count`
// times the tiles.
int gemm_f32_group_entry(const void* const* A, const void* const* W, const void* const* bias, const void* const* residual,
                         void* const* out, int64_t count, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldw,
                         int64_t ldc, int64_t ldr, int trans_b, int act, cudaStream_t st) {
    if (M * N == 0) return XG_OK;
    if ((M + 15) / 16 > 65535) return fail(XG_ERR_TOO_LARGE, "xg_gemm_group_bias_act(f32): M too large");
    for (int64_t first = 0; first < count; first += kF32GroupMax) {
        const int n = (int)((count - first) < kF32GroupMax ? (count - first) : kF32GroupMax);
        GemmF32Group g;
        bool aligned = true;
        for (int e = 0; e < kF32GroupMax; ++e) {
            const int64_t i = first + (e < n ? e : 0);  // unused slots repeat the first entry and are never read
            if (!A[i] || !W[i] || !out[i])
                return fail(XG_ERR_INVALID_ARG, "xg_gemm_group_bias_act: null pointer in entry %lld", (long long)i);
            g.A[e] = A[i];
            g.B[e] = W[i];
            g.bias[e] = bias ? bias[i] : nullptr;
            g.residual[e] = residual ? residual[i] : nullptr;
            g.out[e] = out[i];
            aligned = aligned && aligned16(A[i]) && aligned16(W[i]);
        }
        GemmF32Params p{nullptr, nullptr, nullptr, nullptr, nullptr, M, N, K, lda, ldw, ldc, ldr, trans_b, act};
        const int64_t tiles64 = ((M + 63) / 64) * ((N + 63) / 64) * n;
        const bool panel_ok = trans_b && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && aligned;
        int rc;
        if (panel_ok && tiles64 < num_sms()) {
            const int64_t tiles_32x64 = ((M + 31) / 32) * ((N + 63) / 64) * n;
            rc = tiles_32x64 * 3 >= 2LL * num_sms() ? launch_panel_group<4, 4>(p, g, n, st) : launch_panel_group<2, 2>(p, g, n, st);
        } else if (((M + 127) / 128) * ((N + 127) / 128) * n >= 2LL * num_sms()) {
            dim3 grid((unsigned)((N + 127) / 128), (unsigned)((M + 127) / 128), (unsigned)n);
            launch_with({.early = false}, gemm_f32_group_kernel<float, 8, 8, 16>, grid, 256, 0, st, p, g);
            rc = check_launch("xg_gemm_group_bias_act(f32)");
        } else {
            dim3 grid((unsigned)((N + 63) / 64), (unsigned)((M + 63) / 64), (unsigned)n);
            launch_with({.early = false}, gemm_f32_group_kernel<float, 4, 4, 16>, grid, 256, 0, st, p, g);
            rc = check_launch("xg_gemm_group_bias_act(f32)");
        }
        if (rc != XG_OK) return rc;
    }
    return XG_OK;
}

int read_f32_status(unsigned int* host_out, int reset) {
    unsigned int v[4] = {0, 0, 0, 0};
    if (cudaMemcpyFromSymbol(v, g_f32_status, sizeof(v)) != cudaSuccess) {
        cudaGetLastError();
        return fail(XG_ERR_DEVICE, "xg_tc_status: cannot read device status");
    }
    *host_out = v[0];
    if (reset && v[0] != 0) {
        unsigned int z[4] = {0, 0, 0, 0};
        cudaMemcpyToSymbol(g_f32_status, z, sizeof(z));
    }
    return XG_OK;
}

}  // namespace xg
