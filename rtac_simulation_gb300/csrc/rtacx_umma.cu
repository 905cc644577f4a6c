// 16-bit tensor-core contractions on sm_103a, fp32 accumulation, operands
// K-major ("TN") and both bf16 or both fp16.
//
//   k_gemm_split  the contraction of the precision form (rtacx_precision.cu):
//                 C = row_scale * col_scale * (A B^T) with A and B given as
//                 hi + lo halves side by side, [hi (K) | lo (K)] per row, as the
//                 three products hi hi + hi lo + lo hi of each block of K. The
//                 four tiles of a block are loaded once for its three products
//                 (with the halves repeated along K, [hi|hi|lo] x [hi|lo|hi],
//                 six tiles; the operands' tiles come through L2, which bounded
//                 that form). A list of blocks per column tile leaves out those
//                 where B is zero.
//   k_gemm_tn     plain C = A B^T (the diagnostic entry point).
//
// One CTA computes a 128 x BN tile with four warps:
//   warp 0, lane 0  TMA producer: cp.async.bulk.tensor 2D loads of 128 x 64 and
//                   BN x 64 tiles (128-byte swizzle) into a shared-memory ring
//                   guarded by mbarriers;
//   warp 1, lane 0  MMA issuer: tcgen05.mma.kind::f16 (K = 16 each) into a
//                   128-lane x BN-column fp32 TMEM accumulator, tcgen05.commit
//                   frees the stage;
//   warps 0-3       epilogue: tcgen05.ld 32x32b of their TMEM lane quadrant,
//                   optional row / column scaling, fp32 stores of whole
//                   128-byte row segments.
// Every mbarrier wait is bounded (about two seconds); a timeout sets an
// error bit and the CTA skips its remaining work, still waiting (bounded) for
// issued MMAs and freeing its TMEM.
#include "rtacx_internal.cuh"
#include "rtacx_tcgen05.cuh"

#include <algorithm>
#include <cmath>
#include <cuda_bf16.h>

namespace rtacx {

namespace {

constexpr int BM = 128, BK = 64;
constexpr int kThreads = 128;
constexpr uint32_t A_BYTES = BM * BK * 2;

template <int BN_, int STAGES_>
struct Tile {
    static constexpr int BN = BN_, STAGES = STAGES_;
    static constexpr uint32_t B_BYTES = BN * BK * 2;
    static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr uint32_t TMEM_COLS = BN;           // power of two >= 32
    static constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_BYTES + 1024 + 256;
    static constexpr int CTAS_PER_SM = BN == 128 ? 2 : 1;
};
using TileWide = Tile<256, 4>;
using TileNarrow = Tile<128, 3>;
constexpr long long kWaitCycles = 4000000000ll;

// Instruction descriptor of tcgen05.mma.kind::f16: D = f32 (bits 4-5 = 1),
// A and B format at bits 7-9 and 10-12 (0 = f16, 1 = bf16; always the same
// type for both), both K-major (bits 15, 16 = 0), N >> 3 at bits 17-22,
// M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t idesc_for(bool f16, int bn)
{
    return (1u << 4) | ((f16 ? 0u : 1u) << 7) | ((f16 ? 0u : 1u) << 10) | ((uint32_t)(bn >> 3) << 17) |
           ((uint32_t)(BM >> 4) << 24);
}

// Bounded wait of the GEMM (about two seconds).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag)
{
    return mbar_wait_bounded(bar, parity, abort_flag, kWaitCycles);
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}

template <bool kF16, int BN>
__device__ __forceinline__ void umma_16bit(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc_for(kF16, BN)), "r"(accumulate)
                 : "memory");
}

// Epilogue of one warp: its TMEM lane quadrant -> rows m0 + 32 warp + lane. lo_at
// (not 0): the sum of two accumulators, so many columns apart.
template <int BN>
__device__ __forceinline__ void store_tile(uint32_t tmem, float* __restrict__ C, int m0, int n0, int ldc, int warp, int lane,
                                           const float* __restrict__ row_scale, const float* __restrict__ col_scale,
                                           bool any, bool add, uint32_t lo_at = 0)
{
    const int row = m0 + warp * 32 + lane;
    float* crow = C + (size_t)row * ldc + n0;
    const float rs = row_scale ? row_scale[row] : 1.0f;
#pragma unroll 1
    for(int c = 0; c < BN / 32; c++) {
        uint32_t r[32];
        const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 32);
        float v[32];
        if(lo_at) {
            uint32_t lo[32];
            tmem_ld32_two(at, r, at + lo_at, lo);
#pragma unroll
            for(int q = 0; q < 32; q++) v[q] = __uint_as_float(r[q]) + __uint_as_float(lo[q]);
        }
        else {
            tmem_ld32(at, r);
#pragma unroll
            for(int q = 0; q < 32; q++) v[q] = __uint_as_float(r[q]);
        }
        if(!any) {
#pragma unroll
            for(int q = 0; q < 32; q++) v[q] = 0.0f;
        }
        if(row_scale) {
#pragma unroll
            for(int q = 0; q < 32; q++) v[q] *= rs;
        }
        if(col_scale) {
            const float4* cs = reinterpret_cast<const float4*>(col_scale + n0 + c * 32);
#pragma unroll
            for(int q = 0; q < 8; q++) {
                const float4 s4 = __ldg(cs + q);
                v[4 * q] *= s4.x; v[4 * q + 1] *= s4.y; v[4 * q + 2] *= s4.z; v[4 * q + 3] *= s4.w;
            }
        }
        float4* dst = reinterpret_cast<float4*>(crow + c * 32);
        if(add) {
#pragma unroll
            for(int q = 0; q < 8; q++)
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                             ::"l"(dst + q), "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]), "f"(v[4 * q + 3]) : "memory");
            continue;
        }
#pragma unroll
        for(int q = 0; q < 8; q++) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, T::CTAS_PER_SM)
k_gemm_tn(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
          float* __restrict__ C, int K, int ldc, uint32_t* __restrict__ err)
{
    constexpr int BN = T::BN, STAGES = T::STAGES;
    constexpr uint32_t STAGE_BYTES = T::STAGE_BYTES, TMEM_COLS = T::TMEM_COLS;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    unsigned char* base = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + STAGES * STAGE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int nkb = K / BK;
    auto full_bar = [&](int s) { return smem_u32(bars + s); };
    auto empty_bar = [&](int s) { return smem_u32(bars + STAGES + s); };
    const uint32_t accum_bar = smem_u32(bars + 2 * STAGES);

    if(threadIdx.x == 0) {
        for(int s = 0; s < 2 * STAGES + 1; s++) mbar_init(smem_u32(bars + s), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if(warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if(warp == 0 && lane == 0) {
        // TMA producer.
        for(int kb = 0; kb < nkb; kb++) {
            const int s = kb % STAGES;
            if(kb >= STAGES && !mbar_wait(empty_bar(s), ((kb / STAGES) - 1) & 1, abort_flag)) break;
            unsigned char* a = base + s * STAGE_BYTES;
            mbar_expect_tx(full_bar(s), STAGE_BYTES);
            tma_load_2d(smem_u32(a), &tmA, kb * BK, m0, full_bar(s));
            tma_load_2d(smem_u32(a + A_BYTES), &tmB, kb * BK, n0, full_bar(s));
        }
    }
    else if(warp == 1 && lane == 0) {
        // MMA issuer.
        for(int kb = 0; kb < nkb; kb++) {
            const int s = kb % STAGES;
            if(!mbar_wait(full_bar(s), (kb / STAGES) & 1, abort_flag)) break;
            tc_fence_after();
            const uint32_t a = smem_u32(base + s * STAGE_BYTES);
            const uint64_t ad = smem_desc(a), bd = smem_desc(a + A_BYTES);
#pragma unroll
            for(int kk = 0; kk < BK / 16; kk++)   // 32 bytes of K per MMA: +2 in descriptor units
                umma_16bit<false, BN>(tmem, ad + 2 * kk, bd + 2 * kk, (kb > 0 || kk > 0) ? 1u : 0u);
            umma_commit(empty_bar(s));
        }
        umma_commit(accum_bar);   // arrives once every MMA issued above has completed
    }
    __syncwarp();
    const bool ok = mbar_wait(accum_bar, 0, abort_flag);
    __syncwarp();
    tc_fence_after();
    if(__all_sync(0xffffffffu, ok ? 1 : 0)) store_tile<BN>(tmem, C, m0, n0, ldc, warp, lane, nullptr, nullptr, true, false);
    else if(lane == 0 && err) atomicOr(err, kErrGemmTimeout);
    tc_fence_before();
    __syncthreads();
    if(warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// The split contraction. Stage: A hi, A lo, B hi, B lo of one block of 64
// along K; the hi and the lo tiles have a barrier each, so that hi hi starts
// before the lo tiles are in. In long sums (lo_at = BN) the products with a lo
// half have an accumulator of their own: the tensor cores truncate as they
// accumulate, so in one accumulator the two products that add next to nothing
// to the sum cost it digits too (2^24 samples, 512 x 4096: 1.0e-5 from 64 bits,
// 7.3e-6 with two, the time within 0.2 us; short sums keep one, since reading
// two would cost them 0.2 of 19.5 us). blockIdx.z: its share of the column tile's list
// of blocks (blocks: [column tiles][1 + all blocks], the count first), into its
// own partial product C + z rows ldc, or (add) added into C.
template <int BN_, int STAGES_>
struct SplitTile {
    static constexpr int BN = BN_, STAGES = STAGES_;
    static constexpr uint32_t B_BYTES = BN * BK * 2;
    static constexpr uint32_t STAGE_BYTES = 2 * (A_BYTES + B_BYTES);
    static constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_BYTES + 1024 + 256;
};
using SplitWide = SplitTile<256, 2>;
using SplitNarrow = SplitTile<128, 3>;

template <bool kF16, typename T>
__global__ void __launch_bounds__(kThreads, 1)
k_gemm_split(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, float* __restrict__ C,
             int rows, int K, int ldc, const uint16_t* __restrict__ blocks, const float* __restrict__ row_scale,
             const float* __restrict__ col_scale, int add, uint32_t lo_at, uint32_t* __restrict__ err)
{
    constexpr int BN = T::BN, STAGES = T::STAGES;
    constexpr uint32_t TMEM_COLS = 2 * BN;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    unsigned char* base = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + STAGES * T::STAGE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const uint16_t* list = blocks + (size_t)blockIdx.x * (K / BK + 1);
    const int total = list[0];
    const int begin = total * (int)blockIdx.z / (int)gridDim.z, count = total * ((int)blockIdx.z + 1) / (int)gridDim.z - begin;
    list += 1 + begin;
    if(!add) C += (size_t)blockIdx.z * (size_t)rows * ldc;
    auto hi_bar = [&](int s) { return smem_u32(bars + s); };
    auto lo_bar = [&](int s) { return smem_u32(bars + STAGES + s); };
    auto empty_bar = [&](int s) { return smem_u32(bars + 2 * STAGES + s); };
    const uint32_t accum_bar = smem_u32(bars + 3 * STAGES);

    chain_next();
    if(threadIdx.x == 0) {
        for(int s = 0; s < 3 * STAGES + 1; s++) mbar_init(smem_u32(bars + s), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
    }
    if(warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    chain_wait();
    row_scale = after_chain(row_scale);

    if(warp == 0 && lane == 0) {
        // TMA producer.
        for(int i = 0; i < count; i++) {
            const int s = i % STAGES, x = (int)list[i] * BK;
            if(i >= STAGES && !mbar_wait(empty_bar(s), ((i / STAGES) - 1) & 1, abort_flag)) break;
            const uint32_t a = smem_u32(base + s * T::STAGE_BYTES), b = a + 2 * A_BYTES;
            mbar_expect_tx(hi_bar(s), A_BYTES + T::B_BYTES);
            tma_load_2d(a, &tmA, x, m0, hi_bar(s));
            tma_load_2d(b, &tmB, x, n0, hi_bar(s));
            mbar_expect_tx(lo_bar(s), A_BYTES + T::B_BYTES);
            tma_load_2d(b + T::B_BYTES, &tmB, K + x, n0, lo_bar(s));
            tma_load_2d(a + A_BYTES, &tmA, K + x, m0, lo_bar(s));
        }
    }
    else if(warp == 1 && lane == 0) {
        // MMA issuer.
        for(int i = 0; i < count; i++) {
            const int s = i % STAGES;
            const uint32_t parity = (uint32_t)(i / STAGES) & 1u;
            const uint32_t a = smem_u32(base + s * T::STAGE_BYTES), b = a + 2 * A_BYTES;
            const uint64_t ahi = smem_desc(a), alo = smem_desc(a + A_BYTES);
            const uint64_t bhi = smem_desc(b), blo = smem_desc(b + T::B_BYTES);
            if(!mbar_wait(hi_bar(s), parity, abort_flag)) break;
            tc_fence_after();
#pragma unroll
            for(int kk = 0; kk < BK / 16; kk++)   // 32 bytes of K per MMA: +2 in descriptor units
                umma_16bit<kF16, BN>(tmem, ahi + 2 * kk, bhi + 2 * kk, (i > 0 || kk > 0) ? 1u : 0u);
            if(!mbar_wait(lo_bar(s), parity, abort_flag)) break;
            tc_fence_after();
#pragma unroll
            for(int kk = 0; kk < BK / 16; kk++) umma_16bit<kF16, BN>(tmem + lo_at, ahi + 2 * kk, blo + 2 * kk, (!lo_at || i > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
            for(int kk = 0; kk < BK / 16; kk++) umma_16bit<kF16, BN>(tmem + lo_at, alo + 2 * kk, bhi + 2 * kk, 1u);
            umma_commit(empty_bar(s));
        }
        umma_commit(accum_bar);   // arrives once every MMA issued above has completed
    }
    __syncwarp();
    const bool ok = mbar_wait(accum_bar, 0, abort_flag);
    __syncwarp();
    tc_fence_after();
    if(__all_sync(0xffffffffu, ok ? 1 : 0))
        store_tile<BN>(tmem, C, m0, n0, ldc, warp, lane, row_scale, col_scale, count > 0, add != 0, lo_at);
    else if(lane == 0 && err) atomicOr(err, kErrGemmTimeout);
    tc_fence_before();
    __syncthreads();
    if(warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if(!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
           q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
        else
            cudaGetLastError();
    }
    return fn;
}

bool make_map(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t k, uint32_t box_rows, bool f16)
{
    EncodeTiledFn enc = encode_fn();
    if(!enc) return false;
    cuuint64_t dims[2] = {k, rows};
    cuuint64_t strides[1] = {k * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
               const_cast<void*>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

} // namespace

// C = A * B^T; A [M][K], B [N][K] bf16 (16-byte aligned, row stride K), C
// [M][N] fp32. Shapes must be multiples of the tile (128, 128, 64).
static rtacx_status gemm_tn(std::string& error, const void* A, const void* B, float* C, int M, int N, int K,
                            cudaStream_t stream, uint32_t* err)
{
    if(M <= 0 || N <= 0 || K <= 0 || M % BM || N % 128 || K % BK) {
        error = "gemm shape must be multiples of 128 x 128 x 64";
        return RTACX_ERR_INVALID_ARGUMENT;
    }
    // 128 x 256 tiles when N allows them and they cover more than half of
    // the SMs; 128 x 128 tiles (two CTAs per SM) otherwise. Measured on the
    // 4096 x 1024 x 3072 contraction (128 wide tiles): 27 us wide, 30 us
    // narrow (the narrow grid re-reads A twice as often through L2); with
    // half the SMs or fewer, wide tiles leave the tensor cores of the rest
    // idle for the whole launch.
    int dev = 0, sms = 0;
    if(cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        error = "cannot query the current device";
        return RTACX_ERR_CUDA;
    }
    const bool wide = N % 256 == 0 && 2ll * (N / 256) * (M / BM) > (long long)sms;
    const int bn = wide ? TileWide::BN : TileNarrow::BN;
    if((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) % 16 || reinterpret_cast<uintptr_t>(C) % 16) {
        error = "gemm operands must be 16-byte aligned";
        return RTACX_ERR_INVALID_ARGUMENT;
    }
    CUtensorMap ma, mb;
    if(!make_map(&ma, A, (uint64_t)M, (uint64_t)K, BM, false) || !make_map(&mb, B, (uint64_t)N, (uint64_t)K, bn, false)) {
        error = "cuTensorMapEncodeTiled failed";
        return RTACX_ERR_CUDA;
    }
    auto fn = wide ? k_gemm_tn<TileWide> : k_gemm_tn<TileNarrow>;
    const size_t smem = wide ? TileWide::SMEM_BYTES : TileNarrow::SMEM_BYTES;
    cudaError_t e = raise_smem_limit((const void*)fn, smem);
    if(e == cudaSuccess) {
        fn<<<dim3(N / bn, M / BM), kThreads, smem, stream>>>(ma, mb, C, K, N, err);
        e = cudaGetLastError();
    }
    if(e != cudaSuccess) { error = std::string("k_gemm_tn: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    return RTACX_OK;
}

namespace {

auto split_kernel(int bn, bool f16)
{
    return bn == 256 ? (f16 ? k_gemm_split<true, SplitWide> : k_gemm_split<false, SplitWide>)
                     : (f16 ? k_gemm_split<true, SplitNarrow> : k_gemm_split<false, SplitNarrow>);
}
size_t split_smem(int bn) { return bn == 256 ? SplitWide::SMEM_BYTES : SplitNarrow::SMEM_BYTES; }

} // namespace

// Parts of K, at most (16384 grid bearings' real and imaginary parts are 15 of
// kMaxTerms), and terms of a part's sum.
constexpr int kMaxParts = 16, kMaxTerms = 2200;
// Terms of a part's sum from which the lo products have their own accumulator.
constexpr int kLoApart = 512;

// Tile width, K split and block lists of the contraction of A [M][2 K] with
// B [N][2 K] (b: its host copy), M % 128 == 0, N % 256 == 0, K % 64 == 0.
//
// Choice: the fewest microseconds by waves x (blocks per CTA x time of a block
// + fixed time) + the filter's reading of the partial products, with the
// measured times below. 4096 ranges x 512 bearings: 68 wide tiles x 2 parts;
// 512 ranges x 128 bearings: 6 narrow tiles x 8 parts.
rtacx_status plan_gemm_split(std::string& error, GemmPlan& g, const void* A, const void* B, const uint16_t* b, int M, int N,
                             int K, bool f16, int sm_count)
{
    const int nkb = K / BK;
    // Blocks of 64 columns in which a tile of `width` rows of B has a nonzero.
    std::vector<unsigned char> used((size_t)(N / 128) * nkb, 0);
    for(int n = 0; n < N; n++)
        for(int kb = 0; kb < nkb; kb++) {
            unsigned char& u = used[(size_t)(n / 128) * nkb + kb];
            const uint16_t* row = b + (size_t)n * 2 * K + (size_t)kb * BK;
            for(int k = 0; k < BK && !u; k++) u = ((row[k] | row[K + k]) & 0x7fff) != 0;
        }
    double best = 1e30;
    for(int bn : {256, 128}) {
        std::vector<uint16_t> lists((size_t)(N / bn) * (nkb + 1), 0);
        size_t longest = 0;
        for(int t = 0; t < N / bn; t++) {
            uint16_t* l = lists.data() + (size_t)t * (nkb + 1);
            for(int kb = 0; kb < nkb; kb++)
                if(used[(size_t)t * (bn / 128) * nkb + kb] || (bn == 256 && used[((size_t)t * 2 + 1) * nkb + kb])) l[++l[0]] = (uint16_t)kb;
            longest = std::max<size_t>(longest, l[0]);
        }
        for(int ks = 1; ks <= kMaxParts; ks *= 2) {
            if(ks > 1 && longest < (size_t)2 * ks) continue;
            // A sum of K terms of one sign in one accumulator comes out about 6e-9
            // K too small (measured with fp16 operands, up to 16384 grid bearings
            // in 8 parts), a split one its parts' share. So no part takes more
            // than kMaxTerms (1.32e-5), and the time decides among the splits
            // that keep to that.
            if(longest * BK > (size_t)kMaxTerms * ks && ks < kMaxParts) continue;
            const double ctas = (double)(N / bn) * (M / BM) * ks, waves = std::ceil(ctas / sm_count);
            const double t = waves * ((double)longest / ks * (bn == 256 ? 1.0 : 0.6) + 4.0) + (double)ks * M * N * 4.0 / 4e6;
            if(t < best) { best = t; g.bn = bn; g.ksplit = ks; g.lists = lists; g.lo_apart = longest * BK > (size_t)kLoApart * ks; }
        }
    }
    if(!make_map(&g.ma, A, (uint64_t)M, 2 * (uint64_t)K, BM, f16) || !make_map(&g.mb, B, (uint64_t)N, 2 * (uint64_t)K, g.bn, f16)) {
        error = "cuTensorMapEncodeTiled failed";
        return RTACX_ERR_CUDA;
    }
    if(raise_smem_limit((const void*)split_kernel(g.bn, f16), split_smem(g.bn)) != cudaSuccess) {
        error = "cannot reserve shared memory for the tensor-core contraction";
        return RTACX_ERR_CUDA;
    }
    return RTACX_OK;
}

// C + z M N (z < g.parts()) = partial products of the planned contraction (added
// into a zeroed C where g.adds()), in
// A's and B's current values (16-byte aligned scales optional).
rtacx_status gemm_split(std::string& error, const GemmPlan& g, const uint16_t* d_blocks, float* C, int M, int N, int K,
                        cudaStream_t stream, uint32_t* err, bool f16, const float* row_scale, const float* col_scale)
{
    const cudaError_t e = launch_chained(split_kernel(g.bn, f16), dim3(N / g.bn, M / BM, g.ksplit), kThreads,
                                         split_smem(g.bn), stream, g.ma, g.mb, C, M, K, N, d_blocks, row_scale, col_scale,
                                         g.adds() ? 1 : 0, (uint32_t)(g.lo_apart ? g.bn : 0), err);
    if(e != cudaSuccess) { cudaGetLastError(); error = std::string("k_gemm_split: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    return RTACX_OK;
}

} // namespace rtacx

namespace {
__device__ uint32_t g_gemm_check_err;
}

// Diagnostic entry point (include/rtacx.h): synchronous C = A * B^T.
extern "C" rtacx_status rtacx_gemm_bf16_tn(const void* A, const void* B, float* C, int M, int N, int K, void* stream)
{
    std::string error;
    uint32_t* err = nullptr;
    if(cudaGetSymbolAddress(reinterpret_cast<void**>(&err), g_gemm_check_err) != cudaSuccess) {
        cudaGetLastError();
        return RTACX_ERR_CUDA;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if(cudaMemsetAsync(err, 0, sizeof(uint32_t), s) != cudaSuccess) { cudaGetLastError(); return RTACX_ERR_CUDA; }
    rtacx_status st = rtacx::gemm_tn(error, A, B, C, M, N, K, s, err);
    if(st != RTACX_OK) return st;
    uint32_t word = 0;
    if(cudaStreamSynchronize(s) != cudaSuccess ||
       cudaMemcpyFromSymbol(&word, g_gemm_check_err, sizeof(word)) != cudaSuccess) {
        cudaGetLastError();
        return RTACX_ERR_CUDA;
    }
    return word ? RTACX_ERR_DEVICE : RTACX_OK;
}
