// sg_kernels.cu — device kernels of the screening surrogate (include/surrogate_b200.h).
//
// The GEMM is the Blackwell tensor-core path: a 128 x BN output tile per CTA
// (BN = 64, 128 or 256), K consumed 64 bf16 at a time through a ring of
// shared-memory buffers that TMA fills (128-byte swizzled, the layout tcgen05
// reads), one elected thread issuing tcgen05.mma into an fp32 accumulator in
// tensor memory, and all eight warps reading it back (tcgen05.ld) for the fused
// epilogue (bias, ReLU, ReLU-derivative mask, fp32 or bf16 store).
// The weight gradients dY^T X are the same path with both operands MN-major, so
// that the row-major activations are read as they lie, and with those of all
// layers in one launch.
// The other kernels are the surrogate's memory-bound glue: patch gathers for
// the convolutions and their adjoint, transposes, column sums, Adam and the loss.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <mutex>

#include "sg_tc.cuh"
#include "surrogate_b200.h"

namespace {

constexpr int kBM = 128;
constexpr int kBK = 64;  // bf16 per 128-byte swizzled row
// Deepest operand ring: enough 64-deep K slices in flight to cover a TMA round
// trip behind the MMAs of the slices before it (24, 32 and 48 KB a stage).
template <int BN>
__host__ __device__ constexpr int max_stages() { return BN >= 256 ? 4 : BN >= 128 ? 6 : 8; }
template <int BN>
__host__ __device__ constexpr int stage_bytes() { return kBM * kBK * 2 + BN * kBK * 2; }

struct GemmArgs {
    int M, N, K;
    void* D;
    int ldd, d_bf16;
    const float* bias;
    int relu;
    const __nv_bfloat16* mask;
    int ldm;
    int* err;
    int stages;          // depth of the operand ring
    const float* cinit;  // accumulators start at row crow[m] of cinit (row stride ldc), or 0 when NULL
    const int* crow;
    int ldc;
};

// Words of one epilogue row in shared memory: 32 columns, padded so that 16-byte
// accesses by rows and by columns fall on different banks.
constexpr int kGemmWarps = 8;
constexpr int kEpiLd = 36;
constexpr size_t kEpiBytes = kGemmWarps * 32 * kEpiLd * sizeof(float);

// The operand ring, which the epilogue's staging reuses, and the barriers.
template <int BN>
__host__ __device__ constexpr size_t ring_bytes(int stages) {
    return (size_t)stages * stage_bytes<BN>() > kEpiBytes ? (size_t)stages * stage_bytes<BN>() : kEpiBytes;
}
template <int BN>
constexpr size_t gemm_smem_bytes(int stages) {
    return 1024 + ring_bytes<BN>(stages) + 256;
}

static_assert(gemm_smem_bytes<64>(max_stages<64>()) <= 232448 && gemm_smem_bytes<128>(max_stages<128>()) <= 232448 &&
                  gemm_smem_bytes<256>(max_stages<256>()) <= 232448,
              "operand ring above the 227 KB of shared memory a CTA may use");

template <int BN>
__global__ void __launch_bounds__(32 * kGemmWarps, 4)
    gemm_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const GemmArgs g) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = smem_raw + ((1024u - (sg::smem_addr(smem_raw) & 1023u)) & 1023u);
    const int kStages = g.stages;
    constexpr uint32_t kABytes = kBM * kBK * 2, kBBytes = BN * kBK * 2, kStage = kABytes + kBBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + ring_bytes<BN>(kStages));
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);
    const uint32_t sbase = sg::smem_addr(base);
    const uint32_t bar0 = sg::smem_addr(bars);
    auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
    auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(kStages + s); };
    const uint32_t done = bar0 + 8u * (uint32_t)(2 * kStages);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // uniform over the warp
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;  // M tiles on x: no 65535 limit on M
    const int nk = (g.K + kBK - 1) / kBK;

    // The first loads need the barriers alone, so they go out while another warp
    // allocates the accumulator (1,200 cycles to there).
    const int first = min(nk, kStages);
    auto load = [&](int s, int kb) {
        sg::mbar_expect_tx(full(s), kStage);
        sg::tma_load_2d(sbase + (uint32_t)s * kStage, &ta, full(s), kb * kBK, m0);
        sg::tma_load_2d(sbase + (uint32_t)s * kStage + kABytes, &tb, full(s), kb * kBK, n0);
    };
    if (warp == 0) {
        if (sg::elect_one()) {
            sg::tma_prefetch(&ta);
            sg::tma_prefetch(&tb);
            for (int s = 0; s < kStages; ++s) {
                sg::mbar_init(full(s), 1);
                sg::mbar_init(empty(s), 1);
            }
            sg::mbar_init(done, 1);
            sg::mbar_fence_init();
            sg::fence_proxy_async();
            for (int s = 0; s < first; ++s) load(s, s);
        }
        __syncwarp();
    } else if (warp == 1) {
        sg::tmem_alloc(sg::smem_addr(tmem_slot), (uint32_t)BN);
        sg::tmem_relinquish();
    }
    sg::tc_fence_before();
    __syncthreads();
    sg::tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    if (g.cinit) {
        // the accumulators' start: a lane writes its row, a warp every second 32 columns
        const int gm = m0 + (warp & 3) * 32 + lane;
        const float* c = gm < g.M ? g.cinit + (size_t)(g.crow ? g.crow[gm] : gm) * g.ldc : nullptr;
#pragma unroll 1
        for (int cc = (warp >> 2) * 32; cc < BN; cc += 64) {
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = c && n0 + cc + j < g.N ? c[n0 + cc + j] : 0.0f;
            sg::tmem_st32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cc, v);
        }
        sg::tc_fence_before();
        __syncthreads();
        sg::tc_fence_after();
    }

    bool ok = true;
    if (warp == 0) {
        // TMA producer: stage s is refilled once the MMAs that read it have completed
        const bool one = sg::elect_one();
        int s = 0;
        uint32_t ph = 0u;
        for (int kb = first; kb < nk; ++kb) {
            if (!__all_sync(0xffffffffu, sg::mbar_wait(empty(s), ph))) {
                ok = false;
                break;
            }
            if (one) load(s, kb);
            __syncwarp();
            if (++s == kStages) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        // MMA issuer: four K=16 steps per stage, advancing 32 bytes inside the swizzle atom
        constexpr uint32_t idesc = sg::idesc_bf16_f32(kBM, BN);
        const bool one = sg::elect_one();
        const uint64_t d0 = sg::desc_kmajor_sw128(0u);
        int s = 0;
        uint32_t ph = 0u;
        for (int kb = 0; kb < nk; ++kb) {
            if (!__all_sync(0xffffffffu, sg::mbar_wait(full(s), ph))) {
                ok = false;
                break;
            }
            sg::tc_fence_after();
            const uint64_t a = d0 | ((sbase + (uint32_t)s * kStage) >> 4), b = a + (kABytes >> 4);
            if (one) {
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k)
                    sg::mma_bf16(tmem, a + 2u * k, b + 2u * k, idesc, (kb > 0 || k > 0 || g.cinit) ? 1u : 0u);
                sg::mma_commit(empty(s));
            }
            __syncwarp();
            if (++s == kStages) {
                s = 0;
                ph ^= 1u;
            }
        }
        // arrives once every MMA issued above has completed (also after a failed wait)
        if (one) sg::mma_commit(done);
    }
    __syncwarp();

    // epilogue: warps w and w + 4 share accumulator rows 32 w .. + 31, a row per lane
    // (TMEM lane), and take 32 columns in turn.  The columns go through the warp's
    // slice of shared memory (the operand ring, which every MMA has left), so that
    // its lanes store whole lines of a row instead of 16 bytes in each of 32 rows,
    // and four columns a lane, since a warp that is alone on its scheduler pays for
    // every instruction: a row a step took 3,000 cycles for 32 x 32 values, longer
    // than the K loop of most layers.  The 65536 x 320 fp32 gradient of the second
    // convolution's patches, 84 MB: 22.6 us (83 from the accumulator's rows, 24.7 a
    // row a step); 8192 x 512 x 512: 10.4 (12.4 a row a step).
    const bool got = sg::mbar_wait(done, 0);
    sg::tc_fence_after();
    if ((!ok || !got) && lane == 0) atomicExch(g.err, 1);
    __syncthreads();  // every warp has left its wait on the ring
    float* st = reinterpret_cast<float*>(base) + warp * 32 * kEpiLd;
    const int row0 = m0 + (warp & 3) * 32;
    const int rows = got ? min(32, g.M - row0) : 0;
    // four columns a lane where rows of D and of the mask allow aligned stores and loads
    auto quad = [](const void* p, int ld, int bytes) {
        return ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & (4u * bytes - 1u)) == 0;
    };
    const bool quads = quad(g.D, g.ldd, g.d_bf16 ? 2 : 4) && (!g.mask || quad(g.mask, g.ldm, 2));
#pragma unroll 1
    for (int c = (warp >> 2) * 32; c < BN && n0 + c < g.N; c += 64) {
        const bool wide = quads && n0 + c + 32 <= g.N;
        const int qc = n0 + c + 4 * (lane & 7), qr = lane >> 3;  // the lane's columns and first row
        float bq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint2 mk[8];
        if (wide) {  // on their way while the accumulator is read
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (g.bias) bq[j] = g.bias[qc + j];
            if (g.mask)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    mk[i] = 4 * i + qr < rows
                                ? *reinterpret_cast<const uint2*>(g.mask + (size_t)(row0 + 4 * i + qr) * g.ldm + qc)
                                : make_uint2(0u, 0u);
        }
        {
            float v[32];
            sg::tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, v);
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(st + lane * kEpiLd + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        }
        __syncwarp();
        auto finish = [&](float x, float b, int gm, int col) {
            if (g.bias) x += b;
            if (g.relu) x = fmaxf(x, 0.0f);
            if (g.mask && !(__bfloat162float(g.mask[(size_t)gm * g.ldm + col]) > 0.0f)) x = 0.0f;
            return x;
        };
        if (wide) {
            auto live = [](uint32_t bf16_bits) { return __uint_as_float(bf16_bits) > 0.0f; };
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int rr = 4 * i + qr;
                float4 x = *reinterpret_cast<const float4*>(st + rr * kEpiLd + 4 * (lane & 7));
                if (g.bias) x.x += bq[0], x.y += bq[1], x.z += bq[2], x.w += bq[3];
                if (g.relu)
                    x.x = fmaxf(x.x, 0.0f), x.y = fmaxf(x.y, 0.0f), x.z = fmaxf(x.z, 0.0f), x.w = fmaxf(x.w, 0.0f);
                if (g.mask) {
                    if (!live(mk[i].x << 16)) x.x = 0.0f;
                    if (!live(mk[i].x & 0xffff0000u)) x.y = 0.0f;
                    if (!live(mk[i].y << 16)) x.z = 0.0f;
                    if (!live(mk[i].y & 0xffff0000u)) x.w = 0.0f;
                }
                const size_t o = (size_t)(row0 + rr) * g.ldd + qc;
                if (rr < rows) {
                    if (g.d_bf16) {
                        __nv_bfloat162 h[2] = {__floats2bfloat162_rn(x.x, x.y), __floats2bfloat162_rn(x.z, x.w)};
                        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(g.D) + o) =
                            *reinterpret_cast<const uint2*>(h);
                    } else {
                        *reinterpret_cast<float4*>(reinterpret_cast<float*>(g.D) + o) = x;
                    }
                }
            }
        } else {
            const int col = n0 + c + lane;
            if (col < g.N) {
                const float b = g.bias ? g.bias[col] : 0.0f;
                for (int r0 = 0; r0 < rows; r0 += 8) {
                    float x[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[i] = st[(r0 + i) * kEpiLd + lane];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = r0 + i;
                        if (r >= rows) break;
                        const float y = finish(x[i], b, row0 + r, col);
                        const size_t o = (size_t)(row0 + r) * g.ldd + col;
                        if (g.d_bf16)
                            reinterpret_cast<__nv_bfloat16*>(g.D)[o] = __float2bfloat16_rn(y);
                        else
                            reinterpret_cast<float*>(g.D)[o] = y;
                    }
                }
            }
        }
        __syncwarp();  // the next columns overwrite the slice
    }
    sg::tc_fence_before();
    __syncthreads();
    if (warp == 1) sg::tmem_dealloc(tmem, (uint32_t)BN);
}

// ─── tensor maps ────────────────────────────────────────────────────────────
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// Row-major bf16 (rows, cols) with row stride ld (elements), boxes of box_rows x
// box_cols (16, 32 or 64), swizzled over their width.
bool make_map_box(CUtensorMap* map, const void* ptr, int rows, int cols, int ld, int box_rows, int box_cols) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const CUtensorMapSwizzle swizzle = box_cols == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
                                       : box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                        : CU_TENSOR_MAP_SWIZZLE_32B;
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_map(CUtensorMap* map, const void* ptr, int rows, int cols, int ld, int box_rows) {
    return make_map_box(map, ptr, rows, cols, ld, box_rows, kBK);
}

template <int BN>
int launch_gemm(GemmArgs g, const void* A, int lda, const void* B, int ldb, cudaStream_t st) {
    CUtensorMap ta, tb;
    if (!make_map(&ta, A, g.M, g.K, lda, kBM) || !make_map(&tb, B, g.N, g.K, ldb, BN)) return SG_ERR_CUDA;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] {
        attr = cudaFuncSetAttribute(gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)gemm_smem_bytes<BN>(max_stages<BN>()));
    });
    if (attr != cudaSuccess) return SG_ERR_CUDA;
    dim3 grid((g.M + kBM - 1) / kBM, (g.N + BN - 1) / BN);
    // the ring is as deep as K needs; with more tiles than SMs it leaves room for a
    // second CTA, whose loads and MMAs run under the first one's epilogue
    g.stages = std::min((g.K + kBK - 1) / kBK, max_stages<BN>());
    if ((long long)grid.x * grid.y > 148) g.stages = std::min(g.stages, 100 * 1024 / stage_bytes<BN>());
    gemm_kernel<BN><<<grid, 32 * kGemmWarps, gemm_smem_bytes<BN>(g.stages), st>>>(ta, tb, g);
    return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ─── weight gradients ───────────────────────────────────────────────────────
// G (N, K) = dY^T X and gb (N) = column sums of dY over R rows, for several layers
// in one launch.  Both operands are read row by row, which is the MN-major layout
// of tcgen05, so nothing is transposed: X's columns are the M dimension of a tile
// (wa of them), dY's the N dimension (wb).  Every sum runs over the rows in order,
// sixteen at a time, as the product of the transposed operands (sg_gemm) does, and
// the column sums keep sg_colsum's order: the same bits.
//
// What bounds it: the chain of the longest layer.  The first convolution's gradient
// for 256 patches is 32 x 64 entries over 262,144 rows, 16,384 MMAs one after
// another on one accumulator, and the operands pass through one SM; narrow tiles
// (16 + 16 columns, 64 bytes a row) keep that stream small, and the other layers'
// tiles run on the other SMs meanwhile.  One layer at a time, with two transposes,
// a product and a column sum each, the eight layers of a training step on 256
// patches took 5.2 ms (the first layer's product 1.19 ms and column sums 2.70 ms);
// in one launch 0.43 ms, which is the first layer's chain.
constexpr int kWgMaxJobs = 16;
constexpr int kWgThreads = 256;
constexpr int kWgRing = 192 * 1024;  // operand ring
constexpr int kWgMaxStages = 12;

struct WgJob {
    CUtensorMap tx, ty;
    int R, N, K;
    int wa, wb;       // tile columns of X (16, 32, 64 or 128: two boxes of 64) and of dY (32 or 64)
    int rows;         // rows of a stage
    int stages;
    int mt;           // tiles along K
    int first;        // first CTA
    float *G, *gb;
};
struct WgBatch {
    WgJob job[kWgMaxJobs];
    int count;
    int* err;
};

constexpr size_t kWgSmem = 1024 + kWgRing + 256 + 8 * 64 * sizeof(float);
static_assert(kWgSmem <= 232448 && 2 * kWgMaxStages + 1 <= 28, "weight-gradient ring and its barriers");

// Warp 0 loads, warp 1 issues the MMAs, warps 4 to 7 sum columns; warps 0 to 3 store.
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_kernel(const __grid_constant__ WgBatch w) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* base = smem_raw + ((1024u - (sg::smem_addr(smem_raw) & 1023u)) & 1023u);
    int ji = 0;
    while (ji + 1 < w.count && (int)blockIdx.x >= w.job[ji + 1].first) ++ji;
    const WgJob& g = w.job[ji];
    const int tile = (int)blockIdx.x - g.first;
    const int m0 = tile % g.mt * g.wa, n0 = tile / g.mt * g.wb;
    const bool sums = m0 == 0;  // this CTA also sums dY's columns
    const int abox = min(g.wa, 64);                       // columns of a box of X
    const uint32_t pa = 2u * abox, pb = 2u * g.wb;        // bytes of a box row
    const uint32_t abytes = (uint32_t)g.rows * pa, bbytes = (uint32_t)g.rows * pb;
    const uint32_t aall = abytes * (g.wa / abox), stage = aall + bbytes;
    const int kStages = g.stages;
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + kWgRing);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
    float* part = reinterpret_cast<float*>(bars + 32);  // [8][64] column sums of the row classes
    const uint32_t sbase = sg::smem_addr(base), bar0 = sg::smem_addr(bars);
    auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
    auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(kStages + s); };
    const uint32_t done = bar0 + 8u * (uint32_t)(2 * kStages);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // uniform over the warp
    const int nk = (g.R + g.rows - 1) / g.rows;
    const int rows = g.rows;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            sg::mbar_init(full(s), 1);
            sg::mbar_init(empty(s), sums ? 5 : 1);  // the MMAs, and the four summing warps
        }
        sg::mbar_init(done, 1);
        sg::mbar_fence_init();
        sg::tma_prefetch(&g.tx);
        sg::tma_prefetch(&g.ty);
    }
    if (warp == 0) {
        sg::tmem_alloc(sg::smem_addr(tmem_slot), 64u);
        sg::tmem_relinquish();
    }
    sg::tc_fence_before();
    __syncthreads();
    sg::tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
    bool ok = true;
    if (warp == 0) {
        const bool one = sg::elect_one();
        int s = 0;
        uint32_t ph = 1u;
        for (int kb = 0; kb < nk; ++kb) {
            if (!__all_sync(0xffffffffu, sg::mbar_wait(empty(s), ph))) {
                ok = false;
                break;
            }
            if (one) {
                sg::mbar_expect_tx(full(s), stage);
                const uint32_t d = sbase + (uint32_t)s * stage;
                sg::tma_load_2d(d, &g.tx, full(s), m0, kb * rows);
                if (g.wa > 64) sg::tma_load_2d(d + abytes, &g.tx, full(s), m0 + 64, kb * rows);
                sg::tma_load_2d(d + aall, &g.ty, full(s), n0, kb * rows);
            }
            __syncwarp();
            if (++s == kStages) {
                s = 0;
                ph ^= 1u;
            }
        }
    } else if (warp == 1) {
        const bool one = sg::elect_one();
        // the accumulator has 64 rows (128 for two boxes of X) whatever wa is: with
        // one narrow box the M blocks all read that box (leading offset 0), and
        // their copies are not stored
        const uint32_t idesc = sg::idesc_bf16_f32_mn(g.wa > 64 ? 128 : 64, g.wb);
        const uint64_t ad = sg::desc_mnmajor(0u, pa, g.wa > 64 ? abytes : 0u), bd = sg::desc_mnmajor(0u, pb, 0u);
        const uint32_t astep = 16u * pa >> 4, bstep = 16u * pb >> 4;  // 16 rows of K
        int s = 0;
        uint32_t ph = 0u;
        for (int kb = 0; kb < nk; ++kb) {
            if (!__all_sync(0xffffffffu, sg::mbar_wait(full(s), ph))) {
                ok = false;
                break;
            }
            sg::tc_fence_after();
            uint64_t a = ad | ((sbase + (uint32_t)s * stage) >> 4), b = bd | ((sbase + (uint32_t)s * stage + aall) >> 4);
            if (one) {
                for (int k = 0; k < rows / 64; ++k) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        sg::mma_bf16(tmem, a, b, idesc, (kb > 0 || k > 0 || u > 0) ? 1u : 0u);
                        a += astep;
                        b += bstep;
                    }
                }
                sg::mma_commit(empty(s));
            }
            __syncwarp();
            if (++s == kStages) {
                s = 0;
                ph ^= 1u;
            }
        }
        if (one) sg::mma_commit(done);
    } else if (warp >= 4 && sums) {
        // column sums from the staged tiles: row class y = r mod 8 of two columns a
        // thread and turn, each class summed in row order, then the classes in order
        const int t = threadIdx.x - 128, y = t & 7, c0 = t >> 3, pairs = g.wb / 2;
        const uint32_t swz = pb == 128u ? 7u : pb == 64u ? 3u : 1u;
        float acc[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
        int s = 0;
        uint32_t ph = 0u;
        for (int kb = 0; kb < nk; ++kb) {
            if (!__all_sync(0xffffffffu, sg::mbar_wait(full(s), ph))) {
                ok = false;
                break;
            }
            const unsigned char* box = base + (size_t)s * stage + aall;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (c0 + 16 * u >= pairs) break;
                // rows 8 apart have the same swizzle
                uint32_t o = (uint32_t)y * pb + 4u * (uint32_t)(c0 + 16 * u);
                o ^= ((o >> 7) & swz) << 4;
                const unsigned char* q = box + o;
                for (int i = 0; i < rows / 8; i += 8, q += 64u * pb) {  // eight reads ahead of their sums
                    uint32_t v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = *reinterpret_cast<const uint32_t*>(q + (uint32_t)j * 8u * pb);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        acc[u][0] += __uint_as_float(v[j] << 16);
                        acc[u][1] += __uint_as_float(v[j] & 0xffff0000u);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) sg::mbar_arrive(empty(s));
            if (++s == kStages) {
                s = 0;
                ph ^= 1u;
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (c0 + 16 * u < pairs) {
                part[y * 64 + 2 * (c0 + 16 * u)] = acc[u][0];
                part[y * 64 + 2 * (c0 + 16 * u) + 1] = acc[u][1];
            }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (t < g.wb && n0 + t < g.N) {
            float sum = 0.0f;
            for (int j = 0; j < 8; ++j) sum += part[j * 64 + t];
            g.gb[n0 + t] = sum;
        }
    }
    __syncwarp();
    const bool got = sg::mbar_wait(done, 0);
    sg::tc_fence_after();
    if ((!ok || !got) && lane == 0) atomicExch(w.err, 1);
    if (warp < 4) {
        // TMEM lane = column of X (an accumulator of 64 rows has 16 in each warp's
        // lanes): for each column of dY the lanes store consecutive words
        const int ml = g.wa > 64 ? warp * 32 + lane : warp * 16 + lane, m = m0 + ml;
        const bool mine = got && (g.wa > 64 || lane < 16) && ml < g.wa && m < g.K;
#pragma unroll 1
        for (int c = 0; c < g.wb && n0 + c < g.N; c += 32) {
            float v[32];
            sg::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
            if (!mine) continue;
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (c + j < g.wb && n0 + c + j < g.N) g.G[(size_t)(n0 + c + j) * g.K + m] = v[j];
        }
    }
    sg::tc_fence_before();
    __syncthreads();
    if (warp == 0) sg::tmem_dealloc(tmem, 64u);
}

// ─── glue kernels ───────────────────────────────────────────────────────────
// The rows of the kernels below are counted in unsigned: up to 2^31 of them and a
// step of the grid beyond stay in range.
// im2col for channel counts that are multiples of 8: a thread per 16-byte chunk of
// a patch row, which lies within one tap.  blockDim.x is the chunks of a row, so
// that a thread's tap and channel stay the same and its rows advance.  The
// second convolution of 256 patches, 42 MB written: 14.4 us.  (A thread per bf16
// with 64-bit divisions: 147 us.)
__global__ void im2col8_kernel(int rows, int H, int W, int C, const __nv_bfloat16* __restrict__ X, int kpad,
                               __nv_bfloat16* __restrict__ cols) {
    const unsigned Ho = H / 2, Wo = W / 2;
    const int k = threadIdx.x * 8, t = k / C, c = k % C, ky = t / 3, kx = t % 3;
    const bool live = k < 9 * C;
    for (unsigned r = blockIdx.x * blockDim.y + threadIdx.y; r < (unsigned)rows; r += gridDim.x * blockDim.y) {
        const unsigned ox = r % Wo, q = r / Wo, oy = q % Ho, b = q / Ho;
        const int iy = 2 * (int)oy - 1 + ky, ix = 2 * (int)ox - 1 + kx;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (live && iy >= 0 && iy < H && ix >= 0 && ix < W)
            v = *reinterpret_cast<const uint4*>(X + (((size_t)b * H + iy) * W + ix) * C + c);
        *reinterpret_cast<uint4*>(cols + (size_t)r * kpad + k) = v;
    }
}

// The same for one channel: chunk 0 holds taps 0..7, chunk 1 tap 8, the rest zeros.
__global__ void im2col1_kernel(int rows, int H, int W, const __nv_bfloat16* __restrict__ X, int kpad,
                               __nv_bfloat16* __restrict__ cols) {
    const unsigned Ho = H / 2, Wo = W / 2;
    const int k = threadIdx.x * 8;
    for (unsigned r = blockIdx.x * blockDim.y + threadIdx.y; r < (unsigned)rows; r += gridDim.x * blockDim.y) {
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __float2bfloat16_rn(0.0f);
        if (k < 9) {
            const unsigned ox = r % Wo, q = r / Wo, oy = q % Ho, b = q / Ho;
            const __nv_bfloat16* img = X + (size_t)b * H * W;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int t = k + j, iy = 2 * (int)oy - 1 + t / 3, ix = 2 * (int)ox - 1 + t % 3;
                if (t < 9 && iy >= 0 && iy < H && ix >= 0 && ix < W) v[j] = img[(size_t)iy * W + ix];
            }
        }
        *reinterpret_cast<uint4*>(cols + (size_t)r * kpad + k) = *reinterpret_cast<const uint4*>(v);
    }
}

// col2im for channel counts that are multiples of 8: a thread per 8 channels of a
// pixel, the taps in the same (ky, kx) order.  The second
// convolution's 84 MB of patch gradients: 27 us.  (A thread per channel: 90 us.)
__global__ void col2im8_kernel(int pixels, int H, int W, int C, const float* __restrict__ dcols, int kpad,
                               const __nv_bfloat16* __restrict__ act, __nv_bfloat16* __restrict__ dX) {
    const unsigned Ho = H / 2, Wo = W / 2;
    const int c = threadIdx.x * 8;
    for (unsigned p = blockIdx.x * blockDim.y + threadIdx.y; p < (unsigned)pixels; p += gridDim.x * blockDim.y) {
        const unsigned ix = p % W, q = p / W, iy = q % H, b = q / H;
        float s[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int ky = 0; ky < 3; ++ky) {
            const int ty = (int)iy + 1 - ky;
            if (ty < 0 || (ty & 1) || (ty >> 1) >= (int)Ho) continue;
            for (int kx = 0; kx < 3; ++kx) {
                const int tx = (int)ix + 1 - kx;
                if (tx < 0 || (tx & 1) || (tx >> 1) >= (int)Wo) continue;
                const size_t row = ((size_t)b * Ho + (ty >> 1)) * Wo + (tx >> 1);
                const float4* d = reinterpret_cast<const float4*>(dcols + row * kpad + (ky * 3 + kx) * C + c);
                const float4 x = d[0], y = d[1];
                s[0] += x.x;
                s[1] += x.y;
                s[2] += x.z;
                s[3] += x.w;
                s[4] += y.x;
                s[5] += y.y;
                s[6] += y.z;
                s[7] += y.w;
            }
        }
        const size_t o = (size_t)p * C + c;
        if (act) {
            const uint4 w = *reinterpret_cast<const uint4*>(act + o);
            const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&w);
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (!(__bfloat162float(h[j]) > 0.0f)) s[j] = 0.0f;
        }
        __nv_bfloat162 h2[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) h2[j] = __floats2bfloat162_rn(s[2 * j], s[2 * j + 1]);
        *reinterpret_cast<uint4*>(dX + o) = *reinterpret_cast<const uint4*>(h2);
    }
}

// One Adam step on several matrices: a CTA per tile of 32 rows x 64 columns, four
// columns a thread, the bf16 transpose through shared memory (written 64 bytes at
// a time; straight from the rows it was 2 bytes in each of 32 lines).
constexpr int kAdamMax = 32;
struct AdamBatch {
    SgAdamParam q[kAdamMax];
    int first[kAdamMax + 1];  // first tile of each matrix
    int count;
};

__global__ void __launch_bounds__(256) adam_batch_kernel(const __grid_constant__ AdamBatch a, float lr, float b1, float b2,
                                                         float eps, float c1, float c2) {
    __shared__ __nv_bfloat16 tile[32][66];
    int i = 0;
    while (i + 1 < a.count && (int)blockIdx.x >= a.first[i + 1]) ++i;
    const SgAdamParam& q = a.q[i];
    const int tiles_c = (q.cols + 63) / 64, t = (int)blockIdx.x - a.first[i];
    const int r0 = t / tiles_c * 32, c0 = t % tiles_c * 64;
    __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(q.w);
    __nv_bfloat16* wt = reinterpret_cast<__nv_bfloat16*>(q.wt);
    float* p = reinterpret_cast<float*>(q.p);
    const float* g = reinterpret_cast<const float*>(q.g);
    float *m = reinterpret_cast<float*>(q.m), *v = reinterpret_cast<float*>(q.v);
    auto one = [&](float pi, float gi, float& mi, float& vi) {
        mi = b1 * mi + (1.0f - b1) * gi;
        vi = b2 * vi + (1.0f - b2) * gi * gi;
        return pi - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    };
    const bool vec = (q.cols % 4) == 0 &&
                     ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
                       reinterpret_cast<uintptr_t>(v)) & 15u) == 0;
    for (int rr = threadIdx.x / 16; rr < 32; rr += 16) {
        const int r = r0 + rr, cc = (threadIdx.x % 16) * 4, c = c0 + cc;
        if (r >= q.rows || c >= q.cols) continue;
        const size_t o = (size_t)r * q.cols + c;
        if (vec) {
            float4 pi = *reinterpret_cast<float4*>(p + o), mi = *reinterpret_cast<float4*>(m + o),
                   vi = *reinterpret_cast<float4*>(v + o);
            const float4 gi = *reinterpret_cast<const float4*>(g + o);
            pi.x = one(pi.x, gi.x, mi.x, vi.x);
            pi.y = one(pi.y, gi.y, mi.y, vi.y);
            pi.z = one(pi.z, gi.z, mi.z, vi.z);
            pi.w = one(pi.w, gi.w, mi.w, vi.w);
            *reinterpret_cast<float4*>(p + o) = pi;
            *reinterpret_cast<float4*>(m + o) = mi;
            *reinterpret_cast<float4*>(v + o) = vi;
            const float x[4] = {pi.x, pi.y, pi.z, pi.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) tile[rr][cc + j] = __float2bfloat16_rn(x[j]);
        } else {
            for (int j = 0; j < 4 && c + j < q.cols; ++j) {
                float mi = m[o + j], vi = v[o + j];
                const float pi = one(p[o + j], g[o + j], mi, vi);
                p[o + j] = pi;
                m[o + j] = mi;
                v[o + j] = vi;
                tile[rr][cc + j] = __float2bfloat16_rn(pi);
            }
        }
    }
    __syncthreads();
    for (int x = threadIdx.x; x < 32 * 64; x += 256) {
        const int rr = x / 64, cc = x % 64;
        if (r0 + rr < q.rows && c0 + cc < q.cols) w[(size_t)(r0 + rr) * q.ldw + c0 + cc] = tile[rr][cc];
    }
    if (!wt) return;
    for (int x = threadIdx.x; x < 32 * 64; x += 256) {
        const int rr = x % 32, cc = x / 32;
        if (r0 + rr < q.rows && c0 + cc < q.cols) wt[(size_t)(c0 + cc) * q.ldwt + r0 + rr] = tile[rr][cc];
    }
}

__global__ void im2col_kernel(int B, int H, int W, int C, const __nv_bfloat16* __restrict__ X, int kpad,
                              __nv_bfloat16* __restrict__ cols) {
    const int Ho = H / 2, Wo = W / 2;
    const long long total = (long long)B * Ho * Wo * kpad;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(i % kpad);
        const long long r = i / kpad;
        __nv_bfloat16 v = __float2bfloat16_rn(0.0f);
        if (k < 9 * C) {
            const int c = k % C, t = k / C, kx = t % 3, ky = t / 3;
            const int ox = (int)(r % Wo), oy = (int)((r / Wo) % Ho), b = (int)(r / ((long long)Wo * Ho));
            const int iy = 2 * oy - 1 + ky, ix = 2 * ox - 1 + kx;
            if (iy >= 0 && iy < H && ix >= 0 && ix < W) v = X[(((long long)b * H + iy) * W + ix) * C + c];
        }
        cols[i] = v;
    }
}

__global__ void col2im_kernel(int B, int H, int W, int C, const float* __restrict__ dcols, int kpad,
                              const __nv_bfloat16* __restrict__ act, __nv_bfloat16* __restrict__ dX) {
    const int Ho = H / 2, Wo = W / 2;
    const long long total = (long long)B * H * W * C;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i % C);
        const long long p = i / C;
        const int ix = (int)(p % W), iy = (int)((p / W) % H), b = (int)(p / ((long long)W * H));
        float s = 0.0f;
        // patches (oy, ox) with iy = 2 oy - 1 + ky, ix = 2 ox - 1 + kx, in (ky, kx) order
        for (int ky = 0; ky < 3; ++ky) {
            const int ty = iy + 1 - ky;
            if (ty < 0 || (ty & 1) || (ty >> 1) >= Ho) continue;
            for (int kx = 0; kx < 3; ++kx) {
                const int tx = ix + 1 - kx;
                if (tx < 0 || (tx & 1) || (tx >> 1) >= Wo) continue;
                const long long row = ((long long)b * Ho + (ty >> 1)) * Wo + (tx >> 1);
                s += dcols[row * kpad + (ky * 3 + kx) * C + c];
            }
        }
        if (act && !(__bfloat162float(act[i]) > 0.0f)) s = 0.0f;
        dX[i] = __float2bfloat16_rn(s);
    }
}

__global__ void transpose_kernel(int rows, int cols, const __nv_bfloat16* __restrict__ in, int ld_in,
                                 __nv_bfloat16* __restrict__ out, int ld_out) {
    __shared__ __nv_bfloat16 tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = by + j, c = bx + threadIdx.x;
        if (r < rows && c < cols) tile[j][threadIdx.x] = in[(size_t)r * ld_in + c];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int c = bx + j, r = by + threadIdx.x;
        if (r < rows && c < cols) out[(size_t)c * ld_out + r] = tile[threadIdx.x][j];
    }
}

// column sums: block (x) = 32 columns, threads (32, 8) walk the rows in a
// fixed interleave, then the 8 partial sums of a column are added in order
__global__ void colsum_kernel(int rows, int cols, const void* __restrict__ in, int ld, int in_bf16,
                              float* __restrict__ out) {
    __shared__ float part[8][33];
    const int c = blockIdx.x * 32 + threadIdx.x;
    float s = 0.0f;
    if (c < cols) {
        for (int r = threadIdx.y; r < rows; r += 8) {
            const size_t o = (size_t)r * ld + c;
            s += in_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(in)[o])
                         : reinterpret_cast<const float*>(in)[o];
        }
    }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && c < cols) {
        float t = 0.0f;
        for (int j = 0; j < 8; ++j) t += part[j][threadIdx.x];
        out[c] = t;
    }
}

__global__ void adam_kernel(int rows, int cols, float* __restrict__ p, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2, float eps,
                            float c1, float c2, __nv_bfloat16* __restrict__ w, int ldw, __nv_bfloat16* __restrict__ wt,
                            int ldwt) {
    const long long n = (long long)rows * cols;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        const int r = (int)(i / cols), c = (int)(i % cols);
        const __nv_bfloat16 h = __float2bfloat16_rn(pi);
        w[(size_t)r * ldw + c] = h;
        if (wt) wt[(size_t)c * ldwt + r] = h;
    }
}

// one block: each thread sums a strided share, then a fixed-order tree
__global__ void mse_kernel(int rows, int n_out, const float* __restrict__ pred, int ldp,
                           const float* __restrict__ target, int ldt, __nv_bfloat16* __restrict__ grad, int ldg,
                           float* __restrict__ loss) {
    __shared__ float red[1024];
    const float inv = 1.0f / ((float)rows * (float)n_out);
    float s = 0.0f;
    auto entry = [&](int r, int c) {
        float gv = 0.0f;
        if (c < n_out) {
            const float d = pred[(size_t)r * ldp + c] - target[(size_t)r * ldt + c];
            s += d * d;
            gv = 2.0f * d * inv;
        }
        grad[(size_t)r * ldg + c] = __float2bfloat16_rn(gv);
    };
    if (blockDim.x % ldg == 0) {
        // whole rows a step: the same entries for every thread without a division each
        const int c = threadIdx.x % ldg, step = blockDim.x / ldg;
        for (unsigned r = threadIdx.x / ldg; r < (unsigned)rows; r += step) entry((int)r, c);
    } else {
        const long long total = (long long)rows * ldg;
        for (long long i = threadIdx.x; i < total; i += blockDim.x) entry((int)(i / ldg), (int)(i % ldg));
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[0] = red[0] * inv;
}

__global__ void pack_rows_kernel(int rows, int enc_dim, const __nv_bfloat16* __restrict__ enc, int ld_enc,
                                 const int* __restrict__ enc_row, int n_extra, const float* __restrict__ extra,
                                 int ld_extra, __nv_bfloat16* __restrict__ x, int ldx) {
    const long long total = (long long)rows * ldx;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / ldx), c = (int)(i % ldx);
        __nv_bfloat16 v = __float2bfloat16_rn(0.0f);
        if (c < enc_dim) {
            const int er = enc_row ? enc_row[r] : r;
            v = enc[(size_t)er * ld_enc + c];
        } else if (c < enc_dim + n_extra) {
            v = __float2bfloat16_rn(extra[(size_t)r * ld_extra + (c - enc_dim)]);
        }
        x[i] = v;
    }
}

// The same with 8 columns a thread (16-byte stores), a row per step of a block:
// encoder columns are copied 16 bytes at a time.  256 rows of 2304
// in 4.3 us, 8192 of 256 in 5.0.  (A bf16 per thread with 64-bit divisions: 45 us
// for 8192 rows of 2304.)
__global__ void pack_rows8_kernel(int rows, int enc_dim, const __nv_bfloat16* __restrict__ enc, int ld_enc,
                                  const int* __restrict__ enc_row, int n_extra, const float* __restrict__ extra,
                                  int ld_extra, __nv_bfloat16* __restrict__ x, int ldx) {
    for (unsigned r = blockIdx.x * blockDim.y + threadIdx.y; r < (unsigned)rows; r += gridDim.x * blockDim.y) {
        const __nv_bfloat16* er = enc ? enc + (size_t)(enc_row ? enc_row[r] : (int)r) * ld_enc : nullptr;
        for (int c = threadIdx.x * 8; c < ldx; c += blockDim.x * 8) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (c < enc_dim) {
                v = *reinterpret_cast<const uint4*>(er + c);
            } else if (c < enc_dim + n_extra) {
                const float* s = extra + (size_t)r * ld_extra + (c - enc_dim);
                const int m = enc_dim + n_extra - c;
                __nv_bfloat162 h[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    h[j] = __floats2bfloat162_rn(2 * j < m ? s[2 * j] : 0.0f, 2 * j + 1 < m ? s[2 * j + 1] : 0.0f);
                v = *reinterpret_cast<const uint4*>(h);
            }
            *reinterpret_cast<uint4*>(x + (size_t)r * ldx + c) = v;
        }
    }
}

__global__ void unpack_grad_kernel(int rows, int enc_dim, const __nv_bfloat16* __restrict__ dx, int ldx,
                                   const __nv_bfloat16* __restrict__ act, __nv_bfloat16* __restrict__ d_enc) {
    const long long total = (long long)rows * enc_dim;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / enc_dim), c = (int)(i % enc_dim);
        __nv_bfloat16 v = dx[(size_t)r * ldx + c];
        if (act && !(__bfloat162float(act[i]) > 0.0f)) v = __float2bfloat16_rn(0.0f);
        d_enc[i] = v;
    }
}

// out[r, :] = in[idx[r], :], rows of `bytes` bytes (16-byte units when aligned)
__global__ void gather_rows_kernel(int rows, long long bytes, const unsigned char* __restrict__ in, long long ld_in,
                                   const int* __restrict__ idx, unsigned char* __restrict__ out, long long ld_out,
                                   int vec16) {
    const long long per = vec16 ? bytes / 16 : bytes;
    const long long total = (long long)rows * per;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / per);
        const long long o = i % per;
        const unsigned char* src = in + (long long)idx[r] * ld_in;
        unsigned char* dst = out + (long long)r * ld_out;
        if (vec16)
            reinterpret_cast<uint4*>(dst)[o] = reinterpret_cast<const uint4*>(src)[o];
        else
            dst[o] = src[o];
    }
}

__global__ void to_bf16_kernel(long long n, const float* __restrict__ in, __nv_bfloat16* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = __float2bfloat16_rn(in[i]);
}

int grid_for(long long work, int threads = 256) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms < 1) sms = 148;
    }
    const long long b = (work + threads - 1) / threads;
    return (int)std::max<long long>(1, std::min<long long>(b, (long long)sms * 16));
}

int launched() { return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA; }

}  // namespace

extern "C" {

int sg_gemm(int32_t M, int32_t N, int32_t K, const void* A, int32_t lda, const void* B, int32_t ldb, void* D,
            int32_t ldd, int32_t d_dtype, const float* bias, int32_t relu, const void* mask, int32_t ldm, int32_t* err,
            void* stream) {
    return sg_gemm_from(M, N, K, A, lda, B, ldb, D, ldd, d_dtype, bias, relu, mask, ldm, nullptr, nullptr, 0, err, stream);
}

int sg_gemm_from(int32_t M, int32_t N, int32_t K, const void* A, int32_t lda, const void* B, int32_t ldb, void* D,
                 int32_t ldd, int32_t d_dtype, const float* bias, int32_t relu, const void* mask, int32_t ldm,
                 const float* cinit, const int32_t* crow, int32_t ldc, int32_t* err, void* stream) {
    if (cinit && ldc < N) return SG_ERR_INVALID;
    if (M < 1 || N < 1 || K < 1 || !A || !B || !D || !err) return SG_ERR_INVALID;
    if (lda < K || ldb < K || (lda % 8) || (ldb % 8) || !aligned16(A) || !aligned16(B)) return SG_ERR_INVALID;
    if (ldd < N || (d_dtype != SG_OUT_F32 && d_dtype != SG_OUT_BF16)) return SG_ERR_INVALID;
    if (mask && ldm < N) return SG_ERR_INVALID;
    if ((N + 63) / 64 > 65535) return SG_ERR_INVALID;
    GemmArgs g{M, N, K, D, ldd, d_dtype == SG_OUT_BF16 ? 1 : 0, bias, relu ? 1 : 0,
               reinterpret_cast<const __nv_bfloat16*>(mask), ldm, err, 0, cinit, crow, ldc};
    cudaStream_t st = (cudaStream_t)stream;
    if (N <= 64) return launch_gemm<64>(g, A, lda, B, ldb, st);
    // 128 x 256 tiles halve the re-reads of A, but leave fewer CTAs to take turns
    // on an SM, so they want several waves of the 148 SMs: 32768 x 512 x 2304 in 83
    // us against 106 with 128 x 128 tiles, 16384 x 1024 x 1024 in 42 against 47
    // (512 of the wide tiles both); 8192 x 512 x 512 in 10.7 against 10.4 and 8192 x
    // 512 x 256 in 10.4 against 8.3 (128).
    const long long tiles256 = (long long)((M + kBM - 1) / kBM) * ((N + 255) / 256);
    if (N >= 512 && tiles256 >= 512) return launch_gemm<256>(g, A, lda, B, ldb, st);
    // narrow tiles while even those leave SMs without one, half of B and of the
    // epilogue for each CTA: 256 x 512 x 512 in 6.8 us against 8.3, 256 x 512 x 2304 in
    // 10.7 against 12.4, 4096 x 128 x 1152 in 8.3 against 10.4
    if ((long long)((M + kBM - 1) / kBM) * ((N + 63) / 64) <= 148) return launch_gemm<64>(g, A, lda, B, ldb, st);
    return launch_gemm<128>(g, A, lda, B, ldb, st);
}

int sg_im2col(int32_t B, int32_t H, int32_t W, int32_t C, const void* X, int32_t kpad, void* cols, void* stream) {
    if (B < 1 || H < 2 || W < 2 || (H & 1) || (W & 1) || C < 1 || kpad < 9 * C || !X || !cols) return SG_ERR_INVALID;
    const long long rows = (long long)B * (H / 2) * (W / 2);
    cudaStream_t st = (cudaStream_t)stream;
    if (rows <= INT_MAX && kpad % 8 == 0 && kpad / 8 <= 1024 && aligned16(cols) && (C == 1 || (C % 8 == 0 && aligned16(X)))) {
        const dim3 block(kpad / 8, std::max(1, 256 / (kpad / 8)));
        const int grid = (int)std::min<long long>((rows + block.y - 1) / block.y, 148 * 16);
        if (C == 1)
            im2col1_kernel<<<grid, block, 0, st>>>((int)rows, H, W, reinterpret_cast<const __nv_bfloat16*>(X), kpad,
                                                   reinterpret_cast<__nv_bfloat16*>(cols));
        else
            im2col8_kernel<<<grid, block, 0, st>>>((int)rows, H, W, C, reinterpret_cast<const __nv_bfloat16*>(X), kpad,
                                                   reinterpret_cast<__nv_bfloat16*>(cols));
        return launched();
    }
    const long long work = rows * kpad;
    im2col_kernel<<<grid_for(work), 256, 0, (cudaStream_t)stream>>>(
        B, H, W, C, reinterpret_cast<const __nv_bfloat16*>(X), kpad, reinterpret_cast<__nv_bfloat16*>(cols));
    return launched();
}

int sg_conv_forward(int32_t P, int32_t size, const void* x, int32_t count, const SgConvLayer* layers, int32_t* err,
                    void* stream) {
    if (count < 1 || !layers || P < 1 || size < 2) return SG_ERR_INVALID;
    for (int i = 0; i < count; ++i) {
        const SgConvLayer& q = layers[i];
        int rc = sg_im2col(P, size, size, q.cin, x, q.kpad, q.cols, stream);
        size /= 2;
        const long long rows = (long long)P * size * size;
        if (rc == SG_OK && rows > INT_MAX) rc = SG_ERR_INVALID;
        if (rc == SG_OK)
            rc = sg_gemm((int32_t)rows, q.cout, q.kpad, q.cols, q.kpad, q.w, q.ldw, q.act, q.cout, SG_OUT_BF16, q.bias, 1,
                         nullptr, 0, err, stream);
        if (rc != SG_OK) return rc;
        x = q.act;
    }
    return SG_OK;
}

int sg_dense_forward(int32_t rows, const void* x, int32_t ldx, int32_t count, const SgDenseLayer* layers, int32_t* err,
                     void* stream) {
    if (count < 1 || !layers) return SG_ERR_INVALID;
    for (int i = 0; i + 1 < count; ++i)  // the next layer's operand
        if (layers[i].d_dtype != SG_OUT_BF16) return SG_ERR_INVALID;
    for (int i = 0; i < count; ++i) {
        const SgDenseLayer& q = layers[i];
        const int rc = q.cinit ? sg_gemm_from(rows, q.N, q.K, x, ldx, q.w, q.ldw, q.out, q.ldd, q.d_dtype, q.bias, q.relu,
                                              nullptr, 0, q.cinit, q.crow, q.ldc, err, stream)
                               : sg_gemm(rows, q.N, q.K, x, ldx, q.w, q.ldw, q.out, q.ldd, q.d_dtype, q.bias, q.relu,
                                         nullptr, 0, err, stream);
        if (rc != SG_OK) return rc;
        x = q.out;
        ldx = q.ldd;
    }
    return SG_OK;
}

int sg_col2im(int32_t B, int32_t H, int32_t W, int32_t C, const float* dcols, int32_t kpad, const void* act,
              void* dX, void* stream) {
    if (B < 1 || H < 2 || W < 2 || (H & 1) || (W & 1) || C < 1 || kpad < 9 * C || !dcols || !dX) return SG_ERR_INVALID;
    const long long pixels = (long long)B * H * W;
    if (pixels <= INT_MAX && C % 8 == 0 && C / 8 <= 1024 && kpad % 4 == 0 && aligned16(dcols) && aligned16(dX) &&
        (!act || aligned16(act))) {
        const dim3 block(C / 8, std::max(1, 256 / (C / 8)));
        const int grid = (int)std::min<long long>((pixels + block.y - 1) / block.y, 148 * 16);
        col2im8_kernel<<<grid, block, 0, (cudaStream_t)stream>>>((int)pixels, H, W, C, dcols, kpad,
                                                                 reinterpret_cast<const __nv_bfloat16*>(act),
                                                                 reinterpret_cast<__nv_bfloat16*>(dX));
        return launched();
    }
    const long long work = pixels * C;
    col2im_kernel<<<grid_for(work), 256, 0, (cudaStream_t)stream>>>(
        B, H, W, C, dcols, kpad, reinterpret_cast<const __nv_bfloat16*>(act), reinterpret_cast<__nv_bfloat16*>(dX));
    return launched();
}

int sg_transpose(int32_t rows, int32_t cols, const void* in, int32_t ld_in, void* out, int32_t ld_out,
                 void* stream) {
    if (rows < 1 || cols < 1 || !in || !out || ld_in < cols || ld_out < rows) return SG_ERR_INVALID;
    if ((cols + 31) / 32 > 2147483647 || (rows + 31) / 32 > 65535) return SG_ERR_INVALID;
    dim3 grid((cols + 31) / 32, (rows + 31) / 32);
    transpose_kernel<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>(
        rows, cols, reinterpret_cast<const __nv_bfloat16*>(in), ld_in, reinterpret_cast<__nv_bfloat16*>(out), ld_out);
    return launched();
}

int sg_colsum(int32_t rows, int32_t cols, const void* in, int32_t ld, int32_t in_bf16, float* out, void* stream) {
    if (rows < 1 || cols < 1 || !in || !out || ld < cols) return SG_ERR_INVALID;
    colsum_kernel<<<(cols + 31) / 32, dim3(32, 8), 0, (cudaStream_t)stream>>>(rows, cols, in, ld, in_bf16 ? 1 : 0,
                                                                              out);
    return launched();
}

int sg_adam(int32_t rows, int32_t cols, float* p, const float* g, float* m, float* v, float lr, float beta1,
            float beta2, float eps, int32_t t, void* w, int32_t ldw, void* wt, int32_t ldwt, void* stream) {
    if (rows < 1 || cols < 1 || !p || !g || !m || !v || !w || t < 1 || ldw < cols || (wt && ldwt < rows))
        return SG_ERR_INVALID;
    const float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
    adam_kernel<<<grid_for((long long)rows * cols), 256, 0, (cudaStream_t)stream>>>(
        rows, cols, p, g, m, v, lr, beta1, beta2, eps, c1, c2, reinterpret_cast<__nv_bfloat16*>(w), ldw,
        reinterpret_cast<__nv_bfloat16*>(wt), ldwt);
    return launched();
}

int sg_adam_batch(int32_t count, const SgAdamParam* params, float lr, float beta1, float beta2, float eps, int32_t t,
                  void* stream) {
    if (count < 1 || count > kAdamMax || !params || t < 1) return SG_ERR_INVALID;
    AdamBatch a;
    a.count = count;
    a.first[0] = 0;
    for (int i = 0; i < count; ++i) {
        const SgAdamParam& q = params[i];
        if (q.rows < 1 || q.cols < 1 || !q.p || !q.g || !q.m || !q.v || !q.w || q.ldw < q.cols || (q.wt && q.ldwt < q.rows))
            return SG_ERR_INVALID;
        const long long tiles = ((long long)q.rows + 31) / 32 * (((long long)q.cols + 63) / 64);
        if (a.first[i] + tiles > INT_MAX) return SG_ERR_INVALID;
        a.q[i] = q;
        a.first[i + 1] = a.first[i] + (int)tiles;
    }
    const float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
    adam_batch_kernel<<<a.first[count], 256, 0, (cudaStream_t)stream>>>(a, lr, beta1, beta2, eps, c1, c2);
    return launched();
}

int sg_weight_grads(int32_t count, const SgWeightGrad* jobs, int32_t* err, void* stream) {
    if (count < 1 || count > kWgMaxJobs || !jobs || !err) return SG_ERR_INVALID;
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] {
        attr = cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgSmem);
    });
    if (attr != cudaSuccess) return SG_ERR_CUDA;
    WgBatch b;
    b.count = count;
    b.err = err;
    // the layers with the longest chains first, so that their CTAs start first
    int order[kWgMaxJobs];
    for (int i = 0; i < count; ++i) order[i] = i;
    std::stable_sort(order, order + count, [&](int x, int y) { return jobs[x].R > jobs[y].R; });
    long long ctas = 0;
    for (int i = 0; i < count; ++i) {
        const SgWeightGrad& q = jobs[order[i]];
        if (q.R < 1 || q.N < 1 || q.K < 1 || !q.dY || !q.X || !q.G || !q.gb) return SG_ERR_INVALID;
        if (q.ldy < q.N || q.ldx < q.K || (q.ldy % 8) || (q.ldx % 8) || !aligned16(q.dY) || !aligned16(q.X))
            return SG_ERR_INVALID;
        WgJob& g = b.job[i];
        // Tile: the widest whose operand stream through one SM stays under 8.5 MB
        // (of the order of 100 us); narrow ones for the longest chains.
        static const int tiles[4][2] = {{128, 64}, {64, 64}, {32, 32}, {16, 32}};
        int c = 0;
        while (c < 3 && (long long)q.R * 2 * (tiles[c][0] + tiles[c][1]) > 8500000LL) ++c;
        g.wa = tiles[c][0];
        g.wb = tiles[c][1];
        g.R = q.R;
        g.N = q.N;
        g.K = q.K;
        g.G = q.G;
        g.gb = q.gb;
        const int abox = std::min(g.wa, 64);
        g.rows = 64 * 64 / abox;  // a box of 8 KB
        const int stage = 2 * g.rows * (g.wa + g.wb);
        g.stages = std::min(kWgRing / stage, kWgMaxStages);
        g.mt = (q.K + g.wa - 1) / g.wa;
        g.first = (int)ctas;
        ctas += (long long)g.mt * ((q.N + g.wb - 1) / g.wb);
        if (ctas > INT_MAX) return SG_ERR_INVALID;
        if (!make_map_box(&g.tx, q.X, q.R, q.K, q.ldx, g.rows, abox) ||
            !make_map_box(&g.ty, q.dY, q.R, q.N, q.ldy, g.rows, g.wb))
            return SG_ERR_CUDA;
    }
    wgrad_kernel<<<(unsigned)ctas, kWgThreads, kWgSmem, (cudaStream_t)stream>>>(b);
    return launched();
}

int sg_mse(int32_t rows, int32_t n_out, const float* pred, int32_t ldp, const float* target, int32_t ldt,
           void* grad, int32_t ldg, float* loss, void* stream) {
    if (rows < 1 || n_out < 1 || !pred || !target || !grad || !loss || ldp < n_out || ldt < n_out || ldg < n_out)
        return SG_ERR_INVALID;
    mse_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(rows, n_out, pred, ldp, target, ldt,
                                                     reinterpret_cast<__nv_bfloat16*>(grad), ldg, loss);
    return launched();
}

int sg_pack_rows(int32_t rows, int32_t enc_dim, const void* enc, int32_t ld_enc, const int32_t* enc_row,
                 int32_t n_extra, const float* extra, int32_t ld_extra, void* x, int32_t ldx, void* stream) {
    if (rows < 1 || enc_dim < 0 || n_extra < 0 || ldx < enc_dim + n_extra || !x) return SG_ERR_INVALID;
    if ((enc_dim > 0 && (!enc || ld_enc < enc_dim)) || (n_extra > 0 && (!extra || ld_extra < n_extra)))
        return SG_ERR_INVALID;
    if (ldx % 8 == 0 && aligned16(x) && enc_dim % 8 == 0 && (enc_dim == 0 || (ld_enc % 8 == 0 && aligned16(enc)))) {
        const int tx = std::min(256, ldx / 8);
        const dim3 block(tx, std::max(1, 256 / tx));
        const int grid = (int)std::min<long long>(((long long)rows + block.y - 1) / block.y, 148 * 8);
        pack_rows8_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(
            rows, enc_dim, reinterpret_cast<const __nv_bfloat16*>(enc), ld_enc, enc_row, n_extra, extra, ld_extra,
            reinterpret_cast<__nv_bfloat16*>(x), ldx);
        return launched();
    }
    pack_rows_kernel<<<grid_for((long long)rows * ldx), 256, 0, (cudaStream_t)stream>>>(
        rows, enc_dim, reinterpret_cast<const __nv_bfloat16*>(enc), ld_enc, enc_row, n_extra, extra, ld_extra,
        reinterpret_cast<__nv_bfloat16*>(x), ldx);
    return launched();
}

int sg_unpack_grad(int32_t rows, int32_t enc_dim, const void* dx, int32_t ldx, const void* act, void* d_enc,
                   void* stream) {
    if (rows < 1 || enc_dim < 1 || !dx || !d_enc || ldx < enc_dim) return SG_ERR_INVALID;
    unpack_grad_kernel<<<grid_for((long long)rows * enc_dim), 256, 0, (cudaStream_t)stream>>>(
        rows, enc_dim, reinterpret_cast<const __nv_bfloat16*>(dx), ldx, reinterpret_cast<const __nv_bfloat16*>(act),
        reinterpret_cast<__nv_bfloat16*>(d_enc));
    return launched();
}

int sg_gather_rows(int32_t rows, int64_t row_bytes, const void* in, int64_t ld_in_bytes, const int32_t* idx,
                   void* out, int64_t ld_out_bytes, void* stream) {
    if (rows < 1 || row_bytes < 1 || !in || !idx || !out || ld_in_bytes < row_bytes || ld_out_bytes < row_bytes)
        return SG_ERR_INVALID;
    const bool v16 = (row_bytes % 16) == 0 && (ld_in_bytes % 16) == 0 && (ld_out_bytes % 16) == 0 && aligned16(in) &&
                     aligned16(out);
    const long long work = (long long)rows * (v16 ? row_bytes / 16 : row_bytes);
    gather_rows_kernel<<<grid_for(work), 256, 0, (cudaStream_t)stream>>>(
        rows, row_bytes, reinterpret_cast<const unsigned char*>(in), ld_in_bytes, idx,
        reinterpret_cast<unsigned char*>(out), ld_out_bytes, v16 ? 1 : 0);
    return launched();
}

int sg_to_bf16(int64_t n, const float* in, void* out, void* stream) {
    if (n < 0 || (n > 0 && (!in || !out))) return SG_ERR_INVALID;
    if (n == 0) return SG_OK;
    to_bf16_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(n, in, reinterpret_cast<__nv_bfloat16*>(out));
    return launched();
}

}  // extern "C"
