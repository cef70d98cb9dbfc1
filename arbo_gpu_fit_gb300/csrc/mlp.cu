// mlp.cu — the learned surrogate of the simulator: a multilayer perceptron (SiLU hidden layers)
// trained on the GPU with BF16 operands and FP32 accumulation. Every matrix product runs on the
// fifth-generation tensor cores (tcgen05.mma into tensor memory, tc.cuh); the epilogues fuse bias,
// activation, activation derivative and the transposed copies the next products need; Adam updates
// FP32 master weights and writes the BF16 copies. No reference counterpart: the reference has no
// surrogate (include/arbo.h, section "surrogate").
//
// Products, all C = A * B^T with K-major BF16 operands (row-major A [M][K], B [N][K]):
//   forward  Z_l  = H_{l-1} W_l^T          A = H_{l-1} [B][in],  B = W_l  [out][in]
//   backward dH   = dZ_l W_l               A = dZ_l    [B][out], B = W_l^T [in][out]
//   weights  dW_l = dZ_l^T H_{l-1}         A = dZ_l^T  [out][B], B = H_{l-1}^T [in][B]
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/arbo.h"
#include "launch.cuh"
#include "philox.cuh"
#include "sim_internal.h"
#include "tc.cuh"

using namespace arbo;

namespace {

typedef __nv_bfloat16 bf16;

enum Epi : int { kEpiHidden = 0, kEpiLinear = 1, kEpiBackward = 2, kEpiStore = 3, kEpiLoss = 4 };

// One product C = A B^T and its epilogue.
struct GemmArgs {
    const bf16* A;
    const bf16* B;
    uint32_t lda, ldb, M, N, K;
    int epi;
    const float* bias;   // [N]
    const float* zprev;  // [M][ldz] pre-activation whose derivative scales the product (backward)
    uint32_t ldz;
    float* outf;         // [M][ldof]
    uint32_t ldof;
    bf16* outb;          // [M][ldob]
    uint32_t ldob;
    bf16* outt;          // [N][ldot] transposed copy
    uint32_t ldot;
    const float* target;  // [M][nout] (loss)
    uint32_t nout;
    float* loss;
};

// Column sums of a matrix given by its transposed copy (bias gradients): sums[c] = sum over n rows.
struct ColumnSums {
    const bf16* t;  // [cols][ld]
    uint32_t ld, n, cols;
    float* sums;
};

// What one launch of k_gemm_tn does: one or two independent products and optional column sums.
struct GemmLaunch {
    CUtensorMap map[2][2];  // A and B of each product
    GemmArgs g[2];
    uint32_t tn[2], tiles[2];
    uint32_t stages, stage_size, acc_cols;  // operand ring; columns of one tensor-memory accumulator
    ColumnSums cs;
    uint32_t* err;  // bit 0: an mbarrier wait ran out
};

constexpr uint32_t kTileM = 128, kTileK = 64, kMaxStages = 8;
constexpr uint32_t kMinTileN = 32, kMaxTileN = 256;
constexpr uint32_t kStageBudget = 192 * 1024;  // shared memory of the operand ring
constexpr uint32_t kEpiWarps = 16;  // four per quarter of the 128 tensor-memory lanes
constexpr uint32_t kEpiPitch = 12;  // words per staged row of 8 columns
constexpr uint32_t kEpiBytes = kEpiWarps * 32 * kEpiPitch * 4;  // one staging block per epilogue warp
constexpr uint32_t kGemmThreads = 64 + kEpiWarps * 32 + 64;

// Dynamic shared memory: the ring, the epilogue's staging and 1 KB of alignment slack.
constexpr uint32_t kGemmSmemMax = kStageBudget + kEpiBytes + 1024;
static_assert(kGemmSmemMax <= 232448 - 256, "dynamic and static shared memory of one CTA");

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
    const float s = 1.0f / (1.0f + expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) |
           ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16);
}

// The epilogue's copies between a warp's block of 32 rows (one per lane) and 8 columns and row-major
// FP32 memory, through the warp's staging block, so that a warp instruction touches sixteen whole
// 32-byte sectors. `rows` is the number of live rows.
__device__ __forceinline__ void block_store_f32(float* st, const float (&v)[8], float* out, uint32_t ld, uint32_t rows,
                                                uint32_t lane)
{
#pragma unroll
    for (int k = 0; k < 2; ++k)
        *reinterpret_cast<float4*>(st + lane * kEpiPitch + 4 * k) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    __syncwarp();
    const uint32_t c = (lane & 1u) * 4;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const uint32_t r = it * 16 + (lane >> 1);
        if (r < rows)
            *reinterpret_cast<float4*>(out + (size_t)r * ld + c) = *reinterpret_cast<const float4*>(st + r * kEpiPitch + c);
    }
    __syncwarp();
}

__device__ __forceinline__ void block_fetch_f32(float4 (&f)[2], const float* in, uint32_t ld, uint32_t rows, uint32_t lane)
{
    const uint32_t c = (lane & 1u) * 4;
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const uint32_t r = it * 16 + (lane >> 1);
        f[it] = r < rows ? *reinterpret_cast<const float4*>(in + (size_t)r * ld + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

__device__ __forceinline__ void block_row_f32(const float* st, float (&v)[8], uint32_t lane)
{
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(st + lane * kEpiPitch + 4 * k);
        v[4 * k] = x.x;
        v[4 * k + 1] = x.y;
        v[4 * k + 2] = x.z;
        v[4 * k + 3] = x.w;
    }
    __syncwarp();
}

__device__ __forceinline__ void block_spread_f32(float* st, const float4 (&f)[2], float (&v)[8], uint32_t lane)
{
    const uint32_t c = (lane & 1u) * 4;
#pragma unroll
    for (int it = 0; it < 2; ++it) *reinterpret_cast<float4*>(st + (it * 16 + (lane >> 1)) * kEpiPitch + c) = f[it];
    __syncwarp();
    block_row_f32(st, v, lane);
}

// The block as BF16: row-major to `out`, transposed to `outt` (column n of the block at outt + n * ldt,
// the lane's row advancing along it). w[j] packs columns 2j and 2j+1 of the lane's row; neighbouring
// lanes swap halves so that each store of the transposed copy carries two rows of one column. Rows come
// in pairs: the products with a transposed copy have a multiple of 16 of them.
__device__ __forceinline__ void block_store_bf16(const uint32_t (&w)[4], bf16* out, uint32_t ld, bf16* outt, uint32_t ldt,
                                                 uint32_t rows, uint32_t lane)
{
    if (lane < rows) *reinterpret_cast<uint4*>(out + (size_t)lane * ld) = make_uint4(w[0], w[1], w[2], w[3]);
    const uint32_t c = lane & 1u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, w[j], 1);
        const uint32_t v = c ? __byte_perm(other, w[j], 0x7632) : __byte_perm(w[j], other, 0x5410);
        if (lane < rows) *reinterpret_cast<uint32_t*>(outt + (size_t)(2 * j + c) * ldt + lane - c) = v;
    }
}

// Column sums by the warps w, w + nw, ... of the launch, two columns at a time so that a warp keeps
// 16 loads in flight. Each column is summed by lane-strided rows, then across the lanes.
__device__ __forceinline__ void column_sums(const ColumnSums& cs, uint32_t w, uint32_t nw, uint32_t lane)
{
    for (uint32_t c = 2 * w; c < cs.cols; c += 2 * nw) {  // cols is a multiple of 16
        const bf16* t = cs.t + (size_t)c * cs.ld;
        float s[2] = {0.0f, 0.0f};
        for (uint32_t r0 = lane; r0 < cs.n; r0 += 256) {
            bf16 x[2][8];
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    x[q][k] = r0 + 32 * k < cs.n ? t[(size_t)q * cs.ld + r0 + 32 * k] : __float2bfloat16_rn(0.0f);
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int q = 0; q < 2; ++q) s[q] += __bfloat162float(x[q][k]);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
            if (lane == 0) cs.sums[c + q] = s[q];
        }
    }
}

// Tile t of a launch: which product, and where in it.
struct TileAt {
    uint32_t q, m0, n0, nt, tn, nk;
};
__device__ __forceinline__ TileAt tile_at(const GemmLaunch& p, uint32_t t)
{
    TileAt x;
    x.q = t >= p.tiles[0] ? 1u : 0u;
    const uint32_t i = x.q ? t - p.tiles[0] : t;
    const GemmArgs& g = p.g[x.q];
    const uint32_t mtiles = (g.M + kTileM - 1) / kTileM;
    x.tn = p.tn[x.q];
    x.m0 = (i % mtiles) * kTileM;
    x.n0 = (i / mtiles) * x.tn;
    x.nt = min(x.tn, g.N - x.n0);
    x.nk = (g.K + kTileK - 1) / kTileK;
    return x;
}

// Persistent, warp-specialised product: each CTA (640 threads) walks output tiles of kTileM x tn
// (tn = 32, 64, 128 or 256) in a grid-stride loop over the tiles of one or two independent products.
//   warp 0, one thread: TMA producer. Each 64-wide K chunk of A and B is one box per operand in
//     the 128-byte-swizzled K-major layout; up to eight chunks are in flight ("full" / "empty"
//     mbarriers per stage), which for the narrow tiles is the whole K of a 512-wide layer.
//   warp 1, one thread: issues the four K=16 tcgen05 products of each chunk into one of two
//     tensor-memory accumulators (tile parity), commits each chunk to the stage's "empty" barrier
//     and each finished tile to the accumulator's "full" barrier.
//   warps 2-17: epilogue. Warp w reads tensor-memory lanes 32*(w mod 4) .. +31 with tcgen05.ld, 8
//     columns at a time (four warps share a lane quarter's columns: the activation's exponential and
//     division are one long chain per output, which only other warps hide),
//     applies the fused epilogue and writes whole sectors through shared memory (block_store_*), then
//     releases the accumulator ("empty"), so the products of the next tile overlap the epilogue of
//     this one.
//   warps 18-19: the launch's column sums (bias gradients), beside the products.
// The backward pass of a layer is one launch: its weight gradient, the signal of the layer below and
// its bias gradient all read the same dZ. Launched with programmatic serialization: barriers and
// tensor memory are set up while the previous launch ends. The next launch is let in only after this
// CTA holds its tensor memory, so a later CTA can never take columns that an earlier one waits for.
// Every wait is bounded; a role that runs out records the error and stops, which bounds the waits
// of the others; tensor memory is freed at the end in every case.
//
// What bounds it: the small products of training (256 x 512 x 512) one tile's chain of load, product
// and epilogue; the large ones (4096 x 1024 x 1024) the epilogue's traffic (FP32 pre-activation, BF16
// activation and its transpose, 33.6 MB) and the operand loads from L2. With one column per store
// instruction (32 rows apart) and tiles of 128 columns the first took 41.7 us and a
// training step of the second shape 85 us a product; now 10.7 and 34 us (profiler, cold caches), and the
// fit network's training step 573 -> 245 us.
__global__ void __launch_bounds__(kGemmThreads, 1) k_gemm_tn(const __grid_constant__ GemmLaunch p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ unsigned long long full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    constexpr uint32_t aBytes = kTileM * kTileK * 2;
    const uint32_t tiles = p.tiles[0] + p.tiles[1], S = p.stages;
    if (warp == 0) tc_alloc(&tmem_slot, 2 * p.acc_cols);
    if (tid == 0) {
        for (uint32_t s = 0; s < S; ++s) {
            tc_bar_init(&full[s], 1);
            tc_bar_init(&empty[s], 1);
        }
        for (uint32_t a = 0; a < 2; ++a) {
            tc_bar_init(&acc_full[a], 1);
            tc_bar_init(&acc_empty[a], kEpiWarps);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    griddep_launch_dependents();
    griddep_wait();
    bool ok = true;
    if (warp == 0 && lane == 0) {  // producer
        uint32_t s = 0, round = 0;
        for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            const TileAt x = tile_at(p, t);
            const uint32_t bytes = aBytes + x.tn * kTileK * 2;
            for (uint32_t c = 0; c < x.nk && ok; ++c) {
                if (round > 0) ok = tc_bar_wait(&empty[s], (round - 1) & 1u);
                if (!ok) break;
                uint8_t* sa = smem + s * p.stage_size;
                tc_bar_expect_tx(&full[s], bytes);
                tc_tma_load_2d(sa, &p.map[x.q][0], (int32_t)(c * kTileK), (int32_t)x.m0, &full[s]);
                tc_tma_load_2d(sa + aBytes, &p.map[x.q][1], (int32_t)(c * kTileK), (int32_t)x.n0, &full[s]);
                if (++s == S) {
                    s = 0;
                    ++round;
                }
            }
        }
    } else if (warp == 1 && lane == 0) {  // tensor-core issuer
        uint32_t s = 0, round = 0, li = 0;
        for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++li) {
            const TileAt x = tile_at(p, t);
            const uint32_t a = li & 1u, K = p.g[x.q].K;
            if (li >= 2) ok = tc_bar_wait(&acc_empty[a], ((li >> 1) - 1) & 1u);
            if (!ok) break;
            tc_fence_after();
            const uint32_t idesc = tc_idesc_bf16(kTileM, x.nt), d = tmem + a * p.acc_cols;
            for (uint32_t c = 0; c < x.nk; ++c) {
                ok = tc_bar_wait(&full[s], round & 1u);
                if (!ok) break;
                tc_fence_after();
                const uint32_t sa = tc_smem(smem + s * p.stage_size), sb = sa + aBytes;
                const uint32_t ks = min(4u, (K - c * kTileK + 15) / 16);
                for (uint32_t kk = 0; kk < ks; ++kk)
                    tc_mma(d, tc_desc_sw128(sa + kk * 32), tc_desc_sw128(sb + kk * 32), idesc, c > 0 || kk > 0);
                tc_commit(&empty[s]);
                if (++s == S) {
                    s = 0;
                    ++round;
                }
            }
            tc_commit(&acc_full[a]);
        }
    } else if (warp >= 2 && warp < 2 + kEpiWarps) {  // epilogue
        const uint32_t quarter = warp & 3u, part = (warp - 2) >> 2;
        float* st = reinterpret_cast<float*>(smem + S * p.stage_size) + (warp - 2) * 32 * kEpiPitch;
        constexpr uint32_t kStep = 8 * (kEpiWarps / 4);  // columns between a warp's blocks
        uint32_t li = 0;
        for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++li) {
            const TileAt x = tile_at(p, t);
            const GemmArgs& g = p.g[x.q];
            const uint32_t a = li & 1u, n0 = x.n0, nt = x.nt;
            const uint32_t r0 = x.m0 + quarter * 32;
            const uint32_t rows = r0 < g.M ? min(32u, g.M - r0) : 0u;
            float4 zf[2];  // pre-activations of the next block, in flight while the current one is done
            if (g.epi == kEpiBackward && part * 8 < nt)
                block_fetch_f32(zf, g.zprev + (size_t)r0 * g.ldz + n0 + part * 8, g.ldz, rows, lane);
            float e2 = 0.0f;
            ok = __all_sync(0xffffffffu, tc_bar_wait(&acc_full[a], (li >> 1) & 1u));  // warp-uniform
            if (!ok) break;
            tc_fence_after();
            for (uint32_t c0 = part * 8; c0 < nt; c0 += kStep) {
                const uint32_t n = n0 + c0;
                float v[8], z[8];
                uint32_t w[4];
                if (g.epi == kEpiLoss) {  // targets of the block, four rows per instruction
#pragma unroll
                    for (int it = 0; it < 8; ++it) {
                        const uint32_t r = 4 * it + (lane >> 3), c = n + (lane & 7u);
                        z[it] = (r < rows && c < g.nout) ? g.target[(size_t)(r0 + r) * g.nout + c] : 0.0f;
                    }
                }
                tc_ld8(tmem + a * p.acc_cols + ((quarter * 32u) << 16) + c0, v);
                if (g.epi == kEpiHidden || g.epi == kEpiLinear || g.epi == kEpiLoss) {
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float4 b = __ldg(reinterpret_cast<const float4*>(g.bias + n) + k);
                        v[4 * k] += b.x;
                        v[4 * k + 1] += b.y;
                        v[4 * k + 2] += b.z;
                        v[4 * k + 3] += b.w;
                    }
                }
                if (g.epi == kEpiHidden) {
                    block_store_f32(st, v, g.outf + (size_t)r0 * g.ldof + n, g.ldof, rows, lane);
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[j] = pack_bf16(silu(v[2 * j]), silu(v[2 * j + 1]));
                } else if (g.epi == kEpiBackward) {
                    block_spread_f32(st, zf, z, lane);
                    if (c0 + kStep < nt)
                        block_fetch_f32(zf, g.zprev + (size_t)r0 * g.ldz + n + kStep, g.ldz, rows, lane);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        w[j] = pack_bf16(v[2 * j] * dsilu(z[2 * j]), v[2 * j + 1] * dsilu(z[2 * j + 1]));
                } else if (g.epi == kEpiLoss) {
                    // Mean squared error over the real outputs and its gradient 2 (Y - T) / (rows * nout).
                    const float cells = (float)(g.M * g.nout);
#pragma unroll
                    for (int it = 0; it < 8; ++it) st[(4 * it + (lane >> 3)) * kEpiPitch + (lane & 7u)] = z[it];
                    __syncwarp();
                    block_row_f32(st, z, lane);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float grad = 0.0f;
                        if (lane < rows && n + j < g.nout) {
                            const float e = v[j] - z[j];
                            e2 += e * e;
                            grad = 2.0f * e / cells;
                        }
                        v[j] = grad;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) w[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
                } else {
                    block_store_f32(st, v, g.outf + (size_t)r0 * g.ldof + n, g.ldof, rows, lane);
                }
                if (g.epi == kEpiHidden || g.epi == kEpiBackward || g.epi == kEpiLoss)
                    block_store_bf16(w, g.outb + (size_t)r0 * g.ldob + n, g.ldob, g.outt + (size_t)n * g.ldot + r0,
                                     g.ldot, rows, lane);
            }
            if (g.epi == kEpiLoss) {
                for (int o = 16; o > 0; o >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
                if (lane == 0 && e2 != 0.0f) atomicAdd(g.loss, e2 / (float)(g.M * g.nout));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_bar_arrive(&acc_empty[a]);
        }
    } else if (warp >= 2 + kEpiWarps && p.cs.cols) {
        column_sums(p.cs, blockIdx.x * 2 + (warp - 2 - kEpiWarps), gridDim.x * 2, lane);
    }
    if (!ok) atomicOr(p.err, 1u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(tmem, 2 * p.acc_cols);
}

// Tensor map of a row-major BF16 matrix [rows][ld] whose first `cols` columns are the operand:
// boxes of {64 columns x box_rows rows} written 128-byte swizzled, zero fill outside.
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

int tensor_map(CUtensorMap* map, const bf16* base, uint32_t rows, uint32_t cols, uint32_t ld, uint32_t box_rows)
{
    if (!g_encode) {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn)
            return set_error(ARBO_ERR_CUDA, "cuTensorMapEncodeTiled not available");
        g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    if ((reinterpret_cast<uintptr_t>(base) & 15u) || (ld * 2) % 16)
        return set_error(ARBO_ERR_INVALID, "tensor map: base and row pitch must be 16-byte aligned");
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, es,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(ARBO_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return ARBO_OK;
}

uint32_t tile_count(const GemmArgs& g, uint32_t tn)
{
    return ((g.M + kTileM - 1) / kTileM) * ((g.N + tn - 1) / tn);
}

// Model of a CTA's time on one tile (cycles): its operand loads, (128 + tn) rows of 128 bytes per K
// chunk, and its epilogue, 32 columns at a time.
uint64_t tile_cost(const GemmArgs& g, uint32_t tn)
{
    return (uint64_t)((g.K + kTileK - 1) / kTileK) * (kTileM + tn) * 2 + 500ull * (tn / 32);
}

// Columns per tile of each of the n products of a launch on num_sm SMs: the pair with the smallest
// modelled time. Narrow tiles win while wide ones leave SMs idle (a 256 x 512 layer: 32 tiles of 32
// columns instead of 8 of 128), wide ones once every SM has work (fewer operand loads per output):
// the step of a 1024-wide network at 4,096 rows took 570, 522, 496 and 450 us with forward tiles and
// backward pairs of 32, 64, 128 and 256 columns, and 480 us with the long weight-gradient tiles first.
void choose_tiles(const GemmArgs* g, uint32_t n, uint32_t num_sm, uint32_t (&tn)[2])
{
    uint64_t best = ~0ull;
    for (uint32_t a = kMinTileN; a <= kMaxTileN; a *= 2)
        for (uint32_t b = kMinTileN; b <= (n > 1 ? kMaxTileN : kMinTileN); b *= 2) {
            const uint64_t ca = tile_cost(g[0], a), cb = n > 1 ? tile_cost(g[1], b) : 0;
            const uint64_t ta = tile_count(g[0], a), tb = n > 1 ? tile_count(g[1], b) : 0;
            const uint64_t waves = (ta + tb + num_sm - 1) / num_sm;
            // One product fills whole waves; two of different cost fill the gaps of each other.
            const uint64_t cost = waves <= 1 ? std::max(ca, cb)
                                  : n == 1   ? waves * ca
                                             : (ta * ca + tb * cb) / num_sm + std::max(ca, cb) / 2;
            if (cost < best) {
                best = cost;
                tn[0] = a;
                tn[1] = b;
            }
        }
}

// Launches one or two independent products (g[i]: C = A B^T with its epilogue) and optional column
// sums on persistent CTAs, at most one per SM. Returns a cudaError_t (invalid value when a tensor map
// cannot be built; the reason is then in arbo_last_error).
int gemm_launch(const GemmArgs* g, uint32_t n, const ColumnSums& cs, uint32_t* err, cudaStream_t st, uint32_t num_sm,
                bool pdl)
{
    GemmLaunch p{};
    uint32_t nk = 0;
    choose_tiles(g, n, num_sm, p.tn);
    for (uint32_t i = 0; i < n; ++i) {
        p.g[i] = g[i];
        p.tiles[i] = tile_count(g[i], p.tn[i]);
        if (tensor_map(&p.map[i][0], g[i].A, g[i].M, g[i].K, g[i].lda, kTileM) ||
            tensor_map(&p.map[i][1], g[i].B, g[i].N, g[i].K, g[i].ldb, p.tn[i]))
            return (int)cudaErrorInvalidValue;
        p.acc_cols = std::max(p.acc_cols, p.tn[i]);
        nk = std::max(nk, (g[i].K + kTileK - 1) / kTileK);
    }
    p.stage_size = (kTileM + p.acc_cols) * kTileK * 2;
    p.stages = std::min({kStageBudget / p.stage_size, kMaxStages, nk * (p.tiles[0] + p.tiles[1] > num_sm ? 2u : 1u)});
    p.cs = cs;
    p.err = err;
    // CTAs without a tile only add column sums (four columns each pass).
    const uint32_t ctas = std::min(std::max(p.tiles[0] + p.tiles[1], (cs.cols + 3) / 4), num_sm);
    return launch_pdl(k_gemm_tn, dim3(ctas), dim3(kGemmThreads),
                      p.stages * p.stage_size + kEpiBytes + 1024, st, pdl, p);
}

// Inputs: FP32 [n][nin] -> BF16 [n][ldx] (zero padded) and transposed [ldx][ldt]; the loss is zeroed
// for the sums of the last layer's epilogue.
__global__ void k_stage_input(const float* __restrict__ x, uint32_t n, uint32_t nin, uint32_t ldx, bf16* xb, bf16* xt,
                              uint32_t ldt, float* loss)
{
    griddep_launch_dependents();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *loss = 0.0f;
    if (i >= n * ldx) return;
    const uint32_t r = i / ldx, c = i - r * ldx;
    const bf16 v = __float2bfloat16_rn(c < nin ? x[(size_t)r * nin + c] : 0.0f);
    xb[i] = v;
    xt[(size_t)c * ldt + r] = v;
}

// One parameter array of the optimiser: a layer's weights [rows][cols] with their BF16 copy and its
// transpose [cols][rows], or its bias (rows 1, no copies). `first` is its first 32 x 32 block.
struct AdamArray {
    float *w, *m, *v;
    const float* g;
    bf16 *wb, *wt;
    uint32_t rows, cols, first;
};

// Adam (Kingma & Ba 2015) on FP32 master weights, all arrays of the network in one launch: one block
// of 256 threads per 32 x 32 weights, the transposed copy written through shared memory. One launch
// per array, each thread writing its own transposed element, took 48 us of the fit network's step
// (ten launches of 3-6 us) and 70 us of a 1024-wide network's. Nothing is updated when a wait of this
// step's products ran out (*err != 0).
__global__ void __launch_bounds__(256) k_adam(const AdamArray* __restrict__ arrays, uint32_t count, float lr, float b1,
                                              float b2, float eps, float c1, float c2, const uint32_t* err)
{
    __shared__ uint16_t tile[32][33];
    uint32_t lo = 0, hi = count - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (arrays[mid].first <= blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const AdamArray a = arrays[lo];
    griddep_wait();
    if (*err) return;
    const uint32_t cb = (a.cols + 31) / 32, k = blockIdx.x - a.first;
    const uint32_t r0 = (k / cb) * 32, col = (k % cb) * 32 + (threadIdx.x & 31u);
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t rr = (threadIdx.x >> 5) + 8 * j, r = r0 + rr;
        if (r >= a.rows || col >= a.cols) continue;
        const size_t i = (size_t)r * a.cols + col;
        const float gi = a.g[i];
        const float mi = b1 * a.m[i] + (1.0f - b1) * gi;
        const float vi = b2 * a.v[i] + (1.0f - b2) * gi * gi;
        a.m[i] = mi;
        a.v[i] = vi;
        const float wi = a.w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        a.w[i] = wi;
        if (a.wb) {
            const bf16 b = __float2bfloat16_rn(wi);
            a.wb[i] = b;
            tile[rr][threadIdx.x & 31u] = __bfloat16_as_ushort(b);
        }
    }
    if (!a.wb) return;
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t cc = (threadIdx.x >> 5) + 8 * j, c = (k % cb) * 32 + cc, r = r0 + (threadIdx.x & 31u);
        if (c < a.cols && r < a.rows)
            a.wt[(size_t)c * a.rows + r] = __ushort_as_bfloat16(tile[threadIdx.x & 31u][cc]);
    }
}

__global__ void k_cast_weights(const float* __restrict__ w, uint32_t rows, uint32_t cols, bf16* wb, bf16* wt)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * cols) return;
    const uint32_t r = i / cols, c = i - r * cols;
    const bf16 b = __float2bfloat16_rn(w[i]);
    wb[i] = b;
    wt[(size_t)c * rows + r] = b;
}

int ufail(int code, const std::string& msg) { return set_error(code, msg); }

#define UCUDA(expr)                                                                                     \
    do {                                                                                                \
        cudaError_t e_ = (expr);                                                                        \
        if (e_ != cudaSuccess) return ufail(ARBO_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

uint32_t up16(uint32_t x) { return (x + 15u) & ~15u; }

}  // namespace

struct arbo_mlp {
    int device = 0;
    uint32_t L = 0;                    // linear layers
    std::vector<uint32_t> dim;         // padded widths, dim[0] = input, dim[L] = output
    uint32_t nin = 0, nout = 0, maxb = 0;
    std::vector<float*> w, b, mw, vw, mb, vb, dw, db;
    std::vector<bf16*> wb, wt;
    bf16 *x = nullptr, *xt = nullptr;
    std::vector<float*> z;             // pre-activations of hidden layers [maxb][dim]
    std::vector<bf16*> h, ht;          // activations of hidden layers
    float* y = nullptr;                // outputs [maxb][dim[L]]
    bf16 *d0 = nullptr, *d0t = nullptr, *d1 = nullptr, *d1t = nullptr;  // ping-pong dZ and transposes
    float *xin = nullptr, *tin = nullptr, *loss = nullptr;
    uint32_t* err = nullptr;
    uint32_t steps = 0;
    uint32_t num_sm = 152;
    AdamArray* adam = nullptr;         // device table of the optimiser's arrays
    uint32_t adam_arrays = 0, adam_blocks = 0;
    // What the host reads back every call: loss and error word, device (adjacent) and pinned.
    uint32_t* back = nullptr;
    cudaEvent_t done = nullptr;
    // Captured kernel sequences of the row counts in use. A row count is launched directly the first
    // time and captured the second, so that one call on a new network pays for no capture.
    struct Captured {
        uint32_t rows = 0;
        bool train = false;
        uint64_t used = 0;
        cudaGraphExec_t exec = nullptr;
    };
    Captured graphs[8];
    uint64_t calls = 0;
    cudaStream_t cap = nullptr;
    std::vector<void*> allocs;
};

namespace {

// train: the last layer's epilogue goes straight to the loss and its gradient (no outputs kept).
int mlp_forward(arbo_mlp* n, uint32_t rows, bool train, cudaStream_t st)
{
    const uint32_t ld = n->maxb, L = n->L;
    k_stage_input<<<(rows * n->dim[0] + 255) / 256, 256, 0, st>>>(n->xin, rows, n->nin, n->dim[0], n->x, n->xt, ld, n->loss);
    int e = (int)cudaGetLastError();
    for (uint32_t l = 0; l < L && !e; ++l) {
        const uint32_t in = n->dim[l], out = n->dim[l + 1];
        GemmArgs g{};
        g.A = l == 0 ? n->x : n->h[l - 1];
        g.B = n->wb[l];
        g.lda = g.ldb = in;
        g.M = rows;
        g.N = out;
        g.K = in;
        g.bias = n->b[l];
        g.ldof = g.ldob = out;
        g.ldot = ld;
        if (l + 1 < L) {
            g.epi = kEpiHidden;
            g.outf = n->z[l];
            g.outb = n->h[l];
            g.outt = n->ht[l];
        } else if (train) {
            g.epi = kEpiLoss;
            g.outb = n->d0;
            g.outt = n->d0t;
            g.target = n->tin;
            g.nout = n->nout;
            g.loss = n->loss;
        } else {
            g.epi = kEpiLinear;
            g.outf = n->y;
        }
        e = gemm_launch(&g, 1, ColumnSums{}, n->err, st, n->num_sm, true);
    }
    return e;
}

// One launch per layer: dZ_{l-1} = (dZ_l W_l) * silu'(Z_{l-1}) (M = rows, N = in, K = out), dW_l =
// dZ_l^T H_{l-1} (M = out, N = in, K = rows) and db_l = column sums of dZ_l.
int mlp_backward(arbo_mlp* n, uint32_t rows, cudaStream_t st)
{
    const uint32_t ld = n->maxb, L = n->L;
    bf16 *dz = n->d0, *dzt = n->d0t, *nd = n->d1, *ndt = n->d1t;
    int e = 0;
    for (uint32_t l = L; l-- > 0 && !e;) {
        const uint32_t in = n->dim[l], out = n->dim[l + 1];
        GemmArgs g[2] = {};
        GemmArgs& w = g[l > 0 ? 1 : 0];
        w.A = dzt;
        w.B = l == 0 ? n->xt : n->ht[l - 1];
        w.lda = w.ldb = ld;
        w.M = out;
        w.N = in;
        w.K = rows;
        w.epi = kEpiStore;
        w.outf = n->dw[l];
        w.ldof = in;
        if (l > 0) {
            g[0].A = dz;
            g[0].B = n->wt[l];
            g[0].lda = g[0].ldb = out;
            g[0].M = rows;
            g[0].N = in;
            g[0].K = out;
            g[0].epi = kEpiBackward;
            g[0].zprev = n->z[l - 1];
            g[0].ldz = g[0].ldob = in;
            g[0].outb = nd;
            g[0].outt = ndt;
            g[0].ldot = ld;
        }
        e = gemm_launch(g, l > 0 ? 2 : 1, ColumnSums{dzt, ld, rows, out, n->db[l]}, n->err, st, n->num_sm, true);
        std::swap(dz, nd);
        std::swap(dzt, ndt);
    }
    return e;
}

int mlp_upload(arbo_mlp* n, const float* x, const float* t, uint32_t rows, cudaStream_t st)
{
    if (rows == 0 || rows > n->maxb || rows % 16) return ufail(ARBO_ERR_INVALID, "batch rows must be a multiple of 16 in [16, max_batch]");
    UCUDA(cudaMemcpyAsync(n->xin, x, (size_t)rows * n->nin * 4, cudaMemcpyHostToDevice, st));
    if (t) UCUDA(cudaMemcpyAsync(n->tin, t, (size_t)rows * n->nout * 4, cudaMemcpyHostToDevice, st));
    return ARBO_OK;
}

int mlp_kernels(arbo_mlp* n, uint32_t rows, bool train, cudaStream_t st)
{
    int e = mlp_forward(n, rows, train, st);
    if (!e && train) e = mlp_backward(n, rows, st);
    return e;
}

// The forward pass, or the forward and backward pass, of `rows` rows already in xin (and tin). From
// the second call of a row count on it is one graph launch instead of 6 or 11 kernel launches (each
// with its tensor maps to encode): training step of the fit network 132 -> 109 us, prediction at 64
// rows 84 -> 79 us.
int mlp_enqueue(arbo_mlp* n, uint32_t rows, bool train, cudaStream_t st)
{
    n->calls += 1;
    arbo_mlp::Captured* slot = nullptr;
    for (auto& g : n->graphs)
        if (g.rows == rows && g.train == train) slot = &g;
    if (!slot) {
        slot = &n->graphs[0];
        for (auto& g : n->graphs)
            if (g.used < slot->used) slot = &g;
        // An evicted graph may still run on another stream.
        if (slot->exec && (cudaDeviceSynchronize() != cudaSuccess || cudaGraphExecDestroy(slot->exec) != cudaSuccess))
            return (int)cudaErrorUnknown;
        *slot = {rows, train, n->calls, nullptr};
        return mlp_kernels(n, rows, train, st);
    }
    slot->used = n->calls;
    if (!slot->exec) {
        cudaGraph_t g = nullptr;
        cudaError_t e = n->cap ? cudaSuccess : cudaStreamCreateWithFlags(&n->cap, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaStreamBeginCapture(n->cap, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return (int)e;
        const int k = mlp_kernels(n, rows, train, n->cap);
        e = cudaStreamEndCapture(n->cap, &g);
        if (!k && e == cudaSuccess) e = cudaGraphInstantiate(&slot->exec, g, 0);
        if (g) cudaGraphDestroy(g);
        if (k || e != cudaSuccess) return k ? k : (int)e;
    }
    return (int)cudaGraphLaunch(slot->exec, st);
}

// Waits for what was enqueued before (and for the copy of loss and error word, which it enqueues).
int mlp_read_back(arbo_mlp* n, cudaStream_t st)
{
    UCUDA(cudaMemcpyAsync(n->back, n->loss, 8, cudaMemcpyDeviceToHost, st));
    UCUDA(cudaEventRecord(n->done, st));
    return ARBO_OK;
}

int mlp_check_err(arbo_mlp* n)
{
    UCUDA(cudaEventSynchronize(n->done));
    const uint32_t e = n->back[1];
    if (e) return ufail(ARBO_ERR_CUDA, "tensor-core product: an mbarrier wait ran out (error word " + std::to_string(e) + ")");
    return ARBO_OK;
}

// Upload, forward and backward pass and the copy of the loss, all enqueued on st.
int mlp_gradients(arbo_mlp* n, const float* x, const float* t, uint32_t rows, cudaStream_t st)
{
    int e = mlp_upload(n, x, t, rows, st);
    if (e) return e;
    if ((e = mlp_enqueue(n, rows, true, st)))
        return ufail(ARBO_ERR_CUDA, std::string("forward/backward: ") + cudaGetErrorString((cudaError_t)e));
    return mlp_read_back(n, st);
}

}  // namespace

extern "C" {

int arbo_mlp_create(uint32_t n_in, uint32_t hidden, uint32_t hidden_layers, uint32_t n_out, uint32_t max_batch,
                    uint64_t seed, arbo_mlp** out)
{
    if (!out || n_in == 0 || n_in > 4096 || hidden == 0 || hidden % 16 || hidden > 8192 || hidden_layers == 0 ||
        n_out == 0 || n_out > 8192 || max_batch == 0 || max_batch % 16 || max_batch > (1u << 16))
        return ufail(ARBO_ERR_INVALID, "arbo_mlp_create: hidden and max_batch multiples of 16; sizes within limits");
    *out = nullptr;
    arbo_mlp* n = new arbo_mlp();
    UCUDA(cudaGetDevice(&n->device));
    UCUDA(cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmemMax));
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, n->device) == cudaSuccess && sms > 0)
        n->num_sm = (uint32_t)sms;
    n->L = hidden_layers + 1;
    n->nin = n_in;
    n->nout = n_out;
    n->maxb = max_batch;
    n->dim.push_back(up16(n_in));
    for (uint32_t l = 0; l < hidden_layers; ++l) n->dim.push_back(hidden);
    n->dim.push_back(up16(n_out));
    auto alloc = [&](size_t bytes) -> void* {
        void* p = nullptr;
        if (cudaMalloc(&p, bytes ? bytes : 16) != cudaSuccess) return nullptr;
        cudaMemset(p, 0, bytes ? bytes : 16);
        n->allocs.push_back(p);
        return p;
    };
    bool okm = true;
    auto F = [&](size_t cnt) {
        float* p = (float*)alloc(cnt * 4);
        okm = okm && p;
        return p;
    };
    auto H = [&](size_t cnt) {
        bf16* p = (bf16*)alloc(cnt * 2);
        okm = okm && p;
        return p;
    };
    std::vector<float> hw;
    for (uint32_t l = 0; l < n->L; ++l) {
        const uint32_t in = n->dim[l], o = n->dim[l + 1];
        const size_t cnt = (size_t)in * o;
        n->w.push_back(F(cnt));
        n->mw.push_back(F(cnt));
        n->vw.push_back(F(cnt));
        n->dw.push_back(F(cnt));
        n->b.push_back(F(o));
        n->mb.push_back(F(o));
        n->vb.push_back(F(o));
        n->db.push_back(F(o));
        n->wb.push_back(H(cnt));
        n->wt.push_back(H(cnt));
        if (!okm) break;
        // Uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) from the keyed stream; padded inputs and outputs
        // have zero weights.
        const uint32_t fan = l == 0 ? n_in : n->dim[l];
        const float bound = 1.0f / std::sqrt((float)fan);
        const uint32_t ro = (l + 1 == n->L) ? n_out : o, ri = l == 0 ? n_in : in;
        hw.assign(cnt, 0.0f);
        const Key key{(uint32_t)seed, (uint32_t)(seed >> 32), 0};
        for (uint32_t r = 0; r < ro; ++r)
            for (uint32_t c = 0; c < ri; c += 4) {
                const U4 u = draw4(key, 0x3Fu, l, r, c);
                for (uint32_t q = 0; q < 4 && c + q < ri; ++q) hw[(size_t)r * in + c + q] = (2.0f * u01(u.v[q]) - 1.0f) * bound;
            }
        UCUDA(cudaMemcpy(n->w[l], hw.data(), cnt * 4, cudaMemcpyHostToDevice));
        k_cast_weights<<<(uint32_t)((cnt + 255) / 256), 256>>>(n->w[l], o, in, n->wb[l], n->wt[l]);
    }
    const uint32_t B = max_batch;
    n->x = H((size_t)B * n->dim[0]);
    n->xt = H((size_t)B * n->dim[0]);
    uint32_t widest = 0;
    for (uint32_t d : n->dim) widest = std::max(widest, d);
    for (uint32_t l = 0; l + 1 < n->L; ++l) {
        n->z.push_back(F((size_t)B * n->dim[l + 1]));
        n->h.push_back(H((size_t)B * n->dim[l + 1]));
        n->ht.push_back(H((size_t)B * n->dim[l + 1]));
    }
    n->y = F((size_t)B * n->dim[n->L]);
    n->d0 = H((size_t)B * widest);
    n->d0t = H((size_t)B * widest);
    n->d1 = H((size_t)B * widest);
    n->d1t = H((size_t)B * widest);
    n->xin = F((size_t)B * n_in);
    n->tin = F((size_t)B * n_out);
    n->loss = F(2);  // and the error word beside it
    n->err = (uint32_t*)n->loss + 1;
    if (!okm || cudaMallocHost(&n->back, 8) != cudaSuccess ||
        cudaEventCreateWithFlags(&n->done, cudaEventDisableTiming) != cudaSuccess) {
        arbo_mlp_destroy(n);
        return ufail(ARBO_ERR_ALLOC, "arbo_mlp_create: device allocation failed");
    }
    std::vector<AdamArray> arrays;
    for (uint32_t l = 0; l < n->L; ++l) {
        const uint32_t in = n->dim[l], o = n->dim[l + 1];
        arrays.push_back({n->w[l], n->mw[l], n->vw[l], n->dw[l], n->wb[l], n->wt[l], o, in, n->adam_blocks});
        n->adam_blocks += ((o + 31) / 32) * ((in + 31) / 32);
        arrays.push_back({n->b[l], n->mb[l], n->vb[l], n->db[l], nullptr, nullptr, 1, o, n->adam_blocks});
        n->adam_blocks += (o + 31) / 32;
    }
    n->adam_arrays = (uint32_t)arrays.size();
    n->adam = (AdamArray*)alloc(arrays.size() * sizeof(AdamArray));
    if (!n->adam) {
        arbo_mlp_destroy(n);
        return ufail(ARBO_ERR_ALLOC, "arbo_mlp_create: device allocation failed");
    }
    UCUDA(cudaMemcpy(n->adam, arrays.data(), arrays.size() * sizeof(AdamArray), cudaMemcpyHostToDevice));
    UCUDA(cudaDeviceSynchronize());
    *out = n;
    return ARBO_OK;
}

int arbo_mlp_destroy(arbo_mlp* n)
{
    if (!n) return ARBO_OK;
    cudaSetDevice(n->device);
    for (auto& g : n->graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    if (n->cap) cudaStreamDestroy(n->cap);
    if (n->done) cudaEventDestroy(n->done);
    if (n->back) cudaFreeHost(n->back);
    for (void* p : n->allocs) cudaFree(p);
    delete n;
    return ARBO_OK;
}

int arbo_mlp_dims(const arbo_mlp* n, uint32_t* layers, uint32_t* dims)
{
    if (!n) return ufail(ARBO_ERR_INVALID, "null network");
    if (layers) *layers = n->L;
    if (dims)
        for (uint32_t l = 0; l <= n->L; ++l) dims[l] = n->dim[l];
    return ARBO_OK;
}

int arbo_mlp_forward(arbo_mlp* n, const float* x, uint32_t rows, float* y, void* stream)
{
    if (!n || !x || !y) return ufail(ARBO_ERR_INVALID, "null argument");
    UCUDA(cudaSetDevice(n->device));
    cudaStream_t st = (cudaStream_t)stream;
    int e = mlp_upload(n, x, nullptr, rows, st);
    if (e) return e;
    if ((e = mlp_enqueue(n, rows, false, st))) return ufail(ARBO_ERR_CUDA, std::string("forward: ") + cudaGetErrorString((cudaError_t)e));
    const uint32_t w = n->dim[n->L];
    if (w == n->nout) {
        UCUDA(cudaMemcpyAsync(y, n->y, (size_t)rows * w * 4, cudaMemcpyDeviceToHost, st));
    } else {
        UCUDA(cudaMemcpy2DAsync(y, n->nout * 4, n->y, w * 4, n->nout * 4, rows, cudaMemcpyDeviceToHost, st));
    }
    if ((e = mlp_read_back(n, st))) return e;
    return mlp_check_err(n);
}

int arbo_mlp_gradients(arbo_mlp* n, const float* x, const float* t, uint32_t rows, float* loss, void* stream)
{
    if (!n || !x || !t) return ufail(ARBO_ERR_INVALID, "null argument");
    UCUDA(cudaSetDevice(n->device));
    int e = mlp_gradients(n, x, t, rows, (cudaStream_t)stream);
    if (!e) e = mlp_check_err(n);
    if (!e && loss) std::memcpy(loss, &n->back[0], 4);
    return e;
}

// The optimiser's launch follows the gradients without a wait in between (it does nothing when their
// products failed); the call returns with the loss while it runs.
int arbo_mlp_train_step(arbo_mlp* n, const float* x, const float* t, uint32_t rows, float lr, float* loss, void* stream)
{
    if (!n || !x || !t) return ufail(ARBO_ERR_INVALID, "null argument");
    UCUDA(cudaSetDevice(n->device));
    cudaStream_t st = (cudaStream_t)stream;
    int e = mlp_gradients(n, x, t, rows, st);
    if (e) return e;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f, step = (float)(n->steps + 1);
    const float c1 = 1.0f - std::pow(b1, step), c2 = 1.0f - std::pow(b2, step);
    k_adam<<<n->adam_blocks, 256, 0, st>>>(n->adam, n->adam_arrays, lr, b1, b2, eps, c1, c2, n->err);
    UCUDA(cudaGetLastError());
    if ((e = mlp_check_err(n))) return e;
    n->steps += 1;
    if (loss) std::memcpy(loss, &n->back[0], 4);
    return ARBO_OK;
}

int arbo_mlp_get_layer(const arbo_mlp* n, uint32_t layer, float* w, float* b, float* dw, float* db)
{
    if (!n || layer >= n->L) return ufail(ARBO_ERR_INVALID, "bad layer");
    UCUDA(cudaSetDevice(n->device));
    UCUDA(cudaDeviceSynchronize());
    const size_t cnt = (size_t)n->dim[layer] * n->dim[layer + 1], o = n->dim[layer + 1];
    if (w) UCUDA(cudaMemcpy(w, n->w[layer], cnt * 4, cudaMemcpyDeviceToHost));
    if (b) UCUDA(cudaMemcpy(b, n->b[layer], o * 4, cudaMemcpyDeviceToHost));
    if (dw) UCUDA(cudaMemcpy(dw, n->dw[layer], cnt * 4, cudaMemcpyDeviceToHost));
    if (db) UCUDA(cudaMemcpy(db, n->db[layer], o * 4, cudaMemcpyDeviceToHost));
    return ARBO_OK;
}

int arbo_mlp_set_layer(arbo_mlp* n, uint32_t layer, const float* w, const float* b)
{
    if (!n || layer >= n->L) return ufail(ARBO_ERR_INVALID, "bad layer");
    UCUDA(cudaSetDevice(n->device));
    const uint32_t in = n->dim[layer], o = n->dim[layer + 1];
    const size_t cnt = (size_t)in * o;
    if (w) {
        UCUDA(cudaMemcpy(n->w[layer], w, cnt * 4, cudaMemcpyHostToDevice));
        k_cast_weights<<<(uint32_t)((cnt + 255) / 256), 256>>>(n->w[layer], o, in, n->wb[layer], n->wt[layer]);
        UCUDA(cudaGetLastError());
    }
    if (b) UCUDA(cudaMemcpy(n->b[layer], b, o * 4, cudaMemcpyHostToDevice));
    UCUDA(cudaDeviceSynchronize());
    return ARBO_OK;
}

// One tensor-core product C = A B^T of BF16 inputs given as FP32 (rounded to BF16 here), FP32
// result: exposes the GEMM kernel alone for checks and timing. A [M][K], B [N][K], C [M][N].
int arbo_tc_gemm(const float* a, const float* b, uint32_t M, uint32_t N, uint32_t K, float* c, uint32_t reps,
                 float* ms)
{
    if (!a || !b || !c || M == 0 || N == 0 || K == 0 || N % 16 || K % 16)
        return ufail(ARBO_ERR_INVALID, "arbo_tc_gemm: N and K multiples of 16");
    UCUDA(cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmemMax));
    std::vector<bf16> ha((size_t)M * K), hb((size_t)N * K);
    for (size_t i = 0; i < ha.size(); ++i) ha[i] = __float2bfloat16_rn(a[i]);
    for (size_t i = 0; i < hb.size(); ++i) hb[i] = __float2bfloat16_rn(b[i]);
    bf16 *da = nullptr, *db = nullptr;
    float* dc = nullptr;
    uint32_t* derr = nullptr;
    auto cleanup = [&]() {
        cudaFree(da);
        cudaFree(db);
        cudaFree(dc);
        cudaFree(derr);
    };
    if (cudaMalloc(&da, ha.size() * 2) || cudaMalloc(&db, hb.size() * 2) || cudaMalloc(&dc, (size_t)M * N * 4) ||
        cudaMalloc(&derr, 4)) {
        cleanup();
        return ufail(ARBO_ERR_ALLOC, "arbo_tc_gemm: allocation");
    }
    cudaMemcpy(da, ha.data(), ha.size() * 2, cudaMemcpyHostToDevice);
    cudaMemcpy(db, hb.data(), hb.size() * 2, cudaMemcpyHostToDevice);
    cudaMemset(derr, 0, 4);
    GemmArgs g{};
    g.A = da;
    g.B = db;
    g.lda = g.ldb = K;
    g.M = M;
    g.N = g.ldof = N;
    g.K = K;
    g.epi = kEpiStore;
    g.outf = dc;
    int sms = 152, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto product = [&]() { return gemm_launch(&g, 1, ColumnSums{}, derr, nullptr, (uint32_t)sms, false); };
    int le = product();
    const std::string map_err = le ? std::string(arbo_last_error()) : std::string();
    cudaEventRecord(e0);
    for (uint32_t r = 0; r < reps && !le; ++r) le = product();
    cudaEventRecord(e1);
    cudaError_t ce = cudaEventSynchronize(e1);
    float t = 0;
    cudaEventElapsedTime(&t, e0, e1);
    if (ms) *ms = reps ? t / reps : 0.0f;
    uint32_t herr = 0;
    if (ce == cudaSuccess) ce = cudaMemcpy(c, dc, (size_t)M * N * 4, cudaMemcpyDeviceToHost);
    if (ce == cudaSuccess) ce = cudaMemcpy(&herr, derr, 4, cudaMemcpyDeviceToHost);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cleanup();
    if (le) return ufail(ARBO_ERR_CUDA, "arbo_tc_gemm: launch failed: " + map_err + " " + cudaGetErrorString((cudaError_t)le));
    if (ce != cudaSuccess) return ufail(ARBO_ERR_CUDA, std::string("arbo_tc_gemm: ") + cudaGetErrorString(ce));
    if (herr) return ufail(ARBO_ERR_CUDA, "arbo_tc_gemm: an mbarrier wait ran out");
    return ARBO_OK;
}

}  // extern "C"
