// mlp.cu — the learned surrogate of the simulator: a multilayer perceptron (SiLU hidden layers)
// trained on the GPU with BF16 operands and FP32 accumulation. Every matrix product runs on the
// fifth-generation tensor cores (tcgen05.mma into tensor memory, tc.cuh); the epilogues fuse bias,
// activation, activation derivative and the transposed copies the next products need; Adam updates
// FP32 master weights and writes the BF16 copies. No reference counterpart: the reference has no
// surrogate (include/arbo.h, section "surrogate").
//
// Products, all C = A * B^T with K-major BF16 operands (row-major A [M][K], B [N][K]), C written
// transposed (row-major [N][M]):
//   forward  Z_l^T  = W_l H_{l-1}^T        A = W_l   [out][in],      B = H_{l-1} [rows][in]
//   backward dH^T   = W_l^T dZ_l^T         A = W_l^T [in][out],      B = dZ_l    [rows][out]
//   weights  dW_l^T = H_{l-1}^T dZ_l       A = H_{l-1}^T [in][rows], B = dZ_l^T  [out][rows]
// A is at least two launches old in each, which lets the kernel fetch it before the launch that it
// depends on has ended (k_gemm_tn).
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

// One product C = A B^T, M a multiple of 16, and its epilogue, which writes C transposed. A, bias, zprev and
// target were written before the launch that precedes this one began (they are read before it has ended).
struct GemmArgs {
    const bf16* A;
    const bf16* B;
    uint32_t lda, ldb, M, N, K;
    int epi;
    const float* bias;   // [M]
    const float* zprev;  // [N][ldz] pre-activation whose derivative scales the product (backward)
    uint32_t ldz;
    float* outf;         // [N][ldof]
    uint32_t ldof;
    bf16* outb;          // [N][ldob]; with it N is a multiple of 16
    uint32_t ldob;
    bf16* outt;          // [M][ldot] copy of outb the other way round
    uint32_t ldot;
    const float* target;  // [N][nout] (loss)
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
    // Operand ring: stages of `group` K chunks; columns of one tensor-memory accumulator.
    uint32_t stages, group, stage_size, acc_cols;
    ColumnSums cs;
    uint32_t* err;       // bit 0: an mbarrier wait ran out
    uint32_t* host_err;  // the same in host memory, or null
    const float* loss;   // if not null, a finished loss and where in host memory it goes
    float* host_loss;
    uint32_t polls;      // bound of the roles' waits (kTcMaxPolls; 0 in the self-test: every wait runs out)
};

constexpr uint32_t kTileM = 128, kTileK = 64, kMaxStages = 8;
constexpr uint32_t kMinTileN = 16, kMaxTileN = 256;
constexpr uint32_t kStageBudget = 192 * 1024;  // shared memory of the operand ring
constexpr uint32_t kEpiWarps = 16;  // four per quarter of the 128 tensor-memory lanes
constexpr uint32_t kGemmThreads = 64 + kEpiWarps * 32 + 64;

// Dynamic shared memory: the ring and 1 KB of alignment slack.
constexpr uint32_t kGemmSmemMax = kStageBudget + 1024;
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

// The epilogue's copies between a warp's block of the accumulator, 32 lanes (rows of C) by C columns, and
// row-major FP32 memory that holds the matrix transposed: an instruction touches 128 consecutive bytes. Lanes
// from M on and columns from N on are left out.
template <int C>
__device__ __forceinline__ void block_store_f32(const float (&v)[C], float* out, uint32_t ld, bool live, uint32_t cols)
{
#pragma unroll
    for (uint32_t k = 0; k < C; ++k)
        if (live && k < cols) out[(size_t)k * ld] = v[k];
}

template <int C>
__device__ __forceinline__ void block_fetch_f32(float (&v)[C], const float* in, uint32_t ld, bool live)
{
#pragma unroll
    for (uint32_t k = 0; k < C; ++k) v[k] = live ? __ldcg(in + (size_t)k * ld) : 0.0f;
}

// The block as BF16, w[j] packing columns 2j and 2j+1 of the lane's row: the lane's columns in one store to
// `outt`, and transposed to `out` (row k of it is column k), where neighbouring lanes swap halves so that a
// store carries two lanes of one column.
template <int C>
__device__ __forceinline__ void block_store_bf16(const uint32_t (&w)[C / 2], bf16* out, uint32_t ld, bf16* outt, bool live,
                                                 uint32_t lane)
{
    if (live) {
        if constexpr (C == 8) *reinterpret_cast<uint4*>(outt) = make_uint4(w[0], w[1], w[2], w[3]);
        else *reinterpret_cast<uint2*>(outt) = make_uint2(w[0], w[1]);
    }
    const uint32_t c = lane & 1u;
#pragma unroll
    for (int j = 0; j < C / 2; ++j) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, w[j], 1);
        const uint32_t v = c ? __byte_perm(other, w[j], 0x7632) : __byte_perm(w[j], other, 0x5410);
        if (live) *reinterpret_cast<uint32_t*>(out + (size_t)(2 * j + c) * ld - c) = v;
    }
}

// Epilogue of one tile by one of the warps of a quarter of its rows (lane: row m): blocks of C columns, block
// `part` and every (kEpiWarps / 4)-th after it. `ready` waits for the accumulator (tensor-memory address d) and
// returns false when the wait ran out; what else the first block needs is fetched before it. Returns the
// lane's sum of squared errors (loss).
template <int C, typename Ready>
__device__ __forceinline__ float tile_epilogue(const GemmArgs& g, uint32_t m, uint32_t n0, uint32_t nt, uint32_t part,
                                               uint32_t d, uint32_t lane, Ready ready)
{
    constexpr uint32_t kStep = C * (kEpiWarps / 4);
    const bool live = m < g.M;
    float z[C] = {};
    const float* zin = g.epi == kEpiBackward ? g.zprev : g.target;
    const uint32_t ldz = g.epi == kEpiBackward ? g.ldz : g.nout;
    const bool zlive = g.epi == kEpiBackward ? live : g.epi == kEpiLoss && m < g.nout;
    if (part * C < nt) block_fetch_f32(z, zin + (size_t)(n0 + part * C) * ldz + m, ldz, zlive);
    const float bias = live && g.bias ? __ldcg(g.bias + m) : 0.0f;
    float e2 = 0.0f;
    if (!ready()) return 0.0f;
    for (uint32_t c0 = part * C; c0 < nt; c0 += kStep) {
        const uint32_t n = n0 + c0;
        float v[C];
        uint32_t w[C / 2];
        tc_ld(d + c0, v);
        if (g.epi != kEpiBackward && g.epi != kEpiStore) {
#pragma unroll
            for (int k = 0; k < C; ++k) v[k] += bias;
        }
        if (g.epi == kEpiHidden) {
            block_store_f32(v, g.outf + (size_t)n * g.ldof + m, g.ldof, live, C);
#pragma unroll
            for (int j = 0; j < C / 2; ++j) w[j] = pack_bf16(silu(v[2 * j]), silu(v[2 * j + 1]));
        } else if (g.epi == kEpiBackward) {
#pragma unroll
            for (int j = 0; j < C / 2; ++j)
                w[j] = pack_bf16(v[2 * j] * dsilu(z[2 * j]), v[2 * j + 1] * dsilu(z[2 * j + 1]));
        } else if (g.epi == kEpiLoss) {
            // Mean squared error over the real outputs and its gradient 2 (Y - T) / (rows * nout).
            const float cells = (float)(g.N * g.nout);
#pragma unroll
            for (int j = 0; j < C; ++j) {
                float grad = 0.0f;
                if (m < g.nout) {
                    const float e = v[j] - z[j];
                    e2 += e * e;
                    grad = 2.0f * e / cells;
                }
                v[j] = grad;
            }
#pragma unroll
            for (int j = 0; j < C / 2; ++j) w[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
        } else {
            block_store_f32(v, g.outf + (size_t)n * g.ldof + m, g.ldof, live, n < g.N ? g.N - n : 0u);
        }
        if (g.epi == kEpiHidden || g.epi == kEpiBackward || g.epi == kEpiLoss) {
            if (c0 + kStep < nt) block_fetch_f32(z, zin + (size_t)(n + kStep) * ldz + m, ldz, zlive);
            block_store_bf16<C>(w, g.outb + (size_t)n * g.ldob + m, g.ldob, g.outt + (size_t)m * g.ldot + n, live, lane);
        }
    }
    return e2;
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
    x.nt = min(x.tn, (g.N - x.n0 + 15u) & ~15u);
    x.nk = (g.K + kTileK - 1) / kTileK;
    return x;
}

// Persistent, warp-specialised product: each CTA (640 threads) walks output tiles of kTileM x tn
// (tn = 16, 32, 64, 128 or 256) in a grid-stride loop over the tiles of one or two independent products.
//   warp 0: TMA producer. Each 64-wide K chunk of A and B is one box per operand in the
//     128-byte-swizzled K-major layout. A stage of the operand ring ("full" / "empty" mbarriers) holds
//     one to four chunks: a wait on an mbarrier costs some 180 cycles even when its phase is over, more
//     than the products of a narrow chunk (4 x 20 cycles).
//   warp 1: issues the four K=16 tcgen05 products of each chunk into one of two tensor-memory
//     accumulators (tile parity), commits each stage that is filled again to its "empty" barrier
//     and each finished tile to the accumulator's "full" barrier. The whole warp runs the loop and an
//     elected lane issues: from a branch on the lane, an issue took some 100 cycles.
//   warps 2-17: epilogue (tile_epilogue). Warp w reads tensor-memory lanes 32*(w mod 4) .. +31 with
//     tcgen05.ld, 8 columns at a time, or 4 of a tile of 16 (four warps share a lane quarter's columns: the
//     activation's exponential and division are one long chain per output, which only other warps hide),
//     applies the fused epilogue, writes, and releases the accumulator ("empty"), so the products of the
//     next tile overlap the epilogue of this one. A's rows are the lanes, so the row-major outputs are
//     written 128 bytes an instruction straight from registers.
//   warps 18-19: the launch's column sums (bias gradients), beside the products.
// The backward pass of a layer is one launch: its weight gradient, the signal of the layer below and
// its bias gradient all read the same dZ.
// Launched with programmatic serialization: barriers and tensor memory are set up and A, the larger operand
// of a narrow tile, and the epilogue's first inputs are fetched while the previous launch runs. That is sound
// because a launch lets the next one in only after its own wait: when a CTA starts, every launch but the
// previous one has ended, and A, bias, zprev and target are older than that (GemmArgs). What the passes of
// the same step wrote among them (activations and pre-activations, read by the backward launches) is in L2 by
// then, and the early reads are TMA copies and ld.cg, which go to L2 and not through L1. By then the CTA also
// holds its tensor memory, so a later CTA can never take columns that an earlier one waits for.
// Every wait is bounded; a role that runs out records the error and stops, which bounds the waits
// of the others. The CTA then waits, bounded again, for its copies and products in flight, which write its
// shared and tensor memory; tensor memory is freed at the end in every case.
//
// What bounds it: the small products of training (256 x 512 x 512, one tile a CTA) the chain of B's load
// (0.4 us), products (0.6), epilogue (1.0) and the hand-over to the next launch (1.2): 6.5 us a layer with A
// loaded after the wait, the roles of A and B exchanged and one chunk a stage, now 3.5 (backward 4.1); the fit
// network's training step 103 -> 71.5 us. The large ones (4096 x 1024 x 1024) the epilogue, issue of the
// activation's instructions and 33.6 MB of outputs (FP32 pre-activation, BF16 activation and its transpose):
// the step of a 1024-wide network at 4,096 rows 399 -> 304 us. 4096^3 alone 165 -> 104 us.
__global__ void __launch_bounds__(kGemmThreads, 1) k_gemm_tn(const __grid_constant__ GemmLaunch p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ unsigned long long full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t tmem_slot;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
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
        tc_bar_init(&drained, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    bool ok = true;
    const uint32_t ring = tc_smem(smem), stage = p.stage_size, ring_end = ring + S * stage, G = p.group;
    const uint32_t full0 = tc_smem(full), empty0 = tc_smem(empty), polls = p.polls;
    uint32_t fills = 0;  // of ring stages, by the producing lane
    if (warp == 0) {  // producer
        uint32_t t = blockIdx.x;
        TileAt x = tile_at(p, min(t, tiles - 1));
        const CUtensorMap *ma = &p.map[x.q][0], *mb = &p.map[x.q][1];
        uint32_t early = t < tiles ? min(x.nk, S * G) : 0;
        const bool one = tc_elect();
        auto load = [&](const CUtensorMap* map, uint32_t to, uint32_t pitch, uint32_t c, uint32_t end, uint32_t row, uint32_t bar) {
            for (; c < end; ++c, to += pitch) tc_tma_load_2d(to, map, (int32_t)(c * kTileK), (int32_t)row, bar);
        };
        // A of the first tile's chunks that the ring holds; after the wait their B.
        if (one)
            for (uint32_t c = 0, s = 0; c < early; c += G, ++s) {
                const uint32_t end = min(c + G, x.nk);
                tc_bar_expect_tx(full0 + 8 * s, (end - c) * (aBytes + x.tn * kTileK * 2));
                load(ma, ring + s * stage, aBytes, c, end, x.m0, full0 + 8 * s);
            }
        griddep_wait();
        if (one) {
            uint32_t s = 0, round = 0;
            for (uint32_t c = 0; c < early; c += G, ++s)
                load(mb, ring + s * stage + G * aBytes, x.tn * kTileK * 2, c, min(c + G, x.nk), x.n0, full0 + 8 * s);
            griddep_launch_dependents();
            if (s == S) {
                s = 0;
                round = 1;
            }
            // The rest, as stages come free.
            while (t < tiles && ok) {
                for (uint32_t c = early; c < x.nk; c += G) {
                    if (round > 0) ok = tc_bar_wait(empty0 + 8 * s, (round - 1) & 1u, polls);
                    if (!ok) break;
                    const uint32_t bar = full0 + 8 * s, sa = ring + s * stage, end = min(c + G, x.nk);
                    tc_bar_expect_tx(bar, (end - c) * (aBytes + x.tn * kTileK * 2));
                    load(ma, sa, aBytes, c, end, x.m0, bar);
                    load(mb, sa + G * aBytes, x.tn * kTileK * 2, c, end, x.n0, bar);
                    if (++s == S) {
                        s = 0;
                        ++round;
                    }
                }
                early = 0;
                t += gridDim.x;
                if (t < tiles) {
                    x = tile_at(p, t);
                    ma = &p.map[x.q][0];
                    mb = &p.map[x.q][1];
                }
            }
            fills = round * S + s;
        }
    } else if (warp == 1) {  // tensor-core issuer
        uint32_t sa = ring, bar = full0, phase = 0, li = 0;
        for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++li) {
            const TileAt x = tile_at(p, t);
            const uint32_t a = li & 1u, idesc = tc_idesc_bf16(kTileM, x.nt), d = tmem + a * p.acc_cols;
            if (li >= 2) ok = __all_sync(0xffffffffu, tc_bar_wait(tc_smem(&acc_empty[a]), ((li >> 1) - 1) & 1u, polls));
            if (!ok) break;
            tc_fence_after();
            // Steps whose stage is filled again: all but the CTA's last S.
            const uint32_t steps = (x.nk + G - 1) / G, refilled = t + gridDim.x < tiles ? x.nk : (steps - min(steps, S)) * G;
            const uint32_t bstep = x.tn * kTileK * 2 / 16;
            for (uint32_t c = 0; c < x.nk; c += G) {
                ok = __all_sync(0xffffffffu, tc_bar_wait(bar, phase, polls));
                if (!ok) break;
                tc_fence_after();
                const uint64_t da = tc_desc_sw128(sa), db = tc_desc_sw128(sa + G * aBytes);
                const uint32_t n = min(G, x.nk - c);
                if (tc_elect()) {
                    uint64_t ag = da, bg = db;
                    uint32_t g = 0;
                    do {
#pragma unroll
                        for (uint32_t kk = 0; kk < 4; ++kk)  // a K=16 slice is 32 bytes on: 2 in the descriptor
                            tc_mma(d, ag + 2 * kk, bg + 2 * kk, idesc, c + g + kk > 0);
                        ag += aBytes / 16;
                        bg += bstep;
                    } while (++g < n);
                    if (c < refilled) tc_commit(bar + (empty0 - full0));
                }
                sa += stage;
                bar += 8;
                if (sa == ring_end) {
                    sa = ring;
                    bar = full0;
                    phase ^= 1u;
                }
            }
            if (tc_elect() && ok) tc_commit(tc_smem(&acc_full[a]));
        }
    } else if (warp >= 2 && warp < 2 + kEpiWarps) {  // epilogue
        const uint32_t quarter = warp & 3u, part = (warp - 2) >> 2;
        uint32_t li = 0;
        for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++li) {
            const TileAt x = tile_at(p, t);
            const GemmArgs& g = p.g[x.q];
            const uint32_t a = li & 1u, m = x.m0 + quarter * 32 + lane;
            const uint32_t d = tmem + a * p.acc_cols + ((quarter * 32u) << 16);
            auto ready = [&] {
                if (li == 0) griddep_wait();
                ok = __all_sync(0xffffffffu, tc_bar_wait(tc_smem(&acc_full[a]), (li >> 1) & 1u, polls));  // warp-uniform
                tc_fence_after();
                return ok;
            };
            // A tile of 16 columns gives each of the four warps four.
            float e2 = x.tn < 32 ? tile_epilogue<4>(g, m, x.n0, x.nt, part, d, lane, ready)
                                 : tile_epilogue<8>(g, m, x.n0, x.nt, part, d, lane, ready);
            if (!ok) break;
            if (g.epi == kEpiLoss) {
                for (int o = 16; o > 0; o >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, o);
                if (lane == 0 && e2 != 0.0f) atomicAdd(g.loss, e2 / (float)(g.N * g.nout));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_bar_arrive(tc_smem(&acc_empty[a]));
        }
    } else if (warp >= 2 + kEpiWarps && p.cs.cols) {
        griddep_wait();
        if (p.loss && blockIdx.x == 0 && warp == 2 + kEpiWarps && lane == 0) *(volatile float*)p.host_loss = __ldcg(p.loss);
        column_sums(p.cs, blockIdx.x * 2 + (warp - 2 - kEpiWarps), gridDim.x * 2, lane);
    }
    if (!ok) {
        atomicOr(p.err, 1u);
        if (p.host_err) *(volatile uint32_t*)p.host_err = 1u;
    }
    tc_fence_before();
    if (__syncthreads_or(!ok)) {
        for (uint32_t f = fills - min(fills, S); f < fills; ++f) tc_bar_wait(full0 + 8 * (f % S), (f / S) & 1u);
        if (warp == 1 && tc_elect()) {
            tc_commit(tc_smem(&drained));
            tc_bar_wait(tc_smem(&drained), 0u);
        }
        tc_fence_before();
        __syncthreads();
    }
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

// Model of a CTA's time on one tile, in cycles: its operands and products, (128 + tn) rows of 128 bytes per K
// chunk at 90 bytes a cycle, and its epilogue, by 32 columns: 2,500 with an activation or a loss and BF16
// copies (16 columns 1,700), 900 for a plain store.
struct TileCost {
    double main, epi;
};
TileCost tile_cost(const GemmArgs& g, uint32_t tn)
{
    const bool plain = g.epi == kEpiStore || g.epi == kEpiLinear;
    const double per = plain ? 900.0 : 2500.0;
    return {(g.K + kTileK - 1) / kTileK * (kTileM + tn) * 1.4,
            tn < 32 ? (plain ? 700.0 : 1700.0) : per * tn / 32};
}

// Columns per tile of each of the n products of a launch on num_sm SMs: the pair with the smallest
// modelled time. Narrow tiles win while wide ones leave SMs idle, wide ones once every SM has work (fewer
// operand loads per output) up to where the epilogue of a CTA's last tile, which nothing overlaps, weighs
// more. Measured with forward and signal tiles of a columns and weight-gradient tiles of b (a/b): training
// step of the fit network (256 x 512) 71.8 us at 16/32, 71.8 at 16/64, 75.5 at 32/32, 83 at 32/128 and 97 at
// 64/64; of a 1024-wide network at 4,096 rows 304 at 128/64, 314 at 128/128, 326 at 64/64 and 256/64, 335 at
// 256/256.
void choose_tiles(const GemmArgs* g, uint32_t n, uint32_t num_sm, uint32_t (&tn)[2])
{
    constexpr double kPerTile = 1500.0;  // barriers and hand-over of a tile
    double best = 1e300;
    for (uint32_t a = kMinTileN; a <= kMaxTileN; a *= 2)
        for (uint32_t b = kMinTileN; b <= (n > 1 ? kMaxTileN : kMinTileN); b *= 2) {
            double work = 0.0, longest = 0.0;
            uint32_t tiles = 0;
            for (uint32_t i = 0; i < n; ++i) {
                const TileCost c = tile_cost(g[i], i ? b : a);
                const uint32_t t = tile_count(g[i], i ? b : a);
                tiles += t;
                work += t * (std::max(c.main, c.epi) + kPerTile);  // loads overlap the epilogue before them
                longest = std::max(longest, c.main + c.epi + kPerTile);
            }
            const uint32_t waves = (tiles + num_sm - 1) / num_sm;
            // One product fills whole waves; two of different cost fill the gaps of each other.
            const double cost = waves <= 1 ? longest
                                : n == 1   ? waves * work / tiles + std::min(tile_cost(g[0], a).main, tile_cost(g[0], a).epi)
                                           : work / num_sm + 0.75 * longest;
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
int gemm_launch(const GemmArgs* g, uint32_t n, const ColumnSums& cs, uint32_t* err, uint32_t* host_err, cudaStream_t st,
                uint32_t num_sm, bool pdl, const float* loss = nullptr, float* host_loss = nullptr,
                uint32_t polls = kTcMaxPolls)
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
    p.group = std::min(p.acc_cols <= 64 ? 4u : p.acc_cols <= 128 ? 2u : 1u, nk);
    p.stage_size = p.group * (kTileM + p.acc_cols) * kTileK * 2;
    p.stages = std::min({kStageBudget / p.stage_size, kMaxStages,
                         (nk + p.group - 1) / p.group * (p.tiles[0] + p.tiles[1] > num_sm ? 2u : 1u)});
    p.cs = cs;
    p.err = err;
    p.host_err = host_err;
    p.loss = loss;
    p.host_loss = host_loss;
    p.polls = polls;
    // CTAs without a tile only add column sums (four columns each pass).
    const uint32_t ctas = std::min(std::max(p.tiles[0] + p.tiles[1], (cs.cols + 3) / 4), num_sm);
    return launch_pdl(k_gemm_tn, dim3(ctas), dim3(kGemmThreads),
                      p.stages * p.stage_size + 1024, st, pdl, p);
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
size_t up256(size_t x) { return (x + 255) & ~(size_t)255; }

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
    // Pinned: loss and error word, written by the products.
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
        g.A = n->wb[l];
        g.B = l == 0 ? n->x : n->h[l - 1];
        g.lda = g.ldb = in;
        g.M = out;
        g.N = rows;
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
        e = gemm_launch(&g, 1, ColumnSums{}, n->err, &n->back[1], st, n->num_sm, true);
    }
    return e;
}

// One launch per layer: dZ_{l-1} = (dZ_l W_l) * silu'(Z_{l-1}) (M = in, N = rows, K = out), dW_l =
// dZ_l^T H_{l-1} (M = in, N = out, K = rows) and db_l = column sums of dZ_l.
int mlp_backward(arbo_mlp* n, uint32_t rows, cudaStream_t st)
{
    const uint32_t ld = n->maxb, L = n->L;
    bf16 *dz = n->d0, *dzt = n->d0t, *nd = n->d1, *ndt = n->d1t;
    int e = 0;
    for (uint32_t l = L; l-- > 0 && !e;) {
        const uint32_t in = n->dim[l], out = n->dim[l + 1];
        GemmArgs g[2] = {};
        GemmArgs& w = g[l > 0 ? 1 : 0];
        w.A = l == 0 ? n->xt : n->ht[l - 1];
        w.B = dzt;
        w.lda = w.ldb = ld;
        w.M = in;
        w.N = out;
        w.K = rows;
        w.epi = kEpiStore;
        w.outf = n->dw[l];
        w.ldof = in;
        if (l > 0) {
            g[0].A = n->wt[l];
            g[0].B = dz;
            g[0].lda = g[0].ldb = out;
            g[0].M = in;
            g[0].N = rows;
            g[0].K = out;
            g[0].epi = kEpiBackward;
            g[0].zprev = n->z[l - 1];
            g[0].ldz = g[0].ldob = in;
            g[0].outb = nd;
            g[0].outt = ndt;
            g[0].ldot = ld;
        }
        e = gemm_launch(g, l > 0 ? 2 : 1, ColumnSums{dzt, ld, rows, out, n->db[l]}, n->err, &n->back[1], st, n->num_sm, true,
                        l + 1 == L ? n->loss : nullptr, (float*)n->back);
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

// Waits for the event recorded behind the products; the loss is in back[0] then.
int mlp_check_err(arbo_mlp* n)
{
    UCUDA(cudaEventSynchronize(n->done));
    const uint32_t e = n->back[1];
    if (e) return ufail(ARBO_ERR_CUDA, "tensor-core product: an mbarrier wait ran out (error word " + std::to_string(e) + ")");
    return ARBO_OK;
}

// Upload, forward and backward pass, all enqueued on st with the event behind them.
int mlp_gradients(arbo_mlp* n, const float* x, const float* t, uint32_t rows, cudaStream_t st)
{
    int e = mlp_upload(n, x, t, rows, st);
    if (e) return e;
    if ((e = mlp_enqueue(n, rows, true, st)))
        return ufail(ARBO_ERR_CUDA, std::string("forward/backward: ") + cudaGetErrorString((cudaError_t)e));
    UCUDA(cudaEventRecord(n->done, st));
    return ARBO_OK;
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
    std::memset(n->back, 0, 8);
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
    UCUDA(cudaEventRecord(n->done, st));
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
    g.A = db;
    g.B = da;
    g.lda = g.ldb = K;
    g.M = g.ldof = N;
    g.N = M;
    g.K = K;
    g.epi = kEpiStore;
    g.outf = dc;
    int sms = 152, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto product = [&]() { return gemm_launch(&g, 1, ColumnSums{}, derr, nullptr, nullptr, (uint32_t)sms, false); };
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

// A product of zeros whose waits all run out at once, with the first copies in flight: its error word.
int arbo_selftest_stalled_product(uint32_t M, uint32_t N, uint32_t K, uint32_t* err)
{
    if (!err || M == 0 || N == 0 || K == 0 || N % 16 || K % 16)
        return ufail(ARBO_ERR_INVALID, "arbo_selftest_stalled_product: N and K multiples of 16");
    UCUDA(cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmemMax));
    const size_t na = up256((size_t)N * K * 2), nb = up256((size_t)M * K * 2), nc = up256((size_t)M * N * 4);
    char* base = nullptr;
    UCUDA(cudaMalloc(&base, na + nb + nc + 256));
    GemmArgs g{};
    g.A = (const bf16*)base;
    g.B = (const bf16*)(base + na);
    g.lda = g.ldb = K;
    g.M = g.ldof = N;
    g.N = M;
    g.K = K;
    g.epi = kEpiStore;
    g.outf = (float*)(base + na + nb);
    uint32_t* derr = (uint32_t*)(base + na + nb + nc);
    int sms = 152, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaMemset(base, 0, na + nb + nc + 256);
    if (e == cudaSuccess)
        e = (cudaError_t)gemm_launch(&g, 1, ColumnSums{}, derr, nullptr, nullptr, (uint32_t)sms, false, nullptr, nullptr, 0);
    if (e == cudaSuccess) e = cudaMemcpy(err, derr, 4, cudaMemcpyDeviceToHost);
    cudaFree(base);
    if (e != cudaSuccess) return ufail(ARBO_ERR_CUDA, std::string("stalled product: ") + cudaGetErrorString(e));
    return ARBO_OK;
}

}  // extern "C"
