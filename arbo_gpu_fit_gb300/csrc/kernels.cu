// kernels.cu — sm_103a kernels of one simulation time step and of its initialisation.
//
// One step is three launches (captured in CUDA graphs by the host after a handle's first steps):
//   k_demog   human and mosquito demographic passes over the whole census (HBM stream: a
//             human's next event time, a mosquito slot's event code; ages are birth times,
//             so a survivor without a transition writes nothing), per-tile
//             mosquito recruitment, counter deltas; replaces nBlockBirthDeath + resetIncidence
//             + mBlockBirthDeath (cpp/ndemographic.cu:32-120, cpp/mdemographic.cu:22-150).
//   k_foi     per (serotype, community): the series row of the next time point, then the
//             force of infection both ways with stay / long-distance / CSR-local dispersal;
//             replaces dataCollect + initialTransmission + nVisitingInfected +
//             mVisitingInfected (cpp/datacollect.cu:10-189, cpp/epidemic.cu:12-29,
//             cpp/nepidemic.cu:28-142, cpp/mepidemic.cu:28-138).
//   k_infect  one warp per community: event-parallel infection draws resolved to the
//             reference's serial order among the warp's lanes or by a minimum order key per target, external
//             introductions, application of the winners; replaces nmTransmission +
//             mnTransmission (cpp/mepidemic.cu:143-246, cpp/nepidemic.cu:146-319).
// No tensor cores: the work is integer streaming and scattered events.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "../../include/arbo.h"
#include "launch.cuh"
#include "sim_internal.h"

namespace arbo {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t comm_of(const uint32_t* __restrict__ loc, uint32_t P, uint32_t i)
{
    // Largest c < P with loc[c] <= i: the community whose contiguous range holds index i.
    uint32_t lo = 0, hi = P;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&loc[mid]) <= i) lo = mid; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ float cdf_at(const float* __restrict__ t, uint32_t n, int32_t a)
{
    const uint32_t i = a < 0 ? 0u : (uint32_t)a;
    return __ldg(&t[i < n ? i : n - 1]);
}

__device__ __forceinline__ uint32_t lower_bound_f(const float* __restrict__ t, uint32_t n, float v)
{
    // First index with t[index] >= v (n-1 if none): the first age whose cumulative survival
    // reaches the drawn value, as the linear scans of cpp/demographicintial.cu:124-137.
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&t[mid]) >= v) hi = mid; else lo = mid + 1;
    }
    return lo;
}

__device__ __forceinline__ Key load_key(const Ctrl* c)
{
    Key k;
    k.k0 = c->k0;
    k.k1 = c->k1;
    k.instance = c->instance;
    return k;
}

// The step a body works on: its number, its winner epoch and the random key of the simulation.
struct StepAt {
    uint32_t t, epoch;
    Key key;
};

__device__ __forceinline__ StepAt load_step(const Ctrl* c, uint32_t koff)
{
    StepAt at;
    at.t = c->t + koff;
    at.epoch = c->epoch + koff;
    at.key = load_key(c);
    return at;
}

__device__ __forceinline__ void counter_dec(uint32_t* p, Ctrl* ctrl)
{
    if (atomicSub(p, 1u) == 0u) atomicOr(&ctrl->err, ARBO_DEVERR_COUNTER);
}

__device__ __forceinline__ unsigned long long order_key(uint32_t hiword, uint32_t j, uint32_t intro, uint32_t e)
{
    return ((unsigned long long)hiword << 32) | ((j << 29) | (intro << 28) | e);
}

// ------------------------------------------------------------------ demographic pass

// First age whose CDF reaches ple: the death test "ple <= CDF(age)" of the reference
// (cpp/ndemographic.cu:62, cpp/mdemographic.cu:72) holds exactly when age >= this value, because
// the CDF table is non-decreasing; it is evaluated once per birth instead of a table gather (or
// powf/expf) per agent per step. Inverse bucket table of 2^bits + 2 entries: with
// j = floor(ple * 2^bits), minv[j] (first age with CDF >= j / 2^bits) and minv[j+1] bracket the
// answer, so a short binary search between them is exact. minv[2^bits + 1] = table size (none).
__device__ __forceinline__ int32_t death_age_inv(const float* __restrict__ cdf, const uint32_t* __restrict__ minv,
                                                 uint32_t n, float ple, float scale)
{
    const uint32_t j = (uint32_t)(ple * scale);
    uint32_t lo = __ldg(&minv[j]), hi = __ldg(&minv[j + 1]);
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&cdf[mid]) >= ple) hi = mid; else lo = mid + 1;
    }
    return lo >= n ? INT_MAX : (int32_t)lo;
}

// The same for mosquitoes with the bucket's first age and the CDF there in one load: a bucket of 1/4096
// holds at most one age step except in the far tail (ages past 60 at a mean of 10 days), where the
// search runs.
__device__ __forceinline__ int32_t death_age_lut(const Dev& d, float ple)
{
    const uint2 e = __ldg(&d.mlut[(uint32_t)(ple * 4096.0f)]);
    if (e.x & kLutWide) return death_age_inv(d.cdfm, d.minv, d.am, ple, 4096.0f);
    const uint32_t a = e.x + (__uint_as_float(e.y) >= ple ? 0u : 1u);
    return a >= d.am ? INT_MAX : (int32_t)a;
}

// Per-warp shared staging of the demographic pass.
struct QuadSmem {
    uint4 code[32];
    uint32_t c0[kQuad], end[kQuad], end2[kQuad];  // community of each tile's first slot; where it and the next end
    uint4 draw[32];  // rebirth draws of ranks 4s .. 4s+3 of tile u, by the lane 8u + s that made them; 31: quota draws
    union {
        uint8_t slot[kQuad][kTile];    // reborn slot offsets by rank
        uint16_t deep[kQuad * kTile];  // slots with a deep event; a human pass's agents with an event due
    };
};

// Community of human i.
__device__ __forceinline__ uint32_t human_comm(const uint32_t* __restrict__ nloc, const uint32_t* __restrict__ hcomm,
                                               uint32_t P, uint32_t i)
{
    const uint32_t h = __ldg(&hcomm[i / kHumanBlock]);
    uint32_t c = h & ~kTileSpans;
    if (h & kTileSpans)
        while (c + 1 < P && __ldg(&nloc[c + 1]) <= i) ++c;
    return c;
}

// Human i in the step that reaches time tn, at or after its next event time: a transition of an
// exposed or infectious human, a death with rebirth, or (after a census write) neither yet.
__device__ __forceinline__ void human_due(const Dev& d, const Key key, uint32_t i, int32_t tn)
{
    uint32_t st = d.n_status[i];
    const int32_t dt = d.n_dtime[i], born = d.n_born[i], ex = d.n_exposed[i], rec = d.n_recovery[i];
    const uint32_t s = d.n_strain[i], c = human_comm(d.nloc, d.hcomm, d.P, i);
    if (tn < dt) {
        const int32_t a = tn - born;
        if (st == 2 && rec < a) {
            counter_dec(&d.infh[s * d.P + c], d.ctrl);
            d.n_status[i] = (uint8_t)(st = 0);
        } else if (st == 1 && ex < a) {
            atomicAdd(&d.inc[s * d.P + c], 1u);
            atomicAdd(&d.infh[s * d.P + c], 1u);
            d.n_status[i] = (uint8_t)(st = 2);
        }
        d.n_next[i] = human_next(st, dt, born, st == 1 ? ex : rec);
        return;
    }
    if (st == 2) counter_dec(&d.infh[s * d.P + c], d.ctrl);
    const U4 r = draw4(key, kHumanRebirth, i >> 2, (uint32_t)(tn - 1));
    const float ple = u01(r.v[i & 3]);
    const int32_t nd = death_time(tn, death_age_inv(d.cdfh, d.minvh, d.ah, ple, 65536.0f));
    d.n_ple[i] = ple;
    d.n_born[i] = tn;
    d.n_dtime[i] = nd;
    d.n_next[i] = nd;
    d.n_imm[i] = 0;
    d.n_status[i] = 0;
}

// Human pass of one warp over U rows of 32 groups of four, `stride` groups apart (g0: this lane's
// first group; cpp/ndemographic.cu:32-105): ageing is implicit in the birth times, and each human's
// next event time (its death, or its exposed-to-infectious or recovery step, whichever comes first)
// is kept up to date by every writer of its status, so the pass streams only that time. The agents
// with an event due are listed and taken one per lane: their status, times and ages are one round
// trip for the whole warp. Worked off by the lane that streamed them, four agents in turn and each
// kind of event by itself, the chain of the last warps set the end of the pass (a step of 5e4 agents
// 18.9 -> 15.0 us, of 7 M 34 -> 28 us, with the mosquitoes' deep events taken the same way).
template <int U>
__device__ __forceinline__ void demog_humans(const Dev& d, const Key key, uint32_t g0, uint32_t stride, uint32_t t,
                                             QuadSmem& sm)
{
    const uint32_t lane = threadIdx.x & 31u;
    int4 X[U];
    const int32_t tn = (int32_t)t + 1;
    int32_t first = INT_MAX;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t g = g0 + u * stride;
        X[u] = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);  // as padding
        if (g < d.nvec) X[u] = __ldcs(reinterpret_cast<const int4*>(d.n_next) + g);
        first = min(first, min(min(X[u].x, X[u].y), min(X[u].z, X[u].w)));
    }
    if (!__any_sync(kFull, tn >= first)) return;
    uint32_t n = 0;
    const uint32_t below = (1u << lane) - 1u;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int32_t x[4] = {X[u].x, X[u].y, X[u].z, X[u].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned bal = __ballot_sync(kFull, tn >= x[k]);
            if (tn >= x[k]) sm.deep[n + __popc(bal & below)] = (uint16_t)((u << 7) | (lane << 2) | k);
            n += __popc(bal);
        }
    }
    __syncwarp();
    for (uint32_t j = lane; j < n; j += 32) {
        const uint32_t e = sm.deep[j];
        human_due(d, key, 4 * (g0 - lane + (e >> 7) * stride) + (e & 127u), tn);
    }
    __syncwarp();
}

// Community of slot i at or after community c, which ends at slot `end`, the next one at `end2` (c and
// end move on; few tiles reach into a third community).
__device__ __forceinline__ void comm_forward(const Dev& d, uint32_t i, uint32_t& c, uint32_t& end, uint32_t end2)
{
    if (i >= end && end < end2) ++c, end = end2;
    while (i >= end) end = __ldg(&d.mloc[++c + 1]);
}

__device__ __forceinline__ uint32_t slot_comm(const Dev& d, uint32_t c0, uint32_t i)
{
    uint32_t c = c0;
    while (c + 1 < d.P && __ldg(&d.mloc[c + 1]) <= i) ++c;
    return c;
}

// Community of mosquito slot i.
__device__ __forceinline__ uint32_t mosq_comm(const Dev& d, uint32_t i)
{
    const uint32_t c = __ldg(&d.tcomm[i / kTile]);
    return (c & kTileSpans) ? slot_comm(d, c & ~kTileSpans, i) : c;
}

// A live slot whose event is due in the step that reaches time tn and is not the plain death of a
// susceptible mosquito: its death, its latent-to-infectious transition, or neither yet. Returns its
// new code. c, end, end2: the community of its tile's first slot and where that and the next one end.
__device__ __forceinline__ uint32_t mosq_deep(const Dev& d, uint32_t i, int32_t tn, uint32_t c, uint32_t end, uint32_t end2)
{
    const int2 r = *reinterpret_cast<const int2*>(d.m_life + i);  // born, dtime
    uint32_t st = d.m_stat[i] & 3u;
    const int32_t ex = d.m_exposed[i];
    const uint32_t s = d.m_strain[i];
    comm_forward(d, i, c, end, end2);
    if (tn >= r.y) {
        if (st == 2) counter_dec(&d.infm[s * d.P + c], d.ctrl);
        return st ? (uint32_t)(kDead | kDeep) : (uint32_t)kDead;
    }
    if (st == 1 && ex < tn - r.x) {
        st = 2;
        d.m_stat[i] = 2;
        atomicAdd(&d.infm[s * d.P + c], 1u);
    }
    return mosq_code(mosq_next(st, r.y, r.x, ex), tn, st != 0);
}

// Bit 7 of each byte of x (the other bits zero) gathered into a 4-bit mask (byte k -> bit k).
__device__ __forceinline__ uint32_t nibble7(uint32_t x)
{
    return ((x >> 7) * 0x01020408u) >> 24;
}

__device__ __forceinline__ uint32_t pick4(const U4& v, uint32_t i)
{
    return i == 0 ? v.v[0] : i == 1 ? v.v[1] : i == 2 ? v.v[2] : v.v[3];
}

// What a quad needs that no step kernel writes, made while the previous pass ends: the tile's community,
// the expected mosquitoes, and (left in the staging) the quad's quota draws and the draws of the first 28
// births of each tile, which are keyed by rank and not by slot.
struct QuadStart {
    uint32_t c0, end, end2;
    float target;
};

__device__ __forceinline__ QuadStart quad_start(const Dev& d, const Key key, uint32_t q, uint32_t lane, uint32_t t,
                                                QuadSmem& sm)
{
    const uint32_t u = lane >> 3, b = q * kQuad + u;
    const bool live = b < d.tiles;
    QuadStart at;
    at.c0 = live ? __ldg(&d.tcomm[b]) : 0u;
    at.end = at.end2 = ~0u;
    if (at.c0 & kTileSpans) {
        at.end = __ldg(&d.mloc[(at.c0 & ~kTileSpans) + 1]);
        at.end2 = __ldg(&d.mloc[(at.c0 & ~kTileSpans) + 2]);
    }
    if ((lane & 7u) == 0) {
        sm.c0[u] = at.c0 & ~kTileSpans;
        sm.end[u] = at.end;
        sm.end2[u] = at.end2;
    }
    at.target = __ldg(&d.etab[t + 1]);
    const bool quota = lane == 31;  // one Philox call a lane: the last one makes the quota draws
    const U4 r = draw4(key, quota ? kMosquitoTile : kMosquitoRebirth, quota ? q : b, t, quota ? 0u : lane & 7u);
    sm.draw[lane] = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
    return at;
}

// The carried dead count of the lane's tile. The last step's pass wrote it, so it is loaded after the wait,
// in the same round trip as the codes.
__device__ __forceinline__ int32_t quad_ledger(const Dev& d, uint32_t q, uint32_t lane)
{
    const uint32_t b = q * kQuad + (lane >> 3);
    return b < d.tiles ? d.ledger[b] : 0;
}

// One warp, tiles 4q..4q+3; lane l holds the codes of slots 16(l mod 8) .. +15 of tile 4q + l/8, four
// words. Per tile: deaths (a live slot dies in the step that reaches its death time), the birth quota
// (cpp/mdemographic.cu:104-129) from the carried dead count, rebirth of the lowest-index dead slots, the
// net change of each community's alive count. The quota draws of the four tiles come from one Philox
// call; the r-th reborn slot of tile b takes component r&3 of the call keyed (b, t, r>>2).
//
// What bounds it: instruction issue. The whole test of a slot is a byte compare (three instructions for
// four slots): its code holds the low bits of its next event time, and a susceptible mosquito's event is
// its death, so nothing else is read. Before, a slot's state byte and 4-byte death time were streamed
// and tested one slot at a time (1,150 warp instructions a quad); demographic phase of 14 M agents 60 ->
// 42 us, of 128 instances of 7e4 agents 79 -> 42 us (with the human pass above). Owner lanes post the offset of each
// reborn slot under its rank; one lane per reborn slot then draws its PLE and writes its life record
// (one sector instead of three) and its code, which the owners write back with one 16-byte store.
__device__ __forceinline__ void mosquito_quad_core(const Dev& d, const Key key, uint32_t q, uint32_t lane, uint32_t t,
                                                   QuadSmem& sm, const QuadStart& at, const int32_t led, const uint4 A)
{
    const int32_t tn = (int32_t)t + 1;
    const uint32_t u = lane >> 3, seg = lane & 7u, b = q * kQuad + u;
    const bool live = b < d.tiles;
    const uint32_t c0 = at.c0;

    uint32_t aw[4] = {A.x, A.y, A.z, A.w}, z[4], deep = 0;
    const uint32_t now4 = ((uint32_t)tn & 63u) * 0x01010101u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        // Bytes with code == now: the sum reaches bit 7 in every other byte (no carry between bytes).
        z[j] = ~((((aw[j] & 0x3F3F3F3Fu) ^ now4) + 0x7F7F7F7Fu) | aw[j]) & 0x80808080u;
        deep |= z[j] & (aw[j] << 1);
    }
    bool chg = (z[0] | z[1] | z[2] | z[3]) != 0;
    uint32_t dead[4] = {0, 0, 0, 0};  // died in the deep path
    if (__any_sync(kFull, deep != 0)) {
        // One lane per deep event of the quad, whoever owns its slot: its loads are one round trip.
        uint32_t zd[4], m = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            zd[j] = z[j] & (aw[j] << 1);
            z[j] &= ~zd[j];
            m |= nibble7(zd[j]) << (4 * j);
        }
        const uint32_t cnt = __popc(m);
        uint32_t at = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, at, off);
            if (lane >= (uint32_t)off) at += y;
        }
        const uint32_t total = __shfl_sync(kFull, at, 31);
        for (at -= cnt; m; m &= m - 1) sm.deep[at++] = (uint16_t)(16 * lane + __ffs(m) - 1);
        sm.code[lane] = make_uint4(aw[0], aw[1], aw[2], aw[3]);
        __syncwarp();
        for (uint32_t j = lane; j < total; j += 32) {
            const uint32_t o = sm.deep[j];
            reinterpret_cast<uint8_t*>(sm.code)[o] = (uint8_t)mosq_deep(d, q * kQuad * kTile + o, tn, sm.c0[o / kTile], sm.end[o / kTile], sm.end2[o / kTile]);
        }
        __syncwarp();
        const uint4 B = sm.code[lane];
        aw[0] = B.x, aw[1] = B.y, aw[2] = B.z, aw[3] = B.w;
#pragma unroll
        for (int j = 0; j < 4; ++j) dead[j] = zd[j] & aw[j];
    }
    // Plain deaths become kDead exactly; died: both kinds.
    uint32_t dm = 0, died = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        aw[j] = (aw[j] & ~((z[j] >> 7) * 0xFFu)) | z[j];
        z[j] |= dead[j];
        uint32_t dj = aw[j] & 0x80808080u;
        if (b == d.tiles - 1) dj &= ~__vcmpeq4(aw[j], 0xFFFFFFFFu);  // padding is in the last tile only
        dm |= nibble7(dj) << (4 * j);
        died |= z[j] >> (7 - j);  // byte k, bit j
    }
    if (!live) dm = 0;
    // Counts of the tile's eight lanes: exclusive dead count before this lane's slots (slot order) and
    // the tile's totals, dead in the low and died in the high half.
    const uint32_t own = (uint32_t)__popc(dm) | ((uint32_t)__popc(died) << 16);
    uint32_t incl = own;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, off, 8);
        if (seg >= (uint32_t)off) incl += y;
    }
    const uint32_t excl = (incl - own) & 0xFFFFu, tot = __shfl_sync(kFull, incl, 7, 8);
    const uint32_t dead_tot = tot & 0xFFFFu, died_tot = tot >> 16;
    // The quota, by every lane of the tile alike.
    uint32_t nb = 0;
    __syncwarp();
    if (live) {
        const uint32_t start = b * kTile;
        const uint32_t bt = (d.M - start) < kTile ? (d.M - start) : kTile;
        const uint32_t L = (uint32_t)led + died_tot;
        const float fbt = (float)bt;
        float x = __fmul_rn(at.target, fbt);
        x = __fdiv_rn(x, (float)d.M);
        x = __fsub_rn(x, fbt);
        x = __fadd_rn(x, (float)L);
        const int births = (int)resolve(x, reinterpret_cast<const uint32_t*>(sm.draw)[31 * 4 + u]);
        if (seg == 0) d.ledger[b] = (int32_t)L - births;
        nb = births > 0 ? min((uint32_t)births, dead_tot) : 0u;
    }
    const uint32_t mine = min(nb > excl ? nb - excl : 0u, own & 0xFFFFu);
    // The lowest `mine` dead slots of the lane, posted under their ranks.
    uint32_t born = 0;
    {
        uint32_t m = dm;
        for (uint32_t r = excl, n = mine; n; --n, ++r) {
            const uint32_t low = m & (0u - m);
            sm.slot[u][r] = (uint8_t)(16 * seg + 31 - __clz(low));
            m ^= low;
        }
        born = dm ^ m;
    }
    chg |= born != 0;
    if (live && (c0 & kTileSpans)) {
        // A tile across communities: the net change slot by slot.
        uint32_t died16 = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) died16 |= nibble7(z[j]) << (4 * j);
        uint32_t c = c0 & ~kTileSpans, end = at.end;
        for (uint32_t m = born ^ died16; m; m &= m - 1) {
            const uint32_t k = __ffs(m) - 1;
            comm_forward(d, b * kTile + 16 * seg + k, c, end, at.end2);
            atomicAdd(&d.mcnt[c], ((born >> k) & 1u) ? 1u : ~0u);
        }
    } else if (seg == 0 && nb != died_tot) {
        atomicAdd(&d.mcnt[c0], nb - died_tot);  // one atomic per tile
    }
    const uint32_t n0 = __shfl_sync(kFull, nb, 0), n1 = n0 + __shfl_sync(kFull, nb, 8), n2 = n1 + __shfl_sync(kFull, nb, 16);
    const uint32_t rtot = n2 + __shfl_sync(kFull, nb, 24);
    if (rtot) {
        sm.code[lane] = make_uint4(aw[0], aw[1], aw[2], aw[3]);
        __syncwarp();
        uint8_t* codes = reinterpret_cast<uint8_t*>(sm.code);
        for (uint32_t j = lane; j < rtot; j += 32) {
            const uint32_t v = (j >= n0 ? 1u : 0u) + (j >= n1 ? 1u : 0u) + (j >= n2 ? 1u : 0u);
            const uint32_t r = j - (v == 0 ? 0u : v == 1 ? n0 : v == 2 ? n1 : n2);
            uint32_t x;
            if (r < 28) x = reinterpret_cast<const uint32_t*>(sm.draw)[32 * v + r];
            else x = pick4(draw4(key, kMosquitoRebirth, q * kQuad + v, t, r >> 2), r & 3u);
            const float ple = u01(x);
            const uint32_t o = v * kTile + sm.slot[v][r], i = q * kQuad * kTile + o;
            const int32_t dt = death_time(tn, death_age_lut(d, ple));
            *reinterpret_cast<int4*>(d.m_life + i) = make_int4(tn, dt, __float_as_int(ple), 0);
            if (codes[o] & kDeep) d.m_stat[i] = 0;
            codes[o] = mosq_code(dt, tn, false);
        }
        __syncwarp();
        if (chg) reinterpret_cast<uint4*>(d.m_code)[q * 32 + lane] = sm.code[lane];
        __syncwarp();
    } else if (chg) {
        reinterpret_cast<uint4*>(d.m_code)[q * 32 + lane] = make_uint4(aw[0], aw[1], aw[2], aw[3]);
    }
}

// What a phase's work waits for once it has done what does not depend on the previous phase: nothing, the
// previous kernel of the stream, or (PendingWait) the previous phase of a cluster, once per warp and phase.
struct NoWait {
    __device__ __forceinline__ void operator()() const {}
};
struct GridWait {
    __device__ __forceinline__ void operator()() const { griddep_wait(); }
};
// In the infection pass the next step's demographic pass may be scheduled only then, so that when a pass
// starts, every kernel but the one before it has ended. What a pass reads before its own wait (step control,
// tables, network) no step kernel writes: an early start is promised earlier kernels' writes only after it.
struct GridWaitRelease {
    __device__ __forceinline__ void operator()() const
    {
        griddep_wait();
        griddep_launch_dependents();
    }
};

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Its two halves, for warps whose lanes the compiler may have apart.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

struct PendingWait {
    bool& pending;  // warp-uniform
    __device__ __forceinline__ void operator()() const
    {
        if (pending) cluster_wait();
        pending = false;
    }
};

// Quad with its codes loaded straight from global memory. The wait for the previous phase
// stands between what does not depend on it and the codes, which its infections change.
template <typename Wait>
__device__ __forceinline__ void demog_mosquito_quad(const Dev& d, const Key key, uint32_t q, uint32_t lane, uint32_t t,
                                                    QuadSmem& sm, Wait wait)
{
    const QuadStart at = quad_start(d, key, q, lane, t, sm);
    wait();
    uint4 A = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (q * kQuad + (lane >> 3) < d.tiles) A = reinterpret_cast<const uint4*>(d.m_code)[q * 32 + lane];
    mosquito_quad_core(d, key, q, lane, t, sm, at, quad_ledger(d, q, lane), A);
}

// ------------------------------------------------------------------ TMA-staged pipeline

// One warp's double buffer of quad codes, filled by bulk asynchronous copies.
struct TmaWarpSmem {
    uint4 stage[2][32];
    QuadSmem qs;
    unsigned long long mbar[2];
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// One arrival that also announces `bytes` of asynchronous transfers for the current phase.
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Bulk copy global -> shared (16-byte aligned addresses, size a multiple of 16) completing on bar.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Waits for the phase of `bar` with the given parity; gives up after a bounded number of polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity)
{
    const uint32_t a = smem_u32(bar);
    for (uint32_t it = 0; it < (1u << 20); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Lane 0 starts the copy of quad q into `st`.
__device__ __forceinline__ void issue_quad(const Dev& d, uint32_t q, uint4* st, unsigned long long* bar)
{
    const uint32_t b0 = q * kQuad;
    const uint32_t nt = min(kQuad, d.tiles - b0);
    // Order the warp's earlier generic reads of this buffer before the asynchronous writes.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(bar, nt * kTile);
    bulk_load(st, d.m_code + (size_t)b0 * kTile, nt * kTile, bar);
}

// Persistent demographic pass with TMA staging. Every warp first walks chunks of 32*U human
// groups (grid-stride), then its mosquito quads: lane 0 starts the bulk copy of the warp's next
// quad into the other half of its double buffer before the current quad is processed, so the
// census streams of all warps overlap with their arithmetic. Waits are bounded: on a timeout the
// kernel records ARBO_DEVERR_STALL, waits (bounded) for its own copy in flight and stops.
template <int U>
__global__ void __launch_bounds__(128, 4) k_demog_tma(Dev d, uint32_t koff)
{
    __shared__ TmaWarpSmem ws_all[4];
    const uint32_t t = d.ctrl->t + koff;
    const Key key = load_key(d.ctrl);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + warp, nw = gridDim.x * (blockDim.x >> 5);
    TmaWarpSmem& ws = ws_all[warp];
    const uint32_t quads = (d.tiles + kQuad - 1) / kQuad;
    if (lane == 0) {
        mbar_init(&ws.mbar[0], 1);
        mbar_init(&ws.mbar[1], 1);
        mbar_fence_init();
        if (gw < quads) issue_quad(d, gw, ws.stage[0], &ws.mbar[0]);
    }
    __syncwarp();
    const uint32_t hchunks = (d.nvec + 32 * U - 1) / (32 * U);
    for (uint32_t ch = gw; ch < hchunks; ch += nw) demog_humans<U>(d, key, ch * 32 * U + lane, 32, t, ws.qs);
    uint32_t phase = 0;  // bit s: parity to wait for on stage s
    uint32_t i = 0;
    for (uint32_t q = gw; q < quads; q += nw, ++i) {
        const uint32_t sidx = i & 1u;
        const uint32_t nq = q + nw;
        if (lane == 0 && nq < quads) issue_quad(d, nq, ws.stage[sidx ^ 1u], &ws.mbar[sidx ^ 1u]);
        const bool ok = mbar_wait(&ws.mbar[sidx], (phase >> sidx) & 1u);
        phase ^= 1u << sidx;
        if (!__all_sync(kFull, ok)) {
            if (lane == 0) {
                atomicOr(&d.ctrl->err, ARBO_DEVERR_STALL);
                if (nq < quads) mbar_wait(&ws.mbar[sidx ^ 1u], (phase >> (sidx ^ 1u)) & 1u);
            }
            break;
        }
        uint4 A = make_uint4(~0u, ~0u, ~0u, ~0u);
        if (q * kQuad + (lane >> 3) < d.tiles) A = ws.stage[sidx][lane];
        __syncwarp();  // every lane has its words before the buffer is refilled next iteration
        const int32_t led = quad_ledger(d, q, lane);
        mosquito_quad_core(d, key, q, lane, t, ws.qs, quad_start(d, key, q, lane, t, ws.qs), led, A);
    }
    griddep_launch_dependents();
}

// Demographic pass of one simulation, one warp item per warp: the mosquito quads first, then the rows of
// 32 * U human groups. With `spread`, neighbouring items go to different blocks, so that every block has
// its share of the long items (quads) and of the short ones; else blocks take consecutive items and the
// human blocks, which are short but end in latency chains, come last and fill the SMs that the last
// mosquito blocks leave idle. 40 registers, so that six blocks fit an SM; the body takes a little more and
// spills 8 bytes a thread.
template <int U>
__global__ void __launch_bounds__(256, 6) k_demog(Dev d, uint32_t spread, uint32_t koff)
{
    __shared__ QuadSmem wsm[8];
    const uint32_t t = d.ctrl->t + koff;
    const Key key = load_key(d.ctrl);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t quads = (d.tiles + kQuad - 1) / kQuad, rows = (d.nvec + 32 * U - 1) / (32 * U);
    const uint32_t it = spread ? warp * gridDim.x + blockIdx.x : blockIdx.x * (blockDim.x >> 5) + warp;
    if (it < quads) {
        demog_mosquito_quad(d, key, it, lane, t, wsm[warp], GridWait{});
    } else if (it - quads < rows) {
        griddep_wait();
        demog_humans<U>(d, key, (it - quads) * 32 * U + lane, 32, t, wsm[warp]);
    }
    griddep_launch_dependents();
}

// ------------------------------------------------------------------ series + force of infection

// Event count of a source and its split (cpp/nepidemic.cu:65-136): a noDistance share stays
// home (added to trans[pidx] here), a longDistance share of the rest goes to uniform
// communities, the remainder to uniform CSR neighbours; an isolated community keeps all.
__device__ __forceinline__ void split_events(const Dev& d, uint32_t* trans, float x, const U4& r, uint32_t pidx,
                                             uint32_t deg, uint32_t* nlocal, uint32_t* nlong)
{
    uint32_t n = (uint32_t)resolve(x, r.v[0]);
    if (n >= (1u << 26)) {
        atomicOr(&d.ctrl->err, ARBO_DEVERR_EVENT_OVERFLOW);
        n = (1u << 26) - 1;
    }
    uint32_t stay = n, lng = 0;
    if (deg > 0) {
        stay = (uint32_t)resolve(__fmul_rn((float)n, d.noDist), r.v[1]);
        n -= stay;
        lng = (uint32_t)resolve(__fmul_rn((float)n, d.longDist), r.v[2]);
        n -= lng;
    } else {
        n = 0;
    }
    if (stay) atomicAdd(&trans[pidx], stay);
    *nlocal = n;
    *nlong = lng;
}

// A count at or above 2^31 is a counter that went below zero (counter_dec records
// ARBO_DEVERR_COUNTER when that happens): it is read as 0, so that an inconsistent state cannot turn
// into an unbounded number of events.
__device__ __forceinline__ uint32_t checked_count(uint32_t x, uint32_t* bad)
{
    *bad |= x & 0x80000000u;
    return (x & 0x80000000u) ? 0u : x;
}

// Series row of the step and the reset of the incidence counters, by one warp for one serotype and 256
// consecutive communities (item s * series_chunks + chunk): its loads are one round trip, then one
// reduction and one atomic per series. Beside the force of infection and not in it: summed by the warps
// that spread the events, the row stood between their counters and their events.
__device__ __forceinline__ uint32_t series_chunks(uint32_t P) { return (P + 255) / 256; }

template <typename Wait>
__device__ __forceinline__ void foi_series(const Dev& d, uint32_t item, int collect_only, const StepAt& at, Wait wait)
{
    const uint32_t lane = threadIdx.x & 31u, S = d.S, P = d.P, chunks = series_chunks(P);
    const uint32_t s = item / chunks, c0 = (item - s * chunks) * 256 + lane;
    const uint32_t row = collect_only ? 0u : at.t + 1;
    uint32_t humans = 0;
    if (s == 0)
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
            if (c0 + 32 * k < P) humans += __ldg(&d.ncnt[c0 + 32 * k]);
    wait();
    uint32_t ih[8], im[8], ic[8], mc[8];
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t c = c0 + 32 * k;
        const bool ok = c < P;
        ih[k] = ok ? d.infh[s * P + c] : 0u;
        im[k] = ok ? d.infm[s * P + c] : 0u;
        ic[k] = ok ? d.inc[s * P + c] : 0u;
        mc[k] = ok && s == 0 ? d.mcnt[c] : 0u;
    }
    uint32_t si = 0, sm = 0, sc = 0, mosq = 0, bad = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t c = c0 + 32 * k;
        if (ic[k]) d.inc[s * P + c] = 0u;
        const uint32_t x = checked_count(ih[k], &bad);
        si += x;
        sm += checked_count(im[k], &bad);
        sc += checked_count(ic[k], &bad);
        mosq += checked_count(mc[k], &bad);
        if (c == 0) d.s_one[row * S + s] = x;
        if (d.recordSpatial && c < P) d.s_spatial[(size_t)row * S * P + s * P + c] = x;
    }
    if (bad) atomicOr(&d.ctrl->err, ARBO_DEVERR_COUNTER);
    si = __reduce_add_sync(kFull, si);
    sc = __reduce_add_sync(kFull, sc);
    sm = __reduce_add_sync(kFull, sm);
    if (lane == 0 && si) atomicAdd(&d.s_ninf[row * S + s], si);
    if (lane == 1 && sc) atomicAdd(&d.s_ninc[row * S + s], sc);
    if (lane == 2 && sm) atomicAdd(&d.s_minf[row * S + s], sm);
    if (s == 0) {
        humans = __reduce_add_sync(kFull, humans);
        mosq = __reduce_add_sync(kFull, mosq);
        if (lane == 3 && humans) atomicAdd(&d.s_ncount[row], humans);
        if (lane == 4 && mosq) atomicAdd(&d.s_mcount[row], mosq);
    }
}

// Force of infection, by one warp for kFoiPairs consecutive (serotype, community) pairs: lane l splits
// the events of pair l mod 16 in one direction (below 16 human to mosquito, else mosquito to human);
// then the 32 lanes spread the flattened events of the warp's 64 (lane, kind) entries, four per Philox
// call. No block barrier: a warp is a chain of two dependent round trips and its draws, so the more warps
// in flight the better. The wait for the previous phase stands between the loads of static
// data and those of its results.
constexpr uint32_t kFoiPairs = 16;

struct __align__(16) FoiWarpSmem {
    uint32_t to[kFoiPairs][8];  // CSR row of each pair's source community (degree <= 8)
    uint32_t base[32];          // first group of four events of each lane
    uint32_t local[32], far[32];  // a lane's events to neighbours and to any community
    uint32_t loc[kFoiPairs], deg[kFoiPairs], row[kFoiPairs];  // CSR row, its length, first counter of the serotype
};

template <typename Wait>
__device__ __forceinline__ void foi_events(const Dev& d, uint32_t p0, const StepAt& at, FoiWarpSmem& sh, Wait wait)
{
    const uint32_t lane = threadIdx.x & 31u, SP = d.S * d.P, P = d.P;
    const uint32_t slot = lane & (kFoiPairs - 1), p = p0 + slot;
    const bool hm = lane < kFoiPairs, valid = p < SP;
    uint32_t ncc = 0, loc = 0, deg = 0, s = 0, c = 0;
    U4 r;
    if (valid) {
        s = p / P;
        c = p - s * P;
        ncc = __ldg(&d.ncnt[c]);
        loc = __ldg(&d.csr_loc[c]);
        deg = __ldg(&d.csr_loc[c + 1]) - loc;
        if (deg <= 8)  // the two lanes of a pair fetch every second neighbour
            for (uint32_t q = hm ? 0u : 1u; q < deg; q += 2) sh.to[slot][q] = __ldg(&d.csr_to[loc + q]);
        if (hm) {
            sh.loc[slot] = loc;
            sh.deg[slot] = deg;
            sh.row[slot] = s * P;
        }
        r = draw4(at.key, hm ? kFoiHM : kFoiMH, p, at.t);
    }
    wait();
    uint32_t nlocal = 0, nfar = 0;
    if (valid) {
        uint32_t bad = 0;
        const uint32_t inf = checked_count(hm ? d.infh[p] : d.infm[p], &bad);
        const uint32_t mcc = checked_count(hm ? d.mcnt[c] : 0u, &bad);
        if (bad) atomicOr(&d.ctrl->err, ARBO_DEVERR_COUNTER);
        if (inf) {
            // Human to mosquito (cpp/nepidemic.cu:28-142), mosquito to human (cpp/mepidemic.cu:28-138).
            float x = hm ? __fmul_rn(__fmul_rn(__fdiv_rn((float)mcc, (float)ncc), d.biting), d.nmSuccess)
                         : __fmul_rn(d.biting, d.mnSuccess);
            x = __fmul_rn(x, (float)inf);
            split_events(d, hm ? d.transm : d.transh, x, r, p, deg, &nlocal, &nfar);
        }
    }
    const uint32_t own = ((nlocal + 3) >> 2) + ((nfar + 3) >> 2);
    sh.local[lane] = nlocal;
    sh.far[lane] = nfar;
    uint32_t v = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, v, off);
        if (lane >= (uint32_t)off) v += y;
    }
    sh.base[lane] = v - own;
    __syncwarp();
    const uint32_t G = __shfl_sync(kFull, v, 31);
    for (uint32_t gi = lane; gi < G; gi += 32) {
        uint32_t o = 0;  // last lane whose first group is <= gi
#pragma unroll
        for (uint32_t half = 16; half; half >>= 1)
            if (sh.base[o + half] <= gi) o += half;
        const uint32_t rel = gi - sh.base[o], nl = sh.local[o], gl = (nl + 3) >> 2;
        const bool far = rel >= gl, human = o < kFoiPairs;
        const uint32_t r4 = far ? rel - gl : rel, n = far ? sh.far[o] : nl, q = o & (kFoiPairs - 1);
        const uint32_t stream = human ? (far ? kFoiHMLong : kFoiHMLocal) : (far ? kFoiMHLong : kFoiMHLocal);
        uint32_t* trans = (human ? d.transm : d.transh) + sh.row[q];
        const U4 x = draw4(at.key, stream, p0 + q, at.t, r4);
        const uint32_t dg = sh.deg[q];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (4 * r4 + e >= n) break;
            uint32_t dest;
            if (far) dest = bounded(x.v[e], P);
            else {
                const uint32_t nb = bounded(x.v[e], dg);
                dest = dg <= 8 ? sh.to[q][nb] : __ldg(&d.csr_to[sh.loc[q] + nb]);
            }
            atomicAdd(&trans[dest], 1u);
        }
    }
    __syncwarp();  // the tables are reused for the warp's next pairs
}

// Items of the pass of one simulation: the event items first, then those of the series row.
__device__ __forceinline__ uint32_t foi_event_items(const Dev& d) { return (d.S * d.P + kFoiPairs - 1) / kFoiPairs; }

template <typename Wait>
__device__ __forceinline__ void foi_item(const Dev& d, uint32_t item, int collect_only, const StepAt& at, FoiWarpSmem& sh, Wait wait)
{
    const uint32_t ev = foi_event_items(d);
    if (item >= ev) foi_series(d, item - ev, collect_only, at, wait);
    else if (!collect_only) foi_events(d, kFoiPairs * item, at, sh, wait);
}

// Warp w of block b takes item b * W + w, then every gridDim.x * W further (W = blockDim.x / 32; W
// per-warp tables in dynamic shared memory).
__global__ void __launch_bounds__(512) k_foi(Dev d, int collect_only, uint32_t koff)
{
    extern __shared__ __align__(16) unsigned char foi_dyn[];
    const uint32_t warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    FoiWarpSmem& sh = reinterpret_cast<FoiWarpSmem*>(foi_dyn)[warp];
    const uint32_t items = foi_event_items(d) + d.S * series_chunks(d.P);
    griddep_launch_dependents();  // the infection kernel may be scheduled; it waits for this grid
    const StepAt at = load_step(d.ctrl, koff);
    for (uint32_t g = blockIdx.x * W + warp; g < items; g += gridDim.x * W) foi_item(d, g, collect_only, at, sh, GridWait{});
}

// ------------------------------------------------------------------ infection draws

// Infection of human i in step t, after the demographic pass of the step. `imm`, `born` and
// `dtime` are its immunity byte, birth and death times, loaded by the caller together with the
// winner key (its age is t + 1 - born); its next event time becomes its exposed-to-infectious
// step or its death.
__device__ __forceinline__ void infect_human(const Dev& d, uint32_t i, uint32_t s, const U4& r, uint32_t t,
                                             uint32_t imm, int32_t born, int32_t dtime)
{
    d.n_status[i] = 1;
    d.n_strain[i] = (uint8_t)s;
    d.n_imm[i] = (uint8_t)(imm | (1u << s));
    const int32_t age = (int32_t)t + 1 - born;
    const int32_t ex = (int32_t)resolve(__fadd_rn((float)age, d.nExposed), r.v[0]);
    d.n_exposed[i] = ex;
    d.n_recovery[i] = (int32_t)resolve(__fadd_rn((float)ex, d.recovery), r.v[1]);
    d.n_next[i] = human_next(1, dtime, born, ex);
}

// The same for mosquito slot i.
__device__ __forceinline__ void infect_mosquito(const Dev& d, uint32_t i, uint32_t s, uint32_t r, uint32_t t, int32_t born,
                                                int32_t dtime)
{
    d.m_stat[i] = 1;
    d.m_strain[i] = (uint8_t)s;
    const int32_t now = (int32_t)t + 1;
    const int32_t ex = (int32_t)resolve(__fadd_rn((float)(now - born), d.mExposed), r);
    d.m_exposed[i] = ex;
    d.m_code[i] = mosq_code(mosq_next(1, dtime, born, ex), now, true);
}

// Target of mosquito event e: the first alive slot of its attempt sequence (dead slots are
// retried, cpp/mepidemic.cu:206-235). Returns UINT_MAX when the attempts run out. The four
// candidates of one Philox call are loaded together (one memory round trip) and the first alive
// one in attempt order is taken; its status is left in *state (a live slot without kDeep is susceptible). `first` is the draw of the
// first four attempts (the caller computes it together with other lanes' draws); a0 (a multiple of
// four): the first attempt.
__device__ __forceinline__ uint32_t mosquito_target(const Dev& d, const Key& key, uint32_t pidx, uint32_t e,
                                                    uint32_t base, uint32_t size, uint32_t t, uint32_t* state,
                                                    const U4& first, uint32_t a0 = 0)
{
    for (uint32_t a = a0; a < d.maxTarget; a += 4) {
        const U4 r = a == 0 ? first : draw4(key, kInfMTarget, pidx, t, e, a >> 2);
        uint32_t slot[4], st[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) slot[q] = base + bounded(r.v[q], size);
#pragma unroll
        for (int q = 0; q < 4; ++q) st[q] = (a + q < d.maxTarget) ? __ldcg(&d.m_code[slot[q]]) : (uint32_t)kDead;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (!(st[q] & kDead)) {
                *state = (st[q] & kDeep) ? __ldcg(&d.m_stat[slot[q]]) & 3u : 0u;
                return slot[q];
            }
    }
    return UINT_MAX;
}

// Per-warp tables of the infection pass: one community and its events of every serotype
// flattened into one index space.
constexpr uint32_t kIntroScan = 1024;   // humans of a community up to which failed introductions look at all of them
constexpr uint32_t kFewEvents = 32;
// Items past which a block of a batch works off a community together. Infection phase of 64 uneven
// instances of a heavy epidemic (2.3e5 human infections a step) at 64, 128, 256 and 512: 369, 353, 340 and
// 415 us, of 16 smaller ones 32, 29, 33 and 41.
constexpr uint32_t kHeavyItems = 128;
constexpr uint32_t kHeavyList = 64;     // such communities that a block can list
constexpr uint32_t kTargetCache = 128;  // items whose targets Phase A keeps for Phase C

struct InfectWarpSmem {
    union {
        uint4 target[kTargetCache];     // per item: four human targets, or a mosquito slot in .x
        uint2 bid[kFewEvents];          // of few events the eligible ones: {target (mosquito slots with bit
                                        // 31), serotype position}
    };
    // First item of each serotype position and events by position, humans (groups of four) and
    // mosquitoes; positions past the last serotype start at UINT_MAX.
    uint4 hstart[2], mstart[2];
    uint32_t kh[ARBO_MAX_STRAINS], km[ARBO_MAX_STRAINS];
};
static_assert(ARBO_MAX_STRAINS == 8, "tables of eight serotype positions");

// Serotype position of item `rel` and its number within it, from a table of starts: the last position
// whose start is <= rel (positions without items share the next one's start).
__device__ __forceinline__ uint32_t item_position(const uint4* start, uint32_t rel, uint32_t* idx)
{
    const uint4 a = start[0], b = start[1];
    const uint32_t s[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t j = 0, at = 0;
#pragma unroll
    for (uint32_t k = 1; k < 8; ++k)
        if (s[k] <= rel) {
            j = k;
            at = s[k];
        }
    *idx = rel - at;
    return j;
}

__device__ __forceinline__ uint32_t wrap(uint32_t x, uint32_t n) { return x >= n ? x - n : x; }

// Infection draws of community c, by one warp. Lanes 0..S-1 read the community's event counts
// and draw its introduction counts, lanes 8 and 9 the first serotypes; the events (groups of
// four human events, single mosquito events) then form one index space walked by the 32 lanes:
// Up to 32 events, which is most communities in most steps, the warp resolves among its lanes, one event to
// a lane: every lane loads all that its event may need in one round trip, and the eligible events on a
// target are found by matching the lanes' targets; lanes are in serial order, so the lowest one holds it.
// The two round trips that the bids in memory cost are gone: infection pass of 5e4 agents 5.1 -> 3.6 us, of
// 7e6 9.1 -> 6.6. One item (four human events) to a lane, which covers more of them, took twice the
// registers: 64 leave twice the warps in flight in batches (phase of 512 instances of 7e4 agents 104 -> 90
// us, of 64 uneven ones 228 -> 200) and fit the clusters that share SMs, which had gone without (step of
// 128 such instances 63.4 -> 56.3 us at the peak, of 32 21.0 -> 19.8, of 8 16.9 -> 15.2).
// More items go through the targets' winner keys in memory, three phases:
//   A: every event whose target is eligible at the start of the pass bids its serial order
//      (serotype position j, event index) for the target with atomicMin; the targets of the first
//      kTargetCache items are kept in shared memory for phase C;
//   B: external introductions (cpp/nepidemic.cu:261-309) in serial order, 32 attempts at a time, then 128;
//   C: each event that won its target applies its infection.
// This reproduces the serial loops of nmTransmission / mnTransmission (cpp/mepidemic.cu:143-246,
// cpp/nepidemic.cu:146-319): a target is infected by the first eligible event in serial order.
// Every target of community c's events and introductions lies in c's own census range, so no
// other warp reads or writes them during the pass and warp barriers order the phases. One warp
// per community with no block barrier: the pass is a chain of dependent round trips per
// community, so the more communities in flight per SM the better.
//
// By: one warp alone; one warp that leaves a community of more than kHeavyItems items untouched and lists it
// (works it off itself when the list is full); or a whole block (every warp calls with the same community
// and the same tables).
// Communities that the warps of a block leave to the whole block: {instance, community}.
struct HeavyList {
    uint32_t n;
    uint2 at[kHeavyList];
};

enum InfectBy : int { kByWarp = 0, kByWarpDefer = 1, kByBlock = 2 };

template <int kBy, typename Wait>
__device__ __forceinline__ void infect_unit(const Dev& d, uint32_t c, const StepAt& at, InfectWarpSmem& sh, Wait wait,
                                            HeavyList* heavy = nullptr, uint32_t inst = 0)
{
    constexpr bool kFew = kBy != kByBlock;  // may find few events
    const uint32_t lane = threadIdx.x & 31u;
    const bool lead = kBy != kByBlock || threadIdx.x < 32;
    const uint32_t gl = kBy == kByBlock ? threadIdx.x : lane, gt = kBy == kByBlock ? blockDim.x : 32u;
    auto sync = [] {
        if (kBy == kByBlock) __syncthreads();
        else __syncwarp();
    };
    const uint32_t t = at.t;
    const uint32_t hiword = ~at.epoch;
    const Key key = at.key;
    const uint32_t S = d.S, P = d.P;
    const float ext = __fdiv_rn(d.extInf, (float)P);
    // Static loads and keyed draws first; the event counts and alive mosquitoes written by the
    // previous kernels are read after the programmatic-launch wait.
    const uint32_t ns = __ldg(&d.nsize[c]), ms = __ldg(&d.msize[c]);
    const uint32_t nbase = __ldg(&d.nloc[c]), mbase = __ldg(&d.mloc[c]);
    const uint32_t pl = lane * P + c;
    // One draw per lane in one pass: introduction counts (lanes < S), first serotypes (8, 9).
    const U4 rd = draw4(key, lane < S ? (uint32_t)kIntroCount : lane == 8 ? (uint32_t)kInfMStart : (uint32_t)kInfHStart,
                        lane < S ? pl : c, t);
    wait();
    const uint32_t mc = d.mcnt[c];
    uint32_t kh = lane < S ? d.transh[pl] : 0u;
    uint32_t km = lane < S ? d.transm[pl] : 0u;
    const bool had_h = kh != 0, had_m = km != 0;
    uint32_t sv = 0, ne = 0;
    if (lane < S) {
        if (ns == 0) kh = 0;
        else ne = (uint32_t)resolve(ext, rd.v[0]);
        if (mc == 0) km = 0;
        if (kh >= kMaxEventsPerPair || km >= kMaxEventsPerPair) {
            atomicOr(&d.ctrl->err, ARBO_DEVERR_EVENT_OVERFLOW);
            kh = min(kh, kMaxEventsPerPair - 1);
            km = min(km, kMaxEventsPerPair - 1);
        }
    } else if (lane == 8) {
        if (mc) sv = bounded(rd.v[0], S);
    } else if (lane == 9) {
        if (ns) sv = bounded(rd.v[0], S);
    }
    const uint32_t s0m = __shfl_sync(kFull, sv, 8), s0h = __shfl_sync(kFull, sv, 9);
    // Lane j: serotype position j (the j-th serotype from the first of each species).
    const uint32_t hs = wrap(s0h + (lane & 7u), S), ms_ = wrap(s0m + (lane & 7u), S);
    uint32_t khj = __shfl_sync(kFull, kh, hs), kmj = __shfl_sync(kFull, km, ms_), nej = __shfl_sync(kFull, ne, hs);
    if (lane >= S) khj = kmj = nej = 0;
    uint32_t hi = (khj + 3) >> 2, mi = kmj, he = khj;  // groups of human events, mosquito events, human events
    const uint32_t h0 = hi, m0 = mi;
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, hi, off), x = __shfl_up_sync(kFull, mi, off);
        const uint32_t z = kFew ? __shfl_up_sync(kFull, he, off) : 0u;
        if (lane >= (uint32_t)off) {
            hi += y;
            mi += x;
            he += z;
        }
    }
    const uint32_t H = __shfl_sync(kFull, hi, 7), Mt = __shfl_sync(kFull, mi, 7);
    const uint32_t items = H + Mt, Hev = kFew ? __shfl_sync(kFull, he, 7) : 0u;
    const bool few = kFew && Hev + Mt <= kFewEvents;
    if (kBy == kByWarpDefer && items > kHeavyItems) {
        uint32_t i = 0;
        if (lane == 0) {
            i = atomicAdd(&heavy->n, 1u);
            if (i < kHeavyList) heavy->at[i] = make_uint2(inst, c);
        }
        if (__shfl_sync(kFull, i, 0) < kHeavyList) return;
    }
    if (kBy == kByBlock) __syncthreads();  // every warp has read the event counts
    if (lead && had_h) d.transh[pl] = 0;
    if (lead && had_m) d.transm[pl] = 0;
    if (lead && lane < 8) {
        reinterpret_cast<uint32_t*>(sh.hstart)[lane] = lane < S ? (few ? he - khj : hi - h0) : UINT_MAX;
        reinterpret_cast<uint32_t*>(sh.mstart)[lane] = lane < S ? mi - m0 : UINT_MAX;
        sh.kh[lane] = khj;
        sh.km[lane] = kmj;
    }
    const unsigned intro = __ballot_sync(kFull, nej != 0);  // positions with introductions
    sync();
    if (items == 0 && !intro) return;
    // The first introduction's first 32 attempts load everything but the bids together with the events'
    // targets: nothing before them changes it.
    uint32_t ii = 0, iim = 0, ist = 1;
    int32_t ibn = 0, idt = 0;
    if (lead && intro && lane < d.maxIntro) {
        const uint32_t ph = wrap(s0h + __ffs(intro) - 1, S) * P + c;
        const U4 r = draw4(key, kIntroTarget, ph, t, lane >> 2);
        ii = nbase + bounded(pick4(r, lane & 3u), ns);
        iim = __ldcg(&d.n_imm[ii]);
        ist = __ldcg(&d.n_status[ii]);
        ibn = __ldcg(&d.n_born[ii]);
        idt = __ldcg(&d.n_dtime[ii]);
    }

    // External introductions, position by position: open_to(i, j, a) says whether no event before attempt a
    // of position j holds human i, took(i, a, j) notes that the attempt has taken i.
    auto introductions = [&](auto open_to, auto took) {
        uint32_t avail = 0xFFu;  // bit s clear: no human of the community can take serotype s
        bool scanned = false;
        for (unsigned left_pos = intro; left_pos; left_pos &= left_pos - 1) {
            const uint32_t j = __ffs(left_pos) - 1, s = wrap(s0h + j, S), ph = s * P + c;
            uint32_t left = __shfl_sync(kFull, nej, j);
            uint32_t a0 = (avail >> s) & 1u ? 0u : d.maxIntro;
            // The first 32 attempts one per lane (most introductions find someone there), later ones
            // 128 at a time, four to a lane and to a Philox call.
            for (uint32_t per = 1; left > 0 && a0 < d.maxIntro; per = 4) {
                uint32_t i[4], im[4], elig = 0;
                int32_t bn = 0, dt = 0;  // times of the lane's one attempt
                const uint32_t av = a0 + per * lane;  // a0 is a multiple of four
                if (per == 1) {
                    i[1] = i[2] = i[3] = im[1] = im[2] = im[3] = 0;
                    if (left_pos != intro) {
                        const U4 r = draw4(key, kIntroTarget, ph, t, av >> 2);
                        ii = nbase + bounded(pick4(r, av & 3u), ns);
                        if (av < d.maxIntro) {
                            iim = __ldcg(&d.n_imm[ii]);
                            ist = __ldcg(&d.n_status[ii]);
                            ibn = __ldcg(&d.n_born[ii]);
                            idt = __ldcg(&d.n_dtime[ii]);
                        }
                    }
                    i[0] = ii, im[0] = iim, bn = ibn, dt = idt;
                    if (av < d.maxIntro && ist == 0 && !((iim >> s) & 1u) &&
                        open_to(ii, j, av))
                        elig = 1;
                } else {
                    const U4 r = draw4(key, kIntroTarget, ph, t, av >> 2);
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) {
                        i[q] = im[q] = 0;
                        if (av + q < d.maxIntro) {
                            i[q] = nbase + bounded(r.v[q], ns);
                            im[q] = __ldcg(&d.n_imm[i[q]]);
                            if (__ldcg(&d.n_status[i[q]]) == 0 && !((im[q] >> s) & 1u) &&
                                open_to(i[q], j, av + q))
                                elig |= 1u << q;
                        }
                    }
                }
                // The eligible attempts in order; a human taken by one is lost to the later ones.
                while (left > 0) {
                    const unsigned bal = __ballot_sync(kFull, elig != 0);
                    if (!bal) break;
                    const uint32_t first = __ffs(bal) - 1;
                    uint32_t q = elig ? __ffs(elig) - 1 : 0;
                    const uint32_t iq = q == 0 ? i[0] : q == 1 ? i[1] : q == 2 ? i[2] : i[3];
                    const uint32_t mq = q == 0 ? im[0] : q == 1 ? im[1] : q == 2 ? im[2] : im[3];
                    const uint32_t taken = __shfl_sync(kFull, iq, first);
                    took(taken, __shfl_sync(kFull, av + q, first), j);
                    if (lane == first) {
                        if (per != 1) {
                            bn = __ldcg(&d.n_born[iq]);
                            dt = __ldcg(&d.n_dtime[iq]);
                        }
                        infect_human(d, iq, s, draw4(key, kIntroExposed, ph, t, av + q), t, mq, bn, dt);
                    }
#pragma unroll
                    for (q = 0; q < 4; ++q)
                        if (i[q] == taken) elig &= ~(1u << q);
                    left -= 1;
                }
                __syncwarp();
                a0 += 32 * per;
                if (left > 0 && !scanned && ns <= kIntroScan) {
                    // Is there anyone left to infect? In a small population the attempts would else run
                    // to their limit (1,000) in every community that is immune, 32 a round trip: once a small
                    // population was immune its step took 42 us (2,000 humans) and 27 us (10,000), now 18
                    // and 19; 512 instances of 1e4 humans 300 -> 255 us.
                    scanned = true;
                    uint32_t open = 0;
                    for (uint32_t h = lane; h < ns; h += 32)
                        if (__ldcg(&d.n_status[nbase + h]) == 0) open |= ~(uint32_t)__ldcg(&d.n_imm[nbase + h]);
                    avail = __reduce_or_sync(kFull, open & 0xFFu);
                }
                if (!((avail >> s) & 1u)) break;
            }
            if (left > 0 && lane == 0) atomicAdd(&d.ctrl->diag[1], 1u);
        }
    };
    if (few) {
        // One event per lane.
        const bool act = lane < Hev + Mt, hum = lane < Hev;
        uint32_t idx = 0, sp = 0, pp = 0, tg = 0, j = 0, im = 0;
        int32_t bn = 0, dt = 0;
        bool elig = false;
        U4 rx;  // exposed-age draw
        if (act) {
            j = item_position(hum ? sh.hstart : sh.mstart, hum ? lane : lane - Hev, &idx);
            sp = wrap((hum ? s0h : s0m) + j, S);
            pp = sp * P + c;
            const U4 r = draw4(key, hum ? (uint32_t)kInfHTarget : (uint32_t)kInfMTarget, pp, t, hum ? idx >> 2 : idx);
            // Both kinds of event load alike, so that they wait together: a human's status, immunity, birth
            // and death time, a mosquito slot's code, status, birth and death time; of the slots of a
            // mosquito event's further attempts, which few events get to, the codes.
            const uint32_t base = hum ? nbase : mbase, size = hum ? ns : ms;
            tg = base + bounded(hum ? pick4(r, idx & 3u) : r.v[0], size);
            const uint32_t step = hum ? 1u : sizeof(Life) / 4;
            uint32_t st[4] = {kDead, kDead, kDead, kDead};
            if (hum || d.maxTarget) st[0] = (hum ? d.n_status : d.m_code)[tg];
            im = (hum ? d.n_imm : d.m_stat)[tg];
            bn = (hum ? d.n_born : &d.m_life->born)[(size_t)tg * step];
            dt = (hum ? d.n_dtime : &d.m_life->dtime)[(size_t)tg * step];
#pragma unroll
            for (uint32_t q = 1; q < 4; ++q)
                if (!hum && q < d.maxTarget) st[q] = d.m_code[mbase + bounded(r.v[q], ms)];
            rx = draw4(key, hum ? (uint32_t)kInfHExposed : (uint32_t)kInfMExposed, pp, t, hum ? idx : idx >> 2);
            if (hum) {
                elig = st[0] == 0 && !((im >> sp) & 1u);
            } else {
                uint32_t state = im & 3u;
                if (st[0] & kDead) {
                    tg = UINT_MAX;
#pragma unroll
                    for (int q = 3; q >= 1; --q)
                        if (!(st[q] & kDead)) tg = mbase + bounded(r.v[q], ms);
                    if (tg == UINT_MAX) tg = mosquito_target(d, key, pp, idx, mbase, ms, t, &state, r, 4);
                    if (tg == UINT_MAX) {
                        atomicAdd(&d.ctrl->diag[0], 1u);
                    } else {
                        state = d.m_stat[tg] & 3u;
                        bn = d.m_life[tg].born;
                        dt = d.m_life[tg].dtime;
                    }
                }
                elig = tg != UINT_MAX && state == 0;
                tg |= 0x80000000u;
            }
        }
        // Lanes are in serial order within a species, so of the eligible events on a target the lowest lane
        // holds it.
        const unsigned open_events = __ballot_sync(kFull, elig);
        const unsigned same = __match_any_sync(kFull, tg) & open_events;
        bool won = elig && __ffs(same) - 1 == (int)lane;
        if (intro) {
            const uint32_t nb = __popc(open_events);
            if (elig) sh.bid[__popc(open_events & ((1u << lane) - 1u))] = make_uint2(tg, j);
            __syncwarp();
            introductions(
                [&](uint32_t i, uint32_t jj, uint32_t) {
                    bool open = true;  // no event of this position or an earlier one is on i
                    for (uint32_t b = 0; b < nb; ++b) open &= sh.bid[b].x != i || sh.bid[b].y > jj;
                    return open;
                },
                [&](uint32_t i, uint32_t, uint32_t) { won = won && tg != i; });
        }
        if (won) {
            if (hum) infect_human(d, tg, sp, rx, t, im, bn, dt);
            else infect_mosquito(d, tg & 0x7FFFFFFFu, sp, pick4(rx, idx & 3u), t, bn, dt);
        }
        __syncwarp();  // the warp's tables are reused for its next community
        return;
    }
    // Phase A. Human groups and mosquito events draw their targets in one pass (the first four
    // attempts of a mosquito event).
    for (uint32_t it = gl; it < items; it += gt) {
        const bool hum = it < H;
        const uint32_t rel = hum ? it : it - H;
        uint32_t idx;
        const uint32_t j = item_position(hum ? sh.hstart : sh.mstart, rel, &idx);
        const uint32_t sp = wrap((hum ? s0h : s0m) + j, S), pp = sp * P + c;
        const U4 r = draw4(key, hum ? (uint32_t)kInfHTarget : (uint32_t)kInfMTarget, pp, t, idx);
        if (hum) {
            const uint32_t s = sp, k = sh.kh[j];
            uint32_t tg[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) tg[q] = nbase + bounded(r.v[q], ns);
            if (it < kTargetCache) sh.target[it] = make_uint4(tg[0], tg[1], tg[2], tg[3]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t e = 4 * idx + q;
                if (e >= k) break;
                const uint32_t st = d.n_status[tg[q]], im = d.n_imm[tg[q]];
                if (st == 0 && !((im >> s) & 1u)) atomicMin(&d.winh[tg[q]], order_key(hiword, j, 0, e));
            }
        } else {
            uint32_t st = 0;
            const uint32_t slot = mosquito_target(d, key, pp, idx, mbase, ms, t, &st, r);
            if (it < kTargetCache) sh.target[it].x = slot;
            if (slot == UINT_MAX) atomicAdd(&d.ctrl->diag[0], 1u);
            else if (st == 0) atomicMin(&d.winm[slot], order_key(hiword, j, 0, idx));
        }
    }
    sync();
    // Phase B
    if (intro && lead) {
        introductions([&](uint32_t i, uint32_t j, uint32_t a) { return __ldcg(&d.winh[i]) > order_key(hiword, j, 1, a); },
                      [&](uint32_t i, uint32_t a, uint32_t j) {
                          if (lane == 0) d.winh[i] = order_key(hiword, j, 1, a);
                      });
        __syncwarp();
    }
    if (kBy == kByBlock && intro) __syncthreads();
    // Phase C
    for (uint32_t it = gl; it < items; it += gt) {
        if (it < H) {
            uint32_t idx;
            const uint32_t j = item_position(sh.hstart, it, &idx);
            const uint32_t s = wrap(s0h + j, S), ph = s * P + c, k = sh.kh[j];
            uint32_t tg[4];
            if (it < kTargetCache) {
                const uint4 v = sh.target[it];
                tg[0] = v.x;
                tg[1] = v.y;
                tg[2] = v.z;
                tg[3] = v.w;
            } else {
                const U4 r = draw4(key, kInfHTarget, ph, t, idx);
#pragma unroll
                for (int q = 0; q < 4; ++q) tg[q] = nbase + bounded(r.v[q], ns);
            }
            // Winner keys and the inputs of the infection in one round trip: only the winner of a
            // target writes it, so the values read here are the ones the infection needs.
            unsigned long long wk[4];
            uint32_t im[4];
            int32_t bn[4], dt[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                wk[q] = 0;
                im[q] = 0;
                bn[q] = dt[q] = 0;
                if (4 * idx + q < k) {
                    wk[q] = __ldcg(&d.winh[tg[q]]);
                    im[q] = __ldcg(&d.n_imm[tg[q]]);
                    bn[q] = __ldcg(&d.n_born[tg[q]]);
                    dt[q] = __ldcg(&d.n_dtime[tg[q]]);
                }
            }
            // The group's winning events, then one pass per winner of the lane (the warp runs as
            // many passes as its busiest lane has winners, not one per event position).
            uint32_t won = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (4 * idx + q < k && wk[q] == order_key(hiword, j, 0, 4 * idx + q)) won |= 1u << q;
            while (won) {
                const uint32_t q = __ffs(won) - 1;
                won &= won - 1;
                const uint32_t e = 4 * idx + q;
                const uint32_t tq = q == 0 ? tg[0] : q == 1 ? tg[1] : q == 2 ? tg[2] : tg[3];
                const uint32_t iq = q == 0 ? im[0] : q == 1 ? im[1] : q == 2 ? im[2] : im[3];
                const int32_t bq = q == 0 ? bn[0] : q == 1 ? bn[1] : q == 2 ? bn[2] : bn[3];
                const int32_t dq = q == 0 ? dt[0] : q == 1 ? dt[1] : q == 2 ? dt[2] : dt[3];
                infect_human(d, tq, s, draw4(key, kInfHExposed, ph, t, e), t, iq, bq, dq);
            }
        } else {
            uint32_t idx;
            const uint32_t rel = it - H, j = item_position(sh.mstart, rel, &idx);
            const uint32_t sm = wrap(s0m + j, S), pm = sm * P + c;
            uint32_t st = 0;
            const uint32_t slot = it < kTargetCache
                                      ? sh.target[it].x
                                      : mosquito_target(d, key, pm, idx, mbase, ms, t, &st, draw4(key, kInfMTarget, pm, t, idx));
            unsigned long long wk = 0;
            int2 life = make_int2(0, 0);
            if (slot != UINT_MAX) {  // winner key and times in one round trip
                wk = __ldcg(&d.winm[slot]);
                life = __ldcg(reinterpret_cast<const int2*>(d.m_life + slot));
            }
            const U4 r = draw4(key, kInfMExposed, pm, t, idx >> 2);  // while they are on their way
            if (slot != UINT_MAX && wk == order_key(hiword, j, 0, idx))
                infect_mosquito(d, slot, sm, pick4(r, idx & 3u), t, life.x, life.y);
        }
    }
    sync();  // the tables are reused for the next community
}

// One warp per community: warp w of block b takes communities b*K + w (per-warp tables in dynamic shared
// memory).
__device__ __forceinline__ void infect_communities(const Dev& d, uint32_t koff)
{
    extern __shared__ __align__(16) unsigned char infect_dyn[];
    const uint32_t warp = threadIdx.x >> 5, K = blockDim.x >> 5;
    InfectWarpSmem& sh = reinterpret_cast<InfectWarpSmem*>(infect_dyn)[warp];
    const StepAt at = load_step(d.ctrl, koff);
    for (uint32_t c = blockIdx.x * K + warp; c < d.P; c += gridDim.x * K)
        infect_unit<kByWarp>(d, c, at, sh, GridWaitRelease{});
}

// Few communities to an SM: the shortest chain per warp (116 registers). Many: 80 registers, so that more
// warps are in flight and the next kernels' blocks find room beside them. Step with the first and the
// second: 100 communities 10.2 and 10.35 us, 400 10.8 and 10.9, 900 11.65 and 11.4, 2,500 18.65 and 18.6,
// 3,969 38.4 and 37.7.
__global__ void __launch_bounds__(512) k_infect(Dev d, uint32_t koff) { infect_communities(d, koff); }
__global__ void __maxnreg__(80) k_infect_many(Dev d, uint32_t koff) { infect_communities(d, koff); }

// ------------------------------------------------------------------ batched steps

// Instance owning flattened block b: the largest i with off[i] <= b.
__device__ __forceinline__ uint32_t batch_instance(const uint32_t* __restrict__ off, uint32_t n, uint32_t b)
{
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(&off[mid]) <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Warp runs over the concatenated items of a batch's instances (off[i] = first item of instance
// i): warps take runs of `run` consecutive items, strided over the grid, so that a warp restages
// its instance descriptor (per-warp copy in shared memory, wdev) about once per run while every
// instance is spread over many warps; fn(dev, item within the instance, instance) runs each item.
// kAcross: consecutive runs go to different blocks.
template <bool kAcross, typename Fn>
__device__ __forceinline__ void batch_warp_items(const BatchDev& bd, const uint32_t* __restrict__ off, uint32_t run,
                                                 unsigned long long* wdev, Fn fn)
{
    const uint32_t lane = threadIdx.x & 31u, W = blockDim.x >> 5;
    const Dev& d = *reinterpret_cast<const Dev*>(wdev);
    const uint32_t total = __ldg(&off[bd.n]);
    const uint32_t runs = (total + run - 1) / run;
    const uint32_t w = threadIdx.x >> 5, gw = kAcross ? w * gridDim.x + blockIdx.x : blockIdx.x * W + w;
    const uint32_t nw = gridDim.x * W;
    uint32_t inst = UINT_MAX, lo = 0, hi = 0;  // current instance and its item range
    for (uint32_t r = gw; r < runs; r += nw) {
        const uint32_t end = min(total, (r + 1) * run);
        for (uint32_t it = r * run; it < end; ++it) {
            if (inst == UINT_MAX || it < lo || it >= hi) {
                inst = batch_instance(off, bd.n, it);
                lo = __ldg(&off[inst]);
                hi = __ldg(&off[inst + 1]);
                __syncwarp();  // every lane is done with the previous descriptor
                const unsigned long long* src = reinterpret_cast<const unsigned long long*>(bd.devs + inst);
                for (uint32_t i = lane; i < sizeof(Dev) / 8; i += 32) wdev[i] = src[i];
                __syncwarp();
            }
            fn(d, it - lo, inst);
        }
    }
}

// Demographic pass of a batch. Work items are per warp: 32*U-lane groups of humans or one
// mosquito quad, instance by instance (bd.demog_off counts warp items, bd.demog_h the human items
// of each instance). Warps take runs of bd.demog_chunk consecutive items from a device counter
// (reset by the force-of-infection kernel once this kernel has finished), single items once fewer
// than bd.demog_tail are left, so uneven instances balance across the GPU, and each warp keeps a
// private copy of its current instance's descriptor in shared memory: no block-wide barrier
// anywhere.
template <int U>
__global__ void __launch_bounds__(256, 5) k_demog_batch(BatchDev bd, uint32_t koff)
{
    __shared__ QuadSmem wsm[8];
    __shared__ __align__(16) unsigned long long wdev[8][sizeof(Dev) / 8];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const Dev& d = *reinterpret_cast<const Dev*>(wdev[warp]);
    const uint32_t total = __ldg(&bd.demog_off[bd.n]);
    uint32_t inst = UINT_MAX, lo = 0, hi = 0;  // current instance and its item range
    uint32_t chunk = bd.demog_chunk;
    for (;;) {
        uint32_t it0 = 0;
        if (lane == 0) it0 = atomicAdd(bd.work, chunk);
        it0 = __shfl_sync(kFull, it0, 0);
        if (it0 >= total) break;
        const uint32_t end = min(it0 + chunk, total);
        if (total - end < bd.demog_tail) chunk = 1u;
        for (uint32_t it = it0; it < end; ++it) {
            if (inst == UINT_MAX || it >= hi) {
                // Items arrive in increasing order: usually the next instance, else search.
                const bool next = inst != UINT_MAX && inst + 2 <= bd.n && it < __ldg(&bd.demog_off[inst + 2]);
                inst = next ? inst + 1 : batch_instance(bd.demog_off, bd.n, it);
                lo = __ldg(&bd.demog_off[inst]);
                hi = __ldg(&bd.demog_off[inst + 1]);
                __syncwarp();
                const unsigned long long* src = reinterpret_cast<const unsigned long long*>(bd.devs + inst);
                for (uint32_t i = lane; i < sizeof(Dev) / 8; i += 32) wdev[warp][i] = src[i];
                __syncwarp();
            }
            const uint32_t local = it - lo, hw = __ldg(&bd.demog_h[inst]);
            const uint32_t t = d.ctrl->t + koff;
            const Key key = load_key(d.ctrl);
            if (local < hw) demog_humans<U>(d, key, local * 32 * U + lane, 32, t, wsm[warp]);
            else demog_mosquito_quad(d, key, local - hw, lane, t, wsm[warp], NoWait{});
        }
    }
    griddep_launch_dependents();
}

// Force-of-infection pass of a batch: one warp per item of an instance (foi_item; bd.foi_off counts them), in runs of bd.foi_run items per warp. With
// collect_only, only series row 0 of every instance (the end of its initialisation).
__global__ void __launch_bounds__(512) k_foi_batch(BatchDev bd, int collect_only, uint32_t koff)
{
    extern __shared__ __align__(16) unsigned char foi_dyn[];
    const uint32_t warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    FoiWarpSmem& sh = reinterpret_cast<FoiWarpSmem*>(foi_dyn)[warp];
    unsigned long long* wdev =
        reinterpret_cast<unsigned long long*>(foi_dyn + W * sizeof(FoiWarpSmem)) + warp * (sizeof(Dev) / 8);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        griddep_wait();  // the demographic kernel has finished taking items
        *bd.work = 0u;
    }
    griddep_launch_dependents();  // the infection kernel may be scheduled; it waits for this grid
    batch_warp_items<false>(bd, bd.foi_off, bd.foi_run, wdev, [&](const Dev& d, uint32_t item, uint32_t) {
        foi_item(d, item, collect_only, load_step(d.ctrl, koff), sh, GridWait{});
    });
}

// Infection pass of a batch: one warp per community over the concatenated communities of all
// instances (bd.infect_off counts communities), in runs of bd.infect_run communities per warp. kHeavy: the
// block then works off together those with more than kHeavyItems items, of which a warp alone takes 32 in
// some 4 us, and neighbouring runs, mostly of one instance with many events or with few, go to different
// blocks. 64 uneven instances (1.9e8 agents) in the steps of a heavy epidemic: phase 631 -> 202, 896 -> 270
// and 775 -> 288 us; with few events 79 -> 85, and 24 such instances 38 -> 41.
// 80 registers; phase of 512 instances of 7e4 agents and of 24 uneven ones at 64, 72, 80 and 96: 90, 82, 79
// and 84 us, 40, 37, 35 and 39.
template <bool kHeavy>
__global__ void __maxnreg__(80) k_infect_batch(BatchDev bd, uint32_t koff)
{
    extern __shared__ __align__(16) unsigned char infect_dyn[];
    const uint32_t warp = threadIdx.x >> 5, K = blockDim.x >> 5;
    InfectWarpSmem* tables = reinterpret_cast<InfectWarpSmem*>(infect_dyn);
    unsigned long long* descs = reinterpret_cast<unsigned long long*>(infect_dyn + K * sizeof(InfectWarpSmem));
    unsigned long long* wdev = descs + warp * (sizeof(Dev) / 8);
    if constexpr (!kHeavy) {
        batch_warp_items<false>(bd, bd.infect_off, bd.infect_run, wdev, [&](const Dev& d, uint32_t c, uint32_t) {
            infect_unit<kByWarp>(d, c, load_step(d.ctrl, koff), tables[warp], GridWaitRelease{});
        });
    } else {
        __shared__ HeavyList heavy;
        if (threadIdx.x == 0) heavy.n = 0;
        __syncthreads();
        batch_warp_items<true>(bd, bd.infect_off, bd.infect_run, wdev, [&](const Dev& d, uint32_t c, uint32_t inst) {
            const StepAt at = load_step(d.ctrl, koff);
            infect_unit<kByWarpDefer>(d, c, at, tables[warp], GridWaitRelease{}, &heavy, inst);
        });
        __syncthreads();
        const uint32_t n = min(heavy.n, kHeavyList);
        for (uint32_t i = 0; i < n; ++i) {
            const uint2 h = heavy.at[i];
            const unsigned long long* src = reinterpret_cast<const unsigned long long*>(bd.devs + h.x);
            for (uint32_t j = threadIdx.x; j < sizeof(Dev) / 8; j += blockDim.x) descs[j] = src[j];
            __syncthreads();
            const Dev& d = *reinterpret_cast<const Dev*>(descs);
            infect_unit<kByBlock>(d, h.y, load_step(d.ctrl, koff), tables[0], NoWait{});
        }
    }
}

static_assert(16 * (sizeof(InfectWarpSmem) + sizeof(Dev)) <= 48 * 1024 && 16 * (sizeof(FoiWarpSmem) + sizeof(Dev)) <= 48 * 1024,
              "per-warp tables of a 512-thread block must fit the default dynamic shared memory");

// Dynamic shared memory of the infection kernels for blocks of `threads` threads.
size_t infect_smem(uint32_t threads, bool batch)
{
    return (size_t)(threads / 32) * (sizeof(InfectWarpSmem) + (batch ? sizeof(Dev) : 0));
}

// Dynamic shared memory of the force-of-infection kernels for blocks of `threads` threads.
size_t foi_smem(uint32_t threads, bool batch)
{
    return (size_t)(threads / 32) * (sizeof(FoiWarpSmem) + (batch ? sizeof(Dev) : 0));
}

// ------------------------------------------------------------------ many steps of small simulations

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

constexpr uint32_t kStepsWarps = 16;  // warps per CTA of k_steps
union __align__(16) StepsScratch {  // a warp works on one phase at a time
    QuadSmem demog;
    FoiWarpSmem foi;
    InfectWarpSmem infect;
};
constexpr uint32_t kStepsSmem = kStepsWarps * (uint32_t)sizeof(StepsScratch);
static_assert(kStepsSmem + sizeof(Dev) + 64 <= 48 * 1024, "shared memory of k_steps");

// Many steps of a batch of few small simulations in one launch: one thread-block cluster of C CTAs per
// simulation runs `nsteps` whole steps, its phases separated by cluster barriers. Simulations need
// nothing from one another, so each cluster goes on by itself; the per-phase batch kernels wait for the
// slowest simulation at each phase and hand out items through one counter, which with few items is all
// latency: 32 simulations of 7e4 agents took 39 us a step, now 17, 8 of them 35 and 14. The bodies are
// the per-phase kernels' own. Sixteen warps to a CTA and B CTAs to an SM (64 registers at two).
//
// Two forms. With few demographic items to a warp (kMany false) they go in a fixed order, and each phase's
// first item does what does not depend on the phase before (draws, constant tables) before it waits for
// that phase: 8 simulations of 7e4 agents 17.4 -> 16.8 us a step, 32 of them 21.5 -> 21.0. With many (items
// are of uneven cost) a CTA's warps take its share of them from a counter: 128 of them 65.4 -> 62.8 us,
// later 38.2 -> 36.1; half an item to a warp by the counter took 18.4 for 17.8. Both together, in one
// kernel of 64 registers, took 64.5 and 37.5 on 128. At 64 registers the infection body spills: 104 bytes a
// thread in the first form, 64 in the second; at 128 (CTAs with an SM each) nothing.
template <uint32_t B, bool kMany>
__global__ void __launch_bounds__(kStepsWarps * 32, B) k_steps(const Dev* devs, uint32_t C, uint32_t nsteps)
{
    extern __shared__ __align__(16) unsigned char steps_dyn[];
    __shared__ __align__(16) unsigned long long dev_copy[sizeof(Dev) / 8];
    __shared__ uint32_t next[2];  // items taken, by parity of the step
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x < 2) next[threadIdx.x] = 0;
    {
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(devs + blockIdx.x / C);
        for (uint32_t i = threadIdx.x; i < sizeof(Dev) / 8; i += blockDim.x) dev_copy[i] = src[i];
    }
    __syncthreads();
    const Dev& d = *reinterpret_cast<const Dev*>(dev_copy);
    StepsScratch& scratch = reinterpret_cast<StepsScratch*>(steps_dyn)[warp];
    // Neighbouring warps of the cluster's order sit on different SMs.
    const uint32_t rank = cluster_rank(), w = warp * C + rank, nw = kStepsWarps * C;
    StepAt at = load_step(d.ctrl, 0);
    const uint32_t quads = (d.tiles + kQuad - 1) / kQuad, hw = (d.nvec + 31) / 32;
    const uint32_t foi = foi_event_items(d) + d.S * series_chunks(d.P);
    for (uint32_t k = 0; k < nsteps; ++k, ++at.t, ++at.epoch) {
        auto human = [&](uint32_t it) { demog_humans<1>(d, at.key, (it - quads) * 32 + lane, 32, at.t, scratch.demog); };
        if constexpr (kMany) {
            auto take = [&] {
                uint32_t i = 0;
                if (lane == 0) i = atomicAdd(&next[k & 1u], 1u);
                return __shfl_sync(kFull, i, 0) * C + rank;
            };
            for (uint32_t it = take(); it < quads + hw; it = take()) {
                if (it < quads) demog_mosquito_quad(d, at.key, it, lane, at.t, scratch.demog, NoWait{});
                else human(it);
            }
            cluster_barrier();
            if (threadIdx.x == 0) next[(k + 1) & 1u] = 0;
            for (uint32_t g = w; g < foi; g += nw) foi_item(d, g, 0, at, scratch.foi, NoWait{});
            cluster_barrier();
            for (uint32_t c = w; c < d.P; c += nw) infect_unit<kByWarp>(d, c, at, scratch.infect, NoWait{});
            cluster_barrier();
        } else {
            bool pending = k > 0;
            const PendingWait later{pending};
            auto end_phase = [&] {
                later();  // a warp without items has not waited for the phase before
                cluster_arrive();
                pending = true;
            };
            for (uint32_t it = w; it < quads + hw; it += nw) {
                if (it < quads) {
                    demog_mosquito_quad(d, at.key, it, lane, at.t, scratch.demog, later);
                } else {
                    later();
                    human(it);
                }
            }
            end_phase();
            for (uint32_t g = w; g < foi; g += nw) foi_item(d, g, 0, at, scratch.foi, later);
            end_phase();
            for (uint32_t c = w; c < d.P; c += nw) infect_unit<kByWarp>(d, c, at, scratch.infect, later);
            end_phase();
        }
    }
    if (!kMany && nsteps) cluster_wait();
    if (rank == 0 && threadIdx.x == 0) {
        d.ctrl->t = at.t;
        d.ctrl->epoch = at.epoch;
    }
}

__global__ void k_advance_batch(BatchDev bd, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < bd.n) {
        Ctrl* c = bd.devs[i].ctrl;
        c->t += n;
        c->epoch += n;
    }
}

// ------------------------------------------------------------------ initialisation

// nDemographicInitialization (cpp/demographicintial.cu:86-180), one thread per human slot.
__device__ __forceinline__ void init_human(const Dev& d, const Key& key, uint32_t j)
{
    if (j >= d.N) {
        d.n_status[j] = kPad;
        d.n_born[j] = 0;
        d.n_dtime[j] = INT_MAX;
        d.n_next[j] = INT_MAX;
        d.n_ple[j] = 0.0f;
        d.n_strain[j] = 0;
        d.n_imm[j] = 0;
        d.n_exposed[j] = 0;
        d.n_recovery[j] = 0;
        return;
    }
    const U4 r0 = draw4(key, kInitHuman, j, 0, 0);
    const U4 r1 = draw4(key, kInitHuman, j, 0, 1);
    const U4 r2 = draw4(key, kInitHuman, j, 0, 2);
    const uint32_t dr[12] = {r0.v[0], r0.v[1], r0.v[2], r0.v[3], r1.v[0], r1.v[1],
                             r1.v[2], r1.v[3], r2.v[0], r2.v[1], r2.v[2], r2.v[3]};
    const float randCSF = __fmul_rn(__ldg(&d.survh[d.yh]), u01(dr[0]));
    const uint32_t y = lower_bound_f(d.survh, d.yh + 1, randCSF);
    const int32_t age = (int32_t)(365u * y + bounded(dr[1], 365u));
    const float base = cdf_at(d.cdfh, d.ah, age != 0 ? age - 1 : 0);
    const float ple = __fadd_rn(__fmul_rn(__fsub_rn(1.0f, base), u01(dr[2])), base);
    uint32_t imm = 0;
    for (uint32_t s = 0; s < d.S; ++s)
        if (u01(dr[3 + s]) < d.seroPrev) imm |= 1u << s;
    const int32_t dt = death_time(-age, death_age_inv(d.cdfh, d.minvh, d.ah, ple, 65536.0f));
    d.n_born[j] = -age;  // age `age` at time 0
    d.n_ple[j] = ple;
    d.n_dtime[j] = dt;
    d.n_next[j] = dt;
    d.n_status[j] = 0;
    d.n_strain[j] = 0;
    d.n_imm[j] = (uint8_t)imm;
    d.n_exposed[j] = 0;
    d.n_recovery[j] = 0;
}

__global__ void k_init_humans(Dev d)
{
    const Key key = load_key(d.ctrl);
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < d.nvec * 4) init_human(d, key, j);
}

// mDemographicInitialization (cpp/demographicintial.cu:183-297): one warp per 128-slot tile;
// the tile's dead count starts the carried count of the recruitment quota.
__device__ __forceinline__ void init_mosquito_tile(const Dev& d, const Key& key, uint32_t b, uint32_t lane)
{
    const float alive_p = __fdiv_rn(__ldg(&d.etab[0]), (float)d.M);
    const uint32_t c0 = __ldg(&d.tcomm[b]) & ~kTileSpans;
    uint32_t codes = 0;
    uint32_t ndead = 0, ndead0 = 0;  // dead slots of the tile; of them, in the tile's first community
    for (int k = 0; k < 4; ++k) {
        const uint32_t i = 4 * (b * 32 + lane) + k;
        d.m_stat[i] = 0;
        d.m_strain[i] = 0;
        d.m_exposed[i] = 0;
        Life life{0, INT_MIN, 0.0f, 0};  // padding, or never alive: age 0, death age 0
        uint32_t code = kPad;
        if (i < d.M) {
            const U4 r = draw4(key, kInitMosquito, i, 0);
            if (!(u01(r.v[0]) < alive_p)) {
                code = kDead;
                ndead += 1;
                const uint32_t cc = slot_comm(d, c0, i);
                if (cc == c0) ndead0 += 1;
                else atomicSub(&d.mcnt[cc], 1u);
            } else {
                const float randCSF = __fmul_rn(__ldg(&d.survm[d.dm]), u01(r.v[1]));
                const uint32_t a = lower_bound_f(d.survm, d.dm + 1, randCSF);
                const float base = cdf_at(d.cdfm, d.am, a != 0 ? (int32_t)a - 1 : 0);
                life.ple = __fadd_rn(__fmul_rn(__fsub_rn(1.0f, base), u01(r.v[2])), base);
                life.born = -(int32_t)a;
                life.dtime = death_time(-(int32_t)a, death_age_lut(d, life.ple));
                code = mosq_code(life.dtime, 0, false);
            }
        }
        codes |= code << (8 * k);
        d.m_life[i] = life;
    }
    reinterpret_cast<uint32_t*>(d.m_code)[b * 32 + lane] = codes;
    // One atomic per tile for its first community (a community's alive count would otherwise
    // take one same-address atomic per dead slot).
    const uint32_t tile_dead = __reduce_add_sync(kFull, ndead);
    const uint32_t dead0 = __reduce_add_sync(kFull, ndead0);
    if (lane == 0) {
        d.ledger[b] = (int32_t)tile_dead;
        if (dead0) atomicSub(&d.mcnt[c0], dead0);
    }
}

__global__ void k_init_mosquitoes(Dev d)
{
    const Key key = load_key(d.ctrl);
    const uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b < d.tiles) init_mosquito_tile(d, key, b, threadIdx.x & 31u);  // warp-uniform
}

// nEpidemicInitial / mEpidemicInitial (cpp/epidemicinitial.cu:27-99): the seeded agents are
// elements 0..k-1 of a keyed bijection of the census. Thread 0 also resets the step control.
__device__ __forceinline__ void seed_one(const Dev& d, const Key& key, uint32_t j)
{
    if (j == 0) {
        d.ctrl->t = 0;
        d.ctrl->err = 0;
        d.ctrl->done = 0;
        d.ctrl->epoch += 1;
        for (int q = 0; q < 4; ++q) d.ctrl->diag[q] = 0;
    }
    if (j < d.nInit) {
        const uint32_t i = seed_perm(key, 0, d.N, j);
        const U4 r = draw4(key, kSeedHuman, j, 0);
        const uint32_t s = bounded(r.v[0], d.S);
        d.n_status[i] = 2;
        d.n_strain[i] = (uint8_t)s;
        d.n_imm[i] = (uint8_t)(d.n_imm[i] | (1u << s));
        const uint32_t rr = (uint32_t)resolve(d.recovery, r.v[2]);
        const uint32_t m = rr > 1u ? rr - 1u : 1u;
        const int32_t dur = (int32_t)(bounded(r.v[1], m) + 1u);
        const int32_t born = d.n_born[i];
        const int32_t rec = (d.quirks & ARBO_QUIRK_SEED_RECOVERY_DURATION) ? dur : dur - born;  // age + dur
        d.n_recovery[i] = rec;
        d.n_next[i] = human_next(2, d.n_dtime[i], born, rec);
        atomicAdd(&d.infh[s * d.P + comm_of(d.nloc, d.P, i)], 1u);
    }
    if (j < d.mInit) {
        const uint32_t i = seed_perm(key, 1, d.M, j);
        const uint8_t code = d.m_code[i];
        if ((code & kDead) && !(d.quirks & ARBO_QUIRK_SEED_DEAD_MOSQUITO)) return;
        const U4 r = draw4(key, kSeedMosquito, j, 0);
        const uint32_t s = bounded(r.v[0], d.S);
        d.m_stat[i] = 2;
        d.m_code[i] = (code & kDead) ? (uint8_t)(kDead | kDeep) : mosq_code(d.m_life[i].dtime, 0, true);
        d.m_strain[i] = (uint8_t)s;
        atomicAdd(&d.infm[s * d.P + comm_of(d.mloc, d.P, i)], 1u);
    }
}

__global__ void k_seed(Dev d)
{
    const Key key = load_key(d.ctrl);
    seed_one(d, key, blockIdx.x * blockDim.x + threadIdx.x);
}

// ------------------------------------------------------------------ batched initialisation
//
// arbo_sim_init of every instance of a batch in five launches: the same per-agent bodies, with
// the blocks of all instances concatenated (off[i] = first block of instance i, every instance
// at least one block) and each block's instance descriptor staged in shared memory.

// Instance of block blockIdx.x and its first block; the descriptor copied into `buf` by the block.
__device__ __forceinline__ const Dev& stage_block_desc(const BatchDev& bd, const uint32_t* __restrict__ off,
                                                       uint32_t& inst, uint32_t& first, unsigned long long* buf)
{
    inst = batch_instance(off, bd.n, blockIdx.x);
    first = __ldg(&off[inst]);
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(bd.devs + inst);
    for (uint32_t i = threadIdx.x; i < sizeof(Dev) / 8; i += blockDim.x) buf[i] = src[i];
    __syncthreads();
    return *reinterpret_cast<const Dev*>(buf);
}

// The cudaMemsetAsync / cudaMemcpyAsync calls of arbo_sim_init: counters, event counts and
// series zeroed, each community's alive mosquito count restarted from its slot count. The blocks
// of one instance stride over its arrays.
__global__ void __launch_bounds__(256) k_reset_batch(BatchDev bd)
{
    __shared__ __align__(16) unsigned long long buf[sizeof(Dev) / 8];
    uint32_t inst, first;
    const Dev& d = stage_block_desc(bd, bd.init_off[3], inst, first, buf);
    const uint32_t nb = __ldg(&bd.init_off[3][inst + 1]) - first;
    const uint32_t i0 = (blockIdx.x - first) * blockDim.x + threadIdx.x, stride = nb * blockDim.x;
    const uint32_t SP = d.S * d.P, R = d.T + 1, RS = R * d.S;
    for (uint32_t i = i0; i < SP; i += stride) {
        d.infh[i] = 0u;
        d.infm[i] = 0u;
        d.inc[i] = 0u;
        d.transh[i] = 0u;
        d.transm[i] = 0u;
    }
    for (uint32_t i = i0; i < RS; i += stride) {
        d.s_ninc[i] = 0u;
        d.s_ninf[i] = 0u;
        d.s_one[i] = 0u;
        d.s_minf[i] = 0u;
    }
    for (uint32_t i = i0; i < R; i += stride) {
        d.s_ncount[i] = 0u;
        d.s_mcount[i] = 0u;
    }
    if (d.s_spatial)
        for (size_t i = i0; i < (size_t)R * SP; i += stride) d.s_spatial[i] = 0u;
    for (uint32_t i = i0; i < d.P; i += stride) d.mcnt[i] = d.msize[i];
}

__global__ void __launch_bounds__(256) k_init_humans_batch(BatchDev bd)
{
    __shared__ __align__(16) unsigned long long buf[sizeof(Dev) / 8];
    uint32_t inst, first;
    const Dev& d = stage_block_desc(bd, bd.init_off[0], inst, first, buf);
    const Key key = load_key(d.ctrl);
    const uint32_t j = (blockIdx.x - first) * blockDim.x + threadIdx.x;
    if (j < d.nvec * 4) init_human(d, key, j);
}

__global__ void __launch_bounds__(256) k_init_mosquitoes_batch(BatchDev bd)
{
    __shared__ __align__(16) unsigned long long buf[sizeof(Dev) / 8];
    uint32_t inst, first;
    const Dev& d = stage_block_desc(bd, bd.init_off[1], inst, first, buf);
    const Key key = load_key(d.ctrl);
    const uint32_t b = (blockIdx.x - first) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (b < d.tiles) init_mosquito_tile(d, key, b, threadIdx.x & 31u);  // warp-uniform
}

__global__ void __launch_bounds__(256) k_seed_batch(BatchDev bd)
{
    __shared__ __align__(16) unsigned long long buf[sizeof(Dev) / 8];
    uint32_t inst, first;
    const Dev& d = stage_block_desc(bd, bd.init_off[2], inst, first, buf);
    const Key key = load_key(d.ctrl);
    seed_one(d, key, (blockIdx.x - first) * blockDim.x + threadIdx.x);
}


// Reads a buffer larger than L2 so that the next kernel starts with a cold cache. The loads
// feed a comparison that never holds for the zero-filled buffer, so they cannot be elided.
__global__ void __launch_bounds__(256) k_l2_flush(const int4* __restrict__ buf, size_t n, uint32_t* sink)
{
    uint32_t acc = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int4 v = __ldcs(buf + i);
        acc ^= (uint32_t)(v.x ^ v.y ^ v.z ^ v.w);
    }
    if (acc == 0x9E3779B9u) *sink = acc;
}

// Advances the step counter and the winner epoch after `n` captured steps (steps inside a
// graph read ctrl->t plus their baked offset).
__global__ void k_advance(Dev d, uint32_t n)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        d.ctrl->t += n;
        d.ctrl->epoch += n;
    }
}

// Census export in the reference's types (arbo_sim_export_census): one thread per agent.
__global__ void k_export_humans(Dev d, arbo_census_export x)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N) return;
    const int32_t now = (int32_t)d.ctrl->t;
    if (x.n_age) x.n_age[i] = (uint16_t)(now - d.n_born[i]);
    if (x.n_exposed) x.n_exposed[i] = (uint16_t)d.n_exposed[i];
    if (x.n_recovery) x.n_recovery[i] = (uint16_t)d.n_recovery[i];
    if (x.n_infect_status) x.n_infect_status[i] = d.n_status[i];
    if (x.n_ple) x.n_ple[i] = d.n_ple[i];
    if (x.n_strain) x.n_strain[i] = d.n_strain[i];
    if (x.n_sub_population) x.n_sub_population[i] = human_comm(d.nloc, d.hcomm, d.P, i);
    if (x.n_sub_pop_index) x.n_sub_pop_index[i] = i;
    if (x.n_history) {
        const uint32_t imm = d.n_imm[i];
        for (uint32_t s = 0; s < d.S; ++s) x.n_history[(size_t)s * d.N + i] = ((imm >> s) & 1u) ? -2 : -1;
    }
}

__global__ void k_export_mosquitoes(Dev d, arbo_census_export x)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.M) return;
    const int32_t now = (int32_t)d.ctrl->t;
    const bool dead = (d.m_code[i] & kDead) != 0;
    const Life life = d.m_life[i];
    if (x.m_age) {
        // Alive: steps since birth; dead: the age it died at (0 for a slot dead since initialisation).
        const int32_t b = life.born, dt = life.dtime;
        int32_t a = now - b;
        if (dead) a = dt == INT_MIN ? 0 : max(dt, max(b, 0) + 1) - b;
        x.m_age[i] = (uint16_t)a;
    }
    if (x.m_dead) x.m_dead[i] = dead ? 1 : 0;
    if (x.m_exposed) x.m_exposed[i] = (uint16_t)d.m_exposed[i];
    if (x.m_infect_status) x.m_infect_status[i] = (uint8_t)(d.m_stat[i] & 3u);
    if (x.m_ple) x.m_ple[i] = life.ple;
    if (x.m_strain) x.m_strain[i] = d.m_strain[i];
    if (x.m_sub_population) x.m_sub_population[i] = mosq_comm(d, i);
    if (x.m_sub_pop_index) x.m_sub_pop_index[i] = i;
}

// Words of the life records to or from a dense array.
__global__ void k_life_words(Dev d, uint32_t first, uint32_t n, int word, int words, int32_t* array, int store)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int32_t* w = reinterpret_cast<int32_t*>(d.m_life + first + i) + word;
    int32_t* a = array + (size_t)i * words;
    for (int k = 0; k < words; ++k) {
        if (store) w[k] = a[k];
        else a[k] = w[k];
    }
}

// After a census write; with the arrays brought to the host and the codes made there, a write of 6e6 slots'
// status took 24.7 ms, now 0.08.
__global__ void k_refresh_codes(Dev d, int flags)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.M) return;
    const uint32_t code = d.m_code[i], st = d.m_stat[i] & 3u;
    const Life life = d.m_life[i];
    const bool dead = flags ? code != 0 : (code & kDead) != 0;
    d.m_stat[i] = (uint8_t)st;
    d.m_code[i] = dead ? (uint8_t)(kDead | (st ? kDeep : 0u))
                       : mosq_code(mosq_next(st, life.dtime, life.born, d.m_exposed[i]), (int32_t)d.ctrl->t, st != 0);
}

}  // namespace

int launch_life_words(const Dev& d, uint32_t first, uint32_t n, int word, int words, void* array, bool store, void* stream)
{
    k_life_words<<<cdiv(n, 256), 256, 0, (cudaStream_t)stream>>>(d, first, n, word, words, (int32_t*)array, store ? 1 : 0);
    return (int)cudaGetLastError();
}

int launch_refresh_codes(const Dev& d, bool flags, void* stream)
{
    k_refresh_codes<<<cdiv(d.M, 256), 256, 0, (cudaStream_t)stream>>>(d, flags ? 1 : 0);
    return (int)cudaGetLastError();
}

int launch_export(const Dev& d, const arbo_census_export& x, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (d.N) k_export_humans<<<cdiv(d.N, 256), 256, 0, st>>>(d, x);
    if (d.M) k_export_mosquitoes<<<cdiv(d.M, 256), 256, 0, st>>>(d, x);
    return (int)cudaGetLastError();
}

int launch_l2_flush(const void* buf, size_t bytes, uint32_t* sink, uint32_t num_sm, cudaStream_t st)
{
    k_l2_flush<<<4 * (num_sm ? num_sm : 152), 256, 0, st>>>((const int4*)buf, bytes / 16, sink);
    return (int)cudaGetLastError();
}

int demog_tma_blocks_per_sm(uint32_t unroll)
{
    int n = 0;
    cudaError_t e;
    if (unroll == 4) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_demog_tma<4>, 128, 0);
    else if (unroll == 2) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_demog_tma<2>, 128, 0);
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_demog_tma<1>, 128, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

int launch_demog(const Dev& d, const Launch& l, cudaStream_t st, uint32_t koff)
{
    const uint32_t U = l.demogUnroll;
    if (l.demogPipeline) {
        const uint32_t quads = cdiv(d.tiles, kQuad);
        const uint32_t hchunks = cdiv(d.nvec, 32 * U);
        const uint32_t need = cdiv(quads > hchunks ? quads : hchunks, 4);
        uint32_t grid = (l.numSM ? l.numSM : 152u) * (l.demogTmaBlocksPerSM ? l.demogTmaBlocksPerSM : 1u);
        if (grid > need) grid = need;
        if (U == 4) k_demog_tma<4><<<grid, 128, 0, st>>>(d, koff);
        else if (U == 2) k_demog_tma<2><<<grid, 128, 0, st>>>(d, koff);
        else k_demog_tma<1><<<grid, 128, 0, st>>>(d, koff);
        return (int)cudaGetLastError();
    }
    const uint32_t items = cdiv(d.tiles, kQuad) + cdiv(d.nvec, (uint64_t)32 * U), sms = l.numSM ? l.numSM : 152u;
    // With blocks of 8 warps and fewer than two of them per SM, the items are spread and the blocks made
    // smaller, down to 4 warps, so that no SM gets two full blocks while others have none: step of 7e5
    // agents 11.5 -> 10.8 us (and up to 13 when the early start placed the blocks badly), of 5e4 10.6 ->
    // 10.4. From there on larger blocks are better (128 threads: 18.6 -> 21.4 us at 7e6 agents), and a
    // grid of resident blocks striding over the items is not (20.5 us).
    uint32_t warps = l.demogBlock / 32;
    const bool spread = items <= 2 * warps * sms;
    if (spread && warps == 8) warps = std::min(8u, std::max(4u, cdiv(items, 2 * sms)));
    // Within a run of steps the previous kernel is the last step's infection pass, which leaves the step
    // control and the tables alone, so the pass may begin before it ends. At a run's
    // first step (koff 0) it may be the kernel that advances the step control.
    return launch_pdl(U == 4 ? k_demog<4> : U == 2 ? k_demog<2> : k_demog<1>, dim3(cdiv(items, warps)), dim3(32 * warps), 0,
                      st, l.pdl && koff > 0, d, spread ? 1u : 0u, koff);
}

uint32_t foi_items(uint32_t S, uint32_t P) { return cdiv((uint64_t)S * P, kFoiPairs) + S * cdiv(P, 256); }

int launch_foi(const Dev& d, const Launch& l, cudaStream_t st, int collect_only, uint32_t koff)
{
    return launch_pdl(k_foi, dim3(cdiv(foi_items(d.S, d.P), l.foiBlock / 32)), dim3(l.foiBlock), foi_smem(l.foiBlock, false), st,
                      l.pdl && !collect_only, d, collect_only, koff);
}

typedef void (*InfectKernel)(Dev, uint32_t);
static InfectKernel infect_kernel(uint32_t P, const Launch& l)
{
    return P >= 4 * (l.numSM ? l.numSM : 152u) ? k_infect_many : k_infect;
}

int launch_infect(const Dev& d, const Launch& l, cudaStream_t st, uint32_t koff)
{
    const uint32_t per = l.infectBlock / 32;
    uint32_t blocks = cdiv(d.P, per);
    const uint32_t cap = 16u * (l.numSM ? l.numSM : 152u);
    if (blocks > cap) blocks = cap;
    return launch_pdl(infect_kernel(d.P, l), dim3(blocks), dim3(l.infectBlock), infect_smem(l.infectBlock, false), st,
                      l.pdl != 0, d, koff);
}

int launch_init(const Dev& d, const Launch& l, void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    k_init_humans<<<cdiv((uint64_t)d.nvec * 4, 256), 256, 0, st>>>(d);
    k_init_mosquitoes<<<cdiv((uint64_t)d.tiles * 32, 256), 256, 0, st>>>(d);
    const uint32_t nseed = d.nInit > d.mInit ? d.nInit : d.mInit;
    k_seed<<<cdiv(nseed ? nseed : 1, 256), 256, 0, st>>>(d);
    int e = (int)cudaGetLastError();
    if (e) return e;
    return launch_foi(d, l, st, 1, 0);
}

int launch_step(const Dev& d, const Launch& l, void* stream, void* events, uint32_t koff)
{
    cudaStream_t st = (cudaStream_t)stream;
    cudaEvent_t* ev = (cudaEvent_t*)events;
    int e;
    if (ev) cudaEventRecord(ev[0], st);
    if ((e = launch_demog(d, l, st, koff))) return e;
    if (ev) cudaEventRecord(ev[1], st);
    if ((e = launch_foi(d, l, st, 0, koff))) return e;
    if (ev) cudaEventRecord(ev[2], st);
    if ((e = launch_infect(d, l, st, koff))) return e;
    if (ev) cudaEventRecord(ev[3], st);
    return 0;
}

int launch_advance(const Dev& d, uint32_t n, void* stream)
{
    k_advance<<<1, 32, 0, (cudaStream_t)stream>>>(d, n);
    return (int)cudaGetLastError();
}

int share_carveout()
{
    const int pct = 44;  // 100 KB of 228: five blocks of the demographic kernel, and 128 KB of L1
    const void* f[] = {(const void*)k_demog<1>, (const void*)k_demog<2>, (const void*)k_demog<4>, (const void*)k_foi,
                       (const void*)k_infect, (const void*)k_infect_many};
    for (const void* k : f) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

uint32_t launches_per_step() { return 3; }

int preload_step_kernels(const Launch& l)
{
    cudaFuncAttributes a;
    cudaError_t e;
    if (l.demogPipeline)
        e = l.demogUnroll == 4   ? cudaFuncGetAttributes(&a, k_demog_tma<4>)
            : l.demogUnroll == 2 ? cudaFuncGetAttributes(&a, k_demog_tma<2>)
                                 : cudaFuncGetAttributes(&a, k_demog_tma<1>);
    else
        e = l.demogUnroll == 4   ? cudaFuncGetAttributes(&a, k_demog<4>)
            : l.demogUnroll == 2 ? cudaFuncGetAttributes(&a, k_demog<2>)
                                 : cudaFuncGetAttributes(&a, k_demog<1>);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_foi);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_infect);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_infect_many);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k_advance);
    return (int)e;
}

int batch_blocks_per_sm(const Launch& l, uint32_t out[3])
{
    int n = 0;
    cudaError_t e;
    if (l.demogUnroll == 4) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_demog_batch<4>, (int)l.demogBlock, 0);
    else if (l.demogUnroll == 2) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_demog_batch<2>, (int)l.demogBlock, 0);
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_demog_batch<1>, (int)l.demogBlock, 0);
    if (e != cudaSuccess) return (int)e;
    out[0] = n > 0 ? (uint32_t)n : 1u;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_foi_batch, (int)l.foiBlock, foi_smem(l.foiBlock, true))) !=
        cudaSuccess)
        return (int)e;
    out[1] = n > 0 ? (uint32_t)n : 1u;
    const auto infect = l.infectHeavy ? k_infect_batch<true> : k_infect_batch<false>;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, infect, (int)l.infectBlock,
                                                            infect_smem(l.infectBlock, true))) != cudaSuccess)
        return (int)e;
    out[2] = n > 0 ? (uint32_t)n : 1u;
    return 0;
}

int launch_step_batch(const BatchDev& bd, const Launch& l, void* stream, void* events, uint32_t koff)
{
    cudaStream_t st = (cudaStream_t)stream;
    cudaEvent_t* ev = (cudaEvent_t*)events;
    int e;
    if (ev) cudaEventRecord(ev[0], st);
    const dim3 gd(bd.grid_demog), bdm(l.demogBlock);
    if (l.demogUnroll == 4) k_demog_batch<4><<<gd, bdm, 0, st>>>(bd, koff);
    else if (l.demogUnroll == 2) k_demog_batch<2><<<gd, bdm, 0, st>>>(bd, koff);
    else k_demog_batch<1><<<gd, bdm, 0, st>>>(bd, koff);
    if ((e = (int)cudaGetLastError())) return e;
    if (ev) cudaEventRecord(ev[1], st);
    if ((e = launch_pdl(k_foi_batch, dim3(bd.grid_foi), dim3(l.foiBlock), foi_smem(l.foiBlock, true), st, l.pdl != 0, bd,
                        0, koff)))
        return e;
    if (ev) cudaEventRecord(ev[2], st);
    if ((e = launch_pdl(l.infectHeavy ? k_infect_batch<true> : k_infect_batch<false>, dim3(bd.grid_infect),
                        dim3(l.infectBlock), infect_smem(l.infectBlock, true), st, l.pdl != 0, bd, koff)))
        return e;
    if (ev) cudaEventRecord(ev[3], st);
    return 0;
}

int launch_init_batch(const BatchDev& bd, const Launch& l, void* stream, const uint32_t blocks[4])
{
    cudaStream_t st = (cudaStream_t)stream;
    k_reset_batch<<<blocks[3], 256, 0, st>>>(bd);
    k_init_humans_batch<<<blocks[0], 256, 0, st>>>(bd);
    k_init_mosquitoes_batch<<<blocks[1], 256, 0, st>>>(bd);
    k_seed_batch<<<blocks[2], 256, 0, st>>>(bd);
    const int e = (int)cudaGetLastError();
    if (e) return e;
    // Series row 0 of every instance (the collect-only pass of arbo_sim_init).
    return launch_pdl(k_foi_batch, dim3(bd.grid_foi), dim3(l.foiBlock), foi_smem(l.foiBlock, true), st, false, bd, 1,
                      0u);
}

// Launch configuration of k_steps with clusters of C CTAs (attr: one attribute, kept by the caller).
static cudaLaunchConfig_t steps_config(uint32_t n, uint32_t C, cudaLaunchAttribute* attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n * C);
    cfg.blockDim = dim3(kStepsWarps * 32);
    cfg.dynamicSmemBytes = kStepsSmem;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = C;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

typedef void (*StepsKernel)(const Dev*, uint32_t, uint32_t);

// Largest cluster of which n fit the device at once with kernel k and have `ctas` CTAs at most (0: none).
static uint32_t largest_cluster(StepsKernel k, uint32_t n, uint64_t ctas)
{
    // Sixteen CTAs per cluster are more than the portable eight.
    const bool wide = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    uint32_t found = 0;
    for (uint32_t C = wide ? 16 : 8; C >= 1 && !found; C /= 2) {
        if ((uint64_t)n * C > ctas) continue;
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = steps_config(1, C, &attr);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, k, &cfg) == cudaSuccess && fit > 0 && (uint32_t)fit >= n) found = C;
    }
    (void)cudaGetLastError();
    return found;
}

// CTAs that have an SM each keep 128 registers a thread; two to an SM have 64.
static StepsKernel steps_kernel(uint32_t per_sm, bool many)
{
    if (many) return per_sm == 1 ? k_steps<1, true> : k_steps<2, true>;
    return per_sm == 1 ? k_steps<1, false> : k_steps<2, false>;
}

uint32_t steps_cluster(uint32_t n, uint32_t num_sm, uint32_t* per_sm)
{
    // The larger of the two forms, so that either fits (each sets its own attribute).
    const uint64_t sms = num_sm;
    const uint32_t one = std::min(largest_cluster(k_steps<1, false>, n, sms), largest_cluster(k_steps<1, true>, n, sms));
    const uint32_t two =
        std::min(largest_cluster(k_steps<2, false>, n, 2 * sms), largest_cluster(k_steps<2, true>, n, 2 * sms));
    *per_sm = one && one >= two ? 1u : 2u;
    return one && one >= two ? one : two;
}

int launch_steps(const Dev* devs, uint32_t n, uint32_t C, uint32_t per_sm, uint64_t items, uint32_t nsteps,
                 void* stream)
{
    const bool many = items >= 4ull * n * C * kStepsWarps;

    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = steps_config(n, C, &attr);
    cfg.stream = (cudaStream_t)stream;
    return (int)cudaLaunchKernelEx(&cfg, steps_kernel(per_sm, many), devs, C, nsteps);
}

int launch_advance_batch(const BatchDev& bd, uint32_t n, void* stream)
{
    k_advance_batch<<<cdiv(bd.n, 128), 128, 0, (cudaStream_t)stream>>>(bd, n);
    return (int)cudaGetLastError();
}

}  // namespace arbo
