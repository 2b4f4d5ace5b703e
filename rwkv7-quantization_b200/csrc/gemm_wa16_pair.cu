// Weight-only projections of many tokens (W4A16 group 128, W8A16 per tensor) on CTA PAIRS: tcgen05.mma.cta_group::2 with the
// widened weights in tensor memory, 256 weight rows x NB tokens a tile.  The arithmetic is gemm_wa16.cu's (weights widened to
// fp16 integers, scales in fp32 outside the tensor core), which keeps the prompts of fewer tokens.
//
// Why pairs.  The single-CTA form (128 rows x up to 128 tokens) spends a step of 512 tensor-core clocks on 40 KB (INT4) or 48 KB
// (INT8) from L2, more than an SM takes in meanwhile, on widening 128 x 128 weights, which its four warps manage in about as
// long, and on 128 tokens x 128 rows of fp32 work in the epilogue; measured it took 1400 clocks.  In a pair each CTA widens its own
// 128 weight rows once for all NB tokens and loads half of the tokens: the same bytes and half the widening per MMA.
//
// Zero points.  out = sum over groups of scale * (codes . x) + zero * sum(x).  The second part is a product of its own, [rows, groups] x
// [groups, tokens] in fp32: taken with FMAs it costs the epilogue as much as the scales do, and the group sums, the same for
// all 32 lanes, come through 128-byte-per-clock shared-memory loads at 16 bytes of use per warp (a third of the step).  So it is done
// by the tensor core too, after the last group: both fp32 factors are cut into three bf16 parts of 8 mantissa bits each (exact from
// 2^-110 up: below, what lies under bf16's 2^-133 is lost), and all products but zl xl, which is below 2^-30 of the whole, are
// eight k of an MMA, 16 groups a step.  (The parts are cut, not rounded, so zm xl and zl xm each reach 2^-22.)  An infinity or NaN has no
// parts: it is multiplied once, as the highest one.
//
// Centred codes.  The two parts cancel where the activations have a mean, and they are added one after the other, so what either
// loses is lost at its own size, and the tensor core cuts towards zero, always to the same side: with codes 0 to 15 and activations of
// mean 3 the error of [4096, 16384] against 64 bits was 7.75e-4, of which 6.62e-4 are the rounding to fp16.  So a code goes in as code -
// 7.5 (2 * code - 15, an exact fp16 integer) and its zero point as zero + 7.5 * scale, the middle of the group's range: 6.62e-4, as
// with fp32 sums that add both parts group by group.  It costs the widening warps 64 fp16 FMAs a step: 15 ns with 256 tokens, 67 with 128,
// where they are what a step waits for.  Without zeros (zero = -8 * scale) the codes are centred at 8 and there is no second part.
//
// A step is 128 k of one tile; its tokens are units of UN columns with an accumulator each, so that the epilogue adds one unit's
// group while the tensor core works on others.  What limits a step is less the work (the MMAs of 256 tokens take 1024 clocks) than
// the roles' own instruction streams and the signals between them: an arrival at the other CTA that orders memory costs 0.4 us
// (1.92 us a step), a branch around each arrival instead of a predicate 0.13, two units of 128 columns from one issuing warp
// instead of four of 64 from two 0.07, an epilogue at 200 registers that crowds the widening warps 0.1.  Tensor memory: 256
// columns of accumulators, then kA slots of 64 columns of widened weights; more accumulators and fewer slots change nothing.
//
// Measured in a graph, us with the activations' kernel, single CTAs -> pairs.  INT4: [4096, 4096] 200 / 1000 / 2048 rows 21.4 -> 18.6, 56.2 ->
// 35.3, 106.8 -> 63.1; [16384, 4096] 53.4 -> 33.2, 177.9 -> 118.5, 356.3 -> 218.1; [4096, 16384] 56.0 -> 38.1, 198.6 -> 122.4, 381.9 -> 248.6.
// INT8: [4096, 4096] 1000 / 2048 rows 33.7 -> 26.3, 62.5 -> 48.0; [4096, 16384] 122.9 -> 93.1, 259.8 -> 201.6.
//
// Roles per CTA (512 threads): warps 0-3 widen (lane quarter = warp), 12 TMA producer, 13 (which owns tensor memory) and 14 MMA
// issuers in the leader CTA, each with every other unit of a step, 4-7 and 8-11 the epilogue of warp 13's and warp 14's units.
// wfull[] (this CTA's weights) is local; xfull[] (both CTAs' tokens), aready[] (both CTAs' widened weights) and dempty[] live in
// the leader; empty[] and dfull[] are signalled in both CTAs by a multicast commit.  A slot of widened weights is free when the
// step kA before it has left the tensor core, which is that step's empty[].  Every wait is bounded; the producers wait for the last
// commits and the pair meets before its tensor memory goes.
#include <algorithm>
#include <cstdlib>

#include "tc_pair.cuh"
#include "wa16.cuh"

namespace rwkvq {

constexpr int kP16Threads = 512;
constexpr int kP16MaxStages = 8;

struct P16Maps {
    CUtensorMap w, x, z;
};
struct P16Args {
    const float* scales;      // INT4: [N, groups]; INT8: [1]
    const float* zeros;       // INT4: [N, groups] or null (zero = -8 * scale)
    __half* out;
    float* part;              // slices > 1: fp32 partial sums [slices][M][N]
    int64_t ldo;
    int M, N, ksteps, groups;
    int mtiles, ntiles, slices;
    int* status;
    unsigned long long wait_ns;
};
struct P16Shared {
    uint64_t wfull[kP16MaxStages], xfull[kP16MaxStages], empty[kP16MaxStages], aready[kP16MaxStages], dfull[4], dempty[4];
    uint32_t tmem_base;
    int abort_flag;
};

template <int FMT, int NB>
struct P16Tile {
    static constexpr bool kGroup = FMT == W16_INT4_GROUP;
    static constexpr int kUN = kGroup ? 64 : 128;                        // tokens of a unit
    static constexpr int kU = NB / kUN / 2;                              // units of a step for each issuing warp
    static constexpr uint32_t kWBytes = 128u * (kGroup ? kW16K / 2 : kW16K);
    static constexpr uint32_t kXSlab = (uint32_t)NB / 2 * 128u;          // 64 k of this CTA's tokens
    static constexpr uint32_t kXBytes = 2 * kXSlab;
    static constexpr uint32_t kStage = kWBytes + kXBytes;
    static constexpr int kS = (int)((kW16SmemBudget - 1024) / kStage) < kP16MaxStages ? (int)((kW16SmemBudget - 1024) / kStage) : kP16MaxStages;
    static constexpr int kD = 256 / kUN;                                 // accumulators, half of them for each issuing warp
    static constexpr uint32_t kACol = 256;
    static constexpr int kA = 4;                                         // slots of widened weights
    static constexpr size_t kSmem = 1024 + (size_t)kS * kStage;
    static_assert(NB % (2 * kUN) == 0 && kU >= 1 && kA <= kS && (kU <= kD / 2 || kGroup), "tile");
};
// the epilogue keeps up to 128 sums a thread and 64 loaded values; widening and issuing warps give their registers to it:
// 80 + 2 * 192 + 48 = 4 * 128, the launch's own total
constexpr int kP16RegsLaunch = 128;

__device__ __forceinline__ void p16_abort(P16Shared& s, const P16Args& a) {
    s.abort_flag = 1;
    if (a.status) atomicExch(a.status, RWKVQ_E_TIMEOUT);
}
// D[tmem of both CTAs] (+)= A[tmem of both] * B[smem of both], 16-bit operands, fp32 accumulator
__device__ __forceinline__ void tc_mma_f16_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with the accumulator multiplied by 2^-4 before the sum
__device__ __forceinline__ void tc_mma_f16_ts_pair_d16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p, 4;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc) : "memory");
}

template <int FMT, int NB>
__global__ void __launch_bounds__(kP16Threads, 1) gemm_wa16_pair_kernel(const __grid_constant__ P16Maps maps, const P16Args a) {
    using TL = P16Tile<FMT, NB>;
    constexpr bool kGroup = TL::kGroup;
    constexpr int UN = TL::kUN;
    extern __shared__ uint8_t smem_raw[];
    __shared__ P16Shared s;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = warp_uniform((int)(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();          // 0 = leader of the pair
    const int pair = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);

    griddep_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < TL::kS; ++i) {
            mbar_init(&s.wfull[i], 1);
            mbar_init(&s.xfull[i], 1);                // the leader's expect_tx arrival; both CTAs' bytes
            mbar_init(&s.empty[i], 2);                // a multicast commit of each issuing warp
        }
        for (int i = 0; i < TL::kA; ++i) mbar_init(&s.aready[i], 8);      // four widening warps of each CTA
        for (int i = 0; i < TL::kD; ++i) {
            mbar_init(&s.dfull[i], 1);
            mbar_init(&s.dempty[i], 8);               // four epilogue warps of each CTA
        }
        s.abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
        prefetch_tmap(&maps.w);
        prefetch_tmap(&maps.x);
        if (kGroup) prefetch_tmap(&maps.z);
    }
    if (warp == 13) tmem_alloc_pair(&s.tmem_base, 512);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();                               // the peer's barriers exist before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = warp_uniform(s.tmem_base);
    const volatile int* abort_flag = &s.abort_flag;
    const int items = a.mtiles * a.ntiles * a.slices;
    // item -> (token tile, tile of 256 weight rows, K range); token tiles fastest, so the pairs at work share weight tiles
    // through L2.  K slices start at multiples of 4 steps (16-byte vectors of scales, whole MMAs of zero points).
    struct Item { int mt, nt, sl, k0, k1, nz; };      // nz: steps of zero points after the groups
    auto item_of = [&](int t) {
        Item it;
        it.mt = t % a.mtiles;
        const int r = t / a.mtiles;
        it.nt = r % a.ntiles;
        it.sl = r / a.ntiles;
        const int q4 = (a.ksteps + 3) >> 2;
        it.k0 = (int)((uint32_t)(q4 * it.sl) / (uint32_t)a.slices) * 4;             // below 2^21 * 16
        it.k1 = min((int)((uint32_t)(q4 * (it.sl + 1)) / (uint32_t)a.slices) * 4, a.ksteps);
        it.nz = kGroup && a.zeros ? (it.k1 - it.k0 + 15) >> 4 : 0;
        return it;
    };

    if (warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        if (warp == 12) {
            // ============================== TMA producer (both CTAs) ==============================
            const bool issuer = elect_one();
            constexpr int kWRow = kGroup ? kW16K / 2 : kW16K;
            // weights of a step; a step of zero points has none, its barrier just goes on with the ring
            auto fetch_w = [&](const Item& it, int k, int st) {
                if (!issuer) return;
                if (k < it.k1) {
                    mbar_expect_tx(&s.wfull[st], TL::kWBytes);
                    tma_load_2d(ring + (size_t)st * TL::kStage, &maps.w, k * kWRow, it.nt * 256 + (int)rank * 128, &s.wfull[st]);
                } else {
                    mbar_arrive(&s.wfull[st]);
                }
            };
            // first pass over the ring: weights never depend on the kernels in front, so they are requested before the
            // dependency wait of programmatic dependent launch
            int npre = 0;
            for (int t = pair; t < items && npre < TL::kS; t += npairs) {
                const Item it = item_of(t);
                for (int k = it.k0; k < it.k1 + it.nz && npre < TL::kS; ++k, ++npre) fetch_w(it, k, npre);
            }
            griddep_wait();
            bool ok = true;
            RingPos rp;
            for (int t = pair; t < items && ok; t += npairs) {
                const Item it = item_of(t);
                const int y0 = it.mt * NB + (int)rank * (NB / 2);
                for (int k = it.k0; k < it.k1 + it.nz; ++k, rp.next(TL::kS)) {
                    const int st = rp.i;
                    const bool refill = --npre < 0;
                    if (refill && !mbar_wait(&s.empty[st], rp.phase ^ 1, abort_flag, a.wait_ns)) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { p16_abort(s, a); break; }
                    if (refill) fetch_w(it, k, st);
                    if (issuer) {
                        const uint32_t leader_bar = smem_u32(&s.xfull[st]) & 0xFEFFFFFFu;        // the barrier of the even CTA
                        if (rank == 0) mbar_expect_tx(&s.xfull[st], 2 * TL::kXBytes);
                        uint8_t* dst = ring + (size_t)st * TL::kStage + TL::kWBytes;
                        const bool zstep = kGroup && k >= it.k1;
                        const CUtensorMap* m = zstep ? &maps.z : &maps.x;
                        const int x0 = zstep ? (it.k0 + 16 * (k - it.k1)) * (2 * kW16ZSlots) : k * 256;
                        tma_load_2d_pair(dst, m, x0, y0, leader_bar);
                        tma_load_2d_pair(dst + TL::kXSlab, m, x0 + 128, y0, leader_bar);
                    }
                }
            }
            if (ok && !(ok = pair_drain_ring(s.empty, rp, TL::kS, abort_flag, a.wait_ns))) p16_abort(s, a);
            if (!ok) {   // give copies already in flight a bounded time to land before the CTA's memory is released
                const unsigned long long t0 = global_ns();
                while (global_ns() - t0 < 2000000ull) {}
            }
        } else if (warp < 15 && rank == 0) {
            // ============================== MMA issuers (leader CTA) ==============================
            const bool issuer = elect_one();
            const int j = warp - 13;
            const uint32_t idesc = (1u << 4) | ((uint32_t)(UN >> 3) << 17) | (16u << 24);     // f32 += f16 * f16, both K-major, M = 256
            const uint32_t idesc_z = idesc | (1u << 7) | (1u << 10);                          // bf16 operands
            const uint32_t ring_addr = warp_uniform(smem_u32(ring));
            RingPos rp, ap, fp;                  // ring stage, widened weights, accumulator
            bool ok = true;
            for (int t = pair; t < items && ok; t += npairs) {
                const Item it = item_of(t);
                for (int k = it.k0; k < it.k1 + it.nz && ok; ++k, rp.next(TL::kS), ap.next(TL::kA)) {
                    const int st = rp.i;
                    const bool zstep = kGroup && k >= it.k1, fresh = kGroup || k == it.k0, last = kGroup || k == it.k1 - 1;
                    ok = mbar_wait(&s.xfull[st], rp.phase, abort_flag, a.wait_ns) && mbar_wait(&s.aready[ap.i], ap.phase, abort_flag, a.wait_ns);
                    const uint32_t at = tmem_base + TL::kACol + (uint32_t)ap.i * 64;
                    const uint64_t b = umma_desc_sw128(ring_addr + (uint32_t)st * TL::kStage + TL::kWBytes);
                    // the zero points of two groups are one MMA
                    const int zmma = kGroup ? (min(16, it.k1 - it.k0 - 16 * (k - it.k1)) + 1) >> 1 : 0;
                    RingPos f = fp;
#pragma unroll 1
                    for (int i = 0; i < TL::kU; ++i) {
                        const int buf = 2 * f.i + j;
                        if (fresh) ok = ok && mbar_wait(&s.dempty[buf], f.phase ^ 1, abort_flag, a.wait_ns);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) { p16_abort(s, a); break; }
                        tc_fence_after_sync();
                        const uint32_t d = tmem_base + (uint32_t)(buf * UN);
                        const uint64_t b0 = b + (uint64_t)(((2 * i + j) * (UN / 2) * 128) >> 4), b1 = b0 + (uint64_t)(TL::kXSlab >> 4);
                        if (issuer) {
                            if (zstep) {
                                for (int n = 0; n < zmma; ++n)
                                    tc_mma_f16_ts_pair(d, at + n * 8, (n < 4 ? b0 : b1) + (uint64_t)((n & 3) * 2), idesc_z, n ? 1u : 0u);
                            } else {
#pragma unroll
                                for (int n = 0; n < kW16K / 16; ++n) {
                                    const int c = kGroup ? (n < 4 ? 2 * n : 2 * n - 7) : n;          // INT4: the odd k (c even) first
                                    const uint64_t bc = (c < 4 ? b0 : b1) + (uint64_t)((c & 3) * 2);
                                    if (kGroup && n == 4) tc_mma_f16_ts_pair_d16(d, at + c * 8, bc, idesc);
                                    else tc_mma_f16_ts_pair(d, at + c * 8, bc, idesc, (fresh && n == 0) ? 0u : 1u);
                                }
                            }
                            if (last) tc_commit_pair(&s.dfull[buf]);
                            if (i == TL::kU - 1) tc_commit_pair(&s.empty[st]);      // both CTAs: this warp's MMAs have read the stage and the widened weights
                        }
                        f.next(TL::kD / 2);
                    }
                    if (last) fp = f;
                }
            }
        }
    } else if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        // ============================== weights: packed -> 16 bits in tensor memory ==============================
        const uint32_t lane_addr = tmem_base + TL::kACol + ((uint32_t)(warp * 32) << 16);
        const int row = warp * 32 + lane;
        const uint32_t centre = a.zeros ? 15 : 16;
        const uint32_t leader_aready = mapa_u32(smem_u32(&s.aready[0]), 0);
        const bool vec = (a.groups & 3) == 0;    // host: scales and zeros are 16-byte aligned
        RingPos rp, ap, freed;                   // freed: the step whose MMAs read this slot last
        int slots = TL::kA;
        bool ok = true;
        for (int t = pair; t < items && ok; t += npairs) {
            const Item it = item_of(t);
            for (int k = it.k0; k < it.k1 + it.nz; ++k, rp.next(TL::kS), ap.next(TL::kA)) {
                const int st = rp.i;
                const uint32_t dst = lane_addr + (uint32_t)ap.i * 64;
                const bool zstep = kGroup && k >= it.k1;
                ok = mbar_wait(&s.wfull[st], rp.phase, abort_flag, a.wait_ns);
                if (--slots < 0) {
                    ok = ok && mbar_wait(&s.empty[freed.i], freed.phase, abort_flag, a.wait_ns);
                    freed.next(TL::kS);
                }
                ok = __all_sync(0xffffffffu, ok);            // the tensor-memory stores are warp-wide
                if (!ok) { p16_abort(s, a); break; }
                tc_fence_after_sync();
                if (zstep) {
                    griddep_wait();                          // zeros may come from the kernel in front
                    const int g0 = it.k0 + 16 * (k - it.k1);
                    const int64_t at = (int64_t)min(it.nt * 256 + (int)rank * 128 + row, a.N - 1) * a.groups;
#pragma unroll 1
                    for (int h = 0; h < 2 && g0 + 8 * h < it.k1; ++h) {
                        float z[8], sc[8];                   // all loads at once: what is past the end is read from the last group
                        if (vec) {
#pragma unroll
                            for (int j = 0; j < 8; j += 4) {
                                const int g = min(g0 + 8 * h + j, it.k1 - 4);
                                *reinterpret_cast<float4*>(z + j) = __ldg(reinterpret_cast<const float4*>(a.zeros + at + g));
                                *reinterpret_cast<float4*>(sc + j) = __ldg(reinterpret_cast<const float4*>(a.scales + at + g));
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                const int g = min(g0 + 8 * h + j, it.k1 - 1);
                                z[j] = __ldg(a.zeros + at + g);
                                sc[j] = __ldg(a.scales + at + g);
                            }
                        }
                        uint32_t r[32];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            // zh zh' | zh' zm | zm zl | zm zl against xh xm | xl xh' | xm xh' | xl xm (a primed part is zero beside an infinity or NaN)
                            const Bf16Parts p = bf16_parts(g0 + 8 * h + j < it.k1 ? fmaf(7.5f, sc[j], z[j]) : 0.f);      // of centred codes
                            r[4 * j] = p.h | (p.h1 << 16);
                            r[4 * j + 1] = p.h1 | (p.m << 16);
                            r[4 * j + 2] = p.m | (p.l << 16);
                            r[4 * j + 3] = p.m | (p.l << 16);
                        }
                        tmem_st32(dst + h * 32, r);
                    }
                } else {
                    const uint8_t* wrow = ring + (size_t)st * TL::kStage + row * (kGroup ? 64 : 128);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {                // 64 k = 32 columns at a time
                        uint32_t r[32];
                        if constexpr (kGroup) {
#pragma unroll
                            for (int c = 0; c < 2; ++c) {        // 64-byte swizzle: 16-byte piece p of row r sits at p ^ ((r / 2) % 4)
                                const uint4 v = *reinterpret_cast<const uint4*>(wrow + (((h * 2 + c) ^ ((row >> 1) & 3)) << 4));
                                widen_nibbles_centred(v.x, centre, r + c * 16, r + c * 16 + 8);
                                widen_nibbles_centred(v.y, centre, r + c * 16 + 2, r + c * 16 + 10);
                                widen_nibbles_centred(v.z, centre, r + c * 16 + 4, r + c * 16 + 12);
                                widen_nibbles_centred(v.w, centre, r + c * 16 + 6, r + c * 16 + 14);
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < 4; ++c) {        // 128-byte swizzle: piece p at p ^ (r % 8)
                                const uint4 v = *reinterpret_cast<const uint4*>(wrow + (((h * 4 + c) ^ (row & 7)) << 4));
                                s8x4_to_f16x4(v.x, r + c * 8);
                                s8x4_to_f16x4(v.y, r + c * 8 + 2);
                                s8x4_to_f16x4(v.z, r + c * 8 + 4);
                                s8x4_to_f16x4(v.w, r + c * 8 + 6);
                            }
                        }
                        tmem_st32(dst + h * 32, r);
                    }
                }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                mbar_arrive_cluster_relaxed(leader_aready + (uint32_t)ap.i * 8, lane);
            }
        }
    } else {
        // ============================== epilogue ==============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
        griddep_wait();
        const int q = warp & 3, j = (warp - 4) >> 2;     // lane quarter; the issuing warp whose units these are
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
        const uint32_t leader_dempty = mapa_u32(smem_u32(&s.dempty[0]), 0);
        // columns 32 c .. 32 c + 31 of unit 2 i + j are 32 neighbouring tokens of one CTA's half of the tile
        auto first_token = [&](int i, int c) { return c / (UN / 64) * (NB / 2) + (2 * i + j) * (UN / 2) + c % (UN / 64) * 32; };
        auto release = [&](int buf) {
            tc_fence_before_sync();
            __syncwarp();
            mbar_arrive_cluster_relaxed(leader_dempty + (uint32_t)buf * 8, lane);
        };
        RingPos fp;
        bool ok = true;
        for (int t = pair; t < items && ok; t += npairs) {
            const Item it = item_of(t);
            const int row = it.nt * 256 + (int)rank * 128 + q * 32 + lane;
            // a warp's 32 lanes are 32 neighbouring weight rows: 64 (fp16) or 128 (fp32) contiguous bytes per token
            const int mend = row < a.N ? a.M : 0;
            const int64_t pitch = a.slices > 1 ? (int64_t)a.N * 4 : a.ldo * 2;
            uint8_t* const base = a.slices > 1 ? reinterpret_cast<uint8_t*>(a.part + (int64_t)it.sl * a.M * a.N + row) : reinterpret_cast<uint8_t*>(a.out + row);
            auto store = [&](int m, float v0, float v1) {
                uint8_t* p = base + m * pitch;
                if (a.slices > 1) {
                    if (m < mend) *reinterpret_cast<float*>(p) = v0;
                    if (m + 1 < mend) *reinterpret_cast<float*>(p + pitch) = v1;
                } else {
                    if (m < mend) *reinterpret_cast<__half*>(p) = __float2half_rn(v0);
                    if (m + 1 < mend) *reinterpret_cast<__half*>(p + pitch) = __float2half_rn(v1);
                }
            };
            if constexpr (kGroup) {
                uint64_t acc[TL::kU][UN / 2];
#pragma unroll
                for (int i = 0; i < TL::kU; ++i)
#pragma unroll
                    for (int n = 0; n < UN / 2; ++n) acc[i][n] = 0;
                const float* srow = a.scales + (int64_t)min(row, a.N - 1) * a.groups;
                // scale of group k, or what undoes the factor 2^23 for a step of zero points; three steps under way.  2^23: twice a centred
                // code is widened to a multiple of 2^-24.
                auto scale_of = [&](int k) { return k < it.k1 ? __ldg(srow + k) : 1.f / 8388608.f; };
                float s0 = scale_of(it.k0), s1 = scale_of(it.k0 + 1), s3 = scale_of(it.k0 + 2);
#pragma unroll 1
                for (int k = it.k0; k < it.k1 + it.nz && ok; ++k) {
                    const float sc = s0 * 8388608.f;
                    s0 = s1;
                    s1 = s3;
                    s3 = scale_of(k + 3);
                    const uint64_t s2 = pack2(sc, sc);
#pragma unroll
                    for (int i = 0; i < TL::kU; ++i) {
                        const int buf = 2 * fp.i + j;
                        ok = ok && mbar_wait(&s.dfull[buf], fp.phase, abort_flag, a.wait_ns);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) { p16_abort(s, a); break; }
                        tc_fence_after_sync();
                        uint32_t r[UN / 32][32];
#pragma unroll
                        for (int c = 0; c < UN / 32; ++c) tmem_ld32(lane_addr + (uint32_t)(buf * UN) + c * 32, r[c]);
                        tmem_ld_wait();
                        release(buf);
                        fp.next(TL::kD / 2);
#pragma unroll
                        for (int c = 0; c < UN / 32; ++c)
#pragma unroll
                            for (int n = 0; n < 16; ++n) fma2_loaded(acc[i][c * 16 + n], s2, r[c][2 * n], r[c][2 * n + 1]);
                    }
                }
                if (!ok) break;
#pragma unroll
                for (int i = 0; i < TL::kU; ++i)
#pragma unroll
                    for (int n = 0; n < UN / 2; ++n) {
                        const float2 v = unpack2(acc[i][n]);
                        store(it.mt * NB + first_token(i, n / 16) + 2 * (n % 16), v.x, v.y);
                    }
            } else {
                const float ts = a.slices > 1 ? 1.f : __ldg(a.scales);
#pragma unroll
                for (int i = 0; i < TL::kU; ++i) {
                    const int buf = 2 * fp.i + j;
                    ok = ok && mbar_wait(&s.dfull[buf], fp.phase, abort_flag, a.wait_ns);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { p16_abort(s, a); break; }
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < UN / 32; ++c) {
                        uint32_t r[32];
                        tmem_ld32(lane_addr + (uint32_t)(buf * UN) + c * 32, r);
                        tmem_ld_wait();
                        if (c == UN / 32 - 1) release(buf);
#pragma unroll
                        for (int n = 0; n < 16; ++n)
                            store(it.mt * NB + first_token(i, c) + 2 * n, __uint_as_float(r[2 * n]) * ts, __uint_as_float(r[2 * n + 1]) * ts);
                    }
                    fp.next(TL::kD / 2);
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();      // both CTAs have read their last accumulator: the pair's tensor memory and the leader's barriers may go
    if (warp == 13) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------------ host side
// the register split adds up only if a thread starts with 128 registers
template <int FMT, int NB>
static bool p16_regs_fit() {
    static const bool fit = [] {
        cudaFuncAttributes fa{};
        return cudaFuncGetAttributes(&fa, gemm_wa16_pair_kernel<FMT, NB>) == cudaSuccess && fa.numRegs == kP16RegsLaunch;
    }();
    return fit;
}
bool wa16_pair_fits(int fmt) {
    return fmt == W16_INT4_GROUP ? p16_regs_fit<W16_INT4_GROUP, 128>() && p16_regs_fit<W16_INT4_GROUP, 256>() : p16_regs_fit<W16_INT8_TENSOR, 256>();
}

template <int FMT, int NB>
static int32_t launch_p16(const P16Maps& maps, const P16Args& a, cudaStream_t st, const char* who) {
    using TL = P16Tile<FMT, NB>;
    auto kern = gemm_wa16_pair_kernel<FMT, NB>;
    const int32_t rc = ensure_smem_optin(reinterpret_cast<const void*>(kern), (int)kW16SmemBudget, who);
    if (rc != RWKVQ_OK) return rc;
    const bool fit = p16_regs_fit<FMT, NB>();           // wa16_pair_fits keeps the plan from it
    RWKVQ_REQUIRE(fit, RWKVQ_E_LAUNCH, "%s: the register split needs a build with 128 per thread", who);
    const int64_t pairs = std::min<int64_t>(std::max(1, sm_count() / 2), (int64_t)a.mtiles * a.ntiles * a.slices);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(kP16Threads);
    cfg.dynamicSmemBytes = TL::kSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl() ? 2 : 1;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, maps, a);
    if (err != cudaSuccess) {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return fail(RWKVQ_E_LAUNCH, "%s: %s", who, cudaGetErrorString(err));
    }
    return check_launch(who);
}

int32_t run_wa16_pair(const W16PairCall& c, cudaStream_t st, const char* who) {
    const bool group = c.fmt == W16_INT4_GROUP;
    P16Args a{};
    a.scales = c.scales; a.zeros = c.zeros; a.out = c.out; a.part = c.part; a.ldo = c.ldo; a.M = (int)c.M; a.N = (int)c.N;
    a.ksteps = (int)((c.K + kW16K - 1) / kW16K);
    a.groups = (int)(c.K / kW16K);
    a.mtiles = (int)((c.M + c.NB - 1) / c.NB);
    a.ntiles = (int)((c.N + 255) / 256);
    a.slices = c.slices;
    a.status = device_status_ptr();
    a.wait_ns = wait_limit_ns();
    RWKVQ_REQUIRE((int64_t)a.mtiles * a.ntiles * a.slices < (int64_t(1) << 30), RWKVQ_E_SHAPE, "%s: too many tiles", who);
    P16Maps maps;
    int32_t rc = w16_map(&maps.w, c.w, c.N, group ? c.K / 2 : c.K, c.ldw, 128, group ? 64 : 128, who);
    if (rc != RWKVQ_OK) return rc;
    rc = make_map(&maps.x, c.x, c.M, c.K * 2, c.ldx * 2, c.NB / 2, who);
    if (rc != RWKVQ_OK) return rc;
    rc = group ? make_map(&maps.z, c.xz, c.M, (int64_t)a.groups * kW16ZSlots * 2, (int64_t)a.groups * kW16ZSlots * 2, c.NB / 2, who) : RWKVQ_OK;
    if (rc != RWKVQ_OK) return rc;
    if (!group) maps.z = maps.x;
    if (group) return c.NB == 128 ? launch_p16<W16_INT4_GROUP, 128>(maps, a, st, who) : launch_p16<W16_INT4_GROUP, 256>(maps, a, st, who);
    return launch_p16<W16_INT8_TENSOR, 256>(maps, a, st, who);
}

}  // namespace rwkvq
