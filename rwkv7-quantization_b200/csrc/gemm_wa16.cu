// Weight-only projections of many tokens (W4A16 group 128, W8A16 per tensor; fp16 activations) on the tensor cores:
// the weights are read from HBM in packed form, widened to fp16 INTEGERS in registers, written to TENSOR MEMORY and
// multiplied from there (tcgen05.mma.kind::f16, A operand in tensor memory, tokens = B operand from shared memory).
//
// Arithmetic.  An INT4 code (0 .. 15) and an INT8 code (-128 .. 127) are exact in fp16, so the products with the fp16
// activations and their fp32 sums are those of the decode kernel (gemv_int4.cu).  Scales stay in fp32 and are never
// multiplied into a 16-bit operand: INT4 accumulates one group of 128 k in its own tensor-memory accumulator and the
// epilogue warps add  scale[n,g] * acc + zero[n,g] * sum_{k in g} x[k]  to fp32 registers, group after group, while the
// tensor core works on the next group; INT8 accumulates all of K and multiplies by the tensor scale once.
//
// Why A in tensor memory.  A 128 x 128 x 16 step with both operands in shared memory reads 128 bytes per clock, all an
// SM's shared memory gives, before the widened weights have even been written there.  A lane of tensor memory is one
// weight row, so the thread that widens row r stores its own lane (tcgen05.st, no swizzle, no bank conflicts), the MMA
// reads 64 bytes per clock of activations from shared memory, and the epilogue thread of lane r needs exactly the
// scale and zero of row r.
//
// Nibbles.  A nibble left in the low mantissa bits of an fp16 is the SUBNORMAL n * 2^-24, which the tensor core
// multiplies exactly: w & 0x000F000F is the pair (n0, n4) * 2^-24, w & 0x00F000F0 is (n1, n5) * 2^-20, and the same masks
// on w >> 8 give (n2, n6) and (n3, n7) -- 5 instructions for 8 weights.  An MMA sums over k in any order as long as both
// operands agree, so each run of 32 k is stored as its 16 odd k, then its 16 even ones (wa16_prep_kernel does the same to
// the activations, converts bf16 to fp16 and forms the group sums on the way): of a step's eight MMAs the four odd ones
// run first, and the first even one multiplies the accumulator by 2^-4 as it adds to it (scale-input-d), which is exact.
// 2^24 joins the scale.  The activations are never scaled themselves: a sixteenth of an fp16 value below 2^-10 would be
// rounded.
//
// Roles (512 threads, one persistent CTA per SM): warps 0-3 widen weights (lane quarter = warp), warps 4-11 are the
// epilogue (two warps per lane quarter, half of the tokens each), warp 12 = TMA producer, warp 13 = MMA issuer.
// Stage n of the ring carries 128 k of 128 weight rows and of NB tokens; its widened weights live in tensor-memory
// columns of the same stage index, so one "empty" barrier (the MMA's commit) frees both.  Work items are (K slice,
// row tile, token tile); with more than one slice the fp32 partial sums go to a buffer that wa16_reduce_kernel adds in
// slice order.
#include <algorithm>
#include <cstdlib>

#include "wa16.cuh"

namespace rwkvq {

constexpr int kW16Threads = 512;                // four warpgroups
constexpr int kW16MaxStages = 7;

struct W16Maps {
    CUtensorMap w, x;
};
struct W16Args {
    const float* scales;      // INT4: [N, groups]; INT8: [1]
    const float* zeros;       // INT4: [N, groups] or null (zero = -8 * scale)
    const float* xsum;        // INT4: [token tile][group][NB] sums of the activations
    __half* out;
    float* part;              // slices > 1: fp32 partial sums [slices][M][N]
    int64_t ldo;
    int M, N, ksteps, groups;
    int mtiles, ntiles, slices;
    int* status;
    unsigned long long wait_ns;
};
struct W16Shared {
    uint64_t full[kW16MaxStages], empty[kW16MaxStages], aready[kW16MaxStages], dfull[2], dempty[2];
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ void w16_abort(W16Shared& s, const W16Args& a) {
    s.abort_flag = 1;
    if (a.status) atomicExch(a.status, RWKVQ_E_TIMEOUT);
}
// D[tmem] (+)= A[tmem] * B[smem], fp16 operands, fp32 accumulator
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with the accumulator multiplied by 2^-4 before the sum
__device__ __forceinline__ void tc_mma_f16_ts_d16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 4;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc) : "memory");
}
template <int FMT, int NB>
struct W16Tile {
    static constexpr bool kGroup = FMT == W16_INT4_GROUP;
    static constexpr uint32_t kWBytes = 128u * (kGroup ? kW16K / 2 : kW16K);
    static constexpr uint32_t kXSlab = (uint32_t)NB * 128u;             // 64 k of the token tile, 128-byte swizzled rows
    static constexpr uint32_t kStage = kWBytes + 2 * kXSlab;
    static constexpr uint32_t kTx = kStage + (kGroup ? (uint32_t)NB * 4u : 0u);
    static constexpr uint32_t kACol = 2 * NB;                           // two accumulators, then the widened weights (64 columns a stage)
    static constexpr int kS = (512 - 2 * NB) / 64 < kW16MaxStages ? (512 - 2 * NB) / 64 : kW16MaxStages;    // ring stages
    static constexpr int kXS = kS + 2;
    // the group sums live in their own ring of stages + 2 slots: the epilogue of step n has read them before the MMA of
    // step n + 2 may start, hence before stage n + 2 is released and the load of step n + 2 + stages is issued
    // 96 and 128 tokens, INT4: an epilogue thread keeps up to 64 sums and 64 loaded values, more than the 128 registers of 512
    // threads; the widening warps (104) and the TMA / MMA warps (56) hand theirs to the two epilogue warpgroups (176):
    // 104 + 56 + 2 * 176 = 4 * 128, the launch's own total
    static constexpr bool kRegSplit = kGroup && NB > 64;
    static constexpr size_t kSmem = 1024 + (size_t)kS * kStage + (kGroup ? (size_t)kXS * NB * 4 : 0);
    static_assert(kSmem <= kW16SmemBudget, "ring");
};

template <int FMT, int NB>
__global__ void __launch_bounds__(kW16Threads, 1) gemm_wa16_kernel(const __grid_constant__ W16Maps maps, const W16Args a) {
    using TL = W16Tile<FMT, NB>;
    constexpr bool kGroup = TL::kGroup;
    extern __shared__ uint8_t smem_raw[];
    __shared__ W16Shared s;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* xsring = reinterpret_cast<float*>(ring + (size_t)TL::kS * TL::kStage);
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;

    griddep_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < TL::kS; ++i) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], 1);
            mbar_init(&s.aready[i], 4);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s.dfull[i], 1);
            mbar_init(&s.dempty[i], 8);
        }
        s.abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
        prefetch_tmap(&maps.w);
        prefetch_tmap(&maps.x);
    }
    if (warp == 13) tmem_alloc(&s.tmem_base, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = warp_uniform(s.tmem_base);
    const volatile int* abort_flag = &s.abort_flag;
    const int items = a.mtiles * a.ntiles * a.slices;
    // item -> (token tile, row tile, K range); token tiles fastest, so the CTAs at work share weight tiles through L2.
    // K slices start at multiples of 4 steps (16-byte vectors of scales).
    struct Item { int mt, nt, sl, k0, k1; };
    auto item_of = [&](int t) {
        Item it;
        it.mt = t % a.mtiles;
        const int r = t / a.mtiles;
        it.nt = r % a.ntiles;
        it.sl = r / a.ntiles;
        const int q4 = (a.ksteps + 3) >> 2;
        it.k0 = (int)((uint32_t)(q4 * it.sl) / (uint32_t)a.slices) * 4;             // below 2^21 * 16
        it.k1 = min((int)((uint32_t)(q4 * (it.sl + 1)) / (uint32_t)a.slices) * 4, a.ksteps);
        return it;
    };

    if (warp >= 12) {
        if constexpr (TL::kRegSplit) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 12) {
        // ============================== TMA producer ==============================
        {
            const bool leader = elect_one();
            constexpr int kWRow = kGroup ? kW16K / 2 : kW16K;
            int npre = 0;
            // first pass over the ring: weights never depend on the kernels in front, so they are requested before the
            // dependency wait of programmatic dependent launch
            for (int t = blockIdx.x; t < items && npre < TL::kS; t += gridDim.x) {
                const Item it = item_of(t);
                for (int k = it.k0; k < it.k1 && npre < TL::kS; ++k, ++npre) {
                    if (leader) {
                        mbar_expect_tx(&s.full[npre], TL::kTx);
                        tma_load_2d(ring + (size_t)npre * TL::kStage, &maps.w, k * kWRow, it.nt * 128, &s.full[npre]);
                    }
                }
            }
            griddep_wait();
            bool ok = true;
            RingPos rp;
            RingPos xp;
            for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
                const Item it = item_of(t);
                const float* xsrc = kGroup ? a.xsum + ((int64_t)it.mt * a.groups + it.k0) * NB : nullptr;
                for (int k = it.k0; k < it.k1; ++k, rp.next(TL::kS), xp.next(TL::kXS)) {
                    const int st = rp.i;
                    uint8_t* dst = ring + (size_t)st * TL::kStage;
                    const bool refill = --npre < 0;
                    if (refill && !mbar_wait(&s.empty[st], rp.phase ^ 1, abort_flag, a.wait_ns)) ok = false;
                    if (!__all_sync(0xffffffffu, ok)) { w16_abort(s, a); ok = false; break; }
                    if (leader) {
                        if (refill) {
                            mbar_expect_tx(&s.full[st], TL::kTx);
                            tma_load_2d(dst, &maps.w, k * kWRow, it.nt * 128, &s.full[st]);
                        }
                        tma_load_2d(dst + TL::kWBytes, &maps.x, k * 256, it.mt * NB, &s.full[st]);
                        tma_load_2d(dst + TL::kWBytes + TL::kXSlab, &maps.x, k * 256 + 128, it.mt * NB, &s.full[st]);
                        if constexpr (kGroup) bulk_load_1d(xsring + (size_t)xp.i * NB, xsrc, NB * 4, &s.full[st]);
                    }
                    if constexpr (kGroup) xsrc += NB;
                }
            }
            if (!ok) {   // give copies already in flight a bounded time to land before the CTA's memory is released
                const unsigned long long t0 = global_ns();
                while (global_ns() - t0 < 2000000ull) {}
            }
        }
        } else if (warp == 13) {
        // ============================== MMA issuer ==============================
        {
            const bool leader = elect_one();
            const uint32_t idesc = (1u << 4) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);      // f32 += f16 * f16, both K-major, M = 128
            RingPos rp;
            RingPos fp;                          // accumulator fill
            const uint32_t ring_addr = warp_uniform(smem_u32(ring));
            bool ok = true;
            for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
                const Item it = item_of(t);
                for (int k = it.k0; k < it.k1; ++k, rp.next(TL::kS)) {
                    const int st = rp.i;
                    const bool fresh = kGroup || k == it.k0;
                    ok = (!fresh || mbar_wait(&s.dempty[fp.i], fp.phase ^ 1, abort_flag, a.wait_ns)) && mbar_wait(&s.full[st], rp.phase, abort_flag, a.wait_ns) &&
                         mbar_wait(&s.aready[st], rp.phase, abort_flag, a.wait_ns);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { w16_abort(s, a); break; }
                    tc_fence_after_sync();
                    const uint32_t d = tmem_base + (uint32_t)(fp.i * NB), at = tmem_base + TL::kACol + (uint32_t)st * 64;
                    const uint32_t sb = ring_addr + (uint32_t)st * TL::kStage + TL::kWBytes;
                    const uint64_t b0 = umma_desc_sw128(sb), b1 = umma_desc_sw128(sb + TL::kXSlab);
                    const bool last = kGroup || k == it.k1 - 1;
                    if (leader) {
#pragma unroll
                        for (int i = 0; i < kW16K / 16; ++i) {
                            const int j = kGroup ? (i < 4 ? 2 * i : 2 * i - 7) : i;          // INT4: the odd k (j even) first
                            const uint64_t b = (j < 4 ? b0 : b1) + (uint64_t)((j & 3) * 2);
                            if (kGroup && i == 4) tc_mma_f16_ts_d16(d, at + j * 8, b, idesc);
                            else tc_mma_f16_ts(d, at + j * 8, b, idesc, (fresh && i == 0) ? 0u : 1u);
                        }
                        tc_commit(&s.empty[st]);
                        if (last) tc_commit(&s.dfull[fp.i]);
                    }
                    if (last) fp.next(2);
                }
            }
        }
        }
    } else if (warp < 4) {
        if constexpr (TL::kRegSplit) asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
        // ============================== weights: packed -> fp16 in tensor memory ==============================
        const uint32_t lane_addr = tmem_base + TL::kACol + ((uint32_t)(warp * 32) << 16);
        const int row = warp * 32 + lane;
        RingPos rp;
        bool ok = true;
        for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
            const Item it = item_of(t);
            for (int k = it.k0; k < it.k1; ++k, rp.next(TL::kS)) {
                const int st = rp.i;
                ok = mbar_wait(&s.full[st], rp.phase, abort_flag, a.wait_ns);
                ok = __all_sync(0xffffffffu, ok);           // the tensor-memory stores are warp-wide
                if (!ok) { w16_abort(s, a); break; }
                tc_fence_after_sync();                       // the stage's columns were read by MMAs that the full barrier implies complete
                const uint8_t* wrow = ring + (size_t)st * TL::kStage + row * (kGroup ? 64 : 128);
#pragma unroll
                for (int h = 0; h < 2; ++h) {                // 64 k = 32 columns at a time
                    uint32_t r[32];
                    if constexpr (kGroup) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {        // 64-byte swizzle: 16-byte piece p of row r sits at p ^ ((r / 2) % 4)
                            const uint4 v = *reinterpret_cast<const uint4*>(wrow + (((h * 2 + c) ^ ((row >> 1) & 3)) << 4));
                            widen_nibbles(v.x, r + c * 16, r + c * 16 + 8);
                            widen_nibbles(v.y, r + c * 16 + 2, r + c * 16 + 10);
                            widen_nibbles(v.z, r + c * 16 + 4, r + c * 16 + 12);
                            widen_nibbles(v.w, r + c * 16 + 6, r + c * 16 + 14);
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
                    tmem_st32(lane_addr + (uint32_t)st * 64 + h * 32, r);
                }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s.aready[st]);
            }
        }
    } else {
        // ============================== epilogue ==============================
        if constexpr (TL::kRegSplit) asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
        griddep_wait();
        constexpr int NH = NB / 2;                       // tokens of this warp
        constexpr int CH = NH % 32 == 0 ? 32 : 16;       // tensor-memory columns per load
        const int q = warp & 3, half = (warp - 4) >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + half * NH;
        RingPos xp;
        RingPos fp;
        bool ok = true;
        for (int t = blockIdx.x; t < items && ok; t += gridDim.x) {
            const Item it = item_of(t);
            const int row = it.nt * 128 + q * 32 + lane;
            uint64_t acc[NH / 2];
#pragma unroll
            for (int j = 0; j < NH / 2; ++j) acc[j] = 0;
            if constexpr (kGroup) {
                const int64_t srow = (int64_t)min(row, a.N - 1) * a.groups;
                const bool vec = (a.groups & 3) == 0;    // host: scales and zeros are 16-byte aligned
                float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f), z4 = s4, s4n = s4, z4n = s4;
                auto load4 = [&](int k, float4& sv, float4& zv) {
                    if (k >= it.k1) return;
                    if (vec) {
                        sv = __ldg(reinterpret_cast<const float4*>(a.scales + srow + k));
                        if (a.zeros) zv = __ldg(reinterpret_cast<const float4*>(a.zeros + srow + k));
                    } else {
                        const float* p = a.scales + srow;
                        const int last = a.groups - 1;
                        sv = make_float4(__ldg(p + k), __ldg(p + min(k + 1, last)), __ldg(p + min(k + 2, last)), __ldg(p + min(k + 3, last)));
                        if (a.zeros) {
                            const float* z = a.zeros + srow;
                            zv = make_float4(__ldg(z + k), __ldg(z + min(k + 1, last)), __ldg(z + min(k + 2, last)), __ldg(z + min(k + 3, last)));
                        }
                    }
                    if (!a.zeros) zv = make_float4(-8.f * sv.x, -8.f * sv.y, -8.f * sv.z, -8.f * sv.w);
                };
                load4(it.k0, s4n, z4n);
#pragma unroll 1
                for (int k = it.k0; k < it.k1; ++k, xp.next(TL::kXS), fp.next(2)) {
                    const int j4 = k & 3;                // k0 is a multiple of 4
                    if (j4 == 0) {
                        s4 = s4n;
                        z4 = z4n;
                        load4(k + 4, s4n, z4n);          // in flight during four steps
                    }
                    const float sc = j4 == 0 ? s4.x : (j4 == 1 ? s4.y : (j4 == 2 ? s4.z : s4.w));
                    const float ze = j4 == 0 ? z4.x : (j4 == 1 ? z4.y : (j4 == 2 ? z4.z : z4.w));
                    const uint64_t s2 = pack2(sc * 16777216.f, sc * 16777216.f), z2 = pack2(ze, ze);
                    ok = mbar_wait(&s.dfull[fp.i], fp.phase, abort_flag, a.wait_ns);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { w16_abort(s, a); break; }
                    tc_fence_after_sync();
                    const float* xs = xsring + (size_t)xp.i * NB + half * NH;
                    uint32_t r[NH / CH][CH];
#pragma unroll
                    for (int c = 0; c < NH / CH; ++c) {
                        if constexpr (CH == 32) tmem_ld32(lane_addr + (uint32_t)(fp.i * NB) + c * CH, r[c]);
                        else tmem_ld16(lane_addr + (uint32_t)(fp.i * NB) + c * CH, r[c]);
                    }
#pragma unroll
                    for (int i = 0; i < NH / 4; ++i) {               // the zeros' part while the loads are under way
                        const float4 xv = *reinterpret_cast<const float4*>(xs + 4 * i);
                        fma2(acc[2 * i], z2, pack2(xv.x, xv.y));
                        fma2(acc[2 * i + 1], z2, pack2(xv.z, xv.w));
                    }
                    tmem_ld_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&s.dempty[fp.i]);     // sums and accumulator of this step have been read
#pragma unroll
                    for (int c = 0; c < NH / CH; ++c)
#pragma unroll
                        for (int i = 0; i < CH / 2; ++i) fma2_loaded(acc[c * (CH / 2) + i], s2, r[c][2 * i], r[c][2 * i + 1]);
                }
                if (!ok) break;
            } else {
                ok = mbar_wait(&s.dfull[fp.i], fp.phase, abort_flag, a.wait_ns);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { w16_abort(s, a); break; }
                tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < NH; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(lane_addr + (uint32_t)(fp.i * NB) + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[c / 2 + i] = pack2_loaded(r[2 * i], r[2 * i + 1]);
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s.dempty[fp.i]);
                fp.next(2);
            }
            // a warp's 32 lanes are 32 neighbouring weight rows: 64 (fp16) or 128 (fp32) contiguous bytes per token
            if (row < a.N) {
                const int m0 = it.mt * NB + half * NH;
                const int cnt = min(NH, a.M - m0);
                const float ts = kGroup ? 1.f : __ldg(a.scales);
                if (a.slices > 1) {
                    float* p = a.part + ((int64_t)it.sl * a.M + m0) * a.N + row;
#pragma unroll
                    for (int j = 0; j < NH / 2; ++j) {
                        const float2 v = unpack2(acc[j]);
                        if (2 * j < cnt) p[(int64_t)(2 * j) * a.N] = v.x;
                        if (2 * j + 1 < cnt) p[(int64_t)(2 * j + 1) * a.N] = v.y;
                    }
                } else {
                    __half* p = a.out + (int64_t)m0 * a.ldo + row;
#pragma unroll
                    for (int j = 0; j < NH / 2; ++j) {
                        const float2 v = unpack2(acc[j]);
                        if (2 * j < cnt) p[(int64_t)(2 * j) * a.ldo] = __float2half_rn(v.x * ts);
                        if (2 * j + 1 < cnt) p[(int64_t)(2 * j + 1) * a.ldo] = __float2half_rn(v.y * ts);
                    }
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 13) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

// Activations for the INT4 kernel: fp16 rows with each run of 32 stored as [1,5,3,7, 9,13,11,15, ...] and then
// [0,4,2,6, 8,12,10,14, ...], and the sums of each group of 128 (of the fp16 values), [token tile][group][NB].  16 lanes hold a group; bound by the one read and one write, so a thread
// has four vectors under way: 1 << lgP of a row and the same of the next 4 >> lgP of its CTA's rows.
template <int DT>
__global__ void __launch_bounds__(256) wa16_prep_kernel(const uint16_t* __restrict__ x, int64_t ldx, int M, int kv, __half* xp, float* xsum, uint4* xz, int NB,
                                                        int groups, int cpr, int lgP) {
    griddep_launch_dependents();
    const int seg = (int)blockIdx.x % cpr, rstep = (int)gridDim.x / cpr, cstep = cpr * 256, P = 1 << lgP;
    const uint32_t mask = 0xffffu << (threadIdx.x & 16);
    griddep_wait();
    for (int r0 = (int)blockIdx.x / cpr; r0 < M; r0 += rstep << (2 - lgP)) {
        for (int base = seg * 256; base < kv; base += P * cstep) {
            uint4 v4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int m = r0 + (j >> lgP) * rstep, i = base + (j & (P - 1)) * cstep + (int)threadIdx.x;
                if (m < M && i < kv) v4[j] = ldg_l2_16(x + (int64_t)m * ldx + (int64_t)i * 8);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int m = r0 + (j >> lgP) * rstep, i = base + (j & (P - 1)) * cstep + (int)threadIdx.x;
                if (m >= M || i >= kv) continue;           // kv is a multiple of 16: the half-warps stay whole
                uint4 v = v4[j];
                float2 f[4] = {cvt2<DT>(v.x), cvt2<DT>(v.y), cvt2<DT>(v.z), cvt2<DT>(v.w)};
                if constexpr (DT == RWKVQ_BF16) {
                    uint32_t h[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const __half2 hh = __floats2half2_rn(f[q].x, f[q].y);
                        h[q] = *reinterpret_cast<const uint32_t*>(&hh);
                        f[q] = cvt2<RWKVQ_F16>(h[q]);
                    }
                    v = make_uint4(h[0], h[1], h[2], h[3]);
                }
                __half* run = xp + ((int64_t)m * kv + (i & ~3)) * 8 + (i & 3) * 4;       // a row is a whole number of runs (K % 128 == 0)
                *reinterpret_cast<uint2*>(run) = make_uint2(__byte_perm(v.x, v.z, 0x7632), __byte_perm(v.y, v.w, 0x7632));
                *reinterpret_cast<uint2*>(run + 16) = make_uint2(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.y, v.w, 0x5410));
                float sum = ((f[0].x + f[0].y) + (f[1].x + f[1].y)) + ((f[2].x + f[2].y) + (f[3].x + f[3].y));
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(mask, sum, o);
                if ((threadIdx.x & 15) == 0) {
                    if (xz) {
                        const Bf16Parts p = bf16_parts(sum);
                        xz[(int64_t)m * groups + (i >> 4)] = make_uint4(p.h | (p.m << 16), p.l | (p.h1 << 16), p.m | (p.h1 << 16), p.l | (p.m << 16));
                    } else {
                        xsum[((int64_t)(m / NB) * groups + (i >> 4)) * NB + m % NB] = sum;
                    }
                }
            }
        }
    }
}

// out[m][n] = fp16(scale * sum over slices, in slice order, of part[s][m][n]); four columns per thread
__global__ void __launch_bounds__(256) wa16_reduce_kernel(const float* __restrict__ part, int slices, int M, int N, const float* scale, __half* out, int64_t ldo) {
    griddep_launch_dependents();
    const float ts = scale ? __ldg(scale) : 1.f;
    griddep_wait();
    const int64_t total = (int64_t)M * N;
    const bool vec = (N & 3) == 0;
    const int64_t step = vec ? 4 : 1;
    for (int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * step; i < total; i += (int64_t)gridDim.x * 256 * step) {
        const int64_t m = i / N;
        __half* o = out + m * ldo + (i - m * N);
        if (vec) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int sl = 0; sl < slices; ++sl) {
                const float4 p = __ldcg(reinterpret_cast<const float4*>(part + (int64_t)sl * total + i));
                v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
            }
            const __half h[4] = {__float2half_rn(v.x * ts), __float2half_rn(v.y * ts), __float2half_rn(v.z * ts), __float2half_rn(v.w * ts)};
            if ((ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0) *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(h);
            else for (int j = 0; j < 4; ++j) o[j] = h[j];
        } else {
            float v = 0.f;
            for (int sl = 0; sl < slices; ++sl) v += __ldcg(part + (int64_t)sl * total + i);
            *o = __float2half_rn(v * ts);
        }
    }
}

// ------------------------------------------------------------------------------------------------ host side
struct W16Plan { int NB, slices; bool pair; };

// Form (single CTAs or pairs), token tile and K slices: those with the least estimated time.  Measured on [4096, 4096], [16384, 4096],
// [4096, 16384], [2560, 2560], [10240, 2560], [2560, 10240], [1024, 1024] and [4096, 1024] at 8 to 2048 rows: a step (128 k of a tile)
// takes 0.40 / 0.52 / 0.65 / 0.76 us with 32 / 64 / 96 / 128 tokens on one CTA (INT4: the widened weights and the accumulators share
// tensor memory's ports with the MMAs) and 0.40 / 0.43 / 0.48 / 0.55 us (INT8: what an SM takes in from L2); on a pair, with 256 weight
// rows, 0.58 / 0.88 us with 128 / 256 tokens (INT4) and 0.73 us with 256 (INT8); K slices cost 3.4 us for the second launch plus
// the round trip of the partial sums.  Of the forms timed for each size the estimate takes one within 10 % of the best.
// The register split of the INT4 kernels with 96 and 128 tokens adds up only if a thread starts with 128 registers; a compiler
// that gives them another number leaves the narrower tiles.  RWKVQ_WA16_MAX_NB lowers the limit (read once).
template <int NB>
static bool w16_regs_fit() {
    static const bool fit = [] {
        cudaFuncAttributes fa{};
        return cudaFuncGetAttributes(&fa, gemm_wa16_kernel<W16_INT4_GROUP, NB>) == cudaSuccess && fa.numRegs == 128;
    }();
    return fit;
}
static int w16_max_tokens(int fmt) {
    static const int cap = std::getenv("RWKVQ_WA16_MAX_NB") ? std::max(32, std::atoi(std::getenv("RWKVQ_WA16_MAX_NB"))) : 256;
    return fmt == W16_INT8_TENSOR || (w16_regs_fit<96>() && w16_regs_fit<128>()) ? cap : std::min(cap, 64);
}
static W16Plan wa16_plan(int fmt, int64_t M, int64_t N, int64_t K) {
    static constexpr double kStep[2][4] = {{400., 520., 650., 760.}, {400., 430., 480., 550.}};      // ns
    static constexpr double kPairStep[2][2] = {{575., 875.}, {0., 730.}};                            // 0: no such tile
    // RWKVQ_WA16_PAIR=0 switches the pairs off, =force uses them wherever they are legal (read once)
    static const char mode = std::getenv("RWKVQ_WA16_PAIR") ? std::getenv("RWKVQ_WA16_PAIR")[0] : 0;
    const int64_t ksteps = (K + kW16K - 1) / kW16K, q4 = (ksteps + 3) / 4;
    const int max_nb = w16_max_tokens(fmt);
    W16Plan best{32, 1, false};
    double best_t = 1e30;
    for (int i = 0; i < 6; ++i) {
        const bool pair = i >= 4;
        const int nb = pair ? 128 << (i - 4) : 32 * (i + 1);
        if (nb > max_nb || (pair && (kPairStep[fmt][i - 4] == 0. || mode == '0' || !wa16_pair_fits(fmt))) || (!pair && mode == 'f')) continue;
        const int64_t mt = (M + nb - 1) / nb, nt = pair ? (N + 255) / 256 : (N + 127) / 128, units = pair ? sm_count() / 2 : sm_count();
        for (int64_t sl = 1; sl <= 16 && sl <= q4; ++sl) {
            const int64_t waves = (mt * nt * sl + units - 1) / units, len = std::min((q4 + sl - 1) / sl * 4, ksteps);
            double t = (double)waves * ((double)len * (pair ? kPairStep[fmt][i - 4] : kStep[fmt][i]) + 300.0);
            if (pair) t += waves * (fmt == W16_INT4_GROUP ? (len + 15) / 16 : 0) * kPairStep[fmt][i - 4] + 500.0;
            if (sl > 1) t += 3400.0 + (double)sl * M * N * 8.0 / 8000.0;
            if (t < best_t) { best_t = t; best = {nb, (int)sl, pair}; }
        }
    }
    return best;
}

template <int FMT, int NB>
static int32_t launch_wa16(const W16Maps& maps, W16Args a, cudaStream_t st, const char* who) {
    using TL = W16Tile<FMT, NB>;
    auto kern = gemm_wa16_kernel<FMT, NB>;
    const int32_t rc = ensure_smem_optin(reinterpret_cast<const void*>(kern), (int)kW16SmemBudget, who);
    if (rc != RWKVQ_OK) return rc;
    if constexpr (TL::kRegSplit)        // w16_max_tokens keeps the plan from it
        RWKVQ_REQUIRE(w16_regs_fit<NB>(), RWKVQ_E_LAUNCH, "%s: the register split of %d-token tiles needs a build with 128 per thread", who, NB);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::min<int64_t>(sm_count(), (int64_t)a.mtiles * a.ntiles * a.slices));
    cfg.blockDim = dim3(kW16Threads);
    cfg.dynamicSmemBytes = TL::kSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl() ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, maps, a);
    if (err != cudaSuccess) {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return fail(RWKVQ_E_LAUNCH, "%s: %s", who, cudaGetErrorString(err));
    }
    return check_launch(who);
}

template <typename Kern, typename... Args>
static int32_t launch_plain(Kern kern, int64_t blocks, cudaStream_t st, const char* who, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(blocks, 8 * (int64_t)sm_count())));
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = use_pdl() ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, args...);
    if (err != cudaSuccess) {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return fail(RWKVQ_E_LAUNCH, "%s: %s", who, cudaGetErrorString(err));
    }
    return check_launch(who);
}

struct W16Layout { int64_t xp, xsum, part, total; };     // byte offsets in the workspace, 256-byte aligned
static W16Layout wa16_layout(int fmt, int64_t M, int64_t N, int64_t K, const W16Plan& p) {
    auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
    W16Layout l{};
    int64_t at = 0;
    if (fmt == W16_INT4_GROUP) {
        l.xp = at; at += up(M * K * 2);
        l.xsum = at; at += up(p.pair ? M * (K / kW16K) * kW16ZSlots * 2 : (M + p.NB - 1) / p.NB * p.NB * (K / kW16K) * 4);
    }
    l.part = at;
    if (p.slices > 1) at += up((int64_t)p.slices * M * N * 4);
    l.total = std::max<int64_t>(at, 256);
    return l;
}

static int32_t run_wa16(int fmt, const void* x, int x_dtype, int64_t ldx, const void* w, int64_t ldw, const float* scales, const float* zeros,
                        void* out, int64_t ldo, int64_t M, int64_t N, int64_t K, void* workspace, int64_t workspace_bytes, cudaStream_t st, const char* who) {
    const bool group = fmt == W16_INT4_GROUP;
    RWKVQ_REQUIRE(M >= 0 && N >= 0 && K >= 0 && M < (int64_t(1) << 30) && N < (int64_t(1) << 30) && K < (int64_t(1) << 30), RWKVQ_E_SHAPE,
                  "%s: M=%lld, N=%lld, K=%lld", who, (long long)M, (long long)N, (long long)K);
    if (M == 0 || N == 0) return RWKVQ_OK;
    RWKVQ_REQUIRE(x && w && scales && out, RWKVQ_E_BADARG, "%s: null pointer", who);
    RWKVQ_REQUIRE(x_dtype == RWKVQ_F16 || (group && x_dtype == RWKVQ_BF16), RWKVQ_E_BADARG, "%s: activation type %d", who, x_dtype);
    RWKVQ_REQUIRE(K > 0 && K % (group ? kW16K : 16) == 0, RWKVQ_E_SHAPE, "%s: K=%lld must be a multiple of %d", who, (long long)K, group ? kW16K : 16);
    RWKVQ_REQUIRE(aligned16(w) && ldw % 16 == 0 && ldw >= (group ? K / 2 : K), RWKVQ_E_ALIGN, "%s: weight rows must be 16-byte aligned", who);
    RWKVQ_REQUIRE(aligned16(x) && ldx % 8 == 0 && ldx >= K, RWKVQ_E_ALIGN, "%s: activation rows must be 16-byte aligned", who);
    RWKVQ_REQUIRE(!group || (aligned16(scales) && (zeros == nullptr || aligned16(zeros))), RWKVQ_E_ALIGN, "%s: scales / zeros must be 16-byte aligned", who);
    RWKVQ_REQUIRE(ldo >= N, RWKVQ_E_SHAPE, "%s: ldo < N", who);
    const W16Plan p = wa16_plan(fmt, M, N, K);
    const W16Layout l = wa16_layout(fmt, M, N, K, p);
    RWKVQ_REQUIRE(workspace && ((uintptr_t)workspace & 255) == 0 && workspace_bytes >= l.total, RWKVQ_E_WORKSPACE,
                  "%s: %lld bytes of 256-byte aligned workspace needed", who, (long long)l.total);
    uint8_t* base = reinterpret_cast<uint8_t*>(workspace);
    W16Args a{};
    a.scales = scales; a.zeros = zeros; a.out = (__half*)out; a.ldo = ldo; a.M = (int)M; a.N = (int)N;
    a.ksteps = (int)((K + kW16K - 1) / kW16K);
    a.groups = (int)(K / kW16K);
    a.mtiles = (int)((M + p.NB - 1) / p.NB);
    a.ntiles = (int)((N + 127) / 128);
    a.slices = p.slices;
    a.part = reinterpret_cast<float*>(base + l.part);
    a.status = device_status_ptr();
    a.wait_ns = wait_limit_ns();
    RWKVQ_REQUIRE((int64_t)a.mtiles * a.ntiles * a.slices < (int64_t(1) << 30), RWKVQ_E_SHAPE, "%s: too many tiles", who);
    int32_t rc;
    const void* xb = x;
    int64_t ldxb = ldx;
    if (group) {
        __half* xp = reinterpret_cast<__half*>(base + l.xp);
        float* xsum = reinterpret_cast<float*>(base + l.xsum);
        a.xsum = xsum;
        const int kv = (int)(K / 8);
        int cpr = 1, lgP = 0;                            // CTAs per row: two CTAs per SM in all, 256+ vectors each
        while (M * cpr < 2 * (int64_t)sm_count() && cpr * 512 <= kv) cpr <<= 1;
        while (lgP < 2 && (cpr * 256 << lgP) < kv) ++lgP;
        const int64_t blocks = std::min<int64_t>(M, std::max<int64_t>(1, 6 * (int64_t)sm_count() / cpr)) * cpr;
        uint4* xz = p.pair ? reinterpret_cast<uint4*>(xsum) : nullptr;
        rc = x_dtype == RWKVQ_F16
                 ? launch_plain(wa16_prep_kernel<RWKVQ_F16>, blocks, st, who, (const uint16_t*)x, ldx, (int)M, kv, xp, xsum, xz, p.NB, a.groups, cpr, lgP)
                 : launch_plain(wa16_prep_kernel<RWKVQ_BF16>, blocks, st, who, (const uint16_t*)x, ldx, (int)M, kv, xp, xsum, xz, p.NB, a.groups, cpr, lgP);
        if (rc != RWKVQ_OK) return rc;
        xb = xp;
        ldxb = K;
    }
    if (p.pair) {
        W16PairCall c{};
        c.fmt = fmt; c.NB = p.NB; c.slices = p.slices; c.w = w; c.ldw = ldw; c.x = xb; c.ldx = ldxb; c.xz = a.xsum; c.scales = scales; c.zeros = zeros;
        c.out = (__half*)out; c.part = a.part; c.ldo = ldo; c.M = M; c.N = N; c.K = K;
        rc = run_wa16_pair(c, st, who);
    } else {
        W16Maps maps;
        rc = w16_map(&maps.w, w, N, group ? K / 2 : K, ldw, 128, group ? 64 : 128, who);
        if (rc != RWKVQ_OK) return rc;
        rc = w16_map(&maps.x, xb, M, K * 2, ldxb * 2, p.NB, 128, who);
        if (rc != RWKVQ_OK) return rc;
        if (group) {
            rc = p.NB == 32 ? launch_wa16<W16_INT4_GROUP, 32>(maps, a, st, who) : p.NB == 64 ? launch_wa16<W16_INT4_GROUP, 64>(maps, a, st, who)
                 : p.NB == 96 ? launch_wa16<W16_INT4_GROUP, 96>(maps, a, st, who) : launch_wa16<W16_INT4_GROUP, 128>(maps, a, st, who);
        } else {
            rc = p.NB == 32 ? launch_wa16<W16_INT8_TENSOR, 32>(maps, a, st, who) : p.NB == 64 ? launch_wa16<W16_INT8_TENSOR, 64>(maps, a, st, who)
                 : p.NB == 96 ? launch_wa16<W16_INT8_TENSOR, 96>(maps, a, st, who) : launch_wa16<W16_INT8_TENSOR, 128>(maps, a, st, who);
        }
    }
    if (rc != RWKVQ_OK || p.slices == 1) return rc;
    const int64_t per = (N & 3) == 0 ? 1024 : 256;
    return launch_plain(wa16_reduce_kernel, (M * N + per - 1) / per, st, who, (const float*)a.part, p.slices, (int)M, (int)N,
                        group ? (const float*)nullptr : scales, (__half*)out, ldo);
}

}  // namespace rwkvq

using namespace rwkvq;

extern "C" {

int32_t rwkvq_tc_gemm_wa16_form(int64_t M, int64_t N, int64_t K, int32_t bits) {
    if (M < 1 || N < 1 || K < 1 || (bits != 4 && bits != 8) || K % (bits == 4 ? kW16K : 16)) return 0;
    const W16Plan p = wa16_plan(bits == 4 ? W16_INT4_GROUP : W16_INT8_TENSOR, M, N, K);
    return p.slices * 1000 + (p.pair ? -p.NB : p.NB);
}

/* Bytes of workspace that the tensor-core weight-only GEMMs need for these sizes (256-byte aligned, contents irrelevant);
 * bits = 4 (group 128) or 8 (per tensor); 0: sizes these kernels do not take. */
int64_t rwkvq_tc_gemm_wa16_workspace_bytes(int64_t M, int64_t N, int64_t K, int32_t bits) {
    if (M < 1 || N < 1 || K < 1 || (bits != 4 && bits != 8) || K % (bits == 4 ? kW16K : 16)) return 0;
    return wa16_layout(bits == 4 ? W16_INT4_GROUP : W16_INT8_TENSOR, M, N, K, wa16_plan(bits == 4 ? W16_INT4_GROUP : W16_INT8_TENSOR, M, N, K)).total;
}

int32_t rwkvq_tc_gemm_int4_group(const void* x, int32_t x_dtype, int64_t ldx, const uint8_t* packed, int64_t ldw, const float* scales,
                                 const float* zeros, void* out_f16, int64_t ldo, int64_t M, int64_t N, int64_t K, void* workspace,
                                 int64_t workspace_bytes, void* stream) {
    return run_wa16(W16_INT4_GROUP, x, x_dtype, ldx, packed, ldw, scales, zeros, out_f16, ldo, M, N, K, workspace, workspace_bytes,
                    (cudaStream_t)stream, "tc_gemm_int4_group");
}

int32_t rwkvq_tc_gemm_int8_w8a16(const void* x_f16, int64_t ldx, const int8_t* w, int64_t ldw, const float* scale, void* out_f16, int64_t ldo,
                                 int64_t M, int64_t N, int64_t K, void* workspace, int64_t workspace_bytes, void* stream) {
    return run_wa16(W16_INT8_TENSOR, x_f16, RWKVQ_F16, ldx, w, ldw, scale, nullptr, out_f16, ldo, M, N, K, workspace, workspace_bytes,
                    (cudaStream_t)stream, "tc_gemm_int8_w8a16");
}

}  // extern "C"
