// NVFP4 (W4A4) GEMM for many tokens on CTA PAIRS: tcgen05.mma.cta_group::2 with block scales, 256 tokens x 256 weight rows a tile.
// Operands, scale factors and arithmetic are gemm_tc_nvfp4.cu's, which keeps the calls of fewer tokens and the pushed ones.
//
// Why pairs.  A stage (256 values of k) of a 128 x 256 tile on one CTA is 54 KB from L2 for 512 clocks of tensor-core work, more than
// an SM takes in: measured 0.40 us instead of 0.27.  In a pair each CTA loads its own 128 token rows, HALF of the weight rows and the
// scales of its tokens and of all 256 weight rows, 38 KB.  The leader's MMA reads both halves of the weight tile and
// accumulates each CTA's 128 x 256 block in that CTA's tensor memory; tcgen05.cp.cta_group::2 copies each CTA's scales from its own
// shared memory into its own tensor memory.  No load is multicast.
//
// The block-scaled accumulator takes 256 columns and the scales 128, so there is one accumulator and the next tile's MMAs wait for the
// epilogue: its eight warps read all their columns into registers before they convert or store anything.
//
// 2048 rows, us without the quantizer, one CTA -> pairs: [4096, 4096] 18.9 -> 17.0, [16384, 4096] 61.4 -> 52.6, [4096, 16384] 54.4 -> 47.9.  A stage takes 0.32 us:
// 38 KB at the 64 bytes a clock that an SM takes in.
#include <algorithm>
#include <cstdlib>

#include "tc_host.cuh"
#include "tc_pair.cuh"
#include "w8a8.cuh"

namespace rwkvq {
using namespace tc;

constexpr int kN2Threads = 320;
constexpr int kN2MaxStages = 5;
constexpr uint32_t kN2Tile = 128 * 128;                       // 128 rows x 128 bytes (256 values of k)
constexpr uint32_t kN2Stage = 2 * kN2Tile + 3 * kNfSfStage;   // tokens, half of the weight rows, scales of 128 tokens and of 256 weight rows
constexpr uint32_t kN2SfCol = 256;                            // first tensor-memory column of the scale factors

struct N2Maps {
    CUtensorMap a, w;          // packed codes, box 128 rows x 128 bytes
    CUtensorMap sfa, sfw;      // blocked scales as rows of 128 bytes, box 16 rows (one stage of a 128-row tile)
};
struct N2Args {
    const float* a_pts;
    const float* w_pts;
    __half* out;
    int64_t ldo;
    int M, N, kstages, ptiles, qtiles;
    int* status;
    unsigned long long wait_ns;
};
struct N2Shared {
    uint64_t full[kN2MaxStages], empty[kN2MaxStages], tfull, tempty;
    uint32_t tmem_base;
    int abort_flag;
};

__device__ __forceinline__ void n2_abort(N2Shared& s, const N2Args& a) {
    s.abort_flag = 1;
    if (a.status) atomicExch(a.status, RWKVQ_E_TIMEOUT);
}
__device__ __forceinline__ void tc_cp_sf_pair(uint32_t tmem_dst, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(desc) : "memory");
}
__device__ __forceinline__ void tc_mma_nvfp4_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t tsfa, uint32_t tsfb, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(tsfa), "r"(tsfb) : "memory");
}

__global__ void __launch_bounds__(kN2Threads, 1) gemm_tc2_nvfp4_kernel(const __grid_constant__ N2Maps maps, const N2Args a) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ N2Shared s;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = warp_uniform((int)(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();          // 0 = leader of the pair
    const int pair = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);
    const int total = a.ptiles * a.qtiles;

    griddep_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < kN2MaxStages; ++i) {
            mbar_init(&s.full[i], 1);                 // the leader's expect_tx arrival; both CTAs' bytes
            mbar_init(&s.empty[i], 1);                // one multicast commit per use
        }
        mbar_init(&s.tfull, 1);
        mbar_init(&s.tempty, 16);                     // eight epilogue warps of each CTA (used in the leader only)
        s.abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
        prefetch_tmap(&maps.a);
        prefetch_tmap(&maps.w);
        prefetch_tmap(&maps.sfa);
        prefetch_tmap(&maps.sfw);
    }
    if (warp == 1) tmem_alloc_pair(&s.tmem_base, 512);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();                               // the peer's barriers exist before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = warp_uniform(s.tmem_base);
    const volatile int* abort_flag = &s.abort_flag;

    if (warp == 0) {
        // ============================== TMA producer (both CTAs; the warp walks the loop, one lane issues) ==============================
        const bool issuer = elect_one();
        const int sfrow = a.kstages * 16;             // rows of 128 bytes that a 128-row tile's scales take
        auto fetch_w = [&](int qt, int kc, int st) {
            const uint32_t bar = smem_u32(&s.full[st]) & 0xFEFFFFFFu;      // the barrier of the even CTA
            uint8_t* dst = ring + (size_t)st * kN2Stage;
            if (rank == 0) mbar_expect_tx(&s.full[st], 2 * kN2Stage);
            tma_load_2d_pair(dst + kN2Tile, &maps.w, kc * 128, qt * 256 + (int)rank * 128, bar);
            tma_load_2d_pair(dst + 2 * kN2Tile + kNfSfStage, &maps.sfw, 0, (2 * qt) * sfrow + kc * 16, bar);
            tma_load_2d_pair(dst + 2 * kN2Tile + 2 * kNfSfStage, &maps.sfw, 0, (2 * qt + 1) * sfrow + kc * 16, bar);
        };
        // first pass over the ring: the weights and their scales do not depend on the kernels in front, so they are requested
        // before the dependency wait of programmatic dependent launch
        int npre = 0;
        for (int t = pair; t < total && npre < kN2MaxStages; t += npairs)
            for (int kc = 0; kc < a.kstages && npre < kN2MaxStages; ++kc, ++npre)
                if (issuer) fetch_w(t / a.ptiles, kc, npre);
        griddep_wait();                               // activation codes and scales come from the previous kernels
        RingPos rp;
        bool ok = true;
        for (int t = pair; t < total && ok; t += npairs) {
            const int pt = t % a.ptiles, qt = t / a.ptiles;       // token tiles fastest: the pairs running together share weight tiles
            for (int kc = 0; kc < a.kstages; ++kc, rp.next(kN2MaxStages)) {
                const int st = rp.i;
                const bool refill = --npre < 0;
                if (refill) ok = mbar_wait(&s.empty[st], rp.phase ^ 1, abort_flag, a.wait_ns);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { n2_abort(s, a); break; }
                if (issuer) {
                    if (refill) fetch_w(qt, kc, st);
                    const uint32_t bar = smem_u32(&s.full[st]) & 0xFEFFFFFFu;
                    uint8_t* dst = ring + (size_t)st * kN2Stage;
                    tma_load_2d_pair(dst, &maps.a, kc * 128, pt * 256 + (int)rank * 128, bar);
                    tma_load_2d_pair(dst + 2 * kN2Tile, &maps.sfa, 0, (2 * pt + (int)rank) * sfrow + kc * 16, bar);
                }
            }
        }
        if (ok && !(ok = pair_drain_ring(s.empty, rp, kN2MaxStages, abort_flag, a.wait_ns))) n2_abort(s, a);
        if (!ok) {      // give copies already in flight a bounded time to land before the CTA's memory is released
            const unsigned long long t0 = global_ns();
            while (global_ns() - t0 < 2000000ull) {}
        }
    } else if (warp == 1) {
        // ============================== MMA issuer (leader CTA only) ==============================
        if (rank == 0) {
            const bool issuer = elect_one();
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);       // e2m1 x e2m1, e4m3 scales, N = M = 256
            const uint32_t ring_addr = warp_uniform(smem_u32(ring));
            RingPos rp, fp;
            uint32_t n = 0;
            bool ok = true;
            for (int t = pair; t < total && ok; t += npairs, fp.next(1)) {
                ok = __all_sync(0xffffffffu, mbar_wait(&s.tempty, fp.phase ^ 1, abort_flag, a.wait_ns));
                if (!ok) { n2_abort(s, a); break; }
                tc_fence_after_sync();
                for (int kc = 0; kc < a.kstages; ++kc, ++n, rp.next(kN2MaxStages)) {
                    const int st = rp.i;
                    ok = __all_sync(0xffffffffu, mbar_wait(&s.full[st], rp.phase, abort_flag, a.wait_ns));
                    if (!ok) { n2_abort(s, a); break; }
                    tc_fence_after_sync();
                    const uint32_t sa = ring_addr + (uint32_t)st * kN2Stage, ssf = sa + 2 * kN2Tile;
                    // two alternating column sets, so a copy never lands in columns that the previous stage's MMAs may still read
                    const uint32_t tsfa = tmem_base + kN2SfCol + (n & 1) * 64, tsfb = tsfa + 16;
                    const uint64_t da = umma_desc_sw128(sa), db = umma_desc_sw128(sa + kN2Tile);
                    if (issuer) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            tc_cp_sf_pair(tsfa + k * 4, sf_desc(ssf + k * kNfSfChunk));
                            tc_cp_sf_pair(tsfb + k * 8, sf_desc(ssf + kNfSfStage + k * kNfSfChunk));
                            tc_cp_sf_pair(tsfb + k * 8 + 4, sf_desc(ssf + 2 * kNfSfStage + k * kNfSfChunk));
                        }
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tc_mma_nvfp4_pair(tmem_base, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, tsfa + k * 4, tsfb + k * 8, (kc > 0 || k > 0) ? 1u : 0u);
                        tc_commit_pair(&s.empty[st]);      // both CTAs may refill the stage once these MMAs have read it
                        if (kc == a.kstages - 1) tc_commit_pair(&s.tfull);     // both CTAs' epilogues
                    }
                }
            }
        }
    } else {
        // ============================== epilogue (both CTAs, each its own 128 token rows) ==============================
        griddep_wait();
        const int q = warp & 3, half = (warp - 2) >> 2;       // lane quarter; half of the tile's columns
        const float scale = a.a_pts[0] * a.w_pts[0];
        const bool vec16 = rows_vec16(a.out, a.ldo), vec32 = rows_vec32(a.out, a.ldo);
        const uint32_t leader_tempty = mapa_u32(smem_u32(&s.tempty), 0);
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + half * 128;
        RingPos fp;
        for (int t = pair; t < total; t += npairs, fp.next(1)) {
            const int pt = t % a.ptiles, qt = t / a.ptiles;
            const int m = pt * 256 + (int)rank * 128 + q * 32 + lane;
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&s.tfull, fp.phase, abort_flag, a.wait_ns));
            if (!ok) { n2_abort(s, a); break; }
            tc_fence_after_sync();
            uint32_t r[8][16];
#pragma unroll
            for (int i = 0; i < 8; ++i) tmem_ld16(taddr + i * 16, r[i]);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            mbar_arrive_cluster_relaxed(leader_tempty, lane);        // the accumulator may be overwritten
            if (m >= a.M) continue;
            __half* o = a.out + (int64_t)m * a.ldo;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int n0 = qt * 256 + half * 128 + i * 16;
                uint32_t h[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const __half2 hh = __floats2half2_rn(__uint_as_float(r[i][2 * j]) * scale, __uint_as_float(r[i][2 * j + 1]) * scale);
                    h[j] = *reinterpret_cast<const uint32_t*>(&hh);
                }
                store_f16x16(o + n0, h, a.N - n0, vec16, vec32);
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();      // both CTAs have read their last accumulator: the pair's tensor memory and the leader's barriers may go
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------------ host side
// Weight rows per tile of the single-CTA form (128 or 256), or 0 for pairs: the form with the least estimated time.  Fitted to 129 to
// 2048 rows of [4096, 4096], [16384, 4096], [4096, 16384], [10240, 2560], [2560, 10240], [8192, 2048], [2560, 2560], [1024, 1024] and [3072, 768], from a
// graph: a wave of tiles takes 0.29 us a stage + 0.3 (128 rows), 0.37 + 2.6 (256: the epilogue is exposed) and 0.32 + 1.7 (pairs), a
// launch 4.4 / 1.9 / 3.2 us besides.  Measured, us, 128 / 256 / pairs: [4096, 4096] 200 rows 8.1 / 9.8 / 9.6, 2048 rows 24.0 / 18.9 / 17.0; [16384,
// 4096] 2048 rows 73.1 / 61.4 / 52.6; [4096, 16384] 79.4 / 54.4 / 47.9; [10240, 2560] 33.0 / 30.8 / 23.1; [1024, 1024] 5.5 / 5.9 / 6.3.
int tc_nvfp4_form(int64_t M, int64_t N, int64_t K) {
    const int64_t sms = sm_count(), pairs = std::max<int64_t>(1, sms / 2), mt = (M + 127) / 128;
    const double st = (double)(K / 256);
    auto waves = [](int64_t tiles, int64_t units) { return (double)((tiles + units - 1) / units); };
    const double us128 = 4.4 + waves(mt * ((N + 127) / 128), sms) * (st * 0.289 + 0.3), us256 = 1.9 + waves(mt * ((N + 255) / 256), sms) * (st * 0.37 + 2.6);
    const double us2 = 3.2 + waves(((M + 255) / 256) * ((N + 255) / 256), pairs) * (st * 0.323 + 1.7);
    if (M > 128 && N > 128 && us2 <= us128 && us2 <= 0.95 * us256) return 0;  // up to 128 half of a pair's tile is empty
    return us256 < us128 ? 256 : 128;
}

// blocked scales [tiles][K / 64][512] as rows of 128 bytes; one box = the 2048 bytes of a stage
static int32_t n2_sf_map(CUtensorMap* m, const void* ptr, int64_t rows, int64_t K, const char* who) {
    EncodeTiledFn fn = encode_fn();
    RWKVQ_REQUIRE(fn != nullptr, RWKVQ_E_LAUNCH, "%s: cuTensorMapEncodeTiled is not available from the driver", who);
    const cuuint64_t dims[2] = {128, (cuuint64_t)((rows + 255) / 256 * 2 * (K / 64) * 4)};
    const cuuint64_t strides[1] = {128};
    const cuuint32_t box[2] = {128u, 16u};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    RWKVQ_REQUIRE(r == CUDA_SUCCESS, RWKVQ_E_LAUNCH, "%s: cuTensorMapEncodeTiled failed (%d)", who, (int)r);
    return RWKVQ_OK;
}

int32_t run_tc2_nvfp4(const uint8_t* a_codes, int64_t lda, const uint8_t* a_scales_blocked, const float* a_pts, const uint8_t* w_codes, int64_t ldw,
                      const uint8_t* w_scales_blocked, const float* w_tscale, __half* out, int64_t ldo, int64_t M, int64_t N, int64_t K, int* status,
                      cudaStream_t st, const char* who) {
    N2Args a{};
    a.a_pts = a_pts; a.w_pts = w_tscale; a.out = out; a.ldo = ldo; a.M = (int)M; a.N = (int)N;
    a.kstages = (int)(K / 256);
    a.ptiles = (int)((M + 255) / 256);
    a.qtiles = (int)((N + 255) / 256);
    a.status = status;
    a.wait_ns = wait_limit_ns();
    RWKVQ_REQUIRE((int64_t)a.ptiles * a.qtiles < (int64_t(1) << 30) && ((int64_t)std::max(a.ptiles, a.qtiles) * 2 + 2) * a.kstages * 16 < (int64_t(1) << 31),
                  RWKVQ_E_SHAPE, "%s: too many tiles", who);
    N2Maps maps;
    int32_t rc = make_map(&maps.a, a_codes, M, K / 2, lda, 128, who);
    if (rc) return rc;
    rc = make_map(&maps.w, w_codes, N, K / 2, ldw, 128, who);
    if (rc) return rc;
    rc = n2_sf_map(&maps.sfa, a_scales_blocked, M, K, who);
    if (rc) return rc;
    rc = n2_sf_map(&maps.sfw, w_scales_blocked, N, K, who);
    if (rc) return rc;
    const size_t smem = (size_t)kN2MaxStages * kN2Stage + 1024;
    rc = ensure_smem_optin(reinterpret_cast<const void*>(gemm_tc2_nvfp4_kernel), (int)smem, who);
    if (rc) return rc;
    const int64_t pairs = std::min<int64_t>(std::max(1, sm_count() / 2), (int64_t)a.ptiles * a.qtiles);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(kN2Threads);
    cfg.dynamicSmemBytes = smem;
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
    const cudaError_t err = cudaLaunchKernelEx(&cfg, gemm_tc2_nvfp4_kernel, maps, a);
    if (err != cudaSuccess) {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return fail(RWKVQ_E_LAUNCH, "%s: %s", who, cudaGetErrorString(err));
    }
    return check_launch(who);
}

}  // namespace rwkvq
