// W8A8 GEMM for many tokens on CTA PAIRS: tcgen05.mma.cta_group::2 (two SMs work on one tile of 256 tokens x bn weight rows,
// bn = 128 to 256, see tc2_tile).
//
// Why pairs.  With one CTA per 128 x 256 tile (gemm_tc.cu) every 128-byte step of K needs 48 KB of operands from L2
// per SM for 512 cycles of tensor-core work -- 96 bytes per clock, more than an SM gets from L2, so the tensor pipe
// idles a third of the time.  In a pair each CTA loads its own 128 token rows and only HALF of the bn weight rows (bn = 256:
// 32 KB per step per SM, 64 bytes per clock; bn = 128: 24 KB for half the work, 96 again, taken where it fills a wave); the MMA
// issued by the pair's leader reads both halves of the weight tile from the two CTAs' shared memory and accumulates each CTA's
// 128 x bn block in that CTA's own tensor memory.
// No multicast is involved: every TMA load lands in the shared memory of the CTA that issued it.
//
// Roles per CTA as in gemm_tc.cu: warp 0 = TMA producer, warp 1 = tensor-memory owner and -- in the leader CTA only --
// MMA issuer (one elected lane each), warps 2-9 = epilogue (tc_epilogue.cuh).  Barriers: full[] lives in the leader (both producers' bytes are
// counted there: the loads carry .cta_group::2 and name the leader's barrier), empty[] and tfull[] are signalled in both
// CTAs at once by a multicast tcgen05.commit, tempty[] of the leader collects the arrivals of both CTAs' epilogue warps.
// Every wait is bounded; the producers wait for the last commits and the pair meets at a cluster barrier before the tensor memory is
// released.
#include <algorithm>
#include <cstdlib>

#include "tc_common.cuh"
#include "tc_epilogue.cuh"
#include "tc_host.cuh"
#include "tc_pair.cuh"
#include "w8a8.cuh"

namespace rwkvq {
using namespace tc;

constexpr int kT2Threads = 320;
constexpr int kT2MaxStages = 6;
constexpr int kT2Chunk = 128;                 // bytes of K per stage
constexpr int kT2Rows = 128;                  // rows of each operand tile per CTA
constexpr uint32_t kT2TileBytes = kT2Rows * kT2Chunk;      // 16 KB
constexpr uint32_t kT2StageBytes = 2 * kT2TileBytes;       // tokens + this CTA's half of the weight tile
constexpr int kT2N = 256;                     // most weight rows per pair tile (the instruction's N)

struct Tc2Maps {
    CUtensorMap a[3];   // activation codes [M, K], box 128 rows x 128 bytes
    CUtensorMap w[3];   // weights [N, K], box bn / 2 rows x 128 bytes
};

struct Tc2Args {
    const float* a_scale[3];   // FP8 amax-or-scale [1]; INT8 row scales [M]
    const float* ws[3];        // weight scale: one value, or N with RWKVQ_FLAG_WSCALE_PER_ROW
    __half* out[3];
    int32_t* acc[3];           // INT8: optional raw accumulators
    float* ffn_amax;           // RWKVQ_FLAG_RELU2: maximum of the relu^2 results -- FP8: one word; INT8: one per token row
    int* status;
    unsigned long long wait_ns;
    int64_t ldo, ldacc;
    int M, N, K, nmat;
    int bn;                                   // weight rows per tile: a multiple of 16 (FP8) or 32 (INT8) from 128 to 256
    int kchunks, ptiles, qtiles, stages;      // ptiles: 256-token pair tiles, qtiles: weight tiles
    int div_mode, amax_is_amax;
    uint32_t flags;
};

struct Tc2Shared {
    uint64_t full[kT2MaxStages], empty[kT2MaxStages], tfull[2], tempty[2], done;
    uint32_t tmem_base;
    int abort_flag;
};

template <int KIND>
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (KIND == KIND_F8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
    }
}

__device__ __forceinline__ void t2_abort(Tc2Shared& s, const Tc2Args& a) {
    s.abort_flag = 1;
    if (a.status) atomicExch(a.status, RWKVQ_E_TIMEOUT);
}

template <int KIND>
__global__ void __launch_bounds__(kT2Threads, 1) gemm_tc2_kernel(const __grid_constant__ Tc2Maps maps, const Tc2Args a) {
    using T = typename Acc<KIND == KIND_F8 ? QT_FP8 : QT_INT8>::T;
    extern __shared__ uint8_t smem_raw[];
    __shared__ Tc2Shared s;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = warp_uniform((int)(threadIdx.x >> 5)), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();          // 0 = leader of the pair
    const int pair = (int)(blockIdx.x >> 1), npairs = (int)(gridDim.x >> 1);
    const int per_mat = a.ptiles * a.qtiles, total = a.nmat * per_mat;
    constexpr uint32_t kCols = 512;                   // two 256-column accumulators

    griddep_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < a.stages; ++i) {
            mbar_init(&s.full[i], 1);                 // the leader's expect_tx arrival; both CTAs' bytes
            mbar_init(&s.empty[i], 1);                // one multicast commit per use
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s.tfull[i], 1);
            mbar_init(&s.tempty[i], 16);              // eight epilogue warps of each CTA (used in the leader only)
        }
        mbar_init(&s.done, 8);
        s.abort_flag = 0;
        fence_barrier_init();
        fence_proxy_async();
        for (int i = 0; i < a.nmat; ++i) {
            prefetch_tmap(&maps.a[i]);
            prefetch_tmap(&maps.w[i]);
        }
    }
    if (warp == 1) tmem_alloc_pair(&s.tmem_base, kCols);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();                               // the peer's barriers exist before anything signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = warp_uniform(s.tmem_base);
    const volatile int* abort_flag = &s.abort_flag;
    const int wrows = a.bn >> 1;                      // weight rows of a tile that this CTA loads
    const uint32_t tx = 2 * (kT2TileBytes + (uint32_t)wrows * kT2Chunk);      // the four tiles of the pair

    auto tile_rows = [&](int t, int& mrow, int& nrow) {       // token tiles fastest: the pairs running together share weight tiles
        const int mat = (t >= per_mat) + (t >= 2 * per_mat);
        t -= mat * per_mat;
        mrow = (t % a.ptiles) * 256;
        nrow = (t / a.ptiles) * a.bn;
        return mat;
    };

    if (warp == 0) {
        // ============================== TMA producer (both CTAs; the warp walks the loop, one lane issues) ==============================
        {
            const bool issuer = elect_one();
            // first pass over the ring: the weights do not depend on the kernel in front, so they are requested before the
            // dependency wait of programmatic dependent launch
            int npre = 0;
            for (int t = pair; t < total && npre < a.stages; t += npairs) {
                int mrow, nrow;
                const int mat = tile_rows(t, mrow, nrow);
                for (int kc = 0; kc < a.kchunks && npre < a.stages; ++kc, ++npre) {
                    if (!issuer) continue;
                    if (rank == 0) mbar_expect_tx(&s.full[npre], tx);
                    tma_load_2d_pair(ring + (size_t)npre * kT2StageBytes + kT2TileBytes, &maps.w[mat], kc * kT2Chunk, nrow + (int)rank * wrows,
                                     smem_u32(&s.full[npre]) & 0xFEFFFFFFu);
                }
            }
            griddep_wait();                           // the activation codes come from the previous kernel
            RingPos rp;
            bool ok = true;
            for (int t = pair; t < total && ok; t += npairs) {
                int mrow, nrow;
                const int mat = tile_rows(t, mrow, nrow);
                for (int kc = 0; kc < a.kchunks; ++kc, rp.next(a.stages)) {
                    const int st = rp.i;
                    const bool refill = --npre < 0;
                    if (refill) ok = mbar_wait(&s.empty[st], rp.phase ^ 1, abort_flag, a.wait_ns);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { t2_abort(s, a); break; }
                    uint8_t* dst = ring + (size_t)st * kT2StageBytes;
                    if (issuer) {
                        const uint32_t leader_bar = smem_u32(&s.full[st]) & 0xFEFFFFFFu;         // the barrier of the even CTA
                        if (refill) {
                            if (rank == 0) mbar_expect_tx(&s.full[st], tx);
                            tma_load_2d_pair(dst + kT2TileBytes, &maps.w[mat], kc * kT2Chunk, nrow + (int)rank * wrows, leader_bar);
                        }
                        tma_load_2d_pair(dst, &maps.a[mat], kc * kT2Chunk, mrow + (int)rank * kT2Rows, leader_bar);
                    }
                }
            }
            if (ok && !(ok = pair_drain_ring(s.empty, rp, a.stages, abort_flag, a.wait_ns))) t2_abort(s, a);
            if (!ok) {      // give copies already in flight a bounded time to land before the CTA's memory is released
                const unsigned long long t0 = global_ns();
                while (global_ns() - t0 < 2000000ull) {}
            }
        }
    } else if (warp == 1) {
        // ============================== MMA issuer (leader CTA only) ==============================
        if (rank == 0) {
            const bool issuer = elect_one();
            const uint32_t idesc = umma_idesc(KIND, 256, a.bn), ring_addr = warp_uniform(smem_u32(ring));
            RingPos rp, fp;                                // ring stage, accumulator
            bool ok = true;
            for (int t = pair; t < total && ok; t += npairs, fp.next(2)) {
                ok = __all_sync(0xffffffffu, mbar_wait(&s.tempty[fp.i], fp.phase ^ 1, abort_flag, a.wait_ns));
                if (!ok) { t2_abort(s, a); break; }
                tc_fence_after_sync();
                const uint32_t d = tmem_base + (uint32_t)(fp.i * kT2N);
                for (int kc = 0; kc < a.kchunks; ++kc, rp.next(a.stages)) {
                    const int st = rp.i;
                    ok = __all_sync(0xffffffffu, mbar_wait(&s.full[st], rp.phase, abort_flag, a.wait_ns));
                    if (!ok) { t2_abort(s, a); break; }
                    tc_fence_after_sync();
                    const uint32_t sa = ring_addr + (uint32_t)st * kT2StageBytes;
                    const uint64_t da = umma_desc_sw128(sa), db = umma_desc_sw128(sa + kT2TileBytes);
                    if (issuer) {
#pragma unroll
                        for (int k = 0; k < kT2Chunk / 32; ++k)
                            tc_mma_pair<KIND>(d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kc > 0 || k > 0) ? 1u : 0u);
                        tc_commit_pair(&s.empty[st]);      // both CTAs may refill the stage once these MMAs have read it
                        if (kc == a.kchunks - 1) tc_commit_pair(&s.tfull[fp.i]);     // both CTAs' epilogues
                    }
                }
            }
        }
    } else {
        // ============================== epilogue (both CTAs, each its own 128 token rows) ==============================
        griddep_wait();
        const int q = warp & 3;                         // tensor-memory lane quarter this warp may read
        const int c0 = warp < 6 ? 0 : ((a.bn + 31) >> 5) << 4, cols = warp < 6 ? ((a.bn + 31) >> 5) << 4 : a.bn - c0;     // its columns of the tile
        const int row_l = q * 32 + lane;
        const uint32_t leader_tempty[2] = {mapa_u32(smem_u32(&s.tempty[0]), 0), mapa_u32(smem_u32(&s.tempty[1]), 0)};
        RingPos fp;
        for (int t = pair; t < total; t += npairs, fp.next(2)) {
            int mrow, nrow;
            const int mat = tile_rows(t, mrow, nrow);
            const int m = mrow + (int)rank * kT2Rows + row_l;
            // what the tile needs from global memory is fetched while its MMAs still run
            EpiRow e;
            if constexpr (KIND == KIND_F8) {
                const float am = a.a_scale[mat][0];
                e.actscale = a.amax_is_amax ? div_mode_f32(fmaxf(am, 1e-12f), 448.f, a.div_mode) : am;
            } else {
                e.actscale = m < a.M ? a.a_scale[mat][m] : 0.f;
            }
            e.ws = a.ws[mat];
            e.rowscale = e.actscale * e.ws[0];
            e.out = a.out[mat] + (int64_t)m * a.ldo;
            e.acc = KIND == KIND_I8 && a.acc[mat] ? a.acc[mat] + (int64_t)m * a.ldacc : nullptr;
            e.N = a.N;
            e.live = m < a.M;
            e.vec_ok = rows_vec16(a.out[mat], a.ldo);
            e.vec32 = rows_vec32(a.out[mat], a.ldo);
            e.flags = a.flags;
            if (!mbar_wait(&s.tfull[fp.i], fp.phase, abort_flag, a.wait_ns)) { t2_abort(s, a); break; }
            tc_fence_after_sync();
            float hmax = 0.f;
            epi_tile<KIND, true>(e, tmem_base + (uint32_t)(fp.i * kT2N) + ((uint32_t)(q * 32) << 16) + c0, nrow + c0, cols, hmax);
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_tempty[fp.i]);       // this accumulator may be overwritten
            if (a.flags & RWKVQ_FLAG_RELU2) {
                if constexpr (KIND == KIND_F8) {
                    hmax = warp_max(hmax);
                    if (lane == 0 && hmax > 0.f) atomic_max_nonneg(a.ffn_amax, hmax);
                } else {                                 // INT8 scales its activations per row
                    if (m < a.M && hmax > 0.f) atomic_max_nonneg(a.ffn_amax + m, hmax);
                }
            }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s.done);
    }

    __syncwarp();            // single-lane roles: the other lanes wait here for their lane 0
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        if (!mbar_wait(&s.done, 0, abort_flag, a.wait_ns)) t2_abort(s, a);     // this CTA's epilogue has read its last accumulator
    }
    cluster_sync_all();      // ... and so has the peer's: the pair's tensor memory (and the leader's barriers) may go
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, kCols);
    }
}

// ------------------------------------------------------------------------------------------------ host side
static int t2_grid_pairs() { return std::max(1, sm_count() / 2); }

// Weight rows per pair tile.  A tile of 256 leaves pairs idle wherever the tiles are not a multiple of the pairs: [4096, 4096] at 717
// rows is 48 tiles for 74 pairs, [2560, 10240] at 2048 rows 80.  tcgen05.mma.cta_group::2 with 256 rows takes N in steps of 16 for
// kind::f8f6f4 and of 32 for kind::i8; of these widths the one with the least estimated time is taken: a 128-byte step of K takes 0.094 us +
// 0.00073 a row, a launch 3.2 us + 0.009 a row and up to 1.6 where all SMs store their results.  Measured, us, tiles of 256 / the tile
// taken, FP8: [4096, 4096] 717 rows 15.5 / 12.8 (176), [4096, 16384] 717 rows 44.3 / 36.0, [2560, 10240] 1000 rows 29.6 / 19.4 (144), 2048 rows
// 50.7 / 35.7, [2560, 2560] 2048 rows 16.2 / 13.5, [16384, 4096] 717 rows 36.3 / 35.2 (224).  INT8: 15.1 / 12.8 (192), 42.5 / 34.7, 28.6 / 19.6 (160),
// 49.8 / 34.4, 15.8 / 12.8, 37.5 / 34.9 (224).
struct T2Tile { int bn; double us; };
static bool t2_forced() {
    static const bool force = std::getenv("RWKVQ_TC2") && std::getenv("RWKVQ_TC2")[0] == 'f';
    return force;
}
static T2Tile tc2_tile(int kind, int64_t M, int64_t N, int64_t K, int nmat) {
    const int step = kind == KIND_I8 ? 32 : 16;
    const char* bn_env = t2_forced() ? std::getenv("RWKVQ_TC2_BN") : nullptr;      // read per call: a test switches tiles in one process
    const int forced = bn_env ? std::atoi(bn_env) : 0;
    const int64_t pairs = t2_grid_pairs(), pt = nmat * ((M + 255) / 256);
    const double kc = (double)((K + kT2Chunk - 1) / kT2Chunk), inv_pairs = 1.0 / (double)pairs;
    T2Tile best{0, 0.};
    for (int bn = kT2N; bn >= 128; bn -= step) {                 // on the path of every call: one short division a width where all tiles run at once
        if (forced >= 128 && forced <= kT2N && forced % step == 0 && bn != forced) continue;
        const int64_t tiles = pt * (int64_t)(((uint32_t)N + (uint32_t)bn - 1) / (uint32_t)bn);      // N < 2^30
        const int64_t waves = tiles <= pairs ? 1 : (tiles + pairs - 1) / pairs;
        const double us = 3.15 + 0.009 * bn + 1.6 * std::min(1.0, (double)tiles * inv_pairs) + (double)waves * kc * (0.094 + 0.000731 * bn);
        if (best.bn == 0 || us < best.us) best = {bn, us};
    }
    return best;
}
// RWKVQ_TC2=0 switches the pairs off, =force uses them wherever they are legal, RWKVQ_TC2_MIN_M raises their first row count (129: below it a pair tile is half empty).
// Pairs or single CTAs?  The estimate above against that of the single form: 3.3 / 4.0 / 3.5 us and 0.37 / 0.22 / 0.19 a step with 256 / 128 /
// 64 weight rows per tile.  Measured, us, single / pairs: FP8 [16384, 4096] 384 rows 26.9 / 24.0, 2048 rows 93.6 / 84.6; [4096, 16384] 717 rows 49.4 /
// 35.9; [4096, 4096] 1000 rows 15.6 / 16.3; [8192, 2048] 384 rows 10.2 / 11.3, 2048 rows 28.3 / 25.3; [2560, 2560] 1500 rows 11.5 / 11.9.
bool tc2_eligible(int kind, int64_t M, int64_t N, int64_t K, int nmat, int single_nb) {
    static const int64_t min_m = [] {
        const char* off = std::getenv("RWKVQ_TC2");
        if (off && off[0] == '0') return (int64_t)1 << 62;
        const char* e = std::getenv("RWKVQ_TC2_MIN_M");
        const long long v = e ? std::atoll(e) : 129;
        return (int64_t)std::max<long long>(v, 129);
    }();
    if (M < min_m || N < kT2N || K % 16 || (kind != KIND_F8 && kind != KIND_I8)) return false;
    if (t2_forced()) return true;
    const int64_t pairs = t2_grid_pairs();
    const int64_t single = nmat * ((M + 127) / 128) * ((N + single_nb - 1) / single_nb);
    const double kc = (double)((K + kT2Chunk - 1) / kT2Chunk), step1 = single_nb > 128 ? 0.369 : (single_nb > 64 ? 0.218 : 0.193);
    const double t2 = tc2_tile(kind, M, N, K, nmat).us, t1 = (single_nb > 128 ? 3.3 : (single_nb > 64 ? 4.0 : 3.5)) + (double)((single + 2 * pairs - 1) / (2 * pairs)) * kc * step1;
    return t2 <= t1;
}

int tc2_width(int kind, int64_t M, int64_t N, int64_t K, int nmat) { return tc2_tile(kind, M, N, K, nmat).bn; }

int32_t run_tc2(const Tc2Call& c, int* status, cudaStream_t st, const char* who) {
    Tc2Args a{};
    const int kind = c.kind;
    a.ffn_amax = c.ffn_amax; a.status = status; a.wait_ns = wait_limit_ns();
    a.ldo = c.ldo; a.ldacc = c.ldacc; a.M = c.M; a.N = c.N; a.K = c.K; a.nmat = c.nmat; a.div_mode = c.div_mode; a.amax_is_amax = c.amax_is_amax; a.flags = c.flags;
    a.kchunks = (c.K + kT2Chunk - 1) / kT2Chunk;
    a.bn = tc2_tile(c.kind, c.M, c.N, c.K, c.nmat).bn;
    a.ptiles = (c.M + 255) / 256;
    a.qtiles = (c.N + a.bn - 1) / a.bn;
    a.stages = kT2MaxStages;
    const size_t smem = (size_t)a.stages * kT2StageBytes + 1024;
    Tc2Maps maps;
    int32_t rc;
    for (int i = 0; i < c.nmat; ++i) {
        a.a_scale[i] = c.a_scale[i]; a.ws[i] = c.ws[i]; a.out[i] = c.out[i]; a.acc[i] = c.acc[i];
        rc = make_map(&maps.a[i], c.codes[i], c.M, c.K, c.lda, kT2Rows, who);
        if (rc) return rc;
        rc = make_map(&maps.w[i], c.w[i], c.N, c.K, c.ldw, a.bn / 2, who);
        if (rc) return rc;
    }
    const void* kern = kind == KIND_F8 ? (const void*)gemm_tc2_kernel<KIND_F8> : (const void*)gemm_tc2_kernel<KIND_I8>;
    rc = ensure_smem_optin(kern, (int)smem, who);
    if (rc) return rc;
    const int pairs = (int)std::min<int64_t>(t2_grid_pairs(), (int64_t)a.nmat * a.ptiles * a.qtiles);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(kT2Threads);
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
    const cudaError_t err = kind == KIND_F8 ? cudaLaunchKernelEx(&cfg, gemm_tc2_kernel<KIND_F8>, maps, a)
                                            : cudaLaunchKernelEx(&cfg, gemm_tc2_kernel<KIND_I8>, maps, a);
    if (err != cudaSuccess) {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return fail(RWKVQ_E_LAUNCH, "%s: %s", who, cudaGetErrorString(err));
    }
    return check_launch(who);
}

}  // namespace rwkvq
