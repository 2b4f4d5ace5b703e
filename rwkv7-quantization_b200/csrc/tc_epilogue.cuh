// Epilogue of the tiled W8A8 GEMMs (gemm_tc.cu, gemm_tc2.cu): accumulator columns of one token row -> scaled fp16.
//
// With one or two waves of tiles the last tile's epilogue is exposed at the end of the launch, so it is written for its own
// latency: what a tile needs is decided once per tile (EPI), not per pair of columns -- the run-time tests for relu^2 and
// per-row scales kept the loads of one 16-column step from starting before the stores of the one before --, two
// tensor-memory loads are under way, and eight warps share a tile (two per lane quarter, half of the columns each).
// Measured, us, before -> after (GEMM alone): FP8 [4096, 4096] 717 rows 20.4 -> 16.3, [2560, 2560] 1024 rows 16.1 -> 12.7, [16384,
// 4096] 256 rows 26.6 -> 22.4; INT8 22.9 -> 15.5, 18.7 -> 12.0, 27.8 -> 20.9.
#pragma once

#include "tc_common.cuh"
#include "w8a8.cuh"

namespace rwkvq {

enum { EPI_PLAIN = 0, EPI_BF16 = 1, EPI_RELU2 = 2, EPI_RELU2_BF16 = 3, EPI_ANY = 4 };

struct EpiRow {
    float rowscale, actscale;      // activation scale times the matrix's weight scale; activation scale alone (per-row weight scales)
    const float* ws;
    __half* out;                   // this token's row of the result
    int32_t* acc;                  // INT8: this token's row of raw accumulators, or null (EPI_ANY only)
    int N;
    bool live, vec_ok, vec32;      // the token exists; 16- / 32-byte stores are possible
    uint32_t flags;
};

// columns [n0, n0 + 16) of the result from the accumulator values r; hmax: running maximum of the relu^2 results
template <int KIND, int EPI>
__device__ __forceinline__ void epi_convert16(const EpiRow& e, const uint32_t (&r)[16], int n0, uint32_t (&h)[8], float& hmax) {
    const bool via = EPI == EPI_BF16 || EPI == EPI_RELU2_BF16 || (EPI == EPI_ANY && (e.flags & RWKVQ_FLAG_OUT_VIA_BF16));
    const bool relu2 = EPI == EPI_RELU2 || EPI == EPI_RELU2_BF16 || (EPI == EPI_ANY && (e.flags & RWKVQ_FLAG_RELU2));
    const bool per_row = EPI == EPI_ANY && (e.flags & RWKVQ_FLAG_WSCALE_PER_ROW);
    const bool hmax_bf16 = (e.flags & RWKVQ_FLAG_AMAX_AFTER_BF16) != 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        float s0 = e.rowscale, s1 = e.rowscale;
        if (per_row) {
            s0 = e.actscale * e.ws[min(n0 + 2 * j, e.N - 1)];
            s1 = e.actscale * e.ws[min(n0 + 2 * j + 1, e.N - 1)];
        }
        float2 f;
        if constexpr (KIND == tc::KIND_F8) f = make_float2(__uint_as_float(r[2 * j]) * s0, __uint_as_float(r[2 * j + 1]) * s1);
        else f = make_float2((float)(int32_t)r[2 * j] * s0, (float)(int32_t)r[2 * j + 1] * s1);
        if (via) f = bf16_round2(f);
        __half2 hh = __floats2half2_rn(f.x, f.y);
        if (relu2) {
            // the engine's relu_square on the fp16 result, fp32 arithmetic; its maximum (over the bf16-rounded values where the
            // consumer takes its amax there) goes to the projection that follows
            const float2 y = __half22float2(hh);
            const float v0 = y.x < 0.f ? 0.f : y.x, v1 = y.y < 0.f ? 0.f : y.y;      // NaN stays NaN, as in a relu of its own
            hh = __floats2half2_rn(v0 * v0, v1 * v1);
            float2 hv = __half22float2(hh);
            if (hmax_bf16) hv = bf16_round2(hv);
            if (n0 + 2 * j < e.N) hmax = fmaxf(hmax, hv.x);
            if (n0 + 2 * j + 1 < e.N) hmax = fmaxf(hmax, hv.y);
        }
        h[j] = *reinterpret_cast<const uint32_t*>(&hh);
    }
}

template <int KIND, int EPI>
__device__ __forceinline__ void epi_store16(const EpiRow& e, const uint32_t (&r)[16], int n0, float& hmax) {
    if (!e.live || n0 >= e.N) return;
    uint32_t h[8];
    epi_convert16<KIND, EPI>(e, r, n0, h, hmax);
    store_f16x16(e.out + n0, h, e.N - n0, e.vec_ok, e.vec32);
    if constexpr (KIND == tc::KIND_I8 && EPI == EPI_ANY) {
        if (e.acc) {
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (n0 + j < e.N) e.acc[n0 + j] = (int32_t)r[j];
        }
    }
}

// `cols` accumulator columns (a multiple of 32, with ODD of 16) at taddr, result columns from n0 on
template <int KIND, int EPI, bool ODD>
__device__ __forceinline__ void epi_cols(const EpiRow& e, uint32_t taddr, int n0, int cols, float& hmax) {
#pragma unroll 1
    for (int c0 = 0; c0 < cols; c0 += 32) {
        uint32_t r0[16], r1[16];
        const bool two = !ODD || c0 + 16 < cols;
        tc::tmem_ld16(taddr + c0, r0);
        if (two) tc::tmem_ld16(taddr + c0 + 16, r1);
        tc::tmem_ld_wait();
        epi_store16<KIND, EPI>(e, r0, n0 + c0, hmax);
        if (two) epi_store16<KIND, EPI>(e, r1, n0 + c0 + 16, hmax);
    }
}

template <int KIND, bool ODD = false>
__device__ __forceinline__ void epi_tile(const EpiRow& e, uint32_t taddr, int n0, int cols, float& hmax) {
    const bool any = (e.flags & RWKVQ_FLAG_WSCALE_PER_ROW) || (KIND == tc::KIND_I8 && e.acc);
    const bool via = (e.flags & RWKVQ_FLAG_OUT_VIA_BF16) != 0, relu2 = (e.flags & RWKVQ_FLAG_RELU2) != 0;
    if (any) epi_cols<KIND, EPI_ANY, ODD>(e, taddr, n0, cols, hmax);
    else if (relu2 && via) epi_cols<KIND, EPI_RELU2_BF16, ODD>(e, taddr, n0, cols, hmax);
    else if (relu2) epi_cols<KIND, EPI_RELU2, ODD>(e, taddr, n0, cols, hmax);
    else if (via) epi_cols<KIND, EPI_BF16, ODD>(e, taddr, n0, cols, hmax);
    else epi_cols<KIND, EPI_PLAIN, ODD>(e, taddr, n0, cols, hmax);
}

}  // namespace rwkvq
