// Whole projections in one boundary crossing: the activation quantizer and the GEMM behind it (single matrix or r/k/v), and
// the FFN pair of many rows.  Host code only: the kernels are those of the entries called here, in the same order on the
// same stream, so the results are the same bits.
//
// Why.  From 9 rows on a projection is two launches (the FFN pair four), and from Python each crossing costs the
// marshalling of some 20 arguments plus an allocation per intermediate: 193 us for the three calls of a layer at 201
// rows of width 2560, whose kernels take about 60.  Here a call packs one descriptor and one scratch buffer carries the
// intermediates: 94 us.
#include "common.cuh"

using namespace rwkvq;

namespace {
int64_t up256(int64_t v) { return (v + 255) / 256 * 256; }
}  // namespace

extern "C" {

int64_t rwkvq_linear_scratch_bytes(int32_t kind, int32_t nmat, int64_t M, int64_t K) {
    if (nmat < 1 || nmat > 3 || M < 0 || K < 0 || (kind != RWKVQ_LINEAR_FP8 && kind != RWKVQ_LINEAR_INT8)) return 0;
    return nmat * up256(M * K) + (kind == RWKVQ_LINEAR_FP8 ? 256 : nmat * up256(4 * M));
}

int32_t rwkvq_linear(const rwkvq_linear_desc* d) {
    const char* who = "linear";
    RWKVQ_REQUIRE(d != nullptr, RWKVQ_E_BADARG, "%s: null descriptor", who);
    const bool fp8 = d->kind == RWKVQ_LINEAR_FP8;
    RWKVQ_REQUIRE((fp8 || d->kind == RWKVQ_LINEAR_INT8) && (d->nmat == 1 || d->nmat == 3), RWKVQ_E_BADARG, "%s: kind %d, %d matrices", who, d->kind, d->nmat);
    RWKVQ_REQUIRE(d->M > 0 && d->N >= 0 && d->K > 0 && d->M < (int64_t(1) << 30) && d->K < (int64_t(1) << 30), RWKVQ_E_SHAPE, "%s: M=%lld K=%lld", who,
                  (long long)d->M, (long long)d->K);
    RWKVQ_REQUIRE(d->scratch && ((uintptr_t)d->scratch & 255) == 0 && d->scratch_bytes >= rwkvq_linear_scratch_bytes(d->kind, d->nmat, d->M, d->K),
                  RWKVQ_E_WORKSPACE, "%s: %lld bytes of 256-byte aligned scratch needed", who, (long long)rwkvq_linear_scratch_bytes(d->kind, d->nmat, d->M, d->K));
    RWKVQ_REQUIRE(!d->relu2 || (d->nmat == 1 && d->x_dtype == RWKVQ_F16), RWKVQ_E_BADARG, "%s: relu2 takes one matrix and fp16 rows", who);
    uint8_t* c[3] = {nullptr, nullptr, nullptr};
    const int64_t M = d->M, N = d->N, K = d->K, cb = up256(M * K);
    for (int i = 0; i < d->nmat; ++i) c[i] = reinterpret_cast<uint8_t*>(d->scratch) + i * cb;
    float* sc = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(d->scratch) + d->nmat * cb);
    int32_t rc;
    if (fp8) {
        float* scale = d->by_scale ? sc + 4 : nullptr;                 // linear_fp8: the quantizer's own scale, not amax / 448
        const float* a = d->by_scale ? sc + 4 : sc;
        const int32_t is_amax = d->by_scale ? 0 : 1;
        if (d->nmat == 1) {
            rc = d->relu2 ? rwkvq_actq_fp8_relu2(d->x[0], M, K, d->ldx, c[0], K, sc, scale, d->act_div, d->act_flags, d->stream)
                          : rwkvq_actq_fp8_fused(d->x[0], d->x_dtype, M, K, d->ldx, c[0], K, sc, scale, d->actq_scratch, d->actq_scratch_bytes, nullptr,
                                                 d->act_div, d->act_flags, d->stream);
            if (rc != RWKVQ_OK) return rc;
            const uint8_t* w = (const uint8_t*)d->w[0];
            return d->decode ? rwkvq_gemm_fp8(c[0], K, a, is_amax, w, d->ldw, d->w_scale[0], d->out[0], d->ldo, M, N, K, d->gemm_div, d->gemm_flags, d->stream)
                             : rwkvq_tc_gemm_fp8(c[0], K, a, is_amax, w, d->ldw, d->w_scale[0], d->out[0], d->ldo, M, N, K, d->gemm_div, d->gemm_flags,
                                                 d->workspace, d->workspace_bytes, d->stream);
        }
        RWKVQ_REQUIRE(!d->by_scale, RWKVQ_E_BADARG, "%s: by_scale takes one matrix", who);
        rc = rwkvq_actq_fp8_fused3(d->x[0], d->x[1], d->x[2], d->x_dtype, M, K, d->ldx, c[0], c[1], c[2], K, sc, d->actq_scratch, d->actq_scratch_bytes, nullptr,
                                   d->act_div, d->act_flags, d->stream);
        if (rc != RWKVQ_OK) return rc;
        const uint8_t *w0 = (const uint8_t*)d->w[0], *w1 = (const uint8_t*)d->w[1], *w2 = (const uint8_t*)d->w[2];
        return d->decode ? rwkvq_gemm_fp8_rkv(c[0], c[1], c[2], K, sc, 1, w0, w1, w2, d->ldw, d->w_scale[0], d->w_scale[1], d->w_scale[2], d->out[0], d->out[1],
                                              d->out[2], d->ldo, M, N, K, d->gemm_div, d->gemm_flags, d->stream)
                         : rwkvq_tc_gemm_fp8_rkv(c[0], c[1], c[2], K, sc, 1, w0, w1, w2, d->ldw, d->w_scale[0], d->w_scale[1], d->w_scale[2], d->out[0],
                                                 d->out[1], d->out[2], d->ldo, M, N, K, d->gemm_div, d->gemm_flags, d->workspace, d->workspace_bytes, d->stream);
    }
    const int64_t sb = up256(4 * M) / 4;
    float* s[3] = {sc, sc + sb, sc + 2 * sb};
    int8_t* q[3] = {(int8_t*)c[0], (int8_t*)c[1], (int8_t*)c[2]};
    const int8_t *w0 = (const int8_t*)d->w[0], *w1 = (const int8_t*)d->w[1], *w2 = (const int8_t*)d->w[2];
    if (d->nmat == 1) {
        rc = d->relu2 ? rwkvq_prep_x_int8_relu2(d->x[0], M, K, d->ldx, q[0], K, s[0], d->act_div, d->stream)
                      : rwkvq_prep_x_int8(d->x[0], d->x_dtype, M, K, d->ldx, q[0], K, s[0], d->act_div, d->stream);
        if (rc != RWKVQ_OK) return rc;
        return d->decode ? rwkvq_gemm_int8(q[0], K, s[0], w0, d->ldw, d->w_scale[0], d->out[0], d->ldo, nullptr, N, M, N, K, d->gemm_flags, d->stream)
                         : rwkvq_tc_gemm_int8(q[0], K, s[0], w0, d->ldw, d->w_scale[0], d->out[0], d->ldo, nullptr, N, M, N, K, d->gemm_flags, d->workspace,
                                              d->workspace_bytes, d->stream);
    }
    rc = rwkvq_prep3_x_int8(d->x[0], d->x[1], d->x[2], d->x_dtype, M, K, d->ldx, q[0], q[1], q[2], K, s[0], s[1], s[2], d->act_div, d->stream);
    if (rc != RWKVQ_OK) return rc;
    return d->decode ? rwkvq_gemm_int8_rkv(q[0], q[1], q[2], K, s[0], s[1], s[2], w0, w1, w2, d->ldw, d->w_scale[0], d->w_scale[1], d->w_scale[2], d->out[0],
                                           d->out[1], d->out[2], d->ldo, M, N, K, d->gemm_flags, d->stream)
                     : rwkvq_tc_gemm_int8_rkv(q[0], q[1], q[2], K, s[0], s[1], s[2], w0, w1, w2, d->ldw, d->w_scale[0], d->w_scale[1], d->w_scale[2], d->out[0],
                                              d->out[1], d->out[2], d->ldo, M, N, K, d->gemm_flags, d->workspace, d->workspace_bytes, d->stream);
}

int64_t rwkvq_linear_nvfp4_scratch_bytes(int64_t M, int64_t K) {
    if (M < 0 || K < 0 || K % 64) return 0;
    return up256(M * (K / 2)) + up256(rwkvq_nvfp4_blocked_scale_bytes(M, K)) + 256;
}

int32_t rwkvq_linear_nvfp4(const rwkvq_nvfp4_desc* d) {
    const char* who = "linear_nvfp4";
    RWKVQ_REQUIRE(d != nullptr, RWKVQ_E_BADARG, "%s: null descriptor", who);
    const int64_t M = d->M, N = d->N, K = d->K;
    RWKVQ_REQUIRE(M > 0 && N >= 0 && K > 0 && K % 256 == 0 && M < (int64_t(1) << 30) && K < (int64_t(1) << 30), RWKVQ_E_SHAPE, "%s: M=%lld K=%lld", who,
                  (long long)M, (long long)K);
    RWKVQ_REQUIRE(d->scratch && ((uintptr_t)d->scratch & 255) == 0 && d->scratch_bytes >= rwkvq_linear_nvfp4_scratch_bytes(M, K), RWKVQ_E_WORKSPACE,
                  "%s: %lld bytes of 256-byte aligned scratch needed", who, (long long)rwkvq_linear_nvfp4_scratch_bytes(M, K));
    uint8_t* codes = reinterpret_cast<uint8_t*>(d->scratch);
    uint8_t* scales = codes + up256(M * (K / 2));
    float* pts = reinterpret_cast<float*>(scales + up256(rwkvq_nvfp4_blocked_scale_bytes(M, K)));
    const int32_t rc = rwkvq_actq_nvfp4_fused(d->x, (int32_t)d->x_dtype, M, K, d->ldx, codes, K / 2, nullptr, K / 16, scales, pts, d->actq_scratch,
                                              d->actq_scratch_bytes, nullptr, d->stream);
    if (rc != RWKVQ_OK) return rc;
    return rwkvq_tc_gemm_nvfp4(codes, K / 2, scales, pts, d->w, d->ldw, d->w_scales_blocked, d->w_tscale, d->out, d->ldo, M, N, K, d->workspace,
                               d->workspace_bytes, d->stream);
}

int64_t rwkvq_ffn_scratch_bytes(int32_t kind, int64_t M, int64_t K, int64_t F) {
    if (M < 0 || K < 0 || F < 0 || (kind != RWKVQ_LINEAR_FP8 && kind != RWKVQ_LINEAR_INT8)) return 0;
    return up256(M * K) + up256(M * F) + (kind == RWKVQ_LINEAR_FP8 ? 256 : 2 * up256(4 * M));
}

int32_t rwkvq_ffn_relu2(const rwkvq_ffn_desc* d) {
    const char* who = "ffn_relu2";
    RWKVQ_REQUIRE(d != nullptr, RWKVQ_E_BADARG, "%s: null descriptor", who);
    const bool fp8 = d->kind == RWKVQ_LINEAR_FP8;
    RWKVQ_REQUIRE(fp8 || d->kind == RWKVQ_LINEAR_INT8, RWKVQ_E_BADARG, "%s: kind %d", who, d->kind);
    const int64_t M = d->M, K = d->K, F = d->F, N = d->N;
    RWKVQ_REQUIRE(M > 0 && K > 0 && F > 0 && N >= 0 && M < (int64_t(1) << 30) && K < (int64_t(1) << 30) && F < (int64_t(1) << 30), RWKVQ_E_SHAPE,
                  "%s: M=%lld K=%lld F=%lld", who, (long long)M, (long long)K, (long long)F);
    RWKVQ_REQUIRE(d->scratch && ((uintptr_t)d->scratch & 255) == 0 && d->scratch_bytes >= rwkvq_ffn_scratch_bytes(d->kind, M, K, F), RWKVQ_E_WORKSPACE,
                  "%s: %lld bytes of 256-byte aligned scratch needed", who, (long long)rwkvq_ffn_scratch_bytes(d->kind, M, K, F));
    uint8_t* xc = reinterpret_cast<uint8_t*>(d->scratch);
    uint8_t* hc = xc + up256(M * K);
    float* sc = reinterpret_cast<float*>(hc + up256(M * F));
    int32_t rc;
    if (fp8) {
        // sc: amax / scale of x, amax / scale of the hidden activations
        rc = rwkvq_actq_fp8_fused(d->x, d->x_dtype, M, K, d->ldx, xc, K, sc, sc + 4, d->actq_scratch, d->actq_scratch_bytes, nullptr, d->act_div, d->act_flags, d->stream);
        if (rc != RWKVQ_OK) return rc;
        const int32_t is_amax = d->by_scale ? 0 : 1;
        rc = rwkvq_tc_gemm_fp8_relu2(xc, K, d->by_scale ? sc + 4 : sc, is_amax, (const uint8_t*)d->w_key, d->ldw_key, d->s_key, d->hidden, F, M, F, K, d->gemm_div,
                                     d->key_flags, d->ffn_scratch, d->workspace, d->workspace_bytes, d->stream);
        if (rc != RWKVQ_OK) return rc;
        rc = rwkvq_actq_fp8_given(d->hidden, RWKVQ_F16, M, F, F, hc, F, sc + 8, sc + 12, d->ffn_scratch, d->act_div, RWKVQ_FLAG_QUANT_FROM_BF16, d->stream);
        if (rc != RWKVQ_OK) return rc;
        return rwkvq_tc_gemm_fp8(hc, F, d->by_scale ? sc + 12 : sc + 8, is_amax, (const uint8_t*)d->w_value, d->ldw_value, d->s_value, d->out, d->ldo, M, N, F,
                                 d->gemm_div, d->value_flags, d->workspace, d->workspace_bytes, d->stream);
    }
    float* hs = sc + up256(4 * M) / 4;
    rc = rwkvq_prep_x_int8(d->x, d->x_dtype, M, K, d->ldx, (int8_t*)xc, K, sc, d->act_div, d->stream);
    if (rc != RWKVQ_OK) return rc;
    rc = rwkvq_tc_gemm_int8_relu2((int8_t*)xc, K, sc, (const int8_t*)d->w_key, d->ldw_key, d->s_key, d->hidden, F, M, F, K, d->key_flags, (float*)d->ffn_scratch,
                                  d->workspace, d->workspace_bytes, d->stream);
    if (rc != RWKVQ_OK) return rc;
    rc = rwkvq_actq_int8_given(d->hidden, RWKVQ_F16, M, F, F, (int8_t*)hc, F, hs, (float*)d->ffn_scratch, d->act_div, d->stream);
    if (rc != RWKVQ_OK) return rc;
    return rwkvq_tc_gemm_int8((int8_t*)hc, F, hs, (const int8_t*)d->w_value, d->ldw_value, d->s_value, d->out, d->ldo, nullptr, N, M, N, F, d->value_flags,
                              d->workspace, d->workspace_bytes, d->stream);
}

}  // extern "C"
