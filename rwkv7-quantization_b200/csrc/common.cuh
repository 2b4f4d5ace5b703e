// Shared device helpers and host-side error plumbing of librwkvq (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/rwkvq.h"

namespace rwkvq {

// ----------------------------------------------------------------------------- host side
extern thread_local char g_err[512];
extern std::atomic<int64_t> g_launches;

int32_t fail(int32_t code, const char* fmt, ...);
int32_t check_launch(const char* what);   // cudaGetLastError() -> status, counts the launch
int sm_count();
// wall-time limit of every bounded device-side wait, nanoseconds: 1.5 s unless RWKVQ_WAIT_LIMIT_US (read once) or
// rwkvq_set_wait_limit_us changed it
unsigned long long wait_limit_ns();
// per kernel and device: opt in to `bytes` of dynamic shared memory (once)
int32_t ensure_smem_optin(const void* kern, int bytes, const char* who);
// per (kernel, device, dynamic shared memory size): the opt-in above plus the resident CTAs per SM, looked up once
int32_t kernel_plan(const void* kern, int threads, size_t smem, int optin_bytes, int* per_sm, const char* who);
// programmatic dependent launch unless RWKVQ_PDL=0 (read once)
bool use_pdl();
// The library's per-device status word (device address): kernels whose entry points take no status pointer set it to
// RWKVQ_E_TIMEOUT when a bounded wait gives up; rwkvq_device_status reads it.  Null if the lookup failed.
int* device_status_ptr();

// CTAs of an elementwise pass over `vecs` vectors by 256-thread CTAs that load four vectors per thread at a time: enough for
// two per SM where the block allows it, then four vectors per thread, at most `most`.  (One vector per thread and one CTA per
// 256: 717 rows of 4096 took 8.7 instead of 5.3 us, the CTAs' arrivals on one counter queueing up.)
inline int64_t elementwise_ctas(int64_t vecs, int64_t most) {
    return std::max<int64_t>(1, std::min((vecs + 255) / 256, std::min(most, std::max<int64_t>(2 * (int64_t)sm_count(), (vecs + 1023) / 1024))));
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

#define RWKVQ_REQUIRE(cond, code, ...) \
    do {                               \
        if (!(cond)) return ::rwkvq::fail(code, __VA_ARGS__); \
    } while (0)

// ----------------------------------------------------------------------------- device side
__device__ __forceinline__ float div_full(float a, float b) {
    float r;
    asm("div.full.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float div_mode_f32(float a, float b, int mode) {
    return mode == RWKVQ_DIV_FULL ? div_full(a, b) : __fdiv_rn(a, b);
}

// qmax / amax and amax / qmax of the activation scales.  RWKVQ_DIV_TORCH: what torch's GPU kernels compute for
// `scalar / tensor` (reciprocal, then a product) and `tensor / scalar` (product with the rounded reciprocal).
__device__ __forceinline__ float scale_inv(float qmax, float amax, int mode) {
    if (mode == RWKVQ_DIV_TORCH) return __fmul_rn(__frcp_rn(amax), qmax);
    return div_mode_f32(qmax, amax, mode);
}
__device__ __forceinline__ float scale_fwd(float amax, float qmax, int mode) {
    if (mode == RWKVQ_DIV_TORCH) return __fmul_rn(amax, __frcp_rn(qmax));
    return div_mode_f32(amax, qmax, mode);
}

template <int DT>
__device__ __forceinline__ float2 cvt2(uint32_t v) {   // two packed 16-bit values -> fp32
    if (DT == RWKVQ_F16) {
        return __half22float2(*reinterpret_cast<const __half2*>(&v));
    } else {
        return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
    }
}
__device__ __forceinline__ float bf16_round(float v) {  // fp32 -> bf16 (RNE) -> fp32
    return __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&p);
}
__device__ __forceinline__ float2 bf16_round2(float2 f) {   // both in one conversion
    const uint32_t p = pack_bf16x2(f.x, f.y);
    return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}
// two fp32 -> two e4m3 bytes (lo in bits 0-7), round-to-nearest-even, saturating.  One hardware instruction
// (written as PTX: the cuda_fp8.h helper may pick its software path, hundreds of instructions per pair).
__device__ __forceinline__ uint32_t e4m3x2(float lo, float hi) {
    unsigned short r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return (uint32_t)r;
}
// two e4m3 bytes (bits 0-15) -> two f16 (exact), low byte in the low half
__device__ __forceinline__ uint32_t e4m3x2_to_f16x2(uint32_t two_codes) {
    uint32_t r;
    const unsigned short c = (unsigned short)two_codes;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(c));
    return r;
}

// two floats -> one byte of two e2m1 codes (lo in the low nibble), round-to-nearest-even, saturating
__device__ __forceinline__ uint32_t e2m1x2(float lo, float hi) {
    unsigned short r;
    asm("{ .reg .b8 t; cvt.rn.satfinite.e2m1x2.f32 t, %1, %2; cvt.u16.u8 %0, t; }" : "=h"(r) : "f"(hi), "f"(lo));
    return (uint32_t)r;
}
// one byte of two e2m1 codes -> f16 pair (low nibble in the low half), exact
__device__ __forceinline__ uint32_t e2m1x2_to_f16x2(uint32_t byte) {
    uint32_t r;
    const unsigned short b = (unsigned short)(byte & 0xffu);
    asm("{ .reg .b8 t; cvt.u8.u16 t, %1; cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(r) : "h"(b));
    return r;
}
__device__ __forceinline__ float e4m3_to_float(uint32_t code) {
    const uint32_t h2 = e4m3x2_to_f16x2(code & 0xffu);
    return __half2float(__ushort_as_half((unsigned short)(h2 & 0xffffu)));
}
// two fp32 values in a 64-bit register pair, and arithmetic on both halves in one instruction
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack_f32x2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// the engine's relu_square of 8 fp16 values: fp16(max(y, 0)^2) in fp32 arithmetic, NaN kept
__device__ __forceinline__ uint4 relu2_f16x8(const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t h[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float2 f = cvt2<RWKVQ_F16>(w[q]);
        f.x = f.x < 0.f ? 0.f : f.x;
        f.y = f.y < 0.f ? 0.f : f.y;
        const __half2 r = __floats2half2_rn(f.x * f.x, f.y * f.y);
        h[q] = *reinterpret_cast<const uint32_t*>(&r);
    }
    return make_uint4(h[0], h[1], h[2], h[3]);
}

// 1 / bs, correctly rounded, of an NVFP4 block scale: bs = (8 + m) / 8 * 2^e as an e4m3 code (2^-6 ... 448, always normal), so
// its reciprocal is the rounded 8 / (8 + m) times an exact power of two.  Lane m (mod 8) of the warp holds 8 / (8 + m) and
// one shuffle fetches it.  __frcp_rn per block instead costs the quantizers 1 %, the fused GEMV's prologue 3 % of the
// call ([4096, 4096] 7 rows 7.96 -> 8.25 us), and a table in constant memory misses its cache once per launch (+0.5 us).
// Whole warps only.
__device__ __forceinline__ float eighth_rcp() {
    const int m = threadIdx.x & 7;
    const float lo = m & 2 ? (m & 1 ? 8.f / 11.f : 8.f / 10.f) : (m & 1 ? 8.f / 9.f : 1.f);
    const float hi = m & 2 ? (m & 1 ? 8.f / 15.f : 8.f / 14.f) : (m & 1 ? 8.f / 13.f : 8.f / 12.f);
    return m & 4 ? hi : lo;
}
__device__ __forceinline__ float block_scale_rcp(uint32_t code, float eighth) {
    const float r = __shfl_sync(0xffffffffu, eighth, code & 7);
    return __uint_as_float(__float_as_uint(r) - (((code >> 3) - 7u) << 23));
}

// e2m1 codes of 8 values of one NVFP4 block: e2m1_rn((f * inv_pts) / bs), the quotient correctly rounded, with bs an e4m3
// block scale (2^-6 ... 448) and rc = 1 / bs.  The quotient is a product with the reciprocal, its exact remainder and one correction
// (P. Markstein, IBM J. Res. Dev. 34(1), 1990: with a correctly rounded reciprocal the corrected quotient is correctly
// rounded; |t| is far from overflow, and where the remainder underflows the code is a zero either way).  t is kept negated,
// so that the remainder of a zero is +0 and the correction leaves the zero's sign, which the code carries, alone.  The 16
// values of a block share one reciprocal: a division for each took half of the quantizers' instructions.
__device__ __forceinline__ uint32_t nvfp4_codes8(const float (&f)[8], float inv_pts, float bs, float rc) {
    const uint64_t ninv = pack_f32x2(-inv_pts, -inv_pts), nrc = pack_f32x2(-rc, -rc), bs2 = pack_f32x2(bs, bs);
    uint32_t out = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint64_t nt = mul_f32x2(pack_f32x2(f[2 * q], f[2 * q + 1]), ninv);        // -t
        const uint64_t u = mul_f32x2(nt, nrc);                                          // t * rc
        const float2 v = unpack_f32x2(fma_f32x2(fma_f32x2(u, bs2, nt), nrc, u));
        out |= e2m1x2(v.x, v.y) << (8 * q);
    }
    return out;
}
__device__ __forceinline__ float clamp448(float v) { return fminf(fmaxf(v, -448.f), 448.f); }

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// streaming 128-bit weight load: read-only path, do not keep the line in L1
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

// 16 fp16 values of a result row: one 32-byte store where the row allows it (two 16-byte stores of a lane send each sector to
// L2 twice, as halves), `left` = columns from here to the row's end
__device__ __forceinline__ void store_f16x16(__half* o, const uint32_t (&h)[8], int left, bool vec16, bool vec32) {
    if (vec32 && left >= 16) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(o), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]), "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7]) : "memory");
    } else if (vec16 && left >= 16) {
        reinterpret_cast<uint4*>(o)[0] = make_uint4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<uint4*>(o)[1] = make_uint4(h[4], h[5], h[6], h[7]);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (j < left) o[j] = __ushort_as_half((unsigned short)((h[j >> 1] >> ((j & 1) * 16)) & 0xffff));
    }
}
// rows of a result start on 16- / 32-byte boundaries
__device__ __forceinline__ bool rows_vec16(const void* out, int64_t ldo) { return (ldo % 8 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0); }
__device__ __forceinline__ bool rows_vec32(const void* out, int64_t ldo) { return (ldo % 16 == 0) && ((reinterpret_cast<uintptr_t>(out) & 31) == 0); }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)::"memory");
    return t;
}
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded wait for *p == want (a flag another CTA of the same cooperative launch publishes with st_release_u32).
// The clock costs hundreds of nanoseconds to read, so it is consulted only after a few hundred failed polls.
__device__ __forceinline__ bool wait_flag_eq(const uint32_t* p, uint32_t want, unsigned long long limit_ns) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i) {
        if (ld_acquire_u32(p) == want) return true;
        __nanosleep(64);
    }
    const unsigned long long t0 = global_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 256; ++i) {
            if (ld_acquire_u32(p) == want) return true;
            __nanosleep(128);
        }
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// atomic max of a non-negative float through its bit pattern
__device__ __forceinline__ void atomic_max_nonneg(float* addr, float v) {
    atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));
}

}  // namespace rwkvq
