// What the two tensor-core forms of the weight-only projections share (gemm_wa16.cu: one CTA per tile, gemm_wa16_pair.cu: CTA
// pairs): formats, widening of the packed weights, tensor-memory loads and stores of 32 columns, tensor maps.
#pragma once

#include "tc_common.cuh"
#include "tc_host.cuh"
#include "w8a8.cuh"

namespace rwkvq {
using namespace tc;

enum { W16_INT4_GROUP = 0, W16_INT8_TENSOR = 1 };
constexpr int kW16K = 128;                    // k per ring stage = one INT4 group
constexpr size_t kW16SmemBudget = 225 * 1024;

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {     // this thread's lane, 32 columns
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 8 nibbles of a word -> fp16 pairs odd = (n1,n5), (n3,n7) * 2^-20 and even = (n0,n4), (n2,n6) * 2^-24
__device__ __forceinline__ void widen_nibbles(uint32_t w, uint32_t* odd, uint32_t* even) {
    const uint32_t h = w >> 8;
    odd[0] = w & 0x00F000F0u;
    odd[1] = h & 0x00F000F0u;
    even[0] = w & 0x000F000Fu;
    even[1] = h & 0x000F000Fu;
}
// the same of 2 * code - centre, exact (multiples of 2^-24 below 2^-13)
__device__ __forceinline__ void widen_nibbles_centred(uint32_t w, uint32_t centre, uint32_t* odd, uint32_t* even) {
    widen_nibbles(w, odd, even);
    const uint32_t e = 0x80008000u | centre * 0x00010001u, o = 0x80008000u | centre * 0x00100010u;       // - centre * 2^-24, - centre * 2^-20
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        asm("fma.rn.f16x2 %0, %0, %1, %2;" : "+r"(odd[i]) : "r"(0x40004000u), "r"(o));
        asm("fma.rn.f16x2 %0, %0, %1, %2;" : "+r"(even[i]) : "r"(0x40004000u), "r"(e));
    }
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t pack2_loaded(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm volatile("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
// two independent fp32 fused multiply-adds in one instruction
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t x, uint64_t y) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y));
}
// the same on a register pair of a tensor-memory load: volatile, so that it stays behind the load's wait
__device__ __forceinline__ void fma2_loaded(uint64_t& acc, uint64_t x, uint32_t lo, uint32_t hi) {
    asm volatile("{\n\t.reg .b64 t;\n\tmov.b64 t, {%2, %3};\n\tfma.rn.f32x2 %0, %1, t, %0;\n\t}" : "+l"(acc) : "l"(x), "r"(lo), "r"(hi));
}

// byte matrix, tiles of box_rows x box_bytes; 64-byte boxes take the 64-byte swizzle
inline int32_t w16_map(CUtensorMap* m, const void* ptr, int64_t rows, int64_t row_bytes, int64_t ld, int box_rows, int box_bytes, const char* who) {
    if (box_bytes == 128) return make_map(m, ptr, rows, row_bytes, ld, box_rows, who);
    EncodeTiledFn fn = encode_fn();
    RWKVQ_REQUIRE(fn != nullptr, RWKVQ_E_LAUNCH, "%s: cuTensorMapEncodeTiled is not available from the driver", who);
    RWKVQ_REQUIRE(aligned16(ptr) && ld % 16 == 0 && ld >= row_bytes, RWKVQ_E_ALIGN, "%s: TMA needs a 16-byte aligned base and row pitch", who);
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld};
    const cuuint32_t box[2] = {(cuuint32_t)box_bytes, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    RWKVQ_REQUIRE(r == CUDA_SUCCESS, RWKVQ_E_LAUNCH, "%s: cuTensorMapEncodeTiled failed (%d)", who, (int)r);
    return RWKVQ_OK;
}

// An fp32 value of 2^-110 and more as three bf16 values of 8 mantissa bits each that add up to it exactly (cut, not rounded: no part
// overflows; of a smaller one what is below bf16's least, 2^-133, is lost).
// An infinity or NaN is its own highest part and has no others; h1 is the highest part of a finite value only.
struct Bf16Parts { uint32_t h, h1, m, l; };
__device__ __forceinline__ Bf16Parts bf16_parts(float v) {
    const uint32_t u = __float_as_uint(v);
    Bf16Parts p;
    if ((u & 0x7f800000u) == 0x7f800000u) {
        p.h = (u >> 16) | ((u & 0x007fffffu) ? 0x40u : 0u);
        p.h1 = p.m = p.l = 0;
        return p;
    }
    const float rest = v - __uint_as_float(u & 0xffff0000u);
    const uint32_t um = __float_as_uint(rest);
    p.h = p.h1 = u >> 16;
    p.m = um >> 16;
    p.l = __float_as_uint(rest - __uint_as_float(um & 0xffff0000u)) >> 16;
    return p;
}

// ---- CTA pairs (gemm_wa16_pair.cu)
// zero points of the INT4 codes: three bf16 parts of each fp32 value on either side, kW16ZSlots products per group
constexpr int kW16ZSlots = 8;
struct W16PairCall {
    int fmt, NB, slices;
    const void* w;                // packed weights, ldw bytes between rows
    const void* x;                // INT4: the permuted activations (wa16_prep_kernel), INT8: fp16 activations; ldx elements
    const void* xz;               // INT4: the groups' sums in bf16 parts [M][groups][kW16ZSlots]
    const float* scales;
    const float* zeros;
    __half* out;
    float* part;
    int64_t ldw, ldx, ldo, M, N, K;
};
bool wa16_pair_fits(int fmt);     // the build's kernels have the registers that their split counts on
int32_t run_wa16_pair(const W16PairCall& c, cudaStream_t st, const char* who);

}  // namespace rwkvq
