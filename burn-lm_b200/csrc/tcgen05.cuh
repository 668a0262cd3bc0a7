// Shared helpers of kernels that form 32-bit products on the 5th-generation tensor cores: mbarriers, TMA loads, tcgen05
// instructions and descriptors, and the split of a float into three bfloat16 numbers.
//
// A float has 24 bits of mantissa, a bfloat16 number 8 and the same exponents, so x = x1 + x2 + x3 exactly (x1 = x's first bits,
// x2 = the next, x3 = what is left; split3_as).  x w is then nine products that the tensor cores form exactly; the six with i + j <= 4 are
// summed (in float32, the smallest first), the other three are below 2^-21 of the product and 2^-24 on average.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace tc5 {

constexpr unsigned kSpinLimit = 1u << 18;
// what a kernel whose wait ran out leaves in the status word: a code for every file that includes this one
enum { TC5_OK = 0, TC5_TIMEOUT_PRODUCT = 15, TC5_TIMEOUT_SCAN_CHUNKS = 16, TC5_TIMEOUT_SCAN_LONG = 17, TC5_TIMEOUT_QUADS = 18 };

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Waits for a phase, a bounded number of times (false: it ran out).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
    const unsigned addr = smem_u32(bar);
    unsigned done;
    asm volatile(                              // a phase that is over already answers at once
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    for (unsigned spin = 0; !done && spin < kSpinLimit; ++spin)
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
    return done;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int w, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
        : "memory");
}
// one lane of a converged warp
__device__ __forceinline__ bool elect() {
    unsigned is;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(is));
    return is;
}
// what a thread wrote to shared memory becomes visible to the tensor cores and the TMA
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Operand descriptor in shared memory, rows of 128 (swizzle 2) or 64 bytes (swizzle 4), eight rows `group` bytes apart; `lead`: MN-major
// operands of more than one swizzled row's length, the distance of the next piece.
__device__ __forceinline__ unsigned long long operand(const void* tile, int swizzle, int group, int lead = 16) {
    return (unsigned long long)((smem_u32(tile) >> 4) & 0x3fff) | (unsigned long long)(lead >> 4) << 16 |
           (unsigned long long)(group >> 4) << 32 | (unsigned long long)1 << 46 | (unsigned long long)swizzle << 61;
}
// Instruction descriptor of kind::f16: fp32 accumulator, bf16 operands, M 128.
__host__ __device__ constexpr unsigned instruction(int n, bool a_mn = false, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u) | ((unsigned)(n >> 3) << 17) |
           ((unsigned)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma(unsigned tmem_d, unsigned long long a, unsigned long long b, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"((unsigned)accumulate)
        : "memory");
}
// the A operand from tensor memory: a row a lane, two places of K a column
__device__ __forceinline__ void mma_ts(unsigned tmem_d, unsigned tmem_a, unsigned long long b, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(b), "r"(idesc), "r"((unsigned)accumulate)
        : "memory");
}
__device__ __forceinline__ void commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// Sixteen columns of the warp's 32 lanes; wait_ld before the registers are read.
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float* v) {
    unsigned* r = reinterpret_cast<unsigned*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(unsigned taddr, const unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st8(unsigned taddr, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// The whole warp takes (gives back) `cols` columns of tensor memory, a power of two of at least 32; the address lands in `slot`.
__device__ __forceinline__ void tmem_alloc(unsigned* slot, int cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
}
__device__ __forceinline__ void tmem_free(unsigned base, int cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(base), "r"(cols));
}

// Two floats as three pairs of bfloat16 numbers (the first float in the lower half); x3 is exact whichever of the first two are rounded.
// Where all are cut off in both operands, the products left out have the product's own sign and add up: errors of recurrences and products
// 1.1 to 1.7 times as large.  Rounding either operand's leaves them of either sign.  With x1 cut off no finite float becomes an infinity, so
// that is what recurrences take, x2 rounded.  As many instructions each; a conversion takes longer than a byte permutation.
template <bool ROUND1, bool ROUND2>
__device__ __forceinline__ void split3_as(float a, float b, unsigned& p1, unsigned& p2, unsigned& p3) {
    auto part = [&](bool round) {
        const __nv_bfloat162 m = __floats2bfloat162_rn(a, b);
        const unsigned p = round ? *reinterpret_cast<const unsigned*>(&m) : __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
        a -= __uint_as_float(round ? p << 16 : __float_as_uint(a) & 0xffff0000u);
        b -= __uint_as_float(round ? p & 0xffff0000u : __float_as_uint(b) & 0xffff0000u);
        return p;
    };
    p1 = part(ROUND1);
    p2 = part(ROUND2);
    p3 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ void split3(float a, float b, unsigned& p1, unsigned& p2, unsigned& p3) { split3_as<false, true>(a, b, p1, p2, p3); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static inline EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q);
        return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? (EncodeTiledFn)f : nullptr;
    }();
    return fn;
}
// A view of R dimensions (strides of all but the first in bytes, multiples of 16); what lies outside reads as zero.
template <int R>
static inline bool make_map(CUtensorMap* out, CUtensorMapDataType type, const void* base, const long long (&dims)[R],
                            const long long (&strides)[R - 1], const int (&box)[R], CUtensorMapSwizzle swizzle) {
    const EncodeTiledFn encode = encode_tiled();
    if (!encode) return false;
    cuuint64_t d[R], s[R - 1];
    cuuint32_t b[R], e[R];
    for (int i = 0; i < R; ++i) {
        d[i] = (cuuint64_t)dims[i];
        b[i] = (cuuint32_t)box[i];
        e[i] = 1;
        if (i) s[i - 1] = (cuuint64_t)strides[i - 1];
    }
    return encode(out, type, R, const_cast<void*>(base), d, s, b, e, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static inline bool make_map_3d(CUtensorMap* out, CUtensorMapDataType type, const void* base, const long long (&dims)[3],
                               const long long (&strides)[2], const int (&box)[3], CUtensorMapSwizzle swizzle) {
    return make_map<3>(out, type, base, dims, strides, box, swizzle);
}
static inline bool make_map_4d(CUtensorMap* out, CUtensorMapDataType type, const void* base, const long long (&dims)[4],
                               const long long (&strides)[3], const int (&box)[4], CUtensorMapSwizzle swizzle) {
    return make_map<4>(out, type, base, dims, strides, box, swizzle);
}

}  // namespace tc5
