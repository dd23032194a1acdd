// A float32 as three bfloat16 numbers: x = x0 + x1 + x2 exactly from 2^-110 on (8 + 8 + 8 significant bits, each part the rounding of what the parts before
// it leave; smaller numbers lose what is below 2^-133).  Six products of parts stand for one float32 product, x0 w0 + (x0 w1 + x1 w0) + (x0 w2 + x1 w1 + x2 w0); what they leave out is at most
// 2^-24 + 2^-34 of |x w| and of either sign (x = w = 1 + 2^-8 - 2^-17; the rounding of one float32 product is as much), and a product of two bfloat16 numbers is exact in the tensor core's float32 sum.  (Dekker, "A floating-point
// technique for extending the available precision", 1971; Ozaki et al., 2012, for matrix products on short formats.)
#pragma once
#include "sm100.cuh"

namespace mi {
namespace split3 {

constexpr int PARTS = 3, PRODUCTS = 6;
// the parts of the two operands, small products first: the tensor core cuts off instead of rounding when it adds
__device__ constexpr int PART_A[PRODUCTS] = {2, 1, 0, 1, 0, 0}, PART_B[PRODUCTS] = {0, 1, 2, 0, 1, 0};

// a, b -> their next part side by side; a and b become what is left
__device__ __forceinline__ uint32_t take_part(float& a, float& b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
    a -= __uint_as_float(w << 16);
    b -= __uint_as_float(w & 0xffff0000u);
    return w;
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
                 :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                    "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

}  // namespace split3
}  // namespace mi
