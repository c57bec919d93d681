// Device helpers shared by the bit-pack kernels (pack.cu, fused_encode.cu, dense.cu).
#pragma once
#include "common.cuh"

namespace pkv {

constexpr int kWarpsPerCta = 4;

// ---- per-pack helpers --------------------------------------------------------------------

// bytewise bit_length of four packed bytes, summed
__device__ __forceinline__ unsigned sum_bitlen4(unsigned d) {
    return bit_length_u32(d & 0xFFu) + bit_length_u32((d >> 8) & 0xFFu) + bit_length_u32((d >> 16) & 0xFFu) +
           bit_length_u32(d >> 24);
}

__device__ __forceinline__ void store_pack_smem(uint8_t* dst, uint64_t w, int len) {
    // dst is 2-byte aligned; the pack takes 2*len bytes = len u16 words
    uint16_t* q = reinterpret_cast<uint16_t*>(dst);
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (i < len) q[i] = (uint16_t)(w >> (16 * i));
}

// Copies `size` bytes (plus up to 16 bytes of slack on either side, inside the stream
// allocation) from global `src` into shared memory so that the shared copy of src[0] has
// the same address modulo 16.  Returns the shared pointer that mirrors src.
__device__ __forceinline__ const uint8_t* warp_copy_in(uint8_t* sbuf16, const uint8_t* src, int size, int lane,
                                                       const uint8_t* lo, const uint8_t* hi) {
    int phase = (int)(reinterpret_cast<uintptr_t>(src) & 15);
    const uint8_t* a = src - phase;                 // 16-byte aligned start
    int total = (phase + size + 15) & ~15;
    for (int i = 16 * lane; i < total; i += 16 * 32) {
        const uint8_t* p = a + i;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (p >= lo && p + 16 <= hi) {
            v = *reinterpret_cast<const uint4*>(p);
        } else {                                    // ragged edge of the allocation
            unsigned q[4] = {0, 0, 0, 0};
#pragma unroll
            for (int b = 0; b < 16; b++)
                if (p + b >= lo && p + b < hi) q[b >> 2] |= (unsigned)p[b] << (8 * (b & 3));
            v = make_uint4(q[0], q[1], q[2], q[3]);
        }
        *reinterpret_cast<uint4*>(sbuf16 + i) = v;
    }
    return sbuf16 + phase;
}

// Copies `size` bytes from shared `src` to global `dst`; both have the same address modulo
// 16 and are 2-byte aligned.  Warp-cooperative.
__device__ __forceinline__ void warp_copy_out(uint8_t* dst, const uint8_t* src, int size, int lane) {
    int head = (16 - (int)(reinterpret_cast<uintptr_t>(dst) & 15)) & 15;
    if (head > size) head = size;
    for (int i = 2 * lane; i < head; i += 64)
        *reinterpret_cast<uint16_t*>(dst + i) = *reinterpret_cast<const uint16_t*>(src + i);
    int body = (size - head) & ~15;
    for (int i = 16 * lane; i < body; i += 16 * 32)
        *reinterpret_cast<uint4*>(dst + head + i) = *reinterpret_cast<const uint4*>(src + head + i);
    for (int i = head + body + 2 * lane; i < size; i += 64)
        *reinterpret_cast<uint16_t*>(dst + i) = *reinterpret_cast<const uint16_t*>(src + i);
}

}  // namespace pkv
