// wire.cuh -- reading a compact down row (kernels.h WIRE_*): the escape bits and the two roundings of the reference's result.
#pragma once
#include <stdint.h>
#include "kernels.h"

// escape code (2 bits) -> bits 16.. of (dot + 32768): 0, +1 or -1
__device__ __forceinline__ int wire_hi(uint32_t code) { return ((int)(code ^ 2u) - 2) << 16; }
__device__ __forceinline__ float wire_scale(float dot, float qs, float s) { return __fmul_rn(__fmul_rn(dot, qs), s); }
// A warp adds one pair's contribution to rows 128 rb + 4 lane .. + 3 of acc: raw = the row's eight bytes there, qs = the scale of the pair's int8 row,
// s = the expert's down scales of those rows, esc = the record's escape bits.  A block that did not fit 16 bits (rare) also reads its escape plane and
// leaves it and the record's bit clean for the next layer.
__device__ __forceinline__ void wire_add(float4 &acc, const uint2 raw, const float w, const float qs, const float4 s, const int esc, const int rb, const int lane,
                                         uint8_t *wire, const int np_cap, const int slot) {
    // 2^23 + h as a float is the 16 bits h under the bytes 4B 00: a byte permute and an exact subtraction give (float)dot, instead of a mask, a subtraction and a
    // conversion (2048 tokens: 156.4 -> 155.3 us per layer)
    float d[4] = {__uint_as_float(__byte_perm(raw.x, 0x4B000000u, 0x7610)) - 8421376.0f, __uint_as_float(__byte_perm(raw.x, 0x4B000000u, 0x7632)) - 8421376.0f,
                  __uint_as_float(__byte_perm(raw.y, 0x4B000000u, 0x7610)) - 8421376.0f, __uint_as_float(__byte_perm(raw.y, 0x4B000000u, 0x7632)) - 8421376.0f};
    if ((esc >> rb) & 1) {
        uint32_t *pw = reinterpret_cast<uint32_t *>(wire + (size_t)slot * WIRE_PITCH + 4096) + ((rb * 128 + 4 * lane) >> 4);
        const uint32_t bits = (*pw >> ((lane & 3) * 8)) & 0xFFu;
#pragma unroll
        for (int i = 0; i < 4; i++) d[i] += (float)wire_hi((bits >> (2 * i)) & 3u);
        __syncwarp();
        if ((lane & 3) == 0) *pw = 0u;
        if (lane == 0) atomicAnd(reinterpret_cast<int *>(wire + (size_t)np_cap * WIRE_PITCH + (size_t)slot * WIRE_REC + 8), ~(1 << rb));
    }
    acc.x = __fmaf_rn(w, wire_scale(d[0], qs, s.x), acc.x); acc.y = __fmaf_rn(w, wire_scale(d[1], qs, s.y), acc.y);
    acc.z = __fmaf_rn(w, wire_scale(d[2], qs, s.z), acc.z); acc.w = __fmaf_rn(w, wire_scale(d[3], qs, s.w), acc.w);
}
