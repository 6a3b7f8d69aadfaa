// Packed weights to bf16 / fp16 pairs with the reference's two roundings, as the fused kernel and the dequantisation pre-pass do it.
#pragma once
#include "wqbmm_decode_common.cuh"

namespace opsnn {

namespace {

enum class MixW { kInt4, kInt8, kE4m3 };

// A pair of weights, codes in the low bits of the two halves (other bits arbitrary), to the 16-bit type, exactly (int4: the caller has
// shifted the nibble down). e4m3's two NaN codes read as +-480 here; fix_nan below puts that right.
template <MixW kW, bool kBf16>
__device__ __forceinline__ uint32_t mix_exact(uint32_t p)
{
    using N = Num<kBf16>;
    uint32_t v;
    if (kW == MixW::kInt4) {
        asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(v) : "r"(p), "n"(0x000F000F), "n"(N::kMagic));  // (nibble ^ 8) | magic
        return N::sub(v, N::kBias);
    }
    if (kW == MixW::kInt8) {
        if (kBf16) {  // (128 + low seven bits) - (128 or 256)
            uint32_t s;
            asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(p), "n"(0x007F007F), "n"(0x43004300));
            asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(s) : "r"(p), "n"(0x00800080), "n"(0x43004300));
            return N::sub(v, s);
        }
        asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(v) : "r"(p), "n"(0x00FF00FF), "n"(0x64806480));  // 1024 + (byte ^ 0x80)
        return N::sub(v, 0x64806480u);
    }
    constexpr uint32_t kMag = kBf16 ? 0x07F007F0u : 0x3F803F80u, kRebias = kBf16 ? 0x7B807B80u : 0x5C005C00u;
    v = (p << (kBf16 ? 4 : 7)) & kMag;  // the magnitude under the wider type's sign bit reads as w * 2^-120 (bf16) / 2^-8 (fp16)
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(p << 8), "n"(0x80008000), "r"(v));
    return N::mul(v, kRebias);
}

template <bool kBf16, bool kOff>
__device__ __forceinline__ uint32_t mix_scale(uint32_t v, uint32_t sc, uint32_t of)
{
    using N = Num<kBf16>;
    if (kOff) v = N::add(v, of);
    return N::mul(v, sc);
}

// Any of the four bytes an e4m3 NaN (low seven bits all set)?
__device__ __forceinline__ uint32_t has_nan8(uint32_t r) { return ((r & 0x7F7F7F7Fu) + 0x01010101u) & 0x80808080u; }
// Replaces the halves of `v` whose code byte (bytes 0 and 2 of p) is a NaN code.
__device__ __forceinline__ uint32_t fix_nan(uint32_t v, uint32_t p)
{
    if ((p & 0x7Fu) == 0x7Fu) v |= 0x00007FFFu;
    if ((p & 0x7F0000u) == 0x7F0000u) v |= 0x7FFF0000u;
    return v;
}

}  // namespace

}  // namespace opsnn
