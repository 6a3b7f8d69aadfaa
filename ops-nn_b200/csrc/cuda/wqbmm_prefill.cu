// Weight-only quant matmul for m beyond the decode range ("prefill"): the weight is dequantised once into the workspace as
// a k-contiguous (n, k) matrix in x's dtype, then the tcgen05 kind::f16 matmul of qmm_umma.cu runs on x and that matrix.
//
// Reference: weight_quant_batch_matmul_v2/op_kernel/arch35/weight_quant_batch_matmul_v2_reg_base_common.h:164-286 (vector
// cores dequantise the weight tile by tile into L1, the cube unit multiplies in bf16/fp16); arithmetic of the golden
// weight_quant_batch_matmul_v2/tests/assets/wqbmmv2_kernel_golden.py:199-297:
//   w' = cast_x( cast_x( float(w) + float(offset) ) * float(scale) )     two roundings in x's dtype, as the decode kernel
//   y  = cast_x( sum_k x * w' (fp32) + bias )
// The dequantised weight is what the reference's cube unit sees too, so the result differs from the golden only by fp32
// summation order.
//
// HBM cost of the pre-pass: n*k/2 (int4) read + 2*n*k written, then 2*n*k read once by the matmul (x stays in L2):
// worthwhile once the matmul's 2*m*n*k flops dominate; up to m = 1152 the fused kernel (wqbmm_mixed.cu) and the streaming decode
// kernels take what they can.
#include <cstdlib>
#include <type_traits>

#include "common.cuh"
#include "wq_convert.cuh"
#include "wqbmm_decode_common.cuh"

namespace opsnn {

bool qmm_umma_eligible(const OpsnnQmmParams* p);
int32_t qmm_umma_launch(const OpsnnQmmParams* p, cudaStream_t stream);

namespace {

constexpr int TK = 64, TN = 64, NT = 256;

template <bool kBf16>
__device__ __forceinline__ float round_x(float v)
{
    if (kBf16) return __bfloat162float(__float2bfloat16_rn(v));
    return __half2float(__float2half_rn(v));
}
template <bool kBf16>
__device__ __forceinline__ float load_x(const void* base, int64_t idx)
{
    if (kBf16) return __uint_as_float((uint32_t)__ldg(reinterpret_cast<const uint16_t*>(base) + idx) << 16);
    return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const uint16_t*>(base) + idx)));
}
template <bool kBf16>
__device__ __forceinline__ uint16_t bits_x(float v)
{
    if (kBf16) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
    return __half_as_ushort(__float2half_rn(v));
}

// One CTA: a TK x TN tile of the weight -> dst[n][k] (row pitch kp elements). Any storage, one element at a time.
template <bool kBf16>
__global__ void __launch_bounds__(NT) wq_dequant_nk_kernel(const OpsnnWqbmmParams p, uint16_t* __restrict__ dst, int64_t kp,
                                                           float* __restrict__ one)
{
    __shared__ __align__(16) uint16_t tile[TN][TK + 8];  // row pitch 144 bytes: 16-byte aligned rows, skewed banks
    const int tid = threadIdx.x;
    const int64_t tiles_n = (p.n + TN - 1) / TN;
    const int64_t k0 = ((int64_t)blockIdx.x / tiles_n) * TK, n0 = ((int64_t)blockIdx.x % tiles_n) * TN;
    if (blockIdx.x == 0 && tid == 0) *one = 1.0f;  // the unit dequant scale the matmul's epilogue multiplies by
    for (int e = tid; e < TK * TN; e += NT) {
        int kk, nn;
        if (p.trans_w) { nn = e / TK; kk = e % TK; } else { kk = e / TN; nn = e % TN; }
        const int64_t gn = n0 + nn, gk = k0 + kk;
        float w = 0.f;
        if (gn < p.n && gk < p.k) {
            const int64_t idx = p.trans_w ? gn * p.w_ld + gk : gk * p.w_ld + gn;
            w = load_as_float(p.w, idx, p.w_dtype);
            const int64_t g = p.group_size > 0 ? gk / p.group_size : 0;
            const int64_t sidx = g * p.scale_sg + gn * p.scale_sn;
            if (p.offset != nullptr) w = round_x<kBf16>(__fadd_rn(w, load_x<kBf16>(p.offset, sidx)));
            w = round_x<kBf16>(__fmul_rn(w, load_wq_scale(p.scale, sidx, p.scale_dtype, kBf16)));
        }
        tile[nn][kk] = bits_x<kBf16>(w);
    }
    __syncthreads();
    // 64 rows (n) x 128 bytes (64 k): 16-byte pieces, 8 per row; kp % 8 == 0 and k0 % 64 == 0 keep them aligned
    for (int e = tid; e < TN * (TK / 8); e += NT) {
        const int nn = e / (TK / 8), c = e % (TK / 8);
        const int64_t gn = n0 + nn, gk = k0 + c * 8;
        if (gn < p.n && gk < kp)
            *reinterpret_cast<uint4*>(dst + gn * kp + gk) = *reinterpret_cast<const uint4*>(&tile[nn][c * 8]);
    }
}

// two fp32 -> packed pair in x's dtype (lo in the low half), and back
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
    if (kBf16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <bool kBf16>
__device__ __forceinline__ float2 unpack2(uint32_t v)
{
    if (kBf16) return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
    return __half22float2(*reinterpret_cast<const __half2*>(&v));
}

// Weight stored (k,n): a tile of 64 k rows x 32 words (256 int4 or 128 8-bit columns), so that a row of it is 128 bytes in the weight and
// a column 128 bytes in the image. A thread owns one word column over 8 k rows; a pair conversion gives two columns of one row, two
// rows' results are re-paired into (k, k + 1) words with byte permutes and kept at word (k pair ^ word column), which is free of bank
// conflicts both ways and leaves a 16-byte piece together (in another order). Bound by HBM: 0.5 (1) bytes in, 2 out per weight; with
// 32-byte pieces of rows and 4-byte stores it was 252 us for 8192 x 28672 int4, 588 MB.
// Needs word-aligned rows, n a multiple of a word's columns, scales in x's dtype, groups of a multiple of 8 rows.
template <MixW kW, bool kBf16, bool kOff>
__global__ void __launch_bounds__(NT) wq_dequant_kn_kernel(const OpsnnWqbmmParams p, uint16_t* __restrict__ dst, int64_t kp, float* __restrict__ one,
                                                           uint32_t tiles_n)
{
    pdl_trigger();
    pdl_wait();
    constexpr int kCols = kW == MixW::kInt4 ? 8 : 4, kPairs = kCols / 2, kTileN = 32 * kCols;
    __shared__ __align__(16) uint32_t tile[kTileN * 32];
    const int tid = threadIdx.x, wj = tid & 31, kr = tid >> 5;
    const uint32_t tk = blockIdx.x / tiles_n;
    const int64_t k0 = (int64_t)tk * 64, n0 = (int64_t)(blockIdx.x - tk * tiles_n) * kTileN;
    if (blockIdx.x == 0 && tid == 0) *one = 1.0f;
    const int64_t gn = n0 + wj * kCols, gk = k0 + 8 * kr;
    const bool col_live = gn < p.n;
    uint32_t w[8];
    const uint8_t* src = static_cast<const uint8_t*>(p.w) + (gk * p.w_ld + gn) * (32 / kCols) / 8;
    const int64_t pitch = p.w_ld * (32 / kCols) / 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = (col_live && gk + i < p.k) ? __ldcs(reinterpret_cast<const uint32_t*>(src + i * pitch)) : 0u;
    uint32_t sp[kPairs], op[kPairs];  // scale / offset of columns (j, j + kCols / 2)
    {
        const int64_t g = p.group_size > 0 ? min(gk, p.k - 1) / p.group_size : 0;
        const int64_t at = g * p.scale_sg + (col_live ? gn : 0) * p.scale_sn;
        const uint16_t *sc = reinterpret_cast<const uint16_t*>(p.scale) + at, *of = reinterpret_cast<const uint16_t*>(p.offset) + at;
#pragma unroll
        for (int j = 0; j < kPairs; ++j) {
            sp[j] = (uint32_t)__ldg(sc + j * p.scale_sn) | ((uint32_t)__ldg(sc + (j + kPairs) * p.scale_sn) << 16);
            op[j] = kOff ? (uint32_t)__ldg(of + j * p.scale_sn) | ((uint32_t)__ldg(of + (j + kPairs) * p.scale_sn) << 16) : 0u;
        }
    }
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) {
        const int at = (4 * kr + rp) ^ wj;
#pragma unroll
        for (int j = 0; j < kPairs; ++j) {
            // the codes of columns j and j + kCols / 2 in the low bits of the halves
            const uint32_t c0 = w[2 * rp] >> ((kW == MixW::kInt4 ? 4 : 8) * j), c1 = w[2 * rp + 1] >> ((kW == MixW::kInt4 ? 4 : 8) * j);
            uint32_t t0 = mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(c0), sp[j], op[j]);
            uint32_t t1 = mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(c1), sp[j], op[j]);
            if (kW == MixW::kE4m3) {
                t0 = fix_nan(t0, c0);
                t1 = fix_nan(t1, c1);
            }
            if (gk + 2 * rp >= p.k) t0 = 0u;  // rows past k are zeros in the image (an offset would make them something else)
            if (gk + 2 * rp + 1 >= p.k) t1 = 0u;
            tile[(wj * kCols + j) * 32 + at] = prmt(t0, t1, 0x5410);
            tile[(wj * kCols + j + kPairs) * 32 + at] = prmt(t0, t1, 0x7632);
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = tid; e < kTileN * 8; e += NT) {
        const int nn = e >> 3, c = e & 7, x = nn / kCols;  // column, 16-byte piece (8 k), its word column
        const int64_t on = n0 + nn, ok = k0 + c * 8;
        uint4 v = *reinterpret_cast<const uint4*>(&tile[nn * 32 + ((c ^ (x >> 2)) << 2)]);
        if (x & 1) v = make_uint4(v.y, v.x, v.w, v.z);
        if (x & 2) v = make_uint4(v.z, v.w, v.x, v.y);
        if (on < p.n && ok < kp) *reinterpret_cast<uint4*>(dst + on * kp + ok) = v;
    }
}

// Weight stored (n,k): the destination has the same orientation. A thread turns 32-bit words of a column into 16 (int4) or 8 bytes of
// pairs, four words in flight, words of a warp side by side; a block is one column's stretch, so scales cost no division per word.
// (n, k) = (18432, 7168) int4: 91 us one element at a time, 330 MB.
template <MixW kW, bool kBf16, bool kOff>
__global__ void __launch_bounds__(NT) wq_dequant_nk_kernel_fast(const OpsnnWqbmmParams p, uint16_t* __restrict__ dst, int64_t kp, float* __restrict__ one,
                                                                uint32_t chunks)
{
    pdl_trigger();
    pdl_wait();
    constexpr int kPer = kW == MixW::kInt4 ? 8 : 4;  // weights in a word
    const uint32_t row = blockIdx.x / chunks, chunk = blockIdx.x - row * chunks;
    if (blockIdx.x == 0 && threadIdx.x == 0) *one = 1.0f;
    const uint32_t words = (uint32_t)(p.k / kPer), w0 = chunk * (4 * NT) + threadIdx.x, group = p.group_size > 0 ? (uint32_t)p.group_size : 0x7FFFFFFFu;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(p.w) + (int64_t)row * p.w_ld * (32 / kPer) / 8);
    uint32_t w[4], sc[4], of[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t at = w0 + i * NT;
        if (at >= words) continue;
        w[i] = __ldcs(src + at);
        const int64_t s = (int64_t)(at * kPer / group) * p.scale_sg + (int64_t)row * p.scale_sn;
        sc[i] = __ldg(reinterpret_cast<const uint16_t*>(p.scale) + s);
        of[i] = kOff ? __ldg(reinterpret_cast<const uint16_t*>(p.offset) + s) : 0u;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t at = w0 + i * NT;
        if (at >= words) continue;
        const uint32_t s2 = sc[i] | (sc[i] << 16), o2 = of[i] | (of[i] << 16);
        uint32_t o[kPer / 2];
#pragma unroll
        for (int j = 0; j < kPer / 2; ++j) {
            // weights 2 j and 2 j + 1: nibbles of byte j (it and the word shifted by four), or bytes 2 j and 2 j + 1
            const uint32_t c = kW == MixW::kInt4 ? prmt(w[i], w[i] >> 4, (uint32_t)(j | ((4 + j) << 8))) : prmt(w[i], 0u, j == 0 ? 0x4140u : 0x4342u);
            o[j] = mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(c), s2, o2);
            if (kW == MixW::kE4m3) o[j] = fix_nan(o[j], c);
        }
        uint16_t* d = dst + (int64_t)row * kp + (int64_t)at * kPer;
        if constexpr (kPer == 8) *reinterpret_cast<uint4*>(d) = make_uint4(o[0], o[1], o[2], o[3]);
        else *reinterpret_cast<uint2*>(d) = make_uint2(o[0], o[1]);
    }
}

template <MixW kW>
void dequant_fast(const OpsnnWqbmmParams* p, uint16_t* dst, int64_t kp, float* one, cudaStream_t stream)
{
    constexpr int kPer = kW == MixW::kInt4 ? 8 : 4;
    const bool bf = p->x_dtype == ACL_BF16, off = p->offset != nullptr;
    auto go = [&](auto bf_c, auto off_c) {
        constexpr bool kB = decltype(bf_c)::value, kO = decltype(off_c)::value && kW != MixW::kE4m3;
        if (p->trans_w) {
            const uint32_t chunks = (uint32_t)((p->k / kPer + 4 * NT - 1) / (4 * NT));
            launch_dependent(wq_dequant_nk_kernel_fast<kW, kB, kO>, dim3((unsigned)(p->n * chunks)), NT, 0, stream, *p, dst, kp, one, chunks);
        } else {
            const uint32_t tiles_n = (uint32_t)((p->n + 32 * kPer - 1) / (32 * kPer));
            launch_dependent(wq_dequant_kn_kernel<kW, kB, kO>, dim3((unsigned)(tiles_n * ((p->k + 63) / 64))), NT, 0, stream, *p, dst, kp, one, tiles_n);
        }
    };
    if (bf && off) go(std::true_type{}, std::true_type{});
    else if (bf) go(std::true_type{}, std::false_type{});
    else if (off) go(std::false_type{}, std::true_type{});
    else go(std::false_type{}, std::false_type{});
}

// Layouts of the two kernels above.
bool dequant_fast_takes(const OpsnnWqbmmParams* p)
{
    if (env("OPSNN_WQ_PREFILL_SIMPLE") || p->scale_dtype == ACL_FLOAT8_E8M0 || (reinterpret_cast<uintptr_t>(p->w) & 3) != 0) return false;
    if (p->w_dtype != ACL_INT4 && p->w_dtype != ACL_INT8 && p->w_dtype != ACL_FLOAT8_E4M3FN) return false;
    if (p->w_dtype == ACL_FLOAT8_E4M3FN && p->offset != nullptr) return false;
    const int per = p->w_dtype == ACL_INT4 ? 8 : 4;
    if (p->w_ld % per != 0 || p->k >= ((int64_t)1 << 30)) return false;
    if (p->trans_w) return p->k % per == 0 && p->group_size % per == 0 && p->n * ((p->k / per + 4 * NT - 1) / (4 * NT)) <= 0x7FFFFFFF;
    return p->n % per == 0 && p->group_size % 8 == 0 && ((p->n + 32 * per - 1) / (32 * per)) * ((p->k + 63) / 64) <= 0x7FFFFFFF;
}

// fp8 weights stored (k,n) that the kernels above do not take (e5m2, or with an offset): a thread owns one 32-bit word (4 columns) over 4 consecutive k rows, the two row
// pairs of a column leave as packed words; 64 x 64 tile with 33-word rows. Needs n % 4 == 0, word-aligned rows,
// group_size % 4 == 0 and scales in x's dtype.
template <bool kBf16>
__global__ void __launch_bounds__(NT) wq_dequant_nk_bytes_kernel(const OpsnnWqbmmParams p, uint16_t* __restrict__ dst, int64_t kp,
                                                                 float* __restrict__ one)
{
    __shared__ uint32_t tile[TN][TK / 2 + 1];
    const int tid = threadIdx.x;
    const int64_t tiles_n = (p.n + TN - 1) / TN;
    const int64_t k0 = ((int64_t)blockIdx.x / tiles_n) * TK, n0 = ((int64_t)blockIdx.x % tiles_n) * TN;
    if (blockIdx.x == 0 && tid == 0) *one = 1.0f;
    const int wj = tid & 15, kq = tid >> 4;
    const int64_t gn = n0 + wj * 4, gk = k0 + 4 * kq;
    const bool col_live = gn < p.n;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = (col_live && gk + i < p.k) ? __ldcs(reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(p.w) + (gk + i) * p.w_ld + gn)) : 0u;
    float sc[4], of[4];
    const bool has_off = p.offset != nullptr;
    {
        const int64_t g = p.group_size > 0 ? min(gk, p.k - 1) / p.group_size : 0;
        const int64_t sidx = g * p.scale_sg + (col_live ? gn : 0) * p.scale_sn;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            sc[j] = load_x<kBf16>(p.scale, sidx + j * p.scale_sn);
            of[j] = has_off ? load_x<kBf16>(p.offset, sidx + j * p.scale_sn) : 0.f;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t byte = (w[i] >> (8 * j)) & 0xFFu;
            v[i] = fp8_to_float((uint8_t)byte, p.w_dtype);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float a = v[2 * h], b = v[2 * h + 1];
            if (has_off) {
                const float2 r = unpack2<kBf16>(pack2<kBf16>(__fadd_rn(a, of[j]), __fadd_rn(b, of[j])));
                a = r.x;
                b = r.y;
            }
            tile[wj * 4 + j][2 * kq + h] = pack2<kBf16>(__fmul_rn(a, sc[j]), __fmul_rn(b, sc[j]));
        }
    }
    __syncthreads();
    uint32_t* out = reinterpret_cast<uint32_t*>(dst);
    for (int e = tid; e < TN * (TK / 2); e += NT) {
        const int nn = e >> 5, c = e & 31;
        const int64_t on = n0 + nn, ok = k0 + 2 * c;
        if (on < p.n && ok < kp) out[(on * kp + ok) >> 1] = tile[nn][c];
    }
}

// fp4 / fp8 weight stored (n,k) that the kernel above does not take: the destination has the same orientation, so a
// thread dequantises one 32-bit word - kPer consecutive k of one column (8 for 4-bit, 4 for 8-bit weights) - and stores it as
// one 16- / 8-byte piece. One scale / offset per word (groups are multiples of kPer, or per-channel).
template <bool kBf16, int kPer>
__global__ void __launch_bounds__(NT) wq_dequant_nk_rows_kernel(const OpsnnWqbmmParams p, uint16_t* __restrict__ dst, int64_t kp,
                                                                float* __restrict__ one)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *one = 1.0f;
    const int64_t wpr = p.k / kPer, total = p.n * wpr;  // words per row
    const bool has_off = p.offset != nullptr;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t nn = i / wpr, kw = i % wpr, kk = kw * kPer;
        const uint32_t word = __ldcs(reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(p.w) + (nn * p.w_ld + kk) * (32 / kPer) / 8));
        const int64_t g = p.group_size > 0 ? kk / p.group_size : 0;
        const int64_t sidx = g * p.scale_sg + nn * p.scale_sn;
        const float sc = load_x<kBf16>(p.scale, sidx), of = has_off ? load_x<kBf16>(p.offset, sidx) : 0.f;
        uint32_t outw[kPer / 2];
#pragma unroll
        for (int h = 0; h < kPer / 2; ++h) {
            float a, b;
            if (kPer == 8) {
                const uint32_t n0 = (word >> (8 * h)) & 0xFu, n1 = (word >> (8 * h + 4)) & 0xFu;
                a = fp4_e2m1_to_float((uint8_t)n0);
                b = fp4_e2m1_to_float((uint8_t)n1);
            } else {
                const uint32_t b0 = (word >> (16 * h)) & 0xFFu, b1 = (word >> (16 * h + 8)) & 0xFFu;
                a = fp8_to_float((uint8_t)b0, p.w_dtype);
                b = fp8_to_float((uint8_t)b1, p.w_dtype);
            }
            if (has_off) {
                const float2 r = unpack2<kBf16>(pack2<kBf16>(__fadd_rn(a, of), __fadd_rn(b, of)));
                a = r.x;
                b = r.y;
            }
            outw[h] = pack2<kBf16>(__fmul_rn(a, sc), __fmul_rn(b, sc));
        }
        uint16_t* o = dst + nn * kp + kk;
        if (kPer == 8) *reinterpret_cast<uint4*>(o) = make_uint4(outw[0], outw[1], outw[kPer / 2 - 2], outw[kPer / 2 - 1]);
        else *reinterpret_cast<uint2*>(o) = make_uint2(outw[0], outw[1]);
    }
}

int64_t padded_k(const OpsnnWqbmmParams* p) { return (p->k + 7) / 8 * 8; }

// The matmul the pre-pass leaves behind, as parameters of the quantised-matmul launcher.
void gemm_view(const OpsnnWqbmmParams* p, OpsnnQmmParams* q, void* wdeq, const void* one)
{
    *q = OpsnnQmmParams{};
    q->mode = OPSNN_QMM_DEQ;
    q->a_dtype = q->b_dtype = q->out_dtype = p->x_dtype;
    q->bias_dtype = p->bias != nullptr ? p->bias_dtype : -1;
    q->scale_b_dtype = ACL_FLOAT;
    q->trans_a = 0;
    q->trans_b = 1;
    q->batch = 1; q->m = p->m; q->n = p->n; q->k = p->k;
    q->a = p->x; q->a_ld = p->x_ld;
    q->b = wdeq; q->b_ld = padded_k(p);
    q->scale_b = one; q->scale_b_len = 1;
    q->group_m = q->group_n = q->group_k = 1;
    q->bias = p->bias;
    q->out = p->y; q->out_ld = p->y_ld; q->out_bs = p->m * p->y_ld;
}

}  // namespace

uint64_t wqbmm_prefill_image_size(const OpsnnWqbmmParams* p)
{
    return (uint64_t)p->n * (uint64_t)padded_k(p) * 2u + 512u;  // dequantised weight, alignment slack, the unit scale
}

uint64_t wqbmm_prefill_workspace_size(const OpsnnWqbmmParams* p) { return p->prep_w != nullptr ? 0 : wqbmm_prefill_image_size(p); }

bool wqbmm_prefill_eligible(const OpsnnWqbmmParams* p)
{
    if (env("OPSNN_WQ_NO_PREFILL")) return false;
    if (p->x_dtype != ACL_BF16 && p->x_dtype != ACL_FLOAT16) return false;
    if (p->w_dtype != ACL_INT4 && p->w_dtype != ACL_INT8 && p->w_dtype != ACL_FLOAT8_E4M3FN && p->w_dtype != ACL_FLOAT8_E5M2 &&
        p->w_dtype != ACL_FLOAT4_E2M1)
        return false;
    if (p->m < 1 || p->n < 1 || p->k < 1) return false;
    if (p->x_ld % 8 != 0 || (p->x != nullptr && (reinterpret_cast<uintptr_t>(p->x) & 15) != 0)) return false;
    OpsnnQmmParams q;
    gemm_view(p, &q, reinterpret_cast<void*>(uintptr_t(256)), reinterpret_cast<const void*>(uintptr_t(256)));
    q.a = nullptr;  // alignment of x was checked above; the stand-in addresses only serve the shape rules
    return qmm_umma_eligible(&q);
}

// The dequantisation pre-pass alone: the (n, padded k) 16-bit weight and the unit scale behind it, at `ws` (256-byte aligned).
int32_t wqbmm_prefill_prepass(const OpsnnWqbmmParams* p, uint8_t* ws, cudaStream_t stream)
{
    const int64_t kp = padded_k(p);
    uint16_t* wdeq = reinterpret_cast<uint16_t*>(ws);
    float* one = reinterpret_cast<float*>(ws + (((uint64_t)p->n * kp * 2u + 15u) & ~(uint64_t)15u));
    const int64_t tiles = ((p->n + TN - 1) / TN) * ((p->k + TK - 1) / TK);
    if (tiles > 0x7FFFFFFF) return (int32_t)cudaErrorInvalidConfiguration;
    const bool bf = p->x_dtype == ACL_BF16;
    const bool four = p->w_dtype == ACL_FLOAT4_E2M1, fp8 = p->w_dtype == ACL_FLOAT8_E4M3FN || p->w_dtype == ACL_FLOAT8_E5M2;
    const int per = four ? 8 : 4;
    const bool rows_path = (four || fp8) && p->trans_w && p->k % per == 0 && p->w_ld % per == 0 && (p->group_size == 0 || p->group_size % per == 0) &&
                           p->scale_dtype != ACL_FLOAT8_E8M0 && (reinterpret_cast<uintptr_t>(p->w) & 3) == 0 &&
                           env("OPSNN_WQ_PREFILL_SIMPLE") == nullptr;
    if (dequant_fast_takes(p)) {
        if (p->w_dtype == ACL_INT4) dequant_fast<MixW::kInt4>(p, wdeq, kp, one, stream);
        else if (p->w_dtype == ACL_INT8) dequant_fast<MixW::kInt8>(p, wdeq, kp, one, stream);
        else dequant_fast<MixW::kE4m3>(p, wdeq, kp, one, stream);
    } else if (rows_path) {
        const int64_t work = p->n * (p->k / per);
        int64_t grid = (work + NT - 1) / NT;
        if (grid > 148 * 32) grid = 148 * 32;
        if (grid < 1) grid = 1;
        if (bf && four) wq_dequant_nk_rows_kernel<true, 8><<<(unsigned)grid, NT, 0, stream>>>(*p, wdeq, kp, one);
        else if (bf) wq_dequant_nk_rows_kernel<true, 4><<<(unsigned)grid, NT, 0, stream>>>(*p, wdeq, kp, one);
        else if (four) wq_dequant_nk_rows_kernel<false, 8><<<(unsigned)grid, NT, 0, stream>>>(*p, wdeq, kp, one);
        else wq_dequant_nk_rows_kernel<false, 4><<<(unsigned)grid, NT, 0, stream>>>(*p, wdeq, kp, one);
    } else if (fp8 && !p->trans_w &&
               p->n % 4 == 0 && p->w_ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p->w) & 3) == 0 &&
               (p->group_size == 0 || p->group_size % 4 == 0) && p->scale_dtype != ACL_FLOAT8_E8M0 &&
               env("OPSNN_WQ_PREFILL_SIMPLE") == nullptr) {
        if (bf) wq_dequant_nk_bytes_kernel<true><<<(unsigned)tiles, NT, 0, stream>>>(*p, wdeq, kp, one);
        else wq_dequant_nk_bytes_kernel<false><<<(unsigned)tiles, NT, 0, stream>>>(*p, wdeq, kp, one);
    } else if (bf) wq_dequant_nk_kernel<true><<<(unsigned)tiles, NT, 0, stream>>>(*p, wdeq, kp, one);
    else wq_dequant_nk_kernel<false><<<(unsigned)tiles, NT, 0, stream>>>(*p, wdeq, kp, one);
    note_launch("wq_dequant_nk");
    return (int32_t)cudaGetLastError();
}

int32_t wqbmm_prefill_launch(const OpsnnWqbmmParams* p, cudaStream_t stream)
{
    uint8_t* ws;
    if (p->prep_w != nullptr) {
        if ((reinterpret_cast<uintptr_t>(p->prep_w) & 255) != 0) return (int32_t)cudaErrorInvalidValue;
        ws = const_cast<uint8_t*>(static_cast<const uint8_t*>(p->prep_w));  // prepared once: nothing to do per call
    } else {
        if (p->workspace == nullptr || p->workspace_size < wqbmm_prefill_workspace_size(p)) return (int32_t)cudaErrorInvalidValue;
        ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p->workspace) + 255) & ~(uintptr_t)255);
        const int32_t rc = wqbmm_prefill_prepass(p, ws, stream);
        if (rc != 0) return rc;
    }
    const int64_t kp = padded_k(p);
    uint16_t* wdeq = reinterpret_cast<uint16_t*>(ws);
    float* one = reinterpret_cast<float*>(ws + (((uint64_t)p->n * kp * 2u + 15u) & ~(uint64_t)15u));
    OpsnnQmmParams q;
    gemm_view(p, &q, wdeq, one);
    if (!qmm_umma_eligible(&q)) return (int32_t)cudaErrorInvalidValue;
    return qmm_umma_launch(&q, stream);
}

}  // namespace opsnn
