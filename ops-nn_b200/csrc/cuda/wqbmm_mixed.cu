// Weight-only quant matmul: the packed weight is dequantised straight into tensor memory and multiplied there
// (tcgen05 kind::f16 with A in TMEM), one pass over the weight for up to 128 rows of x. No 16-bit image of the weight in HBM.
//
// Reference: weight_quant_batch_matmul_v2/op_kernel/arch35/weight_quant_batch_matmul_v2_reg_base_common.h:164-286 (vector cores
// dequantise tile by tile, the cube unit multiplies in bf16 / fp16); arithmetic of the golden wqbmmv2_kernel_golden.py:199-297:
//   w' = rn_x(rn_x(w + offset) * scale),  y = rn_x(sum_k x * w' (fp32) + bias)
//
// Orientation: D^T = W'^T x^T. The MMA's 128 rows are weight columns, its N is the rows of x (16 ... 128 of them, a multiple of 16), so
// the tensor core's work shrinks with m while the dequantisation - what bounds this kernel - is done once whatever m is.
//   CTA tile: 256 weight columns (two M = 128 accumulators) x N rows of x; persistent, one CTA per SM (all 512 TMEM columns).
//   The (tile, k stage of 128 rows) pairs lie in one line, and every CTA has a contiguous piece of it (mix_plan):
//     a tile into `split` equal pieces, launched as a cluster: every CTA sums the rows of the tile that the cluster's CTAs send it (mix_push); or
//     stream-k, all CTAs the same share: a tile that several CTAs share is combined through workspace by whichever arrives last.
//   Pieces are added in the order of k either way (deterministic; in the second nobody waits for anybody).
//   warps 0-15   dequantise. Warp w serves TMEM lanes 32 (w % 4) .. (a hardware rule), accumulator half (w / 4) % 2, and every other
//                stage (w / 8). packed words -> registers (ldmatrix.trans for (k,n) storage: a register then holds nibbles /
//                bytes of k rows 2q, 2q + 1, already the pair that a TMEM cell of A wants; a row per lane for (n,k) storage) ->
//                the decode kernels' pair arithmetic -> tcgen05.st.
//   warps 16-19  epilogue of all but the CTA's last tile, overlapped with the next tile's main loop; the last is finished by warps 0-15.
//   warp 20      TMA producer (packed weight, x, scale / offset rows), warps 21 and 22 MMA issuers, one for each accumulator half.
// A operand buffers: four of 128 k x 128 columns (64 TMEM columns each) at columns 256-511, one for either half of two stages in turn;
// accumulators at 0-255 (two sets while N <= 64).
// What bounds it: no single unit, but a stage's chain of steps: wait for the packed words, shared loads, arithmetic, wait for the A buffer, stores
// to tensor memory and their wait, arrival, MMAs, commit. Every wait, even for a barrier long completed, is 80 clocks, and a third to a half of
// the schedulers' cycles have no warp that could issue. us, weights from HBM, whole / without the arithmetic / without the MMAs / without the stores
// (results kept alive by a XOR and a compare, which cost more than the stores did): 16 x 8192 x 28672 int4 with offset 37.4 / 29.2 / 35.5 / 39.5,
// 77 x 7168 x 18432 int4 (n,k) fp16 24.6 / 21.5 / 21.2 / 26.9, 4 x 4096 x 14336 int8 (n,k) fp16 15.7 / 15.0 / 15.2 / 17.9, 1 x 4096 x 4096
// 9.2 / 7.6 / 8.6 / 9.5. So the stores cost less than that, the arithmetic a twentieth to a fifth, and what is left is the chain and the two ends.
// Therefore buffers change hands by the stage and not by 64 rows of k, a warp arrives under a predicate instead of a branch, and scales that allow
// it save the magic number (MixFast). Before / after, the same calls, weights from HBM (in brackets out of L2): 39.4 / 37.5, 27.9 / 24.5
// (25.9 / 21.7), 17.7 / 15.7 (15.5 / 13.1), 9.5 / 9.2 (9.1 / 8.8).
// Clocks, 16 x 8192 x 28672: 65000 a CTA, 3900 until the first stage is there, 6000 from the last sums to the end; the busiest unit, the 16-bit pipe, works for 37400. A
// warp waits for A buffers 7000, but others compute meanwhile: a third stage of buffers in place of the second accumulator set took 38.6 us, with
// two 38.3 by the same code, 37.6 by this.
// Every wait is bounded; a wait that gives up raises the CTA's abort flag, records a code and the CTA tears down (TMEM freed).
#include <algorithm>
#include <cstdio>
#include <type_traits>

#include "common.cuh"
#include "sm100_ptx.cuh"
#include "wq_convert.cuh"
#include "wqbmm_decode_common.cuh"

namespace opsnn {

int32_t umma_prelaunch_check(cudaStream_t stream, unsigned int** mirror);

namespace {

constexpr int kMixTileN = 256;
constexpr int kMixDqWarps = 16, kMixEpWarps = 4;
constexpr int kMixMmaWarps = 2;
constexpr int kMixThreads = (kMixDqWarps + kMixEpWarps + 1 + kMixMmaWarps) * 32;
constexpr int kMixMaxRows = 128;   // rows of x per pass over the weight
constexpr int kMixABufs = 4;
constexpr uint32_t kMixACol = 256;  // first TMEM column of the A buffers
constexpr int kMixMaxStages = 16;
constexpr int kMixSmemMax = 225 * 1024;

// How a CTA sums its piece over k. The tensor core cuts each addition to an accumulator off instead of rounding it, so the error grows with
// the length of the chain of MMAs on one accumulator. Up to 48 rows of x the streaming kernels, which cut k over more CTAs, chain a quarter
// as many MMAs as a piece here has; the sums are to be as exact as theirs (outputs that are not the rounded exact sum, fp16,
// 16 x 8192 x 28672: 2.1 % as one chain, 0.8 % there, 0.65 % here).
//   kChain    one accumulator: the chain is no longer than that of the matmul on a dequantised weight
//   kCopies   4 or 8 accumulators take turns, MMA by MMA (they fit for 16 rows, or 32 where one set is enough)
//   kChunks   the accumulator is added to a sum in tensor memory, with rounding, every few stages, by the epilogue warps
enum class MixSum { kChain, kCopies, kChunks };

struct MixArgs {
    int32_t m, t_tiles, rows;  // rows: rows of x per tile (N of the MMA)
    uint32_t n, k, kb;         // kb: k stages per tile
    uint32_t grid, units;      // units = tiles * kb, cut into `grid` contiguous pieces; units * grid < 2^32
    uint32_t copies, chunk;    // MixSum: accumulators, k stages to a chunk
    uint32_t split;            // > 0: grid = tiles * split, so that a tile is `split` whole pieces, launched as a cluster; 0: stream-k
    uint32_t stages, stage_bytes, x_off, sc_off, sc_rows, sc_vec;  // sc_rows: scale rows a stage needs (2: groups that end inside a stage)
    const void* scale;
    const void* offset;
    int64_t scale_sg, scale_sn;
    uint32_t group;       // rows of k per group (one group: at least k)
    const void* bias;
    int32_t bias_dtype;
    void* y;
    int64_t y_ld;
    float4* part;                  // [2 grid][2 rows / 4][128]
    unsigned long long* count;     // [tiles] (nonce << 8) | arrivals
    unsigned long long nonce;
    uint32_t idesc;
    volatile unsigned int* status_host;  // pinned mirror of the error word that later launches look at; nullptr: none
    uint32_t test_stop;  // tests of the give-up path only: stages that a CTA's producer copies before it stops; otherwise all
};

__device__ unsigned int g_mix_status = 0;

// (Out of line: a dozen calls of it are in the kernel, none of them on the way that it takes.)
static __device__ __noinline__ void mix_report_at(volatile unsigned int* status_host, volatile uint32_t* abort_flag, unsigned int code)
{
    *abort_flag = 1u;
    atomicCAS(&g_mix_status, 0u, code);
    if (status_host != nullptr) {
        *status_host = code;
        __threadfence_system();
    }
}
__device__ __forceinline__ void mix_report(const MixArgs& a, volatile uint32_t* abort_flag, unsigned int code) { mix_report_at(a.status_host, abort_flag, code); }

__device__ __forceinline__ void mix_tma_2d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_addr, int32_t c0, int32_t c1)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_addr), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void mix_arrive(uint32_t bar_addr)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_addr) : "memory");
}
// Has the phase completed? Does not wait.
__device__ __forceinline__ bool mix_test(uint32_t bar_addr, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar_addr), "r"(parity)
                 : "memory");
    return ok != 0;
}
// A wait for a whole tile's sums, which nobody waits for in turn: the four epilogue warps sleep between polls, else their polling is a fifth of all
// instructions issued. Not for the sums of a chunk, due every stage or few, with the last of which the CTA ends: asleep for them, 17 - 32 rows
// with chunks of one stage took 12.4 us for 11.8 (24 x 4096 x 8192 int4 with offset; 24 x 2048 x 16384 int8 12.5 / 12.0), with longer ones 0.5 - 1 %
// more (24 x 4096 x 14336 16.15 / 16.02).
static __device__ __noinline__ bool mix_wait_asleep(uint32_t bar_addr, uint32_t parity, volatile uint32_t* abort_flag)
{
    const uint32_t limit = ptx::g_spin_limit / 64u + 1u;
    for (uint32_t i = 0; i < limit; ++i) {
        if (ptx::mbar_try_wait_a(bar_addr, parity)) return true;
        if (*abort_flag != 0u) return false;
        __nanosleep(1000);
    }
    *abort_flag = 1u;
    return false;
}
// Bounded wait with one answer for the warp: what follows it is .sync.aligned.
__device__ __forceinline__ bool mix_wait(uint32_t bar_addr, uint32_t parity, volatile uint32_t* abort_flag)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tvote.sync.all.pred q, p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(bar_addr), "r"(parity)
        : "memory");
    return done != 0u || __all_sync(0xffffffffu, ptx::mbar_wait_slow_a<>(bar_addr, parity, abort_flag));
}
// A warp's arrival: one for all its lanes' earlier accesses (predicated: no branch).
__device__ __forceinline__ void mix_arrive_warp(uint32_t bar_addr, int lane)
{
    __syncwarp();
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar_addr), "r"(lane) : "memory");
}
// Barrier of kThreads threads that tells all of them whether every one came with `ok`: they go on, or leave, together.
template <int kBar, int kThreads>
__device__ __forceinline__ bool mix_all_ok(bool ok)
{
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, %2, %3, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r)
                 : "r"(ok ? 1u : 0u), "n"(kBar), "n"(kThreads)
                 : "memory");
    return r != 0u;
}
__device__ __forceinline__ void mix_init(uint32_t bar_addr, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_addr), "r"(count) : "memory");
}
__device__ __forceinline__ void mix_ldsm4_trans(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ uint4 mix_lds128(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
// 16 TMEM lanes x 16 columns: register pairs (2c, 2c + 1) hold, in lane (g, q), rows g and g + 8 of columns 4c + q
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// 32 TMEM lanes x 8 columns, a lane's columns in its registers
__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// 32 TMEM lanes x 32 columns of 32-bit sums
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// kind::f16, A (128 x 16) in tensor memory, B in shared memory
__device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same weights in fewer instructions, where a lane's scales allow it. Integer and 16-bit-pair instructions both take two clocks a warp, and
// a pair of int4 weights was 1.75 - 2.25 of the first and two of the second.
// A code (less its sign flip: w + z, z = 8 or 128) left in the low bits of a 16-bit half is a subnormal there: it reads as (w + z) * 2^-E, E by the
// bit it starts at, without a magic number to take off again. So fma(code, s * 2^E, -z * s) = rn(w * s): product and subtrahend are exact,
// one rounding, one instruction. Needs s * 2^E finite: |s| < 2^-5 (bf16; fp16 int4), 2^-8 (fp16 int8). (e4m3: its magnitude bits read as
// w * 2^-120 / 2^-8 already, and the product with s * 2^120 / 2^8 is the one rounding; |s| < 2^8.)
// A warp one of whose lanes has other scales in a stage (infinities and NaN among them) takes the general arithmetic for that stage: us, weights from
// HBM, short / general / the kernel before there was a choice: 16 x 8192 x 28672 int4 bf16 (k,n) 32.8 / 33.7 / 34.5, (n,k) 36.5 / 40.6 / 43.0,
// 77 x 7168 x 18432 int4 (n,k) fp16 24.6 / 26.9 / 28.0, int8 (k,n) bf16 29.4 / 30.7 / 30.6, 4 x 4096 x 14336 int8 (n,k) bf16 15.7 / 18.1 / 19.3.
// With an offset (two roundings) the same idea saves no 16-bit instruction, and what the scaled offsets cost is more than the two shifts it
// saves (16 x 8192 x 28672 bf16: 38.6 -> 40.0 us): general arithmetic.
template <MixW kW, bool kNK, bool kBf16, bool kOff>
struct MixFast {
    using N = Num<kBf16>;
    static constexpr bool kHas = !kOff;
    static constexpr uint32_t pow2(int e)
    {
        const uint32_t v = kBf16 ? (uint32_t)(127 + e) << 7 : (uint32_t)(15 + e) << 10;
        return v | (v << 16);
    }
    static constexpr int kTop = kBf16 ? 127 : 15;  // the largest power of two
    // E of the code of word position b ((k,n) int4: the word's columns alternate between two)
    static constexpr int exponent(int b)
    {
        if (kW == MixW::kE4m3) return kBf16 ? 120 : 8;
        if (kW == MixW::kInt8) return kBf16 ? 133 : 24;
        if (kNK) return kBf16 ? 133 : 21;
        return kBf16 ? ((b & 1) ? 129 : 133) : ((b & 1) ? 17 : 21);
    }
    static constexpr uint32_t kZero = kW == MixW::kInt4 ? (kBf16 ? 0xC100C100u : 0xC800C800u) : (kBf16 ? 0xC300C300u : 0xD800D800u);  // -z
    __device__ __forceinline__ static uint32_t lop(uint32_t a, uint32_t mask, uint32_t flip)
    {
        uint32_t v;
        asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(v) : "r"(a), "r"(mask), "r"(flip));
        return v;
    }
    // Scales of two columns (or one, twice) whose word positions are b0 (low half) and b1: multiplier and addend of `pair` below. Returns whether
    // they allow it.
    __device__ __forceinline__ static bool prepare(uint32_t sc, int b0, int b1, uint32_t& mul, uint32_t& add)
    {
        if (kW == MixW::kE4m3) {
            mul = N::mul(sc, pow2(exponent(0)));
        } else {
            const uint32_t rest = (pow2(exponent(b0) > kTop ? exponent(b0) - kTop : 0) & 0xFFFFu) | (pow2(exponent(b1) > kTop ? exponent(b1) - kTop : 0) & 0xFFFF0000u);
            mul = N::mul(N::mul(sc, pow2(kTop)), rest);
        }
        add = N::mul(sc, kZero);
        // an infinity or NaN carries into bit 15 or 31
        return (((mul & 0x7FFF7FFFu) + (kBf16 ? 0x00800080u : 0x04000400u)) & 0x80008000u) == 0u;
    }
    __device__ __forceinline__ static uint32_t pair(uint32_t code, uint32_t mul, uint32_t add) { return kW == MixW::kE4m3 ? N::mul(code, mul) : N::fma(code, mul, add); }
    // (k,n) int4: the pair of column b of a word (its nibble b and nibble 4 + b)
    __device__ __forceinline__ static void codes4(uint32_t w, uint32_t (&c)[4])
    {
        const uint32_t lo = kBf16 ? w : w << 3, hi = kBf16 ? w >> 8 : w >> 5;
        constexpr uint32_t m0 = kBf16 ? 0x000F000Fu : 0x00780078u, f0 = kBf16 ? 0x00080008u : 0x00400040u;
        constexpr uint32_t m1 = kBf16 ? 0x00F000F0u : 0x07800780u, f1 = kBf16 ? 0x00800080u : 0x04000400u;
        c[0] = lop(lo, m0, f0);
        c[1] = lop(lo, m1, f1);
        c[2] = lop(hi, m0, f0);
        c[3] = lop(hi, m1, f1);
    }
    // (n,k) int4: the pairs of nibbles 2 b and 2 b + 1. A byte's zero top bit, replicated, is the half's upper byte.
    __device__ __forceinline__ static void codes4_nk(uint32_t w, uint32_t (&c)[4])
    {
        const uint32_t a = kBf16 ? lop(w, 0x0F0F0F0Fu, 0x08080808u) : lop(w << 3, 0x78787878u, 0x40404040u);
        const uint32_t d = kBf16 ? lop(w >> 4, 0x0F0F0F0Fu, 0x08080808u) : lop(w >> 1, 0x78787878u, 0x40404040u);
        c[0] = prmt(a, d, 0xC480u);
        c[1] = prmt(a, d, 0xD591u);
        c[2] = prmt(a, d, 0xE6A2u);
        c[3] = prmt(a, d, 0xF7B3u);
    }
    // (k,n), 8 bits: the pair of column b; (n,k), 8 bits: the pair of bytes 2 b, 2 b + 1
    __device__ __forceinline__ static void codes8(uint32_t w, uint32_t (&c)[2])
    {
        if constexpr (kW == MixW::kE4m3) {
            c[0] = e4m3_bits(kNK ? prmt(w, 0u, 0x4140u) : w);
            c[1] = e4m3_bits(kNK ? prmt(w, 0u, 0x4342u) : w >> 8);
        } else if constexpr (kNK) {
            const uint32_t x = w ^ 0x80808080u;
            c[0] = prmt(x, 0u, 0x4140u);
            c[1] = prmt(x, 0u, 0x4342u);
        } else {
            c[0] = lop(w, 0x00FF00FFu, 0x00800080u);
            c[1] = lop(w >> 8, 0x00FF00FFu, 0x00800080u);
        }
    }
    __device__ __forceinline__ static uint32_t e4m3_bits(uint32_t p)
    {
        uint32_t v = (p << (kBf16 ? 4 : 7)) & (kBf16 ? 0x07F007F0u : 0x3F803F80u);
        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(p << 8), "n"(0x80008000), "r"(v));
        return v;
    }
};

// One stage: 128 rows of k x 256 columns. (With 64-row stages the producer's and the MMA issuer's fixed cost per stage showed.)
template <MixW kW>
struct MixCfg {
    static constexpr int kBits = kW == MixW::kInt4 ? 4 : 8;
    static constexpr int kBK = 128;
    static constexpr int kWBytes = kMixTileN * kBK * kBits / 8;
};

// TMEM lane (within a warp's 32) -> weight column (within the warp's 32)
template <MixW kW, bool kNK>
__device__ __forceinline__ int mix_col_of_lane(int l)
{
    if (kNK) return l;
    return kW == MixW::kInt4 ? 4 * (l & 7) + (l >> 3) : 16 * (l >> 4) + 2 * (l & 7) + ((l >> 3) & 1);
}

// The rows past `live` of a unit of A (64 rows of k, two to a column) cleared, this warp's 32 lanes of it at `abase`. A stage's rows past k
// are zero in x and in the packed weight, but their dequantised weight is (0 + offset) * scale, and zero times an infinity is NaN.
__device__ __forceinline__ void mix_clear_past(uint32_t abase, uint32_t live)
{
    tmem_st_wait();
#pragma unroll 1
    for (uint32_t c = live / 32u * 16u; c < 32u; c += 16u) {
        uint32_t v[16], lo[8], hi[8];
        ptx::tmem_ld16(abase + c, v);
        ptx::tmem_ld_wait();
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) {
            const uint32_t row = 2u * (c + i);
            const uint32_t kept = row + 1u < live ? v[i] : (row < live ? v[i] & 0xFFFFu : 0u);
            if (i < 8) lo[i] = kept;
            else hi[i - 8] = kept;
        }
        tmem_st_32x32b_x8(abase + c, lo);
        tmem_st_32x32b_x8(abase + c + 8u, hi);
    }
}

// A CTA's contiguous piece of the (tile, stage) line.
__device__ __forceinline__ uint32_t mix_begin(const MixArgs& a, uint32_t c) { return c * a.units / a.grid; }
__device__ __forceinline__ uint32_t mix_owner(const MixArgs& a, uint32_t unit)
{
    uint32_t c = unit * a.grid / a.units;
    while (mix_begin(a, c + 1) <= unit) ++c;
    while (mix_begin(a, c) > unit) --c;
    return c;
}

// One column of 16 rows of y.
template <bool kBf16>
__device__ __forceinline__ void mix_store(const MixArgs& a, uint32_t n, uint32_t r0, const float (&f)[16])
{
    if (n >= a.n) return;
    const float b = a.bias != nullptr ? load_as_float(a.bias, n, a.bias_dtype) : 0.f;
    uint16_t* y = reinterpret_cast<uint16_t*>(a.y) + (int64_t)r0 * a.y_ld + n;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if ((int)r0 + i >= a.m) break;
        const float v = a.bias != nullptr ? __fadd_rn(f[i], b) : f[i];
        y[(int64_t)i * a.y_ld] = kBf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
    }
}

// 16 columns of a piece's sums. kMany: of `n` accumulators (1 or an even number), `step` columns apart.
template <bool kMany>
__device__ __forceinline__ void mix_sums16(uint32_t acc, uint32_t n, uint32_t step, float (&f)[16])
{
    uint32_t v[16];
    ptx::tmem_ld16(acc, v);
    if constexpr (!kMany) {
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
    } else {
        uint32_t q[16];
        if (n > 1u) ptx::tmem_ld16(acc + step, q);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = n > 1u ? __fadd_rn(__uint_as_float(v[i]), __uint_as_float(q[i])) : __uint_as_float(v[i]);
#pragma unroll 1
        for (uint32_t j = 2; j < n; j += 2) {
            ptx::tmem_ld16(acc + j * step, v);
            ptx::tmem_ld16(acc + (j + 1u) * step, q);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] = __fadd_rn(f[i], __fadd_rn(__uint_as_float(v[i]), __uint_as_float(q[i])));
        }
    }
}

// sum = acc (the first chunk) or sum + acc, `cols` columns (a multiple of 32) of this warp's lanes.
__device__ __forceinline__ void mix_promote(uint32_t acc, uint32_t sum, uint32_t cols, bool first)
{
#pragma unroll 1
    for (uint32_t c = 0; c < cols; c += 32) {
        uint32_t v[32], q[32];
        ptx::tmem_ld32(acc + c, v);
        if (!first) {
            ptx::tmem_ld32(sum + c, q);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__fadd_rn(__uint_as_float(q[i]), __uint_as_float(v[i])));
        } else {
            ptx::tmem_ld_wait();
        }
        tmem_st_32x32b_x32(sum + c, v);
    }
    tmem_st_wait();
}

// A finished piece of tile t (stages kb .. kb + cnt of it) out of the accumulators at TMEM address `acc` (this warp's lanes): stored
// if it is the whole tile, else parked in workspace, and combined by whoever arrives last. Run by kWarps warps (four per TMEM lane
// quarter and column share): 4 of them beside the main loop, or 16 at the end of the CTA's work.
template <bool kBf16, int kWarps, bool kMany>
__device__ __forceinline__ void mix_finish(const MixArgs& a, uint32_t acc, uint32_t n_acc, uint32_t step, uint32_t t, uint32_t cnt, int col, int qd, int lane, int share, bool leader,
                                           volatile uint32_t* s_last, volatile uint32_t* abort_flag)
{
    constexpr int kBar = kWarps == 4 ? 1 : 2;
    constexpr uint32_t kStep = 16u * (kWarps / 4);
    const uint32_t rows = (uint32_t)a.rows, tn = t / (uint32_t)a.t_tiles, tt = t - tn * (uint32_t)a.t_tiles;
    const uint32_t n0 = tn * kMixTileN + col;
    const bool whole = cnt == a.kb;
    const uint32_t slot = (rows / 2) * 128u, row = (uint32_t)(qd * 32 + lane);
    unsigned long long* const cnt_p = a.count + t;
    unsigned long long cur = 0ull;
    if (leader && !whole) cur = *reinterpret_cast<volatile unsigned long long*>(cnt_p);  // (a guess, here while the sums are parked)
    float4* mine = a.part + (2u * blockIdx.x + (t == mix_begin(a, blockIdx.x) / a.kb ? 0u : 1u)) * slot + row;
#pragma unroll 1
    for (uint32_t hc = 16u * share; hc < 2u * rows; hc += kStep) {
        float f[16];
        mix_sums16<kMany>(acc + hc, n_acc, step, f);
        if (whole) {
            const uint32_t h = hc >= rows ? 1u : 0u;
            mix_store<kBf16>(a, n0 + 128u * h, tt * rows + hc - h * rows, f);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) __stcg(mine + (hc / 4 + i) * 128u, make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]));
        }
    }
    if (whole) return;
    const uint32_t c0 = mix_owner(a, t * a.kb), c1 = mix_owner(a, (t + 1u) * a.kb - 1u);  // the CTAs whose pieces meet this tile
    asm volatile("bar.sync %0, %1;" ::"n"(kBar), "n"(kWarps * 32) : "memory");  // all of this CTA's partial sums are written
    if (leader) {
        __threadfence();  // for all of them: the barrier puts them before it
        unsigned long long want = 0ull;
        bool done = false;
        for (int it = 0; it < 4096 && !done; ++it) {  // at most c1 - c0 other CTAs can get in between
            want = ((cur >> 8) == a.nonce) ? cur + 1ull : ((a.nonce << 8) | 1ull);
            const unsigned long long prev = atomicCAS(cnt_p, cur, want);
            done = prev == cur;
            cur = prev;
        }
        if (!done) mix_report(a, abort_flag, (4u << 8) | 2u);
        const bool last = done && (uint32_t)(want & 0xFFull) == c1 - c0 + 1u;
        if (last) *reinterpret_cast<volatile unsigned long long*>(cnt_p) = 0ull;  // a replay of this launch starts clean
        __threadfence();
        *s_last = last ? 1u : 0u;
    }
    asm volatile("bar.sync %0, %1;" ::"n"(kBar), "n"(kWarps * 32) : "memory");
    if (*s_last == 0u) return;
#pragma unroll 1
    for (uint32_t hc = 16u * share; hc < 2u * rows; hc += kStep) {
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = 0.f;
#pragma unroll 2
        for (uint32_t c = c0; c <= c1; ++c) {
            // only the first of a CTA's tiles can be shared with the CTAs before it: its other shared tile starts with it
            const uint32_t sl = 2u * c + (c == c0 && mix_begin(a, c) / a.kb != t ? 1u : 0u);
            const float4* p = a.part + sl * slot + (hc / 4) * 128u + row;
            float4 q[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = __ldcg(p + i * 128);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                f[4 * i] += q[i].x; f[4 * i + 1] += q[i].y; f[4 * i + 2] += q[i].z; f[4 * i + 3] += q[i].w;
            }
        }
        const uint32_t h = hc >= rows ? 1u : 0u;
        mix_store<kBf16>(a, n0 + 128u * h, tt * rows + hc - h * rows, f);
    }
}

// A tile that is `split` whole pieces is dealt to the CTAs in parts of four live rows x 64 columns, mix_share parts each in order of rank; every CTA
// stores its sums of them in their owner's shared memory, [piece][part of the share][64 columns][4 rows] fp32 in the place of the stages (at
// most 143 KB, less than the stages of any form), and the owner adds the pieces up. Bound by latency: two cluster barriers, a remote store, and
// code that runs once and so is fetched while everybody waits for it: fewer instructions here are microseconds. us, graph replay, weights from
// HBM, before (sums, abort flags and bias fetched out of the others' memory and HBM between two barriers) / dealt as four rows of all columns, a
// piece alone stored through shared memory too / now: 1 x 4096 x 4096 8.45 / 8.28 / 7.99, 4 x 4096 x 14336 int8 (n,k) fp16 16.3 / 15.5 / 15.2,
// 4 x 11776 x 8192 with bias 20.2 / 19.1 / 19.2, 6 x 3072 x 1728 int8 7.63 / 7.68 / 6.83, 21 x 1792 x 25440 (n,k) 16.2 / 15.3 / 14.7, 173 x 1280 x 17184
// (n,k) 14.1 / 14.1 / 11.9. (Sent row by row 77 x 7168 x 18432 lost 2 %.)
__device__ __forceinline__ uint32_t mix_parts(uint32_t live) { return (live + 3u) / 4u * (kMixTileN / 64); }
__device__ __forceinline__ uint32_t mix_share(uint32_t live, uint32_t split) { return (mix_parts(live) + split - 1u) / split; }
constexpr uint32_t kMixPartBytes = 64u * 16u;

// This CTA's sums (sixteen warps) to their owners. Within a part they lie in the order of the TMEM lanes (`lane`, of 128) and not of the columns, which in
// (k,n) storage are permuted: in their order eight neighbouring lanes met in two of a shared memory's eight 16-byte banks (int4; in four, 8 bits):
// us, graph replay, fetched / sent in the columns' order / in the lanes': 128 x 2048 x 12544 int4 15.7 / 16.3 / 15.6, 244 x 2560 x 8544 16.9 / 17.4 / 16.7.
// With many rows (kTurn) each CTA begins a quarter of its sums further on than the one before it: all beginning with the first rows, they were all sending
// to the same few owners. fetched / from the first / further on and with four pieces on their way to an owner's registers instead of two, where they
// go worked out before the cluster meets: 128 rows, eight pieces, 2048 x 4608 int4 12.8 / 13.0 / 11.9, five, 2048 x 7424 12.7 / 13.4 / 12.6 (112 rows 12.1 / 12.8 /
// 11.9), seven, 339 x 1408 x 1696 11.9 / 12.1 / 11.2, fourteen, 2048 x 2560 13.0 / 12.2 / 11.4. (16 rows do not need it, and its code cost them 1 %: 4 x 4096 x
// 14336 int8 (n,k) 15.1 / 15.2, without it, worked out before the cluster meets, 15.0.)
struct MixPush {
    uint32_t live, per, inverse, mine, hc, left;
};
template <bool kTurn>
__device__ __forceinline__ MixPush mix_push_plan(const MixArgs& a, uint32_t smem, uint32_t live, uint32_t rank, uint32_t lane, uint32_t share)
{
    MixPush q;
    q.live = live;
    q.per = mix_share(live, a.split);
    q.inverse = 65535u / q.per + 1u;  // part * per < 2^16: the quotient is exact
    q.mine = smem + rank * q.per * kMixPartBytes + (lane & 63u) * 16u;
    q.hc = 16u * share + (kTurn ? 64u * (rank & 3u) : 0u);
    q.left = (2u * (uint32_t)a.rows + 48u - 16u * share) / 64u;
    return q;
}
template <bool kMany, bool kTurn>
__device__ __forceinline__ void mix_push(const MixArgs& a, uint32_t acc, uint32_t n_acc, uint32_t step, const MixPush& q, uint32_t lane, uint32_t share)
{
    const uint32_t rows = (uint32_t)a.rows, live = q.live, per = q.per, inverse = q.inverse, mine = q.mine;
#pragma unroll 1
    for (uint32_t left = q.left, hc = q.hc; kTurn ? left != 0u : hc < 2u * rows; --left, hc += 64u) {
        if (kTurn && hc >= 2u * rows) hc = 16u * share;  // (round to the first)
        const uint32_t h = hc >= rows ? 1u : 0u, r0 = hc - h * rows;
        if (r0 >= live) continue;
        float f[16];
        mix_sums16<kMany>(acc + hc, n_acc, step, f);
        uint32_t part = r0 + 2u * h + (lane >> 6), owner = part * inverse >> 16, slot = part - owner * per;
#pragma unroll
        for (uint32_t i = 0; i < 16; i += 4) {
            if (r0 + i >= live) break;
            uint32_t to;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine + slot * kMixPartBytes), "r"(owner));
            for (slot += 4u; slot >= per; slot -= per) ++owner;  // the next four rows
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(f[i]), "f"(f[i + 1]), "f"(f[i + 2]), "f"(f[i + 3]) : "memory");
        }
    }
}

// This CTA's share of its tile: the pieces added in their order, + bias (s_bias: the tile's columns), stored (512 threads, one column of four rows each).
struct MixOwn {
    uint32_t live, per, first, n0, col;  // first: of this CTA's parts; n0: the tile's first column; col: of a part, this thread's
    uint16_t* out;                       // the tile's first row
};
template <MixW kW, bool kNK>
__device__ __forceinline__ MixOwn mix_own(const MixArgs& a, uint32_t t, uint32_t live, uint32_t rank, uint32_t tid)
{
    const uint32_t tn = t / (uint32_t)a.t_tiles, tt = t - tn * (uint32_t)a.t_tiles;
    MixOwn q;
    q.live = live;
    q.per = mix_share(live, a.split);
    q.first = rank * q.per;
    q.n0 = tn * kMixTileN;
    q.col = (tid & 32u) + (uint32_t)mix_col_of_lane<kW, kNK>((int)(tid & 31u));
    q.out = reinterpret_cast<uint16_t*>(a.y) + (int64_t)(tt * (uint32_t)a.rows) * a.y_ld;
    return q;
}
template <bool kBf16, int kAtOnce>
__device__ __forceinline__ void mix_sum_and_store(const MixArgs& a, uint32_t smem, const MixOwn& q, uint32_t tid, const float* s_bias)
{
    const uint32_t live = q.live, per = q.per, parts = mix_parts(live), col = q.col;
    uint16_t* out = q.out;
#pragma unroll 1
    for (uint32_t slot = tid / 64u; slot < per; slot += kMixDqWarps * 32 / 64) {
        const uint32_t part = q.first + slot, row = part & ~3u, n = q.n0 + (part & 3u) * 64u + col;
        if (part >= parts || n >= a.n) continue;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t at = smem + slot * kMixPartBytes + tid % 64u * 16u;
#pragma unroll kAtOnce
        for (uint32_t j = 0; j < a.split; ++j, at += per * kMixPartBytes) {
            const uint4 p = mix_lds128(at);
            v[0] += __uint_as_float(p.x); v[1] += __uint_as_float(p.y); v[2] += __uint_as_float(p.z); v[3] += __uint_as_float(p.w);
        }
        uint16_t* y = out + (int64_t)row * a.y_ld + n;
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r) {
            if (row + r >= live) break;
            const float f = a.bias != nullptr ? __fadd_rn(v[r], s_bias[(part & 3u) * 64u + col]) : v[r];
            y[(int64_t)r * a.y_ld] = kBf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(f)) : __half_as_ushort(__float2half_rn(f));
        }
    }
}

// kRagged: k is not a whole number of stages. (As a question asked in every stage it cost the calls with whole ones up to 3 %: 4 x 4096 x 14336
// int8 18.1 -> 18.7 us.)
template <MixW kW, bool kNK, bool kBf16, bool kOff, MixSum kSum, bool kRagged>
__global__ void __launch_bounds__(kMixThreads, 1)
wqbmm_mixed_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ MixArgs a)
{
    using C = MixCfg<kW>;
    using F = MixFast<kW, kNK, kBf16, kOff>;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    extern __shared__ uint8_t dyn_raw[];
    const uint32_t smem0 = (ptx::smem_u32(dyn_raw) + 1023u) & ~1023u;
    // `full` has two barriers a slot, used in turn: so one belongs to one group of dequantising warps, which sees every one of its phases (with an
    // odd number of slots a group meets a slot in every second phase only, and a parity does not tell a phase from the one two before it)
    __shared__ __align__(8) uint64_t s_bars[3 * kMixMaxStages + 2 * kMixABufs + 6];
    __shared__ uint32_t s_tmem;
    __shared__ volatile uint32_t s_abort;
    __shared__ volatile uint32_t s_last[2];
    __shared__ volatile uint32_t s_bad;   // a CTA of the cluster gave up a wait
    __shared__ float s_bias[kMixTileN];  // of the tile's columns, where its pieces are a cluster
    const uint32_t full0 = ptx::smem_u32(s_bars), empty0 = full0 + 16u * kMixMaxStages;
    const uint32_t afull0 = empty0 + 8u * kMixMaxStages, aempty0 = afull0 + 8u * kMixABufs;
    const uint32_t dfull0 = aempty0 + 8u * kMixABufs, dempty0 = dfull0 + 16u, fin0 = dempty0 + 16u, fsum0 = fin0 + 8u;
    volatile uint32_t* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        s_abort = 0u;
        s_bad = 0u;
        for (uint32_t i = 0; i < a.stages; ++i) {
            mix_init(full0 + 8u * i, 1u);
            mix_init(full0 + 8u * (a.stages + i), 1u);
            mix_init(empty0 + 8u * i, kMixDqWarps / 2 + kMixMmaWarps);
        }
        for (int i = 0; i < kMixABufs; ++i) {
            mix_init(afull0 + 8u * i, 4u);
            mix_init(aempty0 + 8u * i, 1u);
        }
        for (int i = 0; i < 2; ++i) {
            mix_init(dfull0 + 8u * i, kMixMmaWarps);
            mix_init(dempty0 + 8u * i, kMixEpWarps);
        }
        // the last piece's sums, and those of its chunks before the last (barriers of their own: the warps that wait for them have not
        // followed the others' phases)
        mix_init(fin0, kMixMmaWarps);
        mix_init(fsum0, kMixEpWarps);
        ptx::fence_mbar_init();
        ptx::fence_proxy_async();
    }
    if (warp == kMixDqWarps + kMixEpWarps + 1) ptx::tmem_alloc(&s_tmem, 512);
    if (warp == kMixDqWarps + kMixEpWarps && lane == 0) {
        ptx::tma_prefetch_desc(&map_w);
        ptx::tma_prefetch_desc(&map_x);
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_trigger();
    pdl_wait();  // nothing another kernel may have written is read before this

    const uint32_t u_begin = mix_begin(a, blockIdx.x), u_end = mix_begin(a, blockIdx.x + 1);
    const uint32_t stages = a.stages, stage_bytes = a.stage_bytes;
    auto rows_live = [&] { return min((uint32_t)a.rows, (uint32_t)a.m - (blockIdx.x / a.split) % (uint32_t)a.t_tiles * (uint32_t)a.rows); };  // rows of x in the (only) tile
    const uint32_t xunit = (uint32_t)a.rows * 128u;  // bytes of x per 64-row unit of k
    // accumulators: two sets where there is room, beside them the sums of the chunks that are done
    const uint32_t d_one = 2u * (uint32_t)a.rows, d_set = kSum == MixSum::kCopies ? a.copies * d_one : d_one;
    const bool two_d = kSum == MixSum::kChain ? a.rows <= 64 : (kSum == MixSum::kCopies ? a.split == 0u : a.rows <= 32);
    const uint32_t d_sum = two_d ? 2u * d_set : d_set;

    if (warp == kMixDqWarps + kMixEpWarps) {
        // ======================= TMA producer =======================
        // Its time per stage bounds the stream: no division but one by the group size, everything else counted along.
        uint32_t s = 0, par = 0, second = 0;  // second: the slot's other barrier
        const uint32_t kbs = a.kb, rows = (uint32_t)a.rows, n_all = a.n, x_off = a.x_off, sc_off = a.sc_off, nrows_sc = a.sc_rows, k_last = a.k - 1u, group = a.group;
        const int64_t scale_sg = a.scale_sg;
        const uint16_t *scale = reinterpret_cast<const uint16_t*>(a.scale), *offset = reinterpret_cast<const uint16_t*>(a.offset);
        const uint32_t t0 = u_begin / kbs;
        uint32_t kb = u_begin - t0 * kbs;
        uint32_t n0 = t0 / (uint32_t)a.t_tiles, r0 = (t0 - n0 * (uint32_t)a.t_tiles) * rows;
        const uint32_t r_end = (uint32_t)(a.t_tiles * a.rows);
        n0 *= kMixTileN;
        const uint32_t sc_rows = kNK ? 0u : nrows_sc * (kOff ? 2u : 1u), u_stop = u_begin + min(u_end - u_begin, a.test_stop);
        for (uint32_t u = u_begin; u < u_stop; ++u) {
            if (!mix_wait(empty0 + 8u * s, par ^ 1u, abort_flag)) {
                mix_report(a, abort_flag, (1u << 8) | 1u);
                break;
            }
            if (ptx::elect_one()) {
                const uint32_t k0 = kb * C::kBK, fb = full0 + 8u * (s + second), dst = smem0 + s * stage_bytes;
                const uint32_t sc_bytes = min((uint32_t)kMixTileN, n_all - n0) * 2u;
                ptx::mbar_expect_tx_a(fb, (uint32_t)C::kWBytes + 2u * xunit + sc_bytes * sc_rows);
                if (kNK) {
                    mix_tma_2d(dst, &map_w, fb, (int32_t)(k0 * C::kBits / 8), (int32_t)n0);
                } else {
                    mix_tma_2d(dst, &map_w, fb, (int32_t)(n0 * C::kBits / 8), (int32_t)k0);
                    if (C::kBits == 8) mix_tma_2d(dst + C::kWBytes / 2, &map_w, fb, (int32_t)n0 + 128, (int32_t)k0);
                }
                mix_tma_2d(dst + x_off, &map_x, fb, (int32_t)k0 * 2, (int32_t)r0);
                mix_tma_2d(dst + x_off + xunit, &map_x, fb, (int32_t)k0 * 2 + 128, (int32_t)r0);
                if (!kNK) {
                    uint32_t sd = dst + sc_off;
                    for (uint32_t i = 0; i < nrows_sc; ++i) {
                        const int64_t at = (int64_t)(min(k0 + 64u * i, k_last) / group) * scale_sg + n0;
                        ptx::bulk_load_a(sd, scale + at, sc_bytes, fb);
                        if (kOff) ptx::bulk_load_a(sd + kMixTileN * 2, offset + at, sc_bytes, fb);
                        sd += kMixTileN * 4;
                    }
                }
            }
            __syncwarp();
            if (++s == stages) { s = 0; par ^= 1u; second ^= stages; }
            if (++kb == kbs) {
                kb = 0;
                r0 += rows;
                if (r0 == r_end) { r0 = 0; n0 += kMixTileN; }
            }
        }
    } else if (warp > kMixDqWarps + kMixEpWarps) {
        // ======================= MMA issuers =======================
        // Two warps, one for each accumulator half (and so on schedulers of their own): a buffer's MMAs are few and short (N = 16: 20 clocks
        // each), so what else it costs shows: a wait for a barrier that has long completed is 80 clocks of latency. So the next buffer's
        // barrier is looked at before this one's MMAs are issued, and the stage's own barrier not at all: the dequantising warps have
        // waited for it before they arrived on `afull`.
        const uint64_t db = ptx::make_smem_desc(smem0 + a.x_off, 0, 1024, 2);
        const uint32_t b_lo = (uint32_t)db;
        const uint64_t b_hi = db & 0xFFFFFFFF00000000ull;
        const uint32_t h = (uint32_t)(warp - (kMixDqWarps + kMixEpWarps + 1));
        uint32_t s = 0, ab = h, apar = 0, dbuf = 0, dpar = 0;
        bool ok = true, ready = false;
        const uint32_t kbs = a.kb, rows = (uint32_t)a.rows, idesc = a.idesc, chunk = kSum == MixSum::kChunks ? a.chunk : kbs;
        const uint32_t copies = a.copies, turn1 = d_one, turn2 = 2u * d_one, turn3 = 3u * d_one;
        uint32_t u = u_begin, kb = u_begin % kbs;
        while (u < u_end && ok) {
            const uint32_t cnt = min(min(kbs - kb, u_end - u), chunk);
            if (!mix_wait(dempty0 + 8u * dbuf, dpar ^ 1u, abort_flag)) {
                mix_report(a, abort_flag, (2u << 8) | 1u);
                break;
            }
            const uint32_t d0 = tmem + dbuf * d_set + h * rows;
            uint32_t acc = 0u;
            for (uint32_t i = 0; i < cnt; ++i) {
                if (!__all_sync(0xffffffffu, ready) && !mix_wait(afull0 + 8u * ab, apar, abort_flag)) {
                    mix_report(a, abort_flag, (2u << 8) | 3u);
                    ok = false;
                    break;
                }
                const uint32_t a0 = tmem + kMixACol + ab * 64u, freed = aempty0 + 8u * ab;
                ab ^= 2u;
                if (ab == h) apar ^= 1u;
                ready = mix_test(afull0 + 8u * ab, apar);
                ptx::tc_fence_after();
                if (ptx::elect_one()) {
                    const uint32_t bl = b_lo + ((s * stage_bytes) >> 4);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {
                        uint32_t d = d0, go_on = kk == 0 ? acc : 1u;
                        if (kSum == MixSum::kCopies) {
                            d += (kk & 3) == 0 ? 0u : ((kk & 3) == 1 ? turn1 : ((kk & 3) == 2 ? turn2 : turn3));
                            if (kk >= 4) d += copies == 8u ? 4u * d_one : 0u;
                            go_on = kk < 4 || copies == 8u ? acc : 1u;
                        }
                        umma_f16_ta(d, a0 + kk * 8, b_hi | (uint64_t)(bl + (kk >= 4 ? xunit >> 4 : 0u) + 2u * (kk & 3)), idesc, go_on);
                    }
                    ptx::umma_commit_a(freed);
                    ptx::umma_commit_a(empty0 + 8u * s);
                }
                __syncwarp();
                acc = 1u;
                if (++s == stages) s = 0;
            }
            if (!ok) break;
            u += cnt;
            if (ptx::elect_one()) ptx::umma_commit_a(u < u_end ? dfull0 + 8u * dbuf : fin0);
            __syncwarp();
            kb += cnt;
            if (kb == kbs) kb = 0;
            if (two_d) dbuf ^= 1u;
            if (dbuf == 0u) dpar ^= 1u;
        }
    } else if (warp < kMixDqWarps) {
        // ======================= dequantisation =======================
        // Eight warps take the even stages of the CTA's piece, eight the odd ones: one wait, one read of the scales and one release per
        // 128 rows of k. A warp fills its lanes of one A buffer a stage (its half), so the four buffers alternate between the two groups.
        const int qd = warp & 3, h = (warp >> 2) & 1;
        const uint32_t grp = (uint32_t)warp >> 3;
        const int g = lane >> 2;
        const uint32_t tlane = (uint32_t)(qd * 32) << 16;
        const int wcol = h * 128 + qd * 32;  // the warp's first column in the tile
        const uint32_t ab = 2u * grp + h;  // the warp's A buffer, shared with the three other lane quarters
        uint32_t s = grp, fs = grp, par = 0, apar = 0;  // slot and its barrier (two or more slots)
        bool ok = true;
        const bool two_rows = a.sc_rows == 2u;  // a stage's units have scale rows of their own
        const uint32_t k_in_last = a.k - (a.kb - 1u) * (uint32_t)C::kBK;  // rows of k in a tile's last stage
        uint32_t ragged = (u_begin / a.kb + 1u) * a.kb - 1u;  // the next last stage
        // (n,k) storage: the lane's own scales and offsets, an iteration ahead. The group of a stage is counted along (a division per
        // stage was a tenth of this loop): k0 = first row of the stage, k0_in = its place in group gi.
        uint32_t sc_next[2] = {0, 0}, of_next[2] = {0, 0};
        uint32_t t = 0, kb = 0, k0_in = 0, gi = 0;
        const uint32_t step_g = 2u * C::kBK / a.group, step_in = 2u * C::kBK - step_g * a.group;
        int64_t col_at = 0;
        // rows of scales whose groups lie side by side: eight groups in one 16-byte load (a lane's 2-byte loads each drag a sector of their
        // own through L2, as many bytes as the weight itself)
        const bool vec = a.sc_vec != 0;
        uint4 sc_v = make_uint4(0, 0, 0, 0), of_v = sc_v;
        uint32_t have = 0xFFFFFFFFu;
        uint32_t sel = 0;
        auto pick = [](const uint4& v, uint32_t i, uint32_t (&out)[2]) {  // group i; where a stage has two (i even), the next one too
            const uint32_t w = (i & 4u) ? ((i & 2u) ? v.w : v.z) : ((i & 2u) ? v.y : v.x);
            out[0] = prmt(w, w, (i & 1u) ? 0x3232u : 0x1010u);
            out[1] = prmt(w, w, 0x3232u);
        };
        auto seek = [&](uint32_t unit) {
            t = unit / a.kb;
            kb = unit - t * a.kb;
            gi = (kb * (uint32_t)C::kBK) / a.group;
            k0_in = kb * (uint32_t)C::kBK - gi * a.group;
            col_at = (int64_t)min((t / (uint32_t)a.t_tiles) * kMixTileN + wcol + lane, a.n - 1u) * a.scale_sn;
            have = 0xFFFFFFFFu;
        };
        auto fetch = [&]() {
            if (vec) {
                sel = gi & 7u;
                if ((gi >> 3) != have) {
                    have = gi >> 3;
                    sc_v = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.scale) + col_at + 8u * have));
                    if (kOff) of_v = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.offset) + col_at + 8u * have));
                }
                return;
            }
            int64_t at = (int64_t)gi * a.scale_sg + col_at;
            sc_next[0] = __ldg(reinterpret_cast<const uint16_t*>(a.scale) + at);
            if (kOff) of_next[0] = __ldg(reinterpret_cast<const uint16_t*>(a.offset) + at);
            if (two_rows && k0_in + 64u >= a.group && kb * (uint32_t)C::kBK + 64u < a.k) at += a.scale_sg;
            sc_next[1] = two_rows ? __ldg(reinterpret_cast<const uint16_t*>(a.scale) + at) : sc_next[0];
            if (kOff) of_next[1] = two_rows ? __ldg(reinterpret_cast<const uint16_t*>(a.offset) + at) : of_next[0];
        };
        if (kNK && u_begin + grp < u_end) {
            seek(u_begin + grp);
            fetch();
        }
        for (uint32_t u = u_begin + grp; u < u_end; u += 2) {
            uint32_t sc_n[2], of_n[2];
            if constexpr (kRagged) {
                while (ragged < u) ragged += a.kb;
            }
            if (kNK) {
                if (vec) {
                    pick(sc_v, sel, sc_n);
                    if (kOff) pick(of_v, sel, of_n);
                    else of_n[0] = of_n[1] = 0u;
                } else {
#pragma unroll
                    for (int un = 0; un < 2; ++un) {
                        sc_n[un] = sc_next[un] | (sc_next[un] << 16);
                        of_n[un] = of_next[un] | (of_next[un] << 16);
                    }
                }
                if (u + 2 < u_end) {
                    kb += 2;
                    if (kb < a.kb) {
                        k0_in += step_in;
                        gi += step_g;
                        if (k0_in >= a.group) { k0_in -= a.group; ++gi; }
                    } else {
                        seek(u + 2);
                    }
                    fetch();
                }
            }
            if (!mix_wait(full0 + 8u * fs, par, abort_flag)) {
                mix_report(a, abort_flag, (3u << 8) | 1u);
                ok = false;
                break;
            }
            const uint32_t base = smem0 + s * stage_bytes;
            // scales and offsets (or what MixFast makes of them) of the lane's columns: int4 4g .. 4g + 3, 8 bits 2g, 2g + 1 of each 16, or its one
            uint32_t sc[4], of[4];
            bool fast = false;
            auto load_scales = [&](uint32_t un) {
                const uint32_t at = base + a.sc_off + un * (kMixTileN * 4u) + 2u * wcol + (kW == MixW::kInt4 ? 8u * g : 4u * g);
                uint32_t r0, r1, o0 = 0, o1 = 0;
                if (kW == MixW::kInt4) {
                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(at) : "memory");
                    if (kOff) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(o0), "=r"(o1) : "r"(at + kMixTileN * 2) : "memory");
                } else {
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r0) : "r"(at) : "memory");
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r1) : "r"(at + 32u) : "memory");
                    if (kOff) {
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(o0) : "r"(at + kMixTileN * 2) : "memory");
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(o1) : "r"(at + kMixTileN * 2 + 32u) : "memory");
                    }
                }
                if constexpr (F::kHas) {
                    uint32_t m0, m1, a0, a1;
                    const bool f0 = F::prepare(r0, 0, 1, m0, a0), f1 = F::prepare(r1, 0, 1, m1, a1);
                    fast = __all_sync(0xffffffffu, f0 && f1);
                    if (fast) { r0 = m0; r1 = m1; o0 = a0; o1 = a1; }
                }
                sc[0] = prmt(r0, r0, 0x1010); sc[1] = prmt(r0, r0, 0x3232); sc[2] = prmt(r1, r1, 0x1010); sc[3] = prmt(r1, r1, 0x3232);
                of[0] = prmt(o0, o0, 0x1010); of[1] = prmt(o0, o0, 0x3232); of[2] = prmt(o1, o1, 0x1010); of[3] = prmt(o1, o1, 0x3232);
            };
            auto own_scales = [&](uint32_t un) {
                sc[0] = sc_n[un];
                of[0] = of_n[un];
                if constexpr (F::kHas) {
                    uint32_t m0, a0;
                    fast = __all_sync(0xffffffffu, F::prepare(sc[0], 0, 0, m0, a0));
                    if (fast) { sc[0] = m0; of[0] = a0; }
                }
            };
            if (kNK) own_scales(0);
            else load_scales(0);
            const int r = lane & 7, j = lane >> 3;
            // (k,n) int4: rows of 128 bytes; matrix j of an ldmatrix = rows 8 j .. of a half of 32, the warp's 16 bytes of the row
            uint32_t w4[4][4];
            if constexpr (!kNK && kW == MixW::kInt4) {
                const uint32_t at = base + (uint32_t)(8 * j + r) * 128u + (uint32_t)(((h * 4 + qd) ^ r) << 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) mix_ldsm4_trans(at + i * 32 * 128, w4[i]);
                if (!two_rows) mix_arrive_warp(empty0 + 8u * s, lane);  // the packed words and the scale rows of this stage are in registers
            }
            const uint32_t abase0 = tmem + kMixACol + ab * 64u + tlane;
            auto need_buffer = [&]() {  // the MMAs that read this A buffer's previous contents are done
                if (!mix_wait(aempty0 + 8u * ab, apar ^ 1u, abort_flag)) {
                    mix_report(a, abort_flag, (3u << 8) | 2u);
                    ok = false;
                }
                ptx::tc_fence_after();
            };
            auto unit = [&](auto fast_c, auto un_c) {  // 64 rows of packed words -> half of the A buffer
                constexpr bool kFast = decltype(fast_c)::value;
                constexpr int un = decltype(un_c)::value;
                const uint32_t abase = abase0 + un * 32u;
                // one word of four columns, or of one column's four bytes / eight nibbles
                auto word8 = [&](uint32_t w, int at, uint32_t& o0, uint32_t& o1) {
                    if constexpr (kFast) {
                        uint32_t c[2];
                        F::codes8(w, c);
                        o0 = F::pair(c[0], sc[at], of[at]);
                        o1 = kNK ? F::pair(c[1], sc[0], of[0]) : F::pair(c[1], sc[at + 1], of[at + 1]);
                    } else {
                        o0 = mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(kNK ? prmt(w, 0u, 0x4140) : w), sc[at], of[at]);
                        o1 = kNK ? mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(prmt(w, 0u, 0x4342)), sc[0], of[0])
                                 : mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(w >> 8), sc[at + 1], of[at + 1]);
                    }
                };
                if constexpr (!kNK) {
                    if constexpr (kW == MixW::kInt4) {
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            uint32_t o[2][8];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t w = w4[2 * un + half][i];
                                uint32_t c[4];
                                if constexpr (kFast) F::codes4(w, c);
#pragma unroll
                                for (int b = 0; b < 4; ++b) {
                                    if constexpr (kFast) o[b >> 1][2 * i + (b & 1)] = F::pair(c[b], sc[b], of[b]);
                                    else o[b >> 1][2 * i + (b & 1)] = mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(w >> (4 * b)), sc[b], of[b]);
                                }
                            }
                            if (un == 0 && half == 0) need_buffer();
                            tmem_st_16x128b_x4(abase + half * 16, o[0]);
                            tmem_st_16x128b_x4(abase + half * 16 + (16u << 16), o[1]);
                        }
                    } else {
                        const uint32_t box = base + h * (C::kWBytes / 2) + un * (64u * 128u) + (uint32_t)(8 * j + r) * 128u;
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
#pragma unroll
                            for (int cc = 0; cc < 2; ++cc) {
                                uint32_t w[4], o[8];
                                mix_ldsm4_trans(box + half * 32 * 128 + (uint32_t)(((2 * qd + cc) ^ r) << 4), w);
#pragma unroll
                                for (int i = 0; i < 4; ++i) word8(w[i], 2 * cc, o[2 * i], o[2 * i + 1]);
                                if (kW == MixW::kE4m3) {
                                    const uint32_t any = has_nan8(w[0]) | has_nan8(w[1]) | has_nan8(w[2]) | has_nan8(w[3]);
                                    if (any != 0u) {
#pragma unroll
                                        for (int i = 0; i < 4; ++i) {
                                            o[2 * i] = fix_nan(o[2 * i], w[i]);
                                            o[2 * i + 1] = fix_nan(o[2 * i + 1], w[i] >> 8);
                                        }
                                    }
                                    __syncwarp();
                                }
                                if (un == 0 && half == 0 && cc == 0) need_buffer();
                                tmem_st_16x128b_x4(abase + half * 16 + ((uint32_t)(16 * cc) << 16), o);
                            }
                        }
                    }
                } else {
                    const int row = wcol + lane;
                    if constexpr (kW == MixW::kInt4) {
                        const uint32_t rb = base + (uint32_t)row * 64u;
                        const uint32_t x = (uint32_t)(row >> 1) & 3u;  // 64-byte swizzle
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const uint4 v = mix_lds128(rb + (((2u * un + c) ^ x) << 4));
                            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                uint32_t o[8];
#pragma unroll
                                for (int i = 0; i < 2; ++i) {
                                    const uint32_t lo = w[2 * hh + i], hi = lo >> 4;
                                    uint32_t code[4];
                                    if constexpr (kFast) F::codes4_nk(lo, code);
#pragma unroll
                                    for (int b = 0; b < 4; ++b) {  // nibbles 2 b and 2 b + 1: byte b of the word and of the word shifted by four
                                        if constexpr (kFast) o[4 * i + b] = F::pair(code[b], sc[0], of[0]);
                                        else o[4 * i + b] = mix_scale<kBf16, kOff>(mix_exact<kW, kBf16>(prmt(lo, hi, (uint32_t)(b | ((4 + b) << 8)))), sc[0], of[0]);
                                    }
                                }
                                if (un == 0 && c == 0 && hh == 0) need_buffer();
                                tmem_st_32x32b_x8(abase + c * 16 + hh * 8, o);
                            }
                        }
                    } else {
                        const uint32_t rb = base + (uint32_t)row * 128u;
                        const uint32_t x = (uint32_t)row & 7u;  // 128-byte swizzle
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const uint4 v = mix_lds128(rb + (((4u * un + c) ^ x) << 4));
                            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                            uint32_t o[8];
#pragma unroll
                            for (int i = 0; i < 4; ++i) word8(w[i], 0, o[2 * i], o[2 * i + 1]);
                            if (kW == MixW::kE4m3) {
                                const uint32_t any = has_nan8(w[0]) | has_nan8(w[1]) | has_nan8(w[2]) | has_nan8(w[3]);
                                if (any != 0u) {
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        o[2 * i] = fix_nan(o[2 * i], prmt(w[i], 0u, 0x4140));
                                        o[2 * i + 1] = fix_nan(o[2 * i + 1], prmt(w[i], 0u, 0x4342));
                                    }
                                }
                                __syncwarp();
                            }
                            if (un == 0 && c == 0) need_buffer();
                            tmem_st_32x32b_x8(abase + c * 8, o);
                        }
                    }
                }
            };
            using U0 = std::integral_constant<int, 0>;
            using U1 = std::integral_constant<int, 1>;
            using Fast = std::bool_constant<F::kHas>;
            if (!two_rows) {  // (one branch for the stage)
                if (fast) {
                    unit(Fast{}, U0{});
                    unit(Fast{}, U1{});
                } else {
                    unit(std::false_type{}, U0{});
                    unit(std::false_type{}, U1{});
                }
            } else {  // groups that end inside a stage: scales for each unit
                if (fast) unit(Fast{}, U0{});
                else unit(std::false_type{}, U0{});
                if (kNK) own_scales(1);
                else load_scales(1);
                if (fast) unit(Fast{}, U1{});
                else unit(std::false_type{}, U1{});
            }
            if (!ok) break;
            if constexpr (kRagged) {
                if (u == ragged) {
                    if (k_in_last < 64u) mix_clear_past(abase0, k_in_last);
                    mix_clear_past(abase0 + 32u, k_in_last > 64u ? k_in_last - 64u : 0u);
                }
            }
            tmem_st_wait();
            ptx::tc_fence_before();
            mix_arrive_warp(afull0 + 8u * ab, lane);
            // (the packed words of the other layouts are read on the way)
            if (kNK || kW != MixW::kInt4 || two_rows) mix_arrive_warp(empty0 + 8u * s, lane);
            apar ^= 1u;
            fs += 2u;
            if (fs >= 2u * stages) { fs -= 2u * stages; par ^= 1u; }
            s = fs >= stages ? fs - stages : fs;
        }
        // the CTA's last (often only) piece: nothing is left to dequantise, all sixteen warps finish it
        const uint32_t t_first = u_begin / a.kb, t_last = (u_end - 1u) / a.kb;
        const uint32_t last_cnt = min(u_end - t_last * a.kb, u_end - u_begin);
        uint32_t before = t_last - t_first;  // accumulator sets used before the last one
        bool has_sum = false;
        if constexpr (kSum == MixSum::kChunks) {
            auto chunks = [&](uint32_t c) { return (c + a.chunk - 1u) / a.chunk; };
            const uint32_t n = chunks(last_cnt);
            has_sum = n > 1u;
            before = n - 1u + (t_first == t_last ? 0u : chunks((t_first + 1u) * a.kb - u_begin) + (t_last - t_first - 1u) * chunks(a.kb));
        }
        const uint32_t dbuf = two_d ? (before & 1u) : 0u;
        if (ok && (!mix_wait(fin0, 0u, abort_flag) || (has_sum && !mix_wait(fsum0, 0u, abort_flag)))) {
            mix_report(a, abort_flag, (3u << 8) | 3u);
            ok = false;
        }
        constexpr bool kMany = kSum != MixSum::kChain, kTurn = kSum != MixSum::kCopies;
        const uint32_t acc = tmem + tlane + dbuf * d_set;
        // (with chunks: the last one and the sum of those before it)
        const uint32_t n_acc = kSum == MixSum::kCopies ? a.copies : (has_sum ? 2u : 1u), step = kSum == MixSum::kCopies ? d_one : tmem + tlane + d_sum - acc;
        const int col = qd * 32 + mix_col_of_lane<kW, kNK>(lane);
        if (a.split > 1u) {
            // Its pieces ran as one thread-block cluster: where every CTA of it is done with its stages, the sums go to their owners. What a CTA that
            // gave up a wait sends is not used.
            ptx::tc_fence_after();
            __syncwarp();
            ptx::cluster_arrive();
            const MixPush plan = mix_push_plan<kTurn>(a, smem0, rows_live(), ptx::cluster_ctarank(), (uint32_t)(qd * 32 + lane), (uint32_t)warp >> 2);
            ptx::cluster_wait();
            mix_push<kMany, kTurn>(a, acc, n_acc, step, plan, (uint32_t)(qd * 32 + lane), (uint32_t)warp >> 2);
        } else if (mix_all_ok<2, kMixDqWarps * 32>(ok)) {
            ptx::tc_fence_after();
            mix_finish<kBf16, 16, kMany>(a, acc, n_acc, step, t_last, last_cnt, col, qd, lane, warp >> 2, threadIdx.x == 0, &s_last[1], abort_flag);
        }
    } else {
        // ======================= epilogue of all but the last piece, beside the main loop; chunks are added up =======================
        const int qd = warp & 3;
        const uint32_t tlane = (uint32_t)(qd * 32) << 16;
        const int col = qd * 32 + mix_col_of_lane<kW, kNK>(lane);
        const bool leader = warp == kMixDqWarps && lane == 0;
        uint32_t dbuf = 0, dpar = 0, u = u_begin, t = u_begin / a.kb, kb = u_begin - t * a.kb;
        if (a.split > 1u && a.bias != nullptr) {  // these warps have the time; read at the end it cost up to 0.6 us, by the dequantising warps 0.1 - 0.2
            for (uint32_t c = threadIdx.x - kMixDqWarps * 32; c < (uint32_t)kMixTileN; c += kMixEpWarps * 32)
                s_bias[c] = load_as_float(a.bias, min(t / (uint32_t)a.t_tiles * kMixTileN + c, a.n - 1u), a.bias_dtype);
        }
        auto next_set = [&](bool urgent) {  // waits for an accumulator set; the four warps go on, or leave, together
            const bool got = urgent ? mix_wait(dfull0 + 8u * dbuf, dpar, abort_flag) : __all_sync(0xffffffffu, mix_wait_asleep(dfull0 + 8u * dbuf, dpar, abort_flag));
            if (!got) mix_report(a, abort_flag, (4u << 8) | 1u);
            const bool ok = mix_all_ok<1, kMixEpWarps * 32>(got);
            ptx::tc_fence_after();
            return ok;
        };
        auto give_back = [&]() {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) mix_arrive(dempty0 + 8u * dbuf);
            if (two_d) dbuf ^= 1u;
            if (dbuf == 0u) dpar ^= 1u;
        };
        if constexpr (kSum != MixSum::kChunks) {
            while (u + (a.kb - kb) < u_end) {
                const uint32_t cnt = a.kb - kb;
                if (!next_set(!two_d)) break;  // (with one set the MMA issuers wait for this)
                mix_finish<kBf16, 4, kSum == MixSum::kCopies>(a, tmem + tlane + dbuf * d_set, a.copies, d_one, t, cnt, col, qd, lane, 0, leader, &s_last[0], abort_flag);
                give_back();
                u += cnt;
                kb = 0;
                ++t;
            }
        } else {
            const uint32_t sum = tmem + tlane + d_sum;
            bool ok = true;
            while (u < u_end && ok) {
                const uint32_t cnt = min(a.kb - kb, u_end - u);
                const bool mine = u + cnt < u_end;  // the last chunk of the last piece is the dequantising warps'
                for (uint32_t c = 0; (mine ? c : c + a.chunk) < cnt; c += a.chunk) {
                    ok = next_set(true);
                    if (!ok) break;
                    mix_promote(tmem + tlane + dbuf * d_set, sum, d_one, c == 0u);
                    give_back();
                }
                if (mine && ok) mix_finish<kBf16, 4, false>(a, sum, 1u, 0u, t, cnt, col, qd, lane, 0, leader, &s_last[0], abort_flag);
                u += cnt;
                kb = 0;
                ++t;
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (ok && lane == 0) mix_arrive(fsum0);
        }
    }
    if (a.split > 1u) {
        if (warp >= kMixDqWarps) {
            __syncwarp();
            ptx::cluster_arrive();
            ptx::cluster_wait();
        }
        // every warp's waits lie behind it, so the abort flag is final
        if (threadIdx.x < a.split && *abort_flag != 0u) {
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(ptx::smem_u32(const_cast<uint32_t*>(&s_bad))), "r"(threadIdx.x));
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(1u) : "memory");
        }
        __syncwarp();
        ptx::cluster_arrive();
        const MixOwn own = mix_own<kW, kNK>(a, blockIdx.x / a.split, rows_live(), ptx::cluster_ctarank(), threadIdx.x);
        ptx::cluster_wait();
        // (nobody reaches into another CTA's shared memory from here on: they leave when they are done)
        if (warp < kMixDqWarps && s_bad == 0u) mix_sum_and_store<kBf16, kSum == MixSum::kCopies ? 2 : 4>(a, smem0, own, threadIdx.x, s_bias);
    }
    // ---- teardown: everyone meets here, also after an aborted wait; then the allocating warp frees TMEM ----
    if (*abort_flag != 0u) __nanosleep(200000);  // lets bulk copies that are still in flight land before the CTA leaves
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == kMixDqWarps + kMixEpWarps + 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 512);
    }
}

using MixEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
MixEncodeFn mix_encoder()
{
    static MixEncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
        return reinterpret_cast<MixEncodeFn>(p);
    }();
    return fn;
}
bool mix_map(CUtensorMap* map, const void* base, uint64_t inner_bytes, uint64_t rows, uint64_t pitch, uint32_t box_inner, uint32_t box_rows,
             CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_L2_256B)
{
    MixEncodeFn enc = mix_encoder();
    if (enc == nullptr) return false;
    cuuint64_t dims[2] = {inner_bytes, rows};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2] = {box_inner, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               box_inner == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, promotion,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct MixPlan {
    int t_tiles, rows, split, copies, chunk;
    MixSum sum;
    int64_t n_tiles, kb, grid, units, tiles;
};

// How the (tile, k stage) line is cut. Either every tile into `split` equal pieces, one CTA each, launched as a cluster and summed over
// distributed shared memory; or stream-k, all SMs the same share, the tiles that straddle pieces summed through workspace. The first ends
// sooner for the same number of stages per CTA, so stream-k has to save stages to win. `clusters(split)` is how many clusters of that
// size the device keeps resident.
template <typename F>
MixPlan mix_plan(const OpsnnWqbmmParams* p, int sms, F&& clusters)
{
    MixPlan q;
    q.t_tiles = (int)((p->m + kMixMaxRows - 1) / kMixMaxRows);
    const int64_t per = (p->m + q.t_tiles - 1) / q.t_tiles;
    q.rows = (int)((per + 15) / 16 * 16);
    q.t_tiles = (int)((p->m + q.rows - 1) / q.rows);
    q.n_tiles = (p->n + kMixTileN - 1) / kMixTileN;
    q.kb = (p->k + 127) / 128;
    q.tiles = q.n_tiles * q.t_tiles;
    q.units = q.tiles * q.kb;
    q.split = 0;
    q.grid = q.units / 4;  // stages a CTA should at least see: a shorter piece is mostly ramp and combination
    if (q.grid > sms) q.grid = sms;
    if (q.grid < 1) q.grid = 1;
    int64_t stream_extra = 6 + q.rows / 4;
    if (const char* e = env("OPSNN_WQ_MIXED_STREAM")) stream_extra = atoi(e);
    int64_t best = (q.units + q.grid - 1) / q.grid + stream_extra;
    int64_t most = sms / q.tiles;
    if (most > 16) most = 16;
    if (most > q.kb) most = q.kb;
    for (int s = (int)most; s >= 1; --s) {
        const int64_t cost = (q.kb + s - 1) / s + (s > 1 ? 3 : 0);
        if (cost >= best || (s > 1 && (int64_t)clusters(s) < q.tiles)) continue;
        best = cost;
        q.split = s;
        q.grid = q.tiles * s;
    }
    if (const char* e = env("OPSNN_WQ_MIXED_SPLIT")) {  // experiments
        const int v = atoi(e);
        if (v >= 1 && v <= most) { q.split = v; q.grid = q.tiles * v; }
    }
    // The longest chain of MMAs (8 a stage) that leaves the sums as exact as the streaming kernels' (MixSum): a quarter of an SM's share of
    // the work, or what is left of k when they have cut it sixteen ways. They took more than 16 rows of x from 2^24 weights on, more than 32
    // from 3 x 2^24 (16 rows a launch).
    const int64_t chain = std::max<int64_t>(2 * q.units / sms, (q.kb * 9 + 19) / 20), piece = (q.units + q.grid - 1) / q.grid;
    q.sum = MixSum::kChain;
    q.copies = 1;
    q.chunk = (int)std::min<int64_t>(std::max<int64_t>(1, chain / 8), q.kb);
    if (q.rows == 16 || (q.rows == 32 && q.split != 0 && 2 * piece <= chain)) {
        q.sum = MixSum::kCopies;
        q.copies = q.split != 0 && 2 * piece > chain ? 8 : 4;
    } else if ((q.rows == 32 && p->k * p->n >= ((int64_t)1 << 24)) || (q.rows == 48 && p->k * p->n >= ((int64_t)3 << 24))) {
        q.sum = MixSum::kChunks;
    }
    return q;
}

using MixKernel = void (*)(const CUtensorMap, const CUtensorMap, const MixArgs);
template <MixW kW, bool kNK, MixSum kSum, bool kRagged>
MixKernel mix_kernel_of(bool bf16, bool off)
{
    if constexpr (kW != MixW::kE4m3) {
        if (off) return bf16 ? &wqbmm_mixed_kernel<kW, kNK, true, true, kSum, kRagged> : &wqbmm_mixed_kernel<kW, kNK, false, true, kSum, kRagged>;
    }
    return bf16 ? &wqbmm_mixed_kernel<kW, kNK, true, false, kSum, kRagged> : &wqbmm_mixed_kernel<kW, kNK, false, false, kSum, kRagged>;
}
template <MixSum kSum, bool kRagged>
MixKernel mix_kernel_of(int w, bool nk, bool bf16, bool off)
{
    switch (w) {
        case 0: return nk ? mix_kernel_of<MixW::kInt4, true, kSum, kRagged>(bf16, off) : mix_kernel_of<MixW::kInt4, false, kSum, kRagged>(bf16, off);
        case 1: return nk ? mix_kernel_of<MixW::kInt8, true, kSum, kRagged>(bf16, off) : mix_kernel_of<MixW::kInt8, false, kSum, kRagged>(bf16, off);
        default: return nk ? mix_kernel_of<MixW::kE4m3, true, kSum, kRagged>(bf16, off) : mix_kernel_of<MixW::kE4m3, false, kSum, kRagged>(bf16, off);
    }
}
template <bool kRagged>
MixKernel mix_kernel_of(MixSum sum, int w, bool nk, bool bf16, bool off)
{
    switch (sum) {
        case MixSum::kChain: return mix_kernel_of<MixSum::kChain, kRagged>(w, nk, bf16, off);
        case MixSum::kCopies: return mix_kernel_of<MixSum::kCopies, kRagged>(w, nk, bf16, off);
        default: return mix_kernel_of<MixSum::kChunks, kRagged>(w, nk, bf16, off);
    }
}
// The kernel of a form, ready to launch on the current device.
cudaError_t mix_kernel(const OpsnnWqbmmParams* p, MixSum sum, MixKernel* kern)
{
    static std::atomic<uint64_t> configured[2 * 3 * 24];
    const bool bf16 = p->x_dtype == ACL_BF16, off = p->offset != nullptr, nk = p->trans_w != 0, ragged = p->k % 128 != 0;
    const int w = p->w_dtype == ACL_INT4 ? 0 : (p->w_dtype == ACL_INT8 ? 1 : 2);
    const MixKernel k = ragged ? mix_kernel_of<true>(sum, w, nk, bf16, off) : mix_kernel_of<false>(sum, w, nk, bf16, off);
    *kern = k;
    return once_per_device(configured[(ragged ? 72 : 0) + (int)sum * 24 + w * 8 + (nk ? 4 : 0) + (bf16 ? 2 : 0) + (off ? 1 : 0)], [&] {
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMixSmemMax);
    });
}

// A call's plan and its kernel. (Every form takes an SM for itself, so clusters of one are placed as those of the others.)
cudaError_t mix_prepare(const OpsnnWqbmmParams* p, MixKernel* kern, MixPlan* plan)
{
    MixKernel any;
    if (const cudaError_t rc = mix_kernel(p, MixSum::kCopies, &any); rc != cudaSuccess) return rc;
    *plan = mix_plan(p, current_sm_count(), [&](int s) { return max_active_clusters(reinterpret_cast<const void*>(any), kMixThreads, kMixSmemMax, s, 0); });
    return mix_kernel(p, plan->sum, kern);
}

}  // namespace

// Layouts the kernel takes: int4 / int8 / e4m3 weights in either storage order with 16-byte aligned rows, one group or groups of whole
// 64-row units, scales in x's dtype - for (k,n) storage contiguous along n (their rows are bulk-copied), any strides for (n,k).
bool wqbmm_mixed_eligible(const OpsnnWqbmmParams* p)
{
    if (env("OPSNN_WQ_NO_MIXED")) return false;
    if (p->nz_k0 != 0 || p->scale_dtype == ACL_FLOAT8_E8M0) return false;
    if (p->w_dtype != ACL_INT4 && p->w_dtype != ACL_INT8 && p->w_dtype != ACL_FLOAT8_E4M3FN) return false;
    if (p->w_dtype == ACL_FLOAT8_E4M3FN && p->offset != nullptr) return false;
    if (p->x_dtype != ACL_BF16 && p->x_dtype != ACL_FLOAT16) return false;
    if (p->m < 1 || p->n < 1 || p->k < 64 || p->m >= (1 << 24) || p->n >= ((int64_t)1 << 30) || p->k >= ((int64_t)1 << 29)) return false;
    const int bits = p->w_dtype == ACL_INT4 ? 4 : 8;
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (!al16(p->w) || !al16(p->x) || p->x_ld % 8 != 0 || (p->w_ld * bits / 8) % 16 != 0 || (p->w_ld * bits) % 8 != 0) return false;
    if (p->group_size != 0 && p->group_size % 64 != 0) return false;
    if ((p->m + 15) / 16 * ((p->n + kMixTileN - 1) / kMixTileN) * ((p->k + 127) / 128) >= (1 << 24)) return false;  // 32-bit piece arithmetic
    if (p->trans_w) {
        if (bits == 4 && p->k % 2 != 0) return false;
        if (p->scale_sn < 0 || p->scale_sg < 0) return false;
    } else {
        if (p->n % 8 != 0 || p->scale_sn != 1 || !al16(p->scale) || (p->offset != nullptr && !al16(p->offset))) return false;
        if (p->group_size != 0 && p->scale_sg % 8 != 0) return false;
    }
    return true;
}

uint64_t wqbmm_mixed_workspace_size(const OpsnnWqbmmParams* p)
{
    // without a device (planning only) the stream-k form's need, which covers the other's
    MixKernel kern;
    MixPlan q;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0 || mix_prepare(p, &kern, &q) != cudaSuccess) {
        cudaGetLastError();
        q = mix_plan(p, 148, [](int) { return 0; });
    }
    if (q.split != 0) return 0;
    const uint64_t counters = ((uint64_t)q.tiles * 8u + 255u) & ~(uint64_t)255u;
    return 256u + counters + 2u * (uint64_t)q.grid * (uint64_t)q.rows * kMixTileN * 4u;
}

int32_t wqbmm_mixed_launch(const OpsnnWqbmmParams* p, cudaStream_t stream)
{
    MixKernel kern;
    MixPlan q;
    if (const cudaError_t rc = mix_prepare(p, &kern, &q); rc != cudaSuccess) return (int32_t)rc;
    if (q.split == 0 && (p->workspace == nullptr || p->workspace_size < wqbmm_mixed_workspace_size(p))) return (int32_t)cudaErrorInvalidValue;
    const bool nk = p->trans_w != 0, bf16 = p->x_dtype == ACL_BF16;
    const int bits = p->w_dtype == ACL_INT4 ? 4 : 8;
    MixArgs a{};
    a.m = (int32_t)p->m;
    a.n = (uint32_t)p->n;
    a.k = (uint32_t)p->k;
    a.t_tiles = q.t_tiles;
    a.rows = q.rows;
    a.kb = (uint32_t)q.kb;
    a.units = (uint32_t)q.units;
    a.grid = (uint32_t)q.grid;
    a.split = (uint32_t)q.split;
    a.copies = (uint32_t)q.copies;
    a.chunk = (uint32_t)q.chunk;
    a.group = p->group_size > 0 ? (uint32_t)p->group_size : 0x7FFFFFFFu;
    a.sc_rows = p->group_size % 128 == 0 ? 1 : 2;
    {
        auto al16 = [](const void* v) { return (reinterpret_cast<uintptr_t>(v) & 15) == 0; };
        // Eight groups a load where every column's rows of eight are whole and aligned. Groups of 64 are two a stage, the first an even one. (Read one by
        // one they had become 1 % slower with buffers that change hands by the stage: 77 x 8192 x 18432 int4 bf16 with offset 50.0 -> 50.5 us,
        // 34.8 with one load; 16 rows 45.5 / 34.3, int8 59.9 / 43.7.)
        a.sc_vec = nk && (a.sc_rows == 1 || p->group_size == 64) && p->group_size > 0 && p->scale_sg == 1 && p->scale_sn % 8 == 0 && (p->k / p->group_size) % 8 == 0 &&
                   p->k % p->group_size == 0 && al16(p->scale) && (p->offset == nullptr || al16(p->offset));
    }
    a.x_off = kMixTileN * 128 * bits / 8;
    a.sc_off = a.x_off + q.rows * 256;
    a.stage_bytes = a.sc_off + (nk ? 0 : 1024 * a.sc_rows);
    a.stages = (kMixSmemMax - 2048) / a.stage_bytes;
    if (a.stages > (uint32_t)kMixMaxStages) a.stages = kMixMaxStages;
    size_t smem = (size_t)a.stages * a.stage_bytes + 1024;
    if (smem < 116 * 1024) smem = 116 * 1024;  // one CTA per SM: the kernel owns all of the SM's tensor memory
    a.scale = p->scale;
    a.offset = p->offset;
    a.scale_sg = p->group_size > 0 ? p->scale_sg : 0;
    a.scale_sn = p->scale_sn;
    a.bias = p->bias;
    a.bias_dtype = p->bias_dtype;
    a.y = p->y;
    a.y_ld = p->y_ld;
    if (q.split == 0) {
        uint8_t* ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p->workspace) + 255) & ~(uintptr_t)255);
        a.count = reinterpret_cast<unsigned long long*>(ws);
        a.part = reinterpret_cast<float4*>(ws + (((uint64_t)q.tiles * 8u + 255u) & ~(uint64_t)255u));
    }
    a.nonce = next_nonce() & 0x00FFFFFFFFFFFFFFull;
    const uint32_t f = bf16 ? 1u : 0u;
    a.idesc = make_idesc(1u, f, f, 0u, 0u, 128u, (uint32_t)q.rows);
    // More than 16 rows: as a dequantised weight's matmul would, a call after one that gave up a wait is refused.
    if (p->m > 16) {
        unsigned int* mirror;
        if (const int32_t bad = umma_prelaunch_check(stream, &mirror)) return bad;
        a.status_host = mirror;
    }
    a.test_stop = 0xFFFFFFFFu;
    if (const char* e = env("OPSNN_TEST_MIXED_STALL_STAGE")) {  // tests of the give-up path only
        a.test_stop = (uint32_t)atoi(e);
        const char* pl = env("OPSNN_TEST_UMMA_POLL_LIMIT");
        const uint32_t limit = pl != nullptr ? (uint32_t)atoi(pl) : 20000u;
        cudaMemcpyToSymbolAsync(ptx::g_spin_limit, &limit, sizeof(limit), 0, cudaMemcpyHostToDevice, stream);
    }
    CUtensorMap mw, mx;
    const bool ok = nk ? mix_map(&mw, p->w, (uint64_t)p->k * bits / 8, (uint64_t)p->n, (uint64_t)p->w_ld * bits / 8, bits == 4 ? 64u : 128u, kMixTileN)
                       : mix_map(&mw, p->w, (uint64_t)p->n * bits / 8, (uint64_t)p->k, (uint64_t)p->w_ld * bits / 8, 128u, 128u,
                                // a tile is 128 bytes of an int4 row: fetching 256 for it reads the neighbour's half twice (4.2 -> 5.5 TB/s)
                                bits == 4 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B : CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    if (!ok || !mix_map(&mx, p->x, (uint64_t)p->k * 2, (uint64_t)p->m, (uint64_t)p->x_ld * 2, 128u, (uint32_t)q.rows)) return (int32_t)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(a.grid, 1, 1);
    cfg.blockDim = dim3(kMixThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = a.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.split > 1u ? 2 : 1;
    const int32_t rc = (int32_t)cudaLaunchKernelEx(&cfg, kern, mw, mx, a);
    note_launch("wqbmm_mixed");
    return rc;
}

// Error word of this file's kernel on the current device (see opsnn_wqbmm_decode_status).
uint32_t wqbmm_mixed_status(int reset)
{
    unsigned int v = 0;
    cudaMemcpyFromSymbol(&v, g_mix_status, sizeof(v));
    if (reset) {
        unsigned int z = 0;
        cudaMemcpyToSymbol(g_mix_status, &z, sizeof(z));
        const uint32_t limit = ptx::kSpinLimit;  // a test may have shortened the waits
        cudaMemcpyToSymbol(ptx::g_spin_limit, &limit, sizeof(limit));
    }
    return v;
}

}  // namespace opsnn
