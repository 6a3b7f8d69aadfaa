// Per-block (1x128 / 128x128 fp32 scales) fp8 and int8 matmul on CTA pairs (tcgen05 cta_group::2). Included by qmm_umma.cu.
//
// Why. The single-CTA per-block kernel uses 128 x 128 tiles (the promotion epilogue keeps 128 fp32 sums per thread), which
// pull 32 KB of operands from L2 per 128-deep k-block of 256 clocks of tensor work. A CTA pair shares a 256 x 128 tile: each
// CTA loads its own 128 rows of A and 64 of the 128 rows of B (24 KB per k-block), keeps a 128 x 128 accumulator in its own
// TMEM and runs the same promotion on it.
//
// B per CTA is half of the tile's 128 columns. k-major (x2 stored (n,k)): 64 rows of 128 swizzled bytes. n-major (x2 stored
// (k,n)): half a 128-byte swizzle row is not a legal operand, so the 64 columns x 128 k rows are loaded and described in the
// 64-byte swizzle (TMA box 64 x 128, descriptor layout type 4, 512 bytes per 8 rows).
//
// Choreography per k-block (= one accumulation group), four TMEM buffers of 128 columns:
//   producers (both CTAs) : wait own empty[s]; even CTA arms full[s] for both CTAs' bytes; each loads A (128 rows) and B (64 rows)
//   MMA warp (even CTA)   : wait tempty[buf] (all epilogue warps of the pair), wait full[s], 4 pair MMAs (first overwrites),
//                           commit -> empty[s] and tfull[buf] of both CTAs
//   epilogue (both CTAs)  : wait own tfull[buf]; TMEM -> registers; acc += part * (s1 * s2); arrive on the even CTA's tempty[buf]
//   scale loaders         : two warps keep s1 of the CTA's rows and s2 of the tile's column blocks two runs of k-blocks ahead in shared
//                           memory
// Bound by the epilogue warps' chain per k-block (barrier, TMEM reads beside the running MMA, multiply-adds of 128 x 256 sums: ~900
// clocks for 512 of tensor work) and, at 4096 x 7168 x 18432, by the power limit as well. Every epilogue thread used to read its scales
// from global memory (32 sectors a load) and to store its row 16 bytes at a time: 180 and 120 of 1117 clocks. A run's scales are in
// registers before its first k-block: read per k-block, they cost 8 % of the chain. fp8, bf16 out: 4096 x 7168 x 18432 655 -> 600 us,
// 1024 x 4096 x 7168 51.5 -> 42.5, 512 x 7168 x 4608 27.3 -> 19.5, 2000 x 2048 x 2048 18.4 -> 16.
// Neither the MMAs nor the TMEM port are the bound: 901 clocks a k-block, 962 (instrumented) without any MMA, 577 - 640 for a skeleton of the same TMEM
// loads and multiply-adds. Tried besides: products of the scales from the loaders, one k-block an iteration, waits without divergence (878 clocks;
// 593 / 595 us under the power limit); 32-byte stores from registers (883).
// Tried: two N = 128 MMAs a k-block on four half buffers (57 us at 1024 x 4096 x 7168), 32 columns a TMEM load (spills, 54 us).
namespace {

// Two neighbouring columns; fp8's fused multiply-adds go as one packed instruction (each half rounded on its own).
template <ptx::MmaKind kKind>
__device__ __forceinline__ void promote2(uint32_t v0, uint32_t v1, float sc, float& a0, float& a1)
{
    if constexpr (kKind != ptx::MmaKind::kI8) {
        asm("{\n\t.reg .b64 a, v, s;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\tfma.rn.f32x2 a, v, s, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
            : "+f"(a0), "+f"(a1)
            : "r"(v0), "r"(v1), "f"(sc));
        return;
    }
    a0 = promote<kKind>(v0, sc, a0);
    a1 = promote<kKind>(v1, sc, a1);
}

// 256-column tiles: 128 sums per epilogue thread need more registers than an even split of the register file over the CTA's
// warps gives (168 with ten warps), so the block is three whole warpgroups - epilogue warps 0..7, then {producer, MMA issuer, two
// scale loaders} - and setmaxnreg moves registers from the third group (40 each) to the first two (232 each): per scheduler
// 2 x 232 + 40 = 504 of the 512 registers per lane.
// (Code that runs under setmaxnreg cannot call an out-of-line function: the bounded spin is inlined for those instances.)
template <bool kInline>
__device__ __forceinline__ bool pb_wait(uint32_t bar_addr, uint32_t parity, volatile uint32_t* abort_flag)
{
    if (!kInline) return ptx::mbar_wait_a(bar_addr, parity, abort_flag);
    if (ptx::mbar_try_wait_a(bar_addr, parity)) return true;
    const uint32_t limit = ptx::g_spin_limit;
    for (uint32_t i = 0; i < limit; ++i) {
        if (ptx::mbar_try_wait_a(bar_addr, parity)) return true;
        if ((i & 1023u) == 1023u && *abort_flag != 0u) return false;
    }
    *abort_flag = 1u;
    return false;
}

template <int EW, bool kAsym>
constexpr int pair_pb_threads() { return (EW + (kAsym ? 2 : 4)) * 32; }

constexpr int kPbScaleRun = 4;  // k-blocks of scales per buffer of the ring

// kAsym: INT4 x INT4 asymmetric per-group (quant_batch_matmul_v4_pertoken_pergroup.h; golden qbmmv4_kernel_golden.py:328-395), both
// operands widened to INT8 beforehand. An accumulation group is two k-blocks (256 of k); per group and element
// tot += (part - rowsum(x1 over the group)[m] * x2Offset[g, n]) * x2Scale[g, n], four separately rounded fp32 operations as in
// the golden, and at the end out = tot * x1Scale[m]. x2Offset / x2Scale of the tile's columns are staged in shared memory one
// group ahead (three buffers, one named barrier per group whose reduced predicate also carries the abort flag, so that the
// epilogue warps can only leave together).
template <ptx::MmaKind kKind, int EW, int BN, bool kAsym = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_pb_threads<EW, kAsym>(), 1)
qmm_umma_pair_pb_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const UmmaArgs a)
{
    static_assert(BN == 128 || (BN == 256 && EW == 8), "256-column tiles keep 128 sums per thread: eight epilogue warps");
    static_assert(!kAsym || (BN == 128 && EW == 4 && kKind == ptx::MmaKind::kI8), "the asymmetric per-group epilogue: int8, 128 columns, four warps");
    __shared__ float s_cols[kAsym ? 3 * 2 * BN : 1];  // kAsym: [buffer][offset | scale][column]
    // otherwise: scales of a run of k-blocks, two buffers ([k-block][row], then [k-block][128-column block]), and 2 KB per epilogue warp
    // through which its rows leave as 64-byte pieces
    __shared__ __align__(16) float s_scale[kAsym ? 1 : 2][kAsym ? 1 : kPbScaleRun * 130];
    __shared__ __align__(16) uint8_t s_out[kAsym ? 16 : EW * 2048];
    __shared__ uint64_t s_bars[4];  // scale buffers: [2] full, [2] empty
    constexpr int NBUF = 512 / BN;              // accumulator buffers in the 512 TMEM columns
    constexpr int kCols = BN * 4 / EW;          // accumulator columns per epilogue thread
    constexpr uint32_t kBHalf = (BN / 2) * BK;  // this CTA's half of the B tile
    constexpr uint32_t kStage = kATile + kBHalf;
    constexpr uint32_t kTmemCols = 512;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)a.stages * kStage);
    uint64_t* full = bars;                    // [stages]  used in the even CTA only
    uint64_t* empty = bars + a.stages;        // [stages]
    uint64_t* tfull = bars + 2 * a.stages;    // [NBUF]
    uint64_t* tempty = tfull + NBUF;          // [NBUF]    used in the even CTA only
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tempty + NBUF);
    volatile uint32_t* abort_flag = tmem_ptr + 1;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < NBUF; ++b) {
            ptx::mbar_init(&tfull[b], 1);
            ptx::mbar_init(&tempty[b], 2 * EW);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(&s_bars[b], 2);       // two loading warps
            ptx::mbar_init(&s_bars[2 + b], EW);  // the epilogue warps
        }
        *abort_flag = 0u;
        ptx::fence_mbar_init();
    }
    if (warp == EW + 1) ptx::tmem_alloc_pair(tmem_ptr, kTmemCols);
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr;
    pdl_trigger();
    pdl_wait();

    const uint32_t tiles_per_batch = (uint32_t)a.tiles_m * (uint32_t)a.tiles_n;
    const uint32_t ntiles = (uint32_t)a.num_tiles;
    const uint32_t pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const uint32_t smem0 = ptx::smem_u32(smem), full0 = ptx::smem_u32(full), empty0 = ptx::smem_u32(empty);
    const uint32_t tfull0 = ptx::smem_u32(tfull), tempty0 = ptx::smem_u32(tempty);
    const uint32_t stages = (uint32_t)a.stages;
    const uint32_t sfull0 = ptx::smem_u32(s_bars), sempty0 = sfull0 + 16u;
    const int kblocks = a.kblocks;

    if (warp == EW) {
        // ======================= TMA producer (both CTAs) =======================
        if (BN == 256) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (lane == 0) {
            ptx::tma_prefetch_desc(&map_a);
            ptx::tma_prefetch_desc(&map_b);
        }
        __syncwarp();
        uint32_t s = 0, par = 0;
        bool ok = true;
        const bool a_mn = a.a_mn_major != 0, b_mn = a.b_mn_major != 0;
        const uint32_t lead_full0 = full0 & ptx::kPeerBitMask;
        for (uint32_t tile = pair; tile < ntiles && ok; tile += npairs) {
            const uint32_t b = tile / tiles_per_batch, r = tile % tiles_per_batch;
            uint32_t tm, tn;
            tile_of<8>(r, (uint32_t)a.tiles_m, (uint32_t)a.tiles_n, tm, tn);
            const int32_t m0 = (int32_t)tm * 256 + (int32_t)rank * 128;
            const int32_t n0 = (int32_t)tn * BN + (int32_t)rank * (BN / 2);
            const int32_t ba = a.a_batched ? (int32_t)b : 0, bb = a.b_batched ? (int32_t)b : 0;
            int32_t kk = 0;
            for (int kb = 0; kb < kblocks; ++kb) {
                if (!pb_wait<BN == 256>(empty0 + 8u * s, par ^ 1u, abort_flag)) {
                    report(abort_flag, (1u << 8) | 1u);
                    ok = false;
                    break;
                }
                if (ptx::elect_one()) {
                    const uint32_t fb = lead_full0 + 8u * s, sa = smem0 + s * kStage, sb = sa + (uint32_t)kATile;
                    if (leader) ptx::mbar_expect_tx_a(full0 + 8u * s, 2u * kStage);
                    ptx::tma_load_3d_pair(sa, &map_a, fb, a_mn ? m0 : kk, a_mn ? kk : m0, ba);
                    if (b_mn) ptx::tma_load_3d_pair(sb, &map_b, fb, n0, kk, bb);  // BN / 2 columns x 128 k rows (64 columns: 64-byte swizzle)
                    else ptx::tma_load_3d_pair(sb, &map_b, fb, kk, n0, bb);
                }
                __syncwarp();
                kk += BK;
                if (++s == stages) {
                    s = 0;
                    par ^= 1u;
                }
            }
        }
    } else if (warp == EW + 1) {
        // ======================= MMA issuer (even CTA only): every k-block is its own accumulation group =======================
        if (BN == 256) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (leader) {
            uint32_t s = 0, par = 0, buf = 0, bpar = 0;
            bool ok = true;
            const uint64_t da0 = a.a_mn_major ? ptx::make_smem_desc(smem0, 128 * BK, 1024, 2) : ptx::make_smem_desc(smem0, 0, 1024, 2);
            // B k-major: 64 rows of 128 swizzled bytes. B n-major (x2 stored (k,n)): 128 k rows of this CTA's 64 columns in the
            // 64-byte swizzle (layout type 4): 8 rows = 512 bytes (stride byte offset), one MMA = 32 rows = 2 KB
            // 128 columns (BN = 256) are whole 128-byte swizzle rows, described like an m-major A
            const uint64_t db0 = !a.b_mn_major ? ptx::make_smem_desc(smem0 + kATile, 0, 1024, 2)
                                 : (BN == 128 ? ptx::make_smem_desc(smem0 + kATile, 64 * BK, 512, 4)
                                              : ptx::make_smem_desc(smem0 + kATile, 128 * BK, 1024, 2));
            const uint32_t a_lo = (uint32_t)da0, b_lo = (uint32_t)db0;
            const uint64_t a_hi = da0 & 0xFFFFFFFF00000000ull, b_hi = db0 & 0xFFFFFFFF00000000ull;
            const uint32_t a_k1 = a.a_mn_major ? 256u : 2u, b_k1 = a.b_mn_major ? (BN == 128 ? 128u : 256u) : 2u;
            const uint32_t idesc = a.idesc;
            for (uint32_t tile = pair; tile < ntiles && ok; tile += npairs) {
                for (int kb = 0; kb < kblocks; ++kb) {
                    // kAsym: k-blocks 2g and 2g + 1 accumulate into one buffer; otherwise every k-block is its own group
                    const bool first = !kAsym || (kb & 1) == 0, last = !kAsym || (kb & 1) == 1 || kb == kblocks - 1;
                    if (first && !pb_wait<BN == 256>(tempty0 + 8u * buf, bpar ^ 1u, abort_flag)) {
                        report(abort_flag, (2u << 8) | 1u);
                        ok = false;
                        break;
                    }
                    if (!pb_wait<BN == 256>(full0 + 8u * s, par, abort_flag)) {
                        report(abort_flag, (2u << 8) | 2u);
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    if (ptx::elect_one()) {
                        const uint32_t stage_off = (s * kStage) >> 4;
                        const uint32_t d = tmem_base + buf * BN;
                        const uint32_t al = a_lo + stage_off, bl = b_lo + stage_off;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            ptx::umma_pair<kKind>(d, a_hi | (uint64_t)(al + k * a_k1), b_hi | (uint64_t)(bl + k * b_k1), idesc,
                                                  (k == 0 && first) ? 0u : 1u);
                        ptx::umma_commit_pair(empty0 + 8u * s, (uint16_t)3);
                        if (last) ptx::umma_commit_pair(tfull0 + 8u * buf, (uint16_t)3);
                    }
                    __syncwarp();
                    if (++s == stages) {
                        s = 0;
                        par ^= 1u;
                    }
                    if (last && ++buf == NBUF) {
                        buf = 0;
                        bpar ^= 1u;
                    }
                }
            }
        }
    } else if (warp < EW) {
        // ======================= epilogue warps (both CTAs): own 128 rows, kCols columns each =======================
        if (BN == 256) asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        const int quad = warp & 3, part = warp >> 2;
        const uint32_t lane_addr = ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * kCols);
        const uint32_t lead_tempty0 = tempty0 & ptx::kPeerBitMask;
        uint32_t buf = 0, bpar = 0, sbuf = 0, spar = 0;
        bool ok = true;
        for (uint32_t tile = pair; tile < ntiles && ok; tile += npairs) {
            const uint32_t b = tile / tiles_per_batch, r = tile % tiles_per_batch;
            uint32_t tm, tn;
            tile_of<8>(r, (uint32_t)a.tiles_m, (uint32_t)a.tiles_n, tm, tn);
            const int64_t m0 = (int64_t)tm * 256 + (int64_t)rank * 128, n0 = (int64_t)tn * BN;
            const int64_t row = m0 + quad * 32 + lane;
            const bool row_ok = row < a.m;
            uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + b * a.out_bs * out_elem_bytes(a.out_dtype);
            const int64_t colbase = n0 + part * kCols;
            float acc[kCols];
#pragma unroll
            for (int i = 0; i < kCols; ++i) acc[i] = 0.f;
            if constexpr (kAsym) {
                const int groups = a.groups;
                const float* rsp = a.row_sums + (row_ok ? row : 0) * (int64_t)groups;
                const __half* offp = reinterpret_cast<const __half*>(a.b_offset);
                const float* scp = reinterpret_cast<const float*>(a.scale_b);
                const int tcol = quad * 32 + lane;  // the column of the tile whose offset and scale this thread stages
                const int64_t gcol = n0 + tcol;
                auto stage_cols = [&](int g) {
                    float o = 0.f, sc = 0.f;
                    if (g < groups && gcol < a.n) {
                        o = __half2float(offp[(int64_t)g * a.n + gcol]);
                        sc = __ldg(scp + (int64_t)g * a.n + gcol);
                    }
                    float* dst = s_cols + (g % 3) * 2 * BN;
                    dst[tcol] = o;
                    dst[BN + tcol] = sc;
                };
                asm volatile("bar.sync 1, 128;" ::: "memory");  // the previous tile's readers of the column buffers are done
                stage_cols(0);
                float rs_next = __ldg(rsp);
                for (int g = 0; g < groups; ++g) {
                    const float rsg = rs_next;
                    if (g + 1 < groups) rs_next = __ldg(rsp + g + 1);
                    stage_cols(g + 1);  // buffer (g + 1) % 3: last read in group g - 2, which every warp has left (barrier of g - 1)
                    const bool arrived = pb_wait<false>(tfull0 + 8u * buf, bpar, abort_flag);
                    if (!arrived) report(abort_flag, (3u << 8) | 2u);
                    // One barrier per group: group g's columns are visible to all four warps, and its reduced predicate tells every
                    // warp the same thing about a give-up anywhere in the CTA - they can only leave together.
                    const int bad = (!arrived || *abort_flag != 0u) ? 1 : 0;
                    int any_bad;
                    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.or.pred p, 1, 128, q;\n\tselp.s32 %0, 1, 0, p;\n\t}"
                                 : "=r"(any_bad)
                                 : "r"(bad)
                                 : "memory");
                    if (any_bad != 0) {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const float* cur = s_cols + (g % 3) * 2 * BN;
                    const uint32_t t0 = tmem_base + lane_addr + buf * BN;
                    // (part - rowsum * offset) * scale, then the running sum: four roundings, none fused, as in the golden
                    auto fold = [&](const uint32_t(&v)[16], int c) {
#pragma unroll
                        for (int i = 0; i < 16; i += 4) {
                            const float4 o4 = *reinterpret_cast<const float4*>(cur + c + i);
                            const float4 s4 = *reinterpret_cast<const float4*>(cur + BN + c + i);
                            const float oo[4] = {o4.x, o4.y, o4.z, o4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float f = __fsub_rn(__uint_as_float(v[i + j] + 0x4B400000u), 12582912.f);  // exact int -> float, |part| < 2^22
                                const float w = __fmul_rn(__fsub_rn(f, __fmul_rn(rsg, oo[j])), ss[j]);
                                acc[c + i + j] = __fadd_rn(acc[c + i + j], w);
                            }
                        }
                    };
                    uint32_t va[16], vb[16];
                    ptx::tmem_ld16(t0, va);
#pragma unroll
                    for (int c = 0; c < kCols; c += 32) {
                        ptx::tmem_ld_wait();
                        ptx::tmem_ld16(t0 + c + 16, vb);
                        fold(va, c);
                        ptx::tmem_ld_wait();
                        if (c + 32 < kCols) {
                            ptx::tmem_ld16(t0 + c + 32, va);
                        } else {
                            ptx::tc_fence_before();
                            __syncwarp();
                            if (lane == 0) ptx::mbar_arrive_cluster(lead_tempty0 + 8u * buf);
                        }
                        fold(vb, c + 16);
                    }
                    if (++buf == NBUF) {
                        buf = 0;
                        bpar ^= 1u;
                    }
                }
                if (row_ok) {  // out = tot * x1Scale[m]
                    const float sa = __ldg(reinterpret_cast<const float*>(a.scale_a) + row);
#pragma unroll
                    for (int i = 0; i < kCols; ++i) acc[i] = __fmul_rn(acc[i], sa);
                }
            } else {
                const uint32_t nb = (uint32_t)(part * kCols) >> 7;  // 128-column block of the tile
                for (int kb0 = 0; kb0 < kblocks && ok; kb0 += kPbScaleRun) {
                    if (!__all_sync(0xffffffffu, pb_wait<BN == 256>(sfull0 + 8u * sbuf, spar, abort_flag))) {
                        report(abort_flag, (3u << 8) | 3u);
                        ok = false;
                        break;
                    }
                    float run[kPbScaleRun];  // the run's scales; the buffer goes back at once
#pragma unroll
                    for (int j = 0; j < kPbScaleRun; ++j)
                        run[j] = __fmul_rn(s_scale[sbuf][j * 128 + quad * 32 + lane], s_scale[sbuf][kPbScaleRun * 128 + 2 * j + nb]);
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(&s_bars[2 + sbuf]);
                    sbuf ^= 1u;
                    if (sbuf == 0u) spar ^= 1u;
#pragma unroll
                    for (int j = 0; j < kPbScaleRun; ++j) {
                        if (kb0 + j >= kblocks) break;
                        const float sc = run[j];
                        if (!pb_wait<BN == 256>(tfull0 + 8u * buf, bpar, abort_flag)) {
                            report(abort_flag, (3u << 8) | 2u);
                            ok = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        constexpr int W = 16;  // staging registers per TMEM load (two sets in flight)
                        const uint32_t t0 = tmem_base + lane_addr + buf * BN;
                        uint32_t va[W], vb[W];
                        ptx::tmem_ld_n(t0, va);
#pragma unroll
                        for (int c = 0; c < kCols; c += 2 * W) {
                            ptx::tmem_ld_wait();
                            ptx::tmem_ld_n(t0 + c + W, vb);
#pragma unroll
                            for (int i = 0; i < W; i += 2) promote2<kKind>(va[i], va[i + 1], sc, acc[c + i], acc[c + i + 1]);
                            ptx::tmem_ld_wait();
                            if (c + 2 * W < kCols) {
                                ptx::tmem_ld_n(t0 + c + 2 * W, va);
                            } else {
                                ptx::tc_fence_before();
                                __syncwarp();
                                if (lane == 0) ptx::mbar_arrive_cluster(lead_tempty0 + 8u * buf);
                            }
#pragma unroll
                            for (int i = 0; i < W; i += 2) promote2<kKind>(vb[i], vb[i + 1], sc, acc[c + W + i], acc[c + W + i + 1]);
                        }
                        if (++buf == NBUF) {
                            buf = 0;
                            bpar ^= 1u;
                        }
                    }
                }
            }
            if constexpr (!kAsym) {
                // Whole tiles with 16-byte rows: a thread's row goes through shared memory and leaves with its neighbours as 64-byte
                // pieces (pieces of a row XOR-swizzled by the row pair: no bank conflicts either way).
                const int es = out_elem_bytes(a.out_dtype);
                if (ok && colbase + kCols <= a.n && ((reinterpret_cast<uintptr_t>(out) | (uintptr_t)(a.out_ld * es)) & 15) == 0) {
                    uint8_t* st = s_out + warp * 2048;
                    const uint8_t* bias = a.bias == nullptr ? nullptr : reinterpret_cast<const uint8_t*>(a.bias) +
                                              b * a.bias_bs * ((a.bias_dtype == ACL_FLOAT || a.bias_dtype == ACL_INT32) ? 4 : 2);
                    auto piece = [&](int p) { return st + lane * 64 + ((p ^ ((lane >> 1) & 3)) << 4); };
                    uint8_t* orow = out + (m0 + quad * 32 + (lane >> 2)) * a.out_ld * es + colbase * es + (lane & 3) * 16;
                    const int64_t rows_left = a.m - (m0 + quad * 32 + (lane >> 2));
                    auto flush = [&](int c) {  // the warp's 32 rows x 64 bytes, from column c
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int r = (lane >> 2) + 8 * i;
                            const uint4 v = *reinterpret_cast<const uint4*>(st + r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) << 4));
                            if (8 * i < rows_left) *reinterpret_cast<uint4*>(orow + (int64_t)(8 * i) * a.out_ld * es + c * es) = v;
                        }
                        __syncwarp();
                    };
#pragma unroll
                    for (int c = 0; c < kCols; c += 32) {
                        float f[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) f[i] = acc[c + i];
                        if (bias != nullptr) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) f[i] = __fadd_rn(f[i], load_as_float(bias, colbase + c + i, a.bias_dtype));
                        }
                        if (a.out_dtype == ACL_FLOAT) {
#pragma unroll
                            for (int h = 0; h < 32; h += 16) {
#pragma unroll
                                for (int i = 0; i < 4; ++i)
                                    *reinterpret_cast<float4*>(piece(i)) = make_float4(f[h + 4 * i], f[h + 4 * i + 1], f[h + 4 * i + 2], f[h + 4 * i + 3]);
                                flush(c + h);
                            }
                        } else {
                            uint32_t pk[16];
                            pack16(a.out_dtype, f, pk);
#pragma unroll
                            for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(piece(i)) = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
                            flush(c);
                        }
                    }
                    continue;
                }
            }
            if (ok && row_ok) {
#pragma unroll
                for (int c = 0; c < kCols; c += 32) {
                    const int64_t col = colbase + c;
                    const int valid = (int)max((int64_t)0, min((int64_t)32, a.n - col));
                    if (valid > 0) {
                        float f[32];
#pragma unroll
                        for (int i = 0; i < 32; ++i) f[i] = acc[c + i];
                        if (a.bias != nullptr) {
                            const uint8_t* bias = reinterpret_cast<const uint8_t*>(a.bias) +
                                                  b * a.bias_bs * ((a.bias_dtype == ACL_FLOAT || a.bias_dtype == ACL_INT32) ? 4 : 2);
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (i < valid) f[i] = __fadd_rn(f[i], load_as_float(bias, col + i, a.bias_dtype));
                        }
                        store_row32(a, out, row, col, f, valid);
                    }
                }
            }
        }
    } else if constexpr (!kAsym) {
        // ======================= scale loaders (two warps): s1 of this CTA's 128 rows, s2 of the tile's column blocks =======================
        if (BN == 256) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        const int t = (int)threadIdx.x - (EW + 2) * 32;  // 0 .. 63: rows t and t + 64
        const uint32_t n_mg = (uint32_t)((a.m + a.group_m - 1) / a.group_m), n_ng = (uint32_t)((a.n + 127) / 128);
        const uint32_t rs = a.trans_a ? 1u : (uint32_t)kblocks, ks = a.trans_a ? n_mg : 1u;  // strides of s1 per row group and per k-block
        const bool vec = !a.trans_a && kblocks % 4 == 0 && (reinterpret_cast<uintptr_t>(a.scale_a) & 15) == 0 && (a.sa_bs & 3) == 0;
        uint32_t sbuf = 0, spar = 0;
        bool ok = true;
        for (uint32_t tile = pair; tile < ntiles && ok; tile += npairs) {
            const uint32_t b = tile / tiles_per_batch, r = tile % tiles_per_batch;
            uint32_t tm, tn;
            tile_of<8>(r, (uint32_t)a.tiles_m, (uint32_t)a.tiles_n, tm, tn);
            const uint32_t row = tm * 256u + rank * 128u + (uint32_t)t, last = (uint32_t)a.m - 1u;
            const float* s1 = reinterpret_cast<const float*>(a.scale_a) + b * a.sa_bs;
            const float* r0 = s1 + (int64_t)(min(row, last) / (uint32_t)a.group_m) * rs;
            const float* r1 = s1 + (int64_t)(min(row + 64u, last) / (uint32_t)a.group_m) * rs;
            // the first threads: s2 of k-block t / 2 of the run, column block t % 2
            const uint32_t ng = min(tn * (BN / 128) + (uint32_t)(t & 1), n_ng - 1u);
            const float* s2 = reinterpret_cast<const float*>(a.scale_b) + b * a.sb_bs + (a.trans_b ? (int64_t)ng * kblocks : (int64_t)ng);
            const uint32_t s2k = a.trans_b ? 1u : n_ng;
            for (int kb = 0; kb < kblocks; kb += kPbScaleRun) {
                float v0[kPbScaleRun], v1[kPbScaleRun], w = 0.f;
                if (vec) {
                    const float4 x = __ldg(reinterpret_cast<const float4*>(r0 + kb)), y = __ldg(reinterpret_cast<const float4*>(r1 + kb));
                    v0[0] = x.x; v0[1] = x.y; v0[2] = x.z; v0[3] = x.w;
                    v1[0] = y.x; v1[1] = y.y; v1[2] = y.z; v1[3] = y.w;
                } else {
#pragma unroll
                    for (int h = 0; h < kPbScaleRun; ++h) {
                        const int64_t at = (int64_t)min(kb + h, kblocks - 1) * ks;
                        v0[h] = __ldg(r0 + at);
                        v1[h] = __ldg(r1 + at);
                    }
                }
                if (t < 2 * kPbScaleRun) w = __ldg(s2 + (int64_t)min(kb + (t >> 1), kblocks - 1) * s2k);
                if (!__all_sync(0xffffffffu, pb_wait<BN == 256>(sempty0 + 8u * sbuf, spar ^ 1u, abort_flag))) {
                    report(abort_flag, (4u << 8) | 1u);
                    ok = false;
                    break;
                }
                float* d = s_scale[sbuf];
#pragma unroll
                for (int h = 0; h < kPbScaleRun; ++h) {
                    d[h * 128 + t] = v0[h];
                    d[h * 128 + 64 + t] = v1[h];
                }
                if (t < 2 * kPbScaleRun) d[kPbScaleRun * 128 + t] = w;
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&s_bars[sbuf]);
                sbuf ^= 1u;
                if (sbuf == 0u) spar ^= 1u;
            }
        }
    }
    // ---- teardown ----
    if (*abort_flag != 0u) __nanosleep(200000);
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();
    if (warp == EW + 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

template <ptx::MmaKind KIND, int EW, int BN = 128, bool ASYM = false>
int32_t launch_pair_pb(const CUtensorMap& ma, const CUtensorMap& mb, UmmaArgs& a, cudaStream_t stream)
{
    constexpr int kStage = kATile + (BN / 2) * BK;
    constexpr int kDynMax = 227 * 1024 - (ASYM ? 4096 : 5 * 1024 + EW * 2048);  // less the static buffers
    int stages = (kDynMax - 2048) / kStage;
    if (stages > 8) stages = 8;
    if (stages > a.kblocks + 1) stages = a.kblocks + 1 > 2 ? a.kblocks + 1 : 2;
    a.stages = stages;
    const size_t smem = (size_t)stages * kStage + 1024 + 256;
    auto kern = qmm_umma_pair_pb_kernel<KIND, EW, BN, ASYM>;
    static std::atomic<uint64_t> configured{0};
    if (once_per_device(configured, [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kDynMax); }) != cudaSuccess)
        return (int32_t)cudaGetLastError();
    int64_t pairs = sm_count() / 2;
    if (a.num_tiles < pairs) pairs = a.num_tiles;
    launch_dependent(kern, dim3((unsigned)(2 * pairs)), pair_pb_threads<EW, ASYM>(), smem, stream, ma, mb, a);
    note_launch(ASYM ? "qmm_umma_pair_pergroup_asym" : "qmm_umma_pair_perblock");
    return (int32_t)cudaGetLastError();
}

// Sums of x1's rows over each k-group, as floats (exact: at most 256 values of magnitude <= 128), for the asymmetric per-group
// epilogue. One thread per (row, group); x1 is the widened INT8 operand, stored (m,k) or, transposed, (k,m).
__global__ void row_sums_kernel(const int8_t* __restrict__ x1, int64_t ld, int trans, int64_t m, int64_t k, int32_t groups, int32_t group_k,
                                float* __restrict__ out)
{
    const int64_t total = m * groups;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        // transposed storage: consecutive threads take consecutive rows (contiguous in memory); else consecutive groups of one row
        const int64_t row = trans ? i % m : i / groups;
        const int g = (int)(trans ? i / m : i % groups);
        const int64_t k0 = (int64_t)g * group_k, k1 = min(k, k0 + group_k);
        int sum = 0;
        if (trans) {
            for (int64_t kk = k0; kk < k1; ++kk) sum += x1[kk * ld + row];
        } else {
            for (int64_t kk = k0; kk < k1; ++kk) sum += x1[row * ld + kk];
        }
        out[row * groups + g] = (float)sum;
    }
}

// Pair tiles for per-block problems: worthwhile once there are enough 256 x 128 tiles to fill the pairs.
bool pair_pb_worthwhile(const OpsnnQmmParams* p)
{
    if (p->mode != OPSNN_QMM_PERBLOCK) return false;
    if (const char* e = env("OPSNN_QMM_PAIR")) return atoi(e) != 0;
    const int64_t tiles = p->batch * ((p->m + 255) / 256) * ((p->n + 127) / 128);
    return p->m >= 256 && tiles >= 74;
}

// Tile width of the per-block pair kernel: 256 columns (32 KB of operands per CTA and k-block for twice the tensor work of the
// 128-column tile's 24 KB, and one hand-over of an accumulator instead of two) once there are enough such tiles for every pair.
// OPSNN_QMM_PB_BN=128|256 fixes it.
int pair_pb_bn(const OpsnnQmmParams* p)
{
    if (const char* e = env("OPSNN_QMM_PB_BN")) return atoi(e) == 256 ? 256 : 128;
    const int64_t tiles = p->batch * ((p->m + 255) / 256) * ((p->n + 255) / 256);
    return tiles >= sm_count() / 2 ? 256 : 128;
}

}  // namespace
