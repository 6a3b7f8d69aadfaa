// int8 / fp8 matmul with too few tiles for every SM: the k range is split, weight columns as the MMA's M. Included by qmm_umma.cu.
//
// What bounds such a call with one CTA per output tile is the serial chain of k-blocks of the few CTAs that have one, or a last wave that
// is nearly empty; and for a decode-sized m the epilogue of 128-row tiles that are mostly padding. Here
//   D^T = W^T x^T: the MMA's 128 rows are weight columns, its N the rows of x (a multiple of 16), so a tile is 256 columns x up to 128 rows
//   (two M = 128 accumulators) or 128 columns x up to 256 rows, and tensor work, operand traffic and epilogue shrink with m;
//   the (tile, k-block) pairs form one line that is cut into pieces: a tile into `split` equal ones, launched as a cluster and summed over
//   distributed shared memory, or all tiles together into one piece per SM (stream-k), straddled tiles summed through workspace by
//   whichever CTA arrives last. Pieces are added in k order, so results do not depend on timing; int8 sums are exact.
//   warps 0-7  epilogue: warp w reads TMEM lanes 32 (w % 4) .. (weight columns), accumulator half w / 4. Per-block mode promotes every
//              k-block into registers as the other kernels do (fma(part, s1 * s2, acc)); s1 * s2 of the rows of x come from a per-warp
//              ring in shared memory, filled a k-block ahead.
//   warp 8     TMA producer, warp 9 MMA issuer. All waits are bounded as in qmm_umma_kernel.
// x2 in either storage order (A operand of the MMA), x1 stored (m,k).
namespace {

struct SplitArgs {
    int64_t n, k, out_ld, out_bs, bias_bs, sa_bs, sb_bs;
    uint32_t m, rows, halves, t_tiles, n_tiles, kb, grid, units, split, stages, stage_bytes, x_off, dbufs;
    uint32_t w_mn, w_batched, x_batched, idesc;
    int32_t is_int, out_dtype, bias_dtype, scale_b_dtype, deq_flags, trans_sa, trans_sb;
    uint32_t group_m;
    const void* scale_a;
    const void* scale_b;
    int64_t scale_a_len, scale_b_len;
    const void* bias;
    void* out;
    uint32_t* part;                // [2 grid][rows][128 halves] raw 32-bit sums
    unsigned long long* count;     // [tiles] (nonce << 8) | arrivals
    unsigned long long nonce;
    uint32_t test_stop;  // tests of the give-up path only: k-blocks that a CTA's producer copies before it stops; otherwise all
};

constexpr int kSplitThreads = 320;
constexpr int kSplitMaxStages = 8;
constexpr uint32_t kSplitSmem = 225 * 1024;
constexpr uint32_t kSplitRing = 8 * 2 * 128 * 4;  // per-block: 8 warps x 2 k-blocks x 128 rows of x

__device__ __forceinline__ uint32_t split_begin(const SplitArgs& a, uint32_t c) { return (uint32_t)((uint64_t)c * a.units / a.grid); }
__device__ __forceinline__ uint32_t split_owner(const SplitArgs& a, uint32_t unit)
{
    uint32_t c = (uint32_t)((uint64_t)unit * a.grid / a.units);
    while (split_begin(a, c + 1) <= unit) ++c;
    while (split_begin(a, c) > unit) --c;
    return c;
}

// What turns a sum into an output element, for one weight column.
struct SplitCol {
    float sb, fbias;
    int32_t ibias;
};
template <bool kPerBlock>
__device__ __forceinline__ SplitCol split_col(const SplitArgs& a, uint32_t b, int64_t n)
{
    SplitCol c{1.f, 0.f, 0};
    if (!kPerBlock) c.sb = load_deq_scale(a.scale_b, a.scale_b_len == 1 ? 0 : n, a.scale_b_dtype);
    if (a.bias != nullptr) {
        if (a.bias_dtype == ACL_INT32 && !kPerBlock) c.ibias = __ldg(reinterpret_cast<const int32_t*>(a.bias) + b * a.bias_bs + n);
        else c.fbias = load_as_float(a.bias, b * a.bias_bs + n, a.bias_dtype);
    }
    return c;
}
template <bool kPerBlock>
__device__ __forceinline__ float split_value(const SplitArgs& a, uint32_t v, const SplitCol& c, float sa)
{
    const bool fb = a.bias != nullptr && (kPerBlock || a.bias_dtype != ACL_INT32);
    if (kPerBlock) return fb ? __fadd_rn(__uint_as_float(v), c.fbias) : __uint_as_float(v);
    const float f = a.is_int ? (float)((int32_t)v + c.ibias) : __uint_as_float(v);
    return deq_epilogue(f, c.sb, sa, a.scale_a != nullptr, c.fbias, fb, a.deq_flags);
}
template <bool kPerBlock>
__device__ __forceinline__ float split_sa(const SplitArgs& a, uint32_t row)
{
    return !kPerBlock && a.scale_a != nullptr ? __ldg(reinterpret_cast<const float*>(a.scale_a) + (a.scale_a_len == 1 ? 0 : row)) : 1.f;
}

struct SplitTile {
    uint32_t b, n0, r0, live;  // batch, first column, first row of x, rows of x inside m
};
__device__ __forceinline__ SplitTile split_tile(const SplitArgs& a, uint32_t t)
{
    SplitTile s;
    const uint32_t per = a.n_tiles * a.t_tiles;
    s.b = t / per;
    const uint32_t r = t - s.b * per, tn = r / a.t_tiles;
    s.n0 = tn * 128u * a.halves;
    s.r0 = (r - tn * a.t_tiles) * a.rows;
    s.live = min(a.rows, a.m - s.r0);
    return s;
}

// This CTA's slice of a tile whose pieces lie in the cluster's shared memory as [row of x][column] raw sums: 256 threads, 4 columns each.
// `sa`: the tile's x1 scales in shared memory; `c`: those of the thread's columns (split_cols4), both fetched during the main loop.
struct SplitCols4 {
    SplitCol c[4];
};
template <bool kPerBlock, uint32_t kHalves>
__device__ __forceinline__ SplitCols4 split_cols4(const SplitArgs& a, const SplitTile& t, uint32_t tid)
{
    SplitCols4 r;
    const uint32_t n = t.n0 + (tid % (32u * kHalves)) * 4u;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) r.c[i] = split_col<kPerBlock>(a, t.b, min((int64_t)n + i, a.n - 1));
    return r;
}
template <bool kPerBlock, uint32_t kHalves>
__device__ __forceinline__ void split_sum_and_store(const SplitArgs& a, uint32_t smem, const SplitTile& t, uint32_t rank, uint32_t tid, const float* s_sa,
                                                    const SplitCols4& cols4)
{
    constexpr uint32_t vecs = 32u * kHalves;  // 4-column pieces in a row; 256 is a multiple of it
    const uint32_t total = t.live * vecs;
    const uint32_t split = a.split;
    const uint32_t begin = (total * rank / split) / vecs * vecs, end = rank + 1u == split ? total : (total * (rank + 1u) / split) / vecs * vecs;
    const uint32_t n = t.n0 + (tid % vecs) * 4u;
    if (n >= a.n) return;
    const uint32_t cols = (uint32_t)min((int64_t)4, a.n - n);
    const int out_dtype = a.out_dtype, ob = out_elem_bytes(out_dtype);
    uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + (t.b * a.out_bs + n) * ob;
    const int64_t pitch = a.out_ld * ob;
    const bool is_int = a.is_int && !kPerBlock;
    constexpr int kBatch = 4;  // rows of x in flight: what bounds this loop is the latency of the reads from the other CTAs
    for (uint32_t i0 = begin + tid; i0 < end; i0 += 256u * kBatch) {
        uint32_t v[kBatch][4];
        for (uint32_t j = 0; j < split; ++j) {
            uint32_t q[kBatch][4];
#pragma unroll
            for (int r = 0; r < kBatch; ++r) {
                const uint32_t at = smem + min(i0 + 256u * r, total - 1u) * 16u;
                uint32_t remote = at;
                if (split > 1u) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(at), "r"(j));
                asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(q[r][0]), "=r"(q[r][1]), "=r"(q[r][2]), "=r"(q[r][3]) : "r"(remote));
            }
#pragma unroll
            for (int r = 0; r < kBatch; ++r)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    v[r][e] = j == 0 ? q[r][e]
                                     : (is_int ? v[r][e] + q[r][e] : __float_as_uint(__fadd_rn(__uint_as_float(v[r][e]), __uint_as_float(q[r][e]))));
        }
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
            const uint32_t i = i0 + 256u * r;
            if (i >= end) break;
            const uint32_t row = i / vecs;
            const float sa = kPerBlock ? 1.f : s_sa[row];
            float f[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) f[e] = split_value<kPerBlock>(a, v[r][e], cols4.c[e], sa);
            uint8_t* o = out + (int64_t)(t.r0 + row) * pitch;
            if (cols == 4u && out_dtype != ACL_FLOAT && (reinterpret_cast<uintptr_t>(o) & 7) == 0) {
                uint2 w;
                if (out_dtype == ACL_BF16) {
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(f[0], f[1]), hi = __floats2bfloat162_rn(f[2], f[3]);
                    w = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                } else {
                    const __half2 lo = __floats2half2_rn(f[0], f[1]), hi = __floats2half2_rn(f[2], f[3]);
                    w = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
                }
                *reinterpret_cast<uint2*>(o) = w;
            } else if (cols == 4u && out_dtype == ACL_FLOAT && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
                *reinterpret_cast<float4*>(o) = make_float4(f[0], f[1], f[2], f[3]);
            } else {
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e)
                    if (e < cols) store_out(o, e, f[e], out_dtype);
            }
        }
    }
}

// The same tile where few rows are left to a CTA (split_launch: `push`). Its live rows of x, four at a time, are dealt to the CTAs, split_share fours
// each in order of rank; every CTA stores its sums of them in their owner's shared memory, [piece][four of the share][columns][4 rows] in the
// place of the stages (at least 12 KB less than the stages of any form), and the owner adds the pieces up. Nobody reads another CTA's memory,
// so there is no second trip for the sums and nobody waits to leave.
__host__ __device__ __forceinline__ uint32_t split_share(uint32_t live, uint32_t split) { return ((live + 3u) / 4u + split - 1u) / split; }

// 16 rows of this thread's column, from row `row` of the tile on (a multiple of 16), to their owners.
template <uint32_t kHalves>
__device__ __forceinline__ void split_push16(uint32_t smem, uint32_t live, uint32_t split, uint32_t rank, uint32_t row, uint32_t col, const uint32_t (&v)[16])
{
    constexpr uint32_t kFour = 128u * kHalves * 16u;  // bytes of four rows
    const uint32_t per = split_share(live, split), mine = smem + rank * per * kFour + col * 16u;
    uint32_t owner = row / 4u / per, four = row / 4u - owner * per;
#pragma unroll
    for (uint32_t i = 0; i < 16; i += 4) {
        if (row + i >= live) break;
        uint32_t to;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine), "r"(owner));
        asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + four * kFour), "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]) : "memory");
        if (++four == per) { four = 0; ++owner; }
    }
}

// This CTA's share of a tile: the pieces added in their order and stored (256 threads, one column of four rows each; `c`: the column's scale and
// bias, `s_sa`: the tile's x1 scales, both fetched during the main loop).
template <uint32_t kHalves>
__device__ __forceinline__ void split_sum_fours(const SplitArgs& a, uint32_t smem, const SplitTile& t, uint32_t rank, uint32_t tid, const float* s_sa, const SplitCol& c)
{
    constexpr uint32_t kWidth = 128u * kHalves, kFour = kWidth * 16u;
    const uint32_t split = a.split, per = split_share(t.live, split), n = t.n0 + tid % kWidth;
    if (n >= a.n) return;
    const bool is_int = a.is_int != 0;
    const int64_t base = t.b * a.out_bs + n;
#pragma unroll 1
    for (uint32_t four = tid / kWidth; four < per; four += 256u / kWidth) {
        const uint32_t row = (rank * per + four) * 4u;
        uint32_t at = smem + four * kFour + tid % kWidth * 16u;
        uint32_t v[4];
#pragma unroll 2
        for (uint32_t j = 0; j < split; ++j, at += per * kFour) {
            uint32_t q[4];
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]) : "r"(at) : "memory");
#pragma unroll
            for (int e = 0; e < 4; ++e)
                v[e] = j == 0 ? q[e] : (is_int ? v[e] + q[e] : __float_as_uint(__fadd_rn(__uint_as_float(v[e]), __uint_as_float(q[e]))));
        }
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            if (row + e >= t.live) break;
            store_out(a.out, base + (int64_t)(t.r0 + row + e) * a.out_ld, split_value<false>(a, v[e], c, s_sa[row + e]), a.out_dtype);
        }
    }
}

// One thread's column of 16 rows of x, straight to the output (stream-k form).
template <bool kPerBlock>
__device__ __forceinline__ void split_store16(const SplitArgs& a, const SplitTile& t, int64_t n, const SplitCol& c, uint32_t row, const uint32_t (&v)[16])
{
    if (n >= a.n) return;
    const int64_t base = t.b * a.out_bs + n;
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) {
        if (row + i >= t.live) break;
        const uint32_t r = t.r0 + row + i;
        store_out(a.out, base + (int64_t)r * a.out_ld, split_value<kPerBlock>(a, v[i], c, split_sa<kPerBlock>(a, r)), a.out_dtype);
    }
}

// A finished piece in the stream-k form: stored if it is the whole tile, else parked in workspace and, by whoever arrives last, summed in
// k order. `get(i, v)` hands out sums i .. i + 15 of this thread. 256 threads; ends with all of them past their last use of `get`.
template <bool kPerBlock, typename Get>
__device__ __forceinline__ void split_finish(const SplitArgs& a, uint32_t t, uint32_t cnt, uint32_t cnt_rows, uint32_t row0, uint32_t col, bool leader,
                                             volatile uint32_t* s_last, volatile uint32_t* abort_flag, Get&& get)
{
    const SplitTile tile = split_tile(a, t);
    const int64_t n = (int64_t)tile.n0 + col;
    const uint32_t width = 128u * a.halves;
    const bool whole = cnt == a.kb;
    uint32_t* mine = a.part + (size_t)(2u * blockIdx.x + (t == split_begin(a, blockIdx.x) / a.kb ? 0u : 1u)) * a.rows * width + (size_t)row0 * width + col;
    const SplitCol c = split_col<kPerBlock>(a, tile.b, min(n, a.n - 1));
#pragma unroll
    for (uint32_t i = 0; i < 128; i += 16) {
        if (i >= cnt_rows) break;
        uint32_t v[16];
        get(i, v);
        if (whole) {
            split_store16<kPerBlock>(a, tile, n, c, row0 + i, v);
        } else {
#pragma unroll
            for (uint32_t e = 0; e < 16; ++e) __stcg(mine + (size_t)(i + e) * width, v[e]);
        }
    }
    if (whole) return;
    const uint32_t c0 = split_owner(a, t * a.kb), c1 = split_owner(a, (t + 1u) * a.kb - 1u);  // the CTAs whose pieces meet this tile
    __threadfence();
    asm volatile("bar.sync 1, 256;" ::: "memory");  // all of this CTA's sums are written and fenced
    if (leader) {
        unsigned long long* cnt_p = a.count + t;
        unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(cnt_p), want = 0ull;
        bool done = false;
        for (int it = 0; it < 4096 && !done; ++it) {  // at most c1 - c0 other CTAs can get in between
            want = ((cur >> 8) == a.nonce) ? cur + 1ull : ((a.nonce << 8) | 1ull);
            const unsigned long long prev = atomicCAS(cnt_p, cur, want);
            done = prev == cur;
            cur = prev;
        }
        if (!done) report(abort_flag, (3u << 8) | 3u);
        const bool last = done && (uint32_t)(want & 0xFFull) == c1 - c0 + 1u;
        if (last) *reinterpret_cast<volatile unsigned long long*>(cnt_p) = 0ull;  // a replay of this launch starts clean
        *s_last = last ? 1u : 0u;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (*s_last == 0u) return;
    __threadfence();
#pragma unroll 1
    for (uint32_t i = 0; i < cnt_rows; i += 16) {
        if (row0 + i >= tile.live) break;
        uint32_t v[16];
#pragma unroll
        for (uint32_t e = 0; e < 16; ++e) v[e] = 0u;
#pragma unroll 2
        for (uint32_t j = c0; j <= c1; ++j) {
            // only the first of a CTA's tiles can be shared with the CTAs before it: its other shared tile starts with it
            const uint32_t slot = 2u * j + (j == c0 && split_begin(a, j) / a.kb != t ? 1u : 0u);
            const uint32_t* p = a.part + (size_t)slot * a.rows * width + (size_t)(row0 + i) * width + col;
            uint32_t q[16];
#pragma unroll
            for (uint32_t e = 0; e < 16; ++e) q[e] = __ldcg(p + (size_t)e * width);
#pragma unroll
            for (uint32_t e = 0; e < 16; ++e)
                v[e] = a.is_int && !kPerBlock ? v[e] + q[e] : (j == c0 ? q[e] : __float_as_uint(__fadd_rn(__uint_as_float(v[e]), __uint_as_float(q[e]))));
        }
        split_store16<kPerBlock>(a, tile, n, c, row0 + i, v);
    }
}

// kAcc: sums one epilogue thread keeps in registers (per-block mode), at least the rows of x that it serves. kOrder: how x2 is stored (kMe). kForm: how the
// line is cut and its pieces come together. An instance each: the forms' ends in one kernel cost all of them registers and instruction fetches. us, weights
// from HBM, one instance / each its own: streams 64 x 384 x 40960 int8 24.2 / 23.6, 60 x 512 x 36864 10.7 / 9.5, 48 x 7168 x 30720 fp8 39.6 / 38.6; fetched
// 128 x 4096 x 4096 int8 9.9 / 9.7, 717 x 7168 x 2304 fp8 17.5 / 17.1, 300 x 4096 x 2048 int8 10.8 / 10.5; sent 16 x 1472 x 4880 int8 6.2 / 6.1; per-block
// 128 x 4096 x 4096 12.5 / 12.1, (n,k) 100 x 7168 x 4096 14.6 / 13.9.
constexpr int kOrderAny = 0, kOrderKN = 1, kOrderNK = 2;
constexpr int kFormStream = 1, kFormFetch = 2, kFormPush = 3;  // kFormFetch: also one piece a tile
template <ptx::MmaKind kKind, bool kPerBlock, int kAcc, uint32_t kHalves, int kOrder, int kForm>
__global__ void __launch_bounds__(kSplitThreads, 1)
qmm_umma_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ SplitArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    // The out-of-line part of the waits, shared by all kernels of the file, is compiled to a convention that all of them can live with. Where the chain of
    // waits is most of a call it is worth a copy for the instance alone: us, graph replay, weights from HBM, shared / own, 128 x 4096 x 4096 int8 10.6 / 9.9,
    // 717 x 7168 x 2304 fp8 18.7 / 17.2, 14 x 8640 x 6048 fp8 17.9 / 16.0, 300 x 4096 x 2048 int8 11.6 / 10.8; per-block on weights stored (n,k)
    // 5 x 8320 x 14080 27.6 / 24.9 (25.8 since the forms are instances), 14 x 4480 x 15872 17.3 / 16.2, 24 x 7168 x 18432 25.4 / 25.3. Per-block on (k,n) it is not: 16 x 10368 x 3584 15.3 / 14.8, but
    // 5 x 8320 x 14080 28.3 / 28.8, 14 x 4480 x 15872 18.9 / 19.1, 100 x 7168 x 4096 15.9 / 16.2. That is why the order is a template argument there.
    // (The fused weight-only, pair and block-scaled kernels do not change.)
    constexpr int kMe = !kPerBlock ? 100 * kForm + (int)kKind * 2 + (int)kHalves : (kOrder == kOrderNK ? 1000 * kForm + kAcc + (int)kHalves : 0);
    const bool w_mn = kOrder == kOrderAny ? a.w_mn != 0u : kOrder == kOrderKN;
    const uint32_t smem0 = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    __shared__ __align__(8) uint64_t s_bars[2 * kSplitMaxStages + 8];
    __shared__ uint32_t s_tmem;
    __shared__ volatile uint32_t s_abort, s_last, s_bad;  // s_bad: a CTA of the cluster gave up a wait
    __shared__ float s_sa[256];  // x1 scales of the tile's rows (one piece per CTA)
    const uint32_t full0 = ptx::smem_u32(s_bars), empty0 = full0 + 8u * kSplitMaxStages, tfull0 = empty0 + 8u * kSplitMaxStages, tempty0 = tfull0 + 32u;
    volatile uint32_t* abort_flag = &s_abort;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;

    // programmatic dependent launch: placed and set up under the tail of the kernel before it, reads nothing until that has finished
    if (threadIdx.x == 0) {
        s_abort = 0u;
        s_bad = 0u;
        for (uint32_t i = 0; i < a.stages; ++i) {
            ptx::mbar_init(&s_bars[i], 1);
            ptx::mbar_init(&s_bars[kSplitMaxStages + i], 1);
        }
        for (uint32_t i = 0; i < 4; ++i) {
            ptx::mbar_init(&s_bars[2 * kSplitMaxStages + i], 1);
            ptx::mbar_init(&s_bars[2 * kSplitMaxStages + 4 + i], 8);  // one arrival per epilogue warp
        }
        ptx::fence_mbar_init();
    }
    if (warp == 9) ptx::tmem_alloc(&s_tmem, 512);
    if (warp == 8 && lane == 0) {
        ptx::tma_prefetch_desc(&map_w);
        ptx::tma_prefetch_desc(&map_x);
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_trigger();
    pdl_wait();

    const uint32_t u_begin = split_begin(a, blockIdx.x), u_end = split_begin(a, blockIdx.x + 1);
    SplitCols4 cols4;  // (per-block: only a bias, read at the end; 16 registers the sums need)
    constexpr bool push = kForm == kFormPush;  // a cluster's sums are sent to their owners (split_push16), not fetched
    constexpr bool stream = kForm == kFormStream;
    SplitCol own{1.f, 0.f, 0};  // push: of the column that this thread serves in the end
    bool met = false;           // push: this warp has met the cluster's others at the end of the stages
    if (warp < 8 && !stream) {
        const SplitTile tile = split_tile(a, blockIdx.x / a.split);
        if constexpr (!kPerBlock) {
            if (push) own = split_col<false>(a, tile.b, min((int64_t)tile.n0 + threadIdx.x % (128u * kHalves), a.n - 1));
            else cols4 = split_cols4<kPerBlock, kHalves>(a, tile, threadIdx.x);
        }
        if (!kPerBlock && threadIdx.x < a.rows) s_sa[threadIdx.x] = split_sa<kPerBlock>(a, tile.r0 + min(threadIdx.x, tile.live - 1u));
    }
    const uint32_t set = kHalves * a.rows;  // TMEM columns of one accumulator buffer

    if (warp == 8) {
        // ======================= TMA producer =======================
        // One warp with nothing to hide latency behind: everything the loop uses is in registers (with the launch parameters read where
        // they are used, a k-block cost this warp and the next 0.6 us each, more than its copies and its MMAs).
        const uint32_t stages = a.stages, stage_bytes = a.stage_bytes, x_off = a.x_off, kbs = a.kb, bytes = kHalves * kATile + a.rows * BK;
        const bool w_batched = a.w_batched != 0, x_batched = a.x_batched != 0;
        uint32_t s = 0, par = 0, t = u_begin / kbs, kb = u_begin - t * kbs;
        SplitTile tile = split_tile(a, t);
        const uint32_t u_stop = u_begin + min(u_end - u_begin, a.test_stop);
        for (uint32_t u = u_begin; u < u_stop; ++u) {
            if (!ptx::mbar_wait_a<kMe>(empty0 + 8u * s, par ^ 1u, abort_flag)) {
                report(abort_flag, (1u << 8) | 1u);
                break;
            }
            if (ptx::elect_one()) {
                const uint32_t fb = full0 + 8u * s, dst = smem0 + s * stage_bytes;
                const int32_t k0 = (int32_t)(kb * BK), bw = w_batched ? (int32_t)tile.b : 0, bx = x_batched ? (int32_t)tile.b : 0;
                ptx::mbar_expect_tx_a(fb, bytes);
#pragma unroll
                for (uint32_t h = 0; h < kHalves; ++h) {
                    const int32_t n0 = (int32_t)(tile.n0 + 128u * h);
                    ptx::tma_load_3d_a(dst + h * kATile, &map_w, fb, w_mn ? n0 : k0, w_mn ? k0 : n0, bw);
                }
                ptx::tma_load_3d_a(dst + x_off, &map_x, fb, k0, (int32_t)tile.r0, bx);
            }
            __syncwarp();
            if (++s == stages) { s = 0; par ^= 1u; }
            if (++kb == kbs) {
                kb = 0;
                if (u + 1 < u_end) tile = split_tile(a, ++t);
            }
        }
    } else if (warp == 9) {
        // ======================= MMA issuer =======================
        const uint64_t dw = w_mn ? ptx::make_smem_desc(smem0, 128 * BK, 1024, 2) : ptx::make_smem_desc(smem0, 0, 1024, 2);
        const uint64_t dx = ptx::make_smem_desc(smem0 + a.x_off, 0, 1024, 2);
        const uint32_t w_lo = (uint32_t)dw, x_lo = (uint32_t)dx, w_k = w_mn ? 256u : 2u;
        const uint64_t w_hi = dw & 0xFFFFFFFF00000000ull, x_hi = dx & 0xFFFFFFFF00000000ull;
        const uint32_t stages = a.stages, stage16 = a.stage_bytes >> 4, rows = a.rows, idesc = a.idesc, kbs = a.kb, dbufs = a.dbufs;
        uint32_t s = 0, par = 0, off = 0, buf = 0, bpar = 0, kb = u_begin % kbs;
        uint32_t acc = 0u;
        bool fresh = true;
        for (uint32_t u = u_begin; u < u_end; ++u) {
            if (kPerBlock || fresh) {
                if (!ptx::mbar_wait_a<kMe>(tempty0 + 8u * buf, bpar ^ 1u, abort_flag)) {
                    report(abort_flag, (2u << 8) | 1u);
                    break;
                }
                fresh = false;
            }
            if (!ptx::mbar_wait_a<kMe>(full0 + 8u * s, par, abort_flag)) {
                report(abort_flag, (2u << 8) | 2u);
                break;
            }
            ptx::tc_fence_after();
            const bool last = kPerBlock || kb + 1 == kbs || u + 1 == u_end;
            if (ptx::elect_one()) {
                const uint32_t d = tmem + buf * set, wl = w_lo + off, xl = x_lo + off;
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (uint32_t h = 0; h < kHalves; ++h)
                        ptx::umma<kKind>(d + h * rows, w_hi | (uint64_t)(wl + h * (kATile >> 4) + k * w_k), x_hi | (uint64_t)(xl + 2u * k), idesc,
                                         k == 0 ? acc : 1u);
                ptx::umma_commit_a(empty0 + 8u * s);
                if (last) ptx::umma_commit_a(tfull0 + 8u * buf);
            }
            __syncwarp();
            acc = last ? 0u : 1u;
            if (last) {
                fresh = true;
                if (++buf == dbufs) { buf = 0; bpar ^= 1u; }
            }
            off += stage16;
            if (++s == stages) { s = 0; off = 0; par ^= 1u; }
            if (++kb == kbs) kb = 0;
        }
    } else {
        // ======================= epilogue =======================
        const uint32_t quad = warp & 3, hf = (uint32_t)warp >> 2;
        const uint32_t cnt_rows = kHalves == 2u ? a.rows : a.rows / 2u;  // rows of x this thread serves, of its one column
        const uint32_t col = (kHalves == 2u ? hf * 128u : 0u) + quad * 32u + lane, row0 = kHalves == 2u ? 0u : hf * cnt_rows;
        const uint32_t tbase = tmem + ((quad * 32u) << 16) + hf * cnt_rows;
        const uint32_t ring = smem0 + a.stages * a.stage_bytes + (uint32_t)warp * (2u * 128u * 4u);
        uint32_t buf = 0, bpar = 0, u = u_begin, t = u_begin / a.kb, kb = u_begin - t * a.kb;
        bool ok = true;
        while (u < u_end && ok) {
            const uint32_t cnt = min(a.kb - kb, u_end - u);
            float acc[kPerBlock ? kAcc : 1];
            uint32_t done_buf = 0;
            if constexpr (kPerBlock) {
                const SplitTile tile = split_tile(a, t);
#pragma unroll
                for (int i = 0; i < kAcc; ++i) acc[i] = 0.f;
                const uint32_t groups = (a.m + a.group_m - 1) / a.group_m, ngroups = (uint32_t)((a.n + 127) / 128);
                const uint32_t ng = min((tile.n0 + col) / 128u, ngroups - 1);
                const float* s1 = reinterpret_cast<const float*>(a.scale_a) + tile.b * a.sa_bs;
                const float* s2 = reinterpret_cast<const float*>(a.scale_b) + tile.b * a.sb_bs;
                constexpr int kPerLane = (kAcc + 31) / 32;
                float s1v[kPerLane], s2v = 0.f;
                auto fetch = [&](uint32_t k) {  // scales of k-block k: the warp's rows of x over the lanes, its column block's
                    k = min(k, a.kb - 1u);
#pragma unroll
                    for (int i = 0; i < kPerLane; ++i) {
                        const uint32_t g = min(tile.r0 + row0 + 32u * i + lane, a.m - 1u) / a.group_m;
                        s1v[i] = __ldg(s1 + (a.trans_sa ? (int64_t)k * groups + g : (int64_t)g * a.kb + k));
                    }
                    s2v = __ldg(s2 + (a.trans_sb ? (int64_t)ng * a.kb + k : (int64_t)k * ngroups + ng));
                };
                auto publish = [&](uint32_t k) {
#pragma unroll
                    for (int i = 0; i < kPerLane; ++i)
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(ring + (k & 1u) * 512u + (32u * i + lane) * 4u), "f"(__fmul_rn(s1v[i], s2v)) : "memory");
                };
                fetch(kb);
                publish(kb);
                fetch(kb + 1);
                for (uint32_t k = kb; k < kb + cnt; ++k) {
                    publish(k + 1);
                    fetch(k + 2);
                    if (!__all_sync(0xffffffffu, ptx::mbar_wait_a<kMe>(tfull0 + 8u * buf, bpar, abort_flag))) {
                        report(abort_flag, (3u << 8) | 2u);
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t t0 = tbase + buf * set, rk = ring + (k & 1u) * 512u;
                    // 16 sums at a time, the next 16 on their way while these are promoted
                    uint32_t va[16], vb[16];
                    auto promote16 = [&](const uint32_t (&v)[16], int i) {
#pragma unroll
                        for (int e = 0; e < 16; e += 4) {
                            float4 sc;
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(sc.x), "=f"(sc.y), "=f"(sc.z), "=f"(sc.w) : "r"(rk + (i + e) * 4));
                            acc[i + e] = fmaf(__uint_as_float(v[e]), sc.x, acc[i + e]);
                            acc[i + e + 1] = fmaf(__uint_as_float(v[e + 1]), sc.y, acc[i + e + 1]);
                            acc[i + e + 2] = fmaf(__uint_as_float(v[e + 2]), sc.z, acc[i + e + 2]);
                            acc[i + e + 3] = fmaf(__uint_as_float(v[e + 3]), sc.w, acc[i + e + 3]);
                        }
                    };
                    ptx::tmem_ld16(t0, va);
#pragma unroll
                    for (int i = 0; i < kAcc; i += 32) {
                        if ((uint32_t)i < cnt_rows) {
                            ptx::tmem_ld_wait();
                            if ((uint32_t)(i + 16) < cnt_rows) ptx::tmem_ld16(t0 + i + 16, vb);
                            promote16(va, i);
                        }
                        if ((uint32_t)(i + 16) < cnt_rows) {
                            ptx::tmem_ld_wait();
                            if (i + 32 < kAcc && (uint32_t)(i + 32) < cnt_rows) ptx::tmem_ld16(t0 + i + 32, va);
                            promote16(vb, i + 16);
                        }
                    }
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(&s_bars[2 * kSplitMaxStages + 4 + buf]);
                    if (++buf == a.dbufs) { buf = 0; bpar ^= 1u; }
                }
            } else {
                if (!__all_sync(0xffffffffu, ptx::mbar_wait_relaxed(&s_bars[2 * kSplitMaxStages + buf], bpar, abort_flag))) {
                    report(abort_flag, (3u << 8) | 1u);
                    ok = false;
                }
                done_buf = buf;
                if (++buf == a.dbufs) { buf = 0; bpar ^= 1u; }
            }
            {  // the eight warps go on, or leave, together
                uint32_t r;
                asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 1, 256, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(r)
                             : "r"(ok ? 1u : 0u)
                             : "memory");
                ok = r != 0u;
            }
            if (!ok) break;
            ptx::tc_fence_after();
            auto get = [&](uint32_t i, uint32_t (&v)[16]) {
                if constexpr (kPerBlock) {
#pragma unroll
                    for (int j = 0; j < kAcc; j += 16)
                        if ((uint32_t)j == i) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) v[e] = __float_as_uint(acc[j + e]);
                        }
                } else {
                    ptx::tmem_ld16(tbase + done_buf * set + i, v);
                    ptx::tmem_ld_wait();
                }
            };
            if (stream) {
                split_finish<kPerBlock>(a, t, cnt, cnt_rows, row0, col, threadIdx.x == 0, &s_last, abort_flag, get);
            } else if (push) {
                // where every CTA of the cluster is done with its stages, the sums go to their owners
                const uint32_t live = split_tile(a, t).live;
                __syncwarp();
                ptx::cluster_arrive();
                ptx::cluster_wait();
                met = true;
#pragma unroll 1
                for (uint32_t i = 0; i < cnt_rows && row0 + i < live; i += 16) {
                    uint32_t v[16];
                    get(i, v);
                    split_push16<kHalves>(smem0, live, a.split, ptx::cluster_ctarank(), row0 + i, col, v);
                }
            } else {
                // the tile's only piece here: into shared memory (no copy is in flight any more), as [row of x][column]
                constexpr uint32_t width = 128u * kHalves;
                constexpr int kUnroll = kPerBlock ? 8 : 1;  // (per-block: its sums are registers)
#pragma unroll kUnroll
                for (uint32_t i = 0; i < 128; i += 16) {
                    if (i >= cnt_rows) break;
                    uint32_t v[16];
                    get(i, v);
#pragma unroll
                    for (uint32_t e = 0; e < 16; ++e)
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(smem0 + ((row0 + i + e) * width + col) * 4u), "r"(v[e]) : "memory");
                }
                if (a.split == 1u) {
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if constexpr (kPerBlock) cols4 = split_cols4<kPerBlock, kHalves>(a, split_tile(a, t), threadIdx.x);
                    split_sum_and_store<kPerBlock, kHalves>(a, smem0, split_tile(a, t), 0u, threadIdx.x, s_sa, cols4);
                }
            }
            if (!kPerBlock) {
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&s_bars[2 * kSplitMaxStages + 4 + done_buf]);
            }
            u += cnt;
            kb = 0;
            ++t;
        }
    }
    if (push) {
        // A CTA that gave up a wait joins both barriers too; what it sends is not used, and then nobody writes.
        if (!met) {
            __syncwarp();
            ptx::cluster_arrive();
            ptx::cluster_wait();
        }
        if (threadIdx.x < a.split && *abort_flag != 0u) {  // (final: every warp's waits lie behind it)
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(ptx::smem_u32(const_cast<uint32_t*>(&s_bad))), "r"(threadIdx.x));
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(1u) : "memory");
        }
        __syncwarp();
        ptx::cluster_arrive();
        ptx::cluster_wait();
        if (warp < 8 && s_bad == 0u) split_sum_fours<kHalves>(a, smem0, split_tile(a, blockIdx.x / a.split), ptx::cluster_ctarank(), threadIdx.x, s_sa, own);
    } else if (!stream && a.split > 1u) {
        // the pieces of the tile meet; a CTA that gave up a wait still joins both barriers, and then nobody writes
        __syncwarp();
        ptx::cluster_sync();
        if (warp < 8) {
            uint32_t bad = 0u;
            if ((uint32_t)lane < a.split) {
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(ptx::smem_u32(const_cast<uint32_t*>(&s_abort))), "r"((uint32_t)lane));
                asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(bad) : "r"(remote) : "memory");
            }
            if constexpr (kPerBlock) cols4 = split_cols4<kPerBlock, kHalves>(a, split_tile(a, blockIdx.x / a.split), threadIdx.x);
            if (!__any_sync(0xffffffffu, bad != 0u))
                split_sum_and_store<kPerBlock, kHalves>(a, smem0, split_tile(a, blockIdx.x / a.split), ptx::cluster_ctarank(), threadIdx.x, s_sa, cols4);
        }
        ptx::cluster_sync();
    }
    if (*abort_flag != 0u) __nanosleep(200000);  // lets bulk copies that are still in flight land before the CTA leaves
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 512);
    }
}

using SplitKernel = void (*)(const CUtensorMap, const CUtensorMap, const SplitArgs);

struct SplitPlan {
    uint32_t rows = 0, halves = 0, t_tiles = 0, n_tiles = 0, kb = 0, split = 0, stages = 0, stage_bytes = 0;
    int64_t tiles = 0, units = 0, grid = 0;
    double cost = 1e30;  // us
    int acc = 0;
};

// Whether the split kernel takes the call at all.
bool split_takes(const OpsnnQmmParams* p)
{
    if (env("OPSNN_QMM_NO_SPLIT")) return false;
    // beyond this the promotion (per-block) or the two-byte stores of shared tiles (dequant) cost more than idle SMs do
    if (p->mode == OPSNN_QMM_PERBLOCK && p->m > 128) return false;
    const bool i8 = p->a_dtype == ACL_INT8, f8 = is_fp8(p->a_dtype);
    // int8 per-block sums are tested bit for bit against the reference's order of k-blocks: they are not split
    if (!(p->mode == OPSNN_QMM_DEQ && (i8 || f8)) && !(p->mode == OPSNN_QMM_PERBLOCK && f8)) return false;
    if (p->out_dtype != ACL_BF16 && p->out_dtype != ACL_FLOAT16 && p->out_dtype != ACL_FLOAT) return false;
    if (p->trans_a || (p->deq_flags & OPSNN_DEQ_REQUANT)) return false;
    if (p->m >= (1 << 24) || p->n >= (1 << 30) || p->k >= (1 << 30)) return false;
    return p->batch * ((p->m + 15) / 16) * ((p->n + 127) / 128) * ((p->k + 127) / 128) < ((int64_t)1 << 31);
}

// One candidate tile shape (halves; t_tiles row tiles more than needed), cut in the cheapest way. The costs (us) were fitted to fp8 and
// int8 calls of 16 to 717 rows: launch and ramp, a k-block's fixed part, its tensor work (or promotion) and its share of a stream of
// weights out of HBM, and the combination, which grows with the tile. `most_cost`: a way that costs as much is of no use, so that the device is not
// asked about its clusters (asked about all of them, eight candidates of up to sixteen, it took most of a call's 11 - 17 us on the host).
template <typename F>
SplitPlan split_candidate(const OpsnnQmmParams* p, uint32_t halves, uint32_t more, int sms, double most_cost, F&& clusters)
{
    SplitPlan q;
    const bool pb = p->mode == OPSNN_QMM_PERBLOCK;
    const uint32_t most_rows = halves == 2 ? 128 : 256, unit = halves == 2 ? 16 : 32;
    q.halves = halves;
    q.t_tiles = (uint32_t)((p->m + most_rows - 1) / most_rows) + more;
    const uint32_t per = (uint32_t)((p->m + q.t_tiles - 1) / q.t_tiles);
    q.rows = (per + unit - 1) / unit * unit;
    q.t_tiles = (uint32_t)((p->m + q.rows - 1) / q.rows);
    q.n_tiles = (uint32_t)((p->n + 128 * halves - 1) / (128 * halves));
    q.kb = (uint32_t)((p->k + BK - 1) / BK);
    q.tiles = p->batch * q.n_tiles * q.t_tiles;
    q.units = q.tiles * q.kb;
    const uint32_t served = halves == 2 ? q.rows : q.rows / 2;
    if (pb && served > 64) return q;
    q.acc = served <= 32 ? 32 : 64;
    q.stage_bytes = halves * kATile + q.rows * BK;
    q.stages = (kSplitSmem - 2048 - (pb ? kSplitRing : 0u)) / q.stage_bytes;
    if (q.stages > (uint32_t)kSplitMaxStages) q.stages = kSplitMaxStages;
    const double area = (double)q.rows * halves;
    q.cost = most_cost;
    auto cost_of = [&](int64_t grid, double extra) {
        double w = 0.12 + (pb ? 0.0075 * served : 0.00135 * area);
        const double hbm = (double)grid * halves * kATile / q.t_tiles / 5.8e6;  // all CTAs' weights of one k-block
        if (hbm > w) w = hbm;
        return 5.5 + (double)((q.units + grid - 1) / grid) * w + extra;
    };
    auto take = [&](int64_t grid, uint32_t split, double cost) {
        q.cost = cost;
        q.grid = grid;
        q.split = split;
    };
    const int64_t all = q.units < sms ? q.units : sms;
    // Whoever arrives last adds a tile's pieces up alone, 0.6 us each: few tiles with a long k are many pieces (us, before / since that was counted:
    // 8 x 7168 x 512 int8 56.0 / 8.4, 16 x 16384 x 256 fp8 131.6 / 11.4, per-block 24 x 7168 x 384 43.4 / 8.1, 1 x 8192 x 1024 35.5 / 9.0).
    const double stream = cost_of(all, 1.0 + area * 0.05 + 0.6 * std::max(0.0, (double)q.kb * all / q.units - 4.0));
    if (stream < q.cost) take(all, 0, stream);
    int64_t most = sms / q.tiles;
    if (most > 16) most = 16;
    if (most > q.kb) most = q.kb;
    // of the cheapest first, so that one answer is enough nearly always
    for (uint32_t refused = 0;;) {
        int best = 0;
        double cost = q.cost;
        for (int s = (int)most; s >= 1; --s) {
            if ((refused >> s) & 1u) continue;
            const double c = cost_of(q.tiles * s, s > 1 ? std::max(0.4, 0.6 * s + 0.012 * area - 1.8) : 0.02 * area);
            if (c < cost) {
                cost = c;
                best = s;
            }
        }
        if (best == 0) break;
        if (best == 1 || (int64_t)clusters(q, best) >= q.tiles) {
            take(q.tiles * best, (uint32_t)best, cost);
            break;
        }
        refused |= 1u << best;
    }
    return q;
}

template <uint32_t kHalves, int kOrder, int kForm>
SplitKernel split_per_block(int acc)
{
    if (acc == 32) return &qmm_umma_split_kernel<ptx::MmaKind::kF8F6F4, true, 32, kHalves, kOrder, kForm>;
    return &qmm_umma_split_kernel<ptx::MmaKind::kF8F6F4, true, 64, kHalves, kOrder, kForm>;
}
template <ptx::MmaKind kKind, uint32_t kHalves>
SplitKernel split_kernel_of(bool per_block, int acc, bool w_mn, int form)
{
    if constexpr (kKind == ptx::MmaKind::kF8F6F4) {
        if (per_block) {
            if (form == kFormStream) return w_mn ? split_per_block<kHalves, kOrderKN, kFormStream>(acc) : split_per_block<kHalves, kOrderNK, kFormStream>(acc);
            return w_mn ? split_per_block<kHalves, kOrderKN, kFormFetch>(acc) : split_per_block<kHalves, kOrderNK, kFormFetch>(acc);
        }
    }
    if (form == kFormPush) return &qmm_umma_split_kernel<kKind, false, 16, kHalves, kOrderAny, kFormPush>;
    if (form == kFormStream) return &qmm_umma_split_kernel<kKind, false, 16, kHalves, kOrderAny, kFormStream>;
    return &qmm_umma_split_kernel<kKind, false, 16, kHalves, kOrderAny, kFormFetch>;
}
// The kernel of a plan, ready to launch on the current device; nullptr when it cannot be made ready.
SplitKernel split_kernel(bool i8, bool per_block, bool w_mn, const SplitPlan& q, int form)
{
    const SplitKernel k = i8 ? (q.halves == 2 ? split_kernel_of<ptx::MmaKind::kI8, 2>(per_block, q.acc, w_mn, form) : split_kernel_of<ptx::MmaKind::kI8, 1>(per_block, q.acc, w_mn, form))
                             : (q.halves == 2 ? split_kernel_of<ptx::MmaKind::kF8F6F4, 2>(per_block, q.acc, w_mn, form) : split_kernel_of<ptx::MmaKind::kF8F6F4, 1>(per_block, q.acc, w_mn, form));
    static std::atomic<uint64_t> configured[2 * 14];
    const int index = (q.halves == 2 ? 14 : 0) + (!per_block ? (i8 ? 0 : 3) + form - 1 : 6 + (q.acc == 32 ? 0 : 4) + (w_mn ? 2 : 0) + form - 1);
    const cudaError_t rc = once_per_device(configured[index], [&] {
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem);
    });
    return rc == cudaSuccess ? k : nullptr;
}

// Sent or fetched: a column of four rows at a time is summed with less code and fewer waits, but by 256 threads whose stores are two bytes wide; up to four
// fours a thread it is the faster. us, graph replay, weights from HBM, fetched / sent, where it is sent: 16 x 1472 x 4880 int8 6.65 / 6.07, 24 x 7168 x 384 7.82 /
// 6.89, 32 x 4096 x 3072 fp8 8.53 / 8.06, 64 x 4096 x 3072 8.91 / 8.87, 83 x 4096 x 3072 int8 8.96 / 8.78, 200 x 4096 x 1024 8.96 / 7.79 (14 x 8640 x 6048 fp8 15.70 /
// 15.86); where it is fetched: 96 x 4096 x 4096 int8 9.78 / 10.25, 128 rows 9.92 / 10.35, 300 x 4096 x 2048 10.46 / 11.18, 717 x 7168 x 2304 fp8 16.9 / 18.9.
// Per-block, whose sums are in registers, it is 3 - 6 % slower at 14 and 100 rows.
int split_form(const OpsnnQmmParams* p, const SplitPlan& q)
{
    if (q.split == 0) return kFormStream;
    if (p->mode == OPSNN_QMM_PERBLOCK) return kFormFetch;
    if (const char* e = env("OPSNN_QMM_SPLIT_PUSH")) return q.split > 1u && atoi(e) != 0 ? kFormPush : kFormFetch;  // tests and experiments (any share fits)
    return q.split > 1u && split_share(std::min(q.rows, (uint32_t)p->m), q.split) * q.halves <= 4u ? kFormPush : kFormFetch;
}

cudaError_t split_prepare(const OpsnnQmmParams* p, SplitKernel* kern, SplitPlan* plan)
{
    const bool i8 = p->a_dtype == ACL_INT8, pb = p->mode == OPSNN_QMM_PERBLOCK;
    int device = -1;
    const bool have_device = cudaGetDevice(&device) == cudaSuccess;
    const int sms = have_device ? sm_count() : 148;
    const char* only = env("OPSNN_QMM_SPLIT_HALVES");  // experiments
    *plan = SplitPlan{};
    for (uint32_t c = 0; c < 8; ++c) {
        const uint32_t halves = 2u - (c & 1u);
        if (only != nullptr && atoi(only) != (int)halves) continue;
        const SplitPlan q = split_candidate(p, halves, c >> 1, sms, plan->cost, [&](const SplitPlan& c, int s) -> int {
            const SplitKernel k = have_device ? split_kernel(i8, pb, p->trans_b == 0, c, kFormFetch) : nullptr;  // (clusters of all forms are placed alike)
            return k == nullptr ? 0 : max_active_clusters(reinterpret_cast<const void*>(k), kSplitThreads, kSplitSmem, s, 0);
        });
        if (q.grid != 0 && q.cost < plan->cost) *plan = q;
    }
    if (plan->grid == 0) return cudaErrorNotSupported;
    *kern = nullptr;
    if (!have_device) return cudaErrorNoDevice;
    *kern = split_kernel(i8, pb, p->trans_b == 0, *plan, split_form(p, *plan));
    return *kern != nullptr ? cudaSuccess : cudaGetLastError();
}

uint64_t split_workspace(const SplitPlan& q)
{
    if (q.split != 0) return 0;
    const uint64_t counters = ((uint64_t)q.tiles * 8u + 255u) & ~(uint64_t)255u;
    return 256u + counters + 2u * (uint64_t)q.grid * q.rows * 128u * q.halves * 4u;
}

// A call's kernel and plan, made once by whoever asks first.
struct SplitChoice {
    SplitKernel kern = nullptr;
    SplitPlan plan;
    int known = 0;  // 1: they are there, -1: there are none
    bool get(const OpsnnQmmParams* p)
    {
        if (known == 0) {
            known = split_prepare(p, &kern, &plan) == cudaSuccess ? 1 : -1;
            if (known < 0) cudaGetLastError();
        }
        return known > 0;
    }
};

// 0: launched (or a CUDA error); -1: not this kernel's call.
int32_t split_launch(const OpsnnQmmParams* p, SplitChoice& choice, cudaStream_t stream)
{
    if (!choice.get(p)) return -1;
    const SplitKernel kern = choice.kern;
    const SplitPlan& q = choice.plan;
    if (q.split == 0 && (p->workspace == nullptr || p->workspace_size < split_workspace(q))) return -1;
    const bool pb = p->mode == OPSNN_QMM_PERBLOCK;
    SplitArgs a{};
    a.n = p->n; a.k = p->k; a.m = (uint32_t)p->m;
    a.rows = q.rows; a.halves = q.halves; a.t_tiles = q.t_tiles; a.n_tiles = q.n_tiles; a.kb = q.kb;
    a.grid = (uint32_t)q.grid; a.units = (uint32_t)q.units; a.split = q.split; a.stages = q.stages; a.stage_bytes = q.stage_bytes;
    a.x_off = q.halves * kATile;
    a.dbufs = pb ? std::min(4u, 512u / (q.halves * q.rows)) : 2u;
    a.w_mn = p->trans_b ? 0 : 1;
    a.w_batched = p->b_bs != 0;
    a.x_batched = p->a_bs != 0;
    a.is_int = p->a_dtype == ACL_INT8;
    const uint32_t fw = a.is_int ? 1u : (p->b_dtype == ACL_FLOAT8_E5M2 ? 1u : 0u), fx = a.is_int ? 1u : (p->a_dtype == ACL_FLOAT8_E5M2 ? 1u : 0u);
    a.idesc = make_idesc(a.is_int ? 2u : 1u, fw, fx, a.w_mn, 0u, 128u, q.rows);
    a.out_dtype = p->out_dtype; a.bias_dtype = p->bias_dtype; a.scale_b_dtype = p->scale_b_dtype; a.deq_flags = p->deq_flags;
    a.trans_sa = p->trans_a; a.trans_sb = p->trans_b;
    a.group_m = p->group_m > 0 ? (uint32_t)p->group_m : 1u;
    a.scale_a = p->scale_a; a.scale_b = p->scale_b; a.scale_a_len = p->scale_a_len; a.scale_b_len = p->scale_b_len;
    a.sa_bs = p->sa_bs; a.sb_bs = p->sb_bs;
    a.bias = p->bias; a.bias_bs = p->bias_bs;
    a.out = p->out; a.out_ld = p->out_ld; a.out_bs = p->out_bs;
    if (q.split == 0) {
        uint8_t* ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p->workspace) + 255) & ~(uintptr_t)255);
        a.count = reinterpret_cast<unsigned long long*>(ws);
        a.part = reinterpret_cast<uint32_t*>(ws + (((uint64_t)q.tiles * 8u + 255u) & ~(uint64_t)255u));
    }
    a.nonce = next_ks_nonce();
    a.test_stop = 0xFFFFFFFFu;
    if (const char* e = env("OPSNN_TEST_SPLIT_STALL_KBLOCK")) {  // tests of the give-up path only
        a.test_stop = (uint32_t)atoi(e);
        const char* pl = env("OPSNN_TEST_UMMA_POLL_LIMIT");
        const uint32_t limit = pl != nullptr ? (uint32_t)atoi(pl) : 20000u;
        cudaMemcpyToSymbolAsync(ptx::g_spin_limit, &limit, sizeof(limit), 0, cudaMemcpyHostToDevice, stream);
    }
    CUtensorMap mw, mx;
    const uint64_t nbw = a.w_batched ? (uint64_t)p->batch : 1, nbx = a.x_batched ? (uint64_t)p->batch : 1;
    bool ok = a.w_mn ? make_map(&mw, p->b, (uint64_t)p->n, (uint64_t)p->k, nbw, (uint64_t)p->b_ld, (uint64_t)p->b_bs, 128)
                     : make_map(&mw, p->b, (uint64_t)p->k, (uint64_t)p->n, nbw, (uint64_t)p->b_ld, (uint64_t)p->b_bs, 128);
    ok = ok && make_map(&mx, p->a, (uint64_t)p->k, (uint64_t)p->m, nbx, (uint64_t)p->a_ld, (uint64_t)p->a_bs, q.rows);
    if (!ok) return (int32_t)cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(a.grid, 1, 1);
    cfg.blockDim = dim3(kSplitThreads, 1, 1);
    cfg.dynamicSmemBytes = (size_t)q.stages * q.stage_bytes + 1024 + (pb ? kSplitRing : 0u);
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
    note_launch(pb ? "qmm_umma_split_perblock" : "qmm_umma_split_deq");
    return rc;
}

}  // namespace
