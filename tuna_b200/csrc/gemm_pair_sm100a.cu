// FP16 x 4-bit(codebook) GEMM for large token counts (prefill) on the 5th-generation tensor cores
// of sm_100a, two SMs per tile.  Counterpart of the reference's Tuna<> kernel and its cp.async /
// ldmatrix / mma.sync main loop (kernel.cu:1043-2505, 2816-2960); the orientation is kept
// (weights are MMA operand A, tokens operand B, the accumulator is an o^T tile,
// kernel.cu:2182-2192) and nothing else.
//
// What bounds it.  The tensor pipe needs N/2 clocks for one 128 x N x 16 step; in the same time the
// step's operands have to pass the SM's 128 B/clk of shared memory.  With one SM per tile every SM
// stages and reads all N tokens: N/4 + N/4 wavefronts for the activations, 32 for the table lookups
// of its 2048 weights, 16 for their packed bytes, ~13 for the tensor-memory stores - 189 at N = 256
// against 128 clocks, which is where the one-SM version of this kernel stopped (0.69 of cuBLAS'
// bf16 rate).  A CTA pair (cta_group::2, M = 256) stages half of the tokens per SM: 125 at N = 256.  ncu at 57344x8192 and 256
// tokens in 256-token tiles counts 48 of them per step for lookups and weight bytes and 32 for the MMAs' operand reads, and sees the tensor
// pipe active for 87 % of the SMs' active clocks (the one-SM kernel: 49 % of the launch, this one 82 %); in 128-token tiles with 16 dequant warps,
// twice the lookups, 91 and 85 %.
//
// One persistent CTA pair per two SMs; each CTA dequantizes its own 128 rows into its own tensor
// memory, the leader (rank 0) issues the MMAs for both.  16 or 24 warps per CTA:
//   warp 0      leader: MMA issue (M = 256, N = the tile's tokens, K = 16, fp32 accumulate): A from
//               tensor memory, B through a shared-memory descriptor, D in tensor memory.
//               follower: tells the leader which of its activation stages have landed
//   warp 1      copy producer of the packed weights (TMA into a ring of KC-column stages)
//   warp 2      copy producer of the activations (TMA, this CTA's half of the tile's tokens)
//   warp 3      tensor-memory allocation
//   warps 4-7   epilogue: tensor memory -> registers -> scale by absmax -> fp16 -> stmatrix into a
//               staging tile -> TMA store; split-K partials and fix-up
//   warps 8 on   dequant (8 or 16, pair_split): packed bytes (shared memory) -> byte->half2 table lookups -> tcgen05.st.  A
//               thread owns one weight row (= one TMEM lane): a 32-bit word of the packed layout is
//               8 consecutive columns of one row (test.py:58-65), i.e. four TMEM columns in K order
// The dequantised fp16 weights never touch shared or global memory.  The scale is constant along K
// (one block per row, test.py:81, kernel.cu:2178-2180) and is applied once, in fp32, to the sum.
//
// KC, the columns of a stage: 64 for more than 128 tokens per tile, else 128, so that a stage is at
// least 512 clocks of MMAs per wait and commit (that fixed cost is ~230 clocks).
//
// Work decomposition.  A tile is 256 rows x N tokens.  Whole waves of tiles are handed out one tile
// per pair (all pairs walk K together, so the tiles that share weights or activations share them in
// L2; tiles are numbered so that a wave covers at most 8 token tiles).  What is left over - or, when there are
// fewer tiles than pairs, everything - is cut evenly along K ("stream-K"), first in the pair's
// order so that the exchange of partial sums overlaps the whole tiles.  A tile cut across pairs is finished
// by the CTA that arrives last at the tile's counter (per 32-row quarter): it adds the fp32 partials in K
// order, so the result does not depend on arrival order (the reference adds fp16 partials with
// atomicAdd, kernel.cu:2739-2745).  No floating-point atomics, no zero-filled output.
//
// Every wait is bounded: when one runs out the CTA records where in the device status word, raises its
// abort flag and unwinds to the common exit, where the pair meets and releases the tensor memory.
#include <cuda.h>
#include <algorithm>
#include <cstring>
#include <mutex>
#include "common.cuh"
#include "launchers.h"
#include "ring_plan.h"
#include "sm100_ptx.cuh"
#include "tcgen05.cuh"

namespace tuna {

constexpr int kPairRows = 2 * kBlockRows;   // rows of a tile
constexpr int kPairEpilogueWarp0 = 4;
constexpr int kPairDequantWarp0 = 8;
constexpr int kPairBars = 3 * kPairMaxStages + 2 * kPairMaxWStages + 4;
constexpr int kPairTokGroup = 8;            // token tiles of a wave's working set
// Up to here weights and codebook are taken from ahead of the dependency wait, as the weight-streaming kernels do (the
// header's contract); more tokens see ordinary stream order.  There the weights are read after the wait, and the lookup table
// is still built before it, from a copy of the codebook that is compared with the codebook after it.  Graph replay, us,
// all ahead / so / all after the wait: 512x512 at 100 tokens 3.4 / 3.9 / 5.5, 6144x4096 at 256 16.4 / 16.1 / 17.4, 28672x4096 at
// 1024 167 / 167 / 168; below the line 2048x2048 at 48 6.1 / 7.8, 28672x4096 at 64 25.4 / 25.7.
constexpr int kPairAheadTokens = 64;

static_assert((size_t)kBlockRows * 256 * 4 <= kMaxPartialSlotBytes, "partial sums of the widest tile");

struct PairParams {
    const float *code;
    const float *absmax;
    __half *o;
    float *partials;
    unsigned int *counters;
    DeviceStatus *status;
    int m, n, k;
    int tile_tok;     // N: tokens of a tile, a multiple of 32 up to 256 (the last token tile may use fewer)
    int chunks;       // ceil(k / KC)
    int row_tiles;    // ceil(m / 256)
    int tok_tiles;    // ceil(n / N)
    int stages;       // unit stages
    int w_stages;
    int nd;           // accumulator buffers
    int ahead;        // weights and codebook are taken from before the dependency wait
    int q3d;          // the weights' tensor map is the 3-D view (WMODE 0)
    int sk_tiles;     // tiles 0 .. sk_tiles - 1 are cut along K over pairs 0 .. sk_pairs - 1 ...
    int sk_pairs;
    int rot_step;     // see pair_first_chunk
    int sk_q, sk_r;   // ... in ranges of sk_q units, the first sk_r pairs one more
};

// The segments of a pair in order: its range of the tiles cut along K, then whole tiles.
struct PairSegs {
    int u, u_end, dp, dp_step, tiles;
    int tile, c0, c1;
    __device__ void init(const PairParams &p, int pair, int pairs)
    {
        u = pair * p.sk_q + min(pair, p.sk_r);
        u_end = u + (pair < p.sk_pairs ? p.sk_q + (pair < p.sk_r ? 1 : 0) : 0);
        dp = p.sk_tiles + pair;
        dp_step = pairs;
        tiles = p.row_tiles * p.tok_tiles;
    }
    __device__ bool more() const { return u < u_end || dp < tiles; }
    __device__ bool next(const PairParams &p)
    {
        if (u < u_end) {
            tile = u / p.chunks;
            c0 = u - tile * p.chunks;
            c1 = min(p.chunks, c0 + (u_end - u));
            u += c1 - c0;
            return true;
        }
        if (dp < tiles) {
            tile = dp;
            c0 = 0;
            c1 = p.chunks;
            dp += dp_step;
            return true;
        }
        return false;
    }
    __device__ int total_units(const PairParams &p) const
    {
        return (u_end - u) + (dp < tiles ? ((tiles - 1 - dp) / dp_step + 1) * p.chunks : 0);
    }
};

// Row tile and token tile of a tile number: groups of up to kPairTokGroup token tiles, row tiles inside a
// group, token tiles fastest.
__device__ __forceinline__ void pair_tile(const PairParams &p, int tile, int &rt, int &tt)
{
    const int per_group = p.row_tiles * kPairTokGroup;
    const int g = tile / per_group, r = tile - g * per_group;
    const int w = min(kPairTokGroup, p.tok_tiles - g * kPairTokGroup);
    rt = r / w;
    tt = g * kPairTokGroup + (r - rt * w);
}

// Where along K a whole tile starts: the chunks are taken cyclically from here.  Pairs that walk K in step would all read
// weights at one offset of rows 4k bytes apart (k = 8192: every 32 KB), which L2 serves at 2 TB/s; spread over K by
// row tile it is not what bounds the kernel (57344x8192, copies of weights alone: 114 us in step).  The pairs that share
// weights (same row tile) still read them together.
__device__ __forceinline__ int pair_first_chunk(const PairParams &p, const PairSegs &s, int rt)
{
    if (s.c0 != 0 || s.c1 != p.chunks) return s.c0;  // a range of a cut tile: as it lies
    return (int)((unsigned)rt * (unsigned)p.rot_step % (unsigned)p.chunks);
}

// Tokens the tile's MMAs cover: N, or what is left rounded up to the MMA's granule.
__device__ __forceinline__ int pair_tile_cols(const PairParams &p, int tt)
{
    return min(p.tile_tok, (p.n - tt * p.tile_tok + 31) & ~31);
}

// Table lookup: byte C of w (two 4-bit codes) -> half2 of the two code values, from this lane's copy of the table.
//   WIDE: the table lies kPairLutWide into the shared window with 256 bytes per entry (half of them unused), so that ONE prmt
//   builds the address (window | byte << 8 | lane * 4, `lane_key` = window | lane * 4) and the offset is the load's immediate;
//   otherwise 128 bytes per entry at `lane_key` - lane * 4, one multiply-add more per lookup.
template <bool WIDE, int C>
__device__ __forceinline__ uint32_t pair_lookup(uint32_t w, uint32_t lane_key)
{
    uint32_t a, v;
    // not volatile: the table is constant once built, so the compiler may schedule lookups freely
    if (WIDE) {
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(lane_key), "n"(0x7604 | (C << 4)));
        asm("ld.shared.u32 %0, [%1 + %2];" : "=r"(v) : "r"(a), "n"(kPairLutWide));
    } else {
        asm("prmt.b32 %0, %1, 0, %2;" : "=r"(a) : "r"(w), "n"(0x4440 | C));
        asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(lane_key + (a << 7)));
    }
    return v;
}

// KC: columns of a stage (64 or 128).  WMODE: layout of a weight stage, as in the weight-streaming kernel:
//   1  [32-row block][step pair][row group of the block][step of the pair][128 bytes]: one 5-D box per stage
//      that reads global memory in runs of 256 bytes (m % 32 == 0 and k % 64 == 0); TMEM lane l holds row l;
//   0  [step][row group][128 bytes]: one 3-D box per stage (k % 32 == 0) or one 2-D box per step; rows
//      assigned to lanes by lane_row_group().
// DW: dequant warps, 8 or 16 (pair_split).
template <int KC, int WMODE, int DW>
__global__ void __launch_bounds__(32 * (kPairDequantWarp0 + DW), 1)
gemm_w4a16_pair_kernel(const __grid_constant__ PairParams p, const __grid_constant__ CUtensorMap tmap_q,
                       const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_o)
{
    constexpr int STEPS = KC / 32;
    constexpr int kPairWarps = kPairDequantWarp0 + DW;
    constexpr int kPairGroups = DW / 4;  // a group of four warps (one per 32-lane quarter) converts every kPairGroups-th stage
    constexpr bool kWide = DW == 16;
    constexpr int kSlotCols = KC / 2;
    constexpr uint32_t kWBytes = kBlockRows * KC / 2;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kPairBars];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ float s_code[16];  // the codebook as it was before the dependency wait
    __shared__ int s_fix[4];   // quarters this CTA finishes with all its warps at the end

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int N = p.tile_tok, S = p.stages, SW = p.w_stages;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const uint32_t x_tile_bytes = (uint32_t)N * 64;             // N/2 tokens x 64 columns
    const uint32_t x_stage_bytes = x_tile_bytes * (KC / 64);
    const uint32_t window = smem_u32(smem) & 0xFFFF0000u;       // in a cluster a CTA's shared addresses carry its rank in their upper bits
    const uint32_t lut_addr = kWide ? window + kPairLutWide : smem_u32(smem);
    const uint32_t staging = lut_addr + (kWide ? kPairLutWideBytes : kPairLutBytes);          // [2 halves of 64 rows][N tokens][128 bytes], 128-byte swizzle
    const uint32_t xring = staging + (uint32_t)N * 256;
    const uint32_t wring = xring + (uint32_t)S * x_stage_bytes;

    const uint32_t u_full = smem_u32(&bars[0]), u_empty = u_full + 8 * kPairMaxStages, x_full = u_empty + 8 * kPairMaxStages;
    const uint32_t w_full = x_full + 8 * kPairMaxStages, w_empty = w_full + 8 * kPairMaxWStages;
    const uint32_t d_full = w_empty + 8 * kPairMaxWStages, d_empty = d_full + 16;
    volatile int *abort_flag = &s_abort;
    if (kWide && smem_u32(smem) > lut_addr) {  // the host checks it too; both CTAs leave, since they have the same layout
        if (threadIdx.x == 0 && atomicCAS(&p.status->code, 0, 109) == 0) p.status->detail = (int)smem_u32(smem);
        return;
    }

    if (warp == 1) {  // the barriers, 32 at a time
        auto count = [](int i) {
            if (i < kPairMaxStages) return 10;                            // u_full: two activation copies, four dequant warps of each CTA
            if (i < 3 * kPairMaxStages + kPairMaxWStages) return 1;       // u_empty, x_full (follower only), w_full
            if (i < 3 * kPairMaxStages + 2 * kPairMaxWStages) return 4;   // w_empty
            return i < kPairBars - 2 ? 1 : 8;                             // d_full, d_empty
        };
        for (int i = lane; i < kPairBars; i += 32) mbar_init(u_full + 8 * i, count(i));
        if (lane == 0) s_abort = 0;
        if (lane < 4) s_fix[lane] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
    }
    if (warp == 2 && elect_one_sync()) {
        prefetch_map(&tmap_x);
        prefetch_map(&tmap_o);
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(kPairTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    if (!p.ahead && threadIdx.x >= 64 && threadIdx.x < 80) s_code[threadIdx.x - 64] = p.code[threadIdx.x - 64];
    __syncthreads();  // this CTA's barriers are initialised: its weight producer may start

    // What a kernel before this one wrote is there only after this wait: its end alone, or its letting dependents start, is no
    // promise.  The copies of x and the epilogue always wait; up to kPairAheadTokens the weights are copied ahead of it, and
    // the dequant warps fill the A slots meanwhile.
    auto depend = [] { asm volatile("griddepcontrol.wait;" ::: "memory"); };

    PairSegs segs;
    segs.init(p, pair, pairs);
    const int total = segs.total_units(p);

    // The byte -> half2 table (even column = high nibble in the low half), its entries shared out over `step` warps.
    auto build_table = [&](float cv, int first, int step) {
        const uint32_t ch = (uint32_t)__half_as_ushort(__float2half_rn(cv));
        for (int e = first; e < 256; e += step) {
            const uint32_t v = __shfl_sync(0xffffffffu, ch, e >> 4) | (__shfl_sync(0xffffffffu, ch, e & 15) << 16);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(lut_addr + (uint32_t)e * (kWide ? 256 : 128) + lane * 4), "r"(v) : "memory");
        }
    };
    // Rest of the prologue, run by every warp inside its own role's branch: the table, then the barrier of the
    // pair, which publishes both CTAs' barriers and tables.
    // depend() comes after it in every role that needs it, and in whoever is about to make a bounded wait that
    // ends only after the kernels before this one.
    auto table_share = [&] { build_table(p.ahead ? p.code[lane & 15] : s_code[lane & 15], warp, kPairWarps); };
    auto finish_prologue = [&]() -> uint32_t {
        table_share();
        tc_fence_before();
        cluster_sync_all();
        tc_fence_after();
        return s_tmem_base;
    };
    uint32_t tmem = 0;
    const uint32_t d_cols = (uint32_t)N;
    const uint32_t a_off = (uint32_t)p.nd * d_cols;  // first A slot
    const uint32_t leader_u_full = map_to_rank(u_full, 0), leader_d_empty = map_to_rank(d_empty, 0);

    // The first CTA pair of a cut tile's segments, and their number.
    auto tile_segments = [&](int tile, int &first) {
        auto pair_of = [&](int unit) {
            const int big = p.sk_r * (p.sk_q + 1);
            return unit < big ? unit / (p.sk_q + 1) : p.sk_r + (unit - big) / p.sk_q;
        };
        first = pair_of(tile * p.chunks);
        return pair_of((tile + 1) * p.chunks - 1) - first + 1;
    };
    // Adds the partials of COLS columns from `col` on of TMEM lane 32*quarter + lane over all segments of a tile, in K
    // order, and stores the row.  The loads of SG segments are in flight at a time, the adds keep the order; their addresses are 32-bit offsets into the
    // partial sums (partial_region_bytes, far below 4 GB), which is less code for a part that runs once.
    auto fix_piece = [&](auto cols_, auto sg, int tile, int first, int nseg, int quarter, int col) {
        constexpr int COLS = decltype(cols_)::value, SG = decltype(sg)::value;
        int rt, tt;
        pair_tile(p, tile, rt, tt);
        const int row_in_block = WMODE == 1 ? 32 * quarter + lane : 8 * lane_row_group(quarter, lane) + (lane & 7);
        const int row = rt * kPairRows + rank * kBlockRows + row_in_block;
        const uint32_t slot_bytes = (uint32_t)N * (kBlockRows * 4u);
        const uint32_t at = (uint32_t)(2 * (2 * first + rank)) * slot_bytes + (uint32_t)(col / 4 * kBlockRows + 32 * quarter + lane) * 16u;
        auto seg_ptr = [&](int s) {
            return reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(p.partials) + (at + (uint32_t)(4 * s + (s == 0 ? 1 : 0)) * slot_bytes));
        };
        float acc[COLS];
#pragma unroll
        for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
        for (int s = 0; s < nseg; s += SG) {
            float4 v[SG][COLS / 4];
#pragma unroll
            for (int j = 0; j < SG; ++j)
                if (s + j < nseg) {
                    const float4 *src = seg_ptr(s + j);
#pragma unroll
                    for (int i = 0; i < COLS / 4; ++i) v[j][i] = __ldcg(src + i * kBlockRows);
                }
#pragma unroll
            for (int j = 0; j < SG; ++j)
                if (s + j < nseg) {
#pragma unroll
                    for (int i = 0; i < COLS / 4; ++i) { acc[4 * i] += v[j][i].x; acc[4 * i + 1] += v[j][i].y; acc[4 * i + 2] += v[j][i].z; acc[4 * i + 3] += v[j][i].w; }
                }
        }
        if (row < p.m) {
            const float sc = p.absmax[row];
#pragma unroll
            for (int i = 0; i < COLS; ++i) {
                const int tok = tt * N + col + i;
                if (tok < p.n) p.o[(size_t)tok * p.m + row] = __float2half_rn(acc[i] * sc);
            }
        }
    };

    if (warp == 0) {
        tmem = finish_prologue();
        depend();
        if (rank == 0) {
            // -------------------------------------------------------------- MMA issue
            // The warp stays converged: every lane runs the loop and the waits, one elected lane issues.
            constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8-token groups 1024 bytes apart, version 1, 128-byte swizzle
            Ring ru, rd;
            bool ok = true;
            while (ok && segs.next(p)) {
                int rt, tt;
                pair_tile(p, segs.tile, rt, tt);
                const uint32_t idesc = (1u << 4) | ((uint32_t)(pair_tile_cols(p, tt) >> 3) << 17) | ((uint32_t)(kPairRows >> 4) << 24);
                ok = mbar_wait_warp(d_empty + 8 * rd.idx, rd.phase ^ 1, abort_flag, p.status, 103);
                const uint32_t dbase = tmem + (uint32_t)rd.idx * d_cols;
                for (int c = segs.c0; ok && c < segs.c1; ++c) {
                    ok = mbar_wait_warp(u_full + 8 * ru.idx, ru.phase, abort_flag, p.status, 104);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one_sync()) {
                        const uint32_t abase = tmem + a_off + (uint32_t)ru.idx * kSlotCols;
                        const uint32_t desc_lo = ((xring + (uint32_t)ru.idx * x_stage_bytes) & 0x3FFFFu) >> 4;
#pragma unroll
                        for (int kk = 0; kk < KC / 16; ++kk) {
                            const uint64_t bdesc = ((uint64_t)desc_hi << 32) | (uint64_t)(desc_lo + (kk >> 2) * (x_tile_bytes >> 4) + (kk & 3) * 2);
                            tc_mma_ts_pair(dbase, abase + kk * 8, bdesc, idesc, (c == segs.c0 && kk == 0) ? 0u : 1u);
                        }
                        tc_commit_pair(u_empty + 8 * ru.idx);
                        if (c + 1 == segs.c1) tc_commit_pair(d_full + 8 * rd.idx);
                    }
                    __syncwarp();
                    ru.advance(S);
                }
                rd.advance(p.nd);
            }
        } else {
            // -------------------------------------------------------------- follower: activation stages that have landed
            Ring ru;
            for (int u = 0; u < total; ++u, ru.advance(S)) {
                if (!mbar_wait_warp(x_full + 8 * ru.idx, ru.phase, abort_flag, p.status, 102)) break;
                if (lane == 0) mbar_arrive_cluster(leader_u_full + 8 * ru.idx);
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ weight producer
        // One elected lane of the converged warp issues the copies, the first ones before the rest of the prologue.
        Ring rw;
        int u = 0;
        bool ok = segs.next(p);
        int rt = 0, c = 0, left = 0;  // row tile, chunk, chunks of the segment still to load
        auto enter = [&]() {
            int tt;
            pair_tile(p, segs.tile, rt, tt);
            c = pair_first_chunk(p, segs, rt);
            left = segs.c1 - segs.c0;
        };
        if (ok) enter();
        auto issue_until = [&](int end) {
            for (; ok && u < end; ++u, rw.advance(SW)) {
                ok = mbar_wait_warp(w_empty + 8 * rw.idx, rw.phase ^ 1, abort_flag, p.status, 100);
                if (!ok) break;
                if (elect_one_sync()) {
                    const int block = 2 * rt + rank;  // 128-row block
                    const uint32_t dst = wring + (uint32_t)rw.idx * kWBytes, bar = w_full + 8 * rw.idx;
                    mbar_expect_tx(bar, kWBytes);
                    if (WMODE == 1) {
                        tma_load_5d(dst, &tmap_q, 0, 0, 0, c * (STEPS / 2), block * 4, bar);
                    } else if (p.q3d) {
                        tma_load_3d(dst, &tmap_q, 0, block * 16, c * STEPS, bar);
                    } else {
#pragma unroll
                        for (int st = 0; st < STEPS; ++st) tma_load_2d(dst + st * 2048u, &tmap_q, c * KC + 32 * st, block * 16, bar);
                    }
                }
                __syncwarp();
                if (++c == p.chunks) c = 0;
                if (--left == 0 && u + 1 < total) {
                    segs.next(p);
                    enter();
                }
            }
        };
        // The copies of a ring-full take longer than the rest of the prologue: the other warps do not wait for them.
        table_share();
        cluster_arrive();
        if (p.ahead) issue_until(min(SW, total));
        cluster_wait();
        if (p.ahead) issue_until(min(SW + S, total));  // the stages the dequant warps empty before the first MMA
        depend();
        issue_until(total);
    } else if (warp == 2) {
        // ------------------------------------------------------------------ activation producer
        tmem = finish_prologue();
        depend();
        Ring ru;
        const uint32_t full = rank == 0 ? u_full : x_full;
        bool ok = true;
        while (ok && segs.next(p)) {
            int rt, tt;
            pair_tile(p, segs.tile, rt, tt);
            const int tok = tt * N + rank * (pair_tile_cols(p, tt) >> 1);
            int c = pair_first_chunk(p, segs, rt);
            for (int i = segs.c0; i < segs.c1; ++i, ru.advance(S)) {
                ok = mbar_wait_warp(u_empty + 8 * ru.idx, ru.phase ^ 1, abort_flag, p.status, 101);
                if (!ok) break;
                if (elect_one_sync()) {
                    mbar_expect_tx(full + 8 * ru.idx, x_stage_bytes);
#pragma unroll
                    for (int t = 0; t < KC / 64; ++t)
                        tma_load_2d(xring + (uint32_t)ru.idx * x_stage_bytes + (uint32_t)t * x_tile_bytes, &tmap_x, c * KC + 64 * t, tok, full + 8 * ru.idx);
                }
                __syncwarp();
                if (++c == p.chunks) c = 0;
            }
        }
        // The MMAs' commits arrive at both CTAs' barriers: neither leaves before the last ones have, one per stage in use.
        for (int i = min(S, total); ok && i > 0; --i, ru.advance(S)) {
            if (total < S && i == total) ru = Ring();
            ok = mbar_wait_warp(u_empty + 8 * ru.idx, total < S ? 0u : ru.phase ^ 1, abort_flag, p.status, 110);
        }
    } else if (warp == 3) {
        tmem = finish_prologue();
    } else if (warp < kPairDequantWarp0) {
        // ------------------------------------------------------------------ epilogue
        tmem = finish_prologue();
        depend();
        const int quarter = warp & 3;
        const uint32_t tmem_q = tmem + ((uint32_t)(32 * quarter) << 16);
        Ring rd;
        while (segs.next(p)) {
            int rt, tt;
            pair_tile(p, segs.tile, rt, tt);
            const int cols = pair_tile_cols(p, tt);
            const bool full = segs.c0 == 0 && segs.c1 == p.chunks;
            const int row0 = rt * kPairRows + rank * kBlockRows;
            if (full) {
                // Fragments of 8 rows x 8 tokens, packed to fp16, are written transposed (stmatrix): 16 bytes =
                // 8 rows of one token.  8-row chunk j of this warp's 32 lanes is rows 8 * chunk(j) .. + 7.
                float sc[4];
                int chunk[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    chunk[j] = WMODE == 1 ? 4 * quarter + j : lane_row_group(quarter, 8 * j);
                    const int row = row0 + 8 * chunk[j] + (lane >> 2);
                    sc[j] = row < p.m ? p.absmax[row] : 0.f;
                }
                const int my_chunk = WMODE == 1 ? 4 * quarter + (lane >> 3) : lane_row_group(quarter, lane);
                const uint32_t st_base = staging + (uint32_t)(my_chunk >> 3) * (uint32_t)N * 128u;
                if (threadIdx.x == 32 * kPairEpilogueWarp0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                __syncwarp();
                // the previous tile has left the staging buffer; the four warps stop together or not at all, since they meet here
                if (bar_any(1, 128, *abort_flag != 0)) break;
                const bool ok = mbar_wait_warp(d_full + 8 * rd.idx, rd.phase, abort_flag, p.status, 106);
                tc_fence_after();
                for (int t0 = 0; ok && t0 < cols; t0 += 32) {
                    uint32_t lo[16], hi[16];
                    tc_ld_16x256b_x4(tmem_q + (uint32_t)rd.idx * d_cols + t0, lo);
                    tc_ld_16x256b_x4(tmem_q + (16u << 16) + (uint32_t)rd.idx * d_cols + t0, hi);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t r0 = pack_half2(__uint_as_float(lo[4 * i]) * sc[0], __uint_as_float(lo[4 * i + 1]) * sc[0]);
                        const uint32_t r1 = pack_half2(__uint_as_float(lo[4 * i + 2]) * sc[1], __uint_as_float(lo[4 * i + 3]) * sc[1]);
                        const uint32_t r2 = pack_half2(__uint_as_float(hi[4 * i]) * sc[2], __uint_as_float(hi[4 * i + 1]) * sc[2]);
                        const uint32_t r3 = pack_half2(__uint_as_float(hi[4 * i + 2]) * sc[3], __uint_as_float(hi[4 * i + 3]) * sc[3]);
                        const uint32_t tok = (uint32_t)(t0 + 8 * i + (lane & 7));
                        stmatrix_x4_trans(st_base + tok * 128u + ((((uint32_t)my_chunk & 7u) ^ (tok & 7u)) << 4), r0, r1, r2, r3);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_d_empty + 8 * rd.idx);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (ok && threadIdx.x == 32 * kPairEpilogueWarp0) {
                    // rows past m and tokens past n are clipped by the copy
                    for (int h = 0; h < 2; ++h)
                        if (row0 + 64 * h < p.m) tma_store_2d(&tmap_o, row0 + 64 * h, tt * N, staging + (uint32_t)h * (uint32_t)N * 128u);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            } else {
                if (!mbar_wait_warp(d_full + 8 * rd.idx, rd.phase, abort_flag, p.status, 106)) continue;  // the flag is up: see above
                tc_fence_after();
                // [4-token group][128 lanes] float4: a warp store is 512 contiguous bytes
                float4 *dst = reinterpret_cast<float4 *>(p.partials + (size_t)(2 * blockIdx.x + (segs.c0 == 0 ? 1 : 0)) * ((size_t)kBlockRows * N)) + 32 * quarter + lane;
                for (int t0 = 0; t0 < cols; t0 += 16) {
                    float v[16];
                    tc_ld_x16(tmem_q + (uint32_t)rd.idx * d_cols + t0, v);
#pragma unroll
                    for (int i = 0; i < 4; ++i) dst[(size_t)(t0 / 4 + i) * kBlockRows] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(leader_d_empty + 8 * rd.idx);
                int first;
                const int nseg = tile_segments(segs.tile, first);
                unsigned int *counter = p.counters + (size_t)(2 * segs.tile + rank) * 4 + quarter;
                unsigned int old = 0;
                // releases the warp's partials (the __syncwarp above orders them before it) and acquires the others'
                if (lane == 0) asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
                old = __shfl_sync(0xffffffffu, old, 0);
                if (old == (unsigned)nseg - 1) {
                    if (lane == 0) *counter = 0;  // leave the counter clean for the next call
                    // the pair's last segment: all warps of the CTA finish it together, below
                    if (segs.more()) {
                        for (int col = 0; col < cols; col += 16) fix_piece(Int<16>(), Int<DW == 8 ? 4 : 2>(), segs.tile, first, nseg, quarter, col);
                    } else if (lane == 0) {
                        s_fix[quarter] = 1;
                    }
                }
            }
            rd.advance(p.nd);
        }
        if (threadIdx.x == 32 * kPairEpilogueWarp0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        // ------------------------------------------------------------------ dequant
        tmem = finish_prologue();
        if (!p.ahead) {
            depend();
            const float cv = __ldcg(p.code + (lane & 15));
            // the kernel before has written another codebook: all the dequant warps see it, and nobody has looked anything up yet
            if (__any_sync(0xffffffffu, __float_as_uint(cv) != __float_as_uint(s_code[lane & 15]))) {
                asm volatile("bar.sync 2, %0;" ::"n"(32 * DW) : "memory");
                build_table(cv, warp - kPairDequantWarp0, DW);
                asm volatile("bar.sync 2, %0;" ::"n"(32 * DW) : "memory");
            }
        }
        const int quarter = warp & 3, group = (warp - kPairDequantWarp0) >> 2;
        const uint32_t lane_key = (kWide ? window : lut_addr) + (uint32_t)lane * 4u;
        const uint32_t a_lane = tmem + ((uint32_t)(32 * quarter) << 16) + a_off;
        // This thread's row inside a weight stage (see the weight-streaming kernel): word r%4 of 16-byte chunk
        // 2 kt + r/4 of the 128-byte row of (row group, step), XORed with that row's index mod 8.
        const int r = lane & 7;
        const int rg = WMODE == 1 ? (lane >> 3) : lane_row_group(quarter, lane);
        const uint32_t row0 = WMODE == 1 ? (uint32_t)(quarter * (STEPS / 2) * 8 + 2 * rg) : (uint32_t)rg;
        const uint32_t xor0 = WMODE == 1 ? (uint32_t)(2 * rg) : (uint32_t)(rg & 7);
        uint32_t soff[4];
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) soff[kt] = row0 * 128u + (((uint32_t)(2 * kt + (r >> 2)) ^ xor0) << 4) + (uint32_t)(r & 3) * 4u;
        auto w_addr = [&](uint32_t stage, int st, int kt) -> uint32_t {
            if (WMODE == 1) return stage + (soff[kt] ^ ((st & 1) ? 16u : 0u)) + (uint32_t)((st >> 1) * 1024 + (st & 1) * 128);
            return stage + soff[kt] + (uint32_t)st * 2048u;
        };
        auto skip = [](Ring &ring, int by, int depth) {
            ring.idx += by;
            while (ring.idx >= depth) { ring.idx -= depth; ring.phase ^= 1u; }
        };
        Ring rw, ru;  // the groups share both rings: rings_shareable() says when they may
        skip(rw, group, SW);
        skip(ru, group, S);
        for (int u = group; u < total; u += kPairGroups) {
            if (!mbar_wait_warp(w_full + 8 * rw.idx, rw.phase, abort_flag, p.status, 107)) break;
            const uint32_t stage = wring + (uint32_t)rw.idx * kWBytes;
            uint32_t w[STEPS][4];
#pragma unroll
            for (int st = 0; st < STEPS; ++st)
#pragma unroll
                for (int kt = 0; kt < 4; ++kt) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[st][kt]) : "r"(w_addr(stage, st, kt)));
            uint32_t v[32];
            auto lookups = [&](int st0) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t word = w[st0 + (i >> 2)][i & 3];
                    v[4 * i] = pair_lookup<kWide, 0>(word, lane_key);
                    v[4 * i + 1] = pair_lookup<kWide, 1>(word, lane_key);
                    v[4 * i + 2] = pair_lookup<kWide, 2>(word, lane_key);
                    v[4 * i + 3] = pair_lookup<kWide, 3>(word, lane_key);
                }
            };
            lookups(0);
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty + 8 * rw.idx);  // all of the stage's loads have returned (they return in order)
            if (u >= S && u < S + kPairGroups) depend();  // the first stages whose A slot has to be emptied first
            if (!mbar_wait_warp(u_empty + 8 * ru.idx, ru.phase ^ 1, abort_flag, p.status, 108)) break;
            tc_fence_after();
            const uint32_t slot = a_lane + (uint32_t)ru.idx * kSlotCols;
            tc_st_x32(slot, v);
#pragma unroll
            for (int st0 = 2; st0 < STEPS; st0 += 2) {
                lookups(st0);
                tc_st_x32(slot + 16 * st0, v);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(leader_u_full + 8 * ru.idx);
            skip(rw, kPairGroups, SW);
            skip(ru, kPairGroups, S);
        }
    }

    // ------------------------------------------------------------------ common exit
    __syncwarp();
    __syncthreads();
    {
        // the tile whose last partials this CTA wrote in its last segment: (piece, quarter) over all warps
        int tile = -1, cols = 0, first = 0, nseg = 0;
        PairSegs s;
        s.init(p, pair, pairs);
        if (s_fix[0] | s_fix[1] | s_fix[2] | s_fix[3]) {
            while (s.next(p)) tile = s.tile;
            int rt, tt;
            pair_tile(p, tile, rt, tt);
            cols = pair_tile_cols(p, tt);
            nseg = tile_segments(tile, first);
        }
        // 24 warps have registers for half as many loads in flight as 16: twice the segments where there is a warp for every eight columns
        // (16 columns of two segments / 8 of four, us: 800x6464 at 52 tokens 10.7 / 10.3, 512x27392 at 60 13.1 / 12.1; where that takes a second
        // round of pieces, 64-token tiles, 768x22400 at 97 16.1 / 16.9)
        if (DW == 16 && cols / 8 * 4 <= kPairWarps) {
            if ((warp >> 2) * 8 < cols && s_fix[warp & 3]) fix_piece(Int<8>(), Int<4>(), tile, first, nseg, warp & 3, (warp >> 2) * 8);
        } else {
            for (int item = warp; (item >> 2) * 16 < cols; item += kPairWarps)
                if (s_fix[item & 3]) fix_piece(Int<16>(), Int<DW == 16 ? 2 : 4>(), tile, first, nseg, item & 3, (item >> 2) * 16);
        }
    }
    tc_fence_before();
    __syncwarp();
    cluster_sync_all();
    if (warp == 3) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPairTmemCols) : "memory");
    }
}

// ------------------------------------------------------------------ host side

// The estimates below are fitted to 16000 launches: in short runs (graph replay) 350 shapes of 512 to 55000 rows, 512 to 28000 columns and
// 25 to 3900 tokens in every token tile, with 8 and 16 dequant warps, uncut and cut in every way that pair_split considers; and 170 shapes of
// 3e10 operations or more under the power cap.  What they choose takes 0.7 % (short runs) and 1.9 % (power cap) longer than the fastest launch of its shape
// in the mean, 16 % at worst; with 16 warps wherever they fit and cuts priced by their number of segments alone it was 4 and 3.7 %, and 38 % at worst.  Fitted
// to the short runs alone it was 0.7 and 3 %, and on 40 other shapes whose activations are a good part of L2 or more 1.4 % slower than so.  Those are
// the least predictable: 6 % longer than the fastest launch in the mean, 31 % at worst (tiles out of step no longer share what L2 holds).

// Microseconds per 16 columns of K of a tile of `tok` tokens: the clocks of the lookups and what goes with them plus the activations',
// at the 1.7 GHz of a short run, or the tensor pipe's N/2 clocks and what the dequantisation adds to them, at a clock between that and the one
// that the power cap leaves (128 / 192 / 256 tokens: 0.052 / 0.075 / 0.101 in short runs, 0.059 / 0.088 / 0.117 under the cap).
static double pair_step_us(int tok, int warps)
{
    return std::max((warps == 16 ? 50 + 0.25 * tok : 73 + 0.26 * tok) / 1700.0, (tok / 2 + 14) / 1540.0);
}

// How the tiles of a launch are handed out (see the head of the file): sk_tiles of them are cut along K over
// sk_pairs pairs, the others go out in whole waves.
struct PairSplit {
    int sk_tiles, sk_pairs;
    int warps;  // dequant warps
    double us;  // the estimate
};

// What an uncut launch takes beside its steps.  16 dequant warps convert four stages at once and the MMAs of all four are still to come: on
// short tiles that takes longer than what the warps save (us, 8 / 16: 3192x1048 at 613 tokens, 128-token tiles, 9.1 / 9.6; 12496x512 at 738 12.9 / 13.5;
// 2048x4096 at 1140 16.5 / 16.4; 6144x4096 at 256, 96-token tiles, 15.8 / 14.5).  Where the weights come after the dependency wait, narrow tiles
// have most of the dequantisation still before them then and want the warps (1792x896 at 78 tokens, 32-token tiles, 5.2 / 4.8; 2944x768 at 100,
// 64-token tiles, 5.1 / 4.9; ahead of it 3072x768 at 60 3.9 / 4.0).
static double pair_uncut_us(int cols, int warps, bool ahead)
{
    return 2.6 + 0.007 * cols + (warps == 16 ? 0.95 : (ahead ? 0.0 : std::max(0.0, 0.7 - 0.006 * cols)));
}
// What cutting costs: partial sums written, an arrival, and adding them up.
static double pair_cut_us(int cols, int warps) { return 5.2 + 0.029 * cols + 0.008 * std::max(0, cols - 128) + (warps == 16 ? 0.65 : 0.0); }
// Adding up `segs` segments of a tile at the end of a CTA: a round is as many loads as its warps have in flight.
static double pair_add_us(int cols, int warps, int segs)
{
    const int rounds = warps == 8 ? div_up(segs, 4) * div_up(cols / 4, 16) : (cols == 32 ? div_up(segs, 4) : div_up(segs, 2) * div_up(cols / 4, 24));
    return 0.9 * rounds;
}
// Ranges that do not end where a tile does: their CTAs work on two tiles, and a tile has one segment more (528x4480 at 44 tokens, 35 chunks a
// tile: four segments 10.2 us, five 8.4).
static double pair_ragged_us(int cols) { return 2.0 + 0.01 * cols; }
// Cut tiles in front of whole ones.
constexpr double kPairMixedUs = 1.7;
// A launch that leaves half of the pairs idle: the next one starts on those (6272x1792 at 42 tokens: one tile of 64 per 256 rows 6.5 us, two
// of 32 8.0).
constexpr double kPairOverlapUs = 1.2;

static PairSplit pair_split(int m, int n, int k, int tile_tok, int pairs)
{
    const int row_tiles = div_up(m, kPairRows), full = n / tile_tok, last = n - full * tile_tok, last_cols = (last + 31) / 32 * 32;
    const int tok_tiles = full + (last ? 1 : 0), chunks = div_up(k, pair_kc(tile_tok)), cols = full ? tile_tok : last_cols;
    const long long tiles = (long long)row_tiles * tok_tiles;
    const long long waves = tiles / pairs;
    const int rest = (int)(tiles - waves * pairs);
    const double steps = k / 16.0;
    auto overlap = [&](long long busy) { return 2 * busy <= pairs ? kPairOverlapUs : 0.0; };
    PairSplit best = {0, 0, 0, 0.0};
    for (int warps = pair_dequant_warps(tile_tok); warps >= 8; warps -= 8) {
        const double last_us = last ? steps * pair_step_us(last_cols, warps) : 0.0;
        const double tile_us = full ? steps * pair_step_us(tile_tok, warps) : last_us;  // of the widest tile
        const double work_us = row_tiles * (full * tile_us + last_us) / pairs;          // per pair, evenly cut
        auto consider = [&](int sk_tiles, int sk_pairs, double us) {
            if (best.warps == 0 || us < best.us) best = {sk_tiles, sk_pairs, warps, us};
        };
        const double uncut_us = pair_uncut_us(cols, warps, n <= kPairAheadTokens), cut_us = pair_cut_us(cols, warps);
        // a wave of tiles of two widths takes as long as something between their mean and the wider one
        const double wave_us = (tile_us + 2 * work_us * pairs / tiles) / 3;
        consider(0, 0, waves == 0 ? uncut_us + tile_us - overlap(tiles) : uncut_us + (waves + (rest ? 1 : 0)) * wave_us);
        // where there is more than one wave of whole tiles, adding up hides behind them
        if (rest > 0 && waves > 0)
            consider(pairs + rest, pairs, work_us + cut_us + kPairMixedUs + (waves > 1 ? 0.0 : pair_add_us(cols, warps, 2)));
        if (waves == 0) {
            int s = 2;
            for (; s * tiles <= pairs && s <= chunks; ++s) {
                const bool ragged = chunks % s != 0;
                consider((int)tiles, s * (int)tiles,
                         tile_us * div_up(chunks, s) / chunks + cut_us + pair_add_us(cols, warps, s + ragged) + (ragged ? pair_ragged_us(cols) : 0.0) - overlap(s * tiles));
            }
            // all pairs, where whole segments leave more than a tenth of them idle
            if (s <= chunks && (s - 1) * tiles * 10 < pairs * 9)
                consider((int)tiles, pairs, work_us + cut_us + pair_add_us(cols, warps, pairs / (int)tiles + 1) + pair_ragged_us(cols));
        }
    }
    return best;
}

// Tokens per tile: the multiple of 32 with the lowest estimate; the smaller one where two are equal.
static int pair_pick_tile_tok(int m, int n, int k, int pairs)
{
    int best = 32;
    double best_us = -1;
    for (int t = 32; t <= 256; t += 32) {
        const double us = pair_split(m, n, k, t, pairs).us;
        if (best_us < 0 || us < best_us) { best = t; best_us = us; }
        if (t >= n) break;
    }
    return best;
}

static int pair_count(const tuna_config &c) { return c.ctas / 2 > 0 ? c.ctas / 2 : 1; }

// of a normalized configuration
static int pair_tile_tok(const tuna_config &c) { return c.tile_tok < 32 ? 32 : c.tile_tok; }

// The fields of an explicit configuration describe a tile of one SM - `row_blocks` x 128 rows x `tile_tok` tokens in stages
// of 64 columns - and what does not fit one SM's tensor or shared memory is refused, although this kernel takes no
// more than the token tile from them.
static bool umma_fields_fit(int n, const tuna_config &c)
{
    constexpr int kSlot = 32, kLut = 32 * 1024, kBlock = 4096, kSmem = 225 * 1024;  // A-slot columns; bytes
    const int t = c.tile_tok ? c.tile_tok : (n <= 16 ? 16 : n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : 256);
    const int rb = c.row_blocks ? c.row_blocks : (t <= 32 ? 4 : (t <= 64 ? 2 : 1));
    if (rb * t + 2 * rb * kSlot > kPairTmemCols) return false;
    const int bufs = 2 * rb * t + 2 * rb * kSlot <= kPairTmemCols ? 2 : 1;
    const int sw = c.stages_w ? c.stages_w : (rb == 4 ? 4 : (rb == 2 ? 6 : 8));
    const int sx = c.stages_x ? c.stages_x : 2;  // left free, as few as it takes
    return sx <= (kPairTmemCols - bufs * rb * t) / (rb * kSlot) && kLut + sw * rb * kBlock + sx * t * 128 <= kSmem;
}

int gemm_umma_normalize_config(int m, int n, int k, int sm_count, tuna_config *c)
{
    const int t = c->tile_tok;
    if (t < 0 || t > 256 || (t != 16 && t % 32 != 0)) return TUNA_ERR_BAD_CONFIG;
    if (c->row_blocks != 0 && c->row_blocks != 1 && c->row_blocks != 2 && c->row_blocks != 4) return TUNA_ERR_BAD_CONFIG;
    if (c->dequant_warps != 0 && c->dequant_warps != 8 && c->dequant_warps != 16) return TUNA_ERR_BAD_CONFIG;
    if (c->k_accs != 0 && c->k_accs != 1) return TUNA_ERR_BAD_CONFIG;
    if (c->stages_x != 0 && (c->stages_x < 2 || c->stages_x > 16)) return TUNA_ERR_BAD_CONFIG;
    if (c->stages_w != 0 && (c->stages_w < 4 || c->stages_w > 16)) return TUNA_ERR_BAD_CONFIG;
    if (!umma_fields_fit(n, *c)) return TUNA_ERR_BAD_CONFIG;
    if (c->ctas < 0) return TUNA_ERR_BAD_CONFIG;
    if (c->ctas == 0 || c->ctas > sm_count) c->ctas = sm_count;
    // what the launch takes, for whoever looks it up (stages follow from the token tile and stay 0)
    if (t == 0) c->tile_tok = pair_pick_tile_tok(m, n, k, pair_count(*c));
    if (c->row_blocks == 0) c->row_blocks = 1;
    if (c->dequant_warps == 0) c->dequant_warps = pair_split(m, n, k, pair_tile_tok(*c), pair_count(*c)).warps;
    if (c->k_accs == 0) c->k_accs = 1;
    return TUNA_OK;
}

size_t gemm_umma_workspace_bytes(int m, int n, int k, const tuna_config &c, int sm_count)
{
    (void)k;
    const long long tiles = (long long)div_up(m, kPairRows) * div_up(n, pair_tile_tok(c));
    const long long cut = tiles < sm_count ? tiles : sm_count;  // fewer than two waves of tiles are cut along K
    return partial_region_bytes(sm_count) + ((size_t)cut * 32 + 255) / 256 * 256;  // one counter per tile, CTA and TMEM lane quarter
}

template <int KC, int WMODE, int DW>
static int launch_pair(const PairParams &p, const CUtensorMap &mq, const CUtensorMap &mx, const CUtensorMap &mo, int ctas, cudaStream_t stream)
{
    static bool attr_set[64] = {false};  // one-time, per device, opt-in to large dynamic shared memory
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TUNA_ERR_NO_DEVICE;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!attr_set[dev]) {
            if (cudaFuncSetAttribute(gemm_w4a16_pair_kernel<KC, WMODE, DW>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemDynamic) != cudaSuccess)
                return TUNA_ERR_NO_DEVICE;
            // pair_plan counts on 1 KB of the system's and up to 1 KB of static shared memory before the dynamic part
            cudaFuncAttributes fa;
            int reserved = 0;
            if (cudaFuncGetAttributes(&fa, gemm_w4a16_pair_kernel<KC, WMODE, DW>) != cudaSuccess ||
                cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess ||
                fa.sharedSizeBytes + (size_t)reserved > kPairSmemStart)
                return TUNA_ERR_NO_DEVICE;
            attr_set[dev] = true;
        }
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)ctas);
    lc.blockDim = dim3(32 * (kPairDequantWarp0 + DW));
    lc.dynamicSmemBytes = kPairSmemDynamic;
    lc.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 2;
    return cudaLaunchKernelEx(&lc, gemm_w4a16_pair_kernel<KC, WMODE, DW>, p, mq, mx, mo) == cudaSuccess ? TUNA_OK : TUNA_ERR_LAUNCH;
}

int launch_gemm_umma(const GemmArgs &a, const tuna_config &c)
{
    int pairs = pair_count(c);
    const PairSplit split = pair_split(a.m, a.n, a.k, pair_tile_tok(c), pairs);
    const PairPlan l = pair_plan(pair_tile_tok(c), pair_kc(pair_tile_tok(c)), split.warps);
    PairParams p;
    std::memset(&p, 0, sizeof(p));
    p.code = a.code; p.absmax = a.absmax; p.o = (__half *)a.o;
    p.m = a.m; p.n = a.n; p.k = a.k;
    p.tile_tok = l.tile_tok;
    p.chunks = div_up(a.k, l.kc);
    p.row_tiles = div_up(a.m, kPairRows);
    p.tok_tiles = div_up(a.n, l.tile_tok);
    p.rot_step = p.chunks * 5 / 8 | 1;
    p.stages = l.stages; p.w_stages = l.w_stages; p.nd = l.nd;
    p.ahead = a.n <= kPairAheadTokens;
    if (a.workspace == nullptr || a.workspace_bytes < gemm_umma_workspace_bytes(a.m, a.n, a.k, c, a.sm_count)) return TUNA_ERR_WORKSPACE;
    p.partials = (float *)a.workspace;
    p.counters = (unsigned int *)((uint8_t *)a.workspace + partial_region_bytes(a.sm_count));

    const long long tiles_ll = (long long)p.row_tiles * p.tok_tiles;
    // the kernel numbers tiles, the units (tile, chunk) of cut tiles and a pair's units in 32 bits
    constexpr long long kLimit = 1ll << 30;
    if (tiles_ll >= kLimit || (long long)split.sk_tiles * p.chunks >= kLimit || (tiles_ll / pairs + 2) * p.chunks >= kLimit) return TUNA_ERR_TOO_LARGE;
    p.status = device_status_word();
    if (!p.status) return TUNA_ERR_NO_DEVICE;
    const int tiles = (int)tiles_ll;
    p.sk_tiles = split.sk_tiles;
    p.sk_pairs = split.sk_pairs;
    if (p.sk_tiles) {
        const int units = p.sk_tiles * p.chunks;
        if (p.sk_pairs > units) p.sk_pairs = units;
        p.sk_q = units / p.sk_pairs;
        p.sk_r = units % p.sk_pairs;
    }
    const int busy = tiles - p.sk_tiles > p.sk_pairs ? tiles - p.sk_tiles : p.sk_pairs;  // pairs with work
    if (pairs > busy) pairs = busy;

    CUtensorMap mq, mx, mo;
    const int steps = l.kc / 32;
    int w_mode = weight_map_has_runs(a.m, a.k) ? 1 : 0;
    if (!make_weight_map(&mq, a.q, a.m, a.k, steps, &w_mode, &p.q3d)) return TUNA_ERR_NO_DEVICE;
    // activations as [n] x [k] fp16; box = half a tile's tokens x 64 columns
    if (!make_tensor_map_2d(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x, (uint64_t)a.k, (uint64_t)a.n, (uint64_t)a.k * 2, 64,
                            (uint32_t)l.tile_tok / 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return TUNA_ERR_NO_DEVICE;
    // output as [n] x [m] fp16; box = a tile's tokens x 64 rows
    if (!make_tensor_map_2d(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.o, (uint64_t)a.m, (uint64_t)a.n, (uint64_t)a.m * 2, 64,
                            (uint32_t)l.tile_tok, CU_TENSOR_MAP_SWIZZLE_128B))
        return TUNA_ERR_NO_DEVICE;
    switch (split.warps * 1000 + l.kc + w_mode) {
        case 8064: return launch_pair<64, 0, 8>(p, mq, mx, mo, 2 * pairs, a.stream);
        case 8065: return launch_pair<64, 1, 8>(p, mq, mx, mo, 2 * pairs, a.stream);
        case 8128: return launch_pair<128, 0, 8>(p, mq, mx, mo, 2 * pairs, a.stream);
        case 8129: return launch_pair<128, 1, 8>(p, mq, mx, mo, 2 * pairs, a.stream);
        case 16064: return launch_pair<64, 0, 16>(p, mq, mx, mo, 2 * pairs, a.stream);
        case 16065: return launch_pair<64, 1, 16>(p, mq, mx, mo, 2 * pairs, a.stream);
        case 16128: return launch_pair<128, 0, 16>(p, mq, mx, mo, 2 * pairs, a.stream);
        default: return launch_pair<128, 1, 16>(p, mq, mx, mo, 2 * pairs, a.stream);
    }
}

}  // namespace tuna
