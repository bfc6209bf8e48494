// Weight-streaming FP16 x 4-bit(codebook) GEMM on tcgen05 for small token counts (one pass
// covers 16, 32 or 64 tokens) on sm_100a: the memory-bound regime every row of the
// reference's README table is measured in.  Counterpart of the reference's Tuna<> kernel and its
// cp.async / ldmatrix / mma.sync main loop (kernel.cu:1043-2505, 2816-2960); the orientation
// is kept (weights are MMA operand A, tokens operand B, the accumulator is an o^T tile,
// kernel.cu:2182-2192) and nothing else.
//
// The idea.  The packed layout stores an 8x8 weight tile as 32 bytes (test.py:58-65: byte j =
// row j/4, column pair j%4), so the 8 columns of one row are one 32-bit word of the tile.  A
// dequant thread owns one weight row = one tensor-memory lane: per 32-column step it reads the
// row's four words (one per tile), turns their 16 bytes into 16 half2 by 16 table lookups and
// writes them to 16 consecutive tensor-memory columns with one tcgen05.st (shape 32x32b).  K
// stays in natural order, so the activations need no re-ordering at all: TMA writes x straight
// into the 128-byte-swizzled K-major tiles the MMA's shared-memory descriptor reads.  The
// dequantised weights exist only in registers and tensor memory.  (An earlier version used the
// 16x256b store shape, whose fragment is exactly a 16-byte piece of the packed layout: no
// row permutation to undo, but a K permutation that two extra warps had to apply to x through
// shared memory, and a store shape that costs the tensor-memory write path a third more.)
// Which row a lane holds is chosen for the shared-memory reads: lane 32q + l holds row
// 8*rg + l%8 with rg = 8*(q/2) + q%2 + 2*(l/8), so the four row groups a warp reads at once
// differ in bits 1-2 of rg - the bits the 128-byte swizzle XORs into the 16-byte chunk index -
// and the warp's 32-bit reads are bank-conflict free.  The epilogue undoes it (one lane per thread).
//
// The packed weights are staged by TMA: per slot (16 row groups x 512 or 1024 bytes = 128 rows
// x 128 or 256 columns) one 3-D box, or one 2-D box per step where the 3-D view does not exist
// (k not a multiple of 32), into an mbarrier-tracked ring of [step][row group][128 bytes]
// stages, 128-byte swizzled, that takes all the shared memory left; out-of-range rows and
// columns are zero-filled by the copy engine.  (A first version streamed the weights with
// ld.global into a per-lane register ring: 64 KB per SM at best, less whenever a warp was busy
// converting, and the loaded HBM latency of ~2 us capped it near 3.3 TB/s.)
//
// One persistent CTA per SM, warp-specialised (24 warps; 80 registers per
// thread.  Re-balancing registers between warpgroups with setmaxnreg made ptxas spill more,
// not less, in this kernel):
//   warp 0       MMA issue: tcgen05.mma (M=128, N=tile_tok, K=16, fp32 accumulate), A from tensor
//                memory, B through a 128-byte-swizzle shared-memory descriptor, D in tensor memory.
//                The warp stays converged and one elected lane issues (a lone diverged thread
//                running this loop needed ~80 clocks per MMA instead of ~12); a slot is 8 or 16
//                MMAs per wait and commit, because that fixed cost per slot is what limits it
//   warp 1       copy producer of x (fp16 [n,k], L2 resident; one box per 64 columns) into the activation ring
//   warp 2       copy producer of the packed weights (TMA boxes into the weight ring); it initialises the barriers and issues the
//                first ring-full ahead of everything: 2000 clocks that the others waited for (4096x4096 at 1 token 7.3 -> 6.8 us, graph replay)
//   warp 3       no role
//   warps 4-7    epilogue: tcgen05.ld of the accumulator, fp32 scale by absmax, fp16 store,
//                split-K partials and fix-up
//   warps 8-23   dequant: ld.shared.u32 -> prmt + ld.shared table lookups -> tcgen05.st into the A
//                slots.  A warp handles rows 32q..+31 (q = its 32-lane quarter) and four
//                32-column steps of a slot; with 128-column slots four groups of four warps
//                convert four slots at once, with 256-column slots two groups of eight warps two.
// The scale is constant along K (one block per row, test.py:81, kernel.cu:2178-2180) and is
// applied once, in fp32, to the accumulated sum.
//
// Work decomposition ("stream-K"): a unit is (tile of 128*row_blocks rows, 128- or 256-column chunk) =
// row_blocks slots; the units, tile-major, are cut into one contiguous range per CTA so that
// every SM streams the same number of bytes whatever the shape (a single GEMM may take fewer CTAs, so that its tiles
// are cut into whole segments: ts_pick_split).  A tile cut across CTAs is finished by whichever CTA arrives last at
// the tile's counter (per 32-row quarter): it adds the fp32 partials from the workspace in range order, so the
// result does not depend on arrival order (the reference adds fp16 partials with atomicAdd, kernel.cu:2739-2745).  No
// floating-point atomics, no zero-filled output.  This tail is what a single small GEMM waits for: at 28672x4096 and 16
// tokens the last MMA was done at 16.7 us of 24.1.  Hence only token groups that exist are exchanged, one
// acquire-release atomic per warp replaces two fences, and at the end of the range all 24 warps add up the tile, eight
// tokens of 32 rows each, instead of four warps 16 tokens at a time (graph replay, 16 tokens unless said, us):
// 4096x4096 10.3 -> 9.9, 57344x8192 67.0 -> 65.2, 4096x4096 at 64 tokens 20.1 -> 14.2, 768x4096 at 64 49.7 -> 12.9; with that
// code in one place only, outside the roles, 4096x4096 7.8, 57344x8192 53.5, 4096x4096 at 64 10.9.
//
// Programmatic dependent launch: the kernel lets its successor start as SMs free up and itself waits for its predecessors
// only before it touches what they may have written (activations, workspace, output); the weights and the
// codebook are constants, requested before, and dequantised into the A-slot ring meanwhile.
//
// Every wait is bounded: when one runs out the CTA records where in the device status word,
// raises a CTA-wide abort flag and unwinds to the common exit, where tensor memory is released.
#include <cstring>
#include <mutex>
#include "common.cuh"
#include "launchers.h"
#include "ring_plan.h"
#include "sm100_ptx.cuh"
#include "tcgen05.cuh"

// Optional per-warp timing (debug builds with -DTUNA_TS_PROFILE only): absolute times of the
// warp's milestones and the clocks it spent in each kind of wait.
#ifdef TUNA_TS_PROFILE
__device__ long long g_ts_prof[160 * 24 * 8];
__device__ __forceinline__ long long ts_gtime()
{
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define TS_PROF_DECL long long pw_[4] = {0, 0, 0, 0}, pt_ = 0, pg_[4] = {ts_gtime(), 0, 0, 0}; (void)pt_;
#define TS_PROF_MARK(i) pg_[i] = ts_gtime();
#define TS_PROF_BEGIN pt_ = clock64();
#define TS_PROF_END(i) pw_[i] += clock64() - pt_;
#define TS_PROF_STORE                                                                     \
    if ((threadIdx.x & 31) == 0) {                                                        \
        long long *d_ = g_ts_prof + ((size_t)blockIdx.x * 24 + (threadIdx.x >> 5)) * 8;   \
        for (int i_ = 0; i_ < 4; ++i_) { d_[i_] = pg_[i_]; d_[4 + i_] = pw_[i_]; }        \
    }
#else
#define TS_PROF_DECL
#define TS_PROF_MARK(i)
#define TS_PROF_BEGIN
#define TS_PROF_END(i)
#define TS_PROF_STORE
#endif

namespace tuna {

constexpr int kTsMaxASlots = 8;       // A-slot ring: as many slots as the accumulators leave room for
constexpr int kTsTmemCols = 512;
constexpr int kTsMaxXStages = 6;
constexpr int kTsMaxWStages = 16;     // weight ring: as many stages as shared memory holds
constexpr int kTsLutBytes = 256 * 128;    // byte -> half2 table: 256 entries, 32 copies (one per bank) of 4 bytes
constexpr int kTsSmemTotal = 227 * 1024;             // static + dynamic shared memory of a CTA on sm_100
constexpr int kTsSmemDynamic = kTsSmemTotal - 1024;  // the static part (barriers) stays below 1 KB
constexpr int kTsBars = 2 * kTsMaxASlots + 2 * kTsMaxXStages + 4 + 2 * kTsMaxWStages;
constexpr int kTsXWarp = 1, kTsWeightWarp = 2, kTsEpilogueWarp0 = 4;
constexpr int kTsDequantWarp0 = 8;
#ifndef TS_DEQUANT_WARPS
#define TS_DEQUANT_WARPS 16
#endif
constexpr int kTsDequantWarps = TS_DEQUANT_WARPS;
constexpr int kTsThreads = 32 * (kTsDequantWarp0 + kTsDequantWarps);

constexpr int kTsMaxSeq = kSequenceMax;  // GEMMs of one launch (tuna_matmul_sequence)
constexpr int kMaxPeers = TUNA_MAX_PEERS;

// One GEMM of a launch.  The two tensor maps are what the copy producer hands to TMA; everything
// else is read by the epilogue warps and the cursors.
struct __align__(64) TsGemm {
    CUtensorMap map_q;   // packed weights: the 5-D view (w_mode 1), else the 3-D view if q3d, else [m/8 row groups] x [k 32-bit words]
    CUtensorMap map_x;   // activations as [n] x [k] fp16
    const float *absmax;
    __half *o;
    int m, n, k;
    int chunks;       // ceil(k / chunk columns)
    int row_tiles;    // ceil(m / (128 RB))
    int unit0;        // index of its first unit in the launch's unit sequence
    int tile0;        // index of its first tile among the launch's tiles (arrival counters)
    int q3d;          // map_q is the 3-D view (one copy per slot) rather than the 2-D one (one copy per step)
    long long slab_off;  // exchange launches: offset of this rank's slab for this GEMM inside a parity region, -1: none (o is written)
};

struct TsParams {
    const float *code;
    float *partials;
    unsigned int *counters;
    DeviceStatus *status;
    int count;        // GEMMs of this launch
    int tok0;         // first token of this pass (0 unless a single GEMM runs as several passes)
    int row_blocks;   // RB: 128-row blocks per tile
    int a_slots;      // A-slot ring depth
    int a_base;       // first tensor-memory column of the A slots (behind the two accumulator buffers)
    int acc_cols;     // columns of one accumulator buffer
    int units;        // units of all the GEMMs
    int units_q, units_r;  // units = units_q * CTAs + units_r: the first units_r CTAs take units_q + 1
    int w_mode;       // layout of the weight stages (the kernel's WMODE)
    // Exchange launches (K-split GEMMs whose partial outputs every rank sums): instead of o, a
    // finished row goes to this rank's slab ([row][tile_tok] fp16) in the exchange buffer of every
    // rank, with ordinary stores to peer memory; the reduce kernel that follows sums the slabs.
    int n_peers;                 // 0: an ordinary launch
    unsigned char *peer[kMaxPeers];
    const unsigned int *epoch;   // exchanges completed so far on this rank (device counter): its parity selects the region
    long long region0, region_bytes;  // offset of parity region 0 inside an exchange buffer, and the size of a region
};

template <int MAXG>
struct __align__(64) TsLaunch {
    TsParams c;
    TsGemm g[MAXG];
};

// Table lookup: the selected byte of w (two 4-bit codes) -> half2 of the two code values.  Entry e
// of the table lies at 128 * e, one copy per bank: conflict free.
__device__ __forceinline__ uint32_t ts_lookup(uint32_t w, uint32_t lane_base, uint32_t selector)
{
    uint32_t b, v;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(b) : "r"(w), "r"(selector));
    // not volatile: the table is constant once built, so the compiler may schedule lookups freely
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(lane_base + (b << 7)));
    return v;
}

// The same lookup when the table lies at shared address 0x10000 with 256 bytes per entry: the
// address 0x10000 + 256 * byte + 4 * lane is assembled by ONE prmt from `key` = 0x00010000 | 4 * lane
// (bytes 0, 2, 3) and the selected byte of w (byte 1); `selector` = 0x7604 | (byte index << 4).
__device__ __forceinline__ uint32_t ts_lookup256(uint32_t w, uint32_t key, uint32_t selector)
{
    uint32_t a, v;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(a) : "r"(w), "r"(key), "r"(selector));
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// Weight stages below the lookup table, and all of them, where the first one starts at shared address `w_low`.
__host__ __device__ constexpr int ts_low_stages(bool lut256, uint32_t w_low, uint32_t slot_bytes)
{
    return lut256 && w_low < 0x10000u ? (int)((0x10000u - w_low) / slot_bytes) : 0;
}
__host__ __device__ constexpr int ts_w_stages(bool lut256, uint32_t w_low, uint32_t smem_end, uint32_t slot_bytes)
{
    const int n = ts_low_stages(lut256, w_low, slot_bytes) + (int)((smem_end - (lut256 ? 0x20000u : w_low)) / slot_bytes);
    return n < kTsMaxWStages ? n : kTsMaxWStages;
}
// Columns of one accumulator buffer (32 is the allocation granule), and A slots behind the two of them.
__host__ __device__ constexpr int ts_acc_cols(int row_blocks, int tile_tok) { return row_blocks * tile_tok < 32 ? 32 : row_blocks * tile_tok; }
__host__ __device__ constexpr int ts_a_slots(int acc_cols, int steps)
{
    const int n = (kTsTmemCols - 2 * acc_cols) / (16 * steps);
    return n < kTsMaxASlots ? n : kTsMaxASlots;
}
// Whether the dequant groups may share the rings (ring_plan.h) wherever dynamic shared memory begins, which is checked to be in the first 4 KB.
constexpr bool ts_rings_shareable(int tile_tok, int steps, bool lut256, uint32_t x_ring_bytes)
{
    for (int rb = 1; rb == 1 || rb * tile_tok <= 64; rb *= 2)
        for (uint32_t dyn0 = 1024; dyn0 <= 4096; dyn0 += 1024) {
            const uint32_t w_low = dyn0 + (lut256 ? 0u : kTsLutBytes) + x_ring_bytes;
            const int w = ts_w_stages(lut256, w_low, dyn0 + kTsSmemDynamic, 16 * 32 * 4 * steps);
            if (!rings_shareable(w, ts_a_slots(ts_acc_cols(rb, tile_tok), steps), kTsDequantWarps / steps)) return false;
        }
    return true;
}

// The CTA whose range holds unit u.
__device__ __forceinline__ int ts_cta_of_unit(const TsParams &p, int u)
{
    const int big = p.units_r * (p.units_q + 1);
    return u < big ? u / (p.units_q + 1) : p.units_r + (u - big) / p.units_q;
}

// Position in a CTA's contiguous range of the launch's unit sequence (GEMM after GEMM, each
// tile-major): which GEMM, which row tile, which K chunk.
struct TsCursor {
    int g, tile, chunk;
    int chunks, row_tiles;  // of GEMM g
    int left;               // units of the range still ahead, including the current one
    bool seg_first;         // the current unit starts a segment (the units of one tile inside the range)
    template <class Launch>
    __device__ void init(const Launch &L, int u_begin, int n_units)
    {
        g = 0;
        while (g + 1 < L.c.count && L.g[g + 1].unit0 <= u_begin) ++g;
        chunks = L.g[g].chunks;
        row_tiles = L.g[g].row_tiles;
        const int r = u_begin - L.g[g].unit0;
        tile = r / chunks;
        chunk = r - tile * chunks;
        left = n_units;
        seg_first = true;
    }
    __device__ bool seg_last() const { return chunk + 1 == chunks || left == 1; }
    template <class Launch>
    __device__ void next(const Launch &L)
    {
        seg_first = seg_last();
        --left;
        if (++chunk == chunks) {
            chunk = 0;
            if (++tile == row_tiles && left > 0) {
                tile = 0;
                ++g;
                chunks = L.g[g].chunks;
                row_tiles = L.g[g].row_tiles;
            }
        }
    }
};

// STEPS: 32-column steps per slot (4 or 8).  MAXG: capacity of the launch's GEMM table (1 for a
// single GEMM, kTsMaxSeq for a sequence).  WMODE: layout of a weight stage (128-byte rows, 128-byte
// swizzle), the same for all GEMMs of a launch:
//   1  [32-row block][step pair][row group of the block][step of the pair]: one 5-D box per slot
//      that reads global memory in runs of 256 contiguous bytes (m % 32 == 0 and k % 64 == 0);
//      a warp's four row groups are consecutive and the swizzle separates them, so tensor-memory
//      lane l holds row l of the 128;
//   0  [step][row group]: one 3-D box per slot (k % 32 == 0; 128-byte runs, measured 8 % slower in
//      the copy alone) or one 2-D box per step (any k); rows assigned to lanes by lane_row_group().
template <int N_TILE, int STEPS, int MAXG, int WMODE>
__global__ void __launch_bounds__(kTsThreads, 1) gemm_w4a16_tstream_kernel(const __grid_constant__ TsLaunch<MAXG> L)
{
    const TsParams &p = L.c;
    constexpr int kChunkK = 32 * STEPS;                     // columns of a unit / slot
    constexpr int kSlotCols = 16 * STEPS;                   // tensor-memory columns of one A slot
    constexpr int kSlotBytes = 16 * kChunkK * 4;            // packed bytes of a slot: 16 row groups x 4 bytes per column
    constexpr int kHalves = STEPS / 4;                      // warps that share a quarter of a slot
    constexpr int kGroups = kTsDequantWarps / (4 * kHalves);  // slots converted at once
    // Activations of a unit: one tile of [token][64 columns] fp16 (128-byte rows, 128-byte swizzle,
    // 8-token groups 1024 bytes apart) per 64 columns, as TMA writes it and the MMA descriptor reads it.
    constexpr int kXTiles = kChunkK / 64;
    constexpr uint32_t kXTileBytes = N_TILE * 128;
    constexpr uint32_t kXStageBytes = kXTiles * kXTileBytes;
    // activation stages (TMA -> MMA); up to 32 tokens the ring has to fit below the lookup table (shared address 0x10000)
    constexpr int kXS = (N_TILE >= 64 || 4 * kXStageBytes + 4096 > 0x10000) ? 3 : 4;
    constexpr uint32_t kStepBytes = 16 * 128;                         // one step of a weight stage: 16 row groups x 128 bytes
    static_assert(kXS <= kTsMaxXStages, "barrier arrays too small");
    static_assert(N_TILE > 32 || kXS * kXStageBytes + 4096 <= 0x10000, "the activation ring must end below the lookup table");
    static_assert(kXStageBytes % 1024 == 0 && kSlotBytes % 1024 == 0, "swizzle atoms are 1024 bytes");
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kTsBars];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    // The cut tiles of the CTA's range, at most its first [0] and its last [1], that this CTA finishes at its end
    __shared__ int s_fix[2][4];   // by quarter
    __shared__ int s_tile[2][4];  // GEMM, tile, first CTA and segments

    TS_PROF_DECL
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int cta = blockIdx.x;
    const int RB = p.row_blocks;

    // Let the next kernel in the stream become resident as SMs free up.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // Shared memory (everything 1024-byte aligned): the byte -> half2 table (256 entries, one copy per
    // bank), the activation ring, and weight stages in everything that is left.
    //   kLut256 (token tiles up to 32): the table occupies shared addresses [0x10000, 0x20000) with 256
    //   bytes per entry (half of them unused), which lets one prmt build a lookup's address; the
    //   activation ring and the first weight stages lie below it, the other weight stages above.
    //   Otherwise (64-token tiles need the room): 128 bytes per entry at the start of dynamic shared memory.
    constexpr bool kLut256 = N_TILE <= 32;
    const uint32_t dyn0 = smem_u32(smem);
    const uint32_t smem_end = dyn0 + kTsSmemDynamic;
    const uint32_t lut_addr = kLut256 ? 0x10000u : dyn0;
    const uint32_t xring = kLut256 ? dyn0 : dyn0 + kTsLutBytes;
    const uint32_t w_low = xring + kXS * kXStageBytes;                       // first weight stage
    const int n_low = ts_low_stages(kLut256, w_low, kSlotBytes);  // weight stages below the table
    const uint32_t w_high = kLut256 ? 0x20000u : w_low;
    const int WS = ts_w_stages(kLut256, w_low, smem_end, kSlotBytes);
    static_assert(ts_rings_shareable(N_TILE, STEPS, kLut256, kXS * kXStageBytes), "a dequant group could pass its wait for a weight stage a phase early");
    auto w_stage = [&](int i) -> uint32_t { return i < n_low ? w_low + (uint32_t)i * kSlotBytes : w_high + (uint32_t)(i - n_low) * kSlotBytes; };
    if (kLut256 && dyn0 > 4096u) {  // the layout above assumes that dynamic shared memory starts within the first 4 KB
        if (threadIdx.x == 0 && atomicCAS(&p.status->code, 0, 97) == 0) p.status->detail = (int)dyn0;
        return;
    }

    const uint32_t bar0 = smem_u32(&bars[0]);
    const uint32_t a_full = bar0, a_empty = a_full + 8 * kTsMaxASlots;
    const uint32_t x_full = a_empty + 8 * kTsMaxASlots, x_empty = x_full + 8 * kTsMaxXStages;
    const uint32_t d_full = x_empty + 8 * kTsMaxXStages, d_empty = d_full + 16;
    const uint32_t w_full = d_empty + 16, w_empty = w_full + 8 * kTsMaxWStages;
    volatile int *abort_flag = &s_abort;

    // this CTA's contiguous range of units
    const int u_begin = cta * p.units_q + min(cta, p.units_r);
    const int n_units = p.units_q + (cta < p.units_r ? 1 : 0);

    // The weight producer initialises the barriers, 32 at a time, and goes on to its copies without waiting for anyone:
    // issuing a ring-full takes longer than the rest of the prologue.
    if (warp == kTsWeightWarp) {
        auto count = [](int i) {
            if (i < kTsMaxASlots) return 4 * kHalves;                  // a_full
            i -= 2 * kTsMaxASlots + 2 * kTsMaxXStages + 4;
            if (i < -2 || (i >= 0 && i < kTsMaxWStages)) return 1;     // a_empty, x_full, x_empty, d_full; w_full
            return i < 0 ? 4 : 4 * kHalves;                            // d_empty; w_empty
        };
        for (int i = lane; i < kTsBars; i += 32) mbar_init(bar0 + 8 * i, count(i));
        if (lane == 0) s_abort = 0;
        if (lane < 8) s_fix[lane >> 2][lane & 3] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
    } else if (warp == kTsXWarp) {
        if (elect_one_sync()) prefetch_map(&L.g[0].map_x);
    } else if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                     "r"(kTsTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }

    const int quarter = warp & 3;          // the 32 tensor-memory lanes this warp may access
    const int total_slots = n_units * RB;

    // Rest of the prologue, run by every other warp inside its own role's branch: the byte -> half2
    // table (even column = high nibble in the low half), one copy per bank, by the epilogue and dequant warps - the
    // codebook is a constant, so this needs no dependency wait - then the CTA barrier that publishes barriers, table and
    // tensor-memory base.  Only what reads or writes data of the kernels before this one waits for
    // them (depend(): the copies of x, the epilogue, and before their bounded waits the MMA warp and
    // whoever has filled its ring), so the dequant warps fill the A-slot ring meanwhile.
    auto finish_prologue = [&]() -> uint32_t {
        if (warp >= kTsEpilogueWarp0) {
            const float cv = p.code[lane & 15];
            const uint32_t ch = (uint32_t)__half_as_ushort(__float2half_rn(cv));
            for (int e = warp - kTsEpilogueWarp0; e < 256; e += kTsThreads / 32 - kTsEpilogueWarp0) {
                const uint32_t v = __shfl_sync(0xffffffffu, ch, e >> 4) | (__shfl_sync(0xffffffffu, ch, e & 15) << 16);
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(lut_addr + (uint32_t)e * (kLut256 ? 256 : 128) + lane * 4), "r"(v) : "memory");
            }
        }
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(kTsThreads) : "memory");
        tc_fence_after();
        TS_PROF_MARK(1)
        return s_tmem_base;
    };
    auto depend = [] { asm volatile("griddepcontrol.wait;" ::: "memory"); };

    const size_t slot_floats = (size_t)RB * kBlockRows * N_TILE;
    // the row of a block that lane `lane` of quarter q holds
    auto row_in_block = [&](int q) { return WMODE == 1 ? 32 * q + lane : 8 * lane_row_group(q, lane) + (lane & 7); };
    // groups of four tokens of the tile that exist (an exchange slab takes the whole tile)
    auto token_groups = [&](const TsGemm &G) { return p.n_peers > 0 ? N_TILE / 4 : (min(G.n - p.tok0, N_TILE) + 3) >> 2; };
    // NT tokens from token `t0` of the tile on of one finished row, scaled: to o, or (16 tokens) to every rank's slab
    auto store_row = [&](const TsGemm &G, int row, int t0, const auto &v, float sc) __attribute__((always_inline)) {
        constexpr int NT = sizeof(v) / sizeof(float);
        if (NT == 16 && p.n_peers > 0 && G.slab_off >= 0) {
            uint32_t h[NT / 2];
#pragma unroll
            for (int i = 0; i < NT / 2; ++i) {
                const __half2 t = __floats2half2_rn(v[2 * i] * sc, v[2 * i + 1] * sc);
                h[i] = *reinterpret_cast<const uint32_t *>(&t);
            }
            // where this launch's slabs start: every caller is past the dependency wait
            const long long region = p.region0 + (long long)((__ldcg(p.epoch) + 1u) & 1u) * p.region_bytes;
            const long long off = region + G.slab_off + ((long long)row * N_TILE + t0) * 2;
            for (int pr = 0; pr < p.n_peers; ++pr) {
                uint4 *dst = reinterpret_cast<uint4 *>(p.peer[pr] + off);
#pragma unroll
                for (int i = 0; i < NT / 8; ++i) dst[i] = make_uint4(h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int tok = p.tok0 + t0 + i;
                if (tok < G.n) G.o[(size_t)tok * G.m + row] = __float2half_rn(v[i] * sc);
            }
        }
    };
    // Adds the partials of GR four-token groups from group g0 on (the last group that exists stands in for those after it) of 32 rows (block rb, quarter q of the tile) over its
    // segments, which CTAs `first` .. first + nseg - 1 wrote, and stores the rows.  The loads of SG segments are
    // in flight at a time, the adds keep the range order.  Their addresses are 32-bit offsets into the partial sums (partial_region_bytes, far
    // below 4 GB): this runs once per CTA, out of a cold instruction cache, and with 64-bit arithmetic per load eight in flight took longer than four
    // (768x2304 at 15 tokens, nine segments, by four / by eight / so: 5.63 / 6.06 / 5.63 us; 1152x3328 at 11 6.14 / 6.06 / 5.72).
    auto add_partials = [&](auto gr, auto sg, const TsGemm &G, int tile, int first, int nseg, int q, int rb, int g0, int last) __attribute__((always_inline)) {
        constexpr int GR = decltype(gr)::value, SG = decltype(sg)::value;
        const int row = (tile * RB + rb) * kBlockRows + row_in_block(q);
        if (row >= G.m) return;
        const float sc = G.absmax[row];
        const uint32_t slot_bytes = (uint32_t)slot_floats * 4u;
        const uint32_t at = (uint32_t)(2 * first) * slot_bytes + (uint32_t)(rb * (N_TILE / 4) * kBlockRows + 32 * q + lane) * 16u;
        float acc[4 * GR];
#pragma unroll
        for (int i = 0; i < 4 * GR; ++i) acc[i] = 0.f;
#pragma unroll 1
        for (int sgm = 0; sgm < nseg; sgm += SG) {
            float4 a[SG][GR];
#pragma unroll
            for (int j = 0; j < SG; ++j) {
                const int seg = min(sgm + j, nseg - 1);
                const uint32_t off = at + (uint32_t)(2 * seg + (seg == 0 ? 1 : 0)) * slot_bytes;
#pragma unroll
                for (int i = 0; i < GR; ++i)
                    a[j][i] = __ldcg(reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(p.partials) + (off + (uint32_t)min(g0 + i, last) * (kBlockRows * 16u))));
            }
#pragma unroll
            for (int j = 0; j < SG; ++j) {
                const bool live = sgm + j < nseg;
#pragma unroll
                for (int i = 0; i < GR; ++i)
                    if (live) { acc[4 * i] += a[j][i].x; acc[4 * i + 1] += a[j][i].y; acc[4 * i + 2] += a[j][i].z; acc[4 * i + 3] += a[j][i].w; }
            }
        }
        store_row(G, row, 4 * g0, acc, sc);
    };
    // The flagged quarters of a tile whose partials are all there, shared out over warps `w0`, w0 + step, ... : a warp
    // takes eight tokens of 32 rows at a time, so that all of a tile is in flight at once (28672x4096 at 16 tokens, two row blocks: by
    // four 18.0 us, by eight 17.7), four of them where that takes no second round and there are more than four segments, eight of which
    // are in flight then (1152x3328 at 11 tokens 6.1 -> 5.7), in exchange launches 16, whole sectors of a peer's slab.
    auto finish_tile = [&](const TsGemm &G, int tile, int first, int nseg, const int *flagged, int w0, int step) __attribute__((always_inline)) {
        const int groups4 = token_groups(G), rb_shift = RB >> 1;
        const int per = p.n_peers > 0 ? 4 : nseg <= 4 || (groups4 << (2 + rb_shift)) > step ? 2 : 1;
        for (int item = w0; (item >> (2 + rb_shift)) * per < groups4; item += step) {
            const int q = item & 3, rest = item >> 2;
            const int g = (rest >> rb_shift) * per, rb = rest & (RB - 1);  // RB is 1, 2 or 4
            if (!flagged[q]) continue;
            if (per == 1) add_partials(Int<1>(), Int<8>(), G, tile, first, nseg, q, rb, g, groups4 - 1);
            else if (per == 2) add_partials(Int<2>(), Int<4>(), G, tile, first, nseg, q, rb, g, groups4 - 1);
            else add_partials(Int<4>(), Int<2>(), G, tile, first, nseg, q, rb, g, groups4 - 1);
        }
    };
    auto first_cta = [&](const TsGemm &G, int tile) { return ts_cta_of_unit(p, G.unit0 + tile * G.chunks); };
    auto last_cta = [&](const TsGemm &G, int tile) { return ts_cta_of_unit(p, G.unit0 + (tile + 1) * G.chunks - 1); };
    uint32_t tmem = 0;

    if (warp == 0) {
        // ------------------------------------------------------------------ MMA issue
        // The warp stays converged: every lane runs the loop and the waits, one elected lane
        // issues the MMAs and the commits.  Descriptors (K-major, 128-byte swizzle): the high word
        // is constant (8-token groups 1024 bytes apart, version 1, layout type 2), the low word is the
        // start address; 16 columns further along K is 32 bytes further inside the 128-byte row.
        constexpr uint32_t idesc = make_idesc(N_TILE);
        constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
        Ring ra, rx, rd;
        TsCursor cur;
        cur.init(L, u_begin, n_units);
        tmem = finish_prologue();
        depend();
        bool ok = true;
        for (int u = 0; ok && u < n_units; ++u, cur.next(L)) {
            const bool seg_first = cur.seg_first, seg_last = cur.seg_last();
            TS_PROF_BEGIN
            if (seg_first) ok = mbar_wait(d_empty + 8 * rd.idx, rd.phase ^ 1, abort_flag, p.status, 3);
            TS_PROF_END(0)
            TS_PROF_BEGIN
            ok = ok && mbar_wait(x_full + 8 * rx.idx, rx.phase, abort_flag, p.status, 4);
            ok = __all_sync(0xffffffffu, ok) != 0;
            TS_PROF_END(1)
            if (!ok) break;
            const uint32_t desc_lo0 = ((xring + (uint32_t)rx.idx * kXStageBytes) & 0x3FFFFu) >> 4;
            const uint32_t dbase = tmem + (uint32_t)(rd.idx * p.acc_cols);
            for (int rb = 0; rb < RB; ++rb) {
                TS_PROF_BEGIN
                ok = mbar_wait_warp(a_full + 8 * ra.idx, ra.phase, abort_flag, p.status, 5);
                TS_PROF_END(2)
                if (!ok) break;
                tc_fence_after();
                TS_PROF_BEGIN
                if (elect_one_sync()) {
                    const uint32_t abase = tmem + (uint32_t)p.a_base + (uint32_t)ra.idx * kSlotCols;
#pragma unroll
#ifdef TS_ABL_NOMMA  // timing experiment: commits only
                    for (int mm = 0; mm < 0; ++mm) {
#else
                    for (int mm = 0; mm < 2 * STEPS; ++mm) {  // columns 16 mm .. 16 mm + 15 of the slot: 64-column tile mm/4
#endif
                        const uint64_t bdesc = ((uint64_t)desc_hi << 32) | (uint64_t)(desc_lo0 + (mm >> 2) * (kXTileBytes >> 4) + (mm & 3) * 2);
                        tc_mma_ts(dbase + (uint32_t)rb * N_TILE, abase + mm * 8, bdesc, idesc, (seg_first && mm == 0) ? 0u : 1u);
                    }
                    tc_commit(a_empty + 8 * ra.idx);
                    if (rb + 1 == RB) {
                        tc_commit(x_empty + 8 * rx.idx);
                        if (seg_last) tc_commit(d_full + 8 * rd.idx);
                    }
                }
                __syncwarp();
                TS_PROF_END(3)
                ra.advance(p.a_slots);
            }
            rx.advance(kXS);
            if (seg_last) rd.advance(2);
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------------ no role after the prologue
        tmem = finish_prologue();
    } else if (warp == kTsXWarp) {
        // ------------------------------------------------------------------ copy producer of the activations
        // One elected lane of the converged warp issues, per unit, kChunkK/64 boxes of x (tile_tok tokens x 64
        // columns, L2 resident; tokens past n and columns past k zero-filled) into the activation ring, released by the
        // MMAs' commit.
        Ring rn;
        TsCursor xc;
        xc.init(L, u_begin, n_units);
        finish_prologue();
        depend();
        for (int u = 0; u < n_units; ++u, xc.next(L)) {
            if (!mbar_wait_warp(x_empty + 8 * rn.idx, rn.phase ^ 1, abort_flag, p.status, 9)) break;
            if (elect_one_sync()) {
                mbar_expect_tx(x_full + 8 * rn.idx, kXStageBytes);
#pragma unroll
                for (int t = 0; t < kXTiles; ++t)
                    tma_load_2d(xring + (uint32_t)rn.idx * kXStageBytes + (uint32_t)t * kXTileBytes, &L.g[xc.g].map_x,
                                xc.chunk * kChunkK + 64 * t, p.tok0, x_full + 8 * rn.idx);
            }
            __syncwarp();
            rn.advance(kXS);
        }
    } else if (warp == kTsWeightWarp) {
        // ------------------------------------------------------------------ copy producer of the weights
        // Per slot one elected lane of the converged warp issues the packed weights (16 row groups x kChunkK 32-bit words;
        // one 5-D or 3-D box, or one 2-D box per step) into the weight ring.  The weights are constants:
        // the first ring-full of their copies is issued before the dependency wait.
        asm volatile("bar.arrive 1, %0;" ::"n"(kTsThreads) : "memory");
        Ring rw;
        int w_rb = 0;
        TsCursor wc;
        wc.init(L, u_begin, n_units);
        for (int sl = 0; sl < total_slots; ++sl) {
            if (sl == WS) depend();
            TS_PROF_BEGIN
            const bool ok = mbar_wait_warp(w_empty + 8 * rw.idx, rw.phase ^ 1, abort_flag, p.status, 1);
            TS_PROF_END(0)
            if (!ok) break;
            if (elect_one_sync()) {
                const TsGemm &G = L.g[wc.g];
                mbar_expect_tx(w_full + 8 * rw.idx, kSlotBytes);
                if (WMODE == 1) {
                    tma_load_5d(w_stage(rw.idx), &G.map_q, 0, 0, 0, wc.chunk * (STEPS / 2), (wc.tile * RB + w_rb) * 4, w_full + 8 * rw.idx);
                } else if (G.q3d) {
                    tma_load_3d(w_stage(rw.idx), &G.map_q, 0, (wc.tile * RB + w_rb) * 16, wc.chunk * STEPS, w_full + 8 * rw.idx);
                } else {
#pragma unroll
                    for (int st = 0; st < STEPS; ++st)
                        tma_load_2d(w_stage(rw.idx) + (uint32_t)st * kStepBytes, &G.map_q, wc.chunk * kChunkK + 32 * st,
                                    (wc.tile * RB + w_rb) * 16, w_full + 8 * rw.idx);
                }
            }
            __syncwarp();
            rw.advance(WS);
            if (++w_rb == RB) {
                w_rb = 0;
                wc.next(L);
            }
        }
    } else if (warp < kTsDequantWarp0) {
        // ------------------------------------------------------------------ epilogue
        Ring rd;
        TsCursor cur;
        cur.init(L, u_begin, n_units);
        tmem = finish_prologue();
        depend();
        int u = 0;
        while (u < n_units) {
            // the segment: chunks [c0, c1) of tile `tile` of GEMM `cur.g`
            const TsGemm &G = L.g[cur.g];
            const int tile = cur.tile, c0 = cur.chunk;
            const int c1 = min(G.chunks, c0 + cur.left);
            const bool full = (c0 == 0 && c1 == G.chunks);
            TS_PROF_BEGIN
            if (!mbar_wait_warp(d_full + 8 * rd.idx, rd.phase, abort_flag, p.status, 6)) break;
            TS_PROF_END(0)
            tc_fence_after();
            TS_PROF_BEGIN
            const int groups4 = token_groups(G);
            float *my_partial = p.partials + (size_t)(2 * cta + (c0 == 0 ? 1 : 0)) * slot_floats;
            for (int rb = 0; rb < RB; ++rb) {
                const int row = (tile * RB + rb) * kBlockRows + row_in_block(quarter);
                const float sc = (full && row < G.m) ? G.absmax[row] : 0.f;
#pragma unroll 1
                for (int piece = 0; 4 * piece < groups4; ++piece) {
                    float v[16];
                    tc_ld_x16(tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(rd.idx * p.acc_cols) + (uint32_t)rb * N_TILE + piece * 16, v);
                    if (full) {
                        if (row < G.m) store_row(G, row, 16 * piece, v, sc);
                    } else {
                        // [rb][4-token group][128 lanes] float4: a warp store is 512 contiguous bytes
                        float4 *dst = reinterpret_cast<float4 *>(my_partial) + ((size_t)rb * (N_TILE / 4) + piece * 4) * kBlockRows + 32 * quarter + lane;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (4 * piece + i < groups4) dst[i * kBlockRows] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty + 8 * rd.idx);
            if (!full) {
                // Each epilogue warp arrives for its own 32 lanes at the counter of (tile, quarter).  Whoever arrives
                // last has all the partials; its CTA adds them up at the end of its range, with all its warps.  That is
                // the CTA whose range ends with the tile, unless the tile's other CTA started late.
                // lane 0's atomic releases the warp's partials and acquires the others'
                __syncwarp();
                const int first = first_cta(G, tile), nseg = last_cta(G, tile) - first + 1;
                unsigned int *counter = p.counters + (size_t)(G.tile0 + tile) * 4 + quarter;
                unsigned int old = 0;
                if (lane == 0) asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
                old = __shfl_sync(0xffffffffu, old, 0);
                if (old == (unsigned)nseg - 1) {
                    if (lane == 0) *counter = 0;  // leave the counter clean for the next call
                    if (lane == 0) {
                        const int e = u + (c1 - c0) < n_units ? 0 : 1;
                        s_fix[e][quarter] = 1;
                        // the same values from every flagged quarter
                        s_tile[e][0] = cur.g; s_tile[e][1] = tile; s_tile[e][2] = first; s_tile[e][3] = nseg;
                    }
                }
            }
            TS_PROF_END(1)
            for (int i = c0; i < c1; ++i) cur.next(L);
            u += c1 - c0;
            rd.advance(2);
        }
    } else {
        // ------------------------------------------------------------------ dequant
        // A group (4 * kHalves warps: one per 32-lane quarter and per four steps of a slot) converts
        // the slots j, j + kGroups, ... of this CTA: one wait / fence / arrival per slot and warp.
        // The groups work on different slots at once, so the latency of a slot's chain (shared
        // loads -> lookups -> tcgen05.st -> wait::st -> arrive) is overlapped kGroups times.
        const int dq = warp - kTsDequantWarp0;
        const int half = (dq >> 2) % kHalves;      // which four steps of the slot
        const int group = dq / (4 * kHalves);
        tmem = finish_prologue();
        const uint32_t lane_key = lut_addr + (uint32_t)(lane * 4);  // this lane's copy of the table (kLut256: also the prmt's second operand)
        const uint32_t a_lane0 = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)p.a_base + 64u * (uint32_t)half;
        // This thread's row inside a stage: word r%4 of 16-byte chunk 2 kt + r/4 of the 128-byte row
        // of (row group, step), the chunk index XORed with (index of that 128-byte row in the stage) % 8.
        //   WMODE 0: row index = 16 step + row group: offsets lane_soff[kt] + step * 2048;
        //   WMODE 1: row index = ((quarter * STEPS/2 + step/2) * 4 + l/8) * 2 + step%2, whose low three
        //            bits are 2 (l/8) + step%2: an odd step flips bit 0 of the chunk index (^ 16 bytes).
        const int r = lane & 7;
        const int rg = WMODE == 1 ? (lane >> 3) : lane_row_group(quarter, lane);
        const uint32_t row0 = WMODE == 1 ? (uint32_t)((quarter * (STEPS / 2) + 2 * half) * 8 + 2 * rg) : (uint32_t)(64 * half + rg);
        const uint32_t xor0 = WMODE == 1 ? (uint32_t)(2 * rg) : (uint32_t)(rg & 7);
        uint32_t lane_soff[4];
#pragma unroll
        for (int kt = 0; kt < 4; ++kt)
            lane_soff[kt] = row0 * 128u + (((uint32_t)(2 * kt + (r >> 2)) ^ xor0) << 4) + (uint32_t)(r & 3) * 4u;
        auto w_addr = [&](uint32_t stage, int st, int kt) -> uint32_t {
            if (WMODE == 1) return stage + (lane_soff[kt] ^ ((st & 1) ? 16u : 0u)) + (uint32_t)((st >> 1) * 1024 + (st & 1) * 128);
            return stage + lane_soff[kt] + (uint32_t)st * kStepBytes;
        };
        const int A = p.a_slots;
        int a_idx = group % A, w_idx = group % WS;  // ring positions of slot `sl`: sl % A, sl % WS
        uint32_t a_phase = (uint32_t)(group / A) & 1u, w_phase = (uint32_t)(group / WS) & 1u;
        bool ok = true;
        if (MAXG > 1) depend();  // a sequence is too long to gain from a head start
#ifdef TUNA_TS_PROFILE
        const long long loop_c0 = clock64();
#endif
        for (int sl = group; ok && sl < total_slots; sl += kGroups) {
            TS_PROF_BEGIN
            ok = mbar_wait_warp(w_full + 8 * w_idx, w_phase, abort_flag, p.status, 8);
            TS_PROF_END(3)
            if (!ok) break;
            uint32_t wv[4][4];  // [step][tile]: the row's 8 columns of that tile
            {
                const uint32_t src = w_stage(w_idx);
#pragma unroll
                for (int st = 0; st < 4; ++st)
#pragma unroll
                    for (int kt = 0; kt < 4; ++kt)
#ifdef TS_ABL_LDS4  // timing experiment: a quarter of the weight loads
                        if (kt > 0) wv[st][kt] = wv[st][0] + kt; else
#endif
                        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(wv[st][kt]) : "r"(w_addr(src, st, kt)));
            }
            // software pipeline: the 16 lookups of step st + 1 are in flight while step st is stored
            uint32_t v[2][16];
            auto lookups = [&](const uint32_t (&w)[4], uint32_t (&o)[16]) {
#pragma unroll
                for (int kt = 0; kt < 4; ++kt) {  // byte c of word kt = column pair c of tile kt
#ifdef TS_ABL_NOLUT  // timing experiment: no table lookups
                    o[4 * kt] = w[kt]; o[4 * kt + 1] = w[kt] + lane_key; o[4 * kt + 2] = w[kt] ^ lane_key; o[4 * kt + 3] = w[kt] >> 1;
#else
                    if (kLut256) {
                        o[4 * kt] = ts_lookup256(w[kt], lane_key, 0x7604);
                        o[4 * kt + 1] = ts_lookup256(w[kt], lane_key, 0x7614);
                        o[4 * kt + 2] = ts_lookup256(w[kt], lane_key, 0x7624);
                        o[4 * kt + 3] = ts_lookup256(w[kt], lane_key, 0x7634);
                    } else {
                        o[4 * kt] = ts_lookup(w[kt], lane_key, 0x4440);
                        o[4 * kt + 1] = ts_lookup(w[kt], lane_key, 0x4441);
                        o[4 * kt + 2] = ts_lookup(w[kt], lane_key, 0x4442);
                        o[4 * kt + 3] = ts_lookup(w[kt], lane_key, 0x4443);
                    }
#endif
                }
            };
            lookups(wv[0], v[0]);
            // All sixteen shared loads of the stage have been issued and the first have returned
            // (their data fed the lookups; they return in order): hand the stage back to the
            // producer.  The arrival is a release: it is ordered after this warp's loads.
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty + 8 * w_idx);
            if (MAXG == 1 && sl >= A && sl < A + kGroups) depend();  // the first slots whose A-slot has to be emptied first
            TS_PROF_BEGIN
            ok = mbar_wait_warp(a_empty + 8 * a_idx, a_phase ^ 1, abort_flag, p.status, 7);
            TS_PROF_END(0)
            if (!ok) break;
            tc_fence_after();
            TS_PROF_BEGIN
            const uint32_t ta = a_lane0 + (uint32_t)a_idx * kSlotCols;
#pragma unroll
            for (int st = 0; st < 4; ++st) {
                if (st < 3) lookups(wv[st + 1], v[(st + 1) & 1]);
                uint32_t (&c)[16] = v[st & 1];
#ifdef TS_ABL_NOST  // timing experiment: keep the lookups alive, skip the stores
                asm volatile("" ::"r"(c[0] ^ c[1] ^ c[2] ^ c[3] ^ c[4] ^ c[5] ^ c[6] ^ c[7] ^ c[8] ^ c[9] ^ c[10] ^ c[11] ^ c[12] ^ c[13] ^ c[14] ^ c[15]), "r"(ta));
#else
                tc_st_x16(ta + 16u * st, c);  // columns 16 st .. + 15 of this warp's half slot = the step's 32 columns of K
#endif
            }
            TS_PROF_END(1)
            TS_PROF_BEGIN
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            TS_PROF_END(2)
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full + 8 * a_idx);
            a_idx += kGroups;
            while (a_idx >= A) { a_idx -= A; a_phase ^= 1u; }
            w_idx += kGroups;
            while (w_idx >= WS) { w_idx -= WS; w_phase ^= 1u; }
        }
#ifdef TUNA_TS_PROFILE
        pg_[3] = clock64() - loop_c0;
#endif
    }

    // ------------------------------------------------------------------ common exit
    TS_PROF_MARK(2)
    tc_fence_before();
    __syncthreads();
    {
        // One copy of that code, outside any loop: half of the warps take the first tile where there is one.  A second copy in the
        // epilogue, for first tiles, or a loop over the two here took registers and instruction cache from the roles above
        // (us with the copy / the loop / as it is: 28672x4096 at 16 tokens 22.6 / 20.2 / 20.0, 57344x64 at 5 8.0 / 6.7 / 6.7,
        // 64 GEMMs of 1032x520 at 8 23.9 / 27.1 / 22.4, 47 of 4096x4096 at 16 95 / 83 / 82).
        const bool first = (s_fix[0][0] | s_fix[0][1] | s_fix[0][2] | s_fix[0][3]) != 0;
        const int e = first ? warp & 1 : 1;
        if (s_fix[e][0] | s_fix[e][1] | s_fix[e][2] | s_fix[e][3])
            finish_tile(L.g[s_tile[e][0]], s_tile[e][1], s_tile[e][2], s_tile[e][3], s_fix[e], first ? warp >> 1 : warp, first ? kTsThreads / 64 : kTsThreads / 32);
    }
    if (warp < kTsDequantWarp0) { TS_PROF_MARK(3) }
    TS_PROF_STORE
    if (warp == 0) {
        __syncwarp();  // lanes of rows past the matrix leave finish_tile early
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTsTmemCols) : "memory");
    }
}

// ------------------------------------------------------------------ host side

static int ts_steps(const tuna_config &c) { return c.k_steps == 4 ? 4 : 8; }

// Row blocks per tile and CTAs of a single GEMM, the free ones of them: the lowest estimate in microseconds.  A
// 128 x 256 slot takes 0.66 us, less where row blocks share its activations.  What comes on top depends on how the
// tiles are cut: not at all, into whole segments per tile, or anywhere (every CTA the same number of units); the partial
// sums of a cut tile cost by tokens and row blocks.  The constants are fitted to launches of 512x512 to
// 57344x8192 at 1 to 32 tokens; examples (us) at 16 tokens: 4096x4096 128 CTAs 7.8, 148 8.7; 4096x14336 two row blocks
// and 128 CTAs 13.8, two and 148 15.9, one and 148 14.5; 28672x4096 two row blocks and 148 CTAs 19.8, two and 112 21.0, one and
// 148 20.6; 57344x8192 four, two, one on 148 CTAs: 52.4, 52.1, 59.9.
static void ts_pick_split(int m, int n, int k, int sm_count, tuna_config *c)
{
    const int chunks = div_up(k, 32 * ts_steps(*c));
    const int groups = div_up(n < c->tile_tok ? n : c->tile_tok, 4);
    const int rb_wanted = c->row_blocks, ctas_wanted = c->ctas;
    double best = -1;
    for (int rb = 1; rb <= 4; rb *= 2) {
        if ((rb_wanted && rb != rb_wanted) || (!rb_wanted && rb * c->tile_tok > 64)) continue;
        const double unit_us = rb == 1 ? 0.66 : (rb == 2 ? 1.15 : 2.13);
        const long long tiles = div_up(m, kBlockRows * rb), units = tiles * chunks;
        auto consider = [&](long long ctas) {
            const long long per = (units + ctas - 1) / ctas;
            const bool whole = ctas % tiles == 0 && chunks % (ctas / tiles) == 0;
            double us = per * unit_us;
            if (whole && ctas == tiles) us = 1.15 * us + 3.1 + 0.2 * groups;  // fewer SMs draw on HBM
            else if (whole) us += 4.8 + (0.3 + 0.1 * rb) * groups + 0.17 * (ctas / tiles);
            else us += 6.3 + 0.55 * groups + 0.12 * rb * (groups - 1) + 0.17 * (ctas / tiles);
            if (best < 0 || us < best) {
                best = us;
                c->row_blocks = rb;
                c->ctas = (int)ctas;
            }
        };
        if (ctas_wanted) {
            consider(ctas_wanted);
            continue;
        }
        consider(sm_count < units ? sm_count : units);
        for (long long ctas = tiles; ctas <= sm_count && ctas <= units; ctas += tiles) consider(ctas);
    }
    if (ctas_wanted) c->ctas = ctas_wanted;
}

int gemm_tstream_normalize_config(int m, int n, int k, int sm_count, tuna_config *c)
{
    if (c->tile_tok == 0) c->tile_tok = (n <= 16) ? 16 : (n <= 32 ? 32 : (n <= 64 ? 64 : 128));
    if (c->tile_tok != 16 && c->tile_tok != 32 && c->tile_tok != 64 && c->tile_tok != 128) return TUNA_ERR_BAD_CONFIG;
    if (c->tile_tok == 128) {
        // 128-token tiles (token counts above 64 run as passes of 128): the tensor pipe needs 64 clocks
        // per MMA there, as long as the dequantisation of 16 columns, so a slot is 128 columns (8 MMAs per
        // wait and commit are enough) and a tile one row block (the accumulators take 2 x 128 columns)
        if (c->row_blocks == 0) c->row_blocks = 1;
        if (c->k_steps == 0) c->k_steps = 4;
        if (c->row_blocks != 1 || c->k_steps != 4) return TUNA_ERR_BAD_CONFIG;
    }
    if (c->row_blocks != 0 && c->row_blocks != 1 && c->row_blocks != 2 && c->row_blocks != 4) return TUNA_ERR_BAD_CONFIG;
    if (c->row_blocks != 0 && c->tile_tok <= 64 && c->row_blocks * c->tile_tok > 64) return TUNA_ERR_BAD_CONFIG;
    if (c->ctas < 0) return TUNA_ERR_BAD_CONFIG;
    if (c->ctas > sm_count) c->ctas = sm_count;
    // 256-column slots (16 MMAs per wait and commit of the issuing warp) unless one of 128 holds the whole of K:
    // 128-column slots measured 10 to 30 % slower even where they balance better over the CTAs
    if (c->k_steps == 0) c->k_steps = k > 128 ? 8 : 4;
    if (c->k_steps != 4 && c->k_steps != 8) return TUNA_ERR_BAD_CONFIG;
    if (c->row_blocks == 0 || c->ctas == 0) ts_pick_split(m, n, k, sm_count, c);
    return TUNA_OK;
}

size_t gemm_tstream_workspace_bytes(int m, int n, int k, const tuna_config &c, int sm_count)
{
    (void)n; (void)k;
    const size_t tiles = (size_t)div_up(m, kBlockRows * c.row_blocks);
    const size_t counters = (tiles * 16 + 255) / 256 * 256;  // one counter per tile and 32-row quarter
    return partial_region_bytes(sm_count) + counters;
}

template <int N_TILE, int STEPS, int MAXG, int WMODE>
static int launch_ts(const TsLaunch<MAXG> &L, int ctas, cudaStream_t stream)
{
    static bool attr_set[64] = {false};  // one-time, per device, opt-in to large dynamic shared memory
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TUNA_ERR_NO_DEVICE;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!attr_set[dev]) {
            if (cudaFuncSetAttribute(gemm_w4a16_tstream_kernel<N_TILE, STEPS, MAXG, WMODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kTsSmemDynamic) != cudaSuccess)
                return TUNA_ERR_NO_DEVICE;
            // The kernel places its lookup table at shared address 0x10000 and what lies below it right
            // after the start of dynamic shared memory, which must therefore begin within the first 4 KB
            // (static shared memory of the kernel + what the system reserves per block; the kernel checks too).
            cudaFuncAttributes fa;
            int reserved = 0;
            if (cudaFuncGetAttributes(&fa, gemm_w4a16_tstream_kernel<N_TILE, STEPS, MAXG, WMODE>) != cudaSuccess ||
                cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
                return TUNA_ERR_NO_DEVICE;
            if ((fa.sharedSizeBytes + (size_t)reserved + 1023) / 1024 * 1024 > 4096) return TUNA_ERR_NO_DEVICE;
            attr_set[dev] = true;
        }
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)ctas);
    lc.blockDim = dim3(kTsThreads);
    lc.dynamicSmemBytes = kTsSmemDynamic;
    lc.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, gemm_w4a16_tstream_kernel<N_TILE, STEPS, MAXG, WMODE>, L) == cudaSuccess ? TUNA_OK : TUNA_ERR_LAUNCH;
}

template <int MAXG>
static int launch_ts_dispatch(const TsLaunch<MAXG> &L, int tile_tok, int steps, int ctas, cudaStream_t stream)
{
    // sequences: 256-column slots and up to 64 tokens only
    switch (tile_tok * 100 + steps * 10 + L.c.w_mode) {
        case 1680: return launch_ts<16, 8, MAXG, 0>(L, ctas, stream);
        case 1681: return launch_ts<16, 8, MAXG, 1>(L, ctas, stream);
        case 3280: return launch_ts<32, 8, MAXG, 0>(L, ctas, stream);
        case 3281: return launch_ts<32, 8, MAXG, 1>(L, ctas, stream);
        case 6480: return launch_ts<64, 8, MAXG, 0>(L, ctas, stream);
        case 6481: return launch_ts<64, 8, MAXG, 1>(L, ctas, stream);
    }
    if constexpr (MAXG == 1) {
        switch (tile_tok * 100 + steps * 10 + L.c.w_mode) {
            case 1640: return launch_ts<16, 4, MAXG, 0>(L, ctas, stream);
            case 1641: return launch_ts<16, 4, MAXG, 1>(L, ctas, stream);
            case 3240: return launch_ts<32, 4, MAXG, 0>(L, ctas, stream);
            case 3241: return launch_ts<32, 4, MAXG, 1>(L, ctas, stream);
            case 6440: return launch_ts<64, 4, MAXG, 0>(L, ctas, stream);
            case 6441: return launch_ts<64, 4, MAXG, 1>(L, ctas, stream);
            case 12840: return launch_ts<128, 4, MAXG, 0>(L, ctas, stream);
            case 12841: return launch_ts<128, 4, MAXG, 1>(L, ctas, stream);
        }
    }
    return TUNA_ERR_BAD_CONFIG;
}

// Fills the table entry of one GEMM (tensor maps, geometry); `unit0` / `tile0` are where its units
// and tiles start in the launch.  Returns its unit count, or a negative status.
static long long ts_fill_gemm(TsGemm *g, const void *q, const void *x, const float *absmax, void *o, int m, int n, int k,
                              int row_blocks, int steps, int tile_tok, int unit0, int tile0, const int w_mode_wanted)
{
    int w_mode = w_mode_wanted;
    const int chunk_k = 32 * steps;
    std::memset(g, 0, sizeof(*g));
    g->absmax = absmax; g->o = (__half *)o;
    g->m = m; g->n = n; g->k = k;
    g->chunks = div_up(k, chunk_k);
    g->row_tiles = div_up(m, kBlockRows * row_blocks);
    g->unit0 = unit0;
    g->tile0 = tile0;
    if (!make_weight_map(&g->map_q, q, m, k, steps, &w_mode, &g->q3d)) return TUNA_ERR_NO_DEVICE;
    if (w_mode != w_mode_wanted) return TUNA_ERR_BAD_CONFIG;  // the driver refused the 5-D view: the caller falls back
    // activations as [n tokens] x [k] fp16; box = tile_tok tokens x 64 columns (128-byte rows, swizzled)
    if (!make_tensor_map_2d(&g->map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, (uint64_t)k, (uint64_t)n, (uint64_t)k * 2, 64,
                            (uint32_t)tile_tok, CU_TENSOR_MAP_SWIZZLE_128B))
        return TUNA_ERR_NO_DEVICE;
    return (long long)g->row_tiles * g->chunks;
}

static void ts_fill_common(TsParams *p, const tuna_config &c, int steps, void *workspace, int sm_count)
{
    p->row_blocks = c.row_blocks;
    p->acc_cols = ts_acc_cols(c.row_blocks, c.tile_tok);
    p->a_base = 2 * p->acc_cols;
    p->a_slots = ts_a_slots(p->acc_cols, steps);
    p->partials = (float *)workspace;
    p->counters = (unsigned int *)((uint8_t *)workspace + partial_region_bytes(sm_count));
}

int launch_gemm_tstream(const GemmArgs &a, const tuna_config &c)
{
    const int steps = ts_steps(c);
    TsLaunch<1> L;
    std::memset(&L.c, 0, sizeof(L.c));
    L.c.code = a.code;
    L.c.count = 1;
    L.c.status = device_status_word();
    if (!L.c.status) return TUNA_ERR_NO_DEVICE;
    if (a.workspace == nullptr || a.workspace_bytes < gemm_tstream_workspace_bytes(a.m, a.n, a.k, c, a.sm_count))
        return TUNA_ERR_WORKSPACE;
    ts_fill_common(&L.c, c, steps, a.workspace, a.sm_count);
    L.c.w_mode = weight_map_has_runs(a.m, a.k) ? 1 : 0;
    long long units = ts_fill_gemm(&L.g[0], a.q, a.x, a.absmax, a.o, a.m, a.n, a.k, c.row_blocks, steps, c.tile_tok, 0, 0, L.c.w_mode);
    if (units == TUNA_ERR_BAD_CONFIG && L.c.w_mode == 1) {  // the driver refused the 5-D view
        L.c.w_mode = 0;
        units = ts_fill_gemm(&L.g[0], a.q, a.x, a.absmax, a.o, a.m, a.n, a.k, c.row_blocks, steps, c.tile_tok, 0, 0, 0);
    }
    if (units < 0) return (int)units;
    if (units >= (1ll << 30)) return TUNA_ERR_TOO_LARGE;
    L.c.units = (int)units;
    int ctas = c.ctas;
    if (ctas > L.c.units) ctas = L.c.units;
    L.c.units_q = L.c.units / ctas;
    L.c.units_r = L.c.units % ctas;
    for (int tok0 = 0; tok0 < a.n; tok0 += c.tile_tok) {
        L.c.tok0 = tok0;
        const int st = launch_ts_dispatch(L, c.tile_tok, steps, ctas, a.stream);
        if (st != TUNA_OK) return st;
    }
    return TUNA_OK;
}

// ---- a sequence of independent GEMMs in one persistent launch

size_t gemm_tstream_sequence_workspace_bytes(const tuna_gemm_desc *d, int count, int sm_count)
{
    size_t tiles = 0;  // an upper bound: one 128-row block per tile
    for (int i = 0; i < count; ++i) tiles += (size_t)div_up(d[i].m, kBlockRows);
    return partial_region_bytes(sm_count) + (tiles * 16 + 255) / 256 * 256;
}

// Token tile and row blocks per tile of a launch whose largest token count is max_n: as many row
// blocks as the accumulator columns allow, because they share one activation stage (measured on the
// Mistral MLP sweep: 3.53 / 4.00 / 4.27 TB/s with 1 / 2 / 4 row blocks); the sequence as a whole is
// still balanced at unit granularity (64 KB).
static int ts_sequence_tile_tok(int max_n) { return max_n <= 16 ? 16 : (max_n <= 32 ? 32 : 64); }
static int ts_sequence_row_blocks(int tile_tok) { return 64 / tile_tok; }

size_t gemm_tstream_sequence_min_workspace_bytes(const tuna_gemm_desc *d, int count, int sm_count)
{
    size_t tiles = 0;
    for (int first = 0; first < count; first += kTsMaxSeq) {
        const int cnt = count - first < kTsMaxSeq ? count - first : kTsMaxSeq;
        int max_n = 1;
        for (int i = 0; i < cnt; ++i) max_n = d[first + i].n > max_n ? d[first + i].n : max_n;
        const int rows = kBlockRows * ts_sequence_row_blocks(ts_sequence_tile_tok(max_n));
        for (int i = 0; i < cnt; ++i) tiles += (size_t)div_up(d[first + i].m, rows);
    }
    return partial_region_bytes(sm_count) + (tiles * 16 + 255) / 256 * 256;
}

// Whether the sequence kernel can take these GEMMs (token counts of one pass; the rest is checked by the caller).
bool gemm_tstream_sequence_supported(const tuna_gemm_desc *d, int count)
{
    if (count < 1) return false;
    for (int i = 0; i < count; ++i)
        if (d[i].n > 64) return false;
    return true;
}

int launch_gemm_tstream_sequence(const tuna_gemm_desc *d, int count, const float *code, void *workspace, size_t workspace_bytes,
                                 int sm_count, cudaStream_t stream, const tuna_exchange *ex)
{
    if (workspace == nullptr || workspace_bytes < gemm_tstream_sequence_min_workspace_bytes(d, count, sm_count)) return TUNA_ERR_WORKSPACE;
    DeviceStatus *status = device_status_word();
    if (!status) return TUNA_ERR_NO_DEVICE;
    int tile0 = 0;  // tiles of the GEMMs launched so far: every launch has its own counters
    for (int first = 0; first < count; first += kTsMaxSeq) {
        const int cnt = count - first < kTsMaxSeq ? count - first : kTsMaxSeq;
        int max_n = 1;
        for (int i = 0; i < cnt; ++i) max_n = d[first + i].n > max_n ? d[first + i].n : max_n;
        tuna_config c;
        std::memset(&c, 0, sizeof(c));
        c.path = TUNA_PATH_TSTREAM;
        c.tile_tok = ts_sequence_tile_tok(max_n);
        c.row_blocks = ts_sequence_row_blocks(c.tile_tok);
        c.k_steps = 8;
        c.ctas = sm_count;
        static thread_local TsLaunch<kTsMaxSeq> L;  // ~20 KB: not on the stack
        std::memset(&L.c, 0, sizeof(L.c));
        L.c.code = code;
        L.c.count = cnt;
        L.c.status = status;
        ts_fill_common(&L.c, c, 8, workspace, sm_count);
        long long slab0[kTsMaxSeq];  // exchange launches: rank 0's slab of each GEMM inside a parity region
        long long region_bytes = 0;
        if (ex) {
            region_bytes = (long long)((ex->bytes - kExHeaderBytes) / 2 / 256 * 256);
            L.c.n_peers = ex->world;
            for (int j = 0; j < ex->world; ++j) L.c.peer[j] = (unsigned char *)ex->buffer[j];
            L.c.epoch = (const unsigned int *)ex->buffer[ex->rank];
            L.c.region0 = kExHeaderBytes;
            L.c.region_bytes = region_bytes;
            long long off = 0;
            for (int i = 0; i < cnt; ++i) {
                slab0[i] = -1;
                if (!(d[first + i].flags & TUNA_GEMM_PARTIAL)) continue;
                slab0[i] = off;
                off += (long long)ex->world * d[first + i].m * c.tile_tok * 2;
            }
            if (off > region_bytes) return TUNA_ERR_WORKSPACE;
        }
        // one stage layout per launch: the 256-byte-run one if every GEMM has it
        L.c.w_mode = 1;
        for (int i = 0; i < cnt; ++i)
            if (!weight_map_has_runs(d[first + i].m, d[first + i].k)) L.c.w_mode = 0;
        long long units = 0;
        const int tile0_launch = tile0;
        for (int attempt = 0; attempt < 2; ++attempt) {
            units = 0;
            tile0 = tile0_launch;
            bool refused = false;
            for (int i = 0; i < cnt; ++i) {
                const tuna_gemm_desc &g = d[first + i];
                const long long u = ts_fill_gemm(&L.g[i], g.q, g.x, (const float *)g.absmax, g.o, g.m, g.n, g.k, c.row_blocks, 8, c.tile_tok,
                                                 (int)units, tile0, L.c.w_mode);
                if (u == TUNA_ERR_BAD_CONFIG && L.c.w_mode == 1) { refused = true; break; }  // the driver refused the 5-D view
                if (u < 0) return (int)u;
                if (ex) L.g[i].slab_off = slab0[i] < 0 ? -1 : slab0[i] + (long long)ex->rank * g.m * c.tile_tok * 2;
                units += u;
                tile0 += L.g[i].row_tiles;
                if (units >= (1ll << 30)) return TUNA_ERR_TOO_LARGE;
            }
            if (!refused) break;
            L.c.w_mode = 0;
        }
        L.c.units = (int)units;
        int ctas = c.ctas;
        if (ctas > L.c.units) ctas = L.c.units;
        L.c.units_q = L.c.units / ctas;
        L.c.units_r = L.c.units % ctas;
        int st = launch_ts_dispatch(L, c.tile_tok, 8, ctas, stream);
        if (st == TUNA_OK && ex) st = launch_exchange_reduce(*ex, d + first, slab0, cnt, c.tile_tok, region_bytes, stream);
        if (st != TUNA_OK) return st;
    }
    return TUNA_OK;
}

}  // namespace tuna

#ifdef TUNA_TS_PROFILE
extern "C" int tuna_debug_ts_profile(void *host_out, size_t bytes)
{
    if (bytes > sizeof(long long) * 160 * 24 * 8) bytes = sizeof(long long) * 160 * 24 * 8;
    return (int)cudaMemcpyFromSymbol(host_out, g_ts_prof, bytes);
}
#endif
