// Depths of the rings that several dequant groups share, and the pair kernel's choice of them.  Host code without CUDA, all of it
// constexpr: the kernels assert what they rely on at compile time, and a test compiles this file by itself.
#pragma once

namespace tuna {

// Whether `groups` of dequant warps, group g taking the units g, g + groups, ..., may share a ring of `w_stages` weight stages
// and one of `a_slots` A slots.  Both are waited on by parity, which cannot tell a use of a stage from the use before the last:
//   a stage: at unit u a group needs to know that unit u - w_stages has landed.  Either that was its own unit, or the MMAs have
//   consumed it, which holds for all units up to u - groups - a_slots since the group's last wait for a slot;
//   a slot: likewise unit u - 2 a_slots has to be consumed, which that wait says where a_slots >= groups.
// Otherwise a group that is ahead passes its wait a phase early, reads stale bytes and hands back a stage whose copy is still
// in flight; the producer's next copy then arrives in a phase that expects none, which is undefined (a launch failure at best).
constexpr bool rings_shareable(int w_stages, int a_slots, int groups)
{
    return a_slots >= groups && w_stages >= groups && (w_stages % groups == 0 || w_stages >= a_slots + groups);
}

constexpr int kPairTmemCols = 512;
constexpr int kPairLutBytes = 256 * 128;    // byte -> half2 table: 256 entries, one copy per bank
constexpr int kPairLutWide = 4096, kPairLutWideBytes = 256 * 256;  // its place and size with 256 bytes per entry (pair_lookup)
constexpr int kPairMaxStages = 8;           // unit stages: activations in shared memory + an A slot in tensor memory
constexpr int kPairMaxWStages = 8;
constexpr int kPairSmemDynamic = 226 * 1024;
constexpr int kPairSmemStart = 2048;        // where in the shared window dynamic shared memory begins (launch_pair checks it)

// The most dequant warps of a tile, 8 or 16: 16 as long as the tensor pipe needs fewer clocks per step than the table lookups and
// what goes with them; with them comes the table that one instruction per lookup addresses (pair_lookup), which leaves too little shared
// memory for the stages of wider tiles.  Graph replay, us, 8 / 16 warps / 16 and the wide table: 11000x4104 at 43
// tokens 13.5 / 12.6 / 12.5, 6144x4096 at 256 (96-token tiles) 15.5 / 14.5 / 14.1, 57344x8192 at 64 81 / 70 / 70, 8192x8192 at 192
// 27.5 / 25.5 / 24.3; 57344x8192 at 256 (256-token tiles) 166 / 167, 28672x4096 at 224 47 / 46.  Fewer on short tiles (pair_split).
constexpr int pair_dequant_warps(int tile_tok) { return tile_tok <= 192 ? 16 : 8; }

constexpr int pair_kc(int tile_tok) { return tile_tok > 128 ? 64 : 128; }

struct PairPlan {
    int tile_tok, kc;
    int stages, w_stages;  // unit stages, weight stages
    int nd;                // accumulator buffers
    bool fits;             // shared memory holds it
};

// of tiles of `tile_tok` tokens with stages of `kc` columns and `warps` dequant warps
constexpr PairPlan pair_plan(int tile_tok, int kc, int warps)
{
    PairPlan l = {tile_tok, kc, 0, kPairMaxWStages, 1, false};
    const int slot = kc / 2, w_bytes = 128 * kc / 2;
    // two accumulator buffers (the epilogue of one tile overlaps the MMAs of the next) where they leave four A slots
    if (2 * tile_tok + 4 * slot <= kPairTmemCols) l.nd = 2;
    l.stages = (kPairTmemCols - l.nd * tile_tok) / slot;
    if (l.stages > kPairMaxStages) l.stages = kPairMaxStages;
    const int groups = warps / 4;
    const int lut = groups == 4 ? kPairLutWide - kPairSmemStart + kPairLutWideBytes : kPairLutBytes;
    const int beside = kPairSmemDynamic - lut - tile_tok * 256;  // what the table and the staging tile leave
    while (l.stages > 4 && l.stages * tile_tok * kc + l.w_stages * w_bytes > beside) --l.stages;
    while (l.w_stages > 4 && l.stages * tile_tok * kc + l.w_stages * w_bytes > beside) --l.w_stages;
    if (!rings_shareable(l.w_stages, l.stages, groups)) l.w_stages -= l.w_stages % groups;
    l.fits = l.stages * tile_tok * kc + l.w_stages * w_bytes <= beside && rings_shareable(l.w_stages, l.stages, groups);
    return l;
}
constexpr PairPlan pair_plan(int tile_tok, int kc) { return pair_plan(tile_tok, kc, pair_dequant_warps(tile_tok)); }

constexpr bool pair_plans_fit()
{
    for (int t = 32; t <= 256; t += 32)
        for (int warps = 8; warps <= pair_dequant_warps(t); warps += 8)
            if (!pair_plan(t, pair_kc(t), warps).fits) return false;
    return true;
}
static_assert(pair_plans_fit(), "every token tile has its rings");

}  // namespace tuna
