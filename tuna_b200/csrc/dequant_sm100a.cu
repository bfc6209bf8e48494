// Standalone dequantisation kernel for sm_100a: packed 4-bit codes -> fp16.
//
// Replaces the reference's dequantize_4bit (kernel.cu:3158-3241) and is
// bit-exact to it: out = (half)(code[nibble] * absmax[row]) with the multiply
// in fp32 (kernel.cu:3223-3228).  HBM-bound: reads m*k/2 bytes, writes 2*m*k.
//
// Mapping: one warp owns one 8-row group and walks along K.  A lane reads 16 packed bytes (half of
// an 8x8 tile: 4 rows x 8 columns) with one 128-bit load, turns each row's word into fp16 with the
// row's table in registers (CodePlanes; the tables are built once per warp with the fp32 multiply)
// and writes four 16-byte row segments.  Across a warp each of those stores covers 256 contiguous
// bytes of two rows.
// HBM bounds it: a copy of as many bytes in all (294 MB at 28672x4096) takes 45 us at the 6.55 TB/s a copy reaches.  28672x4096: 58.9 -> 49.5 us (5.93 TB/s) against lookups in a per-row table in shared memory, one
// load in flight.
#include <algorithm>
#include "common.cuh"
#include "launchers.h"

namespace tuna {

constexpr int kDqWarps = 8;
constexpr int kDqUnroll = 2;     // loads in flight per lane
constexpr int kDqCtasPerSm = 3;  // 80 registers: four tables of 8 and two passes of data
constexpr int kDqWaves = 6;      // 28672x4096: 56.5 us with one wave of longer-lived warps, 53.4 with 4, 49.5 with 6, 49.3 with 8

__global__ void __launch_bounds__(kDqWarps * 32, kDqCtasPerSm)
dequant_w4_kernel(const uint8_t *__restrict__ q, const float *__restrict__ absmax,
                  const float *__restrict__ code, __half *__restrict__ out, int k, int per_warp, int extra)
{
    __shared__ __align__(16) __half lut[kDqWarps][8][kCodeSize];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_kt = k >> 3;
    const int half_sel = lane & 1;  // which 4 rows of the tile this lane holds
    constexpr int kPassTiles = 16 * kDqUnroll;
    const int passes = (n_kt + kPassTiles - 1) / kPassTiles;  // of a row group
    // this warp's contiguous range of (row group, pass)
    const int w = blockIdx.x * kDqWarps + warp;
    int it = w * per_warp + min(w, extra);
    const int it_end = it + per_warp + (w < extra ? 1 : 0);

    while (it < it_end) {
        const int rg = it / passes, p0 = it - rg * passes;
        const int n_pass = min(passes - p0, it_end - it);
        it += n_pass;
        const int kt_end = min(n_kt, (p0 + n_pass) * kPassTiles);
        const uint8_t *src = q + (size_t)rg * row_group_bytes(k) + half_sel * 16;
        __half *dst_rows = out + (size_t)(rg * 8 + half_sel * 4) * k;
        int kt = p0 * kPassTiles + (lane >> 1);
        uint4 v[kDqUnroll];
        auto load = [&](int kt0) {
#pragma unroll
            for (int u = 0; u < kDqUnroll; ++u) v[u] = ldg_stream_pred(src + (size_t)(kt0 + 16 * u) * 32, kt0 + 16 * u < kt_end);
        };
        load(kt);  // in flight while the tables are built

        // 128 table entries per warp, 4 per lane: row = e / 16, nibble = e % 16
        __syncwarp();  // the previous row group's tables have been read
        for (int e = lane; e < 8 * kCodeSize; e += 32)
            lut[warp][e >> 4][e & 15] = __float2half_rn(code[e & 15] * absmax[rg * 8 + (e >> 4)]);
        __syncwarp();
        CodePlanes row[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 *t = reinterpret_cast<const uint4 *>(&lut[warp][half_sel * 4 + i][0]);
            const uint4 a = t[0], b = t[1];
            const uint32_t e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            row[i].init(e);
        }

        for (; kt < kt_end; kt += kPassTiles) {
            uint4 c[kDqUnroll];
#pragma unroll
            for (int u = 0; u < kDqUnroll; ++u) c[u] = v[u];
            load(kt + kPassTiles);
#pragma unroll
            for (int u = 0; u < kDqUnroll; ++u) {
                if (kt + 16 * u >= kt_end) break;
                const uint32_t words[4] = {c[u].x, c[u].y, c[u].z, c[u].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {  // row 4*half_sel + i, columns 8kt .. 8kt+7
                    uint32_t o[4];
                    row[i].convert(words[i], o);
                    *reinterpret_cast<uint4 *>(dst_rows + (size_t)i * k + (size_t)(kt + 16 * u) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            }
        }
    }
}

// Small matrices and narrow rows, where a warp has hardly more to do than to build its tables: they stay in shared memory,
// one entry looked up per weight, and a warp's share is as little as 128 columns of one row group.
__global__ void __launch_bounds__(kDqWarps * 32)
dequant_lookup_kernel(const uint8_t *__restrict__ q, const float *__restrict__ absmax, const float *__restrict__ code,
                      __half *__restrict__ out, int m, int k, int tiles_per_warp)
{
    __shared__ __align__(16) __half lut[kDqWarps][8][kCodeSize];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rg = blockIdx.x * kDqWarps + warp;
    if (rg >= (m >> 3)) return;
    for (int e = lane; e < 8 * kCodeSize; e += 32)
        lut[warp][e >> 4][e & 15] = __float2half_rn(code[e & 15] * absmax[rg * 8 + (e >> 4)]);
    __syncwarp();

    const int kt_end = min(k >> 3, ((int)blockIdx.y + 1) * tiles_per_warp);
    const int half_sel = lane & 1;  // which 4 rows of the tile this lane holds
    const uint8_t *src = q + (size_t)rg * row_group_bytes(k) + half_sel * 16;
    const __half(*table)[kCodeSize] = &lut[warp][half_sel * 4];
    __half *dst_rows = out + (size_t)(rg * 8 + half_sel * 4) * k;
    for (int kt = (int)blockIdx.y * tiles_per_warp + (lane >> 1); kt < kt_end; kt += 16) {
        const uint4 v = ldg_stream_u4(src + (size_t)kt * 32);
        const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t o[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {  // even column: high nibble
                const uint32_t byte = (words[i] >> (8 * b)) & 0xffu;
                o[b] = (uint32_t)__half_as_ushort(table[i][byte >> 4]) | ((uint32_t)__half_as_ushort(table[i][byte & 15]) << 16);
            }
            *reinterpret_cast<uint4 *>(dst_rows + (size_t)i * k + (size_t)kt * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// Measured (graph replay, us, lookups in shared memory / tables in registers): 57344x8 4.0 / 5.5, 57344x128 5.2 / 5.6, 57344x160 7.4 / 7.1;
// 8x4096 2.1 / 2.6, 512x512 2.3 / 2.5, 4096x256 2.3 / 2.5, 4096x384 2.8 / 2.5, 6144x160 2.7 / 2.5.
static bool dequant_by_lookup(int m, int k) { return k <= 128 || (m <= 4096 && (long long)m * k <= 1 << 20); }

cudaError_t launch_dequant(const void *q, const void *absmax, const void *code, void *o, int m,
                           int k, int sm_count, cudaStream_t stream)
{
    if (dequant_by_lookup(m, k)) {
        const int tiles = k / 8, gx = div_up(m / 8, kDqWarps);
        // eight CTAs per SM if the columns give as many, a whole number of warp passes (16 tiles) each
        const int wanted = std::max(1, std::min(div_up(sm_count * 8, gx), div_up(tiles, 16)));
        const int per_warp = div_up(div_up(tiles, wanted), 16) * 16;
        dequant_lookup_kernel<<<dim3(gx, div_up(tiles, per_warp)), kDqWarps * 32, 0, stream>>>(
            (const uint8_t *)q, (const float *)absmax, (const float *)code, (__half *)o, m, k, per_warp);
        return cudaGetLastError();
    }
    const int items = (m / 8) * div_up(k / 8, 16 * kDqUnroll);  // below 2^31: m * k <= 2^41
    const int grid = std::min(sm_count * kDqCtasPerSm * kDqWaves, div_up(items, kDqWarps));
    const int warps = grid * kDqWarps;
    dequant_w4_kernel<<<grid, kDqWarps * 32, 0, stream>>>((const uint8_t *)q, (const float *)absmax, (const float *)code, (__half *)o, k,
                                                          items / warps, items % warps);
    return cudaGetLastError();
}

}  // namespace tuna
