// Row-wise absmax quantizer + packer on the device: the reference's
// quantize_blockwise_dynamic_4bit(w, block_size=k, preprocess=True) (test.py:7-68), which the
// reference runs as a chain of torch kernels (clone, abs, max, divide, a [16, chunk] distance
// tensor, argmin, reshape/permute, multiply-add):
//   absmax[r]  = max_c |w[r, c]|
//   code(r, c) = argmin_i | fp32(w[r,c]) / absmax[r] - code[i] |   (first index on ties, as
//      torch.argmin; the quotient is an fp32 division because the reference converts absmax to
//      fp32 before dividing, test.py:16,42), packed into the [m/8, k/8, 32] tile layout
//      (test.py:55-65): one thread produces the 32-bit word that holds its row's 8 columns of a
//      tile, a warp writes 128 contiguous bytes.
//
// quantize_rows_kernel does it in one pass over memory.  A CTA stages its share of an 8-row group
// (up to 4096 columns, 64 KB: three CTAs per SM keep ~190 KB of copies in flight) in shared memory
// with one cp.async.bulk per row, reduces the row maxima from there - row groups wider than one
// share belong to a cluster of up to 8 CTAs that exchange theirs through distributed shared memory -
// and quantizes from there: 2 bytes read and half a byte written per weight.
//
// The division and the 16 distances per weight are ~70 instructions and were what bounded the
// two-pass version (435 us on 28672x4096, 0.68 TB/s); the floor of the traffic is 46 us, i.e. ~14
// instructions per weight.  They go like this: for a fixed row the code is a step function of the
// fp16 weight (fp32 division and subtraction round monotonically), so the row's 15 step positions
// are found first, as exact fp16 thresholds, by evaluating the reference's own expression around
// (code[i] + code[i+1]) / 2 * absmax.  Then one packed half FMA maps two weights to buckets
// 1..127 (monotonically, whatever its rounding), and the row's table says for a bucket which
// threshold lies in it, if any, and the codes below and above: one lookup and one exact fp16
// comparison per weight.  The table is exact because a threshold is filed under the bucket the same
// FMA gives it.  Rows it cannot represent (two thresholds in one bucket, a zero, tiny or
// non-finite absmax, codes that are equal, closer than fp32 can separate, or not finite) take the
// literal expression.  28672x4096: 436 -> 67 us (0.68 -> 4.4 TB/s of its 294 MB).
#include <cuda_fp16.h>
#include <mutex>
#include "common.cuh"
#include "launchers.h"
#include "sm100_ptx.cuh"

namespace tuna {

constexpr int kQuantThreads = 256;
constexpr int kQuantShareCols = 4096;      // columns of a CTA's share a cluster is chosen for
constexpr int kQuantMaxShareCols = 13936;  // what shared memory holds at one CTA per SM (beside the tables)
constexpr int kQuantMaxCluster = 8;
constexpr int kBuckets = 128;
// The "NormalFloat4" levels the reference's quantizer emits (test.py:19-40); codebooks.py has the same list.
__constant__ float kNf4[16] = {-1.0f, -0.6961928009986877f, -0.5250730514526367f, -0.39491748809814453f, -0.28444138169288635f,
                               -0.18477343022823334f, -0.09105003625154495f, 0.0f, 0.07958029955625534f, 0.16093020141124725f,
                               0.24611230194568634f, 0.33791524171829224f, 0.44070982933044434f, 0.5626170039176941f,
                               0.7229568362236023f, 1.0f};

// The rows' tables lie side by side, bucket by bucket, each row's twice: lane l of a warp (row l % 8) looks up in column
// l % 16, so that two lanes share a bank at most (rows' tables one after another, where random
// lookups meet three or four at a time: 84 us against 80 on 28672x4096; 64 buckets with a column per bank, and the code that
// chooses between the two, 84: the lookups are not what bounds it any more, the phases' instructions are).
constexpr int kTableCols = 16;
constexpr int kThrStride = 17;  // words of a row's thresholds: the eight rows' lie in different banks

// The reference's expression for one weight.
__device__ __forceinline__ uint32_t nearest_code(float w, float scale, const float *cb)
{
    const float x = __fdiv_rn(w, scale);
    float best = fabsf(x - cb[0]);
    uint32_t idx = 0;
#pragma unroll
    for (int c = 1; c < 16; ++c) {
        const float d = fabsf(x - cb[c]);
        if (d < best) { best = d; idx = c; }  // strict: ties and NaN keep the lower index
    }
    return idx;
}

// fp16 bit patterns in the order of their values (-inf .. inf -> ascending integers), and back.
__device__ __forceinline__ int half_rank(uint32_t h) { return (h & 0x8000u) ? 0x8000 - (int)h : (int)h; }
__device__ __forceinline__ uint32_t half_of_rank(int r) { return r < 0 ? (uint32_t)(0x8000 - r) : (uint32_t)r; }

__device__ __forceinline__ uint32_t habs2_bits(uint32_t v) { return v & 0x7fff7fffu; }
__device__ __forceinline__ uint32_t hmax2_nan_bits(uint32_t a, uint32_t b)
{
    const __half2 r = __hmax2_nan(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}

// cluster = gridDim.x / (m / 8) CTAs per 8-row group, `share` columns each (the last one the rest).
// code == nullptr: the NF4 levels, which are also written to code_out (the caller needs no copy of its own).
__global__ void __launch_bounds__(kQuantThreads) quantize_rows_kernel(const __half *__restrict__ w, const float *__restrict__ code,
                                                                      float *__restrict__ code_out, uint8_t *__restrict__ q, float *__restrict__ absmax,
                                                                      DeviceStatus *status, int k, int share, int cluster)
{
    extern __shared__ __align__(16) uint8_t stage[];  // [8 rows][2 share + 16 bytes]: the 16 bytes separate the rows' banks
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_abort;
    __shared__ float s_code[16], s_sorted[16];
    __shared__ uint32_t s_sorted_idx[16];
    __shared__ uint32_t s_warp_max[kQuantThreads / 32][8];
    __shared__ uint32_t s_row_max[8];  // fp16 bits; read by the other CTAs of the cluster
    __shared__ float s_scale[8];
    __shared__ uint32_t s_bucket_scale[8];  // half2
    __shared__ uint32_t s_thr[8][kThrStride];  // fp16 bits of threshold i | its bucket << 16
    __shared__ int s_row_ok[8];
    __shared__ uint32_t s_table[kBuckets * kTableCols];  // fp16 threshold | codes (below << 4 | (below ^ above)) << 16

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rg = blockIdx.x / cluster, rank = blockIdx.x - rg * cluster;
    const int col0 = rank * share, cols = min(share, k - col0);
    const int tiles = cols >> 3;
    const uint32_t pitch = 2u * (uint32_t)share + 16u;
    const uint32_t stage0 = smem_u32(stage), bar = smem_u32(&s_bar);

    if (tid == 0) {
        s_abort = 0;
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(bar, 16u * (uint32_t)cols);
        for (int r = 0; r < 8; ++r)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(stage0 + r * pitch),
                         "l"(w + ((size_t)rg * 8 + r) * k + col0), "r"(2u * (uint32_t)cols), "r"(bar)
                         : "memory");
    }
    if (tid < 16) {
        const float c = code ? code[tid] : kNf4[tid];
        s_code[tid] = c;
        s_sorted[tid] = __int_as_float(0x7fffffff);  // stays NaN, and every row literal, where a NaN code leaves a gap in the order
        s_sorted_idx[tid] = 0;
        if (code_out && blockIdx.x == 0) code_out[tid] = c;
    }
    if (tid < 8) s_row_ok[tid] = 1;
    __syncthreads();
    if (tid < 16) {  // the codes in ascending order (equal ones by index)
        const float c = s_code[tid];
        int pos = 0;
        for (int j = 0; j < 16; ++j) pos += (s_code[j] < c || (s_code[j] == c && j < tid)) ? 1 : 0;
        s_sorted[pos] = c;
        s_sorted_idx[pos] = (uint32_t)tid;
    }
    bool landed = mbar_wait(bar, 0, &s_abort, status, 60);
    __syncthreads();

    // ---- row maxima (NaN propagates like torch.max)
    const int r = lane & 7, tl = lane >> 3;  // row of the group, tile among the warp's four
    const uint32_t row_addr = stage0 + (uint32_t)r * pitch;
    auto load8 = [&](int kt) {
        uint4 v;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(row_addr + (uint32_t)kt * 16u));
        return v;
    };
    constexpr int kTilesPerPass = 4 * (kQuantThreads / 32);
    {
        uint32_t best = 0;
        if (landed)
            for (int kt = 4 * warp + tl; kt < tiles; kt += kTilesPerPass) {
                const uint4 v = load8(kt);
                best = hmax2_nan_bits(hmax2_nan_bits(best, habs2_bits(v.x)), hmax2_nan_bits(habs2_bits(v.y), hmax2_nan_bits(habs2_bits(v.z), habs2_bits(v.w))));
            }
        best = hmax2_nan_bits(best, __byte_perm(best, 0, 0x1032));
        best = hmax2_nan_bits(best, __shfl_xor_sync(0xffffffffu, best, 8));
        best = hmax2_nan_bits(best, __shfl_xor_sync(0xffffffffu, best, 16));
        if (lane < 8) s_warp_max[warp][lane] = best & 0xffffu;
    }
    __syncthreads();
    if (tid < 8) {
        uint32_t best = 0;
        for (int i = 0; i < kQuantThreads / 32; ++i) best = hmax2_nan_bits(best, s_warp_max[i][tid]);
        s_row_max[tid] = best;
    }
    if (cluster > 1) {
        __syncwarp();  // the aligned barriers want converged warps, and lanes take different ways before each of them
        asm volatile("barrier.cluster.arrive.aligned;\n barrier.cluster.wait.aligned;" ::: "memory");
        if (tid < 8) {
            uint32_t best = 0;
            for (int c = 0; c < cluster; ++c) {
                uint32_t remote, v;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(&s_row_max[tid])), "r"(c));
                asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
                best = hmax2_nan_bits(best, v);
            }
            s_warp_max[0][tid] = best;  // not s_row_max: the other CTAs may still be reading it
        }
        // the matching wait stands at the end: no CTA leaves while another may read its maxima
        __syncwarp();
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    } else if (tid < 8) {
        s_warp_max[0][tid] = s_row_max[tid];
    }
    if (tid < 8) {
        const float s = __half2float(__ushort_as_half((unsigned short)s_warp_max[0][tid]));
        s_scale[tid] = s;
        if (rank == 0 && landed) absmax[(size_t)rg * 8 + tid] = s;
        // weights map to buckets 64 + round(w * 63 / absmax): 1 .. 127
        const __half b = __float2half_rn(63.0f / s);
        const uint32_t hb = (uint32_t)__half_as_ushort(b);
        s_bucket_scale[tid] = hb | (hb << 16);
        if (!(s > 0.f) || !(s < 65536.f) || (hb & 0x7c00u) == 0x7c00u) s_row_ok[tid] = 0;
    }
    __syncthreads();

    // The bucket of a weight: its low byte after one FMA into [1024, 2048), where an fp16 step is 1.
    const __half2 kMagic = __floats2half2_rn(1024.f + 64.f, 1024.f + 64.f);
    auto buckets2 = [&](uint32_t w2, uint32_t scale2) {
        const __half2 h = __hfma2(*reinterpret_cast<const __half2 *>(&w2), *reinterpret_cast<const __half2 *>(&scale2), kMagic);
        return *reinterpret_cast<const uint32_t *>(&h);
    };

    // ---- thresholds: thread (row, i) finds the smallest fp16 weight whose code lies above sorted code i
    if (tid < 128) {
        const int row = tid & 7, i = tid >> 3;
        uint32_t thr = 0x7fffu, bkt = 255u;  // a NaN no weight compares >= to, in no bucket
        if (i < 15 && s_row_ok[row]) {
            const float s = s_scale[row], a = s_sorted[i], b = s_sorted[i + 1];
            const bool tie_up = s_sorted_idx[i + 1] < s_sorted_idx[i];  // equal distances keep the lower original index
            // fp32 distances up to 1 + |code| carry an error of half an ulp: codes closer than this might tie at a distance
            if (!(b - a > 1e-5f * (1.f + fmaxf(fabsf(a), fabsf(b)))) || !(b - a < 1e30f)) {
                s_row_ok[row] = 0;
            } else {
                auto above = [&](int rk) {
                    const float x = __fdiv_rn(__half2float(__ushort_as_half((unsigned short)half_of_rank(rk))), s);
                    const float da = fabsf(x - a), db = fabsf(x - b);
                    return db < da || (tie_up && db == da);
                };
                // bracket (lo: not above, hi: above), growing from the midpoint, then bisect
                constexpr int kLowest = -0x7bff, kHighest = 0x7bff;  // finite fp16
                int g = half_rank(__half_as_ushort(__float2half_rn(0.5f * (a + b) * s)));
                g = min(max(g, kLowest), kHighest);
                int lo, hi, step = 1;
                if (above(g)) {
                    hi = g;
                    lo = g - 1;
                    while (lo >= kLowest && above(lo)) { hi = lo; lo -= step; step *= 2; }
                    lo = max(lo, kLowest - 1);
                } else {
                    lo = g;
                    hi = g + 1;
                    while (hi <= kHighest && !above(hi)) { lo = hi; hi += step; step *= 2; }
                    hi = min(hi, kHighest + 1);
                }
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;  // arithmetic shift: floor
                    if (above(mid)) hi = mid; else lo = mid;
                }
                const float t = hi > kHighest ? 1e30f : __half2float(__ushort_as_half((unsigned short)half_of_rank(hi)));
                if (t > s) {
                    // above every weight of the row
                } else if (t <= -s) {
                    thr = (uint32_t)__half_as_ushort(__float2half_rn(-s));  // at or below every weight: "bucket 0" lies before all
                    bkt = 0u;
                } else {
                    thr = half_of_rank(hi);
                    bkt = buckets2(thr, s_bucket_scale[row]) & 0xffu;
                }
            }
        }
        s_thr[row][i] = thr | (bkt << 16);
    }
    __syncthreads();

    // ---- the rows' tables: thread (row, i, half) fills every other bucket after threshold i - 1's up to threshold i's
    // (filling by bucket, which counts the thresholds below each, was a quarter of the kernel's instructions: 28672x4096 75.2 us, so 67.3)
    {
        const int row = tid & 7, i = (tid >> 3) & 15, half = tid >> 7;
        const uint32_t t = s_thr[row][i], bkt = t >> 16, prev = i > 0 ? s_thr[row][i - 1] >> 16 : 0u;
        const uint32_t lo = s_sorted_idx[i], hi = s_sorted_idx[min(i + 1, 15)];
        const uint32_t codes = ((lo << 4) | (lo ^ hi)) << 16;
        for (uint32_t b = prev + 1 + half; b <= min(bkt, (uint32_t)kBuckets - 1); b += 2) {
            const uint32_t e = (b == bkt ? t & 0xffffu : 0x7fffu) | codes;
            s_table[b * kTableCols + row] = e;
            s_table[b * kTableCols + 8 + row] = e;
        }
        if (i > 0 && bkt == prev && bkt > 0 && bkt < kBuckets) s_row_ok[row] = 0;  // two thresholds in one bucket
    }
    __syncthreads();

    // ---- codes: one 32-bit word (the row's 8 columns of a tile) per thread and step
    if (landed) {
        uint8_t *dst = q + (size_t)rg * row_group_bytes(k) + (size_t)col0 * 4 + r * 4;
        if (s_row_ok[r]) {
            const uint32_t scale2 = s_bucket_scale[r];
            const uint32_t table = smem_u32(&s_table[lane & (kTableCols - 1)]);
            for (int kt = 4 * warp + tl; kt < tiles; kt += kTilesPerPass) {
                const uint4 v = load8(kt);
                const uint32_t u[4] = {v.x, v.y, v.z, v.w};
                uint32_t e0[4], e1[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t b2 = buckets2(u[i], scale2);
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e0[i]) : "r"(table + 4u * kTableCols * (b2 & 0xffu)));
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e1[i]) : "r"(table + 4u * kTableCols * __byte_perm(b2, 0, 0x4442)));
                }
                // two pairs at a time, a byte per weight: the code below in the high nibble, the difference to the one above in the low one
                uint32_t half_word[2];
#pragma unroll
                for (int i = 0; i < 4; i += 2) {
                    uint32_t c[2], m[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t t2 = __byte_perm(e0[i + j], e1[i + j], 0x5410);
                        m[j] = __hge2_mask(*reinterpret_cast<const __half2 *>(&u[i + j]), *reinterpret_cast<const __half2 *>(&t2));
                        c[j] = __byte_perm(e0[i + j], e1[i + j], 0x0062);
                    }
                    const uint32_t codes = __byte_perm(c[0], c[1], 0x5410), above = __byte_perm(m[0], m[1], 0x6420);
                    const uint32_t sel = codes ^ ((codes << 4) & above);                    // the code in each high nibble
                    half_word[i >> 1] = (sel & 0x00f000f0u) | ((sel >> 12) & 0x000f000fu);  // even column high: bytes 0 and 2
                }
                const uint32_t word = __byte_perm(half_word[0], half_word[1], 0x6420);
                *reinterpret_cast<uint32_t *>(dst + (size_t)kt * 32) = word;
            }
        } else {
            const float scale = s_scale[r];
            for (int kt = 4 * warp + tl; kt < tiles; kt += kTilesPerPass) {
                const uint4 v = load8(kt);
                const uint32_t u[4] = {v.x, v.y, v.z, v.w};
                uint32_t word = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half2 h = *reinterpret_cast<const __half2 *>(&u[i]);
                    word |= ((nearest_code(__low2float(h), scale, s_code) << 4) | nearest_code(__high2float(h), scale, s_code)) << (8 * i);
                }
                *reinterpret_cast<uint32_t *>(dst + (size_t)kt * 32) = word;
            }
        }
    }
    if (cluster > 1) {
        __syncwarp();
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    }
}

// ---- rows too wide for a cluster's shared memory (k > 111488), and many narrow rows (quantize_in_two_passes): two passes
// over memory, the literal expression

__global__ void __launch_bounds__(256) row_absmax_kernel(const __half *__restrict__ w, float *__restrict__ absmax, int m, int k)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int chunks = k >> 3;  // 16-byte pieces of a row
    for (int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < m; row += warps) {
        const uint4 *src = reinterpret_cast<const uint4 *>(w + (size_t)row * k);
        float best = 0.f;
        for (int c = lane; c < chunks; c += 32) {
            const uint4 v = ldg_stream_u4(src + c);
            const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __half2 h = *reinterpret_cast<const __half2 *>(&u[i]);
                // NaN propagates like torch.max: fmaxf would drop it
                const float a = fabsf(__low2float(h)), b = fabsf(__high2float(h));
                best = (a > best || a != a) ? a : best;
                best = (b > best || b != b) ? b : best;
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float o = __shfl_xor_sync(0xffffffffu, best, off);
            best = (o > best || o != o) ? o : best;
        }
        if (lane == 0) absmax[row] = best;
    }
}

__global__ void __launch_bounds__(256) quantize_pack_kernel(const __half *__restrict__ w, const float *__restrict__ code,
                                                            float *__restrict__ code_out, const float *__restrict__ absmax, uint8_t *__restrict__ q,
                                                            int m, int k)
{
    __shared__ float s_code[16];
    if (threadIdx.x < 16) {
        s_code[threadIdx.x] = code ? code[threadIdx.x] : kNf4[threadIdx.x];
        if (code_out && blockIdx.x == 0) code_out[threadIdx.x] = s_code[threadIdx.x];
    }
    __syncthreads();
    float cb[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) cb[i] = s_code[i];

    const int lane = threadIdx.x & 31;
    const int r = lane & 7, tl = lane >> 3;  // row inside the 8-row group, tile among the warp's four
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const int tiles_k = k >> 3;
    const int quads = (tiles_k + 3) >> 2;  // groups of four tiles along K
    const long long items = (long long)(m >> 3) * quads;
    for (long long it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < items; it += warps) {
        const int rg = (int)(it / quads);
        const int kt = (int)(it - (long long)rg * quads) * 4 + tl;
        if (kt >= tiles_k) continue;
        const int row = rg * 8 + r;
        const float scale = absmax[row];
        const uint4 v = ldg_stream_u4(reinterpret_cast<const uint4 *>(w + (size_t)row * k + (size_t)kt * 8));
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        uint32_t word = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 h = *reinterpret_cast<const __half2 *>(&u[i]);
            // nearest_code of both columns side by side: 32 registers; by two calls of it 41 (1024x120000: 503 us against 609)
            const float x[2] = {__fdiv_rn(__low2float(h), scale), __fdiv_rn(__high2float(h), scale)};
            uint32_t nib[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float best = fabsf(x[e] - cb[0]);
                uint32_t idx = 0;
#pragma unroll
                for (int c = 1; c < 16; ++c) {
                    const float d = fabsf(x[e] - cb[c]);
                    if (d < best) { best = d; idx = c; }
                }
                nib[e] = idx;
            }
            word |= ((nib[0] << 4) | nib[1]) << (8 * i);  // even column in the high nibble
        }
        *reinterpret_cast<uint32_t *>(q + (size_t)rg * row_group_bytes(k) + (size_t)kt * 32 + r * 4) = word;
    }
}

// Whether two passes are the faster way.  A CTA of the single pass spends ~1.8 us on its row group before the first code,
// whatever the width; on many very narrow rows the literal expression is done with them sooner.  The estimates (us) are fitted to 8 to
// 229376 rows of 8 to 512 columns; two passes / one: 57344x8 17.4 / 30.4, 57344x64 22.0 / 30.8, 57344x128 33.2 / 31.5, 8192x64
// 6.9 / 6.4, 8192x128 8.6 / 6.5, 4096x64 5.7 / 3.9.
static bool quantize_in_two_passes(int m, int k, int sm_count)
{
    const double groups_per_sm = (m / 8) / (double)sm_count;
    return 4.6 + groups_per_sm * (0.15 + 0.00355 * k) < 2.2 + groups_per_sm / 3 * (1.72 + 0.001 * k);
}

cudaError_t launch_quantize(const void *w, const void *code, void *code_out, void *q, void *absmax, int m, int k, int sm_count,
                            cudaStream_t stream)
{
    const int want = div_up(k, kQuantShareCols);
    const int cluster0 = want < kQuantMaxCluster ? want : kQuantMaxCluster;
    const int share = div_up(k / 8, cluster0) * 8;
    if (share > kQuantMaxShareCols || quantize_in_two_passes(m, k, sm_count)) {
        const int blocks = sm_count * 8;
        row_absmax_kernel<<<blocks, 256, 0, stream>>>((const __half *)w, (float *)absmax, m, k);
        quantize_pack_kernel<<<blocks, 256, 0, stream>>>((const __half *)w, (const float *)code, (float *)code_out,
                                                         (const float *)absmax, (uint8_t *)q, m, k);
        return cudaGetLastError();
    }
    const int cluster = div_up(k, share);
    DeviceStatus *status = device_status_word();
    if (!status) return cudaErrorInitializationError;
    static bool attr_set[64] = {false};  // one-time, per device, opt-in to large dynamic shared memory
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!attr_set[dev]) {
            e = cudaFuncSetAttribute(quantize_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * (2 * kQuantMaxShareCols + 16));
            if (e != cudaSuccess) return e;
            attr_set[dev] = true;
        }
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(m / 8) * (unsigned)cluster);
    lc.blockDim = dim3(kQuantThreads);
    lc.dynamicSmemBytes = 8 * (2 * (size_t)share + 16);
    lc.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = cluster > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&lc, quantize_rows_kernel, (const __half *)w, (const float *)code, (float *)code_out, (uint8_t *)q,
                              (float *)absmax, status, k, share, cluster);
}

}  // namespace tuna
