// Device-side building blocks of the counting sort (shared by the per-ping
// binning kernels and the fused batched kernel): the tiled pass over a chunk
// of samples, the count and scatter passes of one chunk, the block scan and
// the reference windows. Internal linkage: every translation unit that
// includes this header gets its own copy.
#pragma once

#include "rtacx_internal.cuh"

#include <climits>

namespace rtacx {

namespace {

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

constexpr int kTileLoads = 4;        // independent record loads per thread and tile

// Block-uniform pass over chunk `c` of `nc` equal chunks of the input in
// tiles of blockDim.x * kTileLoads samples: the loads of tile t + 1 are
// issued before tile t is processed, then the keys are computed and
// f(valid[], record[], key[], side[]) is called -- the same number of times
// in every thread, so f may synchronise the block.
template <typename F>
__device__ __forceinline__ void for_chunk(const float* samples, uint64_t n, const BinParams& p,
                                          uint32_t c, uint32_t nc, F&& f)
{
    const uint64_t chunk = (n + nc - 1) / nc;
    const uint64_t begin = (uint64_t)c * chunk;
    const uint64_t end = min(begin + chunk, n);
    const uint64_t tile = (uint64_t)blockDim.x * kTileLoads;
    float4 next[kTileLoads];
    auto load_tile = [&](uint64_t t0) {
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            const uint64_t i = t0 + (uint64_t)u * blockDim.x + threadIdx.x;
            next[u] = i < end ? load_record(samples, i, p) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    if(begin < end) load_tile(begin);
    for(uint64_t t0 = begin; t0 < end; t0 += tile) {
        bool valid[kTileLoads];
        float4 rec[kTileLoads];
        uint32_t key[kTileLoads];
        int side[kTileLoads];
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            valid[u] = t0 + (uint64_t)u * blockDim.x + threadIdx.x < end;
            rec[u] = next[u];
        }
        if(t0 + tile < end) load_tile(t0 + tile);
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            key[u] = kOutOfRange;
            side[u] = 0;
            if(valid[u]) key[u] = sample_key(p, rec[u].z, rec[u].w, side[u]);
        }
        f(valid, rec, key, side);
    }
}

// Count pass of chunk c of nc (shared-memory histogram sh of p.nBins
// words), added into totals[0, nBins) (zeroed by the caller). With `nonempty`
// also the bitmap of the range bins that hold a sample (sh then has
// (nR + 31) / 32 words more), which the cell order's histogram does not tell.
__device__ __forceinline__ void count_chunk(const float* __restrict__ samples, uint64_t n, const BinParams& p, uint32_t c,
                            uint32_t nc, uint32_t* __restrict__ totals, unsigned long long* __restrict__ oor,
                            uint32_t* sh, unsigned long long* s_oor, uint32_t* __restrict__ nonempty = nullptr)
{
    const uint32_t words = nonempty ? (p.key.nR + 31) / 32 : 0u;
    uint32_t* s_bits = sh + p.nBins;
    for(uint32_t b = threadIdx.x; b < p.nBins + words; b += blockDim.x) sh[b] = 0u;
    if(threadIdx.x < 2) s_oor[threadIdx.x] = 0ull;
    __syncthreads();

    uint32_t low = 0, high = 0;
    for_chunk(samples, n, p, c, nc, [&](const bool* valid, const float4* rec, const uint32_t* key, const int* side) {
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            if(valid[u] && key[u] != kOutOfRange) {
                atomicAdd(&sh[key[u]], 1u);
                if(words) {
                    int unused;
                    const uint32_t r = range_key(p.key, rec[u].z, unused), bit = 1u << (r & 31u);
                    if(!(s_bits[r >> 5] & bit)) atomicOr(&s_bits[r >> 5], bit);
                }
            }
            else if(valid[u]) {
                if(side[u] < 0) low++; else high++;
            }
        }
    });
    for(int o = 16; o > 0; o >>= 1) {
        low += __shfl_down_sync(0xffffffffu, low, o);
        high += __shfl_down_sync(0xffffffffu, high, o);
    }
    if(lane_id() == 0 && (low | high)) {
        atomicAdd(&s_oor[0], (unsigned long long)low);
        atomicAdd(&s_oor[1], (unsigned long long)high);
    }
    __syncthreads();
    if(threadIdx.x == 0) {
        if(s_oor[0]) atomicAdd(&oor[0], s_oor[0]);
        if(s_oor[1]) atomicAdd(&oor[1], s_oor[1]);
    }
    for(uint32_t b = threadIdx.x; b < p.nBins; b += blockDim.x)
        if(sh[b]) atomicAdd(&totals[b], sh[b]);
    for(uint32_t b = threadIdx.x; b < words; b += blockDim.x)
        if(s_bits[b]) atomicOr(&nonempty[b], s_bits[b]);
    // Per-block sums of kScanBlock bins (totals[nBins + blk]) for the
    // parallel bin scan: one warp per block of bins.
    const uint32_t blocks = (p.nBins + kScanBlock - 1) / kScanBlock;
    for(uint32_t blk = threadIdx.x >> 5; blk < blocks; blk += blockDim.x >> 5) {
        uint32_t s = 0;
        for(uint32_t b = blk * kScanBlock + lane_id(); b < min((blk + 1) * kScanBlock, p.nBins); b += 32) s += sh[b];
        for(int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if(lane_id() == 0 && s) atomicAdd(&totals[p.nBins + blk], s);
    }
}

// Exclusive block scan of one value per thread (any blockDim.x that is a
// multiple of 32, at most 1024).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t& total)
{
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t x = v;
    for(int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if(lane >= (unsigned)o) x += y;
    }
    if(lane == 31) s_warp[warp] = x;
    __syncthreads();
    const unsigned nw = blockDim.x >> 5;
    if(warp == 0) {
        uint32_t w = lane < nw ? s_warp[lane] : 0u;
        for(int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if(lane >= (unsigned)o) w += y;
        }
        if(lane < nw) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[nw - 1];
    const uint32_t before = warp ? s_warp[warp - 1] : 0u;
    __syncthreads();
    return before + x - v;
}

// Scatter pass of chunk c of nc. Per tile: rank of each sample among the
// tile's samples of its bin (shared-memory histogram sh of p.nBins words,
// zero between tiles); the first sample of each (tile, bin) reserves the
// bin's run with one atomicAdd on the shared cursor and leaves the run's
// base in sh; every sample is written at base + rank.
__device__ __forceinline__ void scatter_chunk(const float* __restrict__ samples, uint64_t n, const BinParams& p, uint32_t c,
                              uint32_t nc, uint32_t* __restrict__ cursor, const uint32_t* __restrict__ offsets,
                              float4* __restrict__ sorted, uint32_t* __restrict__ err, uint32_t* sh)
{
    for(uint32_t b = threadIdx.x; b < p.nBins; b += blockDim.x) sh[b] = 0u;
    const uint32_t total = offsets[p.nBins];
    __syncthreads();

    for_chunk(samples, n, p, c, nc, [&](const bool* valid, const float4* rec, const uint32_t* key, const int*) {
        uint32_t rank[kTileLoads];
#pragma unroll
        for(int u = 0; u < kTileLoads; u++)
            rank[u] = (valid[u] && key[u] != kOutOfRange) ? atomicAdd(&sh[key[u]], 1u) : UINT_MAX;
        __syncthreads();
#pragma unroll
        for(int u = 0; u < kTileLoads; u++)
            if(rank[u] == 0u) sh[key[u]] = atomicAdd(&cursor[cursor_word(key[u])], sh[key[u]]);
        __syncthreads();
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            if(rank[u] == UINT_MAX) continue;
            const uint32_t pos = sh[key[u]] + rank[u];
            float4 out = rec[u];
            if(p.echo_flags) {
                const float2 v = apply_echo(p, make_float2(out.x, out.y), out.z);
                out.x = v.x; out.y = v.y;
            }
            if(pos < total) sorted[pos] = out;
            else atomicOr(err, kErrScatterOverflow);
        }
        __syncthreads();
#pragma unroll
        for(int u = 0; u < kTileLoads; u++)
            if(rank[u] == 0u) sh[key[u]] = 0u;
        __syncthreads();
    });
}

__device__ __forceinline__ uint32_t bin_count(const uint32_t* off, uint32_t nBB, int j)
{
    return off[(size_t)(j + 1) * nBB] - off[(size_t)j * nBB];
}

// Does row r's reference window hold at least two non-empty range bins of the
// bitmap (the view of src/Binner.cu:90-102 is empty otherwise)?
__device__ __forceinline__ bool row_on(const uint32_t* nonempty, int nR, int ov, int r)
{
    const int lo = max(0, r - ov), hi = (int)min((long long)nR - 1, (long long)r + ov);
    int seen = 0;
    for(int w = lo >> 5; w <= hi >> 5 && seen < 2; w++) {
        uint32_t bits = nonempty[w];
        if(w == lo >> 5) bits &= 0xFFFFFFFFu << (lo & 31);
        if(w == hi >> 5) bits &= 0xFFFFFFFFu >> (31 - (hi & 31));
        seen += __popc(bits);
    }
    return seen >= 2;
}

// First / last non-empty range bin of row r's reference window
// [max(0, r - ov), min(nR - 1, r + ov)]; returns false for the empty view
// (no non-empty bin, or istart >= iend: src/Binner.cu:90-102).
__device__ __forceinline__ bool ref_window(const uint32_t* off, uint32_t nBB, uint32_t nR, int ov, int r,
                                           int& f, int& l)
{
    const long long lo = max(0ll, (long long)r - ov);
    const long long hi = min((long long)nR - 1, (long long)r + ov);
    long long a = lo;
    while(a <= hi && bin_count(off, nBB, (int)a) == 0u) a++;
    if(a >= hi) return false;
    long long z = hi;
    while(z > a && bin_count(off, nBB, (int)z) == 0u) z--;
    if(a >= z) return false;
    f = (int)a; l = (int)z;
    return true;
}

// Effective window of output row r: the reference window's first / last
// non-empty bins intersected with the row's PSF support.
__device__ __forceinline__ void window_row(const uint32_t* __restrict__ off, uint32_t nBB, uint32_t nR, int ov,
                           const int2* __restrict__ support, int2* __restrict__ win, int r)
{
    if(r >= (int)nR) return;
    int f, l;
    int2 w = make_int2(1, 0);
    if(ref_window(off, nBB, nR, ov, r, f, l)) {
        const int2 s = support[r];
        w = make_int2(max(f, s.x), min(l, s.y));
    }
    win[r] = w;
}

// Exclusive scan of bins [blk kScanBlock, (blk + 1) kScanBlock) of
// totals[0, nBins), offset by the count of every bin before the block: the
// sum of the block sums before it (totals[nBins + j], j < blk, accumulated by
// the count pass) when block_sums, else the sum of totals[0, blk kScanBlock)
// taken by the whole CTA. Writes offsets (and offsets[nBins] from the block
// holding the last bin) and the scatter's per-bin cursors. Each thread scans
// kScanBlock / blockDim.x consecutive bins; blockDim.x divides kScanBlock.
__device__ __forceinline__ void scan_bin_block(const uint32_t* __restrict__ totals, uint32_t nBins, uint32_t blk,
                                               uint32_t* __restrict__ offsets, uint32_t* __restrict__ cursor,
                                               uint32_t* s_warp, uint32_t* s_prefix, bool block_sums = true)
{
    if(block_sums) {
        if(threadIdx.x < 32) {
            uint32_t s = 0;
            for(uint32_t j = threadIdx.x; j < blk; j += 32) s += totals[nBins + j];
            for(int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if(threadIdx.x == 0) *s_prefix = s;
        }
    }
    else {
        if(threadIdx.x == 0) *s_prefix = 0u;
        __syncthreads();
        uint32_t s = 0;
#pragma unroll 16
        for(uint32_t i = threadIdx.x; i < blk * kScanBlock; i += blockDim.x) s += totals[i];
        for(int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if(lane_id() == 0 && s) atomicAdd(s_prefix, s);
    }
    const uint32_t per = kScanBlock / blockDim.x;
    const uint32_t b0 = blk * kScanBlock + threadIdx.x * per;
    uint32_t sum = 0;
    for(uint32_t u = 0; u < per; u++) sum += b0 + u < nBins ? totals[b0 + u] : 0u;
    uint32_t blk_total;
    uint32_t o = block_exclusive_scan(sum, s_warp, blk_total);   // synchronises: s_prefix is visible
    o += *s_prefix;
    for(uint32_t u = 0; u < per; u++) {
        const uint32_t b = b0 + u;
        if(b >= nBins) break;
        const uint32_t v = totals[b];
        offsets[b] = o;
        cursor[cursor_word(b)] = o;
        o += v;
        if(b == nBins - 1) offsets[nBins] = o;
    }
}

// Count pass of chunk c of nc straight into totals[0, nBins) with one global
// atomic per sample (no shared histogram: the fused batched kernel keeps its
// shared memory for the gather). Out-of-range counts and the bitmap as
// count_chunk's (a set bit is read before it is written again).
__device__ __forceinline__ void count_chunk_global(const float* __restrict__ samples, uint64_t n, const BinParams& p,
                                                   uint32_t c, uint32_t nc, uint32_t* __restrict__ totals,
                                                   unsigned long long* __restrict__ oor, unsigned long long* s_oor,
                                                   uint32_t* nonempty = nullptr)
{
    if(threadIdx.x < 2) s_oor[threadIdx.x] = 0ull;
    __syncthreads();
    uint32_t low = 0, high = 0;
    for_chunk(samples, n, p, c, nc, [&](const bool* valid, const float4* rec, const uint32_t* key, const int* side) {
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            if(valid[u] && key[u] != kOutOfRange) {
                atomicAdd(&totals[key[u]], 1u);
                if(nonempty) {
                    int unused;
                    const uint32_t r = range_key(p.key, rec[u].z, unused), bit = 1u << (r & 31u);
                    if(!(__ldcg(nonempty + (r >> 5)) & bit)) atomicOr(nonempty + (r >> 5), bit);
                }
            }
            else if(valid[u]) {
                if(side[u] < 0) low++; else high++;
            }
        }
    });
    for(int o = 16; o > 0; o >>= 1) {
        low += __shfl_down_sync(0xffffffffu, low, o);
        high += __shfl_down_sync(0xffffffffu, high, o);
    }
    if(lane_id() == 0 && (low | high)) {
        atomicAdd(&s_oor[0], (unsigned long long)low);
        atomicAdd(&s_oor[1], (unsigned long long)high);
    }
    __syncthreads();
    if(threadIdx.x == 0) {
        if(s_oor[0]) atomicAdd(&oor[0], s_oor[0]);
        if(s_oor[1]) atomicAdd(&oor[1], s_oor[1]);
    }
}

// Scatter pass of chunk c of nc with one global atomic per sample on its
// bin's cursor (no shared histogram); positions past the counted total set
// kErrScatterOverflow instead of being written.
__device__ __forceinline__ void scatter_chunk_global(const float* __restrict__ samples, uint64_t n, const BinParams& p,
                                                     uint32_t c, uint32_t nc, uint32_t* __restrict__ cursor,
                                                     const uint32_t* __restrict__ offsets, float4* __restrict__ sorted,
                                                     uint32_t* __restrict__ err)
{
    const uint32_t total = offsets[p.nBins];
    for_chunk(samples, n, p, c, nc, [&](const bool* valid, const float4* rec, const uint32_t* key, const int*) {
#pragma unroll
        for(int u = 0; u < kTileLoads; u++) {
            if(!valid[u] || key[u] == kOutOfRange) continue;
            const uint32_t pos = atomicAdd(&cursor[cursor_word(key[u])], 1u);
            float4 out = rec[u];
            if(p.echo_flags) {
                const float2 v = apply_echo(p, make_float2(out.x, out.y), out.z);
                out.x = v.x; out.y = v.y;
            }
            if(pos < total) sorted[pos] = out;
            else atomicOr(err, kErrScatterOverflow);
        }
    });
}

// Ranks of chunk c of nc (at most THREADS x LOADS samples) among the samples of
// their bins: a shared histogram gives each sample's rank in the chunk (kept
// with its key in one register), one 64-bit atomic per pair of bins adds the
// chunk's counts to the totals and returns what its ranks start at; the ranks
// are stored in input order. Also the bitmap of range bins and, with
// block_sums, the sums of kScanBlock bins (totals[nBins + block]).
constexpr int kRankKeyBits = 14;                     // nBins <= 2^14, a chunk's ranks < 2^18
template <int THREADS, int LOADS>
__device__ __forceinline__ void count_ranked(const float* __restrict__ samples, uint64_t n, const BinParams& p, uint32_t c,
                                             uint32_t nc, uint32_t* __restrict__ totals, uint32_t* __restrict__ nonempty,
                                             uint32_t* __restrict__ ranks, uint32_t* sh, bool block_sums)
{
    static_assert(THREADS * LOADS <= 1 << (32 - kRankKeyBits), "key and rank share a word");
    const uint32_t tid = threadIdx.x, pairs = (p.nBins + 1) / 2, words = (p.key.nR + 31) / 32;
    const uint32_t blocks = (p.nBins + kScanBlock - 1) / kScanBlock;
    uint32_t *s_bits = sh + 2 * pairs, *s_blk = s_bits + words;
    uint2* s_pair = reinterpret_cast<uint2*>(sh);
    for(uint32_t b = tid; b < 2 * pairs + words + blocks; b += THREADS) sh[b] = 0u;
    __syncthreads();
    const uint64_t chunk = (n + nc - 1) / nc, begin = c * chunk, end = min(begin + chunk, n);
    uint32_t kr[LOADS];                     // key | rank in the CTA << kRankKeyBits
#pragma unroll
    for(int g = 0; g < LOADS; g += 4) {
        float4 rec[4];
        if(begin + (uint64_t)g * THREADS >= end) {
#pragma unroll
            for(int u = 0; u < 4; u++) kr[g + u] = kOutOfRange;
            continue;
        }
#pragma unroll
        for(int u = 0; u < 4; u++) {
            const uint64_t i = begin + (uint64_t)(g + u) * THREADS + tid;
            rec[u] = i < end ? load_record(samples, i, p) : make_float4(0.f, 0.f, INFINITY, 0.f);
        }
#pragma unroll
        for(int u = 0; u < 4; u++) {
            int side;
            const uint32_t r = range_key(p.key, rec[u].z, side);
            const uint32_t k = begin + (uint64_t)(g + u) * THREADS + tid < end ? sample_key(p, rec[u].z, rec[u].w, side)
                                                                                : kOutOfRange;
            kr[g + u] = kOutOfRange;
            if(k == kOutOfRange) continue;
            kr[g + u] = k | atomicAdd(&sh[k], 1u) << kRankKeyBits;
            const uint32_t bit = 1u << (r & 31u);
            if(!(s_bits[r >> 5] & bit)) atomicOr(&s_bits[r >> 5], bit);
        }
    }
    __syncthreads();
    // The CTA's counts into the totals; the bins' entries become the first ranks.
    constexpr int kBatch = 4;
    for(uint32_t w0 = tid & ~31u; w0 < pairs; w0 += kBatch * THREADS) {
        const uint32_t b0 = w0 + (tid & 31u);
        uint2 v[kBatch];
        unsigned long long old[kBatch];
#pragma unroll
        for(int q = 0; q < kBatch; q++) {
            const uint32_t b = b0 + q * THREADS;
            v[q] = b < pairs ? s_pair[b] : make_uint2(0u, 0u);
            // (an odd last bin's neighbour is the first block sum)
            if(!(v[q].x | v[q].y)) old[q] = 0ull;
            else if(2 * b + 1 < p.nBins) old[q] = atomicAdd(reinterpret_cast<unsigned long long*>(totals) + b,
                                                            (unsigned long long)v[q].y << 32 | v[q].x);
            else old[q] = atomicAdd(&totals[2 * b], v[q].x);
        }
#pragma unroll
        for(int q = 0; q < kBatch; q++) {
            const uint32_t b = b0 + q * THREADS;
            if(b < pairs) s_pair[b] = make_uint2((uint32_t)old[q], (uint32_t)(old[q] >> 32));
            // (a warp's pairs lie in one block of kScanBlock bins)
            const uint32_t sum = __reduce_add_sync(0xffffffffu, v[q].x + v[q].y);
            if((tid & 31) == 0 && sum) atomicAdd(&s_blk[2 * b / kScanBlock], sum);
        }
    }
    __syncthreads();
#pragma unroll
    for(int u = 0; u < LOADS; u++) {
        const uint64_t i = begin + (uint64_t)u * THREADS + tid;
        if(kr[u] != kOutOfRange) ranks[i] = sh[kr[u] & ((1u << kRankKeyBits) - 1u)] + (kr[u] >> kRankKeyBits);
    }
    for(uint32_t b = tid; b < words; b += THREADS)
        if(s_bits[b]) atomicOr(&nonempty[b], s_bits[b]);
    for(uint32_t b = tid; b < blocks; b += THREADS)
        if(block_sums && s_blk[b]) atomicAdd(&totals[p.nBins + b], s_blk[b]);
}

// Scatter of chunk c of nc straight to offsets[bin] + rank, kRankedLoads records
// per thread in flight (bound by the latency of the loads). Batch of 16 pings,
// 2.5e6 2D samples, us: count 75 with one global atomic per sample, 45 with
// count_ranked; scatter 55 with a cursor atomic per sample, 43.
constexpr int kRankedLoads = 8;

__device__ __forceinline__ void scatter_chunk_ranked(const float* __restrict__ samples, uint64_t n, const BinParams& p,
                                                     uint32_t c, uint32_t nc, const uint32_t* ranks,
                                                     const uint32_t* offsets, float4* __restrict__ sorted,
                                                     uint32_t* __restrict__ err)
{
    const uint32_t total = offsets[p.nBins];
    const uint64_t chunk = (n + nc - 1) / nc, begin = c * chunk, end = min(begin + chunk, n);
    for(uint64_t t0 = begin + threadIdx.x; t0 < end; t0 += (uint64_t)kRankedLoads * blockDim.x) {
        float4 rec[kRankedLoads];
        uint32_t pos[kRankedLoads];
#pragma unroll
        for(int u = 0; u < kRankedLoads; u++) {
            const uint64_t i = t0 + (uint64_t)u * blockDim.x;
            rec[u] = i < end ? load_record(samples, i, p) : make_float4(0.f, 0.f, INFINITY, 0.f);
            pos[u] = i < end ? ranks[i] : 0u;
        }
#pragma unroll
        for(int u = 0; u < kRankedLoads; u++) {
            int side;
            const uint32_t k = t0 + (uint64_t)u * blockDim.x < end ? sample_key(p, rec[u].z, rec[u].w, side) : kOutOfRange;
            pos[u] = k != kOutOfRange ? offsets[k] + pos[u] : kOutOfRange;
        }
#pragma unroll
        for(int u = 0; u < kRankedLoads; u++) {
            if(pos[u] == kOutOfRange) continue;
            if(p.echo_flags) {
                const float2 v = apply_echo(p, make_float2(rec[u].x, rec[u].y), rec[u].z);
                rec[u].x = v.x; rec[u].y = v.y;
            }
            if(pos[u] < total) sorted[pos[u]] = rec[u];
            else atomicOr(err, kErrScatterOverflow);
        }
    }
}

} // namespace

} // namespace rtacx
