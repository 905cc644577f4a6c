// Range-cell form of the plain reduction: device building blocks (shared by
// the single-ping kernels and the batched kernel) and what they need.
//
// The pulse table is piecewise linear (a linear-filtered texture). When its
// taps are one output range apart, the knots that all output rows put on the
// travel axis fall on one grid: between two neighbouring knots (a range
// cell) every row's pulse weight is linear in the travel. A sample of cell C
// at fraction alpha then reaches row r with
//   P[C - r] + (alpha + e_r) D[C - r],   D[i] = P[i + 1] - P[i],
// where e_r is the distance of row r's float range from the grid, so the
// ping is, exactly,
//   T[C][b] = sum v beam(theta - theta_b),  M[C][b] = sum alpha v beam(...)
//   out(r, b) = sum_i P[i] T[r + i][b] + D[i] (M[r + i][b] + e_r T[r + i][b]).
// Each (sample, bearing) pair costs one beam lookup and four multiply-adds
// whatever the pulse's length, instead of one product per output row.
// Samples within `knot` of a grid knot, which the rows' e_r put into
// different pieces for different rows, are reduced row by row.
//
// Row pairs: a pulse that reaches at most two output rows (the reference's
// adaptive duration, one range bin) uses the same accumulation with the
// cells between rows: T and M then hold the sample's contributions to the
// cell's two rows, with the rows' own pulse weights, whatever the table.
#pragma once

#include "rtacx_bin_device.cuh"
#include "rtacx_internal.cuh"

namespace rtacx {

namespace {

// Two floats in one 64-bit register (sm_100 packed single-precision
// arithmetic: one instruction, two lanes, each rounded to nearest).
using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Reductions into buffers that the reducing kernel never reads: no memory
// clobber, so that loads move across them.
__device__ __forceinline__ void red_add_f4(float4* addr, float x, float y, float z, float w)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(x), "f"(y), "f"(z), "f"(w));
}

__device__ __forceinline__ void red_add_f2(float2* addr, float x, float y)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(x), "f"(y));
}

// Pulse weight at delta = travel - output range: the lerp of the zero-padded
// pulse table (pad[0] = pad[n + 1] = 0) in global memory, as the gathers of
// rtacx_reduce.cu evaluate it.
__device__ __forceinline__ float2 pulse_at(const float2* __restrict__ pad, const AxisLerp& ax, float delta)
{
    const float x1 = fmaf(delta, ax.k_hi, ax.c);
    const float fi = floorf(x1);
    if(!(fi >= -1.0f && fi <= (float)(ax.n - 1))) return make_float2(0.f, 0.f);
    const float alpha = fmaf(delta, ax.k_lo, fmaf(delta, ax.k_hi, ax.c - fi));
    const int i = (int)fi + 1;
    const float2 lo = __ldg(pad + i), hi = __ldg(pad + i + 1);
    return make_float2(fmaf(alpha, hi.x - lo.x, lo.x), fmaf(alpha, hi.y - lo.y, lo.y));
}

// ---- the beam table in shared memory ---------------------------------------
// Entry i of the table is the linear piece left of texel i: {value at its
// left end, slope}, entry 0 the rise from the zero border to texel 0, entry W
// the fall after texel W - 1, entry W + 1 zero (every coordinate outside).
// An even table's texel coordinates are half-integers: its entries are stored
// from the middle of the piece, so that the constant of the fraction is a
// whole number either way (see BeamLookup).
// COPIES 16: entry i of copy k at 16 i + k, so that lanes that read the copy of
// their own pair of banks never conflict (see k_cells).
template <int COPIES = 1>
__device__ __forceinline__ void load_beam_table(float2* tab, const float* __restrict__ beam_pad, const AxisLerp& ax, int tid,
                                                int threads)
{
    const int W = ax.n;
    const bool whole = ax.c == floorf(ax.c);         // texel coordinates are whole numbers (an odd table)
    for(int k = tid; k < (W + 2) * COPIES; k += threads) {
        const int i = k / COPIES;
        float2 e = make_float2(0.f, 0.f);
        if(i <= W) {
            const float lo = beam_pad[i], hi = beam_pad[i + 1];
            e.y = hi - lo;
            e.x = whole ? lo : fmaf(0.5f, e.y, lo);
        }
        tab[k] = e;
    }
}

// Beam weights of one sample at a pair of bearings: x = (theta - theta_b) k +
// c + 1/2 rounded to a whole number by adding 1.5 * 2^23 (the piece's index,
// in the low mantissa bits), the fraction in one more fused multiply-add from
// the exact difference of the constant and that number, then the piece's
// line. An index below 0 or above W lands on the zero entry.
constexpr float kRoundMagic = 12582912.0f;          // 1.5 * 2^23
constexpr uint32_t kRoundMagicBits = 0x4B400000u;

// tab: the table, at the lane's copy.
template <int COPIES = 1>
struct BeamLookup {
    f32x2 k2, k_lo2, c2, magic2, frac2, minus2;
    uint32_t last;                                   // W + 1
    __device__ __forceinline__ void init(const AxisLerp& ax)
    {
        k2 = pack2(ax.k_hi, ax.k_hi);
        k_lo2 = pack2(ax.k_lo, ax.k_lo);
        const float c = ax.c + 0.5f;                 // floor(x) + 1 = round(x + 1/2)
        c2 = pack2(c, c);
        magic2 = pack2(kRoundMagic, kRoundMagic);
        // fraction = d k + (ax.c + 1 - index); the half of an even table's
        // coordinate is in its entries instead.
        const float f = kRoundMagic + (ax.c == floorf(ax.c) ? ax.c + 1.0f : ax.c + 0.5f);
        frac2 = pack2(f, f);
        minus2 = pack2(-1.0f, -1.0f);
        last = (uint32_t)ax.n + 1u;
    }
    // theta2: the sample's bearing twice; minus_tb2: minus the two bearings.
    __device__ __forceinline__ f32x2 operator()(const float2* __restrict__ tab, f32x2 theta2, f32x2 minus_tb2) const
    {
        const f32x2 d = add2(theta2, minus_tb2);
        const f32x2 y = add2(fma2(d, k2, c2), magic2);
        const f32x2 a = fma2(d, k2, fma2(d, k_lo2, fma2(y, minus2, frac2)));
        const float2 yu = unpack2(y), au = unpack2(a);
        const float2 e0 = tab[min(__float_as_uint(yu.x) - kRoundMagicBits, last) * COPIES];
        const float2 e1 = tab[min(__float_as_uint(yu.y) - kRoundMagicBits, last) * COPIES];
        return pack2(fmaf(au.x, e0.y, e0.x), fmaf(au.y, e1.y, e1.x));
    }
};

// ---- accumulation of one ping's samples into the cell rows ------------------
// The samples are sorted by (bearing window, block of cells). A warp takes
// units of up to kUnit consecutive samples, so of one window or two and of
// few cells. Lane l holds the bearings at positions l, l + 32, ... of a
// window. The unit's samples are listed by cell in shared memory, each value
// twice (the packed operands); all lanes then walk a cell's list, summing T
// and M for their bearings in registers, and add the sums to the cell row in
// 16-byte reductions. Windows that are shared out (wide beams: every sample
// reaches every window) walk the same list one after the other.
constexpr int kUnit = 128;                 // samples per warp and unit, at most
constexpr int kUnitLoads = kUnit / 32;
constexpr int kListCells = 32;             // cells listed at a time

// A listed sample, each value twice: theta, v.x, v.y, alpha; for row pairs
// theta and the two rows' weighted values.
template <bool PAIR> struct CellEntry { ulonglong2 v[PAIR ? 3 : 2]; };

template <bool PAIR>
struct CellWarpSmem {
    CellEntry<PAIR> list[kUnit];
    float4 w[kUnit];                        // {v.x, v.y, alpha, -}; row-by-row samples: travel for alpha; pairs: both rows'
    uint32_t count[kListCells], start[kListCells];
};

// One sample next to a knot, row by row: the lanes take 32 rows at a time,
// then every row's weight is broadcast and reduced into the (zeroed) ping.
template <int BPL, int COPIES>
__device__ __forceinline__ void reduce_row_by_row(const CellPing& P, float4 w, float theta, int C, const float2* tab,
                                                  const BeamLookup<COPIES>& beam, const f32x2 (&minus_tb)[BPL / 2],
                                                  const int* bearing)
{
    const int lane = threadIdx.x & 31;
    const f32x2 th = pack2(theta, theta);
    float bv[BPL];
#pragma unroll
    for(int p = 0; p < BPL / 2; p++) {
        const float2 x = unpack2(beam(tab, th, minus_tb[p]));
        bv[2 * p] = x.x;
        bv[2 * p + 1] = x.y;
    }
    // Rows whose pulse reaches cells C - 1 .. C + 1.
    const int r_lo = max(0, C - P.cp.taps - 1), r_hi = min((int)P.nR - 1, C + 2);
    for(int r0 = r_lo; r0 <= r_hi; r0 += 32) {
        float2 u = make_float2(0.f, 0.f);
        if(r0 + lane <= r_hi) {
            const float2 f = pulse_at(P.pulse, P.range_axis, w.z - P.ranges[r0 + lane]);
            u = make_float2(w.x * f.x - w.y * f.y, w.x * f.y + w.y * f.x);
        }
        const int rows = min(32, r_hi - r0 + 1);
        for(int q = 0; q < rows; q++) {
            const float ux = __shfl_sync(0xffffffffu, u.x, q), uy = __shfl_sync(0xffffffffu, u.y, q);
            if(ux == 0.0f && uy == 0.0f) continue;
#pragma unroll
            for(int p = 0; p < BPL; p++) {
                const int b = bearing[p];
                if(b >= 0) red_add_f2(P.out + (size_t)(r0 + q) * P.nB + b, ux * bv[p], uy * bv[p]);
            }
        }
    }
}

// Accumulates samples [first, first + count) (count <= kUnit) of the sorted
// order into the cell rows. SHARED: for the windows win0, win0 + win_step, ...;
// otherwise for each sample's own window.
// FLOOR (lobe form): the beam table holds what the lobe stands out of the
// floor; the floor times the cells' sums of v and alpha v goes into one more
// column (no sample is next to a knot).
template <int BPL, bool SHARED, bool PAIR, bool FLOOR = false, int COPIES>
__device__ __forceinline__ void accumulate_unit(const CellPing& P, uint32_t first, uint32_t count, int win0,
                                                int win_step, CellWarpSmem<PAIR>& S, const float2* tab,
                                                const BeamLookup<COPIES>& beam)
{
    constexpr int NP = BPL / 2;
    const int lane = threadIdx.x & 31;
    float theta[kUnitLoads];
    int cell[kUnitLoads];                  // storage row; -1 dropped; -2 - row: reduced row by row
    int win[kUnitLoads];
    int cur = INT_MAX;
    bool near_knot = false;
    __syncwarp();
#pragma unroll
    for(int q = 0; q < kUnitLoads; q++) {
        const uint32_t i = (uint32_t)(q * 32 + lane);
        cell[q] = -1;
        win[q] = INT_MAX;
        theta[q] = 0.0f;
        if(i < count) {
            const float4 rec = __ldcs(P.sorted + first + i);
            float alpha;
            const int c = range_cell(P.cp, rec.z, alpha);
            const bool near = !PAIR && !FLOOR && !(alpha >= P.cp.knot && alpha <= 1.0f - P.cp.knot);
            // Bearings far outside (and NaN) move to a bearing that no beam reaches.
            theta[q] = fminf(fmaxf(rec.w, P.theta_lo), P.theta_hi);
            if(PAIR) {
                // Storage row c holds the shares of output rows c - 1 and c.
                float2 f[2];
                int side;
                const int key = (int)range_key(P.key, rec.z, side);
#pragma unroll
                for(int k = 0; k < 2; k++) {
                    const int r = c - 1 + k;
                    const bool on = c >= 0 && r >= 0 && r < (int)P.nR && abs(key - r) <= P.overlap;
                    f[k] = on ? pulse_at(P.pulse, P.range_axis, rec.z - P.ranges[on ? r : 0]) : make_float2(0.f, 0.f);
                }
                S.w[i] = make_float4(rec.x * f[0].x - rec.y * f[0].y, rec.x * f[0].y + rec.y * f[0].x,
                                     rec.x * f[1].x - rec.y * f[1].y, rec.x * f[1].y + rec.y * f[1].x);
            }
            else S.w[i] = make_float4(rec.x, rec.y, near ? rec.z : alpha, 0.0f);
            if(c >= 0) {
                cell[q] = near ? -2 - c : c;
                near_knot |= near;
                win[q] = SHARED ? 0 : (int)bearing_bin(P.win_scale, P.win_offset, (uint32_t)P.windows, rec.w);
                cur = min(cur, win[q]);
            }
        }
    }
    // Every lane reads S.w below, also where no sample is listed (all of them
    // next to knots): the votes converge the lanes but order no memory.
    __syncwarp();
    near_knot = __any_sync(0xffffffffu, near_knot);
    for(cur = __reduce_min_sync(0xffffffffu, cur); cur != INT_MAX;) {
        const int w_begin = SHARED ? win0 : cur, w_end = SHARED ? P.windows : cur + 1;
        int base = INT_MAX, next_win = INT_MAX;
#pragma unroll
        for(int q = 0; q < kUnitLoads; q++) {
            if(win[q] == cur && cell[q] >= 0) base = min(base, cell[q]);
            if(win[q] > cur) next_win = min(next_win, win[q]);
        }
        base = __reduce_min_sync(0xffffffffu, base);
        while(base != INT_MAX) {
            // List the window's samples of cells base .. base + kListCells - 1, by cell.
            uint32_t rank[kUnitLoads];
            int next = INT_MAX;
            S.count[lane] = 0u;
            __syncwarp();
#pragma unroll
            for(int q = 0; q < kUnitLoads; q++) {
                const bool in = win[q] == cur && cell[q] >= base;
                rank[q] = in && cell[q] - base < kListCells ? atomicAdd(&S.count[cell[q] - base], 1u) : 0xFFFFFFFFu;
                if(in && cell[q] - base >= kListCells) next = min(next, cell[q]);
            }
            __syncwarp();
            const uint32_t mine = S.count[lane];
            uint32_t upto = mine;
            for(int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, upto, o);
                if(lane >= o) upto += y;
            }
            S.start[lane] = upto - mine;
            __syncwarp();
#pragma unroll
            for(int q = 0; q < kUnitLoads; q++) {
                if(rank[q] == 0xFFFFFFFFu) continue;
                const uint32_t at = S.start[cell[q] - base] + rank[q];
                const float4 w = S.w[q * 32 + lane];
                S.list[at].v[0] = make_ulonglong2(pack2(theta[q], theta[q]), pack2(w.x, w.x));
                S.list[at].v[1] = make_ulonglong2(pack2(w.y, w.y), pack2(w.z, w.z));
                if constexpr(PAIR) S.list[at].v[2].x = pack2(w.w, w.w);
            }
            __syncwarp();
            const uint32_t filled = __ballot_sync(0xffffffffu, mine != 0u);
            for(int w = w_begin; w < w_end; w += win_step) {
                const int pos0 = w * 32 * BPL + lane;
                f32x2 minus_tb[NP];
                int2 col[NP];
#pragma unroll
                for(int p = 0; p < NP; p++) {
                    minus_tb[p] = pack2(-P.pos_theta[pos0 + 64 * p], -P.pos_theta[pos0 + 64 * p + 32]);
                    if(!SHARED) col[p] = make_int2(P.pos_col[pos0 + 64 * p], P.pos_col[pos0 + 64 * p + 32]);
                }
                int s = 0;
                for(uint32_t left = filled; left; left &= left - 1u) {
                    const int k = __ffs(left) - 1;
                    const int end = (int)__shfl_sync(0xffffffffu, upto, k);
                    if(FLOOR) {
                        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
                        for(int i = s + lane; i < end; i += 32) {
                            const float* e = reinterpret_cast<const float*>(&S.list[i]);
                            const float vx = e[2], vy = e[4], alpha = e[6];
                            sum.x += vx; sum.y += vy;
                            sum.z = fmaf(alpha, vx, sum.z); sum.w = fmaf(alpha, vy, sum.w);
                        }
                        for(int o = 16; o > 0; o >>= 1) {
                            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o); sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
                            sum.z += __shfl_xor_sync(0xffffffffu, sum.z, o); sum.w += __shfl_xor_sync(0xffffffffu, sum.w, o);
                        }
                        if(lane == 0)
                            red_add_f4(P.cells + (size_t)(base + k) * P.pitch + P.floor_col, P.floor * sum.x, P.floor * sum.y,
                                       P.floor * sum.z, P.floor * sum.w);
                    }
                    f32x2 acc[NP][4];
#pragma unroll
                    for(int p = 0; p < NP; p++)
#pragma unroll
                        for(int e = 0; e < 4; e++) acc[p][e] = 0ull;
#pragma unroll COPIES > 1 ? 4 : BPL
                    for(; s < end; s++) {
                        const ulonglong2 e0 = S.list[s].v[0], e1 = S.list[s].v[1];
                        f32x2 e2 = 0ull;
                        if constexpr(PAIR) e2 = S.list[s].v[2].x;
#pragma unroll
                        for(int p = 0; p < NP; p++) {
                            const f32x2 B = beam(tab, e0.x, minus_tb[p]);
                            acc[p][0] = fma2(e0.y, B, acc[p][0]);
                            acc[p][1] = fma2(e1.x, B, acc[p][1]);
                            if constexpr(PAIR) {
                                acc[p][2] = fma2(e1.y, B, acc[p][2]);
                                acc[p][3] = fma2(e2, B, acc[p][3]);
                            }
                            else {
                                const f32x2 aB = mul2(e1.y, B);
                                acc[p][2] = fma2(e0.y, aB, acc[p][2]);
                                acc[p][3] = fma2(e1.x, aB, acc[p][3]);
                            }
                        }
                    }
                    float4* row = P.cells + (size_t)(base + k) * P.pitch;
#pragma unroll
                    for(int p = 0; p < NP; p++) {
                        const float2 a = unpack2(acc[p][0]), b = unpack2(acc[p][1]);
                        const float2 c = unpack2(acc[p][2]), d = unpack2(acc[p][3]);
                        // (shared-out windows reload the columns: registers)
                        if(SHARED) col[p] = make_int2(P.pos_col[pos0 + 64 * p], P.pos_col[pos0 + 64 * p + 32]);
                        if(col[p].x >= 0) red_add_f4(row + col[p].x, a.x, b.x, c.x, d.x);
                        if(col[p].y >= 0) red_add_f4(row + col[p].y, a.y, b.y, c.y, d.y);
                    }
                }
            }
            base = __reduce_min_sync(0xffffffffu, next);
            __syncwarp();
        }
        if(!PAIR && !FLOOR && near_knot) {
            for(int w = w_begin; w < w_end; w += win_step) {
                const int pos0 = w * 32 * BPL + lane;
                f32x2 minus_tb[NP];
                int bearing[BPL];
#pragma unroll
                for(int p = 0; p < NP; p++)
                    minus_tb[p] = pack2(-P.pos_theta[pos0 + 64 * p], -P.pos_theta[pos0 + 64 * p + 32]);
#pragma unroll
                for(int p = 0; p < BPL; p++) {
                    const int col = P.pos_col[pos0 + 32 * p];
                    bearing[p] = col < 0 ? -1 : P.col_bearing[col];
                }
#pragma unroll 1
                for(int q = 0; q < kUnitLoads; q++) {
                    // (no register array indexing: the values go through selects)
                    int c = cell[0], v = win[0];
                    float th = theta[0];
#pragma unroll
                    for(int z = 1; z < kUnitLoads; z++) {
                        c = q == z ? cell[z] : c;
                        v = q == z ? win[z] : v;
                        th = q == z ? theta[z] : th;
                    }
                    uint32_t near = __ballot_sync(0xffffffffu, c <= -2 && v == cur);
                    for(; near; near &= near - 1u) {
                        const int l = __ffs(near) - 1;
                        reduce_row_by_row<BPL>(P, S.w[q * 32 + l], __shfl_sync(0xffffffffu, th, l),
                                               -3 - __shfl_sync(0xffffffffu, c, l), tab, beam, minus_tb, bearing);
                    }
                }
            }
        }
        cur = __reduce_min_sync(0xffffffffu, next_win);
    }
}

// ---- 1D sensors --------------------------------------------------------------
// Without bearings a sample's sums are two complex numbers, so nothing is
// gained by sorting: each sample is one 16-byte reduction {v, alpha v} into
// its cell (ROWS: one 8-byte reduction per output row it reaches, into float2
// rows), straight from the input order. Samples [begin, end) by one CTA,
// kLoads1D records per thread in flight. cells: the copy of the cell rows that
// the CTA adds into (copy_1d). s_bits: the CTA's bitmap of range bins. The records (echo
// model applied) are kept in `copy` for the diagnostic copy of the sorted scratch.
constexpr int kLoads1D = 4;
// Copies of the cell rows, taken in turn by the CTAs. On large pings one queues
// at its L2 addresses: 3e6 samples on 4161 cells, whole ping, 55.5 us; 41.6 with
// 8 copies, 41.1 with 32, 33 without the reductions. And a word that many
// samples add into one after the other loses digits: 1.3e5 samples on 2070 to
// 2113 cells (63 each) 4.1e-7 and 4.4e-7 from 64 bits with one copy, 2.7e-7 and
// 3.3e-7 with 4, 2.7e-7 and 3.0e-7 with 8; 10.6 and 11.4 us, 10.3 and 11.4, 10.8
// and 12.2. Row by row, 20000 samples on 1049 rows (95 each): 1.7e-7, 8 copies
// 9e-8.
constexpr int kReplicas1D = 8;

__device__ __forceinline__ float4* copy_1d(const CellPing& P, bool rows, uint32_t cta)
{
    const size_t k = cta % (uint32_t)P.replicas;
    return rows ? reinterpret_cast<float4*>(reinterpret_cast<float2*>(P.cells) + k * P.nR) : P.cells + k * P.cp.cells;
}

template <bool ROWS>
__device__ __forceinline__ void accumulate_1d(const CellPing& P, const BinParams& p, const float* __restrict__ samples,
                                              uint64_t begin, uint64_t end, float4* cells, uint32_t* s_bits,
                                              float4* copy)
{
    const int lane = threadIdx.x & 31;
    // Whole warps run every iteration (the row-by-row samples are shared out
    // over the lanes).
    for(uint64_t i0 = begin + threadIdx.x - lane; i0 < end; i0 += (uint64_t)blockDim.x * kLoads1D) {
        float4 rec[kLoads1D];
#pragma unroll
        for(int u = 0; u < kLoads1D; u++) {
            const uint64_t i = i0 + (uint64_t)u * blockDim.x + lane;
            rec[u] = i < end ? load_record(samples, i, p) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for(int u = 0; u < kLoads1D; u++) {
            const uint64_t i = i0 + (uint64_t)u * blockDim.x + lane;
            const float t = rec[u].z;
            int side;
            const uint32_t key = i < end ? range_key(p.key, t, side) : kOutOfRange;
            float2 v = make_float2(rec[u].x, rec[u].y);
            if(p.echo_flags) v = apply_echo(p, v, t);
            if(i < end) __stcs(copy + i, make_float4(v.x, v.y, t, 0.0f));
            float alpha = 0.5f;
            const int row = key != kOutOfRange ? range_cell(P.cp, t, alpha) : -1;
            if(key != kOutOfRange) {
                const uint32_t bit = 1u << (key & 31u);
                if(!(s_bits[key >> 5] & bit)) atomicOr(&s_bits[key >> 5], bit);
            }
            if(ROWS) {
                if(row < 0) continue;
                const int r0 = row - (P.rows - 1);
#pragma unroll 4
                for(int r = max(r0, 0); r < min(r0 + P.rows, (int)P.nR); r++) {
                    if(abs((int)key - r) > P.overlap) continue;
                    const float2 f = pulse_at(P.pulse, P.range_axis, t - P.ranges[r]);
                    if(f.x != 0.0f || f.y != 0.0f)
                        red_add_f2(reinterpret_cast<float2*>(cells) + r, v.x * f.x - v.y * f.y, v.x * f.y + v.y * f.x);
                }
                continue;
            }
            const bool near = row >= 0 && !(alpha >= P.cp.knot && alpha <= 1.0f - P.cp.knot);
            if(row >= 0 && !near) red_add_f4(cells + row, v.x, v.y, alpha * v.x, alpha * v.y);
            // Next to a knot: row by row (rows whose pulse reaches cells C - 1 .. C + 1).
            for(uint32_t m = __ballot_sync(0xffffffffu, near); m; m &= m - 1u) {
                const int l = __ffs(m) - 1;
                const float vx = __shfl_sync(0xffffffffu, v.x, l), vy = __shfl_sync(0xffffffffu, v.y, l);
                const float tl = __shfl_sync(0xffffffffu, t, l);
                const int C = __shfl_sync(0xffffffffu, row, l) - 1;
                for(int r = max(0, C - P.cp.taps - 1) + lane; r <= min((int)P.nR - 1, C + 2); r += 32) {
                    const float2 f = pulse_at(P.pulse, P.range_axis, tl - P.ranges[r]);
                    if(f.x != 0.0f || f.y != 0.0f) red_add_f2(P.out + r, vx * f.x - vy * f.y, vx * f.y + vy * f.x);
                }
            }
        }
    }
}

// Output row r of a ping summed row by row.
__device__ __forceinline__ void join_rows_1d(const CellPing& P, int r, const uint32_t* nonempty)
{
    float2 v = make_float2(0.f, 0.f);
#pragma unroll 8
    for(int k = 0; k < P.replicas; k++) {
        const float2 x = __ldcg(reinterpret_cast<const float2*>(P.cells) + (size_t)k * P.nR + r);
        v.x += x.x; v.y += x.y;
    }
    P.out[r] = row_on(nonempty, (int)P.nR, P.overlap, r) ? v : make_float2(0.f, 0.f);
}

// Range filter of a 1D ping: four threads per output row, every fourth tap
// each. s: the cells of the CTA's rows and the taps.
constexpr int kFilterRows1D = 32;          // rows per CTA of 4 kFilterRows1D threads
__host__ __device__ __forceinline__ size_t filter_smem_1d(int H, int rows)
{
    return (size_t)(rows + 2 * (H + 1)) * sizeof(float4);
}

template <int ROWS>
__device__ __forceinline__ void filter_rows_1d(const CellPing& P, int tile, float4* s, const uint32_t* nonempty)
{
    const int n = P.cp.taps + 1, rows0 = tile * ROWS;
    float4 *s_cells = s, *s_taps = s + ROWS + n;
    for(int i = threadIdx.x; i < ROWS + n; i += 4 * ROWS)
    {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        if(rows0 + i < P.cp.cells)
            for(int k = 0; k < P.replicas; k++) {
                const float4 x = __ldcg(P.cells + (size_t)k * P.cp.cells + rows0 + i);
                a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
            }
        s_cells[i] = a;
    }
    for(int i = threadIdx.x; i < n; i += 4 * ROWS) s_taps[i] = P.taps[i];
    __syncthreads();
    const int q = threadIdx.x >> 2, r = rows0 + q;
    const float e = r < (int)P.nR ? P.row_dev[r] : 0.0f;
    float2 acc = make_float2(0.f, 0.f);
    for(int t = threadIdx.x & 3; t < n; t += 4) {
        const float4 c = s_taps[t], a = s_cells[q + t];
        const float mx = fmaf(e, a.x, a.z), my = fmaf(e, a.y, a.w);
        acc.x = fmaf(c.x, a.x, fmaf(-c.y, a.y, fmaf(c.z, mx, fmaf(-c.w, my, acc.x))));
        acc.y = fmaf(c.x, a.y, fmaf(c.y, a.x, fmaf(c.z, my, fmaf(c.w, mx, acc.y))));
    }
    for(int o = 1; o < 4; o <<= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if((threadIdx.x & 3) == 0 && r < (int)P.nR) {
        const float2 v = __ldcg(P.out + r);
        P.out[r] = row_on(nonempty, (int)P.nR, P.overlap, r) ? make_float2(v.x + acc.x, v.y + acc.y) : make_float2(0.f, 0.f);
    }
}

// ---- range filter over the cell rows ----------------------------------------
// A CTA of WARPS warps filters 32 columns x WARPS * kFilterRows output rows. The
// cell rows it needs are staged in shared memory by 16-byte asynchronous
// copies, kFilterChunk rows at a time, all of them in flight together. Each thread holds one column and kFilterRows consecutive output
// rows and walks the staged cells; the taps of its rows slide through
// registers (the tap of row q at a cell is the tap of row q + 1 at the next).
// What is in the ping already is loaded before the cells arrive. Bound by
// issue; 33 taps, us per filter: 512 x 1024 20.2 with 8 rows per thread, 4
// warps and the ping loaded last, 16.5 with 4 rows and 8 warps (fewer
// registers, twice the warps); 512 x 4096 73 -> 49.
// taps[t] = {P[t - 1], D[t - 1]}, t = 0 .. H, zero beyond.
constexpr int kFilterWarps = 8, kFilterRows = 4;
constexpr int kFilterChunk = 72;           // staged cell rows: a 33-tap pulse's tile in one chunk

// Entries of the tap table: H + 1 taps, the sliding window's steps beyond
// them, rounded up to whole blocks of kFilterRows.
__host__ __device__ __forceinline__ int cell_tap_entries(int H) { return (H + 2 * kFilterRows - 1) / kFilterRows * kFilterRows; }
__host__ __device__ __forceinline__ size_t filter_smem(int H)
{
    return (size_t)cell_tap_entries(H) * sizeof(float4) + (size_t)kFilterChunk * 32 * sizeof(float4);
}

// Columns [32 tile_c, +32) and rows [WARPS kFilterRows tile_r, + WARPS
// kFilterRows) of a ping. Called by 32 WARPS threads; synchronises.
template <int WARPS, bool FLOOR = false>
__device__ __forceinline__ void filter_tile(const CellPing& P, int tile_c, int tile_r, float4* s_raw,
                                            const uint32_t* nonempty)
{
    constexpr int kThreads = 32 * WARPS, kFilterTile = WARPS * kFilterRows;
    __shared__ int s_on[kFilterTile];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4* s_taps = s_raw;
    float4* s_cells = s_raw + cell_tap_entries(P.cp.taps);
    const int rows0 = tile_r * kFilterTile, r0 = rows0 + warp * kFilterRows, col = tile_c * 32 + lane;
    const int span = P.cp.taps + kFilterRows;                  // cells that reach a thread's rows
    const int total = min(P.cp.taps + kFilterTile, P.cp.cells - rows0);   // cells of the tile
    if(tid < kFilterTile) {
        const int r = rows0 + tid;
        s_on[tid] = r < (int)P.nR && row_on(nonempty, (int)P.nR, P.overlap, r) ? 1 : 0;
    }
    for(int i = tid; i < cell_tap_entries(P.cp.taps); i += kThreads) s_taps[i] = P.taps[i];
    const int b = P.col_bearing[col];
    float2 acc[kFilterRows];
    float e[kFilterRows];
    float4 c[kFilterRows];
#pragma unroll
    for(int q = 0; q < kFilterRows; q++) {
        acc[q] = b >= 0 && r0 + q < (int)P.nR ? __ldcg(P.out + (size_t)(r0 + q) * P.nB + b) : make_float2(0.f, 0.f);
        e[q] = r0 + q < (int)P.nR ? P.row_dev[r0 + q] : 0.0f;
        c[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float4* src = P.cells + (size_t)rows0 * P.pitch + tile_c * 32;
    for(int k0 = 0; k0 < total; k0 += kFilterChunk) {
        const int rows = min(kFilterChunk, total - k0);
        if(k0) __syncthreads();
        for(int i = warp; i < kFilterChunk; i += WARPS) {
            float4* dst = s_cells + i * 32 + lane;
            if(i < rows)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)),
                             "l"(src + (size_t)(k0 + i) * P.pitch + lane) : "memory");
            else *dst = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if(FLOOR) {
            // Lobe form: the floor's column joins every column's sums (each thread's own copies).
#pragma unroll
            for(int i = warp; i < kFilterChunk; i += WARPS)
                if(i < rows) {
                    const float4 f = __ldcg(P.cells + (size_t)(rows0 + k0 + i) * P.pitch + P.floor_col);
                    float4& a = s_cells[i * 32 + lane];
                    a = make_float4(a.x + f.x, a.y + f.y, a.z + f.z, a.w + f.w);
                }
        }
        __syncthreads();
        // The thread's cell j (from its first row) is the tile's cell
        // j + warp * kFilterRows; output row r0 + q takes tap j - q there.
        const int j0 = max(0, k0 - warp * kFilterRows), j1 = min(span, k0 + kFilterChunk - warp * kFilterRows);
        for(int j = j0; j < j1; j += kFilterRows) {
            const float4* a_row = s_cells + (j + warp * kFilterRows - k0) * 32 + lane;
#pragma unroll
            for(int u = 0; u < kFilterRows; u++) {
                const float4 a = a_row[u * 32];
                c[u] = s_taps[j + u];
#pragma unroll
                for(int q = 0; q < kFilterRows; q++) {
                    const float4 t = c[(u - q + kFilterRows) % kFilterRows];
                    const float mx = fmaf(e[q], a.x, a.z), my = fmaf(e[q], a.y, a.w);
                    acc[q].x = fmaf(t.x, a.x, fmaf(-t.y, a.y, fmaf(t.z, mx, fmaf(-t.w, my, acc[q].x))));
                    acc[q].y = fmaf(t.x, a.y, fmaf(t.y, a.x, fmaf(t.z, my, fmaf(t.w, mx, acc[q].y))));
                }
            }
        }
    }
    if(b < 0) return;
#pragma unroll
    for(int q = 0; q < kFilterRows; q++)
        if(r0 + q < (int)P.nR) P.out[(size_t)(r0 + q) * P.nB + b] = s_on[warp * kFilterRows + q] ? acc[q] : make_float2(0.f, 0.f);
}

// Row pairs of output row r into the ping, by every thread of the CTA: T of
// storage row r + 1 and M of storage row r.
__device__ __forceinline__ void join_pairs(const CellPing& P, int r, const uint32_t* nonempty)
{
    const bool on = row_on(nonempty, (int)P.nR, P.overlap, r);
    for(int col = threadIdx.x; col < (int)P.pitch; col += blockDim.x) {
        const int b = P.col_bearing[col];
        if(b < 0) continue;
        const float4 t = __ldcg(P.cells + (size_t)(r + 1) * P.pitch + col), m = __ldcg(P.cells + (size_t)r * P.pitch + col);
        P.out[(size_t)r * P.nB + b] = on ? make_float2(t.x + m.z, t.y + m.w) : make_float2(0.f, 0.f);
    }
}

} // namespace

} // namespace rtacx
