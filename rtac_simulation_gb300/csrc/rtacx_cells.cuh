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
#pragma once

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

__device__ __forceinline__ void red_add_f4(float4* addr, float x, float y, float z, float w)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

__device__ __forceinline__ void red_add_f2(float2* addr, float x, float y)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(x), "f"(y) : "memory");
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

// Range cell of a travel and its fraction of the cell: floor and fraction of
// travel * k + b, with the product's exact residual (fmaf) and the low part
// of k added to the fraction (k * travel reaches the row count, a fraction of
// which a plain float product would round away). Returns the cell's storage
// row C + 1 (C = -1: the first cell any row's pulse reaches) or -1 for a
// travel that reaches no row, NaN and infinities included.
__device__ __forceinline__ int range_cell(const CellParams& cp, float travel, float& alpha)
{
    const float prod = travel * cp.k_hi;
    const float err = fmaf(travel, cp.k_hi, -prod);
    const float whole = rintf(prod);
    const float f = (prod - whole) + (err + fmaf(travel, cp.k_lo, cp.b_frac));
    const float fl = floorf(f);
    alpha = f - fl;
    const float row = whole + fl + cp.b_row;      // whole numbers below 2^22: exact
    return row >= 0.0f && row < (float)cp.cells ? (int)row : -1;
}

// ---- the beam table in shared memory ---------------------------------------
// Entry i of the table is the linear piece left of texel i: {value at its
// left end, slope}, entry 0 the rise from the zero border to texel 0, entry W
// the fall after texel W - 1, entry W + 1 zero (every coordinate outside).
// An even table's texel coordinates are half-integers: its entries are stored
// from the middle of the piece, so that the constant of the fraction is a
// whole number either way (see BeamLookup).
__device__ __forceinline__ void load_beam_table(float2* tab, const float* __restrict__ beam_pad, int W, int tid,
                                                int threads)
{
    for(int i = tid; i <= W + 1; i += threads) {
        float2 e = make_float2(0.f, 0.f);
        if(i <= W) {
            const float lo = beam_pad[i], hi = beam_pad[i + 1];
            e.y = hi - lo;
            e.x = (W & 1) ? lo : fmaf(0.5f, e.y, lo);
        }
        tab[i] = e;
    }
}

// Beam weights of one sample at a pair of bearings: x = (theta - theta_b) k +
// c + 1/2 rounded to a whole number by adding 1.5 * 2^23 (the piece's index,
// in the low mantissa bits), the fraction in one more fused multiply-add from
// the exact difference of the constant and that number, then the piece's
// line. An index below 0 or above W lands on the zero entry.
constexpr float kRoundMagic = 12582912.0f;          // 1.5 * 2^23
constexpr uint32_t kRoundMagicBits = 0x4B400000u;

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
        const float f = kRoundMagic + ((ax.n & 1) ? ax.c + 1.0f : ax.c + 0.5f);
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
        const float2 e0 = tab[min(__float_as_uint(yu.x) - kRoundMagicBits, last)];
        const float2 e1 = tab[min(__float_as_uint(yu.y) - kRoundMagicBits, last)];
        return pack2(fmaf(au.x, e0.y, e0.x), fmaf(au.y, e1.y, e1.x));
    }
};

// ---- accumulation of one ping's samples into the cell rows ------------------
// A warp takes units of kUnit consecutive samples of the sorted order (so of
// few cells and, with bearing sub-bins, of few bearings) and, one after the
// other, the segments of 32 BPL bearings that the unit's bearings can reach:
// lane l holds bearings at positions l, l + 32, ... of the segment and the
// sums of three consecutive cells for them in registers. Per chunk of 32
// samples the lanes list the samples of those cells and this segment, in
// shared memory, each value twice (the packed operands); all lanes then walk
// the list. A unit's sums go to the cell rows as 16-byte reductions.
constexpr int kUnit = 128;                 // samples per warp and unit
constexpr int kCellClasses = 3;            // consecutive cells held in registers

struct CellEntry {                          // a listed sample
    f32x2 theta, w0x, w0y, w1x, w1y, pad;
};

struct CellWarpSmem {
    float4 w[kUnit];                        // {w0.x, w0.y, w1.x, w1.y}; row-by-row samples: {v.x, v.y, travel, -}
    float theta[kUnit];
    int cell[kUnit];                        // storage row; -1 dropped; -2 - row: reduced row by row
    CellEntry list[32];
};

// Samples of a unit that fall next to a knot, row by row: the lanes take 32
// rows at a time, then every row's weight is broadcast and reduced into the
// (zeroed) ping.
template <int BPL>
__device__ __forceinline__ void reduce_row_by_row(const CellPing& P, const CellWarpSmem& S, const float2* tab,
                                                  const BeamLookup& beam, const f32x2 (&minus_tb)[BPL / 2],
                                                  const int* s_b, int s)
{
    const int lane = threadIdx.x & 31;
    const float4 w = S.w[s];
    const int C = -2 - S.cell[s] - 1;                       // cell index
    const f32x2 th = pack2(S.theta[s], S.theta[s]);
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
                const int b = s_b[p];
                if(b >= 0) red_add_f2(P.out + (size_t)(r0 + q) * P.nB + b, ux * bv[p], uy * bv[p]);
            }
        }
    }
}

// Accumulates samples [first, first + count) (count <= kUnit) of the sorted
// order into the cell rows, for the segments seg0, seg0 + seg_step, ....
template <int BPL>
__device__ __forceinline__ void accumulate_unit(const CellPing& P, uint32_t first, uint32_t count, int seg0,
                                                int seg_step, CellWarpSmem& S, const float2* tab,
                                                const BeamLookup& beam)
{
    constexpr int NP = BPL / 2;
    const int lane = threadIdx.x & 31;
    float th_lo = INFINITY, th_hi = -INFINITY;
    int c_lo = INT_MAX, any_near = 0;
    __syncwarp();
#pragma unroll
    for(int q = 0; q < kUnit / 32; q++) {
        const uint32_t i = (uint32_t)(q * 32 + lane);
        int cell = -1;
        if(i < count) {
            const float4 rec = __ldcs(P.sorted + first + i);
            float alpha;
            cell = range_cell(P.cp, rec.z, alpha);
            // Bearings far outside (and NaN) move to a bearing that no beam reaches.
            const float th = fminf(fmaxf(rec.w, P.theta_lo), P.theta_hi);
            S.theta[i] = th;
            S.w[i] = make_float4(rec.x, rec.y, alpha * rec.x, alpha * rec.y);
            if(cell >= 0) {
                th_lo = fminf(th_lo, th);
                th_hi = fmaxf(th_hi, th);
                if(!(alpha >= P.cp.knot && alpha <= 1.0f - P.cp.knot)) {
                    S.w[i] = make_float4(rec.x, rec.y, rec.z, 0.0f);
                    cell = -2 - cell;
                    any_near = 1;
                }
                else c_lo = min(c_lo, cell);
            }
        }
        S.cell[i] = cell;
    }
    any_near = __any_sync(0xffffffffu, any_near);
    for(int o = 16; o > 0; o >>= 1) {
        th_lo = fminf(th_lo, __shfl_xor_sync(0xffffffffu, th_lo, o));
        th_hi = fmaxf(th_hi, __shfl_xor_sync(0xffffffffu, th_hi, o));
    }
    c_lo = __reduce_min_sync(0xffffffffu, c_lo);
    __syncwarp();
    for(int seg = seg0; seg < P.segs; seg += seg_step) {
        const float2 reach = P.seg_reach[seg];
        if(!(th_hi >= reach.x && th_lo <= reach.y)) continue;
        const int pos0 = seg * 32 * BPL + lane;
        f32x2 minus_tb[NP];
#pragma unroll
        for(int p = 0; p < NP; p++)
            minus_tb[p] = pack2(-P.pos_theta[pos0 + 64 * p], -P.pos_theta[pos0 + 64 * p + 32]);
        for(int base = c_lo; base != INT_MAX;) {
            f32x2 acc[kCellClasses][NP][4];
#pragma unroll
            for(int k = 0; k < kCellClasses; k++)
#pragma unroll
                for(int p = 0; p < NP; p++)
#pragma unroll
                    for(int e = 0; e < 4; e++) acc[k][p][e] = 0ull;
            int next = INT_MAX;
            uint32_t held = 0;
#pragma unroll 1
            for(uint32_t q = 0; q < count; q += 32) {
                const int i = (int)q + lane;
                const int cell = S.cell[i];
                const float th = cell >= 0 ? S.theta[i] : 0.0f;
                const bool rel = cell >= base && th >= reach.x && th <= reach.y;
                const int off = cell - base;
                if(rel && off >= kCellClasses) next = min(next, cell);
                const uint32_t m0 = __ballot_sync(0xffffffffu, rel && off == 0);
                const uint32_t m1 = __ballot_sync(0xffffffffu, rel && off == 1);
                const uint32_t m2 = __ballot_sync(0xffffffffu, rel && off == 2);
                const int n0 = __popc(m0), n1 = __popc(m1), n2 = __popc(m2);
                if(n0 + n1 + n2 == 0) continue;
                if(rel && off < kCellClasses) {
                    const uint32_t below = (1u << lane) - 1u;
                    const int at = off == 0 ? __popc(m0 & below)
                                 : off == 1 ? n0 + __popc(m1 & below) : n0 + n1 + __popc(m2 & below);
                    const float4 w = S.w[i];
                    CellEntry* e = S.list + at;
                    e->theta = pack2(th, th);
                    e->w0x = pack2(w.x, w.x);
                    e->w0y = pack2(w.y, w.y);
                    e->w1x = pack2(w.z, w.z);
                    e->w1y = pack2(w.w, w.w);
                }
                held |= (n0 ? 1u : 0u) | (n1 ? 2u : 0u) | (n2 ? 4u : 0u);
                __syncwarp();
                int s = 0;
#pragma unroll
                for(int k = 0; k < kCellClasses; k++) {
                    const int end = k == 0 ? n0 : k == 1 ? n0 + n1 : n0 + n1 + n2;
#pragma unroll 2
                    for(; s < end; s++) {
                        const CellEntry& e = S.list[s];
                        const f32x2 th2 = e.theta, w0x = e.w0x, w0y = e.w0y, w1x = e.w1x, w1y = e.w1y;
#pragma unroll
                        for(int p = 0; p < NP; p++) {
                            const f32x2 B = beam(tab, th2, minus_tb[p]);
                            acc[k][p][0] = fma2(w0x, B, acc[k][p][0]);
                            acc[k][p][1] = fma2(w0y, B, acc[k][p][1]);
                            acc[k][p][2] = fma2(w1x, B, acc[k][p][2]);
                            acc[k][p][3] = fma2(w1y, B, acc[k][p][3]);
                        }
                    }
                }
                __syncwarp();
            }
#pragma unroll
            for(int k = 0; k < kCellClasses; k++) {
                if(!(held & (1u << k))) continue;
                float4* row = P.cells + (size_t)(base + k) * P.pitch + pos0;
#pragma unroll
                for(int p = 0; p < NP; p++) {
                    const float2 a = unpack2(acc[k][p][0]), b = unpack2(acc[k][p][1]);
                    const float2 c = unpack2(acc[k][p][2]), d = unpack2(acc[k][p][3]);
                    red_add_f4(row + 64 * p, a.x, b.x, c.x, d.x);
                    red_add_f4(row + 64 * p + 32, a.y, b.y, c.y, d.y);
                }
            }
            base = __reduce_min_sync(0xffffffffu, next);
        }
        if(any_near) {
            int s_b[BPL];
#pragma unroll
            for(int p = 0; p < BPL; p++) s_b[p] = P.pos_bearing[pos0 + 32 * p];
            for(uint32_t q = 0; q < count; q += 32) {
                const int i = (int)q + lane;
                uint32_t m = __ballot_sync(0xffffffffu, S.cell[i] <= -2 && S.theta[i] >= reach.x && S.theta[i] <= reach.y);
                for(; m; m &= m - 1u)
                    reduce_row_by_row<BPL>(P, S, tab, beam, minus_tb, s_b, (int)q + __ffs(m) - 1);
            }
        }
    }
}

// ---- range filter over the cell rows ----------------------------------------
// Thread: one position (bearing) and kFilterRows consecutive output rows. It
// walks the cells that reach them, one 16-byte load each; the taps of the
// kFilterRows rows slide through registers (the tap of row q at a cell is the
// tap of row q + 1 at the next). taps[i] = {P[i], D[i]} for i = -1 ..
// H - 1, zero beyond on both sides by kFilterRows entries.
constexpr int kFilterRows = 8;

__device__ __forceinline__ void filter_rows(const CellPing& P, int pos, int r0, const float4* __restrict__ s_taps,
                                            const int* __restrict__ s_on)
{
    const int n = P.cp.taps + 1;                              // taps i = -1 .. H - 1
    float2 acc[kFilterRows];
    float e[kFilterRows];
    float4 c[kFilterRows];
#pragma unroll
    for(int q = 0; q < kFilterRows; q++) {
        acc[q] = make_float2(0.f, 0.f);
        e[q] = r0 + q < (int)P.nR ? P.row_dev[r0 + q] : 0.0f;
        c[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // Storage row j of cell C = j - 1; row r takes tap index i + 1 = C - r + 1
    // = j - r. Cells j = r0 .. r0 + n - 1 + kFilterRows - 1.
    const float4* col = P.cells + (size_t)r0 * P.pitch + pos;
    const int last = min(n + kFilterRows - 1, P.cp.cells - r0);
    for(int j0 = 0; j0 < last; j0 += kFilterRows) {
        float4 a[kFilterRows];
#pragma unroll
        for(int u = 0; u < kFilterRows; u++)
            a[u] = j0 + u < last ? __ldg(col + (size_t)(j0 + u) * P.pitch) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for(int u = 0; u < kFilterRows; u++) {
            // Row q's tap at cell j0 + u: slot (u - q) mod kFilterRows.
            c[u] = s_taps[j0 + u];
#pragma unroll
            for(int q = 0; q < kFilterRows; q++) {
                const float4 t = c[(u - q + kFilterRows) % kFilterRows];
                const float mx = fmaf(e[q], a[u].x, a[u].z), my = fmaf(e[q], a[u].y, a[u].w);
                acc[q].x = fmaf(t.x, a[u].x, fmaf(-t.y, a[u].y, fmaf(t.z, mx, fmaf(-t.w, my, acc[q].x))));
                acc[q].y = fmaf(t.x, a[u].y, fmaf(t.y, a[u].x, fmaf(t.z, my, fmaf(t.w, mx, acc[q].y))));
            }
        }
    }
    const int b = P.pos_bearing[pos];
    if(b < 0) return;
#pragma unroll
    for(int q = 0; q < kFilterRows; q++) {
        if(r0 + q >= (int)P.nR) break;
        float2* o = P.out + (size_t)(r0 + q) * P.nB + b;
        const float2 v = *o;
        *o = s_on[q] ? make_float2(v.x + acc[q].x, v.y + acc[q].y) : make_float2(0.f, 0.f);
    }
}

} // namespace

} // namespace rtacx
