// Plain reduction over range cells (see rtacx_cells.cuh): configuration and
// the single-ping kernels.
//
//   k_cells         the sorted samples of one ping into the cell rows;
//   k_cells_filter  the pulse's taps over the cell rows, rows without a
//                   reference window zeroed (k_pairs_join: row pairs);
//   k_cells_1d, k_cells_filter_1d, k_rows_join_1d  the same for 1D sensors,
//                   from the input order.
// Measured against the per-row gathers on the same pings (whole rtacx_reduce,
// us): 2^20 samples, 512 x 1024, 33 taps, narrow beams: 1380 -> 96; 2^22 samples,
// 512 x 4096, wide beams on a floor: 14430 -> 418 (1180 with the whole beam);
// 150003 samples, 387 x 777, 24 taps: 246 -> 42; 20000 samples, 256 x 500, row
// pairs: 94 -> 22. k_cells is bound by the beam lookups' shared memory (single
// tables) and by the FMA pipe (16 copies), at one lookup per (sample, bearing).
// 1D: 20000 samples, 1049 ranges (row by row) 33 -> 11; 3e6 samples, 4096
// ranges, 65 taps 381 -> 38.
#include "rtacx_cells.cuh"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace rtacx {

namespace {

// Warps per CTA: 8, two or three CTAs per SM; with a replicated table one CTA
// of as many warps. Narrow beams' tables (up to 606 taps for 64-bearing
// windows, 1006 for 128) fit 16 times: a copy for each pair of banks, so that
// a lookup takes two wavefronts instead of three and more, and four samples'
// lookups in flight pay off. 2^20 samples, 512 x 1024: 111 -> 101 us; 150003
// samples, 387 x 777: 49 -> 46.6. Fewer warps (20): 109.
__host__ __device__ constexpr int cell_warps(int bpl, int copies) { return copies == 1 ? 8 : bpl == 2 ? 24 : 16; }
constexpr int kTableCopies = 16;
constexpr size_t kMaxCellBytes = (size_t)1 << 30;      // cell rows of one context
constexpr size_t kMaxCellSmem = 226 * 1024;
constexpr double kMaxKnot = 0.01;
constexpr uint32_t kCellBins = 12288;
// Fewest samples of a warp's unit (20000 samples, 256 x 500, us per ping: 8
// 29.0, 16 26.1, 32 25.9; 150003 samples: 64 7 us more than 32). Units of equal
// size for the resident warps instead of 128 samples each end together: 2^20
// samples, 512 x 1024, 135 -> 124 us.
constexpr uint32_t kMinUnit = 32;

size_t cells_smem(int W, bool pairs, int bpl, int copies)
{
    return cell_warps(bpl, copies) * (pairs ? sizeof(CellWarpSmem<true>) : sizeof(CellWarpSmem<false>)) +
           (size_t)(W + 2) * copies * sizeof(float2);
}

// begin (null: 0), end: where the sorted samples that it takes start and end.
template <int BPL, bool SHARED, bool PAIR, int COPIES, bool FLOOR = false>
__global__ void __launch_bounds__(32 * cell_warps(BPL, COPIES), COPIES > 1 ? 1 : BPL == 2 ? 3 : 2)
k_cells(const CellPing ping, const uint32_t* begin, const uint32_t* end, uint32_t min_unit)
{
    constexpr int kWarps = cell_warps(BPL, COPIES);
    CellPing P = ping;
    extern __shared__ __align__(16) unsigned char s_raw[];
    CellWarpSmem<PAIR>& S = reinterpret_cast<CellWarpSmem<PAIR>*>(s_raw)[threadIdx.x >> 5];
    float2* tab = reinterpret_cast<float2*>(s_raw + kWarps * sizeof(CellWarpSmem<PAIR>));
    chain_next();
    load_beam_table<COPIES>(tab, P.beam, P.beam_axis, threadIdx.x, 32 * kWarps);
    __syncthreads();
    chain_wait();
    P.sorted = after_chain(P.sorted);
    BeamLookup<COPIES> beam;
    beam.init(P.beam_axis);
    tab += threadIdx.x & (COPIES - 1);
    const uint32_t first = begin ? *after_chain(begin) : 0u, m = *after_chain(end) - first;
    // Equal units, so that the resident warps all end in the same round.
    const uint64_t warps = (uint64_t)gridDim.x * kWarps, rounds = (m + warps * kUnit - 1) / (warps * kUnit);
    const uint32_t unit = max(min_unit, (uint32_t)((m + warps * rounds - 1) / max(warps * rounds, (uint64_t)1)));
    for(uint64_t u = (uint64_t)(blockIdx.x * kWarps + (threadIdx.x >> 5)) * unit; u < m; u += warps * unit)
        accumulate_unit<BPL, SHARED, PAIR, FLOOR>(P, first + (uint32_t)u, min(unit, m - (uint32_t)u), blockIdx.y, gridDim.y, S,
                                                  tab, beam);
}

using CellsFn = void (*)(const CellPing, const uint32_t*, const uint32_t*, uint32_t);
CellsFn lobe_fn(int bpl) { return bpl == 4 ? k_cells<4, false, false, kTableCopies, true> : k_cells<2, false, false, kTableCopies, true>; }
CellsFn cells_fn(int bpl, bool shared_out, bool pairs, int copies)
{
    if(copies > 1) return bpl == 4 ? k_cells<4, false, false, kTableCopies> : k_cells<2, false, false, kTableCopies>;
    if(pairs)
        return shared_out ? (bpl == 4 ? k_cells<4, true, true, 1> : k_cells<2, true, true, 1>)
                          : (bpl == 4 ? k_cells<4, false, true, 1> : k_cells<2, false, true, 1>);
    return shared_out ? (bpl == 4 ? k_cells<4, true, false, 1> : k_cells<2, true, false, 1>)
                      : (bpl == 4 ? k_cells<4, false, false, 1> : k_cells<2, false, false, 1>);
}
CellsFn cells_fn(const Context& c) { return cells_fn(c.cell_bpl, c.cell_shared, c.cell_pairs, c.cell_copies); }
size_t cells_smem(const Context& c) { return cells_smem((int)c.W, c.cell_pairs, c.cell_bpl, c.cell_copies); }

// Zeroes what a ping's passes add into: the bin totals, the range-bin bitmap,
// the cell rows and the ping (8-byte stores: the ping's alignment). Notes the
// order that the ping leaves in the sorted scratch.
__global__ void k_cells_clear(unsigned long long* __restrict__ sorted_order, unsigned long long order,
                              uint32_t* __restrict__ totals, uint32_t n_totals, uint32_t* __restrict__ bits,
                              uint32_t n_bits, float4* __restrict__ cells, uint64_t n_cells, float2* __restrict__ out,
                              uint64_t n_out)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    chain_next();
    chain_wait();
    if(i0 == 0) *sorted_order = order;
    for(uint64_t i = i0; i < n_totals; i += stride) totals[i] = 0u;
    for(uint64_t i = i0; i < n_bits; i += stride) bits[i] = 0u;
    for(uint64_t i = i0; i < n_cells; i += stride) cells[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for(uint64_t i = i0; i < n_out; i += stride) out[i] = make_float2(0.f, 0.f);
}

template <bool FLOOR>
__global__ void __launch_bounds__(32 * kFilterWarps)
k_cells_filter(const CellPing ping, const uint32_t* nonempty)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    CellPing P = ping;
    chain_next();
    chain_wait();
    P.cells = after_chain(P.cells);
    P.out = after_chain(P.out);
    filter_tile<kFilterWarps, FLOOR>(P, blockIdx.x, blockIdx.y, reinterpret_cast<float4*>(s_raw), after_chain(nonempty));
}

// One CTA per output row.
__global__ void __launch_bounds__(256)
k_pairs_join(const CellPing ping, const uint32_t* nonempty)
{
    CellPing P = ping;
    chain_next();
    chain_wait();
    P.cells = after_chain(P.cells);
    join_pairs(P, blockIdx.x, after_chain(nonempty));
}

// 1D pings: the samples into the cells (or rows), then the taps.
constexpr int kThreads1D = 256;
template <bool ROWS>
__global__ void __launch_bounds__(kThreads1D)
k_cells_1d(const CellPing P, const BinParams p, const float* __restrict__ samples, uint64_t n,
           uint32_t* __restrict__ nonempty, float4* __restrict__ copy)
{
    extern __shared__ uint32_t s_bits[];
    const uint32_t words = (P.nR + 31) / 32;
    chain_next();
    for(uint32_t i = threadIdx.x; i < words; i += kThreads1D) s_bits[i] = 0u;
    __syncthreads();
    chain_wait();
    const uint64_t chunk = (n + gridDim.x - 1) / gridDim.x, begin = blockIdx.x * chunk;
    accumulate_1d<ROWS>(P, p, after_chain(samples), begin, min(begin + chunk, n), copy_1d(P, ROWS, blockIdx.x), s_bits, copy);
    __syncthreads();
    for(uint32_t i = threadIdx.x; i < words; i += kThreads1D)
        if(s_bits[i]) atomicOr(&nonempty[i], s_bits[i]);
}

__global__ void __launch_bounds__(4 * kFilterRows1D)
k_cells_filter_1d(const CellPing ping, const uint32_t* nonempty)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    CellPing P = ping;
    chain_next();
    chain_wait();
    P.cells = after_chain(P.cells);
    P.out = after_chain(P.out);
    filter_rows_1d<kFilterRows1D>(P, blockIdx.x, reinterpret_cast<float4*>(s_raw), after_chain(nonempty));
}

__global__ void k_rows_join_1d(const CellPing ping, const uint32_t* nonempty)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    CellPing P = ping;
    chain_next();
    chain_wait();
    P.cells = after_chain(P.cells);
    if(r < (int)P.nR) join_rows_1d(P, r, after_chain(nonempty));
}

} // namespace

void free_cells(Context& c)
{
    if(c.d_cells) cudaFree(c.d_cells);
    c.d_cells = nullptr;
    c.d_nonempty = nullptr;
    c.lobe_on = false;
    c.cells_on = false;
}

void ensure_cells(Context& c)
{
    if(!c.cells_on || c.d_cells || cudaMalloc(&c.d_cells, c.cell_bytes) == cudaSuccess) return;
    cudaGetLastError();
    free_cells(c);
}

void bind_cells(Context& c)
{
    c.cell.pulse = c.d_pulse; c.cell.beam = c.d_beam; c.cell.ranges = c.d_ranges;
    if(c.lobe_on) {
        CellPing& L = c.lobe;
        L.pulse = c.cell.pulse; L.ranges = c.cell.ranges; L.taps = c.cell.taps; L.row_dev = c.cell.row_dev;
        L.col_bearing = c.cell.col_bearing;
    }
}

namespace {

// The best line (least squares) through the rows' float ranges, and how far
// each row lies from it, in taps.
struct RowFit {
    double k = 0.0, spacing = 0.0, R0 = 0.0, worst = 0.0, last = 0.0;   // taps per metre; metres; taps; metres
    std::vector<float> dev;
};

bool fit_rows(const Context& c, RowFit& f)
{
    const int nR = (int)c.nR;
    if(nR < 2 || c.H < 1) return false;
    f.k = (double)c.red.range_axis.k_hi + (double)c.red.range_axis.k_lo;
    double sr = 0.0, sx = 0.0;
    for(int r = 0; r < nR; r++) {
        sr += c.ranges[r];
        sx += ((double)r - 0.5 * (nR - 1)) * c.ranges[r];
    }
    f.spacing = sx / ((double)nR * ((double)nR * nR - 1.0) / 12.0);
    f.R0 = sr / nR - 0.5 * (nR - 1) * f.spacing;
    if(!(f.spacing > 0.0) || !std::isfinite(f.spacing)) return false;
    f.dev.resize(nR);
    for(int r = 0; r < nR; r++) {
        const double e = f.k * (f.R0 + r * f.spacing - c.ranges[r]);
        f.dev[r] = (float)e;
        f.worst = std::max(f.worst, std::fabs(e));
        f.last = std::max(f.last, std::fabs((double)c.ranges[r]));
    }
    return true;
}

// Cell coordinate y = travel / spacing + b, storage row floor(y) + shift.
bool set_cell_axis(CellParams& cp, const RowFit& f, double b, int shift, int cells, double knot, int taps)
{
    const double kc = 1.0 / f.spacing;
    cp.k_hi = (float)kc;
    cp.k_lo = (float)(kc - (double)cp.k_hi);
    cp.b_row = (float)(std::floor(b) + shift);
    cp.b_frac = (float)(b - std::floor(b));
    cp.knot = (float)knot;
    cp.cells = cells;
    cp.taps = taps;
    return std::fabs(b) + cells <= (double)(1 << 21);
}

// Half of the travels that reach a row, with a hair of the spacing for the
// float cell index and the rows' deviations.
double row_reach(const Context& c, const RowFit& f)
{
    return 0.5 * ((double)c.H / f.k) * (1.0 + 1.0 / c.H) + 1e-4 * f.spacing + f.worst / f.k + 1e-6 * f.last;
}

// Knot cells: the pulse's taps one output range apart, up to what the knot
// band covers (it costs one product per row and pair, so it is kept under a
// hundredth of a cell), and every row's PSF support inside its reference
// window, so that the window only decides whether the row is on.
bool knot_cells(Context& c, const RowFit& f)
{
    const int nR = (int)c.nR, H = (int)c.H;
    // What moves a row's knots against the grid: its own deviation, the tap
    // spacing's over half the pulse, and the rounding of travel - range.
    const double knot = 1.01 * (f.worst + std::fabs(f.k * f.spacing - 1.0) * (0.5 * H + 1.0)) + 2e-6 + 1.5e-7 * H;
    if(!(knot <= kMaxKnot)) return false;
    for(int r = 0; r < nR; r++)
        if(c.support[r].x < std::max(0ll, (long long)r - c.overlap) ||
           c.support[r].y > std::min((long long)nR - 1, (long long)r + c.overlap)) return false;
    return set_cell_axis(c.cell.cp, f, 0.5 * H - 0.5 - f.R0 / f.spacing, 1, nR + H, knot, H);
}

// Window x cell block bins, the blocks as small as kCellBins allows.
void set_cell_blocks(BinParams& bin, int cells)
{
    for(bin.cell_shift = 0;; bin.cell_shift++) {
        bin.cell_blocks = (uint32_t)((cells - 1) >> bin.cell_shift) + 1u;
        if(bin.nBB * bin.cell_blocks <= kCellBins || bin.cell_blocks == 1u) break;
    }
    bin.nBins = bin.nBB * bin.cell_blocks;
}

// Taps of the knot cells' filter.
std::vector<float4> cell_taps(const Context& c, const RowFit& f)
{
    const int H = (int)c.H;
    const double kappa = f.k * f.spacing;
    std::vector<float4> taps((size_t)cell_tap_entries(H), make_float4(0.f, 0.f, 0.f, 0.f));
    for(int i = -1; i < H; i++) {
        double p[2], d[2];
        for(int q = 0; q < 2; q++) {
            const double lo = i >= 0 ? c.pulse[2 * (size_t)i + q] : 0.0, hi = i + 1 < H ? c.pulse[2 * ((size_t)i + 1) + q] : 0.0;
            p[q] = lo + (hi - lo) * (kappa - 1.0) * ((double)i - (0.5 * H - 0.5));
            d[q] = (hi - lo) * kappa;
        }
        taps[i + 1] = make_float4((float)p[0], (float)p[1], (float)d[0], (float)d[1]);
    }
    return taps;
}

void set_ping_params(Context& c)
{
    CellPing& P = c.cell;
    P.range_axis = c.red.range_axis; P.beam_axis = c.red.beam_axis;
    P.key = c.key; P.overlap = c.overlap;
    P.nR = c.nR; P.nB = c.nB;
    P.floor = 0.0f; P.floor_col = -1;
}

// A beam table that is one level, not zero, at both ends: the texels between
// its flat tails (the lobe), how far the lobe reaches, and the sample bearings
// from which every output bearing lies within the table.
struct Lobe { int first = 0, last = 0; float level = 0.0f, in_lo = 0.0f, in_hi = 0.0f; double support = 0.0; };

bool find_lobe(const Context& c, Lobe& l)
{
    const int W = (int)c.W;
    l.level = c.beam[0];
    if(W < 8 || l.level == 0.0f || !std::isfinite(l.level) || c.beam[W - 1] != l.level) return false;
    l.first = 0;
    l.last = W - 1;
    while(l.first < W && c.beam[l.first] == l.level) l.first++;
    while(l.last >= 0 && c.beam[l.last] == l.level) l.last--;
    if(l.first > l.last) return false;
    const AxisLerp& ax = c.red.beam_axis;
    const double k = (double)ax.k_hi + (double)ax.k_lo;
    auto at = [&](double x) { return (x - (double)ax.c) / k; };
    l.support = std::max(std::fabs(at(l.first - 1)), std::fabs(at(l.last + 1)));
    const auto mm = std::minmax_element(c.bearings.begin(), c.bearings.end());
    l.in_lo = (float)(*mm.second + at(2.0));             // two texels from the ends
    l.in_hi = (float)(*mm.first + at(W - 3.0));
    return k > 0.0 && l.support > 0.0 && l.in_lo < l.in_hi;
}

// Lobe form of a sensor whose wide beam is a lobe on a flat floor: beam =
// floor + lobe, so a sample inside [in_lo, in_hi] adds floor v to the cell
// sums of all bearings (one column more, which the filter adds to the others)
// and the lobe's part to the few bearings that the lobe reaches, in windows
// like a narrow beam's. The other samples and those next to a knot take the
// whole table, in the last window of the sort; their bearings lie side by side
// on the lanes, since row by row the reductions bound it (161 -> 61 us against
// the order that spares the table's banks). Whole pings without / with, us:
// 2^22 samples, 512 x 4096 1178 -> 418; 2^20, 600 x 2048 429 -> 138; 2^16, 512 x
// 128 60 -> 40; 2^16, 300 x 1024 58 -> 47; 2^14, 600 x 300 43 -> 50; 2^14, 300 x
// 1024 38 -> 52: one more launch and short lists, hence kLobeFrom (samples x
// bearings).
constexpr uint64_t kLobeFrom = 1ull << 24;

} // namespace

// 1D sensors: knot cells where the pulse's taps allow them, else row by row.
bool configure_cells_1d(Context& c, ConfigArena& arena)
{
    free_cells(c);
    RowFit f;
    if(c.dims != 1 || !fit_rows(c, f)) return false;
    const int nR = (int)c.nR;
    bool ok = filter_smem_1d((int)c.H, kFilterRows1D) <= 200 * 1024 && knot_cells(c, f);
    c.cell_pairs = false;
    c.cell_rows = !ok;
    if(c.cell_rows) {
        const double reach = row_reach(c, f), rows = std::floor(2.0 * reach / f.spacing) + 1.0;
        if(!(rows <= 64.0)) return false;
        c.cell.rows = (int)rows;
        // First row reached: floor(y) + 1 with y = (travel - reach - R0) / spacing.
        ok = set_cell_axis(c.cell.cp, f, -(reach + f.R0) / f.spacing, c.cell.rows, nR + c.cell.rows - 1, 0.0, (int)c.H);
    }
    if(!ok || raise_smem_limit((const void*)k_cells_filter_1d, filter_smem_1d(c.cell_rows ? 1 : (int)c.H, kFilterRows1D)) != cudaSuccess)
        return false;
    arena.table(c.cell.row_dev, f.dev);
    arena.table(c.cell.taps, cell_taps(c, f));
    arena.table(c.d_nonempty, std::vector<uint32_t>((nR + 127) / 128 * 4, 0u));
    c.cell_bytes = (size_t)kReplicas1D * (c.cell_rows ? nR * sizeof(float2) : c.cell.cp.cells * sizeof(float4));
    set_ping_params(c);
    c.cell.pitch = 1;
    c.cells_on = true;
    return true;
}

// Row by row is bound by the reductions queueing at the output rows, the
// sorted gather by its launches until the samples outweigh them. Whole pings,
// us, row by row / sorted: 1049 ranges, 5 rows, 2^15 samples 19 / 33, 2^17 31 /
// 35, 2^19 134 / 51; 4096 ranges, 32 rows, 2^15 32 / 33, 2^17 82 / 40; 9 rows
// 2^17 30 / 35. They meet near 512 reductions per row, or a million in all.
// 2D: see cell_from_2d.
bool takes_cells(const Context& c, uint64_t n)
{
    if(!c.cells_on || !c.d_cells) return false;
    if(c.dims == 1) return !c.cell_rows || n * (uint64_t)c.cell.rows <= std::min<uint64_t>(512ull * c.nR, 1ull << 20);
    return n == 0 || n >= c.cell_from;
}

// More than one copy where a row takes more than 8 reductions, or a cell 48 (4
// copies; 8 from 2^18 samples, below which clearing them costs more than they
// save).
int cell_replicas(const Context& c, uint64_t n)
{
    if(c.cell_rows) return n * (uint64_t)c.cell.rows > 8ull * c.nR ? kReplicas1D : 1;
    return n >= (1ull << 18) ? kReplicas1D : n >= 48ull * c.cell.cp.cells ? 4 : 1;
}

// 16-byte words of the cell rows that a 1D ping uses.
uint64_t cell_words_1d(const Context& c, uint64_t n)
{
    const uint64_t copies = (uint64_t)cell_replicas(c, n);
    return c.cell_rows ? (copies * c.nR + 1) / 2 : copies * c.cell.cp.cells;
}

// Samples from which a 2D ping takes the cell form. It clears and filters all
// cell rows whatever the sample count; the gathers' work follows the samples,
// and the tiles that any sample reaches. Whole pings, us, cell form / gather, 33
// taps, uniform scene (half of the samples in 1 % of the ranges): 512 x 1024
// 2^9 56 / 62; 512 x 2048 2^9 66 / 66; 512 x 4096 2^7 91 / 89 (76), 2^9 91 / 85
// (99), 2^12 89 / 83 (115), 2^13 87 / 89 (122); 1024 x 4096 2^10 144 / 93 (103),
// 2^14 138 / 117 (130), 2^15 138 / 150 (153), with 9 taps 2^10 103 / 96 (87),
// 2^12 99 / 91 (116); 1024 x 8192 2^10 244 / 126 (132), 2^15 234 / 199 (218),
// 2^16 236 / 289 (324). Wide beams: 1024 x 8192 2^14 302 / 224 (234), 2^15 298 /
// 339 (355). Row pairs, which have no filter: 1024 x 4096 2^8 70 / 62 (64), 2^9
// 68 / 72 (74); 1024 x 8192 2^10 107 / 101 (101), 2^12 113 / 126 (122). So the
// cell form takes 40 us and, per million entries, 12 and 0.36 per tap (7.5 for
// pairs); the gather 65 us (52) at 64 samples, up to 10 more with every
// doubling, in the end 2 us per 1000 samples (wide beams 4 per 1024 bearings).
uint64_t cell_from_2d(const Context& c)
{
    const double entries = 1e-6 * (double)c.cell.cp.cells * c.cell.pitch;
    const double cells = 40.0 + entries * (c.cell_pairs ? 7.5 : 12.0 + 0.36 * c.H);
    double from = 64.0 * std::exp2(std::min((cells - (c.cell_pairs ? 52.0 : 65.0)) / 10.0, 40.0));
    if(!c.cell_pairs)
        from = std::min(from, 1e3 * (cells - 55.0 - 9.0 * entries) / (c.cell_shared ? std::max(2.0, c.nB / 256.0) : 2.0));
    return from > 100.0 ? (uint64_t)from : 0;
}

// Decides whether a configured 2D sensor takes the cell form and builds its
// tables: row pairs where no travel reaches three rows, else knot cells where
// the pulse's taps allow them, and the cell rows and the beam table have to
// fit (everything else keeps the per-row gathers). Returns whether the form
// is on.
bool configure_cells(Context& c, double beam_support, ConfigArena& arena)
{
    free_cells(c);
    const int nR = (int)c.nR, nB = (int)c.nB, H = (int)c.H, W = (int)c.W;
    RowFit f;
    if(c.dims != 2 || !fit_rows(c, f)) return false;
    CellParams& cp = c.cell.cp;
    c.cell_rows = false;
    const double reach = row_reach(c, f);
    c.cell_pairs = reach < f.spacing;
    // Pairs: the first row reached is floor(y) + 1, its storage row one more.
    if(!(c.cell_pairs ? set_cell_axis(cp, f, -(reach + f.R0) / f.spacing, 2, nR + 1, 0.0, H) : knot_cells(c, f))) return false;
    // Beam coordinates far below the rounding trick's 2^22.
    const auto mm = std::minmax_element(c.bearings.begin(), c.bearings.end());
    const double fan = (double)*mm.second - (double)*mm.first, span = c.span;
    if((fan + 4.0 * span) / span * W + W > (double)(1 << 20)) return false;
    c.cell.theta_lo = (float)(*mm.first - 2.0 * span);
    c.cell.theta_hi = (float)(*mm.second + 2.0 * span);

    // Windows. Narrow beams: equal intervals of sample bearings, each with the
    // consecutive output bearings that its samples reach; every sample is in
    // exactly one. As few as keep the bearings of each within 64 (else 128),
    // unless a window would be narrower than half a beam's half width (its
    // sums would be flushed after too few samples). Wide beams: the bearings
    // are shared out among windows that all take every sample.
    std::vector<int> sorted_b(nB);
    std::iota(sorted_b.begin(), sorted_b.end(), 0);
    std::stable_sort(sorted_b.begin(), sorted_b.end(), [&](int x, int y) { return c.bearings[x] < c.bearings[y]; });
    std::vector<double> theta_sorted(nB);
    for(int i = 0; i < nB; i++) theta_sorted[i] = c.bearings[sorted_b[i]];
    double lo = 0.0, hi = 0.0;
    std::vector<int2> span_of;              // [first, end) sorted bearings of each window
    auto find_windows = [&](double support) {
        lo = (double)*mm.first - support;
        hi = (double)*mm.second + support;
        const int max_windows = std::max(1, (int)std::min(4096.0, (hi - lo) / (0.5 * support)));
        // The most bearings within two supports: some window takes them all,
        // whatever the windows, so where they do not fit none are tried (for
        // bearings in a cluster the search took up to 0.1 s).
        int densest = 0;
        for(int first = 0, end = 0; first < nB; first++) {
            while(end < nB && theta_sorted[end] <= theta_sorted[first] + 2.0 * support) end++;
            densest = std::max(densest, end - first);
        }
        for(int cand = densest <= 64 ? 2 : densest <= 128 ? 4 : 6; cand <= 4; cand += 2)
            for(int w = std::max(1, nB / (32 * cand)); w <= max_windows; w++) {
                const double step = (hi - lo) / w, slack = 1e-5 * (hi - lo) + support;   // 1e-5: the float window index
                bool fits = true;
                span_of.clear();
                for(int q = 0; q < w && fits; q++) {
                    const auto f = std::lower_bound(theta_sorted.begin(), theta_sorted.end(), lo + q * step - slack);
                    const auto e = std::upper_bound(f, theta_sorted.end(), lo + (q + 1) * step + slack);
                    span_of.push_back(make_int2((int)(f - theta_sorted.begin()), (int)(e - theta_sorted.begin())));
                    fits = e - f <= 32 * cand;
                }
                if(fits) return cand;
            }
        return 0;
    };
    int bpl = find_windows(beam_support);
    const bool shared_out = bpl == 0;
    if(shared_out) bpl = nB > 64 ? 4 : 2;
    Lobe lobe;
    const bool with_lobe = shared_out && !c.cell_pairs && nB > 128 && find_lobe(c, lobe);
    const int len = 32 * bpl;
    const int copies = !shared_out && !c.cell_pairs && cells_smem(W, false, bpl, kTableCopies) <= kMaxCellSmem ? kTableCopies : 1;
    // Order of the bearings in a window. For one sample the table entries of
    // two bearings differ by their distance in taps, whatever the sample;
    // lanes whose distances differ modulo the 16 eight-byte banks of shared
    // memory never conflict. Bearings sorted by that remainder and dealt to
    // the groups of 16 lanes in turn are about one bank apart: 3.1 to 3.5
    // wavefronts per lookup instead of 3.8 to 4.8 in the bearings' own order
    // (counted for the tables of the imaging sensors).
    const double kb = (double)c.red.beam_axis.k_hi;
    auto deal = [&](std::vector<int> order, std::vector<int>& pos, size_t at) {
        if(copies > 1) { std::copy(order.begin(), order.end(), pos.begin() + at); return; }
        auto bank = [&](int i) { const double x = (double)c.bearings[i] * kb; return x - 16.0 * std::floor(x / 16.0); };
        std::stable_sort(order.begin(), order.end(), [&](int a, int d) { return bank(a) < bank(d); });
        const size_t groups = std::max<size_t>(1, (order.size() + 15) / 16);
        for(size_t q = 0; q < order.size(); q++) pos[at + (q % groups) * 16 + q / groups] = order[q];
    };
    std::vector<int> pos;
    if(shared_out) {
        const int wins = (nB + len - 1) / len;
        pos.assign((size_t)wins * len, -1);
        deal(sorted_b, pos, 0);
    }
    else {
        pos.assign(span_of.size() * len, -1);
        for(size_t w = 0; w < span_of.size(); w++)
            deal(std::vector<int>(sorted_b.begin() + span_of[w].x, sorted_b.begin() + span_of[w].y), pos, w * len);
    }
    c.cell_bpl = bpl;
    c.cell_shared = shared_out;
    c.cell_copies = copies;
    c.cell.windows = (int)(pos.size() / len);
    // Sort order: window x cell block, with as many bins as the pipelined
    // scatter takes at one reservation batch per thread.
    BinParams& bin = c.cell_bin;
    bin = c.bin;
    bin.cell = cp;
    bin.nBB = shared_out ? 1u : (uint32_t)span_of.size();
    bin.bb_scale = (float)(bin.nBB / (hi - lo));
    bin.bb_offset = (float)(-lo * (bin.nBB / (hi - lo)));
    set_cell_blocks(bin, cp.cells);
    c.cell.win_scale = bin.bb_scale;
    c.cell.win_offset = bin.bb_offset;
    // Columns: the lanes' order for shared-out windows (whole rows of 512
    // bytes per reduction), the bearings' own order for overlapping ones.
    // (and, with one more for the floor, where the lobe form has such).
    const bool lane_order = shared_out && !with_lobe;
    const uint32_t pitch = lane_order ? (uint32_t)pos.size() : (uint32_t)((nB + (with_lobe ? 1 : 0) + 31) / 32 * 32);
    c.cell.pitch = pitch;
    std::vector<int> col(pos.size()), col_bearing(pitch, -1);
    std::vector<float> theta(pos.size(), c.bearings[sorted_b[nB - 1]]);
    for(size_t p = 0; p < pos.size(); p++) {
        col[p] = pos[p] < 0 ? -1 : lane_order ? (int)p : pos[p];
        if(pos[p] < 0) continue;
        theta[p] = c.bearings[pos[p]];
        col_bearing[col[p]] = pos[p];
    }
    c.cell_bytes = (size_t)cp.cells * pitch * sizeof(float4);
    if(c.cell_bytes > kMaxCellBytes || cells_smem(c) > kMaxCellSmem ||
       (!c.cell_pairs && filter_smem(H) > 200 * 1024)) return false;
    if(raise_smem_limit((const void*)cells_fn(c), cells_smem(c)) != cudaSuccess ||
       (!c.cell_pairs && raise_smem_limit((const void*)k_cells_filter<false>, filter_smem(H)) != cudaSuccess) ||
       cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c.cell_ctas, cells_fn(c), 32 * cell_warps(bpl, copies),
                                                     cells_smem(c)) != cudaSuccess || c.cell_ctas < 1) {
        cudaGetLastError();
        return false;
    }
    arena.table(c.cell.taps, cell_taps(c, f));
    arena.table(c.cell.row_dev, f.dev);
    arena.table(c.d_nonempty, std::vector<uint32_t>((nR + 127) / 128 * 4, 0u));
    arena.table(c.cell.pos_theta, theta);
    arena.table(c.cell.pos_col, col);
    arena.table(c.cell.col_bearing, col_bearing);
    set_ping_params(c);
    c.cells_on = true;
    c.cell_from = cell_from_2d(c);

    // The lobe form's tables.
    if(!with_lobe || (c.lobe_bpl = find_windows(lobe.support)) == 0) return true;
    const int n_lobe = lobe.last - lobe.first + 1, l_len = 32 * c.lobe_bpl, windows = (int)span_of.size();
    const size_t l_smem = cells_smem(n_lobe, false, c.lobe_bpl, kTableCopies);
    if(l_smem > kMaxCellSmem || raise_smem_limit((const void*)lobe_fn(c.lobe_bpl), l_smem) != cudaSuccess ||
       raise_smem_limit((const void*)k_cells_filter<true>, filter_smem(H)) != cudaSuccess) return true;
    c.lobe_on = true;
    std::vector<float> table(n_lobe + 2, 0.0f);
    for(int i = 0; i < n_lobe; i++) table[i + 1] = c.beam[lobe.first + i] - lobe.level;
    // (behind the lobe's windows: the whole beam's, in the bearings' order)
    const size_t whole = (size_t)windows * l_len;
    std::vector<int> l_col(whole + pos.size(), -1);
    std::vector<float> l_theta(whole + pos.size(), c.bearings[sorted_b[nB - 1]]);
    for(int q = 0; q < nB; q++) {
        l_col[whole + q] = sorted_b[q];
        l_theta[whole + q] = c.bearings[sorted_b[q]];
    }
    for(int w = 0; w < windows; w++)
        for(int q = span_of[w].x; q < span_of[w].y; q++) {
            l_col[w * l_len + (q - span_of[w].x)] = sorted_b[q];
            l_theta[w * l_len + (q - span_of[w].x)] = c.bearings[sorted_b[q]];
        }
    CellPing& L = c.lobe;
    L = c.cell;
    L.windows = windows;
    arena.table(L.beam, table);
    arena.table(L.pos_theta, l_theta);
    arena.table(L.pos_col, l_col);
    L.beam_axis.c = (float)(c.red.beam_axis.c - lobe.first);
    L.beam_axis.n = n_lobe;
    L.floor = lobe.level;
    L.floor_col = nB;
    BinParams& lb = c.lobe_bin;
    lb = c.cell_bin;
    lb.split = 1;
    lb.in_lo = lobe.in_lo;
    lb.in_hi = lobe.in_hi;
    lb.nBB = (uint32_t)windows + 1u;
    lb.bb_scale = L.win_scale = (float)(windows / (hi - lo));
    lb.bb_offset = L.win_offset = (float)(-lo * (windows / (hi - lo)));
    set_cell_blocks(lb, cp.cells);
    return true;
}

static rtacx_status run_cells_1d(Context& c, const void* samples, uint64_t n, float2* out, cudaStream_t stream)
{
    CellPing P = c.cell;
    P.cells = c.d_cells;
    P.out = out;
    P.replicas = cell_replicas(c, n);
    const uint64_t cells = cell_words_1d(c, n), cells_out = c.cell_rows && n ? 0 : c.nR;   // (joined rows are all written)
    c.mark(1, false, stream);
    cudaError_t e = launch_chained(k_cells_clear, (uint32_t)std::min<uint64_t>((cells + c.nR + 255) / 256, (uint64_t)c.sm_count * 8),
                                   256, 0, stream, c.d_oor + 2, kInputOrder | n, c.d_totals, 0u, c.d_nonempty, (c.nR + 31) / 32, c.d_cells, cells, out,
                                   cells_out);
    c.mark(1, true, stream);
    if(e == cudaSuccess && n) {
        c.mark(5, false, stream);
        // One record per thread while that fills the SMs, more beyond.
        const uint32_t grid = (uint32_t)std::min<uint64_t>((n + kThreads1D - 1) / kThreads1D, (uint64_t)c.sm_count * 8);
        const size_t bits = (c.nR + 31) / 32 * sizeof(uint32_t);
        auto fn = c.cell_rows ? k_cells_1d<true> : k_cells_1d<false>;
        e = launch_chained(fn, grid, kThreads1D, bits, stream, P, c.bin, static_cast<const float*>(samples), n,
                           c.d_nonempty, c.d_sorted);
        if(e == cudaSuccess)
            e = c.cell_rows ? launch_chained(k_rows_join_1d, (c.nR + 255) / 256, 256, 0, stream, P, c.d_nonempty)
                            : launch_chained(k_cells_filter_1d, (c.nR + kFilterRows1D - 1) / kFilterRows1D, 4 * kFilterRows1D,
                                             filter_smem_1d(P.cp.taps, kFilterRows1D), stream, P, c.d_nonempty);
        c.mark(5, true, stream);
    }
    if(e != cudaSuccess) { cudaGetLastError(); c.error = std::string("cell form: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    return RTACX_OK;
}

rtacx_status run_cells(Context& c, const void* samples, uint64_t n, float2* out, cudaStream_t stream)
{
    if(c.dims == 1) return run_cells_1d(c, samples, n, out, stream);
    CellPing P = c.cell;
    P.cells = c.d_cells;
    P.sorted = c.d_sorted;
    P.out = out;
    const bool lobe = c.lobe_on && n * (uint64_t)c.nB >= kLobeFrom;
    BinParams bin = lobe ? c.lobe_bin : c.cell_bin;
    bin.vec4 = c.bin.vec4;
    bin.echo_flags = c.cell_bin.echo_flags; bin.echo_cycles = c.cell_bin.echo_cycles;
    bin.echo_k_hi = c.cell_bin.echo_k_hi; bin.echo_k_lo = c.cell_bin.echo_k_lo;
    const uint32_t totals = bin.nBins + (bin.nBins + kScanBlock - 1) / kScanBlock;
    const uint64_t cells = (uint64_t)P.cp.cells * P.pitch, cells_out = c.cell_pairs && n ? 0 : (uint64_t)c.nR * c.nB;   // (the pairs' join writes every cell)
    c.mark(1, false, stream);
    cudaError_t e = launch_chained(k_cells_clear, (uint32_t)std::min<uint64_t>((cells + 255) / 256, (uint64_t)c.sm_count * 8),
                                   256, 0, stream, c.d_oor + 2, n ? kBinsOrder | bin.nBins : +kInputOrder,
                                   c.d_totals, totals, c.d_nonempty, (c.nR + 31) / 32, c.d_cells, cells,
                                   out, cells_out);
    c.mark(1, true, stream);
    if(e == cudaSuccess && n) {
        const rtacx_status st = run_sort(c, bin, lobe ? c.lobe_sort : c.cell_sort, samples, n, c.d_nonempty, stream);
        if(st != RTACX_OK) return st;
        c.mark(5, false, stream);
        // As many CTAs as are resident (twice that for wide beams, whose units
        // are long: the SMs' shares even out, 2^22 samples 1240 -> 1222 us);
        // wide beams' windows are also shared out over blockIdx.y where the
        // samples alone leave SMs idle.
        const uint32_t warps = (uint32_t)cell_warps(c.cell_bpl, c.cell_copies);
        const uint32_t resident = (uint32_t)(c.sm_count * c.cell_ctas);
        uint32_t gx = (uint32_t)std::min<uint64_t>((n + kMinUnit * warps - 1) / (kMinUnit * warps),
                                                   c.cell_shared ? 2 * resident : resident);
        uint32_t gy = c.cell_shared ? std::min((uint32_t)P.windows, std::max(1u, resident / gx)) : 1u;
        const uint32_t* split_at = nullptr;
        CellPing whole = P;
        if(lobe) {
            CellPing L = c.lobe;
            L.cells = P.cells; L.sorted = P.sorted; L.out = out;
            // The samples left are few and mostly next to knots (row by row):
            // one per warp, all windows side by side.
            gy = (uint32_t)P.windows;
            gx = std::max(1u, 4 * resident / gy);
            whole.pos_theta = L.pos_theta + (size_t)L.windows * 32 * c.lobe_bpl;
            whole.pos_col = L.pos_col + (size_t)L.windows * 32 * c.lobe_bpl;
            split_at = c.d_offsets + (bin.nBB - 1u) * bin.cell_blocks;
            const uint32_t lw = (uint32_t)cell_warps(c.lobe_bpl, kTableCopies);
            e = launch_chained(lobe_fn(c.lobe_bpl), (uint32_t)std::min<uint64_t>((n + kMinUnit * lw - 1) / (kMinUnit * lw), (uint64_t)c.sm_count),
                               32 * lw, cells_smem(L.beam_axis.n, false, c.lobe_bpl, kTableCopies), stream, L,
                               static_cast<const uint32_t*>(nullptr), split_at, kMinUnit);
        }
        if(e == cudaSuccess)
            e = launch_chained(cells_fn(c), dim3(gx, gy), 32 * warps, cells_smem(c), stream, whole, split_at, c.d_offsets + bin.nBins,
                               lobe ? 1u : kMinUnit);
        P.floor_col = lobe ? c.lobe.floor_col : -1;
        const dim3 fgrid(P.pitch / 32, (c.nR + kFilterWarps * kFilterRows - 1) / (kFilterWarps * kFilterRows));
        if(e == cudaSuccess)
            e = c.cell_pairs ? launch_chained(k_pairs_join, c.nR, std::min(256u, P.pitch), 0, stream, P, c.d_nonempty)
                             : launch_chained(lobe ? k_cells_filter<true> : k_cells_filter<false>, fgrid, 32 * kFilterWarps, filter_smem(P.cp.taps), stream, P,
                                              c.d_nonempty);
        c.mark(5, true, stream);
    }
    if(e != cudaSuccess) { cudaGetLastError(); c.error = std::string("cell form: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    return RTACX_OK;
}

} // namespace rtacx
