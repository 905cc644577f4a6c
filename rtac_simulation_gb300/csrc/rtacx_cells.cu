// Plain 2D reduction over range cells (see rtacx_cells.cuh): configuration
// and the single-ping kernels.
//
//   k_cells         the sorted samples of one ping into the cell rows;
//   k_cells_filter  the pulse's taps over the cell rows, rows without a
//                   reference window zeroed.
// Measured against the tensor-core gather on the same pings (whole
// rtacx_reduce, us): 2^20 samples, 512 x 1024, 33 taps, narrow beams: 1384 ->
// 152; 2^22 samples, 512 x 4096, wide beams: 14433 -> 1339; 150003 samples,
// 387 x 777, 24 taps: 246 -> 82. k_cells is bound by the beam lookups' shared
// memory and issue slots, at one lookup per (sample, bearing).
#include "rtacx_bin_device.cuh"
#include "rtacx_cells.cuh"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace rtacx {

namespace {

constexpr int kCellThreads = 256, kCellWarps = kCellThreads / 32;
constexpr size_t kMaxCellBytes = (size_t)1 << 30;      // cell rows of one context
constexpr double kMaxKnot = 0.01;
constexpr uint32_t kCellBins = 12288;

size_t cells_smem(int W, bool pairs)
{
    return kCellWarps * (pairs ? sizeof(CellWarpSmem<true>) : sizeof(CellWarpSmem<false>)) + (size_t)(W + 2) * sizeof(float2);
}

template <int BPL, bool SHARED, bool PAIR>
__global__ void __launch_bounds__(kCellThreads, BPL == 2 ? 3 : 2)
k_cells(const CellPing P, const uint32_t* __restrict__ total, uint32_t unit)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    CellWarpSmem<PAIR>& S = reinterpret_cast<CellWarpSmem<PAIR>*>(s_raw)[threadIdx.x >> 5];
    float2* tab = reinterpret_cast<float2*>(s_raw + kCellWarps * sizeof(CellWarpSmem<PAIR>));
    load_beam_table(tab, P.beam, P.beam_axis.n, threadIdx.x, kCellThreads);
    __syncthreads();
    BeamLookup beam;
    beam.init(P.beam_axis);
    const uint32_t m = *total;
    for(uint64_t u = (uint64_t)(blockIdx.x * kCellWarps + (threadIdx.x >> 5)) * unit; u < m;
        u += (uint64_t)gridDim.x * kCellWarps * unit)
        accumulate_unit<BPL, SHARED, PAIR>(P, (uint32_t)u, min(unit, m - (uint32_t)u), blockIdx.y, gridDim.y, S, tab, beam);
}

using CellsFn = void (*)(const CellPing, const uint32_t*, uint32_t);
template <bool PAIR>
CellsFn cells_fn_of(int bpl, bool shared_out)
{
    if(shared_out) return bpl == 4 ? k_cells<4, true, PAIR> : k_cells<2, true, PAIR>;
    return bpl == 4 ? k_cells<4, false, PAIR> : k_cells<2, false, PAIR>;
}
CellsFn cells_fn(int bpl, bool shared_out, bool pairs)
{
    return pairs ? cells_fn_of<true>(bpl, shared_out) : cells_fn_of<false>(bpl, shared_out);
}

// Zeroes what a ping's passes add into: the bin totals, the range-bin bitmap,
// the cell rows and the ping (8-byte stores: the ping's alignment).
__global__ void k_cells_clear(uint32_t* __restrict__ totals, uint32_t n_totals, uint32_t* __restrict__ bits,
                              uint32_t n_bits, float4* __restrict__ cells, uint64_t n_cells, float2* __restrict__ out,
                              uint64_t n_out)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for(uint64_t i = i0; i < n_totals; i += stride) totals[i] = 0u;
    for(uint64_t i = i0; i < n_bits; i += stride) bits[i] = 0u;
    for(uint64_t i = i0; i < n_cells; i += stride) cells[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for(uint64_t i = i0; i < n_out; i += stride) out[i] = make_float2(0.f, 0.f);
}

__global__ void __launch_bounds__(32 * kFilterWarps)
k_cells_filter(const CellPing P, const uint32_t* __restrict__ nonempty, int ov)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_on[kFilterTile];
    if(threadIdx.x < kFilterTile) {
        const int r = blockIdx.y * kFilterTile + threadIdx.x;
        s_on[threadIdx.x] = r < (int)P.nR && row_on(nonempty, (int)P.nR, ov, r) ? 1 : 0;
    }
    filter_tile(P, blockIdx.x, blockIdx.y, reinterpret_cast<float4*>(s_raw), s_on);   // synchronises before it reads s_on
}

// Row pairs into the ping: row r takes T of storage row r + 1 and M of storage
// row r.
__global__ void __launch_bounds__(256)
k_pairs_join(const CellPing P, const uint32_t* __restrict__ nonempty, int ov)
{
    const int r = blockIdx.y, col = blockIdx.x * blockDim.x + threadIdx.x;
    if(col >= (int)P.pitch) return;
    const int b = P.col_bearing[col];
    if(b < 0) return;
    const float4 t = P.cells[(size_t)(r + 1) * P.pitch + col], m = P.cells[(size_t)r * P.pitch + col];
    P.out[(size_t)r * P.nB + b] = row_on(nonempty, (int)P.nR, ov, r) ? make_float2(t.x + m.z, t.y + m.w) : make_float2(0.f, 0.f);
}

template <typename T>
void drop(T*& p)
{
    if(p) cudaFree(p);
    p = nullptr;
}

template <typename T>
bool put(T*& dst, const std::vector<T>& src)
{
    if(cudaMalloc(&dst, src.size() * sizeof(T)) != cudaSuccess ||
       cudaMemcpy(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

} // namespace

void free_cells(Context& c)
{
    drop(c.d_cells); drop(c.d_cell_taps); drop(c.d_row_dev); drop(c.d_nonempty);
    drop(c.d_pos_theta); drop(c.d_pos_col); drop(c.d_col_bearing);
    c.cells_on = false;
    c.sorted_cells_n = 0;
}

// Decides whether a configured 2D sensor takes the cell form and builds its
// tables. The rule (everything else keeps the per-row gathers):
//   * the pulse's taps are one output range apart: the best line through the
//     rows' float ranges has k * spacing = 1 up to what the knot band covers,
//     and every row lies within the band of it (the band costs one product
//     per row and pair, so it is kept under a hundredth of a cell);
//   * every row's PSF support lies inside its reference window, so the window
//     only decides whether the row is on;
//   or (row pairs) no travel reaches more than two rows;
//   * the cell rows and the beam table fit.
// Returns whether the form is on; a failed allocation leaves it off.
bool configure_cells(Context& c, double beam_support)
{
    free_cells(c);
    const int nR = (int)c.nR, nB = (int)c.nB, H = (int)c.H, W = (int)c.W;
    if(c.dims != 2 || nR < 2 || H < 1) return false;
    const double k = (double)c.red.range_axis.k_hi + (double)c.red.range_axis.k_lo, center = 0.5 * H - 0.5;
    // Least-squares line through the rows' float ranges.
    std::vector<double> R(nR);
    double sr = 0.0, sx = 0.0;
    for(int r = 0; r < nR; r++) {
        R[r] = host_linspace_at(c.rmin, c.rmax, c.nR, (uint32_t)r);
        sr += R[r];
        sx += ((double)r - 0.5 * (nR - 1)) * R[r];
    }
    const double spacing = sx / ((double)nR * ((double)nR * nR - 1.0) / 12.0);
    const double R0 = sr / nR - 0.5 * (nR - 1) * spacing;
    if(!(spacing > 0.0) || !std::isfinite(spacing)) return false;
    const double kappa = k * spacing;
    double worst = 0.0;
    std::vector<float> dev(nR);
    for(int r = 0; r < nR; r++) {
        const double e = k * (R0 + r * spacing - R[r]);
        dev[r] = (float)e;
        worst = std::max(worst, std::fabs(e));
    }
    const double ext = (double)H / k;
    CellParams& cp = c.cell.cp;
    const double kc = 1.0 / spacing;
    cp.k_hi = (float)kc;
    cp.k_lo = (float)(kc - (double)cp.k_hi);
    double b;                                // cell coordinate y = travel / spacing + b
    // Row pairs: no travel within `half` of three rows (a hair of the spacing
    // covers the float cell index and the rows' deviations). Storage row
    // floor(y) + 2 = first row reached + 1.
    const double half = 0.5 * ext * (1.0 + 1.0 / H) + 1e-4 * spacing + worst / k + 1e-6 * std::fabs(R[nR - 1]);
    c.cell_pairs = half < spacing;
    if(c.cell_pairs) {
        b = -(half + R0) / spacing;
        cp.b_row = (float)(std::floor(b) + 2.0);
        cp.knot = 0.0f;
        cp.cells = nR + 1;
    }
    else {
        // What moves a row's knots against the grid: its own deviation, the tap
        // spacing's over half the pulse, and the rounding of travel - range.
        const double knot = 1.01 * (worst + std::fabs(kappa - 1.0) * (0.5 * H + 1.0)) + 2e-6 + 1.5e-7 * H;
        if(!(knot <= kMaxKnot)) return false;
        // Rows' supports inside their windows.
        for(int r = 0; r < nR; r++) {
            const double reach = 0.5 * ext * (1.0 + 1.0 / H) * (1.0 + 1e-4);
            const double slack = 1e-6 * (std::fabs(R[r]) + reach) + 1e-30;
            const int lo = (int)host_range_key_clamped(c.key, (float)(R[r] - reach - slack));
            const int hi = (int)host_range_key_clamped(c.key, (float)(R[r] + reach + slack));
            if(lo < std::max(0ll, (long long)r - c.overlap) || hi > std::min((long long)nR - 1, (long long)r + c.overlap)) return false;
        }
        b = center - kc * R0;                // storage row = cell + 1
        cp.b_row = (float)(std::floor(b) + 1.0);
        cp.knot = (float)knot;
        cp.cells = nR + H;
    }
    cp.b_frac = (float)(b - std::floor(b));
    cp.taps = H;
    c.cell.key = c.key;
    c.cell.overlap = c.overlap;
    if(std::fabs(b) + cp.cells > (double)(1 << 21)) return false;
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
    const double lo = (double)*mm.first - beam_support, hi = (double)*mm.second + beam_support;
    std::vector<double> theta_sorted(nB);
    for(int i = 0; i < nB; i++) theta_sorted[i] = c.bearings[sorted_b[i]];
    const int max_windows = std::max(1, (int)std::min(4096.0, (hi - lo) / (0.5 * beam_support)));
    std::vector<int2> span_of;              // [first, end) sorted bearings of each window
    int bpl = 0;
    for(int cand = 2; cand <= 4 && !bpl; cand += 2)
        for(int w = std::max(1, nB / (32 * cand)); w <= max_windows && !bpl; w++) {
            const double step = (hi - lo) / w, slack = 1e-5 * (hi - lo) + beam_support;   // 1e-5: the float window index
            bool fits = true;
            span_of.clear();
            for(int q = 0; q < w && fits; q++) {
                const auto f = std::lower_bound(theta_sorted.begin(), theta_sorted.end(), lo + q * step - slack);
                const auto e = std::upper_bound(f, theta_sorted.end(), lo + (q + 1) * step + slack);
                span_of.push_back(make_int2((int)(f - theta_sorted.begin()), (int)(e - theta_sorted.begin())));
                fits = e - f <= 32 * cand;
            }
            if(fits) bpl = cand;
        }
    const bool shared_out = bpl == 0;
    if(shared_out) bpl = nB > 64 ? 4 : 2;
    const int len = 32 * bpl;
    // Order of the bearings in a window. For one sample the table entries of
    // two bearings differ by their distance in taps, whatever the sample;
    // lanes whose distances differ modulo the 16 eight-byte banks of shared
    // memory never conflict. Bearings sorted by that remainder and dealt to
    // the groups of 16 lanes in turn are about one bank apart: 3.1 to 3.5
    // wavefronts per lookup instead of 3.8 to 4.8 in the bearings' own order
    // (counted for the tables of the imaging sensors).
    const double kb = (double)c.red.beam_axis.k_hi;
    auto deal = [&](std::vector<int> order, std::vector<int>& pos, size_t at) {
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
    c.cell.windows = (int)(pos.size() / len);
    // Sort order: window x cell block, with as many bins as the pipelined
    // scatter takes at one reservation batch per thread.
    BinParams& bin = c.cell_bin;
    bin = c.bin;
    bin.cell = cp;
    bin.nBB = shared_out ? 1u : (uint32_t)span_of.size();
    bin.bb_scale = (float)(bin.nBB / (hi - lo));
    bin.bb_offset = (float)(-lo * (bin.nBB / (hi - lo)));
    for(bin.cell_shift = 0;; bin.cell_shift++) {
        bin.cell_blocks = (uint32_t)((cp.cells - 1) >> bin.cell_shift) + 1u;
        if(bin.nBB * bin.cell_blocks <= kCellBins || bin.cell_blocks == 1u) break;
    }
    bin.nBins = bin.nBB * bin.cell_blocks;
    c.cell.win_scale = bin.bb_scale;
    c.cell.win_offset = bin.bb_offset;
    // Columns: the lanes' order for shared-out windows (whole rows of 512
    // bytes per reduction), the bearings' own order for overlapping ones.
    const uint32_t pitch = shared_out ? (uint32_t)pos.size() : (uint32_t)((nB + 31) / 32 * 32);
    c.cell.pitch = pitch;
    std::vector<int> col(pos.size()), col_bearing(pitch, -1);
    std::vector<float> theta(pos.size(), c.bearings[sorted_b[nB - 1]]);
    for(size_t p = 0; p < pos.size(); p++) {
        col[p] = pos[p] < 0 ? -1 : shared_out ? (int)p : pos[p];
        if(pos[p] < 0) continue;
        theta[p] = c.bearings[pos[p]];
        col_bearing[col[p]] = pos[p];
    }
    const size_t cell_bytes = (size_t)cp.cells * pitch * sizeof(float4);
    if(cell_bytes > kMaxCellBytes || cells_smem(W, c.cell_pairs) > 200 * 1024 ||
       (!c.cell_pairs && filter_smem(H) > 200 * 1024)) return false;
    std::vector<float4> taps((size_t)cell_tap_entries(H), make_float4(0.f, 0.f, 0.f, 0.f));
    for(int i = -1; i < H; i++) {
        double p[2], d[2];
        for(int q = 0; q < 2; q++) {
            const double lo = i >= 0 ? c.pulse[2 * (size_t)i + q] : 0.0, hi = i + 1 < H ? c.pulse[2 * ((size_t)i + 1) + q] : 0.0;
            p[q] = lo + (hi - lo) * (kappa - 1.0) * ((double)i - center);
            d[q] = (hi - lo) * kappa;
        }
        taps[i + 1] = make_float4((float)p[0], (float)p[1], (float)d[0], (float)d[1]);
    }
    bool ok = put(c.d_cell_taps, taps) && put(c.d_row_dev, dev) && put(c.d_nonempty, std::vector<uint32_t>((nR + 31) / 32, 0u)) &&
              put(c.d_pos_theta, theta) && put(c.d_pos_col, col) && put(c.d_col_bearing, col_bearing);
    if(ok && cudaMalloc(&c.d_cells, cell_bytes) != cudaSuccess) { cudaGetLastError(); ok = false; }
    if(ok) ok = raise_smem_limit((const void*)cells_fn(bpl, shared_out, c.cell_pairs), cells_smem(W, c.cell_pairs)) == cudaSuccess &&
                (c.cell_pairs ||
                 raise_smem_limit((const void*)k_cells_filter, filter_smem(H)) == cudaSuccess);
    if(!ok) { free_cells(c); return false; }
    CellPing& P = c.cell;
    P.cells = c.d_cells;
    P.row_dev = c.d_row_dev; P.taps = c.d_cell_taps;
    P.pos_theta = c.d_pos_theta; P.pos_col = c.d_pos_col; P.col_bearing = c.d_col_bearing;
    P.range_axis = c.red.range_axis; P.beam_axis = c.red.beam_axis;
    P.nR = c.nR; P.nB = c.nB;
    c.cells_on = true;
    return true;
}

rtacx_status run_cells(Context& c, const void* samples, uint64_t n, float2* out, cudaStream_t stream)
{
    CellPing P = c.cell;
    P.sorted = c.d_sorted;
    P.out = out;
    BinParams bin = c.cell_bin;
    bin.vec4 = c.bin.vec4;
    const uint32_t totals = bin.nBins + (bin.nBins + kScanBlock - 1) / kScanBlock;
    const uint64_t cells = (uint64_t)P.cp.cells * P.pitch, cells_out = c.cell_pairs && n ? 0 : (uint64_t)c.nR * c.nB;   // (the pairs' join writes every cell)
    c.mark(1, false, stream);
    k_cells_clear<<<(uint32_t)std::min<uint64_t>((cells + 255) / 256, (uint64_t)c.sm_count * 8), 256, 0, stream>>>(
        c.d_totals, totals, c.d_nonempty, (c.nR + 31) / 32, c.d_cells, cells, out, cells_out);
    cudaError_t e = cudaGetLastError();
    c.mark(1, true, stream);
    c.sorted_cells_n = 0;
    if(e == cudaSuccess && n) {
        const rtacx_status st = run_sort(c, bin, c.cell_sort, samples, n, c.d_nonempty, stream);
        if(st != RTACX_OK) return st;
        c.sorted_cells_n = n;
        c.mark(5, false, stream);
        // Units of fewer samples while that leaves the SMs' warps without one;
        // wide beams' windows are then also shared out over blockIdx.y.
        const uint32_t warps = (uint32_t)c.sm_count * 3u * kCellWarps;
        uint32_t unit = kUnit;
        while(unit > 32 && n < (uint64_t)warps * unit * 2) unit /= 2;
        const uint64_t ctas = (n + (uint64_t)unit * kCellWarps - 1) / ((uint64_t)unit * kCellWarps);
        const uint32_t gx = (uint32_t)std::min<uint64_t>(ctas, (uint64_t)c.sm_count * 12u);
        const uint32_t gy = c.cell_shared ? (uint32_t)std::min<uint64_t>((uint64_t)P.windows,
                                                std::max<uint64_t>(1, (uint64_t)c.sm_count * 3u / gx)) : 1u;
        cells_fn(c.cell_bpl, c.cell_shared, c.cell_pairs)<<<dim3(gx, gy), kCellThreads,
                                                            cells_smem(P.beam_axis.n, c.cell_pairs), stream>>>(
            P, c.d_offsets + bin.nBins, unit);
        const dim3 fgrid(P.pitch / 32, (c.nR + kFilterTile - 1) / kFilterTile);
        if(c.cell_pairs) k_pairs_join<<<dim3((P.pitch + 255) / 256, c.nR), 256, 0, stream>>>(P, c.d_nonempty, c.overlap);
        else k_cells_filter<<<fgrid, 32 * kFilterWarps, filter_smem(P.cp.taps), stream>>>(P, c.d_nonempty, c.overlap);
        e = cudaGetLastError();
        c.mark(5, true, stream);
    }
    if(e != cudaSuccess) { c.error = std::string("cell form: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    return RTACX_OK;
}

} // namespace rtacx
