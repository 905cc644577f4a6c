// Plain 2D reduction over range cells (see rtacx_cells.cuh): configuration
// and the single-ping kernels.
//
//   k_cells         the sorted samples of one ping into the cell rows;
//   k_cells_filter  the pulse's taps over the cell rows, rows without a
//                   reference window zeroed.
// Measured against the tensor-core gather on the same pings (whole
// rtacx_reduce, us): 2^20 samples, 512 x 1024, 33 taps, narrow beams: 1384 ->
// 170; 2^22 samples, 512 x 4096, wide beams: 14433 -> 1278; 150003 samples,
// 387 x 777, 24 taps: 246 -> 90. k_cells is bound by the beam lookups' shared
// memory and issue slots, at one lookup per (sample, bearing).
#include "rtacx_bin_device.cuh"
#include "rtacx_cells.cuh"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace rtacx {

namespace {

constexpr int kCellThreads = 256, kCellWarps = kCellThreads / 32;
constexpr int kFilterWarps = 4;
constexpr size_t kMaxCellBytes = (size_t)1 << 30;      // cell rows of one context
constexpr double kMaxKnot = 0.01;

size_t cells_smem(int W) { return kCellWarps * sizeof(CellWarpSmem) + (size_t)(W + 2) * sizeof(float2); }

// Entries of the tap table: H + 1 taps, kFilterRows - 1 steps of the sliding
// window beyond them, rounded up to whole blocks of kFilterRows.
__host__ __device__ __forceinline__ int cell_tap_entries(int H) { return (H + kFilterRows + kFilterRows - 1) / kFilterRows * kFilterRows; }

template <int BPL>
__global__ void __launch_bounds__(kCellThreads, 2)
k_cells(const CellPing P, const uint32_t* __restrict__ total)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    CellWarpSmem& S = reinterpret_cast<CellWarpSmem*>(s_raw)[threadIdx.x >> 5];
    float2* tab = reinterpret_cast<float2*>(s_raw + kCellWarps * sizeof(CellWarpSmem));
    load_beam_table(tab, P.beam, P.beam_axis.n, threadIdx.x, kCellThreads);
    __syncthreads();
    BeamLookup beam;
    beam.init(P.beam_axis);
    const uint32_t m = *total, units = (m + kUnit - 1) / kUnit;
    for(uint32_t u = blockIdx.x * kCellWarps + (threadIdx.x >> 5); u < units; u += gridDim.x * kCellWarps)
        accumulate_unit<BPL>(P, u * kUnit, min((uint32_t)kUnit, m - u * kUnit), blockIdx.y, gridDim.y, S, tab, beam);
}

// One CTA: 32 positions x kFilterWarps * kFilterRows rows, the warps below
// each other so that they share the cell rows through L1.
__global__ void __launch_bounds__(32 * kFilterWarps)
k_cells_filter(const CellPing P, const uint32_t* __restrict__ off, uint32_t nBB, int ov)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    float4* s_taps = reinterpret_cast<float4*>(s_raw);
    __shared__ int s_on[kFilterWarps * kFilterRows];
    const int rows0 = blockIdx.y * (kFilterWarps * kFilterRows), warp = threadIdx.x >> 5;
    for(int i = threadIdx.x; i < cell_tap_entries(P.cp.taps); i += 32 * kFilterWarps) s_taps[i] = P.taps[i];
    if(threadIdx.x < kFilterWarps * kFilterRows) {
        const int r = rows0 + threadIdx.x;
        int f, l;
        s_on[threadIdx.x] = r < (int)P.nR && ref_window(off, nBB, P.nR, ov, r, f, l) ? 1 : 0;
    }
    __syncthreads();
    const int r0 = rows0 + warp * kFilterRows;
    if(r0 < (int)P.nR) filter_rows(P, blockIdx.x * 32 + (threadIdx.x & 31), r0, s_taps, s_on + warp * kFilterRows);
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
    drop(c.d_cells); drop(c.d_cell_taps); drop(c.d_row_dev); drop(c.d_seg_reach);
    drop(c.d_pos_theta); drop(c.d_pos_bearing);
    c.cells_on = false;
}

// Decides whether a configured 2D sensor takes the cell form and builds its
// tables. The rule (everything else keeps the per-row gathers):
//   * the pulse's taps are one output range apart: the best line through the
//     rows' float ranges has k * spacing = 1 up to what the knot band covers,
//     and every row lies within the band of it (the band costs one product
//     per row and pair, so it is kept under a hundredth of a cell);
//   * every row's PSF support lies inside its reference window, so the window
//     only decides whether the row is on;
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
    // What moves a row's knots against the grid: its own deviation, the tap
    // spacing's over half the pulse, and the rounding of travel - range.
    const double knot = 1.01 * (worst + std::fabs(kappa - 1.0) * (0.5 * H + 1.0)) + 2e-6 + 1.5e-7 * H;
    if(!(knot <= kMaxKnot)) return false;
    // Rows' supports inside their windows.
    for(int r = 0; r < nR; r++) {
        const double ext = 1.0 / (k / H), half = 0.5 * ext * (1.0 + 1.0 / H) * (1.0 + 1e-4);
        const double slack = 1e-6 * (std::fabs(R[r]) + half) + 1e-30;
        const int lo = (int)host_range_key_clamped(c.key, (float)(R[r] - half - slack));
        const int hi = (int)host_range_key_clamped(c.key, (float)(R[r] + half + slack));
        if(lo < std::max(0ll, (long long)r - c.overlap) || hi > std::min((long long)nR - 1, (long long)r + c.overlap)) return false;
    }
    // Cell coordinate y = travel / spacing + b; storage row = cell + 1.
    CellParams& cp = c.cell.cp;
    const double kc = 1.0 / spacing, b = center - kc * R0;
    cp.k_hi = (float)kc;
    cp.k_lo = (float)(kc - (double)cp.k_hi);
    cp.b_row = (float)(std::floor(b) + 1.0);
    cp.b_frac = (float)(b - std::floor(b));
    cp.knot = (float)knot;
    cp.cells = nR + H;
    cp.taps = H;
    if(std::fabs(b) + cp.cells > (double)(1 << 21)) return false;
    // Beam coordinates far below the rounding trick's 2^22.
    const auto mm = std::minmax_element(c.bearings.begin(), c.bearings.end());
    const double fan = (double)*mm.second - (double)*mm.first, span = c.span;
    if((fan + 4.0 * span) / span * W + W > (double)(1 << 20)) return false;
    c.cell.theta_lo = (float)(*mm.first - 2.0 * span);
    c.cell.theta_hi = (float)(*mm.second + 2.0 * span);

    // Bearings per lane: four where a sample reaches most of the fan (fewer
    // list reads per pair), two where beams are narrow (shorter segments).
    const bool wide = 4.0 * beam_support >= fan;
    c.cell_bpl = wide && nB > 64 ? 4 : 2;
    const int seg_len = 32 * c.cell_bpl, segs = (nB + seg_len - 1) / seg_len;
    c.cell.segs = segs;
    c.cell.pitch = (uint32_t)(segs * seg_len);
    const size_t cell_bytes = (size_t)cp.cells * c.cell.pitch * sizeof(float4);
    if(cell_bytes > kMaxCellBytes || cells_smem(W) > 200 * 1024) return false;

    // Order of the bearings. For one sample the table entries of two bearings
    // differ by their distance in taps, whatever the sample; lanes whose
    // distances differ modulo the 16 eight-byte banks of shared memory never
    // conflict. Bearings sorted by that remainder and dealt to the groups of
    // 16 lanes in turn are about one bank apart. Dealt over the whole fan for
    // wide beams, inside each segment for narrow ones.
    const double kb = (double)c.red.beam_axis.k_hi;
    std::vector<int> pos(c.cell.pitch, -1);
    const int scope = wide ? (int)c.cell.pitch : seg_len;
    for(int s0 = 0; s0 < (int)c.cell.pitch; s0 += scope) {
        std::vector<int> order;
        for(int i = s0; i < std::min(nB, s0 + scope); i++) order.push_back(i);
        auto bank = [&](int i) { const double x = (double)c.bearings[i] * kb; return x - 16.0 * std::floor(x / 16.0); };
        std::stable_sort(order.begin(), order.end(), [&](int a, int d) { return bank(a) < bank(d); });
        // Deal the bearings to as many whole groups as they fill.
        const int groups = std::max(1, ((int)order.size() + 15) / 16);
        for(size_t q = 0; q < order.size(); q++) pos[s0 + (int)(q % groups) * 16 + (int)(q / groups)] = order[q];
    }
    std::vector<float> theta(c.cell.pitch, c.bearings[nB - 1]);
    std::vector<float2> reach(segs, make_float2(INFINITY, -INFINITY));
    for(int p = 0; p < (int)c.cell.pitch; p++) {
        if(pos[p] < 0) continue;
        const float t = c.bearings[pos[p]];
        theta[p] = t;
        float2& s = reach[p / seg_len];
        s.x = std::min(s.x, (float)(t - beam_support));
        s.y = std::max(s.y, (float)(t + beam_support));
    }
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
    bool ok = put(c.d_cell_taps, taps) && put(c.d_row_dev, dev) && put(c.d_seg_reach, reach) &&
              put(c.d_pos_theta, theta) && put(c.d_pos_bearing, pos);
    if(ok && cudaMalloc(&c.d_cells, cell_bytes) != cudaSuccess) { cudaGetLastError(); ok = false; }
    const void* fn = c.cell_bpl == 4 ? (const void*)k_cells<4> : (const void*)k_cells<2>;
    if(ok) ok = raise_smem_limit(fn, cells_smem(W)) == cudaSuccess &&
                raise_smem_limit((const void*)k_cells_filter, cell_tap_entries(H) * sizeof(float4)) == cudaSuccess;
    if(!ok) { free_cells(c); return false; }
    CellPing& P = c.cell;
    P.cells = c.d_cells;
    P.pulse = c.d_pulse; P.beam = c.d_beam; P.ranges = c.d_ranges;
    P.row_dev = c.d_row_dev; P.taps = c.d_cell_taps; P.seg_reach = c.d_seg_reach;
    P.pos_theta = c.d_pos_theta; P.pos_bearing = c.d_pos_bearing;
    P.range_axis = c.red.range_axis; P.beam_axis = c.red.beam_axis;
    P.nR = c.nR; P.nB = c.nB;
    c.cells_on = true;
    return true;
}

rtacx_status run_cells(Context& c, uint64_t n, float2* out, cudaStream_t stream)
{
    CellPing P = c.cell;
    P.sorted = c.d_sorted;
    P.out = out;
    cudaError_t e = cudaMemsetAsync(c.d_cells, 0, (size_t)P.cp.cells * P.pitch * sizeof(float4), stream);
    if(e == cudaSuccess) e = cudaMemsetAsync(out, 0, (size_t)c.nR * c.nB * sizeof(float2), stream);
    if(e != cudaSuccess) { c.error = std::string("clearing the cell rows: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    // As many units as there are; the segments of a unit are shared out over
    // blockIdx.y when there are too few units to fill the SMs.
    const uint64_t ctas = std::max<uint64_t>(1, (n + (uint64_t)kUnit * kCellWarps - 1) / ((uint64_t)kUnit * kCellWarps));
    const uint32_t full = (uint32_t)c.sm_count * 3u;
    const uint32_t gx = (uint32_t)std::min<uint64_t>(ctas, (uint64_t)full * 4u);
    const uint32_t gy = (uint32_t)std::min<uint64_t>((uint64_t)P.segs, std::max<uint64_t>(1, full / gx));
    const dim3 grid(gx, gy);
    const size_t smem = cells_smem(P.beam_axis.n);
    if(c.cell_bpl == 4) k_cells<4><<<grid, kCellThreads, smem, stream>>>(P, c.d_offsets + c.bin.nBins);
    else k_cells<2><<<grid, kCellThreads, smem, stream>>>(P, c.d_offsets + c.bin.nBins);
    const dim3 fgrid(P.pitch / 32, (c.nR + kFilterWarps * kFilterRows - 1) / (kFilterWarps * kFilterRows));
    k_cells_filter<<<fgrid, 32 * kFilterWarps, cell_tap_entries(P.cp.taps) * sizeof(float4), stream>>>(
        P, c.d_offsets, c.bin.nBB, c.overlap);
    e = cudaGetLastError();
    if(e != cudaSuccess) { c.error = std::string("cell form: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    return RTACX_OK;
}

} // namespace rtacx
