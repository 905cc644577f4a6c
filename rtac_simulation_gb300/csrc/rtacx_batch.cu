// Batched plain form: many pings from heterogeneous sensors in one CUDA graph.
//
// A batch holds up to thousands of pings, each bound to its own configured
// context (1D or 2D). rtacx_batch_plan builds, once:
//   * a device descriptor per ping (PingDev: its samples, scratch, tables);
//   * (ping, index) maps of the binning work of every ping (totals to zero,
//     count / scatter chunks, bin-scan blocks, window row groups);
//   * the gather work list: 2D output tiles and 1D row groups of every ping,
//     heaviest first;
// then captures the batch into a CUDA graph. By default the graph holds one
// kernel: k_batch_fused, a cooperative persistent launch (one or two CTAs per
// SM, all resident) that runs every phase of every ping, taking work from
// atomic queues and separating the phases with bounded grid barriers (and a
// memset node that resets the barrier and the queues). Pings that rtacx_reduce
// takes through the cell form go through it here too (choose_form): 16 mixed
// pings of 2^13 to 2^20 samples 10.0 -> 0.63 ms. With
// RTACX_BATCH_STAGED the graph holds one launch per binning stage and a
// persistent gather kernel instead. rtacx_batch_run replays the graph with one
// cudaGraphLaunch. With RTACX_BATCH_AUTOTUNE the plan times every candidate
// (gather tile shape x samples per binning chunk) on the real batch and keeps
// the fastest.
#include "rtacx_internal.cuh"

#include <algorithm>
#include <cmath>
#include <set>
#include <vector>

namespace rtacx {

namespace {

struct Candidate {
    int shape;
    uint32_t per_cta;
};

uint64_t ceil_div(uint64_t a, uint64_t b) { return (a + b - 1) / b; }

} // namespace

struct Batch {
    int device = 0;
    int sm_count = 0;
    std::string error;
    cudaStream_t stream = nullptr;
    std::vector<rtacx_ping_desc> pings;
    // Device arrays of the current plan.
    PingDev* d_pings = nullptr;
    uint2* d_chunk_map = nullptr;
    uint2* d_col_map = nullptr;
    uint2* d_win_map = nullptr;
    uint2* d_scan_map = nullptr;
    uint4* d_items = nullptr;
    uint4* d_filters = nullptr;
    ZeroItem* d_zero16 = nullptr;
    ZeroItem* d_zero8 = nullptr;
    uint32_t* d_counter = nullptr;
    BatchSync* d_sync = nullptr;
    uint32_t* d_status = nullptr;
    uint32_t n_chunks_all = 0, n_filters = 0, n_zero16 = 0, n_zero8 = 0;
    bool cells = false;             // the fused kernel with the cell form
    bool per_row_2d = false;        // some 2D ping takes the per-row gather
    uint32_t n_chunks = 0, n_col = 0, n_win = 0, n_scan = 0, n_items = 0, max_bins = 0;
    size_t gather_smem = 0;
    uint32_t gather_grid = 0;
    bool staged = false;            // RTACX_BATCH_STAGED
    FusedBatch fb{};
    size_t fused_smem = 0;
    uint32_t fused_grid = 0;
    uint32_t graph_kernels = 0;     // kernel nodes of the captured graph
    uint32_t diag_extra = 0;        // extra barrier arrivals (diagnostic)
    uint32_t wait_ms = 1000;        // bound of one grid-barrier wait
    Candidate chosen{2, 4096};
    float tuned_ms = 0.0f;
    cudaGraphExec_t exec = nullptr;

    template <typename T>
    void drop(T*& p) { if(p) cudaFree(p); p = nullptr; }

    void free_plan()
    {
        if(exec) cudaGraphExecDestroy(exec);
        exec = nullptr;
        drop(d_pings); drop(d_chunk_map); drop(d_col_map); drop(d_win_map); drop(d_scan_map); drop(d_items);
        drop(d_filters); drop(d_zero16); drop(d_zero8);
        graph_kernels = 0;
    }

    template <typename T>
    bool put(T*& dst, const std::vector<T>& src)
    {
        drop(dst);
        const size_t bytes = std::max<size_t>(1, src.size()) * sizeof(T);
        if(cudaMalloc(&dst, bytes) != cudaSuccess) { cudaGetLastError(); error = "cudaMalloc failed"; return false; }
        if(!src.empty() && cudaMemcpy(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
            cudaGetLastError();
            error = "cudaMemcpy failed";
            return false;
        }
        return true;
    }

    // Samples of a ping's cell form that one work item takes: about kItemSamples
    // of a 64-bearing window's work, in whole rounds of the CTA's warps (16
    // pings, 2.5e6 2D samples, us for the phase: 2048 243, its last items
    // leaving SMs idle; 1024 226; 512 247, units of 64 samples).
    static constexpr uint64_t kItemSamples = 1024;
    static uint32_t cells_per_item(const Context& c)
    {
        const uint64_t pairs = c.cell_shared ? c.cell.pitch : 32u * (uint32_t)c.cell_bpl;
        uint64_t want = kItemSamples;
        while(want > 256 && want * pairs > kItemSamples * 64) want /= 2;
        return (uint32_t)want;
    }

    // Estimates of a ping in the fused kernel (us): of the per-row gathers,
    // with the default tiles and `alone` the time of its tiles one behind the
    // other on one CTA each, and of the cell form.
    static double rows_us(const Context& c, uint64_t n, double& alone)
    {
        const double samples = (double)n, TR = gather_shape_rows(2), TB = gather_shape_bearings(2);
        if(c.dims == 1) { alone = 0.0; return 0.09e-3 * samples; }
        const double tr = std::ceil(c.nR / TR), tb = std::ceil(c.nB / TB);
        const double pulse_rows = (double)c.duration * c.c * (c.nR - 1.0) / std::max(1e-30, (double)c.rmax - c.rmin);
        double entered = std::min(tr, 1.0 + pulse_rows / TR), across = tb;      // tiles that a sample enters
        if(c.bin.nBB > 1) {
            const double fan = c.bin.nBB / (double)c.bin.bb_scale;
            across = std::min(tb, tb / fan * ((fan - c.span) * TB / c.nB + c.span + fan / c.bin.nBB));
        }
        entered *= across;
        alone = 0.35 * samples * entered / (tr * tb);
        return 5e-6 * c.nR * c.nB + samples * entered * TR * TB / 4e6;
    }
    static double cells_us(const Context& c, uint64_t n)
    {
        if(c.dims == 1) return 0.015e-3 * n;
        const double entries = 1e-6 * (double)c.cell.cp.cells * c.cell.pitch;
        return entries * (c.cell_pairs ? 13.0 : 18.0 + 0.4 * c.H) +
               0.8e-6 * n * (c.cell_shared ? c.cell.pitch : 32.0 * c.cell_bpl);
    }

    // Whether the batch runs on the fused kernel with the cell form: where that
    // is estimated to be faster (it clears and filters every cell row, whatever
    // the samples), and when the per-row gathers' share of the work (samples x
    // bearings) is at most half, since that kernel keeps fewer of their CTAs
    // resident. us per batch, per-row / cell form, samples spread evenly (a
    // floor in view): one ping of 512 x 1024, 33 taps, 2^12 samples 57 / 118 (89
    // / 113), 2^14 78 / 116 (147 / 109), 2^16 159 / 113 (443 / 108); six of them
    // 2^12 98 / 210 (127 / 201), 2^14 198 / 202 (245 / 202); six of 512 x 4096
    // 2^14 251 / 500 (278 / 503), 2^16 647 / 558 (683 / 531); six of 1024 x 8192
    // 2^15 824 / 1632 (851 / 1636), 2^17 2572 / 1778 (2640 / 1731); six wide beams
    // of 512 x 1024 2^10 90 / 244 (119 / 248), 2^13 336 / 216 (457 / 228); six row
    // pairs of 1024 x 4096 2^13 346 / 565 (336 / 562), 2^15 726 / 582 (749 / 646);
    // six 1D pings 2^8 44 / 30, 2^17 113 / 45. The estimates are fitted to both
    // scenes, towards the cell form where they differ.
    void choose_form()
    {
        double per_row = 0.0, cell = 0.0, rows = 0.0, longest = 0.0, form = 28.0;
        bool any_2d = false;
        for(const rtacx_ping_desc& p : pings) {
            const Context& c = p.ctx->impl;
            const bool takes = takes_cells(c, p.n);
            (takes ? cell : per_row) += (double)p.n * c.nB;
            double alone;
            const double r = rows_us(c, p.n, alone);
            rows += r;
            longest = std::max(longest, alone);
            form += takes ? cells_us(c, p.n) : r;
            any_2d |= takes && c.dims == 2;
        }
        cells = !staged && cell > 0.0 && per_row <= cell && form + (any_2d ? 70.0 : 0.0) < 35.0 + std::max(rows, longest);
        per_row_2d = false;
        for(const rtacx_ping_desc& p : pings)
            if(p.ctx->impl.dims == 2 && !(cells && takes_cells(p.ctx->impl, p.n))) per_row_2d = true;
    }

    // Descriptors, maps and work items for one candidate; captures the graph.
    rtacx_status build(const Candidate& cand)
    {
        free_plan();
        const int TR = gather_shape_rows(cand.shape), TB = gather_shape_bearings(cand.shape);
        std::vector<PingDev> descs;
        std::vector<uint2> chunk_map, chunk_map_1d, col_map, win_map, scan_map;
        std::vector<uint4> filters;
        std::vector<ZeroItem> zero16, zero8;
        auto zero = [](std::vector<ZeroItem>& list, void* p, uint64_t n, size_t elem) {
            for(uint64_t i = 0; i < n; i += 4096)
                list.push_back(ZeroItem{static_cast<unsigned char*>(p) + i * elem, std::min<uint64_t>(4096, n - i)});
        };
        struct Item { uint4 v; double cost; };
        std::vector<Item> items;
        max_bins = 1;
        gather_smem = 0;
        for(uint32_t i = 0; i < pings.size(); i++) {
            Context& c = pings[i].ctx->impl;
            const uint64_t n = pings[i].n;
            PingDev d{};
            const bool cell_form = cells && takes_cells(c, n);
            d.form = !cell_form ? kPerRow
                   : c.dims == 1 ? (c.cell_rows ? kRows1D : kCells1D) : (c.cell_pairs ? kPairs2D : kCells2D);
            d.samples = static_cast<const float*>(pings[i].samples);
            d.n = n;
            d.bin = cell_form && c.dims == 2 ? c.cell_bin : c.bin;
            d.bin.vec4 = (c.dims == 2 && reinterpret_cast<uintptr_t>(pings[i].samples) % 16 == 0) ? 1 : 0;
            d.chunks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(c.sort.hist_ctas, ceil_div(n, cand.per_cta)));
            d.hist = c.d_hist; d.totals = c.d_totals; d.offsets = c.d_offsets; d.oor = c.d_oor; d.err = c.d_err;
            d.sorted = c.d_sorted;
            d.nR = c.nR; d.overlap = c.overlap; d.support = c.d_support; d.win = c.d_win;
            d.red = c.red; d.bb_tiles = c.d_bb_tiles; d.ranges = c.d_ranges; d.bearings = c.d_bearings;
            d.pulse = c.d_pulse; d.beam = c.d_beam; d.out = reinterpret_cast<float2*>(pings[i].out);
            if(c.dims == 2) d.bb_tiles = (TB == 64) ? c.d_bb_tiles64 : c.d_bb_tiles128;   // ranges for width TB
            if(cell_form) {
                d.order = c.dims == 1 ? kInputOrder | n : kBinsOrder | d.bin.nBins;
                d.cell = c.cell;
                d.cell.cells = c.d_cells;
                d.cell.sorted = c.d_sorted;
                d.cell.out = d.out;
                d.cell.replicas = c.dims == 1 ? cell_replicas(c, n) : 1;
                d.nonempty = c.d_nonempty;
                d.bpl = c.cell_bpl;
                d.shared = c.cell_shared ? 1 : 0;
                zero(zero16, c.d_nonempty, (c.nR + 127) / 128, 16);
                zero(zero16, c.d_cells, c.dims == 1 ? cell_words_1d(c, n) : (uint64_t)c.cell.cp.cells * c.cell.pitch, 16);
                if(d.form != kPairs2D && d.form != kRows1D) zero(zero8, d.out, (uint64_t)c.nR * c.nB, 8);
                uint32_t columns;
                const uint32_t rows = batch_filter_tiles(c, columns);
                for(uint32_t y = 0; y < rows; y++)
                    for(uint32_t x = 0; x < columns; x++) filters.push_back(make_uint4(i, x, y, 0));
                gather_smem = std::max(gather_smem, batch_cells_smem(c));
                if(c.dims == 2 && c.cell_sort.ranked && n <= std::min(c.n_ranks, kMaxRanked)) {
                    d.ranks = c.d_ranks;
                    d.chunks = (uint32_t)std::max<uint64_t>(1, ceil_div(n, kRankedChunk));
                    gather_smem = std::max(gather_smem, ranked_smem(d.bin.nBins, c.nR));
                }
            }
            if(cell_form && c.dims == 1) {
                d.chunks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)sm_count * 8, ceil_div(n, cand.per_cta)));
                for(uint32_t k = 0; k < d.chunks; k++) chunk_map_1d.push_back(make_uint2(i, k));
                descs.push_back(d);
                continue;
            }
            for(uint32_t k = 0; k < d.chunks; k++) chunk_map.push_back(make_uint2(i, k));
            for(uint32_t k = 0; k < ceil_div(d.bin.nBins, 256); k++) col_map.push_back(make_uint2(i, k));
            for(uint32_t k = 0; k < ceil_div(d.bin.nBins, kScanBlock); k++) scan_map.push_back(make_uint2(i, k));
            max_bins = std::max(max_bins, d.bin.nBins);
            const double density = (double)n / c.nR;     // samples per range bin
            if(cell_form) {
                d.per_item = cells_per_item(c);
                d.unit = std::min(128u, std::max(32u, d.per_item / 8));
                const double pairs = c.cell_shared ? c.cell.pitch : 32.0 * c.cell_bpl;
                for(uint64_t k = 0; k < ceil_div(n, d.per_item); k++)
                    items.push_back({make_uint4(i, (uint32_t)k, 0, 2), (double)std::min<uint64_t>(n, d.per_item) * pairs / 64.0});
                descs.push_back(d);
                continue;
            }
            descs.push_back(d);
            for(uint32_t k = 0; k < ceil_div(c.nR, 256); k++) win_map.push_back(make_uint2(i, k));
            if(c.dims == 2) {
                const uint32_t tb = (c.nB + TB - 1) / TB, tr = (c.nR + TR - 1) / TR;
                for(uint32_t y = 0; y < tr; y++)
                    for(uint32_t x = 0; x < tb; x++) items.push_back({make_uint4(i, x, y, 0), density * TR * TB});
                gather_smem = std::max(gather_smem, gather_batch_smem(cand.shape, c.H, c.W));
            }
            else {
                for(uint32_t g = 0; g < ceil_div(c.nR, 8); g++) items.push_back({make_uint4(i, g, 0, 1), density * 8.0});
                gather_smem = std::max(gather_smem, (size_t)(c.H + 2) * sizeof(float2));
            }
        }
        std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.cost > b.cost; });
        std::vector<uint4> iv(items.size());
        for(size_t k = 0; k < items.size(); k++) iv[k] = items[k].v;
        n_chunks = (uint32_t)chunk_map.size();
        chunk_map.insert(chunk_map.end(), chunk_map_1d.begin(), chunk_map_1d.end());
        n_chunks_all = (uint32_t)chunk_map.size();
        n_filters = (uint32_t)filters.size(); n_zero16 = (uint32_t)zero16.size(); n_zero8 = (uint32_t)zero8.size();
        n_col = (uint32_t)col_map.size();
        n_win = (uint32_t)win_map.size(); n_scan = (uint32_t)scan_map.size(); n_items = (uint32_t)iv.size();
        if(!put(d_pings, descs) || !put(d_chunk_map, chunk_map) || !put(d_col_map, col_map) ||
           !put(d_win_map, win_map) || !put(d_scan_map, scan_map) || !put(d_items, iv) || !put(d_filters, filters) ||
           !put(d_zero16, zero16) || !put(d_zero8, zero8))
            return RTACX_ERR_OUT_OF_MEMORY;
        if(gather_smem > 227 * 1024) { error = "PSF tables too large for the batched gather"; return RTACX_ERR_UNSUPPORTED; }
        if(staged && (size_t)max_bins * 4 > 227 * 1024) { error = "histograms too large for the batched binning"; return RTACX_ERR_UNSUPPORTED; }
        chosen = cand;
        return staged ? capture_staged(cand, (uint32_t)descs.size()) : capture_fused(cand);
    }

    // Graph of the fused form: reset of the barrier and queues, one
    // cooperative launch.
    rtacx_status capture_fused(const Candidate& cand)
    {
        fused_smem = gather_smem;
        rtacx_status prep = prepare_fused_batch(error, cand.shape, cells, fused_smem, sm_count, fused_grid);
        if(prep != RTACX_OK) return prep;
        fb = FusedBatch{};
        fb.pings = d_pings;
        fb.col_map = d_col_map; fb.n_col = n_col;
        fb.chunk_map = d_chunk_map; fb.n_chunks = n_chunks; fb.n_chunks_all = n_chunks_all;
        fb.zero16 = d_zero16; fb.n_zero16 = n_zero16;
        fb.zero8 = d_zero8; fb.n_zero8 = n_zero8;
        fb.filters = d_filters; fb.n_filters = n_filters;
        fb.scan_map = d_scan_map; fb.n_scan = n_scan;
        fb.win_map = d_win_map; fb.n_win = n_win;
        fb.items = d_items; fb.n_items = n_items;
        fb.sync = d_sync;
        fb.status = d_status;
        fb.arrivals = fused_grid + diag_extra;
        fb.wait_ns = (unsigned long long)wait_ms * 1000000ull;
        cudaGraph_t graph = nullptr;
        if(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            error = "cudaStreamBeginCapture failed";
            return RTACX_ERR_CUDA;
        }
        rtacx_status st = RTACX_OK;
        if(cudaMemsetAsync(d_sync, 0, sizeof(BatchSync), stream) != cudaSuccess) st = RTACX_ERR_CUDA;
        if(st == RTACX_OK) st = launch_fused_batch(error, cand.shape, cells, fb, fused_smem, fused_grid, stream);
        return finish_capture(st, graph);
    }

    // Graph of the staged form: reset of the work counter, five binning
    // launches, one persistent gather.
    rtacx_status capture_staged(const Candidate& cand, uint32_t n_pings)
    {
        gather_grid = (uint32_t)sm_count * (gather_smem <= 100 * 1024 ? 2u : 1u);
        rtacx_status prep = prepare_bin_batch(error, max_bins);
        if(prep == RTACX_OK) prep = prepare_gather_batch(error, cand.shape, gather_smem);
        if(prep != RTACX_OK) return prep;
        cudaGraph_t graph = nullptr;
        if(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            cudaGetLastError();
            error = "cudaStreamBeginCapture failed";
            return RTACX_ERR_CUDA;
        }
        rtacx_status st = RTACX_OK;
        if(cudaMemsetAsync(d_counter, 0, sizeof(uint32_t), stream) != cudaSuccess) st = RTACX_ERR_CUDA;
        if(st == RTACX_OK)
            st = launch_bin_batch(error, d_pings, n_pings, d_chunk_map, n_chunks, d_col_map, n_col,
                                  d_win_map, n_win, max_bins, stream);
        if(st == RTACX_OK)
            st = launch_gather_batch(error, cand.shape, d_pings, d_items, n_items, d_counter, gather_smem, gather_grid,
                                     stream);
        return finish_capture(st, graph);
    }

    rtacx_status finish_capture(rtacx_status st, cudaGraph_t graph)
    {
        const cudaError_t ec = cudaStreamEndCapture(stream, &graph);
        if(st != RTACX_OK || ec != cudaSuccess) {
            cudaGetLastError();
            if(graph) cudaGraphDestroy(graph);
            if(st == RTACX_OK) { error = std::string("stream capture failed: ") + cudaGetErrorString(ec); st = RTACX_ERR_CUDA; }
            return st;
        }
        size_t n_nodes = 0;
        graph_kernels = 0;
        if(cudaGraphGetNodes(graph, nullptr, &n_nodes) == cudaSuccess && n_nodes) {
            std::vector<cudaGraphNode_t> nodes(n_nodes);
            if(cudaGraphGetNodes(graph, nodes.data(), &n_nodes) == cudaSuccess)
                for(size_t k = 0; k < n_nodes; k++) {
                    cudaGraphNodeType t;
                    if(cudaGraphNodeGetType(nodes[k], &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) graph_kernels++;
                }
        }
        cudaGetLastError();
        const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if(ei != cudaSuccess) {
            cudaGetLastError();
            exec = nullptr;
            error = std::string("cudaGraphInstantiate failed: ") + cudaGetErrorString(ei);
            return RTACX_ERR_CUDA;
        }
        return RTACX_OK;
    }

    // Median device time of `reps` replays of the current graph.
    bool time_plan(int reps, float& ms)
    {
        cudaEvent_t a, b;
        if(cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) { cudaGetLastError(); return false; }
        std::vector<float> t;
        bool ok = cudaGraphLaunch(exec, stream) == cudaSuccess;   // warm-up
        for(int r = 0; ok && r < reps; r++) {
            float x = 0.0f;
            ok = cudaEventRecord(a, stream) == cudaSuccess && cudaGraphLaunch(exec, stream) == cudaSuccess &&
                 cudaEventRecord(b, stream) == cudaSuccess && cudaEventSynchronize(b) == cudaSuccess &&
                 cudaEventElapsedTime(&x, a, b) == cudaSuccess;
            t.push_back(x);
        }
        cudaEventDestroy(a); cudaEventDestroy(b);
        if(!ok) { cudaGetLastError(); return false; }
        std::sort(t.begin(), t.end());
        ms = t[t.size() / 2];
        return true;
    }
};

} // namespace rtacx

struct rtacx_batch {
    rtacx::Batch impl;
};

using namespace rtacx;

extern "C" {

rtacx_status rtacx_batch_create(rtacx_batch** out, int device)
{
    if(!out) return RTACX_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if(cudaSetDevice(device) != cudaSuccess) { cudaGetLastError(); return RTACX_ERR_CUDA; }
    rtacx_batch* b = new rtacx_batch();
    Batch& B = b->impl;
    B.device = device;
    if(cudaDeviceGetAttribute(&B.sm_count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
       cudaStreamCreateWithFlags(&B.stream, cudaStreamNonBlocking) != cudaSuccess ||
       cudaMalloc(&B.d_counter, sizeof(uint32_t)) != cudaSuccess ||
       cudaMalloc(&B.d_sync, sizeof(BatchSync)) != cudaSuccess ||
       cudaMalloc(&B.d_status, sizeof(uint32_t)) != cudaSuccess ||
       cudaMemset(B.d_status, 0, sizeof(uint32_t)) != cudaSuccess) {
        cudaGetLastError();
        rtacx_batch_destroy(b);
        return RTACX_ERR_CUDA;
    }
    *out = b;
    return RTACX_OK;
}

void rtacx_batch_destroy(rtacx_batch* b)
{
    if(!b) return;
    Batch& B = b->impl;
    cudaSetDevice(B.device);
    B.free_plan();
    B.drop(B.d_counter);
    B.drop(B.d_sync);
    B.drop(B.d_status);
    if(B.stream) cudaStreamDestroy(B.stream);
    delete b;
}

const char* rtacx_batch_last_error(const rtacx_batch* b)
{
    return b ? b->impl.error.c_str() : "null batch";
}

rtacx_status rtacx_batch_plan(rtacx_batch* b, const rtacx_ping_desc* pings, uint32_t count, uint32_t flags)
{
    if(!b) return RTACX_ERR_INVALID_ARGUMENT;
    Batch& B = b->impl;
    if(!pings || count == 0) { B.error = "empty batch"; return RTACX_ERR_INVALID_ARGUMENT; }
    if(cudaSetDevice(B.device) != cudaSuccess) { cudaGetLastError(); B.error = "cudaSetDevice failed"; return RTACX_ERR_CUDA; }
    std::set<const rtacx_ctx*> seen;
    for(uint32_t i = 0; i < count; i++) {
        const rtacx_ping_desc& p = pings[i];
        if(!p.ctx || !p.samples || !p.out || p.n == 0) { B.error = "ping " + std::to_string(i) + ": null pointer or no samples"; return RTACX_ERR_INVALID_ARGUMENT; }
        Context& c = p.ctx->impl;
        if(!c.configured) { B.error = "ping " + std::to_string(i) + ": context not configured"; return RTACX_ERR_NOT_CONFIGURED; }
        if(c.psf_tex) { B.error = "ping " + std::to_string(i) + ": RTACX_FLAG_TEXTURE_PSF is not supported in batches"; return RTACX_ERR_UNSUPPORTED; }
        if(c.device != B.device) { B.error = "ping " + std::to_string(i) + ": context on another device"; return RTACX_ERR_INVALID_ARGUMENT; }
        if(!seen.insert(p.ctx).second) { B.error = "ping " + std::to_string(i) + ": every ping needs its own context"; return RTACX_ERR_INVALID_ARGUMENT; }
        if(p.n >= (1ull << 32)) { B.error = "at most 2^32 - 1 samples per ping"; return RTACX_ERR_UNSUPPORTED; }
        if(reinterpret_cast<uintptr_t>(p.samples) % 4 != 0) { B.error = "sample buffers must be 4-byte aligned"; return RTACX_ERR_INVALID_ARGUMENT; }
        if(reinterpret_cast<uintptr_t>(p.out) % 8 != 0) { B.error = "pings must be 8-byte aligned"; return RTACX_ERR_INVALID_ARGUMENT; }
        if(!ensure_capacity(c, p.n)) { B.error = c.error; return RTACX_ERR_OUT_OF_MEMORY; }
    }
    B.pings.assign(pings, pings + count);
    B.staged = (flags & RTACX_BATCH_STAGED) != 0;
    B.choose_form();
    if(!(flags & RTACX_BATCH_AUTOTUNE)) {
        const rtacx_status st = B.build(Candidate{2, 4096});
        B.tuned_ms = 0.0f;
        return st;
    }
    // Autotune: every candidate is built, captured and timed on this batch.
    Candidate best{2, 4096};
    float best_ms = 1e30f;
    for(int shape = 0; shape < (B.per_row_2d ? 3 : 1); shape++)     // (the tile shape is the per-row 2D gather's)
        for(uint32_t per : {2048u, 4096u, 8192u}) {
            const Candidate cand{shape, per};
            if(B.build(cand) != RTACX_OK) continue;
            float ms;
            if(B.time_plan(3, ms) && ms < best_ms) { best_ms = ms; best = cand; }
        }
    if(best_ms >= 1e30f) { if(B.error.empty()) B.error = "no batch plan could be built"; return RTACX_ERR_CUDA; }
    const rtacx_status st = B.build(best);
    B.tuned_ms = best_ms;
    return st;
}

rtacx_status rtacx_batch_run(rtacx_batch* b, void* stream)
{
    if(!b) return RTACX_ERR_INVALID_ARGUMENT;
    Batch& B = b->impl;
    if(!B.exec) { B.error = "plan the batch first"; return RTACX_ERR_NOT_CONFIGURED; }
    if(cudaSetDevice(B.device) != cudaSuccess ||
       cudaGraphLaunch(B.exec, static_cast<cudaStream_t>(stream)) != cudaSuccess) {
        cudaGetLastError();
        B.error = "cudaGraphLaunch failed";
        return RTACX_ERR_CUDA;
    }
    return RTACX_OK;
}

rtacx_status rtacx_batch_status(rtacx_batch* b, void* stream)
{
    if(!b) return RTACX_ERR_INVALID_ARGUMENT;
    Batch& B = b->impl;
    if(cudaSetDevice(B.device) != cudaSuccess) { cudaGetLastError(); B.error = "cudaSetDevice failed"; return RTACX_ERR_CUDA; }
    const cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if(e != cudaSuccess) { B.error = std::string("stream: ") + cudaGetErrorString(e); return RTACX_ERR_CUDA; }
    uint32_t word = 0;
    if(cudaMemcpy(&word, B.d_status, sizeof(word), cudaMemcpyDeviceToHost) != cudaSuccess ||
       cudaMemset(B.d_status, 0, sizeof(word)) != cudaSuccess) {
        cudaGetLastError();
        B.error = "reading the batch status word failed";
        return RTACX_ERR_CUDA;
    }
    if(word) {
        B.error = "batch status word " + std::to_string(word) +
                  ((word & kErrBatchWaitTimeout) ? " (a grid-barrier wait expired; the batch's pings are incomplete)" : "");
        return RTACX_ERR_DEVICE;
    }
    return RTACX_OK;
}

rtacx_status rtacx_batch_graph_kernels(const rtacx_batch* b, uint32_t* kernels)
{
    if(!b || !kernels) return RTACX_ERR_INVALID_ARGUMENT;
    *kernels = b->impl.exec ? b->impl.graph_kernels : 0u;
    return RTACX_OK;
}

rtacx_status rtacx_diag_batch_barrier(rtacx_batch* b, uint32_t extra_arrivals, uint32_t wait_ms)
{
    if(!b || wait_ms == 0 || wait_ms > 10000 || extra_arrivals > 1) return RTACX_ERR_INVALID_ARGUMENT;
    b->impl.diag_extra = extra_arrivals;
    b->impl.wait_ms = wait_ms;
    return RTACX_OK;
}

rtacx_status rtacx_batch_tuning(const rtacx_batch* b, uint32_t* tile_rows, uint32_t* tile_bearings,
                                uint32_t* samples_per_cta, float* tuned_ms)
{
    if(!b) return RTACX_ERR_INVALID_ARGUMENT;
    const Batch& B = b->impl;
    if(tile_rows) *tile_rows = (uint32_t)gather_shape_rows(B.chosen.shape);
    if(tile_bearings) *tile_bearings = (uint32_t)gather_shape_bearings(B.chosen.shape);
    if(samples_per_cta) *samples_per_cta = B.chosen.per_cta;
    if(tuned_ms) *tuned_ms = B.tuned_ms;
    return RTACX_OK;
}

} // extern "C"
