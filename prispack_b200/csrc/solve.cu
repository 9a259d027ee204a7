// Device-resident operator, triangular preconditioners and the FCG driver.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <future>
#include <limits>

#include "../../include/prism_solve.h"
#include "kernels.cuh"
#include "solve.cuh"
#include "stream_sweep.cuh"
#include "flow_sweep.cuh"

namespace prism {

std::atomic<uint64_t>& launch_counter() {
    static std::atomic<uint64_t> c{0};
    return c;
}

namespace {
constexpr unsigned long long kWaitNs = 1000000000ull;  // 1 s per dependency wait
constexpr int kSpmvSubG = 8;                           // lanes per row in k_spmv_sub
constexpr int kSpmvG = 1, kSpmvU = 2;                  // k_spmv: lanes per row, rows per group and pass
// Rows of a dataflow slab the tuner tries.  More slabs share a wavefront's rows among more SMs
// and let a CTA take its next slab while the wavefront is elsewhere; fewer pay fewer hand-overs
// from slab to slab (about 1 us each).  Measured (us an M^-1 apply, 512 / 1024 / 2048 / 4096
// rows): IC 64^2 FP64 135 / 147 / 148 / 150, IC 512^2 FP64 2388 / 1759 / 1272 / 1088, IC 40^3
// FP64 443 / 431 / 483 / 567, AMSED 64^3 FP64 1601 / 1726 / 2055 / 2682, GMSLR 50^3 with float
// arithmetic 805 / 856 / 904 / 1020, AMSED 128^3 with float arithmetic 6483 / 5283 / 4563 / 5387.
// With 256 rows the first is 153 and only AMSED 64^3 gains (1500).
constexpr int kFlowSizes = 4;
constexpr uint32_t kFlowSlabRows[kFlowSizes] = {512, 1024, 2048, 4096};
// Rows of a slab of a block sweep: as many slabs as let the few CTAs of a group keep up with the
// wavefront (512^2, k = 64, 2 columns: 5,266 us with 2,048 rows, 3,047 with 4,096; 192^2: 682 with
// 1,024, 805 with 2,048).
static uint32_t block_slab_rows(uint32_t n) { return std::max(1024u, n / 64u); }
// the shapes A's SpMV may take (lanes per row, rows per group and pass): one lane per row
// suits short rows such as stencils, a group of lanes per row longer ones
constexpr int kSpmvShapes = 6;
constexpr int kSpmvShapeG[kSpmvShapes] = {1, 1, 2, 4, 8, 16};
constexpr int kSpmvShapeU[kSpmvShapes] = {2, 4, 2, 1, 1, 1};
}  // namespace

int vec_grid(const Handle& h, uint32_t n) {
    long want = ((long)n + kBlock - 1) / kBlock;
    long cap = (long)h.info.sms * 4;
    if (want < 1) want = 1;
    return (int)(want < cap ? want : cap);
}

void launch_fill(cudaStream_t st, const Handle& h, uint32_t n, double* p) {
    if (!n) return;
    k_fill_pending<<<vec_grid(h, n), kBlock, 0, st>>>(n, reinterpret_cast<unsigned long long*>(p));
    PRISM_LAUNCHED();
}

static void* slab_kernel(bool fp32, int op) {
    if (fp32) {
        switch (op) {
            case SWEEP_DIV: return (void*)k_sweep_slab<float, OP_DIV>;
            case SWEEP_MUL: return (void*)k_sweep_slab<float, OP_MUL>;
            case SWEEP_NONE: return (void*)k_sweep_slab<float, OP_NONE>;
            default: return (void*)k_sweep_slab<float, OP_PREDIV>;
        }
    }
    switch (op) {
        case SWEEP_DIV: return (void*)k_sweep_slab<double, OP_DIV>;
        case SWEEP_MUL: return (void*)k_sweep_slab<double, OP_MUL>;
        case SWEEP_NONE: return (void*)k_sweep_slab<double, OP_NONE>;
        default: return (void*)k_sweep_slab<double, OP_PREDIV>;
    }
}

static constexpr int kSlabThreads = 1024;

// acc32: single-precision arithmetic (float factor values only)
static void* stream_kernel(bool fp32, int op, bool acc32) {
    if (acc32) {
        switch (op) {
            case SWEEP_DIV: return (void*)k_sweep_stream<float, OP_DIV, float>;
            case SWEEP_MUL: return (void*)k_sweep_stream<float, OP_MUL, float>;
            case SWEEP_NONE: return (void*)k_sweep_stream<float, OP_NONE, float>;
            default: return (void*)k_sweep_stream<float, OP_PREDIV, float>;
        }
    }
    if (fp32) {
        switch (op) {
            case SWEEP_DIV: return (void*)k_sweep_stream<float, OP_DIV, double>;
            case SWEEP_MUL: return (void*)k_sweep_stream<float, OP_MUL, double>;
            case SWEEP_NONE: return (void*)k_sweep_stream<float, OP_NONE, double>;
            default: return (void*)k_sweep_stream<float, OP_PREDIV, double>;
        }
    }
    switch (op) {
        case SWEEP_DIV: return (void*)k_sweep_stream<double, OP_DIV, double>;
        case SWEEP_MUL: return (void*)k_sweep_stream<double, OP_MUL, double>;
        case SWEEP_NONE: return (void*)k_sweep_stream<double, OP_NONE, double>;
        default: return (void*)k_sweep_stream<double, OP_PREDIV, double>;
    }
}

// acc32 as above; entries: E of the layout; cols: as DevSweep::fl_cols (4 entries where not 0)
template <typename Low, typename Acc, int E, int C>
static void* flow_kernel_of(int op) {
    switch (op) {
        case SWEEP_DIV: return (void*)k_sweep_flow<Low, OP_DIV, Acc, E, C>;
        case SWEEP_MUL: return (void*)k_sweep_flow<Low, OP_MUL, Acc, E, C>;
        case SWEEP_NONE: return (void*)k_sweep_flow<Low, OP_NONE, Acc, E, C>;
        default: return (void*)k_sweep_flow<Low, OP_PREDIV, Acc, E, C>;
    }
}
static void* flow_kernel(bool fp32, int op, bool acc32, uint32_t entries, uint32_t cols) {
    switch (cols) {
        case 1: return fp32 ? flow_kernel_of<float, double, 4, 1>(op) : flow_kernel_of<double, double, 4, 1>(op);
        case 2: return fp32 ? flow_kernel_of<float, double, 4, 2>(op) : flow_kernel_of<double, double, 4, 2>(op);
        case 4: return fp32 ? flow_kernel_of<float, double, 4, 4>(op) : flow_kernel_of<double, double, 4, 4>(op);
        default: break;
    }
    if (entries == 4) {
        if (acc32) return flow_kernel_of<float, float, 4, 0>(op);
        return fp32 ? flow_kernel_of<float, double, 4, 0>(op) : flow_kernel_of<double, double, 4, 0>(op);
    }
    if (acc32) return flow_kernel_of<float, float, 8, 0>(op);
    return fp32 ? flow_kernel_of<float, double, 8, 0>(op) : flow_kernel_of<double, double, 8, 0>(op);
}

static FlowArgs flow_args(const Handle& h, const DevSweep& s, const double* in, double* out) {
    FlowArgs a;
    a.chunks = s.fl_chunks.get();
    a.hdr = reinterpret_cast<const uint4*>(s.fl_hdr.get());
    a.dg = s.fl_dg.get();
    a.warp = reinterpret_cast<const uint4*>(s.fl_warp.get());
    a.halo_ptr = s.fl_halo_ptr.get();
    a.halo = reinterpret_cast<const uint2*>(s.fl_halo.get());
    a.xch = s.fl_xch.get();
    a.ctl = s.fl_ctl.get();
    a.in = in;
    a.out = out;
    a.status = h.status.get();
    a.wait_ns = h.info.wait_ns;
    a.slabs = s.fl_slabs;
    a.slots = s.str_slots;
    a.dd = s.fl_dd.get();
    a.members = s.str_ctas;
    a.k = 1;
    return a;
}

// Columns a CTA of a block sweep takes, for k columns of an n-row operator.  One column has
// the shortest chain as long as the groups of CTAs that share the slabs are six or more; wider
// ones read a record for more columns.  Measured (us an IC apply, float values; 1 / 2 / 4
// columns): 192^2, k = 24: 524 / 560 / 764; 192^2, k = 64: 909 / 682 / 836; 512^2, k = 64:
// - / 3,047 / 2,672.  On 3D operators this choice against level order: IC 64^3 FP64, k = 8 / 24 /
// 64, 1,134 / 2,486 / 3,998 and 16,847 / 17,232 / 10,633; 100^3, k = 64, 14,505 and 18,211 (there
// choose_block_sweep mixes the two: 12,190).
uint32_t block_columns(uint32_t k, uint32_t n) { return k <= 24 ? 1u : (n < 131072 ? 2u : 4u); }

void launch_flow_block(const Handle& h, cudaStream_t st, const DevSweep& s, uint32_t k, const double* in, double* out) {
    FlowArgs a = flow_args(h, s, in, out);
    const uint32_t groups = (k + s.fl_cols - 1) / s.fl_cols;
    a.members = std::max(1u, std::min((uint32_t)h.info.sms / groups, s.fl_slabs));
    a.k = k;
    void* args[] = {&a};
    PRISM_CUDA(cudaLaunchCooperativeKernel(flow_kernel(s.fp32, s.op, false, s.fl_entries, s.fl_cols),
                                           dim3(groups * a.members), dim3(kFlowThreads), args, s.str_smem, st));
    PRISM_LAUNCHED();
}

void launch_sweep_prepare(const Handle& h, cudaStream_t st, const DevSweep& s, const double* in, double* out) {
    if (!s.n) return;
    if (s.layout == LAYOUT_FLOW) {
        if (s.paired) {
            k_flow_pair_rhs<<<vec_grid(h, s.n), kBlock, 0, st>>>(s.n, s.pair_ptr.get(), s.pair_dep.get(),
                                                                s.pair_coef.get(), in, s.pair_rhs.get());
            PRISM_LAUNCHED();
        }
        return;
    }
    if (s.layout != LAYOUT_STREAM) {
        launch_fill(st, h, s.n, out);
        return;
    }
    if (s.paired) {
        // the prep reads other rows of `in`: when in == out, the outputs are marked afterwards
        const int mark = in != out ? 1 : 0;
        if (s.acc32)
            k_stream_prep_pair<float><<<vec_grid(h, s.n), kBlock, 0, st>>>(
                s.n, s.str_in_slot.get(), s.pair_ptr.get(), s.pair_dep.get(), s.pair_coef.get(), in,
                reinterpret_cast<float*>(s.str_blob.get()), reinterpret_cast<unsigned long long*>(out), mark);
        else
            k_stream_prep_pair<double><<<vec_grid(h, s.n), kBlock, 0, st>>>(
                s.n, s.str_in_slot.get(), s.pair_ptr.get(), s.pair_dep.get(), s.pair_coef.get(), in,
                reinterpret_cast<double*>(s.str_blob.get()), reinterpret_cast<unsigned long long*>(out), mark);
        PRISM_LAUNCHED();
        if (!mark) launch_fill(st, h, s.n, out);
        return;
    }
    if (s.acc32)
        k_stream_prep<float><<<vec_grid(h, s.n), kBlock, 0, st>>>(s.n, s.str_in_slot.get(), in,
                                                                  reinterpret_cast<float*>(s.str_blob.get()),
                                                                  reinterpret_cast<unsigned long long*>(out));
    else
        k_stream_prep<double><<<vec_grid(h, s.n), kBlock, 0, st>>>(s.n, s.str_in_slot.get(), in,
                                                                   reinterpret_cast<double*>(s.str_blob.get()),
                                                                   reinterpret_cast<unsigned long long*>(out));
    PRISM_LAUNCHED();
}

void launch_sweep_kernel(const Handle& h, cudaStream_t st, const DevSweep& s, const double* in, double* out) {
    if (!s.n) return;
    if (s.layout == LAYOUT_FLOW) {
        FlowArgs a = flow_args(h, s, s.paired ? s.pair_rhs.get() : in, out);
        void* args[] = {&a};
        PRISM_CUDA(cudaLaunchCooperativeKernel(flow_kernel(s.fp32, s.op, s.acc32, s.fl_entries, 0), dim3(s.str_ctas), dim3(kFlowThreads),
                                               args, s.str_smem, st));
        PRISM_LAUNCHED();
        return;
    }
    if (s.layout == LAYOUT_STREAM) {
        (void)in;
        StreamArgs a;
        a.blob = s.str_blob.get();
        a.meta = reinterpret_cast<const uint4*>(s.str_meta.get());
        a.cta_round = s.str_cta_round.get();
        a.slab_start = s.str_slab_start.get();
        a.halo_ptr = s.str_halo_ptr.get();
        a.halo_row = s.str_halo_row.get();
        a.halo_sw = s.str_halo_sw.get();
        a.n = s.n;
        a.ring_bytes = s.str_ring;
        a.meta_slots = s.str_meta_slots;
        a.slots = s.str_slots;
        a.out = out;
        a.status = h.status.get();
        a.wait_ns = kWaitNs;
        void* args[] = {&a};
        PRISM_CUDA(cudaLaunchCooperativeKernel(stream_kernel(s.fp32, s.op, s.acc32), dim3(s.str_ctas), dim3(kStrThreads), args,
                                               s.str_smem, st));
        PRISM_LAUNCHED();
        return;
    }
    if (s.num_ctas > 0) {
        void* fn = slab_kernel(s.fp32, s.op);
        uint32_t n = s.n, rpc = s.rows_per_cta, smem_rows = s.smem_rows;
        const uint32_t* cta_pos = s.cta_pos.get();
        const uint32_t* order = s.order.get();
        const uint32_t* rowptr = s.rowptr.get();
        const uint32_t* col = s.col.get();
        const void* val = s.fp32 ? (const void*)s.val32.get() : (const void*)s.val64.get();
        const double* diag = s.diag.get();
        int* status = h.status.get();
        unsigned long long wait = kWaitNs;
        void* args[] = {&n, &rpc, &smem_rows, &cta_pos, &order, &rowptr, &col, &val, &diag, &in, &out, &status, &wait};
        PRISM_CUDA(cudaLaunchCooperativeKernel(fn, dim3(s.num_ctas), dim3(kSlabThreads), args,
                                               (size_t)s.smem_rows * sizeof(double), st));
        PRISM_LAUNCHED();
        return;
    }
    long want = ((long)s.n * 32 + kBlock - 1) / kBlock;
    long cap = (long)h.info.sms * h.info.sweep_blocks_per_sm;
    int grid = (int)(want < cap ? want : cap);
    void* fn = nullptr;
    if (s.fp32) {
        switch (s.op) {
            case SWEEP_DIV: fn = (void*)k_sweep<float, OP_DIV>; break;
            case SWEEP_MUL: fn = (void*)k_sweep<float, OP_MUL>; break;
            case SWEEP_NONE: fn = (void*)k_sweep<float, OP_NONE>; break;
            default: fn = (void*)k_sweep<float, OP_PREDIV>; break;
        }
    } else {
        switch (s.op) {
            case SWEEP_DIV: fn = (void*)k_sweep<double, OP_DIV>; break;
            case SWEEP_MUL: fn = (void*)k_sweep<double, OP_MUL>; break;
            case SWEEP_NONE: fn = (void*)k_sweep<double, OP_NONE>; break;
            default: fn = (void*)k_sweep<double, OP_PREDIV>; break;
        }
    }
    uint32_t n = s.n;
    const uint32_t* order = s.order.get();
    const uint32_t* rowptr = s.rowptr.get();
    const uint32_t* col = s.col.get();
    const void* val = s.fp32 ? (const void*)s.val32.get() : (const void*)s.val64.get();
    const double* diag = s.diag.get();
    int* status = h.status.get();
    unsigned long long wait = kWaitNs;
    void* args[] = {&n, &order, &rowptr, &col, &val, &diag, &in, &out, &status, &wait};
    // Cooperative launch: all blocks co-resident, which the level-order
    // progress argument of k_sweep relies on.
    PRISM_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kBlock), args, 0, st));
    PRISM_LAUNCHED();
}

void launch_sweep(const Handle& h, cudaStream_t st, const DevSweep& s, const double* in, double* out) {
    if (s.streamed()) launch_sweep_prepare(h, st, s, in, out);
    launch_sweep_kernel(h, st, s, in, out);
}

void launch_spmv(const Handle& h, cudaStream_t st, uint32_t nrows, const uint32_t* rowptr, const uint32_t* col,
                 const double* val, const double* x, double* y, int sub) {
    if (!nrows) return;
    long cap = (long)h.info.sms * 8;
    ReduceSlot none{nullptr, nullptr, nullptr};
    if (sub) {
        long want = ((long)nrows * kSpmvSubG + kBlock - 1) / kBlock;
        k_spmv_sub<kSpmvSubG><<<(int)(want < cap ? want : cap), kBlock, 0, st>>>(nrows, rowptr, col, val, x, y);
    } else {
        const long rows_per_block = (long)(kBlock / 32) * (32 / kSpmvG) * kSpmvU;
        long want = ((long)nrows + rows_per_block - 1) / rows_per_block;
        k_spmv<kSpmvG, kSpmvU, 0><<<(int)(want < cap ? want : cap), kBlock, 0, st>>>(nrows, rowptr, col, val, x, y,
                                                                                   nullptr, nullptr, none);
    }
    PRISM_LAUNCHED();
}

void launch_adjoint_outer(const Handle& h, cudaStream_t st, const double* lambda, const double* x, double* grad) {
    k_adjoint_outer<<<vec_grid(h, h.A.n), kBlock, 0, st>>>(h.A.n, h.A.rowptr.get(), h.A.col.get(), lambda, x, grad);
    PRISM_LAUNCHED();
}

// ============================================================================
// Bounded-wait self test: a two-row sweep whose first position depends on the
// second one, run by a single warp.  The warp reaches position 0 first, so the
// value it waits for is never produced; the wait must run out after wait_ns,
// raise status 6 and return, leaving the context usable (checked by a normal
// sweep afterwards).
// ============================================================================
int selftest_wait_timeout(int device, unsigned long long wait_ns, int* device_status) {
    PRISM_CUDA(cudaSetDevice(device));
    cudaStream_t st;
    PRISM_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    // position 0 = row 0 (depends on row 1), position 1 = row 1 (no dependency)
    const uint32_t h_order[2] = {0, 1}, h_rowptr[3] = {0, 1, 1}, h_col[1] = {1};
    const double h_val[1] = {0.5}, h_diag[2] = {1.0, 1.0}, h_in[2] = {1.0, 2.0};
    DevBuf<uint32_t> order(2), rowptr(3), col(1);
    DevBuf<double> val(1), diag(2), in(2), out(2);
    DevBuf<int> status(1);
    order.upload(h_order, 2, st); rowptr.upload(h_rowptr, 3, st); col.upload(h_col, 1, st);
    val.upload(h_val, 1, st); diag.upload(h_diag, 2, st); in.upload(h_in, 2, st);
    PRISM_CUDA(cudaMemsetAsync(status.get(), 0, sizeof(int), st));
    k_fill_pending<<<1, 32, 0, st>>>(2, reinterpret_cast<unsigned long long*>(out.get()));
    PRISM_LAUNCHED();
    k_sweep<double, OP_NONE><<<1, 32, 0, st>>>(2, order.get(), rowptr.get(), col.get(), val.get(), diag.get(),
                                               in.get(), out.get(), status.get(), wait_ns);
    PRISM_LAUNCHED();
    int s = -1;
    PRISM_CUDA(cudaMemcpyAsync(&s, status.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
    PRISM_CUDA(cudaStreamSynchronize(st));
    *device_status = s;
    // the context is still usable: the same rows in a valid order solve normally
    const uint32_t g_order[2] = {1, 0}, g_rowptr[3] = {0, 0, 1};
    order.upload(g_order, 2, st); rowptr.upload(g_rowptr, 3, st);
    PRISM_CUDA(cudaMemsetAsync(status.get(), 0, sizeof(int), st));
    k_fill_pending<<<1, 32, 0, st>>>(2, reinterpret_cast<unsigned long long*>(out.get()));
    PRISM_LAUNCHED();
    k_sweep<double, OP_NONE><<<1, 32, 0, st>>>(2, order.get(), rowptr.get(), col.get(), val.get(), diag.get(),
                                               in.get(), out.get(), status.get(), wait_ns);
    PRISM_LAUNCHED();
    double h_out[2] = {0, 0};
    int s2 = -1;
    PRISM_CUDA(cudaMemcpyAsync(h_out, out.get(), sizeof(h_out), cudaMemcpyDeviceToHost, st));
    PRISM_CUDA(cudaMemcpyAsync(&s2, status.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
    PRISM_CUDA(cudaStreamSynchronize(st));
    PRISM_CUDA(cudaStreamDestroy(st));
    // row 1 = 2, row 0 = 1 - 0.5 * 2 = 0
    if (s2 != 0 || h_out[0] != 0.0 || h_out[1] != 2.0)
        throw Error(PRISM_ERR_CUDA, "context unusable after a timed-out wait");
    return 0;
}

// ============================================================================
// Handle
// ============================================================================
void init_device_info(DeviceInfo& info, int device) {
    info.device = device;
    PRISM_CUDA(cudaDeviceGetAttribute(&info.sms, cudaDevAttrMultiProcessorCount, device));
    info.co_resident = info.sms;
    int occ = 0, occ2 = 0;
    PRISM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sweep<double, OP_DIV>, kBlock, 0));
    PRISM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, k_sweep<float, OP_DIV>, kBlock, 0));
    occ = occ < occ2 ? occ : occ2;
    // a fraction of the co-resident capacity: enough warps to cover a wavefront,
    // few enough pollers to leave L2 bandwidth to the producers
    int want = 4;
    if (const char* e = std::getenv("PRISM_SWEEP_BLOCKS_PER_SM")) want = std::atoi(e);
    if (want < 1) want = 1;
    info.sweep_blocks_per_sm = occ < want ? (occ > 0 ? occ : 1) : want;
    PRISM_CUDA(cudaDeviceGetAttribute(&info.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    if (const char* e = std::getenv("PRISM_SWEEP_KERNEL")) {
        const std::string k(e);
        info.sweep_kernel = k == "global" ? 1 : (k == "slab" ? 2 : (k == "stream" ? 3 : (k == "rounds" ? 4 : 0)));
    }
    if (const char* e = std::getenv("PRISM_SLAB_MIN_ROWS")) info.slab_min_rows = (uint32_t)std::atoi(e);
    if (const char* e = std::getenv("PRISM_SLAB_MAX_ROWS")) info.slab_max_rows = (uint32_t)std::atoi(e);
    if (info.slab_min_rows < 32) info.slab_min_rows = 32;
    // the slab kernel runs one 1024-thread CTA per SM with up to the whole opt-in shared memory
    if (const char* e = std::getenv("PRISM_STREAM_MIN_ROWS")) info.stream_min_rows = (uint32_t)std::atoi(e);
    if (const char* e = std::getenv("PRISM_STREAM_PAIR")) {  // 0 never, 1 the tuner decides, 2 always
        const int v = std::atoi(e);
        info.stream_pair = v < 0 ? 0 : (v > 2 ? 2 : v);
    }
    if (info.stream_min_rows < 32) info.stream_min_rows = 32;
    if (const char* e = std::getenv("PRISM_FLOW_ROWS")) info.flow_rows = (uint32_t)std::max(32, std::atoi(e));
    for (bool f32 : {false, true})
        for (int op = 0; op < 4; ++op) {
            PRISM_CUDA(cudaFuncSetAttribute(slab_kernel(f32, op), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            info.max_smem_optin));
            PRISM_CUDA(cudaFuncSetAttribute(stream_kernel(f32, op, false), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            info.max_smem_optin));
            for (uint32_t e : {4u, 8u}) {
                PRISM_CUDA(cudaFuncSetAttribute(flow_kernel(f32, op, false, e, 0),
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, info.max_smem_optin));
                if (f32)
                    PRISM_CUDA(cudaFuncSetAttribute(flow_kernel(true, op, true, e, 0),
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, info.max_smem_optin));
            }
            for (uint32_t c : {1u, 2u, 4u})
                PRISM_CUDA(cudaFuncSetAttribute(flow_kernel(f32, op, false, 4, c),
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, info.max_smem_optin));
            if (f32)
                PRISM_CUDA(cudaFuncSetAttribute(stream_kernel(true, op, true),
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, info.max_smem_optin));
        }
}

Handle::~Handle() {
    P.reset();
    if (pinned) cudaFreeHost(pinned);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (own_stream && stream) cudaStreamDestroy(stream);
}

void Handle::ensure_workspace() {
    const uint32_t n = A.n;
    if (y.size() < n) {  // the last one: all are there
        r.alloc(n); w.alloc(n); d.alloc(n); v.alloc(n); y.alloc(n);
    }
}

namespace {
template <int G, int U>
void spmv_shape_launch(const Handle& h, const double* x, double* yout, int ndot, const double* z, const double* q,
                       ReduceSlot slot) {
    const uint32_t n = h.A.n;
    const long rows_per_block = (long)(kBlock / 32) * (32 / G) * U;
    long want = ((long)n + rows_per_block - 1) / rows_per_block;
    long cap = (long)h.info.sms * 8;
    int grid = (int)(want < cap ? want : cap);
    if (grid > Reducer::kMaxGrid) grid = Reducer::kMaxGrid;
    const uint32_t* rp = h.A.rowptr.get();
    const uint32_t* ci = h.A.col.get();
    const double* va = h.A.val.get();
    if (ndot == 0) k_spmv<G, U, 0><<<grid, kBlock, 0, h.stream>>>(n, rp, ci, va, x, yout, z, q, slot);
    else if (ndot == 1) k_spmv<G, U, 1><<<grid, kBlock, 0, h.stream>>>(n, rp, ci, va, x, yout, z, q, slot);
    else k_spmv<G, U, 2><<<grid, kBlock, 0, h.stream>>>(n, rp, ci, va, x, yout, z, q, slot);
    PRISM_LAUNCHED();
}
}  // namespace

void Handle::spmv(const double* x, double* yout, int ndot, const double* z, const double* q, int scalar) {
    if (!A.n) return;
    const ReduceSlot slot = red.slot(scalar);
    switch (spmv_shape) {
        case 1: spmv_shape_launch<kSpmvShapeG[1], kSpmvShapeU[1]>(*this, x, yout, ndot, z, q, slot); break;
        case 2: spmv_shape_launch<kSpmvShapeG[2], kSpmvShapeU[2]>(*this, x, yout, ndot, z, q, slot); break;
        case 3: spmv_shape_launch<kSpmvShapeG[3], kSpmvShapeU[3]>(*this, x, yout, ndot, z, q, slot); break;
        case 4: spmv_shape_launch<kSpmvShapeG[4], kSpmvShapeU[4]>(*this, x, yout, ndot, z, q, slot); break;
        case 5: spmv_shape_launch<kSpmvShapeG[5], kSpmvShapeU[5]>(*this, x, yout, ndot, z, q, slot); break;
        default: spmv_shape_launch<kSpmvShapeG[0], kSpmvShapeU[0]>(*this, x, yout, ndot, z, q, slot); break;
    }
}

void Handle::spmv_shape_of(int* lanes_per_row, int* rows_per_pass) const {
    const int s = spmv_shape >= 0 && spmv_shape < kSpmvShapes ? spmv_shape : 0;
    if (lanes_per_row) *lanes_per_row = kSpmvShapeG[s];
    if (rows_per_pass) *rows_per_pass = kSpmvShapeU[s];
}

// Times A x with each shape (one warm-up and three timed launches, the plain product
// without fused dot products) and keeps the fastest; PRISM_SPMV_SHAPE (0..5) forces one.
void Handle::tune_spmv() {
    spmv_shape = 0;
    if (const char* e = std::getenv("PRISM_SPMV_SHAPE")) {
        const int v = std::atoi(e);
        spmv_shape = v >= 0 && v < kSpmvShapes ? v : 0;
        return;
    }
    if (A.n == 0) return;
    DevBuf<double> x(A.n), y(A.n);
    std::vector<double> ones(A.n, 1.0);
    x.upload(ones.data(), A.n, stream);
    float best = 0.f;
    int best_s = 0;
    for (int s = 0; s < kSpmvShapes; ++s) {
        spmv_shape = s;
        spmv(x.get(), y.get());
        PRISM_CUDA(cudaEventRecord(ev0, stream));
        for (int it = 0; it < 3; ++it) spmv(x.get(), y.get());
        PRISM_CUDA(cudaEventRecord(ev1, stream));
        PRISM_CUDA(cudaEventSynchronize(ev1));
        float ms = 0.f;
        PRISM_CUDA(cudaEventElapsedTime(&ms, ev0, ev1));
        if (s == 0 || ms < best) {
            best = ms;
            best_s = s;
        }
    }
    spmv_shape = best_s;
}

void Handle::check_status() {
    int s = 0;
    PRISM_CUDA(cudaMemcpyAsync(&s, status.get(), sizeof(int), cudaMemcpyDeviceToHost, stream));
    PRISM_CUDA(cudaStreamSynchronize(stream));
    if (s != 0) {
        PRISM_CUDA(cudaMemsetAsync(status.get(), 0, sizeof(int), stream));
        throw Error(s, "device-side wait ran out of time in a triangular sweep (status " + std::to_string(s) + ")");
    }
}

// ============================================================================
// Sweeps and triangular preconditioners
// ============================================================================
void DevSweep::release() {
    order.release(); rowptr.release(); col.release(); cta_pos.release();
    val64.release(); diag.release(); val32.release();
    str_blob.release(); str_meta.release(); str_cta_round.release(); str_slab_start.release(); str_in_slot.release();
    str_halo_ptr.release(); str_halo_row.release(); str_halo_sw.release();
    num_ctas = rows_per_cta = smem_rows = 0;
    str_ctas = str_ring = str_meta_slots = str_slots = str_rounds = str_smem = 0;
    str_nnz = 0;
    str_round_cap = 0;
    fl_chunks.release(); fl_dg.release(); fl_xch.release();
    fl_hdr.release(); fl_warp.release(); fl_halo_ptr.release(); fl_halo.release(); fl_ctl.release();
    fl_slabs = fl_entries = fl_published = fl_cols = 0;
    fl_dd.release();
    pair_ptr.release(); pair_dep.release(); pair_coef.release(); pair_rhs.release();
    paired = false;
    n = num_levels = 0;  // empty: nothing launches on a released sweep
}

template <typename Low>
StreamPlan plan_stream(const Sweep<Low>& s0, const DeviceInfo& info, bool acc32) {
    // One persistent CTA per SM (fewer for small sweeps); shared memory holds the
    // round table, the value slots and, in what is left, the ring the round
    // records stream through.
    StreamPlan P;
    const uint32_t nn = s0.n;
    if (nn == 0) return P;
    const uint32_t ctas_req = stream_slab_count(nn, (uint32_t)info.sms, info.stream_min_rows);
    const std::vector<uint32_t> start = slab_ranges<Low>(s0, ctas_req);
    if (start.size() - 1 > (size_t)info.co_resident) return P;  // one co-resident CTA a slab: too many independent blocks
    const uint64_t smem = (uint64_t)info.max_smem_optin;
    StreamLayout& L = P.L;
    const bool a32 = acc32 && std::is_same<Low, float>::value;
    const uint32_t slot_bytes = a32 ? 4 : 8;  // one value slot
    const uint32_t vb = (uint32_t)sizeof(Low);
    const uint64_t base_smem = stream_smem(0, 0, slot_bytes, vb, 0).total;  // everything but table and slots
    if (smem <= base_smem) return P;
    const uint32_t slot_cap = (uint32_t)std::min<uint64_t>(kNoSlot, (smem - base_smem) / slot_bytes / 2);
    // While round i is computed the row threads hold rounds i and i + 1 and wait for
    // round i + 2's record: two live records and room for a third, which a circular ring
    // of four of the largest records always has in one piece.  Where a round's record
    // is too large for that (rows of many entries), the rounds are cut shorter.
    uint32_t cap = 0;
    uint64_t fixed = 0;
    bool fits = false;
    for (int attempt = 0; attempt < 4 && !fits; ++attempt) {
        L = StreamLayout();
        if (!stream_layout<Low>(s0, start, slot_cap, slot_bytes, L, nullptr, nullptr, nullptr, cap)) return P;
        if (L.max_rounds_per_cta > smem / 16 || L.slots > kNoSlot) return P;
        fixed = stream_smem(L.max_rounds_per_cta, L.slots, slot_bytes, vb, 0).total;
        fits = fixed + 4ull * L.max_round_bytes <= smem;
        if (!fits) {
            if (fixed + 4096 >= smem) return P;
            const uint64_t room = (smem - fixed) / 4 * 7 / 8 >> attempt;  // margin for rounds and slots
            cap = (uint32_t)std::max<uint64_t>(room & ~15ull, 1024);
        }
    }
    if (!fits) return P;
    P.ok = true;
    P.fp32 = std::is_same<Low, float>::value;
    P.a32 = a32;
    P.n = s0.n;
    P.num_levels = s0.num_levels;
    P.op = s0.op;
    P.ctas = (uint32_t)start.size() - 1;
    P.ctas_req = ctas_req;
    P.slot_bytes = slot_bytes;
    P.cap = cap;
    P.ring = (uint32_t)((smem - fixed) & ~15ull);
    P.smem = stream_smem(L.max_rounds_per_cta, L.slots, slot_bytes, vb, P.ring).total;  // <= smem
    P.nnz = s0.val.size();
    return P;
}
template StreamPlan plan_stream<double>(const Sweep<double>&, const DeviceInfo&, bool);
template StreamPlan plan_stream<float>(const Sweep<float>&, const DeviceInfo&, bool);

template <typename Low>
StreamPlan plan_flow(const Sweep<Low>& s0, const DeviceInfo& info, bool acc32, uint32_t rows, uint32_t cols) {
    StreamPlan P;
    const uint32_t nn = s0.n;
    if (nn == 0) return P;
    P.a32 = acc32 && std::is_same<Low, float>::value;
    P.cols = cols;
    P.slot_bytes = (P.a32 ? 4 : 8) * std::max(cols, 1u);
    const uint32_t cap = ((uint32_t)info.max_smem_optin - flow_smem(0, P.slot_bytes)) / P.slot_bytes;
    // A slab whose rows and halo do not fit in shared memory is split further.
    uint32_t want = std::max(1u, (nn + rows - 1) / rows);
    for (;; want *= 2) {
        const std::vector<uint32_t> start = slab_ranges<Low>(s0, want);
        if (flow_layout<Low>(s0, start, cap, P.F, nullptr, nullptr, cols ? 4 : 0)) break;
        if (nn / want < 64) return P;
    }
    P.ok = P.flow = true;
    P.fp32 = std::is_same<Low, float>::value;
    P.n = s0.n;
    P.num_levels = s0.num_levels;
    P.op = s0.op;
    P.ctas_req = want;
    P.ctas = std::min(P.F.slabs, (uint32_t)info.sms);
    P.smem = flow_smem(P.F.slots, P.slot_bytes);
    P.nnz = s0.val.size();
    return P;
}
template StreamPlan plan_flow<double>(const Sweep<double>&, const DeviceInfo&, bool, uint32_t, uint32_t);
template StreamPlan plan_flow<float>(const Sweep<float>&, const DeviceInfo&, bool, uint32_t, uint32_t);

void DevSweep::commit_stream(StreamPlan&& P, cudaStream_t st) {
    const StreamLayout& L = P.L;
    release();
    n = P.n;
    num_levels = P.num_levels;
    op = P.op;
    fp32 = P.fp32;
    acc32 = P.a32;
    str_ctas = P.ctas;
    str_ctas_req = P.ctas_req;
    str_nnz = P.nnz;
    str_smem = P.smem;
    if (P.pm) {
        paired = true;
        pair_ptr.upload(P.pm->ptr.data(), P.pm->ptr.size(), st);
        pair_dep.upload(P.pm->dep.data(), P.pm->dep.size(), st);
        pair_coef.upload(P.pm->coef.data(), P.pm->coef.size(), st);
        if (pair_dep.size() == 0) pair_dep.alloc(1);  // valid pointers for the prep
        if (pair_coef.size() == 0) pair_coef.alloc(1);
    }
    if (P.flow) {
        const FlowLayout& F = P.F;
        layout = LAYOUT_FLOW;
        fl_slabs = F.slabs;
        str_slots = F.slots;
        fl_entries = F.entries;
        fl_chunks.alloc(F.chunks.size() + kFlowPad);  // the kernel brings lines past the end into L2
        fl_chunks.upload(F.chunks.data(), F.chunks.size(), st);
        fl_hdr.upload(F.hdr.data(), F.hdr.size(), st);
        fl_warp.upload(F.warp.data(), F.warp.size(), st);
        fl_halo_ptr.upload(F.halo_ptr.data(), F.halo_ptr.size(), st);
        fl_halo.upload(F.halo.data(), F.halo.size(), st);
        if (fl_halo.size() == 0) fl_halo.alloc(2);
        std::vector<float> dgf;
        if (acc32) {
            dgf.assign(F.dg.begin(), F.dg.end());
            fl_dg.upload(reinterpret_cast<const unsigned char*>(dgf.data()), dgf.size() * sizeof(float), st);
        } else {
            fl_dg.upload(reinterpret_cast<const unsigned char*>(F.dg.data()), F.dg.size() * sizeof(double), st);
        }
        fl_cols = P.cols;
        fl_published = F.published;
        if (fl_cols) {
            std::vector<double> dd(F.dg.size(), 1.0);
            if (op == SWEEP_DIV || op == SWEEP_PREDIV)
                for (uint32_t r = 0; r < n; ++r) dd[F.dg_pos[r]] = P.diag[r];
            fl_dd.upload(dd.data(), dd.size(), st);
            PRISM_CUDA(cudaStreamSynchronize(st));
        } else {
            // epoch 0 everywhere: the first sweep is epoch 1
            fl_xch.alloc((size_t)std::max(F.published, 1u) * (acc32 ? sizeof(FlowWord<float>) : sizeof(FlowWord<double>)));
            PRISM_CUDA(cudaMemsetAsync(fl_xch.get(), 0, fl_xch.size(), st));
        }
        fl_ctl.alloc(2);
        PRISM_CUDA(cudaMemsetAsync(fl_ctl.get(), 0, 2 * sizeof(uint32_t), st));
        if (paired) pair_rhs.alloc(n);
        PRISM_CUDA(cudaStreamSynchronize(st));
        return;
    }
    layout = LAYOUT_STREAM;
    str_slot_bytes = P.slot_bytes;
    str_round_cap = P.cap;
    str_ring = P.ring;
    str_meta_slots = L.max_rounds_per_cta;
    str_slots = L.slots;
    str_rounds = L.num_rounds;
    str_blob.upload(L.blob.data(), L.blob.size(), st);
    str_meta.upload(L.meta.data(), L.meta.size(), st);
    str_cta_round.upload(L.cta_round.data(), L.cta_round.size(), st);
    str_slab_start.upload(L.slab_start.data(), L.slab_start.size(), st);
    str_in_slot.upload(L.in_slot.data(), L.in_slot.size(), st);
    str_halo_ptr.upload(L.halo_ptr.data(), L.halo_ptr.size(), st);
    str_halo_row.upload(L.halo_row.data(), L.halo_row.size(), st);
    str_halo_sw.upload(L.halo_sw.data(), L.halo_sw.size(), st);
    if (str_halo_row.size() == 0) str_halo_row.alloc(1);  // valid pointers for the kernel
    if (str_halo_sw.size() == 0) str_halo_sw.alloc(1);
    PRISM_CUDA(cudaStreamSynchronize(st));
}

template <typename Low>
void DevSweep::upload_block(const Sweep<Low>& s, const DeviceInfo& info, uint32_t cols, cudaStream_t st) {
    if (s.n > 0) {
        StreamPlan P = plan_flow<Low>(s, info, false, info.flow_rows ? info.flow_rows : block_slab_rows(s.n), cols);
        if (P.ok) {
            if (s.op == SWEEP_DIV || s.op == SWEEP_PREDIV) {
                P.diag.resize(s.n);
                for (uint32_t p = 0; p < s.n; ++p) P.diag[s.order[p]] = s.diag[p];
            }
            commit_stream(std::move(P), st);
            return;
        }
    }
    upload(s, info, LAYOUT_LEVEL, st);
}
template void DevSweep::upload_block<double>(const Sweep<double>&, const DeviceInfo&, uint32_t, cudaStream_t);
template void DevSweep::upload_block<float>(const Sweep<float>&, const DeviceInfo&, uint32_t, cudaStream_t);

void DevSweep::block_workspace(uint32_t k, cudaStream_t st) {
    if (!fl_cols) return;
    const size_t groups = (k + fl_cols - 1) / fl_cols;
    const size_t bytes = std::max(fl_published, 1u) * groups * fl_cols * sizeof(FlowWord<double>);
    if (fl_xch.size() >= bytes) return;
    fl_xch.alloc(bytes);
    PRISM_CUDA(cudaMemsetAsync(fl_xch.get(), 0, bytes, st));  // no entry of the epochs to come
}

template <typename Low>
bool DevSweep::upload(const Sweep<Low>& sweep, const DeviceInfo& info, int lay, cudaStream_t st) {
    if (lay == LAYOUT_STREAM || lay == LAYOUT_FLOW) {
        StreamPlan P = lay == LAYOUT_FLOW
                           ? plan_flow<Low>(sweep, info, acc32, info.flow_rows ? info.flow_rows : kFlowSlabRows[0])
                           : plan_stream<Low>(sweep, info, acc32);
        if (!P.ok) return false;
        commit_stream(std::move(P), st);
        return true;
    }
    const Sweep<Low>& s0 = sweep;
    release();
    layout = lay;
    n = s0.n;
    num_levels = s0.num_levels;
    op = s0.op;
    fp32 = std::is_same<Low, float>::value;
    const Sweep<Low>* s = &s0;
    Sweep<Low> slab;
    std::vector<uint32_t> cpos;
    if (lay == LAYOUT_SLAB && n > 0) {
        // As many rows per slab as shared memory holds: the dependencies of a
        // row reach back about one grid plane, so large slabs keep most of them
        // (and the critical path through them) inside one CTA, where a
        // dependency costs a shared-memory poll instead of an L2 round trip.
        const uint32_t cap = (uint32_t)(info.max_smem_optin / sizeof(double));
        uint32_t per = std::max<uint32_t>(std::min<uint32_t>(cap, info.slab_max_rows), info.slab_min_rows);
        uint32_t ctas = (n + per - 1) / per;
        if (ctas > (uint32_t)info.sms) ctas = (uint32_t)info.sms;
        if (ctas < 1) ctas = 1;
        rows_per_cta = (n + ctas - 1) / ctas;
        num_ctas = (n + rows_per_cta - 1) / rows_per_cta;
        smem_rows = std::min<uint32_t>(rows_per_cta, (uint32_t)(info.max_smem_optin / sizeof(double)));
        slab_layout<Low>(s0, num_ctas, rows_per_cta, cpos, slab);
        s = &slab;
        cta_pos.upload(cpos.data(), cpos.size(), st);
    } else {
        layout = LAYOUT_LEVEL;
    }
    order.upload(s->order.data(), s->order.size(), st);
    rowptr.upload(s->rowptr.data(), s->rowptr.size(), st);
    col.upload(s->col.data(), s->col.size(), st);
    diag.upload(s->diag.data(), s->diag.size(), st);
    if (fp32) val32.upload(reinterpret_cast<const float*>(s->val.data()), s->val.size(), st);
    else val64.upload(reinterpret_cast<const double*>(s->val.data()), s->val.size(), st);
    // keep at least one element so kernels always get valid pointers
    if (col.size() == 0) col.alloc(1);
    if (fp32 && val32.size() == 0) val32.alloc(1);
    if (!fp32 && val64.size() == 0) val64.alloc(1);
    PRISM_CUDA(cudaStreamSynchronize(st));
    return true;
}

uint32_t stream_slab_count(uint32_t n, uint32_t num_ctas, uint32_t min_rows) {
    if (min_rows < 1) min_rows = 1;
    uint32_t c = std::min<uint32_t>(num_ctas, (n + min_rows - 1) / min_rows);
    return c < 1 ? 1 : c;
}

template <typename Low>
bool DevSweep::stream_order(const Sweep<Low>& sweep, StreamOrder& o) const {
    if (!streamed() || sweep.n != n) return false;
    Sweep<Low> ps;
    PairMap pm;
    if (paired) pair_sweep<Low>(sweep, ps, pm);
    const Sweep<Low>& s = paired ? ps : sweep;
    StreamLayout L;
    FlowLayout F;
    std::string why;
    if (layout == LAYOUT_FLOW) {
        if (!flow_layout<Low>(s, slab_ranges<Low>(s, str_ctas_req), str_slots, F, &o))
            throw Error(PRISM_ERR_CUDA, "dataflow layout could not be rebuilt");
    } else if (!stream_layout<Low>(s, slab_ranges<Low>(s, str_ctas_req), kNoSlot, str_slot_bytes, L, &why, &o, nullptr,
                            str_round_cap))
        throw Error(PRISM_ERR_CUDA, "streamed layout could not be rebuilt: " + why);
    if (paired) {
        o.mptr = std::move(pm.ptr);
        o.mdep = std::move(pm.dep);
        o.mcoef = std::move(pm.coef);
    }
    return true;
}
template bool DevSweep::stream_order<double>(const Sweep<double>&, StreamOrder&) const;
template bool DevSweep::stream_order<float>(const Sweep<float>&, StreamOrder&) const;

template <typename Low>
void stream_sweep_run(int device, const Sweep<Low>& s, bool acc32, uint32_t num_ctas, const double* in,
                      double* out) {
    Handle h;
    init_device_info(h.info, device);
    h.info.sms = (int)std::min<uint32_t>(num_ctas, (uint32_t)h.info.sms);
    h.info.stream_min_rows = 32;
    PRISM_CUDA(cudaStreamCreateWithFlags(&h.stream, cudaStreamNonBlocking));
    h.own_stream = true;
    h.status.alloc(1);
    PRISM_CUDA(cudaMemsetAsync(h.status.get(), 0, sizeof(int), h.stream));
    DevSweep d;
    d.acc32 = acc32 && std::is_same<Low, float>::value;
    if (!d.upload(s, h.info, LAYOUT_STREAM, h.stream))
        throw Error(PRISM_ERR_UNSUPPORTED, "the sweep does not fit the streamed layout");
    DevBuf<double> din(s.n), dout(s.n);
    din.upload(in, s.n, h.stream);
    launch_sweep(h, h.stream, d, din.get(), dout.get());
    PRISM_CUDA(cudaMemcpyAsync(out, dout.get(), s.n * sizeof(double), cudaMemcpyDeviceToHost, h.stream));
    h.check_status();
}
template void stream_sweep_run<double>(int, const Sweep<double>&, bool, uint32_t, const double*, double*);
template void stream_sweep_run<float>(int, const Sweep<float>&, bool, uint32_t, const double*, double*);

// ============================================================================
// Bounded-wait self test of the dataflow sweep: four slabs of 128 rows whose first one keeps the
// value of its last row to itself, so the second waits for an exchange entry that is never
// written.  The wait runs out after wait_ns, every CTA leaves, and status 6 is raised; with the
// header put right the same layout, exchange entries and all, then sweeps to the replay's bits.
// ============================================================================
void selftest_flow_timeout(int device, uint32_t cols, unsigned long long wait_ns, int* device_status) {
    Handle h;
    init_device_info(h.info, device);
    h.info.wait_ns = wait_ns;
    PRISM_CUDA(cudaStreamCreateWithFlags(&h.stream, cudaStreamNonBlocking));
    h.own_stream = true;
    h.status.alloc(1);
    PRISM_CUDA(cudaMemsetAsync(h.status.get(), 0, sizeof(int), h.stream));
    // row r reads rows r - 1 and r - 37
    const uint32_t n = 512, slab = 128, k = std::max(cols, 1u);
    std::vector<uint32_t> rp{0}, ci;
    std::vector<double> val;
    for (uint32_t r = 0; r < n; ++r) {
        if (r >= 37) ci.push_back(r - 37), val.push_back(0.25);
        if (r >= 1) ci.push_back(r - 1), val.push_back(-0.5);
        rp.push_back((uint32_t)ci.size());
    }
    Sweep<double> s;
    build_sweep<double>(n, rp, ci, val, nullptr, SWEEP_NONE, true, s);
    StreamPlan P = plan_flow<double>(s, h.info, false, slab, cols);
    if (!P.ok || P.F.slabs != n / slab) throw Error(PRISM_ERR_CUDA, "four slabs expected");
    FlowLayout good;
    flow_layout<double>(s, slab_ranges<double>(s, P.ctas_req), P.F.slots, good, nullptr, nullptr, P.F.entries);
    bool found = false;
    for (size_t i = 0; i < P.F.hdr.size(); i += 4)
        if (P.F.hdr[i] == slab - 1) {
            found = P.F.hdr[i + 1] != kFlowNone;
            P.F.hdr[i + 1] = kFlowNone;
        }
    if (!found) throw Error(PRISM_ERR_CUDA, "a published row expected");
    DevSweep d;
    d.commit_stream(std::move(P), h.stream);
    d.block_workspace(k, h.stream);
    std::vector<double> in((size_t)n * k), got((size_t)n * k), one(n), want(n);
    for (size_t i = 0; i < in.size(); ++i) in[i] = 1.0 + (double)(i % 11) * 0.125;
    DevBuf<double> din(in.size()), dout(in.size());
    din.upload(in.data(), in.size(), h.stream);
    auto sweep = [&]() {
        if (cols) launch_flow_block(h, h.stream, d, k, din.get(), dout.get());
        else launch_sweep(h, h.stream, d, din.get(), dout.get());
        h.check_status();
    };
    *device_status = 0;
    try {
        sweep();
    } catch (const Error& e) {
        if (e.status == PRISM_ERR_CUDA) throw;
        *device_status = e.status;
    }
    d.fl_hdr.upload(good.hdr.data(), good.hdr.size(), h.stream);
    sweep();
    PRISM_CUDA(cudaMemcpy(got.data(), dout.get(), got.size() * sizeof(double), cudaMemcpyDeviceToHost));
    for (uint32_t c = 0; c < k; ++c) {
        for (uint32_t r = 0; r < n; ++r) one[r] = in[(size_t)r * k + c];
        const std::string why = flow_layout_replay<double>(s, good, false, one.data(), want.data());
        if (!why.empty()) throw Error(PRISM_ERR_CUDA, "dataflow layout: " + why);
        for (uint32_t r = 0; r < n; ++r)
            if (got[(size_t)r * k + c] != want[r])
                throw Error(PRISM_ERR_CUDA, "the sweep after the one that was given up differs in row " + std::to_string(r));
    }
}

// Sweep-kernel autotuner: uploads the sweep in one device layout after another
// (level order for k_sweep, slabs for k_sweep_slab, dataflow slabs for k_sweep_flow
// or, where they do not fit, rounds for k_sweep_stream), times a few launches of
// each, output marking included, on a fixed right-hand side with CUDA events, and
// keeps the fastest.  Which kernel wins depends on how many rows a wavefront holds
// and how far dependencies reach.
//
// Single-precision arithmetic: only the streamed kernels have it (the other layouts,
// where no streamed one fits, compute in double).  Slab sizes are climbed from one to its
// neighbours, the sweep's time having one minimum over them (kFlowSlabRows), and the paired
// sweep is laid out for its own minimum only where at the unpaired sweep's best size it is within
// a quarter of it.  At most two layouts are in host memory, and the paired sweep, which is worked
// out while the unpaired ones are timed (all sizes, paired and not, laid out at once held eight
// layouts, 450 MB each for the level-0 sweep of 128^3 with float values, and four paired sweeps).
template <typename Low>
void tune_sweep(Handle& h, DevSweep& d, const Sweep<Low>& s, bool acc32, bool pair) {
    const int mode = h.info.sweep_kernel;
    const bool a32 = acc32 && std::is_same<Low, float>::value;
    // Pairing keeps the arithmetic's precision class only where the derived coefficients are
    // stored in the arithmetic's own type: double values (FP64) or float values with float
    // arithmetic; float values with double arithmetic (<float,double>) stay unpaired.
    const bool pp = pair && h.info.stream_pair != 0 && (a32 || std::is_same<Low, double>::value);
    const bool only_paired = pp && h.info.stream_pair == 2;  // paired where it fits
    const bool any = mode == 0 && !a32 && !only_paired;      // every layout is a candidate
    auto untimed = [&](int layout) {
        DevSweep t;
        t.acc32 = a32;
        t.upload(s, h.info, layout, h.stream);
        d = std::move(t);
    };
    if (s.n == 0 || ((mode == 1 || mode == 2) && !a32 && !only_paired)) {
        untimed(s.n != 0 && mode == 2 ? LAYOUT_SLAB : LAYOUT_LEVEL);
        return;
    }
    struct Paired {
        Sweep<Low> s;
        PairMap m;
    };
    std::future<Paired> pairing;
    if (pp)
        pairing = std::async([&s] {
            Paired p;
            pair_sweep<Low>(s, p.s, p.m);
            return p;
        });
    DevBuf<double> in(s.n), out(s.n);
    std::vector<double> rhs(s.n);
    for (uint32_t i = 0; i < s.n; ++i) rhs[i] = 1.0 + (double)(i % 7) * 0.125;
    in.upload(rhs.data(), s.n, h.stream);
    struct Events {
        cudaEvent_t e[2] = {};
        ~Events() {
            for (cudaEvent_t x : e)
                if (x) cudaEventDestroy(x);
        }
    } ev;
    for (cudaEvent_t& x : ev.e) PRISM_CUDA(cudaEventCreate(&x));
    constexpr float kNever = std::numeric_limits<float>::infinity();
    float best = kNever;
    DevSweep kept;  // the fastest candidate so far, kept uploaded
    auto time = [&](DevSweep&& t) {
        float least = kNever;
        for (int it = 0; it < 4; ++it) {
            PRISM_CUDA(cudaEventRecord(ev.e[0], h.stream));
            launch_sweep_prepare(h, h.stream, t, in.get(), out.get());
            launch_sweep_kernel(h, h.stream, t, in.get(), out.get());
            PRISM_CUDA(cudaEventRecord(ev.e[1], h.stream));
            PRISM_CUDA(cudaEventSynchronize(ev.e[1]));
            float ms = 0.f;
            PRISM_CUDA(cudaEventElapsedTime(&ms, ev.e[0], ev.e[1]));
            if (it > 0) least = std::min(least, ms);  // first launch is a warm-up
        }
        h.check_status();
        if (least < best) {
            best = least;
            kept = std::move(t);
        }
        return least;
    };
    auto plain = [&](int layout) {
        DevSweep t;
        t.acc32 = a32;
        if (t.upload(s, h.info, layout, h.stream)) time(std::move(t));
    };
    const bool rounds = mode == 4;
    // small sweeps: the smallest size (64^2: 8% faster than the others)
    const bool climbs = !rounds && !h.info.flow_rows && s.n > 32 * kFlowSlabRows[0];
    const uint32_t only_rows = h.info.flow_rows ? h.info.flow_rows : kFlowSlabRows[0];
    // the unpaired layouts that are needed in any case: on the host while the one before is timed
    int size = 1;
    uint32_t ahead_rows = 0;
    std::future<StreamPlan> ahead;
    auto lay_ahead = [&](uint32_t rows) {
        ahead_rows = rows;
        ahead = std::async([&s, &h, a32, rows] { return plan_flow<Low>(s, h.info, a32, rows); });
    };
    // the streamed layouts of sw, starting from kFlowSlabRows[at]; returns the best size
    auto streamed = [&](const Sweep<Low>& sw, const PairMap* pm, int at) {
        auto upload = [&](StreamPlan&& P) {
            P.pm = pm;
            DevSweep t;
            t.acc32 = a32;
            t.commit_stream(std::move(P), h.stream);
            return time(std::move(t));
        };
        bool first = true;
        auto flow = [&](uint32_t rows) {
            StreamPlan P;
            if (!rounds) P = rows == ahead_rows ? ahead.get() : plan_flow<Low>(sw, h.info, a32, rows);
            ahead_rows = 0;
            if (first && !pm && climbs) lay_ahead(kFlowSlabRows[at - 1]);
            if (!P.ok && first) P = plan_stream<Low>(sw, h.info, a32);
            // slabs that had to be split are those of a smaller size
            const bool split = P.ok && P.flow && P.ctas_req > (s.n + rows - 1) / rows;
            if (!P.ok || (split && !first)) return kNever;
            first = false;
            return upload(std::move(P));
        };
        if (!climbs) {
            flow(only_rows);
            return 0;
        }
        const float unpaired = best;
        float here = flow(kFlowSlabRows[at]);
        if (pm && here > 1.25f * unpaired) return at;
        for (int step : {-1, 1}) {
            const int from = at;
            while (at + step >= 0 && at + step < kFlowSizes) {
                const float t = flow(kFlowSlabRows[at + step]);
                if (t >= here) break;
                here = t;
                at += step;
            }
            if (at != from) break;
        }
        return at;
    };
    if (!only_paired && !rounds) lay_ahead(climbs ? kFlowSlabRows[size] : only_rows);
    if (any) {
        plain(LAYOUT_LEVEL);
        plain(LAYOUT_SLAB);
    }
    if (!only_paired) size = streamed(s, nullptr, size);
    if (pairing.valid()) {
        const Paired p = pairing.get();
        streamed(p.s, &p.m, size);
    }
    if (best == kNever) {  // nothing fitted (streamed layouts only): level order, double arithmetic
        untimed(LAYOUT_LEVEL);
        return;
    }
    d = std::move(kept);
    d.tuned_ms = best;
}
template void tune_sweep<double>(Handle&, DevSweep&, const Sweep<double>&, bool, bool);
template void tune_sweep<float>(Handle&, DevSweep&, const Sweep<float>&, bool, bool);

namespace {
std::atomic<uint64_t> g_precond_uid{0};
}
Precond::Precond() : uid(++g_precond_uid) {}
void Precond::renew_uid() { uid = ++g_precond_uid; }

TriangularPrecond::TriangularPrecond(Handle& h, std::shared_ptr<const HostFactor> f) : h_(h), f_(std::move(f)) {
    // the streamed kernel may run the sweeps paired (refactor() tunes them again unpaired)
    if (f_->fp32) {
        tune_sweep(h_, lower_, f_->lower32, f_->apply32, true);
        tune_sweep(h_, upper_, f_->upper32, f_->apply32, true);
    } else {
        tune_sweep(h_, lower_, f_->lower64, false, true);
        tune_sweep(h_, upper_, f_->upper64, false, true);
    }
    tmp_.alloc(h_.A.n);  // here rather than at the first apply, which may be under graph capture
}

void TriangularPrecond::apply(cudaStream_t st, const double* in, double* out) {
    const uint32_t n = h_.A.n;
    if (tmp_.size() < n) tmp_.alloc(n);
    if (!lower_.self_filling()) launch_fill(st, h_, n, tmp_.get());
    if (in != out && !upper_.self_filling()) launch_fill(st, h_, n, out);
    launch_sweep(h_, st, lower_, in, tmp_.get());
    if (in == out && !upper_.self_filling()) launch_fill(st, h_, n, out);
    launch_sweep(h_, st, upper_, tmp_.get(), out);
}

bool TriangularPrecond::run_sweep(cudaStream_t st, int sweep, const double* in, double* out, int prepare) {
    const DevSweep& s = sweep == 0 ? lower_ : upper_;
    if (prepare != 0) launch_sweep_prepare(h_, st, s, in, out);
    if (prepare != 2) launch_sweep_kernel(h_, st, s, in, out);
    return true;
}

bool TriangularPrecond::sweep_info(int sweep, uint32_t* n, uint64_t* nnz, uint32_t* vbytes, uint32_t* levels,
                                   uint32_t* kernel) const {
    const DevSweep& s = sweep == 0 ? lower_ : upper_;
    if (kernel) *kernel = s.kernel_id();
    if (n) *n = s.n;
    if (nnz) *nnz = s.entries();
    if (vbytes) *vbytes = s.fp32 ? 4 : 8;
    if (levels) *levels = s.num_levels;
    return true;
}

bool TriangularPrecond::sweep_order(int sweep, StreamOrder& o) const {
    const DevSweep& s = sweep == 0 ? lower_ : upper_;
    if (f_->fp32) return s.stream_order<float>(sweep == 0 ? f_->lower32 : f_->upper32, o);
    return s.stream_order<double>(sweep == 0 ? f_->lower64 : f_->upper64, o);
}

int export_host_factor(const HostFactor& f, int which, uint32_t* n, uint64_t* nnz, uint32_t* rowptr, uint32_t* col,
                       double* val, double* diag) {
    if (which != 0 && !(which == 1 && f.kind == PRISM_PRECOND_ILUT)) return PRISM_ERR_ARG;
    const CsrT<double>& m = which == 0 ? f.f0 : f.f1;
    if (n) *n = m.n;
    if (nnz) *nnz = m.nnz();
    if (rowptr) std::memcpy(rowptr, m.rowptr.data(), m.rowptr.size() * sizeof(uint32_t));
    if (col) std::memcpy(col, m.col.data(), m.col.size() * sizeof(uint32_t));
    if (val) std::memcpy(val, m.val.data(), m.val.size() * sizeof(double));
    if (diag && !f.diag.empty()) std::memcpy(diag, f.diag.data(), f.diag.size() * sizeof(double));
    return 0;
}

int TriangularPrecond::export_factor(int which, uint32_t* n, uint64_t* nnz, uint32_t* rowptr, uint32_t* col,
                                     double* val, double* diag) const {
    if (rf_) return export_refactored(which, n, nnz, rowptr, col, val, diag);
    return export_host_factor(*f_, which, n, nnz, rowptr, col, val, diag);
}

// ============================================================================
// Flexible / normal preconditioned CG  (CG<double>::solve, CG.cpp:34-83)
//
// Same recurrence, same stopping test on the recursive residual, same
// iteration count convention (numIter = m + 1).  The reference recomputes
// v = A d at the top of every iteration (CG.cpp:68) although d has not
// changed since v = A d at the end of the previous one (CG.cpp:75); the
// SpMV and the d.v reduction are deterministic here, so that product and its
// d.v are reused instead of recomputed: one SpMV per iteration, not two.
// ============================================================================
void fcg_solve(Handle& h, const prism_solve_opts& o, const double* b, double* x, prism_solve_stats* st) {
    const uint32_t n = h.A.n;
    h.ensure_workspace();
    cudaStream_t s = h.stream;
    const bool flexible = o.solver == PRISM_SOLVER_FCG;
    Precond* P = h.P.get();
    double* r = h.r.get();
    double* w = h.w.get();
    double* d = h.d.get();
    double* v = h.v.get();
    double* y = h.y.get();
    double* sc = h.red.scalars.get();
    const int vg = vec_grid(h, n);
    uint32_t applies = 0, spmvs = 0, syncs = 0;

    PRISM_CUDA(cudaEventRecord(h.ev0, s));
    // r = b - A x ; Σ b²
    h.spmv(x, y);
    ++spmvs;
    k_residual<<<vg, kBlock, 0, s>>>(n, b, y, r, h.red.slot(SC_BB));
    PRISM_LAUNCHED();
    // w = M^{-1} r ; d = w
    if (P) { P->apply(s, r, w); ++applies; }
    else PRISM_CUDA(cudaMemcpyAsync(w, r, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    PRISM_CUDA(cudaMemcpyAsync(d, w, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    // v = A d ; Σ v·d , Σ d·r
    h.spmv(d, v, 2, d, r, SC_DV);
    ++spmvs;
    // x += a d ; r -= a v ; Σ r²
    k_fcg_step<<<vg, kBlock, 0, s>>>(n, x, r, d, v, sc + SC_DR, sc + SC_DV, h.red.slot(SC_RR));
    PRISM_LAUNCHED();

    PRISM_CUDA(cudaMemcpyAsync(h.pinned, sc, kNumScalars * sizeof(double), cudaMemcpyDeviceToHost, s));
    h.check_status();
    ++syncs;
    const double norm_b = std::sqrt(h.pinned[SC_BB]);
    uint32_t m = o.max_iter;
    double norm = -1.0;
    bool converged = false;
    for (uint32_t i = 1; i < o.max_iter; ++i) {
        if (i > 1) {
            PRISM_CUDA(cudaMemcpyAsync(h.pinned + SC_RR, sc + SC_RR, sizeof(double), cudaMemcpyDeviceToHost, s));
            h.check_status();
            ++syncs;
        }
        norm = std::sqrt(h.pinned[SC_RR]) / norm_b;
        if (!std::isfinite(norm)) throw Error(PRISM_ERR_NONFINITE, "non-finite residual norm in CG iteration " + std::to_string(i));
        if (norm < o.tol) {
            converged = true;
            m = i;
            break;
        }
        if (flexible && P) { P->apply(s, r, w); ++applies; }
        else PRISM_CUDA(cudaMemcpyAsync(w, r, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
        // v still holds A d and sc[DV] its d.v: c = (w.v)/(d.v); d = w - c d; Σ d·r
        k_dot<<<vg, kBlock, 0, s>>>(n, w, v, h.red.slot(SC_WV));
        PRISM_LAUNCHED();
        k_fcg_direction<<<vg, kBlock, 0, s>>>(n, w, d, r, sc + SC_WV, sc + SC_DV, h.red.slot(SC_DR2));
        PRISM_LAUNCHED();
        // v = A d ; Σ v·d
        h.spmv(d, v, 1, d, nullptr, SC_DV);
        ++spmvs;
        k_fcg_step<<<vg, kBlock, 0, s>>>(n, x, r, d, v, sc + SC_DR2, sc + SC_DV, h.red.slot(SC_RR));
        PRISM_LAUNCHED();
    }
    // true FP64 residual
    h.spmv(x, y);
    ++spmvs;
    k_residual<<<vg, kBlock, 0, s>>>(n, b, y, nullptr, h.red.slot(SC_BB));
    PRISM_LAUNCHED();
    PRISM_CUDA(cudaEventRecord(h.ev1, s));
    PRISM_CUDA(cudaMemcpyAsync(h.pinned, sc, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    h.check_status();
    ++syncs;
    float ms = 0.f;
    PRISM_CUDA(cudaEventElapsedTime(&ms, h.ev0, h.ev1));
    if (st) {
        st->num_iter = (int32_t)(m + 1);
        st->converged = converged;
        st->final_error = norm;
        st->true_rel_residual = std::sqrt(h.pinned[SC_RES]) / std::sqrt(h.pinned[SC_BB]);
        st->precond_applies = applies;
        st->spmv_count = spmvs;
        st->device_ms = ms;
        st->host_syncs = syncs;
        st->graph_nodes = 0;
    }
}

double forward_error(Handle& h, const double* x, const double* xref) {
    const uint32_t n = h.A.n;
    if (!n) return 0.0;
    // { Σ xref_i^2, Σ (xref_i - x_i)^2 } into the two scratch scalars
    k_residual<<<vec_grid(h, n), kBlock, 0, h.stream>>>(n, xref, x, nullptr, h.red.slot(SC_TMP));
    PRISM_LAUNCHED();
    double v[2] = {0.0, 0.0};
    PRISM_CUDA(cudaMemcpyAsync(v, h.red.scalars.get() + SC_TMP, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                               h.stream));
    PRISM_CUDA(cudaStreamSynchronize(h.stream));
    return v[0] > 0.0 ? std::sqrt(v[1]) / std::sqrt(v[0]) : std::sqrt(v[1]);
}

}  // namespace prism
