// A batch of independent systems solved together: the handle's matrix is block
// diagonal, rows [seg_ptr[s], seg_ptr[s+1]) forming system s, and so is any
// incomplete factorisation of it (an ICT / ILDLT / ILUT of a block-diagonal
// matrix eliminates each block on its own), so one SpMV and one pair of
// triangular sweeps serve every system at once -- the sweep kernels' slabs
// follow the block boundaries.  Each system runs the recurrence of
// CG<double>::solve (CG.cpp:34-83) on its own scalars: the Krylov reductions
// are per system (fixed chunks in a fixed order, so repeated solves give
// identical bits), a system that has converged stops changing,
// and stats[s] reports exactly what a solve of system s alone reports.
#include <cmath>
#include <cstring>

#include "../../include/prism_solve.h"
#include "kernels.cuh"
#include "solve.cuh"

namespace prism {

namespace {

// Per-system scalars, each an array of nseg doubles.
enum SegScalar : int { SG_BB = 0, SG_RES, SG_RR, SG_WV, SG_DV, SG_DR, SG_DR2, kSegScalars };

// The systems' rows in chunks of at most kSegChunk: a block takes a chunk, the last block of a
// system adds up its partial sums in chunk order.  A block a system left 100 SMs idle on 48
// systems of up to 25,600 rows: 35 to 56 us a kernel.
constexpr uint32_t kSegChunk = 4096;
struct SegTable {
    uint32_t chunks;
    const uint32_t* lo;      // chunks + 1: chunk c is the rows [lo[c], lo[c + 1])
    const uint32_t* seg;     // chunk -> system
    const uint32_t* first;   // system -> its first chunk, and the end
    double* partial;         // 2 per chunk
    unsigned* ticket;        // per system, 0 between launches
};

template <int NV>
__device__ __forceinline__ void seg_store(double (&v)[NV], double* const (&out)[NV], const SegTable& T, uint32_t c) {
    __shared__ double smem[NV * 32];
    __shared__ bool last;
    const uint32_t s = __ldg(T.seg + c), c0 = __ldg(T.first + s), c1 = __ldg(T.first + s + 1);
    block_sum<NV>(v, smem);
    if (c1 - c0 > 1) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int q = 0; q < NV; ++q) T.partial[2 * (size_t)c + q] = v[q];
            __threadfence();
            last = atomicAdd(T.ticket + s, 1u) == c1 - c0 - 1;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = 0.0;
        for (uint32_t i = c0 + threadIdx.x; i < c1; i += blockDim.x) {
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] += __ldcg(T.partial + 2 * (size_t)i + q);
        }
        block_sum<NV>(v, smem);
        if (threadIdx.x == 0) T.ticket[s] = 0u;
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) out[q][s] = v[q];
    }
}

// r = b - y (r may be null); bb[s] = Σ b², res[s] = Σ (b - y)²
template <int B>
__global__ void __launch_bounds__(B) k_seg_residual(const SegTable T, const double* __restrict__ b,
                                                    const double* __restrict__ y, double* __restrict__ r,
                                                    double* bb, double* res) {
    for (uint32_t c = blockIdx.x; c < T.chunks; c += gridDim.x) {
        double v[2] = {0.0, 0.0};
#pragma unroll 4
        for (uint32_t i = T.lo[c] + threadIdx.x; i < T.lo[c + 1]; i += B) {
            const double bi = b[i], ri = bi - y[i];
            if (r) r[i] = ri;
            v[0] += bi * bi;
            v[1] += ri * ri;
        }
        double* const out[2] = {bb, res};
        seg_store<2>(v, out, T, c);
    }
}

// out[s] = Σ a b over the system's rows
template <int B>
__global__ void __launch_bounds__(B) k_seg_dot(const SegTable T, const double* __restrict__ a,
                                               const double* __restrict__ b, double* out) {
    for (uint32_t c = blockIdx.x; c < T.chunks; c += gridDim.x) {
        double v[1] = {0.0};
#pragma unroll 4
        for (uint32_t i = T.lo[c] + threadIdx.x; i < T.lo[c + 1]; i += B) v[0] += a[i] * b[i];
        double* const o[1] = {out};
        seg_store<1>(v, o, T, c);
    }
}

// vd[s] = Σ v d, dr[s] = Σ d r
template <int B>
__global__ void __launch_bounds__(B) k_seg_dot2(const SegTable T, const double* __restrict__ v,
                                                const double* __restrict__ d, const double* __restrict__ r,
                                                double* vd, double* dr) {
    for (uint32_t c = blockIdx.x; c < T.chunks; c += gridDim.x) {
        double acc[2] = {0.0, 0.0};
#pragma unroll 4
        for (uint32_t i = T.lo[c] + threadIdx.x; i < T.lo[c + 1]; i += B) {
            acc[0] += v[i] * d[i];
            acc[1] += d[i] * r[i];
        }
        double* const out[2] = {vd, dr};
        seg_store<2>(acc, out, T, c);
    }
}

// active systems: c = (w.v)/(d.v); d = w - c d.  dr[s] = Σ d r (frozen systems keep d)
template <int B>
__global__ void __launch_bounds__(B) k_seg_direction(const SegTable T, const double* __restrict__ w,
                                                     double* __restrict__ d, const double* __restrict__ r,
                                                     const double* __restrict__ wv,
                                                     const double* __restrict__ dv,
                                                     const int* __restrict__ active, double* dr) {
    for (uint32_t k = blockIdx.x; k < T.chunks; k += gridDim.x) {
        const uint32_t s = __ldg(T.seg + k);
        const bool on = active[s] != 0 && dv[s] != 0.0;  // dv = 0: a zero right-hand side, nothing to do
        const double c = on ? wv[s] / dv[s] : 0.0;
        double v[1] = {0.0};
#pragma unroll 4
        for (uint32_t i = T.lo[k] + threadIdx.x; i < T.lo[k + 1]; i += B) {
            double di = d[i];
            if (on) {
                di = w[i] - c * di;
                d[i] = di;
            }
            v[0] += di * r[i];
        }
        double* const o[1] = {dr};
        seg_store<1>(v, o, T, k);
    }
}

// active systems: a = (d.r)/(d.v); x += a d; r -= a v.  rr[s] = Σ r²
template <int B>
__global__ void __launch_bounds__(B) k_seg_step(const SegTable T, double* __restrict__ x,
                                                double* __restrict__ r, const double* __restrict__ d,
                                                const double* __restrict__ v, const double* __restrict__ dr,
                                                const double* __restrict__ dv, const int* __restrict__ active,
                                                double* rr) {
    for (uint32_t c = blockIdx.x; c < T.chunks; c += gridDim.x) {
        const uint32_t s = __ldg(T.seg + c);
        const bool on = active[s] != 0 && dv[s] != 0.0;
        const double a = on ? dr[s] / dv[s] : 0.0;
        double acc[1] = {0.0};
#pragma unroll 4
        for (uint32_t i = T.lo[c] + threadIdx.x; i < T.lo[c + 1]; i += B) {
            double ri = r[i];
            if (on) {
                x[i] = x[i] + a * d[i];
                ri = ri - a * v[i];
                r[i] = ri;
            }
            acc[0] += ri * ri;
        }
        double* const o[1] = {rr};
        seg_store<1>(acc, o, T, c);
    }
}

// The kernels for blocks of `threads` threads.
struct SegKernels {
    int threads;
    decltype(&k_seg_residual<32>) residual;
    decltype(&k_seg_dot<32>) dot;
    decltype(&k_seg_dot2<32>) dot2;
    decltype(&k_seg_direction<32>) direction;
    decltype(&k_seg_step<32>) step;
};
template <int B>
SegKernels seg_kernels_of() {
    return {B, k_seg_residual<B>, k_seg_dot<B>, k_seg_dot2<B>, k_seg_direction<B>, k_seg_step<B>};
}
// By the rows of a chunk: as many blocks as fill the SMs go over small systems, a few rows a thread
// (Krylov loop without preconditioner, 12 iterations, us: 20,000 systems of 16 rows 6,340 with 512
// threads, 4,300 now; 4,096 of 64 rows 1,950, 1,580; 2,000 of 256 rows 1,370, 1,200).
SegKernels seg_kernels(uint32_t rows) {
    if (rows <= 64) return seg_kernels_of<32>();
    if (rows <= 256) return seg_kernels_of<64>();
    return rows <= 1024 ? seg_kernels_of<256>() : seg_kernels_of<512>();
}

}  // namespace

struct SegWork {
    std::vector<uint32_t> seg;   // the segment table the device copy holds
    uint32_t chunks = 0;
    DevBuf<uint32_t> lo, of, first;  // SegTable
    DevBuf<double> partial;
    DevBuf<unsigned> ticket;
    DevBuf<double> sc;           // kSegScalars * nseg
    DevBuf<int> active;
    std::vector<double> host;
};

void seg_release(SegWork* w) { delete w; }

void segmented_fcg_solve(Handle& h, const prism_solve_opts& o, uint32_t nseg, const uint32_t* seg_ptr,
                         const double* b, double* x, prism_solve_stats* st) {
    const uint32_t n = h.A.n;
    if (nseg == 0) throw Error(PRISM_ERR_ARG, "no systems");
    if (seg_ptr[0] != 0 || seg_ptr[nseg] != n) throw Error(PRISM_ERR_ARG, "system offsets must run from 0 to n");
    for (uint32_t s = 0; s < nseg; ++s)
        if (seg_ptr[s + 1] <= seg_ptr[s]) throw Error(PRISM_ERR_ARG, "a system without rows");
    if (!h.seg || h.seg->seg.size() != (size_t)nseg + 1 ||
        std::memcmp(h.seg->seg.data(), seg_ptr, ((size_t)nseg + 1) * sizeof(uint32_t)) != 0) {
        // a row may only couple to rows of its own system
        const CsrHost& A = h.A_host;
        for (uint32_t s = 0; s < nseg; ++s)
            for (uint32_t i = seg_ptr[s]; i < seg_ptr[s + 1]; ++i)
                for (uint32_t k = A.rowptr[i]; k < A.rowptr[i + 1]; ++k)
                    if (A.col[k] < seg_ptr[s] || A.col[k] >= seg_ptr[s + 1])
                        throw Error(PRISM_ERR_ARG, "row " + std::to_string(i) + " couples system " +
                                                       std::to_string(s) + " to another one");
        h.seg.reset();
        std::unique_ptr<SegWork, void (*)(SegWork*)> w(new SegWork(), seg_release);
        w->seg.assign(seg_ptr, seg_ptr + nseg + 1);
        std::vector<uint32_t> lo, of, first;
        for (uint32_t s = 0; s < nseg; ++s) {
            first.push_back((uint32_t)lo.size());
            for (uint64_t r = seg_ptr[s]; r < seg_ptr[s + 1]; r += kSegChunk) {
                lo.push_back((uint32_t)r);
                of.push_back(s);
            }
        }
        first.push_back((uint32_t)lo.size());
        w->chunks = (uint32_t)lo.size();
        lo.push_back(n);
        w->lo.upload(lo.data(), lo.size(), h.stream);
        w->of.upload(of.data(), of.size(), h.stream);
        w->first.upload(first.data(), first.size(), h.stream);
        w->partial.alloc(2 * (size_t)w->chunks);
        w->ticket.alloc(nseg);
        PRISM_CUDA(cudaMemsetAsync(w->ticket.get(), 0, nseg * sizeof(unsigned), h.stream));
        PRISM_CUDA(cudaStreamSynchronize(h.stream));  // the host arrays end here
        w->sc.alloc((size_t)kSegScalars * nseg);
        w->active.alloc(nseg);
        w->host.assign((size_t)kSegScalars * nseg, 0.0);
        h.seg = std::move(w);  // whole
    }
    SegWork& w = *h.seg;
    h.ensure_workspace();
    cudaStream_t s = h.stream;
    const bool flexible = o.solver == PRISM_SOLVER_FCG;
    Precond* P = h.P.get();
    double *r = h.r.get(), *wv = h.w.get(), *d = h.d.get(), *v = h.v.get(), *y = h.y.get();
    const SegTable T{w.chunks, w.lo.get(), w.of.get(), w.first.get(), w.partial.get(), w.ticket.get()};
    auto sc = [&](int k) { return w.sc.get() + (size_t)k * nseg; };
    const SegKernels K = seg_kernels(n / w.chunks);
    const int per_sm = 2048 / K.threads;
    const int grid = (int)std::min<uint32_t>(w.chunks, (uint32_t)(h.info.sms * per_sm));
    uint32_t applies = 0, spmvs = 0;
    std::vector<int> act(nseg, 1);
    PRISM_CUDA(cudaMemcpyAsync(w.active.get(), act.data(), nseg * sizeof(int), cudaMemcpyHostToDevice, s));

    PRISM_CUDA(cudaEventRecord(h.ev0, s));
    h.spmv(x, y);
    ++spmvs;
    K.residual<<<grid, K.threads, 0, s>>>(T, b, y, r, sc(SG_BB), sc(SG_RES));
    PRISM_LAUNCHED();
    if (P) { P->apply(s, r, wv); ++applies; }
    else PRISM_CUDA(cudaMemcpyAsync(wv, r, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    PRISM_CUDA(cudaMemcpyAsync(d, wv, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    h.spmv(d, v);
    ++spmvs;
    K.dot2<<<grid, K.threads, 0, s>>>(T, v, d, r, sc(SG_DV), sc(SG_DR));
    PRISM_LAUNCHED();
    K.step<<<grid, K.threads, 0, s>>>(T, x, r, d, v, sc(SG_DR), sc(SG_DV), w.active.get(), sc(SG_RR));
    PRISM_LAUNCHED();
    PRISM_CUDA(cudaMemcpyAsync(w.host.data(), w.sc.get(), (size_t)kSegScalars * nseg * sizeof(double),
                               cudaMemcpyDeviceToHost, s));
    h.check_status();
    std::vector<double> norm_b(nseg), norm(nseg, 0.0);
    std::vector<uint32_t> m(nseg, o.max_iter);
    std::vector<int> conv(nseg, 0);
    uint32_t remaining = nseg;
    for (uint32_t q = 0; q < nseg; ++q) {
        norm_b[q] = std::sqrt(w.host[(size_t)SG_BB * nseg + q]);
        if (norm_b[q] == 0.0) {  // b = 0: x = 0 solves it; nothing to iterate
            conv[q] = 1;
            m[q] = 0;
            act[q] = 0;
            --remaining;
        }
    }
    for (uint32_t i = 1; i < o.max_iter && remaining > 0; ++i) {
        if (i > 1) {
            PRISM_CUDA(cudaMemcpyAsync(w.host.data() + (size_t)SG_RR * nseg, sc(SG_RR), nseg * sizeof(double),
                                       cudaMemcpyDeviceToHost, s));
            h.check_status();
        }
        bool changed = false;
        for (uint32_t q = 0; q < nseg; ++q) {
            if (!act[q]) continue;
            norm[q] = std::sqrt(w.host[(size_t)SG_RR * nseg + q]) / norm_b[q];
            if (!std::isfinite(norm[q]))
                throw Error(PRISM_ERR_NONFINITE, "non-finite residual norm of system " + std::to_string(q) +
                                                     " in CG iteration " + std::to_string(i));
            if (norm[q] < o.tol) {
                conv[q] = 1;
                m[q] = i;
                act[q] = 0;
                --remaining;
                changed = true;
            }
        }
        if (remaining == 0) break;
        if (changed)
            PRISM_CUDA(cudaMemcpyAsync(w.active.get(), act.data(), nseg * sizeof(int), cudaMemcpyHostToDevice, s));
        if (flexible && P) { P->apply(s, r, wv); ++applies; }
        else PRISM_CUDA(cudaMemcpyAsync(wv, r, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
        K.dot<<<grid, K.threads, 0, s>>>(T, wv, v, sc(SG_WV));
        PRISM_LAUNCHED();
        K.direction<<<grid, K.threads, 0, s>>>(T, wv, d, r, sc(SG_WV), sc(SG_DV), w.active.get(),
                                               sc(SG_DR2));
        PRISM_LAUNCHED();
        h.spmv(d, v);
        ++spmvs;
        K.dot<<<grid, K.threads, 0, s>>>(T, v, d, sc(SG_DV));
        PRISM_LAUNCHED();
        K.step<<<grid, K.threads, 0, s>>>(T, x, r, d, v, sc(SG_DR2), sc(SG_DV), w.active.get(),
                                          sc(SG_RR));
        PRISM_LAUNCHED();
    }
    h.spmv(x, y);
    ++spmvs;
    K.residual<<<grid, K.threads, 0, s>>>(T, b, y, nullptr, sc(SG_BB), sc(SG_RES));
    PRISM_LAUNCHED();
    PRISM_CUDA(cudaEventRecord(h.ev1, s));
    PRISM_CUDA(cudaMemcpyAsync(w.host.data(), w.sc.get(), 2 * (size_t)nseg * sizeof(double), cudaMemcpyDeviceToHost,
                               s));
    h.check_status();
    float ms = 0.f;
    PRISM_CUDA(cudaEventElapsedTime(&ms, h.ev0, h.ev1));
    if (st) {
        for (uint32_t q = 0; q < nseg; ++q) {
            const double bb = w.host[(size_t)SG_BB * nseg + q], res = w.host[(size_t)SG_RES * nseg + q];
            st[q].num_iter = (int32_t)(m[q] + 1);
            st[q].converged = conv[q];
            st[q].final_error = norm[q];
            st[q].true_rel_residual = bb > 0.0 ? std::sqrt(res) / std::sqrt(bb) : 0.0;
            st[q].precond_applies = applies;
            st[q].spmv_count = spmvs;
            st[q].device_ms = ms;
            st[q].forward_error = -1.0;  // no reference solution for block / batch solves
            st[q].host_syncs = 0;  // not counted for block / batch solves
            st[q].graph_nodes = 0;
        }
    }
}

}  // namespace prism
