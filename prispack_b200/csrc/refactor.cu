// Device numeric refactorisation of an IC / ILDLT factor on its own pattern.
//
// The host factorisation (IncompleteCholesky::setup, IncompleteCholesky.cpp:
// 96-246; IncompleteLDLT::setup, IncompleteLDLT.cpp:39-186) is left-looking:
// column j starts from the matrix entries of row j on or below the diagonal,
// subtracts L_ik * L_jk (* D_k) for every finished column k with an entry in
// row j, in the order of its linked lists, drops small entries, and divides by
// the pivot.  Which entries survive depends on the values, but once the
// pattern is fixed, the order of every operation on a kept entry depends only
// on the pattern, and the host records it (RefactorPlan).  k_refactor replays
// it for new matrix values: one warp per column, columns taken in order by
// co-resident warps (cooperative launch), a finished column published with a
// release store of the refactorisation's epoch and awaited with bounded
// acquire polls, the column's accumulators in shared memory, every
// floating-point operation the host's, in the host's order, correctly
// rounded and never contracted.  With the matrix the factor was built from it
// reproduces the host factor bit for bit; with new values it computes the
// incomplete factor of the same pattern.
//
// The factor values then go into every device layout of the preconditioner's
// sweeps through maps built once from the factor's pattern: the level-order and
// slab layouts' value and diagonal arrays, the dataflow layout's chunks and diagonals,
// the rounds' records (coefficients, and each row's diagonal or its reciprocal).
#include <algorithm>
#include <cmath>
#include <memory>

#include "kernels.cuh"
#include "solve.cuh"

namespace prism {

namespace {
constexpr int kRfWarps = kBlock / 32;
// A dependency wait is bounded by 1 s and 20 us for each chunk on the longest chain of columns:
// columns of a full factor wait for one another's whole work (8 us a chunk, 2.1 s for 1,024 of them).
constexpr unsigned long long kRfWaitNs = 1000000000ull, kRfChunkNs = 20000ull;
constexpr uint32_t kRfMaxCol = 1024;                      // longest column a warp holds in shared memory

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

struct RfArgs {
    uint32_t n, max_col, smax, epoch;
    const uint32_t* lt_rowptr;
    const uint32_t* lt_col;
    const uint32_t* a_col;
    const double* a_val;
    const uint32_t* a_ptr;
    const uint32_t* a_pos;
    const uint32_t* up_ptr;
    const uint32_t* up_k;
    const uint32_t* up_start;
    const uint32_t* sched;   // the columns in order of their depth in the dependency graph
    const uint64_t* uo;      // per column: offset of its first update entry in `place`
    const uint16_t* place;   // per update entry: where its product goes in the chunk (kRfPlace)
    const uint64_t* so;      // per column: offset of its first chunk in `seg`
    const uint16_t* seg;     // per chunk: the first product of each slot, and the end
    uint32_t* done;     // per column: the epoch that finished it
    int* status;        // 0, PRISM_ERR_NOT_SPD, PRISM_ERR_ZERO_PIVOT or PRISM_ERR_TIMEOUT
    int* bad_col;       // the first column that raised it
    unsigned long long wait_ns;
};
// An update entry's word: the place of its product, the update's number in the chunk, and
// whether its row is not in the column.
constexpr uint32_t kRfPlace = 1023, kRfUpdateAt = 10, kRfDrop = 0x8000;
static_assert(kRfMaxCol <= kRfPlace + 1, "a chunk's products");

// Per-warp shared memory of k_refactor: the column's accumulators and rows (max_col each), a
// chunk's products and their words (smax each) and its slots' first products (max_col + 1), and
// per update of the chunk its L_jk, D_k and first entry.
__host__ __device__ inline size_t rf_warp_bytes(uint32_t max_col, uint32_t smax) {
    return ((size_t)max_col * (8 + 4) + (size_t)smax * (8 + 2) + 32 * (8 + 8 + 4) + ((size_t)max_col + 1) * 2 + 15) &
           ~(size_t)15;
}

// The chunk of updates from u0 on: the longest prefix of up to 32 updates whose entries fit smax
// (each update alone does: c <= max_col <= smax).  Lane q has update u0 + q's column k, its first
// entry and their number, and the entries before it in the chunk.
struct RfChunk {
    uint32_t k = 0, st = 0, c = 0, off = 0, total = 0;
    int nu = 0;
    __device__ RfChunk(const RfArgs& a, uint32_t u0, uint32_t uend, int lane) {
        const uint32_t u = u0 + lane;
        if (u < uend) {
            k = a.up_k[u];
            st = a.up_start[u];
            c = a.lt_rowptr[k + 1] - st;
        }
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += t;
        }
        nu = __popc(__ballot_sync(0xFFFFFFFFu, u < uend && incl <= a.smax));
        total = __shfl_sync(0xFFFFFFFFu, incl, nu - 1);
        off = incl - c;
    }
};

// The column of each slot's row (slot 0: row j), in increasing order, and binary search.
struct RfCol {
    const uint32_t* rows;
    uint32_t m;
    __device__ int find(uint32_t i) const {
        uint32_t lo = 0, hi = m;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (rows[mid] < i) lo = mid + 1;
            else hi = mid;
        }
        return (lo < m && rows[lo] == i) ? (int)lo : -1;
    }
};

// Once per pattern: where the product of every entry an update brings in (the entries of
// column k from row j down) goes.  A chunk's products are laid out slot after slot, and in the
// order of the updates within one.
__global__ void __launch_bounds__(kBlock) k_rf_places(const RfArgs a, uint16_t* place, uint16_t* seg, int ldlt) {
    extern __shared__ __align__(16) unsigned char rf_smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t* rows = reinterpret_cast<uint32_t*>(rf_smem) + (size_t)wid * 2 * a.max_col;
    uint32_t* cur = rows + a.max_col;
    const uint32_t nwarps = gridDim.x * kRfWarps;
    for (uint32_t j = blockIdx.x * kRfWarps + wid; j < a.n; j += nwarps) {
        const uint32_t b = a.lt_rowptr[j], e = a.lt_rowptr[j + 1];
        const uint32_t m = ldlt ? e - b + 1 : e - b, off0 = ldlt ? b - 1 : b;
        for (uint32_t s = lane; s < m; s += 32) rows[s] = s == 0 ? j : a.lt_col[off0 + s];
        __syncwarp();
        const RfCol col{rows, m};
        uint16_t* f = place + a.uo[j];
        uint16_t* g = seg + a.so[j];
        const uint32_t uend = a.up_ptr[j + 1];
        for (uint32_t u0 = a.up_ptr[j]; u0 < uend;) {
            const RfChunk h(a, u0, uend, lane);
            for (uint32_t s = lane; s < m; s += 32) cur[s] = 0;
            __syncwarp();
            // how many products a slot has (a row appears once per update)
            for (int q = 0; q < h.nu; ++q) {
                const uint32_t st = __shfl_sync(0xFFFFFFFFu, h.st, q), c = __shfl_sync(0xFFFFFFFFu, h.c, q);
                const uint32_t o = __shfl_sync(0xFFFFFFFFu, h.off, q);
                for (uint32_t t = lane; t < c; t += 32) {
                    const int s = col.find(a.lt_col[st + t]);
                    f[o + t] = s < 0 ? (uint16_t)kRfDrop : (uint16_t)s;
                    if (s >= 0) ++cur[s];
                }
                __syncwarp();
            }
            if (lane == 0) {
                uint32_t sum = 0;
                for (uint32_t s = 0; s < m; ++s) {
                    const uint32_t c = cur[s];
                    g[s] = (uint16_t)sum;
                    cur[s] = sum;
                    sum += c;
                }
                g[m] = (uint16_t)sum;
            }
            __syncwarp();
            for (int q = 0; q < h.nu; ++q) {
                const uint32_t c = __shfl_sync(0xFFFFFFFFu, h.c, q), o = __shfl_sync(0xFFFFFFFFu, h.off, q);
                for (uint32_t t = lane; t < c; t += 32) {
                    const uint32_t s = f[o + t];
                    const uint32_t at = s == kRfDrop ? kRfDrop : cur[s]++;
                    f[o + t] = (uint16_t)(at | (uint32_t)q << kRfUpdateAt);
                }
                __syncwarp();
            }
            u0 += h.nu;
            f += h.total;
            g += m + 1;
        }
    }
}

// Column j of the factor, one warp per column, columns taken in the order of `sched`
// (by depth in the dependency graph: a column's updates come from shallower columns, so
// the columns in flight at any time span a few levels of the graph, not a few planes of
// the natural order).  The updates are taken in chunks: first every product
// L_ik L_jk (D_k) of the chunk into shared memory, all loads independent, then a lane a slot
// subtracts the slot's products in the host's update order.
//
// The time is the depth of the graph times what lies between a column's last update and its
// own publication, so everything that the pattern gives (the updates' columns and entries,
// the products' places, the matrix row) is loaded before the wait, L_jk and L_ik are asked for
// together, and the subtractions are one short chain a lane instead of a pass of the warp per
// update.  (Sleeping between polls, or one lane polling for the warp, gains nothing.)  Measured:
// IC 40^3 FP64, 735 levels: 9,985 us with a pass of the warp per update, now 2,950.
template <typename Low, bool LDLT>
__global__ void __launch_bounds__(kBlock) k_refactor(const RfArgs a, Low* __restrict__ lt, double* __restrict__ D) {
    extern __shared__ __align__(16) unsigned char rf_smem[];
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* base = rf_smem + (size_t)wid * rf_warp_bytes(a.max_col, a.smax);
    double* acc = reinterpret_cast<double*>(base);
    double* tv = acc + a.max_col;
    double* cL = tv + a.smax;
    double* cD = cL + 32;
    uint32_t* rows = reinterpret_cast<uint32_t*>(cD + 32);
    uint32_t* cst = rows + a.max_col;
    uint16_t* tw = reinterpret_cast<uint16_t*>(cst + 32);
    uint16_t* sg = tw + a.smax;
    const uint32_t nwarps = gridDim.x * kRfWarps;
    auto fail = [&](int code, uint32_t col) {
        if (atomicCAS(a.status, 0, code) == 0) *a.bad_col = (int)col;
    };
    for (uint32_t w = blockIdx.x * kRfWarps + wid; w < a.n; w += nwarps) {
        const uint32_t j = a.sched[w];
        const uint32_t b = a.lt_rowptr[j], e = a.lt_rowptr[j + 1];
        // IC: the column's first entry is its diagonal; ILDLT stores none (slot 0 is row j anyway)
        const uint32_t m = LDLT ? e - b + 1 : e - b;
        const uint32_t off0 = LDLT ? b - 1 : b;  // entry of slot s is off0 + s (s >= 1)
        for (uint32_t s = lane; s < m; s += 32) {
            rows[s] = s == 0 ? j : a.lt_col[off0 + s];
            acc[s] = 0.0;
        }
        __syncwarp();
        const RfCol col{rows, m};
        // the matrix entries of row j at or below the diagonal, in stored order (duplicates add up)
        const uint32_t qend = a.a_ptr[j + 1];
        for (uint32_t q0 = a.a_ptr[j]; q0 < qend; q0 += 32) {
            int s = -1;
            double v = 0.0;
            if (q0 + lane < qend) {
                const uint32_t p = a.a_pos[q0 + lane];
                s = col.find(a.a_col[p]);
                v = a.a_val[p];
            }
            const int cnt = (int)min(32u, qend - q0);
            for (int i = 0; i < cnt; ++i) {
                const int si = __shfl_sync(kAll, s, i);
                const double vi = __shfl_sync(kAll, v, i);
                if (lane == 0 && si >= 0) acc[si] = __dadd_rn(acc[si], vi);
            }
        }
        __syncwarp();
        bool ok = __all_sync(kAll, ld_relaxed_s32(a.status) == 0);  // the same in every lane
        const uint16_t* f = a.place + a.uo[j];
        const uint16_t* g = a.seg + a.so[j];
        const uint32_t uend = a.up_ptr[j + 1];
        for (uint32_t u0 = a.up_ptr[j]; u0 < uend && ok;) {
            const RfChunk h(a, u0, uend, lane);
            if (lane < h.nu) cst[lane] = h.st - h.off;  // entry t of the chunk: cst[its update] + t
            for (uint32_t t = lane; t < h.total; t += 32) tw[t] = f[t];
            for (uint32_t s = lane; s <= m; s += 32) sg[s] = g[s];
            // wait for the chunk's columns
            bool have = lane >= h.nu || ld_acquire_u32(a.done + h.k) == a.epoch;
            if (!__all_sync(kAll, have)) {
                const unsigned long long t0 = globaltimer_ns();
                unsigned spins = 0;
                do {
                    if (!have) have = ld_acquire_u32(a.done + h.k) == a.epoch;
                    if ((++spins & 15u) == 0u)
                        ok = __all_sync(kAll, ld_relaxed_s32(a.status) == 0 && globaltimer_ns() - t0 <= a.wait_ns);
                } while (ok && !__all_sync(kAll, have));
            }
            if (!ok) break;
            __syncwarp();
            double L = 0.0, dk = 0.0;
            if (lane < h.nu) {
                L = (double)lt[h.st];
                if (LDLT) dk = D[h.k];
            }
            // every product of the chunk, to its place
            constexpr int B = 8;
            for (uint32_t t0 = 0; t0 < h.total; t0 += 32 * B) {
                uint32_t wd[B];
                double Lik[B];
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const uint32_t t = t0 + 32 * i + lane;
                    wd[i] = t < h.total ? tw[t] : kRfDrop;
                    Lik[i] = wd[i] & kRfDrop ? 0.0 : (double)lt[cst[wd[i] >> kRfUpdateAt] + t];
                }
                if (t0 == 0) {
                    if (lane < h.nu) {
                        cL[lane] = L;
                        cD[lane] = dk;
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    if (wd[i] & kRfDrop) continue;
                    const uint32_t q = wd[i] >> kRfUpdateAt;
                    const double v = __dmul_rn(Lik[i], cL[q]);
                    tv[wd[i] & kRfPlace] = LDLT ? __dmul_rn(v, cD[q]) : v;
                }
            }
            __syncwarp();
            // the subtractions, in the order of the updates
            for (uint32_t s = lane; s < m; s += 32) {
                double x = acc[s];
                const uint32_t t1 = sg[s + 1];
#pragma unroll 4
                for (uint32_t t = sg[s]; t < t1; ++t) x = __dsub_rn(x, tv[t]);
                acc[s] = x;
            }
            __syncwarp();
            u0 += h.nu;
            f += h.total;
            g += m + 1;
        }
        if (!ok) {
            if (lane == 0) fail(PRISM_ERR_TIMEOUT, j);
            return;
        }
        // the pivot, then the column divided by it
        double piv = acc[0];
        if (LDLT) {
            if (fabs(piv) < 1e-15 && lane == 0) fail(PRISM_ERR_ZERO_PIVOT, j);
            if (lane == 0) D[j] = piv;
        } else {
            if (!(piv > 0.0) && lane == 0) fail(PRISM_ERR_NOT_SPD, j);
            piv = __dsqrt_rn(piv);
            if (lane == 0) lt[b] = (Low)piv;
        }
        for (uint32_t s = 1 + lane; s < m; s += 32) lt[off0 + s] = (Low)__ddiv_rn(acc[s], piv);
        // every lane's values are ordered before lane 0's release by the warp's barrier
        __syncwarp();
        if (lane == 0) st_release_u32(a.done + j, a.epoch);
    }
}

// dst[cdst[t]] = src[csrc[t]]: new coefficients into a layout.  An index outside its
// array is not followed: the first such t is recorded (t + 1) in *bad for the host.
template <typename Low>
__global__ void __launch_bounds__(kBlock) k_rf_coef(uint32_t count, const uint32_t* __restrict__ cdst,
                                                    const uint32_t* __restrict__ csrc, const Low* __restrict__ src,
                                                    uint64_t src_n, Low* __restrict__ dst, uint64_t dst_n,
                                                    unsigned* bad) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const uint32_t d = cdst[t], s = csrc[t];
        if (d >= dst_n || s >= src_n) {
            atomicCAS(bad, 0u, t + 1);
            continue;
        }
        dst[d] = src[s];
    }
}

// New diagonals into a layout: d = (double)lt[idx] (IC) or D[idx] (ILDLT), stored as d or
// 1/d (the streamed records of the dividing operations), in D2 (double or float).
template <typename Low, typename D2>
__global__ void __launch_bounds__(kBlock) k_rf_diag(uint32_t count, const uint32_t* __restrict__ ddst,
                                                    const uint32_t* __restrict__ dsrc, const Low* __restrict__ lt,
                                                    const double* __restrict__ D, uint64_t src_n, int ic, int recip,
                                                    D2* __restrict__ dst, uint64_t dst_n, unsigned* bad) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < count; t += gridDim.x * blockDim.x) {
        const uint32_t di = ddst[t], si = dsrc[t];
        if (di >= dst_n || si >= src_n) {
            atomicCAS(bad, 0u, t + 1);
            continue;
        }
        const double d = ic ? (double)lt[si] : D[si];
        dst[di] = (D2)(recip ? 1.0 / d : d);
    }
}

int rf_grid(const Handle& h, uint64_t items) {
    uint64_t want = (items + kBlock - 1) / kBlock;
    const uint64_t cap = (uint64_t)h.info.sms * 8;
    if (want < 1) want = 1;
    return (int)(want < cap ? want : cap);
}
}  // namespace

// The maps of one device sweep: coefficient positions (in factor-value units) and
// diagonal positions (in the layout's diagonal units) with the factor entries they
// come from.
struct SweepValueMap {
    DevBuf<uint32_t> cdst, csrc, ddst, dsrc;
    uint32_t ncoef = 0, ndiag = 0;
    bool built = false;
};

struct RefactorState {
    uint32_t epoch = 0;
    DevBuf<uint32_t> lt_rowptr, lt_col, a_ptr, a_pos, up_ptr, up_k, up_start, done;
    DevBuf<uint32_t> sched;   // columns by depth in the dependency graph
    DevBuf<uint64_t> uo, so;  // per column: its first update entry; its first chunk's segments
    DevBuf<uint16_t> place, seg;  // as RfArgs
    uint32_t smax = 0;
    unsigned long long wait_ns = kRfWaitNs;
    // the factor values and pivots the sweeps hold, and those a refactorisation writes: swapped
    // where it succeeds, so that one that fails leaves the factor as it was
    DevBuf<float> lt32, lt32_new;
    DevBuf<double> lt64, lt64_new, D, D_new;
    DevBuf<int> status;       // [status, first bad column]
    DevBuf<unsigned> bad;     // first out-of-range map entry: [coefficients, diagonals]
    SweepValueMap lower, upper;
    SweepValueMap lower_bk[kBlockWidths + 1], upper_bk[kBlockWidths + 1];  // of the copies for blocks (the last: level order)
    bool refactored = false;  // the device factor differs from the host one
};
void refactor_release(RefactorState* r) { delete r; }

namespace {
void upload_map(SweepValueMap& M, const std::vector<uint32_t>& cd, const std::vector<uint32_t>& cs,
                const std::vector<uint32_t>& dd, const std::vector<uint32_t>& ds, cudaStream_t st) {
    M.ncoef = (uint32_t)cd.size();
    M.ndiag = (uint32_t)dd.size();
    M.cdst.upload(cd.data(), cd.size(), st);
    M.csrc.upload(cs.data(), cs.size(), st);
    M.ddst.upload(dd.data(), dd.size(), st);
    M.dsrc.upload(ds.data(), ds.size(), st);
    M.built = true;
}

// The map of device sweep d, uploaded from host sweep s (idx: the same sweep with factor
// entry indices as values and diagonal sources as diag).
template <typename Low>
void build_map(const DevSweep& d, const Sweep<Low>& s, const Sweep<double>& idx, SweepValueMap& M, cudaStream_t st) {
    std::vector<uint32_t> cd, cs, dd, ds;
    const bool has_diag = s.op != SWEEP_NONE;
    if (d.layout == LAYOUT_FLOW) {
        FlowLayout F;
        std::vector<uint32_t> cmap;
        if (!flow_layout<Low>(s, slab_ranges<Low>(s, d.str_ctas_req), d.str_slots, F, nullptr, &cmap, d.fl_entries))
            throw Error(PRISM_ERR_CUDA, "dataflow layout could not be rebuilt");
        cd.reserve(cmap.size() / 2);
        cs.reserve(cmap.size() / 2);
        for (size_t t = 0; t < cmap.size(); t += 2) {
            cd.push_back(cmap[t]);
            cs.push_back((uint32_t)idx.val[cmap[t + 1]]);
        }
        if (has_diag) {
            for (uint32_t p = 0; p < idx.n; ++p) {
                dd.push_back(F.dg_pos[idx.order[p]]);
                ds.push_back((uint32_t)idx.diag[p]);
            }
        }
    } else if (d.layout == LAYOUT_STREAM) {
        StreamLayout L;
        std::vector<uint32_t> cmap;
        std::string why;
        if (!stream_layout<Low>(s, slab_ranges<Low>(s, d.str_ctas_req), kNoSlot, d.str_slot_bytes, L, &why, nullptr,
                                &cmap, d.str_round_cap))
            throw Error(PRISM_ERR_CUDA, "streamed layout could not be rebuilt: " + why);
        cd.reserve(cmap.size() / 2);
        cs.reserve(cmap.size() / 2);
        for (size_t t = 0; t < cmap.size(); t += 2) {
            cd.push_back(cmap[t]);
            cs.push_back((uint32_t)idx.val[cmap[t + 1]]);
        }
        if (has_diag) {
            // each row's diagonal sits right after its right-hand side in its record
            for (uint32_t p = 0; p < idx.n; ++p) {
                dd.push_back(L.in_slot[idx.order[p]] + 1);
                ds.push_back((uint32_t)idx.diag[p]);
            }
        }
    } else {
        const Sweep<double>* src = &idx;
        Sweep<double> slab;
        if (d.layout == LAYOUT_SLAB) {
            std::vector<uint32_t> cpos;
            slab_layout<double>(idx, d.num_ctas, d.rows_per_cta, cpos, slab);
            src = &slab;
        }
        cd.resize(src->val.size());
        cs.resize(src->val.size());
        for (size_t t = 0; t < src->val.size(); ++t) {
            cd[t] = (uint32_t)t;
            cs[t] = (uint32_t)src->val[t];
        }
        if (has_diag) {
            dd.resize(src->n);
            ds.resize(src->n);
            for (uint32_t p = 0; p < src->n; ++p) {
                dd[p] = p;
                ds[p] = (uint32_t)src->diag[p];
            }
        }
    }
    upload_map(M, cd, cs, dd, ds, st);
}

// New values into device sweep d through its map (lt: lt_n factor values, D: n pivots);
// `bad` (two words, zero before) receives the first out-of-range map entry of each kernel.
template <typename Low>
void apply_map(const Handle& h, cudaStream_t st, DevSweep& d, const SweepValueMap& M, const Low* lt, uint64_t lt_n,
               const double* D, bool ic, unsigned* bad) {
    if (!d.n) return;
    if (M.ncoef) {
        const bool stream = d.streamed();
        DevBuf<unsigned char>& blob = d.layout == LAYOUT_FLOW ? d.fl_chunks : d.str_blob;
        Low* dst = stream ? reinterpret_cast<Low*>(blob.get())
                          : (std::is_same<Low, float>::value ? reinterpret_cast<Low*>(d.val32.get())
                                                             : reinterpret_cast<Low*>(d.val64.get()));
        const uint64_t dst_n = stream ? blob.size() / sizeof(Low)
                                      : (std::is_same<Low, float>::value ? d.val32.size() : d.val64.size());
        k_rf_coef<Low><<<rf_grid(h, M.ncoef), kBlock, 0, st>>>(M.ncoef, M.cdst.get(), M.csrc.get(), lt, lt_n, dst,
                                                               dst_n, bad);
        PRISM_LAUNCHED();
    }
    if (M.ndiag) {
        const int recip = d.streamed() && (d.op == SWEEP_DIV || d.op == SWEEP_PREDIV);
        const uint64_t src_n = ic ? lt_n : d.n;
        DevBuf<unsigned char>& blob = d.layout == LAYOUT_FLOW ? d.fl_dg : d.str_blob;
        if (d.streamed() && d.acc32) {
            k_rf_diag<Low, float><<<rf_grid(h, M.ndiag), kBlock, 0, st>>>(
                M.ndiag, M.ddst.get(), M.dsrc.get(), lt, D, src_n, ic, recip, reinterpret_cast<float*>(blob.get()),
                blob.size() / sizeof(float), bad + 1);
        } else {
            const bool stream = d.streamed();
            double* dst = stream ? reinterpret_cast<double*>(blob.get()) : d.diag.get();
            const uint64_t dst_n = stream ? blob.size() / sizeof(double) : d.diag.size();
            k_rf_diag<Low, double><<<rf_grid(h, M.ndiag), kBlock, 0, st>>>(M.ndiag, M.ddst.get(), M.dsrc.get(), lt,
                                                                            D, src_n, ic, recip, dst, dst_n, bad + 1);
        }
        PRISM_LAUNCHED();
        if (d.fl_cols && recip) {  // blocks hold the diagonals themselves, too
            k_rf_diag<Low, double><<<rf_grid(h, M.ndiag), kBlock, 0, st>>>(M.ndiag, M.ddst.get(), M.dsrc.get(), lt, D,
                                                                            src_n, ic, 0, d.fl_dd.get(),
                                                                            d.fl_dd.size(), bad + 1);
            PRISM_LAUNCHED();
        }
    }
}
}  // namespace

namespace {
// the scatter kernels' record of an out-of-range map entry, as an error
void check_maps(RefactorState& R, cudaStream_t st, const char* what) {
    unsigned b[2] = {0, 0};
    PRISM_CUDA(cudaMemcpyAsync(b, R.bad.get(), 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    PRISM_CUDA(cudaStreamSynchronize(st));
    if (b[0] || b[1])
        throw Error(PRISM_ERR_CUDA, std::string("refactorisation: a value map of ") + what +
                                        " points outside its arrays (coefficient entry " + std::to_string(b[0]) +
                                        ", diagonal entry " + std::to_string(b[1]) + ")");
}
}  // namespace

void TriangularPrecond::refactor() {
    const HostFactor& F = *f_;
    if ((F.kind != 1 && F.kind != 3) || !F.plan)
        throw Error(PRISM_ERR_UNSUPPORTED, "device refactorisation covers IC and ILDLT factors");
    const RefactorPlan& P = *F.plan;
    if (P.n != h_.A.n) throw Error(PRISM_ERR_ARG, "the factor does not belong to this operator");
    if (P.max_col > kRfMaxCol)
        throw Error(PRISM_ERR_UNSUPPORTED, "a factor column longer than " + std::to_string(kRfMaxCol) + " entries");
    cudaStream_t st = h_.stream;
    const bool ldlt = F.kind == 3;
    // A paired sweep's coefficients combine several factor entries, which the value maps
    // below cannot rebuild: such sweeps are tuned again without pairing first.  Their old
    // device arrays go, so what was captured from them (a GMRES cycle graph) must not run again.
    if (!rf_ && (lower_.paired || upper_.paired)) {
        renew_uid();
        if (F.fp32) {
            if (lower_.paired) tune_sweep(h_, lower_, F.lower32, F.apply32, false);
            if (upper_.paired) tune_sweep(h_, upper_, F.upper32, F.apply32, false);
        } else {
            if (lower_.paired) tune_sweep(h_, lower_, F.lower64, false, false);
            if (upper_.paired) tune_sweep(h_, upper_, F.upper64, false, false);
        }
    }
    if (!rf_) {
        std::unique_ptr<RefactorState, void (*)(RefactorState*)> built(new RefactorState(), refactor_release);
        RefactorState& R = *built;
        // a diagonal factor has no updates and, ILDLT, no entries
        auto put = [&](DevBuf<uint32_t>& d, const std::vector<uint32_t>& v) {
            d.alloc(std::max<size_t>(v.size(), 1));
            d.upload(v.data(), v.size(), st);
        };
        R.lt_rowptr.upload(F.f0.rowptr.data(), F.f0.rowptr.size(), st);
        put(R.lt_col, F.f0.col);
        R.a_ptr.upload(P.a_ptr.data(), P.a_ptr.size(), st);
        put(R.a_pos, P.a_pos);
        R.up_ptr.upload(P.up_ptr.data(), P.up_ptr.size(), st);
        put(R.up_k, P.up_k);
        put(R.up_start, P.up_start);
        R.done.alloc(P.n);
        PRISM_CUDA(cudaMemsetAsync(R.done.get(), 0, (size_t)P.n * sizeof(uint32_t), st));
        // Longer columns leave one CTA an SM in any case, so their chunks take all the products a
        // place can name (columns of 600 entries, a full factor, ms: 534 with one update a chunk,
        // 384 now; a warp pass per update took 464).
        R.smax = P.max_col <= 512 ? 512u : kRfPlace + 1;
        // where each column's update entries start, and the segments of its chunks (cut as RfChunk
        // cuts them); what stands there is found on the device, once
        std::vector<uint64_t> uo((size_t)P.n + 1, 0), so((size_t)P.n + 1, 0), chain((size_t)P.n, 0);
        uint64_t longest = 0;
        for (uint32_t j = 0; j < P.n; ++j) {
            uint64_t c = 0, chunks = 0, in_chunk = 0;
            uint32_t updates = 32;
            for (uint32_t u = P.up_ptr[j]; u < P.up_ptr[j + 1]; ++u) {
                const uint64_t one = F.f0.rowptr[P.up_k[u] + 1] - P.up_start[u];
                if (updates == 32 || in_chunk + one > R.smax) {
                    ++chunks;
                    updates = 0;
                    in_chunk = 0;
                }
                ++updates;
                in_chunk += one;
                c += one;
                chain[j] = std::max(chain[j], chain[P.up_k[u]]);
            }
            chain[j] += chunks;
            longest = std::max(longest, chain[j]);
            uo[j + 1] = uo[j] + c;
            so[j + 1] = so[j] + chunks * (F.f0.rowptr[j + 1] - F.f0.rowptr[j] + (ldlt ? 2u : 1u));
        }
        R.wait_ns = kRfWaitNs + longest * kRfChunkNs;
        R.uo.upload(uo.data(), uo.size(), st);
        R.so.upload(so.data(), so.size(), st);
        // depth of each column in the dependency graph (its updates come from columns k < j),
        // and the columns ordered by depth, then index
        std::vector<uint32_t> depth(P.n, 0), sched(std::max<uint32_t>(P.n, 1), 0);
        uint32_t maxd = 0;
        for (uint32_t j = 0; j < P.n; ++j) {
            uint32_t d = 0;
            for (uint32_t u = P.up_ptr[j]; u < P.up_ptr[j + 1]; ++u) d = std::max(d, depth[P.up_k[u]] + 1);
            depth[j] = d;
            maxd = std::max(maxd, d);
        }
        std::vector<uint32_t> start((size_t)maxd + 2, 0);
        for (uint32_t j = 0; j < P.n; ++j) ++start[depth[j] + 1];
        for (uint32_t d = 0; d <= maxd; ++d) start[d + 1] += start[d];
        for (uint32_t j = 0; j < P.n; ++j) sched[start[depth[j]]++] = j;
        R.sched.upload(sched.data(), sched.size(), st);
        R.place.alloc(std::max<uint64_t>(uo[P.n], 1));
        R.seg.alloc(std::max<uint64_t>(so[P.n], 1));
        const size_t nnz = std::max<size_t>(F.f0.col.size(), 1);
        if (F.fp32) R.lt32.alloc(nnz), R.lt32_new.alloc(nnz);
        else R.lt64.alloc(nnz), R.lt64_new.alloc(nnz);
        R.D.alloc(std::max<uint32_t>(P.n, 1));
        R.D_new.alloc(std::max<uint32_t>(P.n, 1));
        R.status.alloc(2);
        R.bad.alloc(2);
        Sweep<double> ilo, iup;
        factor_index_sweeps(F, ilo, iup);
        if (F.fp32) {
            build_map<float>(lower_, F.lower32, ilo, R.lower, st);
            build_map<float>(upper_, F.upper32, iup, R.upper, st);
        } else {
            build_map<double>(lower_, F.lower64, ilo, R.lower, st);
            build_map<double>(upper_, F.upper64, iup, R.upper, st);
        }
        PRISM_CUDA(cudaStreamSynchronize(st));
        rf_ = std::move(built);  // whole
    }
    RefactorState& R = *rf_;
    RfArgs a;
    a.n = P.n;
    a.max_col = std::max<uint32_t>(P.max_col, 1);
    a.smax = R.smax;
    a.sched = R.sched.get();
    a.uo = R.uo.get();
    a.place = R.place.get();
    a.so = R.so.get();
    a.seg = R.seg.get();
    a.lt_rowptr = R.lt_rowptr.get();
    a.lt_col = R.lt_col.get();
    a.a_col = h_.A.col.get();
    a.a_val = h_.A.val.get();
    a.a_ptr = R.a_ptr.get();
    a.a_pos = R.a_pos.get();
    a.up_ptr = R.up_ptr.get();
    a.up_k = R.up_k.get();
    a.up_start = R.up_start.get();
    a.done = R.done.get();
    a.status = R.status.get();
    a.bad_col = R.status.get() + 1;
    a.wait_ns = R.wait_ns;
    if (R.epoch == 0) {  // the products' places, once per pattern
        const size_t ssm = (size_t)kRfWarps * a.max_col * 2 * sizeof(uint32_t);
        PRISM_CUDA(cudaFuncSetAttribute(k_rf_places, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm));
        const uint64_t want = ((uint64_t)P.n + kRfWarps - 1) / kRfWarps;
        const int g = (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)h_.info.sms * 4));
        k_rf_places<<<g, kBlock, ssm, st>>>(a, R.place.get(), R.seg.get(), ldlt ? 1 : 0);
        PRISM_LAUNCHED();
        PRISM_CUDA(cudaStreamSynchronize(st));
    }
    ++R.epoch;
    a.epoch = R.epoch;
    PRISM_CUDA(cudaMemsetAsync(R.status.get(), 0, 2 * sizeof(int), st));
    const size_t smem = (size_t)kRfWarps * rf_warp_bytes(a.max_col, a.smax);
    void* fn = F.fp32 ? (ldlt ? (void*)k_refactor<float, true> : (void*)k_refactor<float, false>)
                      : (ldlt ? (void*)k_refactor<double, true> : (void*)k_refactor<double, false>);
    PRISM_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int occ = 0;
    PRISM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBlock, smem));
    if (occ < 1) throw Error(PRISM_ERR_UNSUPPORTED, "the refactorisation kernel does not fit on an SM");
    const uint64_t want = ((uint64_t)P.n + kRfWarps - 1) / kRfWarps;
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)h_.info.sms * occ));
    void* lt = F.fp32 ? (void*)R.lt32_new.get() : (void*)R.lt64_new.get();
    double* D_new = R.D_new.get();
    void* args[] = {&a, &lt, &D_new};
    PRISM_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kBlock), args, smem, st));
    PRISM_LAUNCHED();
    int hs[2] = {0, 0};
    PRISM_CUDA(cudaMemcpyAsync(hs, R.status.get(), 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    PRISM_CUDA(cudaStreamSynchronize(st));
    if (hs[0] == PRISM_ERR_NOT_SPD)
        throw Error(PRISM_ERR_NOT_SPD, "refactorisation: non-positive pivot in column " + std::to_string(hs[1]));
    if (hs[0] == PRISM_ERR_ZERO_PIVOT)
        throw Error(PRISM_ERR_ZERO_PIVOT, "refactorisation: zero pivot in column " + std::to_string(hs[1]));
    if (hs[0] != 0) throw Error(hs[0], "refactorisation: a dependency wait ran out in column " + std::to_string(hs[1]));
    std::swap(R.lt32, R.lt32_new);
    std::swap(R.lt64, R.lt64_new);
    std::swap(R.D, R.D_new);
    const double* D = R.D.get();
    // the new values into every device layout of the two sweeps
    const bool ic = F.kind == 1;
    const uint64_t lt_n = F.f0.col.size();
    PRISM_CUDA(cudaMemsetAsync(R.bad.get(), 0, 2 * sizeof(unsigned), st));
    if (F.fp32) {
        apply_map<float>(h_, st, lower_, R.lower, R.lt32.get(), lt_n, D, ic, R.bad.get());
        apply_map<float>(h_, st, upper_, R.upper, R.lt32.get(), lt_n, D, ic, R.bad.get());
    } else {
        apply_map<double>(h_, st, lower_, R.lower, R.lt64.get(), lt_n, D, ic, R.bad.get());
        apply_map<double>(h_, st, upper_, R.upper, R.lt64.get(), lt_n, D, ic, R.bad.get());
    }
    for (uint32_t c = 0; c <= kBlockWidths; ++c) {
        DevSweep& lo = c < kBlockWidths ? lower_bk_.flow[c] : lower_bk_.level;
        DevSweep& up = c < kBlockWidths ? upper_bk_.flow[c] : upper_bk_.level;
        if (lo.n) refresh_block_copy(lo, R.lower_bk[c], true);
        if (up.n) refresh_block_copy(up, R.upper_bk[c], false);
    }
    check_maps(R, st, "the sweeps");
    R.refactored = true;
    PRISM_CUDA(cudaStreamSynchronize(st));
}

// The refactored values into a copy for the block sweeps; its map is built once.  (Copies uploaded
// again after each refactorisation, laid out twice on the host: IC 64^3, 8 columns, refactorisation
// and block apply 1,308 ms.)
void TriangularPrecond::refresh_block_copy(DevSweep& d, SweepValueMap& M, bool lower) {
    const HostFactor& F = *f_;
    RefactorState& R = *rf_;
    cudaStream_t st = h_.stream;
    const uint64_t lt_n = F.f0.col.size();
    if (!M.built) {
        Sweep<double> ilo, iup;
        factor_index_sweeps(F, ilo, iup);
        const Sweep<double>& idx = lower ? ilo : iup;
        if (F.fp32) build_map<float>(d, lower ? F.lower32 : F.upper32, idx, M, st);
        else build_map<double>(d, lower ? F.lower64 : F.upper64, idx, M, st);
    }
    if (F.fp32) apply_map<float>(h_, st, d, M, R.lt32.get(), lt_n, R.D.get(), F.kind == 1, R.bad.get());
    else apply_map<double>(h_, st, d, M, R.lt64.get(), lt_n, R.D.get(), F.kind == 1, R.bad.get());
}

// A copy for the block sweeps uploaded from the host factor: nothing to do until the device has
// refactored it.
void TriangularPrecond::refresh_block_copy(DevSweep& d, uint32_t copy, bool lower) {
    if (!rf_ || !rf_->refactored) return;
    RefactorState& R = *rf_;
    PRISM_CUDA(cudaMemsetAsync(R.bad.get(), 0, 2 * sizeof(unsigned), h_.stream));
    refresh_block_copy(d, lower ? R.lower_bk[copy] : R.upper_bk[copy], lower);
    check_maps(R, h_.stream, "a block copy");
}

int TriangularPrecond::export_refactored(int which, uint32_t* n, uint64_t* nnz, uint32_t* rowptr, uint32_t* col,
                                         double* val, double* diag) const {
    const HostFactor& F = *f_;
    const RefactorState& R = *rf_;
    if (which != 0) return 9;
    const uint32_t nn = F.f0.n;
    const size_t m = F.f0.col.size();
    if (n) *n = nn;
    if (nnz) *nnz = m;
    if (rowptr) std::copy(F.f0.rowptr.begin(), F.f0.rowptr.end(), rowptr);
    if (col) std::copy(F.f0.col.begin(), F.f0.col.end(), col);
    if (val) {
        if (F.fp32) {
            std::vector<float> v(m);
            PRISM_CUDA(cudaMemcpy(v.data(), R.lt32.get(), m * sizeof(float), cudaMemcpyDeviceToHost));
            for (size_t t = 0; t < m; ++t) val[t] = (double)v[t];
        } else {
            PRISM_CUDA(cudaMemcpy(val, R.lt64.get(), m * sizeof(double), cudaMemcpyDeviceToHost));
        }
    }
    if (diag && F.kind == 3) PRISM_CUDA(cudaMemcpy(diag, R.D.get(), nn * sizeof(double), cudaMemcpyDeviceToHost));
    return 0;
}

}  // namespace prism
