// Dataflow triangular sweep: one triangular sweep (IncompleteCholesky /
// IncompleteLDLT / IncompleteLU MSolve*UsePtr, IncompleteCholesky.cpp:249-295,
// IncompleteLDLT.cpp:188-233, IncompleteLU.cpp:268-297) over the layout of
// flow_layout.hpp.
//
// What bounds it.  A sweep is a chain of dependency wavefronts, so its time is their
// number times the latency of one; the bytes would take a tenth of that.  What a warp
// does once between two wavefronts therefore counts in instructions (4-5 cycles each,
// dependent), and everything else must happen beside the chain.  Where the chain crosses
// slabs, as on every 3D operator, the hop from one to the next (store, L2, poll, store into
// the slot, poll: about 1.3 us against 0.12 inside a slab) is most of it: of the 921 us of
// the level-0 lower sweep of AMSED 128^3 a model of the chain gives 338 to 260 hops and 247 to
// the rest; the workers' tasks, spread over all of them, would take 144.
//
//  - A slab belongs to one CTA at a time and its values to that CTA's shared memory, each
//    in a slot of its own that holds a sentinel until the value is there.  No slot is used
//    twice within a slab, so nothing has to be waited for before a write, and a reader
//    needs no flag.
//  - kFlowWorkers warps take the tasks in turn.  A task takes a warp some 1,700 cycles, 256
//    instructions that mostly wait for one another, so several must be under way for each
//    wavefront of a slab, and 16 warps are what 128 registers a thread leave.  13 and three for the halo: IC 512^2 FP64 1,034 us an
//    apply, FCG with AMSED on 64^3 91.9 ms, FGMRES with GMSLR on 50^3 30.1 ms; 12 and four
//    1,070, 91.1, 31.3; 14 and two 1,004, 93.5, 29.3.  A warp sums the front of its task, whose
//    values are mostly there, while the others finish the levels before; the level itself
//    opens with a named barrier on which only the workers of two neighbouring levels meet
//    (a hand-over of 93 cycles; polling the last values takes 2 to 3 times that, and
//    polling warps slow down the one that the chain waits for).  Only then come the four
//    tail values, their multiply-adds, the result's store and the next hand-over.
//  - Four lanes a row: short tasks, so that the workers keep up with the chain (a lane a row:
//    0.26 us a level on 3D factors against 0.19).
//  - Records come by plain 16-byte loads one chunk ahead into registers, from lines brought
//    into L2 12 KB ahead; bulk copies into shared memory cost the worker more (a proxy fence
//    waits for its global stores: 540 cycles a chunk).
//  - Values that other slabs read go into an exchange array as {value, epoch} in one 8- or
//    16-byte word; three warps a CTA copy the slab's halo from it into its slots.  The epoch
//    counts the sweeps of the layout, so nothing is marked before a sweep, the output can
//    be the input, and a sweep that was given up leaves nothing that the next could take
//    for its own.
//  - There are more slabs than CTAs where a wavefront is wide: a CTA takes its next slab
//    while the wavefront is elsewhere.
//
// Blocks of columns run the same kernel with 1, 2 or 4 columns a lane (block_columns): a record
// serves them all, groups of CTAs take the columns. Us a sweep, level order before: IC 192^2,
// 64 columns 4,208, now 311; AMSED 95x71 FP64, 13 columns 485 to 1,540, now 31.
//
// Measured against the streamed rounds (us an M^-1 apply): IC 64^2 FP64 135 against 334, IC
// 512^2 FP64 1,034 against 2,948, ILUT 61x53x47 with float values 365 against 950 (level
// order), AMSED 64^3 FP64 1,600 against 2,200, AMSED 128^3 with float arithmetic 4,500
// against 5,140.
//
// Progress: a task waits for earlier levels of its slab, held by warps that are ahead of it
// or on their way there, and for slabs of a lower number; CTA b takes the slabs b, b + grid,
// ... in turn and all CTAs are co-resident (cooperative launch), so the lowest unfinished
// slab is always in work.  Every wait on a value is a bounded poll: when it runs out, the
// status is raised, the CTA told to leave, and its warps go on without waiting, barriers
// included, until they are through.
#pragma once

#include "flow_layout.hpp"
#include "kernels.cuh"
#include "stream_sweep.cuh"

namespace prism {

constexpr int kFlowHaloWarps = 3;
constexpr int kFlowThreads = 32 * ((int)kFlowWorkers + kFlowHaloWarps);
constexpr uint32_t kFlowFixedSmem = 128;    // "leave" word, then the value slots
constexpr unsigned kFlowPolls = 1024;       // polls of a value slot between looks at the clock
constexpr uint32_t kFlowAhead = 12288;      // bytes of a worker's stream brought into L2 ahead of its reads
constexpr uint32_t kFlowPad = kFlowAhead + 4096;  // ... and thus allocated past the end of `chunks`
PRISM_HD inline uint32_t flow_smem(uint32_t slots, uint32_t ab) { return kFlowFixedSmem + slots * ab; }

struct FlowArgs {
    const unsigned char* chunks;
    const uint4* hdr;
    const void* dg;             // Acc per (task, row)
    const uint4* warp;
    const uint32_t* halo_ptr;
    const uint2* halo;
    void* xch;                  // exchange entries: FlowWord<Acc>
    uint32_t* ctl;              // [epoch, ticket]
    const double* in;
    double* out;
    int* status;
    unsigned long long wait_ns;
    uint32_t slabs, slots;
    // blocks of columns (interleaved, X[row * k + c]): `members` CTAs a group of columns
    const double* dd;           // the diagonal itself, per (task, row)
    uint32_t members, k;
};

// record words: read once, in order, by one warp
__device__ __forceinline__ uint4 ldg_stream_u4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A value and the epoch of the sweep it belongs to, written and read as one word.
template <typename Acc>
struct FlowWord;
template <>
struct FlowWord<float> {
    unsigned long long w;
    static __device__ __forceinline__ void put(FlowWord* p, float v, uint32_t epoch) {
        st_relaxed_u64(p, ((unsigned long long)epoch << 32) | __float_as_uint(v));
    }
    static __device__ __forceinline__ bool get(const FlowWord* p, float& v, uint32_t epoch) {
        const unsigned long long w = ld_relaxed_u64(p);
        v = __uint_as_float((uint32_t)w);
        return (uint32_t)(w >> 32) == epoch;
    }
};
template <>
struct alignas(16) FlowWord<double> {
    unsigned long long v, e;
    static __device__ __forceinline__ void put(FlowWord* p, double v, uint32_t epoch) {
        asm volatile(
            "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
            "l"(__double_as_longlong(v)), "l"((unsigned long long)epoch)
            : "memory");
    }
    static __device__ __forceinline__ bool get(const FlowWord* p, double& v, uint32_t epoch) {
        unsigned long long lo, hi;
        asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                     : "=l"(lo), "=l"(hi)
                     : "l"(p)
                     : "memory");
        v = __longlong_as_double((long long)lo);
        return (uint32_t)hi == epoch;
    }
};

// A value slot's sentinel: a signalling NaN, which no arithmetic returns.
constexpr uint32_t kFlowPendF = 0x7FA0BEEFu;
__device__ __forceinline__ bool flow_pending(float v) { return __float_as_uint(v) == kFlowPendF; }
__device__ __forceinline__ bool flow_pending(double v) { return (uint32_t)__double2hiint(v) == (uint32_t)(kPending >> 32); }
__device__ __forceinline__ void flow_load(uint32_t at, float& v) {
    asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
}
__device__ __forceinline__ void flow_load(uint32_t at, double& v) {
    asm volatile("ld.volatile.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
}
// Named barriers.  The id in a register makes a hand-over 93 cycles, not the 30 of an
// immediate one, but a switch over the ids costs more than that.
__device__ __forceinline__ void flow_bar_sync(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void flow_bar_arrive(uint32_t id, uint32_t threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void flow_load2(uint32_t at, double& v, double& w) {
    asm volatile("ld.volatile.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v), "=d"(w) : "r"(at) : "memory");
}
__device__ __forceinline__ void flow_peek2(uint32_t at, double& v, double& w) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v), "=d"(w) : "r"(at));
}
__device__ __forceinline__ void flow_store2(uint32_t at, double v, double w) {
    asm volatile("st.volatile.shared.v2.f64 [%0], {%1, %2};" ::"r"(at), "d"(v), "d"(w) : "memory");
}
// a first look: may miss a value just written, so only a loop of flow_load may wait
__device__ __forceinline__ void flow_peek(uint32_t at, float& v) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
}
__device__ __forceinline__ void flow_peek(uint32_t at, double& v) {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at));
}
__device__ __forceinline__ void flow_store(uint32_t at, float v) {
    asm volatile("st.volatile.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
__device__ __forceinline__ void flow_store(uint32_t at, double v) {
    asm volatile("st.volatile.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

// v / d from r = 1 / d rounded: one step that takes the product's error out again.
__device__ __forceinline__ double flow_quotient(double v, double d, double r) {
    const double q = acc_mul(v, r), e = acc_fma(acc_fma(-q, d, v), r, q);
    return isfinite(q) ? e : q;
}

// C = 0: one vector.  C = 1, 2, 4: C columns of a block at once (double arithmetic); CTA
// g * members + m takes the slabs m, m + members, ... for the columns C g .. C g + C - 1.
template <typename Low, int OP, typename Acc, int E, int C>
static __global__ void __launch_bounds__(kFlowThreads, 1) k_sweep_flow(const FlowArgs a) {
    extern __shared__ __align__(128) unsigned char fsm[];
    constexpr uint32_t vb = sizeof(Low);
    constexpr int N = C == 0 ? 1 : C;
    constexpr int CQ = E * (int)vb / 16;         // 16-byte words of a lane's coefficients
    constexpr uint32_t LB = E * (2 + vb);         // bytes of a lane in a chunk
    constexpr int V = N == 1 ? 1 : 2, PL = N / V; // columns of a slot word, planes of slot words
    constexpr uint32_t sb = sizeof(Acc) * V;      // bytes of a slot word
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t xs = smem_addr(fsm + kFlowFixedSmem), plane = a.slots * sb;
    volatile uint32_t* leave = reinterpret_cast<volatile uint32_t*>(fsm);
    const uint32_t group = C == 0 ? 0u : blockIdx.x / a.members, groups = C == 0 ? 1u : gridDim.x / a.members;
    const uint32_t first_slab = C == 0 ? blockIdx.x : blockIdx.x % a.members, step = C == 0 ? gridDim.x : a.members;
    const uint32_t col = group * N;               // first column
    FlowWord<Acc>* xch = static_cast<FlowWord<Acc>*>(a.xch) + group * N;
    auto word_of = [&](uint32_t e) { return xch + (C == 0 ? (size_t)e : (size_t)e * (groups * N)); };
    // the N values of a slot
    auto peek = [&](uint32_t at, Acc(&x)[N]) {
        if constexpr (N == 1) {
            flow_peek(at, x[0]);
        } else {
#pragma unroll
            for (int p = 0; p < PL; ++p) flow_peek2(at + p * plane, x[2 * p], x[2 * p + 1]);
        }
    };
    auto look = [&](uint32_t at, Acc(&x)[N]) {
        if constexpr (N == 1) {
            flow_load(at, x[0]);
        } else {
#pragma unroll
            for (int p = 0; p < PL; ++p) flow_load2(at + p * plane, x[2 * p], x[2 * p + 1]);
        }
        bool pend = false;
#pragma unroll
        for (int j = 0; j < N; ++j) pend = pend || flow_pending(x[j]);
        return pend;
    };
    auto store = [&](uint32_t at, const Acc(&x)[N]) {
        if constexpr (N == 1) {
            flow_store(at, x[0]);
        } else {
#pragma unroll
            for (int p = 0; p < PL; ++p) flow_store2(at + p * plane, x[2 * p], x[2 * p + 1]);
        }
    };
    uint32_t epoch;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(epoch) : "l"(a.ctl) : "memory");
    ++epoch;
    if (threadIdx.x == 0) *leave = 0;
    bool dead = false;  // this lane's wait ran out, or another's did
    unsigned long long since = 0;
    // after kFlowPolls polls without success
    auto expired = [&]() {
        const unsigned long long now = globaltimer_ns();
        if (since == 0) since = now;
        if (*leave != 0u || ld_relaxed_s32(a.status) != 0 || now - since > a.wait_ns) {
            atomicCAS(a.status, 0, 6);
            *leave = 1u;
            dead = true;
        }
    };
    for (uint32_t b = first_slab; b < a.slabs; b += step) {
        for (uint32_t i = threadIdx.x; i < a.slots; i += blockDim.x) {
            Acc v;
            if constexpr (sizeof(Acc) == 4) v = __uint_as_float(kFlowPendF);
            else v = __longlong_as_double((long long)kPending);
            Acc x[N];
#pragma unroll
            for (int j = 0; j < N; ++j) x[j] = i == 0 ? (Acc)0 : v;
            store(xs + i * sb, x);
        }
        __syncthreads();
        if (warp < (int)kFlowWorkers) {
            const uint4 wi = __ldg(a.warp + ((size_t)b * kFlowWorkers + warp) * 2);
            const uint4 we = __ldg(a.warp + ((size_t)b * kFlowWorkers + warp) * 2 + 1);
            const uint32_t nt = wi.z, nch = wi.w;
            const uint4* hp = a.hdr + (size_t)wi.y * kFlowRows + lane / (int)kFlowLanes;
            const Acc* dp = static_cast<const Acc*>(a.dg) + (size_t)wi.y * kFlowRows + lane / (int)kFlowLanes;
            const double* ep = a.dd + (size_t)wi.y * kFlowRows + lane / (int)kFlowLanes;
            const unsigned char* src = a.chunks + (size_t)we.x * 16;
            for (uint32_t o = (uint32_t)lane * 128; o < kFlowAhead && o < we.y * 16u; o += 4096) prefetch_l2(src + o);
            uint4 h0 = make_uint4(kFlowNone, kFlowNone, 0, 0), h1 = h0;
            Acc d0 = (Acc)1, d1 = (Acc)1;
            double e0 = 1.0;
            double v0[N];
#pragma unroll
            for (int j = 0; j < N; ++j) v0[j] = 0.0;
            if (nt > 0) h0 = __ldg(hp), d0 = __ldg(dp);
            uint32_t t = 0;
            // the next task's header and this one's right-hand side
            auto ahead = [&]() {
                h1.x = kFlowNone;
                if (t + 1 < nt) h1 = __ldg(hp + (size_t)(t + 1) * kFlowRows), d1 = __ldg(dp + (size_t)(t + 1) * kFlowRows);
                if (C != 0 && (OP == OP_DIV || OP == OP_PREDIV) && t < nt) e0 = __ldg(ep + (size_t)t * kFlowRows);
                if (h0.x != kFlowNone) {
                    if constexpr (C == 0) {
                        v0[0] = a.in[h0.x];
                    } else {
#pragma unroll
                        for (int j = 0; j < N; ++j) v0[j] = col + j < a.k ? a.in[(size_t)h0.x * a.k + col + j] : 0.0;
                    }
                }
            };
            ahead();
            // the chunk in work and the next one (lanes without a row read slot 0)
            uint4 q[CQ], qn[CQ];
            uint32_t sl[E / 2], sn[E / 2];
            constexpr int TQ = (int)vb / 4;
            uint4 tq[TQ];  // the task's tail
            uint2 ts = make_uint2(0, 0);
#pragma unroll
            for (int i = 0; i < TQ; ++i) tq[i] = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < CQ; ++i) q[i] = qn[i] = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < E / 2; ++i) sl[i] = sn[i] = 0;
            auto fetch = [&](uint32_t(&s)[E / 2], uint4(&r)[CQ], uint32_t m) {
                const uint32_t lanes = m * kFlowLanes;
                if ((uint32_t)lane < lanes) {
                    const unsigned char* p = src + (uint32_t)lane * (2 * E);
                    if constexpr (E == 8) {
                        const uint4 v = ldg_stream_u4(p);
                        s[0] = v.x, s[1] = v.y, s[E / 2 - 2] = v.z, s[E / 2 - 1] = v.w;
                    } else {
                        const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
                        s[0] = v.x, s[1] = v.y;
                    }
                    const unsigned char* c = src + lanes * (2 * E) + (uint32_t)lane * 16u;
#pragma unroll
                    for (int i = 0; i < CQ; ++i) r[i] = ldg_stream_u4(c + (uint32_t)i * lanes * 16u);
                } else {
#pragma unroll
                    for (int i = 0; i < E / 2; ++i) s[i] = 0;
                }
                const uint32_t o = (uint32_t)lane * 128;
                const uint32_t bytes = lanes * LB;
                if (o < bytes) prefetch_l2(src + kFlowAhead + o);  // past the end at times, within the padding
                src += bytes;
            };
            uint32_t left = h0.w & 0xFFu;
            if (nch > 0) fetch(sl, q, h0.w >> 8 & 15u);
            auto fetch_tail = [&](uint32_t m) {
                ts = make_uint2(0, 0);
                if ((uint32_t)lane < m * kFlowLanes) {
                    const unsigned char* p = src + (uint32_t)lane / kFlowLanes * 16u;
#pragma unroll
                    for (int i = 0; i < TQ; ++i) tq[i] = ldg_stream_u4(p + (uint32_t)i * m * 16u);
                    ts = __ldg(reinterpret_cast<const uint2*>(src + m * (4 * vb) + (uint32_t)lane / kFlowLanes * 8u));
                }
                src += flow_tail_bytes(m, vb);
            };
            auto coef_of = [](const uint4& v, int i) {
                if constexpr (vb == 4)
                    return (Acc)__uint_as_float((i & 3) == 0 ? v.x : ((i & 3) == 1 ? v.y : ((i & 3) == 2 ? v.z : v.w)));
                else
                    return (i & 1) ? __hiloint2double((int)v.w, (int)v.z) : __hiloint2double((int)v.y, (int)v.x);
            };
            Acc c[N];
#pragma unroll
            for (int j = 0; j < N; ++j) c[j] = (Acc)0;
            const bool first = (lane & ((int)kFlowLanes - 1)) == 0;
#pragma unroll 1
            for (uint32_t ch = 0; ch < nch; ++ch) {
                if (left == 1) fetch_tail(h0.w >> 8 & 15u);
                if (ch + 1 < nch) fetch(sn, qn, (left > 1 ? h0.w >> 8 : h0.w >> 12) & 15u);
                auto at = [&](int i) { return xs + ((sl[i / 2] >> (16 * (i & 1))) & 0xFFFFu) * sb; };
                auto coef = [&](int i) { return coef_of(q[i * (int)vb / 16], i); };
                // the chunk's positions onto c, each value awaited.  A sentinel makes the chain
                // a NaN: no NaN, nothing was pending.  The warp stays together (lanes that spin
                // apart starve one another).
                auto add = [&]() {
                    constexpr int B = N == 4 ? 4 : E;  // positions in flight
                    Acc g[N];
#pragma unroll
                    for (int j = 0; j < N; ++j) g[j] = c[j];
#pragma unroll
                    for (int i0 = 0; i0 < E; i0 += B) {
                        Acc x[B][N];
#pragma unroll
                        for (int i = 0; i < B; ++i) peek(at(i0 + i), x[i]);
#pragma unroll
                        for (int i = 0; i < B; ++i)
#pragma unroll
                            for (int j = 0; j < N; ++j) g[j] = acc_fma(coef(i0 + i), x[i][j], g[j]);
                    }
                    bool nan = false;
#pragma unroll
                    for (int j = 0; j < N; ++j) nan = nan || g[j] != g[j];
                    if (!__any_sync(0xFFFFFFFFu, nan)) {
#pragma unroll
                        for (int j = 0; j < N; ++j) c[j] = g[j];
                        return;
                    }
#pragma unroll
                    for (int i = 0; i < E; i += 2) {
                        Acc y[2][N];
                        bool p;
                        unsigned polls = 0;
                        do {
                            p = look(at(i), y[0]);
                            p = look(at(i + 1), y[1]) || p;
                            p = __any_sync(0xFFFFFFFFu, p) && !dead;
                            if (p && ++polls >= kFlowPolls) {
                                polls = 0;
                                expired();
                                dead = __any_sync(0xFFFFFFFFu, dead);
                            }
                        } while (p);
#pragma unroll
                        for (int j = 0; j < N; ++j) c[j] = acc_fma(coef(i + 1), y[1][j], acc_fma(coef(i), y[0][j], c[j]));
                    }
                    since = 0;
                };
                add();
                if (--left == 0) {
                    const uint32_t slot_at = xs + (h0.z & 0xFFFFu) * sb, sync = h0.w >> 17 & 31u, id = h0.z >> 16 & 15u, arrive = h0.w >> 22;
                    const bool mine = first && h0.x != kFlowNone;
                    Acc s[N], vin[N];
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        vin[j] = (Acc)v0[j];
                        if (OP == OP_PREDIV) {
                            if constexpr (C == 0) vin[j] = acc_mul(vin[j], d0);
                            else vin[j] = flow_quotient(vin[j], e0, d0);
                        }
                        s[j] = acc_add(c[j], __shfl_xor_sync(0xFFFFFFFFu, c[j], 1));
                        s[j] = acc_add(s[j], __shfl_xor_sync(0xFFFFFFFFu, s[j], 2));
                    }
                    // the tail: rows of this slab alone, ready once the level before is
                    if (sync != 0u) flow_bar_sync(id, sync * 32u);
                    Acc x[4][N], res[N];
#pragma unroll
                    for (int i = 0; i < 4; ++i) peek(xs + (((i < 2 ? ts.x : ts.y) >> (16 * (i & 1))) & 0xFFFFu) * sb, x[i]);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < N; ++j) s[j] = acc_fma(coef_of(tq[i * (int)vb / 16], i), x[i][j], s[j]);
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        res[j] = acc_sub(vin[j], s[j]);
                        if (OP == OP_MUL || (OP == OP_DIV && C == 0)) res[j] = acc_mul(res[j], d0);
                        else if constexpr (OP == OP_DIV && C != 0) res[j] = flow_quotient(res[j], e0, d0);
                    }
                    if (mine) store(slot_at, res);
                    if (arrive != 0u) flow_bar_arrive(id == kFlowBars ? 1u : id + 1u, arrive * 32u);
                    if (mine) {
                        if (h0.y != kFlowNone) {
                            FlowWord<Acc>* w = word_of(h0.y);
#pragma unroll
                            for (int j = 0; j < N; ++j) FlowWord<Acc>::put(w + j, res[j], epoch);
                        }
#pragma unroll
                        for (int j = 0; j < N; ++j) {
                            const double rd = (double)res[j];
                            const double o = rd != rd ? __longlong_as_double((long long)kCanonicalNaN) : rd;
                            if constexpr (C == 0) a.out[h0.x] = o;
                            else if (col + j < a.k) a.out[(size_t)h0.x * a.k + col + j] = o;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < N; ++j) c[j] = (Acc)0;
                    ++t;
                    h0 = h1, d0 = d1;
                    left = h0.w & 0xFFu;
                    ahead();
                }
#pragma unroll
                for (int i = 0; i < CQ; ++i) q[i] = qn[i];
#pragma unroll
                for (int i = 0; i < E / 2; ++i) sl[i] = sn[i];
            }
        } else {
            const uint32_t h1 = __ldg(a.halo_ptr + b + 1);
            constexpr uint32_t S = 32 * kFlowHaloWarps;
            uint32_t i = __ldg(a.halo_ptr + b) + (uint32_t)(warp - (int)kFlowWorkers) * 32 + (uint32_t)lane;
            // One entry of the list a lane and the next one known: four in flight a lane cost more
            // registers and a longer way round the loop, which is what a value that is not there
            // yet waits for (sweeps of 64^2 to 50^3: 2 to 5% slower)
            uint2 e = i < h1 ? __ldg(a.halo + i) : make_uint2(kFlowNone, 0);
            uint2 nx = i + S < h1 ? __ldg(a.halo + i + S) : make_uint2(kFlowNone, 0);
            i += 2 * S;
            unsigned idle = 0;
            bool more = e.x != kFlowNone;
            while (__any_sync(0xFFFFFFFFu, more)) {
                Acc v[N];
                bool some = false, ok = true;
                // no branch between the loads: all are in flight at once
                const FlowWord<Acc>* w = word_of(more ? e.x : 0u);
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const bool in = FlowWord<Acc>::get(w + j, v[j], epoch);
                    ok = in && ok;
                }
                if (ok && more) {
                    store(xs + e.y * sb, v);
                    e = nx;
                    nx = i < h1 ? __ldg(a.halo + i) : make_uint2(kFlowNone, 0);
                    i += S;
                    some = true;
                    more = e.x != kFlowNone;
                }
                if (__any_sync(0xFFFFFFFFu, some)) {
                    idle = 0;
                    since = 0;
                } else {
                    if (++idle > 8) __nanosleep(64);
                    if ((idle & 255u) == 0u) expired();
                    if (__any_sync(0xFFFFFFFFu, dead)) break;
                }
            }
        }
        if (__syncthreads_or(*leave != 0u ? 1 : 0)) break;
    }
    // the last CTA opens the next epoch; the others have read this one
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.ctl + 1, 1u) == gridDim.x - 1) {
            a.ctl[1] = 0;
            a.ctl[0] = epoch;
        }
    }
}

// Right-hand side of a paired sweep: b'_r = b_r - sum m b_dep (one fused multiply-add per
// entry, in stored order, in double).
static __global__ void __launch_bounds__(kBlock) k_flow_pair_rhs(uint32_t n, const uint32_t* __restrict__ mptr,
                                                                 const uint32_t* __restrict__ mdep,
                                                                 const double* __restrict__ mcoef,
                                                                 const double* __restrict__ in,
                                                                 double* __restrict__ bp) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        double v = in[r];
        for (uint32_t q = __ldg(mptr + r); q < __ldg(mptr + r + 1); ++q)
            v = __fma_rn(-__ldg(mcoef + q), in[__ldg(mdep + q)], v);
        bp[r] = v;
    }
}

}  // namespace prism
