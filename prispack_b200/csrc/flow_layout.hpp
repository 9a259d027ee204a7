// Dataflow layout of a triangular sweep (k_sweep_flow, flow_sweep.cuh).
//
// The rows are split into slabs of contiguous rows; a slab's rows, in (level, row)
// order, into tasks of up to kFlowRows rows of one level (kFlowLanes lanes each), and
// task t of a slab belongs to worker warp t mod kFlowWorkers.  Every row of the slab
// and every row of another slab that it reads ("halo", always upstream) has a
// shared-memory value slot of its own, which holds a sentinel until the value is there:
// readiness travels with the value.
//
// A row's entries are sorted by the level of the row they read (a halo row counts as
// kFlowHaloLag levels later).  The tail, its four latest entries that read rows of the
// slab, is read once the level before the task's is done; the others, the front,
// before.  Both are padded in front with entries of slot 0 (value 0.0) and coefficient
// 0.  Front position p belongs to lane p mod 4 of the row's four, which adds it to its
// chain c_i = fma(coef, x, c_i);  then s = (c0 + c1) + (c2 + c3), and s = fma(coef, x, s)
// over the tail in order.
//
//   chunks   per worker warp of a slab, in the order it reads them; one chunk is E
//            front positions (4 or 8, per layout) of each lane of a task's m rows: slots
//            [4 m] x E x u16, then coefficients [E * vb / 16][4 m] x 16 B (vb bytes a
//            value); a task's last chunk ends with the tails: coefficients
//            [vb / 4][m] x 16 B, slots [m] x 4 x u16 (padded to 16 B)
//   hdr      per task and row: {row (kFlowNone: no row), exchange entry its value is
//            published in (kFlowNone: read by no other slab), slot | barrier << 16,
//            chunks of the task | m << 8 | m of the worker's next task << 12 | sync << 17 |
//            arrive << 22}.
//            Level l of a slab opens when named barrier 1 + l mod kFlowBars completes, on which
//            the workers of levels l - 1 and l meet: sync is their number where the task
//            waits for its level (0: an earlier task of the worker did, or the first
//            level), arrive that of the next level where the worker is done with this one
//            and has no task of the next (0 otherwise)
//   dg       per task and row: the diagonal, or its reciprocal for the dividing operations
//   warp     per slab and worker: {0, first task, tasks, chunks, start and length in
//            `chunks` / 16, 0, 0}
//   halo     per slab, by level: {exchange entry, slot}
// Slabs are numbered from upstream to downstream.
#pragma once

#include <memory>
#include <string>

#include "host_setup.hpp"

namespace prism {

constexpr uint32_t kFlowWorkers = 13;
// Named barriers in turn over a slab's levels.  A worker that waits for level l did its task
// before at a level >= l - kFlowWorkers, whose barrier is done, so no barrier is taken up
// again before it opened as long as there are at least kFlowWorkers of them.
constexpr uint32_t kFlowBars = 15;
static_assert(kFlowBars >= kFlowWorkers && kFlowBars <= 15, "named barriers");
constexpr uint32_t kFlowLanes = 4, kFlowRows = 32 / kFlowLanes;
constexpr uint32_t kFlowTail = 4;
PRISM_HD constexpr uint32_t flow_tail_bytes(uint32_t m, uint32_t vb) { return (m * (4u * vb + 8u) + 15u) & ~15u; }
constexpr uint32_t kFlowNone = 0xFFFFFFFFu;
constexpr uint32_t kFlowHaloLag = 8;

// Bytes that alloc leaves untouched: each slab's thread clears and fills its own.
class FlowBytes {
  public:
    void alloc(size_t count) {
        p_.reset(new uint8_t[count]);
        n_ = count;
    }
    const uint8_t* data() const { return p_.get(); }
    size_t size() const { return n_; }
    uint8_t& operator[](size_t i) { return p_[i]; }
    const uint8_t& operator[](size_t i) const { return p_[i]; }

  private:
    std::unique_ptr<uint8_t[]> p_;
    size_t n_ = 0;
};

struct FlowLayout {
    uint32_t entries = 0;              // E
    uint32_t slabs = 0, slots = 0, published = 0, tasks = 0;  // slots: of the slab that needs most
    FlowBytes chunks;
    std::vector<uint32_t> hdr, warp, halo_ptr, halo;
    std::vector<double> dg;
    std::vector<uint32_t> dg_pos;  // per row: its entry of dg
};

// Lays the sweep out for slabs [start[b], start[b + 1]), with E = entries (0: by the rows'
// lengths).  False when a slab needs more than max_slots value slots or a task more than 255 chunks
// (a row of 4,080 or 8,160 front entries).  order, coef_map: as for stream_layout (every position
// is an early one; coef_map in units of the factor value within `chunks`).
template <typename Low>
bool flow_layout(const Sweep<Low>& s, const std::vector<uint32_t>& start, uint32_t max_slots, FlowLayout& out,
                 StreamOrder* order = nullptr, std::vector<uint32_t>* coef_map = nullptr, uint32_t entries = 0);

// Replays k_sweep_flow on the host, in its arithmetic (float when acc32): every index of the
// layout checked against its array, each worker's tasks taken in order as their values become
// ready, every row computed exactly once.  Returns an empty string, or what is wrong.
template <typename Low>
std::string flow_layout_replay(const Sweep<Low>& s, const FlowLayout& L, bool acc32, const double* in, double* out);

}  // namespace prism
