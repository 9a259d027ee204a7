// Host side of the dataflow sweep layout (flow_layout.hpp).
#include "flow_layout.hpp"
#include "host_threads.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

namespace prism {
namespace {

// An entry of a row: {level (halo rows later) << 32 | row read, stored entry, slot}.
struct Item {
    uint64_t key;
    uint32_t k, slot;
};

struct SlabPlan {
    std::vector<uint32_t> pos;        // positions of the sweep, in (level, row) order
    std::vector<uint32_t> task;       // first row (index into pos) of each task, and the end
    std::vector<uint32_t> chunks;     // chunks of each task
    std::vector<uint32_t> level;      // first task of each level of the slab, and the end
    std::vector<std::pair<uint32_t, uint32_t>> halo;  // {row, slot}
    std::vector<uint32_t> up;         // the slabs it reads
};

// Rows of other slabs -> their slots in the slab in work: open addressing, at most half full.
// Entries of the slabs before are told apart by their tag, so nothing is cleared between slabs.
class HaloSlots {
  public:
    HaloSlots() : tab_(1024, Entry{0, 0}) {}
    void start() {
        ++tag_;
        count_ = 0;
    }
    // the slot of `row`: `fresh` where it has none yet
    uint32_t put(uint32_t row, uint32_t fresh) {
        Entry& e = find(row);
        if (e.key >> 32 == tag_) return e.slot;
        e = Entry{(uint64_t)tag_ << 32 | row, fresh};
        if (++count_ * 2 > tab_.size()) grow();
        return fresh;
    }

  private:
    struct Entry {
        uint64_t key;
        uint32_t slot;
    };
    // the entry of `row`, or the free one where it goes
    Entry& find(uint32_t row) {
        const uint64_t key = (uint64_t)tag_ << 32 | row;
        for (uint64_t i = (row * 0x9E3779B97F4A7C15ull) >> 32;; ++i) {
            Entry& e = tab_[i & (tab_.size() - 1)];
            if (e.key == key || e.key >> 32 != tag_) return e;
        }
    }
    void grow() {
        std::vector<Entry> old(tab_.size() * 2, Entry{0, 0});
        old.swap(tab_);
        for (const Entry& e : old)
            if (e.key >> 32 == tag_) find((uint32_t)e.key) = e;
    }
    std::vector<Entry> tab_;
    uint32_t tag_ = 0;
    size_t count_ = 0;
};

}  // namespace

template <typename Low>
bool flow_layout(const Sweep<Low>& s, const std::vector<uint32_t>& start, uint32_t max_slots, FlowLayout& out,
                 StreamOrder* order, std::vector<uint32_t>* coef_map, uint32_t entries) {
    const uint32_t n = s.n, ns = (uint32_t)start.size() - 1;
    max_slots = std::min<uint32_t>(max_slots, 0xFFFFu);
    out = FlowLayout();
    out.slabs = ns;
    const bool recip = s.op == SWEEP_DIV || s.op == SWEEP_PREDIV;
    constexpr uint32_t vb = (uint32_t)sizeof(Low), Q = kFlowLanes;
    // rows of up to 16 positions in one chunk of four a lane
    const uint32_t E = entries ? entries : (s.val.size() <= 12 * (uint64_t)n ? 4 : 8), RB = Q * E * (2 + vb);
    out.entries = E;
    auto tail_bytes = [](uint32_t m) { return flow_tail_bytes(m, vb); };
    for (uint32_t b = 0; b < ns; ++b)
        if (start[b + 1] - start[b] >= max_slots) return false;
    std::vector<uint32_t> owner(n), slot(n);
    for (uint32_t b = 0; b < ns; ++b)
        for (uint32_t r = start[b]; r < start[b + 1]; ++r) owner[r] = b;
    std::vector<SlabPlan> plan(ns);
    for (uint32_t b = 0; b < ns; ++b) plan[b].pos.reserve(start[b + 1] - start[b]);
    for (uint32_t p = 0; p < n; ++p) {
        const uint32_t r = s.order[p];
        SlabPlan& P = plan[owner[r]];
        P.pos.push_back(p);
        slot[r] = (uint32_t)P.pos.size();  // slot 0 holds the padding's zero
    }
    std::vector<std::atomic<uint8_t>> pub(n);
    for (auto& x : pub) x.store(0, std::memory_order_relaxed);
    std::atomic<bool> fits{true};
    std::atomic<uint32_t> most{0}, next{0};
    const uint32_t T = std::min<uint32_t>(layout_threads(), ns);
    host_parallel_for(T, T, [&](uint32_t) {
        HaloSlots seen;
        for (uint32_t b = next++; b < ns && fits; b = next++) {
            SlabPlan& P = plan[b];
            const uint32_t m = (uint32_t)P.pos.size(), r0 = start[b], r1 = start[b + 1];
            seen.start();
            uint32_t longest = 0, used = m + 1;
            auto close = [&]() { P.chunks.push_back(std::max(1u, (longest + Q * E - 1) / (Q * E))); };
            for (uint32_t i = 0; i < m && used <= max_slots; ++i) {
                const uint32_t p = P.pos[i];
                const bool opens = i == 0 || s.level[s.order[p]] != s.level[s.order[P.pos[i - 1]]];
                if (opens || i - P.task.back() == kFlowRows) {
                    if (i) close();
                    if (opens) P.level.push_back((uint32_t)P.task.size());
                    P.task.push_back(i);
                    longest = 0;
                }
                uint32_t own = 0;
                for (uint32_t k = s.rowptr[p]; k < s.rowptr[p + 1]; ++k) {
                    const uint32_t c = s.col[k];
                    if (c >= r0 && c < r1) {
                        ++own;
                    } else if (used <= max_slots && seen.put(c, used) == used) {
                        P.halo.push_back({c, used++});
                        pub[c].store(1, std::memory_order_relaxed);
                    }
                }
                longest = std::max(longest, s.rowptr[p + 1] - s.rowptr[p] - std::min(own, kFlowTail));
            }
            if (used > max_slots) {
                fits = false;
                return;
            }
            close();
            P.level.push_back((uint32_t)P.task.size());
            P.task.push_back(m);
            uint32_t cur = most.load();
            while (cur < used && !most.compare_exchange_weak(cur, used)) {
            }
            // values arrive by level
            std::sort(P.halo.begin(), P.halo.end(), [&](const auto& x, const auto& y) {
                return s.level[x.first] != s.level[y.first] ? s.level[x.first] < s.level[y.first] : x.first < y.first;
            });
            for (uint32_t c : P.chunks)
                if (c > 0xFFu) fits = false;
            P.up.reserve(P.halo.size());
            for (const auto& h : P.halo)
                if (P.up.empty() || P.up.back() != owner[h.first]) P.up.push_back(owner[h.first]);
            std::sort(P.up.begin(), P.up.end());
            P.up.erase(std::unique(P.up.begin(), P.up.end()), P.up.end());
        }
    });
    if (!fits) return false;
    // Slabs from upstream to downstream, by their depth in the graph of slabs: independent
    // blocks advance side by side where a CTA takes several slabs.
    std::vector<uint32_t> range_of(ns);  // slab number -> its rows' range in `start`
    {
        std::vector<uint32_t> depth(ns, 0);
        for (uint32_t i = 0; i < ns; ++i) {
            const uint32_t b = s.lower ? i : ns - 1 - i;
            for (uint32_t u : plan[b].up) depth[b] = std::max(depth[b], depth[u] + 1);
            range_of[i] = b;
        }
        std::stable_sort(range_of.begin(), range_of.end(),
                         [&](uint32_t x, uint32_t y) { return depth[x] < depth[y]; });
        std::vector<SlabPlan> sorted(ns);
        for (uint32_t i = 0; i < ns; ++i) sorted[i] = std::move(plan[range_of[i]]);
        plan.swap(sorted);
    }
    out.slots = most;
    // exchange entries, in the order the rows are computed
    std::vector<uint32_t> entry(n, kFlowNone);
    for (const SlabPlan& P : plan)
        for (uint32_t p : P.pos)
            if (pub[s.order[p]].load(std::memory_order_relaxed)) entry[s.order[p]] = out.published++;
    // where each worker's tasks and chunks start
    out.warp.assign((size_t)ns * kFlowWorkers * 8, 0);
    out.halo_ptr.assign((size_t)ns + 1, 0);
    uint64_t chunk = 0, bytes = 0;
    for (uint32_t b = 0; b < ns; ++b) {
        const SlabPlan& P = plan[b];
        const uint32_t nt = (uint32_t)P.chunks.size();
        for (uint32_t w = 0; w < kFlowWorkers; ++w) {
            uint32_t* q = &out.warp[((size_t)b * kFlowWorkers + w) * 8];
            q[1] = out.tasks;
            q[4] = (uint32_t)(bytes / 16);
            for (uint32_t t = w; t < nt; t += kFlowWorkers) {
                const uint32_t m = P.task[t + 1] - P.task[t];
                ++q[2];
                q[3] += P.chunks[t];
                bytes += (uint64_t)P.chunks[t] * m * RB + tail_bytes(m);
            }
            q[5] = (uint32_t)(bytes / 16) - q[4];
            out.tasks += q[2];
            chunk += q[3];
        }
        out.halo_ptr[b + 1] = out.halo_ptr[b] + (uint32_t)P.halo.size();
    }
    if (chunk > 0xFFFFFFFFull || bytes / vb > 0xFFFFFFFFull) return false;  // u32 positions (coef_map)
    out.chunks.alloc(bytes);
    out.hdr.assign((size_t)out.tasks * kFlowRows * 4, 0);
    out.dg.assign((size_t)out.tasks * kFlowRows, 1.0);
    out.dg_pos.assign(n, 0);
    out.halo.assign((size_t)out.halo_ptr[ns] * 2, 0);
    std::vector<uint32_t> eptr;
    if (order) {
        order->eptr.assign((size_t)n + 1, 0);
        order->kptr.assign((size_t)n + 1, 0);
        for (uint32_t r = 0; r <= n; ++r) order->kptr[r] = r * kFlowTail;
        order->kdep.assign((size_t)n * kFlowTail, kFlowNone);
        order->kcoef.assign((size_t)n * kFlowTail, 0.0);
        order->diag.assign(n, 1.0);
        for (uint32_t p = 0; p < n; ++p) order->diag[s.order[p]] = s.diag[p];
        order->op = s.op;
        order->lower = s.lower;
        for (const SlabPlan& P : plan)
            for (size_t t = 0; t < P.chunks.size(); ++t)
                for (uint32_t i = P.task[t]; i < P.task[t + 1]; ++i)
                    order->eptr[s.order[P.pos[i]] + 1] = P.chunks[t] * Q * E;
        for (uint32_t r = 0; r < n; ++r) order->eptr[r + 1] += order->eptr[r];
        order->edep.assign(order->eptr[n], kFlowNone);
        order->ecoef.assign(order->eptr[n], 0.0);
    }
    if (coef_map) coef_map->assign(s.val.size() * 2, 0);
    auto lay = [&](uint32_t b, HaloSlots& hs, std::vector<Item>& it) {
        const SlabPlan& P = plan[b];
        const uint32_t r0 = start[range_of[b]], r1 = start[range_of[b] + 1];
        hs.start();
        for (size_t i = 0; i < P.halo.size(); ++i) {
            hs.put(P.halo[i].first, P.halo[i].second);
            out.halo[2 * (out.halo_ptr[b] + i)] = entry[P.halo[i].first];
            out.halo[2 * (out.halo_ptr[b] + i) + 1] = P.halo[i].second;
        }
        // the workers of each level, as bits; the level and barrier counts of each task
        const uint32_t nl = (uint32_t)P.level.size() - 1;
        std::vector<uint32_t> who(nl + 1, 0), meet((size_t)P.chunks.size(), 0), lev(P.chunks.size());
        for (uint32_t l = 0; l < nl; ++l)
            for (uint32_t t = P.level[l]; t < P.level[l + 1]; ++t) who[l] |= 1u << t % kFlowWorkers, lev[t] = l;
        for (uint32_t l = 0; l < nl; ++l)
            for (uint32_t t = P.level[l]; t < P.level[l + 1]; ++t) {
                const uint32_t w = 1u << t % kFlowWorkers;
                if (l > 0 && t < P.level[l] + kFlowWorkers) meet[t] |= (uint32_t)__builtin_popcount(who[l - 1] | who[l]) << 17;
                if (l + 1 < nl && t + kFlowWorkers >= P.level[l + 1] && !(who[l + 1] & w))
                    meet[t] |= (uint32_t)__builtin_popcount(who[l] | who[l + 1]) << 22;
            }
        for (uint32_t w = 0; w < kFlowWorkers; ++w) {
            const uint32_t* q = &out.warp[((size_t)b * kFlowWorkers + w) * 8];
            uint64_t start16 = (uint64_t)q[4] * 16;
            if (q[5]) std::memset(&out.chunks[start16], 0, (size_t)q[5] * 16);
            uint32_t task = q[1];
            for (size_t t = w; t < P.chunks.size(); t += kFlowWorkers, ++task) {
                const uint32_t nc = P.chunks[t], m = P.task[t + 1] - P.task[t];
                const size_t tn = t + kFlowWorkers;
                const uint32_t mn = tn < P.chunks.size() ? P.task[tn + 1] - P.task[tn] : 0u;
                for (uint32_t j8 = 0; j8 < kFlowRows; ++j8) {
                    uint32_t* h = &out.hdr[((size_t)task * kFlowRows + j8) * 4];
                    h[0] = h[1] = kFlowNone;
                    h[2] = (1 + lev[t] % kFlowBars) << 16;
                    h[3] = nc | m << 8 | mn << 12 | meet[t];
                    const uint32_t i = P.task[t] + j8;
                    if (i >= P.task[t + 1]) continue;
                    const uint32_t p = P.pos[i], r = s.order[p];
                    h[0] = r;
                    h[1] = entry[r];
                    h[2] |= slot[r];
                    const double d = s.op == SWEEP_NONE ? 1.0 : s.diag[p];
                    out.dg[(size_t)task * kFlowRows + j8] = recip ? 1.0 / d : d;
                    out.dg_pos[r] = task * kFlowRows + j8;
                    it.clear();
                    for (uint32_t k = s.rowptr[p]; k < s.rowptr[p + 1]; ++k) {
                        const uint32_t c = s.col[k];
                        const bool own = c >= r0 && c < r1;
                        it.push_back({(uint64_t)(s.level[c] + (own ? 0u : kFlowHaloLag)) << 32 | c, k,
                                      own ? slot[c] : hs.put(c, 0)});
                    }
                    std::sort(it.begin(), it.end(),
                              [](const Item& x, const Item& y) { return x.key != y.key ? x.key < y.key : x.k < y.k; });
                    // the latest rows of the slab to the end, the others' order kept
                    const uint32_t all = (uint32_t)it.size();
                    uint32_t tail = 0;
                    Item last[kFlowTail];
                    uint32_t to = all;  // where the entries kept are moved to, from the end
                    for (uint32_t j = all; j-- > 0;) {
                        const uint32_t c = (uint32_t)it[j].key;
                        if (tail < kFlowTail && c >= r0 && c < r1) last[tail++] = it[j];
                        else it[--to] = it[j];
                    }
                    // entries [to, all) are the front now; to == tail
                    const uint32_t front = all - tail;
                    for (uint32_t j = 0; j < all; ++j) {
                        const Item& en = j < front ? it[tail + j] : last[all - 1 - j];
                        const uint32_t dep = (uint32_t)en.key;
                        const uint16_t sl = (uint16_t)en.slot;
                        uint64_t at;  // where the coefficient goes
                        if (j < front) {
                            // position, its lane, chunk and place in the chunk
                            const uint32_t e = Q * nc * E - (front - j);
                            const uint32_t lane = j8 * Q + e % Q, ch = e / Q / E, c = e / Q % E;
                            const uint64_t base = start16 + (uint64_t)ch * m * RB;
                            std::memcpy(&out.chunks[base + (lane * E + c) * 2], &sl, 2);
                            at = base + 2 * E * Q * m + (uint64_t)(c * vb / 16) * 16 * Q * m + lane * 16 + c * vb % 16;
                            if (order) {
                                order->edep[order->eptr[r] + e] = dep;
                                order->ecoef[order->eptr[r] + e] = (double)s.val[en.k];
                            }
                        } else {
                            const uint32_t c = kFlowTail - (all - j);
                            const uint64_t base = start16 + (uint64_t)nc * m * RB;
                            std::memcpy(&out.chunks[base + 4 * vb * m + j8 * 8 + c * 2], &sl, 2);
                            at = base + (uint64_t)(c * vb / 16) * 16 * m + j8 * 16 + c * vb % 16;
                            if (order) {
                                order->kdep[r * kFlowTail + c] = dep;
                                order->kcoef[r * kFlowTail + c] = (double)s.val[en.k];
                            }
                        }
                        std::memcpy(&out.chunks[at], &s.val[en.k], vb);
                        if (coef_map) {
                            (*coef_map)[2 * (size_t)en.k] = (uint32_t)(at / vb);
                            (*coef_map)[2 * (size_t)en.k + 1] = en.k;
                        }
                    }
                }
                start16 += (uint64_t)nc * m * RB + tail_bytes(m);
            }
        }
    };
    next = 0;
    host_parallel_for(T, T, [&](uint32_t) {
        HaloSlots hs;
        std::vector<Item> it;
        for (uint32_t b = next++; b < ns; b = next++) lay(b, hs, it);
    });
    return true;
}
template bool flow_layout<double>(const Sweep<double>&, const std::vector<uint32_t>&, uint32_t, FlowLayout&,
                                  StreamOrder*, std::vector<uint32_t>*, uint32_t);
template bool flow_layout<float>(const Sweep<float>&, const std::vector<uint32_t>&, uint32_t, FlowLayout&,
                                 StreamOrder*, std::vector<uint32_t>*, uint32_t);

namespace {
template <typename Low, typename Acc>
std::string flow_replay(const Sweep<Low>& s, const FlowLayout& L, const double* in, double* out) {
    constexpr uint32_t vb = (uint32_t)sizeof(Low), Q = kFlowLanes;
    const uint32_t E = L.entries, RB = Q * E * (2 + vb);
    if (L.warp.size() != (size_t)L.slabs * kFlowWorkers * 8 || L.halo_ptr.size() != (size_t)L.slabs + 1 ||
        L.hdr.size() != (size_t)L.tasks * kFlowRows * 4 || L.dg.size() != (size_t)L.tasks * kFlowRows ||
        L.halo.size() != 2 * (size_t)L.halo_ptr[L.slabs])
        return "array sizes";
    std::vector<Acc> xch(L.published);
    std::vector<char> sent(L.published, 0), done(s.n, 0);
    for (uint32_t b = 0; b < L.slabs; ++b) {
        std::vector<Acc> xs(L.slots, (Acc)0);
        std::vector<char> ready(L.slots, 0);
        ready[0] = 1;
        for (uint32_t i = L.halo_ptr[b]; i < L.halo_ptr[b + 1]; ++i) {
            const uint32_t e = L.halo[2 * i], sl = L.halo[2 * i + 1];
            if (e >= L.published || sl >= L.slots || !sent[e] || ready[sl]) return "halo entry";
            xs[sl] = xch[e];
            ready[sl] = 1;
        }
        uint32_t next[kFlowWorkers] = {};   // tasks done
        uint64_t chunk[kFlowWorkers] = {}, at[kFlowWorkers] = {};  // chunks, bytes read
        // named barriers: workers met so far, workers expected, times opened
        uint32_t met[16] = {}, want[16] = {};
        uint64_t done_of[16] = {}, target[kFlowWorkers] = {};
        auto meet = [&](uint32_t id, uint32_t count, uint64_t& until) {
            if (id < 1 || id > kFlowBars || count > kFlowWorkers) return false;
            if (met[id] == 0) want[id] = count;
            if (want[id] != count) return false;
            until = done_of[id] + 1;
            if (++met[id] == count) ++done_of[id], met[id] = 0;
            return true;
        };
        bool moved = true;
        while (moved) {
            moved = false;
            for (uint32_t w = 0; w < kFlowWorkers; ++w) {
                const uint32_t* q = &L.warp[((size_t)b * kFlowWorkers + w) * 8];
                if (next[w] == q[2]) continue;
                const uint32_t task = q[1] + next[w];
                if (task >= L.tasks) return "task index";
                const uint32_t hw = L.hdr[(size_t)task * kFlowRows * 4 + 3], nc = hw & 0xFFu, m = hw >> 8 & 15u;
                const uint32_t id = L.hdr[(size_t)task * kFlowRows * 4 + 2] >> 16;
                const uint64_t a0 = (uint64_t)q[4] * 16 + at[w];
                if (nc == 0 || m == 0 || m > kFlowRows || chunk[w] + nc > q[3] ||
                    a0 + (uint64_t)nc * m * RB + flow_tail_bytes(m, vb) > L.chunks.size())
                    return "chunk index";
                auto slot_of = [&](uint32_t c, uint32_t lane, uint32_t p) {
                    uint16_t sl;
                    std::memcpy(&sl, &L.chunks[a0 + (uint64_t)c * m * RB + (lane * E + p) * 2], 2);
                    return (uint32_t)sl;
                };
                // the front positions await their values; the tail is read when the barrier opens
                bool all = true;
                for (uint32_t c = 0; c < nc; ++c)
                    for (uint32_t t = 0; t < Q * m * E; ++t) {
                        const uint32_t sl = slot_of(c, t / E, t % E);
                        if (sl >= L.slots) return "value slot";
                        all = all && ready[sl];
                    }
                if (!all) continue;
                const uint32_t sync = hw >> 17 & 31u, arrive = hw >> 22;
                if (sync != 0 && target[w] == 0) {
                    if (!meet(id, sync, target[w])) return "barrier count";
                    moved = true;
                }
                if (sync != 0 && done_of[id] < target[w]) continue;
                auto tail_of = [&](uint32_t j8, uint32_t p) {
                    uint16_t sl;
                    std::memcpy(&sl, &L.chunks[a0 + (uint64_t)nc * m * RB + 4 * vb * m + j8 * 8 + p * 2], 2);
                    return (uint32_t)sl;
                };
                for (uint32_t t = 0; t < m * kFlowTail; ++t) {
                    const uint32_t sl = tail_of(t / kFlowTail, t % kFlowTail);
                    if (sl >= L.slots || !ready[sl]) return "a tail value that the barrier does not cover";
                }
                Acc res[kFlowRows];
                for (uint32_t j8 = 0; j8 < kFlowRows; ++j8) {
                    const uint32_t* h = &L.hdr[((size_t)task * kFlowRows + j8) * 4];
                    if (h[3] != hw || h[2] >> 16 != id || (h[0] == kFlowNone) != (j8 >= m)) return "task header";
                    if (h[0] == kFlowNone) continue;
                    Acc c[4] = {0, 0, 0, 0};
                    for (uint32_t e = 0; e < Q * nc * E; ++e) {
                        const uint32_t lane = j8 * Q + e % Q, ch = e / Q / E, p = e / Q % E;
                        Low cf;
                        std::memcpy(&cf, &L.chunks[a0 + (uint64_t)ch * m * RB + 2 * E * Q * m + (uint64_t)(p * vb / 16) * 16 * Q * m + lane * 16 + p * vb % 16], vb);
                        c[e & 3] = std::fma((Acc)cf, xs[slot_of(ch, lane, p)], c[e & 3]);
                    }
                    if (h[0] >= s.n || done[h[0]]) return "row";
                    Acc sum = (c[0] + c[1]) + (c[2] + c[3]);
                    for (uint32_t p = 0; p < kFlowTail; ++p) {
                        Low cf;
                        std::memcpy(&cf, &L.chunks[a0 + (uint64_t)nc * m * RB + (uint64_t)(p * vb / 16) * 16 * m + j8 * 16 + p * vb % 16], vb);
                        sum = std::fma((Acc)cf, xs[tail_of(j8, p)], sum);
                    }
                    const Acc v = (Acc)in[h[0]];
                    const Acc d = (Acc)L.dg[(size_t)task * kFlowRows + j8];
                    res[j8] = s.op == SWEEP_NONE ? v - sum : s.op == SWEEP_PREDIV ? v * d - sum : (v - sum) * d;
                }
                for (uint32_t j8 = 0; j8 < kFlowRows; ++j8) {
                    const uint32_t* h = &L.hdr[((size_t)task * kFlowRows + j8) * 4];
                    if (h[0] == kFlowNone) continue;
                    const uint32_t sl = h[2] & 0xFFFFu;
                    if (sl >= L.slots || ready[sl]) return "result slot";
                    xs[sl] = res[j8];
                    ready[sl] = 1;
                    done[h[0]] = 1;
                    out[h[0]] = (double)res[j8];
                    if (h[1] != kFlowNone) {
                        if (h[1] >= L.published || sent[h[1]]) return "exchange entry";
                        xch[h[1]] = res[j8];
                        sent[h[1]] = 1;
                    }
                }
                if (arrive != 0) {
                    uint64_t unused;
                    if (!meet(id == kFlowBars ? 1 : id + 1, arrive, unused)) return "barrier count";
                }
                target[w] = 0;
                ++next[w];
                if (next[w] < q[2]) {
                    const uint32_t nw = L.hdr[(size_t)(task + 1) * kFlowRows * 4 + 3];
                    if ((hw >> 12 & 15u) != (nw >> 8 & 15u)) return "next task";
                }
                chunk[w] += nc;
                at[w] += (uint64_t)nc * m * RB + flow_tail_bytes(m, vb);
                moved = true;
            }
        }
        for (uint32_t w = 0; w < kFlowWorkers; ++w)
            if (next[w] != L.warp[((size_t)b * kFlowWorkers + w) * 8 + 2]) return "a task that never becomes ready";
        for (uint32_t i = 0; i < 16; ++i)
            if (met[i] != 0) return "a barrier left open";
    }
    for (char d : done)
        if (!d) return "a row that is not computed";
    return "";
}
}  // namespace

template <typename Low>
std::string flow_layout_replay(const Sweep<Low>& s, const FlowLayout& L, bool acc32, const double* in, double* out) {
    return acc32 ? flow_replay<Low, float>(s, L, in, out) : flow_replay<Low, double>(s, L, in, out);
}
template std::string flow_layout_replay<double>(const Sweep<double>&, const FlowLayout&, bool, const double*, double*);
template std::string flow_layout_replay<float>(const Sweep<float>&, const FlowLayout&, bool, const double*, double*);

}  // namespace prism
