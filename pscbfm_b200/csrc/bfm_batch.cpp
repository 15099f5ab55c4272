// Batch: many independent systems advanced together on one GPU.
//
// Systems whose lattices (and, in the bond-code representation, packed coordinates and bond
// codes) fit one CTA's shared memory run in the resident kernel, one CTA per system; where such systems
// leave SMs idle, the largest of them run on clusters of CTAs (planClusters).
// Larger systems of the bond-code representation run in the slab sweep, each on CTAs of its
// own, several systems in one cooperative launch (plan_slab_waves; runs of few MCS take the grid phase where
// the launches' loading of the slots would take longer). A launch of these kernels runs up to
// kLaunchSteps sub-steps. What fits neither shares the grid-phase kernels: one check and one perform launch per
// sub-step and representation cover the active colour group of every such system at once, and
// chunks of those launches are captured into a CUDA graph once and replayed. Each system draws its
// own sub-steps from its own stream exactly as it would alone, so its trajectory is unchanged by
// batching.
//
// A run stages the members' streams, and the step entries that no kernel makes from them (grid-phase
// members, callbacks), with one host-to-device copy; the resident
// and the grid-phase launches then proceed on two streams without meeting until the run ends, and
// the host returns as soon as the work is queued. The slab sweeps run on a stream of
// their own, each group of clusters on another. Member streams are ordered before the run and
// after it with events, never with host waits.

#include <algorithm>
#include <atomic>
#include <cstring>
#include <stdexcept>

#include "bfm_engine.hpp"

namespace bfm {

namespace {
constexpr double kClusterGain = 0.9;      // clusters are taken for at least a tenth of a batch's time
constexpr uint32_t kBatchChunk = 64;      // sub-steps per captured graph of the grid phase
constexpr uint32_t kCalmRuns = 8;         // runs beside fewer others before a batch's share of the SMs grows
size_t up256(size_t v) { return (v + 255) & ~size_t(255); }
}  // namespace

Batch::Batch(int gpu, Updater* const* members, uint32_t n) : gpu_(gpu)
{
    validateMembers(members, n);
    members_.assign(members, members + n);
    cuda_check(cudaSetDevice(gpu_), "cudaSetDevice");
    cuda_check(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate");
    cuda_check(cudaStreamCreateWithFlags(&stream2_, cudaStreamNonBlocking), "cudaStreamCreate");
    for (cudaEvent_t* e : {&join_, &fork_, &stepsFree_, &done_, &ready_})
        cuda_check(cudaEventCreateWithFlags(e, cudaEventDisableTiming), "cudaEventCreate");
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, gpu_) == cudaSuccess && sms > 0)
        smCount_ = slabSms_ = share_ = (uint32_t)sms;
}

Batch::~Batch()
{
    SweepUsers::end(gpu_, this);
    cudaSetDevice(gpu_);
    if (stream_) cudaStreamSynchronize(stream_);
    if (stream2_) cudaStreamSynchronize(stream2_);
    for (Side const& q : side_) cudaStreamSynchronize(q.stream);
    if (graph_) cudaGraphExecDestroy(graph_);
    if (arena_) cudaFreeAsync(arena_, stream_);
    if (dStepsAll_) cudaFreeAsync(dStepsAll_, stream_);
    if (stream_) cudaStreamSynchronize(stream_);
    cudaFreeHost(hSteps_);
    for (cudaEvent_t e : {join_, fork_, stepsFree_, done_, ready_})
        if (e) cudaEventDestroy(e);
    for (Side const& q : side_) {
        if (q.join) cudaEventDestroy(q.join);
        cudaStreamDestroy(q.stream);
    }
    if (stream_) cudaStreamDestroy(stream_);
    if (stream2_) cudaStreamDestroy(stream2_);
}

uint32_t Batch::residentCount() const
{
    uint32_t n = 0;
    for (auto const& g : resident_) n += (uint32_t)g.members.size();
    return n;
}

uint32_t Batch::clusterCount() const
{
    uint32_t n = 0;
    for (auto const& w : slab_)
        for (SlabRef const& r : w.refs) n += r.rank == 0 ? 1u : 0u;
    for (auto const& g : cluster_) n += (uint32_t)g.members.size();
    return n;
}

void Batch::setMembers(Updater* const* members, uint32_t n)
{
    validateMembers(members, n);
    members_.assign(members, members + n);
    built_ = false;
}

void Batch::validateMembers(Updater* const* members, uint32_t n) const
{
    if (n == 0) throw std::invalid_argument("[Batch] no systems");
    for (uint32_t i = 0; i < n; ++i) {
        Updater* u = members[i];
        if (!u) throw std::invalid_argument("[Batch] null system");
        if (!u->initialized()) throw std::runtime_error("[Batch] every system must be initialized");
        if (u->gpu() != gpu_) throw std::invalid_argument("[Batch] every system must live on the batch GPU");
        for (uint32_t j = 0; j < i; ++j)
            if (members[j] == u) throw std::invalid_argument("[Batch] a system appears twice");
    }
}

void Batch::rebuild()
{
    // the previous launches may still read the arena
    cuda_check(cudaStreamSynchronize(stream_), "batch");
    cuda_check(cudaStreamSynchronize(stream2_), "batch");
    for (Side const& q : side_) cuda_check(cudaStreamSynchronize(q.stream), "batch");
    uint32_t const M = (uint32_t)members_.size();
    grid_.clear();
    resident_.clear();
    wholeRun_.assign(M, 0);
    auto gridGroup = [&](uint32_t mode) -> GridGroup& {
        for (auto& g : grid_)
            if (g.codeMode == mode) return g;
        grid_.push_back(GridGroup{mode, {}, nullptr, {}, nullptr, {}});
        return grid_.back();
    };
    auto resGroup = [&](uint32_t mode) -> ResidentGroup& {
        for (auto& g : resident_)
            if (g.codeMode == mode) return g;
        resident_.push_back(ResidentGroup{mode, {}, nullptr, 1, 0});
        return resident_.back();
    };
    SlabWaves plan = planSlabs();
    slab_.swap(plan.waves);
    residentsAfter_ = plan.residentsAfter;
    leastMcs_ = plan.leastMcs;
    shortMembers_ = false;
    std::vector<char> const slabbed = std::move(plan.taken);
    std::vector<char> clustered;
    cluster_ = planClusters(clustered);
    sides_ = std::max<size_t>(cluster_.size(), slab_.empty() ? 0 : 1);
    while (side_.size() < sides_) {   // kept from one plan to the next
        cudaStream_t q = nullptr;
        cuda_check(cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking), "cudaStreamCreate");
        side_.push_back(Side{q, nullptr});
        cuda_check(cudaEventCreateWithFlags(&side_.back().join, cudaEventDisableTiming), "cudaEventCreate");
    }
    bool faulted = false;   // a report belongs to the member it was made for: kept by it, not reused
    for (uint32_t m = 0; m < reportCap_; ++m) faulted = faulted || reports_.get()[m].fault != 0u;
    if (!slab_.empty() && (M > reportCap_ || faulted)) {
        void* p = nullptr;
        void* d = nullptr;
        cuda_check(cudaHostAlloc(&p, sizeof(GridFault) * M, cudaHostAllocMapped), "cudaHostAlloc(reports)");
        std::memset(p, 0, sizeof(GridFault) * M);
        reports_ = std::shared_ptr<GridFault>(static_cast<GridFault*>(p), [](GridFault* q) { cudaFreeHost(q); });
        cuda_check(cudaHostGetDevicePointer(&d, p, 0), "reports device address");
        dReports_ = static_cast<GridFault*>(d);
        reportCap_ = M;
    }
    for (uint32_t m = 0; m < M; ++m) {
        Updater* u = members_[m];
        if (clustered[m]) {
            wholeRun_[m] = 1;
        } else if (residentOn_ && u->residentEligible()) {
            ResidentGroup& g = resGroup(u->codeMode());
            g.members.push_back(m);
            g.smem = std::max(g.smem, u->residentSmem());
            while (g.perThread * kResidentBlock < u->maxGroup()) g.perThread *= 2;
            wholeRun_[m] = 1;
        } else if (slabbed[m]) {
            wholeRun_[m] = 1;
        } else {
            GridGroup& g = gridGroup(u->codeMode());
            uint32_t const span = u->codeMode() == kCodeNone ? kGridBlock : kBcTileSpan;
            uint32_t const t = u->gridTiles();
            for (uint32_t k = 0; k < t; ++k) g.tiles.push_back(TileRef{m, k * span});
            g.members.push_back(m);
        }
    }
    for (auto& g : grid_) g.ptiles = g.codeMode == kCodeNone ? g.tiles : perform_tile_list(g.tiles);
    stepCap_ = kBatchChunk;
    size_t total = up256(sizeof(SysDev) * M) + up256(sizeof(StepEntry) * stepCap_ * M);
    for (auto const& g : grid_) total += up256(sizeof(TileRef) * g.tiles.size()) + up256(sizeof(TileRef) * g.ptiles.size());
    for (auto const& g : resident_) total += up256(sizeof(uint32_t) * g.members.size());
    for (auto const& w : slab_) total += up256(sizeof(SlabRef) * w.refs.size());
    for (auto const& g : cluster_) total += up256(sizeof(uint32_t) * g.members.size());
    if (total > arenaBytes_) {   // grows only: membership changes reuse the arena
        if (arena_) cuda_check(cudaFreeAsync(arena_, stream_), "cudaFreeAsync(batch)");
        arena_ = nullptr;
        arenaBytes_ = 0;
        cuda_check(cudaMallocAsync(&arena_, total * 2, stream_), "cudaMallocAsync(batch)");
        arenaBytes_ = total * 2;
    }
    char* p = static_cast<char*>(arena_);
    dSys_ = reinterpret_cast<SysDev*>(p);
    p += up256(sizeof(SysDev) * M);
    dWindow_ = reinterpret_cast<StepEntry*>(p);
    p += up256(sizeof(StepEntry) * stepCap_ * M);
    std::vector<SysDev> descs(M);
    for (uint32_t m = 0; m < M; ++m) descs[m] = members_[m]->desc();
    cuda_check(cudaMemcpyAsync(dSys_, descs.data(), sizeof(SysDev) * M, cudaMemcpyHostToDevice, stream_),
               "upload descriptors");
    for (auto& g : grid_) {
        g.dTiles = reinterpret_cast<TileRef*>(p);
        p += up256(sizeof(TileRef) * g.tiles.size());
        cuda_check(cudaMemcpyAsync(g.dTiles, g.tiles.data(), sizeof(TileRef) * g.tiles.size(), cudaMemcpyHostToDevice,
                                   stream_),
                   "upload tiles");
        g.dPTiles = reinterpret_cast<TileRef*>(p);
        p += up256(sizeof(TileRef) * g.ptiles.size());
        cuda_check(cudaMemcpyAsync(g.dPTiles, g.ptiles.data(), sizeof(TileRef) * g.ptiles.size(),
                                   cudaMemcpyHostToDevice, stream_),
                   "upload perform tiles");
    }
    for (auto& g : resident_) {
        g.dList = reinterpret_cast<uint32_t*>(p);
        p += up256(sizeof(uint32_t) * g.members.size());
        cuda_check(cudaMemcpyAsync(g.dList, g.members.data(), sizeof(uint32_t) * g.members.size(),
                                   cudaMemcpyHostToDevice, stream_),
                   "upload resident list");
    }
    for (auto& w : slab_) {
        w.dRefs = reinterpret_cast<SlabRef*>(p);
        p += up256(sizeof(SlabRef) * w.refs.size());
        cuda_check(cudaMemcpyAsync(w.dRefs, w.refs.data(), sizeof(SlabRef) * w.refs.size(), cudaMemcpyHostToDevice,
                                   stream_),
                   "upload slab CTAs");
    }
    for (auto& g : cluster_) {
        g.dList = reinterpret_cast<uint32_t*>(p);
        p += up256(sizeof(uint32_t) * g.members.size());
        cuda_check(cudaMemcpyAsync(g.dList, g.members.data(), sizeof(uint32_t) * g.members.size(),
                                   cudaMemcpyHostToDevice, stream_),
                   "upload cluster list");
    }
    // the host vectors above die with this call: finish their copies now
    cuda_check(cudaStreamSynchronize(stream_), "batch uploads");
    if (graph_) {
        cudaGraphExecDestroy(graph_);
        graph_ = nullptr;
    }
    built_ = true;
}

namespace {
// The fewest of at most `most` CTAs that hold the member in the slab sweep, and how; false: it does not fit.
template <typename Plan>
bool slab_least(Plan const& plan, uint32_t most, SlabPlan& out)
{
    for (uint32_t C = 1; C <= most; ++C)
        if (plan(C, out) && out.cache) return true;
    return false;
}
}  // namespace

bool Batch::slabFits(Updater const& u) const
{
    SlabPlan plan;
    return slab_least([&](uint32_t C, SlabPlan& p) { return u.slabPlan(C, p); }, std::min(smCount_ / 2u, slabSms_), plan);
}

SlabWaves plan_slab_waves(std::vector<SlabMember> const& members, uint32_t sms, uint32_t share, uint32_t most)
{
    // The members in the slab sweep (taken) and their CTAs, in cooperative launches of at most `budget` CTAs
    // that run one after the other. Each CTA takes an SM, so the fewest CTAs that hold a member do the most
    // work per SM (moves per us and SM at 0.9K, 1.9K, 3.7K and 7.5K slots per CTA and colour: 208, 331, 419
    // and 458); members are packed by those, longest first. The SMs a wave leaves idle then go, one by one,
    // to its member with the most slots per CTA, which runs longest. A member the grid-phase kernels
    // have to take anyway (it does not fit the budget, or gathers) keeps half of the SMs.
    SlabWaves out;
    out.taken.assign(members.size(), 0);
    uint32_t residents = 0;
    for (SlabMember const& m : members) residents += m.resident ? 1u : 0u;
    // A cooperative launch waits until all its CTAs have found an SM, so it must never queue behind the
    // batch's own resident kernels, which keep theirs for the whole run: a few residents get SMs of
    // their own, many run after the slab sweeps.
    bool const residentsAfter = residents > share / 4u;
    struct Item {
        uint32_t m;
        SlabPlan plan;
    };
    std::vector<Item> items;
    bool gridAnyway = false;
    uint32_t budget = 0;
    for (;;) {   // a member that does not fit leaves the others half of the SMs, which one more may not fit
        budget = std::max(1u, gridAnyway ? share / 2u : share - (residentsAfter ? 0u : residents));
        bool const before = gridAnyway;
        items.clear();
        for (uint32_t m = 0; m < (uint32_t)members.size(); ++m) {
            if (members[m].resident) continue;
            Item it{m, {}};
            if (slab_least(members[m].plan, std::min(budget, sms / 2u), it.plan)) items.push_back(it);
            else gridAnyway = true;
        }
        if (gridAnyway == before) break;
    }
    out.residentsAfter = residentsAfter;
    std::stable_sort(items.begin(), items.end(),
                     [&](Item const& a, Item const& b) { return members[a.m].monomers > members[b.m].monomers; });
    struct Wave {
        uint32_t codeMode, used = 0;
        uint64_t monomers = 0;
        std::vector<Item> items;
    };
    auto put = [&](Wave& w, Item const& it) {
        w.items.push_back(it);
        w.used += it.plan.ctas;
        w.monomers += members[it.m].monomers;
    };
    auto takes = [&](Wave const& w, Item const& it) {
        return w.codeMode == members[it.m].codeMode && w.used + it.plan.ctas <= budget;
    };
    // The idle SMs of each wave handed out; returns the waves' time in all, us per MCS: a CTA's time grows with
    // its slots per colour, and jumps where the movers of a sub-step, about an eighth, pass one per thread
    // (one wave each, 128^3 boxes, at 640, 1664, 3350, 4928 and 6048 slots: 8, 11, 17, 21 and 41).
    auto grow = [&](std::vector<Wave>& waves) {
        double time = 0.0;
        for (Wave& w : waves) {
            uint32_t slots = 0;
            for (;;) {
                Item* pick = nullptr;
                for (Item& it : w.items)
                    if (!pick || it.plan.perCta > pick->plan.perCta) pick = &it;
                slots = pick->plan.perCta;
                SlabPlan next;
                if (slots <= kSlabGrowSlots || w.used >= budget || !members[pick->m].plan(pick->plan.ctas + 1u, next) ||
                    !next.cache)
                    break;
                pick->plan = next;
                ++w.used;
            }
            time += 5.5 + 0.0033 * slots + (slots > kSlabPassSlots ? 14.0 : 0.0);
        }
        return time;
    };
    // Members by first fit, the fewest waves; or as evenly over as many waves, each member, longest first, into
    // the one of its kind with the fewest monomers: whichever takes less time. First fit fills its waves to
    // the brim and leaves little to the last (32 systems of 60K, 29 and 3, 50 us per MCS and, 16 and 16, 38;
    // 64 systems of 30K, 49 of 3 CTAs each and 15, 31 and, 32 and 32, 35).
    std::vector<Wave> first;
    for (Item const& it : items) {
        auto w = std::find_if(first.begin(), first.end(), [&](Wave const& q) { return takes(q, it); });
        if (w == first.end()) w = first.insert(w, Wave{members[it.m].codeMode});
        put(*w, it);
    }
    if (first.size() > most) {
        out.residentsAfter = false;
        return out;
    }
    std::vector<Wave> even;
    for (Wave const& w : first) even.push_back(Wave{w.codeMode});
    bool room = first.size() > 1;
    for (size_t i = 0; room && i < items.size(); ++i) {
        Wave* best = nullptr;
        for (Wave& w : even)
            if (takes(w, items[i]) && (!best || w.monomers < best->monomers)) best = &w;
        room = best != nullptr;
        if (room) put(*best, items[i]);
    }
    double const time = grow(first);
    if (room && grow(even) < time) first.swap(even);
    // A launch loads its CTAs' slots and writes them back, about 10 us per 1000 slots of a CTA and colour. us
    // of 1, 2, 4 and 6 MCS in the grid phase and in the sweeps, `load` their launches' slots: 16 x 60K (load 3350)
    // 59, 102, 180, 264 and 61, 77, 114, 153; 12 x 118K (4928) 67, 112, 200, 291 and 77, 100, 143, 188; 32 x 60K
    // (6700) 92, 154, 277, 403 and 118, 156, 225, 301; 48 x 60K (10048) 124, 211, 385, 562 and 174, 227, 322,
    // 424; 100 x 30K (10368) 138, 204, 347, 481 and 198, 248, 347, 448. Residents that run after the sweeps run
    // beside the grid phase: 64 mixed systems 145, 212, 333, 469 and 195, 248, 356, 467; 256 624, 822, 1251, 1669 and
    // 808, 961, 1266, 1565.
    uint32_t load = 0;
    for (Wave const& w : first) {
        uint32_t slots = 0;
        for (Item const& it : w.items) slots = std::max(slots, it.plan.perCta);
        load += slots;
    }
    out.leastMcs = load <= 4000u ? 1u : (load <= 9500u ? 2u : 4u) + (residentsAfter ? 2u : 0u);
    for (Wave const& w : first) {
        SlabWave wave{w.codeMode, {}, 0, nullptr};
        for (Item const& it : w.items) {
            for (uint32_t r = 0; r < it.plan.ctas; ++r) wave.refs.push_back(SlabRef{it.m, r, it.plan.ctas, 0u});
            wave.smem = std::max(wave.smem, it.plan.smem);
            out.taken[it.m] = 1;
        }
        out.waves.push_back(std::move(wave));
    }
    return out;
}

SlabWaves Batch::planSlabs() const
{
    std::vector<SlabMember> members;
    if (clusterOn_)
        for (Updater const* u : members_)
            members.push_back(SlabMember{u->nMonomers(), u->codeMode(), residentOn_ && u->residentEligible(),
                                         [u](uint32_t C, SlabPlan& p) { return u->slabPlan(C, p); }});
    SlabWaves plan = plan_slab_waves(members, smCount_, share_, slabLaunches_);
    plan.taken.resize(members_.size(), 0);
    return plan;
}

std::vector<Batch::ClusterGroup> Batch::planClusters(std::vector<char>& taken) const
{
    // A batch lasts as long as its largest member, and a member that fits one CTA takes longer there than
    // on a cluster's CTAs. The weights, us per MCS with g slots per colour, 2.9 + 0.00185 g on one CTA and
    // 4.4 + 0.0046 g / C on C, are those of lone systems on earlier forms of the kernels. A lone cluster takes
    // less now (3.7 + 0.006 g / C), but many at once take longer than one, and with that fit the plans
    // were worse (16 systems of 8K monomers 8.8 -> 11.2), so the older weights stay. Where every member fits one CTA and SMs are left over, the k largest go
    // to clusters: C and k with the least time of the longest member. Sixteen systems of 0.4K to 10.5K
    // monomers, on one CTA each, with slab sweeps on the SMs left over, and so: 14.2, 9.4 and 6.8 us per MCS;
    // 7, 9, 16, 32 and 36 systems of 8K monomers 10.8 -> 5.8, 7.2, 9.5, 9.8 and 10.9.
    uint32_t const M = (uint32_t)members_.size();
    taken.assign(M, 0);
    std::vector<ClusterGroup> groups;
    if (!clusterOn_ || !residentOn_) return groups;
    std::vector<uint32_t> order;
    for (uint32_t m = 0; m < M; ++m) {
        if (!members_[m]->residentEligible()) return groups;
        if (members_[m]->codeMode() != kCodeNone) order.push_back(m);
    }
    std::stable_sort(order.begin(), order.end(),
                     [&](uint32_t a, uint32_t b) { return members_[a]->maxGroup() > members_[b]->maxGroup(); });
    auto slots = [&](size_t k) { return k < order.size() ? (double)members_[order[k]]->maxGroup() : 0.0; };
    auto alone = [](double g) { return 2.9 + 0.00185 * g; };
    auto spread = [](double g, double C) { return 4.4 + 0.0046 * g / C; };
    double best = alone(slots(0)) * kClusterGain;
    size_t bestCount = 0;
    uint32_t bestLog = 0;
    for (uint32_t logC = 4; logC >= 2; --logC) {
        uint32_t const C = 1u << logC;
        uint32_t atOnce = ~0u;   // clusters of the batch's share of the SMs
        for (size_t k = 0; k < order.size(); ++k) {
            ClusterPlan plan;
            atOnce = std::min(atOnce, members_[order[k]]->clusterPlan(logC, plan) * share_ / smCount_);
            if (k + 1 > atOnce || (k + 1) * (C - 1u) + M > share_) break;
            double const time = std::max(spread(slots(0), C), alone(slots(k + 1)));
            if (time < best) {
                best = time;
                bestCount = k + 1;
                bestLog = logC;
            }
        }
    }
    for (size_t k = 0; k < bestCount; ++k) {
        uint32_t const m = order[k];
        Updater const& u = *members_[m];
        ClusterPlan plan;
        u.clusterPlan(bestLog, plan);
        auto g = std::find_if(groups.begin(), groups.end(), [&](ClusterGroup const& c) { return c.codeMode == u.codeMode(); });
        if (g == groups.end()) g = groups.insert(g, ClusterGroup{u.codeMode(), plan, {}, nullptr});
        // one launch has one number of chunks per warp and one size of shared memory (descending groups: the
        // first member's chunks do for all)
        size_t const smem = u.clusterSmem(bestLog, g->plan.chunks);
        if (smem > kResidentMaxSmem) continue;
        g->plan.smem = std::max(g->plan.smem, smem);
        g->members.push_back(m);
        taken[m] = 1;
    }
    return groups;
}

void Batch::setSlabLaunches(uint32_t most)
{
    if (most != slabLaunches_) built_ = false;
    slabLaunches_ = most;
}

void Batch::setSlabSms(uint32_t sms)
{
    if (sms != slabSms_) built_ = false;
    slabSms_ = share_ = sms;
    calm_ = 0;
}

void Batch::takeShare()
{
    // Beside other users of the device (SweepUsers) the plan takes their number's share of the SMs: sweeps of
    // batches in several threads then run at once instead of one after the other (us per MCS of all, 8 threads with
    // a batch each: 2 systems of 60K monomers 76 and 20, 8 of 30K 76 and 35, 4 of 8K 24 and 9; 16 of 60K 155 and
    // 171, each batch then several launches).
    // The share shrinks at once and by halves, and grows after kCalmRuns runs in which it could have: a new
    // plan costs the host what several short runs take.
    if (!clusterOn_ || slabSms_ < smCount_) return;   // (a server's lanes have their shares)
    if (built_ && slab_.empty() && cluster_.empty() && share_ == slabSms_) return;
    uint32_t parts = 1;
    for (uint32_t const n = SweepUsers::others(gpu_, this) + 1u; parts < n;) parts *= 2u;
    uint32_t const want = std::max(1u, std::min(slabSms_, smCount_ / parts));
    calm_ = want > share_ ? calm_ + 1u : 0u;
    if (want >= share_ && calm_ < kCalmRuns) return;
    share_ = want;
    calm_ = 0;
    built_ = false;
}

cudaError_t Batch::launchGrid(StepEntry const* e)
{
    SysDev const unused{};   // multi-system launches read each CTA's descriptor from dSys_
    PerformArgs pa;
    pa.warps = perfWarps_;
    pa.group = perfGroup_;
    for (auto const& g : grid_) {
        uint32_t const n = (uint32_t)g.tiles.size();
        if (g.members.size() == 1) {
            // a lone system runs the single-system kernels, as it would alone (descriptor as a launch
            // parameter, several tiles per perform CTA): a long job left alone in a server lane
            // then runs at its own speed
            uint32_t const m = g.members[0];
            Updater const& u = *members_[m];
            cudaError_t err = g.codeMode == kCodeNone
                                  ? launch_check(u.deviceDesc(), nullptr, n, kGridBlock, e + m, stream_)
                                  : launch_check_bc(u.desc(), u.deviceDesc(), nullptr, n, e + m, g.codeMode, stream_, shape_, block_);
            if (err != cudaSuccess) return err;
            err = g.codeMode == kCodeNone
                      ? launch_perform(u.deviceDesc(), nullptr, n, kGridBlock, e + m, stream_)
                      : launch_perform_bc(u.desc(), u.deviceDesc(), nullptr, n, e + m, g.codeMode, stream_, shape_, pa);
            if (err != cudaSuccess) return err;
            continue;
        }
        cudaError_t err = g.codeMode == kCodeNone
                              ? launch_check(dSys_, g.dTiles, n, kGridBlock, e, stream_)
                              : launch_check_bc(unused, dSys_, g.dTiles, n, e, g.codeMode, stream_, shape_, block_);
        if (err != cudaSuccess) return err;
        err = g.codeMode == kCodeNone
                  ? launch_perform(dSys_, g.dTiles, n, kGridBlock, e, stream_)
                  : launch_perform_bc(unused, dSys_, g.dPTiles, (uint32_t)g.ptiles.size(), e, g.codeMode, stream_, shape_, pa);
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

void Batch::reserveSteps(size_t entries)
{
    // the previous run's copy has read the host staging once stepsFree_ has passed
    cuda_check(cudaEventSynchronize(stepsFree_), "batch staging");
    if (entries > hStepsCap_) {
        cudaFreeHost(hSteps_);
        hSteps_ = nullptr;
        hStepsCap_ = 0;
        cuda_check(cudaMallocHost(&hSteps_, sizeof(StepEntry) * entries * 2), "cudaMallocHost(batch steps)");
        hStepsCap_ = entries * 2;
    }
    if (entries > dStepsCap_) {
        if (dStepsAll_) cuda_check(cudaFreeAsync(dStepsAll_, stream_), "cudaFreeAsync(batch steps)");
        dStepsAll_ = nullptr;
        dStepsCap_ = 0;
        cuda_check(cudaMallocAsync(&dStepsAll_, sizeof(StepEntry) * entries * 2, stream_),
                   "cudaMallocAsync(batch steps)");
        dStepsCap_ = entries * 2;
    }
}

void Batch::ensureGraph()
{
    if (graph_) return;
    uint32_t const M = (uint32_t)members_.size();
    cudaGraph_t g;
    cuda_check(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal), "begin capture");
    cudaError_t err = cudaSuccess;
    for (uint32_t t = 0; t < stepCap_ && err == cudaSuccess; ++t) err = launchGrid(dWindow_ + (size_t)t * M);
    cudaError_t const endErr = cudaStreamEndCapture(stream_, &g);
    cuda_check(err, "capture batch launches");
    cuda_check(endErr, "end capture");
    cudaError_t const ie = cudaGraphInstantiate(&graph_, g, 0);
    cudaGraphDestroy(g);
    cuda_check(ie, "graph instantiate");
}

bool Batch::ownEntries(uint32_t m) const
{
    // a kernel that runs all of the member's sub-steps makes their entries (bond codes, counter stream)
    return wholeRun_[m] && members_[m]->codeMode() != kCodeNone && members_[m]->countsDraws();
}

bool Batch::hostEntries() const
{
    for (uint32_t m = 0; m < (uint32_t)members_.size(); ++m)
        if (!ownEntries(m)) return true;
    return false;
}

size_t Batch::streamUnits() const
{
    return (sizeof(StepStream) * members_.size() + sizeof(StepEntry) - 1) / sizeof(StepEntry);
}

uint32_t Batch::longest(int32_t const* mcs) const
{
    uint64_t T = 0;
    for (size_t m = 0; m < members_.size(); ++m) {
        if (mcs[m] < 0) throw std::invalid_argument("[Batch::run] negative MCS count");
        T = std::max(T, (uint64_t)mcs[m] * members_[m]->nColors());
    }
    // the kernels count the sub-steps of a run in 32 bits, as Updater::run does
    if (T > 0xFFFFFFFFull) throw std::invalid_argument("[Batch::run] too many sub-steps in one call");
    return (uint32_t)T;
}

Batch* Batch::shortFor(int32_t const* mcs)
{
    if (!shortRuns_ || leastMcs_ <= 1 || slab_.empty()) return nullptr;
    for (size_t m = 0; m < members_.size(); ++m)
        if ((uint32_t)mcs[m] >= leastMcs_) return nullptr;
    if (!short_) {
        short_.reset(new Batch(gpu_, members_.data(), (uint32_t)members_.size()));
        short_->setClusterEnabled(false);
    } else if (!shortMembers_) {
        short_->setMembers(members_.data(), (uint32_t)members_.size());
    }
    shortMembers_ = true;
    short_->setResidentEnabled(residentOn_);
    short_->setShape(shape_);
    short_->setBlock(block_);
    short_->setPerformShape(perfWarps_, perfGroup_);
    return short_.get();
}

void Batch::prepare(int32_t const* mcs)
{
    // one-time host work of a run (staging growth, graph capture), done ahead of a timed run
    uint32_t const M = (uint32_t)members_.size();
    uint32_t const T = longest(mcs);
    if (T == 0) return;
    if (Batch* const b = shortFor(mcs)) {
        if (!b->built_) b->rebuild();
        b->prepare(mcs);
        return;
    }
    reserveSteps(streamUnits() + (hostEntries() ? (size_t)T * M : 0));
    if (!grid_.empty() && T >= stepCap_) ensureGraph();
}

void Batch::run(int32_t nMcs)
{
    if (nMcs <= 0) return;
    std::vector<int32_t> each(members_.size(), nMcs);
    run(each.data());
}

void Batch::run(int32_t const* mcs)
{
    uint32_t const T = longest(mcs);
    cuda_check(cudaSetDevice(gpu_), "cudaSetDevice");
    takeShare();
    if (!built_) rebuild();
    if (Batch* const b = shortFor(mcs)) {
        b->run(mcs);   // (the members' streams order it after this batch's runs and before the next)
        cuda_check(cudaStreamWaitEvent(stream_, b->done_, 0), "wait");
        return;
    }
    enqueue(mcs, T);
}

void Batch::enqueue(int32_t const* mcs, uint32_t T)
{
    uint32_t const M = (uint32_t)members_.size();
    // pending grid-path marks of members that run in a resident or cluster kernel are cleared on
    // their own streams; then the batch waits for every member stream (uploads, scrubs,
    // observables) on the device
    for (uint32_t m = 0; m < M; ++m)
        if (wholeRun_[m]) members_[m]->scrubPending(members_[m]->stream());
    for (Updater* u : members_) {
        u->endSweep();       // (this run comes after the member's own)
        u->flushTickets();   // a member's ticket still waiting for a snapshot reads its counters now
        cuda_check(cudaEventRecord(ready_, u->stream()), "event");
        cuda_check(cudaStreamWaitEvent(stream_, ready_, 0), "wait");
    }

    std::vector<uint32_t> need(M);
    for (uint32_t m = 0; m < M; ++m) need[m] = (uint32_t)mcs[m] * members_[m]->nColors();   // at most T
    if (T > 0) {
        // the members' streams, and the entries of those whose kernels don't make them
        size_t const units = streamUnits(), entries = units + (hostEntries() ? (size_t)T * M : 0);
        reserveSteps(entries);
        StepStream* const streams = reinterpret_cast<StepStream*>(hSteps_);
        StepEntry* const host = hSteps_ + units;
        std::vector<uint32_t> drawn;
        for (uint32_t m = 0; m < M; ++m) {
            streams[m] = StepStream{};
            if (!ownEntries(m) || !members_[m]->streamSteps(need[m], streams[m])) drawn.push_back(m);
        }
        // sub-step by sub-step: members may share a callback's generator
        for (uint32_t t = 0; t < T && !drawn.empty(); ++t)
            for (uint32_t m : drawn)
                host[(size_t)t * M + m] = t < need[m] ? members_[m]->nextStep()
                                                      : StepEntry{kNoColor, 0u, 0u, kNoColor, 0u, 0u, 0u, 0u};
        StepEntry const* const dEntries = dStepsAll_ + units;
        cuda_check(cudaMemcpyAsync(dStepsAll_, hSteps_, sizeof(StepEntry) * entries, cudaMemcpyHostToDevice, stream_),
                   "batch steps H2D");
        cuda_check(cudaEventRecord(stepsFree_, stream_), "event");
        if (!resident_.empty() || sides_ != 0) cuda_check(cudaEventRecord(fork_, stream_), "event");
        // a whole-run kernel's launches on one stream: launch(source, sub-steps), kLaunchSteps at a time
        auto wholeRun = [&](char const* what, auto const& launch) {
            for (uint32_t t0 = 0, n = 0; t0 < T; t0 += n) {
                n = std::min(T - t0, kLaunchSteps);
                cuda_check(launch(StepSource{dEntries + (size_t)t0 * M, reinterpret_cast<StepStream const*>(dStepsAll_),
                                             StepStream{}, M, t0},
                                  n),
                           what);
                ++launches_;
            }
        };
        for (size_t i = 0; i < sides_; ++i) {
            // a cluster group each, side by side; or all slab sweeps, one after the other
            cudaStream_t const q = side_[i].stream;
            cuda_check(cudaStreamWaitEvent(q, fork_, 0), "wait");
            if (i < cluster_.size()) {
                ClusterGroup const& g = cluster_[i];
                wholeRun("batch cluster", [&](StepSource const& src, uint32_t n) {
                    return launch_cluster_bc(dSys_, g.dList, (uint32_t)g.members.size(), g.plan.logC, g.plan.chunks,
                                             src, n, g.plan.smem, g.codeMode, q);
                });
            }
            for (size_t k = 0; i == 0 && k < slab_.size(); ++k) {
                SlabWave const& w = slab_[k];
                for (SlabRef const& r : w.refs)
                    if (r.rank == 0) members_[r.sys]->applyStall(q);
                wholeRun("batch slab", [&](StepSource const& src, uint32_t n) {
                    return launch_slab_batch(dSys_, w.dRefs, (uint32_t)w.refs.size(), w.smem, src, n, dReports_,
                                             w.codeMode, q);
                });
            }
            cuda_check(cudaEventRecord(side_[i].join, q), "event");
        }
        if (!resident_.empty()) {
            // on the second stream
            cuda_check(cudaStreamWaitEvent(stream2_, fork_, 0), "wait");
            if (!slab_.empty() && residentsAfter_) cuda_check(cudaStreamWaitEvent(stream2_, side_[0].join, 0), "wait");
            for (auto const& g : resident_)
                wholeRun("batch resident", [&](StepSource const& src, uint32_t n) {
                    return g.codeMode == kCodeNone
                               ? launch_resident(dSys_, g.dList, (uint32_t)g.members.size(), g.perThread, src.steps, M,
                                                 n, g.smem, stream2_)
                               : launch_resident_bc(dSys_, g.dList, (uint32_t)g.members.size(), g.perThread, src, n,
                                                    g.smem, g.codeMode, stream2_);
                });
        }
        if (!grid_.empty()) {
            for (uint64_t t0 = 0; t0 < T; t0 += stepCap_) {
                uint32_t const chunk = (uint32_t)std::min<uint64_t>(stepCap_, T - t0);
                if (chunk == stepCap_) {
                    // the captured graph reads its entries from the window
                    cuda_check(cudaMemcpyAsync(dWindow_, dEntries + t0 * M, sizeof(StepEntry) * stepCap_ * M,
                                               cudaMemcpyDeviceToDevice, stream_),
                               "batch window");
                    ensureGraph();
                    cuda_check(cudaGraphLaunch(graph_, stream_), "batch graph launch");
                } else {
                    for (uint32_t t = 0; t < chunk; ++t)
                        cuda_check(launchGrid(dEntries + (t0 + t) * M), "batch grid launch");
                }
                launches_ += 2ull * chunk * grid_.size();
            }
        }
        if (!resident_.empty()) {
            cuda_check(cudaEventRecord(join_, stream2_), "event");
            cuda_check(cudaStreamWaitEvent(stream_, join_, 0), "wait");
        }
        for (size_t i = 0; i < sides_; ++i) cuda_check(cudaStreamWaitEvent(stream_, side_[i].join, 0), "wait");
    }
    cuda_check(cudaEventRecord(done_, stream_), "event");
    if (sides_ != 0) SweepUsers::add(gpu_, this, done_);
    for (uint32_t m = 0; m < M; ++m) {
        members_[m]->noteExternalRun((uint64_t)mcs[m], !wholeRun_[m], members_[m]->lastColor(),
                                     slab_.empty() ? nullptr : std::shared_ptr<GridFault>(reports_, reports_.get() + m));
        members_[m]->streamWait(done_);
    }
}

void Batch::setShape(int shape)
{
    if (shape >= kGridShapes) throw std::invalid_argument("[Batch::setShape] unknown kernel shape");
    if (shape != shape_) built_ = false;   // the captured graph holds the old kernels
    shape_ = shape;
}

void Batch::setBlock(int block)
{
    if (block != 0 && !check_block_ok(block))
        throw std::invalid_argument("[Batch::setBlock] the check's CTA size must be 128, 256 or 512 threads");
    if (block != block_) built_ = false;   // the captured graph holds the old kernels
    block_ = block;
}

void Batch::setPerformShape(int warps, int group)
{
    if (!perform_shape_ok(warps, group))
        throw std::invalid_argument("[Batch::setPerformShape] warps per CTA and per tile must be 1, 2, 4 or 8, "
                                    "the second at most the first (0, 0: the default)");
    if (warps != perfWarps_ || group != perfGroup_) built_ = false;   // the captured graph holds the old kernels
    perfWarps_ = warps;
    perfGroup_ = group;
}

std::vector<Batch::Trial> Batch::autotune(int32_t mcsPerTrial)
{
    // Every configuration gives the same trajectories, so the trials are ordinary MCS of the run:
    // each configuration runs 1 MCS and then mcsPerTrial MCS, both timed. What a run costs however long it is
    // (slots loaded and written back, streams joined) would have few MCS per trial choose for runs as short as
    // the trials (40 systems of 60K, 2 MCS 95 us per MCS in slab sweeps and 88 in the grid phase, 100 MCS 46
    // and 65): the paths are compared by the time that the further MCS take, their kernels' shapes by the
    // longer run less the path's fixed time.
    if (mcsPerTrial <= 0) throw std::invalid_argument("[Batch::autotune] trials need at least one MCS");
    cuda_check(cudaSetDevice(gpu_), "cudaSetDevice");
    if (!built_) rebuild();
    // cluster on and off differ only where a member that does not run resident fits the slab sweep
    bool anyResident = false, anyCluster[2] = {false, false};
    for (Updater* u : members_) {
        anyResident = anyResident || u->residentEligible();
        bool const cl = slabFits(*u);
        anyCluster[0] = anyCluster[0] || cl;
        anyCluster[1] = anyCluster[1] || (cl && !u->residentEligible());
    }
    if (residentOn_ && clusterOn_) anyCluster[1] = anyCluster[1] || !cluster_.empty();
    // Three stages, each configuration timed over the same kind of MCS: first the paths (resident
    // kernel on / off x cluster kernel on / off, where either can matter) with the grid kernels'
    // defaults; then, for the best paths under which some member runs on the grid-phase kernels (with the
    // slab sweeps off where they take every member), the
    // check's register budget (kGridShapes) x its CTA size (128, 256, 512 threads), as the
    // reference sweeps its block size (CRITICAL.cu:445-487); last, for the best of those, the
    // perform's warps per CTA x warps per tile.
    struct Whole {   // the trials are of the paths they name, however short
        bool& on;
        explicit Whole(bool& o) : on(o) { on = false; }
        ~Whole() { on = true; }
    } const whole(shortRuns_);
    std::vector<Trial> trials;
    float fixed[2][2] = {};   // ms of a run on each path before its first MCS
    auto time_it = [&](bool resident, bool cl, int shape, int block, int pw, int pg, bool path = false) {
        setResidentEnabled(resident);
        setClusterEnabled(cl);
        setShape(shape);
        setBlock(block);
        setPerformShape(pw, pg);
        rebuild();
        std::vector<int32_t> const none(members_.size(), 0);
        float idle = 0.f;   // every kernel, all members idle (the first time it is loaded as well)
        for (int rep = 0; rep < 4; ++rep) {
            for (Updater* u : members_) u->synchronize();
            float const t = timed([&] { enqueue(none.data(), 1); });
            idle = rep < 2 ? t : std::min(idle, t);
        }
        float const one = runTimed(1), ms = runTimed(mcsPerTrial), k = (float)mcsPerTrial;
        float& f = fixed[resident][cl];
        // (a run of 1 MCS that was held up must not make a path look fast: the MCS take at least the time
        // of the run less that of an idle one)
        if (path && mcsPerTrial > 1) f = std::max(0.f, ms - std::max(k * (ms - one) / (k - 1.f), ms - idle));
        trials.push_back(Trial{shape_, resident, cl, block_, pw, pg, std::max(ms - f, 0.1f * ms) / k});
        return trials.back();
    };
    Trial best{};
    bool first = true;
    for (int resident = 1; resident >= 0; --resident) {
        if (!resident && !anyResident) break;   // the same configuration as resident on
        for (int cl = 1; cl >= 0; --cl) {
            if (!cl && !anyCluster[resident]) break;   // the same configuration as cluster on
            Trial const t = time_it(resident != 0, cl != 0, -1, 0, 0, 0, true);
            if (first || t.msPerMcs < best.msPerMcs) best = t;
            first = false;
        }
    }
    bool clusterOn = best.cluster;
    for (;;) {
        setResidentEnabled(best.resident);
        setClusterEnabled(clusterOn);
        rebuild();
        if (!grid_.empty() || !clusterOn) break;
        clusterOn = false;
    }
    if (!grid_.empty()) {
        Trial grid{};
        for (int block : {128, 256, 512})
            for (int sh = 0; sh < kGridShapes; ++sh) {
                Trial const t = time_it(best.resident, clusterOn, sh, block, 0, 0);
                if (grid.msPerMcs == 0.f || t.msPerMcs < grid.msPerMcs) grid = t;
            }
        Trial const base = grid;
        for (auto pw : kPerformShapeTrials) {
            Trial const t = time_it(base.resident, base.cluster, base.shape, base.block, pw[0], pw[1]);
            if (t.msPerMcs < grid.msPerMcs) grid = t;
        }
        if (grid.msPerMcs < best.msPerMcs) best = grid;
    }
    setResidentEnabled(best.resident);
    setClusterEnabled(best.cluster);
    setShape(best.shape);
    setBlock(best.block);
    setPerformShape(best.perfWarps, best.perfGroup);
    return trials;
}

template <typename Queue>
float Batch::timed(Queue const& queue)
{
    cudaEvent_t a, b;
    cuda_check(cudaEventCreate(&a), "cudaEventCreate");
    cuda_check(cudaEventCreate(&b), "cudaEventCreate");
    cuda_check(cudaEventRecord(a, stream_), "event");
    queue();   // the other streams join stream_ before it returns
    cuda_check(cudaEventRecord(b, stream_), "event");
    cuda_check(cudaEventSynchronize(b), "timed batch");
    float ms = 0.f;
    cuda_check(cudaEventElapsedTime(&ms, a, b), "elapsed");
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    checkReports();
    return ms;
}

float Batch::runTimed(int32_t nMcs)
{
    cuda_check(cudaSetDevice(gpu_), "cudaSetDevice");
    for (Updater* u : members_) u->synchronize();
    if (!built_) rebuild();
    if (nMcs > 0) {
        std::vector<int32_t> each(members_.size(), nMcs);
        prepare(each.data());
    }
    return timed([&] { run(nMcs); });
}

void Batch::synchronize()
{
    cuda_check(cudaStreamSynchronize(stream_), "batch");
    cuda_check(cudaStreamSynchronize(stream2_), "batch");
    checkReports();
}

void Batch::checkReports()
{
    std::atomic_thread_fence(std::memory_order_acquire);
    for (auto const& w : slab_)
        for (SlabRef const& r : w.refs)
            if (static_cast<GridFault const volatile*>(reports_.get())[r.sys].fault)
                throw CudaError("[Batch::run] a grid barrier of a member's slab sweep timed out; the state of member " +
                                std::to_string(r.sys) + " is not usable");
}

}  // namespace bfm
