// Host check of plan_slab_waves: members drawn over the range of sizes, shares of the SMs from a few to all.
// No launch has more CTAs than its share leaves it; every member is taken once, on CTAs that hold it, or
// left to the grid-phase kernels because the share does not hold it.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "bfm_engine.hpp"

using namespace bfm;

#define REQUIRE(c)                                                                                  \
    do {                                                                                            \
        if (!(c)) {                                                                                 \
            std::printf("line %d: %s (case %d)\n", __LINE__, #c, number);                           \
            return 1;                                                                               \
        }                                                                                           \
    } while (0)

static SlabMember member(uint32_t n, uint32_t mode, bool resident, uint32_t nwords = 1u << 18)
{
    return SlabMember{n, mode, resident, [=](uint32_t C, SlabPlan& p) {
                          uint32_t const grp[2] = {n / 2, n - n / 2};
                          return slab_plan(grp, 2, mode == kCode64 ? 4 : 2, nwords, mode, C, p);
                      }};
}

static bool fits(SlabMember const& m, uint32_t most)
{
    SlabPlan p;
    for (uint32_t C = 1; C <= most; ++C)
        if (m.plan(C, p) && p.cache) return true;
    return false;
}

static int check(int number, std::vector<SlabMember> const& members, uint32_t sms, uint32_t share)
{
    SlabWaves const w = plan_slab_waves(members, sms, share);
    REQUIRE(w.taken.size() == members.size());
    uint32_t residents = 0;
    bool grid = false;
    for (size_t m = 0; m < members.size(); ++m) {
        residents += members[m].resident;
        grid = grid || (!members[m].resident && !w.taken[m]);
        REQUIRE(!(members[m].resident && w.taken[m]));
    }
    REQUIRE(w.residentsAfter == (residents > share / 4));
    uint32_t const budget = std::max(1u, grid ? share / 2 : share - (w.residentsAfter ? 0 : residents));
    std::vector<uint32_t> seen(members.size(), 0);
    for (SlabWave const& wave : w.waves) {
        REQUIRE(!wave.refs.empty() && wave.refs.size() <= budget);
        for (size_t i = 0; i < wave.refs.size();) {
            SlabRef const r = wave.refs[i];
            SlabPlan p;
            REQUIRE(members[r.sys].codeMode == wave.codeMode && w.taken[r.sys] && ++seen[r.sys] == 1);
            REQUIRE(members[r.sys].plan(r.ctas, p) && p.cache && p.smem <= wave.smem && wave.smem <= kSlabMaxSmem);
            for (uint32_t k = 0; k < r.ctas; ++k, ++i)
                REQUIRE(i < wave.refs.size() && wave.refs[i].sys == r.sys && wave.refs[i].rank == k &&
                        wave.refs[i].ctas == r.ctas);
        }
    }
    for (size_t m = 0; m < members.size(); ++m) {
        REQUIRE(seen[m] == (w.taken[m] ? 1u : 0u));
        if (!members[m].resident && members[m].codeMode != kCodeNone)
            REQUIRE(w.taken[m] == fits(members[m], std::min(budget, sms / 2)));
    }
    return 0;
}

int main()
{
    // a server lane of 37 SMs: 700K monomers need 43 CTAs, more than the lane has
    int number = -1;
    SlabPlan p;
    REQUIRE(member(700000, kCode32, false).plan(74, p) && p.cache && !fits(member(700000, kCode32, false), 37));
    if (check(0, {member(700000, kCode32, false), member(60000, kCode32, false)}, 148, 37)) return 1;
    // beside a gathering member the lane's sweeps have 18 SMs: 300K need 19
    if (check(1, {member(300000, kCode32, false), member(9000, kCodeNone, false), member(30000, kCode32, false)}, 148, 37))
        return 1;
    // two waves where one is not enough, as evenly as their sizes allow: none to the brim beside one nearly empty
    {
        number = 2;
        std::vector<SlabMember> const members(32, member(60288, kCode32, false, 1u << 15));
        SlabWaves const w = plan_slab_waves(members, 148, 148);
        REQUIRE(w.waves.size() == 2 && w.waves[0].refs.size() == 148 && w.waves[1].refs.size() == 148);
        size_t first = 0;
        for (SlabRef const& r : w.waves[0].refs) first += r.rank == 0;
        REQUIRE(first == 16);
        // at most one launch: none for these, one for a lane's few
        SlabWaves const none = plan_slab_waves(members, 148, 148, 1), few = plan_slab_waves({members[0], members[1]}, 148, 37, 1);
        REQUIRE(none.waves.empty() && none.taken == std::vector<char>(32, 0) && few.waves.size() == 1 && few.taken[1]);
    }
    std::mt19937 rng(12345);
    for (number = 3; number < 3000; ++number) {
        std::uniform_real_distribution<double> u(0.0, 1.0);
        std::vector<SlabMember> members;
        size_t const count = 1 + size_t(40 * u(rng) * u(rng));
        for (size_t k = 0; k < count; ++k) {
            uint32_t const n = (uint32_t)(20000 * std::pow(60.0, u(rng)));
            double const kind = u(rng);
            uint32_t const mode = kind < 0.03 ? kCodeNone : kind < 0.2 ? kCode64 : kCode32;
            bool const resident = u(rng) < 0.3;
            members.push_back(resident ? member(3000, mode, true) : member(n, mode, false));
        }
        uint32_t const share = u(rng) < 0.4 ? 148 : 1 + (uint32_t)(147 * u(rng));
        if (check(number, members, 148, share)) return 1;
    }
    std::printf("ok\n");
    return 0;
}
