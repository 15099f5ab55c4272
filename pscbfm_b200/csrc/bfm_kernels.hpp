// Host-callable launchers of the sweep kernels (bfm_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "bfm_device.cuh"

namespace bfm {

constexpr uint32_t kGridBlock = 256;          // threads per CTA of the grid-phase kernels
constexpr uint32_t kResidentBlock = 1024;     // threads per CTA of the resident kernel
constexpr uint32_t kClusterSmallBlock = 512;  // threads per CTA of the cluster kernel with few slots per CTA
// dynamic shared memory of the resident kernel: the 227 KB opt-in limit minus room for its
// static shared memory (the copied system descriptor)
constexpr size_t kResidentMaxSmem = 226 * 1024;
// Raises a kernel's dynamic shared memory limit to kResidentMaxSmem, once per device and thread (done: that
// kernel's own flags). Always to the same value: the limit belongs to the function, not to the
// launch, so a thread that set what its own launch needs would lower it under another thread's.
template <typename F>
cudaError_t allow_smem(F* kernel, bool (&done)[64])
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || done[dev & 63]) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kResidentMaxSmem);
    done[dev & 63] = e == cudaSuccess;
    return e;
}
// Sub-steps of one launch of the kernels that run many (resident, cluster, slab), at most; a longer run is
// several launches. A CTA holds at most kCtaSlots slots of a colour and counts its moves in 32 bits, and no
// CTA keeps its SM from other work for more than a second or so (65536 sub-steps of 8K slots in one CTA 0.35 s).
constexpr uint32_t kLaunchSteps = 1u << 16, kCtaSlots = 16 * kResidentBlock;
static_assert((unsigned long long)kLaunchSteps * kCtaSlots < (1ull << 32), "a launch's move counts fit 32 bits");
constexpr int32_t kPadCoord = INT32_MIN;      // x of an unused (padding) slot

// One CTA of a grid-phase launch: system index and first in-colour index it covers.
struct TileRef {
    uint32_t sys;
    uint32_t start;
    uint32_t count = 1;   // consecutive tiles from start (bond-code perform lists group up to 4)
};

// dTiles == nullptr: single system 0, CTA b covers [b*tileSpan, (b+1)*tileSpan).
cudaError_t launch_check(SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles, uint32_t tileSpan,
                         StepEntry const* dSteps, cudaStream_t s);
// next != nullptr (one system): CTA 0 writes the following sub-step's entry there (write_next_step)
cudaError_t launch_perform(SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles, uint32_t tileSpan,
                           StepEntry const* dSteps, cudaStream_t s, StepEntry* next = nullptr);

// Resident kernel: CTA b runs system dList[b] through sub-steps 0..nSteps-1 of dSteps
// ([nSteps][nSys] entries). perThread = ceil(largest colour group / kResidentBlock), in {1,2,4,8,16}.
size_t resident_smem_bytes(uint32_t nwords, uint32_t ntab);
cudaError_t launch_resident(SysDev const* dSys, uint32_t const* dList, uint32_t nCta, uint32_t perThread,
                            StepEntry const* dSteps, uint32_t nSys, uint32_t nSteps, size_t smem, cudaStream_t s);

// Bond-code kernels (SysDev::codeMode kCode32 / kCode64). Tiles span kBcTileSpan in-colour
// indices. As in the gather representation, the perform zeroes the previous sub-step's marks, so a
// stand-alone scrub is a perform launch whose entry has color == kNoColor.
constexpr int kCheckMpt = 2;                                   // monomers per thread (256-thread CTAs)
constexpr uint32_t kBcTileSpan = kGridBlock * kCheckMpt;       // 512 in-colour indices per tile
// CTA sizes of the bond-code check: 128, 256 or 512 threads over the same tile (4, 2 or 1
// monomers per thread); every size gives the same results
constexpr uint32_t kCheckBlockDefault = 256;
inline bool check_block_ok(int block) { return block == 128 || block == 256 || block == 512; }
// dTiles == nullptr: single system, descriptor passed by value (hostDesc); otherwise the tile
// list selects the system per CTA from dSys and hostDesc is unused. shape picks the check's register
// budget (resident threads per SM), 0 .. kGridShapes-1, and block its CTA size (check_block_ok);
// negative / 0: the defaults. Every shape and block gives the same results.
constexpr int kGridShapes = 4;
// The perform launch's tile list for a check tile list of bond-code systems: one tile per entry.
std::vector<TileRef> perform_tile_list(std::vector<TileRef> const& tiles);
// snap != nullptr (one system): the check first writes the snapshot of the move counters as the
// work before it left them into that ring (snapshot_stats; the sequence word follows the 4 x
// kSnapRing slot words). The check counts attempted moves (CTA 0, after the snapshot) and the
// perform the tentative ones (list lengths) and the accepted ones.
cudaError_t launch_check_bc(SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles,
                            StepEntry const* dSteps, uint32_t codeMode, cudaStream_t s, int shape = -1,
                            int block = 0, unsigned long long* snap = nullptr);
// The perform takes one warp per tile. A single-system launch may carry the sub-step's parity and
// scope (kPerfCur: walk its tentative movers, kPerfPrev: zero the previous sub-step's marks), so
// it reads no step entry; parity == kParityFromEntry reads both from dSteps[0]. next != nullptr
// (one system): CTA 0 writes the following sub-step's entry there (write_next_step). Tile lists
// (several systems) always read each system's entry; parity, scope and next are ignored.
constexpr uint32_t kParityFromEntry = 0xFFFFFFFFu;
constexpr uint32_t kPerformWarpsDefault = 4;   // warps per CTA of the perform
constexpr uint32_t kPerformGroupDefault = 4;   // warps per tile of the perform
// the perform shapes (warps per CTA, warps per tile) an autotuner tries beside the default
constexpr int kPerformShapeTrials[][2] = {{8, 4}, {4, 2}, {8, 8}, {2, 2}};
constexpr uint32_t kPerfCur = 1u, kPerfPrev = 2u;
struct PerformArgs {
    uint32_t parity = kParityFromEntry;
    uint32_t scope = kPerfCur | kPerfPrev;
    StepEntry* next = nullptr;
    unsigned long long* snap = nullptr;   // the check's counter snapshot ring (launch_check_bc)
    int warps = 0;   // warps per CTA (1, 2, 4, 8; 0: the default)
    int group = 0;   // warps per tile (1, 2, 4, 8, at most `warps`; 0: the default)
};
inline bool perform_shape_ok(int warps, int group)
{
    auto ok = [](int v) { return v == 1 || v == 2 || v == 4 || v == 8; };
    return (warps == 0 && group == 0) || (ok(warps) && ok(group) && group <= warps);
}
cudaError_t launch_perform_bc(SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles,
                              StepEntry const* dSteps, uint32_t codeMode, cudaStream_t s, int shape = -1,
                              PerformArgs const& pa = PerformArgs{});
// Slab sweeps (bond codes): nSteps sub-steps of a system by plan.ctas CTAs of a cooperative launch, each
// holding its share of the slots in shared memory (slab_sweep): one system (k_slab_bc), or several in one
// launch (k_slab_batch_bc). slab_plan returns false where the system does not fit ctas CTAs (more than
// kSlabColors colours, or too many slots per CTA). report (mapped host memory): its fault word is set
// when a grid-barrier wait ran out; the system's state is then not usable.
// threads per CTA (one CTA per SM); 64-bit codes keep up to six neighbours of a mover in registers
constexpr uint32_t kSlabBlock32 = 640, kSlabBlock64 = 512, kSlabBlockSmall = 256;
constexpr uint32_t kSlabSmallSlots = 1024;   // slots per CTA and colour, at most, of the small CTAs
constexpr uint32_t kSlabColors = 8;          // bond codes: at most 6 bonds, so at most 7 colours
constexpr uint32_t kSlabEntBits = 13;         // list entries: a slot's index in its colour's part, and 3 direction bits
// bits of a local index in a 16-bit neighbour reference, below the reverse slot (0-2, or 0-5 with 64-bit codes)
__host__ __device__ constexpr uint32_t slab_ref_bits(bool code64) { return code64 ? 13u : 14u; }
constexpr uint32_t kSlabMinChunks = 8;       // chunks of 32 slots per CTA and colour, before more CTAs join
constexpr size_t kSlabMaxSmem = kResidentMaxSmem;
struct SlabPlan {
    uint32_t ctas = 0;         // 0: the system does not fit
    uint32_t cap = 0, perCta = 0;   // slots a CTA holds in all, and of the largest colour group
    uint32_t threads = 0;      // threads per CTA
    bool clearAll = false;     // the temporary lattice is zeroed whole
    bool cache = false;        // the neighbour references and inner direction hashes fit in shared memory too
    size_t smem = 0;           // dynamic shared memory per CTA
};
bool slab_plan(uint32_t const* grpSize, uint32_t nColors, uint32_t maxc, uint32_t nwords, uint32_t codeMode,
               uint32_t ctas, SlabPlan& plan);
// CTAs of a cooperative launch for a system whose largest colour group is maxGroup
uint32_t slab_ctas(uint32_t maxGroup, uint32_t sms);
// CTAs of such a launch that an SM holds at a time (0: the question failed).
uint32_t slab_ctas_per_sm(SlabPlan const& plan, uint32_t codeMode);
cudaError_t launch_slab_bc(SysDev const& hostDesc, StepSource const& src, uint32_t nSteps, SlabPlan const& plan,
                           GridFault* report, uint32_t codeMode, cudaStream_t s);
// Plans with the cache only; dRefs: the launch's CTAs; the reports are report[system].
cudaError_t launch_slab_batch(SysDev const* dSys, SlabRef const* dRefs, uint32_t ctas, size_t smem,
                              StepSource const& src, uint32_t nSteps, GridFault* report, uint32_t codeMode,
                              cudaStream_t s);
// Dynamic shared memory of the bond-code resident kernel, with the neighbour references where they fit too.
size_t resident_bc_smem_bytes(uint32_t nwords, uint32_t npad, uint32_t maxGroup, uint32_t maxc, uint32_t codeMode);
// Cluster-resident sweep (bond codes): one cluster of 2^logC CTAs per
// system of dList[0..nClusters) (logC 1..4), state in the cluster's shared memory for nSteps
// sub-steps; at most `chunks` (16, 32: CTAs of kClusterSmallBlock threads; 64, 128, 256: of kResidentBlock)
// chunks of 32 slots per CTA and colour. cluster_bc_runnable: how many such clusters the device runs at a time.
size_t cluster_bc_smem_bytes(uint32_t nwords, uint32_t npad, uint32_t logC, uint32_t chunks, uint32_t maxc,
                             uint32_t codeMode);
uint32_t cluster_bc_runnable(uint32_t logC, uint32_t chunks, size_t smem, uint32_t codeMode);
cudaError_t launch_cluster_bc(SysDev const* dSys, uint32_t const* dList, uint32_t nClusters, uint32_t logC,
                              uint32_t chunks, StepSource const& src, uint32_t nSteps, size_t smem,
                              uint32_t codeMode, cudaStream_t s);
cudaError_t launch_resident_bc(SysDev const* dSys, uint32_t const* dList, uint32_t nCta, uint32_t perThread,
                               StepSource const& src, uint32_t nSteps, size_t smem, uint32_t codeMode, cudaStream_t s);

// Observables (bfm_observables.cu). Molecule of every slot (kNoColor for padding), first and last
// slot of every molecule, and the reference positions for the mean squared displacement.
struct ObsDev {
    uint32_t const* molOfSlot;
    uint32_t const* ends;       // [2 * nMol]
    int32_t const* rx;
    int32_t const* ry;
    int32_t const* rz;
    uint32_t nMol;
};
inline size_t obs_words(uint32_t nMol) { return 5ull * nMol + 512 + 1; }
cudaError_t launch_observables(SysDev const* dSys, ObsDev const& o, long long* dOut, uint32_t npad, cudaStream_t s);

// Sets the occupancy bit of every non-padding slot of system dSys[0] (lat must be zeroed).
cudaError_t launch_build_lattice(SysDev const* dSys, uint32_t npad, cudaStream_t s);
// Positions in the caller's order, x y z interleaved (out[3 i + a] from sorted slot slotOf[i]).
cudaError_t launch_gather_positions(SysDev const& h, uint32_t const* slotOf, uint32_t n, int32_t* out,
                                    DoneSignal const& done, cudaStream_t s);
// Unfolded positions of every slot of bond-code system dSys[0] (image offsets plus the coordinates
// of the lattice addresses) into ox, oy, oz, in slot order.
cudaError_t launch_unfold_positions(SysDev const* dSys, uint32_t npad, int32_t* ox, int32_t* oy, int32_t* oz,
                                    cudaStream_t s);
// Writes the sums over the kStatSlots slots of the three move counters (attempted, tentative,
// accepted) into out[0..3), mapped pinned host memory.
cudaError_t launch_publish_stats(unsigned long long const* stats, unsigned long long* out, cudaStream_t s);
// A counter snapshot (snapshot_stats) as a one-warp launch: a captured sweep graph's last node
// when its handle's counters are read by ticket; k_publish_snap copies one slot of the snapshot
// ring into host memory, on another stream.
cudaError_t launch_snapshot_stats(unsigned long long const* stats, unsigned long long* ring, unsigned long long* seq,
                                  cudaStream_t s);
cudaError_t launch_publish_snap(unsigned long long const* slot, unsigned long long* out, cudaStream_t s);

}  // namespace bfm
