// Bond-code kernels of the BFM sweep (sm_100a).
//
// The same sub-step as the gather kernels (check: CRITICAL.cu:298-374, perform + apply:
// CRITICAL.cu:376-411, clear: :561-573), on a different state: each monomer keeps the lattice
// address of its corner (pk: brick word << 6 | bit; moves and front planes are adds confined to one
// axis's address bits) and a bond-code word whose 9-bit fields are the reference's bond-table
// indices of its bonds, so the check needs no neighbour positions. When a monomer moves by d, its
// own fields change by -d and the reverse field of every neighbour by +d; the reverse field's old
// value is the negation (mod 8) of the monomer's own field, so the update needs no extra load.
//
// Grid phase (k_check_bc, k_perform_bc): the check lists its tentative movers per tile, with the
// address of the temporary-lattice cell each one marked (mover lists, double-buffered by sub-step
// parity); the perform walks only those lists, and the perform of sub-step t also zeroes the words
// listed at t-1. Every independent load of a pass is issued before any dependent one; a single-system
// launch takes the descriptor as a grid-constant parameter.
//
// Persistent (k_slab_bc): a whole run of sub-steps in one cooperative launch with time-bounded grid
// barriers; the lattices in global memory, each CTA's share of the slots in its shared memory.
//
// Resident (k_resident_bc): one CTA owns a small system for a chunk of sub-steps; lattice, temporary
// lattices, addresses, bond codes and neighbour references in shared memory; tentative movers go to
// a shared list (warp ballot + one atomic per warp), so the perform runs with full warps.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "bfm_device.cuh"
#include "bfm_kernels.hpp"

namespace bfm {

namespace {


__device__ __forceinline__ void copy_desc(SysDev& dst, SysDev const* src)
{
    static_assert(sizeof(SysDev) % 4 == 0, "SysDev is copied word by word");
    uint32_t const* s = reinterpret_cast<uint32_t const*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
    for (uint32_t w = threadIdx.x; w < sizeof(SysDev) / 4; w += blockDim.x) d[w] = s[w];
}

// True if every bond of the code word stays allowed after the move along dir: the AND of the move
// table's entries over all fields (an unused field is index 0, whose entry allows every move).
template <typename W, bool kSharedTables>
__device__ __forceinline__ bool bonds_ok(W code, uint32_t dir, uint8_t const* ok)
{
    uint32_t m = 0xFFu;
#pragma unroll
    for (uint32_t k = 0; k < CodeWord<W>::kSlots; ++k) {
        uint32_t const idx = uint32_t(code >> (9u * k)) & 511u;
        m &= kSharedTables ? ok[idx] : __ldg(ok + idx);
    }
    return (m >> dir) & 1u;
}

constexpr uint32_t kStepBlock = 8;   // step entries staged in shared memory at a time (static shared memory stays below 1 KB)

// Adds v to a counter in shared memory and returns its old value, as one instruction: written with
// atomicAdd, the compiler gathers the adds of a warp first, 20 instructions for the one lane that adds.
__device__ __forceinline__ uint32_t shared_add(uint32_t* p, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;"
                 : "=r"(old)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v)
                 : "memory");
    return old;
}
__device__ __forceinline__ void shared_xor(uint32_t* p, uint32_t v) { atomicXor(p, v); }
// (a 64-bit exclusive or as two on the halves: shared memory has no native 64-bit one)
__device__ __forceinline__ void shared_xor(unsigned long long* p, unsigned long long v)
{
    unsigned int* const h = reinterpret_cast<unsigned int*>(p);
    if ((unsigned int)v) atomicXor(h, (unsigned int)v);
    if ((unsigned int)(v >> 32)) atomicXor(h + 1, (unsigned int)(v >> 32));
}

// The words a front plane touches and their masks, prepared ahead of the reads (a word that is not
// touched has an empty mask; reads of it are left out).
struct PlaneRef {
    uint32_t w[4];
    unsigned long long m[4];
};
__device__ __forceinline__ void plane_ref(PlaneRef& r, unsigned long long const* ptab, DirParams const& D,
                                          uint32_t base, uint32_t da, uint32_t dir)
{
    uint32_t ti, touch;
    front_plane_words(r.w, ti, touch, D, base, da, dir);
    // entry ti / 4, its first two masks in the table's first half and the others in the second: 16-byte
    // entries spread over all banks (21 wavefronts per warp, 28 with the 32-byte entries of planeTab)
    ulonglong2 const m01 = *reinterpret_cast<ulonglong2 const*>(ptab + ti / 2u);
    ulonglong2 const m23 = *reinterpret_cast<ulonglong2 const*>(ptab + 384u + ti / 2u);
    r.m[0] = m01.x;
    r.m[1] = m01.y;
    r.m[2] = m23.x;
    r.m[3] = m23.y;
}
// Mover lists: the check of sub-step t appends each tentative mover of tile k (kBcTileSpan
// in-colour indices) to segment k of list[parity] (entry: slot g in bits 0-26, direction in
// 27-29), the lattice address of its target (the temporary-lattice cell it marked) to the same
// place of word[parity], and stores the segment's length in count[parity][k]. The perform of
// sub-step t walks only the listed movers, and zeroes the words of the targets listed at t-1
// (nobody reads tmp[parity^1] during sub-step t, and the check of t+1, which marks it again,
// comes after).
constexpr uint32_t kEntSlotMask = (1u << 27) - 1u;
// Tentative movers a lane of the grid perform takes per pass over its tile's list: 32 x kPerfQ
// entries, loaded together with the list's length (about a sixth of a dense tile's 512 monomers
// move tentatively, so one pass covers a tile of a dense system; longer lists take more passes).
constexpr int kPerfQ = 4;

// ---------------------------------------------------------------------------------- check

template <typename W, int MPT>
__device__ __forceinline__ void check_body(SysDev const& S, uint32_t const* dtab, StepEntry const& st, uint32_t start,
                                           uint32_t* segCount, uint2* stage)
{
    uint32_t const B = blockDim.x, tid = threadIdx.x;
    using RV = typename SlotRec<W>::V;
    RV const* const REC = reinterpret_cast<RV const*>(S.rec);
    uint32_t const tile = start / kBcTileSpan;
    unsigned long long* const tcur = S.tmp + (size_t)st.parity * S.nwords;
    size_t const seg = (size_t)st.parity * S.listStride + (size_t)tile * kBcTileSpan;
    uint32_t* const lcur = S.mlist + seg;
    uint32_t* const wcur = S.mword + seg;

    // stage 1: every independent load of the pass; they stay in flight across the barrier that
    // publishes the caller's shared writes (the direction table, the segment count)
    uint32_t pk[MPT];
    W code[MPT];
#pragma unroll
    for (int q = 0; q < MPT; ++q) {
        uint32_t const i = start + tid + (uint32_t)q * B;
        RV const r = i < st.cnt ? __ldg(REC + st.off + i) : RV{};
        pk[q] = r.x;
        code[q] = rec_code_of(r);
    }
    __syncthreads();
    // stage 2: direction, walls, bonds; the monomers that pass go to this warp's part of the
    // stage (address, slot | direction << 27), packed, so that the front-plane and occupancy work
    // below runs on full warps of candidates only (about half the monomers fail here)
    uint32_t const lane = tid & 31u;
    uint32_t const lanesBelow = (1u << lane) - 1u;
    uint2* const ws = stage + (tid >> 5) * (32u * MPT);
    uint32_t n = 0;
    bool const walled = S.walls != 0u;   // uniform: a periodic box skips the wall test's table reads
#pragma unroll
    for (int q = 0; q < MPT; ++q) {
        uint32_t const i = start + tid + (uint32_t)q * B;
        uint32_t const dir = move_dir(i, st.seed);
        bool free = true;
        if (walled) {
            uint2 const mw = make_uint2(dtab[dir * 4u], dtab[kDirHalf + dir * 4u + 3u]);   // Ma, wall
            free = (pk[q] & mw.x) != mw.y;
        }
        bool const ok = i < st.cnt && free && bonds_ok<W, false>(code[q], dir, S.moveOk);
        uint32_t const bal = __ballot_sync(0xffffffffu, ok);
        if (ok) ws[n + __popc(bal & lanesBelow)] = make_uint2(pk[q], (st.off + i) | (dir << 27));
        n += (uint32_t)__popc(bal);
    }
    __syncwarp();
    // stage 3: per candidate, the front plane from its address, the occupancy words, and for a
    // free plane the mark and the list entries (one shared-memory atomic per warp and pass)
    for (uint32_t b = 0; b < n; b += 32u) {
        bool const live = b + lane < n;
        uint2 const it = live ? ws[b + lane] : make_uint2(0u, 0u);
        uint32_t const dir = it.y >> 27;   // 0 for a dead lane: table reads stay in range
        DirParams const D = dir_params(dtab, dir);
        Plane pl;
        front_plane<false>(pl, S.planeTab, D, it.x, D.front, dir);
        uint32_t const to = addr_add(it.x, D.ma, D.step);
        unsigned long long hit = 0ull;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (live && ((pl.touch >> r) & 1u)) hit |= __ldg(S.lat + pl.w[r]) & pl.m[r];
        bool const go = live && hit == 0ull;
        uint32_t const bal = __ballot_sync(0xffffffffu, go);
        uint32_t base = 0;
        if (lane == 0 && bal) base = atomicAdd(segCount, (uint32_t)__popc(bal));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (go) {
            atomicOr(tcur + (to >> 6), 1ull << (to & 63u));
            uint32_t const slot = base + __popc(bal & lanesBelow);
            lcur[slot] = it.y;
            wcur[slot] = to;
        }
    }
}

// ---------------------------------------------------------------------------------- perform

// Image offsets (x, y, z with bond codes, see SysDev) of slot g after a move along axis a by s from
// lattice address p0 to p1 (ma: the axis's address bits): they change only when the move wraps the
// periodic axis, i.e. reaches coordinate 0 going up or leaves it going down; a walled axis never
// wraps. About one move in a lattice side along that axis writes here.
__device__ __forceinline__ void image_step(SysDev const& S, uint32_t g, uint32_t a, int32_t s, uint32_t p0,
                                           uint32_t p1, uint32_t ma)
{
    if (((s > 0 ? p1 : p0) & ma) == 0u)
        atomicAdd((a == 0 ? S.x : (a == 1 ? S.y : S.z)) + g, s * int32_t(S.mask[a] + 1u));
}

// Movers ent[q] (list entries: slot | direction << 27) with targets to[q], for the q with
// live[q]: re-test the front plane on the temporary lattice and apply the free moves. The plane
// and the old position follow from the target's address, so the monomer's own address is not
// loaded. Returns the moves applied.
template <typename W, int N>
__device__ __forceinline__ uint32_t perform_movers(SysDev const& S, uint32_t const* dtab,
                                                   unsigned long long const* tcur, uint32_t const (&ent)[N],
                                                   uint32_t const (&to)[N], bool const (&live)[N])
{
    using RV = typename SlotRec<W>::V;
    RV* const REC = reinterpret_cast<RV*>(S.rec);
    Plane pl[N];
    W code[N];
    uint32_t nbr[N][CodeWord<W>::kSlots];
#pragma unroll
    for (int q = 0; q < N; ++q) {
        uint32_t const g = live[q] ? ent[q] & kEntSlotMask : 0u;
        code[q] = live[q] ? *rec_code<W>(S.rec, g) : W(0);
#pragma unroll
        for (uint32_t k = 0; k < CodeWord<W>::kSlots; ++k)
            nbr[q][k] = (live[q] && k < S.maxc) ? __ldg(S.nbrr + (size_t)k * S.npad + g) : 0u;
    }
#pragma unroll
    for (int q = 0; q < N; ++q) {
        // a lane past its list's end may hold any stale word: direction 0 keeps its table reads in
        // range (the direction table has six entries, the plane table three axes)
        uint32_t const d = live[q] ? (ent[q] >> 27) & 7u : 0u;
        DirParams const D = dir_params(dtab, d);
        front_plane<false>(pl[q], S.planeTab, D, to[q], D.step, d);
    }
    unsigned long long hit[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
        hit[q] = 0ull;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (live[q] && ((pl[q].touch >> r) & 1u)) hit[q] |= __ldg(tcur + pl[q].w[r]) & pl[q].m[r];
    }
    uint32_t nAcc = 0;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        if (!live[q] || hit[q] != 0ull) continue;
        ++nAcc;
        uint32_t const g = ent[q] & kEntSlotMask;
        uint32_t const dir = (ent[q] >> 27) & 7u;
        uint32_t const a = dir >> 1;
        int32_t const s = (dir & 1u) ? 1 : -1;
        uint2 const ms = *reinterpret_cast<uint2 const*>(dtab + dir * 4u);   // words 0, 1: Ma, step
        uint32_t const pk1 = to[q];
        uint32_t const pk0 = addr_add(pk1, ms.x, addr_back(ms.x, ms.y));
        uint32_t const w0 = pk0 >> 6, w1 = pk1 >> 6;
        if (w0 == w1) {
            atomicXor(S.lat + w0, (1ull << (pk0 & 63u)) | (1ull << (pk1 & 63u)));
        } else {
            atomicXor(S.lat + w0, 1ull << (pk0 & 63u));
            atomicXor(S.lat + w1, 1ull << (pk1 & 63u));
        }
        image_step(S, g, a, s, pk0, pk1, ms.x);
        W const own = code[q];
        REC[g] = make_rec(pk1, code_shift(own, a, -s));   // new address and code word in one store
        uint32_t const n = uint32_t(own >> CodeWord<W>::kCountShift) & 7u;
#pragma unroll
        for (uint32_t k = 0; k < CodeWord<W>::kSlots; ++k) {
            if (k < n) {
                uint32_t const nb = nbr[q][k];
                uint32_t const c = (0u - (uint32_t(own >> (9u * k + 3u * a)) & 7u)) & 7u;   // reverse field
                uint32_t const nc = uint32_t(int32_t(c) + s) & 7u;
                atomicXor(rec_code<W>(S.rec, nb & kSlotMask), W(c ^ nc) << (9u * (nb >> kSlotShift) + 3u * a));
            }
        }
    }
    return nAcc;
}

// Grid-phase perform of one tile by a group of G warps (`sub` = this warp's index in the group):
// the group walks list segment `tile` of this sub-step (parity p: its tentative movers) and of the
// previous one (parity p ^ 1: it zeroes the temporary-lattice words those movers marked), warp
// `sub` taking entries sub * 32 + lane + 32 G q. Every load of the first pass is independent of the
// others: both list lengths and Q entries, target addresses and previous targets per lane come in
// one round trip, so no length scan or barrier precedes the movers' own loads; entries past a
// list's end lie inside the tile's segment and are ignored. The lengths are exact for every tile of
// the launch: a check CTA whose tile lies beyond its colour group stores a zero length. Longer lists
// take further passes. The warp's copy of the direction table (dtab) is written from d0, d1 (words
// lane and lane + 32, loaded by the caller) once those loads are out, so the table's round trip
// overlaps the lists'. Returns the moves this warp applied.
template <typename W, int Q>
__device__ __forceinline__ uint32_t perform_tile(SysDev const& S, uint32_t* dtab, uint32_t d0, uint32_t d1,
                                                 uint32_t p, uint32_t tile, bool doCur, bool doPrev, uint32_t sub,
                                                 uint32_t G, uint32_t& listLen)
{
    uint32_t const lane = threadIdx.x & 31u;
    size_t const seg = (size_t)tile * kBcTileSpan;
    uint32_t const* const lc = S.mlist + (size_t)p * S.listStride + seg;
    uint32_t const* const wc = S.mword + (size_t)p * S.listStride + seg;
    uint32_t const* const wp = S.mword + (size_t)(p ^ 1u) * S.listStride + seg;
    unsigned long long const* const tcur = S.tmp + (size_t)p * S.nwords;
    unsigned long long* const tprev = S.tmp + (size_t)(p ^ 1u) * S.nwords;
    uint32_t const cnt = doCur ? __ldg(S.mcount + (size_t)p * S.countStride + tile) : 0u;
    uint32_t const pcnt = doPrev ? __ldg(S.mcount + (size_t)(p ^ 1u) * S.countStride + tile) : 0u;
    listLen = cnt;
    uint32_t const first = sub * 32u + lane, stride = 32u * G;
    uint32_t ent[Q], to[Q], pw[Q];
    bool live[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        uint32_t const e = first + stride * (uint32_t)q;   // < 32 G Q <= kBcTileSpan
        ent[q] = doCur ? __ldg(lc + e) : 0u;
        to[q] = doCur ? __ldg(wc + e) : 0u;
        pw[q] = doPrev ? __ldg(wp + e) : 0u;
    }
    dtab[lane] = d0;
    if (lane + 32u < kDirTab) dtab[lane + 32u] = d1;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q) live[q] = first + stride * (uint32_t)q < cnt;
    uint32_t nAcc = perform_movers<W, Q>(S, dtab, tcur, ent, to, live);
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (first + stride * (uint32_t)q < pcnt) tprev[pw[q] >> 6] = 0ull;
    uint32_t const pass = stride * (uint32_t)Q;
    for (uint32_t b = pass; b < cnt; b += pass) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            uint32_t const e = b + first + stride * (uint32_t)q;
            live[q] = e < cnt;
            ent[q] = live[q] ? __ldg(lc + e) : 0u;
            to[q] = live[q] ? __ldg(wc + e) : 0u;
        }
        nAcc += perform_movers<W, Q>(S, dtab, tcur, ent, to, live);
    }
    for (uint32_t b = pass; b < pcnt; b += pass) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            uint32_t const e = b + first + stride * (uint32_t)q;
            if (e < pcnt) tprev[__ldg(wp + e) >> 6] = 0ull;
        }
    }
    return nAcc;
}

}  // namespace

// ---------------------------------------------------------------------------------- kernels

// Grid-phase check: CTA b of B threads covers tile b (kBcTileSpan in-colour indices, kBcTileSpan / B
// per thread); a tile list (kMulti) gives each CTA its system and tile.
template <typename W, int B, bool kMulti, int kMinBlocks = 1>
__global__ void __launch_bounds__(B, kMinBlocks) k_check_bc(const __grid_constant__ SysDev S1,
                                                         SysDev const* __restrict__ sysv,
                                                         TileRef const* __restrict__ tiles,
                                                         StepEntry const* __restrict__ steps,
                                                         unsigned long long* snap)
{
    __shared__ SysDev Sm;
    __shared__ __align__(16) uint32_t dtab[kDirTab];
    constexpr int MPT = (int)kBcTileSpan / B;
    static_assert(B * MPT == (int)kBcTileSpan, "a CTA covers one list segment");
    // one system, snap != nullptr: the first warp of CTA 0 first takes the snapshot of the move
    // counters as the work before this launch left them (snapshot_stats). No CTA of the check adds to
    // the tentative count (the perform does) and CTA 0 adds the attempted count only after this, so
    // no other update of this launch can reach the counters before it.
    if (!kMulti && snap != nullptr && blockIdx.x == 0 && threadIdx.x < 32u)
        snapshot_stats(S1.stats, snap, snap + 4 * kSnapRing);
    uint32_t sys = 0, start = blockIdx.x * kBcTileSpan;
    // one system: the direction table's load goes out with the step entry's
    uint32_t dv = (!kMulti && threadIdx.x < kDirTab) ? S1.dirTab[threadIdx.x] : 0u;
    if (kMulti) {
        TileRef const tr = tiles[blockIdx.x];
        sys = tr.sys;
        start = tr.start;
    }
    StepEntry const st = steps[sys];
    if (st.color == kNoColor) return;
    if (start >= st.cnt) {
        // one system: the tile lies beyond this colour group; its list length becomes 0, so every
        // length the perform reads is this sub-step's (it does not read the step entry)
        if (!kMulti && threadIdx.x == 0) S1.mcount[(size_t)st.parity * S1.countStride + start / kBcTileSpan] = 0u;
        return;
    }
    if (kMulti) {
        copy_desc(Sm, sysv + sys);
        __syncthreads();
        if (threadIdx.x < kDirTab) dv = Sm.dirTab[threadIdx.x];
    }
    SysDev const& S = kMulti ? Sm : S1;
    __shared__ uint32_t segCount;
    __shared__ uint2 stage[kBcTileSpan];   // the warps' candidates (check_body)
    if (threadIdx.x < kDirTab) dtab[threadIdx.x] = dv;
    if (threadIdx.x == 0) segCount = 0;
    check_body<W, MPT>(S, dtab, st, start, &segCount, stage);   // publishes both with its first barrier
    __syncthreads();
    if (threadIdx.x == 0 && st.color != kNoColor) {
        // the list length; the perform that walks the list counts its entries as tentative moves
        S.mcount[(size_t)st.parity * S.countStride + start / kBcTileSpan] = segCount;
        if (start == 0) tally_flush(st.cnt, S.stats, 0);
    }
}

// Grid-phase perform: groups of G warps per tile of kBcTileSpan in-colour indices (perform_tile),
// PW warps per CTA (PW / G tiles); the groups of a CTA share nothing and never wait for each other.
// One system: `parity` and `scope` (kPerfCur: walk this sub-step's movers, kPerfPrev: scrub the
// previous sub-step's marks) come with the launch, so no load precedes the lists'; with parity ==
// kParityFromEntry they come from the step entry (a launch captured once and replayed on other
// entries). `next` != nullptr: the first warp of tile 0 also writes the following sub-step's entry
// there (write_next_step; the producer's state is loaded first, the entry stored after the warp's
// share of the tile). A tile list (kMulti): group b takes tile tiles[b] of system tiles[b].sys,
// whose step entry says what to do. nTiles: tiles of the launch (groups past it leave at once).
// Every warp of a group has 32 x max(4 / G, 1) list slots per pass.
template <typename W, bool kMulti, int PW, int G>
__global__ void __launch_bounds__(32 * PW) k_perform_bc(const __grid_constant__ SysDev S1, SysDev const* __restrict__ sysv,
                                                        TileRef const* __restrict__ tiles,
                                                        StepEntry const* __restrict__ steps, uint32_t parity,
                                                        uint32_t scope, StepEntry* next, uint32_t nTiles)
{
    static_assert(PW % G == 0, "whole groups per CTA");
    constexpr int Q = kPerfQ / G > 0 ? kPerfQ / G : 1;   // list slots per lane and pass
    __shared__ SysDev Sm[kMulti ? PW : 1];
    __shared__ __align__(16) uint32_t dtabs[PW][kDirTab];
    uint32_t const lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint32_t const wt = (blockIdx.x * PW + wid) / G;   // this group's tile (single) or tile-list entry
    uint32_t const sub = wid % G;
    if (wt >= nTiles) return;
    bool const writer = !kMulti && next != nullptr && wt == 0 && sub == 0 && lane == 0;
    StepGen gen{};
    if (writer) gen = *S1.gen;
    uint32_t p = parity, tile = wt, d0, d1;
    bool cur = (scope & kPerfCur) != 0u, prev = (scope & kPerfPrev) != 0u;
    if (!kMulti) {
        d0 = S1.dirTab[lane];
        d1 = lane + 32u < kDirTab ? S1.dirTab[lane + 32u] : 0u;
        if (parity == kParityFromEntry) {
            StepEntry const st = steps[0];
            uint32_t const start = tile * kBcTileSpan;
            p = st.parity;
            cur = st.color != kNoColor && start < st.cnt;
            prev = st.prevColor != kNoColor && start < st.pcnt;
        }
    } else {
        TileRef const tr = tiles[wt];
        SysDev& D = Sm[kMulti ? wid : 0];
        {   // the warp copies its system's descriptor
            static_assert(sizeof(SysDev) % 4 == 0, "SysDev is copied word by word");
            uint32_t const* src = reinterpret_cast<uint32_t const*>(sysv + tr.sys);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&D);
            for (uint32_t w = lane; w < sizeof(SysDev) / 4; w += 32u) dst[w] = src[w];
        }
        StepEntry const st = steps[tr.sys];
        p = st.parity;
        tile = tr.start / kBcTileSpan;
        cur = st.color != kNoColor && tr.start < st.cnt;
        prev = st.prevColor != kNoColor && tr.start < st.pcnt;
        __syncwarp();
        d0 = D.dirTab[lane];
        d1 = lane + 32u < kDirTab ? D.dirTab[lane + 32u] : 0u;
    }
    if (cur || prev) {
        SysDev const& S = kMulti ? Sm[kMulti ? wid : 0] : S1;
        uint32_t listLen = 0;
        uint32_t const nAcc = __reduce_add_sync(
            0xffffffffu,
            perform_tile<W, Q>(S, dtabs[wid], d0, d1, p, tile, cur, prev, sub, (uint32_t)G, listLen));
        uint32_t const stripe = (blockIdx.x * PW + wid) % kStatSlots;
        // the tile's list length (its tentative moves) is counted once, by the group's first warp
        if (lane == 0 && sub == 0 && listLen)
            atomicAdd(S.stats + kStatSlots + stripe, (unsigned long long)listLen);
        if (lane == 0 && nAcc) atomicAdd(S.stats + 2 * kStatSlots + stripe, (unsigned long long)nAcc);
    }
    if (writer) write_next_step(S1.gen, gen, S1.grp, next);
}

// ---------------------------------------------------------------------------------- persistent

// A wait longer than this is a fault. The CTAs of a cooperative launch start together, once all of them have
// an SM (B200: behind a kernel that holds 100 SMs for 50 ms all 148 start within 10 us of its end, behind
// another cooperative launch they never start between its CTAs), so other streams' kernels delay a launch
// but none of its waits. kBarrierPolls bounds a wait without the timer (as many polls take longer).
constexpr unsigned long long kBarrierTimeoutNs = 2000000000ull;
constexpr unsigned int kBarrierPolls = 1u << 24;

__device__ __forceinline__ unsigned int ld_acquire_gpu(unsigned int const* p)
{
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One thread of each CTA, after a CTA barrier that ordered the CTA's earlier writes before it: adds
// the CTA's arrival to a count that only grows (a release add) and waits with acquire loads until
// the count reaches this barrier's target, nCtas above the previous one (the first one's is
// base + nCtas). Nothing is reset between barriers, and the signed difference keeps the comparison right
// across a wrap of the count. The wait is bounded by time and by a poll count; false if it ran out or
// another CTA's did (GridSync::fault): the kernel then leaves, and the host reports the fault.
__device__ __forceinline__ bool grid_meet(GridSync* gs, unsigned int& target, unsigned int nCtas)
{
    target += nCtas;
    red_release_gpu_add(&gs->count, 1u);
    if (int(ld_acquire_gpu(&gs->count) - target) < 0) {
        unsigned long long const t0 = global_ns();
        unsigned int polls = 0u;
        while (int(ld_acquire_gpu(&gs->count) - target) < 0) {
            // a time limit, and a poll count as a second bound that does not trust the timer
            if ((++polls & 255u) == 0u) {
                if (ld_acquire_gpu(&gs->fault) != 0u) return false;
                if (global_ns() - t0 > kBarrierTimeoutNs || polls > kBarrierPolls) {
                    gs->fault = 1u;
                    return false;
                }
            }
            __nanosleep(20);
        }
    }
    return true;
}

// The two halves of a cluster barrier: after the first every earlier access of the thread is on its
// way, after the second those of all threads of the cluster are in place.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Slab layout (slab_sweep): CTA r of C holds, of every colour group of n slots in
// chunks of 32, chunks [r nch / C, (r + 1) nch / C), nch = ceil(n / 32): contiguous slots, in the
// group's order, so the neighbours of a chain numbered along its bonds mostly lie in the same CTA.
struct SlabPart {
    uint32_t first[kSlabColors], count[kSlabColors], base[kSlabColors];   // first slot, slots, local index
};

// A code word's top bit in shared memory (above the fields and the count): some neighbour of the slot
// lies in another CTA, so its code word lives in global memory, where that CTA can change it.
template <typename W>
__device__ __forceinline__ constexpr W slab_shared_flag()
{
    return W(1) << (8 * sizeof(W) - 1);
}

// Local index of slot g in this CTA, or kNoMark if another CTA holds it.
__device__ __forceinline__ uint32_t slab_local(SlabPart const& P, uint32_t nColors, uint32_t g)
{
    for (uint32_t c = 0; c < nColors; ++c) {
        uint32_t const d = g - P.first[c];
        if (d < P.count[c]) return P.base[c] + d;
    }
    return kNoMark;
}

// An 8-byte load where `on`, else 0, as one predicated instruction: the loads of a plane go out back
// to back. Coherent with other CTAs' writes after a grid barrier (its acquire drops the L1's lines),
// cached in the L1 within a phase.
__device__ __forceinline__ unsigned long long load_if(unsigned long long const* p, bool on)
{
    unsigned long long v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u64 %0, 0;\n\t@q ld.global.u64 %0, [%1];\n\t}"
                 : "=l"(v)
                 : "l"(p), "r"((uint32_t)on)
                 : "memory");
    return v;
}
// The set cells of the plane in lattice L (0 where not live).
__device__ __forceinline__ unsigned long long plane_hits(PlaneRef const& r, bool live, unsigned long long const* L)
{
    unsigned long long v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = load_if(L + r.w[k], live && r.m[k] != 0ull);
    return (v[0] & r.m[0]) | (v[1] & r.m[1]) | (v[2] & r.m[2]) | (v[3] & r.m[3]);
}

// Shared memory of a CTA of the slab sweeps: cap slots in all, capG of the largest colour group.
__host__ __device__ __forceinline__ size_t slab_layout(uint32_t cap, uint32_t capG, bool clearAll, bool cache,
                                                       uint32_t maxc, uint32_t codeBytes)
{
    return 768 * 8 + kDirTab * 4 + (size_t)cap * (codeBytes + 4) + (size_t)capG * (clearAll ? 4 : 8) + 512 +
           (cache ? (size_t)cap * 4 + (size_t)maxc * cap * 2 : 0);
}
// Slots a CTA of C holds at most of all colour groups and of the largest one, and the system's slots.
template <typename F>
__host__ __device__ __forceinline__ void slab_caps(F size, uint32_t nColors, uint32_t C, uint32_t& cap, uint32_t& capG,
                                                   uint32_t& n)
{
    cap = capG = n = 0;
    for (uint32_t c = 0; c < nColors; ++c) {
        uint32_t const own = 32u * ((((size(c) + 31u) >> 5) + C - 1u) / C);
        cap += own;
        capG = capG > own ? capG : own;
        n += size(c);
    }
}
// Dense systems clear the temporary lattice whole: nwords x 8 B written in order, against one scattered
// write per mark. The two draw level at about two words per slot (us per MCS, whole and per mark: 128^3 at 6.3
// words per slot 7.72 and 7.42, 3.1 7.75 and 7.67, 2.0 7.68 and 7.68, 1.6 7.61 and 7.63; 256^3 at 6.3 8.22 and 7.92,
// 2.0 8.32 and 8.26, 1.25 8.75 and 8.71, 0.6 10.25 and 10.31, 0.3 14.23 and 14.37).
__host__ __device__ __forceinline__ bool slab_clear_all(uint32_t nwords, uint32_t nSlots) { return nwords <= 2u * nSlots; }

// The sweep of one system by C CTAs (this one's rank among them), a whole run of sub-steps in one launch.
// Lattice and temporary lattices stay in global memory (the L2); each CTA keeps the lattice addresses and
// code words of its slots (SlabPart) in shared memory. Per sub-step two barriers of the CTAs: after the
// check (every mark is set) and after the perform (the lattice is settled). The last warp sees the CTA's
// writes through and waits; the others meanwhile do all of the next phase that depends on this CTA's own
// slots only: bond tests, candidates and their planes before the check's lattice reads; the list of
// movers, their codes, neighbour references and planes, the clearing of the previous marks and the
// directions of the next sub-step before the perform's temporary-lattice reads. What is left between two
// barriers is one round of L2 reads and the writes that follow from it.
//   kCache: the slots' inner direction hashes and neighbour references in shared memory too.
// The CTAs are part of a cooperative launch and meet at a count in global memory (S.gs). A thread-block
// cluster and its barrier in hardware were no faster (131K monomers on 16 CTAs 9.7 us per sub-step
// against 8.9: every warp's wait drops the SM's L1 lines), and its CTAs have to fit one GPC.
// kIdle: entries may be idle (kNoColor). cap, capG: slots of a CTA in all and of the largest colour group,
// at most (slab_caps). The waiter fetches the step entries a block ahead, during a perform.
// Bound: on the 256^3 melt (N = 1,048,576, 148 CTAs) by the scattered L2 accesses (about 0.8 loads and
// 0.57 atomics per clock and SM), the integer pipe and instruction issue (24 K warp instructions per SM
// and sub-step); below 200K monomers by the barriers (1.3-1.8 us each with the writes before them) and
// one L2 round trip after each. Per MCS: melt 14.9 us (graph of launches 21.7), 131K monomers 9.6 (13.4;
// 15 with the cooperative sweep that kept every record in global memory), 60K 8.6 (15.2).
// 640 threads: 20 warps of 96 registers hold two prepared candidates per thread (the melt has 1.9
// per thread) and its movers fit one pass; 512 threads took 17.6 us per MCS there, 768 16.3, 1024 18.
// CTAs with at most kSlabSmallSlots slots per colour have 256: fewer warps meet faster at the CTA's own
// barriers (131K monomers 9.0 against 9.6 us per MCS, 210K 9.3 against 9.9, 60K 7.9 against 8.5).
template <typename W, int B, bool kCache, bool kIdle>
__device__ __forceinline__ void slab_sweep(SysDev const& S, StepSource const& src, StepStream const& own,
                                           uint32_t sysId, uint32_t nSteps, uint32_t C, uint32_t rank, uint32_t cap, uint32_t capG, bool clearAll,
                                           GridFault* report)
{
    constexpr uint32_t kSlots = CodeWord<W>::kSlots;
    constexpr W kShared = slab_shared_flag<W>();
    constexpr uint32_t nWork = B / 32 - 1, kThreads = nWork * 32;   // the last warp waits at the barriers
    constexpr uint32_t kGroup = 3;   // slots of a thread worked on together, so that their latencies overlap
    constexpr uint32_t kDirs = 9;    // directions (3 bits each) a thread keeps at a time
    constexpr int kPre = 2;          // candidates of a thread prepared ahead of the barrier
    constexpr uint32_t kEntMask = (1u << kSlabEntBits) - 1u;   // list entries: index in the part | dir << kSlabEntBits
    constexpr uint32_t kRefBits = slab_ref_bits(sizeof(W) == 8), kRefMask = (1u << kRefBits) - 1u, kAway = 0xFFFFu;
    constexpr uint32_t kFarBit = 1u << 31;
    __shared__ SlabPart P;
    __shared__ __align__(16) StepEntry stepSm[2][kStepBlock];   // the block of entries in use, and the next
    __shared__ uint32_t nCand, nMov, tallyA;
    extern __shared__ unsigned long long smem[];
    uint32_t const tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    bool const waiter = warp == nWork;
    GridSync* const gs = S.gs;
    // an earlier launch failed: the state is not usable, and this run's caller learns of it too (asked here, and in
    // a batch's launch with the tables' barrier: the other way round the kernels were built 0.6 and 1.3 % slower)
    if constexpr (!kIdle) {
        if (__syncthreads_or(tid == 0 && ld_acquire_gpu(&gs->fault) != 0u) != 0) {
            if (tid == 0) report->fault = 1u;   // (where: the barrier it failed at, where the report is the same)
            return;
        }
    }
    uint32_t const nColors = S.nColors, np = S.npad;
    if (tid == 0) {
        uint32_t b = 0;
        for (uint32_t c = 0; c < nColors; ++c) {
            uint32_t const nch = (S.grp[2 * c + 1] + 31u) >> 5;
            uint32_t const lo = rank * nch / C, hi = (rank + 1u) * nch / C;
            P.first[c] = S.grp[2 * c] + 32u * lo;
            P.count[c] = 32u * (hi - lo);
            P.base[c] = b;
            b += 32u * (hi - lo);
        }
        nCand = nMov = tallyA = 0u;
    }
    unsigned long long* const ptab = smem;                                   // 768 plane masks
    uint32_t* const dtab = reinterpret_cast<uint32_t*>(smem + 768);          // kDirTab words
    W* const code = reinterpret_cast<W*>(smem + 768 + kDirTab / 2);          // cap slots
    uint32_t* const pk = reinterpret_cast<uint32_t*>(code + cap);            // cap slots
    uint16_t* const cand = reinterpret_cast<uint16_t*>(pk + cap);            // capG candidates
    uint16_t* const list = cand + capG;                                      // capG movers
    uint32_t* const tgt = reinterpret_cast<uint32_t*>(list + capG);          // !clearAll: capG marked addresses
    uint8_t* const mok = reinterpret_cast<uint8_t*>(tgt + (clearAll ? 0u : capG));   // 512 move-table bytes
    uint32_t* const inner = reinterpret_cast<uint32_t*>(mok + 512);          // kCache: cap hashes
    uint16_t* const refs = reinterpret_cast<uint16_t*>(inner + cap);         // kCache: maxc x cap references
    for (uint32_t w = tid; w < 768; w += B) ptab[(w & 2u ? 384u : 0u) + (w >> 2) * 2u + (w & 1u)] = S.planeTab[w];
    if (tid < kDirTab) dtab[tid] = S.dirTab[tid];
    for (uint32_t w = tid; w < 512; w += B) mok[w] = S.moveOk[w];
    if constexpr (kIdle) {
        if (__syncthreads_or(tid == 0 && ld_acquire_gpu(&gs->fault) != 0u) != 0) {
            if (tid == 0) report->fault = 1u;   // (where: the barrier it failed at, where the report is the same)
            return;
        }
    } else {
        __syncthreads();
    }
    using RV = typename SlotRec<W>::V;
    for (uint32_t c = 0; c < nColors; ++c)
        for (uint32_t d = tid; d < P.count[c]; d += B) {
            uint32_t const g = P.first[c] + d, l = P.base[c] + d;
            RV const r = reinterpret_cast<RV const*>(S.rec)[g];
            W cw = rec_code_of(r);
            uint32_t const n = uint32_t(cw >> CodeWord<W>::kCountShift) & 7u;
            for (uint32_t q = 0; q < n; ++q) {
                uint32_t const ref = S.nbrr[(size_t)q * np + g], at = slab_local(P, nColors, ref & kSlotMask);
                if (at == kNoMark) cw |= kShared;
                if (kCache) refs[q * cap + l] = at == kNoMark ? kAway : at | ((ref >> kSlotShift) << kRefBits);
            }
            code[l] = cw;
            pk[l] = r.x;
            if (kCache) inner[l] = move_hash(g - S.grp[2 * c]);
        }
    __syncthreads();
    if (kCache) {
        // a neighbour held here whose code word other CTAs change too lives in global memory as well
        for (uint32_t c = 0; c < nColors; ++c)
            for (uint32_t d = tid; d < P.count[c]; d += B) {
                uint32_t const l = P.base[c] + d, n = uint32_t(code[l] >> CodeWord<W>::kCountShift) & 7u;
                for (uint32_t q = 0; q < n; ++q) {
                    uint32_t const r = refs[q * cap + l];
                    if (r != kAway && (code[r & kRefMask] & kShared) != W(0)) refs[q * cap + l] = kAway;
                }
            }
        __syncthreads();
    }
    // neighbour q of slot g (local index l): the local index of its slot | its reverse slot << kSlotShift,
    // or the slot itself with kFarBit where its code word lives in global memory
    auto neighbour = [&](uint32_t q, uint32_t g, uint32_t l) {
        if (kCache) {
            uint32_t const r = refs[q * cap + l];
            if (r != kAway) return (r & kRefMask) | ((r >> kRefBits) << kSlotShift);
            return __ldg(S.nbrr + (size_t)q * np + g) | kFarBit;
        }
        uint32_t const ref = __ldg(S.nbrr + (size_t)q * np + g), at = slab_local(P, nColors, ref & kSlotMask);
        if (at == kNoMark || (code[at] & kShared) != W(0)) return ref | kFarBit;
        return at | ((ref >> kSlotShift) << kSlotShift);
    };
    // directions of this thread's slots tid + k kThreads of the part, k from k0, of a sub-step
    auto directions = [&](StepEntry const& e, uint32_t k0) {
        uint32_t const n = P.count[e.color], i0 = P.first[e.color] - e.off;
        uint32_t const* const h = inner + P.base[e.color];
        uint32_t d = 0;
        for (uint32_t k = 0, i = tid + k0 * kThreads; k < kDirs && i < n; k += kGroup) {
#pragma unroll
            for (uint32_t q = 0; q < kGroup; ++q, i += kThreads) {
                uint32_t const in = kCache ? h[i < n ? i : tid] : move_hash(i0 + i);
                d |= (move_hash(in ^ e.seed) % 6u) << (3u * (k + q));
            }
        }
        return d;
    };
    // a warp's append: the place of each lane with `on` in a list whose length is *count
    uint32_t const lanesBelow = (1u << lane) - 1u;
    auto append = [&](bool on, uint32_t* count) {
        uint32_t const bal = __ballot_sync(0xffffffffu, on);
        uint32_t at = 0;
        if (lane == 0) at = shared_add(count, (uint32_t)__popc(bal));
        return __shfl_sync(0xffffffffu, at, 0) + __popc(bal & lanesBelow);
    };
    // a barrier of the CTAs in two halves, between which the workers prepare; a CTA barrier comes before
    // the first. The waiter alone carries the CTA's writes over (it orders them after the CTA barrier)
    unsigned int target = gs->base;   // (the waiter's) count target of the next barrier
    auto meet_begin = [&]() {   // false on the waiter if a wait ran out
        bool met = true;
        if (waiter && lane == 0) met = grid_meet(gs, target, C);
        __syncwarp();
        return met;
    };
    auto meet_end = [&](bool met) {   // whether every CTA came
        if (__syncthreads_or(!met) == 0) return true;
        if (waiter && lane == 0) *report = GridFault{1u, (target - gs->base) / C};
        return false;
    };
    bool const walled = S.walls != 0u;
    uint32_t const cw0 = (uint32_t)((uint64_t)S.nwords * rank / C), cw1 = (uint32_t)((uint64_t)S.nwords * (rank + 1u) / C);
    uint32_t prevMov = 0u, nAcc = 0u, nTent = 0u, par = 0u, dirs = 0u;
    bool began = false, drawn = false;   // a sub-step has run; dirs belong to the next one
    unsigned long long att = 0ull;
    auto fetch_steps = [&](uint32_t block) {   // the waiter's lanes
        uint32_t const t = block * kStepBlock + lane;
        if (lane < kStepBlock && t < nSteps) stepSm[block & 1u][lane] = step_entry(src, own, sysId, t, S.grp, nColors);
    };
    if (waiter) {
        fetch_steps(0);
        fetch_steps(1);
    }
    __syncthreads();
    for (uint32_t t = 0; t < nSteps; ++t) {
        StepEntry const st = stepSm[t / kStepBlock & 1u][t % kStepBlock];
        StepEntry const& next = stepSm[(t + 1u) / kStepBlock & 1u][(t + 1u) % kStepBlock];
        // the block before the one in use has been read by all: the next one takes its place
        bool const refill = t != 0 && t % kStepBlock == 0;
        if (kIdle && st.color == kNoColor) {
            if (refill) {   // (the same on every thread)
                __syncthreads();
                if (waiter) fetch_steps(t / kStepBlock + 1u);
                __syncthreads();
            }
            continue;
        }
        par = st.parity;
        att += st.cnt;
        uint32_t const first = P.first[st.color], base = P.base[st.color];
        unsigned long long* const tcur = S.tmp + (size_t)par * S.nwords;
        // check, part 1 (own slots only): walls and bonds -> candidates, and their planes
        uint32_t nc = 0, ent[kPre], to[kPre], far = 0u, go = 0u;   // far, go: bit q, candidate q
        PlaneRef pr[kPre];
        auto candidate = [&](bool live, uint32_t e, uint32_t& en, uint32_t& target1, PlaneRef& r) {
            en = live ? cand[e] : 0u;
            uint32_t const l = base + (en & kEntMask), p = pk[l], dir = en >> kSlabEntBits;
            DirParams const D = dir_params(dtab, dir);
            plane_ref(r, ptab, D, p, D.front, dir);
            target1 = addr_add(p, D.ma, D.step);
            return (code[l] & kShared) != W(0);
        };
        // the bond test of a candidate whose code word lives in global memory
        auto far_ok = [&](uint32_t en) {
            return bonds_ok<W, true>(__ldcg(rec_code<W>(S.rec, first + (en & kEntMask))), en >> kSlabEntBits, mok);
        };
        if (waiter && lane == 0) nMov = 0u;
        bool met = began ? meet_begin() : true;
        if (!waiter) {
            if (!drawn) dirs = directions(st, 0);
            // slots held here, and those before the group's end (the last chunk may be padded)
            uint32_t const n = P.count[st.color], left = min(n, st.cnt - (first - st.off));
            uint32_t const t0 = warp * 32u;   // (n is a multiple of 32: a warp's slots end together)
            for (uint32_t k = 0; t0 + k * kThreads < n; k += kGroup) {
                if (k != 0 && k % kDirs == 0) dirs = directions(st, k);
                W cw[kGroup];
                uint32_t bal[kGroup], dir[kGroup], total = 0;
#pragma unroll
                for (uint32_t q = 0; q < kGroup; ++q) {
                    uint32_t const i = tid + (k + q) * kThreads;
                    cw[q] = i < n ? code[base + i] : W(0);
                    dir[q] = dirs & 7u;
                    dirs >>= 3;
                }
#pragma unroll
                for (uint32_t q = 0; q < kGroup; ++q) {
                    uint32_t const i = tid + (k + q) * kThreads;
                    bool ok = bonds_ok<W, true>(cw[q], dir[q], mok) || (cw[q] & kShared) != W(0);
                    ok = ok && i < left;
                    if (walled && ok) {
                        uint2 const mw = make_uint2(dtab[dir[q] * 4u], dtab[kDirHalf + dir[q] * 4u + 3u]);   // Ma, wall
                        ok = (pk[base + i] & mw.x) != mw.y;
                    }
                    bal[q] = __ballot_sync(0xffffffffu, ok);
                    total += __popc(bal[q]);
                }
                uint32_t at = 0;
                if (lane == 0) at = shared_add(&nCand, total);
                at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
                for (uint32_t q = 0; q < kGroup; ++q) {
                    if ((bal[q] >> lane) & 1u)
                        cand[at + __popc(bal[q] & lanesBelow)] =
                            (uint16_t)((tid + (k + q) * kThreads) | (dir[q] << kSlabEntBits));
                    at += __popc(bal[q]);
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");   // the working warps
            nc = nCand;
#pragma unroll
            for (int q = 0; q < kPre; ++q) {
                // (a thread without a candidate takes entry 0's slot, and its answer is not used)
                bool const live = q * kThreads + tid < nc;
                if (q * kThreads + t0 < nc && candidate(live, q * kThreads + tid, ent[q], to[q], pr[q]) && live)
                    far |= 1u << q;
            }
        }
        if (began) {
            if (!meet_end(met)) return;
        } else {
            __syncthreads();
        }
        began = true;
        // check, part 2: the front planes; free candidates mark their target
        if (!waiter) {
            uint32_t const w0 = warp * 32u;   // (the tests on it are the same for the whole warp)
            unsigned long long hit[kPre];
#pragma unroll
            for (int q = 0; q < kPre; ++q)
                if (q * kThreads + w0 < nc) hit[q] = plane_hits(pr[q], q * kThreads + tid < nc, S.lat);
#pragma unroll
            for (int q = 0; q < kPre; ++q)
                if (q * kThreads + tid < nc && hit[q] == 0ull && (!((far >> q) & 1u) || far_ok(ent[q]))) {
                    atomicOr(tcur + (to[q] >> 6), 1ull << (to[q] & 63u));
                    go |= 1u << q;
                }
            for (uint32_t e0 = kPre * kThreads + w0; e0 < nc; e0 += kThreads) {
                uint32_t en = 0, target1 = 0;
                PlaneRef r;
                bool ok = e0 + lane < nc;
                bool const f = candidate(ok, e0 + lane, en, target1, r);
                ok = ok && plane_hits(r, ok, S.lat) == 0ull && (!f || far_ok(en));
                if (ok) atomicOr(tcur + (target1 >> 6), 1ull << (target1 & 63u));
                uint32_t const at = append(ok, &nMov);
                if (ok) list[at] = (uint16_t)en;
            }
        }
        __syncthreads();
        // perform, part 1: the movers, and what they need besides the temporary lattice
        uint32_t nm = 0, mL = 0, mTo = 0, mW0 = 0, mW1 = 0, nb[kSlots];
        W moved = W(0), flip[kSlots];
        unsigned long long mB0 = 0ull, mB1 = 0ull;
        PlaneRef mr{};
        bool mFar = false;
        int32_t wraps = -1;   // the periodic axis the move wraps, + 4 going up
        auto fetch = [&](uint32_t e) {
            uint32_t const en = list[e], dir = en >> kSlabEntBits, g = first + (en & kEntMask);
            mL = base + (en & kEntMask);
            DirParams const D = dir_params(dtab, dir);
            uint32_t const from = pk[mL];
            mTo = addr_add(from, D.ma, D.step);
            plane_ref(mr, ptab, D, mTo, D.step, dir);
            W own = code[mL];
            mFar = (own & kShared) != W(0);
            if (mFar) own = __ldcg(rec_code<W>(S.rec, g));
            W f;
            moved = code_move(own, dir, f);
            uint32_t const n = uint32_t(own >> CodeWord<W>::kCountShift) & 7u;
#pragma unroll
            for (uint32_t q = 0; q < kSlots; ++q) {
                flip[q] = W(0);
                if (q < n) {
                    nb[q] = neighbour(q, g, mL);
                    flip[q] = code_flip(f, q, (nb[q] >> kSlotShift) & 7u);
                }
            }
            mW0 = from >> 6;
            mW1 = mTo >> 6;
            mB0 = 1ull << (from & 63u);
            mB1 = 1ull << (mTo & 63u);
            if (mW0 == mW1) {
                mB0 |= mB1;
                mB1 = 0ull;
            }
            wraps = (((dir & 1u) ? mTo : from) & D.ma) == 0u ? int32_t((dir >> 1) | ((dir & 1u) << 2)) : -1;
        };
        if (waiter && lane == 0) nCand = 0u;
        met = meet_begin();
        drawn = t + 1 < nSteps && (!kIdle || next.color != kNoColor);
        if (!waiter) {
            if (warp * 32u < nc) {
                static_assert(kPre == 2, "the candidates of a warp go to the list together");
                uint32_t const b0 = __ballot_sync(0xffffffffu, go & 1u), b1 = __ballot_sync(0xffffffffu, go & 2u);
                uint32_t at = 0;
                if (lane == 0) at = shared_add(&nMov, (uint32_t)(__popc(b0) + __popc(b1)));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (go & 1u) list[at + __popc(b0 & lanesBelow)] = (uint16_t)ent[0];
                if (go & 2u) list[at + __popc(b0) + __popc(b1 & lanesBelow)] = (uint16_t)ent[1];
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
            nm = nMov;
            if (tid < nm) fetch(tid);
            unsigned long long* const tprev = S.tmp + (size_t)(par ^ 1u) * S.nwords;
            if (clearAll) {
                for (uint32_t w = cw0 + tid; w < cw1; w += kThreads) tprev[w] = 0ull;
            } else {
                for (uint32_t e = tid; e < prevMov || e < nm; e += kThreads) {
                    if (e < prevMov) tprev[tgt[e] >> 6] = 0ull;
                    if (e < nm) {
                        uint32_t const en = list[e];
                        DirParams const D = dir_params(dtab, en >> kSlabEntBits);
                        tgt[e] = addr_add(pk[base + (en & kEntMask)], D.ma, D.step);
                    }
                }
            }
            if (drawn) dirs = directions(next, 0);
        }
        if (!meet_end(met)) return;
        // perform, part 2: front planes on the temporary lattice; the free movers move
        if (!waiter) {
            for (uint32_t e = tid; e < nm; e += kThreads) {
                if (e != tid) fetch(e);
                if (plane_hits(mr, true, tcur) != 0ull) continue;
                ++nAcc;
                atomicXor(S.lat + mW0, mB0);
                if (mB1 != 0ull) atomicXor(S.lat + mW1, mB1);
                pk[mL] = mTo;
                if (mFar) *rec_code<W>(S.rec, first + (mL - base)) = moved;
                else code[mL] = moved;
#pragma unroll
                for (uint32_t q = 0; q < kSlots; ++q) {
                    if (flip[q] == W(0)) continue;
                    if (nb[q] & kFarBit) atomicXor(rec_code<W>(S.rec, nb[q] & kSlotMask), flip[q]);
                    else shared_xor(code + (nb[q] & kSlotMask), flip[q]);
                }
                if (wraps >= 0) {   // about one move in a lattice side: the image offset changes
                    int32_t const a = wraps & 3, side = int32_t(S.mask[a] + 1u);
                    atomicAdd((a == 0 ? S.x : (a == 1 ? S.y : S.z)) + first + (mL - base), (wraps & 4) ? side : -side);
                }
            }
        }
        if (waiter && refill) fetch_steps(t / kStepBlock + 1u);
        nTent += nm;
        prevMov = nm;
        __syncthreads();   // this CTA's slots are settled for the next check's first part
    }
    // every perform has read the last marks: zero them, and write the slots back
    if (began && !meet_end(meet_begin())) return;
    if (began && rank == 0 && waiter && lane == 0) gs->base = target;   // (every CTA has read it)
    unsigned long long* const tlast = S.tmp + (size_t)par * S.nwords;
    if (clearAll) {
        for (uint32_t w = cw0 + tid; w < cw1; w += B) tlast[w] = 0ull;
    } else if (!waiter) {
        for (uint32_t e = tid; e < prevMov; e += kThreads) tlast[tgt[e] >> 6] = 0ull;
    }
    for (uint32_t c = 0; c < nColors; ++c)
        for (uint32_t d = tid; d < P.count[c]; d += B) {
            uint32_t const g = P.first[c] + d, l = P.base[c] + d;
            if ((code[l] & kShared) != W(0)) *rec_pk<W>(S.rec, g) = pk[l];   // its code word is in place
            else reinterpret_cast<RV*>(S.rec)[g] = make_rec(pk[l], code[l]);
        }
    uint32_t const asum = __reduce_add_sync(0xffffffffu, nAcc);
    if (lane == 0 && asum) atomicAdd(&tallyA, asum);
    __syncthreads();
    if (tid == 0) {
        tally_flush(nTent, S.stats, 1);
        tally_flush(tallyA, S.stats, 2);
        if (rank == 0 && att) atomicAdd(S.stats, att);
    }
}

template <typename W, int B, bool kCache>
__global__ void __launch_bounds__(B, 1)
    k_slab_bc(const __grid_constant__ SysDev S, const __grid_constant__ StepSource src, uint32_t nSteps, uint32_t cap,
              uint32_t capG, uint32_t clearAll, GridFault* report)
{
    slab_sweep<W, B, kCache, false>(S, src, src.own, 0u, nSteps, gridDim.x, blockIdx.x, cap, capG, clearAll != 0u,
                                    report);
}

// Many systems in one cooperative launch: CTA b runs share refs[b].rank of system refs[b].sys with the
// other CTAs of that system, and waits for no others; the reports are report[system].
template <typename W, int B>
__global__ void __launch_bounds__(B, 1)
    k_slab_batch_bc(SysDev const* __restrict__ sysv, SlabRef const* __restrict__ refs,
                    const __grid_constant__ StepSource src, uint32_t nSteps, GridFault* report)
{
    __shared__ SysDev S;
    __shared__ StepStream own;
    __shared__ uint32_t caps[3];
    SlabRef const r = refs[blockIdx.x];
    if (threadIdx.x == 0) own = step_stream(src, r.sys);
    copy_desc(S, sysv + r.sys);
    __syncthreads();
    if (threadIdx.x == 0)
        slab_caps([&](uint32_t c) { return S.grp[2 * c + 1]; }, S.nColors, r.ctas, caps[0], caps[1], caps[2]);
    if (threadIdx.x == 32) step_stream_from(own, src.first);
    __syncthreads();
    slab_sweep<W, B, true, true>(S, src, own, r.sys, nSteps, r.ctas, r.rank, caps[0], caps[1],
                                 slab_clear_all(S.nwords, caps[2]), report + r.sys);
}

// ---------------------------------------------------------------------------------- resident

// Half bricks: the kernels that keep the lattices in shared memory read them as 32-bit words of
// 4 x 4 x 2 cells (word a >> 5 of lattice address a; the z axis's in-word coordinate has one bit). A
// front plane still touches at most 2 x 2 of them, with half the bytes of the lattice and of the
// masks to read: shared-memory wavefronts (bank conflicts of random words) bound those kernels, and a
// plane on 64-bit words took 52 of a warp's 80 per check, on half bricks 25. Marks and flips
// are 32-bit atomics (shared memory has no native 64-bit ones).
constexpr uint32_t kHalfPlanes = 3 * 32;   // table entries of four masks: axis, in-word position

// Entry e of the mask table: for the axis e >> 5 and the first cell's position e & 31 in its word, the
// plane's cells in the word itself and its neighbours along v, u, and both (front_plane_words' order).
__device__ __forceinline__ uint4 half_plane_masks(uint32_t e)
{
    uint32_t const a = e >> 5, u = a == 0 ? 1u : 0u, v = a == 2 ? 1u : 2u;
    uint32_t m[4] = {0u, 0u, 0u, 0u};
    for (uint32_t k = 0; k < 9; ++k) {
        uint32_t const c[3] = {e & 3u, (e >> 2) & 3u, (e >> 4) & 1u}, size[3] = {4u, 4u, 2u};
        uint32_t w = 0, bit = 0;
        for (uint32_t ax = 0; ax < 3; ++ax) {
            uint32_t const at = c[ax] + (ax == u ? k % 3u : 0u) + (ax == v ? k / 3u : 0u);
            if (at >= size[ax]) w |= ax == u ? 2u : 1u;
            bit |= (at % size[ax]) << (2u * ax);
        }
        for (uint32_t j = 0; j < 4; ++j)
            if (w == j) m[j] |= 1u << bit;
    }
    return make_uint4(m[0], m[1], m[2], m[3]);
}

// The tables of the kernels with half bricks, by the CTA's threads: masks, and the direction table
// with the u and v masks of a half-brick index in place of those of a brick index.
__device__ __forceinline__ void half_tables(SysDev const& S, uint4* masks, uint32_t* dtab)
{
    for (uint32_t e = threadIdx.x; e < kHalfPlanes; e += blockDim.x) masks[e] = half_plane_masks(e);
    if (threadIdx.x < kDirTab) {
        uint32_t const w = threadIdx.x, d = w % 24u / 4u, k = w % 4u;
        bool const uv = w >= kDirHalf && (k == 1u || k == 2u);
        dtab[w] = uv ? S.dirTab[d * 4u + k + 1u] >> 5 : S.dirTab[w];
    }
}

// The set cells of the front plane of a move along dir in lattice L of half bricks (front_plane's
// arguments): all four words are read, each is a word of the lattice.
struct HalfPlane {
    uint32_t w[4];
    uint4 m;
};
__device__ __forceinline__ void half_plane(HalfPlane& r, uint4 const* masks, DirParams const& D, uint32_t base,
                                           uint32_t da, uint32_t dir)
{
    uint32_t const f = ((((base | ~D.ma) + da) & D.ma) | (((base | ~D.mu) + D.mu) & D.mu)) |
                       (((base | ~D.mv) + D.mv) & D.mv);
    r.w[0] = f >> 5;
    r.w[1] = addr_add(r.w[0], D.bv, 1u);
    r.w[2] = addr_add(r.w[0], D.bu, 1u);
    r.w[3] = addr_add(r.w[2], D.bv, 1u);
    r.m = masks[(dir >> 1) * 32u + (f & 31u)];
}
__device__ __forceinline__ uint32_t half_hits(HalfPlane const& r, uint32_t const* L)
{
    return (L[r.w[0]] & r.m.x) | (L[r.w[1]] & r.m.y) | (L[r.w[2]] & r.m.z) | (L[r.w[3]] & r.m.w);
}

// Shared memory of k_resident_bc (resident_bc_smem_bytes); nb: neighbour references kept here (0: they
// stay in global memory).
__host__ __device__ __forceinline__ size_t resident_layout(uint32_t nwords, uint32_t npad, uint32_t maxGroup,
                                                           uint32_t codeBytes, uint32_t nb)
{
    return kHalfPlanes * 16 + kDirTab * 4 + (size_t)nwords * 3 * 8 + (size_t)npad * (codeBytes + 4) + 512 +
           (size_t)((maxGroup + 1u) & ~1u) * 4 + (size_t)nb * npad * 2;
}

// The whole system in one CTA's shared memory for nSteps sub-steps: lattice, one temporary
// lattice per sub-step parity (the previous one cleared while the next check runs), lattice
// addresses, bond codes, neighbour references (where they fit: 2 bytes each) and lists; one CTA per
// system of sysList.
// The bond test and the front plane's masks are read side by side, so that their chains of dependent
// reads overlap, the lattice only for slots that pass the test: two thirds of a melt's do not, and their
// reads cost more in bank conflicts than the wait for the test. The directions of sub-step t + 1 are
// drawn during the perform of t, whose movers take the threads from the last one down, where a small
// system has no slots.
// Two forms of the check:
//   kDirect: each slot's bonds and plane by its own thread, two CTA barriers per sub-step (groups of at
//   most 1024 slots, and those too large for 16-bit list entries);
//   else the slots that pass the wall and bond tests (a third of a melt's) are listed first, so the
//   planes run on full warps: three barriers, and less work from 2 slots per thread on.
// Bound by shared-memory wavefronts (bank conflicts), the integer pipe and the chain of dependent reads
// of each phase (1.2K monomers: about 1700 cycles of a sub-step in the check, 1300 in the perform). us per
// MCS, with every slot's plane read and so: 1.2K-monomer chains 3.4 and 3.3, 1.6K 3.9 and 3.6, 2K 4.3 and
// 4.1; 3.3K 5.3, 8K 10.6. Slower: each thread performing its own mover, all but the temporary lattice
// read before the barrier and no list (3 %, issue); the movers spread over more warps (20 %).
template <typename W, bool kDirect>
__global__ void __launch_bounds__(kResidentBlock, 1) k_resident_bc(SysDev const* __restrict__ sysv,
                                                                    uint32_t const* __restrict__ sysList,
                                                                    StepSource const src, uint32_t nSteps)
{
    constexpr uint32_t kSlots = CodeWord<W>::kSlots, B = kResidentBlock, kDirs = 10;
    constexpr uint32_t kRefBits = slab_ref_bits(sizeof(W) == 8), kRefMask = (1u << kRefBits) - 1u;
    __shared__ SysDev S;
    __shared__ __align__(16) StepEntry stepSm[kStepBlock];
    __shared__ StepStream own;
    __shared__ uint32_t nMov[2], nCand, maxGroup;   // nMov: per sub-step parity
    extern __shared__ unsigned long long smem[];
    uint32_t const sysId = sysList[blockIdx.x];
    if (threadIdx.x == 0) own = step_stream(src, sysId);
    copy_desc(S, sysv + sysId);
    __syncthreads();
    if (threadIdx.x == 32) step_stream_from(own, src.first);   // (read after the next barrier)
    uint32_t const nw = S.nwords, np = S.npad, maxc = S.maxc;
    uint32_t const tid = threadIdx.x, lane = tid & 31u;
    if (tid == 0) {
        uint32_t m = 0;
        for (uint32_t c = 0; c < S.nColors; ++c) m = max(m, S.grp[2 * c + 1]);
        maxGroup = m;
        nMov[0] = nMov[1] = nCand = 0u;
    }
    __syncthreads();
    uint4* const masks = reinterpret_cast<uint4*>(smem);    // kHalfPlanes entries
    uint32_t* const dtab = reinterpret_cast<uint32_t*>(masks + kHalfPlanes);   // kDirTab words (16-byte aligned)
    uint32_t* const lat = dtab + kDirTab;                   // 2 nw half bricks
    uint32_t* const tmp = lat + 2u * nw;                    // twice 2 nw half bricks (per sub-step parity)
    W* const code = reinterpret_cast<W*>(tmp + 4u * nw);
    uint32_t* const pk = reinterpret_cast<uint32_t*>(code + np);
    uint8_t* const mok = reinterpret_cast<uint8_t*>(pk + np);   // 512 move-table bytes
    uint32_t const mg = (maxGroup + 1u) & ~1u;
    // kDirect: movers, slot | dir << 28; else candidates and movers, index in the group | dir << 13
    uint32_t* const list = reinterpret_cast<uint32_t*>(mok + 512);
    uint16_t* const cand = reinterpret_cast<uint16_t*>(list);
    uint16_t* const movers = cand + mg;
    uint16_t* const refs = movers + mg;                     // maxc x np references, where they fit
    uint32_t dynBytes;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dynBytes));
    bool const cached = np < (1u << kRefBits) && resident_layout(nw, np, maxGroup, sizeof(W), maxc) <= dynBytes;
    half_tables(S, masks, dtab);
    for (uint32_t w = tid; w < 512; w += B) mok[w] = S.moveOk[w];
    for (uint32_t w = tid; w < 2u * nw; w += B) {
        lat[w] = reinterpret_cast<uint32_t const*>(S.lat)[w];
        tmp[w] = 0u;
        tmp[2u * nw + w] = 0u;
    }
    for (uint32_t g = tid; g < np; g += B) {
        code[g] = *rec_code<W>(S.rec, g);
        pk[g] = *rec_pk<W>(S.rec, g);
    }
    if (cached)
        for (uint32_t g = tid; g < maxc * np; g += B) {   // reference q of slot g at q np + g, as in nbrr
            uint32_t const r = S.nbrr[g];
            refs[g] = (uint16_t)((r & kSlotMask) | ((r >> kSlotShift) << kRefBits));
        }
    uint32_t nAcc = 0, nTent = 0;
    unsigned long long nAtt = 0;
    bool const walled = S.walls != 0u;

    uint32_t const lanesBelow = (1u << lane) - 1u;
    auto append = [&](bool on, uint32_t* count) {
        uint32_t const bal = __ballot_sync(0xffffffffu, on);
        uint32_t at = 0;
        if (lane == 0) at = shared_add(count, (uint32_t)__popc(bal));
        return __shfl_sync(0xffffffffu, at, 0) + __popc(bal & lanesBelow);
    };
    // directions of in-colour indices tid + k B, k from k0, 3 bits each
    auto directions = [&](StepEntry const& e, uint32_t k0) {
        uint32_t d = 0;
        for (uint32_t k = 0, i = tid + k0 * B; k < kDirs && i < e.cnt; ++k, i += B) d |= move_dir(i, e.seed) << (3u * k);
        return d;
    };
    // the check of slot l: the move's target, and whether the front plane is free and, if asked, the
    // wall and bond tests pass; only slots that pass them read the lattice
    auto check = [&](uint32_t l, uint32_t dir, bool tests, uint32_t& to) {
        uint32_t const p = pk[l];
        DirParams const D = dir_params(dtab, dir);
        bool const ok = !tests || (bonds_ok<W, true>(code[l], dir, mok) & ((p & D.ma) != D.wall));
        HalfPlane pl;
        half_plane(pl, masks, D, p, D.front, dir);
        to = addr_add(p, D.ma, D.step);
        if (!ok) return false;
        return half_hits(pl, lat) == 0u;
    };
    uint32_t par = 0, dirs = 0;
    bool drawn = false;   // dirs belong to the next active sub-step
    for (uint32_t t = 0; t < nSteps; ++t) {
        if (t % kStepBlock == 0) {   // (the last barrier of the sub-step before ended the reads of the old ones)
            uint32_t const n = min(kStepBlock, nSteps - t);
            if (tid < n) stepSm[tid] = step_entry(src, own, sysId, t + tid, S.grp, S.nColors);
            __syncthreads();   // (the first also publishes the state loaded above)
            drawn = false;
        }
        uint32_t const ts = t % kStepBlock;
        StepEntry const st = stepSm[ts];
        if (st.color == kNoColor) continue;
        if (!drawn) dirs = directions(st, 0);
        nAtt += st.cnt;
        uint32_t* const marks = tmp + par * 2u * nw;
        uint32_t const cnt = st.cnt, off = st.off;
        if (kDirect) {
            for (uint32_t k = 0, i0 = tid & ~31u; i0 < cnt; ++k, i0 += B) {   // warp-uniform
                if (k != 0 && k % kDirs == 0) dirs = directions(st, k);
                uint32_t const i = i0 + lane, dir = dirs & 7u, l = off + min(i, cnt - 1u);
                dirs >>= 3;
                uint32_t to;
                bool const go = check(l, dir, true, to) & (i < cnt);
                if (go) atomicOr(marks + (to >> 5), 1u << (to & 31u));
                uint32_t const at = append(go, &nMov[par]);
                if (go) list[at] = l | (dir << kSlotShift);
            }
        } else {
            for (uint32_t k = 0, i0 = tid & ~31u; i0 < cnt; ++k, i0 += B) {
                if (k != 0 && k % kDirs == 0) dirs = directions(st, k);
                uint32_t const i = i0 + lane, dir = dirs & 7u, l = off + min(i, cnt - 1u);
                dirs >>= 3;
                bool ok = bonds_ok<W, true>(code[l], dir, mok) & (i < cnt);
                if (walled) {
                    uint2 const mw = make_uint2(dtab[dir * 4u], dtab[kDirHalf + dir * 4u + 3u]);   // Ma, wall
                    ok = ok & ((pk[l] & mw.x) != mw.y);
                }
                uint32_t const at = append(ok, &nCand);
                if (ok) cand[at] = (uint16_t)(i | (dir << kSlabEntBits));
            }
        }
        // the previous sub-step's marks and mover count: read by no thread after the barrier that
        // ended that sub-step, written by none before the barrier that ends this check
        for (uint32_t w = B - 1u - tid; w < nw; w += B)
            reinterpret_cast<unsigned long long*>(tmp + (par ^ 1u) * 2u * nw)[w] = 0ull;
        if (tid == 0) nMov[par ^ 1u] = 0u;
        if (!kDirect) {
            __syncthreads();
            uint32_t const nc = nCand;
            for (uint32_t e0 = tid & ~31u; e0 < nc; e0 += B) {
                bool const live = e0 + lane < nc;
                uint32_t const en = live ? cand[e0 + lane] : 0u;
                uint32_t to;
                bool const go = check(off + (en & ((1u << kSlabEntBits) - 1u)), en >> kSlabEntBits, false, to) & live;
                if (go) atomicOr(marks + (to >> 5), 1u << (to & 31u));
                uint32_t const at = append(go, &nMov[par]);
                if (go) movers[at] = (uint16_t)en;
            }
        }
        __syncthreads();
        // perform over the movers
        uint32_t const n = nMov[par];
        if (!kDirect && tid == 0) nCand = 0u;
        for (uint32_t e = B - 1u - tid; e < n; e += B) {
            uint32_t l, dir;
            if (kDirect) {
                l = list[e] & kSlotMask;
                dir = list[e] >> kSlotShift;
            } else {
                l = off + (movers[e] & ((1u << kSlabEntBits) - 1u));
                dir = movers[e] >> kSlabEntBits;
            }
            uint32_t const p = pk[l];
            W const own = code[l];
            uint32_t const nn = uint32_t(own >> CodeWord<W>::kCountShift) & 7u;
            uint32_t nb[kSlots];
#pragma unroll
            for (uint32_t q = 0; q < kSlots; ++q) {
                nb[q] = 0u;
                if (q < maxc) {
                    if (cached) {
                        uint32_t const r = refs[q * np + l];
                        nb[q] = (r & kRefMask) | ((r >> kRefBits) << kSlotShift);
                    } else if (q < nn) {
                        nb[q] = __ldg(S.nbrr + (size_t)q * np + l);
                    }
                }
            }
            DirParams const D = dir_params(dtab, dir);
            uint32_t const to = addr_add(p, D.ma, D.step);
            HalfPlane pl;
            half_plane(pl, masks, D, to, D.step, dir);
            W flip;
            W const moved = code_move(own, dir, flip);
            if (half_hits(pl, marks) != 0u) continue;
            atomicXor(lat + (p >> 5), 1u << (p & 31u));
            atomicXor(lat + (to >> 5), 1u << (to & 31u));
            pk[l] = to;
            code[l] = moved;
#pragma unroll
            for (uint32_t q = 0; q < kSlots; ++q) {
                W const f = code_flip(flip, q, nb[q] >> kSlotShift);
                if (f != W(0)) shared_xor(code + (nb[q] & kSlotMask), f);   // (f is 0 past the last bond)
            }
            image_step(S, l, dir >> 1, (dir & 1u) ? 1 : -1, p, to, D.ma);
            ++nAcc;
        }
        nTent += n;
        drawn = t + 1 < nSteps && ts + 1u < kStepBlock && stepSm[ts + 1u].color != kNoColor;
        if (drawn) dirs = directions(stepSm[ts + 1u], 0);
        __syncthreads();   // every perform is done: the lattice is settled for the next check
        par ^= 1u;
    }
    __syncthreads();   // (a run that ended with idle sub-steps)
    for (uint32_t w = tid; w < 2u * nw; w += B) reinterpret_cast<uint32_t*>(S.lat)[w] = lat[w];
    for (uint32_t g = tid; g < np; g += B) {
        *rec_code<W>(S.rec, g) = code[g];
        *rec_pk<W>(S.rec, g) = pk[g];
    }
    uint32_t const asum = __reduce_add_sync(0xffffffffu, nAcc);
    if (lane == 0) tally_flush(asum, S.stats, 2);
    if (tid == 0) {
        tally_flush(nTent, S.stats, 1);
        if (nAtt) atomicAdd(S.stats + (blockIdx.x % kStatSlots), nAtt);
    }
}

// ---------------------------------------------------------------------------------- cluster-resident

// Distributed shared memory: the address of p (this CTA's shared memory) in the CTA of the given
// rank, a read, and atomics without result where `on`. All are 32 bits wide: 64-bit bitwise atomics on
// another CTA's shared memory (through map_shared_rank, or atom.shared::cluster.*.b64) were measured
// on a B200 to lose updates when several CTAs hit the same word, 32-bit ones are exact.
__device__ __forceinline__ uint32_t cluster_map(uint32_t sharedAddr, uint32_t rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(sharedAddr), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t cluster_load(uint32_t a, bool on)
{
    uint32_t v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u32 %0, 0;\n\t@q ld.shared::cluster.u32 %0, [%1];\n\t}"
                 : "=r"(v) : "r"(a), "r"((uint32_t)on) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_or(uint32_t a, uint32_t v, bool on)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;\n\t}"
                 :: "r"(a), "r"(v), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void cluster_xor(uint32_t a, uint32_t v, bool on)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q red.relaxed.cluster.shared::cluster.xor.b32 [%0], %1;\n\t}"
                 :: "r"(a), "r"(v), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void cluster_xor(uint32_t a, unsigned long long v, bool on)
{
    cluster_xor(a, (uint32_t)v, on && (uint32_t)v != 0u);
    cluster_xor(a + 4u, (uint32_t)(v >> 32), on && (v >> 32) != 0ull);
}
// Shared memory of k_cluster_bc per CTA (cluster_bc_smem_bytes); nb: neighbour references kept here (0:
// they stay in global memory).
__host__ __device__ __forceinline__ size_t cluster_layout(uint32_t nwords, uint32_t npad, uint32_t logC,
                                                          uint32_t groupSlots, uint32_t codeBytes, uint32_t nb)
{
    size_t const cap = cluster_slots_per_cta(npad, logC);
    return kHalfPlanes * 16 + kDirTab * 4 + (size_t)(nwords >> logC) * 3 * 8 + cap * (codeBytes + 4) + 512 +
           (size_t)groupSlots * 4 + cap * nb * 4;
}

// One thread-block cluster of 2^logC CTAs (kBlock threads each) owns a system whose lattice,
// temporary lattices, addresses and codes fit their shared memory together, for a whole run of
// sub-steps (half bricks dealt out as cluster_word_rank says, slots as cluster_slot_rank). Each CTA
// checks the slots it holds, lists its own tentative movers and performs them; words and
// neighbours' codes held by another CTA are reached through distributed shared memory, the
// neighbours' at addresses mapped once. Two cluster barriers per sub-step (after the check, after the
// perform); the temporary lattice has one copy per sub-step parity. Between the two halves of the
// first barrier a CTA clears its words of the previous copy, draws the directions of the next sub-step and
// makes the step entries a block ahead (made at the start of their block, with a barrier and the first
// directions after them, they took 4 % of the run), which nobody waits for. Every CTA of a cluster runs the same system and so reaches the
// same barriers. A CTA leaves only after the last barrier, when no other CTA accesses its shared
// memory any more. Grid: one cluster per system of sysList. K: chunks of 32 slots per warp and colour, at most.
// CTAs of at most 32 chunks per colour have 512 threads: half of the warps of 1024 had nothing to do but
// arrive at the barriers (8K chains, 8 chunks per CTA, 5.5 -> 5.0 us per MCS on 512 threads, 5.1 on 256; 16K,
// 16 chunks, 7.2 -> 6.7, 7.2 on 256; 26K, 26 chunks, 9.8 -> 9.2 with two chunks per warp).
// Bound by remote accesses (0.33 remote atomics per clock and SM), two barriers of 0.3 us and the
// chain of dependent reads of each phase; a lattice word is read only where the bond test passed and the
// plane touches it. us per MCS, 16 CTAs: 4K chains 4.3, 8K 5.0, 16K 6.7, the 11K network 6.2.
template <typename W, int K, int kBlock>
__global__ void __launch_bounds__(kBlock, 1) k_cluster_bc(SysDev const* __restrict__ sysv,
                                                          uint32_t const* __restrict__ sysList,
                                                          StepSource const src, uint32_t nSteps)
{
    namespace cg = cooperative_groups;
    constexpr uint32_t kSlots = CodeWord<W>::kSlots, B = kBlock, kFetchWarp = B / 64 - 1;
    static_assert(K <= 10, "a thread's directions share one word, three bits each");
    cg::cluster_group cluster = cg::this_cluster();
    uint32_t const C = cluster.num_blocks(), rank = cluster.block_rank();
    uint32_t logC = 0;
    while ((1u << logC) < C) ++logC;   // a power of two (launch_cluster_bc)
    __shared__ SysDev S;
    __shared__ __align__(16) StepEntry stepSm[2][kStepBlock];   // the block of entries in use, and the next
    __shared__ StepStream own;
    __shared__ uint32_t nMov[2];   // per sub-step parity
    extern __shared__ unsigned long long smem[];
    uint32_t const sysId = sysList[blockIdx.x >> logC];
    if (threadIdx.x == 0) own = step_stream(src, sysId);
    copy_desc(S, sysv + sysId);
    __syncthreads();
    if (threadIdx.x == 32) step_stream_from(own, src.first);   // (read after the next barrier)
    uint32_t const np = S.npad, nwC = S.nwords >> logC, cap = cluster_slots_per_cta(np, logC), maxc = S.maxc;
    uint32_t const tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint4* const masks = reinterpret_cast<uint4*>(smem);                     // kHalfPlanes entries
    uint32_t* const dtab = reinterpret_cast<uint32_t*>(masks + kHalfPlanes); // kDirTab words
    uint32_t* const lat = dtab + kDirTab;                                    // 2 nwC half bricks
    uint32_t* const tmp = lat + 2u * nwC;                                    // twice 2 nwC half bricks
    W* const code = reinterpret_cast<W*>(tmp + 4u * nwC);                    // cap slots
    uint32_t* const pk = reinterpret_cast<uint32_t*>(code + cap);            // cap slots
    uint8_t* const mok = reinterpret_cast<uint8_t*>(pk + cap);               // 512 move-table bytes
    uint32_t* const list = reinterpret_cast<uint32_t*>(mok + 512);           // K x B movers: local slot | dir << 28
    uint32_t* const refs = list + K * B;                                     // maxc x cap references, where they fit
    uint32_t dynBytes;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dynBytes));
    bool const cached = cluster_layout(S.nwords, np, logC, K * B, sizeof(W), maxc) <= dynBytes;
    uint32_t const latAddr = (uint32_t)__cvta_generic_to_shared(lat), tmpAddr = (uint32_t)__cvta_generic_to_shared(tmp),
                   codeAddr = (uint32_t)__cvta_generic_to_shared(code);
    // neighbour reference (slot | reverse slot << 28): the mapped address of its code word, with the
    // reverse slot (0-2, or 0-5 with 64-bit codes) in the low bits the word's alignment leaves free
    auto mapped = [&](uint32_t ref) {
        uint32_t const g = ref & kSlotMask;
        return cluster_map(codeAddr + cluster_slot_local(g, logC) * (uint32_t)sizeof(W), cluster_slot_rank(g, logC)) |
               (ref >> kSlotShift);
    };
    half_tables(S, masks, dtab);
    for (uint32_t w = tid; w < 512; w += B) mok[w] = S.moveOk[w];
    for (uint32_t l = tid; l < 2u * nwC; l += B) {
        lat[l] = reinterpret_cast<uint32_t const*>(S.lat)[(l << logC) | rank];
        tmp[l] = 0u;
        tmp[2u * nwC + l] = 0u;
    }
    for (uint32_t l = tid; l < cap; l += B) {
        uint32_t const g = cluster_slot_of(l, rank, logC);
        bool const in = g < np;
        code[l] = in ? *rec_code<W>(S.rec, g) : W(0);
        pk[l] = in ? *rec_pk<W>(S.rec, g) : 0u;
        if (cached)
            for (uint32_t q = 0; q < maxc; ++q) refs[q * cap + l] = in ? mapped(S.nbrr[(size_t)q * np + g]) : 0u;
    }
    if (tid < 2) nMov[tid] = 0u;
    cluster.sync();   // every CTA's part of the state is in place before any remote access

    auto wordAt = [&](uint32_t base, uint32_t w) {
        return cluster_map(base + 4u * cluster_word_local(w, logC), cluster_word_rank(w, logC));
    };
    auto hits = [&](HalfPlane const& r, uint32_t base, bool on) {
        uint32_t const v0 = cluster_load(wordAt(base, r.w[0]), on), v1 = cluster_load(wordAt(base, r.w[1]), on && r.m.y),
                       v2 = cluster_load(wordAt(base, r.w[2]), on && r.m.z), v3 = cluster_load(wordAt(base, r.w[3]), on && r.m.w);
        return (v0 & r.m.x) | (v1 & r.m.y) | (v2 & r.m.z) | (v3 & r.m.w);
    };
    // this warp's chunks of a colour group (which starts at a chunk): the k-th starts at slot
    // chunk(e) * 32 + k * B C
    auto chunk = [&](StepEntry const& e) {
        uint32_t const c0 = e.off >> 5;
        return c0 + ((rank - c0) & (C - 1u)) + warp * C;
    };
    auto directions = [&](StepEntry const& e) {
        uint32_t const c = chunk(e), i0 = c * 32u + lane - e.off;
        uint32_t d = 0;
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)K; ++k) {
            uint32_t const i = i0 + k * B * C;
            if (i - lane >= e.cnt) break;   // the same for the whole warp
            d |= move_dir(i, e.seed) << (3u * k);
        }
        return d;
    };
    uint32_t const lanesBelow = (1u << lane) - 1u;
    uint32_t nTent = 0, nAcc = 0, par = 0, dirs = 0;
    bool drawn = false;   // dirs belong to the next active sub-step
    unsigned long long nAtt = 0;
    auto fetch_steps = [&](uint32_t block) {   // one warp
        uint32_t const k = tid - kFetchWarp * 32u, t = block * kStepBlock + k;
        if (k < kStepBlock && t < nSteps) stepSm[block & 1u][k] = step_entry(src, own, sysId, t, S.grp, S.nColors);
    };
    fetch_steps(0);
    fetch_steps(1);
    __syncthreads();
    for (uint32_t t = 0; t < nSteps; ++t) {
        StepEntry const st = stepSm[t / kStepBlock & 1u][t % kStepBlock];
        StepEntry const& next = stepSm[(t + 1u) / kStepBlock & 1u][(t + 1u) % kStepBlock];
        // the block before the one in use has been read by all: the next one takes its place
        bool const refill = t != 0 && t % kStepBlock == 0;
        if (st.color == kNoColor) {
            if (refill) {   // (the same on every thread)
                __syncthreads();
                fetch_steps(t / kStepBlock + 1u);
                __syncthreads();
            }
            continue;
        }
        if (!drawn) dirs = directions(st);
        if (rank == 0) nAtt += st.cnt;
        uint32_t const marks = tmpAddr + par * 8u * nwC;
        // check: this warp's chunks of the colour group
        uint32_t const end = st.off + st.cnt, c0 = chunk(st);
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)K; ++k) {
            uint32_t const g = (c0 + k * (B / 32u) * C) * 32u + lane;
            if (g - lane >= end) break;   // the same for the whole warp
            uint32_t const l = cluster_slot_local(g, logC), dir = (dirs >> (3u * k)) & 7u, p = pk[l];
            DirParams const D = dir_params(dtab, dir);
            bool const ok = bonds_ok<W, true>(code[l], dir, mok) & ((p & D.ma) != D.wall) & (g < end);
            HalfPlane pl;
            half_plane(pl, masks, D, p, D.front, dir);
            uint32_t const to = addr_add(p, D.ma, D.step);
            bool const go = ok & (hits(pl, latAddr, ok) == 0u);
            cluster_or(wordAt(marks, to >> 5), 1u << (to & 31u), go);
            uint32_t const bal = __ballot_sync(0xffffffffu, go);
            uint32_t at = 0;
            if (lane == 0) at = shared_add(&nMov[par], (uint32_t)__popc(bal));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & lanesBelow);
            if (go) list[at] = l | (dir << kSlotShift);
        }
        cluster_arrive();   // this CTA's marks are on their way
        // the previous sub-step's marks and mover count: no CTA reads them after the barrier that
        // ended that sub-step, and none writes them before the barrier that ends this one
        for (uint32_t w = B - 1u - tid; w < nwC; w += B)
            reinterpret_cast<unsigned long long*>(tmp + (par ^ 1u) * 2u * nwC)[w] = 0ull;
        if (tid == 0) nMov[par ^ 1u] = 0u;
        drawn = t + 1 < nSteps && next.color != kNoColor;
        if (drawn) dirs = directions(next);
        if (refill) fetch_steps(t / kStepBlock + 1u);
        cluster_wait();   // every CTA's marks are in place
        // perform over this CTA's movers, from the last thread down
        uint32_t const n = nMov[par];
        for (uint32_t e = B - 1u - tid; e < n; e += B) {
            uint32_t const l = list[e] & kSlotMask, dir = list[e] >> kSlotShift, p = pk[l];
            W const own = code[l];
            uint32_t const nn = uint32_t(own >> CodeWord<W>::kCountShift) & 7u;
            uint32_t nb[kSlots];
#pragma unroll
            for (uint32_t q = 0; q < kSlots; ++q) {
                nb[q] = 0u;
                if (q < nn)
                    nb[q] = cached ? refs[q * cap + l]
                                   : mapped(__ldg(S.nbrr + (size_t)q * np + cluster_slot_of(l, rank, logC)));
            }
            DirParams const D = dir_params(dtab, dir);
            uint32_t const to = addr_add(p, D.ma, D.step);
            HalfPlane pl;
            half_plane(pl, masks, D, to, D.step, dir);
            W flip;
            W const moved = code_move(own, dir, flip);
            bool const free = hits(pl, marks, true) == 0u;
            cluster_xor(wordAt(latAddr, p >> 5), 1u << (p & 31u), free);
            cluster_xor(wordAt(latAddr, to >> 5), 1u << (to & 31u), free);
#pragma unroll
            for (uint32_t q = 0; q < kSlots; ++q)
                cluster_xor(nb[q] & ~(uint32_t)(sizeof(W) - 1), code_flip(flip, q, nb[q] & (uint32_t)(sizeof(W) - 1)),
                            free && q < nn);
            if (free) {
                pk[l] = to;
                code[l] = moved;
                image_step(S, cluster_slot_of(l, rank, logC), dir >> 1, (dir & 1u) ? 1 : -1, p, to, D.ma);
                ++nAcc;
            }
        }
        nTent += n;
        cluster_arrive();
        cluster_wait();   // every perform is done: the lattice is settled for the next check
        par ^= 1u;
    }
    // after the last cluster barrier no CTA reaches into another's shared memory
    for (uint32_t l = tid; l < 2u * nwC; l += B) reinterpret_cast<uint32_t*>(S.lat)[(l << logC) | rank] = lat[l];
    for (uint32_t l = tid; l < cap; l += B) {
        uint32_t const g = cluster_slot_of(l, rank, logC);
        if (g < np) {
            *rec_code<W>(S.rec, g) = code[l];
            *rec_pk<W>(S.rec, g) = pk[l];
        }
    }
    uint32_t const asum = __reduce_add_sync(0xffffffffu, nAcc);
    if (lane == 0) tally_flush(asum, S.stats, 2);
    if (tid == 0) {
        tally_flush(nTent, S.stats, 1);
        if (nAtt) atomicAdd(S.stats + (blockIdx.x % kStatSlots), nAtt);
    }
}

// ---------------------------------------------------------------------------------- launchers

namespace {

// CTAs per SM the compiler must fit (register budget) for check / perform: shape 0 leaves the
// registers free (64 / 80), 1 asks 6 / 5 (40 / 48), 2 asks 6 / 6, 3 (the default) asks 7 / 5: the
// check at 32 registers with a 20-byte spill runs the 1024 tiles of the 256^3 melt in one wave
// (7 x 148 CTAs), 4-5 % faster than shape 1. A launch names its shape (Batch::autotune picks one);
// a negative shape means the default, which the environment variable BFM_GRID_SHAPE can change.
int default_grid_shape()
{
    static int const shape = [] {
        char const* e = std::getenv("BFM_GRID_SHAPE");
        int const v = e ? std::atoi(e) : 3;
        return (v >= 0 && v < kGridShapes) ? v : 3;
    }();
    return shape;
}

// SMs of the current device (cached per device)
int sm_count()
{
    static thread_local int count[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 148;
    int& c = count[dev & 63];
    if (!c && cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) c = 148;
    return c;
}

// the perform's warps per CTA and per tile: BFM_PERFORM_WARPS (1, 2, 4, 8) and BFM_PERFORM_GROUP
// (1, 2, 4, 8; at most the warps per CTA) override the defaults
int perform_env(char const* name, int dflt, int maxv)
{
    char const* e = std::getenv(name);
    int const v = e ? std::atoi(e) : dflt;
    return (v == 1 || v == 2 || v == 4 || v == 8) && v <= maxv ? v : dflt;
}
int perform_warps()
{
    static int const w = perform_env("BFM_PERFORM_WARPS", (int)kPerformWarpsDefault, 8);
    return w;
}
int perform_group()
{
    static int const g = std::min(perform_env("BFM_PERFORM_GROUP", (int)kPerformGroupDefault, 8), perform_warps());
    return g;
}

template <typename W, bool kMulti, int PW, int G>
void launch_perform_k(SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles,
                      StepEntry const* dSteps, PerformArgs const& pa, cudaStream_t s)
{
    uint32_t const tilesPerCta = PW / G;
    k_perform_bc<W, kMulti, PW, G><<<(nTiles + tilesPerCta - 1) / tilesPerCta, 32 * PW, 0, s>>>(
        hostDesc, dSys, dTiles, dSteps, pa.parity, pa.scope, pa.next, nTiles);
}

template <typename W, bool kMulti, int PW>
void launch_perform_g(SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles,
                      StepEntry const* dSteps, PerformArgs const& pa, cudaStream_t s)
{
    int const g = pa.group > 0 ? pa.group : perform_group();
    if (g >= 8 && PW >= 8) launch_perform_k<W, kMulti, PW, (PW >= 8 ? 8 : 1)>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s);
    else if (g >= 4 && PW >= 4) launch_perform_k<W, kMulti, PW, (PW >= 4 ? 4 : 1)>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s);
    else if (g >= 2 && PW >= 2) launch_perform_k<W, kMulti, PW, (PW >= 2 ? 2 : 1)>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s);
    else launch_perform_k<W, kMulti, PW, 1>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s);
}

template <typename W, bool kMulti, int B, int kMinCheck>
void launch_grid_bc_k(bool check, SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles,
                      uint32_t nTiles, StepEntry const* dSteps, PerformArgs const& pa, cudaStream_t s)
{
    if (check) {
        k_check_bc<W, B, kMulti, kMinCheck><<<nTiles, B, 0, s>>>(hostDesc, dSys, dTiles, dSteps, pa.snap);
        return;
    }
    switch (pa.warps > 0 ? pa.warps : perform_warps()) {
    case 1: launch_perform_g<W, kMulti, 1>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    case 2: launch_perform_g<W, kMulti, 2>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    case 8: launch_perform_g<W, kMulti, 8>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    default: launch_perform_g<W, kMulti, 4>(hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    }
}

// shape: the check's register budget in resident threads per SM, 0: the compiler's choice, 1: 1536,
// 2: 1280, 3: 1792 (the default; BFM_GRID_SHAPE overrides it); block: the check's CTA size (128, 256
// or 512 threads over the same 512-monomer tile). The perform (one warp per tile) has one form.
template <typename W, bool kMulti, int B>
void launch_grid_bc_b(bool check, SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles,
                      uint32_t nTiles, StepEntry const* dSteps, PerformArgs const& pa, int shape, cudaStream_t s)
{
    switch (shape < 0 ? default_grid_shape() : shape) {
    case 1: launch_grid_bc_k<W, kMulti, B, 1536 / B>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    case 2: launch_grid_bc_k<W, kMulti, B, 1280 / B>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    case 3: launch_grid_bc_k<W, kMulti, B, 1792 / B>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    default: launch_grid_bc_k<W, kMulti, B, 1>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, s); break;
    }
}

template <typename W, bool kMulti>
void launch_grid_bc_m(bool check, SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles,
                      uint32_t nTiles, StepEntry const* dSteps, PerformArgs const& pa, int shape, int block,
                      cudaStream_t s)
{
    if (!check) {   // the perform's form does not depend on shape or block
        launch_grid_bc_k<W, kMulti, 256, 1>(false, hostDesc, dSys, dTiles, nTiles, dSteps, pa, s);
        return;
    }
    if (block == 128) launch_grid_bc_b<W, kMulti, 128>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape, s);
    else if (block == 512) launch_grid_bc_b<W, kMulti, 512>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape, s);
    else launch_grid_bc_b<W, kMulti, 256>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape, s);
}

template <typename W>
cudaError_t launch_grid_bc(bool check, SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles,
                           uint32_t nTiles, StepEntry const* dSteps, PerformArgs const& pa, int shape, int block,
                           cudaStream_t s)
{
    if (shape >= kGridShapes || !check_block_ok(block) || !perform_shape_ok(pa.warps, pa.group))
        return cudaErrorInvalidValue;
    if (dTiles) launch_grid_bc_m<W, true>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape, block, s);
    else launch_grid_bc_m<W, false>(check, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape, block, s);
    return cudaGetLastError();
}

}  // namespace

std::vector<TileRef> perform_tile_list(std::vector<TileRef> const& tiles)
{
    // the perform takes one tile per warp, like the check's list
    std::vector<TileRef> out(tiles);
    for (auto& t : out) t.count = 1;
    return out;
}

cudaError_t launch_check_bc(SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles,
                            StepEntry const* dSteps, uint32_t codeMode, cudaStream_t s, int shape, int block,
                            unsigned long long* snap)
{
    if (nTiles == 0) return cudaSuccess;
    if (dTiles && snap) return cudaErrorInvalidValue;   // snapshots are taken for one system only
    PerformArgs none{};
    none.snap = snap;
    if (block <= 0) block = (int)kCheckBlockDefault;
    if (codeMode == kCode32)
        return launch_grid_bc<uint32_t>(true, hostDesc, dSys, dTiles, nTiles, dSteps, none, shape, block, s);
    if (codeMode == kCode64)
        return launch_grid_bc<unsigned long long>(true, hostDesc, dSys, dTiles, nTiles, dSteps, none, shape, block, s);
    return cudaErrorInvalidValue;
}

cudaError_t launch_perform_bc(SysDev const& hostDesc, SysDev const* dSys, TileRef const* dTiles, uint32_t nTiles,
                              StepEntry const* dSteps, uint32_t codeMode, cudaStream_t s, int shape,
                              PerformArgs const& pa)
{
    if (nTiles == 0) return cudaSuccess;
    if (codeMode == kCode32)
        return launch_grid_bc<uint32_t>(false, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape,
                                        (int)kCheckBlockDefault, s);
    if (codeMode == kCode64)
        return launch_grid_bc<unsigned long long>(false, hostDesc, dSys, dTiles, nTiles, dSteps, pa, shape,
                                                  (int)kCheckBlockDefault, s);
    return cudaErrorInvalidValue;
}

bool slab_plan(uint32_t const* grpSize, uint32_t nColors, uint32_t maxc, uint32_t nwords, uint32_t codeMode,
               uint32_t ctas, SlabPlan& plan)
{
    plan = SlabPlan{};
    if (codeMode == kCodeNone || nColors == 0 || nColors > kSlabColors || ctas == 0) return false;
    uint32_t cap, capG, n;
    slab_caps([&](uint32_t c) { return grpSize[c]; }, nColors, ctas, cap, capG, n);
    if (capG > 1u << kSlabEntBits) return false;
    uint32_t const w = codeMode == kCode64 ? 8 : 4;
    bool const clearAll = slab_clear_all(nwords, n);
    size_t const least = slab_layout(cap, capG, clearAll, false, maxc, w), all = slab_layout(cap, capG, clearAll, true, maxc, w);
    if (least > kSlabMaxSmem) return false;
    bool const cache = all <= kSlabMaxSmem && cap < (1u << slab_ref_bits(w == 8));
    uint32_t const threads = cache && capG <= kSlabSmallSlots ? kSlabBlockSmall : (w == 8 ? kSlabBlock64 : kSlabBlock32);
    plan = SlabPlan{ctas, cap, capG, threads, clearAll, cache, cache ? all : least};
    return true;
}

uint32_t slab_ctas(uint32_t maxGroup, uint32_t sms)
{
    return std::min(sms, std::max(1u, (((maxGroup + 31u) >> 5) + kSlabMinChunks - 1u) / kSlabMinChunks));
}

namespace {

template <typename W, int B, bool kCache>
cudaError_t launch_slab_bc_w(SysDev const& S, StepSource src, uint32_t nSteps, SlabPlan const& plan,
                             GridFault* report, cudaStream_t s)
{
    static thread_local bool done[64] = {};
    cudaError_t const e = allow_smem(k_slab_bc<W, B, kCache>, done);
    if (e != cudaSuccess) return e;
    uint32_t cap = plan.cap, perCta = plan.perCta, clearAll = plan.clearAll ? 1u : 0u;
    void* args[] = {const_cast<SysDev*>(&S), &src, &nSteps, &cap, &perCta, &clearAll, &report};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void const*>(k_slab_bc<W, B, kCache>), dim3(plan.ctas), dim3(B),
                                       args, plan.smem, s);
}

// Calls f.operator()<W, B, kCache>() for a code mode and a plan.
template <typename W, int B, typename F>
auto slab_dispatch_w(SlabPlan const& plan, F f)
{
    if (plan.threads == kSlabBlockSmall) return f.template operator()<W, (int)kSlabBlockSmall, true>();
    return plan.cache ? f.template operator()<W, B, true>() : f.template operator()<W, B, false>();
}
template <typename F>
auto slab_dispatch(uint32_t codeMode, SlabPlan const& plan, F f)
{
    return codeMode == kCode64 ? slab_dispatch_w<unsigned long long, (int)kSlabBlock64>(plan, f)
                               : slab_dispatch_w<uint32_t, (int)kSlabBlock32>(plan, f);
}

struct SlabLaunch {
    SysDev const& S;
    StepSource const& src;
    uint32_t nSteps;
    SlabPlan const& plan;
    GridFault* report;
    cudaStream_t s;
    template <typename W, int B, bool kCache>
    cudaError_t operator()() const { return launch_slab_bc_w<W, B, kCache>(S, src, nSteps, plan, report, s); }
};

struct SlabPerSm {
    SlabPlan const& plan;
    template <typename W, int B, bool kCache>
    uint32_t operator()() const
    {
        static thread_local bool done[64] = {};
        int n = 0;
        if (allow_smem(k_slab_bc<W, B, kCache>, done) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_slab_bc<W, B, kCache>, B, plan.smem) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return (uint32_t)n;
    }
};

template <typename W, int B>
cudaError_t launch_slab_batch_w(SysDev const* dSys, SlabRef const* dRefs, uint32_t ctas, size_t smem, StepSource src,
                                uint32_t nSteps, GridFault* report, cudaStream_t s)
{
    static thread_local bool done[64] = {};
    cudaError_t const e = allow_smem(k_slab_batch_bc<W, B>, done);
    if (e != cudaSuccess) return e;
    void* args[] = {&dSys, &dRefs, &src, &nSteps, &report};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void const*>(k_slab_batch_bc<W, B>), dim3(ctas), dim3(B), args,
                                       smem, s);
}

}  // namespace

uint32_t slab_ctas_per_sm(SlabPlan const& plan, uint32_t codeMode)
{
    return plan.ctas == 0 || codeMode == kCodeNone ? 0u : slab_dispatch(codeMode, plan, SlabPerSm{plan});
}

cudaError_t launch_slab_bc(SysDev const& hostDesc, StepSource const& src, uint32_t nSteps, SlabPlan const& plan,
                           GridFault* report, uint32_t codeMode, cudaStream_t s)
{
    if (nSteps == 0) return cudaSuccess;
    if (plan.ctas == 0 || codeMode == kCodeNone || nSteps > kLaunchSteps) return cudaErrorInvalidValue;
    return slab_dispatch(codeMode, plan, SlabLaunch{hostDesc, src, nSteps, plan, report, s});
}

cudaError_t launch_slab_batch(SysDev const* dSys, SlabRef const* dRefs, uint32_t ctas, size_t smem,
                              StepSource const& src, uint32_t nSteps, GridFault* report, uint32_t codeMode,
                              cudaStream_t s)
{
    if (ctas == 0 || nSteps == 0) return cudaSuccess;
    if (nSteps > kLaunchSteps) return cudaErrorInvalidValue;
    if (codeMode == kCode32)
        return launch_slab_batch_w<uint32_t, (int)kSlabBlock32>(dSys, dRefs, ctas, smem, src, nSteps, report, s);
    if (codeMode == kCode64)
        return launch_slab_batch_w<unsigned long long, (int)kSlabBlock64>(dSys, dRefs, ctas, smem, src, nSteps, report, s);
    return cudaErrorInvalidValue;
}

size_t resident_bc_smem_bytes(uint32_t nwords, uint32_t npad, uint32_t maxGroup, uint32_t maxc, uint32_t codeMode)
{
    uint32_t const w = codeMode == kCode64 ? 8 : 4;
    size_t const all = resident_layout(nwords, npad, maxGroup, w, maxc);
    return all <= kResidentMaxSmem ? all : resident_layout(nwords, npad, maxGroup, w, 0);
}

namespace {

template <typename W, bool kDirect>
cudaError_t launch_resident_bc_k(SysDev const* dSys, uint32_t const* dList, uint32_t nCta, StepSource const& src,
                                 uint32_t nSteps, size_t smem, cudaStream_t s)
{
    static thread_local bool done[64] = {};
    cudaError_t const e = allow_smem(k_resident_bc<W, kDirect>, done);
    if (e != cudaSuccess) return e;
    k_resident_bc<W, kDirect><<<nCta, kResidentBlock, smem, s>>>(dSys, dList, src, nSteps);
    return cudaGetLastError();
}

template <typename W>
cudaError_t launch_resident_bc_w(SysDev const* dSys, uint32_t const* dList, uint32_t nCta, uint32_t perThread,
                                 StepSource const& src, uint32_t nSteps, size_t smem, cudaStream_t s)
{
    // lists of 16-bit entries index up to 1 << kSlabEntBits slots of a group
    constexpr uint32_t kListed = (1u << kSlabEntBits) / kResidentBlock;
    if (perThread < 1 || perThread > 16) return cudaErrorInvalidValue;
    return perThread == 1 || perThread > kListed
               ? launch_resident_bc_k<W, true>(dSys, dList, nCta, src, nSteps, smem, s)
               : launch_resident_bc_k<W, false>(dSys, dList, nCta, src, nSteps, smem, s);
}

}  // namespace

cudaError_t launch_resident_bc(SysDev const* dSys, uint32_t const* dList, uint32_t nCta, uint32_t perThread,
                               StepSource const& src, uint32_t nSteps, size_t smem, uint32_t codeMode,
                               cudaStream_t s)
{
    if (nCta == 0 || nSteps == 0) return cudaSuccess;
    if (smem > kResidentMaxSmem || nSteps > kLaunchSteps) return cudaErrorInvalidValue;
    if (codeMode == kCode32)
        return launch_resident_bc_w<uint32_t>(dSys, dList, nCta, perThread, src, nSteps, smem, s);
    if (codeMode == kCode64)
        return launch_resident_bc_w<unsigned long long>(dSys, dList, nCta, perThread, src, nSteps, smem, s);
    return cudaErrorInvalidValue;
}

size_t cluster_bc_smem_bytes(uint32_t nwords, uint32_t npad, uint32_t logC, uint32_t chunks, uint32_t maxc,
                             uint32_t codeMode)
{
    uint32_t const w = codeMode == kCode64 ? 8 : 4;
    size_t const all = cluster_layout(nwords, npad, logC, chunks * 32u, w, maxc);
    return all <= kResidentMaxSmem ? all : cluster_layout(nwords, npad, logC, chunks * 32u, w, 0);
}

namespace {

// The launch of nClusters clusters of 2^logC CTAs of `block` threads.
cudaLaunchConfig_t cluster_bc_config(uint32_t logC, uint32_t block, size_t smem, cudaLaunchAttribute* attr,
                                     uint32_t nClusters, cudaStream_t s)
{
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << logC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nClusters << logC);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// How many clusters of 2^logC CTAs the device runs at a time, with all the shared memory a CTA may take:
// asked once per device, thread, kernel and size (the question takes the driver most of a millisecond).
template <typename W, int K, int B>
uint32_t cluster_bc_check(uint32_t logC)
{
    static thread_local short known[64][5] = {};
    static thread_local bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    short& k = known[dev & 63][logC];
    if (k == 0) {
        auto kernel = k_cluster_bc<W, K, B>;
        cudaLaunchAttribute attr[1];
        cudaLaunchConfig_t const cfg = cluster_bc_config(logC, B, kResidentMaxSmem, attr, 1, nullptr);
        int clusters = 0;
        cudaError_t e = allow_smem(kernel, done);
        if (e == cudaSuccess && logC > 3)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
        if (e != cudaSuccess) cudaGetLastError();   // a configuration the device refuses is an answer, not an error
        k = e == cudaSuccess && clusters >= 1 ? (short)clusters : -1;
    }
    return k > 0 ? (uint32_t)k : 0u;
}

template <typename W, int K, int B>
cudaError_t launch_cluster_bc_k(SysDev const* dSys, uint32_t const* dList, uint32_t nClusters, uint32_t logC,
                                StepSource const& src, uint32_t nSteps, size_t smem,
                                cudaStream_t s)
{
    if (cluster_bc_check<W, K, B>(logC) == 0) return cudaErrorInvalidConfiguration;
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t const cfg = cluster_bc_config(logC, B, smem, attr, nClusters, s);
    return cudaLaunchKernelEx(&cfg, k_cluster_bc<W, K, B>, dSys, dList, src, nSteps);
}

template <typename W>
cudaError_t launch_cluster_bc_w(SysDev const* dSys, uint32_t const* dList, uint32_t nClusters, uint32_t logC,
                                uint32_t chunks, StepSource const& src, uint32_t nSteps,
                                size_t smem, cudaStream_t s)
{
    switch (chunks) {
    case 16: return launch_cluster_bc_k<W, 1, kClusterSmallBlock>(dSys, dList, nClusters, logC, src, nSteps, smem, s);
    case 32: return launch_cluster_bc_k<W, 2, kClusterSmallBlock>(dSys, dList, nClusters, logC, src, nSteps, smem, s);
    case 64: return launch_cluster_bc_k<W, 2, kResidentBlock>(dSys, dList, nClusters, logC, src, nSteps, smem, s);
    case 128: return launch_cluster_bc_k<W, 4, kResidentBlock>(dSys, dList, nClusters, logC, src, nSteps, smem, s);
    case 256: return launch_cluster_bc_k<W, 8, kResidentBlock>(dSys, dList, nClusters, logC, src, nSteps, smem, s);
    default: return cudaErrorInvalidValue;
    }
}

template <typename W>
uint32_t cluster_bc_runnable_w(uint32_t logC, uint32_t chunks)
{
    switch (chunks) {
    case 16: return cluster_bc_check<W, 1, kClusterSmallBlock>(logC);
    case 32: return cluster_bc_check<W, 2, kClusterSmallBlock>(logC);
    case 64: return cluster_bc_check<W, 2, kResidentBlock>(logC);
    case 128: return cluster_bc_check<W, 4, kResidentBlock>(logC);
    case 256: return cluster_bc_check<W, 8, kResidentBlock>(logC);
    default: return 0;
    }
}

}  // namespace

uint32_t cluster_bc_runnable(uint32_t logC, uint32_t chunks, size_t smem, uint32_t codeMode)
{
    if (logC < 1 || logC > 4 || smem > kResidentMaxSmem) return 0;
    if (codeMode == kCode32) return cluster_bc_runnable_w<uint32_t>(logC, chunks);
    if (codeMode == kCode64) return cluster_bc_runnable_w<unsigned long long>(logC, chunks);
    return 0;
}

cudaError_t launch_cluster_bc(SysDev const* dSys, uint32_t const* dList, uint32_t nClusters, uint32_t logC,
                              uint32_t chunks, StepSource const& src, uint32_t nSteps,
                              size_t smem, uint32_t codeMode, cudaStream_t s)
{
    if (nClusters == 0 || nSteps == 0) return cudaSuccess;
    if (logC < 1 || logC > 4 || smem > kResidentMaxSmem || nSteps > kLaunchSteps) return cudaErrorInvalidValue;
    if (codeMode == kCode32)
        return launch_cluster_bc_w<uint32_t>(dSys, dList, nClusters, logC, chunks, src, nSteps, smem, s);
    if (codeMode == kCode64)
        return launch_cluster_bc_w<unsigned long long>(dSys, dList, nClusters, logC, chunks, src, nSteps,
                                                       smem, s);
    return cudaErrorInvalidValue;
}

}  // namespace bfm
