// matrix_tc.cu -- the filter-matrix comparison counted on the tensor cores.
//
// popcount(a & b) of two 2048-bit filters is the dot product of their bit
// vectors.  With every bit widened to an e2m1 value (4 bits) and fp32
// accumulation, tcgen05.mma.kind::mxf4 computes it exactly: bit k of each
// nibble keeps its place in the target filters (values 0.5, 1, 2, 2) and the
// reference filters hold the reciprocal (2, 1, 0.5, 0.5), so every product of
// two set bits is 1, all block scales are 1 and the sums are integers up to
// 2,048.  Widening permutes K inside each 32-bit word identically for both.
//
// One persistent CTA per SM multiplies 128 reference filters (TMEM lanes, a
// "pass": their 128 KB of e2m1 stay in shared memory) by tiles of up to 192
// target filters (TMEM columns) over K = 2048 in eight chunks of 256.  Five
// roles run as a pipeline over the tiles, joined by mbarriers only:
//   compose (1 warp)  takes work units, writes the rows of a pass and the
//                     columns of a tile (filter, hamming weight, element
//                     count, target) into a ring of four tiles;
//   widen (6 warps)   widen a pass's reference rows, then chunk by chunk the
//                     tile's target filters (bits read from global memory four
//                     chunks ahead) into two 24 KB stages;
//   mma (1 warp)      four K=64 MMAs per chunk into one of two accumulators;
//   mark (4 warps)    read the counts with tcgen05.ld, one row per lane, and
//                     mark the columns above the pair's cut: one subtraction
//                     and one funnel shift per column (the sign bit) when
//                     the slice's element counts are equal, else a table
//                     lookup per column;
//   check (8 warps)   recompute the marked pairs (about 1 % on unrelated
//                     content) from the filters in memory, eight lanes a
//                     pair: full count and the reference's staged exits
//                     (bf_utils.cc:114-206), and add the row's maximum.
// A pair can score above 0 only if its full count exceeds the cut, so what
// is not marked contributes 0.
//
// A digest pair's score is floor(100 * sum / denominator + 0.5) of the row
// maxima's sum in double precision, in filter order.  The row maxima are
// summed here as integers of 2^-23 (any order gives the same sum); each is
// within two units of the true ratio, so the score is the reference's unless
// 100 * sum / denominator + 0.5 lies within that error of a whole number.
// Such a pair (about 1 in 20,000 of those above 0, or an exact half), and a
// ratio that is not in [0, 1] (possible when --fast digests meet unfolded
// ones), is marked and k_matrix_finish scores it with the ordered sum in
// double precision.  Marks and sums live in the score array itself for units
// of several reference digests.
//
// Every mbarrier wait is bounded; a role whose wait gives up sets P.error
// and leaves, the others follow when their own waits run out, and the MMAs in
// flight are waited for before the TMEM is released.
//
// What bounds it: shared-memory bandwidth and the hand-over between the
// roles.  A tile takes about 10.4 K cycles, of which its 32 MMAs need 3 K on
// the tensor pipe; they read 10 KB of shared memory each (2.5 K cycles of
// its bandwidth a tile) beside 1.5 K cycles of widened stores.  Pairs of 128 x
// 192 filters: 5.6e11 filter pairs/s (400 uneven digests, 4.7e9 pairs: 8.5
// ms; 2,048 queries against 4 image segments, 8e8 pairs: 1.5 ms), against
// 1.2e11 for e4m3 operands widened for both sides in every tile, one row per
// scoring lane and ordered sums in the kernel (39 and 5.7 ms).  Measured on
// the way: every check warp a share of the tile's marked pairs instead of
// its own rows (three barriers a tile: 10.1 against 9.0 ms); the marks of a
// row listed and folded by its own lane (a last filter of few elements has
// most of a tile's marks: 64 x 64 digests 240 against 145 us); unrolled role
// loops (15 ms: the five roles share the instruction cache, and instruction
// fetch was the first stall); a proxy fence in the widening warps (18.4 ms:
// it waits for their loads in flight).
#include <cstdint>
#include <cuda_runtime.h>

#include "compare_device.cuh"
#include "compare_kernels.h"
#include "sdbf_device.cuh"

namespace sdbfg {

namespace {

constexpr uint32_t kTcRows = 128;       // reference rows per pass = TMEM lanes
constexpr uint32_t kTcCols = 192;       // target filters per tile = MMA N (max)
constexpr uint32_t kTcSlices = kTcCols / 32;
constexpr uint32_t kTcMark = 4, kTcCheck = 8, kTcWiden = 6;  // warps of each role
constexpr uint32_t kTcThreads = (kTcMark + kTcCheck + kTcWiden + 2) * 32;
constexpr uint32_t kTcComposeWarp = kTcMark + kTcCheck + kTcWiden, kTcMmaWarp = kTcComposeWarp + 1;
constexpr uint32_t kTcChunks = 8;                       // chunks of 256 bits: 128 bytes of e2m1 per row
constexpr uint32_t kTcAChunk = kTcRows * 128, kTcA = kTcChunks * kTcAChunk;
constexpr uint32_t kTcBStage = kTcCols * 128;
constexpr uint32_t kTcRing = 4;         // composed tiles in flight
constexpr uint32_t kTcScaleCol = 2 * kTcCols, kTcScaleCols = 32;  // TMEM columns of block scales (all 1.0)
constexpr uint32_t kTcTmemCols = 512;
constexpr uint32_t kTcMasks = 4;        // marked tiles in flight
constexpr uint32_t kTcDense = 96;       // marked pairs a check warp takes at a time
constexpr uint32_t kTcSpins = 1u << 20;

enum : uint32_t { kTileFirst = 1u, kTilePassEnd = 2u, kTileUnitEnd = 4u, kTileExit = 8u, kTileFast = 16u };

struct alignas(16) TcTile {
    uint32_t gidx[kTcCols];                 // filter of each column
    alignas(16) uint32_t meta[kTcCols];     // its hamming weight << 16 | element count (read four at a time)
    uint16_t te[kTcCols];                   // its target's place in the unit's run
    uint32_t e2min[kTcSlices];              // smallest hamming weight of the slice's columns that count
    uint32_t kmask[kTcSlices];              // columns that count (elements >= 16)
    uint32_t su[kTcSlices];                 // their element count where it is the same for all, else ~0
    uint32_t ste[kTcSlices];                // their target's place where it is the same for all, else ~0
    uint32_t nt, flags, pass, pseq, rc;     // columns, kTile*, pass slot and number, first row of the pass
    MatUnit unit;
};

struct TcPass {
    uint32_t rowf[kTcRows], rowmeta[kTcRows];  // filter of each row (~0: none), its meta word
    uint32_t gref[kTcRows];                    // reference digests of the unit
    uint8_t rowk[kTcRows];                     // the row's digest among them
};

// element-count sums of kTcSumMax and more share one cut: CUTOFFS256[0..3]
// are equal (4096 / sum <= 3), and CUTOFFS64[0..3] (1024 / sum <= 3)
constexpr uint32_t kTcSumMax = 1025;

struct TcSmem {
    TcTile tile[kTcRing];
    TcPass pass[kTcRing];
    uint32_t cm[kTcMasks][kTcSlices][kTcRows];     // marked columns of each row
    float thr[kTcSumMax + 1], thr64[kTcSumMax + 1];  // cut by element-count sum
    uint16_t dense[kTcCheck][kTcDense];     // check: marked pairs (row << 8 | column)
    uint32_t res[kTcCheck][kTcDense];       // check: their ratios in units of 2^-23 (0: none)
    // check: a row's open target (pass number << 9 | place) in the high half, its
    // maximum so far in the low one.  The mark warps read it while it changes: one 64-bit access.
    unsigned long long rowbest[kTcRows];
    uint32_t run[kMatMaxTargets];           // sums of the pass per target (one reference digest)
    unsigned long long run64[kMatMaxTargets];  // and of the unit
    uint32_t seg_first[kTcCols], seg_start[kTcCols + 1], seg_te[kTcCols];  // compose: one segment per target
    uint32_t gfirst[kTcRows], gstart[kTcRows + 1];                          // compose: rows of a group
    uint32_t tmem, fail;
    alignas(8) uint64_t tile_full[kTcRing], tile_empty[kTcRing], stage_full[2], stage_empty[2], acc_full[2],
        acc_empty[2], mask_full[kTcMasks], mask_empty[kTcMasks], check_bar, a_free, drain;
};

constexpr size_t kTcSmemBytes = 1024 /* alignment */ + kTcA + 2 * kTcBStage + sizeof(TcSmem);
static_assert(kTcSmemBytes <= 227 * 1024, "tensor-core kernel exceeds the shared memory of one CTA");
static_assert(sizeof(TcTile) % 16 == 0 && alignof(TcSmem) >= 16, "meta words are read as uint4");
static_assert(kTcWiden * 32 == kTcCols, "eight lanes a row, whole rows to a warp");

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
// By a whole warp; false: the wait gave up (the limit is about a second).
// The vote keeps the lanes together: without it they leave the loop one by
// one and run what follows in parts.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity) {
    const uint32_t addr = smem_addr(b);
#pragma unroll 1
    for (uint32_t i = 0; i < kTcSpins; i++) {
        uint32_t done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(addr), "r"(parity), "r"(1000u)
            : "memory");
        if (__all_sync(0xffffffffu, done)) return true;
    }
    return false;
}
// mbar_wait that, when phases are counted (kPhases), adds the cycles waited
// by the first lane of each of a role's warps (and the warp's other time)
// when the role ends
template <bool kPhases>
struct TcWait {
    unsigned long long* phase;
    int what;
    long long t0 = 0, waited = 0;
    __device__ __forceinline__ TcWait(unsigned long long* p, int w) : phase(p), what(w) {
        if constexpr (kPhases) t0 = clock64();
    }
    __device__ __forceinline__ bool operator()(uint64_t* b, uint32_t parity) {
        if constexpr (!kPhases) return mbar_wait(b, parity);
        const long long a = clock64();
        const bool ok = mbar_wait(b, parity);
        waited += clock64() - a;
        return ok;
    }
    __device__ __forceinline__ ~TcWait() {
        if (kPhases && (threadIdx.x & 31) == 0) {
            atomicAdd(phase + what, (unsigned long long)(clock64() - t0 - waited));
            atomicAdd(phase + kTcPhWaits + what, (unsigned long long)waited);
        }
    }
};
__device__ __forceinline__ void mma_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(b))
                 : "memory");
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// One filter word as the 16-byte granule q of row r of a chunk, at its
// swizzled place.
template <bool kRef>
__device__ __forceinline__ void widen_word(uint8_t* chunk, uint32_t r, uint32_t q, uint32_t x) {
    uint4 g;
    if (kRef) {
        g.x = (x & 0x11111111u) << 2;
        g.y = x & 0x22222222u;
        g.z = (x & 0x44444444u) >> 2;
        g.w = (x >> 3) & 0x11111111u;
    } else {
        g.x = x & 0x11111111u;
        g.y = x & 0x22222222u;
        g.z = x & 0x44444444u;
        g.w = (x >> 1) & 0x44444444u;
    }
    *reinterpret_cast<uint4*>(chunk + r * 128 + ((q ^ (r & 7)) << 4)) = g;
}

__device__ __forceinline__ uint2 row_best(const TcSmem& S, uint32_t row) {
    const unsigned long long v = *const_cast<const volatile unsigned long long*>(&S.rowbest[row]);
    return make_uint2((uint32_t)(v >> 32), (uint32_t)v);
}
__device__ __forceinline__ void set_row_best(TcSmem& S, uint32_t row, uint32_t tag, uint32_t best) {
    *const_cast<volatile unsigned long long*>(&S.rowbest[row]) = (unsigned long long)tag << 32 | best;
}

// slot j of a composed tile: its segment k (seg_start[k] <= j < seg_start[k+1])
__device__ __forceinline__ uint32_t find_segment(const uint32_t* seg_start, uint32_t nseg, uint32_t j) {
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (seg_start[mid] <= j) lo = mid;
        else hi = mid;
    }
    return lo;
}

// barrier of the check warps (bounded, unlike a hardware one); global
// additions of a thread before it are seen by the others' L2 reads after it
__device__ __forceinline__ bool check_sync(TcSmem& S, uint32_t lane, uint32_t& phase) {
    __threadfence();
    __syncwarp();
    if (lane == 0) mbar_arrive(&S.check_bar);
    const bool ok = mbar_wait(&S.check_bar, phase);
    phase ^= 1u;
    return ok;
}

// ------------------------------------------------------------- compose
template <bool kPhases>
__device__ __forceinline__ void tc_compose(const MatParams& P, TcSmem& S, uint32_t lane) {
    TcWait<kPhases> twait(P.phase, kTcPhCompose);
    uint32_t t = 0, pass = 0;  // tiles composed, passes begun
    uint32_t next = 0;
    if (lane == 0) next = atomicAdd(P.next_unit, 1u);
    for (;;) {
        const uint32_t u = __shfl_sync(0xffffffffu, next, 0);
        if (u >= P.nunits) {
            TcTile& T = S.tile[t % kTcRing];
            if (!twait(&S.tile_empty[t % kTcRing], ((t / kTcRing) & 1) ^ 1)) S.fail = 1;
            if (lane == 0) {
                T.flags = kTileExit;
                T.nt = 0;
                mbar_arrive(&S.tile_full[t % kTcRing]);
            }
            return;
        }
        if (lane == 0) next = atomicAdd(P.next_unit, 1u);  // the next unit, while this one is composed
        const MatUnit U = P.units[u];
        const uint32_t rs = U.flags & kUnitRefSide1 ? 1 : 0, ts = U.flags & kUnitTgtSide1 ? 1 : 0;
        const bool split = (U.flags & kUnitSplit) != 0, group = (U.flags & kUnitGroup) != 0;
        const uint32_t nref = group ? U.nref : 1, nT = U.t1 - U.t0;
        if (group) {  // first rows of the group's digests
            uint32_t base = 0;
            for (uint32_t b = 0; b < nref; b += 32) {
                const uint32_t k = b + lane;
                uint32_t n = 0, first = 0;
                if (k < nref) {
                    const CmpDigest D = P.digests[rs][P.refs[U.ref + k]];
                    n = D.nfilters;
                    first = D.first;
                }
                uint32_t incl = n;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= (uint32_t)d) incl += v;
                }
                if (k < nref) {
                    S.gfirst[k] = first;
                    S.gstart[k] = base + incl - n;
                }
                base += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) S.gstart[nref] = base;
            __syncwarp();
        }
        const CmpDigest A = P.digests[rs][group ? P.refs[U.ref] : U.ref];
        const uint32_t fast = A.flags & kDigestFast ? (uint32_t)kTileFast : 0u;
        for (uint32_t rc = U.r0; rc < U.r1; rc += kTcRows) {
            uint32_t ct = 0, cf = split ? U.c0 : 0u;  // target of the run, filter in it
            uint32_t wb = 0, wn = 0, wfirst = 0;       // 32 targets from wb: filters, first filter
            auto window = [&]() {
                wb = ct;
                wn = 0;
                if (wb + lane < nT) {
                    const CmpDigest B = P.digests[ts][P.targets[U.t0 + wb + lane]];
                    wn = split ? U.c1 : B.nfilters;
                    wfirst = B.first;
                }
            };
            window();
            bool first = true;
            while (ct < nT) {
                const uint32_t slot = t % kTcRing;
                TcTile& T = S.tile[slot];
                if (!twait(&S.tile_empty[slot], ((t / kTcRing) & 1) ^ 1)) {
                    S.fail = 1;
                    return;
                }
                if (first) {  // the rows of the pass (its slot was released with the tile's)
                    TcPass& R = S.pass[pass % kTcRing];
                    const uint32_t rows = U.r1 - rc;
#pragma unroll
                    for (uint32_t i = 0; i < kTcRows / 32; i++) {
                        const uint32_t row = 32 * i + lane;
                        uint32_t f = 0xFFFFFFFFu, m = 0, k = 0;
                        if (row < rows) {
                            if (group) {
                                k = find_segment(S.gstart, nref, row);
                                f = S.gfirst[k] + (row - S.gstart[k]);
                            } else {
                                f = A.first + rc + row;
                            }
                            m = P.meta[rs][f];
                        }
                        R.rowf[row] = f;
                        R.rowmeta[row] = m;
                        R.rowk[row] = (uint8_t)k;
                        if (row < nref) R.gref[row] = group ? P.refs[U.ref + row] : U.ref;
                    }
                }
                // targets from (ct, cf) on, up to kTcCols filters
                uint32_t filled = 0, nseg = 0;
                while (filled < kTcCols && ct < nT) {
                    if (ct >= wb + 32) window();
                    const uint32_t te = wb + lane;
                    const uint32_t f0 = te == ct ? cf : 0u;
                    const uint32_t rem = te >= ct && te < nT ? wn - f0 : 0u;
                    uint32_t incl = rem;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
                        if (lane >= (uint32_t)d) incl += v;
                    }
                    const uint32_t excl = incl - rem, room = kTcCols - filled;
                    const bool has = rem > 0 && excl < room;
                    const uint32_t has_mask = __ballot_sync(0xffffffffu, has);
                    if (has) {
                        const uint32_t k = nseg + __popc(has_mask & ((1u << lane) - 1u));
                        S.seg_first[k] = wfirst + f0;
                        S.seg_start[k] = filled + excl;
                        S.seg_te[k] = te;
                    }
                    nseg += __popc(has_mask);
                    const uint32_t over = __ballot_sync(0xffffffffu, rem > 0 && incl > room);
                    if (over) {  // the first target that does not fit (any more)
                        const uint32_t l = __ffs(over) - 1;
                        const uint32_t ex_l = __shfl_sync(0xffffffffu, excl, l), f0_l = __shfl_sync(0xffffffffu, f0, l);
                        ct = wb + l;
                        cf = f0_l + (room - ex_l);
                        filled = kTcCols;
                    } else {
                        filled += __shfl_sync(0xffffffffu, incl, 31);
                        ct = min(wb + 32u, nT);
                        cf = 0;
                    }
                }
                if (lane == 0) S.seg_start[nseg] = filled;
                __syncwarp();
                uint32_t mj[kTcSlices];
#pragma unroll 1
                for (uint32_t j = lane; j < kTcCols; j += 32) {
                    uint32_t f = 0, te = 0;
                    if (j < filled) {
                        const uint32_t k = find_segment(S.seg_start, nseg, j);
                        f = S.seg_first[k] + (j - S.seg_start[k]);
                        te = S.seg_te[k];
                    }
                    T.gidx[j] = f;
                    T.te[j] = (uint16_t)te;
                }
#pragma unroll
                for (uint32_t i = 0; i < kTcSlices; i++)  // (each lane reads what it wrote)
                    mj[i] = 32 * i + lane < filled ? P.meta[ts][T.gidx[32 * i + lane]] : 0u;
#pragma unroll
                for (uint32_t i = 0; i < kTcSlices; i++) T.meta[32 * i + lane] = mj[i];
#pragma unroll 1
                for (uint32_t i = 0; i < kTcSlices; i++) {
                    const uint32_t j = 32 * i + lane, m = T.meta[j], te = T.te[j];
                    const uint32_t e = m & 0xFFFFu, s2 = min(e, kTcSumMax);
                    const bool counts = j < filled && e >= (uint32_t)kMinElem;
                    const uint32_t km = __ballot_sync(0xffffffffu, counts);
                    const uint32_t lo = __reduce_min_sync(0xffffffffu, counts ? s2 : 0xFFFFu);
                    const uint32_t hi = __reduce_max_sync(0xffffffffu, counts ? s2 : 0u);
                    const uint32_t tlo = __reduce_min_sync(0xffffffffu, counts ? te : 0xFFFFu);
                    const uint32_t thi = __reduce_max_sync(0xffffffffu, counts ? te : 0u);
                    const uint32_t em = __reduce_min_sync(0xffffffffu, counts ? m >> 16 : 0xFFFFu);
                    if (lane == 0) {
                        T.kmask[i] = km;
                        T.su[i] = lo == hi ? lo : 0xFFFFFFFFu;
                        T.ste[i] = tlo == thi ? tlo : 0xFFFFFFFFu;
                        T.e2min[i] = em;
                    }
                }
                if (lane == 0) {
                    const bool pass_end = ct >= nT;
                    T.nt = filled;
                    T.pass = pass % kTcRing;
                    T.pseq = pass & 0x3FFFFFu;
                    T.rc = rc;
                    T.unit = U;
                    T.flags = fast | (first ? (uint32_t)kTileFirst : 0u) | (pass_end ? (uint32_t)kTilePassEnd : 0u) |
                              (pass_end && rc + kTcRows >= U.r1 ? (uint32_t)kTileUnitEnd : 0u);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.tile_full[slot]);
                first = false;
                t++;
            }
            pass++;
        }
    }
}

// a read-only load that stays where it is written: the compiler moves a
// plain one down to its use, behind the waits it is to overlap with
__device__ __forceinline__ uint4 ldg_here(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// --------------------------------------------------------------- widen
// A warp load takes 128 bytes of four rows (eight lanes a row, four words a
// lane: one "block" of four chunks), four cache lines instead of the sixteen
// that 32-byte pieces of sixteen rows touch; chunk j of the block is word j of every
// lane.  The order of the words in K is the same for both operands.
template <bool kPhases>
__device__ __forceinline__ void tc_widen(const MatParams& P, TcSmem& S, uint8_t* a_smem, uint8_t* b_smem, uint32_t wt,
                                         uint32_t lane) {
    TcWait<kPhases> twait(P.phase, kTcPhWiden);
    const uint32_t g = wt & 7, r0 = wt >> 3;  // lane g of rows r0 + 24 k
    constexpr uint32_t kRowStep = kTcWiden * 4, kRows = kTcCols / kRowStep;
    const uint4 z = make_uint4(0, 0, 0, 0);
    uint32_t pass = 0, q = 0;  // passes widened, chunks widened
    uint4 x[kRows], y[kRows];  // this block's words, the next block's
    uint32_t pt = 0, pb = 0;   // the next block: block pb of tile pt
    bool more = true, ok = true;
    auto fetch = [&]() {
#pragma unroll
        for (uint32_t k = 0; k < kRows; k++) y[k] = z;
        if (!more) return;
        const TcTile& T = S.tile[pt % kTcRing];
        if (pb == 0) {
            if (!twait(&S.tile_full[pt % kTcRing], (pt / kTcRing) & 1)) {
                ok = more = false;
                return;
            }
            if (T.flags & kTileExit) {
                more = false;
                return;
            }
        }
        const uint32_t* f = P.filters[T.unit.flags & kUnitTgtSide1 ? 1 : 0];
#pragma unroll
        for (uint32_t k = 0; k < kRows; k++)
            if (r0 + kRowStep * k < T.nt)
                y[k] = ldg_here(reinterpret_cast<const uint4*>(f + (size_t)T.gidx[r0 + kRowStep * k] * 64) + 8 * pb + g);
        if (++pb == (T.flags & kTileFast ? 1u : 2u)) {
            pb = 0;
            pt++;
        }
    };
    fetch();
    uint32_t t = 0, blk = 0;
    // one copy of the loop's code: five roles share the instruction cache
#pragma unroll 1
    while (ok) {
        const uint32_t slot = t % kTcRing;
        const TcTile& T = S.tile[slot];
        // (its descriptor has arrived: the fetch position is past it or at the exit)
        if (T.flags & kTileExit) return;
        const uint32_t ncols = (T.nt + 15) & ~15u, nblk = T.flags & kTileFast ? 1u : 2u;
        if (blk == 0 && (T.flags & kTileFirst)) {  // the pass's reference rows
            if (pass > 0 && !twait(&S.a_free, (pass - 1) & 1)) break;
            const TcPass& R = S.pass[T.pass];
            const uint32_t* f = P.filters[T.unit.flags & kUnitRefSide1 ? 1 : 0];
#pragma unroll 1
            for (uint32_t i0 = wt; i0 < kTcRows * 8 * nblk; i0 += 4 * kTcWiden * 32) {
                uint4 v[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) {  // lane g of row (i >> 3) & 127, block i >> 10
                    const uint32_t i = i0 + k * kTcWiden * 32;
                    v[k] = z;
                    if (i < kTcRows * 8 * nblk) {
                        const uint32_t fr = R.rowf[(i >> 3) & (kTcRows - 1)];
                        // fast mode counts the first 16 words: four lanes
                        if (fr != 0xFFFFFFFFu && (nblk == 2 || g < 4))
                            v[k] = __ldg(reinterpret_cast<const uint4*>(f + (size_t)fr * 64) + 8 * (i >> 10) + g);
                    }
                }
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) {
                    const uint32_t i = i0 + k * kTcWiden * 32;
                    if (i < kTcRows * 8 * nblk) {
                        uint8_t* a = a_smem + 4 * (i >> 10) * kTcAChunk;
                        const uint32_t r = (i >> 3) & (kTcRows - 1);
                        widen_word<true>(a, r, g, v[k].x);
                        widen_word<true>(a + kTcAChunk, r, g, v[k].y);
                        widen_word<true>(a + 2 * kTcAChunk, r, g, v[k].z);
                        widen_word<true>(a + 3 * kTcAChunk, r, g, v[k].w);
                    }
                }
            }
            pass++;
        }
#pragma unroll
        for (uint32_t k = 0; k < kRows; k++) x[k] = y[k];
        fetch();
#pragma unroll 1
        for (uint32_t j = 0; j < 4 && ok; j++, q++) {
            const uint32_t s = q & 1;
            ok = twait(&S.stage_empty[s], ((q >> 1) & 1) ^ 1);
            uint8_t* sb = b_smem + s * kTcBStage;
#pragma unroll
            for (uint32_t k = 0; k < kRows; k++) {
                const uint32_t r = r0 + kRowStep * k;
                if (r < ncols) widen_word<false>(sb, r, g, x[k].x);
                x[k].x = x[k].y;
                x[k].y = x[k].z;
                x[k].z = x[k].w;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.stage_full[s]);
        }
        if (++blk == nblk) {
            blk = 0;
            if (lane == 0) mbar_arrive(&S.tile_empty[slot]);
            t++;
        }
    }
    S.fail = 1;
}

// ----------------------------------------------------------------- mma
template <bool kPhases>
__device__ __forceinline__ void tc_mma(const MatParams& P, TcSmem& S, uint32_t a_addr, uint32_t b_addr, uint32_t tmem, uint32_t lane) {
    TcWait<kPhases> twait(P.phase, kTcPhMma);
    uint32_t q = 0;
    for (uint32_t t = 0;; t++) {
        const uint32_t slot = t % kTcRing, b = t & 1;
        bool ok = twait(&S.tile_full[slot], (t / kTcRing) & 1);
        const TcTile& T = S.tile[slot];
        if (ok && (T.flags & kTileExit)) return;
        ok = ok && twait(&S.acc_empty[b], ((t >> 1) & 1) ^ 1);
        if (!ok) {
            S.fail = 1;
            return;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t nch = T.flags & kTileFast ? 4u : kTcChunks, ncols = (T.nt + 15) & ~15u;
        const bool pass_end = (T.flags & kTilePassEnd) != 0;
        if (kPhases && lane == 0) atomicAdd(P.phase + kTcPhTiles, 1ull);
        // kind::mxf4: both operands e2m1 (1), N / 8, ue8m0 scales, M / 16, K = 64
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((ncols >> 3) << 17) | (1u << 23) | ((kTcRows >> 4) << 24);
        const uint32_t dacc = tmem + b * kTcCols;
        for (uint32_t c = 0; c < nch; c++, q++) {
            const uint32_t s = q & 1;
            if (!twait(&S.stage_full[s], (q >> 1) & 1)) {
                S.fail = 1;
                return;
            }
            if (lane == 0) {
                // the widening warps' writes, seen through the barrier, become
                // visible to the tensor core here: a fence in those warps
                // would wait for their loads in flight
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t a0 = a_addr + c * kTcAChunk, b0 = b_addr + s * kTcBStage;
#pragma unroll
                for (uint32_t kk = 0; kk < 4; kk++) {
                    const uint64_t ad = sw128_desc(a0 + kk * 32), bd = sw128_desc(b0 + kk * 32);
                    const uint32_t acc = (c > 0 || kk > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                        " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n}\n" ::"r"(
                            dacc),
                        "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(tmem + kTcScaleCol), "r"(tmem + kTcScaleCol + kTcScaleCols / 2));
                }
                mma_commit(&S.stage_empty[s]);
                if (c + 1 == nch) {
                    mma_commit(&S.acc_full[b]);
                    if (pass_end) mma_commit(&S.a_free);
                }
            }
            __syncwarp();
        }
        if (lane == 0) mbar_arrive(&S.tile_empty[slot]);
    }
}

// ---------------------------------------------------------------- mark
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
        "%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
// the loads' registers pass through the wait, so that no use moves before it
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
                 :
                 : "memory");
    asm volatile("" : "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]),
                 "+r"(v[23]), "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]),
                 "+r"(v[31]));
}
template <bool kPhases>
__device__ __forceinline__ void tc_mark(const MatParams& P, TcSmem& S, uint32_t tmem, uint32_t warp, uint32_t lane) {
    TcWait<kPhases> twait(P.phase, kTcPhMark);
    const uint32_t row = warp * 32 + lane;
    uint32_t s1 = 0, e1 = 0;
    bool active = false;
    for (uint32_t t = 0;; t++) {
        const uint32_t slot = t % kTcRing, b = t & 1;
        bool ok = twait(&S.tile_full[slot], (t / kTcRing) & 1);
        const TcTile& T = S.tile[slot];
        if (ok && (T.flags & kTileExit)) return;
        const uint32_t mb = t % kTcMasks;
        ok = ok && twait(&S.mask_empty[mb], ((t / kTcMasks) & 1) ^ 1) && twait(&S.acc_full[b], (t >> 1) & 1);
        if (!ok) {
            S.fail = 1;
            return;
        }
        if (T.flags & kTileFirst) {
            const uint32_t m = S.pass[T.pass].rowmeta[row] & 0xFFFFu;
            active = m >= (uint32_t)kMinElem;
            s1 = min(m, kTcSumMax);
            e1 = S.pass[T.pass].rowmeta[row] >> 16;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const float* thr = T.flags & kTileFast ? S.thr64 : S.thr;
        const uint32_t nsl = (T.nt + 31) / 32;
        const uint2 rb = row_best(S, row);
        const uint32_t tacc = tmem + ((warp * 32) << 16) + b * kTcCols;
        // columns of slice i above the cut: the sign of cut - count, four
        // chains of eight columns.  A row that has a maximum r of the
        // slice's target already only improves on it where
        // count - cut > r (weight - cut), weight the smaller hamming weight of the pair.
        auto slice = [&](uint32_t i, const uint32_t (&v)[32]) {
            const uint32_t km = T.kmask[i], su = T.su[i];
            uint32_t m[4] = {0, 0, 0, 0};
            if (km != 0) {
                float r = 0.0f;
                if (rb.x == (T.pseq << 9 | T.ste[i])) r = fmaxf((float)rb.y - 8.0f, 0.0f) * (1.0f / 8388608.0f);
                const float keep = 1.0f - r, fe1 = (float)e1;
                if (su != 0xFFFFFFFFu) {
                    float cut = thr[min(s1 + su, kTcSumMax)];
                    cut = fmaxf(cut, fmaf(cut, keep, r * fminf(fe1, (float)T.e2min[i]) - 0.0625f));
#pragma unroll
                    for (int q = 7; q >= 0; q--)
#pragma unroll
                        for (int z = 0; z < 4; z++)
                            m[z] = __funnelshift_l(__float_as_uint(cut - __uint_as_float(v[8 * z + q])), m[z], 1);
                } else {
                    const uint4* m4 = reinterpret_cast<const uint4*>(&T.meta[32 * i]);
#pragma unroll
                    for (int z = 0; z < 4; z++) {
                        const uint4 w = m4[2 * z], x = m4[2 * z + 1];
                        const uint32_t mt[8] = {w.x, w.y, w.z, w.w, x.x, x.y, x.z, x.w};
#pragma unroll
                        for (int q = 7; q >= 0; q--) {
                            float cut = thr[min(s1 + (mt[q] & 0xFFFFu), kTcSumMax)];
                            const float we = fminf(fe1, (float)(mt[q] >> 16));
                            cut = fmaxf(cut, fmaf(cut, keep, fmaf(r, we, -0.0625f)));
                            m[z] = __funnelshift_l(__float_as_uint(cut - __uint_as_float(v[8 * z + q])), m[z], 1);
                        }
                    }
                }
            }
            S.cm[mb][i][row] = active ? (m[0] | m[1] << 8 | m[2] << 16 | m[3] << 24) & km : 0u;
        };
#pragma unroll 1
        for (uint32_t i = 0; i < nsl; i++) {
            uint32_t v[32];
            tmem_ld32(tacc + 32 * i, v);
            tmem_ld_wait(v);
            slice(i, v);
        }
        for (uint32_t i = nsl; i < kTcSlices; i++) S.cm[mb][i][row] = 0;
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&S.acc_empty[b]);
            mbar_arrive(&S.mask_full[mb]);
            mbar_arrive(&S.tile_empty[slot]);
        }
    }
}

// --------------------------------------------------------------- check
template <bool kPhases>
__device__ __forceinline__ void tc_check(const MatParams& P, TcSmem& S, uint32_t cw, uint32_t lane) {
    TcWait<kPhases> twait(P.phase, kTcPhCheck);
    const uint32_t half = lane >> 4, row = cw * 16 + (lane & 15);  // slices 3 half .. 3 half + 2 of the row
    const uint32_t ct = cw * 32 + lane;                            // thread of the role
    const uint32_t sub = lane & 7, grp = lane >> 3;
    uint16_t* dense = S.dense[cw];
    uint32_t* res = S.res[cw];
    uint32_t phase = 0;
#pragma unroll 1
    for (uint32_t t = 0;; t++) {
        const uint32_t slot = t % kTcRing, b = t % kTcMasks;
        bool ok = twait(&S.tile_full[slot], (t / kTcRing) & 1);
        const TcTile& T = S.tile[slot];
        if (ok && (T.flags & kTileExit)) return;
        ok = ok && twait(&S.mask_full[b], (t / kTcMasks) & 1);
        if (!ok) break;
        uint32_t m[3];
#pragma unroll
        for (int k = 0; k < 3; k++) m[k] = S.cm[b][3 * half + k][row];
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.mask_empty[b]);
        const uint32_t n = __popc(m[0]) + __popc(m[1]) + __popc(m[2]);
        uint32_t incl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        const uint32_t off = incl - n, total = __shfl_sync(0xffffffffu, incl, 31);
        const TcPass& R = S.pass[T.pass];
        const uint32_t uflags = T.unit.flags;
        const uint32_t rs = uflags & kUnitRefSide1 ? 1 : 0, ts = uflags & kUnitTgtSide1 ? 1 : 0;
        const bool split = (uflags & kUnitSplit) != 0, fast = (T.flags & kTileFast) != 0;
        const uint32_t nref = uflags & kUnitGroup ? T.unit.nref : 1u;
        if (T.flags & kTileFirst) {
            if (half == 0) set_row_best(S, row, 0xFFFFFFFFu, 0);
            __syncwarp();
        }
        const uint32_t* __restrict__ fr = P.filters[rs];
        const uint32_t* __restrict__ ft = P.filters[ts];
        const float* thr = fast ? S.thr64 : S.thr;
        if (kPhases && lane == 0) atomicAdd(P.phase + kTcPhMarked, (unsigned long long)total);
        // the warp's marked pairs in one list, kTcDense of them at a time: by
        // lane (a row's first half before its second), then column.  The
        // warp writes one mask word at a time, so a row with many marks (a
        // digest's last filter, of few elements and a low cut) costs it no more than others.
#pragma unroll 1
        for (uint32_t base = 0; base < total; base += kTcDense) {
            const uint32_t lim = min(total - base, kTcDense);
            uint32_t at = off - base;  // place of the lane's next word (wraps below the round)
#pragma unroll
            for (int k = 0; k < 3; k++) {
                uint32_t lanes = __ballot_sync(0xffffffffu, m[k] != 0);
#pragma unroll 1
                while (lanes) {
                    const uint32_t l = __ffs(lanes) - 1;
                    lanes &= lanes - 1u;
                    const uint32_t w = __shfl_sync(0xffffffffu, m[k], l), o = __shfl_sync(0xffffffffu, at, l);
                    const uint32_t i = o + __popc(w & ((1u << lane) - 1u));
                    if (((w >> lane) & 1u) && i < lim)
                        dense[i] = (uint16_t)((cw * 16 + (l & 15)) << 8 | (96 * (l >> 4) + 32 * k + lane));
                }
                at += __popc(m[k]);
            }
            __syncwarp();
            constexpr uint32_t kSteps = 3;  // pairs in flight per eight lanes
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < lim; i0 += 4 * kSteps) {
                uint4 x[kSteps][2], y[kSteps][2];
                uint32_t e[kSteps];
#pragma unroll
                for (uint32_t s = 0; s < kSteps; s++) {  // (past the end: the last pair again)
                    e[s] = dense[min(i0 + 4 * s + grp, lim - 1)];
                    const uint4* a = reinterpret_cast<const uint4*>(fr + (size_t)R.rowf[e[s] >> 8] * 64) + sub;
                    const uint4* c = reinterpret_cast<const uint4*>(ft + (size_t)T.gidx[e[s] & 0xFFu] * 64) + sub;
                    x[s][0] = __ldg(a);
                    x[s][1] = __ldg(a + 8);
                    y[s][0] = __ldg(c);
                    y[s][1] = __ldg(c + 8);
                }
                uint32_t pk0 = 0, pk1 = 0, ee = 0;  // lane sub < kSteps: step sub's counts (packed) and pair
#pragma unroll
                for (uint32_t s = 0; s < kSteps; s++) {
                    uint32_t p[2];
#pragma unroll
                    for (int z = 0; z < 2; z++)
                        p[z] = __popc(x[s][z].x & y[s][z].x) + __popc(x[s][z].y & y[s][z].y) +
                               __popc(x[s][z].z & y[s][z].z) + __popc(x[s][z].w & y[s][z].w);
                    // first of the eight lanes: counts of the first 8, 16 and
                    // 32 words, and above them those of the words 32 later
                    uint32_t c = p[0] | p[1] << 16;
                    const uint32_t c1 = c + __shfl_xor_sync(0xffffffffu, c, 1);
                    const uint32_t c2 = c1 + __shfl_xor_sync(0xffffffffu, c1, 2);
                    const uint32_t c3 = c2 + __shfl_xor_sync(0xffffffffu, c2, 4);
                    const uint32_t k0 = __shfl_sync(0xffffffffu, (c1 & 0xFFFFu) | c2 << 16, lane & 24);
                    const uint32_t k1 = __shfl_sync(0xffffffffu, c3, lane & 24);
                    if (sub == s) {
                        pk0 = k0;
                        pk1 = k1;
                        ee = e[s];
                    }
                }
                const uint32_t i = i0 + 4 * sub + grp;
                if (sub < kSteps && i < lim) {
                    const uint32_t p = pk0 & 0xFFFFu, p1 = pk0 >> 16, p2 = pk1 & 0xFFFFu, p3 = p2 + (pk1 >> 16);
                    const uint32_t mr = R.rowmeta[ee >> 8], mc = T.meta[ee & 0xFFu];
                    const uint32_t cut = (uint32_t)thr[min(min(mr & 0xFFFFu, kTcSumMax) + min(mc & 0xFFFFu, kTcSumMax), kTcSumMax)];
                    const uint32_t cnt = fast ? p1 : p3;
                    const bool out = fast ? 2 * p + 48 < cut : (8 * p + 48 < cut || 4 * p1 + 48 < cut || 2 * p2 + 48 < cut);
                    uint32_t r = 0;
                    if (!out && cnt > cut) {
                        const uint32_t num = cnt - cut, den = min(mr >> 16, mc >> 16) - cut;
                        // within two units of 2^-23 of num / den (two ulps of the quotient, rounding)
                        r = num <= den ? (uint32_t)(__fdividef((float)num, (float)den) * 8388608.0f + 0.5f) : 0xFFFFFFFFu;
                    }
                    res[i] = r;
                }
            }
            __syncwarp();
            // the rows' maxima, 32 entries at a time: the maximum of every run
            // of one row and target, then the runs' last lanes update the
            // rows (a row's runs one after another, in order)
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < lim; i0 += 32) {
                const uint32_t e = dense[min(i0 + lane, lim - 1)];
                uint32_t r = i0 + lane < lim ? res[i0 + lane] : 0u;
                const uint32_t te = T.te[e & 0xFFu], row = e >> 8, key = row << 9 | te;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t kr = __shfl_up_sync(0xffffffffu, key, d), rr = __shfl_up_sync(0xffffffffu, r, d);
                    if (lane >= (uint32_t)d && kr == key) r = max(r, rr);
                }
                const uint32_t next = __shfl_down_sync(0xffffffffu, key, 1);
                uint32_t todo = __ballot_sync(0xffffffffu, r != 0 && (lane == 31 || next != key));
                const uint32_t same = __match_any_sync(0xffffffffu, row);
#pragma unroll 1
                while (todo) {
                    const uint32_t mine = same & todo;
                    if (((todo >> lane) & 1u) && (uint32_t)(__ffs(mine) - 1) == lane) {
                        const uint32_t tag = T.pseq << 9 | te;
                        const uint2 st = row_best(S, row);
                        const uint32_t best = st.x == tag ? st.y : 0u;
                        if (r > best) {
                            set_row_best(S, row, tag, r);  // (the mark warps raise the row's cuts by it)
                            // the sum grows by what the maximum grows
                            if (split) {
                                atomicMax(reinterpret_cast<uint32_t*>(P.slots) + P.split[T.unit.split].slot_base + T.rc + row, r);
                            } else {
                                uint32_t* sum;
                                if (nref == 1) sum = &S.run[te];
                                else
                                    sum = reinterpret_cast<uint32_t*>(P.scores) +
                                          out_index(P, rs != 0, R.gref[R.rowk[row]], P.targets[T.unit.t0 + te]);
                                if (r == 0xFFFFFFFFu) atomicOr(sum, 0x80000000u);  // left to k_matrix_finish
                                else atomicAdd(sum, r - best);
                            }
                        }
                    }
                    todo &= ~__ballot_sync(0xffffffffu, ((todo >> lane) & 1u) && (uint32_t)(__ffs(mine) - 1) == lane);
                    __syncwarp();
                }
            }
            __syncwarp();
        }
        if (!split && (T.flags & kTilePassEnd)) {
            const uint32_t nT = T.unit.t1 - T.unit.t0;
            if (!check_sync(S, lane, phase)) break;
            if (nref == 1)
                for (uint32_t k = ct; k < nT; k += kTcCheck * 32) {
                    const uint32_t v = S.run[k];
                    S.run[k] = 0;
                    S.run64[k] = (S.run64[k] + (v & 0x7FFFFFFFu)) | ((unsigned long long)(v >> 31) << 63);
                }
            if (T.flags & kTileUnitEnd) {
                for (uint32_t k = ct; k < nref * nT; k += kTcCheck * 32) {
                    const uint32_t g = k % nref, te = k / nref;
                    const uint32_t ref = R.gref[g], tgt = P.targets[T.unit.t0 + te];
                    const uint64_t o = out_index(P, rs != 0, ref, tgt);
                    unsigned long long sum;
                    if (nref == 1) {
                        sum = S.run64[te];
                        S.run64[te] = 0;
                    } else {
                        const uint32_t v = (uint32_t)__ldcg(P.scores + o);
                        sum = (v & 0x7FFFFFFFu) | ((unsigned long long)(v >> 31) << 63);
                    }
                    P.scores[o] = fixed_score(P, rs, ref, ts, tgt, sum);
                }
            }
            if (!check_sync(S, lane, phase)) break;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.tile_empty[slot]);
    }
    S.fail = 1;
}

}  // namespace

template <bool kPhases>
__global__ void __launch_bounds__(kTcThreads, 1) k_matrix_tc(MatParams P) {
    extern __shared__ uint8_t tc_smem_raw[];
    const uint32_t raw = smem_addr(tc_smem_raw);
    uint8_t* a_smem = tc_smem_raw + (((raw + 1023) & ~1023u) - raw);
    uint8_t* b_smem = a_smem + kTcA;
    TcSmem& S = *reinterpret_cast<TcSmem*>(b_smem + 2 * kTcBStage);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (uint32_t i = tid; i <= kTcSumMax; i += kTcThreads) {
        // below 32 (8) the quotient is past the tables' end, as in the reference's last bin
        S.thr[i] = (float)P.cutoffs[i >= 32 ? min(4096u / i, (uint32_t)SDBF_CUTOFF_BINS - 1) : (uint32_t)SDBF_CUTOFF_BINS - 1];
        S.thr64[i] = (float)P.cutoffs64[i >= 8 ? min(1024u / i, (uint32_t)SDBF_CUTOFF_BINS - 1) : (uint32_t)SDBF_CUTOFF_BINS - 1];
    }
    for (uint32_t i = tid; i < kTcRows; i += kTcThreads) S.rowbest[i] = ~0ull << 32;
    for (uint32_t i = tid; i < kMatMaxTargets; i += kTcThreads) {
        S.run[i] = 0;
        S.run64[i] = 0;
    }
    if (tid == 0) {
        S.fail = 0;
        for (uint32_t i = 0; i < kTcRing; i++) {
            mbar_init(&S.tile_full[i], 1);
            mbar_init(&S.tile_empty[i], kTcMark + kTcCheck + kTcWiden + 1);
        }
        for (uint32_t i = 0; i < 2; i++) {
            mbar_init(&S.stage_full[i], kTcWiden);
            mbar_init(&S.stage_empty[i], 1);
            mbar_init(&S.acc_full[i], 1);
            mbar_init(&S.acc_empty[i], kTcMark);
        }
        for (uint32_t i = 0; i < kTcMasks; i++) {
            mbar_init(&S.mask_full[i], kTcMark);
            mbar_init(&S.mask_empty[i], kTcCheck);
        }
        mbar_init(&S.check_bar, kTcCheck);
        mbar_init(&S.a_free, 1);
        mbar_init(&S.drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&S.tmem)),
                     "r"(kTcTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = S.tmem;
    if (warp < 4) {  // every block scale is 1.0 (ue8m0 127), whatever its place in these columns
        const uint32_t one = 0x7F7F7F7Fu;
        const uint32_t taddr = tmem + ((warp * 32) << 16) + kTcScaleCol;
#pragma unroll
        for (uint32_t c = 0; c < kTcScaleCols; c += 8)
            asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr + c), "r"(one)
                         : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");

    if (warp < kTcMark) tc_mark<kPhases>(P, S, tmem, warp, lane);
    else if (warp < kTcMark + kTcCheck) tc_check<kPhases>(P, S, warp - kTcMark, lane);
    else if (warp < kTcComposeWarp) tc_widen<kPhases>(P, S, a_smem, b_smem, (warp - kTcMark - kTcCheck) * 32 + lane, lane);
    else if (warp == kTcComposeWarp) tc_compose<kPhases>(P, S, lane);
    else tc_mma<kPhases>(P, S, smem_addr(a_smem), smem_addr(b_smem), tmem, lane);
    __syncwarp();
    if (warp == kTcMmaWarp && S.fail) {
        // wait (bounded) for any MMA still reading shared memory or writing TMEM
        if (lane == 0) mma_commit(&S.drain);
        __syncwarp();
        mbar_wait(&S.drain, 0);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0 && S.fail) atomicAdd(P.error, 1u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcTmemCols));
}

cudaError_t launch_matrix_tc(const MatParams& P, uint32_t grid, cudaStream_t st) {
    if (P.nunits == 0) return cudaSuccess;
    if (P.phase) k_matrix_tc<true><<<grid, kTcThreads, kTcSmemBytes, st>>>(P);
    else k_matrix_tc<false><<<grid, kTcThreads, kTcSmemBytes, st>>>(P);
    return cudaGetLastError();
}

int matrix_tc_ctas_per_sm() {
    cudaFuncSetAttribute(k_matrix_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmemBytes);
    cudaFuncSetAttribute(k_matrix_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmemBytes);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_matrix_tc<false>, kTcThreads, kTcSmemBytes);
    return n > 0 ? n : 1;
}

}  // namespace sdbfg
