// gen_kernels.cu -- SDBF digest generation on sm_103a.
//
// Restates sdhash's generation path (sdbf/sdbf_core.cc:21-324) as three
// kernels over a batch of files resident in HBM:
//
//  k_stream_tiles   one CTA per tile of kTileL window steps of a 32 MiB
//                   stream chunk: bytes -> ranks (rolling 64-byte entropy,
//                   gen_chunk_ranks :21-45) -> popularity scores
//                   (gen_chunk_scores :50-89, parallelised below) ->
//                   selection score > 16 -> SHA-1 of every selected 64-byte
//                   feature.  Writes the ordered feature digests of the tile.
//  k_stream_fix     one CTA per chunk: finds tiles whose speculative entry
//                   state differs from their predecessor's exit state and
//                   recomputes them in place from the true state.
//  k_stream_commit  one CTA per file: the ordered filter fill of
//                   gen_chunk_hash (:93-136) -- 256-byte filter insert with
//                   zero-new-bit suppression, the 16 KiB "big filter"
//                   dedupe (bloom_filter.cc:333-359), roll-over at 160
//                   elements, big-filter roll-over at 8738 per chunk, and the
//                   final chop (:235-238).  A file that a batch waits for
//                   commits through links instead (k_stream_chain).
//  k_block_digest   one CTA per dd block (gen_block_sdbf_mt :251-324,
//                   gen_block_hash :141-191): histogram threshold, <=192
//                   ordered inserts.
//
// Popularity scores in parallel.  gen_chunk_scores is a sequential state
// machine over window steps i with state (P, M) = (min_pos, min_rank).  A
// step is either a "cheap slide" (depends on (P, M) and rank[i+64]) or a full
// rescan of window [i, i+63], whose result depends on i only.  Hence two
// walks that reach the same state at the same step agree from then on.  Each
// thread walks one segment of steps, starting kLead steps early with an
// assumed full rescan; the state it reaches at its segment start is compared
// with the state its left neighbour reaches at the same step.  Equal states
// prove the segment exact (induction from step 0, which is always a full
// rescan); a mismatch is re-walked from the neighbour's state.  The same
// check links consecutive tiles of a chunk (k_stream_fails / k_stream_fix).
#include <cstdint>
#include <mutex>

#include <cuda_runtime.h>

#include "gen_kernels.h"
#include "sdbf_device.cuh"

namespace sdbfg {

// ------------------------------------------------------------ smem layout
struct TileGeom {
    uint32_t n;      // chunk length
    uint32_t t0;     // first step owned by the tile
    uint32_t S0;     // first step whose credits the tile needs (t0-64, or 0)
    uint32_t SE;     // end of steps (exclusive), <= n-64
    uint32_t Q0;     // first step simulated (lead-in), multiple of 64 rel. chunk
    uint32_t RE;     // end of rank positions (exclusive)
    uint32_t BE;     // end of bytes (exclusive)
    uint32_t L;      // positions owned: [t0, t0+L)
};

// Shared-memory carve-up for a tile of at most Lmax owned positions.
struct TileSmem {
    uint32_t* bytes32;     // chunk bytes [Q0, BE) (+pad)
    uint16_t* ranks;       // ranks [Q0, RE)
    uint8_t* hist;         // per-thread byte histograms (phase 2 only)
    uint16_t* fres;        // full-rescan result per step [Q0, SE)
    uint32_t* score32;     // u8 scores of [t0, t0+L) packed 4 per word
    uint32_t* list;        // selected positions (relative to t0)
    uint64_t* sig;         // per-segment entry state
    uint64_t* tau;         // per-segment exit state
    uint32_t* own;         // block mode, insert phase: 2,048 owners over dead space
    uint32_t* misc;        // scalars
};

__host__ __device__ constexpr uint32_t align_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// Padded index of the per-position uint16 arrays (ranks, full-rescan
// results): one spare word after every 64 entries, so 32 lanes that each
// scan their own aligned 64-position block address 32 different banks.
__host__ __device__ constexpr uint32_t pidx(uint32_t o) { return o + 2 * (o >> 6); }
__host__ __device__ constexpr uint32_t padded_len(uint32_t n) { return pidx(n) + 2; }

// Byte address of thread t's counter for byte value v in the histogram area:
// each lane's 256 counters occupy 64 words of its own bank.
static_assert(kRankThreads % 32 == 0, "histogram layout assumes full warps");
__device__ __forceinline__ uint32_t hist_off(uint32_t t, uint32_t v) {
    return ((((t >> 5) * 64 + (v >> 2)) * 32 + (t & 31)) << 2) | (v & 3);
}

// Layout: bytes | ranks | union { histograms (ranks phase) ;
//                                 fres | scores | list | sig | tau } | misc
__host__ __device__ inline uint32_t phase3_bytes(uint32_t Lmax) {
    return align_up(padded_len(Lmax + 64 + kLead) * 2, 16) + align_up(Lmax + 16, 16) +
           align_up(((Lmax + 64) / 15 + 8) * 4, 16) + 2 * kSegs * 8;
}

// Offset in the union of the block-mode insert's owner table (8 KiB): the
// full-rescan table when it is that large (dead once the scores are
// known), else past the phase-3 layout.
constexpr uint32_t kOwnBytes = 2048 * 4;
__host__ __device__ inline uint32_t own_offset(uint32_t Lmax) {
    return align_up(padded_len(Lmax + 64 + kLead) * 2, 16) >= kOwnBytes ? 0u : phase3_bytes(Lmax);
}

__host__ __device__ inline uint32_t union_bytes(uint32_t Lmax) {
    const uint32_t hist = 256 * kRankThreads, p3 = phase3_bytes(Lmax), own = own_offset(Lmax) + kOwnBytes;
    return max(max(hist, p3), own);
}

__host__ __device__ inline uint32_t tile_smem_bytes(uint32_t Lmax) {
    const uint32_t span = Lmax + 64 + kLead + 64;           // rank positions
    uint32_t b = 0;
    b += align_up(span + 64 + 16, 16);                       // bytes
    b += align_up(padded_len(span) * 2, 16);                 // ranks
    b += union_bytes(Lmax);                                  // union
    b += 64 * 4;                                             // misc
    return b;
}

__device__ inline TileSmem carve(uint8_t* base, uint32_t Lmax) {
    TileSmem s;
    const uint32_t span = Lmax + 64 + kLead + 64;
    uint8_t* p = base;
    s.bytes32 = reinterpret_cast<uint32_t*>(p); p += align_up(span + 64 + 16, 16);
    s.ranks = reinterpret_cast<uint16_t*>(p); p += align_up(padded_len(span) * 2, 16);
    uint8_t* u = p;
    s.hist = u;
    s.fres = reinterpret_cast<uint16_t*>(u); u += align_up(padded_len(Lmax + 64 + kLead) * 2, 16);
    s.score32 = reinterpret_cast<uint32_t*>(u); u += align_up(Lmax + 16, 16);
    s.list = reinterpret_cast<uint32_t*>(u); u += align_up(((Lmax + 64) / 15 + 8) * 4, 16);
    s.sig = reinterpret_cast<uint64_t*>(u); u += kSegs * 8;
    s.tau = reinterpret_cast<uint64_t*>(u); u += kSegs * 8;
    s.own = reinterpret_cast<uint32_t*>(p + own_offset(Lmax));
    p += union_bytes(Lmax);
    s.misc = reinterpret_cast<uint32_t*>(p);
    return s;
}

// Layout of a stream tile whose ranks come precomputed (k_stream_ranks):
// ranks | fres (the compaction list reuses it) | scores | sig | tau | misc.
// No bytes or histograms: 42.9 KB, so five tiles fit on an SM.
__host__ __device__ inline uint32_t fres_bytes(uint32_t Lmax) { return align_up(padded_len(Lmax + 64 + kLead) * 2, 16); }
__host__ __device__ inline uint32_t tile_smem_bytes_pre(uint32_t Lmax) {
    const uint32_t span = Lmax + 64 + kLead + 64;
    return align_up(padded_len(span) * 2, 16) + fres_bytes(Lmax) + align_up(Lmax + 16, 16) + 2 * kSegs * 8 + 64 * 4;
}
__device__ inline TileSmem carve_pre(uint8_t* base, uint32_t Lmax) {
    TileSmem s;
    const uint32_t span = Lmax + 64 + kLead + 64;
    uint8_t* p = base;
    s.bytes32 = nullptr;
    s.hist = nullptr;
    s.own = nullptr;
    s.ranks = reinterpret_cast<uint16_t*>(p); p += align_up(padded_len(span) * 2, 16);
    s.fres = reinterpret_cast<uint16_t*>(p);
    s.list = reinterpret_cast<uint32_t*>(p); p += fres_bytes(Lmax);
    s.score32 = reinterpret_cast<uint32_t*>(p); p += align_up(Lmax + 16, 16);
    s.sig = reinterpret_cast<uint64_t*>(p); p += kSegs * 8;
    s.tau = reinterpret_cast<uint64_t*>(p); p += kSegs * 8;
    s.misc = reinterpret_cast<uint32_t*>(p);
    return s;
}
static_assert(((kTileL + 64) / 15 + 8) * 4 <= (kTileL + 64 + kLead) * 2, "the list fits in the fres area");

// Ranks [Q0, RE) of a tile from the chunk's precomputed ranks (src = the
// chunk's first rank, 16-byte aligned; Q0 is a multiple of 64, and the
// chunk's ranks extend to a multiple of 8), eight per 16-byte load.  The
// last 64 positions have rank 0 (a dd block inside a longer run of ranks has
// a size that is a multiple of 8, so they are whole loads there).
template <bool kBlock>
__device__ inline void load_ranks(const uint16_t* __restrict__ src, const TileGeom& g, uint16_t* dst) {
    const uint32_t n8 = (g.RE - g.Q0 + 7) / 8;
    const uint4* s4 = reinterpret_cast<const uint4*>(src + g.Q0);
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < n8; i += blockDim.x) {
        uint4 v = __ldg(s4 + i);
        if (kBlock && g.Q0 + 8 * i >= g.n - kWin) v = make_uint4(0, 0, 0, 0);
        uint32_t* d = reinterpret_cast<uint32_t*>(dst + pidx(8 * i));
        d[0] = v.x;
        d[1] = v.y;
        d[2] = v.z;
        d[3] = v.w;
    }
}

// ------------------------------------------------------- phase 1: bytes
__device__ inline void load_bytes(const uint8_t* __restrict__ chunk, const TileGeom& g, uint32_t* dst32) {
    // [Q0, BE) -> dst; Q0 is a multiple of 64 relative to the chunk start and
    // chunks start 16-byte aligned, so the bulk moves as 16-byte vectors.
    const uint32_t nbytes = g.BE - g.Q0;
    const uint8_t* src = chunk + g.Q0;
    // dd blocks of a size that is not a multiple of 16 start unaligned
    const uint32_t nvec = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) ? nbytes / 16 : 0;
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4 = reinterpret_cast<uint4*>(dst32);
    for (uint32_t i = threadIdx.x; i < nvec; i += blockDim.x) d4[i] = __ldg(s4 + i);
    uint8_t* d8 = reinterpret_cast<uint8_t*>(dst32);
    for (uint32_t i = nvec * 16 + threadIdx.x; i < nbytes + 8; i += blockDim.x)
        d8[i] = (i < nbytes) ? src[i] : 0;
}

// ------------------------------------------------------- phase 2: ranks
// dtab[c] = T[c+1] - T[c] (c = 0..63): entropy change when a byte value's
// count in the window goes from c to c+1 (entr64_inc_int, entr64.cc:47-71,
// written as differences of the table of entr64_table_init_int); dtab[64]
// = 0 pads the table for the branch-free step pair.
//
// Each of kRankThreads threads owns a run of positions starting at a
// multiple of 8 and keeps the byte counts of its window in its own
// histogram.  The counts are the only thing carried from step to step, so
// everything else is moved out of that chain: bytes are read as words a
// group ahead, two steps share one round of count loads (the second step's
// counts corrected for the first step in registers), and the eight ranks of
// a group are stored together as four words.
__device__ __forceinline__ uint32_t byte_of(uint32_t w, uint32_t k) { return __byte_perm(w, 0, 0x4440u | k); }

// Two window steps: bytes a0, a1 leave, b0, b1 enter; e0 / e1 receive the
// entropy after each step.
__device__ __forceinline__ void rank_pair(uint8_t* h, uint32_t hbase, const int32_t* dtab, int32_t& e, uint32_t a0,
                                          uint32_t b0, uint32_t a1, uint32_t b1, int32_t& e0, int32_t& e1) {
    const uint32_t ha0 = hbase + ((a0 >> 2) << 7) + (a0 & 3), hb0 = hbase + ((b0 >> 2) << 7) + (b0 & 3);
    const uint32_t ha1 = hbase + ((a1 >> 2) << 7) + (a1 & 3), hb1 = hbase + ((b1 >> 2) << 7) + (b1 & 3);
    const int32_t ca0 = h[ha0], cb0 = h[hb0];
    int32_t ca1 = h[ha1], cb1 = h[hb1];
    // no branches: when a step's leaving and entering bytes are equal, its
    // two counters are one, the stores below write that count back
    // unchanged, its entropy change is dropped, and the second step's
    // corrections are 0 (dtab has a 0 at index 64 for a count of 64 there)
    const int32_t d0 = (int32_t)(a0 != b0), d1 = (int32_t)(a1 != b1);
    const int32_t x0 = dtab[cb0] - dtab[ca0 - 1];
    ca1 += (int32_t)(a1 == b0) - (int32_t)(a1 == a0);
    cb1 += (int32_t)(b1 == b0) - (int32_t)(b1 == a0);
    e += d0 ? x0 : 0;
    e0 = e;
    const int32_t x1 = dtab[cb1] - dtab[ca1 - 1];
    e += d1 ? x1 : 0;
    e1 = e;
    h[ha0] = (uint8_t)(ca0 - d0);
    h[hb0] = (uint8_t)(cb0 + d0);
    h[ha1] = (uint8_t)(ca1 - d1);
    h[hb1] = (uint8_t)(cb1 + d1);
}

// One window step: byte a leaves, byte b enters.
__device__ __forceinline__ void rank_single(uint8_t* h, uint32_t hbase, const int32_t* dtab, int32_t& e, uint32_t a,
                                            uint32_t b) {
    if (a != b) {
        const uint32_t ha = hbase + ((a >> 2) << 7) + (a & 3);
        const uint32_t hb = hbase + ((b >> 2) << 7) + (b & 3);
        const uint32_t ca = h[ha], cb = h[hb];
        h[ha] = (uint8_t)(ca - 1);
        h[hb] = (uint8_t)(cb + 1);
        e += dtab[cb] - dtab[ca - 1];
    }
}

// Where a run of ranks goes: the tile's padded shared-memory array, or a
// chunk's ranks in global memory (a group of eight as one 16-byte store).
struct SmemRanks {
    uint16_t* r;
    __device__ __forceinline__ void one(uint32_t o, uint16_t v) const { r[pidx(o)] = v; }
    __device__ __forceinline__ void eight(uint32_t o, const uint32_t (&w)[4]) const {
        uint32_t* p = reinterpret_cast<uint32_t*>(r + pidx(o));
#pragma unroll
        for (int k = 0; k < 4; k++) p[k] = w[k];
    }
};
struct GlobalRanks {
    uint16_t* r;  // 16-byte aligned
    __device__ __forceinline__ void one(uint32_t o, uint16_t v) const { r[o] = v; }
    __device__ __forceinline__ void eight(uint32_t o, const uint32_t (&w)[4]) const {
        *reinterpret_cast<uint4*>(r + o) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};

// Ranks of positions [lo, hi) of the bytes at b32 (lo a multiple of 8):
// entropy ranks for [lo, vend), 0 for [vend, hi).  Bytes up to vend+62
// must be present, plus 8 bytes of padding; h + hbase is the thread's
// cleared histogram (hist_off layout).
template <class Out>
__device__ __forceinline__ void rank_run(const uint32_t* b32, uint8_t* h, uint32_t hbase, const uint16_t* rank_tab,
                                         const int32_t* dtab, uint32_t lo, uint32_t vend, uint32_t hi,
                                         const Out& out) {
    const uint8_t* b8 = reinterpret_cast<const uint8_t*>(b32);
    int32_t e = 0;
    uint32_t r = lo;
    if (r < vend) {
        // entr64_init_int (entr64.cc:27-41) built incrementally, two bytes
        // per round of count loads; lo is a multiple of 8, so the window's 64
        // bytes are 16 aligned words, read four at a time
#pragma unroll 1
        for (int q = 0; q < 16; q += 4) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; k++) w[k] = b32[(lo >> 2) + q + k];
#pragma unroll
            for (int k = 0; k < 16; k += 2) {
                const uint32_t v0 = byte_of(w[k >> 2], k & 3), v1 = byte_of(w[k >> 2], (k & 3) + 1);
                const uint32_t o0 = hbase + ((v0 >> 2) << 7) + (v0 & 3), o1 = hbase + ((v1 >> 2) << 7) + (v1 & 3);
                const int32_t c0 = h[o0];
                const int32_t c1 = h[o1] + (int32_t)(v0 == v1);
                e += dtab[c0] + dtab[c1];
                h[o0] = (uint8_t)(c0 + 1);
                h[o1] = (uint8_t)(c1 + 1);  // the same counter when v0 == v1: this store wins
            }
        }
        out.one(r, rank_tab[e >> 10]);
        r++;
    }
    // single steps up to the next multiple of 8
    for (; r < vend && (r & 7u); r++) {
        rank_single(h, hbase, dtab, e, b8[r - 1], b8[r + 63]);
        out.one(r, rank_tab[e >> 10]);
    }
    // groups of eight: leaving bytes r-1..r+6, entering r+63..r+70 (three
    // aligned words each, the next group's words loaded ahead)
    if (r + 8 <= vend) {
        uint32_t lw0 = b32[(r - 4) >> 2], lw1 = b32[r >> 2], lw2 = b32[(r + 4) >> 2];
        uint32_t ew0 = b32[(r + 60) >> 2], ew1 = b32[(r + 64) >> 2], ew2 = b32[(r + 68) >> 2];
        for (; r + 8 <= vend; r += 8) {
            uint32_t nl0 = 0, nl1 = 0, nl2 = 0, ne0 = 0, ne1 = 0, ne2 = 0;
            if (r + 16 <= vend) {
                nl0 = b32[(r + 4) >> 2];
                nl1 = b32[(r + 8) >> 2];
                nl2 = b32[(r + 12) >> 2];
                ne0 = b32[(r + 68) >> 2];
                ne1 = b32[(r + 72) >> 2];
                ne2 = b32[(r + 76) >> 2];
            }
            uint32_t a[8], b[8];
            a[0] = byte_of(lw0, 3);
            b[0] = byte_of(ew0, 3);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                a[1 + k] = byte_of(lw1, k);
                b[1 + k] = byte_of(ew1, k);
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                a[5 + k] = byte_of(lw2, k);
                b[5 + k] = byte_of(ew2, k);
            }
            int32_t ev[8];
#pragma unroll
            for (int k = 0; k < 8; k += 2) rank_pair(h, hbase, dtab, e, a[k], b[k], a[k + 1], b[k + 1], ev[k], ev[k + 1]);
            uint32_t rk[4];
#pragma unroll
            for (int k = 0; k < 4; k++)
                rk[k] = (uint32_t)rank_tab[ev[2 * k] >> 10] | ((uint32_t)rank_tab[ev[2 * k + 1] >> 10] << 16);
            out.eight(r, rk);
            lw0 = nl0;
            lw1 = nl1;
            lw2 = nl2;
            ew0 = ne0;
            ew1 = ne1;
            ew2 = ne2;
        }
    }
    for (; r < vend; r++) {
        rank_single(h, hbase, dtab, e, b8[r - 1], b8[r + 63]);  // byte r-1 leaves, byte r+63 enters
        out.one(r, rank_tab[e >> 10]);
    }
    for (; r < hi; r++) out.one(r, 0);  // the last 64 positions of a chunk
}

__device__ inline void compute_ranks(const TileGeom& g, const TileSmem& s, const uint16_t* rank_tab,
                                     const int32_t* dtab) {
    const uint32_t np = g.RE - g.Q0;
    const uint32_t per = ((np + kRankThreads - 1) / kRankThreads + 7) & ~7u;
    const uint32_t tid = threadIdx.x;
    if (tid >= (uint32_t)kRankThreads) return;
    const uint32_t lo = min(np, tid * per), hi = min(np, lo + per);
    const uint32_t last = g.n - kWin;  // ranks exist for o < n-64 only
    const uint32_t vend = last > g.Q0 ? min(hi, last - g.Q0) : lo;  // [lo, vend): entropy ranks
    rank_run(s.bytes32, s.hist, hist_off(tid, 0), rank_tab, dtab, lo, vend, hi, SmemRanks{s.ranks});
}

// ------------------------------------- phase 3: full-rescan result per step
// For step k with rank[k] > 0 the full rescan of gen_chunk_scores picks the
// smallest non-zero rank m of window [k, k+63], at its leftmost position f,
// extended right over the run of equal ranks (capped at k+63).  Stored as
// (m << 6) | (p - k); kNoRes when rank[k] == 0 (no credit, next step rescans).
//
// A position's key is (its rank, the end of its run of equal ranks): the
// smallest key of a window is the leftmost run of its smallest rank, and it
// holds that run's end.  Keys are (r - 1) * 64 + e, so that a rank of 0 wraps
// around to above every key.  One thread per aligned 64-step block A (steps
// base..base+63); the window of step base+u is A[u..63] followed by
// B[0..u-1], B the next block.
//  pass 1, u = 63..0: suffix minimum of A's keys (run ends inside A), written
//    to fres[base+u] (kNoRes when rank[base+u] == 0);
//  pass 2, v = 0..62: the smallest rank of the prefix B[0..v] and the end of
//    its leftmost run so far.  T is what a rank's (r - 1) * 64 + 63 may be at
//    most to change them: that of the minimum while its run is open (an equal
//    rank extends the run), less than it once the run has ended.  Step
//    u = v+1 takes A's minimum on ties (leftmost); when A's is the run that
//    ends at A's last position and B starts with the same rank, the run goes
//    on into B.  Run ends stay within the window, so no cap is needed.
// Positions past the tile's last step are read but only feed steps that no
// walk uses (every array extends past them).
//
// What bounds the tile kernels is the integer pipe (79 % busy, issue 72 %):
// both passes are a handful of compares, selects and minima per step, the
// multiplications and additions left to the other pipe: 8,300 cycles of a
// tile's 47,600 (running minimum, run end and previous rank as separate states:
// 12,100), the tile kernel 14.8 to 13.7 ms on 3.1 GB, k_block_digest 5.1 to
// 4.6 ms on 1 GiB.
//
// Both passes move eight steps at a time: the next group's ranks (two per
// 32-bit word; pidx keeps a block contiguous and 4-byte aligned) are loaded
// before the current group's results are stored, so no load waits behind a
// store.
constexpr uint32_t kNoRes = kNoRank << 6;  // full-rescan result: no rank
__device__ inline void compute_fres(const TileGeom& g, const TileSmem& s) {
    const uint32_t nsteps = g.SE - g.Q0;
    const uint32_t nblk = (nsteps + 63) / 64;
    for (uint32_t j = threadIdx.x; j < nblk; j += blockDim.x) {
        const uint32_t base = j * 64;
        const uint32_t* __restrict__ Ra = reinterpret_cast<const uint32_t*>(s.ranks + pidx(base));
        const uint32_t* __restrict__ Rb = reinterpret_cast<const uint32_t*>(s.ranks + pidx(base + 64));
        uint32_t* __restrict__ Fa = reinterpret_cast<uint32_t*>(s.fres + pidx(base));
        // pass 1: suffix minima of A's keys, steps 63..0
        uint32_t key = 0xFFFFFFFFu, e = 0, rn = 0xFFFFu;  // e: the run's end - 64
        uint32_t cur[4], nxt[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; q++) cur[q] = Ra[28 + q];
        uint32_t first = 0;  // key of step 0
        uint32_t any = 0;    // OR of block A's ranks
        uint32_t u0 = 0u - 8u;  // position of the group's first step - 64
#pragma unroll 1
        for (int gi = 7; gi >= 0; gi--, u0 -= 8) {
            any |= cur[0] | cur[1] | cur[2] | cur[3];
            if (gi > 0) {
#pragma unroll
                for (int q = 0; q < 4; q++) nxt[q] = Ra[4 * (gi - 1) + q];
            }
            uint32_t out[4];
#pragma unroll
            for (int q = 3; q >= 0; q--) {
                uint32_t o2[2];
#pragma unroll
                for (int h = 1; h >= 0; h--) {
                    const uint32_t r = h ? (cur[q] >> 16) : (cur[q] & 0xFFFFu);
                    e = r == rn ? e : u0 + 2 * q + h;
                    key = min(key, r * 64 + e);
                    o2[h] = r == 0 ? kNoRes : key;
                    rn = r;
                }
                out[q] = __byte_perm(o2[0], o2[1], 0x5410);
            }
            first = out[0] & 0xFFFFu;
#pragma unroll
            for (int q = 0; q < 4; q++) Fa[4 * gi + q] = out[q];
#pragma unroll
            for (int q = 0; q < 4; q++) cur[q] = nxt[q];
        }
        // a block whose ranks are all 0 (low-entropy content) is done: no
        // step has a result, as pass 1 wrote
        if (any == 0) continue;
        // pass 2: prefix states of B, steps u = v + 1 = 1..63; results are
        // packed into aligned words with the previous group's last one
        uint32_t rb[4], fa[5], nrb[4] = {0, 0, 0, 0}, nfa[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; q++) rb[q] = Rb[q];
#pragma unroll
        for (int q = 0; q < 5; q++) fa[q] = Fa[q];
        // A's run up to its last position goes on into B's leading run
        const uint32_t rb0 = rb[0] & 0xFFFFu, r63 = Ra[31] >> 16;
        const bool cont = r63 != 0 && r63 == rb0;
        const uint32_t tail = cont ? r63 * 64 - 1 : 0xFFFFFFFFu;  // that run's key in A
        bool lead_open = true;
        uint32_t lead = tail;  // with its end so far in B
        uint32_t pm = kNoRes - 1, T = pm, pval = 0;  // smallest rank of B's prefix as (r - 1) * 64 + 63; its key
        uint32_t carry = first == kNoRes ? kNoRes : first + 64;
        uint32_t v0 = 0;
#pragma unroll 1
        for (uint32_t gi = 0; gi < 8; gi++, v0 += 8) {
            if (gi < 7) {
#pragma unroll
                for (int q = 0; q < 4; q++) nrb[q] = Rb[4 * (gi + 1) + q];
#pragma unroll
                for (int q = 0; q < 4; q++) nfa[q] = Fa[4 * (gi + 1) + q];
                nfa[4] = gi < 6 ? Fa[4 * (gi + 1) + 4] : 0u;
            }
            uint32_t res[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const uint32_t r = (t & 1) ? (rb[t >> 1] >> 16) : (rb[t >> 1] & 0xFFFFu);
                lead_open = lead_open && r == rb0;
                lead += lead_open;
                const uint32_t q = r * 64 - 1;
                const bool upd = q <= T;
                pm = upd ? q : pm;
                pval = upd ? q + v0 + (t + 1) : pval;
                T = upd ? q : pm - 1;
                // step u = v + 1: its suffix minimum is halfword t + 1 of fa
                const uint32_t sv = ((t + 1) & 1) ? (fa[(t + 1) >> 1] >> 16) : (fa[(t + 1) >> 1] & 0xFFFFu);
                const uint32_t a = sv == tail ? lead : sv;
                const uint32_t w = sv <= pm ? a : pval;
                res[t] = sv == kNoRes ? kNoRes : w + (63 - t) - v0;  // + 64 - u
            }
            // steps 8gi .. 8gi+7 as words 4gi .. 4gi+3 (step 8gi from the carry)
            Fa[4 * gi] = __byte_perm(carry, res[0], 0x5410);
            Fa[4 * gi + 1] = __byte_perm(res[1], res[2], 0x5410);
            Fa[4 * gi + 2] = __byte_perm(res[3], res[4], 0x5410);
            Fa[4 * gi + 3] = __byte_perm(res[5], res[6], 0x5410);
            carry = res[7];  // step 8gi + 8 (the next block's step 0 when gi == 7: dropped)
#pragma unroll
            for (int q = 0; q < 4; q++) rb[q] = nrb[q];
#pragma unroll
            for (int q = 0; q < 5; q++) fa[q] = nfa[q];
        }
    }
}

// ------------------------------------------------------ phase 4: chains
// Run-length credit accumulator: a cheap slide credits the same position
// many times in a row, so credits are added to the shared score array only
// when the credited position changes.
template <int kSign>
struct Credit {
    uint32_t score;       // the score array's shared-memory address
    uint32_t lo, hi;      // credited positions [lo, hi) (chunk-relative)
    uint32_t cur, start;  // position credited by the open run of steps (~0u: none) and its first step
    // adds the run's steps [start, i) to cur's score where it is in range and
    // `when` holds: one predicated reduction, where the branch the compiler
    // puts around an atomicAdd was a tenth of the walk (19,700 to 17,600
    // cycles of a tile; tiles of 3.1 GB 13.6 to 13.0 ms)
    __device__ __forceinline__ void close(uint32_t i, bool when) {
        const uint32_t o = cur - lo;
        const uint32_t inc = __funnelshift_l(0u, kSign > 0 ? i - start : start - i, 8 * o);  // shifts by 8 * (o & 3)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p red.shared.add.u32 [%0], %1;\n\t}"
                     ::"r"(score + (o & ~3u)), "r"(inc), "r"((uint32_t)(when && o < hi - lo)) : "memory");
    }
    // closes the open run at step i
    __device__ __forceinline__ void flush(uint32_t i) { close(i, i > start); }
    // step i credits p when act (its window has a rank); a step that
    // credits nothing opens a run of ~0u, which is never added
    __device__ __forceinline__ void add(uint32_t i, uint32_t p, bool act) {
        const uint32_t key = act ? p : ~0u;
        const bool chg = key != cur;
        close(i, chg);
        cur = key;
        start = chg ? i : start;
    }
};

// One step of gen_chunk_scores (sdbf_core.cc:59-80) from state st, given
// rank[i+64] and the full-rescan result of step i.
template <typename CR>
__device__ __forceinline__ void walk_step(ChainState& st, uint32_t i, uint32_t r64, uint32_t f, CR* cr) {
    const bool cheap = (r64 >= st.M) & (i < st.P);  // never with M == kNoRank
    const uint32_t cheapP = (r64 == st.M) ? i + 64 : st.P;
    st.P = cheap ? cheapP : i + (f & 63);
    st.M = cheap ? st.M : (f >> 6);
    if (cr) cr->add(i, st.P, st.M != kNoRank);
}

// Eight consecutive 16-bit entries starting at an 8-aligned index (inside
// one 64-block of the padded layout), one load each: the load path has room,
// taking words apart would be two more instructions per step on the integer
// pipe that bounds the kernel.
__device__ __forceinline__ void load8(const uint16_t* p, uint32_t* w) {
#pragma unroll
    for (int k = 0; k < 8; k++) w[k] = p[k];
}

// Walk steps [a, b) of gen_chunk_scores from state `st` (st.M == kNoRank makes step
// a a full rescan: the speculative start, or step 0).  Single steps up to an
// 8-aligned step (Q0 is a multiple of 64, so tile offsets are aligned too),
// then groups of eight whose operands (rank[i+64..], fres[i..]) are loaded
// one group ahead.  With rec set, the state entering step chk is stored
// there (the steps before chk then run one at a time).
template <typename CR>
__device__ __forceinline__ ChainState walk(const TileGeom& g, const TileSmem& s, uint32_t a, uint32_t b,
                                           ChainState st, CR* cr, uint32_t chk = 0, uint64_t* rec = nullptr) {
    const uint16_t* __restrict__ R = s.ranks;
    const uint16_t* __restrict__ Fr = s.fres;
    uint32_t i = a;
    if (rec && chk >= a && chk < b) {
        for (; i < chk; i++) walk_step(st, i, R[pidx(i + 64 - g.Q0)], Fr[pidx(i - g.Q0)], cr);
        *rec = pack_state(st);
    }
    for (; i < b && (i & 7u); i++) walk_step(st, i, R[pidx(i + 64 - g.Q0)], Fr[pidx(i - g.Q0)], cr);
    if (i + 8 <= b) {
        uint32_t rw[8], fw[8];
        load8(R + pidx(i + 64 - g.Q0), rw);
        load8(Fr + pidx(i - g.Q0), fw);
        for (; i + 8 <= b; i += 8) {
            uint32_t nrw[8] = {}, nfw[8] = {};
            if (i + 16 <= b) {
                load8(R + pidx(i + 72 - g.Q0), nrw);
                load8(Fr + pidx(i + 8 - g.Q0), nfw);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) walk_step(st, i + k, rw[k], fw[k], cr);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                rw[k] = nrw[k];
                fw[k] = nfw[k];
            }
        }
    }
    for (; i < b; i++) walk_step(st, i, R[pidx(i + 64 - g.Q0)], Fr[pidx(i - g.Q0)], cr);
    return st;
}

// Re-walk segment [St, Et) from its true entry state `nw` next to the chain
// it was credited with (`old`, from its speculative entry).  Both walks run
// in lockstep; credits differ only until the two states coincide, after
// which the rest of the old walk (and its exit state) stands.  Returns the
// segment's exit state.
__device__ uint64_t relink_segment(const TileGeom& g, const TileSmem& s, uint32_t St, uint32_t Et, ChainState old,
                                   ChainState nw, uint32_t chk, uint64_t old_exit) {
    Credit<-1> un{(uint32_t)__cvta_generic_to_shared(s.score32), g.t0, g.t0 + g.L, ~0u, St};
    Credit<1> re{(uint32_t)__cvta_generic_to_shared(s.score32), g.t0, g.t0 + g.L, ~0u, St};
    uint32_t i = St;
    for (; i < Et; i++) {
        if (pack_state(old) == pack_state(nw)) break;
        if (i == chk) *reinterpret_cast<uint64_t*>(&s.misc[10]) = pack_state(nw);
        const uint32_t r64 = s.ranks[pidx(i + 64 - g.Q0)], f = s.fres[pidx(i - g.Q0)];
        walk_step(old, i, r64, f, &un);
        walk_step(nw, i, r64, f, &re);
    }
    un.flush(i);
    re.flush(i);
    return i < Et ? old_exit : pack_state(nw);
}

__device__ __forceinline__ void stamp(long long* tm, int k) {
    if (tm && threadIdx.x == 0) tm[k] = clock64();
}

// Walk segment [St, Et) from `st` with credits of sign kSign; records the
// state entering step chk (the next tile's first credited step) when the
// segment contains it.
template <int kSign>
__device__ __forceinline__ ChainState walk_segment(const TileGeom& g, const TileSmem& s, uint32_t St, uint32_t Et,
                                                   ChainState st, uint32_t chk) {
    Credit<kSign> cr{(uint32_t)__cvta_generic_to_shared(s.score32), g.t0, g.t0 + g.L, ~0u, St};
    st = walk(g, s, St, Et, st, &cr, chk, kSign > 0 ? reinterpret_cast<uint64_t*>(&s.misc[10]) : nullptr);
    cr.flush(Et);
    return st;
}

// Runs all phases for one tile.  entry != nullptr: the state entering step
// S0 is known (re-computation after a failed link check); otherwise thread 0
// starts speculatively `lead` steps early.  Writes sig_in / tau_out.
// kPre: the ranks come from pre_ranks (the chunk's precomputed ranks)
// instead of the chunk bytes.
template <bool kPre = false, bool kBlock = kPre>
__device__ void tile_pipeline(const uint8_t* __restrict__ chunk, const TileGeom& g, const TileSmem& s,
                              const uint16_t* rank_tab, const int32_t* dtab, const uint64_t* entry,
                              uint64_t* sig_in, uint64_t* tau_out, uint32_t lead, long long* tm,
                              const uint16_t* pre_ranks = nullptr) {
    stamp(tm, 0);
    if constexpr (kPre) {
        load_ranks<kBlock>(pre_ranks, g, s.ranks);
        __syncthreads();
        stamp(tm, 1);
    } else {
        load_bytes(chunk, g, s.bytes32);
        {
            uint4* h4 = reinterpret_cast<uint4*>(s.hist);
            for (uint32_t i = threadIdx.x; i < 256 * kRankThreads / 16; i += blockDim.x)
                h4[i] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
        stamp(tm, 1);
        compute_ranks(g, s, rank_tab, dtab);
        __syncthreads();
    }
    stamp(tm, 2);
    compute_fres(g, s);
    // clear scores (in-tile ranks: aliases the histogram area, free after phase 2)
    for (uint32_t i = threadIdx.x; i < (g.L + 3) / 4 + 1; i += blockDim.x) s.score32[i] = 0;
    if (threadIdx.x == 0) {
        s.misc[9] = 0;
        s.misc[10] = 0;
        s.misc[11] = 0;
    }
    __syncthreads();
    stamp(tm, 3);
    // segments over steps [S0, SE)
    const uint32_t total = g.SE > g.S0 ? g.SE - g.S0 : 0;
    // segment length a multiple of 8 (S0 is a multiple of 64): every walk then
    // starts and ends on a group of eight steps (trailing threads may idle)
    const uint32_t SL = ((total + kSegs - 1) / kSegs + 7) & ~7u;
    const uint32_t chk = g.t0 + g.L - 64;  // next tile's S0
    const uint32_t t = threadIdx.x;
    const uint32_t St = g.S0 + t * SL;
    const uint32_t Et = min(St + SL, g.SE);
    const bool has_seg = t < kSegs && SL > 0 && St < g.SE;
    if (t < kSegs) {
        if (has_seg) {
            ChainState st{0, kNoRank};
            if (t == 0 && entry) {
                st = unpack_state(*entry);
            } else {
                // lead-in, not below the first simulated step; a lead-in
                // from step 0 makes the walk exact.  The tile's first segment
                // has the same lead as the others (a longer one would hold up
                // its warp): its rare mis-speculation costs a tile recompute
                // in k_stream_fix.
                const uint32_t Ls = St - min(St - g.Q0, lead);
                st = walk(g, s, Ls, St, st, (Credit<1>*)nullptr);
            }
            s.sig[t] = pack_state(st);
            s.tau[t] = pack_state(walk_segment<1>(g, s, St, Et, st, chk));
        } else {
            s.sig[t] = ~0ull;
            s.tau[t] = ~0ull;
        }
    }
    __syncthreads();
    stamp(tm, 4);
    // phase 5: link segments.  A segment is exact iff its entry state equals
    // its left neighbour's exit state; mismatched segments are re-walked in
    // parallel rounds until every link holds (normally zero rounds).
    while (true) {
        bool need = false;
        uint64_t from = 0;
        if (has_seg && t >= 1) {
            from = s.tau[t - 1];
            need = s.sig[t] != from;
        }
        if (!__syncthreads_or(need)) break;
        if (need) {
            const uint64_t out = relink_segment(g, s, St, Et, unpack_state(s.sig[t]), unpack_state(from), chk,
                                                s.tau[t]);
            s.sig[t] = from;
            s.tau[t] = out;
            atomicAdd(&s.misc[9], 1u);
        }
        __syncthreads();
    }
    if (t == 0) {
        if (sig_in) *sig_in = s.sig[0];
        if (tau_out) *tau_out = *reinterpret_cast<uint64_t*>(&s.misc[10]);
    }
    __syncthreads();
    stamp(tm, 5);
}

// ------------------------------------------- phase 6: ordered compaction
// The positions (relative to t0) whose score is at least kGe, in one pass.
// Warp w writes its own to lists + w * stride and their number to counts[w];
// entry f of all is entry f - (the counts of earlier warps) of the first warp
// list that reaches it.  A lane reads 16 scores (one 16-byte load; a warp's
// 32 loads are one contiguous 512-byte run) and gets their selection bits
// from four byte-parallel compares; a shuffle scan of the lanes' counts
// places them.  (Bytes are scores <= 65, so no byte borrows from its
// neighbour.)  Each step credits one position in [i, i+64], so at most
// (R + 64) / kGe positions of a warp's range of R reach kGe.
__device__ __forceinline__ uint32_t sel4(uint32_t w, uint32_t t4) {
    const uint32_t hb = ((w | 0x80808080u) - t4) & 0x80808080u;
    return (hb >> 7 | hb >> 14 | hb >> 21 | hb >> 28) & 0xFu;
}
template <uint32_t kGe, class T>
__device__ __forceinline__ uint32_t compact_warp(const uint32_t* score32, uint32_t nown, T* lists, uint32_t stride) {
    const uint32_t nq = (nown + 15) / 16;  // 16-position quads
    const uint32_t nwarps = blockDim.x / 32, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t per = ((nq + nwarps - 1) / nwarps + 31) / 32 * 32;
    const uint32_t q0 = min(nq, wid * per), q1 = min(nq, q0 + per);
    T* list = lists + wid * stride;
    const uint4* sc4 = reinterpret_cast<const uint4*>(score32);
    const uint32_t t4 = kGe * 0x01010101u;
    uint32_t n = 0;
    for (uint32_t qb = q0; qb < q1; qb += 32) {
        const uint32_t q = qb + lane;
        uint32_t m = 0;
        if (q < q1) {
            const uint4 w = sc4[q];
            m = sel4(w.x, t4) | (sel4(w.y, t4) << 4) | (sel4(w.z, t4) << 8) | (sel4(w.w, t4) << 12);
            if (16 * q + 16 > nown) m &= (1u << (nown - 16 * q)) - 1u;
        }
        const uint32_t c = __popc(m);
        uint32_t incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        uint32_t pos = n + incl - c;
        while (m) {
            list[pos++] = (T)(16 * q + (uint32_t)(__ffs(m) - 1));
            m &= m - 1u;
        }
        n += __shfl_sync(0xffffffffu, incl, 31);
    }
    return n;
}
constexpr uint32_t kWarpList = 128;  // stream tiles: at most (2,048 + 64) / 17 = 124 per warp

// ---------------------------------------------------------- stream tiles
__device__ inline TileGeom stream_geom(uint32_t n, uint32_t t0) {
    TileGeom g;
    g.n = n;
    g.t0 = t0;
    g.L = kTileL;
    g.S0 = t0 >= 64 ? t0 - 64 : 0;
    const uint32_t last = n - kWin;
    g.SE = min(t0 + kTileL, last);
    g.Q0 = g.S0 > kLead ? g.S0 - kLead : 0;
    g.RE = min(g.SE + 64, n);
    g.BE = min(g.RE + 63, n);
    return g;
}

// A tile's features in GenParams::features: words 0..3 of each feature as one
// uint4, then the fifth words.
__device__ __forceinline__ uint32_t feat_word(uint32_t f, int k) { return k < 4 ? 4 * f + k : 4 * kTileCap + f; }

// kPre: ranks precomputed in P.ranks (tile_smem_bytes_pre layout); the
// SHA-1 phase then reads the feature bytes from global memory.
template <bool kPre>
__device__ void stream_tile_body(const GenParams& P, uint32_t tile, const uint64_t* entry, uint8_t* smem) {
    const GenTile T = P.tiles[tile];
    const GenChunk C = P.chunks[T.chunk];
    const TileGeom g = stream_geom(C.n, T.t0);
    TileSmem s = kPre ? carve_pre(smem, kTileL) : carve(smem, kTileL);
    const uint16_t* rank_tab = nullptr;
    const int32_t* dt = nullptr;
    if constexpr (!kPre) {
        __shared__ int32_t dtab[65];
        for (uint32_t i = threadIdx.x; i < 65; i += blockDim.x)
            dtab[i] = i < 64 ? (int32_t)P.ent_tab[i + 1] - (int32_t)P.ent_tab[i] : 0;
        // the rank table (2 KB) in shared memory: a lookup is one shared-memory read
        __shared__ uint16_t s_rank[(SDBF_RANK_BINS + 7) / 8 * 8];
        for (uint32_t i = threadIdx.x; i < SDBF_RANK_BINS; i += blockDim.x) s_rank[i] = P.rank_tab[i];
        __syncthreads();
        rank_tab = s_rank;
        dt = dtab;
    }
    TileOut* out = P.tile_out + tile;
    long long tm[9];
    const uint8_t* chunk = P.data + C.data_off;
    tile_pipeline<kPre, false>(chunk, g, s, rank_tab, dt, entry, &out->sig_in, &out->tau_out, P.lead,
                        P.phase ? tm : nullptr, kPre ? P.ranks + (size_t)C.rank_off8 * 8 : nullptr);
    const uint32_t nown = g.SE > g.t0 ? g.SE - g.t0 : 0;
    __shared__ uint32_t counts[kGenThreads / 32];
    static_assert(kGenThreads / 32 == 4 && 4 * kWarpList <= (kTileL + 64) / 15 + 8, "stream list layout");
    const uint32_t nsel = compact_warp<kThreshold + 1>(s.score32, nown, s.list, kWarpList);
    if ((threadIdx.x & 31) == 0) counts[threadIdx.x >> 5] = nsel;
    __syncthreads();
    const uint32_t c1 = counts[0], c2 = c1 + counts[1], c3 = c2 + counts[2], nf = c3 + counts[3];
    stamp(P.phase ? tm : nullptr, 6);
    // SHA-1 of each selected feature (sdbf_core.cc:103-105)
    uint32_t* feat = P.features + (size_t)tile * 5 * kTileCap;
    const uint32_t off = g.t0 - g.Q0;
    for (uint32_t f = threadIdx.x; f < nf; f += blockDim.x) {
        const uint32_t wl = (f >= c1) + (f >= c2) + (f >= c3);
        const uint32_t before = wl == 0 ? 0u : wl == 1 ? c1 : wl == 2 ? c2 : c3;
        const uint32_t p = s.list[wl * kWarpList + (f - before)] + off;
        uint32_t w[16], h[5];
        if constexpr (kPre)
            load_be16_global(chunk + g.Q0 + p, w);
        else
            load_be16(s.bytes32, p, w);
        sha1_feature(w, h);
        static_assert(5 * kTileCap % 4 == 0, "a tile's features start 16-byte aligned");
        reinterpret_cast<uint4*>(feat)[f] = make_uint4(h[0], h[1], h[2], h[3]);
        feat[4 * kTileCap + f] = h[4];
    }
    if (threadIdx.x == 0) {
        out->count = nf;
        out->fixups = s.misc[9];
    }
    if (P.phase) {
        __syncthreads();
        stamp(tm, 7);
        if (threadIdx.x == 0) {
            for (int k = 0; k < 7; k++) atomicAdd(P.phase + k, (unsigned long long)(tm[k + 1] - tm[k]));
            atomicAdd(P.phase + kPhTiles, 1ull);
            atomicAdd(P.phase + kPhFixups, (unsigned long long)s.misc[9]);
        }
    }
}

__global__ void __launch_bounds__(kGenThreads, 4) k_stream_tiles(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    for (uint32_t tile = blockIdx.x; tile < P.ntiles; tile += gridDim.x) {
        stream_tile_body<false>(P, tile, nullptr, smem);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kGenThreads, 5) k_stream_tiles_pre(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    for (uint32_t tile = blockIdx.x; tile < P.ntiles; tile += gridDim.x) {
        stream_tile_body<true>(P, tile, nullptr, smem);
        __syncthreads();
    }
}

// Link tiles of a chunk: a tile's speculative entry state must equal its
// predecessor's exit state (tiles whose lead-in reaches step 0 are exact).
// k_stream_fix (one CTA per chunk) first checks all links of its chunk, with
// no exit from the loop so that the loads overlap (a 32 MiB chunk has 4,229;
// a warp per chunk that left at the first failing link spent 84 us on the
// six full chunks of a 200 MiB file), and normally ends there; else it recomputes the first failing tile from
// the true entry state and moves on through the chunk: its threads check
// the links of the next kGenThreads tiles at once, and the first failing
// one (a later tile whose entry no longer matches, or an unrelated
// mis-speculation) is recomputed next.
__device__ __forceinline__ bool link_fails(const GenParams& P, const GenChunk& C, uint32_t tile) {
    const TileGeom g = stream_geom(C.n, P.tiles[tile].t0);
    return g.S0 > P.lead && P.tile_out[tile - 1].tau_out != P.tile_out[tile].sig_in;
}

// Before k_stream_fix: every tile whose link fails goes
// to P.fix_list (fix_list[0] = their number, zeroed by the host), and
// k_stream_fix_list recomputes them all at once, one CTA each, from their
// predecessors' exit states as they stand.  A tile whose predecessor is
// recomputed in the same launch may start from the stale state; the
// serial pass that follows finds and redoes it (normally nothing is left).
// A group of at most one tile per resident CTA needs no list: fix_list is
// null and each CTA checks its own tile's link (a stale or a fresh exit state
// read there decides only what the serial pass is left with), which saves a
// memset and a launch, 5 us of the 64 KiB file's digest.
__global__ void __launch_bounds__(256) k_stream_fails(GenParams P) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < P.ntiles; t += gridDim.x * blockDim.x) {
        const GenChunk C = P.chunks[P.tiles[t].chunk];
        if (t > C.first_tile && link_fails(P, C, t)) P.fix_list[1 + atomicAdd(P.fix_list, 1u)] = t;
    }
}

template <bool kPre>
__global__ void __launch_bounds__(kGenThreads) k_stream_fix_list(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t entry;
    const uint32_t n = P.fix_list ? P.fix_list[0] : P.ntiles;
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        uint32_t tile = k;
        if (P.fix_list) {
            tile = P.fix_list[1 + k];
        } else {
            const GenChunk C = P.chunks[P.tiles[k].chunk];
            bool fails = false;
            if (threadIdx.x == 0) fails = k > C.first_tile && link_fails(P, C, k);
            if (!__syncthreads_or(fails)) continue;
        }
        if (threadIdx.x == 0) entry = P.tile_out[tile - 1].tau_out;
        __syncthreads();
        stream_tile_body<kPre>(P, tile, &entry, smem);
        if (threadIdx.x == 0) atomicAdd(P.counters + 0, 1u);
        __syncthreads();
    }
}

template <bool kPre>
__global__ void __launch_bounds__(kGenThreads) k_stream_fix(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t entry;
    __shared__ uint32_t bad_first;
    for (uint32_t c = blockIdx.x; c < P.nchunks; c += gridDim.x) {
        const GenChunk C = P.chunks[c];
        __syncthreads();  // the previous chunk is done with bad_first
        if (threadIdx.x == 0) bad_first = 0xFFFFFFFFu;
        __syncthreads();
        uint32_t mine = 0xFFFFFFFFu;
#pragma unroll 4
        for (uint32_t jj = 1 + threadIdx.x; jj < C.ntiles; jj += blockDim.x)
            if (link_fails(P, C, C.first_tile + jj)) mine = min(mine, jj);
        if (mine != 0xFFFFFFFFu) atomicMin(&bad_first, mine);
        __syncthreads();
        uint32_t j = bad_first;
        __syncthreads();
        while (j < C.ntiles) {  // ~0: every link holds
            // the first failing link among tiles [j, j + blockDim.x); tiles
            // recomputed before it are visible here (same CTA, after a barrier)
            if (threadIdx.x == 0) bad_first = 0xFFFFFFFFu;
            __syncthreads();
            const uint32_t jj = j + threadIdx.x;
            if (jj < C.ntiles && link_fails(P, C, C.first_tile + jj)) atomicMin(&bad_first, jj);
            __syncthreads();
            const uint32_t f = bad_first;
            if (f == 0xFFFFFFFFu) {
                j += blockDim.x;
                continue;
            }
            const uint32_t tile = C.first_tile + f;
            if (threadIdx.x == 0) entry = P.tile_out[tile - 1].tau_out;
            __syncthreads();
            stream_tile_body<kPre>(P, tile, &entry, smem);
            if (threadIdx.x == 0) atomicAdd(P.counters + 0, 1u);
            __syncthreads();
            j = f + 1;
        }
    }
}

// ------------------------------------------------------ async copies
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }
// The L2 prefetch of [gmem, gmem+bytes) (16-byte aligned, a multiple of 16 bytes).
__device__ __forceinline__ void prefetch_l2(const void* gmem, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(gmem), "r"(bytes) : "memory");
}

// ------------------------------------------------ precomputed ranks
// Entropy ranks of a stream launch group ahead of its tile kernel.  One CTA
// item is a stretch of kRkThreads x rk_per positions of a chunk, its bytes staged in
// shared memory by 16-byte asynchronous copies (the CTA's next stretch
// prefetched into L2 meanwhile); each thread ranks rk_per consecutive
// positions with its own histogram (rank_run, the tile kernel's rank loop),
// so a thread's 64-byte window set-up is spread over up to 312 positions
// instead of a tile thread's 88.  Ranks of positions >= n-64 are 0; the
// chunk's ranks run to a multiple of 8 (GenChunk::rank_off8).
//
// Positions per thread: the kernel's time is that of a thread's chain of
// 64 + rk_per steps times the number of waves of stretches over the SMs
// (three to an SM).  312 has the least set-up, but leaves most SMs idle
// below 18 MB: rk_choose takes the smallest product.  One file of 64 KiB, 1, 4,
// 8 and 16 MiB: 11, 13, 18, 24 and 37 us; always 312: 21, 21, 22, 27 and 36.
constexpr uint32_t kRkBytes = align_up(rk_span(kRkPerMax) + 64 + 16, 16);  // staged bytes + zero padding
constexpr uint32_t kRkSmem = 256 * kRkThreads + kRkBytes;

__global__ void __launch_bounds__(kRkThreads, 3) k_stream_ranks(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* hist = smem;
    uint32_t* b32 = reinterpret_cast<uint32_t*>(smem + 256 * kRkThreads);
    __shared__ int32_t dtab[65];
    __shared__ uint16_t s_rank[(SDBF_RANK_BINS + 7) / 8 * 8];
    for (uint32_t i = threadIdx.x; i < 65; i += blockDim.x) dtab[i] = i < 64 ? (int32_t)P.ent_tab[i + 1] - (int32_t)P.ent_tab[i] : 0;
    for (uint32_t i = threadIdx.x; i < SDBF_RANK_BINS; i += blockDim.x) s_rank[i] = P.rank_tab[i];
    const uint32_t tid = threadIdx.x, per = P.rk_per, span = rk_span(per);
    for (uint32_t item = blockIdx.x; item < P.nrk_items; item += gridDim.x) {
        const uint2 it = P.rk_items[item];
        const GenChunk C = P.chunks[it.x];
        const uint32_t s0 = it.y, n = C.n;
        const uint32_t np = min(span, align_up(n, 8) - s0);  // positions [s0, s0+np)
        const uint32_t nb = min(span + 64, n - s0);          // bytes [s0, s0+nb)
        __syncthreads();  // the previous stretch is done with the bytes and histograms
        // the stretch's bytes: 16-byte asynchronous copies, all in flight at once
        const uint8_t* src = P.data + C.data_off + s0;
        const uint32_t nvec = ((reinterpret_cast<uintptr_t>(src) & 15) == 0) ? nb / 16 : 0;
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
        uint4* d4 = reinterpret_cast<uint4*>(b32);
        for (uint32_t i = tid; i < nvec; i += blockDim.x) cp_async16(d4 + i, s4 + i);
        cp_async_commit();
        uint8_t* d8 = reinterpret_cast<uint8_t*>(b32);
        for (uint32_t i = nvec * 16 + tid; i < nb + 8; i += blockDim.x) d8[i] = (i < nb) ? src[i] : 0;
        uint4* h4 = reinterpret_cast<uint4*>(hist);
        for (uint32_t i = tid; i < 256 * kRkThreads / 16; i += blockDim.x) h4[i] = make_uint4(0, 0, 0, 0);
        // the CTA's next stretch into L2 while this one is ranked
        if (tid == 0 && item + gridDim.x < P.nrk_items) {
            const uint2 nx = P.rk_items[item + gridDim.x];
            const GenChunk Cn = P.chunks[nx.x];
            const uint8_t* ns = P.data + Cn.data_off + nx.y;
            const uint32_t nnb = min(span + 64, Cn.n - nx.y) & ~15u;
            if ((reinterpret_cast<uintptr_t>(ns) & 15) == 0 && nnb) prefetch_l2(ns, nnb);
        }
        cp_async_wait_all();
        __syncthreads();
        const uint32_t lo = min(np, tid * per), hi = min(np, lo + per);
        const uint32_t last = n > kWin ? n - kWin : 0;  // ranks exist for o < n-64 only
        const uint32_t vend = last > s0 ? min(hi, last - s0) : lo;
        rank_run(b32, hist, hist_off(tid, 0), s_rank, dtab, lo, vend, hi,
                 GlobalRanks{P.ranks + (size_t)C.rank_off8 * 8 + s0});
    }
}

// ------------------------------------------------------- ordered commit
// The ordered filter fill (gen_chunk_hash, sdbf_core.cc:93-136): a feature
// is counted iff it sets a new bit in the 256-byte filter F (bf_sha1_insert)
// and a new bit in the 16 KiB big filter G (query_and_set); F keeps the bits
// of features that fail G.  F rolls over at 160 counted features, G at 8,738
// counted per chunk (the counter is local to a chunk, sdbf_core.cc:100; G
// itself continues).
//
// One CTA per file takes a window of up to kCmWin consecutive features per
// pass, one per thread; the order inside the window is recovered without a
// serial step:
//  * every hash word puts its feature's number into a table of the smallest
//    feature number per 12-bit index (atomicMin; the pass number, counting
//    down, is the key's high part, so a pass overrides its predecessors and
//    the table is never cleared).  The 11-bit filter index of a word is new
//    in F iff it is unset before the window and neither of its two 12-bit
//    entries names an earlier feature;
//  * a big-filter bit whose 12-bit entry names this very feature has no
//    earlier holder in the window, so it is new in G iff it was unset.  A
//    feature whose unset big-filter bits all have an earlier 12-bit holder
//    is compared with the 17-bit values of the earlier F-passing features
//    (slow path; 0.3 features per pass on mixture content);
//  * a prefix count of the counted flags cuts the window behind the feature
//    at which F or G rolls over: exactly the features with fewer counted
//    predecessors than that are applied, the rest start the next pass.
// A filter takes ~163 features, so a pass is normally one whole filter.
// Three barriers per pass: (1) table filled and the last window's bits
// applied, (2) flags known, (3) the window's end known; (2) and (3) are the
// window's threads' only.  A separate warp streams the
// tiles' features into a ring; it meets the others once a pass, at (1), and
// what it publishes there counts from the next pass on, so that its copies
// and its own instructions have a whole pass.
//
// What bounds it: the chain of passes of the largest file -- about 1,000
// cycles of shared-memory work (random words: four cycles per warp
// instruction) and the latency of the barriers.  One 200 MiB file (2.7 M
// features, 16,720 passes of 1,885 cycles) commits in 15.2 ms, 64 files of
// 1 MiB in 0.107 ms; one warp per file taking 32 features per pass took 87.2
// and 0.543 ms.  Measured beside it: a lane per (feature, hash word), 30
// warps: 3,225 cycles per pass; the loading warp taking part in barrier (2):
// 2,740; the window's end found by every warp instead of at barrier (3), and
// F read when it is known to be empty: 2,270.
//
// With an index being built (sdhash --index: sdbf_core.cc:108-114), a
// feature whose filter insert set a new bit is inserted into the index and
// is skipped unless that set a new index bit -- so each file depends on
// every earlier file's features.  Two ways to get that order:
// * k_stream_commit_index: one warp commits all files in input order, one
//   feature at a time, the index in global memory;
// * k_stream_commit_round: one round of a fixed point.  Files commit in
//   parallel; a feature is taken as setting a new index bit iff no feature
//   inserted in the previous round precedes it as the first setter of one of
//   its bits (GenParams::index_pred, one bit per feature), and the inserted
//   features are recorded (GenParams::index_seen).  A file's commit depends
//   only on its own features and their predicate bits, so later rounds
//   re-commit only the files whose bits changed (GenParams::commit_dirty),
//   after clearing their seen bits, from the last checkpoint before the
//   first change.  A round that inserts the same features as the previous
//   one reproduces the sequential result: by induction over the input order,
//   every decision then depends only on earlier decisions that already agree.
constexpr uint32_t kCmWarps = kCmWin / 32;
constexpr uint32_t kCmRing = 1024;  // features staged ahead (a tile has at most kTileCap)
constexpr uint32_t kCmTiles = 4;    // tiles the loading warp starts per pass
static_assert(kCmWin % 32 == 0 && kCmWin <= 256 && kCmThreads == (int)kCmWin + 32, "one thread per window feature");
static_assert(kCmWarps == 6, "the warps' flags are read as a uint4 and a uint2");
static_assert(kCmRing >= kTileCap + 2 * kCmWin, "a tile fits the ring beside two windows");

template <bool kRound>
struct CommitSmem {
    uint4 feat4[kCmRing];                   // hash words 0..3 of the staged features
    uint32_t feat1[kCmRing];                // hash word 4
    alignas(16) uint32_t G[kBigBytes / 4];  // current big filter (cleared and copied in 16-byte words)
    uint32_t tab[4096];                     // (pass key << 8 | feature) of each 12-bit index
    uint32_t F[2][64];                      // current filter (the other one is being written out)
    uint32_t match[kCmWin];                 // slow path: big-filter values held by an earlier feature
    alignas(16) uint32_t counted[8], ambig[8];  // per warp
    uint32_t end;                           // features the pass consumes, when F or G rolls over
    // published before barrier (1) of a pass, by pass parity (a reader may be
    // late by the time until the next barrier (1)):
    uint32_t pos[2];     // the window's start, for the loading warp
    uint32_t avail[2];   // features of the file in the ring so far (end position)
    uint32_t final_[2];  // avail is the end of the segment
    uint32_t seg_pos;    // the segment's end position, once it is through
    uint32_t ord[kRound ? kCmRing : 1];     // index rounds: the feature's ordinal
};
// barrier of the window's threads (the loading warp does not take part)
__device__ __forceinline__ void commit_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCmWin) : "memory"); }

__device__ inline uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_2() { asm volatile("cp.async.wait_group 2;\n" ::); }

// The chop of sdbf_core.cc:235-238: a last filter of few elements is dropped.
__device__ __forceinline__ bool commit_chops(uint32_t bf_count, uint32_t last_count) {
    return bf_count > 1 && last_count < (uint32_t)kMaxElem / 8;
}

// The last filter is out: the file's result.
__device__ __forceinline__ void commit_result(const GenParams& P, uint32_t file, uint32_t bf_count, uint32_t last_count) {
    if (commit_chops(bf_count, last_count)) {
        bf_count--;
        last_count = kMaxElem;
    }
    P.out_info[file].bf_count = bf_count;
    P.out_info[file].last_count = last_count;
}

template <bool kRound>
__device__ __forceinline__ void commit_files(const GenParams& P, uint8_t* smem) {
    CommitSmem<kRound>& S = *reinterpret_cast<CommitSmem<kRound>*>(smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool loader = wid == kCmWarps;
    for (uint32_t i = tid; i < 4096; i += kCmThreads) S.tab[i] = 0xFFFFFFFFu;
    for (uint32_t i = tid; i < kCmWin; i += kCmThreads) S.match[i] = 0;
    uint32_t epoch = 0xFFFFFFu;  // counts down: a later pass has smaller keys
    for (uint32_t fi = blockIdx.x; fi < P.nfiles; fi += gridDim.x) {
        const uint32_t file = P.file_order[fi];
        if (kRound && P.commit_dirty && !P.commit_dirty[file]) continue;
        const GenFile Fd = P.files[file];
        if (Fd.nchunks == 0) continue;
        uint32_t* out = P.out_filters + (size_t)Fd.filter_base * 64;
        // the file's tiles are one contiguous range
        const GenChunk c0 = P.chunks[Fd.first_chunk];
        const GenChunk cl = P.chunks[Fd.first_chunk + Fd.nchunks - 1];
        const uint32_t t_first = c0.first_tile, t_end = cl.first_tile + cl.ntiles;
        const uint32_t chunk_end = Fd.first_chunk + Fd.nchunks;
        uint32_t chunk = Fd.first_chunk;
        uint32_t next_chunk_tile = (Fd.nchunks > 1) ? P.chunks[chunk + 1].first_tile : 0xFFFFFFFFu;
        uint32_t bf_count = 1, last_count = 0, bigfi = 0;
        // tiles [ts, t_end) commit now: a later index round restarts from the
        // last checkpoint at or before the first changed predicate (nothing
        // before it changed, so the state there is the one recorded)
        uint32_t ts = t_first;
        if (kRound && P.commit_dirty) {
            const uint32_t from = P.commit_from[file];
            const uint32_t tc = from == 0xFFFFFFFFu ? 0u : from / kTileCap / kCkptTiles * kCkptTiles;
            if (tc > t_first && tc < t_end) ts = tc;
            if (P.phase && tid == 0 && ts > t_first) atomicAdd(P.phase + kPhCkptRestarts, 1ull);
        }
        __syncthreads();  // the previous file is done with the shared state
        if (ts > t_first) {
            const uint32_t* ck = P.commit_ckpt + (size_t)(ts / kCkptTiles) * kCkptWords;
            for (uint32_t i = tid; i < 64; i += kCmThreads) {
                S.F[0][i] = ck[i];
                S.F[1][i] = 0;
            }
            const uint4* g4 = reinterpret_cast<const uint4*>(ck + 64);
            for (uint32_t i = tid; i < kBigBytes / 16; i += kCmThreads) reinterpret_cast<uint4*>(S.G)[i] = g4[i];
            bf_count = ck[64 + 4096];
            last_count = ck[64 + 4096 + 1];
            bigfi = ck[64 + 4096 + 2];
            // the chunk holding tile ts - 1, as the segment loop leaves it
            while (next_chunk_tile < ts) {
                chunk++;
                next_chunk_tile = chunk + 1 < chunk_end ? P.chunks[chunk + 1].first_tile : 0xFFFFFFFFu;
            }
        } else {
            for (uint32_t i = tid; i < 128; i += kCmThreads) S.F[0][i] = 0;
            for (uint32_t i = tid; i < kBigBytes / 16; i += kCmThreads)
                reinterpret_cast<uint4*>(S.G)[i] = make_uint4(0, 0, 0, 0);
        }
        if (kRound && P.commit_dirty && ts < t_end) {
            // clear the file's seen bits, ordinals [ts, t_end) * kTileCap;
            // inner words are the file's alone, edge words shared with neighbours
            const uint32_t o0 = ts * kTileCap, o1 = t_end * kTileCap - 1;
            for (uint32_t w = (o0 >> 5) + tid; w <= (o1 >> 5); w += kCmThreads) {
                const uint32_t lo = w == (o0 >> 5) ? (o0 & 31u) : 0u, hi = w == (o1 >> 5) ? (o1 & 31u) : 31u;
                const uint32_t m = (0xffffffffu >> (31u - hi)) & (0xffffffffu << lo);
                if (m == 0xffffffffu) P.index_seen[w] = 0;
                else atomicAnd(P.index_seen + w, ~m);
            }
        }
        __syncthreads();
        long long t_file = P.phase ? clock64() : 0, t_wait = 0;
        uint32_t n_pass = 0, n_ambig = 0;
        uint32_t cur = 0;            // F[cur] fills
        bool fresh = ts == t_first;  // F[cur] holds no bit
        bool flush = false;          // F[cur ^ 1] is complete: filter bf_count - 2 goes out
        uint32_t pos = 0, avail = 0; // window start, end of the staged features (positions in the file)
        // segments of tiles: a chunk (the big-filter counter restarts behind
        // it), in index rounds also cut at checkpoints
        uint32_t t_seg = ts;
        while (t_seg < t_end) {
            if (kRound && t_seg > ts && t_seg % kCkptTiles == 0) {
                // checkpoint of the state entering tile t_seg
                uint32_t* ck = P.commit_ckpt + (size_t)(t_seg / kCkptTiles) * kCkptWords;
                __syncthreads();  // the last pass's bits are applied
                for (uint32_t i = tid; i < 64; i += kCmThreads) ck[i] = S.F[cur][i];
                uint4* g4 = reinterpret_cast<uint4*>(ck + 64);
                for (uint32_t i = tid; i < kBigBytes / 16; i += kCmThreads) g4[i] = reinterpret_cast<const uint4*>(S.G)[i];
                if (tid == 0) {
                    ck[64 + 4096] = bf_count;
                    ck[64 + 4096 + 1] = last_count;
                    ck[64 + 4096 + 2] = bigfi;
                }
            }
            while (t_seg >= next_chunk_tile) {
                bigfi = 0;
                chunk++;
                next_chunk_tile = chunk + 1 < chunk_end ? P.chunks[chunk + 1].first_tile : 0xFFFFFFFFu;
            }
            uint32_t seg_end = min(next_chunk_tile, t_end);
            if (kRound) seg_end = min(seg_end, (t_seg / kCkptTiles + 1) * kCkptTiles);
            // the loading warp and the window's threads run the same number of
            // passes: both see what was published before barrier (1)
            if (loader) {
                // tiles [tn, seg_end) to come, their counts 32 at a time (lane
                // l: tile cb + l), e0 >= e1 >= e2 the staged ends after this
                // pass's copies, the last pass's, the one's before
                uint32_t tn = t_seg, cb = t_seg, cnt = 0, cnt_next = 0, e0 = pos, e1 = pos, e2 = pos, par = 0;
                if (cb + lane < seg_end) cnt = P.tile_out[cb + lane].count;
                if (cb + 32 + lane < seg_end) cnt_next = P.tile_out[cb + 32 + lane].count;
                while (true) {
                    // stage the next tiles that fit (positions below the last
                    // window's start are free), then publish the end of what
                    // has arrived: copies started two passes ago, or all of
                    // them when the next windows would run short
                    uint32_t started = 0;
                    while (tn < seg_end && started < kCmTiles) {
                        const uint32_t c = min(__shfl_sync(0xffffffffu, cnt, tn - cb), kTileCap);
                        if (e0 - pos + c > kCmRing) break;
                        const uint32_t* src = P.features + (size_t)tn * 5 * kTileCap;
                        for (uint32_t q = lane; q < c; q += 32) {
                            const uint32_t d = (e0 + q) & (kCmRing - 1);
                            cp_async16(&S.feat4[d], src + 4 * q);
                            cp_async4(&S.feat1[d], src + 4 * kTileCap + q);
                            if (kRound) S.ord[d] = tn * kTileCap + q;
                        }
                        e0 += c;
                        tn++;
                        started += c != 0;
                        if (tn - cb == 32) {
                            cb += 32;
                            cnt = cnt_next;
                            cnt_next = cb + 32 + lane < seg_end ? P.tile_out[cb + 32 + lane].count : 0;
                        }
                    }
                    cp_async_commit();
                    const long long w0 = P.phase ? clock64() : 0;
                    const bool all = e2 - pos < 3 * kCmWin;
                    if (all) cp_async_wait_all();
                    else cp_async_wait_2();
                    if (P.phase) t_wait += clock64() - w0;
                    const uint32_t got = all ? e0 : e2;
                    e2 = all ? e0 : e1;
                    e1 = e0;
                    const bool fin = tn == seg_end && got == e0;
                    __syncwarp();
                    if (lane == 0) {
                        S.avail[par] = got;
                        S.final_[par] = fin;
                    }
                    __syncthreads();  // (1)
                    pos = S.pos[par];
                    par ^= 1u;
                    if (fin) break;
                }
            }
            // window's threads: after a pass whose barrier (1) carried
            // final_, the rest of the segment runs without the loading warp
            bool final_ = false;
            uint32_t par = 0;
            while (!loader && (!final_ || pos != avail)) {
                if (epoch == 0) {  // once in 2^24 passes
                    commit_sync();
                    for (uint32_t i = tid; i < 4096; i += kCmWin) S.tab[i] = 0xFFFFFFFFu;
                    epoch = 0xFFFFFFu;
                    commit_sync();
                }
                epoch--;
                n_pass++;
                const uint32_t W = min((uint32_t)kCmWin, avail - pos);
                const bool have = tid < W;
                const uint32_t key = (epoch << 8) | tid;
                const uint32_t slot = (pos + tid) & (kCmRing - 1);
                uint32_t h[5] = {0, 0, 0, 0, 0};
                uint32_t ord = 0;
                bool ipred = true;
                if (have) {
                    const uint4 v = S.feat4[slot];
                    h[0] = v.x;
                    h[1] = v.y;
                    h[2] = v.z;
                    h[3] = v.w;
                    h[4] = S.feat1[slot];
#pragma unroll
                    for (int k = 0; k < 5; k++) atomicMin(&S.tab[h[k] & 0xFFFu], key);
                    if (kRound) {
                        ord = S.ord[slot];
                        ipred = (__ldg(P.index_pred + (ord >> 5)) >> (ord & 31u)) & 1u;
                    }
                }
                if (tid == 0) S.pos[par] = pos;
                uint32_t avail_next = avail;
                if (final_) {
                    commit_sync();  // (1)
                } else {
                    __syncthreads();  // (1)
                    avail_next = S.avail[par];
                    final_ = S.final_[par] != 0;
                    par ^= 1u;
                }
                if (flush) {
                    if (tid < 64) {
                        if (bf_count - 1 <= Fd.filter_cap) out[(size_t)(bf_count - 2) * 64 + tid] = S.F[cur ^ 1u][tid];
                        else if (tid == 0) atomicAdd(P.counters + 1, 1u);
                        S.F[cur ^ 1u][tid] = 0;
                    }
                    flush = false;
                }
                bool fnew = false, gate = false, cnt_def = false, amb = false;
                uint32_t gun = 0;  // big-filter bits unset before the window
                if (have) {
                    bool gnew = false;
#pragma unroll
                    for (int k = 0; k < 5; k++) {
                        const uint32_t i12 = h[k] & 0xFFFu, a = h[k] & kBfMask, b = h[k] & kBigMask;
                        const uint32_t t0 = S.tab[i12], t1 = S.tab[i12 ^ 0x800u];
                        const uint32_t fw = fresh ? 0u : S.F[cur][a >> 5] >> (a & 31), gw = S.G[b >> 5] >> (b & 31);
                        fnew |= t0 == key && t1 >= key && !(fw & 1u);
                        gnew |= t0 == key && !(gw & 1u);
                        gun |= (~gw & 1u) << k;
                    }
                    gate = fnew && ipred;
                    cnt_def = gate && gnew;
                    amb = gate && !gnew && gun;
                }
                {
                    const uint32_t mc = __ballot_sync(0xffffffffu, cnt_def), ma = __ballot_sync(0xffffffffu, amb);
                    if (lane == 0) {
                        S.counted[wid] = mc;
                        S.ambig[wid] = ma;
                    }
                }
                commit_sync();  // (2)
                uint32_t m[kCmWarps], am_[kCmWarps];
                auto read_flags = [&](const uint32_t* src, uint32_t (&v)[kCmWarps]) {
                    const uint4 x = *reinterpret_cast<const uint4*>(src);
                    const uint2 y = *reinterpret_cast<const uint2*>(src + 4);
                    v[0] = x.x;
                    v[1] = x.y;
                    v[2] = x.z;
                    v[3] = x.w;
                    v[4] = y.x;
                    v[5] = y.y;
                };
                read_flags(S.counted, m);
                read_flags(S.ambig, am_);
                if (am_[0] | am_[1] | am_[2] | am_[3] | am_[4] | am_[5]) {
                    // an ambiguous feature's value k is held by an earlier
                    // F-passing feature of the window?
#pragma unroll
                    for (uint32_t w = 0; w < kCmWarps; w++) {
                        for (uint32_t am = am_[w]; am; am &= am - 1u) {
                            const uint32_t j = 32 * w + (uint32_t)(__ffs(am) - 1);
                            n_ambig++;
                            if (wid > w) continue;  // later features only
                            uint32_t mm = 0;
                            if (gate && tid < j) {
                                const uint32_t js = (pos + j) & (kCmRing - 1);
                                const uint4 v4 = S.feat4[js];
                                const uint32_t v[5] = {v4.x, v4.y, v4.z, v4.w, S.feat1[js]};
#pragma unroll
                                for (int k = 0; k < 5; k++)
#pragma unroll
                                    for (int q = 0; q < 5; q++) mm |= (uint32_t)(((h[q] ^ v[k]) & kBigMask) == 0) << k;
                            }
                            mm = __reduce_or_sync(0xffffffffu, mm);
                            if (lane == 0 && mm) atomicOr(&S.match[j], mm);
                        }
                    }
                    commit_sync();
                    if (amb) {
                        cnt_def = (gun & ~S.match[tid]) != 0;
                        S.match[tid] = 0;
                    }
                    const uint32_t mc = __ballot_sync(0xffffffffu, cnt_def);
                    if (lane == 0) S.counted[wid] = mc;
                    commit_sync();
                    read_flags(S.counted, m);
                }
                // counted features before this one and in all
                uint32_t before = 0, total = 0;
#pragma unroll
                for (uint32_t w = 0; w < kCmWarps; w++) {
                    const uint32_t c = __popc(m[w]);
                    before += w < wid ? c : w == wid ? __popc(m[w] & lanemask_lt()) : 0u;
                    total += c;
                }
                const uint32_t need_s = (uint32_t)kMaxElem - last_count, need_b = (uint32_t)kBigElem - bigfi;
                const uint32_t need = min(need_s, need_b);
                const bool roll = total >= need;  // the need-th counted feature ends the pass
                if (roll && cnt_def && before + 1 == need) S.end = tid + 1;
                commit_sync();  // (3)
                const uint32_t n = roll ? S.end : W;
                const bool roll_small = roll && need == need_s, roll_big = roll && need == need_b;
                if (have && before < need) {
#pragma unroll
                    for (int k = 0; k < 5; k++) {
                        const uint32_t a = h[k] & kBfMask, b = h[k] & kBigMask;
                        atomicOr(&S.F[cur][a >> 5], 1u << (a & 31));
                        if (gate && !roll_big) atomicOr(&S.G[b >> 5], 1u << (b & 31));
                    }
                    // the inserted features of this pass
                    if (kRound && fnew) atomicOr(P.index_seen + (ord >> 5), 1u << (ord & 31u));
                }
                if (roll_big)
                    for (uint32_t i = tid; i < kBigBytes / 16; i += kCmWin)
                        reinterpret_cast<uint4*>(S.G)[i] = make_uint4(0, 0, 0, 0);
                fresh = roll_small || (fresh && n == 0);
                last_count += min(total, need);
                bigfi += min(total, need);
                if (roll_small) {
                    bf_count++;
                    last_count = 0;
                    cur ^= 1u;
                    flush = true;
                }
                if (roll_big) bigfi = 0;
                pos += n;
                avail = avail_next;
            }
            if (tid == 0) S.seg_pos = pos;
            __syncthreads();  // the segment's last bits are applied
            pos = avail = S.seg_pos;
            t_seg = seg_end;
        }
        __syncthreads();
        if (flush && tid < 64) {
            if (bf_count - 1 <= Fd.filter_cap) out[(size_t)(bf_count - 2) * 64 + tid] = S.F[cur ^ 1u][tid];
            else if (tid == 0) atomicAdd(P.counters + 1, 1u);
        }
        // emit the current (last) filter, if it stays (out may be the caller's
        // buffer, whose slots behind the result are not written)
        if (bf_count <= Fd.filter_cap) {
            if (tid < 64 && !commit_chops(bf_count, last_count)) out[(size_t)(bf_count - 1) * 64 + tid] = S.F[cur][tid];
        } else if (tid == 0) {
            atomicAdd(P.counters + 1, 1u);
        }
        if (tid == 0) {
            commit_result(P, file, bf_count, last_count);
            if (P.phase) {
                const long long busy = clock64() - t_file;
                atomicAdd(P.phase + kPhCommitBusy, (unsigned long long)busy);
                atomicAdd(P.phase + kPhCommitGroups, (unsigned long long)n_pass);
                atomicAdd(P.phase + kPhCommitLoops, (unsigned long long)n_ambig);
                atomicMax(P.phase + kPhCommitMaxFile, (unsigned long long)busy);
            }
        }
        if (P.phase && loader && lane == 0) atomicAdd(P.phase + kPhCommitWait, (unsigned long long)t_wait);
    }
}

__global__ void __launch_bounds__(kCmThreads) k_stream_commit(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    commit_files<false>(P, smem);
}

__global__ void __launch_bounds__(kCmThreads) k_stream_commit_round(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    commit_files<true>(P, smem);
}

// The sequential commit of an index build: one warp, files in input order,
// one feature at a time, lane k (< 5) holding its k-th hash word.  Setting a
// bit and learning whether it was new is one atomic each on the filter, the
// index and the big filter.
__global__ void __launch_bounds__(32) k_stream_commit_index(GenParams P) {
    __shared__ uint32_t F[64], G[kBigBytes / 4];
    __shared__ __align__(16) uint32_t feat[2][5 * kTileCap];  // double-buffered features of a tile
    const uint32_t lane = threadIdx.x;
    const uint32_t k = min(lane, 4u);
    auto stage = [&](uint32_t buf, uint32_t t, uint32_t nf) {
        const uint32_t* src = P.features + (size_t)t * 5 * kTileCap;
        for (uint32_t q = lane; q < nf; q += 32) cp_async16(&feat[buf][4 * q], src + 4 * q);
        for (uint32_t q = lane; q < (nf + 3) / 4; q += 32)
            cp_async16(&feat[buf][4 * (kTileCap + q)], src + 4 * (kTileCap + q));
        cp_async_commit();
    };
    for (uint32_t fi = 0; fi < P.nfiles; fi++) {
        const uint32_t file = P.file_order[fi];
        const GenFile Fd = P.files[file];
        if (Fd.nchunks == 0) continue;
        uint32_t* out = P.out_filters + (size_t)Fd.filter_base * 64;
        for (uint32_t i = lane; i < 64; i += 32) F[i] = 0;
        for (uint32_t i = lane; i < kBigBytes / 4; i += 32) G[i] = 0;
        __syncwarp();
        uint32_t bf_count = 1, last_count = 0;
        auto emit = [&]() {
            __syncwarp();
            const bool fits = bf_count <= Fd.filter_cap;
            for (uint32_t i = lane; i < 64; i += 32) {
                if (fits) out[(size_t)(bf_count - 1) * 64 + i] = F[i];
                F[i] = 0;
            }
            if (!fits && lane == 0) atomicAdd(P.counters + 1, 1u);
            __syncwarp();
        };
        for (uint32_t c = Fd.first_chunk; c < Fd.first_chunk + Fd.nchunks; c++) {
            const uint32_t ta = P.chunks[c].first_tile, tb = ta + P.chunks[c].ntiles;
            uint32_t bigfi = 0;  // local to the chunk
            uint32_t nf = ta < tb ? P.tile_out[ta].count : 0;
            if (ta < tb) stage(0, ta, nf);
            for (uint32_t t = ta; t < tb; t++) {
                const uint32_t cur = (t - ta) & 1u;
                cp_async_wait_all();
                __syncwarp();
                const uint32_t nf_next = t + 1 < tb ? P.tile_out[t + 1].count : 0;
                if (t + 1 < tb) stage(cur ^ 1u, t + 1, nf_next);
                for (uint32_t g = 0; g < nf; g++) {
                    const uint32_t h = feat[cur][feat_word(g, k)];
                    const uint32_t a = h & kBfMask, b = h & kBigMask, pos = h & P.index_mask;
                    bool nw = false;
                    if (lane < 5) nw = !((atomicOr(&F[a >> 5], 1u << (a & 31)) >> (a & 31)) & 1u);
                    if (!__any_sync(0xffffffffu, nw)) continue;
                    nw = false;
                    if (lane < 5) nw = !((atomicOr(P.index_bits + (pos >> 5), 1u << (pos & 31)) >> (pos & 31)) & 1u);
                    if (!__any_sync(0xffffffffu, nw)) continue;
                    if (lane == 0) atomicAdd(P.index_new, 1ull);
                    nw = false;
                    if (lane < 5) nw = !((atomicOr(&G[b >> 5], 1u << (b & 31)) >> (b & 31)) & 1u);
                    if (!__any_sync(0xffffffffu, nw)) continue;
                    last_count++;
                    bigfi++;
                    if (last_count == (uint32_t)kMaxElem) {
                        emit();
                        bf_count++;
                        last_count = 0;
                    }
                    if (bigfi == (uint32_t)kBigElem) {
                        __syncwarp();
                        for (uint32_t i = lane; i < kBigBytes / 4; i += 32) G[i] = 0;
                        __syncwarp();
                        bigfi = 0;
                    }
                }
                nf = nf_next;
            }
        }
        emit();
        if (lane == 0) commit_result(P, file, bf_count, last_count);
        __syncwarp();
    }
}

// Features of a stream launch recorded in a seen bitmap (ordinal = tile *
// kTileCap + feature): the first setter of each of their index bits, then
// (once the rounds agree) the bits and the count of first setters.
// k_stream_index_pred: for every feature, whether it would own the first
// setting of one of its bits (one bit per ordinal, a warp per word).
__global__ void k_stream_index_pred(const uint32_t* __restrict__ feats, const TileOut* __restrict__ tile_out,
                                    uint32_t ntiles, const uint32_t* __restrict__ first, uint32_t mask,
                                    uint32_t* __restrict__ pred) {
    const uint64_t n = (uint64_t)ntiles * kTileCap, npad = (n + 31) & ~31ull;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npad; i += (uint64_t)gridDim.x * blockDim.x) {
        bool p = false;
        if (i < n) {
            const uint32_t t = (uint32_t)(i / kTileCap), g = (uint32_t)(i - (uint64_t)t * kTileCap);
            if (g < tile_out[t].count) {
                const uint32_t* w = feats + (size_t)t * 5 * kTileCap;
#pragma unroll
                for (int k = 0; k < 5; k++) p |= __ldg(first + (w[feat_word(g, k)] & mask)) >= (uint32_t)i + 1u;
            }
        }
        const uint32_t word = __ballot_sync(0xffffffffu, p);
        if ((threadIdx.x & 31) == 0) pred[i >> 5] = word;
    }
}

__global__ void k_stream_index_first(const uint32_t* __restrict__ feats, const TileOut* __restrict__ tile_out,
                                     uint32_t ntiles, const uint32_t* __restrict__ seen, uint32_t mask,
                                     uint32_t* __restrict__ first) {
    const uint64_t n = (uint64_t)ntiles * kTileCap;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!((seen[i >> 5] >> (i & 31)) & 1u)) continue;
        const uint32_t t = (uint32_t)(i / kTileCap), g = (uint32_t)(i - (uint64_t)t * kTileCap);
        if (g >= tile_out[t].count) continue;
        const uint32_t* w = feats + (size_t)t * 5 * kTileCap;
#pragma unroll
        for (int k = 0; k < 5; k++) atomicMin(first + (w[feat_word(g, k)] & mask), (uint32_t)i + 1u);
    }
}

__global__ void k_stream_index_mark(const uint32_t* __restrict__ feats, const TileOut* __restrict__ tile_out,
                                    uint32_t ntiles, const uint32_t* __restrict__ seen, uint32_t mask,
                                    const uint32_t* __restrict__ first, uint32_t* __restrict__ bits,
                                    unsigned long long* __restrict__ count) {
    const uint64_t n = (uint64_t)ntiles * kTileCap;
    uint32_t mine = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!((seen[i >> 5] >> (i & 31)) & 1u)) continue;
        const uint32_t t = (uint32_t)(i / kTileCap), g = (uint32_t)(i - (uint64_t)t * kTileCap);
        if (g >= tile_out[t].count) continue;
        const uint32_t* w = feats + (size_t)t * 5 * kTileCap;
        bool fresh = false;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const uint32_t pos = w[feat_word(g, k)] & mask;
            fresh |= first[pos] == (uint32_t)i + 1u;
            atomicOr(bits + (pos >> 5), 1u << (pos & 31));
        }
        mine += fresh;
    }
    for (int d = 16; d > 0; d >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, d);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(count, (unsigned long long)mine);
}

__global__ void k_pred_dirty(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint64_t nwords,
                             const GenTile* __restrict__ tiles, const GenChunk* __restrict__ chunks, uint32_t ntiles,
                             uint8_t* __restrict__ dirty, uint32_t* __restrict__ from,
                             unsigned int* __restrict__ ndirty) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nwords;
         w += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t x = a[w] ^ b[w];
        while (x) {
            const uint64_t ord = w * 32 + (uint32_t)(__ffs(x) - 1);
            x &= x - 1u;
            const uint64_t t = ord / kTileCap;
            if (t >= ntiles) continue;
            const uint32_t f = chunks[tiles[t].chunk].file;
            atomicMin(from + f, (uint32_t)ord);
            if (!dirty[f]) {
                dirty[f] = 1;
                atomicAdd(ndirty, 1u);
            }
        }
    }
}

// ------------------------------------------------------ linked commit
// The ordered filter fill again, for files long enough that its chain of
// passes is what a batch waits for.  Whether a feature sets a new bit in the
// filter F does not need F: F holds exactly the bits of the features since
// the filter's start fs (a feature that fails either test sets no bit that is
// new), so feature i passes iff one of its five bits was last held before fs,
// that is iff min over its words of (place of the last earlier holder of the
// same 11-bit index) is before fs.  That minimum depends on the features
// alone and is computed for all of them at once:
//  k_feat_scan   the place of every tile's features in its file;
//  k_feat_pack   the features packed per file: five 17-bit big-filter indices
//                (the filter's are their low 11 bits);
//  k_feat_last   per block of kLkBlock features, the last holder of each
//                filter bit in the block;
//  k_feat_carry  per block, the last holder before it;
//  k_feat_links  the minimum (0: a bit that no earlier feature holds, else
//                place + 1), and for each word whether a feature of the last
//                kLkNear may hold the same big-filter index.
// k_stream_chain then walks a file's features in windows as k_stream_commit
// does, with one compare for F; the big filter G is kept, and its bits that
// are unset before a window and near no other holder are new.  It leaves the
// ends of the filters; k_stream_emit fills them.
//
// What bounds it: the chain, ~200 instructions a pass that wait for one
// another, three barriers, the random reads and stores of G (a byte per bit,
// so that its bits are set without atomics).  One 200 MiB file: 16,693 passes
// of 1,034 cycles, 8.35 ms, and 0.43 ms for links and filters; k_stream_commit
// takes 15.2 ms.  On the way: G as bits set by atomics, one table of 13 bits
// for the near flags (0.44 ambiguous features a pass, 1,100 cycles each; with
// two tables 0.02): 1,745 cycles; the next window's features read only after
// barrier (1): 1,135.
constexpr uint32_t kLkNear = 192 + 32;  // a window, and what a stale place in the table may be off
static_assert(kLkNear % 32 == 0 && kLkBlock % 32 == 0 && kLkNear <= kLkBlock && kLkBlock + kLkNear < 65535, "places in whole groups, in 16 bits");

__global__ void __launch_bounds__(1024) k_feat_scan(GenParams P) {
    __shared__ uint32_t warp_sums[32];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (uint32_t f = blockIdx.x; f < P.nfiles; f += gridDim.x) {
        const GenFile Fd = P.files[f];
        if (Fd.nchunks == 0) {
            if (threadIdx.x == 0) P.file_total[f] = 0;
            continue;
        }
        const GenChunk cl = P.chunks[Fd.first_chunk + Fd.nchunks - 1];
        const uint32_t t0 = P.chunks[Fd.first_chunk].first_tile, t1 = cl.first_tile + cl.ntiles;
        uint32_t run = t0 * kTileCap;
        for (uint32_t b = t0; b < t1; b += 4096) {
            uint32_t c[4], sum = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t t = b + 4 * threadIdx.x + k;
                c[k] = t < t1 ? min(P.tile_out[t].count, kTileCap) : 0u;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) sum += c[k];
            uint32_t incl = sum;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= (uint32_t)d) incl += y;
            }
            __syncthreads();  // the last stretch's sums are read
            if (lane == 31) warp_sums[wid] = incl;
            __syncthreads();
            uint32_t ws = warp_sums[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, ws, d);
                if (lane >= (uint32_t)d) ws += y;
            }
            uint32_t at = run + incl - sum + (wid ? __shfl_sync(0xffffffffu, ws, wid - 1) : 0u);
            run += __shfl_sync(0xffffffffu, ws, 31);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t t = b + 4 * threadIdx.x + k;
                if (t < t1) P.tile_base[t] = at;
                at += c[k];
            }
        }
        if (threadIdx.x == 0) P.file_total[f] = run - t0 * kTileCap;
    }
}

// links entry: x = index 0 | low 15 bits of index 3 << 17, y = index 1 | low
// 15 bits of index 4 << 17, z = index 2 | high bits of 3 << 17 | of 4 << 19 |
// near flags << 21, w = the minimum
__device__ __forceinline__ void link_unpack(const uint4& v, uint32_t (&b)[5]) {
    b[0] = v.x & kBigMask;
    b[1] = v.y & kBigMask;
    b[2] = v.z & kBigMask;
    b[3] = (v.x >> 17) | ((v.z >> 2) & 0x18000u);
    b[4] = (v.y >> 17) | ((v.z >> 4) & 0x18000u);
}

__global__ void __launch_bounds__(256) k_feat_pack(GenParams P) {
    const uint32_t lane = threadIdx.x & 31, w0 = blockIdx.x * 8 + (threadIdx.x >> 5), nw = gridDim.x * 8;
    for (uint32_t t = w0; t < P.ntiles; t += nw) {
        const uint32_t c = min(P.tile_out[t].count, kTileCap);
        const uint32_t* src = P.features + (size_t)t * 5 * kTileCap;
        uint4* dst = P.links + P.tile_base[t];
        for (uint32_t q = lane; q < c; q += 32) {
            const uint4 h = __ldg(reinterpret_cast<const uint4*>(src) + q);
            const uint32_t b3 = h.w & kBigMask, b4 = __ldg(src + 4 * kTileCap + q) & kBigMask;
            dst[q] = make_uint4((h.x & kBigMask) | (b3 << 17), (h.y & kBigMask) | (b4 << 17),
                                (h.z & kBigMask) | ((b3 >> 15) << 17) | ((b4 >> 15) << 19), 0u);
        }
    }
}

// first place of a file's features in links
__device__ __forceinline__ uint32_t link_base(const GenParams& P, const GenFile& Fd) {
    return P.chunks[Fd.first_chunk].first_tile * kTileCap;
}

__global__ void __launch_bounds__(32) k_feat_last(GenParams P) {
    __shared__ uint32_t last[kLkTab];
    const uint32_t lane = threadIdx.x;
    for (uint32_t f = blockIdx.y; f < P.nfiles; f += gridDim.y) {
        const uint32_t total = P.file_total[f];
        if (total <= kLkBlock) continue;
        const uint4* v = P.links + link_base(P, P.files[f]);
        const uint32_t nblk = (total + kLkBlock - 1) / kLkBlock;
        for (uint32_t b = blockIdx.x; b + 1 < nblk; b += gridDim.x) {  // (nothing follows the last block)
            for (uint32_t i = lane; i < kLkTab; i += 32) last[i] = 0;
            __syncwarp();
#pragma unroll 4
            for (uint32_t q = lane; q < kLkBlock; q += 32) {
                const uint32_t o = b * kLkBlock + q;
                uint32_t x[5];
                link_unpack(v[o], x);
#pragma unroll
                for (int k = 0; k < 5; k++) atomicMax(&last[x[k] & kBfMask], o + 1);
            }
            __syncwarp();
            uint32_t* row = P.last_tab + ((size_t)P.link_first[f] + b) * kLkTab;
            for (uint32_t i = lane; i < kLkTab; i += 32) row[i] = last[i];
            __syncwarp();
        }
    }
}

// Rows of a file: last holder in the block -> last holder before the block.
__global__ void __launch_bounds__(128) k_feat_carry(GenParams P) {
    const uint32_t col = blockIdx.x * 128 + threadIdx.x;
    for (uint32_t f = blockIdx.y; f < P.nfiles; f += gridDim.y) {
        const uint32_t total = P.file_total[f];
        if (total <= kLkBlock) continue;
        const uint32_t nblk = (total + kLkBlock - 1) / kLkBlock;
        uint32_t* c = P.last_tab + (size_t)P.link_first[f] * kLkTab + col;
        uint32_t run = 0;
        for (uint32_t b = 0; b < nblk; b += 16) {
            uint32_t x[16];
#pragma unroll
            for (uint32_t k = 0; k < 16; k++) x[k] = b + k + 1 < nblk ? c[(size_t)(b + k) * kLkTab] : 0u;
#pragma unroll
            for (uint32_t k = 0; k < 16; k++) {
                if (b + k < nblk) c[(size_t)(b + k) * kLkTab] = run;
                run = max(run, x[k]);
            }
        }
    }
}

struct LinkSmem {
    uint32_t last[kLkTab];   // place + 1 of the last holder of each filter bit
    uint32_t own[kLkTab];    // lanes of the current 32 features that hold it
    uint32_t idx[32][5];     // their big-filter indices
    // place (from the first one looked at) + 1 of a late holder of an index's
    // low and of its high 13 bits: an index held late is late in both (chance
    // matches in both are one in 50, in one table one in 7)
    uint16_t near_[2][8192];
};
__global__ void __launch_bounds__(32) k_feat_links(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    LinkSmem& S = *reinterpret_cast<LinkSmem*>(smem);
    const uint32_t lane = threadIdx.x;
    for (uint32_t i = lane; i < kLkTab; i += 32) S.own[i] = 0;
    for (uint32_t f = blockIdx.y; f < P.nfiles; f += gridDim.y) {
        const uint32_t total = P.file_total[f];
        if (total == 0) continue;
        uint4* v = P.links + link_base(P, P.files[f]);
        const uint32_t nblk = (total + kLkBlock - 1) / kLkBlock;
        for (uint32_t b = blockIdx.x; b < nblk; b += gridDim.x) {
            __syncwarp();
            const uint32_t* row = P.last_tab + ((size_t)P.link_first[f] + b) * kLkTab;
            for (uint32_t i = lane; i < kLkTab; i += 32) S.last[i] = b ? __ldg(row + i) : 0u;
            uint4* n4 = reinterpret_cast<uint4*>(S.near_);
            for (uint32_t i = lane; i < sizeof S.near_ / 16; i += 32) n4[i] = make_uint4(0, 0, 0, 0);
            const uint32_t o0 = b * kLkBlock, o1 = min(total, o0 + kLkBlock), h0 = b ? o0 - kLkNear : 0u;
            __syncwarp();
            // the features before the block that a window may still hold
            // (other blocks' warps write these entries' flags meanwhile; the
            // indices stay)
            for (uint32_t o = h0 + lane; o < o0; o += 32) {  // whole groups of 32
                uint32_t x[5];
                link_unpack(v[o], x);
#pragma unroll
                for (int k = 0; k < 5; k++) S.near_[0][x[k] & 8191u] = S.near_[1][x[k] >> 4] = (uint16_t)(o - h0 + 1);
                __syncwarp();
            }
            __syncwarp();
            uint4 cur = o0 + lane < o1 ? v[o0 + lane] : make_uint4(0, 0, 0, 0);
            for (uint32_t g = o0; g < o1; g += 32) {
                const uint32_t o = g + lane;
                const bool have = o < o1;
                const uint4 nxt = o + 32 < o1 ? v[o + 32] : make_uint4(0, 0, 0, 0);
                uint32_t x[5], held[5], own[5], nr[5], nh[5];
                link_unpack(cur, x);
                const uint32_t here = o - h0 + 1;
#pragma unroll
                for (int k = 0; k < 5; k++) {
                    held[k] = S.last[x[k] & kBfMask];
                    nr[k] = S.near_[0][x[k] & 8191u];
                    nh[k] = S.near_[1][x[k] >> 4];
                    if (have) atomicOr(&S.own[x[k] & kBfMask], 1u << lane);
                    S.idx[lane][k] = x[k];
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 5; k++) own[k] = S.own[x[k] & kBfMask];
                __syncwarp();
                if (have) {
                    uint32_t least = 0xFFFFFFFFu, flags = 0;
#pragma unroll
                    for (int k = 0; k < 5; k++) {
                        const uint32_t lower = own[k] & lanemask_lt();
                        least = min(least, lower ? g + 32 - __clz(lower) : held[k]);
                        const bool late = nr[k] != 0 && nh[k] != 0 && here - min(nr[k], nh[k]) < kLkNear;
                        bool same = late;
                        for (uint32_t l = lower; l && !same; l &= l - 1u) {  // earlier ones of these 32, word by word
                            const uint32_t* e = S.idx[31 - __clz(l & (0u - l))];
                            same = e[0] == x[k] || e[1] == x[k] || e[2] == x[k] || e[3] == x[k] || e[4] == x[k];
                        }
                        flags |= (uint32_t)same << k;
                        if ((own[k] >> lane) == 1u) S.last[x[k] & kBfMask] = o + 1;
                        S.own[x[k] & kBfMask] = 0;
                        S.near_[0][x[k] & 8191u] = S.near_[1][x[k] >> 4] = (uint16_t)here;
                    }
                    reinterpret_cast<uint2*>(v + o)[1] = make_uint2((cur.z & 0x1FFFFFu) | (flags << 21), least);
                }
                __syncwarp();
                cur = nxt;
            }
        }
    }
}

constexpr uint32_t kChRing = 1024;
struct ChainSmem {
    uint4 ring[kChRing];                  // links staged ahead
    alignas(16) uint8_t G[kBigMask + 1];  // big filter, a byte per bit: set by plain stores
    uint32_t match[kCmWin];               // slow path: big-filter values held by an earlier feature
    alignas(8) uint8_t counted[8];        // features counted per warp
    uint32_t ambig[8];                    // slow path, per warp
    uint32_t end;                         // features the pass consumes, when F or G rolls over
};
static_assert(offsetof(ChainSmem, G) % 16 == 0 && offsetof(ChainSmem, counted) % 8 == 0, "read as 16- and 8-byte words");

__global__ void __launch_bounds__(kCmWin) k_stream_chain(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    ChainSmem& S = *reinterpret_cast<ChainSmem*>(smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    S.match[tid] = 0;
    // ones in the bytes of the warps before this one
    const uint32_t below_x = wid >= 4 ? 0x01010101u : 0x01010101u & ((1u << (8 * wid)) - 1u);
    const uint32_t below_y = wid == 5 ? 1u : 0u;
    for (uint32_t fi = blockIdx.x; fi < P.nfiles; fi += gridDim.x) {
        const uint32_t file = P.file_order[fi];
        const GenFile Fd = P.files[file];
        if (Fd.nchunks == 0) continue;
        const GenChunk cl = P.chunks[Fd.first_chunk + Fd.nchunks - 1];
        const uint32_t t_end = cl.first_tile + cl.ntiles, base = link_base(P, Fd), total = P.file_total[file];
        const uint4* v = P.links + base;
        uint32_t* ends = P.ends + Fd.filter_base;
        // a chunk's first feature; the big filter's counter restarts there
        uint32_t chunk = 0;
        const auto chunk_start = [&](uint32_t k) {
            if (k >= Fd.nchunks) return total;
            const uint32_t t = P.chunks[Fd.first_chunk + k].first_tile;
            return t < t_end ? P.tile_base[t] - base : total;
        };
        uint32_t seg_end = chunk_start(1);
        uint32_t bf_count = 1, last_count = 0, bigfi = 0, fs = 0, pos = 0;
        uint32_t e0 = 0, e1 = 0, e2 = 0, e3 = 0;  // ends of the copies started up to this pass, the ones before
        uint32_t n_pass = 0, n_ambig = 0;
        const long long t_file = P.phase ? clock64() : 0;
        // this thread's feature of the window: five indices, near flags, last holder
        uint32_t h[5] = {0, 0, 0, 0, 0}, near_ = 0, held = 0;
        bool loaded = false;
        __syncthreads();  // the previous file is done with the shared state
        for (uint32_t i = tid; i < sizeof S.G / 16; i += kCmWin) reinterpret_cast<uint4*>(S.G)[i] = make_uint4(0, 0, 0, 0);
        for (; e0 < min(total, 4u * kCmWin); e0 += kCmWin)
            if (e0 + tid < total) cp_async16(&S.ring[e0 + tid], v + e0 + tid);
        e0 = min(e0, total);
        while (pos < total) {
            while (pos == seg_end) {
                bigfi = 0;
                seg_end = chunk_start(++chunk + 1);
            }
            n_pass++;
            // stage on: places below this window's start are free (reads that
            // may still be under way are of this window's features)
            e3 = e2;
            e2 = e1;
            e1 = e0;
            const uint32_t room = min(min((uint32_t)kCmWin, total - e0), pos + kChRing - e0);
            if (tid < room) cp_async16(&S.ring[(e0 + tid) & (kChRing - 1)], v + e0 + tid);
            e0 += room;
            cp_async_commit();
            uint32_t avail = e3;
            if (e3 - pos < min((uint32_t)kCmWin, total - pos)) {
                cp_async_wait_all();
                avail = e3 = e2 = e1 = e0;
            } else {
                asm volatile("cp.async.wait_group 3;\n" ::);
            }
            __syncthreads();  // (1) copies and the last pass's big-filter bits are there
            const uint32_t W = min(min((uint32_t)kCmWin, avail - pos), seg_end - pos);
            const bool have = tid < W;
            if (have && !loaded) {
                const uint4 x = S.ring[(pos + tid) & (kChRing - 1)];
                link_unpack(x, h);
                near_ = x.z >> 21;
                held = x.w;
            }
            const bool gate = have && held <= fs;
            // a big-filter bit that is unset (0) before the window, and one
            // that is unset and near no other holder
            uint32_t g[5], un = 1, sure = 1;
#pragma unroll
            for (int k = 0; k < 5; k++) g[k] = S.G[h[k]];
#pragma unroll
            for (int k = 0; k < 5; k++) {
                un = min(un, g[k]);
                sure = min(sure, g[k] | (near_ & (1u << k)));
            }
            bool cnt_def = gate && sure == 0;
            const bool amb = gate && un == 0 && sure != 0;
            uint32_t mc = __ballot_sync(0xffffffffu, cnt_def);
            if (lane == 0) S.counted[wid] = (uint8_t)__popc(mc);
            if (__syncthreads_or(amb)) {  // (2)
                // an ambiguous feature's value k is held by an earlier
                // F-passing feature of the window?
                const uint32_t ma = __ballot_sync(0xffffffffu, amb);
                if (lane == 0) S.ambig[wid] = ma;
                __syncthreads();
                for (uint32_t w = 0; w < (uint32_t)kCmWarps; w++) {
                    for (uint32_t am = S.ambig[w]; am; am &= am - 1u) {
                        const uint32_t j = 32 * w + (uint32_t)(__ffs(am) - 1);
                        n_ambig++;
                        if (wid > w) continue;  // later features only
                        uint32_t mm = 0;
                        if (gate && tid < j) {
                            uint32_t x[5];
                            link_unpack(S.ring[(pos + j) & (kChRing - 1)], x);
#pragma unroll
                            for (int k = 0; k < 5; k++)
#pragma unroll
                                for (int q = 0; q < 5; q++) mm |= (uint32_t)(h[q] == x[k]) << k;
                        }
                        mm = __reduce_or_sync(0xffffffffu, mm);
                        if (lane == 0 && mm) atomicOr(&S.match[j], mm);
                    }
                }
                __syncthreads();
                if (amb) {
                    const uint32_t mm = S.match[tid];
#pragma unroll
                    for (int k = 0; k < 5; k++) cnt_def |= g[k] == 0 && !((mm >> k) & 1u);
                    S.match[tid] = 0;
                }
                mc = __ballot_sync(0xffffffffu, cnt_def);
                if (lane == 0) S.counted[wid] = (uint8_t)__popc(mc);
                __syncthreads();
            }
            // counted features before this one and in all: byte sums
            const uint2 cw = *reinterpret_cast<const uint2*>(S.counted);
            const uint32_t all = __dp4a(cw.x, 0x01010101u, __dp4a(cw.y, 0x00000101u, 0u));
            const uint32_t before = __dp4a(cw.x, below_x, __dp4a(cw.y, below_y, (uint32_t)__popc(mc & lanemask_lt())));
            const uint32_t need_s = (uint32_t)kMaxElem - last_count, need_b = (uint32_t)kBigElem - bigfi;
            const uint32_t need = min(need_s, need_b);
            const bool roll = all >= need;  // the need-th counted feature ends the pass
            if (roll && cnt_def && before + 1 == need) S.end = tid + 1;
            __syncthreads();  // (3)
            const uint32_t n = roll ? S.end : W;
            const bool roll_small = roll && need == need_s, roll_big = roll && need == need_b;
            // the next window's feature is read while this one's bits are set
            const uint32_t next = pos + n + tid;
            loaded = next < avail;
            uint4 x = make_uint4(0, 0, 0, 0);
            if (loaded) x = S.ring[next & (kChRing - 1)];
            if (gate && tid < n && !roll_big) {
#pragma unroll
                for (int k = 0; k < 5; k++) S.G[h[k]] = 1;
            }
            if (roll_big)
                for (uint32_t i = tid; i < sizeof S.G / 16; i += kCmWin)
                    reinterpret_cast<uint4*>(S.G)[i] = make_uint4(0, 0, 0, 0);
            link_unpack(x, h);
            near_ = x.z >> 21;
            held = x.w;
            last_count += min(all, need);
            bigfi += min(all, need);
            pos += n;
            if (roll_small) {
                if (tid == 0) {
                    if (bf_count <= Fd.filter_cap) ends[bf_count - 1] = pos;
                    else atomicAdd(P.counters + 1, 1u);
                }
                bf_count++;
                last_count = 0;
                fs = pos;
            }
            if (roll_big) bigfi = 0;
        }
        cp_async_wait_all();
        if (tid == 0) {
            if (bf_count <= Fd.filter_cap) ends[bf_count - 1] = total;
            else atomicAdd(P.counters + 1, 1u);
            commit_result(P, file, bf_count, last_count);
            if (P.phase) {
                const long long busy = clock64() - t_file;
                atomicAdd(P.phase + kPhCommitBusy, (unsigned long long)busy);
                atomicAdd(P.phase + kPhCommitGroups, (unsigned long long)n_pass);
                atomicAdd(P.phase + kPhCommitLoops, (unsigned long long)n_ambig);
                atomicMax(P.phase + kPhCommitMaxFile, (unsigned long long)busy);
            }
        }
    }
}

// A warp per filter: the bits of its features, written to the file's output
// slots (dst_off; null: a batch of one file, from slot 0).
__global__ void __launch_bounds__(256) k_stream_emit(GenParams P, const uint64_t* __restrict__ dst_off,
                                                     uint32_t* __restrict__ dst, uint64_t dst_cap) {
    __shared__ uint32_t F[8][64];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (uint32_t f = blockIdx.y; f < P.nfiles; f += gridDim.y) {
        const GenFile Fd = P.files[f];
        if (Fd.nchunks == 0) continue;
        const uint32_t nf = P.out_info[f].bf_count;
        const uint4* v = P.links + link_base(P, Fd);
        const uint32_t* ends = P.ends + Fd.filter_base;
        const uint64_t slot = dst_off ? dst_off[f] : 0;
        for (uint32_t k = blockIdx.x * 8 + wid; k < nf && k < Fd.filter_cap && slot + k < dst_cap; k += gridDim.x * 8) {
            F[wid][lane] = 0;
            F[wid][lane + 32] = 0;
            __syncwarp();
            const uint32_t b = k ? ends[k - 1] : 0u, e = ends[k];
            for (uint32_t o = b + lane; o < e; o += 32) {
                uint32_t x[5];
                link_unpack(__ldg(v + o), x);
#pragma unroll
                for (int q = 0; q < 5; q++) atomicOr(&F[wid][(x[q] & kBfMask) >> 5], 1u << (x[q] & 31));
            }
            __syncwarp();
            reinterpret_cast<uint2*>(dst + (slot + k) * 64)[lane] = reinterpret_cast<const uint2*>(F[wid])[lane];
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------ block mode
// kPre: the block's ranks come from k_stream_ranks (64-byte windows do not
// know about blocks; only a block's last 64 positions have rank 0), and the
// block is walked as one or two tiles of kBlkL steps, the second entered
// with the first one's exit state.  55 KB of shared memory then hold four
// blocks on an SM.  Without (block sizes that are no multiple of 8, few blocks,
// or no room for the ranks) the whole block is ranked and walked at once, two
// blocks to an SM.  A 1 GiB image at 16 KiB blocks: ranks 1.6 ms and this
// kernel 4.45 ms; when the ranks left the tile the two went from 10.9 to 8.2 ms,
// most of it the set-up of 96 threads' windows for 170 positions each.
constexpr uint32_t kBlkL = 8192;
static_assert(kBlkL / kSegs == 64 && kBlkL % 64 == 0, "a segment is one block of the full-rescan table");

__device__ inline TileGeom block_geom(uint32_t n) {
    TileGeom g;
    g.n = n;
    g.t0 = 0;
    g.S0 = 0;
    g.Q0 = 0;
    g.SE = n - kWin;
    g.L = n - kWin;
    g.RE = n;
    g.BE = n;
    return g;
}

// tile h of a block with precomputed ranks: entered with a known state, so
// no lead-in before its first credited step
__device__ inline TileGeom block_tile_geom(uint32_t n, uint32_t h) {
    TileGeom g;
    g.n = n;
    g.t0 = h * kBlkL;
    g.S0 = g.t0 >= 64 ? g.t0 - 64 : 0;
    g.Q0 = g.S0;
    g.L = min(kBlkL, n - kWin - g.t0);
    g.SE = g.t0 + g.L;
    g.RE = min(g.SE + 64, n);
    g.BE = n;
    return g;
}

// ranks | fres (afterwards the insert's owner table) | scores of the whole
// block | sig | tau | misc
constexpr uint32_t kBlkRanks = align_up(padded_len(kBlkL + 128 + 8) * 2, 16), kBlkFres = align_up(padded_len(kBlkL + 64) * 2, 16);
static_assert(kOwnBytes <= kBlkFres, "the owner table fits the full-rescan table");
constexpr uint32_t kBlkSmem = kBlkRanks + kBlkFres + align_up(kMaxBlockBytes + 32, 16) + 2 * kSegs * 8 + 64 * 4;
__device__ inline TileSmem carve_block_pre(uint8_t* p) {
    TileSmem s;
    s.bytes32 = nullptr;
    s.hist = nullptr;
    s.ranks = reinterpret_cast<uint16_t*>(p); p += kBlkRanks;
    s.list = nullptr;
    s.fres = reinterpret_cast<uint16_t*>(p);
    s.own = reinterpret_cast<uint32_t*>(p); p += kBlkFres;
    s.score32 = reinterpret_cast<uint32_t*>(p); p += align_up(kMaxBlockBytes + 32, 16);
    s.sig = reinterpret_cast<uint64_t*>(p); p += kSegs * 8;
    s.tau = reinterpret_cast<uint64_t*>(p); p += kSegs * 8;
    s.misc = reinterpret_cast<uint32_t*>(p);
    return s;
}

// Selection and ordered insert (kind 0: thread_gen_block_sdbf's histogram
// threshold, sdbf_core.cc:271-276; kind 1, a tail: 16, sdbf_core.cc:315).
// The block's positions of score >= 15 are listed once (a threshold is never
// lower), the histogram counts the list, every warp finds the threshold from
// its suffix sums, and each warp drops the entries below it from its list.
// The insert (gen_block_hash, sdbf_core.cc:157-183) takes kGenThreads
// candidates at once, one per thread: a candidate is eligible if its score is
// above the threshold k, or equal to it while `allowed` lasts; an eligible one
// sets its 5 filter bits and is counted if one was new -- unset before, with
// this candidate as its smallest holder (a table of the smallest candidate
// per filter bit; the key's high part counts passes down, so a pass overrides
// its predecessors).  A pass takes every candidate as eligible, then keeps
// those before the first one counted past the allowance (it is skipped and
// the rest re-run with the allowance spent) and stops after the one that
// reaches 192.
// (One warp that inserted 32 candidates at a time after the whole CTA had
// counted all 16 K scores one by one and compacted them in two passes: 54 K
// of a block's 119 K cycles; 6.6 ms for a 1 GiB image became 5.1.)
constexpr uint32_t kBlkWarpList = ((kMaxBlockBytes / (kGenThreads / 32)) + 64) / 15 + 3;  // scores >= 15 in a warp's range

// Index of the n-th (from 1) set bit of a mask of kGenThreads bits that has as many.
__device__ __forceinline__ uint32_t nth_bit(const uint32_t* m, uint32_t n) {
    uint32_t w = 0;
    while (n > (uint32_t)__popc(m[w])) n -= __popc(m[w++]);
    return 32 * w + __fns(m[w], 0, (int)n);
}

template <bool kPre>
__global__ void __launch_bounds__(kGenThreads, kPre ? 4 : 1) k_block_digest(GenParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t histo[66];
    constexpr uint32_t kWarps = kGenThreads / 32;
    static_assert(kWarps == 4, "candidate lists are walked as four");
    __shared__ uint32_t counts[kWarps];
    __shared__ uint32_t filt[64];
    __shared__ uint16_t lists[kWarps][kBlkWarpList];
    __shared__ uint32_t madd[kWarps], maddk[kWarps];  // candidates counted in a pass; those of score k
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint16_t* rank_tab = nullptr;
    const int32_t* dt = nullptr;
    if constexpr (!kPre) {
        __shared__ int32_t dtab[65];
        __shared__ uint16_t s_rank[(SDBF_RANK_BINS + 7) / 8 * 8];
        for (uint32_t i = threadIdx.x; i < 65; i += blockDim.x) dtab[i] = i < 64 ? (int32_t)P.ent_tab[i + 1] - (int32_t)P.ent_tab[i] : 0;
        for (uint32_t i = threadIdx.x; i < SDBF_RANK_BINS; i += blockDim.x) s_rank[i] = P.rank_tab[i];
        __syncthreads();
        rank_tab = s_rank;
        dt = dtab;
    }
    TileSmem s = kPre ? carve_block_pre(smem) : carve(smem, P.block_lmax);
    for (uint32_t b = blockIdx.x; b < P.nchunks; b += gridDim.x) {
        const GenChunk C = P.chunks[b];
        const uint8_t* chunk = P.data + C.data_off;
        const uint32_t nown = C.n - kWin;
        if (threadIdx.x < 66) histo[threadIdx.x] = 0;
        if (threadIdx.x < 64) filt[threadIdx.x] = 0;
        if constexpr (kPre) {
            __shared__ uint64_t carry;
            const uint32_t ntile = (nown + kBlkL - 1) / kBlkL;
            for (uint32_t h = 0; h < ntile; h++) {
                const TileGeom g = block_tile_geom(C.n, h);
                TileSmem st = s;
                st.score32 += g.t0 / 4;
                tile_pipeline<true>(chunk, g, st, nullptr, nullptr, h ? &carry : nullptr, nullptr, nullptr, P.lead, nullptr,
                                    P.ranks + (size_t)C.rank_off8 * 8);
                if (threadIdx.x == 0) carry = *reinterpret_cast<uint64_t*>(&s.misc[10]);
                __syncthreads();
            }
        } else {
            tile_pipeline(chunk, block_geom(C.n), s, rank_tab, dt, nullptr, nullptr, nullptr, P.lead, nullptr);
        }
        const uint8_t* sc = reinterpret_cast<const uint8_t*>(s.score32);
        uint16_t* list = lists[wid];
        uint32_t nw = compact_warp<kThreshold - 1>(s.score32, nown, &lists[0][0], kBlkWarpList);
        __syncwarp();
        if (C.kind == 0)
            for (uint32_t i = lane; i < nw; i += 32) atomicAdd(&histo[sc[list[i]]], 1u);
        uint4* own4 = reinterpret_cast<uint4*>(s.own);
        for (uint32_t i = threadIdx.x; i < kOwnBytes / 16; i += kGenThreads) own4[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        __syncthreads();
        // threshold k: the largest score >= 16 that more than 192 positions
        // reach (15 if none does); the allowance is what those above it leave
        uint32_t k = kThreshold, allowed = kMaxElemDD;
        if (C.kind == 0) {
            static_assert(66 - kThreshold == 2 * 25, "two scores per lane");
            const uint32_t c0 = lane < 25 ? histo[kThreshold + 2 * lane] : 0u;
            const uint32_t c1 = lane < 25 ? histo[kThreshold + 1 + 2 * lane] : 0u;
            uint32_t s0 = c0 + c1;  // positions of score >= 16 + 2 lane
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_down_sync(0xffffffffu, s0, d);
                if (lane + d < 32) s0 += y;
            }
            const uint32_t s1 = s0 - c0;  // of score >= 17 + 2 lane
            const uint32_t over = __ballot_sync(0xffffffffu, s0 > (uint32_t)kMaxElemDD);
            const uint32_t odd = __ballot_sync(0xffffffffu, s1 > (uint32_t)kMaxElemDD);
            const uint32_t L = over ? 31 - __clz(over) : 0;
            const bool hi = (odd >> L) & 1u;
            const uint32_t above = __shfl_sync(0xffffffffu, hi ? s1 - c1 : s1, L);
            const uint32_t all = __shfl_sync(0xffffffffu, s0, 0);
            k = over ? kThreshold + 2 * L + hi : kThreshold - 1;
            allowed = kMaxElemDD - (over ? above : all);
        }
        if (k >= kThreshold) {
            uint32_t m = 0;
            for (uint32_t i0 = 0; i0 < nw; i0 += 32) {
                const bool have = i0 + lane < nw;
                const uint16_t p = have ? list[i0 + lane] : (uint16_t)0;
                const bool sel = have && sc[p] >= k;
                const uint32_t bm = __ballot_sync(0xffffffffu, sel);
                if (sel) list[m + __popc(bm & lanemask_lt())] = p;
                m += __popc(bm);
                __syncwarp();
            }
            nw = m;
        }
        if (lane == 0) counts[wid] = nw;
        __syncthreads();
        const uint32_t n1 = counts[0], n2 = n1 + counts[1], n3 = n2 + counts[2], ncand = n3 + counts[3];
        uint32_t hashed = 0, pass = 0xFFFFu;
        for (uint32_t base = 0; base < ncand && hashed < (uint32_t)kMaxElemDD; base += kGenThreads) {
            const uint32_t f = base + threadIdx.x;
            const bool have = f < ncand;
            uint32_t h[5] = {0, 0, 0, 0, 0};
            bool isk = false;
            if (have) {
                const uint32_t wl = (f >= n1) + (f >= n2) + (f >= n3);
                const uint32_t before = wl == 0 ? 0u : wl == 1 ? n1 : wl == 2 ? n2 : n3;
                const uint32_t p = lists[wl][f - before];
                isk = sc[p] == k;
                uint32_t w[16];
                if constexpr (kPre)
                    load_be16_global(chunk + p, w);
                else
                    load_be16(s.bytes32, p, w);
                sha1_feature(w, h);
            }
            uint32_t start = 0;
            while (true) {
                const bool act = have && threadIdx.x >= start && (!isk || allowed > 0);
                const uint32_t key = (--pass << 16) | threadIdx.x;
                uint32_t fresh = 0;
                if (act) {
#pragma unroll
                    for (int z = 0; z < 5; z++) {
                        const uint32_t a = h[z] & kBfMask;
                        fresh |= (~(filt[a >> 5] >> (a & 31)) & 1u) << z;
                        atomicMin(&s.own[a], key);
                    }
                }
                __syncthreads();
                bool added = false;
                if (act) {
#pragma unroll
                    for (int z = 0; z < 5; z++) added |= ((fresh >> z) & 1u) && s.own[h[z] & kBfMask] == key;
                }
                const uint32_t bm = __ballot_sync(0xffffffffu, added), bk = __ballot_sync(0xffffffffu, added && isk);
                if (lane == 0) {
                    madd[wid] = bm;
                    maddk[wid] = bk;
                }
                __syncthreads();
                uint32_t total = 0, totalk = 0, before = __popc(bm & lanemask_lt());
#pragma unroll
                for (uint32_t q = 0; q < kWarps; q++) {
                    total += __popc(madd[q]);
                    totalk += __popc(maddk[q]);
                    if (q < wid) before += __popc(madd[q]);
                }
                uint32_t end = kGenThreads;  // candidates [start, end) stand
                bool skip = false, full = false;
                if (totalk > allowed) {
                    end = nth_bit(maddk, allowed + 1);
                    skip = true;
                }
                if (hashed + total >= (uint32_t)kMaxElemDD) {
                    const uint32_t last = nth_bit(madd, kMaxElemDD - hashed);  // the block's 192nd
                    if (last < end) {
                        end = last + 1;
                        full = true;
                    }
                }
                if (act && threadIdx.x < end) {
#pragma unroll
                    for (int z = 0; z < 5; z++) {
                        const uint32_t a = h[z] & kBfMask;
                        atomicOr(&filt[a >> 5], 1u << (a & 31));
                    }
                    if (added) {
                        const uint32_t idx = hashed + before;
                        if (P.feats) {  // index build: every counted feature (sdbf_core.cc:164-167)
                            uint32_t* fw = P.feats + (size_t)C.filter * kFeatWords + idx * 5;
#pragma unroll
                            for (int z = 0; z < 5; z++) fw[z] = h[z];
                        }
                        if (P.probes && (idx & 3) == 0) {  // index search sample (sdbf_core.cc:168-175)
                            uint32_t* pr = P.probes + (size_t)C.filter * kProbeWords + (idx >> 2) * 5;
#pragma unroll
                            for (int z = 0; z < 5; z++) pr[z] = h[z];
                        }
                    }
                }
                if (end < (uint32_t)kGenThreads) {  // count those that stand only
                    total = totalk = 0;
#pragma unroll
                    for (uint32_t q = 0; q < kWarps; q++) {
                        const uint32_t keep = end >= 32 * q + 32 ? 0xffffffffu : end <= 32 * q ? 0u : (1u << (end - 32 * q)) - 1u;
                        total += __popc(madd[q] & keep);
                        totalk += __popc(maddk[q] & keep);
                    }
                }
                hashed += total;
                allowed -= totalk;
                __syncthreads();  // the filter's bits are set, the masks read
                if (full || !skip) break;
                start = end + 1;  // candidate `end` is skipped (allowance spent)
            }
        }
        if (threadIdx.x < 64) P.out_filters[(size_t)C.filter * 64 + threadIdx.x] = filt[threadIdx.x];
        if (threadIdx.x == 0) P.out_counts[C.filter] = (uint16_t)hashed;
        if (threadIdx.x == 0 && P.nprobes) P.nprobes[C.filter] = (uint8_t)((hashed + 3) >> 2);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- launch
size_t stream_tile_smem() { return tile_smem_bytes(kTileL); }
size_t stream_tile_smem_pre() { return tile_smem_bytes_pre(kTileL); }
size_t block_smem(uint32_t lmax) { return tile_smem_bytes(lmax); }

// Attributes belong to a device: they are set once on each (contexts may be
// used from several threads).
static void set_stream_attrs_here() {
    const int sm = (int)stream_tile_smem(), smp = (int)stream_tile_smem_pre();
    cudaFuncSetAttribute(k_stream_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_stream_fix<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_stream_tiles_pre, cudaFuncAttributeMaxDynamicSharedMemorySize, smp);
    cudaFuncSetAttribute(k_stream_fix<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smp);
    cudaFuncSetAttribute(k_stream_fix_list<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_stream_fix_list<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smp);
    cudaFuncSetAttribute(k_stream_ranks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRkSmem);
    cudaFuncSetAttribute(k_stream_commit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CommitSmem<false>));
    cudaFuncSetAttribute(k_stream_commit_round, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(CommitSmem<true>));
    cudaFuncSetAttribute(k_stream_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChainSmem));
    cudaFuncSetAttribute(k_feat_links, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LinkSmem));
    // one shared-memory / L1 split for every kernel of the stream pipeline
    // (the largest shared memory): CTAs of different kernels can then share
    // an SM
    for (const void* f : {(const void*)k_stream_ranks, (const void*)k_stream_tiles, (const void*)k_stream_tiles_pre,
                          (const void*)k_stream_fails, (const void*)k_stream_fix_list<false>,
                          (const void*)k_stream_fix_list<true>,
                          (const void*)k_stream_fix<false>, (const void*)k_stream_fix<true>,
                          (const void*)k_stream_commit, (const void*)k_stream_commit_round,
                          (const void*)k_stream_commit_index, (const void*)k_feat_scan, (const void*)k_feat_pack,
                          (const void*)k_feat_last, (const void*)k_feat_carry, (const void*)k_feat_links,
                          (const void*)k_stream_chain, (const void*)k_stream_emit})
        cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
}
static void set_stream_attrs() {
    static std::once_flag done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) std::call_once(done[dev], set_stream_attrs_here);
    else set_stream_attrs_here();
}

int rk_choose(const uint64_t* stretches, uint32_t sms) {
    const uint64_t slots = (uint64_t)sms * 3;
    int best = 0;
    uint64_t cost = ~0ull;
    for (int k = 0; k < kRkChoices; k++) {
        const uint64_t c = (stretches[k] + slots - 1) / slots * (64 + kRkPers[k]);
        if (c < cost) {
            cost = c;
            best = k;
        }
    }
    return best;
}

cudaError_t launch_stream_ranks(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    if (grid) k_stream_ranks<<<grid, kRkThreads, kRkSmem, st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_tiles(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    if (P.ranks)
        k_stream_tiles_pre<<<grid, kGenThreads, stream_tile_smem_pre(), st>>>(P);
    else
        k_stream_tiles<<<grid, kGenThreads, stream_tile_smem(), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_fails(const GenParams& P, uint32_t grid, cudaStream_t st) {
    if (grid) k_stream_fails<<<grid, 256, 0, st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_fix_list(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    if (P.ranks)
        k_stream_fix_list<true><<<grid, kGenThreads, stream_tile_smem_pre(), st>>>(P);
    else
        k_stream_fix_list<false><<<grid, kGenThreads, stream_tile_smem(), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_fix(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    if (P.ranks)
        k_stream_fix<true><<<grid, kGenThreads, stream_tile_smem_pre(), st>>>(P);
    else
        k_stream_fix<false><<<grid, kGenThreads, stream_tile_smem(), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_commit_index(const GenParams& P, cudaStream_t st) {
    k_stream_commit_index<<<1, 32, 0, st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_commit_round(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    k_stream_commit_round<<<grid, kCmThreads, sizeof(CommitSmem<true>), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_index_pred(const GenParams& P, const uint32_t* first, uint32_t* pred, uint32_t grid,
                                     cudaStream_t st) {
    k_stream_index_pred<<<grid, 256, 0, st>>>(P.features, P.tile_out, P.ntiles, first, P.index_mask, pred);
    return cudaGetLastError();
}

cudaError_t launch_stream_index_first(const GenParams& P, const uint32_t* seen, uint32_t* first, uint32_t grid,
                                      cudaStream_t st) {
    k_stream_index_first<<<grid, 256, 0, st>>>(P.features, P.tile_out, P.ntiles, seen, P.index_mask, first);
    return cudaGetLastError();
}

cudaError_t launch_stream_index_mark(const GenParams& P, const uint32_t* seen, const uint32_t* first, uint32_t grid,
                                     cudaStream_t st) {
    k_stream_index_mark<<<grid, 256, 0, st>>>(P.features, P.tile_out, P.ntiles, seen, P.index_mask, first,
                                              P.index_bits, P.index_new);
    return cudaGetLastError();
}

cudaError_t launch_pred_dirty(const GenParams& P, const uint32_t* a, const uint32_t* b, uint64_t nwords,
                              uint8_t* dirty, uint32_t* from, unsigned int* ndirty, uint32_t grid, cudaStream_t st) {
    k_pred_dirty<<<grid, 256, 0, st>>>(a, b, nwords, P.tiles, P.chunks, P.ntiles, dirty, from, ndirty);
    return cudaGetLastError();
}

cudaError_t launch_stream_links(const GenParams& P, uint32_t sms, cudaStream_t st) {
    set_stream_attrs();
    const uint32_t files = min(P.nfiles, 4096u);
    // CTAs per file: enough to fill the SMs with one-warp CTAs
    const uint32_t x = max(4u, 24 * sms / files);
    k_feat_scan<<<min(P.nfiles, 2 * sms), 1024, 0, st>>>(P);
    k_feat_pack<<<min((P.ntiles + 7) / 8, 8 * sms), 256, 0, st>>>(P);
    k_feat_last<<<dim3(x, files), 32, 0, st>>>(P);
    k_feat_carry<<<dim3(kLkTab / 128, files), 128, 0, st>>>(P);
    k_feat_links<<<dim3(x, files), 32, sizeof(LinkSmem), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_chain(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    k_stream_chain<<<grid, kCmWin, sizeof(ChainSmem), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_stream_emit(const GenParams& P, const uint64_t* dst_off, uint32_t* dst, uint64_t dst_cap, uint32_t sms,
                               cudaStream_t st) {
    const uint32_t files = min(P.nfiles, 4096u);
    k_stream_emit<<<dim3(max(1u, 8 * sms / files), files), 256, 0, st>>>(P, dst_off, dst, dst_cap);
    return cudaGetLastError();
}

cudaError_t launch_stream_commit(const GenParams& P, uint32_t grid, cudaStream_t st) {
    set_stream_attrs();
    k_stream_commit<<<grid, kCmThreads, sizeof(CommitSmem<false>), st>>>(P);
    return cudaGetLastError();
}

cudaError_t launch_block(const GenParams& P, uint32_t sms, cudaStream_t st) {
    if (P.nchunks == 0) return cudaSuccess;
    if (P.ranks) {
        cudaFuncSetAttribute(k_block_digest<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlkSmem);
        cudaFuncSetAttribute(k_block_digest<true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
        k_block_digest<true><<<min(P.nchunks, sms * 4 * 8), kGenThreads, kBlkSmem, st>>>(P);
    } else {
        const size_t sm = block_smem(P.block_lmax);
        cudaFuncSetAttribute(k_block_digest<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        k_block_digest<false><<<min(P.nchunks, sms * 2 * 8), kGenThreads, sm, st>>>(P);
    }
    return cudaGetLastError();
}

}  // namespace sdbfg
