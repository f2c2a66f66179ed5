// ctx_internal.h -- the context and digest-set objects behind the C ABI,
// shared by the generation (sdbf_api.cu) and comparison (compare_api.cu)
// host code.  Not part of the public interface.
#pragma once
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/sdbf_gb300.h"
#include "compare_kernels.h"
#include "gen_kernels.h"

using namespace sdbfg;

namespace sdbfg_host {

constexpr uint32_t kMaxTilesPerLaunch = 1u << 18;  // 2 GiB of stream input per launch group
constexpr uint64_t kMaxBytesPerLaunch = 2ull << 30;
// Block-mode input whose ranks are held at once (512 MiB of them).  On the
// device 1 GiB in blocks of 16 KiB: 6.13 ms, with 128 MiB 6.29, with 512 MiB
// 6.03; 400 uneven files in blocks of 4 KiB: 5.32, 5.40 and 5.27.
constexpr uint64_t kBlockSlabBytes = 256ull << 20;
// First slab of a host-input block batch (each later one at most twice it).
// 768 fragments of 140 MB: 2.40 ms, with 8 MiB 2.54, with 32 MiB 2.40; 100
// files of 600 KiB: 1.61, 1.65 and 1.67; four of 128 MiB: 4.81, 4.64 and 4.86.
constexpr uint64_t kFirstHostSlabBytes = 16ull << 20;
// Stream batches (inputs sorted by size, largest first) in groups of this size:
// a group's ordered commits, which one large file can draw out, run beside
// the tiles of the groups behind it, and the last group's files are small.
// On the device 64 files of 40 MiB: 18.6 ms, in groups of 128 MiB 19.1, of 512
// MiB 18.5; 1,000 of 1 MiB: 6.20, 6.31 and 6.21.  From the host 300 uneven files
// of up to 16 MiB: 7.85, 7.46 and 8.10; 400 of 1 MiB: 4.24, 4.18 and 4.27.
constexpr uint64_t kStreamGroupBytes = 256ull << 20;
// A long batch keeps the GPU busy whatever the groups' size, and many commits in
// flight take the registers that the staging gather's CTAs need on an SM: groups
// of 1 GiB, four in flight.  28.4 GB: 160 ms on the device and 201 from the
// host (eight in flight: 160 and 287); groups of 256 MiB, eight in flight: 164
// and 303.  1,500 files of 4 MiB: 35.8 and 54.2, in groups of 256 MiB 36.1 and
// 71.9; 2,500 from the host 88.0, in groups of 512 MiB 89.0, of 2 GiB 91.5.  The
// line is not sharp: 2.4 GiB from the host take 23.2 ms either way, 3.7 GiB
// 41.3 and with the long batches' groups 35.4.
constexpr uint64_t kLongBatchBytes = 4ull << 30;
constexpr uint64_t kLongGroupBytes = 1ull << 30;
// First group of a host-input stream batch (each later one at most twice it):
// its copy is the one nothing hides.  64 files of 1 MiB: 1.06 ms, with 16 MiB
// 1.11, with 64 MiB (one group) 1.17; 200 of 200 KiB: 0.86, 0.78 and 0.85; 600 of
// 1 MiB: 6.23, 6.28 and 6.27; 160 uneven ones of 0.86 GB: 9.68, 9.52 and 9.70.
constexpr uint64_t kFirstHostGroupBytes = 32ull << 20;
// A group with a file of this many tiles, and at least half of all, commits
// through links (k_stream_chain): there the group waits for that one file's
// chain.  One file of 2, 3, 8 and 32 MiB on the device: 209, 267, 537 and 1,698
// us, through k_stream_commit 191, 289, 717 and 2,646; of 5 and 100 MiB 380 and
// 5,110 against 464 and 8,280; two files of 4 MiB 384 against 440.  Where many files'
// commits run beside tiles anyway, the links are only more work: 3.1 GB of
// uneven files 22.9 ms against 21.2.
constexpr uint32_t kChainTiles = 384;
constexpr uint64_t kFirstIndexGroupBytes = 256ull << 20;  // with an index being built (groups one after another)
// Output filters (128 KiB) that a host batch reads back with its results: one
// file of 200 and 900 KiB 113 and 164 us, without 118 and 171.
constexpr uint64_t kFetchFilters = 512;
constexpr uint32_t kMinFile = 512;                 // MIN_FILE_SIZE (sdbf_defines.h:56)
constexpr uint64_t kPairsPerLaunch = 1ull << 22;
constexpr int kSlots = 8;  // stream-mode launch groups in flight (at most)
// host-input stream batches up to this size (and half the free device
// memory) are staged whole on the device, where it can read the host's memory
constexpr uint64_t kStageMaxBytes = 64ull << 30;
constexpr uint64_t kStagePiece = 1ull << 20;  // work item of the staging gather
struct StagePiece {
    uint64_t dst;  // staging offset (16-byte aligned)
    uint64_t src;  // the host bytes as the device addresses them
    uint64_t len;
};


// Device / pinned-host arrays that grow on demand and free themselves with
// their owner (not copyable).
struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), cap(o.cap) {
        o.p = nullptr;
        o.cap = 0;
    }
    DevBuf& operator=(DevBuf&& o) noexcept {
        if (this != &o) {
            release();
            p = o.p;
            cap = o.cap;
            o.p = nullptr;
            o.cap = 0;
        }
        return *this;
    }
    ~DevBuf() { release(); }
    cudaError_t ensure(size_t bytes) {
        if (bytes <= cap) return cudaSuccess;
        const size_t want = std::max(bytes, cap + cap / 2);
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        cudaError_t e = cudaMalloc(&p, want);
        if (e == cudaSuccess) cap = want;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

// A part of a DevBuf.
struct DevView {
    void* p = nullptr;
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

struct HostBuf {
    void* p = nullptr;
    size_t cap = 0;
    HostBuf() = default;
    HostBuf(const HostBuf&) = delete;
    HostBuf& operator=(const HostBuf&) = delete;
    HostBuf(HostBuf&& o) noexcept : p(o.p), cap(o.cap) {
        o.p = nullptr;
        o.cap = 0;
    }
    HostBuf& operator=(HostBuf&& o) noexcept {
        if (this != &o) {
            release();
            p = o.p;
            cap = o.cap;
            o.p = nullptr;
            o.cap = 0;
        }
        return *this;
    }
    ~HostBuf() { release(); }
    cudaError_t ensure(size_t bytes) {
        if (bytes <= cap) return cudaSuccess;
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
        cudaError_t e = cudaMallocHost(&p, bytes);
        if (e == cudaSuccess) cap = bytes;
        return e;
    }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

}  // namespace sdbfg_host

using namespace sdbfg_host;

struct KernelTimer {
    const char* name;
    cudaEvent_t a, b;
};

struct KernelStat {
    std::string name;
    double ms = 0;
    uint64_t launches = 0;
};

struct sdbfg_ctx {
    bool profile = false;
    std::vector<KernelTimer> pending;
    std::vector<KernelStat> stats;
    int device = 0;
    cudaStream_t own = nullptr;
    cudaStream_t stream = nullptr;
    std::string err;
    uint64_t launches = 0;
    int sms = 152;
    uint32_t lead = kDefaultLead;
    bool pre_ranks = true;  // stream mode: ranks by k_stream_ranks ahead of the tile kernel
    DevBuf d_ranks;         // their ranks (two halves, by launch-group parity)
    bool reads_pageable = false;  // the device reads pageable memory through the host's page tables
    // constant tables
    DevBuf d_rank, d_ent, d_cut, d_cut64;
    // generation buffers
    DevBuf d_data, d_chunks, d_counters, d_out_filters, d_out_counts;
    HostBuf h_flags;  // pinned words: [0] small read-backs, [1] set when a comparison gave up
    uint32_t* gave_up() const { return static_cast<uint32_t*>(h_flags.p) + 1; }
    // comparison buffers
    DevBuf d_pairs, d_scores;
    // stream-mode pipeline: launch-group slots on their own streams
    struct Slot {
        cudaStream_t stream = nullptr;
        cudaEvent_t done = nullptr;
        bool used = false;
        DevBuf data, tile_out, features, work;
        DevBuf links, last_tab, chain;  // linked commit; chain: tile places, file totals, filter ends
        // chunks, tiles, files, order, rank stretches and the (zero) head of
        // the list of failing links, uploaded in one copy; the list follows
        DevBuf tables;
        HostBuf h_tables;
    } slot[kSlots];
    int depth = kSlots;  // launch groups in flight (at kSlots: fewer in long batches)
    DevBuf d_result, d_phase;  // of a stream batch: total filters, per-file info and output slots
    HostBuf h_result;
    HostBuf h_block;  // a block-mode launch group's tables
    // host-input stream batches staged whole on the device: per-file copies
    // in launch-group order on their own stream, one event per group
    DevBuf d_stage_in, d_stage_items;
    bool staging = false;  // a batch reads d_stage_in
    HostBuf h_stage_items;
    cudaStream_t copy_stream = nullptr;
    std::vector<cudaEvent_t> ev_copy;
    cudaEvent_t ev_scan[kSlots] = {};
    cudaEvent_t ev_tiles[kSlots] = {};  // a group's tile kernels done
    cudaEvent_t ev_start = nullptr;
    // A buffer that a call cannot do without.  Where there is no room for it,
    // what earlier calls left and later ones can do without or make again goes
    // first: the linked commit's buffers (1.4 bytes per byte of a file) and the
    // staging copy (cudaFree waits for their users).
    cudaError_t must(DevBuf& b, size_t bytes) {
        cudaError_t e = b.ensure(bytes);
        if (e != cudaErrorMemoryAllocation) return e;
        cudaGetLastError();
        for (Slot& s : slot) {
            s.links.release();
            s.last_tab.release();
        }
        if (!staging) d_stage_in.release();
        return b.ensure(bytes);
    }
    // comparison engine: tuning and cached plans (work units + CUDA graph)
    int mat_variant = kMatVariantTc;  // tensor-core counting
    uint64_t mat_unit_work = 1ull << 22;
    bool mat_graphs = true;
    std::vector<struct MatPlan*> plans;
    cudaEvent_t ev_plan = nullptr;      // behind the last copy of a plan's tables,
    bool plan_tables_queued = false;    //   which may not have run yet
    DevBuf d_match_counts, d_match_offs, d_matches, d_mphase;
    // index search: per-slot probe words and counts of the group being
    // digested (set around a block-mode batch), the device index table
    uint32_t* probe_words = nullptr;
    uint8_t* probe_counts = nullptr;
    DevBuf d_probes, d_nprobes, d_hits, d_index_tab;
    // index build: counted features of the group being digested (block
    // mode), the index bits, the first setter of every bit, the new-insert count
    uint32_t* feat_words = nullptr;
    DevBuf d_feats, d_idx_bits, d_idx_first, d_idx_count;
    // stream-mode index build: fixed-point rounds before the sequential
    // commit takes over (0: sequential only), rounds the last launch group took
    uint32_t index_max_rounds = 16;
    uint32_t index_rounds_used = 0;
    DevBuf d_seen[2], d_pred, d_diff, d_ckpt, d_from;
};

// A resident index filter (bloom_filter of an index file).
struct sdbfg_index {
    sdbfg_ctx* ctx = nullptr;
    uint64_t bf_size = 0, elem_count = 0, bit_mask = 0;
    uint32_t hash_count = 0;
    std::string name;
    DevBuf d_bits;
};

// Block-mode index build over one launch group's slots [0, nslots) (global
// slots from slot0): each bit's first setter in input order, then the bits
// and the count of features that set a new one (bloom_filter::insert_sha1
// in that order, bloom_filter.cc:333-359).
int index_build_group(sdbfg_ctx* c, const uint32_t* d_feats, const uint16_t* d_counts, uint64_t nslots,
                      uint64_t slot0, uint32_t mask, uint32_t* d_first, uint32_t* d_bits,
                      unsigned long long* d_count, cudaStream_t st);
// first[p] = 0 for bits already set, ~0 otherwise.
int index_first_init(sdbfg_ctx* c, const uint32_t* d_bits, uint32_t* d_first, uint64_t nbits, cudaStream_t st);

// Hits of every probe slot against every index (k_index_query).
int index_query(sdbfg_ctx* c, const uint32_t* d_probes, const uint8_t* d_nprobes, uint64_t nslots,
                const sdbfg_index* const* indexes, uint32_t nidx, uint8_t* d_hits, cudaStream_t st);

struct sdbfg_set {
    sdbfg_ctx* ctx = nullptr;
    uint32_t n = 0;
    std::vector<std::string> names;
    std::vector<uint32_t> bf_count;
    std::vector<uint32_t> last_elem;  // element count of the last filter (swap rule)
    std::vector<uint8_t> fast;         // per digest: folded by sdbfg_set_fast
    // header fields of the SDBF text form (sdbf::to_string, sdbf_class.cc:293-334)
    std::vector<uint64_t> orig_size;
    std::vector<uint32_t> max_elem, last_count, dd_block;  // dd_block 0: stream digest
    uint64_t serial = 0;               // identifies the set in cached comparison plans
    uint64_t total_filters = 0;
    std::vector<uint32_t> first;       // first filter of each digest in d_filters
    DevBuf d_all;  // one allocation: filters, meta, digests
    DevView d_filters, d_meta, d_digests;
    static uint64_t meta_at(uint64_t filters) { return std::max<uint64_t>(1, filters) * 256; }
    static uint64_t digests_at(uint64_t filters) { return meta_at(filters) + (filters * 4 + 255) / 256 * 256; }
    static uint64_t bytes(uint64_t filters, uint64_t digests) { return digests_at(filters) + (digests + 1) * sizeof(CmpDigest); }
    cudaError_t allocate(uint64_t filters, uint64_t digests) {
        const cudaError_t e = ctx->must(d_all, bytes(filters, digests));
        if (e != cudaSuccess) return e;
        d_filters.p = d_all.p;
        d_meta.p = d_all.as<uint8_t>() + meta_at(filters);
        d_digests.p = d_all.as<uint8_t>() + digests_at(filters);
        return e;
    }
};

// Serial number of a new set (cached comparison plans are keyed by it).
uint64_t next_set_serial();

// Waits until the tables of the context's plans are on the device: before
// work on another stream than the one their copies are queued on.
cudaError_t plan_tables_arrived(sdbfg_ctx* c);

// A comparison job prepared for the matrix engine: work units sorted by
// size, the target list, split-pair table and slot array, and (once run) a
// CUDA graph of its launches.
struct MatPlan {
    uint64_t serial_a = 0, serial_b = 0;
    uint32_t mode = 0;
    int variant = 0;
    uint64_t unit_work = 0;
    uint32_t nunits = 0, nsplit = 0;
    uint64_t nscores = 0, nslots = 0;
    uint64_t filter_pairs = 0;  // sum over scored pairs of n_ref * n_tgt
    DevBuf d_all;  // one allocation: units, targets, refs, split | redo list | counters, slots
    DevView d_units, d_targets, d_refs, d_split, d_redo, d_counter;
    std::vector<uint8_t> tables;  // the uploaded tables: alive for their copy, which is only queued
    cudaGraphExec_t graph = nullptr;
    int32_t* graph_out = nullptr;  // output of the captured (or, before that, of the last) run
    uint64_t last_use = 0;
    ~MatPlan() {
        if (graph) cudaGraphExecDestroy(graph);
        d_all.release();  // waits for the device: the tables' copy is done
    }
};

// Per-kernel CUDA-event timing on the launch stream (only when enabled).
inline void timer_begin(sdbfg_ctx* c, const char* name, cudaEvent_t* a, cudaStream_t st) {
    *a = nullptr;
    if (!c->profile) return;
    cudaEventCreate(a);
    cudaEventRecord(*a, st);
    (void)name;
}

inline void timer_end(sdbfg_ctx* c, const char* name, cudaEvent_t a, cudaStream_t st) {
    if (!c->profile || !a) return;
    cudaEvent_t b;
    cudaEventCreate(&b);
    cudaEventRecord(b, st);
    c->pending.push_back({name, a, b});
}

inline void timer_collect(sdbfg_ctx* c) {
    for (KernelTimer& t : c->pending) {
        cudaEventSynchronize(t.b);
        float ms = 0;
        cudaEventElapsedTime(&ms, t.a, t.b);
        KernelStat* st = nullptr;
        for (KernelStat& k : c->stats)
            if (k.name == t.name) st = &k;
        if (!st) {
            c->stats.push_back(KernelStat{t.name, 0, 0});
            st = &c->stats.back();
        }
        st->ms += ms;
        st->launches += 1;
        cudaEventDestroy(t.a);
        cudaEventDestroy(t.b);
    }
    c->pending.clear();
}

#define TIMED_LAUNCH_ON(c, name, st_, expr)     \
    do {                                        \
        cudaEvent_t ev_;                        \
        timer_begin((c), (name), &ev_, (st_));  \
        cudaError_t le_ = (expr);               \
        timer_end((c), (name), ev_, (st_));     \
        if (le_ != cudaSuccess)                 \
            return fail((c), SDBFG_ERR_CUDA, "%s launch: %s", (name), cudaGetErrorString(le_)); \
        (c)->launches += 1;                     \
    } while (0)
#define TIMED_LAUNCH(c, name, expr) TIMED_LAUNCH_ON(c, name, (c)->stream, expr)

inline int fail(sdbfg_ctx* c, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    return code;
}

#define CUDA_TRY(ctx, call)                                                                       \
    do {                                                                                         \
        cudaError_t e_ = (call);                                                                 \
        if (e_ != cudaSuccess)                                                                   \
            return fail((ctx), e_ == cudaErrorMemoryAllocation ? SDBFG_ERR_NOMEM : SDBFG_ERR_CUDA, \
                        "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);    \
    } while (0)

