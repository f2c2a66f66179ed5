// compare_api.cu -- digest sets on the device and the comparison entry
// points of the C ABI (include/sdbf_gb300.h).
#include <algorithm>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include <atomic>

#include "ctx_internal.h"
#include "matrix_plan.h"

static std::atomic<uint64_t> g_set_serial{1};

uint64_t next_set_serial() { return g_set_serial.fetch_add(1); }

// -------------------------------------------------------------- comparison
extern "C" int sdbfg_set_upload(sdbfg_ctx* c, const sdbfg_digest_desc* ds, uint32_t n, sdbfg_set** out) {
    if (!c || !out || (n && !ds)) return SDBFG_ERR_ARG;
    *out = nullptr;
    CUDA_TRY(c, cudaSetDevice(c->device));
    auto* s = new sdbfg_set();
    s->ctx = c;
    s->n = n;
    s->serial = next_set_serial();
    uint64_t total = 0;
    std::vector<CmpDigest> dig(n);
    for (uint32_t i = 0; i < n; i++) {
        if (ds[i].bf_count == 0 || !ds[i].filters) {
            delete s;
            return fail(c, SDBFG_ERR_ARG, "digest %u has no filters", i);
        }
        dig[i] = {(uint32_t)total, ds[i].bf_count, 0, 0, 0};
        total += ds[i].bf_count;
    }
    if (total >= (1ull << 32)) {
        delete s;
        return fail(c, SDBFG_ERR_ARG, "set too large");
    }
    s->total_filters = total;
    std::vector<uint8_t> image(sdbfg_set::bytes(total, n));  // the set's device memory, copied at once
    uint8_t* filt = image.data();
    uint32_t* meta = reinterpret_cast<uint32_t*>(filt + sdbfg_set::meta_at(total));
    s->names.resize(n);
    s->fast.assign(n, 0);
    s->bf_count.resize(n);
    s->last_elem.resize(n);
    s->orig_size.resize(n);
    s->max_elem.resize(n);
    s->last_count.resize(n);
    s->dd_block.resize(n);
    s->first.resize(n);
    for (uint32_t i = 0; i < n; i++) {
        const sdbfg_digest_desc& d = ds[i];
        s->names[i] = d.name ? d.name : "";
        s->bf_count[i] = d.bf_count;
        s->orig_size[i] = d.orig_size;
        s->max_elem[i] = d.max_elem;
        s->last_count[i] = d.elem_counts ? 0 : d.last_count;
        s->dd_block[i] = d.elem_counts ? d.dd_block_size : 0;
        s->first[i] = dig[i].first;
        memcpy(filt + (uint64_t)dig[i].first * 256, d.filters, (uint64_t)d.bf_count * 256);
        for (uint32_t f = 0; f < d.bf_count; f++) {
            // get_elem_count (sdbf_class.cc:406-415)
            uint32_t e = d.elem_counts ? d.elem_counts[f] : (f + 1 < d.bf_count ? d.max_elem : d.last_count);
            uint32_t h = 0;
            const uint8_t* p = d.filters + (uint64_t)f * 256;
            for (int b = 0; b < 256; b += 8) {
                uint64_t w;
                memcpy(&w, p + b, 8);
                h += (uint32_t)__builtin_popcountll(w);
            }
            meta[dig[i].first + f] = (h << 16) | (e & 0xFFFFu);
            if (f + 1 == d.bf_count) s->last_elem[i] = e;
        }
        digest_stats(dig[i], meta);
    }
    if (n) memcpy(filt + sdbfg_set::digests_at(total), dig.data(), n * sizeof(CmpDigest));
    if (s->allocate(total, n) != cudaSuccess) {
        cudaGetLastError();
        delete s;
        return fail(c, SDBFG_ERR_NOMEM, "set upload: out of device memory");
    }
    cudaMemcpy(s->d_all.p, image.data(), image.size(), cudaMemcpyHostToDevice);
    *out = s;
    return SDBFG_OK;
}

static void drop_plans(sdbfg_ctx* c, uint64_t serial) {
    auto& plans = c->plans;
    for (size_t k = 0; k < plans.size();) {
        if (plans[k]->serial_a == serial || plans[k]->serial_b == serial) {
            delete plans[k];
            plans.erase(plans.begin() + k);
        } else {
            k++;
        }
    }
}

extern "C" int sdbfg_set_fast(sdbfg_ctx* c, sdbfg_set* s, uint32_t first, uint32_t count) {
    if (!c || !s || first > s->n || count > s->n - first) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (!count) return SDBFG_OK;
    TIMED_LAUNCH(c, "k_fold", launch_fold(s->d_filters.as<uint32_t>(), s->d_meta.as<uint32_t>(),
                                          s->d_digests.as<CmpDigest>(), first, count, c->stream));
    CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    for (uint32_t i = first; i < first + count; i++) s->fast[i] = 1;
    drop_plans(c, s->serial);  // group units are formed per fast mode
    return SDBFG_OK;
}

extern "C" void sdbfg_set_free(sdbfg_set* s) {
    if (!s) return;
    cudaSetDevice(s->ctx->device);
    drop_plans(s->ctx, s->serial);
    s->d_all.release();
    delete s;
}

extern "C" uint32_t sdbfg_set_size(const sdbfg_set* s) { return s ? s->n : 0; }

// Orientation of a pair: sdbf_score's swap rule (sdbf_core.cc:351-359).
static CmpPair orient(const sdbfg_set* a, uint32_t i, const sdbfg_set* b, uint32_t j) {
    const uint32_t n1 = a->bf_count[i], n2 = b->bf_count[j];
    const bool swap = n1 > n2 || (n1 == n2 && (a->last_elem[i] > b->last_elem[j] ||
                                               strcmp(a->names[i].c_str(), b->names[j].c_str()) > 0));
    if (swap) return CmpPair{j, i, n2, 1u | 0u};  // ref from b (side 1), tgt from a (side 0)
    return CmpPair{i, j, n1, 2u};                  // ref from a (side 0), tgt from b (side 1)
}

static int run_pairs(sdbfg_ctx* c, const sdbfg_set* a, const sdbfg_set* b, const std::vector<CmpPair>& pairs,
                     int32_t* out) {
    cudaStream_t st = c->stream;
    CUDA_TRY(c, c->must(c->d_pairs, std::max<size_t>(1, pairs.size()) * sizeof(CmpPair)));
    CUDA_TRY(c, c->must(c->d_scores, std::max<size_t>(1, pairs.size()) * 4));
    CUDA_TRY(c, cudaMemcpyAsync(c->d_pairs.p, pairs.data(), pairs.size() * sizeof(CmpPair), cudaMemcpyHostToDevice,
                                st));
    CmpParams P{};
    P.filters[0] = a->d_filters.as<uint32_t>();
    P.meta[0] = a->d_meta.as<uint32_t>();
    P.digests[0] = a->d_digests.as<CmpDigest>();
    P.filters[1] = b->d_filters.as<uint32_t>();
    P.meta[1] = b->d_meta.as<uint32_t>();
    P.digests[1] = b->d_digests.as<CmpDigest>();
    P.pairs = c->d_pairs.as<CmpPair>();
    P.npairs = pairs.size();
    P.scores = c->d_scores.as<int32_t>();
    P.cutoffs = c->d_cut.as<uint16_t>();
    P.cutoffs64 = c->d_cut64.as<uint16_t>();
    const uint32_t grid = (uint32_t)std::min<uint64_t>(pairs.size(), (uint64_t)c->sms * 16);
    TIMED_LAUNCH(c, "k_compare_pairs", launch_compare_pairs(P, std::max(1u, grid), st));
    CUDA_TRY(c, cudaMemcpyAsync(out, c->d_scores.p, pairs.size() * 4, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(c, cudaStreamSynchronize(st));
    return SDBFG_OK;
}

extern "C" int sdbfg_score_pairs(sdbfg_ctx* c, const sdbfg_set* a, const sdbfg_set* b, const uint32_t* ia,
                                 const uint32_t* ib, uint64_t npairs, int32_t* out) {
    if (!c || !a || !b || (npairs && (!ia || !ib || !out))) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    for (uint64_t base = 0; base < npairs; base += kPairsPerLaunch) {
        const uint64_t m = std::min<uint64_t>(kPairsPerLaunch, npairs - base);
        std::vector<CmpPair> pairs(m);
        for (uint64_t k = 0; k < m; k++) {
            const uint32_t i = ia[base + k], j = ib[base + k];
            if (i >= a->n || j >= b->n) return fail(c, SDBFG_ERR_ARG, "pair %llu out of range", (unsigned long long)k);
            pairs[k] = orient(a, i, b, j);
        }
        int rc = run_pairs(c, a, b, pairs, out + base);
        if (rc) return rc;
    }
    return SDBFG_OK;
}

// ------------------------------------------------------- matrix engine
// Orientation of pair (x of set a, y of set b) called as sdbf_score(x, y):
// true when y becomes the reference (the swap rule, sdbf_core.cc:351-359).
static bool swaps(const sdbfg_set* a, uint32_t x, const sdbfg_set* b, uint32_t y) {
    const uint32_t n1 = a->bf_count[x], n2 = b->bf_count[y];
    return n1 > n2 ||
           (n1 == n2 && (a->last_elem[x] > b->last_elem[y] || strcmp(a->names[x].c_str(), b->names[y].c_str()) > 0));
}

static MatPlan* find_plan(sdbfg_ctx* c, uint64_t sa, uint64_t sb, uint32_t mode) {
    static uint64_t tick = 0;
    for (MatPlan* p : c->plans)
        if (p->serial_a == sa && p->serial_b == sb && p->mode == mode && p->variant == c->mat_variant &&
            p->unit_work == c->mat_unit_work) {
            p->last_use = ++tick;
            return p;
        }
    return nullptr;
}

static int upload_plan(sdbfg_ctx* c, MatPlan* p, UnitBuilder& ub, const std::vector<uint32_t>& targets) {
    const std::vector<MatUnit> units = ub.sorted_units();
    p->nunits = (uint32_t)units.size();
    p->nsplit = (uint32_t)ub.split.size();
    p->nslots = ub.slots;
    p->filter_pairs = ub.filter_pairs;
    const auto up = [](uint64_t v) { return (v + 255) / 256 * 256; };
    const uint64_t at_targets = up(units.size() * sizeof(MatUnit)), at_refs = at_targets + up(targets.size() * 4),
                   at_split = at_refs + up(ub.refs.size() * 4), at_redo = at_split + up(ub.split.size() * sizeof(MatSplit)),
                   at_counter = at_redo + up(kRedoBytes);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CUDA_TRY(c, cudaStreamIsCapturing(c->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone)
        return fail(c, SDBFG_ERR_CUDA, "a comparison's first run cannot be captured");
    CUDA_TRY(c, c->must(p->d_all, at_counter + kMatCounterBytes + std::max<uint64_t>(1, ub.slots) * 8));
    uint8_t* d = p->d_all.as<uint8_t>();
    p->d_units.p = d;
    p->d_targets.p = d + at_targets;
    p->d_refs.p = d + at_refs;
    p->d_split.p = d + at_split;
    p->d_redo.p = d + at_redo;
    p->d_counter.p = d + at_counter;
    p->tables.resize(at_redo);
    const auto put = [&](uint64_t at, const void* src, uint64_t bytes) {
        if (bytes) memcpy(p->tables.data() + at, src, bytes);
    };
    put(0, units.data(), units.size() * sizeof(MatUnit));
    put(at_targets, targets.data(), targets.size() * 4);
    put(at_refs, ub.refs.data(), ub.refs.size() * 4);
    put(at_split, ub.split.data(), ub.split.size() * sizeof(MatSplit));
    if (at_redo) {
        // queued only: runs on this stream come behind it, and a change of the
        // stream waits for it (plan_tables_arrived)
        CUDA_TRY(c, cudaMemcpyAsync(d, p->tables.data(), at_redo, cudaMemcpyHostToDevice, c->stream));
        if (!c->ev_plan) CUDA_TRY(c, cudaEventCreateWithFlags(&c->ev_plan, cudaEventDisableTiming));
        CUDA_TRY(c, cudaEventRecord(c->ev_plan, c->stream));
        c->plan_tables_queued = true;
    }
    return SDBFG_OK;
}

cudaError_t plan_tables_arrived(sdbfg_ctx* c) {
    if (!c->plan_tables_queued) return cudaSuccess;
    // (the caller may be capturing another stream)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaError_t e = cudaEventSynchronize(c->ev_plan);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e == cudaSuccess) c->plan_tables_queued = false;
    return e;
}

// All pairs i<j of one set.  Digests sorted by filter count: a digest is the
// reference for every digest with more filters and for the equal-count digests
// the swap rule gives it.  Bundles of neighbours in that order take the digests
// behind their last class (of equal counts) as shared targets, a suffix of the
// sorted order; what a digest is the reference for before that suffix is an
// explicit list appended to the target list.
static int build_plan_all(sdbfg_ctx* c, const sdbfg_set* s, MatPlan* p) {
    const uint32_t n = s->n;
    std::vector<uint32_t> sorted(n);
    std::iota(sorted.begin(), sorted.end(), 0u);
    std::stable_sort(sorted.begin(), sorted.end(),
                     [&](uint32_t x, uint32_t y) { return s->bf_count[x] < s->bf_count[y]; });
    std::vector<uint32_t> targets(sorted);
    const auto count = [&](uint32_t k) { return s->bf_count[sorted[k]]; };
    std::vector<uint64_t> sum(n + 1, 0);          // filters of the first k digests
    std::vector<uint32_t> first(n), end(n + 1, n);  // a position's class [first, end)
    for (uint32_t k = 0; k < n; k++) {
        sum[k + 1] = sum[k] + count(k);
        first[k] = k && count(k) == count(k - 1) ? first[k - 1] : k;
    }
    for (uint32_t k = n; k-- > 0;) end[k] = k + 1 < n && count(k) == count(k + 1) ? end[k + 1] : k + 1;
    // A bundle is a class, or (tensor cores, whose passes cost 128 rows
    // whatever they fill) several small digests of neighbouring classes that
    // fit one pass together.  That saves passes over the suffix and costs
    // explicit pairs between the bundle's classes, a unit's start (about three
    // tiles) each: a class joins while the suffix is longer than that.
    // 400 digests of 1 to 2,000 filters: 8.57 ms by classes, 8.22 by bundles;
    // 200 of 2 to 1,300: 2.12 and 2.06 (the text they are read from included).
    const bool tc = c->mat_variant == kMatVariantTc;
    const uint64_t pad = tc ? (uint64_t)kMatVariantTable[c->mat_variant].rows : 1;
    const uint64_t start = 3ull * kMatVariantTable[c->mat_variant].tile;
    std::vector<uint32_t> cut;  // bundles [cut[i], cut[i + 1])
    for (uint32_t k = 0; k < n;) {
        cut.push_back(k);
        uint32_t e = end[k];
        if (tc && sum[e] - sum[k] <= pad) {
            uint64_t pairs = 0;  // explicit target filters between the classes
            while (e < n && sum[end[e]] - sum[k] <= pad && s->fast[sorted[e]] == s->fast[sorted[k]]) {
                const uint32_t f = end[e];
                pairs += (uint64_t)(e - k) * (sum[f] - sum[e]);
                if (pairs + start * (f - k) > sum[n] - sum[f]) break;
                e = f;
            }
        }
        k = e;
    }
    cut.push_back(n);
    // the job's work: every bundle (its rows packed) against the rest of the
    // sorted order, half of its own class
    const uint64_t ctas = (uint64_t)c->sms * matrix_ctas_per_sm(c->mat_variant);
    uint64_t total = 0;
    for (size_t i = 0; i + 1 < cut.size(); i++) {
        const uint64_t rows = sum[cut[i + 1]] - sum[cut[i]];
        total += (rows + pad - 1) / pad * pad * (sum[n] - sum[cut[i + 1]] + rows / 2);
    }
    UnitBuilder ub(effective_unit_budget(c->mat_unit_work, total, ctas, c->mat_variant), c->mat_variant);
    const auto nf = [&](uint32_t e) { return s->bf_count[targets[e]]; };
    const auto id = [&](uint32_t e) { return targets[e]; };
    const auto nf_ref = [&](uint32_t d) { return s->bf_count[d]; };
    for (size_t i = 0; i + 1 < cut.size(); i++) {
        const uint32_t k0 = cut[i], k1 = cut[i + 1];
        // every digest of the bundle is the reference of the whole suffix
        const std::vector<uint32_t> ids(sorted.begin() + k0, sorted.begin() + k1);
        ub.add_shared(ids, nf_ref, [&](uint32_t d) { return (uint32_t)s->fast[d]; }, 0u, k1, n, nf, id);
        // of the equal-count digests the swap rule gives it, and of the
        // bundle's later classes
        for (uint32_t k = k0; k < k1; k++) {
            const uint32_t a = sorted[k];
            const uint32_t own0 = (uint32_t)targets.size();
            for (uint32_t m = first[k]; m < end[k]; m++) {
                const uint32_t b = sorted[m];
                if (b == a) continue;
                const uint32_t lo = std::min(a, b), hi = std::max(a, b);
                const uint32_t ref = swaps(s, lo, s, hi) ? hi : lo;
                if (ref == a) targets.push_back(b);
            }
            targets.insert(targets.end(), sorted.begin() + end[k], sorted.begin() + k1);
            ub.add(a, s->bf_count[a], 0u, own0, (uint32_t)targets.size(), nf, id);
        }
    }
    p->nscores = (uint64_t)n * (n - 1) / 2;
    return upload_plan(c, p, ub, targets);
}

// Every query of set q against every target of set t (sdbf_score(q_i, t_j)).
static int build_plan_cross(sdbfg_ctx* c, const sdbfg_set* q, const sdbfg_set* t, MatPlan* p) {
    if ((uint64_t)q->n * t->n + q->n + t->n >= (1ull << 32))
        return fail(c, SDBFG_ERR_ARG, "compare_to: too many pairs for one plan");
    const uint64_t ctas = (uint64_t)c->sms * matrix_ctas_per_sm(c->mat_variant);
    UnitBuilder ub(effective_unit_budget(c->mat_unit_work, cross_work(q->total_filters, t->total_filters, c->mat_variant), ctas,
                                         c->mat_variant),
                   c->mat_variant);
    std::vector<uint32_t> targets;
    build_cross_units(
        ub, targets, q->n, t->n, [&](uint32_t i, uint32_t j) { return swaps(q, i, t, j); },
        [&](uint32_t i) { return q->bf_count[i]; }, [&](uint32_t j) { return t->bf_count[j]; },
        [&](uint32_t i) { return (uint32_t)q->fast[i]; }, [&](uint32_t j) { return (uint32_t)t->fast[j]; });
    p->nscores = (uint64_t)q->n * t->n;
    return upload_plan(c, p, ub, targets);
}

static int get_plan(sdbfg_ctx* c, const sdbfg_set* a, const sdbfg_set* b, uint32_t mode, MatPlan** out) {
    const uint64_t sb = b ? b->serial : 0;
    MatPlan* p = find_plan(c, a->serial, sb, mode);
    if (!p) {
        if (c->plans.size() >= 8) {  // drop the least recently used plan
            auto it = std::min_element(c->plans.begin(), c->plans.end(),
                                       [](MatPlan* x, MatPlan* y) { return x->last_use < y->last_use; });
            delete *it;
            c->plans.erase(it);
        }
        p = new MatPlan();
        p->serial_a = a->serial;
        p->serial_b = sb;
        p->mode = mode;
        p->variant = c->mat_variant;
        p->unit_work = c->mat_unit_work;
        const int rc = mode == kMatModeAll ? build_plan_all(c, a, p) : build_plan_cross(c, a, b, p);
        if (rc) {
            delete p;
            return rc;
        }
        c->plans.push_back(p);
        find_plan(c, a->serial, sb, mode);
    }
    *out = p;
    return SDBFG_OK;
}

static MatParams plan_params(sdbfg_ctx* c, const MatPlan* p, const sdbfg_set* a, const sdbfg_set* b,
                             int32_t* scores) {
    MatParams P{};
    const sdbfg_set* s1 = b ? b : a;
    P.filters[0] = a->d_filters.as<uint32_t>();
    P.meta[0] = a->d_meta.as<uint32_t>();
    P.digests[0] = a->d_digests.as<CmpDigest>();
    P.filters[1] = s1->d_filters.as<uint32_t>();
    P.meta[1] = s1->d_meta.as<uint32_t>();
    P.digests[1] = s1->d_digests.as<CmpDigest>();
    P.units = p->d_units.as<MatUnit>();
    P.nunits = p->nunits;
    P.next_unit = p->d_counter.as<uint32_t>();
    P.targets = p->d_targets.as<uint32_t>();
    P.refs = p->d_refs.as<uint32_t>();
    P.split = p->d_split.as<MatSplit>();
    P.nsplit = p->nsplit;
    P.slots = p->d_counter.as<double>() + kMatCounterBytes / 8;
    P.nslots = p->nslots;
    P.scores = scores;
    P.nscores = p->nscores;
    P.mode = p->mode;
    P.n = p->mode == kMatModeAll ? a->n : b->n;
    P.cutoffs = c->d_cut.as<uint16_t>();
    P.cutoffs64 = c->d_cut64.as<uint16_t>();
    P.redo = redo_list(p->d_redo.p, P.next_unit);
    P.error = p->d_counter.as<uint32_t>() + 1;
    P.gave_up = c->gave_up();
    P.phase = c->profile ? c->d_mphase.as<unsigned long long>() : nullptr;
    return P;
}

static int enqueue_plan(sdbfg_ctx* c, const MatPlan* p, const MatParams& P, cudaStream_t st) {
    const uint32_t grid = (uint32_t)(c->sms * matrix_ctas_per_sm(p->variant));
    uint64_t launched = 0;
    TIMED_LAUNCH_ON(c, "k_matrix", st, run_matrix(P, p->variant, grid, (uint32_t)c->sms, st, &launched));
    c->launches += launched - 1;  // one is counted with the timer
    return SDBFG_OK;
}

// Runs a plan on the context stream: launch by launch the first time (a
// capture costs more than it saves there), and through a CUDA graph once the
// output array is that of the run before.
static int run_plan(sdbfg_ctx* c, MatPlan* p, const sdbfg_set* a, const sdbfg_set* b, int32_t* dev_scores) {
    cudaStream_t st = c->stream;
    const MatParams P = plan_params(c, p, a, b, dev_scores);
    matrix_ctas_per_sm(p->variant);  // sets the kernel's attributes outside any capture
    if (!c->mat_graphs || c->profile) return enqueue_plan(c, p, P, st);
    if (p->graph_out != dev_scores) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        CUDA_TRY(c, cudaStreamIsCapturing(st, &cap));
        if (cap == cudaStreamCaptureStatusNone) {
            if (p->graph) cudaGraphExecDestroy(p->graph);
            p->graph = nullptr;
            p->graph_out = dev_scores;
            return enqueue_plan(c, p, P, st);
        }
    }
    const uint64_t kernels = p->variant == kMatVariantTc ? 3 : 1 + (P.nsplit ? 1 : 0), before = c->launches;
    if (p->graph && p->graph_out == dev_scores) {
        CUDA_TRY(c, cudaGraphLaunch(p->graph, st));
        c->launches += kernels;
        return SDBFG_OK;
    }
    if (p->graph) {
        cudaGraphExecDestroy(p->graph);
        p->graph = nullptr;
    }
    // capture on a private stream so a caller's stream in capture mode is not disturbed
    cudaStream_t cs;
    CUDA_TRY(c, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    int rc = SDBFG_OK;
    if (e == cudaSuccess) {
        rc = enqueue_plan(c, p, P, cs);
        e = cudaStreamEndCapture(cs, &g);
    }
    cudaStreamDestroy(cs);
    if (rc) return rc;
    c->launches = before;  // counted when the graph runs
    if (e == cudaSuccess) e = cudaGraphInstantiate(&p->graph, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(c, SDBFG_ERR_CUDA, "comparison graph: %s", cudaGetErrorString(e));
    p->graph_out = dev_scores;
    CUDA_TRY(c, cudaGraphLaunch(p->graph, st));
    c->launches += kernels;
    return SDBFG_OK;
}

// Copies a run's scores to out, waits, and reports a bounded wait that gave up.
static int fetch_scores(sdbfg_ctx* c, const MatPlan* p, int32_t* out) {
    uint32_t* err = static_cast<uint32_t*>(c->h_flags.p);  // pinned: this copy does not block
    CUDA_TRY(c, cudaMemcpyAsync(err, p->d_counter.as<uint32_t>() + 1, 4, cudaMemcpyDeviceToHost, c->stream));
    if (out) CUDA_TRY(c, cudaMemcpyAsync(out, c->d_scores.p, p->nscores * 4, cudaMemcpyDeviceToHost, c->stream));
    CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    if (*err) {
        *c->gave_up() = 0;  // reported here
        return fail(c, SDBFG_ERR_CUDA, "comparison kernel: %u CTAs gave up waiting for the tensor cores", *err);
    }
    return SDBFG_OK;
}

extern "C" int sdbfg_compare_all_device(sdbfg_ctx* c, const sdbfg_set* s, int32_t* dev_scores) {
    if (!c || !s || (!dev_scores && s->n > 1)) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (s->n < 2) return SDBFG_OK;
    MatPlan* p;
    int rc = get_plan(c, s, nullptr, kMatModeAll, &p);
    if (rc) return rc;
    return run_plan(c, p, s, nullptr, dev_scores);
}

extern "C" int sdbfg_compare_to_device(sdbfg_ctx* c, const sdbfg_set* q, const sdbfg_set* t, int32_t* dev_scores) {
    if (!c || !q || !t || (!dev_scores && q->n && t->n)) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (!q->n || !t->n) return SDBFG_OK;
    MatPlan* p;
    int rc = get_plan(c, q, t, kMatModeCross, &p);
    if (rc) return rc;
    return run_plan(c, p, q, t, dev_scores);
}

extern "C" int sdbfg_compare_all(sdbfg_ctx* c, const sdbfg_set* s, int32_t* out) {
    if (!c || !s || (!out && s->n > 1)) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (s->n < 2) return SDBFG_OK;
    MatPlan* p;
    int rc = get_plan(c, s, nullptr, kMatModeAll, &p);
    if (rc) return rc;
    CUDA_TRY(c, c->must(c->d_scores, p->nscores * 4));
    rc = run_plan(c, p, s, nullptr, c->d_scores.as<int32_t>());
    if (rc) return rc;
    return fetch_scores(c, p, out);
}

extern "C" int sdbfg_compare_to(sdbfg_ctx* c, const sdbfg_set* q, const sdbfg_set* t, int32_t* out) {
    if (!c || !q || !t || (!out && q->n && t->n)) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (!q->n || !t->n) return SDBFG_OK;
    MatPlan* p;
    int rc = get_plan(c, q, t, kMatModeCross, &p);
    if (rc) return rc;
    CUDA_TRY(c, c->must(c->d_scores, p->nscores * 4));
    rc = run_plan(c, p, q, t, c->d_scores.as<int32_t>());
    if (rc) return rc;
    return fetch_scores(c, p, out);
}

// scores (already queued into c->d_scores) -> matches on the host
static int collect_matches(sdbfg_ctx* c, uint64_t nscores, uint32_t mode, uint64_t dim, int32_t threshold,
                           sdbfg_match* out, uint64_t cap, uint64_t* count) {
    cudaStream_t st = c->stream;
    const uint64_t nb = (nscores + kMatchBlockScores - 1) / kMatchBlockScores;
    CUDA_TRY(c, c->must(c->d_match_counts, std::max<uint64_t>(1, nb) * 4));
    CUDA_TRY(c, c->must(c->d_match_offs, (nb + 1) * 8));
    const int32_t* sc = c->d_scores.as<int32_t>();
    TIMED_LAUNCH_ON(c, "k_match_count", st, launch_match_count(sc, nscores, threshold, c->d_match_counts.as<uint32_t>(), st));
    TIMED_LAUNCH_ON(c, "k_match_scan", st, launch_match_scan(c->d_match_counts.as<uint32_t>(), nb,
                                                             c->d_match_offs.as<uint64_t>(), st));
    uint64_t total = 0;
    CUDA_TRY(c, cudaMemcpyAsync(&total, c->d_match_offs.as<uint64_t>() + nb, 8, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(c, cudaStreamSynchronize(st));
    *count = total;
    if (total > cap) return fail(c, SDBFG_ERR_CAPACITY, "%llu matches, room for %llu", (unsigned long long)total,
                                 (unsigned long long)cap);
    if (!total) return SDBFG_OK;
    CUDA_TRY(c, c->must(c->d_matches, total * sizeof(sdbfg_match)));
    TIMED_LAUNCH_ON(c, "k_match_write", st, launch_match_write(sc, nscores, threshold, c->d_match_offs.as<uint64_t>(),
                                                               mode, dim, c->d_matches.as<uint32_t>(), total, st));
    CUDA_TRY(c, cudaMemcpyAsync(out, c->d_matches.p, total * sizeof(sdbfg_match), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(c, cudaStreamSynchronize(st));
    return SDBFG_OK;
}

extern "C" int sdbfg_compare_all_matches(sdbfg_ctx* c, const sdbfg_set* s, int32_t threshold, sdbfg_match* out,
                                         uint64_t cap, uint64_t* count) {
    if (!c || !s || !count || (cap && !out)) return SDBFG_ERR_ARG;
    *count = 0;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (s->n < 2) return SDBFG_OK;
    MatPlan* p;
    int rc = get_plan(c, s, nullptr, kMatModeAll, &p);
    if (rc) return rc;
    CUDA_TRY(c, c->must(c->d_scores, p->nscores * 4));
    rc = run_plan(c, p, s, nullptr, c->d_scores.as<int32_t>());
    if (rc) return rc;
    if ((rc = fetch_scores(c, p, nullptr))) return rc;
    return collect_matches(c, p->nscores, kMatModeAll, s->n, threshold, out, cap, count);
}

extern "C" int sdbfg_compare_to_matches(sdbfg_ctx* c, const sdbfg_set* q, const sdbfg_set* t, int32_t threshold,
                                        sdbfg_match* out, uint64_t cap, uint64_t* count) {
    if (!c || !q || !t || !count || (cap && !out)) return SDBFG_ERR_ARG;
    *count = 0;
    CUDA_TRY(c, cudaSetDevice(c->device));
    if (!q->n || !t->n) return SDBFG_OK;
    MatPlan* p;
    int rc = get_plan(c, q, t, kMatModeCross, &p);
    if (rc) return rc;
    CUDA_TRY(c, c->must(c->d_scores, p->nscores * 4));
    rc = run_plan(c, p, q, t, c->d_scores.as<int32_t>());
    if (rc) return rc;
    if ((rc = fetch_scores(c, p, nullptr))) return rc;
    return collect_matches(c, p->nscores, kMatModeCross, t->n, threshold, out, cap, count);
}

extern "C" int sdbfg_ctx_set_compare_tuning(sdbfg_ctx* c, int variant, uint64_t unit_work, int use_graphs) {
    if (!c || variant < 0 || variant >= kMatVariants || unit_work == 0) return SDBFG_ERR_ARG;
    c->mat_variant = variant;
    c->mat_unit_work = unit_work;
    c->mat_graphs = use_graphs != 0;
    return SDBFG_OK;
}

extern "C" int sdbfg_ctx_get_compare_tuning(const sdbfg_ctx* c, int* variant, uint64_t* unit_work) {
    if (!c) return SDBFG_ERR_ARG;
    if (variant) *variant = c->mat_variant;
    if (unit_work) *unit_work = c->mat_unit_work;
    return SDBFG_OK;
}

extern "C" uint64_t sdbfg_compare_filter_pairs(sdbfg_ctx* c, const sdbfg_set* a, const sdbfg_set* b) {
    if (!c || !a || cudaSetDevice(c->device) != cudaSuccess) return 0;
    MatPlan* p;
    if (get_plan(c, a, b, b ? kMatModeCross : kMatModeAll, &p)) return 0;
    return p->filter_pairs;
}

// Times every kernel variant and unit budget on a sample of the plan's units
// (every k-th unit, about `sample_pairs` filter pairs) and keeps the fastest.
extern "C" int sdbfg_compare_autotune(sdbfg_ctx* c, const sdbfg_set* a, const sdbfg_set* b, uint64_t sample_pairs,
                                      int* out_variant, uint64_t* out_unit_work, double* out_rate) {
    if (!c || !a) return SDBFG_ERR_ARG;
    CUDA_TRY(c, cudaSetDevice(c->device));
    const uint32_t mode = b ? kMatModeCross : kMatModeAll;
    const uint64_t budgets[3] = {1ull << 20, 1ull << 22, 1ull << 24};
    const int saved_v = c->mat_variant;
    const uint64_t saved_w = c->mat_unit_work;
    int best_v = saved_v;
    uint64_t best_w = saved_w;
    double best_rate = -1;
    cudaEvent_t e0, e1;
    CUDA_TRY(c, cudaEventCreate(&e0));
    CUDA_TRY(c, cudaEventCreate(&e1));
    for (uint64_t w : budgets) {
        for (int v = 0; v < kMatVariants; v++) {
            c->mat_variant = v;
            c->mat_unit_work = w;
            MatPlan* p;
            int rc = get_plan(c, a, b, mode, &p);
            if (rc) return rc;
            // sampled unit list: every k-th unit (the plan is sorted largest first)
            // (from the host's tables: their copy to the device may still be queued)
            const MatUnit* units = reinterpret_cast<const MatUnit*>(p->tables.data());
            const uint32_t* targets = reinterpret_cast<const uint32_t*>(
                p->tables.data() + (static_cast<const uint8_t*>(p->d_targets.p) - p->d_all.as<uint8_t>()));
            const uint64_t avg = std::max<uint64_t>(1, p->filter_pairs / std::max<uint32_t>(1, p->nunits));
            const uint64_t want = std::max<uint64_t>(1, sample_pairs / avg);
            const uint64_t step = std::max<uint64_t>(1, p->nunits / want);
            std::vector<MatUnit> sample;
            for (uint64_t k = 0; k < p->nunits; k += step)
                if (!(units[k].flags & kUnitSplit)) sample.push_back(units[k]);
            if (sample.empty()) continue;
            uint64_t pairs = 0;
            DevBuf d_sample;
            CUDA_TRY(c, c->must(d_sample, sample.size() * sizeof(MatUnit)));
            CUDA_TRY(c, cudaMemcpy(d_sample.p, sample.data(), sample.size() * sizeof(MatUnit), cudaMemcpyHostToDevice));
            CUDA_TRY(c, c->must(c->d_scores, p->nscores * 4));
            MatParams P = plan_params(c, p, a, b, c->d_scores.as<int32_t>());
            P.units = d_sample.as<MatUnit>();
            P.nunits = (uint32_t)sample.size();
            P.nsplit = 0;
            {
                // count filter pairs of the sample from the target list
                const sdbfg_set* ts_all = b ? b : a;
                for (const MatUnit& u : sample) {
                    const sdbfg_set* tset = (u.flags & kUnitTgtSide1) ? ts_all : a;
                    for (uint32_t e = u.t0; e < u.t1; e++) pairs += (uint64_t)(u.r1 - u.r0) * tset->bf_count[targets[e]];
                }
            }
            cudaStream_t st = c->stream;
            float best_ms = 1e30f;
            for (int rep = 0; rep < 2; rep++) {
                CUDA_TRY(c, cudaMemsetAsync(p->d_counter.p, 0, kMatCounterBytes, st));
                CUDA_TRY(c, cudaEventRecord(e0, st));
                const uint32_t grid = (uint32_t)(c->sms * matrix_ctas_per_sm(v));
                CUDA_TRY(c, launch_matrix(P, v, std::max(1u, std::min(grid, P.nunits)), st));
                CUDA_TRY(c, cudaEventRecord(e1, st));
                CUDA_TRY(c, cudaEventSynchronize(e1));
                float ms = 0;
                CUDA_TRY(c, cudaEventElapsedTime(&ms, e0, e1));
                best_ms = std::min(best_ms, ms);
            }
            d_sample.release();
            const double rate = pairs / (best_ms * 1e-3);
            if (rate > best_rate) {
                best_rate = rate;
                best_v = v;
                best_w = w;
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    c->mat_variant = best_v;
    c->mat_unit_work = best_w;
    (void)saved_v;
    (void)saved_w;
    if (out_variant) *out_variant = best_v;
    if (out_unit_work) *out_unit_work = best_w;
    if (out_rate) *out_rate = best_rate;
    return SDBFG_OK;
}
