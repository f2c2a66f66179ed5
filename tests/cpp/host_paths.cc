// Cases of the library's host code against fake_cuda.h: one per run, by name.
// Exit status 0: the case holds.
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "../../include/sdbf_gb300.h"
#include "../../sdhash_gb300/csrc/compare_kernels.h"
#include "../../sdhash_gb300/csrc/gen_kernels.h"
#include "fake_cuda.h"

#define REQUIRE(c)                                                      \
    do {                                                                \
        if (!(c)) {                                                     \
            fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c);     \
            exit(1);                                                    \
        }                                                               \
    } while (0)

namespace {

sdbfg_ctx* context(int device = 0) {
    sdbfg_ctx* c = nullptr;
    REQUIRE(sdbfg_ctx_create(device, &c) == SDBFG_OK);
    return c;
}

// n digests of 1, 2, 3, ... filters
sdbfg_set* digests(sdbfg_ctx* c, uint32_t n) {
    std::vector<uint8_t> filters(n * 256);
    for (size_t i = 0; i < filters.size(); i++) filters[i] = (uint8_t)(i * 2654435761u >> 13);
    std::vector<sdbfg_digest_desc> ds(n);
    for (uint32_t i = 0; i < n; i++) {
        ds[i] = {};
        ds[i].name = "d";
        ds[i].filters = filters.data();
        ds[i].bf_count = i + 1;
        ds[i].last_count = ds[i].max_elem = 160;
        ds[i].orig_size = 4096;
    }
    sdbfg_set* s = nullptr;
    REQUIRE(sdbfg_set_upload(c, ds.data(), n, &s) == SDBFG_OK);
    return s;
}

template <class T>
T* device_array(size_t n) {
    void* p = nullptr;
    REQUIRE(cudaMalloc(&p, n * sizeof(T)) == cudaSuccess);
    return static_cast<T*>(p);
}

uint8_t* host_array(size_t n) {  // (never touched as a whole)
    void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    REQUIRE(p != MAP_FAILED);
    return static_cast<uint8_t*>(p);
}

// every comparison kernel that runs has its units and targets
int matrix_runs = 0;
void expect_tables() {
    fake::on_launch("k_matrix", [](void** args) {
        const sdbfg::MatParams P = *static_cast<sdbfg::MatParams*>(args[0]);
        return [P] {
            matrix_runs++;
            uint32_t poison;
            memset(&poison, fake::kPoison, 4);
            for (uint32_t u = 0; u < P.nunits; u++) {
                REQUIRE(P.units[u].ref != poison && P.units[u].t1 != poison);
                for (uint32_t t = P.units[u].t0; t < P.units[u].t1; t++) REQUIRE(P.targets[t] != poison);
            }
        };
    });
}

// a plan's tables reach the device before a comparison on another stream than
// the one it was made under
void plan_other_stream(bool first_compared) {
    sdbfg_ctx* c = context();
    sdbfg_set* s = digests(c, 40);
    int32_t* out = device_array<int32_t>(2 * 780);
    expect_tables();
    cudaStream_t a, b;
    cudaStreamCreateWithFlags(&a, cudaStreamNonBlocking);
    cudaStreamCreateWithFlags(&b, cudaStreamNonBlocking);
    REQUIRE(sdbfg_ctx_set_stream(c, a) == SDBFG_OK);
    if (first_compared) REQUIRE(sdbfg_compare_all_device(c, s, out) == SDBFG_OK);
    else REQUIRE(sdbfg_compare_filter_pairs(c, s, nullptr) > 0);
    REQUIRE(sdbfg_ctx_set_stream(c, b) == SDBFG_OK);
    REQUIRE(sdbfg_compare_all_device(c, s, out + 780) == SDBFG_OK);
    cudaStreamSynchronize(b);
    REQUIRE(matrix_runs > 0);
    sdbfg_set_free(s);
    sdbfg_ctx_destroy(c);
}

// the tuner samples a plan's units as they are
void autotune() {
    sdbfg_ctx* c = context();
    sdbfg_set* s = digests(c, 40);
    expect_tables();
    REQUIRE(sdbfg_compare_autotune(c, s, nullptr, 1 << 20, nullptr, nullptr, nullptr) == SDBFG_OK);
    REQUIRE(matrix_runs > 0);
    sdbfg_set_free(s);
    sdbfg_ctx_destroy(c);
}

// a stream batch reads its inputs and nothing behind them
void copies_end_with_the_input() {
    sdbfg_ctx* c = context();
    const std::vector<std::vector<uint64_t>> batches = {{1001}, {512}, {70'001}, {4096, 513}, {1040, 700, 1003}};
    for (const bool page_locked : {false, true})
        for (uint64_t shift = 0; shift < 16; shift += 3)
            for (const auto& lens : batches) {
                std::vector<uint64_t> offs;
                uint64_t end = shift;
                for (uint64_t n : lens) {  // each 16-byte aligned to the first: one contiguous range
                    end = (end - shift + 15) / 16 * 16 + shift;
                    offs.push_back(end);
                    end += n;
                }
                void* p = nullptr;
                if (page_locked) REQUIRE(cudaMallocHost(&p, end) == cudaSuccess);
                else p = malloc(end);
                const uint8_t* data = static_cast<uint8_t*>(p);
                const uint64_t cap = sdbfg_digest_capacity(lens.data(), (uint32_t)lens.size(), 0);
                std::vector<uint8_t> out(cap * 256);
                std::vector<sdbfg_digest_result> res(lens.size());
                fake::copies.clear();
                REQUIRE(sdbfg_digest_batch(c, data, offs.data(), lens.data(), (uint32_t)lens.size(), 0, out.data(), cap,
                                           nullptr, res.data()) == SDBFG_OK);
                for (const fake::Copy& k : fake::copies) {
                    const uint8_t* s = static_cast<const uint8_t*>(k.src);
                    if (k.kind == cudaMemcpyHostToDevice && s >= data && s < data + end) REQUIRE(s + k.bytes <= data + end);
                }
                if (page_locked) cudaFreeHost(p);
                else free(p);
            }
    sdbfg_ctx_destroy(c);
}

// every kernel can be launched on each device of a process (fake_cuda refuses
// more than 48 KB of dynamic shared memory on a device it was not asked for on)
void second_device() {
    std::vector<uint8_t> data(4 << 20), index(1 << 16);
    for (size_t i = 0; i < data.size(); i++) data[i] = (uint8_t)(i * i >> 7);
    for (int device = 0; device < 3; device++) {
        sdbfg_ctx* c = context(device);
        fake::launches.clear();
        const std::vector<std::vector<uint64_t>> batches = {{4 << 20}, {1 << 20, 1 << 20, 70'000}};
        for (const auto& lens : batches)
            for (const uint32_t dd : {0u, 4096u, 1001u}) {
                std::vector<uint64_t> offs(lens.size(), 0);
                for (size_t i = 1; i < lens.size(); i++) offs[i] = offs[i - 1] + lens[i - 1];
                const uint32_t n = (uint32_t)lens.size();
                const uint64_t cap = sdbfg_digest_capacity(lens.data(), n, dd);
                std::vector<uint8_t> out(cap * 256);
                std::vector<uint16_t> counts(cap);
                std::vector<sdbfg_digest_result> res(n);
                uint64_t added = 0;
                REQUIRE(sdbfg_digest_batch(c, data.data(), offs.data(), lens.data(), n, dd, out.data(), cap, counts.data(),
                                           res.data()) == SDBFG_OK);
                REQUIRE(sdbfg_digest_batch_index(c, data.data(), offs.data(), lens.data(), n, dd, out.data(), cap,
                                                 counts.data(), res.data(), index.data(), index.size(), &added) == SDBFG_OK);
            }
        sdbfg_set* s = digests(c, 40);
        std::vector<int32_t> scores(780);
        for (int variant = 0; variant < 6; variant++) {
            REQUIRE(sdbfg_ctx_set_compare_tuning(c, variant, 1 << 22, 1) == SDBFG_OK);
            REQUIRE(sdbfg_compare_all(c, s, scores.data()) == SDBFG_OK);
        }
        REQUIRE(fake::launched("k_stream_chain(") && fake::launched("k_stream_commit(") &&
                fake::launched("k_stream_commit_round(") && fake::launched("k_block_digest<true>") &&
                fake::launched("k_block_digest<false>") && fake::launched("k_matrix_tc<false>"));
        for (const fake::Launch& l : fake::launches) REQUIRE(l.device == device);
        sdbfg_set_free(s);
        sdbfg_ctx_destroy(c);
    }
}

// precomputed ranks are addressed in 32 bits of eight ranks: of an input
// above 32 GiB they are not used
void ranks_of_a_huge_input() {
    for (const bool huge : {false, true}) {
        sdbfg_ctx* c = context();
        const std::vector<uint64_t> lens = huge ? std::vector<uint64_t>{(33ull << 30) + 5, 1 << 20} : std::vector<uint64_t>{31ull << 30, 1 << 20};
        const std::vector<uint64_t> offs = {0, 34ull << 30};
        uint8_t* data = device_array<uint8_t>(35ull << 30);
        const uint64_t cap = sdbfg_digest_capacity(lens.data(), 2, 0);
        uint8_t* out = device_array<uint8_t>(cap * 256);
        sdbfg_digest_result res[2];
        static uint64_t ranked, wrapped;
        ranked = wrapped = 0;
        fake::launches.clear();
        fake::on_launch("k_stream_ranks", [](void** args) {
            const sdbfg::GenParams P = *static_cast<sdbfg::GenParams*>(args[0]);
            return [P] {  // every chunk's ranks lie behind those of the chunk before
                for (uint32_t k = 1; k < P.nchunks; k++)
                    wrapped += P.chunks[k].rank_off8 != P.chunks[k - 1].rank_off8 + (P.chunks[k - 1].n + 7) / 8 ||
                               P.chunks[k].rank_off8 < P.chunks[k - 1].rank_off8;
                ranked++;
            };
        });
        REQUIRE(sdbfg_digest_batch_device(c, data, offs.data(), lens.data(), 2, 0, out, cap, nullptr, res) == SDBFG_OK);
        REQUIRE(fake::launched("k_stream_tiles"));
        REQUIRE(wrapped == 0);
        REQUIRE(huge || ranked > 0);
        sdbfg_ctx_destroy(c);
        cudaFree(data);
        cudaFree(out);
    }
}

// a comparison whose kernel gave up (an error word that the kernel sets) is
// reported once: by the calls that wait, else by the next synchronisation
void comparison_gave_up() {
    sdbfg_ctx* c = context();
    sdbfg_set* s = digests(c, 40);
    int32_t* out = device_array<int32_t>(780);
    std::vector<int32_t> scores(780);
    static bool fails = true;
    fake::on_launch("k_matrix_tc", [](void** args) {
        const sdbfg::MatParams P = *static_cast<sdbfg::MatParams*>(args[0]);
        return [P] { *P.error = fails; };
    });
    fake::on_launch("k_matrix_finish", [](void** args) {  // (the kernel's part of it: test_gpu_gave_up.py)
        const sdbfg::MatParams P = *static_cast<sdbfg::MatParams*>(args[0]);
        return [P] {
            if (*P.error && P.gave_up) *P.gave_up = 1;
        };
    });
    for (int k = 0; k < 3; k++) {  // launched, launched, from the graph
        REQUIRE(sdbfg_compare_all_device(c, s, out) == SDBFG_OK);
        REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_ERR_CUDA);
        REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_OK);
    }
    REQUIRE(sdbfg_compare_to_device(c, s, s, device_array<int32_t>(1600)) == SDBFG_OK);
    REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_ERR_CUDA);
    REQUIRE(sdbfg_compare_all(c, s, scores.data()) == SDBFG_ERR_CUDA);
    REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_OK);
    fails = false;
    REQUIRE(sdbfg_compare_all_device(c, s, out) == SDBFG_OK);
    REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_OK);
    REQUIRE(sdbfg_compare_all(c, s, scores.data()) == SDBFG_OK);
    sdbfg_set_free(s);
    sdbfg_ctx_destroy(c);
}

// a served batch whose kernel gave up comes back with an error for each of
// its queries, and the next one is served
void server_batch_gave_up() {
    sdbfg_ctx* c = context();
    sdbfg_set* s = digests(c, 10);
    static int runs = 0;
    fake::on_launch("k_matrix_tc", [](void** args) {
        const sdbfg::MatParams P = *static_cast<sdbfg::MatParams*>(args[0]);
        return [P] { *P.error = runs++ < 1; };
    });
    fake::on_launch("k_matrix_finish", [](void** args) {  // (the kernel's part of it: test_gpu_gave_up.py)
        const sdbfg::MatParams P = *static_cast<sdbfg::MatParams*>(args[0]);
        return [P] {
            if (*P.error && P.gave_up) *P.gave_up = 1;
            const int32_t score = *P.error ? SDBFG_SCORE_INVALID : 7;
            for (uint64_t k = 0; k < P.nscores; k++) P.scores[k] = score;
        };
    });
    const sdbfg_server_config cfg{1, 4, 8ull << 20, 1, 0, 0};
    sdbfg_server* srv = nullptr;
    REQUIRE(sdbfg_server_create(c, s, &cfg, &srv) == SDBFG_OK);
    const std::vector<uint8_t> filter(256, 0x11);
    sdbfg_digest_desc q{};
    q.name = "q";
    q.filters = filter.data();
    q.bf_count = 1;
    q.last_count = q.max_elem = 160;
    for (uint64_t tag = 0; tag < 2; tag++) {
        REQUIRE(sdbfg_server_submit(srv, &q, tag) == SDBFG_OK);
        sdbfg_server_result r{};
        std::vector<int32_t> row(10);
        uint32_t n = 0;
        REQUIRE(sdbfg_server_poll(srv, &r, row.data(), 1, &n, 10'000) == SDBFG_OK);
        REQUIRE(n == 1 && r.tag == tag);
        REQUIRE(r.status == (tag ? SDBFG_OK : SDBFG_ERR_CUDA));
        REQUIRE(r.best_score == (tag ? 7 : -1) && r.matches == (tag ? 10u : 0u));
        for (int32_t v : row) REQUIRE(v == (tag ? 7 : SDBFG_SCORE_INVALID));
    }
    sdbfg_server_destroy(srv);
    REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_OK);  // the server's runs are not the context's
    sdbfg_set_free(s);
    sdbfg_ctx_destroy(c);
}

// where device memory is short, what earlier calls left for later ones (the
// links of a large file, the staging copy of a pageable batch) makes room
void room_is_made() {
    const auto limit_to = [](uint64_t more) {
        size_t free_ = 0, total = 0;
        fake::memory_limit = 1ull << 40;
        cudaMemGetInfo(&free_, &total);
        fake::memory_limit = total - free_ + more;
    };
    constexpr uint64_t kGiB = 1ull << 30, kMiB = 1ull << 20;
    fake::reads_pageable = true;
    const uint64_t len = kGiB, off = 0, cap = sdbfg_digest_capacity(&len, 1, 0);
    uint8_t* file = device_array<uint8_t>(len);
    uint8_t* filters = device_array<uint8_t>(cap * 256);
    uint8_t* data = host_array(3 * kGiB);
    uint8_t* out = host_array(cap * 3 * 256);
    std::vector<uint16_t> counts(3 * kGiB / 4096);
    std::vector<int32_t> scores(499'500);
    const std::vector<uint64_t> lens(12, kGiB / 4);
    std::vector<uint64_t> offs(12);
    for (size_t i = 0; i < offs.size(); i++) offs[i] = i * (kGiB / 4);
    std::vector<sdbfg_digest_result> res(12);
    for (const bool staging : {false, true}) {
        // each call on a context of its own, which the call before filled
        for (int call = 0; call < 4; call++) {
            fake::memory_limit = 1ull << 40;
            sdbfg_ctx* c = context();
            sdbfg_set* s = call == 2 ? digests(c, 1000) : nullptr;
            if (staging)
                REQUIRE(sdbfg_digest_batch(c, data, offs.data(), lens.data(), 12, 0, out, 3 * cap, nullptr, res.data()) == SDBFG_OK);
            else
                REQUIRE(sdbfg_digest_batch_device(c, file, &off, &len, 1, 0, filters, cap, nullptr, res.data()) == SDBFG_OK);
            REQUIRE(fake::launched(staging ? "k_stage_gather" : "k_stream_chain"));
            limit_to(call == 2 ? 1 * kMiB : 64 * kMiB);
            if (call == 0) s = digests(c, 1000);  // 128 MB of filters
            if (call == 1)
                REQUIRE(sdbfg_digest_batch(c, data, &off, &len, 1, 4096, out, cap, counts.data(), res.data()) == SDBFG_OK);
            if (call == 2) REQUIRE(sdbfg_compare_all(c, s, scores.data()) == SDBFG_OK);
            if (call == 3) {
                const std::vector<uint64_t> small(1000, 300'000);
                std::vector<uint64_t> at(1000);
                for (size_t i = 0; i < at.size(); i++) at[i] = i * 300'000;
                std::vector<sdbfg_digest_result> r(1000);
                const uint64_t room = sdbfg_digest_capacity(small.data(), 1000, 0);
                std::vector<uint8_t> f(room * 256), bits(16 << 20);
                uint64_t added = 0;
                REQUIRE(sdbfg_digest_batch_index(c, data, at.data(), small.data(), 1000, 0, f.data(), room, nullptr, r.data(),
                                                 bits.data(), bits.size(), &added) == SDBFG_OK);
            }
            if (s) sdbfg_set_free(s);
            sdbfg_ctx_destroy(c);
        }
    }
}

// a context's memory is on its own device, whichever device is current when it
// is called
void other_device_current() {
    sdbfg_ctx* c = context(1);
    sdbfg_set* s = digests(c, 40);
    int32_t* out = device_array<int32_t>(780);
    static int runs = 0;
    fake::on_launch("k_matrix", [](void** args) {
        const sdbfg::MatParams P = *static_cast<sdbfg::MatParams*>(args[0]);
        return [P] {
            runs++;
            REQUIRE(fake::device_of(P.units) == 1 && fake::device_of(P.filters[0]) == 1);
            REQUIRE(!P.phase || fake::device_of(P.phase) == 1);
        };
    });
    cudaSetDevice(0);
    REQUIRE(sdbfg_compare_filter_pairs(c, s, nullptr) > 0);
    REQUIRE(sdbfg_compare_all_device(c, s, out) == SDBFG_OK);
    cudaSetDevice(0);
    REQUIRE(sdbfg_ctx_profile(c, 1) == SDBFG_OK);
    REQUIRE(sdbfg_compare_all_device(c, s, out) == SDBFG_OK);
    REQUIRE(sdbfg_ctx_synchronize(c) == SDBFG_OK);
    REQUIRE(runs > 0);
    sdbfg_set_free(s);
    sdbfg_ctx_destroy(c);
}

const std::map<std::string, std::function<void()>> kCases = {
    {"plan_other_stream", [] { plan_other_stream(false); }},
    {"plan_other_stream_compared", [] { plan_other_stream(true); }},
    {"autotune", autotune},
    {"copies_end_with_the_input", copies_end_with_the_input},
    {"second_device", second_device},
    {"ranks_of_a_huge_input", ranks_of_a_huge_input},
    {"comparison_gave_up", comparison_gave_up},
    {"server_batch_gave_up", server_batch_gave_up},
    {"room_is_made", room_is_made},
    {"other_device_current", other_device_current},
};

}  // namespace

int main(int argc, char** argv) {
    const auto it = argc > 1 ? kCases.find(argv[1]) : kCases.end();
    REQUIRE(it != kCases.end());
    it->second();
    return 0;
}
