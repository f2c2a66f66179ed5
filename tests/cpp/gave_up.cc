// k_matrix_finish after a comparison kernel that gave up: every score is
// invalid and the host's word is set; without an error the scores stay.
#include <climits>
#include <cstdio>
#include <vector>

#include <cuda_runtime.h>

#include "../../sdhash_gb300/csrc/compare_kernels.h"

namespace sdbfg {
void k_matrix_finish(MatParams);  // (the kernel's host symbol)
}

#define REQUIRE(c)                                                  \
    do {                                                            \
        if (!(c)) {                                                 \
            fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #c); \
            return 1;                                               \
        }                                                           \
    } while (0)

int main() {
    constexpr size_t kScores = 5000, kCutoffs = 64 << 10;
    uint8_t* mem = nullptr;
    uint32_t* word = nullptr;
    REQUIRE(cudaMalloc(&mem, kScores * 4 + 256 + kCutoffs) == cudaSuccess);
    REQUIRE(cudaMallocHost(&word, 64) == cudaSuccess);
    REQUIRE(cudaMemset(mem, 0, kScores * 4 + 256 + kCutoffs) == cudaSuccess);
    std::vector<int32_t> start(kScores + 1), got(kScores + 1);
    for (size_t k = 0; k <= kScores; k++) start[k] = (int32_t)(k * 7919 % (1u << 30));  // sums of units left undone
    for (const uint32_t error : {0u, 3u}) {
        sdbfg::MatParams P{};
        P.scores = reinterpret_cast<int32_t*>(mem);
        P.nscores = kScores;
        uint32_t* counters = reinterpret_cast<uint32_t*>(mem + kScores * 4 + 64);
        P.next_unit = counters;
        P.error = counters + 1;
        P.redo = sdbfg::redo_list(mem, counters);  // (no entry is written: nothing is marked)
        P.gave_up = word;
        P.mode = sdbfg::kMatModeAll;
        P.n = 100;
        P.cutoffs = P.cutoffs64 = reinterpret_cast<uint16_t*>(mem + kScores * 4 + 256);
        word[0] = word[1] = 0;
        REQUIRE(cudaMemcpy(mem, start.data(), kScores * 4 + 4, cudaMemcpyHostToDevice) == cudaSuccess);
        REQUIRE(cudaMemcpy(P.error, &error, 4, cudaMemcpyHostToDevice) == cudaSuccess);
        void* args[] = {&P};
        REQUIRE(cudaLaunchKernel(reinterpret_cast<const void*>(sdbfg::k_matrix_finish), dim3(7), dim3(sdbfg::kCmpThreads), args,
                                 0, nullptr) == cudaSuccess);
        REQUIRE(cudaDeviceSynchronize() == cudaSuccess);
        REQUIRE(cudaMemcpy(got.data(), mem, kScores * 4 + 4, cudaMemcpyDeviceToHost) == cudaSuccess);
        for (size_t k = 0; k < kScores; k++) REQUIRE(got[k] == (error ? INT32_MIN : start[k]));
        REQUIRE(got[kScores] == start[kScores]);
        REQUIRE(word[0] == (error ? 1u : 0u) && word[1] == 0);
    }
    return 0;
}
