// compare_device.cuh -- device helpers shared by the comparison kernels
// (compare_kernels.cu: CUDA-core paths, matrix_tc.cu: tensor-core path).
#pragma once
#include <cstdint>

#include "compare_kernels.h"

namespace sdbfg {

__device__ __forceinline__ uint32_t cut_for(const uint16_t* cut_sum, const uint16_t* cut256, uint32_t s1,
                                            uint32_t s2) {
    const uint32_t sum = s1 + s2;
    return sum < 1024 ? cut_sum[sum] : cut256[4096u / sum];
}

// A filter's maximum against one target as the reference's double:
// -1 when no target filter has >= 16 elements, else num / den (den is the
// reference's uint32 max_est - cut, which wraps when the hamming weights do
// not describe the compared bits -- mixed --fast comparisons).
__device__ __forceinline__ double max_value(bool active, uint32_t bnum, uint32_t bden, bool counted) {
    if (!active) return 0.0;
    if (!counted) return -1.0;
    return bnum == 0 ? 0.0 : __ddiv_rn((double)bnum, (double)bden);
}

__device__ __forceinline__ uint64_t out_index(const MatParams& P, bool ref_side1, uint32_t ref, uint32_t tgt) {
    if (P.mode == kMatModeAll) {
        const uint64_t i = min(ref, tgt), j = max(ref, tgt);
        return i * (2ull * P.n - i - 1) / 2 + (j - i - 1);
    }
    const uint64_t q = ref_side1 ? tgt : ref, t = ref_side1 ? ref : tgt;
    return q * P.n + t;
}

__device__ __forceinline__ int32_t final_score(double sum, uint32_t n1, uint32_t sparse) {
    uint64_t denom = n1;
    if (n1 > 1) denom -= sparse;
    if (denom == 0 || sum < 0) return -1;
    return (int32_t)floor(__dadd_rn(__ddiv_rn(__dmul_rn(100.0, sum), (double)denom), 0.5));
}

// Marks of scores that only the ordered sum in double precision decides: the
// reference digest is the pair's first (-2) or second (-3) digest.
constexpr int32_t kScoreRedoFirst = -2, kScoreRedoSecond = -3;

// The score of (ref, tgt) from the sum of its row maxima in units of 2^-23
// (each within two units; bit 63: left to exact arithmetic), or a mark.
// score = floor(100 sum / denom + 0.5); the reference's sum in double
// precision differs from the true one by far less than the rows' units do,
// so the score is its score unless 100 sum / denom + 0.5 is closer to a whole
// number than that.  A target without a filter of 16 elements gives every
// active row -1 and every other row 0: the running sum is then -1 after an
// active row and 0 after another one, so the last row decides.
__device__ __forceinline__ int32_t fixed_score(const MatParams& P, uint32_t rs, uint32_t ref, uint32_t ts,
                                               uint32_t tgt, unsigned long long sum) {
    const CmpDigest A = P.digests[rs][ref], B = P.digests[ts][tgt];
    const uint64_t denom = A.nfilters > 1 ? A.nfilters - A.sparse : A.nfilters;
    if (denom == 0) return -1;
    if (B.sparse == B.nfilters) return A.flags & kDigestLastActive ? -1 : 0;
    const bool second = P.mode == kMatModeAll ? ref > tgt : rs != 0;
    const int32_t redo = second ? kScoreRedoSecond : kScoreRedoFirst;
    if (sum >> 63) return redo;
    if (sum == 0) return 0;
    const uint64_t one = denom << 24;  // a score of 1 in the units of t
    const uint64_t t = 200ull * sum + (denom << 23);
    const uint64_t score = t / one, rem = t - score * one;
    const uint64_t tol = 400ull * denom;
    return rem < tol || one - rem <= tol ? redo : (int32_t)score;
}


}  // namespace sdbfg
