// launch_rules.h -- rules of the host side that decide which kernel a call may take, in plain C++ (no
// CUDA), so that they can be checked at sizes no test machine holds.
#pragma once

#include <limits.h>

namespace pasc {

// The mixed FEM-SUM kernels (fem.cu) index timesteps as int, a thread past the end included, and
// coarse entries as unsigned int: signals within these limits.  Larger ones take the general
// reduction and prolongation, which index in 64 bits (T1 of 2^31 at K = 1 is about 100 GB of state,
// so such signals exist).
constexpr long FEM_SUM_THREADS = 256;  // a block's
inline bool fem_sum_indexable(long T1, long T2, int K)
{
    return T2 >= 1 && T2 <= T1 && T1 <= (long)INT_MAX - FEM_SUM_THREADS &&
           T2 <= ((long)UINT_MAX - FEM_SUM_THREADS) / K;
}

// Tags of the words that the blocks of a cooperative launch exchange (grid_words.cuh).  A word is valid
// when it carries the sweep's tag, so no tag may come twice while a word of its first use may still lie
// in the buffer (a plan with more blocks leaves words that a smaller one never writes), and cleared
// words carry tag 0, which is never used.  take gives a launch the tags first .. first + n - 1, and
// says whether the buffer has to be cleared before it: once in 2^32 tags.
struct WordTags {
    unsigned int next = 1;
    bool take(unsigned int n, unsigned int *first)
    {
        const bool wrap = n > UINT_MAX - next;
        if (wrap) next = 1;
        *first = next;
        next += n;
        return wrap;
    }
};

}  // namespace pasc
