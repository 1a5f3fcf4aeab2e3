// tc_words.h -- walking the words of a row.
//
// A matrix holds up to 2^31 - 1 words, so the position a strided loop steps to
// past the end of a row near the last word does not fit an int: it would come
// out negative, compare as before the end, and be read.  Walks therefore count
// what is left of the row and keep their position unsigned.
#pragma once

#ifdef __CUDACC__
#define TC_WORDS_FN __host__ __device__ __forceinline__
#else
#define TC_WORDS_FN inline
#endif

namespace tc {

// The words [b, e) of a row from word b + skipped on.
struct Words {
    unsigned at;      // position of the first of them
    int left;         // how many there are (none when <= 0)
    TC_WORDS_FN Words(int b, int e, int skipped = 0) : at((unsigned)b + (unsigned)skipped), left(e - b - skipped) {}
    // n words on, n at most a few thousand; not past an end that `left` shows
    TC_WORDS_FN void skip(int n)
    {
        at += (unsigned)n;
        left -= n;
    }
};

// f(position, words left) every `step` words of [b, e) from word b + skipped
// on: the same walk with signed positions, which stay inside the row because
// the last step is not taken (SpMM of the power-law R-MAT scale 20 at k = 3:
// 169 us, 175 with Words).
template <class F>
TC_WORDS_FN void each_step(int b, int e, int skipped, int step, F &&f)
{
    if (e - b <= skipped) return;
    for (int j = b + skipped;; j += step) {
        f(j, e - j);
        if (e - j <= step) break;
    }
}

// The end of the first `most` of the words [b, e).
TC_WORDS_FN int words_upto(int b, int e, int most) { return e - b > most ? b + most : e; }

}  // namespace tc
