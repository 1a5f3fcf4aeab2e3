// tc_words.h -- walking the words of a row.
//
// A matrix holds up to 2^31 - 1 words, so the position a strided loop steps to
// past the end of a row near the last word does not fit an int: it would come
// out negative, compare as before the end, and be read.  Three forms of a walk
// that stays inside the row; which one is the fastest differs from kernel to
// kernel by up to 8 %.
#pragma once

#ifdef __CUDACC__
#define TC_WORDS_FN __host__ __device__ __forceinline__
#else
#define TC_WORDS_FN inline
#endif

namespace tc {

// Counted: the words [b, e) of a row from word b + skipped on, at an unsigned
// position.
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

// By hand: the position `skipped` words from b, which may lie past
// 2^31 - 1 (and then comes out negative), and the words from position j to e,
// right for such a position too (and then not above 0).  A position is read,
// and stepped on from, only where words are left for that.
TC_WORDS_FN int words_from(int b, int skipped) { return (int)((unsigned)b + (unsigned)skipped); }
TC_WORDS_FN int words_left(int j, int e) { return (int)((unsigned)e - (unsigned)j); }

// Signed: f(position, words left) every `step` words of [b, e) from word b +
// skipped on; the step past the end is not taken.
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
