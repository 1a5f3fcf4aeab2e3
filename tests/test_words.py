"""Walks over the words of a row (tc_words.h), compiled for the host: every
strided walk visits its words and no others, also where the row ends at or
near word 2^31 - 1, the largest position a matrix can have."""
import os
import subprocess

from tests.test_host_checks import CSRC

PROGRAM = r'''
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include "tc_words.h"

// The words a kernel reads: `round` of them, every by-th, per step.
static long walk(int b, int e, int lane, int by, int round)
{
    const long begin = b, end = e;
    long want = begin + lane, bad = 0, steps = 0;
    for (tc::Words a(b, e, lane); a.left > 0; a.skip(round * by)) {
        if (++steps > 1 << 20) return -1;                       // does not end
        for (int w = 0; w < round; ++w) {
            if (w * by >= a.left) break;
            const long at = (long)(uintptr_t)(a.at + (unsigned)(w * by));
            bad += at != want || at >= end;
            want += by;
        }
    }
    return bad + (want < end);                                  // a word left out
}

// The same with each_step.
static long steps(int b, int e, int lane, int by, int round)
{
    long want = (long)b + lane, bad = 0;
    tc::each_step(b, e, lane, round * by, [&](int j, int left) {
        bad += j < b || j >= e || left != (long)e - j;
        for (int w = 0; w < round && w * by < left; ++w) {
            bad += (long)j + w * by != want;
            want += by;
        }
    });
    return bad + (want < e);
}

// The same by hand.
static long by_hand(int b, int e, int lane, int by, int round)
{
    long want = (long)b + lane, bad = 0;
    int j = tc::words_from(b, lane);
    for (;;) {
        for (int w = 0; w < round && w * by < tc::words_left(j, e); ++w) {
            bad += (long)j + w * by != want || want >= e;
            want += by;
        }
        if (tc::words_left(j, e) <= round * by) break;
        j += round * by;
    }
    return bad + (want < e);
}

int main()
{
    const int top = 2147483647;
    const int lens[] = {0, 1, 2, 3, 4, 5, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 5000};
    const int bys[] = {1, 2, 4, 8, 16, 32, 64, 128, 256}, rounds[] = {1, 2, 3, 4, 6, 8};
    long bad = 0;
    for (int end : {5000, top - 4096, top - 1024, top - 7, top - 1, top})
        for (int n : lens)
            for (int by : bys)
                for (int r : rounds)
                    for (int lane : {0, 1, by / 2, by - 1})
                        if (lane < by && (walk(end - n, end, lane, by, r) || steps(end - n, end, lane, by, r) ||
                                           by_hand(end - n, end, lane, by, r))) ++bad;
    for (int b : {0, 77, top - 100, top - 16384, top - 16385})
        for (int e : {b, b + 1, top - (top - b) / 2, top}) {
            const long want = (long)e - b > 16384 ? (long)b + 16384 : (long)e;
            if (tc::words_upto(b, e, 16384) != want) ++bad;
        }
    std::printf("%ld\n", bad);
    return bad != 0;
}
'''


def test_walks(tmp_path):
    src, exe = tmp_path / "words.cpp", tmp_path / "words"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
