"""Descriptors of the Float32 precision line: which of them run as TF32 is recorded in golden/float32_line.txt."""
import math
import random

PATTERNS = ["abcdef geac dfgb", "abcdef gfac degb", "abcdef dfgb geac", "abcdef dega gfbc", "abcdef efgb gdac", "abcdef gdab efgc",
            "abcd deca be", "abcd aebf fdec", "abcd aedf fbec", "abcde efba cfd", "abc adc db", "abcde efbad cf", "bcdea bagf fcged"]
EXTENTS = [3, 4, 4, 5, 6, 7, 8, 8, 9, 10, 11, 12, 12, 13, 15, 16, 16, 18, 20, 21, 24, 24, 27, 30, 32, 36, 40, 48, 52, 60, 64, 72, 80, 96,
           100, 120, 128, 192, 256, 512]


def descriptors(count=6000):
    rng = random.Random(20)
    while count:
        C, A, B = rng.choice(PATTERNS).split()
        ext = {m: rng.choice(EXTENTS) for m in sorted(set(C + A + B))}
        if max(math.prod(ext[m] for m in t) for t in (A, B, C)) < 2**31:
            count -= 1
            yield C, A, B, ext
