// The part of a field's span that a line of the float TBC copies to shared memory.
#pragma once

#ifdef __CUDACC__
#define VHSD_HD __host__ __device__
#else
#define VHSD_HD
#endif

namespace vhsd {

struct TbcStretch {
    bool staged;   // false: the line is read from global memory tap by tap
    int lo, len;   // floats [lo, lo + len), four at a time
};

// The stretch for a line whose first and last output samples lie at span
// samples `first` and `last` (positions run one way along the line): their
// taps, x - 7 .. x + 8, and what load_taps reads beside them.  A line whose
// taps leave the span of n samples or the stage (its locations are no line's)
// is not staged.  The chroma copy starts up to three floats before lo (in the
// row of lo's block, whose kept samples have others ahead of them) and ends up
// to four after lo + len: still inside the span.  The positions are compared
// before any sum is formed: they saturate at the ends of the int range, and
// such a sum would wrap.
VHSD_HD inline TbcStretch tbc_stretch(int first, int last, int n, int stage_cap) {
    const int low = first < last ? first : last, high = first < last ? last : first;
    TbcStretch s{false, 0, 0};
    if (low < 7 || n < 26 || high > n - 19) return s;
    s.lo = (low - 7) & ~3;
    s.len = (high - 7 + 19 - s.lo + 3) & ~3;
    s.staged = s.len + 4 <= stage_cap;
    return s;
}

}  // namespace vhsd
