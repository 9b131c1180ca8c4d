// Which segment an outer tile belongs to, for kernels that find their tiles without a list (simt_tiles.cuh): tile t of
// segment s has slot floor(first_row(s) / 64) + s + t, so first slots grow from segment to segment.
//
// All threads of a CTA look at once, each at one candidate, and the number of them whose segment starts at or before the slot
// narrows the candidates to one of `threads` pieces: one round up to 256 segments, two up to 65 536.  (A binary search is a chain of
// global loads, a third of a microsecond each; a look at every segment by every CTA grows with the square of the segments: fp32
// self-attention over segments of 8-64 rows, 2 heads of 64, forward with a binary search | with a look at every segment | now:
// 64 segments 52 | 55 | 55 us, 1000 111 | 100 | 96, 4096 371 | 311 | 279, 16 384 1390 | 1843 | 1000.)  The answer
// follows from the prefix sums alone, whatever they hold: CTAs of one cluster, which ask for the same slot, get the same one.
//
// No CUDA in here beyond the two qualifiers: the CPU tests compile it as it is.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define VAFA_HD __host__ __device__ __forceinline__
#else
#define VAFA_HD inline
#endif

namespace vafa {
namespace tiles {

constexpr int kRows = 64;  // outer rows per CTA

VAFA_HD long long first_slot(const int32_t* cu, int seg, int stack) { return (long long)cu[seg] * stack / kRows + seg; }

struct SegSearch {
  unsigned lo, hi, step;  // candidates [lo, hi); thread i looks at lo + i step

  VAFA_HD SegSearch(int n_seg, int threads) : lo(0), hi((unsigned)n_seg), step(((unsigned)n_seg - 1) / threads + 1) {}
  VAFA_HD bool done() const { return hi - lo <= 1; }
  VAFA_HD bool starts_by(const int32_t* cu, int stack, long long slot, int thread) const {
    const unsigned i = lo + (unsigned)thread * step;
    return i < hi && first_slot(cu, (int)i, stack) <= slot;
  }
  // `count`: of how many threads starts_by() is true.  (None: the first piece, whose first slot is behind the one that was asked for.)
  VAFA_HD void narrow(int count, int threads) {
    if (count > 0) lo += (unsigned)(count - 1) * step;
    if (hi - lo > step) hi = lo + step;
    step = (hi - lo - 1) / threads + 1;
  }
};

}  // namespace tiles
}  // namespace vafa
