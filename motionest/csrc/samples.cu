// Host side of me_samples: the per-shot sample lists of plane masks.  Plain C++ on host memory;
// the meaning is that of motionest/sampling.py's _python_lists, which took 11 ms for 32 shots of
// 128x112 (most of a synthetic acquisition's 13.3 ms, now 6.4) and 48 ms for 64 shots of 256x224
// where this takes 0.6 and 3 ms.
#include <algorithm>
#include <cstring>
#include <exception>
#include <numeric>
#include <vector>

#include "common.cuh"

namespace me {

// Bins by decreasing sample count (stable), the bins of one count reordered so that each window
// of 16 positions holds bins of distinct residues mod 16 where it can, and none moved across
// position `split` (see spread_residues in motionest/sampling.py).
static void order_bins(const int* off, int ny, int split, int* order, std::vector<int>& sorted,
                       std::vector<int>& next) {
  sorted.resize(ny);
  next.resize(ny + 1);
  std::iota(sorted.begin(), sorted.end(), 0);
  auto count = [&](int b) { return off[b + 1] - off[b]; };
  std::stable_sort(sorted.begin(), sorted.end(),
                   [&](int a, int b) { return count(a) > count(b); });
  for (int start = 0; start < ny;) {
    int stop = start + 1;
    while (stop < ny && count(sorted[stop]) == count(sorted[start]) && stop != split) stop++;
    // the run's remaining bins as a list in their order: next[i] follows i, `head` leads
    int head = start;
    for (int i = start; i < stop; i++) next[i] = i + 1;
    for (int i = start; i < stop; i++) {
      unsigned used = 0;
      for (int k = i - i % 16; k < i; k++) used |= 1u << (order[k] % 16);
      int prev = -1, pick = head;
      while (pick < stop && (used >> (sorted[pick] % 16) & 1)) {
        prev = pick;
        pick = next[pick];
      }
      if (pick >= stop) {
        prev = -1;
        pick = head;
      }
      order[i] = sorted[pick];
      if (prev < 0) head = next[pick];
      else next[prev] = next[pick];
    }
    start = stop;
  }
}

}  // namespace me

using namespace me;

extern "C" int me_sample_lists(const unsigned char* planes, int nshots, int nx, int ny,
                               long long total, int* shot_off, int* kx, int* ky, int* ky_off,
                               int* ky_order) {
  if (!planes || !shot_off || !ky_off || !ky_order || (total > 0 && (!kx || !ky)))
    return fail("me_sample_lists: NULL pointer");
  if (nshots < 1 || nx < 1 || ny < 1 || (i64)nx * ny > 0x7fffffff)
    return fail("me_sample_lists: dims must be positive, nx * ny below 2^31");
  if (total < 0 || total > 0x7fffffff)  // the offsets are 32-bit
    return fail("me_sample_lists: `total` outside 0 .. 2^31 - 1");
  try {
    std::vector<int> at(ny), sorted, next, found;
    const int split = (ny > 128 && ny < 256) ? 256 - ny : 0;
    long long n = 0;
    shot_off[0] = 0;
    for (int s = 0; s < nshots; s++) {
      const unsigned char* p = planes + (i64)s * nx * ny;
      int* off = ky_off + (i64)s * (ny + 1);
      // the sampled points in memory order, eight bytes of a sparse mask at a time
      found.clear();
      const i64 cells = (i64)nx * ny;
      for (i64 i = 0; i < cells; i += 8) {
        uint64_t word = 0;
        std::memcpy(&word, p + i, (size_t)std::min<i64>(8, cells - i));
        if (word == 0) continue;
        for (i64 k = i; k < std::min(i + 8, cells); k++)
          if (p[k]) found.push_back((int)k);
      }
      std::fill(at.begin(), at.end(), 0);
      for (const int k : found) at[k % ny]++;
      off[0] = 0;
      for (int y = 0; y < ny; y++) off[y + 1] = off[y] + at[y];
      if (n + off[ny] > total) return fail("me_sample_lists: more samples than `total`");
      std::copy(off, off + ny, at.begin());
      for (const int k : found) {
        const int x = k / ny, y = k - x * ny;
        const long long i = n + at[y]++;
        kx[i] = x;
        ky[i] = y;
      }
      n += off[ny];
      shot_off[s + 1] = (int)n;
      order_bins(off, ny, split, ky_order + (i64)s * ny, sorted, next);
    }
    if (n != total) return fail("me_sample_lists: `total` is not the number of samples");
  } catch (const std::exception& e) {
    return fail(std::string("me_sample_lists: ") + e.what());
  }
  return ME_OK;
}
