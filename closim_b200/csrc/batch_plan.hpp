// How a batch's sheets are spread over the SMs: size classes and, for a given
// batch, whether a class's sheets are stepped by clusters or by lone blocks.
#pragma once
#include <algorithm>
#include <vector>

namespace cs {

// CTAs that step a sheet of n vertices together (a cluster). A function of the sheet
// alone, because it fixes the shape of the sheet's reductions: its result is the same
// in every batch. Below 1,500 vertices (three per thread) a cluster's barriers cost
// what its SMs save.
constexpr int kBatchClasses = 3;
constexpr int kBatchSize[kBatchClasses] = {4, 2, 1};
inline int batch_class(int n) { return n > 3000 ? 0 : n > 1500 ? 1 : 2; }

// Time of one sheet's step by `size` CTAs of 512 threads, in passes of a vertex
// per thread (about 6.2 ms at the reference budget on a B200). Measured, ms a step:
// lone blocks 18.4 at 1,444 vertices, 25.4 at 2,025, 37.9 at 3,025, 49.4 at 4,096, 85
// at 6,400, 119 at 10,000; pairs 16.0 at 2,025; clusters of four 15.0 at 3,025, 15.3
// at 4,096, 23.6 at 6,400, 35.3 at 10,000.
inline double batch_sheet_cost(int n, int size) { return n / (512.0 * size) + (size > 1 ? 0.6 : 0.13); }

// Estimated time of a step when class c's sheets (verts[c], largest first) go to
// groups of size[c] CTAs: the groups take sheets as they come free, a class starts on
// the SMs that the classes before it leave. maxGroups[c]: clusters of that class the
// device holds at once.
inline double batch_makespan(const std::vector<int> (&verts)[kBatchClasses], const int (&size)[kBatchClasses], int sms,
                             const int (&maxGroups)[kBatchClasses]) {
  std::vector<double> freeAt(sms, 0.0), ready;
  for (int c = 0; c < kBatchClasses; c++) {
    const int s = size[c], count = (int)verts[c].size();
    if (count == 0) continue;
    const int groups = std::min(count, s > 1 ? std::min(maxGroups[c], sms / s) : sms);
    if (groups < 1) return 1e300;
    std::sort(freeAt.begin(), freeAt.end());
    ready.resize(groups);
    for (int j = 0; j < groups; j++) ready[j] = -freeAt[j * s + s - 1];  // a heap of the earliest
    std::make_heap(ready.begin(), ready.end());
    for (int n : verts[c]) {
      std::pop_heap(ready.begin(), ready.end());
      ready.back() -= batch_sheet_cost(n, s);
      std::push_heap(ready.begin(), ready.end());
    }
    for (int j = 0; j < groups; j++)
      for (int q = 0; q < s; q++) freeAt[j * s + q] = -ready[j];
  }
  return *std::max_element(freeAt.begin(), freeAt.end());
}

// CTAs per sheet for each class: kBatchSize, or 1 where lone blocks, which reproduce
// the cluster's reductions, are expected to finish the batch as soon (3% go to the
// estimate's error). A cluster shortens the tail, a lone block spends fewer SM-cycles
// on a sheet: equal sheets that fill the device with one block each run best alone, few
// or very uneven ones in clusters. Measured on a B200 (33 clusters of four, 74 of two),
// ms a step, lone / clusters: 64 x 64 vertices, 74 sheets 52 / 46, 111 sheets 55 / 61,
// 148 sheets 57 / 77; 55 x 55, 37 sheets 38 / 30, 74 sheets 38 / 45, 160 sheets 77 / 76;
// 45 x 45, 74 sheets 25 / 16, 148 sheets 26 / 32, 222 sheets 50 / 48; 100 x 100, 60 sheets
// 131 / 71, 100 sheets 133 / 137; 16 to 128 a side, 64 sheets 189 / 55, 256 sheets
// 212 / 198, 384 sheets 225 / 274, 512 sheets 301 / 369. The estimate takes the
// smaller of each of these.
inline void batch_route(const std::vector<int> (&verts)[kBatchClasses], int sms,
                        const int (&maxGroups)[kBatchClasses], int (&size)[kBatchClasses]) {
  for (int c = 0; c < kBatchClasses; c++) size[c] = 1;
  double best = batch_makespan(verts, size, sms, maxGroups) * 0.97;
  for (int m = 1; m < 4; m++) {
    int s[kBatchClasses];
    for (int c = 0; c < kBatchClasses; c++) s[c] = (m >> c) & 1 ? kBatchSize[c] : 1;
    const double t = batch_makespan(verts, s, sms, maxGroups);
    if (t < best) {
      best = t;
      std::copy(s, s + kBatchClasses, size);
    }
  }
}

}  // namespace cs
