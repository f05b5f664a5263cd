// Check of the staged host transfers (ops::h2d_staged, d2h_staged): values of both strides
// below, at and above the sizes where the pinned buffers come into play, nothing written
// beside the elements, and the buffers made only once they repay it.
#include <cstdio>
#include <vector>
#include "../../cc4s_b200/csrc/ops.h"
using namespace cc4s_b200;

int main() {
  Stream s = ops::stream_create(0);
  const int64_t most = (int64_t(1) << 23) + 12345;
  double* d = ops::alloc(most);
  std::vector<double> h(2 * most + 1), r(2 * most + 1);
  for (size_t k = 0; k < h.size(); ++k) h[k] = 0.25 + double(k);
  // a first upload of the smallest staged size goes straight
  {
    ops::HostStage st;
    ops::h2d_staged(d, h.data(), ops::STAGED_MIN, 1, st, s);
    if (st.pinned) { printf("pinned for one small transfer\n"); return 1; }
    for (int k = 0; k < 8; ++k) ops::h2d_staged(d, h.data(), ops::STAGED_MIN, 1, st, s);
    if (!st.pinned) { printf("not pinned after many\n"); return 1; }
  }
  for (int64_t n : {int64_t(1), int64_t(1000), ops::STAGED_MIN - 1, ops::STAGED_MIN, ops::STAGED_MIN + 1,
                    (int64_t(1) << 22) + 77, most})
    for (int stride : {1, 2})
      for (int warm = 0; warm < 2; ++warm) {
        ops::HostStage st;
        if (warm) st.lost = ops::STAGED_LOST;
        const int off = stride - 1;  // the second plane of interleaved values
        ops::zero(d, most, s);
        ops::h2d_staged(d, h.data() + off, n, stride, st, s);
        std::fill(r.begin(), r.end(), -1.0);
        ops::d2h_staged(r.data() + off, stride, d, n, st, s);
        if (warm && n >= ops::STAGED_MIN && !st.pinned) { printf("not staged\n"); return 1; }
        for (int64_t k = 0; k < 2 * most + 1; ++k) {
          const int64_t e = (k - off) / stride;
          const bool in = k >= off && (k - off) % stride == 0 && e < n;
          if (r[k] != (in ? h[k] : -1.0)) {
            printf("n=%ld stride=%d warm=%d: element %ld is %g\n", (long)n, stride, warm, (long)k, r[k]);
            return 1;
          }
        }
      }
  ops::release(d);
  ops::stream_destroy(s);
  printf("ok\n");
  return 0;
}
