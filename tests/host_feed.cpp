// Host build of volume-compressor_gb300/csrc/feed_extent.cuh, run through the
// orders in which the GPU may run the warps that use it: between two meetings
// every warp puts its part for the coming atom, and the first one then takes the
// atom's. Output: atoms whose extent was another's, atoms checked.
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#define __device__
#define __forceinline__ inline

#include "feed_extent.cuh"

using namespace vcg;

constexpr int W = 3;

static float norm_of(uint32_t i, int w) { return (float)(1000 * i + 10 * w + 1); }
static uint32_t far_of(uint32_t i, int w) { return 7 * ((i * 31 + w * 17) % 97) + 1; }

int main() {
    // between the meetings of atoms i and i + 1: warp 0 takes atom i (step 0), then puts its
    // part of i + 1 (step 1); the other warps put theirs (steps 2, 3), in any order with those
    std::vector<std::vector<int>> orders;
    std::vector<int> o = {0, 1, 2, 3};
    do {
        if (std::find(o.begin(), o.end(), 0) < std::find(o.begin(), o.end(), 1)) orders.push_back(o);
    } while (std::next_permutation(o.begin(), o.end()));
    int wrong = 0, checked = 0;
    for (size_t a = 0; a < orders.size(); ++a)
        for (size_t b = 0; b < orders.size(); ++b) {
            FeedExtent<W> x;
            for (int w = 0; w < W; ++w) x.put(0, w, norm_of(0, w), far_of(0, w));
            for (uint32_t i = 0; i < 8; ++i) {
                float n = 0.0f;
                uint32_t f = 0;
                for (int step : orders[i & 1 ? b : a]) {
                    if (step == 0) x.take(i, n, f);
                    else x.put(i + 1, step - 1, norm_of(i + 1, step - 1), far_of(i + 1, step - 1));
                }
                float wn = norm_of(i, 0);
                uint32_t wf = far_of(i, 0);
                for (int w = 1; w < W; ++w) {
                    wn += norm_of(i, w);
                    wf = std::max(wf, far_of(i, w));
                }
                wrong += n != wn || f != wf;
                ++checked;
            }
        }
    printf("%d %d\n", wrong, checked);
    return 0;
}
