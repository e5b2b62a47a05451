// The march segments (vah_kernels.cuh) against a search over every number of parts.
#include <cuda_runtime.h>

#include "vah_kernels.cuh"

extern "C" {

// The segment length for n cells and `strips` strips; calls: how many lengths were priced.
int sc_segment(int n, int minb, long long strips, int *calls) {
    *calls = 0;
    return vah::march_segment(n, minb, [&](int len) {
        ++*calls;
        return strips * ((n + len - 1) / len);
    });
}

int sc_search(int n, int minb, long long strips) {
    const long long wave = 148 * 4 * minb;
    int best = 1;
    double cost = 1e300;
    for (int parts = 1; parts <= n; ++parts) {
        const int len = (n + parts - 1) / parts;
        const double c = (double)((strips * ((n + len - 1) / len) + wave - 1) / wave) * (len + 1.5);
        if (c < cost) {
            cost = c;
            best = len;
        }
    }
    return best;
}

}  // extern "C"
