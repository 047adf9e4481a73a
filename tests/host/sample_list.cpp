// The sample list of a metric whose fixed mask admits one voxel of a whole grid: as long as it
// has to be, not as long as the grid.
#include <cstdio>
#include <vector>

#include "internal.h"
#include "runtime.h"

int main() {
    mi_context* ctx = new mi_context();
    ctx->num_sms = 148;
    mi_geometry g = {{128, 128, 128}, {1, 1, 1}, {0, 0, 0}, {1, 0, 0, 0, 1, 0, 0, 0, 1}};
    const int64_t n = 128 * 128 * 128;
    mi_image img[3];
    for (mi_image& i : img) {
        i.ctx = ctx;
        i.geo = g;
        i.n = n;
        if (mi::dev_alloc(ctx, &i.data, (size_t)n * 4) != cudaSuccess) return 1;
    }
    mi_metric_options opt = {};
    opt.metric = MI_METRIC_MEAN_SQUARES;
    mi_metric* m = nullptr;
    const mi_status s = mi_metric_create_ex(ctx, &img[0], &img[1], &img[2], nullptr, nullptr, 32, &opt, &m);
    if (s != MI_OK) {
        std::printf("create: %d %s\n", (int)s, mi_last_error(ctx));
        return 1;
    }
    const size_t bytes = fake::live.at(m->samples);
    std::printf("%lld samples in %zu bytes\n", (long long)m->n_samples, bytes);
    return m->n_samples == 1 && bytes <= 4096 ? 0 : 1;  // (the runtime's words are all 1)
}
