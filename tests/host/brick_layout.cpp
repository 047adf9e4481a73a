// The staged-tile layout of a metric, each of its allocations refused in turn: the call fails
// with the setting off and nothing of the layout left, and the next call builds it whole.
#include <cstdio>
#include <new>

#include "internal.h"
#include "runtime.h"

#define CHECK(x)                                                                \
    do {                                                                        \
        if (!(x)) {                                                             \
            std::printf("refused %ld: %s does not hold\n", refused, #x);        \
            return 1;                                                           \
        }                                                                       \
    } while (0)

int main() {
    mi_context* ctx = new mi_context();
    ctx->num_sms = 148;
    int failures = 0;
    for (long refused = 0;; ++refused) {
        mi_metric* m = new mi_metric();
        m->ctx = ctx;
        m->tile_capable = true;
        m->n_samples = 64;
        m->brick_bl = 3;
        for (int d = 0; d < 3; ++d) m->fgeo.size[d] = 16;
        CHECK(mi::dev_alloc(ctx, &m->samples, 64 * 4) == cudaSuccess);
        CHECK(mi::dev_alloc(ctx, &m->fbin, 64) == cudaSuccess);
        const size_t before = fake::live.size();
        // (the second try of a refused allocation, after what the context keeps went back, too)
        fake::allocations = 0;
        fake::fail_at = refused;
        fake::fail_on = 1;
        const mi_status s = mi_metric_set_tile_staging(m, 1);
        fake::fail_at = -1;
        int on = -1;
        CHECK(mi_metric_get_tile_staging(m, &on, nullptr) == MI_OK);
        if (s == MI_OK) {
            CHECK(on == 1);
            CHECK(failures >= 5);  // one for each of the layout's arrays at least
            std::printf("%d allocations refused in turn\n", failures);
            return 0;
        }
        ++failures;
        CHECK(s == MI_ERR_OUT_OF_MEMORY);
        CHECK(on == 0);
        CHECK(fake::live.size() == before);
        CHECK(mi_metric_set_tile_staging(m, 1) == MI_OK);
        CHECK(mi_metric_get_tile_staging(m, &on, nullptr) == MI_OK && on == 1);
        CHECK(m->codes && m->chunk_run && m->run_brick && m->run_start && m->run_chunk0);
        CHECK(m->nchunks > 0 && m->nruns > 0);
    }
}
