// be_check_status reports the workspace of the last union-find call: an error word written into the
// workspace of a form (from outside, after the call) is reported while that form was the last one called,
// and the scan's flag is reported as its own site.  Exits 1 at the first wrong report.
#include "be_api_internal.h"

#include <cstdio>
#include <vector>

static be_ctx *c;
static uint8_t *in;
static int32_t *out;

static int call(int dims, int algo)
{
    const int rc = dims == 2 ? be_label2d(c, in, 64, 64, 64, 0, BE_COH_DEFAULT, algo, out, 64, nullptr, nullptr)
                             : be_label3d(c, in, 16, 16, 16, 0, algo, out, nullptr, nullptr);
    return rc ? rc : int(cudaDeviceSynchronize());
}

static int status(int dims)
{
    uint32_t s[3] = {99, 99, 99};
    return be_check_status(c, dims, s) ? -1 : int(s[0]);
}

#define EXPECT(x, y)                                                          \
    if ((x) != (y)) {                                                         \
        std::printf("line %d: %d, not %d\n", __LINE__, int(x), int(y));       \
        return 1;                                                             \
    }

int main()
{
    EXPECT(be_create(&c, 0), BE_OK);
    EXPECT(cudaMalloc(&in, 4096), cudaSuccess);
    EXPECT(cudaMalloc(&out, 4096 * 4), cudaSuccess);
    EXPECT(cudaMemset(in, 1, 4096), cudaSuccess);
    const uint32_t site[4] = {77, 5, 0, 0}, wait[4] = {0, 0, 0, 1}, none[4] = {};
    for (int dims = 2; dims <= 3; ++dims) {
        EXPECT(status(dims), 0);   // no call yet
        for (int algo : {BE_ALGO_PIXEL, BE_ALGO_RUNS, BE_ALGO_UF}) {
            if (dims == 3 && algo == BE_ALGO_RUNS) continue;
            EXPECT(call(dims, algo), 0);
            EXPECT(status(dims), 0);
            const bool form = algo != BE_ALGO_UF;
            const be::Workspace &ws = dims == 2 ? (form ? c->wsform2d : c->ws2d) : (form ? c->wsform3d : c->ws3d);
            EXPECT(cudaMemcpy(ws.w.err, site, sizeof(site), cudaMemcpyHostToDevice), cudaSuccess);
            EXPECT(status(dims), 77);
            EXPECT(cudaMemcpy(ws.w.err, wait, sizeof(wait), cudaMemcpyHostToDevice), cudaSuccess);
            EXPECT(status(dims), int(be::kSiteScanWait));
            EXPECT(cudaMemcpy(ws.w.err, none, sizeof(none), cudaMemcpyHostToDevice), cudaSuccess);
            EXPECT(status(dims), 0);
        }
    }
    EXPECT(be_destroy(c), BE_OK);
    return 0;
}
