// Launches whose border components would not have ids of their own in 32 bits are refused before any CUDA
// call (this runs without a GPU), the largest that have them are not: exits 1 at a wrong answer.
#include "be_api_internal.h"
#include "be_kernels.h"

#include <cstdio>

using namespace be;

int main()
{
    const Geometry g[] = {uf2d_geometry(0), uf2d_geometry(1), uf2d_geometry(2), uf2d_geometry(kShapePixel2D), geometry_3d()};
    for (const Geometry &x : g) {
        const int64_t most = int64_t(kNone - 1) / x.maxb;   // tiles whose last node has an id below kNone
        if (!node_ids_fit(x, most) || node_ids_fit(x, most + 1)) {
            std::printf("%d nodes a tile\n", x.maxb);
            return 1;
        }
        be_ctx c;
        Workspace ws;
        if (ws.ensure(&c, x, (int64_t(1) << 32) / x.maxb + 1, 1, 1, nullptr) != BE_ERR_TOO_LARGE || ws.base) {
            std::printf("%d nodes a tile: not refused\n", x.maxb);
            return 1;
        }
    }
    return 0;
}
