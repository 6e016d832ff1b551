// Workspace layouts of random pairs of launches in one allocation (host code only): prints the first pair
// in which the head of one -- launch epoch, error flags, scan status words -- is not the head of the other,
// or meets another array of either, and exits 1; exits 0 when there is none.
#include "be_api_internal.h"
#include "be_kernels.h"

#include <cstdio>
#include <random>
#include <vector>

using namespace be;

struct Launch {
    Geometry g;
    int64_t tiles, segs;
};

static Launch launch(std::mt19937_64 &r)
{
    auto side = [&](double hi) { return int(std::exp2(std::uniform_real_distribution<double>(0, hi)(r))); };
    const int shape = int(r() % (kNumShapes2D + 2));
    if (shape > kShapePixel2D) {
        Img3D im;
        fill_img3d(im, nullptr, side(9), side(9), side(9), 0, nullptr, 0, 0, 0);
        return {geometry_3d(), int64_t(im.t0) * im.t1 * im.t2, int64_t(im.d0) * im.d1 * im.t2};
    }
    Img2D im;
    const int rows = side(16), cols = side(14);
    fill_img2d(im, nullptr, cols, rows, cols, 0, nullptr, cols, 0, 0, 0, shape);
    return {uf2d_geometry(shape), int64_t(im.tiles_x) * im.tiles_y, int64_t(rows) * im.tiles_x};
}

int main()
{
    std::mt19937_64 r(1);
    int fits = 0;
    for (int i = 0; i < 20000; ++i) {
        const Launch a = launch(r), b = launch(r);
        // As Workspace::ensure sizes an allocation for the first, and takes it again for the second.
        const size_t need = layout_work(a.g, a.tiles, a.segs, 1, nullptr, nullptr), body = need + need / 4;
        const int64_t cap = max_chunks(body);
        const size_t bytes = head_bytes(cap) + body;
        char *base = reinterpret_cast<char *>(size_t(1) << 40);
        if (layout_work(b.g, b.tiles, b.segs, 1, nullptr, nullptr, cap) > bytes) continue;
        ++fits;
        Work w[2];
        size_t end[2] = {layout_work(a.g, a.tiles, a.segs, 1, base, &w[0], cap), layout_work(b.g, b.tiles, b.segs, 1, base, &w[1], cap)};
        const char *head_end = base + head_bytes(cap);
        bool ok = w[0].epoch == w[1].epoch && w[0].err == w[1].err && w[0].scan_status == w[1].scan_status;
        for (int k = 0; k < 2; ++k) {
            const Work &x = w[k];
            const void *arrays[] = {x.lab, x.perim, x.rbits, x.nb, x.timg, x.gp, x.nroot, x.nlink, x.segcnt, x.segpref, x.chunksum, x.queue, x.ncomp};
            for (const void *p : arrays) ok = ok && (!p || static_cast<const char *>(p) >= head_end);
            ok = ok && end[k] <= bytes && x.n_chunks <= cap && reinterpret_cast<const char *>(x.scan_status + x.n_chunks) <= head_end;
        }
        if (!ok) {
            std::printf("pair %d: %lld tiles %lld segments, then %lld tiles %lld segments\n", i, (long long)a.tiles, (long long)a.segs,
                        (long long)b.tiles, (long long)b.segs);
            return 1;
        }
    }
    std::printf("%d pairs share an allocation\n", fits);
    return fits > 1000 ? 0 : 1;
}
