// be_api.cu -- host side of the C ABI in include/be.h: contexts, scratch workspaces and the
// launch sequences of the 2D / 3D pipelines.
//
// The reference allocates its block buffers per call (clCreateBuffer in InitSPixels,
// LabelingAlgs.cpp:996-997 / 1451-1452) and frees them after (FreeSPixels, :1059-1063).  Here a
// context keeps one workspace per pipeline and grows it only when a larger image arrives, so a
// steady stream of calls allocates nothing.
#include "be.h"
#include "be_api_internal.h"
#include "be_kernels.h"

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>

namespace be {

int set_error(be_ctx *ctx, int code, const char *fmt, ...)
{
    if (ctx) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        ctx->err = buf;
    }
    return code;
}

int cuda_error(be_ctx *ctx, cudaError_t e, const char *what)
{
    return set_error(ctx, e == cudaErrorMemoryAllocation ? BE_ERR_OOM : BE_ERR_CUDA, "%s: %s (%s)",
                     what, cudaGetErrorName(e), cudaGetErrorString(e));
}

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

Geometry geometry_2d() { return uf2d_geometry(0); }

Geometry geometry_3d()
{
    Geometry g;
    g.lab_bytes_per_tile = size_t(T3_LAB_WORDS) * sizeof(uint32_t);
    g.rbits_bytes_per_tile = size_t(T3_NROW) * sizeof(uint32_t);
    g.nperim = T3_EDGE;
    g.maxb = T3_MAXB;
    g.links = true;
    return g;
}

// The head of a workspace: launch epoch, error flags and the status words of the segment scan.  A status word
// is taken for this launch's when it carries its epoch, so whatever else may be in the scratch, these words
// must never be anything but status words: the head comes first and has one size for all the launches that
// use an allocation.
static size_t take_head(int64_t chunks, char *base, Work &t)
{
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char *p = base ? base + off : nullptr;
        off = align_up(off + bytes, 256);
        return p;
    };
    t.epoch = reinterpret_cast<uint32_t *>(take(2 * sizeof(uint32_t)));
    t.err = reinterpret_cast<uint32_t *>(take(16 * sizeof(uint32_t)));
    t.scan_status = reinterpret_cast<uint64_t *>(take(size_t(std::max<int64_t>(chunks, 1)) * sizeof(uint64_t)));
    return off;
}

size_t head_bytes(int64_t chunks)
{
    Work t{};
    return take_head(chunks, nullptr, t);
}

// A segment takes at least five bytes of a launch's arrays, its count and its prefix.
int64_t max_chunks(size_t bytes) { return int64_t(bytes / (5 * size_t(kScanChunk))) + 1; }

// Carves the workspace of a launch with n_tiles tiles, n_segs segments and n_imgs images out of
// one allocation (or only computes its size when base == nullptr).  head_chunks: the scan chunks that the
// allocation's head holds (0: as many as this launch has).
size_t layout_work(const Geometry &g, int64_t n_tiles, int64_t n_segs, int n_imgs, char *base, Work *w,
                   int64_t head_chunks)
{
    const int64_t n_chunks = (n_segs + kScanChunk - 1) / kScanChunk;
    Work t{};
    size_t off = take_head(head_chunks ? head_chunks : n_chunks, base, t);
    auto take = [&](size_t bytes) {
        size_t o = off;
        off = align_up(off + bytes, 256);
        return base ? base + o : nullptr;
    };
    const size_t nodes = size_t(n_tiles) * g.maxb;
    t.lab = take(size_t(n_tiles) * g.lab_bytes_per_tile);
    t.perim = reinterpret_cast<uint16_t *>(take(size_t(n_tiles) * g.nperim * sizeof(uint16_t)));
    t.rbits = reinterpret_cast<uint32_t *>(take(size_t(n_tiles) * g.rbits_bytes_per_tile));
    t.nb = reinterpret_cast<uint32_t *>(take(size_t(n_tiles) * sizeof(uint32_t)));
    t.timg = reinterpret_cast<uint32_t *>(take(n_imgs > 1 ? size_t(n_tiles) * sizeof(uint32_t) : 0));
    t.gp = reinterpret_cast<unsigned long long *>(take(nodes * sizeof(unsigned long long)));
    t.nroot = reinterpret_cast<uint16_t *>(take(nodes * sizeof(uint16_t)));
    t.nlink = g.links ? reinterpret_cast<uint2 *>(take(nodes * sizeof(uint2))) : nullptr;
    t.segcnt = reinterpret_cast<uint8_t *>(take(align_up(size_t(n_segs) * g.seg_bytes, 16) + 16));
    t.segpref = reinterpret_cast<uint32_t *>(take((size_t(n_segs) + 1) * sizeof(uint32_t)));
    t.chunksum = reinterpret_cast<uint32_t *>(take(size_t(std::max<int64_t>(n_chunks, 1)) * sizeof(uint32_t)));
    t.queue = reinterpret_cast<uint32_t *>(take(kQueueWords * sizeof(uint32_t)));
    t.ncomp = reinterpret_cast<int64_t *>(take(size_t(std::max(n_imgs, 1)) * sizeof(int64_t)));
    t.n_tiles = n_tiles;
    t.n_segs = n_segs;
    t.n_chunks = int32_t(n_chunks);
    t.n_imgs = n_imgs;
    if (w) *w = t;
    return off;
}

cudaError_t reset_scan_state(const Work &w, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(w.epoch, 0, 2 * sizeof(uint32_t), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(w.scan_status, 0, size_t(std::max(w.n_chunks, 1)) * sizeof(uint64_t), s);
    return e;
}

int Workspace::ensure(be_ctx *ctx, const Geometry &g, int64_t n_tiles, int64_t n_segs, int n_imgs, cudaStream_t s)
{
    if (!node_ids_fit(g, n_tiles)) return set_error(ctx, BE_ERR_TOO_LARGE, "more than 2^32 - 2 tile border components in one launch");
    // Node links name a segment in 32 bits.
    if (n_segs >= int64_t(kNone)) return set_error(ctx, BE_ERR_TOO_LARGE, "more than 2^32 - 2 image rows in one launch");
    if (!base || layout_work(g, n_tiles, n_segs, n_imgs, nullptr, nullptr, cap_chunks) > bytes) {
        if (base) {
            cudaError_t e = cudaFree(base);
            base = nullptr;
            bytes = 0;
            if (e != cudaSuccess) return cuda_error(ctx, e, "cudaFree(workspace)");
        }
        const size_t need = layout_work(g, n_tiles, n_segs, n_imgs, nullptr, nullptr);
        size_t body = need + need / 4;   // headroom for slightly larger later calls
        cudaError_t e = cudaMalloc(&base, head_bytes(max_chunks(body)) + body);
        if (e == cudaErrorMemoryAllocation) {   // without it
            cudaGetLastError();
            body = need;
            e = cudaMalloc(&base, head_bytes(max_chunks(body)) + body);
        }
        const size_t head = head_bytes(max_chunks(body));
        if (e != cudaSuccess) {
            base = nullptr;
            cudaGetLastError();
            return cuda_error(ctx, e, "cudaMalloc(workspace)");
        }
        // The scan's status words and the launch epoch start at zero once; every later run tells
        // its own status words from older ones by the epoch it increments.  (On the call's stream: a clear on the
        // default stream does not hold up a non-blocking one, and could come after its first kernels.)
        e = cudaMemsetAsync(base, 0, head, s);
        if (e != cudaSuccess) return cuda_error(ctx, e, "cudaMemsetAsync(workspace)");
        bytes = head + body;
        cap_chunks = max_chunks(body);   // of any launch whose arrays fit beside the head
    }
    layout_work(g, n_tiles, n_segs, n_imgs, static_cast<char *>(base), &w, cap_chunks);
    cap_tiles = n_tiles;
    cap_segs = n_segs;
    cap_imgs = n_imgs;
    return BE_OK;
}

void Workspace::release()
{
    if (base) cudaFree(base);
    base = nullptr;
    bytes = 0;
    cap_tiles = cap_segs = 0;
    cap_imgs = 0;
}

// ---------------------------------------------------------------------------------------------
// Launch sequences.
// ---------------------------------------------------------------------------------------------
void fill_img2d(Img2D &im, const uint8_t *in, int64_t in_pitch, int32_t rows, int32_t cols, int thr,
                int32_t *out, int64_t out_pitch, int64_t tile_base, int64_t seg_base, int index,
                int shape)
{
    const int tw = kShapes2D[shape].tw, th = kShapes2D[shape].th;
    im.in = in;
    im.out = out;
    im.in_pitch = in_pitch;
    im.out_pitch = out_pitch;
    im.rows = rows;
    im.cols = cols;
    im.tiles_x = (cols + tw - 1) / tw;
    im.tiles_y = (rows + th - 1) / th;
    im.tile_base = tile_base;
    im.seg_base = seg_base;
    im.thr = thr;
    im.index = index;
}

void fill_img3d(Img3D &im, const uint8_t *in, int32_t d0, int32_t d1, int32_t d2, int thr,
                int32_t *out, int64_t tile_base, int64_t seg_base, int index)
{
    im.in = in;
    im.out = out;
    im.d0 = d0;
    im.d1 = d1;
    im.d2 = d2;
    im.t0 = (d0 + 2 * T3_TB0 - 1) / (2 * T3_TB0);
    im.t1 = (d1 + 2 * T3_TB1 - 1) / (2 * T3_TB1);
    im.t2 = (d2 + 2 * T3_TB2 - 1) / (2 * T3_TB2);
    im.tile_base = tile_base;
    im.seg_base = seg_base;
    im.thr = thr;
    im.index = index;
}

// Whether the pixel and run forms leave an image of n pixels to the iterative forms, which give the same
// labels with about 4.5 bytes of scratch a pixel: the tile pipeline's is a fixed 17 KB a tile, whatever part
// of the tile the image fills.  Images of up to four rows or eight columns take more than 32 bytes a pixel so; where
// that comes to more than half a gigabyte, it is not taken.  Measured, 4-connected, by tiles / iterative: 1 x 2^25
// pixels, half of them set, 3404 us and 5.4 GB / 1402 us and 0.17 GB, nearly all set 3501 / 5766 us; 2^23 x 1
// 2813 us and 2.8 GB / 345 us and 0.04 GB, nearly all set 3057 / 1490 us; 4 x 2^22 574 us and 0.7 GB / 1171 us
// and 0.09 GB; but 8 x 2^22 617 us and 0.7 GB / 2992 us and 0.17 GB.
constexpr size_t kThinBytes = size_t(1) << 29;
static bool tiles_nearly_empty(size_t bytes, int64_t n) { return bytes > kThinBytes && bytes > 32 * size_t(n); }

// The tile pipeline on one image, in the context's workspace of the block form or of the others.
// BE_ERR_OOM when there is no memory for its scratch, or `form` has a better use for it.
static int run_tiles2d(be_ctx *c, bool form, int shape, const Img2D &im, bool count, cudaStream_t s)
{
    const Geometry g = uf2d_geometry(shape);
    const int64_t n_tiles = int64_t(im.tiles_x) * im.tiles_y, n_segs = int64_t(im.rows) * im.tiles_x;
    if (form && tiles_nearly_empty(layout_work(g, n_tiles, n_segs, 1, nullptr, nullptr), int64_t(im.rows) * im.cols)) return BE_ERR_OOM;
    Workspace &ws = form ? c->wsform2d : c->ws2d;
    c->last_ws[0] = &ws;
    int rc = ws.ensure(c, g, n_tiles, n_segs, 1, s);
    if (rc) return rc;
    ImgList2D L{nullptr, 1, im};
#ifdef BE_BOUNDS_CHECK
    cudaMemsetAsync(ws.w.err, 0, 16 * sizeof(uint32_t), s);
#endif
    const bool timed = c->timing && !form;
    Work w = ws.w;
    w.host_count = count ? c->h_ncomp : nullptr;   // the count straight to the host, no copy after
    const cudaError_t e = uf2d_launch(shape, L, w, c->sms, false, s, timed ? c->stage_ev : nullptr);
    c->timed_stages = timed ? kStages2D : 0;
    c->last_ncomp = ws.w.ncomp;
    return e == cudaSuccess ? BE_OK : cuda_error(c, e, "be_label2d launch");
}

static int run_tiles3d(be_ctx *c, bool form, const Img3D &im, bool count, cudaStream_t s)
{
    const Geometry g = geometry_3d();
    const int64_t n_tiles = int64_t(im.t0) * im.t1 * im.t2, n_segs = int64_t(im.d0) * im.d1 * im.t2;
    if (form && tiles_nearly_empty(layout_work(g, n_tiles, n_segs, 1, nullptr, nullptr), int64_t(im.d0) * im.d1 * im.d2)) return BE_ERR_OOM;
    Workspace &ws = form ? c->wsform3d : c->ws3d;
    c->last_ws[1] = &ws;
    int rc = ws.ensure(c, g, n_tiles, n_segs, 1, s);
    if (rc) return rc;
    ImgList3D L{nullptr, 1, im};
#ifdef BE_BOUNDS_CHECK
    cudaMemsetAsync(ws.w.err, 0, 16 * sizeof(uint32_t), s);
#endif
    const bool timed = c->timing && !form;
    Work w = ws.w;
    w.host_count = count ? c->h_ncomp : nullptr;   // as in 2D
    const cudaError_t e = launch_uf3d(L, w, c->sms, false, s, timed ? c->stage_ev : nullptr);
    c->timed_stages = timed ? kStages3D : 0;
    c->last_ncomp = ws.w.ncomp;
    return e == cudaSuccess ? BE_OK : cuda_error(c, e, "be_label3d launch");
}

// The end of a label call: notes what ran and, where the caller wants the count, waits for it.
static int finish_label(be_ctx *c, bool iter, int64_t *n_components, const char *what, cudaStream_t s)
{
    c->last_iter = iter;
    if (iter) c->last_ncomp = c->wsiter.w.ncomp;
    if (!n_components) return BE_OK;
    cudaError_t e = cudaSuccess;
    if (iter) e = cudaMemcpyAsync(c->h_ncomp, c->last_ncomp, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(c, e, what);
    if (iter && c->iter_err && *c->iter_err) return set_error(c, BE_ERR_NO_CONVERGENCE, "%s: iteration cap reached", what);
    *n_components = c->h_ncomp[0];
    return BE_OK;
}

}  // namespace be

using namespace be;

// ---------------------------------------------------------------------------------------------
// C ABI.
// ---------------------------------------------------------------------------------------------
extern "C" {

const char *be_version(void) { return "0.1.0"; }

int be_create(be_ctx **out, int device)
{
    if (!out) return BE_ERR_INVALID;
    *out = nullptr;
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess) return BE_ERR_CUDA;
    if (device < 0 || device >= ndev) return BE_ERR_INVALID;
    be_ctx *c = new be_ctx();
    c->device = device;
    e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&c->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&c->ev1);
    if (e == cudaSuccess) e = cudaMallocHost(&c->h_ncomp, 64 * sizeof(int64_t));
    for (int i = 0; i <= kStages && e == cudaSuccess; ++i) e = cudaEventCreate(&c->stage_ev[i]);
    if (e != cudaSuccess) {
        be_destroy(c);
        return e == cudaErrorMemoryAllocation ? BE_ERR_OOM : BE_ERR_CUDA;
    }
    *out = c;
    return BE_OK;
}

int be_destroy(be_ctx *c)
{
    if (!c) return BE_OK;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    c->ws2d.release();
    c->ws3d.release();
    c->wsiter.release();
    c->wsform2d.release();
    c->wsform3d.release();
    for (be_iter_graph &g : c->iter_graph) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        if (g.graph) cudaGraphDestroy(g.graph);
    }
    if (c->d_in) cudaFree(c->d_in);
    if (c->d_out) cudaFree(c->d_out);
    if (c->slab_buf) cudaFree(c->slab_buf);
    if (c->h_ncomp) cudaFreeHost(c->h_ncomp);
    for (int i = 0; i <= kStages; ++i)
        if (c->stage_ev[i]) cudaEventDestroy(c->stage_ev[i]);
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
    return BE_OK;
}

const char *be_last_error(const be_ctx *c) { return c ? c->err.c_str() : "no context"; }

int be_check_status(be_ctx *c, int dims, uint32_t *out3)
{
    if (!c || !out3 || (dims != 2 && dims != 3)) return BE_ERR_INVALID;
    out3[0] = out3[1] = out3[2] = 0;
    const Workspace *ws = c->last_ws[dims - 2];
    if (!ws || !ws->base) return BE_OK;
    uint32_t err[4] = {};
    cudaError_t e = cudaMemcpy(err, ws->w.err, sizeof(err), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_error(c, e, "be_check_status");
    std::copy(err, err + 3, out3);
    if (!out3[0] && err[3]) out3[0] = kSiteScanWait;
    return BE_OK;
}

int be_set_stage_timing(be_ctx *c, int enable)
{
    if (!c) return BE_ERR_INVALID;
    c->timing = enable != 0;
    c->timed_stages = 0;
    return BE_OK;
}

int be_stage_times(be_ctx *c, float *ms, int max_stages, int *n_stages)
{
    if (!c || !n_stages) return BE_ERR_INVALID;
    *n_stages = c->timed_stages;
    if (!c->timed_stages) return BE_OK;
    cudaError_t e = cudaEventSynchronize(c->stage_ev[c->timed_stages]);
    if (e != cudaSuccess) return cuda_error(c, e, "be_stage_times");
    for (int i = 0; i < c->timed_stages && i < max_stages; ++i) {
        e = cudaEventElapsedTime(&ms[i], c->stage_ev[i], c->stage_ev[i + 1]);
        if (e != cudaSuccess) return cuda_error(c, e, "be_stage_times");
    }
    return BE_OK;
}

int be_label2d(be_ctx *c, const uint8_t *in, int64_t in_pitch, int32_t rows, int32_t cols,
               int threshold, int coh, int algo, int32_t *out, int64_t out_pitch,
               int64_t *n_components, void *stream)
{
    if (!c) return BE_ERR_INVALID;
    c->err.clear();
    if (!in || !out) return set_error(c, BE_ERR_INVALID, "be_label2d: null buffer");
    if (rows <= 0 || cols <= 0 || int64_t(rows) * cols >= (int64_t(1) << 31))
        return set_error(c, BE_ERR_INVALID, "be_label2d: bad size %d x %d", rows, cols);
    if (in_pitch < cols || out_pitch < cols)
        return set_error(c, BE_ERR_INVALID, "be_label2d: pitch smaller than the row");
    if (threshold < 0 || threshold > 255)
        return set_error(c, BE_ERR_INVALID, "be_label2d: threshold %d outside 0..255", threshold);
    if (algo < BE_ALGO_AUTO || algo > BE_ALGO_RUNS)
        return set_error(c, BE_ERR_INVALID, "be_label2d: unknown algorithm %d", algo);
    if (coh == BE_COH_4 && algo != BE_ALGO_PIXEL && algo != BE_ALGO_RUNS)
        return set_error(c, BE_ERR_INVALID, "be_label2d: block equivalence does not support 4-connectivity");
    if (coh != BE_COH_4 && coh != BE_COH_8 && coh != BE_COH_DEFAULT)
        return set_error(c, BE_ERR_INVALID, "be_label2d: unknown connectivity %d", coh);
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_error(c, e, "cudaSetDevice");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = BE_OK, shape;
    pick2d(c, rows, cols, algo, &algo, &shape);
    const bool form = algo == BE_ALGO_PIXEL || algo == BE_ALGO_RUNS;
    bool iter = algo == BE_ALGO_ITER;
    if (form) {
        // The pixel and run forms give the components of their connectivity in canonical order: 4
        // by the pipeline on pixel runs, 8 by the block pipeline.  (Sizes as their own key space --
        // rows of a power of two -- takes them.)
        if ((int64_t(rows) << ceil_log2(cols)) >= (int64_t(1) << 31))
            return set_error(c, BE_ERR_INVALID, algo == BE_ALGO_PIXEL ? "label equivalence: %d x %d exceeds its key space"
                                                                      : "run equivalence: %d x %d exceeds its key space", rows, cols);
        shape = coh == BE_COH_8 ? 0 : kShapePixel2D;
    }
    if (!iter) {
        Img2D im;
        fill_img2d(im, in, in_pitch, rows, cols, threshold, out, out_pitch, 0, 0, 0, shape);
        rc = run_tiles2d(c, form, shape, im, n_components != nullptr, s);
        if (rc && !(form && rc == BE_ERR_OOM)) return rc;
        iter = rc != BE_OK;   // scratch refused: the same components with less of it
    }
    if (iter) {
        c->err.clear();
        rc = form && coh != BE_COH_8 ? run_lbeq2d(c, in, in_pitch, rows, cols, threshold, out, out_pitch, s)
                                     : run_iter2d(c, in, in_pitch, rows, cols, threshold, out, out_pitch, s);
        if (rc) return rc;
    }
    return finish_label(c, iter, n_components, "be_label2d", s);
}

int be_label3d(be_ctx *c, const uint8_t *in, int32_t d0, int32_t d1, int32_t d2, int threshold,
               int algo, int32_t *out, int64_t *n_components, void *stream)
{
    if (!c) return BE_ERR_INVALID;
    c->err.clear();
    if (!in || !out) return set_error(c, BE_ERR_INVALID, "be_label3d: null buffer");
    if (d0 <= 0 || d1 <= 0 || d2 <= 0 || int64_t(d0) * d1 * d2 >= (int64_t(1) << 31))
        return set_error(c, BE_ERR_INVALID, "be_label3d: bad size %d x %d x %d", d0, d1, d2);
    if (threshold < 0 || threshold > 255)
        return set_error(c, BE_ERR_INVALID, "be_label3d: threshold %d outside 0..255", threshold);
    if (algo < BE_ALGO_AUTO || algo > BE_ALGO_PIXEL)
        return set_error(c, BE_ERR_INVALID, algo == BE_ALGO_RUNS ? "be_label3d: run equivalence is 2D only"
                                                                 : "be_label3d: unknown algorithm %d", algo);
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_error(c, e, "cudaSetDevice");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int rc = BE_OK;
    pick3d(c, int64_t(d0) * d1 * d2, algo, &algo);
    const bool form = algo == BE_ALGO_PIXEL;
    bool iter = algo == BE_ALGO_ITER;
    if (form && (int64_t(d0) << (ceil_log2(d1) + ceil_log2(d2))) >= (int64_t(1) << 31))   // as in 2D
        return set_error(c, BE_ERR_INVALID, "label equivalence: volume exceeds its key space");
    if (!iter) {
        Img3D im;
        fill_img3d(im, in, d0, d1, d2, threshold, out, 0, 0, 0);
        rc = run_tiles3d(c, form, im, n_components != nullptr, s);
        if (rc && !(form && rc == BE_ERR_OOM)) return rc;
        iter = rc != BE_OK;   // as in 2D
    }
    if (iter) {
        c->err.clear();
        rc = run_iter3d(c, in, d0, d1, d2, threshold, out, s);
        if (rc) return rc;
    }
    return finish_label(c, iter, n_components, "be_label3d", s);
}

static int ensure_staging(be_ctx *c, size_t in_bytes, size_t out_bytes)
{
    cudaError_t e;
    if (in_bytes > c->d_in_bytes) {
        if (c->d_in) cudaFree(c->d_in);
        c->d_in = nullptr;
        c->d_in_bytes = 0;
        e = cudaMalloc(&c->d_in, in_bytes);
        if (e != cudaSuccess) return cuda_error(c, e, "cudaMalloc(input staging)");
        c->d_in_bytes = in_bytes;
    }
    if (out_bytes > c->d_out_bytes) {
        if (c->d_out) cudaFree(c->d_out);
        c->d_out = nullptr;
        c->d_out_bytes = 0;
        e = cudaMalloc(&c->d_out, out_bytes);
        if (e != cudaSuccess) return cuda_error(c, e, "cudaMalloc(output staging)");
        c->d_out_bytes = out_bytes;
    }
    return BE_OK;
}

int be_label2d_host(be_ctx *c, const uint8_t *in, int64_t in_pitch, int32_t rows, int32_t cols,
                    int threshold, int coh, int algo, int32_t *out, int64_t out_pitch,
                    int64_t *n_components, double *elapsed_us)
{
    if (!c) return BE_ERR_INVALID;
    c->err.clear();
    if (!in || !out) return set_error(c, BE_ERR_INVALID, "be_label2d_host: null buffer");
    if (rows <= 0 || cols <= 0 || in_pitch < cols || out_pitch < cols)
        return set_error(c, BE_ERR_INVALID, "be_label2d_host: bad size or pitch");
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_error(c, e, "cudaSetDevice");
    // Rows without gaps in host memory stay without gaps on the device, so that each way is one flat
    // copy.  A pageable copy of rows into or out of padded rows is twice as slow as a flat one (a whole
    // call at 1021x1787 1080-1170 us, flat 580-610; 100x100 113, flat 80), where the labeling itself
    // loses a few us to unaligned rows.
    const int64_t dpi = in_pitch == cols ? cols : (int64_t(cols) + 15) / 16 * 16;
    const int64_t dpo = out_pitch == cols ? cols : (int64_t(cols) + 3) / 4 * 4;
    int rc = ensure_staging(c, size_t(dpi) * rows, size_t(dpo) * rows * sizeof(int32_t));
    if (rc) return rc;
    cudaStream_t s = c->stream;
    e = in_pitch == cols ? cudaMemcpyAsync(c->d_in, in, size_t(cols) * rows, cudaMemcpyHostToDevice, s)
                         : cudaMemcpy2DAsync(c->d_in, dpi, in, in_pitch, cols, rows, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_error(c, e, "upload");
    cudaEventRecord(c->ev0, s);
    int64_t n = 0;
    rc = be_label2d(c, static_cast<const uint8_t *>(c->d_in), dpi, rows, cols, threshold, coh, algo,
                    static_cast<int32_t *>(c->d_out), dpo, nullptr, s);
    if (rc) return rc;
    cudaEventRecord(c->ev1, s);
    e = out_pitch == cols ? cudaMemcpyAsync(out, c->d_out, size_t(cols) * rows * sizeof(int32_t), cudaMemcpyDeviceToHost, s)
                          : cudaMemcpy2DAsync(out, out_pitch * sizeof(int32_t), c->d_out, dpo * sizeof(int32_t),
                                              cols * sizeof(int32_t), rows, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return cuda_error(c, e, "download");
    e = cudaMemcpyAsync(c->h_ncomp, c->last_ncomp, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(c, e, "be_label2d_host sync");
    if (c->last_iter && c->iter_err && *c->iter_err)
        return set_error(c, BE_ERR_NO_CONVERGENCE, "be_label2d_host: iteration cap reached");
    n = c->h_ncomp[0];
    if (n_components) *n_components = n;
    if (elapsed_us) {
        float ms = 0;
        cudaEventElapsedTime(&ms, c->ev0, c->ev1);
        *elapsed_us = double(ms) * 1000.0;
    }
    return BE_OK;
}

int be_label3d_host(be_ctx *c, const uint8_t *in, int32_t d0, int32_t d1, int32_t d2,
                    int threshold, int algo, int32_t *out, int64_t *n_components,
                    double *elapsed_us)
{
    if (!c) return BE_ERR_INVALID;
    c->err.clear();
    if (!in || !out) return set_error(c, BE_ERR_INVALID, "be_label3d_host: null buffer");
    if (d0 <= 0 || d1 <= 0 || d2 <= 0)
        return set_error(c, BE_ERR_INVALID, "be_label3d_host: bad size");
    cudaError_t e = cudaSetDevice(c->device);
    if (e != cudaSuccess) return cuda_error(c, e, "cudaSetDevice");
    const size_t n = size_t(d0) * d1 * d2;
    int rc = ensure_staging(c, n, n * sizeof(int32_t));
    if (rc) return rc;
    cudaStream_t s = c->stream;
    e = cudaMemcpyAsync(c->d_in, in, n, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_error(c, e, "upload");
    cudaEventRecord(c->ev0, s);
    rc = be_label3d(c, static_cast<const uint8_t *>(c->d_in), d0, d1, d2, threshold, algo,
                    static_cast<int32_t *>(c->d_out), nullptr, s);
    if (rc) return rc;
    cudaEventRecord(c->ev1, s);
    e = cudaMemcpyAsync(out, c->d_out, n * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return cuda_error(c, e, "download");
    e = cudaMemcpyAsync(c->h_ncomp, c->last_ncomp, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(c, e, "be_label3d_host sync");
    if (c->last_iter && c->iter_err && *c->iter_err)
        return set_error(c, BE_ERR_NO_CONVERGENCE, "be_label3d_host: iteration cap reached");
    if (n_components) *n_components = c->h_ncomp[0];
    if (elapsed_us) {
        float ms = 0;
        cudaEventElapsedTime(&ms, c->ev0, c->ev1);
        *elapsed_us = double(ms) * 1000.0;
    }
    return BE_OK;
}

}  // extern "C"
