// be_common.cuh -- shared device code for the B200 Block-Equivalence labeler.
//
// Terminology (follows the reference's BE method, LabelingAlgs.cl:133-319 / 737-979):
//   block      2x2 pixels (2D) or 2x2x2 voxels (3D); the reference's "super pixel".
//   mask       which pixels/voxels of a block are foreground (4 / 8 bits).
//   tile       the rectangle (box) of blocks one CTA labels in shared memory.
//   key        the raster index of a pixel/voxel inside its image (row-major, last dim fastest).
//              A component is represented by its smallest key (its first pixel in raster order);
//              that is what makes the output canonical.
//   node       a tile-local component that touches the tile border; nodes are merged across
//              tiles with a global union-find.
//   segment    the part of one image row (a line along the fastest dimension) that lies in one
//              tile; per-segment root counts give each component its canonical rank.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>
#include <utility>

namespace be {

constexpr uint32_t kNone = 0xFFFFFFFFu;

// ---------------------------------------------------------------------------------------------
// Image descriptors.  One pipeline launch labels a list of images (the plain API passes one).
// ---------------------------------------------------------------------------------------------
struct Img2D {
    const uint8_t *in;   // row-major uint8, in_pitch bytes per row
    int32_t *out;        // row-major int32 labels, out_pitch elements per row
    int64_t in_pitch;
    int64_t out_pitch;
    int32_t rows, cols;
    int32_t tiles_x, tiles_y;
    int64_t tile_base;   // index of the image's first tile in the launch
    int64_t seg_base;    // index of the image's first segment in the launch
    int32_t thr;         // foreground is pixel > thr
    int32_t index;       // position in the caller's list (for per-image outputs)
};

struct Img3D {
    const uint8_t *in;   // dense [d0][d1][d2] uint8, d2 fastest
    int32_t *out;        // dense [d0][d1][d2] int32 labels
    int32_t d0, d1, d2;
    int32_t t0, t1, t2;  // tile counts per dimension
    int64_t tile_base;
    int64_t seg_base;
    int32_t thr;
    int32_t index;
};

// The images of one launch: a device array, or a single descriptor passed by value (plain calls
// need no descriptor upload).
template <class Img>
struct ImgList {
    const Img *ptr;
    int n;
    Img one;
    __device__ __forceinline__ Img find(int64_t tile, uint32_t *timg) const;
    __device__ __forceinline__ Img get(int64_t tile, const uint32_t *timg) const;
};

// Global scratch of one pipeline launch ("workspace").  Sizes are per tile so that every tile
// owns fixed-size slices and no kernel needs a prefix sum to find its data.
struct Work {
    void *lab;            // per-block tile-local labels: uint16 (2D) / uint32 (3D), NBLK per tile
    uint16_t *perim;      // per tile NPERIM border entries: (node << 4) | side bits, 0 = empty
    uint32_t *nb;         // per tile: number of nodes
    uint32_t *timg;       // per tile: its image's place in the launch's list (launches of several images)
    unsigned long long *gp;   // per node (tile * MAXB + j): union-find entry (key of the parent << 32) |
                              // parent (global node id); see gentry
    uint16_t *nroot;      // per node: tile-local block index of the node's root block
    uint2 *nlink;         // per node, after the merge: x = segment of its global root's first pixel
                          // (kNone when the node is a root itself), y = (root block << 16) | rank
                          // of that first pixel among the roots left in its segment
    uint32_t *rbits;      // per tile: bitmap of the tile's components that are still roots (the merge
                          // clears the ones it links): 2D a bit per run, 3D a bit per first voxel
    uint8_t *segcnt;      // per segment: number of component roots (uint8, or uint16 in a pipeline whose segments
                          // can hold more than 255; word-padded)
    uint32_t *segpref;    // per segment + 1: exclusive prefix of segcnt over the launch
    uint32_t *chunksum;   // per scan chunk: sum of segcnt
    uint32_t *queue;      // work-queue counters (persistent mode); zeroed before a launch
    int64_t *ncomp;       // per image: number of components
    int64_t *host_count;  // the first image's count once more, in pinned host memory (or null)
    uint32_t *err;        // error flags (bounded waits / iteration caps)
    uint32_t *epoch;      // [0] launch epoch (+1 per pipeline run), [1] scan ticket counter
    uint64_t *scan_status;  // per scan chunk: (epoch << 34 | state << 32) | prefix value
    int64_t n_tiles;
    int64_t n_segs;
    int32_t n_chunks;
    int32_t n_imgs;
};

constexpr int kScanChunk = 4096;    // segments per scan chunk (one CTA)

// ---------------------------------------------------------------------------------------------
// Bounds-checked build (-DBE_BOUNDS_CHECK): GUARD(w, cond, site, value) is false when `cond`
// fails; the first failure of a launch records (site, value) in w.err[0..2] and the guarded
// access is skipped.  In normal builds GUARD is the constant true and costs nothing.
// ---------------------------------------------------------------------------------------------
#ifdef BE_BOUNDS_CHECK
__device__ __forceinline__ bool be_guard(uint32_t *err, bool ok, uint32_t site, uint64_t val)
{
    if (!ok && atomicCAS(err, 0u, site) == 0u) {
        err[1] = uint32_t(val);
        err[2] = uint32_t(val >> 32);
    }
    return ok;
}
#define GUARD(w, cond, site, val) be_guard((w).err, bool(cond), (site), uint64_t(val))
#else
#define GUARD(w, cond, site, val) (true)
#endif

// ---------------------------------------------------------------------------------------------
// Small helpers.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p)
{
    return *reinterpret_cast<const volatile uint32_t *>(p);
}

// Union-find find over a shared-memory parent array (parents never exceed their child), with
// path halving: each visited entry is pointed at its grandparent.  Every stored value is an
// ancestor of the entry at the time it was read, so concurrent merges stay correct: a pointer
// never leaves the entry's component, and a merge that loses a race to such a store retries
// from the parent it displaced (see smerge).
__device__ __forceinline__ uint32_t sfind(uint32_t *P, uint32_t a)
{
    uint32_t p = P[a];
    while (p != a) {
        const uint32_t g = P[p];
        if (g != p) P[a] = g;
        a = p;
        p = g;
    }
    return a;
}

// Merge of two shared-memory union-find trees that keeps the smaller index as the root
// (the atomicMin formulation of Playne & Hawick's union-find, safe under concurrent merges).
__device__ __forceinline__ void smerge(uint32_t *P, uint32_t a, uint32_t b)
{
    for (;;) {
        a = sfind(P, a);
        b = sfind(P, b);
        if (a == b) return;
        if (a < b) {
            uint32_t old = atomicMin(&P[b], a);
            if (old == b) return;
            b = old;
        } else {
            uint32_t old = atomicMin(&P[a], b);
            if (old == a) return;
            a = old;
        }
    }
}

// Points entries first, first + step, ... below n of a shared-memory parent array straight at their
// roots while no link happens (a read-only walk, then one store: whatever a walk meets is an
// ancestor, so any interleaving is right).  Entries are taken in ascending order by all threads at
// once, so a walk soon meets entries that are done.  (Sweeps of pointer jumping with four entries in
// flight, and one state machine per lane over its entries, were measured slower: the loop is bound by
// instruction issue, not by the latency of a walk.)
__device__ __forceinline__ void sflatten_all(uint32_t *P, uint32_t first, uint32_t step, uint32_t n)
{
    for (uint32_t i = first; i < n; i += step) {
        uint32_t x = P[i];
        if (x == i) continue;
        uint32_t y = P[x];
        if (y == x) continue;   // at its root already
        while (y != x) {
            x = y;
            y = P[x];
        }
        P[i] = x;
    }
}

// First pass over pairs of a flat parent array (every entry at its root), by one warp over its own
// part q[0 .. n) of the pairs ((a << 16) | b): pairs of one root are dropped, the others hook the larger
// root under the smaller (atomicMin) and stay, as roots, at the front of q; returns how many.  A hook
// can be overwritten by another one, and can land on an entry hooked meanwhile, so after a barrier the
// pairs that stay are merged for good (smerge) -- by then most are one set already.
__device__ __forceinline__ uint32_t shook_pairs(uint32_t *P, uint32_t *q, uint32_t n)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t kept = 0;
    for (uint32_t k = 0; k < n; k += 32) {
        uint32_t x = 0, y = 0;
        if (k + lane < n) {
            const uint32_t e = q[k + lane];
            x = P[e >> 16];
            y = P[e & 0xFFFFu];
        }
        const uint32_t keep = __ballot_sync(0xFFFFFFFFu, x != y);   // (the pairs of this turn are read)
        if (x != y) {
            atomicMin(&P[max(x, y)], min(x, y));
            q[kept + __popc(keep & ((1u << lane) - 1u))] = (x << 16) | y;
        }
        kept += __popc(keep);
    }
    __syncwarp();
    return kept;
}

// Appends this lane's `n` merge pairs to a shared queue with one atomic per warp; returns the
// lane's first position (positions >= capacity mean the queue is full for those pairs).
__device__ __forceinline__ uint32_t warp_reserve(uint32_t *count, uint32_t n)
{
    const int lane = threadIdx.x & 31;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    uint32_t base = 0;
    if (lane == 31 && total) base = atomicAdd(count, total);
    base = __shfl_sync(0xFFFFFFFFu, base, 31);
    return base + incl - n;
}

// Global union-find entries: gp[x] = (key of x's parent << 32) | parent, a root holding its own key
// and index.  Keys (first-pixel raster indices) are distinct, and a parent's key is always smaller
// than its child's, so no path can close a cycle whatever other threads link meanwhile, and one
// load of an entry gives both the parent and the key that decides which way a union goes.
__device__ __forceinline__ unsigned long long gentry(uint32_t key, uint32_t id)
{
    return (static_cast<unsigned long long>(key) << 32) | id;
}

// Union of nodes a and b after Rem's algorithm, lock-free: the two sides climb in turn, always
// the side whose parent has the larger key (the order keys are linked in), with path halving on
// the way; the walk ends where the two parents meet (already one set), or when the climbing side
// stands on a root, which is linked (CAS) under the other side's parent -- a node of b's set with
// a smaller key.  A walk that reaches the common ancestor stops there instead of going on to both
// roots.  Latency, not work, is the cost: each step is one L2 round trip, and one load gives the
// parent and its key.  on_link(node, key) is called with the root that was linked and its key.  (Rem's
// splicing -- re-pointing the climbing node at the other side's parent -- was measured: it merged
// the long paths of one-pixel spirals into deep trees.)
template <typename OnLink>
__device__ __forceinline__ void gunion_keyed(unsigned long long *gp, uint32_t a, uint32_t b, OnLink on_link)
{
    volatile unsigned long long *vp = gp;
    unsigned long long ea = vp[a], eb = vp[b];
    for (;;) {
        if (uint32_t(ea) == uint32_t(eb)) return;   // same parent: one set
        if ((ea >> 32) < (eb >> 32)) {               // climb on the side with the larger parent key
            const uint32_t t = a; a = b; b = t;
            const unsigned long long u = ea; ea = eb; eb = u;
        }
        const uint32_t pa = uint32_t(ea);
        if (pa == a) {   // a root
            const unsigned long long old = atomicCAS(gp + a, ea, eb);
            if (old == ea) {
                on_link(a, uint32_t(ea >> 32));
                return;
            }
            ea = old;
            eb = vp[b];
            continue;
        }
        const unsigned long long ga = vp[pa];
        if (uint32_t(ga) != pa) vp[a] = ga;   // halving
        a = pa;
        ea = ga;
    }
}

// Points node x at its parent's parent (one jump; a root and a root's child stay).
__device__ __forceinline__ void gjump(unsigned long long *gp, uint32_t x)
{
    volatile unsigned long long *vp = gp;
    const uint32_t p = uint32_t(vp[x]);
    if (p == x) return;
    const unsigned long long ep = vp[p];
    if (uint32_t(ep) != p) vp[x] = ep;
}

// Root of node x after all merges of the launch are complete, by pointer jumping that writes only
// x's own entry: each step x is pointed at its parent's parent as that entry reads now.  When every
// node of a deep tree runs this at once, each read lands on an entry that its own thread has
// already shortened, so the walks take about log2(depth) steps instead of depth (and no two
// threads write the same entry).  The cap only bounds the walk should the forest ever hold a cycle
// (it cannot).
__device__ __forceinline__ uint32_t gfind_jump(unsigned long long *gp, uint32_t x)
{
    volatile unsigned long long *vp = gp;
    uint32_t p = uint32_t(vp[x]);
    if (p == x) return x;
    for (int it = 0; it < (1 << 24); ++it) {
        const unsigned long long ep = vp[p];
        const uint32_t g = uint32_t(ep);
        if (g == p) break;   // p is the root
        vp[x] = ep;
        p = g;
    }
    return p;
}

// Decrement a uint8 or uint16 counter packed in a 32-bit word (the counter is >= 1 when this is called).
template <class Count>
__device__ __forceinline__ void dec_count(uint8_t *base, int64_t idx)
{
    const int64_t at = idx * int64_t(sizeof(Count));
    uint32_t *w = reinterpret_cast<uint32_t *>(base + (at & ~int64_t(3)));
    atomicSub(w, 1u << (8 * (at & 3)));
}

// Block-wide exclusive scan of one uint32 per thread; returns the thread's prefix and writes the
// total to *total.  `tmp` must hold blockDim.x / 32 + 1 words.
template <int NT>
__device__ __forceinline__ uint32_t block_exscan(uint32_t v, uint32_t *tmp, uint32_t *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tmp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < NT / 32 ? tmp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < NT / 32) tmp[lane] = s;
        if (lane == NT / 32 - 1) tmp[NT / 32] = s;
    }
    __syncthreads();
    uint32_t r = x - v + (warp ? tmp[warp - 1] : 0);
    *total = tmp[NT / 32];
    __syncthreads();
    return r;
}

// Index of the image that owns global item `t`, by binary search over the images' bases.
template <class Img>
__device__ __forceinline__ int find_img_tile(const Img *imgs, int n, int64_t t)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (imgs[mid].tile_base <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The image of a tile: by search in the first launch, which leaves its index for the later ones.
template <class Img>
__device__ __forceinline__ Img ImgList<Img>::find(int64_t tile, uint32_t *timg) const
{
    if (n == 1) return one;
    const int i = find_img_tile(ptr, n, tile);
    if (threadIdx.x == 0) timg[tile] = uint32_t(i);
    return ptr[i];
}

template <class Img>
__device__ __forceinline__ Img ImgList<Img>::get(int64_t tile, const uint32_t *timg) const
{
    return n == 1 ? one : ptr[__ldcg(timg + tile)];
}

using ImgList2D = ImgList<Img2D>;
using ImgList3D = ImgList<Img3D>;

// ---- Pixel rows as bit words ------------------------------------------------------------------
// Byte-wise x > thr for four pixels: bit 7 of each byte.  K = 0x7F - (thr & 0x7F) in every byte;
// `hi` = thr >= 128.  (x & 0x7F) + K carries into bit 7 exactly when the low seven bits exceed
// thr's; the high bit decides the rest.
__device__ __forceinline__ uint32_t gt_bytes(uint32_t x, uint32_t K, bool hi)
{
    const uint32_t s = (x & 0x7F7F7F7Fu) + K;
    return (hi ? (x & s) : (x | s)) & 0x80808080u;
}

// Bits 7, 15, 23, 31 -> bits 0..3 (the four partial products land on distinct bits, no carries).
__device__ __forceinline__ uint32_t gather4(uint32_t g) { return (g * 0x00204081u) >> 28; }

// 16 pixels of one row -> foreground bits of their even (left) and odd (right) pixels: 8 blocks.
__device__ __forceinline__ void split16(uint4 v, uint32_t K, bool hi, uint32_t &ev, uint32_t &od)
{
    ev = gather4(gt_bytes(__byte_perm(v.x, v.y, 0x6420), K, hi)) |
         (gather4(gt_bytes(__byte_perm(v.z, v.w, 0x6420), K, hi)) << 4);
    od = gather4(gt_bytes(__byte_perm(v.x, v.y, 0x7531), K, hi)) |
         (gather4(gt_bytes(__byte_perm(v.z, v.w, 0x7531), K, hi)) << 4);
}

// 16 pixels of one row -> their foreground bits in order.
__device__ __forceinline__ uint32_t bits16(uint4 v, uint32_t K, bool hi)
{
    return gather4(gt_bytes(v.x, K, hi)) | (gather4(gt_bytes(v.y, K, hi)) << 4) | (gather4(gt_bytes(v.z, K, hi)) << 8) |
           (gather4(gt_bytes(v.w, K, hi)) << 12);
}

// Bits 0..15 of x -> bits 0, 2, .. 30.
__device__ __forceinline__ uint32_t spread16(uint32_t x)
{
    x &= 0xFFFFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

// Foreground bits of the n (1..64) pixels at p, split as split16 (bit k of left / right: pixel
// 2k / 2k + 1), whatever p's alignment: the up to five 16-byte chunks that hold the pixels are
// loaded whole and the words shifted into place -- an odd offset swaps the even and odd words.  A
// chunk that would reach outside [lo, hi), the image's bytes, is read byte by byte.  (One byte
// load per pixel cost a tile kernel 64 dependent load-and-or steps per row for every image whose
// width is not a multiple of 16.)
__device__ __forceinline__ void row_bits(const uint8_t *p, int n, const uint8_t *lo, const uint8_t *hi,
                                         uint32_t K, bool thr_hi, int thr, uint32_t &left, uint32_t &right)
{
    const int a = int(reinterpret_cast<uintptr_t>(p) & 15u);
    const uint8_t *base = p - a;
    uint4 v[5];
    uint32_t bytewise = 0;   // chunks to read byte by byte
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        v[i] = make_uint4(0, 0, 0, 0);
        if (16 * i < a + n) {
            const uint8_t *c = base + 16 * i;
            if (c >= lo && c + 16 <= hi) v[i] = __ldg(reinterpret_cast<const uint4 *>(c));
            else bytewise |= 1u << i;
        }
    }
    uint32_t ev = 0, od = 0, ev4 = 0, od4 = 0;   // even / odd bytes of chunks 0..3, of chunk 4
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        uint32_t e8, o8;
        split16(v[i], K, thr_hi, e8, o8);
        if ((bytewise >> i) & 1u) {
            e8 = o8 = 0;
#pragma unroll 1
            for (int k = 0; k < 16; ++k) {
                const uint8_t *c = base + 16 * i + k;
                const uint32_t bit = (c >= lo && c < hi && *c > thr) ? 1u << (k >> 1) : 0u;
                if (k & 1) o8 |= bit;
                else e8 |= bit;
            }
        }
        if (i < 4) {
            ev |= e8 << (8 * i);
            od |= o8 << (8 * i);
        } else {
            ev4 = e8;
            od4 = o8;
        }
    }
    const uint32_t h = uint32_t(a) >> 1;
    const uint32_t el = __funnelshift_r(ev, ev4, h), ol = __funnelshift_r(od, od4, h);
    const uint32_t er = __funnelshift_r(ev, ev4, h + 1u);
    left = (a & 1) ? ol : el;
    right = (a & 1) ? er : ol;
    const int nl = (n + 1) >> 1, nr = n >> 1;   // valid left / right pixels
    left &= 0xFFFFFFFFu >> (32 - nl);
    right &= nr ? 0xFFFFFFFFu >> (32 - nr) : 0u;
}

// Stores one row's labels from a group of W neighbouring lanes, lane g holding the four pixels
// v of the row at dst (n of them, 0..4, are inside the row; a lane's are full before the next
// lane has any), with aligned 16-byte stores whatever the row's alignment: when dst is m elements
// past a 16-byte boundary, each lane stores the quad of the m last pixels of the lane before it
// and its own first 4 - m; the group's ends and the row's end are stored pixel by pixel.  Every
// lane of the warp calls this (dst & 15 is the same over a group).
template <int W>
__device__ __forceinline__ void store_row(int32_t *dst, int4 v, int n)
{
    const uint32_t m = uint32_t(reinterpret_cast<uintptr_t>(dst) >> 2) & 3u;
    const int py = __shfl_up_sync(0xFFFFFFFFu, v.y, 1, W), pz = __shfl_up_sync(0xFFFFFFFFu, v.z, 1, W);
    const int pw = __shfl_up_sync(0xFFFFFFFFu, v.w, 1, W), pn = __shfl_up_sync(0xFFFFFFFFu, n, 1, W);
    const int g = int(threadIdx.x) & (W - 1);
    int4 q = v;
    if (m == 1) q = make_int4(pw, v.x, v.y, v.z);
    else if (m == 2) q = make_int4(pz, pw, v.x, v.y);
    else if (m == 3) q = make_int4(py, pz, pw, v.x);
    const int have = g ? max(0, pn - (4 - int(m))) : 0;          // pixels of the lane before in the quad
    int32_t *d = dst - m;
    if (have == int(m) && n >= 4 - int(m)) {
        __stcs(reinterpret_cast<int4 *>(d), q);
    } else {
        const int b = g ? 0 : int(m), e = n > 0 ? int(m) + min(n, 4 - int(m)) : have;   // elements [b, e) of the quad
        if (b <= 0 && 0 < e) d[0] = q.x;
        if (b <= 1 && 1 < e) d[1] = q.y;
        if (b <= 2 && 2 < e) d[2] = q.z;
        if (b <= 3 && 3 < e) d[3] = q.w;
    }
    if (g == W - 1 && m) {   // the group's last lane: its own pixels past its quad
        const int b = 4 - int(m);
        if (b <= 1 && 1 < n) dst[1] = v.y;
        if (b <= 2 && 2 < n) dst[2] = v.z;
        if (b <= 3 && 3 < n) dst[3] = v.w;
    }
}

// Programmatic dependent launch (sm_90 and later).  A launch made with programmatic stream
// serialization may put its CTAs on the SMs while the grid before it in the stream still runs:
// grid_dep_wait() blocks until that grid has completed and its writes are visible (for a normal
// launch it returns at once), and grid_dep_release() lets the next grid's CTAs be scheduled once
// every CTA of this grid has called it or exited.  The pipeline kernels wait before their first
// global access, so the overlap only hides launch and ramp-up time, never a dependency.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Asynchronous global -> shared copies (cp.async, through L1): the data lands in shared memory
// without passing through registers, so a CTA can fetch its next tile's small arrays while it
// works on the current one.  cp_async_wait() waits for all of this thread's copies; a barrier
// after it makes every thread's copies visible to the CTA.
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)   // L2 only
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Launches kernel k, with programmatic stream serialization when `overlap` is set, and always with
// the whole of the SM's L1 / shared memory asked for as shared memory.  Left to itself the runtime picks
// a split per kernel from its occupancy; an SM drains before it changes its split, so a launch whose
// split differs from its predecessor's cannot overlap it (measured, 2048^2: 58 us a call with
// differing splits, 43 us with one).
template <typename... P, typename... A>
inline cudaError_t launch_k(void (*k)(P...), unsigned grid, unsigned block, cudaStream_t s, bool overlap,
                            A &&...args)
{
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[0].val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 2u : 1u;
    return cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

// Work distribution: with a queue (Q) every CTA pulls items from a counter until none are left
// (persistent launch); without one, CTA b takes items b, b + grid, ...  The counter's answer takes an L2
// round trip, so a CTA asks for its next item (request) while it still works on the current one and
// reads the answer (next) after the barrier that ends it -- or an earlier one, where it prefetches.
template <bool Q>
struct ItemLoop {
    uint32_t *queue;
    uint32_t ticket = 0;   // thread 0: the item asked for
    __device__ __forceinline__ int64_t first(uint32_t *slot)
    {
        if (!Q) return blockIdx.x;
        if (threadIdx.x == 0) *slot = atomicAdd(queue, 1u);
        __syncthreads();
        const int64_t v = *slot;
        __syncthreads();
        return v;
    }
    __device__ __forceinline__ void request()
    {
        if (Q && threadIdx.x == 0) ticket = atomicAdd(queue, 1u);
    }
    // Publishes the answer; a barrier goes between this and next(), and another between next() and the
    // following publish().
    __device__ __forceinline__ void publish(uint32_t *slot)
    {
        if (Q && threadIdx.x == 0) *slot = ticket;
    }
    __device__ __forceinline__ int64_t next(int64_t cur, const uint32_t *slot) const
    {
        return Q ? int64_t(*slot) : cur + gridDim.x;
    }
};

// Label writes of few tiles: several CTAs share a tile's rows, each working out the tile's labels for
// itself, so that a launch of fewer tiles than the SMs can hold CTAs does not take as long as one CTA
// needs for a whole tile's stores.  CTAs per tile, from a launch's tiles and the CTAs it may have (a whole
// number, so that the kernel reads it off its grid).  Measured, whole calls: 200x300 31.3 -> 30.2 us,
// 513x700 35.3 -> 33.5, 48^3 41.0 -> 38.4, 191x223x157 68.3 -> 66.1.
constexpr int kMaxWriteSplit = 8;
// A CTA writes whole tiles; shares one with others; or shares the only tile (2D, without a merge).
enum WriteForm { kWriteTiles, kWriteShared, kWriteOne };
inline int write_split(int64_t n_tiles, int64_t ctas)
{
    return int(std::max<int64_t>(1, std::min<int64_t>(kMaxWriteSplit, ctas / std::max<int64_t>(1, n_tiles))));
}

}  // namespace be
