// be_uf3d.cu -- 3D Block-Equivalence labeling, union-find form (26-connectivity, 2x2x2 blocks).
//
// Replaces the reference's BLEQ3D_Init / BLEQ3D_Scan / BLEQ3D_Analyze / BLEQ3D_SetFinalLabels
// (LabelingAlgs.cl:740-979) and their host loop (LabelingAlgs.cpp:1443-1536) with the same
// four-launch structure as the 2D pipeline (be_uf2d_impl.cuh):
//
//   k_tile_local_3d   one CTA per 16 x 32 x 64-voxel tile (8 x 16 x 32 blocks): 16-byte loads,
//                     voxel-class words per block row, runs along d2 and their links to the four
//                     preceding rows by bit operations, a shared-memory union-find over run numbers
//                     (the run of the component's first voxel stays the root); writes the tile's bit
//                     words, the root run of every run, a bitmap of the root runs and the segments'
//                     root counts, and exports border components as nodes.
//   k_merge_3d        links of block rows across tile borders, and the global union-find over the nodes
//                     they join; a root linked under another leaves its segment count and its
//                     tile's bitmap.
//   k_scan_link_3d    exclusive scan of the segment counts (single pass, look-back) and, in the
//                     same launch, every linked node pointed at its global root with the segment
//                     and in-segment rank of that root's first voxel resolved.
//   k_tile_write_3d   resolves the label of every run (segment prefix + rank among the segment's roots)
//                     and writes int32 voxels with 16-byte stores.
//
// Volume layout is the reference's cv::Mat 3-D order [d0][d1][d2] with d2 fastest
// (Read3DImage, main.cpp:191-203; kernel addressing x*h*d + y*d + z, LabelingAlgs.cl:974).
// Mask bit v = 4i + 2j + k is the voxel at offset (i, j, k) in (d0, d1, d2); the lowest set bit
// is the block's first voxel in raster order.
//
// Block connectivity.  Two blocks A and B = A + d are 26-connected iff A has a foreground voxel
// on its side facing B and B has one on its side facing A: along an axis with d = -1 only offset
// 0 of A and offset 1 of B can touch, along an axis with d = 0 every offset can.  This is the
// predicate the reference evaluates voxel by voxel with TEST_CONN1/2/4 (LabelingAlgs.cl:770-856).
//
// Within a tile runs are numbered by block row; the union-find entries carry the slot (b0, i, b1, j, b2)
// of a run, (i, j) being the voxel row of its first voxel, whose order is the raster order of first
// voxels, and the atomicMin union keeps the smaller slot as the root: the root run of a component holds
// its first voxel.
#include "be_common.cuh"
#include "be_kernels.h"
#include "be_scan.cuh"

#include "be_api_internal.h"

#include <algorithm>

namespace be {

namespace {

constexpr int TB0 = T3_TB0, TB1 = T3_TB1, TB2 = T3_TB2;   // tile in blocks
constexpr int TX = 2 * TB0, TY = 2 * TB1, TZ = 2 * TB2;   // tile in voxels
constexpr int NBLK = T3_NBLK;
constexpr int MAXB = T3_MAXB;
constexpr int NT = kT3Threads;
constexpr int NROW = T3_NROW;               // block rows along d2 per tile: one 32-bit word each

static_assert(TB2 == 32, "a block row along d2 is one 32-bit word");
static_assert(NBLK <= 4096, "a run number must fit 12 bits");
static_assert(MAXB <= 2048, "node indices of the merge queue");

// A tile's border as the merge kernel reads it (Work::perim, uint16): for every run the node of its
// component, where that is one (T3_NBLK); for every block row the nodes of its first and last block's
// runs, low and high half of a word (2 * NROW); and for every block row the voxels of the first block on
// the - d2 face and of the last block on the + d2 face, as bits 2i + j of the low and high half of a
// byte (NROW / 2).
constexpr int kZNode = NBLK, kZFace = NBLK + 2 * NROW;
static_assert(T3_EDGE == kZFace + NROW / 2 && T3_EDGE % 2 == 0, "border words");
constexpr uint32_t kNoNode = 0xFFFFu;

// A tile's labels as the write kernel reads them (Work::lab), in 32-bit words: the voxel-class words
// 0..3 and 4..7 of its block rows (two arrays of uint4), (run starts, runs before, starts whose first
// voxel is of voxel row (0, 0), of (0, 1)) and the starts of voxel row (1, 0) per row, then the root run
// of every run (uint16).
constexpr int kHdr3 = 13 * NROW;
static_assert(T3_LAB_WORDS == kHdr3 + NBLK / 2, "tile words");
static_assert(TZ / 2 <= 0xFF, "a segment's root count fits its uint8");

// Of the starts, those of voxel row ij (2i + j) of their block row: the four sets of `first voxel in that
// voxel row`.
__device__ __forceinline__ uint32_t starts_of(int ij, uint32_t S, uint32_t S00, uint32_t S01, uint32_t S10)
{
    return ij == 0 ? S00 : ij == 1 ? S01 : ij == 2 ? S10 : S & ~(S00 | S01 | S10);
}

// Global keys: segment (one voxel row inside one tile, numbered in raster order) * seg_width + the place
// of the root run among the runs whose first voxel is in that segment -- the order of the components'
// first voxels.
__device__ __forceinline__ uint32_t seg_width3(const Img3D &im) { return uint32_t(min(im.d2, TZ) + 1) >> 1; }

// Selector over face bits (a*2 + b) for the tangent offsets (da, db).
__device__ __forceinline__ uint32_t face_sel(int da, int db)
{
    const uint32_t sa = da < 0 ? 0x3u : da > 0 ? 0xCu : 0xFu;
    const uint32_t sb = db < 0 ? 0x5u : db > 0 ? 0xAu : 0xFu;
    return sa & sb;
}

struct TileGeo {
    int tx0, tx1, tx2;      // tile coordinates
    int x0, y0, z0;         // first voxel
    int nx, ny, nz;         // valid voxels
    int n0, n1, n2;         // valid blocks
};

__device__ __forceinline__ TileGeo tile_geo(const Img3D &im, int64_t t)
{
    TileGeo g;
    const uint32_t lt = uint32_t(t - im.tile_base);   // (an image has fewer than 2^31 tiles)
    const uint32_t l12 = lt / uint32_t(im.t2);
    g.tx2 = int(lt - l12 * uint32_t(im.t2));
    g.tx0 = int(l12 / uint32_t(im.t1));
    g.tx1 = int(l12 - uint32_t(g.tx0) * uint32_t(im.t1));
    g.x0 = g.tx0 * TX; g.y0 = g.tx1 * TY; g.z0 = g.tx2 * TZ;
    g.nx = min(TX, im.d0 - g.x0); g.ny = min(TY, im.d1 - g.y0); g.nz = min(TZ, im.d2 - g.z0);
    g.n0 = (g.nx + 1) >> 1; g.n1 = (g.ny + 1) >> 1; g.n2 = (g.nz + 1) >> 1;
    return g;
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Tile-local labeling.  One thread per block row along d2: the tile is TB2 = 32 blocks deep, so a
// row is one 32-bit word per voxel class (v = 4i + 2j + k, the voxel's offsets in its block).
// Faces, runs along d2, run starts and the links to the four preceding rows are bit operations;
// only runs enter the union-find, ordered by the raster position of their first voxel.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int NT1 = kT3LocalThreads;   // threads of the tile-local kernel: one per block row
static_assert(NT1 == NROW && NT1 == 128, "thread layout");
constexpr int kRawWords = 3 * 4 * NROW;         // raw links of the rows (three uint4 per row)
constexpr int MQ1 = 2048;                       // union-queue capacity (more take further rounds)
static_assert(kRawWords <= MQ1, "the raw links live in the queue's memory");

// Word of the blocks whose side toward (dx, dy, dz) holds a foreground voxel: the OR of the
// classes with offset 0 along an axis where d < 0, offset 1 where d > 0.
template <int DX, int DY, int DZ>
__device__ __forceinline__ uint32_t face_word(const uint32_t (&c)[8])
{
    uint32_t r = 0;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        const int i = v >> 2, j = (v >> 1) & 1, k = v & 1;
        if ((DX < 0 && i) || (DX > 0 && !i) || (DY < 0 && j) || (DY > 0 && !j) || (DZ < 0 && k) || (DZ > 0 && !k))
            continue;
        r |= c[v];
    }
    return r;
}

// Slot of the run that starts at block b2 of row (b0, b1) and has its first voxel in the row's voxel
// row ij = 2i + j: the raster order of first voxels is the order of (b0, i, b1, j) and, in one voxel
// row, the order of the runs.
__device__ __forceinline__ uint32_t slot3(uint32_t b0, uint32_t b1, uint32_t ij, uint32_t b2)
{
    return (((b0 * 2 + (ij >> 1)) * TB1 + b1) * 2 + (ij & 1)) * TB2 + b2;
}

// Union-find over run numbers, the slot carried in the entry: (slot << 12) | parent, a root holding its
// own.  The union (atomicMin of the smaller entry into the other root, Playne-Hawick) leaves the run
// of the first voxel as the root.
__device__ __forceinline__ uint32_t efind3(uint32_t *P, uint32_t x, uint32_t &ev)
{
    uint32_t v = P[x];
    while ((v & 0xFFFu) != x) {
        const uint32_t y = v & 0xFFFu;
        const uint32_t vg = P[y];
        if ((vg & 0xFFFu) != y) P[x] = vg;   // path halving
        x = y;
        v = vg;
    }
    ev = v;
    return x;
}

__device__ __forceinline__ void eunion3(uint32_t *P, uint32_t a, uint32_t b)
{
    for (;;) {
        uint32_t ea, eb;
        a = efind3(P, a, ea);
        b = efind3(P, b, eb);
        if (a == b) return;
        const uint32_t hi = ea < eb ? b : a;
        const uint32_t old = atomicMin(&P[hi], min(ea, eb)) & 0xFFFu;
        if (old == hi) return;
        b = ea < eb ? a : b;
        a = old;
    }
}

// As sflatten_all, on entries: every run's entry becomes its root's.
__device__ __forceinline__ void eflatten3_all(uint32_t *P, uint32_t first, uint32_t step, uint32_t n)
{
    for (uint32_t i = first; i < n; i += step) {
        uint32_t x = P[i] & 0xFFFu;
        if (x == i) continue;
        uint32_t v = P[x];
        while ((v & 0xFFFu) != x) {
            x = v & 0xFFFu;
            v = P[x];
        }
        P[i] = v;
    }
}

// As shook_pairs, on entries.
__device__ __forceinline__ uint32_t ehook3_pairs(uint32_t *P, uint32_t *q, uint32_t n)
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
        const uint32_t keep = __ballot_sync(0xFFFFFFFFu, x != y);
        if (x != y) {
            atomicMin(&P[max(x, y) & 0xFFFu], min(x, y));
            q[kept + __popc(keep & ((1u << lane) - 1u))] = ((x & 0xFFFu) << 16) | (y & 0xFFFu);
        }
        kept += __popc(keep);
    }
    __syncwarp();
    return kept;
}

// Of the run starts S, those whose run holds a bit of x (every bit of x lies in a run): from each bit a
// carry runs down -- in reversed bits -- to the start it belongs to.
__device__ __forceinline__ uint32_t starts_with(uint32_t S, uint32_t x)
{
    const uint32_t rS = __brev(S), rx = __brev(x);
    return __brev(((~rS + (rx & ~rS)) | rx) & rS);
}

// Links of a block row (classes c, joins hz) to its preceding row nr -- 0..2: d0-1 with d1-1 / d1 / d1+1,
// 3: d0 with d1-1 -- whose classes are ua, ub and joins uhz, at the offsets dz = 0 / -1 / +1 along d2 (n /
// w / e).  raw: as found.  Returned: without those that an earlier one (further along d2, or dz = 0
// before dz = +-1 at the same block) stands for because it joins the same two runs.
struct Links {
    uint32_t n, w, e;
};
__device__ __forceinline__ Links row_links(int nr, const uint32_t (&c)[8], uint32_t hz, uint4 ua, uint4 ub, uint32_t uhz,
                                           Links &raw)
{
    const uint32_t u[8] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
    uint32_t A0, Am, Ap, B0, Bm, Bp;   // own sides toward dz = 0/-1/+1, neighbour's opposite sides
    if (nr == 0) {
        A0 = face_word<-1, -1, 0>(c); Am = face_word<-1, -1, -1>(c); Ap = face_word<-1, -1, 1>(c);
        B0 = face_word<1, 1, 0>(u); Bm = face_word<1, 1, 1>(u); Bp = face_word<1, 1, -1>(u);
    } else if (nr == 1) {
        A0 = face_word<-1, 0, 0>(c); Am = face_word<-1, 0, -1>(c); Ap = face_word<-1, 0, 1>(c);
        B0 = face_word<1, 0, 0>(u); Bm = face_word<1, 0, 1>(u); Bp = face_word<1, 0, -1>(u);
    } else if (nr == 2) {
        A0 = face_word<-1, 1, 0>(c); Am = face_word<-1, 1, -1>(c); Ap = face_word<-1, 1, 1>(c);
        B0 = face_word<1, -1, 0>(u); Bm = face_word<1, -1, 1>(u); Bp = face_word<1, -1, -1>(u);
    } else {
        A0 = face_word<0, -1, 0>(c); Am = face_word<0, -1, -1>(c); Ap = face_word<0, -1, 1>(c);
        B0 = face_word<0, 1, 0>(u); Bm = face_word<0, 1, 1>(u); Bp = face_word<0, 1, -1>(u);
    }
    const uint32_t hl = hz << 1, uhl = uhz << 1;
    raw = Links{A0 & B0, Am & (Bm << 1), Ap & (Bp >> 1)};
    const uint32_t Nsh = raw.n << 1, NEsh = raw.e << 1;
    return Links{raw.n & ~(hl & ((Nsh & uhl) | NEsh)), raw.w & ~((raw.n & uhl) | (hl & Nsh)),
                 raw.e & ~((raw.n & uhz) | (hl & NEsh & uhz))};
}

// Joins along d2 of a row's classes: bit k, block k touches block k + 1.
__device__ __forceinline__ uint32_t row_joins(const uint32_t (&c)[8])
{
    return face_word<0, 0, 1>(c) & (face_word<0, 0, -1>(c) >> 1);
}

// Class words of the CTA's block rows of a tile whose rows are whole and 16-byte aligned (p: its first
// voxel; rs0, rs1: strides of d0 and d1; nx, ny: voxels inside the volume).  A warp instruction reads
// whole 64-byte rows, four lanes a row -- with each thread reading its own four rows every load touched
// 32 cache lines, and those lookups took 60% of the load / store unit's time.  Lane 4 Y' + j of a warp loads
// chunk j of row Y of every plane X; two exchanges inside the four lanes leave lane j the words of planes
// 4 j .. 4 j + 3, and one with the lanes of row Y ^ 1 leaves it the two planes of block row (load_b0(tid),
// load_b1(tid)) in both rows.
__device__ __forceinline__ int load_b0(int tid) { return 2 * (tid & 3) + ((tid >> 2) & 1); }
__device__ __forceinline__ int load_b1(int tid) { return tid >> 3; }
static_assert(TB0 == 8 && TY * 4 == NT1, "the load's lanes");
__device__ __forceinline__ void load_rows(const uint8_t *p, int64_t rs0, int64_t rs1, int nx, int ny, uint32_t K, bool hi,
                                          uint32_t (&c)[8])
{
    const int Y = int(threadIdx.x) >> 2, j = int(threadIdx.x) & 3, s = Y & 1;
    const uint4 *q = reinterpret_cast<const uint4 *>(p + Y * rs1) + j;
    const int64_t step = rs0 / 16;
    uint32_t r[8];   // bytes: even and odd bits of plane k, of plane k + 8
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint4 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = 8 * h + k < nx && Y < ny ? __ldg(q + (8 * h + k) * step) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint32_t ev, od;
            split16(v[k], K, hi, ev, od);
            if (8 * h + k >= nx || Y >= ny) ev = od = 0;
            const uint32_t x = ev | (od << 8);
            r[k] = h ? r[k] | (x << 16) : x;
        }
    }
    // Lanes 0, 1 of the four keep planes 0..7, lanes 2, 3 planes 8..15.
    uint32_t own[4], oth[4];   // planes 2 m, 2 m + 1 of the kept eight: chunk j, chunk j ^ 2
    const bool up = j & 2;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        own[m] = __byte_perm(r[2 * m], r[2 * m + 1], up ? 0x7632 : 0x5410);
        oth[m] = __shfl_xor_sync(0xFFFFFFFFu, __byte_perm(r[2 * m], r[2 * m + 1], up ? 0x5410 : 0x7632), 2);
    }
    // Then lanes 0, 2 the first four of their eight planes, lanes 1, 3 the others.
    const bool hi2 = j & 1;
    uint32_t W[4][2];   // planes 4 j + 0..3: even, odd words
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const uint32_t a = hi2 ? own[m + 2] : own[m], b = hi2 ? oth[m + 2] : oth[m];                 // chunks j, j ^ 2
        const uint32_t x = __shfl_xor_sync(0xFFFFFFFFu, hi2 ? own[m] : own[m + 2], 1);               // chunk j ^ 1
        const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, hi2 ? oth[m] : oth[m + 2], 1);               // chunk j ^ 3
        const uint32_t a0 = hi2 ? x : a, a1 = hi2 ? a : x, b0 = hi2 ? y : b, b1 = hi2 ? b : y;
        const uint32_t k0 = up ? b0 : a0, k1 = up ? b1 : a1, k2 = up ? a0 : b0, k3 = up ? a1 : b1;   // chunks 0..3
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t lo = __byte_perm(k0, k1, h ? 0x7362 : 0x5140), hi4 = __byte_perm(k2, k3, h ? 0x7362 : 0x5140);
            W[2 * m + h][0] = __byte_perm(lo, hi4, 0x5410);
            W[2 * m + h][1] = __byte_perm(lo, hi4, 0x7632);
        }
    }
    // Planes 2 s, 2 s + 1 of the four stay, the others go to the lane of the row beside.
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t keep = s ? W[2 + i][k] : W[i][k];
            const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, s ? W[i][k] : W[2 + i][k], 4);
            c[4 * i + k] = s ? got : keep;        // row 2 b1
            c[4 * i + 2 + k] = s ? keep : got;    // row 2 b1 + 1
        }
}

// row_bits out of line: inlined into the four unrolled rows it slowed the aligned path by 1%.
__device__ __noinline__ uint2 row_bits_call(const uint8_t *p, int n, const uint8_t *lo, const uint8_t *hi,
                                            uint32_t K, bool thr_hi, int thr)
{
    uint2 r;
    row_bits(p, n, lo, hi, K, thr_hi, thr, r.x, r.y);
    return r;
}

}  // namespace

// One thread per block row (32 blocks along d2, one word per voxel class).  Bound by instruction issue
// and shared-memory latency: of a tile's time on noise of density 0.3, 13% are the loads, 16% links and
// first links, 18% queueing the other links and flattening, 38% the unions of about 700 kept links, 10%
// nodes and border data; on smooth fields (long runs) the loads are a third.  Measured (this launch on
// 512^3, us; slots of first voxels as run numbers and every link a union -> dense run numbers, links that
// close a triangle dropped, hooking before the unions, whole-row loads): density 0.3 390 -> 199, smooth
// half-full fields 196 -> 87.  128 threads, 31 KB and 72 registers: 7 CTAs per SM.
template <bool Q>
__global__ void __launch_bounds__(NT1, kT3LocalPerSM) k_tile_local_3d(ImgList3D L, Work w)
{
    grid_dep_release();   // the merge launch may take free SMs during this grid's last wave
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // a new epoch for the segment scan of this run
        w.epoch[0] += 1u;
        w.epoch[1] = 0u;
    }
    __shared__ uint32_t P[NBLK];               // per run: (slot << 12) | parent
    __shared__ __align__(16) uint4 CA[NROW], CB[NROW];   // class words 0..3, 4..7 of every row
    __shared__ __align__(16) uint4 WR[NROW];   // run starts, joins along d2, runs before, -
    __shared__ __align__(16) uint32_t MQ[MQ1]; // raw links, then the union queue: (run_a << 16) | run_b
    __shared__ uint32_t BF[NBLK / 32];         // runs that are border components
    __shared__ uint32_t BP[NBLK / 32];         // nodes before each word of BF
    __shared__ uint32_t mqn;
    __shared__ uint32_t wtot[NT1 / 32], ntot[NBLK / 32 / 32];
    __shared__ uint32_t qslot;
    uint4 *const RW = reinterpret_cast<uint4 *>(MQ);   // raw links: of row r straight below, below right, beside

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = tid / TB1, b1 = tid % TB1;
    uint32_t *lab = reinterpret_cast<uint32_t *>(w.lab);
    ItemLoop<Q> loop{w.queue + 0};
    for (int64_t t = loop.first(&qslot); t < w.n_tiles; t = loop.next(t, &qslot)) {
        const Img3D im = L.find(t, w.timg);
        const TileGeo g = tile_geo(im, t);
        const uint32_t K = (0x7Fu - (uint32_t(im.thr) & 0x7Fu)) * 0x01010101u;
        const bool hi = im.thr >= 128;
        const int64_t rs0 = int64_t(im.d1) * im.d2;   // stride of d0 in voxels

        BF[tid] = 0;
        if (tid == 0) mqn = 0;

        // Phase A: class words, runs along d2, run numbers.
        uint32_t c[8];
#pragma unroll
        for (int v = 0; v < 8; ++v) c[v] = 0;
        if (g.nz == TZ && ((reinterpret_cast<uintptr_t>(im.in) | uintptr_t(im.d2)) & 15) == 0) {
            // The lanes that loaded a row are not those that go on with it: through shared memory.
            load_rows(im.in + g.x0 * rs0 + int64_t(g.y0) * im.d2 + g.z0, rs0, im.d2, g.nx, g.ny, K, hi, c);
            const int row = load_b0(tid) * TB1 + load_b1(tid);
            CA[row] = make_uint4(c[0], c[1], c[2], c[3]);
            CB[row] = make_uint4(c[4], c[5], c[6], c[7]);
            __syncthreads();
            const uint4 ca = CA[tid], cb = CB[tid];
            c[0] = ca.x; c[1] = ca.y; c[2] = ca.z; c[3] = ca.w;
            c[4] = cb.x; c[5] = cb.y; c[6] = cb.z; c[7] = cb.w;
        } else if (b0 < g.n0 && b1 < g.n1) {
#pragma unroll
            for (int ij = 0; ij < 4; ++ij) {
                const int X = 2 * b0 + (ij >> 1), Y = 2 * b1 + (ij & 1);
                if (X >= g.nx || Y >= g.ny) continue;
                const uint8_t *row = im.in + (g.x0 + X) * rs0 + int64_t(g.y0 + Y) * im.d2 + g.z0;
                const uint2 eo = row_bits_call(row, g.nz, im.in, im.in + im.d0 * rs0, K, hi, im.thr);
                c[2 * ij] = eo.x;
                c[2 * ij + 1] = eo.y;
            }
        }
        const uint32_t Fw = c[0] | c[1] | c[2] | c[3] | c[4] | c[5] | c[6] | c[7];
        const uint32_t hz = row_joins(c);                                          // k joined to k + 1
        const uint32_t hl = hz << 1;                                               // k joined to k - 1
        const uint32_t S = Fw & ~hl;
        // The voxel row of each run's first voxel.
        const uint32_t S00 = starts_with(S, c[0] | c[1]);
        const uint32_t S01 = starts_with(S, c[2] | c[3]) & ~S00;
        const uint32_t S10 = starts_with(S, c[4] | c[5]) & ~(S00 | S01);
        uint32_t incl = __popc(S);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) wtot[warp] = incl;
        CA[tid] = make_uint4(c[0], c[1], c[2], c[3]);
        CB[tid] = make_uint4(c[4], c[5], c[6], c[7]);
        WR[tid] = make_uint4(S, hz, incl - __popc(S), 0u);
        __syncthreads();
        uint32_t woff = 0, nrun = 0;
#pragma unroll
        for (int i = 0; i < NT1 / 32; ++i) {
            const uint32_t n = wtot[i];
            if (i < warp) woff += n;
            nrun += n;
        }
        const uint32_t base = woff + incl - __popc(S);
        {
            uint32_t *h = lab + t * T3_LAB_WORDS;
            reinterpret_cast<uint4 *>(h)[tid] = make_uint4(c[0], c[1], c[2], c[3]);
            reinterpret_cast<uint4 *>(h)[NROW + tid] = make_uint4(c[4], c[5], c[6], c[7]);
            reinterpret_cast<uint4 *>(h)[2 * NROW + tid] = make_uint4(S, base, S00, S01);
            h[12 * NROW + tid] = S10;
        }

        // Phase B: links to the four preceding rows, as found and with the ones dropped that an earlier
        // link to the same row stands for.
        uint32_t LN[4], LW[4], LE[4];
        uint32_t n1 = 0, w1 = 0, e1 = 0, n3 = 0, w3 = 0, e3 = 0;   // as found, straight below and beside
        uint32_t n2 = 0, w2 = 0, e2 = 0;                           // below right
#pragma unroll
        for (int nr = 0; nr < 4; ++nr) {
            const int r0 = b0 + (nr < 3 ? -1 : 0), r1 = b1 + (nr < 3 ? nr - 1 : -1);
            Links l{0u, 0u, 0u}, raw{0u, 0u, 0u};
            if (Fw && r0 >= 0 && r1 >= 0 && r1 < TB1) {
                const int ur = r0 * TB1 + r1;
                l = row_links(nr, c, hz, CA[ur], CB[ur], WR[ur].y, raw);
            }
            if (nr == 1) { n1 = raw.n; w1 = raw.w; e1 = raw.e; }
            if (nr == 2) { n2 = raw.n; w2 = raw.w; e2 = raw.e; }
            if (nr == 3) { n3 = raw.n; w3 = raw.w; e3 = raw.e; }
            LN[nr] = l.n;
            LW[nr] = l.w;
            LE[nr] = l.e;
        }
        RW[tid] = make_uint4(n1, w1, e1, 0u);
        RW[NROW + tid] = make_uint4(n2, w2, e2, 0u);
        RW[2 * NROW + tid] = make_uint4(n3, w3, e3, 0u);
        __syncthreads();
        // A link is also dropped when two others close a triangle with it over a block of the row
        // straight below, or beside: own - below left over own - below and below - below left, and so
        // on, all as found, dropped or not.  Every reason uses links of earlier rows, or of this
        // row to `below` (dropped only by the rules above) or `beside` (dropped only over `below`), so
        // the reasons of a dropped link end at links that are kept.  This keeps 65% of the links of
        // Bernoulli 0.3 and 39% of those of 0.5 for about 60 instructions a row.
        {
            const uint4 z = make_uint4(0u, 0u, 0u, 0u);
            const uint4 p = b0 > 0 ? RW[2 * NROW + tid - TB1] : z;                      // below - below left
            const uint4 r = b0 > 0 && b1 + 1 < TB1 ? RW[2 * NROW + tid - TB1 + 1] : z;   // below right - below
            const uint4 s = b1 > 0 ? RW[tid - 1] : z;                                   // beside - below left
            const uint4 v = b1 > 0 ? RW[NROW + tid - 1] : z;                            // beside - below
            LN[0] &= ~((n1 & p.x) | (n3 & s.x));
            LW[0] &= ~((n1 & p.y) | (w1 & (p.x << 1)) | (n3 & s.y) | (w3 & (s.x << 1)));
            LE[0] &= ~((n1 & p.z) | (e1 & (p.x >> 1)) | (n3 & s.z) | (e3 & (s.x >> 1)));
            LN[2] &= ~(n1 & r.x);
            LW[2] &= ~((n1 & (r.z << 1)) | (w1 & (r.x << 1)));
            LE[2] &= ~((n1 & (r.y >> 1)) | (e1 & (r.x >> 1)));
            LN[3] &= ~(n1 & v.x);
            LW[3] &= ~((n1 & (v.z << 1)) | (w1 & (v.x << 1)));
            LE[3] &= ~((n1 & (v.y >> 1)) | (e1 & (v.x >> 1)));
        }
        // The first link of a run into the preceding layer (d0 - 1, whose slots are all smaller than
        // this row's) becomes its parent by a plain store: straight below if it has one there, else
        // below left, else below right.  Its entry holds key 0, the smallest value.  The other runs are
        // roots for now, with their slot.  (First links by a carry, as in 2D, from the starts whose run
        // has a link.)
        auto up_row = [&](int nr) -> int { return tid + (nr < 3 ? nr - 1 - TB1 : -1); };
        auto take = [&](int nr, uint32_t uS, uint32_t ubase, uint32_t b, uint32_t &own, uint32_t &up) {
            const uint32_t bit = 1u << b, upto = (bit << 1) - 1u;
            own = base + __popc(S & upto) - 1u;
            const bool isN = LN[nr] & bit, isW = !isN && (LW[nr] & bit), isE = !isN && !isW;
            LN[nr] &= isN ? ~bit : ~0u;
            LW[nr] &= isW ? ~bit : ~0u;
            LE[nr] &= isE ? ~bit : ~0u;
            up = ubase + __popc(uS & (isN ? upto : isW ? bit - 1u : (bit << 2) - 1u)) - 1u;   // (b = 30: all)
        };
        auto warp_base = [&](int row) -> uint32_t {   // runs before the warp of a row
            uint32_t n = 0;
#pragma unroll
            for (int i = 0; i < NT1 / 32 - 1; ++i)
                if (i < (row >> 5)) n += wtot[i];
            return n;
        };
        uint32_t rem = S;   // runs without a parent
#pragma unroll
        for (int o = 0; o < 3; ++o) {
            const int nr = o == 0 ? 1 : o == 1 ? 0 : 2;
            const uint32_t lk = LN[nr] | LW[nr] | LE[nr];
            if (!lk) continue;
            const uint32_t with = starts_with(S, lk) & rem;
            uint32_t first = lk & ((~lk + (with & ~lk)) | with);
            rem &= ~with;
            const int ur = up_row(nr);
            const uint4 uw = WR[ur];
            const uint32_t ub = uw.z + warp_base(ur);
            while (first) {
                const uint32_t b = __ffs(first) - 1;
                first &= first - 1;
                uint32_t own, up;
                take(nr, uw.x, ub, b, own, up);
                if (GUARD(w, own < nrun && up < own, 101, (uint64_t(own) << 32) | up)) P[own & (NBLK - 1)] = up & (NBLK - 1);
            }
        }
        for (uint32_t ss = rem; ss; ss &= ss - 1) {
            const uint32_t b = __ffs(ss) - 1, bit = 1u << b;
            const uint32_t ij = (S00 & bit) ? 0u : (S01 & bit) ? 1u : (S10 & bit) ? 2u : 3u;
            const uint32_t id = base + __popc(S & (bit - 1u));
            P[id] = (slot3(b0, b1, ij, b) << 12) | id;
        }
        // The remaining links are unions: queued and merged by every lane.
        uint32_t n = 0;
#pragma unroll
        for (int nr = 0; nr < 4; ++nr) n += __popc(LN[nr]) + __popc(LW[nr]) + __popc(LE[nr]);
        uint32_t pos = warp_reserve(&mqn, n);
        auto push = [&](uint32_t lo, uint32_t end) {   // links at queue positions [lo, end) go in
#pragma unroll
            for (int nr = 0; nr < 4; ++nr) {
                if (!(LN[nr] | LW[nr] | LE[nr])) continue;
                const int ur = up_row(nr);
                const uint4 uw = WR[ur];
                const uint32_t ub = uw.z + warp_base(ur);
                while (pos < end) {
                    const uint32_t b = __ffs(LN[nr] | LW[nr] | LE[nr]);
                    if (!b) break;
                    uint32_t own, up;
                    take(nr, uw.x, ub, b - 1u, own, up);
                    MQ[pos - lo] = GUARD(w, own < nrun && up < own, 103, (uint64_t(own) << 32) | up) ? (own << 16) | up : 0u;
                    ++pos;
                }
            }
        };
        __syncthreads();   // the raw links are used up
        push(0u, uint32_t(MQ1));
        // The forest of first links is flattened before the unions, as in 2D.
        eflatten3_all(P, tid, NT1, nrun);
        __syncthreads();
        const uint32_t total = mqn;
        for (uint32_t lo = 0; lo < total; lo += MQ1) {
            if (lo) {
                eflatten3_all(P, tid, NT1, nrun);   // ehook3_pairs wants every run at its root
                push(lo, lo + MQ1);
                __syncthreads();
            }
            const uint32_t nq = min(total - lo, uint32_t(MQ1)), per = (nq + NT1 / 32 - 1) / (NT1 / 32);
            const uint32_t q0 = min(nq, warp * per);
            const uint32_t kept = ehook3_pairs(P, MQ + q0, min(nq - q0, per));
            __syncthreads();
            for (uint32_t k = lane; k < kept; k += 32) eunion3(P, MQ[q0 + k] >> 16, MQ[q0 + k] & 0xFFFFu);
            __syncthreads();
        }

        // Phase C: every run's entry becomes its root's.
        if (total) eflatten3_all(P, tid, NT1, nrun);
        __syncthreads();
        loop.request();
        // Phase D: the root bitmap (a bit per run start, so a word per row) and the segments' root
        // counts.
        uint32_t roots = 0;
        for (uint32_t ss = rem; ss; ss &= ss - 1) {
            const uint32_t bit = ss & (0u - ss);
            const uint32_t id = base + __popc(S & (bit - 1u));
            if ((P[id] & 0xFFFu) == id) roots |= bit;
        }
        w.rbits[t * NROW + tid] = roots;
#pragma unroll
        for (int ij = 0; ij < 4; ++ij) {
            const int X = 2 * b0 + (ij >> 1), Y = 2 * b1 + (ij & 1);
            if (X >= g.nx || Y >= g.ny) continue;
            const int64_t si = im.seg_base + (int64_t(g.x0 + X) * im.d1 + (g.y0 + Y)) * im.t2 + g.tx2;
            if (GUARD(w, si >= 0 && si < w.n_segs, 104, si)) w.segcnt[si] = uint8_t(__popc(roots & starts_of(ij, S, S00, S01, S10)));
        }
        // Border components -> nodes: the runs of the rows on a face that has a tile behind it, and the
        // runs of the first and last blocks of every row where a tile lies behind those.
        const bool zlo = g.tx2 > 0 && (S & 1u), zhi = g.tx2 + 1 < im.t2 && (Fw >> 31);
        {
            const bool face = (b0 == 0 && g.tx0 > 0) || (b0 == TB0 - 1 && g.tx0 + 1 < im.t0) || (b1 == 0 && g.tx1 > 0) ||
                              (b1 == TB1 - 1 && g.tx1 + 1 < im.t1);
            uint32_t ss = face ? S : (zlo ? 1u : 0u) | (zhi ? 0x80000000u >> __clz(S) : 0u);
            for (; ss; ss &= ss - 1) {
                const uint32_t id = base + __popc(S & ((ss & (0u - ss)) - 1u));
                const uint32_t rt = P[id] & 0xFFFu;
                atomicOr(&BF[rt >> 5], 1u << (rt & 31));
            }
        }
        __syncthreads();
        uint32_t nin = __popc(BF[tid]);   // nodes up to this word, within the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, nin, o);
            if (lane >= o) nin += v;
        }
        BP[tid] = nin - __popc(BF[tid]);
        if (lane == 31) ntot[warp] = nin;
        __syncthreads();
        uint32_t noff[NBLK / 32 / 32 + 1];
        noff[0] = 0;
#pragma unroll
        for (int i = 0; i < NBLK / 32 / 32; ++i) noff[i + 1] = noff[i] + ntot[i];
        auto node_of = [&](uint32_t rt) -> uint32_t {   // node of a root run's component
            const uint32_t f = BF[rt >> 5], bit = 1u << (rt & 31), q = rt >> 10;
            if (!(f & bit)) return kNoNode;
            return (q == 0 ? noff[0] : q == 1 ? noff[1] : q == 2 ? noff[2] : noff[3]) + BP[rt >> 5] + __popc(f & (bit - 1u));
        };
        // Node records, by the row of the root run; root and node of every run; the row's ends.
        for (uint32_t ss = roots; ss; ss &= ss - 1) {
            const uint32_t bit = ss & (0u - ss), id = base + __popc(S & (bit - 1u));
            const uint32_t j = node_of(id);
            if (j == kNoNode) continue;
            if (!GUARD(w, j < uint32_t(MAXB), 102, j)) break;
            const uint32_t ij = (S00 & bit) ? 0u : (S01 & bit) ? 1u : (S10 & bit) ? 2u : 3u;
            const uint32_t place = __popc(starts_of(int(ij), S, S00, S01, S10) & (bit - 1u));
            const int64_t seg = (int64_t(g.x0 + 2 * b0 + (ij >> 1)) * im.d1 + (g.y0 + 2 * b1 + (ij & 1))) * im.t2 + g.tx2;
            const int64_t node = t * MAXB + j;
            w.nroot[node] = uint16_t(tid * TB2 + __ffs(bit) - 1);
            w.gp[node] = gentry(uint32_t(seg) * seg_width3(im) + place, uint32_t(node));
        }
        {
            uint32_t *rl = lab + t * T3_LAB_WORDS + kHdr3;
            uint32_t *nl = reinterpret_cast<uint32_t *>(w.perim + t * T3_EDGE);
            for (uint32_t i = 2 * tid; i < nrun; i += 2 * NT1) {
                const uint32_t ra = P[i] & 0xFFFu, rb = P[i + 1 < nrun ? i + 1 : i] & 0xFFFu;
                rl[i >> 1] = ra | (rb << 16);
                nl[i >> 1] = node_of(ra) | (node_of(rb) << 16);
            }
            const uint32_t na = zlo ? node_of(P[base] & 0xFFFu) : kNoNode;
            const uint32_t nz = zhi ? node_of(P[base + __popc(S) - 1u] & 0xFFFu) : kNoNode;
            nl[kZNode / 2 + tid] = na | (nz << 16);
            reinterpret_cast<uint8_t *>(w.perim + t * T3_EDGE + kZFace)[tid] =
                uint8_t((c[0] & 1u) | ((c[2] & 1u) << 1) | ((c[4] & 1u) << 2) | ((c[6] & 1u) << 3) | ((c[1] >> 31) << 4) |
                        ((c[3] >> 31) << 5) | ((c[5] >> 31) << 6) | ((c[7] >> 31) << 7));
        }
        if (tid == 0) w.nb[t] = noff[NBLK / 32 / 32];
        if (!Q) break;   // one tile per CTA
        loop.publish(&qslot);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Cross-tile merge.
// ---------------------------------------------------------------------------------------------
namespace {

// Union of two nodes of one volume; the root linked under the other leaves its segment's root
// count and its tile's root bitmap.
__device__ void gunion3d(const Img3D &im, Work &w, uint32_t a, uint32_t b)
{
    gunion_keyed(w.gp, a, b, [&](uint32_t node, uint32_t key) {
        dec_count<uint8_t>(w.segcnt, im.seg_base + key / seg_width3(im));
        const uint32_t blk = w.nroot[node];
        atomicAnd(w.rbits + int64_t(node / MAXB) * NROW + blk / TB2, ~(1u << (blk % TB2)));
    });
}

}  // namespace

// Cross-tile merge.  One CTA per tile: the links of its block rows to those of their four preceding rows
// that lie in other tiles, by the same bit operations as inside a tile (row_links), and the links of
// their first and last blocks across d2 to the tiles beside (one byte of face voxels per row and two
// nodes, written by the tile kernel).  Of the 512 (row, preceding row) pairs only 70 leave the tile: one
// warp takes those of one direction, a lane a pair.  The links go through a shared queue and are shared
// by all lanes; a pair of nodes that the CTA has just seen -- most links join the same few large
// components -- is dropped by a small table, and the others are unions, whose walks (dependent loads
// through L2) end as soon as the two sides have one parent.  Bound by the latency of its loads: 16 tiles
// in flight per SM (8 / 12 / 16: 127 / 110 / 107 us before the direction split).  Measured (this launch on
// 512^3, us; voxel pairs through a CTA-local union-find -> this): density 0.3 150 -> 68, smooth fields
// 143 -> 44, density 0.1 79 -> 70.
constexpr int kMQ3 = 1024;     // queued links (more take further rounds)
constexpr int kSeen3 = 256;    // table of node pairs seen

template <bool Q>
__global__ void __launch_bounds__(kT3MergeThreads, kT3MergePerSM) k_merge_3d(ImgList3D L, Work w)
{
    grid_dep_wait();
    grid_dep_release();
    __shared__ uint32_t LQ[kMQ3];
    __shared__ unsigned long long seen[kSeen3];
    __shared__ uint32_t nq;
    __shared__ uint32_t qslot;
    static_assert(kT3MergeThreads == NROW && TB1 + TB0 - 1 <= 32, "one thread per block row; a warp's lanes take a direction");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = tid / TB1, b1 = tid % TB1;
    const uint32_t *lab = reinterpret_cast<const uint32_t *>(w.lab);
    ItemLoop<Q> loop{w.queue + 1};
    for (int64_t t = loop.first(&qslot); t < w.n_tiles; t = loop.next(t, &qslot)) {
        const Img3D im = L.get(t, w.timg);
        loop.request();
        const TileGeo g = tile_geo(im, t);
        for (int i = tid; i < kSeen3; i += kT3MergeThreads) seen[i] = ~0ull;
        if (tid == 0) nq = 0;
        __syncthreads();

        // Preceding row nr of row (a, b): its row in its tile, and that tile's offset code
        // 4 * (o0 + 1) + (o1 + 1) with o0 in {-1, 0}; 16 when there is no such tile.
        auto preceding = [&](int a, int b, int nr, int &rr) -> int {
            const int r0 = a + (nr < 3 ? -1 : 0), r1 = b + (nr < 3 ? nr - 1 : -1);
            const int o0 = r0 < 0 ? -1 : 0, o1 = r1 < 0 ? -1 : r1 >= TB1 ? 1 : 0;
            rr = (r0 & (TB0 - 1)) * TB1 + (r1 & (TB1 - 1));
            if (g.tx0 + o0 < 0 || g.tx1 + o1 < 0 || g.tx1 + o1 >= im.t1) return 16;
            return 4 * (o0 + 1) + (o1 + 1);
        };
        auto tile_at = [&](int code, int o2) -> int64_t {
            const int64_t tt = t + (int64_t((code >> 2) - 1) * im.t1 + (code & 3) - 1) * im.t2 + o2;
            return GUARD(w, tt >= im.tile_base && tt < w.n_tiles, 201, tt) ? tt : t;
        };
        constexpr int kOwn = 5;   // code of the row's own tile
        // Links to rows of other tiles: warp 0 straight below (the rows of the first layer), warp 1 below
        // left (the first layer; the others' first row), warp 2 below right (.. last row), warp 3 beside
        // (every layer's first row).
        const int nr = warp == 0 ? 1 : warp == 1 ? 0 : warp;
        const int ra = nr == 3 ? lane : lane < TB1 ? 0 : lane - TB1 + 1;
        const int rb = nr == 3 ? 0 : lane < TB1 ? lane : nr == 0 ? 0 : TB1 - 1;
        Links lk{0u, 0u, 0u};
        uint32_t S = 0, base = 0, uS = 0, ubase = 0;
        int code = 16;
        if (ra < g.n0 && rb < g.n1 && lane < (nr == 1 ? TB1 : nr == 3 ? TB0 : TB1 + TB0 - 1)) {
            int rr;
            code = preceding(ra, rb, nr, rr);
            if (code != kOwn && code != 16) {
                const uint4 *h = reinterpret_cast<const uint4 *>(lab + t * T3_LAB_WORDS);
                const uint4 *uh = reinterpret_cast<const uint4 *>(lab + tile_at(code, 0) * T3_LAB_WORDS);
                const int row = ra * TB1 + rb;
                const uint4 ca = __ldcg(h + row), cb = __ldcg(h + NROW + row), rw = __ldcg(h + 2 * NROW + row);
                const uint4 ua = __ldcg(uh + rr), ub = __ldcg(uh + NROW + rr), uw = __ldcg(uh + 2 * NROW + rr);
                // Below left / right: also the row straight below, over which most of them are dropped.
                uint4 va = make_uint4(0, 0, 0, 0), vb = va;
                if (nr == 0 || nr == 2) {
                    int r1;
                    const int c1 = preceding(ra, rb, 1, r1);
                    if (c1 != 16) {
                        const uint4 *vh = reinterpret_cast<const uint4 *>(lab + tile_at(c1, 0) * T3_LAB_WORDS);
                        va = __ldcg(vh + r1);
                        vb = __ldcg(vh + NROW + r1);
                    }
                }
                const uint32_t c[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
                const uint32_t u[8] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
                const uint32_t v[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
                const uint32_t hz = row_joins(c), uhz = row_joins(u);
                S = rw.x;
                base = rw.y;
                uS = uw.x;
                ubase = uw.y;
                Links raw, r1, p;
                if (nr == 1) lk = row_links(1, c, hz, ua, ub, uhz, raw);
                else if (nr == 3) lk = row_links(3, c, hz, ua, ub, uhz, raw);
                else if (nr == 0) {   // the triangle rule of the tile kernel over own - below - below left
                    lk = row_links(0, c, hz, ua, ub, uhz, raw);
                    row_links(1, c, hz, va, vb, 0u, r1);
                    row_links(3, v, 0u, ua, ub, 0u, p);
                    lk.n &= ~(r1.n & p.n);
                    lk.w &= ~((r1.n & p.w) | (r1.w & (p.n << 1)));
                    lk.e &= ~((r1.n & p.e) | (r1.e & (p.n >> 1)));
                } else {              // over own - below - below right
                    lk = row_links(2, c, hz, ua, ub, uhz, raw);
                    row_links(1, c, hz, va, vb, 0u, r1);
                    row_links(3, u, 0u, va, vb, 0u, p);
                    lk.n &= ~(r1.n & p.n);
                    lk.w &= ~((r1.n & (p.e << 1)) | (r1.w & (p.n << 1)));
                    lk.e &= ~((r1.n & (p.w >> 1)) | (r1.e & (p.n >> 1)));
                }
            }
        }
        // Links across d2: bits 0..3, own first block to preceding row nr of the tiles before; bit 4, to
        // the same row; bits 5..8, own last block to preceding row nr of the tiles after.
        auto zface = [&](int64_t tt, int row) -> uint32_t {
            return __ldcg(reinterpret_cast<const uint8_t *>(w.perim + tt * T3_EDGE + kZFace) + row);
        };
        uint32_t zm = 0;
        if (b0 < g.n0 && b1 < g.n1) {
            const uint32_t f = zface(t, tid);
            const uint32_t lo = g.tx2 > 0 ? f & 15u : 0u, hi = g.tx2 + 1 < im.t2 ? f >> 4 : 0u;
            // The same row beside: a link before (after, one that the tile there makes), over which those
            // to the preceding rows that its face voxels touch too are dropped.
            const uint32_t before = lo ? zface(t - 1, tid) >> 4 : 0u, after = hi ? zface(t + 1, tid) & 15u : 0u;
            if (before) zm |= 16u;
            if (lo | hi) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int rr;
                    const int cd = preceding(b0, b1, k, rr);
                    if (cd == 16) continue;
                    const int dx = k < 3 ? -1 : 0, dy = k < 3 ? k - 1 : -1;
                    const uint32_t own = face_sel(dx, dy), opp = face_sel(-dx, -dy);
                    if ((lo & own) && !(before & own) && ((zface(tile_at(cd, -1), rr) >> 4) & opp)) zm |= 1u << k;
                    if ((hi & own) && !(after & own) && (zface(tile_at(cd, 1), rr) & opp)) zm |= 32u << k;
                }
            }
        }
        // Queue entries: run links, own run | other run << 12 | code << 24; links across d2, own node |
        // other node << 11 | code << 24 | (o2 < 0: 1, o2 > 0: 2) << 29.
        uint32_t pos = warp_reserve(&nq, __popc(zm) + __popc(lk.n) + __popc(lk.w) + __popc(lk.e));
        auto push = [&](uint32_t from, uint32_t end) {   // links at queue positions [from, end) go in
            while (pos < end) {
                const uint32_t f = __ffs(lk.n | lk.w | lk.e);
                if (!f) break;
                const uint32_t b = f - 1, bit = 1u << b, upto = (bit << 1) - 1u;
                const bool isN = lk.n & bit, isW = !isN && (lk.w & bit), isE = !isN && !isW;
                lk.n &= isN ? ~bit : ~0u;
                lk.w &= isW ? ~bit : ~0u;
                lk.e &= isE ? ~bit : ~0u;
                const uint32_t own = base + __popc(S & upto) - 1u;
                const uint32_t up = ubase + __popc(uS & (isN ? upto : isW ? bit - 1u : (bit << 2) - 1u)) - 1u;
                LQ[pos++ - from] = own | (up << 12) | (uint32_t(code) << 24);
            }
            if (zm && pos < end) {
                auto znodes = [&](int64_t tt, int row) -> uint32_t {
                    return __ldcg(reinterpret_cast<const uint32_t *>(w.perim + tt * T3_EDGE + kZNode) + row);
                };
                const uint32_t zo = znodes(t, tid);
                while (zm && pos < end) {
                    const int k = __ffs(zm) - 1;
                    zm &= zm - 1;
                    int rr = tid, cd = kOwn;
                    if (k != 4) cd = preceding(b0, b1, k < 4 ? k : k - 5, rr);
                    const uint32_t zu = znodes(tile_at(cd, k < 5 ? -1 : 1), rr);
                    const uint32_t a = k < 5 ? zo & 0xFFFFu : zo >> 16, b = k < 5 ? zu >> 16 : zu & 0xFFFFu;
                    LQ[pos++ - from] = a | (b << 11) | (uint32_t(cd) << 24) | (k < 5 ? 1u << 29 : 2u << 29);
                }
            }
        };
        push(0u, uint32_t(kMQ3));
        __syncthreads();
        const uint32_t total = nq;
        for (uint32_t from = 0; from < total; from += kMQ3) {
            if (from) {
                push(from, from + kMQ3);
                __syncthreads();
            }
            const uint32_t cnt = min(total - from, uint32_t(kMQ3));
            for (uint32_t i = tid; i < cnt; i += kT3MergeThreads) {
                const uint32_t e = LQ[i], z = e >> 29;
                const int64_t tt = tile_at(int(e >> 24) & 31, z == 0 ? 0 : z == 1 ? -1 : 1);
                uint32_t a, b;
                if (z) {
                    a = e & 0x7FFu;
                    b = (e >> 11) & 0x7FFu;
                } else {
                    if (!GUARD(w, (e & 0xFFFu) < uint32_t(NBLK) && ((e >> 12) & 0xFFFu) < uint32_t(NBLK), 203, e)) continue;
                    a = __ldcg(w.perim + t * T3_EDGE + (e & 0xFFFu));
                    b = __ldcg(w.perim + tt * T3_EDGE + ((e >> 12) & 0xFFFu));
                }
                if (!GUARD(w, a < w.nb[t] && b < w.nb[tt], 204, (uint64_t(tt) << 32) | e)) continue;
                const uint32_t nA = uint32_t(t * MAXB + a), nB = uint32_t(tt * MAXB + b);
                const unsigned long long key = (static_cast<unsigned long long>(nA) << 32) | nB;
                const uint32_t slot = (nA * 0x9E3779B1u ^ nB * 0x85EBCA77u) >> 24;
                static_assert(kSeen3 == 256, "eight hash bits");
                if (atomicExch(&seen[slot], key) == key) continue;   // the lane that put it there unites the two
                gunion3d(im, w, nA, nB);
            }
            __syncthreads();
        }
        if (!Q) break;   // one tile per CTA
        loop.publish(&qslot);
        __syncthreads();   // every lane has read this tile's count
    }
}

// ---------------------------------------------------------------------------------------------
// Segment scan and node links, one launch: items below n_chunks scan a chunk of segment counts
// (single pass, look-back); the others resolve the linked nodes of one tile (link_tile_nodes):
// each is pointed straight at its global root, and the segment and in-segment rank of that root's
// first voxel are stored with it.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kScanThreads) k_scan_link_3d(ImgList3D L, Work w)
{
    grid_dep_wait();
    grid_dep_release();   // after the wait: the label-write launch relies on it
    __shared__ uint32_t tmp[kScanThreads / 32 + 1];
    __shared__ uint32_t sh[2];
    const int64_t n = int64_t(w.n_chunks) + w.n_tiles;
    for (int64_t it = blockIdx.x; it < n; it += gridDim.x) {   // (in a fixed order: the items are short)
        if (it < w.n_chunks) {
            segscan_lb_chunk<kScanThreads>(w, tmp, sh);
            continue;
        }
        const int64_t t = it - w.n_chunks;
        const Img3D im = L.get(t, w.timg);
        link_tile_nodes(w, t, MAXB, [&](uint32_t root, uint32_t key, uint32_t &seg, uint32_t &rank) {
            // The root's segment, and the roots left in it before the root.
            const uint32_t sg = key / seg_width3(im), line = sg / uint32_t(im.t2);   // line = X * d1 + Y
            const uint32_t X = line / uint32_t(im.d1), Y = line - X * uint32_t(im.d1);
            const uint32_t blk = w.nroot[root], row = blk / TB2;
            const int64_t tile = root / MAXB;
            const uint32_t *h = reinterpret_cast<const uint32_t *>(w.lab) + tile * T3_LAB_WORDS;
            const uint4 rw = reinterpret_cast<const uint4 *>(h)[2 * NROW + row];
            const uint32_t st = starts_of(int(X & 1) * 2 + int(Y & 1), rw.x, rw.z, rw.w, h[12 * NROW + row]);
            rank = __popc(w.rbits[tile * NROW + row] & st & ((1u << (blk % TB2)) - 1u));
            seg = uint32_t(im.seg_base) + sg;
        });
    }
}

// ---------------------------------------------------------------------------------------------
// Label resolve and write.
// ---------------------------------------------------------------------------------------------
// As k_tile_write_2d, with the nodes' links resolved by the launch before and one lookup per block pair for
// its four voxel rows.  Bound by the stores: of 111 us for the 537 MB of a 512^3 volume a bare kernel that
// stores the same tiles takes 87.  4 CTAs of 256 threads per SM, for their 64 registers: with 6 / 5 / 4 / 3
// a 512^3 volume takes 121 / 114 / 111 / 110 us, a 511x511x509 one, whose rows have every alignment, - /
// 243 / 181 / 177, and 191x223x157 - / 24.5 / 18.6 / 24.
// CTAs per SM up to which CTAs share a tile's rows (191x223x157, 252 tiles: one CTA a tile 68.3 us, two
// 65.8; 200^3, 364 tiles: the same with 2 to 5).
constexpr int kSplitPerSM3 = 4;
constexpr int kNLCap = 512;        // node links a write CTA stages in shared memory (later ones: from L2)
constexpr int kStageRuns3 = 2048;  // run entries likewise

template <bool Q, bool SHARED>
__global__ void __launch_bounds__(NT, kT3WritePerSM) k_tile_write_3d(ImgList3D L, Work w)
{
    __shared__ __align__(16) uint4 H[3 * NROW];   // class words 0..3, 4..7, (starts, runs before, S00, S01)
    __shared__ uint32_t H10[NROW];
    __shared__ uint32_t LT[NBLK + 1];             // label of run i at i + 1
    __shared__ uint32_t RB[NROW];                 // roots left, a bit per run start
    __shared__ uint32_t segb[TX * TY + 1];   // segment prefixes of the tile's voxel rows; [TX * TY]: the volume's first
    __shared__ __align__(16) uint2 NL[kNLCap];
    __shared__ __align__(16) uint32_t E[kStageRuns3 / 2];
    __shared__ uint32_t snb;
    __shared__ uint32_t qslot;

    const int tid = threadIdx.x;
    const uint32_t *lab = reinterpret_cast<const uint32_t *>(w.lab);
    static_assert(3 * NROW <= 2 * NT && NROW <= NT, "tile words per thread");
    static_assert(TX * TY == 2 * NT && kNLCap == 2 * NT && kStageRuns3 == 8 * NT, "fetched words per thread");
    // The tile's words, root bitmaps and node counts were final before this grid's predecessor (the
    // scan and link pass) started: that grid waits for the merge to complete before it lets this
    // one launch.  So they are read before the wait -- the words into registers, the rest into shared
    // memory (cp.async) -- and the segment prefixes and node links, which the predecessor writes, are
    // copied after it.  The next tile's fetches are issued before the current tile's labels are written.
    uint4 nH[2];
    uint32_t n10 = 0;
    auto fetch = [&](int64_t t) {
        const uint32_t *h = lab + t * T3_LAB_WORDS;
        nH[0] = __ldcg(reinterpret_cast<const uint4 *>(h) + tid);
        if (tid + NT < 3 * NROW) nH[1] = __ldcg(reinterpret_cast<const uint4 *>(h) + tid + NT);
        if (tid < NROW) {
            n10 = __ldcg(h + 12 * NROW + tid);
            cp_async4(&RB[tid], w.rbits + t * NROW + tid);
        }
        cp_async16(&E[4 * tid], h + kHdr3 + 4 * tid);
        if (tid == NT - 1) cp_async4(&snb, w.nb + t);
        cp_async_commit();
    };
    auto fetch_links = [&](int64_t t) {
        const Img3D im = L.get(t, w.timg);
        const TileGeo g = tile_geo(im, t);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = tid + i * NT;
            cp_async8(&NL[r], w.nlink + t * MAXB + r);
            const int X = r / TY, Y = r % TY;
            if (X < g.nx && Y < g.ny)
                cp_async4(&segb[r], w.segpref + im.seg_base + (int64_t(g.x0 + X) * im.d1 + (g.y0 + Y)) * im.t2 + g.tx2);
        }
        if (tid == 0) cp_async4(&segb[TX * TY], w.segpref + im.seg_base);
        cp_async_commit();
    };
    ItemLoop<Q> loop{w.queue + 4};
    int64_t t = loop.first(&qslot);
    int part = 0, split = 1;   // of the tile's rows
    if (SHARED) {
        split = int(gridDim.x / uint32_t(w.n_tiles));
        part = int(blockIdx.x % uint32_t(split));
        t = blockIdx.x / uint32_t(split);
    }
    if (t < w.n_tiles) fetch(t);
    if (t < w.n_tiles) {
        grid_dep_wait();   // segment prefixes and node links from here on
        fetch_links(t);
    }
    while (t < w.n_tiles) {
        loop.request();
        const Img3D im = L.get(t, w.timg);
        const TileGeo g = tile_geo(im, t);
        const int64_t rs0 = int64_t(im.d1) * im.d2;
        H[tid] = nH[0];
        if (tid + NT < 3 * NROW) H[tid + NT] = nH[1];
        if (tid < NROW) H10[tid] = n10;
        cp_async_wait();
        __syncthreads();
        const uint32_t nb = snb, base0 = segb[TX * TY];
        const uint4 *HR = H + 2 * NROW;
        const uint32_t nrun = HR[NROW - 1].y + __popc(HR[NROW - 1].x);
        if (t == im.tile_base && tid == 0 && part == 0) {
            const int64_t n = int64_t(w.segpref[im.seg_base + int64_t(im.d0) * im.d1 * im.t2] - base0);
            w.ncomp[im.index] = n;
            if (w.host_count) *w.host_count = n;
        }
        // Surviving roots, by block row and voxel row: rank = roots before it in its segment.
#pragma unroll
        for (int i = 0; i < 4 * NROW / NT; ++i) {
            const int u = tid + i * NT, row = u / 4, ij = u % 4;
            const uint4 rw = HR[row];
            uint32_t bits = RB[row] & starts_of(ij, rw.x, rw.z, rw.w, H10[row]);
            uint32_t label = 1u + segb[(2 * (row / TB1) + (ij >> 1)) * TY + 2 * (row % TB1) + (ij & 1)] - base0;
            while (bits) {
                const uint32_t bit = bits & (0u - bits);
                if (!GUARD(w, rw.y + __popc(rw.x) <= uint32_t(NBLK), 401, rw.y)) break;
                LT[rw.y + __popc(rw.x & (bit | (bit - 1u)))] = label++;
                bits &= bits - 1;
            }
        }
        // Border components linked under another tile's component: the label of that root, its
        // segment's prefix plus its rank among the roots left there (both resolved by the link pass).
        for (uint32_t j = tid; j < nb; j += NT) {
            const uint2 e = j < uint32_t(kNLCap) ? NL[j] : __ldcg(w.nlink + t * MAXB + j);
            if (e.x == kNone) continue;
            const uint32_t blk = e.y >> 16;
            if (GUARD(w, blk < uint32_t(NBLK) && e.x < w.n_segs, 402, t * MAXB + j)) {
                const uint4 rw = HR[blk / TB2];
                LT[rw.y + __popc(rw.x & ((2u << (blk % TB2)) - 1u))] = 1u + (__ldcg(w.segpref + e.x) - base0) + (e.y & 0xFFFFu);
            }
        }
        __syncthreads();
        // Every other run takes the label of its root run.
        for (uint32_t i = 2 * tid; i < nrun; i += 2 * NT) {
            const uint32_t e = i < uint32_t(kStageRuns3) ? E[i >> 1] : __ldcg(lab + t * T3_LAB_WORDS + kHdr3 + (i >> 1));
            const uint32_t a = e & 0xFFFFu, b = e >> 16;
            if (!GUARD(w, a < nrun && (i + 1 >= nrun || b < nrun), 403, e)) continue;
            if (a != i) LT[i + 1] = LT[a + 1];
            if (i + 1 < nrun && b != i + 1) LT[i + 2] = LT[b + 1];
        }
        loop.publish(&qslot);
        __syncthreads();
        const int64_t tn = SHARED ? w.n_tiles : loop.next(t, &qslot);   // the next tile's data come while this one's labels go
        if (tn < w.n_tiles) {   // RB, NL, E, segb and snb are free now
            fetch(tn);
            fetch_links(tn);
        }

        // Output: one unit = two blocks along d2 in all four voxel rows (X, Y) they cover: the
        // labels are looked up once for four 16-byte stores.  A thread keeps its place along d2.
        const bool vec_ok = ((reinterpret_cast<uintptr_t>(im.out) | (uintptr_t(im.d2) * 4)) & 15) == 0;
        const int q = tid % (TB2 / 2);
        const uint32_t bit0 = 1u << (2 * q), bit1 = 2u << (2 * q), upto0 = bit0 | (bit0 - 1u);
        const int n = min(4, max(0, g.nz - 4 * q));   // voxels of the thread's place inside the volume
        for (int row = tid / (TB2 / 2) + NT / (TB2 / 2) * part; row < NROW; row += NT / (TB2 / 2) * split) {
            const int b0 = row / TB1, b1 = row % TB1;
            if (vec_ok && (n == 0 || 2 * b0 >= g.nx || 2 * b1 >= g.ny)) continue;
            const uint4 a = H[row], b = H[NROW + row], rw = HR[row];
            const uint32_t i0 = rw.y + __popc(rw.x & upto0);
            const uint32_t l0 = LT[i0], l1 = LT[i0 + ((rw.x & bit1) ? 1u : 0u)];
#pragma unroll
            for (int ij = 0; ij < 4; ++ij) {
                const int X = 2 * b0 + (ij >> 1), Y = 2 * b1 + (ij & 1);
                const uint32_t ce = ij == 0 ? a.x : ij == 1 ? a.z : ij == 2 ? b.x : b.z;   // even, odd voxels
                const uint32_t co = ij == 0 ? a.y : ij == 1 ? a.w : ij == 2 ? b.y : b.w;
                int4 v;
                v.x = (ce & bit0) ? int(l0) : 0;
                v.y = (co & bit0) ? int(l0) : 0;
                v.z = (ce & bit1) ? int(l1) : 0;
                v.w = (co & bit1) ? int(l1) : 0;
                int32_t *dst = im.out + (g.x0 + X) * rs0 + int64_t(g.y0 + Y) * im.d2 + g.z0 + 4 * q;
                const bool in = X < g.nx && Y < g.ny;
                if (!vec_ok) {   // rows of any alignment: 16-byte stores across the row's lanes
                    store_row<TB2 / 2>(dst, v, in ? n : 0);
                } else if (in) {   // (vec_ok: d2 is a multiple of 4, so is every row's end)
                    __stcs(reinterpret_cast<int4 *>(dst), v);
                }
            }
        }
        __syncthreads();
        t = tn;
    }
}

// ---------------------------------------------------------------------------------------------
// Launch sequence.
// ---------------------------------------------------------------------------------------------
cudaError_t launch_uf3d(const ImgList3D &L, const Work &w, int sms, bool persistent, cudaStream_t s,
                        cudaEvent_t *ev)
{
    auto mark = [&](int i) {
        if (ev) cudaEventRecord(ev[i], s);
    };
    auto grid = [&](int64_t items, int per_sm) -> unsigned {
        int64_t g = persistent ? std::min<int64_t>(items, int64_t(sms) * per_sm) : items;
        return unsigned(std::max<int64_t>(g, 1));
    };
    // The launches after the first overlap their start with the tail of the one before (they
    // wait for it on the device); not when events are recorded between them.
    const bool ov = !persistent && !ev;
    cudaError_t e = cudaSuccess;
    auto keep = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
    };
    mark(0);
    keep(launch_k(persistent ? k_tile_local_3d<true> : k_tile_local_3d<false>, grid(w.n_tiles, kT3LocalPerSM), kT3LocalThreads, s, false, L, w));
    mark(1);
    keep(launch_k(persistent ? k_merge_3d<true> : k_merge_3d<false>, grid(w.n_tiles, kT3MergePerSM), kT3MergeThreads, s, ov, L, w));
    mark(2);
    keep(launch_k(k_scan_link_3d, grid(int64_t(w.n_chunks) + w.n_tiles, 8), kScanThreads, s, ov, L, w));
    mark(3);
    const int64_t ctas = int64_t(sms) * kT3WritePerSM;
    const int split = persistent ? 1 : write_split(w.n_tiles, int64_t(sms) * kSplitPerSM3);
    // The label writes run a fixed tile order over kT3WritePerSM CTAs per SM (they prefetch their next tile).
    const auto write = persistent ? k_tile_write_3d<true, false> : split > 1 ? k_tile_write_3d<false, true> : k_tile_write_3d<false, false>;
    keep(launch_k(write, unsigned(std::max<int64_t>(1, std::min(w.n_tiles * split, ctas))), kT3Threads, s, ov, L, w));
    mark(4);
    return e;
}

}  // namespace be
