// be_uf2d_impl.cuh -- the 2D union-find pipeline for one tile shape.  Included by be_uf2d.cu
// once per supported shape, inside a namespace that defines
//   CELL      2: 2x2 blocks, 8-connectivity; 1: pixels, 4-connectivity
//   TBW, TBH  tile width and height in cells (TBW a power of two in [64, 256], TBW * TBH / 32 threads)
// Comments speak of blocks; with CELL 1 a block is one pixel, in pixel row and block row alike, every
// run is a T run (below), and the only link is the one straight up.
namespace {

constexpr int TW = CELL * TBW, TH = CELL * TBH;    // tile in pixels
constexpr int NBLK = TBW * TBH;                    // blocks per tile
constexpr int MAXRUN = CELL == 2 ? NBLK : NBLK / 2;   // runs per tile (between two pixel runs is a gap)
constexpr int NPERIM = 2 * (TBW + TBH);            // border positions per tile
constexpr int MAXB = NPERIM;                       // nodes per tile
constexpr int WPR = TBW / 32;                      // 32-block words per block row
constexpr int NWORD = NBLK / 32;                   // words per tile
constexpr int K1_NT = NWORD;                       // one thread per (block row, word)
constexpr int K1_PER_SM = CELL == 2 ? 7 : 4;       // resident tile CTAs per SM (26 KB of shared memory, 66 registers)
constexpr int MQCAP = 1024;                        // union-queue capacity (more take further rounds)
constexpr int RBWORDS = MAXRUN / 32;               // root-bitmap words per tile: a bit per run
// A tile's labels as the write kernel reads them (Work::lab): for each of its 32-block words the four
// pixel-class words (uint4) and the run words (uint4: starts of the runs with a top pixel, of the
// others, blocks of the former, runs of either kind before the word), then for every run of the
// tile its component's root run (uint16, at most MAXRUN).  With CELL 1 there are no class words, and
// the run words' second word is the pixels.
constexpr int kHdr = (CELL == 2 ? 8 : 4) * NWORD;
constexpr int kLabWords = kHdr + MAXRUN / 2;

// Roots of a segment: at most its runs, every two of them with a background pixel between.
using SegCount = std::conditional_t<TW / 2 <= 255, uint8_t, uint16_t>;
static_assert(TW / 2 <= 0xFFFF, "a segment's root count fits");

static_assert(MAXRUN == 4096, "a run number must fit 12 bits; 128 words of run flags");
static_assert(MAXB < 4096, "node index must fit 12 bits");
static_assert(K1_NT % 128 == 0 && K1_NT >= RBWORDS && (WPR & (WPR - 1)) == 0 && WPR <= 32, "thread layout");

// Block position of border position p of a tile with nbr x nbc valid blocks.
__device__ __forceinline__ bool perim_pos(int p, int nbr, int nbc, int &r, int &c)
{
    if (p < TBW) { r = 0; c = p; return c < nbc; }
    if (p < 2 * TBW) { r = nbr - 1; c = p - TBW; return c < nbc; }
    if (p < 2 * TBW + TBH) { r = p - 2 * TBW; c = 0; return r < nbr; }
    r = p - 2 * TBW - TBH; c = nbc - 1;
    return r < nbr;
}

// Global keys.  A component is known by (segment, place of its root run among the segment's runs):
// segments -- the part of one pixel row that lies in one tile -- are numbered in raster order, and a
// tile numbers the runs of a segment by their first pixel, so key = segment * seg_width + place orders
// components as their first pixels do.  A segment has at most seg_width runs, every two of them with
// a background pixel between, so keys stay below 2^31 with the pixel count.
__device__ __forceinline__ uint32_t seg_width(const Img2D &im) { return uint32_t(min(im.cols, TW) + 1) >> 1; }

// Blocks that n pixels take.
__device__ __forceinline__ int cells(int n) { return CELL == 2 ? (n + 1) >> 1 : n; }

// Set bits of the bitmap b in positions [lo, hi).
__device__ __forceinline__ uint32_t count_bits(const uint32_t *b, uint32_t lo, uint32_t hi)
{
    uint32_t n = 0;
    for (uint32_t i = lo >> 5; 32 * i < hi; ++i) {
        uint32_t x = __ldcg(b + i);
        if (i == lo >> 5) x &= ~0u << (lo & 31u);
        if (32 * i + 32 > hi) x &= (1u << (hi & 31u)) - 1u;
        n += __popc(x);
    }
    return n;
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Tile-local labeling.  One thread per 32 blocks of a block row (a "word"): the four pixel
// classes of the blocks (top-left, top-right, bottom-left, bottom-right) are 32-bit words, so
// horizontal runs of joined blocks, their starts and the links to the row above are bitwise
// operations.  Runs are numbered 0.. over the tile in the raster order of their first pixels: row by
// row, in a row the runs with a top pixel ("T runs") first, then those without ("B runs"), each by
// column.  So the run of a block is `runs of its kind before the word + starts of its kind in the
// word up to the block - 1` -- one popc, no search -- and the union-find over run numbers in shared
// memory, where the smaller number wins, leaves the run of a component's first pixel as its root.
// The loops over runs and links are shared evenly by the CTA's threads, and the tile is handed on as
// bit words and one number per run, not as an entry per block.
//
// Bound by instruction issue (65% of the issue slots, four instructions of a 32-lane warp per block) and
// the latency of shared-memory chains behind it, not by the image's bytes (67 MB of an 8192^2 image, 10
// us).  Measured (this launch on 8192^2, us; one thread's serial loops over its word's runs, entries per
// block -> this form): noise of density 0.6 150 -> 88, 0.4 158 -> 94, 0.1 73 -> 59, spiral 129 -> 87.
// The 64 x 256 tile and 7 CTAs of 128 threads are what its 26 KB and 66 registers leave room for; the
// pixel form (256 threads of 32 pixels) runs 4.
// ---------------------------------------------------------------------------------------------
template <bool Q>
__global__ void __launch_bounds__(K1_NT, K1_PER_SM) k_tile_local_2d(ImgList2D L, Work w)
{
    grid_dep_release();   // the merge launch may take free SMs during this grid's last wave
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // a new epoch for the segment scan of this run
        w.epoch[0] += 1u;
        w.epoch[1] = 0u;
    }
    __shared__ __align__(16) uint32_t P[MAXRUN]; // per run: parent run
    __shared__ __align__(16) uint4 CW[CELL == 2 ? NWORD : 1];   // class words: TL, TR, BL, BR
    __shared__ __align__(16) uint4 WR[NWORD];    // T starts, B starts (CELL 1: pixels), blocks of T runs,
                                                 // runs before (T | B << 16)
    __shared__ uint32_t WHC[NWORD];              // joins to the right
    __shared__ uint32_t MQ[MQCAP];               // union queue: (run_a << 16) | run_b
    __shared__ uint32_t BF[RBWORDS];             // runs that are border components
    __shared__ uint32_t BP[RBWORDS];             // runs that are roots; then nodes before each word of BF
    __shared__ uint32_t mqn;
    __shared__ uint32_t wtot[K1_NT / 32], ntot[RBWORDS / 32];   // run starts / nodes per warp
    __shared__ uint32_t qslot;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r = tid / WPR, q = tid % WPR;
    uint32_t *lab = reinterpret_cast<uint32_t *>(w.lab);
    ItemLoop<Q> loop{w.queue + 0};
    for (int64_t t = loop.first(&qslot); t < w.n_tiles; t = loop.next(t, &qslot)) {
        const Img2D im = L.find(t, w.timg);
        const int64_t lt = t - im.tile_base;
        const int ty = int(uint32_t(lt) / uint32_t(im.tiles_x)), tx = int(uint32_t(lt) - uint32_t(ty) * uint32_t(im.tiles_x));
        const int y0 = ty * TH, x0 = tx * TW;
        const int nrp = min(TH, im.rows - y0), ncp = min(TW, im.cols - x0);
        const int nbr = cells(nrp), nbc = cells(ncp);
        const uint32_t K = (0x7Fu - (uint32_t(im.thr) & 0x7Fu)) * 0x01010101u;
        const bool hi = im.thr >= 128;

        if (tid == 0) mqn = 0;
        if (tid < RBWORDS) BF[tid] = 0;
        for (int i = tid; i < MAXRUN / 4; i += K1_NT)   // every run its own root
            reinterpret_cast<uint4 *>(P)[i] = make_uint4(4 * i, 4 * i + 1, 4 * i + 2, 4 * i + 3);

        // Phase A: pixel words, runs, run starts.
        uint32_t TLw = 0, TRw = 0, BLw = 0, BRw = 0;   // CELL 2: pixel classes
        uint32_t F = 0;                                // CELL 1: pixels
        if constexpr (CELL == 2) {
            if (r < nbr && 64 * q < ncp) {
                const uint8_t *row0 = im.in + int64_t(y0 + 2 * r) * im.in_pitch + x0 + 64 * q;
                const bool row1 = 2 * r + 1 < nrp;
                const bool vec = (64 * q + 64 <= ncp) &&
                                 ((reinterpret_cast<uintptr_t>(row0) | uintptr_t(im.in_pitch)) & 15) == 0;
                if (vec) {
                    const uint4 *p0 = reinterpret_cast<const uint4 *>(row0);
                    uint4 v[4], u[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = __ldg(p0 + i);
                    if (row1) {
                        const uint4 *p1 = reinterpret_cast<const uint4 *>(row0 + im.in_pitch);
#pragma unroll
                        for (int i = 0; i < 4; ++i) u[i] = __ldg(p1 + i);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t ev, od;
                        split16(v[i], K, hi, ev, od);
                        TLw |= ev << (8 * i);
                        TRw |= od << (8 * i);
                        if (row1) {
                            split16(u[i], K, hi, ev, od);
                            BLw |= ev << (8 * i);
                            BRw |= od << (8 * i);
                        }
                    }
                } else {
                    const int n = min(64, ncp - 64 * q);
                    const uint8_t *hi_px = im.in + int64_t(im.rows - 1) * im.in_pitch + im.cols;
                    row_bits(row0, n, im.in, hi_px, K, hi, im.thr, TLw, TRw);
                    if (row1) row_bits(row0 + im.in_pitch, n, im.in, hi_px, K, hi, im.thr, BLw, BRw);
                }
            }
        } else if (r < nbr && 32 * q < ncp) {
            const uint8_t *row = im.in + int64_t(y0 + r) * im.in_pitch + x0 + 32 * q;
            if (32 * q + 32 <= ncp && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
                const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row)), u = __ldg(reinterpret_cast<const uint4 *>(row) + 1);
                F = bits16(v, K, hi) | (bits16(u, K, hi) << 16);
            } else {
                uint32_t even, odd;
                row_bits(row, min(32, ncp - 32 * q), im.in, im.in + int64_t(im.rows - 1) * im.in_pitch + im.cols, K, hi,
                         im.thr, even, odd);
                F = spread16(even) | (spread16(odd) << 1);
            }
        }
        const uint32_t Lw = CELL == 2 ? TLw | BLw : F, Rw = CELL == 2 ? TRw | BRw : F, Tw = CELL == 2 ? TLw | TRw : F;
        // hc bit k: block k is joined to block k + 1 (a right pixel of k touches a left pixel of
        // k + 1 -- every such pair is 8-adjacent); bit 31 looks at the next word.
        const uint32_t Lnext = __shfl_down_sync(0xFFFFFFFFu, Lw, 1, WPR);
        const uint32_t hc = (Rw & (Lw >> 1)) | ((q + 1 < WPR) ? (Rw & (Lnext << 31)) : 0u);
        const uint32_t hcprev = __shfl_up_sync(0xFFFFFFFFu, hc, 1, WPR);
        const uint32_t cin = q > 0 ? (hcprev >> 31) : 0u;   // block 0 continues a run from the left
        const uint32_t hl = (hc << 1) | cin;                  // bit k: block k joined to block k - 1
        const uint32_t S = (Lw | Rw) & ~hl;                   // run starts
        // T runs: the starts whose run has a top pixel.  Within the word, from each top pixel a carry
        // runs down (in reversed bits) to the start it belongs to.  A run that goes on past its word
        // with no top pixel yet takes it from the words it goes on into.
        uint32_t ST = S, CT = ~0u;
        if constexpr (CELL == 2) {
            const uint32_t rS = __brev(S), rT = __brev(Tw);
            ST = __brev(((~rS + (rT & ~rS)) | rT) & rS);
            const uint32_t cm = (S & (0u - S)) - 1u;   // blocks before the word's first start
            const uint32_t mine = ((cin && (Tw & cm)) ? 1u : 0u) | ((cin && !S && (hc >> 31)) ? 2u : 0u);
            const uint32_t last = S ? 0x80000000u >> __clz(S) : 0u;
            bool open = last && (hc >> 31) && !(ST & last);
#pragma unroll
            for (int d = 1; d < WPR; ++d) {
                const uint32_t pj = __shfl_down_sync(0xFFFFFFFFu, mine, d, WPR);
                if (open && q + d < WPR) {
                    if (pj & 1u) ST |= last;
                    open = pj == 2u;
                }
            }
            // Blocks of T runs: from each T start up to the next start; a run carried in has the kind
            // of the last start before the word.
            uint32_t v = S ? 2u | ((ST & last) ? 1u : 0u) : 0u;
#pragma unroll
            for (int o = 1; o < WPR; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o, WPR);
                if (q >= o && !v) v = u;
            }
            const uint32_t vp = __shfl_up_sync(0xFFFFFFFFu, v, 1, WPR);
            uint32_t pr = ~S;
            CT = ST | (q > 0 ? vp & pr & 1u : 0u);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                CT |= (CT << o) & pr;
                pr &= pr << o;
            }
        }
        const uint32_t SB = CELL == 2 ? S & ~ST : 0u;
        // Runs before this word: in its row (T runs in the low half, B runs in the high half), and in
        // the rows before it -- over the warp here, the warps' totals are added after the barrier.
        uint32_t bTB, rowsum;
        {
            const uint32_t c = __popc(ST) | (__popc(SB) << 16);
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < WPR; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o, WPR);
                if (q >= o) x += u;
            }
            const uint32_t row = __shfl_sync(0xFFFFFFFFu, x, WPR - 1, WPR);
            const uint32_t rt = (row & 0xFFFFu) + (row >> 16);
            rowsum = rt;
#pragma unroll
            for (int o = WPR; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, rowsum, o);
                if (lane >= o) rowsum += u;
            }
            bTB = x - c + (row << 16) + (rowsum - rt) * 0x10001u;   // B runs follow the row's T runs
        }
        if (lane == 31) wtot[warp] = rowsum;
        if constexpr (CELL == 2) CW[tid] = make_uint4(TLw, TRw, BLw, BRw);
        WR[tid] = make_uint4(ST, CELL == 2 ? SB : F, CT, bTB);
        WHC[tid] = hc;
        __syncthreads();   // words of every row written
        uint32_t woff = 0, nrun = 0, uoff = 0;
#pragma unroll
        for (int i = 0; i < K1_NT / 32; ++i) {
            const uint32_t n = wtot[i];
            if (i < warp) woff += n;
            if (i < int(uint32_t(tid - WPR) >> 5)) uoff += n;
            nrun += n;
        }
        bTB += woff * 0x10001u;
        const uint32_t bT = bTB & 0xFFFFu, bB = bTB >> 16;   // T, B runs numbered before this word's
        {
            uint4 *h = reinterpret_cast<uint4 *>(lab + t * kLabWords);
            if constexpr (CELL == 2) h[tid] = make_uint4(TLw, TRw, BLw, BRw);
            h[kHdr / 4 - NWORD + tid] = make_uint4(ST, CELL == 2 ? SB : F, CT, bTB);
        }

        // Phase B: links to the block row above.  For block b of this row: N (straight up, a top
        // pixel over a bottom pixel), NW (top-left pixel to the bottom-right pixel of b - 1 above)
        // and NE (top-right to the bottom-left pixel of b + 1 above).  A link is dropped when an
        // earlier link (further left, or N before NW / NE at the same block) joins the same two
        // runs; every chain of such reasons ends at a link that is kept.
        uint32_t Nm = 0, NWm = 0, NEm = 0;
        uint32_t uST = 0, uSB = 0, ubTB = 0;              // the word above: starts, runs before
        uint32_t uC = 0, uCl = 0, uCr = 0, uSn = 0;       // kind of the block above, above left, above right
        const bool above = r > 0 && r < nbr;
        if constexpr (CELL == 2) {
            if (above) {
                const int u = tid - WPR;   // same word, row above
                const uint32_t uBL = CW[u].z, uBR = CW[u].w;
                const uint32_t uBRp = q > 0 ? CW[u - 1].w >> 31 : 0u;
                const uint32_t uBLn = q + 1 < WPR ? CW[u + 1].z & 1u : 0u;
                const uint4 ur = WR[u];
                uST = ur.x;
                uSB = ur.y;
                uC = ur.z;
                ubTB = ur.w + uoff * 0x10001u;
                uCl = uC << 1;
                uCr = uC >> 1;
                if (q > 0) uCl |= WR[u - 1].z >> 31;
                if (q + 1 < WPR) {
                    const uint4 un = WR[u + 1];
                    uCr |= un.z << 31;
                    uSn = (un.x | un.y) & 1u;   // a run starts at the next word's first block
                }
                Nm = Tw & (uBL | uBR);
                NWm = TLw & ((uBR << 1) | uBRp);
                NEm = TRw & ((uBL >> 1) | (uBLn << 31));
            }
            {
                // bit 31 of the previous word's raw N / NE, for the rules at block 0
                const uint32_t Np = __shfl_up_sync(0xFFFFFFFFu, Nm, 1, WPR);
                const uint32_t NEp = __shfl_up_sync(0xFFFFFFFFu, NEm, 1, WPR);
                if (above) {
                    const int u = tid - WPR;
                    const uint32_t uhc = WHC[u];
                    const uint32_t uhl = (uhc << 1) | (q > 0 ? WHC[u - 1] >> 31 : 0u);
                    const uint32_t N = Nm, NE = NEm;
                    const uint32_t Nsh = (N << 1) | (q > 0 ? Np >> 31 : 0u);
                    const uint32_t NEsh = (NE << 1) | (q > 0 ? NEp >> 31 : 0u);
                    Nm = N & ~(hl & ((Nsh & uhl) | NEsh));
                    NWm &= ~((N & uhl) | (hl & Nsh));
                    NEm = NE & ~((N & uhc) | (hl & NEsh & uhc));
                }
            }
        } else {
            if (above) {
                const uint4 ur = WR[tid - WPR];
                uST = ur.x;
                ubTB = ur.w + uoff * 0x10001u;
                Nm = F & ur.y;
            }
            // A pixel pair left of another one is joined to it in both rows.
            const uint32_t Np = __shfl_up_sync(0xFFFFFFFFu, Nm, 1, WPR);
            Nm &= ~((Nm << 1) | (q > 0 ? Np >> 31 : 0u));
        }
        // Takes one kept link of block b off the masks (N, else NW, else NE): its two runs.
        auto take = [&](uint32_t b, uint32_t &own, uint32_t &up) {
            const uint32_t bit = 1u << b, upto = (bit << 1) - 1u;
            if constexpr (CELL == 1) {
                Nm ^= bit;
                own = bT + __popc(ST & upto) - 1u;
                up = (ubTB & 0xFFFFu) + __popc(uST & upto) - 1u;
                return;
            }
            const bool tt = CT & bit;
            own = (tt ? bT : bB) + __popc((tt ? ST : SB) & upto) - 1u;
            const bool isN = Nm & bit, isW = !isN && (NWm & bit), isE = !isN && !isW;
            Nm &= isN ? ~bit : ~0u;
            NWm &= isW ? ~bit : ~0u;
            NEm &= isE ? ~bit : ~0u;
            // Blocks of the word above up to the link's (NW at b = 0: none, its block is the last of the
            // word before; NE at b >= 30: all, at b = 31 and the first block of the word after).
            const uint32_t m = isN ? upto : isW ? bit - 1u : (bit << 2) - 1u;
            const bool ut = (isN ? uC : isW ? uCl : uCr) & bit;
            up = (ut ? ubTB & 0xFFFFu : ubTB >> 16) + __popc((ut ? uST : uSB) & m) + (isE && b == 31u ? uSn : 0u) - 1u;
        };
        // The first link of every run that starts in this word becomes the run's parent by a plain
        // store: the parent is in the row above, whose numbers are all smaller, so no cycle is
        // possible and no atomic is needed.  First links by a carry: adding the starts that hold no
        // link to ~links ripples from each of them to the next link bit and stops there; a start
        // without any link ripples on into the next start, which absorbs the carry or is itself a link.
        {
            const uint32_t lk = Nm | NWm | NEm;
            uint32_t first = lk & ((~lk + (S & ~lk)) | S);
            while (first) {
                const uint32_t b = __ffs(first) - 1;
                first &= first - 1;
                uint32_t own, up;
                take(b, own, up);
                if (GUARD(w, own < nrun && up < own, 112, (uint64_t(own) << 32) | up)) P[own & (MAXRUN - 1)] = up & (MAXRUN - 1);
            }
        }
        // The remaining links are unions: queued and merged by every lane.
        const uint32_t n = __popc(Nm) + __popc(NWm) + __popc(NEm);
        uint32_t pos = warp_reserve(&mqn, n);
        auto push = [&](uint32_t lo, uint32_t end) {   // links at queue positions [lo, end) go in
            while (pos < end) {
                const uint32_t b = __ffs(Nm | NWm | NEm);
                if (!b) break;
                uint32_t own, up;
                take(b - 1u, own, up);
                MQ[pos - lo] = GUARD(w, own < nrun && up < own, 114, (uint64_t(own) << 32) | up) ? (own << 16) | up : 0u;
                ++pos;
            }
        };
        push(0u, uint32_t(MQCAP));
        __syncthreads();
        WR[tid].w = bTB;   // from here on the runs before each word over the whole tile
        // The forest of first links is as deep as the tile has rows; every run of it is pointed at its
        // tree's root before the unions, in ascending order, so that a walk meets runs already done.
        sflatten_all(P, tid, K1_NT, nrun);
        __syncthreads();
        // Rounds of the queue, each warp with its quarter.
        const uint32_t total = mqn;
        uint32_t kept = 0;
        for (uint32_t lo = 0; lo < total; lo += MQCAP) {
            if (lo) {
                sflatten_all(P, tid, K1_NT, nrun);   // shook_pairs wants every run at its root
                push(lo, lo + MQCAP);
                __syncthreads();
            }
            const uint32_t nq = min(total - lo, uint32_t(MQCAP)), per = (nq + K1_NT / 32 - 1) / (K1_NT / 32);
            const uint32_t q0 = min(nq, warp * per);
            kept = shook_pairs(P, MQ + q0, min(nq - q0, per));
            __syncthreads();
            for (uint32_t k = lane; k < kept; k += 32) smerge(P, MQ[q0 + k] >> 16, MQ[q0 + k] & 0xFFFFu);
            __syncthreads();
        }

        // Phase C: what the unions linked is the roots of kept pairs; these are pointed at their roots,
        // so that every run is at most one step from its own (root_of).  With several rounds of the
        // queue every run is.  Roots are flagged in bit words.
        if (total > uint32_t(MQCAP)) {
            sflatten_all(P, tid, K1_NT, nrun);
        } else if (total) {
            const uint32_t per = (total + K1_NT / 32 - 1) / (K1_NT / 32), q0 = min(total, warp * per);
            for (uint32_t k = lane; k < kept; k += 32) {
                const uint32_t e = MQ[q0 + k];
#pragma unroll
                for (int side = 0; side < 2; ++side) {
                    const uint32_t i = side ? e & 0xFFFFu : e >> 16;
                    uint32_t x = i, y = P[i];
                    while (y != x) {
                        x = y;
                        y = P[x];
                    }
                    if (x != i) P[i] = x;
                }
            }
        }
        for (uint32_t i0 = 32 * warp; i0 < nrun; i0 += K1_NT) {
            const uint32_t i = i0 + lane;
            const uint32_t roots = __ballot_sync(0xFFFFFFFFu, i < nrun && P[i] == i);
            if (lane == 0) BP[i0 >> 5] = roots;
        }
        __syncthreads();

        loop.request();
        // Phase D: every run's root, the tile's root bitmap and the segments' root counts out.
        auto root_of = [&](uint32_t id) -> uint32_t { return P[P[id & (MAXRUN - 1)]]; };
        {
            uint32_t *rl = lab + t * kLabWords + kHdr;
            for (uint32_t i = 2 * tid; i < nrun; i += 2 * K1_NT)
                rl[i >> 1] = root_of(i) | (root_of(i + 1 < nrun ? i + 1 : i) << 16);
        }
        if (tid < RBWORDS) w.rbits[t * RBWORDS + tid] = 32u * tid < nrun ? BP[tid] : 0u;
        if (tid < TH && tid < nrp) {   // runs [s, e) start in pixel row tid
            const int br = tid / CELL;
            const bool low = CELL == 2 && (tid & 1);
            const uint32_t b = WR[br * WPR].w;
            const uint32_t s = low ? b >> 16 : b & 0xFFFFu;
            const uint32_t e = !low ? b >> 16 : br + 1 < TBH ? WR[(br + 1) * WPR].w & 0xFFFFu : nrun;
            uint32_t c = 0;
            for (uint32_t i = s >> 5; 32 * i < e; ++i)
                c += __popc(BP[i] & (i == s >> 5 ? ~0u << (s & 31u) : ~0u) & (32 * i + 32 > e ? (1u << (e & 31u)) - 1u : ~0u));
            const int64_t si = im.seg_base + int64_t(y0 + tid) * im.tiles_x + tx;
            if (GUARD(w, si >= 0 && si < w.n_segs, 116, si)) reinterpret_cast<SegCount *>(w.segcnt)[si] = SegCount(c);
        }
        // Border positions: component (root run), mask, and whether this position
        // claimed the node (the one that sets the component's flag writes the node's record).
        constexpr uint32_t kOwner = 1u << 20;
        uint32_t prb[(NPERIM + K1_NT - 1) / K1_NT];
#pragma unroll
        for (int i = 0; i < (NPERIM + K1_NT - 1) / K1_NT; ++i) {
            const int p = tid + i * K1_NT;
            int br, bc;
            prb[i] = kNone;
            if (p >= NPERIM || !perim_pos(p, nbr, nbc, br, bc)) continue;
            const int wi = br * WPR + (bc >> 5), k = bc & 31;
            const uint4 wr = WR[wi];
            uint32_t m;
            if constexpr (CELL == 2) {
                const uint4 cw = CW[wi];
                m = ((cw.x >> k) & 1u) | (((cw.y >> k) & 1u) << 1) | (((cw.z >> k) & 1u) << 2) | (((cw.w >> k) & 1u) << 3);
            } else {
                m = (wr.y >> k) & 1u;
            }
            if (!m) continue;
            const uint32_t upto = (2u << k) - 1u;
            const uint32_t id = (CELL == 1 || ((wr.z >> k) & 1u) ? (wr.w & 0xFFFFu) + __popc(wr.x & upto) : (wr.w >> 16) + __popc(wr.y & upto)) - 1u;
            if (!GUARD(w, id < nrun, 113, id)) continue;
            const uint32_t c = root_of(id);
            const uint32_t bit = 1u << (c & 31);
            const uint32_t old = atomicOr(&BF[c >> 5], bit);
            prb[i] = c | (m << 16) | ((old & bit) ? 0u : kOwner);
        }
        __syncthreads();   // node flags complete
        if (tid < RBWORDS) {   // nodes before each word of flags, within the warp; the warps' totals beside them
            const uint32_t c = __popc(BF[tid]);
            uint32_t x = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += v;
            }
            BP[tid] = x - c;
            if (lane == 31) ntot[warp] = x;
        }
        __syncthreads();
        // Every border position writes its entry; the position that claimed its node writes the
        // node's record.
        uint32_t noff[RBWORDS / 32 + 1];
        noff[0] = 0;
#pragma unroll
        for (int i = 0; i < RBWORDS / 32; ++i) noff[i + 1] = noff[i] + ntot[i];
#pragma unroll
        for (int i = 0; i < (NPERIM + K1_NT - 1) / K1_NT; ++i) {
            const int p = tid + i * K1_NT;
            if (p >= NPERIM) continue;
            uint16_t ent = 0;
            if (prb[i] != kNone) {
                const uint32_t c = prb[i] & 0xFFFFu, m = (prb[i] >> 16) & 15u;
                const uint32_t cw = c >> 5, g = cw >> 5;
                const uint32_t j = (g == 0 ? noff[0] : g == 1 ? noff[1] : g == 2 ? noff[2] : noff[3]) + BP[cw] +
                                   __popc(BF[cw] & ((1u << (c & 31)) - 1u));
                const bool ok = GUARD(w, j < uint32_t(MAXB), 115, j);
                ent = ok ? uint16_t((j << 4) | m) : uint16_t(0);
                if ((prb[i] & kOwner) && ok) {
                    int row = 0;   // the block row of run c
#pragma unroll
                    for (int h = TBH / 2; h; h >>= 1)
                        if ((WR[(row + h) * WPR].w & 0xFFFFu) <= c) row += h;
                    const uint32_t b = WR[row * WPR].w;
                    const bool low = CELL == 2 && c >= b >> 16;   // a run without a top pixel
                    const uint32_t place = c - (low ? b >> 16 : b & 0xFFFFu);
                    const int64_t seg = int64_t(y0 + CELL * row + (low ? 1 : 0)) * im.tiles_x + tx;
                    const int64_t node = t * MAXB + j;
                    w.nroot[node] = uint16_t(c);
                    w.gp[node] = gentry(uint32_t(seg) * seg_width(im) + place, uint32_t(node));
                }
            }
            w.perim[t * NPERIM + p] = ent;
        }
        if (tid == 0) w.nb[t] = noff[RBWORDS / 32];
        if (!Q) break;   // one tile per CTA
        loop.publish(&qslot);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Cross-tile merge.
// ---------------------------------------------------------------------------------------------
namespace {

// Union of two nodes of one image; the root with the larger key is linked under the other, and
// the linked root leaves its segment's root count and its tile's root bitmap (so that after the merge
// the bitmaps hold exactly the components' root runs).
__device__ void gunion2d(const Img2D &im, Work &w, uint32_t a, uint32_t b)
{
    gunion_keyed(w.gp, a, b, [&](uint32_t node, uint32_t key) {
        dec_count<SegCount>(w.segcnt, im.seg_base + key / seg_width(im));
        const uint32_t run = w.nroot[node];
        atomicAnd(w.rbits + int64_t(node / MAXB) * RBWORDS + (run >> 5), ~(1u << (run & 31u)));
    });
}

}  // namespace

constexpr int K2_NP = TBH + TBW;               // border positions a merge CTA looks at
constexpr int K2_NT = 64;                      // threads of a merge CTA (small: many tiles per SM)
constexpr int K2_PER_SM = 28;                  // resident merge CTAs per SM
constexpr int kGQ2 = 256;                      // queued global unions per tile (more are done at once)
constexpr int kSeen2 = 256;                    // table of pairs seen

// Positions p < TBH are the right border's rows, the others the bottom border's columns
// (p - TBH).  The border entries across the right border (the next tile's left column) and the
// bottom border (the top row of the tile below, widened by one block into the two diagonal tiles)
// are staged in shared memory.  Most links join the same few pairs of border components; a table
// of the pairs seen lets one link of each through, to a shared queue that both warps empty by global
// unions once all of the tile's links are seen.  The merge is bound by the latency of those unions
// (dependent L2 round trips), so a CTA is two warps that loop over the positions: many tiles are in
// flight on each SM at once.  Measured (this launch, us; a CTA-local union-find before the queue ->
// the table; 8192^2 noise of density 0.6: 29.0 -> 24.4, 0.1: 19.4 -> 14.6; 2048^2 disks 19.0 -> 16.4),
// and with the jumps after the unions 25.7, 15.7 and 16.6 -- for an 8192^2 spiral 101 -> 54, for a
// 2048^2 one 31 -> 22.
template <bool Q>
__global__ void __launch_bounds__(K2_NT, K2_PER_SM) k_merge_2d(ImgList2D L, Work w)
{
    grid_dep_wait();
    grid_dep_release();
    __shared__ uint32_t qslot;
    __shared__ uint16_t st[TBH + TBW + 2];    // staged border entries (0 = background)
    __shared__ uint32_t seen[kSeen2];
    __shared__ uint2 gq[kGQ2];
    __shared__ uint32_t nq;
    ItemLoop<Q> loop{w.queue + 1};
    for (int64_t t = loop.first(&qslot); t < w.n_tiles; t = loop.next(t, &qslot)) {
        const Img2D im = L.get(t, w.timg);
        loop.request();
        const int64_t lt = t - im.tile_base;
        const int ty = int(uint32_t(lt) / uint32_t(im.tiles_x)), tx = int(uint32_t(lt) - uint32_t(ty) * uint32_t(im.tiles_x));
        const int nbr = cells(min(TH, im.rows - ty * TH));
        const int nbc = cells(min(TW, im.cols - tx * TW));
        const uint16_t *pe = w.perim;
        for (int i = threadIdx.x; i < kSeen2; i += K2_NT) seen[i] = kNone;
        if (threadIdx.x == 0) nq = 0;
        // Stage: position p < TBH stages right-column row p; the others bottom-row column p - TBH,
        // and the first two of those also columns -1 and TBW.  Each position's own entry is loaded
        // with the staging loads.
        constexpr int NI = (K2_NP + K2_NT - 1) / K2_NT;
        uint32_t own[NI];
        bool right = tx + 1 < im.tiles_x, below = ty + 1 < im.tiles_y;
        if (!GUARD(w, t + (below ? im.tiles_x : 0) + (right ? 1 : 0) < w.n_tiles, 201, t)) right = below = false;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int p = threadIdx.x + i * K2_NT;
            own[i] = 0;
            if (p < TBH) {
                uint16_t B = 0;
                if (p < nbr && right) {
                    own[i] = pe[t * NPERIM + 2 * TBW + TBH + p];
                    B = pe[(t + 1) * NPERIM + 2 * TBW + p];
                }
                st[p] = B;
            } else if (p < K2_NP) {
                const int c = p - TBH;
                uint16_t B = 0;
                if (c < nbc && below) {
                    own[i] = pe[t * NPERIM + TBW + c];
                    B = pe[(t + im.tiles_x) * NPERIM + c];
                }
                st[p + 1] = B;
                if (c == 0) st[TBH] = tx > 0 && below ? pe[(t + im.tiles_x - 1) * NPERIM + TBW - 1] : uint16_t(0);
                // column TBW: block 0 of the tile below-right (a tile with a right neighbour is
                // full-width; a narrower tile's column nbc is staged empty by its own position)
                if (c == 1) st[TBH + TBW + 1] = nbc == TBW && right && below ? pe[(t + im.tiles_x + 1) * NPERIM] : uint16_t(0);
            }
        }
        __syncthreads();
        // Links of every position to the staged positions at offsets -1, 0, 1.  Neighbouring staged
        // positions of one node need one link; a pair of nodes in the table has its union queued.
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int p = threadIdx.x + i * K2_NT;
            const uint32_t A = own[i];
            if (!A) continue;
            const uint32_t ja = A >> 4;
            const bool col = p < TBH;            // right border: the same rows of the tile to the right
            const int k0 = col ? p : p + 1;      // staged position straight across
            uint32_t last = kNone;
#pragma unroll
            for (int dd = 0; dd < (CELL == 1 ? 1 : 3); ++dd) {
                const int d = dd == 0 ? 0 : dd == 1 ? -1 : 1, k = k0 + d;
                if (d < 0 && col && p == 0) continue;
                if (d > 0 && col && p == TBH - 1) continue;
                const uint32_t B = st[k];
                if constexpr (CELL == 2) {
                    const uint32_t a = col ? (d == 0 ? 0xAu : d < 0 ? 2u : 8u) : (d == 0 ? 0xCu : d < 0 ? 4u : 8u);
                    const uint32_t b = col ? (d == 0 ? 0x5u : d < 0 ? 4u : 1u) : (d == 0 ? 0x3u : d < 0 ? 2u : 1u);
                    if (!(A & a) || !(B & b)) continue;
                } else if (!B) {
                    continue;
                }
                // the staged position's tile: to the right, below left, below, below right
                const uint32_t side = col ? 0u : k == TBH ? 1u : k <= TBH + TBW ? 2u : 3u;
                const uint32_t key = (side << 24) | ((B >> 4) << 12) | ja;
                if (key == last) continue;
                last = key;
                if (atomicExch(&seen[(key * 0x9E3779B1u) >> 24], key) == key) continue;
                const int64_t tB = col ? t + 1 : t + im.tiles_x + int(side) - 2;
                if (!GUARD(w, ja < w.nb[t] && (B >> 4) < w.nb[tB], 203, (uint64_t(tB) << 32) | (B << 16) | A)) continue;
                const uint32_t nA = uint32_t(t * MAXB + ja);
                const uint32_t nB = uint32_t(tB * MAXB + (B >> 4));
                const uint32_t slot = atomicAdd(&nq, 1u);
                if (slot < uint32_t(kGQ2)) gq[slot] = make_uint2(nA, nB);
                else gunion2d(im, w, nA, nB);
            }
        }
        __syncthreads();
        const uint32_t nqt = min(nq, uint32_t(kGQ2));
        const uint32_t nb = w.nb[t];
        for (uint32_t i = threadIdx.x; i < nqt; i += K2_NT) gunion2d(im, w, gq[i].x, gq[i].y);
        __syncthreads();
        // Every node of the tile then jumps to its parent's parent, all tiles at once: a component that
        // winds through many tiles is a path as long as the tiles it crosses, and the union that closes
        // it climbs what nobody has shortened.
        for (uint32_t j = threadIdx.x; j < nb; j += K2_NT) gjump(w.gp, uint32_t(t * MAXB + j));
        if (!Q) break;   // one tile per CTA
        loop.publish(&qslot);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Segment scan and node flatten, one launch: items below n_chunks scan a chunk of segment counts
// (single pass, look-back); the others point every linked node of one tile straight at its global
// root (flatten_tile_nodes: all unions are done; the nodes of all tiles jump at once), so that the
// label writes find each root in one step however long the merge's chains grew.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kScanThreads) k_scan_flatten_2d(Work w)
{
    grid_dep_wait();
    grid_dep_release();   // after the wait: the label-write launch relies on it
    __shared__ uint32_t tmp[kScanThreads / 32 + 1];
    __shared__ uint32_t sh[2];
    const int64_t n = int64_t(w.n_chunks) + w.n_tiles;
    for (int64_t it = blockIdx.x; it < n; it += gridDim.x) {   // (in a fixed order: the items are short)
        if (it < w.n_chunks) {
            segscan_lb_chunk<kScanThreads, SegCount>(w, tmp, sh);
            continue;
        }
        flatten_tile_nodes(w, it - w.n_chunks, MAXB);
    }
}

// ---------------------------------------------------------------------------------------------
// Label resolve and write.
// ---------------------------------------------------------------------------------------------
constexpr int K3_NT = 256;
// CTAs per SM up to which CTAs share a tile's rows: with 4, a 2048^2 call (256 tiles) is 0.5 us slower, and
// none is faster than with 2.
constexpr int kSplitPerSM2 = 2;
// Resident CTAs per SM.  Fewer have registers for rows of any alignment (48 instead of 32 a thread), and
// four to five full of stores keep the memory as busy as eight: 8 / 7 / 6 / 5 / 4 take 58.0 / 59.0 / 59.5 /
// 57.5 / 61.3 us for 8192^2 noise, 83.0 / 85.4 / 82.2 / 79.9 / 84.7 for 8191x8189, 12.3 / 12.4 / 10.3 / 10.3 / 10.2
// for 1021x1787.
constexpr int K3_PER_SM = 5;

// A CTA works out the label of every run (roots by rank in their segment, linked border components
// through their global root, the others through their root run), then writes the rows; with a fixed tile
// order it fetches its next tile's words while it writes.  Bound by the stores: of 57 us for the 268 MB
// of an 8192^2 image a bare kernel that stores the same tiles takes 44 (6.1 TB/s); the rest is the first
// tile's set-up and the last, half-full round of tiles.  Copying the segment prefixes and node entries
// ahead too, and starting an SM's CTAs apart, changed nothing.  Four pixels a thread and row,
// as one 16-byte store; rows of any other alignment go through store_row.
//
// kWriteOne (a plain launch of one tile): the tile kernel's launch goes straight before this one -- there is
// nothing to merge and no prefix beyond the tile's own rows, which the CTA sums itself -- so that the
// smallest images take two launches: 16^2 17.4 -> 13.1 us, 64^2 18.5 -> 16.1 us.  (Doing without the scan
// launch for images of several tiles, every CTA scanning the counts, was slower: 2048^2 43.0 -> 44.7 us.)
template <bool Q, WriteForm F>
__global__ void __launch_bounds__(K3_NT, K3_PER_SM) k_tile_write_2d(ImgList2D L, Work w)
{
    constexpr bool ONE = F == kWriteOne, SHARED = F != kWriteTiles;
    __shared__ __align__(16) uint4 H[kHdr / 4];   // class words, then run words
    __shared__ uint32_t LT[MAXRUN + 1];   // label of run i at i + 1 (0: the place of "no run yet")
    constexpr int kStageRuns = 2048;      // run entries staged in shared memory (later ones: from L2)
    __shared__ __align__(16) uint32_t RB[RBWORDS + 1];
    __shared__ __align__(16) uint32_t E[kStageRuns / 2];
    __shared__ uint32_t segb[TH];
    __shared__ uint32_t qslot;

    const int tid = threadIdx.x;
    const uint32_t *lab = reinterpret_cast<const uint32_t *>(w.lab);
    // The tile's words and the root bitmap (first pixels of the components that stayed roots through
    // the merge) were final before this grid's predecessor (segment scan and node flatten) started:
    // that grid waits for the merge to complete before it lets this one launch.  So they are read
    // before the wait (through L2), and only the segment prefixes, which the scan writes, after it.
    // The words go into registers, the root bitmap and run entries into shared memory (cp.async).
    static_assert(TW % 128 == 0, "a warp's output units lie in one row");
    static_assert(kHdr == 4 * K3_NT && TH * WPR == K3_NT && kStageRuns == 8 * K3_NT, "prefetched words per thread");
    uint4 nH;
    uint32_t nNb = 0;
    auto fetch_words = [&](int64_t t) {
        nH = __ldcg(reinterpret_cast<const uint4 *>(lab + t * kLabWords) + tid);
        nNb = __ldcg(w.nb + t);
    };
    auto fetch_roots = [&](int64_t t) {
        if (tid < RBWORDS) cp_async4(&RB[tid], w.rbits + t * RBWORDS + tid);
        cp_async_commit();
    };
    auto fetch_runs = [&](int64_t t) {
        cp_async16(&E[4 * tid], lab + t * kLabWords + kHdr + 4 * tid);
        cp_async_commit();
    };
    auto fetch = [&](int64_t t) {
        fetch_words(t);
        fetch_roots(t);
        fetch_runs(t);
    };
    ItemLoop<Q> loop{w.queue + 4};
    int64_t t = loop.first(&qslot);
    int part = 0, split = 1;   // of the tile's rows
    if (SHARED) {
        split = int(gridDim.x / uint32_t(w.n_tiles));
        part = int(blockIdx.x % uint32_t(split));
        t = blockIdx.x / uint32_t(split);
    }
    if (ONE) grid_dep_wait();   // the tile kernel is this grid's predecessor
    if (t < w.n_tiles) fetch(t);
    while (t < w.n_tiles) {
        loop.request();
        const Img2D im = L.get(t, w.timg);
        const int64_t lt = t - im.tile_base;
        const int ty = int(uint32_t(lt) / uint32_t(im.tiles_x)), tx = int(uint32_t(lt) - uint32_t(ty) * uint32_t(im.tiles_x));
        const int y0 = ty * TH, x0 = tx * TW;
        const int nrp = min(TH, im.rows - y0), ncp = min(TW, im.cols - x0);
        H[tid] = nH;
        const uint32_t nb = nNb;
        // The next tile's data come while this one's labels are worked out and written, each part as soon
        // as its place is free -- and the tile is known, which with a work queue is before the writes.
        int64_t tn = Q || SHARED ? w.n_tiles : t + gridDim.x;
        if (tn < w.n_tiles) fetch_words(tn);
        cp_async_wait();
        auto put_count = [&](int64_t n) {
            w.ncomp[im.index] = n;
            if (w.host_count) *w.host_count = n;
        };
        uint32_t base0 = 0;
        if (ONE) {
            constexpr int PER = TH / 32;
            if (tid < 32) {
                uint32_t c[PER], sum = 0;
#pragma unroll
                for (int i = 0; i < PER; ++i) sum += c[i] = PER * tid + i < nrp ? reinterpret_cast<const SegCount *>(w.segcnt)[PER * tid + i] : 0u;
                uint32_t x = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, x, o);
                    if (tid >= o) x += v;
                }
                if (tid == 31 && part == 0) put_count(int64_t(x));
                x -= sum;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    segb[PER * tid + i] = x;
                    x += c[i];
                }
            }
        } else {
            grid_dep_wait();   // segment prefixes from here on (returns at once after the first tile)
            base0 = w.segpref[im.seg_base];
            if (tid < TH && tid < nrp)
                segb[tid] = w.segpref[im.seg_base + int64_t(y0 + tid) * im.tiles_x + tx] - base0;
            if (lt == 0 && tid == 0 && part == 0) put_count(int64_t(w.segpref[im.seg_base + int64_t(im.rows) * im.tiles_x] - base0));
        }
        __syncthreads();
        const uint4 *HR = H + kHdr / 4 - NWORD;   // run words
        // The last B run is the last run.
        uint32_t nrun = (HR[NWORD - 1].w >> 16) + (CELL == 2 ? __popc(HR[NWORD - 1].y) : 0);
        if (!GUARD(w, nrun <= uint32_t(MAXRUN), 404, nrun)) nrun = MAXRUN;

        // Surviving roots: rank = roots before it in its segment.  One thread per word and kind of run:
        // WPR consecutive lanes hold a segment's words, a shuffle scan gives each word's prefix, and the
        // word's runs are consecutive bits of the root bitmap.
        {
            const int seg = tid / WPR, wi = (seg / CELL) * WPR + tid % WPR;   // segment = pixel row
            const bool low = CELL == 2 && (seg & 1);
            const uint4 wr = HR[wi];
            const uint32_t c = __popc(low ? wr.y : wr.x), b = low ? wr.w >> 16 : wr.w & 0xFFFFu;
            const uint32_t g = b >> 5;   // (RB has a word past its end; b = MAXRUN only with c = 0)
            uint32_t bits = c ? __funnelshift_r(RB[g], RB[min(g + 1, uint32_t(RBWORDS))], b & 31u) & (0xFFFFFFFFu >> (32 - c)) : 0u;
            uint32_t pre = __popc(bits);
#pragma unroll
            for (int o = 1; o < WPR; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, pre, o, WPR);
                if (tid % WPR >= o) pre += v;
            }
            uint32_t label = 1u + segb[seg] + pre - __popc(bits);
            while (bits) {
                if (!GUARD(w, b + __ffs(bits) <= uint32_t(MAXRUN), 401, b)) break;
                LT[b + __ffs(bits)] = label++;   // run i's place is i + 1
                bits &= bits - 1;
            }
        }
        // Border components linked under another tile's component: the label of that root, its
        // segment's prefix plus its rank among the first pixels left in its row of its tile.
        for (uint32_t j = tid; !ONE && j < nb; j += K3_NT) {
            const int64_t node = t * MAXB + j;
            const unsigned long long e = __ldcg(w.gp + node);   // its root's own entry (flatten_tile_nodes)
            const uint32_t g = uint32_t(e), kg = uint32_t(e >> 32);
            if (g == uint32_t(node)) continue;
            const uint32_t sg = kg / seg_width(im);
            if (!GUARD(w, g < w.n_tiles * MAXB && sg < uint32_t(im.rows) * uint32_t(im.tiles_x), 402, e)) continue;
            const uint32_t run = __ldcg(w.nroot + g);
            const uint32_t rank = count_bits(w.rbits + int64_t(g / MAXB) * RBWORDS, run - (kg - sg * seg_width(im)), run);
            const uint32_t sb = w.segpref[im.seg_base + sg] - base0;
            LT[__ldcg(w.nroot + node) + 1u] = 1u + sb + rank;
        }
        __syncthreads();
        if (tn < w.n_tiles) fetch_roots(tn);
        // Every other run takes the label of its root run.
        for (uint32_t i = 2 * tid; i < nrun; i += 2 * K3_NT) {
            const uint32_t e = i < uint32_t(kStageRuns) ? E[i >> 1] : __ldcg(lab + t * kLabWords + kHdr + (i >> 1));
            const uint32_t a = e & 0xFFFFu, b = e >> 16;
            if (!GUARD(w, a < nrun && (i + 1 >= nrun || b < nrun), 403, e)) continue;
            if (a != i) LT[i + 1] = LT[a + 1];
            if (i + 1 < nrun && b != i + 1) LT[i + 2] = LT[b + 1];
        }
        loop.publish(&qslot);
        __syncthreads();
        if (Q) {
            tn = loop.next(t, &qslot);
            if (tn < w.n_tiles) fetch(tn);
        } else if (tn < w.n_tiles) {
            fetch_runs(tn);
        }

        // Output: one unit = 4 pixels in each row of a block row (two 2x2 blocks, or four pixel cells).
        const bool vec_ok = ((reinterpret_cast<uintptr_t>(im.out) | uintptr_t(im.out_pitch * 4)) & 15) == 0;
        // A thread keeps its column: unit i is UR block rows further down.
        constexpr int UPR = TW / 4, UR = K3_NT / UPR;   // units per block row, block rows per turn
        constexpr int UPW = CELL == 2 ? 16 : 8;         // units per word
        const int q = tid % UPR, k = (32 / UPW) * (q % UPW);
        const uint32_t bit0 = 1u << k, bit1 = 2u << k, upto0 = bit0 | (bit0 - 1u), upto1 = bit1 | (bit1 - 1u);
        const int n = min(4, max(0, ncp - 4 * q));       // pixels of the thread's column inside the image
        auto unit = [&](int br, int4 &a, int4 &b) {
            const int wi = br * WPR + q / UPW;
            if constexpr (CELL == 1) {
                const uint4 wr = HR[wi];
                const uint32_t st = wr.x >> k, f = wr.y >> k;
                uint32_t i = (wr.w & 0xFFFFu) + __popc(wr.x & upto0);
                a.x = (f & 1u) ? int(LT[i]) : 0;
                i += (st >> 1) & 1u;
                a.y = (f & 2u) ? int(LT[i]) : 0;
                i += (st >> 2) & 1u;
                a.z = (f & 4u) ? int(LT[i]) : 0;
                i += (st >> 3) & 1u;
                a.w = (f & 8u) ? int(LT[i]) : 0;
                return;
            }
            const uint4 c = H[wi], wr = HR[wi];
            const uint32_t bT = wr.w & 0xFFFFu, bB = wr.w >> 16;
            const bool t0 = wr.z & bit0, t1 = wr.z & bit1;
            const int l0 = int(LT[(t0 ? bT : bB) + __popc((t0 ? wr.x : wr.y) & upto0)]);
            const int l1 = int(LT[(t1 ? bT : bB) + __popc((t1 ? wr.x : wr.y) & upto1)]);
            a.x = (c.x & bit0) ? l0 : 0; a.y = (c.y & bit0) ? l0 : 0;
            a.z = (c.x & bit1) ? l1 : 0; a.w = (c.y & bit1) ? l1 : 0;
            b.x = (c.z & bit0) ? l0 : 0; b.y = (c.w & bit0) ? l0 : 0;
            b.z = (c.z & bit1) ? l1 : 0; b.w = (c.w & bit1) ? l1 : 0;
        };
        const int br0 = tid / UPR + UR * part, brs = UR * split;
        int32_t *dst = im.out + int64_t(y0 + CELL * br0) * im.out_pitch + x0 + 4 * q;
        const int64_t turn = CELL * brs * im.out_pitch;
        if (vec_ok) {
            if (n > 0)
                for (int br = br0; CELL * br < nrp; br += brs, dst += turn) {
                    int4 a, b;
                    unit(br, a, b);
                    const bool row2 = CELL == 2 && 2 * br + 1 < nrp;
                    if (n == 4) {
                        __stcs(reinterpret_cast<int4 *>(dst), a);
                        if (row2) __stcs(reinterpret_cast<int4 *>(dst + im.out_pitch), b);
                    } else {
                        const int va[4] = {a.x, a.y, a.z, a.w}, vb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            if (i >= n) break;
                            dst[i] = va[i];
                            if (row2) dst[im.out_pitch + i] = vb[i];
                        }
                    }
                }
        } else {
            for (int br = br0; CELL * br < nrp; br += brs, dst += turn) {   // rows of any alignment (whole warps)
                int4 a, b;
                unit(br, a, b);
                store_row<32>(dst, a, n);
                if (CELL == 2 && 2 * br + 1 < nrp) store_row<32>(dst + im.out_pitch, b, n);
            }
        }
        __syncthreads();
        t = tn;
    }
}

// ---------------------------------------------------------------------------------------------
// Geometry and launch sequence of this tile shape.
// ---------------------------------------------------------------------------------------------
inline Geometry geometry()
{
    Geometry g;
    g.lab_bytes_per_tile = size_t(kLabWords) * sizeof(uint32_t);
    g.rbits_bytes_per_tile = size_t(RBWORDS) * sizeof(uint32_t);
    g.nperim = NPERIM;
    g.seg_bytes = int(sizeof(SegCount));
    g.maxb = MAXB;
    return g;
}

inline cudaError_t launch(const ImgList2D &L, const Work &w, int sms, bool persistent, cudaStream_t s,
                          cudaEvent_t *ev)
{
    auto grid = [&](int64_t items, int per_sm) -> unsigned {
        int64_t g = persistent ? std::min<int64_t>(items, int64_t(sms) * per_sm) : items;
        return unsigned(std::max<int64_t>(g, 1));
    };
    auto mark = [&](int i) {
        if (ev) cudaEventRecord(ev[i], s);
    };
    // The launches after the first overlap their start with the tail of the one before (they
    // wait for it on the device); not when events are recorded between them.
    const bool ov = !persistent && !ev;
    cudaError_t e = cudaSuccess;
    auto keep = [&](cudaError_t r) {
        if (e == cudaSuccess) e = r;
    };
    mark(0);
    keep(launch_k(persistent ? k_tile_local_2d<true> : k_tile_local_2d<false>, grid(w.n_tiles, K1_PER_SM), K1_NT, s, false, L, w));
    mark(1);
    const bool one = !persistent && w.n_tiles == 1;
    if (!one) keep(launch_k(persistent ? k_merge_2d<true> : k_merge_2d<false>, grid(w.n_tiles, K2_PER_SM), K2_NT, s, ov, L, w));
    mark(2);
    if (!one) keep(launch_k(k_scan_flatten_2d, grid(int64_t(w.n_chunks) + w.n_tiles, 8), kScanThreads, s, ov, w));
    mark(3);
    const int64_t ctas = int64_t(sms) * K3_PER_SM;
    const int split = persistent ? 1 : write_split(w.n_tiles, int64_t(sms) * kSplitPerSM2);
    // The label writes run a fixed tile order over K3_PER_SM CTAs per SM (they prefetch their next tile).
    const auto write = persistent ? k_tile_write_2d<true, kWriteTiles>
                       : one ? k_tile_write_2d<false, kWriteOne>
                       : split > 1 ? k_tile_write_2d<false, kWriteShared> : k_tile_write_2d<false, kWriteTiles>;
    keep(launch_k(write, unsigned(std::max<int64_t>(1, std::min(w.n_tiles * split, ctas))), K3_NT, s, ov, L, w));
    mark(4);
    return e;
}
