"""The 3D kernels' link filters restated on whole tiles and checked against the oracle
(labeling_b200/csrc/be_uf3d.cu).  In a tile (k_tile_local_3d phase B) a link to a preceding row is dropped
when an earlier one to that row joins the same two runs, or when two others close a triangle with it over
the row straight below or the row beside.  Across tiles (k_merge_3d) links below left and below right are
dropped over the row straight below, wherever that lies, and links across d2 to the preceding rows over the
same row of the tile before or after.  Uniting the runs over the links that are kept must give exactly the
26-connected components: a rule that dropped a needed link would split one."""
import numpy as np
import pytest

from oracle import oracle as O

TB0, TB1, TB2 = 8, 16, 32
M = 0xFFFFFFFF


def face(c, dx, dy, dz):
    r = 0
    for v in range(8):
        i, j, k = v >> 2, (v >> 1) & 1, v & 1
        if (dx < 0 and i) or (dx > 0 and not i) or (dy < 0 and j) or (dy > 0 and not j) or (dz < 0 and k) or (dz > 0 and not k):
            continue
        r |= c[v]
    return r


def joins(c):
    return face(c, 0, 0, 1) & (face(c, 0, 0, -1) >> 1)


OFF = ((-1, -1), (-1, 0), (-1, 1), (0, -1))   # preceding rows 0..3


def row_links(nr, c, hz, u, uhz):
    """(kept n, w, e), (raw n, w, e)."""
    dx, dy = OFF[nr]
    a0, am, ap = (face(c, dx, dy, dz) for dz in (0, -1, 1))
    b0, bm, bp = (face(u, -dx, -dy, -dz) for dz in (0, -1, 1))
    hl, uhl = (hz << 1) & M, (uhz << 1) & M
    n, w, e = a0 & b0, am & (bm << 1) & M, ap & (bp >> 1)
    nsh, esh = (n << 1) & M, (e << 1) & M
    return (n & ~(hl & ((nsh & uhl) | esh)), w & ~((n & uhl) | (hl & nsh)), e & ~((n & uhz) | (hl & esh & uhz))), (n, w, e)


def bits(x):
    while x:
        b = x & -x
        yield b.bit_length() - 1
        x ^= b


def sh(x, s):
    return (x << s) & M if s > 0 else x >> -s


class Model:
    def __init__(self, vol):
        self.t = [-(-n // (2 * b)) for n, b in zip(vol.shape, (TB0, TB1, TB2))]
        pad = np.zeros([t * 2 * b for t, b in zip(self.t, (TB0, TB1, TB2))], bool)
        pad[:vol.shape[0], :vol.shape[1], :vol.shape[2]] = vol > 0
        self.cls, self.S, self.hz = {}, {}, {}
        for r0 in range(self.t[0] * TB0):
            for r1 in range(self.t[1] * TB1):
                for t2 in range(self.t[2]):
                    z = slice(t2 * 64, t2 * 64 + 64)
                    c = []
                    for v in range(8):
                        i, j, k = v >> 2, (v >> 1) & 1, v & 1
                        c.append(int(sum(1 << int(b) for b in np.flatnonzero(pad[2 * r0 + i, 2 * r1 + j, z][k::2]))))
                    key = (r0, r1, t2)
                    self.cls[key], self.hz[key] = c, joins(c)
                    f = 0
                    for x in c:
                        f |= x
                    self.S[key] = f & ~(self.hz[key] << 1) & M
        self.parent = {}

    def run(self, key, k):
        return key, (self.S[key] & ((2 << k) - 1)).bit_length() - 1

    def find(self, x):
        p = self.parent.setdefault(x, x)
        while p != x:
            g = self.parent[p]
            self.parent[x] = g
            x, p = p, self.parent[p]
        return x

    def unite(self, a, b):
        assert a[1] >= 0 and b[1] >= 0
        a, b = self.find(a), self.find(b)
        if a != b:
            self.parent[max(a, b)] = min(a, b)

    def unite_links(self, key, up, kept):
        for d, x in zip((0, -1, 1), kept):
            for k in bits(x):
                self.unite(self.run(key, k), self.run(up, k + d))

    def preceding(self, key, nr):
        """Key of a preceding row, or None outside the volume's tiles."""
        r0, r1 = key[0] + OFF[nr][0], key[1] + OFF[nr][1]
        return (r0, r1, key[2]) if r0 >= 0 and 0 <= r1 < self.t[1] * TB1 else None

    @staticmethod
    def tile(key):
        return key[0] // TB0, key[1] // TB1, key[2]

    def raw(self, key, up):
        """Raw links of a row to its preceding row `up` of the same tile (zeros elsewhere)."""
        nr = OFF.index((up[0] - key[0], up[1] - key[1]))
        if up not in self.cls or self.tile(up) != self.tile(key):
            return 0, 0, 0
        return row_links(nr, self.cls[key], self.hz[key], self.cls[up], self.hz[up])[1]

    def local(self, key):
        kept, raw = {}, {}
        for nr in range(4):
            up = self.preceding(key, nr)
            if up is None or self.tile(up) != self.tile(key):
                kept[nr], raw[nr] = (0, 0, 0), (0, 0, 0)
            else:
                kept[nr], raw[nr] = row_links(nr, self.cls[key], self.hz[key], self.cls[up], self.hz[up])
        r0, r1, t2 = key
        below, beside = (r0 - 1, r1, t2), (r0, r1 - 1, t2)
        zero = (0, 0, 0)
        in_below, in_beside = r0 % TB0 > 0, r1 % TB1 > 0
        p = self.raw(below, (r0 - 1, r1 - 1, t2)) if in_below else zero
        r = self.raw((r0 - 1, r1 + 1, t2), below) if in_below and (r1 + 1) % TB1 else zero
        s = self.raw(beside, (r0 - 1, r1 - 1, t2)) if in_beside else zero
        v = self.raw(beside, below) if in_beside else zero
        (n1, w1, e1), (n3, w3, e3) = raw[1], raw[3]
        n, w, e = kept[0]
        kept[0] = (n & ~((n1 & p[0]) | (n3 & s[0])),
                   w & ~((n1 & p[1]) | (w1 & sh(p[0], 1)) | (n3 & s[1]) | (w3 & sh(s[0], 1))),
                   e & ~((n1 & p[2]) | (e1 & sh(p[0], -1)) | (n3 & s[2]) | (e3 & sh(s[0], -1))))
        for nr, q in ((2, r), (3, v)):
            n, w, e = kept[nr]
            kept[nr] = (n & ~(n1 & q[0]), w & ~((n1 & sh(q[2], 1)) | (w1 & sh(q[0], 1))), e & ~((n1 & sh(q[1], -1)) | (e1 & sh(q[0], -1))))
        for nr in range(4):
            if any(kept[nr]):
                self.unite_links(key, self.preceding(key, nr), kept[nr])

    def across(self, key):
        c, hz = self.cls[key], self.hz[key]
        for nr in range(4):
            up = self.preceding(key, nr)
            if up is None or self.tile(up) == self.tile(key):
                continue
            u, uhz = self.cls[up], self.hz[up]
            (n, w, e), _ = row_links(nr, c, hz, u, uhz)
            if nr in (0, 2):
                below = self.preceding(key, 1)
                v = self.cls[below] if below else [0] * 8
                r1 = row_links(1, c, hz, v, 0)[1]
                if nr == 0:
                    p = row_links(3, v, 0, u, 0)[1]
                    n, w, e = n & ~(r1[0] & p[0]), w & ~((r1[0] & p[1]) | (r1[1] & sh(p[0], 1))), e & ~((r1[0] & p[2]) | (r1[2] & sh(p[0], -1)))
                else:
                    p = row_links(3, u, 0, v, 0)[1]
                    n, w, e = (n & ~(r1[0] & p[0]), w & ~((r1[0] & sh(p[2], 1)) | (r1[1] & sh(p[0], 1))),
                               e & ~((r1[0] & sh(p[1], -1)) | (r1[2] & sh(p[0], -1))))
            self.unite_links(key, up, (n, w, e))
        # Across d2: face voxels of the first and the last block, bits 2i + j.
        def first(k):
            return sum(((self.cls[k][2 * ij] & 1) << ij) for ij in range(4))

        def last(k):
            return sum(((self.cls[k][2 * ij + 1] >> 31) << ij) for ij in range(4))

        def sel(dx, dy):
            return (0x3 if dx < 0 else 0xC if dx > 0 else 0xF) & (0x5 if dy < 0 else 0xA if dy > 0 else 0xF)

        r0, r1, t2 = key
        lo = first(key) if t2 > 0 else 0
        hi = last(key) if t2 + 1 < self.t[2] else 0
        before = last((r0, r1, t2 - 1)) if lo else 0
        after = first((r0, r1, t2 + 1)) if hi else 0
        if before:
            self.unite(self.run(key, 0), self.run((r0, r1, t2 - 1), 31))
        for nr in range(4):
            up = self.preceding(key, nr)
            if up is None:
                continue
            own, opp = sel(*OFF[nr]), sel(-OFF[nr][0], -OFF[nr][1])
            if lo & own and not before & own and last((up[0], up[1], t2 - 1)) & opp:
                self.unite(self.run(key, 0), self.run((up[0], up[1], t2 - 1), 31))
            if hi & own and not after & own and first((up[0], up[1], t2 + 1)) & opp:
                self.unite(self.run(key, 31), self.run((up[0], up[1], t2 + 1), 0))

    def check(self, ref):
        to_label, to_root = {}, {}
        for X, Y, Z in np.argwhere(ref > 0):
            key = (int(X) // 2, int(Y) // 2, int(Z) // 64)
            root = self.find(self.run(key, (int(Z) % 64) // 2))
            label = int(ref[X, Y, Z])
            assert to_label.setdefault(root, label) == label, "joined apart"
            assert to_root.setdefault(label, root) == root, "split"


def volumes():
    rng = np.random.default_rng(11)
    for shape in ((18, 34, 66), (33, 70, 20), (5, 36, 130), (17, 33, 129)):
        for p in (0.02, 0.06, 0.12, 0.3, 0.55):
            yield shape, f"noise {p}", rng.random(shape) < p
        x, y, z = np.indices(shape)
        yield shape, "tile corners", (np.isin(x % 16, (0, 15)) & np.isin(y % 32, (0, 31)) & np.isin(z % 64, (0, 63))) & (rng.random(shape) < 0.5)
        yield shape, "tile faces", (np.isin(x % 16, (0, 1, 14, 15)) | np.isin(y % 32, (0, 31)) | np.isin(z % 64, (0, 1, 62, 63))) & (rng.random(shape) < 0.08)
        yield shape, "sheets", ((x + y + z) % 5 == 0) & (rng.random(shape) < 0.7)
    # Clusters of few voxels apart from one another, so that most links are the only ones: on a grid that
    # meets every alignment to blocks and tile borders.
    for i, (p, q) in enumerate(((0.08, 9), (0.12, 9), (0.16, 8), (0.2, 8), (0.25, 7), (0.12, 7), (0.16, 6), (0.2, 6)) * 2):
        shape = (36, 72, 132) if i < 8 else (19, 67, 1500)
        x, y, z = (c + o for c, o in zip(np.indices(shape), rng.integers(0, q, 3)))
        yield shape, f"clusters {p}", (x % q > 1) & (y % q > 1) & (z % q > 1) & (rng.random(shape) < p)


@pytest.mark.parametrize("case", range(48))
def test_kept_links_join_the_components(case):
    shape, name, mask = list(volumes())[case]
    m = Model(mask)
    for key in m.cls:
        if any(m.cls[key]):
            m.local(key)
            m.across(key)
    m.check(O.ccl3d(mask.astype(np.uint8))[0])
