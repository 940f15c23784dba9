"""H-matrix (hierarchical low-rank) representation of the BEM matrices on the GPU.

Host side (geometry only, once per mesh / wavelength):

* ``ClusterTree``   -- recursive bisection of the face centroids with a first
  split per particle (reference mnpbem/greenfun/clustertree.py:7-380, after
  Boerm et al., Eng. Anal. Bound. Elem. 27, 405 (2003));
* ``block_partition`` -- admissibility recursion over cluster pairs: leaf x
  leaf pairs are dense blocks, admissible pairs low-rank blocks
  (clustertree.py:304-376), with the wavenumber-aware criterion of
  ``make_kaware_fadmiss`` (mnpbem/greenfun/hmatrix.py:1284-1310).

Device side (libbem200, csrc/hmat.cu):

* the dense BEM matrix is gathered into cluster order; low-rank blocks are
  compressed by partially pivoted adaptive cross approximation, one CTA per
  block, with the reference's pivoting and stopping rule
  (hmatrix.py:195-336, tolerance ``htol``, rank <= ``kmax``); dense leaves are
  packed;
* the product H x runs in two kernels: T_b = V_b^T x for every low-rank block,
  then one CTA per block adds its rows, M_b times the block's x (or T) slice,
  into y (reference HMatrix.mtimes_vec, hmatrix.py:450-541).

The reference compresses each region-pair Green matrix (G11, G21, ...) and
forms G1 = G11 - G21 by H-matrix addition with QR/SVD recompression
(hmatrix.py:580-737).  Here the combined BEM matrices G1, G2, H1, H2 are
assembled densely on the GPU and compressed directly, which approximates the
same operators to the same tolerance.
"""
import ctypes

import numpy as np

from . import _native as nat


def _torch():
    import torch
    return torch


# --------------------------------------------------------------------------- tree
class ClusterTree:
    """Cluster tree of face centroids (reference clustertree.py:7-146).

    Attributes (0-based): son (nnodes, 2) children or -1, cind (nnodes, 2)
    first/last cluster index, mid (nnodes, 3), rad (nnodes,), ipart (nnodes,)
    particle of the node or -1, ind (n, 2): ind[c, 0] = face of cluster index
    c, ind[f, 1] = cluster index of face f.
    """

    def __init__(self, pos, cleaf=32, ipart_arr=None):
        self.pos = np.asarray(pos, dtype=np.float64)
        self.n = self.pos.shape[0]
        self._ipart = (np.zeros(self.n, dtype=np.int64) if ipart_arr is None
                       else np.asarray(ipart_arr, dtype=np.int64))
        self._build(int(cleaf))

    def _sphere(self, ind):
        p = self.pos[ind]
        lo, hi = p.min(axis=0), p.max(axis=0)
        return 0.5 * (lo + hi), 0.5 * float(np.linalg.norm(hi - lo))

    def _split(self, ind):
        ip = self._ipart[ind]
        if np.any(ip != ip[0]):  # first split: first particle against the rest
            mask = ip == ip[0]
            return ind[mask], ind[~mask], True
        p = self.pos[ind]
        lo, hi = p.min(axis=0), p.max(axis=0)
        ext = hi - lo
        k = int(np.argmax(ext))
        mask = self.pos[ind, k] < lo[k] + 0.5 * ext[k]
        i1, i2 = ind[mask], ind[~mask]
        if len(i1) == 0:
            i1, i2 = ind[:1], ind[1:]
        elif len(i2) == 0:
            i1, i2 = ind[:-1], ind[-1:]
        return i1, i2, False

    def _build(self, cleaf):
        n = self.n
        lo, hi = self.pos.min(axis=0), self.pos.max(axis=0)
        nodes = [dict(cs=0, ce=n - 1, mid=0.5 * (lo + hi), rad=0.5 * float(np.linalg.norm(hi - lo)), s1=-1, s2=-1,
                      leaf=None)]
        # explicit stack in the reference's recursion order (son 1 subtree, then son 2)
        stack = [(0, np.arange(n, dtype=np.int64), np.arange(n, dtype=np.int64))]
        while stack:
            ic, ind, cind = stack.pop()
            base = len(nodes)
            nodes[ic]["s1"], nodes[ic]["s2"] = base, base + 1
            i1, i2, psplit = self._split(ind)
            c1, c2 = cind[:len(i1)], cind[len(i1):]
            for ii, cc in ((i1, c1), (i2, c2)):
                m, r = self._sphere(ii)
                nodes.append(dict(cs=int(cc[0]), ce=int(cc[-1]), mid=m, rad=r, s1=-1, s2=-1, leaf=None))
            todo = []
            for off, ii, cc in ((0, i1, c1), (1, i2, c2)):
                if len(ii) > cleaf or psplit:
                    todo.append((base + off, ii, cc))
                else:
                    nodes[base + off]["leaf"] = ii
            stack.extend(reversed(todo))  # son 1 is expanded first
        nn = len(nodes)
        self.son = np.array([[d["s1"], d["s2"]] for d in nodes], dtype=np.int64)
        self.cind = np.array([[d["cs"], d["ce"]] for d in nodes], dtype=np.int64)
        self.mid = np.array([d["mid"] for d in nodes], dtype=np.float64)
        self.rad = np.array([d["rad"] for d in nodes], dtype=np.float64)
        c2p = np.empty(n, dtype=np.int64)
        for d in nodes:
            if d["leaf"] is not None:
                c2p[d["cs"]:d["ce"] + 1] = d["leaf"]
        p2c = np.empty(n, dtype=np.int64)
        p2c[c2p] = np.arange(n)
        self.ind = np.stack([c2p, p2c], axis=1)
        ip = np.empty(nn, dtype=np.int64)
        for i, d in enumerate(nodes):
            a, b = self._ipart[c2p[d["cs"]]], self._ipart[c2p[d["ce"]]]
            ip[i] = a if a == b else -1
        self.ipart = ip

    def is_leaf(self, i):
        return self.son[i, 0] == -1


def eta_fadmiss(eta=2.5):
    """Boerm's criterion eta * min(rad1, rad2) < dist (clustertree.py:311)."""
    return lambda r1, r2, d: eta * min(r1, r2) < d


def make_kaware_fadmiss(k, eta0=2.5):
    """Wavenumber-aware admissibility (reference hmatrix.py:1284-1310): the
    Boerm criterion, and for clusters wider than 1/|k| also a distance of at
    least one wavelength."""
    if k is None or not np.isfinite(k) or abs(k) < 1e-12:
        return eta_fadmiss(eta0)
    ka = abs(complex(k))
    lam = 2.0 * np.pi / ka

    def fadmiss(r1, r2, d):
        rmin = min(r1, r2)
        if eta0 * rmin >= d:
            return False
        if ka * rmin > 1.0 and d < lam:
            return False
        return True

    def many(r1, r2, d):  # the same test on arrays
        rmin = np.minimum(r1, r2)
        return ~((eta0 * rmin >= d) | ((ka * rmin > 1.0) & (d < lam)))
    fadmiss.many = many
    return fadmiss


def block_partition(tree, fadmiss):
    """Dense (leaf x leaf) and low-rank (admissible) cluster pairs, in the
    reference's recursion order (clustertree.py:324-376)."""
    many = getattr(fadmiss, "many", None)
    if many is not None:
        return _block_partition_arrays(tree, many)
    dense, lowrank = [], []

    def admissible(i1, i2):
        if tree.is_leaf(i1) and tree.is_leaf(i2):
            return 2
        if tree.ipart[i1] == -1 or tree.ipart[i2] == -1:
            return 0
        d = float(np.linalg.norm(tree.mid[i1] - tree.mid[i2]))
        return 1 if fadmiss(tree.rad[i1], tree.rad[i2], d) else 0

    stack = [(0, 0)]
    while stack:
        i1, i2 = stack.pop()
        ad = admissible(i1, i2)
        if ad == 2:
            dense.append((i1, i2))
        elif ad == 1:
            lowrank.append((i1, i2))
        else:
            s1 = [i1] if tree.is_leaf(i1) else [tree.son[i1, 0], tree.son[i1, 1]]
            s2 = [i2] if tree.is_leaf(i2) else [tree.son[i2, 0], tree.son[i2, 1]]
            stack.extend(reversed([(a, b) for a in s1 for b in s2]))
    return dense, lowrank


def _block_partition_arrays(tree, many):
    """The same recursion, one level of all pairs at a time: a pair is replaced
    in place by its son pairs, so the sequence stays in recursion order."""
    leaf = tree.son[:, 0] == -1
    i1 = i2 = np.zeros(1, dtype=np.int64)
    kind = np.zeros(1, dtype=np.int8)  # 0 open, 1 low rank, 2 dense
    while True:
        o = np.flatnonzero(kind == 0)
        if len(o) == 0:
            break
        a, b = i1[o], i2[o]
        both = leaf[a] & leaf[b]
        d = np.sqrt(np.sum((tree.mid[a] - tree.mid[b]) ** 2, axis=1))
        adm = (tree.ipart[a] != -1) & (tree.ipart[b] != -1) & many(tree.rad[a], tree.rad[b], d)
        kind[o] = np.where(both, 2, np.where(adm, 1, 0))
        n1 = np.where(leaf[i1], 1, 2)
        n2 = np.where(leaf[i2], 1, 2)
        reps = np.where(kind == 0, n1 * n2, 1)
        src = np.repeat(np.arange(len(kind)), reps)
        pos = np.arange(len(src)) - np.repeat(np.cumsum(reps) - reps, reps)  # son pair within its parent
        grow = kind[src] == 0
        p1, p2 = pos // n2[src], pos % n2[src]
        j1 = np.where(grow & ~leaf[i1[src]], tree.son[i1[src], np.minimum(p1, 1)], i1[src])
        j2 = np.where(grow & ~leaf[i2[src]], tree.son[i2[src], np.minimum(p2, 1)], i2[src])
        i1, i2, kind = j1, j2, kind[src]
    pairs = np.stack([i1, i2], axis=1)
    return ([tuple(v) for v in pairs[kind == 2].tolist()], [tuple(v) for v in pairs[kind == 1].tolist()])


# --------------------------------------------------------------------------- device H-matrix
class _Layout:
    """Block structure of H-matrices on one partition: block tables, storage
    offsets and work items, on the host and on the device."""

    _RUN = 512

    def __init__(self, tree, dense, lowrank, kmax, dev):
        torch = _torch()
        lo = tree.cind[:, 0].astype(np.int32)
        ln = (tree.cind[:, 1] - tree.cind[:, 0] + 1).astype(np.int32)

        def table(pairs):
            p = np.asarray(pairs, dtype=np.int64).reshape(-1, 2)
            a, b = p[:, 0], p[:, 1]
            return np.ascontiguousarray(np.stack([lo[a], ln[a], lo[b], ln[b]], axis=1))

        # dense leaves (r0, m, c0, nb) and packed offsets; low-rank blocks,
        # storage for the maximum rank min(m, nb, kmax)
        self.db, self.lb = db, lb = table(dense), table(lowrank)
        self.kcap = kcap = np.minimum(np.minimum(lb[:, 1], lb[:, 3]), kmax).astype(np.int64)

        def offsets(sizes):
            off = np.zeros(len(sizes) + 1, dtype=np.int64)
            off[1:] = np.cumsum(sizes)
            return off
        self.doff, self.uoff = offsets(db[:, 1].astype(np.int64) * db[:, 3]), offsets(lb[:, 1].astype(np.int64) * kcap)
        self.voff, self.toff = offsets(lb[:, 3].astype(np.int64) * kcap), offsets(kcap)

        def split(rows, step, first=0):  # (block, first row) for every `step` rows of every block
            cnt = (rows.astype(np.int64) + step - 1) // step
            blk = np.repeat(np.arange(len(rows)), cnt)
            j = np.arange(len(blk)) - np.repeat(np.cumsum(cnt) - cnt, cnt)
            return np.stack([blk + first, j * step], axis=1).astype(np.int32)
        vit = split(lb[:, 3], 128)
        bit = np.concatenate([split(db[:, 1], 32), split(lb[:, 1], 32, first=len(db))])
        tiles, blist = self._row_tiles(tree, lo, ln)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        self.dev = {k: t(v) for k, v in dict(
            dblk=db.reshape(-1), doff=self.doff, lblk=lb.reshape(-1), uoff=self.uoff, voff=self.voff, toff=self.toff,
            kcap=kcap.astype(np.int32), c2p=tree.ind[:, 0].astype(np.int32), p2c=tree.ind[:, 1].astype(np.int32),
            vitems=vit.reshape(-1), bitems=bit.reshape(-1), tiles=tiles.reshape(-1), blist=blist).items()}
        self.nvitems, self.nbitems, self.ntiles = len(vit), len(bit), len(tiles)

    def _row_tiles(self, tree, lo, ln):
        """Phase B of the operator product: up to 32 rows of a leaf cluster with
        a run of at most 128 of the blocks over them (every block's rows are a
        union of whole leaf clusters), about _RUN matrix columns per run."""
        leaf = np.flatnonzero(tree.son[:, 0] == -1)
        leaf = leaf[np.argsort(lo[leaf], kind="stable")]
        start = lo[leaf]
        blocks = np.concatenate([self.db, self.lb])
        cost = np.concatenate([self.db[:, 3].astype(np.int64), np.minimum(self.kcap, 24)]) + 8
        # leaves covered by each block
        f = np.searchsorted(start, blocks[:, 0])
        e = np.searchsorted(start, blocks[:, 0] + blocks[:, 1])
        cnt = e - f
        blk = np.repeat(np.arange(len(blocks)), cnt)
        lf = np.arange(len(blk)) - np.repeat(np.cumsum(cnt) - cnt, cnt) + np.repeat(f, cnt)
        order = np.lexsort((blk, lf))
        blk, lf = blk[order].astype(np.int32), lf[order]
        begin = np.searchsorted(lf, np.arange(len(leaf)))
        c = np.cumsum(cost[blk]) if len(blk) else np.zeros(0, np.int64)
        base = np.concatenate([[0], c])[begin] if len(blk) else np.zeros(len(leaf), np.int64)
        run = (c - cost[blk] - base[lf]) // self._RUN if len(blk) else c
        head = np.flatnonzero(np.concatenate([[True], (lf[1:] != lf[:-1]) | (run[1:] != run[:-1])])) if len(blk) else \
            np.zeros(0, np.int64)
        tail = np.concatenate([head[1:], [len(blk)]]).astype(np.int64) if len(head) else head
        rows, first = ln[leaf][lf[head]].astype(np.int64), start[lf[head]].astype(np.int64)
        parts = (rows + 31) // 32
        src = np.repeat(np.arange(len(head)), parts)
        k = np.arange(len(src)) - np.repeat(np.cumsum(parts) - parts, parts)
        tiles = np.stack([first[src] + 32 * k, np.minimum(32, rows[src] - 32 * k), head[src], tail[src]], axis=1)
        return tiles.astype(np.int32), blk


class HMatrixGPU:
    """Compressed n x n complex128 matrix on the device (cluster order).

    ``compress(M)`` takes the dense matrix in particle order; ``matvec(x, y)``
    computes y = H x for n x w row-major device arrays in cluster order.
    """

    def __init__(self, tree, dense, lowrank, htol=1e-6, kmax=100, device="cuda", layout=None):
        torch = _torch()
        self.tree = tree
        self.n = tree.n
        self.htol = float(htol)
        self.kmax = int(kmax)
        dev = torch.device(device)
        self.dev = dev
        self.layout = L = layout if layout is not None else _Layout(tree, dense, lowrank, self.kmax, dev)
        self.ndense, self.nlow = len(L.db), len(L.lb)
        self._db, self._lb, self._kcap = L.db, L.lb, L.kcap
        self._doff_h, self._uoff_h, self._voff_h = L.doff, L.uoff, L.voff
        for k in ("dblk", "doff", "lblk", "uoff", "voff", "toff", "kcap", "c2p", "p2c", "vitems", "bitems"):
            setattr(self, k, L.dev[k])
        self.nvitems, self.nbitems = L.nvitems, L.nbitems
        self.D = torch.empty(max(int(L.doff[-1]), 1), dtype=torch.complex128, device=dev)
        self.U = torch.empty(max(int(L.uoff[-1]), 1), dtype=torch.complex128, device=dev)
        self.V = torch.empty(max(int(L.voff[-1]), 1), dtype=torch.complex128, device=dev)
        self.rank = torch.zeros(max(self.nlow, 1), dtype=torch.int32, device=dev)
        self.ranks = None

    def compress(self, M, scratch=None):
        """Compress the dense n x n complex128 device matrix M (particle order)."""
        torch = _torch()
        n = self.n
        Mc = scratch if scratch is not None else torch.empty((n, n), dtype=torch.complex128, device=self.dev)
        s = nat.stream_ptr()
        nat.call("bem200_hmat_permute", n, nat.ptr(M), nat.ptr(self.c2p), nat.ptr(Mc), s)
        if self.ndense:
            nat.call("bem200_hmat_pack_dense", self.ndense, nat.ptr(self.dblk), nat.ptr(self.doff), n, nat.ptr(Mc),
                     nat.ptr(self.D), s)
        if self.nlow:
            max_rows = int(max(self._lb[:, 1].max(), self._lb[:, 3].max()))
            nat.call("bem200_hmat_aca", self.nlow, nat.ptr(self.lblk), nat.ptr(self.uoff), nat.ptr(self.voff),
                     nat.ptr(self.kcap), n, nat.ptr(Mc), self.htol, nat.ptr(self.U), nat.ptr(self.V),
                     nat.ptr(self.rank), max_rows, int(self._kcap.max()), s)
            self.ranks = self.rank.cpu().numpy()[:self.nlow].copy()
        else:
            self.ranks = np.zeros(0, dtype=np.int32)
        return self

    def compress_green(self, g, enei, which, fetch=True):
        """Compress BEM matrix ``which`` (0 = G1, 1 = G2, 2 = H1, 3 = H2) of the
        Green function ``g`` (a CompGreenRet) at ``enei`` with every entry of the
        dense leaves and of the ACA rows and columns computed on demand: no
        n x n matrix is formed (bem200_hmat_compress_green).  fetch=False leaves
        the ranks on the device (``fetch_ranks`` reads them later)."""
        ks = g.wavenumbers(enei)
        kmat = (ctypes.c_double * (2 * len(ks)))(*[v for k in ks for v in (k.real, k.imag)])
        blk = g._blk_mat([(0, 0), (1, 0), (1, 1), (0, 1)])
        r = g.refined
        has_ref = r.nref > 0
        max_rows = int(max(self._lb[:, 1].max(), self._lb[:, 3].max())) if self.nlow else 1
        max_kcap = int(self._kcap.max()) if self.nlow else 1
        nat.call("bem200_hmat_compress_green", int(which), self.n, g.npart, nat.ptr(g.pid), nat.ptr(blk), len(ks),
                 ctypes.cast(kmat, ctypes.c_void_p), nat.ptr(g.pos), nat.ptr(g.nvec), nat.ptr(g.area),
                 nat.ptr(r.row_ptr) if has_ref else None, nat.ptr(r.col) if has_ref else None, g.order,
                 nat.ptr(r.g) if has_ref else None, nat.ptr(r.fn) if has_ref else None, nat.ptr(self.c2p),
                 self.ndense, nat.ptr(self.dblk), nat.ptr(self.doff), nat.ptr(self.D), self.nlow, nat.ptr(self.lblk),
                 nat.ptr(self.uoff), nat.ptr(self.voff), nat.ptr(self.kcap), self.htol, nat.ptr(self.U),
                 nat.ptr(self.V), nat.ptr(self.rank), max_rows, max_kcap, nat.stream_ptr())
        return self.fetch_ranks() if fetch else self

    def fetch_ranks(self):
        self.ranks = self.rank.cpu().numpy()[:self.nlow].copy() if self.nlow else np.zeros(0, dtype=np.int32)
        return self

    def compression(self):
        """Stored elements / n^2 (reference HMatrix.compression, hmatrix.py:739-756)."""
        ne = int(self._doff_h[-1]) + int(np.sum(self.ranks.astype(np.int64) * (self._lb[:, 1] + self._lb[:, 3])))
        return ne / float(self.n * self.n)

    def matvec(self, x, y, w):
        """y = H x, x and y n x w row-major complex128 in cluster order, with
        large blocks split over several CTAs (bem200_hmat_matvec_items)."""
        torch = _torch()
        tbuf = getattr(self, "_tbuf", None)
        need = max(int(np.sum(self._kcap)) * w, 1)
        if tbuf is None or tbuf.numel() < need:
            self._tbuf = tbuf = torch.empty(need, dtype=torch.complex128, device=self.dev)
        nat.call("bem200_hmat_matvec_items", self.n, w, nat.ptr(x), self.nlow, nat.ptr(self.lblk),
                 nat.ptr(self.voff), nat.ptr(self.uoff), nat.ptr(self.toff), nat.ptr(self.kcap), nat.ptr(self.rank),
                 nat.ptr(self.U), nat.ptr(self.V), nat.ptr(tbuf), int(np.sum(self._kcap)) * w, self.ndense,
                 nat.ptr(self.dblk), nat.ptr(self.doff), nat.ptr(self.D), self.nvitems, nat.ptr(self.vitems),
                 self.nbitems, nat.ptr(self.bitems), nat.ptr(y), nat.stream_ptr())

    def matvec_per_block(self, x, y, w):
        """y = H x with one CTA per block (bem200_hmat_matvec)."""
        torch = _torch()
        tbuf = getattr(self, "_tbuf", None)
        need = max(int(np.sum(self._kcap)) * w, 1)
        if tbuf is None or tbuf.numel() < need:
            self._tbuf = tbuf = torch.empty(need, dtype=torch.complex128, device=self.dev)
        nat.call("bem200_hmat_matvec", self.n, w, nat.ptr(x), self.nlow, nat.ptr(self.lblk), nat.ptr(self.voff),
                 nat.ptr(self.uoff), nat.ptr(self.toff), nat.ptr(self.kcap), nat.ptr(self.rank), nat.ptr(self.U),
                 nat.ptr(self.V), nat.ptr(tbuf), self.ndense, nat.ptr(self.dblk), nat.ptr(self.doff),
                 nat.ptr(self.D), nat.ptr(y), nat.stream_ptr())


def particle_index(p):
    """Particle of every face of a compound particle (or None for one particle)."""
    if not hasattr(p, "p") or len(p.p) <= 1:
        return None
    off = np.asarray(p.offsets)
    return np.repeat(np.arange(len(p.p)), np.diff(off)).astype(np.int64)


class BEMHMatrices:
    """G1, G2, H1, H2 of the BEM as device H-matrices and the BEM operator on them.

    ``build(enei)`` compresses the four matrices (wavenumber-aware
    admissibility at k = 2 pi / enei, as the reference ACACompGreenRet.eval,
    aca_compgreen_ret.py:156-164): from dense matrices already at hand, or
    with entries computed on demand from the Green function (the default when
    none are given); ``apply`` is the FP64 operator of ``bem200_bem_apply``
    with the four products done by H-matrix matvecs.
    """

    def __init__(self, p, g, htol=1e-6, kmax=(4, 100), cleaf=200, eta=2.5):
        self.p = p
        self.g = g
        self.n = p.n
        self.htol = float(max(htol) if hasattr(htol, "__iter__") else htol)
        self.kmax = int(max(kmax) if hasattr(kmax, "__iter__") else kmax)
        self.cleaf = int(cleaf)
        self.eta = float(eta)
        self.tree = ClusterTree(p.pos, cleaf=self.cleaf, ipart_arr=particle_index(p))
        self.H = None
        self.enei = None

    def build(self, enei, mats=None, fill="green"):
        """Compress G1, G2, H1, H2 at ``enei``.  ``mats`` may hand in the four
        dense complex128 matrices already assembled at this wavelength;
        without them, fill='green' computes every stored entry on demand from
        the Green function (no n x n matrix), fill='dense' assembles the dense
        matrices first."""
        torch = _torch()
        n = self.n
        fad = make_kaware_fadmiss(2.0 * np.pi / enei, eta0=self.eta)
        dense, low = block_partition(self.tree, fad)
        dev = self.g.device
        if mats is None and fill == "green":
            self.H = None
            layout = _Layout(self.tree, dense, low, self.kmax, dev)
            self.H = [HMatrixGPU(self.tree, dense, low, htol=self.htol, kmax=self.kmax, layout=layout)
                      for _ in range(4)]
            # the four fills side by side: each is paced by its few largest
            # blocks (one CTA per block, 1.1 ms at 3600 faces)
            cur = torch.cuda.current_stream()
            sides = [torch.cuda.Stream() for _ in range(4)]
            try:
                for w, (h, s) in enumerate(zip(self.H, sides)):
                    s.wait_stream(cur)
                    with torch.cuda.stream(s):
                        h.compress_green(self.g, enei, w, fetch=False)
            except BaseException:
                self.H = None  # its memory is free for work behind the fills already queued
                raise
            finally:
                for s in sides:
                    cur.wait_stream(s)
            for h in self.H:
                h.fetch_ranks()
            self.enei = enei
            return self
        if fill not in ("green", "dense"):
            raise ValueError("BEMHMatrices.build: fill must be 'green' or 'dense'")
        if mats is None:
            mats = [torch.empty((n, n), dtype=torch.complex128, device=dev) for _ in range(4)]
            self.g.bem_matrices(enei, dtype="c128", out=mats)
        self.H = None
        scratch = torch.empty((n, n), dtype=torch.complex128, device=dev)
        layout = _Layout(self.tree, dense, low, self.kmax, dev)
        self.H = [HMatrixGPU(self.tree, dense, low, htol=self.htol, kmax=self.kmax, layout=layout).compress(M, scratch)
                  for M in mats]
        del mats, scratch
        self.enei = enei
        return self

    def compression(self):
        return [h.compression() for h in self.H]

    def apply(self, npol, eps_mode, e1p, e2p, nvec, k0, x, out):
        """out = A x (the full BEM operator) for x in the solution layout."""
        torch = _torch()
        n = self.n
        L = self.H[0].layout
        d = L.dev
        t_len = int(L.toff[-1]) * 8 * npol
        need = int(nat.lib().bem200_hmat_operator_workspace_size(n, npol, t_len))
        buf = getattr(self, "_opbuf", None)
        if buf is None or buf.numel() < need:
            self._opbuf = buf = torch.empty(need, dtype=torch.uint8, device=x.device)

        def four(name):
            return (ctypes.c_void_p * 4)(*[getattr(h, name).data_ptr() for h in self.H])
        nat.call("bem200_hmat_operator", n, npol, nat.ptr(x), eps_mode, e1p, e2p, nat.ptr(nvec), k0, nat.ptr(d["c2p"]),
                 nat.ptr(d["p2c"]), len(L.lb), nat.ptr(d["lblk"]), nat.ptr(d["voff"]), nat.ptr(d["uoff"]),
                 nat.ptr(d["toff"]), nat.ptr(d["kcap"]), t_len, len(L.db), nat.ptr(d["dblk"]), nat.ptr(d["doff"]),
                 four("D"), four("U"), four("V"), four("rank"), L.nvitems, nat.ptr(d["vitems"]), L.ntiles,
                 nat.ptr(d["tiles"]), nat.ptr(d["blist"]), nat.ptr(buf), None, nat.ptr(out), nat.stream_ptr())
