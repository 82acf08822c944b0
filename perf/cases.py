"""Performance cases of the quantized H-matrix apply.

Every case is one pass of what a program does with a resident matrix: it
holds the matrix (built from its QHMAT001 image, as a loaded file is) and a
right-hand side, and applies one to the other through the package's public
entry points.

The matrices are synthetic, so that they can be made in a second: the
partition is the real one (``spatial_partition`` of seeded uniform points, the
workloads' leaf sizes), the ranks and the share of each code width follow what
``from_kernel`` gives for the benchmark's kernels (log on the square at 1e-6,
Yukawa on the cube at 1e-5, 1/(r + 0.4) on the line at 1e-6), and the codes,
scales and dense diagonal entries are random.
"""

from __future__ import annotations

import numpy as np
import torch

from qhmat_gb300 import HMatrix, PrecisionHMatrix, load_library
from qhmat_gb300.batching import BatchedHMatrices
from qhmat_gb300.construct import spatial_partition

DEVICE = 0

# Rank of a neighbouring leaf block (not admissible) and of an admissible one,
# by dimension of the points; the spread is about +-20%.
RANKS = {1: (6.0, 6.0), 2: (17.5, 11.0), 3: (33.0, 21.0)}
# Code widths in the order of the components (widest first) and the share of
# the components up to and including each.
WIDTHS = np.array([32, 24, 16, 12, 8, 4])
WIDTH_SHARE = np.array([0.20, 0.45, 0.56, 0.67, 0.80, 1.0])


# ------------------------------------------------------------------ matrices

def _structure(n, dim, leaf, seed):
    """Permutation, blocks (row0, row1, col0, col1, admissible) and the rank
    of every block (0 for a dense diagonal one)."""
    rng = np.random.default_rng(seed)
    perm, rects = spatial_partition(rng.random((n, dim)), leaf)
    r = np.array([b[:4] for b in rects], np.int64)
    adm = np.array([b[4] for b in rects], bool)
    dense = (r[:, 0] == r[:, 2]) & (r[:, 1] == r[:, 3])
    rows, cols = r[:, 1] - r[:, 0], r[:, 3] - r[:, 2]
    near, far = RANKS[dim]
    mean = np.where(adm, far, near)
    rank = np.rint(mean * (1.0 + 0.2 * np.clip(rng.standard_normal(len(r)), -2, 2))).astype(np.int64)
    # a block cannot have more than its smaller side; leaves smaller than the
    # workloads' keep about half of it
    rank = np.clip(rank, 1, np.maximum(1, np.minimum(rows, cols) // 2))
    rank[dense] = 0
    return perm, r, adm, dense, rank


class _Arrays:
    """A matrix as flat arrays: the blocks in order, their components'
    widths and scales, the packed words of each side and the dense entries."""

    def __init__(self, n, dim, leaf, seed):
        perm, r, adm, dense, rank = _structure(n, dim, leaf, seed)
        rng = np.random.default_rng(seed + 1)
        self.n, self.perm, self.rects, self.adm, self.dense, self.rank = n, perm, r, adm, dense, rank
        rows, cols = r[:, 1] - r[:, 0], r[:, 3] - r[:, 2]
        self.comp0 = np.concatenate([[0], np.cumsum(rank)])
        self.block = np.repeat(np.arange(len(r)), rank)
        j = np.arange(self.comp0[-1]) - self.comp0[self.block]
        share = (j + 0.5) / rank[self.block]
        self.width = WIDTHS[np.searchsorted(WIDTH_SHARE, share)].astype(np.int64)
        self.m, self.k = rows[self.block], cols[self.block]
        # singular values over about six decades, split evenly on the factors
        sigma = 10.0 ** (-6.0 * share) * rng.uniform(0.5, 1.5, len(j))
        q = 2.0 ** (self.width - 1) - 1
        self.left_scale = np.sqrt(sigma / self.m) * 2.0 / q
        self.right_scale = np.sqrt(sigma / self.k) * 2.0 / q
        self.left_words, self.left_off = self._words(rng, self.m)
        self.right_words, self.right_off = self._words(rng, self.k)
        self.dense_off = np.concatenate([[0], np.cumsum(np.where(dense, rows * cols, 0))])
        self.dense_values = rng.standard_normal(int(self.dense_off[-1]))

    def _words(self, rng, count):
        """One run of words per component: uniform codes in [-q, q], each run
        on a fresh word with zero bits after its last code."""
        bits = count * self.width
        nw = (bits + 31) // 32
        off = np.concatenate([[0], np.cumsum(nw)])
        w = rng.integers(0, 1 << 63, (int(off[-1]) + 1) // 2 + 1, np.int64, endpoint=False)
        w = (w ^ (w << 1)).view(np.uint32)[: int(off[-1])].copy()
        # the code -2^(b-1), which the writer never makes, becomes 0 (widths
        # whose codes lie inside one word)
        for b, ones in ((4, 0x11111111), (8, 0x01010101), (16, 0x00010001), (32, 1)):
            sel = np.repeat(self.width == b, nw)
            v = w[sel]
            top = np.uint32(ones << (b - 1) & 0xFFFFFFFF)
            low = v & ~top
            w[sel] = low | (v & top & (low + (top - np.uint32(ones))))
        last, rest = off[1:] - 1, bits % 32
        cut = rest > 0
        w[last[cut]] &= ((1 << rest[cut]) - 1).astype(np.uint32)
        return w, off

    def image(self):
        """The QHMAT001 bytes of this matrix."""
        r, le = self.rects, "<u8"
        parts = [b"QHMAT001", np.array([1, self.n, len(r)], le).tobytes(), np.asarray(self.perm, le).tobytes()]
        lw, rw = self.left_words.data, self.right_words.data
        heads = r.astype(le).tobytes()
        width = self.width.astype(np.uint8).tobytes()
        ls, rs, dv = self.left_scale.tobytes(), self.right_scale.tobytes(), self.dense_values.tobytes()
        comp0, lo, ro, do = (a.tolist() for a in (self.comp0, self.left_off, self.right_off, self.dense_off))
        adm, dense = self.adm.tolist(), self.dense.tolist()
        bounds = np.array([1e-7, 1e-7]).tobytes()
        for b in range(len(r)):
            parts.append(heads[32 * b:32 * b + 32])
            parts.append(bytes((adm[b], dense[b])))
            if dense[b]:
                parts.append(dv[8 * do[b]:8 * do[b + 1]])
                continue
            c0, c1 = comp0[b], comp0[b + 1]
            parts += [(c1 - c0).to_bytes(8, "little"), len(WIDTHS).to_bytes(8, "little"), bounds, width[c0:c1],
                      ls[8 * c0:8 * c1], rs[8 * c0:8 * c1], lw[lo[c0]:lo[c1]], rw[ro[c0]:ro[c1]]]
        body = b"".join(parts)
        return body + int(load_library().qh_fnv1a64(body, len(body))).to_bytes(8, "little")

    def bytes_and_codes(self):
        """Packed bytes of the matrix (words, scales, dense entries) and the
        multiply-adds of one column."""
        code_bytes = 4 * (len(self.left_words) + len(self.right_words)) + 16 * len(self.width)
        macs = int((self.m + self.k).sum()) + int(self.dense_off[-1])
        return code_bytes + 8 * int(self.dense_off[-1]), macs

    # ---- the represented matrix in 64 bits

    def _codes(self, words, off, sel, count, width):
        """Codes of the components ``sel`` (all of ``width`` bits, ``count``
        of them each) as float64 [component][entry]."""
        dev = words.device
        bit = torch.arange(count, device=dev, dtype=torch.int64) * width
        base = off[sel][:, None] + (bit >> 5)[None, :]
        lo = words[base].to(torch.int64) & 0xFFFFFFFF
        hi = words[torch.clamp(base + 1, max=len(words) - 1)].to(torch.int64) & 0xFFFFFFFF
        sh = (bit & 31)[None, :]
        v = (lo >> sh) | torch.where(sh + width > 32, hi << (32 - sh), torch.zeros_like(hi))
        v = v & ((1 << width) - 1)
        return torch.where(v >= 1 << (width - 1), v - (1 << width), v).to(torch.float64)

    def _groups(self, *by):
        """Component numbers, grouped by equal values of ``by``, at most 2^22
        codes to a group."""
        key = np.stack([self.width, *by], 1)
        uniq, inv = np.unique(key, axis=0, return_inverse=True)
        inv = inv.reshape(-1)
        order = np.argsort(inv, kind="stable")
        ends = np.concatenate([[0], np.cumsum(np.bincount(inv, minlength=len(uniq)))])
        for g, values in enumerate(uniq):
            most = max(1, (1 << 22) // int(max(values[1:])))
            for a in range(int(ends[g]), int(ends[g + 1]), most):
                yield [int(v) for v in values], order[a:min(a + most, int(ends[g + 1]))]

    def exact_apply(self, x):
        """y = A x in 64 bits (x: [n][p] on the device, source order)."""
        dev = x.device
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        perm = up(self.perm)
        xc = x[perm]
        u = torch.zeros(len(self.width), x.shape[1], dtype=torch.float64, device=dev)
        y = torch.zeros_like(xc)
        col0, row0 = up(self.rects[self.block, 2]), up(self.rects[self.block, 0])
        sl, sr = up(self.left_scale), up(self.right_scale)
        for words, off, side in ((self.right_words, self.right_off, 1), (self.left_words, self.left_off, 0)):
            words, off = up(words.view(np.int32)), up(off)
            for (w, count), sel in self._groups(self.k if side else self.m):
                sel = up(sel)
                codes = self._codes(words, off, sel, count, w)
                for a in range(0, x.shape[1], 8):
                    if side:
                        at = col0[sel][:, None] + torch.arange(count, device=dev)
                        u[sel, a:a + 8] = sr[sel][:, None] * torch.einsum("ci,cip->cp", codes, xc[:, a:a + 8][at])
                    else:
                        at = (row0[sel][:, None] + torch.arange(count, device=dev)).reshape(-1)
                        add = (codes[:, :, None] * (sl[sel][:, None] * u[sel, a:a + 8])[:, None, :])
                        y[:, a:a + 8].index_add_(0, at, add.reshape(-1, add.shape[2]))
        dv = up(self.dense_values)
        for b in np.flatnonzero(self.dense):
            r0, r1, c0, c1 = (int(v) for v in self.rects[b])
            blk = dv[int(self.dense_off[b]):int(self.dense_off[b + 1])].reshape(r1 - r0, c1 - c0)
            y[r0:r1] += blk @ xc[c0:c1]
        out = torch.empty_like(y)
        out[perm] = y
        return out

    def exact_dense(self):
        """The represented matrix in 64 bits, source order."""
        dev = torch.device("cuda", DEVICE)
        return self.exact_apply(torch.eye(self.n, dtype=torch.float64, device=dev))


def _image(n, dim, leaf, seed):
    return _Arrays(n, dim, leaf, seed).image()


# --------------------------------------------------------------------- cases
#
# op: "plain" and "precision" are the two forms of matmul, "batch" many
# matrices in one graph launch, "dense" the reconstruction.  io: where the
# right-hand side lives (NumPy array, or tensor on the device); loop: an
# iterative solver's call, which keeps a workspace and leaves the status
# unread until later.

def listed():
    return [
        # one step of an iterative solver on a small matrix: launches and latency
        {"name": "solve-1d-2048", "op": "plain", "n": 2048, "dim": 1, "leaf": 32, "rhs": 1, "io": "device", "loop": True},
        # the quick-start call: a small matrix, four columns, NumPy in and out
        {"name": "numpy-1d-2048x4", "op": "plain", "n": 2048, "dim": 1, "leaf": 32, "rhs": 4, "io": "host", "loop": False},
        # the headline workload: one large matrix, one column, in a solver
        {"name": "solve-2d-32768", "op": "plain", "n": 32768, "dim": 2, "leaf": 64, "rhs": 1, "io": "device", "loop": True},
        # the same kind of apply from NumPy, an odd order
        {"name": "numpy-2d-12345", "op": "plain", "n": 12345, "dim": 2, "leaf": 64, "rhs": 1, "io": "host", "loop": False},
        # a few columns (block solvers, gradient estimates), odd sizes
        {"name": "few-2d-9001x3", "op": "plain", "n": 9001, "dim": 2, "leaf": 32, "rhs": 3, "io": "device", "loop": False},
        # the columns one served batch of a tight-tolerance matrix holds
        {"name": "served-2d-16384x16", "op": "plain", "n": 16384, "dim": 2, "leaf": 64, "rhs": 16, "io": "device", "loop": False},
        # a wide block of columns at full precision on a 3-D matrix
        {"name": "block-3d-8192x64", "op": "plain", "n": 8192, "dim": 3, "leaf": 64, "rhs": 64, "io": "device", "loop": False},
        # the precision form: 64 columns in one pass, and a narrow odd count
        {"name": "precision-3d-8192x64", "op": "precision", "n": 8192, "dim": 3, "leaf": 64, "rhs": 64, "io": "device", "loop": False},
        {"name": "precision-2d-5003x11", "op": "precision", "n": 5003, "dim": 2, "leaf": 64, "rhs": 11, "io": "host", "loop": False},
        # many small matrices with a few columns each, one graph launch
        {"name": "batch-24", "op": "batch", "n": 2048, "dim": 2, "leaf": 32, "rhs": 16, "count": 24, "form": "plain"},
        # the dense matrix, to inspect or to hand to a dense solver
        {"name": "dense-2d-2048", "op": "dense", "n": 2048, "dim": 2, "leaf": 64},
    ]


def draw(rng):
    def log(a, b):
        return int(round(a * (b / a) ** rng.random()))

    op = rng.choice(["plain", "plain", "plain", "precision", "batch", "dense"])
    dim = rng.choice([1, 2, 2, 3])
    c = {"op": op, "dim": dim, "leaf": 64 if dim == 3 else rng.choice([32, 64])}
    if op == "dense":
        return dict(c, n=log(300, 2048))
    if op == "batch":
        return dict(c, n=log(512, 2048), dim=min(dim, 2), rhs=log(1, 32), count=rng.randint(8, 24),
                    form=rng.choice(["plain", "plain", "precision"]))
    c["io"] = rng.choice(["device", "device", "host"])
    c["loop"] = c["io"] == "device" and rng.random() < 0.5
    if op == "precision":
        return dict(c, n=log(1000, 8192), rhs=log(2, 64))
    rhs = rng.choice([1, log(2, 64)])
    return dict(c, n=log(1000, 8192 if dim == 3 else 32768 if rhs == 1 else 16384), rhs=rhs)


def _batch_specs(case):
    """(order, columns) of each matrix of a batch: orders down to a quarter
    of the largest, one to ``rhs`` columns each."""
    rng = np.random.default_rng(case["count"])
    orders = np.rint(case["n"] * 0.25 ** rng.random(case["count"])).astype(int)
    return [(int(n), int(p)) for n, p in zip(orders, rng.integers(1, case["rhs"] + 1, case["count"]))]


def _rhs(case, seed):
    """N(0, 1) columns, as the workloads have them."""
    if case["op"] == "batch":
        return np.random.default_rng(seed + 2).standard_normal(sum(n * p for n, p in _batch_specs(case)))
    x = np.random.default_rng(seed + 2).standard_normal((case["n"], case["rhs"]))
    return x[:, 0].copy() if case["rhs"] == 1 else x


def prepare(case, seed):
    op, dev = case["op"], torch.device("cuda", DEVICE)
    s = {"case": case}
    if op == "batch":
        specs = _batch_specs(case)
        images = [_image(n, case["dim"], case["leaf"], seed + 100 * k) for k, (n, _) in enumerate(specs)]
        s["b"] = BatchedHMatrices(images, [p for _, p in specs], device=DEVICE, forms=case["form"], autotune=False)
        s["x"] = torch.from_numpy(_rhs(case, seed)).to(dev)
        s["y"] = torch.zeros_like(s["x"])
        s["b"].capture(s["x"], s["y"])
        return s
    image = _image(case["n"], case["dim"], case["leaf"], seed)
    s["h"] = (PrecisionHMatrix if op == "precision" else HMatrix).from_bytes(image, device=DEVICE)
    if op == "dense":
        return s
    s["x"] = _rhs(case, seed)
    if case["io"] == "device":
        s["x"] = torch.from_numpy(s["x"]).to(dev)
    if case["loop"]:
        s["ws"] = torch.empty(s["h"].workspace_bytes(case["rhs"]), dtype=torch.uint8, device=dev)
    return s


def run(s):
    op = s["case"]["op"]
    if op == "batch":
        s["b"].replay()
        return s["y"]
    if op == "dense":
        return s["h"].to_dense()
    if s["case"]["loop"]:
        return s["h"].matmul(s["x"], workspace=s["ws"], check=False)
    return s["h"].matmul(s["x"])


def work(case):
    if case["op"] == "batch":
        specs = [(n, p, _Arrays(n, case["dim"], case["leaf"], 7 * k)) for k, (n, p) in enumerate(_batch_specs(case))]
    else:
        specs = [(case["n"], case.get("rhs", 0), _Arrays(case["n"], case["dim"], case["leaf"], 7))]
    total = {"bytes": 0, "flops": 0}
    for n, p, a in specs:
        b, macs = a.bytes_and_codes()
        if case["op"] == "dense":
            total["bytes"] += b + 8 * n * n
            total["flops"] += 2 * int((a.m * a.k).sum())
        else:
            total["bytes"] += b + 16 * n * p
            total["flops"] += 2 * macs * p
    return total


def exact(case, seed):
    dev = torch.device("cuda", DEVICE)
    if case["op"] == "batch":
        x, out, at = torch.from_numpy(_rhs(case, seed)).to(dev), [], 0
        for k, (n, p) in enumerate(_batch_specs(case)):
            a = _Arrays(n, case["dim"], case["leaf"], seed + 100 * k)
            out.append(a.exact_apply(x[at:at + n * p].reshape(n, p)).reshape(-1))
            at += n * p
        return torch.cat(out)
    a = _Arrays(case["n"], case["dim"], case["leaf"], seed)
    if case["op"] == "dense":
        return a.exact_dense().cpu().numpy()
    x = torch.from_numpy(_rhs(case, seed)).to(dev)
    y = a.exact_apply(x.reshape(case["n"], -1)).reshape(x.shape)
    return y.cpu().numpy() if case["io"] == "host" else y
