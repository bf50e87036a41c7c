"""Host-side construction of "dense plans" for ``e3b_dense_fwd`` (layouts in csrc/dense.cu and csrc/dense_tile.cu).

The first part of a plan lists, per output irrep, the (path, u, v) triples that are contracted against the
shared weights, and for every path the Clebsch-Gordan non-zeros (with the path coefficient
folded in) that turn a pair of input rows into the left operand of that contraction.  The second part describes the
same contraction by whole paths, cut into chunks of 32 channels, for the register-tile kernels; the plan's last word
is its offset.
"""
from __future__ import annotations

import struct
from itertools import chain
from typing import List, Optional, Sequence, Tuple

import numpy as np

from ._irreps import Irreps
from ._wigner import wigner_3j_numpy

MAGIC = 0x65336251          # (..50: plans of the first part alone)


_FLOAT, _INT = struct.Struct("<f"), struct.Struct("<i")


def _f2i(v: float) -> int:
    return _INT.unpack(_FLOAT.pack(v))[0]


class _Builder:
    def __init__(self, d1: int, d2: int, dout: int):
        self.d1, self.d2, self.dout = d1, d2, dout
        self.groups: List[List[int]] = []
        self.kent: List[int] = []
        self.paths: List[List[Tuple[int, int]]] = []   # per path, per k: (cg_start, cg_count)
        self.cg: List[int] = []
        self.max_k = 0
        # second part
        self.wpaths: List[dict] = []
        self.wgroups: List[Tuple[int, int, int, List[int]]] = []     # out_off, mul_out, dim3, whole paths

    def add_whole_path(self, **path) -> int:
        """x1off, m1, d1; x2off (-1: no second operand), m2, d2; out_off, mo, d3; wbase, su, sv, sw; c [d1, d2, d3] or coef."""
        self.wpaths.append(path)
        return len(self.wpaths) - 1

    def add_whole_group(self, out_off: int, mul_out: int, dim3: int, paths: Sequence[int]):
        self.wgroups.append((out_off, mul_out, dim3, list(paths)))

    def add_path(self, per_k: Sequence[Sequence[Tuple[int, int, float]]]) -> int:
        entry = []
        for triples in per_k:
            start = len(self.cg) // 3
            for i, j, c in triples:
                self.cg += [i, j, _f2i(c)]
            entry.append((start, len(triples)))
        self.paths.append(entry)
        return len(self.paths) - 1

    def add_group(self, out_off: int, mul_out: int, dim3: int, kents: Sequence[Tuple[int, int, int, int]], w_stride: int = 1):
        start = len(self.kent) // 4
        self.kent += chain.from_iterable(kents)
        self.groups.append([out_off, mul_out, dim3, len(kents), start, w_stride])
        self.max_k = max(self.max_k, len(kents))

    def finish(self) -> np.ndarray:
        header = 12
        off_groups = header
        off_kent = off_groups + 6 * len(self.groups)
        off_pathk = off_kent + len(self.kent)
        n_paths = len(self.paths)
        pathk_words: List[int] = []
        dir_words = []
        base = off_pathk + n_paths
        for entry in self.paths:
            dir_words.append(base + len(pathk_words))
            for s, c in entry:
                pathk_words += [s, c]
        off_cg = base + len(pathk_words)
        second, where = self._second_part(off_cg + len(self.cg))
        total = off_cg + len(self.cg) + len(second) + 1
        words = [MAGIC, self.d1, self.d2, self.dout, len(self.groups), n_paths, total,
                 off_groups, off_kent, off_pathk, off_cg, self.max_k]
        for g in self.groups:
            words += g
        words += self.kent + dir_words + pathk_words + self.cg + second + [where]
        assert len(words) == total
        return np.asarray(words, dtype=np.int64).astype(np.int32)

    def _second_part(self, base: int) -> Tuple[List[int], int]:
        """Words of the second part, which starts at word ``base`` of the plan, and the offset of its header."""
        words: List[int] = []

        def segments(lists) -> int:
            """Pairs (index, coefficient) of every list, then the word offsets of the lists' ends; returns where those start."""
            ends = [base + len(words)]
            for pairs in lists:
                for i, c in pairs:
                    words.extend([i, _f2i(c)])
                ends.append(base + len(words))
            at = base + len(words)
            words.extend(ends)
            return at

        swapped = self._swaps()
        if swapped:
            paths = [dict(p, x1off=p["x2off"], m1=p["m2"], d1=p["d2"], x2off=p["x1off"], m2=p["m1"], d2=p["d1"], su=p["sv"], sv=p["su"],
                          c=p["c"].transpose(1, 0, 2)) for p in self.wpaths]
        else:
            paths = self.wpaths
        rows, d1max, d3max = [], 1, 1
        for p in paths:
            d1, d2, d3 = p["d1"], p["d2"], p["d3"]
            d1max, d3max = max(d1max, d1), max(d3max, d3)
            ki = jj = 0
            if p["x2off"] >= 0:
                c = p["c"].tolist()
                ki = segments([[(j, c[i][j][k]) for j in range(d2) if c[i][j][k] != 0.0] for k in range(d3) for i in range(d1)])
                jj = segments([[(i * d3 + k, c[i][j][k]) for i in range(d1) for k in range(d3) if c[i][j][k] != 0.0] for j in range(d2)])
            rows.append([d1, d2, d3, p["su"], p["sw"], ki, jj, p["x1off"], p["m1"], p["x2off"], p["m2"], p["out_off"], p["mo"],
                         p["wbase"], p["sv"], _f2i(p.get("coef", 0.0))])
        chunks, groups = [], []
        for out_off, mo, d3, members in self.wgroups:
            first = len(chunks)
            for n in members:
                p = paths[n]
                for v in range(p["m2"]):
                    x2off = p["x2off"] + v * p["d2"] if p["x2off"] >= 0 else -1
                    for u0 in range(0, p["m1"], 32):
                        chunks.append([n, p["x1off"] + u0 * p["d1"], min(32, p["m1"] - u0), x2off,
                                       p["wbase"] + u0 * p["su"] + v * p["sv"], int(u0 == 0)])
            groups.append([out_off, mo, d3, first, len(chunks) - first, 0])
        # the paths that leave each block of the first operand (operand gradients of a product)
        blocks = {}
        for n, p in enumerate(paths):
            if p["x2off"] >= 0 and p["m1"] * p["m2"] * p["mo"] > 0:
                blocks.setdefault((p["x1off"], p["m1"], p["d1"]), []).append(n)
        in_paths = [n for members in blocks.values() for n in members]
        in_groups, at = [], 0
        for (x1off, m1, d1), members in blocks.items():
            in_groups.append([x1off, m1, d1, at, len(members)])
            at += len(members)
        covered = sum(m1 * d1 for _, m1, d1 in blocks) == (self.d2 if swapped else self.d1)
        offs = []
        for table in (groups, chunks, rows, in_groups):
            offs.append(base + len(words))
            for r in table:
                words.extend(r)
        offs.append(base + len(words))
        words.extend(in_paths)
        header = base + len(words)
        words.extend([len(groups), offs[0], len(chunks), offs[1], len(rows), offs[2], len(in_groups), offs[3], d1max, d3max, offs[4],
                      int(covered), int(swapped), sum(c[2] for c in chunks)])
        return words, header

    def _swaps(self) -> bool:
        """Whether the second part describes a product with its operands exchanged: the kernels take 32 channels of the first
        operand at a time for every single channel of the second, so the one that gives fewer such chunks goes first (8 x 64
        channels: 64 chunks of 8 a path, or 16 of 32; 10,000 rows, l <= 2, forward 5.5 -> 0.78 ms, all gradients 18 -> 3.4; 1 x 128
        -> 32 channels 16 -> 0.22 and 57 -> 0.70 ms), unless that takes an irrep of l > 3 into the first place, where the row
        kernels do not have it."""
        paths = [p for p in self.wpaths if p["m1"] * p["m2"] * p["mo"] > 0]
        if not paths or paths[0]["x2off"] < 0:
            return False
        if max(p["d2"] for p in paths) > 7 >= max(p["d1"] for p in paths):
            return False
        return sum(p["m1"] * -(-p["m2"] // 32) for p in paths) < sum(p["m2"] * -(-p["m1"] // 32) for p in paths)


def uvw_plan(spec, instruction_ids: Optional[Sequence[int]] = None) -> Tuple[np.ndarray, List[int]]:
    """Plan of the 'uvw' paths of a `TPSpec`.  Returns (plan words, output irreps written)."""
    i1, i2, io = spec.irreps_in1, spec.irreps_in2, spec.irreps_out
    o1, o2, oo = i1.offsets(), i2.offsets(), io.offsets()
    woffs = spec.weight_offsets()
    b = _Builder(i1.dim, i2.dim, io.dim)
    live = [(n, ins) for n, ins in spec.live_instructions() if ins.connection_mode == "uvw"]
    if instruction_ids is not None:
        live = [(n, ins) for n, ins in live if n in set(instruction_ids)]
    written = sorted({ins.i_out for _, ins in live})
    for out_idx in written:
        kents, whole = [], []
        mul_out, ir_out = io[out_idx]
        for n, ins in live:
            if ins.i_out != out_idx:
                continue
            (m1, ir1), (m2, ir2) = i1[ins.i_in1], i2[ins.i_in2]
            c = wigner_3j_numpy(ir1.l, ir2.l, ir_out.l) * ins.path_weight
            cl, x1off, x2off, d1, d2 = c.tolist(), o1[ins.i_in1], o2[ins.i_in2], ir1.dim, ir2.dim
            pid = b.add_path([[(i, j, cl[i][j][k]) for i in range(d1) for j in range(d2) if cl[i][j][k] != 0.0]
                              for k in range(ir_out.dim)])
            kents += [(pid, x1off + u * d1, x2off + v * d2, woffs[n] + (u * m2 + v) * mul_out) for u in range(m1) for v in range(m2)]
            whole.append(b.add_whole_path(x1off=o1[ins.i_in1], m1=m1, d1=ir1.dim, x2off=o2[ins.i_in2], m2=m2, d2=ir2.dim,
                                          out_off=oo[out_idx], mo=mul_out, d3=ir_out.dim, wbase=woffs[n], su=m2 * mul_out, sv=mul_out,
                                          sw=1, c=c))
        b.add_group(oo[out_idx], mul_out, ir_out.dim, kents, 1)
        b.add_whole_group(oo[out_idx], mul_out, ir_out.dim, whole)
    return b.finish(), written


def linear_plan(irreps_in: Irreps, irreps_out: Irreps, instructions, transpose: bool = False) -> Tuple[np.ndarray, List[int]]:
    """Plan of a Linear (weight instructions only).  ``transpose``: the map from output
    cotangents back to input cotangents (same weights, read with a stride).  In the first part of a transposed plan a
    target may have several groups (to be added up); in the second part, which ``e3b_dense_fwd`` runs, it has one."""
    oi, oo = irreps_in.offsets(), irreps_out.offsets()
    woff, offs = 0, []
    for ins in instructions:
        if ins.i_in == -1:
            offs.append(-1)
            continue
        offs.append(woff)
        woff += ins.path_shape[0] * ins.path_shape[1]
    src, dst = (irreps_out, irreps_in) if transpose else (irreps_in, irreps_out)
    so, do = (oo, oi) if transpose else (oi, oo)
    b = _Builder(src.dim, 0, dst.dim)
    live = [(n, ins) for n, ins in enumerate(instructions) if ins.i_in != -1 and 0 not in ins.path_shape
            and irreps_in[ins.i_in].dim > 0 and irreps_out[ins.i_out].dim > 0]
    targets = sorted({(ins.i_in if transpose else ins.i_out) for _, ins in live})
    for t in targets:
        mul_t, ir = dst[t]
        # a group reads W with one stride: forward 1; transposed the output multiplicity of the path, so the
        # paths out of one input irrep are grouped by it (the caller accumulates the groups of a target)
        by_stride, whole = {}, []
        for n, ins in live:
            if (ins.i_in if transpose else ins.i_out) != t:
                continue
            s = ins.i_out if transpose else ins.i_in
            mul_s = src[s].mul
            pid = b.add_path([[(k, 0, float(ins.path_weight))] for k in range(ir.dim)])
            mul_in, mul_out = ins.path_shape
            kents = by_stride.setdefault(mul_out if transpose else 1, [])
            for q in range(mul_s):
                # forward: W[u=q, w] contiguous in w; transpose: W[u, w=q] strided by mul_out in u
                wbase = offs[n] + (q if transpose else q * mul_out)
                kents.append((pid, so[s] + q * ir.dim, -1, wbase))
            whole.append(b.add_whole_path(x1off=so[s], m1=mul_s, d1=ir.dim, x2off=-1, m2=1, d2=1, out_off=do[t], mo=mul_t, d3=ir.dim,
                                          wbase=offs[n], su=1 if transpose else mul_out, sv=0, sw=mul_out if transpose else 1,
                                          coef=float(ins.path_weight)))
        for stride, kents in by_stride.items():
            b.add_group(do[t], mul_t, ir.dim, kents, stride)
        b.add_whole_group(do[t], mul_t, ir.dim, whole)
    return b.finish(), targets
