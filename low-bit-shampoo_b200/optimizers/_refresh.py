"""Plan of the refresh of the eigen-factor statistics and their inverse roots: per order class one host call
(qt_refresh_class) over tables laid out once.  Only the addresses of the gradients change from step to step; every
intermediate result lives in a workspace that is allocated for the call.
"""
import ctypes as ct
from collections import defaultdict

import numpy as np
import torch

import qtensor.functional as F
from optimizers import _engine as E
from optimizers._apply import GRAD_STAT, PIECE, SPLIT, _ITEM, _up

MAX_ORDER = 1216                # the panel kernel's (see _qr.py)


class Group(ct.Structure):
    _fields_ = [("slots", ct.c_void_p), ("hi_off", ct.c_longlong), ("lo_off", ct.c_longlong)] + \
               [(k, ct.c_int) for k in ("rows", "cols", "count", "axis", "first", "reserved")]


class Desc(ct.Structure):
    _fields_ = [(k, ct.c_void_p) for k in ("stat_codes", "stat_absmax", "prec_codes", "prec_absmax", "prec_diag", "S", "keep_idx", "max_eig",
                                           "code", "groups", "grad_stat_items", "grad_split_items", "grads", "part_amax", "part_ss", "gexp")] + \
               [(k, ct.c_longlong) for k in ("stride_codes", "grad_plane_bytes")] + \
               [(k, ct.c_int) for k in ("n", "count", "keep", "bits", "blocksize", "rect_t1", "rect_t2", "do_stat", "do_root", "n_groups",
                                        "n_grad_stat", "n_grad_split")] + \
               [(k, ct.c_float) for k in ("w1", "w2", "eps", "inv_p")]


def plannable(cls, inv_root_mode):
    s, p = cls.stat, cls.prec
    return (cls.flavour == "s2" and inv_root_mode == 0 and s.lowbit and p.lowbit and s.bits == p.bits and s.blocksize == p.blocksize
            and 64 <= cls.n <= MAX_ORDER and s.var.is_cuda)


class _Batch:
    """Consecutive matrices a .. a+m-1 of a class."""

    def __init__(self, cls, entries, a, m):
        """entries: (slot, param, offset of the block, rows, cols, row length of the parameter, axis), one per matrix, by slot."""
        dev, n = cls.device, cls.n
        self._keep = []
        by_shape = defaultdict(lambda: ([], []))
        for slot, param, off, rows, cols, ld, axis in entries:
            by_shape[(rows, cols, ld)][axis].append((slot - a, param, off))
        stat, split, groups = [], [], []
        pieces = blocks = elems = 0
        for (rows, cols, ld), axes in by_shape.items():
            same = [[e[1:] for e in x] for x in axes]
            shared = same[0] == same[1]                       # square blocks: both sides read the same planes
            regions = {}
            for axis in (0, 1):
                if not axes[axis]:
                    continue
                if axis == 1 and shared:
                    region = regions[0]
                else:
                    lp, cnt = _up(cols, 16), len(axes[axis])
                    hi, lo = elems, elems + _up(cnt * rows * lp, 64)
                    elems = lo + _up(cnt * rows * lp, 64)
                    region = regions[axis] = (hi, lo, blocks)
                    step = max(1, PIECE // cols)
                    for j, (_, param, off) in enumerate(axes[axis]):
                        first = pieces
                        for r in range(0, rows, step):
                            k = min(step, rows - r)
                            o = off + r * ld
                            flat = cols == ld
                            stat.append((GRAD_STAT, param, 1 if flat else k, k * cols if flat else cols, k * cols if flat else ld, pieces, 0, 0, o, 0, 0, 0, 0, 0))
                            at = 2 * (j * rows + r) * lp
                            split.append([SPLIT, param, k, cols, ld, first, 0, blocks, o, 2 * hi + at, 2 * lo + at, lp, int(r == 0), 0])
                            pieces += 1
                        for it in split[len(split) - (pieces - first):]:
                            it[6] = pieces - first
                        blocks += 1
                slots = torch.tensor([e[0] for e in axes[axis]], dtype=torch.int32).to(dev)
                self._keep.append(slots)
                groups.append((slots.data_ptr(), 2 * region[0], 2 * region[1], rows, cols, len(axes[axis]), axis, region[2], 0))

        def up(rows_):
            t = torch.from_numpy(np.frombuffer(np.array([tuple(r) for r in rows_], dtype=_ITEM).tobytes(), dtype=np.uint8).copy()).to(dev)
            self._keep.append(t)
            return t.data_ptr()
        self.groups = (Group * max(1, len(groups)))(*[Group(*g) for g in groups])
        part = torch.zeros(2, max(1, pieces), dtype=torch.float32, device=dev)
        gexp = torch.zeros(max(1, blocks), dtype=torch.int32, device=dev)
        self._keep += [part, gexp, cls]
        s, p = cls.stat, cls.prec
        d = self.desc = Desc()
        d.stat_codes, d.stat_absmax = s.var[a].data_ptr(), s.absmax[a].data_ptr()
        d.prec_codes, d.prec_absmax, d.prec_diag = p.var[a].data_ptr(), p.absmax[a].data_ptr(), p.diag[a].data_ptr()
        d.S, d.keep_idx, d.max_eig = cls.S[a].data_ptr(), cls.keep_idx[a].data_ptr(), cls.max_eig[a].data_ptr()
        d.code, d.groups, d.n_groups = s.code.data_ptr(), ct.addressof(self.groups), len(groups)
        d.grad_stat_items, d.n_grad_stat, d.grad_split_items, d.n_grad_split = up(stat), len(stat), up(split), len(split)
        d.part_amax, d.part_ss, d.gexp = part[0].data_ptr(), part[1].data_ptr(), gexp.data_ptr()
        d.stride_codes, d.grad_plane_bytes = s.row_bytes, 2 * elems
        d.n, d.count, d.keep, d.bits, d.blocksize = n, m, cls.keep, s.bits, s.blocksize
        d.rect_t1, d.rect_t2 = cls.rect_t1, cls.rect_t2
        self.bytes = {}


class RefreshPlan:
    def __init__(self, params, states, inv_root_mode):
        by_class = defaultdict(list)
        for i, (p, st) in enumerate(zip(params, states)):
            pre = st['preconditioner']
            if not pre.statistics:
                continue
            ld = p.numel() // pre._partitioner._shape[0]
            for j, (rs, cs) in enumerate(pre._partitioner.block_slices()):
                for axis in (0, 1):
                    cls, slot = pre._slots[2 * j + axis]
                    by_class[cls].append((slot, i, rs.start * ld + cs.start, rs.stop - rs.start, cs.stop - cs.start, ld, axis))
        self.batches = {}
        self.rest = False                                     # some class is left to the general engine
        for cls, entries in by_class.items():
            entries.sort()
            slots = [e[0] for e in entries]
            if not plannable(cls, inv_root_mode) or slots != list(range(slots[0], slots[0] + len(slots))):
                self.rest = True
                continue
            cap = cls.sub_batch()
            self.batches[cls] = [_Batch(cls, entries[k: k + cap], slots[k], len(entries[k: k + cap])) for k in range(0, len(entries), cap)]

    def run(self, cls, grads, stat, root, w1, w2, eps):
        """Statistics and / or roots of one class on the current stream."""
        lib = F.lib
        for b in self.batches[cls]:
            d = b.desc
            d.grads = grads.data_ptr() if grads is not None else None
            d.do_stat, d.do_root = int(stat), int(root)
            d.w1, d.w2, d.eps, d.inv_p = w1, w2, eps, 0.25
            need = b.bytes.get((stat, root))
            if need is None:
                need = b.bytes[(stat, root)] = lib.qt_refresh_workspace_bytes(ct.byref(d))
            ws = torch.empty(need, dtype=torch.uint8, device=cls.device)
            rc = lib.qt_refresh_class(ct.byref(d), ws.data_ptr(), need, F._stream(ws))
            F._check(rc, f"refresh of order {cls.n}")
