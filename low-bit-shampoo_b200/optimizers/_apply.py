"""Plan of the part of a step that runs every time (qt_apply_run): preconditioned directions of all gradient
blocks, norm grafting and the AdamW / SGD tail, five launches over tables laid out once.

A plan belongs to one list of parameters with one pattern of active preconditioners.  It owns the tables, the
operand-plane workspace and the buffer of directions; from step to step only the addresses of the gradients (and
the step's scalars) change.  Nothing computed in one step is kept for the next: planes, exponents and norms are
formed anew from the stored state and the gradients.

Blocks with two 4/8-bit preconditioners are multiplied on the tensor cores, blocks of one shape forming a group;
where an order is below min_lowbit_size (a plain fp32 preconditioner) both products run in fp32.
"""
import ctypes as ct
import math
from collections import defaultdict

import numpy as np
import torch

import qtensor.functional as F
from optimizers import _gemm

# Planes of the blocks of one wave: P0, P1, G and T, two 16-bit planes each.  Larger models go through the same
# workspace in several waves, so that it stays bounded whatever the model.
WAVE_BYTES = 3 << 29
PIECE = 1 << 14                 # elements per work item of the streaming launches
MAX_GROUPS = 256
SIMT_FLOPS = 1 << 30            # largest block taken by the fp32 product

_ITEM = np.dtype([("type", "i4"), ("param", "i4"), ("rows", "i4"), ("cols", "i4"), ("ld", "i4"), ("aux0", "i4"), ("aux1", "i4"),
                  ("aux2", "i4"), ("off", "i8"), ("p0", "i8"), ("p1", "i8"), ("p2", "i8"), ("p3", "i8"), ("p4", "i8")])
_TENSOR = np.dtype([("p", "i8"), ("m", "i8"), ("v", "i8"), ("d", "i8"), ("numel", "i8"), ("param", "i4"), ("flags", "i4"),
                    ("g0", "i4"), ("g1", "i4"), ("r0", "i4"), ("r1", "i4"), ("pad", "i8")])
GRAD_STAT, STATE_EXP, SIMT_FIRST, SPLIT, DEQUANT, SIMT_SECOND = range(6)
GROUP_BYTES = 640               # the stride of the groups in device memory (include/qtensor_b200.h)


class Wave(ct.Structure):
    _fields_ = [("plane_items", ct.c_void_p), ("groups1", ct.c_void_p), ("groups2", ct.c_void_p), ("tiles1", ct.c_void_p),
                ("tiles2", ct.c_void_p), ("n_plane_items", ct.c_int), ("n_groups", ct.c_int), ("n_tiles1", ct.c_int),
                ("n_tiles2", ct.c_int), ("bn1", ct.c_int), ("bn2", ct.c_int)]


class Desc(ct.Structure):
    _fields_ = [(k, ct.c_void_p) for k in ("stat_items", "waves", "grads", "code", "part_amax", "part_ss", "pexp", "gexp", "tensors",
                                           "chunk_tensor", "chunk_index", "ranges", "scalars")] + \
               [(k, ct.c_int) for k in ("n_stat_items", "n_waves", "target", "n_chunks", "chunk_elems", "kind", "nesterov", "reserved")] + \
               [(k, ct.c_float) for k in ("s0", "s1", "s2", "beta1", "beta2", "a1", "a2", "eps", "lr", "momentum", "weight_decay")]


class PointerTable:
    """Device copy of a list of addresses, refreshed without blocking when they change: the host may run steps ahead
    of the device, so a pinned buffer is written again only after the copy that read it has completed."""

    def __init__(self, n, device):
        self.dev = torch.zeros(n, dtype=torch.int64, device=device)
        self.ptrs = None
        self.ring, self.next = [], 0

    def set(self, ptrs):
        if ptrs == self.ptrs:
            return
        if len(self.ring) < 4:
            self.ring.append([torch.empty(len(ptrs), dtype=torch.int64).pin_memory(), torch.cuda.Event()])
            slot = self.ring[-1]
        else:
            slot = self.ring[self.next]
            self.next = (self.next + 1) % len(self.ring)
            slot[1].synchronize()
        slot[0].numpy()[:] = ptrs
        self.dev.copy_(slot[0], non_blocking=True)
        slot[1].record(torch.cuda.current_stream(self.dev.device))
        self.ptrs = ptrs


class _Block:
    __slots__ = ("param", "r0", "c0", "m", "k", "s0", "s1", "stat", "index")


def _tile_width(waves, sms):
    """Tile width of one product of all blocks; waves: lists of (rows, columns, K, blocks).  A tile's time is linear in
    K: operand delivery from L2 per k - wider tiles need less of it per result - and the part of its epilogue that the next
    tile's products do not hide.  Tiles go to the SMs in turn, so a plan's time is the longest sum over an SM.  Microseconds of
    both products, 128 / 192 / 256: ViT-B/32 905 / 891 / 849, ResNet-34 215 / 225 / 208, 8 x (512 x 1000) 52 / 65 / 56."""
    def cost(width, per_k, fixed):
        total = 0.0
        for groups in waves:
            times = np.concatenate([np.full(math.ceil(m / 128) * math.ceil(n / width) * count, per_k * k + fixed) for m, n, k, count in groups])
            total += np.pad(times, (0, -len(times) % sms)).reshape(-1, sms).sum(0).max()
        return total
    if not waves:
        return 128
    return min(((cost(w, *c), w) for w, c in ((128, (0.0147, 1.0)), (192, (0.0174, 1.9)), (256, (0.0215, 3.5)))))[1]


def _up(x, q):
    return (x + q - 1) // q * q


def _storage(arena, slot):
    """(codes or fp32 matrix, scales, diagonal) addresses and bits | block shift << 8 of one stored matrix."""
    if not arena.lowbit:
        return arena.var.data_ptr() + 4 * slot * arena.n * arena.n, 0, 0, 32
    return (arena.var.data_ptr() + slot * arena.row_bytes, arena.absmax.data_ptr() + 4 * slot * arena.n * arena.nb,
            arena.diag.data_ptr() + 4 * slot * arena.n, arena.bits | (arena.blocksize.bit_length() - 1) << 8)


def _collect(params, states, grafted):
    """Gradient blocks in parameter order, or None if some block fits neither kind of product."""
    blocks = []
    for i, (p, st) in enumerate(zip(params, states)):
        pre = st['preconditioner']
        if not (grafted[i] and pre.preconditioners):
            continue
        for j, (rs, cs) in enumerate(pre._partitioner.block_slices()):
            b = _Block()
            b.param, b.r0, b.c0 = i, rs.start, cs.start
            b.m, b.k = rs.stop - rs.start, cs.stop - cs.start
            b.s0, b.s1 = pre._slots[2 * j], pre._slots[2 * j + 1]
            a0, a1 = b.s0[0].prec, b.s1[0].prec
            if any(not a.lowbit and a.bits != 32 for a in (a0, a1)):
                return None
            if not (a0.lowbit and a1.lowbit) and 2 * b.m * b.k * (b.m + b.k) > SIMT_FLOPS:
                return None
            blocks.append(b)
    return blocks


class ApplyPlan:
    def __init__(self, params, states, grafted, kind, moments):
        """grafted[i]: parameter i has an active preconditioner (or none) and its step is not before start_prec_step.
        kind 0: AdamW, 1: SGD.  moments: names of the moment tensors in the states."""
        self.ok = False
        blocks = _collect(params, states, grafted)
        if blocks is None:
            return
        self.params, self.states, self.kind, self.moments = params, states, kind, moments
        self.device = dev = params[0].device
        self._keep = []
        numels = [p.numel() for p in params]
        widths = {}                                           # row length of the matrix a parameter is reshaped to
        for b in blocks:
            if b.param not in widths:
                widths[b.param] = numels[b.param] // states[b.param]['preconditioner']._partitioner._shape[0]

        # directions: one buffer, parameters on 128-byte boundaries
        off, d_off = 0, {}
        for i in widths:
            d_off[i] = off
            off += _up(numels[i], 32)
        self.directions = torch.empty(max(off, 1), dtype=torch.float32, device=dev)
        d_base = self.directions.data_ptr()

        # ---- pieces of the gradients: magnitudes and sums of squares
        stat, g_range = [], [(0, 0)] * len(params)
        by_param = defaultdict(list)
        for b in blocks:
            by_param[b.param].append(b)
        pieces = 0

        def piece(param, offset, rows, cols, ld):
            nonlocal pieces
            stat.append((GRAD_STAT, param, rows, cols, ld, pieces, 0, 0, offset, 0, 0, 0, 0, 0))
            pieces += 1
        for i, n in enumerate(numels):
            if not grafted[i]:
                continue
            first = pieces
            for b in by_param.get(i, ()):
                ld, b0 = widths[i], pieces
                step = max(1, PIECE // b.k)
                for r in range(0, b.m, step):
                    rows = min(step, b.m - r)
                    o = (b.r0 + r) * ld + b.c0
                    if b.k == ld:
                        piece(i, o, 1, rows * b.k, rows * b.k)
                    else:
                        piece(i, o, rows, b.k, ld)
                b.stat = (b0, pieces - b0)
            if i not in by_param:
                for o in range(0, n, PIECE):
                    piece(i, o, 1, min(PIECE, n - o), min(PIECE, n - o))
            g_range[i] = (first, pieces)

        # ---- groups of equal shape (and row length of the parameter: the pitch of the result), cut into waves that share one plane workspace
        groups, simt = defaultdict(list), []
        for b in blocks:
            if b.s0[0].prec.lowbit and b.s1[0].prec.lowbit:
                groups[(b.m, b.k, widths[b.param])].append(b)
            else:
                simt.append(b)
        order = sorted(groups.items(), key=lambda kv: -(kv[0][0] * kv[0][1] * (kv[0][0] + kv[0][1])))
        waves, used = [[]], 0
        for (m, k, _), bs in order:
            lm, lk = _up(m, 16), _up(k, 16)
            size = 4 * (m * lm + k * lk + 2 * m * lk)
            while bs:
                room = int(max(0, WAVE_BYTES - used) // size)
                if waves[-1] and (room == 0 or len(waves[-1]) == MAX_GROUPS):
                    waves.append([])
                    used = 0
                    continue
                take = bs[: max(1, room)]
                bs = bs[len(take):]
                waves[-1].append((m, k, take))
                used += size * len(take)
        waves = [w for w in waves if w]
        tc = sum(len(g[2]) for w in waves for g in w)
        ints = torch.zeros(max(1, 4 * tc), dtype=torch.int32, device=dev)    # exponents: P0, P1, G, T
        self._keep.append(ints)
        exp = lambda kind_, i: ints.data_ptr() + 4 * (kind_ * tc + i)

        sms = torch.cuda.get_device_properties(dev).multi_processor_count
        bn1 = _tile_width([[(m, k, m, len(bs)) for m, k, bs in w] for w in waves], sms)
        bn2 = _tile_width([[(m, k, k, len(bs)) for m, k, bs in w] for w in waves], sms)

        # ---- work items and groups of every wave
        ranges = defaultdict(list)                            # per parameter: pieces of the direction's sum of squares
        parts = pieces
        wave_tables, max_elems, index = [], 0, 0
        layout = []                                           # deferred until the workspace exists
        for w in waves:
            cursor, entry = 0, []
            for m, k, bs in w:
                lm, lk, n = _up(m, 16), _up(k, 16), len(bs)
                regions = []
                for rows, ld in ((m, lm), (k, lk), (m, lk), (m, lk)):          # P0, P1, G, T
                    regions.append((cursor, cursor + _up(n * rows * ld, 64)))
                    cursor += 2 * _up(n * rows * ld, 64)
                nt = math.ceil(m / 128) * math.ceil(k / bn2)
                for j, b in enumerate(bs):
                    b.index = index + j
                    ranges[b.param].append((parts + 8 * nt * j, 8 * nt))
                entry.append((m, k, bs, regions, index, parts))
                parts += 8 * nt * n
                index += n
            max_elems = max(max_elems, cursor)
            layout.append(entry)
        ws = torch.empty(max(max_elems, 1), dtype=torch.int16, device=dev)
        self._keep.append(ws)
        wb = ws.data_ptr()

        for b in simt:
            nt = math.ceil(b.m / 32) * math.ceil(b.k / 32)
            ranges[b.param].append((parts, nt))
            b.index = parts
            parts += nt
        self.part_ss = torch.zeros(max(parts, 1), dtype=torch.float32, device=dev)
        self.part_amax = torch.zeros(max(pieces, 1), dtype=torch.float32, device=dev)
        part = lambda i: self.part_ss.data_ptr() + 4 * i

        simt_second = []
        for b in simt:
            T = torch.empty(b.m, b.k, dtype=torch.float32, device=dev)
            self._keep.append(T)
            ld = widths[b.param]
            p0, p1 = _storage(b.s0[0].prec, b.s0[1]), _storage(b.s1[0].prec, b.s1[1])
            o = b.r0 * ld + b.c0
            for tm in range(math.ceil(b.m / 32)):
                for tn in range(math.ceil(b.k / 32)):
                    stat.append((SIMT_FIRST, b.param, b.m, b.k, ld, p0[3], tm, tn, o, p0[0], p0[1], p0[2], 0, T.data_ptr()))
                    simt_second.append((SIMT_SECOND, b.param, b.m, b.k, ld, p1[3], tm, tn, b.index + tm * math.ceil(b.k / 32) + tn,
                                        p1[0], p1[1], p1[2], d_base + 4 * (d_off[b.param] + o), T.data_ptr()))

        lib = F.lib
        for entry in layout:
            items, g1, g2, t1, t2 = [], [], [], [0], [0]
            for m, k, bs, regions, i0, part0 in entry:
                lm, lk, n = _up(m, 16), _up(k, 16), len(bs)
                dptrs, wide = [], 1
                for j, b in enumerate(bs):
                    ld = widths[b.param]
                    o = b.r0 * ld + b.c0
                    dptrs.append(d_base + 4 * (d_off[b.param] + o))
                    wide &= int(ld % 8 == 0 and o % 8 == 0)
                    step = max(1, PIECE // k)
                    for r in range(0, m, step):
                        at = 2 * (j * m + r) * lk
                        items.append((SPLIT, b.param, min(step, m - r), k, ld, b.stat[0], b.stat[1], b.index, o + r * ld,
                                      wb + 2 * regions[2][0] + at, wb + 2 * regions[2][1] + at, lk, int(r == 0), 0))
                    for side, (arena, slot), order_, lo_ in ((0, (b.s0[0].prec, b.s0[1]), m, lm), (1, (b.s1[0].prec, b.s1[1]), k, lk)):
                        var, absmax, diag, bits = _storage(arena, slot)
                        e = side * tc + b.index
                        stat.append((STATE_EXP, 0, arena.n * arena.nb, arena.n, 0, e, 0, 0, 0, absmax, diag, 0, 0, 0))
                        step = max(1, 2 * PIECE // order_)
                        at = 2 * j * order_ * lo_
                        for r in range(0, order_, step):
                            items.append((DEQUANT, 0, min(step, order_ - r), order_, lo_, bits, e, 0, r, var, absmax, diag,
                                          wb + 2 * regions[side][0] + at, wb + 2 * regions[side][1] + at))
                dp = torch.tensor(dptrs, dtype=torch.int64).to(dev)
                self._keep.append(dp)
                count = lambda bn: math.ceil(m / 128) * math.ceil(k / bn) * n
                rel = _gemm.F16_MAX_EXP - _gemm._ceil_log2(m) - 2 * _gemm.SPLIT_TARGET
                at = lambda q, h: wb + 2 * regions[q][h]
                for lst, tl, bn, args in (
                        (g1, t1, bn1, (at(0, 0), at(0, 1), lm, m * lm, at(2, 0), at(2, 1), lk, m * lk, m, k, m, n, bn1, t1[-1], exp(0, i0), exp(2, i0),
                                  at(3, 0), at(3, 1), lk, m * lk, exp(3, i0), rel, None, 0, 0, None)),
                        (g2, t2, bn2, (at(3, 0), at(3, 1), lk, m * lk, at(1, 0), at(1, 1), lk, k * lk, m, k, k, n, bn2, t2[-1], exp(3, i0), exp(1, i0),
                                  None, None, 0, 0, None, 0, dp.data_ptr(), widths[bs[0].param], wide, part(part0)))):
                    buf = ct.create_string_buffer(GROUP_BYTES)
                    F._check(lib.qt_apply_group(buf, *args), "apply group")
                    lst.append(buf.raw)
                    tl.append(tl[-1] + count(bn))
            wave_tables.append((items, g1, g2, t1, t2))
        if simt_second:
            if not wave_tables:
                wave_tables.append(([], [], [], [0], [0]))
            wave_tables[0][0].extend(simt_second)

        # ---- upload
        def up(data):
            t = torch.from_numpy(np.frombuffer(data, dtype=np.uint8).copy()).to(dev) if len(data) else torch.zeros(8, dtype=torch.uint8, device=dev)
            self._keep.append(t)
            return t.data_ptr()
        # slowest items first: the fp32 products, then the state's exponents, then the streaming pieces
        rank = {SIMT_FIRST: 0, SIMT_SECOND: 0, STATE_EXP: 1, GRAD_STAT: 2, DEQUANT: 3, SPLIT: 4}
        table = lambda rows: np.array(sorted(rows, key=lambda r: rank[r[0]]), dtype=_ITEM).tobytes()
        self.waves = (Wave * max(1, len(wave_tables)))()
        for wv, (items, g1, g2, t1, t2) in zip(self.waves, wave_tables):
            wv.plane_items, wv.n_plane_items = up(table(items)), len(items)
            wv.groups1, wv.groups2, wv.n_groups, wv.bn1, wv.bn2 = up(b"".join(g1)), up(b"".join(g2)), len(g1), bn1, bn2
            wv.tiles1, wv.tiles2 = up(np.array(t1, dtype=np.int32).tobytes()), up(np.array(t2, dtype=np.int32).tobytes())
            wv.n_tiles1, wv.n_tiles2 = t1[-1], t2[-1]
        total = sum(numels)
        chunk = min(1 << 15, max(1 << 11, _up(total // (148 * 16), 1024)))
        ct_, ci_, rr, self._tensors = [], [], [], np.zeros(len(params), dtype=_TENSOR)
        for i, n in enumerate(numels):
            for c in range((n + chunk - 1) // chunk):
                ct_.append(i)
                ci_.append(c)
            r0 = len(rr)
            rr += ranges.get(i, [])
            flags = int(grafted[i]) | (2 if i not in widths else 0)
            self._tensors[i] = (0, 0, 0, d_base + 4 * d_off[i] if i in widths else 0, n, i, flags, *g_range[i], r0, len(rr), 0)
        self._tensor_table = torch.zeros(self._tensors.nbytes, dtype=torch.uint8, device=dev)
        self._state_ptrs = None
        d = self.desc = Desc()
        d.stat_items, d.n_stat_items = up(table(stat)), len(stat)
        d.waves, d.n_waves = ct.addressof(self.waves), len(wave_tables)
        codes = [c.prec.code for b in blocks for c in (b.s0[0], b.s1[0]) if c.prec.lowbit]
        d.code = codes[0].data_ptr() if codes else None
        self._keep.append(codes[:1])
        d.part_amax, d.part_ss = self.part_amax.data_ptr(), self.part_ss.data_ptr()
        d.pexp, d.gexp = ints.data_ptr(), exp(2, 0)
        d.tensors = self._tensor_table.data_ptr()
        d.chunk_tensor, d.chunk_index = up(np.array(ct_, dtype=np.int32).tobytes()), up(np.array(ci_, dtype=np.int32).tobytes())
        d.ranges = up(np.array(rr, dtype=np.int32).tobytes())
        d.target, d.n_chunks, d.chunk_elems, d.kind = _gemm.SPLIT_TARGET, len(ct_), chunk, kind
        self.ok = True

    def bind_state(self):
        """Addresses of parameters and moments into the tail's table; False if one of them is not a dense fp32 tensor
        on this device."""
        names = self.moments
        ptrs = [p.data_ptr() for p in self.params]
        for name in names:
            ptrs += [st[name].data_ptr() for st in self.states]
        if ptrs == self._state_ptrs:
            return True
        n = len(self.params)
        for i, (p, st) in enumerate(zip(self.params, self.states)):
            for t in (p, *(st[name] for name in names)):
                if not (t.dtype == torch.float32 and t.is_contiguous() and t.device == self.device and t.numel() == self._tensors[i]["numel"]):
                    return False
        if torch.cuda.is_current_stream_capturing():
            return False
        self._tensors["p"], self._tensors["m"] = ptrs[:n], ptrs[n: 2 * n]
        self._tensors["v"] = ptrs[2 * n:] if len(names) > 1 else ptrs[n: 2 * n]
        self._tensor_table.copy_(torch.from_numpy(self._tensors.view(np.uint8).copy()))
        self._state_ptrs = ptrs
        return True

    def run(self, grads, stream, scalars=None, **hyper):
        """`grads`: device table of the gradients' addresses; hyper: scalar fields of the descriptor."""
        d = self.desc
        d.grads = grads.data_ptr()
        d.scalars = scalars.data_ptr() if scalars is not None else None
        for k, v in hyper.items():
            setattr(d, k, v)
        rc = F.lib.qt_apply_run(ct.byref(d), stream)
        if rc != 0:
            F._check(rc, "apply step")
